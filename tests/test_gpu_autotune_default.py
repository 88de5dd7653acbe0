"""Where the default shape wins, the autotuner reports it as it ran and keeps it as the default:
its threshold depends on a launch's bins, its work items on the kernel."""
import ctypes

import numpy as np
import pytest

from hussar_gb300 import PathTracer, _lib, gb300, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1], ids=["wavefront", "per-thread"])
@pytest.mark.parametrize("bins", [256, 1536, 1537, 2048])
def test_the_default_is_reported_as_it_ran(product_lib, kernel, bins):
    """A single work item, on which no shape can gain: a candidate wins only by the noise of its
    timing, so the default does (its time is then the best time) within a few attempts."""
    w = scenes.dihedral_workload(poses=1)
    be = gb300.Backend(w.mesh, None)
    t = PathTracer()
    t.doGuiding, t.maxDepth = False, 2
    rf = scenes.rf_77ghz(bins, 5e6 * bins / 256)[0]
    product_lib.hsr_set_path_kernel(kernel)
    try:
        for _ in range(500):
            got = be.autotune(rf, bins, t, w.tx, w.rx, np.full(1, 256))
            if got["trace_ms"] == got["default_trace_ms"]:
                break
    finally:
        product_lib.hsr_set_path_kernel(0)
    assert got["trace_ms"] == got["default_trace_ms"], got
    threshold = 256 if bins <= 1536 else 128
    assert got["queue_threshold"] == threshold and got["tile"] == (4096 if kernel else 16384), got
    kept = _lib.LaunchConfigC()
    _lib.check(product_lib.hsr_get_launch_config(be.handle, ctypes.byref(kept)))
    assert (kept.tile, kept.ctas_per_sm, kept.queue_threshold) == (0, 0, threshold)
