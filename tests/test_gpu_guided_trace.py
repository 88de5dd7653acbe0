"""Guided runs on the one-thread-per-sample kernel (no geometrical optics, or chosen): their passes
are short, so their work items have to be small enough to reach every SM."""
import time

import pytest

from hussar_gb300 import FrameConfig, PathTracer, Scene, gb300, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel, optics", [(0, False), (1, True)], ids=["no-optics", "chosen"])
def test_passes_fill_the_chip(product_lib, kernel, optics):
    """A guided run of 2^18 samples traces twice as many in five passes, each path a few times as
    long as the plain run's, most of which miss: three to four times its time. With 4096-sample
    items, of which the passes have 4 to 32 for 304 CTAs, it was sixteen to twenty times."""
    w = scenes.dihedral_workload(poses=3)
    took = {}
    product_lib.hsr_set_path_kernel(kernel)
    try:
        for guided in (False, True):
            t = PathTracer()
            t.useGeometricalOptics, t.doGuiding, t.maxDepth = optics, guided, 2
            t.configureFrame(FrameConfig(1, 256, 1))
            be, scene = gb300.Backend(w.mesh, t), Scene(w.rf, w.tx[1], w.rx[1])
            times = []
            for _ in range(8):
                start = time.perf_counter()
                t.run(be, scene, 1 << 18)
                times.append(time.perf_counter() - start)
            took[guided] = min(times)
    finally:
        product_lib.hsr_set_path_kernel(0)
    assert took[True] < 10 * took[False], took
