"""The next-event occlusion query runs last and only for estimates that are not exactly
zero: the flags that make an estimate zero (the sphere filter's taper, the hard cut of
correctPhase, the angular filter) and the ones that change what a zero means
(produceDebugImage) against the oracle, which asks first, at the parity tolerance (1e-4
relative L2). Sparse boxes on 30 m: most estimates are out of the taper's reach and walls
hide others."""
import numpy as np
import pytest

from hussar_gb300 import PathTracer, gb300, scenes

pytestmark = pytest.mark.gpu

N, BUDGET = 200, 1 << 15
FLAGS = [dict(), dict(correctPhase=True), dict(correctPhase=True, filterGuiding=False), dict(filteringSphere=False),
         dict(doFiltering=False), dict(produceDebugImage=True), dict(onlyIndirect=False), dict(poDiffraction=True)]


@pytest.fixture(scope="module")
def setup(product_lib, oracle_lib):
    mesh = scenes.boxes_mesh(11, 60, 30.0)
    return gb300.Backend(mesh, None), oracle_lib.Scene(mesh), scenes.plane_poses(3, 12, 30.0)


@pytest.mark.parametrize("flags", FLAGS, ids=lambda f: "-".join("%s=%d" % i for i in f.items()) or "default")
def test_rows_match_the_oracle(setup, flags):
    be, ora, ants = setup
    t = PathTracer()
    t.doGuiding = False
    t.maxDepth = 4
    for k, v in flags.items():
        setattr(t, k, v)
    rf, _ = scenes.rf_77ghz(N, 5e6)
    # the receiver stands apart from the transmitter, so that the direct term exists
    rx = [type(a)(a.position() + np.float32([0.3, 0.2, 0.1]), a.rotation()) for a in ants]
    rows = be.simulate_batch(rf, N, t, ants, rx, [BUDGET] * 3)
    for row, a, b in zip(rows, ants, rx):
        ref = np.asarray(ora.fetch_row(rf, N, a, b, t, BUDGET), np.complex128)
        assert np.linalg.norm(row - ref) <= 1e-4 * np.linalg.norm(ref)
