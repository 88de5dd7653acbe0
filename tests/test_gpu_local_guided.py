"""Guided paths on a dense scene: their weights, pdfs and training sums go with them through the
two-ended path stack and through rays the list leaves to the tree. Against the oracle on
the same guiding tree, at the tolerances of the guided parity tests: 1e-4 relative L2 of a
frame, 1e-4 of the largest leaf sum."""
import numpy as np
import pytest

from hussar_gb300 import FrameConfig, NFAntenna, PathTracer, Scene, gb300, scenes

pytestmark = pytest.mark.gpu

N, BUDGET = 100, 12345


@pytest.fixture(scope="module")
def setup(product_lib, oracle_lib):
    mesh = scenes.boxes_mesh(5, 4000, 20.0)
    return mesh, gb300.Backend(mesh, None), oracle_lib.Scene(mesh), oracle_lib


def tracer(**flags):
    t = PathTracer()
    t.maxDepth = 4
    for k, v in flags.items():
        setattr(t, k, v)
    t.configureFrame(FrameConfig(1, N, 1))
    return t


def sensors():
    out = [NFAntenna(p, scenes.looking(0.3 * k)) for k, p in enumerate(
        [(0.0, 1.0, 0.0), (3.3, 0.4, -2.1), (-4.0, 1.7, 5.0), (2.0, 7.0, 2.0)])]
    return out + scenes.plane_poses(4, 3, 18.0)


@pytest.mark.parametrize("pose", [0, 1, 2, 3])
def test_an_iteration_from_a_trained_tree(setup, pose):
    _, be, ora, oracle_lib = setup
    rf, frame = scenes.rf_77ghz(N, 5e6)
    t, a = tracer(), sensors()[pose]
    sc, g = Scene(rf, a, a), gb300.Guide(be)

    def iterate():
        t.clearFrame()
        t.sampleIndexOffset = 0
        g.run_iteration(t, sc, BUDGET, True)
        return t.frame.data[0, :, 0].copy()

    for _ in range(3):
        iterate()
        g.step()
    start = oracle_lib.GuideState(*g.read())
    assert (start.samp_child >= 0).sum() > 4  # a tree that warps samples
    og = oracle_lib.Guide()
    og.set(start)
    row = iterate()
    want, _ = og.run_pass(ora, rf, t.frame.config(), a, a, t, BUDGET, train=True)
    assert np.linalg.norm(row - want[0, :, 0]) <= 1e-4 * np.linalg.norm(want[0, :, 0])
    got, ref = oracle_lib.GuideState(*g.read()), og.get()
    leaves = [n for n in ref.reachable("train") if ref.train_child[n] < 0]
    x, y = got.acc2[leaves].astype(np.float64), ref.acc2[leaves].astype(np.float64)
    assert np.count_nonzero(y) > 4 and np.abs(x - y).max() <= 1e-4 * np.abs(y).max()


@pytest.mark.parametrize("flags", [dict(), dict(onlyIndirect=False), dict(maxDepth=9), dict(doFiltering=False)],
                         ids=lambda f: "-".join("%s=%d" % i for i in f.items()) or "default")
def test_batches_of_one_iteration(setup, flags):
    """Receivers beside and away from their transmitters, one iteration each."""
    _, be, ora, oracle_lib = setup
    rf, frame = scenes.rf_77ghz(N, 5e6)
    t, tx = tracer(**flags), sensors()
    for gap in (0.01, 0.3, 3.0):
        rx = [NFAntenna(a.position() + np.float32([gap, 0.5 * gap, -gap]), a.rotation()) for a in tx]
        rows = be.simulate_batch(rf, N, t, tx, rx, [BUDGET] * len(tx))
        for k, (row, a, b) in enumerate(zip(rows, tx, rx)):
            fr, tw = oracle_lib.Guide().path_tracer_run(ora, rf, t.frame.config(), a, b, t, BUDGET)
            want = fr[0, :, 0] / tw
            assert np.linalg.norm(row - want) <= 1e-4 * np.linalg.norm(want), (gap, k)
