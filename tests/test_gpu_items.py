"""Work items of the wavefront launch: 256-sample items pulled in shrinking runs. Budgets at
the edges of an item and of a run, poses without samples between them, and tiles that are
and are not whole numbers of items, against the oracle at the parity tolerance (1e-4
relative L2 of the IF signal) on the same Halton samples."""
import numpy as np
import pytest

from hussar_gb300 import PathTracer, gb300, scenes

pytestmark = pytest.mark.gpu

N = 128
BUDGETS = [1, 255, 256, 257, 0, 511, 4095, 4096, 4097, 0, 0, 16385, 70001]


@pytest.fixture(scope="module")
def setup(product_lib, oracle_lib):
    mesh = scenes.boxes_mesh(5, 40, 10.0)
    t = PathTracer()
    t.doGuiding = False
    t.maxDepth = 3
    rf, _ = scenes.rf_77ghz(N, 5e6)
    ants = scenes.plane_poses(len(BUDGETS), 6, 10.0)
    offset = np.arange(len(BUDGETS), dtype=np.int64) * 1000003
    ora = oracle_lib.Scene(mesh)
    refs = [ora.fetch_row(rf, N, a, a, t, b, offset=int(o)) if b else None
            for a, b, o in zip(ants, BUDGETS, offset)]
    return gb300.Backend(mesh, None), rf, t, ants, offset, refs


@pytest.mark.parametrize("tile", [0, 256, 1000, 16384])
@pytest.mark.parametrize("poses", [1, len(BUDGETS)])
def test_every_sample_is_traced_once(setup, tile, poses):
    be, rf, t, ants, offset, refs = setup
    be.set_launch_config(tile=tile, default=tile == 0)
    first = len(BUDGETS) - poses  # one pose: the largest budget, spread over the grid
    rows = be.simulate_batch(rf, N, t, ants[first:], ants[first:], BUDGETS[first:], offset[first:])
    for row, ref, b in zip(rows, refs[first:], BUDGETS[first:]):
        if b:
            ref = np.asarray(ref, np.complex128)
            assert np.linalg.norm(row - ref) <= 1e-4 * np.linalg.norm(ref), (tile, b)


@pytest.mark.parametrize("poses", [1023, 1024, 1025, 2049])
def test_prefix_over_many_poses(setup, oracle_lib, poses):
    """The items' prefix is formed 1024 poses at a time; poses without samples lie between.
    Every 97th pose and the ones around a chunk's end against the oracle."""
    be, rf, t, _, _, _ = setup
    be.set_launch_config(default=True)
    rng = np.random.default_rng(poses)
    budget = rng.integers(0, 700, poses) * (rng.random(poses) < 0.8)
    budget[-1] = 300
    offset = rng.integers(0, 1 << 20, poses)
    ants = scenes.plane_poses(poses, 9, 10.0)
    rows = be.simulate_batch(rf, N, t, ants, ants, budget, offset)
    ora = oracle_lib.Scene(scenes.boxes_mesh(5, 40, 10.0))
    for k in sorted({*range(0, poses, 97), 1022, min(1023, poses - 1), min(1024, poses - 1), poses - 1}):
        if budget[k]:
            ref = np.asarray(ora.fetch_row(rf, N, ants[k], ants[k], t, int(budget[k]), offset=int(offset[k])),
                             np.complex128)
            assert np.linalg.norm(rows[k] - ref) <= 1e-4 * np.linalg.norm(ref), k


@pytest.mark.parametrize("weight", [1.0, 0.1, 3.0, 1e-3, 0.0, 1e30])
def test_total_weight_is_the_sum_of_additions(product_lib, weight):
    """hsr_backend_run's total weight against adding the float weight sample by sample."""
    mesh = scenes.dihedral_mesh()
    from hussar_gb300 import FrameConfig, Scene
    t = PathTracer()
    t.doGuiding = False
    t.configureFrame(FrameConfig(1, 8, 1))
    rf, _ = scenes.rf_77ghz(8, 5e6)
    a = scenes.dihedral_workload(poses=2).tx[0]
    budget = 70001
    t.currentSampleWeight = weight
    gb300.Backend(mesh, t).run(Scene(rf, a, a), budget)
    assert t.totalWeight == np.cumsum(np.full(budget, np.float64(np.float32(weight))))[-1]
