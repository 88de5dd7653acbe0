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
