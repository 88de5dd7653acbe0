"""Served requests on dense scenes, whose poses get neighbourhood lists in the tick: rows against
the oracle at the parity tolerance (1e-4 relative L2) and against the same request alone
(1e-5), in ticks of one scene and chirp and of several, dense and open together, plain
and guided."""
import numpy as np
import pytest

from hussar_gb300 import PathTracer, Server, gb300, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def resident(product_lib, oracle_lib):
    """(poses, backend, oracle scene): two dense scenes and two open ones."""
    meshes = [scenes.boxes_mesh(5, 4000, 20.0), scenes.boxes_mesh(6, 1500, 13.0),
              scenes.sphere_ground_workload(level=4).mesh, scenes.boxes_mesh(7, 500, 60.0)]
    poses = [scenes.plane_poses(8, 3, 18.0), scenes.plane_poses(8, 4, 12.0), scenes.sphere_ground_workload().tx * 8,
             scenes.plane_poses(8, 5, 50.0)]
    return [(p, gb300.Backend(m, None), oracle_lib.Scene(m)) for p, m in zip(poses, meshes)]


@pytest.mark.parametrize("guided", [False, True], ids=["plain", "guided"])
@pytest.mark.parametrize("kinds", [(0,), (0, 1), (0, 2), (2, 3, 1), (0, 1, 2, 3)],
                         ids=lambda k: "".join("DdOo"[i] for i in k))
def test_rows(resident, kinds, guided):
    t = PathTracer()
    t.doGuiding, t.maxDepth = guided, 3
    rng = np.random.default_rng(len(kinds))
    reqs = []
    for k in range(12):
        si = kinds[k % len(kinds)]
        bins = 128 if len(kinds) == 1 else int(rng.choice([100, 128, 333]))
        budget = int(rng.integers(3000, 16000))  # guided: one iteration
        reqs.append((si, scenes.rf_chirp(2e9, bins), bins, resident[si][0][k % 8], budget, 0 if guided else 77 * k))
    with Server(flags=t, max_slots=16, max_samples_per_chirp=512) as srv:
        ids = [srv.add_scene(be) for _, be, _ in resident]
        handles = [srv.submit(ids[si], rf, n, a, a, b, off) for si, rf, n, a, b, off in reqs]
        rows = [h.result(timeout=60)[0] for h in handles]
    for (si, rf, n, a, b, off), row in zip(reqs, rows):
        _, be, ora = resident[si]
        alone = be.simulate_batch(rf, n, t, [a], [a], [b], index_offset=[off])[0]
        assert np.linalg.norm(row - alone) <= 1e-5 * np.linalg.norm(alone)
        if not guided:
            want = ora.fetch_row(rf, n, a, a, t, b, offset=off)
            assert np.linalg.norm(row - want) <= 1e-4 * np.linalg.norm(want)
