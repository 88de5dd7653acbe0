"""Neighbourhood lists (dense scenes): rows of the wavefront kernel, whose queries near the
sensor the list answers, against the oracle's tree on the same samples at the parity
tolerance (1e-4 relative L2). Sensors inside the boxes, between them and above them (lists
that settle most queries, some, and none), receivers inside and outside the cube, the
flags that change a query, and a scene moved under its tree."""
import numpy as np
import pytest

from hussar_gb300 import (HSR_PHASE_REFERENCE_FP32, HSR_PHASE_SPLIT_FP64, HSR_SPLAT_DIRICHLET16, HSR_SPLAT_FINE_SYNTH,
                          NFAntenna, PathTracer, TriangleMesh, gb300, scenes)

pytestmark = pytest.mark.gpu

N, BUDGET = 100, 12345


def tracer(**flags):
    t = PathTracer()
    t.doGuiding = False
    t.maxDepth = 4
    for k, v in flags.items():
        setattr(t, k, v)
    return t


def sensors():
    out = [NFAntenna(p, scenes.looking(0.3 * k)) for k, p in enumerate(
        [(0.0, 1.0, 0.0), (3.3, 0.4, -2.1), (-4.0, 1.7, 5.0), (1.0, 4.9, 1.0), (2.0, 7.0, 2.0), (30.0, 2.0, 0.0)])]
    return out + scenes.plane_poses(6, 3, 18.0)


@pytest.fixture(scope="module")
def scene(product_lib, oracle_lib):
    mesh = scenes.boxes_mesh(5, 4000, 20.0)
    return mesh, gb300.Backend(mesh, None), oracle_lib.Scene(mesh)


def check(be, ora, t, tx, rx, tol=1e-4, **modes):
    rf, _ = scenes.rf_77ghz(N, 5e6)
    rows = be.simulate_batch(rf, N, t, tx, rx, [BUDGET] * len(tx), **modes)
    for k, (row, a, b) in enumerate(zip(rows, tx, rx)):
        ref = np.asarray(ora.fetch_row(rf, N, a, b, t, BUDGET), np.complex128)
        # the direct term of a receiver at its transmitter is 0 / 0, on both sides
        fine = np.isfinite(ref)
        assert np.array_equal(fine, np.isfinite(row)), k
        assert np.linalg.norm((row - ref)[fine]) <= tol * np.linalg.norm(ref[fine]), k


@pytest.mark.parametrize("flags", [dict(), dict(onlyIndirect=False), dict(maxDepth=1), dict(maxDepth=9),
                                   dict(doFiltering=False), dict(filteringSphere=False)],
                         ids=lambda f: "-".join("%s=%d" % i for i in f.items()) or "default")
def test_rows_match_the_oracle(scene, product_lib, flags):
    _, be, ora = scene
    before = product_lib.hsr_launch_count()
    check(be, ora, tracer(**flags), sensors(), sensors())
    assert product_lib.hsr_launch_count() - before == 4  # prefix, lists, trace, finalize


@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("gap", [0.01, 0.3, 3.0])
def test_receiver_apart_from_the_transmitter(scene, gap, direct):
    """The cube is the receiver's; the transmitter may lie outside it."""
    _, be, ora = scene
    rx = [NFAntenna(a.position() + np.float32([gap, 0.5 * gap, -gap]), a.rotation()) for a in sensors()]
    check(be, ora, tracer(onlyIndirect=not direct), sensors(), rx)


def test_phase_and_splat_modes_agree_with_the_per_thread_kernel(scene, product_lib):
    """The split phase and the synthesis take the same path: against the one-thread-per-
    sample kernel, which walks the tree for every query (1e-3: the two translation units
    contract multiply-adds differently)."""
    _, be, _ = scene
    rf, _ = scenes.rf_77ghz(N, 5e6)
    for phase, splat in ((HSR_PHASE_SPLIT_FP64, HSR_SPLAT_DIRICHLET16), (HSR_PHASE_SPLIT_FP64, HSR_SPLAT_FINE_SYNTH),
                         (HSR_PHASE_REFERENCE_FP32, HSR_SPLAT_FINE_SYNTH)):
        args = (rf, N, tracer(), sensors(), sensors(), [BUDGET] * len(sensors()), None, phase, splat)
        rows = be.simulate_batch(*args)
        product_lib.hsr_set_path_kernel(1)
        try:
            ref = be.simulate_batch(*args)
        finally:
            product_lib.hsr_set_path_kernel(0)
        err = np.linalg.norm(rows - ref) / np.linalg.norm(ref)
        assert err <= (1e-3 if phase == HSR_PHASE_SPLIT_FP64 else 1e-4), (phase, splat)


def test_moved_scene(scene, oracle_lib):
    """A refit keeps the scene's list radius; the lists are formed from the moved boxes."""
    mesh, _, _ = scene
    be = gb300.Backend(mesh, None)
    v = mesh.vertexBuffer
    moved = TriangleMesh(v + (0.3 * np.sin(3.0 * v[:, [2, 0, 1]])).astype(np.float32), mesh.indexBuffer)
    be.refit(moved)
    check(be, oracle_lib.Scene(moved), tracer(), sensors(), sensors())
