"""Scenes whose tree is a chain: thousands of triangles on one place, which the clustering merges
one by one (ties go to the lower index) and no insertion pass untangles. They build, with
every triangle reachable, and rays that keep away from the place are answered as without it."""
import numpy as np
import pytest

from hussar_gb300 import TriangleMesh, gb300

pytestmark = pytest.mark.gpu


def cloud(rng, count):
    c = rng.uniform(-5, 5, (count, 1, 3))
    return c + rng.uniform(-0.5, 0.5, (count, 3, 3))


def mesh(triangles):
    return TriangleMesh(np.asarray(triangles, np.float32).reshape(-1, 3), np.arange(3 * len(triangles)).reshape(-1, 3))


@pytest.mark.parametrize("copies", [100, 1000, 1023, 1024, 1025, 1026, 3000, 9001])
@pytest.mark.parametrize("builder", [0, 1], ids=["ploc", "lbvh"])
def test_coincident_triangles(product_lib, copies, builder):
    rng = np.random.default_rng(copies)
    around = cloud(rng, 300)
    place = np.tile([[[20, 0, 0], [21, 0, 0], [20, 1, 0]]], (copies, 1, 1))
    product_lib.hsr_set_bvh_builder(builder)
    try:
        be, ref = gb300.Backend(mesh(np.concatenate([around, place])), None), gb300.Backend(mesh(around), None)
    finally:
        product_lib.hsr_set_bvh_builder(0)
    # every triangle is in one leaf, and the nodes are stored depth first
    nodes, tris = be.device_bvh()
    slots, stack, met = np.zeros(len(tris), int), [0], 0
    while stack:
        at = stack.pop()
        assert at == met
        met += 1
        for c in reversed(nodes["child"][at].tolist()):
            if c >= 0:
                stack.append(c)
            else:
                slots[(~c >> 3): (~c >> 3) + (~c & 7) + 1] += 1
    assert met == len(nodes) and (slots == 1).all()
    ids = tris[:, 3].view(np.int32)
    assert np.array_equal(np.sort(ids), np.arange(300 + copies))
    # rays that leave the cloud on its other sides
    o = rng.uniform(-6, 6, (2000, 3)).astype(np.float32)
    d = rng.normal(size=(2000, 3))
    d[:, 0] = -np.abs(d[:, 0])
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    for got, want in zip(be.intersect(o, d), ref.intersect(o, d)):
        assert got.tobytes() == want.tobytes()
    far = np.full(2000, 4, np.float32)
    assert be.visible(o, d, far).tobytes() == ref.visible(o, d, far).tobytes()
