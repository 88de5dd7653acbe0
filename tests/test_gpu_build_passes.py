"""The build at its edges: clusters around a warp's and a block's share of the nearest-neighbour
search (four and 32), around its window (256 either side) and, for the insertion passes, a
small and a large tree. Each tree is complete and conservative, and the passes leave the
surface-area cost lower than they found it."""
import numpy as np
import pytest

from hussar_gb300 import TriangleMesh, gb300, scenes
from hussar_gb300.core import child_boxes
from test_gpu_bvh import check_tree

pytestmark = pytest.mark.gpu


def cost(be):
    """Sum of the child boxes' areas: what the passes lower."""
    lo, hi = child_boxes(be.device_bvh()[0])
    d = (hi - lo).astype(np.float64)
    return (d[..., 0] * d[..., 1] + d[..., 1] * d[..., 2] + d[..., 2] * d[..., 0]).sum()


@pytest.mark.parametrize("nt", [31, 32, 33, 255, 257, 511, 514, 20001])
def test_tree(product_lib, nt):
    mesh = scenes.boxes_mesh(7, (nt + 11) // 12, 30.0 if nt < 1000 else 100.0)
    assert mesh.triangleCount() >= nt
    mesh = TriangleMesh(mesh.vertexBuffer, np.asarray(mesh.indexBuffer)[:nt])
    product_lib.hsr_set_bvh_leaf_size(1)
    try:
        be = gb300.Backend(mesh, None)
        assert check_tree(be, mesh)[2] == nt
        product_lib.hsr_set_bvh_optimize(0)
        assert cost(be) <= cost(gb300.Backend(mesh, None))
    finally:
        product_lib.hsr_set_bvh_leaf_size(4)
        product_lib.hsr_set_bvh_optimize(32)
