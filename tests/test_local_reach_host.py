"""That the CPU check of the neighbourhood lists' queries has something to compare: on every
kind of mesh there is a cube, queries its list settles and segments that are occluded, also
where coordinates are large beside the boxes."""
import subprocess

import numpy as np
import pytest

import test_local_host as lists
from hussar_gb300 import TriangleMesh, scenes
from test_local_host import checker  # noqa: F401 (the compiled check)


def far_boxes(offset):
    m = scenes.boxes_mesh(9, 400, 7.0)
    return TriangleMesh(m.vertexBuffer + np.float32(offset), m.indexBuffer)


MESHES = {k: (v, 0.0) for k, v in lists.MESHES.items() if k != "far boxes"}
MESHES |= {"boxes %d m away" % d: (lambda rng, d=d: far_boxes(d), float(d)) for d in (20, 100)}


@pytest.mark.parametrize("name", MESHES)
def test_there_is_something_to_settle(checker, tmp_path, name):  # noqa: F811
    make, offset = MESHES[name]
    rng = np.random.default_rng(len(name))
    mesh = make(rng)
    v, f = mesh.vertexBuffer, mesh.indexBuffer
    total = {"half": 0.0, "settled": 0.0, "occluded": 0.0}
    for k in range(6):
        c = np.array([0.3, 1.0, -0.2]) + rng.uniform(-1, 1, 3) + offset
        n = 1500
        rays = rng.uniform(-1, 1, (n, 7))
        d = rng.normal(size=(n, 3))
        rays[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
        path = tmp_path / ("in%d.bin" % k)
        with open(path, "wb") as fh:
            fh.write(np.array([len(v), len(f), n], np.int64).tobytes())
            for a, t in ((v, np.float32), (f, np.int32), (c, np.float32), (rays, np.float32)):
                fh.write(np.ascontiguousarray(a, t).tobytes())
        out = subprocess.run([checker, str(path)], check=True, capture_output=True, text=True).stdout.split()
        res = {out[i]: float(out[i + 1]) for i in range(0, len(out), 2)}
        assert res["wrong"] == 0 and res["missed"] == 0 and res["any_wrong"] == 0, res
        for q in total:
            total[q] += max(0.0, res[q])
    assert total["half"] > 0 and total["settled"] > 100 and total["occluded"] > 0, total
