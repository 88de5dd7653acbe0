"""The neighbourhood lists' queries on the CPU (hussar_gb300/csrc/hsr_local.cuh compiled
with g++): every answer a list gives equals brute force over the whole mesh, and it answers
whenever the hit lies inside the cube."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from hussar_gb300 import TriangleMesh, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")) or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("local") / "local_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "tests", "native"),
                    "-I", os.path.join(ROOT, "hussar_gb300", "csrc"), "-I", CUDA_INC, "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "native", "local_check.cpp"),
                    "-o", exe], check=True)
    return exe


def turned(mesh, angle):
    """The mesh turned about an oblique axis: no plane is parallel to an axis."""
    k = np.array([1.0, 2.0, 3.0]) / np.sqrt(14.0)
    K = np.array([[0, -k[2], k[1]], [k[2], 0, -k[0]], [-k[1], k[0], 0]])
    R = np.eye(3) + np.sin(angle) * K + (1 - np.cos(angle)) * K @ K
    m = TriangleMesh()
    m.append(mesh.vertexBuffer.astype(np.float64) @ R.T, mesh.indexBuffer)
    return m


def slivers(rng, count):
    """Thin and degenerate triangles of every size: some of zero area, some 1e-4 as high as
    wide, some through the origin."""
    a = rng.normal(size=(count, 3))
    e = rng.normal(size=(count, 3)) * 10.0 ** rng.uniform(-2, 1, (count, 1))
    g = rng.normal(size=(count, 3)) * 10.0 ** rng.uniform(-4, 0, (count, 1)) + e * rng.uniform(0, 1, (count, 1))
    g[::17] = e[::17] * 0.5
    a[::5] *= 0.05
    m = TriangleMesh()
    m.append(np.stack([a, a + e, a + g], 1).reshape(-1, 3), np.arange(3 * count).reshape(-1, 3))
    return m


MESHES = {
    "boxes": lambda rng: scenes.boxes_mesh(7, 400, 7.0),
    "turned boxes": lambda rng: turned(scenes.boxes_mesh(8, 400, 40.0), 0.7),
    "slivers": lambda rng: slivers(rng, 600),
    "sphere": lambda rng: scenes.sphere_ground_workload(level=3).mesh,
    "far boxes": lambda rng: TriangleMesh(scenes.boxes_mesh(9, 400, 7.0).vertexBuffer + np.float32(500),
                                          scenes.boxes_mesh(9, 400, 7.0).indexBuffer),
}


@pytest.mark.parametrize("name", MESHES)
def test_answers_equal_brute_force(checker, tmp_path, name):
    rng = np.random.default_rng(len(name))
    mesh = MESHES[name](rng)
    v, f = mesh.vertexBuffer, mesh.indexBuffer
    settled = 0
    for k in range(6):
        c = np.array([0.3, 1.0, -0.2]) + rng.uniform(-1, 1, 3)
        if name == "far boxes":
            c += 500
        n = 1500
        rays = rng.uniform(-1, 1, (n, 7))
        d = rng.normal(size=(n, 3))
        d[: n // 8, 0] = 0.0  # parallel to a plane, and to an axis
        d[n // 8: n // 4] = np.eye(3)[rng.integers(0, 3, n // 4 - n // 8)] * rng.choice([-1, 1], (n // 4 - n // 8, 1))
        rays[: n // 16, :3] = rng.choice([-1.0, 0.0, 1.0], (n // 16, 3))  # the cube's corners, edges, centre
        rays[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
        path = tmp_path / ("in%d.bin" % k)
        with open(path, "wb") as fh:
            fh.write(np.array([len(v), len(f), n], np.int64).tobytes())
            for a, t in ((v, np.float32), (f, np.int32), (c, np.float32), (rays, np.float32)):
                fh.write(np.ascontiguousarray(a, t).tobytes())
        out = subprocess.run([checker, str(path)], check=True, capture_output=True, text=True).stdout.split()
        res = {out[i]: float(out[i + 1]) for i in range(0, len(out), 2)}
        assert res["wrong"] == 0 and res["missed"] == 0 and res["any_wrong"] == 0, res
        settled += res["settled"]
    assert settled > 0 or name == "far boxes"
