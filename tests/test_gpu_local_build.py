"""The neighbourhood lists the device builds (hussar_gb300/csrc/hsr_local.cu) are those brute
force forms, and a pose has one wherever it would settle a good part of its queries."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from hussar_gb300 import scenes

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda"


@pytest.fixture(scope="module")
def checker(product_lib, tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")) or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("local") / "local_build_check")
    libs = [os.path.join(ROOT, "hussar_gb300"), os.path.join(CUDA, "lib64")]
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "tests", "native"),
                    "-I", os.path.join(ROOT, "hussar_gb300", "csrc"), "-I", os.path.join(CUDA, "include"), "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "native", "local_build_check.cpp"),
                    *[x for d in libs for x in ("-L", d, "-Wl,-rpath," + d)], "-lhsr_gb300", "-lcudart", "-o", exe],
                   check=True)
    return exe


def build(checker, tmp_path, mesh, tx, rx):
    v, f = mesh.vertexBuffer, mesh.indexBuffer
    path = tmp_path / "in.bin"
    with open(path, "wb") as fh:
        fh.write(np.array([len(v), len(f), len(tx)], np.int64).tobytes())
        for a, t in ((v, np.float32), (f, np.int32), (np.concatenate([tx, rx], 1), np.float32)):
            fh.write(np.ascontiguousarray(a, t).tobytes())
    lines = subprocess.run([checker, str(path)], check=True, capture_output=True, text=True).stdout.splitlines()
    return float(lines[0].split()[1]), [dict(zip(w[::2], map(int, w[1::2]))) for w in (x.split() for x in lines[1:])]


def judge(poses):
    """Differences, and lists that are there though they settle next to nothing or missing though
    they settle half of the rays (8 of 32 is the line; directions round differently here)."""
    assert all(p["wrong"] == 0 for p in poses), poses
    assert all(p["planes"] > 0 for p in poses if p["near"] >= 12), poses
    assert all(p["planes"] == 0 for p in poses if p["near"] <= 4), poses


@pytest.mark.parametrize("boxes, extent", [(4000, 20.0), (400, 7.0), (20000, 49.0)])
def test_lists_equal_brute_force(checker, tmp_path, boxes, extent):
    rng = np.random.default_rng(boxes)
    c = rng.uniform([-extent / 3, 0.2, -extent / 3], [extent / 3, 1.8, extent / 3], (40, 3))
    radius, poses = build(checker, tmp_path, scenes.boxes_mesh(5, boxes, extent), c, c)
    assert radius > 0  # a dense scene
    judge(poses)
    # between the boxes most poses have a list
    assert sum(p["planes"] > 0 for p in poses) >= 30, poses


def test_transmitter_apart_and_sensors_outside(checker, tmp_path):
    """A transmitter outside the receiver's cube, and receivers far above the boxes, have none."""
    rng = np.random.default_rng(2)
    c = rng.uniform([-6, 0.2, -6], [6, 1.8, 6], (16, 3))
    mesh = scenes.boxes_mesh(5, 4000, 20.0)
    for gap in (0.02, 0.3, 4.0):
        _, poses = build(checker, tmp_path, mesh, c + [gap, gap, 0], c)
        judge(poses)
        assert gap < 4 or all(p["planes"] == 0 for p in poses), poses
    _, poses = build(checker, tmp_path, mesh, c + [0, 200, 0], c + [0, 200, 0])
    assert all(p["planes"] == 0 for p in poses), poses
