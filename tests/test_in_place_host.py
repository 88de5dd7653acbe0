"""Caller arrays that kernels may use where they are: aligned for their elements and apart from
every result (usable_in_place compiled with g++, on made-up addresses)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def usable(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")) or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("in_place") / "in_place_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "hussar_gb300", "csrc"), "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "native", "in_place_check.cpp"), "-o", exe], check=True)
    return lambda *arrays: subprocess.run([exe, *arrays], check=True, capture_output=True, text=True).stdout == "1\n"


@pytest.mark.parametrize("off", [0, 1, 2, 3, 4, 6])
def test_alignment(usable, off):
    """Words from any byte: in place at whole words only, whichever array is off."""
    assert usable("i:%d:400:4" % (4096 + off), "o:8192:400:4") == (off % 4 == 0)
    assert usable("i:4096:400:4", "o:%d:400:4" % (8192 + off)) == (off % 4 == 0)
    assert usable("i:4096:400:4", "i:%d:80:8" % (4800 + off), "o:8192:400:4") == (off % 8 == 0)


@pytest.mark.parametrize("at, apart", [(4096, False), (4092, False), (4496, True), (4492, False), (3696, True),
                                       (3700, False), (4200, False), (0, True)])
def test_overlap(usable, at, apart):
    """A result of 400 bytes against an input and another result at 4096 .. 4495; 0: not wanted."""
    assert usable("i:4096:400:4", "o:%d:400:4" % at) == apart
    assert usable("i:20000:400:4", "o:4096:400:4", "o:%d:400:4" % at) == apart
    # inputs may share memory
    assert usable("i:4096:400:4", "i:4100:400:4", "o:20000:400:4")
