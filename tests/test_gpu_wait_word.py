"""Error words of the FP64 contraction's device-side waits (tests/cpp/test_wait_word.cpp): each
context and each block product reports its own."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "tamm_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_words_are_apart(tmp_path):
    exe = os.path.join(str(tmp_path), "test_wait_word")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", os.path.join(ROOT, "tests", "cpp", "test_wait_word.cpp"),
                        f"-I{ROOT}/include", f"-I{LIBDIR}/csrc", f"-I{CUDA}/include", f"-L{LIBDIR}", "-ltamm_b200",
                        f"-Wl,-rpath,{LIBDIR}", f"-L{CUDA}/lib64", "-lcudart", f"-Wl,-rpath,{CUDA}/lib64", "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ALL PASSED" in r.stdout, r.stdout + r.stderr
