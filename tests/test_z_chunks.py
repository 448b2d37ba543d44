"""The split of a z-marching launch (csrc/z_chunks.h): within 2% of the best of
all splits, planned in microseconds whatever the number of planes, and used by
every kernel that plans one at each launch."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "libgeodecomp_gb300", "csrc")


def test_near_the_best_split(tmp_path):
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, "-include", "cmath",
                    os.path.join(ROOT, "tests", "cpp", "z_chunks_test.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "ok\n", res.returncode


def test_default_kernels_plan_with_it():
    for name in ("k_tb.cu", "k_vctb.cu", "conv_tc.cu", "wgrad_tc.cu"):
        src = open(os.path.join(CSRC, name)).read()
        assert "least_planes(" in src, name
        assert not re.search(r"for \(int split = 1;", src), name
