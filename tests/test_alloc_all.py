"""Buffers made together on first use (csrc/alloc_all.h): an allocation that
fails leaves none of them, so that a second call fails the same way instead of
running with the rest missing.  Host code, with a failing allocator."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "libgeodecomp_gb300", "csrc")


def test_all_or_none(tmp_path):
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, os.path.join(ROOT, "tests", "cpp", "alloc_all_test.cpp"), "-o", exe],
                   check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "ok\n"


def test_the_networks_mma_buffers_are_made_together():
    """ensure_dense takes one of its buffers as the sign that all exist."""
    src = open(os.path.join(CSRC, "surrogate.cu")).read()
    body = re.search(r"static void ensure_dense\(Net& n\)\n\{(.*?)\n\}", src, re.S).group(1)
    assert "allocate_all(" in body and "LGD_CHECK_CUDA(cudaMalloc" not in body


def test_gradients_share_no_line_with_the_loss():
    """They are one allocation; the gradients' atomics add whole 128-byte lines."""
    src = open(os.path.join(CSRC, "surrogate.cu")).read()
    at = re.search(r"constexpr size_t GRADS_AT = (\d+);", src)
    assert at and int(at.group(1)) % 128 == 0 and int(at.group(1)) >= 128
    assert re.search(r"n->grads = .*n->d_loss\) \+ GRADS_AT\)", src)


def test_error_words(tmp_path):
    """The pool of the handles' error words (csrc/error_words.h), and that handles use it."""
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "error_words_test.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "ok\n", res.returncode
    for name in ("api.cu", "surrogate.cu"):
        src = open(os.path.join(CSRC, name)).read()
        assert "= take_error_word()" in src and not re.search(r"cudaHostAlloc\(&(g\.|n->)", src)
