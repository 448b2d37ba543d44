"""Every tensor-memory load (csrc/tc_common.cuh) hands its registers through the
wait that completes it: otherwise the compiler may use them before it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libgeodecomp_gb300", "csrc")


def functions_with(text, what):
    for m in re.finditer(r"__device__ __forceinline__ [^;{]*\{", text):
        body = text[m.end():text.index("\n}\n", m.end())]
        if what in body:
            yield body


def test_loaded_registers_pass_through_the_wait():
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        for body in functions_with(text, "tcgen05.ld."):
            loaded = re.findall(r'"=r"\((\w+)', body)
            waits = re.findall(r'"tcgen05\.wait::ld\.sync\.aligned;"(.*?)\);\n', body, re.S)
            assert len(waits) == 1, name
            width = int(re.search(r"uint32_t r\[(\d+)\]", body).group(1)) if "uint32_t r[" in body else 1
            assert loaded and len(re.findall(r'"\+r"\(', waits[0])) == width, (name, body)
            seen += 1
    assert seen >= 3
