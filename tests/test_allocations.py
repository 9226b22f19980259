"""Every device allocation of the library goes through device_malloc, which gives the kept blocks back before it fails; only the
few made at initialisation, before there are any, do not."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepj_b200", "csrc")


def test_allocations_go_through_device_malloc():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh", ".cpp", ".h")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name), encoding="utf-8").read())
        if name == "runtime.cu":
            a, b = text.index("void ensure_init() {"), text.index("void drop_graphs() {")
            text = text[:a] + text[b:]
            a = text.index("cudaError_t device_malloc(")
            text = text[:a] + text[text.index("return e;", a):]
        assert "cudaMalloc(" not in text and "cudaMallocAsync(" not in text, name
