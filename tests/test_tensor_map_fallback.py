"""Kernels on tensor copies, read from their sources: where the driver gives no tensor map a projection takes another form, it is not
refused (a driver without the encoder cannot be had for a test on a GPU; the other forms are tested there behind the setting that picks them)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepj_b200", "csrc")


def test_a_refused_tensor_map_is_no_error():
    calls = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name), encoding="utf-8").read())
        for m in re.finditer(r"if \([^;{]*!(?:q8_)?encode_\w+\([^;{]*\)\s*(\w+)", text):
            calls += 1
            assert m.group(1) != "throw", (name, m.group(0))
    assert calls >= 5
