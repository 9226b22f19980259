"""Cluster barriers in their .aligned forms, read from the kernels' sources: every thread of a warp has to execute them together, so a
warp-wide or block-wide barrier stands before each, with nothing between that threads of one warp could do differently."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepj_b200", "csrc")
HELPERS = ("cluster_barrier", "cluster_sync_all")


def barriers():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name), encoding="utf-8").read())
        for m in re.finditer(r'asm volatile\("barrier\.cluster\.[^"]*\.aligned|\b(?:%s)\(\);' % "|".join(HELPERS), text):
            head = text[:m.start()]
            if not re.search(r"void (?:%s)\(\) \{\s*$" % "|".join(HELPERS), head):      # inside a helper: its calls are looked at
                yield name, m.group(0), head


def test_warps_are_whole_at_every_aligned_cluster_barrier():
    seen = 0
    for name, what, head in barriers():
        seen += 1
        if "arrive.relaxed" in what:                 # at a kernel's start: no thread has branched yet
            start = head[head.rindex("__global__"):]
            assert not re.search(r"\b(if \((?!constexpr)|for \(|while \()", start), (name, what)
            continue
        at = max(head.rfind("__syncwarp();"), head.rfind("__syncthreads();"), head.rfind("barrier.cluster."), *(head.rfind(h + "();") for h in HELPERS))
        between = head[at:]
        assert not re.search(r"\b(tid|lane|threadIdx|gl|group|t4)\b", between), (name, what, between)
    assert seen >= 8
