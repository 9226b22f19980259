"""Order of waits in the many-row Q8 kernel, read from its source (a kernel whose bound runs out under an earlier kernel's time
is not something to provoke on a GPU): every role waits for the earlier kernels before its first bounded wait that ends only
with their data.  The activation images are such data; the raw codes are not."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepj_b200", "csrc", "q8_tc.cu")


def roles():
    text = open(SRC, encoding="utf-8").read()
    text = text[text.index("k_q8_gemm_tc(const __grid_constant__"):text.index("struct TcPlan")]
    text = re.sub(r"//[^\n]*", "", text)
    heads = ["if (warp < kPromoteWarps) {", "if (warp < kPromoteWarps + kConvertWarps) {", "} else if (warp == kCopyWarp) {", "} else if (warp >= kMmaWarp) {",
             "} else if (warp == kRawWarp) {"]
    at = [text.index(h) for h in heads] + [len(text)]
    assert at == sorted(at)
    return dict(zip(("promote", "convert", "copy", "mma", "raw"), (text[a:b] for a, b in zip(at, at[1:]))))


def test_dependency_wait_precedes_the_waits_that_need_the_images():
    for name, body in roles().items():
        waits = [m.start() for m in re.finditer(r"warp_wait\((accFull|accEmpty|full|empty|rawEmpty)\(", body)]
        assert waits and "pdl_wait();" in body, name
        assert body.index("pdl_wait();") < waits[0], name
    # a converter's wait for raw codes may come first: they are copied without any earlier kernel's data
    conv = roles()["convert"]
    assert "i >= S::kStages" in conv[:conv.index("pdl_wait();")]


def test_no_results_are_stored_after_an_expired_wait():
    body = roles()["promote"]
    assert re.search(r"mEnd = s_abort \? 0 :", body) and body.index("s_abort ? 0") > body.index("cluster_sync_all()")
