"""What can only be read: the ends of the tcgen05 pipeline's roles after a bounded wait has run out, which no test may bring about
on a GPU.  No GPU."""
import os
import re

from conftest import ROOT


def _kernel(path, name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "rwkv_quant_b200", "csrc", path)).read())
    at = src.index(name + "(")
    return src[at:src.index("\n}\n", at)]


def test_copies_in_flight_are_waited_for_by_the_warps_that_issue_them():
    """Also where a wait ran out, and by the issuer itself: it may reach the end of the kernel before another role has failed."""
    body = _kernel("rwkvq_gemm_sb.cu", "gemm_sb_kernel")
    raw = body[body.index("warp == kSbRawWarp) {"):body.index("warp == kSbTmaWarp) {", body.index("warp == kSbRawWarp) {"))]
    rows = body[body.index("warp == kSbTmaWarp) {", body.index("warp == kSbRawWarp) {")):body.index("const __half* dp")]
    for role, bar, depth in ((raw, "raw_full", "G::AHEAD"), (rows, "bar_empty", "G::U")):
        assert role.count("if (!alive) break;") == 1 and role.count("if (!alive || ti == n_my - 1)") == 1
        drain = role[role.index("if (!alive || ti == n_my - 1)"):]
        assert re.search(r"for \(int (\w) = max\(0, (\w+) - %s\); \1 < \2; \+\+\1\) mbar_poll_bounded\(&%s\[\1 %% %s\], \(\1 / %s\) & 1\)"
                         % (depth, bar, depth, depth), drain), drain


def test_a_weight_warp_whose_wait_ran_out_arrives_no_more():
    """Its arrivals would complete phases of units whose copies are still on their way."""
    body = _kernel("rwkvq_gemm_sb.cu", "gemm_sb_kernel")
    weights = body[body.index("const __half* dp"):body.index("sb_before += n_super")]
    assert re.findall(r"if \(([^)]*)\)\s*mbar_arrive\(&(\w+)", weights) == [("lane == 0 && alive", "raw_empty"), ("lane == 0 && alive", "bar_full")]
    assert weights.count("mbar_arrive") == 2
