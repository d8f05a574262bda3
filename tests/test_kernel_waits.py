"""CPU, by reading the source: where a warp whose wait ran out may leave, and where the others meet."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ubridge_b200", "csrc")


def test_summing_warps_of_the_integer_kernel_agree_before_their_exchange():
    """qgemm_unit.cu: a summing warp leaves its super-block loop on its own verdict.  With a K split the four meet at a named
    barrier behind it, which has no limit: the verdict has to be a common one before any of them leaves the tile."""
    src = open(os.path.join(CSRC, "qgemm_unit.cu")).read()
    role = src[src.index("group sums -> y"):src.index("MMA issuers")]
    after = role[role.index("acc[t] += part[t]"):]  # the last thing a super-block does
    tail = after[after.index("\n      }\n"):]  # behind the loop over super-blocks
    agreed = re.search(r"if \(KS > 1\) ok = agree\(ok\);", tail)
    assert agreed
    for way_out in (r"\bbreak;", r"\bcontinue;", r"\breturn;", "barrier.cluster.wait", "tc_wait"):
        m = re.search(way_out, tail)
        assert m is None or m.start() > agreed.start(), way_out
    # every barrier of the four is such an agreement
    assert len(re.findall(r"bar\.(?:sync|red)", role)) == 1 and "auto agree" in role
