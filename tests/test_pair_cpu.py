"""The prefill kernel on pairs of SMs, as far as the CPU can check it."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "qwen3-27b-thor-runner_b200", "csrc")


def test_issuing_warps_decide_as_a_whole():
    """The issuers elect a lane of the full warp for every MMA and commit, so a lane that leaves the loop alone (its wait ran out,
    another lane's did not) would leave the rest waiting without a limit.  No wait on a GPU can be made to run out in some lanes
    only, hence the source: behind the loop's last wait the warp votes, and nothing but the vote decides whether it goes on."""
    src = open(os.path.join(CSRC, "prefill_pair.cu")).read()
    issuer = src[src.index("MMA issuers (leader only)"):src.index("dequantise into TMEM")]
    loop = issuer[issuer.index("for (int turn = 0;"):]
    assert re.match(r"for \(int turn = 0; turn < turns; \+\+turn\)", loop)            # not on the lane's own `ok`
    vote = loop.index("ok = __all_sync(0xffffffffu, ok);")
    elections = [loop.index(f) for f in ("mma8_ss(", "mma8_ts(", "commit_leader(")]
    assert loop.rindex("ptx::mbar_wait(") < vote < loop.index("break;") < min(elections)
    assert loop.count("break;") == 1 and "return" not in loop and "continue" not in loop
