"""What the kernels' sources have to keep to around their bounded waits and no run can show: where a wait runs out, the threads that
meet in a barrier leave together; what one lane has seen land is ordered before what another lane issues."""
import itertools
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "kinetics_b200" / "csrc"


def _consumers_of_selection():
    text = (CSRC / "ktk_select.cu").read_text()
    return text[text.index("// ---------------- consumer warps ----------------"):text.index("// ---- the k-th largest")]


def _stuck(vote):
    """Two warps at the point of leaving: whether the waits of each came through, and what a look at the flag shows each of them, which may
    be raised in between.  The cases in which one leaves and the other goes on to the next barrier."""
    cases = []
    for came_a, came_b, flag_a, flag_b in itertools.product((True, False), repeat=4):
        alone = [not came or flag for came, flag in ((came_a, flag_a), (came_b, flag_b))]
        left = [not came_a or not came_b] * 2 if vote else alone
        if left[0] != left[1]:
            cases.append((came_a, came_b, flag_a, flag_b))
    return cases


def test_consumers_of_the_selection_leave_together():
    assert _stuck(vote=False) and not _stuck(vote=True)
    body = _consumers_of_selection()
    # the one way out of the item loop: behind a vote of all consumers
    outs = [x.strip() for x in body.splitlines() if re.search(r"\bbreak;", x) and x.strip() != "break;"]
    assert len(outs) == 1 and outs[0].startswith("if (consumer_any(!ok)) break;")
    alone = re.findall(r"\{\s*ok = false;\s*break;\s*\}", body)            # out of the loop over an item's stages, to the vote behind it
    assert len(re.findall(r"^\s*break;", body, re.M)) == len(alone) == 1
    assert "abort_flag)" not in body.replace("&abort_flag)", "")             # no look of a warp's own


def test_a_lane_that_looks_for_another_hands_on_what_it_saw():
    """Two lanes look at a barrier each and any lane may issue the products: a vote orders control flow, __syncwarp memory."""
    text = (CSRC / "layers" / "ktl_moe_umma.cu").read_text()
    look = text[text.index("auto both_landed"):]
    look = look[:look.index("return true;")]
    assert look.index("__ballot_sync(") < look.index("__syncwarp();")


def test_lanes_of_a_warp_give_up_together():
    """Behind these waits stand shuffles and votes over the whole warp: one lane alone may not leave."""
    look = (CSRC / "layers" / "ktl_moe_umma.cu").read_text()
    look = look[look.index("auto both_landed"):look.index("if (PAIR && rank == 1)")]
    assert re.findall(r"if \((.*)\) return false;", look) == ["(i & 63u) == 63u && __any_sync(0xffffffffu, *(volatile int*)&abort_flag)"]
    walk = (CSRC / "layers" / "ktl_norm.cu").read_text()
    walk = walk[walk.index("residual_norm_walk_kernel(const"):]
    assert re.findall(r"if \((.*mbar_wait.*)\) break;", walk) == ["!__all_sync(0xffffffffu, mbar_wait(&full[s], parity, &abort_flag))"]
