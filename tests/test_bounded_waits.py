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
    """Two warps and what each sees at its two points of leaving (its wait for the item, then the flag behind the item's barrier, raised
    in between): the cases in which one has left and the other stands in a barrier."""
    cases = []
    for item_a, item_b, flag_a, flag_b in itertools.product((True, False), repeat=4):
        left = []
        for mine, flag in ((item_a, flag_a), (item_b, flag_b)):
            if vote:
                left.append(not (item_a and item_b) or flag_a or flag_b)
            else:
                left.append(not mine or flag)
        if left[0] != left[1]:
            cases.append((item_a, item_b, flag_a, flag_b))
    return cases


def test_consumers_of_the_selection_leave_together():
    assert _stuck(vote=False) and not _stuck(vote=True)
    body = _consumers_of_selection()
    # every way out of the item loop: behind a vote of all consumers, or behind a rank that is the same for all of them
    for line in (x.strip() for x in body.splitlines()):
        if re.search(r"\bbreak;", line) and line != "break;":
            assert "consumer_any(" in line or line == "if (rank < 0) break;", line
    alone = re.findall(r"\{\s*ok = false;\s*break;\s*\}", body)            # out of the loop over an item's stages, to the vote behind it
    assert len(re.findall(r"^\s*break;", body, re.M)) == len(alone) == 1
    assert "abort_flag)" not in body.replace("&abort_flag)", "")             # no look of a warp's own


def test_the_producer_of_the_selection_hands_out_nothing_after_giving_up():
    text = (CSRC / "ktk_select.cu").read_text()
    wait, hand_out = text.index("mbar_wait(&item_free[slot]"), text.index("mbar_arrive(&item_full[slot])")
    assert "*(volatile int*)&abort_flag) break;" in text[wait:hand_out]


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
