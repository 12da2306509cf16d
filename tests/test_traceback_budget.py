"""A traceback slot counts its age in 16 bits (TbSlot::it0): a hand-on budget that
no such count reaches would never hand a tree on.  Read from csrc/bulge.cu: every
budget, the largest that COF_TB_BUDGET may set among them, is within that count."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "cas-offinder-rust-old_b200", "csrc", "bulge.cu")


def test_budgets_are_within_a_slots_count():
    text = open(SRC).read()
    bits = int(re.search(r"uint(\d+)_t it0;", text).group(1))
    budgets = {m[0]: int(m[1]) for m in re.findall(r"constexpr uint32_t (kTb\w*Budget\w*) = (\d+);", text)}
    assert len(budgets) >= 5
    assert all(0 < b <= 2**bits - 1 for b in budgets.values()), budgets
    # the environment's value is cut to the largest
    env = text[text.index('std::getenv("COF_TB_BUDGET")'):]
    assert "std::min<long>(kTbBudgetMax," in env[:env.index(";")]
