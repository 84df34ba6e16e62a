"""The choice between the chained forward and the two kernels in front of the intra stage depends on process-wide
testing switches that another thread may move: one call asks once, and every stage follows that answer."""

import os
import re

from conftest import ROOT


def test_one_call_asks_once():
    csrc = os.path.join(ROOT, "delta_feedback_experiment_b200", "csrc")
    uses = []
    for name in sorted(os.listdir(csrc)):
        code = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, name)).read())
        uses += [(name, line.strip()) for line in code.splitlines() if "forward_chain_possible(" in line]
    assert len(uses) == 2, uses  # its definition and the one question
    assert uses[0][1].startswith("static bool") and uses[1][1].startswith("const bool chained =")
