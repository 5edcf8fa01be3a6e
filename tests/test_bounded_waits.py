"""Bounded waits whose outcome decides what a warp does next: the whole warp has to agree on it.

The kernels' softmax, epilogue and issuing warps go on with votes, shuffles and tcgen05 loads of all lanes.  A wait that runs out
for some lanes only must not let them go alone, so those warps use the form that votes; a lane's own form is left to waits that a
block-wide vote or one thread's loop follows, and to the drains, whose outcome nobody looks at.  Read from the sources: no wait is
made to run out here."""
import os
import re

import pytest

from transformer_b200.csrc import build


def _text(name):
    with open(os.path.join(build.HERE, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_the_warps_form_votes():
    body = _text("tc_common.cuh").split("bool mbar_wait_warp(", 1)[1].split("}", 1)[0]
    assert "return __all_sync(0xffffffffu, mbar_wait(bar, parity, error, code));" in body


@pytest.mark.parametrize("name", [f for f in build.sources() if "mbar_wait" in _text(f)])
def test_no_lane_decides_alone(name):
    """Every ``mbar_wait`` of a lane is a statement by itself (a drain), voted on in the same expression, of a product kernel's
    one issuing thread (``agreed``), behind ``if (lane == 0)`` with the answer passed on, or followed by a vote of the block."""
    text = _text(name)
    for m in re.finditer(r"\bmbar_wait\(", text):
        line = text[text.rfind("\n", 0, m.start()) + 1:text.find("\n", m.start())].strip()
        before = text[:m.start()].rstrip()
        drain = before[-1] in ";{})"
        voted = before.endswith(("__all_sync(0xffffffffu,", "agreed("))
        block = "const bool ok = mbar_wait(" in line and "__syncthreads_and(ok)" in text[m.start():m.start() + 400]
        passed_on = line.startswith("if (i >= S) ok = mbar_wait(") and "ok = __shfl_sync(0xffffffffu, ok, 0);" in text[m.start():]
        assert drain or voted or block or passed_on, line
