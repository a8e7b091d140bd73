"""Bounded waits give every lane a verdict of its own, so a warp votes before a branch on one that guards instructions of the whole warp.
Read from the source: to reach such a branch on a GPU a wait has to run out for some lanes of a warp alone."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "sapient_b200" / "csrc"
WAIT, VOTE, BRANCH = re.compile(r"\.(full|empty)\(bars\."), "__all_sync(", re.compile(r"\bif \((?:.*&& )?ok\) \{")


def _blocks(text):
    """(line number of the branch, its body) of every branch on `ok`."""
    for m in BRANCH.finditer(text):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.start(), text[m.end():end]


@pytest.mark.parametrize("name", ["gemm_dq.cu"])
def test_branches_around_warp_instructions_are_voted_on(name):
    text = (CSRC / name).read_text()
    guarded = [at for at, body in _blocks(text) if "sync.aligned" in body]
    assert guarded
    for at in guarded:
        before = text[:at]
        wait = max(m.start() for m in WAIT.finditer(before))
        line = before[before.rfind("\n", 0, wait) + 1: before.find("\n", wait)]
        assert VOTE in line or before.rfind(VOTE) > wait, f"line {before.count(chr(10)) + 1}: no vote after `{line.strip()}`"
