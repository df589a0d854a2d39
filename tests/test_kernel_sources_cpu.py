"""Rules of the kernel sources that show in their text: what a run on a GPU could only show by hanging it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "mindspeed_rl_b200" / "csrc"
SOURCES = sorted(p for p in (*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")) if "mbar_wait(" in p.read_text())


def lone_waits(text: str):
    """Lines of bounded waits that the lanes of a warp take one by one: outside code of one lane, and with no vote on the outcome."""
    text = re.sub(r"//[^\n]*", "", text)
    enclosing, start, found = [], 0, []
    for m in re.finditer(r"[{};]|\bmbar_wait\(", text):
        if m.group() == "{":
            enclosing.append(text[start:m.start()])
        elif m.group() == "}":
            enclosing.pop()
        elif m.group() != ";":
            around = enclosing + [text[start:m.start()]]
            own = re.search(r"\bbool\s+$", around[-1])                       # the definition
            if not own and not any(re.search(r"elect_one\(\)|lane == 0|__all_sync\(", s) for s in around):
                found.append(text.count("\n", 0, m.start()) + 1)
            continue
        start = m.end()
    return found


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_lanes_of_a_warp_leave_a_bounded_wait_together(path):
    """A wait that ran out in some lanes only leaves the others in front of a warp-wide barrier that these never reach: a hang in
    place of an error code.  One lane waits, or all agree (``mbar_wait_warp``)."""
    assert lone_waits(path.read_text()) == []
