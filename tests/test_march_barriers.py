"""The uniform marches' rings of primitives, on the CPU: no slot is written in a turn of the march while
a slower warp may still read it from the turn before.

A turn j reads planes (rows) j - ZH .. j + ZH and writes plane j + ZH at its top, in a ring of 2 ZH + 1
slots: the slot it writes is the one that plane j - 1 - ZH had, which the turn before reads. So a barrier
stands between a turn's reads and its end in every turn but the last. The turn of a lower ghost leaves the
loop's body early, ahead of the barriers at the faces, and needs one of its own."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "shaderous_b200" / "csrc"


@pytest.mark.parametrize("zh", [1, 2])
def test_a_turn_writes_the_slot_the_turn_before_reads(zh):
    ring = 2 * zh + 1
    for j in range(-1, 9):
        reads_before = {p % ring: p for p in range(j - 1 - zh, j + zh)}
        assert reads_before[(j + zh) % ring] == j - 1 - zh


def _block(text, start):
    """The braces that open at or after start, and what they hold."""
    a = text.index("{", start)
    depth, i = 0, a
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[a:i]


@pytest.mark.parametrize("name,ghost", [("sweep.cu", "zg"), ("sweep_rows.cu", "yg")])
def test_every_turn_but_the_last_ends_behind_a_barrier(name, ghost):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    body = _block(text, text.index("for (int j = jb; j <= je; j++"))
    # the lower ghost's turn, the one early end that another turn follows (the upper ghost's is the last)
    early = _block(body, body.index(f"if ({ghost}_lo || {ghost}_hi)"))
    lower = _block(early, early.index(f"if ({ghost}_lo)"))
    assert re.search(r"__syncthreads\(\);\s*}$", lower), lower
    assert early.rstrip("} \n").endswith("continue;") and body.count("continue;") == 1
    # any other turn: a barrier after the last read of the ring
    last_read = max(m.start() for m in re.finditer(r"ringk\(|sWj\b", body))
    assert "__syncthreads" in body[last_read:]
