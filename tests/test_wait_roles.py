"""Bounded waits of whole-warp roles give every lane of the warp the same answer.

A lane that gives up while another saw the phase would leave its warp split in front of ``elect.sync``, ``tcgen05.ld`` or
``__syncwarp``, which wait for all 32 lanes.  That cannot be provoked on a GPU without hanging it, so the sources are read: the
per-lane waits may stand only where one thread runs, the warp waits only where whole warps do."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mlperf_training_b200" / "csrc"
FILES = sorted(p for p in (*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")) if p.name != "common.cuh" and "_wait" in p.read_text())
ONE_THREAD = re.compile(r"lane == 0|threadIdx\.x == 0|elect_one\(\)")
# one thread calls the function, or all but one have returned
ONE_THREAD_BODY = re.compile(r"if \((?:lane|threadIdx\.x) != 0\) return;")


def _code(path):
    text = re.sub(r"/\*.*?\*/", lambda m: " " * len(m.group()), path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), text)


def _single(text, at):
    """Whether position ``at`` lies in a block that one thread of the warp runs."""
    depth, before = 0, ""                   # ``before``: what stands ahead of ``at`` in the block itself, without nested blocks
    for i in range(at - 1, -1, -1):
        if text[i] == "}":
            depth += 1
        elif text[i] == "{" and depth:
            depth -= 1
        elif text[i] == "{":
            head = text[max(text.rfind(c, 0, i) for c in ";{}") + 1:i]
            if ONE_THREAD.search(head) or ONE_THREAD_BODY.search(before[::-1]):
                return True
            before = ""
        elif not depth:
            before += text[i]
    return False


@pytest.mark.parametrize("path", FILES, ids=lambda p: p.name)
def test_waits_match_their_roles(path):
    text = _code(path)
    for m in re.finditer(r"\b(mbar_wait|mbar_wait_spin|warp_wait|warp_wait_spin)\(", text):
        where = f"{path.name}:{text.count(chr(10), 0, m.start()) + 1}"
        assert _single(text, m.start()) == m.group(1).startswith("mbar"), where


def test_warp_waits_leave_as_one():
    text = _code(CSRC / "common.cuh")
    body = re.search(r"bool warp_wait_impl\([^)]*\) \{(.*?)\n\}", text, re.S).group(1)
    exits = re.findall(r"if \((.*)\) return (true|false);|while \((.*)\) \{", body)
    assert len(exits) == 3 and all((a or b).lstrip("!").startswith(("__all_sync(0xffffffffu,", "__any_sync(0xffffffffu,"))
                                   for a, _, b in exits)
