"""Instructions that a whole warp issues together (`.sync.aligned` loads of tensor memory,
`bar.sync`): on every way from a branch that lanes take differently to the next of them the
warp has to meet again in the source, since neither a loop's back edge nor the end of an `if`
promises it. Read from the kernels' sources: a divergence that the compiler happens to undo
shows in no result."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "lattica_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
LOADS = re.compile(r"\btmem_ld(?:4|8|16|_planes)\(|\breduce16\(")


def _code(path):
    """The source without comments, loops of loads alone as one load."""
    with open(path, encoding="utf-8") as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    return re.sub(r"\bfor \([^\n]*\) \{((?:\s*tc::tmem_ld[48]\([^{};]*;)+)\s*\}", r"\1", text)


def _block(text, at):
    """The text between the brace at `at` and its partner."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise ValueError("unbalanced braces")


def _flat(body):
    """A block without its nested blocks."""
    out, depth = [], 0
    for ch in body:
        depth += ch == "{"
        if depth == 0:
            out.append(ch)
        depth -= ch == "}"
    return "".join(out)


def _loops(text):
    """Bodies of the braced loops whose own statements load tensor memory."""
    for m in re.finditer(r"\bfor \(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        brace = re.match(r"\s*\{", text[i:])
        if brace:
            body = _block(text, i + brace.end() - 1)
            if LOADS.search(_flat(body)):
                yield body


def _meets(body):
    """The warp is whole before the body's loads in every turn: it meets at the turn's end,
    or first thing in the next one, and no turn ends early for some lanes."""
    ends = body.rstrip().endswith("__syncwarp();")
    begins = "lane0_wait(" in LOADS.split(_flat(body))[0]
    return (ends or begins) and "continue;" not in _flat(body)


def test_loops_over_tensor_memory_meet_between_turns():
    found = [(os.path.basename(p), body) for p in FILES for body in _loops(_code(p))]
    assert len(found) >= 8
    assert [name for name, body in found if not _meets(body)] == []


def test_the_rule_refuses_a_loop_that_parts():
    """The check itself: the same loop with the lanes parted, and met again."""
    loop = "\nfor (int n0 = 0; n0 < N; n0 += 8) {\n tmem_ld8(t, e);\n %s\n}\n"
    parted = ["if (m >= M) continue;\n store(e);", "if (m < M) {\n store(e);\n }"]
    for tail in parted:
        assert not any(_meets(b) for b in _loops(loop % tail))
    assert all(_meets(b) for b in _loops(loop % (parted[1] + "\n __syncwarp();")))


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_named_barriers_follow_a_meeting(path):
    text = _code(path)
    for m in re.finditer(r"\bbar\.(?:sync|red)", text):
        before = text[:m.start()]
        opened = before.rfind("asm volatile")
        between = before[before.rfind("__syncwarp();"):opened]
        assert between and "{" not in between and "if" not in between
