"""How the kernels use their bounded waits, read from the sources: what happens when a wait gives up cannot be tried on a GPU
(it would take a kernel that is broken on purpose)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastnn_b200", "csrc")


def code_of(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def block_after(text, at):
    """The span of the braces that open behind `at`."""
    first = text.index("{", at)
    depth = 0
    for i in range(first, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return first, i
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("name", ["qmm_tc.cu", "qmm_tc_pair.cu"])
def test_waits_of_whole_warps_have_one_answer(name):
    """Outside the blocks of an elected thread every lane of a warp waits by itself, and what follows is for converged warps:
    tensor-memory accesses and cluster arrivals.  So either the wait votes, or its answer decides over nothing but one
    lane's arrival, and the lanes stay together whatever it is."""
    text = code_of(name)
    elected = [block_after(text, m.start()) for m in re.finditer(r"if \(elect_one\(\)\)", text)]
    assert elected
    inside = lambda at: any(a <= at <= b for a, b in elected)
    whole = [m.start() for m in re.finditer(r"\bmbar_wait_warp\(", text)]
    assert whole and not any(inside(at) for at in whole)
    lone = [m for m in re.finditer(r"(?:const bool (\w+) = )?\bmbar_wait\(", text) if not inside(m.start())]
    assert len(lone) == 1
    answer = lone[0].group(1)
    assert answer, text[lone[0].start():][:80]
    def statements(word):
        return [u.strip() for u in re.findall(rf"[^;{{}}]*\b{word}\b[^;]*;", text)]
    kept = re.fullmatch(rf"(\w+) &= {answer};", statements(answer)[1])   # once it is false it stays false
    assert kept and len(statements(answer)) == 2, statements(answer)
    uses = statements(kept.group(1))
    assert len(uses) == 3 and uses[0] == f"bool {kept.group(1)} = true;", uses
    assert uses[2].startswith(f"if (lane == 0 && {kept.group(1)}) mbar_arrive"), uses


@pytest.mark.parametrize("name", ["qmm_mma8.cu", "qmm_tc.cu", "qmm_tc_pair.cu"])
def test_no_answer_of_a_wait_is_dropped(name):
    """What a wait was for is not there when it gives up: the kernel has to leave without using it."""
    text = code_of(name)
    calls = list(re.finditer(r"\bmbar_wait(?:_warp)?\(", text))
    assert calls
    for m in calls:
        head = re.split(r"[;{}]", text[:m.start()])[-1].strip()
        assert re.search(r"(=|&&|!|if \()\s*(tc::)?$", head), head


def test_rows_that_never_came_end_the_fragment_kernel():
    """The 8-bit fragment kernel: the block leaves as a whole between the wait for its rows and the first weight."""
    text = code_of("qmm_mma8.cu")
    wait = re.search(r"(\w+) = tc::mbar_wait\(s_rows_bar", text)
    leave = re.search(rf"if \(!__syncthreads_and\({wait.group(1)}\)\) ", text)
    assert leave and leave.start() > wait.start()
    first, last = block_after(text, leave.end() - 1)
    assert "cp_async_wait<0>()" in text[first:last] and "return;" in text[first:last]
    assert last < text.index("for (int tl = 0; tl < tiles_here; ++tl)")
