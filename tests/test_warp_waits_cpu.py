"""Bounded waits of the kernels on the fifth-generation tensor cores: a warp whose lanes meet again (``__syncwarp``, a shuffle, a read
of tensor memory) gives a wait up as a whole.  Lanes that ran out, or saw another warp's flag, one by one would leave the others
waiting for them.  Read from the sources: on a GPU it could only be seen as a hang."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tiny_llm_infer_b200" / "csrc"
MEET = re.compile(r"__syncwarp|__shfl|__any_sync|__all_sync|tmem_ld|\bldmatrix|sync\.aligned")
WAIT = re.compile(r"\b(?:mbar_wait|wait)\(&")
VOTE = re.compile(r"__(?:any|all)_sync")


def code_of(text):
    return re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), text)


def blocks_of(code):
    """(start, end, header) of every brace block, inner ones too."""
    out, stack = [], []
    for i, c in enumerate(code):
        if c == "{":
            head = code[max(code.rfind(x, 0, i) for x in ";{}") + 1:i].strip()
            stack.append((i, head))
        elif c == "}":
            start, head = stack.pop()
            out.append((start, i, head))
    assert not stack
    return out


def lone_waits(text):
    """Places of waits whose lanes decide one by one, in a role (a branch on the warp) in which lanes meet."""
    code = code_of(text)
    blocks, bad = blocks_of(code), []
    for m in WAIT.finditer(code):
        around = sorted((b for b in blocks if b[0] < m.start() < b[1]), key=lambda b: b[0])
        if any(re.search(r"lane == 0|threadIdx\.x == 0|leader", head) for _, _, head in around):
            continue                                     # one thread
        role = [b for b in around if re.search(r"\bwarp\b|else$", b[2])]
        if not role or not MEET.search(code[role[-1][0]:role[-1][1]]):
            continue
        after = code[m.end():role[-1][1]]
        vote, parting = VOTE.search(after), re.search(r"\bbreak\b|\breturn\b", after)
        if vote and not (parting and parting.start() < vote.start()):
            continue                                     # decided together before any lane may leave
        bad.append(text.count("\n", 0, m.start()) + 1)
    return bad


@pytest.mark.parametrize("name", ["gemm_f32.cu", "gemm_tcgen05.cu", "attention_prefill_tc.cu"])
def test_a_warp_gives_a_wait_up_as_one(name):
    assert lone_waits((CSRC / name).read_text()) == []


def test_flags_are_not_read_lane_by_lane_where_lanes_meet():
    """A loop that every lane leaves by its own read of the block's flag parts the warp as a wait does."""
    code = code_of((CSRC / "gemm_f32.cu").read_text())
    for start, end, head in blocks_of(code):
        if re.search(r"\bfor\b.*(abort_flag|\*aborted)", head):
            assert not MEET.search(code[start:end]), head


def test_the_reading_finds_what_it_looks_for():
    kernel = """__global__ void k() { if (warp == 1) { if (lane == 0) { mbar_wait(&a, 0); } } else {
        for (;;) { if (!%s) { *aborted = 1; }
        if (%s) break; tmem_ld16(x, r); } } }"""
    assert lone_waits(kernel % ("mbar_wait(&b, 0)", "*aborted")) == [2]
    assert lone_waits(kernel % ("mbar_wait(&b, 0)", "__any_sync(0xffffffffu, *aborted != 0)")) == []
    assert lone_waits(kernel % ("warp_wait(&b, 0)", "*aborted")) == []
