"""Tensor-memory loads (tcgen05.ld .sync.aligned) need their whole warp together. In the sources: a
loop body that lanes can leave early (`continue`, or `return` from a lambda in it) brings the warp together again (__syncwarp) before
a load in it."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "iane_gb300" / "csrc"
CALL = re.compile(r"\btc::ld_32x32b\w*\(")


def loops_around(text, at):
    """(start, end) of the braces of every for/while loop around position `at`."""
    stack, spans = [], []
    for i, c in enumerate(text):
        if c == "{":
            stack.append(i)
        elif c == "}":
            spans.append((stack.pop(), i))
    for start, end in spans:
        if start < at < end and re.search(r"\b(for|while)\s*\([^{}]*\)\s*$", text[:start]):
            yield start, end


def offences(text):
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), text)
    for call in CALL.finditer(text):
        for start, end in loops_around(text, call.start()):
            if re.search(r"\b(continue|return);", text[start:end]) and "__syncwarp()" not in text[start:call.start()]:
                yield text[:call.start()].count("\n") + 1


@pytest.mark.parametrize("path", sorted(p for p in CSRC.glob("*.cu*") if CALL.search(p.read_text())),
                         ids=lambda p: p.name)
def test_warps_are_together_before_a_tensor_memory_load(path):
    assert not list(offences(path.read_text()))


def test_the_batch_s_warps_sum_together():
    # thread 0 takes tiles from the queue while its warp waits for one: brought together before the sums, or
    # the two parts sum one after the other
    text = (CSRC / "rl_batch_kernel.cu").read_text()
    loop = text[text.index("for (unsigned int n = 0;; ++n)"):]
    wait, sums = loop.index("mbar_wait_bounded(&sh->full"), loop.index("item_sums(tile")
    assert "__syncwarp();" in loop[wait:sums]
