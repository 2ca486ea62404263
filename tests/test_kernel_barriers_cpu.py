"""CPU test over the kernel sources: no __syncthreads() under a branch on the warp.

__syncthreads() may stand in conditional code only where the whole block takes
the same branch.  Warps that branch apart (`switch (warp)`) and meet at a barrier
all the same need one that counts arrivals whatever instruction they come from (a
numbered PTX barrier)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gf2_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def body(text, at):
    """The {...} block that opens at or after `at`."""
    start = i = text.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


def functions(text):
    """Device functions by name: their bodies."""
    out = {}
    for m in re.finditer(r"__device__[^;{}()]*?(\w+)\s*\(", text):
        close = text.find(")", m.end())
        semi, brace = text.find(";", close), text.find("{", close)
        if 0 <= brace < (semi if semi >= 0 else len(text)):
            out.setdefault(m.group(1), []).append(body(text, close))
    return out


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_block_barrier_under_a_branch_on_the_warp(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    funcs = functions(text)
    for m in re.finditer(r"switch\s*\(\s*(warp|wib|wid)\s*\)", text):
        seen, todo = set(), [body(text, m.end())]
        while todo:
            block = todo.pop()
            assert "__syncthreads" not in block
            for name in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", block)) & (set(funcs) - seen):
                seen.add(name)
                todo += funcs[name]
