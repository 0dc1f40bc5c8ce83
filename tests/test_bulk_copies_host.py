"""Shared memory that a bulk copy (cp.async.bulk) still reads is not written again: looked up in the sources, as no run can show it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmq_b200", "csrc")
WAIT, COMMIT = "cp.async.bulk.wait_group.read", "cp.async.bulk.commit_group"


def text_of(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def conditions(text, at):
    """what stands before each block around the statement at text[at], outermost first; the statement's own `if`"""
    heads, start, depth = [], 0, 0
    for i, c in enumerate(text[:at]):
        if c == "(":
            depth += 1
        elif c == ")":
            depth -= 1
        elif c == "{" and depth == 0:
            heads.append(" ".join(text[start:i].split()))
            start = i + 1
        elif c == "}" and depth == 0 and heads:
            heads.pop()
            start = i + 1
        elif c == ";" and depth == 0:
            start = i + 1
    return heads, [" ".join(text[start:at].split())] if text[start:at].strip() else []


def waits():
    """(file, its text, place, groups that may be pending) of every wait that leaves some"""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = text_of(name)
            for m in re.finditer(re.escape(WAIT) + r' (?:%0;" ::"n"\((.*?)\)|(\d+);)', text):
                if (m.group(1) or m.group(2)) != "0":
                    yield name, text, text.rindex("asm", 0, m.start())


@pytest.mark.parametrize("name,text,at", [pytest.param(*w, id=w[0]) for w in waits()])
def test_every_use_of_a_buffer_is_a_group(name, text, at):
    """A wait that leaves groups pending counts groups, not buffers: in its loop every use of a buffer commits one, whether or not it copies
    anything, under the condition of the wait and no other"""
    block, own = conditions(text, at)
    assert [h for h in block if "for (" in h], "a wait outside a loop"
    inside = []
    for m in re.finditer(re.escape(COMMIT), text):
        heads, last = conditions(text, text.rindex("asm", 0, m.start()))
        if heads[:len(block)] == block:
            inside.append([h for h in heads[len(block):] + last if h not in own])
    assert inside and not any(inside), ("a group only where", inside)


def test_the_waits_are_found():
    assert {w[0] for w in waits()} >= {"prefill_attn.cu", "gemm_rows.cu"}
