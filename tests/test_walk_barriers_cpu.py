"""Shared-memory order of the tree walks' stacks, read from the source.

A warp's lanes push children for one another, so a store to the stack has to be
followed by a warp barrier before any load of it (and a load by one before the
next stores), on every path through the walk's loop.  Such a race need not show
in a run: the compiled code may keep the lanes together by itself.  The test
takes the loads, stores and barriers of the loop in text order, with the brace
blocks that they stand in, and asks for a barrier between each store and each
load that every lane passes whenever it passes one of the two.
"""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "n-body-2d_b200" / "csrc"


def _loop_body(text, head="while (size > 0) {"):
    text = re.sub(r"//[^\n]*", "", text)
    assert text.count(head) == 1
    at = text.index(head) + len(head)
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end - 1]


def _events(body):
    """[(kind, path of the enclosing blocks)] in text order."""
    access = re.compile(r"(?:\bL\.stack|\bdst)\[")
    found = []
    for m in access.finditer(body):
        depth, end = 1, m.end()
        while depth:
            depth += {"[": 1, "]": -1}.get(body[end], 0)
            end += 1
        store = re.match(r"\s*=[^=]", body[end:]) is not None
        found.append((m.start(), "store" if store else "load"))
    for m in re.finditer(r"__sync(?:warp|threads)\(\)", body):
        before = body[:m.start()].rstrip()
        assert before == "" or before[-1] in ";{}", "a barrier under a condition without a block"
        found.append((m.start(), "barrier"))
    out, path, opened = [], [], 0
    marks = dict(found)
    for k, ch in enumerate(body):
        if k in marks:
            out.append((marks[k], tuple(path)))
        if ch == "{":
            opened += 1
            path.append(opened)
        elif ch == "}":
            path.pop()
    return out


def _passed(barrier, access):
    """Lanes that pass `access` pass `barrier` in the same iteration."""
    return access[:len(barrier)] == barrier


@pytest.mark.parametrize("name", ["k_force32.cu", "k_force64.cu"])
def test_a_barrier_between_pushes_and_pops(name):
    events = _events(_loop_body((CSRC / name).read_text()))
    kinds = [k for k, _ in events]
    assert "load" in kinds and "store" in kinds and "barrier" in kinds
    twice = events + events  # the next iteration
    for i in range(len(events)):
        a, pa = events[i]
        for j in range(i + 1, i + len(events)):
            b, pb = twice[j]
            if {a, b} != {"store", "load"}:
                continue
            between = [p for k, p in twice[i + 1:j] if k == "barrier"]
            assert any(_passed(p, pa) or _passed(p, pb) for p in between), (
                f"{name}: {a} {i} and {b} {j % len(events)} of the stack have no barrier between")
