"""How a column CTA takes the picked determinant over from the leader
(column_body, mcdfci_b200/csrc/column_kernel.cu), on the CPU.

The CTA reads the picks once before the leader has ended and, when its column
was not among them, again after it.  Both readings pass their answer through
one word of shared memory: warp 0 writes it, a barrier follows, every warp
reads it.  The steps are taken from the source in their order, and every
interleaving of two warps is walked through, with each pair of answers that
the two readings can give: the warps must agree on what they read, and meet at
the same barriers.
"""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "mcdfci_b200", "csrc", "column_kernel.cu")


def _function(name):
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    at = re.search(r"__device__ __forceinline__ \w+ %s\([^)]*\) \{" % name, text).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end - 1]


def _steps():
    """The hand-over of column_body: ("read", i) the i-th call of read_picked,
    ("barrier",) a __syncthreads between them."""
    body = _function("column_body")
    body = body[:body.index("const int total")]
    tokens = re.findall(r"read_picked\(|__syncthreads\(\)", body)
    assert tokens.count("read_picked(") == 2 and tokens[0] == tokens[-1] == "read_picked("
    steps, reads = [], 0
    for t in tokens:
        if t == "__syncthreads()":
            steps.append(("barrier",))
        else:
            steps.append(("read", reads))
            reads += 1
    return steps


def _program(warp, steps, answers):
    """One warp: yields ("write", value), ("barrier",) or ("read",), is sent
    the word at a read; returns whether the column is computed, and by which
    reading."""
    for s in steps:
        if s[0] == "barrier":
            yield s
            continue
        if warp == 0:
            yield ("write", answers[s[1]])
        yield ("barrier",)
        if (yield ("read",)):
            return s[1]
    return None


def _outcomes(steps, answers):
    """Every result (a tuple over the warps; "stuck" for barriers that do not
    match) over the interleavings, each replayed from its schedule."""
    found, todo = set(), [()]
    while todo:
        schedule = todo.pop()
        warps = [_program(w, steps, answers) for w in range(2)]
        at = [next(w) for w in warps]
        word, result = None, [None, None]
        done = [False, False]

        def move(w, value=None):
            try:
                at[w] = warps[w].send(value)
            except StopIteration as e:
                done[w], result[w], at[w] = True, e.value, ("end",)

        def settle():
            while at[0] == at[1] == ("barrier",):
                move(0)
                move(1)

        settle()
        for w in schedule:
            if at[w][0] == "write":
                word = at[w][1]
                move(w)
            else:
                move(w, word)
            settle()
        free = [w for w in range(2) if at[w][0] in ("write", "read")]
        if not free:
            found.add(tuple(result) if all(done) else "stuck")
        todo.extend(schedule + (w,) for w in free)
    return found


@pytest.mark.parametrize("first", [False, True])
@pytest.mark.parametrize("second", [False, True])
def test_warps_agree_on_the_reading(first, second):
    want = 0 if first else 1 if second else None
    assert _outcomes(_steps(), (first, second)) == {(want, want)}


def test_walk_finds_a_missing_barrier():
    """Two readings with nothing between them: a late warp takes the second
    answer for the first."""
    found = _outcomes([("read", 0), ("read", 1)], (False, True))
    assert found - {(1, 1)}


def test_slice_is_taken_of_the_own_sector_only():
    """A CTA that finds after the leader's end that its first reading named
    another determinant probes the new one over the slice it already has.  The
    number of entries depends on the electrons per spin alone, so the first
    reading counts only with those of the launch; anything else (the zeroed state
    of a column that no iteration has had) waits for the second reading."""
    body = _function("column_body")
    first = re.search(r"early = ([^;]*);", body[body.index("pdl_trigger"):]).group(1)
    assert re.fullmatch(r"read_picked\([^)]*\) && S\.P\.na == L\.na && S\.P\.nb == L\.nb", first)
