"""The order of equal scores from 32 orbitals on.

The reference compares the words of two determinants by the sign of their
wrapped difference (detComp_global, src/wavefunction.h:30-36).  Words that reach
2^63 need not have an order then: of two that differ in bit 63 alone neither
sorts first, and three can each sort after the next.  The leader's ranking must
still give every pick a place of its own.  Its rule: the number of equal-score
picks that sort before, and where that is equal the larger (alpha, beta).
"""
import itertools
import random

import pytest

TOP = 1 << 63


def _words(a, b):
    w = 0
    for p in range(64):
        w |= ((a >> p) & 1) << (2 * p) | ((b >> p) & 1) << (2 * p + 1)
    return w & (2**64 - 1), w >> 64


def _after(x, y):
    """det_ref_compare(x, y) > 0 on (alpha, beta) pairs."""
    xw, yw = _words(*x), _words(*y)
    i = 0 if xw[0] != yw[0] else 1
    diff = (xw[i] - yw[i]) % 2**64
    return xw[i] > yw[i] if diff == TOP else 0 < diff < TOP


def _ranks(dets):
    before = [sum(_after(e, d) for e in dets) for d in dets]
    return [sum((before[j], -e[0], -e[1]) < (before[i], -d[0], -d[1]) for j, e in enumerate(dets) if j != i)
            for i, d in enumerate(dets)]


def _det(r, s):
    return 1 << r, 1 << s


def test_ranks_are_places():
    # beta 31 against beta 32: word 0 differs in bit 63 alone; then a circle
    pair = [_det(3, 31), _det(3, 32)]
    assert sorted(_ranks(pair)) == [0, 1]
    circle = [_det(1, 32), _det(1, 30), _det(2, 31)]
    assert _after(circle[1], circle[0]) and _after(circle[2], circle[1]) and _after(circle[0], circle[2])
    assert [sum(_after(e, d) for e in circle) for d in circle] == [1, 1, 1]  # counting alone: places 0 and 2 empty
    rng = random.Random(1)
    for n in (2, 3, 5, 40):
        for _ in range(50):
            dets = rng.sample([_det(r, s) for r in range(34) for s in range(34)], n)
            ranks = _ranks(dets)
            assert sorted(ranks) == list(range(n))
            if all(_words(*d)[0] < TOP for d in dets) and all(_words(*d)[1] < TOP for d in dets):
                order = [d for _, d in sorted(zip(ranks, dets))]
                assert all(_after(x, y) for x, y in itertools.pairwise(order))


@pytest.mark.gpu
@pytest.mark.parametrize("k", [3, 32, 33, 128])
def test_picks_without_an_order(tmp_path, k):
    """One alpha and one beta electron in 34 orbitals, every double excitation of
    the reference coupled to it equally and nothing else: the candidates of the
    first column are the reference and k - 1 doubles with one score, among them
    circles and pairs that differ in bit 63 alone."""
    import mcdfci_b200 as m

    n = 34
    lines = [f"&FCI NORB={n},NELEC=2,MS2=0,", " ORBSYM=" + "1," * n, " ISYM=1,", "&END"]
    for r in range(1, n):
        lines += [f"0.125 {r + 1} 1 {s + 1} 1" for s in range(1, r + 1)]
    lines += ["-10.0 1 1 0 0"] + [f"1.0 {r + 1} {r + 1} 0 0" for r in range(1, n)] + ["0.0 0 0 0 0"]
    p = tmp_path / "equal.fcidump"
    p.write_text("\n".join(lines) + "\n")
    s = m.CDFCI(m.Fcidump(str(p)), num_of_coordinate=k, estimate=k, max_memory=0.05, threshold=0.0, z_threshold=0.0)
    s.reset()
    s.run_iterations(1)
    picked = [(int(a), int(b)) for a, b in zip(*s.picked()[:2])]
    x_size = s.report()["x_size"]
    s.close()
    assert len(set(picked)) == len(picked) == k and x_size == k
    assert picked[0] == (1, 1)
    doubles = picked[1:]
    assert all(a.bit_count() == b.bit_count() == 1 and a != 1 and b != 1 for a, b in doubles)
    ranks = _ranks(doubles)
    assert ranks == list(range(k - 1))
