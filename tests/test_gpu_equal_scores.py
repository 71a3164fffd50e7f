"""Equal scores at the last place of a column's candidate list.

Of a column's determinants with equal scores the larger (alpha, beta) strings
stay.  So the list follows from the scores alone, whatever the CTAs, blocks and
lists a column is cut into and whichever warp comes first, and with one
coordinate per iteration (no two additions to one z) a solve repeats itself bit
for bit.
"""
import numpy as np
import pytest

import mcdfci_b200 as m
from mcdfci_b200 import synth
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


# 254, 1,060 (more than one block), 2,761 and 5,871 entries; open and closed shells
SECTORS = [(7, 3, 2), (10, 4, 3), (12, 5, 5), (19, 5, 4)]


@pytest.fixture(scope="module")
def problems(tmp_path_factory):
    """Integrals rounded to sixteenths (`coarse`) or, off the diagonal, to one
    of -1/8, 0 and 1/8: every matrix element is exact, and equal ones are few
    at a place, or hundreds."""
    d = tmp_path_factory.mktemp("equal")
    out = {}
    for n, na, nb in SECTORS:
        for coarse in (True, False):
            spec = synth.SynthSpec(n, na, nb, -20.0, 1.0, 0.1, 2 * n)
            _, h1, eri, ecore = synth.make_integrals(spec, 7)
            diag = np.diag(np.arange(-20.0, n - 20.0))
            if coarse:
                h1, eri = np.round(16 * h1) / 16, np.round(16 * eri) / 16
            else:
                h1, eri = np.sign(np.round(4 * h1)) / 8, np.sign(np.round(2 * eri)) / 8
            h1 = np.where(np.eye(n, dtype=bool), diag, h1)
            p = str(d / f"n{n}_{na}a{nb}b_{coarse}.fcidump")
            with open(p, "w") as f:
                f.write(synth.fcidump_text(spec, h1, eri, np.floor(ecore) - 200.0))
            out[n, coarse] = (p, Oracle(p, 0.0))
    return out


@pytest.mark.parametrize("mm,groups", [(1, 1), (8, 3), (33, 0), (100, 1), (128, 2), (128, 24)])
@pytest.mark.parametrize("coarse", [True, False])
@pytest.mark.parametrize("sector", SECTORS, ids=lambda s: f"n{s[0]}")
def test_larger_determinants_stay(problems, sector, coarse, mm, groups):
    path, o = problems[sector[0], coarse]
    s = m.CDFCI(m.Fcidump(path), num_of_coordinate=mm, estimate=mm, max_memory=0.05, threshold=0.0, z_threshold=0.0,
                groups=groups)
    s.reset()
    ra, rb, _ = s.picked()
    ref = (int(ra[0]), int(rb[0]))
    s.run_iterations(1)
    picked = [(int(a), int(b)) for a, b in zip(*s.picked()[:2])]
    s.close()
    ca, cb, cv = o.column_ab_arrays(*ref)
    value = {(int(a), int(b)): v + (1.0 if (int(a), int(b)) == ref else 0.0) for a, b, v in zip(ca, cb, cv)}
    value = {d: v for d, v in value.items() if v != 0.0}  # a single of value 0 is not inserted
    want = sorted(value, key=lambda d: (-abs(value[d]), -d[0], -d[1]))[:mm]
    assert set(picked) == set(want) and len(picked) == len(want)


@pytest.mark.parametrize("name", ["n12_6a6b", "n24_6a6b"])
def test_one_coordinate_repeats(synth_fcidumps, name):
    """Closed shell, k = m = 1: the best of a column is most often one of a
    mirror pair with equal scores."""
    runs = []
    for _ in range(6):
        s = m.CDFCI(m.Fcidump(synth_fcidumps[name]), num_of_coordinate=1, estimate=1, max_memory=0.5, threshold=0.0,
                    z_threshold=0.0)
        s.reset()
        s.run_iterations(256)
        a, b, x = s.wavefunction()
        order = np.lexsort((b, a))
        runs.append((a[order].tolist(), b[order].tolist(), x[order].tobytes(), s.report()["energy"]))
        s.close()
    assert all(r == runs[0] for r in runs[1:])


def test_circular_order_repeats(tmp_path):
    """34 orbitals, where the reference's order of determinants has circles (alpha
    30 and beta 32 sorts after 31 and 31, that after 33 and 31, and that after the
    first): picks among 127 equal scores."""
    n = 34
    lines = [f"&FCI NORB={n},NELEC=2,MS2=0,", " ORBSYM=" + "1," * n, " ISYM=1,", "&END"]
    for r in range(1, n):
        lines += [f"0.125 {r + 1} 1 {s + 1} 1" for s in range(1, r + 1)]
    lines += ["-10.0 1 1 0 0"] + [f"1.0 {r + 1} {r + 1} 0 0" for r in range(1, n)]
    lines += ["-10.0 1 0 0 0"] + [f"1.0 {r + 1} 0 0 0" for r in range(1, n)] + ["0.0 0 0 0 0"]
    p = tmp_path / "equal.fcidump"
    p.write_text("\n".join(lines) + "\n")
    for k in (8, 64):
        seen = set()
        for groups in (1, 2, 5) * 4:
            s = m.CDFCI(m.Fcidump(str(p)), num_of_coordinate=k, estimate=128, max_memory=0.05, threshold=0.0,
                        z_threshold=0.0, groups=groups)
            s.reset()
            s.run_iterations(1)
            seen.add(tuple(zip(*(v.tolist() for v in s.picked()[:2]))))
            s.close()
        assert len(seen) == 1
