"""The column kernel's candidate selection (cta_select): the m largest of a
column whatever the CTAs per column, the blocks per CTA and the range of the
scores.

After reset the first iteration's candidates are the m best entries of the
reference determinant's column, with scores |1 + H_ref,ref| and |H_d,ref|
(x = e_ref), so with k = m the picks must be the oracle's column's m largest
scores.  Equal scores make the determinants ambiguous, not the scores, so the
sorted scores are compared: 1e-12 relative, the agreement of the matrix
elements themselves.
"""
import numpy as np
import pytest

from oracle.oracle import Oracle

import mcdfci_b200 as m
from mcdfci_b200 import synth

pytestmark = pytest.mark.gpu

# orbitals, alpha, beta: entries 35 (fewer than m), 254, 1,060 (one block and
# a ragged one), 5,871, and 14,469 (15 blocks)
SECTORS = [(4, 2, 1), (7, 3, 2), (10, 4, 3), (19, 5, 4), (24, 6, 5)]


@pytest.fixture(scope="module")
def problems(tmp_path_factory):
    d = tmp_path_factory.mktemp("candidates")
    out = {}
    for n, na, nb in SECTORS:
        for spread in (0, 18):
            spec = synth.SynthSpec(n, na, nb, -20.0, 1.0, 0.1, 2 * n)
            _, h1, eri, ecore = synth.make_integrals(spec, 3)
            if spread:
                # Couplings over 18 decades (60 binades), 8-fold symmetric.
                rng = np.random.default_rng(5)
                w = rng.uniform(-spread / 2, 0, size=(n, n))
                w = np.triu(w, 1)
                w = 10.0 ** (w + w.T)
                eri = eri * w[:, :, None, None] * w[None, None, :, :]
                h1 = np.where(np.eye(n, dtype=bool), h1, h1 * w)
                ecore -= 200.0
            p = str(d / f"n{n}_{na}a{nb}b_{spread}.fcidump")
            with open(p, "w") as f:
                f.write(synth.fcidump_text(spec, h1, eri, ecore))
            out[n, spread] = (p, Oracle(p, 0.0))
    return out


@pytest.mark.parametrize("spread", [0, 18])
@pytest.mark.parametrize("sector", SECTORS, ids=lambda s: f"n{s[0]}")
@pytest.mark.parametrize("mm,groups", [(1, 0), (1, 96), (31, 3), (32, 1), (33, 0), (64, 5), (100, 0), (128, 0), (128, 1),
                                       (128, 96)])
def test_first_candidates_are_the_largest(problems, sector, spread, mm, groups):
    path, o = problems[sector[0], spread]
    s = m.CDFCI(m.Fcidump(path), num_of_coordinate=mm, estimate=mm, max_memory=0.05, threshold=0.0, z_threshold=0.0,
                groups=groups)
    s.reset()
    ra, rb, _ = s.picked()
    ref = (int(ra[0]), int(rb[0]))
    s.run_iterations(1)
    pa, pb, _ = s.picked()
    s.close()
    ca, cb, cv = o.column_ab_arrays(*ref)
    score = {(int(a), int(b)): abs(v + (1.0 if (int(a), int(b)) == ref else 0.0)) for a, b, v in zip(ca, cb, cv)}
    picked = [(int(a), int(b)) for a, b in zip(pa, pb)]
    want = np.sort(np.array(list(score.values())))[::-1][:mm]
    assert len(set(picked)) == len(picked) == len(want)
    got = np.sort(np.array([score[d] for d in picked]))[::-1]
    assert np.all(np.abs(got - want) <= 1e-12 * want)


@pytest.mark.parametrize("groups", [1, 60, 96])
def test_launch_forms_agree(problems, groups):
    """One CTA a column, several waves of CTAs started beside the leader, and
    more waves than that, against one wave: 32 columns, the same table and
    energy after a few iterations up to the order of the sums (64-bit sums of
    at most 1e5 terms, 1e-16 each, relative to the energy)."""
    path, _ = problems[19, 0]
    sums = []
    for g in (18, groups):
        s = m.CDFCI(m.Fcidump(path), num_of_coordinate=32, estimate=128, max_memory=0.05, threshold=0.0,
                    z_threshold=0.0, groups=g)
        s.reset()
        s.run_iterations(6)
        r = s.report()
        sums.append((r["energy"], r["z_size"], r["x_size"], s.table_sums()))
        s.close()
    (e0, z0, x0, t0), (e1, z1, x1, t1) = sums
    assert abs(e0 - e1) <= 1e-11 * abs(e0)
    assert (z0, x0, t0["occupied"]) == (z1, x1, t1["occupied"])
