"""The calls that read a solved vector out of the table, against the table
itself: its nonzero coefficients in slot order, the residual, and the density
matrices by both ways of finding the connected pairs, from one determinant up
and over the edges of the comparison's tiles (8 by 256)."""
import numpy as np
import pytest

import mcdfci_b200 as m

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,iterations", [(1, 0), (1, 7), (4, 2), (8, 32), (8, 33), (16, 60)])
def test_readout_matches_table(fcidumps, k, iterations):
    s = m.CDFCI(m.Fcidump(fcidumps["n7_5a5b"]), num_of_coordinate=k, estimate=2 * k, max_memory=0.001,
                threshold=0.0, num_iterations=1000, report_interval=1000)
    s.reset()
    s.run_iterations(iterations)
    sa, sb, sx, sz = s.slots()
    keep = sx != 0.0
    a, b, x = s.wavefunction()
    # The slots come in no particular order beyond the table's own.
    order, want = np.lexsort((b, a)), np.lexsort((sb[keep], sa[keep]))
    np.testing.assert_array_equal(a[order], sa[keep][want])
    np.testing.assert_array_equal(b[order], sb[keep][want])
    np.testing.assert_array_equal(x[order], sx[keep][want])
    if not len(x):
        return
    lx, lz = sx.astype(np.longdouble), sz.astype(np.longdouble)
    e = (lx @ lz) / (lx @ lx)
    r = float(np.sqrt(((lz - e * lx) ** 2).sum() / (lx @ lx)))
    # 64-bit-mantissa sums of r, of size 1e-2 or more against |E x| of 1e2.
    assert abs(s.residual() - r) <= 1e-12 * max(r, 1.0)
    # An element sums at most one term x x' / x'x per determinant, each below 1.
    tol = 4 * len(x) * np.finfo(float).eps
    g1, g2 = s.rdm()
    for route in (1, 2):
        h1, h2 = s.debug_rdm(route)
        assert np.max(np.abs(g1 - h1)) <= tol * 10  # ten electrons' terms at most in an element of rdm1
        assert np.max(np.abs(g2 - h2)) <= tol * 10
    assert abs(np.trace(g1) - 10) <= 100 * tol
