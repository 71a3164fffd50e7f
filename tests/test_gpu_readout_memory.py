"""When device memory is short, and what the calls that read a solved vector out
keep.

- An allocation that fails is reported by its own call alone.
- The scratch that a read-out leaves is given back to the solver's other
  allocations.
- Coefficients need no memory beside the table: the list of determinants is
  made in ranges of the table that fit what there is, down to the solver's own
  partial sums.
- Density matrices summed from parts of the list equal those from all of it.
- The matrices leave through a pinned block of 32 MB, in several pieces from 45
  orbitals on.
"""
import ctypes

import numpy as np
import pytest

import mcdfci_b200 as m
from mcdfci_b200 import synth

pytestmark = pytest.mark.gpu


class _Full:
    """The device's free memory, allocated down to pieces of 4 KB."""

    def __enter__(self):
        self.cu, self.held = ctypes.CDLL("libcuda.so.1"), []
        size = 1 << 37
        while size >= 4096:
            p = ctypes.c_uint64()
            if self.cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
                self.held.append(p)
            else:
                size //= 2
        assert self.held
        return self

    def __exit__(self, *_):
        for p in self.held:
            self.cu.cuMemFree_v2(p)


def _solver(path, k, iterations, **kw):
    s = m.CDFCI(m.Fcidump(path), num_of_coordinate=k, estimate=k, max_memory=0.5, threshold=0.0, **kw)
    s.reset()
    s.run_iterations(iterations)
    s.report()
    return s


def test_an_error_is_reported_once(synth_fcidumps):
    """A growth without memory fails; the calls after it do not fail again."""
    s = _solver(synth_fcidumps["n24_6a6b"], 1, 0, num_iterations=1, report_interval=1)
    with _Full():
        with pytest.raises(m.McdError, match="out of memory"):
            s.grow()
    before = s.report()["occupied"]
    s.grow()
    assert s.report()["occupied"] == before and s.table_info()["capacity"] == 1 << 17
    s.close()


def test_growth_takes_the_scratch(synth_fcidumps):
    """A table of 2 MB grows to 4 MB with nothing free but the 8 MB that the
    density matrices of 24 orbitals left."""
    path = synth_fcidumps["n24_6a6b"]
    for full in (False, True):
        s = _solver(path, 1, 0, num_iterations=1, report_interval=1)
        s.rdm()
        before = s.table_info()["capacity"]
        assert before == 1 << 16
        if full:
            with _Full():
                s.grow(0)
        else:
            s.grow(0)
        assert s.table_info()["capacity"] == 2 * before
        s.close()


def test_coefficients_without_memory(synth_fcidumps):
    """3,000 determinants and more in a table of 2^22 slots: several times the 591
    that the partial sums hold."""
    path = synth_fcidumps["n16_5a5b"]
    first = _solver(path, 64, 8)
    first.wavefunction()  # (its kernels are loaded with memory at hand)
    first.close()
    s = _solver(path, 64, 96, table_growth=False)
    with _Full():
        a, b, x = s.wavefunction()
    sa, sb, sx, _ = s.slots()
    keep = sx != 0.0
    assert keep.sum() > 3000
    np.testing.assert_array_equal(a, sa[keep])
    np.testing.assert_array_equal(b, sb[keep])
    np.testing.assert_array_equal(x, sx[keep])
    s.close()


def test_matrices_from_parts(synth_fcidumps):
    s = _solver(synth_fcidumps["n16_5a5b"], 64, 96)
    n = len(s.wavefunction()[2])
    assert n > 3000
    g1, g2 = s.debug_rdm(2)
    h1, h2 = s.debug_rdm(3)
    s.close()
    # An element sums at most one term per determinant and electron, each below 1.
    tol = 4 * n * np.finfo(float).eps * 10
    assert np.max(np.abs(g1 - h1)) <= tol and np.max(np.abs(g2 - h2)) <= tol


def test_matrices_in_pieces(tmp_path):
    """48 orbitals, 42.5 MB: partial traces that every element takes part in,
    sum_q Gamma_pqrq = (N - 1) gamma_pr, and the symmetry Gamma_pqrs = Gamma_qpsr."""
    spec = synth.SynthSpec(48, 2, 1, -3.0, 1.0, 0.08, 48, decay=6.0)
    p = str(tmp_path / "n48.fcidump")
    synth.write_fcidump(p, spec, seed=2, drop_below=1e-3)
    s = _solver(p, 64, 40, z_threshold=1e-6)
    g1, g2 = s.rdm()
    s.close()
    assert abs(np.trace(g1) - 3) < 1e-12
    assert np.max(np.abs(np.einsum("pqrq->pr", g2) - 2 * g1)) < 1e-12
    assert np.max(np.abs(g2 - g2.transpose(1, 0, 3, 2))) < 1e-12
    assert all(np.count_nonzero(part) for part in (g2[:8], g2[8:30], g2[30:37], g2[38:]))
