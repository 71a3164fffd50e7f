"""When device memory is short, and what the calls that read a solved vector out
keep.

- An allocation that fails is reported by its own call alone.
- The scratch that a read-out leaves is given back to the solver's other
  allocations.
"""
import ctypes

import pytest

import mcdfci_b200 as m

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
