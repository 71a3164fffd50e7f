"""The leader's pick and eig update inside a solve, at the edges of its layouts
(rows per warp and registers per lane of the bordered fixed point: 8, 16, 32,
64, 128; candidates per thread: 1, 4 and more).

Each iteration's subspace problem is read back and solved with numpy in 64
bits: the lowest eigenpair (lambda, v) of B = [[a, b'], [b, H]] with |rest|^2 =
xx - x'x, a = (xz - 2 x'z + x'Hx) / |rest|^2 and b = (z - Hx) / |rest| gives
dx = v_{i+1} |rest| / v_0 - x (src/solver.h:333-538).  Tolerance 1e-9 (1 +
|dx|), that of the recorded reference calls.  The picks must be distinct.
"""
import numpy as np
import pytest

import mcdfci_b200 as m
from mcdfci_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def path(tmp_path_factory):
    p = str(tmp_path_factory.mktemp("leader") / "n11.fcidump")
    synth.write_fcidump(p, synth.SynthSpec(11, 5, 4, -20.0, 1.0, 0.1, 22), seed=4)
    return p


@pytest.mark.parametrize("k,mm", [(1, 1), (7, 8), (8, 100), (9, 20), (16, 32), (17, 40), (32, 64), (33, 64), (64, 100),
                                  (65, 128), (96, 128), (127, 128), (128, 128)])
def test_update_matches_numpy(path, k, mm):
    s = m.CDFCI(m.Fcidump(path), num_of_coordinate=k, estimate=mm, max_memory=0.02, threshold=0.0, z_threshold=0.0)
    s.reset()
    for it in range(12):
        s.run_iterations(1)
        steps = s.report()["inv_steps_last"]  # of the bordered form; 0 when the reduction ran
        pa, pb, dx = s.picked()
        assert len(set(zip(pa.tolist(), pb.tolist()))) == len(pa)
        e = s.last_eig_inputs()
        H, x, z = e["hsub"], e["x"], e["z"]
        assert np.array_equal(H, H.T)
        xx, xz = float(e["xx"].sum()), float(e["xz"].sum())
        rest = xx - float(x @ x)
        if it == 0 or rest <= 1e-10:
            continue
        n = e["k"]
        B = np.zeros((n + 1, n + 1))
        B[0, 0] = (xz - 2.0 * float(x @ z) + float(x @ H @ x)) / rest
        B[0, 1:] = B[1:, 0] = (z - H @ x) / np.sqrt(rest)
        B[1:, 1:] = H
        w, u = np.linalg.eigh(B)
        v = u[:, 0]
        want = v[1:] / v[0] * np.sqrt(rest) - x
        assert np.max(np.abs(dx - want) / (1.0 + np.abs(want))) < 1e-9, it
        # The bordered form certifies only an eigenvalue below H's Gershgorin bound.
        g = np.min(np.diag(H) - (np.abs(H).sum(axis=1) - np.abs(np.diag(H))))
        assert steps == 0 or w[0] < g + 1e-9
    s.close()


def _fixed_point(H, x, z, xx, xz):
    """The bordered fixed point of the leader (eig_bordered) with numpy: the
    steps it takes to converge, or None when it gives up, and its tolerance."""
    d = np.diag(H).copy()
    E = H - np.diag(d)
    rest = xx - float(x @ x)
    a, b = (xz - 2.0 * float(x @ z) + float(x @ H @ x)) / rest, (z - H @ x) / np.sqrt(rest)
    off = np.abs(E).sum(axis=1)
    g = np.min(d - off)
    tol = 1e-15 * max(np.max(np.abs(d) + off + np.abs(b)), abs(a) + np.abs(b).sum())
    y = x / np.sqrt(rest)
    lam = a + b @ y
    cold = not lam < g
    if cold:
        y, lam = np.zeros_like(x), min(a, g) - 1e-3 * (1.0 + abs(a))
    last = np.inf
    for t in range(64):
        s = b + E @ y
        new = -s / (d - lam)
        r = np.linalg.norm((d - lam) * (y - new)) / np.sqrt(1.0 + y @ y)
        if t % 2 == 0:
            if (r <= tol or (t >= 2 and r > 0.25 * last and r <= 16 * tol)) and not (cold and t == 0):
                return t + 1, tol
            if not r < 1e140 or (t >= 8 and r > 0.8 * last) or (t >= 4 and not lam < g):
                return None, tol
            last = r
        y = new
        lam = a + b @ y
    return None, tol


@pytest.mark.parametrize("k", [8, 33, 65, 96, 127, 128])
def test_bordered_form_is_taken(tmp_path, k):
    """Where the fixed point converges (in 48 steps or fewer, the limit being 64),
    the leader takes its result, with a residual of at most 16 times its
    tolerance (17 for the rounding of dx, 2^-53 |x + dx| times a row of B, below
    a tenth of it)."""
    p = str(tmp_path / "n16.fcidump")
    synth.write_fcidump(p, synth.SynthSpec(16, 5, 4, -20.0, 1.0, 0.1, 32), seed=4)
    s = m.CDFCI(m.Fcidump(p), num_of_coordinate=k, estimate=min(128, 2 * k), max_memory=1.0, threshold=0.0,
                z_threshold=0.0)
    s.reset()
    taken = 0
    for it in range(24):
        s.run_iterations(1)
        if it == 0:
            continue
        steps = s.report()["inv_steps_last"]
        e = s.last_eig_inputs()
        H, x, z, xx, xz = e["hsub"], e["x"], e["z"], float(e["xx"].sum()), float(e["xz"].sum())
        want, tol = _fixed_point(H, x, z, xx, xz)
        if want is not None and want <= 48:
            assert steps > 0, (it, want)
        if steps == 0:
            continue
        taken += 1
        rest = xx - float(x @ x)
        b = (z - H @ x) / np.sqrt(rest)
        y = (x + s.picked()[2]) / np.sqrt(rest)
        lam = (xz - 2.0 * float(x @ z) + float(x @ H @ x)) / rest + b @ y
        assert np.linalg.norm(b + H @ y - lam * y) <= 17.0 * tol * np.sqrt(1.0 + y @ y)
    s.close()
    assert taken >= 12
