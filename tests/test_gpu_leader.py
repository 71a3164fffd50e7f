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
