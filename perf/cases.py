"""Timed work of the mCDFCI solver, through the calls a program makes.

A case is one of five kinds:

solve     ``CDFCI.solve()`` on a solver that the program holds: from the
          reference determinant, a fixed number of iterations with a report
          every few of them, as a program reads them to watch the energy.
point     one point of a curve from its FCIDUMP: create, solve, close.
batch     ``CDFCIBatch.solve()`` over the points of a dissociation curve.
readout   after a solve: the residual ||H c - E c|| / ||c|| and the 1- and
          2-RDM (the energy gradient), ``CDFCI.residual()`` and ``CDFCI.rdm()``.
coefs     after a solve: the determinants and coefficients,
          ``CDFCI.wavefunction()``, in determinant order.
eig       one subspace eigen-update on host buffers, ``eig_update_static()``.

The integrals are those of ``mcdfci_b200.synth``, drawn from the seed.
"""
import math
import os
import tempfile

import numpy as np

import mcdfci_b200 as mc
from mcdfci_b200 import synth

ENTRY_BYTES = 40  # 16-byte key, x, and z read and written, per column entry
SLOT_BYTES = 32


def _case(kind, name=None, **kw):
    c = dict(kind=kind, **kw)
    if name is not None:
        c["name"] = name
    return c


# The list of candidates per column (`m`, the solver's `estimate`) is its
# default of 100 or longer than k by a third and more, and the shells are
# open.  With m = k, or with the mirror-image determinants of a closed shell,
# which of two nearly equal determinants is picked follows the order of
# concurrent additions, and a solve's path does not repeat.


def listed():
    return [
        # 735 determinants: the smallest problem, all launch latency.
        _case("solve", "tiny_n7_k8", norb=7, na=5, nb=4, k=8, m=100, iterations=600, report=300, max_memory=0.005,
              zt=0.0),
        # The solver's default options (one coordinate, 100 candidates).
        _case("solve", "defaults_n12_k1", norb=12, na=6, nb=6, k=1, m=100, iterations=512, report=128,
              max_memory=0.1, zt=0.0),
        # The size of the energy-gradient workload, on the way to its converged vector.
        _case("solve", "gradient_n12_k32", norb=12, na=6, nb=5, k=32, m=64, iterations=256, report=128,
              max_memory=0.1, zt=0.0),
        # Ragged sizes.
        _case("solve", "ragged_n19_k24", norb=19, na=5, nb=4, k=24, m=100, iterations=200, report=50,
              max_memory=0.8, zt=1e-9),
        # The throughput workload: 1.2e10 determinants, a table far larger than L2.
        _case("solve", "throughput_n24_k32", norb=24, na=6, nb=5, k=32, m=64, iterations=256, report=128,
              max_memory=16.0, zt=1e-9),
        # Many coordinates per iteration.
        _case("solve", "wide_n24_k96", norb=24, na=6, nb=5, k=96, m=128, iterations=64, report=64,
              max_memory=16.0, zt=1e-9),
        # The large active space: about 265,000 entries per column.
        _case("solve", "large_n42_k64", norb=42, na=24, nb=23, k=64, m=128, iterations=16, report=16,
              max_memory=24.0, zt=1e-9),
        # One curve point on its own, from its FCIDUMP to its energy.
        _case("point", "point_n16_k16", norb=16, na=5, nb=4, k=16, m=32, iterations=200, report=100,
              max_memory=1.0, zt=0.0),
        # The whole curve as a batch.
        _case("batch", "curve32_n16_k16", norb=16, na=5, nb=4, points=32, k=16, m=32, iterations=128, report=64,
              max_memory=1.0, zt=0.0),
        # Residual and gradient of a solved vector in a 4.3 GB table.
        _case("readout", "readout_n24", norb=24, na=6, nb=5, k=32, m=64, iterations=24, max_memory=4.0),
        # Coefficients of a solved vector.
        _case("coefs", "coefs_n16", norb=16, na=5, nb=4, k=16, m=32, iterations=64, max_memory=1.0),
        # A host program's own subspace update.
        _case("eig", "eig_k48", k=48),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sector(rng, lo, hi):
    """Orbitals and electrons with at least 2000 determinants."""
    while True:
        n = _logint(rng, lo, hi)
        na = rng.randint(2, max(2, min(n - 2, 24)))
        nb = max(1, na - rng.choice([1, 1, 2]))
        if math.comb(n, na) * math.comb(n, nb) >= 2000:
            return n, na, nb


def entries(norb, na, nb):
    """Entries of one Hamiltonian column."""
    va, vb = norb - na, norb - nb
    return (1 + na * va + nb * vb + math.comb(na, 2) * math.comb(va, 2) + math.comb(nb, 2) * math.comb(vb, 2)
            + na * nb * va * vb)


def _max_memory(slots_wanted, norb):
    """The max_memory (GB) that gives the smallest power of two of slots above slots_wanted."""
    slots = 1 << max(16, math.ceil(math.log2(slots_wanted)))
    return slots * (8 * (1 + (2 * norb - 1) // 64) + 16) * 1.01 / 2**30


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "point", "batch", "readout", "coefs", "eig"])
    if kind == "eig":
        return _case(kind, k=_logint(rng, 2, 128))
    n, na, nb = _sector(rng, 7, {"solve": 42, "point": 24, "batch": 18, "readout": 26, "coefs": 24}[kind])
    e = entries(n, na, nb)
    dets = math.comb(n, na) * math.comb(n, nb)
    if kind in ("solve", "point"):
        k = min(_logint(rng, 1, 96 if kind == "solve" else 32), max(1, dets // 20))
        m = min(128, rng.choice([2 * k + 2, 100, rng.randint(k, 128)]))
        m = max(m, k + max(k // 3, 12))
        its = max(4, min(_logint(rng, 40, 600), int(1.2e8 / (k * e))))
        return _case(kind, norb=n, na=na, nb=nb, k=k, m=m, iterations=its, report=max(1, its // rng.choice([1, 2, 3])),
                  max_memory=round(_max_memory(min(dets, its * k * e) * 2.0, n), 4),
                  zt=rng.choice([0.0, 0.0, 1e-10, 1e-9]))
    if kind == "batch":
        k = min(_logint(rng, 4, 32), max(1, dets // 20))
        points = rng.randint(2, 32)
        its = max(4, min(rng.randint(32, 160), int(1.5e8 / (points * k * e))))
        return _case(kind, norb=n, na=na, nb=nb, points=points, k=k, m=rng.choice([2 * k + 16, 100]), iterations=its,
                     report=max(1, its // 2), max_memory=round(_max_memory(min(dets, its * k * e) * 2.0, n), 4),
                     zt=0.0)
    k = min(_logint(rng, 4, 32), max(1, dets // 20))
    its = max(4, min(rng.randint(8, 48), int(3e7 / (k * e))))
    return _case(kind, norb=n, na=na, nb=nb, k=k, m=2 * k + 16, iterations=its,
                 max_memory=round(_max_memory(max(min(dets, its * k * e) * 2.0, _logint(rng, 2**18, 2**26)), n), 4))


# ---------------------------------------------------------------------------

def _spec(norb, na, nb):
    """The value distributions of the nearest named workload."""
    if norb <= 16:
        return synth.SynthSpec(norb, na, nb, -20.0, 1.0, 0.1, 2 * norb)
    if norb <= 30:
        return synth.SynthSpec(norb, na, nb, -5.0, 2.0, 0.05, 2 * norb)
    return synth.SynthSpec(norb, na, nb, -3.0, 1.0, 0.08, 2 * norb, decay=6.0)


def _write(d, case, seed, t=None):
    spec = _spec(case["norb"], case["na"], case["nb"])
    path = os.path.join(d, "t%s.fcidump" % ("" if t is None else "%.4f" % t))
    synth.write_fcidump(path, spec, seed=seed, t=t)
    return path


def _options(case):
    return dict(num_of_coordinate=case["k"], estimate=case["m"], max_memory=case["max_memory"],
                z_threshold=case.get("zt", 0.0), threshold=0.0, num_iterations=case["iterations"],
                report_interval=case.get("report", case["iterations"]), device=0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "eig":
        return {"kind": kind, "args": _eig_inputs(case["k"], seed)}
    with tempfile.TemporaryDirectory() as d:
        if kind == "batch":
            n = case["points"]
            fcs = [mc.Fcidump(_write(d, case, seed, t=i / (n - 1))) for i in range(n)]
            return {"kind": kind, "batch": mc.CDFCIBatch(fcs, **_options(case))}
        fc = mc.Fcidump(_write(d, case, seed))
    if kind == "point":
        return {"kind": kind, "fcidump": fc, "options": _options(case)}
    if kind == "solve":
        return {"kind": kind, "solver": mc.CDFCI(fc, **_options(case))}
    s = mc.CDFCI(fc, table_growth=False, **_options(case))
    s.solve()
    # At most k determinants per iteration, and the first, carry a coefficient.
    return {"kind": kind, "solver": s, "rows": case["k"] * case["iterations"] + 1}


def _columns(reports):
    """The energy and the scale of every report, and the last energy."""
    return {"energy": np.array([r["energy"] for r in reports]), "scale": np.array([r["scale"] for r in reports]),
            "final": np.float64(reports[-1]["energy"])}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        s = state["solver"]
        s.solve()
        return _columns(s.reports)
    if kind == "point":
        s = mc.CDFCI(state["fcidump"], **state["options"])
        s.solve()
        s.close()
        return _columns(s.reports)
    if kind == "batch":
        b = state["batch"]
        b.solve()
        return _columns([r for reports in b.reports for r in reports])
    if kind == "readout":
        s = state["solver"]
        residual = s.residual()
        rdm1, rdm2 = s.rdm()
        return {"residual": np.float64(residual), "rdm1": rdm1, "rdm2": rdm2}
    if kind == "coefs":
        a, b, x = state["solver"].wavefunction()
        order = np.lexsort((b, a))
        out = {"alpha": np.zeros(state["rows"], np.int64), "beta": np.zeros(state["rows"], np.int64),
               "x": np.zeros(state["rows"])}
        for name, v in (("alpha", a.view(np.int64)), ("beta", b.view(np.int64)), ("x", x)):
            out[name][: len(order)] = v[order]
        return out
    dx, xx, scale, branch = mc.eig_update_static(*state["args"])
    return {"dx": dx, "xx": np.float64(xx[0]), "scale": np.float64(scale[0]), "branch": branch}


# ---------------------------------------------------------------------------
# The eigen-update's inputs: the current vector is sqrt(rest) times a
# normalised rest vector of energy e0 plus x on the k picked determinants;
# H is their block, b its coupling to the rest.

def _eig_inputs(k, seed):
    rng = np.random.default_rng(seed)
    h = np.diag(rng.uniform(-100.0, -95.0, size=k))
    off = np.triu(rng.normal(0.0, 0.05, size=(k, k)) * (rng.random((k, k)) < 0.2), 1)
    h = h + off + off.T
    b = rng.normal(0.0, 0.05, size=k)
    x = rng.normal(0.0, 0.01, size=k) * (rng.random(k) < 0.7)
    y1, e0 = 10.2, -105.0
    z = h @ x + b * y1
    xx = y1 * y1 + float(x @ x)
    xz = y1 * y1 * e0 + 2.0 * y1 * float(b @ x) + float(x @ h @ x)
    return h, x, z, (xx, 0.0), (xz, 0.0)


def _eig_exact(k, seed):
    """The lowest eigenpair (lam, v) of the bordered matrix, by LAPACK in 64
    bits, gives gamma = v0 / y1, scale = gamma sqrt(-lam), xx = -lam / scale^2
    and dx = v / gamma - x."""
    h, x, z, (xx, _), (xz, _) = _eig_inputs(k, seed)
    hx = h @ x
    yy = xx - x @ x
    y1 = math.sqrt(yy)
    big = np.zeros((k + 1, k + 1))
    big[0, 0] = (xz - 2.0 * (x @ z) + x @ hx) / yy
    big[0, 1:] = big[1:, 0] = (z - hx) / y1
    big[1:, 1:] = h
    lam, v = np.linalg.eigh(big)
    v = v[:, 0] * (1.0 if v[0, 0] >= 0 else -1.0)
    lam = float(v @ big @ v)
    gamma = v[0] / y1
    scale = gamma * math.sqrt(-lam)
    return {"dx": v[1:] / gamma - x, "xx": np.float64(-lam / scale**2), "scale": np.float64(scale), "branch": 1}


def _dense_energy(case, seed):
    """Lowest eigenvalue of the Hamiltonian in the whole sector, assembled
    from one- and two-body operators on occupation strings."""
    n, na, nb = case["norb"], case["na"], case["nb"]
    _, h1, eri, ecore = synth.make_integrals(_spec(n, na, nb), seed)
    import itertools

    def strings(k):
        return [sum(1 << p for p in c) for c in itertools.combinations(range(n), k)]

    def singles(strs):  # E[p, q] = a+_p a_q as matrices over the strings
        index = {s: i for i, s in enumerate(strs)}
        e = np.zeros((n, n, len(strs), len(strs)))
        for s, i in index.items():
            for q in range(n):
                if not (s >> q) & 1:
                    continue
                s1, sign = s ^ (1 << q), (-1) ** bin(s & ((1 << q) - 1)).count("1")
                for p in range(n):
                    if (s1 >> p) & 1:
                        continue
                    e[p, q, index[s1 | (1 << p)], i] = sign * (-1) ** bin(s1 & ((1 << p) - 1)).count("1")
        return e

    ea, eb = singles(strings(na)), singles(strings(nb))
    # H = sum (h_pq - 1/2 sum_r (pr|rq)) E_pq + 1/2 sum (pq|rs) E_pq E_rs, E = E_a + E_b
    h = h1 - 0.5 * np.einsum("prrq->pq", eri)

    def one_spin(e):
        m = np.einsum("pq,pqij->ij", h, e)
        g = np.einsum("pqrs,rsij->pqij", eri, e, optimize=True)
        return m + 0.5 * np.einsum("pqik,pqkj->ij", e, g, optimize=True)

    ia, ib = np.eye(ea.shape[-1]), np.eye(eb.shape[-1])
    big = np.kron(one_spin(ea), ib) + np.kron(ia, one_spin(eb))
    w = np.einsum("pqrs,pqij->rsij", eri, ea, optimize=True)
    big += np.einsum("rsij,rskl->ikjl", w, eb, optimize=True).reshape(big.shape)
    return float(np.linalg.eigvalsh(big)[0]) + ecore


def exact(case, seed):
    if case["kind"] == "eig":
        return _eig_exact(case["k"], seed)
    # A solve's reports after a fixed number of iterations follow its own
    # trajectory; where it picks every determinant many times over, the last
    # energy is the sector's lowest eigenvalue.
    if case["kind"] in ("solve", "point"):
        dets = math.comb(case["norb"], case["na"]) * math.comb(case["norb"], case["nb"])
        if dets <= 900 and case["k"] * case["iterations"] >= 6 * dets and case.get("zt", 0.0) == 0.0:
            return {"energy": None, "scale": None, "final": np.float64(_dense_energy(case, seed))}
    return None


def work(case):
    kind = case["kind"]
    if kind == "eig":
        n = case["k"] + 1
        return {"bytes": 8.0 * (n * n + 4 * n), "flops": 4.0 / 3.0 * n**3}
    e = entries(case["norb"], case["na"], case["nb"])
    if kind in ("solve", "point", "batch"):
        columns = case["iterations"] * case["k"] * case.get("points", 1)
        return {"bytes": float(ENTRY_BYTES * columns * e), "flops": 0.0}
    slots = 2 ** math.ceil(math.log2(case["max_memory"] * 2**30 / (8 * (1 + (2 * case["norb"] - 1) // 64) + 16)) - 1)
    x = case["iterations"] * case["k"]  # at most so many determinants carry a coefficient
    if kind == "coefs":
        return {"bytes": float(SLOT_BYTES * slots + 24 * x), "flops": 0.0}
    # The residual reads the table once; the RDMs look up every connected determinant.
    return {"bytes": float(SLOT_BYTES * slots + 24 * x * e), "flops": 0.0}
