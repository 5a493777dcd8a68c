"""Measured cases of the KKT solve path.

Each case is a call that a program using this package makes in earnest:

* ``solve``  one KKT system solved by a plan that the program keeps for its
  sparsity (an interior-point step): values on the device (the caller's
  derivatives live there) or on the host (the drop-in's form);
* ``batch``  several plans of one sparsity solving at once, one stream each;
* ``chol``   the Cholesky component: one factorization and a few solves;
* ``ruiz``   the Ruiz equilibration component on device arrays.

The systems are synthetic power grids of the shape that the benchmark and the
tests use (buses, 0.2 generators and 1.4 branches per bus; H the branch-weighted
Laplacian plus generator costs plus a log-uniform barrier diagonal; two balance
rows per bus in Jc, two limit rows per branch in Jd; log-uniform Ds), generated
here from the seed alone: another seed draws another grid and other values.

Solves run with refinement on the full KKT system, so that a solution is
determined by the inputs down to the last digits and not by where the conjugate
gradient happens to stop.
"""
import math
import os

# plans that solve at once run on streams of their own; more hardware queues
# than the default 8 keep them from waiting behind one another
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np
import torch

import hykkt_gb300 as hk
from hykkt_gb300 import gridgen as gg

#: (gamma, range of the barrier diagonal D_x, range of D_s)
VALUES = {
    # well into the feasible region: few CG iterations, the factorization counts
    "mild": (1e4, (1e-4, 1e4), (1e-4, 1e4)),
    # the single-solve benchmark's ranges
    "wide": (1e4, (1e-8, 1e4), (1e-8, 1e8)),
    # the benchmark sequence's ranges, late interior-point iterations
    "late": (1e5, (1e-10, 1e8), (1e-10, 1e8)),
}


def listed():
    return [
        # the smallest call: a 200-bus system (the smoke test's size and ranges)
        {"name": "grid200", "kind": "solve", "n_bus": 200, "values": "mild", "where": "device", "ineq": True, "piece": 0},
        # the benchmark's single solve
        {"name": "grid500", "kind": "solve", "n_bus": 500, "values": "wide", "where": "device", "ineq": True, "piece": 0},
        # a served client: host arrays in, host arrays out
        {"name": "grid1000_host", "kind": "solve", "n_bus": 1000, "values": "wide", "where": "host", "ineq": True, "piece": 0},
        # odd size, no inequality block (Jd and Ds empty)
        {"name": "grid1777_eq", "kind": "solve", "n_bus": 1777, "values": "wide", "where": "device", "ineq": False, "piece": 0},
        # the size of the larger fixture
        {"name": "grid2000", "kind": "solve", "n_bus": 2000, "values": "mild", "where": "device", "ineq": True, "piece": 0},
        # a mid-sized served client
        {"name": "grid5000_host", "kind": "solve", "n_bus": 5000, "values": "wide", "where": "host", "ineq": True, "piece": 0},
        # the headline benchmark's system, one plan alone
        {"name": "grid10k", "kind": "solve", "n_bus": 10000, "values": "late", "where": "device", "ineq": True, "piece": 0},
        # the largest: few CG iterations, bound by the factorization
        {"name": "grid14k", "kind": "solve", "n_bus": 14000, "values": "mild", "where": "device", "ineq": True, "piece": 0},
        # plans solving at once, wide supernodes cut into pieces as the batched benchmark does
        {"name": "batch8_5000", "kind": "batch", "n_bus": 5000, "plans": 8, "values": "wide", "piece": 2048},
        # the Cholesky component on a dense 2,600-column matrix, the widest that the tests factor
        {"name": "chol_dense2600", "kind": "chol", "n": 2600, "border": 2600, "block": 0, "solves": 2},
        # ... and on 40 blocks of 50 columns coupled to a dense border of 1,200
        {"name": "chol_arrow3200", "kind": "chol", "n": 3200, "border": 1200, "block": 50, "solves": 2},
        # the equilibration component on the benchmark's system
        {"name": "ruiz10k", "kind": "ruiz", "n_bus": 10000, "sweeps": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.7:
        values = rng.choice(["mild", "mild", "wide", "late"])
        n_bus = _log_int(rng, 200, 12000 if values == "mild" else 8000)
        return {"kind": "solve", "n_bus": n_bus, "values": values, "where": rng.choice(["device", "host"]),
                "ineq": rng.random() < 0.8, "piece": rng.choice([0, 0, 0, 1024]) if n_bus > 2000 else 0}
    if pick < 0.8:
        return {"kind": "batch", "n_bus": _log_int(rng, 500, 4000), "plans": rng.randint(2, 8),
                "values": rng.choice(["mild", "wide"]), "piece": rng.choice([0, 1024])}
    if pick < 0.9:
        block = rng.choice([0, 20, 50, 90])
        border = _log_int(rng, 200, 2500)
        n = border + (block * rng.randint(2, 20) if block else 0)
        return {"kind": "chol", "n": n, "border": border, "block": block, "solves": rng.randint(1, 4)}
    return {"kind": "ruiz", "n_bus": _log_int(rng, 200, 14000), "sweeps": rng.randint(1, 4)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _csr(n, rows, cols, vals):
    """(rowptr, colidx, vals) with sorted columns; duplicates are summed."""
    m = int(cols.max(initial=0)) + 1
    key, inv = np.unique(rows * m + cols, return_inverse=True)
    v = np.bincount(inv, weights=vals, minlength=key.size)
    rp = np.concatenate([[0], np.cumsum(np.bincount(key // m, minlength=n))])
    return rp.astype(np.int32), (key % m).astype(np.int32), v


def _grid(n_bus, seed, values, ineq=True):
    """The blocks of one system: {"H", "Jc", "Jd": (rowptr, colidx, vals), "ds", "rx", "rs", "ry", "ryd"}."""
    gamma, dxr, dsr = VALUES[values]
    rng = np.random.default_rng([seed, n_bus])
    n_gen, n_br = int(round(0.2 * n_bus)), int(round(1.4 * n_bus))
    # random recursive spanning tree and random chords, no parallel branches
    child = np.arange(1, n_bus)
    tree = np.stack([(rng.random(n_bus - 1) * child).astype(np.int64), child], 1)
    more = np.sort(rng.integers(0, n_bus, (3 * n_br, 2)), 1)
    more = more[more[:, 0] != more[:, 1]]
    both = np.concatenate([tree, more])
    _, at = np.unique(both[:, 0] * n_bus + both[:, 1], return_index=True)
    br = both[np.sort(at)][:n_br]
    a, b = br[:, 0], br[:, 1]
    gen_bus = rng.integers(0, n_bus, n_gen)
    n_x = 2 * n_bus + 2 * n_gen
    w, rho = rng.uniform(0.1, 10.0, len(br)), rng.uniform(-0.9, 0.9, len(br))
    rows, cols, vals = [], [], []
    for p, q in ((0, 0), (1, 1), (0, 1), (1, 0)):
        c = w if p == q else w * rho
        rows += [2 * a + p, 2 * b + p, 2 * a + p, 2 * b + p]
        cols += [2 * a + q, 2 * b + q, 2 * b + q, 2 * a + q]
        vals += [c, c, -c, -c]
    diag = np.arange(n_x)
    gens = np.arange(2 * n_bus, n_x)
    dx = np.exp(rng.uniform(math.log(dxr[0]), math.log(dxr[1]), n_x))
    H = _csr(n_x, np.concatenate(rows + [gens, diag]), np.concatenate(cols + [gens, diag]),
             np.concatenate(vals + [rng.uniform(0.1, 10.0, gens.size), dx]))
    # Jc: rows (P, Q) of each bus touch Vm, Va of the bus and its neighbours and its generators' Pg or Qg
    at_bus, nbr = np.concatenate([np.arange(n_bus), a, b]), np.concatenate([np.arange(n_bus), b, a])
    g = np.arange(n_gen)
    rows = [2 * at_bus + pq for pq in (0, 1) for _ in (0, 1)] + [2 * gen_bus + pq for pq in (0, 1)]
    cols = [2 * nbr + v for _ in (0, 1) for v in (0, 1)] + [2 * n_bus + 2 * g + pq for pq in (0, 1)]
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    Jc = _csr(2 * n_bus, rows, cols, rng.standard_normal(rows.size))
    if ineq:  # Jd: two limit rows per branch on the endpoints' Vm, Va
        e = np.arange(len(br))
        rows = np.concatenate([2 * e + s for s in (0, 1) for _ in range(4)])
        cols = np.concatenate([2 * x + v for _ in (0, 1) for x in (a, b) for v in (0, 1)])
        Jd = _csr(2 * len(br), rows, cols, rng.standard_normal(rows.size))
    else:
        Jd = (np.zeros(1, np.int32), np.zeros(0, np.int32), np.zeros(0))
    m_d, m_c = len(Jd[0]) - 1, 2 * n_bus
    ds = np.exp(rng.uniform(math.log(dsr[0]), math.log(dsr[1]), m_d))
    rhs = {k: rng.uniform(-1, 1, n) for k, n in (("rx", n_x), ("rs", m_d), ("ry", m_c), ("ryd", m_d))}
    return {"H": H, "Jc": Jc, "Jd": Jd, "ds": ds, "gamma": gamma, **rhs}


def _system(g, device):
    """The package's view of the blocks, values as numpy arrays or device tensors."""
    n_x, m_c, m_d = len(g["H"][0]) - 1, len(g["Jc"][0]) - 1, len(g["ds"])
    put = (lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda")) if device else (lambda v: v)
    i = np.arange(m_d + 1, dtype=np.int32)
    blocks = [gg.CSR(n, m, rp, ci, put(v)) for n, m, (rp, ci, v) in (
        (n_x, n_x, g["H"]), (m_d, m_d, (i, i[:-1], g["ds"])), (m_c, n_x, g["Jc"]), (m_d, n_x, g["Jd"]))]
    return gg.KKTSystem(*blocks, *[put(g[k]) for k in ("rx", "rs", "ry", "ryd")], g["gamma"])


def _plan(s, piece):
    p = hk.Plan(s, solve_piece=piece)
    p.set_accuracy(cg_itmax=5000, cg_rtol=1e-11, refine_max=4, refine_target=1e-12)
    p.set_refine_rtol(1e-4)
    return p


def _outputs(p):
    return [torch.empty(n, dtype=torch.float64, device="cuda") for n in (p.n_x, p.m_d, p.m_c, p.m_d)]


def _spd(case, seed):
    """The Cholesky cases' matrix (dense, on the device) and right-hand sides: `block`-column diagonal blocks
    coupled to a dense border."""
    n, border, block = case["n"], case["border"], case["block"]
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + n)

    def uniform(*shape):
        return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1

    A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    at = n - border
    for k in range(0, at, block or n):
        G = uniform(block, block)
        A[k:k + block, k:k + block] = G @ G.T / block + torch.eye(block, dtype=torch.float64, device="cuda")
    if at:
        A[at:, :at] = uniform(border, at) * 0.02
    G = uniform(border, border)
    A[at:, at:] = G @ G.T / border + 4 * torch.eye(border, dtype=torch.float64, device="cuda")
    low = torch.tril(A)
    return low + torch.tril(A, -1).T, uniform(case["solves"], n)


def prepare(case, seed):
    if case["kind"] == "chol":
        A, b = _spd(case, seed)
        A, b = A.cpu().numpy(), b.cpu().numpy()
        r, c = np.nonzero(np.tril(A))
        rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=len(A)))]).astype(np.int32)
        ch = hk.Chol(len(A), rp, c.astype(np.int32), ordering=hk.ORDER_IDENTITY)
        return {"case": case, "chol": ch, "vals": np.ascontiguousarray(A[r, c]), "b": list(b)}
    if case["kind"] == "ruiz":
        g = _grid(case["n_bus"], seed, "wide", ineq=False)
        n, m = len(g["H"][0]) - 1, len(g["Jc"][0]) - 1
        rows = np.repeat(np.arange(m), np.diff(g["Jc"][0]))
        Jt = _csr(n, g["Jc"][1].astype(np.int64), rows, g["Jc"][2])
        dev = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
        mats = [[dev(x) for x in (M[2], M[0], M[1])] for M in (g["H"], Jt, g["Jc"])]
        return {"case": case, "n": n, "m": m, "mats": mats, "rhs": [dev(g["rx"]), dev(g["ry"])],
                "max_d": torch.zeros(n + m, dtype=torch.float64, device="cuda")}
    if case["kind"] == "batch":
        ss = [_system(_grid_of(case, seed, i), True) for i in range(case["plans"])]
        first = _plan(ss[0], case["piece"])
        plans = [first] + [first.clone() for _ in ss[1:]]
        for p in plans:
            p.set_concurrency(len(plans))
        return {"case": case, "plans": plans, "systems": ss, "streams": [torch.cuda.Stream() for _ in ss],
                "out": [_outputs(p) for p in plans]}
    device = case["where"] == "device"
    s = _system(_grid_of(case, seed), device)
    p = _plan(s, case["piece"])
    return {"case": case, "plan": p, "system": s, "out": _outputs(p) if device else None}


def _grid_of(case, seed, i=0):
    """System i of a case: one grid, new barrier values and right-hand sides for each i."""
    g = _grid(case["n_bus"], seed, case["values"], case.get("ineq", True))
    if i:
        _, dxr, dsr = VALUES[case["values"]]
        rng = np.random.default_rng([seed, case["n_bus"], i])
        rp, ci, v = g["H"]
        on = np.repeat(np.arange(len(rp) - 1), np.diff(rp)) == ci
        v = v.copy()
        v[on] += np.exp(rng.uniform(math.log(dxr[0]), math.log(dxr[1]), int(on.sum())))
        g["H"] = (rp, ci, v)
        g["ds"] = np.exp(rng.uniform(math.log(dsr[0]), math.log(dsr[1]), len(g["ds"])))
        for k in ("rx", "rs", "ry", "ryd"):
            g[k] = rng.uniform(-1, 1, len(g[k]))
    return g


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _fetch(p, out, stream):
    rc = hk.lib().hykkt_plan_get_solution(p.h, *[t.data_ptr() for t in out], 1, stream)
    if rc != hk.OK:
        raise RuntimeError(hk.lib().hykkt_last_error().decode())
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "chol":
        c = state["chol"]
        if c.factor(state["vals"]) != hk.OK:
            raise RuntimeError("not positive definite")
        return [c.solve(b) for b in state["b"]]
    if kind == "ruiz":
        (hv, hi, hj), (tv, ti, tj), (jv, ji, jj) = state["mats"]
        arrays = (hv, hi, hj, tv, ti, tj, jv, ji, jj, *state["rhs"], state["max_d"])
        rc = hk.lib().hykkt_ruiz_scale(state["case"]["sweeps"], state["n"], state["m"],
                                       *[t.data_ptr() for t in arrays], None)
        if rc != hk.OK:
            raise RuntimeError(hk.lib().hykkt_last_error().decode())
        return [hv, tv, jv, *state["rhs"], state["max_d"]]
    if kind == "batch":
        ps, sts = state["plans"], [s.cuda_stream for s in state["streams"]]
        for p, s, st in zip(ps, state["systems"], sts):
            p.solve(s, on_device=True, stream=st, sync=False)
        for p, st in zip(ps, sts):
            p.wait(st)
        return [_fetch(p, out, st) for p, out, st in zip(ps, state["out"], sts)]
    p = state["plan"]
    if state["out"] is None:
        p.solve(state["system"])
        return list(p.solution())
    p.solve(state["system"], on_device=True)
    return _fetch(p, state["out"], None)


def work(case):
    """Inputs read once, outputs written once, and the operations of a dense factorization where the
    matrix is dense; the operations of a sparse one depend on the ordering and are left out."""
    if case["kind"] == "chol":
        n, border, block = case["n"], case["border"], case["block"]
        at = n - border
        stored = border * (border + 1) / 2 + at * border + at * (block + 1) / 2
        flops = border ** 3 / 3 + at * border ** 2 + at * block * border + at * block ** 2 / 3
        return {"bytes": 8 * (stored + 2 * n * case["solves"]), "flops": flops + 4 * stored * case["solves"]}
    nb = case["n_bus"]
    n_x, m_c, m_d = 2.4 * nb, 2 * nb, 2.8 * nb if case.get("ineq", True) else 0
    nnz = 15.6 * nb + 15.6 * nb + 4 * m_d  # H, Jc, Jd
    if case["kind"] == "ruiz":
        vals = 3 * 15.6 * nb
        return {"bytes": (16 + 4) * vals + 8 * 4 * (n_x + m_c), "flops": 3 * case["sweeps"] * vals}
    one = 8 * (nnz + m_d + n_x + 2 * m_d + m_c + n_x + 2 * m_d + m_c)
    return {"bytes": one * case.get("plans", 1), "flops": 4 * nnz * case.get("plans", 1)}


# ---------------------------------------------------------------------------
# 64-bit answers
# ---------------------------------------------------------------------------
def _kkt_solution(g):
    """[x, s, y, yd] of the 4-block system: dense LU of the condensed matrix, then corrections whose residuals
    are accumulated in extended precision."""
    n_x, m_c, m_d = len(g["H"][0]) - 1, len(g["Jc"][0]) - 1, len(g["ds"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def coo(M):
        return np.repeat(np.arange(len(M[0]) - 1), np.diff(M[0])), M[1].astype(np.int64), M[2]

    H, Jc, Jd = coo(g["H"]), coo(g["Jc"]), coo(g["Jd"])
    K = torch.zeros(n_x + m_c, n_x + m_c, dtype=torch.float64, device=dev)

    def add(r, c, v):
        K.index_put_((torch.as_tensor(r, device=dev), torch.as_tensor(c, device=dev)),
                     torch.as_tensor(v, device=dev), accumulate=True)

    add(*H)
    add(Jc[0] + n_x, Jc[1], Jc[2])
    add(Jc[1], Jc[0] + n_x, Jc[2])
    if m_d:  # Jd^T Ds Jd, four entries per row
        c, v = Jd[1].reshape(m_d, 4), Jd[2].reshape(m_d, 4)
        for i in range(4):
            for j in range(4):
                add(c[:, i], c[:, j], v[:, i] * v[:, j] * g["ds"])
    d = 1.0 / torch.sqrt(K.abs().amax(1))  # symmetric scaling
    K.mul_(d[:, None]).mul_(d[None, :])
    lu, piv = torch.linalg.lu_factor(K)
    del K
    L = np.longdouble

    def times(M, v, rows, transpose=False):
        r, c = (M[1], M[0]) if transpose else (M[0], M[1])
        out = np.zeros(rows, L)
        np.add.at(out, r, M[2].astype(L) * v[c])
        return out

    x, s, y, yd = np.zeros(n_x, L), np.zeros(m_d, L), np.zeros(m_c, L), np.zeros(m_d, L)
    ds = g["ds"].astype(L)
    for _ in range(6):
        r1 = g["rx"] - times(H, x, n_x) - times(Jc, y, n_x, True) - times(Jd, yd, n_x, True)
        r2 = g["rs"] - (ds * s - yd)
        r3 = g["ry"] - times(Jc, x, m_c)
        r4 = g["ryd"] - (times(Jd, x, m_d) - s)
        top = r1 + times(Jd, ds * r4 + r2, n_x, True)
        b = torch.as_tensor(np.concatenate([top, r3]).astype(np.float64), device=dev) * d
        z = (torch.linalg.lu_solve(lu, piv, b[:, None])[:, 0] * d).cpu().numpy()
        dx = z[:n_x].astype(L)
        dsl = times(Jd, dx, m_d) - r4
        x, y, s, yd = x + dx, y + z[n_x:], s + dsl, yd + (ds * dsl - r2)
    return [v.astype(np.float64) for v in (x, s, y, yd)]


def exact(case, seed):
    if case["kind"] == "chol":
        A, b = _spd(case, seed)
        C = torch.linalg.cholesky(A)
        out = []
        for v in b:
            x = torch.cholesky_solve(v[:, None], C)
            for _ in range(2):
                x = x + torch.cholesky_solve(v[:, None] - A @ x, C)
            out.append(x[:, 0].cpu().numpy())
        return out
    if case["kind"] == "ruiz":
        g = _grid(case["n_bus"], seed, "wide", ineq=False)
        n, m = len(g["H"][0]) - 1, len(g["Jc"][0]) - 1
        hr, hc, hv = np.repeat(np.arange(n), np.diff(g["H"][0])), g["H"][1], g["H"][2].copy()
        jr, jc, jv = np.repeat(np.arange(m), np.diff(g["Jc"][0])), g["Jc"][1], g["Jc"][2].copy()
        rx, ry, max_d = g["rx"].copy(), g["ry"].copy(), np.ones(n + m)
        for _ in range(case["sweeps"]):
            top = np.zeros(n + m)
            np.maximum.at(top, hr, np.abs(hv))
            np.maximum.at(top, jc, np.abs(jv))
            np.maximum.at(top, n + jr, np.abs(jv))
            d = 1.0 / np.sqrt(top)
            hv, jv = hv * (d[hr] * d[hc]), jv * (d[n + jr] * d[jc])
            rx, ry, max_d = rx * d[:n], ry * d[n:], max_d * d
        order = np.lexsort((jr, jc))
        return [hv, jv[order], jv, rx, ry, max_d]
    if case["n_bus"] > 5000:
        return None
    first = _kkt_solution(_grid_of(case, seed))
    return [first] + [[None] * 4] * (case["plans"] - 1) if case["kind"] == "batch" else first
