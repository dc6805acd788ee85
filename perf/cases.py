"""What a program that uses this framework has it do, as cases that can be timed.

A case is a dict of plain values with a "kind":

  spmv     one product y = A x through an autotuning-free plan (ispm.spmv_plan)
  refresh  new values of A with the same pattern into the plan, then y = A x
  ppcg     the scalar and vector updates of one pipelined-CG iteration (sblas)
  dot      one inner product (sblas)
  solve    one whole preconditioned solve (ispm.PCGSolver)
  step     one time step: new values of A into the solver, then its solve
  batch    many systems of uneven size solved together (ispm.BatchSolver)
  train    one training step of the drop-tolerance network (ispm.learn.MLP)
  predict  row features of a matrix and the network's prediction for each row

Matrices are the benchmark's families: 7- and 27-point box stencils with
log-normal coefficients, and the 7-point face graph with 5% of its faces
removed under a random numbering.  Their diagonal is 1.05 (solves: an
implicit step's dominance) or 1.01 times the row sum.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "ispm-sparse-lib_b200"))

import ispm  # noqa: E402
import ispm.learn as learn  # noqa: E402

DEV = torch.device("cuda")
NP = {"f32": np.float32, "f64": np.float64}
TT = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # a coarse level or a small block: launch latency is what it costs
        {"name": "spmv_7pt_f64_16", "kind": "spmv", "matrix": "box", "points": 7,
         "nz": 16, "ny": 16, "nx": 16, "T": "f64", "E": "f64"},
        # the headline system's product in the solver's inner precision
        {"name": "spmv_27pt_f32_128", "kind": "spmv", "matrix": "box", "points": 27,
         "nz": 128, "ny": 128, "nx": 128, "T": "f32", "E": "f32"},
        # an unstructured mesh in the order its generator left it, FP32
        # coefficients and FP64 vectors
        {"name": "spmv_graph_f64f32_90", "kind": "spmv", "matrix": "graph", "points": 7,
         "nz": 90, "ny": 90, "nx": 90, "T": "f64", "E": "f32"},
        # a time step's matrix update on an odd, uneven box, then its product
        {"name": "refresh_27pt_f64_75", "kind": "refresh", "matrix": "box", "points": 27,
         "nz": 61, "ny": 75, "nx": 83, "T": "f64", "E": "f64"},
        # vector updates of a caller's own pipelined CG: a small system, odd length
        {"name": "ppcg_f64_35937", "kind": "ppcg", "n": 35937, "T": "f64"},
        # the same for a large one
        {"name": "ppcg_f32_2000003", "kind": "ppcg", "n": 2000003, "T": "f32"},
        # residual norm / monitoring of the largest benchmark system's vectors
        {"name": "dot_f64_7077888", "kind": "dot", "n": 7077888, "T": "f64"},
        # the small end of the solves: plain FP64 pipelined CG, right-hand side on the device
        {"name": "solve_7pt_f64_24", "kind": "solve", "matrix": "box", "points": 7,
         "nz": 24, "ny": 24, "nx": 24, "inner": "f64"},
        # a time-stepping caller: new coefficients, factor rebuilt on the GPU,
        # mixed-precision solve
        {"name": "step_27pt_mixed_72", "kind": "step", "matrix": "box", "points": 27,
         "nz": 72, "ny": 72, "nx": 72, "inner": "f32"},
        # the U/V/W/p solves of one time step: uneven boxes, 1-4 right-hand sides
        {"name": "batch_mixed_16", "kind": "batch", "systems": 16, "lo": 12, "hi": 40,
         "inner": "f32"},
        # the training loop's minibatch
        {"name": "train_65536", "kind": "train", "n": 65536},
        # drop tolerances of every row of a matrix assembled on the device
        {"name": "predict_27pt_80", "kind": "predict", "points": 27, "nz": 80, "ny": 80,
         "nx": 80},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """Sides near one another around a log-uniform length, odd ones among them."""
    s = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return {k: min(hi, max(lo, int(round(s * rng.uniform(0.85, 1.15))))) for k in ("nz", "ny", "nx")}


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "refresh", "ppcg", "dot", "solve", "step", "batch",
                       "train", "predict"])
    c = {"kind": kind}
    if kind == "spmv":
        c["T"], c["E"] = rng.choice([("f32", "f32"), ("f64", "f32"), ("f64", "f64")])
        if rng.random() < 0.3:
            c.update(matrix="graph", points=7, **_box(rng, 16, 90))
        else:
            c.update(matrix="box", points=rng.choice([7, 27]),
                     **_box(rng, 16, 128 if c["E"] == "f32" else 96))
    elif kind == "refresh":
        c["T"], c["E"] = rng.choice([("f32", "f32"), ("f64", "f32"), ("f64", "f64")])
        c.update(matrix="box", points=rng.choice([7, 27]), **_box(rng, 16, 80))
    elif kind in ("ppcg", "dot"):
        c.update(n=_log_int(rng, 4000, 7000000 if kind == "dot" else 4000000),
                 T=rng.choice(["f32", "f64"]))
    elif kind in ("solve", "step"):
        c["inner"] = rng.choice(["f32", "f64"])
        if rng.random() < 0.25:
            c.update(matrix="graph", points=7, **_box(rng, 20, 48))
        else:
            c.update(matrix="box", points=rng.choice([7, 27]), **_box(rng, 16, 72))
    elif kind == "batch":
        c.update(systems=rng.randint(3, 16), lo=12, hi=rng.randint(16, 40), inner="f32")
    elif kind == "train":
        c["n"] = _log_int(rng, 2000, 300000)
    else:
        c.update(points=rng.choice([7, 27]), **_box(rng, 16, 80))
    return c


# ---------------------------------------------------------------- inputs

def _box_csr(nz, ny, nx, points, seed, diag=1.01, sigma=1.0):
    """(row_ptr, cols, vals) on the GPU: coupling exp((c_i + c_j) / 2) / d^2 of
    the box stencil's neighbours, c ~ N(0, sigma^2) per cell, the diagonal
    `diag` times the row sum."""
    n = nz * ny * nx
    cell = torch.from_numpy(np.random.default_rng(seed).standard_normal(n) * sigma).to(DEV)
    i = torch.arange(n, device=DEV)
    z, y, x = i // (ny * nx), (i // nx) % ny, i % nx
    offs = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)
            if points == 27 or abs(a) + abs(b) + abs(c) < 2]
    cols = torch.empty((n, len(offs)), dtype=torch.int32, device=DEV)
    vals = torch.zeros((n, len(offs)), dtype=torch.float64, device=DEV)
    ok = torch.empty((n, len(offs)), dtype=torch.bool, device=DEV)
    for k, (a, b, c) in enumerate(offs):
        ok[:, k] = ((z + a >= 0) & (z + a < nz) & (y + b >= 0) & (y + b < ny) & (x + c >= 0) &
                    (x + c < nx))
        j = torch.where(ok[:, k], i + (a * ny + b) * nx + c, i)
        cols[:, k] = j.to(torch.int32)
        d2 = a * a + b * b + c * c
        if d2:
            vals[:, k] = torch.where(ok[:, k], -torch.exp(0.5 * (cell + cell[j])) / d2, 0.0)
    vals[:, len(offs) // 2] = -diag * vals.sum(1)
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(ok.sum(1), 0)
    return rp.to(torch.int32), cols[ok], vals[ok]


def _graph_csr(nz, ny, nx, seed, diag=1.01):
    """The 7-point face graph with 5% of its faces removed, weights U(0.1, 10),
    under a random numbering.  The mesh (faces, numbering) is fixed by its
    sides; the seed gives the weights."""
    n = nz * ny * nx
    mesh = np.random.default_rng([nz, ny, nx])
    i = torch.arange(n, device=DEV)
    z, y, x = i // (ny * nx), (i // nx) % ny, i % nx
    p = torch.cat([i[x + 1 < nx], i[y + 1 < ny], i[z + 1 < nz]])
    q = torch.cat([i[x + 1 < nx] + 1, i[y + 1 < ny] + nx, i[z + 1 < nz] + ny * nx])
    keep = torch.from_numpy(mesh.random(p.numel()) >= 0.05).to(DEV)
    perm = torch.from_numpy(mesh.permutation(n)).to(DEV)
    p, q = perm[p[keep]], perm[q[keep]]
    w = torch.from_numpy(np.random.default_rng(seed).uniform(0.1, 10.0, p.numel())).to(DEV)
    rows, cols = torch.cat([p, q, i]), torch.cat([q, p, i])
    order = torch.argsort(rows * n + cols)
    rows, cols = rows[order], cols[order]
    vals = torch.cat([-w, -w, torch.zeros(n, dtype=torch.float64, device=DEV)])[order]
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    # row sums in entry order (no atomics: the same bits every time)
    width = int((rp[1:] - rp[:-1]).max())
    at = rp[:-1, None] + torch.arange(width, device=DEV)[None, :]
    total = torch.where(at < rp[1:, None], vals[at.clamp(max=vals.numel() - 1)], 0.0).sum(1)
    vals[rows == cols] = torch.where(total < 0, -diag * total, 1.0)
    return rp.to(torch.int32), cols.to(torch.int32), vals


def _csr(c, seed, diag=1.01):
    if c.get("matrix") == "graph":
        return _graph_csr(c["nz"], c["ny"], c["nx"], seed, diag)
    return _box_csr(c["nz"], c["ny"], c["nx"], c["points"], seed, diag)


def _host(rp, cols, vals):
    """The host CSR that plans and solvers are made from."""
    n = rp.numel() - 1
    return ispm.csr_matrix(n, n, rp.cpu().numpy(), cols.cpu().numpy(), vals.cpu().numpy())


def _uniform(seed, n, dtype):
    v = np.random.default_rng([seed, 7]).uniform(-1.0, 1.0, n)
    return torch.from_numpy(v).to(DEV).to(dtype)


def _padded(n):
    return (n + 511) // 512 * 512


def _product(rp, cols, vals, x):
    """A x in 64 bits, over the padded rows."""
    n = rp.numel() - 1
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (rp[1:] - rp[:-1]).long())
    y = torch.zeros(_padded(n), dtype=torch.float64, device=DEV)
    return y.index_add_(0, rows, vals.double() * x.double()[cols.long()])


# an implicit step's diagonal dominance and a tolerance near round-off: the
# solution is then the same to many digits however its iterations round
SOLVE_DIAG, SOLVE_TOL = 1.05, 1e-12


def _rhs(rp, cols, vals, seed):
    """(b, x_true), b = A x_true over the padded rows (products summed in entry order)."""
    n = rp.numel() - 1
    x = torch.zeros(_padded(n), dtype=torch.float64, device=DEV)
    x[:n] = _uniform(seed, n, torch.float64)
    prod = vals * x[cols.long()]
    width = int((rp[1:] - rp[:-1]).max())
    b = torch.zeros_like(x)
    lo, hi = rp[:-1].long(), rp[1:].long()
    for k in range(width):
        b[:n] += torch.where(lo + k < hi, prod[(lo + k).clamp(max=prod.numel() - 1)], 0.0)
    return b, x


def _batch_systems(c, seed):
    """Box stencils (60% 7-point) with sides lo..hi and 1-4 right-hand sides; the
    shapes are fixed by the case, the coefficients by the seed."""
    shape = np.random.default_rng([c["systems"], c["lo"], c["hi"]])
    out = []
    for k in range(c["systems"]):
        nz, ny, nx = (int(v) for v in shape.integers(c["lo"], c["hi"] + 1, 3))
        points = 7 if shape.random() < 0.6 else 27
        rhs = int(shape.integers(1, 5))
        out.append((_box_csr(nz, ny, nx, points, seed * 1000 + k, SOLVE_DIAG), rhs))
    return out


def _lane_seed(seed, system, rhs):
    return seed * 100 + 4 * system + rhs


def _ppcg_inputs(c, seed):
    rng = np.random.default_rng([seed, 11])
    dt = TT[c["T"]]
    v = {k: torch.from_numpy(rng.uniform(-1.0, 1.0, c["n"])).to(DEV).to(dt) for k in "nmpsqzxruw"}
    # r.u and w.u of a run that converges: beta near 1/2, alpha near 3/4
    s = {"alpha": 0.75, "beta": 0.5, "gamma": 1.0, "gammaold": 2.0, "delta": 2.0}
    s = {k: torch.tensor([a * rng.uniform(0.95, 1.05)], dtype=dt, device=DEV) for k, a in s.items()}
    return v, s


def _train_inputs(c, seed):
    rng = np.random.default_rng([seed, 13])
    n = c["n"]
    # rows as ispm_row_features makes them: neighbour ratios in (0, 1), a few
    # summary columns, a constant one
    f = rng.uniform(0.0, 1.0, (n, learn.N_IN)).astype(np.float32) ** 2
    f[:, 0] = 0.3 * rng.standard_normal(n)
    f[:, 1] = rng.uniform(0.9, 1.0, n)
    f[:, 28] = 1.0
    f[:, 31] = 1.0
    t = np.stack([rng.uniform(-3.0, 3.0, n), np.zeros(n)], 1).astype(np.float32)
    w = rng.uniform(0.5, 1.5, (n, 2)).astype(np.float32)
    return (torch.from_numpy(f).to(DEV).to(torch.bfloat16), torch.from_numpy(t).to(DEV),
            torch.from_numpy(w).to(DEV), learn.init_params(seed))


def prepare(case, seed):
    c, s, kind = case, {"c": case}, case["kind"]
    if kind in ("spmv", "refresh"):
        rp, cols, vals = _csr(c, seed)
        e = TT[c["E"]]
        A = _host(rp, cols, vals.to(e))
        s["plan"] = ispm.spmv_plan(A, T=NP[c["T"]])
        s["x"] = _uniform(seed, A.n_cols, TT[c["T"]])
        s["y"] = torch.zeros(_padded(A.n_rows), dtype=TT[c["T"]], device=DEV)
        if kind == "refresh":
            s["A"], s["vals"] = A, _csr(c, seed + 500000)[2]  # assembled in FP64
    elif kind == "ppcg":
        s["v"], s["s"] = _ppcg_inputs(c, seed)
        s["out"] = torch.zeros(3, dtype=TT[c["T"]], device=DEV)
    elif kind == "dot":
        s["x"], s["y"] = (_uniform(seed + k * 77, c["n"], TT[c["T"]]) for k in (0, 1))
        s["out"] = torch.zeros(1, dtype=TT[c["T"]], device=DEV)
    elif kind in ("solve", "step"):
        m = _csr(c, seed, SOLVE_DIAG)
        s["solver"] = ispm.PCGSolver(_host(*m), inner=NP[c["inner"]], tol=SOLVE_TOL,
                                     prec="fsai_gpu", refresh=kind == "step")
        if kind == "step":
            m = _csr(c, seed + 500000, SOLVE_DIAG)
            s["vals"] = m[2]
        s["b"], _ = _rhs(*m, seed)
        s["x"] = torch.zeros_like(s["b"])
    elif kind == "batch":
        sysm = _batch_systems(c, seed)
        s["solver"] = ispm.BatchSolver([_host(*m) for m, _ in sysm], [r for _, r in sysm],
                                       inner=NP[c["inner"]], tol=SOLVE_TOL)
        s["b"] = torch.zeros(s["solver"].rows, dtype=torch.float64, device=DEV)
        s["x"] = torch.zeros_like(s["b"])
        s["lanes"] = []  # (system, right-hand side, first row, rows)
        for i in map(s["solver"].lane_info, range(s["solver"].lanes)):
            m = sysm[i["system"]][0]
            n = m[0].numel() - 1
            b, _ = _rhs(*m, _lane_seed(seed, i["system"], i["rhs"]))
            s["b"][i["row0"]:i["row0"] + n] = b[:n]
            s["lanes"].append((i["system"], i["rhs"], i["row0"], n))
        s["lanes"].sort()
    elif kind == "train":
        s["f"], s["t"], s["w"], p = _train_inputs(c, seed)
        s["mlp"] = learn.MLP(p)
    else:
        s["rp"], s["cols"], s["vals"] = _box_csr(c["nz"], c["ny"], c["nx"], c["points"], seed)
        s["n"] = s["rp"].numel() - 1
        s["f"] = torch.empty((s["n"], learn.N_IN), dtype=torch.bfloat16, device=DEV)
        s["mlp"] = learn.MLP(learn.init_params(seed))
    return s


def run(state):
    s, c = state, state["c"]
    kind = c["kind"]
    if kind in ("spmv", "refresh"):
        if kind == "refresh":
            ispm.plan_refresh_values(s["plan"], s["A"], s["vals"])
        s["plan"].execute_spmv(s["x"], s["y"])
        return s["y"]
    if kind == "ppcg":
        v, k, o = s["v"], s["s"], s["out"]
        ispm.sblas.ppcg_update_scalars(k["alpha"], k["beta"], k["gamma"], k["gammaold"],
                                       k["delta"])
        ispm.sblas.ppcg_update_vectors(o[0:1], o[1:2], o[2:3], k["alpha"], k["beta"], v["n"],
                                       v["m"], v["p"], v["s"], v["q"], v["z"], v["x"], v["r"],
                                       v["u"], v["w"], c["n"])
        return {"sums": o, "alpha": k["alpha"], "beta": k["beta"],
                **{a: v[a] for a in "psqzxruw"}}
    if kind == "dot":
        ispm.sblas.dot(s["x"], s["y"], s["out"], c["n"])
        return s["out"]
    if kind in ("solve", "step"):
        if kind == "step":
            s["solver"].update_values(s["vals"])
        s["solver"].solve(s["b"], s["x"])
        return s["x"]
    if kind == "batch":
        s["solver"].solve(s["b"], s["x"])
        return [s["x"][at:at + n] for _, _, at, n in s["lanes"]]
    if kind == "train":
        loss, grad = s["mlp"].loss_grad(s["f"], s["t"], s["w"])
        s["mlp"].adam_step(2e-3)
        # the loss is an FP32 sum, handed out as a Python float
        return {"loss": np.float32(loss), "grad": grad, "params": s["mlp"].params()}
    # the C entry point: the matrix is on the device already
    lib = ispm.lib_handle()
    if lib.ispm_row_features(s["n"], s["rp"].data_ptr(), s["cols"].data_ptr(),
                             s["vals"].data_ptr(), c["nx"], c["ny"], s["f"].data_ptr(), None):
        raise RuntimeError(lib.ispm_last_error().decode())
    return {"features": s["f"], "controls": s["mlp"].forward(s["f"])}


def _nnz(c):
    """Entries of the case's matrix (a graph's: its expectation)."""
    d = (c["nz"], c["ny"], c["nx"])
    if c["points"] == 27:
        return math.prod(3 * k - 2 for k in d)
    n = math.prod(d)
    faces = sum(n // k * (k - 1) for k in d)
    return n + int((1.9 if c.get("matrix") == "graph" else 2.0) * faces)


ITERATIONS = 24  # a solve needs at least about this many at SOLVE_DIAG and SOLVE_TOL


def work(case):
    c, kind = case, case["kind"]
    size = {"f32": 4, "f64": 8}
    if kind in ("spmv", "refresh"):
        n, nnz = c["nz"] * c["ny"] * c["nx"], _nnz(c)
        # a stencil's column indices follow from its diagonals; a graph's are read
        idx = 4 * nnz if c["matrix"] == "graph" else 0
        b = size[c["E"]] * nnz + idx + 2 * size[c["T"]] * n
        if kind == "refresh":  # values and their places in, elements out
            b += (8 + 4 + size[c["E"]]) * nnz
        return {"bytes": b, "flops": 2 * nnz}
    if kind == "ppcg":
        return {"bytes": 18 * size[c["T"]] * c["n"], "flops": 22 * c["n"]}
    if kind == "dot":
        return {"bytes": 2 * size[c["T"]] * c["n"], "flops": 2 * c["n"]}
    if kind in ("solve", "step"):
        n, nnz = c["nz"] * c["ny"] * c["nx"], _nnz(c)
        low = (nnz + n) // 2
        e = size[c["inner"]]
        # A, the factor twice (its values 16 bits in a mixed solve), eleven vector passes
        it = e * nnz + 2 * (2 if e == 4 else 8) * low + 11 * e * n
        b = ITERATIONS * it + 2 * (8 * nnz + 24 * n)
        f = ITERATIONS * (2 * nnz + 4 * low + 10 * n)
        if kind == "step":  # values into both copies of A, the factor's rows
            b += (16 + e + 8) * nnz + 24 * low
            k = 14 if c["points"] == 27 else 4
            f += n * k * k * k // 3
        return {"bytes": b, "flops": f}
    if kind == "batch":
        b = f = 0
        shape = np.random.default_rng([c["systems"], c["lo"], c["hi"]])
        for _ in range(c["systems"]):
            nz, ny, nx = (int(v) for v in shape.integers(c["lo"], c["hi"] + 1, 3))
            points = 7 if shape.random() < 0.6 else 27
            rhs = int(shape.integers(1, 5))
            n, nnz = nz * ny * nx, _nnz({"nz": nz, "ny": ny, "nx": nx, "points": points})
            low = (nnz + n) // 2
            # a system's matrices once an iteration for all its right-hand sides
            b += ITERATIONS * (4 * nnz + 8 * low + 11 * 4 * n * rhs)
            f += ITERATIONS * rhs * (2 * nnz + 4 * low + 10 * n)
        return {"bytes": b, "flops": f}
    net = 2 * (32 * 64 + 64 * 64 + 64 * 2)
    if kind == "train":
        return {"bytes": (64 + 16) * c["n"], "flops": 3 * net * c["n"]}
    n, nnz = c["nz"] * c["ny"] * c["nx"], _nnz(c)
    return {"bytes": 12 * nnz + (4 + 64 + 8) * n, "flops": net * n + 4 * nnz}


# ---------------------------------------------------------------- 64-bit answers

def _net64(p, x):
    """The network in 64 bits: (y, hidden pre-activations and activations)."""
    h, i, o = learn.N_H, learn.N_IN, learn.N_OUT
    p = torch.from_numpy(p).to(DEV).double()
    at, parts = 0, []
    for shape in ((h, i), (h,), (h, h), (h,), (o, h), (o,)):
        k = math.prod(shape)
        parts.append(p[at:at + k].reshape(shape))
        at += k
    w1, b1, w2, b2, w3, b3 = parts
    a1 = torch.relu(x @ w1.T + b1)
    a2 = torch.relu(a1 @ w2.T + b2)
    return a2 @ w3.T + b3, a1, a2, parts


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("spmv", "refresh"):
        rp, cols, vals = _csr(c, seed)
        if kind == "refresh":
            vals = _csr(c, seed + 500000)[2]
        return _product(rp, cols, vals.to(TT[c["E"]]), _uniform(seed, rp.numel() - 1, TT[c["T"]]))
    if kind == "ppcg":
        v, k = _ppcg_inputs(c, seed)
        v, k = ({a: t.double() for a, t in d.items()} for d in (v, k))
        beta = k["gamma"] / k["gammaold"]
        alpha = k["gamma"] / (k["delta"] - beta * k["gamma"] / k["alpha"])
        z, q = v["n"] + beta * v["z"], v["m"] + beta * v["q"]
        s, p = v["w"] + beta * v["s"], v["u"] + beta * v["p"]
        u, w = v["u"] - alpha * q, v["w"] - alpha * z
        r, x = v["r"] - alpha * s, v["x"] + alpha * p
        sums = torch.stack([r.abs().sum(), (r * u).sum(), (w * u).sum()])
        return {"sums": sums, "alpha": alpha, "beta": beta, "p": p, "s": s, "q": q, "z": z,
                "x": x, "r": r, "u": u, "w": w}
    if kind == "dot":
        x, y = (_uniform(seed + k * 77, c["n"], TT[c["T"]]).double() for k in (0, 1))
        return (x * y).sum().reshape(1)
    if kind in ("solve", "step"):
        m = _csr(c, seed + (500000 if kind == "step" else 0), SOLVE_DIAG)
        return _rhs(*m, seed)[1]
    if kind == "batch":
        return [_rhs(*m, _lane_seed(seed, k, r))[1][:m[0].numel() - 1]
                for k, (m, rhs) in enumerate(_batch_systems(c, seed)) for r in range(rhs)]
    if kind == "train":
        f, t, w, p = _train_inputs(c, seed)
        f, t, w = f.double(), t.double(), w.double()
        y, a1, a2, (w1, b1, w2, b2, w3, b3) = _net64(p, f)
        e = y - t
        d3 = 2.0 * w * e / c["n"]
        d2 = (d3 @ w3) * (a2 > 0)
        d1 = (d2 @ w2) * (a1 > 0)
        g = torch.cat([(d1.T @ f).ravel(), d1.sum(0), (d2.T @ a1).ravel(), d2.sum(0),
                       (d3.T @ a2).ravel(), d3.sum(0)])
        # Adam's first step moves every parameter by about the rate, whatever
        # its gradient's size: compared by the start's alone
        return {"loss": (w * e * e).sum() / c["n"], "grad": g, "params": None}
    rp, cols, vals = _box_csr(c["nz"], c["ny"], c["nx"], c["points"], seed)
    n, nx, plane = rp.numel() - 1, c["nx"], c["nx"] * c["ny"]
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (rp[1:] - rp[:-1]).long())
    d, a = cols.long() - rows, vals.abs()
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    diag[rows[d == 0]] = vals[d == 0]
    q = torch.zeros_like(d)
    for k, (z, y, x) in enumerate((z, y, x) for z in (-1, 0, 1) for y in (-1, 0, 1)
                                  for x in (-1, 0, 1)):
        q[d == z * plane + y * nx + x] = k if k < 13 else k - 1
    off = d != 0
    f = torch.zeros((n, learn.N_IN), dtype=torch.float64, device=DEV)
    f[rows[off], 2 + q[off]] = a[off] / diag[rows[off]]
    near = f[:, 2:28]
    f[:, 0], f[:, 1] = torch.log(diag) / 8, near.sum(1)
    f[:, 28] = ((rp[1:] - rp[:-1]) > 7).double()
    least = torch.where(near > 0, near, math.inf).amin(1)
    f[:, 29] = torch.log(near.amax(1) / least) / 8
    f[:, 30], f[:, 31] = (rp[1:] - rp[:-1]).double() / 27, 1.0
    return {"features": f, "controls": _net64(learn.init_params(seed), f)[0]}

