"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values: its form (which public entry point), the
matrix (kind, rows m, mean nonzeros per row deg) and the options of the call.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a user's program has in hand before the call
    run(state)           one pass through the public entry points
    work(case)           the bytes and operations that a pass cannot do without
    exact(case, seed)    the outputs of a first pass, from plain torch in FP64

Matrices: "powerlaw" is a graph with Pareto row lengths (exponent 2.1) and
Zipf column popularity, "banded" an FEM-like matrix of 3x3 blocks in a band
with one per cent of entries anywhere, the two families that the benchmark
and the tests use.
"""
from __future__ import annotations

import functools
import math
import random

import torch

DEV = "cuda"
F64 = torch.float64


def listed() -> list[dict]:
    return [
        # a small system solved iteratively by a program that calls the CSR
        # product without a plan: latency and launches count
        _case("csr", "csr_small", kind="powerlaw", m=1500, deg=12.0),
        # the benchmark's graph (PageRank-like iterations), per-call product
        _case("csr", "csr_powerlaw", kind="powerlaw", m=4_000_000, deg=19.1),
        # an FEM operator applied many times: analysed once, FP64 values
        _case("plan", "plan_banded", kind="banded", m=500_000, deg=140.0),
        # an operator with FP32 values in a relaxation y = a*A*x + b*y, odd size
        _case("plan", "plan_f32_update", kind="powerlaw", m=100_003, deg=17.5, values="f32",
              alpha=1.25, beta=0.5),
        # a matrix kept as sorted triplets, multiplied as it is
        _case("coo", "coo_mid", kind="powerlaw", m=1_000_000, deg=17.5),
        # a CSC pattern analysed once, new values for every product (time steps)
        _case("cscplan", "csc_new_values", kind="powerlaw", m=1_000_000, deg=20.0),
        # a CSC matrix multiplied once
        _case("csc", "csc_once", kind="banded", m=150_000, deg=30.0),
        # conversion of a loaded matrix before it is used as CSR
        _case("csc2csr", "csc_to_csr", kind="powerlaw", m=1_000_000, deg=20.0),
        # a frontier or sparse update: a third of x is nonzero
        _case("spmspv", "spmspv_mid", kind="powerlaw", m=300_000, deg=17.5, density=0.3),
        # many uneven matrices, four right-hand sides each, in one launch
        _case("batch", "batch_k4", kind="mixed", m=200_000, deg=24.0, nmat=16, k=4),
        # one training step of a graph layer: forward, gradients of X and values
        _case("autograd", "train_k16", kind="powerlaw", m=1_000_000, deg=20.0, k=16),
        # the reference's C entry point with plain host arrays
        _case("host", "host_v1", kind="powerlaw", m=400_000, deg=17.5, alpha=1.0, beta=0.0),
    ]


# rows (smallest, largest), largest number of nonzeros of each form's drawn cases
_RANGE = {
    "csr": (200, 4_000_000, 70_000_000),
    "plan": (200, 2_000_000, 70_000_000),
    "coo": (1_000, 2_000_000, 24_000_000),
    "cscplan": (1_000, 1_000_000, 20_000_000),
    "csc": (1_000, 1_000_000, 20_000_000),
    "csc2csr": (1_000, 1_000_000, 20_000_000),
    "spmspv": (1_000, 1_000_000, 20_000_000),
    "batch": (2_000, 200_000, 4_000_000),
    "autograd": (1_000, 1_000_000, 20_000_000),
    "host": (1_000, 400_000, 7_000_000),
}


def draw(rng: random.Random) -> dict:
    form = rng.choice(sorted(_RANGE))
    lo, hi, most = _RANGE[form]
    m = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    deg = math.exp(rng.uniform(math.log(4.0), math.log(min(96.0, m / 8))))
    deg = round(min(deg, most / m), 2)
    kind = rng.choice(["powerlaw", "banded"])
    opt = {}
    alpha, beta = rng.choice([(1.0, 0.0), (1.0, 0.0), (0.75, 0.0), (1.25, 0.5)])
    if form in ("csr", "plan"):
        opt["values"] = rng.choice(["f64", "f64", "f32", "pattern"])
    if form == "csr":
        opt["kernel"] = rng.choice([2, 2, 3, 1 if opt["values"] == "f64" else 2])
    if form == "spmspv":
        opt["density"] = rng.choice([0.01, 0.1, 0.3, 1.0])
    if form == "batch":
        kind = "mixed"
        opt["values"] = rng.choice(["f64", "f64", "f32"])
        opt["nmat"] = rng.randint(3, 24)
        opt["k"] = rng.choice([1, 2, 4, 8])
    if form == "autograd":
        alpha, beta = 1.0, 0.0
        opt["values"] = rng.choice(["f64", "f32"])
        opt["k"] = rng.choice([1, 2, 4, 8, 16])
    return _case(form, None, kind=kind, m=m, deg=deg, alpha=alpha, beta=beta, **opt)


def _case(form, name, *, kind, m, deg, values="f64", alpha=1.0, beta=0.0, k=1, nmat=1,
          density=1.0, kernel=2) -> dict:
    c = dict(form=form, kind=kind, m=m, deg=deg, values=values, alpha=alpha, beta=beta, k=k,
             nmat=nmat, density=density, kernel=kernel)
    if name is not None:
        c["name"] = name
    return c


# ---- inputs -----------------------------------------------------------------
def _compress(m, rows, cols, g):
    """CSR pattern of the (row, col) pairs in order; a repeated pair gets
    another column of its row, so that the number of entries is the same for
    every seed."""
    key = torch.sort(rows * m + cols).values
    while True:
        again = torch.zeros_like(key, dtype=torch.bool)
        again[1:] = key[1:] == key[:-1]
        at = again.nonzero().flatten()
        if at.numel() == 0:
            break
        fresh = torch.randint(0, m, (at.numel(),), generator=g, device=DEV)
        key[at] = torch.div(key[at], m, rounding_mode="floor") * m + fresh
        key = torch.sort(key).values
    r = torch.div(key, m, rounding_mode="floor")
    rowptr = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(r, minlength=m), 0)
    return rowptr.to(torch.int32), (key - r * m).to(torch.int32), r


def _pareto_xmin(a: float, dmax: int, mean: float) -> float:
    """Smallest row length giving floor(xmin * U^(-1/a)), cut at dmax, that mean."""
    lo, hi = 0.5, float(dmax)
    for _ in range(60):
        x = 0.5 * (lo + hi)
        got = x * a / (a - 1.0) * (1.0 - (x / dmax) ** (a - 1.0)) + dmax * (x / dmax) ** a - 0.5
        lo, hi = (x, hi) if got < mean else (lo, x)
    return 0.5 * (lo + hi)


def _pattern(kind, m, deg, g):
    if kind == "powerlaw":
        dmax = max(1, min(20_000, m // 2))
        # every quantile of the row lengths once, in the seed's order
        u = (torch.randperm(m, generator=g, device=DEV) + 0.5) / m
        ln = torch.floor(_pareto_xmin(1.1, dmax, deg) * u.to(F64).pow(-1.0 / 1.1))
        rows = torch.repeat_interleave(torch.arange(m, device=DEV), ln.clamp_(1, dmax).long())
        e = 1.0 - 1.0 / 1.1
        u = torch.rand(rows.numel(), generator=g, dtype=F64, device=DEV)
        rank = (((m + 1.0) ** e - 1.0) * u + 1.0).pow(1.0 / e) - 1.0
        cols = torch.randperm(m, generator=g, device=DEV)[rank.floor_().clamp_(0, m - 1).long()]
        return _compress(m, rows, cols, g)
    nb = (m + 2) // 3
    half = max(1, min(20_000, m) // 6)
    per = max(1, round(0.99 * deg / 3))
    br = torch.arange(nb, device=DEV).repeat_interleave(per)
    off = torch.randint(-half, half + 1, (nb * per,), generator=g, device=DEV)
    off.view(nb, per)[:, 0] = 0
    bc = (br + off).abs()                              # reflected at both ends
    bc = torch.where(bc < nb, bc, 2 * (nb - 1) - bc)
    a = torch.arange(3, device=DEV)
    rows = (3 * br[:, None, None] + a[None, :, None]).expand(-1, 3, 3).reshape(-1)
    cols = (3 * bc[:, None, None] + a[None, None, :]).expand(-1, 3, 3).reshape(-1)
    keep = rows < m
    some = int(0.01 * deg * m)
    rows = torch.cat([rows[keep], torch.randint(0, m, (some,), generator=g, device=DEV)])
    cols = torch.cat([cols[keep], torch.randint(0, m, (some,), generator=g, device=DEV)])
    return _compress(m, rows, cols.clamp_(max=m - 1), g)


def _matrix(kind, m, deg, values, g):
    rowptr, col, row = _pattern(kind, m, deg, g)
    if values == "pattern":
        return rowptr, col, row, None
    val = torch.randn(col.numel(), generator=g, dtype=F64, device=DEV)
    if kind == "banded":
        val += (col.long() == row) * (1.0 + deg)   # diagonally dominant
    return rowptr, col, row, val.float() if values == "f32" else val


def _members(case):
    """(kind, rows, row length) of every matrix of a case."""
    if case["form"] != "batch":
        return [(case["kind"], case["m"], case["deg"])]
    r = random.Random(case["m"] * 31 + case["nmat"])
    lo = max(500, case["m"] // 20)
    out = []
    for i in range(case["nmat"]):
        m = int(math.exp(r.uniform(math.log(lo), math.log(case["m"]))))
        out.append(("powerlaw" if i % 2 == 0 else "banded", m,
                    max(3.0, case["deg"] * math.exp(r.uniform(-0.7, 0.7)))))
    return out


def _inputs(case, seed):
    """Every matrix of a case as row-sorted entries, with its x and first y."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    out = []
    k, shape = case["k"], (lambda m: (m, case["k"]) if case["k"] > 1 else (m,))
    for kind, m, deg in _members(case):
        rowptr, col, row, val = _matrix(kind, m, deg, case["values"], g)
        x = torch.rand(shape(m), generator=g, dtype=F64, device=DEV)
        if kind == "banded" or k > 1:
            x = 2.0 * x - 1.0
        if case["density"] < 1.0:
            x *= torch.rand(x.shape, generator=g, dtype=F64, device=DEV) < case["density"]
        y = torch.rand(shape(m), generator=g, dtype=F64, device=DEV)
        out.append(dict(m=m, rowptr=rowptr, col=col, row=row, val=val, x=x, y=y))
    return out


def _to_csc(d):
    """Column-compressed arrays, rows ascending in each column."""
    perm = torch.sort(d["col"].long() * d["m"] + d["row"]).indices
    colptr = torch.zeros(d["m"] + 1, dtype=torch.int64, device=DEV)
    colptr[1:] = torch.cumsum(torch.bincount(d["col"].long(), minlength=d["m"]), 0)
    return colptr.int(), d["row"][perm].int(), d["val"][perm]


# ---- the cases --------------------------------------------------------------
def prepare(case, seed):
    from hpda_sblas_pnnl_gb300 import ops
    form = case["form"]
    mats = _inputs(case, seed)
    d = mats[0]
    s = dict(form=form, m=d["m"], alpha=case["alpha"], beta=case["beta"], kernel=case["kernel"])
    if form == "batch":
        s["ys"] = [q["y"] for q in mats]
        s["plan"] = ops.BatchPlan([(q["rowptr"], q["col"], q["val"]) for q in mats],
                                  [q["x"] for q in mats], s["ys"], case["k"],
                                  alpha=case["alpha"], beta=case["beta"])
    elif form == "autograd":
        from hpda_sblas_pnnl_gb300 import autograd
        s["op"] = autograd.CsrOperator(d["rowptr"], d["col"], d["m"], case["k"], d["val"].dtype)
        s["val"] = d["val"].requires_grad_()
        s["x"] = d["x"].requires_grad_()
        s["gy"] = d["y"]
    elif form == "host":
        for name in ("rowptr", "col", "val", "x", "y"):
            s[name] = d[name].cpu().numpy()
    elif form in ("csc", "cscplan", "csc2csr"):
        s["colptr"], s["rowidx"], s["val"] = _to_csc(d)
        s["x"], s["y"] = d["x"], d["y"]
        if form == "cscplan":
            s["plan"] = ops.CscPlan(d["m"], s["colptr"], s["rowidx"])
    else:
        s |= {name: d[name] for name in ("rowptr", "col", "val", "x", "y")}
        if form == "plan":
            s["plan"] = ops.CsrPlan(d["rowptr"], d["col"], d["val"], n=d["m"],
                                    kernel=case["kernel"])
        elif form == "coo":
            s["row"] = d["row"].int()
    return s


def run(s):
    from hpda_sblas_pnnl_gb300 import api, autograd, ops
    form, alpha, beta = s["form"], s["alpha"], s["beta"]
    if form == "csr":
        return ops.csrmv(s["rowptr"], s["col"], s["val"], s["x"], s["y"], alpha, beta,
                         kernel=s["kernel"])
    if form == "plan":
        return s["plan"](s["x"], s["y"], alpha, beta)
    if form == "coo":
        return ops.coomv(s["row"], s["col"], s["val"], s["x"], s["y"], alpha, beta)
    if form == "cscplan":
        return s["plan"](s["val"], s["x"], s["y"], alpha, beta)
    if form == "csc":
        return ops.cscmv(s["colptr"], s["rowidx"], s["val"], s["x"], s["y"], alpha, beta)
    if form == "csc2csr":
        return ops.csc_to_csr(s["m"], s["m"], s["colptr"], s["rowidx"], s["val"])
    if form == "spmspv":
        return ops.spmspv(s["rowptr"], s["col"], s["val"], s["x"], s["y"], alpha, beta)
    if form == "batch":
        s["plan"]()
        return s["ys"]
    if form == "autograd":
        y = autograd.spmm(s["op"], s["val"], s["x"])
        dval, dx = torch.autograd.grad(y, (s["val"], s["x"]), s["gy"])
        return y.detach(), dval, dx
    api.spMV_mgpu_v1(s["m"], s["m"], s["val"].size, alpha, s["val"], s["rowptr"], s["col"],
                     s["x"], beta, s["y"], ngpu=1, kernel=s["kernel"])
    return s["y"]


@functools.lru_cache(maxsize=None)
def _nnz(kind, m, deg):
    g = torch.Generator(device=DEV)
    g.manual_seed(1)
    return _pattern(kind, m, deg, g)[1].numel()


def work(case):
    k = case["k"]
    vb = {"f64": 8, "f32": 4, "pattern": 0}[case["values"]]
    reads_y = 2 if case["beta"] != 0.0 else 1
    nbytes = flops = 0
    for kind, m, deg in _members(case):
        nnz = _nnz(kind, m, deg)
        a, vec = (vb + 4) * nnz + 4 * (m + 1), 8 * m * k
        if case["form"] == "coo":
            a = (vb + 8) * nnz
        if case["form"] == "cscplan":
            a += 4 * nnz   # where each value goes: the pattern's row order
        if case["form"] == "csc2csr":
            nbytes += 2 * a
            continue
        if case["form"] == "autograd":   # Y = AX; dX = A'G; dval = G.X at the pattern
            nbytes += a + vb * nnz + 4 * vec
            flops += 6 * nnz * k
            continue
        nbytes += a + vec + reads_y * vec
        flops += 2 * nnz * k
    return {"bytes": nbytes, "flops": flops}


# ---- the outputs in plain torch, 64 bits --------------------------------------
def _times(row, col, val, x, m):
    """A x by entries, a column of x at a time."""
    out = torch.zeros((m,) + tuple(x.shape[1:]), dtype=F64, device=DEV)
    for c in range(1 if x.dim() == 1 else x.shape[1]):
        xc, oc = (x, out) if x.dim() == 1 else (x[:, c].contiguous(), out[:, c])
        p = xc[col] if val is None else val.double() * xc[col]
        oc.copy_(torch.zeros(m, dtype=F64, device=DEV).index_add_(0, row, p))
    return out


def exact(case, seed):
    alpha, beta, form = case["alpha"], case["beta"], case["form"]
    outs = []
    for d in _inputs(case, seed):
        row, col, val, x, m = d["row"], d["col"].long(), d["val"], d["x"], d["m"]
        if form == "csc2csr":
            return None, None, val
        y = _times(row, col, val, x, m)
        if form == "autograd":
            gy = d["y"]
            dval = torch.zeros(col.numel(), dtype=F64, device=DEV)
            for c in range(case["k"]):
                gc, xc = (gy, x) if case["k"] == 1 else (gy[:, c].contiguous(), x[:, c].contiguous())
                dval += gc[row] * xc[col]
            return y, dval, _times(col, row, val, gy, m)
        outs.append(alpha * y + beta * d["y"] if beta != 0.0 else alpha * y)
    return outs if form == "batch" else outs[0]
