"""Forms of the public calls that have to keep their results: optional arrays
left out, empty matrices, workspaces at any alignment, one call after another
on the same workspace.  Whole numbers and moved values equal, FP64 sums
within 1e-12 relative L2."""
import ctypes as C
import subprocess
import sys
import time
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RTOL_L2 = 1e-12


def rel_l2(y, ref):
    den = np.linalg.norm(ref)
    num = np.linalg.norm(np.asarray(y) - ref)
    return num / den if den > 0 else num


def csc_pattern(m, n, nnz, seed):
    """Sorted columns with rows in any order: colptr, rows, cols."""
    rng = np.random.default_rng(seed)
    cols = np.sort(rng.integers(0, n, nnz))
    rows = rng.integers(0, m, nnz).astype(np.int32)
    colptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int32)
    return colptr, rows, cols


@pytest.mark.parametrize("nnz", [1, 1025, 40_000, (1 << 19) + 1, (1 << 22) + 1])
@pytest.mark.parametrize("m", [900, 60_000])
def test_csc_to_csr_of_a_pattern(sblas_lib, cuda, nnz, m):
    """No values: the structure, and zeros for the values (one and two passes,
    every tile size)."""
    from hpda_sblas_pnnl_gb300 import ops
    n = 3000
    colptr, rows, cols = csc_pattern(m, n, nnz, nnz)
    rp, c, v = ops.csc_to_csr(m, n, torch.from_numpy(colptr).to(cuda),
                              torch.from_numpy(rows).to(cuda), None)
    order = np.argsort(rows, kind="stable")
    assert np.array_equal(rp.cpu().numpy(),
                          np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]))
    assert np.array_equal(c.cpu().numpy(), cols[order])
    assert not v.any()


@pytest.mark.parametrize("nnz", [1, 5000, (1 << 19) + 1, (1 << 22) + 1])
@pytest.mark.parametrize("m", [900, 60_000, 5_000_000])
@pytest.mark.parametrize("offset", [0, 4, 8, 20])
def test_sort_workspace_at_any_alignment(sblas_lib, cuda, nnz, m, offset):
    """The sorts ask for bytes of workspace, not for an alignment: one, two and
    three passes with the workspace `offset` bytes into an allocation, and
    nothing written past the bytes that were asked for."""
    n = 3000
    colptr, rows, cols = csc_pattern(m, n, nnz, nnz)
    val = np.random.default_rng(1).standard_normal(nnz)
    order = np.argsort(rows, kind="stable")
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))])
    cp, ri, v = (torch.from_numpy(a).to(cuda) for a in (colptr, rows, val))
    rp = torch.empty(m + 1, dtype=torch.int32, device=cuda)
    c, perm = (torch.empty(nnz, dtype=torch.int32, device=cuda) for _ in range(2))
    out = torch.empty(nnz, dtype=torch.float64, device=cuda)
    stream = C.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)

    def work(size):
        t = torch.full((size + offset + 64,), 0x5A, dtype=torch.uint8, device=cuda)
        return t, t.data_ptr() + offset, t[offset + size:]

    wb = sblas_lib.sblas_csc_to_csr_workspace_bytes(m, n, nnz)
    keep, w, rest = work(wb)
    assert sblas_lib.sblas_csc_to_csr(m, n, nnz, v.data_ptr(), cp.data_ptr(), ri.data_ptr(),
                                      out.data_ptr(), rp.data_ptr(), c.data_ptr(), w, wb, stream) == 0
    assert np.array_equal(rp.cpu().numpy(), rowptr)
    assert np.array_equal(c.cpu().numpy(), cols[order])
    assert np.array_equal(out.cpu().numpy(), val[order])
    assert bool((rest == 0x5A).all())
    # the same arrays as a CSR matrix of n rows: its transpose
    wb = sblas_lib.sblas_csr_transpose_workspace_bytes(n, m, nnz)
    keep, w, rest = work(wb)
    assert sblas_lib.sblas_csr_transpose(n, m, nnz, cp.data_ptr(), ri.data_ptr(), rp.data_ptr(),
                                         c.data_ptr(), perm.data_ptr(), w, wb, stream) == 0
    assert np.array_equal(rp.cpu().numpy(), rowptr)
    assert np.array_equal(c.cpu().numpy(), cols[order])
    assert np.array_equal(perm.cpu().numpy(), order)
    assert bool((rest == 0x5A).all())


def test_sort_with_the_most_columns(sblas_lib, cuda):
    """2^31 - 1 columns with entries in the last of them: the search for an entry's
    column stays in 32 bits."""
    from hpda_sblas_pnnl_gb300 import ops
    m, n = 7, (1 << 31) - 1
    at = [n - 90_000, n - 70_000, n - 514, n - 300, n - 258, n - 257, n - 2, n - 1]
    colptr = torch.zeros(n + 1, dtype=torch.int32, device=cuda)
    for c in at:
        colptr[c + 1:] += 1
    rows = torch.tensor([3, 0, 3, 6, 6, 1, 0, 3], dtype=torch.int32, device=cuda)
    val = torch.arange(8, dtype=torch.float64, device=cuda)
    rp, c, v = ops.csc_to_csr(m, n, colptr, rows, val)
    order = np.argsort(rows.cpu().numpy(), kind="stable")
    assert c.cpu().tolist() == [at[i] for i in order]
    assert v.cpu().tolist() == [float(i) for i in order]
    assert rp.cpu().tolist() == [0, 2, 3, 3, 6, 6, 6, 8]


def test_first_call_inside_a_capture(sblas_lib, cuda):
    """The library's first call in a process may be one that is captured: a
    caller's workspace, nothing allocated, nothing run before."""
    code = """
import torch
from hpda_sblas_pnnl_gb300 import ops
m, per = 20_000, 20
col = torch.arange(m * per, device="cuda", dtype=torch.int32) % m
rp = (torch.arange(m + 1, device="cuda") * per).int()
val = torch.ones(m * per, dtype=torch.float64, device="cuda")
x = torch.ones(m, dtype=torch.float64, device="cuda")
y = torch.zeros(m, dtype=torch.float64, device="cuda")
work = torch.empty(ops.workspace_bytes(m * per), dtype=torch.uint8, device="cuda")
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    ops.csrmv(rp, col, val, x, y, work=work)
g.replay()
torch.cuda.synchronize()
assert bool((y == per).all())
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("nnz", [1, 3000, 200_000, 1 << 20])
def test_one_shot_csc_product_leaves_an_analysis(sblas_lib, cuda, nnz):
    """sblas_dcscmv in the caller's workspace, then products with other values
    of the pattern, and with bound ones, from the same workspace."""
    from hpda_sblas_pnnl_gb300 import _lib, ops
    m, n = 70_000, 9000
    colptr, rows, cols = csc_pattern(m, n, nnz, nnz)
    rng = np.random.default_rng(2)
    x, y0 = rng.standard_normal(n), rng.standard_normal(m)
    cp, ri, xd = (torch.from_numpy(a).to(cuda) for a in (colptr, rows, x))
    wb = sblas_lib.sblas_cscmv_workspace_bytes(m, n, nnz)
    work = torch.full((wb,), 0xFF, dtype=torch.uint8, device=cuda)
    stream = C.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)
    for step in range(3):
        val = rng.standard_normal(nnz)
        v, y = torch.from_numpy(val).to(cuda), torch.from_numpy(y0).to(cuda)
        if step == 0:
            ops.cscmv(cp, ri, v, xd, y, 1.5, -0.5, work=work)
        else:
            if step == 2:
                _lib.check(sblas_lib.sblas_csc_bind_values(m, n, nnz, v.data_ptr(), work.data_ptr(),
                                                           wb, stream))
            _lib.check(sblas_lib.sblas_dcscmv_analysed(
                m, n, nnz, 1.5, v.data_ptr() if step == 1 else None, xd.data_ptr(), -0.5,
                y.data_ptr(), work.data_ptr(), wb, stream))
        ref = -0.5 * y0
        np.add.at(ref, rows, 1.5 * val * x[cols])
        assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2, step


@pytest.mark.parametrize("kernel", [1, 2, 3])
def test_spmspv_of_an_empty_matrix(sblas_lib, cuda, kernel):
    """No nonzeros: y = beta * y for every kernel that takes the form of the
    values; kernel 1 refuses a pattern, empty or not."""
    from hpda_sblas_pnnl_gb300 import _lib, ops
    rp = torch.zeros(6, dtype=torch.int32, device=cuda)
    col = torch.zeros(0, dtype=torch.int32, device=cuda)
    val = torch.zeros(0, dtype=torch.float64, device=cuda)
    x = torch.ones(3, dtype=torch.float64, device=cuda)
    y = torch.full((5,), 3.0, dtype=torch.float64, device=cuda)
    ops.spmspv(rp, col, val, x, y, 1.0, 0.5, kernel=kernel)
    assert y.tolist() == [1.5] * 5
    if kernel == 1:
        with pytest.raises(_lib.SblasError):
            ops.spmspv(rp, col, None, x, y, 1.0, 0.5, kernel=kernel)
    else:
        ops.spmspv(rp, col, None, x, y, 1.0, 0.0, kernel=kernel)
        assert y.tolist() == [0.0] * 5


@pytest.mark.parametrize("lengths", [[3, 4], [5, 0, 700, 3] * 40, [60, 600, 7] * 9, [4] * 3000],
                         ids=lambda v: f"{len(v)}x{max(v)}")
@pytest.mark.parametrize("short", [1, 5, 300])
def test_small_matrix_reads_no_entry_past_its_arrays(sblas_lib, cuda, lengths, short):
    """A row pointer that says more than col and val hold (they are views of
    longer arrays with NaN behind): the entries that are there, for lanes, warps
    and the CTA, with and without zeros of x left out."""
    from hpda_sblas_pnnl_gb300 import ops
    rng = np.random.default_rng(short)
    n, m = 400, len(lengths)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    have = max(int(rp[-1]) - short, 1)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val, x = rng.standard_normal(rp[-1]), rng.standard_normal(n)
    ref = np.zeros(m)
    rows = np.repeat(np.arange(m), lengths)
    np.add.at(ref, rows[:have], val[:have] * x[col[:have]])
    val[have:] = np.nan
    trp, tcol, tval, tx = (torch.from_numpy(a).to(cuda) for a in (rp, col, val, x))
    tcol, tval = tcol[:have], tval[:have]
    y = torch.empty(m, dtype=torch.float64, device=cuda)
    for kernel in (2, 3):
        assert rel_l2(ops.csrmv(trp, tcol, tval, tx, y, kernel=kernel).cpu().numpy(), ref) <= RTOL_L2
        assert rel_l2(ops.spmspv(trp, tcol, tval, tx, y, kernel=kernel).cpu().numpy(), ref) <= RTOL_L2
    assert rel_l2(ops.CsrPlan(trp, tcol, tval, n=n)(tx, y).cpu().numpy(), ref) <= RTOL_L2


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("nnz", [1 << 18, 1 << 21, (1 << 22) - 1, 1 << 22, (1 << 24) + 5])
def test_host_call_times_are_of_what_they_say(sblas_lib, cuda, pinned, nnz):
    """comp_time is the kernels' time, with and without chunks: the copies that
    they wait for stay out.  A product reads its 12 bytes per nonzero at several
    TB/s, the copies move them at a few hundred GB/s at most: far below half
    of the copies' time (from 2^21 nonzeros on, where launches count little);
    and the parts of a call are not longer than the call."""
    from hpda_sblas_pnnl_gb300 import api
    rng = np.random.default_rng(nnz)
    m, n = nnz // 20, 40_000
    rp = np.minimum(np.arange(m + 1, dtype=np.int64) * 20, nnz).astype(np.int32)
    rp[-1] = nnz
    col = rng.integers(0, n, nnz).astype(np.int32)
    val, x, y = rng.standard_normal(nnz), rng.standard_normal(n), np.zeros(m)
    if pinned:
        keep = [torch.from_numpy(a).pin_memory() for a in (val, rp, col, x, y)]
        val, rp, col, x, y = (t.numpy() for t in keep)
    share = []
    for _ in range(5):
        t0 = time.perf_counter()
        r = api.spMV_mgpu_v1(m, n, nnz, 1.0, val, rp, col, x, 0.0, y)
        wall = time.perf_counter() - t0
        assert 0 < r.comp_time and 0 < r.comm_time and 0 <= r.merg_time and r.part_time >= 0
        assert max(r.comp_time, r.comm_time, r.merg_time) <= wall
        share.append(r.comp_time / r.comm_time)
    if nnz >= 1 << 21:
        assert min(share) <= 0.5, share     # the least: a host that is held up delays the kernels


@pytest.mark.parametrize("k", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("s", [1, 2])
@pytest.mark.parametrize("vals", ["f64", "f32"])
def test_short_units_by_request(sblas_lib, cuda, k, s, vals):
    """s = 1 and 2, which a plan picks for small matrices at k >= 8: rows at the
    lengths of a unit and of the fix-up's runs, many rows in a unit, empty
    rows; product, values' adjoint, and a plan made again from what it
    reports.  Refused at smaller k, where they are not compiled."""
    from hpda_sblas_pnnl_gb300 import _lib, ops
    from oracle import oracle as O
    unit = 32 * s
    lengths = ([0, 1, unit - 1, 0, 0, unit, unit + 1] + [1] * (2 * unit + 3) + [0] * 40 + [2, 0] * unit +
               [33 * unit, 7, 32 * unit - 7, 31 * unit, 3, 300 * unit + 5, 0])
    n, m = 700, len(lengths)
    rng = np.random.default_rng(k + s)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val = rng.standard_normal(rp[-1])
    trp, tcol, tval = (torch.from_numpy(a).to(cuda) for a in (rp, col, val))
    if vals == "f32":
        tval = tval.float()
        val = tval.double().cpu().numpy()
    if k < 8:
        with pytest.raises(_lib.SblasError):
            ops.SpmmPlan(trp, tcol, tval, n=n, k=k, s=s)
        return
    x, y0 = rng.standard_normal((n, k)), rng.standard_normal((m, k))
    tx = torch.from_numpy(x).to(cuda)
    plan = ops.SpmmPlan(trp, tcol, tval, n=n, k=k, s=s)
    y = torch.from_numpy(y0).to(cuda)
    plan(tx, y, 1.5, -0.5)
    assert rel_l2(y.cpu().numpy(), O.csr_spmm(m, n, rp, col, val, x, y0.copy(), 1.5, -0.5)) <= RTOL_L2
    dval = torch.empty_like(tval)
    plan.sddmm(y, tx, dval)
    ref = O.csr_sddmm(m, n, rp, col, y.cpu().numpy(), x)
    assert rel_l2(dval.double().cpu().numpy(), ref) <= (RTOL_L2 if vals == "f64" else 2.0 ** -24)
    # what a plan picks for a small matrix can be asked for
    small = [torch.from_numpy(a).to(cuda) for a in (rp[:40] * 1, col, val)]
    small[1], small[2] = small[1][:rp[39]].contiguous(), small[2][:rp[39]].contiguous()
    picked = ops.SpmmPlan(*small, n=n, k=k).s
    assert picked == 1
    assert ops.SpmmPlan(*small, n=n, k=k, s=picked).s == picked


def test_kernel_1_on_many_almost_empty_rows(sblas_lib, cuda):
    """4M rows, 100K nonzeros: kernel 1 streams the row pointer and y (12 bytes
    per row, 7 us at the memory's rate) and is not held up row by row."""
    from hpda_sblas_pnnl_gb300 import ops
    m, n, nnz = 4_000_000, 20_000, 100_000
    rng = np.random.default_rng(1)
    rows = np.sort(rng.integers(0, m, nnz))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int32)
    col, val, x = rng.integers(0, n, nnz).astype(np.int32), rng.standard_normal(nnz), rng.standard_normal(n)
    ref = np.zeros(m)
    np.add.at(ref, rows, val * x[col])
    trp, tcol, tval, tx = (torch.from_numpy(a).to(cuda) for a in (rp, col, val, x))
    y = torch.empty(m, dtype=torch.float64, device=cuda)
    for call in (ops.csrmv, ops.spmspv):
        best = 1e9
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            call(trp, tcol, tval, tx, y, kernel=1)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3)
        assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2
        assert best <= 20 * 12 * m / 6.8e12 * 1e6, best


@pytest.mark.parametrize("m", [4865, 9728, 9729, 78_000])
def test_small_matrix_over_several_steps_of_the_grid(sblas_lib, cuda, m):
    """More rows than one step of the grid covers, with rows for a warp and for
    the CTA in the first and in later steps; kernel 1 on both sides of its rule."""
    from hpda_sblas_pnnl_gb300 import ops
    rng = np.random.default_rng(m)
    lengths = rng.integers(0, 2, m)
    for i, r in enumerate(rng.choice(m, 40, replace=False)):
        lengths[r] = (65, 512, 513, 900)[i % 4]
    lengths[-1], lengths[-2] = 700, 100
    n = 3000
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    nnz = int(rp[-1])
    assert nnz <= 131_072
    col, val = rng.integers(0, n, nnz).astype(np.int32), rng.standard_normal(nnz)
    x, y0 = rng.standard_normal(n), rng.standard_normal(m)
    ref = -0.5 * y0
    np.add.at(ref, np.repeat(np.arange(m), lengths), 1.5 * val * x[col])
    trp, tcol, tval, tx = (torch.from_numpy(a).to(cuda) for a in (rp, col, val, x))
    for kernel in (1, 2, 3):
        for call in (ops.csrmv, ops.spmspv):
            y = torch.from_numpy(y0).to(cuda)
            call(trp, tcol, tval, tx, y, 1.5, -0.5, kernel=kernel)
            assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2, (kernel, call)
    y = torch.from_numpy(y0).to(cuda)
    assert rel_l2(ops.CsrPlan(trp, tcol, tval, n=n)(tx, y, 1.5, -0.5).cpu().numpy(), ref) <= RTOL_L2


@pytest.mark.parametrize("m,nnz,long_row", [(3000, 600_000, 9000), (20_000, 100_000, 16_000),
                                            (300_000, 100_000, 500), (200_000, 3_000_000, 11_000)])
def test_spmspv_kernel_1_is_not_held_up_by_long_rows(sblas_lib, cuda, m, nnz, long_row):
    """Kernel 1 with and without a workspace (infinite values at zeros of x left
    out); through ops.spmspv, which passes one, it takes at most twice as long
    as kernel 2."""
    from hpda_sblas_pnnl_gb300 import _lib, ops
    rng = np.random.default_rng(m)
    n = 10_000
    rows = rng.integers(0, m, nnz)
    rows[:long_row] = m // 2
    rows = np.sort(rows)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))]).astype(np.int32)
    col, val = rng.integers(0, n, nnz).astype(np.int32), rng.standard_normal(nnz)
    x = rng.standard_normal(n) * (rng.random(n) < 0.02)
    y0 = rng.standard_normal(m)
    ref = -0.5 * y0
    live = x[col] != 0.0
    np.add.at(ref, rows[live], 1.5 * val[live] * x[col[live]])
    val[~live] = np.inf
    trp, tcol, tval, tx = (torch.from_numpy(a).to(cuda) for a in (rp, col, val, x))
    y = torch.from_numpy(y0).to(cuda)
    stream = C.c_void_p(torch.cuda.current_stream(cuda).cuda_stream)
    _lib.check(sblas_lib.sblas_dspmspv(1, m, n, nnz, 1.5, tval.data_ptr(), trp.data_ptr(),
                                       tcol.data_ptr(), tx.data_ptr(), -0.5, y.data_ptr(), None, 0,
                                       stream))
    assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2
    best = {}
    for kernel in (1, 2):
        best[kernel] = 1e9
        for _ in range(10):
            y.copy_(torch.from_numpy(y0))
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            ops.spmspv(trp, tcol, tval, tx, y, 1.5, -0.5, kernel=kernel)
            b.record()
            b.synchronize()
            best[kernel] = min(best[kernel], a.elapsed_time(b) * 1e3)
        assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2, kernel
    assert best[1] <= 2 * best[2], best


@pytest.mark.parametrize("k", [2, 4, 8, 16])
@pytest.mark.parametrize("m,nnz", [(3_000_000, 4_000_000), (6_000_000, 7_000_000), (700, 300_000),
                                   (2000, 900_000), (30_000, 1_200_000)])
def test_plans_picked_for_short_and_long_rows(sblas_lib, cuda, k, m, nnz):
    """s = 0 on matrices with about one nonzero per row, and with hundreds: one
    matrix and a batch, product and values' adjoint, and no long units where
    a unit would hold more rows than nonzeros fit."""
    from hpda_sblas_pnnl_gb300 import ops
    g = torch.Generator(device=cuda)
    g.manual_seed(nnz + k)
    n = 4000
    rows = torch.sort(torch.randint(0, m, (nnz,), generator=g, device=cuda)).values
    rp = torch.zeros(m + 1, dtype=torch.int32, device=cuda)
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0).int()
    col = torch.randint(0, n, (nnz,), generator=g, device=cuda, dtype=torch.int32)
    val = torch.randn(nnz, generator=g, dtype=torch.float64, device=cuda)
    x = torch.randn((n, k), generator=g, dtype=torch.float64, device=cuda)
    y0 = torch.randn((m, k), generator=g, dtype=torch.float64, device=cuda)
    ref = -0.5 * y0
    ref.index_add_(0, rows, 1.5 * val[:, None] * x[col.long()])
    plan = ops.SpmmPlan(rp, col, val, n=n, k=k)
    y = y0.clone()
    plan(x, y, 1.5, -0.5)
    assert float((y - ref).norm() / ref.norm()) <= RTOL_L2
    dval = torch.empty_like(val)
    plan.sddmm(y0, x, dval)
    dref = (y0[rows] * x[col.long()]).sum(1)
    assert float((dval - dref).norm() / dref.norm()) <= RTOL_L2
    ys = [y0.clone() for _ in range(2)]
    batch = ops.BatchPlan([(rp, col, val)] * 2, [x] * 2, ys, k, alpha=1.5, beta=-0.5)
    batch()
    for y in ys:
        assert float((y - ref).norm() / ref.norm()) <= RTOL_L2
    if nnz < 4 * m:
        assert plan.s <= 8 and batch.s <= 8


@pytest.mark.parametrize("nnz", [5000, 300_000])
def test_analysed_csc_product_without_values_uses_the_last_ones(sblas_lib, cuda, nnz):
    """val = None: the values that the plan holds in row order, whether bind() or
    a product put them there last."""
    from hpda_sblas_pnnl_gb300 import ops
    m, n = 4000, 3000
    colptr, rows, cols = csc_pattern(m, n, nnz, nnz)
    rng = np.random.default_rng(3)
    a, b, x = rng.standard_normal(nnz), rng.standard_normal(nnz), rng.standard_normal(n)
    cp, ri, ta, tb, tx = (torch.from_numpy(t).to(cuda) for t in (colptr, rows, a, b, x))
    plan = ops.CscPlan(m, cp, ri)
    y = torch.empty(m, dtype=torch.float64, device=cuda)
    with pytest.raises(ValueError):
        plan(None, tx, y)
    plan.bind(ta)
    of_a = plan(None, tx, y).clone()
    ref = np.zeros(m)
    np.add.at(ref, rows, a * x[cols])
    assert rel_l2(of_a.cpu().numpy(), ref) <= RTOL_L2
    of_b = plan(tb, tx, y).clone()
    assert torch.equal(plan(None, tx, y), of_b) and not torch.equal(of_a, of_b)
    plan.bind(ta)
    assert torch.equal(plan(None, tx, y), of_a)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("m,nnz,last", [(1, 5, 5), (700, 9000, 1), (700, 300_001, 100_000),
                                        (5000, 300_000, 300_000)])
def test_coo_rows_past_the_end_stay_inside(sblas_lib, cuda, offset, m, nnz, last):
    """Sorted row indices of m and more (counted from one, say): taken as the
    last row by the row pointer and by the tile partition alike, over many
    tiles too; nothing is written behind y or the row pointer."""
    from hpda_sblas_pnnl_gb300 import ops
    rng = np.random.default_rng(nnz)
    n = 300
    rows = np.sort(rng.integers(0, m, nnz)).astype(np.int32)
    rows[nnz - last:] = np.sort(rng.integers(m, m + 3, last))
    col, val, x = rng.integers(0, n, nnz).astype(np.int32), rng.standard_normal(nnz), rng.standard_normal(n)
    ref = np.zeros(m)
    np.add.at(ref, np.minimum(rows, m - 1), val * x[col])
    pad = torch.zeros(nnz + offset, dtype=torch.int32, device=cuda)
    pad[offset:] = torch.from_numpy(rows).to(cuda)
    tc, tv, tx = (torch.from_numpy(a).to(cuda) for a in (col, val, x))
    for sigma in (0, 11, 27):
        y = torch.full((m + 64,), -7.0, dtype=torch.float64, device=cuda)
        rp = torch.full((m + 1 + 64,), -7, dtype=torch.int32, device=cuda)
        ops.coomv(pad[offset:], tc, tv, tx, y[:m], rowptr_work=rp[:m + 1], sigma=sigma)
        assert bool((y[m:] == -7.0).all()) and bool((rp[m + 1:] == -7).all())
        assert int(rp[m]) == nnz
        assert rel_l2(y[:m].cpu().numpy(), ref) <= RTOL_L2
