"""Sizes at which a kernel or a rule that chooses one can go wrong: run
lengths, tile remainders, the smallest and largest sizes of a path.  The
checker is the oracle; bars as in the other GPU tests (relative L2 <= 1e-12
for FP64 sums in another order, whole numbers equal)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

RTOL_L2 = 1e-12


def rel_l2(y, ref):
    den = np.linalg.norm(ref)
    num = np.linalg.norm(np.asarray(y) - ref)
    return num / den if den > 0 else num


def csr_of_lengths(lengths, n, seed, cuda):
    """A CSR matrix with the given row lengths, random columns and values."""
    rng = np.random.default_rng(seed)
    rowptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = rng.integers(0, n, rowptr[-1]).astype(np.int32)
    val = rng.standard_normal(rowptr[-1])
    return (rowptr, col, val), tuple(torch.from_numpy(a).to(cuda) for a in (rowptr, col, val))


@pytest.mark.parametrize("k", [1, 2, 4, 8, 16])
def test_batch_fixup_run_lengths(sblas_lib, cuda, k):
    """Rows over 1, 31, 32, 33 units, over the last run a warp takes and the
    first the whole block takes, and the longest, side by side."""
    from hpda_sblas_pnnl_gb300 import ops
    s, unit, wg = 4, 128, 32 // k
    edge = 64 * wg * unit
    lengths = [5, 1, 3 * unit, 0, 31 * unit, 32 * unit - 3, 33 * unit, 7, edge - unit, edge + unit,
               0, 0, 2 * edge + 17, 40 * unit, 2, 33 * unit, 33 * unit + 1, 1]
    n = 5000
    (rp, col, val), dev = csr_of_lengths(lengths, n, 11 + k, cuda)
    m = len(lengths)
    g = torch.Generator(device=cuda)
    g.manual_seed(k)
    shape = (lambda r: (r, k) if k > 1 else (r,))
    x = torch.randn(shape(n), generator=g, dtype=torch.float64, device=cuda)
    y0 = torch.randn(shape(m), generator=g, dtype=torch.float64, device=cuda)
    plan = ops.SpmmPlan(*dev, n=n, k=k, s=s)
    y = y0.clone()
    plan(x, y, 1.5, -0.5)
    first = y.clone()
    ref = O.csr_spmm(m, n, rp, col, val, x.cpu().numpy().reshape(n, k),
                     y0.cpu().numpy().reshape(m, k), 1.5, -0.5)
    assert rel_l2(y.cpu().numpy().reshape(m, k), ref) <= RTOL_L2
    y.copy_(y0)
    plan(x, y, 1.5, -0.5)
    assert torch.equal(y, first)      # the same bits on every run


@pytest.mark.parametrize("k", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("nnz", [3_000, 20_000, 250_000, 500_000, 1_300_000, 6_100_000])
def test_plan_picks_a_shape_for_every_size(sblas_lib, cuda, k, nnz):
    """s = 0 on both sides of each size at which the pick changes, with a
    permuted transpose product: forward and both gradients."""
    from hpda_sblas_pnnl_gb300 import autograd
    rng = np.random.default_rng(nnz + k)
    m = max(50, nnz // 20)
    lengths = rng.multinomial(nnz, rng.dirichlet(np.ones(m)))
    (rp, col, val), (trp, tcol, tval) = csr_of_lengths(lengths, m, nnz + k, cuda)
    op = autograd.CsrOperator(trp, tcol, m, k)
    x = torch.from_numpy(rng.standard_normal((m, k))).to(cuda)
    gy = torch.from_numpy(rng.standard_normal((m, k))).to(cuda)
    y = op.forward(tval, x)
    ref = O.csr_spmm(m, m, rp, col, val, x.cpu().numpy(), np.zeros((m, k)))
    assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2
    dx = op.grad_x(tval, gy)
    assert rel_l2(dx.cpu().numpy(), O.csr_spmm_t(m, m, rp, col, val, gy.cpu().numpy())) <= RTOL_L2
    dval = op.grad_val(gy, x)
    assert rel_l2(dval.cpu().numpy(), O.csr_sddmm(m, m, rp, col, gy.cpu().numpy(),
                                                   x.cpu().numpy())) <= RTOL_L2


@pytest.mark.parametrize("sigma", [11, 27])
def test_tile_fixup_row_spans(sblas_lib, cuda, sigma):
    """Rows over 2, 3, 9, 10, 11 and 40 tiles, rows that start or end at a tile
    boundary, one matrix and several in a launch."""
    from hpda_sblas_pnnl_gb300 import ops
    tile = 128 * sigma
    lengths = [3, tile - 3, tile, 1, 0, 2 * tile - 1, 5, 9 * tile, 10 * tile - 5, 11 * tile + 2, 0,
               0, 40 * tile, 7, 3 * tile + 1, tile, tile, 2, 2 * tile]
    n = 4000
    (rp, col, val), dev = csr_of_lengths(lengths, n, sigma, cuda)
    m = len(lengths)
    rng = np.random.default_rng(sigma)
    x, y0 = rng.standard_normal(n), rng.standard_normal(m)
    ref = O.csr_spmv(m, n, rp, col, val, x, y0.copy(), 1.5, -0.5)
    tx = torch.from_numpy(x).to(cuda)
    y = torch.from_numpy(y0).to(cuda)
    ops.CsrPlan(*dev, n=n, sigma=sigma)(tx, y, 1.5, -0.5)
    assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2
    if sigma != 11:
        return                    # several matrices in a launch: one compiled shape
    ys = [torch.from_numpy(y0).to(cuda) for _ in range(3)]
    ops.BatchPlan([dev] * 3, [tx] * 3, ys, 1, alpha=1.5, beta=-0.5)()
    for y in ys:
        assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2


@pytest.mark.parametrize("kernel", [1, 2, 3])
@pytest.mark.parametrize("lengths", [[1], [0, 0, 1408, 0], [1407, 1, 1], [1409], [0] * 700 + [3],
                                     [2, 0, 9000, 1, 0, 0, 40, 1500, 7] * 3], ids=str)
@pytest.mark.parametrize("extra", [0, 1, 1408, 4000])
def test_spmspv_leaves_out_zero_x(sblas_lib, cuda, kernel, lengths, extra):
    """Zeros and negative zeros of x meet infinite and NaN values; rows that
    cross tiles, empty rows, more rows than a tile holds; col and val longer
    than the row pointer says."""
    from hpda_sblas_pnnl_gb300 import ops
    n = 300
    (rp, col, val), (trp, _, _) = csr_of_lengths(lengths, n, 5, cuda)
    m, nnz = len(lengths), int(rp[-1])
    rng = np.random.default_rng(nnz)
    x = rng.standard_normal(n)
    x[rng.random(n) < 0.5] = 0.0
    x[rng.random(n) < 0.1] = -0.0
    dead = x[col] == 0.0
    val[dead] = rng.choice([np.inf, -np.inf, np.nan, 2.0], int(dead.sum()))
    y0 = rng.standard_normal(m)
    orp, oc, ov = O.csr_filter_x(m, rp, col, val, x)
    long_col = torch.from_numpy(np.concatenate([col, np.zeros(extra, np.int32)])).to(cuda)
    long_val = torch.from_numpy(np.concatenate([val, np.full(extra, 3.0)])).to(cuda)
    tx = torch.from_numpy(x).to(cuda)
    for alpha, beta in ((1.0, 0.0), (1.5, 0.0), (1.5, -0.5)):
        y = torch.from_numpy(y0).to(cuda)
        ops.spmspv(trp, long_col, long_val, tx, y, alpha, beta, kernel=kernel)
        ref = O.csr_spmv(m, n, orp, oc, ov, x, y0.copy(), alpha, beta)
        assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2
        if kernel == 1:
            continue
        y = torch.from_numpy(y0).to(cuda)
        ops.spmspv(trp, long_col, None, tx, y, alpha, beta, kernel=kernel)
        ref = O.csr_spmv(m, n, orp, oc, np.ones(len(oc)), x, y0.copy(), alpha, beta)
        assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2


@pytest.mark.parametrize("nnz", [1, 31, 1023, 1024, 1025, 40_000, (1 << 19) - 1, (1 << 19) + 1,
                                 (1 << 22) - 1, (1 << 22) + 4097])
@pytest.mark.parametrize("m,n", [(1, 1), (1, 900), (2, 3_000_000), (2048, 7), (2049, 300),
                                 (300_000, 1), (5_000_000, 20_000)])
def test_sorts_at_tile_and_digit_edges(sblas_lib, cuda, nnz, m, n):
    """CSC -> CSR and the transpose at the edges of the sort's tiles (1024,
    2048, 4096 entries), digit widths and passes (rows up to 1, 2, 2048, 2049,
    5M), with few and many, empty and very long columns: whole numbers and
    values equal to numpy's stable sort."""
    from hpda_sblas_pnnl_gb300 import ops
    rng = np.random.default_rng(nnz + m)
    cols = rng.integers(0, n, nnz)
    cols[: nnz // 3] = n // 2                      # one long column
    cols = np.sort(cols)
    rows = rng.integers(0, m, nnz).astype(np.int32)
    rows[nnz // 2:] = np.where(rng.random(nnz - nnz // 2) < 0.5, m - 1, rows[nnz // 2:])
    val = rng.standard_normal(nnz)
    colptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int32)
    order = np.argsort(rows, kind="stable")
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))])
    tc, tr, tv = (torch.from_numpy(a).to(cuda) for a in (colptr, rows, val))
    rp, c, v = ops.csc_to_csr(m, n, tc, tr, tv)
    assert np.array_equal(rp.cpu().numpy(), rowptr)
    assert np.array_equal(c.cpu().numpy(), cols[order])
    assert np.array_equal(v.cpu().numpy(), val[order])
    # the same arrays as a CSR matrix of n rows: its transpose
    rp, c, perm = ops.csr_transpose(n, m, tc, tr)
    assert np.array_equal(rp.cpu().numpy(), rowptr)
    assert np.array_equal(c.cpu().numpy(), cols[order])
    assert np.array_equal(perm.cpu().numpy(), order)


@pytest.mark.parametrize("lengths", [[1], [0, 64, 65, 0, 512, 513], [8192], [8193], [0] * 3000 + [5],
                                     [7, 0, 63, 64, 65, 511, 512, 513, 4097, 1] * 7,
                                     [2] * 16_384, [2] * 16_385, [9] * 3641, [9] * 14_563,
                                     [5, 0, 700, 3] * 40], ids=lambda v: f"{len(v)}x{max(v)}")
def test_small_matrices(sblas_lib, cuda, lengths):
    """Rows at the lengths where lanes, warps and the CTA change over, sizes on
    both sides of the small path's limits, every value kind, alpha and beta,
    kernels 1 to 3, per call and analysed, an explicit tile shape, x zeros
    left out, NaN in y with beta = 0."""
    from hpda_sblas_pnnl_gb300 import ops
    n = 3000
    (rp, col, val), (trp, tcol, tval) = csr_of_lengths(lengths, n, 3, cuda)
    m = len(lengths)
    rng = np.random.default_rng(m)
    x = rng.standard_normal(n)
    tx = torch.from_numpy(x).to(cuda)
    y0 = rng.standard_normal(m)
    vals = {"f64": (tval, val), "f32": (tval.float(), tval.float().double().cpu().numpy()),
            "pattern": (None, np.ones(len(val)))}
    for form, (tv, v) in vals.items():
        plan = ops.CsrPlan(trp, tcol, tv, n=n)
        for alpha, beta in ((1.0, 0.0), (1.5, 0.0), (1.5, -0.5)):
            start = np.full(m, np.nan) if beta == 0.0 else y0
            ref = O.csr_spmv(m, n, rp, col, v, x, np.where(np.isnan(start), 0.0, start), alpha, beta)
            got = {}
            for kernel in (1, 2, 3) if form == "f64" else (2, 3):
                y = torch.from_numpy(start).to(cuda)
                got[f"kernel {kernel}"] = ops.csrmv(trp, tcol, tv, tx, y, alpha, beta, kernel=kernel)
            got["plan"] = plan(tx, torch.from_numpy(start).to(cuda), alpha, beta)
            got["sigma"] = ops.csrmv(trp, tcol, tv, tx, torch.from_numpy(start).to(cuda), alpha,
                                     beta, sigma=15)
            for what, y in got.items():
                assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2, (form, what, alpha, beta)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("nnz", [(1 << 19) - 1, 1 << 19, (1 << 22) - 1, 1 << 22, (1 << 24) + 5])
def test_host_call_chunks(sblas_lib, cuda, pinned, nnz):
    """Host arrays on both sides of each chunk count, pageable and pinned, a row
    over several chunks, empty rows at both ends, beta with y read in."""
    from hpda_sblas_pnnl_gb300 import api
    rng = np.random.default_rng(nnz)
    m, n = nnz // 50, 40_000
    lengths = rng.multinomial(nnz - nnz // 3, np.ones(m) / m)
    lengths[:3] = 0
    lengths[-4:] = 0
    lengths[m // 3] += nnz - int(lengths.sum())
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = rng.integers(0, n, nnz).astype(np.int32)
    val, x, y0 = rng.standard_normal(nnz), rng.standard_normal(n), rng.standard_normal(m)
    y = y0.copy()
    if pinned:
        keep = [torch.from_numpy(a).pin_memory() for a in (val, rp, col, x, y)]
        val, rp, col, x, y = (t.numpy() for t in keep)
    for alpha, beta in ((1.0, 0.0), (1.5, -0.5)):
        y[:] = y0
        api.spMV_mgpu_v1(m, n, nnz, alpha, val, rp, col, x, beta, y)
        ref = O.csr_spmv(m, n, np.array(rp), np.array(col), np.array(val), np.array(x), y0.copy(),
                         alpha, beta)
        assert rel_l2(y, ref) <= RTOL_L2


@pytest.mark.parametrize("nnz", [1, 3, 4, 5, 127, 4095, 4096, 4097, 8191, 131_073, 300_001])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("m", [1, 700, 200_000])
def test_coo_row_pointer_and_partition(sblas_lib, cuda, nnz, offset, m):
    """Sorted triplets at the edges of the row-pointer kernel's CTAs and of the
    tiles, aligned and not, rows missing at both ends and between, one row over
    many tiles: the row pointer equal, products within the bar, every shape."""
    from hpda_sblas_pnnl_gb300 import ops
    rng = np.random.default_rng(nnz + m)
    n = 500
    rows = np.sort(rng.integers(m // 3, max(m - m // 5, m // 3 + 1), nnz)).astype(np.int32)
    rows[nnz // 4: nnz // 2] = rows[nnz // 4]
    rows = np.sort(rows)
    col = rng.integers(0, n, nnz).astype(np.int32)
    val, x = rng.standard_normal(nnz), rng.standard_normal(n)
    y0 = rng.standard_normal(m)
    pad = torch.zeros(nnz + offset, dtype=torch.int32, device=cuda)
    pad[offset:] = torch.from_numpy(rows).to(cuda)
    tr = pad[offset:]
    tc, tv, tx = (torch.from_numpy(a).to(cuda) for a in (col, val, x))
    ref = O.coo_spmv(m, n, rows, col, val, x, y0.copy(), 1.5, -0.5)
    for sigma in (0, 11, 27):
        y = torch.from_numpy(y0).to(cuda)
        work = torch.full((m + 1,), -7, dtype=torch.int32, device=cuda)
        ops.coomv(tr, tc, tv, tx, y, 1.5, -0.5, rowptr_work=work, sigma=sigma)
        assert rel_l2(y.cpu().numpy(), ref) <= RTOL_L2
        want = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=m))])
        assert np.array_equal(work.cpu().numpy(), want)


@pytest.mark.parametrize("nnz", [1 << 20, (1 << 25) - 3, 1 << 25, (1 << 25) + 5])
def test_csc_values_direct_and_staged(sblas_lib, cuda, nnz):
    """An analysed CSC pattern on both sides of the size from which its values
    are staged: new values, bound values, against the one-shot product."""
    from hpda_sblas_pnnl_gb300 import ops
    g = torch.Generator(device=cuda)
    g.manual_seed(nnz)
    m, n = nnz // 40, nnz // 30
    rows = torch.randint(0, m, (nnz,), generator=g, device=cuda, dtype=torch.int32)
    cols = torch.sort(torch.randint(0, n, (nnz,), generator=g, device=cuda)).values
    colptr = torch.zeros(n + 1, dtype=torch.int64, device=cuda)
    colptr[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
    colptr = colptr.int()
    x = torch.randn(n, generator=g, dtype=torch.float64, device=cuda)
    plan = ops.CscPlan(m, colptr, rows)
    for _ in range(2):
        val = torch.randn(nnz, generator=g, dtype=torch.float64, device=cuda)
        ref = torch.zeros(m, dtype=torch.float64, device=cuda).index_add_(0, rows.long(), val * x[cols])
        once = ops.cscmv(colptr, rows, val, x, torch.empty_like(ref))
        assert float((once - ref).norm() / ref.norm()) <= RTOL_L2
        y = plan(val, x, torch.empty_like(ref))
        assert torch.equal(y, once)
        plan.bind(val)
        assert torch.equal(plan(None, x, torch.empty_like(ref)), once)
