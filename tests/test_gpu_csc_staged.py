"""The staged executor of analysed CSC patterns (above 2^25 entries): the values
regrouped by bucket of row positions, then gathered bucket by bucket.  Rows and
columns far longer than a bucket, tiles that lie in one bucket, a bucket with
one entry, alpha and beta, other values, bound values.  The values that reach
the tile kernel are moved, not computed: the bits of the one-shot product,
whose sort carries them; and within 1e-12 relative L2 of plain sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu

RTOL_L2 = 1e-12
LIMIT = 1 << 25                 # entries up to which values are gathered directly
BUCKET = 1 << 20


def pattern(kind, m, n, nnz, cuda, g):
    """rows, cols of the entries in CSC order (rows in any order in a column)"""
    if kind == "random":
        cols = torch.sort(torch.randint(0, n, (nnz,), generator=g, device=cuda)).values
        rows = torch.randint(0, m, (nnz,), generator=g, device=cuda)
    elif kind == "in order":    # CSC order is row order: a tile lies in one bucket
        cols = torch.arange(nnz, device=cuda) * n // nnz
        rows = torch.arange(nnz, device=cuda) * m // nnz
    else:                       # row order is CSC order backwards
        cols = torch.arange(nnz, device=cuda) * n // nnz
        rows = m - 1 - torch.arange(nnz, device=cuda) * m // nnz
    return rows, cols


@pytest.mark.parametrize("kind,m,n,nnz", [
    ("random", 3, 12_000_000, LIMIT + BUCKET + 1),      # three rows over all buckets
    ("random", 700_000, 5, LIMIT + BUCKET + 1),         # five columns over all buckets
    ("random", 1500, 4000, LIMIT + 1),                  # a last bucket with one entry
    ("random", 2_000_000, 3_000_000, LIMIT + 4097),
    ("in order", 1, 1_000_000, LIMIT + BUCKET - 1),
    ("in order", 5_000_000, 5_000_000, LIMIT + 2047),
    ("backwards", 3_000_000, 1_000_000, LIMIT + BUCKET),
    ("backwards", LIMIT + 9, LIMIT + 9, LIMIT + 9),     # one entry in every row and column
])
def test_staged_values(sblas_lib, cuda, kind, m, n, nnz):
    from hpda_sblas_pnnl_gb300 import ops
    # the staged layout holds one more index per entry: a moved limit shows here
    assert (sblas_lib.sblas_cscmv_workspace_bytes(m, n, nnz) -
            sblas_lib.sblas_cscmv_workspace_bytes(m, n, LIMIT)) >= 4 * nnz
    g = torch.Generator(device=cuda)
    g.manual_seed(nnz + m)
    rows, cols = pattern(kind, m, n, nnz, cuda, g)
    colptr = torch.zeros(n + 1, dtype=torch.int32, device=cuda)
    colptr[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0).int()
    x = torch.randn(n, generator=g, dtype=torch.float64, device=cuda)
    y0 = torch.randn(m, generator=g, dtype=torch.float64, device=cuda)
    ri = rows.int()
    plan = ops.CscPlan(m, colptr, ri)
    for alpha, beta in ((0.5, -1.25), (1.0, 0.0)):
        val = torch.randn(nnz, generator=g, dtype=torch.float64, device=cuda)
        start = y0 if beta else torch.full_like(y0, float("nan"))
        once = ops.cscmv(colptr, ri, val, x, start.clone(), alpha, beta)
        assert torch.equal(plan(val, x, start.clone(), alpha, beta), once)
        plan.bind(val)
        assert torch.equal(plan(None, x, start.clone(), alpha, beta), once)
        prod = val * x[cols]
        if m <= 3:
            ref = torch.stack([prod[rows == r].sum() for r in range(m)])
        else:
            ref = torch.zeros_like(y0).index_add_(0, rows, prod)
        ref = alpha * ref + (beta * y0 if beta else 0.0)
        assert float((once - ref).norm() / ref.norm()) <= RTOL_L2
