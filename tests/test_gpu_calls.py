"""Forms of the public calls that have to keep their results: optional arrays
left out, empty matrices, workspaces at any alignment, one call after another
on the same workspace.  Whole numbers and moved values equal, FP64 sums
within 1e-12 relative L2."""
import ctypes as C

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
