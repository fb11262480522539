"""Calls of the C entry points and of the Python layer that are decided on the
host, before anything is launched (no GPU)."""
import contextlib
import ctypes as C

import numpy as np
import pytest
import torch

from hpda_sblas_pnnl_gb300 import _lib, ops

SBLAS_ERR_ARG, SBLAS_ERR_CUDA = -1, -3


def _addr(a):
    return C.c_void_p(a.ctypes.data)


@pytest.mark.parametrize("missing", ["colptr", "rowidx"])
def test_sort_refuses_an_output_without_its_input(sblas_lib, missing):
    """A null array that a pass of the sort would read is an argument error, not
    a launch (host arrays stand in for device arrays: nothing reads them)."""
    m, n, nnz = 50, 40, 300
    ints = {k: np.zeros(nnz + m + n + 2, np.int32) for k in ("colptr", "rowidx", "rp", "col")}
    val = np.zeros(nnz)
    wb = sblas_lib.sblas_csc_to_csr_workspace_bytes(m, n, nnz)
    work = np.zeros(wb + 256, np.uint8)
    ptr = {k: None if k == missing else _addr(a) for k, a in ints.items()}
    for given in (None, _addr(val)):
        rc = sblas_lib.sblas_csc_to_csr(m, n, nnz, given, ptr["colptr"], ptr["rowidx"], _addr(val),
                                        ptr["rp"], ptr["col"], _addr(work), wb, None)
        assert rc == SBLAS_ERR_ARG


@pytest.mark.parametrize("device,index", [(None, 3), ("cuda", 3), ("cuda:1", 1), (2, 2)])
@pytest.mark.parametrize("form", [lambda d: d, torch.device], ids=["plain", "torch.device"])
def test_check_device_takes_every_form_of_a_device(monkeypatch, device, index, form):
    """A device without an index is the current one; texts and numbers as
    torch.cuda.device takes them (a recorder stands in for the library)."""
    seen = []

    class Lib:
        @staticmethod
        def sblas_stream_status(stream, clear):
            seen.append((stream, clear))
            return 0

    monkeypatch.setattr(_lib, "load", lambda *a, **k: Lib)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "device", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 3, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: ("stream of", i),
                        raising=False)
    if device is None:
        ops.check_device()
    else:
        ops.check_device(form(device), clear=False)
    assert seen == [(("stream of", index), 1 if device is None else 0)]
