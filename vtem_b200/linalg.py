"""Linear algebra of the decode path (reference: ``vtem/utils/linalg.py``)."""
from __future__ import annotations

import numpy as np
import torch

from . import _abi
from ._abi import call, dptr, stream_ptr

F64 = torch.float64

# below this size the low-rank solve's steps (0.7 ms at n = 500, against 5.5 for
# the eigendecomposition) save little and a refusal costs most (at n = 300 0.1 to
# 0.4 ms of 3.3)
PSD_MIN_SIZE = 256


def solve_eq_sym(G, q, rcond=1e-8, return_kept=False):
    """Solve G c = q for symmetric G by pseudoinversion, dropping singular
    values at or below ``rcond * s_0`` (linalg.py:591-631).  As in the
    reference, G may be destroyed.  Only G's lower triangle is read.

    A positive semidefinite G of low rank (a spike Gram with more intervals
    than the Dirichlet space has dimensions) is solved through its pivoted
    Cholesky factor where no eigenvalue lies near the truncation; any other G
    by its eigendecomposition, in place."""
    if not isinstance(G, torch.Tensor) or not isinstance(q, torch.Tensor):
        raise TypeError("G, q must be CUDA tensors")
    if G.dtype != q.dtype:
        raise TypeError("G,q must be of the same dtype")
    if G.dtype != F64:
        raise TypeError("the plain solve runs in float64")
    if G.dim() != 2 or G.shape[0] != G.shape[1]:
        raise ValueError("G must be square matrix")
    n = G.shape[0]
    if q.numel() != n:
        raise ValueError("number of columns of G must be the same of size of q")
    if not G.is_contiguous():
        raise ValueError("G must be contiguous")
    nbytes = np.zeros(1, np.int64)
    if n >= PSD_MIN_SIZE:
        call("vtb_solve_psd_workspace", n, nbytes.ctypes.data)
        work = torch.empty(int(nbytes[0]), dtype=torch.uint8, device=G.device)
        qv = q.reshape(-1).contiguous()
        c = torch.empty_like(qv)
        kept = torch.zeros(1, dtype=torch.int32, device=G.device)
        accepted = np.zeros(1, np.int32)
        call("vtb_solve_psd", dptr(G), n, dptr(qv), dptr(c), n, float(rcond), dptr(work), int(nbytes[0]), dptr(kept),
             accepted.ctypes.data, stream_ptr())
        if accepted[0]:
            c = c.reshape(q.shape)
            return (c, int(kept.item())) if return_kept else c
        del work
    call("vtb_solve_eq_sym_workspace", n, nbytes.ctypes.data)
    work = torch.empty(int(nbytes[0]), dtype=torch.uint8, device=G.device)
    qv = q.reshape(-1).contiguous()
    c = torch.empty_like(qv)
    kept = torch.zeros(1, dtype=torch.int32, device=G.device)
    call("vtb_solve_eq_sym", dptr(G), n, dptr(qv), dptr(c), n, float(rcond), dptr(work), int(nbytes[0]),
         dptr(kept), stream_ptr())
    c = c.reshape(q.shape)
    if return_kept:
        return c, int(kept.item())
    return c


def norm(A):
    """2-norm of a vector (linalg.py:341-364)."""
    return float(torch.linalg.vector_norm(A.reshape(-1)).item())
