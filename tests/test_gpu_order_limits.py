"""The largest orders of the solves that hold their right-hand sides in shared memory:
exact at the last order they take (the columns' padding and the staged block leave room
for fewer columns per CTA there), refused one order further, where they always were."""
import ctypes as C

import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300 import lib as L
from magma_gb300.batched import Queue, ptr_array
from tests.util import scaled_residual

pytestmark = pytest.mark.gpu

NOT_SUPPORTED = -103


def _factors(n, dtype, seed):
    """One matrix in storage (n, n): small entries around a diagonal near one, so that it
    serves as L and U or as a Cholesky factor, and solves stay in range."""
    rng = np.random.default_rng(seed)
    S = (rng.random((n, n), dtype=np.float32) - np.float32(0.5)).astype(dtype) * dtype(1.0 / n)
    S[np.arange(n), np.arange(n)] = 1 + rng.uniform(-0.25, 0.25, n).astype(dtype)
    return S


# four columns (or eight, above four right-hand sides) beside a 32 x 33 block in 227 KB
@pytest.mark.parametrize("dtype,n,nrhs", [(np.float32, 7132, 5), (np.float32, 7117, 8), (np.float32, 14264, 2),
                                          (np.float64, 3500, 8), (np.float64, 7000, 3)])
def test_getrs_largest_order(cuda, dtype, n, nrhs):
    S = _factors(n, dtype, n)
    rng = np.random.default_rng(nrhs)
    ipiv = (np.arange(n) + (rng.random(n) * (n - np.arange(n))).astype(np.int64)).clip(max=n - 1).astype(np.int32) + 1
    dS, dP = torch.from_numpy(S[None]).to(cuda), torch.from_numpy(ipiv[None]).to(cuda)
    for trans in (False, True):
        B = rng.uniform(-1, 1, (1, nrhs, n)).astype(dtype)
        dB = torch.from_numpy(B).to(cuda)
        mg.getrs_batched(dS, dP, dB, trans=trans)
        torch.cuda.synchronize()
        (oracle.sgetrs_batched if dtype == np.float32 else oracle.dgetrs_batched)(S[None], ipiv[None], B, trans)
        assert np.array_equal(dB.cpu().numpy(), B)
    if n in (7132, 14264, 3500, 7000):
        f = getattr(L.load(), f"magma_{'s' if dtype == np.float32 else 'd'}getrs_batched")
        one = ptr_array(dS)                      # refused on the host, before a pointer is read
        p = C.c_void_p(one.data_ptr())
        assert f(111, n + 1, nrhs, p, n + 1, p, p, n + 1, 1, Queue.current(cuda).handle) == NOT_SUPPORTED


@pytest.mark.parametrize("dtype,n,nrhs", [(np.float32, 14264, 5), (np.float32, 14233, 1), (np.float64, 7000, 2)])
def test_potrs_largest_order(cuda, dtype, n, nrhs):
    S = _factors(n, dtype, n + 1)
    B = np.random.default_rng(n).uniform(-1, 1, (1, nrhs, n)).astype(dtype)
    dS, dB = torch.from_numpy(S[None]).to(cuda), torch.from_numpy(B).to(cuda)
    f = getattr(L.load(), f"magma_{'s' if dtype == np.float32 else 'd'}potrs_batched")
    q = Queue.current(cuda).handle
    pS, pB = ptr_array(dS), ptr_array(dB)
    dA, dX = C.c_void_p(pS.data_ptr()), C.c_void_p(pB.data_ptr())
    assert f(122, n, nrhs, dA, n, dX, n, 1, q) == 0
    torch.cuda.synchronize()
    rB = B[0].copy()
    oracle.potrs(S, rB)
    assert np.array_equal(dB.cpu().numpy()[0], rB)
    if n in (14264, 7000):
        assert f(122, n + 1, nrhs, dA, n + 1, dX, n + 1, 1, q) == NOT_SUPPORTED


@pytest.mark.parametrize("n", [2200, 2193])
def test_gmres_largest_order(cuda, n):
    g = torch.Generator(device=cuda).manual_seed(n)
    A = torch.rand((2, n, n), dtype=torch.float64, device=cuda, generator=g) - 0.5
    A.diagonal(dim1=1, dim2=2).add_(float(np.sqrt(n)))
    B = torch.rand((2, 5, n), dtype=torch.float64, device=cuda, generator=g) - 0.5
    S = A.transpose(1, 2).contiguous()
    X, _, info, iters = mg.dsgesv_batched(S, B, solver="gmres")
    torch.cuda.synchronize()
    assert (info == 0).all() and (iters >= 0).all()
    res = scaled_residual(A.cpu().numpy(), X.transpose(1, 2).cpu().numpy(), B.transpose(1, 2).cpu().numpy())
    assert res.max() <= 30
    if n == 2200:
        S, B = torch.zeros((1, n + 1, n + 1), dtype=torch.float64, device=cuda), torch.zeros((1, 5, n + 1), dtype=torch.float64, device=cuda)
        with pytest.raises(RuntimeError, match=str(NOT_SUPPORTED)):
            mg.dsgesv_batched(S, B, solver="gmres")
