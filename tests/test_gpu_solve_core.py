"""The triangular sweeps behind getrs, getri, potrs and the refinement: orders at
the edges of the 32-row blocks, every split of the right-hand sides over CTAs and
warps, leading dimensions that do and do not allow 16-byte loads, diagonals that
need the division, and the reciprocal on the integer pipes.  Bit-identical to the
CPU oracle (exact comparison, no tolerance)."""
import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from tests.util import to_storage

pytestmark = pytest.mark.gpu


def _solve_both(cuda, S, B, trans, ld):
    f32 = S.dtype == np.float32
    LU = S.copy()
    ipiv, _ = (oracle.sgetrf_batched if f32 else oracle.dgetrf_batched)(LU)
    rB = B.copy()
    (oracle.sgetrs_batched if f32 else oracle.dgetrs_batched)(LU, ipiv, rB, trans)
    n = S.shape[1]
    P = np.full((S.shape[0], n, ld), 7.0, S.dtype)
    P[:, :, :n] = LU
    dB = torch.from_numpy(B).to(cuda)
    mg.getrs_batched(torch.from_numpy(P).to(cuda), torch.from_numpy(ipiv).to(cuda), dB, trans=trans)
    torch.cuda.synchronize()
    return dB.cpu().numpy(), rB


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("n,nrhs,batch,pad", [(33, 1, 3, 0), (48, 2, 200, 1), (63, 3, 400, 0), (64, 8, 330, 2),
                                              (65, 9, 3, 3), (95, 4, 310, 1), (97, 17, 40, 0), (150, 16, 170, 2),
                                              (257, 7, 2, 4), (513, 5, 160, 3)])
def test_getrs_blocks_and_columns(cuda, n, nrhs, batch, pad, trans, dtype):
    rng = np.random.default_rng(n * 31 + nrhs)
    S = to_storage(rng.uniform(-1, 1, (min(batch, 8), n, n)).astype(dtype))
    S = np.ascontiguousarray(S[np.arange(batch) % len(S)])
    B = rng.uniform(-1, 1, (batch, nrhs, n)).astype(dtype)
    got, want = _solve_both(cuda, S, B, trans, n + pad)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("trans", [False, True])
def test_getrs_subnormal_and_special_diagonal(cuda, trans, dtype):
    # diagonal entries whose reciprocal overflows take the division (LAPACK's sfmin
    # rule); zero, infinite and NaN ones propagate as they do in the oracle
    rng = np.random.default_rng(5)
    n, nrhs, batch = 100, 5, 6
    A = np.tril(rng.uniform(-1, 1, (batch, n, n)), -1) * 1e-3 + np.eye(n)
    A = A.astype(dtype)
    tiny = np.finfo(dtype).smallest_subnormal
    for k, v in enumerate([tiny * 3, np.finfo(dtype).tiny / 2, np.finfo(dtype).max, 0.0, np.inf, np.nan]):
        A[k, 40, 40] = v
        A[k, 99, 99] = v
    B = (rng.uniform(-1, 1, (batch, nrhs, n)) * float(tiny) * 100).astype(dtype)
    S = to_storage(A)
    ipiv = np.tile(np.arange(1, n + 1, dtype=np.int32), (batch, 1))
    rB = B.copy()
    (oracle.sgetrs_batched if dtype == np.float32 else oracle.dgetrs_batched)(S, ipiv, rB, trans)
    dB = torch.from_numpy(B).to(cuda)
    mg.getrs_batched(torch.from_numpy(S).to(cuda), torch.from_numpy(ipiv).to(cuda), dB, trans=trans)
    torch.cuda.synchronize()
    assert np.array_equal(dB.cpu().numpy(), rB, equal_nan=True)


def test_reciprocal_correctly_rounded(cuda):
    # A = diag(p) with a last row of ones: the multipliers of the last row are the
    # correctly rounded 1/p.  Random significands, neighbours of powers of two, the
    # edges of the 24-bit approximation, and the exponents at the ends of the range.
    rng = np.random.default_rng(11)
    batch, n = 1024, 65
    frac = rng.integers(0, 1 << 52, (batch, n - 1), dtype=np.uint64)
    frac[100:200] = rng.integers(0, 64, (100, n - 1), dtype=np.uint64)
    frac[200:300] = np.uint64((1 << 52) - 1) - rng.integers(0, 64, (100, n - 1), dtype=np.uint64)
    frac[300:400] = (rng.integers(0, 1 << 23, (100, n - 1), dtype=np.uint64) << np.uint64(29)) + \
        rng.integers(0, 2, (100, n - 1), dtype=np.uint64) * np.uint64((1 << 29) - 1)
    expo = rng.integers(1023, 1100, (batch, n - 1)).astype(np.uint64)
    expo[400:500] = rng.integers(2040, 2047, (100, n - 1)).astype(np.uint64)
    p = (frac | (expo << np.uint64(52))).view(np.float64) * rng.choice([-1.0, 1.0], (batch, n - 1))
    S = np.zeros((batch, n, n))
    i = np.arange(n - 1)
    S[:, i, i] = p
    S[:, :, n - 1] = 1.0
    dS = torch.from_numpy(S).to(cuda)
    ipiv, info = mg.getrf_batched(dS)
    torch.cuda.synchronize()
    assert np.array_equal(ipiv.cpu().numpy(), np.tile(np.arange(1, n + 1), (batch, 1)))
    assert np.array_equal(dS.cpu().numpy()[:, :n - 1, n - 1], 1.0 / p)
