"""The bounds-check build through the kernels that its first tests' batches do not reach:
one CTA per matrix at orders up to 256 (fixed and variable sizes, FP64 and FP32), the
two-level form, the triangular sweeps.  The record stays empty and every result equals the
oracle's."""
import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300.batched import ptr_array
from tests.test_gpu_bounds_check import _record, _vp, bc  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu
K = 6                                             # different matrices in a batch


def _clean(lib):
    count, where = _record(lib)
    assert count == 0, f"{count} out-of-bounds accesses, first (site, row, col) = {where}"


def _sms(cuda):
    return torch.cuda.get_device_properties(cuda).multi_processor_count


@pytest.mark.parametrize("dtype,m,n", [(np.float64, 129, 129), (np.float64, 130, 130), (np.float64, 160, 160),
                                       (np.float64, 200, 200), (np.float64, 255, 255), (np.float64, 256, 256),
                                       (np.float64, 256, 40), (np.float64, 40, 256), (np.float64, 7, 200),
                                       (np.float32, 33, 33), (np.float32, 40, 40), (np.float32, 47, 48), (np.float32, 48, 48)])
def test_one_cta_per_matrix_within_bounds(cuda, bc, dtype, m, n):  # noqa: F811
    lib, q = bc
    batch = _sms(cuda)
    rng = np.random.default_rng(m * 3 + n)
    A = rng.uniform(-1, 1, (K, n, m + 3)).astype(dtype)
    A[1, min(m, n) // 2] = 0.0
    A[2] = rng.integers(-2, 3, A[2].shape)
    A[3] *= dtype(1e-310 if dtype == np.float64 else 1e-40)
    idx = np.arange(batch) % K
    S = torch.from_numpy(np.ascontiguousarray(A[idx])).to(cuda)
    ipiv = torch.zeros((batch, min(m, n)), dtype=torch.int32, device=cuda)
    info = torch.zeros((batch,), dtype=torch.int32, device=cuda)
    dA, dP = ptr_array(S), ptr_array(ipiv)
    p = "d" if dtype == np.float64 else "s"
    assert getattr(lib, f"magma_{p}getrf_batched")(m, n, _vp(dA), m + 3, _vp(dP), _vp(info), batch, q) == 0
    torch.cuda.synchronize()
    _clean(lib)
    rp, ri = (oracle.dgetrf_batched if p == "d" else oracle.sgetrf_batched)(A, m)
    assert np.array_equal(S.cpu().numpy(), A[idx])
    assert np.array_equal(ipiv.cpu().numpy(), rp[idx][:, :min(m, n)])
    assert np.array_equal(info.cpu().numpy(), ri[idx])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_variable_sizes_within_bounds(cuda, bc, dtype):  # noqa: F811
    lib, q = bc
    rng = np.random.default_rng(9)
    ns = [1, 2, 15, 16, 17, 31, 33, 48, 64, 65, 127, 128, 129, 200, 255, 256, 240, 0]
    rs = [1, 3, 16, 17, 1, 2, 5, 16, 4, 33, 1, 8, 9, 2, 16, 16, 7, 2]
    td = torch.float64 if dtype == np.float64 else torch.float32
    As = [rng.uniform(-1, 1, (n, n + k % 4)).astype(dtype) for k, n in enumerate(ns)]
    Bs = [rng.uniform(-1, 1, (r, n + k % 3)).astype(dtype) for k, (n, r) in enumerate(zip(ns, rs))]
    A = mg.VBatch([a.shape for a in As], ns, td, cuda).load(As)
    B = mg.VBatch([b.shape for b in Bs], ns, td, cuda).load(Bs)
    offs = np.cumsum([0] + [max(n, 1) for n in ns])
    ipiv = torch.zeros((int(offs[-1]),), dtype=torch.int32, device=cuda)
    dP = ipiv.data_ptr() + torch.tensor(offs[:-1], dtype=torch.int64, device=cuda) * 4
    info = torch.empty((len(ns),), dtype=torch.int32, device=cuda)
    f = lib.magma_dgesv_vbatched if dtype == np.float64 else lib.magma_sgesv_vbatched
    assert f(_vp(A.ncols), _vp(B.ncols), _vp(A.ptrs), _vp(A.ld), _vp(dP), _vp(B.ptrs), _vp(B.ld), _vp(info), len(ns), q) == 0
    torch.cuda.synchronize()
    _clean(lib)
    rp, rinfo = (oracle.dgesv_vbatched if dtype == np.float64 else oracle.sgesv_vbatched)(ns, rs, As, Bs)
    assert np.array_equal(info.cpu().numpy(), rinfo)
    for k, n in enumerate(ns):
        assert np.array_equal(ipiv.cpu().numpy()[offs[k]:offs[k] + n], rp[k]), k
        assert np.array_equal(A.view(k).cpu().numpy(), As[k]) and np.array_equal(B.view(k).cpu().numpy(), Bs[k]), k


@pytest.mark.parametrize("m,n", [(257, 257), (300, 180), (129, 300), (513, 400), (1000, 999), (65, 640), (180, 181)])
def test_two_level_within_bounds(cuda, bc, m, n):  # noqa: F811
    lib, q = bc
    batch = -(-_sms(cuda) // -(-(n - 128) // 128))
    A = np.random.default_rng(m + n).uniform(-1, 1, (K, n, m + 3)).astype(np.float32)
    idx = np.arange(batch) % K
    S = torch.from_numpy(np.ascontiguousarray(A[idx])).to(cuda)
    ipiv = torch.zeros((batch, min(m, n)), dtype=torch.int32, device=cuda)
    info = torch.zeros((batch,), dtype=torch.int32, device=cuda)
    dA, dP = ptr_array(S), ptr_array(ipiv)
    assert lib.magma_sgetrf_batched(m, n, _vp(dA), m + 3, _vp(dP), _vp(info), batch, q) == 0
    torch.cuda.synchronize()
    _clean(lib)
    rp, _ = oracle.sgetrf_batched(A, m)
    assert np.array_equal(S.cpu().numpy(), A[idx])
    assert np.array_equal(ipiv.cpu().numpy(), rp[idx][:, :min(m, n)])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("n,nrhs,batch,pad", [(33, 1, 3, 0), (48, 3, 200, 1), (97, 8, 160, 0), (150, 17, 40, 2), (513, 5, 3, 3)])
def test_solves_within_bounds(cuda, bc, dtype, trans, n, nrhs, batch, pad):  # noqa: F811
    lib, q = bc
    rng = np.random.default_rng(n)
    p = "d" if dtype == np.float64 else "s"
    LU = rng.uniform(-1, 1, (2, n, n)).astype(dtype)
    ipiv, _ = (oracle.dgetrf_batched if p == "d" else oracle.sgetrf_batched)(LU)
    B = rng.uniform(-1, 1, (2, nrhs, n)).astype(dtype)
    idx = np.arange(batch) % 2
    P = np.full((batch, n, n + pad), 7.0, dtype)
    P[:, :, :n] = LU[idx]
    S, X = torch.from_numpy(P).to(cuda), torch.from_numpy(np.ascontiguousarray(B[idx])).to(cuda)
    piv = torch.from_numpy(np.ascontiguousarray(ipiv[idx])).to(cuda)
    dA, dP, dB = ptr_array(S), ptr_array(piv), ptr_array(X)
    f = getattr(lib, f"magma_{p}getrs_batched")
    assert f(112 if trans else 111, n, nrhs, _vp(dA), n + pad, _vp(dP), _vp(dB), n, batch, q) == 0
    torch.cuda.synchronize()
    _clean(lib)
    (oracle.dgetrs_batched if p == "d" else oracle.sgetrs_batched)(LU, ipiv, B, trans)
    assert np.array_equal(X.cpu().numpy(), B[idx])
