"""Panels taller than the register kernels take (FP64 above 512 rows, FP32 above 1024), and
interchanges left of the panel applied in every step (more than 1024 rows), fixed and
variable sizes: zero, subnormal, infinite and NaN columns, ties, padding.  Identical to the
oracle."""
import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300 import lib as L
from magma_gb300.batched import Queue, _vp
from tests.util import to_storage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,m,n", [(np.float64, 513, 65), (np.float64, 1025, 64), (np.float64, 1500, 40), (np.float64, 1100, 1100),
                                       (np.float64, 40, 1300), (np.float32, 1025, 130), (np.float32, 1300, 33), (np.float32, 2050, 70)])
def test_tall_panels(cuda, dtype, m, n):
    rng = np.random.default_rng(m + n)
    A = rng.uniform(-1, 1, (6, m, n)).astype(dtype)
    A[1, :, min(m, n) // 2] = 0.0
    A[2] = rng.integers(-2, 3, (m, n))
    A[3, m // 2, :] = np.nan
    A[4, :, 0] = np.inf
    A[5] *= dtype(1e-310 if dtype == np.float64 else 1e-40)
    S = to_storage(A, m + 3)
    S[:, :, m:] = 9.0
    dS = torch.from_numpy(S).to(cuda)
    ipiv, info = mg.getrf_batched(dS, m)
    torch.cuda.synchronize()
    got = dS.cpu().numpy()
    rp, ri = (oracle.dgetrf_batched if dtype == np.float64 else oracle.sgetrf_batched)(S, m)
    assert np.array_equal(info.cpu().numpy(), ri)
    assert np.array_equal(ipiv.cpu().numpy()[:, :min(m, n)], rp[:, :min(m, n)])
    assert np.array_equal(got, S, equal_nan=True)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_variable_sizes_with_left_interchanges(cuda, dtype):
    rng = np.random.default_rng(12)
    shapes = [(1100, 90), (40, 200), (1030, 33), (700, 700), (1, 64), (1100, 1)]
    ms, mn = [m for m, _ in shapes], [min(s) for s in shapes]
    td = torch.float64 if dtype == np.float64 else torch.float32
    As = [rng.uniform(-1, 1, (n, m + 1)).astype(dtype) for m, n in shapes]
    A = mg.VBatch([a.shape for a in As], ms, td, cuda).load(As)
    ipiv = torch.zeros((len(shapes), max(mn)), dtype=torch.int32, device=cuda)
    dP = ipiv.data_ptr() + torch.arange(len(shapes), dtype=torch.int64, device=cuda) * 4 * max(mn)
    info = torch.empty((len(shapes),), dtype=torch.int32, device=cuda)
    f = getattr(L.load(), "magma_dgetrf_vbatched" if dtype == np.float64 else "magma_sgetrf_vbatched")
    assert f(_vp(A.rows), _vp(A.ncols), _vp(A.ptrs), _vp(A.ld), _vp(dP), _vp(info), len(shapes), Queue.current(cuda).handle) == 0
    torch.cuda.synchronize()
    for k, (m, n) in enumerate(shapes):
        r = As[k][None].copy()
        rp, ri = (oracle.dgetrf_batched if dtype == np.float64 else oracle.sgetrf_batched)(r, m)
        assert info[k].item() == ri[0], k
        assert np.array_equal(ipiv[k, :mn[k]].cpu().numpy(), rp[0, :mn[k]]), k
        assert np.array_equal(A.view(k).cpu().numpy(), r[0]), k
