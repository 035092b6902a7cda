"""The factorisation of one matrix by one CTA (orders up to 256): orders around the
16-column panels, the 32-row blocks and the CTA sizes 64, 128 and 256, rectangular
shapes, padding, zero and NaN columns, through the fixed-size and the variable-size
entry points.  Bit-identical to the CPU oracle (exact comparison)."""
import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from tests.util import to_storage

pytestmark = pytest.mark.gpu
BATCH = 160          # one CTA per matrix needs a batch that occupies the SMs


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,n", [(33, 33), (48, 48), (49, 49), (63, 63), (64, 64), (65, 65), (97, 97), (128, 128),
                                 (129, 129), (160, 160), (255, 255), (256, 256), (256, 40), (40, 256), (7, 200),
                                 (200, 7), (130, 65)])
def test_getrf_one_cta_per_matrix(cuda, m, n, dtype):
    rng = np.random.default_rng(m * 7 + n)
    k = 10
    A = rng.uniform(-1, 1, (k, m, n)).astype(dtype)
    A[1, :, min(m, n) // 2] = 0.0                 # a zero column
    A[2] = rng.integers(-2, 3, (m, n))            # ties in the pivot search
    A[3, m // 2, :] = np.nan
    A[4, :, 0] = np.inf
    A[5] *= dtype(1e-310 if dtype == np.float64 else 1e-40)      # subnormal pivots
    S = to_storage(A, m + 3)
    S[:, :, m:] = 9.0
    rS = S.copy()
    ripiv, rinfo = (oracle.dgetrf_batched if dtype == np.float64 else oracle.sgetrf_batched)(rS, m)
    dS = torch.from_numpy(np.ascontiguousarray(S[np.arange(BATCH) % k])).to(cuda)
    ipiv, info = mg.getrf_batched(dS, m)
    torch.cuda.synchronize()
    gS, gi, gp = dS.cpu().numpy(), info.cpu().numpy(), ipiv.cpu().numpy()
    for b in range(BATCH):
        assert gi[b] == rinfo[b % k]
        assert np.array_equal(gp[b, :min(m, n)], ripiv[b % k, :min(m, n)]), b
        assert np.array_equal(gS[b], rS[b % k], equal_nan=True), b


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_gesv_vbatched_edges(cuda, dtype):
    rng = np.random.default_rng(3)
    ns = [1, 2, 15, 16, 17, 31, 33, 48, 64, 65, 127, 128, 129, 200, 255, 256, 240, 0]
    rs = [1, 3, 16, 17, 1, 2, 5, 16, 4, 33, 1, 8, 9, 2, 16, 16, 7, 2]
    As = [rng.uniform(-1, 1, (n, n + k % 4)).astype(dtype) for k, n in enumerate(ns)]
    Bs = [rng.uniform(-1, 1, (r, n + k % 3)).astype(dtype) for k, (n, r) in enumerate(zip(ns, rs))]
    td = torch.float64 if dtype == np.float64 else torch.float32
    A = mg.VBatch([a.shape for a in As], ns, td, cuda).load(As)
    B = mg.VBatch([b.shape for b in Bs], ns, td, cuda).load(Bs)
    ipiv, offs, info = mg.gesv_vbatched(A, B)
    torch.cuda.synchronize()
    rA, rB = [a.copy() for a in As], [b.copy() for b in Bs]
    f = oracle.dgesv_vbatched if dtype == np.float64 else oracle.sgesv_vbatched
    rp, rinfo = f(ns, rs, rA, rB)
    P = ipiv.cpu().numpy()
    assert np.array_equal(info.cpu().numpy(), rinfo)
    for k, n in enumerate(ns):
        assert np.array_equal(P[offs[k]:offs[k] + n], rp[k]), k
        assert np.array_equal(A.view(k).cpu().numpy(), rA[k]), k
        assert np.array_equal(B.view(k).cpu().numpy(), rB[k]), k
