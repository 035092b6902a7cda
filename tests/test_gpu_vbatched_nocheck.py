"""The unchecked variable-size entries: a negative number of right-hand sides means none
for that matrix; its factors are those of the matrix, and the others are solved."""
import ctypes as C

import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300 import lib as L
from magma_gb300.batched import Queue, _vp

pytestmark = pytest.mark.gpu


def test_negative_right_hand_sides(cuda):
    lib, q = L.load(), Queue.current(cuda)
    rng = np.random.default_rng(4)
    ns, rs = [100, 40, 64, 100, 33], [2, -1, -3, 3, -100]
    As = [rng.uniform(-1, 1, (n, n)) for n in ns]
    Bs = [rng.uniform(-1, 1, (3, n)) for n in ns]
    A = mg.VBatch([a.shape for a in As], ns, torch.float64, cuda).load(As)
    B = mg.VBatch([b.shape for b in Bs], ns, torch.float64, cuda).load(Bs)
    nrhs = torch.tensor(rs, dtype=torch.int32, device=cuda)
    ipiv = torch.zeros((5, 100), dtype=torch.int32, device=cuda)
    dP = ipiv.data_ptr() + torch.arange(5, dtype=torch.int64, device=cuda) * 400
    info = torch.empty((5,), dtype=torch.int32, device=cuda)
    lw = C.c_int(-1)
    f = lib.magma_dgesv_vbatched_max_nocheck_work
    args = (_vp(A.ncols), _vp(nrhs), 100, 3, _vp(A.ptrs), _vp(A.ld), _vp(dP), _vp(B.ptrs), _vp(B.ld), _vp(info))
    assert f(*args, None, C.byref(lw), 5, q.handle) == 0
    work = torch.empty((lw.value,), dtype=torch.uint8, device=cuda)
    assert f(*args, _vp(work), C.byref(lw), 5, q.handle) == 0
    torch.cuda.synchronize()
    for k, n in enumerate(ns):
        rA, rB = As[k][None].copy(), Bs[k][None, :max(rs[k], 0)].copy()
        rp, _ = oracle.dgesv_batched(rA, rB) if rs[k] > 0 else oracle.dgetrf_batched(rA)
        assert np.array_equal(ipiv[k, :n].cpu().numpy(), rp[0]), k
        assert np.array_equal(A.view(k).cpu().numpy(), rA[0]), k
        got = B.view(k).cpu().numpy()
        assert np.array_equal(got[:max(rs[k], 0)], rB[0]) and np.array_equal(got[max(rs[k], 0):], Bs[k][max(rs[k], 0):]), k
