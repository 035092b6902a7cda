"""Fewer launches per call: the pointer arrays of a call made by one kernel, on torch's
current stream and on a queue of another stream, and the refinement loop that ends when
no matrix is being refined (results identical to the oracle, which runs every test)."""
import ctypes as C

import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300 import lib as L
from magma_gb300.batched import Queue, _ptrs, ptr_array
from magma_gb300.testing import svd_batch_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 255, 256, 257, 70000])
def test_pointer_arrays(cuda, batch):
    S = torch.empty((batch, 3, 5), dtype=torch.float64, device=cuda)
    P = torch.empty((batch, 4), dtype=torch.int32, device=cuda)[:, :2]      # a stride of its own
    q = Queue.current(cuda)
    a, b, keep = _ptrs(q, S, P)
    torch.cuda.synchronize()
    assert torch.equal(keep[0], ptr_array(S)) and torch.equal(keep[1], ptr_array(P))
    assert a.value == keep[0].data_ptr() and b.value == keep[1].data_ptr()
    assert L.load().magma_lu_set_pointers(None, 7, None, None, 1, q.handle) == -2
    assert L.load().magma_lu_set_pointers(None, 1, None, None, -1, q.handle) == -5
    assert L.load().magma_lu_set_pointers(None, 1, None, None, 0, q.handle) == 0


def test_queue_of_another_stream(cuda):
    rng = np.random.default_rng(1)
    S, B = rng.uniform(-1, 1, (40, 50, 50)), rng.uniform(-1, 1, (40, 2, 50))
    dS, dB = torch.from_numpy(S.copy()).to(cuda), torch.from_numpy(B.copy()).to(cuda)
    side = torch.cuda.Stream(cuda)
    q = Queue(dS.device.index or 0, side.cuda_stream)
    torch.cuda.synchronize()
    info = torch.empty((40,), dtype=torch.int32, device=cuda)
    ipiv = torch.empty((40, 50), dtype=torch.int32, device=cuda)
    arrays = _ptrs(q, dS, ipiv, dB)
    torch.cuda.synchronize()
    assert len(arrays) == 4 and isinstance(arrays[0], C.c_void_p)
    mg.gesv_batched(dS, dB, ipiv, info, queue=q)
    q.sync()
    rS, rB = S.copy(), B.copy()
    oracle.dgesv_batched(rS, rB)
    assert np.array_equal(dB.cpu().numpy(), rB) and np.array_equal(dS.cpu().numpy(), rS)


@pytest.mark.parametrize("kappas,itermax", [([10.0], 30), ([1e2, 1e6], 30), ([1e6], 2), ([1e7], 3), ([1e5], 1), ([1e4], 0)])
def test_refinement_ends_when_converged(cuda, kappas, itermax):
    n, batch = 96, 6
    A = svd_batch_torch(batch, n, [kappas[k % len(kappas)] for k in range(batch)], 3, device="cpu").numpy()
    S = np.ascontiguousarray(A.transpose(0, 2, 1))
    B = np.random.default_rng(2).uniform(-1, 1, (batch, 3, n))
    launches = L.load().magma_lu_launch_count()
    X, ipiv, info, iters = mg.dsgesv_batched(torch.from_numpy(S.copy()).to(cuda), torch.from_numpy(B).to(cuda),
                                             itermax=itermax)
    torch.cuda.synchronize()
    launches = L.load().magma_lu_launch_count() - launches
    rX, ripiv, rinfo, riters = oracle.dsgesv_batched(S.copy(), B, itermax=itermax)
    assert np.array_equal(iters.cpu().numpy(), riters)
    assert np.array_equal(X.cpu().numpy(), rX)
    assert np.array_equal(info.cpu().numpy(), rinfo)
    if itermax == 30 and riters.max() <= 5:
        assert launches < 40                       # 62 for thirty iterations alone
