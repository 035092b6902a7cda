"""The batched inverse on both sides of its two forms (few and many CTAs), at the edges of
the 32-row blocks and of a CTA's eight columns.  Identical to the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from magma_gb300 import lib as L
from magma_gb300.batched import Queue, ptr_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,batch", [(1, 2), (8, 1300), (9, 3), (33, 400), (64, 160), (64, 200), (255, 2), (256, 12), (300, 1)])
def test_inverse(cuda, n, batch, dtype):
    p = "d" if dtype == np.float64 else "s"
    rng = np.random.default_rng(n + batch)
    S = rng.uniform(-1, 1, (3, n, n)).astype(dtype)
    piv, _ = (oracle.dgetrf_batched if p == "d" else oracle.sgetrf_batched)(S)
    idx = np.arange(batch) % 3
    dS, dP = torch.from_numpy(np.ascontiguousarray(S[idx])).to(cuda), torch.from_numpy(np.ascontiguousarray(piv[idx])).to(cuda)
    I, info = torch.empty_like(dS), torch.empty((batch,), dtype=torch.int32, device=cuda)
    a, b, c = ptr_array(dS), ptr_array(dP), ptr_array(I)
    vp = lambda t: C.c_void_p(t.data_ptr())
    f = getattr(L.load(), f"magma_{p}getri_outofplace_batched")
    assert f(n, vp(a), n, vp(b), vp(c), n, vp(info), batch, Queue.current(cuda).handle) == 0
    torch.cuda.synchronize()
    want = np.stack([oracle.getri(S[k], piv[k]) for k in range(3)])
    assert np.array_equal(I.cpu().numpy(), want[idx])
