"""One CTA per matrix or the step kernels, FP64 orders 113 to 256: the batch has to fill its
last round of one matrix per SM.  Both sides of the line run as named (launches counted)
and are exact, at the orders of the 16-column panels' and thread blocks' edges."""
import ctypes as C

import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300 import lib as L
from tests.util import to_storage

pytestmark = pytest.mark.gpu


def _updates(call):
    lib = L.load()
    assert lib.magma_lu_timing_start(L.KERNEL_CLASSES["gemm"], 4096) == 0
    call()
    n, dropped, ms = C.c_int(), C.c_int(), C.c_double()
    assert lib.magma_lu_timing_stop(C.byref(n), C.byref(dropped), C.byref(ms)) == 0
    return n.value


# extra matrices above `rounds` whole rounds of one per SM, and whether one CTA takes them
@pytest.mark.parametrize("m,n,rounds,extra,one", [(255, 255, 1, 0, True), (256, 256, 1, 0, True), (256, 256, 1, 1, False), (256, 256, 2, 0, True),
                                                  (255, 255, 1, 60, False), (256, 40, 1, 0, True), (40, 256, 1, 0, True), (215, 215, 1, 1, False),
                                                  (192, 192, 1, 1, False), (160, 160, 1, 1, False), (160, 160, 1, 60, True), (144, 144, 1, 1, True),
                                                  (129, 129, 1, 1, True), (200, 200, 0, 3, False)])
def test_both_sides_of_the_line(cuda, m, n, rounds, extra, one):
    batch = rounds * torch.cuda.get_device_properties(cuda).multi_processor_count + extra
    rng = np.random.default_rng(m * 3 + n + batch)
    A = rng.uniform(-1, 1, (5, m, n))
    A[1, :, min(m, n) // 2] = 0.0
    A[2] = rng.integers(-2, 3, (m, n))
    A[3, m // 2, :] = np.nan
    A[4] *= 1e-310
    S = to_storage(A, m + 3)
    S[:, :, m:] = 9.0
    idx = np.arange(batch) % 5
    dS = torch.from_numpy(np.ascontiguousarray(S[idx])).to(cuda)
    out = {}
    assert (_updates(lambda: out.update(r=mg.getrf_batched(dS, m))) == 0) == one
    torch.cuda.synchronize()
    rp, ri = oracle.dgetrf_batched(S, m)
    assert np.array_equal(out["r"][1].cpu().numpy(), ri[idx])
    assert np.array_equal(out["r"][0].cpu().numpy()[:, :min(m, n)], rp[idx][:, :min(m, n)])
    assert np.array_equal(dS.cpu().numpy(), S[idx], equal_nan=True)
