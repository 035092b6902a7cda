"""Which form of the factorisation runs, and that each form is exact: batches chosen from
the number of SMs so that the two-level form, the band kernel (with and without
interchanges) and the step kernels are the ones that run -- the launches of a kernel class
are counted -- with guard cells around every operand."""
import ctypes as C

import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300 import lib as L
from magma_gb300.batched import Queue, ptr_array
from tests.test_gpu_canary import GUARD, _guarded, _guarded_ints, _ints_intact, _sentinels_intact

pytestmark = pytest.mark.gpu


def _launches(cls, call):
    lib = L.load()
    assert lib.magma_lu_timing_start(L.KERNEL_CLASSES[cls], 4096) == 0
    call()
    n, dropped, ms = C.c_int(), C.c_int(), C.c_double()
    assert lib.magma_lu_timing_stop(C.byref(n), C.byref(dropped), C.byref(ms)) == 0
    return n.value


def _sms(cuda):
    return torch.cuda.get_device_properties(cuda).multi_processor_count


@pytest.fixture
def keep_tables():
    saved = {dt: mg.getrf_batched_tuning(dt) for dt in (torch.float32, torch.float64)}
    yield
    for dt, t in saved.items():
        mg.set_getrf_batched_tuning([v["two_level"] for v in t.values()], [v["band_ctas"] for v in t.values()],
                                    [v["tile64"] for v in t.values()], dt)


def _getrf(cuda, m, n, batch, cls="outer", k=6):
    """FP32 factorisation of `batch` guarded matrices (k different ones), exact; the
    launches of class cls."""
    rng = np.random.default_rng(m * 31 + n * 7 + batch)
    A = rng.uniform(-1, 1, (k, n, m)).astype(np.float32)          # storage (batch, ncols, m)
    A[1, min(m, n) // 2, :] = 0.0
    A[2] = rng.integers(-2, 3, (n, m))
    big, S = _guarded(np.ascontiguousarray(A[np.arange(batch) % k]), 5, cuda)
    bigP, ipiv = _guarded_ints(batch, min(m, n), cuda)
    out = {}
    count = _launches(cls, lambda: out.update(r=mg.getrf_batched(S, m, ipiv=ipiv)))
    torch.cuda.synchronize()
    rA = A.copy()
    rp, ri = oracle.sgetrf_batched(rA, m)
    assert _sentinels_intact(big, n, m) and _ints_intact(bigP, min(m, n))
    idx = np.arange(batch) % k
    assert np.array_equal(S[:, :, :m].cpu().numpy(), rA[idx])
    assert np.array_equal(ipiv.cpu().numpy(), rp[idx][:, :min(m, n)])
    assert np.array_equal(out["r"][1].cpu().numpy(), ri[idx])
    return count


# partial last blocks, columns right of the last block, tall (m > 512: interchanges by four
# rows a thread) and wide matrices, blocks without rows below them
@pytest.mark.parametrize("m,n", [(512, 512), (300, 700), (900, 300), (1024, 1024), (257, 257), (180, 181), (129, 300),
                                 (700, 180), (200, 260), (1000, 999), (65, 640)])
def test_two_level_form_runs_and_is_exact(cuda, m, n):
    batch = -(-_sms(cuda) // -(-(n - 128) // 128))
    blocks = -(-min(m, n) // 128)
    assert _getrf(cuda, m, n, batch) >= blocks - 1 + (n > min(m, n))
    if batch > 1:
        assert _getrf(cuda, m, n, batch - 1) == 0                 # one matrix less: one level


@pytest.mark.parametrize("m,n,two_level,sms", [(400, 400, 1, 1), (512, 390, 1, 2), (389, 640, 1, 1), (289, 289, 0, 1),
                                               (320, 300, 0, 2), (300, 520, 0, 1), (1100, 64, 0, 4)])
def test_band_kernel_runs_and_is_exact(cuda, keep_tables, m, n, two_level, sms):
    # `band_ctas` that allows the band kernel against one that forbids it: with it a step has
    # no launch of its own for the interchanges and U12
    batch = sms * _sms(cuda)
    swaps = {}
    for band in (1, 4):
        mg.set_getrf_batched_tuning([two_level] * 6, [band] * 6, [1] * 6, torch.float32)
        swaps[band] = _getrf(cuda, m, n, batch // 2 + 1, "swap_trsm")
    assert swaps[1] < swaps[4]


@pytest.mark.parametrize("n,two_level", [(300, 0), (400, 1)])
def test_band_kernel_without_interchanges(cuda, keep_tables, n, two_level):
    lib, q, batch = L.load(), Queue.current(cuda).handle, 2 * _sms(cuda)
    rng = np.random.default_rng(n)
    A = rng.uniform(-1, 1, (5, n, n)).astype(np.float32)
    A[:, np.arange(n), np.arange(n)] += 8.0
    A[1, 40, 40] = 0.0                             # (not the pivot's value any more at step 40)
    A[2, 0, 0] = 0.0                               # a zero pivot: info 1
    r, swaps = [a.copy() for a in A], {}
    ri = [oracle.getrf_nopiv(a) for a in r]
    for band in (1, 4):
        mg.set_getrf_batched_tuning([two_level] * 6, [band] * 6, [1] * 6, torch.float32)
        b = batch if band == 1 else 8
        big, S = _guarded(np.ascontiguousarray(A[np.arange(b) % 5]), 3, cuda)
        info = torch.full((b,), -9, dtype=torch.int32, device=cuda)
        dA = ptr_array(S)
        rc = []
        swaps[band] = _launches("swap_trsm", lambda: rc.append(lib.magma_sgetrf_nopiv_batched(
            n, n, C.c_void_p(dA.data_ptr()), n + 3, C.c_void_p(info.data_ptr()), b, q)))
        torch.cuda.synchronize()
        assert rc == [0] and _sentinels_intact(big, n, n)
        got, gi = S[:, :, :n].cpu().numpy(), info.cpu().numpy()
        for k in range(b):
            assert gi[k] == ri[k % 5] and np.array_equal(got[k], r[k % 5], equal_nan=True), k
    assert swaps[1] < swaps[4]


@pytest.mark.parametrize("n,per_sm", [(300, 1), (512, 1), (129, 2)])
def test_refinement_two_level_writes_stay_inside(cuda, n, per_sm):
    batch, nrhs = per_sm * _sms(cuda) // -(-(n - 128) // 128) + 1, 2
    rng = np.random.default_rng(n)
    A = rng.uniform(-1, 1, (4, n, n))
    A[0] = 0.0                                     # singular: the FP64 fallback
    B = rng.uniform(-1, 1, (4, nrhs, n))
    idx = np.arange(batch) % 4
    bigA, S = _guarded(np.ascontiguousarray(A[idx]), 3, cuda)
    bigB, Bd = _guarded(np.ascontiguousarray(B[idx]), 1, cuda)
    bigX, X = _guarded(np.zeros((batch, nrhs, n)), 4, cuda)
    bigP, ipiv = _guarded_ints(batch, n, cuda)
    work = torch.full((mg.dsgesv_workspace_bytes(n, nrhs, batch) + 2 * GUARD * 8,), 90, dtype=torch.uint8, device=cuda)
    need = mg.dsgesv_workspace_bytes(n, nrhs, batch)
    out = {}
    count = _launches("outer", lambda: out.update(r=mg.dsgesv_batched(S, Bd, X=X, ipiv=ipiv, tol=30.0, work=work)))
    torch.cuda.synchronize()
    assert (count > 0) == (n > 176)
    rS = A.copy()
    rX, _, rinfo, riters = oracle.dsgesv_batched(rS, B.copy(), tol=30.0)
    assert _sentinels_intact(bigA, n, n) and _sentinels_intact(bigB, nrhs, n) and _sentinels_intact(bigX, nrhs, n)
    assert _ints_intact(bigP, n) and bool((work[need:] == 90).all())
    assert np.array_equal(out["r"][3].cpu().numpy(), riters[idx]) and np.array_equal(out["r"][2].cpu().numpy(), rinfo[idx])
    assert np.array_equal(X[:, :, :n].cpu().numpy(), rX[idx], equal_nan=True)
    assert np.array_equal(S[:, :, :n].cpu().numpy(), rS[idx])
