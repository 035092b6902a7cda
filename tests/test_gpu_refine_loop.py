"""The refinement's host loop on the GPU: results and iteration counts of batches that end
at every number of iterations equal the oracle's (which runs every test), a matrix that
never converges costs few questions, and threads that share a queue do not share an answer."""
import threading

import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle
from magma_gb300 import lib as L
from magma_gb300.batched import Queue
from magma_gb300.testing import svd_batch_torch

pytestmark = pytest.mark.gpu


def _storage(kappas, n, seed):
    A = svd_batch_torch(len(kappas), n, kappas, seed, device="cpu").numpy()
    return np.ascontiguousarray(A.transpose(0, 2, 1))


@pytest.mark.parametrize("kappas", [[2.0], [1e3] * 3, [1e5, 1e1], [3e6, 1e2], [1e7, 1e4, 1e6], [2e7], [1e12, 1e2], [1e12] * 2])
@pytest.mark.parametrize("itermax", [30, 4, 9])
def test_every_iteration_count(cuda, kappas, itermax):
    S = _storage(kappas, 64, 7)
    B = np.random.default_rng(3).uniform(-1, 1, (len(kappas), 2, 64))
    X, ipiv, info, iters = mg.dsgesv_batched(torch.from_numpy(S.copy()).to(cuda), torch.from_numpy(B).to(cuda), itermax=itermax)
    torch.cuda.synchronize()
    rS = S.copy()
    rX, _, rinfo, riters = oracle.dsgesv_batched(rS, B, itermax=itermax)
    assert np.array_equal(iters.cpu().numpy(), riters)
    assert np.array_equal(info.cpu().numpy(), rinfo)
    assert np.array_equal(X.cpu().numpy(), rX)


def test_a_matrix_that_never_converges_costs_few_questions(cuda):
    S = _storage([1e2] * 15 + [1e13], 33, 5)
    B = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, (16, 2, 33))).to(cuda)
    count = {}
    for fallback in (False, True):
        before = L.load().magma_lu_launch_count()
        _, _, _, iters = mg.dsgesv_batched(torch.from_numpy(S.copy()).to(cuda), B, fallback=fallback)
        torch.cuda.synchronize()
        count[fallback] = L.load().magma_lu_launch_count() - before
        assert int(iters[15]) == -31
    # the questions, and the FP64 solve of one matrix: compaction, factorisation, solve, info
    assert count[True] - count[False] <= 4 + 6


def test_threads_on_one_queue(cuda):
    q = Queue(cuda.index or 0, torch.cuda.current_stream(cuda).cuda_stream)
    cases = [([1e6, 1e1], 11), ([1e1], 12), ([1e12, 1e2], 13), ([1e4] * 3, 14)]
    got, errors = {}, []

    def work(kappas, seed):
        try:
            S = _storage(kappas, 48, seed)
            B = np.random.default_rng(seed).uniform(-1, 1, (len(kappas), 1, 48))
            for _ in range(8):
                dS, dB = torch.from_numpy(S.copy()).to(cuda), torch.from_numpy(B).to(cuda)
                X, _, info, iters = mg.dsgesv_batched(dS, dB, queue=q)
                torch.cuda.current_stream().synchronize()
                rX, _, rinfo, riters = oracle.dsgesv_batched(S.copy(), B)
                assert np.array_equal(iters.cpu().numpy(), riters) and np.array_equal(X.cpu().numpy(), rX)
            got[seed] = True
        except BaseException as e:                 # noqa: BLE001  (reported below)
            errors.append(e)
    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert len(got) == len(cases)
