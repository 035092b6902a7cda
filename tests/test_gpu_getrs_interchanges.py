"""The interchanges of the blocked solves, 32 at a time: orders at the edges of the blocks,
targets that repeat, and sequences no factorisation makes (targets above the diagonal),
both directions, through getrs and the variable-size solve.  Identical to the oracle, which
swaps row by row."""
import numpy as np
import pytest
import torch

import magma_gb300 as mg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("n,nrhs", [(33, 1), (64, 3), (95, 9), (129, 17), (600, 4), (2049, 2)])
def test_interchange_sequences(cuda, n, nrhs, trans, dtype):
    rng = np.random.default_rng(n + nrhs)
    k = np.arange(n)
    piv = np.stack([k + (rng.random(n) * (n - k)).astype(np.int64), np.full(n, n - 1), np.minimum(k + 1, n - 1),
                    np.maximum(k, (k // 32) * 32 + 31).clip(max=n - 1), rng.integers(0, n, n), k[::-1]]).astype(np.int32) + 1
    S = (rng.uniform(-1, 1, (len(piv), n, n)) / n).astype(dtype)
    S[:, k, k] = 1
    B = rng.uniform(-1, 1, (len(piv), nrhs, n)).astype(dtype)
    dB = torch.from_numpy(B).to(cuda)
    mg.getrs_batched(torch.from_numpy(S).to(cuda), torch.from_numpy(piv).to(cuda), dB, trans=trans)
    torch.cuda.synchronize()
    (oracle.sgetrs_batched if dtype == np.float32 else oracle.dgetrs_batched)(S, piv, B, trans)
    assert np.array_equal(dB.cpu().numpy(), B)
