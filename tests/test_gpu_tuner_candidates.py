"""The autotuners time only settings that launch different kernels, and leave an entry
alone that no setting of its bin changes (it may matter for another batch)."""
import pytest
import torch

import magma_gb300 as mg
from magma_gb300 import lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture
def keep_tables():
    saved = {dt: mg.getrf_batched_tuning(dt) for dt in (torch.float32, torch.float64)}
    vb = {dt: mg.vbatched_tuning(dt) for dt in (torch.float32, torch.float64)}
    yield
    for dt, t in saved.items():
        mg.set_getrf_batched_tuning([v["two_level"] for v in t.values()], [v["band_ctas"] for v in t.values()],
                                    [v["tile64"] for v in t.values()], dt)
    for dt, t in vb.items():
        mg.set_vbatched_tuning([v["nb"] for v in t.values()], [v["tile"] for v in t.values()], dt)


@pytest.mark.parametrize("tile64", [0, 1])
def test_autotuner_keeps_entries_that_no_candidate_reads(cuda, keep_tables, tile64):
    lib = L.load()
    # FP64 orders 48 and 96: one CTA per matrix, no entry is read and nothing is timed
    mg.set_getrf_batched_tuning([1] * 6, [4] * 6, [tile64] * 6, torch.float64)
    before = lib.magma_lu_launch_count()
    t = mg.autotune_getrf_batched(128, 200, torch.float64)
    assert lib.magma_lu_launch_count() == before
    assert [v["tile64"] for v in t.values()] == [tile64] * 6
    # FP32 at a batch too small for two levels: that entry stays; the band kernel runs above
    # order 288 only, so up to 256 nothing is timed
    mg.set_getrf_batched_tuning([tile64] * 6, [4] * 6, [1] * 6, torch.float32)
    before = lib.magma_lu_launch_count()
    t = mg.autotune_getrf_batched(256, 64, torch.float32)
    assert lib.magma_lu_launch_count() == before
    t = mg.autotune_getrf_batched(300, 64, torch.float32)
    assert lib.magma_lu_launch_count() > before
    assert [v["two_level"] for v in t.values()] == [tile64] * 6
    assert [v["band_ctas"] for v in t.values()][:3] == [4] * 3


@pytest.mark.parametrize("nb,candidates", [(32, 2), (16, 2), (8, 4)])
def test_vbatched_autotuner_times_only_different_kernels(cuda, keep_tables, nb, candidates):
    lib = L.load()
    for dt in (torch.float64, torch.float32):
        mg.set_vbatched_tuning([nb] * 8, [1] * 8, dt)
        before = lib.magma_lu_launch_count()
        t = mg.autotune_vbatched(16, dt)
        # the arrays, then tiles 4x4 and 2x2 at width 16 (and the installed 8), twice each:
        # fill, sort, factor
        assert lib.magma_lu_launch_count() - before == 1 + candidates * 2 * 3
        assert t["<=16"]["nb"] in (nb, 16) and t["<=16"]["tile"] in (mg.batched.TILES[1], mg.batched.TILES[2])
