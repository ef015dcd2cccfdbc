"""The chained GEMM launch's task order can always make progress: host model, random interleavings (CPU)."""
import random

import pytest

from ittai_b200.gemm_chain import INPUTS, STAGES, chain_tasks, simulate, simulate_pair

SIGLIP_LAYER = [768, 3072, 768, 2304]          # out-proj, fc1, fc2, next QKV


def test_task_order_is_gemm_then_row_block_then_column():
    t = chain_tasks(700, [512, 256])
    assert t[:7] == [(0, 0, 0), (0, 0, 1), (0, 1, 0), (0, 1, 1), (0, 2, 0), (0, 2, 1), (1, 0, 0)] and len(t) == 9


@pytest.mark.parametrize("m,ns,clusters", [(12544, SIGLIP_LAYER, 74), (12544, [768, 2304], 74), (700, SIGLIP_LAYER, 74),
                                            (300, [256, 256, 256, 256], 3), (2048, [256, 1024], 5), (12544, SIGLIP_LAYER, 33)])
def test_random_interleavings_never_deadlock(m, ns, clusters):
    for seed in range(5):
        r = simulate(m, ns, clusters, random.Random(seed))
        assert r["steps"] == 2 * r["tasks"]


def test_a_task_that_waits_for_a_later_task_is_reported():
    """The model itself: with the GEMMs' dependency reversed by hand (first GEMM waiting on a second one that is listed after
    it) no cluster can move, and the simulator says so instead of spinning."""
    import ittai_b200.gemm_chain as gc
    tasks = gc.chain_tasks(512, [256, 256])
    real = gc.chain_tasks
    try:
        gc.chain_tasks = lambda m, ns: [(1 - g, tm, tn) for g, tm, tn in tasks]      # GEMM 1's tiles first
        with pytest.raises(RuntimeError, match="deadlock"):
            gc.simulate(512, [256, 256], 2, random.Random(0))
    finally:
        gc.chain_tasks = real


def _staging_conflicts(residual, drain_at_step):
    """Chunks of consecutive tiles (``residual[i]``: tile i adds one) as an epilogue warp of the chain kernel stages them, no tile's
    stores awaited at its end: (tile, chunk) pairs written while a bulk store issued before may still read the same staging tile."""
    unread, bad, cc, one_buffer = [], [], 0, False         # staging tiles of the stores that may still be reading, oldest first
    for tile, has_res in enumerate(residual):
        if has_res:
            unread.clear()                                 # staging tiles 1 and 2 become load targets
        for ch in range(4):
            keep = 0 if has_res or (drain_at_step and one_buffer and ch == 0) else 2
            del unread[:max(0, len(unread) - keep)]
            buf = 0 if has_res else cc % 3
            if buf in unread:
                bad.append((tile, ch))
            unread.append(buf)
            cc += 1
        one_buffer = has_res
    return bad


@pytest.mark.parametrize("before", range(6))
def test_staging_tiles_are_read_before_they_are_written_again(before):
    """A layer's order (residual, none, residual, none) with 0 to 5 tiles ahead of it; without the wait at the step from a tile with a
    residual to one without, every third position writes a tile that is still read."""
    order = [False] * before + [True] * 2 + [False] * 3 + [True, False, True, False, False]
    assert not _staging_conflicts(order, True)
    assert any(_staging_conflicts([False] * n + order, False) for n in range(3))


@pytest.mark.parametrize("m,ns,clusters", [(12544, SIGLIP_LAYER, 74), (2048, [256, 1024], 5), (300, [256, 256, 256, 256], 3)])
def test_tiles_counted_late_never_deadlock(m, ns, clusters):
    """Finished tiles told to the publishing warp only with the next one, loads up to the longest lead ahead."""
    for seed in range(3):
        for ahead in (2, 2 + STAGES):
            r = simulate(m, ns, clusters, random.Random(seed), ahead=ahead, late=True)
            assert r["steps"] == 2 * r["tasks"]


@pytest.mark.parametrize("n_kb", [1, 2, 3, 4, 12, 48])
def test_an_inputs_barrier_is_not_completed_again_before_it_was_looked_at(n_kb):
    """K = 64 is the longest lead: two accumulators and five stages.  The ring of four barriers that K >= 192 would do with fails
    there and at K = 128."""
    lead = max(simulate_pair([n_kb] * 40, random.Random(seed)) for seed in range(200))
    assert lead <= STAGES + 2 < INPUTS
    if n_kb == 1:
        assert lead == STAGES + 2
    if n_kb <= 2:
        with pytest.raises(RuntimeError, match="completed again"):
            for seed in range(200):
                simulate_pair([n_kb] * 40, random.Random(seed), inputs=4)


def test_chains_run_where_they_were_faster():
    """Both sides of the two lines of the rule at the sizes that were measured."""
    from ittai_b200.siglip.kernel import chain_pays
    vit, so400m = ((2304, 768), (768, 768), (3072, 768), (768, 3072)), ((3840, 1280), (1280, 1280), (4352, 1280), (1280, 4352))
    for rows, want in ((1024, False), (2156, False), (4096, False), (4097, True), (6272, True), (9408, True), (12544, False), (16384, True)):
        assert chain_pays(rows, vit, 148) == want, rows
    for rows, want in ((1458, False), (2187, False), (2304, False), (2305, True), (5832, True)):
        assert chain_pays(rows, so400m, 148) == want, rows
