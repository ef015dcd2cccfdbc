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


VIT, SO400M = ((2304, 768), (768, 768), (3072, 768), (768, 3072)), ((3840, 1280), (1280, 1280), (4352, 1280), (1280, 4352))
# us a forward on a B200, chained / one by one, by rows: fixed and variable resolution of one tower, and the large one
MEASURED = [(VIT, {1568: (879, 873), 2048: (902, 876), 2156: (945, 927), 3136: (1066, 1068), 4096: (1139, 1089), 4704: (1196, 1212), 6076: (1424, 1377),
                   6144: (1362, 1315), 6272: (1484, 1704), 9408: (1975, 2095), 12152: (2573, 2581), 12288: (2525, 2523), 12348: (2565, 2562),
                   12544: (2676, 2640), 12740: (2716, 2891), 15680: (3312, 3380), 16384: (3397, 3485), 18228: (3879, 3800), 18432: (3817, 3749),
                   18816: (3922, 3797), 18944: (3867, 3741)}),
            (SO400M, {1458: (2781, 2736), 2187: (3011, 2975), 2916: (3638, 3661), 5832: (6335, 6549), 10206: (10149, 10679), 10935: (10932, 11034),
                      11664: (11802, 12550), 18225: (18808, 18498), 21870: (22978, 22539), 25515: (26267, 25656), 26244: (27237, 26273),
                      32805: (33816, 32986), 33534: (34499, 33268), 36450: (37668, 36373), 40095: (41093, 39885), 40824: (41956, 40891),
                      43740: (45352, 44682)})]


@pytest.mark.parametrize("gemms,times", MEASURED)
def test_chains_run_where_they_were_faster(gemms, times):
    """The rule takes the faster of the two at every size that was measured, or one that is at most 1 % behind."""
    from ittai_b200.siglip.kernel import chain_pays
    for rows, (chained, single) in times.items():
        taken = chained if chain_pays(rows, gemms, 148) else single
        assert taken <= 1.01 * min(chained, single), (rows, chained, single)
    chosen = [chain_pays(rows, gemms, 148) for rows in times]
    assert any(chosen) and not all(chosen)
