"""The tile classes picked for batches whose queries are alike, at and around the sizes where the rule changes (one query,
most queries waiting, lengths within and past a quarter of the mean), with both planners against the oracle; and the
time of such a batch against the best class."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sabertooth_b200 import GapCosts, blosum62, tile_classes
from synth import workloads as W
from tests.test_cta_tasks_gpu import all_pairs

pytestmark = pytest.mark.gpu

_MODEL = W.Model()


@pytest.mark.usefixtures("planner")
@pytest.mark.parametrize("nq,nt,m,n,spread", [(1, 7, 90, 50, 0), (20, 30, 60, 80, 0), (20, 30, 60, 80, 10), (20, 30, 60, 80, 60),
                                             (200, 12, 40, 40, 4), (6, 200, 300, 60, 0), (3, 5, 1200, 90, 0)])
def test_scores(ctx, nq, nt, m, n, spread):
    r = W.Rng(nq * 100 + spread)
    rows = [_MODEL.mat.sequence_rows(_MODEL.background(r, m + (k * spread) // max(nq - 1, 1))) for k in range(nq)]
    targets = [_MODEL.background(r, n) for _ in range(nt)]
    ctx.upload_db_list(targets)
    ids = ctx.create_profiles(rows)
    rates = ctx.tuning_rates()
    pairs = all_pairs(np.arange(nq), nt)
    want = O.sw_pairs(O.Arena(rows, targets), pairs["profile"], pairs["target"], 11, 1)
    try:
        for x in (rates, np.where(np.arange(len(rates)) == 5, rates, 0), np.zeros_like(rates)):  # one class's rate, none
            ctx.set_tuning_rates(x)
            assert np.array_equal(ctx.sw_score_pairs(all_pairs(ids, nt), GapCosts(11, 1)), want)
    finally:
        ctx.set_tuning_rates(rates)
        ctx.free_profiles(ids)


def test_close_to_the_best_class(ctx):
    """300 queries x 50 targets of 100 x 160: each query's path weighed by itself counted the same wait 300 times and took a
    class of more lanes, 1.38 times the best class's time."""
    m = blosum62()
    rng = np.random.default_rng(8)
    ctx.upload_db_list([rng.integers(0, 20, 160).astype(np.uint8) for _ in range(50)])
    ids = ctx.create_profiles([m.sequence_rows(rng.integers(0, 20, 100).astype(np.uint8)) for _ in range(300)])
    d = torch.zeros(300 * 50, dtype=torch.int32, device="cuda")

    def ms():
        plan = ctx.plan(all_pairs(ids, 50), GapCosts(11, 1), d.data_ptr())
        t = np.median([sum(t for _, _, t in plan.profile()) for _ in range(9)])
        plan.close()
        return t

    saved = ctx.tuning_table()
    try:
        picked = ms()
        best = np.inf
        for cls in range(len(tile_classes())):
            ctx.set_tuning_table(np.full((10, 8), cls, dtype=np.int32))
            best = min(best, ms())
    finally:
        ctx.set_tuning_table(saved)
        ctx.free_profiles(ids)
    assert picked < 1.2 * best, (picked, best)
