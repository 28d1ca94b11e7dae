"""How a query's warp tasks are cut into CTA tasks: batches below, at and above what is resident at once, one and many
queries, target counts around a unit's, several classes, with both planners, against the oracle; and no warp task that
waits for another where the chip has schedulers for all."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sabertooth_b200 import GapCosts, blosum62, tile_classes
from sabertooth_b200.dtypes import PAIR_DTYPE
from synth import workloads as W

pytestmark = pytest.mark.gpu

_MODEL = W.Model()


def all_pairs(ids, n_targets):
    pairs = np.zeros(len(ids) * n_targets, dtype=PAIR_DTYPE)
    pairs["profile"] = np.repeat(ids, n_targets)
    pairs["target"] = np.tile(np.arange(n_targets), len(ids))
    pairs["band_radius"] = -1
    return pairs


@pytest.mark.usefixtures("planner")
@pytest.mark.parametrize("shape", [(4, 28), (32, 8), (8, 32), (16, 16), None])
@pytest.mark.parametrize("nq,nt", [(1, 1), (1, 65), (1, 1100), (3, 129), (40, 31), (40, 257), (220, 64)])
def test_scores(ctx, shape, nq, nt):
    r = W.Rng(nq * 1000 + nt)
    queries = [_MODEL.background(r, 10 + (37 * k) % 90) for k in range(nq)]
    targets = [_MODEL.background(r, 5 + (13 * k) % 60) for k in range(nt)]
    rows = [_MODEL.mat.sequence_rows(q) for q in queries]
    ctx.upload_db_list(targets)
    ids = ctx.create_profiles(rows)
    saved = ctx.tuning_table()
    try:
        if shape is not None:
            cls = [c[:2] for c in tile_classes()].index(shape)
            ctx.set_tuning_table(np.full((10, 8), cls, dtype=np.int32))
        got = ctx.sw_score_pairs(all_pairs(ids, nt), GapCosts(11, 1))
    finally:
        ctx.set_tuning_table(saved)
        ctx.free_profiles(ids)
    pairs = all_pairs(np.arange(nq), nt)
    want = O.sw_pairs(O.Arena(rows, targets), pairs["profile"], pairs["target"], 11, 1)
    assert np.array_equal(got, want)


def test_fewer_warp_tasks_than_schedulers(ctx):
    """100 queries x 30 targets in <8,32> are 400 warp tasks, four a query, in CTAs of four warps: with 592 schedulers none
    waits for another, so they take as long as the 100 of 100 queries x 8 targets.  Units of one warp task, two or
    three of them in a CTA task by the class's cap, took 1.7 to 2.4 times as long."""
    m = blosum62()
    rng = np.random.default_rng(4)
    ctx.upload_db_list([rng.integers(0, 20, 300).astype(np.uint8) for _ in range(30)])
    ids = ctx.create_profiles([m.sequence_rows(rng.integers(0, 20, 250).astype(np.uint8)) for _ in range(100)])
    saved = ctx.tuning_table()
    ms = {}
    try:
        ctx.set_tuning_table(np.full((10, 8), [c[:2] for c in tile_classes()].index((8, 32)), dtype=np.int32))
        for n in (8, 30):
            d = torch.zeros(n * 100, dtype=torch.int32, device="cuda")
            plan = ctx.plan(all_pairs(ids, n), GapCosts(11, 1), d.data_ptr())
            ms[n] = np.median([plan.profile()[0][2] for _ in range(9)])
            plan.close()
    finally:
        ctx.set_tuning_table(saved)
        ctx.free_profiles(ids)
    assert ms[30] < 1.4 * ms[8], ms
