"""Batches around the sizes where the planner changes its answer: a batch too small to fill the chip takes tile
classes of many lanes (its longest wavefront decides) and spreads its warp tasks over the SMs in CTA tasks of 1, 2
or 4 warp tasks; larger ones use whole CTAs and the cheapest class.  Both planners, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import GapCosts, blosum62
from sabertooth_b200.dtypes import PAIR_DTYPE
from synth import workloads as W

pytestmark = pytest.mark.gpu

_MODEL = W.Model()


@pytest.mark.parametrize("planner", ["device", "host"])
@pytest.mark.parametrize("queries,per_query", [((1,), 1), ((700,), 3), ((250,), 33), ((1500, 40), 130), ((30, 260, 900), 400),
                                               ((120,), 4200)])
def test_scores_match_the_oracle(ctx, monkeypatch, planner, queries, per_query):
    monkeypatch.setenv("ST_DEVICE_PLAN_MIN", "1" if planner == "device" else "100000000")
    r = W.Rng(1000 * len(queries) + per_query)
    rows = [_MODEL.mat.sequence_rows(_MODEL.background(r, m)) for m in queries]
    lens = W.lognormal_lengths(r, per_query, 90, 0.9, 1, 600)
    targets = [_MODEL.background(r, int(n)) for n in lens]
    ctx.upload_db_list(targets)
    ids = ctx.create_profiles(rows)
    pq = np.repeat(np.arange(len(queries), dtype=np.uint32), per_query)
    pt = np.tile(np.arange(per_query, dtype=np.uint32), len(queries))
    pairs = np.zeros(len(pq), dtype=PAIR_DTYPE)
    pairs["profile"], pairs["target"], pairs["band_radius"] = ids[pq], pt, -1
    try:
        got = ctx.sw_score_pairs(pairs, GapCosts(11, 1))
    finally:
        ctx.free_profiles(ids)
    assert np.array_equal(got, O.sw_pairs(O.Arena(rows, targets), pq, pt, 11, 1))


def test_a_batch_with_a_32_bit_list_keeps_its_tasks(ctx, monkeypatch):
    """Pairs for both kernels in one device-planned batch (the 32-bit list is ordered in buffers of the pair sort)."""
    monkeypatch.setenv("ST_DEVICE_PLAN_MIN", "1")
    r = W.Rng(77)
    rows = [_MODEL.mat.sequence_rows(_MODEL.background(r, m)) for m in (60, 300)]
    targets = [_MODEL.background(r, 20 + 3 * i) for i in range(300)]
    ctx.upload_db_list(targets)
    ids = ctx.create_profiles(rows)
    pq = np.arange(600, dtype=np.uint32) % 2
    pt = np.arange(600, dtype=np.uint32) // 2
    pairs = np.zeros(600, dtype=PAIR_DTYPE)
    pairs["profile"], pairs["target"] = ids[pq], pt
    pairs["band_radius"] = np.where(np.arange(600) % 7 == 0, 20, -1)
    try:
        got = ctx.sw_score_pairs(pairs, GapCosts(11, 1))
    finally:
        ctx.free_profiles(ids)
    want = O.sw_pairs(O.Arena(rows, targets), pq, pt, 11, 1, np.zeros(600, np.int64),
                      pairs["band_radius"].astype(np.int64))
    assert np.array_equal(got, want)
