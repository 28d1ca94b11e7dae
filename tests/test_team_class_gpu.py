"""The tile class whose CTA shares each task's passes among its warps (the last class): one pass to several rounds of
eight, targets shorter than the lag between passes, odd target counts, per-call scores that pick it; against the
oracle, with every pair scored by the packed kernel (a wait that ran out would send it to the 32-bit one)."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import GapCosts, Kernel, QueryProfile, blosum62, tile_classes
from synth import workloads as W
from tests.test_sw_gpu import batch_scores

pytestmark = pytest.mark.gpu

_MODEL = W.Model()


@pytest.mark.parametrize("planner_", ["host", "device"])
@pytest.mark.parametrize("m", [1, 255, 256, 257, 512, 513, 1900, 2048, 2049, 4500])
def test_rounds_and_short_targets(ctx, monkeypatch, planner_, m):
    monkeypatch.setenv("ST_DEVICE_PLAN_MIN", "1" if planner_ == "device" else "100000000")
    r = W.Rng(m)
    q = _MODEL.background(r, m)
    targets = []
    for n in (1, 3, 31, 32, 33, 127, 144, 145, 300, 901, 17):
        t = _MODEL.background(r, n)
        k = min(m, n)
        t[n - k:] = _MODEL.mutate(r, q[m - k:], 0.6)
        targets.append(t)
    rows = _MODEL.mat.sequence_rows(q)
    cls = len(tile_classes()) - 1
    assert tile_classes()[cls] == (32, 8, 4)
    saved = ctx.tuning_table()
    try:
        ctx.set_tuning_table(np.full((10, 8), cls, dtype=np.int32))
        got, kern = batch_scores(ctx, [rows], targets, [(0, i) for i in range(len(targets))], GapCosts(11, 1),
                                 with_kernels=True)
    finally:
        ctx.set_tuning_table(saved)
    assert np.array_equal(got, [O.gotoh_score(rows, t, 11, 1) for t in targets])
    assert set(kern.tolist()) == {int(Kernel.GPU16)}


def test_per_call_long_pair(ctx):
    r = W.Rng(8)
    q = _MODEL.background(r, 2000)
    t = np.concatenate([_MODEL.background(r, 1500), _MODEL.mutate(r, q, 0.5, 0.01), _MODEL.background(r, 900)])
    rows = blosum62().sequence_rows(q)
    qp = QueryProfile.from_rows(rows, ctx)
    assert qp.sw_score_with(t, GapCosts(11, 1)) == (O.gotoh_score(rows, t, 11, 1), Kernel.GPU16)
    qp.free()
