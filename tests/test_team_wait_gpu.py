"""A team's wait that runs out: with no polls allowed a warp that finds the pass above it unfinished gives the task up, and
its pairs are scored by the exact 32-bit kernel.  Batches of one and several tasks a CTA, with both planners, per-call
scores, and a context with the usual limit after them."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import Context, GapCosts, Kernel, QueryProfile, tile_classes
from synth import workloads as W
from tests.test_cta_tasks_gpu import all_pairs

pytestmark = pytest.mark.gpu

_MODEL = W.Model()


def inputs():
    r = W.Rng(31)
    q = [_MODEL.background(r, m) for m in (300, 2100, 4500)]
    targets = [_MODEL.background(r, n) for n in (40, 200, 333, 700)]
    targets += [np.concatenate([_MODEL.background(r, 30), _MODEL.mutate(r, x, 0.6, 0.01)[:900]]) for x in q]
    return [_MODEL.mat.sequence_rows(x) for x in q], targets


def context(monkeypatch, spins):
    if spins is None:
        monkeypatch.delenv("ST_TEAM_SPINS", raising=False)
    else:
        monkeypatch.setenv("ST_TEAM_SPINS", str(spins))
    return Context(0)


@pytest.mark.usefixtures("planner")
@pytest.mark.parametrize("copies", [1, 120])
def test_pairs_go_to_the_32_bit_kernel(monkeypatch, copies):
    rows, targets = inputs()
    targets = targets * copies  # 840 targets: more CTA tasks than CTAs, so a CTA gives up one task and begins the next
    pairs = all_pairs(np.arange(3), len(targets))
    want = O.sw_pairs(O.Arena(rows, targets), pairs["profile"], pairs["target"], 11, 1)
    for spins in (0, None):
        c = context(monkeypatch, spins)
        try:
            c.upload_db_list(targets)
            ids = c.create_profiles(rows)
            c.set_tuning_table(np.full((10, 8), len(tile_classes()) - 1, dtype=np.int32))
            for _ in range(2):
                got, kern = c.sw_score_pairs(all_pairs(ids, len(targets)), GapCosts(11, 1), with_kernels=True)
                assert np.array_equal(got, want)
                if spins is None:
                    assert set(kern.tolist()) == {int(Kernel.GPU16)}
                else:  # a pass 36 steps behind another is never there at the first look
                    assert set(kern.tolist()) == {int(Kernel.GPU32)}
        finally:
            c.close()


def test_per_call_score(monkeypatch):
    rows, targets = inputs()
    t = targets[-1]
    want = O.gotoh_score(rows[2], t, 11, 1)
    for spins, kernel in ((0, Kernel.GPU32), (None, Kernel.GPU16)):
        c = context(monkeypatch, spins)
        try:
            qp = QueryProfile.from_rows(rows[2], c)
            for _ in range(3):
                assert qp.sw_score_with(t, GapCosts(11, 1)) == (want, kernel)
            qp.free()
        finally:
            c.close()
