"""The tile class of the fewest rows a pass (32) forced on queries of more than 8,192 rows: up to 256 passes it scores
them itself, past that another class does; both planners, and the autotuner, which times every class on such queries."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import Context, GapCosts, Kernel, tile_classes
from sabertooth_b200.dtypes import PAIR_DTYPE
from synth import workloads as W
from tests.test_sw_gpu import batch_scores

pytestmark = pytest.mark.gpu

_MODEL = W.Model()


def inputs(m):
    r = W.Rng(m)
    q = _MODEL.background(r, m)
    targets = [_MODEL.background(r, n) for n in (40, 333)]
    # homology in the last rows, which only the last passes hold
    targets += [np.concatenate([_MODEL.background(r, 7), _MODEL.mutate(r, q[m - k:], 0.7)]) for k in (60, 250)]
    return _MODEL.mat.sequence_rows(q), targets


@pytest.mark.usefixtures("planner")
@pytest.mark.parametrize("m", [8160, 8192, 8193, 9000, 10048])
def test_forced_class_of_few_rows(ctx, m):
    rows, targets = inputs(m)
    assert tile_classes()[0] == (4, 8, 4)
    saved = ctx.tuning_table()
    try:
        ctx.set_tuning_table(np.zeros((10, 8), dtype=np.int32))
        got, kern = batch_scores(ctx, [rows], targets, [(0, i) for i in range(len(targets))], GapCosts(11, 1),
                                 with_kernels=True)
    finally:
        ctx.set_tuning_table(saved)
    assert np.array_equal(got, [O.gotoh_score(rows, t, 11, 1) for t in targets])
    assert set(kern.tolist()) == {int(Kernel.GPU16)}


def test_autotune_with_long_queries():
    (long_rows, targets), (short_rows, _) = inputs(9000), inputs(500)
    c = Context(0)
    try:
        c.upload_db_list(targets)
        ids = c.create_profiles([long_rows, short_rows])
        pairs = np.zeros(2 * len(targets), dtype=PAIR_DTYPE)
        pairs["profile"] = np.repeat(ids, len(targets))
        pairs["target"] = np.tile(np.arange(len(targets)), 2)
        pairs["band_radius"] = -1
        assert c.autotune(pairs, GapCosts(11, 1)) == len(tile_classes())  # measured on the 500-row query alone
        got = c.sw_score_pairs(pairs, GapCosts(11, 1))
    finally:
        c.close()
    want = [O.gotoh_score(r, t, 11, 1) for r in (long_rows, short_rows) for t in targets]
    assert np.array_equal(got, want)
