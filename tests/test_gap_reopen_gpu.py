"""The packed kernel's gap recurrence at the edges of its rewriting: both gap states open from the match state
and extend at min(open, extend), so gap costs with extend above, equal to and below open, including zero ones,
are scored in every tile class, with one pass and with several, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import GapCosts, blosum62, tile_classes
from tests.refrng import XorShift, rand_seq
from tests.test_sw_gpu import batch_scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("open_,ext", [(0, 0), (0, 3), (1, 5), (3, 16000), (4, 4), (7, 0)])
def test_every_class_matches_the_oracle(ctx, open_, ext):
    m = blosum62()
    rng = XorShift(991 + 17 * open_ + ext)
    rows, targets, want = [], [], []
    for ql, tl in [(1, 1), (8, 33), (33, 8), (97, 64), (129, 250), (300, 31), (800, 120)]:
        q = rand_seq(rng, ql, 6)
        t = np.array(rand_seq(rng, tl, 6), dtype=np.uint8)
        k = min(ql, tl)
        t[k // 3:k] = np.array(q, dtype=np.uint8)[:k - k // 3]  # a homolog behind a gap
        rows.append(m.sequence_rows(q))
        targets.append(t)
        want.append(O.gotoh_score(rows[-1], t, open_, ext))
    pairs = [(i, i) for i in range(len(rows))]
    saved = ctx.tuning_table()
    try:
        for c in range(len(tile_classes())):
            ctx.set_tuning_table(np.full((10, 8), c, dtype=np.int32))
            got = batch_scores(ctx, rows, targets, pairs, GapCosts(open_, ext))
            assert np.array_equal(got, np.array(want, dtype=np.int32)), (tile_classes()[c], got, want)
    finally:
        ctx.set_tuning_table(saved)
