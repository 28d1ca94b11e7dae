"""End cells and spans of the packed kernel's end modes at their edges: every class that tracks end cells, one and
several passes, ties (few letters, zero gap costs), prefixes of one row or one column, scores past the 16-bit
headroom and rows outside int8 (32-bit list), both planners; against the oracle's forward pass and its forward
pass over the reversed prefix."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import GapCosts, blosum62, encode, tile_classes
from sabertooth_b200.dtypes import PAIR_DTYPE
from tests.refrng import XorShift, rand_seq

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("planner")]

END_CLASSES = [(8, 8, 4), (32, 8, 4), (8, 16, 4), (16, 16, 4), (32, 16, 4)]


def want(rows, t, o, e):
    r = O.gotoh_score_end(rows, t, o, e)
    if r is None or r[0] <= 0:
        return (0, -1, -1, -1, -1)
    s, qe, te = r
    back = O.gotoh_score_end(np.ascontiguousarray(rows[:qe + 1][::-1]), np.ascontiguousarray(t[:te + 1][::-1]), o, e)
    assert back[0] == s
    return (s, qe, te, qe - back[1], te - back[2])


def check(ctx, rows, targets, gaps):
    ctx.upload_db_list(targets)
    ids = ctx.create_profiles(rows)
    n = len(rows)
    pairs = np.zeros(n, dtype=PAIR_DTYPE)
    pairs["profile"], pairs["target"], pairs["band_radius"] = ids, np.arange(n), -1
    try:
        s, st, en = ctx.align_span_pairs(pairs, gaps)
        s2, en2 = ctx.sw_score_end_pairs(pairs, gaps)
    finally:
        ctx.free_profiles(ids)
    w = np.array([want(r, t, gaps.open, gaps.extend) for r, t in zip(rows, targets)])
    got = np.stack([s, en[:, 0], en[:, 1], st[:, 0], st[:, 1]], 1)
    assert np.array_equal(got, w), np.nonzero((got != w).any(1))[0][:5]
    assert np.array_equal(s2, s) and np.array_equal(en2, en)


@pytest.mark.parametrize("cls", END_CLASSES)
@pytest.mark.parametrize("gaps", [(11, 1), (0, 0), (2, 3)])
def test_every_end_class(ctx, cls, gaps):
    m = blosum62()
    index = tile_classes().index(cls)
    rng = XorShift(5 + 100 * index)
    rows, targets = [], []
    for ql in (1, 7, 8, 63, 65, 129, 260, 530, 1100, 2100):
        for tl, letters in ((1, 20), (4, 2), (31, 3), (66, 2), (250, 20), (333, 4)):
            q = np.array(rand_seq(rng, ql, letters), dtype=np.uint8)
            t = np.array(rand_seq(rng, tl, letters), dtype=np.uint8)
            k = min(ql, tl) // 2
            if letters == 20 and k:
                t[tl - k:] = q[ql - k:]
            rows.append(m.sequence_rows(q))
            targets.append(t)
    saved = ctx.tuning_table()
    try:
        ctx.set_tuning_table(np.full((10, 8), index, dtype=np.int32))
        check(ctx, rows, targets, GapCosts(*gaps))
    finally:
        ctx.set_tuning_table(saved)


def test_several_targets_of_one_query_and_the_32_bit_list(ctx):
    m = blosum62()
    rng = XorShift(99)
    w = np.full(3300, int(encode("W")[0]), dtype=np.uint8)
    q = np.array(rand_seq(rng, 300, 20), dtype=np.uint8)
    wide = np.full((5, 21), 300, dtype=np.int32)
    rows, targets = [], []
    for i in range(70):
        t = np.array(rand_seq(rng, 1 + rng.range(400), 20), dtype=np.uint8)
        a = rng.range(len(t))
        b = min(len(t) - a, 200)
        t[a:a + b] = q[50:50 + b]
        rows.append(m.sequence_rows(q))
        targets.append(t)
    rows += [m.sequence_rows(w), m.sequence_rows(w), wide, np.zeros((0, 21), np.int32)]
    targets += [w, w[:2000], np.array([1, 2, 3], np.uint8), np.array([1], np.uint8)]
    check(ctx, rows, targets, GapCosts(11, 1))
    check(ctx, rows[:20], targets[:20], GapCosts(20000, 5))  # gap costs outside the 16-bit range


def test_targets_past_the_16_bit_column(ctx):
    m = blosum62()
    rng = XorShift(3)
    q = np.array(rand_seq(rng, 40, 20), dtype=np.uint8)
    rows, targets = [], []
    for n in (65535, 65536, 65600):
        t = np.array(rand_seq(rng, n, 20), dtype=np.uint8)
        t[n - 40:] = q
        rows.append(m.sequence_rows(q))
        targets.append(t)
    check(ctx, rows, targets, GapCosts(11, 1))
