"""Banded pairs around the edges of the kernel that follows the diagonal: radii at the limits of its two lane counts
(68 and 140) and just past them, row counts around a lane's eight rows and a ring's turn, bands leaving the target
on either side, windows as wide as a lane's turn, near-identical pairs past the 16-bit headroom, several radii in
one claim; both planners, against the oracle's band rule."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import GapCosts, blosum62, encode
from sabertooth_b200.dtypes import PAIR_DTYPE
from tests.refrng import XorShift, rand_seq

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("planner")]


def check(ctx, cases, gaps):
    m = blosum62()
    rows = [m.sequence_rows(q) for q, _, _, _ in cases]
    ctx.upload_db_list([t for _, t, _, _ in cases])
    ids = ctx.create_profiles(rows)
    pairs = np.zeros(len(cases), dtype=PAIR_DTYPE)
    pairs["profile"], pairs["target"] = ids, np.arange(len(cases))
    pairs["band_center"] = [c for _, _, c, _ in cases]
    pairs["band_radius"] = [r for _, _, _, r in cases]
    try:
        got = ctx.sw_score_pairs(pairs, GapCosts(*gaps))
    finally:
        ctx.free_profiles(ids)
    want = np.array([O.band_score(rw, t, gaps[0], gaps[1], c, r) for rw, (_, t, c, r) in zip(rows, cases)])
    assert np.array_equal(got, want), np.nonzero(got != want)[0][:8]


def case(rng, ql, tl, c, r, letters=20, plant=True):
    q = np.array(rand_seq(rng, ql, letters), dtype=np.uint8)
    t = np.array(rand_seq(rng, tl, letters), dtype=np.uint8)
    if plant and 0 <= c < tl:
        k = min(ql, tl - c)
        keep = np.arange(k) % 5 != 0
        t[c:c + k][keep] = q[:k][keep]
        if k > 60:
            t[c + 40:c + k] = np.concatenate([t[c + 43:c + k], t[c:c + 3]])  # a deletion inside the band
    return q, t, c, r


@pytest.mark.parametrize("gaps", [(11, 1), (0, 0), (2, 5)])
@pytest.mark.parametrize("radius", [0, 1, 3, 4, 31, 64, 67, 68, 69, 100, 139, 140, 141])
def test_radius_and_row_edges(ctx, radius, gaps):
    rng = XorShift(17 + radius)
    cases = []
    for ql in (1, 7, 8, 9, 64, 127, 128, 129, 136, 257, 600):
        for tl, c in ((1, 0), (40, 5), (300, -10), (300, 120), (900, 250), (200, 195), (150, -140)):
            cases.append(case(rng, ql, tl, c, radius, 4 if ql % 2 else 20))
    check(ctx, cases, gaps)


def test_mixed_radii_and_rescored_pairs(ctx):
    rng = XorShift(2024)
    cases = []
    for i in range(61):
        ql = 1 + rng.range(500)
        tl = 1 + rng.range(1500)
        cases.append(case(rng, ql, tl, int(rng.range(tl + 80)) - 40, [0, 20, 68, 69, 140, 141, 400, -1][i % 8]
                          if i % 8 != 7 else 33))
    w = np.full(3300, int(encode("W")[0]), dtype=np.uint8)
    cases.insert(3, (w, w, 0, 64))
    cases.insert(20, (w, w[:3200], 2, 140))
    check(ctx, cases, (11, 1))
