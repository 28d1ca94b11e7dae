"""How the kernel of banded pairs claims its list: couples of narrow, wide and other pairs in every mix and number,
against the oracle; and two couples of wide bands side by side, not one after the other on one warp."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from sabertooth_b200 import GapCosts, blosum62
from sabertooth_b200.dtypes import PAIR_DTYPE
from tests.refrng import XorShift
from tests.test_band_ring_gpu import case, check

pytestmark = pytest.mark.gpu


@pytest.mark.usefixtures("planner")
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 9, 13])
def test_mixed_claims(ctx, n):
    """Radii at and past the limits of the two rings (68, 140), of nearly the same cost, so that the list, longest
    first, puts them side by side in any order."""
    rng = XorShift(100 + n)
    for radii in ((68, 69), (3, 141), (0, 68, 69, 140, 141, 300), (300, 5)):
        cases = []
        for k in range(n):
            r = radii[rng.range(len(radii))]
            # cost of a narrow band 9/8 rows + 2 radius, of a wide one passes x (window + 31)
            ql = 150 + rng.range(120) if r > 140 else 500 + rng.range(120)
            cases.append(case(rng, ql, 1200, int(rng.range(300)) - 60, r))
        check(ctx, cases, (11, 1))


@pytest.mark.usefixtures("planner")
def test_pairs_left_to_the_32_bit_kernel_between(ctx):
    """Banded pairs whose rows exceed int8 and unbanded ones share the list and are skipped by the claims."""
    rng = XorShift(7)
    m = blosum62()
    cases = [case(rng, 300 + rng.range(60), 900, 50, [40, 100, 200, 30][k % 4]) for k in range(22)]
    scale = [30 if k % 3 == 1 else 1 for k in range(22)]  # 30 x BLOSUM62: outside int8
    rows = [m.sequence_rows(q) * s for (q, _, _, _), s in zip(cases, scale)]
    ctx.upload_db_list([t for _, t, _, _ in cases])
    ids = ctx.create_profiles(rows)
    pairs = np.zeros(22, dtype=PAIR_DTYPE)
    pairs["profile"], pairs["target"] = ids, np.arange(22)
    pairs["band_center"], pairs["band_radius"] = 50, [c[3] for c in cases]
    try:
        got = ctx.sw_score_pairs(pairs, GapCosts(11, 1))
    finally:
        ctx.free_profiles(ids)
    assert np.array_equal(got, [O.band_score(rw, t, 11, 1, 50, r) for rw, (_, t, _, r) in zip(rows, cases)])


@pytest.mark.parametrize("radius", [100, 300])
def test_wide_couples_run_side_by_side(ctx, radius):
    """Four equal pairs take as long as two where the chip has warps to spare: one after the other they take twice as
    long, side by side the same time (within the launch's few microseconds)."""
    rng = np.random.default_rng(radius)
    m = blosum62()
    q = rng.integers(0, 20, 1000).astype(np.uint8)
    ctx.upload_db_list([rng.integers(0, 20, 4000).astype(np.uint8) for _ in range(4)])
    ids = ctx.create_profiles([m.sequence_rows(q)])
    ms = {}
    for n in (2, 4):
        pairs = np.zeros(n, dtype=PAIR_DTYPE)
        pairs["profile"], pairs["target"] = ids[0], np.arange(n)
        pairs["band_center"], pairs["band_radius"] = 500, radius
        d = torch.zeros(n, dtype=torch.int32, device="cuda")
        plan = ctx.plan(pairs, GapCosts(11, 1), d.data_ptr())
        runs = []
        for _ in range(7):
            runs += [t for name, _, t in plan.profile() if name == "band16"]
        ms[n] = min(runs)
        plan.close()
    ctx.free_profiles(ids)
    assert ms[4] < 1.5 * ms[2], ms
