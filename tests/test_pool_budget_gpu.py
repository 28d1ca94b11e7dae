"""Scratch near the memory budget: work whose arenas do not fit beside the pooled ones of earlier work still runs."""
import numpy as np
import pytest

from sabertooth_b200 import Context, GapCosts, PrefilterParams, blosum62
from sabertooth_b200._lib import SEED_HIT_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget_mb,sizes", [(40, (60_000, 220_000, 90_000)), (36, (200_000, 20_000, 200_000))])
def test_larger_work_after_smaller(budget_mb, sizes):
    rng = np.random.default_rng(budget_mb)
    m = blosum62()
    rows = [m.sequence_rows(rng.integers(0, 20, 80).astype(np.uint8)) for _ in range(4)]
    targets = [rng.integers(0, 20, 100).astype(np.uint8) for _ in range(200)]
    got = []
    for budget in (0, budget_mb << 20):
        r = np.random.default_rng(7)
        c = Context(0, hbm_budget_bytes=budget)
        try:
            c.upload_db_list(targets)
            ids = c.create_profiles(rows)
            out = []
            for n in sizes:
                h = np.zeros(n, dtype=SEED_HIT_DTYPE)
                h["query"] = ids[r.integers(0, 4, n)]
                h["target"] = r.integers(0, 200, n)
                h["qpos"] = r.integers(0, 80, n)
                h["diag"] = r.integers(0, 100, n) - h["qpos"]
                cand, counters = c.prefilter_gate(h, PrefilterParams(min_diag_score=20), GapCosts(11, 1))
                out.append((cand, counters))
            got.append(out)
        finally:
            c.close()
    for (a, ca), (b, cb) in zip(*got):
        assert np.array_equal(a, b) and ca == cb
