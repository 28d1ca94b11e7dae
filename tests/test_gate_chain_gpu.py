"""Chains whose segment positions a CTA walks together, against the oracle: group counts at the edges of a CTA's round
(128 and 256 groups), few and many diagonals a group, with and without regions."""
import numpy as np
import pytest

from sabertooth_b200 import blosum62
from sabertooth_b200._lib import SEED_HIT_DTYPE
from tests.seedhits import default_params
from tests.test_gate_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 255, 256, 257, 600])
@pytest.mark.parametrize("kmax,regions", [(2, 1), (4, 0), (4, 1), (5, 1), (16, 0), (16, 1)])
def test_chains_at_round_edges(ctx, n, kmax, regions):
    rng = np.random.default_rng(1000 * n + 10 * kmax + regions)
    q = rng.integers(0, 20, 64).astype(np.uint8)
    targets, hits = [], []
    for t in range(n):
        gap = int(rng.integers(0, 9))  # pieces 0..8 residues apart; the second may come first in the target
        parts = [q[:30], rng.integers(0, 20, gap).astype(np.uint8), q[30:]]
        if t % 5 == 4:
            parts.reverse()
        s = np.concatenate(parts)
        noise = rng.random(len(s)) < 0.2 * (t % 3)
        s = np.where(noise, rng.integers(0, 20, len(s)), s).astype(np.uint8)
        targets.append(s)
        d0, d1 = (34 + gap, -30) if t % 5 == 4 else (0, gap)
        for d in {d0, d1, *(int(x) for x in rng.integers(-20, 21, t % 7))}:
            for p in rng.integers(max(0, -d), min(64, len(s) - d), 1 + t % 3):
                hits.append((0, t, d, int(p)))
    a = np.array(hits, dtype=np.int64)
    h = np.zeros(len(a), dtype=SEED_HIT_DTYPE)
    for k, name in enumerate(("query", "target", "diag", "qpos")):
        h[name] = a[:, k]
    p = default_params(span=6, min_diag_score=25)
    p["max_diagonals"] = kmax
    p["regions"] = regions
    got, st = _check(ctx, [blosum62().sequence_rows(q)], targets, h[rng.permutation(len(h))], p)
    assert len(got)
