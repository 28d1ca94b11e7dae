"""Seed-hit keys of the evidence path that hold the query position (query, target, diagonal and position in 64 bits)
and those whose positions are sorted beside them, against the oracle field for field.

The bits a field takes follow the database and the profiles: 300 profiles (9 bits), one of 8,300 rows (14 bits of
position), 70,000 targets (17 bits) and one of 2^24 residues (25 bits of diagonal) make 65; each of them made smaller
leaves room.
"""
import numpy as np
import pytest

from sabertooth_b200._lib import SEED_HIT_DTYPE
from sabertooth_b200 import PrefilterParams, blosum62
from tests.seedhits import default_params
from tests.test_gate_gpu import _check

pytestmark = pytest.mark.gpu


def _case(rng, n_short, m_long, n_targets, t_long):
    rows = [rng.integers(-4, 6, size=(int(m), 21), dtype=np.int32) for m in rng.integers(1, 60, n_short)]
    for r in rows:
        r[:, 20] = -1
    mat = blosum62()
    q = rng.integers(0, 20, m_long).astype(np.uint8)
    rows.append(mat.sequence_rows(q))
    targets = [t for t in np.split(rng.integers(0, 20, 24 * (n_targets - 1)).astype(np.uint8), n_targets - 1)]
    long_t = rng.integers(0, 20, t_long).astype(np.uint8)
    at = t_long - m_long  # two pieces of the long query, some residues apart, at the far end
    long_t[at:at + m_long // 2] = q[:m_long // 2]
    long_t[at + m_long // 2 + 3:] = q[m_long // 2:m_long - 3]
    targets.append(long_t)
    hits = []
    for _ in range(400):  # the long query on the long target: both pieces, and stray diagonals
        p = int(rng.integers(0, m_long - 16))
        hits.append((n_short, n_targets - 1, at + (3 if p >= m_long // 2 else 0), p))
    for _ in range(300):
        p = int(rng.integers(0, m_long))
        hits.append((n_short, n_targets - 1, int(rng.integers(0, t_long)) - p, p))
    for _ in range(3000):  # all queries on short targets, several hits a pair
        qi = int(rng.integers(0, n_short + 1))
        t = int(rng.choice([0, 1, n_targets - 2, int(rng.integers(0, n_targets - 1))]))
        p = int(rng.integers(0, len(rows[qi])))
        hits.append((qi, t, int(rng.integers(0, len(targets[t]))) - p, p))
    # first and last position of the longest query, which fill the position's bits
    hits += [(n_short, 0, 0, 0), (n_short, n_targets - 1, t_long - m_long, m_long - 1),
             (n_short, n_targets - 1, -(m_long - 1), m_long - 1)]
    a = np.array(hits, dtype=np.int64)
    h = np.zeros(len(a), dtype=SEED_HIT_DTYPE)
    for k, name in enumerate(("query", "target", "diag", "qpos")):
        h[name] = a[:, k]
    return rows, targets, h[rng.permutation(len(h))]


@pytest.mark.parametrize("n_short,m_long,n_targets,t_long", [
    (299, 8300, 70000, 1 << 24),  # 65 bits: positions beside the keys
    (299, 8192, 70000, 1 << 24),  # 64 bits: the last that fits
    (20, 600, 500, 3000),
    (0, 17, 2, 40),
])
@pytest.mark.parametrize("window", [0, 24])
def test_keys_with_and_without_positions(ctx, n_short, m_long, n_targets, t_long, window):
    rng = np.random.default_rng(m_long + n_targets + window)
    rows, targets, hits = _case(rng, n_short, m_long, n_targets, t_long)
    p = default_params(span=6, min_diag_score=12)
    p["diag_window"] = window
    got, _ = _check(ctx, rows, targets, hits, p)
    assert len(got)


@pytest.mark.parametrize("n_short,m_long,n_targets,t_long", [(299, 8300, 70000, 1 << 24), (3, 600, 500, 30000)])
def test_search_from_records_and_from_keys(ctx, n_short, m_long, n_targets, t_long):
    # the prefilter of a batch of queries equals its seed hits through the evidence call, whichever form the hits take
    rng = np.random.default_rng(n_targets)
    rows, targets, _ = _case(rng, n_short, m_long, n_targets, t_long)
    m = blosum62()
    pick = [0, 1, 2, n_short]
    qs = [rng.integers(0, 20, len(rows[i])).astype(np.uint8) for i in pick[:-1]]
    at = t_long - m_long
    qs.append(targets[-1][at:at + m_long].copy())  # the long query is the far end of the long target
    for i, q in zip(pick, qs):
        rows[i] = m.sequence_rows(q)
    ctx.upload_db_list(targets)
    ids = ctx.create_profiles(rows)
    try:
        ctx.seed_index_build("111001101")
        p = PrefilterParams(min_diag_score=43, span=9)
        sel = ids[pick]
        found, evidence, _ = ctx.prefilter_queries(sel, qs, p)
        hits, _ = ctx.seed_hits(sel, qs, p)
        want, counters = ctx.prefilter_gate(hits, p)
        assert len(want) and len(hits) > len(want)
        assert np.array_equal(found, want[np.argsort(want["query"], kind="stable")])
        assert evidence == counters
    finally:
        ctx.free_profiles(ids)
