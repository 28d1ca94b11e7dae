"""The hits kernel's runs at their edges: runs of one query around a CTA's 256 lanes and around a chunk, windows that all
start at the query's first row or at one row, empty windows inside a run, many short runs in a chunk, rows outside
int8, and the longest query that the kernel's shared memory takes; against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from sabertooth_b200 import blosum62
from sabertooth_b200._lib import StError
from sabertooth_b200.dtypes import HIT_DTYPE
from synth import workloads as W

pytestmark = pytest.mark.gpu

_MODEL = W.Model()


def check(ctx, rows, targets, hq, ht, hd):
    ctx.upload_db_list(targets)
    ids = ctx.create_profiles(rows)
    hits = np.zeros(len(hq), dtype=HIT_DTYPE)
    hits["query"], hits["target"], hits["diag"] = ids[hq], ht, hd
    try:
        got = ctx.ungapped_hits(hits, with_pairs=False)
    finally:
        ctx.free_profiles(ids)
    assert np.array_equal(got, O.ungapped_hits(O.Arena(rows, targets), hq, ht, hd))


def inputs(seed, lens, n_targets=60):
    r = W.Rng(seed)
    rows = [_MODEL.mat.sequence_rows(_MODEL.background(r, m)) for m in lens]
    targets = [_MODEL.background(r, int(n)) for n in W.lognormal_lengths(r, n_targets, 120, 0.7, 1, 700)]
    return rows, targets


@pytest.mark.parametrize("n", [1, 255, 256, 257, 300, 1023, 1024, 1025, 9000])
@pytest.mark.parametrize("kind", ["any", "from_zero", "one_row", "empty"])
def test_runs_and_starts(ctx, n, kind):
    rows, targets = inputs(n, [150])
    rng = np.random.default_rng(n)
    t = rng.integers(0, len(targets), n)
    tl = np.array([len(x) for x in targets])[t]
    if kind == "any":
        d = rng.integers(-149, 1 << 30, n) % (149 + tl) - 149
    elif kind == "from_zero":
        d = rng.integers(0, 1 << 30, n) % tl
    elif kind == "one_row":
        d = np.full(n, -32)
    else:
        d = np.where(rng.random(n) < 0.7, tl + 5, -20)  # most windows empty
    check(ctx, rows, targets, np.zeros(n, np.int64), t, d)


def test_many_runs_in_a_chunk_and_wide_rows(ctx):
    rows, targets = inputs(5, [20, 64, 300, 37, 512])
    rows.append(np.where(rows[2] > 3, 900, rows[2]).astype(np.int32))
    rng = np.random.default_rng(3)
    q = np.sort(rng.integers(0, 6, 20000))
    q[4000:6000] = rng.integers(0, 6, 2000)  # unsorted: runs of a few hits
    t = rng.integers(0, len(targets), 20000)
    m = np.array([len(r) for r in rows])[q]
    tl = np.array([len(x) for x in targets])[t]
    check(ctx, rows, targets, q, t, rng.integers(0, 1 << 30, 20000) % (m + tl - 1) - m + 1)


def test_longest_query(ctx):
    r = W.Rng(9)
    long = _MODEL.background(r, 10480)
    rows = [_MODEL.mat.sequence_rows(long)]
    targets = [long[3000:3400].copy(), _MODEL.background(r, 900), long.copy()]
    d = np.arange(-10479, 400, 7)
    check(ctx, rows, targets, np.zeros(3 * len(d), np.int64), np.repeat(np.arange(3), len(d)), np.tile(d, 3))
    with pytest.raises(StError):
        check(ctx, [_MODEL.mat.sequence_rows(_MODEL.background(r, 10481))], targets, np.zeros(1, np.int64),
              np.zeros(1, np.int64), np.zeros(1, np.int64))
