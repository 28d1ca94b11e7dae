"""Kernels whose shared memory is asked for where they are first launched: end cells and spans of the longest queries
that the tile classes stage, and the seed kernel around the size that needs asking, as a context's first work."""
import time

import numpy as np
import pytest

from sabertooth_b200 import Context, GapCosts, PrefilterParams, blosum62
from tests.refrng import XorShift, rand_seq
from tests.test_end_classes_gpu import check
from tests.test_seeds_gpu import _check_hits

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.usefixtures("planner")
@pytest.mark.parametrize("m", [2233, 9984, 9985, 10048, 10049])
def test_spans_of_long_queries(fresh, m):
    """10,048 rows are 157 passes of <8,8> and 221,056 bytes of staged profile; one more is the 32-bit kernel's."""
    rng = XorShift(m)
    q = np.array(rand_seq(rng, m, 20), dtype=np.uint8)
    rows, targets = [], []
    for n in (30, 333):
        t = np.array(rand_seq(rng, n, 20), dtype=np.uint8)
        t[n - 25:] = q[m - 25:]
        rows.append(blosum62().sequence_rows(q))
        targets.append(t)
    check(fresh, rows, targets, GapCosts(11, 1))


@pytest.mark.parametrize("cap", [2559, 2560, 2561, 3000, 4096])
def test_seed_caps(fresh, cap):
    rng = np.random.default_rng(cap)
    rows = [np.full((9, 21), 2, dtype=np.int32), rng.integers(-1, 2, size=(20, 21)).astype(np.int32)]
    targets = [rng.integers(0, 20, int(rng.integers(10, 120))).astype(np.uint8) for _ in range(60)]
    st = _check_hits(fresh, rows, None, targets, "1101",
                     PrefilterParams(kmer_score=2, max_kmers_per_pos=cap, exact_seeds=False))
    assert st["windows_at_cap"] > 0


def test_first_span_call_makes_no_pinned_block():
    """A context's first small span call stages its plan in the pinned block that the database upload made, with the
    streams it needs; a first scoring call makes a block of its own, which is 2 of its 2.5 ms."""
    m = blosum62()
    rng = np.random.default_rng(1)
    rows = [m.sequence_rows(rng.integers(0, 20, 250).astype(np.uint8)) for _ in range(16)]
    targets = [rng.integers(0, 20, 300).astype(np.uint8) for _ in range(64)]
    pairs = np.zeros(64, dtype=[("profile", "<u4"), ("target", "<u4"), ("band_center", "<i4"), ("band_radius", "<i4")])
    pairs["target"], pairs["band_radius"] = np.arange(64), -1

    def first_call(work):
        c = Context(0)
        try:
            c.upload_db_list(targets)
            pairs["profile"] = np.repeat(c.create_profiles(rows), 4)
            c.synchronize()
            t0 = time.perf_counter()
            work(c)
            return time.perf_counter() - t0
        finally:
            c.close()

    for work in (lambda c: c.align_span_pairs(pairs, GapCosts(11, 1)),
                 lambda c: c.sw_score_end_pairs(pairs, GapCosts(11, 1))):
        first_call(work)  # loads the kernels
        ends = [first_call(work) for _ in range(15)]
        scores = [first_call(lambda c: c.sw_score_pairs(pairs, GapCosts(11, 1))) for _ in range(15)]
        assert min(ends) < 0.5 * min(scores), (ends, scores)  # host timings: a busy machine only adds to them
