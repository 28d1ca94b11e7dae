"""Device allocations that the driver refuses: the arena of a size class is replaced by one of the exact size, a call
that does not fit is refused as such, and neither leaves an error behind for the work after it.  The refusals are made
by asking the driver for an impossible size (ST_ALLOC_FAIL_ABOVE, read when a context is made)."""
import numpy as np
import pytest

from sabertooth_b200 import Context, GapCosts, PrefilterParams, blosum62
from sabertooth_b200._lib import SEED_HIT_DTYPE, StError

pytestmark = pytest.mark.gpu

MB = 1 << 20


def gate(c, ids, n):
    r = np.random.default_rng(n)
    h = np.zeros(n, dtype=SEED_HIT_DTYPE)
    h["query"] = ids[r.integers(0, 4, n)]
    h["target"] = r.integers(0, 200, n)
    h["qpos"] = r.integers(0, 80, n)
    h["diag"] = r.integers(0, 100, n) - h["qpos"]
    return c.prefilter_gate(h, PrefilterParams(min_diag_score=20), GapCosts(11, 1))


def context(monkeypatch, limit):
    if limit is None:
        monkeypatch.delenv("ST_ALLOC_FAIL_ABOVE", raising=False)
    else:
        monkeypatch.setenv("ST_ALLOC_FAIL_ABOVE", str(limit))
    rng = np.random.default_rng(3)
    m = blosum62()
    c = Context(0)
    c.upload_db_list([rng.integers(0, 20, 100).astype(np.uint8) for _ in range(200)])
    return c, c.create_profiles([m.sequence_rows(rng.integers(0, 20, 80).astype(np.uint8)) for _ in range(4)])


def test_exact_size_after_a_refused_class(monkeypatch):
    """Arenas between 40 MB (a size class) and the limit of 44 MB are first asked for as 48 MB, which fails."""
    refused = exact = 0
    for n in range(200_000, 620_000, 10_000):
        free, ids = context(monkeypatch, None)
        want = gate(free, ids, n)
        c, ids = context(monkeypatch, 44 * MB)
        try:
            got = gate(c, ids, n)
        except StError as e:
            assert e.code == -3 and "out of memory" in str(e)
            refused += 1
            assert np.array_equal(gate(c, ids, 1000)[0], gate(free, ids, 1000)[0])  # the refusal is not found again
        else:
            assert refused == 0  # the arenas grow
            assert np.array_equal(got[0], want[0]) and got[1] == want[1]
            exact += c.mem_used() < free.mem_used()
        finally:
            c.close()
            free.close()
    assert refused > 0 and exact > 0


def test_refused_call_leaves_no_error(monkeypatch):
    """4 TB of calibration targets are refused; the scores, spans and calibration after that are not."""
    c, ids = context(monkeypatch, None)
    pairs = np.zeros(4, dtype=[("profile", "<u4"), ("target", "<u4"), ("band_center", "<i4"), ("band_radius", "<i4")])
    pairs["profile"], pairs["target"], pairs["band_radius"] = ids, np.arange(4), -1
    try:
        want = c.sw_score_pairs(pairs, GapCosts(11, 1))
        for work in (lambda: c.sw_score_pairs(pairs, GapCosts(11, 1)),
                     lambda: c.align_span_pairs(pairs, GapCosts(11, 1))[0],
                     lambda: c.sw_score_end_pairs(pairs, GapCosts(11, 1))[0]):
            with pytest.raises(StError) as e:
                c.calibrate_profiles(ids, [4_000_000_000], samples=1000)
            assert e.value.code == -3
            assert np.array_equal(work(), want)
        assert all(f is not None for f in c.calibrate_profiles(ids, [100, 200], samples=200))
    finally:
        c.close()
