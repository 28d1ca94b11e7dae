"""The k-mer generator of one warp per window at its edges: caps around a warp's width and the largest that its levels
in shared memory take, the first cap past it (the depth-first form), rows whose scores all tie (the kept ties follow
the rank order from among thousands), rows of one dominant residue, two to six care positions; hits and counters
against the oracle."""
import numpy as np
import pytest

from sabertooth_b200 import PrefilterParams
from tests.test_seeds_gpu import _check_hits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [1, 2, 31, 32, 33, 500, 4095, 4096, 4097])
def test_caps_over_tied_and_steep_rows(ctx, cap):
    rng = np.random.default_rng(cap)
    flat = np.full((9, 21), 2, dtype=np.int32)
    steep = np.full((12, 21), -4, dtype=np.int32)
    steep[np.arange(12), rng.integers(0, 20, 12)] = 9
    rows = [flat, steep, rng.integers(-1, 2, size=(20, 21)).astype(np.int32),
            rng.integers(-30, 31, size=(25, 21)).astype(np.int32)]
    targets = [rng.integers(0, 20, int(rng.integers(10, 120))).astype(np.uint8) for _ in range(80)]
    for mask, thr in (("1101", 2), ("11", 1), ("11011", -3)):
        st = _check_hits(ctx, rows, None, targets, mask,
                         PrefilterParams(kmer_score=thr, max_kmers_per_pos=cap, exact_seeds=False))
        if 20 ** mask.count("1") > cap:  # the flat rows' windows reach the threshold with every k-mer
            assert st["windows_at_cap"] > 0


def test_exact_seeds_inside_and_outside_the_cap(ctx):
    rng = np.random.default_rng(6)
    qs = [rng.integers(0, 21, 60).astype(np.uint8) for _ in range(4)]
    rows = [rng.integers(-3, 4, size=(60, 21)).astype(np.int32) for _ in range(4)]
    targets = [rng.integers(0, 20, 200).astype(np.uint8) for _ in range(100)]
    for cap in (1, 40, 700):
        st = _check_hits(ctx, rows, qs, targets, "110101", PrefilterParams(kmer_score=4, max_kmers_per_pos=cap))
        assert st["exact_seeds_added"] > 0
