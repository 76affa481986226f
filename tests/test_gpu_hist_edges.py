"""Theoretical histograms where their parts meet: two bins (the host library's least) to 2500, one position to the longest
motif, key ranges on both sides of the small arrays, counts too large for exact sums, shared
distributions, p-values outside (0, 1).  Exact against the host library, which restates the
reference operation for operation."""
import numpy as np
import pytest

import oracle
from blamm_gb300 import BlammError, workloads
from blamm_gb300._native import MotifBank

pytestmark = pytest.mark.gpu

BG = np.array([0.31, 0.19, 0.21, 0.29], dtype=np.float32)


def _bank(seed, n, lmin, lmax, revcompl=True):
    rng = np.random.default_rng(seed)
    bank = MotifBank.from_pfms([p for _, p in workloads.random_pfms(rng, n, lmin, lmax)], revcompl=revcompl)
    bank.generate((BG * 1000).astype(np.uint64), 0.25)
    return bank, *bank.matrix()[:2]


@pytest.mark.parametrize("nbins", [2, 31, 250, 257, 1024, 1025, 2500])
@pytest.mark.parametrize("lengths", [(1, 3), (5, 30), (60, 90)])
def test_thresholds_for_bins_and_lengths(scanner, nbins, lengths):
    bank, P, lens = _bank(nbins + lengths[0], 24, *lengths)
    pvals = (0.5, 1e-2, 1e-4)
    thr, _ = scanner.theoretical_hist(P, lens, BG, pvals, hist_of=bank.hist_columns(), nbins=nbins)
    for v, p in enumerate(pvals):
        want = bank.pvalue_thresholds(BG, p, nbins=nbins)
        assert np.array_equal(thr[v].view(np.uint32), want.view(np.uint32)), f"p={p}"


@pytest.mark.parametrize("max_length", [1, 1000, 1 << 40, 1 << 62])
def test_counts_beyond_exact_sums(scanner, max_length):
    bank, P, lens = _bank(7, 16, 5, 20)
    thr, _ = scanner.theoretical_hist(P, lens, BG, (1e-3, 1e-5), hist_of=bank.hist_columns(), max_length=max_length)
    for v, p in enumerate((1e-3, 1e-5)):
        want = bank.pvalue_thresholds(BG, p, max_length=max_length)
        # (no observations at all: 0 / 0, whose NaN has other bits on the host)
        bits = np.where(np.isnan(want), np.isnan(thr[v]), thr[v].view(np.uint32) == want.view(np.uint32))
        assert bits.all(), f"p={p}"


def test_extreme_p_values(scanner):
    bank, P, lens = _bank(8, 12, 5, 20)
    pvals = (0.0, 1.0, 2.0, -1.0)
    thr, _ = scanner.theoretical_hist(P, lens, BG, pvals, hist_of=bank.hist_columns())
    for v, p in enumerate(pvals):
        want = bank.pvalue_thresholds(BG, p)
        assert np.array_equal(thr[v], want, equal_nan=True), f"p={p}"


def test_shared_distributions_give_every_user_the_same(scanner):
    _, P, lens = _bank(9, 20, 5, 20, revcompl=False)
    of = np.array([3, 3, 7, 7, 7] + [11] * 15, dtype=np.int32)
    alone, c1 = scanner.theoretical_hist(P, lens, BG, (1e-4,), counts=True)
    shared, c2 = scanner.theoretical_hist(P, lens, BG, (1e-4,), hist_of=of, counts=True)
    assert np.array_equal(shared[0], alone[0][of]) and np.array_equal(c2, c1[of])


@pytest.mark.parametrize("height,refused", [(0.05, False), (0.2, False), (100.0, True)])
def test_wide_key_ranges_run_again_or_are_refused(scanner, height, refused):
    """20 rows of +height, 20 of -height and a range of 1 in the last: the prefixes reach
    18000 x height keys beyond the histogram's 900 (more than 2048 are run again, more than
    8192 refused)."""
    P = np.full((1, 160), np.float32(height), dtype=np.float32)
    P[0, 80:] = -np.float32(height)
    P[0, 156:] += np.float32([0.0, 0.3, 0.6, 1.0])
    lens = np.array([40], dtype=np.int32)
    if refused:
        with pytest.raises(BlammError):
            scanner.theoretical_hist(P, lens, BG, (1e-2,), nbins=900)
        return
    _, cnt = scanner.theoretical_hist(P, lens, BG, (1e-2,), nbins=900, counts=True)
    assert np.array_equal(cnt[0], oracle.theoretical_hist(P[0].reshape(40, 4), BG, 900, 10_000_000))
