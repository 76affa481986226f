"""The plain FP32 scan and the empirical histograms at the edges of their parts: columns around
the groups of four and the blocks' 64, lengths around the 32 positions kept in registers,
positions around the tiles of 256, masked bases, column subsets, bins kept in shared memory
and not, scores on bin boundaries.  Exact against the oracle / a restatement in numpy."""
import numpy as np
import pytest

import oracle
from bankutil import make_bank, make_stream, same_hits

pytestmark = pytest.mark.gpu


def _hist(bases, runs, P, lens, mn, width, nbins):
    """ScoreHistogram::addObservation over every window inside its run, FP32 in motif order."""
    code = np.full(len(bases) + 2048, 4)
    for b, ch in enumerate(b"ACGT"):
        code[:len(bases)][bases == ch] = b
    ends = np.append(runs[1:], len(bases))
    end = ends[np.searchsorted(runs, np.arange(len(bases)), side="right") - 1]
    out = np.zeros((len(lens), nbins), dtype=np.uint64)
    for c, L in enumerate(lens):
        pos = np.flatnonzero(np.arange(len(bases)) + L <= end)
        rows = np.concatenate([P[c, :4 * L].reshape(L, 4), np.zeros((L, 1), np.float32)], axis=1)
        s = np.zeros(len(pos), dtype=np.float32)
        for j in range(L):
            s = s + rows[j][code[pos + j]]
        b = np.clip(((s - mn[c]) / width[c]).astype(np.int64), 0, nbins - 1)
        out[c] = np.bincount(b, minlength=nbins)
    return out


@pytest.mark.parametrize("cols", [1, 3, 4, 5, 63, 64, 65, 130])
@pytest.mark.parametrize("lengths", [(1, 4), (5, 30), (31, 34), (60, 70)])
def test_plain_scan_columns_and_lengths(scanner, cols, lengths):
    P, lens, thr = make_bank(400 + cols, cols, *lengths, rc=False, rel=0.7)
    bases, runs = make_stream(401, 3_001, nruns=5, lower_frac=0.05)
    scanner.set_mode("fp32")
    scanner.set_motifs(P, lens, thr)
    ok, msg = same_hits(scanner.scan(bases, runs), oracle.scan(bases, runs, P, lens, thr))
    assert ok, msg


@pytest.mark.parametrize("n", [1, 255, 256, 257, 700_001])
def test_plain_scan_positions_and_subset(scanner, n):
    P, lens, thr = make_bank(410, 70, 3, 40, rel=0.75)
    bases, runs = make_stream(411 + n, n, nruns=min(n, 40), lower_frac=0.05)
    scanner.set_mode("fp32")
    scanner.set_motifs(P, lens, thr)
    sub = np.arange(1, len(lens), 3, dtype=np.int32)
    scanner.set_columns(sub)
    got = scanner.scan(bases, runs)
    scanner.set_columns(None)
    want = oracle.scan(bases, runs, P[sub], lens[sub], thr[sub])
    want["col"] = sub[want["col"]]
    ok, msg = same_hits(got, want)
    assert ok, msg


@pytest.mark.parametrize("cols,lengths,nbins", [(1, (5, 9), 250), (33, (5, 30), 250), (66, (30, 36), 100), (5, (4, 12), 1),
                                                (6, (4, 12), 20_000)])
def test_empirical_histograms(scanner, cols, lengths, nbins):
    P, lens, thr = make_bank(420 + cols, cols, *lengths, rc=False)
    bases, runs = make_stream(421, 20_011, nruns=7, lower_frac=0.05)
    rows = P.reshape(len(lens), -1, 4)
    mn, mx = rows.min(2).sum(1), rows.max(2).sum(1)
    width = ((mx - mn) / np.float32(nbins)).astype(np.float32)
    scanner.set_motifs(P, lens, thr)
    got = scanner.score_histograms(bases, runs, mn, width, nbins)
    assert np.array_equal(got, _hist(bases, runs, P, lens, mn, width, nbins))


def test_scores_on_bin_boundaries(scanner):
    """Scores that are multiples of the bin width, and widths whose reciprocal is not exact: the
    rounded quotient decides, also where the score is below the least one."""
    lens = np.full(6, 5, dtype=np.int32)
    P = np.tile(np.float32([0.0, 0.1, 0.2, 0.3]), (6, 5))
    P[3:] = np.tile(np.float32([-0.3, 0.7, 2.1, 0.0]), (3, 5))
    mn = np.float32([0.0, 0.1, 0.25, -1.5, 0.0, 1.0])
    width = np.float32([0.1, 0.3, 0.05, 0.7, 1e-30, 3.0])
    bases, runs = make_stream(431, 50_000, nruns=3)
    scanner.set_motifs(P, lens, np.zeros(6, np.float32))
    got = scanner.score_histograms(bases, runs, mn, width, 40)
    with np.errstate(all="ignore"):
        want = _hist(bases, runs, P, lens, mn, np.maximum(width, np.float32(1e-18)), 40)
    assert np.array_equal(got, want)
