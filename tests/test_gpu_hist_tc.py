"""Empirical histograms on the tensor cores at the edges of their parts: columns around a tile's
64, lengths around the k-steps of four positions (one is taken by the shifted rows), streams
around the blocks of 512 positions, runs shorter and longer than a block, masked bases, bins
from one to many, scores on bin boundaries and beyond the bins.  Exact against a restatement in
numpy.  Streams long enough for this form."""
import numpy as np
import pytest

from bankutil import make_bank, make_stream
from test_gpu_plain_edges import _hist

pytestmark = pytest.mark.gpu


def _check(scanner, P, lens, bases, runs, mn, width, nbins):
    scanner.set_motifs(P, lens, np.zeros(len(lens), np.float32))
    got = scanner.score_histograms(bases, runs, mn, width, nbins)
    assert np.array_equal(got, _hist(bases, runs, P, lens, mn, width, nbins))


def _bins(P, lens, nbins):
    rows = P.reshape(len(lens), -1, 4)
    mn, mx = rows.min(2).sum(1), rows.max(2).sum(1)
    return mn, ((mx - mn) / np.float32(nbins)).astype(np.float32)


@pytest.mark.parametrize("cols,lengths,nbins", [
    (64, (6, 20), 250), (63, (3, 4), 31), (65, (11, 12), 250), (130, (5, 9), 1), (34, (4, 30), 700), (17, (15, 33), 64),
    (20, (40, 47), 100), (128, (7, 8), 250)])
def test_columns_lengths_and_bins(scanner, cols, lengths, nbins):
    P, lens, _ = make_bank(440 + cols, cols, *lengths, rc=False)
    bases, runs = make_stream(441, 480_011, nruns=9, lower_frac=0.05)
    _check(scanner, P, lens, bases, runs, *_bins(P, lens, nbins), nbins)


@pytest.mark.parametrize("n,nruns,lower", [(262_143, 1, 0.0), (262_144, 1, 0.0), (262_145, 2, 0.5), (262_655, 600, 0.05),
                                           (300_000, 9_000, 0.0)])
def test_streams_and_runs(scanner, n, nruns, lower):
    P, lens, _ = make_bank(450, 40, 5, 18, rc=False)
    bases, runs = make_stream(451 + nruns, n, nruns=nruns, lower_frac=lower)
    _check(scanner, P, lens, bases, runs, *_bins(P, lens, 250), 250)


def test_scores_on_boundaries_and_beyond_the_bins(scanner):
    """Scores that are multiples of the bin width to rounding, bins that cover a part of the
    scores, values of very different size."""
    lens = np.full(48, 7, dtype=np.int32)
    P = np.tile(np.float32([0.0, 0.1, 0.2, 0.3]), (48, 7))
    P[16:32] = np.tile(np.float32([-0.3, 0.7, 2.1, 0.0]), (16, 7))
    P[32:] *= (np.float32(10.0) ** np.arange(-8, 8)).astype(np.float32)[:, None]
    mn = np.zeros(48, np.float32)
    mn[16:32] = np.linspace(-2.1, 4.0, 16, dtype=np.float32)
    width = np.full(48, 0.1, np.float32)
    width[8:16] = 0.3
    width[24:32] = 0.05
    width[32:] = (np.float32(0.1) * np.float32(10.0) ** np.arange(-8, 8)).astype(np.float32)
    bases, runs = make_stream(461, 350_000, nruns=3, lower_frac=0.2)
    _check(scanner, P, lens, bases, runs, mn, width, 40)
