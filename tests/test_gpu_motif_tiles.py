"""The tensor-core scan at the edges of its tiles: columns around 128 a tile, positions around
256 a block, motif lengths around the k-steps, banks that need several tile groups, and motifs
too long for shared memory (streamed A).  Exact against the oracle: hit set and score bits."""
import numpy as np
import pytest

import oracle
from bankutil import exact_window_scores, make_bank, make_stream, quantized_columns, same_hits

pytestmark = pytest.mark.gpu

TERMS = {"bf16x2": 2, "bf16": 1, "e4m3": 8}


def _check(scanner, mode, P, lens, thr, n, seed, nruns=3, lower=0.05):
    bases, runs = make_stream(seed, n, nruns=min(nruns, n), lower_frac=lower)
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    ok, msg = same_hits(scanner.scan(bases, runs), oracle.scan(bases, runs, P, lens, thr))
    assert ok, msg


@pytest.mark.parametrize("mode", list(TERMS))
@pytest.mark.parametrize("cols", [1, 127, 128, 129, 257])
def test_columns_at_tile_edges(scanner, mode, cols):
    P, lens, thr = make_bank(300 + cols, cols, 4, 30, rc=False, rel=0.8)
    _check(scanner, mode, P, lens, thr, 20_011, 301)


@pytest.mark.parametrize("mode", list(TERMS))
@pytest.mark.parametrize("n", [31, 32, 33, 255, 256, 257, 511, 513])
def test_positions_at_block_edges(scanner, mode, n):
    P, lens, thr = make_bank(310, 70, 3, 24, rel=0.6)
    thr[::7] = np.float32(-1e3)  # every window of those columns is a hit, up to the last position
    _check(scanner, mode, P, lens, thr, n, 311 + n)


@pytest.mark.parametrize("mode,length", [("bf16", 188), ("bf16", 189), ("bf16", 256), ("bf16x2", 93), ("bf16x2", 96),
                                         ("bf16x2", 189), ("bf16x2", 256), ("e4m3", 63), ("e4m3", 64)])
def test_long_motifs_resident_and_streamed(scanner, mode, length):
    """Raw sums and hits on both sides of the length at which a tile no longer fits."""
    P, lens, thr = make_bank(320 + length, 130, length - 3, length, rc=False, rel=0.5)
    bases, runs = make_stream(321, 6_000, nruns=2, lower_frac=0.02)
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    D = scanner.debug_scores(bases, 100, 300)
    want = exact_window_scores(bases, quantized_columns(P, lens, TERMS[mode]), lens, 100, 300)
    assert np.array_equal(D.astype(np.float64), want)
    ok, msg = same_hits(scanner.scan(bases, runs), oracle.scan(bases, runs, P, lens, thr))
    assert ok, msg


@pytest.mark.parametrize("mode", list(TERMS))
@pytest.mark.parametrize("n", [700, 150_001])
def test_several_tile_groups(scanner, mode, n):
    """A bank larger than shared memory; few blocks (ranges of units) and many (interleaved)."""
    P, lens, thr = make_bank(330, 1100, 5, 30, rel=0.9)
    _check(scanner, mode, P, lens, thr, n, 331, nruns=9)


@pytest.mark.parametrize("mode", list(TERMS))
def test_threshold_zero_with_masked_windows(scanner, mode):
    """A window of lowercase bases scores +0: it is a hit of a column with threshold 0, and none
    of one with the least positive threshold."""
    P, lens, thr = make_bank(340, 9, 5, 12, rel=0.9)
    thr[0::3], thr[1::3] = np.float32(0.0), np.float32(1.1754944e-38)
    bases, runs = make_stream(341, 4_000, nruns=2)
    bases[500:2500] |= 0x20
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    ok, msg = same_hits(scanner.scan(bases, runs), oracle.scan(bases, runs, P, lens, thr))
    assert ok, msg
