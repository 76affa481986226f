"""Candidate thresholds built on the device: columns whose threshold is at, below and above the
scores a window can reach, not a number, or infinite; flat columns; every length.  Exact against
the oracle, and the candidates stay near the hits."""
import numpy as np
import pytest

import oracle
from bankutil import make_bank, make_stream, same_hits

pytestmark = pytest.mark.gpu

MODES = ["bf16", "bf16x2", "e4m3"]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("seed", [0, 1])
def test_thresholds_at_the_ends_of_the_score_range(scanner, mode, seed):
    P, lens, thr = make_bank(500 + seed, 70, 1, 30, rel=0.85)
    for c in range(len(lens)):
        rows = P[c, :4 * lens[c]].reshape(-1, 4)
        mn, mx = oracle.min_max_score(rows)
        thr[c] = [thr[c], mx, np.nextafter(mx, np.float32(np.inf)), mn, np.nextafter(mn, np.float32(-np.inf)),
                  np.float32(np.inf), np.float32(-np.inf), np.float32(np.nan), np.float32(1e30), np.float32(-1e30),
                  (mn + mx) / 2, np.float32(0.0)][c % 12]
    P[5, :4 * lens[5]] = np.float32(0.25)  # a flat column: every window scores the same
    thr[5] = np.float32(0.25) * np.float32(lens[5])
    P[17, :4 * lens[17]] = 0.0
    thr[17] = 0.0
    bases, runs = make_stream(510 + seed, 3_000, nruns=4, lower_frac=0.1)
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    ok, msg = same_hits(scanner.scan(bases, runs), oracle.scan(bases, runs, P, lens, thr))
    assert ok, msg


@pytest.mark.parametrize("mode,most", [("bf16", 1.25), ("bf16x2", 1.02), ("e4m3", 1.35)])
def test_candidates_stay_near_the_hits(scanner, mode, most):
    """Strict thresholds, no masked bases, one run: candidates per hit."""
    P, lens, thr = make_bank(520, 100, 10, 30, rel=0.8)
    bases, runs = make_stream(521, 2_000_000)
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    hits = scanner.scan(bases, runs)
    st = scanner.stats()
    assert len(hits) > 1000 and len(hits) <= st["candidates"] <= most * len(hits)
