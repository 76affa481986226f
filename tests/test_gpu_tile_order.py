"""Two BF16 terms over two to five tiles a unit, where every other unit takes its tiles in reverse: around
the numbers of tiles and the motif length at which that begins and ends, with one, two and many units a CTA,
units dealt in ranges, and banks cut into groups.  Hits and score bits against the oracle."""
import numpy as np
import pytest

import oracle
from bankutil import make_bank, make_stream, same_hits

pytestmark = pytest.mark.gpu


def _check(scanner, bank, n, nruns=4):
    P, lens, thr = bank
    bases, runs = make_stream(n, n, nruns=nruns, lower_frac=0.02)
    scanner.set_mode("bf16x2")
    scanner.set_motifs(P, lens, thr)
    ok, msg = same_hits(scanner.scan(bases, runs), oracle.scan(bases, runs, P, lens, thr))
    assert ok, msg


@pytest.mark.parametrize("cols", [128, 129, 257, 384, 640, 641])
@pytest.mark.parametrize("lmax", [20, 21])  # 5 k-steps, 6
def test_tiles_and_lengths(scanner, cols, lmax):
    P, lens, thr = make_bank(1000 + cols, cols, 5, lmax, rc=False, rel=0.85)
    lens[-1] = lmax  # (columns come by length; the values beyond a column's length are not used)
    assert P.shape[1] >= 4 * lmax
    _check(scanner, (P, lens, thr), 120_000)


@pytest.mark.parametrize("n", [200, 257, 20_000, 39_000, 80_000, 400_001])
def test_units_per_cta(scanner, n):
    _check(scanner, make_bank(1100, 300, 5, 28, rc=False, rel=0.85), n, nruns=3)


@pytest.mark.parametrize("cols,lo,hi", [(400, 30, 60), (900, 20, 44), (260, 80, 89)])
def test_groups(scanner, cols, lo, hi):
    _check(scanner, make_bank(1200 + cols, cols, lo, hi, rc=False, rel=0.7), 60_000)
