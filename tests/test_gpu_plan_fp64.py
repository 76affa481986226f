"""Candidate thresholds are formed in FP64: the number of candidates is that of the FP64 bound.

A window is a candidate iff its quantised sum (exact, here in integers of the accumulator's unit u) reaches
T = floor of the largest of: threshold - guard, and over 64 values of lambda
lambda thr' + sum_j min(0, min_b (q - lambda P)).  The kernel picks lambda in FP32, where neighbouring
values may tie to a fraction of a unit, and its floor may then be one unit lower: so the count lies between
those for T and T - 1.  A threshold formed in FP32 with a margin for that is about (L + 8) 2^-23 sum |P|
lower, 5 to 10 units here.
"""
import numpy as np
import pytest

from bankutil import exact_window_scores, make_bank, make_stream, quantized_columns

pytestmark = pytest.mark.gpu

LAMBDAS = np.array([0.0, 1.0] + [1.0 - 2.0 ** (-1.0 - 0.875 * (i - 2)) for i in range(2, 16)]
                   + [1.0 + 2.0 ** (-14.0 + 0.34 * (i - 16)) for i in range(16, 64)])


def _unit(col, terms):
    f, e = np.frexp(np.abs(col).max())
    e = int(e) - (1 if f == 0.5 else 0)
    return 2.0 ** (e - 15)  # BF16: 2^-(k + 8), k = 7 - e; E4M3: 2^-(9 + k), k = 6 - e


def _threshold(P, q, thr, L, unit):
    """T in units."""
    x, q = P[:4 * L].astype(np.float64).reshape(L, 4) / unit, q[:4 * L].reshape(L, 4) / unit
    u, t = 2.0 ** -24, float(thr) / unit
    guard = np.maximum(0, (x - q).max(1)).sum() + (L - 1) * u / (1 - (L - 1) * u) * np.abs(x).max(1).sum()
    low = t - L * u * np.abs(x).max(1).sum()
    bounds = [lam * low + np.minimum(0, (q - lam * x).min(1)).sum() for lam in LAMBDAS]
    return np.floor(max(t - guard, max(bounds)))


@pytest.mark.parametrize("mode,terms", [("bf16", 1), ("bf16x2", 2), ("e4m3", 8)])
def test_candidates_of_the_fp64_bound(scanner, mode, terms):
    P, lens, thr = make_bank(931, 40, 14, 30, rc=False, rel=0.55)
    n = 300_000
    bases, runs = make_stream(932, n)
    Q = quantized_columns(P, lens, terms)
    S = exact_window_scores(bases, Q, lens, 0, n)
    at_t = below = 0
    for c in range(len(lens)):
        unit = _unit(P[c, :4 * lens[c]], terms)
        T = _threshold(P[c], Q[c], thr[c], int(lens[c]), unit)
        s = S[:, c] / unit
        at_t += int((s >= T).sum())
        below += int((s >= T - 1).sum())
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    hits = scanner.scan(bases, runs)
    got = scanner.stats()["candidates"]
    assert len(hits) <= at_t <= got <= below, (len(hits), at_t, got, below)
