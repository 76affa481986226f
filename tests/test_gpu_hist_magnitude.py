"""Empirical histograms of scores of any size: banks scaled by powers of two around the largest value
whose fixed-point terms are exact (2^40), some columns or all of them.  Exact against the restatement in
numpy, on streams long enough for the tensor-core form."""
import numpy as np
import pytest

from bankutil import make_bank, make_stream
from test_gpu_hist_tc import _bins, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top", [39, 40, 41, 45, 55])
@pytest.mark.parametrize("some", [False, True])
def test_scores_of_any_size(scanner, top, some):
    P, lens, _ = make_bank(470, 48, 6, 18, rc=False)
    scale = 2.0 ** (top - np.ceil(np.log2(np.abs(P).max())))  # the largest |P| in (2^(top - 1), 2^top]
    P[20 if some else 0:] *= np.float32(scale)
    bases, runs = make_stream(471, 480_011, nruns=5, lower_frac=0.05)
    _check(scanner, P, lens, bases, runs, *_bins(P, lens, 250), 250)
