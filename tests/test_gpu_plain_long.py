"""The plain FP32 form beyond the 32 motif positions whose offsets are kept, and with column groups of one,
two and three: lengths around multiples of 32 and up to the longest, masked bases, runs shorter and longer
than the motif.  Hits and score bits against the oracle, histograms against the restatement in numpy."""
import numpy as np
import pytest

import oracle
from bankutil import make_bank, make_stream, same_hits
from test_gpu_plain_edges import _hist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 2, 3, 6])
@pytest.mark.parametrize("lengths", [(30, 33), (62, 65), (95, 97), (127, 300), (1023, 1024)])
def test_hits(scanner, cols, lengths):
    P, lens, thr = make_bank(970 + cols + lengths[0], cols, *lengths, rc=False, rel=0.55)
    bases, runs = make_stream(971 + cols, 9_001, nruns=6, lower_frac=0.1)
    scanner.set_mode("fp32")
    scanner.set_motifs(P, lens, thr)
    want = oracle.scan(bases, runs, P, lens, thr)
    assert len(want) > 0
    ok, msg = same_hits(scanner.scan(bases, runs), want)
    assert ok, msg


@pytest.mark.parametrize("cols", [1, 2, 5])
@pytest.mark.parametrize("lengths", [(32, 33), (60, 200)])
def test_histograms(scanner, cols, lengths):
    P, lens, thr = make_bank(980 + cols, cols, *lengths, rc=False)
    bases, runs = make_stream(981, 12_011, nruns=7, lower_frac=0.1)
    rows = P.reshape(len(lens), -1, 4)
    mn, mx = rows.min(2).sum(1), rows.max(2).sum(1)
    width = ((mx - mn) / np.float32(250)).astype(np.float32)
    scanner.set_motifs(P, lens, thr)
    got = scanner.score_histograms(bases, runs, mn, width, 250)
    assert np.array_equal(got, _hist(bases, runs, P, lens, mn, width, 250))
