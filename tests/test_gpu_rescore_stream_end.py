"""Long motifs with negative thresholds at the end of a stream: every window that reaches beyond it is a
candidate (masked bases add nothing) and none is a hit.  The hits are the oracle's, and the rescoring does
not spend its time there: its slowest warp takes about as long as with one column, not ten times that."""
import numpy as np
import pytest

import oracle
from bankutil import make_bank, make_stream, same_hits

pytestmark = pytest.mark.gpu


def _bank(cols):
    P, lens, _ = make_bank(480, cols, 250, 250, rc=False)
    rows = P.reshape(cols, 250, 4).astype(np.float64)
    bg = np.array([0.3, 0.2, 0.2, 0.3])
    mean = (rows * bg).sum((1, 2))
    sd = np.sqrt(((rows ** 2) * bg).sum((1, 2)) - (((rows * bg).sum(2)) ** 2).sum(1))
    return P, lens, (mean + 3 * sd).astype(np.float32)


def _rescore_ms(scanner, bank, bases, runs):
    torch = pytest.importorskip("torch")
    scanner.set_motifs(*bank)
    d_b, d_r = torch.from_numpy(bases).cuda(), torch.from_numpy(runs).cuda()
    d_h = torch.empty(16 << 16, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ms = []
    for _ in range(11):
        scanner.scan_device(d_b.data_ptr(), len(bases), d_r.data_ptr(), len(runs), d_h.data_ptr(), 1 << 16)
        ms.append(scanner.stats()["rescore_ms"])
    return float(np.median(ms[2:]))


def test_windows_beyond_the_stream(scanner):
    scanner.set_mode("bf16x2")
    bases, runs = make_stream(481, 50_000, nruns=3)
    bank = _bank(64)
    assert (bank[2] < 0).all()
    scanner.set_motifs(*bank)
    got = scanner.scan(bases, runs)
    assert scanner.stats()["candidates"] > len(got) + 64 * 100  # the windows in question
    ok, msg = same_hits(got, oracle.scan(bases, runs, *bank))
    assert ok, msg
    assert _rescore_ms(scanner, bank, bases, runs) < 3 * _rescore_ms(scanner, _bank(1), bases, runs)
