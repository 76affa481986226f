"""Thresholds and banks are uploaded in order with the scans of their context: a scan that was enqueued
before a change uses the old values throughout, one after it the new ones."""
import numpy as np
import pytest

import oracle
from bankutil import make_bank, make_stream, same_hits
from blamm_gb300 import HIT_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
def test_thresholds_changed_behind_an_enqueued_scan(scanner, mode):
    torch = pytest.importorskip("torch")
    P, lens, thr = make_bank(701, 64, 6, 20, rel=0.9)
    higher = (thr + 0.5 * np.abs(thr)).astype(np.float32)
    bases, runs = make_stream(702, 8_000_000, nruns=5)
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    old = scanner.scan(bases, runs)
    d_b, d_r = torch.from_numpy(bases).cuda(), torch.from_numpy(runs).cuda()
    d_h = torch.empty(len(old) * HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    d_c = torch.zeros(4, dtype=torch.int64, device="cuda")
    scanner.reserve(len(bases), 4 * len(old))
    torch.cuda.synchronize()
    scanner.enqueue(d_b.data_ptr(), len(bases), d_r.data_ptr(), len(runs), d_h.data_ptr(), len(old), d_c.data_ptr())
    scanner.set_thresholds(higher)
    new = scanner.scan(bases, runs)
    assert int(d_c[1]) == len(old)
    ok, msg = same_hits(d_h.cpu().numpy().view(HIT_DTYPE), old)
    assert ok, msg
    keep = old["score"] >= higher[old["col"]]
    ok, msg = same_hits(new, old[keep])
    assert ok, msg


def test_banks_in_turn(scanner):
    scanner.set_mode("bf16")
    bases, runs = make_stream(703, 30_000, nruns=3)
    banks = [make_bank(704 + k, 40 + 300 * (k % 2), 5, 12 + 9 * k, rel=0.85) for k in range(3)]
    want = [oracle.scan(bases, runs, *b) for b in banks]
    for _ in range(4):
        for b, w in zip(banks, want):
            scanner.set_motifs(*b)
            ok, msg = same_hits(scanner.scan(bases, runs), w)
            assert ok, msg
