"""What blamm_stats times: scan_ms is the scan kernel alone, rescore_ms the rescoring, kernel_ms all kernels
(the preparation of the stream too, which moves at least 17 bytes a position), total_ms the call with its
copies, by the host's clock."""
import time

import numpy as np
import pytest

from bankutil import make_bank, make_stream

pytestmark = pytest.mark.gpu

HBM_BYTES_PER_MS = 8.0e9  # above what the memory can move


@pytest.mark.parametrize("mode", ["bf16", "e4m3"])
@pytest.mark.parametrize("n", [16_777_216, 24_000_001])  # one scan window, two
def test_scan_time_is_the_scan_kernel_alone(scanner, mode, n):
    P, lens, thr = make_bank(901, 6, 8, 12, rel=0.95)
    bases, runs = make_stream(902, n, nruns=3)
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    t = []
    for _ in range(5):
        t0 = time.perf_counter()
        scanner.scan(bases, runs)
        s = scanner.stats() | {"wall": 1e3 * (time.perf_counter() - t0)}
        assert s["scan_ms"] > 0 and s["rescore_ms"] > 0
        assert s["kernel_ms"] - s["scan_ms"] - s["rescore_ms"] >= 17 * n / HBM_BYTES_PER_MS, s
        assert s["kernel_ms"] < s["total_ms"] <= s["wall"], s
        t.append(s["total_ms"])
    assert np.median(t) >= n / HBM_BYTES_PER_MS
