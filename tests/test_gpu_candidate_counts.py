"""counts[3] of an enqueued scan is the number of candidates whether or not their records fit the
reservation: it is what the caller reserves room for before the scan is run again."""
import numpy as np
import pytest

from bankutil import make_bank, make_stream, same_hits
from blamm_gb300 import HIT_DTYPE

pytestmark = pytest.mark.gpu


def _long_bank():
    """Motifs whose tiles are streamed with two BF16 terms; some 3 % of the windows are hits."""
    P, lens, _ = make_bank(953, 20, 100, 130)
    rows, bg = P.reshape(len(lens), -1, 4).astype(np.float64), np.array([0.3, 0.2, 0.2, 0.3])
    mean = (rows * bg).sum((1, 2))  # (rows beyond a column's length are zero)
    sd = np.sqrt(((rows ** 2) * bg).sum((1, 2)) - (((rows * bg).sum(2)) ** 2).sum(1))
    return P, lens, (mean + 1.9 * sd).astype(np.float32)


@pytest.mark.parametrize("mode,long", [("bf16", False), ("bf16x2", False), ("e4m3", False), ("bf16x2", True)])
def test_candidates_beyond_the_reservation_are_counted(mode, long):
    torch = pytest.importorskip("torch")
    from blamm_gb300 import GpuScanner
    P, lens, thr = _long_bank() if long else make_bank(951, 60, 5, 20, rel=0.8)
    bases, runs = make_stream(952, 1_500_017, nruns=4, lower_frac=0.0 if long else 0.01)
    ref, sc = GpuScanner(0, mode), GpuScanner(0, mode)
    try:
        ref.set_motifs(P, lens, thr)
        want = ref.scan(bases, runs)
        ncand = ref.stats()["candidates"]
        sc.set_motifs(P, lens, thr)
        d_b, d_r = torch.from_numpy(bases).cuda(), torch.from_numpy(runs).cuda()
        d_h = torch.empty((len(want) + 1) * HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        d_c = torch.zeros(4, dtype=torch.int64, device="cuda")

        def enqueue(room):
            sc.reserve(len(bases), room)
            torch.cuda.synchronize()
            sc.enqueue(d_b.data_ptr(), len(bases), d_r.data_ptr(), len(runs), d_h.data_ptr(), len(want) + 1, d_c.data_ptr())
            torch.cuda.synchronize()
            return [int(x) for x in d_c]

        few = enqueue(0)
        assert few[1] < len(want) and few[2] == 0  # some records did not fit
        assert few[3] == ncand
        enough = enqueue(few[3])
        assert enough[1] == len(want) and enough[3] == ncand
        got = d_h.cpu().numpy().view(HIT_DTYPE)[:len(want)]
        ok, msg = same_hits(got, want)
        assert ok, msg
    finally:
        ref.close()
        sc.close()


def test_enqueue_behind_a_scan_without_a_reservation():
    """The buffers that an ordinary scan of the same stream left behind hold an enqueued one too."""
    torch = pytest.importorskip("torch")
    from blamm_gb300 import GpuScanner
    P, lens, thr = make_bank(961, 60, 5, 20, rel=0.9)
    bases, runs = make_stream(962, 1_000_003, nruns=4)
    sc = GpuScanner(0, "bf16")
    try:
        sc.set_motifs(P, lens, thr)
        d_b, d_r = torch.from_numpy(bases).cuda(), torch.from_numpy(runs).cuda()
        cap = 1 << 20
        d_h = torch.zeros(cap * HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        d_c = torch.zeros(4, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        args = (d_b.data_ptr(), len(bases), d_r.data_ptr(), len(runs), d_h.data_ptr(), cap)
        nh = sc.scan_device(*args)
        want = d_h.cpu().numpy().view(HIT_DTYPE)[:nh].copy()
        d_h.zero_()
        torch.cuda.synchronize()
        sc.enqueue(*args, d_c.data_ptr())
        torch.cuda.synchronize()
        assert int(d_c[1]) == nh > 10_000
        ok, msg = same_hits(d_h.cpu().numpy().view(HIT_DTYPE)[:nh], want)
        assert ok, msg
    finally:
        sc.close()
