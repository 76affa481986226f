"""The scan kernel's failure path, role by role and in the middle of the work: a role's wait runs out
at a CTA's first, second or tenth unit (a block of positions and the tiles of its group) while the others
have jobs in flight.  Every role has to leave, the call reports BLAMM_ERR_TIMEOUT, and the same context
then scans correctly.  Three tiles a unit, so that both issuers, both accumulators and every order of the
two come up; long two-term motifs for the streamed tiles."""
import pytest

import oracle
from bankutil import make_bank, make_stream, same_hits
from blamm_gb300 import BlammError
from blamm_gb300._native import BLAMM_ERR_TIMEOUT

pytestmark = pytest.mark.gpu

DRAINS, ONE_DRAIN, LOADER, ISSUER, CHUNKS = 2, 3, 4, 5, 6


def _check(scanner, mode, bank, stalls, n):
    P, lens, thr = bank
    bases, runs = make_stream(92, n, nruns=5)
    scanner.set_mode(mode)
    scanner.set_motifs(P, lens, thr)
    want = oracle.scan(bases, runs, P, lens, thr)
    for role, unit in stalls:
        scanner.debug_stall(role | unit << 8, 2_000_000)  # about a millisecond of SM cycles
        try:
            with pytest.raises(BlammError) as e:
                scanner.scan(bases, runs)
            assert e.value.code == BLAMM_ERR_TIMEOUT
        finally:
            scanner.debug_stall(False)
        ok, msg = same_hits(scanner.scan(bases, runs), want)
        assert ok, (role, unit, msg)


@pytest.mark.parametrize("unit", [0, 1, 9])
@pytest.mark.parametrize("mode", ["bf16", "e4m3"])
def test_resident_tiles(scanner, mode, unit):
    bank = make_bank(91, 150, 5, 20, rel=0.95)  # 300 columns: three tiles
    _check(scanner, mode, bank, [(r, unit) for r in (DRAINS, ONE_DRAIN, LOADER, ISSUER)], 500_000)


@pytest.mark.parametrize("unit", [0, 1, 9])
def test_streamed_tiles(scanner, unit):
    bank = make_bank(93, 20, 100, 130, rel=0.7)
    _check(scanner, "bf16x2", bank, [(r, unit) for r in (DRAINS, ONE_DRAIN, LOADER, ISSUER, CHUNKS)], 500_000)
