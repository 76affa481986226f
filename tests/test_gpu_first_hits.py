"""Hits of a host scan around the number (512 at least) that comes back with the counters: a word planted a
given number of times, found each time, in buffers with and without room for all."""
import ctypes as C

import numpy as np
import pytest

from blamm_gb300 import HIT_DTYPE
from blamm_gb300._native import BLAMM_ERR_OVERFLOW, _ptr

pytestmark = pytest.mark.gpu

WORD = np.frombuffer(b"CGGTCCGTGGCTCGTC", dtype=np.uint8)


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
@pytest.mark.parametrize("hits,room", [(0, 10), (1, 1), (511, 600), (512, 600), (513, 600), (700, 700), (700, 699), (700, 512),
                                       (700, 511), (700, 0)])
def test_planted_words(scanner, mode, hits, room):
    L = len(WORD)
    bases = np.full(60_000, ord("A"), dtype=np.uint8)
    at = 37 + 80 * np.arange(hits)
    for a in at:
        bases[a:a + L] = WORD
    P = np.full((1, 4 * L), -1.0, dtype=np.float32)
    P[0, 4 * np.arange(L) + np.searchsorted(np.frombuffer(b"ACGT", dtype=np.uint8), WORD)] = 1.0
    scanner.set_mode(mode)
    scanner.set_motifs(P, np.array([L], np.int32), np.array([L], np.float32))
    out = np.zeros(room + 1, dtype=HIT_DTYPE)
    out["col"] = -7  # what is not written stays
    n, runs = C.c_int64(0), np.zeros(1, np.int64)
    rc = scanner.lib.blamm_scan(scanner.h, _ptr(bases), len(bases), _ptr(runs), 1, _ptr(out), room, C.byref(n))
    assert rc == (BLAMM_ERR_OVERFLOW if hits > room else 0) and n.value == hits
    got = min(hits, room)
    assert (out["col"][:got] == 0).all() and (out["col"][got:] == -7).all() and (out["score"][:got] == L).all()
    pos = np.sort(out["pos"][:got])
    assert np.array_equal(pos, at) if hits <= room else set(pos.tolist()) <= set(at.tolist()) and len(set(pos.tolist())) == got
