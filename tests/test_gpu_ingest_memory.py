"""The device memory that blamm_stream_load_fasta is documented to take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1, 32_768, 32_769, 3_000_000])
def test_memory_of_a_loaded_text(size):
    from blamm_gb300 import GpuScanner
    raw = (b">s\n" + np.random.default_rng(size).choice(np.frombuffer(b"ACGTN", np.uint8), size=size).tobytes())[:size]
    sc = GpuScanner(0)
    try:
        before = sc.call_bytes()
        nb, nr, ns, _ = sc.stream_load_fasta(raw)
        took = sc.call_bytes() - before
        want = len(raw) + nb + 8 * (3 * nr + ns) + 4704 * -(-len(raw) // 32_768)
        assert want <= took <= want + 256  # (the totals, and arrays of at least one element)
    finally:
        sc.close()
