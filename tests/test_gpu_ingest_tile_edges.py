"""GPU FASTA ingest at the edges of its 32 KB tiles (a tile: 16 warps of 2 KB): one-line sequences, headers
and gaps that end there, and sequence data before the first header that is only found when the tiles are put
together.  Exact against the oracle's restatement of FastaBatch."""
import numpy as np
import pytest

from blamm_gb300 import BlammError
from test_gpu_ingest_tiles import _check, _parse, _seq

pytestmark = pytest.mark.gpu

TILE, WARP = 32_768, 2_048


@pytest.mark.parametrize("size", [TILE - 4, TILE - 3, TILE - 2, TILE - 1, TILE, TILE + 1, 2 * TILE - 3, 2 * TILE + 1])
def test_one_line_sequences(scanner, tmp_path, size):
    rng = np.random.default_rng(size)
    _check(scanner, tmp_path, b">a\n" + _seq(rng, size) + b"\n>b\n" + _seq(rng, size) + b"\n")


@pytest.mark.parametrize("size", [WARP - 1, WARP, TILE - 1, TILE, 3 * TILE])
def test_long_headers_and_gaps(scanner, tmp_path, size):
    rng = np.random.default_rng(size)
    raw = b">" + _seq(rng, size, b"ACGT> ") + b"\n" + _seq(rng, 40) + b"N" * size + _seq(rng, 40, b"ACGT>") + b"\n"
    _check(scanner, tmp_path, raw + b"\n" * size + _seq(rng, 5) + b"\n>\n" + _seq(rng, 90) + b"\n")


@pytest.mark.parametrize("at", [TILE - 1, TILE, TILE + 3, 2 * TILE, 5 * TILE + 7])
@pytest.mark.parametrize("bare", [b"A", b"N"])
def test_data_before_the_first_header_in_a_later_tile(scanner, tmp_path, at, bare):
    """Refused when nothing but newlines comes before it, not when a header does, whatever tile that is in."""
    with pytest.raises(BlammError):
        _parse(scanner, b"\n" * at + bare + b"\n>s\nACGT\n")
    with pytest.raises(BlammError):
        _parse(scanner, b"\n" * at + bare)
    assert _parse(scanner, b"\n" * at + b">s\nACGT\n")[1].tolist() == [0]
    _check(scanner, tmp_path, b">s\n" + b"\n" * at + bare + b"\n>t\nACGT\n")
    _check(scanner, tmp_path, b"\n" * (at // 2) + b">s\n" + b"\n" * (at - at // 2) + bare + b"CGT\n")
