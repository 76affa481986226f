"""GPU FASTA ingest at the edges of warps (2 KB), written parts (16 KB) and tiles (32 KB): gaps,
headers and line ends that start, end or lie there, in text with few and with many bytes per
piece that are no bases.  Exact against the oracle's restatement of FastaBatch."""
import numpy as np
import pytest

from test_gpu_ingest_tiles import _check, _seq

pytestmark = pytest.mark.gpu

WARP, PART, TILE = 2_048, 16_384, 32_768


@pytest.mark.parametrize("width", [12, 13, 21, 60, 64, 1_000])
@pytest.mark.parametrize("at", [WARP, PART, TILE, 2 * TILE])
def test_gaps_and_headers_at_edges(scanner, tmp_path, at, width):
    """Base lines with an N run and a header line placed one byte before, at and after an edge."""
    rng = np.random.default_rng([at, width])
    for shift in (-1, 0, 1):
        for insert in (b"N" * 3, b"N" * 130, b"\n>next\n", b"\n>" + _seq(rng, 300, b"ACGT>") + b"\nN", b"\n\n"):
            body = b"\n".join(_seq(rng, width, b"ACGTacgt") for _ in range(at // width + 2))
            text = b">first\n" + body
            raw = text[:at + shift] + insert + _seq(rng, 5 * width) + b"\n"
            _check(scanner, tmp_path, raw)


@pytest.mark.parametrize("tiles", [1, 2, 3])
def test_tiles_without_line_starts(scanner, tmp_path, tiles):
    """A header line or a base line over whole tiles: their sums depend on what came before."""
    rng = np.random.default_rng(tiles)
    long_header = b">" + _seq(rng, tiles * TILE + 77, b"ACGTN>") + b"\n"
    long_line = _seq(rng, tiles * TILE + 99) + b"\n"
    _check(scanner, tmp_path, long_header + long_line + long_header + long_line)
