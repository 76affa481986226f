"""GPU FASTA ingest at the edges of its pieces (64 bytes a thread, 16 KB a tile): lines, headers
and gaps that span them, '>' inside lines, texts that end anywhere, text at any alignment.
Exact against the oracle's restatement of FastaBatch."""
import numpy as np
import pytest

from test_host_cpu import _oracle_stream

pytestmark = pytest.mark.gpu

TILE = 16_384


def _parse(scanner, raw: bytes, shift: int = 0):
    torch = pytest.importorskip("torch")
    n = len(raw)
    d_raw = torch.frombuffer(bytearray(b"\n" * shift + raw), dtype=torch.uint8).cuda()[shift:]
    d_b = torch.zeros(n + 5, dtype=torch.uint8, device="cuda")[shift % 5:]
    t = [torch.empty(n, dtype=torch.int64, device="cuda") for _ in range(4)]
    nucl = np.zeros(4, dtype=np.uint64)
    nb, nr, ns = scanner.fasta_parse_device(d_raw.data_ptr(), n, d_b.data_ptr(), *(x.data_ptr() for x in t), nucl)
    return d_b[:nb].cpu().numpy(), *(x[:nr].cpu().numpy() for x in t[:3]), t[3][:ns].cpu().numpy(), nucl


def _check(scanner, tmp_path, raw: bytes, shift: int = 0):
    f = tmp_path / "x.fa"
    f.write_bytes(raw)
    want = _oracle_stream([str(f)])
    got = _parse(scanner, raw, shift)
    for name, g, w in zip(("bases", "run_start", "run_seq", "run_seqpos"), got, want):
        assert np.array_equal(g, w), f"{name}: {g[:8]} vs {w[:8]}"
    starts = [0] if raw[:1] == b">" else []
    starts += [i + 1 for i in range(len(raw) - 1) if raw[i:i + 2] == b"\n>"]
    assert got[4].tolist() == starts
    low = np.asarray(want[0]) | 0x20
    assert [int(x) for x in got[5]] == [int(np.count_nonzero(low == ord(c))) for c in "acgt"]


def _seq(rng, n, alphabet=b"ACGTacgtN"):
    return rng.choice(np.frombuffer(alphabet, dtype=np.uint8), size=n).tobytes()


@pytest.mark.parametrize("size", [1, 62, 63, 64, 65, TILE - 4, TILE - 3, TILE - 2, TILE, 2 * TILE + 1])
def test_one_line_sequences(scanner, tmp_path, size):
    """No newline for whole tiles: a tile does not know what line it starts in."""
    rng = np.random.default_rng(size)
    _check(scanner, tmp_path, b">a\n" + _seq(rng, size) + b"\n>b\n" + _seq(rng, size) + b"\n")


@pytest.mark.parametrize("size", [60, 61, 62, TILE - 1, TILE, 3 * TILE])
def test_long_headers_and_gaps(scanner, tmp_path, size):
    """Headers of bases and '>' and N runs that cover pieces and tiles."""
    rng = np.random.default_rng(size)
    raw = b">" + _seq(rng, size, b"ACGT> ") + b"\n" + _seq(rng, 40) + b"N" * size + _seq(rng, 40, b"ACGT>") + b"\n"
    _check(scanner, tmp_path, raw + b"\n" * size + _seq(rng, 5) + b"\n>" + b"\n>\n" * 70 + _seq(rng, 90) + b"\n")


@pytest.mark.parametrize("shift", [0, 1, 15])
def test_any_alignment_and_short_lines(scanner, tmp_path, shift):
    rng = np.random.default_rng(50 + shift)
    raw = b"".join(b">s%d\r\n" % i + b"".join(_seq(rng, int(rng.integers(0, 9))) + b"\r\n" for _ in range(40))
                   for i in range(60))
    _check(scanner, tmp_path, raw, shift)


def test_data_before_the_first_header_in_a_later_tile(scanner):
    from blamm_gb300 import BlammError
    with pytest.raises(BlammError):
        _parse(scanner, b"\n" * (TILE + 3) + b"A\n>s\nACGT\n")
    assert _parse(scanner, b"\n" * (TILE + 3) + b">s\nACGT\n")[1].tolist() == [0]
