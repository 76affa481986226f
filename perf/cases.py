"""Performance cases of the framework: the calls its users make, over the range they make them in.

A case is a dict of plain values; `kind` names the entry points it goes through:

  scan      hits of a base stream against a motif bank, through GpuScanner.scan ("host"), .scan_device
            ("device"), .scan_device_static ("static") or a captured graph ("graph")
  serve     a burst of requests through the scan service (Server.submit / .take)
  fastascan FASTA text to hits: .stream_load_fasta, .stream_tables, .scan_stream
  fasta     FASTA text on the device to the filtered stream and its tables (.fasta_parse_device)
  thr       theoretical score histograms and p-value thresholds (.theoretical_hist)
  emphist   empirical score histograms (.score_histograms)

Banks have forward and reverse-complement columns of motifs whose columns are Multinomial(100,
Dirichlet(0.5)) counts, as log2 odds with pseudocount 0.25; thresholds come from the score
distribution under the background at the case's p-value.  The library returns hits in no order;
the passes put them in order of position and column, as the command line does before it writes
them.  Outputs are buffers of the state of a size that the case gives, filled up to their counts.
Torch work on the library's buffers runs on the library's stream.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from blamm_gb300 import HIT_DTYPE, GpuScanner, Server

COL_BITS = 20  # a hit's key: position << 20 | column
ACGT = (65, 67, 71, 84)


# ---------------------------------------------------------------- the cases
def listed() -> list[dict]:
    scan = {"kind": "scan", "gc": 0.42, "tune": 0, "lower": 0.0, "nfrac": 0.0}
    return [
        # one promoter against a handful of motifs: the smallest call a script makes in a loop
        scan | {"name": "scan_one_promoter", "entry": "host", "mode": "auto", "n": 2_000, "runs": 1, "motifs": 20,
                "lmin": 6, "lmax": 20, "p": 1e-4},
        # the reference's own example size: 32 motifs over 2 x 500 kbp, host buffers
        scan | {"name": "scan_two_sequences", "entry": "host", "mode": "auto", "n": 1_000_000, "runs": 2,
                "motifs": 32, "lmin": 6, "lmax": 20, "gc": 0.4, "p": 1e-4},
        # a soft-masked chromosome arm with N runs and an odd length, two BF16 terms, allocation-free entry
        scan | {"name": "scan_masked_arm", "entry": "static", "mode": "bf16x2", "n": 3_333_331, "runs": 57,
                "motifs": 301, "lmin": 5, "lmax": 30, "lower": 0.3, "p": 1e-4},
        # 10,000 promoter-like sequences in one launch of a captured graph
        scan | {"name": "scan_promoters_graph", "entry": "graph", "mode": "auto", "n": 32_600_000, "runs": 10_000,
                "motifs": 800, "lmin": 6, "lmax": 25, "gc": 0.5, "p": 1e-4},
        # the headline: a 100 Mbp genome against 512 motifs, device-resident, after the autotuner
        scan | {"name": "scan_genome_tuned", "entry": "device", "mode": "auto", "tune": 1, "n": 100_000_000,
                "runs": 24, "motifs": 512, "lmin": 5, "lmax": 30, "p": 1e-4},
        # a big bank at a strict p-value, one E4M3 term
        scan | {"name": "scan_big_bank_e4m3", "entry": "device", "mode": "e4m3", "n": 12_345_678, "runs": 300,
                "motifs": 2000, "lmin": 5, "lmax": 30, "p": 1e-5},
        # the plain FP32 form (any motif length; the form others are compared with)
        scan | {"name": "scan_plain_fp32", "entry": "device", "mode": "fp32", "n": 2_000_003, "runs": 9,
                "motifs": 128, "lmin": 5, "lmax": 30, "p": 1e-4},
        # the scan service: a burst of requests of uneven length over subsets of a resident bank
        {"name": "serve_burst", "kind": "serve", "requests": 16, "nmin": 1_000, "nmax": 300_000, "motifs": 1000,
         "lmin": 5, "lmax": 30, "gc": 0.42},
        # from FASTA text in host memory to hits: what the command line does per piece
        {"name": "fasta_to_hits", "kind": "fastascan", "n": 8_000_000, "seqs": 12, "width": 60, "nfrac": 0.01,
         "motifs": 32, "lmin": 6, "lmax": 20, "gc": 0.42, "p": 1e-5},
        # ingest alone: a 100 MB FASTA text, 60 bases a line
        {"name": "fasta_ingest_genome", "kind": "fasta", "n": 100_000_000, "seqs": 24, "width": 60, "nfrac": 0.01,
         "lower": 0.3, "gc": 0.42},
        # thresholds of a 4000-column bank at three p-values
        {"name": "thresholds_big_bank", "kind": "thr", "motifs": 2000, "lmin": 5, "lmax": 30, "gc": 0.42, "bins": 250,
         "fp64": 0},
        # empirical histograms of a 64-column bank over 8 Mbp (the hist module looks at 10 Mbp at most)
        {"name": "empirical_hist", "kind": "emphist", "n": 8_000_000, "runs": 12, "motifs": 32, "lmin": 6, "lmax": 20,
         "gc": 0.4, "bins": 250, "lower": 0.0},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["scan", "scan", "scan", "scan", "serve", "fastascan", "fasta", "thr", "emphist"])
    lmin = rng.randint(5, 8)
    base = {"kind": kind, "lmin": lmin, "lmax": rng.randint(lmin + 6, 30), "gc": round(rng.uniform(0.35, 0.6), 3)}
    if kind == "scan":
        entry = rng.choice(["host", "static", "device", "device", "graph"])
        mode = rng.choice(["auto", "auto", "bf16x2", "e4m3", "fp32"])
        nmax = {"host": 2_000_000, "static": 4_000_000, "device": 60_000_000, "graph": 30_000_000}[entry]
        motifs = _log(rng, 3, 2000)
        if entry == "static":  # its record scratch is fixed
            nmax = min(nmax, 1e9 / motifs)
        # no more position x column pairs than the largest case (the plain form: a 100th of it)
        n = _log(rng, 1_000, min(nmax, 5e10 / motifs if mode != "fp32" else 5e8 / motifs))
        p = rng.choice([1e-3, 1e-4, 1e-5] if n * motifs < 2e9 and entry != "static" else [1e-4, 1e-5])
        return base | {"entry": entry, "mode": mode, "tune": 0, "n": n, "runs": min(_log(rng, 1, 5_000), 1 + n // 400),
                       "motifs": motifs, "lower": rng.choice([0.0, 0.0, 0.3]), "nfrac": 0.0, "p": p}
    if kind == "serve":
        return base | {"requests": rng.randint(4, 24), "nmin": 1_000, "nmax": _log(rng, 20_000, 400_000),
                       "motifs": _log(rng, 100, 2000)}
    if kind == "fastascan":
        return base | {"n": _log(rng, 50_000, 20_000_000), "seqs": _log(rng, 1, 300), "width": rng.randint(50, 120),
                       "nfrac": rng.choice([0.0, 0.01]), "motifs": _log(rng, 4, 64), "p": 1e-5}
    if kind == "fasta":
        return base | {"n": _log(rng, 100_000, 80_000_000), "seqs": _log(rng, 1, 1_000), "width": rng.randint(30, 200),
                       "nfrac": rng.choice([0.0, 0.01]), "lower": rng.choice([0.0, 0.3])}
    if kind == "thr":
        return base | {"motifs": _log(rng, 8, 2000), "bins": rng.choice([100, 250, 250, 500]),
                       "fp64": rng.choice([0, 0, 1])}
    return base | {"n": _log(rng, 20_000, 10_000_000), "runs": rng.randint(1, 40), "motifs": _log(rng, 4, 100),
                   "bins": rng.choice([100, 250, 250, 300]), "lower": rng.choice([0.0, 0.3])}


# ---------------------------------------------------------------- inputs
def _background(gc: float) -> np.ndarray:
    return np.array([(1 - gc) / 2, gc / 2, gc / 2, (1 - gc) / 2])


def _bank(case: dict, seed: int):
    """(P (columns x 4 lmax) float32, lengths): forward and reverse-complement columns, by length."""
    rng = np.random.default_rng([seed, 1])
    lens = np.sort(rng.integers(case["lmin"], case["lmax"] + 1, size=case["motifs"]))
    lmax = int(lens[-1])
    counts = rng.multinomial(100, rng.dirichlet([0.5] * 4, size=(len(lens), lmax)))
    pwm = np.log2((counts + 0.25) / (101.0 * _background(case["gc"]))).astype(np.float32)
    P = np.zeros((2 * len(lens), 4 * lmax), dtype=np.float32)
    for i, L in enumerate(lens):
        P[2 * i, :4 * L] = pwm[i, :L].ravel()
        P[2 * i + 1, :4 * L] = pwm[i, :L][::-1, ::-1].ravel()
    return P, np.repeat(lens, 2).astype(np.int32)


def _thresholds(P: np.ndarray, lens: np.ndarray, gc: float, pvalues) -> np.ndarray:
    """Per p-value and column the least score of a 2048-step grid whose tail has at most that probability."""
    steps, bg = 2048, _background(gc)
    pos = torch.arange(steps + 64, device="cuda")
    out = []
    for c0 in range(0, len(lens), 1000):
        L, rows = lens[c0:c0 + 1000], P[c0:c0 + 1000].reshape(len(lens[c0:c0 + 1000]), -1, 4).astype(np.float64)
        used = np.arange(rows.shape[1])[None, :] < L[:, None]
        lo, hi = np.where(used, rows.min(2), 0).sum(1), np.where(used, rows.max(2), 0).sum(1)
        width = (hi - lo) / steps
        q = np.where(used[:, :, None], np.rint((rows - rows.min(2, keepdims=True)) / width[:, None, None]), 0)
        q = torch.from_numpy(q).to("cuda", torch.int64)
        d = torch.zeros(len(L), len(pos), dtype=torch.float64, device="cuda")
        d[:, 0] = 1.0
        for j in range(rows.shape[1]):
            new = torch.zeros_like(d)
            for b in range(4):
                src = pos[None, :] - q[:, j, b:b + 1]
                new += bg[b] * torch.where(src >= 0, d.gather(1, src.clamp(min=0)), 0.0)
            keep = torch.from_numpy(used[:, j:j + 1]).cuda()
            d = torch.where(keep, new, d)
        tail = d.flip(1).cumsum(1).flip(1).cpu().numpy()
        for v, p in enumerate(pvalues):
            at = np.minimum((tail > p * (1 + 1e-9)).sum(1), steps)
            out.append((c0, v, lo + (at - 0.5) * width))  # a motif too short for p: its best score
    thr = np.zeros((len(pvalues), len(lens)), dtype=np.float32)
    for c0, v, t in out:
        thr[v, c0:c0 + len(t)] = t
    return thr


def _bases(n: int, gc: float, seed: int, lower: float = 0.0) -> torch.Tensor:
    """n iid bases on the GPU; about `lower` of them in lowercase stretches of 300."""
    g = torch.Generator("cuda").manual_seed(seed * 7919 + 17)
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    edges = torch.tensor(np.cumsum(_background(gc))[:3], dtype=torch.float32, device="cuda")
    acgt = torch.tensor(ACGT, dtype=torch.uint8, device="cuda")
    for a in range(0, n, 1 << 25):
        m = min(1 << 25, n - a)
        out[a:a + m] = acgt[torch.bucketize(torch.rand(m, device="cuda", generator=g), edges, right=True)]
    if lower > 0:
        soft = torch.rand((n + 299) // 300, device="cuda", generator=g) < lower
        out |= (soft.to(torch.uint8) * 0x20).repeat_interleave(300)[:n]
    return out


def _runs(n: int, k: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng([seed, 2])
    cuts = np.unique(rng.integers(1, max(2, n), size=max(0, k - 1)))
    return np.concatenate([[0], cuts[cuts < n]]).astype(np.int64)


def _fasta(case: dict, seed: int) -> torch.Tensor:
    """FASTA text on the GPU: `seqs` sequences of uneven length, N runs, lines of `width` characters."""
    rng = np.random.default_rng([seed, 3])
    body = _bases(case["n"], case["gc"], seed, case.get("lower", 0.0))
    left = int(case["nfrac"] * case["n"])
    while left > 0:
        k = min(left, int(np.exp(rng.uniform(np.log(100), np.log(10_000)))))
        a = int(rng.integers(0, case["n"]))
        body[a:a + k] = 78
        left -= k
    share = np.random.default_rng(case["seqs"]).uniform(0.1, 1.0, size=case["seqs"])  # lengths: the case's
    cuts = np.concatenate([[0], np.cumsum(np.floor(share / share.sum() * (case["n"] - 1)))]).astype(int).tolist()
    cuts[-1] = case["n"]
    w, parts = case["width"], []
    for i in range(case["seqs"]):
        head = np.frombuffer(b">seq%d synthetic sequence\n" % i, dtype=np.uint8).copy()
        s = body[cuts[i]:cuts[i + 1]]
        whole = len(s) // w * w
        lines = torch.full((whole // w, w + 1), 10, dtype=torch.uint8, device="cuda")
        lines[:, :w] = s[:whole].view(-1, w)
        parts += [torch.from_numpy(head).cuda(), lines.view(-1)]
        if whole < len(s):
            parts += [s[whole:], torch.full((1,), 10, dtype=torch.uint8, device="cuda")]
    return torch.cat(parts)


def _requests(case: dict, seed: int) -> list[dict]:
    shape, rng, out = np.random.default_rng(case["requests"]), np.random.default_rng([seed, 4]), []
    for r in range(case["requests"]):  # lengths, subset sizes and threshold sets are the case's
        n = int(round(math.exp(shape.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        m = int(shape.integers(1, case["motifs"] + 1))
        picked = np.sort(rng.choice(case["motifs"], size=m, replace=False))
        out.append({"bases": _bases(n, case["gc"], seed * 131 + r).cpu().numpy(), "runs": np.zeros(1, np.int64),
                    "cols": np.stack([2 * picked, 2 * picked + 1], 1).ravel().astype(np.int32),
                    "set": int(shape.integers(0, 2))})
    return out


def _room(case: dict, n: int, cols: int, p: float) -> int:
    """Hits to make room for: a motif too short for p has its best word's frequency instead."""
    rate = np.mean([max(p, 3.0 * 4.0 ** -L) for L in range(case["lmin"], case["lmax"] + 1)])
    return int(1.1 * n * cols * rate + min(n * cols * 8e-3, 1e6)) + 4096


def _out(cap: int) -> dict:
    return {"where": np.zeros(cap, np.int64), "score": np.zeros(cap, np.float32)}


def _most_runs(case: dict) -> int:
    return min(case["n"], int(case["nfrac"] * case["n"] / 500) + case["seqs"] + 100)


SERVE_P = (1e-4, 1e-5)


def prepare(case: dict, seed: int) -> dict:
    kind, st = case["kind"], {"case": case}
    if kind == "fasta":
        sc = GpuScanner(0)
        raw = _fasta(case, seed)
        st |= {"sc": sc, "raw": raw, "bases": torch.zeros_like(raw), "nucl": np.zeros(4, np.uint64),
               "tables": [torch.zeros(len(raw), dtype=torch.int64, device="cuda") for _ in range(4)]}
        return st
    P, lens = _bank(case, seed)
    if kind == "thr":
        return st | {"sc": GpuScanner(0), "P": P, "lens": lens, "bg": _background(case["gc"]).astype(np.float32),
                     "of": np.repeat(np.arange(0, len(lens), 2), 2).astype(np.int32)}
    if kind == "emphist":
        sc = GpuScanner(0)
        rows = P.reshape(len(lens), -1, 4)
        mn, mx = rows.min(2).sum(1), rows.max(2).sum(1)
        sc.set_motifs(P, lens, np.zeros(len(lens), np.float32))
        return st | {"sc": sc, "bases": _bases(case["n"], case["gc"], seed, case["lower"]).cpu().numpy(),
                     "runs": _runs(case["n"], case["runs"], seed), "min": mn, "width": (mx - mn) / case["bins"]}
    if kind == "serve":
        thr = _thresholds(P, lens, case["gc"], SERVE_P)
        requests = _requests(case, seed)
        return st | {"server": Server(P, lens, thr), "requests": requests,
                     "out": [_out(_room(case, len(r["bases"]), len(r["cols"]), SERVE_P[r["set"]])) for r in requests]}
    thr = _thresholds(P, lens, case["gc"], [case["p"]])[0]
    if kind == "fastascan":
        sc = GpuScanner(0)
        sc.set_motifs(P, lens, thr)
        return st | {"sc": sc, "raw": _fasta(case, seed).cpu().numpy().tobytes(),
                     "tables": [np.zeros(_most_runs(case), np.int64) for _ in range(3)],
                     "out": _out(_room(case, case["n"], len(lens), case["p"]))}
    sc = GpuScanner(0, case["mode"])
    sc.set_motifs(P, lens, thr)
    st |= {"sc": sc, "n": case["n"]}
    bases = _bases(case["n"], case["gc"], seed, case["lower"])
    runs = _runs(case["n"], case["runs"], seed)
    cap = _room(case, case["n"], len(lens), case["p"])
    if case["entry"] == "host":
        return st | {"bases": bases.cpu().numpy(), "runs": runs, "out": _out(cap)}
    st |= {"bases": bases, "runs": torch.from_numpy(runs).cuda(),
           "where_out": torch.zeros(cap, dtype=torch.int64, device="cuda"),
           "score_out": torch.zeros(cap, dtype=torch.float32, device="cuda"),
           "hits": torch.empty(cap * HIT_DTYPE.itemsize, dtype=torch.uint8, device="cuda"),
           "stream": torch.cuda.ExternalStream(sc.stream())}
    torch.cuda.synchronize()
    where = (bases.data_ptr(), case["n"], st["runs"].data_ptr(), len(runs), st["hits"].data_ptr(), cap)
    if case["tune"]:
        sc.autotune(*where[:4])
    if case["entry"] == "static":  # its plan is built by a first ordinary scan
        sc.scan_device(*where)
    if case["entry"] == "graph":
        st["counts"] = torch.zeros(4, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        sc.reserve(case["n"], 3 * cap)
        st["graph"] = sc.graph_create(*where, st["counts"].data_ptr())
    return st | {"where": where}


# ---------------------------------------------------------------- one pass
def _ordered(hits: np.ndarray, out: dict) -> dict:
    key = (hits["pos"] << COL_BITS) | hits["col"]
    order = np.argsort(key)
    np.take(key, order, out=out["where"][:len(key)])
    np.take(hits["score"], order, out=out["score"][:len(key)])
    return out | {"hits": len(key)}


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "scan":
        sc = st["sc"]
        if case["entry"] == "host":
            return _ordered(sc.scan(st["bases"], st["runs"]), st["out"])
        with torch.cuda.stream(st["stream"]):
            if case["entry"] == "graph":
                sc.graph_launch(st["graph"])
                nh = int(st["counts"][1])
            else:
                nh = (sc.scan_device_static if case["entry"] == "static" else sc.scan_device)(*st["where"])
            words = st["hits"].view(torch.int64).view(-1, 2)[:nh]
            key, order = torch.sort(torch.add(words[:, 1] & 0xFFFFFFFF, words[:, 0], alpha=1 << COL_BITS))
            st["where_out"][:nh] = key
            st["score_out"][:nh] = st["hits"].view(torch.float32).view(-1, 4)[:nh, 3][order]
        return {"where": st["where_out"], "score": st["score_out"], "hits": nh}
    if kind == "serve":
        sv = st["server"]
        ids = [sv.submit(r["bases"], r["runs"], r["cols"], r["set"]) for r in st["requests"]]
        return [_ordered(sv.take(i), o) for i, o in zip(ids, st["out"])]
    if kind == "fastascan":
        sc = st["sc"]
        nb, _, _, nucl = sc.stream_load_fasta(st["raw"])
        starts, seq, seqpos, heads = sc.stream_tables()
        for t, v in zip(st["tables"], (starts, seq, seqpos)):
            t[:len(v)] = v
        return {"tables": st["tables"], "headers": heads, "nucl": nucl.astype(np.int64),
                **_ordered(sc.scan_stream(0, nb, starts), st["out"])}
    if kind == "fasta":
        raw, t = st["raw"], st["tables"]
        nb, nr, ns = st["sc"].fasta_parse_device(raw.data_ptr(), len(raw), st["bases"].data_ptr(), t[0].data_ptr(),
                                                 t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), st["nucl"])
        return {"bases": st["bases"], "runs": [x[:_most_runs(case)] for x in t[:3]], "headers": t[3][:case["seqs"]],
                "counts": [nb, nr, ns], "nucl": st["nucl"].astype(np.int64)}
    if kind == "thr":
        thr, counts = st["sc"].theoretical_hist(st["P"], st["lens"], st["bg"], (1e-3, 1e-4, 1e-5), st["of"],
                                                case["bins"], fp64_dp=bool(case["fp64"]), counts=True)
        return {"thr": thr, "counts": counts.astype(np.int64)}
    return st["sc"].score_histograms(st["bases"], st["runs"], st["min"], st["width"], case["bins"]).astype(np.int64)


# ---------------------------------------------------------------- what a pass cannot do without
def work(case: dict) -> dict:
    """Inputs read once and outputs written once; the scans' flops are the one-hot contraction's,
    8 per motif position, column and window start (the plain and histogram forms: one addition)."""
    kind = case["kind"]
    if kind == "fasta":
        text = case["n"] * (1 + 1 / case["width"])
        return {"bytes": text + case["n"] * (1 - case["nfrac"]), "flops": 0}
    cols, mean = 2 * case["motifs"], (case["lmin"] + case["lmax"]) / 2
    bank = 16 * mean * cols
    if kind == "thr":  # the distribution over `bins` keys, advanced by every position and base
        return {"bytes": bank / 2 + cols * (8 * case["bins"] + 12), "flops": case["motifs"] * mean * 8 * case["bins"]}
    if kind == "emphist":
        return {"bytes": case["n"] + bank + 8 * cols * case["bins"], "flops": case["n"] * cols * mean}
    if kind == "serve":
        n = case["requests"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        return {"bytes": n + 16 * n * cols / 2 * sum(SERVE_P) / 2, "flops": 8 * n * cols / 2 * mean}
    text = case["n"] * (1 + 1 / case["width"]) if kind == "fastascan" else case["n"]
    per = 1 if case.get("mode") == "fp32" else 8
    return {"bytes": text + bank + 16 * case["n"] * cols * case["p"], "flops": per * case["n"] * cols * mean}


# ---------------------------------------------------------------- the same in 64 bits
def _exact_hits(bases: torch.Tensor, runs: np.ndarray, P, lens, thr, room: int, cols=None) -> np.ndarray:
    """FP64 scores of the windows whose FP32 score (summed in motif order) reaches the threshold."""
    n = len(bases)
    code = torch.full((n + 64,), 4, dtype=torch.int64, device="cuda")
    for b, ch in enumerate(ACGT):
        code[:n][bases == ch] = b
    ends = torch.from_numpy(np.append(runs[1:], n)).cuda()
    left = ends[torch.searchsorted(torch.from_numpy(runs).cuda(), torch.arange(n, device="cuda"), right=True) - 1]
    left -= torch.arange(n, device="cuda")
    cols = np.arange(len(lens)) if cols is None else cols
    keys, scores = [], []
    for L in np.unique(lens[cols]):
        same = cols[lens[cols] == L]
        for c0 in range(0, len(same), 16):
            cc = same[c0:c0 + 16]
            rows = np.zeros((int(L), 5, len(cc)), np.float32)
            rows[:, :4] = P[cc, :4 * L].reshape(len(cc), int(L), 4).transpose(1, 2, 0)
            rows = torch.from_numpy(rows).cuda()
            t, at = torch.from_numpy(thr[cc]).cuda(), torch.from_numpy(cc.astype(np.int64)).cuda()
            for a in range(0, n, 1 << 22):
                m = min(1 << 22, n - a)
                s = torch.zeros(m, len(cc), dtype=torch.float32, device="cuda")
                for j in range(int(L)):
                    s += rows[j][code[a + j:a + j + m]]
                i, k = torch.nonzero((s >= t) & (left[a:a + m, None] >= int(L)), as_tuple=True)
                e = torch.zeros(len(i), dtype=torch.float64, device="cuda")
                for j in range(int(L)):
                    e += rows[j].double()[code[a + i + j], k]
                keys.append(((a + i) << COL_BITS) | at[k])
                scores.append(e)
    keys, scores = torch.cat(keys), torch.cat(scores)
    out = np.zeros(room)
    out[:len(keys)] = scores[torch.argsort(keys)].cpu().numpy()
    return out


def _exact_thr(case: dict, seed: int) -> np.ndarray:
    P, lens = _bank(case, seed)
    bg, bins, out = _background(case["gc"]).astype(np.float32).astype(np.float64), case["bins"], []
    for c in range(0, len(lens), 2):
        L = int(lens[c])
        pwm = P[c, :4 * L].reshape(L, 4).astype(np.float64)
        mn, mx = pwm.min(1).sum(), pwm.max(1).sum()
        a = bins / (mx - mn)
        b = -a * mn / L
        q = np.floor(np.abs(a * pwm + b) + 0.5) * np.sign(a * pwm + b)
        lo = np.minimum(0, np.minimum.accumulate(np.cumsum(q.min(1)))).min()
        size = int(np.maximum.accumulate(np.cumsum(q.max(1))).max() - lo + 1 + bins)
        d, off = np.zeros(size), int(-lo)
        d[off] = 1.0
        for j in range(L):
            new = np.zeros(size)
            for k in range(4):
                s = int(q[j, k])
                if s >= 0:
                    new[s:] += bg[k] * d[:size - s]
                else:
                    new[:s] += bg[k] * d[-s:]
            d = new
        score = (np.arange(size) - off - L * b) / a
        hist = np.zeros(bins)
        at = np.clip((score - mn) * bins / (mx - mn), 0, bins - 1).astype(np.int64)
        hist[at[d > 0]] = np.floor(1e7 * d[d > 0])
        row = []
        for p in (1e-3, 1e-4, 1e-5):
            left, cut = float(np.float32(p)) * hist.sum(), mx
            for i in range(bins - 1, -1, -1):
                if hist[i] >= left:
                    f = left / hist[i] if hist[i] else 0.0
                    cut = (f * i + (1 - f) * (i + 1)) * (mx - mn) / bins + mn
                    break
                left -= hist[i]
            row.append(cut)
        out += [row, row]
    return np.array(out).T.copy()


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "thr":
        return {"thr": _exact_thr(case, seed), "counts": None}
    if kind not in ("scan", "serve") or case.get("n", 0) * case["motifs"] > 3e9:
        return None
    P, lens = _bank(case, seed)
    if kind == "serve":
        thr = _thresholds(P, lens, case["gc"], SERVE_P)
        return [{"where": None, "hits": None, "score": _exact_hits(
            torch.from_numpy(r["bases"]).cuda(), r["runs"], P, lens, thr[r["set"]],
            _room(case, len(r["bases"]), len(r["cols"]), SERVE_P[r["set"]]), r["cols"])} for r in _requests(case, seed)]
    thr = _thresholds(P, lens, case["gc"], [case["p"]])[0]
    bases = _bases(case["n"], case["gc"], seed, case["lower"])
    room = _room(case, case["n"], len(lens), case["p"])
    return {"where": None, "hits": None,
            "score": _exact_hits(bases, _runs(case["n"], case["runs"], seed), P, lens, thr, room)}
