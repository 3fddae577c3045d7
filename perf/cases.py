"""Performance cases: the suffix-array work that programs hand to this
framework, called through its public Python entry points.

Texts are synthetic and seeded.  DNA-like texts carry planted repeats (copies
of earlier stretches with 1% substitutions), text bytes are words of a skewed
vocabulary, tokens are skewed word ids, and segmented genomes have lognormal
segments, separators and masked runs: the shapes of the repository's own
benchmark workloads.  Unless a case says `host`, texts, positions and outputs
are CUDA tensors, as in a program that keeps its data on the GPU.  One context
(workspace and stream) lives for the whole process, as programs keep it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "caps-sa_gb300"))

import capssa  # noqa: E402

IDX = {"u32": torch.int32, "u64": torch.int64}  # the index types as CUDA tensors
IDX_BYTES = {"u32": 4, "u64": 8}
SYM_BYTES = {"u8": 1, "u16": 2, "u32": 4}


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one read or contig: the smallest calls, where launches and
        # synchronisations are everything
        {"name": "contig_4k", "kind": "dna", "n": 4099, "coverage": 0.0, "index": "u32",
         "host": False},
        # a bacterial-genome-sized uniform text through plain numpy buffers,
        # the first call most users make
        {"name": "uniform_1m_host", "kind": "dna", "n": 1048576, "coverage": 0.0, "index": "u32",
         "host": True},
        # a small eukaryotic genome (odd length) with repeats
        {"name": "genome_16m", "kind": "dna", "n": 16777259, "coverage": 0.3, "index": "u32",
         "host": False},
        # the benchmark workload: a human-chromosome-sized text with repeats
        {"name": "genome_268m", "kind": "dna", "n": 268435456, "coverage": 0.3, "index": "u32",
         "host": False},
        # a text collection in bytes (words, capitals, digits), 64-bit index
        {"name": "bytes_50m", "kind": "bytes", "n": 50000017, "index": "u64"},
        # a tokenised corpus: 32-bit symbols over a vocabulary of 32,000
        {"name": "tokens_8m", "kind": "tokens", "n": 8000009, "symbol": "u32", "vocab": 32000,
         "index": "u32"},
        # a masked genome in segments, only its ACGT positions wanted, 64-bit
        # index, the default boundary order
        {"name": "masked_128m", "kind": "segmented", "n": 134217749, "order": "shorter",
         "want": "positions", "ties": "position", "index": "u64"},
        # the same shape as an aligner builds its index: ACGT selected by the
        # library, segments ordered longer first
        {"name": "aligner_40m", "kind": "segmented", "n": 40000003, "order": "longer",
         "want": "filter", "ties": "position", "index": "u64"},
        # many independent texts in one call
        {"name": "batch_2048", "kind": "batched", "texts": 2048, "min_len": 1024,
         "max_len": 262144, "index": "u32"},
        # the sample-sort builder, streaming the order to a host callback
        {"name": "stream_16m", "kind": "stream", "n": 16000057, "parts": 4096,
         "partition": "splitters"},
        # suffix array plus LCP array into numpy buffers
        {"name": "lcp_4m", "kind": "lcp", "n": 4000037, "index": "u32"},
        # a sparse index: one position in about sixty of a large text
        {"name": "sparse_100m", "kind": "sparse", "n": 100000007, "every": 61, "index": "u32"},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dna", "dna", "dna", "bytes", "tokens", "segmented", "segmented",
                       "batched", "stream", "lcp", "sparse"])
    index = rng.choice(["u32", "u64"])
    if kind == "dna":
        n = _size(rng, 500, 2.4e8)
        return {"kind": kind, "n": n, "coverage": rng.choice([0.0, 0.1, 0.3, 0.5]),
                "index": index, "host": n <= 2000000 and rng.random() < 0.3}
    if kind == "bytes":
        return {"kind": kind, "n": _size(rng, 2000, 5e7), "index": index}
    if kind == "tokens":
        return {"kind": kind, "n": _size(rng, 2000, 1.6e7), "symbol": rng.choice(["u16", "u32"]),
                "vocab": _size(rng, 300, 60000), "index": index}
    if kind == "segmented":
        want = rng.choice(["whole", "positions", "filter"])
        order = rng.choice(["shorter", "longer"])
        # the reference's tie order: an option of the in-memory builders, with
        # an effect under the default boundary order
        ref = want != "filter" and order == "shorter" and rng.random() < 0.4
        return {"kind": kind, "n": _size(rng, 20000, 1.3e8), "order": order, "want": want,
                "ties": "reference" if ref else "position", "index": index}
    if kind == "batched":
        lo = _size(rng, 64, 4096)
        return {"kind": kind, "texts": _size(rng, 8, 2048), "min_len": lo,
                "max_len": lo * _size(rng, 2, 100), "index": index}
    if kind == "stream":
        return {"kind": kind, "n": _size(rng, 100000, 2e7), "parts": _size(rng, 16, 4096),
                "partition": rng.choice(["splitters", "learned"])}
    if kind == "lcp":
        return {"kind": kind, "n": _size(rng, 20000, 6e6), "index": index}
    return {"kind": kind, "n": _size(rng, 1e6, 1.2e8), "every": _size(rng, 9, 1000),
            "index": index}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(g, lo, hi, n, dtype=torch.int64):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=dtype)


def _loguniform(g, lo, hi, n):
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    return torch.exp(math.log(lo) + u * (math.log(hi) - math.log(lo))).to(torch.int64)


def _ranges(start, length):
    """The concatenated ranges start[i] .. start[i] + length[i] - 1."""
    first = torch.cumsum(length, 0) - length
    total = int(length.sum())
    i = torch.repeat_interleave(torch.arange(len(length), device="cuda"), length,
                                output_size=total)
    return torch.arange(total, device="cuda") - first[i] + start[i]


def _plant(text, g, coverage, lmin, lmax, sub, sigma, bounds=None):
    """Copies of earlier stretches over about `coverage` of the text, in two
    waves (the second copies some copies); destinations of a wave do not
    overlap.  `bounds`: (start, end) of the text that holds each position."""
    n = text.numel()
    if coverage <= 0 or n < 4 * lmin:
        return text
    lmax = max(lmin + 1, min(lmax, n // 4))
    mean = (lmax - lmin) / math.log(lmax / lmin)
    for _ in range(2):
        count = int(n / mean) + 16
        length = _loguniform(g, lmin, lmax, count)
        gap = (length.double().mean() * (2.0 / coverage - 1.0) * 2.0 *
               torch.rand(count, generator=g, device="cuda", dtype=torch.float64)).to(torch.int64)
        dst = torch.cumsum(length + gap + 1, 0) - length
        keep = dst + length <= n
        dst, length = dst[keep], length[keep]
        lo = torch.zeros_like(dst)
        if bounds is not None:
            t = torch.searchsorted(bounds, dst, right=True)
            lo = bounds[t - 1]
            length = torch.minimum(length, bounds[t] - dst)
        room = dst - lo - length
        keep = (room > 0) & (length > 0)
        dst, length, lo, room = dst[keep], length[keep], lo[keep], room[keep]
        if not len(dst):
            break
        u = torch.rand(len(dst), generator=g, device="cuda", dtype=torch.float64)
        src = lo + (u * room.double()).to(torch.int64)
        to = _ranges(dst, length)
        sym = text[_ranges(src, length)].to(torch.int32)
        if sub > 0:
            flip = torch.rand(len(to), generator=g, device="cuda") < sub
            step = _ints(g, 1, sigma, len(to), torch.int32)
            sym = torch.where(flip, (sym + step) % sigma, sym)
        text[to] = sym.to(text.dtype)
    return text


def _dna(n, seed, coverage, lmin=100, lmax=10000):
    g = _gen(seed)
    return _plant(_ints(g, 0, 4, n, torch.uint8), g, coverage, lmin, lmax, 0.01, 4)


def _zipf(g, vocab, n):
    """n ids below vocab, id i with a probability about 1 / (i + 2.7)."""
    # summed on the host, in a fixed order
    cdf = torch.from_numpy(np.cumsum(1.0 / (np.arange(vocab) + 2.7))).cuda()
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=vocab - 1)


def _bytes(n, seed):
    """Words of 2..13 characters over 66 byte values, separated by spaces;
    a tenth of the text in quoted passages of 40..4,000 characters."""
    g = _gen(seed)
    vocab = 20000
    chars = np.frombuffer(b"etaoinshrdlcumwfgypbvkjxqzETAOINSHRDLCUMWFGYPBVKJXQZ0123456789.,;-",
                          dtype=np.uint8)
    alphabet = torch.from_numpy(chars.copy()).cuda()
    wlen = _ints(g, 2, 14, vocab)
    woff = torch.cumsum(wlen, 0) - wlen
    letters = alphabet[_zipf(g, len(alphabet), int(wlen.sum()))]
    ids = _zipf(g, vocab, n // 4 + 16)
    span = wlen[ids] + 1
    stop = int(torch.searchsorted(torch.cumsum(span, 0), n, right=False)) + 1
    ids, span = ids[:stop], span[:stop]
    at = _ranges(torch.zeros_like(span), span)
    word = torch.repeat_interleave(ids, span, output_size=len(at))
    text = torch.where(at == wlen[word], 32, letters[(woff[word] + at).clamp_(max=len(letters) - 1)])
    return _plant(text[:n].to(torch.uint8).contiguous(), g, 0.1, 40, 4000, 0.0, 256)


def _tokens(n, seed, vocab, symbol):
    """Skewed ids below vocab; a fifth of the corpus in repeated passages of
    16..2,000 tokens."""
    g = _gen(seed)
    text = _plant(_zipf(g, vocab, n).to(torch.int32), g, 0.2, 16, 2000, 0.01, vocab)
    return text if symbol == "u32" else text.to(torch.uint16)


def _segmented(n, seed):
    """Segments of lognormal length (median 2,000, sigma 1.5), each ended by
    symbol 4; bodies over {0..3}, a tenth of them repeats; 2% of the positions
    in runs of symbol 5.  (text, ends)"""
    g = _gen(seed)
    text = _plant(_ints(g, 0, 4, n, torch.uint8), g, 0.1, 100, 10000, 0.01, 4)
    rmax = max(40, min(50000, n // 100))
    rmin = max(20, rmax // 50)
    runs = max(1, int(0.02 * n / ((rmin + rmax) / 2)))
    length = _ints(g, rmin, rmax + 1, runs)
    start = _ints(g, 0, max(1, n - rmax), runs)
    text[_ranges(start, length)] = 5
    z = torch.randn(int(n / 3000) + 64, generator=g, device="cuda", dtype=torch.float64)
    seg = torch.exp(math.log(2000.0) + 1.5 * z).to(torch.int64).clamp_(min=2)
    ends = torch.cumsum(seg, 0)
    ends = ends[ends < n - 1]
    ends = torch.cat([ends, torch.tensor([n], device="cuda")])
    text[ends - 1] = 4
    return text, ends.cpu().numpy().astype(np.uint64)


def _batched(case, seed):
    # log-uniform lengths, one from the middle of each of `texts` equal shares
    # of the distribution, in random order
    rng = np.random.default_rng(seed)
    share = (rng.permutation(case["texts"]) + 0.5) / case["texts"]
    lens = (case["min_len"] * (case["max_len"] / case["min_len"]) ** share).astype(np.int64)
    offs = np.zeros(case["texts"] + 1, dtype=np.uint64)
    offs[1:] = np.cumsum(lens)
    g = _gen(seed)
    n = int(offs[-1])
    bounds = torch.from_numpy(offs.astype(np.int64)).cuda()
    text = _plant(_ints(g, 0, 4, n, torch.uint8), g, 0.1, 50, 5000, 0.01, 4, bounds)
    return text, offs


def _batched_total(case):
    """The expected number of symbols of a batch (log-uniform lengths)."""
    lo, hi = case["min_len"], case["max_len"]
    return case["texts"] * (hi - lo) / math.log(hi / lo)


# ------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    s = {"case": case, "ctx": capssa.default_context()}
    if kind == "dna":
        text = _dna(n, seed, case["coverage"])
        if case["host"]:
            s["text"] = text.cpu().numpy()
            s["out"] = np.empty(n, dtype=np.uint32 if case["index"] == "u32" else np.uint64)
        else:
            s["text"] = text
    elif kind == "bytes":
        s["text"] = _bytes(n, seed)
    elif kind == "tokens":
        s["text"] = _tokens(n, seed, case["vocab"], case["symbol"])
    elif kind == "segmented":
        s["text"], ends = _segmented(n, seed)
        s["lp"] = capssa.SegmentedText(n, ends, capssa.BoundaryRank.LONGER_FIRST
                                       if case["order"] == "longer"
                                       else capssa.BoundaryRank.SHORTER_FIRST)
        s["opts"] = capssa.Opts(tie_order=capssa.TieOrder.REFERENCE
                                if case["ties"] == "reference" else capssa.TieOrder.POSITION)
        kept = torch.nonzero(s["text"] < 4).flatten()
        if case["want"] == "positions":
            s["positions"] = kept.to(IDX[case["index"]])
        if case["want"] != "whole":  # the count is the text's own: room for all
            s["out"] = torch.zeros(n, dtype=IDX[case["index"]], device="cuda")
    elif kind == "batched":
        s["text"], s["offsets"] = _batched(case, seed)
        n = s["text"].numel()
    elif kind == "stream":
        s["text"] = _dna(n, seed, 0.3).cpu().numpy()
        s["opts"] = capssa.ExtMemOpts(subproblem_count=case["parts"],
                                      partition=capssa.Partition.LEARNED
                                      if case["partition"] == "learned"
                                      else capssa.Partition.SPLITTERS)
        s["out"] = np.empty(n, dtype=np.uint64)
    elif kind == "lcp":
        s["text"] = _dna(n, seed, 0.3).cpu().numpy()
    elif kind == "sparse":
        s["text"] = _dna(n, seed, 0.3)
        step = case["every"]
        g = _gen(seed + 1)
        at = torch.arange(0, n - step, step, device="cuda")
        pos = at + _ints(g, 0, step, len(at))
        s["positions"] = pos[torch.randperm(len(pos), generator=g, device="cuda")].to(
            IDX[case["index"]])
        s["out"] = torch.empty(len(pos), dtype=IDX[case["index"]], device="cuda")
    if "out" not in s and kind != "lcp":
        s["out"] = torch.empty(n, dtype=IDX[case["index"]], device="cuda")
    # the context works on a stream of its own: the inputs have to be there
    torch.cuda.synchronize()
    return s


def _signed(a):
    """A numpy result as the signed type of its width, as the CUDA ones are."""
    return a.view("i%d" % a.itemsize) if isinstance(a, np.ndarray) else a


def run(state):
    case, ctx, text = state["case"], state["ctx"], state["text"]
    kind = case["kind"]
    if kind in ("dna", "bytes", "tokens"):
        return _signed(ctx.build_in_memory(text, out=state["out"]))
    if kind == "segmented":
        if case["want"] == "whole":
            return ctx.build_in_memory(text, state["lp"], state["opts"], out=state["out"])
        if case["want"] == "filter":
            kept = ctx.build_in_memory_for_filter(text, 0, 4, state["lp"], state["opts"],
                                                  out=state["out"])
            return {"count": len(kept), "sa": state["out"]}
        return ctx.build_in_memory_for_positions(text, state["positions"], state["lp"],
                                                 state["opts"], out=state["out"])
    if kind == "batched":
        return ctx.build_batched(text, state["offsets"], out=state["out"])
    if kind == "stream":
        out, at = state["out"], [0]

        def emit(batch):
            out[at[0]:at[0] + len(batch)] = batch
            at[0] += len(batch)

        ctx.build_in_memory_sample_sort(text, state["opts"], emit)
        return _signed(out)
    if kind == "lcp":
        sa, lcp = ctx.build_in_memory_lcp(
            text, index=np.uint32 if case["index"] == "u32" else np.uint64)
        return {"sa": _signed(sa), "lcp": _signed(lcp)}
    return ctx.build_in_memory_for_positions(text, state["positions"], out=state["out"])


def work(case):
    """Bytes that one pass has to read and write: the text, the positions it is
    given and its outputs.  Integer work only."""
    kind = case["kind"]
    ib = IDX_BYTES[case.get("index", "u64")]
    n = _batched_total(case) if kind == "batched" else case["n"]
    if kind == "tokens":
        return {"bytes": n * (SYM_BYTES[case["symbol"]] + ib), "flops": 0}
    if kind == "segmented":
        m = n if case["want"] == "whole" else 0.98 * n
        return {"bytes": n + m * ib * (2 if case["want"] == "positions" else 1), "flops": 0}
    if kind == "lcp":
        return {"bytes": n + 2 * n * ib, "flops": 0}
    if kind == "sparse":
        return {"bytes": n + 2 * (n / case["every"]) * ib, "flops": 0}
    return {"bytes": n + n * ib, "flops": 0}


def exact(case, seed):
    """Every output is a whole number; there is no computed value to compare."""
    return None
