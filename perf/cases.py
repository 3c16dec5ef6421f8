"""The work that a user of this library has it do, as cases to be timed: suffix-array builds from the smallest text to the
benchmark's, of texts on the device and in host memory, resident and part by part; count and locate batches on an index; and
the radix sort. A case is a dict of plain values; `prepare` makes what a user's program holds before the call and `run` is
one pass through the public calls of cascade_b200.api."""
import math

import torch

from cascade_b200 import api

VOCAB = 50257
_ctx = None
_cdf = None


def listed():
    return [
        # One short document or a test text: the call's latency (launches, read-backs) is all there is.
        {"name": "build_3k", "kind": "build", "n": 3001, "p": 1, "text": "zipf", "mean_doc": 512},
        # A small corpus, as the smoke test builds it.
        {"name": "build_262k", "kind": "build", "n": 1 << 18, "p": 8, "text": "zipf", "mean_doc": 512},
        # The small benchmark corpus: 16M tokens in a single partition.
        {"name": "build_16m", "kind": "build", "n": 1 << 24, "p": 1, "text": "zipf", "mean_doc": 512},
        # The headline benchmark: 2e9 tokens, 64 partitions, everything in one GPU's memory.
        {"name": "build_2g", "kind": "build", "n": 2_000_000_000, "p": 64, "text": "zipf", "mean_doc": 1024},
        # Near-duplicate documents (crawls, templates, versions): long shared suffixes, many doubling generations.
        {"name": "build_copies_400m", "kind": "build", "n": 400_000_003, "p": 64, "text": "copies", "mean_doc": 2048},
        # What the `cascade` command does with a file that fits the device: pinned text in, pinned 5-byte array out.
        {"name": "host_100m", "kind": "build_host", "n": 99_999_989, "p": 64, "text": "zipf", "mean_doc": 1024},
        # What it does with a text whose suffix lists do not fit: parts streamed through the device from host memory.
        {"name": "streamed_200m", "kind": "build_streamed", "n": 200_000_000, "p": 1024, "part_suffixes": 1 << 25, "text": "zipf", "mean_doc": 1024},
        # The benchmark's query batch, counts only, everything on the device.
        {"name": "count_4m_of_2g", "kind": "count", "n": 2_000_000_000, "q": 4_000_000, "stride": 32, "mean_doc": 1024},
        # Counts and the first positions of each match, on the device, as a retrieval step of a larger program.
        {"name": "locate_1m_of_200m", "kind": "locate", "n": 200_000_000, "q": 1_000_000, "max_pos": 20, "stride": 32, "mean_doc": 1024},
        # A host batch of counts and up to 100 positions a query, as the `query find` command runs it.
        {"name": "host_queries_1m", "kind": "query_host", "n": 500_000_000, "q": 1_000_000, "max_pos": 100, "stride": 32, "mean_doc": 1024},
        # An interactive request: a handful of patterns, where latency is what counts.
        {"name": "host_queries_50", "kind": "query_host", "n": 1 << 24, "q": 50, "max_pos": 100, "stride": 16, "mean_doc": 512},
        # The radix sort alone, at the size of one partition of the benchmark.
        {"name": "sort_31m", "kind": "sort", "n": 31_250_000, "bits": 64, "val_bytes": 4},
    ]


def _log_size(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "build_copies", "build_host", "build_streamed", "count", "locate", "query_host", "query_host", "sort"])
    if kind == "build":
        return {"kind": "build", "n": _log_size(rng, 1000, 1_000_000_000), "p": _log_size(rng, 1, 256), "text": "zipf", "mean_doc": rng.choice([512, 1024])}
    if kind == "build_copies":
        return {"kind": "build", "n": _log_size(rng, 1_000_000, 200_000_000), "p": _log_size(rng, 1, 256), "text": "copies", "mean_doc": 2048}
    if kind == "build_host":
        return {"kind": "build_host", "n": _log_size(rng, 10_000, 150_000_000), "p": _log_size(rng, 1, 256), "text": "zipf", "mean_doc": rng.choice([512, 1024])}
    if kind == "build_streamed":
        return {"kind": "build_streamed", "n": _log_size(rng, 1_000_000, 100_000_000), "p": _log_size(rng, 64, 4096), "part_suffixes": 1 << rng.randint(22, 26),
                "text": "zipf", "mean_doc": 1024}
    if kind == "sort":
        return {"kind": "sort", "n": _log_size(rng, 1000, 31_250_000), "bits": rng.choice([32, 40, 48, 64]), "val_bytes": rng.choice([4, 4, 8])}
    case = {"kind": kind, "n": _log_size(rng, 100_000, 500_000_000), "q": _log_size(rng, 1, 2_000_000), "stride": rng.choice([16, 32, 64]), "mean_doc": rng.choice([512, 1024])}
    if kind == "locate":
        case["max_pos"] = rng.randint(1, 50)
    if kind == "query_host":
        case["q"] = min(case["q"], 1_000_000)
        case["max_pos"] = rng.randint(1, 100)
    return case


# ---- inputs ----------------------------------------------------------------------------------------------------------------


def _context():
    """The one context that a program keeps for all its calls."""
    global _ctx, _cdf
    if _ctx is None:
        _ctx, _cdf = api.Context(0), api.zipf_cdf(VOCAB)
    return _ctx


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _zipf_text(n, seed, mean_doc):
    return api.gen_corpus_device(_context(), n, seed, mean_doc, _cdf)


def _copies_text(n, seed, mean_doc, base_docs=4096, mutate=0.001):
    """Base documents of Zipf tokens, then copies of random base documents with a small share of their tokens replaced."""
    g = _generator(seed)
    base_docs = max(16, min(base_docs, n // (16 * mean_doc)))
    base = _zipf_text(base_docs * (mean_doc + 1), seed, mean_doc).view(torch.int16)[:-api.TEXT_PAD]
    base[0] = -1
    starts = torch.nonzero(base == -1).flatten()
    lens = torch.diff(starts, append=torch.tensor([base.numel()], device="cuda"))
    text = torch.zeros(n + api.TEXT_PAD, dtype=torch.int16, device="cuda")
    at = min(n, base.numel())
    text[:at] = base[:at]
    while at < n:
        docs = torch.randint(0, starts.numel(), (1 + min(n - at, 1 << 27) // mean_doc,), device="cuda", generator=g)
        counts = lens[docs]
        first = torch.cumsum(counts, 0) - counts
        source = torch.repeat_interleave((starts[docs] - first).to(torch.int32), counts)
        source += torch.arange(source.numel(), device="cuda", dtype=torch.int32)
        piece = base[source]
        hit = torch.rand(piece.numel(), device="cuda", generator=g) < mutate
        fresh = torch.randint(0, VOCAB, (piece.numel(),), device="cuda", generator=g, dtype=torch.int32).to(torch.int16)
        piece = torch.where(hit & (piece != -1), fresh, piece)
        take = min(n - at, piece.numel())
        text[at:at + take] = piece[:take]
        at += take
    return text.view(torch.uint16)


def _text(case, seed):
    return (_copies_text if case["text"] == "copies" else _zipf_text)(case["n"], seed, case["mean_doc"])


def _pinned(count, dtype):
    return torch.zeros(count, dtype=dtype, pin_memory=True)


def _queries(text, n, q, seed):
    """Half pieces of the text, half random tokens, 1 to 16 symbols each; offsets and symbols on the device."""
    g = _generator(seed + 1)
    lens = torch.randint(1, 17, (q,), device="cuda", generator=g)
    pieces = q - q // 2
    at = torch.randint(0, n - 16, (pieces,), device="cuda", generator=g)
    off = torch.zeros(q + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=off[1:])
    sym = torch.randint(0, VOCAB, (int(off[-1]) + 8,), device="cuda", generator=g, dtype=torch.int32).to(torch.int16)
    copied = int(off[pieces])
    source = torch.repeat_interleave(at - off[:pieces], lens[:pieces]) + torch.arange(copied, device="cuda")
    sym[:copied] = text.view(torch.int16)[source]
    return off, sym.view(torch.uint16)


def prepare(case, seed):
    ctx, kind, n = _context(), case["kind"], case["n"]
    state = dict(case, ctx=ctx)
    if kind == "sort":
        g = _generator(seed)
        state["keys"] = torch.randint(-(1 << 62), 1 << 62, (n,), device="cuda", dtype=torch.int64, generator=g)
        state["vals"] = torch.arange(n, device="cuda", dtype=torch.int32 if case["val_bytes"] == 4 else torch.int64)
        return state
    if kind == "build":
        state["text"] = _text(case, seed)
        state["out"] = torch.zeros(5 * n + api.SA_PAD_BYTES, dtype=torch.uint8, device="cuda")
        return state
    if kind in ("build_host", "build_streamed"):
        state["text"] = _pinned(n + api.TEXT_PAD, torch.int16)
        state["text"].copy_(_text(case, seed).view(torch.int16))
        state["out"] = _pinned(5 * n + api.SA_PAD_BYTES, torch.uint8)
        return state
    text = _zipf_text(n, seed, case["mean_doc"])
    sa, _ = api.build_sa(ctx, text, n, 64)
    state["index"] = api.SuffixIndex(ctx, text, sa, n, case["stride"])
    off, sym = _queries(text, n, case["q"], seed)
    if kind == "query_host":
        state["off"], state["sym"] = _pinned(off.numel(), torch.int64), _pinned(sym.numel(), torch.int16)
        state["off"].copy_(off)
        state["sym"].copy_(sym.view(torch.int16))
        q = case["q"]
        state["bufs"] = {"itv": _pinned(2 * q, torch.int64), "cnt": _pinned(q, torch.int32), "pos_off": _pinned(q + 1, torch.int64),
                         "pos": _pinned(q * case["max_pos"], torch.int64)}
    else:
        state["off"], state["sym"] = off, sym
    return state


# ---- one pass --------------------------------------------------------------------------------------------------------------


def _array(out, n):
    """The 5 n bytes of a suffix array, as 8-byte words and the bytes that are left."""
    words = 5 * n // 8
    return [out[:8 * words].view(torch.int64), out[8 * words:5 * n]]


def run(state):
    ctx, kind, n = state["ctx"], state["kind"], state["n"]
    if kind == "build":
        return _array(api.build_sa(ctx, state["text"], n, state["p"], out=state["out"])[0], n)
    if kind == "build_host":
        return _array(api.build_sa_host(ctx, state["text"], n, state["p"], out=state["out"])[0], n)
    if kind == "build_streamed":
        return _array(api.build_sa_streamed(ctx, state["text"], n, state["p"], out=state["out"], part_suffixes=state["part_suffixes"])[0], n)
    if kind == "sort":
        return list(api.sort_pairs(ctx, state["keys"].clone(), state["vals"].clone(), 0, state["bits"]))
    index, q = state["index"], state["q"]
    if kind == "count":
        return index.find(state["off"], state["sym"], q)
    if kind == "locate":
        itv = index.find(state["off"], state["sym"], q)
        pos, cnt = index.locate(itv, q, state["max_pos"])
        # rows are used at their full width: what lies beyond a row's count is padding
        width = torch.arange(state["max_pos"], device=pos.device, dtype=torch.int32)
        return [itv, torch.where(width < cnt[:, None], pos, -1), cnt]
    itv, cnt, pos_off, pos, total = index.query_host(state["off"], state["sym"], state["max_pos"], state["bufs"])
    return [itv, cnt, pos_off, pos, total]      # the positions buffer is the program's own: zeros stand behind the last position


def work(case):
    n, kind = case["n"], case["kind"]
    if kind.startswith("build"):
        return {"bytes": 7 * n, "flops": 0}                 # the text in, 5 bytes a suffix out
    if kind == "sort":
        return {"bytes": 2 * n * (8 + case["val_bytes"]), "flops": 0}
    # offset and 8.5 symbols a query in, its interval out; with positions also its count, and about 11 positions of a
    # hundred asked for (half of the queries match once or never, short ones match as often as they may)
    rows = 0 if kind == "count" else 4 + 8 * min(case["max_pos"], 1 + 0.1 * case["max_pos"])
    return {"bytes": case["q"] * (8 + 17 + 16 + rows), "flops": 0}


def tolerance(case):
    return "exact"      # whole numbers: the suffix array, the intervals and a stable sort are unique
