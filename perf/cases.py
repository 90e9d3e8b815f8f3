"""The work a serving program has this library do, as cases whose time is measured.

Five entry points are covered, each over the range it is called with:

* ``topk``    ``fast_topk_v3``: select of a decode step (few rows, 2 Ki to 8 Mi columns), fp32 and
              16-bit scores, 32- and 64-bit indices, windows, full and ragged rows, with and without
              threshold guesses carried from step to step.
* ``pages``   ``fast_topk_transform_fused``: the same followed by the page-table gather; decode (one
              request per row) and prefill (many query tokens per request, a causal window each).
* ``offsets`` ``fast_topk_transform_ragged_fused``: prefill over a flattened K, an offset per row.
* ``logits``  ``indexer_logits_fp8``: the scores of every key from the fp8 K cache.
* ``step``    ``indexer_topk``: logits and select of a whole decode step, with the buffers, guesses and
              survivor lists that a decoding program keeps from step to step.

A case is a dict of plain values.  ``rows`` are queries, ``width`` the columns of the score matrix,
``shortest`` the smallest length (lengths are uniform between it and ``width``; equal: all full).
"""
import math

import torch

from flash_float_jit_kernels_b200 import (fast_topk_transform_fused, fast_topk_transform_ragged_fused, fast_topk_v3,
                                          new_threshold_hint, workloads)
from flash_float_jit_kernels_b200.indexer_logits import HEAD_DIM, HEADS, indexer_logits_fp8, indexer_topk, new_handover

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}
TOPKS = (512, 1024, 2048)           # what sparse-attention models select
MAX_DECODE_SCORES = 1 << 23         # rows * width of a decode select
MAX_KEYS = 4_000_000                # rows * width of drawn logits and decode steps (the listed batch reads about as many)
MAX_PREFILL_SCORES = 1 << 26        # rows * width of a prefill select
MAX_PREFILL_REQUESTS = 8


def _topk(name, rows, width, k, shortest=None, scores="normal", dtype="float32", int64=False, window=0, guess=False):
    return {"name": name, "op": "topk", "rows": rows, "width": width, "k": k, "shortest": width if shortest is None else shortest,
            "scores": scores, "dtype": dtype, "int64": int64, "window": window, "guess": guess}


def _prefill(name, op, rows, width, requests, k):
    return {"name": name, "op": op, "rows": rows, "width": width, "k": k, "requests": requests}


def listed():
    return [
        # one user, short context: the smallest call, nearly all of it launch and latency
        _topk("decode 1x16Ki", 1, 16384, 2048),
        # one user, a million tokens of context; scores rounded to bf16, many equal ones at the threshold
        _topk("decode 1x1Mi ties", 1, 1 << 20, 2048, scores="ties"),
        # one user, the longest context: a row that only bandwidth bounds
        _topk("decode 1x8Mi", 1, 1 << 23, 2048),
        # few users, smaller k, scores with a dominant tail
        _topk("decode 4x1Mi k512 tail", 4, 1 << 20, 512, scores="tail"),
        # few users, windows that start at odd columns of a wider buffer
        _topk("decode 8x120000 windows", 8, 131072, 2048, shortest=120000, scores="unit255", window=2048),
        # a full serving batch: 64 users with contexts of all lengths, lightning-indexer logits
        _topk("decode 64x128Ki ragged", 64, 131072, 2048, shortest=4096, scores="logits"),
        # bf16 scores in rows of odd width, the layout torch.topk returns, guesses kept between steps
        _topk("decode 16x100003 bf16", 16, 100003, 1024, shortest=20000, dtype="bfloat16", int64=True, guess=True),
        # decode of a paged K cache: top-k and the page-table gather in one call
        {"name": "pages decode 32x64Ki", "op": "pages", "rows": 32, "width": 65536, "k": 2048, "shortest": 2000, "requests": 0},
        # a prefill chunk: 1000 query tokens of two requests, each with its causal window
        _prefill("pages prefill 1000x32Ki", "pages", 1000, 32768, 2, 2048),
        # a large prefill chunk over one flattened K of several short requests
        _prefill("offsets prefill 4096x16Ki", "offsets", 4096, 16384, 3, 2048),
        # scores of a full batch from the fp8 K cache: half a gigabyte of keys
        {"name": "logits 64x128Ki", "op": "logits", "rows": 64, "width": 131072, "shortest": 4096},
        # a whole decode step of a middling batch: logits, survivor lists, select
        {"name": "step 16x40000", "op": "step", "rows": 16, "width": 40000, "k": 2048, "shortest": 8000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A size of [lo, hi], spread over its logarithm: a power of two or any number, odd ones among them."""
    n = _log_int(rng, lo, hi)
    return min(hi, max(lo, 1 << round(math.log2(n)))) if rng.random() < 0.25 else n


def draw(rng):
    kind = rng.choice(("topk", "topk", "topk", "pages", "pages prefill", "offsets", "logits", "step"))
    k = rng.choice(TOPKS)
    if kind in ("pages prefill", "offsets"):
        width = _size(rng, 4096, 65536)
        rows = _size(rng, 128, min(4096, MAX_PREFILL_SCORES // width))
        c = _prefill(None, kind.split()[0], rows, width, rng.randint(1, min(MAX_PREFILL_REQUESTS, width // 2048)), k)
        del c["name"]
        return c
    if kind == "topk":
        rows = _size(rng, 1, 64)
        width = _size(rng, 2048, MAX_DECODE_SCORES // rows)
    else:
        rows = _size(rng, 1, 64)
        width = _size(rng, 2048, min(131072, MAX_KEYS // rows))
    shortest = width if rng.random() < 0.35 else max(1, int(width * rng.uniform(0.02, 0.95)))
    if kind == "topk":
        c = _topk(None, rows, width, k, shortest, rng.choice(("normal", "ties", "tail", "unit255", "logits")),
                  rng.choice(("float32", "float32", "float32", "bfloat16", "float16")), rng.random() < 0.25,
                  rng.choice((0, 0, 1024)), rng.random() < 0.3)
        c["window"] = min(c["window"], width - 1)
        del c["name"]
        return c
    c = {"op": kind, "rows": rows, "width": width, "shortest": shortest}
    if kind == "pages":
        c["requests"] = 0
    if kind != "logits":
        c["k"] = k
    return c


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _scores(kind, rows, width, seed):
    g = _generator(seed)
    if kind == "normal":
        return torch.randn((rows, width), generator=g, device="cuda")
    if kind == "ties":
        return workloads.gaussian_bf16_ties(rows, width, seed, "cuda")[0]
    if kind == "tail":
        return workloads.gaussian_outliers(rows, width, seed, "cuda")[0]
    if kind == "unit255":
        return workloads.reference_style(rows, width, False, "gaussian", seed, "cuda")[0]
    if kind == "logits":
        return workloads.lightning_indexer_logits(rows, width, width, seed, "cuda")[0]
    # "prefill": mean and deviation of lightning-indexer logits without the K cache behind them
    return torch.randn((rows, width), generator=g, device="cuda").mul_(1.8).add_(9.0).clamp_(min=0.0)


def _lengths(case, seed):
    return torch.randint(case["shortest"], case["width"] + 1, (case["rows"],), generator=_generator(seed + 7777), device="cuda",
                         dtype=torch.int32)


def _prefill_plan(case):
    """(request, window start, window length) of every query token: `requests` contexts side by side fill
    the width, and the query tokens are the last ones of their request."""
    n, width, rows = case["requests"], case["width"], case["rows"]
    edges = [width * i // n for i in range(n + 1)]
    tokens = [rows * i // n for i in range(n + 1)]
    plan = []
    for r in range(n):
        context, mine = edges[r + 1] - edges[r], tokens[r + 1] - tokens[r]
        plan += [(r, edges[r], max(1, context - mine + 1 + i)) for i in range(mine)]
    return plan, tokens


def _keys(case, seed):
    g = _generator(seed)
    rows, width = case["rows"], case["width"]
    q = torch.randn((rows, HEADS, HEAD_DIM), generator=g, device="cuda").div_(4)
    w = torch.rand((rows, HEADS), generator=g, device="cuda")
    keys = torch.empty((rows, width, HEAD_DIM), dtype=torch.float8_e4m3fn, device="cuda")
    for b in range(rows):
        keys[b] = torch.randn((width, HEAD_DIM), generator=g, device="cuda").div_(4).to(torch.float8_e4m3fn)
    return q, w, keys, g


def prepare(case, seed):
    op, rows, width = case["op"], case["rows"], case["width"]
    state = {"op": op}
    if op in ("logits", "step"):
        q, w, keys, g = _keys(case, seed)
        state.update(q=q.to(torch.float8_e4m3fn), w=w, keys=keys, lengths=_lengths(case, seed))
        if op == "step":
            # buffers of the decode loop, and the step before this one, which left guesses behind
            state.update(k=case["k"], scores=torch.full((rows, width), float("-inf"), device="cuda"),
                         out=torch.empty((rows, case["k"]), dtype=torch.int32, device="cuda"),
                         hint=new_threshold_hint(rows, "cuda"), handover=new_handover(rows, torch.device("cuda", torch.cuda.current_device())))
            before = (q + 0.02 * torch.randn(q.shape, generator=g, device="cuda")).to(torch.float8_e4m3fn)
            indexer_topk(before, keys, w, state["lengths"], case["k"], scores=state["scores"], out=state["out"],
                         threshold_hint=state["hint"], handover=state["handover"])
        return state
    if op == "topk":
        scores = _scores(case["scores"], rows, width, seed)
        lengths = _lengths(case, seed)
        if case["window"]:
            state["row_starts"] = torch.randint(0, case["window"], (rows,), generator=_generator(seed + 5), device="cuda", dtype=torch.int32)
            lengths = torch.minimum(lengths, width - state["row_starts"])
        state.update(score=scores.to(DTYPES[case["dtype"]]), lengths=lengths, k=case["k"],
                     index_dtype=torch.int64 if case["int64"] else torch.int32)
        if case["guess"]:
            # the step before this one: the same rows, slightly different scores
            noise = torch.randn(scores.shape, generator=_generator(seed + 9), device="cuda")
            before = scores.add(noise.mul_(0.02 * float(scores[0].std()))).to(DTYPES[case["dtype"]])
            state["hint"] = new_threshold_hint(rows, "cuda")
            fast_topk_v3(before, lengths, case["k"], state.get("row_starts"), threshold_hint=state["hint"])
        return state
    g = _generator(seed + 3)
    state["out"] = torch.empty((rows, case["k"]), dtype=torch.int32, device="cuda")
    if case["requests"] == 0:       # decode: a request per row
        state.update(score=_scores("logits", rows, width, seed), lengths=_lengths(case, seed))
        state["table"] = torch.randint(0, 1 << 24, (rows, width), generator=g, device="cuda", dtype=torch.int32)
        state["cu_seqlens"] = torch.arange(rows + 1, device="cuda", dtype=torch.int32)
        return state
    plan, tokens = _prefill_plan(case)
    state.update(score=_scores("prefill", rows, width, seed))
    state["row_starts"] = torch.tensor([s for _, s, _ in plan], device="cuda", dtype=torch.int32)
    state["lengths"] = torch.tensor([n for _, _, n in plan], device="cuda", dtype=torch.int32)
    if op == "pages":
        state["table"] = torch.randint(0, 1 << 24, (case["requests"], width), generator=g, device="cuda", dtype=torch.int32)
        state["cu_seqlens"] = torch.tensor(tokens, device="cuda", dtype=torch.int32)
    else:
        state["offset"] = state["row_starts"].clone()
    return state


def run(state):
    op = state["op"]
    if op == "topk":
        indices = fast_topk_v3(state["score"], state["lengths"], state["k"], state.get("row_starts"),
                               threshold_hint=state.get("hint"), index_dtype=state["index_dtype"])
        return (indices, state["hint"]) if "hint" in state else indices
    if op == "pages":
        fast_topk_transform_fused(state["score"], state["lengths"], state["out"], state["table"], state["cu_seqlens"],
                                  state.get("row_starts"))
        return state["out"]
    if op == "offsets":
        fast_topk_transform_ragged_fused(state["score"], state["lengths"], state["out"], state["offset"], state["row_starts"])
        return state["out"]
    if op == "logits":
        return indexer_logits_fp8(state["q"], state["keys"], state["w"], state["lengths"])
    indices = indexer_topk(state["q"], state["keys"], state["w"], state["lengths"], state["k"], scores=state["scores"],
                           out=state["out"], threshold_hint=state["hint"], handover=state["handover"])
    return {"scores": state["scores"], "indices": indices}


def work(case):
    """Scores (or keys) of the windows read once, results written once."""
    op, rows, width = case["op"], case["rows"], case["width"]
    if op in ("logits", "step"):
        keys = rows * (case["shortest"] + width) / 2
        w = {"bytes": keys * (HEAD_DIM + 4) + rows * (HEADS * HEAD_DIM + 4 * HEADS + 4), "flops": 2 * keys * HEADS * HEAD_DIM}
        if op == "logits":
            w["bytes"] += 4 * (rows * width - keys)     # a fresh result holds -inf behind every row's end
        else:
            w["bytes"] += 4 * rows * case["k"]
        return w
    if op == "topk":
        read = rows * (case["shortest"] + width) / 2 * (4 if case["dtype"] == "float32" else 2)
        return {"bytes": read + rows * (case["k"] * (8 if case["int64"] else 4) + 4), "flops": 0}
    out = 4 * rows * case["k"]
    if case["requests"] == 0:
        return {"bytes": 4 * rows * (case["shortest"] + width) / 2 + 2 * out, "flops": 0}
    read = 4 * sum(n for _, _, n in _prefill_plan(case)[0])
    table = min(out, 4 * case["requests"] * width) if op == "pages" else 4 * rows
    return {"bytes": read + out + table + 8 * rows, "flops": 0}


def tolerance(case):
    """Selects are exact; the guess left for the next step is a score of rank about 1.25 k, any such
    score.  Logits are 32-bit sums of 64 terms, and another order of summation may swap two nearly
    equal scores and so two indices of a step."""
    if case["op"] == "logits":
        return {"rel": 1e-5}
    if case["op"] == "topk" and case["guess"]:
        return {"rel": 0.03, "differ": 0.0}
    if case["op"] == "step":
        return {"rel": 1e-5, "differ": 2e-3}
    return "exact"
