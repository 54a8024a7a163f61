"""What the framework is asked to do in use: the cases that its speed is measured on.

Each case is one call (or, for the selection, the two calls that always go together) of the public surface:

    decode    one step of a decode batch: the op, the older op that returns the output alone, or the FlashMLA-shaped
              call with its metadata object
    prefill   one chunk of query tokens of a prompt
    model1    the 584-byte cache layout, decode and prefill, with and without the second cache
    select    FP8 indexer logits and the top-k of every row (a prompt's chunk, or a few tokens of a decode step)
    step      indexer -> top-k -> attention of one decode step as the captured graph a serving loop replays
    pack      the cache writer

Shapes are those of this repository's benchmark configurations and tests (128 query heads on one GPU, 64 / 32 / 16 / 8
under tensor parallelism, top-k 2048 and below, pages of 64 rows) and sizes between them.
"""
import math

import torch

import sparse_mla_sm120_b200 as smla
from sparse_mla_sm120_b200 import flash_ops, indexer, interface, pipeline

DEVICE = "cuda"
PAGE = 64
ROW, ROW_M1 = 656, 584          # bytes of a cache row in the two layouts
D_QK, D_QK_M1, D_V = 576, 512, 512
POOL_ROWS = 1 << 20             # most rows of a pool that prepare() fills (0.69 GB)


def listed():
    return [
        # The smallest step of serving: one request, its whole latency is what counts.
        dict(name="decode_one_request", kind="decode", surface="op", requests=1, s_q=1, heads=128, topk=2048,
             context=32768, lengths=False, sink=False),
        # A small running batch whose requests have selected different numbers of rows, with attention sinks.
        dict(name="decode_lengths_sink", kind="decode", surface="op", requests=13, s_q=1, heads=128, topk=2048,
             context=8192, lengths=True, sink=True),
        # The benchmark's batch: 64 requests, KV length up to 32768.
        dict(name="decode_batch", kind="decode", surface="op", requests=64, s_q=1, heads=128, topk=2048,
             context=18432, lengths=False, sink=False),
        # One rank of an eight-way tensor-parallel server (16 of 128 heads), through the older op surface.
        dict(name="decode_tensor_parallel", kind="decode", surface="legacy", requests=48, s_q=1, heads=16, topk=2048,
             context=16384, lengths=False, sink=False),
        # Multi-token prediction: two query tokens per request, every layer of a step with one metadata object.
        dict(name="decode_two_tokens", kind="decode", surface="flashmla", requests=64, s_q=2, heads=128, topk=2048,
             context=16384, lengths=False, sink=False),
        # A full prompt chunk over a cache of 8192 rows, causal selection.
        dict(name="prefill_chunk", kind="prefill", tokens=4096, heads=128, topk=2048, context=8192, lengths=False),
        # The start of a prompt on a two-way tensor-parallel rank: token i sees i + 1 rows, the lists are ragged.
        dict(name="prefill_prompt_start", kind="prefill", tokens=1237, heads=64, topk=1024, context=1237, lengths=True),
        # The 584-byte layout with its window in a second cache: the default (exact) numerics.
        dict(name="model1_decode_extra", kind="model1", phase="decode", tokens=32, heads=128, topk=1024, extra=128,
             context=16384, lengths=True, fp8=False),
        # The same layout where FP8-class numerics are chosen: a prompt chunk.
        dict(name="model1_prefill_fp8", kind="model1", phase="prefill", tokens=1024, heads=128, topk=1024, extra=0,
             context=8192, lengths=False, fp8=True),
        # The benchmark's indexer: logits of a prompt chunk against 65536 keys and the best 2048 of every row.
        dict(name="select_prompt_chunk", kind="select", tokens=4096, heads=64, keys=65536, topk=2048),
        # One decode step of a long context, paged cache, as a serving loop replays it.
        dict(name="indexed_step", kind="step", tokens=16, heads=128, index_heads=64, context=131072, topk=2048, paged=True),
        # A chunk's rows on their way into the cache.
        dict(name="pack_chunk", kind="pack", rows=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode"] * 5 + ["prefill"] * 2 + ["model1"] * 2 + ["select", "step", "pack"])
    if kind == "decode":
        surface = rng.choice(["op", "op", "legacy", "flashmla"])
        topk = rng.choice([2048, 2048, _log_int(rng, 64, 2048)])
        s_q = rng.choice([1, 1, 2]) if surface == "flashmla" else 1
        lengths = surface == "op" and rng.random() < 0.5
        return dict(kind=kind, surface=surface, requests=_log_int(rng, 1, 128 // s_q), s_q=s_q,
                    heads=rng.choice([8, 16, 32, 64, 128, 128, 128]), topk=topk, context=_log_int(rng, max(topk, 2048), 32768),
                    lengths=lengths, sink=surface != "legacy" and rng.random() < 0.4)
    if kind == "prefill":
        tokens, topk = _log_int(rng, 65, 4096), rng.choice([2048, 2048, _log_int(rng, 256, 2048)])
        return dict(kind=kind, tokens=tokens, heads=rng.choice([16, 64, 128, 128]), topk=topk,
                    context=tokens + rng.choice([0, _log_int(rng, 1024, 8192)]), lengths=rng.random() < 0.5)
    if kind == "model1":
        phase = rng.choice(["decode", "decode", "prefill"])
        return dict(kind=kind, phase=phase, tokens=_log_int(rng, 1, 64) if phase == "decode" else _log_int(rng, 65, 1024),
                    heads=rng.choice([8, 64, 128, 128]), topk=rng.choice([512, 1024, _log_int(rng, 100, 1024)]),
                    extra=rng.choice([0, 64, 128, 512]), context=_log_int(rng, 2048, 32768),
                    lengths=phase == "decode" and rng.random() < 0.5, fp8=phase == "prefill" or rng.random() < 0.5)
    if kind == "select":
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), heads=rng.choice([32, 64, 64]), keys=_log_int(rng, 4096, 65536),
                    topk=rng.choice([2048, 2048, 512]))
    if kind == "step":
        return dict(kind=kind, tokens=_log_int(rng, 1, 32), heads=rng.choice([64, 128]), index_heads=64,
                    context=_log_int(rng, 4096, 131072), topk=rng.choice([2048, 2048, 1024]), paged=rng.random() < 0.7)
    return dict(kind=kind, rows=_log_int(rng, 1, 65536))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(shape, device=DEVICE, generator=g)


def _latents(g, rows, offset):
    """Latent rows: unit noise around a mean per channel (the channels of a trained projection are not centred)."""
    return (_randn(g, rows, D_QK) + offset).to(torch.bfloat16)


def _pool_v32(g, rows):
    rows = -(-rows // PAGE) * PAGE
    offset = 0.5 * _randn(g, D_QK)
    pool = torch.empty((rows // PAGE, PAGE, 1, ROW), dtype=torch.uint8, device=DEVICE)
    flat = pool.view(rows, ROW)
    for r0 in range(0, rows, 1 << 17):
        r1 = min(r0 + (1 << 17), rows)
        flat[r0:r1] = indexer.pack_kv_cache(_latents(g, r1 - r0, offset))
    return pool


def _pool_m1(g, rows):
    """Pages of 64 tokens: 64 x (448 e4m3 | 64 bf16), then 64 x (7 power-of-two exponents | pad)."""
    pages = -(-rows // PAGE)
    offset = 0.5 * _randn(g, 448)
    nope = ((_randn(g, pages * PAGE, 448) + offset) * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    rope = _randn(g, pages * PAGE, 64).to(torch.bfloat16)
    data = torch.cat([nope.view(torch.uint8), rope.view(torch.uint8)], dim=1).view(pages, PAGE * 576)
    footer = 120 + torch.randint(0, 3, (pages, PAGE, 8), device=DEVICE, generator=g, dtype=torch.uint8)
    footer[..., 7] = 0
    return torch.cat([data, footer.view(pages, PAGE * 8)], dim=1).view(pages, PAGE, 1, ROW_M1)


def _pick(g, visible, topk, chunk=512):
    """Per row t, topk different positions out of [0, visible[t]) in no particular order, -1 where there are fewer."""
    out = torch.empty((visible.numel(), topk), dtype=torch.int32, device=DEVICE)
    for t0 in range(0, visible.numel(), chunk):
        v = visible[t0:t0 + chunk]
        n = max(int(v.max()), topk)
        keys = torch.rand((v.numel(), n), device=DEVICE, generator=g)
        keys.masked_fill_(torch.arange(n, device=DEVICE) >= v.unsqueeze(1), -1.0)
        best, pos = torch.topk(keys, topk, dim=1)
        out[t0:t0 + chunk] = torch.where(best >= 0, pos, -1)
    return out


def _own_rows(g, pos, pool_rows, requests, context):
    """Positions of request r's context -> physical rows: every request owns a run of shuffled pages of the pool."""
    pages_per = -(-context // PAGE)
    pages = torch.randperm(pool_rows // PAGE, device=DEVICE, generator=g)
    per = pos.shape[0] // requests
    first = (torch.arange(pos.shape[0], device=DEVICE) // per) * pages_per
    page = pages[(first.unsqueeze(1) + pos.clamp(min=0) // PAGE) % pages.numel()]
    return torch.where(pos >= 0, page * PAGE + pos.clamp(min=0) % PAGE, -1).to(torch.int32)


def _lengths(g, n, topk):
    """Numbers of selected rows between an eighth of the list and all of it."""
    return torch.randint(max(topk // 8, 1), topk + 1, (n,), device=DEVICE, generator=g, dtype=torch.int32)


def _index_inputs(g, tokens, heads, keys):
    q = _randn(g, tokens, heads, 128).to(torch.float8_e4m3fn)
    kf = _randn(g, keys, 128)
    scale = kf.abs().amax(dim=1) / 448.0
    k = (kf / scale.unsqueeze(1)).to(torch.float8_e4m3fn)
    w = 0.1 * _randn(g, tokens, heads)
    ks = torch.zeros(tokens, dtype=torch.int32, device=DEVICE)
    # the last token sees every key, the ones before it one key less each
    ke = (keys - tokens + 1 + torch.arange(tokens, device=DEVICE)).clamp(min=1).to(torch.int32)
    return q, k, scale, w, ks, ke


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    s = {"case": case}
    if kind == "decode":
        n, tokens, context, topk = case["requests"], case["requests"] * case["s_q"], case["context"], case["topk"]
        s["q"] = (0.5 * _randn(g, tokens, case["heads"], D_QK)).to(torch.bfloat16)
        s["kv"] = _pool_v32(g, min(n * (-(-context // PAGE) * PAGE), POOL_ROWS))
        pos = _pick(g, torch.full((tokens,), context, device=DEVICE), topk)
        s["indices"] = _own_rows(g, pos, s["kv"].shape[0] * PAGE, n, context)
        s["lengths"] = _lengths(g, tokens, topk) if case["lengths"] else None
        s["sink"] = _randn(g, case["heads"]) if case["sink"] else None
        if case["surface"] == "flashmla":
            s["q"] = s["q"].view(n, case["s_q"], case["heads"], D_QK)
            s["indices"] = s["indices"].view(n, case["s_q"], topk)
            s["meta"] = interface.get_mla_metadata()[0]
    elif kind == "prefill":
        tokens, context = case["tokens"], case["context"]
        s["q"] = (0.5 * _randn(g, tokens, case["heads"], D_QK)).to(torch.bfloat16)
        s["kv"] = _pool_v32(g, context)
        visible = context - tokens + 1 + torch.arange(tokens, device=DEVICE)
        s["indices"] = _own_rows(g, _pick(g, visible, case["topk"]), s["kv"].shape[0] * PAGE, 1, context)
        s["lengths"] = visible.clamp(max=case["topk"]).to(torch.int32) if case["lengths"] else None
    elif kind == "model1":
        tokens, context, topk, extra = case["tokens"], case["context"], case["topk"], case["extra"]
        s["q"] = (0.5 * _randn(g, tokens, case["heads"], D_QK_M1)).to(torch.bfloat16)
        owners = tokens if case["phase"] == "decode" else 1
        s["kv"] = _pool_m1(g, min(owners * (-(-context // PAGE) * PAGE), POOL_ROWS // 4))
        pos = _pick(g, torch.full((tokens,), context, device=DEVICE), topk)
        s["indices"] = _own_rows(g, pos, s["kv"].shape[0] * PAGE, owners, context)
        s["lengths"] = _lengths(g, tokens, topk) if case["lengths"] else None
        s["extra"] = {}
        if extra:
            window = owners * 2 * extra
            epos = _pick(g, torch.full((tokens,), 2 * extra, device=DEVICE), extra)
            ekv = _pool_m1(g, window)
            s["extra"] = dict(extra_k_cache=ekv, extra_topk=extra,
                              extra_indices=_own_rows(g, epos, ekv.shape[0] * PAGE, owners, 2 * extra))
    elif kind == "select":
        s["inputs"] = _index_inputs(g, case["tokens"], case["heads"], case["keys"])
    elif kind == "step":
        tokens, context = case["tokens"], case["context"]
        kv = _pool_v32(g, context)
        qi, ki, scale, w, ks, ke = _index_inputs(g, tokens, case["index_heads"], context)
        table = None
        if case["paged"]:
            pages = torch.randperm(kv.shape[0], device=DEVICE, generator=g).to(torch.int32)
            table = pages.unsqueeze(0).expand(tokens, -1).contiguous()
        s["graph"] = pipeline.GraphedIndexedDecode(kv, ki, scale, tokens, case["heads"], case["index_heads"], D_QK ** -0.5,
                                                   topk=case["topk"], block_table=table)
        s["inputs"] = ((0.5 * _randn(g, tokens, case["heads"], D_QK)).to(torch.bfloat16), qi, w, ks, ke)
    else:
        s["kv"] = _latents(g, case["rows"], 0.5 * _randn(g, D_QK))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "decode":
        if case["surface"] == "legacy":
            return smla.sparse_mla_decode_fwd(s["q"], s["kv"], s["indices"], D_QK ** -0.5)
        if case["surface"] == "flashmla":
            return interface.flash_mla_with_kvcache(s["q"], s["kv"], None, None, D_V, s["meta"], None, D_QK ** -0.5, False, True,
                                                    indices=s["indices"], attn_sink=s["sink"])
        return flash_ops.sparse_mla_decode_fwd(s["q"], s["kv"], s["indices"], D_QK ** -0.5, attn_sink=s["sink"],
                                               topk_length=s["lengths"])
    if kind == "prefill":
        return flash_ops.sparse_mla_prefill_fwd(s["q"], s["kv"], s["indices"], D_QK ** -0.5, topk_length=s["lengths"])
    if kind == "model1":
        fn = flash_ops.sparse_mla_decode_fwd if case["phase"] == "decode" else flash_ops.sparse_mla_prefill_fwd
        return fn(s["q"], s["kv"], s["indices"], D_QK_M1 ** -0.5, topk_length=s["lengths"], impl=2 if case["fp8"] else 0,
                  **s["extra"])
    if kind == "select":
        q, k, scale, w, ks, ke = s["inputs"]
        logits = indexer.fp8_mqa_logits(q, k, scale, w, ks, ke)
        return logits, indexer.topk_indices(logits, ks, ke, case["topk"])
    if kind == "step":
        return s["graph"](*s["inputs"])
    return indexer.pack_kv_cache(s["kv"])


def _attention_work(tokens, heads, listed_entries, entries, row, d_qk, distinct_rows, prefill=False):
    """`entries`: list entries that are attended over, all tokens; the rows themselves count once each."""
    io = tokens * heads * (2 * d_qk + 2 * D_V + (8 if prefill else 4)) + 4 * listed_entries
    return {"bytes": distinct_rows * row + io, "flops": 2 * heads * entries * (d_qk + D_V)}


def work(case):
    kind = case["kind"]
    if kind == "decode":
        tokens = case["requests"] * case["s_q"]
        entries = tokens * case["topk"] * (9 / 16 if case["lengths"] else 1)      # lengths are uniform in [1/8, 1]
        rows = min(entries, case["requests"] * case["context"], POOL_ROWS)
        return _attention_work(tokens, case["heads"], tokens * case["topk"], entries, ROW, D_QK, rows)
    if kind == "prefill":
        tokens, context, topk = case["tokens"], case["context"], case["topk"]
        entries = sum(min(context - tokens + 1 + i, topk) for i in range(tokens))
        return _attention_work(tokens, case["heads"], tokens * topk, entries, ROW, D_QK, min(entries, context), prefill=True)
    if kind == "model1":
        tokens, topk, extra = case["tokens"], case["topk"], case["extra"]
        entries = tokens * (topk * (9 / 16 if case["lengths"] else 1) + extra)
        rows = min(entries, POOL_ROWS // 4 + 2 * extra * tokens,
                   (tokens if case["phase"] == "decode" else 1) * (case["context"] + 2 * extra))
        return _attention_work(tokens, case["heads"], tokens * (topk + extra), entries, ROW_M1, D_QK_M1, rows,
                               prefill=case["phase"] == "prefill")
    if kind in ("select", "step"):
        tokens, keys = case["tokens"], case["keys"] if kind == "select" else case["context"]
        heads = case["heads"] if kind == "select" else case["index_heads"]
        pairs = sum(max(keys - i, 1) for i in range(tokens))
        b = tokens * heads * (128 + 4) + keys * (128 + 4) + 8 * tokens
        flops = 2 * heads * 128 * pairs
        if kind == "select":       # the logits are an output and then the selection's input
            return {"bytes": b + 4 * tokens * (2 * keys + case["topk"]), "flops": flops}
        entries = tokens * case["topk"]
        a = _attention_work(tokens, case["heads"], entries, entries, ROW, D_QK, min(entries, keys))
        return {"bytes": a["bytes"] + b, "flops": a["flops"] + flops}
    return {"bytes": case["rows"] * (2 * D_QK + ROW), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "pack":
        return "exact"
    if kind == "select":            # fp32 sums; equal or nearly equal logits may change places at the end of a list
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.01}
    if kind == "step":
        return {"rel": 1e-2, "max": 0.2, "differ": 0.01}
    if kind == "model1" and not case["fp8"]:      # exact products and fp32 sums, results rounded to bf16
        return {"rel": 4e-3, "max": 0.05}
    return {"rel": 1e-2, "max": 0.2}              # queries and weights rounded to e4m3, results to bf16

