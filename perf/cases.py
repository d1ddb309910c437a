"""Performance cases: the calls a serving engine makes of this package for one attention layer, over the range of sizes it
makes them at.

A case is a dict of plain values; `prepare` makes its tensors on the GPU from a seed, `run` is one pass through the
package's public operators, `work` the bytes a pass cannot do without and `tolerance` how far two correct implementations
at the same precision may be apart.

Kinds of case
  prologue      the fused q-norm / RoPE / FP8-insert operator by itself
  decode_step   every operator of one layer of a decode step, in the order a layer calls them
  prefill_step  every operator of one layer of a prefill step (chunk of several requests of different lengths)
  epilogue      inverse RoPE + FP8 quantisation of the attention output
  norm_quant    hidden-state quantiser, q/kv norms and the quantiser behind them: the way into the FP8 projections
  indexer       sparse-indexer q prologue and key insert
  readers       the two cache readers (latent KV de-quantised, indexer keys copied) over ragged sequences
  topk_decode   selection over the indexer logits of a decode batch
  topk_prefill  the same for a causal prefill chunk
"""
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("flaggems-vllm_b200"))
import flaggems_vllm as fg  # noqa: E402

DEV = "cuda"
BLOCK = 64  # tokens per cache block
EPS = 1e-6
HIDDEN, Q_LORA, HEAD = 7168, 1536, 512
INDEX_HEADS, INDEX_DIM = 64, 128
O_GROUPS = 8
WINDOW, RATIO = 128, 4  # sliding window, tokens per compressed key
SOFTMAX_SCALE, HEAD_SCALE = INDEX_DIM ** -0.5, INDEX_HEADS ** -0.5
CACHE_BLOCKS = 16384  # one million cached tokens


def listed():
    return [
        # one user generating: the shortest call there is
        {"name": "prologue, 1 token", "kind": "prologue", "tokens": 1, "heads": 64, "padding": 0.0, "max_pos": 65536, "slots": "random"},
        # decode batch of the benchmark's decode configuration
        {"name": "prologue, decode batch", "kind": "prologue", "tokens": 256, "heads": 128, "padding": 0.0, "max_pos": 65536, "slots": "random"},
        # the benchmark's default workload: long prefill, padded
        {"name": "prologue, long prefill", "kind": "prologue", "tokens": 32768, "heads": 128, "padding": 0.1, "max_pos": 131072, "slots": "random"},
        # a layer's calls for one user
        {"name": "decode step, 1 request", "kind": "decode_step", "requests": 1, "next_n": 1, "heads": 64, "context": 32768, "topk": 512, "fp4": False},
        # a layer's calls for a loaded server: ragged contexts, a batch size that is no multiple of anything
        {"name": "decode step, 61 requests", "kind": "decode_step", "requests": 61, "next_n": 1, "heads": 128, "context": 16384, "topk": 512, "fp4": True},
        # a prefill chunk shared by three requests, one of them with a long cached prefix
        {"name": "prefill step, 1531 tokens", "kind": "prefill_step", "tokens": 1531, "requests": 3, "prefix": 4096, "heads": 128, "topk": 512, "fp4": False},
        # attention output of a full prefill chunk, in the scale format the FP8 projection takes on this GPU
        {"name": "epilogue, 8192 tokens", "kind": "epilogue", "tokens": 8192, "heads": 128, "packed": True},
        # projections' inputs of an odd-sized chunk, float scales, column-major as the GEMM wants them
        {"name": "norm and quant, 4097 tokens", "kind": "norm_quant", "tokens": 4097, "ue8m0": False, "column_major": True},
        # sparse indexer of a long prefill, 4-bit queries
        {"name": "indexer, 16384 tokens", "kind": "indexer", "tokens": 16384, "fp4": True},
        # chunked-context readers: sixteen cached sequences of different lengths
        {"name": "readers, 16 sequences", "kind": "readers", "requests": 16, "longest": 16384},
        # long-context decode batch
        {"name": "top-k, decode 496 x 262144", "kind": "topk_decode", "rows": 496, "width": 262144, "topk": 512, "persistent": False},
        # causal prefill chunk over a long context
        {"name": "top-k, prefill 4096 x 32768", "kind": "topk_prefill", "rows": 4096, "width": 32768, "topk": 2048},
    ]


def _log(rng, low, high):
    """An integer in [low, high], uniform in its logarithm."""
    return max(low, min(high, int(round(low * (high / low) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["prologue", "prologue", "decode_step", "decode_step", "prefill_step", "epilogue", "norm_quant", "indexer", "readers",
                       "topk_decode", "topk_prefill"])
    if kind == "prologue":
        return {"kind": kind, "tokens": _log(rng, 1, 32768), "heads": rng.choice([16, 64, 128]), "padding": rng.choice([0.0, 0.1]),
                "max_pos": rng.choice([65536, 131072]), "slots": rng.choice(["random", "blocks"])}
    if kind == "decode_step":
        context = _log(rng, 2048, 65536)
        return {"kind": kind, "requests": min(_log(rng, 1, 256), (1 << 22) // context), "next_n": rng.choice([1, 1, 2]),
                "heads": rng.choice([16, 64, 128]), "context": context, "topk": rng.choice([512, 1024]), "fp4": rng.random() < 0.5}
    if kind == "prefill_step":
        return {"kind": kind, "tokens": _log(rng, 200, 8192), "requests": rng.randint(1, 8), "prefix": _log(rng, 256, 16384),
                "heads": rng.choice([16, 64, 128]), "topk": rng.choice([512, 1024]), "fp4": rng.random() < 0.5}
    if kind == "epilogue":
        return {"kind": kind, "tokens": _log(rng, 1, 16384), "heads": rng.choice([16, 64, 128]), "packed": rng.random() < 0.5}
    if kind == "norm_quant":
        return {"kind": kind, "tokens": _log(rng, 1, 32768), "ue8m0": rng.random() < 0.5, "column_major": rng.random() < 0.5}
    if kind == "indexer":
        return {"kind": kind, "tokens": _log(rng, 1, 65536), "fp4": rng.random() < 0.5}
    if kind == "readers":
        return {"kind": kind, "requests": rng.randint(1, 32), "longest": _log(rng, 256, 16384)}
    if kind == "topk_decode":
        rows = _log(rng, 1, 512)
        return {"kind": kind, "rows": rows, "width": _log(rng, 2048, 262144), "topk": rng.choice([512, 1024, 2048]), "persistent": rng.random() < 0.5}
    return {"kind": kind, "rows": _log(rng, 64, 4096), "width": _log(rng, 2048, 65536), "topk": rng.choice([512, 1024, 2048])}


# ---- sizes that follow from a case -----------------------------------------------------------------------------------
def _ragged(count, longest):
    """`count` lengths in [longest/4, longest], the first one the longest."""
    return [longest - (i * 7919) % (longest - longest // 4 + 1) for i in range(count)]


def _split(total, parts):
    """`total` tokens over `parts` requests, unevenly, each at least one."""
    weights = [3 + (i * 5) % 7 for i in range(parts)]
    sizes = [max(1, total * w // sum(weights)) for w in weights]
    sizes[0] += total - sum(sizes)
    return sizes


def _prefill_lens(c):
    """(query lengths, sequence lengths, compressed lengths) of the chunk's requests."""
    query = _split(c["tokens"], c["requests"])
    seq = [q + p for q, p in zip(query, _ragged(c["requests"], c["prefix"]))]
    return query, seq, [s // RATIO for s in seq]


# ---- tensors ---------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _act(g, *shape):
    return torch.empty(shape, dtype=torch.bfloat16, device=DEV).normal_(generator=g)


def _int(values, dtype=torch.int32):
    return torch.tensor(values, dtype=dtype, device=DEV)


def _cos_sin(max_pos):
    inv = 10000.0 ** (-torch.arange(0, 64, 2, dtype=torch.float64, device=DEV) / 64)
    angle = torch.outer(torch.arange(max_pos, dtype=torch.float64, device=DEV), inv)
    return torch.cat((angle.cos(), angle.sin()), dim=-1).float().contiguous()


def _latent_cache(g, blocks):
    """A cache in use: e4m3 bytes and bf16 values below 2 in magnitude, scale codes near 2^-5, a zero pad byte."""
    cache = torch.randint(0, 256, (blocks, BLOCK * 584), generator=g, device=DEV, dtype=torch.uint8).bitwise_and_(0xBF)
    codes = torch.randint(118, 126, (blocks, BLOCK, 8), generator=g, device=DEV, dtype=torch.uint8)
    codes[..., 7] = 0
    cache[:, BLOCK * 576:] = codes.view(blocks, -1)
    return cache


def _index_cache(g, blocks):
    """fp8 keys, then one fp32 power-of-two scale per key."""
    cache = torch.randint(0, 256, (blocks, BLOCK, 132), generator=g, device=DEV, dtype=torch.uint8).bitwise_and_(0xBF)
    scale = torch.randint(-9, -3, (blocks, BLOCK), generator=g, device=DEV).float().exp2()
    cache.view(blocks, -1)[:, BLOCK * 128:] = scale.view(torch.uint8).view(blocks, -1)
    return cache


def _table(g, lens, blocks):
    """Block table [requests, most blocks of a request] of distinct random blocks."""
    need = [-(-n // BLOCK) for n in lens]
    perm = torch.randperm(blocks, generator=g, device=DEV).to(torch.int32)
    table = torch.zeros(len(lens), max(need), dtype=torch.int32, device=DEV)
    at = 0
    for r, n in enumerate(need):
        table[r, :n] = perm[at:at + n]
        at += n
    return table


def _slots_of(table, request, position):
    return (table[request, position // BLOCK].to(torch.int64) * BLOCK + position % BLOCK).contiguous()


def _blocks_for(lens):
    return max(CACHE_BLOCKS, sum(-(-n // BLOCK) for n in lens))


def _prepare_prologue(c, g):
    n, h = c["tokens"], c["heads"]
    s = {"q": _act(g, n, h, HEAD), "kv": _act(g, n, HEAD), "cache": _latent_cache(g, CACHE_BLOCKS), "cs": _cos_sin(c["max_pos"])}
    s["pos"] = torch.randint(0, c["max_pos"], (n,), generator=g, device=DEV)
    if c["slots"] == "random":
        slots = torch.randperm(CACHE_BLOCKS * BLOCK, generator=g, device=DEV)[:n]
    else:  # a prefill fills randomly chosen blocks in order
        i = torch.arange(n, device=DEV)
        slots = torch.randperm(CACHE_BLOCKS, generator=g, device=DEV)[i // BLOCK] * BLOCK + i % BLOCK
    padded = torch.randperm(n, generator=g, device=DEV)[: int(n * c["padding"])]
    s["slots"] = slots.contiguous()
    s["slots"][padded] = -1
    hot = torch.randperm(n, generator=g, device=DEV)[: n // 100]  # outlier tokens
    s["q"][hot] *= 50
    s["kv"][hot] *= 50
    return s


def _prepare_layer(g, n, heads, max_pos):
    """Activations and weights both kinds of step have."""
    return {
        "qr": _act(g, n, Q_LORA), "kv": _act(g, n, HEAD), "wq": 1 + 0.1 * _act(g, Q_LORA), "wkv": 1 + 0.1 * _act(g, HEAD),
        "q": _act(g, n, heads, HEAD), "o": _act(g, n, heads, HEAD), "cs": _cos_sin(max_pos),
        "iq": _act(g, n, INDEX_HEADS, INDEX_DIM), "iw": _act(g, n, INDEX_HEADS),
    }


def _prepare_decode(c, g):
    reqs, nn = c["requests"], c["next_n"]
    n = reqs * nn
    lens = _ragged(reqs, c["context"])
    blocks = _blocks_for(lens)
    s = _prepare_layer(g, n, c["heads"], 65536)
    request = torch.arange(n, device=DEV) // nn
    position = _int(lens, torch.int64)[request] - nn + torch.arange(n, device=DEV) % nn
    s["table"] = _table(g, lens, blocks)
    s["request"] = request.to(torch.int32)
    s["pos"] = position.contiguous()
    s["slots"] = _slots_of(s["table"], request, position)
    s["cache"], s["icache"] = _latent_cache(g, blocks), _index_cache(g, blocks)
    s["ik"] = _act(g, n, INDEX_DIM)
    s["seq"] = _int(lens)
    s["logits"] = torch.empty(n, -(-c["context"] // BLOCK) * BLOCK, device=DEV).normal_(generator=g)
    s["picked"] = torch.empty(n, c["topk"], dtype=torch.int32, device=DEV)
    return s


def _prepare_prefill(c, g):
    query, seq, comp = _prefill_lens(c)
    n, reqs, blocks = c["tokens"], c["requests"], _blocks_for(seq)
    s = _prepare_layer(g, n, c["heads"], 65536)
    request = torch.repeat_interleave(torch.arange(reqs, device=DEV), _int(query, torch.int64))
    position = torch.cat([torch.arange(e - q, e, device=DEV) for q, e in zip(query, seq)])
    s["pos"], s["table"] = position.contiguous(), _table(g, seq, blocks)
    s["slots"] = _slots_of(s["table"], request, position)
    s["cache"] = _latent_cache(g, blocks)
    # compressed keys: one per RATIO tokens, those completed by this chunk are inserted
    s["ctable"], s["icache"] = _table(g, comp, CACHE_BLOCKS), _index_cache(g, CACHE_BLOCKS)
    done = ((position + 1) % RATIO == 0).nonzero().flatten()
    s["islots"] = _slots_of(s["ctable"], request[done], (position[done] + 1) // RATIO - 1)
    s["ik"] = _act(g, done.numel(), INDEX_DIM)
    starts = [sum(comp[:r]) for r in range(reqs + 1)]
    s["cu"] = _int(starts)
    s["ik8"] = torch.empty(starts[-1], INDEX_DIM, dtype=torch.float8_e4m3fn, device=DEV)
    s["iks"] = torch.empty(starts[-1], 4, dtype=torch.uint8, device=DEV)
    s["logits"] = torch.empty(n, -(-starts[-1] // 8) * 8, device=DEV).normal_(generator=g)
    s["row_starts"] = s["cu"][request].contiguous()
    s["row_ends"] = (s["row_starts"] + (position + 1) // RATIO).to(torch.int32).contiguous()
    s["picked"] = torch.empty(n, c["topk"], dtype=torch.int32, device=DEV)
    gather = [min(e, q + WINDOW - 1) for q, e in zip(query, seq)]
    s["N"] = max(comp)  # the gathered buffer of a request: compressed keys, then the window's keys
    s["M"] = s["N"] + max(gather)
    s["gathered"] = torch.zeros(reqs, s["M"], HEAD, dtype=torch.bfloat16, device=DEV)
    s["seq"], s["gather"] = _int(seq), _int(gather)
    s["qsl"] = _int([sum(query[:r]) for r in range(reqs + 1)])
    return s


def prepare(case, seed):
    c, g, kind = case, _gen(seed), case["kind"]
    if kind == "prologue":
        s = _prepare_prologue(c, g)
    elif kind == "decode_step":
        s = _prepare_decode(c, g)
    elif kind == "prefill_step":
        s = _prepare_prefill(c, g)
    elif kind == "epilogue":
        s = {"o": _act(g, c["tokens"], c["heads"], HEAD), "pos": torch.randint(0, 65536, (c["tokens"],), generator=g, device=DEV), "cs": _cos_sin(65536)}
    elif kind == "norm_quant":
        n = c["tokens"]
        s = {"x": _act(g, n, HIDDEN), "qr": _act(g, n, Q_LORA), "kv": _act(g, n, HEAD), "wq": 1 + 0.1 * _act(g, Q_LORA), "wkv": 1 + 0.1 * _act(g, HEAD)}
    elif kind == "indexer":
        n = c["tokens"]
        s = {"iq": _act(g, n, INDEX_HEADS, INDEX_DIM), "iw": _act(g, n, INDEX_HEADS), "ik": _act(g, n, INDEX_DIM), "cs": _cos_sin(65536),
             "pos": torch.randint(0, 65536, (n,), generator=g, device=DEV), "icache": _index_cache(g, CACHE_BLOCKS)}
        i = torch.arange(n, device=DEV)
        s["slots"] = (torch.randperm(CACHE_BLOCKS, generator=g, device=DEV)[i // BLOCK] * BLOCK + i % BLOCK).contiguous()
    elif kind == "readers":
        lens = _ragged(c["requests"], c["longest"])
        total = sum(lens)
        blocks = _blocks_for(lens)
        s = {"table": _table(g, lens, blocks), "cache": _latent_cache(g, blocks), "icache": _index_cache(g, blocks), "seq": _int(lens),
             "cu": _int([sum(lens[:r]) for r in range(len(lens) + 1)]),
             "out": torch.zeros(len(lens), c["longest"], HEAD, dtype=torch.bfloat16, device=DEV),
             "ik8": torch.empty(total, INDEX_DIM, dtype=torch.float8_e4m3fn, device=DEV), "iks": torch.empty(total, 4, dtype=torch.uint8, device=DEV)}
    else:
        rows, width = c["rows"], c["width"]
        s = {"logits": torch.empty(rows, width, device=DEV).normal_(generator=g), "picked": torch.empty(rows, c["topk"], dtype=torch.int32, device=DEV)}
        if kind == "topk_decode":
            s["seq"] = _int(_ragged(rows, width))
            s["workspace"] = torch.zeros(1 << 20, dtype=torch.uint8, device=DEV) if c["persistent"] else None
        else:  # causal: the last row sees the whole width
            s["row_starts"] = torch.zeros(rows, dtype=torch.int32, device=DEV)
            s["row_ends"] = (width - (rows - 1) // RATIO + torch.arange(rows, device=DEV) // RATIO).clamp(1, width).to(torch.int32)
    return dict(s, case=c)


# ---- one pass --------------------------------------------------------------------------------------------------------
def _ascending(picked):
    """The selection leaves its positions in no particular order; callers that want reproducible attention sums, and
    cache reads in address order, sort them."""
    return picked.sort(dim=1).values


def _front(s):
    """What both kinds of step begin with, up to the indexer's query."""
    c = s["case"]
    qr, kv = fg.fused_q_kv_rmsnorm(s["qr"], s["kv"], s["wq"], s["wkv"], EPS)
    qr8, qr_scale = fg.per_token_group_quant_fp8(qr, 128, scale_ue8m0=True)
    fg.fused_deepseek_v4_qnorm_rope_kv_rope_quant_insert(s["q"], kv, s["cache"], s["slots"], s["pos"], s["cs"], EPS, BLOCK)
    iq, iw = fg.fused_indexer_q_rope_quant(s["pos"], s["iq"], s["cs"], s["iw"], SOFTMAX_SCALE, HEAD_SCALE, use_fp4=c["fp4"])
    return [qr, kv, qr8, qr_scale, s["q"], s["cache"], iq, iw]


def _epilogue(s, packed):
    return fg.fused_inv_rope_fp8_quant(s["o"], s["pos"], s["cs"], O_GROUPS, s["o"].shape[1] // O_GROUPS, tma_aligned_scales=packed)


def _run_decode(s):
    c, x = s["case"], s["logits"]
    out = _front(s)
    fg.indexer_k_quant_and_cache(s["ik"], s["icache"], s["slots"], 128, "ue8m0")
    fg.top_k_per_row_decode(x, c["next_n"], s["seq"], s["picked"], x.shape[0], x.stride(0), x.stride(1), c["topk"])
    keys, lens = fg.compute_global_topk_indices_and_lens(_ascending(s["picked"]), s["request"], s["table"], BLOCK)
    return out + [s["icache"], keys, lens, _epilogue(s, True)]


def _run_prefill(s):
    c, x = s["case"], s["logits"]
    out = _front(s)
    fg.indexer_k_quant_and_cache(s["ik"], s["icache"], s["islots"], 128, "ue8m0")
    fg.cp_gather_indexer_k_quant_cache(s["icache"], s["ik8"], s["iks"], s["ctable"], s["cu"])
    fg.top_k_per_row_prefill(x, s["row_starts"], s["row_ends"], s["picked"], x.shape[0], x.stride(0), x.stride(1), c["topk"])
    fg.dequantize_and_gather_k_cache(s["gathered"], s["cache"], s["seq"], s["gather"], s["table"], BLOCK, offset=s["N"])
    # unused entries are -1: descending order keeps them behind the selected positions
    picked = s["picked"].sort(dim=1, descending=True).values
    rows, lens = fg.combine_topk_swa_indices(picked, s["qsl"], s["seq"], s["gather"], WINDOW, RATIO, c["topk"], s["M"], s["N"])
    return out + [s["icache"], s["ik8"], s["iks"], s["gathered"], rows, lens, _epilogue(s, True)]


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "prologue":
        fg.fused_deepseek_v4_qnorm_rope_kv_rope_quant_insert(s["q"], s["kv"], s["cache"], s["slots"], s["pos"], s["cs"], EPS, BLOCK)
        return [s["q"], s["cache"]]
    if kind == "decode_step":
        return _run_decode(s)
    if kind == "prefill_step":
        return _run_prefill(s)
    if kind == "epilogue":
        return _epilogue(s, c["packed"])
    if kind == "norm_quant":
        quant = lambda x: fg.per_token_group_quant_fp8(x, 128, column_major_scales=c["column_major"], scale_ue8m0=c["ue8m0"])  # noqa: E731
        hidden = quant(s["x"])
        qr, kv = fg.fused_q_kv_rmsnorm(s["qr"], s["kv"], s["wq"], s["wkv"], EPS)
        return [hidden, qr, kv, quant(qr)]
    if kind == "indexer":
        q = fg.fused_indexer_q_rope_quant(s["pos"], s["iq"], s["cs"], s["iw"], SOFTMAX_SCALE, HEAD_SCALE, use_fp4=c["fp4"])
        fg.indexer_k_quant_and_cache(s["ik"], s["icache"], s["slots"], 128, "ue8m0")
        return [q, s["icache"]]
    if kind == "readers":
        fg.dequantize_and_gather_k_cache(s["out"], s["cache"], s["seq"], None, s["table"], BLOCK)
        fg.cp_gather_indexer_k_quant_cache(s["icache"], s["ik8"], s["iks"], s["table"], s["cu"])
        return [s["out"], s["ik8"], s["iks"]]
    x = s["logits"]
    if kind == "topk_prefill":
        fg.top_k_per_row_prefill(x, s["row_starts"], s["row_ends"], s["picked"], x.shape[0], x.stride(0), x.stride(1), c["topk"])
    elif c["persistent"]:
        fg.persistent_topk(x, s["seq"], s["picked"], s["workspace"], c["topk"], c["width"])
    else:
        fg.top_k_per_row_decode(x, 1, s["seq"], s["picked"], x.shape[0], x.stride(0), x.stride(1), c["topk"])
    return _ascending(s["picked"])


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def _prologue_bytes(tokens, heads, inserted):
    return tokens * (2048 * heads + 264 + 8) + inserted * 1608


def _quant_bytes(tokens, cols):
    return tokens * cols * (2 + 1 + 4 / 128)


def _epilogue_bytes(tokens, heads, packed):
    return tokens * (heads * (1024 + 512 + (4 if packed else 16)) + 264)


def _indexer_q_bytes(tokens, fp4):
    return tokens * (INDEX_HEADS * (256 + (68 if fp4 else 128) + 6) + 264)


def _front_bytes(tokens, heads, fp4):
    return (tokens * (Q_LORA + HEAD) * 4 + _quant_bytes(tokens, Q_LORA) + _prologue_bytes(tokens, heads, tokens) + _indexer_q_bytes(tokens, fp4)
            + _epilogue_bytes(tokens, heads, True))


def _bytes(c):
    kind = c["kind"]
    if kind == "prologue":
        return _prologue_bytes(c["tokens"], c["heads"], c["tokens"] - int(c["tokens"] * c["padding"]))
    if kind == "decode_step":
        n = c["requests"] * c["next_n"]
        return (_front_bytes(n, c["heads"], c["fp4"]) + n * 396 + c["next_n"] * 4 * sum(_ragged(c["requests"], c["context"]))
                + n * c["topk"] * 12)
    if kind == "prefill_step":
        n = c["tokens"]
        query, seq, comp = _prefill_lens(c)
        seen = sum((p + 1) // RATIO for q, e in zip(query, seq) for p in range(e - q, e))
        gathered = sum(min(e, q + WINDOW - 1) for q, e in zip(query, seq))
        width = -(-(c["topk"] + WINDOW) // 128) * 128
        return (_front_bytes(n, c["heads"], c["fp4"]) + n // RATIO * 396 + sum(comp) * 264 + 4 * seen + gathered * 1608
                + n * 4 * (2 * c["topk"] + width + 1))
    if kind == "epilogue":
        return _epilogue_bytes(c["tokens"], c["heads"], c["packed"])
    if kind == "norm_quant":
        return _quant_bytes(c["tokens"], HIDDEN) + _quant_bytes(c["tokens"], Q_LORA) + c["tokens"] * (Q_LORA + HEAD) * 4
    if kind == "indexer":
        return _indexer_q_bytes(c["tokens"], c["fp4"]) + c["tokens"] * 396
    if kind == "readers":
        return sum(_ragged(c["requests"], c["longest"])) * (1608 + 264)
    if kind == "topk_decode":
        return 4 * sum(_ragged(c["rows"], c["width"])) + c["rows"] * c["topk"] * 4
    ends = (min(c["width"], max(1, c["width"] - (c["rows"] - 1) // RATIO + i // RATIO)) for i in range(c["rows"]))
    return 4 * sum(ends) + c["rows"] * c["topk"] * 4


def work(case):
    # under one operation per byte everywhere: memory is the bound
    return {"bytes": float(_bytes(case)), "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("epilogue", "indexer", "readers"):
        return "exact"  # no sum whose order is free
    if kind in ("topk_decode", "topk_prefill"):
        return {"rel": 0.0, "max": 0.0, "differ": 2e-3}  # equal logits at the boundary
    if kind == "prologue":
        # the mean of squares has no fixed order: q may move by one bf16 step; cache bytes do not depend on it
        return {"rel": 2e-3, "max": 0.03, "differ": 0.0}
    # a bf16 step in a normalised value can move an e4m3 code by one step
    return {"rel": 5e-3, "max": 0.15, "differ": 2e-3}
