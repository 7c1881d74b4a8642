"""The serving work whose speed is tracked: steps of the device models and the device sampler.

A serving engine spends its GPU time in `DeviceModel.forward` (one step of the running batch) and in the sampler behind it.
The cases are the steps of the workloads of `bench_serving` at their real widths, with fewer layers than the whole
models (layers repeat, so the mix of kernels stays): single-stream decoding of GGUF weights, batched decoding in bf16 and packed Q4_K_M, prompts of a
batch, suffixes behind a cached prefix, a long prompt's last chunk, the products of fp8 and NVFP4 layers, and stochastic sampling. Decode steps are
captured in a CUDA graph and replayed, as the engine does for its decode buckets; steps with prompts are launched eagerly, as
the engine does too.

Where two experts score almost the same, another rounding ahead of the router sends a row another way, and an activation between two 4- or 8-bit values
becomes one or the other: the numbers behind it are then others, neither right nor wrong, and they differ by more than a kernel's error. So the
mixture of experts is measured in prompt steps with few logit rows and one layer, and fp8 and NVFP4 by the products of a layer on given rows, the
quantiser of the rows included.

Weights come from `init_random` / `init_random_quant`, which draw them from one seeded generator on the GPU; `exact` draws the same numbers and
computes the step in 64 bits with plain torch.
"""
import math

import torch

from oxide_tech_llm_engine_b200 import ops
from oxide_tech_llm_engine_b200.models.config import preset
from oxide_tech_llm_engine_b200.models.llama import DeviceModel, StepInputs

PAGE = 16
MAX_SPLITS = 16
GOLDEN = 0.6180339887498949


def listed():
    return [
        # one user, the smallest model: launches and memory latency (300 prompt tokens + 128 generated, Q4_0 with a Q8_0 head)
        dict(name="single-1b-q4_0", kind="decode", model="tinyllama-1.1b", layers=22, weights="Q4_0", rows=1, ctx_min=428, ctx_max=428),
        # one user of an 8B model in the usual mixed GGUF layout
        dict(name="single-8b-q4_k_m", kind="decode", model="llama3-8b", layers=4, weights="Q4_K_M", rows=1, ctx_min=1531, ctx_max=1531),
        # continuous batching of 64 requests (prompts of 128 to 1024 tokens, up to 512 generated)
        dict(name="batch64-8b", kind="decode", model="llama3-8b", layers=6, weights="bf16", rows=64, ctx_min=128, ctx_max=1536),
        # the headline decode step: 256 requests, prompts of 128 to 4096 tokens and 512 generated
        dict(name="batch256-70b", kind="decode", model="llama3-70b", layers=3, weights="bf16", rows=256, ctx_min=128, ctx_max=4608),
        # packed weights served to a small batch, at a size whose bf16 copy would not fit beside them
        dict(name="batch32-70b-q4_k_m", kind="decode", model="llama3-70b", layers=2, weights="Q4_K_M", rows=32, ctx_min=128, ctx_max=4608),
        # prompts of a batch in one step, ragged
        dict(name="prompts-8b", kind="prompts", model="llama3-8b", layers=4, weights="bf16", prompts=14, len_min=128, len_max=1024, past=0),
        dict(name="prompts-moe", kind="prompts", model="mixtral-8x7b", layers=1, weights="bf16", prompts=4, len_min=256, len_max=2048, past=0),
        # suffixes behind a cached prefix of 2048 tokens, at 70B widths
        dict(name="suffixes-70b", kind="prompts", model="llama3-70b", layers=2, weights="bf16", prompts=16, len_min=128, len_max=128, past=2048),
        # the last 8192 tokens of a prompt of 32768
        dict(name="long-8b", kind="prompts", model="llama3-8b", layers=2, weights="bf16", prompts=1, len_min=8192, len_max=8192, past=24576),
        # the projections of a layer in block-scaled fp8, for an odd number of decode rows
        dict(name="project117-70b-fp8", kind="project", model="llama3-70b", weights="fp8", rows=117),
        # the expert products of a layer in NVFP4, for 128 decode rows with two experts each
        dict(name="project128-moe-nvfp4", kind="project", model="mixtral-8x7b", weights="nvfp4", rows=128),
        # one token for each of 64 requests from their logits: temperature, top-k and top-p
        dict(name="sample64", kind="sample", vocab=128256, rows=64, temperature=0.8, top_k=50, top_p=0.95, min_p=0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; sizes are odd ones as often as not."""
    kind = rng.choice(("decode", "decode", "decode", "decode", "prompts", "prompts", "prompts", "project", "project", "sample"))
    if kind == "sample":
        return dict(kind=kind, vocab=rng.choice((32000, 128256)), rows=_log_int(rng, 1, 256), temperature=round(rng.uniform(0.3, 1.3), 2),
                    top_k=rng.choice((0, 20, 50, 200)), top_p=rng.choice((0.8, 0.9, 0.95, 1.0)), min_p=rng.choice((0.0, 0.0, 0.05)))
    if kind == "project":
        model, weights, top = rng.choice((("llama3-70b", "fp8", 4096), ("llama3-8b", "fp8", 8192), ("mixtral-8x7b", "nvfp4", 4096)))
        return dict(kind=kind, model=model, weights=weights, rows=_log_int(rng, 1, top))
    if kind == "decode":
        model, weights, layers, top = rng.choice((
            ("tinyllama-1.1b", "Q4_0", 22, 4), ("tinyllama-1.1b", "bf16", 22, 64), ("llama3-8b", "Q4_K_M", 4, 4), ("llama3-8b", "bf16", 6, 128),
            ("llama3-70b", "bf16", 3, 256), ("llama3-70b", "Q4_K_M", 2, 64)))
        ctx = _log_int(rng, 128, {"tinyllama-1.1b": 2048, "llama3-8b": 8192}.get(model, 4608))
        rows = _log_int(rng, 1, top)
        return dict(kind=kind, model=model, layers=layers, weights=weights, rows=rows, ctx_min=max(1, ctx // rng.choice((1, 4, 32))), ctx_max=ctx)
    model, weights, layers = rng.choice((("tinyllama-1.1b", "bf16", 22), ("llama3-8b", "bf16", 4), ("llama3-70b", "bf16", 2), ("mixtral-8x7b", "bf16", 1)))
    prompts = _log_int(rng, 1, 16 if model != "mixtral-8x7b" else 4)
    longest = _log_int(rng, 32, min(2048, 8192 // prompts))
    past = rng.choice((0, 0, 2048, PAGE * _log_int(rng, 1, 512))) if model.startswith("llama3") else 0
    return dict(kind=kind, model=model, layers=layers, weights=weights, prompts=prompts, len_min=max(1, longest // rng.choice((1, 2, 8))), len_max=longest,
                past=past)


# ------------------------------------------------------------------------------------------------ the step of a case
def _lens(n, lo, hi):
    """n lengths spread evenly over [lo, hi], in no order; one sequence has the longest."""
    if n == 1:
        return [hi]
    return [hi if i == 0 else lo + int((hi - lo + 1) * ((i * GOLDEN) % 1.0)) for i in range(n)]


def _config(case):
    return preset(case["model"], n_layers=case["layers"])


def _plan(case):
    """(new tokens of every sequence, context lengths with them)."""
    if case["kind"] == "decode":
        ctx = _lens(case["rows"], case["ctx_min"], case["ctx_max"])
        return [1] * len(ctx), ctx
    lens = _lens(case["prompts"], case["len_min"], case["len_max"])
    return lens, [n + case["past"] for n in lens]


def _tables(case, cfg, seed):
    """Token ids and the pages of every sequence, which lie anywhere in the pool."""
    lens, ctx = _plan(case)
    pages = [(c + PAGE - 1) // PAGE for c in ctx]
    g = torch.Generator().manual_seed(seed)
    tokens = torch.randint(0, cfg.vocab_size, (sum(lens),), generator=g)
    order = torch.randperm(sum(pages), generator=g)
    table = torch.zeros(len(ctx), max(pages), dtype=torch.int64)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    return lens, ctx, tokens, table, at


def _fill_cache(cache, cfg, gen):
    """Keys and values of earlier tokens as random projections of normed rows leave them."""
    for t in cache:
        t.normal_(0.0, 0.02 * math.sqrt(cfg.d_model), generator=gen)


def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    if case["kind"] == "project":
        return _prepare_project(case, seed)
    dev = torch.device("cuda", torch.cuda.current_device())
    cfg = _config(case)
    lens, ctx, tokens, table, n_pages = _tables(case, cfg, seed)
    m, n, decode = sum(lens), len(lens), case["kind"] == "decode"
    packed = case["weights"] != "bf16"
    model = DeviceModel(cfg, device=dev, max_tokens=max(m, 64), max_seqs=max(n, 8), num_blocks=n_pages + 1, max_blocks_per_seq=table.shape[1],
                        max_logits=max(n, 64), max_splits=MAX_SPLITS, weight_mode="quant" if packed else "bf16")
    if packed:
        model.init_random_quant(case["weights"], seed)
    else:
        model.init_random(seed)
    if decode or case["past"]:
        gen = torch.Generator(device=dev).manual_seed(seed + 1)
        _fill_cache(model.k_cache, cfg, gen)
        _fill_cache(model.v_cache, cfg, gen)
    i32 = dict(dtype=torch.int32, device=dev)
    pos = torch.cat([torch.arange(c - q, c) for q, c in zip(lens, ctx)])
    seq = torch.repeat_interleave(torch.arange(n), torch.tensor(lens))
    slots = table[seq, pos // PAGE] * PAGE + pos % PAGE
    start = [sum(lens[:i]) for i in range(n)]
    last = torch.full((m,), -1, dtype=torch.int64)
    last[torch.tensor(start) + torch.tensor(lens) - 1] = torch.arange(n)
    tiles = [(i, q0) for i, q in enumerate(lens) for q0 in range(0, q, 128)]
    # the engine's rule for the pages of one KV split
    splits = max(1, min(MAX_SPLITS, -(-(12 if cfg.n_kv_heads >= 4 else 4) * ops.sm_count(dev) // (n * cfg.n_kv_heads))))
    per_split = (max(4, -(-((max(ctx) + PAGE - 1) // PAGE) // splits)) + 3) // 4 * 4
    t32 = lambda v: torch.as_tensor(v).to(**i32)
    step = StepInputs(m=m, n_decode=n if decode else 0, n_prefill=0 if decode else n, n_tiles=0 if decode else len(tiles), n_logits=n,
                      token_ids=t32(tokens), positions=t32(pos), slot_mapping=slots.to(dev), seq_lens=t32(ctx), block_tables=t32(table),
                      pages_per_split=t32([per_split]), tile_seq=t32([t[0] for t in tiles]), tile_q0=t32([t[1] for t in tiles]), q_start=t32(start),
                      q_lens=t32(lens), ctx_lens=t32(ctx), prefill_block_tables=t32(table), logit_map=t32(last), max_ctx=max(ctx))
    state = {"model": model, "step": step, "graph": None}
    if decode:
        model.forward(step)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["logits"] = model.forward(step)
        state["graph"] = graph
    return state


def _prepare_sample(case, seed):
    """Logits as a language model leaves them: a broad bell and a few dozen likely tokens per row."""
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    rows, vocab = case["rows"], case["vocab"]
    logits = torch.randn(rows, vocab, device=dev, generator=gen) * 2.5
    likely = torch.randint(0, vocab, (rows, 48), device=dev, generator=gen)
    logits.scatter_add_(1, likely, torch.empty(rows, 48, device=dev).exponential_(0.4, generator=gen))
    full = lambda v, dt: torch.full((rows,), v, dtype=dt, device=dev)
    return {"logits": logits, "tokens": torch.zeros(rows, dtype=torch.int32, device=dev), "logprob": torch.zeros(rows, device=dev),
            "params": dict(temperature=full(case["temperature"], torch.float32), top_k=full(case["top_k"], torch.int32),
                           top_p=full(case["top_p"], torch.float32), min_p=full(case["min_p"], torch.float32),
                           seeds=torch.randint(0, 1 << 62, (rows,), device=dev, generator=gen),
                           counters=torch.randint(0, 512, (rows,), device=dev, generator=gen))}


def _project_parts(case, seed):
    """Weights and given input rows of every product of a layer: (name, weight [groups, N, K], rows [groups, M, K]), seeded."""
    cfg = preset(case["model"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    d, ff, rows = cfg.d_model, cfg.ffn_dim, case["rows"]
    if case["weights"] == "fp8":
        sizes = [("qkv", 1, cfg.q_dim + 2 * cfg.kv_dim, d, 1.0), ("o", 1, d, cfg.q_dim, 0.5), ("gate_up", 1, 2 * ff, d, 1.0), ("down", 1, d, ff, 0.5)]
    else:
        sizes = [("gate_up", cfg.n_experts, 2 * ff, d, 1.0), ("down", cfg.n_experts, d, ff, 0.5)]
    for name, groups, n, k, std in sizes:
        x = torch.empty(groups, rows, k, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=gen)
        if case["weights"] == "fp8":
            yield name, torch.empty(groups, n, k, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=gen), x
        else:
            yield name, _random_fp4(groups, n, k, gen), x


def _expert_rows(case):
    """Rows of every expert: two per token, unevenly."""
    e = preset(case["model"]).n_experts
    counts = [int(2 * case["rows"] * (0.5 + ((i + 1) * GOLDEN) % 1.0) / e) for i in range(e)]
    counts[0] += 2 * case["rows"] - sum(counts)
    return [min(c, case["rows"]) for c in counts]


def _prepare_project(case, seed):
    rows, parts = case["rows"], []
    for name, w, x in _project_parts(case, seed):
        if case["weights"] == "fp8":
            parts.append((name, ops.quant_weight_fp8_block(w[0]), x[0], None, torch.empty(rows, w.shape[1], dtype=torch.bfloat16, device="cuda")))
            continue
        q, scale = w
        groups, n, k = q.shape[0], q.shape[1], 2 * q.shape[2]
        atoms = torch.full((groups * (n // 128) * (k // 64) * 512,), 0x2E, dtype=torch.uint8, device="cuda")    # e4m3 0.4375
        weight = ops.Nvfp4Weight(q, atoms, torch.full((groups,), scale / 0.4375, device="cuda"), n, k)
        cap = (rows + 127) // 128 * 128     # scale atoms cover 128 rows
        slab = torch.zeros(groups, cap, k, dtype=torch.bfloat16, device="cuda")
        slab[:, :rows] = x
        bufs = (torch.zeros(groups * cap * k // 2, dtype=torch.uint8, device="cuda"),
                torch.zeros(groups * cap // 128 * (k // 64) * 512, dtype=torch.uint8, device="cuda"), torch.ones(groups * cap, device="cuda"))
        out = torch.zeros(groups, cap, n // 2 if name == "gate_up" else n, dtype=torch.bfloat16, device="cuda")
        parts.append((name, weight, slab, bufs, out))
    counts = None
    if case["weights"] == "nvfp4":
        counts = torch.tensor(_expert_rows(case), dtype=torch.int32, device="cuda")
    return {"parts": parts, "counts": counts, "m_tiles": (2 * rows + 127) // 128 + 8}


def _run_project(state):
    counts, got = state["counts"], {}
    for name, weight, x, bufs, out in state["parts"]:
        if counts is None:
            a8, scale = ops.quant_act_fp8(x)
            got[name] = ops.gemm_fp8_block(a8, scale, weight[0], weight[1], out=out)
        else:
            q, atoms, scale = ops.quant_act_nvfp4(x, bufs, counts)
            ops.gemm(q, weight.q, out=out, epi=ops.EPI_SWIGLU_BF16 if name == "gate_up" else ops.EPI_STORE_BF16, group_counts=counts,
                     m_tiles=state["m_tiles"], sfa=atoms, sfb=weight.sf, a_gscale=scale, w_gscale=weight.gscale)
            got[name] = out
    return got


def run(state):
    if "parts" in state:
        return _run_project(state)
    if "params" in state:
        ops.sample(state["logits"], state["tokens"], out_logit=state["logprob"], **state["params"])
        return {"tokens": state["tokens"], "logprob": state["logprob"]}
    model = state["model"]
    if state["graph"] is not None:
        state["graph"].replay()
        logits = state["logits"]
    else:
        logits = model.forward(state["step"])
    # what a step leaves: the logits, and the keys and values of its tokens in the cache (the last layer's stand behind all others)
    return {"logits": logits, "k": model.k_cache[-1], "v": model.v_cache[-1]}


def _stored_bytes(kind, count):
    """Bytes of `count` weights as they are stored."""
    return count * {"bf16": 2.0, "fp8": 1.0, "nvfp4": 0.5625, "Q4_0": 18 / 32, "Q8_0": 34 / 32, "Q4_K": 144 / 256, "Q6_K": 210 / 256}[kind]


def work(case):
    """Weights once, the context's keys and values once (once per query tile's sequence), new ones and logits written once;
    two operations per weight and row, four per visible key, head and value."""
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 4.0 * n, "flops": 3.0 * n}
    if case["kind"] == "project":
        cfg, rows = preset(case["model"]), case["rows"]
        d, ff = cfg.d_model, cfg.ffn_dim
        attn = (cfg.q_dim + 2 * cfg.kv_dim) * d + d * cfg.q_dim
        if case["weights"] == "fp8":
            one = attn + 3 * ff * d
            return {"bytes": float(one) + 2.0 * rows * (5 * d + 3 * ff + 2 * cfg.kv_dim), "flops": 2.0 * rows * one}
        hit, slots = sum(c > 0 for c in _expert_rows(case)), sum(_expert_rows(case))
        return {"bytes": _stored_bytes("nvfp4", 3.0 * ff * d * hit) + 2.0 * slots * (2 * d + 2 * ff), "flops": 6.0 * slots * ff * d}
    cfg, w = _config(case), case["weights"]
    lens, ctx = _plan(case)
    m, n, d = sum(lens), len(lens), cfg.d_model
    seen = sum(q * (c - q) + q * (q + 1) // 2 for q, c in zip(lens, ctx))
    attn = (cfg.q_dim + 2 * cfg.kv_dim) * d + d * cfg.q_dim
    one = 3 * cfg.ffn_dim * d
    experts = max(1, cfg.n_experts)
    per_row = max(1, cfg.n_experts_used)
    hit = experts * (1.0 - (1.0 - per_row / experts) ** m) if cfg.n_experts else 1.0
    dense = "Q4_K" if w == "Q4_K_M" else w
    head = "Q6_K" if w == "Q4_K_M" else "Q8_0" if w == "Q4_0" else "bf16"
    weights = cfg.n_layers * (_stored_bytes(dense, attn) + _stored_bytes(dense, one * hit))
    if w == "Q4_K_M":   # attn_v and every other ffn_down are Q6_K
        more = 210 / 256 - 144 / 256
        weights += more * d * (cfg.n_layers * cfg.kv_dim + (cfg.n_layers + 1) // 2 * cfg.ffn_dim)
    kv = 2.0 * cfg.kv_dim * cfg.n_layers * (sum(ctx) + m) * 2
    io = m * d * 2.0 + _stored_bytes(head, cfg.vocab_size * d) + 4.0 * n * cfg.vocab_size
    flops = cfg.n_layers * (2.0 * m * (attn + one * per_row + experts * d * (cfg.n_experts > 0)) + 4.0 * seen * cfg.q_dim) + 2.0 * n * cfg.vocab_size * d
    return {"bytes": weights + kv + io, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 1e-5, "differ": 0.01}
    if case["kind"] == "project":
        # bf16 results of exact products: 0.0025 from 64 bits; a 4-bit value on the edge between two levels moves a result of NVFP4 rows by 0.013
        return {"rel": 0.01, "max": 0.1} if case["weights"] == "fp8" else {"rel": 0.02, "max": 0.2}
    # a few layers in bf16: logits are 0.007 to 0.02 from 64 bits, and up to 0.005 from themselves where atomic sums come in another order
    return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------------ the step in 64 bits
def _normal(shape, std, gen):
    return torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=gen)


def _halves(v):
    return v.view(torch.float16).double()


def _random_blocks(kind, n, k, gen):
    """The random packed matrix of `init_random_quant`, expanded by the block formats' definitions: [n, k] in 64 bits."""
    block, size, at, header = {"Q8_0": (32, 34, 0, (2.7e-4,)), "Q4_0": (32, 18, 0, (4.3e-3,)), "Q4_K": (256, 144, 0, (1.4e-4, 1.05e-3)),
                               "Q6_K": (256, 210, 208, (1.46e-5,))}[kind]
    raw = torch.randint(0, 256, (n * k // block, size), dtype=torch.uint8, device="cuda", generator=gen)
    head = torch.tensor(header, dtype=torch.float16).view(torch.uint8).cuda()
    raw[:, at:at + head.numel()] = head
    return raw.view(n, k // block, size), kind


def _expand(packed):
    raw, kind = packed
    n, blocks, size = raw.shape
    out = []
    for part in raw.split(max(1, (1 << 26) // (blocks * size))):
        b = part.reshape(-1, size)
        if kind == "Q8_0":
            v = _halves(b[:, :2].contiguous()) * b[:, 2:].contiguous().view(torch.int8).double()
        elif kind == "Q4_0":
            q = b[:, 2:]
            v = _halves(b[:, :2].contiguous()) * (torch.cat([q & 15, q >> 4], 1).double() - 8.0)
        elif kind == "Q4_K":
            d = _halves(b[:, :4].contiguous())
            s, q = b[:, 4:16], b[:, 16:].reshape(-1, 4, 1, 32)
            scale = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1).double()
            least = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1).double()
            q = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32).double()
            v = (d[:, :1] * scale)[..., None] * q - (d[:, 1:] * least)[..., None]
        else:
            low, high = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 1, 32)
            q = torch.cat([low & 15, low >> 4], 2) | (torch.cat([(high >> s) & 3 for s in (0, 2, 4, 6)], 2) << 4)
            scale = b[:, 192:208].contiguous().view(torch.int8).double().reshape(-1, 2, 4, 2, 1)
            v = _halves(b[:, 208:].contiguous())[:, :, None, None, None] * scale * (q.reshape(-1, 2, 4, 2, 16).double() - 32.0)
        out.append(v.reshape(part.shape[0], -1))
    return torch.cat(out)


def _random_fp4(groups, n, k, gen):
    """Uniform e2m1 codes with one scale of 0.4375 per block and a second one that makes them about N(0, 0.02)."""
    q = torch.randint(0, 256, (groups, n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    return q, 0.4375 * float(torch.tensor(0.02 / (2.93 * 0.4375), dtype=torch.float32))


def _fp4_values(q, scale):
    value = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device="cuda")
    value = torch.cat([value, -value]) * scale
    return torch.stack([value[(q & 15).long()], value[(q >> 4).long()]], -1).reshape(q.shape[0], -1)


def _fp8_values(w):
    """A matrix as block-scaled e4m3 keeps it: one 32-bit scale per 128 x 128 values."""
    n, k = w.shape
    b = w.float().view(n // 128, 128, k // 128, 128)
    s = b.abs().amax((1, 3), keepdim=True).clamp_min(1e-10) / 448.0
    return ((b / s).to(torch.float8_e4m3fn).double() * s.double()).view(n, k)


def _fp8_rows(x):
    """Activation rows as the fp8 path takes them: e4m3 with one scale per 128 values."""
    b = x.view(x.shape[0], -1, 128)
    s = b.abs().amax(-1, keepdim=True).clamp_min(1e-10) / 448.0
    return ((b / s).float().to(torch.float8_e4m3fn).double() * s).view(x.shape)


def _fp4_rows(x):
    """Activation rows as the NVFP4 path takes them: e2m1, an e4m3 scale per 16 values (rounded up), a 32-bit one per row."""
    b = x.view(x.shape[0], -1, 16)
    row = b.abs().amax((1, 2), keepdim=True) / (448.0 * 6.0)
    want = (b.abs().amax(-1, keepdim=True) / (6.0 * row)).float()
    s = want.to(torch.float8_e4m3fn)
    s = torch.where(s.float() < want, (s.view(torch.uint8) + 1).view(torch.float8_e4m3fn).double(), s.double()) * row
    v, level = (b / s).abs(), torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device="cuda")
    edge = (level[1:] + level[:-1]) / 2
    return (torch.copysign(level[torch.bucketize(v.clamp_max(6.0), edge)], b) * s).view(x.shape)


def _weights(case, cfg, seed):
    """Embedding, head, and the layers one by one, as 64-bit matrices behind functions."""
    kind, d, ff = case["weights"], cfg.d_model, cfg.ffn_dim
    wide = lambda t: lambda: t.double()
    if kind.startswith("Q"):
        gen = torch.Generator(device="cuda").manual_seed(seed * 1000 + 17)
        base, mixed = ("Q4_K", True) if kind == "Q4_K_M" else (kind, False)
        embed = _random_blocks("Q8_0", cfg.vocab_size, d, gen)
        head = _random_blocks("Q6_K" if mixed else "Q8_0", cfg.vocab_size, d, gen)
        yield lambda ids: _expand((embed[0][ids], embed[1])), lambda: _expand(head)
        for i in range(cfg.n_layers):
            mats = []
            for name, n, k in (("q", cfg.q_dim, d), ("k", cfg.kv_dim, d), ("v", cfg.kv_dim, d), ("o", d, cfg.q_dim), ("gate", ff, d), ("up", ff, d),
                               ("down", d, ff)):
                mats.append(_random_blocks("Q6_K" if mixed and (name == "v" or (name == "down" and i % 2 == 0)) else base, n, k, gen))
            q, k, v, o, gate, up, down = [lambda p=p: _expand(p) for p in mats]
            yield dict(qkv=lambda: torch.cat([q(), k(), v()]), o=o, experts=[(gate, up, down)], router=None)
        return
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000)
    shared = torch.Generator(device="cuda").manual_seed(seed * 1000 + 999)
    embed = _normal((cfg.vocab_size, d), 0.02, shared)
    head = _normal((cfg.vocab_size, d), 0.02, gen)
    yield lambda ids: embed[ids].double(), wide(head)
    for _ in range(cfg.n_layers):
        layer = dict(qkv=wide(_normal((cfg.q_dim + 2 * cfg.kv_dim, d), 0.02, gen)), o=wide(_normal((d, cfg.q_dim), 0.02, gen)), router=None)
        e = max(1, cfg.n_experts)
        if cfg.n_experts:
            layer["router"] = wide(_normal((e, d), 1.0 / math.sqrt(d), shared))
        gu, down = _normal((e, 2 * ff, d), 0.02, gen), _normal((e, d, ff), 0.02, gen)
        pairs = [_gate_up(gu[j], ff) for j in range(e)]
        layer["experts"] = [(lambda p=p: p[0].double(), lambda p=p: p[1].double(), wide(down[j])) for j, p in enumerate(pairs)]
        yield layer


def _gate_up(w, ff):
    """Gate and up rows of a matrix that has them in turns of 32."""
    v = w.view(ff // 32, 2, 32, -1)
    return v[:, 0].reshape(ff, -1), v[:, 1].reshape(ff, -1)


def _norm(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def exact(case, seed):
    if case["kind"] == "sample":
        return _exact_sample(case, seed)
    if case["kind"] == "project":
        return _exact_project(case, seed)
    cfg = _config(case)
    lens, ctx, tokens, table, n_pages = _tables(case, cfg, seed)
    hq, hkv, dim, m, n = cfg.n_heads, cfg.n_kv_heads, cfg.head_dim, sum(lens), len(lens)
    seq = torch.repeat_interleave(torch.arange(n), torch.tensor(lens))
    pos = torch.cat([torch.arange(c - q, c) for q, c in zip(lens, ctx)])
    block, place = table[seq, pos // PAGE].cuda(), (pos % PAGE).cuda()
    angle = pos.cuda().double()[:, None, None] / cfg.rope_theta ** (torch.arange(0, dim, 2, device="cuda").double() / dim)
    cos, sin = angle.cos(), angle.sin()

    def rotate(t):
        a, b = t.chunk(2, -1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    caches = [[torch.zeros(n_pages + 1, hkv, PAGE, dim, dtype=torch.bfloat16, device="cuda") for _ in range(cfg.n_layers)] for _ in range(2)]
    if case["kind"] == "decode" or case["past"]:
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        for cache in caches:
            _fill_cache(cache, cfg, gen)
    parts = _weights(case, cfg, seed)
    embed, head = next(parts)
    x = embed(tokens.cuda())
    start = [sum(lens[:i]) for i in range(n)]
    for li, layer in enumerate(parts):
        q, k, v = (_norm(x, cfg.rms_eps) @ layer["qkv"]().T).split([cfg.q_dim, cfg.kv_dim, cfg.kv_dim], 1)
        q, k, v = rotate(q.view(m, hq, dim)), rotate(k.reshape(m, hkv, dim)), v.reshape(m, hkv, dim)
        kc, vc = (cache[li].double() for cache in caches)
        kc[block, :, place], vc[block, :, place] = k, v
        out = torch.empty(m, hkv, hq // hkv, dim, dtype=torch.float64, device="cuda")
        for i in range(n):
            pages = table[i, :(ctx[i] + PAGE - 1) // PAGE].cuda()
            ks, vs = (t[pages].transpose(0, 1).reshape(hkv, -1, dim)[:, :ctx[i]] for t in (kc, vc))
            for at in range(0, lens[i], 512):
                rows = slice(start[i] + at, start[i] + min(at + 512, lens[i]))
                score = torch.einsum("thgd,hkd->hgtk", q[rows].view(-1, hkv, hq // hkv, dim), ks) / math.sqrt(dim)
                if lens[i] > 1:
                    score.masked_fill_(torch.arange(ctx[i], device="cuda") > pos[rows].cuda()[:, None], -math.inf)
                out[rows] = torch.einsum("hgtk,hkd->thgd", torch.softmax(score, -1), vs)
        x = x + out.reshape(m, -1) @ layer["o"]().T
        h = _norm(x, cfg.rms_eps)
        if layer["router"] is None:
            share = torch.ones(m, 1, dtype=torch.float64, device="cuda")
        else:
            best, which = (h @ layer["router"]().T).topk(cfg.n_experts_used, -1)
            share = torch.zeros(m, cfg.n_experts, dtype=torch.float64, device="cuda").scatter_(1, which, torch.softmax(best, -1))
        for e, (gate, up, down) in enumerate(layer["experts"]):
            rows = share[:, e].nonzero().flatten()
            if rows.numel():
                y = torch.nn.functional.silu(h[rows] @ gate().T) * (h[rows] @ up().T)
                x[rows] += share[rows, e, None] * (y @ down().T)
    last = torch.tensor(start).cuda() + torch.tensor(lens).cuda() - 1
    return {"logits": _norm(x[last], cfg.rms_eps) @ head().T, "k": kc, "v": vc}


def _splitmix(x):
    mask = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & mask
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & mask
    return x ^ (x >> 31)


def _exact_sample(case, seed):
    """The log-probability of the token that each row's draw falls on: the 256 to 1024 likeliest tokens, min-p, top-k, top-p."""
    state = _prepare_sample(case, seed)
    vocab, top_k = case["vocab"], case["top_k"] if 0 < case["top_k"] < case["vocab"] else case["vocab"]
    n = min(max(top_k, 256), 1024, vocab)
    scaled = state["logits"].double() / state["params"]["temperature"].double()[:, None]
    e = torch.exp(scaled.topk(n, -1).values - scaled.amax(-1, keepdim=True))
    total = torch.exp(scaled - scaled.amax(-1, keepdim=True)).sum(-1) if top_k >= vocab > n else e.sum(-1)
    got = []
    for row in range(case["rows"]):
        keep = min(top_k, int((e[row] >= case["min_p"] * e[row, 0]).sum()) if case["min_p"] > 0 else n)
        if case["top_p"] < 1:
            below = (torch.cumsum(e[row, :keep], 0) / total[row] < float(state["params"]["top_p"][row])).sum()
            keep = min(keep, int(below) + 1)
        counter, own = int(state["params"]["counters"][row]), int(state["params"]["seeds"][row])
        u = (_splitmix(own ^ _splitmix((counter + 0x51ED2701) & ((1 << 64) - 1))) >> 40) / (1 << 24)
        upto = torch.cumsum(e[row, :keep], 0)
        pick = min(int((upto <= u * upto[-1]).sum()), keep - 1)
        got.append(torch.log(e[row, pick] / total[row]))
    return {"tokens": None, "logprob": torch.stack(got)}


def _exact_project(case, seed):
    """Products of the quantised rows with the quantised weights."""
    got, rows, counts = {}, case["rows"], _expert_rows(case) if case["weights"] == "nvfp4" else None
    for name, w, x in _project_parts(case, seed):
        if counts is None:
            got[name] = _fp8_rows(x[0].double()) @ _fp8_values(w[0]).T
            continue
        q, scale = w
        out = torch.zeros(q.shape[0], (rows + 127) // 128 * 128, q.shape[1] // (2 if name == "gate_up" else 1), dtype=torch.float64, device="cuda")
        for j, n in enumerate(counts):
            if n:
                y = _fp4_rows(x[j, :n].double()) @ _fp4_values(q[j], scale).T
                if name == "gate_up":
                    v = y.view(n, -1, 2, 32)
                    y = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(n, -1)
                out[j, :n] = y
        got[name] = out
    return got
