"""Workloads of the engine on one GPU, at the sizes of its own model presets: decode steps, prefill, chunked prefill with
decode rows beside it, embeddings of short texts, mixtures of experts, fp8 weights, the hybrid Mamba-2 / latent-attention
decoder, and sampling.

The models have the presets' widths, heads and vocabularies and fewer layers (``num_hidden_layers_override``), so that several
engines fit one card; weights, caches and tokens are random. A step whose shape repeats from token to token (decode, and the
prefill of one prompt) is kept in a CUDA graph, as the engine keeps it with ``tokenweave_cuda_graphs``; steps that mix shapes
are launched kernel by kernel.
"""
import math
import zlib

import numpy as np
import torch
import torch.nn.functional as F

PAGE = 128
BF16 = torch.bfloat16


# ---- cases --------------------------------------------------------------------------------------------------------------
# kind "step": one engine step of ``model``: a run of ``chunk`` tokens behind ``chunk_context`` (0: no such run), then
#   ``batch`` single tokens whose contexts are spread over [low, high]; "prompts" > 1 cuts the run into that many prompts.
# kind "embed": ``LLM.encode`` of ``batch`` texts of [low, high] tokens. kind "moe": one routed layer. kind "sample": one draw.
def _step(name, model, layers, *, batch=0, low=0, high=0, chunk=0, chunk_context=0, prompts=1, quant="", graph=True):
    return dict(name=name, kind="step", model=model, layers=layers, batch=batch, low=low, high=high, chunk=chunk,
                chunk_context=chunk_context, prompts=prompts, quant=quant, graph=graph)


def listed():
    return [
        # one user, one token: the latency of interactive generation
        _step("decode one", "llama-3.1-8b", 8, batch=1, low=1111, high=1111),
        # a server's usual decode batch, requests at every stage of their lives
        _step("decode ragged", "llama-3.1-8b", 8, batch=48, low=60, high=5000),
        # offline generation: the largest batch the scheduler forms, wide model
        _step("decode wide", "llama-3.3-70b", 2, batch=200, low=700, high=2300),
        # decode on fp8 weights (activations quantised per token), per-head norms of queries and keys
        _step("decode fp8", "qwen3-32b", 3, batch=32, low=200, high=3000, quant="fp8"),
        # a batch of short texts to embed, through the offline API
        dict(name="embed texts", kind="embed", model="llama-3.1-8b", layers=8, batch=24, low=7, high=120),
        # the headline's prompt: 8192 tokens
        _step("prefill long", "llama-3.3-70b", 2, chunk=8192),
        # chunked prefill: a piece of a long prompt, and running requests that must not wait for it
        _step("prefill chunk", "qwen2.5-72b", 2, chunk=2011, chunk_context=13000, batch=37, low=150, high=4000, graph=False),
        # a routed layer under decode: every expert's weights are read for a handful of rows
        dict(name="experts decode", kind="moe", model="mixtral-8x22b", inter=16384, tokens=24, graph=True),
        # a routed layer under prefill, one rank's shard of eight
        dict(name="experts prefill", kind="moe", model="mixtral-8x22b", inter=2048, tokens=4003, graph=False),
        # hybrid decoder: prompts through the chunked recurrence and the expanded latent attention
        _step("hybrid prefill", "sidisun-8b", 4, chunk=6007, prompts=3, graph=False),
        # hybrid decoder: recurrent states and latent caches, token by token
        _step("hybrid decode", "sidisun-8b", 4, batch=100, low=300, high=3500),
        # temperature, top-k and top-p over a full vocabulary for a decode batch
        dict(name="sample", kind="sample", vocab=128256, batch=144),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


DENSE = [("llama-3.1-8b", 8), ("llama-3.3-70b", 2), ("qwen2.5-72b", 2), ("qwen3-32b", 3), ("phi-3-medium-4k", 6)]


def draw(rng):
    """One more case: batches of 1 to 256, contexts and prompts up to what the listed cases reach."""
    kind = rng.choice(["decode", "decode", "decode", "prefill", "chunk", "embed", "moe", "moe", "hybrid", "hybrid decode", "sample"])
    if kind == "decode":
        model, layers = rng.choice(DENSE)
        batch = _log_int(rng, 1, 256)
        high = _log_int(rng, 64, min(4000 if "phi" in model else 8000, 400000 // batch))
        case = _step("", model, layers, batch=batch, low=_log_int(rng, 16, high), high=high, quant=rng.choice(["", "", "fp8"]))
    elif kind == "prefill":
        model, layers = rng.choice(DENSE)
        case = _step("", model, layers, chunk=_log_int(rng, 20, 4000))
    elif kind == "chunk":
        model, layers = rng.choice(DENSE[:4])
        high = _log_int(rng, 64, 4000)
        case = _step("", model, layers, chunk=_log_int(rng, 64, 2048), chunk_context=_log_int(rng, 100, 12000),
                     batch=_log_int(rng, 1, 64), low=_log_int(rng, 16, high), high=high, graph=False)
    elif kind == "embed":
        high = _log_int(rng, 20, 500)
        case = dict(kind="embed", model="llama-3.1-8b", layers=8, batch=_log_int(rng, 1, 32), low=_log_int(rng, 5, high), high=high)
    elif kind == "moe":
        tokens = _log_int(rng, 1, 4096)
        case = dict(kind="moe", model="mixtral-8x22b", inter=rng.choice([2048, 4096, 16384]), tokens=tokens, graph=tokens <= 256)
    elif kind == "hybrid":
        chunk = _log_int(rng, 200, 8000)
        case = _step("", "sidisun-8b", 4, chunk=chunk, prompts=rng.randint(1, max(1, min(6, chunk // 100))), graph=False)
    elif kind == "hybrid decode":
        batch = _log_int(rng, 1, 128)
        high = _log_int(rng, 64, 4000)
        case = _step("", "sidisun-8b", 4, batch=batch, low=_log_int(rng, 16, high), high=high)
    else:
        case = dict(kind="sample", vocab=rng.choice([32064, 128256, 151936, 152064]), batch=_log_int(rng, 1, 256))
    case.pop("name", None)
    return case


# ---- inputs -------------------------------------------------------------------------------------------------------------
def _preset(name):
    from tokenweave_b200.config import resolve_model_config
    return resolve_model_config(name)


def _gen(seed, what):
    return torch.Generator(device="cuda").manual_seed((zlib.crc32(what.encode()) ^ (seed * 0x9E3779B1)) & 0x7FFFFFFF)


def _normal(seed, what, shape, std=1.0, dtype=BF16):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=_gen(seed, what))


def _uniform(seed, what, shape, lo, hi):
    return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=_gen(seed, what))


def _dense_tensors(cfg, layers, seed):
    """(checkpoint name, shape, standard deviation or None for norm weights) of a dense model."""
    H, D, I = cfg.hidden_size, cfg.head_dim, cfg.intermediate_size
    q, kv = cfg.num_q_heads * D, cfg.num_kv_heads * D
    yield "model.embed_tokens.weight", (cfg.vocab_size, H), 0.5
    yield "model.norm.weight", (H,), None
    yield "lm_head.weight", (cfg.vocab_size, H), 0.02
    for i in range(layers):
        p = f"model.layers.{i}."
        yield p + "input_layernorm.weight", (H,), None
        yield p + "post_attention_layernorm.weight", (H,), None
        for n, rows, cols in (("q_proj", q, H), ("k_proj", kv, H), ("v_proj", kv, H), ("o_proj", H, q)):
            yield p + f"self_attn.{n}.weight", (rows, cols), cols ** -0.5
        if cfg.qkv_bias:
            for n, rows in (("q_proj", q), ("k_proj", kv), ("v_proj", kv)):
                yield p + f"self_attn.{n}.bias", (rows,), 0.3
        if cfg.qk_norm:
            yield p + "self_attn.q_norm.weight", (D,), None
            yield p + "self_attn.k_norm.weight", (D,), None
        for n, rows, cols in (("gate_proj", I, H), ("up_proj", I, H), ("down_proj", H, I)):
            yield p + f"mlp.{n}.weight", (rows, cols), cols ** -0.5


def _hybrid_tensors(cfg, layers, seed):
    H = cfg.hidden_size
    yield "embed", (cfg.vocab_size, H), 0.5
    yield "final.norm", (H,), None
    yield "head", (cfg.vocab_size, H), 0.02
    for i in range(layers):
        spec, p = cfg.layers[i], f"l{i}.mix."
        m = spec["mixer"]
        yield f"l{i}.norm1", (H,), None
        if spec["type"] == "mamba2":
            inner, gn = m["heads"] * m["vdim"], m["groups"] * m["state"]
            yield p + "in", (2 * inner + 2 * gn + m["heads"], H), H ** -0.5
            yield p + "conv", (inner + 2 * gn, m["conv"]), m["conv"] ** -0.5
            yield p + "conv.b", (inner + 2 * gn,), 0.1
            for n in ("dt_bias", "A_log", "D"):
                yield p + n, (m["heads"],), 1.0
            yield p + "norm", (inner,), None
            yield p + "o", (H, inner), inner ** -0.5
        else:
            h, d, r, v, k, q = (m[n] for n in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
            for n, rows, cols in (("dq", q, H), ("uq", h * (d + r), q), ("dkv", k + r, H), ("uk", h * d, k), ("uv", h * v, k),
                                  ("g", h * v, H), ("o", H, h * v)):
                yield p + n, (rows, cols), cols ** -0.5
            yield p + "dq.norm", (q,), None
            yield p + "dkv.norm", (k,), None
        ff = spec["mlp"]["ff"]
        yield f"l{i}.norm2", (H,), None
        yield f"l{i}.mlp.up", (ff, H), H ** -0.5
        yield f"l{i}.mlp.down", (H, ff), ff ** -0.5
        yield f"l{i}.mlp.act", (4,), 0.4


def _tensor(name, shape, std, seed):
    if std is None:
        return 1 + _normal(seed, name, shape, 0.2)
    if name.endswith(".dt_bias"):           # step sizes of 0.001 to 0.1
        return _uniform(seed, name, shape, -6.9, -2.3).to(BF16)
    if name.endswith(".A_log"):
        return _uniform(seed, name, shape, 0.0, 2.7).to(BF16)
    return _normal(seed, name, shape, std)


def _tensors_of(cfg):
    return _hybrid_tensors if cfg.layers else _dense_tensors


def _spread(n, low, high):
    """n lengths over [low, high], neither sorted nor multiples of anything."""
    if n <= 1:
        return [high] * n
    return [low + (high - low) * ((i * 37 + 11) % n) // (n - 1) if n % 37 else low + (high - low) * i // (n - 1) for i in range(n)]


def _layout(case):
    """(tokens, keys in the cache before them) of every sequence of a step."""
    q, ctx = [], []
    if case["chunk"]:
        n, p = case["chunk"], case["prompts"]
        cuts = [0] + [n * (2 * i + 1) // (2 * p) for i in range(1, p)] + [n]
        q += [b - a for a, b in zip(cuts, cuts[1:])]
        ctx += [case["chunk_context"]] * p
    q += [1] * case["batch"]
    ctx += _spread(case["batch"], case["low"], case["high"])
    return q, ctx


def _tables(q, ctx, seed):
    """Pages of every sequence, scattered over the pool (page 0 stays unused), and the pool's size."""
    need = [(a + b + PAGE - 1) // PAGE for a, b in zip(q, ctx)]
    order = (np.random.RandomState(seed & 0x7FFFFFFF).permutation(sum(need)) + 1).tolist()
    tables, at = [], 0
    for n in need:
        tables.append(order[at:at + n])
        at += n
    return tables, sum(need) + 1


def _ids(seed, n, vocab):
    return torch.randint(0, vocab, (n,), dtype=torch.int32, device="cuda", generator=_gen(seed, "tokens"))


def _cache(seed, name, shape, dtype=BF16, std=1.0):
    return _normal(seed, name, shape, std, dtype)


def _engine(case, seed, *, tokens, longest, blocks, seqs):
    from tokenweave_b200 import LLM
    llm = LLM(case["model"], load_format="dummy", skip_tokenizer_init=True, num_hidden_layers_override=case["layers"],
              max_num_batched_tokens=tokens, max_model_len=longest, max_num_seqs=seqs, block_size=PAGE,
              num_gpu_blocks_override=blocks, enable_prefix_caching=False, seed=0)
    model = llm.llm_engine.core.executor.worker.runner.model
    cfg = _preset(case["model"])
    model.load_weights((n, _tensor(n, s, d, seed)) for n, s, d in _tensors_of(cfg)(cfg, case["layers"], seed))
    if case.get("quant"):
        from tokenweave_b200.models.loader import quantize_linears_fp8_
        quantize_linears_fp8_(model, case["quant"])
    return llm, model


def _captured(fn):
    """``fn`` in a CUDA graph, and the tensors it writes."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


def _prepare_step(case, seed):
    from tokenweave_b200.layers.attention import build_attention_metadata
    from tokenweave_b200.models.decoder import StepInput
    q, ctx = _layout(case)
    tables, blocks = _tables(q, ctx, seed)
    T, kv = sum(q), [a + b for a, b in zip(q, ctx)]
    llm, model = _engine(case, seed, tokens=max(T, 64), longest=max(kv) + 64, blocks=blocks, seqs=len(q))
    runner = llm.llm_engine.core.executor.worker.runner
    for i, t in enumerate(model.cache_tensors()):
        if any(ctx):
            t.copy_(_cache(seed, f"cache {i}", t.shape, t.dtype, 0.2 if t.dtype == torch.float32 else 1.0))
    pos = np.concatenate([np.arange(c, c + n) for n, c in zip(q, ctx)])
    slots = np.concatenate([np.asarray(t)[np.arange(c, c + n) // PAGE] * PAGE + np.arange(c, c + n) % PAGE
                            for n, c, t in zip(q, ctx, tables)])
    table = np.zeros((len(q), max(map(len, tables))), dtype=np.int32)
    for row, t in zip(table, tables):
        row[:len(t)] = t
    plan, extra, host = (model.plan_step(q, kv, list(range(len(q))), [-1] * len(q)) if hasattr(model, "plan_step")
                         else (None, None, None))
    meta = build_attention_metadata(q, kv, pos, slots, table, torch.device("cuda", torch.cuda.current_device()), plan=plan,
                                    extra=extra, extra_cpu=host)
    step = StepInput(_ids(seed, T, _preset(case["model"]).vocab_size), runner.planner.plan(T), meta=meta)
    rows = torch.tensor(np.cumsum(q) - 1, device="cuda")
    kept = model.cache_tensors()
    written = kept[-3:] if model.cfg.layers else kept[-2:]      # the last layers' caches and states

    def one():
        hidden = model(step)
        return {"hidden": hidden, "logits": model.compute_logits(hidden.index_select(0, rows)), "kept": written}
    state = {"llm": llm, "fn": one}
    if case["graph"]:
        state["graph"], state["out"] = _captured(one)
        if any(ctx):                        # recurrent states have moved on while the step was recorded
            for i, t in enumerate(kept):
                t.copy_(_cache(seed, f"cache {i}", t.shape, t.dtype, 0.2 if t.dtype == torch.float32 else 1.0))
    return state


def _embed_lengths(case):
    return _spread(case["batch"], case["low"], case["high"])


def _prepare_embed(case, seed):
    n = _embed_lengths(case)
    llm, _ = _engine(case, seed, tokens=max(sum(n), 64), longest=max(n) + 64, blocks=sum((x + PAGE) // PAGE + 1 for x in n) + 1,
                     seqs=len(n))
    ids = _ids(seed, sum(n), _preset(case["model"]).vocab_size).tolist()
    cuts = np.cumsum([0] + n).tolist()
    return {"llm": llm, "texts": [ids[a:b] for a, b in zip(cuts, cuts[1:])]}


def _moe_tensors(case, seed):
    cfg = _preset(case["model"])
    E, H, I = cfg.num_experts, cfg.hidden_size, case["inter"]
    return (_normal(seed, "gate", (E, H), H ** -0.5), _normal(seed, "w13", (E, 2 * I, H), H ** -0.5),
            _normal(seed, "w2", (E, H, I), I ** -0.5), _normal(seed, "x", (case["tokens"], H)))


def _prepare_moe(case, seed):
    from tokenweave_b200.layers.moe import FusedMoE
    cfg = _preset(case["model"])
    layer = FusedMoE(cfg.num_experts, cfg.num_experts_per_tok, cfg.hidden_size, case["inter"], dtype=BF16, device="cuda")
    gate, w13, w2, x = _moe_tensors(case, seed)
    for p, t in ((layer.gate, gate), (layer.w13, w13), (layer.w2, w2)):
        p.data = t
    out = torch.empty_like(x)
    state = {"fn": lambda: layer(x, out=out)}
    if case["graph"]:
        state["graph"], state["out"] = _captured(state["fn"])
    return state


def _prepare_sample(case, seed):
    from tokenweave_b200 import ops
    B, V = case["batch"], case["vocab"]
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    t = r.uniform(0.5, 1.2, B)
    k = np.where(r.rand(B) < 0.5, r.randint(5, 100, B), 0)
    p = np.where(r.rand(B) < 0.6, r.uniform(0.8, 0.98, B), 1.0)
    m = np.where(r.rand(B) < 0.1, 0.05, 0.0)
    packed = ops.pack_sample_params(t, k, p, m, r.randint(0, 1 << 30, B)).cuda()
    return {"logits": _normal(seed, "logits", (B, V), 2.5, torch.float32), "packed": packed}


def prepare(case, seed):
    torch.cuda.set_device(0)
    return {"step": _prepare_step, "embed": _prepare_embed, "moe": _prepare_moe, "sample": _prepare_sample}[case["kind"]](case, seed)


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    if "fn" in state:
        return state["fn"]()
    if "texts" in state:
        return [o.data for o in state["llm"].encode(state["texts"])]
    from tokenweave_b200 import ops
    return ops.sample(state["logits"], state["packed"])


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def _pairs(q, ctx):
    return sum(n * c + n * (n + 1) // 2 for n, c in zip(q, ctx))


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4 * case["batch"] * case["vocab"], "flops": 5 * case["batch"] * case["vocab"]}
    cfg = _preset(case["model"])
    H = cfg.hidden_size
    if case["kind"] == "moe":
        T, E, k, I = case["tokens"], cfg.num_experts, cfg.num_experts_per_tok, case["inter"]
        used = E * (1 - (1 - k / E) ** T)
        return {"bytes": 2 * (used * 3 * I * H + E * H + 2 * T * H), "flops": 2 * T * k * 3 * I * H}
    if case["kind"] == "embed":
        q = _embed_lengths(case)
        ctx = [0] * len(q)
    else:
        q, ctx = _layout(case)
    T, B, V = sum(q), len(q), cfg.vocab_size
    flops = 2 * B * V * H
    moved = 2 * V * H + 2 * T * H + 4 * B * V + 2 * T * H
    size = 1 if case.get("quant") else 2
    for i in range(case["layers"]):
        if cfg.layers:
            spec = cfg.layers[i]
            m = spec["mixer"]
            w = 2 * H * spec["mlp"]["ff"]
            if spec["type"] == "mamba2":
                inner, gn = m["heads"] * m["vdim"], m["groups"] * m["state"]
                w += H * (2 * inner + 2 * gn + m["heads"]) + inner * H
                moved += B * 4 * inner * m["state"] * (2 if any(ctx) else 1)
                flops += 6 * T * inner * m["state"]
            else:
                h, d, r, v, k, qr = (m[n] for n in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
                w += H * qr + qr * h * (d + r) + H * (k + r) + k * h * (d + v) + 2 * H * h * v
                moved += 2 * (k + r) * (sum(ctx) + T)
                flops += 2 * h * (d + r + v) * _pairs(q, ctx)
        else:
            D, hq, hkv = cfg.head_dim, cfg.num_q_heads, cfg.num_kv_heads
            w = H * D * (2 * hq + 2 * hkv) + 3 * H * cfg.intermediate_size
            moved += 4 * hkv * D * (sum(ctx) + T)
            flops += 4 * hq * D * _pairs(q, ctx)
        moved += size * w
        flops += 2 * T * w
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["kind"] == "moe":               # 0.003 off the same in 64 bits
        return {"rel": 0.01, "max": 0.1}
    # bf16 activations between kernels: 0.007 off the same in 64 bits behind two layers, 0.015 behind eight; behind fp8 a last
    # bit of an activation may turn over its rounding to eight bits (0.07 off)
    return {"rel": 0.03 if case.get("quant") or case["layers"] > 4 else 0.02, "max": 0.5}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------
def _d(t):
    return t.to(torch.float64)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _fp8(x):
    """x rounded to e4m3 with one scale per row, as values."""
    s = (x.abs().amax(-1, keepdim=True) / 448.0).clamp_min(1e-10)
    return _d((x / s).float().clamp(-448, 448).to(torch.float8_e4m3fn)) * s


def _angles(cfg, rot, theta, pos):
    f = theta ** (-torch.arange(0, rot, 2, dtype=torch.float64, device="cuda") / rot)
    s = cfg.rope_scaling
    if s:                                   # Llama 3: long wavelengths stretched, a blend between
        turns = s["original_max_position_embeddings"] * f / (2 * math.pi)
        keep = ((turns - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0, 1)
        f = f / s["factor"] * (1 - keep) + f * keep
    return pos.double()[:, None] * f


def _rotate(x, ang):
    """x [T, heads, dims], pairs of halves."""
    u, v = x.chunk(2, -1)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(q, k, v, first, scale):
    """q [n, h, d], k [m, g, d], v [m, g, e]; query i sees the keys up to first + i."""
    n, h, g = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(n, h, v.shape[-1], dtype=torch.float64, device="cuda")
    keys = torch.arange(k.shape[0], device="cuda")
    step = max(1, int(3e8) // (h * k.shape[0]))
    for a in range(0, n, step):
        b = min(n, a + step)
        m = first + b
        qq = q[a:b].view(b - a, g, h // g, -1).permute(1, 2, 0, 3).reshape(g, -1, q.shape[-1])
        s = torch.bmm(qq, k[:m].permute(1, 2, 0)).view(g, h // g, b - a, m) * scale
        s.masked_fill_(keys[:m] > first + torch.arange(a, b, device="cuda")[:, None], -math.inf)
        o = torch.bmm(torch.softmax(s, -1).view(g, -1, m), v[:m].transpose(0, 1))
        out[a:b] = o.view(g, h // g, b - a, -1).permute(2, 0, 1, 3).reshape(b - a, h, -1)
    return out


def _exact_dense(case, seed, q, ctx, tables, blocks):
    cfg = _preset(case["model"])
    H, D, hq, hkv, eps = cfg.hidden_size, cfg.head_dim, cfg.num_q_heads, cfg.num_kv_heads, cfg.rms_norm_eps
    made = {n: (n, s, d, seed) for n, s, d in _dense_tensors(cfg, case["layers"], seed)}
    w = lambda n: _d(_tensor(*made[n]))
    fp8 = bool(case.get("quant"))

    def linear(x, name):
        if fp8:
            return _fp8(x) @ _fp8(w(name)).T
        return x @ w(name).T
    pos = torch.cat([torch.arange(c, c + n, device="cuda") for n, c in zip(q, ctx)])
    cuts = np.cumsum([0] + q).tolist()
    slots = torch.cat([torch.tensor(t, device="cuda")[torch.arange(c, c + n, device="cuda") // PAGE] * PAGE
                       + torch.arange(c, c + n, device="cuda") % PAGE for n, c, t in zip(q, ctx, tables)])
    ang = _angles(cfg, D, cfg.rope_theta, pos)
    x = w("model.embed_tokens.weight")[_ids(seed, sum(q), cfg.vocab_size).long()]
    kept = None
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w(p + "input_layernorm.weight")
        parts = []
        for n, heads in (("q", hq), ("k", hkv), ("v", hkv)):
            y = linear(h, p + f"self_attn.{n}_proj.weight")
            if cfg.qkv_bias:
                y = y + w(p + f"self_attn.{n}_proj.bias")
            y = y.view(-1, heads, D)
            if cfg.qk_norm and n != "v":
                y = _rms(y, eps) * w(p + f"self_attn.{n}_norm.weight")
            parts.append(y if n == "v" else _rotate(y, ang))
        shape = (blocks, PAGE, hkv, D)
        caches = [_d(_cache(seed, f"cache {2 * i + j}", shape)) if any(ctx) else torch.zeros(shape, dtype=torch.float64, device="cuda")
                  for j in (0, 1)]
        for c, y in zip(caches, parts[1:]):
            c.view(-1, hkv, D)[slots] = y
        att = torch.empty(sum(q), hq, D, dtype=torch.float64, device="cuda")
        for b, (n, c) in enumerate(zip(q, ctx)):
            t = torch.tensor(tables[b], device="cuda")
            kk, vv = (x_[t].reshape(-1, hkv, D)[:n + c] for x_ in caches)
            att[cuts[b]:cuts[b + 1]] = _attend(parts[0][cuts[b]:cuts[b + 1]], kk, vv, c, D ** -0.5)
        x = x + linear(att.view(-1, hq * D), p + "self_attn.o_proj.weight")
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight")
        act = F.silu(linear(h, p + "mlp.gate_proj.weight")) * linear(h, p + "mlp.up_proj.weight")
        x = x + linear(act, p + "mlp.down_proj.weight")
        kept = caches
    hidden = _rms(x, eps) * w("model.norm.weight")
    logits = hidden[torch.tensor(cuts[1:], device="cuda") - 1] @ w("lm_head.weight").T
    return {"hidden": hidden, "logits": logits, "kept": kept}


def _exact_hybrid(case, seed, q, ctx, tables, blocks):
    cfg = _preset(case["model"])
    eps, T = cfg.rms_norm_eps, sum(q)
    made = {n: (n, s, d, seed) for n, s, d in _hybrid_tensors(cfg, case["layers"], seed)}
    w = lambda n: _d(_tensor(*made[n]))
    cuts = np.cumsum([0] + q).tolist()
    pos = torch.cat([torch.arange(c, c + n, device="cuda") for n, c in zip(q, ctx)])
    x = w("embed")[_ids(seed, T, cfg.vocab_size).long()]
    kept = []

    def start(shape, dtype):
        if any(ctx):
            return _d(_cache(seed, f"cache {len(kept)}", shape, dtype, 0.2 if dtype == torch.float32 else 1.0))
        return torch.zeros(shape, dtype=torch.float64, device="cuda")

    def mamba2(h, p, m):
        nh, P, N, G, taps = (m[n] for n in ("heads", "vdim", "state", "groups", "conv"))
        inner, ch = nh * P, nh * P + 2 * G * N
        z, xbc, dt = (h @ w(p + "in").T).split([inner, ch, nh], -1)
        S = start((len(q), nh, P, N), torch.float32)
        kept.append(S)
        tail = start((len(q), taps - 1, ch), BF16)
        kept.append(tail)
        dt = F.softplus(dt + w(p + "dt_bias"))
        decay = torch.exp(-torch.exp(w(p + "A_log")) * dt)
        cw, cb, skip = w(p + "conv"), w(p + "conv.b"), w(p + "D")
        y = torch.empty(T, nh, P, dtype=torch.float64, device="cuda")
        # all sequences at once, one place of every sequence at a time
        longest, n = max(q), torch.tensor(q, device="cuda")
        begin = torch.tensor(cuts[:-1], device="cuda")
        for t in range(longest):
            on = torch.nonzero(n > t).squeeze(1) if min(q) <= t else slice(None)
            row = begin[on] + t
            now = xbc[row]
            act = F.silu((tail[on] * cw.T[:-1]).sum(1) + now * cw[:, -1] + cb)
            tail[on] = torch.cat([tail[on][:, 1:], now[:, None]], 1)
            xx, Bm, Cm = act.split([inner, G * N, G * N], -1)
            xx = xx.view(-1, nh, P)
            Bm, Cm = (v.view(-1, G, N).repeat_interleave(nh // G, 1) for v in (Bm, Cm))
            new = S[on] * decay[row][..., None, None] + (xx * dt[row][..., None])[..., None] * Bm[:, :, None]
            S[on] = new
            y[row] = torch.matmul(new, Cm[..., None]).squeeze(-1) + skip[:, None] * xx
        y = y.view(T, inner) * F.silu(z)
        g = m["norm_groups"]
        return (_rms(y.view(T, g, -1), eps).view(T, inner) * w(p + "norm")) @ w(p + "o").T

    def latent(h, p, m):
        nh, d, r, v, k = (m[n] for n in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
        qq = ((_rms(h @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T).view(T, nh, d + r)
        ang = _angles(cfg, r, m["rot"]["base"], pos)
        qq = torch.cat([qq[..., :d], _rotate(qq[..., d:], ang)], -1)
        down = h @ w(p + "dkv").T
        rows = torch.cat([_rms(down[:, :k], eps) * w(p + "dkv.norm"), _rotate(down[:, None, k:], ang)[:, 0]], -1)
        cache = start((blocks, PAGE, k + r), BF16)
        kept.append(cache)
        uk, uv = w(p + "uk"), w(p + "uv")
        out = torch.empty(T, nh, v, dtype=torch.float64, device="cuda")
        for b, (n, c) in enumerate(zip(q, ctx)):
            t = torch.tensor(tables[b], device="cuda")
            at = torch.arange(c, c + n, device="cuda")
            cache.view(-1, k + r)[t[at // PAGE] * PAGE + at % PAGE] = rows[cuts[b]:cuts[b + 1]]
            lat = cache[t].reshape(-1, k + r)[:n + c]
            keys = torch.cat([(lat[:, :k] @ uk.T).view(-1, nh, d), lat[:, None, k:].expand(-1, nh, r)], -1)
            out[cuts[b]:cuts[b + 1]] = _attend(qq[cuts[b]:cuts[b + 1]], keys, (lat[:, :k] @ uv.T).view(-1, nh, v), c, m["scale"])
        return (out.view(T, -1) * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T

    for i in range(case["layers"]):
        spec, p = cfg.layers[i], f"l{i}."
        mixed = (mamba2 if spec["type"] == "mamba2" else latent)(x, p + "mix.", spec["mixer"])
        x = x + _rms(mixed, eps) * w(p + "norm1")
        z = x @ w(p + "mlp.up").T
        a, b, c, e = w(p + "mlp.act")
        act = a * _rms(z, eps) + b * _rms(z * z, eps) + c * _rms(z * z * z, eps) + e
        x = x + _rms(act @ w(p + "mlp.down").T, eps) * w(p + "norm2")
    hidden = _rms(x, eps) * w("final.norm")
    logits = hidden[torch.tensor(cuts[1:], device="cuda") - 1] @ w("head").T * cfg.logit_scale
    return {"hidden": hidden, "logits": logits, "kept": kept[-3:]}


def exact(case, seed):
    torch.cuda.set_device(0)
    if case["kind"] == "sample":
        return None
    if case["kind"] == "moe":
        gate, w13, w2, x = (_d(t) for t in _moe_tensors(case, seed))
        top, ids = torch.softmax(x @ gate.T, -1).topk(_preset(case["model"]).num_experts_per_tok, -1)
        top = top / top.sum(-1, keepdim=True)
        out = torch.zeros_like(x)
        for e in range(gate.shape[0]):
            row, place = torch.nonzero(ids == e, as_tuple=True)
            g, u = (x[row] @ w13[e].T).chunk(2, -1)
            out.index_add_(0, row, ((F.silu(g) * u) @ w2[e].T) * top[row, place, None])
        return out
    if case["kind"] == "embed":
        n = _embed_lengths(case)
        tables, blocks = _tables(n, [0] * len(n), seed)
        hidden = _exact_dense(case, seed, n, [0] * len(n), tables, blocks)["hidden"]
        return [hidden[i - 1].cpu() for i in np.cumsum(n).tolist()]
    q, ctx = _layout(case)
    tables, blocks = _tables(q, ctx, seed)
    return (_exact_hybrid if _preset(case["model"]).layers else _exact_dense)(case, seed, q, ctx, tables, blocks)
