"""What is measured when the speed of this package is judged: the hot operations of a serving step, called as the
layers call them.

A serving engine runs two kinds of steps: decode steps (one token per request, many times per second) and prompt steps
(chunks of prompts of up to 8192 tokens, alone or beside decoding requests).  The kinds below are the operations that
these steps spend their time in:

    gqa      paged attention of the dense and MoE models (bf16 or e4m3 cache)
    mla      latent attention of DeepSeek-shaped models
    delta    convolution and gated delta rule of the hybrid models (Qwen3-Next: one decay per head; Kimi-Linear: one per
             key channel), with the states it carries
    mlp      SwiGLU feed-forward, bf16 or block-scaled fp8
    moe      routed experts: routing, permutation, grouped GEMMs, weighted sum; bf16 or block-scaled fp8
    sample   top-k / top-p sampling from the logits

Sizes are those of the package's presets and of its benchmark (64 requests of 1024 + 128 tokens, prompt steps of 8192
tokens), ragged where requests differ.  A case says everything but the values; lengths follow from the case alone.
"""
import math
import random

import torch

BLOCK = 16
LATENT, ROPE = 512, 64
DIM, TAPS = 128, 4
FP8_MAX = 448.0

# (q heads, kv heads), head size 128: Llama-3.1-8B, Llama-3.1-70B, Qwen3-30B-A3B, Qwen3-0.6B
GQA_HEADS = ((32, 8), (64, 8), (32, 4), (16, 8))
# (k heads, v heads) of the delta rule: Qwen3-Next whole and on 2 and 4 ranks; Kimi-Linear whole and on 2 ranks
GDN_HEADS, KDA_HEADS = ((16, 32), (8, 16), (4, 8)), ((32, 32), (16, 16))
# (width, feed-forward): Llama-3.1-8B, Llama-3.1-70B on 8 ranks, Qwen3-0.6B
MLP_SIZES = ((4096, 14336), (8192, 3584), (1024, 3072))
# (width, expert feed-forward, experts here, experts per token): Qwen3-30B-A3B, DeepSeek-V3 on 8 ranks (32 of 256)
MOE_SIZES = ((2048, 768, 128, 8), (7168, 2048, 32, 1))
VOCABS = (32000, 128256, 151936)


def _attention(kind, name=None, *, decodes=0, context=0, chunks=0, chunk=0, prefix=0, **kw):
    c = dict(kind=kind, decodes=decodes, context=context, chunks=chunks, chunk=chunk, prefix=prefix, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user of a small deployment: nothing but latency
        _attention("gqa", "gqa_decode_1", decodes=1, context=700, q_heads=32, kv_heads=8, cache="bf16", ragged=False),
        # the decode step of the serving benchmark
        _attention("gqa", "gqa_decode_64", decodes=64, context=1100, q_heads=32, kv_heads=8, cache="bf16", ragged=False),
        # the prompt step of the serving benchmark
        _attention("gqa", "gqa_prefill_8x1024", chunks=8, chunk=1024, q_heads=32, kv_heads=8, cache="bf16", ragged=False),
        # chunks of long prompts beside decoding requests, e4m3 cache
        _attention("gqa", "gqa_mixed_e4m3", decodes=48, context=1500, chunks=3, chunk=677, prefix=1024, q_heads=32,
                   kv_heads=8, cache="e4m3", ragged=True),
        # DeepSeek-V3 with data-parallel attention (all heads on a GPU): decoding and prompts
        _attention("mla", "mla_decode_64", decodes=64, context=2048, heads=128, ragged=True),
        _attention("mla", "mla_prefill_4x2048", chunks=4, chunk=2048, heads=128, ragged=False),
        # Qwen3-Next: a prompt step, a decode step
        _attention("delta", "gdn_prefill_4x2048", chunks=4, chunk=2048, rule="head", k_heads=16, v_heads=32, ragged=False),
        _attention("delta", "gdn_decode_64", decodes=64, context=1500, rule="head", k_heads=16, v_heads=32, ragged=False),
        # Kimi-Linear: second chunks of ragged prompts
        _attention("delta", "kda_prefill_ragged", chunks=5, chunk=813, prefix=512, rule="channel", k_heads=32, v_heads=32,
                   ragged=True),
        # feed-forward of the decode step of the serving benchmark
        dict(name="mlp_decode_64", kind="mlp", tokens=64, width=4096, inter=14336, quant="bf16"),
        # experts of a prompt step
        dict(name="moe_prefill_4096", kind="moe", tokens=4096, width=2048, inter=768, experts=128, top_k=8, quant="bf16"),
        # sampling behind the decode step
        dict(name="sample_64", kind="sample", rows=64, vocab=128256, top_k=50, top_p=0.9, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _draw_lengths(rng, most):
    """Decoding requests, chunks, or both; at most ``most`` prompt tokens."""
    what = rng.choice(("decode", "prefill", "prefill", "mixed"))
    c = dict(decodes=0, context=0, chunks=0, chunk=0, prefix=0, ragged=rng.random() < 0.7)
    if what != "prefill":
        c.update(decodes=_log(rng, 1, 128), context=_log(rng, 64, 3000))
    if what != "decode":
        c["chunks"] = _log(rng, 1, 12)
        c["chunk"] = _log(rng, 17, min(2048, most // c["chunks"]))
        c["prefix"] = rng.choice((0, 0, _log(rng, 16, 2048)))
    return c


def draw(rng):
    kind = rng.choice(("gqa", "gqa", "mla", "mla", "delta", "delta", "mlp", "moe", "sample"))
    if kind == "gqa":
        hq, hkv = rng.choice(GQA_HEADS)
        return _attention(kind, q_heads=hq, kv_heads=hkv, cache=rng.choice(("bf16", "bf16", "e4m3")), **_draw_lengths(rng, 8192))
    if kind == "mla":
        while True:
            c = _attention(kind, heads=rng.choice((16, 32, 64, 128)), **_draw_lengths(rng, 8192))
            if work(c)["flops"] <= work(listed()[5])["flops"]:
                return c
    if kind == "delta":
        rule = rng.choice(("head", "channel"))
        hk, hv = rng.choice(GDN_HEADS if rule == "head" else KDA_HEADS)
        return _attention(kind, rule=rule, k_heads=hk, v_heads=hv, **_draw_lengths(rng, 8192))
    if kind == "mlp":
        width, inter = rng.choice(MLP_SIZES)
        return dict(kind=kind, tokens=_log(rng, 1, 4096), width=width, inter=inter, quant=rng.choice(("bf16", "fp8")))
    if kind == "moe":
        width, inter, experts, k = rng.choice(MOE_SIZES)
        return dict(kind=kind, tokens=_log(rng, 1, 8192), width=width, inter=inter, experts=experts, top_k=k,
                    quant=rng.choice(("bf16", "fp8")))
    top_k, top_p = rng.choice(((50, 0.9), (0, 0.95), (20, 1.0), (0, 1.0)))
    return dict(kind=kind, rows=_log(rng, 1, 256), vocab=rng.choice(VOCABS), top_k=top_k, top_p=top_p,
                dtype=rng.choice(("bf16", "fp32")))


# ---- lengths and work ----------------------------------------------------------------------------------------------
def _lengths(c):
    """[(tokens of the step, tokens with them)] per request, decoding requests first."""
    r = random.Random(repr(sorted((k, v) for k, v in c.items() if k in ("decodes", "context", "chunks", "chunk", "prefix"))))

    def vary(n):
        return n if not c["ragged"] else max(1, round(n * r.uniform(0.4, 1.0)))
    got = [(1, 1 + vary(c["context"])) for _ in range(c["decodes"])]
    for _ in range(c["chunks"]):
        n = vary(c["chunk"])
        got.append((n, n + (vary(c["prefix"]) if c["prefix"] else 0)))
    return got


def work(c):
    kind = c["kind"]
    if kind in ("gqa", "mla", "delta"):
        ls = _lengths(c)
        T = sum(n for n, _ in ls)
        keys = sum(s for _, s in ls)
        pairs = sum(n * s - n * (n - 1) // 2 for n, s in ls)
    if kind == "gqa":
        elem = 1 if c["cache"] == "e4m3" else 2
        return {"bytes": 2 * keys * c["kv_heads"] * DIM * elem + 4 * T * c["q_heads"] * DIM,
                "flops": 4 * pairs * c["q_heads"] * DIM}
    if kind == "mla":
        return {"bytes": 2 * keys * (LATENT + ROPE) + 2 * T * c["heads"] * (2 * LATENT + ROPE),
                "flops": 2 * pairs * c["heads"] * (2 * LATENT + ROPE)}
    if kind == "delta":
        hk, hv = c["k_heads"], c["v_heads"]
        channels = (2 * hk + hv) * DIM
        gates = hv * (DIM + 1 if c["rule"] == "channel" else 2)
        first = sum(1 for n, s in ls if n < s) + len(ls)            # states read (not at a start) and written
        return {"bytes": 2 * T * (channels + gates + hv * DIM) + first * (4 * hv * DIM * DIM + 2 * channels * (TAPS - 1)),
                "flops": T * (hv * 6 * DIM * DIM + 2 * channels * TAPS)}
    if kind == "mlp":
        t, n = c["tokens"], 3 * c["width"] * c["inter"]
        return {"bytes": n * (1 if c["quant"] == "fp8" else 2) + 4 * t * c["width"], "flops": 2 * t * n}
    if kind == "moe":
        t, n = c["tokens"], 3 * c["width"] * c["inter"]
        rows = t * c["top_k"]
        return {"bytes": min(c["experts"], rows) * n * (1 if c["quant"] == "fp8" else 2) + 4 * t * c["width"]
                + 4 * t * c["experts"], "flops": 2 * rows * n}
    return {"bytes": c["rows"] * c["vocab"] * (2 if c["dtype"] == "bf16" else 4) + 4 * c["rows"], "flops": 0}


def tolerance(c):
    """About four times the error against 64 bits (2e-3 to 3e-3 in bf16, 2e-2 where activations are rounded to e4m3 twice):
    bf16 outputs, bf16 probabilities or e4m3 activations in front of the second product; states are 32-bit behind
    bf16 convolutions.  Sampled tokens are whole numbers."""
    if c["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.01}
    if c["kind"] in ("mlp", "moe") and c["quant"] == "fp8":
        return {"rel": 3e-2}
    return {"rel": 1e-2}


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _meta(c, g):
    """The description of the step that the runner hands to every layer; blocks of a request lie anywhere in the pool."""
    from vllm_torchtpu_b200.runner.attn_metadata import AttentionMetadata
    ls = _lengths(c)
    R, T = len(ls), sum(n for n, _ in ls)
    need = [-(-s // BLOCK) for _, s in ls]
    blocks = sum(need) + 1
    ids = (torch.randperm(blocks - 1, generator=g, device="cuda") + 1).cpu().tolist()
    tables = torch.zeros(R, max(need), dtype=torch.int32)
    positions, slots, starts = [], [], [0]
    for r, (n, s) in enumerate(ls):
        mine = [ids.pop() for _ in range(need[r])]
        tables[r, :need[r]] = torch.tensor(mine, dtype=torch.int32)
        positions += range(s - n, s)
        slots += [mine[p // BLOCK] * BLOCK + p % BLOCK for p in range(s - n, s)]
        starts.append(starts[-1] + n)

    def dev(x):
        return torch.tensor(x, dtype=torch.int32, device="cuda")
    m = AttentionMetadata(
        dev(positions), dev(slots), tables.cuda(), dev([s for _, s in ls]), dev(starts), R, T, num_decode_reqs=c["decodes"],
        max_query_len=max(n for n, _ in ls), max_seq_len=max(s for _, s in ls), state_slots=dev(list(range(1, R + 1))),
        padded_num_reqs=R, padded_num_tokens=T, seq_lens_cpu=torch.tensor([s for _, s in ls]),
        query_start_loc_cpu=torch.tensor(starts))
    return m, blocks


def prepare(c, seed):
    g = _gen(seed)
    s = {"case": c}
    kind = c["kind"]
    if kind in ("gqa", "mla", "delta"):
        s["meta"], blocks = _meta(c, g)
        T, R = s["meta"].num_tokens, s["meta"].num_reqs
    if kind == "gqa":
        s["q"] = _normal(g, T, c["q_heads"], DIM)
        kv = _normal(g, blocks, 2, c["kv_heads"], BLOCK, DIM)
        s["cache"] = kv.to(torch.float8_e4m3fn) if c["cache"] == "e4m3" else kv
    elif kind == "mla":
        s["q"] = _normal(g, T, c["heads"], LATENT + ROPE)
        s["cache"] = _normal(g, blocks, BLOCK, LATENT + ROPE)
    elif kind == "delta":
        hk, hv = c["k_heads"], c["v_heads"]
        channels = (2 * hk + hv) * DIM
        channel = c["rule"] == "channel"
        s.update(mixed=_normal(g, T, channels), a=_normal(g, T, hv, DIM) if channel else _normal(g, T, hv),
                 b=_normal(g, T, hv), conv_w=_normal(g, channels, TAPS, std=0.2),
                 A_log=_normal(g, hv, std=0.5, dtype=torch.float32),
                 dt_bias=_normal(g, *((hv, DIM) if channel else (hv,)), std=0.5, dtype=torch.float32),
                 conv=_normal(g, R + 1, channels, TAPS - 1), rec=_normal(g, R + 1, hv, DIM, DIM, std=0.1, dtype=torch.float32))
    elif kind == "mlp":
        w, n = c["width"], c["inter"]
        s.update(x=_normal(g, c["tokens"], w), w13=_normal(g, 2 * n, w, std=0.02), w2=_normal(g, w, n, std=0.02))
        if c["quant"] == "fp8":
            from vllm_torchtpu_b200.quantization.fp8 import quantize_weight_block
            s["w13"], s["s13"] = quantize_weight_block(s["w13"])
            s["w2"], s["s2"] = quantize_weight_block(s["w2"])
    elif kind == "moe":
        w, n, e = c["width"], c["inter"], c["experts"]
        s.update(x=_normal(g, c["tokens"], w), logits=_normal(g, c["tokens"], e, dtype=torch.float32),
                 w13=_normal(g, e, 2 * n, w, std=0.02), w2=_normal(g, e, w, n, std=0.02))
        if c["quant"] == "fp8":
            from vllm_torchtpu_b200.quantization.fp8 import quantize_weight_block
            for k in ("13", "2"):
                both = [quantize_weight_block(t) for t in s.pop("w" + k)]
                s["w" + k], s["s" + k] = (torch.stack(t) for t in zip(*both))
    else:
        R = c["rows"]
        s.update(logits=_normal(g, R, c["vocab"], std=2.0, dtype=torch.bfloat16 if c["dtype"] == "bf16" else torch.float32),
                 temperature=torch.rand(R, generator=g, device="cuda") * 0.8 + 0.4,
                 top_k=torch.full((R,), c["top_k"], dtype=torch.int32, device="cuda"),
                 top_p=torch.full((R,), c["top_p"], device="cuda"), seed=int(seed),
                 step=torch.full((1,), 7, dtype=torch.int64, device="cuda"))
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(s):
    from vllm_torchtpu_b200 import ops
    c = s["case"]
    kind = c["kind"]
    if kind == "gqa":
        return ops.paged_attention(s["q"], s["cache"], s["meta"], DIM ** -0.5)
    if kind == "mla":
        return ops.mla_paged_attention(s["q"], s["cache"], s["meta"], (128 + ROPE) ** -0.5, LATENT)
    cu = ops.cuda_ops()
    if kind == "delta":
        hk, hv, meta = c["k_heads"], c["v_heads"], s["meta"]
        if c["rule"] == "head":
            o = cu.gdn_forward(s["mixed"], s["a"], s["b"], meta, s["conv"], s["rec"], s["conv_w"], s["A_log"], s["dt_bias"],
                               hk, hv, DIM, DIM)
        else:
            y = cu.short_conv(s["mixed"], meta, s["conv"], s["conv_w"])
            q, k, v = y.split([hk * DIM, hk * DIM, hv * DIM], dim=-1)
            T = y.shape[0]
            o = cu.kda_forward(q.reshape(T, hk, DIM), k.reshape(T, hk, DIM), v.reshape(T, hv, DIM), s["a"], s["b"], meta,
                               s["rec"], s["A_log"], s["dt_bias"])
        return {"o": o, "conv": s["conv"][1:], "rec": s["rec"][1:]}
    if kind == "mlp":
        if c["quant"] == "bf16":
            return ops.gemm(ops.gemm_gated(s["x"], s["w13"], "silu"), s["w2"])
        h = cu.fp8_block_gemm(s["x"], s["w13"], s["s13"])
        xq, xs = cu.quant_rows_1x128(h, c["inter"], swiglu=True)
        return cu.fp8_block_gemm_quantised(xq, xs, s["w2"], s["s2"], torch.empty_like(s["x"]))
    if kind == "moe":
        ids, w = ops.moe_route(s["logits"], c["top_k"])
        if c["quant"] == "bf16":
            return cu.moe_experts(s["x"], s["w13"], s["w2"], ids, w)
        return cu.moe_experts_fp8(s["x"], s["w13"], s["s13"], s["w2"], s["s2"], ids, w, 0)
    return cu.sample(s["logits"], s["temperature"], s["top_k"], s["top_p"], None, False, s["seed"], s["step"])


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------
def _softmax_rows(q, k, v, scale, s):
    """q [H, n, d], k and v [H or 1, s, .]; the n queries are the last of s positions."""
    n = q.shape[1]
    a = q @ k.transpose(1, 2) * scale
    hidden = torch.ones(n, s, dtype=torch.bool, device=q.device).triu(s - n + 1)
    return torch.softmax(a.masked_fill_(hidden, float("-inf")), -1) @ v


def _attention_exact(c, s):
    m, ls, outs, at = s["meta"], _lengths(c), [], 0
    for r, (n, total) in enumerate(ls):
        rows = s["cache"][m.block_tables[r, :-(-total // BLOCK)].long()].double()
        q = s["q"][at:at + n].double().transpose(0, 1)
        at += n
        if c["kind"] == "mla":
            kv = rows.reshape(1, -1, LATENT + ROPE)[:, :total]
            heads = [_softmax_rows(x, kv, kv[..., :LATENT], (128 + ROPE) ** -0.5, total) for x in q.split(16)]
        else:
            k, v = (rows[:, i].transpose(0, 1).reshape(c["kv_heads"], -1, DIM)[:, :total] for i in (0, 1))
            G = c["q_heads"] // c["kv_heads"]
            heads = [_softmax_rows(q[h * G:(h + 1) * G], k[h:h + 1], v[h:h + 1], DIM ** -0.5, total) for h in range(c["kv_heads"])]
        outs.append(torch.cat(heads).transpose(0, 1))
    return torch.cat(outs)


def _delta_exact(c, s):
    ls, hk, hv = _lengths(c), c["k_heads"], c["v_heads"]
    R, most = len(ls), max(n for n, _ in ls)
    T = sum(n for n, _ in ls)
    rep = hv // hk
    fresh = torch.tensor([n == t for n, t in ls], device="cuda")
    conv = s["conv"][1:].double().masked_fill(fresh[:, None, None], 0)
    S = s["rec"][1:].double().masked_fill(fresh[:, None, None, None], 0)
    starts = [0]
    for n, _ in ls:
        starts.append(starts[-1] + n)
    y = torch.empty_like(s["mixed"], dtype=torch.float64)
    for r, (n, _) in enumerate(ls):
        win = torch.cat([conv[r].t(), s["mixed"][starts[r]:starts[r + 1]].double()])
        w = s["conv_w"].double()
        y[starts[r]:starts[r + 1]] = torch.nn.functional.silu(sum(win[j:j + n] * w[:, j] for j in range(TAPS)))
        conv[r] = win[-(TAPS - 1):].t()
    q, k, v = y.split([hk * DIM, hk * DIM, hv * DIM], -1)
    q, k = (torch.nn.functional.normalize(x.reshape(T, hk, DIM), dim=-1).repeat_interleave(rep, 1) for x in (q, k))
    q, v = q * DIM ** -0.5, v.reshape(T, hv, DIM)
    z = torch.nn.functional.softplus(s["a"].double() + s["dt_bias"].double())
    A = s["A_log"].double().exp()
    decay = torch.exp(-(A[:, None] if z.ndim == 3 else A) * z)
    decay = decay if decay.ndim == 3 else decay[..., None]
    beta = s["b"].double().sigmoid()
    o = torch.empty(T, hv, DIM, dtype=torch.float64, device="cuda")
    # requests from the longest to the shortest: those that still have a token are the first ones
    order = sorted(range(R), key=lambda r: -ls[r][0])
    S = S[order].contiguous()
    at = torch.tensor([starts[r] for r in order], device="cuda")
    left = [ls[r][0] for r in order]
    live = R
    for t in range(most):
        while left[live - 1] <= t:
            live -= 1
        i = at[:live] + t
        St, kt = S[:live], k[i]
        St *= decay[i][..., None]
        u = (v[i] - (kt[:, :, None] @ St)[:, :, 0]) * beta[i][..., None]
        St += kt[..., None] * u[:, :, None]
        o[i] = (q[i][:, :, None] @ St)[:, :, 0]
    back = torch.empty_like(S)
    back[order] = S
    return {"o": o, "conv": conv, "rec": back}


def _quantised(x):
    """Rows in e4m3 with a scale per 128 values, expanded again."""
    g = x.float().reshape(x.shape[0], -1, 128)
    scale = g.abs().amax(-1, keepdim=True).clamp_min(1e-12) / FP8_MAX
    return ((g / scale).to(torch.float8_e4m3fn).double() * scale.double()).reshape(x.shape)


def _expanded(w, scale):
    return w.double() * scale.double().repeat_interleave(128, 0)[:w.shape[0]].repeat_interleave(128, 1)[:, :w.shape[1]]


def _feed_forward(c, x, w13, w2):
    """x rows already as the first product takes them; the second takes bf16 or e4m3 rows."""
    gate, up = (x @ w13.t()).chunk(2, -1)
    h = torch.nn.functional.silu(gate) * up
    return (_quantised(h) if c["quant"] == "fp8" else h) @ w2.t()


def exact(c, seed):
    if c["kind"] == "sample":
        return None
    s = prepare(c, seed)
    if c["kind"] == "delta":
        return _delta_exact(c, s)
    if c["kind"] in ("gqa", "mla"):
        return _attention_exact(c, s)
    fp8 = c["quant"] == "fp8"
    x = _quantised(s["x"]) if fp8 else s["x"].double()
    if c["kind"] == "mlp":
        ws = [_expanded(s["w" + k], s["s" + k]) if fp8 else s["w" + k].double() for k in ("13", "2")]
        return _feed_forward(c, x, *ws)
    p = torch.softmax(s["logits"].double(), -1)
    w, ids = p.topk(c["top_k"], -1)
    w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(c["experts"]):
        rows, which = (ids == e).nonzero(as_tuple=True)
        if rows.numel():
            ws = [_expanded(s["w" + k][e], s["s" + k][e]) if fp8 else s["w" + k][e].double() for k in ("13", "2")]
            out.index_add_(0, rows, _feed_forward(c, x[rows], *ws) * w[rows, which][:, None])
    return out
