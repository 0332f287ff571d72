"""CUDA kernels vs the plain-PyTorch fp32 statements of the same ops."""
import math

import pytest
import torch

from vllm_torchtpu_b200.ops import reference as ref
from vllm_torchtpu_b200.runner.attn_metadata import AttentionMetadata

pytestmark = pytest.mark.gpu
DEV = "cuda"


def cu():
    from vllm_torchtpu_b200.ops import cuda
    return cuda


def _close(a, b, rtol=2e-2, atol=2e-2):
    torch.testing.assert_close(a.float(), b.float(), rtol=rtol, atol=atol)


@pytest.mark.parametrize("T,H", [(1, 256), (7, 4096), (64, 8192), (33, 1000 * 8)])
def test_rms_norm(T, H):
    g = torch.Generator(device=DEV).manual_seed(0)
    x = torch.randn(T, H, device=DEV, generator=g).bfloat16()
    w = (1 + 0.1 * torch.randn(H, device=DEV, generator=g)).bfloat16()
    _close(cu().rms_norm(x, w, 1e-5), ref.rms_norm(x, w, 1e-5), 1e-2, 1e-2)
    r = torch.randn(T, H, device=DEV, generator=g).bfloat16()
    want_y, want_r = ref.fused_add_rms_norm(x, r.clone(), w, 1e-5)
    got_y, got_r = cu().fused_add_rms_norm(x, r, w, 1e-5)
    assert torch.equal(got_r, want_r)
    _close(got_y, want_y, 1e-2, 1e-2)


def test_silu_and_mul():
    x = torch.randn(77, 2 * 1536, device=DEV).bfloat16()
    _close(cu().silu_and_mul(x), ref.silu_and_mul(x), 1e-2, 1e-2)


def test_embedding_and_rows():
    table = torch.randn(1000, 512, device=DEV).bfloat16()
    ids = torch.randint(0, 1000, (50,), device=DEV, dtype=torch.int32)
    src = torch.full((50,), -1, device=DEV, dtype=torch.int32)
    last = torch.randint(0, 1000, (8,), device=DEV, dtype=torch.int32)
    src[3], src[10] = 2, 7
    want_ids = ids.clone()
    want_ids[3], want_ids[10] = last[2], last[7]
    assert torch.equal(cu().embedding(ids, table, src, last), table[want_ids.long()])
    idx = torch.tensor([4, 0, 49], device=DEV, dtype=torch.int32)
    h, r = cu().gather_rows(table[:50].contiguous(), table[50:100].contiguous(), idx)
    assert torch.equal(h, table[:50][idx.long()]) and torch.equal(r, table[50:100][idx.long()])
    toks = torch.tensor([11, 22, 33], device=DEV, dtype=torch.int32)
    slots = torch.tensor([5, -1, 0], device=DEV, dtype=torch.int32)
    cu().scatter_tokens(toks, slots, last)
    assert last[5] == 11 and last[0] == 33


@pytest.mark.parametrize("D,interleaved,qk_norm", [(128, False, False), (128, False, True), (64, True, False)])
def test_rope_and_cache(D, interleaved, qk_norm):
    T, Hq, Hkv, bs, nb = 37, 8, 2, 16, 12
    g = torch.Generator(device=DEV).manual_seed(1)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, generator=g).bfloat16()
    pos = torch.randint(0, 5000, (T,), device=DEV, dtype=torch.int32)
    inv = ref.rope_inv_freq(D, 500000.0).to(DEV)
    slots = torch.randperm(nb * bs, device=DEV)[:T].to(torch.int32)
    slots[5] = -1
    qn = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16() if qk_norm else None
    kn = (1 + 0.1 * torch.randn(D, device=DEV)).bfloat16() if qk_norm else None
    c1 = torch.zeros(nb, 2, Hkv, bs, D, device=DEV, dtype=torch.bfloat16)
    c2 = c1.clone()
    q1 = cu().rope_and_cache(qkv, pos, inv, c1, slots, Hq, Hkv, D, interleaved, qn, kn, 1e-6)
    q2 = ref.rope_and_cache(qkv, pos, inv, c2, slots, Hq, Hkv, D, interleaved, qn, kn, 1e-6)
    _close(q1, q2, 2e-2, 2e-2)
    _close(c1, c2, 2e-2, 2e-2)


def _attn_case(q_lens, ctx_lens, Hq, Hkv, D, bs=16, window=None, softcap=None, sinks=False, num_decode=0,
               kv_fp8=False, scales=(0.02, 0.03)):
    g = torch.Generator(device=DEV).manual_seed(2)
    R = len(q_lens)
    seq = [q + c for q, c in zip(q_lens, ctx_lens)]
    maxb = max(-(-s // bs) for s in seq) + 1
    nb = sum(-(-s // bs) for s in seq) + 2
    cache = (torch.randn(nb, 2, Hkv, bs, D, device=DEV, generator=g) * 0.5).bfloat16()
    k_scale, v_scale = 1.0, 1.0
    if kv_fp8:
        # e4m3 cache with per-tensor scales: the oracle dequantises the same bytes in fp32
        k_scale, v_scale = scales
        cache = torch.stack([cache[:, 0].float() / k_scale, cache[:, 1].float() / v_scale],
                            1).to(torch.float8_e4m3fn)
    perm = (torch.randperm(nb - 1, device=DEV) + 1).to(torch.int32)
    bt = torch.zeros(R, maxb, dtype=torch.int32, device=DEV)
    off = 0
    for r, s in enumerate(seq):
        n = -(-s // bs)
        bt[r, :n] = perm[off:off + n]
        off += n
    T = sum(q_lens)
    q = torch.randn(T, Hq, D, device=DEV, generator=g).bfloat16()
    qsl = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    sl = torch.tensor(seq, dtype=torch.int32, device=DEV)
    meta = AttentionMetadata(positions=None, slot_mapping=None, block_tables=bt, seq_lens=sl,
                             query_start_loc=qsl, num_reqs=R, num_tokens=T, num_decode_reqs=num_decode,
                             max_query_len=max(q_lens), max_seq_len=max(seq),
                             padded_num_reqs=R, padded_num_tokens=T,
                             query_start_loc_cpu=qsl.cpu().long(), seq_lens_cpu=sl.cpu().long())
    sk = torch.randn(Hq, device=DEV) if sinks else None
    scale = D ** -0.5
    got, got_lse = cu().paged_attention(q, cache, meta, scale, sliding_window=window, softcap=softcap,
                                        sinks=sk, k_scale=k_scale, v_scale=v_scale, return_lse=True)
    want, want_lse = ref.paged_attention(q, cache, bt, sl, qsl, scale, num_reqs=R, sliding_window=window,
                                         softcap=softcap, sinks=sk, k_scale=k_scale, v_scale=v_scale,
                                         return_lse=True)
    _close(got, want, 2e-2, 2e-2)
    fin = torch.isfinite(want_lse)
    _close(got_lse[fin], want_lse[fin], 1e-2, 1e-2)


@pytest.mark.parametrize("Hq,Hkv,D", [(32, 8, 128), (8, 1, 128), (4, 2, 64)])
def test_attention_decode(Hq, Hkv, D):
    ctx = [0, 15, 16, 100, 1023, 2500, 7]
    _attn_case([1] * len(ctx), ctx, Hq, Hkv, D, num_decode=len(ctx))


def test_attention_decode_many_splits(monkeypatch):
    monkeypatch.setenv("B200_ATTN_SPLIT_KV", "5")
    from vllm_torchtpu_b200 import envs
    envs.reset()
    _attn_case([1, 1, 1], [3000, 1, 77], 16, 4, 128, num_decode=3)


def test_attention_spec_verify_rows():
    # q_len 3 with 4 heads per kv head = 12 rows in the 16-row decode tile
    _attn_case([3, 3, 1], [50, 700, 9], 8, 2, 128, num_decode=3)


@pytest.mark.parametrize("Hq,Hkv,D", [(32, 8, 128), (4, 2, 64)])
def test_attention_prefill_and_mixed(Hq, Hkv, D):
    _attn_case([1, 1, 200, 64, 65, 1, 333], [40, 900, 0, 128, 37, 0, 1000], Hq, Hkv, D, num_decode=2)


@pytest.mark.parametrize("Hq,Hkv,D", [(32, 8, 128), (4, 2, 64)])
def test_attention_fp8_kv_cache(Hq, Hkv, D):
    ctx = [0, 15, 16, 100, 1023, 2500, 7]
    _attn_case([1] * len(ctx), ctx, Hq, Hkv, D, num_decode=len(ctx), kv_fp8=True)
    _attn_case([1, 1, 200, 64, 65, 1, 333], [40, 900, 0, 128, 37, 0, 1000], Hq, Hkv, D, num_decode=2,
               kv_fp8=True)
    _attn_case([1, 130, 17], [500, 300, 0], Hq, Hkv, D, window=128, sinks=True, num_decode=1, kv_fp8=True)


# prompts over an e4m3 cache with values of scale one: pages expanded for the tcgen05 kernel.  Pages of 16 and 32, lengths that
# end a page, requests of one token behind and between, no decode range
@pytest.mark.parametrize("Hq,Hkv,bs,kw", [(32, 8, 16, {}), (8, 8, 16, dict(softcap=20.0)), (8, 1, 32, dict(sinks=True))])
def test_attention_fp8_kv_cache_expanded_for_prompts(Hq, Hkv, bs, kw):
    _attn_case([1, 200, 1, 16, 333, 400], [33, 0, 70, 16, 1000, 1500], Hq, Hkv, 128, num_decode=1, kv_fp8=True, scales=(0.7, 1.0),
               bs=bs, **kw)
    _attn_case([3, 700], [1532, 0], Hq, Hkv, 128, num_decode=0, kv_fp8=True, scales=(1.0, 1.0), bs=bs, **kw)


def test_expanded_pages_take_what_the_lengths_need(monkeypatch):
    """One long request beside short ones: a pool of the pages of all of them, not of the longest for each."""
    lens, bs, Hkv = [(300, 3000), (64, 64), (1, 17), (40, 1030)], 16, 8
    g = torch.Generator(device=DEV).manual_seed(12)
    kv = torch.randn(2, Hkv, sum(s for _, s in lens), 128, device=DEV, generator=g).to(torch.float8_e4m3fn).view(torch.uint8)
    pages, meta = _one_request_each(kv, lens, bs)
    pages = pages.view(torch.float8_e4m3fn)
    q = torch.randn(meta.num_tokens, 32, 128, device=DEV, generator=g).bfloat16()
    made, inner = [], cu()._expanded_pages
    monkeypatch.setattr(cu(), "_expanded_pages", lambda *a: made.append(inner(*a)) or made[-1])
    out = cu().paged_attention(q, pages, meta, 128 ** -0.5)
    pool, table = made[0]
    assert pool.shape[0] == sum(-(-s // bs) for _, s in lens) and table.shape[1] == -(-3000 // bs)
    want = ref.paged_attention(q, pages, meta.block_tables, meta.seq_lens, meta.query_start_loc, 128 ** -0.5, num_reqs=len(lens))
    _close(out, want, 2e-2, 2e-2)


def test_attention_window_softcap_sinks():
    _attn_case([1, 130, 17], [500, 300, 0], 8, 2, 128, window=128, num_decode=1)
    _attn_case([1, 130], [500, 300], 8, 2, 128, softcap=30.0, num_decode=1)
    _attn_case([1, 130], [500, 300], 8, 2, 128, sinks=True, num_decode=1)


def _one_request_each(kv, lens, bs=16):
    """Prompt metadata and pages [blocks, 2, Hkv, bs, D] of requests whose keys and values kv [2, Hkv, sum of keys, D] holds."""
    need = [-(-s // bs) for _, s in lens]
    pages = torch.zeros(sum(need) + 1, 2, kv.shape[1], bs, kv.shape[3], dtype=kv.dtype, device=DEV)
    bt = torch.zeros(len(lens), max(need), dtype=torch.int32, device=DEV)
    at, off = 1, 0
    for r, (_, s) in enumerate(lens):
        bt[r, :need[r]] = torch.arange(at, at + need[r], device=DEV)
        rows = torch.zeros(2, kv.shape[1], need[r] * bs, kv.shape[3], dtype=kv.dtype, device=DEV)
        rows[:, :, :s] = kv[:, :, off:off + s]
        pages[at:at + need[r]] = rows.view(2, kv.shape[1], need[r], bs, -1).permute(2, 0, 1, 3, 4)
        at, off = at + need[r], off + s
    qsl = torch.tensor([0] + [n for n, _ in lens], dtype=torch.int32).cumsum(0, dtype=torch.int32)
    sl = torch.tensor([s for _, s in lens], dtype=torch.int32)
    return pages, AttentionMetadata(
        positions=None, slot_mapping=None, block_tables=bt, seq_lens=sl.to(DEV), query_start_loc=qsl.to(DEV), num_reqs=len(lens),
        num_tokens=int(qsl[-1]), num_decode_reqs=0, max_query_len=max(n for n, _ in lens), max_seq_len=int(sl.max()),
        padded_num_reqs=len(lens), padded_num_tokens=int(qsl[-1]), query_start_loc_cpu=qsl.long(), seq_lens_cpu=sl.long())


def test_soft_cap_of_the_prompt_kernel():
    """A row's largest score has weight one exactly: where a row sees one key the log-sum-exp is its capped score to the bit,
    as fp32 gives it.  And outputs against 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(11)
    Hq, Hkv, D, R, cap, scale = 32, 8, 128, 60, 50.0, 128 ** -0.5
    q, kv = torch.zeros(R, Hq, D, device=DEV), torch.zeros(2, Hkv, R, D, device=DEV)
    q[:, :, 0] = torch.randn(R, Hq, device=DEV, generator=g) * 40
    kv[0, :, :, 0] = torch.randn(Hkv, R, device=DEV, generator=g) * 16
    q, kv = q.bfloat16(), kv.bfloat16()
    pages, meta = _one_request_each(kv, [(1, 1)] * R)
    _, lse = cu().paged_attention(q, pages, meta, scale, softcap=cap, return_lse=True)
    s = q[:, :, 0].float() * kv[0, :, :, 0].float().t().repeat_interleave(Hq // Hkv, 1)              # exact in fp32
    log2e = torch.tensor(1.4426950408889634, device=DEV)
    c = cap * log2e
    want = c * torch.tanh(s * (torch.tensor(scale, device=DEV) * log2e) / c) * torch.tensor(0.6931471805599453, device=DEV)
    assert (lse == want).float().mean() > 0.97, (lse == want).float().mean()
    torch.testing.assert_close(lse, want, rtol=3e-7, atol=1e-7)

    n, m = 200, 1100
    q = torch.randn(n, Hq, D, device=DEV, generator=g).bfloat16()
    kv = (torch.randn(2, Hkv, m, D, device=DEV, generator=g) * 4).bfloat16()
    pages, meta = _one_request_each(kv, [(n, m)])
    out = cu().paged_attention(q, pages, meta, scale, softcap=cap)
    k, v = (t.double().repeat_interleave(Hq // Hkv, 0) for t in kv)
    a = cap * torch.tanh(q.double().transpose(0, 1) @ k.transpose(1, 2) * scale / cap)
    a = a.masked_fill(torch.ones(n, m, dtype=torch.bool, device=DEV).triu(m - n + 1), -float("inf"))
    want = (torch.softmax(a, -1) @ v).transpose(0, 1)
    # bf16 probabilities and outputs: 2^-9 each, uniform rounding, so about 2^-9 in the norm
    assert (out.double() - want).norm() / want.norm() < 2 ** -8


def test_argmax_and_sampling():
    R, V = 9, 128256
    g = torch.Generator(device=DEV).manual_seed(3)
    logits = (torch.randn(R, V, device=DEV, generator=g) * 3).bfloat16()
    assert torch.equal(cu().argmax(logits).long(), logits.float().argmax(-1))
    temp = torch.tensor([0.0, 0.7, 1.0, 1.3, 0.5, 1.0, 1.0, 0.9, 2.0], device=DEV)
    top_k = torch.tensor([0, 50, 0, 5, 1, 0, 1000, 20, 0], device=DEV, dtype=torch.int32)
    top_p = torch.tensor([1.0, 1.0, 0.9, 0.8, 1.0, 0.5, 0.95, 1.0, 1.0], device=DEV)
    u = cu().philox_uniform(R, V, 7, 3, DEV)
    assert 0.45 < float(u.mean()) < 0.55 and float(u.min()) > 0 and float(u.max()) < 1
    got = cu().sample(logits, temp, top_k, top_p, uniform=u)
    want = ref.sample(logits, temp, top_k, top_p, uniform=u)
    assert torch.equal(got.long(), want)
    step = torch.tensor([3], dtype=torch.int64, device=DEV)
    got2 = cu().sample(logits, temp, top_k, top_p, uniform=None, seed=7, step_tensor=step)
    assert torch.equal(got2, got)


def test_sampling_cluster_kernel_on_an_odd_vocabulary():
    """Rows of odd length start on odd element offsets (two-byte loads instead of pairs) and the last CTA of
    the cluster holds a ragged tail."""
    R, V = 6, 50001
    g = torch.Generator(device=DEV).manual_seed(5)
    logits = (torch.randn(R, V, device=DEV, generator=g) * 2.5).bfloat16()
    temp = torch.tensor([0.8, 0.0, 1.0, 1.2, 0.6, 1.0], device=DEV)
    top_k = torch.tensor([40, 0, 0, 3, 0, 2000], device=DEV, dtype=torch.int32)
    top_p = torch.tensor([0.9, 1.0, 0.7, 1.0, 1.0, 0.99], device=DEV)
    u = cu().philox_uniform(R, V, 11, 1, DEV)
    got = cu().sample(logits, temp, top_k, top_p, uniform=u)
    want = ref.sample(logits, temp, top_k, top_p, uniform=u)
    assert torch.equal(got.long(), want)


# keys per thread of the cluster kernel (8, 32, 40, 64) at their limits, the single-CTA kernel on both sides of them; lists that
# overflow (equal logits), fewer finite logits than k, k at the limit of the list
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [4095, 4096, 32768, 32770, 131072, 151936, 163841, 262145])
def test_sampling_sizes_and_types(V, dtype):
    R = 12
    g = torch.Generator(device=DEV).manual_seed(V)
    logits = (torch.randn(R, V, device=DEV, generator=g) * 2.0).to(dtype)
    logits[0] = 0.5
    logits[1, 7:] = -float("inf")
    logits[2, ::2] = -float("inf")
    logits[3] *= 100.0
    temp = torch.rand(R, device=DEV, generator=g) + 0.3
    temp[11] = 0.0
    top_k = torch.tensor([50, 50, 512, 511, 1, 0, 0, 20, 600, 2, 3000, 5], device=DEV, dtype=torch.int32)
    top_p = torch.tensor([0.9, 0.9, 0.5, 1.0, 1.0, 0.95, 1.0, 0.3, 0.9, 0.99, 0.8, 1.0], device=DEV)
    u = cu().philox_uniform(R, V, 5, 2, DEV)
    got = cu().sample(logits, temp, top_k, top_p, uniform=u)
    # the statement with ties at a threshold kept (bf16 logits tie): masses in 64 bits
    x = logits.float() * (1.0 / temp.clamp_min(1e-5))[:, None]
    want = logits.float().argmax(-1)
    for r in range(R - 1):
        s = x[r].sort(descending=True).values
        k = int(top_k[r])
        kept = x[r] >= (s[k - 1] if 0 < k < V else s[-1])
        if top_p[r] < 1:
            mass = torch.exp(x[r].double() - s[0].double()) * kept
            order = x[r].argsort(descending=True)
            # the first value at which the mass from the top on, ties included, reaches its share
            at = int((mass[order].cumsum(0) >= top_p[r].double() * mass.sum()).nonzero()[0])
            kept &= x[r] >= x[r][order[at]]
        noisy = x[r] - torch.log(-torch.log(u[r].clamp(1e-20, 1.0 - 1e-7)))
        want[r] = noisy.masked_fill(~kept, float("-inf")).argmax()
    assert torch.equal(got.long(), want)


# clusters of 8, 4, 2 and 1 CTA and their instances of 8, 16 and 32 keys a thread at their limits, rows beyond which a second
# launch takes those of which nothing is cut
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("R,V", [(9, 8193), (10, 8193), (18, 65537), (37, 32768), (38, 8193), (74, 32769), (75, 16384), (150, 8193),
                                 (400, 4097), (130, 32770), (150, 32770), (96, 163000), (64, 163000)])
def test_sampling_of_many_rows_draws_what_few_rows_draw(R, V, dtype):
    """A row's token depends on the row, not on how many there are: the first rows alone take clusters of eight."""
    g = torch.Generator(device=DEV).manual_seed(R)
    logits = (torch.randn(R, V, device=DEV, generator=g) * 2.0).to(dtype)
    logits[1, 5:] = -float("inf")
    temp = torch.rand(R, device=DEV, generator=g) + 0.3
    temp[2] = 0.0
    top_k = torch.tensor([0, 0, 0, 50, 600, 0, 1, V], device=DEV, dtype=torch.int32).repeat(R // 8 + 1)[:R].contiguous()
    top_p = torch.tensor([1.0, 1.0, 0.5, 0.9, 1.0, 0.95, 1.0, 1.0], device=DEV).repeat(R // 8 + 1)[:R].contiguous()
    step = torch.tensor([3], dtype=torch.int64, device=DEV)
    draw = lambda n: cu().sample(logits[:n], temp[:n], top_k[:n], top_p[:n], seed=7, step_tensor=step)       # noqa: E731
    many, few = draw(R), draw(8)
    assert torch.equal(many[:8], few)
    # noise made in front of the call is drawn from element by element
    u = cu().philox_uniform(R, V, 7, 3, DEV)
    assert torch.equal(many, cu().sample(logits, temp, top_k, top_p, uniform=u))
    free = (((top_k <= 0) | (top_k >= V)) & (top_p >= 1) & (temp > 0)).nonzero()[:, 0]
    x = logits.float() * (1.0 / temp.clamp_min(1e-5))[:, None] - torch.log(-torch.log(u.clamp(1e-20, 1.0 - 1e-7)))
    # the kernel's logarithm has an absolute error of 2^-21 near one, where -log(u) of the winners is 1e-5: 0.05 of noise
    got, best = x.gather(1, many.long()[:, None])[:, 0], x.amax(-1)
    assert (best - got)[free].max() < 1.0


def test_logprobs():
    R, V = 5, 32000
    logits = torch.randn(R, V, device=DEV).bfloat16()
    tok = torch.randint(0, V, (R,), device=DEV)
    a = cu().gather_logprobs(logits, tok, 5)
    b = ref.gather_logprobs(logits, tok, 5)
    _close(a[0], b[0], 1e-3, 1e-3)
    _close(a[1], b[1], 1e-3, 1e-3)
    # bf16 logits tie often: ids may differ among equal values, the values they point at may not
    lf = logits.float()
    assert torch.equal(lf.gather(1, a[2].long()), lf.gather(1, b[2]))
    assert torch.equal(a[3].long(), b[3])


@pytest.mark.parametrize("Hq,Hkv,D", [(16, 16, 64), (8, 2, 128)])
def test_encoder_attention_bidirectional(Hq, Hkv, D):
    """Non-causal varlen attention (vision encoder): every token sees its whole sequence."""
    g = torch.Generator(device=DEV).manual_seed(5)
    lens = [1, 63, 64, 200, 577]
    offs = [0]
    for n in lens:
        offs.append(offs[-1] + n)
    T = offs[-1]
    q = torch.randn(T, Hq, D, device=DEV, generator=g).bfloat16()
    k = torch.randn(T, Hkv, D, device=DEV, generator=g).bfloat16()
    v = torch.randn(T, Hkv, D, device=DEV, generator=g).bfloat16()
    got = cu().encoder_attention(q, k, v, offs)
    want = ref.encoder_attention(q, k, v, offs)
    _close(got, want, 2e-2, 2e-2)


@pytest.mark.parametrize("spec", ["silu", "gelu", "gelu_tanh", "swigluoai", "swigluoai:1.5:2", "silu_clamp:3",
                                  "situ:3:none", "situ:3:2"])
def test_gated_activation_kernels(spec):
    from vllm_torchtpu_b200.ops import cuda
    from vllm_torchtpu_b200.ops import reference as ref
    g = torch.Generator(device=DEV).manual_seed(0)
    x = (torch.randn(37, 2 * 1032, device=DEV, generator=g) * 4).bfloat16()
    got = cuda.gated_act_and_mul(x, spec)
    want = ref.gated_act_and_mul(x.float(), spec)
    torch.testing.assert_close(got.float(), want, rtol=2e-2, atol=2e-2)


def test_moe_experts_with_oai_swiglu_on_the_device():
    from vllm_torchtpu_b200.ops import cuda
    from vllm_torchtpu_b200.ops import reference as ref
    g = torch.Generator(device=DEV).manual_seed(1)
    T, H, I, E, k = 50, 256, 128, 8, 2
    x = torch.randn(T, H, device=DEV, generator=g).bfloat16()
    w13 = (torch.randn(E, 2 * I, H, device=DEV, generator=g) * 0.08).bfloat16()
    w2 = (torch.randn(E, H, I, device=DEV, generator=g) * 0.08).bfloat16()
    logits = torch.randn(T, E, device=DEV, generator=g)
    wt, ids = torch.topk(torch.softmax(logits, -1), k, -1)
    ids, wt = ids.int().contiguous(), wt.float().contiguous()
    got = cuda.moe_experts(x, w13, w2, ids, wt, 0, act="swigluoai")
    want = ref.moe_experts(x, w13, w2, ids, wt, 0, act="swigluoai")
    err = (got.float() - want.float()).abs().max().item()
    assert err <= 3e-2 * want.float().abs().max().item() + 2e-2, err
    assert cuda.check_status() == 0
