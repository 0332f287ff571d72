"""MLA latent-cache attention kernel (dense and top-k sparse) and cache write vs the fp32 statements."""
import pytest
import torch

from vllm_torchtpu_b200.ops import reference as ref
from vllm_torchtpu_b200.runner.attn_metadata import AttentionMetadata

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(q_lens, ctx_lens, H, L, R, bs=16, topk=None, seed=0):
    from vllm_torchtpu_b200.ops import cuda
    g = torch.Generator(device=DEV).manual_seed(seed)
    Dq = L + R
    n = len(q_lens)
    seq = [q + c for q, c in zip(q_lens, ctx_lens)]
    maxb = max(-(-s // bs) for s in seq) + 1
    nb = sum(-(-s // bs) for s in seq) + 2
    cache = (torch.randn(nb, bs, Dq, device=DEV, generator=g) * 0.5).bfloat16()
    perm = (torch.randperm(nb - 1, device=DEV, generator=g) + 1).to(torch.int32)
    bt = torch.zeros(n, maxb, dtype=torch.int32, device=DEV)
    off = 0
    for r, s in enumerate(seq):
        k = -(-s // bs)
        bt[r, :k] = perm[off:off + k]
        off += k
    T = sum(q_lens)
    q = (torch.randn(T, H, Dq, device=DEV, generator=g) * 0.3).bfloat16()
    qsl = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    sl = torch.tensor(seq, dtype=torch.int32, device=DEV)
    meta = AttentionMetadata(None, None, bt, sl, qsl, n, T, num_decode_reqs=0, max_query_len=max(q_lens),
                             max_seq_len=max(seq), padded_num_reqs=n, padded_num_tokens=T)
    ti = None
    if topk:
        # per token: a random subset of its visible positions, padded with -1, plus out-of-range junk
        ti = torch.full((T, topk), -1, dtype=torch.int32, device=DEV)
        tok = 0
        for r in range(n):
            for j in range(q_lens[r]):
                vis = seq[r] - q_lens[r] + j + 1
                k = min(topk - 2, vis)
                sel = torch.randperm(vis, device=DEV, generator=g)[:k].to(torch.int32)
                ti[tok, :k] = sel
                ti[tok, topk - 1] = seq[r] + 5            # beyond the context: ignored
                tok += 1
    scale = (L + R) ** -0.5
    got, got_lse = cuda.mla_paged_attention(q, cache, meta, scale, L, topk_indices=ti, return_lse=True)
    want, want_lse = ref.mla_paged_attention(q, cache, bt, sl, qsl, scale, L, num_reqs=n, topk_indices=ti,
                                             return_lse=True)
    torch.testing.assert_close(got.float(), want.float(), rtol=2e-2, atol=2e-2)
    fin = torch.isfinite(want_lse)
    torch.testing.assert_close(got_lse[fin], want_lse[fin], rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("H,L,R", [(128, 512, 64), (16, 512, 64), (4, 64, 16), (8, 128, 32)])
def test_mla_decode(H, L, R):
    _case([1, 1, 1, 1], [0, 15, 300, 1029], H, L, R)


def test_mla_prefill_and_mixed():
    _case([1, 37, 3, 64], [50, 0, 700, 20], 16, 512, 64)


# tiles of 128 (token, head) rows, chunks of 128 keys in pages of 16: one row, rows across tokens, tiles that end inside a
# request, contexts around a page and a chunk, several items per pair of SMs, requests without tokens
@pytest.mark.parametrize("q_lens,ctx,H", [([1], [0], 1), ([1, 1, 1], [15, 16, 17], 3), ([1, 1, 1, 1], [126, 127, 128, 129], 128),
                                          ([45, 0, 130, 1], [0, 64, 200, 3000], 24), ([300], [33], 128)])
def test_mla_tiles_of_128_rows(q_lens, ctx, H):
    _case(q_lens, ctx, H, 512, 64)


# pages of more than 16 rows: several copies of a page, pages that end inside a chunk of 128 keys
@pytest.mark.parametrize("bs", [32, 48, 64, 128])
def test_mla_pages_of_more_rows(bs):
    _case([1, 1, 1, 70, 5], [0, bs - 1, bs, 430, 131], 16, 512, 64, bs=bs)
    _case([1] * 3, [1000, 129, 2050], 128, 512, 64, bs=bs)


def test_mla_captured_step_with_more_splits_than_chunks():
    """The splits of a captured step follow from the batch; replayed on short contexts most of them see no key."""
    from vllm_torchtpu_b200.ops import cuda
    g = torch.Generator(device=DEV).manual_seed(4)
    R, H, L = 4, 16, 512
    cache = torch.randn(1 + R * 64, 16, 576, device=DEV, generator=g).bfloat16()
    bt = (torch.randperm(R * 64, device=DEV, generator=g) + 1).to(torch.int32).view(R, 64).contiguous()
    q = torch.randn(R, H, 576, device=DEV, generator=g).bfloat16()
    sl = torch.full((R,), 1000, dtype=torch.int32, device=DEV)
    qsl = torch.arange(R + 1, dtype=torch.int32, device=DEV)
    meta = AttentionMetadata(None, None, bt, sl, qsl, R, R, num_decode_reqs=R, max_query_len=1, max_seq_len=1000,
                             padded_num_reqs=R, padded_num_tokens=R)
    cuda.mla_paged_attention(q, cache, meta, 576 ** -0.5, L)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = cuda.mla_paged_attention(q, cache, meta, 576 ** -0.5, L)
    for lens in ([1, 16, 129, 300], [1024, 3, 640, 128], [0, 1, 0, 5]):
        sl.copy_(torch.tensor(lens, dtype=torch.int32))
        graph.replay()
        for r, n in enumerate(lens):
            if n == 0:
                assert out[r].eq(0).all()
                continue
            rows = cache[bt[r].long()].view(-1, 576)[:n].double()
            want = torch.softmax(q[r].double() @ rows.t() * 576 ** -0.5, -1) @ rows[:, :L]
            assert (out[r].double() - want).norm() / want.norm() < 2 ** -7
    assert cuda.check_status() == 0


def test_mla_rows_of_the_cache_that_nothing_wrote_do_not_matter():
    from vllm_torchtpu_b200.ops import cuda
    g = torch.Generator(device=DEV).manual_seed(3)
    seq, H = [70, 131, 16], 16
    cache = torch.full((24, 16, 576), float("nan"), dtype=torch.bfloat16, device=DEV)
    bt = torch.zeros(3, 12, dtype=torch.int32, device=DEV)
    at = 1
    for r, s in enumerate(seq):
        n = -(-s // 16)
        bt[r, :n] = torch.arange(at, at + n, device=DEV)
        rows = cache[at:at + n].view(-1, 576)
        rows[:s] = torch.randn(s, 576, device=DEV, generator=g).bfloat16()
        at += n
    # one request decodes, one has a chunk; two rows of padding behind the step's tokens
    lens = [1, 40, 16]
    qsl = torch.tensor([0, 1, 41, 57], dtype=torch.int32, device=DEV)
    q = torch.randn(59, H, 576, device=DEV, generator=g).bfloat16()
    sl = torch.tensor(seq, dtype=torch.int32, device=DEV)
    meta = AttentionMetadata(None, None, bt, sl, qsl, 3, 57, num_decode_reqs=1, max_query_len=40, max_seq_len=131,
                             padded_num_reqs=3, padded_num_tokens=59)
    out, lse = cuda.mla_paged_attention(q, cache, meta, 576 ** -0.5, 512, return_lse=True)
    want = ref.mla_paged_attention(q[:57], torch.nan_to_num(cache), bt, sl, qsl, 576 ** -0.5, 512, num_reqs=3)
    torch.testing.assert_close(out[:57].float(), want.float(), rtol=2e-2, atol=2e-2)
    assert out[57:].eq(0).all() and torch.isneginf(lse[57:]).all()
    assert sum(lens) == 57 and cuda.check_status() == 0


def test_mla_sparse_topk():
    _case([1, 5, 1], [400, 90, 7], 32, 512, 64, topk=64)


def test_mla_write_cache():
    from vllm_torchtpu_b200.ops import cuda
    T, L, R, nb, bs = 23, 512, 64, 5, 16
    kv = torch.randn(T, L + R + 8, device=DEV).bfloat16()
    kv_c, k_pe = kv[:, :L], kv[:, L:L + R]
    slots = torch.randperm(nb * bs, device=DEV)[:T].to(torch.int32)
    slots[3] = -1
    c1 = torch.zeros(nb, bs, L + R, device=DEV, dtype=torch.bfloat16)
    c2 = c1.clone()
    cuda.mla_write_cache(c1, kv_c, k_pe, slots)
    ref.mla_write_cache(c2, kv_c, k_pe, slots)
    assert torch.equal(c1, c2)


def test_deepseek_style_engine_runs_on_gpu_and_matches_dense_logits():
    """MLA + MoE model through the engine on the GPU: first-token logits against the dense fp32
    forward of the same weights, and graph decode == eager decode."""
    import dataclasses

    import numpy as np

    from vllm_torchtpu_b200 import SamplingParams
    from vllm_torchtpu_b200.config import model_preset
    from vllm_torchtpu_b200.engine.llm import LLM
    from vllm_torchtpu_b200.models.reference_forward_mla import dense_mla_logits
    from vllm_torchtpu_b200.ops import cuda
    cfg = dataclasses.replace(model_preset("tiny-mla"), dtype=torch.bfloat16)
    rng = np.random.RandomState(0)
    prompts = [rng.randint(0, cfg.vocab_size, size=n).tolist() for n in (5, 17, 40)]
    sp = SamplingParams(temperature=0.0, max_tokens=6, ignore_eos=True)

    def make(**kw):
        return LLM(cfg, device="cuda", max_num_seqs=8, max_num_batched_tokens=128, block_size=16,
                   num_gpu_blocks_override=64, **kw)
    llm = make(enforce_eager=True)
    eng = llm.engine
    eng.add_request(prompts[2], SamplingParams(max_tokens=1))
    out = eng.scheduler.schedule()
    r = eng.runner
    r._update_batch(out)
    prep = r._prepare_inputs(out)
    prep["bufs"].upload(prep["R_pad"])
    _, logits = r._forward_and_sample(prep["bufs"], r._make_meta(prep), prep["T_pad"], prep["R_pad"], True)
    want = dense_mla_logits(r.model, prompts[2])[-1]
    err = (logits[0].float() - want.to(logits.device)).abs().max().item()
    assert err < 0.08 * want.abs().max().item() + 0.05, err
    eager = [o.outputs[0].token_ids for o in make(enforce_eager=True).generate(prompts, sp)]
    graph = [o.outputs[0].token_ids for o in make().generate(prompts, sp)]
    assert eager == graph
    assert cuda.check_status() == 0


@pytest.mark.parametrize("interleaved", [False, True])
def test_mla_absorb_and_unabsorb_match_einsum(interleaved):
    """W_UK / W_UV as grouped GEMMs over the heads, rope of the rope dims, against fp32 einsum + the
    reference rotary embedding."""
    from vllm_torchtpu_b200.ops import cuda
    from vllm_torchtpu_b200.ops import reference as ref
    T, H, nope, rope, L, v = 37, 16, 128, 64, 512, 128
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(T, H, nope + rope, device="cuda", generator=g).bfloat16()
    kv = torch.randn(T, L + rope, device="cuda", generator=g).bfloat16()
    w_uk = (torch.randn(H, nope, L, device="cuda", generator=g) * 0.05).bfloat16()
    w_uv = (torch.randn(H, L, v, device="cuda", generator=g) * 0.05).bfloat16()
    pos = torch.randint(0, 4000, (T,), device="cuda", generator=g, dtype=torch.int32)
    inv_freq = (1.0 / (10000 ** (torch.arange(0, rope, 2, device="cuda").float() / rope))).contiguous()
    q_latent, k_pe = cuda.mla_absorb(q, kv, pos, inv_freq, w_uk.transpose(1, 2).contiguous(), nope, rope, L,
                                     interleaved)
    torch.cuda.synchronize()
    want_ql = torch.einsum("thn,hnl->thl", q[..., :nope].float(), w_uk.float())
    want_qpe = ref.apply_rope(q[..., nope:], pos, inv_freq, interleaved).float()
    want_kpe = ref.apply_rope(kv[:, L:].reshape(T, 1, rope), pos, inv_freq, interleaved).reshape(T, rope).float()
    assert (q_latent[..., :L].float() - want_ql).abs().max() <= 2e-2 * want_ql.abs().max() + 1e-2
    assert (q_latent[..., L:].float() - want_qpe).abs().max() <= 3e-2
    assert (k_pe.float() - want_kpe).abs().max() <= 3e-2
    o_lat = torch.randn(T, H, L, device="cuda", generator=g).bfloat16()
    y = cuda.mla_unabsorb(o_lat, w_uv.transpose(1, 2).contiguous())
    torch.cuda.synchronize()
    want = torch.einsum("thl,hlv->thv", o_lat.float(), w_uv.float()).reshape(T, H * v)
    assert (y.float() - want).abs().max() <= 2e-2 * want.abs().max() + 1e-2
    assert cuda.check_status() == 0
