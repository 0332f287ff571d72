"""Gated DeltaNet kernels vs the PyTorch recurrence, including state carried across steps."""
import pytest
import torch

from vllm_torchtpu_b200.ops import gdn_reference as g
from vllm_torchtpu_b200.runner.attn_metadata import AttentionMetadata

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _meta(q_lens, ctx, slots):
    qsl = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    sl = torch.tensor([a + b for a, b in zip(q_lens, ctx)], dtype=torch.int32, device=DEV)
    return AttentionMetadata(None, None, None, sl, qsl, len(q_lens), sum(q_lens),
                             padded_num_reqs=len(q_lens), padded_num_tokens=sum(q_lens),
                             state_slots=torch.tensor(slots, dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("Hk,Hv,dk,dv", [(2, 4, 128, 128), (2, 2, 64, 64)])
def test_gdn_forward_two_steps(Hk, Hv, dk, dv):
    from vllm_torchtpu_b200.ops import cuda
    torch.manual_seed(0)
    C = 2 * Hk * dk + Hv * dv
    conv_w = (torch.randn(C, 4, device=DEV) * 0.3).bfloat16()
    A_log = torch.randn(Hv, device=DEV) * 0.3
    dt_bias = torch.randn(Hv, device=DEV) * 0.3
    pools = [(torch.zeros(5, C, 3, device=DEV, dtype=torch.bfloat16), torch.zeros(5, Hv, dk, dv, device=DEV))
             for _ in range(2)]
    for q_lens, ctx in (([17, 1, 40], [0, 0, 0]), ([1, 1, 5], [17, 1, 40])):
        T = sum(q_lens)
        mixed = torch.randn(T, C, device=DEV).bfloat16()
        a, b = torch.randn(T, Hv, device=DEV).bfloat16(), torch.randn(T, Hv, device=DEV).bfloat16()
        meta = _meta(q_lens, ctx, [3, 0, 2])
        got = cuda.gdn_forward(mixed, a, b, meta, pools[0][0], pools[0][1], conv_w, A_log, dt_bias, Hk, Hv, dk, dv)
        want = g.gdn_forward(mixed, a, b, None, meta, pools[1][0], pools[1][1], conv_w, A_log, dt_bias, Hk, Hv, dk, dv)
        err = (got.float() - want.float()).abs().max().item()
        assert err <= 3e-2 * want.float().abs().max().item() + 1e-2, err
    torch.testing.assert_close(pools[0][1], pools[1][1], rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("Hk,Hv,dk,dv,lb", [(2, 2, 128, 128, None), (2, 4, 64, 64, -5.0), (1, 2, 32, 128, None)])
def test_kda_forward_two_steps(Hk, Hv, dk, dv, lb):
    """Per-channel decay (Kimi Delta Attention): both gate forms, state carried across two steps."""
    from vllm_torchtpu_b200.ops import cuda
    torch.manual_seed(1)
    A_log = torch.randn(Hv, device=DEV) * 0.3
    dt_bias = torch.randn(Hv, dk, device=DEV) * 0.3
    pools = [torch.zeros(5, Hv, dk, dv, device=DEV) for _ in range(2)]
    for q_lens, ctx in (([17, 1, 40], [0, 0, 0]), ([1, 1, 5], [17, 1, 40])):
        T = sum(q_lens)
        q = torch.randn(T, Hk, dk, device=DEV).bfloat16()
        k = torch.randn(T, Hk, dk, device=DEV).bfloat16()
        v = torch.randn(T, Hv, dv, device=DEV).bfloat16()
        a = torch.randn(T, Hv, dk, device=DEV).bfloat16()
        b = torch.randn(T, Hv, device=DEV).bfloat16()
        meta = _meta(q_lens, ctx, [3, 0, 2])
        got = cuda.kda_forward(q, k, v, a, b, meta, pools[0], A_log, dt_bias, lb)
        want = g.kda_forward(q, k, v, a, b, meta, pools[1], A_log, dt_bias, lb)
        err = (got.float() - want.float()).abs().max().item()
        assert err <= 3e-2 * want.float().abs().max().item() + 1e-2, err
    torch.testing.assert_close(pools[0], pools[1], rtol=3e-2, atol=3e-2)


# chunks of the convolution (32 tokens), of the rule on the tensor cores (64) and of the staged tokens (16 and 8), portions shorter than the carried window, requests
# without tokens or without a state, rows behind the step's tokens, value widths that are no multiple of the 64 columns of a
# CTA or of a vector, more requests than a warp has lanes
@pytest.mark.parametrize("Hk,Hv,dk,dv", [(1, 2, 128, 128), (1, 1, 64, 72), (2, 2, 32, 33)])
@pytest.mark.parametrize("q_lens,ctx", [([1, 2, 3, 31, 32, 33, 0, 65], [0, 1, 2, 9, 0, 70, 5, 0]), ([1] * 35, [0, 4, 9, 30, 2] * 7),
                                        ([64, 128, 129, 2, 1, 200, 63], [0, 3, 0, 8, 8, 64, 1]), ([3, 2, 5, 1], [0, 1, 4, 2])])
def test_ragged_portions_and_untouched_rows(Hk, Hv, dk, dv, q_lens, ctx):
    from vllm_torchtpu_b200.ops import cuda
    gen = torch.Generator(device=DEV).manual_seed(7)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)                      # noqa: E731
    C, R, T = 2 * Hk * dk + Hv * dv, len(q_lens), sum(q_lens)
    slots = [(3 * r + 1) % (R + 2) if (R + 2) % 3 else r for r in range(R)]
    off = 4 if R > 4 else None
    if off is not None:
        slots[off] = -1                                                               # no state: rows of zeros
    meta = _meta(q_lens, ctx, slots)
    pad = 3
    mixed, conv_w = rnd(T + pad, C).bfloat16(), (rnd(C, 4) * 0.3).bfloat16()
    a, b, ac = rnd(T + pad, Hv).bfloat16(), rnd(T + pad, Hv).bfloat16(), rnd(T + pad, Hv, dk).bfloat16()
    A_log, dt, dtc = rnd(Hv) * 0.3, rnd(Hv) * 0.3, rnd(Hv, dk) * 0.3
    conv, rec = rnd(R + 2, C, 3).bfloat16(), rnd(R + 2, Hv, dk, dv) * 0.1
    got_pools, want_pools = [conv.clone(), rec.clone()], [conv.clone(), rec.clone()]
    got = cuda.gdn_forward(mixed, a, b, meta, *got_pools, conv_w, A_log, dt, Hk, Hv, dk, dv)
    keep = [r for r in range(R) if slots[r] >= 0]
    rows = torch.cat([torch.arange(sum(q_lens[:r]), sum(q_lens[:r + 1]), device=DEV) for r in keep])
    sub = _meta([q_lens[r] for r in keep], [ctx[r] for r in keep], [slots[r] for r in keep])
    want = g.gdn_forward(mixed[rows], a[rows], b[rows], None, sub, *want_pools, conv_w, A_log, dt, Hk, Hv, dk, dv)

    def close(x, y):
        # convolved values are bf16 on both sides: a value that rounds the other way moves a result by 2^-8 of it
        assert (x.float() - y.float()).abs().max() <= 2e-2 * y.float().abs().max() + 1e-3
    rest = torch.ones(T + pad, dtype=torch.bool, device=DEV)
    rest[rows] = False
    close(got[rows], want)
    assert got[rest].eq(0).all()
    assert torch.equal(got_pools[0], want_pools[0])
    close(got_pools[1], want_pools[1])
    y = cuda.short_conv(mixed, meta, conv.clone(), conv_w)
    assert y[rest].eq(0).all()
    q, k, v = y.split([Hk * dk, Hk * dk, Hv * dv], -1)
    q, k, v = q.reshape(-1, Hk, dk), k.reshape(-1, Hk, dk), v.reshape(-1, Hv, dv)
    got_rec, want_rec = rec.clone(), rec.clone()
    got = cuda.kda_forward(q, k, v, ac, b, meta, got_rec, A_log, dtc)
    want = g.kda_forward(q[rows], k[rows], v[rows], ac[rows], b[rows], sub, want_rec, A_log, dtc)
    close(got[rows], want)
    assert got[rest].eq(0).all()
    close(got_rec, want_rec)


def test_decays_that_underflow():
    """A decay of exactly zero forgets the state; products of decays leave the range of fp32 within a few tokens."""
    from vllm_torchtpu_b200.ops import cuda
    gen = torch.Generator(device=DEV).manual_seed(8)
    Hk, Hv, dk, dv, T = 1, 1, 128, 128, 200
    C = 2 * Hk * dk + Hv * dv
    mixed = torch.randn(T, C, device=DEV, generator=gen).bfloat16()
    a = torch.full((T, Hv), 60.0, device=DEV).bfloat16()                 # g = -60 e: below exp's range
    a[::3] = -3.0
    a[100:] = 3.0
    b = torch.randn(T, Hv, device=DEV, generator=gen).bfloat16()
    conv_w = (torch.randn(C, 4, device=DEV, generator=gen) * 0.3).bfloat16()
    A_log, dt = torch.ones(Hv, device=DEV), torch.zeros(Hv, device=DEV)
    pools = [(torch.zeros(1, C, 3, device=DEV, dtype=torch.bfloat16), torch.ones(1, Hv, dk, dv, device=DEV)) for _ in range(2)]
    meta = _meta([T], [5], [0])
    got = cuda.gdn_forward(mixed, a, b, meta, *pools[0], conv_w, A_log, dt, Hk, Hv, dk, dv)
    want = g.gdn_forward(mixed, a, b, None, meta, *pools[1], conv_w, A_log, dt, Hk, Hv, dk, dv)
    assert (got.float() - want.float()).abs().max() <= 2e-2 * want.float().abs().max()
    assert (pools[0][1] - pools[1][1]).abs().max() <= 2e-2 * pools[1][1].abs().max()


def test_silu_of_large_negative_values():
    """silu(-88) is -5.3e-37, a normal bf16 number: 1 + exp(88) is below the largest fp32 number but above 2^126, where the
    approximate division returns zero."""
    from vllm_torchtpu_b200.ops import cuda
    Hk, Hv, D = 1, 2, 128
    C = (2 * Hk + Hv) * D
    conv_w = torch.zeros(C, 4, device=DEV).bfloat16()
    conv_w[:, 3] = 1
    x = torch.full((40, C), -88.0, device=DEV).bfloat16()
    want = -88.0 / (1.0 + torch.exp(torch.tensor(88.0, dtype=torch.float64))).item()
    y = cuda.short_conv(x, _meta([33, 1, 6], [0, 0, 0], [0, 1, 2]), torch.zeros(3, C, 3, device=DEV, dtype=torch.bfloat16), conv_w)
    # (2^-9 for bf16, 2^-16 for the exponential's argument: 88 * log2(e) in fp32)
    torch.testing.assert_close(y.double() / want, torch.ones_like(y, dtype=torch.float64), rtol=0, atol=2 ** -8)
    # single tokens: o = (q k) v, q = k of unit length but for dk^-1/2, beta = 1, state from zero
    x[:, :2 * Hk * D] = 5.0
    big = torch.full((1, Hv), 30.0, device=DEV).bfloat16()
    rec = torch.zeros(1, Hv, D, D, device=DEV)
    o = cuda.gdn_forward(x[:1], big, big, _meta([1], [0], [0]), torch.zeros(1, C, 3, device=DEV, dtype=torch.bfloat16), rec, conv_w,
                         torch.zeros(Hv, device=DEV), torch.zeros(Hv, device=DEV), Hk, Hv, D, D)
    torch.testing.assert_close(o.double() / (want * D ** -0.5), torch.ones_like(o, dtype=torch.float64), rtol=0, atol=2 ** -7)


@pytest.mark.parametrize("what", ["gate", "beta", "key", "query", "value", "value inf", "huge key"])
def test_values_that_are_not_finite_reach_no_token_in_front_of_them(what):
    """Chunks of 64 tokens: what is not finite in token 70 shows in the outputs and states that it reaches token by token, and
    nowhere else.  A key whose square leaves the range of fp32 counts as a zero vector."""
    from vllm_torchtpu_b200.ops import cuda
    gen = torch.Generator(device=DEV).manual_seed(9)
    Hk, Hv, D = 2, 4, 128
    q_lens, ctx, slots = [150, 70, 20], [0, 30, 5], [2, 0, 1]
    T, C, at = sum(q_lens), (2 * Hk + Hv) * D, 70
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)                      # noqa: E731
    mixed, a, b = rnd(T, C).bfloat16(), rnd(T, Hv).bfloat16(), rnd(T, Hv).bfloat16()
    conv_w = (rnd(C, 4) * 0.3).bfloat16()
    conv_w[:, 3] = 0.5
    A_log, dt = rnd(Hv) * 0.3, rnd(Hv) * 0.3
    nan, inf = float("nan"), float("inf")
    if what == "gate":
        a[at, 1] = nan
    elif what == "beta":
        b[at, 1] = nan
    else:
        col = {"query": D + 7, "key": (Hk + 1) * D + 7, "huge key": (Hk + 1) * D + 7}.get(what, (2 * Hk + 1) * D + 7)
        mixed[at, col] = {"value inf": inf, "huge key": 1e20}.get(what, nan)
    meta = _meta(q_lens, ctx, slots)
    conv, rec = rnd(3, C, 3).bfloat16(), rnd(3, Hv, D, D) * 0.1
    got_pools, want_pools = [conv.clone(), rec.clone()], [conv.clone(), rec.clone()]
    got = cuda.gdn_forward(mixed, a, b, meta, *got_pools, conv_w, A_log, dt, Hk, Hv, D, D)
    want = g.gdn_forward(mixed, a, b, None, meta, *want_pools, conv_w, A_log, dt, Hk, Hv, D, D)
    for x, y in ((got, want), (got_pools[1], want_pools[1])):
        assert torch.equal(torch.isfinite(x), torch.isfinite(y))
        x, y = (t.float().nan_to_num(0.0, 0.0, 0.0) for t in (x, y))
        assert (x - y).abs().max() <= 2e-2 * y.abs().max() + 1e-3
    assert torch.isfinite(want[:at]).all() and cuda.check_status() == 0


@pytest.mark.parametrize("off", [1, 2])
@pytest.mark.parametrize("q_lens,ctx", [([1, 1, 1], [0, 4, 9]), ([5, 1, 40], [3, 7, 0])])
def test_states_at_any_address(q_lens, ctx, off):
    """Pools that begin on 4 or 8 bytes are taken by the kernels that read single floats or pairs."""
    from vllm_torchtpu_b200.ops import cuda
    gen = torch.Generator(device=DEV).manual_seed(10)
    Hk, Hv, D, R, T = 2, 4, 128, len(q_lens), sum(q_lens)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)                      # noqa: E731
    C = (2 * Hk + Hv) * D
    mixed, a, ac, b = rnd(T, C).bfloat16(), rnd(T, Hv).bfloat16(), rnd(T, Hv, D).bfloat16(), rnd(T, Hv).bfloat16()
    conv_w, A_log, dt, dtc = (rnd(C, 4) * 0.3).bfloat16(), rnd(Hv) * 0.3, rnd(Hv) * 0.3, rnd(Hv, D) * 0.3
    conv, rec = rnd(R, C, 3).bfloat16(), rnd(R, Hv, D, D) * 0.1
    meta = _meta(q_lens, ctx, list(range(R)))
    apart = torch.empty(rec.numel() + 4, device=DEV)[off:off + rec.numel()].view_as(rec)
    assert apart.data_ptr() % 16 == 4 * off
    q, k, v = (t.reshape(T, -1, D) for t in mixed.split([Hk * D, Hk * D, Hv * D], -1))
    for call in (lambda st: cuda.gdn_forward(mixed, a, b, meta, conv.clone(), st, conv_w, A_log, dt, Hk, Hv, D, D),
                 lambda st: cuda.kda_forward(q, k, v, ac, b, meta, st, A_log, dtc)):
        want_rec = rec.clone()
        apart.copy_(rec)
        got, want = call(apart), call(want_rec)
        # fp32 sums of 128 products in another order (2^-24 * sqrt(128) * a few), bf16 outputs
        torch.testing.assert_close(apart, want_rec, rtol=1e-4, atol=1e-5)
        torch.testing.assert_close(got.float(), want.float(), rtol=2 ** -7, atol=1e-4)


def test_rows_of_a_step_without_requests_are_zeros():
    from vllm_torchtpu_b200.ops import cuda
    Hk, Hv, D, T = 1, 2, 128, 6
    C = (2 * Hk + Hv) * D
    meta = _meta([], [], [])
    used = torch.full((T * C * 8,), float("nan"), device=DEV).bfloat16()
    del used                                                 # (the next tensors lie there)
    x, a = torch.ones(T, C, device=DEV).bfloat16(), torch.ones(T, Hv, device=DEV).bfloat16()
    pools = torch.zeros(1, C, 3, device=DEV).bfloat16(), torch.zeros(1, Hv, D, D, device=DEV)
    w, A, dt = torch.ones(C, 4, device=DEV).bfloat16(), torch.zeros(Hv, device=DEV), torch.zeros(Hv, device=DEV)
    q, v = torch.ones(T, Hk, D, device=DEV).bfloat16(), torch.ones(T, Hv, D, device=DEV).bfloat16()
    for y in (cuda.gdn_forward(x, a, a, meta, *pools, w, A, dt, Hk, Hv, D, D), cuda.short_conv(x, meta, pools[0], w),
              cuda.kda_forward(q, q, v, torch.ones(T, Hv, D, device=DEV).bfloat16(), a, meta, pools[1], A,
                               torch.zeros(Hv, D, device=DEV))):
        assert y.eq(0).all()


def test_chunks_keep_32_bits():
    """Chunks against the rule in 64 bits on the kernel's own convolved rows: 24 chunks with slow decay.  States and sums are
    fp32, every fp32 operand enters as three parts: a lost part would show as 2^-9 or 2^-17."""
    from vllm_torchtpu_b200.ops import cuda
    gen = torch.Generator(device=DEV).manual_seed(13)
    Hk, Hv, D, T = 1, 2, 128, 24 * 64 + 9
    C = (2 * Hk + Hv) * D
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=gen)                      # noqa: E731
    mixed, a, b = rnd(T, C).bfloat16(), (rnd(T, Hv) * 0.3 - 7).bfloat16(), rnd(T, Hv).bfloat16()
    conv_w, A_log, dt = (rnd(C, 4) * 0.3).bfloat16(), rnd(Hv) * 0.3, rnd(Hv) * 0.3
    meta = _meta([T], [64], [0])
    conv, rec = rnd(1, C, 3).bfloat16(), rnd(1, Hv, D, D) * 0.1
    y = cuda.short_conv(mixed, meta, conv.clone(), conv_w).double()
    got_rec = rec.clone()
    got = cuda.gdn_forward(mixed, a, b, meta, conv.clone(), got_rec, conv_w, A_log, dt, Hk, Hv, D, D)
    q, k, v = (t.reshape(T, -1, D) for t in y.split([Hk * D, Hk * D, Hv * D], -1))
    q, k = (torch.nn.functional.normalize(t, dim=-1).repeat_interleave(Hv // Hk, 1) for t in (q, k))
    decay = torch.exp(-A_log.double().exp() * torch.nn.functional.softplus(a.double() + dt.double()))
    S, beta = rec[0].double(), b.double().sigmoid()
    want = torch.empty(T, Hv, D, dtype=torch.float64, device=DEV)
    for t in range(T):
        S = S * decay[t][:, None, None]
        u = (v[t] - torch.einsum("hk,hkv->hv", k[t], S)) * beta[t][:, None]
        S = S + k[t][:, :, None] * u[:, None]
        want[t] = torch.einsum("hk,hkv->hv", q[t], S) * D ** -0.5

    def rel(x, y):
        return float((x.double() - y).norm() / y.norm())
    # decays from the fast exponential and logarithm (2^-21 a token, a memory of some hundred tokens): about 1e-6
    assert rel(got_rec[0], S) < 1e-5
    assert rel(got, want) < 2.5e-3                           # bf16 outputs: 2^-9 at most, 2^-9 / sqrt(3) in the norm
