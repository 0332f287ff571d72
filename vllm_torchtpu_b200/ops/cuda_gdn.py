"""Bindings of the Gated DeltaNet kernels."""
from __future__ import annotations

from ctypes import c_int

import torch

from . import count_launch
from . import cuda as _c


CHUNK_WORDS = 128 * 64 + 4 * 64           # scratch of a (chunk, head) in gdn_chunk.cu
MOST_WORDS = 1 << 28                      # most that a call takes for them (1 GB)


def chunk_words(T: int, R: int, Hv: int) -> int:
    return (T // 64 + R) * Hv * CHUNK_WORDS


def chunk_scratch_bytes(max_tokens: int, max_reqs: int, Hv: int) -> int:
    """Most that ``gdn_forward`` takes for its chunks in a step."""
    return 4 * min(MOST_WORDS, chunk_words(max_tokens, max_reqs, Hv))


def _rows(R: int, *shape, device):
    """Output rows; the kernels write all of them, zeros where there is no request, unless there is none at all."""
    return (torch.empty if R > 0 else torch.zeros)(shape, dtype=torch.bfloat16, device=device)


def gdn_forward(mixed, a, b, meta, conv_pool, rec_pool, conv_w, A_log, dt_bias, Hk, Hv, dk, dv):
    """mixed [T, 2*Hk*dk + Hv*dv] bf16 (may be a column slice), a/b [T, Hv] -> o [T, Hv, dv]."""
    _c._require_bf16(mixed, a, b, conv_w)
    T, C = mixed.shape
    dev = mixed.device
    R = meta.padded_num_reqs if meta.padded_num_reqs is not None else meta.num_reqs
    def new(*shape, dtype=torch.float32):
        return torch.empty(shape, dtype=dtype, device=dev)
    out = _rows(R, T, Hv, dv, device=dev)
    conv_out = qn = kn = g = beta = chunks = None
    # single tokens have their own kernel, which reads weights in pieces of 8 bytes and states in pieces of 16
    step = dk == dv == 128 and conv_w.data_ptr() % 8 == 0 and rec_pool.data_ptr() % 16 == 0
    if not step or T > R:
        conv_out = new(T, C, dtype=torch.bfloat16)
        # Chunks of 64 tokens on the tensor cores, or token by token: a token costs about 0.7 us there, a request's chunk
        # about 8 us with the work in front of it.  A wrong length costs time only.
        longest = meta.max_query_len if meta.max_query_len > 1 else T - R + 1
        words = chunk_words(T, R, Hv)
        if step and longest > 16 and words <= MOST_WORDS:
            chunks = new(words)
        else:
            qn, kn, g, beta = new(T, Hk, dk), new(T, Hk, dk), new(T, Hv), new(T, Hv)
    _c._check(_c.lib().b200_gdn_forward(
        _c._p(mixed), c_int(mixed.stride(0)), _c._p(a), _c._p(b), c_int(a.stride(0)), _c._p(conv_w),
        _c._p(A_log), _c._p(dt_bias), _c._p(conv_pool), _c._p(rec_pool), _c._p(conv_out), _c._p(qn), _c._p(kn),
        _c._p(g), _c._p(beta), _c._p(chunks), _c._p(out), _c._p(meta.query_start_loc), _c._p(meta.seq_lens),
        _c._p(meta.state_slots), c_int(R), c_int(T), c_int(Hk), c_int(Hv), c_int(dk), c_int(dv),
        c_int(conv_w.shape[1]), _c._p(_c.Workspace.get(dev).status), _c._stream()), "gdn_forward")
    count_launch((4 if step else 3) if conv_out is not None else 1)
    return out


def kda_forward(q, k, v, a, b, meta, rec_pool, A_log, dt_bias, lower_bound=None):
    """Kimi Delta Attention (per-channel decay).  q, k [T, Hk, dk], v [T, Hv, dv], a [T, Hv, dk], b [T, Hv]
    bf16; A_log [Hv], dt_bias [Hv, dk] fp32; rec_pool [slots, Hv, dk, dv] fp32 -> o [T, Hv, dv]."""
    from ctypes import c_float
    _c._require_bf16(q, k, v, a, b)
    # heads side by side; the tokens of q, k and v may lie apart (columns of one projection)
    q, k, v = (t if t.stride(2) == 1 and t.stride(1) == t.shape[2] else t.contiguous() for t in (q, k, v))
    a, b = a.contiguous(), b.contiguous()
    T, Hk, dk = q.shape
    Hv, dv = v.shape[1], v.shape[2]
    dev = q.device
    R = meta.padded_num_reqs if meta.padded_num_reqs is not None else meta.num_reqs
    qn = torch.empty((T, Hk, dk), dtype=torch.float32, device=dev)
    kn = torch.empty_like(qn)
    g = torch.empty((T, Hv, dk), dtype=torch.float32, device=dev)
    beta = torch.empty((T, Hv), dtype=torch.float32, device=dev)
    out = _rows(R, T, Hv, dv, device=dev)
    A_log = A_log.float().contiguous()
    dt_bias = dt_bias.float().contiguous()
    lb = float(lower_bound) if lower_bound is not None else 0.0
    _c._check(_c.lib().b200_kda_forward(
        _c._p(q), _c._p(k), _c._p(v), c_int(q.stride(0)), c_int(k.stride(0)), c_int(v.stride(0)), _c._p(a), _c._p(b),
        _c._p(A_log), _c._p(dt_bias), c_float(lb),
        _c._p(rec_pool), _c._p(qn), _c._p(kn), _c._p(g), _c._p(beta), _c._p(out), _c._p(meta.query_start_loc),
        _c._p(meta.seq_lens), _c._p(meta.state_slots), c_int(R), c_int(T), c_int(Hk), c_int(Hv), c_int(dk),
        c_int(dv), _c._stream()), "kda_forward")
    count_launch(2)
    return out


def short_conv(x, meta, conv_pool, conv_w):
    """Causal depth-wise conv (kernel 4) + SiLU with the carried window; x [T, C] bf16 (row stride free)."""
    _c._require_bf16(x, conv_w)
    T, C = x.shape
    R = meta.padded_num_reqs if meta.padded_num_reqs is not None else meta.num_reqs
    y = _rows(R, T, C, device=x.device)
    _c._check(_c.lib().b200_short_conv(
        _c._p(x), c_int(x.stride(0)), _c._p(conv_w), _c._p(conv_pool), _c._p(y), _c._p(meta.query_start_loc),
        _c._p(meta.seq_lens), _c._p(meta.state_slots), c_int(R), c_int(T), c_int(C), c_int(conv_w.shape[1]), _c._stream()),
        "short_conv")
    count_launch()
    return y
