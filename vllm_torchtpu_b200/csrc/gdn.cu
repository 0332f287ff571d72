// Gated DeltaNet kernels: causal depth-wise conv1d with a carried window, gate/normalisation
// prep, and the gated delta-rule recurrence with the per-head state held in registers.
//
// Heads of 128 / 128: single tokens take delta_step_kernel (everything in one launch), longer portions of the scalar rule
// the chunks of gdn_chunk.cu.  Other portions, head sizes and the channel rule take the recurrence: one CTA per
// (request, value head, 64 columns of the [dk, dv] state), the request's tokens in order; columns are independent of each
// other.  State lives in pools indexed by the request's slot; a request whose first token of the step has position 0
// starts from zero.
//
// Math of the reference's fused conv1d + GDN kernels (reference: src/vllm_torchtpu/kernels/gdn/v3/),
// which use a chunked WY form for prefill; the recurrence below is the same function.
#include "common.cuh"

namespace b200 {

constexpr int CONV_ROWS = 32;        // tokens of a request per CTA of the convolution

// Values of VEC neighbouring channels
template <int VEC>
struct Row;
template <>
struct Row<1> {
  __nv_bfloat16 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *p; }
  __device__ __forceinline__ void store(__nv_bfloat16* p) const { *p = v; }
  __device__ __forceinline__ float get(int) const { return __bfloat162float(v); }
  __device__ __forceinline__ void set(const float (&f)[1]) { v = __float2bfloat16(f[0]); }
};
template <>
struct Row<8> {
  __align__(16) __nv_bfloat16 v[8];
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void store(__nv_bfloat16* p) const { *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(v); }
  __device__ __forceinline__ float get(int i) const { return __bfloat162float(v[i]); }
  __device__ __forceinline__ void set(const float (&f)[8]) {      // (two conversions at a time)
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<__nv_bfloat162*>(v)[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  }
};

// x [T, C] bf16 -> y [T, C] bf16 (convolution of 4 taps, then SiLU).  grid (ceil(C / (128 VEC)), T / 32 + R): a CTA takes up
// to 32 tokens of one request and 128 * VEC channels, with the three tokens in front of them.  Bound by memory: one read
// and one write of the rows; eight rows of a thread are in flight.  Only the CTA of a request's first tokens touches
// the carried window: it reads the old one and writes the new one.  Rows of no request become zeros.
// 4 x 2048 tokens and 8192 channels take 100 us (2.7 TB/s): the next eight rows are loaded only once the present ones are
// stored, and every CTA begins with a search, its weights and a halo.  (The division is IEEE's: 3 us of the 100.)  One
// thread per channel through all tokens of a request had one load in flight.
template <int VEC>
__global__ void __launch_bounds__(128)
gdn_conv_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, __nv_bfloat16* conv_pool,
                const __nv_bfloat16* __restrict__ w, const int* __restrict__ qsl, const int* __restrict__ seq_lens,
                const int* __restrict__ slots, int R, int T, int C, int ldx, int skip_single) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, c = (blockIdx.x * 128 + threadIdx.x) * VEC;
  int r = -1, chunk = blockIdx.y;
  for (int b = 0; b < R; b += 32) {
    const int n = b + lane < R ? (max(0, qsl[b + lane + 1] - qsl[b + lane]) + CONV_ROWS - 1) / CONV_ROWS : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int sum = __shfl_sync(0xffffffffu, incl, 31);
    if (chunk < sum) {
      const int src = __ffs(__ballot_sync(0xffffffffu, incl > chunk)) - 1;
      r = b + src;
      chunk -= __shfl_sync(0xffffffffu, incl - n, src);
      break;
    }
    chunk -= sum;
  }
  if (c >= C) return;
  Row<VEC> zero;
  const float nothing[VEC] = {};
  zero.set(nothing);
  for (int t = max(0, qsl[R]) + blockIdx.y; t < T; t += gridDim.y) zero.store(y + (size_t)t * C + c);
  if (r < 0) return;
  const int qs = qsl[r], len = qsl[r + 1] - qs, t0 = chunk * CONV_ROWS, t1 = min(len, t0 + CONV_ROWS);
  if (skip_single && len == 1) return;
  const int slot = slots[r];
  if (slot < 0) {
    for (int t = t0; t < t1; ++t) zero.store(y + (size_t)(qs + t) * C + c);
    return;
  }
  x += (size_t)qs * ldx + c;
  y += (size_t)qs * C + c;
  float win[3][VEC], wt[4][VEC];
  __nv_bfloat16* st = conv_pool + ((size_t)slot * C + c) * 3;
  {
    __align__(16) __nv_bfloat16 raw[4 * VEC];
    if constexpr (VEC == 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) reinterpret_cast<uint4*>(raw)[i] = reinterpret_cast<const uint4*>(w + (size_t)c * 4)[i];
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) raw[i] = w[(size_t)c * 4 + i];
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
#pragma unroll
      for (int j = 0; j < 4; ++j) wt[j][e] = __bfloat162float(raw[4 * e + j]);
    }
  }
  if (t0 == 0) {
    const bool fresh = seq_lens[r] == len;
    __align__(16) __nv_bfloat16 raw[3 * VEC];
    if constexpr (VEC == 8) {
#pragma unroll
      for (int i = 0; i < 3; ++i) reinterpret_cast<uint4*>(raw)[i] = reinterpret_cast<const uint4*>(st)[i];
    } else {
#pragma unroll
      for (int i = 0; i < 3; ++i) raw[i] = st[i];
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
#pragma unroll
      for (int j = 0; j < 3; ++j) win[j][e] = fresh ? 0.f : __bfloat162float(raw[3 * e + j]);
    }
    // the window behind the last token
    Row<VEC> last[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) last[j].load(x + (size_t)max(0, len - 3 + j) * ldx);
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int from = len - 3 + j;      // < 0: of the old window
        raw[3 * e + j] = __float2bfloat16(from >= 0 ? last[j].get(e) : (from == -1 ? win[2][e] : win[1][e]));
      }
    }
    if constexpr (VEC == 8) {
#pragma unroll
      for (int i = 0; i < 3; ++i) reinterpret_cast<uint4*>(st)[i] = reinterpret_cast<const uint4*>(raw)[i];
    } else {
#pragma unroll
      for (int i = 0; i < 3; ++i) st[i] = raw[i];
    }
  } else {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      Row<VEC> v;
      v.load(x + (size_t)(t0 - 3 + j) * ldx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) win[j][e] = v.get(e);
    }
  }
  constexpr int NB = 8;
  for (int t = t0; t < t1; t += NB) {
    Row<VEC> in[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) in[i].load(x + (size_t)min(t + i, t1 - 1) * ldx);
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      if (t + i >= t1) break;
      float o[VEC];
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float v = in[i].get(e);
        float acc = win[0][e] * wt[0][e];
        acc += win[1][e] * wt[1][e];
        acc += win[2][e] * wt[2][e];
        acc += v * wt[3][e];
        o[e] = acc / (1.f + __expf(-acc));
        win[0][e] = win[1][e];
        win[1][e] = win[2][e];
        win[2][e] = v;
      }
      Row<VEC> out;
      out.set(o);
      out.store(y + (size_t)(t + i) * C);
    }
  }
}

static int launch_conv(const void* x, void* y, void* pool, const void* w, const int* qsl, const int* seq_lens,
                       const int* slots, int R, int T, int C, int ldx, int skip_single, cudaStream_t stream) {
  // 16 bytes a thread where the rows allow it; single channels otherwise
  const bool vec = C % 8 == 0 && ldx % 8 == 0 && (((uintptr_t)x | (uintptr_t)y | (uintptr_t)w | (uintptr_t)pool) & 15) == 0;
  const int per = 128 * (vec ? 8 : 1);
  const dim3 grid((C + per - 1) / per, T / CONV_ROWS + R);
  if (grid.y > 65535) {
    b200_set_last_error("short convolution: too many tokens", __FILE__, __LINE__);
    return -1;
  }
  B200_CUDA_CHECK(launch_pdl(vec ? gdn_conv_kernel<8> : gdn_conv_kernel<1>, grid, dim3(128), (size_t)0, stream,
                             (const __nv_bfloat16*)x, (__nv_bfloat16*)y, (__nv_bfloat16*)pool, (const __nv_bfloat16*)w, qsl,
                             seq_lens, slots, R, T, C, ldx, skip_single));
  return 0;
}

// One warp per (token, k head): L2-normalise q and k (q also scaled by dk^-1/2) into fp32;
// one thread per (token, v head): g = exp(-exp(A_log) * softplus(a + dt_bias)), beta = sigmoid(b).
__global__ void gdn_prep_kernel(const __nv_bfloat16* __restrict__ conv_out, const __nv_bfloat16* __restrict__ a,
                                const __nv_bfloat16* __restrict__ b, const float* __restrict__ A_log,
                                const float* __restrict__ dt_bias, float* __restrict__ qn,
                                float* __restrict__ kn, float* __restrict__ g, float* __restrict__ beta, int T,
                                int Hk, int Hv, int dk, int C, int lda) {
  pdl_wait();              // (no early launch of the recurrence: its CTAs would pile up on the SMs that are free first)
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int total = T * Hk;
  if (warp < total) {
    const int t = warp / Hk, h = warp % Hk;
    const __nv_bfloat16* qp = conv_out + (size_t)t * C + h * dk;
    const __nv_bfloat16* kp = conv_out + (size_t)t * C + Hk * dk + h * dk;
    float sq = 0.f, sk = 0.f;
    for (int i = lane; i < dk; i += 32) {
      const float qv = __bfloat162float(qp[i]), kv = __bfloat162float(kp[i]);
      sq += qv * qv;
      sk += kv * kv;
    }
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    const float iq = rsqrtf((float)dk) / fmaxf(sqrtf(sq), 1e-12f), ik = 1.f / fmaxf(sqrtf(sk), 1e-12f);
    for (int i = lane; i < dk; i += 32) {
      qn[((size_t)t * Hk + h) * dk + i] = __bfloat162float(qp[i]) * iq;
      kn[((size_t)t * Hk + h) * dk + i] = __bfloat162float(kp[i]) * ik;
    }
  }
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < T * Hv) {
    const int t = idx / Hv, h = idx % Hv;
    const float av = __bfloat162float(a[(size_t)t * lda + h]) + dt_bias[h];
    const float sp = av > 20.f ? av : log1pf(__expf(av));
    g[idx] = __expf(-__expf(A_log[h]) * sp);
    beta[idx] = 1.f / (1.f + __expf(-__bfloat162float(b[(size_t)t * lda + h])));
  }
}

// two fp32 numbers per register pair: one issue slot for two multiply-adds
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pair2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float add_halves(uint64_t v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void copy4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

constexpr int REC_COLS = 64;         // state columns per CTA

// grid (ceil(dv / 64), Hv, R), 32 threads * (DK / 32): S <- g S;  u = (v - k^T S) beta;  S <- S + k u^T;  o = q^T S.
// KDA (Kimi Delta Attention, reference: src/vllm_torchtpu/kernels/gdn/v3/compute_kda.py:362-423): the decay g is
// per key channel, [T, Hv, DK], instead of one scalar per (token, head); v_base is the column of the
// first value head inside a row of conv_out (row length C).
//
// What bounds it: 3 (4 with KDA) multiply-adds per state element and token, one token behind the other.  A thread owns
// two columns x 32 rows of the state in 64 registers, DK / 32 neighbouring lanes a column, so every q and k value that
// it reads from shared memory feeds two columns, and both dot products are formed on the old state (o = q^T S + (q k) u)
// and reduced together.  Rows go in groups of four to the lanes in turn: reads of 16 bytes without bank conflicts, and
// pairs of rows for the two-wide multiply-adds.  q, k, v, g and beta of the next tokens arrive by asynchronous copies while
// the 16 (KDA: 8) before them are worked on: the loop has no global load in its chain.
template <int DK, bool KDA>
__global__ void __launch_bounds__(DK)
gdn_recurrent_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
                     const __nv_bfloat16* __restrict__ conv_out, const float* __restrict__ g,
                     const float* __restrict__ beta, float* __restrict__ rec_pool,
                     __nv_bfloat16* __restrict__ out, const int* __restrict__ qsl,
                     const int* __restrict__ seq_lens, const int* __restrict__ slots, int R, int T, int Hk, int Hv, int dv,
                     int C, int v_base, int skip_single) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int PARTS = DK / 32, NB = KDA ? 8 : 16;        // tokens staged at a time
  __shared__ __align__(16) float sk[2][NB][DK], sq[2][NB][DK];
  __shared__ __align__(16) float sd[2][NB][KDA ? DK : 4];
  __shared__ __align__(16) __nv_bfloat16 sv[2][NB][REC_COLS];
  __shared__ float sb[2][NB], sqk[2][NB];
  const int hv = blockIdx.y, r = blockIdx.z, tid = threadIdx.x, c0 = blockIdx.x * REC_COLS;
  const int part = tid % PARTS, cp = tid / PARTS, j = c0 + 2 * cp;
  const bool act0 = j < dv, act1 = j + 1 < dv;
  const int qs = qsl[r], n = qsl[r + 1] - qs, slot = slots[r];
  // rows of no request, and of requests without a state, are zeros
  auto zero = [&](int t) {
    if (part == 0 && act0) {
      out[((size_t)t * Hv + hv) * dv + j] = __float2bfloat16(0.f);
      if (act1) out[((size_t)t * Hv + hv) * dv + j + 1] = __float2bfloat16(0.f);
    }
  };
  for (int t = max(0, qsl[R]) + r; t < T; t += R) zero(t);
  if (n <= 0 || (skip_single && n == 1)) return;
  if (slot < 0) {
    for (int t = qs; t < qs + n; ++t) zero(t);
    return;
  }
  const int hk = hv / (Hv / Hk);
  const bool v16 = (((uintptr_t)conv_out & 15) | (C & 7) | ((v_base + hv * dv) & 7) | (dv & 7)) == 0;
  auto stage = [&](int t0, int buf) {
    const int m = min(NB, n - t0);
    for (int i = tid; i < m * (DK / 4); i += DK) {
      const int t = i / (DK / 4), x = i % (DK / 4) * 4;
      const size_t row = (size_t)(qs + t0 + t);
      copy16(&sk[buf][t][x], kn + (row * Hk + hk) * DK + x);
      copy16(&sq[buf][t][x], qn + (row * Hk + hk) * DK + x);
      if constexpr (KDA) copy16(&sd[buf][t][x], g + (row * Hv + hv) * DK + x);
    }
    const __nv_bfloat16* v = conv_out + (size_t)(qs + t0) * C + v_base + hv * dv + c0;
    if (v16) {
      for (int i = tid; i < m * (REC_COLS / 8); i += DK) {
        const int t = i / (REC_COLS / 8), x = i % (REC_COLS / 8) * 8;
        if (c0 + x < dv) copy16(&sv[buf][t][x], v + (size_t)t * C + x);
      }
    } else {
      for (int i = tid; i < m * REC_COLS; i += DK) {
        const int t = i / REC_COLS, x = i % REC_COLS;
        if (c0 + x < dv) sv[buf][t][x] = v[(size_t)t * C + x];
      }
    }
    for (int t = tid; t < m; t += DK) {
      copy4(&sb[buf][t], beta + (size_t)(qs + t0 + t) * Hv + hv);
      if constexpr (!KDA) copy4(&sd[buf][t][0], g + (size_t)(qs + t0 + t) * Hv + hv);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0, 0);
  // S[c][2 x], S[c][2 x + 1]: rows 4 (PARTS x + part) + 0 .. 3 of column j + c
  uint64_t S[2][16];
  float* sp = rec_pool + (((size_t)slot * Hv + hv) * DK + 4 * part) * dv + j;
  const bool fresh = seq_lens[r] == n, wide = (dv & 1) == 0 && ((uintptr_t)rec_pool & 7) == 0;
  if (fresh || !act0) {
#pragma unroll
    for (int x = 0; x < 16; ++x) S[0][x] = S[1][x] = 0ull;
  } else {
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      float2 a, b;
      const float* s = sp + (size_t)(4 * PARTS * (x >> 1) + 2 * (x & 1)) * dv;
      if (wide) {
        a = *reinterpret_cast<const float2*>(s);
        b = *reinterpret_cast<const float2*>(s + dv);
      } else {
        a = make_float2(s[0], act1 ? s[1] : 0.f);
        b = make_float2(s[dv], act1 ? s[dv + 1] : 0.f);
      }
      S[0][x] = pair2(a.x, b.x);
      S[1][x] = pair2(a.y, b.y);
    }
  }
  // scalar decay: the registers hold S / D, D the product of the decays so far
  float D = 1.f;
  for (int t0 = 0, buf = 0; t0 < n; t0 += NB, buf ^= 1) {
    if (t0 + NB < n) {
      stage(t0 + NB, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    // q k of the staged tokens: PARTS lanes a token
    const int m = min(NB, n - t0);
    for (int t = cp; t - cp < NB; t += DK / PARTS) {  // (every lane takes part in the shuffles)
      float s = 0.f;
      if (t < m)
        for (int x = part; x < DK; x += PARTS) s = fmaf(sk[buf][t][x], sq[buf][t][x], s);
      if constexpr (PARTS >= 2) s += __shfl_xor_sync(0xffffffffu, s, 1);
      if constexpr (PARTS == 4) s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (part == 0 && t < NB) sqk[buf][t] = s;
    }
    __syncthreads();
    for (int t = 0; t < m; ++t) {
      uint64_t k[16], m2[2][2] = {{0ull, 0ull}, {0ull, 0ull}}, o2[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
#pragma unroll
      for (int x = 0; x < 16; x += 2) {
        const int row = 2 * PARTS * x + 4 * part;
        const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(&sk[buf][t][row]);
        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(&sq[buf][t][row]);
        k[x] = kv.x;
        k[x + 1] = kv.y;
        if constexpr (KDA) {
          const ulonglong2 dv2 = *reinterpret_cast<const ulonglong2*>(&sd[buf][t][row]);
          S[0][x] = mul2(S[0][x], dv2.x); S[0][x + 1] = mul2(S[0][x + 1], dv2.y);
          S[1][x] = mul2(S[1][x], dv2.x); S[1][x + 1] = mul2(S[1][x + 1], dv2.y);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          m2[c][0] = fma2(kv.x, S[c][x], m2[c][0]);
          m2[c][1] = fma2(kv.y, S[c][x + 1], m2[c][1]);
          o2[c][0] = fma2(qv.x, S[c][x], o2[c][0]);
          o2[c][1] = fma2(qv.y, S[c][x + 1], o2[c][1]);
        }
      }
      float mem[2], o[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        mem[c] = add_halves(m2[c][0]) + add_halves(m2[c][1]);
        o[c] = add_halves(o2[c][0]) + add_halves(o2[c][1]);
        if constexpr (PARTS >= 2) {
          mem[c] += __shfl_xor_sync(0xffffffffu, mem[c], 1);
          o[c] += __shfl_xor_sync(0xffffffffu, o[c], 1);
        }
        if constexpr (PARTS == 4) {
          mem[c] += __shfl_xor_sync(0xffffffffu, mem[c], 2);
          o[c] += __shfl_xor_sync(0xffffffffu, o[c], 2);
        }
      }
      float scale = 1.f;
      if constexpr (!KDA) {
        D *= sd[buf][t][0];
        if (D < 1e-10f) {                  // (the same for the whole CTA) back to D = 1; a decay of zero included
          const uint64_t d = pair2(D, D);
#pragma unroll
          for (int x = 0; x < 16; ++x) { S[0][x] = mul2(S[0][x], d); S[1][x] = mul2(S[1][x], d); }
#pragma unroll
          for (int c = 0; c < 2; ++c) { mem[c] *= D; o[c] *= D; }
          D = 1.f;
        } else {
#pragma unroll
          for (int c = 0; c < 2; ++c) { mem[c] *= D; o[c] *= D; }
          scale = __frcp_rn(D);
        }
      }
      const float bt = sb[buf][t], qk = sqk[buf][t];
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&sv[buf][t][2 * cp]);
      const float u0 = (__low2float(v) - mem[0]) * bt, u1 = act1 ? (__high2float(v) - mem[1]) * bt : 0.f;
      const uint64_t w0 = pair2(u0 * scale, u0 * scale), w1 = pair2(u1 * scale, u1 * scale);
#pragma unroll
      for (int x = 0; x < 16; ++x) {
        S[0][x] = fma2(k[x], w0, S[0][x]);
        S[1][x] = fma2(k[x], w1, S[1][x]);
      }
      if (part == 0 && act0) {
        __nv_bfloat16* d = out + ((size_t)(qs + t0 + t) * Hv + hv) * dv + j;
        const float a = fmaf(qk, u0, o[0]), b = fmaf(qk, u1, o[1]);
        if (wide) {
          *reinterpret_cast<__nv_bfloat162*>(d) = __floats2bfloat162_rn(a, b);
        } else {
          d[0] = __float2bfloat16(a);
          if (act1) d[1] = __float2bfloat16(b);
        }
      }
    }
    __syncthreads();
  }
  if (!act0) return;
  const uint64_t d = pair2(D, D);
#pragma unroll
  for (int x = 0; x < 16; ++x) {
    if constexpr (!KDA) { S[0][x] = mul2(S[0][x], d); S[1][x] = mul2(S[1][x], d); }
    float2 a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(b.x) : "l"(S[0][x]));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.y), "=f"(b.y) : "l"(S[1][x]));
    float* s = sp + (size_t)(4 * PARTS * (x >> 1) + 2 * (x & 1)) * dv;
    if (wide) {
      *reinterpret_cast<float2*>(s) = a;
      *reinterpret_cast<float2*>(s + dv) = b;
    } else {
      s[0] = a.x;
      s[dv] = b.x;
      if (act1) { s[1] = a.y; s[dv + 1] = b.y; }
    }
  }
}

template <bool KDA>
static int launch_recurrence(const float* qn, const float* kn, const void* v, const float* g, const float* beta,
                             float* rec_pool, void* out, const int* qsl, const int* seq_lens, const int* slots, int R, int T,
                             int Hk, int Hv, int dk, int dv, int C, int v_base, int skip_single, cudaStream_t stream) {
  const dim3 grid((dv + REC_COLS - 1) / REC_COLS, Hv, R);
  if (R > 65535 || Hv > 65535) {
    b200_set_last_error("delta rule: too many requests or heads", __FILE__, __LINE__);
    return -1;
  }
#define REC(DKV)                                                                                                           \
  B200_CUDA_CHECK(launch_pdl(gdn_recurrent_kernel<DKV, KDA>, grid, dim3(DKV), (size_t)0, stream, qn, kn,                   \
                             (const __nv_bfloat16*)v, g, beta, rec_pool, (__nv_bfloat16*)out, qsl, seq_lens, slots, R, T,  \
                             Hk, Hv, dv, C, v_base, skip_single))
  if (dk == 128) REC(128);
  else if (dk == 64) REC(64);
  else REC(32);
#undef REC
  return 0;
}

// Requests of one token, heads of 128 / 128: everything in one kernel.  grid (Hk, R), 256 threads: a CTA takes the value
// heads of one key head in turn, so the convolution's channels and their windows have one owner each.  Bound by memory:
// the state is read and written once (64 KB a head).  A warp holds 16 rows of 128 columns (512 bytes a load), all of
// its loads are under way before the convolution; the column sums of the eight warps meet in shared memory.
// KDA: q, k, v are given (token strides ldq, ldk, ldv).  single: only requests of one token; otherwise tokens in order.
struct StepParams {
  const __nv_bfloat16 *x, *w, *q, *k, *v, *a, *b;
  __nv_bfloat16 *pool, *out;
  const float *A_log, *dt_bias;
  float* rec;
  const int *qsl, *seq_lens, *slots;
  int R, T, Hk, Hv, ldx, ldq, ldk, ldv, lda, single;
  float lower_bound;
};
template <bool KDA>
__global__ void __launch_bounds__(256, 2) delta_step_kernel(const StepParams p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int D = 128;
  __shared__ __align__(16) float raw[2 * D], sq[D], sk[D], sd[D], su[D], red[12];
  __shared__ __align__(16) float pm[8][D], po[8][D];
  const int hk = blockIdx.x, r = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = p.Hv / p.Hk, C = (2 * p.Hk + p.Hv) * D;
  const int qs = p.qsl[r], n = p.qsl[r + 1] - qs, slot = p.slots[r];
  auto zero = [&](int t) {
    for (int i = tid; i < G * D; i += 256) p.out[((size_t)t * p.Hv + hk * G) * D + i] = __float2bfloat16(0.f);
  };
  for (int t = max(0, p.qsl[p.R]) + r; t < p.T; t += p.R) zero(t);
  if (n <= 0 || (p.single && n != 1)) return;
  if (slot < 0) {
    for (int t = qs; t < qs + n; ++t) zero(t);
    return;
  }
  const bool fresh = p.seq_lens[r] == n;
  // convolution of channel c at token t of the request, rounded as the convolution kernel does
  auto conv = [&](int t, int c) -> float {
    const __nv_bfloat16* x = p.x + (size_t)qs * p.ldx + c;
    const __nv_bfloat16* st = p.pool + ((size_t)slot * C + c) * 3;
    const uint2 wr = *reinterpret_cast<const uint2*>(p.w + (size_t)c * 4);
    const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(&wr);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int from = t - 3 + j;
      const float v = from >= 0 ? __bfloat162float(x[(size_t)from * p.ldx]) : (fresh ? 0.f : __bfloat162float(st[from + 3]));
      acc += v * __bfloat162float(w[j]);
    }
    return __bfloat162float(__float2bfloat16(acc / (1.f + __expf(-acc))));
  };
  for (int g = 0; g < G; ++g) {
    const int hv = hk * G + g;
    float* st = p.rec + (((size_t)slot * p.Hv + hv) * D + 16 * warp) * D + 4 * lane;
    float4 S[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) S[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!fresh) {
#pragma unroll
      for (int i = 0; i < 16; ++i) S[i] = *reinterpret_cast<const float4*>(st + (size_t)i * D);
    }
    const float ea = __expf(p.A_log[hv]);
    for (int t = 0; t < n; ++t) {
      const size_t row = qs + t;
      float x, v = 0.f, decay = 1.f;
      if constexpr (KDA) {
        x = __bfloat162float(tid < D ? p.q[row * p.ldq + hk * D + tid] : p.k[row * p.ldk + hk * D + tid - D]);
        if (tid < D) {
          v = __bfloat162float(p.v[row * p.ldv + hv * D + tid]);
          const float z = __bfloat162float(p.a[(row * p.Hv + hv) * D + tid]) + p.dt_bias[hv * D + tid];
          sd[tid] = __expf(p.lower_bound < 0.f ? p.lower_bound / (1.f + __expf(-ea * z))
                                               : -ea * (z > 20.f ? z : log1pf(__expf(z))));
        }
      } else {
        x = conv(t, (tid < D ? 0 : p.Hk * D - D) + hk * D + tid);
        if (tid < D) v = conv(t, (2 * p.Hk + hv) * D + tid);
        const float z = __bfloat162float(p.a[row * p.lda + hv]) + p.dt_bias[hv];
        decay = __expf(-ea * (z > 20.f ? z : log1pf(__expf(z))));
      }
      const float beta = 1.f / (1.f + __expf(-__bfloat162float(p.b[KDA ? row * p.Hv + hv : row * p.lda + hv])));
      raw[tid] = x;
      const float s = warp_sum(x * x);
      if (lane == 0) red[warp] = s;
      __syncthreads();
      if (tid < D) {
        const float s2q = red[0] + red[1] + red[2] + red[3], s2k = red[4] + red[5] + red[6] + red[7];
        const float iq = rsqrtf((float)D) * (KDA ? rsqrtf(s2q + 1e-6f) : 1.f / fmaxf(sqrtf(s2q), 1e-12f));
        const float ik = KDA ? rsqrtf(s2k + 1e-6f) : 1.f / fmaxf(sqrtf(s2k), 1e-12f);
        const float qv = x * iq, kv = raw[D + tid] * ik;
        sq[tid] = qv;
        sk[tid] = kv;
        const float d = warp_sum(qv * kv);
        if (lane == 0) red[8 + warp] = d;
      }
      __syncthreads();
      float4 m = make_float4(0.f, 0.f, 0.f, 0.f), o = m;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float kk = sk[16 * warp + i], qq = sq[16 * warp + i], dd = KDA ? sd[16 * warp + i] : decay;
        S[i].x *= dd; S[i].y *= dd; S[i].z *= dd; S[i].w *= dd;
        m.x = fmaf(kk, S[i].x, m.x); m.y = fmaf(kk, S[i].y, m.y); m.z = fmaf(kk, S[i].z, m.z); m.w = fmaf(kk, S[i].w, m.w);
        o.x = fmaf(qq, S[i].x, o.x); o.y = fmaf(qq, S[i].y, o.y); o.z = fmaf(qq, S[i].z, o.z); o.w = fmaf(qq, S[i].w, o.w);
      }
      *reinterpret_cast<float4*>(&pm[warp][4 * lane]) = m;
      *reinterpret_cast<float4*>(&po[warp][4 * lane]) = o;
      __syncthreads();
      if (tid < D) {
        float mem = 0.f, ov = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          mem += pm[i][tid];
          ov += po[i][tid];
        }
        const float u = (v - mem) * beta;
        su[tid] = u;
        p.out[(row * p.Hv + hv) * D + tid] = __float2bfloat16(fmaf(red[8] + red[9] + red[10] + red[11], u, ov));
      }
      __syncthreads();
      const float4 u = *reinterpret_cast<const float4*>(&su[4 * lane]);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float kk = sk[16 * warp + i];
        S[i].x = fmaf(kk, u.x, S[i].x); S[i].y = fmaf(kk, u.y, S[i].y); S[i].z = fmaf(kk, u.z, S[i].z); S[i].w = fmaf(kk, u.w, S[i].w);
      }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) *reinterpret_cast<float4*>(st + (size_t)i * D) = S[i];
  }
  if constexpr (!KDA) {
    __syncthreads();                      // every window of this CTA's channels has been read
    for (int i = tid; i < (2 + G) * D; i += 256) {
      const int c = i < D ? hk * D + i : (i < 2 * D ? (p.Hk + hk - 1) * D + i : (2 * p.Hk + hk * G - 2) * D + i);
      const __nv_bfloat16* x = p.x + (size_t)qs * p.ldx + c;
      __nv_bfloat16* w = p.pool + ((size_t)slot * C + c) * 3;
      __nv_bfloat16 v[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int from = n - 3 + j;
        v[j] = from >= 0 ? x[(size_t)from * p.ldx] : (fresh ? __float2bfloat16(0.f) : w[from + 3]);
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) w[j] = v[j];
    }
  }
}

// The step kernel (and the chunks) read states in pieces of 16 bytes and the convolution's weights in pieces of 8.
static bool step_takes(int dk, int dv, int R, const void* w, const void* rec) {
  return dk == 128 && dv == 128 && R <= 65535 && !((uintptr_t)w & 7) && !((uintptr_t)rec & 15);
}

// 0: the step kernel took every request; 1: those of one token (or none), the others are still to be done; < 0: error
template <bool KDA>
static int launch_step(StepParams p, int dk, int dv, cudaStream_t stream) {
  if (!step_takes(dk, dv, p.R, p.w, p.rec)) return 1;
  // no more tokens than requests: a step of single tokens (should one have more, its tokens go one after the other).  Else
  // single tokens beside prompts: the chunks of the prompt kernels would be nearly empty for them.
  p.single = p.T > p.R;
  cudaError_t e = launch_pdl(delta_step_kernel<KDA>, dim3(p.Hk, p.R), dim3(256), (size_t)0, stream, p);
  if (e != cudaSuccess) {
    b200_set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
    return -1;
  }
  return p.single;
}

}  // namespace b200

using namespace b200;

extern "C" int b200_gdn_chunks(const void* y, int Cy, const void* a, const void* b, int lda, const float* A_log,
                               const float* dt_bias, float* rec_pool, void* out, float* scratch, const int* qsl,
                               const int* seq_lens, const int* slots, int R, int T, int Hk, int Hv, int* status,
                               cudaStream_t stream);

// mixed [T, C] (C = 2*Hk*dk + Hv*dv, row stride ldx), a/b [T, Hv] (row stride lda).
// scratch of the caller: conv_out [T, C] bf16; qn/kn [T, Hk, dk] fp32 and g/beta [T, Hv] fp32, or (heads of 128 / 128) the
// chunks' (gdn_chunk.cu), which selects that path.  With heads of 128 / 128 and T <= R none is used.
extern "C" int b200_gdn_forward(const void* mixed, int ldx, const void* a, const void* b, int lda,
                                const void* conv_w, const float* A_log, const float* dt_bias, void* conv_pool,
                                float* rec_pool, void* conv_out, float* qn, float* kn, float* g, float* beta,
                                float* chunks, void* out, const int* qsl, const int* seq_lens, const int* slots, int R, int T,
                                int Hk, int Hv, int dk, int dv, int conv_k, int* status, cudaStream_t stream) {
  if (R <= 0 || T <= 0) return 0;
  const int C = 2 * Hk * dk + Hv * dv;
  if (conv_k != 4 || dv * (dk / 32) > 512 || (dk != 128 && dk != 64 && dk != 32)) {
    b200_set_last_error("gdn_forward: conv kernel 4, dk in {32,64,128}, dv * dk <= 16384 required", __FILE__,
                        __LINE__);
    return -1;
  }
  StepParams sp{};
  sp.x = (const __nv_bfloat16*)mixed; sp.w = (const __nv_bfloat16*)conv_w; sp.pool = (__nv_bfloat16*)conv_pool;
  sp.a = (const __nv_bfloat16*)a; sp.b = (const __nv_bfloat16*)b; sp.out = (__nv_bfloat16*)out; sp.A_log = A_log;
  sp.dt_bias = dt_bias; sp.rec = rec_pool; sp.qsl = qsl; sp.seq_lens = seq_lens; sp.slots = slots;
  sp.R = R; sp.T = T; sp.Hk = Hk; sp.Hv = Hv; sp.ldx = ldx; sp.lda = lda;
  int rc = launch_step<false>(sp, dk, dv, stream);
  if (rc <= 0) return rc;
  const int skip = step_takes(dk, dv, R, conv_w, rec_pool);
  if (conv_out == nullptr || (chunks != nullptr ? !skip : (qn == nullptr || kn == nullptr || g == nullptr || beta == nullptr))) {
    b200_set_last_error("gdn_forward: scratch is missing", __FILE__, __LINE__);
    return -1;
  }
  rc = launch_conv(mixed, conv_out, conv_pool, conv_w, qsl, seq_lens, slots, R, T, C, ldx, skip, stream);
  if (rc) return rc;
  if (chunks != nullptr)
    return b200_gdn_chunks(conv_out, C, a, b, lda, A_log, dt_bias, rec_pool, out, chunks, qsl, seq_lens, slots, R, T, Hk, Hv,
                           status, stream);
  const int work = T * (Hk * 32 > Hv ? Hk * 32 : Hv);
  B200_CUDA_CHECK(launch_pdl(gdn_prep_kernel, dim3((work + 255) / 256), dim3(256), (size_t)0, stream,
                             (const __nv_bfloat16*)conv_out, (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, A_log, dt_bias,
                             qn, kn, g, beta, T, Hk, Hv, dk, C, lda));
  return launch_recurrence<false>(qn, kn, conv_out, g, beta, rec_pool, out, qsl, seq_lens, slots, R, T, Hk, Hv, dk, dv, C,
                                  2 * Hk * dk, skip, stream);
}

namespace b200 {

// One warp per (token, k head): fp32 L2 normalisation of q (also scaled by dk^-1/2) and k.
// One thread per (token, v head, channel): per-channel decay, its logarithm in the unbounded form
// -exp(A_log) * softplus(a + dt_bias) or, with lower_bound < 0, lower_bound * sigmoid(exp(A_log) *
// (a + dt_bias)) (reference: compute_kda.py:42-63).  One thread per (token, v head): beta = sigmoid(b).
__global__ void kda_prep_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                                const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                const float* __restrict__ A_log, const float* __restrict__ dt_bias,
                                float lower_bound, float* __restrict__ qn, float* __restrict__ kn,
                                float* __restrict__ g, float* __restrict__ beta, int T, int Hk, int Hv, int dk, int ldq,
                                int ldk) {
  pdl_wait();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int warp = idx >> 5, lane = threadIdx.x & 31;
  if (warp < T * Hk) {
    const __nv_bfloat16* qp = q + (size_t)(warp / Hk) * ldq + warp % Hk * dk;
    const __nv_bfloat16* kp = k + (size_t)(warp / Hk) * ldk + warp % Hk * dk;
    float sq = 0.f, sk = 0.f;
    for (int i = lane; i < dk; i += 32) {
      const float qv = __bfloat162float(qp[i]), kv = __bfloat162float(kp[i]);
      sq += qv * qv;
      sk += kv * kv;
    }
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    const float iq = rsqrtf((float)dk) * rsqrtf(sq + 1e-6f), ik = rsqrtf(sk + 1e-6f);
    for (int i = lane; i < dk; i += 32) {
      qn[(size_t)warp * dk + i] = __bfloat162float(qp[i]) * iq;
      kn[(size_t)warp * dk + i] = __bfloat162float(kp[i]) * ik;
    }
  }
  if (idx < T * Hv * dk) {
    const int h = (idx / dk) % Hv, c = idx % dk;
    const float av = __bfloat162float(a[idx]) + dt_bias[h * dk + c];
    const float ea = __expf(A_log[h]);
    if (lower_bound < 0.f) {
      g[idx] = __expf(lower_bound / (1.f + __expf(-ea * av)));
    } else {
      const float sp = av > 20.f ? av : log1pf(__expf(av));
      g[idx] = __expf(-ea * sp);
    }
  }
  if (idx < T * Hv) beta[idx] = 1.f / (1.f + __expf(-__bfloat162float(b[idx])));
}

}  // namespace b200

// Kimi Delta Attention over a ragged batch.  q, k [T, Hk, dk] bf16 (raw; normalised here), v [T, Hv, dv]
// bf16 (tokens ldq, ldk, ldv elements apart), a [T, Hv, dk] bf16 raw gate, b [T, Hv] bf16, A_log [Hv], dt_bias [Hv, dk] fp32; lower_bound < 0
// selects the bounded gate.  rec_pool [slots, Hv, dk, dv] fp32 carries the state between steps (a request
// whose first token of the step is at position 0 starts from zero).  Scratch qn, kn [T, Hk, dk], g [T, Hv,
// dk], beta [T, Hv] fp32 from the caller.
extern "C" int b200_kda_forward(const void* q, const void* k, const void* v, int ldq, int ldk, int ldv, const void* a,
                                const void* b,
                                const float* A_log, const float* dt_bias, float lower_bound, float* rec_pool,
                                float* qn, float* kn, float* g, float* beta, void* out, const int* qsl,
                                const int* seq_lens, const int* slots, int R, int T, int Hk, int Hv, int dk,
                                int dv, cudaStream_t stream) {
  if (R <= 0 || T <= 0) return 0;
  if (dv * (dk / 32) > 512 || (dk != 128 && dk != 64 && dk != 32) || Hv % Hk) {
    b200_set_last_error("kda_forward: dk in {32,64,128}, dv * dk <= 16384, Hv a multiple of Hk required", __FILE__,
                        __LINE__);
    return -1;
  }
  StepParams sp{};
  sp.q = (const __nv_bfloat16*)q; sp.k = (const __nv_bfloat16*)k; sp.v = (const __nv_bfloat16*)v;
  sp.a = (const __nv_bfloat16*)a; sp.b = (const __nv_bfloat16*)b; sp.out = (__nv_bfloat16*)out; sp.A_log = A_log;
  sp.dt_bias = dt_bias; sp.rec = rec_pool; sp.qsl = qsl; sp.seq_lens = seq_lens; sp.slots = slots;
  sp.R = R; sp.T = T; sp.Hk = Hk; sp.Hv = Hv; sp.ldq = ldq; sp.ldk = ldk; sp.ldv = ldv; sp.lower_bound = lower_bound;
  const int rc = launch_step<true>(sp, dk, dv, stream);
  if (rc <= 0) return rc;
  const int skip = step_takes(dk, dv, R, nullptr, rec_pool);
  const long long work = (long long)T * Hv * dk > (long long)T * Hk * 32 ? (long long)T * Hv * dk
                                                                         : (long long)T * Hk * 32;
  B200_CUDA_CHECK(launch_pdl(kda_prep_kernel, dim3((unsigned)((work + 255) / 256)), dim3(256), (size_t)0, stream,
                             (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)a,
                             (const __nv_bfloat16*)b, A_log, dt_bias, lower_bound, qn, kn, g, beta, T, Hk, Hv, dk, ldq, ldk));
  return launch_recurrence<true>(qn, kn, v, g, beta, rec_pool, out, qsl, seq_lens, slots, R, T, Hk, Hv, dk, dv, ldv, 0,
                                 skip, stream);
}

// Causal depth-wise short convolution (kernel 4) + SiLU over a ragged batch with the window carried in
// conv_pool [slots, C, 3] bf16 — the first stage of b200_gdn_forward on its own, for layers that feed
// the convolved q, k, v to another recurrence (Kimi Delta Attention).  x [T, C] row stride ldx -> y [T, C].
extern "C" int b200_short_conv(const void* x, int ldx, const void* conv_w, void* conv_pool, void* y,
                               const int* qsl, const int* seq_lens, const int* slots, int R, int T, int C, int conv_k,
                               cudaStream_t stream) {
  if (R <= 0 || C <= 0 || T <= 0) return 0;
  if (conv_k != 4) {
    b200_set_last_error("short_conv: kernel width 4 required", __FILE__, __LINE__);
    return -1;
  }
  return launch_conv(x, y, conv_pool, conv_w, qsl, seq_lens, slots, R, T, C, ldx, 0, stream);
}
