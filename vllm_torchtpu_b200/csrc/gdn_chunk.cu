// Gated delta rule of prompts in chunks of 64 tokens on tcgen05 (key and value heads of 128, one decay per value head).
//
// With G_i the sum of the log-decays up to token i of the chunk, b the step sizes, k^ and q^ of unit length (q^ scaled) and
// S the state in front of the chunk:
//     R = V - e^G k^ S,   (I + A) U = b R,   A_ij = b_i e^(G_i - G_j) k^_i k^_j  (i > j)
//     O = e^G q^ S + P U,  P_ij = e^(G_i - G_j) q^_i k^_j (i >= j),   S <- e^(G_last) S + k^^T (e^(G_last - G) U)
//
// gdn_chunk_kernel (parallel over chunks and heads) forms T = (I + A)^-1 b and M = P T, so that U = T R and P U = M R.
// gdn_scan_kernel (one CTA per request and head, chunks in order) then needs three products per chunk, all of 128 rows:
//     [K; Q] S     K and Q are the convolution's bf16 values as they are; lengths and decays are factors of rows
//     [T; M] R     [T; M] in tensor memory
//     K^T U
// Everything that is fp32 (S, T, M, R, U) enters as three bf16 parts, which hold its 24 bits; an exact bf16 factor makes three
// products, two split ones six.  (The parts are cut, not rounded: what is left out of a product is below 2^-21 of it, and
// behind 64 terms below the rounding of a chain of fp32 multiply-adds, 6e-8 against 1.5e-7 on normal values.)  Sums are fp32.
//
// What bounds it: the chain of a request, 64 tokens at a time (6.4 us a chunk: 3840 cycles of products, the rest splits and
// barriers between them); token by token (gdn_recurrent_kernel) a token takes 0.67 us.  4 x 2048 tokens, 32 value heads:
// 1369 us there, 198 + 196 us here.
#include <cstring>
#include <type_traits>

#include "common.cuh"

namespace b200 {
namespace gdnc {

constexpr int C = 64, D = 128;
constexpr int FACTORS = 128 * 64;                     // floats of a (chunk, head): [T; M], row factors of k S, q S and U, decay
constexpr int UNIT = FACTORS + 4 * 64;                // and a flag

struct Params {
  const __nv_bfloat16 *y, *a, *b;                     // y: convolved rows [T, Cy]
  const float *A_log, *dt_bias;
  float *rec, *unit;
  __nv_bfloat16* out;
  const int *qsl, *seq_lens, *slots;
  int* status;
  int R, T, Hk, Hv, Cy, lda;
};

// chunks of request i; requests of one token are not taken here
__device__ __forceinline__ int chunks_of(const Params& p, int i) {
  if (i >= p.R) return 0;
  const int n = p.qsl[i + 1] - p.qsl[i];
  return n > 1 && p.slots[i] >= 0 ? (n + C - 1) / C : 0;
}

__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// grid (chunks, Hv), 128 threads.  Scores on mma.sync (exact bf16 operands); decays from a prefix sum in 64 bits, so that
// differences keep their digits; (I + A) is inverted by blocks (columns of 64 by substitution, on half of the threads: 229 us
// instead of 180 for 4 x 2048 tokens and 32 heads).
constexpr int LDT = 136, LDA = 68;
__global__ void __launch_bounds__(128) gdn_chunk_kernel(const Params p) {
  pdl_wait();
  __shared__ __align__(16) uint8_t buf[2 * C * LDT * 2];                // K and Q, then A and P
  __shared__ float sX[C / 2 * C / 2];
  __shared__ double sG[C];
  __shared__ float sbeta[C], sik[2 * C];
  const int hv = blockIdx.y, hk = hv / (p.Hv / p.Hk), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int r = -1, chunk = blockIdx.x;
  for (int b = 0; b < p.R; b += 32) {
    const int n = chunks_of(p, b + lane);
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
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
  if (r < 0) return;
  const int row0 = p.qsl[r] + chunk * C, n = min(C, p.qsl[r + 1] - row0);
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(buf);         // rows 0-63: K, 64-127: Q
  for (int i = tid; i < 2 * C * 16; i += 128) {
    const int row = i >> 4, x = (i & 15) * 8, t = row & 63;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (t < n) v = *reinterpret_cast<const uint4*>(p.y + (size_t)(row0 + t) * p.Cy + (row < C ? p.Hk * D : 0) + hk * D + x);
    *reinterpret_cast<uint4*>(tile + row * LDT + x) = v;
  }
  if (warp == 0) {
    const float ea = __expf(p.A_log[hv]) * 1.4426950408889634f, dt = p.dt_bias[hv];
    double g[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = 2 * lane + e;
      float z = 0.f, be = 0.f;
      if (t < n) {
        const float av = __bfloat162float(p.a[(size_t)(row0 + t) * p.lda + hv]) + dt;
        z = -ea * (av > 20.f ? av : log1pf(__expf(av)));
        be = 1.f / (1.f + __expf(-__bfloat162float(p.b[(size_t)(row0 + t) * p.lda + hv])));
      }
      z = z < -1000.f ? -1000.f : z;                  // (2^-1000 is zero in fp32; differences of sums stay finite; a NaN stays)
      g[e] = (double)z;
      sbeta[t] = be;
    }
    double s = g[0] + g[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double x = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += x;
    }
    sG[2 * lane] = s - g[1];
    sG[2 * lane + 1] = s;
  }
  __syncthreads();
  int odd;                                            // (see token_by_token)
  {
    float s = 0.f;                                    // thread = row of the tile
#pragma unroll 4
    for (int x = 0; x < D; x += 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(tile + tid * LDT + x);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __bfloat1622float2(h[e]);
        s = fmaf(f.x, f.x, fmaf(f.y, f.y, s));
      }
    }
    sik[tid] = (tid < C ? 1.f : rsqrtf((float)D)) / fmaxf(sqrtf(s), 1e-12f);
    odd = !isfinite(s) || (tid < C && !isfinite(sbeta[tid] + (float)sG[tid]));
  }
  float kk[8][4], qk[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) kk[i][e] = qk[i][e] = 0.f;
  const uint32_t tb = smem_u32(tile);
  const int mi = lane >> 3, rr = lane & 7;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    uint32_t ak[4], aq[4];
    const int arow = warp * 16 + (mi & 1) * 8 + rr, acol = ks * 16 + (mi >> 1) * 8;
    ldsm4(ak, tb + (arow * LDT + acol) * 2);
    ldsm4(aq, tb + ((C + arow) * LDT + acol) * 2);
#pragma unroll
    for (int nb = 0; nb < 8; nb += 2) {
      if (nb * 8 > warp * 16 + 15) break;             // above the diagonal
      uint32_t bk[4];
      ldsm4(bk, tb + ((nb * 8 + (mi >> 1) * 8 + rr) * LDT + ks * 16 + (mi & 1) * 8) * 2);
      mma16816(kk[nb], ak, bk[0], bk[1]);
      mma16816(kk[nb + 1], ak, bk[2], bk[3]);
      mma16816(qk[nb], aq, bk[0], bk[1]);
      mma16816(qk[nb + 1], aq, bk[2], bk[3]);
    }
  }
  __syncthreads();
  float* sA = reinterpret_cast<float*>(buf);
  float* sP = sA + C * LDA;
#pragma unroll
  for (int nb = 0; nb < 8; ++nb) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = warp * 16 + (lane >> 2) + (e >> 1) * 8, j = nb * 8 + 2 * (lane & 3) + (e & 1);
      const float d = j <= i ? exp2f((float)(sG[i] - sG[j])) * sik[j] : 0.f;
      sA[i * LDA + j] = j < i ? sbeta[i] * sik[i] * d * kk[nb][e] : 0.f;
      sP[i * LDA + j] = sik[C + i] * d * qk[nb][e];
    }
  }
  odd = __syncthreads_or(odd);
  // ---- (I + A)^-1 in place of A: blocks of 16 by substitution (a thread a column), then two levels of
  // [T1 0; -T2 A21 T1  T2]
  if (tid < C) {
    const int b = tid & ~15, col = tid & 15;
    float x[16];
    const float* a0 = sA + b * LDA + b;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s[4] = {i == col ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int l = 0; l < i; l += 4) {
        const float4 a = *reinterpret_cast<const float4*>(a0 + i * LDA + l);       // zeros from the diagonal on
        s[0] = fmaf(-a.x, x[l], s[0]);
        if (l + 1 < i) s[1] = fmaf(-a.y, x[l + 1], s[1]);
        if (l + 2 < i) s[2] = fmaf(-a.z, x[l + 2], s[2]);
        if (l + 3 < i) s[3] = fmaf(-a.w, x[l + 3], s[3]);
      }
      x[i] = (s[0] + s[1]) + (s[2] + s[3]);
    }
    __syncwarp();                                     // (a block belongs to half a warp)
#pragma unroll
    for (int i = 0; i < 16; ++i) sA[(b + i) * LDA + b + col] = x[i];
  }
  __syncthreads();
  // X = A21 T1, then A21 <- -T2 X, for blocks of H rows; a thread's outputs are PER rows of one column
  auto merge = [&](auto size) {
    constexpr int H = decltype(size)::value, PER = C / 2 * H / 128;
    const int o = tid * PER, pair = o / (H * H), col = tid % H, r0 = (tid / H) * PER % H, b = pair * 2 * H;
    float acc[PER];
#pragma unroll
    for (int e = 0; e < PER; ++e) acc[e] = 0.f;
    const float* a21 = sA + (b + H + r0) * LDA + b;
    const float* t1 = sA + b * LDA + b + col;
#pragma unroll 4
    for (int k = 0; k < H; k += 4) {
      const float t[4] = {t1[k * LDA], t1[(k + 1) * LDA], t1[(k + 2) * LDA], t1[(k + 3) * LDA]};
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const float4 a = *reinterpret_cast<const float4*>(a21 + e * LDA + k);
        acc[e] = fmaf(a.x, t[0], fmaf(a.y, t[1], fmaf(a.z, t[2], fmaf(a.w, t[3], acc[e]))));
      }
    }
    float* x = sX + pair * H * H;
#pragma unroll
    for (int e = 0; e < PER; ++e) x[(r0 + e) * H + col] = acc[e];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < PER; ++e) acc[e] = 0.f;
    const float* t2 = sA + (b + H + r0) * LDA + b + H;
#pragma unroll 4
    for (int k = 0; k < H; k += 4) {
      const float t[4] = {x[k * H + col], x[(k + 1) * H + col], x[(k + 2) * H + col], x[(k + 3) * H + col]};
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const float4 a = *reinterpret_cast<const float4*>(t2 + e * LDA + k);
        acc[e] = fmaf(-a.x, t[0], fmaf(-a.y, t[1], fmaf(-a.z, t[2], fmaf(-a.w, t[3], acc[e]))));
      }
    }
    float* d = sA + (b + H + r0) * LDA + b + col;
#pragma unroll
    for (int e = 0; e < PER; ++e) d[e * LDA] = acc[e];
    __syncthreads();
  };
  merge(std::integral_constant<int, 16>());
  merge(std::integral_constant<int, 32>());
  // ---- M = P T: a thread has 8 rows x 4 columns; both are lower triangular.  Stored in groups of four columns,
  // [16][128 rows][4], so that the scan's threads (a row each) read neighbouring pieces.
  float* unit = p.unit + ((size_t)blockIdx.x * p.Hv + hv) * UNIT;
  {
    const int i0 = (tid >> 4) * 8, j0 = (tid & 15) * 4;
    float m[8][4];
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
      for (int u = 0; u < 4; ++u) m[e][u] = 0.f;
    for (int k = j0; k < i0 + 8; k += 4) {
      float4 t[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) t[u] = *reinterpret_cast<const float4*>(sA + (k + u) * LDA + j0);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 a = *reinterpret_cast<const float4*>(sP + (i0 + e) * LDA + k);
        const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          m[e][0] = fmaf(av[u], t[u].x, m[e][0]);
          m[e][1] = fmaf(av[u], t[u].y, m[e][1]);
          m[e][2] = fmaf(av[u], t[u].z, m[e][2]);
          m[e][3] = fmaf(av[u], t[u].w, m[e][3]);
        }
      }
    }
    const float4 be = make_float4(sbeta[j0], sbeta[j0 + 1], sbeta[j0 + 2], sbeta[j0 + 3]);
    float4* d = reinterpret_cast<float4*>(unit) + (j0 >> 2) * 128 + i0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float4 t = *reinterpret_cast<const float4*>(sA + (i0 + e) * LDA + j0);
      d[e] = make_float4(t.x * be.x, t.y * be.y, t.z * be.z, t.w * be.w);
      d[C + e] = make_float4(m[e][0] * be.x, m[e][1] * be.y, m[e][2] * be.z, m[e][3] * be.w);
    }
  }
  if (tid < C) {
    const int i = tid;
    float* f = unit + FACTORS;
    const float e = exp2f((float)sG[i]);
    f[i] = sik[i] * e;
    f[C + i] = sik[C + i] * e;
    f[2 * C + i] = sik[i] * exp2f((float)(sG[C - 1] - sG[i]));
    if (i == 0) {
      f[3 * C] = exp2f((float)sG[C - 1]);
      f[3 * C + 1] = odd ? 1.f : 0.f;
    }
  }
}

// ------------------------------------------------------------------------------------------- the scan
constexpr int PANEL_S = D * 128, PANEL_R = C * 128;   // 64 columns of S, of R and U
constexpr int SMEM_S = 0, SMEM_R = SMEM_S + 3 * 2 * PANEL_S, SMEM_KQ = SMEM_R + 3 * 2 * PANEL_R;
constexpr int KQ_BYTES = 2 * 128 * 128, SMEM_V = SMEM_KQ + 2 * KQ_BYTES, SMEM_F = SMEM_V + C * 2 * D;
constexpr int SMEM_BAR = SMEM_F + 2 * 256 * 4, SMEM_USED = SMEM_BAR + 64, SMEM_TOTAL = 227 * 1024;
constexpr int TM_1 = 0, TM_2 = 128, TM_3 = 256, TM_A = 384;

// 128-byte swizzle, groups of 8 rows 1024 bytes apart, the next 64 values of an M- or N-major operand `lbo` bytes away
__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr, uint32_t lbo) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)2 << 61;
}
// A from tensor memory
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(
          taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// v = h + m + l, three bf16 numbers each; two values packed per word
struct Parts {
  uint32_t h, m, l;
};
__device__ __forceinline__ Parts parts2(float a, float b) {
  const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
  const float a1 = a - __uint_as_float(ua & 0xffff0000u), b1 = b - __uint_as_float(ub & 0xffff0000u);
  const uint32_t va = __float_as_uint(a1), vb = __float_as_uint(b1);
  const float a2 = a1 - __uint_as_float(va & 0xffff0000u), b2 = b1 - __uint_as_float(vb & 0xffff0000u);
  Parts p;
  p.h = __byte_perm(ua, ub, 0x7632);
  p.m = __byte_perm(va, vb, 0x7632);
  p.l = __byte_perm(__float_as_uint(a2), __float_as_uint(b2), 0x7632);
  return p;
}
// 32 values of a row (128 bytes of 64 columns), its columns 32 * which .., into the three parts, `part` bytes apart
__device__ __forceinline__ void put32(uint8_t* row128, int sw, int which, uint32_t part, const float* v) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    Parts q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) q[e] = parts2(v[8 * c + 2 * e], v[8 * c + 2 * e + 1]);
    uint8_t* d = row128 + (((which * 4 + c) ^ sw) << 4);
    *reinterpret_cast<uint4*>(d) = make_uint4(q[0].h, q[1].h, q[2].h, q[3].h);
    *reinterpret_cast<uint4*>(d + part) = make_uint4(q[0].m, q[1].m, q[2].m, q[3].m);
    *reinterpret_cast<uint4*>(d + 2 * part) = make_uint4(q[0].l, q[1].l, q[2].l, q[3].l);
  }
}

// The rule token by token, for the rest of a request from a chunk on that holds a value that is not finite: in the products
// of a chunk that value would reach the tokens in front of it as 0 * NaN.  (Sums of finite squares in fp32 bound the products
// of q and k; what overflows there counts as not finite.)  Thread = (row ln of the state, 64 of its columns); k S and q S are
// summed over the lanes of a warp (afterwards lane l has columns 2 l and 2 l + 1), then over the four warps of a half.
__device__ __noinline__ void token_by_token(const Params& p, float* red, int qs, int n, int hv, int hk, float* st) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ln = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 64;
  float *rqk = red + 8 * 128, *su = rqk + 4 * 3;      // [8 warps][2][64]; q k, k k, q q of four warps; u
  const float ea = __expf(p.A_log[hv]), dt = p.dt_bias[hv];
  float S[64];
#pragma unroll
  for (int i = 0; i < 64; ++i) S[i] = st[i];
  auto lanes_sum = [&](float factor) -> float2 {
    float a[32];
    const bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      a[i] = factor * (up ? S[32 + i] : S[i]) + __shfl_xor_sync(0xffffffffu, factor * (up ? S[i] : S[32 + i]), 16);
#pragma unroll
    for (int h = 16; h >= 2; h >>= 1) {
      const bool hi = lane & (h >> 1);
#pragma unroll
      for (int i = 0; i < h; ++i) a[i] = (hi ? a[h + i] : a[i]) + __shfl_xor_sync(0xffffffffu, hi ? a[i] : a[h + i], h >> 1);
    }
    return make_float2(a[0], a[1]);
  };
#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    const __nv_bfloat16* y = p.y + (size_t)(qs + t) * p.Cy;
    float kv = __bfloat162float(y[(p.Hk + hk) * D + ln]), qv = __bfloat162float(y[hk * D + ln]);
    const float kk = warp_sum(kv * kv), qq = warp_sum(qv * qv);
    if (warp < 4 && lane == 0) { rqk[4 + warp] = kk; rqk[8 + warp] = qq; }
    __syncthreads();
    auto over_warps = [&](int i) -> float { return (rqk[4 * i] + rqk[4 * i + 1]) + (rqk[4 * i + 2] + rqk[4 * i + 3]); };
    kv *= 1.f / fmaxf(sqrtf(over_warps(1)), 1e-12f);
    qv *= rsqrtf((float)D) / fmaxf(sqrtf(over_warps(2)), 1e-12f);
    const float z = __bfloat162float(p.a[(size_t)(qs + t) * p.lda + hv]) + dt;
    const float dec = __expf(-ea * (z > 20.f ? z : log1pf(__expf(z))));
    const float beta = 1.f / (1.f + __expf(-__bfloat162float(p.b[(size_t)(qs + t) * p.lda + hv])));
#pragma unroll
    for (int i = 0; i < 64; ++i) S[i] *= dec;
    reinterpret_cast<float2*>(red + warp * 128)[lane] = lanes_sum(kv);
    reinterpret_cast<float2*>(red + warp * 128 + 64)[lane] = lanes_sum(qv);
    const float d = warp_sum(kv * qv);
    if (warp < 4 && lane == 0) rqk[warp] = d;
    __syncthreads();
    if (tid < D) {                                    // thread = value column
      const float* x = red + (tid >> 6) * 512 + (tid & 63);
      const float mem = (x[0] + x[128]) + (x[256] + x[384]), o = (x[64] + x[192]) + (x[320] + x[448]);
      const float u = (__bfloat162float(y[(2 * p.Hk + hv) * D + tid]) - mem) * beta;
      su[tid] = u;
      p.out[((size_t)(qs + t) * p.Hv + hv) * D + tid] = __float2bfloat16(fmaf(over_warps(0), u, o));
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 64; ++i) S[i] = fmaf(kv, su[c0 + i], S[i]);
  }
#pragma unroll
  for (int i = 0; i < 64; ++i) st[i] = S[i];
}

// grid (Hv, R), 256 threads: thread = (lane of the tensor memory, half of the 128 value columns).  Lanes 0-63 are the
// chunk's tokens as keys, lanes 64-127 as queries; for the state they are its 128 rows, held in registers.
__global__ void __launch_bounds__(256, 1) gdn_scan_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem + SMEM_USED > smem_raw + SMEM_TOTAL) {     // (the base is 1024-byte aligned: nothing is cut off)
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, ST_OK, ST_BAD_INDEX);
    return;
  }
  float* fac = reinterpret_cast<float*>(smem + SMEM_F);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + SMEM_BAR);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int hv = blockIdx.x, r = blockIdx.y, hk = hv / (p.Hv / p.Hk), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ln = (warp & 3) * 32 + lane, half = warp >> 2, c0 = half * 64;
  pdl_launch_dependents();
  pdl_wait();
  const int qs = p.qsl[r], n = p.qsl[r + 1] - qs, slot = p.slots[r];
  // rows of no request, and of requests without a state, are zeros (single tokens belong to the step kernel)
  const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
  for (int t = max(0, p.qsl[p.R]) + r; t < p.T; t += p.R)
    if (tid < 16) reinterpret_cast<uint4*>(p.out + ((size_t)t * p.Hv + hv) * D)[tid] = z4;
  if (n <= 1) return;
  if (slot < 0) {
    for (int i = tid; i < n * 16; i += 256) reinterpret_cast<uint4*>(p.out + ((size_t)(qs + (i >> 4)) * p.Hv + hv) * D)[i & 15] = z4;
    return;
  }
  if (tid == 0) {
    mbar_init(bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  int first = 0;                                      // chunks of the requests before this one
  for (int b = 0; b < r; b += 32) first += warp_sum(b + lane < r ? chunks_of(p, b + lane) : 0);
  const int chunks = (n + C - 1) / C;
  const float* unit = p.unit + ((size_t)first * p.Hv + hv) * UNIT;
  const size_t unit_step = (size_t)p.Hv * UNIT;

  // K (rows 0-63) and Q (64-127) of a chunk: two panels of 64 channels, rows of 128 bytes, swizzled; zeros behind the end
  auto load_kq = [&](int c) {
    const uint32_t dst = smem_u32(smem + SMEM_KQ + (c & 1) * KQ_BYTES);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int idx = tid + i * 256, row = idx >> 4, ch = idx & 15, t = c * C + (row & 63);
      const __nv_bfloat16* src = p.y + (size_t)(qs + min(t, n - 1)) * p.Cy + (row < C ? p.Hk * D : 0) + hk * D + ch * 8;
      const uint32_t d = dst + (ch >> 3) * (128 * 128) + row * 128 + (((ch & 7) ^ (row & 7)) << 4);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(t < n ? 16 : 0) : "memory");
    }
    // row factors, the decay and the flag: 194 floats
    if (tid < 49) {
      const float* src = unit + (size_t)c * unit_step + FACTORS + tid * 4;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(fac + (c & 1) * 256 + tid * 4)), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // V: 64 tokens of 256 bytes, pieces of 16 bytes swizzled within a half row
  auto load_v = [&](int c) {
    const uint32_t dst = smem_u32(smem + SMEM_V);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256, row = idx >> 4, ch = idx & 15, t = c * C + row;
      const __nv_bfloat16* src = p.y + (size_t)(qs + min(t, n - 1)) * p.Cy + (2 * p.Hk + hv) * D + ch * 8;
      const uint32_t d = dst + row * 256 + (ch >> 3) * 128 + (((ch & 7) ^ (row & 7)) << 4);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(t < n ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float4 traw[8];                                     // [T; M]: 32 values of row ln
  auto load_t = [&](int c) {
    const float4* src = reinterpret_cast<const float4*>(unit + (size_t)c * unit_step) + half * 8 * 128 + ln;
#pragma unroll
    for (int i = 0; i < 8; ++i) traw[i] = src[i * 128];
  };
  load_kq(0);
  load_t(0);
  load_v(0);
  float S[64];
  float* st = p.rec + (((size_t)slot * p.Hv + hv) * D + ln) * D + c0;
  const bool fresh = p.seq_lens[r] == n;
#pragma unroll
  for (int i = 0; i < 64; i += 4) {
    const float4 v = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(st + i);
    S[i] = v.x; S[i + 1] = v.y; S[i + 2] = v.z; S[i + 3] = v.w;
  }
  uint8_t* s_row = smem + SMEM_S + half * PANEL_S + ln * 128;
  uint8_t* r_row = smem + SMEM_R + half * PANEL_R + (ln & 63) * 128;
  const uint8_t* v_row = smem + SMEM_V + (ln & 63) * 256 + half * 128;
  const int sw = ln & 7;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, lane_addr = (uint32_t)((warp & 3) * 32) << 16;
  auto put_t = [&]() {
    const float* t = reinterpret_cast<const float*>(traw);
    uint32_t h[16], m[16], l[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const Parts q = parts2(t[2 * i], t[2 * i + 1]);
      h[i] = q.h; m[i] = q.m; l[i] = q.l;
    }
    const uint32_t a = tmem + lane_addr + TM_A + half * 16;
    tmem_st_16(a, h);
    tmem_st_16(a + 32, m);
    tmem_st_16(a + 64, l);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  };
  put32(s_row, sw, 0, 2 * PANEL_S, S);
  put32(s_row, sw, 1, 2 * PANEL_S, S + 32);
  put_t();
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  constexpr uint32_t idesc_kb = umma_idesc_bf16(128, 128) | (1u << 16);                     // B N-major
  constexpr uint32_t idesc_ab = umma_idesc_bf16(128, 128) | (1u << 16) | (1u << 15);        // A M-major too
  const uint64_t s_desc = desc_sw128(smem_u32(smem + SMEM_S), PANEL_S), r_desc = desc_sw128(smem_u32(smem + SMEM_R), PANEL_R);
  uint32_t phase = 0;
  bool ok = true, odd = false;
  int c = 0;
  for (; c < chunks; ++c) {
    const float* f = fac + (c & 1) * 256;
    const uint32_t kq = smem_u32(smem + SMEM_KQ + (c & 1) * KQ_BYTES);
    fence_proxy_async_smem();
    tc_fence_before();
    if (__syncthreads_or(!ok)) break;
    if (warp == 0 && elect_one()) {                   // [K; Q] S
      tc_fence_after();
      const uint64_t a = umma_desc_k_sw128(kq);
#pragma unroll
      for (int part = 0; part < 3; ++part) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_f16(tmem + TM_1, a + (ks >> 2) * (128 * 128 / 16) + 2 * (ks & 3),
                   s_desc + (((2 - part) * 2 * PANEL_S + ks * 16 * 128) >> 4), idesc_kb, part > 0 || ks > 0 ? 1u : 0u);
      }
      umma_commit(bar);
    }
    __syncwarp();
    if (c + 1 < chunks) load_kq(c + 1);
    odd = f[3 * C + 1] != 0.f;
    {                                                 // the pieces of V that this thread has copied: 0 * infinity is a NaN
      const __nv_bfloat162 z = __float2bfloat162_rn(0.f);
      __nv_bfloat162 s[4] = {z, z, z, z};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint4 q = *reinterpret_cast<const uint4*>(smem + SMEM_V + (tid + i * 256) * 16);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = __hfma2(h[e], z, s[e]);
      }
      const float2 sum = __bfloat1622float2(__hadd2(__hadd2(s[0], s[1]), __hadd2(s[2], s[3])));
      odd |= !(sum.x + sum.y == 0.f);
    }
    ok = mbar_wait(bar, phase, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL) && ok;
    phase ^= 1;
    tc_fence_after();
    if (ln < C) {                                     // R
      const float fk = f[ln];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t d[32];
        float v[32];
        tmem_ld_32x32(tmem + lane_addr + TM_1 + c0 + 32 * x, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          const uint4 q = *reinterpret_cast<const uint4*>(v_row + (((4 * x + (i >> 3)) ^ sw) << 4));
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            v[i + 2 * u] = fmaf(-fk, __uint_as_float(d[i + 2 * u]), __uint_as_float(w[u] << 16));
            v[i + 2 * u + 1] = fmaf(-fk, __uint_as_float(d[i + 2 * u + 1]), __uint_as_float(w[u] & 0xffff0000u));
          }
        }
        put32(r_row, sw, x, 2 * PANEL_R, v);
      }
    }
    fence_proxy_async_smem();
    tc_fence_before();
    if (__syncthreads_or(!ok || odd)) break;          // (the state is still that in front of the chunk)
    if (warp == 0 && elect_one()) {                   // [T; M] R
      tc_fence_after();
      constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};                 // small products first
#pragma unroll
      for (int q = 0; q < 6; ++q) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          umma_ts(tmem + TM_2, tmem + TM_A + pa[q] * 32 + ks * 8, r_desc + ((pb[q] * 2 * PANEL_R + ks * 16 * 128) >> 4),
                  idesc_kb, q > 0 || ks > 0 ? 1u : 0u);
      }
      umma_commit(bar);
    }
    __syncwarp();
    if (c + 1 < chunks) load_t(c + 1);
    ok = mbar_wait(bar, phase, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL) && ok;
    phase ^= 1;
    tc_fence_after();
    if (ln < C) {                                     // U, scaled for the state
      const float fu = f[2 * C + ln];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t d[32];
        float v[32];
        tmem_ld_32x32(tmem + lane_addr + TM_2 + c0 + 32 * x, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = fu * __uint_as_float(d[i]);
        put32(r_row, sw, x, 2 * PANEL_R, v);
      }
    }
    fence_proxy_async_smem();
    tc_fence_before();
    if (__syncthreads_or(!ok)) break;
    if (warp == 0 && elect_one()) {                   // K^T U
      tc_fence_after();
      const uint64_t a = desc_sw128(kq, 128 * 128);
#pragma unroll
      for (int part = 0; part < 3; ++part) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          umma_f16(tmem + TM_3, a + ((ks * 16 * 128) >> 4), r_desc + (((2 - part) * 2 * PANEL_R + ks * 16 * 128) >> 4), idesc_ab,
                   part > 0 || ks > 0 ? 1u : 0u);
      }
      umma_commit(bar);
    }
    __syncwarp();
    // Beside it: the output, the next [T; M] into tensor memory and the next V into shared memory.  (A fence between generic
    // and tensor-core accesses waits for a thread's loads and stores too: those of global memory are issued right behind
    // one.  With the output and V's loads in front of the fence above it took 3000 cycles more.)
    if (c + 1 < chunks) {
      load_v(c + 1);
      put_t();
    }
    if (ln >= C) {                                    // O
      const float fq = f[ln];
      const int t = c * C + ln - C;
      __nv_bfloat16* o = p.out + ((size_t)(qs + t) * p.Hv + hv) * D + c0;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t d[32], e[32];
        tmem_ld_32x32(tmem + lane_addr + TM_1 + c0 + 32 * x, d);
        tmem_ld_32x32(tmem + lane_addr + TM_2 + c0 + 32 * x, e);
        tmem_ld_wait();
        if (t < n && ok) {
#pragma unroll
          for (int i = 0; i < 32; i += 16) {
            uint32_t w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const __nv_bfloat162 b2 =
                  __floats2bfloat162_rn(fmaf(fq, __uint_as_float(d[i + 2 * u]), __uint_as_float(e[i + 2 * u])),
                                        fmaf(fq, __uint_as_float(d[i + 2 * u + 1]), __uint_as_float(e[i + 2 * u + 1])));
              w[u] = *reinterpret_cast<const uint32_t*>(&b2);
            }
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + 32 * x + i), "r"(w[0]), "r"(w[1]),
                         "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                         : "memory");
          }
        }
      }
    }
    ok = mbar_wait(bar, phase, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL) && ok;
    phase ^= 1;
    tc_fence_after();
    const float dec = f[3 * C];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      uint32_t d[32];
      tmem_ld_32x32(tmem + lane_addr + TM_3 + c0 + 32 * x, d);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) S[32 * x + i] = fmaf(dec, S[32 * x + i], __uint_as_float(d[i]));
      if (c + 1 < chunks) put32(s_row, sw, x, 2 * PANEL_S, S + 32 * x);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (ok) {
#pragma unroll
    for (int i = 0; i < 64; i += 4) *reinterpret_cast<float4*>(st + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
  }
  tc_fence_before();
  odd = __syncthreads_or(odd);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (odd && !__syncthreads_or(!ok))
    token_by_token(p, reinterpret_cast<float*>(smem), qs + c * C, n - c * C, hv, hk, st);
}

}  // namespace gdnc
}  // namespace b200

using namespace b200;

// y [T, Cy] convolved rows (16-byte aligned, Cy a multiple of 8), heads of 128 / 128; see gdn.cu for the rest.  Requests of one
// token are left out.  scratch: UNIT floats for each of (T / 64 + R) chunks and Hv heads.
extern "C" int b200_gdn_chunks(const void* y, int Cy, const void* a, const void* b, int lda, const float* A_log,
                               const float* dt_bias, float* rec_pool, void* out, float* scratch, const int* qsl,
                               const int* seq_lens, const int* slots, int R, int T, int Hk, int Hv, int* status,
                               cudaStream_t stream) {
  if (R <= 0 || T <= 0) return 0;
  if (R > 65535 || Hv > 65535 || scratch == nullptr || Cy % 8 || (((uintptr_t)y | (uintptr_t)scratch | (uintptr_t)rec_pool) & 15) ||
      ((uintptr_t)out & 31)) {
    b200_set_last_error("gdn_chunks: aligned rows and scratch required", __FILE__, __LINE__);
    return -1;
  }
  gdnc::Params p;
  p.y = (const __nv_bfloat16*)y; p.a = (const __nv_bfloat16*)a; p.b = (const __nv_bfloat16*)b;
  p.A_log = A_log; p.dt_bias = dt_bias; p.rec = rec_pool; p.unit = scratch; p.out = (__nv_bfloat16*)out;
  p.qsl = qsl; p.seq_lens = seq_lens; p.slots = slots; p.status = status;
  p.R = R; p.T = T; p.Hk = Hk; p.Hv = Hv; p.Cy = Cy; p.lda = lda;
  static unsigned long long seen = 0;
  B200_CUDA_CHECK(ensure_dynamic_smem(gdnc::gdn_scan_kernel, gdnc::SMEM_TOTAL, &seen));
  B200_CUDA_CHECK(launch_pdl(gdnc::gdn_chunk_kernel, dim3(T / gdnc::C + R, Hv), dim3(128), (size_t)0, stream, p));
  B200_CUDA_CHECK(launch_pdl(gdnc::gdn_scan_kernel, dim3(Hv, R), dim3(256), (size_t)gdnc::SMEM_TOTAL, stream, p));
  return 0;
}
