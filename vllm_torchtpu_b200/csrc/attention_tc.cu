// Prefill / mixed ragged paged attention on the 5th-generation tensor cores (head_dim 128, bf16).
//
// Persistent CTAs, one per SM.  A tile has 128 query rows = the G q-heads of one kv head x 128/G consecutive positions of one
// request, so every K/V byte staged in shared memory serves the whole GQA group.  Per 128-key chunk:
//   S = Q K^T        tcgen05.mma (kind::f16), Q and K in shared memory (TMA, SWIZZLE_128B, K-major),
//                    S in TMEM (fp32, 128 columns, two buffers)
//   softmax          eight warps, two threads per row: tcgen05.ld the row, scale / mask / running max
//                    / exp2 / sum in registers, P written as bf16 into shared memory in the K-major
//                    swizzled layout the next MMA reads
//   O_chunk = P V    tcgen05.mma with V as an MN-major operand (the cache stores V with head_dim
//                    contiguous), result in TMEM (two buffers); the softmax threads fold it into
//                    their fp32 register accumulators (acc = acc * alpha + O_chunk), so TMEM is
//                    never rescaled in place.
// Warp roles: warp 0 TMA producer (Q of this tile and the next, K and V rings, one page of 16 tokens per lane and copy), warp 1
// MMA issuer, warps 2-9 softmax + output (two threads per row, one per half of the key columns).  S(j+1) is issued before
// P V(j), so the tensor core works on the next scores while the softmax of the current chunk runs.  512 TMEM columns, 226 KB
// of shared memory.  What bounds it: the chain scores -> softmax -> P V of a chunk; the tensor work of a chunk is 1024 cycles.
// 8 x 1024 tokens, 32 / 8 heads: 237 us with a CTA per tile, the scores read twice from TMEM and K, V and the table entry
// waited for together; 223 us persistent with the scores read once; 200 us with K and V copied as their buffers come free;
// 185 us with capped scores in an instance of their own (fewer registers in this one), 181 us with rounds of tiles back and
// forth.  Every mbarrier wait is bounded (status word + abort flag + TMEM freed on exit).
//
// Same function as the mma.sync prefill kernel in attention.cu (causal ragged batches with prefix
// context, sliding window, soft-cap, sinks, LSE); semantics of the reference's ragged paged
// attention (reference: src/vllm_torchtpu/kernels/ragged_paged_attention/v3/kernel.py:74-214).
#include <cstring>

#include "common.cuh"
#include "gemm_tcgen05.h"

namespace b200 {
namespace fa {

constexpr int D = 128;
constexpr int BM = 128;                  // query rows per tile
constexpr int BKV = 128;                 // keys per chunk
constexpr int HALF_BYTES = 128 * 128;    // 128 rows x 64 bf16: one swizzled half of a 128 x 128 tile
constexpr int TILE_BYTES = 2 * HALF_BYTES;
constexpr int KV_STAGES = 2;
constexpr int SMEM_Q = 0;                               // two buffers: the next tile's queries arrive during this one
constexpr int SMEM_K = SMEM_Q + 2 * TILE_BYTES;
constexpr int SMEM_V = SMEM_K + KV_STAGES * TILE_BYTES;
constexpr int SMEM_P = SMEM_V + KV_STAGES * TILE_BYTES;
constexpr int SMEM_BAR = SMEM_P + TILE_BYTES;
constexpr int SMEM_XCH = SMEM_BAR + 256;                // row-max and row-sum exchange between the two column halves
constexpr int SMEM_USED = SMEM_XCH + 2 * 2 * 128 * 4, SMEM_TOTAL = 227 * 1024;
static_assert(SMEM_USED <= SMEM_TOTAL, "shared memory");
constexpr int NUM_THREADS = 64 + 256;                   // TMA warp, MMA warp, 8 softmax warps

struct Params {
  __nv_bfloat16* out;
  float* lse;
  const int* block_tables;
  const int* seq_lens;
  const int* qsl;
  const float* sinks;
  int* status;
  int max_blocks, block_size, Hq, Hkv, G, BQ, req_begin, req_end, window;
  int ldo;                             // elements between the output rows of neighbouring tokens (without an epilogue)
  int pv_half;                    // 1: values and probabilities in fp16 (an e4m3 cache, whose values are exact in it), 0: bf16
  int non_causal;                 // 1: every query row sees the whole sequence (encoders, diffusion)
  long long num_blocks;
  float scale_log2, softcap;
  HeadFinish fin;                 // with FIN
};

// MN-major operand whose rows (K index) are 128 bytes = 64 elements of the MN dimension, written by
// TMA with SWIZZLE_128B: 8-row groups are 1024 B apart, the next 64 MN elements are `lbo` bytes away.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t lbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(lbo_bytes >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// bf16 x bf16 -> fp32, A K-major, B MN-major
__host__ __device__ constexpr uint32_t umma_idesc_bf16_bmn(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct Tile {
  int h, q0, qs, q_len, seq_len, req, kv_begin, kv_end, n;      // n: chunks
};
__device__ __forceinline__ int tiles_of(const Params& p, int i) {
  return i < p.req_end ? (max(0, p.qsl[i + 1] - p.qsl[i]) + p.BQ - 1) / p.BQ : 0;
}
// Item w of total * Hkv: heads next to each other (they share the block table), late positions, which see the most keys,
// first.  Called by whole warps.
__device__ __forceinline__ Tile find_tile(const Params& p, int w, int total, int lane) {
  Tile t;
  t.h = w % p.Hkv;
  int tile = total - 1 - w / p.Hkv;
  t.req = p.req_begin;
  t.q0 = 0;
  for (int b = p.req_begin; b < p.req_end; b += 32) {
    const int n = tiles_of(p, b + lane);
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int sum = __shfl_sync(0xffffffffu, incl, 31);
    if (tile < sum) {
      const int src = __ffs(__ballot_sync(0xffffffffu, incl > tile)) - 1;
      t.req = b + src;
      t.q0 = (tile - __shfl_sync(0xffffffffu, incl - n, src)) * p.BQ;
      break;
    }
    tile -= sum;
  }
  t.qs = p.qsl[t.req];
  t.q_len = p.qsl[t.req + 1] - t.qs;
  t.seq_len = p.seq_lens[t.req];
  const int ctx = t.seq_len - t.q_len;
  // causal bound of the tile; the whole sequence without the mask
  t.kv_end = t.seq_len > 0 ? (p.non_causal ? t.seq_len : min(t.seq_len, ctx + t.q0 + p.BQ)) : 0;
  t.kv_begin = t.seq_len > 0 ? first_key(p.window, ctx + t.q0) / BKV * BKV : 0;
  t.n = max(0, (t.kv_end - t.kv_begin + BKV - 1) / BKV);
  return t;
}

// The item of round k for this CTA: rounds go back and forth, so that who had the longest item of one round has the shortest
// of the next (in one direction the first CTAs had the longest of all: 1000
// tokens behind 500, 32 / 8 heads, soft cap, 238 us against 185; 8 x 1024 tokens 185 against 181).
__device__ __forceinline__ int item_of(int k) {
  return k * (int)gridDim.x + (k & 1 ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x);
}

// FIN: the epilogue goes on to what p.fin describes.  CAP: scores are capped; the 64 hyperbolic tangents of a thread are
// taken in two rounds on scores read once more (unrolled over registers they outgrow the instruction cache: 1000 tokens
// behind 500, 32 / 8 heads, 290 us against 238).
template <bool FIN, bool CAP>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                       const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem + SMEM_USED > smem_raw + SMEM_TOTAL) {     // (the base is 1024-byte aligned: nothing is cut off)
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, ST_OK, ST_BAD_INDEX);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SMEM_BAR);
  uint64_t* q_full = bars;                 // [2]
  uint64_t* q_empty = bars + 2;            // [2]
  uint64_t* k_full = bars + 4;             // [2]
  uint64_t* k_empty = bars + 6;            // [2]
  uint64_t* v_full = bars + 8;             // [2]
  uint64_t* v_empty = bars + 10;           // [2]
  uint64_t* s_full = bars + 12;            // [2]
  uint64_t* s_empty = bars + 14;           // [2]
  uint64_t* o_full = bars + 16;            // [2]
  uint64_t* o_empty = bars + 18;           // [2]
  uint64_t* p_full = bars + 20;            // 1
  uint64_t* p_empty = bars + 21;           // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1);
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 8);
      mbar_init(&o_full[i], 1); mbar_init(&o_empty[i], 8);
    }
    mbar_init(p_full, 8);
    mbar_init(p_empty, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  pdl_launch_dependents();
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  int total = 0;
  for (int b = p.req_begin; b < p.req_end; b += 32) total += warp_sum(tiles_of(p, b + lane));
  const int items = total * p.Hkv;

  // Every role walks the same items; chunks (c) and tiles with chunks (nq) are counted on across them, so that the buffers
  // and barriers go on and the next tile is copied and its first scores are formed while this one ends.
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // One chunk = 8 pages of K and 8 of V.  Lane l < 8 owns page l and issues its copies.
    int c = 0, nq = 0;
    bool ok = true;
    for (int k = 0, w; (w = item_of(k)) < items && ok; ++k) {
      const Tile t = find_tile(p, w, total, lane);
      if (t.n == 0) continue;
      const int qb = nq & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&q_empty[qb], ((nq >> 1) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY));
      if (!ok) break;
      ++nq;
      if (lane == 0) {
        mbar_expect_tx(&q_full[qb], TILE_BYTES);
        tma_load_3d(smem + SMEM_Q + qb * TILE_BYTES, &tmQ, &q_full[qb], 0, t.h * p.G, t.qs + t.q0);
        tma_load_3d(smem + SMEM_Q + qb * TILE_BYTES + HALF_BYTES, &tmQ, &q_full[qb], 64, t.h * p.G, t.qs + t.q0);
      }
      const int* bt = p.block_tables + (size_t)t.req * p.max_blocks;
      auto entry = [&](int j) -> int {                // block of page `lane` of chunk j
        const int tok = t.kv_begin + j * BKV + lane * 16, page = tok / p.block_size;
        return lane < 8 && j < t.n && tok < t.kv_end && page < p.max_blocks ? bt[page] : -1;
      };
      // its first K row in the cache as [(blocks, 2, Hkv, bs), D]; V's lies Hkv * bs rows behind
      auto rows = [&](int j, long long blk) -> int {
        const int tok = t.kv_begin + j * BKV + lane * 16;
        const bool seen = lane < 8 && j < t.n && tok < t.kv_end;
        if (!seen) {
          blk = 0;
        } else if (blk < 0 || blk >= p.num_blocks) {
          B200_NOTE_BAD_INDEX();
          blk = 0;
        }
        return (int)((blk * 2 * p.Hkv + t.h) * p.block_size + (seen ? tok % p.block_size : 0));
      };
      auto load = [&](uint64_t* empty, uint64_t* full, int base, int cc, int row) -> bool {
        const int st = cc & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(&empty[st], ((cc >> 1) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY))) return false;
        if (lane == 0) mbar_expect_tx(&full[st], TILE_BYTES);
        __syncwarp();
        if (lane < 8) {
          uint8_t* dst = smem + base + st * TILE_BYTES + lane * 16 * 128;
          tma_load_2d(dst, &tmKV, &full[st], 0, row);
          tma_load_2d(dst + HALF_BYTES, &tmKV, &full[st], 64, row);
        }
        return true;
      };
      // In the order in which the buffers come free: K of a chunk, then V of the one before.  The table entries of the
      // chunk after are on their way meanwhile.
      int here = 0, ahead = rows(0, entry(0)), far = entry(1);
      for (int j = 0; j <= t.n && ok; ++j) {
        if (j < t.n) ok = load(k_empty, k_full, SMEM_K, c + j, ahead);
        if (ok && j > 0) ok = load(v_empty, v_full, SMEM_V, c + j - 1, here + p.Hkv * p.block_size);
        here = ahead;
        ahead = rows(j + 1, far);
        far = entry(j + 2);
      }
      c += t.n;
    }
    if (lane == 0 && *abort_flag)
      for (int it = 0; it < 20000; ++it) __nanosleep(100);
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issuer
    constexpr uint32_t idesc_qk = umma_idesc_bf16(BM, BKV);
    const uint32_t idesc_pv = umma_idesc_bf16_bmn(BM, D) & ~(p.pv_half ? (1u << 7) | (1u << 10) : 0u);
    const uint32_t q_addr = smem_u32(smem + SMEM_Q);
    const uint32_t p_addr = smem_u32(smem + SMEM_P);
    // chunks of the next tile that has any, from round k on (0: none)
    auto next_tile = [&](int& k) -> int {
      for (int w; (w = item_of(k)) < items; ++k) {
        const int n = find_tile(p, w, total, lane).n;
        if (n > 0) return n;
      }
      return 0;
    };
    int k = 0, c = 0, nq = 0, n = next_tile(k);
    bool ok = true, first = true;
    while (n > 0 && ok) {
      ++k;
      const int n_next = next_tile(k);
      if (elect_one()) {
        // scores of chunk cc with the queries of tile qi
        auto issue_qk = [&](int cc, int qi, bool begin, bool last) -> bool {
          const int st = cc & 1;
          const uint32_t ph = (cc >> 1) & 1;
          if (begin && !mbar_wait(&q_full[qi & 1], (qi >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) return false;
          if (!mbar_wait(&s_empty[st], ph ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) return false;
          if (!mbar_wait(&k_full[st], ph, abort_flag, p.status, ST_TIMEOUT_FULL)) return false;
          tc_fence_after();
          const uint64_t qd = umma_desc_k_sw128(q_addr + (qi & 1) * TILE_BYTES);
          const uint64_t kd = umma_desc_k_sw128(smem_u32(smem + SMEM_K + st * TILE_BYTES));
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t off = (ks >> 2) * (HALF_BYTES >> 4) + 2 * (ks & 3);
            umma_f16(tmem_base + st * BKV, qd + off, kd + off, idesc_qk, ks > 0 ? 1u : 0u);
          }
          umma_commit(&k_empty[st]);
          umma_commit(&s_full[st]);
          if (last) umma_commit(&q_empty[qi & 1]);
          return true;
        };
        if (first) ok = issue_qk(c, nq, true, n == 1);
        for (int j = 0; j < n && ok; ++j) {
          // the next scores, of the next tile behind the last chunk, before this chunk's P V
          if (j + 1 < n) ok = issue_qk(c + j + 1, nq, false, j + 2 == n);
          else if (n_next > 0) ok = issue_qk(c + n, nq + 1, true, n_next == 1);
          if (!ok) break;
          const int st = (c + j) & 1;
          const uint32_t ph = ((c + j) >> 1) & 1;
          ok = mbar_wait(&o_empty[st], ph ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY) &&
               mbar_wait(&v_full[st], ph, abort_flag, p.status, ST_TIMEOUT_FULL) &&
               mbar_wait(p_full, (c + j) & 1, abort_flag, p.status, ST_TIMEOUT_FULL);
          if (!ok) break;
          tc_fence_after();
          const uint64_t pd = umma_desc_k_sw128(p_addr);
          const uint64_t vd = umma_desc_mn_sw128(smem_u32(smem + SMEM_V + st * TILE_BYTES), HALF_BYTES);
#pragma unroll
          for (int ks = 0; ks < BKV / 16; ++ks)
            umma_f16(tmem_base + 2 * BKV + st * D, pd + (ks >> 2) * (HALF_BYTES >> 4) + 2 * (ks & 3), vd + ks * (16 * 128 / 16),
                     idesc_pv, ks > 0 ? 1u : 0u);
          umma_commit(&v_empty[st]);
          umma_commit(p_empty);
          umma_commit(&o_full[st]);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      first = false;
      c += n;
      ++nq;
      n = n_next;
    }
  } else {
    // ------------------------------------------------ softmax + output: two threads per row
    // Warps 2-5 own key columns [0, 64) of every chunk and output dims [0, 64), warps 6-9 the other
    // halves (a warp may only touch the TMEM lanes of its quarter, so the pair of a row sits in two
    // warps).  The pair agrees on the chunk's row maximum through shared memory; row sums are combined once at the end.
    // It meets at a named barrier of its two warps (256 arrivals at one mbarrier a chunk took longer).  A failed wait
    // leaves the loops running, with no wait behind it, so that the warps of a pair still meet.
    const int qd = warp & 3;
    const int half = (warp - 2) >> 2;                     // 0: columns 0-63, 1: columns 64-127
    const int row = qd * 32 + lane;                       // TMEM lane = tile row
    constexpr int HC = BKV / 2, HD = D / 2;
    float acc[HD];
    const uint32_t lane_addr = (uint32_t)(qd * 32) << 16;
    uint8_t* p_row = smem + SMEM_P + half * HALF_BYTES + row * 128;      // this thread's 64 keys of P
    float* mx_sh = reinterpret_cast<float*>(smem + SMEM_XCH);           // [2 parity][2 half][128]
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + qd) : "memory"); };
    auto fold = [&](int so, float scale) {           // acc = acc * scale + P V of the buffer, which is free then
      const uint32_t o_addr = tmem_base + 2 * BKV + so * D + half * HD + lane_addr;
#pragma unroll
      for (int c0 = 0; c0 < HD; c0 += 32) {
        uint32_t rv[32];
        tmem_ld_32x32(o_addr + c0, rv);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[c0 + i] = acc[c0 + i] * scale + __uint_as_float(rv[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_empty[so]);
    };
    bool ok = true;
    int c = 0;
    for (int k = 0, w; (w = item_of(k)) < items; ++k) {
      const Tile t = find_tile(p, w, total, lane);
      const int h = t.h, qs = t.qs, q0 = t.q0, nchunks = t.n, kv_end = t.kv_end;
      const int pos_local = row / p.G, head = h * p.G + row % p.G;
      const bool row_ok = t.seq_len > 0 && (q0 + pos_local) < t.q_len;
      const int lim = p.non_causal ? t.seq_len - 1 : t.seq_len - t.q_len + q0 + pos_local;    // last visible key of this row
      const int first = first_key(p.window, max(lim, 0));
#pragma unroll
      for (int i = 0; i < HD; ++i) acc[i] = 0.f;
      float m = -INFINITY, l = 0.f, alpha_prev = 0.f;
      for (int j = 0; j < nchunks; ++j, ++c) {
        const int st = c & 1;
        const int tok0 = t.kv_begin + j * BKV + half * HC;
        if (ok) ok = mbar_wait(&s_full[st], (c >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        // this thread's 64 scores, read once
        uint32_t sc[HC];
        tmem_ld_32x32(tmem_base + st * BKV + half * HC + lane_addr, sc);
        tmem_ld_32x32(tmem_base + st * BKV + half * HC + lane_addr + 32, sc + 32);
        tmem_ld_wait();
        auto scores_read = [&]() {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_empty[st]);
        };
        if constexpr (!CAP) scores_read();
        // columns [c_lo, c_hi) of this thread's 64 are visible to the row (causal limit, end of the
        // sequence, sliding window); most chunks are fully visible
        const int c_hi = min(HC, min(lim, kv_end - 1) - tok0 + 1);
        const int c_lo = max(0, first - tok0);
        const bool cut = c_lo > 0 || c_hi < HC;
        if (cut) {
#pragma unroll
          for (int i = 0; i < HC; ++i)
            if (i < c_lo || i >= c_hi) sc[i] = 0xff800000u;
        }
        // row maximum (raw scores; the scale is positive, the soft-cap monotonic)
        float mx = fmaxf(__uint_as_float(sc[0]), __uint_as_float(sc[1]));
#pragma unroll
        for (int i = 2; i < HC; ++i) mx = fmaxf(mx, __uint_as_float(sc[i]));
        mx_sh[(st * 2 + half) * 128 + row] = mx;
        pair_sync();
        mx = fmaxf(mx, mx_sh[(st * 2 + (half ^ 1)) * 128 + row]);
        if (mx != -INFINITY) {
          mx *= p.scale_log2;
          if constexpr (CAP) mx = p.softcap * tanhf(mx / p.softcap);
        }
        const float m_new = fmaxf(m, mx);
        const float base = m_new == -INFINITY ? 0.f : m_new;
        const float alpha = ex2f(m - base);
        m = m_new;
        // probabilities, row sum, P into shared memory, K-major swizzled
        float ps = 0.f;
        auto pack = [&](float e0, float e1) -> uint32_t {
          ps += e0 + e1;
          if (p.pv_half) {
            const __half2 h2 = __floats2half2_rn(e0, e1);
            return *reinterpret_cast<const uint32_t*>(&h2);
          }
          const __nv_bfloat162 b2 = __floats2bfloat162_rn(e0, e1);
          return *reinterpret_cast<const uint32_t*>(&b2);
        };
        auto put = [&](int cc, const uint32_t* pk) {      // 8 keys
          *reinterpret_cast<uint4*>(p_row + ((cc ^ (row & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        };
        // the P buffer is free once P V of the previous chunk has read it
        auto p_free = [&]() {
          if (c > 0 && ok) ok = mbar_wait(p_empty, (c - 1) & 1, abort_flag, p.status, ST_TIMEOUT_EMPTY);
        };
        if constexpr (CAP) {
          p_free();
#pragma unroll 1
          for (int c0 = 0; c0 < HC; c0 += 32) {
            uint32_t rv[32], pk[16];
            float e[32];
            tmem_ld_32x32(tmem_base + st * BKV + half * HC + lane_addr + c0, rv);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) e[i] = ex2f(p.softcap * tanhf(__uint_as_float(rv[i]) * p.scale_log2 / p.softcap) - base);
            if (cut) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c0 + i < c_lo || c0 + i >= c_hi) e[i] = 0.f;
            }
#pragma unroll
            for (int i = 0; i < 32; i += 2) pk[i >> 1] = pack(e[i], e[i + 1]);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) put((c0 >> 3) + cc, pk + 4 * cc);
          }
          scores_read();
        } else {
          uint32_t pk[HC / 2];
#pragma unroll
          for (int i = 0; i < HC; i += 2)
            pk[i >> 1] = pack(ex2f(fmaf(__uint_as_float(sc[i]), p.scale_log2, -base)),
                              ex2f(fmaf(__uint_as_float(sc[i + 1]), p.scale_log2, -base)));
          p_free();
#pragma unroll
          for (int cc = 0; cc < HC / 8; ++cc) put(cc, pk + 4 * cc);
        }
        l = l * alpha + ps;
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
        // fold the previous chunk's P V into the accumulators while the tensor core works on this one
        if (j > 0) {
          const int so = (c - 1) & 1;
          if (ok) ok = mbar_wait(&o_full[so], ((c - 1) >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
          tc_fence_after();
          fold(so, alpha_prev);
        }
        alpha_prev = alpha;
      }
      if (nchunks > 0) {
        const int so = (c - 1) & 1;
        if (ok) ok = mbar_wait(&o_full[so], ((c - 1) >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        fold(so, alpha_prev);
        // row sum of the pair (each thread summed its 64 columns of every chunk)
        float* l_sh = mx_sh + (c & 1) * 256;          // (the maxima there are those of two chunks ago)
        l_sh[half * 128 + row] = l;
        pair_sync();
        l += l_sh[(half ^ 1) * 128 + row];
        pair_sync();                                  // (the next tile's maxima go there)
      }
      if constexpr (FIN) {
        const float inv = ok && l > 0.f ? 1.f / l : 0.f;
#pragma unroll
        for (int i = 0; i < HD; ++i) acc[i] *= inv;
        const long long tok = qs + q0 + pos_local;
        if (p.fin.lam != nullptr) {
          // the maps of a head are neighbouring rows (lanes): each of the two takes half of this thread's columns
          const bool odd = lane & 1;
          const float lam = *p.fin.lam;
          constexpr int HQ = HD / 2;
          float o[HQ], ss = 0.f;
#pragma unroll
          for (int i = 0; i < HQ; ++i) {
            const float got = __shfl_xor_sync(0xffffffffu, odd ? acc[i] : acc[HQ + i], 1);
            o[i] = odd ? got - lam * acc[HQ + i] : acc[i] - lam * got;
            ss += o[i] * o[i];
          }
          ss += __shfl_xor_sync(0xffffffffu, ss, 1);
          if (nchunks > 0) {
            mx_sh[half * 128 + row] = ss;             // (the row maxima have been read)
            pair_sync();
            ss += mx_sh[(half ^ 1) * 128 + row];
            pair_sync();                              // (the next tile writes its maxima there)
          }
          const float sc = p.fin.keep / sqrtf(ss / (float)p.fin.vdim + p.fin.eps);
          if (ok && row_ok) {
#pragma unroll
            for (int i = 0; i < HQ; ++i) o[i] *= sc;
            const int col = half * HD + (odd ? HQ : 0);
            if (p.fin.gate != nullptr) gate_columns<HQ>(p.fin, tok, head >> 1, col, o);
            __nv_bfloat16* dst = p.out + ((size_t)tok * (p.Hq >> 1) + (head >> 1)) * D + col;
#pragma unroll
            for (int i = 0; i < HQ; i += 8) {
              bf16x8 o8;
#pragma unroll
              for (int u = 0; u < 4; ++u) o8.v[u] = __floats2bfloat162_rn(o[i + 2 * u], o[i + 2 * u + 1]);
              *reinterpret_cast<bf16x8*>(dst + i) = o8;
            }
          }
        } else if (ok && row_ok) {
          if (p.fin.gate != nullptr) gate_columns<HD>(p.fin, tok, head, half * HD, acc);
          __nv_bfloat16* dst = p.out + ((size_t)tok * p.Hq + head) * D + half * HD;
#pragma unroll
          for (int i = 0; i < HD; i += 8) {
            bf16x8 o8;
#pragma unroll
            for (int u = 0; u < 4; ++u) o8.v[u] = __floats2bfloat162_rn(acc[i + 2 * u], acc[i + 2 * u + 1]);
            *reinterpret_cast<bf16x8*>(dst + i) = o8;
          }
        }
      } else if (ok && row_ok) {
        float sc = 1.f;
        if (p.sinks != nullptr) {
          const float sk = p.sinks[head] * 1.4426950408889634f;
          const float n = fmaxf(m, sk);
          sc = (m == -INFINITY) ? 0.f : ex2f(m - n);
          l = l * sc + ex2f(sk - n);
          m = n;
        }
        const float inv = l > 0.f ? sc / l : 0.f;
        __nv_bfloat16* dst = p.out + (size_t)(qs + q0 + pos_local) * p.ldo + head * D + half * HD;
#pragma unroll
        for (int i = 0; i < HD; i += 8) {
          uint4 o;
          __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int u = 0; u < 4; ++u) oh[u] = __floats2bfloat162_rn(acc[i + 2 * u] * inv, acc[i + 2 * u + 1] * inv);
          *reinterpret_cast<uint4*>(dst + i) = o;
        }
        if (p.lse != nullptr && half == 0)
          p.lse[(size_t)(qs + q0 + pos_local) * p.Hq + head] =
              l > 0.f ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Pages of an e4m3 cache expanded exactly, keys to bf16 (as the queries are), values to fp16 (so that the probabilities, of
// the same type in one product, have 11 bits, as in the mma.sync kernel): 0.00167 from the result in 64 bits, 0.0022 with
// bf16 values.  The pages of requests nd, nd + 1, .. lie one behind the other in the new pool; values behind a sequence
// become zeros.  grid (total pages, 2 * Hkv); the block table of the new pool is written along.
__global__ void __launch_bounds__(128) expand_pages_kernel(const uint8_t* __restrict__ kv, uint16_t* __restrict__ dst,
                                                           int* __restrict__ table, const int* __restrict__ block_tables,
                                                           const int* __restrict__ seq_lens, int nd, int requests, int max_blocks,
                                                           int block_size, long long num_blocks, int H2, int pages) {
  pdl_launch_dependents();
  pdl_wait();
  const int to = blockIdx.x, lane = threadIdx.x & 31;
  int r = -1, page = to;
  for (int b = 0; b < requests; b += 32) {
    const int n = b + lane < requests ? (max(0, seq_lens[nd + b + lane]) + block_size - 1) / block_size : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int sum = __shfl_sync(0xffffffffu, incl, 31);
    if (page < sum) {
      const int first = __ffs(__ballot_sync(0xffffffffu, incl > page)) - 1;
      r = nd + b + first;
      page -= __shfl_sync(0xffffffffu, incl - n, first);
      break;
    }
    page -= sum;
  }
  if (r < 0 || page >= pages) return;                 // (lengths are those that the host sized the pool for)
  const int seq = seq_lens[r];
  long long blk = page < max_blocks ? block_tables[(size_t)r * max_blocks + page] : -1;
  if (blk < 0 || blk >= num_blocks) {
    B200_NOTE_BAD_INDEX();
    blk = 0;
  }
  if (blockIdx.y == 0 && threadIdx.x == 0) table[(size_t)r * pages + page] = to;
  const uint4* src = reinterpret_cast<const uint4*>(kv + ((size_t)blk * H2 + blockIdx.y) * block_size * D);
  uint4* d = reinterpret_cast<uint4*>(dst + ((size_t)to * H2 + blockIdx.y) * block_size * D);
  const int rows = seq - page * block_size;
  for (int i = threadIdx.x; i < block_size * (D / 16); i += 128) {
    uint32_t o[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (i / (D / 16) < rows) {
      const uint4 v = src[i];
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint32_t h;
        const uint16_t e = (uint16_t)(w[j >> 1] >> (16 * (j & 1)));
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"(e));
        if (2 * blockIdx.y < H2) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
          const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
          o[j] = *reinterpret_cast<const uint32_t*>(&b);
        } else {
          o[j] = h;
        }
      }
    }
    d[2 * i] = make_uint4(o[0], o[1], o[2], o[3]);
    d[2 * i + 1] = make_uint4(o[4], o[5], o[6], o[7]);
  }
}

}  // namespace fa
}  // namespace b200

using namespace b200;

// Requests [req_begin, req_end) of a ragged batch; num_tiles_64 = sum over them of ceil(q_len / 64)
// (the tile count of 64-row query blocks, from which the grid for 128 / G positions per tile is bounded).
// head_dim 128, q heads per kv head in {1, 2, 4, 8}, block_size a multiple of 16.
static int attn_prefill_tc_impl(const void* q, const void* kv, void* out, float* lse, const int* block_tables,
                                const int* seq_lens, const int* qsl, int req_begin, int req_end, int num_tiles_64,
                                int total_tokens, int max_blocks, int block_size, long long num_blocks, int Hq,
                                int Hkv, int D, float scale, int window, float softcap, const float* sinks,
                                int* status, int non_causal, cudaStream_t stream, const HeadFinish* fin = nullptr,
                                int ldo = 0, int pv_half = 0) {
  if (req_end <= req_begin || num_tiles_64 <= 0) return 0;
  const int G = Hkv > 0 ? Hq / Hkv : 0;
  if (D != 128 || Hq % Hkv || (G != 1 && G != 2 && G != 4 && G != 8) || block_size % 16 || ldo % 8) {
    b200_set_last_error("attn_prefill_tc: head_dim 128, q heads per kv head in {1,2,4,8}, block_size % 16 == 0, rows of 16 bytes",
                        __FILE__, __LINE__);
    return -1;
  }
  fa::Params p;
  memset(&p, 0, sizeof(p));
  p.out = (__nv_bfloat16*)out; p.lse = lse; p.block_tables = block_tables; p.seq_lens = seq_lens; p.qsl = qsl;
  p.sinks = sinks; p.status = status;
  p.max_blocks = max_blocks; p.block_size = block_size; p.Hq = Hq; p.Hkv = Hkv; p.G = G; p.BQ = fa::BM / G;
  p.req_begin = req_begin; p.req_end = req_end; p.window = window; p.num_blocks = num_blocks;
  p.non_causal = non_causal;
  p.pv_half = pv_half;
  p.ldo = ldo > 0 ? ldo : Hq * D;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.softcap = softcap > 0.f ? softcap * 1.4426950408889634f : 0.f;
  CUtensorMap tmQ, tmKV;
  // q [T, Hq, D] as (x = D, y = Hq, z = T); a tile is 64 x G x BQ elements, rows ordered (token, head)
  int rc = b200_make_tmap_3d_bf16(&tmQ, q, (uint64_t)D, (uint64_t)Hq, (uint64_t)total_tokens, (uint64_t)D * 2,
                                  (uint64_t)Hq * D * 2, 64, (uint32_t)G, (uint32_t)p.BQ);
  if (rc) return rc;
  // cache [(blocks, 2, Hkv, block_size), D]; one copy = 16 tokens x 64 elements
  rc = b200_make_tmap_2d(&tmKV, kv, 2, (uint64_t)num_blocks * 2 * Hkv * block_size, (uint64_t)D, (uint64_t)D * 2,
                         16, 64);
  if (rc) return rc;
  static unsigned long long attr_seen = 0, attr_seen_fin = 0, attr_seen_cap = 0;
  if (fin != nullptr) {
    if ((fin->lam != nullptr && G % 2) || fin->vdim < 1 || fin->vdim > D) {
      b200_set_last_error("attn_prefill_tc_heads: pairs of maps within a kv head", __FILE__, __LINE__);
      return -1;
    }
    p.fin = *fin;
    B200_CUDA_CHECK(ensure_dynamic_smem(fa::attn_prefill_tc_kernel<true, false>, fa::SMEM_TOTAL, &attr_seen_fin));
  } else if (p.softcap > 0.f) {
    B200_CUDA_CHECK(ensure_dynamic_smem(fa::attn_prefill_tc_kernel<false, true>, fa::SMEM_TOTAL, &attr_seen_cap));
  } else {
    B200_CUDA_CHECK(ensure_dynamic_smem(fa::attn_prefill_tc_kernel<false, false>, fa::SMEM_TOTAL, &attr_seen));
  }
  // ceil(q_len / BQ) <= ceil(q_len / 64) * (64 / BQ) for BQ <= 64; BQ = 128 needs at most as many tiles
  const long long tiles = (p.BQ >= 64 ? num_tiles_64 : num_tiles_64 * (64 / p.BQ)) * (long long)Hkv;
  int dev = 0, sms = 0;
  B200_CUDA_CHECK(cudaGetDevice(&dev));
  B200_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const dim3 grid((unsigned)(tiles < sms ? tiles : sms));
  auto* kernel = fin != nullptr        ? fa::attn_prefill_tc_kernel<true, false>
                 : p.softcap > 0.f ? fa::attn_prefill_tc_kernel<false, true>
                                   : fa::attn_prefill_tc_kernel<false, false>;
  B200_CUDA_CHECK(launch_pdl(kernel, grid, dim3(fa::NUM_THREADS), (size_t)fa::SMEM_TOTAL, stream, tmQ, tmKV, p));
  return 0;
}

extern "C" int b200_attn_prefill_tc(const void* q, const void* kv, void* out, float* lse, const int* block_tables,
                                    const int* seq_lens, const int* qsl, int req_begin, int req_end,
                                    int num_tiles_64, int total_tokens, int max_blocks, int block_size,
                                    long long num_blocks, int Hq, int Hkv, int D, float scale, int window,
                                    float softcap, const float* sinks, int ldo, int pv_half, int* status,
                                    cudaStream_t stream) {
  return attn_prefill_tc_impl(q, kv, out, lse, block_tables, seq_lens, qsl, req_begin, req_end, num_tiles_64,
                              total_tokens, max_blocks, block_size, num_blocks, Hq, Hkv, D, scale, window, softcap,
                              sinks, status, 0, stream, nullptr, ldo, pv_half);
}

// The pages of requests [nd, nd + requests) of an e4m3 cache [num_blocks, 2, Hkv, block_size, 128] expanded: dst [total, 2,
// Hkv, block_size, 128] for the pages of all of them together, table [nd + requests, pages] for the most of one (its first nd
// rows are left alone).
extern "C" int b200_expand_e4m3_pages(const void* kv, void* dst, int* table, const int* block_tables, const int* seq_lens,
                                      int nd, int requests, int total, int pages, int max_blocks, int block_size,
                                      long long num_blocks, int Hkv, cudaStream_t stream) {
  if (requests <= 0 || total <= 0) return 0;
  if (2 * Hkv > 65535 || (((uintptr_t)kv | (uintptr_t)dst) & 15)) {
    b200_set_last_error("expand_e4m3_pages: aligned pools", __FILE__, __LINE__);
    return -1;
  }
  B200_CUDA_CHECK(launch_pdl(fa::expand_pages_kernel, dim3(total, 2 * Hkv), dim3(128), (size_t)0, stream,
                             (const uint8_t*)kv, (uint16_t*)dst, table, block_tables, seq_lens, nd, requests, max_blocks,
                             block_size, num_blocks, 2 * Hkv, pages));
  return 0;
}

// The same with the epilogue of HeadFinish: out [T, lam ? Hq / 2 : Hq, D].
extern "C" int b200_attn_prefill_tc_heads(const void* q, const void* kv, void* out, const int* block_tables,
                                          const int* seq_lens, const int* qsl, int req_begin, int req_end,
                                          int num_tiles_64, int total_tokens, int max_blocks, int block_size,
                                          long long num_blocks, int Hq, int Hkv, int D, float scale, int window,
                                          const float* lam, const void* gate, int ldg, int vdim, float keep, float eps,
                                          int* status, cudaStream_t stream) {
  const HeadFinish fin{lam, (const __nv_bfloat16*)gate, ldg, vdim, keep, eps};
  return attn_prefill_tc_impl(q, kv, out, nullptr, block_tables, seq_lens, qsl, req_begin, req_end, num_tiles_64,
                              total_tokens, max_blocks, block_size, num_blocks, Hq, Hkv, D, scale, window, 0.f, nullptr,
                              status, 0, stream, &fin);
}

// Bidirectional form (vision encoders, diffusion transformers): each request's q_len equals its seq_len and
// every row sees every key.  No window, soft-cap or sinks.
extern "C" int b200_attn_encoder_tc(const void* q, const void* kv, void* out, float* lse, const int* block_tables,
                                    const int* seq_lens, const int* qsl, int req_begin, int req_end,
                                    int num_tiles_64, int total_tokens, int max_blocks, int block_size,
                                    long long num_blocks, int Hq, int Hkv, int D, float scale, int* status,
                                    cudaStream_t stream) {
  return attn_prefill_tc_impl(q, kv, out, lse, block_tables, seq_lens, qsl, req_begin, req_end, num_tiles_64,
                              total_tokens, max_blocks, block_size, num_blocks, Hq, Hkv, D, scale, 0, 0.f, nullptr,
                              status, 1, stream);
}

// see b200_bad_index_count_attention
extern "C" int b200_bad_index_count_attention_tc(unsigned int* out) {
  B200_TAKE_BAD_INDEX_COUNT(out);
  return 0;
}
