// Dense latent attention of DeepSeek's shape (rows of 512 + 64 values, bf16) on two-SM tensor-core instructions:
// decode, chunked prefill and mixed batches.  Same function as mla_attn_kernel of attention_mla.cu, which keeps the
// other shapes and the top-k form.
//
// What bounds it: 1088 multiply-adds per (query row, key) on 1152 bytes per key.  The mma.sync kernel gives a CTA 16 rows,
// so it reads every key once per 16 rows and the tensor path waits for ldmatrix.  Here 128 rows (all heads of a token, or the
// (token, head) rows of several tokens) meet the keys in one pass.  One CTA cannot hold that: the fp32 output of 128 rows
// is 512 columns, all of its tensor memory.  So a pair of CTAs shares the tile, 64 rows each, with
// tcgen05.mma.cta_group::2, M = 128: an accumulator of N columns then takes N / 2 columns of tensor memory (rows in lanes
// 0-63 for the first N / 2 columns, the same rows in lanes 64-127 for the others).  Per chunk of 128 keys:
//   S = Q K^T   9 panels of 64 dims, N = 128: every CTA stages the panels of its 64 keys;   64 columns, two buffers
//   P           8 warps, a thread holds 32 keys of a row (four threads of a row agree on its maximum through shared
//               memory); bf16, K-major swizzled, in the CTA's own shared memory
//   O += P V    two halves with N = 256: every CTA stages its 256 value columns of all 128 keys (MN-major operand);
//               256 columns, accumulated in place and rescaled there when the maximum of a row grew, while S of the next
//               chunk is computed.  (Rescaling only when it grew by more than 2^8 saves nothing visible and loses the
//               exact weight 1 of the largest score: 0.0020 instead of 0.0018 from the result in 64 bits.)
// Query rows 73.7 KB, K 73.7 KB, V 65.5 KB, P 16.4 KB of shared memory: single buffers, refilled by parts (K in three
// groups of panels, V in two halves) while the other product runs, which leaves a part about 1700 cycles to arrive.
// Persistent: pairs take (tile, split) items from the last request to the first and, in a request, from its last tokens,
// which see the most keys, to its first.  (Decoding requests stand first in a batch: they come last, whatever their length.)
// Two warps copy, one issues, eight compute.
//
// Measured on B200 (CUDA events), 128 heads, mma.sync kernel -> this one: 4 x 2048 prompt tokens 32.5 -> 2.22 ms in short runs, 2.58 in
// long ones under the power cap (71.9 -> 1050 and 905 TFLOP/s), 64 requests of 0.9 to 2 K keys 567 -> 61 us.  A chunk takes about
// 4500 cycles where its products need 2176.  What mattered on the way: one elected thread issues (44 -> 32 cycles per product of N = 128),
// the one arrival a chunk on the leader's barrier releases shared memory at cluster scope (all memory: 2.22 -> 2.73 ms),
// K and V have a copying warp each with the table entries fetched ahead.
//
// Semantics of the reference's dense MLA kernels (reference: src/vllm_torchtpu/kernels/mla/v2/).
#include <cstring>

#include "common.cuh"
#include "gemm_tcgen05.h"

namespace b200 {
namespace mlatc {

constexpr int DQ = 576, L = 512, PANELS = DQ / 64;
constexpr int BK = 128;                               // keys per chunk
constexpr int PANEL = 64 * 128;                       // 64 rows of 128 bytes
constexpr int QUERY_BYTES = PANELS * PANEL, K_GROUP = 3 * PANEL, V_HALF = 2 * BK * 128;
constexpr int SMEM_Q = 0, SMEM_K = SMEM_Q + QUERY_BYTES, SMEM_V = SMEM_K + PANELS * PANEL, SMEM_P = SMEM_V + 2 * V_HALF;
constexpr int SMEM_XCH = SMEM_P + 2 * PANEL;          // [2][4][64] row maxima, row sums at the end
constexpr int SMEM_BAR = SMEM_XCH + 2 * 4 * 64 * 4, SMEM_USED = SMEM_BAR + 256;
constexpr int SMEM_TOTAL = 227 * 1024;
constexpr int THREADS = 96 + 256;
constexpr int TM_O = 128;                             // columns: S at 0 and 64, O from 128 on

struct Params {
  __nv_bfloat16* out;                                 // [T, H, L]
  float* part;                                        // splits > 1: normalised fp32 partials [splits, T, H, L] instead
  float* lse;                                         // [T, H] or null; [splits, T, H] with partials
  const int *block_tables, *seq_lens, *qsl;
  int* status;
  int T, H, num_reqs, max_blocks, block_size, splits;
  long long num_blocks;
  float scale_log2;
};

struct Item {
  int i0, rows, qs, ctx, kv_end, lo, n, req, split;   // lo: first chunk, n: chunks
};

__device__ __forceinline__ int tiles_of(const Params& p, int i) {
  return i < p.num_reqs ? (max(0, p.qsl[i + 1] - p.qsl[i]) * p.H + 127) >> 7 : 0;
}
// tile number -> request and row; called by whole warps
__device__ __forceinline__ Item find_item(const Params& p, int w, int total, int lane) {
  Item it;
  it.split = w % p.splits;
  int tile = total - 1 - w / p.splits;                // late tokens see the most keys: from the last to the first
  it.req = 0;
  it.i0 = 0;
  for (int b = 0; b < p.num_reqs; b += 32) {
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
      it.req = b + src;
      it.i0 = (tile - __shfl_sync(0xffffffffu, incl - n, src)) << 7;
      break;
    }
    tile -= sum;
  }
  it.qs = p.qsl[it.req];
  const int q_len = p.qsl[it.req + 1] - it.qs, kv_len = p.seq_lens[it.req];
  it.ctx = kv_len - q_len;
  it.rows = min(128, q_len * p.H - it.i0);
  it.kv_end = max(0, min(kv_len, it.ctx + (it.i0 + it.rows - 1) / p.H + 1));
  const int all = (it.kv_end + BK - 1) / BK, per = (all + p.splits - 1) / p.splits;
  it.lo = it.split * per;
  it.n = max(0, min(all, it.lo + per) - it.lo);
  return it;
}

// 128-byte swizzle, groups of 8 rows `sbo` bytes apart; MN-major: the next 64 values `lbo` bytes away
__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ void umma_2sm(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
// load into this CTA's shared memory whose bytes complete on the leader's barrier
__device__ __forceinline__ void load_pair(uint8_t* dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// two groups of eight cache rows x some panels of 64 values, [group][panel][8 rows of 128 bytes]
__device__ __forceinline__ void load_boxes(uint8_t* dst, const CUtensorMap* m, uint32_t bar, int panel, int group) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %3, %4, %5}], "
      "[%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(0), "r"(panel), "r"(group)
      : "memory");
}
// The leader's product reads what this thread's warp stored to its own CTA's shared memory: the release has cluster scope,
// and covers shared memory only (one that covers all memory waits about 1000 cycles for the way to L2).
__device__ __forceinline__ void arrive_leader(uint64_t* bar) {
  asm volatile(
      "fence.release.sync_restrict::shared::cta.cluster;\n\t"
      "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa_shared(smem_u32(bar), 0))
      : "memory");
}
// mbar_wait (which acquires at CTA scope) for what threads of the other CTA did before they arrived
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  if (!mbar_wait(bar, parity, abort_flag, status, code)) return false;
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\tselp.b32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 32 bytes a thread: whole sectors
__device__ __forceinline__ void st_global_32(void* d, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(d), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void softmax_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
mla_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
              const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmRow, const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem + SMEM_USED > smem_raw + SMEM_TOTAL) {     // (the base is 1024-byte aligned: nothing is cut off)
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, ST_OK, ST_BAD_INDEX);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SMEM_BAR);
  // in the leader only: both CTAs' copies or warps arrive there
  uint64_t *q_full = bars, *k_full = bars + 1, *v_full = bars + 4, *p_full = bars + 6;
  // in each CTA: the leader's commits arrive on both
  uint64_t *q_empty = bars + 7, *k_empty = bars + 8, *v_empty = bars + 11, *s_full = bars + 13, *p_empty = bars + 15;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank(), pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int i = 0; i < 3; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
    }
    mbar_init(p_full, 16);
    mbar_init(p_empty, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmRow);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_launch_dependents();
  pdl_wait();
  tc_fence_before();
  __syncthreads();
  cluster_arrive_release();                           // the peer's barriers must exist before anything arrives on them
  cluster_wait_acquire();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  int total = 0;
  for (int b = 0; b < p.num_reqs; b += 32) total += warp_sum(tiles_of(p, b + lane));
  const int items = total * p.splits;

  if (warp == 0 || warp == 2) {
    // -------------------------------------------------------- copies (both CTAs): warp 0 queries and K, warp 2 V
    const bool keys = warp == 0;
    const int oob = (int)(p.num_blocks * p.block_size);
    int c = 0, nq = 0;                                // chunks and items so far
    bool ok = true;
    for (int w = pair; w < items && ok; w += npairs) {
      const Item it = find_item(p, w, total, lane);
      if (it.n == 0) continue;
      const int* bt = p.block_tables + (size_t)it.req * p.max_blocks;
      // Lane i holds page i of the 32 pages (16 tokens each) of four chunks; the table entries of the next four are on their
      // way meanwhile.
      auto entry = [&](int j) -> int {
        const int tok = (it.lo + j) * BK + lane * 16, page = tok / p.block_size;
        return tok < it.kv_end && page < p.max_blocks ? bt[page] : -1;
      };
      int ahead = entry(0), row = oob;
      if (keys) {
        ok = __all_sync(0xffffffffu, mbar_wait(q_empty, (nq & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY));
        if (!ok) break;
        ++nq;
        if (rank == 0 && lane == 0) mbar_expect_tx(q_full, 2 * QUERY_BYTES);
        __syncwarp();
        if (lane < PANELS)
          load_pair(smem + SMEM_Q + lane * PANEL, &tmQ, mapa_shared(smem_u32(q_full), 0), lane * 64,
                    it.qs * p.H + it.i0 + rank * 64);
      }
      for (int j = 0; j < it.n && ok; ++j, ++c) {
        if ((j & 3) == 0) {
          // first cache row of the page; out of range (the copy fills zeros) behind the last visible token
          const int tok = (it.lo + j) * BK + lane * 16;
          long long blk = ahead;
          if (tok < it.kv_end && (blk < 0 || blk >= p.num_blocks)) {
            B200_NOTE_BAD_INDEX();
            blk = 0;
          }
          row = tok < it.kv_end ? (int)(blk * p.block_size + tok % p.block_size) : oob;
          if (j + 4 < it.n) ahead = entry(j + 4);
        }
        const int y = __shfl_sync(0xffffffffu, row, (j & 3) * 8 + (keys ? rank * 4 + (lane & 3) : lane & 7));
        if (keys) {
          for (int g = 0; g < 3 && ok; ++g) {
            ok = __all_sync(0xffffffffu, mbar_wait(&k_empty[g], (c & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY));
            if (!ok) break;
            if (rank == 0 && lane == 0) mbar_expect_tx(&k_full[g], 2 * K_GROUP);
            __syncwarp();
            if (lane < 4)
              load_boxes(smem + SMEM_K + g * K_GROUP + lane * 6144, &tmK, mapa_shared(smem_u32(&k_full[g]), 0), 3 * g, y >> 3);
          }
        } else {
          // rows behind the last visible token are filled with zeros: their probabilities are zero, the product must be
          // zero whatever the cache holds there.  Whole pages come from an out-of-range row, the ragged one row by row.
          const int left = it.kv_end - (it.lo + j) * BK, part = left < BK && (left & 15) ? left >> 4 : 8;
          const int y0 = __shfl_sync(0xffffffffu, y, part & 7);
          for (int h = 0; h < 2 && ok; ++h) {
            ok = __all_sync(0xffffffffu, mbar_wait(&v_empty[h], (c & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY));
            if (!ok) break;
            if (rank == 0 && lane == 0) mbar_expect_tx(&v_full[h], 2 * V_HALF);
            __syncwarp();
            const uint32_t bar = mapa_shared(smem_u32(&v_full[h]), 0);
            uint8_t* dst = smem + SMEM_V + h * V_HALF;
            if (lane < 8 && lane != part) load_boxes(dst + lane * 4096, &tmV, bar, rank * 4 + h * 2, y >> 3);
            if (part < 8) {
              const int i = lane & 15, pn = lane >> 4;
              load_pair(dst + part * 4096 + (i >> 3) * 2048 + pn * 1024 + (i & 7) * 128, &tmRow, bar,
                        (rank * 4 + h * 2 + pn) * 64, i < (left & 15) ? y0 + i : oob);
            }
          }
        }
      }
    }
    if (*abort_flag)                                  // copies in flight get a bounded time to land
      for (int i = 0; i < 20000; ++i) __nanosleep(100);
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------------ products (leader)
    if (rank == 0) {
      constexpr uint32_t idesc_qk = umma_idesc_bf16(128, BK), idesc_pv = umma_idesc_bf16(128, 256) | (1u << 16);
      const uint64_t q_desc = umma_desc_k_sw128(smem_u32(smem + SMEM_Q)), k_desc = desc_sw128(smem_u32(smem + SMEM_K), 16, 3072);
      const uint64_t p_desc = umma_desc_k_sw128(smem_u32(smem + SMEM_P));
      const uint64_t v_desc = desc_sw128(smem_u32(smem + SMEM_V), 1024, 2048);
      int c = 0, nq = 0;
      bool ok = true;
      for (int w = pair; w < items && ok; w += npairs) {
        const Item it = find_item(p, w, total, lane);
        if (it.n == 0) continue;
        if (elect_one()) {
          auto scores = [&](int j) -> bool {
            const int cc = c + j, b = cc & 1;
            for (int g = 0; g < 3; ++g) {
              if (!mbar_wait(&k_full[g], cc & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) return false;
              tc_fence_after();
#pragma unroll
              for (int x = 0; x < 12; ++x) {
                const int pn = x >> 2;
                umma_2sm(tmem + b * 64, q_desc + (3 * g + pn) * (PANEL >> 4) + 2 * (x & 3),
                         k_desc + ((g * K_GROUP + pn * 1024) >> 4) + 2 * (x & 3), idesc_qk, g > 0 || x > 0 ? 1u : 0u);
              }
              commit_pair(&k_empty[g]);
            }
            commit_pair(&s_full[b]);
            if (j + 1 == it.n) commit_pair(q_empty);
            return true;
          };
          ok = mbar_wait(q_full, nq & 1, abort_flag, p.status, ST_TIMEOUT_FULL) && scores(0);
          for (int j = 0; j < it.n && ok; ++j) {
            if (j + 1 < it.n && !(ok = scores(j + 1))) break;
            const int cc = c + j;
            // P is there, the scores that it is made of have been read and so has the output of the item before
            if (!(ok = wait_cluster(p_full, cc & 1, abort_flag, p.status, ST_TIMEOUT_FULL))) break;
            for (int h = 0; h < 2 && ok; ++h) {
              if (!(ok = mbar_wait(&v_full[h], cc & 1, abort_flag, p.status, ST_TIMEOUT_FULL))) break;
              tc_fence_after();
#pragma unroll
              for (int x = 0; x < 8; ++x)
                umma_2sm(tmem + TM_O + h * 128, p_desc + (x >> 2) * (PANEL >> 4) + 2 * (x & 3),
                         v_desc + ((h * V_HALF + x * 4096) >> 4), idesc_pv, j > 0 || x > 0 ? 1u : 0u);
              commit_pair(&v_empty[h]);
            }
            if (ok) commit_pair(p_empty);             // P is free, and O holds this chunk
          }
        }
        ok = __all_sync(0xffffffffu, ok);
        c += it.n;
        ++nq;
      }
    }
  } else {
    // ------------------------------------------------------------------------------------------ softmax and output
    // A failed wait leaves the loops running (every wait then returns at once), so that the warps still meet.
    const int ln = (warp & 3) * 32 + lane;            // lane of the tensor memory
    const int r = ln & 63, kh = ln >> 6, sh = (warp - 3) >> 2;
    const int part = kh * 2 + sh;                     // which 32 of the 128 keys
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    float* xch = reinterpret_cast<float*>(smem + SMEM_XCH);
    uint8_t* p_row = smem + SMEM_P + kh * PANEL + r * 128;
    int c = 0;
    bool ok = true;
    for (int w = pair; w < items; w += npairs) {
      const Item it = find_item(p, w, total, lane);
      const int i = it.i0 + rank * 64 + r;            // (token, head) row of the request
      const bool row_ok = rank * 64 + r < it.rows;
      const int lim = row_ok ? it.ctx + i / p.H : -1; // last visible key
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < it.n; ++j, ++c) {
        const int b = c & 1;
        if (ok) ok = mbar_wait(&s_full[b], (c >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        uint32_t s[32];
        tmem_ld_32x32(tmem + lane_addr + b * 64 + sh * 32, s);
        tmem_ld_wait();
        const int seen = lim - ((it.lo + j) * BK + part * 32) + 1;       // visible keys among these 32
        if (seen < 32) {
#pragma unroll
          for (int x = 0; x < 32; ++x)
            if (x >= seen) s[x] = 0xff800000u;
        }
        float mx = __uint_as_float(s[0]);
#pragma unroll
        for (int x = 1; x < 32; ++x) mx = fmaxf(mx, __uint_as_float(s[x]));
        float* row_mx = xch + b * 256 + r;
        row_mx[part * 64] = mx;
        softmax_sync();
        mx = fmaxf(fmaxf(row_mx[0], row_mx[64]), fmaxf(row_mx[128], row_mx[192])) * p.scale_log2;
        float alpha = 1.f;
        if (mx > m) {
          alpha = ex2(m - mx);                        // (0 for the first visible chunk)
          l *= alpha;
          m = mx;
        }
        const float base = m == -INFINITY ? 0.f : m;
        float sum = 0.f;
        uint32_t pk[16];
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          const float e0 = ex2(fmaf(__uint_as_float(s[x]), p.scale_log2, -base));
          const float e1 = ex2(fmaf(__uint_as_float(s[x + 1]), p.scale_log2, -base));
          const __nv_bfloat162 e = __floats2bfloat162_rn(e0, e1);
          pk[x >> 1] = *reinterpret_cast<const uint32_t*>(&e);
          // the sum takes the rounded values that the product takes: the weights of a row add up to one
          sum += __uint_as_float(pk[x >> 1] << 16) + __uint_as_float(pk[x >> 1] & 0xffff0000u);
        }
        l += sum;
        // the product of the chunk before has read P and is in O
        if (c > 0 && ok) ok = mbar_wait(p_empty, (c - 1) & 1, abort_flag, p.status, ST_TIMEOUT_EMPTY);
        if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
          tc_fence_after();
#pragma unroll 1
          for (int x = 0; x < 128; x += 64) {
            const uint32_t a = tmem + lane_addr + TM_O + sh * 128 + x;
            uint32_t o[64];
            tmem_ld_32x32(a, o);
            tmem_ld_32x32(a + 32, o + 32);
            tmem_ld_wait();
#pragma unroll
            for (int y = 0; y < 64; ++y) o[y] = __float_as_uint(__uint_as_float(o[y]) * alpha);
            tmem_st_32x32(a, o);
            tmem_st_32x32(a + 32, o + 32);
          }
          tmem_st_wait();
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
          *reinterpret_cast<uint4*>(p_row + (((sh * 4 + x) ^ (r & 7)) << 4)) =
              make_uint4(pk[4 * x], pk[4 * x + 1], pk[4 * x + 2], pk[4 * x + 3]);
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_leader(p_full);
      }
      // ---- row sums, output
      const size_t row = (size_t)it.qs * p.H + i;
      if (it.n > 0) {
        softmax_sync();                               // the maxima have been read
        xch[part * 64 + r] = l;
        softmax_sync();
        l = xch[r] + xch[64 + r] + xch[128 + r] + xch[192 + r];
        softmax_sync();
        if (ok) ok = mbar_wait(p_empty, (c - 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        const float inv = l > 0.f ? 1.f / l : 0.f;
        const size_t col = kh * 256 + sh * 128;
#pragma unroll 1
        for (int x = 0; x < 128; x += 64) {
          uint32_t o[64];
          tmem_ld_32x32(tmem + lane_addr + TM_O + sh * 128 + x, o);
          tmem_ld_32x32(tmem + lane_addr + TM_O + sh * 128 + x + 32, o + 32);
          tmem_ld_wait();
          if (!ok || !row_ok) continue;
          if (p.splits > 1) {
            float* d = p.part + ((size_t)it.split * p.T * p.H + row) * L + col + x;
#pragma unroll
            for (int y = 0; y < 64; y += 8) {
#pragma unroll
              for (int u = 0; u < 8; ++u) o[y + u] = __float_as_uint(__uint_as_float(o[y + u]) * inv);
              st_global_32(d + y, o + y);
            }
          } else {
            __nv_bfloat16* d = p.out + row * L + col + x;
#pragma unroll
            for (int y = 0; y < 64; y += 16) {
              uint32_t v[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const __nv_bfloat162 e =
                    __floats2bfloat162_rn(__uint_as_float(o[y + 2 * u]) * inv, __uint_as_float(o[y + 2 * u + 1]) * inv);
                v[u] = *reinterpret_cast<const uint32_t*>(&e);
              }
              st_global_32(d + y, v);
            }
          }
        }
      } else if (row_ok && p.splits == 1) {           // a request without keys
        uint4* d = reinterpret_cast<uint4*>(p.out + row * L + part * 128);
        for (int x = 0; x < 16; ++x) d[x] = make_uint4(0u, 0u, 0u, 0u);
      }
      if (p.lse != nullptr && part == 0 && row_ok)
        p.lse[(size_t)it.split * p.T * p.H + row] = l > 0.f ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
    // rows behind the step's tokens: zeros (partials: no keys seen)
    const size_t first = (size_t)max(0, p.qsl[p.num_reqs]) * p.H, all = (size_t)p.T * p.H;
    for (size_t f = first + (size_t)blockIdx.x * 8 + warp - 3; f < all; f += (size_t)gridDim.x * 8) {
      if (p.splits == 1) {
        uint4* d = reinterpret_cast<uint4*>(p.out + f * L);
        d[lane] = d[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
      }
      if (p.lse != nullptr)
        for (int s = lane; s < p.splits; s += 32) p.lse[(size_t)s * all + f] = -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_arrive_release();                           // the pair is done with each other's memory
  cluster_wait_acquire();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// out[row] = sum over the splits of softmax(lse) * part; one CTA of 128 threads per (token, head) row.  A row whose splits
// all saw no key keeps zeros and lse = -inf.
__global__ void __launch_bounds__(128) mla_tc_merge_kernel(const float* __restrict__ part, const float* __restrict__ part_lse,
                                                           __nv_bfloat16* __restrict__ out, float* __restrict__ lse, int splits,
                                                           int rows) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t row = blockIdx.x;
  const int col = threadIdx.x * 4;
  float mx = -INFINITY;
  for (int s = 0; s < splits; ++s) mx = fmaxf(mx, part_lse[(size_t)s * rows + row]);
  float den = 0.f, a[4] = {0.f, 0.f, 0.f, 0.f};
  for (int s = 0; s < splits; ++s) {
    const float v = part_lse[(size_t)s * rows + row];
    if (v == -INFINITY) continue;
    const float e = __expf(v - mx);
    const float4 x = *reinterpret_cast<const float4*>(part + ((size_t)s * rows + row) * L + col);
    den += e;
    a[0] = fmaf(e, x.x, a[0]); a[1] = fmaf(e, x.y, a[1]); a[2] = fmaf(e, x.z, a[2]); a[3] = fmaf(e, x.w, a[3]);
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  __nv_bfloat162* d = reinterpret_cast<__nv_bfloat162*>(out + row * L + col);
  d[0] = __floats2bfloat162_rn(a[0] * inv, a[1] * inv);
  d[1] = __floats2bfloat162_rn(a[2] * inv, a[3] * inv);
  if (lse != nullptr && threadIdx.x == 0) lse[row] = den > 0.f ? mx + __logf(den) : -INFINITY;
}

}  // namespace mlatc
}  // namespace b200

using namespace b200;

// q [T, H, 576], cache [num_blocks, block_size, 576], both 16-byte aligned; block_size a multiple of 16; out [T, H, 512], lse
// [T, H] or null.  splits > 1: part [splits, T, H, 512] and part_lse [splits, T, H] fp32 are scratch of the caller.
extern "C" int b200_mla_attention_tc(const void* q, const void* cache, void* out, float* lse, const int* block_tables,
                                     const int* seq_lens, const int* qsl, int T, int num_reqs, int H, int max_blocks,
                                     int block_size, long long num_blocks, float scale, int splits, float* part,
                                     float* part_lse, int* status, int num_sms, cudaStream_t stream) {
  if (T <= 0 || num_reqs <= 0 || H <= 0) return 0;
  if (block_size % 16 || splits < 1 || (splits > 1 && (part == nullptr || part_lse == nullptr)) ||
      num_blocks * block_size > 0x7ffffff0ll || (long long)T * H > 0x7ffffff0ll ||
      ((uintptr_t)q | (uintptr_t)cache) & 15 || ((uintptr_t)out | (uintptr_t)part) & 31) {
    b200_set_last_error("mla_attention_tc: pages of 16 rows, aligned tensors and scratch for the partials required", __FILE__,
                        __LINE__);
    return -1;
  }
  CUtensorMap tmQ, tmK, tmV, tmRow;
  const uint64_t rows = (uint64_t)num_blocks * block_size, ld = mlatc::DQ * 2;
  int rc = b200_make_tmap_2d(&tmQ, q, 2, (uint64_t)T * H, mlatc::DQ, ld, 64, 64);
  // the cache as [groups of 8 rows][panels of 64 values][8 rows][64 values]
  const uint64_t dims[4] = {64, 8, mlatc::PANELS, rows / 8}, strides[3] = {ld, 128, 8 * ld};
  const uint32_t box_k[4] = {64, 8, 3, 2}, box_v[4] = {64, 8, 2, 2};
  if (!rc) rc = b200_make_tmap_4d_bf16(&tmK, cache, dims, strides, box_k);
  if (!rc) rc = b200_make_tmap_4d_bf16(&tmV, cache, dims, strides, box_v);
  if (!rc) rc = b200_make_tmap_2d(&tmRow, cache, 2, rows, mlatc::DQ, ld, 1, 64);
  if (rc) return rc;
  mlatc::Params p;
  memset(&p, 0, sizeof(p));
  p.out = (__nv_bfloat16*)out; p.part = part; p.lse = splits > 1 ? part_lse : lse; p.block_tables = block_tables; p.seq_lens = seq_lens; p.qsl = qsl;
  p.status = status; p.T = T; p.H = H; p.num_reqs = num_reqs; p.max_blocks = max_blocks; p.block_size = block_size;
  p.num_blocks = num_blocks; p.splits = splits; p.scale_log2 = scale * 1.4426950408889634f;
  static unsigned long long seen = 0;
  B200_CUDA_CHECK(ensure_dynamic_smem(mlatc::mla_tc_kernel, mlatc::SMEM_TOTAL, &seen));
  // every request adds at most one tile to those of its rows
  const long long items = ((long long)T * H / 128 + num_reqs) * splits;
  const long long pairs = num_sms / 2 < items ? num_sms / 2 : items;
  B200_CUDA_CHECK(launch_pdl(mlatc::mla_tc_kernel, dim3((unsigned)(2 * pairs)), dim3(mlatc::THREADS),
                             (size_t)mlatc::SMEM_TOTAL, stream, tmQ, tmK, tmV, tmRow, p));
  if (splits > 1)
    B200_CUDA_CHECK(launch_pdl(mlatc::mla_tc_merge_kernel, dim3((unsigned)(T * H)), dim3(128), (size_t)0, stream,
                               (const float*)part, (const float*)part_lse, (__nv_bfloat16*)out, lse, splits, T * H));
  return 0;
}

// see b200_bad_index_count_attention
extern "C" int b200_bad_index_count_attention_mla_tc(unsigned int* out) {
  B200_TAKE_BAD_INDEX_COUNT(out);
  return 0;
}
