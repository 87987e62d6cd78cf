// Flash-attention backward for sm_100a (head_dim 128, bf16 in, fp32 accumulate), two kernels:
//
//  dkdv kernel  one CTA per (128-row KV tile, KV head): K and V stay in shared memory, the CTA
//               streams every (query head of the group, Q tile) pair that can see the tile and keeps
//               dK and dV in TMEM the whole time. It computes the *transposed* scores
//               S^T = K Q^T and dP^T = V dO^T so that P^T and dS^T land in TMEM with KV rows on the
//               lanes, which is exactly the A operand of dV += P^T dO and dK += dS^T Q.
//               The result is added to fp32 dK/dV with red.add (system scope): the destination may
//               be a peer GPU's buffer, which is how a ring step returns gradients to the KV owner.
//               (kv_overwrite: written instead, in fp32 or bf16, when nothing else adds to it.)
//  dq kernel    one CTA per (Q tile, query head): S = Q K^T, dP = dO V^T, dQ += dS K with dS fed
//               from TMEM; deterministic, no atomics.
//
// Both kernels cut a 128 x 128 item into two halves of 64 columns (queries / keys), each with eight compute warps and
// its own score and dP columns in TMEM, and issue from two warps. A half is a dependency cycle scores -> exponentials
// -> product -> next scores; with a single 128-wide cycle the tensor core waited for the exponentials and the
// exponentials for the tensor core (3,620 clk per item in the dK/dV kernel against 2,048 of MMA time), the two halves
// run in opposite phases (2,830 clk). The price is 64-wide products with both operands in shared memory, which run at
// 48 clk per step instead of 32 (6 KB at 128 B/clk): 2,480 clk of MMA time per item in the dK/dV kernel, whose TMEM is
// full. The dQ kernel has room for Q and dO in TMEM and pays nothing (2,110 -> 1,740 clk per item, MMA time 1,536).
// Kernel times, 32 heads over 8 KV heads, causal (before -> now): dK/dV 1,140 -> 797 us at 8,192 tokens, 16.2 -> 13.4 ms
// at 32,768; dQ 709 -> 620 us and 11.0 -> 9.4 ms (the GPU runs at its power cap at 32,768, 1.5 GHz); with a 4,096-token
// window over 65,536 tokens dK/dV 14.6 -> 8.2 ms, dQ 8.9 ms.
// Exponentials are the special-function unit's: taking every second pair as a polynomial on the FMA pipe made no difference
// (28.4 -> 29.1 ms for the whole backward at 32,768 tokens at the time), since instruction issue and the cycle of an item
// bound these kernels.
// All waits are bounded.
#include "../common/ptx.cuh"
#include "../common/device_once.h"
#include "../common/tma_host.h"
#include "attn.h"
#include "dkdv_waits.h"
#include "tile_iter.cuh"
#include "work_order.h"

namespace zx {

void check_attn_common(int Hq, int Hkv, int Sq, int Skv, const AttnLayout& ql, const AttnLayout& kl);

namespace {

constexpr int HD = 128;
constexpr int BT = 128;                    // tile edge in tokens (both Q and KV)
constexpr int TILE_BYTES = BT * HD * 2;    // 32 KB
constexpr int HALF_BYTES = TILE_BYTES / 2; // one 64-wide d chunk
constexpr int HALF_Q = 64 * 128;           // 64 rows of a d chunk: start of a tile's second half of tokens
constexpr int TMEM_COLS = 512;
constexpr float LOG2E = 1.4426950408889634f;

struct BwdParams {
  int B, Hq, Hkv, Sq, Skv;
  float scale, scale_log2;
  int causal, window_blocks, global_every;
  int n_q_tiles, n_kv_tiles;
  int q_tiles_per_chunk, kv_tiles_per_chunk, n_q_chunks, n_kv_chunks;
  int kv_heads_per_group, q_heads_per_group;   // block order, see work_item
  int q_chunk_pos[kAttnMaxChunks];
  int kv_chunk_pos[kAttnMaxChunks];
  const float* lse;
  const float* delta;
  float* dq;
  float* dk;
  float* dv;
  int dq_accumulate, kv_overwrite, out_bf16;
  const uint4* pull_src;
  uint4* pull_dst;
  size_t pull_nvec;
  long long* trace;
  Status* status;
};

// Clock stamps of pipeline events into the caller's trace buffer (first CTA of the dK/dV kernel). Compiled in only
// with -DZX_BWD_TRACE: the stamps cost issue slots in loops that are bound by instruction issue.
#ifdef ZX_BWD_TRACE
#define ZX_TRACE_DKDV(iter, slot)                                                     \
  do {                                                                                \
    if (p.trace != nullptr && blockIdx.x == 0 && (iter) < 64) p.trace[1024 + (iter) * 16 + (slot)] = clock64(); \
  } while (0)
#else
#define ZX_TRACE_DKDV(iter, slot) do { } while (0)
#endif

__device__ __forceinline__ int q_tile_pos(const BwdParams& p, int t) {
  return p.q_chunk_pos[t / p.q_tiles_per_chunk] + (t % p.q_tiles_per_chunk) * BT;
}
__device__ __forceinline__ int kv_tile_pos(const BwdParams& p, int j) {
  return p.kv_chunk_pos[j / p.kv_tiles_per_chunk] + (j % p.kv_tiles_per_chunk) * BT;
}
// The Q tiles that may attend the KV tile at position kpos0, in order. Positions grow with the tile index inside a
// chunk, so without a window the visible tiles of a chunk are its last ones and the walk starts at the first of them
// (a walk that tests every tile from 0 costs a late KV tile several microseconds before its first load, in every
// role); windowed masks use the jumping search. `count` is the number of tiles `next` will return.
template <bool SPARSE>
struct QWalk {
  int t, qpos0, left, c;
  __device__ __forceinline__ void init() { t = -1; qpos0 = 0; left = 0; c = -1; }
  // first visible tile of chunk c
  static __device__ __forceinline__ int first_in_chunk(const BwdParams& p, int c, int kpos0) {
    const int d = p.causal ? (kpos0 - p.q_chunk_pos[c]) / BT : 0;
    return d < 0 ? 0 : (d < p.q_tiles_per_chunk ? d : p.q_tiles_per_chunk);
  }
  __device__ __forceinline__ bool next(const BwdParams& p, int kpos0) {
    if constexpr (SPARSE) {
      t = next_q_tile(p, kpos0, t + 1);
      if (t >= p.n_q_tiles) return false;
      qpos0 = q_tile_pos(p, t);
      return true;
    } else {
      ++t;
      qpos0 += BT;
      while (left == 0) {
        if (++c >= p.n_q_chunks) return false;
        const int i = first_in_chunk(p, c, kpos0);
        left = p.q_tiles_per_chunk - i;
        t = c * p.q_tiles_per_chunk + i;
        qpos0 = p.q_chunk_pos[c] + i * BT;
      }
      --left;
      return true;
    }
  }
  static __device__ __forceinline__ int count(const BwdParams& p, int kpos0) {
    int n = 0;
    if constexpr (SPARSE) {
      QWalk w;
      for (w.init(); w.next(p, kpos0);) ++n;
    } else {
      for (int c = 0; c < p.n_q_chunks; ++c) n += p.q_tiles_per_chunk - first_in_chunk(p, c, kpos0);
    }
    return n;
  }
};
// The KV tiles the Q tile at position qpos0 may attend, in order: without a window the first ones of each chunk.
template <bool SPARSE>
struct KvWalk {
  int j, kpos0, left, c;
  __device__ __forceinline__ void init() { j = -1; kpos0 = 0; left = 0; c = -1; }
  static __device__ __forceinline__ int in_chunk(const BwdParams& p, int c, int qpos0) {
    if (!p.causal) return p.kv_tiles_per_chunk;
    const int d = qpos0 - p.kv_chunk_pos[c];
    return d < 0 ? 0 : (d / BT + 1 < p.kv_tiles_per_chunk ? d / BT + 1 : p.kv_tiles_per_chunk);
  }
  __device__ __forceinline__ bool next(const BwdParams& p, int qpos0) {
    if constexpr (SPARSE) {
      j = next_kv_tile(p, qpos0, j + 1);
      if (j >= p.n_kv_tiles) return false;
      kpos0 = kv_tile_pos(p, j);
      return true;
    } else {
      ++j;
      kpos0 += BT;
      while (left == 0) {
        if (++c >= p.n_kv_chunks) return false;
        left = in_chunk(p, c, qpos0);
        j = c * p.kv_tiles_per_chunk;
        kpos0 = p.kv_chunk_pos[c];
      }
      --left;
      return true;
    }
  }
  static __device__ __forceinline__ int count(const BwdParams& p, int qpos0) {
    int n = 0;
    if constexpr (SPARSE) {
      KvWalk w;
      for (w.init(); w.next(p, qpos0);) ++n;
    } else {
      for (int c = 0; c < p.n_kv_chunks; ++c) n += in_chunk(p, c, qpos0);
    }
    return n;
  }
};

__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const bool ok = mbar_wait(bar, parity, abort_flag);
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void red_add_v4_sys(float* addr, float a, float b, float c, float d) {
  asm volatile("red.relaxed.sys.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

// One warp's 32 rows x 32 columns of an accumulator (row = lane) into a slab of shared memory and from there to global
// memory through the TMA unit, which writes whole lines; rows are swizzled so that the 16-byte writes of eight lanes
// fall into different banks. (Thread-per-row stores, 16 bytes of 32 rows per instruction, took 4 to 6 us at the end of
// every block.) The caller waits for the store before the block ends.
constexpr int SLAB_BYTES = 32 * 128;
__device__ __forceinline__ void store_slab(const CUtensorMap* m, uint8_t* slab, const uint32_t* a, float scale, int bf16,
                                           int lane, int col, int head, int row, int batch) {
  if (bf16) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        w[e] = pack_bf16x2(__uint_as_float(a[8 * c + 2 * e]) * scale, __uint_as_float(a[8 * c + 2 * e + 1]) * scale);
      *reinterpret_cast<uint4*>(slab + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      *reinterpret_cast<float4*>(slab + lane * 128 + ((c ^ (lane & 7)) << 4)) =
          make_float4(__uint_as_float(a[4 * c]) * scale, __uint_as_float(a[4 * c + 1]) * scale,
                      __uint_as_float(a[4 * c + 2]) * scale, __uint_as_float(a[4 * c + 3]) * scale);
  }
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    tma_store_4d(m, slab, col, head, row, batch);
    tma_store_commit();
  }
}

// Base descriptors of a [128 x 128] bf16 tile (built once per tile address) ...
__device__ __forceinline__ uint64_t base_kmajor(uint32_t tile_addr) { return make_smem_desc_sw128(tile_addr, 16, 1024); }
__device__ __forceinline__ uint64_t base_mnmajor(uint32_t tile_addr) {
  return make_smem_desc_sw128(tile_addr, HALF_BYTES, 1024);
}
// ------------------------------------------------------------------------------------------
// delta[b, h, s] = sum_d dO * O
// ------------------------------------------------------------------------------------------
// Bound by memory: one warp takes eight consecutive tokens of one head (two 256-byte rows per load instruction, all
// eight loads of a lane in flight, eight neighbouring results per store). O_VEC: 16-byte loads of o, or two of 8 bytes for
// an o that starts in the middle of a 16-byte unit (d_o is also read by TMA, which takes whole units only).
constexpr int DELTA_TOKENS = 8;
template <typename O_VEC>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o,
                                                         const __nv_bfloat16* __restrict__ d_o,
                                                         float* __restrict__ delta, int S, int H, int n_groups) {
  const int group = blockIdx.x * 8 + (threadIdx.x >> 5);   // (b, s / 8, h)
  if (group >= n_groups) return;
  const int lane = threadIdx.x & 31, sub = lane >> 4;
  const int h = group % H, bs = group / H;   // bs: eighth of a token row over all batches (S is a multiple of 128)
  const size_t row0 = ((size_t)bs * DELTA_TOKENS + sub) * H + h;
  uint4 a[4], g[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t off = (row0 + (size_t)2 * i * H) * (HD / 8) + (lane & 15);
    if constexpr (sizeof(O_VEC) == 16) {
      a[i] = __ldg(reinterpret_cast<const uint4*>(o) + off);
    } else {
      const uint2 lo = __ldg(reinterpret_cast<const uint2*>(o) + 2 * off), hi = __ldg(reinterpret_cast<const uint2*>(o) + 2 * off + 1);
      a[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
    g[i] = __ldg(reinterpret_cast<const uint4*>(d_o) + off);
  }
  float out = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t aw[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = unpack_bf16x2(aw[e]), y = unpack_bf16x2(gw[e]);
      acc += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    // token 2 i + sub of the group: lanes 0..7 end up with one token each
    const float other = __shfl_xor_sync(0xffffffffu, acc, 16);
    if ((lane >> 1) == i) out = (lane & 1) == sub ? acc : other;
  }
  if (lane < DELTA_TOKENS) {
    const int per_batch = S / DELTA_TOKENS;
    const int b = bs / per_batch, s = (bs % per_batch) * DELTA_TOKENS + lane;
    delta[((size_t)b * H + h) * S + s] = out;
  }
}

// ------------------------------------------------------------------------------------------
// dK / dV
// ------------------------------------------------------------------------------------------
// Q lives until dK of its item has been issued, dO only until dV: a 3-deep Q ring and a 2-deep dO
// ring free every slot a full iteration before its next tile is needed, which hides the TMA latency.
constexpr int Q_STAGES = 3, DO_STAGES = 2;
// Sixteen compute warps: four column groups of 32 queries times the four TMEM lane quarters. The
// exponential phase is bound by the special-function unit whatever the warp count; everything
// around it (TMEM round trips, barrier latency, the dS arithmetic) is per-warp serial time, and
// four warps per scheduler overlap it where two could not.
constexpr int KW_COMPUTE = 16, KW_TMA = 16, KW_MMA = 17, KW_MMA_DK = 18, KW_PULL = 19;
constexpr int DKDV_THREADS = (KW_COMPUTE + 4) * 32;   // 5 warps per scheduler: 96 registers each
// Tail of the dK/dV kernel's shared memory: alignment slack, barriers, and two buffers of 256
// per-query statistics (-lse * log2e for 128 queries, then -delta for the same 128).
constexpr int DKDV_ALIGN_SLACK = 768, DKDV_BAR_BYTES = 224, DKDV_STAT_BYTES = 2 * 256 * 4;
constexpr int DKDV_SMEM =
    2 * TILE_BYTES /*K,V*/ + (Q_STAGES + DO_STAGES) * TILE_BYTES + DKDV_ALIGN_SLACK + DKDV_BAR_BYTES + DKDV_STAT_BYTES;
static_assert(DO_STAGES == 2, "the issuing warps use n & 1 as dO's stage");
static_assert(DKDV_SMEM <= 227 * 1024, "dK/dV kernel shared memory");

template <bool SPARSE>
__global__ void __launch_bounds__(DKDV_THREADS, 1)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmGK, const __grid_constant__ CUtensorMap tmGV, BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = smem + TILE_BYTES;
  uint8_t* sQ = smem + 2 * TILE_BYTES;                 // [Q_STAGES]
  uint8_t* sdO = sQ + Q_STAGES * TILE_BYTES;           // [DO_STAGES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sdO + DO_STAGES * TILE_BYTES);
  uint64_t* kv_full = bars;         // 1
  uint64_t* q_full = bars + 1;      // [3]
  uint64_t* q_empty = bars + 4;     // [3]
  uint64_t* do_full = bars + 7;     // [2]
  uint64_t* do_empty = bars + 9;    // [2]
  uint64_t* s_full = bars + 11;     // [2] S^T of query half h is in TMEM
  uint64_t* dp_full = bars + 13;    // [2]
  uint64_t* p_ready = bars + 15;    // [2] (one arrival per compute warp of the half)
  uint64_t* ds_ready = bars + 17;   // [2]
  uint64_t* stat_full = bars + 19;  // [2] statistics of an item are in shared memory
  uint64_t* stat_free = bars + 21;  // [2] (one arrival per compute warp)
  uint64_t* acc_done = bars + 23;   // 1 (one commit per MMA warp)
  uint64_t* drain_bar = bars + 24;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* item_qpos = reinterpret_cast<int*>(bars + 27);   // [2] position of the item's first query
  float* stats = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + DKDV_BAR_BYTES);  // [2][-lse * log2e | -delta][128]
  if (smem - smem_raw > DKDV_ALIGN_SLACK) {  // same verdict in every thread
    if (threadIdx.x == 0) report(p.status, ZX_ERR_ARG, /*site=*/20, (int)(smem - smem_raw));
    return;
  }

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WorkItem wi = work_item(blockIdx.x, p.n_kv_tiles, p.B * p.Hkv, p.kv_heads_per_group);
  const int j = wi.tile;   // early KV tiles have the most work under a causal mask
  const int b = wi.head / p.Hkv, hk = wi.head % p.Hkv;
  const int G = p.Hq / p.Hkv;
  const int kpos0 = kv_tile_pos(p, j);

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < Q_STAGES; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
    }
    for (int s = 0; s < DO_STAGES; ++s) {
      mbar_init(&do_full[s], 1);
      mbar_init(&do_empty[s], 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&s_full[h], 1);
      mbar_init(&dp_full[h], 1);
      mbar_init(&p_ready[h], KW_COMPUTE / 2);      // per-warp arrivals
      mbar_init(&ds_ready[h], KW_COMPUTE / 2);
      mbar_init(&stat_full[h], 1);
      mbar_init(&stat_free[h], KW_COMPUTE);
    }
    mbar_init(acc_done, 2);
    mbar_init(&drain_bar[0], 1);
    mbar_init(&drain_bar[1], 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == KW_MMA) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // number of (head, q tile) items this CTA processes: identical in every role
  const int n_items = G * QWalk<SPARSE>::count(p, kpos0);

  if (warp == KW_PULL) warp_pull_slice(p.pull_src, p.pull_dst, p.pull_nvec, lane);

  if (n_items > 0 && warp != KW_PULL) {
    if (warp == KW_TMA) {
      // ------------------------------- producer -----------------------------------
      // Tiles through the TMA unit (lane 0), and what the compute warps need to know about each item: the position of
      // its first query, -lse * log2e and -delta of its 128 queries. The compute warps so hold no walk state, no
      // pointers and no prefetched values, which is what keeps them under 96 registers: a spilled register costs an
      // L2 round trip here, since shared memory takes almost all of the L1.
      if (lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmdO);
        mbar_expect_tx(kv_full, 2 * TILE_BYTES);
        tma_load_4d(sK, &tmK, kv_full, 0, hk, j * BT, b);
        tma_load_4d(sK + HALF_BYTES, &tmK, kv_full, 64, hk, j * BT, b);
        tma_load_4d(sV, &tmV, kv_full, 0, hk, j * BT, b);
        tma_load_4d(sV + HALF_BYTES, &tmV, kv_full, 64, hk, j * BT, b);
      }
      uint32_t n = 0;
      bool ok = true;
      for (int g = 0; g < G && ok; ++g) {
        const int hq = hk * G + g;
        const size_t row0 = ((size_t)b * p.Hq + hq) * p.Sq + lane;
        QWalk<SPARSE> w;
        for (w.init(); w.next(p, kpos0); ++n) {
          const int t = w.t;
          const int qs = n % Q_STAGES, ds = n % DO_STAGES;
          float x[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            x[i] = __ldg(p.lse + row0 + (size_t)t * BT + 32 * i);
            x[4 + i] = __ldg(p.delta + row0 + (size_t)t * BT + 32 * i);
          }
          if (!mbar_wait_w(&q_empty[qs], ((n / Q_STAGES) & 1) ^ 1, abort_flag)) { ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(&q_full[qs], TILE_BYTES);
            tma_load_4d(sQ + qs * TILE_BYTES, &tmQ, &q_full[qs], 0, hq, t * BT, b);
            tma_load_4d(sQ + qs * TILE_BYTES + HALF_BYTES, &tmQ, &q_full[qs], 64, hq, t * BT, b);
          }
          if (!mbar_wait_w(&do_empty[ds], ((n / DO_STAGES) & 1) ^ 1, abort_flag)) { ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(&do_full[ds], TILE_BYTES);
            tma_load_4d(sdO + ds * TILE_BYTES, &tmdO, &do_full[ds], 0, hq, t * BT, b);
            tma_load_4d(sdO + ds * TILE_BYTES + HALF_BYTES, &tmdO, &do_full[ds], 64, hq, t * BT, b);
          }
          if (!mbar_wait_w(&stat_free[n & 1], ((n >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
          float* st = stats + (n & 1) * 256 + lane;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            st[32 * i] = -LOG2E * x[i];
            st[128 + 32 * i] = -x[4 + i];
          }
          if (lane == 0) item_qpos[n & 1] = w.qpos0;
          mbar_arrive_warp(&stat_full[n & 1]);
        }
      }
      if (!ok) {
        if (lane == 0) report(p.status, ZX_ERR_TIMEOUT, /*site=*/21, (int)n);
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
      }
    } else if (warp == KW_MMA || warp == KW_MMA_DK) {
      // ------------------------------- MMA issuers --------------------------------
      // Two issuing warps: one for S^T and dV (it owns the S^T / P^T columns and the dV accumulator), one for dP^T and
      // dK. A wait costs such a warp some 270 clk even when its barrier completed long ago (a chain of dependent
      // instructions that shares its scheduler with four compute warps), and only two MMAs are queued behind the one
      // that runs, so one warp with all four products leaves the tensor core idle at each of its six waits per item
      // (measured 4,200 clk per item against 2,480 of MMA time). With two, one issues while the other waits.
      // All 32 lanes run the loops; the instructions themselves are issued by one elected lane.
      const bool scores = warp == KW_MMA;
      constexpr uint32_t idesc_kk = make_idesc(BT, BT / 2, 1, 1, 0, 0);  // both operands K-major, 64 queries
      constexpr uint32_t idesc_tm = make_idesc(BT, HD, 1, 1, 0, 1);      // A from TMEM, B MN-major
      // [S^T | dP^T] of both halves and the accumulator [dV | dK] of this warp
      const uint32_t t_x = tmem_base + (scores ? 0 : 128), t_acc = tmem_base + (scores ? 256 : 384);
      const uint64_t kv_addr = base_kmajor(smem_u32(scores ? sK : sV));
      const uint64_t x_k0 = base_kmajor(smem_u32(scores ? sQ : sdO));      // B operand of the first product, as stored
      const uint64_t x_mn0 = base_mnmajor(smem_u32(scores ? sdO : sQ));    // B operand of the second, read transposed
      uint64_t* x_full = scores ? q_full : do_full;
      uint64_t* out_full = scores ? s_full : dp_full;
      uint64_t* in_ready = scores ? p_ready : ds_ready;
      // first product of query half h: 64 rows of the tile are the B operand (HALF_Q bytes further down for h = 1)
      auto first = [&](int h, int stage) {
        umma_ss_k8_kmajor_w<HALF_BYTES / 16>(t_x + 64 * h, kv_addr, desc_advance(x_k0, (uint32_t)stage * TILE_BYTES + h * HALF_Q),
                                             idesc_kk, 0u);
        umma_commit_w(&out_full[h]);
      };
      // dV += P^T dO or dK += dS^T Q over the 64 queries of half h
      auto second = [&](int h, int stage, uint32_t acc) {
        umma_ts_k4_w<8, 32, 40>(t_acc, t_x + 64 * h, desc_advance(x_mn0, (uint32_t)stage * TILE_BYTES + h * HALF_Q), idesc_tm, acc);
      };
      bool ok = mbar_wait_w(kv_full, 0, abort_flag);
      ok = ok && mbar_wait_w(&x_full[0], 0, abort_flag);
      tc_fence_after();
      if (ok) {
        first(0, 0);
        first(1, 0);
      }
      int n = 0, qs = 0, qsn = 1 % Q_STAGES;        // stages of items n and n + 1, phase of the latter
      uint32_t qphn = 0;
      for (; n < n_items && ok; ++n) {
        const int ds = n & 1, dsn = ds ^ 1;
        const uint32_t dphn = ((n + 1) >> 1) & 1;
        const bool has_next = n + 1 < n_items;
        const int s_first = scores ? qsn : dsn, s_second = scores ? ds : qs;
        for (int h = 0; h < 2; ++h) {
          // what each wait covers: dkdv_waits.h
          const unsigned waits = dkdv_waits(scores, h, has_next);
          const bool next = waits & WAIT_NEXT, tile = waits & WAIT_TILE;
          uint64_t* in = &in_ready[h];
          const uint32_t par = n & 1;
          const bool got = waits == WAIT_IN
                               ? mbar_wait_w(in, par, abort_flag)
                               : mbar_wait3_w(in, par, next ? &x_full[s_first] : in, next ? (scores ? qphn : dphn) : par,
                                              tile ? &do_full[ds] : in, tile ? (n >> 1) & 1 : par, abort_flag);
          if (!got) { ok = false; break; }
          tc_fence_after();
          second(h, s_second, (n > 0 || h > 0) ? 1u : 0u);
          if (has_next) first(h, s_first);
        }
        if (!ok) break;
        qs = qsn;
        if (++qsn == Q_STAGES) { qsn = 0; qphn ^= 1u; }
      }
      if (ok) umma_commit_w(acc_done);
      if (!ok) {
        if (lane == 0) report(p.status, ZX_ERR_TIMEOUT, /*site=*/22, n);
        uint64_t* db = &drain_bar[scores ? 0 : 1];
        umma_commit_w(db);
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(db, 0) && globaltimer_ns() - t0 < 50000000ull) {
        }
      }
    } else {
      // ------------------------------- compute warps ------------------------------
      // Four column groups: group wg owns query columns [32 wg, 32 wg + 32) of every KV row; groups 0, 1 are query
      // half 0, groups 2, 3 half 1.
      const int wg = warp >> 2;
      const int half = wg >> 1;
      const int lq = warp & 3;                 // TMEM lane quarter
      const int r = lq * 32 + lane;            // KV row of this thread == TMEM lane
      const int col0 = wg * 32;
      const uint32_t lane_base = (uint32_t)(lq * 32) << 16;
      const uint32_t t_s = tmem_base + lane_base + col0, t_dp = tmem_base + lane_base + 128 + col0;
      const int my_kpos = kpos0 + r;
      int n = 0;
      int qs_prev = Q_STAGES - 1;   // stage of item n - 1
      bool ok = true;
      for (; n < n_items; ++n) {
        const float* st = stats + (n & 1) * 256 + col0;
        if (!wait_warp(&stat_full[n & 1], (n >> 1) & 1, abort_flag)) { ok = false; break; }
        if (!wait_warp(&s_full[half], n & 1, abort_flag)) { ok = false; break; }
        // Stages are handed back here and not by commits of the issuing warps, whose queue they would fill: S^T of half
        // 1 was issued after dV(n-1), so its arrival says that dO(n-1) has been read (and dP^T(n-1) long before) ...
        if (threadIdx.x == 256 && n > 0) mbar_arrive(&do_empty[(n - 1) % DO_STAGES]);
        tc_fence_after();
        if (threadIdx.x == 0) ZX_TRACE_DKDV(n, 0);
        if (threadIdx.x == 256) ZX_TRACE_DKDV(n, 4);
        uint32_t sr[32];
        tmem_ld_32x32b_x32(t_s, sr);
        tmem_wait_ld();
        const int qpos0 = item_qpos[n & 1];
        const float2 sl2 = make_float2(p.scale_log2, p.scale_log2);
        const float4* nl4 = reinterpret_cast<const float4*>(st);   // uniform address: broadcast reads
        static_for<8>([&](auto idx4) {
          constexpr int c4 = decltype(idx4)::value;
          const float4 nl = nl4[c4];
          static_for<2>([&](auto idxh) {
            constexpr int h = decltype(idxh)::value;
            constexpr int c = 2 * c4 + h;
            const float2 x = __ffma2_rn(make_float2(__uint_as_float(sr[2 * c]), __uint_as_float(sr[2 * c + 1])), sl2,
                                        h == 0 ? make_float2(nl.x, nl.y) : make_float2(nl.z, nl.w));
            const float2 e = fast_exp2(x);
            sr[2 * c] = __float_as_uint(e.x);
            sr[2 * c + 1] = __float_as_uint(e.y);
          });
        });
        if (p.causal && kpos0 + BT - 1 > qpos0) {   // only tiles on the diagonal pay for the per-element mask
          const int seen = my_kpos - qpos0 - col0;   // this key is visible to columns c >= seen
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (c < seen) sr[c] = 0u;
        }
        {
          // bf16 P^T of this group goes over the first 16 of the 32 columns this thread just read
          uint32_t pk[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) pk[c] = pack_bf16x2(__uint_as_float(sr[2 * c]), __uint_as_float(sr[2 * c + 1]));
          tmem_st_32x32b_x16(t_s, pk);
        }
        tmem_wait_st();
        if (threadIdx.x == 0) ZX_TRACE_DKDV(n, 1);
        if (threadIdx.x == 256) ZX_TRACE_DKDV(n, 5);
        tc_fence_before();
        mbar_arrive_warp(&p_ready[half]);
        if (!wait_warp(&dp_full[half], n & 1, abort_flag)) { ok = false; break; }
        // ... and dP^T of half 1 after dK(n-1), so Q(n-1) has been read
        if (threadIdx.x == 256) {
          if (n > 0) mbar_arrive(&q_empty[qs_prev]);
          qs_prev = qs_prev + 1 == Q_STAGES ? 0 : qs_prev + 1;
        }
        tc_fence_after();
        if (threadIdx.x == 0) ZX_TRACE_DKDV(n, 2);
        if (threadIdx.x == 256) ZX_TRACE_DKDV(n, 6);
        uint32_t dp[32];
        tmem_ld_32x32b_x32(t_dp, dp);
        tmem_wait_ld();
        {
          uint32_t dsp[16];
          const float4* nd4 = reinterpret_cast<const float4*>(st + BT);
#pragma unroll
          for (int e4 = 0; e4 < 8; ++e4) {
            const float4 nd = nd4[e4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int e = 2 * e4 + h;
              const float2 t2 = __fadd2_rn(make_float2(__uint_as_float(dp[2 * e]), __uint_as_float(dp[2 * e + 1])),
                                           h == 0 ? make_float2(nd.x, nd.y) : make_float2(nd.z, nd.w));
              const float2 d = __fmul2_rn(make_float2(__uint_as_float(sr[2 * e]), __uint_as_float(sr[2 * e + 1])), t2);
              dsp[e] = pack_bf16x2(d.x, d.y);
            }
          }
          tmem_st_32x32b_x16(t_dp, dsp);
        }
        tmem_wait_st();
        if (threadIdx.x == 0) ZX_TRACE_DKDV(n, 3);
        tc_fence_before();
        mbar_arrive_warp(&ds_ready[half]);
        if (lane == 0) mbar_arrive(&stat_free[n & 1]);
      }
      // epilogue: dV and scale * dK, each column group its 32 columns of both accumulators. Written through shared
      // memory (the stages of Q and dO are free once every MMA has finished), or added into the (possibly remote) fp32
      // accumulators.
      if (ok) ok = wait_warp(acc_done, 0, abort_flag);
      tc_fence_after();
      const bool row_ok = ok && ZX_IN_BOUNDS(p.status, j * BT + r, p.Skv, 24);
      if (p.kv_overwrite && __all_sync(0xffffffffu, row_ok)) {
        uint8_t* slab = sQ + warp * (2 * SLAB_BYTES);
        uint32_t a[32];
        tmem_ld_32x32b_x32(tmem_base + lane_base + 256 + col0, a);
        tmem_wait_ld();
        store_slab(&tmGV, slab, a, 1.f, p.out_bf16, lane, col0, hk, j * BT + lq * 32, b);
        tmem_ld_32x32b_x32(tmem_base + lane_base + 384 + col0, a);
        tmem_wait_ld();
        store_slab(&tmGK, slab + SLAB_BYTES, a, p.scale, p.out_bf16, lane, col0, hk, j * BT + lq * 32, b);
        if (lane == 0) tma_store_wait<0>();
      } else if (row_ok) {
        const size_t row_off = (((size_t)b * p.Skv + (size_t)j * BT + r) * p.Hkv + hk) * HD + col0;
        float* dv_row = p.dv + row_off;
        float* dk_row = p.dk + row_off;
        {
          uint32_t a[32];
          tmem_ld_32x32b_x32(tmem_base + lane_base + 256 + col0, a);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e)
            red_add_v4_sys(dv_row + e * 4, __uint_as_float(a[4 * e]), __uint_as_float(a[4 * e + 1]),
                           __uint_as_float(a[4 * e + 2]), __uint_as_float(a[4 * e + 3]));
        }
        {
          uint32_t a[32];
          tmem_ld_32x32b_x32(tmem_base + lane_base + 384 + col0, a);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e)
            red_add_v4_sys(dk_row + e * 4, __uint_as_float(a[4 * e]) * p.scale, __uint_as_float(a[4 * e + 1]) * p.scale,
                           __uint_as_float(a[4 * e + 2]) * p.scale, __uint_as_float(a[4 * e + 3]) * p.scale);
        }
      }
      if (!ok && lane == 0) report(p.status, ZX_ERR_TIMEOUT, /*site=*/23, (int)n);
    }
  } else if (n_items == 0 && p.kv_overwrite && warp < KW_COMPUTE) {   // no query sees this tile
    uint32_t a[32] = {0};
    uint8_t* slab = sQ + warp * SLAB_BYTES;
    const int col = (warp >> 2) * 32, row = j * BT + (warp & 3) * 32;
    store_slab(&tmGV, slab, a, 1.f, p.out_bf16, lane, col, hk, row, b);
    if (lane == 0) {
      tma_store_4d(&tmGK, slab, col, hk, row, b);
      tma_store_commit();
      tma_store_wait<0>();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == KW_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------
// K lives until dQ of its item has been issued, V only until dP.
constexpr int K_STAGES = 4, V_STAGES = 3;
// Sixteen compute warps like the dK/dV kernel, one TMA warp, two MMA warps.
constexpr int QW_TMA = 16, QW_MMA = 17, QW_MMA_DQ = 18;
constexpr int DQ_THREADS = (KW_COMPUTE + 3) * 32;
constexpr int DQ_ALIGN_SLACK = 768, DQ_BAR_BYTES = 256;   // barriers: 28 x 8 B
constexpr int DQ_SMEM = (K_STAGES + V_STAGES) * TILE_BYTES + DQ_ALIGN_SLACK + DQ_BAR_BYTES;
static_assert(DQ_SMEM <= 227 * 1024, "dQ kernel shared memory");

template <bool SPARSE>
__global__ void __launch_bounds__(DQ_THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const __grid_constant__ CUtensorMap tmGQ, BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;                             // [K_STAGES]
  uint8_t* sV = sK + K_STAGES * TILE_BYTES;       // [V_STAGES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + V_STAGES * TILE_BYTES);
  uint64_t* k_full = bars;          // [4]
  uint64_t* k_empty = bars + 4;     // [4]
  uint64_t* v_full = bars + 8;      // [3]
  uint64_t* v_empty = bars + 11;    // [3]
  uint64_t* s_full = bars + 14;     // [2] S of key half h is in TMEM
  uint64_t* dp_full = bars + 16;    // [2]
  uint64_t* s_read = bars + 18;     // [2] (one arrival per compute warp of the half)
  uint64_t* ds_ready = bars + 20;   // [2]
  uint64_t* acc_done = bars + 22;   // 1
  uint64_t* drain_bar = bars + 23;  // [2]
  uint64_t* ab_ready = bars + 25;   // 1 Q and dO are in TMEM (one arrival per compute warp)
  uint64_t* qdo_full = bars + 26;   // 1 Q and dO are in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  if (smem - smem_raw > DQ_ALIGN_SLACK) {  // same verdict in every thread
    if (threadIdx.x == 0) report(p.status, ZX_ERR_ARG, /*site=*/20, (int)(smem - smem_raw));
    return;
  }

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WorkItem wi = work_item(blockIdx.x, p.n_q_tiles, p.B * p.Hq, p.q_heads_per_group);
  const int t = p.n_q_tiles - 1 - wi.tile;   // late Q tiles have the most work under a causal mask
  const int b = wi.head / p.Hq, hq = wi.head % p.Hq;
  const int hk = hq / (p.Hq / p.Hkv);
  const int qpos0 = q_tile_pos(p, t);

  if (threadIdx.x == 0) {
    for (int s = 0; s < K_STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < V_STAGES; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&s_full[h], 1);
      mbar_init(&dp_full[h], 1);
      mbar_init(&s_read[h], KW_COMPUTE / 2);    // per-warp arrivals
      mbar_init(&ds_ready[h], KW_COMPUTE / 2);
      mbar_init(&drain_bar[h], 1);
    }
    mbar_init(acc_done, 1);
    mbar_init(ab_ready, KW_COMPUTE);
    mbar_init(qdo_full, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == QW_MMA) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // TMEM columns: S of both key halves | dP of both (dS over it) | dQ | Q | dO
  constexpr uint32_t C_DP = 128, C_DQ = 256, C_Q = 384, C_DO = 448;

  const int n_items = KvWalk<SPARSE>::count(p, qpos0);

  if (n_items > 0) {
    if (warp == QW_TMA) {
      if (lane == 0) {
        // Q and dO pass through the last K and V stages on their way to TMEM: those stages are not needed before items
        // K_STAGES - 1 and V_STAGES - 1, and waited for below. (Reading the rows from global memory straight into
        // registers, 16 bytes of 32 different rows per load, took 3 us of every block's start.)
        uint8_t* sQ = sK + (K_STAGES - 1) * TILE_BYTES;
        uint8_t* sdO = sV + (V_STAGES - 1) * TILE_BYTES;
        mbar_expect_tx(qdo_full, 2 * TILE_BYTES);
        tma_load_4d(sQ, &tmQ, qdo_full, 0, hq, t * BT, b);
        tma_load_4d(sQ + HALF_BYTES, &tmQ, qdo_full, 64, hq, t * BT, b);
        tma_load_4d(sdO, &tmdO, qdo_full, 0, hq, t * BT, b);
        tma_load_4d(sdO + HALF_BYTES, &tmdO, qdo_full, 64, hq, t * BT, b);
        uint32_t n = 0;
        int ks = 0, vs = 0;
        uint32_t kph = 1, vph = 1;
        bool ok = true;
        KvWalk<SPARSE> w;
        for (w.init(); w.next(p, qpos0); ++n) {
          const int j = w.j;
          if (!mbar_wait(&k_empty[ks], kph, abort_flag)) { ok = false; break; }
          if (n == K_STAGES - 1 && !mbar_wait(ab_ready, 0, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&k_full[ks], TILE_BYTES);
          tma_load_4d(sK + ks * TILE_BYTES, &tmK, &k_full[ks], 0, hk, j * BT, b);
          tma_load_4d(sK + ks * TILE_BYTES + HALF_BYTES, &tmK, &k_full[ks], 64, hk, j * BT, b);
          if (++ks == K_STAGES) { ks = 0; kph ^= 1u; }
          if (!mbar_wait(&v_empty[vs], vph, abort_flag)) { ok = false; break; }
          if (n == V_STAGES - 1 && !mbar_wait(ab_ready, 0, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&v_full[vs], TILE_BYTES);
          tma_load_4d(sV + vs * TILE_BYTES, &tmV, &v_full[vs], 0, hk, j * BT, b);
          tma_load_4d(sV + vs * TILE_BYTES + HALF_BYTES, &tmV, &v_full[vs], 64, hk, j * BT, b);
          if (++vs == V_STAGES) { vs = 0; vph ^= 1u; }
        }
        if (!ok) {
          report(p.status, ZX_ERR_TIMEOUT, /*site=*/21, (int)n);
          const uint64_t t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 2000000ull) {
          }
        }
      }
    } else if (warp == QW_MMA) {
      // S_h(n+1) = Q K_h(n+1)^T as soon as the half's warps hold S_h(n) in registers
      constexpr uint32_t idesc_kk = make_idesc(BT, BT / 2, 1, 1, 0, 0);
      const uint64_t k_k0 = base_kmajor(smem_u32(sK));
      bool ok = mbar_wait_w(ab_ready, 0, abort_flag);
      int n = 0, ks = 0;
      uint32_t kph = 0;
      for (; n < n_items && ok; ++n) {
        for (int h = 0; h < 2; ++h) {
          const bool got = h == 0 ? mbar_wait2_w(&s_read[0], (n & 1) ^ 1, &k_full[ks], kph, abort_flag)
                                  : mbar_wait_w(&s_read[1], (n & 1) ^ 1, abort_flag);
          if (!got) { ok = false; break; }
          tc_fence_after();
          umma_ts_k8_kmajor_w<HALF_BYTES / 16>(tmem_base + 64 * h, tmem_base + C_Q,
                                               desc_advance(k_k0, (uint32_t)ks * TILE_BYTES + h * HALF_Q), idesc_kk, 0u);
          umma_commit_w(&s_full[h]);
        }
        if (++ks == K_STAGES) { ks = 0; kph ^= 1u; }
      }
      if (!ok) {
        if (lane == 0) report(p.status, ZX_ERR_TIMEOUT, /*site=*/22, n);
        umma_commit_w(&drain_bar[0]);
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&drain_bar[0], 0) && globaltimer_ns() - t0 < 50000000ull) {
        }
      }
    } else if (warp == QW_MMA_DQ) {
      // dQ += dS_h(n) K_h(n) (dS from TMEM, K read transposed), then dP_h(n+1) = dO V_h(n+1)^T over that dS
      constexpr uint32_t idesc_kk = make_idesc(BT, BT / 2, 1, 1, 0, 0);
      constexpr uint32_t idesc_tm = make_idesc(BT, HD, 1, 1, 0, 1);
      const uint64_t k_mn0 = base_mnmajor(smem_u32(sK)), v_k0 = base_kmajor(smem_u32(sV));
      auto dprob = [&](int h, int vs) {
        umma_ts_k8_kmajor_w<HALF_BYTES / 16>(tmem_base + C_DP + 64 * h, tmem_base + C_DO,
                                             desc_advance(v_k0, (uint32_t)vs * TILE_BYTES + h * HALF_Q), idesc_kk, 0u);
        umma_commit_w(&dp_full[h]);
      };
      bool ok = mbar_wait_w(ab_ready, 0, abort_flag);
      ok = ok && mbar_wait_w(&v_full[0], 0, abort_flag);
      tc_fence_after();
      if (ok) {
        dprob(0, 0);
        dprob(1, 0);
      }
      int n = 0, ks = 0, vs = 1;   // V stage of item n + 1
      uint32_t vph = 0;
      for (; n < n_items && ok; ++n) {
        const bool has_next = n + 1 < n_items;
        for (int h = 0; h < 2; ++h) {
          const bool got = h == 0 && has_next ? mbar_wait2_w(&ds_ready[0], n & 1, &v_full[vs], vph, abort_flag)
                                              : mbar_wait_w(&ds_ready[h], n & 1, abort_flag);
          if (!got) { ok = false; break; }
          tc_fence_after();
          umma_ts_k4_w<8, 32, 40>(tmem_base + C_DQ, tmem_base + C_DP + 64 * h,
                                  desc_advance(k_mn0, (uint32_t)ks * TILE_BYTES + h * HALF_Q), idesc_tm, (n > 0 || h > 0) ? 1u : 0u);
          if (has_next) dprob(h, vs);
        }
        if (!ok) break;
        if (++ks == K_STAGES) ks = 0;
        if (++vs == V_STAGES) { vs = 0; vph ^= 1u; }
      }
      if (ok) umma_commit_w(acc_done);
      if (!ok) {
        if (lane == 0) report(p.status, ZX_ERR_TIMEOUT, /*site=*/22, n);
        umma_commit_w(&drain_bar[1]);
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&drain_bar[1], 0) && globaltimer_ns() - t0 < 50000000ull) {
        }
      }
    } else {
      // Column group wg owns key columns [32 wg, 32 wg + 32) of every query row; groups 0, 1 are key half 0, 2, 3 half 1.
      const int wg = warp >> 2;
      const int half = wg >> 1;
      const int lq = warp & 3;
      const int r = lq * 32 + lane;  // query row == TMEM lane
      const int col0 = wg * 32;
      const uint32_t lane_base = (uint32_t)(lq * 32) << 16;
      bool ok = true;
      const uint32_t t_s = tmem_base + lane_base + col0, t_dp = t_s + C_DP;
      {
        // Q and dO of this tile into TMEM, where they are the A operands of S and dP (as shared-memory operands they
        // would make 128 x 64 products wait for shared memory: 6 KB per 32 clk of MMA). Groups 0 and 1 take the two
        // halves of the head dimension of Q, 2 and 3 of dO: 64 values of one row per thread, two per 32-bit column.
        const uint8_t* src = (wg < 2 ? sK + (K_STAGES - 1) * TILE_BYTES : sV + (V_STAGES - 1) * TILE_BYTES) +
                             (wg & 1) * HALF_BYTES + r * 128;
        if (!mbar_wait_w(qdo_full, 0, abort_flag)) ok = false;
        uint32_t x[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 u = *reinterpret_cast<const uint4*>(src + ((i ^ (r & 7)) << 4));   // 128-byte swizzle
          x[4 * i] = u.x; x[4 * i + 1] = u.y; x[4 * i + 2] = u.z; x[4 * i + 3] = u.w;
        }
        tmem_st_32x32b_x32(tmem_base + lane_base + C_Q + col0, x);
        tmem_wait_st();
        fence_proxy_async_smem();   // the stages are refilled by TMA once every warp has arrived
        tc_fence_before();
        mbar_arrive_warp(ab_ready);
      }
      const size_t stat_idx = ((size_t)b * p.Hq + hq) * p.Sq + (size_t)t * BT + r;
      const float nlse2 = -p.lse[stat_idx] * LOG2E;
      const float ndlt = -p.delta[stat_idx];
      uint32_t n = 0;
      int vs = 0;
      KvWalk<SPARSE> walk;
      for (walk.init(); ok && walk.next(p, qpos0); ++n) {
        if (!wait_warp(&s_full[half], n & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        uint32_t sr[32];
        tmem_ld_32x32b_x32(t_s, sr);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive_warp(&s_read[half]);
        const float2 sl2 = make_float2(p.scale_log2, p.scale_log2);
        const float2 nl2 = make_float2(nlse2, nlse2);
        static_for<16>([&](auto idx) {   // packed fp32x2 math: two key columns per instruction
          constexpr int c = decltype(idx)::value;
          const float2 x = __ffma2_rn(make_float2(__uint_as_float(sr[2 * c]), __uint_as_float(sr[2 * c + 1])), sl2, nl2);
          const float2 e = fast_exp2(x);
          sr[2 * c] = __float_as_uint(e.x);
          sr[2 * c + 1] = __float_as_uint(e.y);
        });
        if (p.causal && walk.kpos0 + BT - 1 > qpos0) {   // only tiles on the diagonal pay for the per-element mask
          const int last = qpos0 + r - walk.kpos0 - col0;   // columns up to this one are visible to the row
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (c > last) sr[c] = 0u;
        }
        if (!wait_warp(&dp_full[half], n & 1, abort_flag)) { ok = false; break; }
        // dP of half 1 was issued after dQ(n-1): its arrival says that K(n-1) and V(n) have been read. Handed back here
        // and not by commits of the issuing warp, whose queue they would fill.
        if (threadIdx.x == 256) {
          if (n > 0) mbar_arrive(&k_empty[(n - 1) % K_STAGES]);
          mbar_arrive(&v_empty[vs]);
          vs = vs + 1 == V_STAGES ? 0 : vs + 1;
        }
        tc_fence_after();
        uint32_t dp[32];
        tmem_ld_32x32b_x32(t_dp, dp);
        tmem_wait_ld();
        {
          uint32_t dsp[16];
          const float2 ndl = make_float2(ndlt, ndlt);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 t2 = __fadd2_rn(make_float2(__uint_as_float(dp[2 * e]), __uint_as_float(dp[2 * e + 1])), ndl);
            const float2 d = __fmul2_rn(make_float2(__uint_as_float(sr[2 * e]), __uint_as_float(sr[2 * e + 1])), t2);
            dsp[e] = pack_bf16x2(d.x, d.y);
          }
          tmem_st_32x32b_x16(t_dp, dsp);   // bf16 dS over the first 16 of the 32 columns this thread just read
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive_warp(&ds_ready[half]);
      }
      if (ok) ok = wait_warp(acc_done, 0, abort_flag);
      tc_fence_after();
      const bool row_ok = ok && ZX_IN_BOUNDS(p.status, t * BT + r, p.Sq, 25);
      if (!p.dq_accumulate && __all_sync(0xffffffffu, row_ok)) {
        uint32_t a[32];
        tmem_ld_32x32b_x32(tmem_base + lane_base + C_DQ + col0, a);
        tmem_wait_ld();
        store_slab(&tmGQ, sK + warp * SLAB_BYTES, a, p.scale, p.out_bf16, lane, col0, hq, t * BT + lq * 32, b);
        if (lane == 0) tma_store_wait<0>();
      } else if (row_ok) {
        float* dq_row = p.dq + (((size_t)b * p.Sq + (size_t)t * BT + r) * p.Hq + hq) * HD + col0;
        uint32_t a[32];
        tmem_ld_32x32b_x32(tmem_base + lane_base + C_DQ + col0, a);
        tmem_wait_ld();
        float4* dst = reinterpret_cast<float4*>(dq_row);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float4 o = dst[e];
          dst[e] = make_float4(o.x + __uint_as_float(a[4 * e]) * p.scale, o.y + __uint_as_float(a[4 * e + 1]) * p.scale,
                               o.z + __uint_as_float(a[4 * e + 2]) * p.scale, o.w + __uint_as_float(a[4 * e + 3]) * p.scale);
        }
      }
      if (!ok && lane == 0) report(p.status, ZX_ERR_TIMEOUT, /*site=*/23, (int)n);
    }
  } else if (n_items == 0 && !p.dq_accumulate && warp < KW_COMPUTE) {   // this tile sees no key
    uint32_t a[32] = {0};
    store_slab(&tmGQ, sK + warp * SLAB_BYTES, a, 1.f, p.out_bf16, lane, (warp >> 2) * 32, hq, t * BT + (warp & 3) * 32, b);
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == QW_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

CUtensorMap make_qkv_map(const void* base, int B, int S, int H, int64_t tok_stride) {
  uint64_t dims[4] = {(uint64_t)HD, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)HD * 2, (uint64_t)tok_stride * 2, (uint64_t)S * (uint64_t)tok_stride * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  return make_tma_map(base, 2, 4, dims, strides, box, TmaSwizzle::B128);
}

// A gradient [B, S, H, 128], stored 32 columns x 32 rows at a time (one warp's part of an accumulator).
CUtensorMap make_grad_map(const void* base, int B, int S, int H, int bf16) {
  const uint64_t es = bf16 ? 2 : 4;
  uint64_t dims[4] = {(uint64_t)HD, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {HD * es, (uint64_t)H * HD * es, (uint64_t)S * (uint64_t)H * HD * es};
  uint32_t box[4] = {32, 1, 32, 1};
  return make_tma_map(base, (int)es, 4, dims, strides, box, bf16 ? TmaSwizzle::B64 : TmaSwizzle::B128);
}

template <typename K>
void set_smem(K kern, int bytes, const char* name) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess)
    throw std::runtime_error(std::string(name) + ": cannot raise shared memory limit: " + cudaGetErrorString(e));
}

}  // namespace

void launch_attn_bwd(const AttnBwdArgs& a) {
  check_attn_common(a.Hq, a.Hkv, a.Sq, a.Skv, a.q_layout, a.kv_layout);
  if (a.Sq == 0 || a.Skv == 0 || a.B == 0) return;
  // everything that can refuse the call comes before the first launch
  const uintptr_t o_align = reinterpret_cast<uintptr_t>(a.o);
  if (a.compute_delta && o_align % 8 != 0) throw std::runtime_error("attn_bwd: o must be 8-byte aligned");
  CUtensorMap tmQ = make_qkv_map(a.q, a.B, a.Sq, a.Hq, a.q_tok_stride);
  CUtensorMap tmdO = make_qkv_map(a.d_o, a.B, a.Sq, a.Hq, (int64_t)a.Hq * HD);
  CUtensorMap tmK = make_qkv_map(a.k, a.B, a.Skv, a.Hkv, a.k_tok_stride);
  CUtensorMap tmV = make_qkv_map(a.v, a.B, a.Skv, a.Hkv, a.v_tok_stride);
  BwdParams p;
  p.B = a.B; p.Hq = a.Hq; p.Hkv = a.Hkv; p.Sq = a.Sq; p.Skv = a.Skv;
  p.scale = a.scale;
  p.scale_log2 = a.scale * LOG2E;
  p.causal = a.mask.causal; p.window_blocks = a.mask.window_blocks; p.global_every = a.mask.global_every;
  p.n_q_tiles = a.Sq / BT;
  p.n_kv_tiles = a.Skv / BT;
  p.q_tiles_per_chunk = a.q_layout.chunk_len / BT;
  p.kv_tiles_per_chunk = a.kv_layout.chunk_len / BT;
  p.n_q_chunks = a.q_layout.n_chunks;
  p.n_kv_chunks = a.kv_layout.n_chunks;
  for (int c = 0; c < kAttnMaxChunks; ++c) {
    p.q_chunk_pos[c] = c < a.q_layout.n_chunks ? a.q_layout.chunk_pos[c] : 0;
    p.kv_chunk_pos[c] = c < a.kv_layout.n_chunks ? a.kv_layout.chunk_pos[c] : 0;
  }
  p.lse = a.lse; p.delta = a.delta;
  if (a.out_bf16 && (a.dq_accumulate || !a.kv_overwrite))
    throw std::runtime_error("attn_bwd: bf16 gradients can only be written, not added to");
  p.dq = (float*)a.dq; p.dk = (float*)a.dk; p.dv = (float*)a.dv;
  p.dq_accumulate = a.dq_accumulate; p.kv_overwrite = a.kv_overwrite; p.out_bf16 = a.out_bf16;
  const CUtensorMap tmGQ = make_grad_map(a.dq, a.B, a.Sq, a.Hq, a.out_bf16);
  const CUtensorMap tmGK = make_grad_map(a.dk, a.B, a.Skv, a.Hkv, a.out_bf16);
  const CUtensorMap tmGV = make_grad_map(a.dv, a.B, a.Skv, a.Hkv, a.out_bf16);
  if (a.pull_bytes % 16 != 0) throw std::runtime_error("attn_bwd: pull size must be a multiple of 16 bytes");
  p.pull_src = (const uint4*)a.pull_src;
  p.pull_dst = (uint4*)a.pull_dst;
  p.pull_nvec = a.pull_src != nullptr ? a.pull_bytes / 16 : 0;
  p.trace = a.trace;
  p.status = a.status;
  static PerDeviceOnce once;
  bool& configured = once.current();
  if (!configured) {
    set_smem(attn_bwd_dkdv_kernel<false>, DKDV_SMEM, "attn_bwd_dkdv");
    set_smem(attn_bwd_dkdv_kernel<true>, DKDV_SMEM, "attn_bwd_dkdv (windowed)");
    set_smem(attn_bwd_dq_kernel<false>, DQ_SMEM, "attn_bwd_dq");
    set_smem(attn_bwd_dq_kernel<true>, DQ_SMEM, "attn_bwd_dq (windowed)");
    configured = true;
  }
  const bool uniform = !a.mask.causal && a.mask.window_blocks == 0;
  p.kv_heads_per_group = heads_per_group(p.n_q_tiles, a.B * a.Hkv, uniform, a.mask.window_blocks > 0);
  p.q_heads_per_group = heads_per_group(p.n_kv_tiles, a.B * a.Hq, uniform, false);
  const unsigned grid_kv = p.n_kv_tiles * a.B * a.Hkv, grid_q = p.n_q_tiles * a.B * a.Hq;
  if (a.compute_delta) {
    const int groups = (int)((size_t)a.B * a.Sq * a.Hq / DELTA_TOKENS);
    auto delta = o_align % 16 == 0 ? attn_delta_kernel<uint4> : attn_delta_kernel<uint2>;
    delta<<<(groups + 7) / 8, 256, 0, a.stream>>>((const __nv_bfloat16*)a.o, (const __nv_bfloat16*)a.d_o, a.delta, a.Sq, a.Hq,
                                                  groups);
  }
  if (p.window_blocks > 0) {
    attn_bwd_dkdv_kernel<true><<<grid_kv, DKDV_THREADS, DKDV_SMEM, a.stream>>>(tmQ, tmdO, tmK, tmV, tmGK, tmGV, p);
    attn_bwd_dq_kernel<true><<<grid_q, DQ_THREADS, DQ_SMEM, a.stream>>>(tmQ, tmdO, tmK, tmV, tmGQ, p);
  } else {
    attn_bwd_dkdv_kernel<false><<<grid_kv, DKDV_THREADS, DKDV_SMEM, a.stream>>>(tmQ, tmdO, tmK, tmV, tmGK, tmGV, p);
    attn_bwd_dq_kernel<false><<<grid_q, DQ_THREADS, DQ_SMEM, a.stream>>>(tmQ, tmdO, tmK, tmV, tmGQ, p);
  }
}

}  // namespace zx
