// A whole multisplit in one launch, for inputs whose tiles are all resident on
// the device at once: each block stages its tile, ranks and reorders it in
// shared memory, publishes its bucket counts, and meets the other blocks at a
// barrier; every block then reads the counts it needs and scatters the tile it
// still holds.  Same tiles, same order and same count matrix afterwards as the
// three stages.
//
// Bound by latency, not by bandwidth.  The three stages pay three dependent
// launches and read the keys twice; here the only dependent round trips are
// the loads, one barrier (two for large matrices) and the counts.
#pragma once

#include <cooperative_groups.h>

#include "multisplit_kernels.cuh"

namespace gms {

// How the blocks of one launch meet.
enum FusedSync : uint32_t {
  FUSED_ONE_TILE = 0,  // a single block: nothing to wait for
  FUSED_CLUSTER = 1,   // one thread-block cluster: the hardware's cluster barrier
  FUSED_GRID = 2,      // a cooperative launch: all blocks are resident, so the grid barrier ends
};

struct FusedArgs {
  uint32_t num_tiles;
  uint32_t sync;      // FusedSync
  uint32_t* matrix;   // the count matrix, [bucket][tile]; holds global offsets afterwards
  uint32_t* rows;     // the counts as [tile][bucket]
  uint32_t* totals;   // B words for the bucket totals: the columns of rows are scanned, with a
                      // second barrier; null: every block adds up the rows itself
  uint32_t* starts;   // B words for the bucket starts (pinned host memory), or null
};

__device__ __forceinline__ void fused_barrier(uint32_t sync) {
  if (sync == FUSED_GRID) {
    cooperative_groups::this_grid().sync();
  } else if (sync == FUSED_CLUSTER) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// The most tiles one launch can hold: the column scan keeps a thread's rows in
// registers.
constexpr uint32_t FUSED_SCAN_ROWS = 10;    // rows per thread
constexpr uint32_t FUSED_SCAN_GROUPS = 64;  // threads per column
constexpr uint32_t FUSED_MAX_TILES = FUSED_SCAN_ROWS * FUSED_SCAN_GROUPS;

// The tile's global bucket offsets, agreed on with the other blocks of the
// launch (see GivenOffset for the calls).  resolve() is called by every thread
// of the block after the tile is sorted in shared memory.
template <class C>
struct FusedOffsets {
  static constexpr bool KNOWN_EARLY = false;
  static constexpr uint32_t B = C::B;
  FusedArgs a;
  uint32_t tile;
  uint32_t* s_part;  // 2 * THREADS words
  uint32_t goff;

  __device__ __forceinline__ void aggregate(uint32_t b, uint32_t total) {
    if (a.sync == FUSED_ONE_TILE || tile >= a.num_tiles) return;
    a.rows[tile * B + b] = total;
  }

  __device__ __forceinline__ void resolve(uint32_t tid, uint32_t my_total) {
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    uint32_t before = 0, total = my_total;  // of bucket tid (tid < B)
    fused_barrier(a.sync);
    if (a.sync == FUSED_ONE_TILE) {
      // nothing before this tile
    } else if (a.totals == nullptr) {
      // Thread (r, b) adds rows r, r + R, ... of bucket b; the R partial sums
      // meet by shuffles (B < 32) and in shared memory.
      constexpr uint32_t R = uint32_t(C::THREADS) / B;
      const uint32_t b = tid % B;
      total = 0;
#pragma unroll 8
      for (uint32_t t = tid / B; t < a.num_tiles; t += R) {
        const uint32_t v = __ldcg(a.rows + t * B + b);
        total += v;
        before += t < tile ? v : 0u;
      }
      if constexpr (B < 32) {
#pragma unroll
        for (uint32_t d = B; d < 32; d <<= 1) {
          total += __shfl_xor_sync(~0u, total, d);
          before += __shfl_xor_sync(~0u, before, d);
        }
      }
      constexpr uint32_t G = uint32_t(C::THREADS) / (B < 32 ? 32u : B);  // partial sums per bucket left
      if constexpr (G > 1) {
        constexpr uint32_t PW = B < 32 ? 32u : B;  // threads per partial
        if (tid % PW < B) {
          s_part[(tid / PW) * B + tid % PW] = before;
          s_part[C::THREADS + (tid / PW) * B + tid % PW] = total;
        }
        __syncthreads();
        if (tid < B) {
          before = total = 0;
#pragma unroll
          for (uint32_t g = 0; g < G; ++g) {
            before += s_part[g * B + tid];
            total += s_part[C::THREADS + g * B + tid];
          }
        }
        __syncthreads();
      }
    } else {
      // A block scans four columns: 64 threads per column hold its rows, their
      // sums meet in shared memory.  Then a second barrier.
      constexpr uint32_t CB = B < 4 ? B : 4;
      const uint32_t c = tid % CB, r = tid / CB;
      const uint32_t per = (a.num_tiles + FUSED_SCAN_GROUPS - 1) / FUSED_SCAN_GROUPS;
      for (uint32_t col = blockIdx.x * CB; col < B; col += gridDim.x * CB) {
        uint32_t* p = a.rows + col + c;
        uint32_t v[FUSED_SCAN_ROWS], sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < FUSED_SCAN_ROWS; ++k) {
          const uint32_t t = r * per + k;
          v[k] = (r < FUSED_SCAN_GROUPS && k < per && t < a.num_tiles) ? __ldcg(p + t * B) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < FUSED_SCAN_ROWS; ++k) sum += v[k];
        if (r < FUSED_SCAN_GROUPS) s_part[c * FUSED_SCAN_GROUPS + r] = sum;
        __syncthreads();
        if (warp < CB) {
          uint32_t* q = s_part + warp * FUSED_SCAN_GROUPS + 2 * lane;
          const uint32_t x = q[0], y = q[1];
          uint32_t incl = x + y;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(~0u, incl, d);
            if (lane >= uint32_t(d)) incl += t;
          }
          q[0] = incl - x - y;
          q[1] = incl - y;
          if (lane == 31) a.totals[col + warp] = incl;
        }
        __syncthreads();
        if (r < FUSED_SCAN_GROUPS) {
          uint32_t run = s_part[c * FUSED_SCAN_GROUPS + r];
#pragma unroll
          for (uint32_t k = 0; k < FUSED_SCAN_ROWS; ++k) {
            const uint32_t t = r * per + k;
            if (k < per && t < a.num_tiles) p[t * B] = run;
            run += v[k];
          }
        }
        __syncthreads();
      }
      fused_barrier(a.sync);
      if (tid < B && tile < a.num_tiles) {
        before = __ldcg(a.rows + tile * B + tid);
        total = __ldcg(a.totals + tid);
      }
    }
    // Bucket starts: exclusive scan of the totals over the buckets.
    uint32_t incl = tid < B ? total : 0u;
    const uint32_t own = incl;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(~0u, incl, d);
      if (lane >= uint32_t(d)) incl += t;
    }
    constexpr uint32_t SCAN_WARPS = (B + 31) / 32;
    uint32_t start = incl - own;
    if constexpr (SCAN_WARPS > 1) {
      if (lane == 31 && warp < SCAN_WARPS) s_part[warp] = incl;
      __syncthreads();
#pragma unroll
      for (uint32_t w = 0; w < SCAN_WARPS; ++w) start += (w < warp) ? s_part[w] : 0u;
    }
    goff = start + before;
    if (tid < B && tile < a.num_tiles) {
      a.matrix[tid * a.num_tiles + tile] = goff;
      if (tile == 0 && a.starts != nullptr) a.starts[tid] = goff;
    }
  }
  __device__ __forceinline__ uint32_t offset(uint32_t, uint32_t) { return goff; }
};

// Blocks per SM the fused kernel is register-budgeted for (64 registers).
constexpr int FUSED_BLOCKS = 4;

// Stage cnt elements at src into shared memory, all loads in flight together:
// 16-byte loads and up to three single elements when src is 16-byte aligned,
// single elements otherwise.
template <int THREADS, int IPT>
__device__ __forceinline__ void stage_tile(uint32_t* dst, const uint32_t* __restrict__ src, uint32_t cnt) {
  const uint32_t tid = threadIdx.x;
  if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
    const uint32_t nv = cnt / 4u;
    uint4 v[IPT / 4];
#pragma unroll
    for (int k = 0; k < IPT / 4; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      v[k] = i < nv ? ld_nc_v4(src + i * 4u) : make_uint4(0u, 0u, 0u, 0u);
    }
    const uint32_t tail = 4u * nv + tid;
    if (tail < cnt) dst[tail] = src[tail];
#pragma unroll
    for (int k = 0; k < IPT / 4; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      if (i < nv) *reinterpret_cast<uint4*>(dst + i * 4u) = v[k];
    }
  } else {
    uint32_t v[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      v[k] = i < cnt ? src[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      if (i < cnt) dst[i] = v[k];
    }
  }
}

template <class C, class P>
__global__ void __launch_bounds__(C::THREADS, FUSED_BLOCKS) fused_kernel(
    const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t* __restrict__ kout,
    uint32_t* __restrict__ vout, uint32_t n, FusedArgs a, typename P::Params bp, ScratchHeader* hdr) {
  extern __shared__ __align__(128) unsigned char smem[];
  using L = PostLayout<C, P>;
  static_assert(C::KW == 1 && C::VW == 1, "32-bit elements");
  __shared__ uint32_t s_part[2 * C::THREADS];
  const uint32_t tid = threadIdx.x;
  const uint32_t tile = blockIdx.x;  // a cluster may have blocks past the last tile: empty tiles
  const uint32_t base = tile < a.num_tiles ? tile * C::TILE : n;
  const uint32_t cnt = min(C::TILE, n - base);
  if (tile == 0 && tid == 0) {
    hdr->error = 0u;
    hdr->error_info = 0u;
    hdr->ticket = 0u;
    hdr->wait_limit_us = 0u;
  }
  if (tid == 0) *reinterpret_cast<uint32_t*>(smem + L::OFF_FLAG) = 0u;
  stage_tile<C::THREADS, C::IPT>(reinterpret_cast<uint32_t*>(smem + L::OFF_K), kin + base, cnt);
  if constexpr (C::KV) stage_tile<C::THREADS, C::IPT>(reinterpret_cast<uint32_t*>(smem + L::OFF_V), vin + base, cnt);
  P::prepare(reinterpret_cast<uint32_t*>(smem + L::OFF_SPLIT), bp);
  if constexpr (C::LOGB > 5) {
    constexpr uint32_t WORDS = L::SUBWARPS * C::WB * C::WS * sizeof(typename L::WhT) / 4;
    uint32_t* s_wh = reinterpret_cast<uint32_t*>(smem + L::OFF_WH);
    for (uint32_t i = tid; i < WORDS; i += C::THREADS) s_wh[i] = 0u;
  }
  __syncthreads();
  FusedOffsets<C> offs{a, tile, s_part, 0u};
  if (cnt == C::TILE)
    postscan_tile<C, P, true, false, FusedOffsets<C>>(kout, vout, n, cnt, offs, bp, hdr, smem);
  else
    postscan_tile<C, P, false, false, FusedOffsets<C>>(kout, vout, n, cnt, offs, bp, hdr, smem);
}

}  // namespace gms
