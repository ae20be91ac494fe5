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
  FUSED_NONE = 3,      // they cannot: not one launch
};

constexpr uint32_t FUSED_CLUSTER_MAX = 16;  // blocks of one cluster (above 8: opt-in)

// How num_tiles tiles that are resident at once meet.  cluster_placed: the device
// can place a cluster of their size; has_rows: there is room for their counts,
// which only a cluster can do without.
inline uint32_t fused_sync_of(uint32_t num_tiles, bool cluster_placed, bool has_rows) {
  if (num_tiles == 1) return FUSED_ONE_TILE;
  if (num_tiles <= FUSED_CLUSTER_MAX && cluster_placed) return FUSED_CLUSTER;
  return has_rows ? FUSED_GRID : FUSED_NONE;
}

// Launch errors that say that this device (or the part of it that the process
// may use) has no room for the launch's form; the stages run instead.
inline bool fused_declined(cudaError_t e) {
  return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorInvalidClusterSize ||
         e == cudaErrorLaunchOutOfResources;
}

struct FusedArgs {
  uint32_t num_tiles;
  uint32_t sync;      // FusedSync
  uint32_t* matrix;   // the count matrix, [bucket][tile]; holds global offsets afterwards (null: not kept)
  uint32_t* rows;     // the counts as [tile][bucket]; null: the blocks of a cluster read each other's
                      // shared memory
  uint32_t* totals;   // B words for the bucket totals: the columns of rows are scanned, with a
                      // second barrier; null: every block adds up the rows itself
  uint32_t* starts;   // B words for the bucket starts (pinned host memory), or null
};

// Second half of the cluster barrier that FusedOffsets::resolve() arrives at.
__device__ __forceinline__ void fused_counts_read(const FusedArgs& a) {
  if (a.sync == FUSED_CLUSTER && a.rows == nullptr) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

__device__ __forceinline__ void fused_barrier(uint32_t sync) {
  if (sync == FUSED_GRID) {
    cooperative_groups::this_grid().sync();
  } else if (sync == FUSED_CLUSTER) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// A word of another block's shared memory in the same cluster: `local` is the
// word's address in this block's.
__device__ __forceinline__ uint32_t ld_cluster_u32(const uint32_t* local, uint32_t rank) {
  uint32_t addr, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
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
  uint32_t* s_cnt;   // B words: this block's counts, which the blocks of its cluster read
  uint32_t goff;

  __device__ __forceinline__ void aggregate(uint32_t b, uint32_t total) {
    if (a.rows == nullptr)
      s_cnt[b] = total;
    else if (tile < a.num_tiles)
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
        const uint32_t v = a.rows == nullptr ? ld_cluster_u32(s_cnt + b, t) : __ldcg(a.rows + t * B + b);
        total += v;
        before += t < tile ? v : 0u;
      }
      // No block leaves (or counts again) before the others have read its counts:
      // fused_counts_read() waits for this arrival.
      if (a.rows == nullptr) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
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
    if (tid < B && tile < a.num_tiles && a.matrix != nullptr) {
      a.matrix[tid * a.num_tiles + tile] = goff;
      if (tile == 0 && a.starts != nullptr) a.starts[tid] = goff;
    }
  }
  __device__ __forceinline__ uint32_t offset(uint32_t, uint32_t) { return goff; }
};

// Stage cnt 32- or 64-bit elements at src into shared memory, all loads in
// flight together: 16-byte loads and the last few elements singly when src is
// 16-byte aligned, single elements otherwise.  Through L2: a sort's later
// passes read what other blocks of the launch wrote.
template <int THREADS, int IPT, class T>
__device__ __forceinline__ void stage_tile(T* dst, const T* src, uint32_t cnt) {
  constexpr uint32_t EV = 16 / sizeof(T);  // elements per vector
  constexpr int NV = IPT / int(EV);
  static_assert(IPT % int(EV) == 0, "whole vectors per thread");
  const uint32_t tid = threadIdx.x;
  if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
    const uint32_t nv = cnt / EV;
    uint4 v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      v[k] = i < nv ? __ldcg(reinterpret_cast<const uint4*>(src + i * EV)) : make_uint4(0u, 0u, 0u, 0u);
    }
    const uint32_t tail = EV * nv + tid;
    if (tail < cnt) dst[tail] = __ldcg(src + tail);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      if (i < nv) *reinterpret_cast<uint4*>(dst + i * EV) = v[k];
    }
  } else {
    T v[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      v[k] = i < cnt ? __ldcg(src + i) : T(0);
    }
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
      const uint32_t i = uint32_t(k) * THREADS + tid;
      if (i < cnt) dst[i] = v[k];
    }
  }
}

// Blocks per SM the fused kernel is register-budgeted for: four (64
// registers), fewer where 64-bit elements fill the shared memory first.
template <class C, class P>
__host__ __device__ constexpr int fused_blocks() {
  return C::WIDE && PostLayout<C, P, C::KW == 2>::MIN_BLOCKS < 4 ? PostLayout<C, P, C::KW == 2>::MIN_BLOCKS : 4;
}

// One block's tile of one multisplit among the blocks of its launch.
// 64-bit keys: the tile's buckets are computed once, as bytes, from the staged
// keys (the GIVEN form of the tile's work), with the identifier's state at
// s_ident.
template <class C, class P>
__device__ __forceinline__ void fused_tile(const typename C::KT* kin, const typename C::VT* vin, typename C::KT* kout,
                                           typename C::VT* vout, uint32_t n, const FusedArgs& a,
                                           const typename P::Params& bp, ScratchHeader* hdr, unsigned char* smem,
                                           uint32_t* s_part, uint32_t* s_cnt, uint32_t* s_ident) {
  constexpr bool GIVEN = C::KW == 2;
  using L = PostLayout<C, P, GIVEN>;
  using KT = typename C::KT;
  using VT = typename C::VT;
  const uint32_t tid = threadIdx.x;
  const uint32_t tile = blockIdx.x;  // a cluster may have blocks past the last tile: empty tiles
  const uint32_t base = tile < a.num_tiles ? tile * C::TILE : n;
  const uint32_t cnt = min(C::TILE, n - base);
  if (tid == 0) *reinterpret_cast<uint32_t*>(smem + L::OFF_FLAG) = 0u;
  KT* s_k = reinterpret_cast<KT*>(smem + L::OFF_K);
  stage_tile<C::THREADS, C::IPT>(s_k, kin + base, cnt);
  if constexpr (!P::ANY_KEY) {
    if (cnt == 0 && tid == 0) s_k[0] = __ldcg(kin);  // postscan_tile evaluates the identifier on it
  }
  if constexpr (C::KV) stage_tile<C::THREADS, C::IPT>(reinterpret_cast<VT*>(smem + L::OFF_V), vin + base, cnt);
  uint32_t* s_state = GIVEN ? s_ident : reinterpret_cast<uint32_t*>(smem + L::OFF_SPLIT);
  P::prepare(s_state, bp);
  if constexpr (C::ATOMIC) {
    uint32_t* s_wh = reinterpret_cast<uint32_t*>(smem + L::OFF_WH);
    for (uint32_t i = tid; i < C::WARPS * C::WB; i += C::THREADS) s_wh[i] = 0u;
  }
  __syncthreads();
  if constexpr (GIVEN) {
    const typename P::Id ident = P::make(bp, s_state);
    uint8_t* s_rb = reinterpret_cast<uint8_t*>(smem + L::OFF_RB);
    for (uint32_t i = tid; i < cnt; i += C::THREADS) s_rb[i] = uint8_t(ident(s_k[i]));
    __syncthreads();
  }
  FusedOffsets<C> offs{a, tile, s_part, s_cnt, 0u};
  if (cnt == C::TILE)
    postscan_tile<C, P, true, GIVEN, FusedOffsets<C>>(kout, vout, n, cnt, offs, bp, hdr, smem);
  else
    postscan_tile<C, P, false, GIVEN, FusedOffsets<C>>(kout, vout, n, cnt, offs, bp, hdr, smem);
  fused_counts_read(a);
}

__device__ __forceinline__ void fused_reset_header(ScratchHeader* hdr) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    hdr->error = 0u;
    hdr->error_info = 0u;
    hdr->ticket = 0u;
    hdr->wait_limit_us = 0u;
  }
}

// Shared words of a 64-bit identifier's state (32-bit ones keep theirs in the
// tile's layout).
template <class C, class P>
__host__ __device__ constexpr uint32_t fused_ident_words() {
  return C::KW == 2 ? P::SMEM_WORDS : 1u;
}

template <class C, class P>
__global__ void __launch_bounds__(C::THREADS, (fused_blocks<C, P>())) fused_kernel(
    const typename C::KT* __restrict__ kin, const typename C::VT* __restrict__ vin, typename C::KT* __restrict__ kout,
    typename C::VT* __restrict__ vout, uint32_t n, FusedArgs a, typename P::Params bp, ScratchHeader* hdr) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_part[2 * C::THREADS];
  __shared__ uint32_t s_cnt[C::B];
  __shared__ __align__(16) uint32_t s_ident[fused_ident_words<C, P>()];
  fused_reset_header(hdr);
  fused_tile<C, P>(kin, vin, kout, vout, n, a, bp, hdr, smem, s_part, s_cnt, s_ident);
}

// A digit of the key, for the sort below: at most 2^LOGB values.
struct FieldParams {
  uint32_t shift;
  uint32_t mask;
};
struct FieldId {
  FieldParams p;
  template <class K>
  __device__ __forceinline__ uint32_t operator()(K key) const {
    return uint32_t(key >> p.shift) & p.mask;
  }
};
template <bool CHEAP_>
struct FieldPolicy {
  using Params = FieldParams;
  using Id = FieldId;
  template <bool KV>
  static constexpr bool CHEAP = CHEAP_;
  static constexpr bool USES_SMEM = false;
  static constexpr bool ANY_KEY = true;
  static constexpr uint32_t SMEM_WORDS = 1;
  __device__ __forceinline__ static void prepare(uint32_t*, const Params&) {}
  __device__ __forceinline__ static Id make(const Params& p, const uint32_t*) { return Id{p}; }
};

// A whole LSD sort in one launch: one multisplit per digit of at most `digit`
// bits over key bits [begin, end), ping-ponging so that the last lands in
// kout/vout, with a barrier between passes.
struct FusedDigits {
  uint32_t begin, end, digit;
};

template <class C, class P>
__global__ void __launch_bounds__(C::THREADS, (fused_blocks<C, P>())) fused_sort_kernel(
    const typename C::KT* kin, const typename C::VT* vin, typename C::KT* kout, typename C::VT* vout,
    typename C::KT* tk, typename C::VT* tv, uint32_t n, FusedArgs a, FusedDigits d, ScratchHeader* hdr) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_part[2 * C::THREADS];
  __shared__ uint32_t s_cnt[C::B];
  __shared__ uint32_t s_ident[1];
  fused_reset_header(hdr);
  const uint32_t passes = (d.end - d.begin + d.digit - 1) / d.digit;
  const typename C::KT* ki = kin;
  const typename C::VT* vi = vin;
  for (uint32_t p = 0; p < passes; ++p) {
    const bool to_out = ((passes - 1 - p) & 1u) == 0u;
    typename C::KT* ko = to_out ? kout : tk;
    typename C::VT* vo = to_out ? vout : tv;
    const uint32_t shift = d.begin + p * d.digit;
    const FieldParams bp{shift, (1u << min(d.digit, d.end - shift)) - 1u};
    if (p != 0) fused_barrier(a.sync);  // the previous pass's output is complete, its counts are read
    fused_tile<C, P>(ki, vi, ko, vo, n, a, bp, hdr, smem, s_part, s_cnt, s_ident);
    ki = ko;
    vi = vo;
  }
}

}  // namespace gms
