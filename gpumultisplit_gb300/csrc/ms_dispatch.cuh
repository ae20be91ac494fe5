// Launchers for one identifier kind: picks the compiled tile instance for
// log2 B and key/value, sets its shared-memory limit once per device, and
// launches prescan -> scan -> postscan on the caller's stream.
// Included by exactly one inst_*.cu per kind (explicit instantiation).
#pragma once

#include <atomic>

#include "batch_kernels.cuh"
#include "fused.cuh"
#include "histogram_kernels.cuh"
#include "ms_host.h"
#include "multisplit_kernels.cuh"

namespace gms {

// Raise a kernel's dynamic shared-memory limit to `bytes` once per device (bit
// per device id); needed once its static plus dynamic shared memory passes 48 KB.
template <class Kernel>
inline cudaError_t ensure_smem_limit(Kernel k, size_t bytes, std::atomic<uint64_t>& done_mask,
                                     size_t static_bytes = 0) {
  if (bytes + static_bytes <= 48 * 1024) return cudaSuccess;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (done_mask.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
  if (e == cudaSuccess) done_mask.fetch_or(bit, std::memory_order_acq_rel);
  return e;
}

// Grid of a persistent kernel: as many blocks as fit on the device at once
// (cached per kernel; the device's SM count is read per call), capped by `work`.
// Postscan L2 prefetch distance, in quarters of a wave of resident blocks (0 = off).
#ifndef GMS_PREFETCH_WAVES
#define GMS_PREFETCH_WAVES 2
#endif

template <class Kernel>
inline uint32_t persistent_grid(Kernel k, int threads, uint32_t work, std::atomic<int>& per_sm_cache,
                                size_t smem = 0) {
  int per_sm = per_sm_cache.load(std::memory_order_relaxed);
  if (per_sm <= 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem) != cudaSuccess || per_sm <= 0)
      per_sm = 1;
    per_sm_cache.store(per_sm, std::memory_order_relaxed);
  }
  const uint64_t cap = uint64_t(device_sm_count()) * uint64_t(per_sm);
  return uint32_t(work < cap ? work : cap);
}

// A prescan's grid: no more blocks than ranges that one scan of the rows takes.
inline uint32_t rows_grid(uint32_t grid, const uint32_t* rows) {
  if (rows == nullptr) return grid;
  const uint32_t most = scan_rows_limit();
  return grid < most ? grid : most;
}

// Stages of one multisplit with identifier policy P (descriptor kinds here;
// user functors from the drop-in C++ headers).  `scratch` is laid out as
// make_geometry(n, LOGB, KV).  bucket_bytes (n bytes, or null): for
// identifiers that are costly to evaluate, the prescan stores every key's
// bucket there and the postscan reads it instead of evaluating the identifier
// a second time; the prescan and postscan of one multisplit must agree on it.
//
// KW / VW: 32-bit words per key / value.  64-bit keys (KW = 2) are identified
// by the prescan only, which stores every key's bucket in bucket_bytes (then
// required); their postscan reads those bytes.
//
// starts: where the last stage stores the bucket starts (2^LOGB words of
// pinned host memory), or null.
template <int W>
using ElemT = std::conditional_t<W == 2, uint64_t, uint32_t>;

// When a multisplit runs as one launch (fused.cuh): its tiles are resident all
// at once, and for pairs with an identifier the three stages evaluate twice
// (delta, bit field, mask) there are at most FUSED_CHEAP_PAIR_TILES of them.
// Measured against the three stages replayed from a CUDA graph (us per call):
//   keys, delta, 256 buckets   10 k 11.4 -> 6.2   260 k 14.9 -> 9.4   1 Mi 15.9 -> 11.9   2.4 M 23.8 -> 19.9
//   pairs, delta, 32 buckets   10 k  9.1 -> 5.3   260 k 11.2 -> 6.6   1 Mi 13.6 -> 10.3   2.0 M 17.6 -> 17.3
//   pairs, delta, 64 buckets   1.5 M 17.3 -> 16.0, 2.0 M 19.0 -> 19.6: the line for pairs lies between
//   pairs, range, 32 buckets   10 k 13.3 -> 7.3   1 Mi 22.4 -> 12.4   2.4 M 26.8 -> 21.6
// Larger inputs keep the memory busier as three stages, whose tiles are in
// different phases.
//
// Beside large calls on another stream (2^28 pairs into 256 buckets) a small one
// waits for room, three stages three times, one launch once (us until it is done,
// three stages / one launch):
//   keys, 256 buckets    3 k 675 -> 350   50 k 590 -> 320   130 k 895 -> 69   1 Mi 725 -> 49   2.4 M 950 -> 52
//   pairs, 32 buckets   10 k 705 -> 455  300 k 755 -> 71     1 Mi 803 -> 49
// A cooperative grid, from 17 tiles up, seems to be placed ahead of the blocks that
// the large kernel has left.  The large calls take the same time.
//
// Up to FUSED_ADD_MAX counts every block adds up the rows itself (one
// barrier); above, the columns are scanned first (two barriers).  At 256
// buckets: 130 k keys (8192 counts) 10.1 against 11.6 us, 260 k keys 11.7
// against 10.5.
constexpr uint32_t FUSED_CHEAP_PAIR_TILES = 448;
constexpr uint32_t FUSED_ADD_MAX = 8192;

// What a one-launch kernel remembers per process; a bit per device, and per
// cluster size (2, 4, 8, 16) whether a cluster of that size can be placed.
struct FusedKernelState {
  std::atomic<uint64_t> smem_done{0};
  std::atomic<uint64_t> placed[4] = {};
  std::atomic<uint64_t> not_placed[4] = {};
  std::atomic<int> per_sm{0};
};

// Whether the current device can place the cluster that cfg describes.
template <class Kernel>
bool cluster_placed(Kernel kern, const cudaLaunchConfig_t& cfg, uint32_t blocks, FusedKernelState& state) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const uint64_t bit = 1ull << (dev & 63);
  const int size = blocks <= 2 ? 0 : blocks <= 4 ? 1 : blocks <= 8 ? 2 : 3;
  if (state.placed[size].load(std::memory_order_acquire) & bit) return true;
  if (state.not_placed[size].load(std::memory_order_acquire) & bit) return false;
  int clusters = 0;
  const bool yes =
      (blocks <= 8 || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
      cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0;
  if (!yes) cudaGetLastError();
  (yes ? state.placed : state.not_placed)[size].fetch_or(bit, std::memory_order_acq_rel);
  return yes;
}

// Prepares `kern` to run num_tiles tiles in one launch: its limits, the form of
// its barrier (a->sync) and the launch configuration.  *fits: all tiles are
// resident at once and can meet.
template <class C, class Kernel>
cudaError_t fused_config(Kernel kern, size_t smem, size_t static_smem, uint32_t num_tiles, FusedKernelState& state,
                         cudaStream_t stream, FusedArgs* a, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr,
                         bool* fits) {
  *fits = false;
  const cudaError_t e = ensure_smem_limit(kern, smem, state.smem_done, static_smem);
  if (e != cudaSuccess) return e;
  if (persistent_grid(kern, C::THREADS, num_tiles, state.per_sm, smem) < num_tiles) return cudaSuccess;
  a->num_tiles = num_tiles;
  cfg->blockDim = dim3(C::THREADS);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = stream;
  cfg->attrs = attr;
  bool placed = false;
  if (num_tiles > 1 && num_tiles <= FUSED_CLUSTER_MAX) {
    uint32_t blocks = 2;
    while (blocks < num_tiles) blocks <<= 1;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = blocks;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->numAttrs = 1;
    cfg->gridDim = dim3(blocks);
    placed = cluster_placed(kern, *cfg, blocks, state);
  }
  a->sync = fused_sync_of(num_tiles, placed, a->rows != nullptr);
  if (a->sync == FUSED_NONE) return cudaSuccess;
  if (a->sync != FUSED_CLUSTER) {
    cfg->gridDim = dim3(num_tiles);
    attr->id = cudaLaunchAttributeCooperative;
    attr->val.cooperative = 1;
    cfg->numAttrs = a->sync == FUSED_GRID ? 1 : 0;
  }
  *fits = true;
  return cudaSuccess;
}

// The outcome of a one-launch kernel's launch: one that the device has no room
// for is not an error, the stages run instead.
inline cudaError_t fused_launched(cudaError_t e, bool* launched) {
  *launched = !fused_declined(e);
  if (*launched) return e;
  cudaGetLastError();
  return cudaSuccess;
}

// Runs a whole multisplit as one launch if the rule above says so and, beyond
// one cluster, the scratch has room for the counts as [tile][bucket] rows after
// the matrix and status words (every caller that allocated the reported size
// has it there: its byte per key).  *launched says whether it did.
template <class C, class P>
cudaError_t launch_fused(const typename C::KT* kin, const typename C::VT* vin, typename C::KT* kout, typename C::VT* vout,
                         uint32_t n, const typename P::Params& params, unsigned char* scratch, size_t scratch_bytes,
                         const Geometry& g, cudaStream_t stream, uint32_t* starts, bool* launched) {
  static FusedKernelState state;
  *launched = false;
  if (g.num_tiles > (C::KV && P::template CHEAP<true> ? FUSED_CHEAP_PAIR_TILES : FUSED_MAX_TILES)) return cudaSuccess;
  FusedArgs a{};
  a.starts = starts;
  a.matrix = reinterpret_cast<uint32_t*>(scratch + g.off_matrix);
  const size_t rows_bytes = size_t(g.m) * 4, totals_bytes = size_t(C::B) * 4;
  if (g.num_tiles > 1 && scratch_bytes >= g.off_buckets + rows_bytes + totals_bytes) {
    a.rows = reinterpret_cast<uint32_t*>(scratch + g.off_buckets);
    if (g.m > FUSED_ADD_MAX) a.totals = reinterpret_cast<uint32_t*>(scratch + g.off_buckets + rows_bytes);
  } else if (g.num_tiles > FUSED_CLUSTER_MAX) {
    return cudaSuccess;
  }
  auto kern = fused_kernel<C, P>;
  constexpr size_t smem = PostLayout<C, P, C::KW == 2>::BYTES;
  constexpr size_t static_smem = 2 * C::THREADS * 4 + C::B * 4 + fused_ident_words<C, P>() * 4;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  bool fits = false;
  const cudaError_t e =
      fused_config<C>(kern, smem, static_smem, g.num_tiles, state, stream, &a, &cfg, attr, &fits);
  if (e != cudaSuccess || !fits) return e;
  return fused_launched(cudaLaunchKernelEx(&cfg, kern, kin, vin, kout, vout, n, a, params,
                                           reinterpret_cast<ScratchHeader*>(scratch)),
                        launched);
}

// Sorts with digits of LOGB bits and tiles of IPT keys per thread in one launch,
// if its tiles are resident at once and there is room for the count rows (or
// they form one cluster); *launched says whether it did.
template <int LOGB, bool KV, int KW, int VW, int IPT>
cudaError_t launch_fused_sort(const FusedSortCall& c, bool* launched) {
  using C = TileCfg<LOGB, 8, IPT, KV, KW, VW>;
  using P = FieldPolicy<KW == 1>;
  static FusedKernelState state;
  *launched = false;
  const uint32_t num_tiles = uint32_t((uint64_t(c.n) + C::TILE - 1) / C::TILE);
  if (num_tiles > FUSED_MAX_TILES) return cudaSuccess;
  FusedArgs a{};
  const size_t rows_bytes = size_t(num_tiles) * C::B * 4;
  if (num_tiles > 1 && c.rows_bytes >= rows_bytes + C::B * 4) {
    a.rows = reinterpret_cast<uint32_t*>(c.rows);
    if (num_tiles * C::B > FUSED_ADD_MAX) a.totals = reinterpret_cast<uint32_t*>(c.rows + rows_bytes);
  } else if (num_tiles > FUSED_CLUSTER_MAX) {
    return cudaSuccess;
  }
  auto kern = fused_sort_kernel<C, P>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  bool fits = false;
  const cudaError_t e = fused_config<C>(kern, PostLayout<C, P, KW == 2>::BYTES, (2 * C::THREADS + C::B + 1) * 4, num_tiles, state,
                                        c.stream, &a, &cfg, attr, &fits);
  if (e != cudaSuccess || !fits) return e;
  using K = typename C::KT;
  using V = typename C::VT;
  const FusedDigits d{c.begin_bit, c.end_bit, uint32_t(LOGB)};
  return fused_launched(cudaLaunchKernelEx(&cfg, kern, static_cast<const K*>(c.kin), static_cast<const V*>(c.vin),
                                           static_cast<K*>(c.kout), static_cast<V*>(c.vout), static_cast<K*>(c.tk),
                                           static_cast<V*>(c.tv), c.n, a, d, c.hdr),
                        launched);
}

template <class P, int LOGB, bool KV, int KW = 1, int VW = 1>
cudaError_t launch_multisplit(const ElemT<KW>* kin, const ElemT<VW>* vin, ElemT<KW>* kout, ElemT<VW>* vout,
                              uint32_t n, const typename P::Params& params, unsigned char* scratch, int stages,
                              cudaStream_t stream, uint8_t* bucket_bytes = nullptr, size_t scratch_bytes = 0,
                              uint32_t* starts = nullptr, bool keep_matrix = true) {
  if constexpr (P::template CHEAP<KV>) bucket_bytes = nullptr;
  using S = TileShape<LOGB, KV, KW, VW>;
  using C = TileCfg<LOGB, S::WARPS, S::IPT, KV, KW, VW>;
  const Geometry g = make_geometry(n, LOGB, KV, KW, VW);
  if (g.num_tiles == 0) return cudaSuccess;
  auto* hdr = reinterpret_cast<ScratchHeader*>(scratch);
  auto* status = reinterpret_cast<uint64_t*>(scratch + g.off_status);
  auto* matrix = reinterpret_cast<uint32_t*>(scratch + g.off_matrix);

  if (stages == STAGE_ALL) {
    bool launched = false;
    const cudaError_t e =
        launch_fused<C, P>(kin, vin, kout, vout, n, params, scratch, scratch_bytes, g, stream, starts, &launched);
    if (e != cudaSuccess || launched) return e;
  }
  // Counts as rows: in the matrix's place, or beside it when the caller is to
  // find the matrix and the scratch has the room.
  uint32_t* rows = nullptr;
  if (stages == STAGE_ALL && counts_as_rows(LOGB, g.num_tiles) && (!P::USES_SMEM || bucket_bytes != nullptr)) {
    if (!keep_matrix) {
      rows = matrix;
    } else {
      const size_t off = bucket_bytes != nullptr ? g.bytes_full : g.off_buckets;
      if (scratch_bytes >= off + size_t(g.m) * 4) rows = reinterpret_cast<uint32_t*>(scratch + off);
    }
  }
  uint32_t* const counts = rows != nullptr ? rows : matrix;
  uint32_t* const matrix_out = rows != matrix && rows != nullptr ? matrix : nullptr;
  // The postscan's blocks: one per tile, then those that fill in the matrix.
  const uint32_t post_blocks =
      g.num_tiles + (matrix_out != nullptr ? (g.num_tiles + MATRIX_TILES - 1) / MATRIX_TILES : 0u);
  uint32_t rows_per = 0;  // tiles per range, known with the prescan's grid
  auto choose_rows = [&](uint32_t grid) {
    if (rows == nullptr) return;
    rows_per = (g.num_tiles + grid - 1) / grid;
  };

  if constexpr (KW == 2) {
    if (bucket_bytes == nullptr) return cudaErrorInvalidValue;
    if (stages & STAGE_PRESCAN) {
      static std::atomic<int> per_sm{0};
      auto kern = prescan64_kernel<C, P>;
      const uint32_t grid = rows_grid(persistent_grid(kern, C::THREADS, g.num_tiles, per_sm), rows);
      choose_rows(grid);
      kern<<<grid, C::THREADS, 0, stream>>>(kin, n, g.num_tiles, counts, params, hdr, status, g.num_chunks,
                                            bucket_bytes, rows_per);
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    if (stages & STAGE_SCAN) {
      cudaError_t e = rows_per != 0 ? run_scan_rows(rows, C::B, g.num_tiles, rows_per, status, hdr, stream)
                                    : run_scan(matrix, g.m, status, hdr, stream);
      if (e != cudaSuccess) return e;
    }
    if (stages & STAGE_POSTSCAN) {
      static std::atomic<uint64_t> smem_done{0};
      static std::atomic<int> per_sm{0};
      auto kern = postscan_kernel<C, P, true>;
      constexpr size_t smem = PostLayout<C, P, true>::BYTES;
      cudaError_t e = ensure_smem_limit(kern, smem, smem_done);
      if (e != cudaSuccess) return e;
      const uint32_t wave = persistent_grid(kern, C::THREADS, g.num_tiles, per_sm, smem);
      const uint32_t dist = (GMS_PREFETCH_WAVES * wave) / 4u;
      return launch_after_previous(kern, dim3(post_blocks), dim3(C::THREADS), smem, stream, kin, vin, kout, vout, n,
                                   g.num_tiles, counts, params, hdr, dist, bucket_bytes, starts, rows_per, matrix_out);
    }
    return cudaSuccess;
  } else {
  if (stages & STAGE_PRESCAN) {
    static std::atomic<int> per_sm{0};
    auto kern = prescan_kernel<C, P>;
    const uint32_t grid = rows_grid(persistent_grid(kern, C::THREADS, g.num_tiles, per_sm), rows);
    choose_rows(grid);
    kern<<<grid, C::THREADS, 0, stream>>>(kin, n, g.num_tiles, counts, params, hdr, status, g.num_chunks,
                                          bucket_bytes, rows_per);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  if (stages & STAGE_SCAN) {
    cudaError_t e = rows_per != 0 ? run_scan_rows(rows, C::B, g.num_tiles, rows_per, status, hdr, stream)
                                  : run_scan(matrix, g.m, status, hdr, stream);
    if (e != cudaSuccess) return e;
  }
  if constexpr (!P::template CHEAP<KV>) {
    if ((stages & STAGE_POSTSCAN) && bucket_bytes != nullptr) {
      // Buckets from the prescan: no identifier in the postscan at all.
      static std::atomic<uint64_t> smem_done{0};
      static std::atomic<int> per_sm{0};
      auto kern = postscan_kernel<C, P, true>;
      constexpr size_t smem = PostLayout<C, P, true>::BYTES;
      cudaError_t e = ensure_smem_limit(kern, smem, smem_done);
      if (e != cudaSuccess) return e;
      const uint32_t wave = persistent_grid(kern, C::THREADS, g.num_tiles, per_sm, smem);
      const uint32_t dist = (GMS_PREFETCH_WAVES * wave) / 4u;
      return launch_after_previous(kern, dim3(post_blocks), dim3(C::THREADS), smem, stream, kin, vin, kout, vout, n,
                                   g.num_tiles, counts, params, hdr, dist, bucket_bytes, starts, rows_per, matrix_out);
    }
  }
  if ((stages & STAGE_POSTSCAN) && P::USES_SMEM) {
    // Identifiers with a shared area: persistent blocks prepare it once.
    static std::atomic<uint64_t> smem_done{0};
    static std::atomic<int> per_sm{0};
    auto kern = postscan_persistent_kernel<C, P>;
    constexpr size_t smem = PostLayout<C, P>::BYTES;
    cudaError_t e = ensure_smem_limit(kern, smem, smem_done);
    if (e != cudaSuccess) return e;
    const uint32_t grid = persistent_grid(kern, C::THREADS, g.num_tiles, per_sm, smem);
    return launch_after_previous(kern, dim3(grid), dim3(C::THREADS), smem, stream, kin, vin, kout, vout, n,
                                 g.num_tiles, matrix, params, hdr, starts);
  }
  if (stages & STAGE_POSTSCAN) {
    static std::atomic<uint64_t> smem_done{0};
    static std::atomic<int> per_sm{0};
    auto kern = postscan_kernel<C, P>;
    constexpr size_t smem = PostLayout<C, P>::BYTES;
    cudaError_t e = ensure_smem_limit(kern, smem, smem_done);
    if (e != cudaSuccess) return e;
    // Prefetch distance: a fraction of the number of blocks resident at once (one wave).
    const uint32_t wave = persistent_grid(kern, C::THREADS, g.num_tiles, per_sm, smem);
    const uint32_t dist = (GMS_PREFETCH_WAVES * wave) / 4u;
    e = launch_after_previous(kern, dim3(post_blocks), dim3(C::THREADS), smem, stream, kin, vin, kout, vout, n,
                              g.num_tiles, counts, params, hdr, dist, static_cast<const uint8_t*>(nullptr), starts,
                              rows_per, matrix_out);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
  }
}

template <int KIND, int LOGB, bool KV>
cudaError_t run_multisplit_t(const MsCall& c, int stages) {
  return launch_multisplit<DescPolicy<KIND, LOGB>, LOGB, KV>(c.kin, c.vin, c.kout, c.vout, c.n, c.bp, c.scratch,
                                                             stages, c.stream, c.bucket_bytes, c.scratch_bytes, c.starts, c.keep_matrix);
}

template <int KIND, bool KV>
cudaError_t run_multisplit_kv(const MsCall& c, int stages) {
  switch (c.logb) {
    case 1: return run_multisplit_t<KIND, 1, KV>(c, stages);
    case 2: return run_multisplit_t<KIND, 2, KV>(c, stages);
    case 3: return run_multisplit_t<KIND, 3, KV>(c, stages);
    case 4: return run_multisplit_t<KIND, 4, KV>(c, stages);
    case 5: return run_multisplit_t<KIND, 5, KV>(c, stages);
    case 6: return run_multisplit_t<KIND, 6, KV>(c, stages);
    case 7: return run_multisplit_t<KIND, 7, KV>(c, stages);
    case 8: return run_multisplit_t<KIND, 8, KV>(c, stages);
    default: return cudaErrorInvalidValue;
  }
}

template <int KIND>
cudaError_t run_multisplit(const MsCall& c, int stages) {
  return c.kv ? run_multisplit_kv<KIND, true>(c, stages) : run_multisplit_kv<KIND, false>(c, stages);
}

// 64-bit elements: (key words, value words) = (1, 2), (2, 0), (2, 1), (2, 2).
template <int KIND, int LOGB, bool KV, int KW, int VW>
cudaError_t run_multisplit_wide_t(const MsCallWide& c, int stages) {
  using K = ElemT<KW>;
  using V = ElemT<VW>;
  const K* kin = static_cast<const K*>(c.kin);
  const V* vin = static_cast<const V*>(c.vin);
  K* kout = static_cast<K*>(c.kout);
  V* vout = static_cast<V*>(c.vout);
  if constexpr (KW == 2)
    return launch_multisplit<DescPolicy64<KIND, LOGB>, LOGB, KV, KW, VW>(kin, vin, kout, vout, c.n, c.bp64,
                                                                           c.scratch, stages, c.stream,
                                                                           c.bucket_bytes, c.scratch_bytes, c.starts, c.keep_matrix);
  else
    return launch_multisplit<DescPolicy<KIND, LOGB>, LOGB, KV, KW, VW>(kin, vin, kout, vout, c.n, c.bp, c.scratch,
                                                                         stages, c.stream, c.bucket_bytes, c.scratch_bytes, c.starts, c.keep_matrix);
}

template <int KIND, int LOGB>
cudaError_t run_multisplit_wide_l(const MsCallWide& c, int stages) {
  if (c.kw == 1 && c.kv && c.vw == 2) return run_multisplit_wide_t<KIND, LOGB, true, 1, 2>(c, stages);
  if (c.kw == 2 && !c.kv) return run_multisplit_wide_t<KIND, LOGB, false, 2, 1>(c, stages);
  if (c.kw == 2 && c.kv && c.vw == 1) return run_multisplit_wide_t<KIND, LOGB, true, 2, 1>(c, stages);
  if (c.kw == 2 && c.kv && c.vw == 2) return run_multisplit_wide_t<KIND, LOGB, true, 2, 2>(c, stages);
  return cudaErrorInvalidValue;  // 32-bit keys and values take run_multisplit
}

template <int KIND, int LOGB>
cudaError_t run_histogram64_t(const uint64_t* keys, uint32_t n, const BucketParams64& bp, int32_t* hist,
                              cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  static std::atomic<int> per_sm{0};
  auto kern = histogram64_kernel<LOGB, KIND>;
  const uint32_t grid = persistent_grid(kern, HIST_THREADS, uint32_t((uint64_t(n) + HIST_CHUNK - 1) / HIST_CHUNK),
                                        per_sm);
  kern<<<grid, HIST_THREADS, 0, stream>>>(keys, n, hist, bp, bp.num_buckets);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t run_histogram64(const uint64_t* keys, uint32_t n, int logb, const BucketParams64& bp, int32_t* hist,
                            cudaStream_t stream) {
  switch (logb) {
    case 1: return run_histogram64_t<KIND, 1>(keys, n, bp, hist, stream);
    case 2: return run_histogram64_t<KIND, 2>(keys, n, bp, hist, stream);
    case 3: return run_histogram64_t<KIND, 3>(keys, n, bp, hist, stream);
    case 4: return run_histogram64_t<KIND, 4>(keys, n, bp, hist, stream);
    case 5: return run_histogram64_t<KIND, 5>(keys, n, bp, hist, stream);
    case 6: return run_histogram64_t<KIND, 6>(keys, n, bp, hist, stream);
    case 7: return run_histogram64_t<KIND, 7>(keys, n, bp, hist, stream);
    case 8: return run_histogram64_t<KIND, 8>(keys, n, bp, hist, stream);
    default: return cudaErrorInvalidValue;
  }
}

template <int KIND>
cudaError_t run_multisplit_wide(const MsCallWide& c, int stages) {
  switch (c.logb) {
    case 1: return run_multisplit_wide_l<KIND, 1>(c, stages);
    case 2: return run_multisplit_wide_l<KIND, 2>(c, stages);
    case 3: return run_multisplit_wide_l<KIND, 3>(c, stages);
    case 4: return run_multisplit_wide_l<KIND, 4>(c, stages);
    case 5: return run_multisplit_wide_l<KIND, 5>(c, stages);
    case 6: return run_multisplit_wide_l<KIND, 6>(c, stages);
    case 7: return run_multisplit_wide_l<KIND, 7>(c, stages);
    case 8: return run_multisplit_wide_l<KIND, 8>(c, stages);
    default: return cudaErrorInvalidValue;
  }
}

template <int KIND, int LOGB, bool KV, int V>
cudaError_t run_batch_class_t(const BatchClassLaunch& c, int stage) {
  constexpr int WARPS = kTileVariants[V].warps;
  constexpr int IPT = kTileVariants[V].ipt;
  if constexpr (WARPS * 32 < (1 << LOGB)) {
    return cudaErrorInvalidValue;  // the shape has fewer threads than buckets
  } else {
    using C = TileCfg<LOGB, WARPS, IPT, KV>;
    if (c.class_tiles == 0) return cudaSuccess;
    if (stage == STAGE_PRESCAN) {
      static std::atomic<int> per_sm{0};
      auto kern = batch_prescan_kernel<C, KIND>;
      const uint32_t grid = persistent_grid(kern, C::THREADS, c.class_tiles, per_sm);
      kern<<<grid, C::THREADS, 0, c.stream>>>(c.segs, c.tile_map, c.class_tiles, c.matrix, c.byte_area);
      return cudaGetLastError();
    }
    static std::atomic<uint64_t> smem_done{0};
    using P = DescPolicy<KIND, LOGB>;
    constexpr size_t smem = PostLayout<C, P, !P::template CHEAP<KV>>::BYTES;
    auto kern = batch_postscan_kernel<C, KIND>;
    cudaError_t e = ensure_smem_limit(kern, smem, smem_done);
    if (e != cudaSuccess) return e;
    static std::atomic<int> per_sm{0};
    const uint32_t wave = persistent_grid(kern, C::THREADS, c.class_tiles, per_sm, smem);
    kern<<<c.class_tiles, C::THREADS, smem, c.stream>>>(c.segs, c.tile_map, c.matrix, c.hdr, c.byte_area,
                                                        (GMS_PREFETCH_WAVES * wave) / 4u);
    return cudaGetLastError();
  }
}

template <int KIND, bool KV, int V>
cudaError_t run_batch_class_kv(const BatchClassLaunch& c, int stage) {
  switch (c.logb) {
    case 1: return run_batch_class_t<KIND, 1, KV, V>(c, stage);
    case 2: return run_batch_class_t<KIND, 2, KV, V>(c, stage);
    case 3: return run_batch_class_t<KIND, 3, KV, V>(c, stage);
    case 4: return run_batch_class_t<KIND, 4, KV, V>(c, stage);
    case 5: return run_batch_class_t<KIND, 5, KV, V>(c, stage);
    case 6: return run_batch_class_t<KIND, 6, KV, V>(c, stage);
    case 7: return run_batch_class_t<KIND, 7, KV, V>(c, stage);
    case 8: return run_batch_class_t<KIND, 8, KV, V>(c, stage);
    default: return cudaErrorInvalidValue;
  }
}

template <int KIND, int LOGB, bool KV>
cudaError_t run_batch_warp_t(const BatchClassLaunch& c) {
  static_assert(kWarpSegMax == WARP_SEG_MAX, "host and kernel agree on the warp segment size");
  if (c.class_tiles == 0) return cudaSuccess;
  const uint32_t blocks = (c.class_tiles + WARP_SEG_WARPS - 1) / WARP_SEG_WARPS;
  batch_warp_kernel<KIND, LOGB, KV><<<blocks, WARP_SEG_WARPS * 32, 0, c.stream>>>(c.segs, c.seg_ids, c.class_tiles,
                                                                                 c.matrix);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t run_batch_warp(const BatchClassLaunch& c) {
  switch (c.logb) {
    case 1: return c.kv ? run_batch_warp_t<KIND, 1, true>(c) : run_batch_warp_t<KIND, 1, false>(c);
    case 2: return c.kv ? run_batch_warp_t<KIND, 2, true>(c) : run_batch_warp_t<KIND, 2, false>(c);
    case 3: return c.kv ? run_batch_warp_t<KIND, 3, true>(c) : run_batch_warp_t<KIND, 3, false>(c);
    case 4: return c.kv ? run_batch_warp_t<KIND, 4, true>(c) : run_batch_warp_t<KIND, 4, false>(c);
    case 5: return c.kv ? run_batch_warp_t<KIND, 5, true>(c) : run_batch_warp_t<KIND, 5, false>(c);
    case 6: return c.kv ? run_batch_warp_t<KIND, 6, true>(c) : run_batch_warp_t<KIND, 6, false>(c);
    case 7: return c.kv ? run_batch_warp_t<KIND, 7, true>(c) : run_batch_warp_t<KIND, 7, false>(c);
    case 8: return c.kv ? run_batch_warp_t<KIND, 8, true>(c) : run_batch_warp_t<KIND, 8, false>(c);
    default: return cudaErrorInvalidValue;
  }
}

template <int KIND, int V>
cudaError_t run_batch_class_v(const BatchClassLaunch& c, int stage) {
  return c.kv ? run_batch_class_kv<KIND, true, V>(c, stage) : run_batch_class_kv<KIND, false, V>(c, stage);
}

template <int KIND, int LOGB>
cudaError_t run_histogram_t(const uint32_t* keys, uint32_t n, const BucketParams& bp, int32_t* hist,
                            cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  static std::atomic<int> per_sm{0};
  auto kern = histogram_kernel<LOGB, DescPolicy<KIND, LOGB>>;
  const uint32_t grid = persistent_grid(kern, HIST_THREADS, uint32_t((uint64_t(n) + HIST_CHUNK - 1) / HIST_CHUNK), per_sm);
  kern<<<grid, HIST_THREADS, 0, stream>>>(keys, n, hist, bp, bp.num_buckets);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t run_histogram(const uint32_t* keys, uint32_t n, int logb, const BucketParams& bp, int32_t* hist,
                          cudaStream_t stream) {
  switch (logb) {
    case 1: return run_histogram_t<KIND, 1>(keys, n, bp, hist, stream);
    case 2: return run_histogram_t<KIND, 2>(keys, n, bp, hist, stream);
    case 3: return run_histogram_t<KIND, 3>(keys, n, bp, hist, stream);
    case 4: return run_histogram_t<KIND, 4>(keys, n, bp, hist, stream);
    case 5: return run_histogram_t<KIND, 5>(keys, n, bp, hist, stream);
    case 6: return run_histogram_t<KIND, 6>(keys, n, bp, hist, stream);
    case 7: return run_histogram_t<KIND, 7>(keys, n, bp, hist, stream);
    case 8: return run_histogram_t<KIND, 8>(keys, n, bp, hist, stream);
    default: return cudaErrorInvalidValue;
  }
}

// ------------------------------------------- more than 256 buckets
template <int KIND, int LOGB, bool KV>
cudaError_t digit_prescan_scan_t(const DigitPass& c, uint32_t* rows_per, bool* done) {
  using S = TileShape<LOGB, KV>;
  using C = TileCfg<LOGB, S::WARPS, S::IPT, KV>;
  const Geometry g = make_geometry(c.n, LOGB, KV);
  *done = g.num_tiles == 0;
  if (*done) return cudaSuccess;
  if (c.bucket_bytes == nullptr) return cudaErrorInvalidValue;
  cudaError_t e = launch_fused<C, DigitPolicy<KIND, LOGB>>(c.kin, c.vin, c.kout, c.vout, c.n, c.bp, c.scratch,
                                                           g.bytes_full, g, c.stream, nullptr, done);
  if (e != cudaSuccess || *done) return e;
  auto* hdr = reinterpret_cast<ScratchHeader*>(c.scratch);
  auto* status = reinterpret_cast<uint64_t*>(c.scratch + g.off_status);
  auto* matrix = reinterpret_cast<uint32_t*>(c.scratch + g.off_matrix);
  static std::atomic<int> per_sm{0};
  auto kern = prescan_kernel<C, DigitPolicy<KIND, LOGB>>;
  uint32_t* const rows = counts_as_rows(LOGB, g.num_tiles) ? matrix : nullptr;  // nothing reads the matrix afterwards
  const uint32_t grid = rows_grid(persistent_grid(kern, C::THREADS, g.num_tiles, per_sm), rows);
  *rows_per = rows != nullptr ? (g.num_tiles + grid - 1) / grid : 0u;
  kern<<<grid, C::THREADS, 0, c.stream>>>(c.kin, c.n, g.num_tiles, matrix, c.bp, hdr, status, g.num_chunks,
                                          c.bucket_bytes, *rows_per);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (rows != nullptr) return run_scan_rows(rows, C::B, g.num_tiles, *rows_per, status, hdr, c.stream);
  return run_scan(matrix, g.m, status, hdr, c.stream);
}

template <int LOGB, bool KV>
cudaError_t digit_postscan_t(const DigitPass& c) {
  using S = TileShape<LOGB, KV>;
  using C = TileCfg<LOGB, S::WARPS, S::IPT, KV>;
  using P = GivenBytesPolicy;
  const Geometry g = make_geometry(c.n, LOGB, KV);
  if (g.num_tiles == 0) return cudaSuccess;
  if (c.bucket_bytes == nullptr) return cudaErrorInvalidValue;
  auto* hdr = reinterpret_cast<ScratchHeader*>(c.scratch);
  auto* matrix = reinterpret_cast<uint32_t*>(c.scratch + g.off_matrix);
  static std::atomic<uint64_t> smem_done{0};
  static std::atomic<int> per_sm{0};
  auto kern = postscan_kernel<C, P, true>;
  constexpr size_t smem = PostLayout<C, P, true>::BYTES;
  cudaError_t e = ensure_smem_limit(kern, smem, smem_done);
  if (e != cudaSuccess) return e;
  const uint32_t wave = persistent_grid(kern, C::THREADS, g.num_tiles, per_sm, smem);
  const uint32_t dist = (GMS_PREFETCH_WAVES * wave) / 4u;
  return launch_after_previous(kern, dim3(g.num_tiles), dim3(C::THREADS), smem, c.stream, c.kin, c.vin, c.kout,
                               c.vout, c.n, g.num_tiles, matrix, c.bp, hdr, dist, c.bucket_bytes,
                               static_cast<uint32_t*>(nullptr), c.rows_per, static_cast<uint32_t*>(nullptr));
}

#define GMS_DIGIT_SWITCH(ARGS, FN, ...)                           \
  switch (c.logb) {                                               \
    case 1: return c.kv ? FN<__VA_ARGS__ 1, true> ARGS : FN<__VA_ARGS__ 1, false> ARGS; \
    case 2: return c.kv ? FN<__VA_ARGS__ 2, true> ARGS : FN<__VA_ARGS__ 2, false> ARGS; \
    case 3: return c.kv ? FN<__VA_ARGS__ 3, true> ARGS : FN<__VA_ARGS__ 3, false> ARGS; \
    case 4: return c.kv ? FN<__VA_ARGS__ 4, true> ARGS : FN<__VA_ARGS__ 4, false> ARGS; \
    case 5: return c.kv ? FN<__VA_ARGS__ 5, true> ARGS : FN<__VA_ARGS__ 5, false> ARGS; \
    case 6: return c.kv ? FN<__VA_ARGS__ 6, true> ARGS : FN<__VA_ARGS__ 6, false> ARGS; \
    case 7: return c.kv ? FN<__VA_ARGS__ 7, true> ARGS : FN<__VA_ARGS__ 7, false> ARGS; \
    case 8: return c.kv ? FN<__VA_ARGS__ 8, true> ARGS : FN<__VA_ARGS__ 8, false> ARGS; \
    default: return cudaErrorInvalidValue;                        \
  }

template <int KIND>
cudaError_t run_digit_prescan_scan(const DigitPass& c, uint32_t* rows_per, bool* done) {
  GMS_DIGIT_SWITCH((c, rows_per, done), digit_prescan_scan_t, KIND,)
}

template <int KIND>
cudaError_t run_big_histogram(const uint32_t* keys, uint32_t n, const BucketParams& p, uint32_t* hist,
                              cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  const uint32_t work = uint32_t((uint64_t(n) / 4 + HIST_THREADS) / HIST_THREADS);  // blocks of 4-key vectors
  if (p.num_buckets <= BIG_HIST_SMEM_BINS) {
    // Per-block shared histograms; the limit and the occupancy query assume the largest size.
    static std::atomic<int> per_sm{0};
    static std::atomic<uint64_t> smem_done{0};
    auto kern = big_histogram_kernel<KIND, true>;
    const size_t smem = size_t(p.num_buckets) * 4;
    cudaError_t e = ensure_smem_limit(kern, size_t(BIG_HIST_SMEM_BINS) * 4, smem_done,
                                      size_t(big_identifier_smem_words<KIND>()) * 4);
    if (e != cudaSuccess) return e;
    const uint32_t grid = persistent_grid(kern, HIST_THREADS, work, per_sm, size_t(BIG_HIST_SMEM_BINS) * 4);
    kern<<<grid, HIST_THREADS, smem, stream>>>(keys, n, p, hist);
    return cudaGetLastError();
  }
  static std::atomic<int> per_sm{0};
  auto kern = big_histogram_kernel<KIND, false>;
  const uint32_t grid = persistent_grid(kern, HIST_THREADS, work, per_sm);
  kern<<<grid, HIST_THREADS, 0, stream>>>(keys, n, p, hist);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t run_big_offsets(const uint32_t* sorted_keys, uint32_t n, const BucketParams& p, uint32_t* starts,
                            cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  static std::atomic<int> per_sm{0};
  auto kern = big_offsets_kernel<KIND>;
  const uint32_t grid = persistent_grid(kern, HIST_THREADS, uint32_t((uint64_t(n) + HIST_THREADS - 1) / HIST_THREADS),
                                        per_sm);
  kern<<<grid, HIST_THREADS, 0, stream>>>(sorted_keys, n, p, starts);
  return cudaGetLastError();
}

}  // namespace gms

#define GMS_INSTANTIATE_KIND(K)                                                                        \
  template cudaError_t gms::run_multisplit<K>(const gms::MsCall&, int);                                \
  template cudaError_t gms::run_histogram<K>(const uint32_t*, uint32_t, int, const gms::BucketParams&, \
                                             int32_t*, cudaStream_t);

#define GMS_INSTANTIATE_BIG(K)                                                           \
  template cudaError_t gms::run_digit_prescan_scan<K>(const gms::DigitPass&, uint32_t*, bool*);           \
  template cudaError_t gms::run_big_histogram<K>(const uint32_t*, uint32_t, const gms::BucketParams&, uint32_t*, \
                                                 cudaStream_t);                                                 \
  template cudaError_t gms::run_big_offsets<K>(const uint32_t*, uint32_t, const gms::BucketParams&, uint32_t*, \
                                               cudaStream_t);

#define GMS_INSTANTIATE_WIDE(K)                                                                          \
  template cudaError_t gms::run_multisplit_wide<K>(const gms::MsCallWide&, int);                        \
  template cudaError_t gms::run_histogram64<K>(const uint64_t*, uint32_t, int, const gms::BucketParams64&, \
                                               int32_t*, cudaStream_t);

#define GMS_INSTANTIATE_BATCH_WARP(K) template cudaError_t gms::run_batch_warp<K>(const gms::BatchClassLaunch&);

#define GMS_INSTANTIATE_BATCH(K, V) template cudaError_t gms::run_batch_class_v<K, V>(const gms::BatchClassLaunch&, int);
