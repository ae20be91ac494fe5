// Stable multisplit kernels for sm_103a: prescan (per-tile bucket counts) and
// postscan (stable in-tile rank, shared-memory reorder, coalesced scatter).
//
// Semantics follow the reference's block-wide multisplit
// (src/kernels/bms/bms_prescan.cuh, bms_postscan.cuh, bms_postscan_pairs.cuh):
//   * tile t covers keys [t*TILE, (t+1)*TILE) in input order;
//   * the count matrix is bucket-major, counts[b * num_tiles + t]
//     (bms_prescan.cuh:114);
//   * after an exclusive scan of that matrix, the element of bucket b that is
//     the j-th of its bucket inside tile t goes to counts[b*num_tiles+t] + j,
//     which is exactly the order of cpu_multisplit_general
//     (src/cpu_functions.h:155-220).
// The reference pads the last tile into bucket B-1 (bms_prescan.cuh:62-63);
// here the tail is simply not counted, which leaves every global offset the
// same because the padding only ever sits after all real keys.
#pragma once

#include <type_traits>

#include "gms_device.cuh"

// Threads per SM the key-only postscan's register budget is sized for: six
// 256-thread blocks (40 registers) measured 3-5% faster than four (64) at
// B <= 32 and equal above.
#ifndef GMS_KEYS_RESIDENT_THREADS
#define GMS_KEYS_RESIDENT_THREADS 1536
#endif
// The same for the key-value postscan: four blocks of 64 registers (five
// blocks gained 2% at B = 64 and lost 2% at B = 256; six spilled and lost more).
#ifndef GMS_PAIRS_RESIDENT_THREADS
#define GMS_PAIRS_RESIDENT_THREADS 1024
#endif

namespace gms {

// Tile geometry of one (B, key/value, element widths) instance.  KW and VW
// are the 32-bit words of a key and of a value (1 or 2): 64-bit elements.
template <int LOGB_, int WARPS_, int IPT_, bool KV_, int KW_ = 1, int VW_ = 1>
struct TileCfg {
  static constexpr int LOGB = LOGB_;
  static constexpr uint32_t B = 1u << LOGB_;
  static constexpr int WARPS = WARPS_;
  static constexpr int THREADS = WARPS_ * 32;
  static constexpr int IPT = IPT_;  // keys per thread
  static constexpr uint32_t TILE = THREADS * IPT_;
  static constexpr bool KV = KV_;
  static constexpr int KW = KW_;
  static constexpr int VW = VW_;
  static constexpr bool WIDE = KW_ == 2 || (KV_ && VW_ == 2);  // any 64-bit element
  using KT = std::conditional_t<KW_ == 2, uint64_t, uint32_t>;
  using VT = std::conditional_t<VW_ == 2, uint64_t, uint32_t>;
  static_assert((KW_ == 1 || KW_ == 2) && (VW_ == 1 || VW_ == 2), "elements are 32 or 64 bits");
  static constexpr uint32_t WB = B < 32 ? 32 : B;  // row width of the per-warp count table
  // Ranks by shared-memory atomics (postscan_tile); by ballots at the smallest
  // bucket counts, where few ballots suffice and many lanes meet in a counter.
  // At 2^28, ballots / atomics: keys 16 buckets 0.694 / 0.725 ms, 32 buckets
  // 0.770 / 0.692; pairs 32 buckets 0.955 / 0.874.  Pairs into 16 buckets gain
  // on uniform keys (0.893 / 0.866) but lose on skewed ones (2^25 Zipf pairs
  // 123 / 128 us, four of the buckets 121 / 142).
  static constexpr bool ATOMIC = LOGB_ >= 5;
  // Whether the counts can be kept as rows (counts_as_rows in ms_host.h).  Postscans
  // that never meet rows leave that code out: with it, a call at 2^26 pairs took
  // 242 us into 16 buckets instead of 234, 225 into 8 instead of 221.
  static constexpr bool ROWS = LOGB_ >= ROWS_MIN_LOGB;

  static_assert(IPT % 4 == 0, "IPT must be a multiple of 4 (16-byte vector loads)");
  static_assert(TILE <= 65536, "in-tile positions are packed into 16 bits");
  static_assert(THREADS >= static_cast<int>(B), "one thread per bucket in the tile scan");

};

// ------------------------------------------------------------- counting
// Counting keys per bucket.  For the smallest bucket counts every lane keeps
// the count of bucket `lane` in registers, fed by log2(B) ballots per 32 keys;
// otherwise keys are counted with shared-memory atomics into R replicas of a
// B-entry histogram (R = 32/B below 32 buckets, lane l using replica l % R), so
// few lanes of a warp ever hit the same word.
#ifndef GMS_COUNT_BALLOT_MAX_LOGB
#define GMS_COUNT_BALLOT_MAX_LOGB 0
#endif

template <int LOGB, class Id>
struct KeyCounter {
  static constexpr uint32_t B = 1u << LOGB;
  static constexpr bool kBallot = LOGB <= GMS_COUNT_BALLOT_MAX_LOGB;
  static constexpr uint32_t R = B >= 32 ? 1u : 32u / B;  // histogram replicas (atomic path)
  static constexpr uint32_t HIST_WORDS = B * R;         // >= 32
  Id ident;
  uint32_t* s_hist;                      // 2 x HIST_WORDS (atomic path) or WARPS*32 (ballot path)
  uint32_t acc[4] = {0u, 0u, 0u, 0u};    // ballot path: independent accumulators keep the chains parallel
  uint32_t xm[kBallot ? LOGB : 1];
  uint32_t slot;                          // atomic path: this lane's replica offset
  uint32_t buf = 0;                       // atomic path: histogram being filled (0 or HIST_WORDS)

  __device__ __forceinline__ KeyCounter(const Id& id, uint32_t* hist) : ident(id), s_hist(hist) {
    const uint32_t lane = lane_id();
    if constexpr (kBallot) {
#pragma unroll
      for (int i = 0; i < LOGB; ++i) xm[i] = ((lane >> i) & 1u) ? 0u : ~0u;
    }
    slot = lane & (R - 1);
  }

  // Called by all 32 lanes of the warp together; A selects an accumulator.
  template <int A = 0>
  __device__ __forceinline__ void add(uint32_t key, bool valid) {
    add_bucket<A>(ident(key), valid);
  }

  template <int A = 0>
  __device__ __forceinline__ void add_bucket(uint32_t b, bool valid) {
    if constexpr (kBallot) {
      uint32_t m = __ballot_sync(~0u, valid);
#pragma unroll
      for (int i = 0; i < LOGB; ++i) m &= __ballot_sync(~0u, (b >> i) & 1u) ^ xm[i];
      acc[A] += __popc(m);
    } else {
      if (valid) atomicAdd(&s_hist[buf + b * R + slot], 1u);
    }
  }

  // Shared words the counter needs for a block of `warps` warps.  The atomic
  // path keeps two histograms: one tile is read out and cleared while the
  // next one is counted into the other, so a tile needs one barrier.
  __host__ __device__ static constexpr uint32_t smem_words(int warps) {
    return kBallot ? uint32_t(warps) * 32u : 2u * HIST_WORDS;
  }

  // Zero the shared histograms (atomic path); all threads call, a barrier must follow.
  __device__ __forceinline__ void clear_shared() {
    if constexpr (!kBallot) {
      for (uint32_t i = threadIdx.x; i < 2u * HIST_WORDS; i += blockDim.x) s_hist[i] = 0u;
    }
  }

  // Block totals: after the call (which contains a barrier), thread b < B
  // returns the block's count of bucket b, and the counter is ready for the
  // next tile.
  __device__ __forceinline__ uint32_t block_total() {
    const uint32_t tid = threadIdx.x;
    uint32_t total = 0;
    if constexpr (kBallot) {
      const uint32_t lane = tid & 31u, warp = tid >> 5;
      if (lane < B) s_hist[warp * 32 + lane] = acc[0] + acc[1] + acc[2] + acc[3];
      acc[0] = acc[1] = acc[2] = acc[3] = 0u;
      __syncthreads();
      if (tid < B) {
        for (uint32_t w = 0; w < blockDim.x / 32; ++w) total += s_hist[w * 32 + tid];
      }
      __syncthreads();
    } else {
      // The barrier ends this tile's counting; the histogram is cleared here
      // and filled again two tiles later, after the next tile's barrier.
      __syncthreads();
      if (tid < B) {
#pragma unroll
        for (uint32_t r = 0; r < R; ++r) {
          total += s_hist[buf + tid * R + r];
          s_hist[buf + tid * R + r] = 0u;
        }
      }
      buf ^= HIST_WORDS;
    }
    return total;
  }
};

template <int THREADS, int IPT>
__device__ __forceinline__ void load_tile_v4(const uint32_t* __restrict__ keys, uint32_t base, uint4 (&v)[IPT / 4]) {
#pragma unroll
  for (int k = 0; k < IPT / 4; ++k) v[k] = ld_nc_v4(keys + base + (uint32_t(k) * THREADS + threadIdx.x) * 4u);
}

// Counts one tile held as 16-byte vectors (thread t holds keys
// (k*THREADS + t)*4 .. +3 of vector k).  WRITE_BYTES: also stores every key's
// bucket as one byte at bytes_out[(k*THREADS + t)*4 ..] (four per store).
template <int THREADS, int IPT, bool WRITE_BYTES = false, class Counter>
__device__ __forceinline__ void count_v4(const uint4 (&v)[IPT / 4], Counter& c, uint8_t* bytes_out = nullptr) {
#pragma unroll
  for (int k = 0; k < IPT / 4; ++k) {
    const uint32_t b0 = c.ident(v[k].x), b1 = c.ident(v[k].y), b2 = c.ident(v[k].z), b3 = c.ident(v[k].w);
    c.template add_bucket<0>(b0, true);
    c.template add_bucket<1>(b1, true);
    c.template add_bucket<2>(b2, true);
    c.template add_bucket<3>(b3, true);
    if constexpr (WRITE_BYTES)
      reinterpret_cast<uint32_t*>(bytes_out)[uint32_t(k) * THREADS + threadIdx.x] =
          b0 | (b1 << 8) | (b2 << 16) | (b3 << 24);
  }
}

// Counts tiles first, first+stride, ... (tiles of THREADS*IPT keys) and calls
// done(tile) after each one.  The next tile's keys are loaded into registers
// while the current tile is counted, so loads stay in flight.  WRITE_BYTES:
// every key's bucket is also stored as one byte at bytes_out[key index].
template <int THREADS, int IPT, bool WRITE_BYTES = false, class Counter, class Done>
__device__ __forceinline__ void count_tiles(const uint32_t* __restrict__ keys, uint32_t n, uint32_t first,
                                            uint32_t stride, Counter& c, Done done, uint8_t* bytes_out = nullptr,
                                            uint32_t last = ~0u) {
  constexpr uint32_t TILE = uint32_t(THREADS) * IPT;
  const uint32_t num_tiles = min(uint32_t((uint64_t(n) + TILE - 1) / TILE), last);
  const bool vec_ok = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;
  const uint32_t full_tiles = vec_ok ? min(n / TILE, num_tiles) : 0u;  // tiles read with vector loads
  uint4 cur[IPT / 4];
  if (first < full_tiles) load_tile_v4<THREADS, IPT>(keys, first * TILE, cur);
  for (uint32_t tile = first; tile < num_tiles; tile += stride) {
    const uint32_t next = tile + stride;
    uint4 nxt[IPT / 4];
    if (next < full_tiles) load_tile_v4<THREADS, IPT>(keys, next * TILE, nxt);
    if (tile < full_tiles) {
      count_v4<THREADS, IPT, WRITE_BYTES>(cur, c, WRITE_BYTES ? bytes_out + size_t(tile) * TILE : nullptr);
    } else {
      const uint32_t base = tile * TILE;
      const uint32_t cnt = min(TILE, n - base);
#pragma unroll 4
      for (int k = 0; k < IPT; ++k) {
        const uint32_t i = uint32_t(k) * THREADS + threadIdx.x;
        const bool valid = i < cnt;
        const uint32_t b = c.ident(valid ? keys[base + i] : 0u);
        c.add_bucket(b, valid);
        if constexpr (WRITE_BYTES) {
          if (valid) bytes_out[base + i] = uint8_t(b);
        }
      }
    }
    done(tile);
#pragma unroll
    for (int k = 0; k < IPT / 4; ++k) cur[k] = nxt[k];
  }
}

// --------------------------------------------------------------- prescan
// Persistent grid over the tiles.  Writes counts[b * num_tiles + tile] for
// every tile and resets the scan state (ticket, chunk status words, error
// word) for the scan that follows.
//
// bucket_bytes (identifiers costly to evaluate; may be null): every key's
// bucket is also stored there as one byte, so the postscan need not evaluate
// the identifier again.
//
// Each block counts a contiguous run of tiles, ceil(tiles / blocks) of them, and
// keeps the counts of PRESCAN_GROUP tiles in shared memory, then writes them
// bucket by bucket: a warp stores whole runs of consecutive matrix words (the
// matrix is bucket-major) instead of one scattered word per bucket and tile.
// In ranges of at least two groups the groups are those of the matrix, [8 g,
// 8 g + 8), wherever a range begins: groups counted from a range's own start
// write every sector in two parts, which leave L2 separately once the matrix is
// large (256 buckets, us, groups of the range / of the matrix: 2^27 keys 96 / 92,
// 2^28 208 / 183, 2^30 855 / 723).  Shorter ranges count from their start: the
// matrix's groups would cut them in two (2^24 keys 16.9 / 18.4).
//
// rows_per != 0 (the one-call path): the counts go into rows instead,
// counts[tile * B + b], one coalesced store per tile.  A block's range is then
// rows_per tiles, each row holds the counts of the range's earlier tiles, and
// the range's first row, whose sums would be zero, the range's totals; only
// those rows are scanned (scan_rows_kernel), and the postscan adds the two rows
// of its tile, each read as whole sectors.  The bucket-major matrix made the
// postscan read a sector for every bucket: of its 145 us for 2^25 pairs at 256
// buckets (113 for keys) 18 (16) went into those loads, and the scan ran over
// all counts.
constexpr uint32_t PRESCAN_GROUP = 8;

// Tiles of a prescan block's range.  whole_groups: a multiple of the group where
// that lengthens the range by at most a sixteenth, so that no two blocks write
// to one sector.
__host__ __device__ inline uint32_t prescan_tiles_per_block(uint32_t num_tiles, uint32_t blocks, bool whole_groups) {
  const uint32_t per = (num_tiles + blocks - 1) / blocks;
  const uint32_t whole = (per + PRESCAN_GROUP - 1) / PRESCAN_GROUP * PRESCAN_GROUP;
  return whole_groups && (whole - per) * 16u <= per ? whole : per;
}

// Where ranges of whole groups pay: with identifiers that leave the prescan bound
// by memory (us, any range / whole groups: 256 buckets 2^28 keys 183 / 178, 2^30
// 723 / 695; 190 M keys, ranges of 62 / 64 tiles: 16 buckets 128 / 115, 64 130 /
// 115, 128 135 / 118).  A splitter search is bound by its longest range (256
// buckets, 2^28 keys 330 / 340).
template <class P>
__host__ __device__ constexpr bool prescan_whole_groups() {
  return !P::USES_SMEM;
}

template <class C>
struct PrescanCounts {
  static constexpr uint32_t B = C::B;
  static constexpr uint32_t G = PRESCAN_GROUP;
  uint32_t* counts;
  uint32_t* s_cnt;  // B * G words
  uint32_t num_tiles, first, last;
  uint32_t origin;  // where groups are counted from
  bool rows;
  uint32_t run;     // rows: count of bucket tid in the range so far

  __device__ __forceinline__ PrescanCounts(uint32_t* counts_, uint32_t* s_cnt_, uint32_t num_tiles_, uint32_t rows_per,
                                           bool whole_groups)
      : counts(counts_), s_cnt(s_cnt_), num_tiles(num_tiles_), rows(rows_per != 0), run(0) {
    const uint32_t per = rows ? rows_per : prescan_tiles_per_block(num_tiles, gridDim.x, whole_groups);
    first = min(blockIdx.x * per, num_tiles);
    last = min(first + per, num_tiles);
    origin = per < 2 * G ? first : 0u;
  }
  // Called by all threads after each tile; thread tid < B has the tile's count of bucket tid.
  __device__ __forceinline__ void done(uint32_t tile, uint32_t total) {
    const uint32_t tid = threadIdx.x;
    if (rows) {
      if (tid < B) {
        if (tile != first) counts[tile * B + tid] = run;
        run += total;
        if (tile + 1 == last) counts[first * B + tid] = run;
      }
      return;
    }
    const uint32_t g = (tile - origin) % G;
    if (tid < B) s_cnt[tid * G + g] = total;
    if (g == G - 1 || tile + 1 == last) {
      const uint32_t group_first = tile - g;
      __syncthreads();
      for (uint32_t i = tid; i < B * G; i += C::THREADS) {
        const uint32_t t = group_first + i % G;
        if (t >= first && t < last) counts[(i / G) * num_tiles + t] = s_cnt[i];
      }
      __syncthreads();
    }
  }
};

// A splitter search gets the registers of four blocks per SM: at five (48, where
// the compiler may stop by itself) it spills, and each block more prepares the
// splitters once more (2^22 range keys into 4096 buckets 88 us, at four 80).
// Other identifiers: the compiler's choice (0).
template <class C, class P>
__host__ __device__ constexpr int prescan_min_blocks() {
  return P::USES_SMEM ? 1024 / C::THREADS : 0;
}

template <class C, class P>
__global__ void __launch_bounds__(C::THREADS, (prescan_min_blocks<C, P>()))
    prescan_kernel(const uint32_t* __restrict__ keys, uint32_t n, uint32_t num_tiles, uint32_t* __restrict__ counts,
                   typename P::Params bp, ScratchHeader* hdr, uint64_t* __restrict__ status, uint32_t num_chunks,
                   uint8_t* __restrict__ bucket_bytes, uint32_t rows_per) {
  griddep_launch_dependents();  // the scan may be scheduled now; it waits for this grid
  using Counter = KeyCounter<C::LOGB, typename P::Id>;
  constexpr uint32_t G = PRESCAN_GROUP;
  __shared__ uint32_t s_hist[Counter::smem_words(C::WARPS)];
  __shared__ uint32_t s_split[P::SMEM_WORDS];  // identifier state (RANGE splitters + table)
  __shared__ uint32_t s_cnt[C::B * G];         // counts of the current group of tiles, bucket-major

  const uint32_t tid = threadIdx.x;

  // Reset the scan state for this call.
  for (uint32_t i = blockIdx.x * C::THREADS + tid; i < num_chunks; i += gridDim.x * C::THREADS) status[i] = 0ull;
  if (blockIdx.x == 0 && tid == 0) {
    hdr->error = 0u;
    hdr->error_info = 0u;
    hdr->ticket = 0u;
    hdr->wait_limit_us = 0u;
  }

  P::prepare(s_split, bp);
  Counter counter(P::make(bp, s_split), s_hist);
  counter.clear_shared();
  __syncthreads();
  PrescanCounts<C> out(counts, s_cnt, num_tiles, rows_per, prescan_whole_groups<P>());
  auto done = [&](uint32_t tile) { out.done(tile, counter.block_total()); };
  if constexpr (!P::template CHEAP<C::KV>) {
    if (bucket_bytes != nullptr) {
      count_tiles<C::THREADS, C::IPT, true>(keys, n, out.first, 1u, counter, done, bucket_bytes, out.last);
      return;
    }
  }
  count_tiles<C::THREADS, C::IPT>(keys, n, out.first, 1u, counter, done, nullptr, out.last);
}

// ------------------------------------------------ prescan, 64-bit keys
// The prescan for 64-bit keys: the same tiles, counts, group flush and scan
// reset as prescan_kernel, and every key's bucket is always stored as one
// byte (the 64-bit postscan reads them instead of the keys' identifier).
// In a full tile, thread t loads keys 2(k*THREADS + t) and the next one as one
// 16-byte vector, for k < IPT/2; the next tile's vectors are in flight while
// the current tile is counted.
template <int THREADS, int IPT>
__device__ __forceinline__ void load_tile64(const uint64_t* __restrict__ keys, uint32_t base,
                                            uint4 (&v)[IPT / 2]) {
#pragma unroll
  for (int k = 0; k < IPT / 2; ++k)
    v[k] = ld_nc_v4(reinterpret_cast<const uint32_t*>(keys + base + (uint32_t(k) * THREADS + threadIdx.x) * 2u));
}

template <class C, class P>
__global__ void __launch_bounds__(C::THREADS) prescan64_kernel(const uint64_t* __restrict__ keys, uint32_t n,
                                                               uint32_t num_tiles, uint32_t* __restrict__ counts,
                                                               typename P::Params bp, ScratchHeader* hdr,
                                                               uint64_t* __restrict__ status, uint32_t num_chunks,
                                                               uint8_t* __restrict__ bucket_bytes, uint32_t rows_per) {
  griddep_launch_dependents();  // the scan may be scheduled now; it waits for this grid
  using Counter = KeyCounter<C::LOGB, typename P::Id>;
  constexpr uint32_t G = PRESCAN_GROUP;
  constexpr uint32_t TILE = C::TILE;
  constexpr int NV = C::IPT / 2;
  __shared__ uint32_t s_hist[Counter::smem_words(C::WARPS)];
  __shared__ __align__(16) uint32_t s_split[P::SMEM_WORDS];  // RANGE: 64-bit splitters + table
  __shared__ uint32_t s_cnt[C::B * G];

  const uint32_t tid = threadIdx.x;
  for (uint32_t i = blockIdx.x * C::THREADS + tid; i < num_chunks; i += gridDim.x * C::THREADS) status[i] = 0ull;
  if (blockIdx.x == 0 && tid == 0) {
    hdr->error = 0u;
    hdr->error_info = 0u;
    hdr->ticket = 0u;
    hdr->wait_limit_us = 0u;
  }

  P::prepare(s_split, bp);
  Counter counter(P::make(bp, s_split), s_hist);
  counter.clear_shared();
  __syncthreads();
  PrescanCounts<C> out(counts, s_cnt, num_tiles, rows_per, prescan_whole_groups<P>());
  const uint32_t first = out.first, last = out.last;
  const bool vec_ok = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;
  const uint32_t full_tiles = vec_ok ? min(n / TILE, last) : 0u;
  uint4 cur[NV];
  if (first < full_tiles) load_tile64<C::THREADS, C::IPT>(keys, first * TILE, cur);
  for (uint32_t tile = first; tile < last; ++tile) {
    uint4 nxt[NV];
    if (tile + 1 < full_tiles) load_tile64<C::THREADS, C::IPT>(keys, (tile + 1) * TILE, nxt);
    const uint32_t base = tile * TILE;
    if (tile < full_tiles) {
      uint16_t* bytes = reinterpret_cast<uint16_t*>(bucket_bytes + base);
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        const uint32_t b0 = counter.ident(uint64_t(cur[k].x) | (uint64_t(cur[k].y) << 32));
        const uint32_t b1 = counter.ident(uint64_t(cur[k].z) | (uint64_t(cur[k].w) << 32));
        counter.template add_bucket<0>(b0, true);
        counter.template add_bucket<1>(b1, true);
        bytes[uint32_t(k) * C::THREADS + tid] = uint16_t(b0 | (b1 << 8));
      }
    } else {
      const uint32_t cnt = min(TILE, n - base);
#pragma unroll 4
      for (int k = 0; k < C::IPT; ++k) {
        const uint32_t i = uint32_t(k) * C::THREADS + tid;
        const bool valid = i < cnt;
        const uint32_t b = counter.ident(valid ? keys[base + i] : 0ull);
        counter.add_bucket(b, valid);
        if (valid) bucket_bytes[base + i] = uint8_t(b);
      }
    }
    out.done(tile, counter.block_total());
#pragma unroll
    for (int k = 0; k < NV; ++k) cur[k] = nxt[k];
  }
}

// Shared-memory layout of the postscan for identifier policy P (bytes), and
// what phase 3 writes at each key's bucket-sorted position:
//   R_KEYS       the key (key-only, identifier cheap to recompute): phase 4
//                reads keys conflict-free and recomputes their buckets;
//   R_INDEX16    the key's 16-bit in-tile index (key-value, cheap identifier):
//                a small buffer keeps four tiles resident per SM;
//   R_KEYS_B,    the same plus the key's bucket as one byte, for identifiers
//   R_INDEX16_B  that are costly to recompute (RANGE, DIV, EVEN_FLOAT, user
//                functors); index and bucket as one word where there is room.
// With ranks by atomics the source index is always kept (R_INDEX16, R_INDEX16_B):
// it shows whether the ranks kept the input order.  The per-warp count table
// then holds 32-bit entries, which the atomics need, else 16-bit ones (a warp
// counts at most 32 * IPT keys and a tile holds at most 2^16).
enum ReorderMode { R_KEYS = 0, R_INDEX16 = 1, R_KEYS_B = 2, R_INDEX16_B = 3 };

template <class C, class P, bool GIVEN = false>
struct PostLayout {
  static constexpr bool CHEAP = P::template CHEAP<C::KV>;
  static_assert(!GIVEN || !P::template CHEAP<C::KV>, "given bucket bytes are only used for costly identifiers");
  static_assert(C::KW == 1 || GIVEN, "64-bit keys take their buckets from the prescan's bytes");
  // Keys are reordered through a 16-bit index whenever values come along, keys
  // are 64 bits wide (a sorted copy of the keys would take more room) or the
  // ranks come from atomics.
  static constexpr int MODE =
      (C::KV || C::KW == 2 || C::ATOMIC) ? (CHEAP ? R_INDEX16 : R_INDEX16_B) : (CHEAP ? R_KEYS : R_KEYS_B);
  static constexpr bool INDEXED = MODE == R_INDEX16 || MODE == R_INDEX16_B;
  static constexpr bool BUCKET_BYTES = MODE == R_KEYS_B || MODE == R_INDEX16_B;
  using WhT = std::conditional_t<C::ATOMIC, uint32_t, uint16_t>;
  // Blocks per SM the register budget is sized for (64 registers at 16 keys per thread).
  static constexpr int RESIDENT_THREADS = C::IPT <= 8 ? 1536 : (C::KV ? GMS_PAIRS_RESIDENT_THREADS : GMS_KEYS_RESIDENT_THREADS);
  static constexpr int THREAD_BLOCKS = RESIDENT_THREADS / C::THREADS > 0 ? RESIDENT_THREADS / C::THREADS : 1;
  static constexpr size_t OFF_K = 0;
  static constexpr size_t OFF_V = OFF_K + size_t(C::TILE) * sizeof(typename C::KT);
  static constexpr size_t OFF_R = OFF_V + (C::KV ? size_t(C::TILE) * sizeof(typename C::VT) : 0);
  // With ranks by atomics, a kept bucket and the source index go into one
  // 32-bit word (one scattered store instead of two) where that costs no
  // resident block (228 KB per SM, 1 KB of it reserved per block).
  static constexpr size_t REST = OFF_R + size_t(C::WARPS) * C::WB * sizeof(WhT) + C::B * 4 +
                                 (GIVEN ? 0 : P::SMEM_WORDS * 4) + 256;
  static constexpr int blocks_at(size_t per_key) {
    const int by_smem = int((228u * 1024u) / (REST + size_t(C::TILE) * per_key + 1024u));
    return by_smem < THREAD_BLOCKS ? by_smem : THREAD_BLOCKS;
  }
  static constexpr bool WORDS = C::ATOMIC && BUCKET_BYTES && blocks_at(4) >= blocks_at(3);
  static constexpr size_t R_BYTES = size_t(C::TILE) * (INDEXED && !WORDS ? 2 : 4);
  // Bucket bytes; under the words the staged ones lie where the words go, read
  // in phase 1 before phase 3 writes.
  static constexpr size_t OFF_RB = WORDS ? OFF_R : OFF_R + R_BYTES;
  static constexpr size_t END_R = WORDS ? OFF_R + R_BYTES : OFF_RB + (BUCKET_BYTES ? C::TILE : 0);
  static constexpr size_t OFF_WH = (END_R + 15) & ~size_t(15);
  static constexpr size_t OFF_DELTA = (OFF_WH + size_t(C::WARPS) * C::WB * sizeof(WhT) + 15) & ~size_t(15);
  static constexpr size_t OFF_SPLIT = OFF_DELTA + C::B * 4;
  // With bucket bytes from the prescan the identifier is never evaluated, so
  // it needs no shared area.
  static constexpr size_t OFF_SCAN = OFF_SPLIT + (GIVEN ? 0 : P::SMEM_WORDS * 4);
  static constexpr size_t OFF_FLAG = OFF_SCAN + 32 * 4;  // warp totals of the tile scan
  static constexpr size_t OFF_BAR = (OFF_FLAG + 4 + 15) & ~size_t(15);
  static constexpr size_t BYTES = OFF_BAR + 16;
  // With 64-bit elements shared memory bounds the blocks per SM first.
  static constexpr int SMEM_BLOCKS = int((228u * 1024u) / (BYTES + 1024u));
  static constexpr int MIN_BLOCKS =
      C::WIDE ? (SMEM_BLOCKS < THREAD_BLOCKS ? (SMEM_BLOCKS > 0 ? SMEM_BLOCKS : 1) : THREAD_BLOCKS) : THREAD_BLOCKS;
};

// Puts the source indices of one bucket's run into ascending order (the input's
// order).  An insertion sort: runs that are nearly in order cost one pass.
template <class T>
__host__ __device__ inline void sort_run(T* run, uint32_t n) {
  for (uint32_t i = 1; i < n; ++i) {
    const T v = run[i];
    uint32_t k = i;
    for (; k > 0 && run[k - 1] > v; --k) run[k] = run[k - 1];
    run[k] = v;
  }
}

// Peer mask (lanes of this warp whose key in this slot has bucket b) from
// log2(B) bit-plane ballots: lanes agree on bit i iff ballot_i ^ own_i is set,
// with own_i = 0 or ~0 by this lane's bit i.
template <int LOGB>
__device__ __forceinline__ uint32_t peers_by_ballot(uint32_t b) {
  uint32_t peers = ~0u;
#pragma unroll
  for (int i = 0; i < LOGB; ++i) {
    const uint32_t bal = __ballot_sync(~0u, (b >> i) & 1u);
    const uint32_t own = ((b >> i) & 1u) - 1u;  // bit set -> 0, clear -> ~0
    peers &= bal ^ own;
  }
  return peers;
}

// Lanes of a warp's first slot in one bucket from which on the warp treats its
// most frequent buckets apart (with 32 buckets a crowd of 8 is no sign of skew:
// 2^25 Zipf pairs took 130 us at 8 lanes and 124 at 12).
__host__ __device__ constexpr uint32_t rank_crowd(int logb) { return logb <= 5 ? 12u : 8u; }

// Where a tile's global bucket offsets come from.  Thread b < B holds the
// source for bucket b: aggregate() is called once the tile's count of bucket b
// is known (phase 2); offset() returns the bucket's global offset for this
// tile, in phase 2 when KNOWN_EARLY, else after the tile is sorted in shared
// memory (phase 3), just before the global stores.  GivenOffset is an entry of
// the scanned count matrix, loaded when the tile starts.
struct GivenOffset {
  static constexpr bool KNOWN_EARLY = true;  // resolved in phase 2, before the reorder
  uint32_t goff;
  __device__ __forceinline__ void aggregate(uint32_t, uint32_t) {}
  __device__ __forceinline__ uint32_t offset(uint32_t, uint32_t) { return goff; }
};

// Whether a source of offsets is resolved by all threads of the block together
// (it has a resolve()), after phase 3 and before offset().
template <class O, class = void>
struct requires_resolve : std::false_type {};
template <class O>
struct requires_resolve<O, std::void_t<decltype(&O::resolve)>> : std::true_type {};

// The default source of a job's offsets: its entries of the scanned count
// matrix (minus the job's bias in a shared scan).
struct MatrixOffsets {
  template <class Job>
  __device__ __forceinline__ GivenOffset operator()(const Job& job, uint32_t tid, uint32_t num_buckets) const {
    return GivenOffset{tid < num_buckets ? job.offsets[tid * job.num_tiles + job.tile] - job.bias : 0u};
  }
};

// The same from the prescan's rows (per tiles a range, see prescan_kernel);
// per == 0: job.offsets is the bucket-major matrix.
struct RowOffsets {
  uint32_t per;

  template <class Job>
  __device__ __forceinline__ GivenOffset operator()(const Job& job, uint32_t tid, uint32_t num_buckets) const {
    if (per == 0) return MatrixOffsets()(job, tid, num_buckets);
    if (tid >= num_buckets) return GivenOffset{0u};
    const uint32_t first = job.tile - job.tile % per;
    const uint32_t range = job.offsets[first * num_buckets + tid];
    return GivenOffset{job.tile == first ? range : range + job.offsets[job.tile * num_buckets + tid]};
  }
};

// Tiles whose offsets one block moves from the rows to the matrix.
constexpr uint32_t MATRIX_TILES = 32;

// Fills the bucket-major matrix that the caller sees from the rows, for tiles
// [t0, t0 + MATRIX_TILES): through shared memory, whole rows in and runs of 32
// words out.  Extra blocks of the postscan's grid do this while its last tiles
// drain; done by every eighth tile's own block it took 85 us of a 1360 us call
// (2^28 pairs, 256 buckets).
template <uint32_t B>
__device__ __forceinline__ void rows_to_matrix(const uint32_t* __restrict__ rows, uint32_t* __restrict__ matrix,
                                               uint32_t num_tiles, uint32_t per, uint32_t t0, uint32_t* s) {
  const uint32_t tiles = min(MATRIX_TILES, num_tiles - t0);
  for (uint32_t i = threadIdx.x; i < tiles * B; i += blockDim.x) {
    const uint32_t t = t0 + i / B, b = i % B;
    const uint32_t first = t - t % per;
    s[(i / B) * (B + 1) + b] = rows[first * B + b] + (t != first ? rows[t * B + b] : 0u);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < MATRIX_TILES * B; i += blockDim.x) {
    const uint32_t k = i % MATRIX_TILES, b = i / MATRIX_TILES;
    if (k < tiles) matrix[b * num_tiles + t0 + k] = s[k * (B + 1) + b];
  }
}

// Phase 4 of a tile ranked by atomics: calls store(p, source, bucket) for every
// sorted position p < cnt of the staged tile.  Each warp stores runs of RUN times
// 32 positions and checks beside it that (bucket, source) ascends from each
// position to the next, by a shuffle; from run to run one thread each checks.  If
// it does not somewhere in the tile, every bucket's run is put in order and the
// tile is stored again.
// Longer runs leave fewer places between them to check (the 7-bit sort of 2^25
// keys: 551 us at one, 543 at four); at 256 buckets, whose runs are shortest,
// pairs want the block's stores close together (the 8-bit sort of 2^25 pairs: 606
// us at one, 638 at four).
template <class C, class P, bool FULL, bool GIVEN, class Store>
__device__ __forceinline__ void store_in_order(uint32_t cnt, const typename P::Id& ident, unsigned char* smem,
                                               Store store) {
  using L = PostLayout<C, P, GIVEN>;
  using IndexT = std::conditional_t<L::WORDS, uint32_t, uint16_t>;
  constexpr int IPT = C::IPT;
  constexpr uint32_t B = C::B;
  constexpr uint32_t RUN = C::KV && C::LOGB == 8 ? 1 : 4;
  const typename C::KT* s_k = reinterpret_cast<const typename C::KT*>(smem + L::OFF_K);
  IndexT* s_idx = reinterpret_cast<IndexT*>(smem + L::OFF_R);
  const uint8_t* s_rb = reinterpret_cast<const uint8_t*>(smem + L::OFF_RB);
  const typename L::WhT* s_wh = reinterpret_cast<const typename L::WhT*>(smem + L::OFF_WH);
  const uint32_t tid = threadIdx.x;
  const uint32_t lane = tid & 31u;
  const uint32_t warp = tid >> 5;
  // (bucket << 16) | source of sorted position p.
  auto entry = [&](uint32_t p) -> uint32_t {
    const uint32_t e = s_idx[p];
    if constexpr (L::WORDS)
      return e;
    else if constexpr (L::BUCKET_BYTES)
      return (uint32_t(s_rb[p]) << 16) | e;
    else
      return (ident(s_k[e]) << 16) | e;
  };
  for (int attempt = 0; attempt < 2; ++attempt) {
    bool late = false;
    uint32_t before = 0;  // lane 0: entry of the position before its slot
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const uint32_t p = (uint32_t(j) / RUN * C::WARPS + warp) * (32u * RUN) + uint32_t(j) % RUN * 32u + lane;
      uint32_t at = ~0u;
      if (FULL || p < cnt) {
        at = entry(p);
        store(p, at & 0xFFFFu, at >> 16);
      }
      const uint32_t left = __shfl_sync(~0u, at, (lane + 31u) & 31u);
      late |= (lane != 0 ? left : j % RUN == 0 ? 0u : before) > at;
      before = left;
    }
    for (uint32_t p = 32u * RUN * (tid + 1u); p < cnt; p += 32u * RUN * C::THREADS) late |= entry(p - 1) > entry(p);
    if (!__syncthreads_or(late)) break;
    if (tid < B) {  // s_wh[b] of warp 0 is the start of bucket b's run
      const uint32_t first = s_wh[tid], last = tid + 1 < B ? uint32_t(s_wh[tid + 1]) : cnt;
      sort_run(s_idx + first, last - first);
    }
    __syncthreads();
  }
}

// Phases 1-4 of the postscan for one staged tile.  FULL: the tile holds
// exactly TILE keys, so no per-key validity test is needed.
//
// GIVEN: the tile's buckets were staged as bytes at the bucket-byte area (in
// input order) by the caller, so the identifier is not evaluated; phase 3
// overwrites that area with the buckets in sorted order.  Else, unless P::ANY_KEY,
// position 0 holds one of the input's keys even if the tile is empty.
//
// STREAM_HINTS: the output stores mark their L2 lines evict-first (the batch
// queue keeps keys that are read twice in L2 meanwhile; 32-bit elements).
template <class C, class P, bool FULL, bool GIVEN = false, class Offsets = GivenOffset, bool STREAM_HINTS = false>
__device__ __forceinline__ bool postscan_tile(typename C::KT* __restrict__ kout, typename C::VT* __restrict__ vout,
                                              uint32_t n, uint32_t cnt, Offsets& offs, const typename P::Params& bp,
                                              ScratchHeader* hdr, unsigned char* smem) {
  using L = PostLayout<C, P, GIVEN>;
  using WhT = typename L::WhT;
  using KT = typename C::KT;
  using VT = typename C::VT;
  constexpr uint32_t B = C::B;
  constexpr int LOGB = C::LOGB;
  constexpr int IPT = C::IPT;
  constexpr uint32_t WB = C::WB;
  KT* s_k = reinterpret_cast<KT*>(smem + L::OFF_K);
  VT* s_v = reinterpret_cast<VT*>(smem + L::OFF_V);
  uint32_t* s_r = reinterpret_cast<uint32_t*>(smem + L::OFF_R);
  uint8_t* s_rb = reinterpret_cast<uint8_t*>(smem + L::OFF_RB);
  WhT* s_wh = reinterpret_cast<WhT*>(smem + L::OFF_WH);
  uint32_t* s_delta = reinterpret_cast<uint32_t*>(smem + L::OFF_DELTA);
  const uint32_t* s_split = reinterpret_cast<const uint32_t*>(smem + L::OFF_SPLIT);
  uint32_t* s_scan = reinterpret_cast<uint32_t*>(smem + L::OFF_SCAN);
  uint32_t* s_flag = reinterpret_cast<uint32_t*>(smem + L::OFF_FLAG);
  const uint32_t tid = threadIdx.x;
  const uint32_t lane = tid & 31u;
  const uint32_t warp = tid >> 5;

  // ---- 1. stable in-warp ranks
  const typename P::Id ident = P::make(bp, s_split);
  // Bucket of the staged key at in-tile position pos.  Past a partial tile's keys
  // shared memory holds anything: where the identifier is not to see that, those
  // slots take position 0's key.  (A branch around each evaluation kept a warp's
  // searches from overlapping: 10007 range pairs 8.4 -> 10.3 us; and the clamp
  // costs the key-only kernel into 32 buckets a spill, 2 % of a 5-bit sort.)
  auto bucket_at = [&](uint32_t pos) -> uint32_t {
    if constexpr (GIVEN)
      return uint32_t(s_rb[pos]) & (B - 1);
    else
      return ident(s_k[FULL || P::ANY_KEY || pos < cnt ? pos : 0u]);
  };
  uint32_t packed[IPT];  // (bucket << 16) | rank among same-bucket keys of this warp
  const uint32_t wbase = warp * (IPT * 32u);
  const uint32_t lt = lanemask_lt();
  if constexpr (C::ATOMIC) {
    // A key's rank is what an atomic add on its bucket's counter returns.  The
    // adds of a warp do not depend on one another, so all its slots are in
    // flight at once, where ballots took 4 LOGB instructions a slot and a
    // read-modify-write of the count table that each slot waited for: ranking
    // 2^28 keys alone took 0.68 ms with ballots and takes 0.18 at 256 buckets
    // (0.62 and 0.17 at 128).  Lanes of one slot that meet in a bucket are
    // served in lane order on this chip, but nothing promises it: phase 4
    // checks every tile's order and repairs a run that is out of order.
    // Postscan of 2^25 elements, ballots / atomics: keys 128 buckets 112 / 88
    // us, 256 125 / 104; pairs 128 buckets 130 / 111, 256 148 / 143.
    uint32_t* wh = reinterpret_cast<uint32_t*>(s_wh) + warp * WB;
#pragma unroll
    for (int j = 0; j < IPT; ++j) packed[j] = bucket_at(wbase + uint32_t(j) * 32u + lane) << 16;
    // Lanes that meet in a counter are served one after another, so a warp
    // whose first slot is crowded takes its two most frequent buckets by one
    // ballot each, their counts in registers; if a third is crowded too, four
    // (32 lanes have no room for a fifth crowd).
    const uint32_t b0 = packed[0] >> 16;
    const uint32_t peers0 =
        FULL ? peers_by_ballot<LOGB>(b0) : peers_by_ballot<LOGB>(b0) & __ballot_sync(~0u, wbase + lane < cnt);
    const uint32_t crowd = (uint32_t(__popc(peers0)) << 16) | b0;
    const uint32_t most = __reduce_max_sync(~0u, crowd);
    if ((most >> 16) < rank_crowd(LOGB)) {
#pragma unroll
      for (int j = 0; j < IPT; ++j) {
        const uint32_t pos = wbase + uint32_t(j) * 32u + lane;
        if (FULL || pos < cnt) packed[j] |= atomicAdd(wh + (packed[j] >> 16), 1u);
      }
    } else {
      // Ranks with the D most frequent buckets d[] (0xFFFF: none) taken by ballots.
      auto rank_apart = [&](auto count, const uint32_t* d) {
        constexpr int D = decltype(count)::value;
        uint32_t run[D];
#pragma unroll
        for (int i = 0; i < D; ++i) run[i] = 0;
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
          const bool valid = FULL || wbase + uint32_t(j) * 32u + lane < cnt;
          const uint32_t b = packed[j] >> 16;
          bool apart = !valid;
#pragma unroll
          for (int i = 0; i < D; ++i) {
            const bool mine = valid && b == d[i];
            const uint32_t m = __ballot_sync(~0u, mine);
            if (mine) packed[j] |= run[i] + __popc(m & lt);
            apart |= mine;
            run[i] += __popc(m);
          }
          if (!apart) packed[j] |= atomicAdd(wh + b, 1u);
        }
#pragma unroll
        for (int i = 0; i < D; ++i) {
          if (lane == 0 && d[i] < B) wh[d[i]] = run[i];
        }
      };
      uint32_t d[4];
      d[0] = most & 0xFFFFu;
      uint32_t left = b0 == d[0] ? 0u : crowd;
#pragma unroll
      for (int i = 1; i < 4; ++i) {
        const uint32_t next = __reduce_max_sync(~0u, left);
        d[i] = next != 0u ? next & 0xFFFFu : 0xFFFFu;
        if (b0 == d[i]) left = 0u;
        if (i == 2 && (next >> 16) < rank_crowd(LOGB)) d[2] = 0xFFFFu;  // no third crowd: two suffice
      }
      if (d[2] == 0xFFFFu)
        rank_apart(std::integral_constant<int, 2>{}, d);
      else
        rank_apart(std::integral_constant<int, 4>{}, d);
    }
  } else {
    // Lane l counts bucket l: its mask of lanes holding bucket l comes straight
    // from the ballots, and a key's peers and earlier count are read from the
    // lane that owns its bucket.
    uint32_t xm[LOGB];
#pragma unroll
    for (int i = 0; i < LOGB; ++i) xm[i] = ((lane >> i) & 1u) ? 0u : ~0u;
    uint32_t my_cnt = 0;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const uint32_t pos = wbase + uint32_t(j) * 32u + lane;
      const uint32_t b = bucket_at(pos);
      uint32_t m = FULL ? ~0u : __ballot_sync(~0u, pos < cnt);
#pragma unroll
      for (int i = 0; i < LOGB; ++i) m &= __ballot_sync(~0u, (b >> i) & 1u) ^ xm[i];
      const uint32_t peers = __shfl_sync(~0u, m, b);
      const uint32_t before = __shfl_sync(~0u, my_cnt, b);
      packed[j] = (b << 16) | (before + __popc(peers & lt));
      my_cnt += __popc(m);
    }
    if (lane < B) s_wh[warp * WB + lane] = WhT(my_cnt);
  }
  __syncthreads();

  // ---- 2. tile scan: per-warp offsets and bucket starts.  Thread b owns
  // bucket b; the bucket starts come from a block-wide exclusive scan (warp
  // scans + warp totals).
  uint32_t my_total = 0, my_start = 0;
  {
    // Key-value tiles keep the per-warp prefixes in registers across the block
    // scan and write each count-table entry once; key-only tiles, budgeted at
    // 40 registers, write the prefixes and add the start in a second pass.
    constexpr bool PREFIX_IN_REGS = C::KV;
    constexpr int SW = C::WARPS;  // count-table rows
    uint32_t pre[PREFIX_IN_REGS ? SW : 1];
    uint32_t total = 0;
    if (tid < B) {
#pragma unroll
      for (int w = 0; w < SW; ++w) {
        WhT* c_ptr = &s_wh[w * WB + tid];
        const uint32_t c = *c_ptr;
        if constexpr (PREFIX_IN_REGS)
          pre[w] = total;
        else
          *c_ptr = WhT(total);
        total += c;
      }
      offs.aggregate(tid, total);
      if constexpr (Offsets::KNOWN_EARLY) {
        if (uint64_t(offs.offset(tid, total)) + total > n) atomicOr(s_flag, 1u);
      }
    }
    uint32_t incl = total;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(~0u, incl, d);
      if (lane >= uint32_t(d)) incl += t;
    }
    constexpr uint32_t SCAN_WARPS = (B + 31) / 32;
    if (SCAN_WARPS > 1 && lane == 31 && warp < SCAN_WARPS) s_scan[warp] = incl;
    __syncthreads();
    if (tid < B) {
      uint32_t start = incl - total;
      if constexpr (SCAN_WARPS > 1) {
#pragma unroll
        for (uint32_t w = 0; w < SCAN_WARPS; ++w) start += (w < warp) ? s_scan[w] : 0u;
      }
      if constexpr (Offsets::KNOWN_EARLY) {
        s_delta[tid] = offs.offset(tid, total) - start;
      } else {
        my_total = total;
        my_start = start;
      }
#pragma unroll
      for (int w = 0; w < SW; ++w) {
        WhT* c_ptr = &s_wh[w * WB + tid];
        if constexpr (PREFIX_IN_REGS)
          *c_ptr = WhT(pre[w] + start);
        else
          *c_ptr = WhT(*c_ptr + start);
      }
    }
  }
  __syncthreads();
  if constexpr (Offsets::KNOWN_EARLY) {
    if (*s_flag != 0u) {  // block-uniform
      if (tid == 0) record_error(hdr, DEV_ERR_BAD_OFFSET);
      return false;
    }
  }

  // ---- 3. bucket-sorted in-tile order (positions are a permutation of [0, cnt))
  {
    const WhT* wh = s_wh + warp * WB;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
      const uint32_t pos = wbase + uint32_t(j) * 32u + lane;
      if (FULL || pos < cnt) {
        const uint32_t b = packed[j] >> 16;
        const uint32_t d = uint32_t(wh[b]) + (packed[j] & 0xFFFFu);
        if constexpr (L::WORDS)
          s_r[d] = (b << 16) | pos;
        else if constexpr (L::INDEXED)
          reinterpret_cast<uint16_t*>(s_r)[d] = uint16_t(pos);
        else
          s_r[d] = s_k[pos];
        if constexpr (L::BUCKET_BYTES && !L::WORDS) s_rb[d] = uint8_t(b);
      }
    }
  }
  // Offsets resolved only now: the buckets' global offsets, the per-bucket
  // shift delta = global offset - tile start, and a range check of every
  // bucket's output run against n (a corrupt offset can then never cause a
  // store outside the output).
  if constexpr (!Offsets::KNOWN_EARLY) {
    if constexpr (requires_resolve<Offsets>::value) offs.resolve(tid, my_total);
    if (tid < B) {
      const uint32_t g = offs.offset(tid, my_total);
      if (uint64_t(g) + my_total > n) atomicOr(s_flag, 1u);
      s_delta[tid] = g - my_start;
    }
  }
  __syncthreads();
  if constexpr (!Offsets::KNOWN_EARLY) {
    if (*s_flag != 0u) {  // block-uniform
      if (tid == 0) record_error(hdr, DEV_ERR_BAD_OFFSET);
      return false;
    }
  }

  // ---- 4. scatter in bucket-sorted order: each bucket's run is one coalesced store
  static_assert(!STREAM_HINTS || (C::KW == 1 && C::VW == 1), "store hints are for 32-bit elements");
  uint64_t policy = 0;
  if constexpr (STREAM_HINTS) policy = l2_evict_first_policy();
  // The key at in-tile position src goes to sorted position p of bucket b.
  auto store = [&](uint32_t p, uint32_t src, const KT& key, uint32_t b) {
    const uint32_t g = s_delta[b] + p;
    if constexpr (STREAM_HINTS) {
      st_global_hint(kout + g, key, policy);
      if constexpr (C::KV) st_global_hint(vout + g, s_v[src], policy);
    } else {
      kout[g] = key;
      if constexpr (C::KV) vout[g] = s_v[src];
    }
  };
  if constexpr (C::ATOMIC) {
    store_in_order<C, P, FULL, GIVEN>(cnt, ident, smem,
                                      [&](uint32_t p, uint32_t src, uint32_t b) { store(p, src, s_k[src], b); });
    return true;
  }
#pragma unroll
  for (int j = 0; j < IPT; ++j) {
    const uint32_t p = uint32_t(j) * C::THREADS + tid;
    if (FULL || p < cnt) {
      if constexpr (L::MODE == R_KEYS) {
        const uint32_t key = s_r[p];
        kout[s_delta[ident(key)] + p] = key;
      } else if constexpr (L::MODE == R_KEYS_B) {
        kout[s_delta[s_rb[p]] + p] = s_r[p];
      } else {
        const uint32_t src = reinterpret_cast<const uint16_t*>(s_r)[p];
        const KT key = s_k[src];
        uint32_t b;
        if constexpr (L::BUCKET_BYTES)
          b = s_rb[p];
        else
          b = ident(key);
        store(p, src, key, b);
      }
    }
  }
  return true;
}

// -------------------------------------------------------------- postscan
// One tile of one multisplit, as the postscan sees it.
template <class Params, class KT = uint32_t, class VT = uint32_t>
struct TileJob {
  const KT* kin;
  const VT* vin;
  KT* kout;
  VT* vout;
  uint32_t n;                // keys of this multisplit
  uint32_t num_tiles;        // its tiles
  uint32_t tile;             // this tile
  const uint32_t* offsets;   // its scanned count matrix, bucket-major
  uint32_t bias;             // subtracted from the scanned offsets (start of this multisplit in a shared scan)
  uint32_t prefetch_tile;    // a later tile of the same arrays to pull into L2 (>= num_tiles: none)
  Params bp;
  uint32_t owner;            // which multisplit of a batch (tiles with one owner share bp)
  const uint8_t* bucket_bytes;  // every key's bucket, from the prescan (GIVEN postscans only)
};

// Postscan of one tile, run by a whole block:
//  0. bulk-copy the tile's keys (and values) into shared memory, prefetch the
//     tile's B global offsets;
//  1. per warp, stable rank of every key among same-bucket keys earlier in the
//     warp's range (warp-striped slots keep input order: slot j, lane l is
//     key w*IPT*32 + j*32 + l);
//  2. tile scan: per-warp bucket offsets and the per-bucket shift
//     delta[b] = global_offset(b, tile) - tile_start(b);
//  3. write, at each key's bucket-sorted in-tile position, its key or source index;
//  4. walk the bucket-sorted order: out[delta[b] + p] = key (value), so every
//     bucket's run is a contiguous, coalesced store.
//
// PREPARE: fill the identifier's shared area first (false when the caller
// prepared it for several tiles).  Returns false when the block must stop (a
// bulk copy timed out or an offset was out of range; the error is recorded).
// With `*bar_live` the caller learns whether the tile's mbarrier was
// initialised (it must be invalidated before the next tile initialises it).
//
// GIVEN: the prescan stored every key's bucket as a byte (job.bucket_bytes);
// the tile's bytes are staged with its keys and the identifier is never
// evaluated (nor prepared).
//
// make_offsets(job, tid, B) gives thread tid the source of bucket tid's global
// offset (see GivenOffset); it is called while the tile's bulk copy is in flight.
//
// STREAM_HINTS: the tile's keys, values and bucket bytes are read, and its
// outputs written, as evict-first L2 lines (their last use).
template <class C, class P, bool PREPARE = true, bool GIVEN = false, class MakeOffsets = MatrixOffsets,
          bool STREAM_HINTS = false>
__device__ __forceinline__ bool postscan_job(const TileJob<typename P::Params, typename C::KT, typename C::VT>& job,
                                             ScratchHeader* hdr, unsigned char* smem, bool* bar_live = nullptr,
                                             MakeOffsets make_offsets = MakeOffsets()) {
  using L = PostLayout<C, P, GIVEN>;
  using KT = typename C::KT;
  using VT = typename C::VT;
  constexpr uint32_t B = C::B;
  constexpr uint32_t WB = C::WB;
  KT* s_k = reinterpret_cast<KT*>(smem + L::OFF_K);
  VT* s_v = reinterpret_cast<VT*>(smem + L::OFF_V);
  uint32_t* s_wh = reinterpret_cast<uint32_t*>(smem + L::OFF_WH);
  uint32_t* s_split = reinterpret_cast<uint32_t*>(smem + L::OFF_SPLIT);
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);

  const uint32_t tid = threadIdx.x;
  const uint32_t base = job.tile * C::TILE;
  const uint32_t cnt = min(C::TILE, job.n - base);
  const KT* kin = job.kin;
  const VT* vin = job.vin;

  // ---- 0. stage the tile
  uintptr_t addr_bits = reinterpret_cast<uintptr_t>(kin);
  if constexpr (C::KV) addr_bits |= reinterpret_cast<uintptr_t>(vin);
  // Elements moved by the bulk copy: a multiple of 4, so every array's part
  // is a whole number of 16-byte pieces.
  const uint32_t bulk = ((addr_bits & 15u) == 0) ? (cnt & ~3u) : 0u;
  if (tid == 0) *reinterpret_cast<uint32_t*>(smem + L::OFF_FLAG) = 0u;
  // Given bucket bytes: whole 16-byte pieces by the bulk copy, the rest below.
  const uint32_t bulk_b = (GIVEN && bulk != 0) ? (cnt & ~15u) : 0u;
  uint8_t* s_rb = reinterpret_cast<uint8_t*>(smem + L::OFF_RB);
  if (tid == 0 && bulk != 0) {
    mbar_init(s_bar, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(s_bar, bulk * uint32_t(sizeof(KT) + (C::KV ? sizeof(VT) : 0)) + bulk_b);
    if constexpr (STREAM_HINTS) {
      const uint64_t policy = l2_evict_first_policy();
      bulk_copy_g2s_hint(s_k, kin + base, bulk * uint32_t(sizeof(KT)), s_bar, policy);
      if constexpr (C::KV) bulk_copy_g2s_hint(s_v, vin + base, bulk * uint32_t(sizeof(VT)), s_bar, policy);
      if constexpr (GIVEN) {
        if (bulk_b != 0) bulk_copy_g2s_hint(s_rb, job.bucket_bytes + base, bulk_b, s_bar, policy);
      }
    } else {
      bulk_copy_g2s(s_k, kin + base, bulk * uint32_t(sizeof(KT)), s_bar);
      if constexpr (C::KV) bulk_copy_g2s(s_v, vin + base, bulk * uint32_t(sizeof(VT)), s_bar);
      if constexpr (GIVEN) {
        if (bulk_b != 0) bulk_copy_g2s(s_rb, job.bucket_bytes + base, bulk_b, s_bar);
      }
    }
    // Pull a tile that starts about one wave of blocks later into L2, so its
    // bulk copy does not wait on DRAM (only full tiles: never past the arrays).
    if (job.prefetch_tile < job.num_tiles - 1u) {
      bulk_prefetch_l2(kin + size_t(job.prefetch_tile) * C::TILE, C::TILE * uint32_t(sizeof(KT)));
      if constexpr (C::KV)
        bulk_prefetch_l2(vin + size_t(job.prefetch_tile) * C::TILE, C::TILE * uint32_t(sizeof(VT)));
    }
  }
  for (uint32_t i = bulk + tid; i < cnt; i += C::THREADS) {
    s_k[i] = kin[base + i];
    if constexpr (C::KV) s_v[i] = vin[base + i];
  }
  if constexpr (GIVEN) {
    // Through L2: in the batch queue other blocks of the same launch wrote them.
    for (uint32_t i = bulk_b + tid; i < cnt; i += C::THREADS) s_rb[i] = __ldcg(job.bucket_bytes + base + i);
  }
  if (bar_live) *bar_live = bulk != 0;
  auto offs = make_offsets(job, tid, B);
  if constexpr (PREPARE && !GIVEN) P::prepare(s_split, job.bp);
  if constexpr (C::ATOMIC) {
    for (uint32_t i = tid; i < C::WARPS * WB; i += C::THREADS) s_wh[i] = 0u;
  }
  __syncthreads();
  if (bulk != 0) {
    const bool ok = error_recorded(hdr) ? mbar_try_wait(s_bar, 0) : mbar_wait_bounded(s_bar, 0, hdr);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        record_error(hdr, DEV_ERR_BULK_COPY_TIMEOUT);
        mbar_wait_bounded(s_bar, 0, hdr);  // let a late copy land before the block moves on
      }
      return false;
    }
  }

  if (cnt == C::TILE)
    return postscan_tile<C, P, true, GIVEN, decltype(offs), STREAM_HINTS>(job.kout, job.vout, job.n, cnt, offs,
                                                                           job.bp, hdr, smem);
  return postscan_tile<C, P, false, GIVEN, decltype(offs), STREAM_HINTS>(job.kout, job.vout, job.n, cnt, offs,
                                                                          job.bp, hdr, smem);
}

// Persistent postscan over tiles first, first + stride, ... below last, for
// identifiers with a shared area (RANGE): the area is prepared again only when
// the tile's owner (multisplit of a batch) changes, and each tile pulls the
// block's next tile into L2.
template <class C, class P, class JobAt>
__device__ __forceinline__ void postscan_run(uint32_t first, uint32_t last, uint32_t stride, JobAt job_at,
                                             ScratchHeader* hdr, unsigned char* smem) {
  using L = PostLayout<C, P>;
  uint32_t* s_split = reinterpret_cast<uint32_t*>(smem + L::OFF_SPLIT);
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint32_t prepared_for = ~0u;  // owner whose parameters the shared area holds
  for (uint32_t t = first; t < last; t += stride) {
    const TileJob<typename P::Params, typename C::KT, typename C::VT> job =
        job_at(t, last - t > stride ? t + stride : ~0u);
    if (job.owner != prepared_for) {  // block-uniform: every thread reads the same job
      P::prepare(s_split, job.bp);
      prepared_for = job.owner;
    }
    bool bar_live = false;
    const bool ok = postscan_job<C, P, false>(job, hdr, smem, &bar_live);
    __syncthreads();  // shared buffers are reused by the next tile
    if (!ok) return;
    if (bar_live && threadIdx.x == 0) mbar_inval(s_bar);
  }
}

// The bucket starts (column 0 of the scanned matrix, row 0 of the rows), stored
// by the block of tile 0 where the caller wants them: pinned host memory (capi.cu).
__device__ __forceinline__ void store_starts(uint32_t* starts, const uint32_t* offsets, uint32_t stride,
                                             uint32_t num_buckets) {
  if (starts != nullptr && threadIdx.x < num_buckets) starts[threadIdx.x] = offsets[threadIdx.x * stride];
}

// Plain postscan: one block per tile of one multisplit.  GIVEN: the buckets
// come from bucket_bytes (written by the prescan).
template <class C, class P, bool GIVEN = false>
__global__ void __launch_bounds__(C::THREADS, (PostLayout<C, P, GIVEN>::MIN_BLOCKS)) postscan_kernel(
    const typename C::KT* __restrict__ kin, const typename C::VT* __restrict__ vin, typename C::KT* __restrict__ kout,
    typename C::VT* __restrict__ vout, uint32_t n, uint32_t num_tiles, const uint32_t* __restrict__ offsets,
    typename P::Params bp, ScratchHeader* hdr, uint32_t prefetch_dist, const uint8_t* __restrict__ bucket_bytes,
    uint32_t* starts, uint32_t rows_per, uint32_t* matrix) {
  extern __shared__ __align__(128) unsigned char smem[];
  griddep_wait();  // launched while the scan finishes: its offsets are complete past this point
  if constexpr (C::ROWS) {
    if (blockIdx.x >= num_tiles) {  // block-uniform
      static_assert(PostLayout<C, P, GIVEN>::BYTES >= MATRIX_TILES * (C::B + 1) * 4, "the tile's area holds the rows");
      rows_to_matrix<C::B>(offsets, matrix, num_tiles, rows_per, (blockIdx.x - num_tiles) * MATRIX_TILES,
                           reinterpret_cast<uint32_t*>(smem));
      return;
    }
  }
  if (blockIdx.x == 0) store_starts(starts, offsets, C::ROWS && rows_per != 0 ? 1u : num_tiles, C::B);
  const TileJob<typename P::Params, typename C::KT, typename C::VT> job{kin,        vin,     kout, vout,
                                        n,          num_tiles, blockIdx.x, offsets,
                                        0u,         prefetch_dist != 0 ? blockIdx.x + prefetch_dist : ~0u,
                                        bp,         0u,      bucket_bytes};
  if constexpr (C::ROWS)
    postscan_job<C, P, true, GIVEN, RowOffsets>(job, hdr, smem, nullptr, RowOffsets{rows_per});
  else
    postscan_job<C, P, true, GIVEN>(job, hdr, smem);
}

// Persistent plain postscan (identifiers with a shared area): block b runs
// tiles b, b + grid, ...  Blocks that run at the same time then work on
// neighbouring tiles, whose runs of one bucket are neighbours in the output,
// so partly written sectors merge in L2 before they reach DRAM.
template <class C, class P>
__global__ void __launch_bounds__(C::THREADS, (PostLayout<C, P>::MIN_BLOCKS)) postscan_persistent_kernel(
    const typename C::KT* __restrict__ kin, const typename C::VT* __restrict__ vin, typename C::KT* __restrict__ kout,
    typename C::VT* __restrict__ vout, uint32_t n, uint32_t num_tiles, const uint32_t* __restrict__ offsets,
    typename P::Params bp, ScratchHeader* hdr, uint32_t* starts) {
  extern __shared__ __align__(128) unsigned char smem[];
  griddep_wait();  // launched while the scan finishes: its offsets are complete past this point
  if (blockIdx.x == 0) store_starts(starts, offsets, num_tiles, C::B);
  postscan_run<C, P>(
      blockIdx.x, num_tiles, gridDim.x,
      [&](uint32_t t, uint32_t prefetch) {
        return TileJob<typename P::Params, typename C::KT, typename C::VT>{
            kin, vin, kout, vout, n, num_tiles, t, offsets, 0u, prefetch, bp, 0u};
      },
      hdr, smem);
}

}  // namespace gms
