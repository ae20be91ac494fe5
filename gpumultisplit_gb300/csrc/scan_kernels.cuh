// Single-pass exclusive prefix sum with decoupled look-back, in place over a
// uint32 array (the bucket-count matrix), one block per chunk (scan_chunk.cuh).
// Replaces the reference's cub::DeviceScan::ExclusiveSum call
// (src/api/multisplit.cuh:141,258).
//
// Chunks are claimed through an atomic ticket, so a chunk only ever waits on
// chunks that were claimed (and are therefore running) before it.
#pragma once

#include "scan_chunk.cuh"

namespace gms {

// One chunk per block, claimed through the header's ticket counter.
__global__ void __launch_bounds__(SCAN_THREADS) scan_kernel(uint32_t* __restrict__ data, uint32_t m,
                                                            uint64_t* __restrict__ status, ScratchHeader* hdr) {
  __shared__ uint32_t s_chunk;
  griddep_wait();  // launched while the prescan finishes: the counts and the reset ticket are in place
  griddep_launch_dependents();
  if (threadIdx.x == 0) s_chunk = atomicAdd(&hdr->ticket, 1u);
  __syncthreads();
  const uint32_t chunk = s_chunk;
  // Tickets run from 0 when the prescan reset the counter; a block that draws
  // one past the last chunk (a counter not reset) has nothing to scan.
  if (chunk >= gridDim.x) return;
  scan_chunk(data, m, chunk, status, hdr);
}

// Scan of the prescan's range totals: row r * per of rows (num_buckets words
// each) holds range r's counts, and is replaced by the global offsets at which
// the range's buckets start, in bucket-major order of ranges.  A block scans
// SCAN_ROWS_COLS buckets over all ranges and takes the sum of the buckets before
// its own from the earlier blocks' status words (tickets, so those run).
constexpr int SCAN_ROWS_THREADS = 1024;
constexpr uint32_t SCAN_ROWS_COLS = 8;
constexpr uint32_t SCAN_ROWS_KEEP = 10;  // ranges a thread holds in registers

constexpr uint32_t SCAN_ROWS_GROUPS = SCAN_ROWS_THREADS / SCAN_ROWS_COLS;  // threads per column
constexpr uint32_t SCAN_ROWS_MAX_RANGES = SCAN_ROWS_KEEP * SCAN_ROWS_GROUPS;
static_assert((1u << ROWS_MIN_LOGB) % SCAN_ROWS_COLS == 0, "whole blocks of buckets");
// The prescan resets a status word per SCAN_CHUNK counts; every block here uses one.
static_assert(ROWS_MIN_TILES * SCAN_ROWS_COLS >= SCAN_CHUNK, "a reset status word for every block");

__global__ void __launch_bounds__(SCAN_ROWS_THREADS) scan_rows_kernel(uint32_t* __restrict__ rows, uint32_t num_buckets,
                                                                      uint32_t ranges, uint32_t per,
                                                                      uint64_t* __restrict__ status,
                                                                      ScratchHeader* hdr) {
  __shared__ uint32_t s_sum[SCAN_ROWS_THREADS];  // [column][thread of the column]
  __shared__ uint32_t s_start[SCAN_ROWS_COLS];
  __shared__ uint32_t s_blk;
  griddep_wait();  // launched while the prescan finishes: the rows and the reset ticket are in place
  griddep_launch_dependents();
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) s_blk = atomicAdd(&hdr->ticket, 1u);
  __syncthreads();
  const uint32_t blk = s_blk;
  if (blk >= gridDim.x) return;
  constexpr uint32_t cols = SCAN_ROWS_COLS, groups = SCAN_ROWS_GROUPS;
  static_assert(groups % 32 == 0, "a warp scans whole slots of a column's threads");
  const uint32_t c = tid % cols, r = tid / cols;
  const uint32_t each = (ranges + groups - 1) / groups;
  const size_t stride = size_t(per) * num_buckets;
  uint32_t* p = rows + blk * cols + c;
  uint32_t v[SCAN_ROWS_KEEP], sum = 0;
#pragma unroll
  for (uint32_t k = 0; k < SCAN_ROWS_KEEP; ++k) {
    const uint32_t i = r * each + k;
    v[k] = k < each && i < ranges ? __ldcg(p + i * stride) : 0u;
  }
#pragma unroll
  for (uint32_t k = 0; k < SCAN_ROWS_KEEP; ++k) sum += v[k];
  s_sum[c * groups + r] = sum;
  __syncthreads();
  if (warp < cols) {  // warp w: exclusive scan of column w's partial sums
    uint32_t carry = 0;
    for (uint32_t g = 0; g < groups; g += 32) {
      const uint32_t x = s_sum[warp * groups + g + lane];
      uint32_t incl = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(~0u, incl, d);
        if (lane >= uint32_t(d)) incl += t;
      }
      s_sum[warp * groups + g + lane] = carry + incl - x;
      carry += __shfl_sync(~0u, incl, 31);
    }
    if (lane == 0) s_start[warp] = carry;  // the column's total, for now
  }
  __syncthreads();
  if (warp == 0) {
    const uint32_t total = lane < cols ? s_start[lane] : 0u;
    const uint32_t block_total = warp_sum(total);
    if (lane == 0) st_relaxed_u64(&status[blk], (uint64_t(SCAN_FLAG_AGGREGATE) << 32) | block_total);
    uint32_t before = 0;
    for (uint32_t first = 0; first < blk; first += 32) {
      const uint32_t i = first + lane;
      uint64_t w = 0;
      const uint64_t t0 = global_timer_ns();
      const uint64_t limit = error_recorded(hdr) ? 0ull : wait_limit_ns(hdr);
      while (true) {
        w = i < blk ? ld_relaxed_u64(&status[i]) : (uint64_t(SCAN_FLAG_AGGREGATE) << 32);
        if (!__any_sync(~0u, (w >> 32) == 0u)) break;
        const bool late = lane == 0 && global_timer_ns() - t0 > limit;
        if (__shfl_sync(~0u, late ? 1u : 0u, 0)) {
          if (lane == 0) record_error(hdr, DEV_ERR_LOOKBACK_TIMEOUT);
          break;
        }
        __nanosleep(32);
      }
      before += warp_sum(uint32_t(w));
    }
    uint32_t incl = total;
#pragma unroll
    for (int d = 1; d < int(SCAN_ROWS_COLS); d <<= 1) {
      const uint32_t t = __shfl_up_sync(~0u, incl, d);
      if (lane >= uint32_t(d)) incl += t;
    }
    __syncwarp();
    if (lane < cols) s_start[lane] = before + incl - total;
  }
  __syncthreads();
  uint32_t run = s_start[c] + s_sum[c * groups + r];
#pragma unroll
  for (uint32_t k = 0; k < SCAN_ROWS_KEEP; ++k) {
    const uint32_t i = r * each + k;
    if (k < each && i < ranges) p[i * stride] = run;
    run += v[k];
  }
}

}  // namespace gms
