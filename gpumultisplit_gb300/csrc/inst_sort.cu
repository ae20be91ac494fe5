// Sorts in one launch (fused.cuh): which tile and digit width such a sort takes.
#include "ms_dispatch.cuh"

namespace gms {

namespace {

// Small tiles shorten each warp's chain of ranks and spread a small input over
// more SMs; a single block, or one cluster of at most 16, meets without a trip
// through L2.  Measured for 8-bit digits (us per sort of keys, graph replays;
// three launches per pass / 16 / 8 / 4 keys per thread):
//    1 k  40.7 / 18.8 /  --  /  9.3      2 k  --- / 21.1 / 13.2 / 15.0
//   10 k  49.5 / 24.1 /  --  / 15.9     30 k 58.6 / 22.7 / 22.2 /  --
//   65 k  66.9 / 25.3 / 27.8           130 k 68.3 / 33.7 / 31.6
//  260 k  64.3 / 37.2 / 31.9           500 k 56.3 / 38.0 / 39.5
//  2.4 M 102.1 / 82.8
constexpr uint32_t SORT_ONE_BLOCK_4 = 1024;    // one block at 4 keys per thread
constexpr uint32_t SORT_ONE_BLOCK_8 = 2048;    // one block at 8
constexpr uint32_t SORT_CLUSTER_4 = 16384;     // one cluster at 4
constexpr uint32_t SORT_CLUSTER_8 = 32768;     // one cluster at 8
constexpr uint32_t SORT_CLUSTER_16 = 65536;    // one cluster at 16 (32-bit elements)
constexpr uint32_t SORT_GRID_8 = 400000;       // above: the full tile
constexpr uint32_t SORT_MAX = 2500000;         // tried up to here; 608 tiles of 4096 (2,490,368 keys) are resident on 152 SMs
// 64-bit elements with values: 1.8 M at 12 bytes 209 -> 179 us, 2.4 M 226 -> 230.
constexpr uint32_t SORT_MAX_WIDE_PAIRS = 2000000;

template <bool KV, int KW, int VW>
cudaError_t sort_keys(const FusedSortCall& c, bool* launched) {
  const bool wide = KW == 2 || VW == 2;
  if (wide && KV && c.n > SORT_MAX_WIDE_PAIRS) return cudaSuccess;
  if (c.n <= SORT_ONE_BLOCK_4 || (c.n > SORT_ONE_BLOCK_8 && c.n <= SORT_CLUSTER_4))
    return launch_fused_sort<8, KV, KW, VW, 4>(c, launched);
  if (c.n <= SORT_CLUSTER_8 || (c.n <= SORT_GRID_8 && (wide || c.n > SORT_CLUSTER_16)))
    return launch_fused_sort<8, KV, KW, VW, 8>(c, launched);
  return launch_fused_sort<8, KV, KW, VW, tile_ipt(KV, KW, VW)>(c, launched);
}

}  // namespace

size_t fused_sort_rows_bytes(uint32_t n) {
  if (n > SORT_MAX) return 0;
  const uint32_t tile = n <= SORT_CLUSTER_4 ? 1024u : n <= SORT_GRID_8 ? 2048u : 4096u;
  return size_t((n + tile - 1) / tile) * 1024u + 1024u;
}

cudaError_t run_fused_sort(const FusedSortCall& c, bool* launched) {
  *launched = false;
  if (c.n > SORT_MAX) return cudaSuccess;
  if (c.key_bytes == 4 && c.value_bytes == 0) return sort_keys<false, 1, 1>(c, launched);
  if (c.key_bytes == 4 && c.value_bytes == 4) return sort_keys<true, 1, 1>(c, launched);
  if (c.key_bytes == 8 && c.value_bytes == 0) return sort_keys<false, 2, 1>(c, launched);
  if (c.key_bytes == 8 && c.value_bytes == 4) return sort_keys<true, 2, 1>(c, launched);
  if (c.key_bytes == 8 && c.value_bytes == 8) return sort_keys<true, 2, 2>(c, launched);
  if (c.key_bytes == 4 && c.value_bytes == 8) return sort_keys<true, 1, 2>(c, launched);
  return cudaSuccess;
}

}  // namespace gms
