// Phase 4 of the postscan on its own (store_in_order): it takes tiles whose
// buckets' runs are in any order and stores them in the input's.  Here the runs
// come with one exchange at a lane, slot or run boundary, reversed or shuffled,
// for keys and pairs, 32 to 256 buckets, every way a tile keeps its buckets, and
// full and partial tiles; each against the stable order.  Prints "ok".
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <type_traits>
#include <vector>

#include "ms_dispatch.cuh"

using namespace gms;

struct Tile {
  const void* keys;
  const void* vals;
  const uint32_t* order;    // source of each sorted position
  const uint32_t* buckets;  // bucket of each sorted position
  const uint32_t* starts;   // start of each bucket's run
  void* kout;
  void* vout;
  uint32_t* bout;
  uint32_t cnt;
};

template <class C, class P, bool FULL, bool GIVEN>
__global__ void __launch_bounds__(C::THREADS) store_kernel(Tile t, typename P::Params bp) {
  using L = PostLayout<C, P, GIVEN>;
  using KT = typename C::KT;
  using VT = typename C::VT;
  extern __shared__ __align__(128) unsigned char smem[];
  KT* s_k = reinterpret_cast<KT*>(smem + L::OFF_K);
  VT* s_v = reinterpret_cast<VT*>(smem + L::OFF_V);
  auto* s_wh = reinterpret_cast<typename L::WhT*>(smem + L::OFF_WH);
  for (uint32_t i = threadIdx.x; i < t.cnt; i += C::THREADS) {
    s_k[i] = static_cast<const KT*>(t.keys)[i];
    if constexpr (C::KV) s_v[i] = static_cast<const VT*>(t.vals)[i];
    const uint32_t src = t.order[i], b = t.buckets[i];
    if constexpr (L::WORDS) {
      reinterpret_cast<uint32_t*>(smem + L::OFF_R)[i] = (b << 16) | src;
    } else {
      reinterpret_cast<uint16_t*>(smem + L::OFF_R)[i] = uint16_t(src);
      if constexpr (L::BUCKET_BYTES) (smem + L::OFF_RB)[i] = uint8_t(b);
    }
  }
  for (uint32_t b = threadIdx.x; b < C::B; b += C::THREADS) s_wh[b] = t.starts[b];
  __syncthreads();
  const typename P::Id ident = P::make(bp, reinterpret_cast<const uint32_t*>(smem + L::OFF_SPLIT));
  store_in_order<C, P, FULL, GIVEN>(t.cnt, ident, smem, [&](uint32_t p, uint32_t src, uint32_t b) {
    static_cast<KT*>(t.kout)[p] = s_k[src];
    if constexpr (C::KV) static_cast<VT*>(t.vout)[p] = s_v[src];
    t.bout[p] = b;
  });
}

template <class T>
T* upload(const std::vector<T>& v) {
  T* d = nullptr;
  cudaMalloc(&d, std::max<size_t>(v.size(), 1) * sizeof(T));
  cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return d;
}

static uint32_t g_x = 1;
static uint32_t rnd() { return g_x = g_x * 1664525u + 1013904223u; }

template <class C, class P, bool FULL, bool GIVEN>
int one(const std::vector<typename C::KT>& keys, const std::vector<uint32_t>& bucket_of, int pattern) {
  using KT = typename C::KT;
  using VT = typename C::VT;
  const uint32_t cnt = uint32_t(keys.size());
  std::vector<uint32_t> stable(cnt);
  std::iota(stable.begin(), stable.end(), 0u);
  std::stable_sort(stable.begin(), stable.end(), [&](uint32_t a, uint32_t b) { return bucket_of[a] < bucket_of[b]; });
  std::vector<uint32_t> buckets(cnt), starts(C::B, 0), order = stable;
  for (uint32_t p = 0; p < cnt; ++p) buckets[p] = bucket_of[stable[p]];
  for (uint32_t b = 0; b < C::B; ++b)
    starts[b] = uint32_t(std::lower_bound(buckets.begin(), buckets.end(), b) - buckets.begin());
  bool moved = false;
  if (pattern > 0) {  // one exchange, at the first place from `pattern` on that is inside a run
    const uint32_t every = uint32_t(pattern);
    for (uint32_t p = every; p < cnt && !moved; p += every)
      if (buckets[p - 1] == buckets[p]) {
        std::swap(order[p - 1], order[p]);
        moved = true;
      }
  } else if (pattern == -1 || pattern == -2) {
    for (uint32_t b = 0; b < C::B; ++b) {
      const uint32_t lo = starts[b], hi = b + 1 < C::B ? starts[b + 1] : cnt;
      if (pattern == -1)
        std::reverse(order.begin() + lo, order.begin() + hi);
      else
        for (uint32_t p = hi; p > lo + 1; --p) std::swap(order[p - 1], order[lo + (rnd() >> 8) % (p - lo)]);
    }
  }
  std::vector<VT> vals(cnt);
  for (uint32_t i = 0; i < cnt; ++i) vals[i] = VT(i) * 7 + 1;
  Tile t{};
  KT* kout = upload(std::vector<KT>(cnt, 0));
  VT* vout = upload(std::vector<VT>(cnt, 0));
  uint32_t* bout = upload(std::vector<uint32_t>(cnt, ~0u));
  KT* dk = upload(keys);
  VT* dv = upload(vals);
  uint32_t *dord = upload(order), *dbuck = upload(buckets), *dst = upload(starts);
  t = Tile{dk, dv, dord, dbuck, dst, kout, vout, bout, cnt};
  typename P::Params bp{};
  if constexpr (std::is_same_v<typename P::Params, BucketParams>) bp.num_buckets = C::B;
  constexpr size_t smem = PostLayout<C, P, GIVEN>::BYTES;
  auto kern = store_kernel<C, P, FULL, GIVEN>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  kern<<<1, C::THREADS, smem>>>(t, bp);
  int bad = cudaDeviceSynchronize() != cudaSuccess;
  std::vector<KT> gk(cnt);
  std::vector<VT> gv(cnt);
  std::vector<uint32_t> gb(cnt);
  cudaMemcpy(gk.data(), kout, cnt * sizeof(KT), cudaMemcpyDeviceToHost);
  cudaMemcpy(gv.data(), vout, cnt * sizeof(VT), cudaMemcpyDeviceToHost);
  cudaMemcpy(gb.data(), bout, cnt * 4, cudaMemcpyDeviceToHost);
  for (uint32_t p = 0; p < cnt; ++p)
    bad += gk[p] != keys[stable[p]] || gb[p] != buckets[p] || (C::KV && gv[p] != vals[stable[p]]);
  for (void* d : {(void*)kout, (void*)vout, (void*)bout, (void*)dk, (void*)dv, (void*)dord, (void*)dbuck, (void*)dst})
    cudaFree(d);
  return bad;
}

template <template <int, int> class Policy, int KIND, int LOGB, bool KV, int KW, int VW, bool GIVEN>
int tiles(const char* name) {
  using S = TileShape<LOGB, KV, KW, VW>;
  using C = TileCfg<LOGB, S::WARPS, S::IPT, KV, KW, VW>;
  using P = Policy<KIND, LOGB>;
  using KT = typename C::KT;
  int bad = 0;
  for (uint32_t cnt : {C::TILE, C::TILE - 1, 700u, 33u, 1u}) {
    for (int skew : {0, 1}) {
      std::vector<KT> keys(cnt);
      std::vector<uint32_t> bucket_of(cnt);
      for (uint32_t i = 0; i < cnt; ++i) {
        uint32_t k = rnd() ^ (rnd() >> 16);
        if (skew && i % 4 != 0) k = (k >> 8) | 0x7F000000u;  // three of four keys in one bucket
        keys[i] = KT(k);
        bucket_of[i] = k >> (32 - LOGB);
      }
      for (int pattern : {0, 1, 3, 31, 32, 64, 127, 128, 129, 512, 1024, -1, -2}) {
        const int wrong = cnt == C::TILE ? one<C, P, true, GIVEN>(keys, bucket_of, pattern)
                                         : one<C, P, false, GIVEN>(keys, bucket_of, pattern);
        if (wrong != 0) std::printf("%s %d buckets, %u keys, pattern %d: %d wrong\n", name, 1 << LOGB, cnt, pattern, wrong);
        bad += wrong;
      }
    }
  }
  return bad;
}

template <int LOGB>
int widths() {
  return tiles<DescPolicy, KIND_DELTA, LOGB, false, 1, 1, false>("keys, evaluated again") +
         tiles<DescPolicy, KIND_DELTA, LOGB, true, 1, 1, false>("pairs, evaluated again") +
         tiles<DescPolicy, KIND_RANGE, LOGB, false, 1, 1, true>("keys, given") +
         tiles<DescPolicy, KIND_RANGE, LOGB, true, 1, 1, true>("pairs, given") +
         tiles<DescPolicy, KIND_RANGE, LOGB, true, 1, 1, false>("pairs, kept") +
         tiles<DescPolicy, KIND_DELTA, LOGB, true, 1, 2, false>("pairs with 64-bit values") +
         tiles<DescPolicy64, KIND_DELTA, LOGB, false, 2, 1, true>("64-bit keys") +
         tiles<DescPolicy64, KIND_DELTA, LOGB, true, 2, 2, true>("64-bit pairs");
}

int main() {
  const int bad = widths<5>() + widths<6>() + widths<7>() + widths<8>();
  std::printf(bad ? "%d wrong\n" : "ok\n", bad);
  return bad != 0;
}
