// The repair of a tile whose ranks came back out of the input's order
// (sort_run), on the host: runs of every small length in every order, long runs
// with a few and with many inversions, against std::sort.  Prints "ok".
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <numeric>
#include <vector>

#include "multisplit_kernels.cuh"

static bool check(std::vector<uint16_t> v) {
  std::vector<uint16_t> want = v;
  std::sort(want.begin(), want.end());
  v.push_back(0xBEEF);  // past the run: must stay
  gms::sort_run(v.data(), uint32_t(want.size()));
  return v.back() == 0xBEEF && std::equal(want.begin(), want.end(), v.begin());
}

int main() {
  int bad = 0;
  for (int n = 0; n <= 7; ++n) {
    std::vector<uint16_t> v(n);
    std::iota(v.begin(), v.end(), uint16_t(4000));
    do {
      bad += !check(v);
    } while (std::next_permutation(v.begin(), v.end()));
  }
  uint32_t seed = 1;
  auto rnd = [&] { return seed = seed * 1664525u + 1013904223u; };
  for (int n : {31, 32, 512, 4096}) {
    for (int swaps : {0, 1, 16, n}) {
      std::vector<uint16_t> v(n);
      std::iota(v.begin(), v.end(), uint16_t(0));
      for (int s = 0; s < swaps; ++s) std::swap(v[rnd() % n], v[rnd() % n]);
      bad += !check(v);
    }
    std::vector<uint16_t> down(n);
    std::iota(down.rbegin(), down.rend(), uint16_t(0));
    bad += !check(down);
  }
  std::printf(bad ? "%d wrong\n" : "ok\n", bad);
  return bad != 0;
}
