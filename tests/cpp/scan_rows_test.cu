// The scan of the range totals (scan_rows_kernel) on its own: its result for 1
// range up to the most that one launch takes, and its bounded wait: with the
// ticket counter at 1 no block scans the first columns, so the others wait for a
// status word that nothing writes, give up after 2 ms and report it.  Prints "ok".
#include <cstdio>
#include <vector>

#include "scan_kernels.cuh"

using namespace gms;

int main() {
  int bad = 0;
  for (uint32_t B : {128u, 256u}) {
    for (uint32_t ranges : {1u, 31u, 128u, 129u, 760u, SCAN_ROWS_MAX_RANGES}) {
      for (uint32_t per : {1u, 3u}) {
        const uint32_t rows = ranges * per, blocks = B / SCAN_ROWS_COLS;
        std::vector<uint32_t> h(size_t(rows) * B), want;
        uint32_t x = 12345;
        for (auto& v : h) v = (x = x * 1664525u + 1013904223u) >> 20;
        want = h;
        uint32_t run = 0;
        for (uint32_t b = 0; b < B; ++b)
          for (uint32_t r = 0; r < ranges; ++r) {
            want[size_t(r) * per * B + b] = run;
            run += h[size_t(r) * per * B + b];
          }
        uint32_t* d;
        uint64_t* status;
        ScratchHeader* hdr;
        cudaMalloc(&d, h.size() * 4);
        cudaMalloc(&status, blocks * 8);
        cudaMalloc(&hdr, sizeof(ScratchHeader));
        for (bool stuck : {false, true}) {
          ScratchHeader start = {};
          start.ticket = stuck ? 1u : 0u;
          start.wait_limit_us = 2000;
          cudaMemcpy(d, h.data(), h.size() * 4, cudaMemcpyHostToDevice);
          cudaMemset(status, 0, blocks * 8);
          cudaMemcpy(hdr, &start, sizeof(start), cudaMemcpyHostToDevice);
          scan_rows_kernel<<<blocks, SCAN_ROWS_THREADS>>>(d, B, ranges, per, status, hdr);
          if (cudaDeviceSynchronize() != cudaSuccess) {
            std::printf("%s\n", cudaGetErrorString(cudaGetLastError()));
            return 1;
          }
          ScratchHeader end;
          cudaMemcpy(&end, hdr, sizeof(end), cudaMemcpyDeviceToHost);
          bad += end.error != (stuck ? uint32_t(DEV_ERR_LOOKBACK_TIMEOUT) : 0u);
          if (!stuck) {
            std::vector<uint32_t> got(h.size());
            cudaMemcpy(got.data(), d, got.size() * 4, cudaMemcpyDeviceToHost);
            if (got != want) {
              std::printf("B=%u ranges=%u per=%u: wrong\n", B, ranges, per);
              ++bad;
            }
          }
        }
        cudaFree(d);
        cudaFree(status);
        cudaFree(hdr);
      }
    }
  }
  std::printf(bad ? "%d wrong\n" : "ok\n", bad);
  return bad != 0;
}
