// A user functor is evaluated on the input's keys only.  The functor here has a
// limited domain, as one that looks its key up in a table has; it counts every
// key at or above the limit (and reads nothing).  Calls on large keys first
// leave shared memory full of them.  Prints "ok".
#include <stdint.h>
#include <stdio.h>

#include <vector>

#include "api/multisplit.cuh"

struct domain_bucket {
  uint32_t limit;     // keys in use are below it; 0: all keys
  uint32_t* outside;  // device counter
  __host__ __device__ static uint32_t id(uint32_t a) { return (a * 2654435761u) >> 24; }
  __device__ uint32_t operator()(uint32_t a) const {
    if (limit != 0 && a >= limit) atomicAdd(outside, 1u);
    return id(a);
  }
};

static const uint32_t LIMIT = 1u << 20, MOST = 700u * 4096u + 1u, TILE = 4096u;

int main() {
  uint32_t *k, *v, *ko, *vo, *outside, *large;
  std::vector<uint32_t> hk(MOST), hv(MOST), hl(MOST);
  for (uint32_t i = 0; i < MOST; ++i) {
    hk[i] = (i * 2246822519u + 374761393u) >> 12;  // below LIMIT
    hv[i] = i;
    hl[i] = hk[i] | 0xFFF00000u;
  }
  for (uint32_t** p : {&k, &v, &ko, &vo, &large}) cudaMalloc(p, MOST * 4);
  cudaMalloc(&outside, 4);
  cudaMemset(outside, 0, 4);
  cudaMemcpy(k, hk.data(), MOST * 4, cudaMemcpyHostToDevice);
  cudaMemcpy(v, hv.data(), MOST * 4, cudaMemcpyHostToDevice);
  cudaMemcpy(large, hl.data(), MOST * 4, cudaMemcpyHostToDevice);
  int bad = 0;
  for (uint32_t B : {2u, 8u, 32u, 256u}) {
    for (bool pairs : {false, true}) {
      multisplit_context ctx(B);
      (pairs ? multisplit_allocate_key_value : multisplit_allocate_key_only)(MOST, ctx);
      const size_t most_bytes = ctx.temp_storage_bytes;
      auto run = [&](uint32_t* keys, uint32_t n, uint32_t limit) {
        const domain_bucket f{limit, outside};
        if (pairs)
          multisplit_key_value(keys, v, ko, vo, n, ctx, f);
        else
          multisplit_key_only(keys, ko, n, ctx, f);
        return multisplit_last_error();
      };
      // One tile, clusters without and with an empty block, a grid, three stages; each with the reported
      // scratch and with the smallest that is taken (no byte per key).
      for (uint32_t n : {1u, 33u, TILE + 1, 2 * TILE + 1, 20 * TILE + 1, MOST}) {
        for (bool small : {false, true}) {
          ctx.temp_storage_bytes = most_bytes;
          bad += run(large, 600 * TILE, 0) != GMS_SUCCESS;
          if (small) {
            size_t full = 0;
            gms_multisplit_scratch_bytes(n, B, pairs, &full);
            ctx.temp_storage_bytes = full - (size_t(n) + 255) / 256 * 256;
            if (B > 64 && n > 512 * TILE) ctx.temp_storage_bytes -= size_t(B) * ((n + TILE - 1) / TILE) * 4 / 256 * 256;
          }
          cudaMemset(ko, 0x5A, MOST * 4);
          cudaMemset(vo, 0x5A, MOST * 4);
          cudaMemset(outside, 0, 4);
          bad += run(k, n, LIMIT) != GMS_SUCCESS;
          uint32_t seen = 0;
          cudaMemcpy(&seen, outside, 4, cudaMemcpyDeviceToHost);
          if (seen != 0) {
            printf("B=%u pairs=%d n=%u small=%d: evaluated on %u keys that are not the input's\n", B, pairs, n, small, seen);
            ++bad;
          }
          std::vector<uint32_t> pos(B + 1, 0), gk(n), gv(n), wk(n), wv(n);
          for (uint32_t i = 0; i < n; ++i) ++pos[(domain_bucket::id(hk[i]) & (B - 1)) + 1];
          for (uint32_t b = 0; b < B; ++b) pos[b + 1] += pos[b];
          for (uint32_t i = 0; i < n; ++i) {
            const uint32_t p = pos[domain_bucket::id(hk[i]) & (B - 1)]++;
            wk[p] = hk[i];
            wv[p] = i;
          }
          cudaMemcpy(gk.data(), ko, n * 4, cudaMemcpyDeviceToHost);
          if (pairs) cudaMemcpy(gv.data(), vo, n * 4, cudaMemcpyDeviceToHost);
          if (gk != wk || (pairs && gv != wv)) {
            printf("B=%u pairs=%d n=%u small=%d: wrong output\n", B, pairs, n, small);
            ++bad;
          }
        }
      }
      ctx.temp_storage_bytes = most_bytes;
      multisplit_release_memory(ctx);
    }
  }
  if (cudaDeviceSynchronize() != cudaSuccess) ++bad;
  printf(bad ? "%d wrong\n" : "ok\n", bad);
  return bad != 0;
}
