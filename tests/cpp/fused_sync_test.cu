// How the blocks of one launch meet (fused_sync_of), and which launch errors
// hand the call to the stages, on the host.  Prints "ok".
#include <cstdio>

#include "fused.cuh"

int main() {
  int bad = 0;
  for (uint32_t tiles = 1; tiles <= gms::FUSED_MAX_TILES; ++tiles) {
    for (bool placed : {false, true}) {
      for (bool rows : {false, true}) {
        const uint32_t got = gms::fused_sync_of(tiles, placed, rows);
        uint32_t want = rows ? gms::FUSED_GRID : gms::FUSED_NONE;
        if (tiles <= 16 && placed) want = gms::FUSED_CLUSTER;
        if (tiles == 1) want = gms::FUSED_ONE_TILE;
        bad += got != want;
      }
    }
  }
  for (cudaError_t e : {cudaErrorCooperativeLaunchTooLarge, cudaErrorInvalidClusterSize, cudaErrorLaunchOutOfResources})
    bad += !gms::fused_declined(e);
  for (cudaError_t e : {cudaSuccess, cudaErrorInvalidValue, cudaErrorIllegalAddress, cudaErrorStreamCaptureInvalidated})
    bad += gms::fused_declined(e);
  std::printf(bad ? "%d wrong\n" : "ok\n", bad);
  return bad != 0;
}
