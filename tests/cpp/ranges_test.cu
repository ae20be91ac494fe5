// The prescan's ranges of tiles (prescan_tiles_per_block), on the host: they
// cover every tile, are at most a sixteenth longer than even ones, and whole
// groups wherever that bound allows it.  Prints "ok".
#include <cstdio>

#include "multisplit_kernels.cuh"

int main() {
  int bad = 0;
  for (uint32_t blocks : {1u, 2u, 152u, 608u, 760u, 1216u}) {
    for (uint32_t tiles = 1; tiles <= 70000; tiles += 1 + tiles / 64) {
      const uint32_t even = (tiles + blocks - 1) / blocks;
      const uint32_t any = gms::prescan_tiles_per_block(tiles, blocks, false);
      const uint32_t per = gms::prescan_tiles_per_block(tiles, blocks, true);
      const uint32_t up = (even + gms::PRESCAN_GROUP - 1) / gms::PRESCAN_GROUP * gms::PRESCAN_GROUP;
      bad += any != even;
      bad += per < even || (per - even) * 16 > even || uint64_t(per) * blocks < tiles;
      bad += per % gms::PRESCAN_GROUP != 0 && (up - even) * 16 <= even;
    }
  }
  std::printf(bad ? "%d wrong\n" : "ok\n", bad);
  return bad != 0;
}
