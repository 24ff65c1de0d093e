// Host-side check of the bound on the warp-row sweep's 32-bit byte offsets:
// the last byte of an array of 16-byte entries must have one.
#include <cstdio>
#include "mg_tiles.cuh"

int main() {
  int bad = 0;
  const int dims[][3] = {{4, 4, 4},        {514, 258, 258},   {1024, 512, 512}, {1024, 512, 513},
                         {645, 645, 645},  {646, 646, 646},   {2048, 1024, 1023}, {1290, 1290, 1290}};
  for (const auto& m : dims) {
    const vfs::Dims d{m[0], m[1], m[2], 0, 0, 0};
    const bool holds = 16ull * m[0] * m[1] * m[2] - 1 <= 0xffffffffull;
    if (vfs::fits_byte_offsets(d) != holds) {
      std::printf("wrong for %d x %d x %d\n", m[0], m[1], m[2]);
      bad++;
    }
  }
  return bad;
}
