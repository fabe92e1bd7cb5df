// Host check of the blocks of fill-box voxels (qss_box.cuh): the index of voxel q of the
// fill box in loop order, through the block that holds it, against its coordinates, at the
// first and last voxels of the box, on both sides of 2^31 and 2^32 and at random.
// Usage: fill_block_check nx ny nz ghosts size; prints "<checked> <bad>".
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "qss_box.cuh"

int main(int, char** v) {
  const int nx = atoi(v[1]), ny = atoi(v[2]), nz = atoi(v[3]), g = atoi(v[4]), size = atoi(v[5]);
  const qss::Box b{nx + 2 * g, ny + 2 * g, nz + 2 * g, g, g + nx - 1, g, g + ny - 1, g, g + nz - 1};
  const int64_t n = (int64_t)nx * ny * nz;
  std::vector<int64_t> qs;
  for (int64_t at : {(int64_t)0, n, (int64_t)1 << 31, (int64_t)1 << 32, (int64_t)3 << 31})
    for (int64_t d = -3000; d < 3000; d++) qs.push_back(at + d);
  uint64_t r = 12345;
  for (int k = 0; k < 20000; k++) {
    r = r * 6364136223846793005ull + 1442695040888963407ull;
    qs.push_back((int64_t)((r >> 11) % (uint64_t)n));
  }
  long long checked = 0, bad = 0;
  for (int64_t q : qs) {
    if (q < 0 || q / size > (n + size - 1) / size) continue;
    const qss::FillBlock blk(b, q / size, size);
    const uint32_t t = (uint32_t)(q % size);
    checked++;
    if (blk.base + t != q || blk.n != n || blk.in(t) != (q < n)) bad++;
    else if (q < n && blk.at(b, t) != b.idx(g + (int)(q % nx), g + (int)(q / nx % ny), g + (int)(q / nx / ny))) bad++;
  }
  printf("%lld %lld\n", checked, bad);
  return bad != 0;
}
