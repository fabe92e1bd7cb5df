// qss_box.cuh -- index spaces.  The header compiles for the host too (g++), where the
// index arithmetic of boxes too large to run is tested.
#pragma once
#include <cstdint>
#ifdef __CUDACC__
#define QSS_HD __host__ __device__
#else
#define QSS_HD
#endif

namespace qss {

// Index space of one volume: ghost box [0,nx)x[0,ny)x[0,nz), fill box
// [ilo,ihi]x[jlo,jhi]x[klo,khi], column-major with i fastest.
struct Box {
  int nx, ny, nz;
  int ilo, ihi, jlo, jhi, klo, khi;
  QSS_HD int64_t sx() const { return 1; }
  QSS_HD int64_t sy() const { return nx; }
  QSS_HD int64_t sz() const { return (int64_t)nx * ny; }
  QSS_HD int64_t idx(int i, int j, int k) const {
    return (int64_t)i + (int64_t)nx * ((int64_t)j + (int64_t)ny * k);
  }
  QSS_HD int64_t npts() const { return (int64_t)nx * ny * nz; }
  QSS_HD int fbx() const { return ihi - ilo + 1; }
  QSS_HD int fby() const { return jhi - jlo + 1; }
  QSS_HD int fbz() const { return khi - klo + 1; }
};

// `size` consecutive voxels of the fill box in loop order (i fastest), the block-th of
// such runs: 64-bit where the run starts (a box taken by a single-kernel entry point may
// hold more than 2^32 voxels), 32-bit offsets inside it.
struct FillBlock {
  int64_t base, n;  // the run's first voxel; voxels of the fill box
  uint32_t fbx, fby, i0, j0, k0;
  QSS_HD FillBlock(const Box& b, int64_t block, int size) {
    base = block * size;
    n = (int64_t)b.fbx() * b.fby() * b.fbz();
    fbx = (uint32_t)b.fbx();
    fby = (uint32_t)b.fby();
    const uint64_t row0 = (uint64_t)base / fbx;
    k0 = (uint32_t)(row0 / fby);
    i0 = (uint32_t)((uint64_t)base - row0 * fbx);
    j0 = (uint32_t)(row0 - (uint64_t)k0 * fby);
  }
  QSS_HD bool in(uint32_t t) const { return base + t < n; }
  // ghost-box index of the run's voxel t
  QSS_HD int64_t at(const Box& b, uint32_t t) const {
    const uint32_t x = i0 + t, r = x / fbx, y = j0 + r, q = y / fby;
    return b.idx(b.ilo + (int)(x - r * fbx), b.jlo + (int)(y - q * fby), b.klo + (int)(k0 + q));
  }
};

}  // namespace qss
