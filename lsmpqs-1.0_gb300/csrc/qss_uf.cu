// qss_uf.cu -- 26-connected component labelling and trapped-phase masks on GB300.
//
// The reference labels {phi_bin == 1} with a serial union-find whose union
// rule always hangs the smaller root under the larger one
// (src/connectivity/connectivity.c:66-83), so every component ends up named
// by its LARGEST linear ghost-box index, and background is 0 (:201-214).
// That label is a property of the component, not of the visiting order, so a
// concurrent union-find that keeps the same rule (link the smaller root under
// the larger, by compare-and-swap on the root) produces identical labels:
//   1. per tile of 32 x 8 x 8 voxels, in shared memory: the nodes are the runs of
//      foreground voxels in the tile's 64 rows (one 32-bit mask each), named by
//      their last voxel; one thread per row and preceding row unites the runs
//      that touch; parent[v] = the global index of v's tile-local root (0 for
//      background);
//   2. across tiles, in global memory: a warp per row segment unites its runs
//      with those of preceding rows in other tiles, each touching pair once,
//      and its end voxels with the neighbouring segments;
//   3. labels[v] = root(v), 0 for background.
// Every write to parent[] increases it (hooking a root under a larger root,
// or compressing a node to a larger ancestor), so parent[x] > x holds for
// every non-root, the pointer graph has no cycle and every walk ends; the
// walks still carry an iteration cap and set an error flag instead of
// spinning if the cap is ever reached.
#include "qss_kernels.cuh"

namespace qss {

namespace {

// longest pointer walk tolerated before a device-side error is flagged
constexpr int kWalkCap = 1 << 22;

__device__ __forceinline__ int find_root(int* parent, int x, int* err) {
  int r = x;
  int it = 0;
  while (true) {
    int p = __ldcg(parent + r);  // L2-coherent read: other blocks hook roots concurrently
    if (p == r) break;
    r = p;
    if (++it > kWalkCap) {
      *err |= ERR_UF_LIMIT;
      return r;
    }
  }
  // Path compression.  Only nodes below r are rewritten, and only upwards:
  // another thread may already have moved a node of this path above r, and
  // lowering it again (or walking past r) could close a cycle.
  int y = x;
  it = 0;
  while (y < r && it++ < kWalkCap) {
    const int p = __ldcg(parent + y);
    if (p < r) __stcg(parent + y, r);
    y = p;
  }
  return r;
}

__device__ __forceinline__ void unite(int* parent, int a, int b, int* err) {
  int ra = find_root(parent, a, err);
  int rb = find_root(parent, b, err);
  int it = 0;
  while (ra != rb) {
    if (ra > rb) {
      int t = ra;
      ra = rb;
      rb = t;
    }
    const int old = atomicCAS(&parent[ra], ra, rb);  // hang the smaller root under the larger
    if (old == ra) return;
    ra = find_root(parent, old, err);
    rb = find_root(parent, rb, err);
    if (++it > kWalkCap) {
      *err |= ERR_UF_LIMIT;
      return;
    }
  }
}

// Tile of 32 x 8 x 8 voxels.  Rows r = lj + 8 lk, local index 32 r + li: the
// local order is the global linear order restricted to the tile, so hanging the
// smaller root under the larger makes a local root the component's last voxel.
constexpr int kTileY = 8, kTileZ = 8, kRows = kTileY * kTileZ;
constexpr int kTileN = 32 * kRows;
constexpr int kTileThreads = 4 * kRows;  // one per row and preceding row

// the four rows (dj, dk) that precede a row
__device__ __forceinline__ void back_row(int m, int& dj, int& dk) {
  dj = m == 3 ? 1 : (m == 2 ? 0 : -1);
  dk = m == 0 ? 0 : -1;
}

// last position of the run of ones in `mask` that holds position p
__device__ __forceinline__ int run_end(unsigned mask, int p) {
  const unsigned z = ~mask & (0xffffffffu << p);  // zeros from p on
  return z ? __ffs(z) - 2 : 31;
}

__device__ __forceinline__ int lfind(int* lp, int x, int* err) {
  int r = x;
  int it = 0;
  while (true) {
    const int p = lp[r];
    if (p == r) break;
    r = p;
    if (++it > kTileN) {
      *err |= ERR_UF_LIMIT;
      return r;
    }
  }
  int y = x;
  it = 0;
  while (y < r && it++ < kTileN) {  // compression upwards only (see find_root)
    const int p = lp[y];
    if (p < r) lp[y] = r;
    y = p;
  }
  return r;
}

__device__ __forceinline__ void lunite(int* lp, int a, int b, int* err) {
  int ra = lfind(lp, a, err), rb = lfind(lp, b, err);
  int it = 0;
  while (ra != rb) {
    if (ra > rb) {
      const int t = ra;
      ra = rb;
      rb = t;
    }
    const int old = atomicCAS(&lp[ra], ra, rb);
    if (old == ra) return;
    ra = lfind(lp, old, err);
    rb = lfind(lp, rb, err);
    if (++it > 4 * kTileN) {
      *err |= ERR_UF_LIMIT;
      return;
    }
  }
}

// tile-local labelling; writes parent[] for every voxel of the tile
// (background 0, foreground the global index of its local root)
__global__ void __launch_bounds__(kTileThreads) k_uf_tile(Box b, const unsigned char* __restrict__ bin, int* parent,
                                                          Ctl* ctl) {
  __shared__ int lp[kTileN];
  __shared__ unsigned mask[kRows];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * kTileY, z0 = blockIdx.z * kTileZ;
  int err = 0;
  for (int r = warp; r < kRows; r += kTileThreads / 32) {
    const int i = x0 + lane, j = y0 + r % kTileY, k = z0 + r / kTileY;
    const bool in = i < b.nx && j < b.ny && k < b.nz;
    const unsigned m = __ballot_sync(0xffffffffu, in && bin[b.idx(i, j, k)]);
    if (lane == 0) mask[r] = m;
    lp[32 * r + lane] = 32 * r + lane;
  }
  __syncthreads();
  {
    const int r = threadIdx.x % kRows;
    int dj, dk;
    back_row(threadIdx.x / kRows, dj, dk);
    const int lj = r % kTileY + dj, lk = r / kTileY + dk;
    if (lj >= 0 && lj < kTileY && lk >= 0) {
      const int r2 = lj + kTileY * lk;
      const unsigned B = mask[r2];
      for (unsigned A = mask[r]; A;) {
        const int p = __ffs(A) - 1, e = run_end(A, p);
        const unsigned from_p = 0xffffffffu << p, to_e = 0xffffffffu >> (31 - e);
        A &= ~to_e;
        // the runs of B within one position of [p, e]
        for (unsigned W = B & (from_p | (from_p >> 1)) & (to_e | (to_e << 1)); W;) {
          const int e2 = run_end(B, __ffs(W) - 1);
          lunite(lp, 32 * r + e, 32 * r2 + e2, &err);
          W &= ~(0xffffffffu >> (31 - e2));
        }
      }
    }
  }
  __syncthreads();
  for (int r = warp; r < kRows; r += kTileThreads / 32) {
    const int i = x0 + lane, j = y0 + r % kTileY, k = z0 + r / kTileY;
    if (i >= b.nx || j >= b.ny || k >= b.nz) continue;
    int g = 0;
    if (mask[r] >> lane & 1u) {
      const int root = lfind(lp, 32 * r + run_end(mask[r], lane), &err);
      const int rr = root / 32;
      g = (int)b.idx(x0 + root % 32, y0 + rr % kTileY, z0 + rr / kTileY);
    }
    parent[b.idx(i, j, k)] = g;
  }
  if (err && ctl) atomicOr(&ctl->err, err);
}

// The unions across tiles.  Given that voxels next to each other in a row are
// united (in a tile by the runs, across tiles by lane 0 here), a row's voxel x and
// the row before's voxels x-1, x, x+1 need one union where B[x] is set and the row
// has no voxel x-1 (which would touch B[x] itself), and where B[x] is not set one
// with B[x-1] under the same condition and one with B[x+1]: every pair of
// touching runs once.  Lanes of a warp that join the same two tile components
// agree on one of them (the parents are in the same sets as the voxels).
__device__ __forceinline__ void unite_lanes(int* parent, bool pair, int64_t q, int64_t q2, int* err) {
  if (!__any_sync(0xffffffffu, pair)) return;
  const unsigned lane = threadIdx.x & 31u;
  int ra = -1, rb = -1;
  if (pair) {
    ra = __ldcg(parent + q);
    rb = __ldcg(parent + q2);
    pair = ra != rb;
  }
  const unsigned lo = (unsigned)(ra < rb ? ra : rb), hi = (unsigned)(ra < rb ? rb : ra);
  const unsigned long long key = pair ? (((unsigned long long)lo << 32) | hi) : (0xffffffff00000000ull | lane);
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  if (pair && (unsigned)(__ffs(peers) - 1) == lane) unite(parent, ra, rb, err);
}

__global__ void __launch_bounds__(256) k_uf_cross(Box b, const unsigned char* __restrict__ bin, int* parent, Ctl* ctl) {
  const int lane = threadIdx.x & 31;
  const int x = blockIdx.x * 32 + lane, j = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (j >= b.ny) return;  // warp-uniform
  int err = 0;
  for (int k = blockIdx.z; k < b.nz; k += gridDim.z) {
    const int64_t q = b.idx(0, j, k) + x;
    const bool fg = x < b.nx && bin[q];
    const unsigned A = __ballot_sync(0xffffffffu, fg);
    if (!A) continue;
    const bool left_a = lane == 0 && x > 0 && bin[q - 1];
    const unsigned has_left = __ballot_sync(0xffffffffu, left_a) & 1u;  // A[x-1] of lane 0
    const bool prev = lane ? (A >> (lane - 1)) & 1u : has_left;
    unite_lanes(parent, fg && left_a, q, q - 1, &err);
    for (int m = 0; m < 4; m++) {
      int dj, dk;
      back_row(m, dj, dk);
      const int j2 = j + dj, k2 = k + dk;
      if (j2 < 0 || j2 >= b.ny || k2 < 0) continue;  // warp-uniform
      const bool same = j2 / kTileY == j / kTileY && k2 / kTileZ == k / kTileZ;
      const int64_t q2 = b.idx(0, j2, k2) + x;
      // within a tile only the end lanes look across; elsewhere every lane
      const bool look = fg && (!same || lane == 0 || lane == 31);
      const bool c1 = look && bin[q2];
      bool c0 = look && x > 0 && bin[q2 - 1], c2 = look && x + 1 < b.nx && bin[q2 + 1];
      if (same) {
        c0 = c0 && lane == 0;
        c2 = c2 && lane == 31;
      }
      unite_lanes(parent, look && !prev && ((c1 && !same) || (!c1 && c0)), q, c1 ? q2 : q2 - 1, &err);
      unite_lanes(parent, look && !c1 && c2, q, q2 + 1, &err);
    }
  }
  if (err && ctl) atomicOr(&ctl->err, err);
}

__global__ void k_uf_final(int64_t n, const unsigned char* __restrict__ bin, int* parent, Ctl* ctl) {
  int err = 0;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    if (bin[q]) {
      int r = (int)q;
      int it = 0;
      while (parent[r] != r && it++ < kWalkCap) r = parent[r];
      if (it > kWalkCap) err |= ERR_UF_LIMIT;
      parent[q] = r;
    }
  }
  if (err && ctl) atomicOr(&ctl->err, err);
}

// MERGE_SETS(phi, mask_nw) then phi_bin = phi < 0 (trapComponents.c:167-170)
__global__ void k_bin_nw(int64_t n, double* phi, const double* __restrict__ mask_nw, unsigned char* bin) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double m = mask_nw[q];
    double p = phi[q];
    if (m > 0) {
      p = -m;
      phi[q] = p;
    }
    bin[q] = (p < 0.0) ? 1 : 0;
  }
}

// inlet / outlet reservoirs of trapComponents.c:175-194 and 257-299
__global__ void k_set_bin_slab(Box b, unsigned char* bin, int center, int outlet) {
  const int64_t nxy = (int64_t)b.nx * b.ny;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (!outlet) {
    if (center) {
      const int k = (int)(0.5 * (b.klo + b.khi)), i = (int)(0.5 * (b.ilo + b.ihi));
      if (t < b.ny) bin[i + (int64_t)t * b.nx + k * nxy] = 1;
    } else {
      const int i = b.ilo - 1;
      const int64_t cnt = (int64_t)b.fby() * b.fbz();
      if (t < cnt) {
        const int j = b.jlo + t % b.fby(), k = b.klo + t / b.fby();
        bin[i + (int64_t)j * b.nx + k * nxy] = 1;
      }
    }
  } else {
    if (center) {
      if (t < nxy) {
        bin[(int64_t)(b.klo - 1) * nxy + t] = 1;
        bin[(int64_t)(b.khi + 1) * nxy + t] = 1;
      }
      if (t < (int64_t)b.ny * b.nz) {
        const int j = t % b.ny, k = t / b.ny;
        bin[(b.ilo - 1) + (int64_t)j * b.nx + k * nxy] = 1;
        bin[(b.ihi + 1) + (int64_t)j * b.nx + k * nxy] = 1;
      }
    } else {
      const int i = b.ihi + 1;
      const int64_t cnt = (int64_t)b.fby() * b.fbz();
      if (t < cnt) {
        const int j = b.jlo + t % b.fby(), k = b.klo + t / b.fby();
        bin[i + (int64_t)j * b.nx + k * nxy] = 1;
      }
    }
  }
}

// trapComponents.c:226-259: disconnected non-wetting mask, then the masked
// wetting phase in scratch and its binary image
__global__ void k_trap_nw(int64_t n, const int* __restrict__ labels, int main_idx, const double* __restrict__ phi,
                          const double* __restrict__ mask, double* mask_nw, double* scratch, unsigned char* bin,
                          double fill) {
  const int main_label = labels[main_idx];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int l = labels[q];
    const bool disc = !(l == main_label || l == 0);
    const double p = phi[q];
    const double mnw = (disc && p < 0) ? -p : fill;
    mask_nw[q] = mnw;
    double s = -p;
    const double m = mask[q];
    s = (m > s) ? m : s;
    s = (mnw > s) ? mnw : s;
    scratch[q] = s;
    bin[q] = (s < 0.0) ? 1 : 0;
  }
}

__global__ void k_trap_w(int64_t n, const int* __restrict__ labels, int main_idx, const double* __restrict__ scratch,
                         double* mask_w, double fill) {
  const int main_label = labels[main_idx];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int l = labels[q];
    const bool disc = !(l == main_label || l == 0);
    const double s = scratch[q];
    mask_w[q] = (disc && s < 0) ? -s : fill;
  }
}

unsigned grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 152 * 32) b = 152 * 32;
  return (unsigned)(b < 1 ? 1 : b);
}

}  // namespace

void launch_label(cudaStream_t s, const Box& b, const unsigned char* bin, int* labels, Ctl* ctl) {
  const int64_t n = b.npts();
  const unsigned seg = (unsigned)((b.nx + 31) / 32);
  const dim3 tiles(seg, (b.ny + kTileY - 1) / kTileY, (b.nz + kTileZ - 1) / kTileZ);
  k_uf_tile<<<tiles, kTileThreads, 0, s>>>(b, bin, labels, ctl);
  // a plane to a block; a block of a grid at its limit goes on to further planes
  k_uf_cross<<<dim3(seg, (b.ny + 7) / 8, b.nz < 65535 ? b.nz : 65535), 256, 0, s>>>(b, bin, labels, ctl);
  k_uf_final<<<grid_for(n), 256, 0, s>>>(n, bin, labels, ctl);
}

void launch_bin_nw(cudaStream_t s, int64_t n, double* phi, const double* mask_nw, unsigned char* bin) {
  k_bin_nw<<<grid_for(n), 256, 0, s>>>(n, phi, mask_nw, bin);
}

void launch_set_bin_slab(cudaStream_t s, const Box& b, unsigned char* bin, int center_inlet, int outlet) {
  int64_t cnt = (int64_t)b.nx * b.ny;
  if ((int64_t)b.ny * b.nz > cnt) cnt = (int64_t)b.ny * b.nz;
  if ((int64_t)b.fby() * b.fbz() > cnt) cnt = (int64_t)b.fby() * b.fbz();
  k_set_bin_slab<<<(unsigned)((cnt + 255) / 256), 256, 0, s>>>(b, bin, center_inlet, outlet);
}

void launch_trap_nw(cudaStream_t s, int64_t n, const int* labels, int main_idx, const double* phi,
                    const double* mask, double* mask_nw, double* scratch, unsigned char* bin, double fill) {
  k_trap_nw<<<grid_for(n), 256, 0, s>>>(n, labels, main_idx, phi, mask, mask_nw, scratch, bin, fill);
}

void launch_trap_w(cudaStream_t s, int64_t n, const int* labels, int main_idx, const double* scratch,
                   double* mask_w, double fill) {
  k_trap_w<<<grid_for(n), 256, 0, s>>>(n, labels, main_idx, scratch, mask_w, fill);
}

}  // namespace qss
