// qss_volsum.cu -- the reference's loop-order volume sum, in parallel and
// bit-identical.
//
// qss3dVolumeRegionPhiLessThanZero (qss_util3d.f:288-358) adds one
// contribution per fill-box voxel to a running double in loop order.
// Floating-point addition is not associative, so the result is the
// sequentially rounded sum, not the exact one; a dependent chain of FP64
// additions on GB300 costs ~85 ns per voxel.
//
// The contributions (1 - H(phi)) dV are non-negative, so the running sum s
// never decreases.  While s stays inside one binade [2^E, 2^(E+1)), every
// representable value there is a multiple of u = 2^(E-52), and
//     RN(s + c) = s + u * rne(c / u)
// where rne rounds to the nearest integer -- unless c / u is exactly halfway
// between two integers (then the tie goes to the even significand, which
// depends on s).  So for a chunk of contributions and a known binade, the
// chunk's effect on s is one integer R = sum of rne(c / u), computable in
// parallel and exactly (int64), valid when no element is a tie or not a
// finite non-negative number and s / u + R stays below 2^53 - 1.
//
//   1. k_vol_contrib (volumes; the contributions are computed here) or
//      k_vol_chunk_sum (a given sequence): per chunk of 4096 contributions,
//      their sum -- only to estimate where the running sum stands;
//   2. k_vol_scan (more than 4096 chunks only; else each block of 3 sums its
//      predecessors): exclusive scan of those sums -> an estimate of s at the
//      start of each chunk, good to far better than a factor of 2;
//   3. k_vol_chunk_r: per chunk, R and a "not applicable" flag for the
//      estimated binade and its two neighbours;
//   4. k_vol_walk: one block walks the chunks in order with the exact running
//      sum, 256 chunks at a time: a scan of their R finds the first chunk that
//      does not apply (another binade, the top of the binade reached, a tie,
//      special values); the sum advances to it in one integer addition, and
//      that chunk goes the same way by groups of 16 elements, only the group
//      that does not apply being added element by element.
// Every result equals the sequential loop's bit for bit.  With one warp that
// walked chunk by chunk and added a whole chunk element by element, a volume
// took 0.42 ms at 24^3, 3.5 ms at 192^3 and 8.6 ms at 320^3 on GB300.
#include "qss_emu.cuh"
#include "qss_state.h"

namespace qss {

namespace {

constexpr int kVolChunk = 4096;
constexpr int kVolThreads = 256;
constexpr int kVolPer = kVolChunk / kVolThreads;  // elements per thread in the walk
constexpr int kScanChunks = 4096;                 // from here on the estimates are scanned by a kernel
constexpr int kSmallChunks = 4;                   // up to here the walk goes by elements alone

__device__ __forceinline__ uint64_t dbits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double dfrom(uint64_t b) { return __longlong_as_double((long long)b); }

// unbiased exponent of a positive normal double, or a sentinel
__device__ __forceinline__ int exp_of(double x) {
  const uint64_t b = dbits(x);
  const int e = (int)((b >> 52) & 0x7ff);
  if ((b >> 63) || e == 0 || e == 0x7ff) return -100000;
  return e - 1023;
}

// rne(c / u) for u = 2^(E - 52) (below 2^52 + 1, so 4096 of them fit in
// 64 bits); bad = a tie, a negative or non-finite c, or c >= 2^E
__device__ __forceinline__ uint64_t rne_units(double c, int E, bool& bad) {
  const uint64_t b = dbits(c);
  if ((b << 1) == 0) return 0;  // +-0 leaves s unchanged
  const int ec = (int)((b >> 52) & 0x7ff);
  if ((b >> 63) || ec == 0x7ff) {
    bad = true;
    return 0;
  }
  uint64_t m = b & ((1ull << 52) - 1);
  int ce;  // c = m 2^ce
  if (ec == 0) {
    ce = -1074;
  } else {
    m |= 1ull << 52;
    ce = ec - 1075;
  }
  const int sh = (E - 52) - ce;  // c / u = m / 2^sh
  if (sh <= 0) {  // c >= 2^E: s leaves the binade within this chunk
    bad = true;
    return 0;
  }
  if (sh >= 64) return 0;  // m < 2^53 <= 2^(sh-11): far below half a unit
  const uint64_t q = m >> sh, rem = m & ((1ull << sh) - 1), half = 1ull << (sh - 1);
  if (rem == half) bad = true;
  return q + (rem > half ? 1u : 0u);
}

__global__ void __launch_bounds__(kVolThreads) k_vol_chunk_sum(const double* __restrict__ c, int64_t n,
                                                               double* csum) {
  __shared__ double red[kVolThreads];
  const int64_t base = (int64_t)blockIdx.x * kVolChunk;
  double s = 0;
  for (int t = threadIdx.x; t < kVolChunk; t += kVolThreads) {
    const int64_t q = base + t;
    if (q < n) s += c[q];
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = kVolThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) csum[blockIdx.x] = red[0];
}

// contribution of each fill-box voxel in loop order (i fastest), and the sum of
// each quarter chunk.  A voxel outside the smoothing band costs an
// integer comparison; those inside (about 15 % of the voxels, but a lane or more
// of most warps) are first gathered, then evaluated by full warps: their division
// and sine are ~45 FP64 instructions and the kernel's bound.  Blocks of 1024
// voxels, so that small boxes use more SMs (24^3 49 us with whole chunks).
constexpr int kContribVoxels = 1024, kContribThreads = 256;

__global__ void __launch_bounds__(kContribThreads) k_vol_contrib(Box b, const double* __restrict__ phi, double dV,
                                                                 double eps, double* contrib, float* csum) {
  __shared__ double band_p[kContribVoxels];
  __shared__ uint32_t band_q[kContribVoxels];
  __shared__ int band_n;
  __shared__ float red[kContribThreads / 32];
  const double pi = 3.14159265358979323846;
  const double one_over_pi = 0.31830988618379;
  const uint32_t n = (uint32_t)b.fbx() * b.fby() * b.fbz();  // below 2^31
  const uint32_t base = blockIdx.x * (uint32_t)kContribVoxels;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) band_n = 0;
  __syncthreads();
  // a value as a float by its bits (a conversion is an FP64 instruction); values
  // outside the float range do not matter for the estimate
  auto approx = [](double v) {
    const uint32_t h = qss_emu::hi32(v);
    return h - 0x38100000u < 0x0fe00000u ? __uint_as_float((h - 0x38000000u) << 3) : 0.0f;
  };
  float sum = 0.0f;
#pragma unroll
  for (int t = 0; t < kContribVoxels; t += kContribThreads) {
    const uint32_t q = base + t + threadIdx.x;
    bool band = false;
    double p = 0.0;
    if (q < n) {
      const uint32_t r = q / (uint32_t)b.fbx();
      const int i = b.ilo + (int)(q - r * (uint32_t)b.fbx());
      const int k = b.klo + (int)(r / (uint32_t)b.fby());
      const int j = b.jlo + (int)(r - (uint32_t)(k - b.klo) * (uint32_t)b.fby());
      p = phi[b.idx(i, j, k)];
      const bool inside = qss_emu::gt(-eps, p);  // p < -eps
      band = !inside && qss_emu::gt(eps, p);     // p < eps
      if (!band) contrib[q] = inside ? dV : 0.0;
      if (inside) sum += approx(dV);
    }
    const unsigned m = __ballot_sync(0xffffffffu, band);
    int at = 0;
    if (lane == 0 && m) at = atomicAdd(&band_n, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (band) {
      band_p[at] = p;
      band_q[at] = q;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < band_n; t += kContribThreads) {
    const double rr = band_p[t] / eps;
    const double one_minus_H = 0.5 * (1 - rr - one_over_pi * portable_sin(pi * rr));
    const double v = one_minus_H * dV;
    contrib[band_q[t]] = v;
    sum += approx(v);
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if (lane == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kContribThreads / 32; w++) sum += red[w];
    csum[blockIdx.x] = sum;
  }
}

// the estimate of chunk j's sum from PER partial sums (past np: none)
template <typename T, int PER>
__device__ __forceinline__ double chunk_estimate(const T* __restrict__ csum, int64_t np, int64_t j) {
  double s = 0;
#pragma unroll
  for (int q = 0; q < PER; q++)
    if (PER * j + q < np) s += (double)csum[PER * j + q];
  return s;
}

// exclusive scan of nc chunk sums in one block of 1024 threads
template <typename T, int PER>
__global__ void __launch_bounds__(1024) k_vol_scan(const T* __restrict__ csum, int64_t np, int64_t nc, double* est) {
  __shared__ double part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t per = (nc + 1023) / 1024;
  const int64_t lo = threadIdx.x * per, hi = lo + per < nc ? lo + per : nc;
  double s = 0;
  for (int64_t j = lo; j < hi; j++) s += chunk_estimate<T, PER>(csum, np, j);
  double incl = s;
  for (int o = 1; o < 32; o <<= 1) {
    const double x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) part[warp] = incl;
  __syncthreads();
  double run = incl - s;
  for (int w = 0; w < warp; w++) run += part[w];
  for (int64_t j = lo; j < hi; j++) {
    est[j] = run;
    run += chunk_estimate<T, PER>(csum, np, j);
  }
}

// R[3j+q], F[3j+q] for E = exp(est[j]) - 1 + q
template <typename T, int PER>
__global__ void __launch_bounds__(kVolThreads) k_vol_chunk_r(const double* __restrict__ c, int64_t n,
                                                             const T* __restrict__ csum, int64_t np, bool scanned,
                                                             double* est, int64_t* R, int* F) {
  __shared__ unsigned long long rs[3][kVolThreads];
  __shared__ int fs[3][kVolThreads];
  __shared__ double s_est[kVolThreads / 32];
  const int64_t j = blockIdx.x;
  double e = 0;
  if (scanned) {
    e = est[j];
  } else {
    for (int64_t q = threadIdx.x; q < PER * j; q += kVolThreads) e += (double)csum[q];
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) s_est[threadIdx.x >> 5] = e;
    __syncthreads();
    e = 0;
    for (int w = 0; w < kVolThreads / 32; w++) e += s_est[w];
    if (threadIdx.x == 0) est[j] = e;
  }
  const int E0 = exp_of(e);
  const int64_t base = j * kVolChunk;
  unsigned long long r[3] = {0, 0, 0};
  bool bad[3] = {E0 < -1000, E0 < -1000, E0 < -1000};
  if (E0 >= -1000) {
    for (int t = threadIdx.x; t < kVolChunk; t += kVolThreads) {
      const int64_t q = base + t;
      if (q >= n) break;
      const double x = c[q];
#pragma unroll
      for (int k = 0; k < 3; k++) r[k] += rne_units(x, E0 - 1 + k, bad[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    rs[k][threadIdx.x] = r[k];
    fs[k][threadIdx.x] = bad[k] ? 1 : 0;
  }
  __syncthreads();
  for (int w = kVolThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        rs[k][threadIdx.x] += rs[k][threadIdx.x + w];
        fs[k][threadIdx.x] |= fs[k][threadIdx.x + w];
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < 3) {
    const int k = threadIdx.x;
    // a chunk sum that does not fit the significand range is not applicable
    R[3 * j + k] = (int64_t)rs[k][0];
    F[3 * j + k] = (fs[k][0] || rs[k][0] >= (1ull << 53)) ? 1 : 0;
  }
}

// Inclusive scan of r over the block.  Then, with M the running sum in units of
// its binade: the first thread that does not apply (bad, or M + its scan
// reaches the top of the binade), kVolThreads if none, and the scan up to it.
struct WalkScan {
  unsigned long long warp_sum[kVolThreads / 32], before;
  int warp_first[kVolThreads / 32];
};
__device__ __forceinline__ int walk_scan(WalkScan& w, unsigned long long r, bool bad, uint64_t M,
                                         unsigned long long& before) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = r;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) w.warp_sum[warp] = incl;
  __syncthreads();
  for (int q = 0; q < warp; q++) incl += w.warp_sum[q];
  const unsigned stop = __ballot_sync(0xffffffffu, bad || M + incl >= (1ull << 53) - 1);
  if (lane == 0) w.warp_first[warp] = stop ? 32 * warp + __ffs(stop) - 1 : kVolThreads;
  __syncthreads();
  int first = kVolThreads;
  for (int q = 0; q < kVolThreads / 32; q++) first = min(first, w.warp_first[q]);
  if ((int)threadIdx.x == (first < kVolThreads ? first : kVolThreads - 1)) w.before = first < kVolThreads ? incl - r : incl;
  __syncthreads();
  before = w.before;
  return first;
}

// the running sum s, in a valid binade, advanced by R units of it
__device__ __forceinline__ double advance(double s, unsigned long long R) {
  return R ? dfrom(dbits(s) + R) : s;  // below the binade's top: the significand does not carry
}

// one block: the exact running sum over the chunks in loop order
__global__ void __launch_bounds__(kVolThreads) k_vol_walk(const double* __restrict__ c, int64_t n, int64_t nc,
                                                          const double* __restrict__ est, const int64_t* __restrict__ R,
                                                          const int* __restrict__ F, bool have_r, double* out) {
  __shared__ WalkScan w;
  __shared__ double s_sum;
  __shared__ double x[kVolChunk];
  const int t = threadIdx.x;
  constexpr uint64_t hidden = 1ull << 52;
  double s = 0.0;  // the same in every thread
  for (int64_t j = 0; j < nc;) {
    unsigned long long before;
    if (have_r) {
      const int E = exp_of(s);
      bool ok = true;  // chunks past the end stop nothing
      unsigned long long r = 0;
      if (j + t < nc) {
        const int64_t q = j + t;
        const int E0 = exp_of(est[q]), k = E - (E0 - 1);
        ok = E > -1000 && E0 > -1000 && k >= 0 && k <= 2;
        if (ok) ok = F[3 * q + k] == 0;
        if (ok) r = (unsigned long long)R[3 * q + k];
      }
      const int first = walk_scan(w, r, !ok, E > -1000 ? (dbits(s) & (hidden - 1)) | hidden : 0, before);
      s = advance(s, before);
      j += first;
      if (first == kVolThreads || j >= nc) continue;
    }
    // chunk j: windows of kVolThreads * per consecutive elements, per of them to a
    // thread.  The sum takes about as many elements again to leave a binade as it
    // took to enter it, so per grows with the elements behind.
    __syncthreads();  // the previous chunk's elements are no longer read
    const int64_t base = j * kVolChunk;
#pragma unroll
    for (int q = 0; q < kVolPer; q++) {
      const int64_t e = base + q * kVolThreads + t;
      x[q * kVolThreads + t] = e < n ? c[e] : 0.0;
    }
    __syncthreads();
    for (int start = 0; start < kVolChunk;) {
      const int E = exp_of(s);
      const int64_t behind = (base + start) / (2 * kVolThreads);
      const int per = behind < 1 ? 1 : (behind < kVolPer ? (int)behind : kVolPer);
      bool bad = false;
      unsigned long long r = 0;
      const int lo = start + t * per, hi = lo + per < kVolChunk ? lo + per : kVolChunk;
      for (int q = lo; q < hi; q++) r += rne_units(x[q], E, bad);
      const int first = walk_scan(w, r, bad, E > -1000 ? (dbits(s) & (hidden - 1)) | hidden : 0, before);
      s = advance(s, before);
      if (first == kVolThreads) {
        start += kVolThreads * per;
        continue;
      }
      if (t == first) {  // element by element, in loop order, skipping exact zeros
        double v = s;
        for (int q = lo; q < hi; q++) {
          const double y = x[q];
          if ((dbits(y) << 1) != 0) v = v + y;
        }
        s_sum = v;
      }
      __syncthreads();
      s = s_sum;
      start += (first + 1) * per;
    }
    j++;
  }
  if (t == 0) *out = s;
}

}  // namespace

int64_t loop_sum_scratch_doubles(int64_t n) {
  const int64_t nc = (n + kVolChunk - 1) / kVolChunk;
  return 8 * nc + 64;
}

namespace {

// steps 2 to 4; np partial sums, PER a chunk, are at the start of scratch
// (2 nc doubles), then the estimates (nc), R (3 nc) and F (3 nc ints)
template <typename T, int PER>
void sum_chunks(cudaStream_t s, const double* c, int64_t n, int64_t np, double* scratch, double* out) {
  static_assert(PER * sizeof(T) <= 2 * sizeof(double), "partial sums outgrow their part of the scratch");
  const int64_t nc = (n + kVolChunk - 1) / kVolChunk;
  const T* csum = reinterpret_cast<const T*>(scratch);
  double* est = scratch + 2 * nc;
  int64_t* R = reinterpret_cast<int64_t*>(est + nc);
  int* F = reinterpret_cast<int*>(R + 3 * nc);
  const bool have_r = nc > kSmallChunks, scanned = nc > kScanChunks;
  if (scanned) k_vol_scan<T, PER><<<1, 1024, 0, s>>>(csum, np, nc, est);
  if (have_r) k_vol_chunk_r<T, PER><<<(unsigned)nc, kVolThreads, 0, s>>>(c, n, csum, np, scanned, est, R, F);
  k_vol_walk<<<1, kVolThreads, 0, s>>>(c, n, nc, est, R, F, have_r, out);
}

}  // namespace

void launch_loop_sum(cudaStream_t s, const double* c, int64_t n, double* scratch, double* out) {
  if (n <= 0) {
    QSS_CK(cudaMemsetAsync(out, 0, sizeof(double), s));
    return;
  }
  k_vol_chunk_sum<<<(unsigned)((n + kVolChunk - 1) / kVolChunk), kVolThreads, 0, s>>>(c, n, scratch);
  sum_chunks<double, 1>(s, c, n, (n + kVolChunk - 1) / kVolChunk, scratch, out);
}

void launch_volume(cudaStream_t s, const Box& b, const double* phi, double dx, double dy, double dz, double eps,
                   double* scratch, double* out) {
  const int64_t n = (int64_t)b.fbx() * b.fby() * b.fbz();
  if (n <= 0) {
    QSS_CK(cudaMemsetAsync(out, 0, sizeof(double), s));
    return;
  }
  const double dV = dx * dy * dz;
  const unsigned np = (unsigned)((n + kContribVoxels - 1) / kContribVoxels);
  k_vol_contrib<<<np, kContribThreads, 0, s>>>(b, phi, dV, eps, scratch, reinterpret_cast<float*>(scratch + n));
  sum_chunks<float, kVolChunk / kContribVoxels>(s, scratch, n, np, scratch + n, out);
}

}  // namespace qss

using namespace qss;

// ---------------------------------------------------------------------------
extern "C" {

// See include/lsmpqs_gpu.h.
int qssgpu_loop_sum(const double* values, long long n, double* out) {
  try {
    ensure_device();
    if (n < 0 || (n > 0 && !values) || !out) throw Error(QSSGPU_ERR_ARG, "qssgpu_loop_sum: bad argument");
    cudaStream_t s = nullptr;
    QSS_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    double *dv = nullptr, *scratch = nullptr, *dout = nullptr;
    const int64_t nn = n > 0 ? n : 1;
    QSS_CK(cudaMalloc(&dv, nn * sizeof(double)));
    QSS_CK(cudaMalloc(&scratch, loop_sum_scratch_doubles(nn) * sizeof(double)));
    QSS_CK(cudaMalloc(&dout, sizeof(double)));
    if (n > 0) QSS_CK(cudaMemcpyAsync(dv, values, n * sizeof(double), cudaMemcpyHostToDevice, s));
    launch_loop_sum(s, dv, n, scratch, dout);
    QSS_CK(cudaGetLastError());
    QSS_CK(cudaMemcpyAsync(out, dout, sizeof(double), cudaMemcpyDeviceToHost, s));
    QSS_CK(cudaStreamSynchronize(s));
    cudaFree(dv);
    cudaFree(scratch);
    cudaFree(dout);
    cudaStreamDestroy(s);
    return 0;
  } catch (const std::exception& e) {
    return report_exception(e);
  }
}

}  // extern "C"
