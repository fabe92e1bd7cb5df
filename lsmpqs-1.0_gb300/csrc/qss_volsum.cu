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
// where rne rounds to the nearest integer.  If c / u is exactly halfway between
// two integers, the tie goes to the even significand, so what c adds depends on
// the parity of s / u.  A run of contributions in a known binade is therefore two
// integers (struct Units): what it adds to an even and to an odd significand,
// computable in parallel and exactly.  It applies when no element is negative or
// not finite and s / u plus that stays below 2^53 - 1.
//
//   1. k_vol_contrib (volumes; the contributions are computed here) or
//      k_vol_chunk_sum (a given sequence): per chunk of 1024 contributions,
//      their sum -- only to estimate where the running sum stands;
//   2. k_vol_scan (more than 2048 chunks only; else each block of 3 sums its
//      predecessors): exclusive scan of those sums -> an estimate of s at the
//      start of each chunk, good to far better than a factor of 2;
//   3. k_vol_chunk_r: per chunk, its Units and a "not applicable" flag for the
//      estimated binade and its two neighbours, or that all of it is zero;
//   4. k_vol_walk: one block walks the chunks in order with the exact running
//      sum, 256 chunks at a time: a scan of their Units finds the first chunk that
//      does not apply (another binade, the top of the binade reached, special
//      values); the sum advances to it in one integer addition, and that chunk
//      goes the same way by groups of up to 4 elements, the group that does not
//      apply being added element by element (and more where none applies, kWalkClose).
// Every result equals the sequential loop's bit for bit.
//
// The walk is bound by latency: 1 to 2 us for each binade the sum crosses, in opening
// its chunk and scanning windows of it.  Chunks of 4096 elements, whose ties and
// leading zero chunks did not apply and whose windows were four times as long, took
// 49 us at 24^3, 117 us at 64^3 and 224 us at 128^3 on GB300; these chunks of 1024
// take 46, 63 and 109 us.  (One warp walking chunk by chunk, adding a whole chunk
// element by element: 0.42 ms at 24^3, 3.5 ms at 192^3.)  Windows of one warp for the
// first elements, without barriers, were slower; so was the rounding with branches.
#include "qss_emu.cuh"
#include "qss_kernels.cuh"
#include "qss_state.h"

namespace qss {

namespace {

constexpr int kVolThreads = 256;
constexpr int kVolPer = kVolChunk / kVolThreads;  // elements per thread in the walk
constexpr int kScanChunks = 2048;                 // from here on the estimates are scanned by a kernel
constexpr int kSmallChunks = 2;                   // up to here the walk goes by elements alone
constexpr int kWalkChunks = 8;                    // chunks to a thread of the walk, at most
// Stops closer than this cost more than adding the elements between them one by one (a
// window that stops takes about 3 us, an addition 0.042).  1 M negative elements, whole
// call: 424 ms with a window for every 4 of them, 42 now; a negative element in every
// 100, which stay with the windows, 20.  A sum that climbs leaves the binade with each
// stop and is not concerned.
constexpr int kWalkClose = 32;

__device__ __forceinline__ uint64_t dbits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ double dfrom(uint64_t b) { return __longlong_as_double((long long)b); }

// unbiased exponent of a positive normal double, or a sentinel
__device__ __forceinline__ int exp_of(double x) {
  const uint64_t b = dbits(x);
  const int e = (int)((b >> 52) & 0x7ff);
  if ((b >> 63) || e == 0 || e == 0x7ff) return -100000;
  return e - 1023;
}

// c / u rounded to an integer, for u = 2^(E - 52); on a tie, rounded down.  bad: a
// negative or non-finite c, or c >= 2^E.  Without branches, so that a thread's
// elements overlap.
__device__ __forceinline__ uint64_t rne_units(double c, int E, bool& bad, bool& tie) {
  const uint64_t b = dbits(c);
  const uint32_t hi = (uint32_t)(b >> 32), ec = (hi >> 20) & 0x7ffu;
  // c = m 2^(max(ec, 1) - 1075), c / u = m / 2^sh
  const uint64_t m = (b & ((1ull << 52) - 1)) | (ec ? 1ull << 52 : 0ull);
  const int sh = E + 1023 - (ec ? (int)ec : 1);
  // sh <= 0: c >= 2^E, s leaves the binade.  +-0 leaves s unchanged.
  bad = bad || (((hi >> 31) || ec == 0x7ffu || sh <= 0) && (b << 1) != 0);
  const int d = min(max(sh, 1), 55) - 1;  // from 54 on below half a unit
  const uint64_t h = m >> d;              // c / u in halves, rounded down
  tie = (h & 1) && (h << d) == m;
  return (h + (tie ? 0 : 1)) >> 1;
}

// What a run of contributions adds to the significand of s: r units where it is
// even before the run, r + d where it is odd.  A tie goes to the even sum; two
// significands one apart end 0, 1 or 2 apart, and stay so once they are of one
// parity, so d is -1, 0 or 1.
struct Units {
  unsigned long long r;
  int d;
};
__device__ __forceinline__ void add_units(Units& a, uint64_t q, bool tie) {
  if (tie) {
    const unsigned long long even = a.r + q, odd = even + (unsigned long long)(long long)a.d + 1;
    a.d = (int)(odd + (odd & 1) - 1 - even - (even & 1));
    a.r = even + (even & 1);
  } else {
    a.r += q;
  }
}
// a, then b
__device__ __forceinline__ Units join(const Units& a, const Units& b) {
  const bool odd = a.r & 1;
  return {a.r + b.r + (unsigned long long)(long long)(odd ? b.d : 0), a.d != 0 ? a.d : (odd ? -b.d : b.d)};
}
// the significand m after the run
__device__ __forceinline__ unsigned long long after(unsigned long long m, const Units& a) {
  return m + a.r + (unsigned long long)(long long)((m & 1) ? a.d : 0);
}
// kVolPer consecutive elements to a thread, without bank conflicts
constexpr int kVolStage = kVolChunk + kVolChunk / kVolPer;
__device__ __forceinline__ int stage_at(int e) { return e + e / kVolPer; }

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
// each chunk in units of dV.  A voxel outside the smoothing band costs an
// integer comparison; those inside (about 15 % of the voxels, but a lane or more
// of most warps) are first gathered, then evaluated by full warps: their division
// and sine are ~45 FP64 instructions and the kernel's bound.  A block is a chunk:
// 1024 voxels, so that small boxes use more SMs (24^3 49 us with 4096).
constexpr int kContribThreads = 256;

__global__ void __launch_bounds__(kContribThreads) k_vol_contrib(Box b, const double* __restrict__ phi, double dV,
                                                                 double eps, double* contrib, float* csum) {
  __shared__ double band_p[kVolChunk];
  __shared__ uint16_t band_t[kVolChunk];
  __shared__ int band_n;
  __shared__ float red[kContribThreads / 32];
  const double pi = 3.14159265358979323846;
  const double one_over_pi = 0.31830988618379;
  const FillBlock blk(b, blockIdx.x, kVolChunk);
  contrib += blk.base;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) band_n = 0;
  __syncthreads();
  // the estimate is in units of dV, which itself may lie outside the float range; a value
  // as a float by its bits (a conversion is an FP64 instruction)
  auto approx = [](double v) {
    const uint32_t h = qss_emu::hi32(v);
    return h - 0x38100000u < 0x0fe00000u ? __uint_as_float((h - 0x38000000u) << 3) : 0.0f;
  };
  float sum = 0.0f;
#pragma unroll
  for (int t0 = 0; t0 < kVolChunk; t0 += kContribThreads) {
    const uint32_t t = t0 + threadIdx.x;
    bool band = false;
    double p = 0.0;
    if (blk.in(t)) {
      p = phi[blk.at(b, t)];
      const bool inside = qss_emu::gt(-eps, p);  // p < -eps
      band = !inside && qss_emu::gt(eps, p);     // p < eps
      if (!band) contrib[t] = inside ? dV : 0.0;
      if (inside) sum += 1.0f;
    }
    const unsigned m = __ballot_sync(0xffffffffu, band);
    int at = 0;
    if (lane == 0 && m) at = atomicAdd(&band_n, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (band) {
      band_p[at] = p;
      band_t[at] = (uint16_t)t;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < band_n; e += kContribThreads) {
    const double rr = band_p[e] / eps;
    const double one_minus_H = 0.5 * (1 - rr - one_over_pi * portable_sin(pi * rr));
    const double v = one_minus_H * dV;
    contrib[band_t[e]] = v;
    sum += approx(one_minus_H);
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if (lane == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kContribThreads / 32; w++) sum += red[w];
    csum[blockIdx.x] = sum;
  }
}

// exclusive scan of nc chunk sums, in units of `unit`, in one block of 1024 threads
template <typename T>
__global__ void __launch_bounds__(1024) k_vol_scan(const T* __restrict__ csum, int64_t nc, double unit, double* est) {
  __shared__ double part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t per = (nc + 1023) / 1024;
  const int64_t lo = threadIdx.x * per, hi = lo + per < nc ? lo + per : nc;
  double s = 0;
  for (int64_t j = lo; j < hi; j++) s += (double)csum[j];
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
    est[j] = run * unit;
    run += (double)csum[j];
  }
}

// R[3j+q], F[3j+q] for E = exp(est[j]) - 1 + q.  F: kZeroChunk, all contributions
// zero (nothing changes whatever the sum); kBadChunk, not applicable; else d + 1
constexpr int kBadChunk = 4, kZeroChunk = 5;
template <typename T>
__global__ void __launch_bounds__(kVolThreads) k_vol_chunk_r(const double* __restrict__ c, int64_t n,
                                                             const T* __restrict__ csum, double unit,
                                                             bool scanned, double* est, int64_t* R, int* F) {
  __shared__ double x[kVolStage];
  __shared__ Units part[3][kVolThreads / 32];
  __shared__ double s_est[kVolThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t j = blockIdx.x, base = j * kVolChunk;
  bool some = false;
#pragma unroll
  for (int q = 0; q < kVolPer; q++) {
    const int e = q * kVolThreads + threadIdx.x;
    const double v = base + e < n ? c[base + e] : 0.0;
    x[stage_at(e)] = v;
    some = some || (dbits(v) << 1) != 0;
  }
  double e = 0;
  if (scanned) {
    e = est[j];
  } else {
    for (int64_t q = threadIdx.x; q < j; q += kVolThreads) e += (double)csum[q];
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lane == 0) s_est[warp] = e;
  }
  if (!__syncthreads_or(some)) {
    if (threadIdx.x < 3) F[3 * j + threadIdx.x] = kZeroChunk;
    if (threadIdx.x == 0 && !scanned) est[j] = 0.0;  // not used
    return;
  }
  if (!scanned) {
    e = 0;
    for (int w = 0; w < kVolThreads / 32; w++) e += s_est[w];
    e *= unit;
    if (threadIdx.x == 0) est[j] = e;
  }
  const int E0 = exp_of(e);
  Units u[3] = {};
  bool bad[3] = {E0 < -1000, E0 < -1000, E0 < -1000};
  if (E0 >= -1000) {
    for (int q = 0; q < kVolPer; q++) {
      const double v = x[stage_at(threadIdx.x * kVolPer + q)];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        bool tie;
        const uint64_t r = rne_units(v, E0 - 1 + k, bad[k], tie);
        add_units(u[k], r, tie);
      }
    }
  }
  int any = 0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (bad[k] || u[k].r >= (1ull << 53)) {  // the second also keeps the sums below 2^63
      any |= 1 << k;
      u[k] = Units{0, 0};
    }
    for (int o = 1; o < 32; o <<= 1) {
      const Units v{__shfl_down_sync(0xffffffffu, u[k].r, o), __shfl_down_sync(0xffffffffu, u[k].d, o)};
      if ((lane & (2 * o - 1)) == 0) u[k] = join(u[k], v);
    }
    if (lane == 0) part[k][warp] = u[k];
  }
  __shared__ int s_any;
  if (threadIdx.x == 0) s_any = 0;
  __syncthreads();
  if (any) atomicOr(&s_any, any);
  __syncthreads();
  if (threadIdx.x < 3) {
    const int k = threadIdx.x;
    Units t = part[k][0];
    for (int w = 1; w < kVolThreads / 32; w++) t = join(t, part[k][w]);
    // a chunk sum that does not fit the significand range is not applicable
    R[3 * j + k] = (int64_t)t.r;
    F[3 * j + k] = ((s_any >> k) & 1) || t.r >= (1ull << 53) ? kBadChunk : t.d + 1;
  }
}

// The significand m through the block's runs u in thread order: the first thread
// that does not apply (bad, or the top of the binade reached), kVolThreads if none,
// and in `before` the significand ahead of it.
struct WalkScan {
  Units warp_sum[kVolThreads / 32];
  unsigned long long before[kVolThreads / 32];
  int first[kVolThreads / 32];
};
__device__ __forceinline__ Units warp_join(Units u, int lane) {
  if (__any_sync(0xffffffffu, u.d != 0)) {
    for (int o = 1; o < 32; o <<= 1) {
      const Units v{__shfl_up_sync(0xffffffffu, u.r, o), __shfl_up_sync(0xffffffffu, u.d, o)};
      if (lane >= o) u = join(v, u);
    }
  } else {
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, u.r, o);
      if (lane >= o) u.r += v;
    }
  }
  return u;
}
constexpr unsigned long long kBinadeTop = (1ull << 53) - 1;
__device__ __forceinline__ int walk_scan(WalkScan& w, Units u, bool bad, unsigned long long m,
                                         unsigned long long& before) {
  constexpr int kWarps = kVolThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u = warp_join(u, lane);
  if (lane == 31) w.warp_sum[warp] = u;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kWarps - 1; q++) {
    const Units v = w.warp_sum[q];
    if (q < warp) m = after(m, v);
  }
  const unsigned long long end = after(m, u), prev = __shfl_up_sync(0xffffffffu, end, 1);
  const unsigned stop = __ballot_sync(0xffffffffu, bad || end >= kBinadeTop);
  const int at = stop ? __ffs(stop) - 1 : 31;
  if (lane == at) {
    w.first[warp] = stop ? 32 * warp + at : kVolThreads;
    w.before[warp] = !stop ? end : (lane ? prev : m);
  }
  __syncthreads();
  int first = kVolThreads;
  before = w.before[kWarps - 1];
#pragma unroll
  for (int q = kWarps - 1; q >= 0; q--) {
    if (w.first[q] < kVolThreads) {
      first = w.first[q];
      before = w.before[q];
    }
  }
  return first;
}

// the running sum s, with significand m and in a valid binade, once the significand is `to`
__device__ __forceinline__ double advance(double s, unsigned long long m, unsigned long long to) {
  return dfrom(dbits(s) + (to - m));  // below the binade's top: the significand does not carry
}

// the elements [lo, hi) of a staged chunk in the binade E
__device__ __forceinline__ Units window_units(const double* x, int lo, int hi, int E, bool& bad) {
  Units u{0, 0};
  bad = false;
#pragma unroll
  for (int q = 0; q < kVolPer; q++) {
    if (lo + q < hi) {
      bool tie;
      const uint64_t r = rne_units(x[stage_at(lo + q)], E, bad, tie);
      add_units(u, r, tie);
    }
  }
  if (bad || u.r >= (1ull << 53)) {  // past the binade; also keeps sums over the block below 2^63
    bad = true;
    u = Units{0, 0};
  }
  return u;
}

// one block: the exact running sum over the chunks in loop order
__global__ void __launch_bounds__(kVolThreads) k_vol_walk(const double* __restrict__ c, int64_t n, int64_t nc,
                                                          const double* __restrict__ est, const int64_t* __restrict__ R,
                                                          const int* __restrict__ F, bool have_r, double* out) {
  __shared__ WalkScan w;
  __shared__ double s_sum;
  __shared__ int s_start;
  __shared__ unsigned long long s_at;
  __shared__ double x[kVolStage];
  const int t = threadIdx.x;
  constexpr uint64_t hidden = 1ull << 52;
  double s = 0.0;    // the same in every thread
  int64_t born = 0;  // where s left zero, to a few elements
  int one_by_one = 0, stop_E = 0;  // elements added one by one at the last stop, and the binade there
  // of every normal s, so that the top of its binade is seen; zero for any other s, whose
  // windows apply to zeros only
  auto significand = [&](int E) { return E >= -1022 ? (dbits(s) & (hidden - 1)) | hidden : 0ull; };
  for (int64_t j = 0; j < nc;) {
    unsigned long long before;
    if (have_r) {
      // the sum takes about as many chunks again to leave a binade as it took to enter it
      const int E = exp_of(s), cpt = j < 256 ? 1 : (j < 256 * kWalkChunks ? (int)(j / 256) : kWalkChunks);
      auto chunk_units = [&](int64_t q, bool& ok) {  // chunks past the end stop nothing
        if (q >= nc) return Units{0, 0};
        const double e = est[q];
        const int f[3] = {F[3 * q], F[3 * q + 1], F[3 * q + 2]};
        const int64_t r[3] = {R[3 * q], R[3 * q + 1], R[3 * q + 2]};
        if (f[0] == kZeroChunk) return Units{0, 0};
        const int E0 = exp_of(e), k = E - (E0 - 1), fk = k == 0 ? f[0] : (k == 1 ? f[1] : f[2]);
        if (E <= -1000 || E0 <= -1000 || k < 0 || k > 2 || fk == kBadChunk) {
          ok = false;
          return Units{0, 0};
        }
        return Units{(unsigned long long)(k == 0 ? r[0] : (k == 1 ? r[1] : r[2])), fk - 1};
      };
      bool ok = true;
      Units u{0, 0};
      for (int i = 0; i < cpt; i++) u = join(u, chunk_units(j + (int64_t)t * cpt + i, ok));
      const unsigned long long m = significand(E);
      const int first = walk_scan(w, u, !ok, m, before);
      if (first < kVolThreads && cpt > 1) {  // which of the thread's chunks
        if (t == first) {
          int i = 0;
          unsigned long long at = before;
          for (; i < cpt; i++) {
            bool fits = true;
            const unsigned long long end = after(at, chunk_units(j + (int64_t)t * cpt + i, fits));
            if (!fits || end >= kBinadeTop) break;
            at = end;
          }
          s_at = at;
          s_start = i;
        }
        __syncthreads();
        before = s_at;
        j += s_start;
      }
      s = advance(s, m, before);
      j += (int64_t)first * cpt;
      if (first == kVolThreads || j >= nc) continue;
    }
    // chunk j, by windows of consecutive elements, per of them to a thread.  The sum
    // takes about as many elements again to leave a binade as it took to enter it,
    // so per grows with the elements since it left zero.
    __syncthreads();  // the previous chunk's elements are no longer read
    const int64_t base = j * kVolChunk;
#pragma unroll
    for (int q = 0; q < kVolPer; q++) {
      const int64_t e = base + q * kVolThreads + t;
      x[stage_at(q * kVolThreads + t)] = e < n ? c[e] : 0.0;
    }
    __syncthreads();
    int start = 0;
    while (start < kVolChunk) {
      const int E = exp_of(s);
      const int64_t since = base + start - born;
      const int per = since < 512 ? 1 : (since < 512 * kVolPer ? (int)(since / 512) : kVolPer);
      const int lo = start + t * per, hi = lo + per < kVolChunk ? lo + per : kVolChunk;
      bool bad;
      const Units u = window_units(x, lo, hi, E, bad);
      const unsigned long long m = significand(E);
      const int first = walk_scan(w, u, bad, m, before);
      s = advance(s, m, before);
      if (first == kVolThreads) {
        start += kVolThreads * per;
        continue;
      }
      // element by element, in loop order (a zero of either sign leaves the sum, which is
      // never -0, as it is): the group that does not
      // apply, and twice as many elements as at the last stop where that was close and in
      // the same binade (elements or sums that no window takes)
      one_by_one = first * per < kWalkClose && E == stop_E ? max(per, min(2 * one_by_one, kVolChunk)) : per;
      stop_E = E;
      const int from = start + first * per, to = min(from + one_by_one, kVolChunk);
      if (t == first) {
        double v = s;
#pragma unroll 8
        for (int q = from; q < to; q++) v = v + x[stage_at(q)];
        s_sum = v;
      }
      __syncthreads();
      if ((dbits(s) << 1) == 0) born = base + from;
      s = s_sum;
      start = to;
    }
    j++;
  }
  if (t == 0) *out = s;
}

}  // namespace

namespace {

// steps 2 to 4; the chunks' sums in units of `unit` are at the start of scratch, from its
// double 2 nc on the estimates (nc), R (3 nc) and F (3 nc ints)
template <typename T>
void sum_chunks(cudaStream_t s, const double* c, int64_t n, double unit, double* scratch, double* out) {
  const int64_t nc = (n + kVolChunk - 1) / kVolChunk;
  const T* csum = reinterpret_cast<const T*>(scratch);
  double* est = scratch + 2 * nc;
  int64_t* R = reinterpret_cast<int64_t*>(est + nc);
  int* F = reinterpret_cast<int*>(R + 3 * nc);
  const bool have_r = nc > kSmallChunks, scanned = nc > kScanChunks;
  if (scanned) k_vol_scan<<<1, 1024, 0, s>>>(csum, nc, unit, est);
  if (have_r) k_vol_chunk_r<<<(unsigned)nc, kVolThreads, 0, s>>>(c, n, csum, unit, scanned, est, R, F);
  k_vol_walk<<<1, kVolThreads, 0, s>>>(c, n, nc, est, R, F, have_r, out);
}

}  // namespace

void launch_loop_sum(cudaStream_t s, const double* c, int64_t n, double* scratch, double* out) {
  if (n <= 0) {
    QSS_CK(cudaMemsetAsync(out, 0, sizeof(double), s));
    return;
  }
  k_vol_chunk_sum<<<(unsigned)((n + kVolChunk - 1) / kVolChunk), kVolThreads, 0, s>>>(c, n, scratch);
  sum_chunks<double>(s, c, n, 1.0, scratch, out);
}

void launch_volume(cudaStream_t s, const Box& b, const double* phi, double dx, double dy, double dz, double eps,
                   double* scratch, double* out) {
  const int64_t n = (int64_t)b.fbx() * b.fby() * b.fbz();
  if (n <= 0) {
    QSS_CK(cudaMemsetAsync(out, 0, sizeof(double), s));
    return;
  }
  const double dV = dx * dy * dz;
  k_vol_contrib<<<(unsigned)((n + kVolChunk - 1) / kVolChunk), kContribThreads, 0, s>>>(
      b, phi, dV, eps, scratch, reinterpret_cast<float*>(scratch + n));
  sum_chunks<float>(s, scratch, n, dV, scratch + n, out);
}

}  // namespace qss

using namespace qss;

namespace {

// a call's stream and its device arrays
struct SumCall {
  cudaStream_t s = nullptr;
  void* p[3] = {};
  size_t bytes[3] = {};
  int count = 0;
  SumCall() { QSS_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)); }
  ~SumCall() {
    for (int k = 0; k < count; k++) scratch_free(p[k], bytes[k], s);
    cudaStreamDestroy(s);
  }
  SumCall(const SumCall&) = delete;
  SumCall& operator=(const SumCall&) = delete;
  double* get(int64_t n) {
    bytes[count] = (size_t)n * sizeof(double);
    p[count] = scratch_alloc(bytes[count], s);
    return (double*)p[count++];
  }
};

}  // namespace

// ---------------------------------------------------------------------------
extern "C" {

// See include/lsmpqs_gpu.h.
int qssgpu_loop_sum(const double* values, long long n, double* out) {
  try {
    ensure_device();
    if (n < 0 || (n > 0 && !values) || !out) throw Error(QSSGPU_ERR_ARG, "qssgpu_loop_sum: bad argument");
    SumCall call;
    const cudaStream_t s = call.s;
    const int64_t nn = n > 0 ? n : 1;
    double *dv = call.get(nn), *scratch = call.get(loop_sum_scratch_doubles(nn)), *dout = call.get(1);
    if (n > 0) QSS_CK(cudaMemcpyAsync(dv, values, n * sizeof(double), cudaMemcpyHostToDevice, s));
    launch_loop_sum(s, dv, n, scratch, dout);
    QSS_CK(cudaGetLastError());
    QSS_CK(cudaMemcpyAsync(out, dout, sizeof(double), cudaMemcpyDeviceToHost, s));
    QSS_CK(cudaStreamSynchronize(s));
    return 0;
  } catch (const std::exception& e) {
    return report_exception(e);
  }
}

}  // extern "C"
