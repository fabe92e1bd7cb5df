// qss_stage.cuh -- the pointwise part of a right-hand side with its products,
// roots and divisions as straight-line integer-pipe code (qss_emu.cuh): the
// Godunov normal term, the central curvature term, the upwind advection term
// and the TVD-RK combination, shared by the WENO5 combine kernel and the
// ENO2 / ENO3 stage kernel.
//
// One test per group of operands (all raw differences in [2^-127, 2^129), the
// grid factors in [2^-50, 2^50]) keeps every product normal, so the products
// need no test of their own; a voxel that fails it takes the native expression
// of qss_device.cuh, whose bits the fast one reproduces.  What stays on the FP64
// pipe are the additions (28 in the curvature, about 36 in all): they and the
// ~1400 integer instructions take about the same time.
#pragma once
#include "qss_device.cuh"
#include "qss_emu.cuh"
#include "qss_kernels.cuh"

namespace qss {

// |x| in [2^-127, 2^129) where the result is below 2^29; several are tested by
// one OR
__device__ __forceinline__ uint32_t win8(double x) { return qss_emu::hi32(x) * 2u - 0x70000000u; }
constexpr uint32_t kWin8 = 0x20000000u;
__device__ __forceinline__ bool is_zero(double x) { return ((qss_emu::hi32(x) * 2u) | qss_emu::lo32(x)) == 0; }

__device__ __forceinline__ double mulw(double x, double y, int k = 0) {
  return qss_emu::mul_win(qss_emu::hi32(x), qss_emu::lo32(x), qss_emu::hi32(y), qss_emu::lo32(y), k);
}
__device__ __forceinline__ double sqw(double x) { return qss_emu::sq_win(qss_emu::hi32(x), qss_emu::lo32(x)); }

// |v| >= 1e-5 (false for NaN)
__device__ __forceinline__ bool speed_valid(double v) {
  const uint64_t a = qss_emu::mag2(qss_emu::bits(v));
  return a >= 0x7dc9f16b11c6d1e2ull && a <= qss_emu::kInf2;
}

// host: factors the fast paths accept
inline bool stage_factor(double f) { return f >= 0x1p-50 && f <= 0x1p50; }

// Every fallback is out of line: inlined, its FP64 instructions would be issued
// under a predicate by every warp.
static __device__ __noinline__ double curvature_native(const double* __restrict__ phi, const Box& b, int64_t c, Fac f) {
  return curvature(phi, b, c, f);
}

// a + b + c of squares; INT: on the integer pipes
template <bool INT>
__device__ __forceinline__ double sum_sq(double a, double b, double c) {
  return INT ? qss_emu::add_pos(qss_emu::add_pos(a, b), c) : a + b + c;
}

// curvature() (3d.f:2337-2379), the same operations.  ZERO: exact zeros among the
// differences (planes, symmetric parts) stay in the straight line, where a product
// with one holds nothing of use and its term is replaced by a signed zero; otherwise
// they take the native form.  ENO2 on GB300: drainage 64^3, where plane parts are
// common, stages 9.13 -> 8.13 ms.  The WENO5 combine kernel goes without: 24^3 6 % and
// 110^3 1 % faster with it, 192^3 and 320^3 1 % slower (registers).
template <bool INT = false, bool ZERO = false>
__device__ __forceinline__ double curvature_fast(const double* __restrict__ phi, const Box& b, int64_t c,
                                                 const Fac& f) {
  const int64_t sy = b.sy(), sz = b.sz();
  const double* __restrict__ q = phi + c;
  const double cc = __ldg(q);
  const double dx = __ldg(q + 1) - __ldg(q - 1);
  const double dy = __ldg(q + sy) - __ldg(q - sy);
  const double dz = __ldg(q + sz) - __ldg(q - sz);
  // ... - 2 cc: the product of the FMA is exact
  const double dxx = __fma_rn(-2.0, cc, __ldg(q + 2) + __ldg(q - 2));
  const double dzz = __fma_rn(-2.0, cc, __ldg(q + 2 * sz) + __ldg(q - 2 * sz));
  const double dyy = __fma_rn(-2.0, cc, __ldg(q + 2 * sy) + __ldg(q - 2 * sy));
  const double dxy = __ldg(q + 1 + sy) + __ldg(q - 1 - sy) - __ldg(q - 1 + sy) - __ldg(q + 1 - sy);
  const double dxz = __ldg(q + 1 + sz) + __ldg(q - 1 - sz) - __ldg(q - 1 + sz) - __ldg(q + 1 - sz);
  const double dyz = __ldg(q + sy + sz) + __ldg(q - sy - sz) - __ldg(q - sy + sz) - __ldg(q + sy - sz);
  auto zero = [](double d) { return ZERO && is_zero(d); };
  const bool zx = zero(dx), zy = zero(dy), zz = zero(dz);
  const bool zxx = zero(dxx), zyy = zero(dyy), zzz = zero(dzz);
  const bool zxy = zero(dxy), zxz = zero(dxz), zyz = zero(dyz);
  auto out = [](bool z, double d) { return z ? 0u : win8(d); };
  const uint32_t w = out(zx, dx) | out(zy, dy) | out(zz, dz) | out(zxx, dxx) | out(zyy, dyy) | out(zzz, dzz) |
                     out(zxy, dxy) | out(zxz, dxz) | out(zyz, dyz);
  if (w >= kWin8) return curvature_native(phi, b, c, f);
  auto term = [](bool zero, uint32_t sign, double v) {
    return zero ? __hiloint2double((int)(sign & 0x80000000u), 0) : v;
  };
  const uint32_t hx = qss_emu::hi32(dx), hy = qss_emu::hi32(dy), hz = qss_emu::hi32(dz);
  const uint32_t hxx = qss_emu::hi32(dxx), hyy = qss_emu::hi32(dyy), hzz = qss_emu::hi32(dzz);
  const double x = mulw(dx, f.x), y = mulw(dy, f.y), z = mulw(dz, f.z);
  const double g2 = sum_sq<INT>(term(zx, 0, sqw(x)), term(zy, 0, sqw(y)), term(zz, 0, sqw(z)));
  if (qss_emu::bits(g2) < 0x3ee4f8b588e368f1ull) return 0.0;  // 1e-5
  const double xx = mulw(mulw(dxx, f.x), f.x);
  const double yy = mulw(mulw(dyy, f.y), f.y);
  double curv = term(zxx || zy, hxx, mulw(mulw(xx, y), y)) + term(zyy || zx, hyy, mulw(mulw(yy, x), x));
  curv = curv - term(zxy || zx || zy, qss_emu::hi32(dxy) ^ hx ^ hy, mulw(mulw(mulw(mulw(dxy, f.x), f.y, 1), x), y));
  curv = curv + term(zxx || zz, hxx, mulw(mulw(xx, z), z));
  const double zzv = mulw(mulw(dzz, f.z), f.z);
  curv = curv + term(zzz || zx, hzz, mulw(mulw(zzv, x), x));
  curv = curv - term(zxz || zx || zz, qss_emu::hi32(dxz) ^ hx ^ hz, mulw(mulw(mulw(mulw(dxz, f.x), f.z, 1), x), z));
  curv = curv + term(zyy || zz, hyy, mulw(mulw(yy, z), z));
  curv = curv + term(zzz || zy, hzz, mulw(mulw(zzv, y), y));
  curv = curv - term(zyz || zy || zz, qss_emu::hi32(dyz) ^ hy ^ hz, mulw(mulw(mulw(mulw(dyz, f.y), f.z, 1), y), z));
  if (ZERO && is_zero(curv)) return curv;  // over a positive g2
  return qss_emu::div(curv, g2);
}

// whether curvature() is certainly finite: every point it reads below 2^200 in magnitude
// (grid factors of at most 2^50: numerator below 2^810, over at least 1e-5).  25 loads of
// high words in place of the curvature's FP64 instructions: the ENO2 stages with variable
// coefficients take 6.24 ms of a 128^3 step against 6.00 without the look, GB300.
__device__ __forceinline__ bool curvature_finite(const double* __restrict__ phi, const Box& b, int64_t c) {
  const int64_t st[3] = {1, b.sy(), b.sz()};
  const double* __restrict__ q = phi + c;
  uint32_t top = 0;
  auto see = [&](int64_t o) { top = max(top, __ldg(reinterpret_cast<const uint32_t*>(q + o) + 1) * 2u); };
  see(0);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int64_t s = st[d], t = st[(d + 1) % 3];
    see(s);
    see(-s);
    see(2 * s);
    see(-2 * s);
    see(s + t);
    see(s - t);
    see(t - s);
    see(-s - t);
  }
  return top < 0x98e00000u;  // 2 x the high word of 2^200
}

template <int SCHEME>
__device__ __noinline__ double godunov_native(double vel, double px, double py, double pz, double mx, double my,
                                              double mz, double ix, double iy, double iz) {
  const double pp[3] = {px * ix, py * iy, pz * iz}, pm[3] = {mx * ix, my * iy, mz * iz};
  return godunov_norm<SCHEME>(vel, pp, pm);
}

// godunov_norm<SCHEME>() of the one-sided differences pp[d] inv[d], pm[d] inv[d].
// The larger of the two candidates of an axis is picked before it is scaled and
// squared (rounding is monotone), as a signed integer maximum raised to 2^-255:
// beside a largest candidate of 2^-127 or more the floor changes no sum.
template <int SCHEME, bool SCALE, bool INT = false>
__device__ __forceinline__ double godunov_fast(double vel, const double pp[3], const double pm[3], const Inv& inv) {
  using namespace qss_emu;
  const uint64_t sm = gt0(vel) ? 0 : kSign, sp = sm ^ kSign;  // vel > 0: max(pm, -pp, 0), else max(-pm, pp, 0)
  int h[3];
  uint32_t l[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int64_t u = (int64_t)(bits(pm[d]) ^ sm), v = (int64_t)(bits(pp[d]) ^ sp);
    const int64_t w = u > v ? u : v;
    h[d] = max((int)(w >> 32), 0x30000000);
    l[d] = (uint32_t)w;
  }
  const uint32_t top = (uint32_t)max(max(h[0], h[1]), h[2]);
  if (top - 0x38000000u < 0x10000000u && win8(vel) < kWin8) {
    const double iv[3] = {inv.x, inv.y, inv.z};
    double s[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double g = __hiloint2double(h[d], (int)l[d]);
      if (SCALE) g = mulw(g, iv[d]);
      s[d] = sqw(g);
    }
    const double n2 = sum_sq<INT>(s[0], s[1], s[2]);
    const double r = mulw(vel, sqrt_win(hi32(n2), lo32(n2)));
    return SCHEME == WENO5 ? r : neg(r);
  }
  return godunov_native<SCHEME>(vel, pp[0], pp[1], pp[2], pm[0], pm[1], pm[2], SCALE ? inv.x : 1.0, SCALE ? inv.y : 1.0,
                                SCALE ? inv.z : 1.0);
}

static __device__ __noinline__ double advect_native(double sum, double vx, double vy, double vz, double ax, double ay,
                                             double az) {
  return sum + (-(vx * ax + vy * ay + vz * az));
}

// sum + (-(vx ax + vy ay + vz az)), the upwind derivative picked by the sign of
// the velocity.  The velocity is zero in the pore space: a finite derivative
// then adds +-0, which a nonzero sum does not notice.
template <bool SCALE>
__device__ __forceinline__ double add_advection(double sum, double vx, double vy, double vz, const double pp[3],
                                                const double pm[3], const Inv& inv) {
  using namespace qss_emu;
  const double sx = ge0(vx) ? pm[0] : pp[0], sy = ge0(vy) ? pm[1] : pp[1], sz = ge0(vz) ? pm[2] : pp[2];
  if (((bits(vx) | bits(vy) | bits(vz)) << 1) == 0) {
    const uint32_t top = max(max(hi32(sx) * 2u, hi32(sy) * 2u), hi32(sz) * 2u);
    // derivatives below 2^129 (finite after scaling), sum not zero
    if (top < 0x90000000u && (bits(sum) << 1) != 0) return sum;
    return advect_native(sum, vx, vy, vz, SCALE ? sx * inv.x : sx, SCALE ? sy * inv.y : sy, SCALE ? sz * inv.z : sz);
  }
  const double ax = SCALE ? mul(sx, inv.x) : sx, ay = SCALE ? mul(sy, inv.y) : sy, az = SCALE ? mul(sz, inv.z) : sz;
  return sum + neg(mul(vx, ax) + mul(vy, ay) + mul(vz, az));
}

// TVD-RK combination of one stage (0: the right-hand side itself)
template <int STAGE>
__device__ __forceinline__ double rk_combine(double rhs, double dt, double phi, const double* __restrict__ u_cur,
                                             int64_t idx) {
  using namespace qss_emu;
  if (STAGE == 0) return rhs;
  const double e = phi + mul(dt, rhs);
  if (STAGE == 1) return e;
  if (STAGE == 2) return mul(0.75, u_cur[idx]) + scale2(e, -2);
  return mul(1.0 / 3.0, u_cur[idx]) + mul(2.0 / 3.0, e);
}

// the three mask impositions with the comparisons on the integer pipes
__device__ __forceinline__ double impose3_i(double v, int64_t idx, const ImposeArgs& im) {
  double t = im.mask[idx] - im.overlap;
  v = qss_emu::gt(t, v) ? t : v;
  if (im.check_conn) {
    t = im.mask_w[idx] - 0.0;
    v = qss_emu::gt(t, v) ? t : v;
    t = im.mask_nw[idx] - 0.0;
    v = qss_emu::gt(t, v) ? t : v;
  }
  return v;
}

}  // namespace qss
