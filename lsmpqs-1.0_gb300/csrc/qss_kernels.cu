// qss_kernels.cu -- GB300 (sm_103a) kernels of the quasi-static level-set path.
//
// FP64 throughout, compiled with --fmad=false so that each kernel reproduces
// the reference's Fortran arithmetic bit for bit (see qss_device.cuh).  On
// GB300 the FP64 pipe, not HBM, bounds the WENO5 stage kernel; the kernels
// therefore skip work the reference throws away (the per-voxel CFL estimate
// of which only the last voxel survives, 3d.f:490) and read the stencil
// through the read-only cache (the 7/5-point lines along x, y, z and the
// 12 mixed-derivative neighbours are shared between adjacent threads).
#include <cfloat>
#include <cstdlib>
#include <cstdio>
#include <utility>
#include <vector>
#include "qss_emu.cuh"
#include "qss_kernels.cuh"
#include "qss_stage.cuh"

namespace qss {

namespace {

constexpr double kZeroTol = 1.e-5;

inline dim3 fb_grid(const Box& b, dim3 blk) {
  return dim3((b.fbx() + blk.x - 1) / blk.x, (b.fby() + blk.y - 1) / blk.y, (b.fbz() + blk.z - 1) / blk.z);
}

// ---------------------------------------------------------------------------
// inner step: dt

// weno5_side() with its products and divisions on the integer pipes, which here
// are the lower latency
__device__ __forceinline__ double weno5_side_e(double v1, double v2, double v3, double v4, double v5) {
  using namespace qss_emu;
  auto sq = [](double x) { return mul(x, x); };
  const double m = dmax(dmax(dmax(dmax(sq(v1), sq(v2)), sq(v3)), sq(v4)), sq(v5));
  const double eps = mul(1e-6, m) + 1.0e-35;
  const double p1 = mul(1.0 / 3.0, v1) - mul(7.0 / 6.0, v2) + mul(11.0 / 6.0, v3);
  const double p2 = -mul(1.0 / 6.0, v2) + mul(5.0 / 6.0, v3) + mul(1.0 / 3.0, v4);
  const double p3 = mul(1.0 / 3.0, v3) + mul(5.0 / 6.0, v4) - mul(1.0 / 6.0, v5);
  const double k1312 = 13.0 / 12.0;
  const double S1 = mul(k1312, sq(v1 - scale2(v2, 1) + v3)) + scale2(sq(v1 - scale2(v2, 2) + mul(3.0, v3)), -2);
  const double S2 = mul(k1312, sq(v2 - scale2(v3, 1) + v4)) + scale2(sq(v2 - v4), -2);
  const double S3 = mul(k1312, sq(v3 - scale2(v4, 1) + v5)) + scale2(sq(mul(3.0, v3) - scale2(v4, 2) + v5), -2);
  double a1 = div(0.1, sq(S1 + eps)), a2 = div(0.6, sq(S2 + eps)), a3 = div(0.3, sq(S3 + eps));
  const double r = div(1.0, a1 + a2 + a3);
  a1 = mul(a1, r);
  a2 = mul(a2, r);
  a3 = mul(a3, r);
  return mul(a1, p1) + mul(a2, p2) + mul(a3, p3);
}

// one of the six one-sided derivatives of upwind(): axis 0..2, plus or minus
template <int SCHEME>
__device__ __forceinline__ double upwind_one(const double* __restrict__ phi, const Box& b, int i, int j, int k,
                                             const Inv& inv, int axis, bool plus) {
  const int64_t c = b.idx(i, j, k), st = axis == 0 ? 1 : (axis == 1 ? b.sy() : b.sz());
  const double iv = axis == 0 ? inv.x : (axis == 1 ? inv.y : inv.z);
  double p, m;
  if (SCHEME == ENO2) {
    double s[5];
#pragma unroll
    for (int o = -2; o <= 2; o++) s[o + 2] = __ldg(phi + c + o * st);
    eno2_pm(s, iv, p, m);
  } else if (SCHEME == ENO3) {
    double s[7];
#pragma unroll
    for (int o = -3; o <= 3; o++) s[o + 3] = __ldg(phi + c + o * st);
    if (axis == 0) s[6] = __ldg(phi + b.idx(i + 3, j, j));  // 3d.f:677
    eno3_pm(s, iv, inv.x, p, m);
  } else {
    // v1..v5: faces i+3 .. i-1 (plus), i-2 .. i+2 (minus)
    const int64_t d = plus ? -st : st;
    const double* q = phi + c + (plus ? 3 * st : -2 * st);  // upper point of face v1
    double v[5];
#pragma unroll
    for (int o = 0; o < 5; o++) v[o] = qss_emu::mul(__ldg(q + o * d) - __ldg(q + o * d - st), iv);
    return weno5_side_e(v[0], v[1], v[2], v[3], v[4]);
  }
  return plus ? p : m;
}

// cfl_h() from the larger one-sided magnitudes
__device__ __forceinline__ double cfl_h_e(double vel, double pxc, double pyc, double pzc, double dx, double dy,
                                          double dz, const Inv& inv) {
  using namespace qss_emu;
  const double mdx = dmax(dmax(dx, dy), dz);
  const double ngp = qss_emu::sqrt(mul(pxc, pxc) + mul(pyc, pyc) + mul(pzc, pzc) + mul(mdx, mdx));
  return mul(div(qss_emu::abs(vel), ngp), mul(pxc, inv.x) + mul(pyc, inv.y) + mul(pzc, inv.z));
}

// the CFL estimate of a voxel by a group of 8 lanes (of a full warp): one
// one-sided derivative each, the result in the group's first lane
template <int SCHEME, bool VAR>
__device__ __forceinline__ double cfl_h_lanes(const Box& b, const double* __restrict__ phi, const Coef& c, int i, int j,
                                              int k, double dx, double dy, double dz, const Inv& inv) {
  const int l = threadIdx.x & 7;
  const double d = l < 6 ? upwind_one<SCHEME>(phi, b, i, j, k, inv, l >> 1, (l & 1) == 0) : 0.0;
  const double a = qss_emu::abs(d);
  const double o = __shfl_xor_sync(0xffffffffu, a, 1);
  const double mx = (l & 1) == 0 ? dmax(a, o) : dmax(o, a);  // dmax(|plus|, |minus|)
  const double py = __shfl_down_sync(0xffffffffu, mx, 2, 8), pz = __shfl_down_sync(0xffffffffu, mx, 4, 8);
  return cfl_h_e(VAR ? c.vel_n[b.idx(i, j, k)] : c.a_const, mx, py, pz, dx, dy, dz, inv);
}

// One group of 8 lanes per slab, one lane per one-sided derivative: the step's
// time is this kernel's latency (one thread computing all six with native
// divisions took 28 us for WENO5, 8 us for ENO2).
constexpr int kDtThreads = 256;

template <int SCHEME, bool VAR>
__global__ void __launch_bounds__(kDtThreads) k_dt(Box b, const double* __restrict__ phi, Coef c, int nslabs, double dx,
                                                   double dy, double dz, Inv inv, Ctl* ctl) {
  __shared__ double hs[1024];  // nslabs <= 1024
  if (!ctl->active) return;
  const int l = threadIdx.x & 7;
  for (int t0 = 0; t0 < nslabs; t0 += blockDim.x >> 3) {
    const int t = t0 + (threadIdx.x >> 3);
    const int ts = t < nslabs ? t : nslabs - 1;
    const int ns = b.khi - b.klo + 1;
    int k = b.klo + (int)(((int64_t)ns * (ts + 1)) / nslabs) - 1;
    if (k > b.khi) k = b.khi;
    const int i = b.ihi, j = b.jhi;
    const double h = cfl_h_lanes<SCHEME, VAR>(b, phi, c, i, j, k, dx, dy, dz, inv);
    if (l == 0 && t < nslabs) hs[t] = h;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // max over slabs (the reference's critical section), -1 if none
    double cur = -1.0;
    for (int t = 0; t < nslabs; t++) cur = qss_emu::gt(hs[t], cur) ? hs[t] : cur;
    // loop condition of constCurvModel3d.c:127, evaluated before the step
    bool go = ctl->dt_sub < ctl->tplot;
    if (ctl->max_steps > 0 && ctl->steps >= ctl->max_steps) go = false;
    if (!go) {
      ctl->active = 0;
      return;
    }
    double dt = qss_emu::div(0.5, cur + ctl->b_max_over_dx + ctl->max_U_over_dx);
    ctl->cur_max_H = cur;
    ctl->dt = dt;
    ctl->dt_sub = ctl->dt_sub + dt;
    ctl->steps = ctl->steps + 1;
  }
}

// ---------------------------------------------------------------------------
// inner step: stage kernel (RHS fused with the TVD-RK combination and, for the
// last stage, with the three mask impositions)

struct StageArgs {
  Box b;
  Inv inv;
  Fac fac;
  const double* phi_in;
  const double* u_cur;
  double* out;
  double* phi_new;
  Coef c;
  ImposeArgs im;
  const Ctl* ctl;
  int walk;  // planes per block (k_eno2)
};

template <int SCHEME, bool VAR, int STAGE, bool FINAL>
__global__ void __launch_bounds__(128) k_stage(StageArgs a) {
  if (STAGE != 0 && !a.ctl->active) return;
  const Box& b = a.b;
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t idx = b.idx(i, j, k);
  const double* __restrict__ phi = a.phi_in;

  double pp[3], pm[3];
  upwind<SCHEME>(phi, b, i, j, k, a.inv, pp, pm);

  // Godunov normal term.  A voxel whose |vel_n| is below the tolerance keeps
  // the term of the closest preceding voxel of its slab (3d.f:459-486).
  const double vel = VAR ? a.c.vel_n[idx] : a.c.a_const;
  double temp_norm;
  if (fabs(vel) >= kZeroTol) {
    temp_norm = godunov_norm<SCHEME>(vel, pp, pm);
  } else if (VAR) {
    const int src = a.c.nsrc[idx];
    if (src < 0) {
      temp_norm = 0.0;
    } else {
      const int is = src % b.nx, js = (src / b.nx) % b.ny, ks = src / (b.nx * b.ny);
      double qp[3], qm[3];
      upwind<SCHEME>(phi, b, is, js, ks, a.inv, qp, qm);
      temp_norm = godunov_norm<SCHEME>(a.c.vel_n[src], qp, qm);
    }
  } else {
    temp_norm = 0.0;
  }

  double rhs;
  if (VAR) {
    const double vx = a.c.vx[idx], vy = a.c.vy[idx], vz = a.c.vz[idx];
    const double ax = (vx >= 0) ? pm[0] : pp[0];
    const double ay = (vy >= 0) ? pm[1] : pp[1];
    const double az = (vz >= 0) ? pm[2] : pp[2];
    const double temp_vel = -(vx * ax + vy * ay + vz * az);
    const double temp_curv = a.c.b[idx] * curvature(phi, b, idx, a.fac);
    rhs = temp_norm + temp_curv + temp_vel;
  } else {
    const double temp_curv = a.c.b_const * curvature(phi, b, idx, a.fac);
    rhs = temp_norm + temp_curv;
  }

  double out;
  if (STAGE == 0) {
    out = rhs;
  } else {
    const double dt = a.ctl->dt;
    if (STAGE == 1) {
      out = phi[idx] + dt * rhs;
    } else if (STAGE == 2) {
      out = 0.75 * a.u_cur[idx] + 0.25 * (phi[idx] + dt * rhs);
    } else {
      const double one_third = 1.0 / 3.0, two_thirds = 2.0 / 3.0;
      out = one_third * a.u_cur[idx] + two_thirds * (phi[idx] + dt * rhs);
    }
  }
  a.out[idx] = out;
  if (FINAL) a.phi_new[idx] = impose3(out, idx, a.im);
}

// ---------------------------------------------------------------------------
// ENO2 / ENO3 stage at EMU 2: the one-sided differences with native additions and
// integer comparisons, the rest as in qss_stage.cuh.  Blocks of four 8 x 4
// patches (see k_weno_combine).  Bound: FP64 pipe.  ENO2 with every voxel by itself
// takes 63 FP64 instructions a voxel, with the differences shared (k_eno2) 48; a step of
// constant coefficients on GB300 0.54 -> 0.48 ms at 128^3, 0.116 -> 0.109 ms at 64^3
// (two stages, ghost layers and the CFL step).  Walks of k_eno2 as long as
// kEno2Target blocks per SM allow: at 128^3 6 per SM 0.60 ms, 12 0.52, 18 to 40
// 0.48, 60 0.49; 7 or 8 resident blocks the same as 6.
constexpr int kEno2Blocks = 6, kEno2Target = 32, kEno2Walk = 16;

// |x| < |y| (false where y is NaN)
__device__ __forceinline__ bool abs_lt(double x, double y) {
  const uint64_t a = qss_emu::bits(x) << 1, b = qss_emu::bits(y) << 1;
  return a < b && b <= 0xffe0000000000000ull;
}

// eno3_pm without the scaling
__device__ __forceinline__ void eno3_raw(const double s[7], double& plus, double& minus) {
  using qss_emu::mul;
  using qss_emu::neg;
  using qss_emu::scale2;
  const double third = 1.0 / 3.0, sixth = 1.0 / 6.0;
  const double D1 = s[3] - s[2], D1p = s[4] - s[3], D1m = s[2] - s[1], D1mm = s[1] - s[0];
  const double D1pp = s[5] - s[4], D1ppp = s[6] - s[5];
  const double D2 = D1p - D1, D2p = D1pp - D1p, D2m = D1 - D1m, D2pp = D1ppp - D1pp, D2mm = D1m - D1mm;
  const double D3 = D2 - D2m, D3p = D2p - D2, D3pp = D2pp - D2p, D3m = D2m - D2mm;
  // p = D1p - D2* / 2, then -D3 / 6 where D2 was taken, + D3 / 3 where D2p was
  const bool l = abs_lt(D2, D2p);
  const double a = l ? D3 : D3p, b = l ? D3p : D3pp;
  const double tp = mul(l ? sixth : third, abs_lt(a, b) ? a : b);
  plus = (D1p - scale2(l ? D2 : D2p, -1)) + (l ? neg(tp) : tp);
  const bool m = abs_lt(D2m, D2);
  const double c = m ? D3m : D3, d = m ? D3 : D3p;
  const double tm = mul(m ? third : sixth, abs_lt(c, d) ? c : d);
  minus = (D1 + scale2(m ? D2m : D2, -1)) + (m ? tm : neg(tm));
}

// unscaled ENO3 one-sided differences of the three axes at (i, j, k)
__device__ __forceinline__ void eno3_axes(const double* __restrict__ phi, const Box& b, int i, int j, int64_t c,
                                          double pp[3], double pm[3]) {
  const int64_t st[3] = {1, b.sy(), b.sz()};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double s[7];
#pragma unroll
    for (int o = -3; o <= 3; o++) s[o + 3] = __ldg(phi + c + o * st[d]);
    if (d == 0) s[6] = __ldg(phi + b.idx(i + 3, j, j));  // 3d.f:677
    eno3_raw(s, pp[d], pm[d]);
  }
}

template <int SCHEME>
__device__ __noinline__ double carried_norm(const double* __restrict__ phi, const Box& b, int src, const Inv& inv,
                                            const double* __restrict__ vel_n) {
  const int is = src % b.nx, js = (src / b.nx) % b.ny, ks = src / (b.nx * b.ny);
  double qp[3], qm[3];
  upwind<SCHEME>(phi, b, is, js, ks, inv, qp, qm);
  return godunov_norm<SCHEME>(vel_n[src], qp, qm);
}

// the rest of a stage at one voxel from its unscaled one-sided differences
template <int SCHEME, bool VAR, int STAGE, bool FINAL, bool INT>
__device__ __forceinline__ void eno_finish(const StageArgs& a, int64_t idx, const double pp[3], const double pm[3]) {
  const Box& b = a.b;
  const double* __restrict__ phi = a.phi_in;
  const double vel = VAR ? a.c.vel_n[idx] : a.c.a_const;
  double rhs = 0.0;
  if (speed_valid(vel)) {
    rhs = godunov_fast<SCHEME, true, INT>(vel, pp, pm, a.inv);
  } else if (VAR) {
    // a voxel at rest keeps the term of the closest preceding voxel of its slab
    const int src = a.c.nsrc[idx];
    if (src >= 0) rhs = carried_norm<SCHEME>(phi, b, src, a.inv, a.c.vel_n);
  }
  const double bco = VAR ? a.c.b[idx] : a.c.b_const;
  // b * kappa is +-0 where b is +0 and kappa finite, and changes no term but -0
  if (!VAR || qss_emu::bits(bco) != 0 || qss_emu::bits(rhs) == qss_emu::kSign || !curvature_finite(phi, b, idx))
    rhs = rhs + qss_emu::mul(bco, curvature_fast<INT, SCHEME == ENO2>(phi, b, idx, a.fac));
  if (VAR) rhs = add_advection<true>(rhs, a.c.vx[idx], a.c.vy[idx], a.c.vz[idx], pp, pm, a.inv);
  const double out = rk_combine<STAGE>(rhs, STAGE ? a.ctl->dt : 0.0, STAGE ? __ldg(phi + idx) : 0.0, a.u_cur, idx);
  a.out[idx] = out;
  if (FINAL) a.phi_new[idx] = impose3_i(out, idx, a.im);
}

template <bool VAR, int STAGE, bool FINAL>
__global__ void __launch_bounds__(128, 6) k_eno3(StageArgs a) {
  if (STAGE != 0 && !a.ctl->active) return;
  const Box& b = a.b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = b.ilo + blockIdx.x * 32 + 8 * warp + (lane & 7);
  const int j = b.jlo + blockIdx.y * 4 + (lane >> 3);
  const int k = b.klo + blockIdx.z;
  if (i > b.ihi || j > b.jhi) return;
  const int64_t idx = b.idx(i, j, k);
  double pp[3], pm[3];
  eno3_axes(a.phi_in, b, i, j, idx, pp, pm);
  eno_finish<ENO3, VAR, STAGE, FINAL, false>(a, idx, pp, pm);
}

// ENO2 with each difference computed once.  On an axis, with d1(v) = phi(v + 1) -
// phi(v), d2(v) = phi(v + 1) + phi(v - 1) - 2 phi(v) and m(v) the smaller of d2(v)
// and d2(v + 1) in magnitude, the plus difference of v is d1(v) - m(v) / 2 and the
// minus difference d1(v - 1) + m(v - 1) / 2: three FP64 instructions for d1 and d2
// and two for the sums, against ten for a voxel by itself.  A warp owns an 8 x 4
// patch (x neighbours one lane apart, y neighbours eight) and walks `walk` planes
// along k with the z terms carried; d2 outside the patch's four edges, and d1 below
// the two low ones, is one more evaluation by 24 of the lanes.  The sums of squares
// go over the integer pipes, which have the time.
template <bool VAR, int STAGE, bool FINAL>
__global__ void __launch_bounds__(128, kEno2Blocks) k_eno2(StageArgs a) {
  using qss_emu::scale2;
  if (STAGE != 0 && !a.ctl->active) return;
  const Box& b = a.b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int li = lane & 7, lj = lane >> 3;
  const int i0 = b.ilo + blockIdx.x * 32 + 8 * warp, j0 = b.jlo + blockIdx.y * 4;
  if (i0 > b.ihi) return;  // the whole warp
  // lanes past the fill box work on its last row / column and store nothing
  const int lx = min(7, b.ihi - i0), ly = min(3, b.jhi - j0);
  const bool ok = li <= lx && lj <= ly;
  const int k0 = b.klo + blockIdx.z * a.walk, k1 = min(k0 + a.walk - 1, b.khi);
  const int64_t sy = b.sy(), sz = b.sz();
  const double* __restrict__ phi = a.phi_in;
  int64_t c = b.idx(i0 + min(li, lx), j0 + min(lj, ly), k0);
  // the lane's voxel outside the patch: below (0 - 7) and above (8 - 15) in y, below
  // (16 - 19) and above (20 - 23) in x; its own for the rest
  const bool ey = lane < 16;
  const int er = min(lane & 3, ly);
  const int64_t e0 = ey ? b.idx(i0 + min(li, lx), lane < 8 ? j0 - 1 : j0 + ly + 1, k0)
                        : (lane < 24 ? b.idx(lane < 20 ? i0 - 1 : i0 + lx + 1, j0 + er, k0) : c);
  const int64_t eo = e0 - c, es = ey ? sy : 1;
  // an FMA does not overflow in 2 mid: where that is infinite (2^1023 and more), mid is made so
  auto d2_of = [](double lo, double mid, double hi) {
    const uint32_t h = qss_emu::hi32(mid);
    const bool over = (h & 0x7ff00000u) == 0x7fe00000u;
    const double m = __hiloint2double((int)(over ? (h & 0x80000000u) | 0x7ff00000u : h), (int)(over ? 0u : qss_emu::lo32(mid)));
    return __fma_rn(-2.0, m, hi + lo);
  };
  auto pick = [](double x, double y) { return abs_lt(x, y) ? x : y; };
  auto from = [](double v, int src) { return __shfl_sync(0xffffffffu, v, src); };
  double cc = __ldg(phi + c), zp = __ldg(phi + c + sz), d2z, d1zl, mzl;
  {
    const double zm = __ldg(phi + c - sz);
    d1zl = cc - zm;
    d2z = d2_of(zm, cc, zp);
    mzl = pick(d2_of(__ldg(phi + c - 2 * sz), zm, cc), d2z);
  }
  for (int k = k0; k <= k1; k++) {
    const double xp = __ldg(phi + c + 1), xm = __ldg(phi + c - 1), yp = __ldg(phi + c + sy), ym = __ldg(phi + c - sy);
    const double em = __ldg(phi + c + eo - es), ec = __ldg(phi + c + eo), ep = __ldg(phi + c + eo + es);
    const double zpp = __ldg(phi + c + 2 * sz);
    const double d1e = ep - ec, d2e = d2_of(em, ec, ep);
    const double d1x = xp - cc, d1y = yp - cc, d1z = zp - cc;
    const double d2x = d2_of(xm, cc, xp), d2y = d2_of(ym, cc, yp), d2zp = d2_of(cc, zp, zpp);
    double up = __shfl_down_sync(0xffffffffu, d2x, 1), edge = from(d2e, 20 + lj);
    const double mx = pick(d2x, li >= lx ? edge : up);
    up = __shfl_down_sync(0xffffffffu, d2y, 8);
    edge = from(d2e, 8 + li);
    const double my = pick(d2y, lj >= ly ? edge : up);
    const double mz = pick(d2z, d2zp);
    double mxl = __shfl_up_sync(0xffffffffu, mx, 1), d1xl = __shfl_up_sync(0xffffffffu, d1x, 1);
    edge = from(d2e, 16 + lj);
    double d1 = from(d1e, 16 + lj);
    if (li == 0) {
      mxl = pick(edge, d2x);
      d1xl = d1;
    }
    double myl = __shfl_up_sync(0xffffffffu, my, 8), d1yl = __shfl_up_sync(0xffffffffu, d1y, 8);
    edge = from(d2e, li);
    d1 = from(d1e, li);
    if (lj == 0) {
      myl = pick(edge, d2y);
      d1yl = d1;
    }
    const double pp[3] = {d1x - scale2(mx, -1), d1y - scale2(my, -1), d1z - scale2(mz, -1)};
    const double pm[3] = {d1xl + scale2(mxl, -1), d1yl + scale2(myl, -1), d1zl + scale2(mzl, -1)};
    if (ok) eno_finish<ENO2, VAR, STAGE, FINAL, true>(a, c, pp, pm);
    d1zl = d1z;
    mzl = mz;
    d2z = d2zp;
    cc = zp;
    zp = zpp;
    c += sz;
  }
}

template <int SCHEME, bool VAR>
__global__ void k_cfl_at(Box b, const double* __restrict__ phi, Coef c, int i, int j, int k, double dx,
                         double dy, double dz, Inv inv, double* h_out) {
  const double h = cfl_h_lanes<SCHEME, VAR>(b, phi, c, i, j, k, dx, dy, dz, inv);
  if (threadIdx.x == 0) *h_out = h;
}

// ---------------------------------------------------------------------------
// ghost layers

// bc_xyz() of qss_device.cuh for a warp's points at once: each axis has the nearest
// fill-box index f, the one behind it g and the distance d (0 inside).  The axes
// some lane of the warp lies outside of are found by votes, all loads they need
// are issued together, then the extrapolations follow x, y, z.  (Point by point
// with branches the loads came one after the other: 8 us at 24^3.)  32-bit
// indices: the ghost box is below 2^31 points.
struct GhostAxis {
  int f, g, d;
};
__device__ __forceinline__ GhostAxis ghost_axis(int i, int lo, int hi) {
  if (i < lo) return GhostAxis{lo, lo + 1, lo - i};
  if (i > hi) return GhostAxis{hi, hi - 1, i - hi};
  return GhostAxis{i, i, 0};
}
__device__ __forceinline__ double extrap_if(double f, double g, int d) { return d ? extrap(f, g, d) : f; }

__global__ void __launch_bounds__(256) k_ghost(Box b, double* a, double* phi_new, ImposeArgs im, const Ctl* ctl) {
  if (ctl && !ctl->active) return;
  const uint32_t nx = b.nx, nxy = (uint32_t)b.nx * b.ny;
  const uint32_t nzg = b.klo + (b.nz - 1 - b.khi);  // z-ghost planes
  const uint32_t nyg = b.jlo + (b.ny - 1 - b.jhi);  // y-ghost rows per plane
  const uint32_t nxg = b.ilo + (b.nx - 1 - b.ihi);  // x-ghost points per row
  const uint32_t nz_cells = nzg * nxy;
  const uint32_t ny_cells = b.fbz() * nyg * nx;
  const uint32_t total = nz_cells + ny_cells + (uint32_t)b.fbz() * b.fby() * nxg;
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t q0 = blockIdx.x * blockDim.x + threadIdx.x - lane; q0 < total; q0 += gridDim.x * blockDim.x) {
    // lanes past the end repeat the last point and store nothing
    const uint32_t q = q0 + lane < total ? q0 + lane : total - 1;
    int i, j, k;
    if (q < nz_cells) {
      const uint32_t row = q / nx, p = row / (uint32_t)b.ny;
      i = (int)(q - row * nx);
      j = (int)(row - p * b.ny);
      k = (int)p < b.klo ? (int)p : b.khi + 1 + ((int)p - b.klo);
    } else if (q < nz_cells + ny_cells) {
      const uint32_t r = q - nz_cells, row = r / nx, pl = row / nyg;
      const int p = (int)(row - pl * nyg);
      i = (int)(r - row * nx);
      k = b.klo + (int)pl;
      j = p < b.jlo ? p : b.jhi + 1 + (p - b.jlo);
    } else {
      const uint32_t r = q - nz_cells - ny_cells, row = r / nxg, pl = row / (uint32_t)b.fby();
      const int p = (int)(r - row * nxg);
      k = b.klo + (int)pl;
      j = b.jlo + (int)(row - pl * b.fby());
      i = p < b.ilo ? p : b.ihi + 1 + (p - b.ilo);
    }
    const GhostAxis x = ghost_axis(i, b.ilo, b.ihi), y = ghost_axis(j, b.jlo, b.jhi), z = ghost_axis(k, b.klo, b.khi);
    const bool ox = __any_sync(0xffffffffu, x.d), oy = __any_sync(0xffffffffu, y.d), oz = __any_sync(0xffffffffu, z.d);
    double v[2][2][2];  // z, y, x: f, g
#pragma unroll
    for (int m = 0; m < 8; m++) {
      const bool gx = m & 1, gy = m & 2, gz = m & 4;
      if ((!gx || ox) && (!gy || oy) && (!gz || oz))
        v[gz][gy][gx] = a[b.idx(gx ? x.g : x.f, gy ? y.g : y.f, gz ? z.g : z.f)];
    }
#pragma unroll
    for (int gz = 0; gz < 2; gz++) {
      if (gz && !oz) break;
#pragma unroll
      for (int gy = 0; gy < 2; gy++)
        if ((!gy || oy) && ox) v[gz][gy][0] = extrap_if(v[gz][gy][0], v[gz][gy][1], x.d);
      if (oy) v[gz][0][0] = extrap_if(v[gz][0][0], v[gz][1][0], y.d);
    }
    const double r = oz ? extrap_if(v[0][0][0], v[1][0][0], z.d) : v[0][0][0];
    if (q0 + lane < total) {
      const int64_t idx = b.idx(i, j, k);
      a[idx] = r;
      if (phi_new && k >= b.klo - 3 && k <= b.khi + 3) phi_new[idx] = impose3_i(r, idx, im);
    }
  }
}

__global__ void k_face(Box b, double* a, int face) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (face < 2) {  // lines over (j,k)
    if (t >= b.ny * b.nz) return;
    const int j = t % b.ny, k = t / b.ny;
    const int f = face == 0 ? b.ilo : b.ihi, g = face == 0 ? b.ilo + 1 : b.ihi - 1;
    const double vf = a[b.idx(f, j, k)], vg = a[b.idx(g, j, k)];
    if (face == 0)
      for (int i = 0; i < b.ilo; i++) a[b.idx(i, j, k)] = extrap(vf, vg, b.ilo - i);
    else
      for (int i = b.ihi + 1; i < b.nx; i++) a[b.idx(i, j, k)] = extrap(vf, vg, i - b.ihi);
  } else if (face < 4) {  // lines over (i,k)
    if (t >= b.nx * b.nz) return;
    const int i = t % b.nx, k = t / b.nx;
    const int f = face == 2 ? b.jlo : b.jhi, g = face == 2 ? b.jlo + 1 : b.jhi - 1;
    const double vf = a[b.idx(i, f, k)], vg = a[b.idx(i, g, k)];
    if (face == 2)
      for (int j = 0; j < b.jlo; j++) a[b.idx(i, j, k)] = extrap(vf, vg, b.jlo - j);
    else
      for (int j = b.jhi + 1; j < b.ny; j++) a[b.idx(i, j, k)] = extrap(vf, vg, j - b.jhi);
  } else {  // lines over (i,j)
    if (t >= b.nx * b.ny) return;
    const int i = t % b.nx, j = t / b.nx;
    const int f = face == 4 ? b.klo : b.khi, g = face == 4 ? b.klo + 1 : b.khi - 1;
    const double vf = a[b.idx(i, j, f)], vg = a[b.idx(i, j, g)];
    if (face == 4)
      for (int k = 0; k < b.klo; k++) a[b.idx(i, j, k)] = extrap(vf, vg, b.klo - k);
    else
      for (int k = b.khi + 1; k < b.nz; k++) a[b.idx(i, j, k)] = extrap(vf, vg, k - b.khi);
  }
}

__global__ void k_impose_region(Box b, const double* src, double* phi_new, ImposeArgs im, const Ctl* ctl) {
  if (ctl && !ctl->active) return;
  int k0 = b.klo - 3 < 0 ? 0 : b.klo - 3;
  int k1 = b.khi + 3 > b.nz - 1 ? b.nz - 1 : b.khi + 3;
  const int64_t nxy = (int64_t)b.nx * b.ny;
  const int64_t total = (int64_t)(k1 - k0 + 1) * nxy;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
       q += (int64_t)gridDim.x * blockDim.x) {
    int64_t idx = (int64_t)k0 * nxy + q;
    phi_new[idx] = impose3(src[idx], idx, im);
  }
}

// ---------------------------------------------------------------------------
// F8 source map: rows are (j,k) lines of the fill box in loop order

// One warp per row: 32 voxels at a time, the valid ones found by a ballot.  (A
// thread per row read its row alone: 39 us for the fill at 130 x 96 x 75.)
__global__ void k_nsrc_rowlast(Box b, const double* __restrict__ vel, int* rowlast) {
  const int lane = threadIdx.x & 31;
  const int64_t nrows = (int64_t)b.fby() * b.fbz();
  const int64_t r = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= nrows) return;
  const int j = b.jlo + (int)(r % b.fby()), k = b.klo + (int)(r / b.fby());
  const int64_t row = b.idx(b.ilo, j, k);
  int last = -1;
  for (int i0 = (b.fbx() - 1) & ~31; i0 >= 0; i0 -= 32) {
    const bool valid = i0 + lane < b.fbx() && speed_valid(vel[row + i0 + lane]);
    const unsigned m = __ballot_sync(0xffffffffu, valid);
    if (m) {
      last = (int)(row + i0) + 31 - __clz(m);
      break;
    }
  }
  if (lane == 0) rowlast[r] = last;
}

// one block per slab: exclusive running max of rowlast over the slab's rows
__global__ void __launch_bounds__(1024) k_nsrc_carry(Box b, int nslabs, const int* rowlast, int* carry) {
  __shared__ int part[32];
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ns = b.khi - b.klo + 1;
  const int k0 = b.klo + (int)(((int64_t)ns * t) / nslabs);
  int k1 = b.klo + (int)(((int64_t)ns * (t + 1)) / nslabs) - 1;
  if (k1 > b.khi) k1 = b.khi;
  const int64_t r0 = (int64_t)(k0 - b.klo) * b.fby();
  const int64_t r1 = (int64_t)(k1 - b.klo + 1) * b.fby();  // exclusive
  int run = -1;  // over the rows before this round's
  for (int64_t base = r0; base < r1; base += 1024) {
    const int64_t r = base + threadIdx.x;
    const int v = r < r1 ? rowlast[r] : -1;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl = max(incl, x);
    }
    if (lane == 31) part[warp] = incl;
    int excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = -1;
    __syncthreads();
    int all = run;
    for (int w = 0; w < 32; w++) {
      if (w < warp) excl = max(excl, part[w]);
      all = max(all, part[w]);
    }
    if (r < r1) carry[r] = max(run, excl);
    run = all;
    __syncthreads();
  }
}

__global__ void k_nsrc_fill(Box b, const double* __restrict__ vel, const int* carry, int* nsrc,
                            unsigned long long* count) {
  const int lane = threadIdx.x & 31;
  const int64_t nrows = (int64_t)b.fby() * b.fbz();
  const int64_t r = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= nrows) return;
  const int j = b.jlo + (int)(r % b.fby()), k = b.klo + (int)(r / b.fby());
  const int64_t row = b.idx(b.ilo, j, k);
  int cur = carry[r], invalid = 0;
  for (int i0 = 0; i0 < b.fbx(); i0 += 32) {
    const bool in = i0 + lane < b.fbx();
    const bool valid = in && speed_valid(vel[row + i0 + lane]);
    const unsigned m = __ballot_sync(0xffffffffu, valid);
    const unsigned before = m & ((1u << lane) - 1u);
    if (in) nsrc[row + i0 + lane] = valid ? -1 : (before ? (int)(row + i0) + 31 - __clz(before) : cur);
    invalid += __popc(__ballot_sync(0xffffffffu, in && !valid));
    if (m) cur = (int)(row + i0) + 31 - __clz(m);
  }
  if (lane == 0 && invalid) atomicAdd(count, (unsigned long long)invalid);
}

// ---------------------------------------------------------------------------
// reinitialisation (src/reinitialization/qss_reinitialization3d.f:476-746)

// distance0 of a voxel with a neighbour n (x+, x-, y+, y-, z+, z-) across the interface
__device__ __noinline__ double distance0_native(double cc, const double n[6]) {
  double delta = 1.e-5;
#pragma unroll
  for (int q = 0; q < 6; q += 2) {
    const double d1 = fabs(n[q] - n[q + 1]) / 2.0, d2 = fabs(n[q] - cc), d3 = fabs(cc - n[q + 1]);
    delta = dmax(dmax(dmax(d1, d2), d3), delta);
  }
  return cc / delta;
}

// Away from the interface the distance is one constant, and the tests that say so run
// on the integer pipes (a native comparison occupies the FP64 pipe like an addition).
// The voxels next to it, ~10 % but some in most warps of a sphere pack, are gathered
// per block of kNearVoxels and evaluated by full warps: 200^3, 746 us with every warp
// evaluating its own.
constexpr int kNearVoxels = 1024, kNearThreads = 256;

__global__ void __launch_bounds__(kNearThreads) k_distance0(Box b, const double* __restrict__ phi0, double* distance0,
                                                            double max_dx) {
  using namespace qss_emu;
  __shared__ uint16_t near_t[kNearVoxels];
  __shared__ int near_n;
  const FillBlock blk(b, blockIdx.x, kNearVoxels);
  const int64_t st[6] = {1, -1, b.sy(), -b.sy(), b.sz(), -b.sz()};
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) near_n = 0;
  __syncthreads();
  for (int t0 = 0; t0 < kNearVoxels; t0 += kNearThreads) {
    const uint32_t t = t0 + threadIdx.x;
    bool near = false;
    if (blk.in(t)) {
      const int64_t c = blk.at(b, t);
      const double cc = phi0[c];
      // opposite signs, zero counted as negative
      const bool pos = gt0(cc), nonpos = lt0(cc) || mag2(bits(cc)) == 0;
#pragma unroll
      for (int q = 0; q < 6; q++) {
        const double v = phi0[c + st[q]];
        const bool np = gt0(v);
        near = near || (np && nonpos) || (!np && pos && !isnan_bits(bits(v)));
      }
      if (!near) distance0[c] = max_dx * -1000.0;
    }
    const unsigned vote = __ballot_sync(0xffffffffu, near);
    int slot = 0;
    if (lane == 0 && vote) slot = atomicAdd(&near_n, __popc(vote));
    slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(vote & ((1u << lane) - 1u));
    if (near) near_t[slot] = (uint16_t)t;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < near_n; e += kNearThreads) {
    const int64_t c = blk.at(b, near_t[e]);
    const double cc = phi0[c];
    double v[6];
    uint64_t top = mag2(bits(cc));
#pragma unroll
    for (int q = 0; q < 6; q++) {
      v[q] = phi0[c + st[q]];
      const uint64_t m = mag2(bits(v[q]));
      top = m > top ? m : top;
    }
    double r;
    if (top < (0x5fe0000000000000ull << 1)) {  // below 2^511: every difference finite
      // magnitudes order like their bits
      uint64_t delta = bits(1.e-5);
#pragma unroll
      for (int q = 0; q < 6; q += 2) {
        const uint64_t d1 = mag2(bits(scale2(v[q] - v[q + 1], -1))) >> 1, d2 = mag2(bits(v[q] - cc)) >> 1,
                       d3 = mag2(bits(cc - v[q + 1])) >> 1;
        delta = max(max(max(d1, d2), d3), delta);
      }
      r = div(cc, from_bits(delta));
    } else {
      r = distance0_native(cc, v);
    }
    distance0[c] = r;
  }
}

__device__ __forceinline__ double reinit_rhs_at(const double* __restrict__ phi, const double* __restrict__ phi0,
                                                const double* __restrict__ distance0, const Box& b, int64_t c,
                                                const Inv& inv, double max_dx) {
  const double zero_tol = 1.e-5;
  const int64_t sy = b.sy(), sz = b.sz();
  const double cc = __ldg(phi + c);
  double gp[3], gm[3];
  gp[0] = (__ldg(phi + c + 1) - cc) * inv.x;
  gm[0] = (cc - __ldg(phi + c - 1)) * inv.x;
  gp[1] = (__ldg(phi + c + sy) - cc) * inv.y;
  gm[1] = (cc - __ldg(phi + c - sy)) * inv.y;
  gp[2] = (__ldg(phi + c + sz) - cc) * inv.z;
  gm[2] = (cc - __ldg(phi + c - sz)) * inv.z;
  const double p0 = phi0[c];
  const double sgn = (fabs(p0) > zero_tol) ? copysign(1.0, p0) : 0.0;
  const double d0 = distance0[c];
  if (d0 == -1000.0 * max_dx) {
    double gs[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double a_, b_;
      if (cc > 0.0) {
        a_ = dmax(-gp[d], 0.0);
        b_ = dmax(gm[d], 0.0);
      } else {
        a_ = dmax(gp[d], 0.0);
        b_ = dmax(-gm[d], 0.0);
      }
      gs[d] = dmax(a_, b_);
    }
    if (fabs(cc) > zero_tol) {
      double ngps = gs[0] * gs[0] + gs[1] * gs[1] + gs[2] * gs[2];
      return sgn - sgn * sqrt(ngps);
    }
    return 0.0;
  }
  return d0 - sgn * fabs(cc) / max_dx;
}

// The same right-hand side with the sign tests, maxima, absolute values, the
// square root and the division on the integer pipes (qss_emu: IEEE results,
// bit for bit), leaving ~20 FP64 instructions per voxel; at EMU >= 2 the six
// scalings of the one-sided differences move there too.  Every branch
// computes exactly the native version's value:
//   dmax(-g, 0) = (g < 0 ? -g : +0) and dmax(g, 0) = (g > 0 ? g : +0) (only
//   their squares are used, so the sign of a zero does not matter);
//   sgn * s for sgn = +-1 is a sign flip; sgn = 0 keeps the native product.
template <int EMU>
__device__ __forceinline__ double reinit_rhs_e(const double* __restrict__ phi, const double* __restrict__ phi0,
                                               const double* __restrict__ distance0, const Box& b, int64_t c,
                                               const Inv& inv, double max_dx, uint64_t far_bits) {
  using namespace qss_emu;
  const uint64_t tol2 = mag2(bits(1.e-5));
  const int64_t sy = b.sy(), sz = b.sz();
  auto scale = [](double d, double f) -> double { return EMU >= 2 ? qss_emu::mul(d, f) : d * f; };
  const double cc = __ldg(phi + c);
  const double p0 = phi0[c];
  const uint64_t ap0 = mag2(bits(p0));
  const bool sgn_nz = ap0 > tol2 && ap0 <= kInf2;  // fabs(p0) > 1e-5
  const bool sgn_neg = (int64_t)bits(p0) < 0;
  const double sgn = sgn_nz ? (sgn_neg ? -1.0 : 1.0) : 0.0;
  const double d0 = distance0[c];
  if (bits(d0) == far_bits) {
    const bool pos = gt0(cc);
    double gs[3];
    const int64_t st[3] = {1, sy, sz};
    const double iv[3] = {inv.x, inv.y, inv.z};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double gp = scale(__ldg(phi + c + st[d]) - cc, iv[d]);
      const double gm = scale(cc - __ldg(phi + c - st[d]), iv[d]);
      double a_, b_;
      if (pos) {
        a_ = lt0(gp) ? qss_emu::neg(gp) : 0.0;
        b_ = gt0(gm) ? gm : 0.0;
      } else {
        a_ = gt0(gp) ? gp : 0.0;
        b_ = lt0(gm) ? qss_emu::neg(gm) : 0.0;
      }
      gs[d] = max_nonneg(a_, b_);
    }
    const uint64_t acc = mag2(bits(cc));
    if (acc > tol2 && acc <= kInf2) {  // fabs(cc) > 1e-5
      const double ngps = scale(gs[0], gs[0]) + scale(gs[1], gs[1]) + scale(gs[2], gs[2]);
      const double s = qss_emu::sqrt(ngps);
      if (!sgn_nz) return sgn - sgn * s;
      return sgn - (sgn_neg ? qss_emu::neg(s) : s);
    }
    return 0.0;
  }
  // d0 - sgn * fabs(cc) / max_dx
  const double acc = qss_emu::abs(cc);
  const double t = sgn_nz ? (sgn_neg ? qss_emu::neg(acc) : acc) : sgn * acc;
  return d0 - qss_emu::div(t, max_dx);
}

// The reinitialisation right-hand side of one voxel from its six scaled
// one-sided differences gp[d] = (phi(c + e_d) - phi(c)) inv_d and
// gm[d] = (phi(c) - phi(c - e_d)) inv_d, with the operations of reinit_rhs_e.
__device__ __forceinline__ double reinit_rhs_diffs(double cc, double p0, double d0, const double gp[3],
                                                   const double gm[3], double max_dx, uint64_t far_bits) {
  using namespace qss_emu;
  const uint64_t tol2 = mag2(bits(1.e-5));
  auto scale = [](double d, double f) -> double { return qss_emu::mul(d, f); };
  const uint64_t ap0 = mag2(bits(p0));
  const bool sgn_nz = ap0 > tol2 && ap0 <= kInf2;  // fabs(p0) > 1e-5
  const bool sgn_neg = (int64_t)bits(p0) < 0;
  const double sgn = sgn_nz ? (sgn_neg ? -1.0 : 1.0) : 0.0;
  if (bits(d0) == far_bits) {
    const bool pos = gt0(cc);
    double gs[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double a_, b_;
      if (pos) {
        a_ = lt0(gp[d]) ? qss_emu::neg(gp[d]) : 0.0;
        b_ = gt0(gm[d]) ? gm[d] : 0.0;
      } else {
        a_ = gt0(gp[d]) ? gp[d] : 0.0;
        b_ = lt0(gm[d]) ? qss_emu::neg(gm[d]) : 0.0;
      }
      gs[d] = max_nonneg(a_, b_);
    }
    const uint64_t acc = mag2(bits(cc));
    if (acc > tol2 && acc <= kInf2) {  // fabs(cc) > 1e-5
      const double ngps = scale(gs[0], gs[0]) + scale(gs[1], gs[1]) + scale(gs[2], gs[2]);
      const double s = qss_emu::sqrt(ngps);
      if (!sgn_nz) return sgn - sgn * s;
      return sgn - (sgn_neg ? qss_emu::neg(s) : s);
    }
    return 0.0;
  }
  const double acc = qss_emu::abs(cc);
  const double t = sgn_nz ? (sgn_neg ? qss_emu::neg(acc) : acc) : sgn * acc;
  return d0 - qss_emu::div(t, max_dx);
}

// Reinitialisation step at level 2 with each face difference computed once:
// the difference phi(c + e) - phi(c) is the plus difference of c and the
// minus difference of c + e, the same operation on the same operands.  A block
// of 4 warps covers 32 (i) x 4 (j) voxels, each warp an 8 x 4 patch (x
// neighbours one lane apart, y neighbours eight), and walks `walk` planes
// along k carrying the z difference.  The 12 minus differences across the
// patch's low edges are one more instruction: the 4 lanes of the low x edge
// but the corner compute theirs in x, the 8 of the low y edge theirs in y, and
// lane 9 the corner's in x.  Short walks keep small boxes' grids large enough
// to fill the GPU (see reinit_walk_launch).
//
// Away from the interface the arithmetic is straight-line: the larger
// one-sided difference is picked before it is scaled (rounding is monotone),
// picked, cut off at zero and raised to 2^-255 by one integer maximum on its
// high word, and scaled, squared and rooted on the integer pipes without a
// test per operation.  The floor of 2^-255 in place of a zero changes no bit:
// the root it could reach is below 2^-100, and sgn - root, and phi + dt r,
// round to the same number.  Differences of 2^100 or more (infinities and
// NaNs among them) take the general path, reinit_rhs_diffs.  A voxel next to
// the interface differs in two operands only, d0 - |phi| / max_dx in place of
// sgn - root, so it shares the subtraction and the update; the reciprocal of
// max_dx is computed once per thread.  (Sent through the general path, the ~10 %
// of a sphere pack's voxels that lie there cost most warps a second set of FP64
// instructions: 200^3, 311 us a sweep against 185.)
//
// FP64 instructions per voxel: 3 differences and the edges', 2 sums,
// sgn - root, phi + dt r; they take 616 cycles of the ~720 the sweep takes per
// warp and plane, and with one or both sums moved to the integer pipes it is
// 1 and 5 % slower.
//
// GHOST: the layer next to the fill box is not read but extrapolated from the
// two voxels inside it (extrap with distance 1, as k_ghost would leave it), so
// the ghost layers need filling only after the last sweep.
constexpr int kRWalkMax = 16;
constexpr int kReinitFields = 2;

struct ReinitSweep {
  const double* data[kReinitFields];
  const double* phi0[kReinitFields];
  const double* dist[kReinitFields];
  double* next[kReinitFields];
  double dt_r, max_dx;
  Inv inv;
  uint64_t far_bits;
  int walk, chunks, rhs_only;
};

// f + sign(f) |f - g|: extrap(f, g, 1).  Out of line: inlined, its additions
// would be issued under a predicate by every warp, and an FP64 instruction
// with no active lane still takes its turn on the pipe.
__device__ __noinline__ double extrap1(double f, double g) {
  const uint32_t d = qss_emu::hi32(f - g), low = qss_emu::lo32(f - g);
  return f + __hiloint2double((int)((d & 0x7fffffffu) | (qss_emu::hi32(f) & 0x80000000u)), (int)low);
}

__device__ __noinline__ double reinit_general(double cc, double p0, double d0, double px, double py, double pz,
                                              double mx, double my, double mz, Inv inv, double max_dx,
                                              uint64_t far_bits) {
  const double gp[3] = {px * inv.x, py * inv.y, pz * inv.z}, gm[3] = {mx * inv.x, my * inv.y, mz * inv.z};
  return reinit_rhs_diffs(cc, p0, d0, gp, gm, max_dx, far_bits);
}

template <bool GHOST>
__global__ void __launch_bounds__(128, 10) k_reinit_walk(Box b, ReinitSweep a) {
  using namespace qss_emu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int li = lane & 7, lj = lane >> 3;
  const int field = blockIdx.z / a.chunks, chunk = blockIdx.z - field * a.chunks;
  const double* __restrict__ data = a.data[field];
  const int i0 = b.ilo + blockIdx.x * 32 + 8 * warp, j0 = b.jlo + blockIdx.y * 4;
  if (i0 > b.ihi) return;  // the whole warp
  const bool ok = i0 + li <= b.ihi && j0 + lj <= b.jhi;
  // lanes past the fill box work on its last row/column (in the box), store nothing
  const int i = i0 + li <= b.ihi ? i0 + li : b.ihi;
  const int j = j0 + lj <= b.jhi ? j0 + lj : b.jhi;
  const int k0 = b.klo + chunk * a.walk;
  const int k1 = k0 + a.walk - 1 < b.khi ? k0 + a.walk - 1 : b.khi;
  const int64_t sy = b.sy(), sz = b.sz();
  const Inv inv = a.inv;
  const uint32_t dxh = hi32(a.max_dx), dxl = lo32(a.max_dx);
  bool seed_ok = true;
  const uint32_t dx_recip = recip30(mant_hi(dxh), dxl, seed_ok);
  int64_t c = b.idx(i, j, k0);
  // the lane's share of the low edges: a neighbour's offset from c, and whether
  // that neighbour lies in the ghost layer
  const bool edge_y = lj == 0, edge_x = li == 0 && lj != 0, corner_x = lane == 9;
  const bool edge = edge_y || edge_x || corner_x;
  const int64_t ec = corner_x ? b.idx(i0, j0, k0) - 1 - c : (edge_y ? -sy : -1);
  const bool edge_ghost = GHOST && ((edge_y && j0 == b.jlo) || ((edge_x || corner_x) && i0 == b.ilo));
  const bool xlast = GHOST && i == b.ihi, ylast = GHOST && j == b.jhi;
  double cc = __ldg(data + c);
  double zm;
  if (GHOST && k0 == b.klo) zm = extrap1(cc, __ldg(data + c + sz));
  else zm = __ldg(data + c - sz);
  double dzm = cc - zm;
  for (int k = k0; k <= k1; k++) {
    double xp = __ldg(data + c + (xlast ? -1 : 1)), yp = __ldg(data + c + (ylast ? -sy : sy));
    double zp = __ldg(data + c + (GHOST && k == b.khi ? -sz : sz));
    const double cc0 = __shfl_sync(0xffffffffu, cc, 0);
    const double eb = corner_x ? cc0 : cc;
    double em = edge ? __ldg(data + c + ec) : eb;
    if (GHOST) {
      if (xlast) xp = extrap1(cc, xp);
      if (ylast) yp = extrap1(cc, yp);
      if (k == b.khi) zp = extrap1(cc, zp);
      if (i0 == b.ilo || j0 == b.jlo) {  // warp-uniform
        const double xp0 = __shfl_sync(0xffffffffu, xp, 0);
        if (edge_ghost) em = extrap1(eb, corner_x ? xp0 : (edge_y ? yp : xp));
      }
    }
    const double dxp = xp - cc, dyp = yp - cc, dzp = zp - cc, de = eb - em;
    const double xm = __shfl_up_sync(0xffffffffu, dxp, 1);
    const double ym = __shfl_up_sync(0xffffffffu, dyp, 8);
    const double dc = __shfl_sync(0xffffffffu, de, 9);
    const double dxm = li != 0 ? xm : (lj != 0 ? de : dc);
    const double dym = lj != 0 ? ym : de;
    if (ok) {
      const double p0 = __ldg(a.phi0[field] + c), d0 = __ldg(a.dist[field] + c);
      // max(-d+, d-, 0) where phi > 0, max(d+, -d-, 0) elsewhere, as signed
      // 64-bit integers (a negative double is a negative integer)
      const uint64_t sp = gt0(cc) ? kSign : 0, sm = sp ^ kSign;
      const int64_t ux = (int64_t)(bits(dxp) ^ sp), vx = (int64_t)(bits(dxm) ^ sm);
      const int64_t uy = (int64_t)(bits(dyp) ^ sp), vy = (int64_t)(bits(dym) ^ sm);
      const int64_t uz = (int64_t)(bits(dzp) ^ sp), vz = (int64_t)(bits(dzm) ^ sm);
      const int64_t wx = ux > vx ? ux : vx, wy = uy > vy ? uy : vy, wz = uz > vz ? uz : vz;
      const int hx = max((int)(wx >> 32), 0x30000000), hy = max((int)(wy >> 32), 0x30000000),
                hz = max((int)(wz >> 32), 0x30000000);
      const uint64_t acc2 = mag2(bits(cc)), ap02 = mag2(bits(p0)), tol2 = mag2(0x3ee4f8b588e368f1ull);  // 1e-5
      const uint32_t ach = hi32(cc) & 0x7fffffffu;
      const bool far = bits(d0) == a.far_bits;
      const bool plain = far ? max(max(hx, hy), hz) < 0x46300000 && acc2 > tol2 && acc2 <= kInf2
                             : ach - 0x3af00000u < 0x0b400000u && (hi32(d0) & 0x7fffffffu) < 0x46300000u;
      double r;
      if (plain && ap02 > tol2 && ap02 <= kInf2) {
        const uint32_t neg0 = hi32(p0) & 0x80000000u;  // sgn = +-1
        double from = d0, mag;
        if (far) {
          const double gx = mul_win((uint32_t)hx, (uint32_t)wx, hi32(inv.x), lo32(inv.x));
          const double gy = mul_win((uint32_t)hy, (uint32_t)wy, hi32(inv.y), lo32(inv.y));
          const double gz = mul_win((uint32_t)hz, (uint32_t)wz, hi32(inv.z), lo32(inv.z));
          const double n2 = sq_win(hi32(gx), lo32(gx)) + sq_win(hi32(gy), lo32(gy)) + sq_win(hi32(gz), lo32(gz));
          mag = sqrt_win(hi32(n2), lo32(n2));
          from = __hiloint2double((int)(0x3ff00000u | neg0), 0);
        } else {
          mag = div_recip(ach, lo32(cc), dxh, dxl, dx_recip);
        }
        r = from + __hiloint2double((int)(hi32(mag) ^ neg0 ^ 0x80000000u), (int)lo32(mag));
        if (!a.rhs_only) {
          // dt r with |r| raised to 2^-255 (r = 0: phi + tiny rounds to phi)
          const uint32_t ar = hi32(r) & 0x7fffffffu;
          const double dr = mul_win((ar > 0x30000000u ? ar : 0x30000000u) | (hi32(r) & 0x80000000u), lo32(r),
                                    hi32(a.dt_r), lo32(a.dt_r));
          r = cc + dr;
        }
      } else {
        r = reinit_general(cc, p0, d0, dxp, dyp, dzp, dxm, dym, dzm, inv, a.max_dx, a.far_bits);
        if (!a.rhs_only) r = cc + qss_emu::mul(a.dt_r, r);
      }
      a.next[field][c] = r;
    }
    dzm = dzp;
    cc = zp;
    c += sz;
  }
}

template <int EMU>
__global__ void k_reinit_step(Box b, const double* __restrict__ data, const double* __restrict__ phi0,
                              const double* __restrict__ distance0, double* __restrict__ next, double dt_r,
                              Inv inv, double max_dx, int rhs_only, uint64_t far_bits) {
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t c = b.idx(i, j, k);
  const double r = EMU == 0 ? reinit_rhs_at(data, phi0, distance0, b, c, inv, max_dx)
                            : reinit_rhs_e<EMU>(data, phi0, distance0, b, c, inv, max_dx, far_bits);
  next[c] = rhs_only ? r : data[c] + (EMU >= 2 ? qss_emu::mul(dt_r, r) : dt_r * r);
}

// ---------------------------------------------------------------------------
// coefficient set-up (3d.f:13-298, qss_util3d.f:499-581)

__global__ void k_central_grad(Box b, const double* __restrict__ f, double* fx, double* fy, double* fz,
                               Fac fac) {
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t c = b.idx(i, j, k), sy = b.sy(), sz = b.sz();
  fx[c] = (f[c + 1] - f[c - 1]) * fac.x;
  fy[c] = (f[c + sy] - f[c - sy]) * fac.y;
  fz[c] = (f[c + sz] - f[c - sz]) * fac.z;
}

struct MaskGeom {
  double h1, h2, absgrad, s;
};

__device__ __forceinline__ MaskGeom mask_geom(double m, double mx, double my, double mz, double dx) {
  const double eps_var = 1.5 * dx;
  MaskGeom g;
  g.h1 = qss_heaviside(-m, eps_var);
  g.h2 = qss_heaviside(m, eps_var);
  double ag = mx * mx + my * my + mz * mz;
  ag = sqrt(ag);
  double x = m * m + ag * dx * ag * dx;
  x = sqrt(x);
  g.absgrad = ag;
  g.s = m / x;
  return g;
}

// The coefficients from the mask and its gradient: CURV the curvature
// coefficient and the advection velocity with their CFL maxima, otherwise the
// normal velocity.  The smoothed step of the mask is 0 or 1 for most voxels,
// and what is left of the expressions there needs no FP64 instruction in the
// pore space (a0; the curvature coefficient and signed zeros) and four in the
// solid.  The voxels inside the smoothing band, whose sines and divisions are
// ~70 FP64 instructions, and those with operands out of range (SetVar::plain,
// coef_plain) are gathered per block of 1024 voxels and evaluated by full warps.
// The maxima go over integer keys: a native comparison occupies the FP64 pipe
// like an addition.  With everything evaluated natively everywhere the two
// kernels took 2.4 ms each at 192^3.
struct SetVar {
  const double *mask, *mx, *my, *mz, *theta_field;
  double *vel_n, *vb, *vx, *vy, *vz;
  double coef;  // a0, or the constant curvature coefficient
  double theta, dx;
  bool plain;
  unsigned long long* red;
  double eps, inv, coef0;  // 1.5 dx, 1 / dx, 0 coef
};
constexpr int kSetVoxels = 1024, kSetThreads = 256;

struct SetVarOut {
  double a, x, y, z;  // normal velocity; or curvature coefficient and velocity
};

template <bool CURV>
__device__ __noinline__ SetVarOut setvar_native(double m, double gx, double gy, double gz, double theta, double coef,
                                                double dx) {
  const double C2 = 1;
  const MaskGeom g = mask_geom(m, gx, gy, gz, dx);
  if (CURV) return {g.h1 * coef, g.s * C2 * gx * g.h2, g.s * C2 * gy * g.h2, g.s * C2 * gz * g.h2};
  return {g.h1 * coef - g.s * g.h2 * C2 * portable_cos(theta) * g.absgrad, 0.0, 0.0, 0.0};
}

// the mask in [2^-127, 2^129) and the gradient below 2^129
__device__ __forceinline__ bool coef_plain(double m, double gx, double gy, double gz, uint32_t& top) {
  using namespace qss_emu;
  top = max(max(hi32(gx) & 0x7fffffffu, hi32(gy) & 0x7fffffffu), hi32(gz) & 0x7fffffffu);
  return win8(m) < kWin8 && top < 0x48000000u;
}

// s and |gradient| of mask_geom, where the largest component is 2^-127 or more
// (the floor of 2^-255 under the others changes no sum)
__device__ __forceinline__ void sign_geom(double m, double gx, double gy, double gz, double dx, double& s, double& ag) {
  using namespace qss_emu;
  auto sq = [](double v) { return sq_win(max(hi32(v) & 0x7fffffffu, 0x30000000u), lo32(v)); };
  const double a2 = sq(gx) + sq(gy) + sq(gz);
  ag = sqrt_win(hi32(a2), lo32(a2));
  const double x2 = sqw(m) + mulw(mulw(mulw(ag, dx), ag), dx);
  const double x = sqrt_win(hi32(x2), lo32(x2));
  bool ok = true;
  s = div_win(hi32(m), lo32(m), hi32(x), lo32(x), ok);
}

template <bool CURV>
__global__ void __launch_bounds__(kSetThreads) k_setvar(Box b, SetVar a) {
  using namespace qss_emu;
  __shared__ uint16_t band[kSetVoxels];
  __shared__ int band_n;
  __shared__ double cos_theta;
  const FillBlock blk(b, blockIdx.x, kSetVoxels);
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) band_n = 0;
  if (!CURV && !a.theta_field && threadIdx.x < 32) {
    const double ct = portable_cos(a.theta);
    if (threadIdx.x == 0) cos_theta = ct;
  }
  __syncthreads();
  const double eps = a.eps, inv = a.inv;
  unsigned long long bm = 0, um = 0;  // keys, 0: none; NaNs count as none
  auto keep = [&](const SetVarOut& r) {
    const double u = qss_emu::abs(r.x) * inv + qss_emu::abs(r.y) * inv + qss_emu::abs(r.z) * inv;
    const unsigned long long kb = isnan_bits(bits(r.a)) ? 0 : double_to_key(r.a);
    const unsigned long long ku = isnan_bits(bits(u)) ? 0 : double_to_key(u);
    bm = kb > bm ? kb : bm;
    um = ku > um ? ku : um;
  };
  auto put = [&](int64_t c, const SetVarOut& r) {
    if (CURV) {
      a.vb[c] = r.a;
      a.vx[c] = r.x;
      a.vy[c] = r.y;
      a.vz[c] = r.z;
    } else {
      a.vel_n[c] = r.a;
    }
  };
  for (int t0 = 0; t0 < kSetVoxels; t0 += kSetThreads) {
    const uint32_t t = t0 + threadIdx.x;
    bool rest = false;
    if (blk.in(t)) {
      const int64_t c = blk.at(b, t);
      const double m = a.mask[c], gx = a.mx[c], gy = a.my[c], gz = a.mz[c];
      uint32_t top;
      rest = !(a.plain && coef_plain(m, gx, gy, gz, top));
      const bool pore = gt(neg(eps), m), solid = gt(m, eps);
      rest = rest || !(pore || (solid && top >= 0x38000000u));
      if (!CURV && a.theta_field) rest = rest || (hi32(a.theta_field[c]) & 0x7fffffffu) >= 0x41300000u;  // 2^20
      if (!rest) {
        SetVarOut r{};
        if (pore) {
          r.a = a.coef;
          if (CURV) {  // s is negative
            r.x = __hiloint2double((int)(~hi32(gx) & 0x80000000u), 0);
            r.y = __hiloint2double((int)(~hi32(gy) & 0x80000000u), 0);
            r.z = __hiloint2double((int)(~hi32(gz) & 0x80000000u), 0);
            const unsigned long long kb = double_to_key(r.a), ku = double_to_key(0.0);
            bm = kb > bm ? kb : bm;
            um = ku > um ? ku : um;
          }
          put(c, r);
        } else {
          double s, ag;
          sign_geom(m, gx, gy, gz, a.dx, s, ag);
          if (CURV) {
            r.a = a.coef0;
            r.x = mul(s, gx);
            r.y = mul(s, gy);
            r.z = mul(s, gz);
            keep(r);
            put(c, r);
          } else {
            const double v = mul(mul(s, a.theta_field ? portable_cos(a.theta_field[c]) : cos_theta), ag);
            r.a = neg(v);  // 0 a0 - v
            rest = mag2(bits(v)) == 0;
            if (!rest) put(c, r);
          }
        }
      }
    }
    const unsigned vote = __ballot_sync(0xffffffffu, rest);
    int slot = 0;
    if (lane == 0 && vote) slot = atomicAdd(&band_n, __popc(vote));
    slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(vote & ((1u << lane) - 1u));
    if (rest) band[slot] = (uint16_t)t;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < band_n; e += kSetThreads) {
    const int64_t c = blk.at(b, band[e]);
    const double m = a.mask[c], gx = a.mx[c], gy = a.my[c], gz = a.mz[c];
    uint32_t top;
    SetVarOut r{};
    if (a.plain && coef_plain(m, gx, gy, gz, top) && top >= 0x38000000u && gt(m, neg(eps)) && gt(eps, m) &&
        !(!CURV && a.theta_field)) {
      // both smoothed steps from one quotient and one sine, which are odd in m
      double s, ag;
      sign_geom(m, gx, gy, gz, a.dx, s, ag);
      const double pi = 3.14159265358979323846, one_over_pi = 0.31830988618379;
      const double q = div(m, 2 * eps), w = (0.5 * one_over_pi) * portable_sin(div(mul(pi, m), eps));
      const double h1 = 0.5 - q - w, h2 = 0.5 + q + w;
      if (CURV) r = {h1 * a.coef, mul(mul(s, gx), h2), mul(mul(s, gy), h2), mul(mul(s, gz), h2)};
      else r.a = h1 * a.coef - mul(mul(mul(s, h2), cos_theta), ag);
    } else {
      r = setvar_native<CURV>(m, gx, gy, gz, CURV ? 0.0 : (a.theta_field ? a.theta_field[c] : a.theta), a.coef, a.dx);
    }
    if (CURV) keep(r);
    put(c, r);
  }
  if (CURV) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long x = __shfl_down_sync(0xffffffffu, bm, o), y = __shfl_down_sync(0xffffffffu, um, o);
      bm = x > bm ? x : bm;
      um = y > um ? y : um;
    }
    if (lane == 0) {
      atomicMax(&a.red[0], bm);
      atomicMax(&a.red[1], um);
    }
  }
}

__global__ void k_trapvel(Box b, const double* __restrict__ test, double* vel_n, double* vb, double* vx,
                          double* vy, double* vz, double dx) {
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t c = b.idx(i, j, k);
  if (test[c] > 1.5 * dx) {
    vel_n[c] = 0;
    vb[c] = 0;
    vx[c] = 0;
    vy[c] = 0;
    vz[c] = 0;
  }
}

// ---------------------------------------------------------------------------
// whole-array operations

__global__ void k_max_into(int64_t n, double* out, const double* mask, const double* phi) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double m = mask[q], p = phi[q];
    out[q] = (m > p) ? m : p;
  }
}
__global__ void k_min_into(int64_t n, double* out, const double* a, const double* b) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double x = a[q], y = b[q];
    out[q] = (x < y) ? x : y;
  }
}
__global__ void k_merge(int64_t n, double* phi, const double* m) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double v = m[q];
    if (v > 0) phi[q] = -v;
  }
}
__global__ void k_fill(int64_t n, double* out, double v) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    out[q] = v;
}

__global__ void k_rk(Box b, int stage, double* out, const double* u1, const double* u0, const double* rhs,
                     double dt) {
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t c = b.idx(i, j, k);
  if (stage == 1) {
    out[c] = u1[c] + dt * rhs[c];
  } else if (stage == 2) {
    out[c] = 0.75 * u0[c] + 0.25 * (u1[c] + dt * rhs[c]);
  } else {
    const double one_third = 1.0 / 3.0, two_thirds = 2.0 / 3.0;
    out[c] = one_third * u0[c] + two_thirds * (u1[c] + dt * rhs[c]);
  }
}

__global__ void k_impose_slab(Box b, double* out, const double* mask, const double* phi, double overlap, int k0,
                              int k1) {
  const int64_t nxy = (int64_t)b.nx * b.ny;
  const int64_t total = (int64_t)(k1 - k0 + 1) * nxy;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
       q += (int64_t)gridDim.x * blockDim.x) {
    int64_t c = (int64_t)k0 * nxy + q;
    double m = mask[c] - overlap, p = phi[c];
    out[c] = (m > p) ? m : p;
  }
}

// ---------------------------------------------------------------------------
// reductions

__global__ void k_maxnormdiff(Box b, const double* __restrict__ f1, const double* __restrict__ f2, double zone,
                              unsigned long long* key) {
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  // magnitudes compared as integers (-1: none; NaN differences count as none):
  // a native comparison occupies the FP64 pipe like an addition
  long long m = -1;
  if (i <= b.ihi && j <= b.jhi && k <= b.khi) {
    const int64_t c = b.idx(i, j, k);
    const double a = f1[c];
    if (qss_emu::gt(zone, a) && qss_emu::gt(a, -zone)) {  // |a| < zone
      m = (long long)qss_emu::bits(qss_emu::abs(a - f2[c]));
      if (m > 0x7ff0000000000000ll) m = -1;
    }
  }
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
  const int lane = (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)) & 31;
  if (lane == 0 && m >= 0) atomicMax(key, double_to_key(__longlong_as_double(m)));
}

// ---------------------------------------------------------------------------
// geometry (src/geometry/qss_initialization3d.c:33-165, 440-522)

__global__ void k_sphere(Box b, double* phi, double x0, double y0, double z0, double dx, double dy, double dz,
                         double cx, double cy, double cz, double r, int inside) {
  const int64_t n = b.npts();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % b.nx);
    const int64_t rr = q / b.nx;
    const int j = (int)(rr % b.ny), k = (int)(rr / b.ny);
    const double x = x0 + dx * i, y = y0 + dy * j, z = z0 + dz * k;
    double d = sqrt((x - cx) * (x - cx) + (y - cy) * (y - cy) + (z - cz) * (z - cz)) - r;
    if (inside >= 0) d = -d;
    double best = -FLT_MAX;
    if (d > best) best = d;
    phi[q] = best;
  }
}

__global__ void k_box(Box b, double* phi, double x0, double y0, double z0, double dx, double dy, double dz,
                      double c0, double c1, double c2, double s0, double s1, double s2, int inside) {
  const int64_t n = b.npts();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % b.nx);
    const int64_t rr = q / b.nx;
    const int j = (int)(rr % b.ny), k = (int)(rr / b.ny);
    const double x = x0 + dx * i, y = y0 + dy * j, z = z0 + dz * k;
    double best = -FLT_MAX;
#pragma unroll
    for (int p = 0; p < 6; p++) {
      const bool low = p < 3;
      const int ax = p % 3;
      const double px = low ? c0 : c0 + s0, py = low ? c1 : c1 + s1, pz = low ? c2 : c2 + s2;
      const double sg = low ? -1 : 1;
      const double nx = (ax == 0) ? sg : 0, ny = (ax == 1) ? sg : 0, nz = (ax == 2) ? sg : 0;
      const double dot = (x - px) * nx + (y - py) * ny + (z - pz) * nz;
      double nrm = nx * nx + ny * ny + nz * nz;
      nrm = sqrt(nrm);
      const double d = dot / nrm;
      if (d > best) best = d;
    }
    phi[q] = (inside >= 1) ? -best : best;
  }
}

__global__ void k_spheres(Box b, double* phi, double x0, double y0, double z0, double dx, double dy, double dz,
                          const double* __restrict__ cx, const double* __restrict__ cy,
                          const double* __restrict__ cz, const double* __restrict__ rad,
                          const int* __restrict__ inside, int num) {
  const int64_t n = b.npts();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % b.nx);
    const int64_t rr = q / b.nx;
    const int j = (int)(rr % b.ny), k = (int)(rr / b.ny);
    const double x = x0 + dx * i, y = y0 + dy * j, z = z0 + dz * k;
    double best = -FLT_MAX;
    for (int l = 0; l < num; l++) {
      double d = sqrt((x - cx[l]) * (x - cx[l]) + (y - cy[l]) * (y - cy[l]) + (z - cz[l]) * (z - cz[l])) - rad[l];
      if (inside[l] >= 0) d = -d;
      if (d > best) best = d;
    }
    phi[q] = best;
  }
}

__global__ void k_halfspaces(Box b, double* phi, double x0, double y0, double z0, double dx, double dy, double dz,
                             const double* __restrict__ nxv, const double* __restrict__ nyv,
                             const double* __restrict__ nzv, const double* __restrict__ px,
                             const double* __restrict__ py, const double* __restrict__ pz, int num) {
  const int64_t n = b.npts();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % b.nx);
    const int64_t rr = q / b.nx;
    const int j = (int)(rr % b.ny), k = (int)(rr / b.ny);
    const double x = x0 + dx * i, y = y0 + dy * j, z = z0 + dz * k;
    double best = -FLT_MAX;
    for (int l = 0; l < num; l++) {
      const double dot = (x - px[l]) * nxv[l] + (y - py[l]) * nyv[l] + (z - pz[l]) * nzv[l];
      double nrm = nxv[l] * nxv[l] + nyv[l] * nyv[l] + nzv[l] * nzv[l];
      nrm = sqrt(nrm);
      const double d = dot / nrm;
      if (d > best) best = d;
    }
    phi[q] = best;
  }
}

__global__ void k_negate(int64_t n, double* a) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    a[q] = -a[q];
}

}  // namespace

// ===========================================================================
// launch wrappers

static const dim3 kBlk3(32, 4, 1);

// stage-kernel timing (host side): event pairs recorded around each launch
// of a stage kernel on the profiled stream, tagged with the kernel's kind
namespace {
struct StageProfiler {
  bool on = false;
  cudaStream_t stream = nullptr;
  struct Rec {
    int kind;
    cudaEvent_t e0, e1;
  };
  std::vector<Rec> ev;
} g_prof;
}  // namespace

void qss_profile_stage_begin(cudaStream_t s) {
  g_prof.on = true;
  g_prof.stream = s;
  g_prof.ev.clear();
}

void qss_profile_stage_end(double ms[kProfKinds], int launches[kProfKinds]) {
  for (int k = 0; k < kProfKinds; k++) {
    ms[k] = 0;
    launches[k] = 0;
  }
  for (auto& e : g_prof.ev) {
    cudaEventSynchronize(e.e1);
    float t = 0;
    cudaEventElapsedTime(&t, e.e0, e.e1);
    ms[e.kind] += t;
    launches[e.kind]++;
    cudaEventDestroy(e.e0);
    cudaEventDestroy(e.e1);
  }
  g_prof.ev.clear();
  g_prof.on = false;
}

cudaEvent_t prof_open(cudaStream_t s) {
  if (!g_prof.on || s != g_prof.stream) return nullptr;
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  cudaEventRecord(e, s);
  return e;
}

void prof_close(cudaStream_t s, cudaEvent_t e0, int kind) {
  if (!e0) return;
  cudaEvent_t e1 = nullptr;
  cudaEventCreate(&e1);
  cudaEventRecord(e1, s);
  g_prof.ev.push_back({kind, e0, e1});
}

static const int kBlk1 = 256;

static unsigned grid1(int64_t n) {
  int64_t b = (n + kBlk1 - 1) / kBlk1;
  if (b > 152 * 32) b = 152 * 32;
  if (b < 1) b = 1;
  return (unsigned)b;
}

void launch_dt(cudaStream_t s, int scheme, bool var, const Box& b, const double* phi, const Coef& c, int nslabs,
               double dx, double dy, double dz, Ctl* ctl) {
  const Inv inv{1.0 / dx, 1.0 / dy, 1.0 / dz};
#define QSS_DT(S, V) k_dt<S, V><<<1, nslabs <= 4 ? 32 : kDtThreads, 0, s>>>(b, phi, c, nslabs, dx, dy, dz, inv, ctl)
  if (scheme == ENO2) { if (var) QSS_DT(ENO2, true); else QSS_DT(ENO2, false); }
  else if (scheme == ENO3) { if (var) QSS_DT(ENO3, true); else QSS_DT(ENO3, false); }
  else { if (var) QSS_DT(WENO5, true); else QSS_DT(WENO5, false); }
#undef QSS_DT
}

template <int S, bool V>
static void stage_dispatch(cudaStream_t s, int stage, bool fin, dim3 g, dim3 blk, const StageArgs& a) {
  switch (stage) {
    case 0: k_stage<S, V, 0, false><<<g, blk, 0, s>>>(a); break;
    case 1: if (fin) k_stage<S, V, 1, true><<<g, blk, 0, s>>>(a); else k_stage<S, V, 1, false><<<g, blk, 0, s>>>(a); break;
    case 2: if (fin) k_stage<S, V, 2, true><<<g, blk, 0, s>>>(a); else k_stage<S, V, 2, false><<<g, blk, 0, s>>>(a); break;
    default: if (fin) k_stage<S, V, 3, true><<<g, blk, 0, s>>>(a); else k_stage<S, V, 3, false><<<g, blk, 0, s>>>(a); break;
  }
}

template <bool V>
static void eno_dispatch(cudaStream_t s, int scheme, int stage, bool fin, dim3 g, const StageArgs& a) {
#define QSS_ENO(S, F) \
  { if (scheme == ENO2) k_eno2<V, S, F><<<g, 128, 0, s>>>(a); else k_eno3<V, S, F><<<g, 128, 0, s>>>(a); }
  switch (stage) {
    case 0: QSS_ENO(0, false) break;
    case 1: if (fin) QSS_ENO(1, true) else QSS_ENO(1, false) break;
    case 2: if (fin) QSS_ENO(2, true) else QSS_ENO(2, false) break;
    default: if (fin) QSS_ENO(3, true) else QSS_ENO(3, false) break;
  }
#undef QSS_ENO
}

void launch_stage(cudaStream_t s, int scheme, bool var, int stage, bool final_stage, const Box& b, double dx,
                  double dy, double dz, const double* phi_in, const double* u_cur, double* out, double* phi_new,
                  const Coef& c, const ImposeArgs& im, const Ctl* ctl) {
  StageArgs a;
  a.b = b;
  a.inv = Inv{1.0 / dx, 1.0 / dy, 1.0 / dz};
  a.fac = Fac{0.5 / dx, 0.5 / dy, 0.5 / dz};
  a.phi_in = phi_in;
  a.u_cur = u_cur;
  a.out = out;
  a.phi_new = phi_new;
  a.c = c;
  a.im = im;
  a.ctl = ctl;
  dim3 g = fb_grid(b, kBlk3);
  cudaEvent_t e0 = stage != 0 ? prof_open(s) : nullptr;
  // ENO3 scales its y and z minus differences by 1/dx, the plus ones by 1/dy, 1/dz
  const bool fast = emu_level() >= 2 && scheme != WENO5 && stage_factor(a.fac.x) && stage_factor(a.fac.y) &&
                    stage_factor(a.fac.z) && (scheme == ENO2 || (dx == dy && dx == dz));
  dim3 ge((b.fbx() + 31) / 32, (b.fby() + 3) / 4, b.fbz());
  if (fast && scheme == ENO2) {
    const int64_t walk = (int64_t)ge.x * ge.y * b.fbz() / (152 * kEno2Target);
    a.walk = (int)(walk < 1 ? 1 : (walk > kEno2Walk ? kEno2Walk : walk));
    ge.z = (b.fbz() + a.walk - 1) / a.walk;
  }
  if (fast) { if (var) eno_dispatch<true>(s, scheme, stage, final_stage, ge, a); else eno_dispatch<false>(s, scheme, stage, final_stage, ge, a); }
  else if (scheme == ENO2) { if (var) stage_dispatch<ENO2, true>(s, stage, final_stage, g, kBlk3, a); else stage_dispatch<ENO2, false>(s, stage, final_stage, g, kBlk3, a); }
  else if (scheme == ENO3) { if (var) stage_dispatch<ENO3, true>(s, stage, final_stage, g, kBlk3, a); else stage_dispatch<ENO3, false>(s, stage, final_stage, g, kBlk3, a); }
  else { if (var) stage_dispatch<WENO5, true>(s, stage, final_stage, g, kBlk3, a); else stage_dispatch<WENO5, false>(s, stage, final_stage, g, kBlk3, a); }
  prof_close(s, e0, kProfStage);
}

void launch_cfl_at(cudaStream_t s, int scheme, bool var, const Box& b, const double* phi, const Coef& c, int i,
                   int j, int k, double dx, double dy, double dz, double* h_out) {
  const Inv inv{1.0 / dx, 1.0 / dy, 1.0 / dz};
#define QSS_CFL(S, V) k_cfl_at<S, V><<<1, 32, 0, s>>>(b, phi, c, i, j, k, dx, dy, dz, inv, h_out)
  if (scheme == ENO2) { if (var) QSS_CFL(ENO2, true); else QSS_CFL(ENO2, false); }
  else if (scheme == ENO3) { if (var) QSS_CFL(ENO3, true); else QSS_CFL(ENO3, false); }
  else { if (var) QSS_CFL(WENO5, true); else QSS_CFL(WENO5, false); }
#undef QSS_CFL
}

void launch_ghost(cudaStream_t s, const Box& b, double* a, double* phi_new, const ImposeArgs& im, const Ctl* ctl) {
  const int64_t total = b.npts() - (int64_t)b.fbx() * b.fby() * b.fbz();
  k_ghost<<<grid1(total), kBlk1, 0, s>>>(b, a, phi_new, im, ctl);
}

void launch_face(cudaStream_t s, const Box& b, double* a, int face) {
  int lines = face < 2 ? b.ny * b.nz : (face < 4 ? b.nx * b.nz : b.nx * b.ny);
  k_face<<<(lines + 255) / 256, 256, 0, s>>>(b, a, face);
}

void launch_impose_region(cudaStream_t s, const Box& b, const double* src, double* phi_new, const ImposeArgs& im,
                          const Ctl* ctl) {
  k_impose_region<<<grid1(b.npts()), kBlk1, 0, s>>>(b, src, phi_new, im, ctl);
}

void launch_nsrc(cudaStream_t s, const Box& b, const double* vel_n, int* nsrc, int nslabs, int* d_rowlast,
                 int* d_carry, unsigned long long* d_count) {
  const int64_t nrows = (int64_t)b.fby() * b.fbz();
  cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), s);
  const unsigned blocks = (unsigned)((nrows + 7) / 8);  // 8 warps each
  k_nsrc_rowlast<<<blocks, 256, 0, s>>>(b, vel_n, d_rowlast);
  k_nsrc_carry<<<nslabs, 1024, 0, s>>>(b, nslabs, d_rowlast, d_carry);
  k_nsrc_fill<<<blocks, 256, 0, s>>>(b, vel_n, d_carry, nsrc, d_count);
}

void launch_distance0(cudaStream_t s, const Box& b, const double* phi0, double* distance0, double dx, double dy,
                      double dz) {
  const int64_t n = (int64_t)b.fbx() * b.fby() * b.fbz();
  k_distance0<<<(unsigned)((n + kNearVoxels - 1) / kNearVoxels), kNearThreads, 0, s>>>(
      b, phi0, distance0, dx > dy ? (dx > dz ? dx : dz) : (dy > dz ? dy : dz));
}

// $QSSGPU_REINIT_WALK=0 selects the one-voxel-per-thread reinitialisation
// step at level 2 (identical results)
static bool reinit_walk() {
  static const int on = [] {
    const char* e = getenv("QSSGPU_REINIT_WALK");
    return e && atoi(e) == 0 ? 0 : 1;
  }();
  return on != 0;
}

// constants whose products with the kernel's operands stay normal
static bool middling(double x) { return x > 1e-30 && x < 1e30; }

// one sweep of nf <= 2 fields; from_fill: the ghost layers of data are taken to
// be the extrapolation of its fill box and may be stale.  Returns false, having
// done nothing, where this form does not apply.
static bool reinit_walk_launch(cudaStream_t s, const Box& b, const ReinitArrays* f, int nf, bool from_fill, double dt_r,
                               double dx, double dy, double dz, int rhs_only) {
  const double max_dx = (dx > dy ? dx : dy) > dz ? (dx > dy ? dx : dy) : dz;
  if (emu_level() < 2 || !reinit_walk() || !middling(dx) || !middling(dy) || !middling(dz) ||
      !(rhs_only || middling(dt_r)))
    return false;
  ReinitSweep a{};
  for (int q = 0; q < nf; q++) {
    a.data[q] = f[q].data;
    a.phi0[q] = f[q].phi0;
    a.dist[q] = f[q].dist;
    a.next[q] = f[q].next;
  }
  a.dt_r = dt_r;
  a.max_dx = max_dx;
  a.inv = Inv{1.0 / dx, 1.0 / dy, 1.0 / dz};
  a.far_bits = qss_emu::bits(-1000.0 * max_dx);  // distance0 of voxels away from the interface
  a.rhs_only = rhs_only;
  // planes per thread: up to kRWalkMax while the grid keeps ~16 blocks per SM
  const int64_t xy = (int64_t)((b.fbx() + 31) / 32) * ((b.fby() + 3) / 4);
  int64_t walk = xy * nf * b.fbz() / (152 * 16);
  a.walk = (int)(walk < 1 ? 1 : (walk > kRWalkMax ? kRWalkMax : walk));
  a.chunks = (b.fbz() + a.walk - 1) / a.walk;
  const dim3 g((b.fbx() + 31) / 32, (b.fby() + 3) / 4, (unsigned)(a.chunks * nf));
  if (from_fill) k_reinit_walk<true><<<g, 128, 0, s>>>(b, a);
  else k_reinit_walk<false><<<g, 128, 0, s>>>(b, a);
  return true;
}

static void reinit_launch(cudaStream_t s, const Box& b, const ReinitArrays& f, double dt_r, double dx, double dy,
                          double dz, int rhs_only) {
  const double max_dx = (dx > dy ? dx : dy) > dz ? (dx > dy ? dx : dy) : dz;
  const Inv inv{1.0 / dx, 1.0 / dy, 1.0 / dz};
  const uint64_t far_bits = qss_emu::bits(-1000.0 * max_dx);
  const int lvl = emu_level();
  const dim3 grid = fb_grid(b, kBlk3);
  if (lvl >= 2)
    k_reinit_step<2><<<grid, kBlk3, 0, s>>>(b, f.data, f.phi0, f.dist, f.next, dt_r, inv, max_dx, rhs_only, far_bits);
  else if (lvl == 1)
    k_reinit_step<1><<<grid, kBlk3, 0, s>>>(b, f.data, f.phi0, f.dist, f.next, dt_r, inv, max_dx, rhs_only, far_bits);
  else
    k_reinit_step<0><<<grid, kBlk3, 0, s>>>(b, f.data, f.phi0, f.dist, f.next, dt_r, inv, max_dx, rhs_only, far_bits);
}

void launch_reinit_sweep(cudaStream_t s, const Box& b, const ReinitArrays* f, int nf, bool from_fill, double dt_r,
                         double dx, double dy, double dz) {
  if (reinit_walk_launch(s, b, f, nf, from_fill, dt_r, dx, dy, dz, 0)) return;
  for (int q = 0; q < nf; q++) {
    // this form reads the ghost layers
    if (from_fill) launch_ghost(s, b, const_cast<double*>(f[q].data), nullptr, ImposeArgs{}, nullptr);
    reinit_launch(s, b, f[q], dt_r, dx, dy, dz, 0);
  }
}

void launch_reinit_rhs(cudaStream_t s, const Box& b, const double* data, const double* phi0,
                       const double* distance0, double* rhs, bool from_fill, double dx, double dy, double dz) {
  const ReinitArrays f{const_cast<double*>(data), const_cast<double*>(phi0), const_cast<double*>(distance0), rhs};
  if (reinit_walk_launch(s, b, &f, 1, from_fill, 0.0, dx, dy, dz, 1)) return;
  if (from_fill) launch_ghost(s, b, const_cast<double*>(data), nullptr, ImposeArgs{}, nullptr);
  reinit_launch(s, b, f, 0.0, dx, dy, dz, 1);
}

void launch_reinit(cudaStream_t s, const Box& b, ReinitArrays* f, int nf, int iters, double dt_r, double dx, double dy,
                   double dz) {
  if (iters <= 0) return;
  for (int q = 0; q < nf; q++) {
    // the input stays where it is, as phi0; the sweeps alternate between the
    // other two arrays
    std::swap(f[q].data, f[q].phi0);
    launch_distance0(s, b, f[q].phi0, f[q].dist, dx, dy, dz);
  }
  for (int it = 0; it < iters; it++) {
    ReinitArrays g[kReinitFields];
    for (int q = 0; q < nf; q++) {
      g[q] = f[q];
      if (it == 0) g[q].data = f[q].phi0;
    }
    launch_reinit_sweep(s, b, g, nf, it > 0, dt_r, dx, dy, dz);
    for (int q = 0; q < nf; q++) std::swap(f[q].data, f[q].next);
  }
  for (int q = 0; q < nf; q++) launch_ghost(s, b, f[q].data, nullptr, ImposeArgs{}, nullptr);
}

void launch_central_grad(cudaStream_t s, const Box& b, const double* f, double* fx, double* fy, double* fz,
                         double dx, double dy, double dz) {
  k_central_grad<<<fb_grid(b, kBlk3), kBlk3, 0, s>>>(b, f, fx, fy, fz, Fac{0.5 / dx, 0.5 / dy, 0.5 / dz});
}

static unsigned setvar_blocks(const Box& b) {
  return (unsigned)(((int64_t)b.fbx() * b.fby() * b.fbz() + kSetVoxels - 1) / kSetVoxels);
}

void launch_setvarnorm(cudaStream_t s, const Box& b, const double* mask, const double* mx, const double* my,
                       const double* mz, double* vel_n, double a0, const double* theta_field, double theta,
                       double dx) {
  SetVar a{mask, mx, my, mz, theta_field, vel_n, nullptr, nullptr, nullptr, nullptr, a0, theta, dx, false, nullptr, 1.5 * dx, 1.0 / dx, 0.0};
  a.plain = stage_factor(dx) && a0 != 0.0 && isfinite(a0) && (theta_field || fabs(theta) < 0x1p20);
  k_setvar<false><<<setvar_blocks(b), kSetThreads, 0, s>>>(b, a);
}

void launch_setvarcurvadv(cudaStream_t s, const Box& b, const double* mask, const double* mx, const double* my,
                          const double* mz, double* vb, double* vx, double* vy, double* vz, double const_b,
                          double dx, unsigned long long* red) {
  unsigned long long init[2] = {double_to_key(-1.0), double_to_key(-1.0)};
  cudaMemcpyAsync(red, init, sizeof init, cudaMemcpyHostToDevice, s);
  SetVar a{mask, mx, my, mz, nullptr, nullptr, vb, vx, vy, vz, const_b, 0.0, dx, false, red, 1.5 * dx, 1.0 / dx, 0.0 * const_b};
  a.plain = stage_factor(dx) && isfinite(const_b);
  k_setvar<true><<<setvar_blocks(b), kSetThreads, 0, s>>>(b, a);
}

void launch_trapvel(cudaStream_t s, const Box& b, const double* test, double* vel_n, double* vb, double* vx,
                    double* vy, double* vz, double dx) {
  k_trapvel<<<fb_grid(b, kBlk3), kBlk3, 0, s>>>(b, test, vel_n, vb, vx, vy, vz, dx);
}

void launch_max_into(cudaStream_t s, int64_t n, double* out, const double* mask, const double* phi) {
  k_max_into<<<grid1(n), kBlk1, 0, s>>>(n, out, mask, phi);
}
void launch_min_into(cudaStream_t s, int64_t n, double* out, const double* a, const double* b) {
  k_min_into<<<grid1(n), kBlk1, 0, s>>>(n, out, a, b);
}
void launch_merge(cudaStream_t s, int64_t n, double* phi, const double* m) {
  k_merge<<<grid1(n), kBlk1, 0, s>>>(n, phi, m);
}
void launch_fill(cudaStream_t s, int64_t n, double* out, double v) { k_fill<<<grid1(n), kBlk1, 0, s>>>(n, out, v); }

void launch_rk(cudaStream_t s, const Box& b, int stage, double* out, const double* u1, const double* u0,
               const double* rhs, double dt) {
  k_rk<<<fb_grid(b, kBlk3), kBlk3, 0, s>>>(b, stage, out, u1, u0, rhs, dt);
}

void launch_impose_slab(cudaStream_t s, const Box& b, double* out, const double* mask, const double* phi,
                        double overlap, int k0, int k1) {
  if (k1 < k0) return;
  k_impose_slab<<<grid1((int64_t)(k1 - k0 + 1) * b.nx * b.ny), kBlk1, 0, s>>>(b, out, mask, phi, overlap, k0, k1);
}

void launch_maxnormdiff(cudaStream_t s, const Box& b, const double* f1, const double* f2, double zone,
                        unsigned long long* key) {
  cudaMemsetAsync(key, 0, sizeof *key, s);
  k_maxnormdiff<<<fb_grid(b, kBlk3), kBlk3, 0, s>>>(b, f1, f2, zone, key);
}

void launch_sphere(cudaStream_t s, const Box& b, double* phi, const double* x_lo_gb, const double* dxv, double cx,
                   double cy, double cz, double r, int inside_flag) {
  k_sphere<<<grid1(b.npts()), kBlk1, 0, s>>>(b, phi, x_lo_gb[0], x_lo_gb[1], x_lo_gb[2], dxv[0], dxv[1], dxv[2],
                                              cx, cy, cz, r, inside_flag);
}

void launch_box(cudaStream_t s, const Box& b, double* phi, const double* x_lo_gb, const double* dxv,
                const double corner[3], const double side[3], int inside_flag) {
  k_box<<<grid1(b.npts()), kBlk1, 0, s>>>(b, phi, x_lo_gb[0], x_lo_gb[1], x_lo_gb[2], dxv[0], dxv[1], dxv[2],
                                           corner[0], corner[1], corner[2], side[0], side[1], side[2], inside_flag);
}

void launch_spheres(cudaStream_t s, const Box& b, double* phi, const double* x_lo_gb, const double* dxv,
                    const double* cx, const double* cy, const double* cz, const double* r, const int* inside,
                    int num) {
  k_spheres<<<grid1(b.npts()), kBlk1, 0, s>>>(b, phi, x_lo_gb[0], x_lo_gb[1], x_lo_gb[2], dxv[0], dxv[1], dxv[2], cx,
                                               cy, cz, r, inside, num);
}

void launch_halfspaces(cudaStream_t s, const Box& b, double* phi, const double* x_lo_gb, const double* dxv,
                       const double* nx, const double* ny, const double* nz, const double* px, const double* py,
                       const double* pz, int num) {
  k_halfspaces<<<grid1(b.npts()), kBlk1, 0, s>>>(b, phi, x_lo_gb[0], x_lo_gb[1], x_lo_gb[2], dxv[0], dxv[1],
                                                  dxv[2], nx, ny, nz, px, py, pz, num);
}

void launch_negate(cudaStream_t s, int64_t n, double* a) { k_negate<<<grid1(n), kBlk1, 0, s>>>(n, a); }

}  // namespace qss
