// qss_adjoint.cu -- adjoint of the constant-curvature update with respect to a
// spatially varying contact angle (no counterpart in the reference).
//
// Model (the var-coefficient inner step of constCurvModel3d.c:127-243 with
// check_connectivity = 0 and a fixed time step):
//   vel_n(x) = setVarNorm3dTheta(mask, grad mask, a0, theta(x))   (3d.f:94-172)
//   phi^{n+1} = impose(BC(s3)),  s1 = phi^n + dt L(phi^n)          (RK1)
//     s2 = 3/4 phi^n + 1/4 (BC(s1) + dt L(BC(s1)))                 (TVD-RK2 stage, F10)
//     s3 = 1/3 phi^n + 2/3 (BC(s2) + dt L(BC(s2)))                 (TVD-RK3 stage 3)
//   L = vel_n |grad phi|_Godunov(WENO5) + b kappa - V . grad phi_upwind   (getRHS3d5th)
//   BC = signed linear extrapolation of the six faces, impose = max(mask - overlap, .)
//   loss = sum over the fill box of (H_eps(phi^T) - target)^2, eps = 1.5 dx
// The forward runs the production kernels (split WENO5 passes + combine);
// the time step is an input, so no gradient flows through the CFL estimate.
//
// Backward (reverse mode by hand, FP64), per stage: k_adj_point takes each
// fill-box voxel's adjoint weight through the Godunov normal term, the upwind
// advection and the curvature, giving the adjoints of its six one-sided
// WENO5 derivatives and the partials of the curvature with respect to its
// central differences; k_adj_axis (one per axis) takes the derivative
// adjoints back to phi line by line, one WENO5 face window at a time for the
// minus derivative of one voxel and the plus derivative of its neighbour
// together (they share the window's smoothness indicators); k_adj_curv
// gathers the curvature partials.  Every point's adjoint is summed in a fixed
// order (deterministic); voxels whose normal term is carried from an earlier
// voxel (|vel_n| < 1e-5, 3d.f:459-486) add their (rare) contributions to
// that voxel's derivative adjoints by atomics.  The boundary extrapolation
// is reversed face by face (z, then y, then x), the imposition passes the
// adjoint where the stage value was kept.  Steps are
// recomputed from checkpoints every `ckpt` steps, storing the stage states
// of one segment at a time.
//
// This translation unit is compiled with FMA contraction: the reverse
// arithmetic has no reference bit pattern to reproduce (the forward steps run
// the uncontracted production kernels), and fused multiply-adds cut the FP64
// instructions of the reverse kernel, which is bound by the FP64 pipe.
#include <cstdlib>
#include <vector>

#include "qss_emu.cuh"
#include "qss_state.h"

namespace qss {

namespace {

constexpr double k1312 = 13.0 / 12.0, k136 = 13.0 / 6.0;

__device__ __noinline__ double mul_rare(double x, double y) { return x * y; }

// x * y on the integer pipes where zeros are common (adjoints of parts at rest, exactly
// linear parts): qss_emu::mul sends them down the branch of its FP64 instruction, which
// then takes the pipe for the whole warp
__device__ __forceinline__ double mulz(double x, double y) {
  using namespace qss_emu;
  const uint32_t xh = hi32(x), yh = hi32(y);
  const uint32_t wx = win(xh), wy = win(yh);
  const bool zx = mag2(bits(x)) == 0, zy = mag2(bits(y)) == 0;
  double r = mul_win(xh, lo32(x), yh, lo32(y));
  r = zx || zy ? __hiloint2double((int)((xh ^ yh) & 0x80000000u), 0) : r;
  if ((!zx && wx >= 0x40000000u) || (!zy && wy >= 0x40000000u)) r = mul_rare(x, y);
  return r;
}

// Godunov term of WENO5 (3d.f:2251-2276) and its partials: dtn/d(pp, pm), dtn/dvel
__device__ __forceinline__ void godunov_bwd(double vel, const double pp[3], const double pm[3], double ppb[3],
                                              double pmb[3], double& velb) {
  double a[3], c[3];
  bool use_a[3];
  double ngps = 0;
  const bool vpos = qss_emu::gt0(vel);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (vpos) {
      a[d] = qss_emu::gt0(pm[d]) ? pm[d] : 0.0;
      c[d] = qss_emu::lt0(pp[d]) ? pp[d] : 0.0;
    } else {
      a[d] = qss_emu::lt0(pm[d]) ? pm[d] : 0.0;
      c[d] = qss_emu::gt0(pp[d]) ? pp[d] : 0.0;
    }
    const double aa = mulz(a[d], a[d]), cc = mulz(c[d], c[d]);
    use_a[d] = (long long)qss_emu::bits(aa) > (long long)qss_emu::bits(cc);
    ngps += use_a[d] ? aa : cc;
  }
  const double norm = qss_emu::sqrt(ngps);
  velb = norm;
  // vel / (2 norm), the other 2 of the square's derivative folded in
  const double nb = qss_emu::gt0(norm) ? qss_emu::div(vel, norm) : 0.0;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (use_a[d]) pmb[d] = mulz(nb, a[d]);
    else ppb[d] = mulz(nb, c[d]);
  }
}

// |v| >= 1e-5
__device__ __forceinline__ bool moving(double v) {
  const uint64_t a = qss_emu::mag2(qss_emu::bits(v));
  return a >= 0x7dc9f16b11c6d1e2ull && a <= qss_emu::kInf2;
}
__device__ __forceinline__ bool nonzero(double v) { return qss_emu::mag2(qss_emu::bits(v)) != 0; }

struct AdjPointArgs {
  Box b;
  const double* phi;     // stage input, ghosts valid
  const double* dp[3];   // its WENO5 plus/minus derivatives (production axis passes)
  const double* dm[3];
  const double* lam_in;  // adjoint of the stage output; weight of the RHS = coef_l * lam_in (fill box)
  double coef_l;
  const double* vel_n;
  const double* bcoef;
  const double* vx;
  const double* vy;
  const double* vz;
  const int* nsrc;
  double fac[3];         // 1 / (2 dx) per axis
  double f2[6];          // fac products: xx, yy, zz, xy, xz, yz
  double* bp[3];         // out: adjoint of the plus / minus derivative per axis (fill box)
  double* bm[3];
  double* cc;            // out: 9 arrays of npts, the curvature's partials (see k_adj_curv)
  double* adj_vel;       // += dRHS/dvel * weight
  int64_t npts;
};

// Per fill-box voxel: the adjoints of the six one-sided WENO5 derivatives
// (Godunov normal term and upwind advection) and the partials of the
// curvature term b kappa (3d.f:2337-2379) with respect to its ten central
// differences, each times the voxel's adjoint weight.  Voxels whose normal
// term is carried from an earlier voxel leave that term to k_adj_carry.
// A block of 32 x 4 threads covers 32 (i) x 4 (j) voxels; each warp an 8 x 4
// patch of them, so that warps inside the grains (b = 0) skip the curvature
// partials together.
__global__ void __launch_bounds__(128, 7) k_adj_point(AdjPointArgs a) {
  const Box& b = a.b;
  const int lane = threadIdx.x, warp = threadIdx.y;
  const int i = b.ilo + blockIdx.x * 32 + 8 * warp + (lane & 7);
  const int j = b.jlo + blockIdx.y * 4 + (lane >> 3);
  const int k = b.klo + blockIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t q = b.idx(i, j, k);
  const double w = mulz(a.coef_l, a.lam_in[q]);
  const int64_t st[3] = {1, (int64_t)b.nx, (int64_t)b.nx * b.ny};
  const double* __restrict__ phi = a.phi;
  double pp[3], pm[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    pp[d] = a.dp[d][q];
    pm[d] = a.dm[d][q];
  }
  const double vel = a.vel_n[q];
  double ppb[3] = {0, 0, 0}, pmb[3] = {0, 0, 0};
  if (moving(vel)) {
    double velb;
    godunov_bwd(vel, pp, pm, ppb, pmb, velb);
    a.adj_vel[q] += mulz(w, velb);
  }
  const double vxyz[3] = {a.vx[q], a.vy[q], a.vz[q]};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const bool up = qss_emu::ge0(vxyz[d]);
    if (nonzero(vxyz[d])) (up ? pmb[d] : ppb[d]) -= vxyz[d];
    a.bp[d][q] = mulz(w, ppb[d]);
    a.bm[d][q] = mulz(w, pmb[d]);
  }
  double out[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  // nothing flows through b kappa where b is zero (grain interiors)
  const double bco = a.bcoef[q];
  if (nonzero(w) && nonzero(bco)) {
    const double fx = a.fac[0], fy = a.fac[1], fz = a.fac[2];
    // first differences as the forward computes them (the threshold test on
    // their squares must take the forward's branch)
    const double phx = mulz(phi[q + st[0]] - phi[q - st[0]], fx);
    const double phy = mulz(phi[q + st[1]] - phi[q - st[1]], fy);
    const double phz = mulz(phi[q + st[2]] - phi[q - st[2]], fz);
    const double sx = mulz(phx, phx), sy = mulz(phy, phy), sz = mulz(phz, phz);
    const double grad = __dadd_rn(__dadd_rn(sx, sy), sz);
    if (qss_emu::bits(grad) >= 0x3ee4f8b588e368f1ull) {  // grad >= 1e-5
      const double cc = phi[q];
      const double pxx = mulz(fma(-2.0, cc, phi[q + 2 * st[0]] + phi[q - 2 * st[0]]), a.f2[0]);
      const double pyy = mulz(fma(-2.0, cc, phi[q + 2 * st[1]] + phi[q - 2 * st[1]]), a.f2[1]);
      const double pzz = mulz(fma(-2.0, cc, phi[q + 2 * st[2]] + phi[q - 2 * st[2]]), a.f2[2]);
      const double pxy = mulz(phi[q + st[0] + st[1]] + phi[q - st[0] - st[1]] - phi[q - st[0] + st[1]] -
                              phi[q + st[0] - st[1]], a.f2[3]);
      const double pxz = mulz(phi[q + st[0] + st[2]] + phi[q - st[0] - st[2]] - phi[q - st[0] + st[2]] -
                              phi[q + st[0] - st[2]], a.f2[4]);
      const double pyz = mulz(phi[q + st[1] + st[2]] + phi[q - st[1] - st[2]] - phi[q - st[1] + st[2]] -
                              phi[q + st[1] - st[2]], a.f2[5]);
      const double yz = sy + sz, xz = sx + sz, xy = sx + sy;
      const double hxy = mulz(phx, phy), hxz = mulz(phx, phz), hyz = mulz(phy, phz);
      // kappa numerator (3d.f:2337-2379), regrouped
      const double curv = fma(pxx, yz, fma(pyy, xz, mulz(pzz, xy))) -
                          2 * fma(pxy, hxy, fma(pxz, hxz, mulz(pyz, hyz)));
      const double ig = qss_emu::div(1.0, grad);
      const double cb = mulz(mulz(w, bco), ig);         // d RHS / d numerator
      const double gb = -mulz(mulz(cb, curv), ig);      // d RHS / d grad
      const double c2 = cb + cb;
      const double cx = mulz(c2, phx), cy = mulz(c2, phy), cz = mulz(c2, phz), g2 = gb + gb;
      // 2 (ph (cb (the two second differences across) + gb) - cb (mixed terms)) f
      out[0] = mulz(fma(cx, pyy + pzz, fma(g2, phx, -fma(pxy, cy, mulz(pxz, cz)))), fx);
      out[1] = mulz(fma(cy, pxx + pzz, fma(g2, phy, -fma(pxy, cx, mulz(pyz, cz)))), fy);
      out[2] = mulz(fma(cz, pxx + pyy, fma(g2, phz, -fma(pxz, cx, mulz(pyz, cy)))), fz);
      out[3] = mulz(mulz(cb, yz), a.f2[0]);
      out[4] = mulz(mulz(cb, xz), a.f2[1]);
      out[5] = mulz(mulz(cb, xy), a.f2[2]);
      out[6] = -mulz(mulz(cx, phy), a.f2[3]);
      out[7] = -mulz(mulz(cx, phz), a.f2[4]);
      out[8] = -mulz(mulz(cy, phz), a.f2[5]);
    }
  }
#pragma unroll
  for (int o = 0; o < 9; o++) a.cc[o * a.npts + q] = out[o];
}

// Voxels whose normal term is carried from an earlier voxel (|vel_n| < 1e-5,
// 3d.f:459-486): their weight times the source voxel's Godunov partials goes
// to the source's derivative adjoints (atomics; such voxels are rare).  Runs
// after k_adj_point, which writes the source's own values.
__global__ void __launch_bounds__(128) k_adj_carry(AdjPointArgs a) {
  const Box& b = a.b;
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t q = b.idx(i, j, k);
  if (moving(a.vel_n[q])) return;
  const double w = a.coef_l * a.lam_in[q];
  const int src = a.nsrc[q];
  if (w == 0.0 || src < 0) return;
  double sp[3], sm[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    sp[d] = a.dp[d][src];
    sm[d] = a.dm[d][src];
  }
  double spb[3] = {0, 0, 0}, smb[3] = {0, 0, 0}, velb;
  godunov_bwd(a.vel_n[src], sp, sm, spb, smb, velb);
  atomicAdd(a.adj_vel + src, w * velb);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (spb[d] != 0.0) atomicAdd(a.bp[d] + src, w * spb[d]);
    if (smb[d] != 0.0) atomicAdd(a.bm[d] + src, w * smb[d]);
  }
}

// Reverse of the WENO5 one-sided derivatives along one axis (3d.f:1962-2246),
// one face window at a time.  With v(m) = (phi(m) - phi(m-1)) inv the scaled
// difference of face m, the minus derivative of voxel c and the plus
// derivative of voxel c-1 are the same WENO5 reconstruction of the window
// u0..u4 = v(c-2..c+2), read in opposite directions: they share the three
// smoothness indicators (S1+ = S3-, S2+ = S2-, S3+ = S1-) and eps, and
// differ in the ideal weights (0.1, 0.6, 0.3 against 0.3, 0.6, 0.1 on
// S1, S2, S3) and the candidate stencils.  Per window the adjoints of both
// (the minus adjoint of voxel c, the plus adjoint of voxel c-1) are pushed
// to the five faces at once:
//   d value / d T_k = -2 w_k (p_k - value) / T_k,   T_k = S_k + eps,
//   d value / d p_k = w_k,  d eps / d u_j = 2e-6 u_j at the maximum square
// (the later operand of the reference's MAX chain on ties, per side).
// A block holds a tile of 4 lines x up to 58 points and goes through it in
// phases, each value once in shared memory: faces v, centre differences a, the
// windows (their adjoints of five faces and three centre differences, times six),
// the centres' sums, the faces' sums in a fixed order, and lam(p) += inv / 6 (F(p)
// - F(p+1)).  Only distances between the candidates count, so the candidates are
// taken relative to a midpoint, where they are multiples of the centre differences.  A tile recomputes the windows of 3 points on
// either side; tiles of 58 points make 64 windows of them, full warps.
// Bound: FP64 pipe, about 80 % of its time busy with 57 instructions a window and 15 a
// point (145 a window with the candidates as stencils of their own, products and
// comparisons on the FP64 pipe: 72^3, 150 us a pass against 92).  Full tiles and a
// remainder rather than equal ones: their windows are whole rounds of the block.
// With a thread walking a segment of a line instead (32 points and more, so that a 72^3 box
// had 324 warps for 608 schedulers) a pass took 0.30 ms.
struct AdjAxisArgs {
  Box b;
  const double* phi;
  const double* bp;
  const double* bm;
  double* lam;
  double inv;
  int len;  // points per tile
};
constexpr int kAdjL = 4, kAdjP = 58, kAdjThreads = 128;
constexpr int kAdjW = kAdjP + 6;   // windows p0-2 .. p0+P+3
constexpr int kAdjF = kAdjP + 10;  // faces p0-4 .. p0+P+5
constexpr int kAdjC = kAdjP + 8;   // centres p0-3 .. p0+P+4
constexpr size_t kAdjBytes = sizeof(double) * kAdjL * (kAdjF + kAdjC + 8 * kAdjW);
static_assert(kAdjBytes <= 48 * 1024, "dynamic shared memory without the opt-in attribute");

template <int AX>
__global__ void __launch_bounds__(kAdjThreads, 5) k_adj_axis(AdjAxisArgs a) {
  constexpr int L = kAdjL;
  extern __shared__ double adj_smem[];
  double* const sv = adj_smem;             // faces; later the face adjoints F
  double* const sa = sv + L * kAdjF;       // centre differences; later their terms' adjoints
  double* const sd = sa + L * kAdjC;       // [8][window]: d0 .. d4, bS1 .. bS3
  constexpr int W = L * kAdjW;
  const Box& b = a.b;
  const int line = threadIdx.x % L;
  int p, q, lo, hi, plast_line;
  if (AX == 0) {
    p = b.jlo + blockIdx.x * L + line;  // j
    q = b.klo + blockIdx.y;             // k
    plast_line = b.jhi;
    lo = b.ilo;
    hi = b.ihi;
  } else {
    p = b.ilo + blockIdx.x * L + line;  // i
    q = (AX == 1 ? b.klo : b.jlo) + blockIdx.y;
    plast_line = b.ihi;
    lo = (AX == 1) ? b.jlo : b.klo;
    hi = (AX == 1) ? b.jhi : b.khi;
  }
  const bool line_ok = p <= plast_line;
  if (!line_ok) p = plast_line;  // loads stay in the box; nothing is stored
  const int p0 = lo - 3 + (int)blockIdx.z * a.len;  // points lo-3 .. hi+3 in all
  int tp = hi + 3 - p0 + 1;
  if (tp > a.len) tp = a.len;
  const int64_t base = AX == 0 ? b.idx(0, p, q) : (AX == 1 ? b.idx(p, 0, q) : b.idx(p, q, 0));
  const int64_t stride = AX == 0 ? 1 : (AX == 1 ? (int64_t)b.nx : (int64_t)b.nx * b.ny);
  const double* __restrict__ phi = a.phi;
  const double inv = a.inv, inv6 = a.inv * (1.0 / 6.0);
  const int last = (AX == 0 ? b.nx : (AX == 1 ? b.ny : b.nz)) - 1;
  // loads outside the line only feed windows without adjoints
  auto ld = [&](int m) -> double {
    const int mm = m < 0 ? 0 : (m > last ? last : m);
    return __ldg(phi + base + (int64_t)mm * stride);
  };
  auto ldbar = [&](const double* arr, int m) -> double {
    return (m >= lo && m <= hi) ? __ldg(arr + base + (int64_t)m * stride) : 0.0;
  };
  using qss_emu::bits;
  for (int it = threadIdx.x; it < (tp + 10) * L; it += kAdjThreads) {
    const int m = p0 - 4 + it / L;
    sv[it] = (ld(m) - ld(m - 1)) * inv;
  }
  __syncthreads();
  // a(m) = v(m-1) - 2 v(m) + v(m+1); its term 13/12 a^2 enters S1 of window m+1,
  // S2 of window m and S3 of window m-1
  for (int it = threadIdx.x; it < (tp + 8) * L; it += kAdjThreads) {
    const double* const v = sv + it;
    sa[it] = (v[0] - 2.0 * v[L]) + v[2 * L];
  }
  __syncthreads();
  // windows with an adjoint: c = lo .. hi + 1; the others add nothing
  const int w0 = (p0 - 2 < lo ? lo - (p0 - 2) : 0) * L, w1 = (p0 + tp + 3 > hi + 1 ? hi + 1 - (p0 - 2) + 1 : tp + 6) * L;
  for (int it = threadIdx.x; it < (tp + 6) * L; it += kAdjThreads) {
    if (it >= w0 && it < w1) continue;
#pragma unroll
    for (int o = 0; o < 8; o++) sd[o * W + it] = 0.0;
  }
  for (int it = w0 + threadIdx.x; it < w1; it += kAdjThreads) {
    const int c = p0 - 2 + it / L;
    double d0 = 0, d1 = 0, d2 = 0, d3 = 0, d4 = 0, A1 = 0, A2 = 0, A3 = 0;
    double gm = ldbar(a.bm, c), gp = ldbar(a.bp, c - 1);
    if (((bits(gm) | bits(gp)) << 1) != 0) {
      // Adjoints fall off by orders of magnitude per voxel ahead of the front.  Below
      // 2^-160 the window, linear in them, is evaluated on a multiple: their products
      // would leave the range of the integer ones, and one lane's FP64 instruction costs
      // its warp as much as 32.
      using qss_emu::hi32;
      using qss_emu::scale2;
      const uint32_t top = max(hi32(gm) & 0x7fffffffu, hi32(gp) & 0x7fffffffu);
      const int up2 = top >= 0x35f00000u ? 0 : (top >= 0x23300000u ? 300 : 700);
      if (up2) {
        gm = scale2(gm, up2);
        gp = scale2(gp, up2);
      }
      const double* const v = sv + it;
      const double u0 = v[0], u1 = v[L], u2 = v[2 * L], u3 = v[3 * L], u4 = v[4 * L];
      const double* const aa = sa + it;
      // eps and the position of the largest square (of the largest magnitude) for
      // each reading direction
      const uint64_t b0 = bits(u0) << 1, b1 = bits(u1) << 1, b2 = bits(u2) << 1, b3 = bits(u3) << 1,
                     b4 = bits(u4) << 1;
      uint64_t mx = b0;
      int im = 0;  // minus: u0 .. u4, later wins ties
      if (b1 >= mx) { mx = b1; im = 1; }
      if (b2 >= mx) { mx = b2; im = 2; }
      if (b3 >= mx) { mx = b3; im = 3; }
      if (b4 >= mx) { mx = b4; im = 4; }
      int ip = 0;  // plus: u4 .. u0, later wins ties
      if (b0 == mx) ip = 0;
      else if (b1 == mx) ip = 1;
      else if (b2 == mx) ip = 2;
      else if (b3 == mx) ip = 3;
      else ip = 4;
      const double um = im == 0 ? u0 : im == 1 ? u1 : im == 2 ? u2 : im == 3 ? u3 : u4;
      auto sq = [](double x) { return mulz(x, x); };
      const double eps = fma(1e-6, sq(um), 1.0e-35);
      const double a1 = aa[0], a2 = aa[L], a3 = aa[2 * L];
      const double s1 = u2 - u1, s2 = u3 - u2, e2 = s1 + s2;
      const double b1t = fma(2.0, s1, a1), b3t = fma(-2.0, s2, a3);  // u0 - 4 u1 + 3 u2, 3 u2 - 4 u3 + u4
      const double r1 = qss_emu::div(1.0, fma(k1312, sq(a1), fma(0.25, sq(b1t), eps))),
                   r2 = qss_emu::div(1.0, fma(k1312, sq(a2), fma(0.25, sq(e2), eps))),
                   r3 = qss_emu::div(1.0, fma(k1312, sq(a3), fma(0.25, sq(b3t), eps)));
      const double q1 = mulz(r1, r1), q2 = mulz(r2, r2), q3 = mulz(r3, r3);
      const double am2 = mulz(0.6, q2);
      const double am1 = mulz(0.1, q1), am3 = mulz(0.3, q3);  // minus: 0.1, 0.6, 0.3
      const double ap1 = mulz(0.3, q1), ap3 = mulz(0.1, q3);  // plus (on S1, S2, S3): 0.3, 0.6, 0.1
      const double iam = qss_emu::div(1.0, am1 + am2 + am3), iap = qss_emu::div(1.0, ap1 + am2 + ap3);
      // the weights first: in flat parts the sums are 1e70 and their inverses out of range beside gm
      const double wm1 = mulz(am1, iam), wm2 = mulz(am2, iam), wm3 = mulz(am3, iam);
      const double wp1 = mulz(ap1, iap), wp2 = mulz(am2, iap), wp3 = mulz(ap3, iap);
      // candidates, six times their distance from (u2 + u3) / 2 (minus) and
      // (u1 + u2) / 2 (plus): c1, -a2, -a3 and -a1, -a2, c3
      const double a23 = -3.0 * a2, c1 = fma(2.0, a1, a23), c3 = fma(2.0, a3, a23);
      const double vm = fma(-wm3, a3, fma(-wm2, a2, mulz(wm1, c1)));
      const double vp = fma(-wp1, a1, fma(-wp2, a2, mulz(wp3, c3)));
      // three times the adjoints of the indicators, without their sign: P_k (value - p_k) r_k for
      // each direction and both
      const double P1 = mulz(gm, wm1), P2 = mulz(gm, wm2), P3 = mulz(gm, wm3);
      const double Q1 = mulz(gp, wp1), Q2 = mulz(gp, wp2), Q3 = mulz(gp, wp3);
      const double m1 = mulz(r1, mulz(P1, vm - c1)), m2 = mulz(r2, mulz(P2, vm + a2)), m3 = mulz(r3, mulz(P3, vm + a3));
      const double n1 = mulz(r1, mulz(Q1, vp + a1)), n2 = mulz(r2, mulz(Q2, vp + a2)), n3 = mulz(r3, mulz(Q3, vp - c3));
      const double bS1 = m1 + n1, bS2 = m2 + n2, bS3 = m3 + n3;
      // six times everything from here on: adjoints of the centres a1, a2, a3 ...
      A1 = fma(bS1, fma(2.0 * k136, a1, b1t), fma(2.0, P1, -Q1));
      A2 = fma(2.0 * k136, mulz(bS2, a2), fma(-3.0, P1 + Q3, -(P2 + Q2)));
      A3 = fma(bS3, fma(2.0 * k136, a3, b3t), fma(2.0, Q3, -P3));
      // ... of the differences s1, s2 ...
      const double be = mulz(bS2, e2);
      const double g1 = fma(-3.0, gp, fma(2.0, mulz(bS1, b1t), be)), g2 = fma(3.0, gm, fma(-2.0, mulz(bS3, b3t), be));
      // ... and of the faces
      d1 = -g1;
      d2 = fma(6.0, gm + gp, g1 - g2);
      d3 = g2;
      // eps = 1e-6 max(u^2) + 1e-35, per reading direction; two faces of exactly the same
      // magnitude, where the directions differ, are common enough not to branch on
      const double up = ip == 0 ? u0 : ip == 1 ? u1 : ip == 2 ? u2 : ip == 3 ? u3 : u4;
      const double cm = mulz(mulz(4e-6, um), (m1 + m2) + m3), cp = mulz(mulz(4e-6, up), (n1 + n2) + n3);
      const double cs = im == ip ? cm + cp : cm;
      auto ex = [&](int j) { return j == im ? cs : (j == ip ? cp : 0.0); };
      d0 = ex(0);
      d1 += ex(1);
      d2 += ex(2);
      d3 += ex(3);
      d4 = ex(4);
      if (up2) {
        d0 = scale2(d0, -up2);
        d1 = scale2(d1, -up2);
        d2 = scale2(d2, -up2);
        d3 = scale2(d3, -up2);
        d4 = scale2(d4, -up2);
        A1 = scale2(A1, -up2);
        A2 = scale2(A2, -up2);
        A3 = scale2(A3, -up2);
      }
    }
    sd[it] = d0;
    sd[W + it] = d1;
    sd[2 * W + it] = d2;
    sd[3 * W + it] = d3;
    sd[4 * W + it] = d4;
    sd[5 * W + it] = A1;
    sd[6 * W + it] = A2;
    sd[7 * W + it] = A3;
  }
  __syncthreads();
  // adjoint of a(m) for the centres p0-1 .. p0+tp+1 the tile's faces touch (window
  // index w = m - p0 + 2): it is a1 of window w+1, a2 of w, a3 of w-1
  for (int it = threadIdx.x; it < (tp + 3) * L; it += kAdjThreads) {
    const int w = it + L;  // the window of centre m = p0 - 1 + it / L
    sa[it + 2 * L] = (sd[5 * W + w + L] + sd[6 * W + w]) + sd[7 * W + w - L];  // centre m is entry m - p0 + 3
  }
  __syncthreads();
  // face f = p0 .. p0+tp: slot k of window f + 2 - k, and the three centres on it
  for (int it = threadIdx.x; it < (tp + 1) * L; it += kAdjThreads) {
    const double* const d = sd + it + 4 * L;  // window f + 2
    const double* const c = sa + it + 2 * L;  // centre f - 1
    double F = ((d[0] + d[W - L]) + (d[2 * W - 2 * L] + d[3 * W - 3 * L])) + d[4 * W - 4 * L];
    F += fma(-2.0, c[L], c[0] + c[2 * L]);
    sv[it] = F;  // the faces' v is no longer read
  }
  __syncthreads();
  if (!line_ok) return;
  for (int it = threadIdx.x; it < tp * L; it += kAdjThreads)
    a.lam[base + (int64_t)(p0 + it / L) * stride] += inv6 * (sv[it] - sv[it + L]);
}

// lam_out[p] += coef * lam_in[p] (fill box) + the curvature partials of the
// fill-box voxels whose central stencil holds p, in a fixed order:
//   cc[0..2] first derivatives (+ at p-e, - at p+e), cc[3..5] second
//   derivatives (+ at p -+ 2e, -2 at p), cc[6..8] mixed xy, xz, yz
//   (+ at p -+ (e1 + e2), - at p + (e1 - e2) and p - (e1 - e2))
__global__ void k_adj_curv(Box b, const double* __restrict__ cc, int64_t npts, const double* lam_in, double coef,
                           double* lam_out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npts; p += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(p % b.nx);
    const int64_t r = p / b.nx;
    const int j = (int)(r % b.ny), k = (int)(r / b.ny);
    auto in_fill = [&](int ii, int jj, int kk) {
      return ii >= b.ilo && ii <= b.ihi && jj >= b.jlo && jj <= b.jhi && kk >= b.klo && kk <= b.khi;
    };
    auto at = [&](int o, int di, int dj, int dk) -> double {
      const int ii = i + di, jj = j + dj, kk = k + dk;
      return in_fill(ii, jj, kk) ? cc[o * npts + b.idx(ii, jj, kk)] : 0.0;
    };
    double s = in_fill(i, j, k) ? coef * lam_in[p] : 0.0;
    s += at(0, -1, 0, 0) - at(0, 1, 0, 0);
    s += at(1, 0, -1, 0) - at(1, 0, 1, 0);
    s += at(2, 0, 0, -1) - at(2, 0, 0, 1);
    s += at(3, -2, 0, 0) + at(3, 2, 0, 0) - 2.0 * at(3, 0, 0, 0);
    s += at(4, 0, -2, 0) + at(4, 0, 2, 0) - 2.0 * at(4, 0, 0, 0);
    s += at(5, 0, 0, -2) + at(5, 0, 0, 2) - 2.0 * at(5, 0, 0, 0);
    s += at(6, -1, -1, 0) + at(6, 1, 1, 0) - at(6, 1, -1, 0) - at(6, -1, 1, 0);
    s += at(7, -1, 0, -1) + at(7, 1, 0, 1) - at(7, 1, 0, -1) - at(7, -1, 0, 1);
    s += at(8, 0, -1, -1) + at(8, 0, 1, 1) - at(8, 0, 1, -1) - at(8, 0, -1, 1);
    lam_out[p] += s;
  }
}

// adjoint of the ghost extrapolation of one face sweep: per line, the ghost
// layers' adjoints go to the two boundary points they were built from, and
// are cleared.  axis 2: all (i, j); axis 1: all i, k in the fill box;
// axis 0: j, k in the fill box (the forward's sweep domains).
// With t = sign(f) sign(f - g) in {-1, 0, 1}, a layer at distance d adds lam (1 +
// t d) to f and -lam t d to g: two sums per side, all layers' loads first.
__device__ __forceinline__ void extrap_bwd(double* lam, int64_t p0, int64_t st, int layers, double f, double g,
                                           double& fb, double& gb) {
  double s = 0, sd = 0;
  for (int m0 = 0; m0 < layers; m0 += 3) {
    double x[3];
#pragma unroll
    for (int m = 0; m < 3; m++) x[m] = m0 + m < layers ? lam[p0 + (m0 + m) * st] : 0.0;
#pragma unroll
    for (int m = 0; m < 3; m++) {
      s += x[m];
      sd += x[m] * (double)(m0 + m + 1);
      if (m0 + m < layers) lam[p0 + (m0 + m) * st] = 0.0;
    }
  }
  const double d = f - g;
  const bool neg = (int64_t)(qss_emu::bits(f) ^ qss_emu::bits(d)) < 0;
  const double t = (qss_emu::bits(d) << 1) == 0 ? 0.0 : (neg ? -sd : sd);
  fb = s + t;
  gb = -t;
}

__global__ void k_adj_bc(Box b, int axis, const double* __restrict__ val, double* lam) {
  int n1, n2;
  if (axis == 2) {
    n1 = b.nx;
    n2 = b.ny;
  } else if (axis == 1) {
    n1 = b.nx;
    n2 = b.fbz();
  } else {
    n1 = b.fby();
    n2 = b.fbz();
  }
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n1 * n2) return;
  const int u = t % n1, w = t / n1;
  int64_t base, st;
  int lo, hi, len;
  if (axis == 2) {
    base = b.idx(u, w, 0);
    st = (int64_t)b.nx * b.ny;
    lo = b.klo;
    hi = b.khi;
    len = b.nz;
  } else if (axis == 1) {
    base = b.idx(u, 0, b.klo + w);
    st = b.nx;
    lo = b.jlo;
    hi = b.jhi;
    len = b.ny;
  } else {
    base = b.idx(0, b.jlo + u, b.klo + w);
    st = 1;
    lo = b.ilo;
    hi = b.ihi;
    len = b.nx;
  }
  double blo, blo1, bhi, bhi1;
  const double flo = val[base + lo * st], flo1 = val[base + (lo + 1) * st];
  const double fhi = val[base + hi * st], fhi1 = val[base + (hi - 1) * st];
  extrap_bwd(lam, base + (lo - 1) * st, -st, lo, flo, flo1, blo, blo1);
  extrap_bwd(lam, base + (hi + 1) * st, st, len - 1 - hi, fhi, fhi1, bhi, bhi1);
  lam[base + lo * st] += blo;
  lam[base + (lo + 1) * st] += blo1;
  lam[base + hi * st] += bhi;
  lam[base + (hi - 1) * st] += bhi1;
}

// adjoint of phi = max(mask - overlap, s): passes where s was kept
__global__ void k_adj_impose(int64_t n, const double* __restrict__ s, const double* __restrict__ mask,
                             double overlap, const double* lam_in, double* lam_out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const double t = mask[p] - overlap;
    lam_out[p] = (t > s[p]) ? 0.0 : lam_in[p];
  }
}

// loss contributions (H(phi) - target)^2 in loop order, and the adjoint of phi^T
__global__ void k_adj_loss(Box b, const double* __restrict__ phi, const double* __restrict__ target, double eps,
                           double* contrib, double* lam) {
  const int64_t n = (int64_t)b.fbx() * b.fby() * b.fbz();
  const double pi = 3.14159265358979323846;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = b.ilo + (int)(q % b.fbx());
    const int64_t r = q / b.fbx();
    const int j = b.jlo + (int)(r % b.fby());
    const int k = b.klo + (int)(r / b.fby());
    const int64_t p = b.idx(i, j, k);
    const double x = phi[p];
    const double H = qss_heaviside(x, eps);
    const double dH = (x > -eps && x < eps) ? (1.0 + portable_cos(pi * x / eps)) / (2 * eps) : 0.0;
    const double d = H - target[p];
    contrib[q] = d * d;
    lam[p] = 2.0 * d * dH;
  }
}

// lam_out += coef * lam_in on the fill box
__global__ void k_axpy_fill(Box b, const double* __restrict__ lam_in, double coef, double* lam_out) {
  const int64_t n = b.npts();
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(p % b.nx);
    const int64_t r = p / b.nx;
    const int j = (int)(r % b.ny), k = (int)(r / b.ny);
    if (i >= b.ilo && i <= b.ihi && j >= b.jlo && j <= b.jhi && k >= b.klo && k <= b.khi)
      lam_out[p] += coef * lam_in[p];
  }
}

// d vel_n / d theta = s h2 sin(theta) |grad mask| (from setVarNorm3dTheta)
__global__ void k_adj_theta(Box b, const double* __restrict__ mask, const double* __restrict__ mx,
                            const double* __restrict__ my, const double* __restrict__ mz,
                            const double* __restrict__ theta, const double* __restrict__ adj_vel, double dx,
                            double* grad) {
  const int i = b.ilo + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.jlo + blockIdx.y * blockDim.y + threadIdx.y;
  const int k = b.klo + blockIdx.z * blockDim.z + threadIdx.z;
  if (i > b.ihi || j > b.jhi || k > b.khi) return;
  const int64_t c = b.idx(i, j, k);
  const double eps_var = 1.5 * dx;
  const double m = mask[c];
  const double h2 = qss_heaviside(m, eps_var);
  const double absgrad = sqrt(mx[c] * mx[c] + my[c] * my[c] + mz[c] * mz[c]);
  const double x = sqrt(m * m + absgrad * dx * absgrad * dx);
  const double s = m / x;
  grad[c] = adj_vel[c] * s * h2 * portable_sin(theta[c]) * absgrad;
}

// wgt = coef * lam on the fill box, 0 elsewhere
__global__ void k_scale_fill(Box b, const double* __restrict__ lam, double coef, double* wgt) {
  const int64_t n = b.npts();
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(p % b.nx);
    const int64_t r = p / b.nx;
    const int j = (int)(r % b.ny), k = (int)(r / b.ny);
    const bool fill = i >= b.ilo && i <= b.ihi && j >= b.jlo && j <= b.jhi && k >= b.klo && k <= b.khi;
    wgt[p] = fill ? coef * lam[p] : 0.0;
  }
}

unsigned g1(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 152 * 16) b = 152 * 16;
  return (unsigned)(b < 1 ? 1 : b);
}

// the call's stream and, on it, its device arrays; an exception may leave work of
// either stream in flight, which is waited for before they go
struct DBufs {
  cudaStream_t s = nullptr;
  std::vector<std::pair<void*, size_t>> ptrs;
  bool done = false;  // every stream has been waited for
  DBufs() { QSS_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)); }
  DBufs(const DBufs&) = delete;
  DBufs& operator=(const DBufs&) = delete;
  template <class T = double>
  T* get(int64_t n) {
    const size_t bytes = (size_t)(n > 0 ? n : 1) * sizeof(T);
    ptrs.reserve(ptrs.size() + 1);
    void* p = scratch_alloc(bytes, s);
    ptrs.emplace_back(p, bytes);
    return (T*)p;
  }
  ~DBufs() {
    if (!done) cudaDeviceSynchronize();
    for (const auto& p : ptrs) scratch_free(p.first, p.second, s);
    cudaStreamDestroy(s);
  }
};

struct AdjCtx {
  Box b;
  cudaStream_t s;
  int64_t n;
  double dx[3];
  Coef c;
  ImposeArgs im;
  Ctl* ctl;
  double* dp[3];
  double* dm[3];
};

// WENO5 derivatives of the three stage inputs of one step (6 arrays each)
struct StageDerivs {
  double* d[3][6] = {};  // [stage][dp x, y, z, dm x, y, z]
};

// the stage states (and, when device memory allows, the stage inputs' WENO5
// derivatives) of the steps of one checkpoint segment
struct SegBufs {
  std::vector<double*> sphi, ss1, ss2, ss3;
  std::vector<StageDerivs> sder;
  // one allocation for the whole segment (4 states and, with derivs, 18
  // derivative arrays per step, each starting on a 256-byte boundary): a
  // trajectory kept whole at 128^3 / 200 steps is 4400 arrays, and a
  // cudaMalloc / cudaFree pair per array (cudaFree synchronises the device)
  // is host time the GPU waits through
  void alloc(DBufs& buf, int steps, int64_t n, bool derivs) {
    const int64_t pitch = (n + 31) / 32 * 32;
    const int64_t per_step = 4 + (derivs ? 18 : 0);
    double* slab = buf.get(pitch * per_step * steps);
    auto next = [&]() {
      double* p = slab;
      slab += pitch;
      return p;
    };
    for (int q = 0; q < steps; q++) {
      sphi.push_back(next());
      ss1.push_back(next());
      ss2.push_back(next());
      ss3.push_back(next());
    }
    if (derivs) {
      sder.resize(steps);
      for (auto& sd : sder)
        for (int st = 0; st < 3; st++)
          for (int c = 0; c < 6; c++) sd.d[st][c] = next();
    }
  }
  const StageDerivs* keep(int q) const { return sder.empty() ? nullptr : &sder[q]; }
};

// one forward step from phin: stage states s1, s2, s3 (ghosts valid) and
// phi^{n+1}; with keep, the stage inputs' WENO5 derivatives stay in *keep
void fwd_step(AdjCtx& a, const double* phin, double* s1, double* s2, double* s3, double* next,
              const StageDerivs* keep = nullptr) {
  const Box& b = a.b;
  const double* in[3] = {phin, s1, s2};
  double* out[3] = {s1, s2, s3};
  for (int st = 0; st < 3; st++) {
    double* dp[3] = {a.dp[0], a.dp[1], a.dp[2]};
    double* dm[3] = {a.dm[0], a.dm[1], a.dm[2]};
    if (keep)
      for (int d = 0; d < 3; d++) {
        dp[d] = keep->d[st][d];
        dm[d] = keep->d[st][3 + d];
      }
    launch_weno_axes(a.s, b, in[st], a.dx[0], a.dx[1], a.dx[2], dp, dm, a.ctl);
    launch_weno_combine(a.s, st + 1, st == 2, b, a.dx[0], a.dx[1], a.dx[2], in[st], phin, out[st],
                        st == 2 ? next : nullptr, dp, dm, a.c, a.im, a.ctl);
    launch_ghost(a.s, b, out[st], st == 2 ? next : nullptr, a.im, a.ctl);
  }
}

}  // namespace

}  // namespace qss

using namespace qss;

namespace {

// shared by the forward-only and the adjoint entry points
int adjoint_run(Options* o, QSS_DataArrays* p, Grid* g, const double* theta, const double* target, int nsteps,
                double dt, int ckpt, double* loss, double* grad_theta, double* phi_out) {
  CallScope scope;
  try {
    ensure_device();
    if (!o || !p || !g || !theta || !target || !loss || nsteps < 0 || !(dt > 0) || !p->phi || !p->mask)
      throw Error(QSSGPU_ERR_ARG, "qssgpu adjoint: bad arguments");
    validate_grid(g);
    if (ckpt <= 0 || ckpt > nsteps) ckpt = nsteps > 0 ? nsteps : 1;
    const Box b = box_of(g);
    const int64_t n = b.npts();
    const size_t bytes = (size_t)n * sizeof(double);
    AdjCtx a;
    a.b = b;
    a.n = n;
    for (int d = 0; d < 3; d++) a.dx[d] = g->dx[d];
    DBufs buf;
    a.s = buf.s;
    double* mask = buf.get(n);
    double* mxyz[3] = {buf.get(n), buf.get(n), buf.get(n)};
    double* th = buf.get(n);
    double* tgt = buf.get(n);
    double* vel = buf.get(n);
    double* bco = buf.get(n);
    double* vv[3] = {buf.get(n), buf.get(n), buf.get(n)};
    for (int d = 0; d < 3; d++) {
      a.dp[d] = buf.get(n);
      a.dm[d] = buf.get(n);
    }
    int* nsrc = buf.get<int>(n);
    const int64_t rows = (int64_t)b.fby() * b.fbz();
    int* rowlast = buf.get<int>(rows);
    int* carry = buf.get<int>(rows);
    unsigned long long* cnt = buf.get<unsigned long long>(1);
    unsigned long long* red = buf.get<unsigned long long>(4);
    a.ctl = buf.get<Ctl>(1);
    QSS_CK(cudaMemcpyAsync(mask, p->mask, bytes, cudaMemcpyHostToDevice, a.s));
    QSS_CK(cudaMemcpyAsync(th, theta, bytes, cudaMemcpyHostToDevice, a.s));
    QSS_CK(cudaMemcpyAsync(tgt, target, bytes, cudaMemcpyHostToDevice, a.s));
    // coefficients as drain_model3d sets them (3d.f:13-298)
    launch_central_grad(a.s, b, mask, mxyz[0], mxyz[1], mxyz[2], g->dx[0], g->dx[1], g->dx[2]);
    launch_setvarcurvadv(a.s, b, mask, mxyz[0], mxyz[1], mxyz[2], bco, vv[0], vv[1], vv[2], o->b, g->dx[0], red);
    launch_setvarnorm(a.s, b, mask, mxyz[0], mxyz[1], mxyz[2], vel, o->a, th, o->theta, g->dx[0]);
    launch_nsrc(a.s, b, vel, nsrc, 1, rowlast, carry, cnt);
    Ctl init{};
    init.dt = dt;
    init.active = 1;
    init.tplot = 1e300;
    QSS_CK(cudaMemcpyAsync(a.ctl, &init, sizeof(Ctl), cudaMemcpyHostToDevice, a.s));
    a.c = Coef{};
    a.c.vel_n = vel;
    a.c.b = bco;
    a.c.vx = vv[0];
    a.c.vy = vv[1];
    a.c.vz = vv[2];
    a.c.nsrc = nsrc;
    a.im = ImposeArgs{mask, nullptr, nullptr, o->overlap, 0};

    const bool want_grad = grad_theta != nullptr;
    const int nseg = (nsteps + ckpt - 1) / ckpt;
    const int last0 = (nseg - 1) * ckpt;  // first step of the last segment
    // checkpoints phi^{k ckpt} of the segments before the last; the segment
    // buffers hold the stage states of one segment (the last one straight
    // from this forward pass, the others recomputed in the backward pass)
    std::vector<double*> cp(nseg, nullptr);
    // segment buffers; with two sets (when device memory allows) segment k-1
    // is recomputed on a second stream while the reverse sweep runs over
    // segment k
    SegBufs sets[2];
    int nsets = 0;
    if (want_grad) {
      for (int k = 0; k < nseg - 1; k++) cp[k] = buf.get(n);
      size_t free_b = 0, total_b = 0;
      QSS_CK(cudaMemGetInfo(&free_b, &total_b));
      free_b += scratch_idle_bytes();
      const double per_set = (double)ckpt * (4 + 18) * bytes;
      const double rest = (double)(15 + 8) * bytes;
      const bool derivs = per_set + rest < 0.6 * (double)free_b;
      // (two sets need the kept derivatives: without them both streams
      // would share the derivative scratch)
      nsets = (derivs && nseg > 1 && 2 * per_set + rest < 0.6 * (double)free_b) ? 2 : 1;
      for (int k = 0; k < nsets; k++) sets[k].alloc(buf, ckpt, n, derivs);
    }
    double* cur = buf.get(n);
    double* nxt = buf.get(n);
    double* t1 = buf.get(n);
    double* t2 = buf.get(n);
    double* t3 = buf.get(n);
    QSS_CK(cudaMemcpyAsync(cur, p->phi, bytes, cudaMemcpyHostToDevice, a.s));
    for (int st = 0; st < nsteps; st++) {
      if (want_grad && st % ckpt == 0 && st < last0)
        QSS_CK(cudaMemcpyAsync(cp[st / ckpt], cur, bytes, cudaMemcpyDeviceToDevice, a.s));
      if (want_grad && st >= last0) {
        SegBufs& sb = sets[(nseg - 1) % nsets];
        const int q = st - last0;
        if (q == 0) QSS_CK(cudaMemcpyAsync(sb.sphi[0], cur, bytes, cudaMemcpyDeviceToDevice, a.s));
        double* next = (st + 1 < nsteps) ? sb.sphi[q + 1] : nxt;
        fwd_step(a, sb.sphi[q], sb.ss1[q], sb.ss2[q], sb.ss3[q], next, sb.keep(q));
        cur = next;
      } else {
        fwd_step(a, cur, t1, t2, t3, nxt);
        std::swap(cur, nxt);
      }
    }
    // loss
    const int64_t nfb = (int64_t)b.fbx() * b.fby() * b.fbz();
    double* lc = buf.get(volume_scratch_doubles(nfb));
    double* lam = buf.get(n);
    double* dl = buf.get(1);
    launch_fill(a.s, n, lam, 0.0);
    k_adj_loss<<<g1(nfb), 256, 0, a.s>>>(b, cur, tgt, 1.5 * g->dx[0], lc, lam);
    launch_loop_sum(a.s, lc, nfb, lc + nfb, dl);
    QSS_CK(cudaMemcpyAsync(loss, dl, sizeof(double), cudaMemcpyDeviceToHost, a.s));
    if (phi_out) QSS_CK(cudaMemcpyAsync(phi_out, cur, bytes, cudaMemcpyDeviceToHost, a.s));
    QSS_CK(cudaGetLastError());
    if (!want_grad) {
      QSS_CK(cudaStreamSynchronize(a.s));
      buf.done = true;
      return 0;
    }
    // backward
    double* bars = buf.get(6 * n);  // adjoints of the plus / minus derivatives per axis
    double* cc = buf.get(9 * n);    // curvature partials
    launch_fill(a.s, 9 * n, cc, 0.0);  // outside the fill box they stay zero
    double* adj_vel = buf.get(n);
    double* lam3 = buf.get(n);
    double* lam2 = buf.get(n);
    double* lam1 = buf.get(n);
    double* lamphi = buf.get(n);
    double* wgt = buf.get(n);
    double* gth = buf.get(n);
    launch_fill(a.s, n, adj_vel, 0.0);
    AdjPointArgs ar;
    ar.b = b;
    ar.vel_n = vel;
    ar.bcoef = bco;
    ar.vx = vv[0];
    ar.vy = vv[1];
    ar.vz = vv[2];
    ar.nsrc = nsrc;
    for (int d = 0; d < 3; d++) ar.fac[d] = 0.5 / g->dx[d];
    ar.f2[0] = ar.fac[0] * ar.fac[0];
    ar.f2[1] = ar.fac[1] * ar.fac[1];
    ar.f2[2] = ar.fac[2] * ar.fac[2];
    ar.f2[3] = ar.fac[0] * ar.fac[1];
    ar.f2[4] = ar.fac[0] * ar.fac[2];
    ar.f2[5] = ar.fac[1] * ar.fac[2];
    for (int d = 0; d < 3; d++) {
      ar.bp[d] = bars + (int64_t)d * n;
      ar.bm[d] = bars + (int64_t)(3 + d) * n;
    }
    ar.cc = cc;
    ar.adj_vel = adj_vel;
    ar.npts = n;
    const dim3 blk(32, 4, 1);
    const dim3 grd((b.fbx() + 31) / 32, (b.fby() + 3) / 4, b.fbz());
    // the axis passes' tiles: full ones and a remainder; shorter tiles on small boxes, so
    // that four blocks per SM have about two rounds of them
    AdjAxisArgs axs[3];
    dim3 agrid[3];
    for (int d = 0; d < 3; d++) {
      const int len = (d == 0 ? b.fbx() : d == 1 ? b.fby() : b.fbz()) + 6;
      const unsigned lx = (unsigned)(((d == 0 ? b.fby() : b.fbx()) + kAdjL - 1) / kAdjL);
      const unsigned ly = (unsigned)(d == 2 ? b.fby() : b.fbz());
      int cap = kAdjP;
      while (cap > 16 && (int64_t)lx * ly * ((len + cap - 1) / cap) < 152 * 4 * 2) cap /= 2;
      axs[d] = AdjAxisArgs{b, nullptr, ar.bp[d], ar.bm[d], nullptr, 1.0 / g->dx[d], len < cap ? len : cap};
      agrid[d] = dim3(lx, ly, (unsigned)((len + axs[d].len - 1) / axs[d].len));
    }
    auto bc_bwd = [&](const double* val, double* l) {
      const int n2 = b.nx * b.ny, n1 = b.nx * b.fbz(), n0 = b.fby() * b.fbz();
      k_adj_bc<<<(n2 + 255) / 256, 256, 0, a.s>>>(b, 2, val, l);
      k_adj_bc<<<(n1 + 255) / 256, 256, 0, a.s>>>(b, 1, val, l);
      k_adj_bc<<<(n0 + 255) / 256, 256, 0, a.s>>>(b, 0, val, l);
    };
    // lam_out += coef_id * lam_in(fill) + J_L(in)^T (coef_l * lam_in)
    // stage_bwd's derivatives: kept from the forward pass (sd) or recomputed
    auto stage_bwd = [&](const double* in, const double* lam_in, double coef_id, double coef_l, double* lam_out,
                         const StageDerivs* sd, int st) {
      if (sd) {
        for (int d = 0; d < 3; d++) {
          ar.dp[d] = sd->d[st][d];
          ar.dm[d] = sd->d[st][3 + d];
        }
      } else {
        launch_weno_axes(a.s, b, in, a.dx[0], a.dx[1], a.dx[2], a.dp, a.dm, a.ctl);
        for (int d = 0; d < 3; d++) {
          ar.dp[d] = a.dp[d];
          ar.dm[d] = a.dm[d];
        }
      }
      ar.phi = in;
      ar.lam_in = lam_in;
      ar.coef_l = coef_l;
      k_adj_point<<<grd, blk, 0, a.s>>>(ar);
      k_adj_carry<<<grd, blk, 0, a.s>>>(ar);
      for (auto& x : axs) {
        x.phi = in;
        x.lam = lam_out;
      }
      k_adj_axis<0><<<agrid[0], kAdjThreads, kAdjBytes, a.s>>>(axs[0]);
      k_adj_axis<1><<<agrid[1], kAdjThreads, kAdjBytes, a.s>>>(axs[1]);
      k_adj_axis<2><<<agrid[2], kAdjThreads, kAdjBytes, a.s>>>(axs[2]);
      k_adj_curv<<<g1(n), 256, 0, a.s>>>(b, cc, n, lam_in, coef_id, lam_out);
    };
    // recomputation of segment k's states from its checkpoint, on stream st
    AdjCtx a2 = a;
    cudaStream_t s2 = a.s;
    if (nsets == 2) QSS_CK(cudaStreamCreateWithFlags(&s2, cudaStreamNonBlocking));
    a2.s = s2;
    cudaEvent_t recomputed[2] = {}, released[2] = {};
    for (int k = 0; k < 2; k++) {
      QSS_CK(cudaEventCreateWithFlags(&recomputed[k], cudaEventDisableTiming));
      QSS_CK(cudaEventCreateWithFlags(&released[k], cudaEventDisableTiming));
    }
    auto recompute = [&](int k) {
      SegBufs& sb = sets[k % nsets];
      AdjCtx& c = (nsets == 2) ? a2 : a;
      const int s0 = k * ckpt, s1 = std::min(nsteps, s0 + ckpt);
      QSS_CK(cudaMemcpyAsync(sb.sphi[0], cp[k], bytes, cudaMemcpyDeviceToDevice, c.s));
      for (int st = s0; st < s1; st++) {
        const int q = st - s0;
        double* next = (q + 1 < s1 - s0) ? sb.sphi[q + 1] : t1;
        fwd_step(c, sb.sphi[q], sb.ss1[q], sb.ss2[q], sb.ss3[q], next, sb.keep(q));
      }
      QSS_CK(cudaEventRecord(recomputed[k % 2], c.s));
    };
    if (nsets == 2 && nseg >= 2) {
      // the checkpoints and coefficients come from work queued on a.s
      QSS_CK(cudaEventRecord(released[(nseg - 1) % 2], a.s));
      QSS_CK(cudaStreamWaitEvent(s2, released[(nseg - 1) % 2], 0));
      recompute(nseg - 2);
    }
    for (int k = nseg - 1; k >= 0; k--) {
      const int s0 = k * ckpt, s1 = std::min(nsteps, s0 + ckpt);
      SegBufs& sb = sets[k % nsets];
      if (k < nseg - 1) {
        if (nsets == 2) QSS_CK(cudaStreamWaitEvent(a.s, recomputed[k % 2], 0));
        else recompute(k);
      }
      // the set of segment k-1 is the one the reverse sweep of segment k+1
      // has released: recompute it now, beside the sweep over segment k
      if (nsets == 2 && k >= 1 && k - 1 < nseg - 2) {
        QSS_CK(cudaStreamWaitEvent(s2, released[(k + 1) % 2], 0));
        recompute(k - 1);
      }
      for (int st = s1 - 1; st >= s0; st--) {
        const int q = st - s0;
        // phi^{n+1} = impose(BC(s3))
        k_adj_impose<<<g1(n), 256, 0, a.s>>>(n, sb.ss3[q], mask, o->overlap, lam, lam3);
        bc_bwd(sb.ss3[q], lam3);
        // stage 3: s3 = 1/3 phi^n + 2/3 (s2 + dt L(s2))
        launch_fill(a.s, n, lamphi, 0.0);
        launch_fill(a.s, n, lam2, 0.0);
        const StageDerivs* sd = sb.keep(q);
        stage_bwd(sb.ss2[q], lam3, 2.0 / 3.0, 2.0 / 3.0 * dt, lam2, sd, 2);
        k_axpy_fill<<<g1(n), 256, 0, a.s>>>(b, lam3, 1.0 / 3.0, lamphi);
        bc_bwd(sb.ss2[q], lam2);
        // stage 2: s2 = 3/4 phi^n + 1/4 (s1 + dt L(s1))
        launch_fill(a.s, n, lam1, 0.0);
        stage_bwd(sb.ss1[q], lam2, 0.25, 0.25 * dt, lam1, sd, 1);
        k_axpy_fill<<<g1(n), 256, 0, a.s>>>(b, lam2, 0.75, lamphi);
        bc_bwd(sb.ss1[q], lam1);
        // stage 1: s1 = phi^n + dt L(phi^n)
        stage_bwd(sb.sphi[q], lam1, 1.0, dt, lamphi, sd, 0);
        std::swap(lam, lamphi);
      }
      QSS_CK(cudaEventRecord(released[k % 2], a.s));
    }
    QSS_CK(cudaStreamSynchronize(s2));
    for (int k = 0; k < 2; k++) {
      cudaEventDestroy(recomputed[k]);
      cudaEventDestroy(released[k]);
    }
    if (nsets == 2) cudaStreamDestroy(s2);
    k_adj_theta<<<grd, blk, 0, a.s>>>(b, mask, mxyz[0], mxyz[1], mxyz[2], th, adj_vel, g->dx[0], gth);
    QSS_CK(cudaGetLastError());
    // gradient on the fill box, zero on the ghost layers
    k_scale_fill<<<g1(n), 256, 0, a.s>>>(b, gth, 1.0, wgt);
    QSS_CK(cudaMemcpyAsync(grad_theta, wgt, bytes, cudaMemcpyDeviceToHost, a.s));
    QSS_CK(cudaStreamSynchronize(a.s));
    unsigned long long host_err = 0;
    Ctl hc;
    QSS_CK(cudaMemcpy(&hc, a.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost));
    host_err = hc.err;
    buf.done = true;
    if (host_err) throw Error(QSSGPU_ERR_DEVICE_CHECK, "device check failed in the adjoint run");
    return 0;
  } catch (const std::exception& e) {
    return report_exception(e);
  }
}

}  // namespace

extern "C" {

// See include/lsmpqs_gpu.h.
int qssgpu_adjoint_theta(Options* o, QSS_DataArrays* p, Grid* g, const double* theta, const double* target,
                         int nsteps, double dt, int ckpt, double* loss, double* grad_theta) {
  if (!grad_theta) {
    set_error(QSSGPU_ERR_ARG, "qssgpu_adjoint_theta: grad_theta is NULL");
    return QSSGPU_ERR_ARG;
  }
  return adjoint_run(o, p, g, theta, target, nsteps, dt, ckpt, loss, grad_theta, nullptr);
}

// See include/lsmpqs_gpu.h.
int qssgpu_forward_theta(Options* o, QSS_DataArrays* p, Grid* g, const double* theta, const double* target,
                         int nsteps, double dt, double* loss, double* phi_out) {
  return adjoint_run(o, p, g, theta, target, nsteps, dt, 0, loss, nullptr, phi_out);
}

}  // extern "C"
