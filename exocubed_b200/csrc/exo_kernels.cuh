// exo_kernels.cuh -- the device code of one arithmetic build of the step.
//
// Included by kernels.cu (EXO_MIXED 0: everything in FP64, compiled without
// fused multiply-add so it reproduces the CPU restatement bit for bit) and by
// kernels_mixed.cu (EXO_MIXED 1: WENO5, the Riemann solvers and the flux
// divergence in FP32 -- EXO_FLUX_T -- while the hydrostatic decomposition, the
// implicit solve, the equation of state and the conserved state stay FP64;
// compiled with FMA).  EXO_KNS names the namespace of the build.
//
// One stage of SSPRK(3,3) is six launches, each one kernel over every
// member of a batch (a single atmosphere is a batch of one):
//   kb_flux_x1    per radial column: hydrostatic decomposition, WENO5 in x1,
//                 restore, Riemann solve -> x1 face fluxes         (exo3 only)
//   kb_flux_x23   per 32 lines of horizontal faces: WENO5 on both sides; at
//                 panel edges the outer state is the neighbour panel's own
//                 reconstruction, rotated into this panel's basis; Riemann
//                 solve -> x2/x3 fluxes
//   kb_update     per cell: RK register average, flux divergence, geometric
//                 source, gravity / Coriolis -> u (exo2) or du (exo3)
//   kb_implicit   per radial column: forward sweep of the block-tridiagonal
//                 vertical correction (5x5 or 3x3 blocks); kb_implicit_bwd: its
//                 back substitution, u += delta, AirParcel round trip on the
//                 last stage (exo3)
//   kb_prim_ghost per cell incl. ghosts: ConservedToPrimitive of the interior,
//                 of the ghost bands interpolated from the neighbour panels and
//                 of the reflected x1 ghosts; CFL time-step candidate
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <type_traits>
#include <utility>

#include <cuda_runtime.h>

#include "exo_internal.h"
#include "exo_mbarrier.cuh"

// 1: the x1 (radial) Riemann flux, its storage and its divergence stay FP64
// in the mixed build (the reconstruction of the perturbations stays FP32):
// the radial momentum flux carries the full hydrostatic pressure, whose
// difference across a cell is a few per cent of it, so FP32 storage of the
// flux loses the balance against gravity to cancellation
#ifndef EXO_X1_FLUX64
#define EXO_X1_FLUX64 EXO_MIXED
#endif

namespace exo {
namespace EXO_KNS {
namespace {

// the implicit solve's block arithmetic is FP64 or FP32 (template argument
// R): EXO_PREC_MIXED_F32_SOLVE builds and factors its blocks and keeps its
// back-substitution factors in FP32, EXO_PREC_MIXED and the FP64 build in
// FP64.  The state, the explicit update it corrects and the corrected state
// are FP64 in every case.  At the solver's time steps (vertical acoustic
// Courant numbers of tens) FP32 blocks change a corrected update by a few
// 1e-7 of itself.
__device__ __forceinline__ float abs_r(float x) { return fabsf(x); }
__device__ __forceinline__ double abs_r(double x) { return fabs(x); }
// EXO_IMPL_RCP_NR 1: the mixed build's FP64 implicit blocks take 1/x as PTX
// rcp.approx.ftz.f64 refined by two Newton-Raphson steps, r <- r + r (1 - x r)
// (Newton's method for 1/x: the relative error squares each step, so a
// seed good to 2^-14 or better ends within an ulp or two of 1/x), instead of
// an IEEE division.  The mixed build's primitive and
// update kernels take their reciprocals (density, sin^2, volume, radius)
// the same way.  The FP64 build divides.
#ifndef EXO_IMPL_RCP_NR
#define EXO_IMPL_RCP_NR 1
#endif
__device__ __forceinline__ double rcp_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  r = fma(r, e, r);
  e = fma(-x, r, 1.0);
  return fma(r, e, r);
}
__device__ __forceinline__ float inv_r(float x) { return 1.f / x; }
__device__ __forceinline__ double inv_r(double x) {
  if constexpr (EXO_IMPL_RCP_NR && EXO_MIXED) return rcp_nr(x);
  else return 1. / x;
}
__device__ __forceinline__ float sqrt_r(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_r(double x) { return sqrt(x); }
__device__ __forceinline__ float rsqrt_r(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsqrt_r(double x) { return rsqrt(x); }

constexpr double TINY_NUMBER = 1.0e-20;
constexpr double WENO_EPS = 1.0e-7;

__device__ __forceinline__ double sqr(double x) { return x * x; }
__device__ __forceinline__ float sqr(float x) { return x * x; }

// SSPRK(3,3) stage weights beta = 1, 1/4, 2/3
__device__ __forceinline__ double rk_beta(int stage) {
  return stage == 0 ? 1.0 : (stage == 1 ? 0.25 : 2.0 / 3.0);
}

__device__ __forceinline__ size_t idx(const DevView& v, int p, int n, int k, int j, int i) {
  return (size_t)row_place(v.nv, v.nc3, v.nc2, p, n, k, j) * (unsigned)v.nc1 + (unsigned)i;
}
__device__ __forceinline__ double geo(const DevView& v, int f, int p, int k, int j) {
  return v.geo[geo_place(v.nc3, v.nc2, f, p, k, j)];
}

// face-flux and primitive arrays in the type the flux kernels work in
template <class T> __device__ __forceinline__ T* flux_array(const DevView& v, int d);
template <> __device__ __forceinline__ double* flux_array<double>(const DevView& v, int d) {
  return v.flux[d];
}
template <> __device__ __forceinline__ float* flux_array<float>(const DevView& v, int d) {
  return v.flux32[d];
}
// the type of the x1 face fluxes for a build whose flux type is T
template <class T>
using X1Flux = std::conditional_t<(EXO_X1_FLUX64 != 0), double, T>;
template <class T> __device__ __forceinline__ const T* prim_array(const DevView& v);
template <> __device__ __forceinline__ const double* prim_array<double>(const DevView& v) {
  return v.w;
}
template <> __device__ __forceinline__ const float* prim_array<float>(const DevView& v) {
  return v.w32;
}

#if !EXO_MIXED
// a / b without a division's range checks, for b normal in 2^-400..2^400 and
// a quotient that is normal or zero: 1/b by two Newton steps from PTX's
// approximation, q = a r, and one remainder step (Markstein, IBM J. Res. Dev.
// 34, 1990).  The sum it rounds is within 2^-52 of an ulp of a/b, so the
// result is the IEEE quotient unless a/b lies that close to the middle of two
// doubles.
__device__ __forceinline__ double div_nr(double a, double b) {
  const double r = rcp_nr(b);
  const double q = a * r;
  return fma(fma(-b, q, a), r, q);
}
// WENO5's constants as operands from the constant bank (64-bit immediates
// take two instructions each)
__constant__ double kWeno[12] = {1.0 / 3.0, 7.0 / 6.0, 11.0 / 6.0, -1.0 / 6.0, 5.0 / 6.0,
                                 1.0 / 6.0, 13. / 12., 0.25, 1.0e-7, 0.1, 0.6, 0.3};
#endif
// interp_weno5(phip2, phip1, phi, phim1, phim2): the face value between the
// 2nd and 3rd argument (Jiang & Shu 1996; orientation of tests/test_weno.cpp)
template <class T>
__device__ __forceinline__ T weno5(T phip2, T phip1, T phi, T phim1, T phim2) {
#if !EXO_MIXED
  if constexpr (sizeof(T) == 8) {
    const double eps = kWeno[8];
    const double p0 = kWeno[0] * phim2 - kWeno[1] * phim1 + kWeno[2] * phi;
    const double p1 = kWeno[3] * phim1 + kWeno[4] * phi + kWeno[0] * phip1;
    const double p2 = kWeno[0] * phi + kWeno[4] * phip1 - kWeno[5] * phip2;
    const double b0 = kWeno[6] * sqr(phim2 - 2. * phim1 + phi) +
                      kWeno[7] * sqr(phim2 - 4. * phim1 + 3. * phi);
    const double b1 = kWeno[6] * sqr(phim1 - 2. * phi + phip1) + kWeno[7] * sqr(phim1 - phip1);
    const double b2 = kWeno[6] * sqr(phi - 2. * phip1 + phip2) +
                      kWeno[7] * sqr(3. * phi - 4. * phip1 + phip2);
    const double d0 = (b0 + eps) * (b0 + eps), d1 = (b1 + eps) * (b1 + eps),
                 d2 = (b2 + eps) * (b2 + eps);
    // every weight's denominator below 2^400 (they are above eps^2), and so the
    // five values within 2^105 of each other, and one of them below 2^400: the
    // divisions need no further checks.  NaN and infinity fail this.
    const unsigned top = max(max((unsigned)__double2hiint(d0), (unsigned)__double2hiint(d1)),
                             max((unsigned)__double2hiint(d2),
                                 (unsigned)__double2hiint(phi) & 0x7fffffffu));
    double a0, a1, a2;
    if (top < ((1023u + 400u) << 20)) {
      a0 = div_nr(kWeno[9], d0);
      a1 = div_nr(kWeno[10], d1);
      a2 = div_nr(kWeno[11], d2);
      return div_nr(a0 * p0 + a1 * p1 + a2 * p2, a0 + a1 + a2);
    }
    a0 = kWeno[9] / d0;
    a1 = kWeno[10] / d1;
    a2 = kWeno[11] / d2;
    return (a0 * p0 + a1 * p1 + a2 * p2) / (a0 + a1 + a2);
  }
#endif
  const T eps = T(WENO_EPS);
  T p0 = T(1.0 / 3.0) * phim2 - T(7.0 / 6.0) * phim1 + T(11.0 / 6.0) * phi;
  T p1 = T(-1.0 / 6.0) * phim1 + T(5.0 / 6.0) * phi + T(1.0 / 3.0) * phip1;
  T p2 = T(1.0 / 3.0) * phi + T(5.0 / 6.0) * phip1 - T(1.0 / 6.0) * phip2;
  T b0 = T(13. / 12.) * sqr(phim2 - T(2.) * phim1 + phi) +
         T(.25) * sqr(phim2 - T(4.) * phim1 + T(3.) * phi);
  T b1 = T(13. / 12.) * sqr(phim1 - T(2.) * phi + phip1) + T(.25) * sqr(phim1 - phip1);
  T b2 = T(13. / 12.) * sqr(phi - T(2.) * phip1 + phip2) +
         T(.25) * sqr(T(3.) * phi - T(4.) * phip1 + phip2);
  T a0 = T(0.1) / ((b0 + eps) * (b0 + eps));
  T a1 = T(0.6) / ((b1 + eps) * (b1 + eps));
  T a2 = T(0.3) / ((b2 + eps) * (b2 + eps));
  return (a0 * p0 + a1 * p1 + a2 * p2) / (a0 + a1 + a2);
}

// The same reconstruction split so that a cell's smoothness indicators serve
// both of its faces: the right-face value of cell c uses the weights
// 1/(beta_k + eps)^2 of its left, centre and right candidate stencils in that
// order, the left-face value the same three in mirror order.  a..e are the
// cells c-2..c+2.  (A sliding window over a line of faces computes each
// cell's indicators once instead of twice; the indicators of the mirrored
// stencils are the same sums taken in the other order, so results agree
// with weno5 to rounding.)
template <class T>
struct WenoCell {
  T i0, i1, i2;  // 1/(beta+eps)^2 of the stencils {c-2..c}, {c-1..c+1}, {c..c+2}
};
template <class T>
__device__ __forceinline__ WenoCell<T> weno_cell(T a, T b, T c, T d, T e) {
  const T eps = T(WENO_EPS);
  T b0 = T(13. / 12.) * sqr(a - T(2.) * b + c) + T(.25) * sqr(a - T(4.) * b + T(3.) * c);
  T b1 = T(13. / 12.) * sqr(b - T(2.) * c + d) + T(.25) * sqr(b - d);
  T b2 = T(13. / 12.) * sqr(c - T(2.) * d + e) + T(.25) * sqr(T(3.) * c - T(4.) * d + e);
  return {T(1.) / ((b0 + eps) * (b0 + eps)), T(1.) / ((b1 + eps) * (b1 + eps)),
          T(1.) / ((b2 + eps) * (b2 + eps))};
}
template <class T>
__device__ __forceinline__ T weno_right(const WenoCell<T>& w, T a, T b, T c, T d, T e) {
  T p0 = T(1.0 / 3.0) * a - T(7.0 / 6.0) * b + T(11.0 / 6.0) * c;
  T p1 = T(-1.0 / 6.0) * b + T(5.0 / 6.0) * c + T(1.0 / 3.0) * d;
  T p2 = T(1.0 / 3.0) * c + T(5.0 / 6.0) * d - T(1.0 / 6.0) * e;
  T a0 = T(0.1) * w.i0, a1 = T(0.6) * w.i1, a2 = T(0.3) * w.i2;
  return (a0 * p0 + a1 * p1 + a2 * p2) / (a0 + a1 + a2);
}
template <class T>
__device__ __forceinline__ T weno_left(const WenoCell<T>& w, T a, T b, T c, T d, T e) {
  T p0 = T(1.0 / 3.0) * e - T(7.0 / 6.0) * d + T(11.0 / 6.0) * c;
  T p1 = T(-1.0 / 6.0) * d + T(5.0 / 6.0) * c + T(1.0 / 3.0) * b;
  T p2 = T(1.0 / 3.0) * c + T(5.0 / 6.0) * b - T(1.0 / 6.0) * a;
  T a0 = T(0.1) * w.i2, a1 = T(0.6) * w.i1, a2 = T(0.3) * w.i0;
  return (a0 * p0 + a1 * p1 + a2 * p2) / (a0 + a1 + a2);
}

// right-face value (face c+1) and left-face value (face c) of cell c on a
// strided line q[c*s]
// (the stencil values are converted to the reconstruction type T first)
template <class T, class S>
__device__ __forceinline__ T weno_r(const S* q, long s, int c) {
  return weno5<T>(T(q[(c + 2) * s]), T(q[(c + 1) * s]), T(q[c * s]), T(q[(c - 1) * s]),
                  T(q[(c - 2) * s]));
}
template <class T, class S>
__device__ __forceinline__ T weno_l(const S* q, long s, int c) {
  return weno5<T>(T(q[(c - 2) * s]), T(q[(c - 1) * s]), T(q[c * s]), T(q[(c + 1) * s]),
                  T(q[(c + 2) * s]));
}

// ------------------------------------------------------------------ EOS ----
// CubedSphereUtility::CovariantToContravariant (cubed_sphere_utility.hpp:22-31)
// (the mixed build multiplies by one reciprocal instead of four divisions)
__device__ __forceinline__ void cov_to_contra(double* a, double cth) {
  double v = a[IVY], w = a[IVZ];
  double sth2 = 1. - cth * cth;
#if EXO_MIXED
  const double is2 = inv_r(sth2);
  a[IVY] = (v - w * cth) * is2;
  a[IVZ] = (w - v * cth) * is2;
#else
  const SharedDiv by_s2(sth2);
  a[IVY] = by_s2(v) - by_s2(w * cth);
  a[IVZ] = by_s2(-v * cth) + by_s2(w);
#endif
}
__device__ __forceinline__ void contra_to_cov(double* a, double cth) {
  double v = a[IVY], w = a[IVZ];
  a[IVY] = v + w * cth;
  a[IVZ] = w + v * cth;
}

// ConservedToPrimitive of one cell (shallow_yz_hydro.cpp:42-67,
// ideal_moist_hydro.cpp:77-159); returns 1 if the state is invalid
__device__ __forceinline__ int cons_to_prim(const DevView& v, const double* c, double* w,
                                            double cth) {
  int bad = 0;
  if (v.eqn == EXO_EQN_SHALLOW_YZ) {
    double dfloor = (double)sqrtf(1024 * FLT_MIN);
    double ud = c[IDN];
    ud = (ud > dfloor) ? ud : dfloor;
    w[IDN] = ud;
    w[IVX] = 0.;
    w[IVY] = c[IVY];
    w[IVZ] = c[IVZ];
    double di = 1. / ud;
    cov_to_contra(w, cth);
    w[IVY] *= di;
    w[IVZ] *= di;
  } else {
    double gm1 = v.gamma - 1.0;
    double density = 0.;
    density += c[IDN];
    w[IDN] = density;
    double di = inv_r(density);
    if ((w[IDN] < 0.) || isnan(w[IDN])) bad = 1;
    double fsig = 1., feps = 1.;
    w[IVX] = c[IVX] * di;
    w[IVY] = c[IVY] * di;
    w[IVZ] = c[IVZ] * di;
    cov_to_contra(w, cth);
    double KE = 0.5 * (c[IVX] * w[IVX] + c[IVY] * w[IVY] + c[IVZ] * w[IVZ]);
    w[IPR] = gm1 * (c[IEN] - KE) * feps / fsig;
    if ((w[IPR] < 0.) || isnan(w[IPR])) bad = 1;
  }
  return bad;
}

__device__ __forceinline__ void prim_to_cons(const DevView& v, const double* w, double* c,
                                             double cth) {
  if (v.eqn == EXO_EQN_SHALLOW_YZ) {
    double wd = w[IDN];
    c[IDN] = wd;
    c[IVX] = 0.;
    c[IVY] = w[IVY];
    c[IVZ] = w[IVZ];
    contra_to_cov(c, cth);
    c[IVY] *= wd;
    c[IVZ] *= wd;
  } else {
    double igm1 = 1.0 / (v.gamma - 1.0);
    double wd = w[IDN];
    c[IDN] = wd;
    c[IVX] = w[IVX] * wd;
    c[IVY] = w[IVY] * wd;
    c[IVZ] = w[IVZ] * wd;
    contra_to_cov(c, cth);
    double KE = 0.5 * (c[IVX] * w[IVX] + c[IVY] * w[IVY] + c[IVZ] * w[IVZ]);
    double fsig = 1., feps = 1.;
    c[IEN] = igm1 * w[IPR] * fsig / feps + KE;
  }
}

// ------------------------------------------------------ Riemann solvers ----
template <class T>
struct FaceGeo {
  T cosf, sinf, cthp, cthc;
};

template <class T>
__device__ __forceinline__ void prim_to_local(int ivx, const FaceGeo<T>& fg, T* w) {
  if (ivx == IVY) {  // PrimToLocal2, gnomonic_equiangle.cpp:604-660
    T g23 = fg.cosf, g33 = T(1.0), gi22 = T(1.0) / (fg.sinf * fg.sinf);
    T T11 = T(1.0), T22 = T(1.0) / sqrt(gi22), T32 = g23 / sqrt(g33), T33 = sqrt(g33);
    T uu1 = w[IVX], uu2 = w[IVY], uu3 = w[IVZ];
    w[IVX] = T11 * uu1;
    w[IVY] = T22 * uu2;
    w[IVZ] = T32 * uu2 + T33 * uu3;
  } else if (ivx == IVZ) {  // PrimToLocal3, :662-718
    T g23 = fg.cosf, g22 = T(1.0), gi33 = T(1.0) / (fg.sinf * fg.sinf);
    T T11 = T(1.0), T22 = sqrt(g22), T23 = g23 / sqrt(g22), T33 = T(1.0) / sqrt(gi33);
    T uu1 = w[IVX], uu2 = w[IVY], uu3 = w[IVZ];
    w[IVX] = T11 * uu1;
    w[IVY] = T22 * uu2 + T23 * uu3;
    w[IVZ] = T33 * uu3;
  }
}

template <class T>
__device__ __forceinline__ void flux_to_global(int ivx, const FaceGeo<T>& fg, T* f) {
  if (ivx == IVY) {  // FluxToGlobal2, :752-791
    T g23 = fg.cosf, g33 = T(1.0), gi22 = T(1.0) / (fg.sinf * fg.sinf);
    T T11 = T(1.0), T22 = sqrt(gi22), T32 = -sqrt(gi22) * g23 / g33, T33 = T(1.0) / sqrt(g33);
    T txx = f[IVX], txy = f[IVY], txz = f[IVZ];
    f[IVX] = T11 * txx;
    f[IVY] = T22 * txy;
    f[IVZ] = T32 * txy + T33 * txz;
  } else if (ivx == IVZ) {  // FluxToGlobal3, :793-832
    T g23 = fg.cosf, g22 = T(1.0), gi33 = T(1.0) / (fg.sinf * fg.sinf);
    T T11 = T(1.0), T22 = T(1.0) / sqrt(g22), T23 = -g23 / g22 * sqrt(gi33), T33 = sqrt(gi33);
    T txx = f[IVX], txy = f[IVY], txz = f[IVZ];
    f[IVX] = T11 * txx;
    f[IVY] = T22 * txy + T23 * txz;
    f[IVZ] = T33 * txz;
  }
}

// roe_shallow_yz.cpp:18-122
template <class T>
__device__ __forceinline__ void riemann_roe_shallow(int ivx, const FaceGeo<T>& fg, T* wli, T* wri, T* flx) {
  const T h = T(0.5);
  int ivy = ivx == IVY ? IVZ : IVY;
  prim_to_local(ivx, fg, wli);
  prim_to_local(ivx, fg, wri);
  T ubar = (wli[ivx] * sqrt(wli[IDN]) + wri[ivx] * sqrt(wri[IDN])) /
           (sqrt(wli[IDN]) + sqrt(wri[IDN]));
  T vbar = (wli[ivy] * sqrt(wli[IDN]) + wri[ivy] * sqrt(wri[IDN])) /
           (sqrt(wli[IDN]) + sqrt(wri[IDN]));
  T cbar = sqrt(h * (wli[IDN] + wri[IDN]));
  T delh = wri[IDN] - wli[IDN];
  T delu = wri[ivx] - wli[ivx];
  T delv = wri[ivy] - wli[ivy];
  T hbar = sqrt(wli[IDN] * wri[IDN]);
  T a1 = h * (cbar * delh - hbar * delu) / cbar;
  T a2 = hbar * delv;
  T a3 = h * (cbar * delh + hbar * delu) / cbar;
  T w00 = a1, w01 = a1 * (ubar - cbar), w02 = a1 * vbar;
  T w10 = T(0.), w11 = T(0.), w12 = a2;
  T w20 = a3, w21 = a3 * (ubar + cbar), w22 = a3 * vbar;
  T s0 = fabs(ubar - cbar), s1 = fabs(ubar), s2 = fabs(ubar + cbar);
  flx[IVZ] = T(0.);
  flx[IDN] = h * (wli[IDN] * wli[ivx] + wri[IDN] * wri[ivx]);
  flx[ivx] = h * (wli[IDN] * wli[ivx] * wli[ivx] + h * wli[IDN] * wli[IDN] +
                  wri[IDN] * wri[ivx] * wri[ivx] + h * wri[IDN] * wri[IDN]);
  flx[ivy] = h * (wli[IDN] * wli[ivx] * wli[ivy] + wri[IDN] * wri[ivx] * wri[ivy]);
  flx[IVX] = T(0.);
  flx[IDN] -= h * s0 * w00;
  flx[ivx] -= h * s0 * w01;
  flx[ivy] -= h * s0 * w02;
  flx[IDN] -= h * s1 * w10;
  flx[ivx] -= h * s1 * w11;
  flx[ivy] -= h * s1 * w12;
  flx[IDN] -= h * s2 * w20;
  flx[ivx] -= h * s2 * w21;
  flx[ivy] -= h * s2 * w22;
  if (ivx == IVX) {
    flx[IVX] = T(0.);
    return;
  }
  flux_to_global(ivx, fg, flx);
  T ty = flx[ivx], tz = flx[ivy];
  flx[ivx] = ty + tz * fg.cthp;
  flx[ivy] = tz + ty * fg.cthp;
}

// The solvers' functions of gamma: in FP64 those of the view, which the host
// computed (two divisions a face fewer); in FP32 computed where they are used.
template <class T>
__device__ __forceinline__ RiemannGas<T> riemann_gas(const RiemannGas<double>& gas) {
  if constexpr (sizeof(T) == sizeof(double)) return gas;
  else return make_riemann_gas<T>(T(gas.gamma));
}

// lmars.cpp:24-110 (NVAPOR = NCLOUD = 0), no projection
template <class T>
__device__ __forceinline__ void riemann_lmars(const RiemannGas<T>& gas, int ivx, const T* wli, const T* wri, T* flx) {
  const T h = T(0.5), one = T(1.);
  int ivy = IVX + ((ivx - IVX) + 1) % 3;
  int ivz = IVX + ((ivx - IVX) + 2) % 3;
  T hl = wli[IPR] / wli[IDN] * gas.kappa1 +
         h * (sqr(wli[ivx]) + sqr(wli[ivy]) + sqr(wli[ivz]));
  T hr = wri[IPR] / wri[IDN] * gas.kappa1 +
         h * (sqr(wri[ivx]) + sqr(wri[ivy]) + sqr(wri[ivz]));
  T rhobar = h * (wli[IDN] + wri[IDN]);
  T cbar = sqrt(h * gas.cfac * (wli[IPR] + wri[IPR]) / rhobar);
  T pbar = h * (wli[IPR] + wri[IPR]) + h * (rhobar * cbar) * (wli[ivx] - wri[ivx]);
  T ubar = h * (wli[ivx] + wri[ivx]) + h / (rhobar * cbar) * (wli[IPR] - wri[IPR]);
  T rdl = one, rdr = one;
  if (ubar > T(0.)) {
    flx[IDN] = ubar * wli[IDN] * rdl;
    flx[ivx] = ubar * wli[IDN] * wli[ivx] + pbar;
    flx[ivy] = ubar * wli[IDN] * wli[ivy];
    flx[ivz] = ubar * wli[IDN] * wli[ivz];
    flx[IEN] = ubar * wli[IDN] * hl;
  } else {
    flx[IDN] = ubar * wri[IDN] * rdr;
    flx[ivx] = ubar * wri[IDN] * wri[ivx] + pbar;
    flx[ivy] = ubar * wri[IDN] * wri[ivy];
    flx[ivz] = ubar * wri[IDN] * wri[ivz];
    flx[IEN] = ubar * wri[IDN] * hr;
  }
}

// hllc_transform.cpp:24-263
template <class T>
__device__ __forceinline__ void riemann_hllc(const RiemannGas<T>& gas, int ivx, const FaceGeo<T>& fg, T* wl, T* wr, T* flx) {
  const T h = T(.5), one = T(1.0), zero = T(0.0);
  int ivy = IVX + ((ivx - IVX) + 1) % 3;
  int ivz = IVX + ((ivx - IVX) + 2) % 3;
  prim_to_local(ivx, fg, wl);
  prim_to_local(ivx, fg, wr);
  T wli[5], wri[5], fl[5], fr[5];
  wli[IDN] = wl[IDN]; wli[IVX] = wl[ivx]; wli[IVY] = wl[ivy]; wli[IVZ] = wl[ivz]; wli[IPR] = wl[IPR];
  wri[IDN] = wr[IDN]; wri[IVX] = wr[ivx]; wri[IVY] = wr[ivy]; wri[IVZ] = wr[ivz]; wri[IPR] = wr[IPR];
  T cl = sqrt(gas.gam * wli[IPR] / wli[IDN]);
  T cr = sqrt(gas.gam * wri[IPR] / wri[IDN]);
  T KE_l, KE_r;
  if (ivx == IVX) {
    T cth = fg.cthc, vy, vz;
    vy = wli[IVY] + wli[IVZ] * cth;
    vz = wli[IVZ] + wli[IVY] * cth;
    KE_l = h * wli[IDN] * (sqr(wli[IVX]) + wli[IVY] * vy + wli[IVZ] * vz);
    vy = wri[IVY] + wri[IVZ] * cth;
    vz = wri[IVZ] + wri[IVY] * cth;
    KE_r = h * wri[IDN] * (sqr(wri[IVX]) + wri[IVY] * vy + wri[IVZ] * vz);
  } else {
    KE_l = h * wli[IDN] * (sqr(wli[IVX]) + sqr(wli[IVY]) + sqr(wli[IVZ]));
    KE_r = h * wri[IDN] * (sqr(wri[IVX]) + sqr(wri[IVY]) + sqr(wri[IVZ]));
  }
  T el = wli[IPR] * gas.igm1 + KE_l;
  T er = wri[IPR] * gas.igm1 + KE_r;
  T rhoa = h * (wli[IDN] + wri[IDN]);
  T ca = h * (cl + cr);
  T pmid = h * (wli[IPR] + wri[IPR] + (wli[IVX] - wri[IVX]) * rhoa * ca);
  T ql = (pmid <= wli[IPR]) ? one
         : sqrt(one + gas.qfac * (pmid / wli[IPR] - one));
  T qr = (pmid <= wri[IPR]) ? one
         : sqrt(one + gas.qfac * (pmid / wri[IPR] - one));
  T al = wli[IVX] - cl * ql;
  T ar = wri[IVX] + cr * qr;
  T bp = ar > zero ? ar : T(TINY_NUMBER);
  T bm = al < zero ? al : -T(TINY_NUMBER);
  T vxl = wli[IVX] - al;
  T vxr = wri[IVX] - ar;
  T tl = wli[IPR] + vxl * wli[IDN] * wli[IVX];
  T tr = wri[IPR] + vxr * wri[IDN] * wri[IVX];
  T ml = wli[IDN] * vxl;
  T mr = -(wri[IDN] * vxr);
  T am = (tl - tr) / (ml + mr);
  T cp = (ml * tr + mr * tl) / (ml + mr);
  cp = cp > zero ? cp : zero;
  vxl = wli[IVX] - bm;
  vxr = wri[IVX] - bp;
  fl[IDN] = wli[IDN] * vxl;
  fr[IDN] = wri[IDN] * vxr;
  fl[IVX] = wli[IDN] * wli[IVX] * vxl + wli[IPR];
  fr[IVX] = wri[IDN] * wri[IVX] * vxr + wri[IPR];
  fl[IVY] = wli[IDN] * wli[IVY] * vxl;
  fr[IVY] = wri[IDN] * wri[IVY] * vxr;
  fl[IVZ] = wli[IDN] * wli[IVZ] * vxl;
  fr[IVZ] = wri[IDN] * wri[IVZ] * vxr;
  fl[IEN] = el * vxl + wli[IPR] * wli[IVX];
  fr[IEN] = er * vxr + wri[IPR] * wri[IVX];
  T sl, sr, sm;
  if (am >= zero) {
    sl = am / (am - bm);
    sr = zero;
    sm = -bm / (am - bm);
  } else {
    sl = zero;
    sr = -am / (bp - am);
    sm = bp / (bp - am);
  }
  flx[IDN] = sl * fl[IDN] + sr * fr[IDN];
  flx[ivx] = sl * fl[IVX] + sr * fr[IVX] + sm * cp;
  flx[ivy] = sl * fl[IVY] + sr * fr[IVY];
  flx[ivz] = sl * fl[IVZ] + sr * fr[IVZ];
  flx[IEN] = sl * fl[IEN] + sr * fr[IEN] + sm * cp * am;
  flux_to_global(ivx, fg, flx);
  T ty = flx[IVY], tz = flx[IVZ];
  flx[IVY] = ty + tz * fg.cthp;
  flx[IVZ] = tz + ty * fg.cthp;
}

// lmars_shallow_yz.cpp:18-93
template <class T>
__device__ __forceinline__ void riemann_lmars_shallow(int ivx, const FaceGeo<T>& fg, T* wli, T* wri, T* flx) {
  const T h = T(0.5);
  int ivy = ivx == IVY ? IVZ : IVY;
  prim_to_local(ivx, fg, wli);
  prim_to_local(ivx, fg, wri);
  T cbar = sqrt(h * (wli[IDN] + wri[IDN]));
  T hbar = h * (wli[IDN] + wri[IDN]) + h * cbar * (wli[ivx] - wri[ivx]);
  T ubar = h * (wli[ivx] + wri[ivx]) + h / cbar * (wli[IDN] - wri[IDN]);
  flx[IVZ] = T(0.);
  if (ubar > T(0.)) {
    flx[IDN] = ubar * wli[IDN];
    flx[ivx] = ubar * wli[IDN] * wli[ivx] + h * hbar * hbar;
    flx[ivy] = ubar * wli[IDN] * wli[ivy];
  } else {
    flx[IDN] = ubar * wri[IDN];
    flx[ivx] = ubar * wri[IDN] * wri[ivx] + h * hbar * hbar;
    flx[ivy] = ubar * wri[IDN] * wri[ivy];
  }
  flx[IVX] = T(0.);
  if (ivx == IVX) return;
  flux_to_global(ivx, fg, flx);
  T ty = flx[ivx], tz = flx[ivy];
  flx[ivx] = ty + tz * fg.cthp;
  flx[ivy] = tz + ty * fg.cthp;
}

template <class T>
__device__ __forceinline__ void riemann(int rsolver, const RiemannGas<double>& gas, int ivx, const FaceGeo<T>& fg,
                                        T* wl, T* wr, T* flx) {
  switch (rsolver) {
    case EXO_RS_ROE_SHALLOW: riemann_roe_shallow(ivx, fg, wl, wr, flx); break;
    case EXO_RS_LMARS: riemann_lmars(riemann_gas<T>(gas), ivx, wl, wr, flx); break;
    case EXO_RS_HLLC: riemann_hllc(riemann_gas<T>(gas), ivx, fg, wl, wr, flx); break;
    default: riemann_lmars_shallow(ivx, fg, wl, wr, flx); break;
  }
}

// ----------------------------------------------------- k_prim_ghost ------
// The conserved state a ghost-band cell gets from the neighbour panel
// (CubedSphereUtility::PackData with InteprolateX2/X3, cubed_sphere_utility.
// cpp:92-369, as the ghost table e precomputes it): linear interpolation
// along the edge between two source cells, vectors (IVY, IVZ) raised,
// rotated to the receiver's basis through latitude-longitude and lowered.
// src is the source panel's (nv, nc3, nc2, nc1) array.
__device__ __forceinline__ void ghost_interp(const DevView& v, const GhostEntry& e,
                                             const double* src, int i, double* c) {
  const size_t vs = v.cells;
#if EXO_MIXED
  auto by_C = [&](double a) { return a / e.C; };
  auto by_s = [&](double a) { return a / e.ss; };
#else
  // the same quotients from one reciprocal each (and cov_to_contra's: FP64
  // 96^2x64 109 -> 102 us; the mixed build's results would change in the last bit)
  const SharedDiv by_C(e.C), by_s(e.ss);
#endif
  const double* s0 = src + (size_t)(unsigned)(e.k0 * v.nc2 + e.j0) * (unsigned)v.nc1 + i;
  const double* s1 = src + (size_t)(unsigned)(e.k1 * v.nc2 + e.j1) * (unsigned)v.nc1 + i;
  #pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= v.nv) break;
    if (n == IVY || n == IVZ) continue;
    double v1 = s0[n * vs];
    double v2 = s1[n * vs];
    c[n] = by_C(e.A * v1 + e.B * v2);
  }
  double v1y = s0[IVY * vs], v1z = s0[IVZ * vs];
  double v2y = s1[IVY * vs], v2z = s1[IVZ * vs];
  double vy = by_C(e.A * v1y + e.B * v2y);
  double vz = by_C(e.A * v1z + e.B * v2z);
  double cth = e.cs;
  double vyt = vy, vzt = vz;
  vy = by_s(by_s(vyt)) - by_s(by_s(vzt * cth));
  vz = by_s(by_s(vzt)) - by_s(by_s(vyt * cth));
  double U = e.r[0] * vy + e.r[1] * vz;
  double V = e.r[2] * vy + e.r[3] * vz;
  vy = e.q[0] * U + e.q[1] * V;
  vz = e.q[2] * U + e.q[3] * V;
  vyt = vy;
  vzt = vz;
  c[IVY] = vyt + vzt * e.ct;
  c[IVZ] = vzt + vyt * e.ct;
}

// Conserved value of variable n at cell (p,k,j,i) where (k,j) is interior or
// in a ghost band; vectors (IVY, IVZ) come back together.
__device__ __forceinline__ void load_cons(const DevView& v, int p, int k, int j, int i,
                                          bool interior, double* c) {
  if (interior) {
    const double* u = v.u + idx(v, p, 0, k, j, i);
    const size_t vs = v.cells;
    #pragma unroll
    for (int n = 0; n < 5; ++n) {
      if (n >= v.nv) break;
      c[n] = u[n * vs];
    }
    return;
  }
  const GhostEntry& e = v.ghost[v.ghost_map[((size_t)p * v.nc3 + k) * v.nc2 + j]];
  ghost_interp(v, e, v.u + idx(v, e.src_panel, 0, 0, 0, 0), i, c);
}

// the CFL candidate of the block's cells is reduced in shared memory first,
// so one atomic per block reaches the global minimum
__device__ __forceinline__ void block_min_atomic(unsigned long long* target, unsigned long long x) {
  __shared__ unsigned long long warp_min[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long y = __shfl_down_sync(0xffffffffu, x, o);
    x = y < x ? y : x;
  }
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) warp_min[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int nw = (blockDim.x + 31) >> 5;
    x = lane < nw ? warp_min[lane] : ~0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long y = __shfl_down_sync(0xffffffffu, x, o);
      x = y < x ? y : x;
    }
    if (lane == 0 && x != ~0ull) atomicMin(target, x);
  }
}

// Hydro::NewBlockTimeStep with patches/21.new_blockdt.patch:23-35 at an
// interior cell with primitives w: the candidate as the bits of a
// non-negative double, or ~0 when there is none
__device__ __forceinline__ unsigned long long cfl_candidate(const DevView& v, const double* w,
                                                            int p, int k, int j, int i) {
  const bool shallow = (v.eqn == EXO_EQN_SHALLOW_YZ);
  double cs;
  if (shallow) cs = sqrt(w[IDN]);
  else {
    double fsig = 1., feps = 1.;
    cs = sqrt((1. + (v.gamma - 1) * feps / fsig) * w[IPR] / w[IDN]);
  }
  double dt1 = v.dx1f[i], dt2 = v.x1v[i] * geo(v, GDX2A, p, k, j);
  double dt3 = v.x1v[i] * geo(v, GDX3A, p, k, j);
  double speed1 = fmax(0., (fabs(w[IVX]) + cs));
  double speed2 = fmax(0., (fabs(w[IVY]) + cs));
  double speed3 = fmax(0., (fabs(w[IVZ]) + cs));
  if ((v.implicit_flag & 1) && (v.N > 1)) dt1 /= v.cfl * fabs(w[IVX]);
  else dt1 /= speed1;
  if (v.implicit_flag & 2) dt2 /= v.cfl * fabs(w[IVY]);
  else dt2 /= speed2;
  if (v.implicit_flag & 4) dt3 /= v.cfl * fabs(w[IVZ]);
  else dt3 /= speed3;
  double m = fmin(dt2, dt3);
  if (!shallow) m = fmin(dt1, m);
  if (m >= 0.) return (unsigned long long)__double_as_longlong(m);
  return ~0ull;
}

__device__ __forceinline__ unsigned long long prim_ghost_cell(const DevView& v, unsigned tid,
                                                              int compute_dt) {
  const unsigned long long none = ~0ull;
  unsigned total = 6u * (unsigned)v.cells;
  if (tid >= total) return none;
  unsigned r = v.div_nc1(tid);
  unsigned i = tid - r * (unsigned)v.nc1;
  unsigned r2 = v.div_nc2(r);
  int j = (int)(r - r2 * (unsigned)v.nc2);
  unsigned r3 = v.div_nc3(r2);
  int k = (int)(r2 - r3 * (unsigned)v.nc3);
  int p = (int)r3;
  bool kin = (k >= v.ks && k <= v.ke), jin = (j >= v.js && j <= v.je);
  if (!kin && !jin) return none;  // corner: never read on the path
  int ii = i;
  bool mirror = false;
  if (i < v.is) { ii = 2 * v.is - 1 - i; mirror = true; }
  else if (i > v.ie) { ii = 2 * v.ie + 1 - i; mirror = true; }
  double c[5], w[5];
  load_cons(v, p, k, j, ii, kin && jin, c);
  double cth = geo(v, GCOSC, p, k, j);
  int bad = cons_to_prim(v, c, w, cth);
  if (mirror) w[IVX] = -w[IVX];
  const size_t at = idx(v, p, 0, k, j, i), vs = v.cells;
  double* const wo = v.w + at;
  #pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= v.nv) break;
    wo[n * vs] = w[n];
  }
#if EXO_MIXED
  float* const fo = v.w32 + at;
  #pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= v.nv) break;
    fo[n * vs] = (float)w[n];
  }
#endif
  if (!(kin && jin) || mirror) return none;
  if (bad) atomicOr(&v.sc->invalid, 1);
  if (compute_dt) return cfl_candidate(v, w, p, k, j, (int)i);
  return none;
}


__device__ __forceinline__ void prim_ghost_block(const DevView& v, unsigned blk, int compute_dt) {
  unsigned tid = blk * blockDim.x + threadIdx.x;
  unsigned long long m = prim_ghost_cell(v, tid, compute_dt);
  if (compute_dt) block_min_atomic(&v.sc->dtmin_bits, m);
}

// ------------------------------------------------------------ k_flux_x1 ---
// Several radial columns per block (the x1 tile): each column's faces,
// cells and hydrostatic scan are spread over the block's threads, so the
// block's lanes stay busy (one column of L+1 faces leaves most of a warp
// idle) and the columns' scans run side by side.
// What bounds it: instruction issue (mixed build, 96^2x64: 1,692 instructions
// per 32 cells at 0.65 a cycle and scheduler; DRAM 13 %), a third of them FP32
// WENO5, then the FP64 decomposition and the Riemann solve.  It was 2,076 with
// a division for its place per pass and element, a thread's cells converted to
// FP32 five times, the reciprocal of gamma and the solver's functions of it
// per cell, and the series' coefficients as literals.  Per launch (4 columns a
// block), before and now: FP64 40^2x40 84 -> 70 us, 96^2x64 536 -> 422; mixed
// 24^2x32 19 -> 17, 62^2x45 121 -> 109, 96^2x64 312 -> 258, 126^2x70 667 ->
// 542, 192^2x96 1712 -> 1448.
__device__ __forceinline__ int x1_columns_per_block(const DevView& v) {
  return v.tiles[BK_X1] > 0 ? v.tiles[BK_X1] : 1;
}

// q = t / d, r = t - q d for small non-negative t (< 2^20) through a float
// reciprocal, corrected by one step either way
__device__ __forceinline__ void divmod_small(int t, int d, float inv_d, int& q, int& r) {
  q = (int)((float)t * inv_d);
  r = t - q * d;
  if (r < 0) { --q; r += d; }
  else if (r >= d) { ++q; r -= d; }
}

#if EXO_MIXED
// ln(sinh x / x) for |x| <= 0.25: its Taylor series sum_n c_n x^{2n} with
// c_n = 2^{2n} B_{2n} / (2n (2n)!) (B the Bernoulli numbers), seven terms
// (truncation error below 4e-19 there).  The two series' coefficients are read
// from the constant bank: as literals each takes two moves to registers.
__constant__ double kSinhc[7] = {1. / 6,        -1. / 180,           1. / 2835,
                                 -1. / 37800,   1. / 467775,         -691. / 3831077250.,
                                 2. / 127702575.};
__device__ __forceinline__ double ln_sinhc(double x) {
  const double z = x * x;
  double s = kSinhc[6];
#pragma unroll
  for (int k = 5; k >= 0; --k) s = kSinhc[k] + z * s;
  return z * s;
}
// e^y for |y| <= 0.25: its Taylor series to y^13 (truncation below 5e-20)
__constant__ double kInvFact[14] = {1.,
                                    1.,
                                    1. / 2,
                                    1. / 6,
                                    1. / 24,
                                    1. / 120,
                                    1. / 720,
                                    1. / 5040,
                                    1. / 40320,
                                    1. / 362880,
                                    1. / 3628800,
                                    1. / 39916800,
                                    1. / 479001600,
                                    1. / 6227020800.};
__device__ __forceinline__ double exp_small(double y) {
  double s = kInvFact[13];
#pragma unroll
  for (int k = 12; k >= 0; --k) s = s * y + kInvFact[k];
  return s;
}
#endif

template <class T>
__device__ __forceinline__ void flux_x1_block(const DevView& v, unsigned blk) {
  constexpr int NV = 5;  // the ideal gas only
  extern __shared__ double sm[];
  __shared__ double s_igam[X1_MAX_COLUMNS], s_expf[X1_MAX_COLUMNS];
  __shared__ double s_cthp[X1_MAX_COLUMNS], s_cosc[X1_MAX_COLUMNS];
  __shared__ size_t s_base[X1_MAX_COLUMNS];  // the column's first face in the flux array
  const int cpb = x1_columns_per_block(v);
  const int ncol_total = 6 * v.N * v.N;
  const int col0 = (int)blk * cpb;
  const int ncb = min(cpb, ncol_total - col0);  // columns of this block
  const int nc1 = v.nc1, L = v.L, is = v.is, ie = v.ie;
  const int cstride = x1_column_doubles(v);  // shared doubles per column
  const size_t vs = v.cells;
  const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nwarps = (int)blockDim.x >> 5;
  // Every pass runs over (column c, index i) with i up to the nc1 + 1 faces,
  // the widest of them, so that a thread's place is computed once (a block
  // has a thread for each place unless that is more than 1024).
  const int per = nc1 + 1;
  const float inv_per = 1.f / (float)per;
  int c0, i0;
  divmod_small(tid, per, inv_per, c0, i0);
  auto each = [&](auto&& body) {
    int c = c0, i = i0;
#pragma unroll 1
    for (int t = tid; t < ncb * per;) {
      body(c, i);
      t += (int)blockDim.x;
      if (t < ncb * per) divmod_small(t, per, inv_per, c, i);
    }
  };
  // the column's first place in the state array
  auto base = [&](int c) {
    const unsigned col = (unsigned)(col0 + c);
    const unsigned r = v.div_N(col), p = v.div_N(r);
    return idx(v, (int)p, 0, v.ks + (int)(r - p * (unsigned)v.N),
               v.js + (int)(col - r * (unsigned)v.N), 0);
  };
  // Shared memory of column c.  FP64: w [5][nc1] and psf [nc1 + 1].  Mixed:
  // density and pressure [2][nc1], psf, ln psf and the isentropic density at
  // the faces [3][nc1 + 1], then in FP32 what is reconstructed [5][nc1] and
  // both face values of the cells is - 1 .. ie + 1 [2][5][L + 2].
  auto COL = [&](int c) { return sm + (unsigned)(c * cstride); };
#if EXO_MIXED
  const int ncell = L + 2;
  auto WD = [&](int c) { return COL(c); };
  auto WP = [&](int c) { return COL(c) + nc1; };
  auto PSF = [&](int c) { return COL(c) + 2 * nc1; };
  auto WF = [&](int c) { return reinterpret_cast<T*>(COL(c) + 2 * nc1 + 3 * per); };
  auto REC = [&](int c) { return WF(c) + NV * nc1; };
#else
  auto WD = [&](int c) { return COL(c) + IDN * nc1; };
  auto WP = [&](int c) { return COL(c) + IPR * nc1; };
  auto PSF = [&](int c) { return COL(c) + NV * nc1; };
#endif
  if (tid < ncb) {
    const unsigned col = (unsigned)(col0 + tid);
    const unsigned r = v.div_N(col), p = v.div_N(r);
    const int k = v.ks + (int)(r - p * (unsigned)v.N), j = v.js + (int)(col - r * (unsigned)v.N);
    s_base[tid] = idx(v, (int)p, 0, k, j, is);
    s_cthp[tid] = geo(v, GCTHP1, (int)p, k, j);
    s_cosc[tid] = geo(v, GCOSC, (int)p, k, j);
  }
  const bool decomp = (v.grav != 0.);
  each([&](int c, int i) {
    if (i >= nc1) return;
    const double* src = v.w + base(c) + i;
#if EXO_MIXED
    T* f = WF(c) + i;
    const double d = src[0], p = src[IPR * vs];
    WD(c)[i] = d;
    WP(c)[i] = p;
#pragma unroll
    for (int n = IVX; n <= IVZ; ++n) f[n * nc1] = T(src[n * vs]);
    if (!decomp) {
      f[IDN * nc1] = T(d);
      f[IPR * nc1] = T(p);
    }
#else
    double* dst = COL(c) + i;
#pragma unroll
    for (int n = 0; n < NV; ++n) dst[n * nc1] = src[n * vs];
    // the weight of the layer, which the downward scan below adds up
    if (decomp && i >= is && i <= ie) PSF(c)[i] = -v.grav * src[0] * v.dx1f[i];
#endif
  });
  __syncthreads();
  if (decomp) {
    // Decomposition::ChangeToPerturbation (change_to_perturbation.cpp:39-157).
#if EXO_MIXED
    // The downward scan psf[i] = psf[i+1] + g rho_i dx1f_i as a suffix sum,
    // one warp per column: each lane sums a chunk of levels, the lanes'
    // sums are scanned with shuffles, then each lane fills its chunk (FP64
    // throughout; only the order of the additions differs from the serial
    // scan of the FP64 build).  The column's two logarithms share one call
    // (lanes 0 and 1), and its two exponentials another.
    {
      const int chunk = (L + 31) >> 5;
      const double grav = -v.grav;
      for (int c = warp; c < ncb; c += nwarps) {
        double* psf = PSF(c);
        const double* wd = WD(c);
        const double* wp = WP(c);
        const int m0 = is + lane * chunk, m1 = min(m0 + chunk, ie + 1);
        double part = 0.;
        for (int m = m0; m < m1; ++m) part += grav * wd[m] * v.dx1f[m];
        // sum of the parts of the lanes above this one
        double above = part;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const double y = __shfl_down_sync(0xffffffffu, above, off);
          if (lane + off < 32) above += y;
        }
        above = __shfl_down_sync(0xffffffffu, above, 1);
        if (lane == 31) above = 0.;
        double gammad = v.gamma, fsig = 1., feps = 1.;
        double gam = 1. + (gammad - 1.) * feps / fsig;
        double lg = 0., ex = 0.;
        if (lane < 2) lg = log(lane == 0 ? wp[is] : wd[is]);
        const double lgd = __shfl_sync(0xffffffffu, lg, 1);
        lg = __shfl_sync(0xffffffffu, lg, 0);
        double ent = lg - gam * lgd;
        const double RdTv = wp[ie] / wd[ie];
        if (lane < 2) ex = exp(lane == 0 ? -grav * v.dx1f[ie] / (2 * RdTv) : -ent / gam);
        double top = 0.;
        if (lane == 0) {
          top = wp[ie] * ex;
          psf[ie + 1] = top;
        }
        if (lane == 1) {
          s_igam[c] = 1. / gam;
          s_expf[c] = ex;
        }
        top = __shfl_sync(0xffffffffu, top, 0);
        double run = top + above;
        for (int m = m1 - 1; m >= m0; --m) {
          run += grav * wd[m] * v.dx1f[m];
          psf[m] = run;
        }
        __syncwarp();
        if (lane < G) psf[is - 1 - lane] = psf[is + 1 + lane];
        __syncwarp();
        if (lane < G) psf[ie + 2 + lane] = psf[ie - lane];
      }
    }
#else
    // one thread per column for the downward scan over the layers' weights,
    // another warp's for the isentrope of the lowest cell
    if (warp == 0 && lane < ncb) {
      double* psf = PSF(lane);
      const double* wd = WD(lane);
      const double* wp = WP(lane);
      double grav = -v.grav;
      double RdTv = wp[ie] / wd[ie];
      double run = wp[ie] * exp(-grav * v.dx1f[ie] / (2 * RdTv));
      psf[ie + 1] = run;
#pragma unroll 8
      for (int i = ie; i >= is; --i) {
        run = run + psf[i];
        psf[i] = run;
      }
      for (int i = 1; i <= G; ++i) psf[is - i] = psf[is + i];
      for (int i = 1; i <= G; ++i) psf[ie + i + 1] = psf[ie + 1 - i];
    }
    if (warp == (nwarps > 1 ? 1 : 0) && lane < ncb) {
      double gammad = v.gamma, fsig = 1., feps = 1.;
      double gam = 1. + (gammad - 1.) * feps / fsig;
      double ent = log(WP(lane)[is]) - gam * log(WD(lane)[is]);
      s_igam[lane] = 1. / gam;
      s_expf[lane] = exp(-ent / gam);
    }
#endif
    __syncthreads();
#if EXO_MIXED
    // FP64 still, with the powers as exp(log(x) / gamma) and one log per face
    // shared by its two cells: ln psf and the face density of the isentropic
    // reference go to shared memory for the cells and for the restore
    each([&](int c, int i) {
      double* psf = PSF(c) + i;
      const double l = log(psf[0]);
      psf[per] = l;
      psf[2 * per] = exp(l * s_igam[c]) * s_expf[c];
    });
    __syncthreads();
    each([&](int c, int i) {
      if (i >= nc1) return;
      const double* psf = PSF(c) + i;
      const double igam = s_igam[c];
      double psv, dsv;
      if (fabs(psf[0] - psf[1]) < 1.E-6) {
        psv = (psf[0] + psf[1]) * 0.5;
        dsv = exp(log(psv) * igam) * s_expf[c];
      } else {
        // psv, the log-mean of the face pressures, is psf[i+1] (e^d - 1) / d
        // with d = ln psf[i] - ln psf[i+1], so ln psv = ln psf[i+1] + x +
        // ln(sinh x / x) (x = d/2) and psv^(1/gamma) = psf[i+1]^(1/gamma)
        // e^((x + ln(sinh x / x)) / gamma): the face density times two short
        // series instead of a log and an exp (layers thinner than 0.4 scale
        // heights; thicker ones take the log and the exp)
        const double d = psf[per] - psf[per + 1];
        psv = (psf[0] - psf[1]) / d;
        const double x = 0.5 * d;
        if (fabs(x) <= 0.2) dsv = psf[2 * per + 1] * exp_small((x + ln_sinhc(x)) * igam);
        else dsv = exp(log(psv) * igam) * s_expf[c];
      }
      T* f = WF(c) + i;
      f[IPR * nc1] = T(WP(c)[i] - psv);
      f[IDN * nc1] = T(WD(c)[i] - dsv);
    });
#else
    each([&](int c, int i) {
      if (i >= nc1) return;
      const double* psf = PSF(c) + i;
      double psv, dsv;
      if (fabs(psf[0] - psf[1]) < 1.E-6)
        psv = (psf[0] + psf[1]) / 2.;
      else
        psv = (psf[0] - psf[1]) / log(psf[0] / psf[1]);
      dsv = pow(psv, s_igam[c]) * s_expf[c];
      WP(c)[i] -= psv;
      WD(c)[i] -= dsv;
    });
#endif
    __syncthreads();
  }
  using TF = X1Flux<T>;
  TF* F = flux_array<TF>(v, 0);
#if EXO_MIXED
  // both face values of every cell is-1 .. ie+1, the cell's WENO5
  // smoothness indicators computed once for the two (as the x2/x3 kernel does)
  each([&](int c, int i) {
    if (i >= ncell) return;
    const T* q = WF(c) + is - 3 + i;
    T* rec = REC(c) + i;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const T q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4];
      const WenoCell<T> wcl = weno_cell<T>(q0, q1, q2, q3, q4);
      rec[0] = weno_right<T>(wcl, q0, q1, q2, q3, q4);
      rec[NV * ncell] = weno_left<T>(wcl, q0, q1, q2, q3, q4);
      q += nc1;
      rec += ncell;
    }
  });
  __syncthreads();
#endif
  each([&](int c, int f) {
    if (f > L) return;
    const double* psf = PSF(c) + is + f;
    FaceGeo<TF> fg{TF(0.), TF(1.), TF(s_cthp[c]), TF(s_cosc[c])};
    // perturbations are formed in FP64 above; WENO5 runs in T, the restore in
    // FP64 and the Riemann solve in TF
    TF wl[5], wr[5], fx[5];
#if EXO_MIXED
    const T* rec = REC(c) + f;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      wl[n] = TF(rec[0]);               // the upper face of cell i-1
      wr[n] = TF(rec[NV * ncell + 1]);  // the lower face of cell i
      rec += ncell;
    }
#else
    const double* q = COL(c) + is + f;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      wl[n] = weno_r<T>(q, 1, -1);
      wr[n] = weno_l<T>(q, 1, 0);
      q += nc1;
    }
#endif
    if (decomp) {
      // RestoreFromPerturbation (change_to_perturbation.cpp:159-222), in FP64
      double ps = psf[0];
      double xr = wr[IPR], xl = wl[IPR];
      xr += ps;
      if (xr < 0.) xr = ps;
      xl += ps;
      if (xl < 0.) xl = ps;
#if EXO_MIXED
      const double dsf = psf[2 * per];
#else
      double dsf = pow(ps, s_igam[c]) * s_expf[c];
#endif
      double dr = wr[IDN], dl = wl[IDN];
      dr += dsf;
      if (dr < 0.) dr = dsf;
      dl += dsf;
      if (dl < 0.) dl = dsf;
      wr[IPR] = TF(xr);
      wl[IPR] = TF(xl);
      wr[IDN] = TF(dr);
      wl[IDN] = TF(dl);
    }
    // x1 runs for the ideal gas only: LMARS or HLLC
    if (v.rsolver == EXO_RS_HLLC) riemann_hllc<TF>(riemann_gas<TF>(v.gas), IVX, fg, wl, wr, fx);
    else riemann_lmars<TF>(riemann_gas<TF>(v.gas), IVX, wl, wr, fx);
    TF* out = F + s_base[c] + f;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      *out = fx[n];
      out += vs;
    }
  });
}

// ----------------------------------------------------------- k_flux_x23 --
// Interior-side reconstruction of panel p at its own edge face (side s,
// along index a) for radial index i: the state CubedSphere::sendNeighborBlocks
// sends (L at Down/Right edges, R at Up/Left edges).
template <class T>
__device__ __forceinline__ void edge_interior_state(const DevView& v, int p, int s, int a,
                                                    int i, T* st) {
  long s2 = v.nc1, s3 = (long)v.nc1 * v.nc2;
  const T* W = prim_array<T>(v);
  #pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= v.nv) break;
    if (s == UP || s == DOWN) {
      const T* q = W + idx(v, p, n, v.ks + a, 0, i);
      st[n] = (s == DOWN) ? weno_r<T>(q, s2, v.je) : weno_l<T>(q, s2, v.js);
    } else {
      const T* q = W + idx(v, p, n, 0, v.js + a, i);
      st[n] = (s == RIGHT) ? weno_r<T>(q, s3, v.ke) : weno_l<T>(q, s3, v.ks);
    }
  }
}

template <class T>
__device__ __forceinline__ void edge_outer_state(const DevView& v, int p, int side, int a,
                                                 int i, T* st) {
  const EdgeEntry& e = v.edge[((size_t)p * 4 + side) * v.N + a];
  edge_interior_state<T>(v, e.src_panel, e.src_side, e.src_along, i, st);
  T V2 = st[IVY], V3 = st[IVZ];
  T U = T(e.r[0]) * V2 + T(e.r[1]) * V3;
  T V = T(e.r[2]) * V2 + T(e.r[3]) * V3;
  st[IVY] = T(e.q[0]) * U + T(e.q[1]) * V;
  st[IVZ] = T(e.q[2]) * U + T(e.q[3]) * V;
}

// asynchronous 8-byte global -> shared copies (the next level's inputs)
__device__ __forceinline__ void cp_async8(double* smem_dst, const double* gsrc) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
// one value of the implicit solve's factors (4 or 8 bytes)
template <class R>
__device__ __forceinline__ void cp_async_r(R* smem_dst, const R* gsrc) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(gsrc), "n"((int)sizeof(R))
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_one() {
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
}

// Faces staged through shared memory: a block of X23_THREADS threads takes 32
// lines of faces of one panel and direction, one per lane -- consecutive
// (line, radial index) pairs, so that a row of 32 lanes reads runs along i and
// no lane idles whatever the number of levels (with 32 radial indices of one
// line per block, 40 levels kept 62 % of the lanes busy, 45 levels 70 %) --
// and walks a segment of the lines in chunks of x23_chunk<T>() faces:
// the chunk's cells, with the three-cell halos of its stencils, are copied to
// shared memory while the chunk before is finished; one thread per face then
// reconstructs both of the face's states (WENO5) -- at a panel edge the outer
// one is the neighbour panel's rotated state -- and solves the Riemann problem.
// Where x23_shares_beta says so, the mixed build reconstructs per cell first
// (one thread per cell, both of its face values from one set of smoothness
// indicators, through shared memory) and solves per face after a barrier.
// What bounds it: instruction issue (mixed build, IPC 0.66 a scheduler) and
// the FP64 pipe (FP64 build, 67 % busy), not memory (17 % and 14 % of DRAM).
// Per launch, before (32 radial indices of one line per block, or one thread
// per face where those left lanes idle, places recomputed, divisions with
// range checks) and now: FP64 48^2x3 39 -> 23 us, 40^2x40 179 -> 103, 96^2x64
// 1029 -> 573; mixed 24^2x32 30 -> 19, 62^2x45 176 -> 97, 126^2x70 833 -> 454,
// 192^2x96 1626 -> 1120.
#ifndef EXO_X23_THREADS
#define EXO_X23_THREADS 128
#endif
constexpr int X23_THREADS = EXO_X23_THREADS;
// Whether the mixed build shares a cell's smoothness indicators between its
// two faces: a rule on the levels alone, since the two ways round
// differently and a run's results have to depend on nothing but its
// configuration.  (The line is where a block of 32 levels of one line used to
// give way to one thread per face, which did not share them.  Sharing at all
// levels would be faster: 20 levels of 126^2 157 -> 135 us, 33 of 96^2 168 ->
// 151, 41 of 62^2 96 -> 84.)
__host__ __device__ constexpr bool x23_shares_beta(int L) {
  return EXO_MIXED && L * 100 >= 65 * 32 * ((L + 31) / 32);
}
template <class T, bool kShareBeta>
__host__ __device__ constexpr int x23_chunk() {
  return kShareBeta ? 15 : sizeof(T) == 4 ? 16 : 8;
}
// resident blocks per SM: at 128 registers a thread, which the mixed build is
// held to (EXO_X23_MINB) and the FP64 build takes of itself
constexpr unsigned X23_RESIDENT = 4;

// cp.async of 4 or 8 bytes, zero-filled when src_bytes is 0
template <int B>
__device__ __forceinline__ void cp_async_zfill(void* smem_dst, const void* gsrc, int src_bytes) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(sa), "l"(gsrc), "n"(B),
               "r"(src_bytes)
               : "memory");
}

// The faces of a segment chunk by chunk.  Cell m of a line (m = 0 three cells
// below the first face) sits in ring slot (m - the segment's first) mod XR;
// the copies of chunk q + 1's new cells are in flight while chunk q is
// finished.  Slots written for chunk q + 1 held cells at least XR = 2 CF + 5
// below them, which chunk q no longer reads; the copies for chunk q + 2 start
// after the barrier that ends chunk q's reconstruction.  The ring's position,
// the lines' pointers and strides are carried along: recomputed per row of
// copies and per face, with divisions by the chunk's runtime length, they
// were 38 % of the mixed build's instructions.
template <class T, bool kShareBeta>
struct X23Shared {
  static constexpr int CF = x23_chunk<T, kShareBeta>(), XR = 2 * CF + 5;
  static constexpr int NC = kShareBeta ? CF + 1 : 1;
  T ring[5][XR][32];
  T srec[kShareBeta ? 2 : 1][5][NC][32];
};
template <class T, int NV, bool kShareBeta>
__device__ __forceinline__ void flux_x23_pipe(const DevView& v, unsigned blk, X23Shared<T, kShareBeta>& sm) {
  constexpr int CF = X23Shared<T, kShareBeta>::CF;
  constexpr int NC = X23Shared<T, kShareBeta>::NC;
  constexpr int XR = X23Shared<T, kShareBeta>::XR;
  auto& ring = sm.ring;
  auto& srec = sm.srec;
  const int N = v.N, L = v.L;
  const X23Split sp = v.x23;
  unsigned r = blk;
  const unsigned group = r % sp.groups;
  r /= sp.groups;
  const unsigned seg = r % sp.segments;
  r /= sp.segments;
  const int p = (int)(r % 6u);
  const int dir = (int)(r / 6u) + 1;
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
  constexpr int NW = X23_THREADS / 32;
  // this lane's line: place a across (k - ks for x2 faces, j - js for x3) and
  // radial index; lanes past the last line repeat it and store nothing
  const unsigned line = min(group * 32u + (unsigned)lane, (unsigned)(N * L) - 1u);
  const bool active = group * 32u + (unsigned)lane < (unsigned)(N * L);
  const int a = (int)v.div_L(line);
  const int i = v.is + (int)(line - (unsigned)a * (unsigned)L);
  const size_t vs = v.cells;
  const size_t s = dir == 1 ? (size_t)v.nc1 : (size_t)v.nc1 * v.nc2;
  // the first face's place in the state and flux arrays
  const size_t base = dir == 1 ? idx(v, p, 0, v.ks + a, v.js, i) : idx(v, p, 0, v.ks, v.js + a, i);
  const T* const W = prim_array<T>(v) + base - 3 * s;  // cell 0
  T* const F = flux_array<T>(v, dir) + base;           // face 0
  const int q0 = (int)(seg * sp.chunks);
  const int q1 = min((N + CF) / CF, q0 + (int)sp.chunks);
  const int rsolver = v.rsolver;
  // copies of the cells [m0, m0 + n), the first of them in slot slot0
  auto issue = [&](int m0, int n, int slot0) {
#pragma unroll 1
    for (int c = warp; c < n; c += NW) {
      const int m = m0 + c;
      int slot = slot0 + c;
      slot -= (slot >= XR) ? XR : 0;
      const bool ok = m < N + 6;
      const T* src = W + (size_t)(ok ? m : 3) * s;
      T* dst = &ring[0][slot][lane];
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        cp_async_zfill<sizeof(T)>(dst + q * (XR * 32), src, ok ? (int)sizeof(T) : 0);
        src += vs;
      }
    }
    cp_async_commit();
  };
  issue(q0 * CF, CF + 5, 0);
  int islot = CF + 5, rslot = 0;  // slots of the next cell to copy and of cell q CF
#pragma unroll 1
  for (int q = q0; q < q1; ++q) {
    cp_async_wait_all();
    __syncthreads();
    if (q + 1 < q1) {
      issue(q * CF + CF + 5, CF, islot);
      islot += CF;
      islot -= (islot >= XR) ? XR : 0;
    }
    if constexpr (kShareBeta) {
      // both face values of the cells below and above the chunk's faces
#pragma unroll 1
      for (int mc = warp; mc < NC; mc += NW) {
        const T* st[5];  // the cell's stencil
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          int sl = rslot + mc + m;
          sl -= (sl >= XR) ? XR : 0;
          st[m] = &ring[0][sl][lane];
        }
        T* const rec = &srec[0][0][mc][lane];
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const T c0 = st[0][n * (XR * 32)], c1 = st[1][n * (XR * 32)], c2 = st[2][n * (XR * 32)];
          const T c3 = st[3][n * (XR * 32)], c4 = st[4][n * (XR * 32)];
          const WenoCell<T> wc = weno_cell<T>(c0, c1, c2, c3, c4);
          rec[n * (NC * 32)] = weno_right<T>(wc, c0, c1, c2, c3, c4);
          rec[(5 + n) * (NC * 32)] = weno_left<T>(wc, c0, c1, c2, c3, c4);
        }
      }
      __syncthreads();
    }
    // the faces q CF .. q CF + CF - 1 (up to N)
#pragma unroll 1
    for (int mf = warp; mf < CF; mf += NW) {
      const int f = q * CF + mf;
      if (f > N || !active) break;
      T wl[5], wr[5], fx[5] = {T(0.), T(0.), T(0.), T(0.), T(0.)};
      if constexpr (kShareBeta) {
        const T* const rec = &srec[0][0][mf][lane];
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          wl[n] = rec[n * (NC * 32)];
          wr[n] = rec[(5 + n) * (NC * 32) + 32];
        }
      } else {
        const T* st[6];  // the three cells below the face and the three above
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          int sl = rslot + mf + m;
          sl -= (sl >= XR) ? XR : 0;
          st[m] = &ring[0][sl][lane];
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          T c[6];
#pragma unroll
          for (int m = 0; m < 6; ++m) c[m] = st[m][n * (XR * 32)];
          wl[n] = weno5<T>(c[4], c[3], c[2], c[1], c[0]);
          wr[n] = weno5<T>(c[1], c[2], c[3], c[4], c[5]);
        }
      }
      if (dir == 1) {
        if (f == 0) edge_outer_state<T>(v, p, UP, a, i, wl);
        else if (f == N) edge_outer_state<T>(v, p, DOWN, a, i, wr);
        const int k = v.ks + a, j = v.js + f;
        FaceGeo<T> fg{T(geo(v, GCOSF2, p, k, j)), T(geo(v, GSINF2, p, k, j)),
                      T(geo(v, GCTHP2, p, k, j)), T(geo(v, GCOSC, p, k, j))};
        riemann<T>(rsolver, v.gas, IVY, fg, wl, wr, fx);
      } else {
        if (f == 0) edge_outer_state<T>(v, p, LEFT, a, i, wl);
        else if (f == N) edge_outer_state<T>(v, p, RIGHT, a, i, wr);
        const int k = v.ks + f, j = v.js + a;
        FaceGeo<T> fg{T(geo(v, GCOSF3, p, k, j)), T(geo(v, GSINF3, p, k, j)),
                      T(geo(v, GCTHP3, p, k, j)), T(geo(v, GCOSC, p, k, j))};
        riemann<T>(rsolver, v.gas, IVZ, fg, wl, wr, fx);
      }
      T* out = F + (size_t)f * s;
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        *out = fx[n];
        out += vs;
      }
    }
    rslot += CF;
    rslot -= (rslot >= XR) ? XR : 0;
  }
}

template <class T>
__device__ __forceinline__ void flux_x23_block(const DevView& v, unsigned blk) {
  if constexpr (EXO_MIXED) {
    __shared__ union {
      __align__(16) X23Shared<T, true> cells;
      __align__(16) X23Shared<T, false> faces;
    } sm;
    if (x23_shares_beta(v.L)) {
      if (v.nv == 5) flux_x23_pipe<T, 5, true>(v, blk, sm.cells);
      else flux_x23_pipe<T, 4, true>(v, blk, sm.cells);
    } else {
      if (v.nv == 5) flux_x23_pipe<T, 5, false>(v, blk, sm.faces);
      else flux_x23_pipe<T, 4, false>(v, blk, sm.faces);
    }
  } else {
    __shared__ __align__(16) X23Shared<T, false> sm;
    if (v.nv == 5) flux_x23_pipe<T, 5, false>(v, blk, sm);
    else flux_x23_pipe<T, 4, false>(v, blk, sm);
  }
}

// --------------------------------------------------------------- k_update -
template <class T>
__device__ __forceinline__ void update_block(const DevView& v, unsigned blk, int stage) {
  const unsigned tid = blk * blockDim.x + threadIdx.x;
  const unsigned L = v.L, N = v.N;
  if (tid >= 6u * N * N * L) return;
  const unsigned r1 = v.div_L(tid), r2 = v.div_N(r1), r3 = v.div_N(r2);
  const int i = v.is + (int)(tid - r1 * L);
  const int j = v.js + (int)(r1 - r2 * N);
  const int k = v.ks + (int)(r2 - r3 * N);
  const int p = (int)r3;
  const double wght = rk_beta(stage) * v.sc->dt;
  const bool shallow = (v.eqn == EXO_EQN_SHALLOW_YZ);
  const int nv = v.nv;
  // offsets: this cell (variable 0), variable stride, +1 in j and in k
  const size_t c0 = idx(v, p, 0, k, j, i), vs = v.cells;
  const size_t sj = (size_t)v.nc1, sk = (size_t)v.nc2 * v.nc1;
  // geometry of the column (k,j) and of its upper x2/x3 neighbours
  const size_t g0 = ((size_t)p * v.nc3 + k) * v.nc2 + j, gs = (size_t)6 * v.nc3 * v.nc2;
  auto G2 = [&](int f, size_t off) { return __ldg(v.geo + f * gs + g0 + off); };
  const double* uin = v.u + c0;  // read here, written below
  const double* u1in = v.u1 + c0;
  const double* __restrict__ win = v.w + c0;
  const X1Flux<T>* __restrict__ F0 = flux_array<X1Flux<T>>(v, 0) + c0;
  const T* __restrict__ F1 = flux_array<T>(v, 1) + c0;
  const T* __restrict__ F2 = flux_array<T>(v, 2) + c0;
  // every input of the cell is requested before any is used
  double uu[5], u1v[5], wv[5];
  X1Flux<T> f0l[5], f0r[5];
  T f1l[5], f1r[5], f2l[5], f2r[5];
#pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= nv) break;
    uu[n] = uin[n * vs];
    u1v[n] = stage ? u1in[n * vs] : 0.;
    wv[n] = __ldg(win + n * vs);
    f0l[n] = shallow ? X1Flux<T>(0.) : __ldg(F0 + n * vs);
    f0r[n] = shallow ? X1Flux<T>(0.) : __ldg(F0 + n * vs + 1);
    f1l[n] = __ldg(F1 + n * vs);
    f1r[n] = __ldg(F1 + n * vs + sj);
    f2l[n] = __ldg(F2 + n * vs);
    f2r[n] = __ldg(F2 + n * vs + sk);
  }
  const double x1fi = __ldg(v.x1f + i), x1fp = __ldg(v.x1f + i + 1);
  const double x1vi = __ldg(v.x1v + i), dx1fi = __ldg(v.dx1f + i);
  double un[5];
  // WeightedAve(u1, u, ...) then WeightedAve(u, u1, ...) (SSPRK(3,3) registers)
#pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= nv) break;
    if (stage == 0) {
      v.u1[c0 + n * vs] = uu[n];
      un[n] = 0. + 1.0 * uu[n];
    } else if (stage == 1) {
      un[n] = 0.25 * uu[n] + 0.75 * u1v[n];
    } else {
      un[n] = (2.0 / 3.0) * uu[n] + (1.0 / 3.0) * u1v[n];
    }
  }
  // AddFluxDivergence
  const double s = G2(GSINC, 0);
  const double d2 = G2(GDX2A, 0), d3 = G2(GDX3A, 0);
  const double dx3f2 = G2(GDX3A_F2, 0), dx3f2p = G2(GDX3A_F2, 1);
  const double dx2f3 = G2(GDX2A_F3, 0), dx2f3p = G2(GDX2A_F3, v.nc2);
  const double a1 = d2 * d3 * x1fi * x1fi * s;
  const double a1p = d2 * d3 * x1fp * x1fp * s;
  const double a2 = x1vi * dx3f2 * dx1fi;
  const double a2p = x1vi * dx3f2p * dx1fi;
  const double a3 = x1vi * dx2f3 * dx1fi;
  const double a3p = x1vi * dx2f3p * dx1fi;
  const double vol = dx1fi * d2 * d3 * x1vi * x1vi * s;
  // the mixed build multiplies by reciprocals of the volume and the radius
  // (one division each instead of eight); the FP64 build's quotients are the
  // reference's, from one reciprocal each
#if EXO_MIXED
  const double ivol = inv_r(vol), irad = inv_r(x1vi);
#else
  const SharedDiv by_vol(vol), by_radius(x1vi);
#endif
  double du[5];
  // flux divergence in T (the x1 part in FP64 where its fluxes are); the
  // conserved state accumulates in FP64
  const T A1 = T(a1), A1p = T(a1p), A2 = T(a2), A2p = T(a2p), A3 = T(a3), A3p = T(a3p);
#pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= nv) break;
    double change;
#if !EXO_MIXED
    T dflx = (A1p * f0r[n] - A1 * f0l[n]);
    dflx += (A2p * f1r[n] - A2 * f1l[n]);
    dflx += (A3p * f2r[n] - A3 * f2l[n]);
    change = by_vol.finite(wght * dflx);
#else
    if constexpr (sizeof(X1Flux<T>) == sizeof(double)) {
      T d23 = (A2p * f1r[n] - A2 * f1l[n]);
      d23 += (A3p * f2r[n] - A3 * f2l[n]);
      const double d1 = a1p * f0r[n] - a1 * f0l[n];
      change = wght * ((d1 + (double)d23) * ivol);
    } else {
      T dflx = (A1p * f0r[n] - A1 * f0l[n]);
      dflx += (A2p * f1r[n] - A2 * f1l[n]);
      dflx += (A3p * f2r[n] - A3 * f2l[n]);
      change = wght * (double)(dflx / T(vol));
    }
#endif
    if (shallow) {
      un[n] -= change;
    } else {
      du[n] = 0.;
      du[n] -= change;
    }
  }
  double* out = shallow ? un : du;
  // AddCoordTermsDivergence (gnomonic_equiangle.cpp:834-879)
  {
    const double cosine = G2(GCOSC, 0);
    const double sine2 = s * s;
#if EXO_MIXED
    const double x_ov_rD = (x1vi * dx3f2 * dx1fi * G2(GSINF2, 0) -
                            x1vi * dx3f2p * dx1fi * G2(GSINF2, 1)) * ivol;
    const double y_ov_rC = (x1vi * dx2f3 * dx1fi * G2(GSINF3, 0) -
                            x1vi * dx2f3p * dx1fi * G2(GSINF3, v.nc2)) * ivol;
#else
    const double x_ov_rD = by_vol.finite(x1vi * dx3f2 * dx1fi * G2(GSINF2, 0) -
                                  x1vi * dx3f2p * dx1fi * G2(GSINF2, 1));
    const double y_ov_rC = by_vol.finite(x1vi * dx2f3 * dx1fi * G2(GSINF3, 0) -
                                  x1vi * dx2f3p * dx1fi * G2(GSINF3, v.nc2));
#endif
    const double rho = wv[IDN], v1 = wv[IVX], v2 = wv[IVY], v3 = wv[IVZ];
    double pr;
    const double v_2 = v2 + v3 * cosine;
    const double v_3 = v3 + v2 * cosine;
    if (shallow) {
      pr = 0.5 * rho * rho;
    } else {
      pr = wv[IPR];
#if EXO_MIXED
      double src1 = (2.0 * pr + rho * (v2 * v_2 + v3 * v_3)) * irad;
#else
      double src1 = by_radius.finite(2.0 * pr + rho * (v2 * v_2 + v3 * v_3));
#endif
      out[IVX] += wght * src1;
    }
#if EXO_MIXED
    double src2 = -x_ov_rD * (pr + rho * v3 * v3 * sine2) - rho * v1 * v_2 * irad;
    out[IVY] += wght * src2;
    double src3 = -y_ov_rC * (pr + rho * v2 * v2 * sine2) - rho * v1 * v_3 * irad;
#else
    double src2 = -x_ov_rD * (pr + rho * v3 * v3 * sine2) - by_radius.finite(rho * v1 * v_2);
    out[IVY] += wght * src2;
    double src3 = -y_ov_rC * (pr + rho * v2 * v2 * sine2) - by_radius.finite(rho * v1 * v_3);
#endif
    out[IVZ] += wght * src3;
    // constant gravity (patches/25.constant_acc.patch:35-53)
    if (v.grav != 0.) {
      double src = wght * rho * v.grav;
      out[IVX] += src;
      if (!shallow) out[IEN] += src * v1;
    }
    // W92 Coriolis (examples/2023-Chen-exo3/W92.cpp:48-70)
    if (v.coriolis == EXO_CORIOLIS_W92) {
      double f = G2(GFCOR, 0);
      double U = G2(GCR0, 0) * v2 + G2(GCR1, 0) * v3;
      double V = G2(GCR2, 0) * v2 + G2(GCR3, 0) * v3;
      U = -U;
      double llU = f * V, llV = -f * U;
      double mU = -llU;
      double acc2 = G2(GCQ0, 0) * mU + G2(GCQ1, 0) * llV;
      double acc3 = G2(GCQ2, 0) * mU + G2(GCQ3, 0) * llV;
      double a2c = acc2 + acc3 * cosine, a3c = acc3 + acc2 * cosine;
      out[IVY] += wght * rho * a2c;
      out[IVZ] += wght * rho * a3c;
    }
    // CubedSphere::CalculateCoriolisForce3 (cubed_sphere.cpp:197-231): blocks
    // 1 and 5 (panels 0 and 4) carry the rotation axis through their centre
    if (v.coriolis == EXO_CORIOLIS_3D) {
      const double A = G2(GC3A, 0) * rho;
      const double x = G2(GTANX, 0), y = G2(GTANY, 0), C = G2(GC3C, 0), D = G2(GC3D, 0);
      double cF1, cF2, cF3;
      if (p == 0 || p == 4) {
        cF1 = A * (y * C * v2 - x * D * v3);
        cF2 = A * (-y * C * v1 - v3);
        cF3 = A * (x * D * v1 + v2);
      } else {
        cF1 = -A * D * v3;
        cF2 = A * x * v3;
        cF3 = A * (D * v1 - x * v2);
      }
      out[IVX] += wght * cF1;
      out[IVY] += wght * cF2;
      out[IVZ] += wght * cF3;
    }
    // Held-Suarez forcing (examples/2023-Chen-exo3/hs94.cpp:59-155)
    if (v.forcing == EXO_FORCING_HS94) {
      // Coriolis on the momenta in latitude-longitude (hs94.cpp:82-104)
      {
        double f = G2(GFCOR, 0);
        double U = G2(GCR0, 0) * v2 + G2(GCR1, 0) * v3;
        double V = G2(GCR2, 0) * v2 + G2(GCR3, 0) * v3;
        U = -U;
        double m2 = rho * U, m3 = rho * V;
        double llU = f * m3, llV = -f * m2;
        double mU = -llU;
        double acc2 = G2(GCQ0, 0) * mU + G2(GCQ1, 0) * llV;
        double acc3 = G2(GCQ2, 0) * mU + G2(GCQ3, 0) * llV;
        double a2c = acc2 + acc3 * cosine, a3c = acc3 + acc2 * cosine;
        out[IVY] += wght * a2c;
        out[IVZ] += wght * a3c;
      }
      // Rayleigh drag and Newtonian cooling (hs94.cpp:110-153)
      {
        const double* hs = v.hs;
        double scaled_z = pr / hs[HS_P0];
        double sigma = pr / hs[HS_P0];
        double sigma_p = (sigma - hs[HS_SIGMAB]) / (1. - hs[HS_SIGMAB]);
        double Kv = (sigma_p < 0.0) ? 0.0 : sigma_p * hs[HS_KF];
        double Teq_p = hs[HS_TS] - hs[HS_DT] * G2(GSLAT2, 0) -
                       hs[HS_DTHETA] * log(scaled_z) * G2(GCLAT2, 0);
        Teq_p *= pow(scaled_z, hs[HS_KAPPA]);
        double Teq = (Teq_p > 200.) ? Teq_p : 200.;
        double temp = pr / rho / v.Rd;
        sigma_p = (sigma_p < 0.0) ? 0.0 : sigma_p * G2(GCLAT4, 0);
        double Kt = hs[HS_KA] + (hs[HS_KS] - hs[HS_KA]) * sigma_p;
        double m1 = rho * v1, m2 = rho * v2, m3 = rho * v3;
        double m2c = m2 + m3 * cosine, m3c = m3 + m2 * cosine;
        out[IVX] += -wght * Kv * m1;
        out[IVY] += -wght * Kv * m2c;
        out[IVZ] += -wght * Kv * m3c;
        out[IEN] += -wght * hs[HS_CVM] * rho * Kt * (temp - Teq);
      }
    }
  }
  double* uout = v.u + c0;
  if (shallow) {
#pragma unroll
    for (int n = 0; n < 4; ++n) uout[n * vs] = un[n];
  } else if (v.implicit_flag & 1) {
    // the 3x3 correction leaves the tangential momenta's update as it is, so
    // it is applied here and the solve moves neither
    double* duout = v.du + c0;
    const bool partial = !(v.implicit_flag & 8);
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      if (partial && (n == IVY || n == IVZ)) {
        uout[n * vs] = un[n] + 1. * du[n];
      } else {
        uout[n * vs] = un[n];
        duout[n * vs] = du[n];
      }
    }
  } else {
#pragma unroll
    for (int n = 0; n < 5; ++n) uout[n * vs] = un[n] + 1. * du[n];
  }
}

// ------------------------------------------------------------- k_implicit -
// flux_decomposition.hpp:34-120, X1 direction
#if !EXO_MIXED
struct GasDiv {
  SharedDiv gm1, gp1;  // divisions by gamma - 1 and by gamma - 1 + 1
};
__device__ __forceinline__ void roe_average(double* prim, double gm1, const GasDiv& gd,
                                            const double* wl, const double* wr) {
  double sqrtdl = sqrt(wl[IDN]), sqrtdr = sqrt(wr[IDN]);
  double isdlpdr = 1.0 / (sqrtdl + sqrtdr);
  prim[IDN] = sqrtdl * sqrtdr;
  prim[IVX] = (sqrtdl * wl[IVX] + sqrtdr * wr[IVX]) * isdlpdr;
  prim[IVY] = (sqrtdl * wl[IVY] + sqrtdr * wr[IVY]) * isdlpdr;
  prim[IVZ] = (sqrtdl * wl[IVZ] + sqrtdr * wr[IVZ]) * isdlpdr;
  double el = gd.gm1.finite(wl[IPR]) + 0.5 * wl[IDN] * (sqr(wl[IVX]) + sqr(wl[IVY]) + sqr(wl[IVZ]));
  double er = gd.gm1.finite(wr[IPR]) + 0.5 * wr[IDN] * (sqr(wr[IVX]) + sqr(wr[IVY]) + sqr(wr[IVZ]));
  double hbar = ((el + wl[IPR]) / sqrtdl + (er + wr[IPR]) / sqrtdr) * isdlpdr;
  prim[IPR] = gd.gp1.finite((hbar - 0.5 * (sqr(prim[IVX]) + sqr(prim[IVY]) + sqr(prim[IVZ]))) * gm1) *
              prim[IDN];
}
#endif

// Structural non-zeros of the X1 flux Jacobian dF/dq (flux_decomposition.hpp:
// 100-120): row 0 = e_1; rows 2 and 3 carry three entries each.
__host__ __device__ constexpr bool fj_nz(int r, int q) {
  return r == 1 || r == 4 || (r == 0 && q == 1) || (r == 2 && q <= 2) ||
         (r == 3 && (q <= 1 || q == 3));
}
// structural non-zeros of R (right eigenvectors, columns) and R^-1 (rows)
__host__ __device__ constexpr bool r_nz(int r, int c) {
  return c < 3 || (r == 2 && c == 3) || (r == 3 && c == 4) || r == 4;
}
__host__ __device__ constexpr bool ri_nz(int r, int c) {
  return r < 3 || c == 0 || (r == 3 && c == 2) || (r == 4 && c == 3);
}

// One cell of a column, velocities projected (v2 += v3 cos, v3 *= sin): the
// primitives and the two derived quantities of its flux Jacobian.
template <class R>
struct ColCell {
  R rho, v1, v2, v3, p, s2, hr;  // s2 = |v|^2, hr = (g+1)/g * p/rho (g = gamma-1)
  R sq, isq;                     // sqrt(rho), 1/sqrt(rho) (FP32 blocks)
};

// entry (r, q) of dF/dq at a cell, in the reference's expression order
template <int r, int q, class R>
__device__ __forceinline__ R fj_entry(const ColCell<R>& c, R gm1) {
  if constexpr (r == 0) return R(1);
  else if constexpr (r == 1) {
    if constexpr (q == 0) return gm1 * c.s2 / 2 - c.v1 * c.v1;
    else if constexpr (q == 1) return (R(2) - gm1) * c.v1;
    else if constexpr (q == 2) return -gm1 * c.v2;
    else if constexpr (q == 3) return -gm1 * c.v3;
    else return gm1;
  } else if constexpr (r == 2) {
    if constexpr (q == 0) return -c.v1 * c.v2;
    else if constexpr (q == 1) return c.v2;
    else return c.v1;
  } else if constexpr (r == 3) {
    if constexpr (q == 0) return -c.v1 * c.v3;
    else if constexpr (q == 1) return c.v3;
    else return c.v1;
  } else {
    if constexpr (q == 0) return ((gm1 - 1) * c.s2 / 2 - c.hr) * c.v1;
    else if constexpr (q == 1) return c.hr + c.s2 / 2 - gm1 * c.v1 * c.v1;
    else if constexpr (q == 2) return -gm1 * c.v2 * c.v1;
    else if constexpr (q == 3) return -gm1 * c.v3 * c.v1;
    else return (gm1 + 1) * c.v1;
  }
}

// compile-time loops (the matrix entries live in registers, so every index
// has to be a constant)
template <int N, class F, int... I>
__device__ __forceinline__ void unroll_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void unroll(F&& f) {
  unroll_impl<N>(f, std::make_integer_sequence<int, N>{});
}

#if EXO_MIXED
// |A| = R |Lambda| R^-1 at the Roe average of a face (flux_decomposition.hpp:
// 34-98) as |u| I + (|u-c|-|u|) r0 l0^T + (|u+c|-|u|) r2 l2^T (the three |u|
// eigenvalues coincide), with shared reciprocals.  FP32 blocks take sqrt(rho)
// and 1/sqrt(rho) from the cells and the sound speed and its reciprocal from
// one rsqrt (one rsqrt and two reciprocals a face; 1.6 % faster); FP64 blocks
// keep sqrt and division, which measured 3 % faster than the same rewrite in
// FP64.
template <class R>
__device__ __forceinline__ void abs_jacobian(const ColCell<R>& L, const ColCell<R>& R_, R gm1,
                                             R gamma, R A[5][5]) {
  R wl[5] = {L.rho, L.v1, L.v2, L.v3, L.p};
  R wr[5] = {R_.rho, R_.v1, R_.v2, R_.v3, R_.p};
  // FP32 blocks take the cells' sqrt(rho) and 1/sqrt(rho); the same scheme
  // in FP64 (with a Newton-refined rsqrt) measured 0.5 % slower
  constexpr bool f32 = sizeof(R) == 4;
  const R one = R(1), half = R(0.5);
  R sqrtdl, sqrtdr, isl, isr, isdlpdr;
  if constexpr (f32) {
    sqrtdl = L.sq;
    sqrtdr = R_.sq;
    isdlpdr = inv_r(sqrtdl + sqrtdr);
    isl = isdlpdr * L.isq;
    isr = isdlpdr * R_.isq;
  } else {
    sqrtdl = sqrt_r(wl[IDN]);
    sqrtdr = sqrt_r(wr[IDN]);
    isdlpdr = inv_r(sqrtdl + sqrtdr);
    if constexpr (EXO_IMPL_RCP_NR) {
      isl = isdlpdr * inv_r(sqrtdl);
      isr = isdlpdr * inv_r(sqrtdr);
    } else {
      isl = isdlpdr / sqrtdl;
      isr = isdlpdr / sqrtdr;
    }
  }
  R rr = sqrtdl * sqrtdr;
  R u = (sqrtdl * wl[IVX] + sqrtdr * wr[IVX]) * isdlpdr;
  R v = (sqrtdl * wl[IVY] + sqrtdr * wr[IVY]) * isdlpdr;
  R w = (sqrtdl * wl[IVZ] + sqrtdr * wr[IVZ]) * isdlpdr;
  R inv_gm1 = one / gm1;
  R el = wl[IPR] * inv_gm1 + half * wl[IDN] * L.s2;
  R er = wr[IPR] * inv_gm1 + half * wr[IDN] * R_.s2;
  R hbar = (el + wl[IPR]) * isl + (er + wr[IPR]) * isr;
  R ke = half * (u * u + v * v + w * w);
  R p = (hbar - ke) * (gm1 / (gm1 + one)) * rr;
  R irr, cs, i2cshp;
  if constexpr (f32) {
    irr = L.isq * R_.isq;
    const R cs2 = gamma * p * irr;
    const R ics = rsqrt_r(cs2);
    cs = cs2 * ics;
    i2cshp = ics;  // times 1/(2 hp) below
  } else {
    irr = inv_r(rr);
    cs = sqrt_r(gamma * p * irr);
  }
  R hp = (gm1 + one) * inv_gm1 * p * irr;
  R h = hp + ke;
  R ihp = inv_r(hp), i2hp = half * ihp;
  if constexpr (f32)
    i2cshp *= i2hp;
  else if constexpr (EXO_IMPL_RCP_NR)
    i2cshp = i2hp * inv_r(cs);
  else
    i2cshp = i2hp / cs;
  R au = abs_r(u), al = abs_r(u - cs) - au, ar = abs_r(u + cs) - au;
  R l0[5] = {al * (cs * ke + u * hp) * i2cshp, al * (-hp - cs * u) * i2cshp, -al * v * i2hp,
              -al * w * i2hp, al * i2hp};
  R l2[5] = {ar * (cs * ke - u * hp) * i2cshp, ar * (hp - cs * u) * i2cshp, -ar * v * i2hp,
              -ar * w * i2hp, ar * i2hp};
  R r0[5] = {one, u - cs, v, w, h - u * cs};
  R r2[5] = {one, u + cs, v, w, h + u * cs};
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c) A[r][c] = (r == c ? au : R(0)) + r0[r] * l0[c] + r2[r] * l2[c];
}
#else
// |A| = R |Lambda| R^-1 at the Roe average of a face (flux_decomposition.hpp:
// 34-98): the reference's products R*Lambda and (R*Lambda)*R^-1 summed in its
// order, skipping only terms that are structurally zero (the value is the
// same; at most the sign of an exact zero differs).
__device__ __forceinline__ void abs_jacobian(const ColCell<double>& L, const ColCell<double>& R_,
                                             double gm1, double gamma, const GasDiv& gd,
                                             double A[5][5]) {
  const double wl[5] = {L.rho, L.v1, L.v2, L.v3, L.p};
  const double wr[5] = {R_.rho, R_.v1, R_.v2, R_.v3, R_.p};
  double prim[5];
  roe_average(prim, gm1, gd, wl, wr);
  double fsig = 1., feps = 1.;
  double rr = prim[IDN], u = prim[IVX], v = prim[IVY], w = prim[IVZ], p = prim[IPR];
  // divisions by a common denominator share its reciprocal (SharedDiv: the
  // IEEE quotient)
  const SharedDiv by_rr(rr);
  double cs = sqrt(by_rr.finite((1. + (gamma - 1) * feps / fsig) * p));
  double ke = 0.5 * (u * u + v * v + w * w);
  double hp = by_rr.finite((gm1 + 1.) / gm1 * p);
  double h = hp + ke;
  const double Rm[5][5] = {{1., 1., 1., 0., 0.},
                           {u - cs, u, u + cs, 0., 0.},
                           {v, v, v, 1., 0.},
                           {w, w, w, 0., 1.},
                           {h - u * cs, ke, h + u * cs, v, w}};
  const SharedDiv by_hp(hp), by_2hp(2. * hp), by_2cshp(2. * cs * hp);
  double mv2 = by_2hp.finite(-v), mw2 = by_2hp.finite(-w), i2 = by_2hp.r;
  const double Ri[5][5] = {
      {by_2cshp.finite(cs * ke + u * hp), by_2cshp.finite(-hp - cs * u), mv2, mw2, i2},
      {by_hp.finite(hp - ke), by_hp.finite(u), by_hp.finite(v), by_hp.finite(w), -by_hp.r},
      {by_2cshp.finite(cs * ke - u * hp), by_2cshp.finite(hp - cs * u), mv2, mw2, i2},
      {-v, 0., 1., 0., 0.},
      {-w, 0., 0., 1., 0.}};
  const double lam[5] = {fabs(u - cs), fabs(u), fabs(u + cs), fabs(u), fabs(u)};
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      double s = 0.;
      bool first = true;
#pragma unroll
      for (int k = 0; k < 5; ++k)
        if (r_nz(r, k) && ri_nz(k, c)) {
          double term = (Rm[r][k] * lam[k]) * Ri[k][c];
          s = first ? term : s + term;
          first = false;
        }
      A[r][c] = s;
    }
}
#endif

// Solve with the LU factors of implicit_column's mixed build (rows taken in
// the order 1, 4, 2, 3, 0): y holds the right-hand side, its rows already
// swapped as the factors' were, on entry and the solution, unknowns in
// order, on exit.
template <class R>
__device__ __forceinline__ void lu_solve_rows(const R (&t)[5][5], const R (&idg)[5], R* y) {
  constexpr int O[5] = {1, 4, 2, 3, 0};
#pragma unroll
  for (int r = 1; r < 5; ++r)
#pragma unroll
    for (int k = 0; k < r; ++k) y[O[r]] -= t[O[r]][k] * y[O[k]];
  R z[5];
#pragma unroll
  for (int r = 4; r >= 0; --r) {
    R acc = y[O[r]];
#pragma unroll
    for (int q = r + 1; q < 5; ++q) acc -= t[O[r]][q] * z[q];
    z[r] = acc * idg[r];
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) y[r] = z[r];
}

// The forward sweep's inputs, w(i+1) and du(i) of level i, brought in by the
// whole warp four levels at a time (lane -> level lane & 3 of columns
// (lane >> 2) + 8 m).  What limits these loads is not bytes but the 128-byte
// lines of L1 they hold while in flight, one per (column, variable) run,
// whatever the run's length: with copies of one level per lane, and with
// runs of two, more warps per SM made the solve slower (fewer lines left of
// L1 beside their shared memory).  A level takes a warp several
// microseconds among seven others, so the batch is waited for where it is
// issued: a second buffer would only cost shared memory.  Column c keeps
// level k at place (k + c/4) & 3, which keeps a warp's reads of one level on
// distinct banks.
constexpr int LEVEL_TILE_DOUBLES = 10 * 32 * 4;
template <class IO, int ND>
struct LevelTile {
  double* tile;
  int is, L;
  __device__ __forceinline__ static int var(int m) {
    return ND == 5 ? m : (m == 2 ? IEN : m);
  }
  __device__ __forceinline__ LevelTile(const IO&, double* t, int is_, int L_)
      : tile(t), is(is_), L(L_) {}
  // level k's values are about to be read
  __device__ __forceinline__ void ready(const IO& io, int k0) {
    if (k0 & 3) return;
    const int lane = (int)(threadIdx.x & 31), k = k0 + (lane & 3);
    __syncwarp();
    const unsigned long long wo =
        reinterpret_cast<unsigned long long>(io.wptr(is + 1 + k0, 0));
    const unsigned long long uo = reinterpret_cast<unsigned long long>(io.duptr(is + k0, 0));
    const size_t ws = io.wstride(), ds = io.dstride();
#pragma unroll 1
    for (int m = 0; m < 4; ++m) {
      const int c = (lane >> 2) + 8 * m;
      const double* wp = reinterpret_cast<const double*>(__shfl_sync(0xffffffffu, wo, c)) +
                         (lane & 3);
      const double* dp = reinterpret_cast<const double*>(__shfl_sync(0xffffffffu, uo, c)) +
                         (lane & 3);
      if (k < L) {
        double* d = tile + c * 4 + ((k + (c >> 2)) & 3);
#pragma unroll
        for (int n = 0; n < 5; ++n) cp_async8(d + n * 128, wp + n * ws);
#pragma unroll
        for (int n = 0; n < ND; ++n) cp_async8(d + (5 + n) * 128, dp + var(n) * ds);
      }
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncwarp();
  }
  // value n of level k of this lane's column
  __device__ __forceinline__ double* place(int n, int k) const {
    const int lane = (int)(threadIdx.x & 31);
    return tile + n * 128 + lane * 4 + ((k + (lane >> 2)) & 3);
  }
  __device__ __forceinline__ double get(int n, int k) const { return *place(n, k); }
};

// shared memory of a warp of the solve: the level tile, then NE values of R
// per lane, two face matrices (entry e of lane l at [e * 32 + l])
template <class R, bool full>
__host__ __device__ constexpr int impl_warp_doubles() {
  constexpr int ne = full ? 50 : 18;
  return LEVEL_TILE_DOUBLES + ne * 32 * (int)sizeof(R) / 8;
}
// The vertical 5x5 block-tridiagonal correction of one radial column
// (ImplicitSolver::SolveImplicit3D X1 branch, solve_implicit_3d.cpp:102-179,
// with FullCorrection, full_correction.cpp:32-165, and ForwardSweep /
// BackwardSubstitution, forward_backward.hpp:15-126), one thread per column.
//
// Per level the forward sweep builds the rows of a_i, b_i, c_i from the two
// face Jacobians |A|(i-1/2), |A|(i+1/2) and the three cell Jacobians, forms
// t = a_i - b_i (A c)_{i-1} and x = du_i/dt - b_i delta_{i-1} row by row,
// then
//   exact build: inverts t by Gauss-Jordan with partial pivoting (the
//                reference's inverse) and multiplies, every sum in the
//                reference's order: the result is the CPU restatement's to
//                the bit;
//   mixed build: solves t [X | y] = [c_i | x] by LU with partial pivoting
//                (FP32 blocks; FP64 ones run implicit_column_fused).
// (A c)_i (25) and delta_i (5) go to scratch for the back substitution
// (kb_implicit_bwd).
//
// What bounds it: at 252 registers eight warps share an SM, a warp issues
// every 5 to 6 cycles (dependent FP64 operations), so time is instructions;
// and the L1 beside the blocks' shared memory (see LevelTile).  FP64 build,
// 6x96^2x64: 2863 warp instructions per level and 32 columns against 4481
// with a division for every quotient, unconditional swaps and the back
// substitution in the same kernel; forward sweep 964 us and back
// substitution 246 us a solve against 1913.
//   io.w(i, out[5])  primitives of level i (is-1, is), unprojected
//   io.scr_level(lev)[e * io.scr_stride()]  factor e (0..29) of level lev = i - is
//   io.wptr(i, n), io.duptr(i, n)  addresses of w and of the explicit update
//                    du of level i, io.wstride(), io.dstride() from one
//                    variable to the next (LevelTile)
//   sa, ss           this lane's shared memory: entry e of two face matrices
//                    at sa[e * ss]
//   wt               the warp's level tile
template <class IO>
__device__ __forceinline__ void implicit_column(IO& io, typename IO::Real* sa, int ss,
                                                double cos_theta, double sin_theta, double d2,
                                                double d3, const double* x1f, const double* x1v,
                                                const double* dx1f, int is, int ie, double dt,
                                                double gamma, double grav,
                                                double* wt) {
  using R = typename IO::Real;
  using ColCell = exo::EXO_KNS::ColCell<R>;
  const double s = sin_theta;
  // gmm1 of every cell; the face average equals it
  const R gm1 = R((gamma - 1.) * 1. / 1.);
  const R gp = (gm1 + R(1)) / gm1;
  const R gam = R(gamma);
#if EXO_MIXED
  const R grv = R(grav);
#endif
  // the reference's Dt = 1/dt, the same value every time
  const R rdt = R(1. / dt);
  auto cell = [&](const double* w) {
    ColCell c;
    c.rho = R(w[IDN]);
    c.v1 = R(w[IVX]);
    c.v2 = R(w[IVY] + w[IVZ] * cos_theta);
    c.v3 = R(w[IVZ] * sin_theta);
    c.p = R(w[IPR]);
    c.s2 = c.v1 * c.v1 + c.v2 * c.v2 + c.v3 * c.v3;
#if EXO_MIXED
    if constexpr (sizeof(R) == 4) {
      c.isq = rsqrt_r(c.rho);
      c.sq = c.rho * c.isq;
      c.hr = gp * c.p * (c.isq * c.isq);
    } else {
      c.hr = gp * c.p * inv_r(c.rho);
    }
#else
    c.hr = gp * c.p / c.rho;
#endif
    return c;
  };
  LevelTile<IO, 5> lt(io, wt, is, ie - is + 1);
  double raw[5];
  io.w(is - 1, raw);
  ColCell cm = cell(raw);
  io.w(is, raw);
  ColCell c0 = cell(raw);
  auto AMs = [&](int slot, int r, int q) -> R& { return sa[(slot * 25 + r * 5 + q) * ss]; };
#if EXO_MIXED
  auto face_jacobian = [&](const ColCell& lo, const ColCell& hi, R (&A)[5][5]) {
    abs_jacobian(lo, hi, gm1, gam, A);
  };
#else
  const GasDiv gd{SharedDiv(gm1), SharedDiv(gm1 + 1.)};
  const SharedDiv by_dt(dt);
  auto face_jacobian = [&](const ColCell& lo, const ColCell& hi, R (&A)[5][5]) {
    abs_jacobian(lo, hi, gm1, gam, gd, A);
  };
#endif
  {
    R A[5][5];
    face_jacobian(cm, c0, A);
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int q = 0; q < 5; ++q) AMs(0, r, q) = A[r][q];
  }
  R Ap[5][5];  // (A c)_{i-1}
  R dp[5];  // delta_{i-1}
  int cur = 0;
  for (int i = is; i <= ie; ++i) {
    lt.ready(io, i - is);
    double rhs[5];
#pragma unroll
    for (int n = 0; n < 5; ++n) {
      raw[n] = lt.get(n, i - is);
      rhs[n] = lt.get(5 + n, i - is);
    }
    ColCell cp = cell(raw);
    const int nxt = cur ^ 1;
    {
      R A[5][5];
      face_jacobian(c0, cp, A);
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int q = 0; q < 5; ++q) AMs(nxt, r, q) = A[r][q];
    }
    const double aleft = d2 * d3 * x1f[i] * x1f[i] * s;
    const double aright = d2 * d3 * x1f[i + 1] * x1f[i + 1] * s;
    const double vol = dx1f[i] * d2 * d3 * x1v[i] * x1v[i] * s;
#if EXO_MIXED
    const double i2v = 0.5 / vol;
    const R bl = R(aleft * i2v), cr = R(aright * i2v), dd = R((aright - aleft) * i2v);
#else
    const SharedDiv by_2vol(2. * vol);
#endif
    const bool first = (i == is), last = (i == ie);
    R x[5];
    // rows of a, b (and c at the top boundary), then of t = a - b (A c)_{i-1},
    // written over row r of |A|(i-1/2) once that row has been read; and x
    unroll<5>([&](auto Row) {
      constexpr int r = decltype(Row)::value;
      R brow[5], trow[5];
      unroll<5>([&](auto Q) {
        constexpr int q = decltype(Q)::value;
        const R am = AMs(cur, r, q), ap = AMs(nxt, r, q);
#if EXO_MIXED
        R a = am * bl + ap * cr;
        if constexpr (fj_nz(r, q)) a += dd * fj_entry<r, q>(c0, gm1);
        if constexpr (r == q) a += rdt;
        if constexpr ((r == IVX && q == IDN) || (r == IEN && q == IVX)) a -= grv;
        R bm = am;
        if constexpr (fj_nz(r, q)) bm += fj_entry<r, q>(cm, gm1);
        R b = -bm * bl;
        if (first) a += (q == IVX) ? -b : b;
        if (last) {
          R cmv = ap;
          if constexpr (fj_nz(r, q)) cmv -= fj_entry<r, q>(cp, gm1);
          R c = -cmv * cr;
          a += (q == IVX) ? -c : c;
        }
#else
        double num = am * aleft + ap * aright;
        if constexpr (fj_nz(r, q)) num = num + (aright - aleft) * fj_entry<r, q>(c0, gm1);
        double a = by_2vol.finite(num);
        if constexpr (r == q) a = a + rdt;
        if constexpr ((r == IVX && q == IDN) || (r == IEN && q == IVX)) a = a - grav;
        double bm = am;
        if constexpr (fj_nz(r, q)) bm = am + fj_entry<r, q>(cm, gm1);
        double b = by_2vol.finite(-bm * aleft);
        if (first) a = a + ((q == IVX) ? -b : b);
        if (last) {
          double cmv = ap;
          if constexpr (fj_nz(r, q)) cmv = ap - fj_entry<r, q>(cp, gm1);
          double c = by_2vol.finite(-cmv * aright);
          a = a + ((q == IVX) ? -c : c);
        }
#endif
        brow[q] = b;
        trow[q] = a;
      });
#if EXO_MIXED
      x[r] = R(rhs[r]) * rdt;
#else
      x[r] = by_dt(rhs[r]);
#endif
      if (!first) {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          R ba = brow[0] * Ap[0][q];
#pragma unroll
          for (int k = 1; k < 5; ++k) ba += brow[k] * Ap[k][q];
          trow[q] = trow[q] - ba;
        }
        R bd = brow[0] * dp[0];
#pragma unroll
        for (int k = 1; k < 5; ++k) bd += brow[k] * dp[k];
        x[r] = x[r] - bd;
      }
#pragma unroll
      for (int q = 0; q < 5; ++q) AMs(cur, r, q) = trow[q];
    });
    R t[5][5];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int q = 0; q < 5; ++q) t[r][q] = AMs(cur, r, q);
    // c_i column by column, from |A|(i+1/2) in shared memory and the upper cell
    auto ccol = [&](auto Q, R* c) {
      constexpr int q = decltype(Q)::value;
      unroll<5>([&](auto Row) {
        constexpr int r = decltype(Row)::value;
        R cmv = AMs(nxt, r, q);
#if EXO_MIXED
        if constexpr (fj_nz(r, q)) cmv -= fj_entry<r, q>(cp, gm1);
        c[r] = -cmv * cr;
#else
        if constexpr (fj_nz(r, q)) cmv = cmv - fj_entry<r, q>(cp, gm1);
        c[r] = by_2vol.finite(-cmv * aright);
#endif
      });
    };
#if EXO_MIXED
    // LU with the rows taken in the order 1, 4, 2, 3, 0 -- the order partial
    // pivoting ends with for nearly every block of this solve (density last,
    // energy and x1 momentum first) -- and threshold partial pivoting on top:
    // a row swap only where the diagonal falls below a tenth of the largest
    // entry of its column.  The search and the swaps stand behind a vote, so
    // they are skipped almost always.
    constexpr int O[5] = {1, 4, 2, 3, 0};
    unsigned perm = 0;  // 3 bits per step: the position swapped in
    bool swapped = false;
    R idg[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      if (k < 4) {
        const R dk = abs_r(t[O[k]][k]);
        R best = dk;
#pragma unroll
        for (int r = k + 1; r < 5; ++r) best = fmax(best, abs_r(t[O[r]][k]));
        const bool small = dk < R(0.1) * best;
        int piv = k;
        if (__any_sync(0xffffffffu, small)) {
          if (small) {
            best = dk;
#pragma unroll
            for (int r = k + 1; r < 5; ++r) {
              const R m = abs_r(t[O[r]][k]);
              if (m > best) { best = m; piv = r; }
            }
          }
          swapped = true;
#pragma unroll
          for (int r = k + 1; r < 5; ++r) {
            const bool sw = (piv == r);
#pragma unroll
            for (int q = 0; q < 5; ++q) {
              const R a = t[O[k]][q], b = t[O[r]][q];
              t[O[k]][q] = sw ? b : a;
              t[O[r]][q] = sw ? a : b;
            }
          }
        }
        perm |= (unsigned)piv << (3 * k);
      }
      idg[k] = inv_r(t[O[k]][k]);
#pragma unroll
      for (int r = k + 1; r < 5; ++r) {
        const R l = t[O[r]][k] * idg[k];
        t[O[r]][k] = l;
#pragma unroll
        for (int q = k + 1; q < 5; ++q) t[O[r]][q] -= l * t[O[k]][q];
      }
    }
    // the right-hand sides' rows follow the swaps
    auto solve = [&](R* y) {
      if (swapped) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned pk = (perm >> (3 * k)) & 7u;
#pragma unroll
          for (int r = k + 1; r < 5; ++r) {
            const bool sw = (pk == (unsigned)r);
            const R a = y[O[k]], b = y[O[r]];
            y[O[k]] = sw ? b : a;
            y[O[r]] = sw ? a : b;
          }
        }
      }
      lu_solve_rows(t, idg, y);
    };
    solve(x);
    if (!last) {
      unroll<5>([&](auto Q) {
        constexpr int q = decltype(Q)::value;
        R c[5];
        ccol(Q, c);
        solve(c);
#pragma unroll
        for (int r = 0; r < 5; ++r) Ap[r][q] = c[r];
      });
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) dp[r] = x[r];
#else
    // Gauss-Jordan with partial pivoting on [t | I]; columns of t left of the
    // pivot are never read again and are not updated
    double B[5][5];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int q = 0; q < 5; ++q) B[r][q] = (r == q) ? 1. : 0.;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      int piv = k;
      double best = fabs(t[k][k]);
#pragma unroll
      for (int r = k + 1; r < 5; ++r)
        if (fabs(t[r][k]) > best) { best = fabs(t[r][k]); piv = r; }
#pragma unroll
      for (int r = k + 1; r < 5; ++r) {
        bool sw = (piv == r);
        if (!__any_sync(0xffffffffu, sw)) continue;  // most rows are no lane's pivot
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          if (q >= k) {
            double a = t[k][q], b = t[r][q];
            t[k][q] = sw ? b : a;
            t[r][q] = sw ? a : b;
          }
          double a = B[k][q], b = B[r][q];
          B[k][q] = sw ? b : a;
          B[r][q] = sw ? a : b;
        }
      }
      double d = 1.0 / t[k][k];
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        if (q > k) t[k][q] *= d;
        B[k][q] *= d;
      }
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        if (r == k) continue;
        double f = t[r][k];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          if (q > k) t[r][q] -= f * t[k][q];
          B[r][q] -= f * B[k][q];
        }
      }
    }
    // delta_i = B x, (A c)_i = B c_i
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      double acc = B[r][0] * x[0];
#pragma unroll
      for (int k = 1; k < 5; ++k) acc += B[r][k] * x[k];
      dp[r] = acc;
    }
    unroll<5>([&](auto Q) {
      constexpr int q = decltype(Q)::value;
      double c[5];
      ccol(Q, c);
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        double acc = B[r][0] * c[0];
#pragma unroll
        for (int k = 1; k < 5; ++k) acc += B[r][k] * c[k];
        Ap[r][q] = acc;
      }
    });
#endif
    R* const scl = io.scr_level(i - is);
    const size_t scs = io.scr_stride();
    if (!last) {
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int q = 0; q < 5; ++q) scl[(r * 5 + q) * scs] = Ap[r][q];
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) scl[(25 + r) * scs] = dp[r];
    cm = c0;
    c0 = cp;
    cur = nxt;
  }
}

// ImplicitSolver::PartialCorrection (partial_correction.cpp:26-173) of one
// radial column, one thread per column: the 3x3 block-tridiagonal system of
// (rho, m1, E) -- the rows and columns IDN, IVX, IEN of FullCorrection's
// matrices, the same face and cell Jacobians -- solved by ForwardSweep /
// BackwardSubstitution with 3-row blocks (forward_backward.hpp:15-126).  The
// tangential momenta keep their explicit update; the reference's flux
// correction corr is zero (its computation is commented out there).  Each
// 3x3 block is inverted as its adjugate over its determinant, the closed form
// a fixed-size 3x3 inverse takes.  Scratch per level: (A c)_i (9) and
// delta_i (3).  IO and arguments as for implicit_column.  A solve at
// 6x62^2x45 (mixed build) went from 173 to 126 us, at 6x40^3 (FP64 build) from
// 213 to 100 us.
template <class IO>
__device__ __forceinline__ void implicit_column_partial(IO& io, typename IO::Real* sa, int ss,
                                                        double cos_theta, double sin_theta,
                                                        double d2, double d3, const double* x1f,
                                                        const double* x1v, const double* dx1f,
                                                        int is, int ie, double dt, double gamma,
                                                        double grav, double* wt) {
  using R = typename IO::Real;
  using ColCell = exo::EXO_KNS::ColCell<R>;
  constexpr int P[3] = {IDN, IVX, IEN};
  const double s = sin_theta;
  const R gm1 = R((gamma - 1.) * 1. / 1.);
  const R gp = (gm1 + R(1)) / gm1;
  const R gam = R(gamma);
#if EXO_MIXED
  const R grv = R(grav);
#endif
  const R rdt = R(1. / dt);
  auto cell = [&](const double* w) {
    ColCell c;
    c.rho = R(w[IDN]);
    c.v1 = R(w[IVX]);
    c.v2 = R(w[IVY] + w[IVZ] * cos_theta);
    c.v3 = R(w[IVZ] * sin_theta);
    c.p = R(w[IPR]);
    c.s2 = c.v1 * c.v1 + c.v2 * c.v2 + c.v3 * c.v3;
#if EXO_MIXED
    if constexpr (sizeof(R) == 4) {
      c.isq = rsqrt_r(c.rho);
      c.sq = c.rho * c.isq;
      c.hr = gp * c.p * (c.isq * c.isq);
    } else {
      c.hr = gp * c.p * inv_r(c.rho);
    }
#else
    c.hr = gp * c.p / c.rho;
#endif
    return c;
  };
  LevelTile<IO, 3> lt(io, wt, is, ie - is + 1);
  double raw[5];
  io.w(is - 1, raw);
  ColCell cm = cell(raw);
  io.w(is, raw);
  ColCell c0 = cell(raw);
  auto AMs = [&](int slot, int r, int q) -> R& { return sa[(slot * 9 + r * 3 + q) * ss]; };
#if !EXO_MIXED
  const GasDiv gd{SharedDiv(gm1), SharedDiv(gm1 + 1.)};
  const SharedDiv by_dt(dt);
#endif
  auto face = [&](const ColCell& lo, const ColCell& hi, int slot) {
    R A[5][5];
#if EXO_MIXED
    abs_jacobian(lo, hi, gm1, gam, A);
#else
    abs_jacobian(lo, hi, gm1, gam, gd, A);
#endif
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int q = 0; q < 3; ++q) AMs(slot, r, q) = A[P[r]][P[q]];
  };
  face(cm, c0, 0);
  R Ap[3][3];  // (A c)_{i-1}
  R dp[3];     // delta_{i-1}
  int cur = 0;
  for (int i = is; i <= ie; ++i) {
    lt.ready(io, i - is);
    double rhs[3];
#pragma unroll
    for (int n = 0; n < 5; ++n) raw[n] = lt.get(n, i - is);
#pragma unroll
    for (int m = 0; m < 3; ++m) rhs[m] = lt.get(5 + m, i - is);
    ColCell cp = cell(raw);
    const int nxt = cur ^ 1;
    face(c0, cp, nxt);
    const double aleft = d2 * d3 * x1f[i] * x1f[i] * s;
    const double aright = d2 * d3 * x1f[i + 1] * x1f[i + 1] * s;
    const double vol = dx1f[i] * d2 * d3 * x1v[i] * x1v[i] * s;
#if EXO_MIXED
    const double i2v = 0.5 / vol;
    const R bl = R(aleft * i2v), cr = R(aright * i2v), dd = R((aright - aleft) * i2v);
#else
    const SharedDiv by_2vol(2. * vol);
#endif
    const bool first = (i == is), last = (i == ie);
    R t[3][3], cc[3][3], x[3];
    unroll<3>([&](auto Row) {
      constexpr int r = decltype(Row)::value;
      constexpr int pr = P[r];
      R brow[3];
      unroll<3>([&](auto Q) {
        constexpr int q = decltype(Q)::value;
        constexpr int pq = P[q];
        const R am = AMs(cur, r, q), ap = AMs(nxt, r, q);
        // Phi << 0,0,0, grav,0,0, 0,grav,0 and Bnd = diag(1,-1,1)
        constexpr bool phi = (r == 1 && q == 0) || (r == 2 && q == 1);
#if EXO_MIXED
        R a = am * bl + ap * cr;
        if constexpr (fj_nz(pr, pq)) a += dd * fj_entry<pr, pq>(c0, gm1);
        if constexpr (r == q) a += rdt;
        if constexpr (phi) a -= grv;
        R bm = am;
        if constexpr (fj_nz(pr, pq)) bm += fj_entry<pr, pq>(cm, gm1);
        R b = -bm * bl;
        R cmv = ap;
        if constexpr (fj_nz(pr, pq)) cmv -= fj_entry<pr, pq>(cp, gm1);
        R c = -cmv * cr;
        if (first) a += (q == 1) ? -b : b;
        if (last) a += (q == 1) ? -c : c;
#else
        double num = am * aleft + ap * aright;
        if constexpr (fj_nz(pr, pq)) num = num + (aright - aleft) * fj_entry<pr, pq>(c0, gm1);
        double a = by_2vol.finite(num);
        if constexpr (r == q) a = a + rdt;
        if constexpr (phi) a = a - grav;
        double bm = am;
        if constexpr (fj_nz(pr, pq)) bm = am + fj_entry<pr, pq>(cm, gm1);
        double b = by_2vol.finite(-bm * aleft);
        double cmv = ap;
        if constexpr (fj_nz(pr, pq)) cmv = ap - fj_entry<pr, pq>(cp, gm1);
        double c = by_2vol.finite(-cmv * aright);
        if (first) a = a + ((q == 1) ? -b : b);
        if (last) a = a + ((q == 1) ? -c : c);
#endif
        brow[q] = b;
        t[r][q] = a;
        cc[r][q] = c;
      });
#if EXO_MIXED
      x[r] = R(rhs[r]) * rdt;
#else
      x[r] = by_dt(rhs[r]);
#endif
      if (!first) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          R ba = brow[0] * Ap[0][q];
#pragma unroll
          for (int k = 1; k < 3; ++k) ba += brow[k] * Ap[k][q];
          t[r][q] = t[r][q] - ba;
        }
        R bd = brow[0] * dp[0];
#pragma unroll
        for (int k = 1; k < 3; ++k) bd += brow[k] * dp[k];
        x[r] = x[r] - bd;
      }
    });
    // B = t^-1 = adj(t) / det(t): cofactor (i,j) from the cyclic neighbours
    // of row i and column j (which carries its sign), det along column 0
    auto cof = [&](int i0, int j0) {
      const int i1 = (i0 + 1) % 3, i2 = (i0 + 2) % 3, j1 = (j0 + 1) % 3, j2 = (j0 + 2) % 3;
      return t[i1][j1] * t[i2][j2] - t[i1][j2] * t[i2][j1];
    };
    R B[3][3];
    {
      const R c00 = cof(0, 0), c10 = cof(1, 0), c20 = cof(2, 0);
      const R det = c00 * t[0][0] + c10 * t[1][0] + c20 * t[2][0];
      const R id = R(1) / det;
      B[0][0] = c00 * id;
      B[0][1] = c10 * id;
      B[0][2] = c20 * id;
#pragma unroll
      for (int r = 1; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) B[r][q] = cof(q, r) * id;
    }
    // delta_i = B x, (A c)_i = B c_i
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      R acc = B[r][0] * x[0];
#pragma unroll
      for (int k = 1; k < 3; ++k) acc += B[r][k] * x[k];
      dp[r] = acc;
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        R acc = B[r][0] * cc[0][q];
#pragma unroll
        for (int k = 1; k < 3; ++k) acc += B[r][k] * cc[k][q];
        Ap[r][q] = acc;
      }
    R* const scl = io.scr_level(i - is);
    const size_t scs = io.scr_stride();
    if (!last) {
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) scl[(r * 3 + q) * scs] = Ap[r][q];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) scl[(9 + r) * scs] = dp[r];
    cm = c0;
    c0 = cp;
    cur = nxt;
  }
}

// UpdateAllConserved on the last stage with NVAPOR = NCLOUD = 0: the
// AirParcel round trip MassConc -> MoleFrac -> MassConc of one cell
// (impl.cpp:138-304, air_parcel.cpp:190-278)
__device__ __forceinline__ void airparcel_round_trip(double* uu, double Rd, double gammad) {
  const double Rgas = 8.314462;  // src/constants.hpp:5
  double mu0 = Rgas / Rd;
  double inv_mu0 = 1. / (mu0 * 1.);
  double cv0 = 1. * (Rd / (gammad - 1.));
  double w[5];
#pragma unroll
  for (int n = 0; n < 5; ++n) w[n] = uu[n];
  double rho = 0., cvt = 0.;
  rho += w[0];
  cvt += w[0] * cv0;
  double KE = 0.5 / rho * (sqr(w[IVX]) + sqr(w[IVY]) + sqr(w[IVZ]));
  double tem = (w[IEN] - KE) / cvt;
  w[IEN] = cvt * tem;
  {
    double r2 = 0., cv = 0., rhoR = 0.;
    r2 += w[0];
    cv += w[0] * cv0;
    rhoR += w[0] * Rgas * inv_mu0;
    double di = 1. / r2;
    w[IDN] = w[IEN] / cv;
    w[IPR] = rhoR * w[IDN];
    w[IVX] *= di; w[IVY] *= di; w[IVZ] *= di;
  }
  {
    double tt = w[IDN], sum = 1., gg = 1.;
    double r2 = w[IPR] * sum / (Rd * tt * gg);
    w[IDN] = r2;
    w[IEN] = 0.;
    w[IEN] += w[IDN] * cv0 * tt;
    w[IVX] *= r2; w[IVY] *= r2; w[IVZ] *= r2;
  }
  double r2 = 0.;
  r2 += w[0];
  double vx = w[IVX] / r2, vy = w[IVY] / r2, vz = w[IVZ] / r2;
  double e = w[IEN] + 0.5 * w[0] * (sqr(vx) + sqr(vy) + sqr(vz));
#pragma unroll
  for (int n = 0; n < 4; ++n) uu[n] = w[n];
  uu[IEN] = e;
}

// Launch shape of the forward sweep: one thread per radial column, 64
// columns per block.
constexpr int IMPL_THREADS = 64;      // default; 32 and 128 are the other tiles
constexpr int IMPL_MAX_THREADS = 128;
// Two 128-thread blocks per SM: the full register file.  A smaller budget
// spills, and a spill goes past the little L1 that the shared memory leaves
// (FP64 build at 6x96^2x64 capped at 204: 2247 instead of 1905 us).
#define EXO_IMPL_BOUNDS __launch_bounds__(IMPL_MAX_THREADS, 2)
// per block: the warps' shared memory, then x1f (nc1+1), x1v (nc1), dx1f (nc1)
template <class R, bool full>
__host__ __device__ constexpr size_t impl_smem(int threads, int nc1) {
  return ((size_t)impl_warp_doubles<R, full>() * (threads / 32) + 3 * (size_t)(nc1 + 1)) *
         sizeof(double);
}
// this lane's shared memory (arguments sa, ss, wt of implicit_column and
// implicit_column_partial)
template <class R>
struct ImplSlices {
  R* sa;
  int ss;
  double* wt;  // the warp's tiles
};
template <class R, bool full>
__device__ __forceinline__ ImplSlices<R> impl_slices(double* ism) {
  double* w = ism + (threadIdx.x >> 5) * impl_warp_doubles<R, full>();
  return {reinterpret_cast<R*>(w + LEVEL_TILE_DOUBLES) + (threadIdx.x & 31), 32, w};
}
// where the block's copy of the radial geometry starts
template <class R, bool full>
__device__ __forceinline__ double* impl_radial(double* ism) {
  return ism + (blockDim.x >> 5) * impl_warp_doubles<R, full>();
}
// the largest dynamic shared memory a launch may ask for
// (a step's 128 columns of 250 levels take 96 KB, the column hooks up to this)
constexpr int IMPL_SMEM_MAX = 160 * 1024;

// copies the radial geometry of the member into shared memory (all threads
// of the block take part; returns the shared copies)
__device__ __forceinline__ void stage_radial(double* sg, int nc1, const double* x1f,
                                             const double* x1v, const double* dx1f,
                                             const double*& sx1f, const double*& sx1v,
                                             const double*& sdx1f) {
  double* a = sg;
  double* b = sg + nc1 + 1;
  double* c = b + nc1 + 1;
  for (int t = threadIdx.x; t <= nc1; t += blockDim.x) {
    a[t] = x1f[t];
    if (t < nc1) {
      b[t] = x1v[t];
      c[t] = dx1f[t];
    }
  }
  __syncthreads();
  sx1f = a;
  sx1v = b;
  sdx1f = c;
}

// A column of the stepping context: primitives and update from the state
// arrays, factors in the member's scratch.
template <class R>
struct StepColumnIO {
  using Real = R;
  const double* wc;
  const double* duc;
  size_t vs;  // stride between variables
  R* scr0;    // scratch of this column: [level][entry][32 lanes] per warp of columns
  __device__ __forceinline__ void w(int i, double* out) const {
#pragma unroll
    for (int n = 0; n < 5; ++n) out[n] = wc[n * vs + i];
  }
  __device__ __forceinline__ size_t wstride() const { return vs; }
  __device__ __forceinline__ size_t dstride() const { return vs; }
  __device__ __forceinline__ const double* wptr(int i, int n) const { return wc + n * vs + i; }
  __device__ __forceinline__ const double* duptr(int i, int n) const { return duc + n * vs + i; }
  // the factors of a level: entry e at scr_level(lev)[e * 32]
  __device__ __forceinline__ R* scr_level(int lev) const { return scr0 + (size_t)lev * (30 * 32); }
  __device__ __forceinline__ size_t scr_stride() const { return 32; }
};

// The forward sweep of one radial column of the stepping context.
// stage 0..2: a stage of the step (dt = beta_stage * the CFL step);
// stage -1: ImplicitSolver::SolveImplicit3D alone (dt given)
template <class R, bool full>
__device__ __forceinline__ void implicit_block(const DevView& v, unsigned blk, int stage,
                                               double dt_given = 0.) {
  extern __shared__ double ism[];
  const int ncol = 6 * v.N * v.N;
  const int col = (int)(blk * blockDim.x + threadIdx.x);
  // the radial geometry, read every level by every column, staged once per
  // block: kept out of L1, which the columns' strided loads churn each level
  const double* x1f;
  const double* x1v;
  const double* dx1f;
  stage_radial(impl_radial<R, full>(ism), v.nc1, v.x1f, v.x1v, v.dx1f, x1f, x1v, dx1f);
  if ((col & ~31) >= ncol) return;
  // lanes past the last column repeat it: same values to the same places
  // (their own scratch; it holds whole groups of 32 columns)
  const int cc = min(col, ncol - 1);
  const int j = v.js + cc % v.N;
  const int k = v.ks + (cc / v.N) % v.N;
  const int p = cc / (v.N * v.N);
  const double dt = stage < 0 ? dt_given : rk_beta(stage) * v.sc->dt;
  const size_t base = idx(v, p, 0, k, j, 0);
  // scratch in blocks of 32 columns: a warp's 32 entries are 128 (FP32) or
  // 256 (FP64) contiguous bytes
  R* scr0 = reinterpret_cast<R*>(v.scratch) + (size_t)(col >> 5) * v.L * 30 * 32 + (col & 31);
  StepColumnIO<R> io{v.w + base, v.du + base, v.cells, scr0};
  const ImplSlices<R> sl = impl_slices<R, full>(ism);
  if constexpr (full)
    implicit_column(io, sl.sa, sl.ss, geo(v, GCOSC, p, k, j), geo(v, GSINC, p, k, j),
                    geo(v, GDX2A, p, k, j), geo(v, GDX3A, p, k, j), x1f, x1v, dx1f, v.is, v.ie,
                    dt, v.gamma, v.grav, sl.wt);
  else
    implicit_column_partial(io, sl.sa, sl.ss, geo(v, GCOSC, p, k, j), geo(v, GSINC, p, k, j),
                            geo(v, GDX2A, p, k, j), geo(v, GDX3A, p, k, j), x1f, x1v, dx1f, v.is,
                            v.ie, dt, v.gamma, v.grav, sl.wt);
}

#if EXO_MIXED
#include "exo_implicit_fused.cuh"
#endif

// ---------------------------------------------------- kb_implicit_bwd ---
// The back substitution, delta_i -= (A c)_i delta_{i+1} from the top level
// down, u += delta (with the AirParcel round trip on the last stage), as a
// kernel of its own after the forward sweep, which leaves (A c)_i and
// delta_i of every level in scratch.  It streams 240 bytes of factors (FP64,
// 5x5) and 80 bytes of u per cell and computes little, so it is built to
// keep HBM busy: in the forward kernel, whose registers and shared memory
// leave eight warps per SM, it took 1.6 of 3.95 ms per 6x192^2x96 launch
// (FP64 factors); FP32 blocks at 6x126^2x70 went from 1255 to 1170 us a solve.
// A block of three warps takes 32 columns.  The solver warp runs the
// recursion, one column per lane, on factors that arrive level by level in a
// ring of FRING levels: one bulk copy a level (32 columns' factors of a
// level are contiguous), counted on an mbarrier, its wait bounded.  It
// leaves the corrections of CL levels at a time in shared memory; the other
// two warps add them to u meanwhile, a column's CL levels side by side.
template <class R, int NB>
struct BwdLayout {
  static constexpr int NM = NB * NB, NFAC = NM + NB;
  static constexpr int FRING = 4, CL = 4, DS = CL + 1;
  static constexpr size_t level_bytes = (size_t)NFAC * 32 * sizeof(R);
  static constexpr size_t fac_bytes = FRING * level_bytes;
  static constexpr size_t del_bytes = (size_t)2 * NB * 32 * DS * sizeof(double);
  static constexpr size_t bytes = fac_bytes + del_bytes;
  static_assert(level_bytes % 16 == 0 && NM * 32 * sizeof(R) % 16 == 0,
                "bulk copies start on and move multiples of 16 bytes");
};
constexpr int BWD_THREADS = 96;

template <class R>
struct BwdGroup {
  const R* scr;          // factor e of level l of column c: scr[l lstride + e estride + c]
  size_t lstride, estride;
  double* x;             // u (stage >= 0) or du (stage < 0): x[off[c] + n vs + l]
  size_t vs;
  const long long* off;  // shared memory, 32 entries
  int ncols, L, stage;
  double Rd, gamma;
  int* timeout;          // sticky flag of a wait that gave up
};

// kBulk: the factors of 32 columns of a level are contiguous and 16-byte
// aligned (the stepping scratch); otherwise each lane copies its own
template <class R, int NB, bool kBulk>
__device__ __forceinline__ void implicit_bwd_group(const BwdGroup<R>& g, unsigned char* sm) {
  using LY = BwdLayout<R, NB>;
  constexpr int NM = LY::NM, NFAC = LY::NFAC, FRING = LY::FRING, CL = LY::CL, DS = LY::DS;
  static_assert((FRING & (FRING - 1)) == 0, "ring slots by mask");
  __shared__ unsigned long long full[FRING];
  __shared__ int s_stop;  // the first chunk a wait that gave up left unfinished
  R* const ring = reinterpret_cast<R*>(sm);
  double* const del = reinterpret_cast<double*>(sm + LY::fac_bytes);
  const int lane = (int)(threadIdx.x & 31), L = g.L;
  const int nch = (L + CL - 1) / CL;
  auto var = [](int m) { return NB == 5 ? m : (m == 2 ? (int)IEN : m); };
  if (threadIdx.x < 32) {
    // the j-th level from the top, into slot j; of the top level only delta,
    // its (A c) being neither formed nor read
    auto issue = [&](int j) {
      const int l = L - 1 - j, e0 = j == 0 ? NM : 0;
      R* dst = ring + (j & (FRING - 1)) * NFAC * 32;
      if constexpr (kBulk) {
        if (l >= 0 && lane == 0) {
          const unsigned bytes = (unsigned)((NFAC - e0) * 32 * sizeof(R));
          mbar_expect_tx(&full[j & (FRING - 1)], bytes);
          bulk_g2s(dst + e0 * 32, g.scr + (size_t)l * g.lstride + e0 * 32, bytes,
                   &full[j & (FRING - 1)]);
        }
      } else {
        if (l >= 0 && lane < g.ncols) {
          const R* src = g.scr + (size_t)l * g.lstride + lane;
#pragma unroll
          for (int e = 0; e < NFAC; ++e)
            if (e >= e0) cp_async_r(dst + e * 32 + lane, src + e * g.estride);
        }
        cp_async_commit();
      }
    };
    if constexpr (kBulk) {
      if (lane == 0) {
#pragma unroll
        for (int s = 0; s < FRING; ++s) mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
      }
      __syncwarp();
    }
#pragma unroll 1
    for (int j = 0; j < FRING; ++j) issue(j);
    if (lane == 0) s_stop = nch;
    bool ok = true;
    R dp[NB];
#pragma unroll
    for (int r = 0; r < NB; ++r) dp[r] = R(0);
#pragma unroll 1
    for (int c = 0; c <= nch; ++c) {
      const int hi = L - 1 - c * CL, lo = max(0, hi - CL + 1);
      double* const d = del + (c & 1) * NB * 32 * DS + lane * DS;
      if (c < nch && ok) {
#pragma unroll 1
        for (int l = hi; l >= lo; --l) {
          const int j = L - 1 - l;
          if constexpr (kBulk) {
            ok = __all_sync(0xffffffffu, mbar_wait(&full[j & (FRING - 1)], (j / FRING) & 1));
            if (!ok) break;
          } else {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(FRING - 1) : "memory");
            __syncwarp();
          }
          const R* f = ring + (j & (FRING - 1)) * NFAC * 32 + lane;
          // delta of the top level is its own
          R dl[NB];
#pragma unroll
          for (int r = 0; r < NB; ++r) {
            dl[r] = f[(NM + r) * 32];
            if (j > 0) {
              R ad = f[(r * NB) * 32] * dp[0];
#pragma unroll
              for (int k = 1; k < NB; ++k) ad += f[(r * NB + k) * 32] * dp[k];
              dl[r] = dl[r] - ad;
            }
          }
#pragma unroll
          for (int r = 0; r < NB; ++r) {
            dp[r] = dl[r];
            d[r * 32 * DS + (l - lo)] = (double)dl[r];
          }
          __syncwarp();
          issue(j + FRING);
        }
        if (!ok && lane == 0) s_stop = c;
      }
      __syncthreads();
    }
    if (!ok) {
      // a bulk copy did not complete in time: record it, and give every copy
      // still outstanding a bounded wait before the shared memory is released
      if (lane == 0) atomicOr(g.timeout, 1);
      for (int s = 0; s < FRING; ++s) {
        mbar_wait(&full[s], 0);
        mbar_wait(&full[s], 1);
      }
    }
    if constexpr (!kBulk) cp_async_wait_all();
  } else {
    // cells (column, level) of a chunk: two per thread
    const int t0 = (int)threadIdx.x - 32;
    auto place = [&](int c, int m, int& col, int& l) {
      const int t = t0 + 64 * m, hi = L - 1 - c * CL, lo = max(0, hi - CL + 1);
      col = t / CL;
      l = lo + t % CL;
      return col < g.ncols && l <= hi;
    };
    // the 3x3 correction leaves m2 and m3 to the update kernel; the last
    // stage's round trip takes every variable
    const bool all = g.stage == 2;
    auto moved = [&](int n) { return NB == 5 || all || (n != IVY && n != IVZ); };
    auto load = [&](int c, int m, double* u) {
      int col, l;
      if (g.stage < 0 || !place(c, m, col, l)) return;
      const double* p = g.x + g.off[col] + l;
#pragma unroll
      for (int n = 0; n < 5; ++n)
        if (moved(n)) u[n] = p[n * g.vs];
    };
    double cur0[5] = {}, cur1[5] = {}, nxt0[5] = {}, nxt1[5] = {};
#pragma unroll 1
    for (int c = 0; c <= nch; ++c) {
      if (c < nch) {
        load(c, 0, nxt0);
        load(c, 1, nxt1);
      }
      if (c > 0) {
        const double* d = del + ((c - 1) & 1) * NB * 32 * DS;
        const int lo = max(0, L - (c - 1) * CL - CL);
        // not unrolled: one copy of the round trip's code
#pragma unroll 1
        for (int m = 0; m < 2; ++m) {
          int col, l;
          if (!place(c - 1, m, col, l) || c - 1 >= s_stop) continue;
          double* p = g.x + g.off[col] + l;
          double dv[5];
#pragma unroll
          for (int r = 0; r < NB; ++r) dv[var(r)] = d[(r * 32 + col) * DS + (l - lo)];
          if (g.stage < 0) {
#pragma unroll
            for (int r = 0; r < NB; ++r) p[var(r) * g.vs] = dv[var(r)];
          } else {
            double uu[5];
#pragma unroll
            for (int n = 0; n < 5; ++n) {
              uu[n] = m ? cur1[n] : cur0[n];
              if (NB == 5 || (n != IVY && n != IVZ)) uu[n] = uu[n] + 1. * dv[n];
            }
            if (all) airparcel_round_trip(uu, g.Rd, g.gamma);
#pragma unroll
            for (int n = 0; n < 5; ++n)
              if (moved(n)) p[n * g.vs] = uu[n];
          }
        }
      }
#pragma unroll
      for (int n = 0; n < 5; ++n) {
        cur0[n] = nxt0[n];
        cur1[n] = nxt1[n];
      }
      __syncthreads();
    }
  }
}

// Columns 32 group .. of a member: a stage of the step (stage 0..2, u), or
// SolveImplicit3D alone (stage < 0, du).  If a wait gave up, the columns keep
// the forward sweep's state below the last finished chunk.
template <class R, bool full>
__device__ __forceinline__ void implicit_bwd_block(const DevView& v, int group, int stage) {
  extern __shared__ __align__(128) unsigned char bws[];
  __shared__ long long s_off[32];
  const int ncol = 6 * v.N * v.N, col0 = group * 32;
  if (threadIdx.x < 32) {
    const int col = min(col0 + (int)threadIdx.x, ncol - 1);
    const int j = v.js + col % v.N;
    const int k = v.ks + (col / v.N) % v.N;
    const int p = col / (v.N * v.N);
    s_off[threadIdx.x] = (long long)idx(v, p, 0, k, j, v.is);
  }
  __syncthreads();
  BwdGroup<R> g;
  g.scr = reinterpret_cast<const R*>(v.scratch) + (size_t)group * v.L * 30 * 32;
  g.lstride = 30 * 32;
  g.estride = 32;
  g.x = stage < 0 ? v.du : v.u;
  g.vs = v.cells;
  g.off = s_off;
  g.ncols = min(32, ncol - col0);
  g.L = v.L;
  g.stage = stage;
  g.Rd = v.Rd;
  g.gamma = v.gamma;
  g.timeout = &v.sc->timeout;
  implicit_bwd_group<R, full ? 5 : 3, true>(g, bws);
}

// last-stage round trip when the implicit solver is off
__device__ __forceinline__ void roundtrip_block(const DevView& v, unsigned blk) {
  unsigned tid = blk * blockDim.x + threadIdx.x;
  unsigned L = v.L, N = v.N;
  if (tid >= 6u * N * N * L) return;
  const unsigned r1 = v.div_L(tid), r2 = v.div_N(r1), r3 = v.div_N(r2);
  int i = v.is + (int)(tid - r1 * L);
  int j = v.js + (int)(r1 - r2 * N);
  int k = v.ks + (int)(r2 - r3 * N);
  int p = (int)r3;
  double uu[5];
  for (int n = 0; n < 5; ++n) uu[n] = v.u[idx(v, p, n, k, j, i)];
  airparcel_round_trip(uu, v.Rd, v.gamma);
  for (int n = 0; n < 5; ++n) v.u[idx(v, p, n, k, j, i)] = uu[n];
}

__device__ __forceinline__ void p2c_block(const DevView& v, unsigned blk, const double* wsrc) {
  unsigned tid = blk * blockDim.x + threadIdx.x;
  unsigned L = v.L, N = v.N;
  if (tid >= 6u * N * N * L) return;
  const unsigned r1 = v.div_L(tid), r2 = v.div_N(r1), r3 = v.div_N(r2);
  int i = v.is + (int)(tid - r1 * L);
  int j = v.js + (int)(r1 - r2 * N);
  int k = v.ks + (int)(r2 - r3 * N);
  int p = (int)r3;
  double w[5], c[5];
  #pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= v.nv) break;
    w[n] = wsrc[idx(v, p, n, k, j, i)];
  }
  prim_to_cons(v, w, c, geo(v, GCOSC, p, k, j));
  #pragma unroll
  for (int n = 0; n < 5; ++n) {
    if (n >= v.nv) break;
    v.u[idx(v, p, n, k, j, i)] = c[n];
  }
}

__global__ void k_set_dt(DevScalars* sc, double dt) { sc->dt = dt; }

__global__ void k_dt_reset(DevScalars* sc) {
  sc->dtmin_bits = 0x7FEFFFFFFFFFFFFFull;  // DBL_MAX
}

// Mesh::NewTimeStep: dt = min(2 dt, cfl * min over cells); advance time
__global__ void k_dt_finalize(DevScalars* sc, double cfl, double dt_fixed, int advance,
                              int first) {
  if (advance) {
    sc->time += sc->dt;
    sc->ncycle += 1;
  }
  if (dt_fixed > 0.) {
    sc->dt = dt_fixed;
    return;
  }
  double nd = cfl * __longlong_as_double((long long)sc->dtmin_bits);
  sc->dt = first ? nd : fmin(2.0 * sc->dt, nd);
}

// ------------------------------------------------------------ wrappers ----
// Each kernel body above works on one atmosphere and one block index of it.
// The single-atmosphere kernels take the DevView by value; the batched ones
// take a table of DevViews and, per launch, the first block of every member
// (start[m], start[n] = total): block b belongs to the member m with
// start[m] <= b < start[m+1] and works on its block b - start[m].  One
// batched launch per kernel advances every member of an ensemble.
struct Batch {
  const DevView* views;
  const unsigned* start;
  int n;
};

__device__ __forceinline__ int batch_member(const Batch& bt, unsigned b) {
  int lo = 0, hi = bt.n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (bt.start[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// copies the member's view into shared memory, 16 bytes per thread; returns
// the block's index within the member
__device__ __forceinline__ unsigned batch_enter(const Batch& bt, DevView& sv) {
  static_assert(sizeof(DevView) % 16 == 0, "DevView is copied in 16-byte words");
  const int m = batch_member(bt, blockIdx.x);  // the same for every thread
  const int4* src = reinterpret_cast<const int4*>(bt.views + m);
  int4* dst = reinterpret_cast<int4*>(&sv);
  for (int t = threadIdx.x; t < (int)(sizeof(DevView) / 16); t += blockDim.x) dst[t] = src[t];
  const unsigned local = blockIdx.x - bt.start[m];
  __syncthreads();
  return local;
}

// 64 registers (32 warps per SM, 8 bytes of spill): 9 % faster at
// 6x192^2x96 than 48 (which spills 80 bytes), 56 and 74 (no spill)
#ifndef EXO_PRIM_MAXNREG
#define EXO_PRIM_MAXNREG 64
#endif
#ifdef EXO_PRIM_MAXNREG
#define EXO_PRIM_BOUNDS __maxnreg__(EXO_PRIM_MAXNREG)
#else
#define EXO_PRIM_BOUNDS
#endif
__global__ void EXO_PRIM_BOUNDS kb_prim_ghost(Batch bt, int compute_dt) {
  __shared__ __align__(16) DevView sv;
  unsigned b = batch_enter(bt, sv);
  prim_ghost_block(sv, b, compute_dt);
}

// 48 registers and 100 bytes of spill (mixed, 96^2x64: 261 us; 64 and 72
// registers, a block fewer on each SM: 310; 40 gains 3 % there and loses 10 %
// at 24^2x32)
#ifndef EXO_X1_MAXNREG
#define EXO_X1_MAXNREG 48
#endif
#define EXO_X1_BOUNDS __maxnreg__(EXO_X1_MAXNREG)
template <class T>
__global__ void EXO_X1_BOUNDS kb_flux_x1(Batch bt) {
  __shared__ __align__(16) DevView sv;
  unsigned b = batch_enter(bt, sv);
  if (sv.eqn == EXO_EQN_SHALLOW_YZ) return;
  flux_x1_block<T>(sv, b);
}

// the mixed build at 128 registers (4 blocks of 128 threads per SM): 1.64 ms
// per launch at 6x192^2x96 against 1.75 at its natural 148 (measured with
// addresses recomputed per row and face)
#if EXO_MIXED && !defined(EXO_X23_MINB)
#define EXO_X23_MINB 4
#endif
#if defined(EXO_X23_MINB)
#define EXO_X23_BOUNDS __launch_bounds__(X23_THREADS, EXO_X23_MINB)
#else
#define EXO_X23_BOUNDS __launch_bounds__(X23_THREADS)
#endif
template <class T>
__global__ void EXO_X23_BOUNDS kb_flux_x23(Batch bt) {
  __shared__ __align__(16) DevView sv;
  unsigned b = batch_enter(bt, sv);
  flux_x23_block<T>(sv, b);
}

// The update waits for its loads (mixed, 96^2x64: 61 % of the copy rate on the
// bytes it needs, 16 warps per SM).  FP64 at its natural 140 registers has 12:
// 303 us there, at 128 registers 276, at 96 and 80, with the inputs no longer
// all requested at once, 329 and 312 (mixed 246, 276 and 274).  Its quotients
// by the volume and the radius from one reciprocal each: 329 -> 303.
template <class T>
__global__ void __maxnreg__(128) kb_update(Batch bt, int stage) {
  __shared__ __align__(16) DevView sv;
  unsigned b = batch_enter(bt, sv);
  update_block<T>(sv, b, stage);
}

// One kernel per block size (full: 5x5, else 3x3), each over the blocks of
// every member; members of the other kind are skipped.
template <class R, bool full>
__global__ void EXO_IMPL_BOUNDS kb_implicit(Batch bt, int stage, double dt_given) {
  __shared__ __align__(16) DevView sv;
  unsigned b = batch_enter(bt, sv);
  if (sv.eqn == EXO_EQN_SHALLOW_YZ || !(sv.implicit_flag & 1)) return;
  if (((sv.implicit_flag & 8) != 0) != full) return;
  implicit_block<R, full>(sv, b, stage, dt_given);
}

#if EXO_MIXED
template <bool kTile>
__global__ void __maxnreg__(204) kb_implicit_fused(Batch bt, int stage, double dt_given) {
  __shared__ __align__(16) DevView sv;
  unsigned b = batch_enter(bt, sv);
  if (sv.eqn == EXO_EQN_SHALLOW_YZ || !(sv.implicit_flag & 1)) return;
  if (!(sv.implicit_flag & 8)) return;
  implicit_fused_block<double, kTile>(sv, b, stage, dt_given);
}
#endif

// A block per group of 32 columns: implicit block b of a member (its
// columns b*T .. b*T+T-1 at T = the implicit tile) is T/32 blocks here.
template <class R, bool full>
__global__ void __launch_bounds__(BWD_THREADS) kb_implicit_bwd(Batch bt, int stage,
                                                               int groups_per_iblock) {
  __shared__ __align__(16) DevView sv;
  static_assert(sizeof(DevView) % 16 == 0, "DevView is copied in 16-byte words");
  const unsigned ib = blockIdx.x / (unsigned)groups_per_iblock;
  const int m = batch_member(bt, ib);
  {
    const int4* src = reinterpret_cast<const int4*>(bt.views + m);
    int4* dst = reinterpret_cast<int4*>(&sv);
    for (int t = threadIdx.x; t < (int)(sizeof(DevView) / 16); t += blockDim.x) dst[t] = src[t];
  }
  const unsigned local = ib - bt.start[m];
  __syncthreads();
  if (sv.eqn == EXO_EQN_SHALLOW_YZ || !(sv.implicit_flag & 1)) return;
  if (((sv.implicit_flag & 8) != 0) != full) return;
  const int group =
      (int)(local * (unsigned)groups_per_iblock + blockIdx.x % (unsigned)groups_per_iblock);
  if (group * 32 >= 6 * sv.N * sv.N) return;
  implicit_bwd_block<R, full>(sv, group, stage);
}

__global__ void kb_roundtrip(Batch bt) {
  __shared__ __align__(16) DevView sv;
  unsigned b = batch_enter(bt, sv);
  if (sv.eqn == EXO_EQN_SHALLOW_YZ || (sv.implicit_flag & 1)) return;
  roundtrip_block(sv, b);
}

__global__ void k_p2c(DevView v, const double* wsrc) { p2c_block(v, blockIdx.x, wsrc); }

// time-step bookkeeping of every member (one thread per member)
__global__ void kb_dt_reset(const DevView* views, int n) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < n) views[m].sc->dtmin_bits = 0x7FEFFFFFFFFFFFFFull;
}
__global__ void kb_dt_finalize(const DevView* views, int n, int advance) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  DevScalars* sc = views[m].sc;
  if (advance) {
    sc->time += sc->dt;
    sc->ncycle += 1;
  }
  double nd = views[m].cfl * __longlong_as_double((long long)sc->dtmin_bits);
  sc->dt = advance ? fmin(2.0 * sc->dt, nd) : nd;
}

inline int check_launch() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : EXO_ERR_CUDA;
}

inline unsigned nblk(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

// the implicit kernels of a precision: FP32 blocks for
// EXO_PREC_MIXED_F32_SOLVE, FP64 for EXO_PREC_MIXED and the FP64 build; kinds:
// the block sizes the members take (IMPL_FULL, IMPL_PARTIAL)
template <class R>
inline void launch_kb_implicit(unsigned blocks, int threads, int nc1, cudaStream_t st, Batch b,
                               int stage, double dt_given, int kinds) {
  const int per = threads / 32;
  if (kinds & IMPL_FULL) {
#if EXO_MIXED
    if constexpr (sizeof(R) == 8) {
      if (fused_tiles(blocks, threads, nc1))
        kb_implicit_fused<true>
            <<<blocks, threads, fused_smem<true>(threads, nc1), st>>>(b, stage, dt_given);
      else
        kb_implicit_fused<false>
            <<<blocks, threads, fused_smem<false>(threads, nc1), st>>>(b, stage, dt_given);
    } else
#endif
    {
      kb_implicit<R, true><<<blocks, threads, impl_smem<R, true>(threads, nc1), st>>>(b, stage,
                                                                                     dt_given);
      kb_implicit_bwd<R, true>
          <<<blocks * (unsigned)per, BWD_THREADS, BwdLayout<R, 5>::bytes, st>>>(b, stage, per);
    }
  }
  if (kinds & IMPL_PARTIAL) {
    kb_implicit<R, false><<<blocks, threads, impl_smem<R, false>(threads, nc1), st>>>(b, stage,
                                                                                     dt_given);
    kb_implicit_bwd<R, false><<<blocks * (unsigned)per, BWD_THREADS, BwdLayout<R, 3>::bytes, st>>>(
        b, stage, per);
  }
}
inline void launch_kb_implicit(int precision, unsigned blocks, int threads, int nc1,
                               cudaStream_t st, Batch b, int stage, double dt_given, int kinds) {
#if EXO_MIXED
  if (precision == EXO_PREC_MIXED_F32_SOLVE) {
    launch_kb_implicit<float>(blocks, threads, nc1, st, b, stage, dt_given, kinds);
    return;
  }
#endif
  (void)precision;
  launch_kb_implicit<double>(blocks, threads, nc1, st, b, stage, dt_given, kinds);
}

}  // namespace

// The single-atmosphere launches run the batched kernels on a batch of one
// (the view's own device copy and block table), so an atmosphere advanced
// alone executes exactly the code it executes inside an ensemble.
inline Batch one(const DevView& v, int kind) { return Batch{v.self, v.starts + 2 * kind, 1}; }

inline unsigned member_block_count(const DevView& v, int kind) {
  unsigned b[BK_COUNT];
  member_blocks(v, v.tiles, b);
  return b[kind];
}

// 1/x as the FP64 implicit blocks of this compilation take it (inv_r),
// element-wise
__global__ void k_reciprocal(int n, const double* x, double* out) {
  const int m = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (m < n) out[m] = inv_r(x[m]);
}
int launch_reciprocal(int n, const double* x, double* out, void* stream) {
  if (n <= 0) return 0;
  k_reciprocal<<<nblk((size_t)n, 128), 128, 0, (cudaStream_t)stream>>>(n, x, out);
  return check_launch();
}

// Lines are cut into segments where one segment per line would fill the last
// wave of blocks badly: the count of segments whose waves x length is least,
// a segment's length being its chunks and half a chunk for the first cells'
// way in.  (FP64, N = 40, 40 levels, 600 blocks of whole lines: one
// segment 135 us, two 116; N = 48, 3 levels, 60 blocks: seven segments.)  A
// member of a batch keeps the split it has alone; results do not depend on it.
X23Split x23_split(int N, int L) {
  using T = EXO_FLUX_T;
  const unsigned CF = x23_shares_beta(L) ? x23_chunk<T, true>() : x23_chunk<T, false>();
  const unsigned groups = (unsigned)(((size_t)N * (size_t)L + 31) / 32);
  const unsigned nch = ((unsigned)N + CF) / CF, places = 148u * X23_RESIDENT;
  X23Split best{groups, nch, 1};
  size_t least = 0;
  for (unsigned n = 1; n <= nch; ++n) {
    const unsigned per = (nch + n - 1) / n, segments = (nch + per - 1) / per;
    const size_t waves = ((size_t)12 * groups * segments + places - 1) / places;
    const size_t cost = waves * (2 * per + 1);
    if (n == 1 || cost < least) {
      least = cost;
      best = {groups, per, segments};
    }
  }
  return best;
}

int prepare_kernels() {
  cudaError_t e = cudaSuccess;
  auto allow = [&](const void* f, int bytes) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  };
#if EXO_MIXED
  allow((const void*)kb_implicit_fused<true>, IMPL_SMEM_MAX);
  allow((const void*)kb_implicit_fused<false>, IMPL_SMEM_MAX);
#else
  allow((const void*)kb_implicit<double, true>, IMPL_SMEM_MAX);
  allow((const void*)kb_implicit_bwd<double, true>, (int)BwdLayout<double, 5>::bytes);
#endif
  allow((const void*)kb_implicit<double, false>, IMPL_SMEM_MAX);
  allow((const void*)kb_implicit_bwd<double, false>, (int)BwdLayout<double, 3>::bytes);
#if EXO_MIXED
  allow((const void*)kb_implicit<float, true>, IMPL_SMEM_MAX);
  allow((const void*)kb_implicit<float, false>, IMPL_SMEM_MAX);
  allow((const void*)kb_implicit_bwd<float, true>, (int)BwdLayout<float, 5>::bytes);
  allow((const void*)kb_implicit_bwd<float, false>, (int)BwdLayout<float, 3>::bytes);
#endif
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kb_flux_x1<EXO_FLUX_T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             X1_SMEM_MAX);
  return e == cudaSuccess ? 0 : EXO_ERR_CUDA;
}

int launch_prim_ghost(const DevView& v, bool compute_dt, void* stream) {
  kb_prim_ghost<<<member_block_count(v, BK_PRIM), v.tiles[BK_PRIM], 0, (cudaStream_t)stream>>>(
      one(v, BK_PRIM), compute_dt ? 1 : 0);
  return check_launch();
}

int launch_flux_x1(const DevView& v, void* stream) {
  if (v.eqn == EXO_EQN_SHALLOW_YZ) return 0;
  const int threads = x1_threads(v);
  size_t smem = x1_smem_bytes(v);
  kb_flux_x1<EXO_FLUX_T><<<member_block_count(v, BK_X1), threads, smem, (cudaStream_t)stream>>>(
      one(v, BK_X1));
  return check_launch();
}

int launch_flux_x23(const DevView& v, void* stream) {
  kb_flux_x23<EXO_FLUX_T><<<member_block_count(v, BK_X23), X23_THREADS, 0,
                            (cudaStream_t)stream>>>(
      one(v, BK_X23));
  return check_launch();
}

int launch_update(const DevView& v, int stage, void* stream) {
  kb_update<EXO_FLUX_T><<<member_block_count(v, BK_UPDATE), v.tiles[BK_UPDATE], 0,
                          (cudaStream_t)stream>>>(
      one(v, BK_UPDATE), stage);
  int rc = check_launch();
  if (rc) return rc;
  if (v.eqn != EXO_EQN_SHALLOW_YZ && !(v.implicit_flag & 1) && stage == 2) {
    kb_roundtrip<<<member_block_count(v, BK_ROUNDTRIP), v.tiles[BK_ROUNDTRIP], 0,
                   (cudaStream_t)stream>>>(
        one(v, BK_ROUNDTRIP));
    rc = check_launch();
  }
  return rc;
}

int launch_implicit(const DevView& v, int stage, void* stream) {
  if (v.eqn == EXO_EQN_SHALLOW_YZ || !(v.implicit_flag & 1)) return 0;
  launch_kb_implicit(v.precision, member_block_count(v, BK_IMPLICIT), v.tiles[BK_IMPLICIT], v.nc1,
                     (cudaStream_t)stream, one(v, BK_IMPLICIT), stage, 0.,
                     implicit_kind(v));
  return check_launch();
}

int launch_implicit_du(const DevView& v, double dt, void* stream) {
  if (v.eqn == EXO_EQN_SHALLOW_YZ || !(v.implicit_flag & 1)) return 0;
  launch_kb_implicit(v.precision, member_block_count(v, BK_IMPLICIT), v.tiles[BK_IMPLICIT], v.nc1,
                     (cudaStream_t)stream, one(v, BK_IMPLICIT), -1, dt,
                     implicit_kind(v));
  return check_launch();
}

int launch_dt_reset(const DevView& v, void* stream) {
  k_dt_reset<<<1, 1, 0, (cudaStream_t)stream>>>(v.sc);
  return check_launch();
}

int launch_dt_finalize(const DevView& v, double dt_fixed, bool advance_time, void* stream) {
  k_dt_finalize<<<1, 1, 0, (cudaStream_t)stream>>>(v.sc, v.cfl, dt_fixed, advance_time ? 1 : 0,
                                                   advance_time ? 0 : 1);
  return check_launch();
}

int launch_set_dt(const DevView& v, double dt, void* stream) {
  k_set_dt<<<1, 1, 0, (cudaStream_t)stream>>>(v.sc, dt);
  return check_launch();
}

int launch_p2c_interior(const DevView& v, const double* w_src, void* stream) {
  size_t total = (size_t)6 * v.N * v.N * v.L;
  k_p2c<<<nblk(total, 128), 128, 0, (cudaStream_t)stream>>>(v, w_src);
  return check_launch();
}

// One SSPRK(3,3) step of every member of a batch: the stage sequence of
// one_step() (capi.cpp) with each kernel launched once for all members.
int launch_batched_step(const BatchPlan& pl, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (pl.n <= 0) return 0;
  auto B = [&](int kind) { return Batch{pl.views, pl.start[kind], pl.n}; };
  int rc;
  for (int s = 0; s < 3; ++s) {
    if (pl.total[BK_X1]) {
      kb_flux_x1<EXO_FLUX_T><<<pl.total[BK_X1], pl.x1_threads, pl.x1_smem, st>>>(B(BK_X1));
      if ((rc = check_launch())) return rc;
    }
    kb_flux_x23<EXO_FLUX_T><<<pl.total[BK_X23], X23_THREADS, 0, st>>>(
        B(BK_X23));
    if ((rc = check_launch())) return rc;
    kb_update<EXO_FLUX_T><<<pl.total[BK_UPDATE], pl.threads[BK_UPDATE], 0, st>>>(B(BK_UPDATE), s);
    if ((rc = check_launch())) return rc;
    if (s == 2 && pl.total[BK_ROUNDTRIP]) {
      kb_roundtrip<<<pl.total[BK_ROUNDTRIP], pl.threads[BK_ROUNDTRIP], 0, st>>>(B(BK_ROUNDTRIP));
      if ((rc = check_launch())) return rc;
    }
    if (pl.total[BK_IMPLICIT]) {
      launch_kb_implicit(pl.precision, pl.total[BK_IMPLICIT], pl.threads[BK_IMPLICIT],
                         pl.max_nc1, st, B(BK_IMPLICIT), s, 0., pl.implicit_kinds);
      if ((rc = check_launch())) return rc;
    }
    if (s == 2) {
      kb_dt_reset<<<nblk(pl.n, 128), 128, 0, st>>>(pl.views, pl.n);
      if ((rc = check_launch())) return rc;
    }
    kb_prim_ghost<<<pl.total[BK_PRIM], pl.threads[BK_PRIM], 0, st>>>(B(BK_PRIM), s == 2 ? 1 : 0);
    if ((rc = check_launch())) return rc;
  }
  kb_dt_finalize<<<nblk(pl.n, 128), 128, 0, st>>>(pl.views, pl.n, 1);
  return check_launch();
}

}  // namespace EXO_KNS
}  // namespace exo
