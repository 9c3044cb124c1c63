// Device kernels of the per-timestep MHD update.  Included by exactly one
// translation unit per precision: mhd_fp64.cu (built with -fmad=false: FP64
// products are fused only where the code says so, and the edge EMF and metric mode
// round as the reference does) and mhd_fp32.cu (FMA contraction on, the performance path).
//
// Kernel map (reference routine -> kernel):
//   get_bxyz (mhd3d3.f90:2118-2128) + vf of get_eijk_LFM (1766)  -> k_ct_fill,
//     k_fill_bxyz (k_bxyz_vf at init)
//   get_dt   (1608-1639) + diag_rho_neg/diag_overflow (3143-3160) -> cell_dt in k_ct_fill
//     and k_fill_bxyz or in k_cfl, k_cfl_final
//   advance_previous (3794-3819) -> FORM_SAVE of the first stage (metric mode: k_cfl)
//   advance_predictor_ab (3821-3840)                              -> k_predictor_ab
//   get_flux_stress + get_v_face + reconstruct_3d (2385-2615, 833-1596)
//     -> FP32: k_flux (x faces), k_flux_sweep or k_flux_t of D = 1 (y faces, x+y
//        divergence) and D = 2 (z faces + the conserved update below);
//        FP64: k_faces (all axes), batches as FP32 tiles
//   get_eijk_LFM + get_vav_center2corner + interp2_* (1754-2116, 926-1067)
//     -> FP32: k_emf_stream + k_emf_rows or k_emf_pdm (PDM), k_emf_weno, k_emf (TVD);
//        FP64: k_emf64 (PDM, WENO), k_emf (TVD), k_emf_pdm (batches)
//   get_eijk_Yee (1654-1752)                                      -> k_yee_split, k_emf_yee
//   get_conserve + advance_corrector1/2 + RK combines (1641-1650, 3842-3907,
//     3670-3697, 3741-3783) -> cell_update_vals in the z faces (FP64: k_update_faces)
//   advance_bijk + B combines (3909-3933, 3698-3702, 3784-3788) -> k_ct_fill (metric: k_update_b)
//   fill_hydro_mpi / fill_mag_mpi (781-819, 346-616) -> k_fill_bxyz (k_fill at init)
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include <atomic>
#include <math.h>
#include <stdint.h>
#include "mhd_state.h"

namespace mhd {

// R_PDMG: PDM with a limiter constant for which the sign-free form (R_PDM) does not hold
// (pdm_signless; carve() picks it), evaluated as the reference writes the limiter, in the same kernels.
enum { R_PDM = 1, R_TVD = 2, R_WENO = 3, R_MPWENO = 4, R_TVDMC = 5, R_PDMG = 6 };
enum { BC_PERIODIC = 0, BC_EVEN = 1, BC_REFLECT = 2, BC_OUTFLOW = 3 };
enum { EMF_LFM = 0, EMF_YEE = 1 };

// Kernels with more than 48 KB of dynamic shared memory must be enabled per
// device: a launcher sets its attributes the first time it runs on the
// current device (idempotent if two host threads race; the bit is set only
// after the attributes are).
struct PerDevice {
  std::atomic<unsigned long long> done{0};
  bool need(unsigned long long& bit) {
    int dev = 0;
    cudaGetDevice(&dev);
    bit = 1ull << (dev & 63);
    return !(done.load(std::memory_order_acquire) & bit);
  }
  void mark(unsigned long long bit) { done.fetch_or(bit, std::memory_order_release); }
};

// Preferred shared-memory carveout (percent of the SM's maximum) of a kernel,
// set once per device.  The L1-reliant step passes ask for the shared memory
// they need and no more, so that the configuration a preceding
// shared-memory-heavy launch (the EMF slice rings) leaves behind does not
// shrink their L1.
#ifndef MHD_L1_PREF
#define MHD_L1_PREF 0
#endif
template <typename K>
inline void prefer_carveout(K kernel, int pct, PerDevice& attr) {
  if (!MHD_L1_PREF) return;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
    attr.mark(bit);
  }
}

inline dim3 grid3(int ni, int nj, int nk, dim3 b) {
  return dim3((ni + b.x - 1) / b.x, (nj + b.y - 1) / b.y, nk);
}
enum { ST_NAN = 1u, ST_NEG_RHO = 2u, ST_NEG_P = 4u, ST_CFL = 8u };

// ---------------------------------------------------------------- scalar ops
// Fortran sign(1,x) with ifort's default: +1 for x >= 0, including -0.0.
template <typename T> __device__ __forceinline__ T sgn1(T x) { return x >= T(0) ? T(1) : T(-1); }
template <typename T> __device__ __forceinline__ T mx(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T mn(T a, T b) { return a < b ? a : b; }
__device__ __forceinline__ double fab(double x) { return fabs(x); }
__device__ __forceinline__ float fab(float x) { return fabsf(x); }
__device__ __forceinline__ double sq(double x) { return sqrt(x); }
__device__ __forceinline__ float sq(float x) { return sqrtf(x); }
__device__ __forceinline__ double ex(double x) { return exp(x); }
__device__ __forceinline__ float ex(float x) { return expf(x); }
__device__ __forceinline__ double erc(double x) { return erfc(x); }
__device__ __forceinline__ float erc(float x) { return erfcf(x); }

// Division by a constant: exact in FP64 (reference rounding), reciprocal
// multiply in FP32.
template <typename T> struct Div;
template <> struct Div<double> {
  static __device__ __forceinline__ double by(double a, double b) { return a / b; }
};
template <> struct Div<float> {
  static __device__ __forceinline__ float by(float a, float b) { return a * (1.0f / b); }
};

// Divisions on the hot path.  An FP64 division takes about nine operations of
// the FP64 pipe, the bound of every FP64 kernel, so it is kept where the
// quotient is a result by itself (dv); by a cell width it is a multiply by the
// reciprocal (dc, both precisions), and several quotients by one divisor share
// its reciprocal (dvr).  FP32 multiplies by a reciprocal throughout.  The FP64
// metric mode divides (dw) and keeps the reference's roundings everywhere: its
// blast is symmetric to the last bit, and where two slopes tie the corner
// limiter's choice follows the rounding (8 faces of bk move by 1e-7 of 1e-6 in
// the second step after a change of 1e-16).
static __device__ __noinline__ double quot_far(double a, double b) { return a / b; }
template <typename T> struct Ops;
template <> struct Ops<double> {
  static __device__ __forceinline__ double dw(double a, double w, double) { return a / w; }     // metric mode: a / V
  static __device__ __forceinline__ double dc(double a, double, double rw) { return a * rw; }  // a / width
  static __device__ __forceinline__ double dv(double a, double b) { return a / b; }
  static __device__ __forceinline__ double rcp(double b) { return 1.0 / b; }  // used with dvr below
  // a / b from rb = 1 / b and one residual correction (Markstein's theorem:
  // the rounding of the division when a rb is within one unit of it).  Where rb or
  // a rb is beyond the range (a subnormal, zero or infinite b) the correction is
  // NaN, and the quotient divides.
  static __device__ __forceinline__ double dvr(double a, double b, double rb) {
    const double q = a * rb, r = fma(fma(-q, b, a), rb, q);
    return (__double2hiint(r) & 0x7ff00000) < 0x7ff00000 ? r : quot_far(a, b);
  }
};
template <> struct Ops<float> {
  static __device__ __forceinline__ float dw(float a, float, float rw) { return a * rw; }
  static __device__ __forceinline__ float dc(float a, float, float rw) { return a * rw; }
  static __device__ __forceinline__ float dv(float a, float b) { return __fdividef(a, b); }
  static __device__ __forceinline__ float rcp(float b) { return __frcp_rn(b); }
  static __device__ __forceinline__ float dvr(float a, float, float rb) { return a * rb; }
};

// 8-point centred interpolant (interp_pdm, mhd3d3.f90:866-872):
// (-3, 29, -139, 533, 533, -139, 29, -3) / 840.  tap8: the reference's operand
// order (FP32 contracted, with a reciprocal multiply in place of the division;
// FP64 see div_by).  tap8_fused (FP64 face fluxes): eight fused operations with
// the coefficients divided beforehand, the smallest first, so that the rounding
// of the large terms happens once, at the end (rms error 0.4 of the reference
// order's on smooth and random taps).
__device__ __forceinline__ float tap8(float a0, float a1, float a2, float a3, float a4, float a5, float a6, float a7) {
  float s = fmaf(29.0f, a1, -3.0f * a0);
  s = fmaf(533.0f, a3, fmaf(-139.0f, a2, s));
  s = fmaf(-139.0f, a5, fmaf(533.0f, a4, s));
  s = fmaf(-3.0f, a7, fmaf(29.0f, a6, s));
  return s * (1.0f / 840.0f);
}
__device__ __forceinline__ double tap8_fused(double a0, double a1, double a2, double a3, double a4, double a5, double a6,
                                             double a7) {
  constexpr double c0 = -3.0 / 840.0, c1 = 29.0 / 840.0, c2 = -139.0 / 840.0, c3 = 533.0 / 840.0;
  double s = fma(c0, a7, c0 * a0);
  s = fma(c1, a6, fma(c1, a1, s));
  s = fma(c2, a5, fma(c2, a2, s));
  return fma(c3, a4, fma(c3, a3, s));
}

// PDM2 (mhd3d3.f90:1069-1172) for pdmb > 0, without its signs: the
// interpolant fi clamped to the two near cells gives x, and with D(c, f) = 2
// pdmb (c - f) the left state is x kept within [fm1, fm1 + D(fm1, fm2)] -- the
// reference's x - s0 max(0, |x - fm1| - |sm + s0| |dfm|) is exactly that: |sm +
// s0| is 2 where the two slopes agree and 0 where they do not, and in the latter
// case the two intervals share only fm1.  The right state is the mirror image
// about f0.
//
// FP32 keeps the bits of the reference's form (the corner limiter picks the
// larger of two slopes, so a last bit elsewhere can move a cell by 1e-3 within
// a hundred steps): the excess of the displacement d = x - near over D, a soft
// threshold, is d - (d and D of one sign ? the smaller magnitude : 0), the
// product of signs and the smaller magnitude being one instruction (FMNMX with
// xorsign); the same roundings as |d| - |sm + s0| |dfm| and the final
// difference.  24 instructions per state pair and field instead of 35.
//
// FP64: comparisons share the FP64 pipe (2 lanes per SM and cycle, a 32nd of the
// integer pipe), so minima and maxima run on order-preserving integer images
// of the values, and the face fluxes take the state as x held within the two
// intervals at once (within(): one rounding of c + D).
// NaN: of a face's two states one is NaN where one is in the reference's form, and a NaN
// that is only in the interpolant is dropped by the clamp there as here (the larger near
// cell remains).  A right state whose far cell alone is NaN is NaN here and the near cell
// there: sums over both sides or all quadrants do not show it; the Yee EMF, which takes
// one side, passes the near cell as the other bound of the clamp (lim).
template <typename T> struct Sel;
template <> struct Sel<float> {
  typedef float K;
  static __device__ __forceinline__ K key(float x) { return x; }
  static __device__ __forceinline__ K interp(float x) { return x; }
  static __device__ __forceinline__ float val(K k) { return k; }
  static __device__ __forceinline__ K mn(K a, K b) { return fminf(a, b); }
  static __device__ __forceinline__ K mx(K a, K b) { return fmaxf(a, b); }
  static __device__ __forceinline__ K mn_nan(K a, K b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
  }
  static __device__ __forceinline__ K mn3(K a, K b, K c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
  }
  static __device__ __forceinline__ K mx3(K a, K b, K c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
  }
  static __device__ __forceinline__ K mx_nan(K a, K b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
  }
  static __device__ __forceinline__ float keep_nan(float r, float) { return r; }
};
template <> struct Sel<double> {
  typedef long long K;  // ordered as the doubles are: negative values with the magnitude bits inverted
  static __device__ __forceinline__ K flip(K b) { return b ^ ((b >> 63) & 0x7fffffffffffffffLL); }
  static __device__ __forceinline__ K key(double x) { return flip(__double_as_longlong(x)); }
  // of an interpolant: a NaN of either sign is beyond infinity
  static __device__ __forceinline__ K interp(double x) {
    return (unsigned)__double2hiint(x) > 0xfff00000u ? 0x7fffffffffffffffLL : key(x);
  }
  static __device__ __forceinline__ double val(K k) { return __longlong_as_double(flip(k)); }
  static __device__ __forceinline__ K mn(K a, K b) { return a < b ? a : b; }
  static __device__ __forceinline__ K mx(K a, K b) { return a > b ? a : b; }
  static __device__ __forceinline__ K mn_nan(K a, K b) { return mn(a, b); }
  static __device__ __forceinline__ K mn3(K a, K b, K c) { return mn(mn(a, b), c); }
  static __device__ __forceinline__ K mx3(K a, K b, K c) { return mx(mx(a, b), c); }
  static __device__ __forceinline__ K mx_nan(K a, K b) { return mx(a, b); }
  // the integer images order a NaN beyond infinity: hand it on instead
  // (out = c + D(c, outer) is NaN when c or outer is)
  static __device__ __forceinline__ double keep_nan(double r, double out) {
    return (__double2hiint(out) & 0x7fffffff) > 0x7ff00000 ? out : r;
  }
};
// FP32: x clamped to [a, b], and the soft threshold.
__device__ __forceinline__ float clamp2(float a, float b, float x) {
  typedef Sel<float> S;
  return S::mx_nan(S::mn_nan(a, b), S::mn(x, S::mx(a, b)));
}
__device__ __forceinline__ float shrink(float d, float D) {  // d and D of one sign: the smaller, with the sign of d
  float m;
  asm("min.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(m) : "f"(d), "f"(D));
  return copysignf(Sel<float>::mx_nan(m, 0.0f), d);
}
__device__ __forceinline__ void pdm_states(float fm2, float fm1, float f0, float fp1, float fi, float pdmb, float& fl,
                                           float& fr, float lim) {
  const float k = pdmb + pdmb, x = clamp2(lim, f0, fi);
  const float dl = x - fm1, dr = x - f0;
  fl = x - (dl - shrink(dl, k * (fm1 - fm2)));
  fr = x - (dr - shrink(dr, k * (f0 - fp1)));
}
// FP64 face fluxes: x held within [c, far] and [c, out]; lo = min(c, far), hi = max(c, far).
__device__ __forceinline__ double within(long long lo, long long hi, long long c, double out, long long x) {
  typedef Sel<double> S;
  const long long o = S::key(out);
  return S::keep_nan(S::val(S::mx3(lo, S::mn(c, o), S::mn3(hi, S::mx(c, o), x))), out);
}
__device__ __forceinline__ void pdm_states_fused(double fm2, double fm1, double f0, double fp1, double fi, double pdmb,
                                                 double& fl, double& fr, double lim) {
  typedef Sel<double> S;
  const double k = pdmb + pdmb;
  const long long a = S::key(fm1), b = S::key(f0), x = S::interp(fi), m = S::key(lim);
  const long long lo = S::mn(m, b), hi = S::mx(m, b);
  fl = within(lo, hi, a, fma(k, fm1 - fm2, fm1), x);
  fr = within(lo, hi, b, fma(k, f0 - fp1, f0), x);
}

// ------------------------------------------------ edge EMF forms (FP64)
// The FP64 edge EMF keeps the reference's roundings, while the face fluxes take
// the fused forms above: a face-B component that is zero at first takes its
// value from CT differences of E, so the last bit of E shows in it (corner
// velocities or face B rounded otherwise, however exactly, move bz of the
// 12 x 10 x 9 vortex by 1.8e-11 of its own size in 4 steps, the fluxes by 6e-12).
// What the roundings leave free is where the decisions are made: comparisons,
// minima, signs and absolute values run on the integer pipe, and the division
// by 840 takes two operations.  FP32 has one form for both.
//
// x / 840, correctly rounded: x zh + x zl with zh + zl = 1/840 to twice the
// precision errs by about 2^-106 of the quotient before its one rounding,
// while a quotient by 840 = 8 * 105 is never closer than 2^-54 / 105 to the
// midpoint of two doubles (105 times an odd 54-bit integer has more than 53
// bits, so no midpoint is a quotient, and the gap is a whole unit of x).
template <int N> __device__ __forceinline__ double div_by(double x) {
  constexpr double zh = 1.0 / N;
  // 1/N - zh = (1 - N zh) / N: N zh is split so that both products are exact
  constexpr double zt = (zh * 134217729.0) - ((zh * 134217729.0) - zh);  // upper half of zh
  constexpr double zl = ((1.0 - N * zt) - N * (zh - zt)) / N;
  return fma(x, zh, x * zl);
}
__device__ __forceinline__ double abs_bits(double x) {
  return __hiloint2double(__double2hiint(x) & 0x7fffffff, __double2loint(x));
}
// a >= b for |a|, |b| (integer comparison of the magnitudes), false where either is NaN
__device__ __forceinline__ bool abs_ge(double a, double b) {
  const long long x = __double_as_longlong(a) & 0x7fffffffffffffffLL;
  return x >= (__double_as_longlong(b) & 0x7fffffffffffffffLL) && (int)(x >> 32) <= 0x7ff00000;
}
__device__ __forceinline__ bool abs_ge(float a, float b) { return fabsf(a) >= fabsf(b); }
// x >= 0 (-0.0 counts)
__device__ __forceinline__ bool ge0(double x) { return Sel<double>::key(x) >= -1LL; }
__device__ __forceinline__ bool ge0(float x) { return x >= 0.0f; }

__device__ __forceinline__ double tap8(double a0, double a1, double a2, double a3, double a4, double a5, double a6,
                                       double a7) {
  double s = -3.0 * a0;
  s = s + 29.0 * a1;
  s = s - 139.0 * a2;
  s = s + 533.0 * a3;
  s = s + 533.0 * a4;
  s = s - 139.0 * a5;
  s = s + 29.0 * a6;
  s = s - 3.0 * a7;
  return div_by<840>(s);
}
// Limiter states of the FP64 edge EMF.
struct Edge64 {
  typedef Sel<double> S;
  // the clamp of PDM2: x held within [a, b]
  static __device__ __forceinline__ double clamp(S::K a, S::K b, S::K x) {
    return S::val(S::mx(S::mn(a, b), S::mn(x, S::mx(a, b))));
  }
  // fii -+ max(0, |near - fii| - q |dn|), q = 2 where the slopes towards the
  // far cell (up) and from the outer one (dn = pdmb (near - outer)) agree, else
  // 0; - when the far cell is the larger.  2 |dn| is exact, so the fused
  // difference rounds as the reference's product and difference do.
  static __device__ __forceinline__ double limited(double near, double fii, double dn, bool up) {
    const int hd = __double2hiint(dn);
    const double m = (hd >= 0) == up || (hd & 0x7fffffff) > 0x7ff00000 ? abs_bits(dn) : 0.0;  // (NaN stays)
    const double t = fma(-2.0, m, abs_bits(near - fii));
    const int h = __double2hiint(t);
    const bool neg = (unsigned)h - 0x80000000u <= 0x7ff00000u;  // below zero (not NaN)
    const double x = __hiloint2double(neg ? 0 : (up ? h ^ 0x80000000 : h), neg ? 0 : __double2loint(t));
    return fii + x;
  }
  static __device__ __forceinline__ void states(double fm2, double fm1, double f0, double fp1, double fi, double pdmb,
                                                double& fl, double& fr) {
    const S::K a = S::key(fm1), b = S::key(f0);
    const double fii = clamp(a, b, S::interp(fi));
    fl = limited(fm1, fii, pdmb * (fm1 - fm2), b >= a);
    fr = limited(f0, fii, pdmb * (f0 - fp1), a > b);
  }
};

// PDM2 (mhd3d3.f90:1069-1172) as the reference writes it, for any pdmb (R_PDMG).
template <typename T>
__device__ __forceinline__ void pdm2(T fm2, T fm1, T f0, T fp1, T fi, T pdmb, T& fl, T& fr) {
  T maxf = mx(fm1, f0), minf = mn(fm1, f0);
  T fii = mx(minf, mn(fi, maxf));
  T dfm = pdmb * (fm1 - fm2);
  T df0 = pdmb * (f0 - fm1);
  T dfp = pdmb * (fp1 - f0);
  T sm = sgn1(dfm), s0 = sgn1(df0), sp = sgn1(dfp);
  dfm = fab(dfm);
  dfp = fab(dfp);
  T qm = fab(sm + s0), qp = fab(s0 + sp);
  T dfl = fii - fm1, dfr = f0 - fii;
  fl = fii - s0 * mx(T(0), fab(dfl) - qm * dfm);
  fr = fii + s0 * mx(T(0), fab(dfr) - qp * dfp);
}

// TVD (mhd3d3.f90:1238-1248): van Leer b = (a+|a|)/(1+|a|); MC variant
// b = max(0, min(2a, (1+a)/2, 2)) (fi is the centred value, so b is phi(a)).
// Quotients: Ops<T>::dv divides exactly in FP64 (the reference's rounding)
// and multiplies by the hardware reciprocal in FP32.
template <typename T, bool MC>
__device__ __forceinline__ T tvdb(T a) {
  if (MC) return mx(T(0), mn(mn(T(2) * a, T(0.5) * (T(1) + a)), T(2)));
  return Ops<T>::dv(a + fab(a), T(1) + fab(a));
}
template <typename T, bool MC>
__device__ __forceinline__ void tvd(T fm2, T fm1, T f0, T fp1, T fi, T eps, T& fl, T& fr) {
  T a = Ops<T>::dv(fm1 - fm2, f0 - fm1 + eps);
  T b = tvdb<T, MC>(a);
  fl = fm1 - b * (fm1 - fi);
  a = Ops<T>::dv(f0 - fp1, fm1 - f0 + eps);
  b = tvdb<T, MC>(a);
  fr = f0 - b * (f0 - fi);
}

template <typename T>
struct Prm {
  T pdmb, eps, alpha, beta;
  int tvd_shift;
};

// ------------------------------------------------------------------ WENO
// WENO5 (mhd3d3.f90:1329-1375) and the monotonicity-preserving bound of MPWENO5
// (1530-1591).  The right state of a face is the left-state formula on the
// mirrored stencil.
//
// minmod of four (1380-1403, nested): the one nearest zero where all signs
// agree, else zero, i.e. the median of their minimum, their maximum and zero.
template <typename T>
__device__ __forceinline__ T mm4(T a, T b, T c, T d) {
  typedef Sel<T> S;
  const typename S::K p = S::key(a), q = S::key(b), r = S::key(c), s = S::key(d);
  const typename S::K lo = S::mn(S::mn3(p, q, r), s), hi = S::mx(S::mx3(p, q, r), s);
  return S::val(S::mx(lo, S::mn(hi, S::key(T(0)))));
}
// The bounds of the bound: lo = max(min(a1, b0, md), min(a1, ul, lc)), hi = min(max(..), max(..)).
template <typename T>
__device__ __forceinline__ void mp_bounds(T a1, T b0, T md, T ul, T lc, typename Sel<T>::K& lo, typename Sel<T>::K& hi) {
  typedef Sel<T> S;
  const typename S::K p = S::key(a1), q = S::key(b0), m = S::key(md), u = S::key(ul), c = S::key(lc);
  lo = S::mx(S::mn3(p, q, m), S::mn3(p, u, c));
  hi = S::mn(S::mx3(p, q, m), S::mx3(p, u, c));
}

// FP32: one value, or a pair of values in the packed lanes (two fields of a
// face, the two velocity components of an edge, the two sides of a face).  Bound
// by issue and the ALU pipe; the pair halves the arithmetic, the signs, minima
// and maxima of the bound stay per lane.  Every operation rounds as the
// contracted scalar code before it did (the same products fused), because the
// corner velocities choose between two one-sided estimates and a last bit can
// turn the choice: 128^3 RK3 frames keep their bits.
template <typename V> struct VOps;
template <> struct VOps<float> {
  static __device__ __forceinline__ float k(float a) { return a; }
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fadd_rn(a, -b); }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
  static __device__ __forceinline__ float quot(float a, float b) { return __fdividef(a, b); }
  static __device__ __forceinline__ float mm4v(float a, float b, float c, float d) { return mm4(a, b, c, d); }
  // w + minmod(lo - w, hi - w)
  static __device__ __forceinline__ float bound(float w, float a1, float b0, float md, float ul, float lc) {
    float lo, hi;
    mp_bounds(a1, b0, md, ul, lc, lo, hi);
    return __fadd_rn(w, shrink(__fadd_rn(lo, -w), __fadd_rn(hi, -w)));
  }
};
template <> struct VOps<float2> {
  static __device__ __forceinline__ float2 k(float a) { return make_float2(a, a); }
  static __device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
  static __device__ __forceinline__ float2 sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
  static __device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
  static __device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
  static __device__ __forceinline__ float2 quot(float2 a, float2 b) {
    return make_float2(__fdividef(a.x, b.x), __fdividef(a.y, b.y));
  }
  static __device__ __forceinline__ float2 mm4v(float2 a, float2 b, float2 c, float2 d) {
    return make_float2(mm4(a.x, b.x, c.x, d.x), mm4(a.y, b.y, c.y, d.y));
  }
  static __device__ __forceinline__ float2 bound(float2 w, float2 a1, float2 b0, float2 md, float2 ul, float2 lc) {
    float2 lo, hi;
    mp_bounds(a1.x, b0.x, md.x, ul.x, lc.x, lo.x, hi.x);
    mp_bounds(a1.y, b0.y, md.y, ul.y, lc.y, lo.y, hi.y);
    const float2 p = sub(lo, w), q = sub(hi, w);
    return add(w, make_float2(shrink(p.x, q.x), shrink(p.y, q.y)));
  }
};
// State next to the near cell a1 of the stencil (a3, a2, a1 | b0, b1).
template <typename V, int RECON>
__device__ __forceinline__ V weno_side(V a3, V a2, V a1, V b0, V b1, const Prm<float>& P) {
  typedef VOps<V> O;
  const V c13 = O::k(13.0f / 12.0f), c4 = O::k(0.25f), m4 = O::k(-4.0f), m2 = O::k(-2.0f), eps = O::k(P.eps);
  const V m3 = O::mul(O::k(3.0f), a1);
  const V h0 = O::fma(O::k(11.0f), a1, O::fma(O::k(-7.0f), a2, O::add(a3, a3)));
  const V n1 = O::fma(m2, b0, O::fma(O::k(-5.0f), a1, a2));  // -(-a2 + 5 a1 + 2 b0)
  const V h2 = O::sub(O::fma(O::k(5.0f), b0, O::add(a1, a1)), b1);
  const V t0 = O::add(O::fma(m2, a2, a3), a1), t1 = O::add(O::fma(m2, a1, a2), b0);
  const V t2 = O::add(O::fma(m2, b0, a1), b1);
  const V u0 = O::add(O::fma(m4, a2, a3), m3), u1 = O::sub(a2, b0), u2 = O::add(O::fma(m4, b0, m3), b1);
  const V e0 = O::add(eps, O::fma(c13, O::mul(t0, t0), O::mul(c4, O::mul(u0, u0))));
  const V e1 = O::add(eps, O::fma(c4, O::mul(u1, u1), O::mul(c13, O::mul(t1, t1))));
  const V e2 = O::add(eps, O::fma(c13, O::mul(t2, t2), O::mul(c4, O::mul(u2, u2))));
  const V q0 = O::quot(O::k(0.1f), O::mul(e0, e0)), q1 = O::quot(O::k(0.6f), O::mul(e1, e1));
  const V q2 = O::quot(O::k(0.3f), O::mul(e2, e2));
  const V rs = O::quot(O::k(1.0f), O::add(O::add(q0, q1), q2)), r6 = O::k(1.0f / 6.0f);
  const V w = O::fma(O::mul(q2, rs), O::mul(r6, h2),
                     O::fma(O::mul(q0, rs), O::mul(r6, h0), O::mul(O::mul(q1, rs), O::mul(O::k(-1.0f / 6.0f), n1))));
  if (RECON != R_MPWENO) return w;
  const V f1 = O::mul(O::k(4.0f), t1);
  const V s0 = O::mm4v(O::sub(f1, t2), O::sub(O::mul(O::k(4.0f), t2), t1), t1, t2);
  const V w0 = O::mm4v(O::sub(O::mul(O::k(4.0f), t0), t1), O::sub(f1, t0), t0, t1);
  const V ul = O::fma(O::k(P.alpha), O::sub(a1, a2), a1);
  const V md = O::mul(O::k(0.5f), O::sub(O::add(a1, b0), s0));
  const V lc = O::fma(O::k(0.5f), O::sub(m3, a2), O::mul(O::k(1.0f / 3.0f), O::mul(O::k(P.beta), w0)));
  return O::bound(w, a1, b0, md, ul, lc);
}
// Both states of the face between fm1 and f0 (one value: the two sides as a pair).
template <int RECON>
__device__ __forceinline__ void weno_both(float2 fm3, float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fp2,
                                          const Prm<float>& P, float2& fl, float2& fr) {
  fl = weno_side<float2, RECON>(fm3, fm2, fm1, f0, fp1, P);
  fr = weno_side<float2, RECON>(fp2, fp1, f0, fm1, fm2, P);
}
template <int RECON>
__device__ __forceinline__ void weno_both(float fm3, float fm2, float fm1, float f0, float fp1, float fp2,
                                          const Prm<float>& P, float& fl, float& fr) {
  const float2 r = weno_side<float2, RECON>(make_float2(fm3, fp2), make_float2(fm2, fp1), make_float2(fm1, f0),
                                                   make_float2(f0, fm1), make_float2(fp1, fm2), P);
  fl = r.x;
  fr = r.y;
}

// FP64 face fluxes: everything from the first differences, which both sides
// share: the second differences, the slopes of the smoothness indicators, and
// the candidates as offsets from the near cell, so that a state is that cell
// plus a small correction (half a unit of rounding).  48 operations of the FP64
// pipe per state, as the reference writes it about 150: one division instead
// of nine, the weights 1 : 6 : 3 over e^2 brought to their common denominator
// after scaling by a power of two (integer pipe).  Beside a jump whose indicator is 2^450
// times those of the smooth candidates the scaled squares of these vanish: there the
// weights are the quotients.
static __device__ __noinline__ double weno_mix_far(double e0, double e1, double e2, double g0, double g1, double g2) {
  const double a0 = 1.0 / (e0 * e0), a1 = 6.0 / (e1 * e1), a2 = 3.0 / (e2 * e2);
  return (a0 * g0 + a1 * g1 + a2 * g2) / (6.0 * (a0 + a1 + a2));
}
__device__ __forceinline__ double weno_mix(double e0, double e1, double e2, double g0, double g1, double g2) {
  const int x0 = __double2hiint(e0), x1 = __double2hiint(e1), x2 = __double2hiint(e2);
  const int sh = (max(x0, max(x1, x2)) & 0x7ff00000) - 0x3ff00000;
  const double s0 = __hiloint2double(max(x0 - sh, 0x00100000), __double2loint(e0));
  const double s1 = __hiloint2double(max(x1 - sh, 0x00100000), __double2loint(e1));
  const double s2 = __hiloint2double(max(x2 - sh, 0x00100000), __double2loint(e2));
  const double d0 = s0 * s0, d1 = s1 * s1, d2 = s2 * s2;
  const double a0 = d1 * d2, a1 = (6.0 * d0) * d2, a2 = (3.0 * d0) * d1, sum = a0 + a1 + a2;
  if (__double2hiint(sum) < (1023 - 900) << 20) return weno_mix_far(e0, e1, e2, g0, g1, g2);
  return fma(a0, g0, fma(a1, g1, a2 * g2)) / (6.0 * sum);
}
// S = 1 for the left state, -1 for the right one (the stencil mirrored): near
// cell a1, the cell b0 across the face, the first differences dm behind a1 and
// d0 across the face in the direction of increasing index, and the second
// differences t0, t1, t2 about the cell behind a1, a1 and b0.
template <int RECON, int S>
__device__ __forceinline__ double weno_side64(double a1, double b0, double dm, double d0, double t0, double t1,
                                              double t2, const Prm<double>& P) {
  const double c = 13.0 / 3.0, eps = 4.0 * P.eps;  // e_i = 4 (eps + s_i)
  const double u0 = fma(2.0 * S, dm, t0), u1 = dm + d0, u2 = fma(-2.0 * S, d0, t2);
  const double e0 = fma(c * t0, t0, fma(u0, u0, eps)), e1 = fma(c * t1, t1, fma(u1, u1, eps));
  const double e2 = fma(c * t2, t2, fma(u2, u2, eps));
  const double g0 = fma((double)S, u0 + t0, dm), g1 = fma(2.0, d0, dm), g2 = fma(-(double)S, u2, d0);
  const double w = fma((double)S, weno_mix(e0, e1, e2, g0, g1, g2), a1);
  if (RECON != R_MPWENO) return w;
  const double s0 = mm4(fma(4.0, t1, -t2), fma(4.0, t2, -t1), t1, t2);
  const double w0 = mm4(fma(4.0, t0, -t1), fma(4.0, t1, -t0), t0, t1);
  typedef Sel<double> K;
  long long lo, hi;
  mp_bounds(a1, b0, fma(0.5 * S, d0, fma(-0.5, s0, a1)), fma(S * P.alpha, dm, a1),
            fma(0.5 * S, dm, fma(P.beta * (1.0 / 3.0), w0, a1)), lo, hi);
  // w + minmod(lo - w, hi - w): the median of w, lo and hi
  return K::keep_nan(K::val(K::mx(K::mn(lo, hi), K::mn(K::mx(lo, hi), K::key(w)))), w);
}
template <int RECON>
__device__ __forceinline__ void weno_both(double fm3, double fm2, double fm1, double f0, double fp1, double fp2,
                                          const Prm<double>& P, double& fl, double& fr) {
  const double da = fm2 - fm3, db = fm1 - fm2, dc = f0 - fm1, dd = fp1 - f0, de = fp2 - fp1;
  const double ta = db - da, tb = dc - db, tc = dd - dc, td = de - dd;
  fl = weno_side64<RECON, 1>(fm1, f0, db, dc, ta, tb, tc, P);
  fr = weno_side64<RECON, -1>(f0, fm1, dd, dc, td, tc, tb, P);
}

// The state with the reference's roundings (FP64 edge EMF and metric mode):
// products by powers of two are fused, constant divisors take two operations
// and the quotients by the weights' sum share its reciprocal.
template <int RECON>
__device__ __forceinline__ double weno_side_ref(double a3, double a2, double a1, double b0, double b1,
                                                const Prm<double>& P) {
  const double eps = P.eps, c13 = 13.0 / 12.0;
  const double h0 = div_by<6>(fma(2.0, a3, -(7.0 * a2)) + 11.0 * a1);
  const double h1 = div_by<6>(fma(2.0, b0, 5.0 * a1 - a2));
  const double h2 = div_by<6>(fma(2.0, a1, 5.0 * b0) - b1);
  const double t0 = fma(-2.0, a2, a3) + a1, t1 = fma(-2.0, a1, a2) + b0, t2 = fma(-2.0, b0, a1) + b1;
  const double u0 = fma(-4.0, a2, a3) + 3.0 * a1, u1 = a2 - b0, u2 = fma(-4.0, b0, 3.0 * a1) + b1;
  const double e0 = eps + fma(0.25, u0 * u0, c13 * (t0 * t0)), e1 = eps + fma(0.25, u1 * u1, c13 * (t1 * t1));
  const double e2 = eps + fma(0.25, u2 * u2, c13 * (t2 * t2));
  const double s0 = 0.1 / (e0 * e0), s1 = 0.6 / (e1 * e1), s2 = 0.3 / (e2 * e2);
  typedef Ops<double> O;
  const double sum = s0 + s1 + s2, rs = O::rcp(sum);
  const double w = O::dvr(s0, sum, rs) * h0 + O::dvr(s1, sum, rs) * h1 + O::dvr(s2, sum, rs) * h2;
  if (RECON != R_MPWENO) return w;
  typedef Sel<double> S;
  const double m0 = mm4(fma(4.0, t1, -t2), fma(4.0, t2, -t1), t1, t2);
  const double m1 = mm4(fma(4.0, t0, -t1), fma(4.0, t1, -t0), t0, t1);
  long long kl, kh;
  mp_bounds(a1, b0, 0.5 * (a1 + b0 - m0), a1 + P.alpha * (a1 - a2),
            fma(0.5, 3.0 * a1 - a2, div_by<3>(P.beta * m1)), kl, kh);
  const long long lo = S::key(S::val(kl) - w), hi = S::key(S::val(kh) - w);
  return w + S::val(S::mx(S::mn(lo, hi), S::mn(S::mx(lo, hi), S::key(0.0))));
}

// The two states of the edge EMF's reconstructions.
template <int RECON>
__device__ __forceinline__ void weno_edge(double fm3, double fm2, double fm1, double f0, double fp1, double fp2,
                                          const Prm<double>& P, double& fl, double& fr) {
  fl = weno_side_ref<RECON>(fm3, fm2, fm1, f0, fp1, P);
  fr = weno_side_ref<RECON>(fp2, fp1, f0, fm1, fm2, P);
}
template <int RECON, typename V>
__device__ __forceinline__ void weno_edge(V fm3, V fm2, V fm1, V f0, V fp1, V fp2, const Prm<float>& P, V& fl, V& fr) {
  weno_both<RECON>(fm3, fm2, fm1, f0, fp1, fp2, P, fl, fr);
}

// One-sided face states of f at the low face of element c along stride s
// (reconstruct_3d for dirs 1-3, mhd3d3.f90:833-860).
// PDM face states from the 8 taps a0..a7 (cells c-4 .. c+3 along the
// reconstruction axis; the face at the low side of c).
constexpr bool is_weno(int recon) { return recon == R_WENO || recon == R_MPWENO; }
constexpr bool is_pdm(int recon) { return recon == R_PDM || recon == R_PDMG; }
// EDGE: the face-B reconstruction of the edge EMF.
template <typename T, int RECON = R_PDM, bool EDGE = false>
__device__ __forceinline__ void recon_pdm8(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7, T pdmb, T& fl, T& fr) {
  if constexpr (RECON == R_PDM && std::is_same<T, double>::value && !EDGE) {
    pdm_states_fused(a2, a3, a4, a5, tap8_fused(a0, a1, a2, a3, a4, a5, a6, a7), pdmb, fl, fr, a3);
  } else {
    const T fi = tap8(a0, a1, a2, a3, a4, a5, a6, a7);
    if constexpr (RECON != R_PDM) pdm2(a2, a3, a4, a5, fi, pdmb, fl, fr);
    else if constexpr (std::is_same<T, double>::value) Edge64::states(a2, a3, a4, a5, fi, pdmb, fl, fr);
    else pdm_states(a2, a3, a4, a5, fi, pdmb, fl, fr, a3);
  }
}

template <typename T, int RECON, typename I, bool EDGE = false>
__device__ __forceinline__ void recon_face(const T* __restrict__ f, I c, I s, const Prm<T>& P, T& fl, T& fr) {
  if (is_pdm(RECON)) {
    recon_pdm8<T, RECON, EDGE>(f[c - 4 * s], f[c - 3 * s], f[c - 2 * s], f[c - s], f[c], f[c + s], f[c + 2 * s],
                         f[c + 3 * s], P.pdmb, fl, fr);
  } else if (RECON == R_TVD || RECON == R_TVDMC) {
    T fm2 = f[c - 2 * s], fm1 = f[c - s], f0 = f[c], fp1 = f[c + s];
    T fi = (fm1 + f0) / T(2);
    tvd<T, RECON == R_TVDMC>(fm2, fm1, f0, fp1, fi, P.eps, fl, fr);
  } else {
    T fm3 = f[c - 3 * s], fm2 = f[c - 2 * s], fm1 = f[c - s], f0 = f[c], fp1 = f[c + s], fp2 = f[c + 2 * s];
    if constexpr (EDGE) weno_edge<RECON>(fm3, fm2, fm1, f0, fp1, fp2, P, fl, fr);
    else weno_both<RECON>(fm3, fm2, fm1, f0, fp1, fp2, P, fl, fr);
  }
}

// recon_face of the face B in the edge EMF.
template <typename T, int RECON, typename I>
__device__ __forceinline__ void recon_edge(const T* __restrict__ f, I c, I s, const Prm<T>& P, T& fl, T& fr) {
  recon_face<T, RECON, I, true>(f, c, s, P, fl, fr);
}

// PDM part of get_vav_center2corner (mhd3d3.f90:1901-1905, 2056-2108) for
// an edge with upper cell c and transverse axes d1, d2, given the corner
// interpolant vi.  The reference limits vi with four shifted PDM2 pairs, which
// leaves each quadrant cell q two one-sided estimates, one along d1 and one
// along d2, and takes the one whose outward slope is larger (dif >= 0: d1).
// An estimate is PDM2's state on the side of q: vi clamped to [q, far] and kept
// within [q, q + D(q, outer)], far the cell across the edge and outer the one
// behind q along that axis.  The comparison of the two slopes picks (far, q -
// outer) and one state per quadrant is evaluated, by the same instructions on
// either side.  The edge takes the mean of the four.
__device__ __forceinline__ float corner_quad(float q, float far1, float far2, float e1, float e2, float pd, float vi) {
  const bool b = abs_ge(e1, e2);  // q - outer along d1 and d2
  const float x = clamp2(q, b ? far1 : far2, vi), d = x - q;
  return x - (d - shrink(d, (pd + pd) * (b ? e1 : e2)));
}
__device__ __forceinline__ double corner_quad(double q, double far1, double far2, double e1, double e2, double pd,
                                              double vi) {
  typedef Sel<double> S;
  const bool b = abs_ge(e1, e2);
  const S::K c = S::key(q), f = S::key(b ? far1 : far2);
  return Edge64::limited(q, Edge64::clamp(c, f, S::interp(vi)), pd * (b ? e1 : e2), f > c);
}
// The reference's form, for any pdmb (R_PDMG): one half of pdm2 with the clamp
// pair (lo, hi) = (fm1, f0), the cell `outer` beyond the near end and the side
// (left: near = fm1, outer = fm2; right: near = f0, outer = fp1).
template <typename T>
__device__ __forceinline__ T pdm_half(T lo, T hi, T outer, bool left, T fi, T pdmb) {
  const T fii = mx(mn(lo, hi), mn(fi, mx(lo, hi)));
  const T near = left ? lo : hi;
  const T dn = pdmb * (left ? (lo - outer) : (outer - hi));  // pdm2's dfm / dfp
  const T s0 = sgn1(pdmb * (hi - lo));
  const T q = fab(sgn1(dn) + s0);
  const T x = s0 * mx(T(0), fab(near - fii) - q * fab(dn));
  return left ? fii - x : fii + x;
}

// The 12 cells an edge reads, named by (offset along d1, offset along d2)
// from the upper cell: mAB = (-A, -B), pAB = (+A, -B) etc.; quadrant cells
// m11, m01, m10, c0.
template <typename T, int RECON = R_PDM>
__device__ __forceinline__ T corner_pdm_vals(T m11, T m21, T m12, T m01, T p11, T m02, T m10, T m20, T m1p, T c0,
                                             T p10, T p01, T vi, T pd) {
  if (RECON == R_PDM) {
    const T v00 = corner_quad(m11, m01, m10, m11 - m21, m11 - m12, pd, vi);
    const T v10 = corner_quad(m01, m11, c0, m01 - p11, m01 - m02, pd, vi);
    const T v01 = corner_quad(m10, c0, m11, m10 - m20, m10 - m1p, pd, vi);
    const T v11 = corner_quad(c0, m10, m01, c0 - p10, c0 - p01, pd, vi);
    return T(0.25) * (v00 + v01 + v10 + v11);
  }
  const T d00 = fab(m21 - m11) - fab(m12 - m11);
  const T d10 = fab(p11 - m01) - fab(m02 - m01);
  const T d01 = fab(m20 - m10) - fab(m1p - m10);
  const T d11 = fab(p10 - c0) - fab(p01 - c0);
  const bool b00 = d00 >= T(0), b10 = d10 >= T(0), b01 = d01 >= T(0), b11 = d11 >= T(0);
  const T v00 = pdm_half(m11, b00 ? m01 : m10, b00 ? m21 : m12, true, vi, pd);
  const T v10 = pdm_half(b10 ? m11 : m01, b10 ? m01 : c0, b10 ? p11 : m02, !b10, vi, pd);
  const T v01 = pdm_half(b01 ? m10 : m11, b01 ? c0 : m10, b01 ? m20 : m1p, b01, vi, pd);
  const T v11 = pdm_half(b11 ? m10 : m01, c0, b11 ? p10 : p01, false, vi, pd);
  return T(0.25) * (v00 + v01 + v10 + v11);
}

template <typename T, int RECON, typename I>
__device__ __forceinline__ T corner_pdm(const T* __restrict__ v, I c, I s1, I s2, T vi, T pd) {
  return corner_pdm_vals<T, RECON>(v[c - s1 - s2], v[c - 2 * s1 - s2], v[c - s1 - 2 * s2], v[c - s2],
                                   v[c + s1 - s2], v[c - 2 * s2], v[c - s1], v[c - 2 * s1], v[c - s1 + s2], v[c],
                                   v[c + s1], v[c + s2], vi, pd);
}

// Two values carried together (the v_a1 and v_a2 components of an edge): one
// 8-byte (FP32) or 16-byte (FP64) shared-memory access per pair, and FP32
// pair arithmetic on the packed FMA / MUL pipes (each lane rounds as the
// scalar fma / mul does); FP64 stays scalar, with separate mul and add as
// the reference writes them.
template <typename T> struct Pr;
template <> struct Pr<float> {
  typedef float2 V;
  static __device__ __forceinline__ V mk(float a, float b) { return make_float2(a, b); }
  static __device__ __forceinline__ V mul(float k, V a) { return __fmul2_rn(make_float2(k, k), a); }
  static __device__ __forceinline__ V mad(float k, V a, V c) { return __ffma2_rn(make_float2(k, k), a, c); }  // c + k a
  static __device__ __forceinline__ V sub(V a, V b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }  // one rounding
};
template <> struct Pr<double> {
  typedef double2 V;
  static __device__ __forceinline__ V mk(double a, double b) { return make_double2(a, b); }
  static __device__ __forceinline__ V mul(double k, V a) { return make_double2(k * a.x, k * a.y); }
  static __device__ __forceinline__ V mad(double k, V a, V c) { return make_double2(fma(k, a.x, c.x), fma(k, a.y, c.y)); }
  static __device__ __forceinline__ V sub(V a, V b) { return make_double2(a.x - b.x, a.y - b.y); }
};

// tap8 on pairs (same operations per lane)
__device__ __forceinline__ float2 tap8p(float2 a0, float2 a1, float2 a2, float2 a3, float2 a4, float2 a5, float2 a6,
                                        float2 a7) {
  typedef Pr<float> Q;
  float2 s = Q::mad(29.0f, a1, Q::mul(-3.0f, a0));
  s = Q::mad(533.0f, a3, Q::mad(-139.0f, a2, s));
  s = Q::mad(-139.0f, a5, Q::mad(533.0f, a4, s));
  s = Q::mad(-3.0f, a7, Q::mad(29.0f, a6, s));
  return Q::mul(1.0f / 840.0f, s);
}
__device__ __forceinline__ double2 tap8p(double2 a0, double2 a1, double2 a2, double2 a3, double2 a4, double2 a5,
                                         double2 a6, double2 a7) {
  return make_double2(tap8(a0.x, a1.x, a2.x, a3.x, a4.x, a5.x, a6.x, a7.x),
                      tap8(a0.y, a1.y, a2.y, a3.y, a4.y, a5.y, a6.y, a7.y));
}

// corner_quad of both components of a pair.  FP32: the differences on the
// packed pipe, the choice, the clamp and the threshold per lane.
__device__ __forceinline__ float2 corner_quad2(float2 q, float2 far1, float2 far2, float2 out1, float2 out2, float pd,
                                               float2 vi) {
  typedef Pr<float> Q;
  const float2 e1 = Q::sub(q, out1), e2 = Q::sub(q, out2);
  const bool bx = abs_ge(e1.x, e2.x), by = abs_ge(e1.y, e2.y);
  const float2 D = Q::mul(pd + pd, make_float2(bx ? e1.x : e2.x, by ? e1.y : e2.y));
  const float2 x = make_float2(clamp2(q.x, bx ? far1.x : far2.x, vi.x), clamp2(q.y, by ? far1.y : far2.y, vi.y));
  const float2 d = Q::sub(x, q);
  return Q::sub(x, Q::sub(d, make_float2(shrink(d.x, D.x), shrink(d.y, D.y))));
}
__device__ __forceinline__ double2 corner_quad2(double2 q, double2 far1, double2 far2, double2 out1, double2 out2,
                                                double pd, double2 vi) {
  return make_double2(corner_quad(q.x, far1.x, far2.x, q.x - out1.x, q.x - out2.x, pd, vi.x),
                      corner_quad(q.y, far1.y, far2.y, q.y - out1.y, q.y - out2.y, pd, vi.y));
}
// corner_pdm_vals of both components.
template <typename T, int RECON>
__device__ __forceinline__ void corner_pdm_vals2(
    typename Pr<T>::V m11, typename Pr<T>::V m21, typename Pr<T>::V m12, typename Pr<T>::V m01, typename Pr<T>::V p11,
    typename Pr<T>::V m02, typename Pr<T>::V m10, typename Pr<T>::V m20, typename Pr<T>::V m1p, typename Pr<T>::V c0,
    typename Pr<T>::V p10, typename Pr<T>::V p01, typename Pr<T>::V vi, T pd, T& r0, T& r1) {
  if constexpr (RECON != R_PDM) {
    r0 = corner_pdm_vals<T, RECON>(m11.x, m21.x, m12.x, m01.x, p11.x, m02.x, m10.x, m20.x, m1p.x, c0.x, p10.x, p01.x,
                                   vi.x, pd);
    r1 = corner_pdm_vals<T, RECON>(m11.y, m21.y, m12.y, m01.y, p11.y, m02.y, m10.y, m20.y, m1p.y, c0.y, p10.y, p01.y,
                                   vi.y, pd);
    return;
  }
  typedef typename Pr<T>::V V;
  const V v00 = corner_quad2(m11, m01, m10, m21, m12, pd, vi);
  const V v10 = corner_quad2(m01, m11, c0, p11, m02, pd, vi);
  const V v01 = corner_quad2(m10, c0, m11, m20, m1p, pd, vi);
  const V v11 = corner_quad2(c0, m10, m01, p10, p01, pd, vi);
  r0 = T(0.25) * (v00.x + v01.x + v10.x + v11.x);
  r1 = T(0.25) * (v00.y + v01.y + v10.y + v11.y);
}

// Compile-time knob: MHD_RECON_PACKED = 0 keeps the FP32 reconstruction scalar.
#ifndef MHD_RECON_PACKED
#define MHD_RECON_PACKED 1
#endif
namespace p2 {
__device__ __forceinline__ float2 K(float c) { return make_float2(c, c); }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return __ffma2_rn(b, K(-1.0f), a); }  // a - b, one rounding
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// 1/x, 1/sqrt(x) and exp(-x) on the SFU alone: the .ftz forms, which drop the
// rescaling of subnormal operands and results around each (two to three
// instructions; a face takes 18 of these).  Same bits for normal numbers; a
// tail of erfc or exp below 1.2e-38 is zero, and an operand below it counts as zero: the
// reciprocals and roots of lam check for that (lam_roots).
__device__ __forceinline__ float rcp1(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsq1(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// the same with subnormal operands
__device__ __forceinline__ float rcp1s(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsq1s(float x) {
  float r;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ex21(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 rcp(float2 a) { return make_float2(rcp1(a.x), rcp1(a.y)); }
__device__ __forceinline__ float2 rsq(float2 a) { return make_float2(rsq1(a.x), rsq1(a.y)); }
// lam = r / q, ra = 1 / sqrt(lam), a = sqrt(lam) of two values of each of two q.  a ra is one,
// to a few roundings, unless an operand was flushed (or lam is zero, infinite or NaN):
// the forms with the rescaling decide then.  The check takes five instructions on the FMA
// pipe, which has room, where the rescaling of eight operands takes about 20 on any.
__device__ __forceinline__ void lam_roots(float2 r, float2 q, float2 qm, float2& lam, float2& ra, float2& a, float2& am) {
  lam = mul(r, rcp(q));
  ra = rsq(lam);
  a = mul(lam, ra);
  float2 lm = mul(r, rcp(qm)), rm = rsq(lm);
  am = mul(lm, rm);
  const float2 one = mul(mul(a, ra), mul(am, rm));
  if (!(one.x * one.y < 2.0f)) {
    lam = mul(r, make_float2(rcp1s(q.x), rcp1s(q.y)));
    ra = make_float2(rsq1s(lam.x), rsq1s(lam.y));
    a = mul(lam, ra);
    lm = mul(r, make_float2(rcp1s(qm.x), rcp1s(qm.y)));
    am = mul(lm, make_float2(rsq1s(lm.x), rsq1s(lm.y)));
  }
}
__device__ __forceinline__ float2 exp_neg(float2 a) {
  a = mul(a, K(-1.4426950408889634f));
  return make_float2(ex21(a.x), ex21(a.y));
}
}  // namespace p2

// corner_pdm of both components from pair-interleaved shared memory.
template <typename T, int RECON>
__device__ __forceinline__ void corner_pdm_pair(const typename Pr<T>::V* __restrict__ v, int c, int s1, int s2,
                                                typename Pr<T>::V vi, T pd, T& r0, T& r1) {
  typedef typename Pr<T>::V V;
  const V m11 = v[c - s1 - s2], m21 = v[c - 2 * s1 - s2], m12 = v[c - s1 - 2 * s2], m01 = v[c - s2];
  const V p11 = v[c + s1 - s2], m02 = v[c - 2 * s2], m10 = v[c - s1], m20 = v[c - 2 * s1];
  const V m1p = v[c - s1 + s2], c0 = v[c], p10 = v[c + s1], p01 = v[c + s2];
  corner_pdm_vals2<T, RECON>(m11, m21, m12, m01, p11, m02, m10, m20, m1p, c0, p10, p01, vi, pd, r0, r1);
}

// Limited corner value of v at the edge whose two transverse axes have
// strides s1 (d1) and s2 (d2) and whose upper cell is c
// (get_vav_center2corner, mhd3d3.f90:1858-2116).  Quadrant cell q_ab =
// c - (1-a) s1 - (1-b) s2; v_ab_0 / v_ab_1 are the two one-sided estimates.
template <typename T, int RECON>
__device__ __forceinline__ T corner_vel(const T* __restrict__ v, long long c, long long s1, long long s2,
                                        const Prm<T>& P) {
  T v00_0, v00_1, v10_0, v10_1, v01_0, v01_1, v11_0, v11_1;
  if (is_pdm(RECON)) {
    // interp2_pdm (926-989): 8-tap along d1 at the 8 d2-rows, then along d2
    T g[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const T* r = v + c + (long long)(m - 4) * s2;
      g[m] = tap8(r[-4 * s1], r[-3 * s1], r[-2 * s1], r[-s1], r[0], r[s1], r[2 * s1], r[3 * s1]);
    }
    T vi = tap8(g[0], g[1], g[2], g[3], g[4], g[5], g[6], g[7]);
    return corner_pdm<T, RECON>(v, c, s1, s2, vi, P.pdmb);
  } else if (RECON == R_TVD || RECON == R_TVDMC) {
    // interp2_tvd (1037-1067) and TVD with (mhd3d2) or without (mhd3d3) shifts
    constexpr bool MC = (RECON == R_TVDMC);
    T vi = (v[c - s1 - s2] + v[c - s2] + v[c] + v[c - s1]) / T(4);
    long long a = P.tvd_shift ? c - s2 : c;
    long long b = P.tvd_shift ? c - s1 : c;
    tvd<T, MC>(v[a - 2 * s1], v[a - s1], v[a], v[a + s1], vi, P.eps, v00_0, v10_0);
    tvd<T, MC>(v[b - 2 * s2], v[b - s2], v[b], v[b + s2], vi, P.eps, v00_1, v01_1);
    tvd<T, MC>(v[c - 2 * s2], v[c - s2], v[c], v[c + s2], vi, P.eps, v10_1, v11_1);
    tvd<T, MC>(v[c - 2 * s1], v[c - s1], v[c], v[c + s1], vi, P.eps, v01_0, v11_0);
  } else {
    // WENO5 / MPWENO5 two-level reconstruction (1925-2049): "_1" = along d1
    // then d2, "_0" = along d2 then d1, with the reference's output naming.
    T L[6], R[6], a[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const T* r = v + c + (long long)(m - 3) * s2;
#pragma unroll
      for (int t = 0; t < 6; ++t) a[t] = r[(long long)(t - 3) * s1];
      weno_edge<RECON>(a[0], a[1], a[2], a[3], a[4], a[5], P, L[m], R[m]);
    }
    weno_edge<RECON>(L[0], L[1], L[2], L[3], L[4], L[5], P, v00_1, v01_1);
    weno_edge<RECON>(R[0], R[1], R[2], R[3], R[4], R[5], P, v10_1, v11_1);
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const T* r = v + c + (long long)(m - 3) * s1;
#pragma unroll
      for (int t = 0; t < 6; ++t) a[t] = r[(long long)(t - 3) * s2];
      weno_edge<RECON>(a[0], a[1], a[2], a[3], a[4], a[5], P, L[m], R[m]);
    }
    weno_edge<RECON>(L[0], L[1], L[2], L[3], L[4], L[5], P, v00_0, v01_0);
    weno_edge<RECON>(R[0], R[1], R[2], R[3], R[4], R[5], P, v10_0, v11_0);
  }
  // dif signs pick the smoother one-sided estimate per quadrant (2056-2106)
  const long long q00 = c - s1 - s2, q10 = c - s2, q01 = c - s1, q11 = c;
  T d00 = fab(v[q00 - s1] - v[q00]) - fab(v[q00 - s2] - v[q00]);
  T d10 = fab(v[q10 + s1] - v[q10]) - fab(v[q10 - s2] - v[q10]);
  T d01 = fab(v[q01 - s1] - v[q01]) - fab(v[q01 + s2] - v[q01]);
  T d11 = fab(v[q11 + s1] - v[q11]) - fab(v[q11 + s2] - v[q11]);
  T v00 = d00 >= T(0) ? v00_0 : v00_1;
  T v10 = d10 >= T(0) ? v10_0 : v10_1;
  T v01 = d01 >= T(0) ? v01_0 : v01_1;
  T v11 = d11 >= T(0) ? v11_0 : v11_1;
  return T(0.25) * (v00 + v01 + v10 + v11);
}

// The current state as a stage input (RK stages of a batch read their own grid's state).
template <typename T>
__device__ __forceinline__ Inp<T> state_view(const Dev<T>& d) {
  return Inp<T>{d.rho, d.vx, d.vy, d.vz, d.p, d.bx, d.by, d.bz, d.bi, d.bj, d.bk};
}

// ------------------------------------------------------------ kernel args
// Argument of the step kernels that also run batched over an ensemble.
// B = false: one grid, its Dev by value, block index from blockIdx.
// B = true: many grids in one flattened 1-D launch; block b takes its grid
// and block coordinates from map[b] = {grid, bx, by, bz} and its Dev from
// tab[grid], read in place: a copy held the array pointers in registers (x faces
// 56 instead of 40, CT + bxyz 180 bytes spilled under its budget; a stage of 32
// grids 2720 -> 2583 us).
template <typename T, bool B> struct KArg;
template <typename T> struct KArg<T, false> {
  Dev<T> d;
  __device__ __forceinline__ int4 blk() const {
    return make_int4(0, (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z);
  }
  __device__ __forceinline__ const Dev<T>& dev(const int4&) const { return d; }
};
template <typename T> struct KArg<T, true> {
  const Dev<T>* __restrict__ tab;
  const int4* __restrict__ map;
  __device__ __forceinline__ int4 blk() const { return map[blockIdx.x]; }
  __device__ __forceinline__ const Dev<T>& dev(const int4& b) const { return tab[b.x]; }
};
template <typename T>
inline KArg<T, false> one(const Dev<T>& d) { return KArg<T, false>{d}; }

// Resident 256-thread blocks per SM requested for the cell passes (CFL, CT +
// bxyz, fill).  Single grid: none (0; they take 32 registers).  Batched: a
// budget of 40, since these passes wait on memory and live on residency.
#ifndef MHD_BATCH_MINB
#define MHD_BATCH_MINB 6
#endif
constexpr int pass_min_blocks(bool B) { return B ? MHD_BATCH_MINB : 0; }

// ------------------------------------------------------------- small kernels
// dt of the current step in T (FP32: the copy select_tau rounds once; a
// conversion per thread ran on the FP64 pipe, 16 cycles a warp).
template <typename T>
__device__ __forceinline__ T step_tau(const Scal* sc) {
  if constexpr (std::is_same<T, float>::value) return sc->tauf;
  else return sc->tau;
}

template <typename T>
__device__ __forceinline__ long long idx3(const Geom& g, int i, int j, int k) {
  return (long long)i + (long long)g.px * ((long long)j + (long long)g.py * (long long)k);
}

// Metric-mode cell B from the face fluxes of cell c (low / high faces):
// B = sum_a (Phi_a averaged over the two a-faces / V) e_a, e_a the cell's
// edge vector along a (the oracle's get_bxyz_metric, in its operand order).
template <typename T>
__device__ __forceinline__ void cell_b_metric(const Metric<T>& m, long long c, T lo0, T hi0, T lo1, T hi1, T lo2,
                                              T hi2, T& bx, T& by, T& bz) {
  const T V = m.vol[c], rV = m.rvol[c];
  const T p0 = Ops<T>::dw(T(0.5) * (hi0 + lo0), V, rV);
  const T p1 = Ops<T>::dw(T(0.5) * (hi1 + lo1), V, rV);
  const T p2 = Ops<T>::dw(T(0.5) * (hi2 + lo2), V, rV);
  bx = p0 * m.eb[0][0][c] + p1 * m.eb[1][0][c] + p2 * m.eb[2][0][c];
  by = p0 * m.eb[0][1][c] + p1 * m.eb[1][1][c] + p2 * m.eb[2][1][c];
  bz = p0 * m.eb[0][2][c] + p1 * m.eb[1][2][c] + p2 * m.eb[2][2][c];
}

// vf = |v| + |B| / sqrt(rho) of get_eijk_LFM (1766), b2 = |B|^2 (in FP64 with
// the reference's roundings: the edge EMF multiplies the jumps of B by it).
// FP32: the contraction spelled out, so that every kernel that fills vf gives the same bits.
__device__ __forceinline__ float sq3(float a, float b, float c) { return fmaf(c, c, fmaf(a, a, __fmul_rn(b, b))); }
__device__ __forceinline__ double sq3(double a, double b, double c) { return a * a + b * b + c * c; }
template <typename T>
__device__ __forceinline__ T vf_val(T u, T v, T w, T b2, T r0) {
  return sq(sq3(u, v, w)) + sq(b2 / r0);
}
// get_bxyz over all cells (incl. ghosts) and vf = |v| + |B|/sqrt(rho).
template <typename T, bool M>
__global__ void k_bxyz_vf(Dev<T> d, int want_vf) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  int k = blockIdx.z;
  const Geom& g = d.g;
  if (i >= g.nx || j >= g.ny || k >= g.nz) return;
  long long c = idx3<T>(g, i, j, k);
  T bx, by, bz;
  if (M) {
    cell_b_metric<T>(d.m, c, d.bi[c], d.bi[c + 1], d.bj[c], d.bj[c + g.px], d.bk[c], d.bk[c + g.plane], bx, by, bz);
  } else {
    bx = T(0.5) * (d.bi[c + 1] + d.bi[c]);
    by = T(0.5) * (d.bj[c + g.px] + d.bj[c]);
    bz = T(0.5) * (d.bk[c + g.plane] + d.bk[c]);
  }
  d.bx[c] = bx;
  d.by[c] = by;
  d.bz[c] = bz;
  if (want_vf) {
    T u = d.vx[c], v = d.vy[c], w = d.vz[c];
    d.vf[c] = vf_val(u, v, w, sq3(bx, by, bz), d.rho[c]);
  }
}

// get_dt over all cells incl. ghosts: per-block min, then atomicMin on the
// bit pattern (positive doubles order like their bits).  Status bits mirror
// diag_rho_neg / diag_overflow.
// Fast square root for the FP32 CFL estimate; exact in FP64.
__device__ __forceinline__ double cfl_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float cfl_sqrt(float x) { return x > 0.0f ? x * rsqrtf(x) : 0.0f; }

// |v| + fast speed sqrt(B^2 / rho + gam p / rho); FP64 takes one root and one
// reciprocal for the second term (three roots and two divisions as written in get_dt) of a
// cell with p >= 0 and a positive rho whose reciprocal is a normal number.  In any other
// cell the three roots decide what is NaN, and with it out of the minimum.
template <bool M>
__device__ __forceinline__ float cfl_speed(float gam, float r0, float p0, float u, float v, float w, float b2) {
  typedef Ops<float> O;
  const float vv = cfl_sqrt(sq3(u, v, w));
  const float valf = O::dv(cfl_sqrt(b2), cfl_sqrt(r0));
  const float vs = cfl_sqrt(O::dv(gam * p0, r0));
  return vv + cfl_sqrt(valf * valf + vs * vs);
}
template <bool M>
__device__ __forceinline__ double cfl_speed(double gam, double r0, double p0, double u, double v, double w, double b2) {
  if (M || !ge0(p0) || (unsigned)__double2hiint(r0) - 0x00200000u >= 0x7fc00000u - 0x00200000u) {
    const double valf = sqrt(b2) / sqrt(r0), vs = sqrt(gam * p0 / r0);
    return sqrt(u * u + v * v + w * w) + sqrt(valf * valf + vs * vs);
  }
  return sqrt(u * u + v * v + w * w) + sqrt((b2 + gam * p0) * (1.0 / r0));
}

// get_dt of one cell (mhd3d3.f90:1608-1639) from its primitives and cell B,
// with the status bits of its values.
template <typename T, bool M>
__device__ __forceinline__ T cell_dt(const Dev<T>& d, int c, int i, int j, int k, T r0, T p0, T u, T v, T w, T a,
                                     T b, T cc, unsigned& st) {
  typedef Ops<T> O;
  const T vcfl = cfl_speed<M>(d.gam, r0, p0, u, v, w, sq3(a, b, cc));
  T dt;
  if (M)  // metric mode: 1/dx_a -> |mean area vector of the a-faces| / V
    dt = O::dv(d.cfl, O::dw(vcfl * d.m.sa[c], d.m.vol[c], d.m.rvol[c]));
  else
    dt = O::dv(d.cfl, O::dc(vcfl, d.wx[i], d.rwx[i]) + O::dc(vcfl, d.wy[j], d.rwy[j]) +
                          O::dc(vcfl, d.wz[k], d.rwz[k]));
  if (isnan(r0) || isnan(p0) || isnan(u) || isnan(v) || isnan(w)) st |= ST_NAN;
  if (r0 < T(0)) st |= ST_NEG_RHO;
  if (p0 < T(0)) st |= ST_NEG_P;
  if (isnan(dt)) st |= ST_NAN;
  return dt;
}

// Fold a thread's (dt, status) into the accumulators of the next step's
// state: block minimum (warp shuffles, then shared memory), then one atomic
// per block that lowers the running minimum (a plain read first skips the
// rest).  Every thread of the 256-thread block calls it.
template <typename T>
__device__ __forceinline__ void dt_next_accumulate(Scal* sc, T m, unsigned st) {
  for (int o = 16; o > 0; o >>= 1) {
    T y = __shfl_xor_sync(0xffffffffu, m, o);
    m = (y < m) ? y : m;
    st |= __shfl_xor_sync(0xffffffffu, st, o);
  }
  __shared__ T bm[8];
  __shared__ unsigned bs[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { bm[wid] = m; bs[wid] = st; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      m = (bm[w] < m) ? bm[w] : m;
      st |= bs[w];
    }
    const double md = (double)m;
    if (md >= 0.0) {
      const unsigned long long bits = (unsigned long long)__double_as_longlong(md);
      if (bits < *(volatile unsigned long long*)&sc->dtnext_bits) atomicMin(&sc->dtnext_bits, bits);
    }
    if (st) atomicOr(&sc->pend_status, st);
  }
}

// p / (gam - 1): FP64 by the reciprocal (Dev::rgm1), the metric mode divides.
template <bool M>
__device__ __forceinline__ float over_gm1(const Dev<float>& d, float p) { return Ops<float>::dv(p, d.gam - 1.0f); }
template <bool M>
__device__ __forceinline__ double over_gm1(const Dev<double>& d, double p) { return M ? p / (d.gam - 1.0) : p * d.rgm1; }

// save != 0 also stores U^n of the RK stage combines (advance_previous,
// 3794-3819) at interior cells and faces, the only places they are read.
// next != 0: the dt and status go to the next-step accumulators.
// The minimum is reduced in T and converted to FP64 once per block.
template <typename T, bool M, bool B>
__global__ void __launch_bounds__(256, pass_min_blocks(B)) k_cfl(KArg<T, B> ka, int save, int next) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Geom& g = d.g;
  T m = T(INFINITY);
  unsigned st = 0;
  const int i = bb.y * 32 + (threadIdx.x & 31);
  const int j = bb.z * 8 + (threadIdx.x >> 5);
  const int k1 = min(g.nz, (bb.w + 1) * 8);
  for (int k = bb.w * 8; k < k1; ++k) {
    if (i >= g.nx || j >= g.ny) break;
    const int c = i + g.px * (j + g.py * k);
    T r0 = d.rho[c], p0 = d.p[c], u = d.vx[c], v = d.vy[c], w = d.vz[c];
    if (save) {
      const bool ix = i >= g.ng && i < g.ng + g.nx0, iy = j >= g.ng && j < g.ng + g.ny0,
                 iz = k >= g.ng && k < g.ng + g.nz0;
      if (ix && iy && iz) {
        d.q[0][c] = r0;
        d.q[1][c] = r0 * u;
        d.q[2][c] = r0 * v;
        d.q[3][c] = r0 * w;
        d.q[4][c] = T(0.5) * r0 * (u * u + v * v + w * w) + over_gm1<M>(d, p0);
      }
      const bool fx = i >= g.ng && i <= g.ng + g.nx0, fy = j >= g.ng && j <= g.ng + g.ny0,
                 fz = k >= g.ng && k <= g.ng + g.nz0;
      if (fx && iy && iz) d.q[5][c] = d.bi[c];
      if (ix && fy && iz) d.q[6][c] = d.bj[c];
      if (ix && iy && fz) d.q[7][c] = d.bk[c];
    }
    const T dt = cell_dt<T, M>(d, c, i, j, k, r0, p0, u, v, w, d.bx[c], d.by[c], d.bz[c], st);
    m = (dt < m) ? dt : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    T y = __shfl_xor_sync(0xffffffffu, m, o);
    m = (y < m) ? y : m;
    st |= __shfl_xor_sync(0xffffffffu, st, o);
  }
  __shared__ T sm[8];
  __shared__ unsigned ss[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { sm[wid] = m; ss[wid] = st; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w2 = 1; w2 < 8; ++w2) {
      m = (sm[w2] < m) ? sm[w2] : m;
      st |= ss[w2];
    }
    const double md = (double)m;
    if (md >= 0.0) atomicMin(next ? &d.sc->dtnext_bits : &d.sc->dtmin_bits, (unsigned long long)__double_as_longlong(md));
    if (st) atomicOr(next ? &d.sc->pend_status : &d.sc->status, st);
  }
}

// Empties the next-step accumulators before a dt pass refills them.
__device__ __forceinline__ void next_reset(Scal* sc) {
  sc->dtnext_bits = (unsigned long long)__double_as_longlong(INFINITY);
  sc->pend_status = 0;
}
__global__ inline void k_next_reset(Scal* sc) { next_reset(sc); }

// tau selection of step_ab (3609) / step_rk2,3 (3656-3661, 3723-3728).
// mode 0: RK with fixed deck dt; 1: CFL dt every step; 2: AB (CFL dt and the
// predictor coefficient tau/tau0/2, then tau0=tau).
// mode | 4: take the dt and status accumulated for this state by the
// previous step (dtnext_bits, pend_status) and empty them.
__device__ __forceinline__ void select_tau(Scal* s, int mode) {
  double dt;
  if (mode & 4) {
    dt = __longlong_as_double((long long)s->dtnext_bits);
    s->dtnext_bits = (unsigned long long)__double_as_longlong(INFINITY);
    s->status |= s->pend_status;
    s->pend_status = 0;
    mode &= 3;
  } else {
    dt = __longlong_as_double((long long)s->dtmin_bits);
    s->dtmin_bits = (unsigned long long)__double_as_longlong(INFINITY);
  }
  s->dt_cfl = dt;
  if (mode == 0) {
    if (dt < s->tau0) s->status |= ST_CFL;
    s->tau = s->tau0;
  } else if (mode == 1) {
    s->tau = dt;
    s->tau0 = dt;
  } else if (mode == 2) {
    s->tau = dt;
    s->ab_coef = dt / s->tau0 / 2.0;
    s->tau0 = dt;
  }
  // mode 3: read-only (diagnostics); tau untouched
  s->tauf = (float)s->tau;
}
template <typename T>
__global__ void k_cfl_final(Dev<T> d, int mode) { select_tau(d.sc, mode); }

// The same for every grid of a batch, one thread per grid.
template <typename T>
__global__ void k_next_reset_batch(const Dev<T>* __restrict__ tab, int ngrids) {
  const int gi = blockIdx.x * blockDim.x + threadIdx.x;
  if (gi < ngrids) next_reset(tab[gi].sc);
}
template <typename T>
__global__ void k_cfl_final_batch(const Dev<T>* __restrict__ tab, int ngrids, int mode) {
  const int gi = blockIdx.x * blockDim.x + threadIdx.x;
  if (gi < ngrids) select_tau(tab[gi].sc, mode);
}

// advance_predictor_ab (3821-3840): Xh = X + tau/tau0/2*(X-Xp), then Xp = X;
// also vf of the predicted state.
//
// 23 arrays read and 23 written: bytes bound it (0.87 GB at 160^3, 128 us).  A
// thread takes 16 bytes of every array, all of them loaded before the first store,
// and the padding of the rows is left out (a sixth at nx = 168).
// 160^3 FP32: 186 -> 143 us.
template <typename T> struct Vec16 {
  static constexpr int W = 16 / sizeof(T);
  uint4 u;
  __device__ __forceinline__ void load(const T* p) { u = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ T get(int i) const {
    if constexpr (sizeof(T) == 4) return __uint_as_float((&u.x)[i]);
    else return __hiloint2double((int)(&u.x)[2 * i + 1], (int)(&u.x)[2 * i]);
  }
  __device__ __forceinline__ void put(int i, T x) {
    if constexpr (sizeof(T) == 4) {
      (&u.x)[i] = __float_as_uint(x);
    } else {
      (&u.x)[2 * i] = (unsigned)__double2loint(x);
      (&u.x)[2 * i + 1] = (unsigned)__double2hiint(x);
    }
  }
  __device__ __forceinline__ void store(T* p) const { *reinterpret_cast<uint4*>(p) = u; }
};
template <typename T>
__global__ void __launch_bounds__(256, 2) k_predictor_ab(Dev<T> d) {
  typedef Vec16<T> V;
  const Geom& g = d.g;
  const int nq = (g.nx + V::W) / V::W, u = blockIdx.x * blockDim.x + threadIdx.x;  // x = 0 .. nx of a row
  if (u >= nq * g.py * g.pz) return;
  const int c = u / nq * g.px + u % nq * V::W;
  const T cf = (T)d.sc->ab_coef;
  const T* x[11] = {d.rho, d.vx, d.vy, d.vz, d.p, d.bi, d.bj, d.bk, d.bx, d.by, d.bz};
  V xv[11], xp[11], vf;
#pragma unroll
  for (int a = 0; a < 11; ++a) {
    xv[a].load(x[a] + c);
    xp[a].load(d.q[a] + c);
  }
#pragma unroll
  for (int i = 0; i < V::W; ++i) {
    T hv[11];
#pragma unroll
    for (int a = 0; a < 11; ++a) {
      hv[a] = xv[a].get(i) + cf * (xv[a].get(i) - xp[a].get(i));
      xp[a].put(i, hv[a]);
    }
    const T rr = hv[0];
    vf.put(i, (rr > T(0)) ? sq(hv[1] * hv[1] + hv[2] * hv[2] + hv[3] * hv[3]) +
                                sq((hv[8] * hv[8] + hv[9] * hv[9] + hv[10] * hv[10]) / rr)
                          : T(0));
  }
#pragma unroll
  for (int a = 0; a < 11; ++a) {
    xp[a].store(d.h[a] + c);
    xv[a].store(d.q[a] + c);
  }
  vf.store(d.vf + c);
}

// ------------------------------------------------------------------ fluxes
// Gaussian velocity moments of get_v_face (mhd3d3.f90:2594-2615):
//   a = sqrt(lam), b = .5 exp(-lam v^2)/a/sqrt(pi), v0+- = .5 erfc(-+a v),
//   v1+- = v v0+- +- b.
// FP64: CUDA's sqrt/exp/erfc in the reference's operand order (parity mode).
// FP32: erfc from the Chebyshev fit "erfcc" of Numerical Recipes (Press et
// al., 2nd ed., sec. 6.2; fractional error < 1.2e-7 for all arguments),
// rsqrt and exp2-based exp (the performance path).
template <typename T> struct Moments;
template <> struct Moments<double> {
  static __device__ __forceinline__ void hydro(double lam, double vn, bool left, double& v0, double& v1) {
    const double rspi = sqrt(3.14159265358979323846);
    double a = sqrt(lam);
    double b = 0.5 * exp(-lam * (vn * vn)) / a / rspi;
    if (left) {
      v0 = 0.5 * erfc(-a * vn);
      v1 = vn * v0 + b;
    } else {
      v0 = 0.5 * erfc(a * vn);
      v1 = vn * v0 - b;
    }
  }
  static __device__ __forceinline__ double mag(double lam, double vn, bool left) {
    double a = sqrt(lam);
    return left ? 0.5 * erfc(-a * vn) : 0.5 * erfc(a * vn);
  }
  static __device__ __forceinline__ double div(double a, double b) { return a / b; }
};
template <> struct Moments<float> {
  // erfc(z) for z >= 0 (Numerical Recipes erfcc)
  static __device__ __forceinline__ float erfc_pos(float z) {
    float t = p2::rcp1(fmaf(0.5f, z, 1.0f));
    float q = fmaf(t, 0.17087277f, -0.82215223f);
    q = fmaf(t, q, 1.48851587f);
    q = fmaf(t, q, -1.13520398f);
    q = fmaf(t, q, 0.27886807f);
    q = fmaf(t, q, -0.18628806f);
    q = fmaf(t, q, 0.09678418f);
    q = fmaf(t, q, 0.37409196f);
    q = fmaf(t, q, 1.00002368f);
    q = fmaf(t, q, -1.26551223f);
    return t * p2::ex21(1.4426950408889634f * fmaf(-z, z, q));
  }
  // 0.5 erfc(-s x) for the left (s=+1) or 0.5 erfc(x) for the right state
  static __device__ __forceinline__ float half_erfc(float x, bool left) {
    float h = 0.5f * erfc_pos(fabsf(x));
    bool direct = left ? (x <= 0.0f) : (x >= 0.0f);
    return direct ? h : 1.0f - h;
  }
  static __device__ __forceinline__ void hydro(float lam, float vn, bool left, float& v0, float& v1) {
    float ra = p2::rsq1s(lam);
    float a = lam * ra;
    v0 = half_erfc(a * vn, left);
    float b = (0.5f * 0.56418958354775628f) * ra * p2::ex21(1.4426950408889634f * (-lam * vn * vn));
    v1 = left ? fmaf(vn, v0, b) : fmaf(vn, v0, -b);
  }
  static __device__ __forceinline__ float mag(float lam, float vn, bool left) {
    float a = lam * p2::rsq1s(lam);
    return half_erfc(a * vn, left);
  }
  static __device__ __forceinline__ float div(float a, float b) { return a * p2::rcp1s(b); }
};

// ------------------------------------------------ FP32 packed-pair arithmetic
// Blackwell's packed FP32 instructions (FFMA2 / FMUL2 / FADD2) issue once for
// two lanes, each rounded as the scalar fma / mul / add.  The FP32 path
// evaluates the PDM face reconstruction on pairs of fields and the
// Gaussian-split flux on the (left, right) pair of a face with them; absolute
// values, min / max, signs and selects stay per lane, where the absolute
// values fold into the scalar instructions that use them.  Every FP32 face
// kernel (x faces, y / z face tiles and column sweeps, batched or not) goes
// through these functions, so they agree bit for bit.

// pdm2 of two fields (lanes .x and .y), for any pdmb: the differences on the
// packed pipe, the clamp and the limiter per lane.
__device__ __forceinline__ float2 pdm_general_lim(float fii, float dfl, float dfr, float dfm, float df0, float dfp) {
  const float sm = sgn1(dfm), s0 = sgn1(df0), sp = sgn1(dfp);
  const float qm = fabsf(sm + s0), qp = fabsf(s0 + sp);
  return make_float2(fii - s0 * mx(0.0f, fabsf(dfl) - qm * fabsf(dfm)),
                     fii + s0 * mx(0.0f, fabsf(dfr) - qp * fabsf(dfp)));
}
__device__ __forceinline__ void pdm_pair_general(float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fi, float pdmb,
                                                 float2& lr0, float2& lr1) {
  const float2 kp = p2::K(pdmb);
  const float2 dfm = p2::mul(kp, p2::sub(fm1, fm2));
  const float2 df0 = p2::mul(kp, p2::sub(f0, fm1));
  const float2 dfp = p2::mul(kp, p2::sub(fp1, f0));
  const float2 fii = make_float2(mx(mn(fm1.x, f0.x), mn(fi.x, mx(fm1.x, f0.x))),
                                 mx(mn(fm1.y, f0.y), mn(fi.y, mx(fm1.y, f0.y))));
  const float2 dfl = p2::sub(fii, fm1), dfr = p2::sub(f0, fii);
  lr0 = pdm_general_lim(fii.x, dfl.x, dfr.x, dfm.x, df0.x, dfp.x);
  lr1 = pdm_general_lim(fii.y, dfl.y, dfr.y, dfm.y, df0.y, dfp.y);
}

// PDM face states of two fields (lanes .x and .y) from their 8-tap windows (tap
// m = cell c+m-4 for the face at the low side of cell c): pdm_states with the
// differences on the packed pipe, the clamps and thresholds per lane.  lr0 /
// lr1 are the (left, right) states of lane x / lane y.
template <int RECON>
__device__ __forceinline__ void pdm_pair_states(const float2* a, float pdmb, float2& lr0, float2& lr1) {
  const float2 fi = tap8p(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
  if constexpr (RECON != R_PDM) return pdm_pair_general(a[2], a[3], a[4], a[5], fi, pdmb, lr0, lr1);
  const float2 fm2 = a[2], fm1 = a[3], f0 = a[4], fp1 = a[5], k = p2::K(pdmb + pdmb);
  const float2 Dl = p2::mul(k, p2::sub(fm1, fm2)), Dr = p2::mul(k, p2::sub(f0, fp1));
  const float2 x = make_float2(clamp2(fm1.x, f0.x, fi.x), clamp2(fm1.y, f0.y, fi.y));
  const float2 dl = p2::sub(x, fm1), dr = p2::sub(x, f0);
  const float2 l = p2::sub(x, p2::sub(dl, make_float2(shrink(dl.x, Dl.x), shrink(dl.y, Dl.y))));
  const float2 r = p2::sub(x, p2::sub(dr, make_float2(shrink(dr.x, Dr.x), shrink(dr.y, Dr.y))));
  lr0 = make_float2(l.x, r.x);
  lr1 = make_float2(l.y, r.y);
}

// 0.5 erfc(-x.x) (left state, + moment) and 0.5 erfc(x.y) (right state, -
// moment) with the erfcc fit of Moments<float>::erfc_pos: its polynomial is
// evaluated with negated coefficients, so exp(z^2 - (-q)) takes the same
// argument as erfc_pos's exp(-z^2 + q).
__device__ __forceinline__ float2 half_erfc_lr(float2 x) {
  const float2 t = p2::rcp(make_float2(fmaf(0.5f, fabsf(x.x), 1.0f), fmaf(0.5f, fabsf(x.y), 1.0f)));
  float2 nq = p2::fma(t, p2::K(-0.17087277f), p2::K(0.82215223f));
  nq = p2::fma(t, nq, p2::K(-1.48851587f));
  nq = p2::fma(t, nq, p2::K(1.13520398f));
  nq = p2::fma(t, nq, p2::K(-0.27886807f));
  nq = p2::fma(t, nq, p2::K(0.18628806f));
  nq = p2::fma(t, nq, p2::K(-0.09678418f));
  nq = p2::fma(t, nq, p2::K(-0.37409196f));
  nq = p2::fma(t, nq, p2::K(-1.00002368f));
  nq = p2::fma(t, nq, p2::K(1.26551223f));
  const float2 e = p2::exp_neg(p2::fma(x, x, nq));  // of x^2 - q
  const float2 h = p2::mul(p2::K(0.5f), p2::mul(t, e));
  const float2 g = p2::sub(p2::K(1.0f), h);
  return make_float2(x.x <= 0.0f ? h.x : g.x, x.y >= 0.0f ? h.y : g.y);
}

// Fluxes and magnetic stress through one face normal to axis D (the
// formulas of face_flux) with the left state in lane x and the right state
// in lane y of X[q] = (l[q], r[q]); out = left + right.
template <int D>
__device__ __forceinline__ void face_flux_lr(const float2* X, float rg, float* out) {
  using namespace p2;
  const float2 r = X[0], u = X[1], v = X[2], w = X[3], pr = X[4], bx = X[5], by = X[6], bz = X[7];
  const float2 vn = X[1 + D], bn = X[5 + D];
  float2 ke = mul(u, u);
  ke = fma(v, v, ke);
  ke = fma(w, w, ke);
  const float2 leng = fma(pr, K(rg), mul(mul(K(0.5f), r), ke));
  // hydro moments, lam = rho / (2 p)
  float2 lb = mul(bx, bx);
  lb = fma(by, by, lb);
  lb = fma(bz, bz, lb);
  float2 lam, ra, a, am;
  lam_roots(r, mul(K(2.0f), pr), fma(K(2.0f), pr, lb), lam, ra, a, am);
  const float2 v0 = half_erfc_lr(mul(a, vn));
  const float2 lv = mul(mul(lam, vn), vn);
  const float2 b = mul(mul(K(0.5f * 0.56418958354775628f), ra), exp_neg(lv));
  const float2 v1 = fma(vn, v0, make_float2(b.x, -b.y));
  float2 f[8];
  f[0] = mul(r, v1);
  f[1] = mul(mul(r, u), v1);
  f[2] = mul(mul(r, v), v1);
  f[3] = mul(mul(r, w), v1);
  f[4] = mul(fma(K(0.5f), pr, leng), v1);
  f[1 + D] = fma(pr, v0, f[1 + D]);
  f[4] = fma(mul(mul(K(0.5f), pr), vn), v0, f[4]);
  // magnetic stress, lam = rho / (2 p + B^2)
  const float2 m0 = half_erfc_lr(mul(am, vn));
  const float2 nm0 = mul(K(-1.0f), m0);
  const float2 hb = mul(K(0.5f), lb);
  f[5] = (D == 0) ? mul(sub(hb, mul(bx, bx)), m0) : mul(mul(bx, bn), nm0);
  f[6] = (D == 1) ? mul(sub(hb, mul(by, by)), m0) : mul(mul(by, bn), nm0);
  f[7] = (D == 2) ? mul(sub(hb, mul(bz, bz)), m0) : mul(mul(bz, bn), nm0);
#pragma unroll
  for (int q = 0; q < 8; ++q) out[q] = f[q].x + f[q].y;
}

// ------------------------------------------------------- FP64 moments
// 0.5 erfc(|z|) and exp(-z^2) / (2 sqrt(pi)) from one table of polynomials
// (d.gtab: row i about c = i / 32, ten coefficients of each; gauss_table() fills it).
// CUDA's erfc and exp take about 60 and 20 operations of the FP64 pipe; here the
// row index and the offset from its centre take three and each polynomial nine.
// Both are good to 3e-16 of their own value: a stream that leaves a face
// sends v v0 +- b through it, whose terms cancel to 1 / 2 z^2, and a dense one may
// feed a thin cell with it.  Beyond |z| = 6.5 the tails come from erfc and exp; where the
// result is 1 less a tail they are below its rounding and taken as zero (NaN stays NaN).
static __device__ __noinline__ double half_erfc_far(double az) { return 0.5 * erfc(az); }
static __device__ __noinline__ double bell_far(double az) {  // z^2 in two parts
  const double s = az * az, e = 0.28209479177387814 * exp(-s);
  return s < INFINITY ? fma(-e, fma(az, az, -s), e) : 0.0;
}
struct GaussArg {
  const double2* row;
  double d;
  int far;      // 0: in the table, 1: beyond it, 2: NaN
  bool direct;  // the side that a tail is the moment of: z <= 0 for the left (+ moments), z >= 0 for the right state
  __device__ __forceinline__ GaussArg(const double* tab, double z, bool left) {
    const double az = abs_bits(z);
    const double t = fma(az, 32.0, 6755399441055744.0);  // 1.5 * 2^52: the nearest integer in the low word
    d = fma(t - 6755399441055744.0, -0.03125, az);
    const int hi = __double2hiint(az);
    far = hi < 0x401a0000 ? 0 : hi <= 0x7ff00000 ? 1 : 2;
    direct = (__double2hiint(z) < 0) == left;
    const unsigned i = (unsigned)__double2loint(t);
    row = reinterpret_cast<const double2*>(tab) + (i < kGaussRows ? i : kGaussRows - 1) * kGaussTerms;
  }
  __device__ __forceinline__ double poly(const double2* q) const {
    static_assert(kGaussTerms == 10, "five pairs of coefficients");
    double2 a = __ldg(q + 4);
    double s = fma(a.y, d, a.x);
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      a = __ldg(q + k);
      s = fma(fma(s, d, a.y), d, a.x);
    }
    return s;
  }
  // 0.5 erfc(-z) for the left or 0.5 erfc(z) for the right state
  __device__ __forceinline__ double half_erfc(double z) const {
    double h = poly(row);
    if (far) h = far == 2 ? z : direct ? half_erfc_far(abs_bits(z)) : 0.0;
    return direct ? h : 1.0 - h;
  }
  __device__ __forceinline__ double bell(double z) const {
    double e = poly(row + kGaussTerms / 2);
    if (far) e = far == 2 ? z : direct ? bell_far(abs_bits(z)) : 0.0;
    return e;
  }
};

// a = sqrt(r / q) and ia = sqrt(q / r) for the two lam of a face state, q = 2 p and
// q = 2 p + B^2, by one rsqrt each.  The product r q must be a normal number for that:
// where either is not (p = 0, a product below 1e-307 or above 1e308, a negative p,
// NaN) the quotient decides, as the reference writes it.  p = 0 so gives a =
// inf, ia = 0 and with them finite moments of a gas that moves.
__device__ __forceinline__ void lam_roots(double r, double q, double qm, double& a, double& ia, double& am) {
  const double m = q * r, mm = qm * r;
  const unsigned lo = 0x00200000u, n = 0x7fe00000u - lo;  // high words of 2^-1021 .. 2^1023
  if ((unsigned)__double2hiint(m) - lo < n && (unsigned)__double2hiint(mm) - lo < n) {
    const double s = rsqrt(m);
    a = r * s;
    ia = q * s;
    am = r * rsqrt(mm);
  } else {
    a = sqrt(r / q);
    ia = 1.0 / a;
    am = sqrt(r / qm);
  }
}

// One side (left: + moments) of the FP64 flux through a face normal to axis D:
// the formulas of face_flux with lam_roots, the shared products formed once and
// fused operations.  About 85 operations of the FP64 pipe; as written in the
// reference, with two divisions, a root, an exp and two erfc per side, about 240.
template <int D>
__device__ __forceinline__ void face_side64(const double* q, const Dev<double>& dv, bool left, double* f) {
  const double r = q[0], u = q[1], v = q[2], w = q[3], p = q[4], x = q[5], y = q[6], z = q[7];
  const double vn = q[1 + D], bn = q[5 + D];
  const double ke = fma(u, u, fma(v, v, w * w)), p2 = p + p, b2 = fma(x, x, fma(y, y, z * z));
  double a, ia, am;
  lam_roots(r, p2, p2 + b2, a, ia, am);
  a *= vn;
  am *= vn;
  const GaussArg ga(dv.gtab, a, left);
  const double v0 = ga.half_erfc(a);
  const double b = ia * ga.bell(a);
  const double v1 = fma(vn, v0, left ? b : -b);
  const double m = r * v1, pv = p * v0;
  f[0] = m;
  f[1] = m * u;
  f[2] = m * v;
  f[3] = m * w;
  f[1 + D] += pv;
  f[4] = fma(fma(0.5 * ke, r, p * (dv.rgm1 + 0.5)), v1, (0.5 * vn) * pv);
  const double m0 = GaussArg(dv.gtab, am, left).half_erfc(am);
  const double t = -bn * m0;
  f[5] = x * t;
  f[6] = y * t;
  f[7] = z * t;
  f[5 + D] = fma(0.5 * b2, m0, f[5 + D]);
}

// Fluxes and magnetic stress through one face normal to axis D from the
// reconstructed left (l) and right (r) states {rho, vx, vy, vz, p, bx, by, bz}
// (get_flux_stress, mhd3d3.f90:2385-2560): out = {rho, rvx, rvy, rvz, eng,
// s_x, s_y, s_z}.  Left state with the + moments, right with the - moments.
// FP32: on the packed pipe (face_flux_lr).
// FP64: face_side64 per side.
template <int D>
__device__ __forceinline__ void face_flux(const float* l, const float* r, const Dev<float>& d, float* out) {
  float2 X[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) X[q] = make_float2(l[q], r[q]);
  face_flux_lr<D>(X, d.rgm1, out);
}
template <int D>
__device__ __forceinline__ void face_flux(const double* l, const double* r, const Dev<double>& d, double* out) {
  double f[8];
  face_side64<D>(l, d, true, out);
  face_side64<D>(r, d, false, f);
#pragma unroll
  for (int q = 0; q < 8; ++q) out[q] = out[q] + f[q];
}

// Metric-mode flux through a face of unit normal n and area am: the
// Gaussian-split formulas of face_flux with n in place of the axis (vector
// momentum and magnetic stress), left with the + moments and right with the
// - moments, the sum multiplied by am (the oracle's get_flux_stress_metric).
template <typename T>
__device__ __forceinline__ void face_flux_n(const T* l, const T* r, const Dev<T>& d, const T* n, T am, T* out) {
  typedef Moments<T> Mo;
  T tot[8];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const T* s = side ? r : l;
    const T rr = s[0], u0 = s[1], u1 = s[2], u2 = s[3], pr = s[4], b0 = s[5], b1 = s[6], b2 = s[7];
    const T vn = u0 * n[0] + u1 * n[1] + u2 * n[2];
    const T bn = b0 * n[0] + b1 * n[1] + b2 * n[2];
    const T leng = T(0.5) * rr * (u0 * u0 + u1 * u1 + u2 * u2) + over_gm1<true>(d, pr);
    T lam = Mo::div(rr, T(2) * pr);
    T v0, v1;
    Mo::hydro(lam, vn, side == 0, v0, v1);
    T f[8];
    f[0] = rr * v1;
    f[1] = rr * u0 * v1 + pr * n[0] * v0;
    f[2] = rr * u1 * v1 + pr * n[1] * v0;
    f[3] = rr * u2 * v1 + pr * n[2] * v0;
    f[4] = (leng + T(0.5) * pr) * v1 + T(0.5) * pr * vn * v0;
    const T lbsq = b0 * b0 + b1 * b1 + b2 * b2;
    lam = Mo::div(rr, T(2) * pr + lbsq);
    v0 = Mo::mag(lam, vn, side == 0);
    f[5] = (T(0.5) * lbsq * n[0] - b0 * bn) * v0;
    f[6] = (T(0.5) * lbsq * n[1] - b1 * bn) * v0;
    f[7] = (T(0.5) * lbsq * n[2] - b2 * bn) * v0;
#pragma unroll
    for (int q = 0; q < 8; ++q) tot[q] = side ? tot[q] + f[q] : f[q];
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) out[q] = tot[q] * am;
}

// Face flux of axis D at face c, Cartesian or metric.
template <typename T, int D, bool M>
__device__ __forceinline__ void any_face_flux(const Dev<T>& d, long long c, const T* L, const T* R, T* out) {
  if (M) {
    const T n[3] = {d.m.nrm[D][0][c], d.m.nrm[D][1][c], d.m.nrm[D][2][c]};
    face_flux_n<T>(L, R, d, n, d.m.am[D][c], out);
  } else {
    face_flux<D>(L, R, d, out);
  }
}

// One-sided states from an 8-tap register window (tap m = cell c+m-4 for the
// face at the low side of cell c): slot of tap m is (m + PH) & 7.
template <typename T, int RECON, int PH>
__device__ __forceinline__ void recon_win(const T* w, const Prm<T>& P, T& fl, T& fr) {
#define TAP(m) w[((m) + PH) & 7]
  if (is_pdm(RECON)) {
    recon_pdm8<T, RECON>(TAP(0), TAP(1), TAP(2), TAP(3), TAP(4), TAP(5), TAP(6), TAP(7), P.pdmb, fl, fr);
  } else if (RECON == R_TVD || RECON == R_TVDMC) {
    T fi = (TAP(3) + TAP(4)) / T(2);
    tvd<T, RECON == R_TVDMC>(TAP(2), TAP(3), TAP(4), TAP(5), fi, P.eps, fl, fr);
  } else {
    weno_both<RECON>(TAP(1), TAP(2), TAP(3), TAP(4), TAP(5), TAP(6), P, fl, fr);
  }
#undef TAP
}

// One-sided states of the 8 cell fields src[0..7] at the low face of element
// c along stride s (recon_face per field); FP32 PDM on field pairs.
template <typename T, int RECON, bool M, typename I>
__device__ __forceinline__ void face_states(const T* const* src, I c, I s, const Prm<T>& P, T* L, T* R) {
  if constexpr (std::is_same<T, float>::value && is_pdm(RECON) && MHD_RECON_PACKED) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float *fa = src[2 * q], *fb = src[2 * q + 1];
      float2 a[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) a[m] = make_float2(fa[c + (m - 4) * s], fb[c + (m - 4) * s]);
      float2 lr0, lr1;
      pdm_pair_states<RECON>(a, P.pdmb, lr0, lr1);
      L[2 * q] = lr0.x; R[2 * q] = lr0.y;
      L[2 * q + 1] = lr1.x; R[2 * q + 1] = lr1.y;
    }
  } else if constexpr (std::is_same<T, float>::value && is_weno(RECON)) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float *fa = src[2 * q], *fb = src[2 * q + 1];
      float2 a[6], l, r;
#pragma unroll
      for (int m = 0; m < 6; ++m) a[m] = make_float2(fa[c + (m - 3) * s], fb[c + (m - 3) * s]);
      weno_both<RECON>(a[0], a[1], a[2], a[3], a[4], a[5], P, l, r);
      L[2 * q] = l.x; R[2 * q] = r.x;
      L[2 * q + 1] = l.y; R[2 * q + 1] = r.y;
    }
  } else {
#pragma unroll
    for (int v = 0; v < 8; ++v) recon_face<T, RECON, I, M>(src[v], c, s, P, L[v], R[v]);
  }
}

// Face fluxes through the low face of cell c along axis D by direct (cached)
// loads; one face per thread.  Used for the x faces of every stage and, for
// all three axes, by the kernel-level debug entry point.
template <typename T, int RECON, int D, bool M, bool B>
__global__ void k_flux(KArg<T, B> ka, Inp<T> in0, Prm<T> P) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Inp<T> in = B ? state_view(d) : in0;
  const Geom& g = d.g;
  const int ni = g.nx0 + (D == 0), nj = g.ny0 + (D == 1), nk = g.nz0 + (D == 2);
  const int t = bb.y * blockDim.x + threadIdx.x;
  if (t >= ni * nj * nk) return;
  const int i = t % ni + g.ng;
  const int r = t / ni;
  const int j = r % nj + g.ng;
  const int k = r / nj + g.ng;
  const int c = i + g.px * (j + g.py * k);
  const int s = (D == 0) ? 1 : (D == 1) ? g.px : (int)g.plane;
  const T* src[8] = {in.rho, in.vx, in.vy, in.vz, in.p, in.bx, in.by, in.bz};
  T L[8], R[8], out[8];
  face_states<T, RECON, M>(src, c, s, P, L, R);
  any_face_flux<T, D, M>(d, c, L, R, out);
#pragma unroll
  for (int q = 0; q < 8; ++q) d.F[D][q][c] = out[q];
}

// FP64, single grids: the faces of all three axes in one launch, their fluxes
// to memory, and the conserved update of k_update_faces after it.  The FP64 pipe
// bounds the faces, so the fluxes' traffic is free, no face is computed twice
// (the y / z tiles recompute one of nine), the lanes are full whatever the
// extents (nx0 = 16 left half of a tile's idle), and 16^3 cells are spread over
// every SM (blocks of 64 faces while there are few).  The fluxes take arrays that
// are dead meanwhile: y those of dU, z the other half's, face B until CT writes it and
// the primitives until the update does.
template <int D>
__device__ __forceinline__ double* face_flux_ptr(const Dev<double>& d, int q) {
  if (D == 0) return d.F[0][q];
  if (D == 1) return d.dU[q];
  double* const z[8] = {d.orho, d.ovx, d.ovy, d.ovz, d.op, d.obi, d.obj, d.obk};
  return z[q];
}
template <int RECON, int D, bool M>
__device__ __forceinline__ void face_one(const Dev<double>& d, const Inp<double>& in, const Prm<double>& P, int t,
                                         int ni, int nj) {
  typedef double T;
  const Geom& g = d.g;
  const int i = t % ni, r = t / ni, j = r % nj, k = r / nj;
  const int c = i + g.ng + g.px * (j + g.ng + g.py * (k + g.ng));
  const int s = (D == 0) ? 1 : (D == 1) ? g.px : (int)g.plane;
  const T* src[8] = {in.rho, in.vx, in.vy, in.vz, in.p, in.bx, in.by, in.bz};
  T L[8], R[8], out[8];
  face_states<T, RECON, M>(src, c, s, P, L, R);
  any_face_flux<T, D, M>(d, c, L, R, out);
#pragma unroll
  for (int q = 0; q < 8; ++q) face_flux_ptr<D>(d, q)[c] = out[q];
}
template <int RECON, bool M>
__global__ void __launch_bounds__(128) k_faces(Dev<double> d, Inp<double> in, Prm<double> P) {
  const Geom& g = d.g;
  unsigned t = blockIdx.x * blockDim.x + threadIdx.x;  // each axis fits an int, the three together may not
  const unsigned n0 = (g.nx0 + 1) * g.ny0 * g.nz0, n1 = g.nx0 * (g.ny0 + 1) * g.nz0, n2 = g.nx0 * g.ny0 * (g.nz0 + 1);
  if (t < n0) return face_one<RECON, 0, M>(d, in, P, t, g.nx0 + 1, g.ny0);
  t -= n0;
  if (t < n1) return face_one<RECON, 1, M>(d, in, P, t, g.nx0, g.ny0 + 1);
  t -= n1;
  if (t < n2) face_one<RECON, 2, M>(d, in, P, t, g.nx0, g.ny0);
}

// Stage combine of the RK steps (mhd3d3.f90:3674-3702, 3745-3788):
// form 0: (Xp+X)/den, 1: (c*Xp+X)/den, 2: (Xp+c*X)/den.
// FP64: the divisors are 2, 4 and 3 (forms 0, 1, 2), an exact scaling or two
// operations with the division's rounding (div_by).
__device__ __forceinline__ float comb(int form, float c, float xp, float x, float den) {
  if (form == 0) return Ops<float>::dv(xp + x, den);
  if (form == 1) return Ops<float>::dv(c * xp + x, den);
  return Ops<float>::dv(xp + c * x, den);
}
__device__ __forceinline__ double comb(int form, double c, double xp, double x, double) {
  if (form == 0) return 0.5 * (xp + x);
  if (form == 1) return 0.25 * (c * xp + x);
  return div_by<3>(xp + c * x);
}

// One-sided states from a column of taps in shared memory: tap m (cell
// c+m-4 for the face at the low side of cell c) at col[m * RS].
template <typename T, int RECON, int RS>
__device__ __forceinline__ void recon_col(const T* col, const Prm<T>& P, T& fl, T& fr) {
  if (is_pdm(RECON)) {
    recon_pdm8<T, RECON>(col[0], col[RS], col[2 * RS], col[3 * RS], col[4 * RS], col[5 * RS], col[6 * RS], col[7 * RS],
                         P.pdmb, fl, fr);
  } else if (RECON == R_TVD || RECON == R_TVDMC) {
    T fi = (col[3 * RS] + col[4 * RS]) / T(2);
    tvd<T, RECON == R_TVDMC>(col[2 * RS], col[3 * RS], col[4 * RS], col[5 * RS], fi, P.eps, fl, fr);
  } else {
    weno_both<RECON>(col[RS], col[2 * RS], col[3 * RS], col[4 * RS], col[5 * RS], col[6 * RS], P, fl, fr);
  }
}

// y / z faces with the flux divergence fused through shared memory.  A block
// covers 32 cells along x and TD cells along the sweep axis D (1: y, 2: z) at
// one value of the remaining axis.  It stages the 8 reconstructed cell fields
// of TD+8 rows (4-cell halo each side) with independent coalesced loads, its
// TD+1 thread rows compute the TD+1 faces bounding those cells from shared
// memory, and the first TD rows combine the face pair of their cell:
//   D == 1: dU_q = (Fx_q(i+1)-Fx_q(i))/dx + (Fy_q(j+1)-Fy_q(j))/dy, the first
//     two terms of advance_corrector1/2 (mhd3d3.f90:3850-3906) in their order;
//   D == 2: the z term completes advance_corrector1 + stage combine + p +
//     advance_corrector2 + combine + v (RK: 3666-3697 / 3736-3783; AB:
//     3626-3627, 3876, 3901-3905), written to the other half of the
//     double-buffered primitives.
// Tuning knobs (compile time): cells per block along the sweep axis, whether
// the cell tile is staged in shared memory (1) or read through L1 (0), and
// the minimum resident blocks per SM requested from the register allocator.
#ifndef MHD_FLUX_TD
#define MHD_FLUX_TD 8
#endif
#ifndef MHD_FLUX_STAGED
#define MHD_FLUX_STAGED 0
#endif
#ifndef MHD_FLUX_MINB
#define MHD_FLUX_MINB 6
#endif
constexpr int TD = MHD_FLUX_TD;  // default tile length; FP32 PDM also has 4 and 16 (autotuner)
constexpr bool FLUX_STAGED = MHD_FLUX_STAGED != 0;

// Resident blocks per SM requested for the flux tiles: FP32 trades registers
// for occupancy (latency-bound); FP64 needs about twice the registers and
// would spill at the FP32 setting.
// The metric mode's general normal takes more registers as well, and so do the
// packed WENO states (they spilled 0.8 KB at 32).
template <typename T, bool M, int RECON> struct FluxMinB {
  static constexpr int value = sizeof(T) == 8 ? 2 : RECON == R_WENO || RECON == R_MPWENO ? 3 : M ? 4 : MHD_FLUX_MINB;
};

template <typename T, int TDV = TD>
__host__ __device__ constexpr size_t flux_t_smem() {
  // [+ staged cells] + face fluxes of the sweep + the x-face fluxes the y kernel reads (8 x TD x 33)
  return sizeof(T) * ((FLUX_STAGED ? 8 * (TDV + 8) * 32 : 0) + 8 * (TDV + 1) * 32 + 8 * TDV * 33);
}

// The conserved update of one cell from its z-face flux difference dF and the
// x+y divergence in dU (advance_corrector1 + stage combine + p +
// advance_corrector2 + combine + v, mhd3d3.f90:3666-3697 / 3736-3783; AB:
// 3626-3627, 3876, 3901-3905), written to the other half of the
// double-buffered primitives.  cd is the cell's z index.
// du: the x+y divergence dU of the cell; pv: its rho, vx, vy, vz, p; qv: its
// U^n (q[0..4], read only when form >= 0).
template <typename T, bool M>
__device__ __forceinline__ void cell_update_vals(const Dev<T>& d, int c, int cd, const T* dF, const T* du,
                                                 const T* pv, const T* qv, int form, T cw, T den) {
  const T tau = step_tau<T>(d.sc);
  const T gm1 = d.gam - T(1);
  T dv[8];
  if (M) {
    const T V = d.m.vol[c], rV = d.m.rvol[c];
#pragma unroll
    for (int q = 0; q < 8; ++q) dv[q] = Ops<T>::dw(du[q] + dF[q], V, rV);
  } else {
    const T dz = d.wz[cd], rdz = d.rwz[cd];
#pragma unroll
    for (int q = 0; q < 8; ++q) dv[q] = du[q] + Ops<T>::dc(dF[q], dz, rdz);
  }
  // get_conserve of the current state (AB: the state, not the prediction)
  T rr = pv[0], u = pv[1], v = pv[2], ww = pv[3], pr = pv[4];
  T rvx0 = rr * u, rvy0 = rr * v, rvz0 = rr * ww;
  T eng0 = T(0.5) * rr * (u * u + v * v + ww * ww) + over_gm1<M>(d, pr);
  if (form == FORM_SAVE) {  // U^n of the step (this first stage's input), read by the later stages' combines
    d.q[0][c] = rr;
    d.q[1][c] = rvx0;
    d.q[2][c] = rvy0;
    d.q[3][c] = rvz0;
    d.q[4][c] = eng0;
  }
  T rho1 = rr - tau * dv[0];
  T eng1 = eng0 - tau * dv[4];
  T rx = rvx0 - tau * dv[1], ry = rvy0 - tau * dv[2], rz = rvz0 - tau * dv[3];
  T hx = rx, hy = ry, hz = rz;
  if (form >= 0) {
    rho1 = comb(form, cw, qv[0], rho1, den);
    hx = comb(form, cw, qv[1], rx, den);
    hy = comb(form, cw, qv[2], ry, den);
    hz = comb(form, cw, qv[3], rz, den);
    eng1 = comb(form, cw, qv[4], eng1, den);
  }
  constexpr bool EXACT = M && std::is_same<T, double>::value;
  const T rrho = EXACT ? T(0) : Ops<T>::rcp(rho1);
  auto over_rho = [&](T x) { return EXACT ? x / rho1 : Ops<T>::dvr(x, rho1, rrho); };
  T pn = gm1 * (eng1 - over_rho(T(0.5) * (hx * hx + hy * hy + hz * hz)));
  rx = rx - tau * dv[5];
  ry = ry - tau * dv[6];
  rz = rz - tau * dv[7];
  if (form >= 0) {
    rx = comb(form, cw, qv[1], rx, den);
    ry = comb(form, cw, qv[2], ry, den);
    rz = comb(form, cw, qv[3], rz, den);
  }
  d.orho[c] = rho1;
  d.op[c] = pn;
  d.ovx[c] = over_rho(rx);
  d.ovy[c] = over_rho(ry);
  d.ovz[c] = over_rho(rz);
}

template <typename T, bool M>
__device__ __forceinline__ void cell_update(const Dev<T>& d, int c, int cd, const T* dF, int form, T cw, T den) {
  T du[8], pv[5], qv[5];
#pragma unroll
  for (int q = 0; q < 8; ++q) du[q] = d.dU[q][c];
  pv[0] = d.rho[c]; pv[1] = d.vx[c]; pv[2] = d.vy[c]; pv[3] = d.vz[c]; pv[4] = d.p[c];
#pragma unroll
  for (int q = 0; q < 5; ++q) qv[q] = (form >= 0) ? d.q[q][c] : T(0);
  cell_update_vals<T, M>(d, c, cd, dF, du, pv, qv, form, cw, den);
}

// The update after k_faces: the flux divergence in the tiles' order, then
// cell_update_vals, which puts a cell's new primitives where the z fluxes of its low face
// lie.  So a block owns whole columns, TX of them, and walks them in slabs of TZ cells:
// every thread has read both faces of its cell before any writes, and the next slab's
// low faces are beyond what this one writes.  TZ = 32 (or what nz0 needs) by 128 / TZ
// columns, a sector of x.  Bytes and latency bound it; PDM stage in us at one cell a thread
// with the z fluxes in arrays of their own, and at TZ = 8, 16, 32, 64: 16^3 48.8, 53.4
// 48.6 48.4 48.4; 64^3 898.6, 908.8 909.6 899.1 900.3 (256 or 512 threads: no faster).
template <bool M>
__global__ void __launch_bounds__(128) k_update_faces(Dev<double> d, int form, double cw, double den) {
  typedef double T;
  const Geom& g = d.g;
  const int nbx = (g.nx0 + blockDim.x - 1) / blockDim.x;
  const int i0 = blockIdx.x % nbx * blockDim.x + threadIdx.x, j = blockIdx.x / nbx + g.ng, i = i0 + g.ng;
  const int sy = g.px, sz = (int)g.plane;
  for (int k0 = 0; k0 < g.nz0; k0 += blockDim.y) {
    const int k = k0 + threadIdx.y + g.ng, c = i + g.px * (j + g.py * k);
    const bool in = i0 < g.nx0 && k < g.ng + g.nz0;
    T du[8], dF[8], pv[5], qv[5];
    if (in) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const T *fx = face_flux_ptr<0>(d, q), *fy = face_flux_ptr<1>(d, q), *fz = face_flux_ptr<2>(d, q);
        const T dx = fx[c + 1] - fx[c], dy = fy[c + sy] - fy[c];
        du[q] = M ? dx + dy : Ops<T>::dc(dx, d.wx[i], d.rwx[i]) + Ops<T>::dc(dy, d.wy[j], d.rwy[j]);
        dF[q] = fz[c + sz] - fz[c];
      }
      pv[0] = d.rho[c]; pv[1] = d.vx[c]; pv[2] = d.vy[c]; pv[3] = d.vz[c]; pv[4] = d.p[c];
#pragma unroll
      for (int q = 0; q < 5; ++q) qv[q] = (form >= 0) ? d.q[q][c] : T(0);
    }
    __syncthreads();
    if (in) cell_update_vals<T, M>(d, c, k, dF, du, pv, qv, form, cw, den);
  }
}

template <typename T, int RECON, int D, bool M, bool B, int TDV = TD>
__global__ void __launch_bounds__(32 * (TDV + 1), FluxMinB<T, M, RECON>::value)
    k_flux_t(KArg<T, B> ka, Inp<T> in0, Prm<T> P, int form, T cw, T den, int ab) {
  constexpr int TD = TDV;
  constexpr int TROWS = TDV + 8;
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Inp<T> in = B ? state_view(d) : in0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sv = reinterpret_cast<T*>(smem_raw);                      // [8][TROWS][32] cell fields
  T* sF = sv + (FLUX_STAGED ? 8 * TROWS * 32 : 0);             // [8][TD+1][32] face fluxes
  T* sX = sF + 8 * (TD + 1) * 32;                              // [8][TD][33] x-face fluxes (D == 1)
  const Geom& g = d.g;
  const int tx = threadIdx.x, r = threadIdx.y;
  const int i0 = bb.y * 32 + g.ng;
  const int i = i0 + tx;
  const int n0 = (D == 1) ? g.ny0 : g.nz0;
  const int nD = (D == 1) ? g.ny : g.nz;
  const int cd0 = bb.z * TD + g.ng;  // first cell of the tile along D
  const int o = bb.w + g.ng;         // remaining transverse index
  const int s = (D == 1) ? g.px : (int)g.plane;
  const int rowbase = (D == 1) ? i0 + g.px * g.py * o : i0 + g.px * o;  // + cd * s
  const T* src[8] = {in.rho, in.vx, in.vy, in.vz, in.p, in.bx, in.by, in.bz};
  if (D == 1) {
    // The x-face fluxes of the tile's cells (faces i0 .. i0+32 of rows cd0 ..
    // cd0+TD-1) are only needed in the epilogue: copy them asynchronously now
    // so their latency hides behind the reconstructions.
    const int nthr = 32 * (TD + 1);
#pragma unroll
    for (int q = 0; q < 8; ++q) {  // static q: the flux pointers stay in registers
      const T* fq = d.F[0][q];
      for (int t = r * 32 + tx; t < TD * 33; t += nthr) {
        const int rr = t / 33, col = t - rr * 33;
        if (cd0 + rr < g.ng + n0 && i0 + col <= g.ng + g.nx0) {
          const T* gp = fq + rowbase + col + (cd0 + rr) * s;
          const uint32_t sp = (uint32_t)__cvta_generic_to_shared(sX + q * TD * 33 + t);
          if (sizeof(T) == 4)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sp), "l"(gp) : "memory");
          else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sp), "l"(gp) : "memory");
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (FLUX_STAGED) {
    const int nthr = 32 * (TD + 1);
    const bool xok = i0 + tx < g.nx;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const T* sp = src[v] + rowbase + tx;
      for (int t = r * 32 + tx; t < TROWS * 32; t += nthr) {
        const int cd = cd0 - 4 + (t >> 5);
        sv[v * TROWS * 32 + t] = (xok && cd < nD) ? sp[cd * s] : T(0);
      }
    }
    __syncthreads();
  }
  const int cd = cd0 + r;  // cell whose low face this thread computes
  const bool xin = i < g.ng + g.nx0;
  if (xin && cd <= g.ng + n0) {
    T L[8], R[8], F[8];
    if (FLUX_STAGED) {
#pragma unroll
      for (int v = 0; v < 8; ++v) recon_col<T, RECON, 32>(sv + (v * TROWS + r) * 32 + tx, P, L[v], R[v]);
    } else {
      const int cf = rowbase + tx + cd * s;
      face_states<T, RECON, M>(src, cf, s, P, L, R);
    }
    any_face_flux<T, D, M>(d, rowbase + tx + cd * s, L, R, F);
#pragma unroll
    for (int q = 0; q < 8; ++q) sF[(q * (TD + 1) + r) * 32 + tx] = F[q];
  }
  if (D == 1) asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (r >= TD || !xin || cd >= g.ng + n0) return;
  const int c = rowbase + tx + cd * s;
  T dF[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) dF[q] = sF[(q * (TD + 1) + r + 1) * 32 + tx] - sF[(q * (TD + 1) + r) * 32 + tx];
  if (D == 1) {
    if (M) {  // area-weighted fluxes: the sum is divided by V after the z term
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const T* x = sX + (q * TD + r) * 33 + tx;
        d.dU[q][c] = (x[1] - x[0]) + dF[q];
      }
      return;
    }
    const T dx = d.wx[i], dy = d.wy[cd], rdx = d.rwx[i], rdy = d.rwy[cd];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const T* x = sX + (q * TD + r) * 33 + tx;
      d.dU[q][c] = Ops<T>::dc(x[1] - x[0], dx, rdx) + Ops<T>::dc(dF[q], dy, rdy);
    }
    return;
  }
  cell_update<T, M>(d, c, cd, dF, form, cw, den);
  (void)ab;
}

// y / z faces by column sweeps: the FP32 Cartesian PDM alternative to the face
// tiles, one more launch shape for the autotuner.  A thread owns one column of
// cells along D (x from the lane, the remaining axis from the warp) over a
// segment of Dev::seg cells (sweep_seg) and keeps the 8 reconstructed fields of the 8
// cells around its current face in registers: one new cell is loaded per face
// (issued a face ahead, before that face's arithmetic), every face flux is
// computed once, and a cell's face-pair difference is the current minus the
// previous face's flux.  Face arithmetic and epilogues are those of k_flux_t,
// so the two give the same bits.
#ifndef MHD_SWEEP_UNROLL
#define MHD_SWEEP_UNROLL 1
#endif
constexpr int kSweepUnroll = MHD_SWEEP_UNROLL;  // face-loop unroll (compile-time knob)
#ifndef MHD_SWEEP_MINB
#define MHD_SWEEP_MINB 4
#endif
constexpr int kSweepMinB = MHD_SWEEP_MINB;  // resident 128-thread blocks per SM (register budget)

template <typename T, int D, bool B, int RECON = R_PDM>
__global__ void __launch_bounds__(128, kSweepMinB)
    k_flux_sweep(KArg<T, B> ka, Inp<T> in0, Prm<T> P, int form, T cw, T den) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Inp<T> in = B ? state_view(d) : in0;
  const Geom& g = d.g;
  const int n0 = (D == 1) ? g.ny0 : g.nz0;
  const int no = (D == 1) ? g.nz0 : g.ny0;
  // columns are numbered x first, then along the remaining axis (z for y
  // faces, y for z faces), 32 to a warp, so a warp may span rows; lanes past the
  // last column work on a copy of it and store nothing, so the whole warp stays
  // in the loop (warp-synchronous copies below)
  const int tx = threadIdx.x, ncol = g.nx0 * no;
  const int u = (bb.y * 4 + threadIdx.y) * 32 + tx;
  if (u - tx >= ncol) return;
  const bool xin = u < ncol;
  const int uc = xin ? u : ncol - 1;
  const int i = uc % g.nx0 + g.ng, o = uc / g.nx0 + g.ng;
  // y faces: does this lane copy its own x face i + 1 (the next lane holds another row, or there is none)?
  const bool xlast = tx == 31 || i == g.ng + g.nx0 - 1;
  const int seg = d.seg[D - 1];
  const int c0 = g.ng + bb.z * seg;
  const int c1 = min(c0 + seg, g.ng + n0);
  const int s = (D == 1) ? g.px : (int)g.plane;
  const int col = (D == 1) ? i + (int)g.plane * o : i + g.px * o;  // + cd * s
  const T* src[8] = {in.rho, in.vx, in.vy, in.vz, in.p, in.bx, in.by, in.bz};
  // y faces: the x-face fluxes of the next cell are copied asynchronously into
  // a per-warp double buffer one face ahead of the epilogue that reads them
  // (the copies that xlast lanes make follow the warp's 32)
  __shared__ __align__(16) T sxf[D == 1 ? 4 : 1][2][8][64];
  T (*xs)[8][64] = sxf[D == 1 ? threadIdx.y : 0];
  const int xh = xlast ? 32 : 1;  // from a lane's low x face to its high one
  // z faces: dU, the state (rho, v, p) and U^n of the next cell, likewise
  // (each lane reads back only what it copied)
  __shared__ __align__(16) T szf[D == 2 ? 4 : 1][2][18][32];
  T (*zs)[18][32] = szf[D == 2 ? threadIdx.y : 0];
  // the window holds the 8 fields as pairs (rho, vx), (vy, vz), (p, bx),
  // (by, bz), the operands of the packed FP32 reconstruction
  typedef typename Pr<T>::V V2;
  V2 w[4][8], nx[4];
  T Fp[8];
  // window of the first face (cell c0): cells c0-4 .. c0+3; the loop shifts
  // one cell in per face, so w[q][1..7] start as cells c0-4 .. c0+2.  Window
  // cells are clamped to the ghost-inclusive range [0, nD-1]: with fewer than
  // 4 ghost layers (nord 4 or 6: TVD, WENO) the outermost taps lie outside
  // it, and those taps are exactly the ones such a stencil never reads.
  const int nD = (D == 1) ? g.ny : g.nz;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int m = 1; m < 8; ++m) {
      const int x = col + max(c0 - 5 + m, 0) * s;
      w[q][m] = Pr<T>::mk(src[2 * q][x], src[2 * q + 1][x]);
    }
    const int x = col + min(c0 + 3, nD - 1) * s;
    nx[q] = Pr<T>::mk(src[2 * q][x], src[2 * q + 1][x]);
  }
  T dx = T(0), rdx = T(0);
  if (D == 1) {
    dx = d.wx[i];
    rdx = d.rwx[i];
  }
#pragma unroll kSweepUnroll
  for (int cd = c0; cd <= c1; ++cd) {  // the face at the low side of cell cd
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int m = 0; m < 7; ++m) w[q][m] = w[q][m + 1];
      w[q][7] = nx[q];
    }
    if (cd < c1) {
      const int x = col + min(cd + 4, nD - 1) * s;
#pragma unroll
      for (int q = 0; q < 4; ++q) nx[q] = Pr<T>::mk(src[2 * q][x], src[2 * q + 1][x]);
    }
    if (D == 1) {
      __syncwarp();  // every lane is done reading the slot refilled here
      if (cd < c1) {
        const int fl = col + cd * s;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const T* fx = d.F[0][q] + fl;
          const uint32_t sp = (uint32_t)__cvta_generic_to_shared(&xs[cd & 1][q][tx]);
          if (sizeof(T) == 4)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sp), "l"(fx) : "memory");
          else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sp), "l"(fx) : "memory");
          if (xlast) {
            const uint32_t sq = (uint32_t)__cvta_generic_to_shared(&xs[cd & 1][q][tx + 32]);
            if (sizeof(T) == 4)
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sq), "l"(fx + 1) : "memory");
            else
              asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sq), "l"(fx + 1) : "memory");
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");  // one group per face, empty on the last
    } else {
      if (cd < c1) {
        const int c = col + cd * s;
        const T* gsrc[18] = {d.dU[0] + c, d.dU[1] + c, d.dU[2] + c, d.dU[3] + c, d.dU[4] + c, d.dU[5] + c,
                             d.dU[6] + c, d.dU[7] + c, d.rho + c,   d.vx + c,    d.vy + c,    d.vz + c,
                             d.p + c,     d.q[0] + c, d.q[1] + c, d.q[2] + c, d.q[3] + c, d.q[4] + c};
        const int nz = (form >= 0) ? 18 : 13;
#pragma unroll
        for (int a = 0; a < 18; ++a) {
          if (a < nz) {
            const uint32_t sp = (uint32_t)__cvta_generic_to_shared(&zs[cd & 1][a][tx]);
            if (sizeof(T) == 4)
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sp), "l"(gsrc[a]) : "memory");
            else
              asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sp), "l"(gsrc[a]) : "memory");
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    T L[8], R[8], F[8];
    if constexpr (std::is_same<T, float>::value && is_pdm(RECON) && MHD_RECON_PACKED) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 lr0, lr1;
        pdm_pair_states<RECON>(w[q], P.pdmb, lr0, lr1);
        L[2 * q] = lr0.x; R[2 * q] = lr0.y;
        L[2 * q + 1] = lr1.x; R[2 * q + 1] = lr1.y;
      }
    } else if constexpr (std::is_same<T, float>::value && is_weno(RECON)) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 l, r;
        weno_both<RECON>(w[q][1], w[q][2], w[q][3], w[q][4], w[q][5], w[q][6], P, l, r);
        L[2 * q] = l.x; R[2 * q] = r.x;
        L[2 * q + 1] = l.y; R[2 * q + 1] = r.y;
      }
    } else {
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        T wv[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) wv[m] = (v & 1) ? w[v >> 1][m].y : w[v >> 1][m].x;
        recon_win<T, RECON, 0>(wv, P, L[v], R[v]);
      }
    }
    face_flux<D>(L, R, d, F);
    if (cd > c0) {
      const int cc = cd - 1;
      const int c = col + cc * s;
      T dF[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) dF[q] = F[q] - Fp[q];
      if (D == 1) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // the group of cell cc (one face old)
        __syncwarp();
        const T dy = d.wy[cc], rdy = d.rwy[cc];
        if (xin) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const T* x = &xs[cc & 1][q][tx];
            d.dU[q][c] = Ops<T>::dc(x[xh] - x[0], dx, rdx) + Ops<T>::dc(dF[q], dy, rdy);
          }
        }
      } else {
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // this lane's copies of cell cc
        if (xin) {
          const T* zv = &zs[cc & 1][0][tx];
          T du[8], pv[5], qv[5];
#pragma unroll
          for (int q = 0; q < 8; ++q) du[q] = zv[q * 32];
#pragma unroll
          for (int q = 0; q < 5; ++q) pv[q] = zv[(8 + q) * 32];
#pragma unroll
          for (int q = 0; q < 5; ++q) qv[q] = (form >= 0) ? zv[(13 + q) * 32] : T(0);
          cell_update_vals<T, false>(d, c, cc, dF, du, pv, qv, form, cw, den);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) Fp[q] = F[q];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// -------------------------------------------------------------------- EMF
// Edge EMF of family E (0: ei along x, 1: ej along y, 2: ek along z) at the
// edge whose upper cell is c (get_eijk_LFM, 1754-1856).  a1 = E+1, a2 = E+2
// (cyclic): v1 = v_a1, v2 = v_a2; b1 = B_a1 reconstructed along a2 and
// upwinded by sign(v2); b2 = B_a2 reconstructed along a1, upwinded by sign(v1).
// E of an edge from its corner velocities, the one-sided face states of b1
// and b2 and eta = 0.25 (vf[c-s1-s2] + vf[c-s2] + vf[c] + vf[c-s1]): the
// upwinded convective term plus the resistive term (metric: g_e and |dl_e|).
template <typename T>
__device__ __forceinline__ T eta4(T a, T b, T c, T e) {
  return T(0.25) * (a + b + c + e);
}
template <typename T, int E, bool M, typename I>
__device__ __forceinline__ T emf_value(const Dev<T>& d, I c, T v1av, T v2av, T b1l, T b1r, T b2l, T b2r, T eta) {
  const T b1u = ge0(v2av) ? b1l : b1r;
  const T b2u = ge0(v1av) ? b2l : b2r;
  const T e = -v1av * b2u + v2av * b1u;
  if (M)  // E.dl: g_e * (convective term) + eta |dl_e| * (resistive term)
    return d.m.ge[E][c] * e + eta * d.m.dl[E][c] * (b1l + b2r - b1r - b2l);
  return e + eta * (b1l + b2r - b1r - b2l);
}

// One edge of family E from global memory (upper cell index c).
template <typename T, int RECON, int E, bool M>
__device__ __forceinline__ void emf_edge(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, long long c) {
  const long long st[3] = {1, (long long)d.g.px, d.g.plane};
  constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
  const long long s1 = st[A1], s2 = st[A2];
  const T* vel[3] = {in.vx, in.vy, in.vz};
  const T* fb[3] = {in.bi, in.bj, in.bk};
  const T v1av = corner_vel<T, RECON>(vel[A1], c, s1, s2, P);
  const T v2av = corner_vel<T, RECON>(vel[A2], c, s1, s2, P);
  T b1l, b1r, b2l, b2r;
  recon_edge<T, RECON>(fb[A1], c, s2, P, b1l, b1r);
  recon_edge<T, RECON>(fb[A2], c, s1, P, b2l, b2r);
  const T* vf = d.vf;
  const T eta = eta4(vf[c - s1 - s2], vf[c - s2], vf[c], vf[c - s1]);
  d.E[E][c] = emf_value<T, E, M>(d, c, v1av, v2av, b1l, b1r, b2l, b2r, eta);
}

template <typename T, int RECON, int E, bool M>
__global__ void k_emf(Dev<T> d, Inp<T> in, Prm<T> P) {
  const Geom& g = d.g;
  int i = blockIdx.x * blockDim.x + threadIdx.x + g.ng;
  int j = blockIdx.y * blockDim.y + threadIdx.y + g.ng;
  int k = blockIdx.z + g.ng;
  int ni = g.nx0 + (E != 0), nj = g.ny0 + (E != 1), nk = g.nz0 + (E != 2);
  if (i >= g.ng + ni || j >= g.ng + nj || k >= g.ng + nk) return;
  emf_edge<T, RECON, E, M>(d, in, P, idx3<T>(g, i, j, k));
}

// Shared-memory tiled EMF of family E for PDM (the default deck's
// reconstruction).  A block stages v_a1 and v_a2 of its tile of edges plus a
// 4-cell halo in the transverse (a1, a2) plane, computes the first pass of
// interp2_pdm (8-tap along a1, mhd3d3.f90:926-989) once per (a1 face, a2 row)
// into shared memory, and each edge then takes the second pass along a2, the
// limiters (corner_pdm), the upwinded face-B reconstructions and the Alfven
// resistivity term exactly as k_emf does.  Tile (TX, TY, TZ) in edges.
//
// A transverse axis of an edge family holds n0 + 1 edges.  For ej and ek,
// when that count is one more than a multiple of the tile (n0 a multiple of
// 32 along x, of 8 along the other transverse axis), the last tile of the
// axis is one edge wider instead of a block of its own holding a single edge
// row: emf_edge_tiles() counts the tiles, and k_emf_pdm runs the widened
// variant of emf_pdm_tile in those blocks.  ei keeps the plain count (its
// halo-padded tile is large, so a wider variant would cost shared memory and
// occupancy in every block).
// Depth of the ej / ek plane tiles along their second transverse axis
// (32 x kPT edges, 32 kPT threads); compile-time knob.
#ifndef MHD_EMF_PLANE
#define MHD_EMF_PLANE 8
#endif
constexpr int kPT = MHD_EMF_PLANE;
constexpr bool emf_merges(int E, int axis) { return E != 0 && axis != E; }

__host__ __device__ constexpr int emf_edge_tiles(int ext, int t, bool merge) {
  return (merge && t > 1 && ext > t && ext % t == 1) ? ext / t : (ext + t - 1) / t;
}

// dynamic shared memory of k_emf_pdm: enough for the widest tile it runs
template <typename T, int E, int TX, int TY, int TZ>
constexpr size_t emf_pdm_smem() {
  constexpr int WX = TX + emf_merges(E, 0), WY = TY + emf_merges(E, 1), WZ = TZ + emf_merges(E, 2);
  constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
  constexpr int HX = (E == 0) ? 0 : 4, HY = (E == 1) ? 0 : 4, HZ = (E == 2) ? 0 : 4;
  constexpr int NV = (WX + 2 * HX) * (WY + 2 * HY) * (WZ + 2 * HZ);
  constexpr int TE = (E == 0) ? WX : (E == 1) ? WY : WZ;
  constexpr int T1 = (A1 == 0) ? WX : (A1 == 1) ? WY : WZ;
  constexpr int T2 = (A2 == 0) ? WX : (A2 == 1) ? WY : WZ;
  return sizeof(T) * (2 * NV + 2 * TE * T1 * (T2 + 8));
}

inline dim3 emf_grid(int E, const Geom& g, int tx, int ty, int tz) {
  const int ex = g.nx0 + (E != 0), ey = g.ny0 + (E != 1), ez = g.nz0 + (E != 2);
  return dim3(emf_edge_tiles(ex, tx, emf_merges(E, 0)), emf_edge_tiles(ey, ty, emf_merges(E, 1)),
              emf_edge_tiles(ez, tz, emf_merges(E, 2)));
}

template <typename T, int RECON, int E, int TX, int TY, int TZ, bool M>
__device__ __forceinline__ void emf_pdm_tile(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, int ox, int oy,
                                             int oz) {
  constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
  constexpr int HX = (E == 0) ? 0 : 4, HY = (E == 1) ? 0 : 4, HZ = (E == 2) ? 0 : 4;
  constexpr int SX = TX + 2 * HX, SY = TY + 2 * HY, SZ = TZ + 2 * HZ;
  constexpr int NV = SX * SY * SZ;
  constexpr int SE = (E == 0) ? 1 : (E == 1) ? SX : SX * SY;
  constexpr int S1 = (A1 == 0) ? 1 : (A1 == 1) ? SX : SX * SY;
  constexpr int S2 = (A2 == 0) ? 1 : (A2 == 1) ? SX : SX * SY;
  constexpr int TE = (E == 0) ? TX : (E == 1) ? TY : TZ;
  constexpr int T1 = (A1 == 0) ? TX : (A1 == 1) ? TY : TZ;
  constexpr int T2 = (A2 == 0) ? TX : (A2 == 1) ? TY : TZ;
  constexpr int NG = TE * T1 * (T2 + 8);
  // first-pass layout with the x-mapped index contiguous (conflict-free banks)
  constexpr int R2 = T2 + 8;
  constexpr int GE = (E == 0) ? 1 : (A1 == 0) ? T1 : R2;
  constexpr int G1 = (E == 0) ? TE : (A1 == 0) ? 1 : R2 * TE;
  constexpr int G2 = (E == 0) ? TE * T1 : (A1 == 0) ? T1 * TE : 1;
  typedef Pr<T> Q;
  typedef typename Q::V V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* sv = reinterpret_cast<V*>(smem_raw);  // [NV] (v_a1, v_a2) pairs
  V* sg = sv + NV;                         // [NG] first-pass interpolant pairs
  const Geom& g = d.g;
  const T* vel[3] = {in.vx, in.vy, in.vz};
  const T* v1 = vel[A1];
  const T* v2 = vel[A2];
  // stage v_a1, v_a2: one flat pass over the (x, y, z) tile, x fastest, so
  // every lane has an element even when a row is not a multiple of 32 wide
  for (int t = threadIdx.x; t < NV; t += blockDim.x) {
    const int lx = t % SX, row = t / SX;
    const int ly = row % SY, lz = row / SY;
    const int gx = ox - HX + lx, gy = oy - HY + ly, gz = oz - HZ + lz;
    T a = T(0), b = T(0);
    if (gx < g.nx && gy < g.ny && gz < g.nz) {
      const int gi = gx + g.px * (gy + g.py * gz);
      a = v1[gi];
      b = v2[gi];
    }
    sv[t] = Q::mk(a, b);
  }
  __syncthreads();
  // first pass of interp2_pdm over (e, f1, r2), flat with the x-mapped index fastest
  constexpr int NX = (E == 0) ? TE : (A1 == 0) ? T1 : R2;   // x-mapped extent
  for (int t = threadIdx.x; t < NG; t += blockDim.x) {
    const int ix = t % NX, row = t / NX;
    int e, f1, r2;
    if (E == 0) {
      e = ix; f1 = row % T1; r2 = row / T1;
    } else if (A1 == 0) {
      f1 = ix; e = row % TE; r2 = row / TE;
    } else {
      r2 = ix; e = row % TE; f1 = row / TE;
    }
    const int b0 = e * SE + f1 * S1 + r2 * S2;
    const int gi = e * GE + f1 * G1 + r2 * G2;
    const V* a = sv + b0;
    sg[gi] = tap8p(a[0], a[S1], a[2 * S1], a[3 * S1], a[4 * S1], a[5 * S1], a[6 * S1], a[7 * S1]);
  }
  __syncthreads();
  const int n0[3] = {g.nx0, g.ny0, g.nz0};
  const int lim[3] = {g.ng + n0[0] + (E != 0), g.ng + n0[1] + (E != 1), g.ng + n0[2] + (E != 2)};
  const int st[3] = {1, g.px, (int)g.plane};
  const T* fb[3] = {in.bi, in.bj, in.bk};
  for (int t = threadIdx.x; t < TX * TY * TZ; t += blockDim.x) {
    const int lx = t % TX, r = t / TX, ly = r % TY, lz = r / TY;
    const int gx = ox + lx, gy = oy + ly, gz = oz + lz;
    if (gx >= lim[0] || gy >= lim[1] || gz >= lim[2]) continue;
    const int e = (E == 0) ? lx : (E == 1) ? ly : lz;
    const int f1 = (A1 == 0) ? lx : (A1 == 1) ? ly : lz;
    const int f2 = (A2 == 0) ? lx : (A2 == 1) ? ly : lz;
    const int cv = e * SE + (f1 + 4) * S1 + (f2 + 4) * S2;
    const V* gg = sg + e * GE + f1 * G1 + f2 * G2;
    constexpr int GS = G2;
    const V vi = tap8p(gg[0], gg[GS], gg[2 * GS], gg[3 * GS], gg[4 * GS], gg[5 * GS], gg[6 * GS], gg[7 * GS]);
    T v1av, v2av;
    corner_pdm_pair<T, RECON>(sv, cv, S1, S2, vi, P.pdmb, v1av, v2av);
    const int c = gx + g.px * (gy + g.py * gz);
    const int s1 = st[A1], s2 = st[A2];
    T b1l, b1r, b2l, b2r;
    recon_edge<T, RECON>(fb[A1], c, s2, P, b1l, b1r);
    recon_edge<T, RECON>(fb[A2], c, s1, P, b2l, b2r);
    const T* vf = d.vf;
    const T eta = eta4(vf[c - s1 - s2], vf[c - s2], vf[c], vf[c - s1]);
    d.E[E][c] = emf_value<T, E, M>(d, c, v1av, v2av, b1l, b1r, b2l, b2r, eta);
  }
}

// Register budgets of the EMF tiles (resident threads per SM the allocator
// must allow): single grid 2048 (full occupancy); batched 1536 for the plane
// tiles and 1024 for ei, whose shared memory allows 2 blocks anyway (the
// batched kernels carry a grid-table lookup and spill at 32 registers).
// MHD_EMF_FULL_OCC=0 leaves every budget to the compiler.
#ifndef MHD_EMF_FULL_OCC
#define MHD_EMF_FULL_OCC 1
#endif
// FP64 takes 1024 (64 registers): its bound is the FP64 pipe, which a few
// warps fill, and 32 registers spilled 1.4 KB per thread.
template <typename T>
constexpr int emf_min_blocks(int E, int NT, bool B) {
  return !MHD_EMF_FULL_OCC ? 1 : sizeof(T) == 8 ? 1024 / NT : !B ? 2048 / NT : (E == 0 ? 1024 / NT : 1536 / NT);
}
template <typename T, int RECON, int E, int TX, int TY, int TZ, int NT, bool M, bool B>
__global__ void __launch_bounds__(NT, emf_min_blocks<T>(E, NT, B))
    k_emf_pdm(KArg<T, B> ka, Inp<T> in0, Prm<T> P) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Inp<T> in = B ? state_view(d) : in0;
  const Geom& g = d.g;
  const int ox = g.ng + bb.y * TX, oy = g.ng + bb.z * TY, oz = g.ng + bb.w * TZ;
  if constexpr (E == 0) {
    emf_pdm_tile<T, RECON, E, TX, TY, TZ, M>(d, in, P, ox, oy, oz);
  } else {
    // transverse axes a1, a2: is this block the widened last tile of the axis?
    constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
    const int n0[3] = {g.nx0, g.ny0, g.nz0};
    const int org[3] = {ox - g.ng, oy - g.ng, oz - g.ng};
    constexpr int tl[3] = {TX, TY, TZ};
    const bool w1 = tl[A1] > 1 && n0[A1] - org[A1] == tl[A1];
    const bool w2 = tl[A2] > 1 && n0[A2] - org[A2] == tl[A2];
    constexpr int X1 = A1 == 0, Y1 = A1 == 1, Z1 = A1 == 2, X2 = A2 == 0, Y2 = A2 == 1, Z2 = A2 == 2;
    if (w1 && w2)
      emf_pdm_tile<T, RECON, E, TX + X1 + X2, TY + Y1 + Y2, TZ + Z1 + Z2, M>(d, in, P, ox, oy, oz);
    else if (w1)
      emf_pdm_tile<T, RECON, E, TX + X1, TY + Y1, TZ + Z1, M>(d, in, P, ox, oy, oz);
    else if (w2)
      emf_pdm_tile<T, RECON, E, TX + X2, TY + Y2, TZ + Z2, M>(d, in, P, ox, oy, oz);
    else
      emf_pdm_tile<T, RECON, E, TX, TY, TZ, M>(d, in, P, ox, oy, oz);
  }
}

template <typename T, int RECON, int E, int TX, int TY, int TZ, int NT, bool M>
void launch_emf_pdm(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, cudaStream_t st) {
  constexpr size_t bytes = emf_pdm_smem<T, E, TX, TY, TZ>();
  static PerDevice attr;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    cudaFuncSetAttribute(k_emf_pdm<T, RECON, E, TX, TY, TZ, NT, M, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)bytes);
    attr.mark(bit);
  }
  k_emf_pdm<T, RECON, E, TX, TY, TZ, NT, M, false><<<emf_grid(E, d.g, TX, TY, TZ), NT, bytes, st>>>(one(d), in, P);
}

// ------------------------------------------------------ streamed PDM EMF
// The PDM EMF of one family as slice streams.  A block owns a patch of edges
// across the stream axis S (32 lanes along x times NW warps) and walks S over
// a segment of edge positions.  Each step copies one new cell slice of
// (v_a1, v_a2), of the face-B component that is reconstructed across the
// slice and of vf into shared-memory rings, asynchronously and a step ahead,
// and each thread computes the edge of its column at the current position:
// every cell is staged once per segment (no halo re-reads along S, no
// per-tap index arithmetic), and the taps along S come from a register window
// or the ring.
//   ei (E = 0): lanes along x (the edge axis), warps along y = a1, S = z = a2.
//   ek (E = 2): lanes along x = a1, warps along z (the edge axis), S = y = a2.
//   ej (E = 1): lanes along x = a2, warps along y (the edge axis), S = z = a1.
// With S = a2 the first pass of interp2_pdm (8 taps along a1) runs inside
// the new slice and the second pass (along S) on a register window of eight
// first-pass values; with S = a1 the first pass runs across eight ring slices
// into a per-warp row (32 columns plus the 8-column halo) and the second pass
// along x reads that row.  The face-B component reconstructed along S is a
// register window of eight values of the thread's own column.  The
// arithmetic per edge is emf_pdm_tile's and k_emf's (same operands, same
// order), so all three give the same bits.  The in-slice transverse axis
// holds n0 + 1 edges; the tiles cover the first n0 and k_emf_rows the last.
template <typename T, int E, int NW>
struct EmfStream {
  static constexpr bool SA2 = (E != 1);             // S = a2 (ei, ek) or S = a1 (ej)
  static constexpr int NT = 32 * NW;
  static constexpr int C = (E == 0) ? 32 : 40;      // slice columns (x), with the x halo for ek / ej
  static constexpr int R = (E == 0) ? NW + 8 : NW;  // slice rows, with the y halo for ei
  static constexpr int NS = R * C;                  // cells per slice
  static constexpr int NE = (NS + NT - 1) / NT;     // slice cells each thread copies
  static constexpr int TS = (E == 0) ? C : 1;       // in-slice stride of the transverse axis
  static constexpr int DV = SA2 ? 8 : 16;           // (v_a1, v_a2) ring depth
  static constexpr size_t smem =
      sizeof(typename Pr<T>::V) * (DV * NS + (SA2 ? 0 : NW * C)) + sizeof(T) * (2 * NS + 4 * NS);
};

template <typename T>
__device__ __forceinline__ void cp_async_zfill(uint32_t dst, const T* src, bool ok) {
  const int n = ok ? (int)sizeof(T) : 0;  // 0: nothing is read, the element is zeroed
  if (sizeof(T) == 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

#ifndef MHD_EMF_STREAM_MINB
#define MHD_EMF_STREAM_MINB 3
#endif
template <typename T, int RECON, int E, int NW, bool M, bool B>
__global__ void __launch_bounds__(32 * NW, MHD_EMF_STREAM_MINB)
    k_emf_stream(KArg<T, B> ka, Inp<T> in0, Prm<T> P) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Inp<T> in = B ? state_view(d) : in0;
  typedef EmfStream<T, E, NW> K;
  typedef Pr<T> Q;
  typedef typename Q::V V;
  constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
  constexpr int C = K::C, NS = K::NS, TS = K::TS, DV = K::DV, NT = K::NT, NE = K::NE;
  constexpr bool SA2 = K::SA2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* vr = reinterpret_cast<V*>(smem_raw);              // [DV][NS] (v_a1, v_a2)
  V* gr = vr + DV * NS;                                // ej: [NW][C] first-pass rows
  T* br = reinterpret_cast<T*>(gr + (SA2 ? 0 : NW * C));  // [2][NS] face B across the slice
  T* fr = br + 2 * NS;                                 // [4][NS] vf
  const Geom& g = d.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = g.ng + 32 * bb.y;   // first x of the tile (edge or cell index)
  const int w0 = g.ng + NW * bb.z;   // first index along the warp axis (y, z, y)
  const int nS0 = (E == 2) ? g.ny0 : g.nz0;     // interior cells along S
  const int nSg = (E == 2) ? g.ny : g.nz;
  const int nW0 = (E == 2) ? g.nz0 : g.ny0;
  const int seg = d.eseg[E];
  const int s_lo = g.ng + seg * bb.w;
  const int s_hi = (bb.w == emf_stream_segs(nS0, seg) - 1) ? g.ng + nS0 : s_lo + seg - 1;
  const int SS = (E == 2) ? g.px : (int)g.plane;  // global stride along S
  const int ox = x0 + lane, ow = w0 + warp;
  const bool own = ox < g.ng + g.nx0 && ow < g.ng + nW0;
  const int obase = ox + ((E == 2) ? (int)g.plane * ow : g.px * ow);  // own column at S = 0
  const int oi = (E == 0) ? (warp + 4) * C + lane : warp * C + lane + 4;  // own cell in a slice
  // the slice cells this thread copies: global offset at S = 0 and bounds
  int go[NE];
  bool gok[NE];
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    const int idx = tid + k * NT, r = idx / C, q = idx - r * C;
    int x, w;
    if (E == 0) { x = x0 + q; w = w0 - 4 + r; }
    else { x = x0 - 4 + q; w = w0 + r; }
    const int nw = (E == 2) ? g.nz : g.ny;
    gok[k] = idx < NS && (unsigned)x < (unsigned)g.nx && (unsigned)w < (unsigned)nw;
    go[k] = x + ((E == 2) ? (int)g.plane * w : g.px * w);
  }
  const T* vel[3] = {in.vx, in.vy, in.vz};
  const T* fb[3] = {in.bi, in.bj, in.bk};
  const T* v1 = vel[A1];
  const T* v2 = vel[A2];
  const T* bst = SA2 ? fb[A2] : fb[A1];  // reconstructed across the slice (staged)
  const T* bwn = SA2 ? fb[A1] : fb[A2];  // reconstructed along S (own-column window)
  const T* vf = d.vf;
  const uint32_t vr_s = (uint32_t)__cvta_generic_to_shared(vr);
  const uint32_t br_s = (uint32_t)__cvta_generic_to_shared(br);
  const uint32_t fr_s = (uint32_t)__cvta_generic_to_shared(fr);
  auto vslot = [&](int s) { return (s - s_lo + 4) & (DV - 1); };
  // copy slice s of the selected arrays into their ring slots
  auto stage = [&](int s, bool with_v, bool with_bf) {
    const bool sok = (unsigned)s < (unsigned)nSg;
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      if (k * NT + tid < NS) {
        const int idx = tid + k * NT;
        const bool ok = gok[k] && sok;
        const int o = ok ? go[k] + s * SS : 0;
        if (with_v) {
          const uint32_t a = vr_s + (uint32_t)((vslot(s) * NS + idx) * sizeof(V));
          cp_async_zfill<T>(a, v1 + o, ok);
          cp_async_zfill<T>(a + sizeof(T), v2 + o, ok);
        }
        if (with_bf) {
          cp_async_zfill<T>(br_s + (uint32_t)(((s & 1) * NS + idx) * sizeof(T)), bst + o, ok);
          cp_async_zfill<T>(fr_s + (uint32_t)(((s & 3) * NS + idx) * sizeof(T)), vf + o, ok);
        }
      }
    }
  };
  // prologue: v slices s_lo-4 .. s_lo+3, face B at s_lo, vf at s_lo-1 and s_lo
#pragma unroll 1
  for (int m = 0; m < 8; ++m) stage(s_lo - 4 + m, true, m == 3 || m == 4);
  asm volatile("cp.async.commit_group;" ::: "memory");
  T bw[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) bw[m] = own ? bwn[obase + (s_lo - 4 + m) * SS] : T(0);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // first pass along a1 inside slice s (S = a2)
  auto first_a1 = [&](int s) {
    const V* a = vr + vslot(s) * NS + oi;
    return tap8p(a[-4 * TS], a[-3 * TS], a[-2 * TS], a[-TS], a[0], a[TS], a[2 * TS], a[3 * TS]);
  };
  V gw[8];
  if constexpr (SA2) {
#pragma unroll
    for (int m = 0; m < 8; ++m) gw[m] = first_a1(s_lo - 4 + m);
    __syncthreads();  // the first step refills the slot of slice s_lo - 4
  }
  // two steps a turn: half of the windows' register moves (256^3 stage 2301 -> 2285 us; four a turn spill)
#pragma unroll 2
  for (int s = s_lo; s <= s_hi; ++s) {
    const bool more = s < s_hi;
    T bnext = T(0);
    if (more) {  // inputs of the next step
      stage(s + 4, true, false);
      stage(s + 1, false, true);
      if (own) bnext = bwn[obase + (s + 4) * SS];
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    V vi;
    if constexpr (SA2) {
      vi = tap8p(gw[0], gw[1], gw[2], gw[3], gw[4], gw[5], gw[6], gw[7]);
    } else {
      // first pass along a1 = S across the ring into this warp's row
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r2 = lane + 32 * h;
        if (r2 < C) {
          const int col = warp * C + r2;
          gr[col] = tap8p(vr[vslot(s - 4) * NS + col], vr[vslot(s - 3) * NS + col], vr[vslot(s - 2) * NS + col],
                             vr[vslot(s - 1) * NS + col], vr[vslot(s) * NS + col], vr[vslot(s + 1) * NS + col],
                             vr[vslot(s + 2) * NS + col], vr[vslot(s + 3) * NS + col]);
        }
      }
      __syncwarp();
      const V* gg = gr + warp * C + lane;
      vi = tap8p(gg[0], gg[1], gg[2], gg[3], gg[4], gg[5], gg[6], gg[7]);
    }
    // the 12 corner cells, (d1, d2) from the upper cell
    const V* sm2 = vr + vslot(s - 2) * NS + oi;
    const V* sm1 = vr + vslot(s - 1) * NS + oi;
    const V* s00 = vr + vslot(s) * NS + oi;
    const V* sp1 = vr + vslot(s + 1) * NS + oi;
    V m11, m21, m12, m01, p11, m02, m10, m20, m1p, c0, p10, p01;
    if constexpr (SA2) {  // d1 in the slice (stride TS), d2 across slices
      m11 = sm1[-TS]; m21 = sm1[-2 * TS]; m12 = sm2[-TS]; m01 = sm1[0]; p11 = sm1[TS]; m02 = sm2[0];
      m10 = s00[-TS]; m20 = s00[-2 * TS]; m1p = sp1[-TS]; c0 = s00[0]; p10 = s00[TS]; p01 = sp1[0];
    } else {  // d1 across slices, d2 in the slice (stride 1)
      m11 = sm1[-1]; m21 = sm2[-1]; m12 = sm1[-2]; m01 = s00[-1]; p11 = sp1[-1]; m02 = s00[-2];
      m10 = sm1[0]; m20 = sm2[0]; m1p = sm1[1]; c0 = s00[0]; p10 = sp1[0]; p01 = s00[1];
    }
    T v1av, v2av;
    corner_pdm_vals2<T, RECON>(m11, m21, m12, m01, p11, m02, m10, m20, m1p, c0, p10, p01, vi, P.pdmb, v1av, v2av);
    // face B: across the slice from the staged slice, along S from the window
    constexpr int BS = SA2 ? TS : 1;
    const T* bb = br + (s & 1) * NS + oi;
    T sl, sr, wl, wr;
    recon_pdm8<T, RECON, true>(bb[-4 * BS], bb[-3 * BS], bb[-2 * BS], bb[-BS], bb[0], bb[BS], bb[2 * BS], bb[3 * BS],
                               P.pdmb, sl, sr);
    recon_pdm8<T, RECON, true>(bw[0], bw[1], bw[2], bw[3], bw[4], bw[5], bw[6], bw[7], P.pdmb, wl, wr);
    const T* f0 = fr + (s & 3) * NS + oi;
    const T* fm = fr + ((s - 1) & 3) * NS + oi;
    T eta;
    if constexpr (SA2) eta = eta4(fm[-TS], fm[0], f0[0], f0[-TS]);  // s1 in the slice, s2 = S
    else eta = eta4(fm[-1], f0[-1], f0[0], fm[0]);                  // s1 = S, s2 in the slice
    if (own) {
      const int c = obase + s * SS;
      // b1 = B_a1 along a2, b2 = B_a2 along a1
      d.E[E][c] = SA2 ? emf_value<T, E, M>(d, c, v1av, v2av, wl, wr, sl, sr, eta)
                      : emf_value<T, E, M>(d, c, v1av, v2av, sl, sr, wl, wr, eta);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (more) {
#pragma unroll
      for (int m = 0; m < 7; ++m) bw[m] = bw[m + 1];
      bw[7] = bnext;
      if constexpr (SA2) {
#pragma unroll
        for (int m = 0; m < 7; ++m) gw[m] = gw[m + 1];
        gw[7] = first_a1(s + 4);
      }
    }
  }
}

// The (n0+1)-th edge row of the in-slice transverse axis of each streamed
// family, as thin shared-memory tiles of emf_pdm_tile in one launch of
// 256-thread blocks: ei at y = ny0 in 32 x 1 x 8 tiles (x, y, z edges), ek
// at x = nx0 in 1 x 32 x 8 tiles, ej at x = nx0 in 1 x 8 x 32 tiles.
struct EmfRows {
  int bi, bk, bj;  // blocks of the three planes
  __host__ __device__ explicit EmfRows(const Geom& g)
      : bi(((g.nx0 + 31) / 32) * ((g.nz0 + 8) / 8)), bk(((g.ny0 + 32) / 32) * ((g.nz0 + 7) / 8)),
        bj(((g.ny0 + 7) / 8) * ((g.nz0 + 32) / 32)) {}
  __host__ __device__ int blocks() const { return bi + bk + bj; }
};
template <typename T>
constexpr size_t emf_rows_smem() {
  constexpr size_t a = emf_pdm_smem<T, 0, 32, 1, 8>(), b = emf_pdm_smem<T, 2, 1, 32, 8>(),
                   c = emf_pdm_smem<T, 1, 1, 8, 32>();
  return a > b ? (a > c ? a : c) : (b > c ? b : c);
}
template <typename T, int RECON, bool M, bool B>
__global__ void __launch_bounds__(256) k_emf_rows(KArg<T, B> ka, Inp<T> in0, Prm<T> P) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Inp<T> in = B ? state_view(d) : in0;
  const Geom& g = d.g;
  const EmfRows r(g);
  int b = bb.y;
  if (b < r.bi) {
    const int nbx = (g.nx0 + 31) / 32, bx = b % nbx, bz = b / nbx;
    emf_pdm_tile<T, RECON, 0, 32, 1, 8, M>(d, in, P, g.ng + 32 * bx, g.ng + g.ny0, g.ng + 8 * bz);
    return;
  }
  b -= r.bi;
  if (b < r.bk) {
    const int nby = (g.ny0 + 32) / 32, by = b % nby, bz = b / nby;
    emf_pdm_tile<T, RECON, 2, 1, 32, 8, M>(d, in, P, g.ng + g.nx0, g.ng + 32 * by, g.ng + 8 * bz);
    return;
  }
  b -= r.bk;
  const int nby = (g.ny0 + 7) / 8, by = b % nby, bz = b / nby;
  emf_pdm_tile<T, RECON, 1, 1, 8, 32, M>(d, in, P, g.ng + g.nx0, g.ng + 8 * by, g.ng + 32 * bz);
}

// blocks of streamed family E on one grid (x tiles, warp-axis tiles, segments)
inline dim3 emf_stream_grid(int E, const Geom& g, int seg) {
  const int nS0 = (E == 2) ? g.ny0 : g.nz0, nW0 = (E == 2) ? g.nz0 : g.ny0;
  return dim3((g.nx0 + 31) / 32, (nW0 + MHD_EMF_NW - 1) / MHD_EMF_NW,
              emf_stream_segs(nS0, seg));
}
template <typename T, int RECON, int E, bool M, bool B>
void stream_attr() {
  static PerDevice attr;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    cudaFuncSetAttribute(k_emf_stream<T, RECON, E, MHD_EMF_NW, M, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)EmfStream<T, E, MHD_EMF_NW>::smem);
    attr.mark(bit);
  }
}
template <typename T, int RECON, int E, bool M>
void launch_emf_stream(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, cudaStream_t st) {
  typedef EmfStream<T, E, MHD_EMF_NW> K;
  stream_attr<T, RECON, E, M, false>();
  k_emf_stream<T, RECON, E, MHD_EMF_NW, M, false>
      <<<emf_stream_grid(E, d.g, d.eseg[E]), K::NT, K::smem, st>>>(one(d), in, P);
}

template <typename T, int RECON, bool M>
void emf_pdm_stream(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, cudaStream_t st) {
  launch_emf_stream<T, RECON, 0, M>(d, in, P, st);
  launch_emf_stream<T, RECON, 1, M>(d, in, P, st);
  launch_emf_stream<T, RECON, 2, M>(d, in, P, st);
  static_assert(emf_rows_smem<T>() <= 48 * 1024, "k_emf_rows fits the default shared-memory limit");
  k_emf_rows<T, RECON, M, false><<<EmfRows(d.g).blocks(), 256, emf_rows_smem<T>(), st>>>(one(d), in, P);
}

// ------------------------------------------------------------- WENO EMF
// Shared-memory tiled EMF of family E for WENO5 / MP-WENO5.  The corner
// velocity of get_vav_center2corner (mhd3d3.f90:1925-2049) reconstructs six
// rows of cells along d1 and then the six row results along d2 ("_1"), and
// six columns along d2 and then along d1 ("_0").  Neighbouring edges share
// five of the six rows, so a block stages v_a1 and v_a2 of its tile of edges
// with the stencil halo (3 cells below and 2 above on each transverse axis),
// computes every row and column reconstruction of the tile once into shared
// memory (first pass), and each edge then takes its four second-pass
// reconstructions, the dif-sign quadrant choice and the 4-quadrant mean of
// corner_vel, the upwinded face-B reconstructions and the resistivity term
// of k_emf, with the same operands in the same order.

// An (e, a1, a2) array of edge family E with the x-mapped index fastest, so
// that lanes of a warp touch consecutive words.
template <int E, int DE, int D1, int D2>
struct EdgeLay {
  static constexpr int A1 = (E + 1) % 3;
  static constexpr int N = DE * D1 * D2;
  static constexpr int NX = (E == 0) ? DE : (A1 == 0) ? D1 : D2;
  static constexpr int GE = (E == 0) ? 1 : (A1 == 0) ? D1 : D2;
  static constexpr int G1 = (E == 0) ? DE : (A1 == 0) ? 1 : D2 * DE;
  static constexpr int G2 = (E == 0) ? DE * D1 : (A1 == 0) ? D1 * DE : 1;
  // coordinates of flat index t (t == e * GE + f1 * G1 + f2 * G2)
  __device__ static __forceinline__ void coords(int t, int& e, int& f1, int& f2) {
    const int ix = t % NX, row = t / NX;
    if (E == 0) {
      e = ix; f1 = row % D1; f2 = row / D1;
    } else if (A1 == 0) {
      f1 = ix; e = row % DE; f2 = row / DE;
    } else {
      f2 = ix; e = row % DE; f1 = row / DE;
    }
  }
};

template <typename T, int E, int TX, int TY, int TZ>
struct EmfWeno {
  static constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
  // staged cells: the edge axis without halo, each transverse axis [-3, T+2)
  static constexpr int LX = (E == 0) ? 0 : 3, LY = (E == 1) ? 0 : 3, LZ = (E == 2) ? 0 : 3;
  static constexpr int SX = TX + ((E == 0) ? 0 : 5), SY = TY + ((E == 1) ? 0 : 5), SZ = TZ + ((E == 2) ? 0 : 5);
  static constexpr int NV = SX * SY * SZ;
  static constexpr int SE = (E == 0) ? 1 : (E == 1) ? SX : SX * SY;
  static constexpr int S1 = (A1 == 0) ? 1 : (A1 == 1) ? SX : SX * SY;
  static constexpr int S2 = (A2 == 0) ? 1 : (A2 == 1) ? SX : SX * SY;
  static constexpr int TE = (E == 0) ? TX : (E == 1) ? TY : TZ;
  static constexpr int T1 = (A1 == 0) ? TX : (A1 == 1) ? TY : TZ;
  static constexpr int T2 = (A2 == 0) ? TX : (A2 == 1) ? TY : TZ;
  typedef EdgeLay<E, TE, T1, T2 + 5> L1;  // "_1": rows [-3, T2+2) reconstructed along a1 at the a1 faces
  typedef EdgeLay<E, TE, T1 + 5, T2> L0;  // "_0": columns [-3, T1+2) reconstructed along a2 at the a2 faces
  static constexpr int NP = L1::N + L0::N;
  // sv[2][NV] (v_a1, v_a2), then per component: L1, R1 [L1::N], L0, R0 [L0::N]
  static constexpr size_t smem = sizeof(T) * (2 * NV + 4 * NP);
};

template <typename T, int RECON, int E, int TX, int TY, int TZ, int NT, bool M>
__global__ void __launch_bounds__(NT) k_emf_weno(Dev<T> d, Inp<T> in, Prm<T> P) {
  typedef EmfWeno<T, E, TX, TY, TZ> K;
  typedef typename K::L1 L1;
  typedef typename K::L0 L0;
  constexpr int A1 = K::A1, A2 = K::A2, NV = K::NV, NP = K::NP, N1 = L1::N, N0 = L0::N;
  typedef typename Pr<T>::V V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* sv = reinterpret_cast<V*>(smem_raw);  // [NV] (v_a1, v_a2)
  V* sp = sv + NV;                         // L1, R1 [N1], L0, R0 [N0]
  const Geom& g = d.g;
  const int ox = g.ng + blockIdx.x * TX, oy = g.ng + blockIdx.y * TY, oz = g.ng + blockIdx.z * TZ;
  const T* vel[3] = {in.vx, in.vy, in.vz};
  const T* v1 = vel[A1];
  const T* v2 = vel[A2];
  for (int t = threadIdx.x; t < NV; t += blockDim.x) {
    const int lx = t % K::SX, row = t / K::SX;
    const int ly = row % K::SY, lz = row / K::SY;
    const int gx = ox - K::LX + lx, gy = oy - K::LY + ly, gz = oz - K::LZ + lz;
    T a = T(0), b = T(0);
    if (gx < g.nx && gy < g.ny && gz < g.nz) {
      const int gi = gx + g.px * (gy + g.py * gz);
      a = v1[gi];
      b = v2[gi];
    }
    sv[t] = Pr<T>::mk(a, b);
  }
  __syncthreads();
  // first pass: every row ("_1") and column ("_0") reconstruction of the
  // tile, both components; tap q of an entry is the cell at offset q - 3
  for (int u = threadIdx.x; u < NP; u += blockDim.x) {
    int e, f1, f2, step, o1, o2;
    if (u < N1) {  // row f2 - 3 along a2, reconstructed along a1 at the face of cell f1
      L1::coords(u, e, f1, f2);
      step = K::S1;
      o1 = u;
      o2 = N1 + u;
    } else {  // column f1 - 3 along a1, reconstructed along a2 at the face of cell f2
      L0::coords(u - N1, e, f1, f2);
      step = K::S2;
      o1 = 2 * N1 + (u - N1);
      o2 = 2 * N1 + N0 + (u - N1);
    }
    const V* a = sv + e * K::SE + f1 * K::S1 + f2 * K::S2;
    V fl, fr;
    weno_both<RECON>(a[0], a[step], a[2 * step], a[3 * step], a[4 * step], a[5 * step], P, fl, fr);
    sp[o1] = fl;
    sp[o2] = fr;
  }
  __syncthreads();
  const int lim[3] = {g.ng + g.nx0 + (E != 0), g.ng + g.ny0 + (E != 1), g.ng + g.nz0 + (E != 2)};
  const int st[3] = {1, g.px, (int)g.plane};
  const T* fb[3] = {in.bi, in.bj, in.bk};
  for (int t = threadIdx.x; t < TX * TY * TZ; t += blockDim.x) {
    const int lx = t % TX, r = t / TX, ly = r % TY, lz = r / TY;
    const int gx = ox + lx, gy = oy + ly, gz = oz + lz;
    if (gx >= lim[0] || gy >= lim[1] || gz >= lim[2]) continue;
    const int e = (E == 0) ? lx : (E == 1) ? ly : lz;
    const int f1 = (A1 == 0) ? lx : (A1 == 1) ? ly : lz;
    const int f2 = (A2 == 0) ? lx : (A2 == 1) ? ly : lz;
    // dif signs pick the smoother one-sided estimate per quadrant (2056-2106):
    // "_0" (columns, second pass along d1) if |slope along d1| is not the
    // smaller, else "_1" (rows); only that one is evaluated.  v_00 / v_10 are
    // the left states of the L / R stencils, v_01 / v_11 the right states (the
    // left-state formula on the mirrored stencil).
    const V* v = sv + e * K::SE + (f1 + 3) * K::S1 + (f2 + 3) * K::S2;
    constexpr int t1 = K::S1, t2 = K::S2;
    const T* l1 = reinterpret_cast<const T*>(sp + e * L1::GE + f1 * L1::G1 + f2 * L1::G2);           // rows f2 - 3 + m
    const T* l0 = reinterpret_cast<const T*>(sp + 2 * N1 + e * L0::GE + f1 * L0::G1 + f2 * L0::G2);  // columns f1 - 3 + m
    // one quadrant: cell q, outward cells along d1 and d2, first-pass arrays
    // (L or R) and the direction the stencil runs
    auto quad = [&](const V q, const V o1, const V o2, bool rgt, bool mirror) -> V {
      const bool bx = abs_ge(o1.x - q.x, o2.x - q.x), by = abs_ge(o1.y - q.y, o2.y - q.y);
      const T* ax = bx ? l0 + (rgt ? 2 * N0 : 0) : l1 + (rgt ? 2 * N1 : 0);
      const T* ay = (by ? l0 + (rgt ? 2 * N0 : 0) : l1 + (rgt ? 2 * N1 : 0)) + 1;
      int gx2 = 2 * (bx ? L0::G1 : L1::G2), gy2 = 2 * (by ? L0::G1 : L1::G2);
      if (mirror) {
        ax += 5 * gx2; ay += 5 * gy2;
        gx2 = -gx2; gy2 = -gy2;
      }
      return weno_side<V, RECON>(Pr<T>::mk(ax[0], ay[0]), Pr<T>::mk(ax[gx2], ay[gy2]),
                                Pr<T>::mk(ax[2 * gx2], ay[2 * gy2]), Pr<T>::mk(ax[3 * gx2], ay[3 * gy2]),
                                Pr<T>::mk(ax[4 * gx2], ay[4 * gy2]), P);
    };
    const V v00 = quad(v[-t1 - t2], v[-2 * t1 - t2], v[-t1 - 2 * t2], false, false);
    const V v10 = quad(v[-t2], v[t1 - t2], v[-2 * t2], true, false);
    const V v01 = quad(v[-t1], v[-2 * t1], v[-t1 + t2], false, true);
    const V v11 = quad(v[0], v[t1], v[t2], true, true);
    const T v1av = T(0.25) * (v00.x + v01.x + v10.x + v11.x);
    const T v2av = T(0.25) * (v00.y + v01.y + v10.y + v11.y);
    const int c = gx + g.px * (gy + g.py * gz);
    const int s1 = st[A1], s2 = st[A2];
    T b1l, b1r, b2l, b2r;
    recon_edge<T, RECON>(fb[A1], c, s2, P, b1l, b1r);
    recon_edge<T, RECON>(fb[A2], c, s1, P, b2l, b2r);
    const T* vf = d.vf;
    const T eta = eta4(vf[c - s1 - s2], vf[c - s2], vf[c], vf[c - s1]);
    d.E[E][c] = emf_value<T, E, M>(d, c, v1av, v2av, b1l, b1r, b2l, b2r, eta);
  }
}

// ------------------------------------------------------------- FP64 EMF
// The FP64 pipe (2 lanes per SM and cycle) bounds the FP64 edge EMF: a WENO
// state costs it about 100 operations, a PDM interpolant 17.  All three families
// run as one launch of run-time tiles, so that nothing is computed for padding
// and a small grid still reaches every SM, and the states of a tile are spread
// one per thread.
//  - WENO across (a1, a2): at most 9 x 9 edges (6 x 6 while the launch is short of
//    blocks), the n0 + 1 edges of an axis split evenly (17 = 9 + 8).  The first
//    pass reconstructs (t + 5) / t states per edge and direction (1.6 at 9, 2.3
//    at the 4 x 4 tiles before), the second 12 per edge: 4 quadrants of 2
//    components, 2 states of 2 face-B components.
//  - PDM: at most 4 x 33 edges; only the first pass of the interpolant has a halo,
//    along a2: (t2 + 8) / t2 interpolants per edge, 1.25 at 33 (3 in the 4 x 4 ei
//    tiles before, 2 in the 8-deep planes).
//  - Along the edge axis te edges without halo: 4, fewer while there are less
//    than three blocks per SM.
struct Tile64 {
  int te, t1, t2;     // edges per tile along the edge axis, a1, a2
  int ne, n1, n2;     // edges of the family
  int be, b1, b2;     // tiles
};
struct Tiles64 {
  Tile64 f[3];
  int blocks[3];
  size_t smem;
  static int split(int n, int most) {
    const int tiles = (n + most - 1) / most;
    return (n + tiles - 1) / tiles;
  }
  // doubles of shared memory of a tile: cells, first-pass states, second-pass results
  static size_t words(bool weno, int te, int t1, int t2) {
    return weno ? (size_t)te * (2 * (t1 + 5) * (t2 + 5) + 4 * (t1 * (t2 + 5) + (t1 + 5) * t2) + 12 * t1 * t2)
                : (size_t)te * (2 * (t1 + 8) * (t2 + 8) + 2 * t1 * (t2 + 8) + 6 * t1 * t2);
  }
  Tiles64(bool weno, const Geom& g) {
    const int n0[3] = {g.nx0, g.ny0, g.nz0};
    const int m1[2] = {weno ? 9 : 4, weno ? 6 : 4}, m2[2] = {weno ? 9 : 33, weno ? 6 : 9};
    int total = 0;
    for (int small = 0; small < 2; ++small)
      for (int te = 4; te >= 1; te /= 2) {
        total = 0;
        smem = 0;
        for (int e = 0; e < 3; ++e) {
          Tile64& t = f[e];
          t.ne = n0[e];
          t.n1 = n0[(e + 1) % 3] + 1;
          t.n2 = n0[(e + 2) % 3] + 1;
          t.te = te;
          t.t1 = split(t.n1, m1[small]);
          t.t2 = split(t.n2, m2[small]);
          t.be = (t.ne + te - 1) / te;
          t.b1 = (t.n1 + t.t1 - 1) / t.t1;
          t.b2 = (t.n2 + t.t2 - 1) / t.t2;
          total += blocks[e] = t.be * t.b1 * t.b2;
          const size_t w = sizeof(double) * words(weno, te, t.t1, t.t2);
          smem = w > smem ? w : smem;
        }
        if (total >= 3 * 152) return;
      }
  }
  static size_t max_smem(bool weno) { return sizeof(double) * (weno ? words(true, 4, 9, 9) : words(false, 4, 4, 33)); }
};

// The tile's place: edges te x t1 x t2 from (oe, o1, o2), org the element index
// of its first edge's upper cell.
template <int E>
struct Place64 {
  int te, t1, t2, se, s1, s2, org;
  __device__ __forceinline__ Place64(const Geom& g, const Tile64& w, int blk) {
    constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
    const int o1 = (blk % w.b1) * w.t1;
    blk /= w.b1;
    const int o2 = (blk % w.b2) * w.t2, oe = (blk / w.b2) * w.te;
    te = min(w.te, w.ne - oe);
    t1 = min(w.t1, w.n1 - o1);
    t2 = min(w.t2, w.n2 - o2);
    const int st[3] = {1, g.px, (int)g.plane};
    se = st[E];
    s1 = st[A1];
    s2 = st[A2];
    org = (g.ng + oe) * se + (g.ng + o1) * s1 + (g.ng + o2) * s2;
  }
};

template <int RECON, int E, bool M>
__device__ __forceinline__ void emf64_weno(const Dev<double>& d, const Inp<double>& in, const Prm<double>& P,
                                           const Tile64& w, int blk, double* sv) {
  constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
  const Place64<E> p(d.g, w, blk);
  const int te = p.te, t1 = p.t1, t2 = p.t2, st1 = p.s1, st2 = p.s2;
  const int c1 = t1 + 5, c2 = t2 + 5;  // staged cells: [-3, t + 2) about the tile's edges
  const int nv = te * c1 * c2, n1 = te * t1 * c2, n0 = te * c1 * t2, ned = te * t1 * t2;
  double* s1l = sv + 2 * nv;   // sv: cells [2][te][c2][c1]; rows along a1: [2][te][c2][t1], left and right
  double* s1r = s1l + 2 * n1;
  double* s0l = s1r + 2 * n1;  // columns along a2: [2][te][t2][c1]
  double* s0r = s0l + 2 * n0;
  double* sq = s0r + 2 * n0;   // [12][ned]
  const double* vel[3] = {in.vx, in.vy, in.vz};
  for (int t = threadIdx.x; t < 2 * nv; t += blockDim.x) {
    const int c = t >= nv, u = t - c * nv;
    const int i1 = u % c1, r = u / c1, i2 = r % c2, e = r / c2;
    sv[t] = (c ? vel[A2] : vel[A1])[p.org + e * p.se + (i1 - 3) * st1 + (i2 - 3) * st2];
  }
  __syncthreads();
  // first pass, one state per thread: [side][rows of both components, columns of both components]
  const int half = 2 * (n1 + n0);
  for (int t = threadIdx.x; t < 2 * half; t += blockDim.x) {
    const int right = t >= half;
    int u = t - right * half;
    const double* a;
    double* dst;
    int step;
    if (u < 2 * n1) {
      dst = (right ? s1r : s1l) + u;
      const int c = u >= n1;
      u -= c * n1;
      const int f1 = u % t1, r = u / t1;  // r = e c2 + row
      a = sv + c * nv + r * c1 + f1;
      step = 1;
    } else {
      u -= 2 * n1;
      dst = (right ? s0r : s0l) + u;
      const int c = u >= n0;
      u -= c * n0;
      const int i1 = u % c1, r = u / c1, f2 = r % t2, e = r / t2;
      a = sv + c * nv + (e * c2 + f2) * c1 + i1;
      step = c1;
    }
    if (right) {  // the mirrored stencil
      a += 5 * step;
      step = -step;
    }
    *dst = weno_side_ref<RECON>(a[0], a[step], a[2 * step], a[3 * step], a[4 * step], P);
  }
  __syncthreads();
  // second pass, one state per thread: 0-7 quadrant and component, 8-11 face B
  const double* fb[3] = {in.bi, in.bj, in.bk};
  for (int t = threadIdx.x; t < 12 * ned; t += blockDim.x) {
    const int k = t / ned, u = t - k * ned;
    const int f1 = u % t1, r = u / t1, f2 = r % t2, e = r / t2;
    const double* a;
    int step;
    bool right;
    if (k < 8) {
      const int q = k >> 1, c = k & 1;
      const bool q1 = q & 1, q2 = q & 2;  // quadrant cell (f1 - 1 + q1, f2 - 1 + q2)
      const double* v = sv + c * nv + (e * c2 + f2 + 2 + q2) * c1 + f1 + 2 + q1;
      // the smoother one-sided estimate: columns ("_0") if the outward slope along a1 is not the smaller, else rows
      const bool col = abs_ge(v[q1 ? 1 : -1] - v[0], v[q2 ? c1 : -c1] - v[0]);
      // v_10, v_11 (q1) read the R stencils, v_01, v_11 (q2) take the right state
      if (col) {
        a = (q1 ? s0r : s0l) + c * n0 + (e * t2 + f2) * c1 + f1;  // columns f1 - 3 ..
        step = 1;
      } else {
        a = (q1 ? s1r : s1l) + c * n1 + (e * c2 + f2) * t1 + f1;  // rows f2 - 3 ..
        step = t1;
      }
      right = q2;
    } else {  // b_a1 along a2 (8, 9), b_a2 along a1 (10, 11)
      step = k < 10 ? st2 : st1;
      a = (k < 10 ? fb[A1] : fb[A2]) + p.org + e * p.se + f1 * st1 + f2 * st2 - 3 * step;
      right = k & 1;
    }
    if (right) {
      a += 5 * step;
      step = -step;
    }
    sq[t] = weno_side_ref<RECON>(a[0], a[step], a[2 * step], a[3 * step], a[4 * step], P);
  }
  __syncthreads();
  for (int u = threadIdx.x; u < ned; u += blockDim.x) {
    const int f1 = u % t1, r = u / t1, f2 = r % t2, e = r / t2;
    const double* q = sq + u;
    // the mean in the reference's order (00, 01, 10, 11); quadrant index q1 + 2 q2
    const double v1 = 0.25 * (q[0] + q[4 * ned] + q[2 * ned] + q[6 * ned]);
    const double v2 = 0.25 * (q[ned] + q[5 * ned] + q[3 * ned] + q[7 * ned]);
    const int c = p.org + e * p.se + f1 * st1 + f2 * st2;
    const double* vf = d.vf;
    const double eta = eta4(vf[c - st1 - st2], vf[c - st2], vf[c], vf[c - st1]);
    d.E[E][c] = emf_value<double, E, M>(d, c, v1, v2, q[8 * ned], q[9 * ned], q[10 * ned], q[11 * ned], eta);
  }
}

template <int RECON, int E, bool M>
__device__ __forceinline__ void emf64_pdm(const Dev<double>& d, const Inp<double>& in, const Prm<double>& P,
                                          const Tile64& w, int blk, double* sv) {
  constexpr int A1 = (E + 1) % 3, A2 = (E + 2) % 3;
  const Place64<E> p(d.g, w, blk);
  const int te = p.te, t1 = p.t1, t2 = p.t2, st1 = p.s1, st2 = p.s2;
  const int c1 = t1 + 8, c2 = t2 + 8;  // staged cells: [-4, t + 4) about the tile's edges
  const int nv = te * c1 * c2, ng = te * t1 * c2, ned = te * t1 * t2;
  double* sg = sv + 2 * nv;  // sv: cells [2][te][c2][c1]; first pass: [2][te][c2][t1]
  double* sq = sg + 2 * ng;  // [6][ned]
  const double* vel[3] = {in.vx, in.vy, in.vz};
  for (int t = threadIdx.x; t < 2 * nv; t += blockDim.x) {
    const int c = t >= nv, u = t - c * nv;
    const int i1 = u % c1, r = u / c1, i2 = r % c2, e = r / c2;
    sv[t] = (c ? vel[A2] : vel[A1])[p.org + e * p.se + (i1 - 4) * st1 + (i2 - 4) * st2];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * ng; t += blockDim.x) {
    const int f1 = t % t1, r = t / t1;  // r = (component te + e) c2 + row
    const double* a = sv + r * c1 + f1;
    sg[t] = tap8(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]);
  }
  __syncthreads();
  // second pass: 0, 1 corner velocity of a component; 2, 3 states of b_a1 along a2, of b_a2 along a1
  const double* fb[3] = {in.bi, in.bj, in.bk};
  for (int t = threadIdx.x; t < 4 * ned; t += blockDim.x) {
    const int k = t / ned, u = t - k * ned;
    const int f1 = u % t1, r = u / t1, f2 = r % t2, e = r / t2;
    if (k < 2) {
      const double* q = sg + ((k * te + e) * c2 + f2) * t1 + f1;
      const double vi = tap8(q[0], q[t1], q[2 * t1], q[3 * t1], q[4 * t1], q[5 * t1], q[6 * t1], q[7 * t1]);
      const double* v = sv + ((k * te + e) * c2 + f2 + 4) * c1 + f1 + 4;
      sq[t] = corner_pdm<double, RECON>(v, 0, 1, c1, vi, P.pdmb);
    } else {
      const int s = k == 2 ? st2 : st1;
      double l, rr;
      recon_edge<double, RECON>(k == 2 ? fb[A1] : fb[A2], p.org + e * p.se + f1 * st1 + f2 * st2, s, P, l, rr);
      sq[(2 * k - 2) * ned + u] = l;
      sq[(2 * k - 1) * ned + u] = rr;
    }
  }
  __syncthreads();
  for (int u = threadIdx.x; u < ned; u += blockDim.x) {
    const int f1 = u % t1, r = u / t1, f2 = r % t2, e = r / t2;
    const double* q = sq + u;
    const int c = p.org + e * p.se + f1 * st1 + f2 * st2;
    const double* vf = d.vf;
    const double eta = eta4(vf[c - st1 - st2], vf[c - st2], vf[c], vf[c - st1]);
    d.E[E][c] = emf_value<double, E, M>(d, c, q[0], q[ned], q[2 * ned], q[3 * ned], q[4 * ned], q[5 * ned], eta);
  }
}

template <int RECON, bool M>
__global__ void __launch_bounds__(256) k_emf64(Dev<double> d, Inp<double> in, Prm<double> P, Tiles64 w) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  int b = blockIdx.x;
  auto tile = [&](auto fam, int blk) {
    constexpr int E = decltype(fam)::value;
    if constexpr (is_weno(RECON)) emf64_weno<RECON, E, M>(d, in, P, w.f[E], blk, sm);
    else emf64_pdm<RECON, E, M>(d, in, P, w.f[E], blk, sm);
  };
  if (b < w.blocks[0]) return tile(std::integral_constant<int, 0>{}, b);
  b -= w.blocks[0];
  if (b < w.blocks[1]) return tile(std::integral_constant<int, 1>{}, b);
  tile(std::integral_constant<int, 2>{}, b - w.blocks[1]);
}

template <int RECON, bool M>
void launch_emf64(const Dev<double>& d, const Inp<double>& in, const Prm<double>& P, cudaStream_t st) {
  static PerDevice attr;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    cudaFuncSetAttribute(k_emf64<RECON, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)Tiles64::max_smem(is_weno(RECON)));
    attr.mark(bit);
  }
  const Tiles64 w(is_weno(RECON), d.g);
  k_emf64<RECON, M><<<w.blocks[0] + w.blocks[1] + w.blocks[2], 256, w.smem, st>>>(d, in, P, w);
}

template <typename T, int RECON, int E, int TX, int TY, int TZ, int NT, bool M>
void launch_emf_weno(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, cudaStream_t st) {
  constexpr size_t bytes = EmfWeno<T, E, TX, TY, TZ>::smem;
  static PerDevice attr;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    cudaFuncSetAttribute(k_emf_weno<T, RECON, E, TX, TY, TZ, NT, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)bytes);
    attr.mark(bit);
  }
  const Geom& g = d.g;
  const int ex = g.nx0 + (E != 0), ey = g.ny0 + (E != 1), ez = g.nz0 + (E != 2);
  const dim3 grid((ex + TX - 1) / TX, (ey + TY - 1) / TY, (ez + TZ - 1) / TZ);
  k_emf_weno<T, RECON, E, TX, TY, TZ, NT, M><<<grid, NT, bytes, st>>>(d, in, P);
}


// Metric-mode EMF inputs of a stage: w^a = v . nbar_a at every cell and the
// face-normal field b_a = Phi_a / |A_a| at every face (ghosts included),
// which the EMF kernels then treat as the reference treats v and bi/bj/bk.
template <typename T>
__global__ void k_metric_prep(Dev<T> d, Inp<T> in) {
  const Geom& g = d.g;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (i > g.nx || j > g.ny || k > g.nz) return;
  const long long c = idx3<T>(g, i, j, k);
  const Metric<T>& m = d.m;
  if (i < g.nx && j < g.ny && k < g.nz) {
    const T u = in.vx[c], v = in.vy[c], w = in.vz[c];
#pragma unroll
    for (int a = 0; a < 3; ++a) d.mw[a][c] = u * m.nb[a][0][c] + v * m.nb[a][1][c] + w * m.nb[a][2][c];
  }
  if (j < g.ny && k < g.nz) d.mbn[0][c] = Ops<T>::dv(in.bi[c], m.am[0][c]);
  if (i < g.nx && k < g.nz) d.mbn[1][c] = Ops<T>::dv(in.bj[c], m.am[1][c]);
  if (i < g.nx && j < g.ny) d.mbn[2][c] = Ops<T>::dv(in.bk[c], m.am[2][c]);
}

// ------------------------------------------------------------------ update
// advance_bijk (3909-3933) + B combine, interior faces of all three arrays,
// read from the stage's half of the face B and written to the other half.
template <typename T, bool M, bool B>
__global__ void k_update_b(KArg<T, B> ka, int form, T cw, T den) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Geom& g = d.g;
  int i = bb.y * blockDim.x + threadIdx.x + g.ng;
  int j = bb.z * blockDim.y + threadIdx.y + g.ng;
  int k = bb.w + g.ng;
  if (i > g.ng + g.nx0 || j > g.ng + g.ny0 || k > g.ng + g.nz0) return;
  bool in_x = i < g.ng + g.nx0, in_y = j < g.ng + g.ny0, in_z = k < g.ng + g.nz0;
  long long c = idx3<T>(g, i, j, k);
  const long long sy = g.px, sz = g.plane;
  const T tau = step_tau<T>(d.sc);
  const T dx = d.wx[i], dy = d.wy[j], dz = d.wz[k];
  const T rx = d.rwx[i], ry = d.rwy[j], rz = d.rwz[k];
  const T *ei = d.E[0], *ej = d.E[1], *ek = d.E[2];
  typedef Ops<T> O;
  if (M) {  // face fluxes minus tau times the circulation of E.dl
    if (in_y && in_z) {
      T b = d.bi[c] - tau * ((ek[c + sy] - ek[c]) - (ej[c + sz] - ej[c]));
      if (form >= 0) b = comb(form, cw, d.q[5][c], b, den);
      d.obi[c] = b;
    }
    if (in_x && in_z) {
      T b = d.bj[c] - tau * ((ei[c + sz] - ei[c]) - (ek[c + 1] - ek[c]));
      if (form >= 0) b = comb(form, cw, d.q[6][c], b, den);
      d.obj[c] = b;
    }
    if (in_x && in_y) {
      T b = d.bk[c] - tau * ((ej[c + 1] - ej[c]) - (ei[c + sy] - ei[c]));
      if (form >= 0) b = comb(form, cw, d.q[7][c], b, den);
      d.obk[c] = b;
    }
    return;
  }
  if (in_y && in_z) {
    T b = d.bi[c] - tau * (O::dc(ek[c + sy] - ek[c], dy, ry) - O::dc(ej[c + sz] - ej[c], dz, rz));
    if (form >= 0) b = comb(form, cw, d.q[5][c], b, den);
    d.obi[c] = b;
  }
  if (in_x && in_z) {
    T b = d.bj[c] - tau * (O::dc(ei[c + sz] - ei[c], dz, rz) - O::dc(ek[c + 1] - ek[c], dx, rx));
    if (form >= 0) b = comb(form, cw, d.q[6][c], b, den);
    d.obj[c] = b;
  }
  if (in_x && in_y) {
    T b = d.bk[c] - tau * (O::dc(ej[c + 1] - ej[c], dx, rx) - O::dc(ei[c + sy] - ei[c], dy, ry));
    if (form >= 0) b = comb(form, cw, d.q[7][c], b, den);
    d.obk[c] = b;
  }
}

// ------------------------------------------------------------------- fill
// Single-device replacement of fill_hydro_mpi / fill_mag_mpi (781-819): every
// ghost element takes the value of its per-axis image (the x, y, z passes of
// the reference compose to exactly this, since each pass reads only interior
// values along its own axis).  Cell axes: interior [ng, ng+n0); the face
// array's own axis: interior [ng, ng+n0].
__device__ __forceinline__ int ghost_src(int x, int ng, int n0, bool face, int kind, bool& flip) {
  flip = false;
  int hi = face ? ng + n0 : ng + n0 - 1;  // last interior index
  if (x >= ng && x <= hi) return x;
  bool lo = x < ng;
  if (kind == BC_PERIODIC) return lo ? x + n0 : x - n0;
  if (kind == BC_OUTFLOW) return lo ? ng : hi;
  flip = true;  // mirror: even (flip ignored) or odd
  if (!face) return lo ? 2 * ng - 1 - x : 2 * n0 + 2 * ng - 1 - x;
  return lo ? 2 * ng - x : 2 * n0 + 2 * ng - x;
}

template <typename T>
__global__ void k_fill(Dev<T> d) {
  const Geom& g = d.g;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int j = blockIdx.y * blockDim.y + threadIdx.y;
  int k = blockIdx.z;
  if (i > g.nx || j > g.ny || k > g.nz) return;
  T* arr[8] = {d.rho, d.vx, d.vy, d.vz, d.p, d.bi, d.bj, d.bk};
  const int n0[3] = {g.nx0, g.ny0, g.nz0};
  const int x3[3] = {i, j, k};
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    int fa = a - 5;  // own staggering axis of bi/bj/bk
    bool ghost = false, inside = true;
    int s3[3];
    T sgn = T(1);
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      bool face = (fa == ax);
      int ext = (ax == 0 ? g.nx : ax == 1 ? g.ny : g.nz) + (face ? 1 : 0);
      if (x3[ax] >= ext) inside = false;
      bool flip;
      s3[ax] = ghost_src(x3[ax], g.ng, n0[ax], face, d.bc[ax], flip);
      if (s3[ax] != x3[ax]) ghost = true;
      // reflecting wall: the normal velocity is odd (a = 1,2,3 -> vx,vy,vz)
      if (flip && d.bc[ax] == BC_REFLECT && a == 1 + ax) sgn = -sgn;
    }
    if (!inside || !ghost) continue;
    long long c = idx3<T>(g, i, j, k);
    long long s = idx3<T>(g, s3[0], s3[1], s3[2]);
    T val = arr[a][s];
    arr[a][c] = (sgn > T(0)) ? val : -val;
  }
}

// Ghost fill fused with get_bxyz (mhd3d3.f90:2118-2128) and vf: every thread
// fills the ghost elements it owns (as k_fill) and computes the cell-centred
// B and vf of its cell from the ghost images of the faces and cells it needs,
// so no thread reads an element another thread is filling.  Face B is even
// under every boundary kind and vf uses only squares, so the images give
// exactly the values the separate fill followed by get_bxyz produces.  The
// per-axis image of every index comes from d.gmap (ghost_src tabulated at
// set-up): cell maps of x, y, z then face maps of x, y, z, each padded to n+2.
//
// Launch layout (256 threads per block, block index bb.y): first the interior
// tiles, 32 x 8 cells of one z plane each, which take the fast path with no
// divergence; then the shell, every (i <= nx, j <= ny, k <= nz) outside the
// interior box, 256 elements per block in a flattened order (the z slabs,
// then the y slabs, then the x slabs of the remaining rows).
struct FillShape {
  int nbx, nby, nint, nshell;
  __host__ __device__ FillShape(const Geom& g)
      : nbx((g.nx0 + 31) / 32), nby((g.ny0 + 7) / 8), nint(nbx * nby * g.nz0),
        nshell((g.nz + 1 - g.nz0) * (g.ny + 1) * (g.nx + 1) + g.nz0 * (g.ny + 1 - g.ny0) * (g.nx + 1) +
               g.nz0 * g.ny0 * (g.nx + 1 - g.nx0)) {}
  __host__ __device__ int blocks() const { return nint + (nshell + 255) / 256; }
};

// (i, j, k) of shell element u (0 <= u < nshell)
__device__ __forceinline__ void fill_shell_ijk(const Geom& g, int u, int& i, int& j, int& k) {
  const int X = g.nx + 1, Y = g.ny + 1, Z = g.nz + 1;
  const int a = (Z - g.nz0) * Y * X;
  if (u < a) {  // k outside the interior
    const int kk = u / (Y * X), r = u - kk * (Y * X);
    k = kk < g.ng ? kk : kk + g.nz0;
    j = r / X;
    i = r - j * X;
    return;
  }
  u -= a;
  const int yb = (Y - g.ny0) * X, b = g.nz0 * yb;
  if (u < b) {  // k inside, j outside
    const int kk = u / yb, r = u - kk * yb;
    k = g.ng + kk;
    const int jj = r / X;
    j = jj < g.ng ? jj : jj + g.ny0;
    i = r - jj * X;
    return;
  }
  u -= b;  // k, j inside, i outside
  const int xs = X - g.nx0, xb = g.ny0 * xs;
  const int kk = u / xb, r = u - kk * xb;
  k = g.ng + kk;
  const int jj = r / xs;
  j = g.ng + jj;
  const int ii = r - jj * xs;
  i = ii < g.ng ? ii : ii + g.nx0;
}

// One element of k_fill_bxyz; returns the CFL dt of its cell when want_dt
// (its values and widths, as get_dt sees them after the fill), else +inf.
template <typename T, bool M>
__device__ __forceinline__ T fill_bxyz_elem(const Dev<T>& d, int4 bb, int want_vf, int shell_only, int want_dt,
                                            unsigned& st) {
  const Geom& g = d.g;
  const FillShape fs(g);
  const int blk = shell_only ? bb.y + fs.nint : bb.y;
  int i, j, k;
  bool inner;
  if (blk < fs.nint) {
    const int bx = blk % fs.nbx, r = blk / fs.nbx, by = r % fs.nby, kz = r / fs.nby;
    i = g.ng + bx * 32 + (threadIdx.x & 31);
    j = g.ng + by * 8 + (threadIdx.x >> 5);
    k = g.ng + kz;
    if (i >= g.ng + g.nx0 || j >= g.ng + g.ny0) return T(INFINITY);  // those cells belong to no block here
    inner = true;
  } else {
    const int u = (blk - fs.nint) * 256 + threadIdx.x;
    if (u >= fs.nshell) return T(INFINITY);
    fill_shell_ijk(g, u, i, j, k);
    inner = false;
  }
  const int px = g.px, pl = (int)g.plane;
  const int c = i + px * j + pl * k;
  // interior fast path (no ghost element owned, all images are the identity)
  if (inner) {
    T bx, by, bz;
    if (M) {
      cell_b_metric<T>(d.m, c, d.bi[c], d.bi[c + 1], d.bj[c], d.bj[c + px], d.bk[c], d.bk[c + pl], bx, by, bz);
    } else {
      bx = T(0.5) * (d.bi[c + 1] + d.bi[c]);
      by = T(0.5) * (d.bj[c + px] + d.bj[c]);
      bz = T(0.5) * (d.bk[c + pl] + d.bk[c]);
    }
    d.bx[c] = bx;
    d.by[c] = by;
    d.bz[c] = bz;
    if (want_vf || want_dt) {
      const T u = d.vx[c], v = d.vy[c], w = d.vz[c], r0 = d.rho[c];
      if (want_vf) d.vf[c] = vf_val(u, v, w, sq3(bx, by, bz), r0);
      if (want_dt) return cell_dt<T, M>(d, c, i, j, k, r0, d.p[c], u, v, w, bx, by, bz, st);
    }
    return T(INFINITY);
  }
  const int* cx = d.gmap;
  const int* cy = cx + g.nx + 2;
  const int* cz = cy + g.ny + 2;
  const int* fx = cz + g.nz + 2;
  const int* fy = fx + g.nx + 2;
  const int* fz = fy + g.ny + 2;
  // every image index first, then every load, then every store: the loads of
  // one thread are in flight together (no store sits between them)
  const int sci = cx[i], scj = cy[j], sck = cz[k];  // cell images (entries n, n+1 unused)
  const int sfi = fx[i], sfj = fy[j], sfk = fz[k];  // face images
  const int sfi1 = fx[i + 1], sfj1 = fy[j + 1], sfk1 = fz[k + 1];
  const bool cin = i < g.nx && j < g.ny && k < g.nz;
  const bool gx = sci != i, gy = scj != j, gz = sck != k;
  const bool cell_copy = cin && (gx || gy || gz);
  const bool bi_copy = j < g.ny && k < g.nz && (sfi != i || gy || gz);
  const bool bj_copy = i < g.nx && k < g.nz && (gx || sfj != j || gz);
  const bool bk_copy = i < g.nx && j < g.ny && (gx || gy || sfk != k);
  const bool need_cell = cell_copy || (cin && (want_vf || want_dt));
  const int sc = sci + px * scj + pl * sck;
  const int fi0 = sfi + px * scj + pl * sck, fi1 = sfi1 + px * scj + pl * sck;  // faces of the image cell
  const int fj0 = sci + px * sfj + pl * sck, fj1 = sci + px * sfj1 + pl * sck;
  const int fk0 = sci + px * scj + pl * sfk, fk1 = sci + px * scj + pl * sfk1;
  T r0 = T(0), p0 = T(0), ux = T(0), uy = T(0), uz = T(0);
  if (need_cell) {
    r0 = d.rho[sc]; p0 = d.p[sc]; ux = d.vx[sc]; uy = d.vy[sc]; uz = d.vz[sc];
  }
  T bi0 = T(0), bi1 = T(0), bj0 = T(0), bj1 = T(0), bk0 = T(0), bk1 = T(0);
  if (bi_copy || cin) bi0 = d.bi[fi0];
  if (bj_copy || cin) bj0 = d.bj[fj0];
  if (bk_copy || cin) bk0 = d.bk[fk0];
  if (cin) {
    bi1 = d.bi[fi1];
    bj1 = d.bj[fj1];
    bk1 = d.bk[fk1];
  }
  // ghost copies: cell arrays (rho, vx, vy, vz, p), then bi, bj, bk
  if (cell_copy) {
    d.rho[c] = r0;
    d.p[c] = p0;
    d.vx[c] = (gx && d.bc[0] == BC_REFLECT) ? -ux : ux;
    d.vy[c] = (gy && d.bc[1] == BC_REFLECT) ? -uy : uy;
    d.vz[c] = (gz && d.bc[2] == BC_REFLECT) ? -uz : uz;
  }
  if (bi_copy) d.bi[c] = bi0;
  if (bj_copy) d.bj[c] = bj0;
  if (bk_copy) d.bk[c] = bk0;
  if (!cin) return T(INFINITY);
  T bx, by, bz;
  if (M) {  // face fluxes of the images, geometry of this cell (as fill then get_bxyz)
    cell_b_metric<T>(d.m, c, bi0, bi1, bj0, bj1, bk0, bk1, bx, by, bz);
  } else {
    bx = T(0.5) * (bi1 + bi0);
    by = T(0.5) * (bj1 + bj0);
    bz = T(0.5) * (bk1 + bk0);
  }
  d.bx[c] = bx;
  d.by[c] = by;
  d.bz[c] = bz;
  if (want_vf) d.vf[c] = vf_val(ux, uy, uz, bx * bx + by * by + bz * bz, r0);
  return want_dt ? cell_dt<T, M>(d, c, i, j, k, r0, p0, ux, uy, uz, bx, by, bz, st) : T(INFINITY);
}

// shell_only != 0: the launch covers only the shell blocks (block b is shell
// block b), after k_ct_fill has done the interior.  dt_next != 0: the CFL dt
// and status of the cells the launch covers go to the next-step accumulators.
template <typename T, bool M, bool B>
__global__ void __launch_bounds__(256, pass_min_blocks(B))
    k_fill_bxyz(KArg<T, B> ka, int want_vf, int shell_only, int dt_next) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  unsigned st = 0;
  const T m = fill_bxyz_elem<T, M>(d, bb, want_vf, shell_only, dt_next != 0, st);
  if (dt_next) dt_next_accumulate(d.sc, m, st);
}

// CT fused with get_bxyz and vf on Cartesian meshes (advance_bijk + combine,
// mhd3d3.f90:3909-3933, 3698-3702, 3784-3788; get_bxyz 2118-2128; vf of
// get_eijk_LFM 1766): one thread per interior cell, blocks of 32 x 8 cells of
// one z plane (the fill's interior tiles).  The thread advances its cell's
// three low faces into the new half of the face B with k_update_b's
// expressions and recomputes the new values of its three high faces from the
// same inputs (the cell that owns such a face writes it; the last cell of an
// axis writes the boundary face), then forms the cell-centred B from the six
// new faces and vf from the new primitives, which the z sweep wrote into the
// new half.  Every input here is read-only (old half of the face B, EMFs,
// U^n, new primitives), so a recomputed face equals what its owner writes,
// bit for bit, and the result equals k_update_b followed by the fill's
// interior tiles.  The ghost shell of the new half follows in k_fill_bxyz
// (shell_only).  An RK first stage (form FORM_SAVE) also stores its input
// face B as U^n of the later combines; dt_next (the last stage) accumulates
// the CFL dt and status of the new cells for the next step, as k_cfl would
// compute them at its start.
//
// Bytes bound it (20 arrays a cell), and by one cell a thread it waited on them:
// 24 of 31 cycles a warp on loads at 44 % of DRAM, ei, ej and bk fetched again by
// the next plane, their face computed twice.  A thread now walks Dev::ctk cells up
// z: the upper z face and edges of a cell are the lower ones of the next, and
// the next cell's inputs are loaded before this one's stores.  RK stage: 256^3
// 2285 -> 2202 us, 32 grids in a batch 2583 -> 2397.
//
// A sum that no product before it is contracted into (the faces as they are stored).
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return a + b; }
template <typename T>
struct CtIn {  // what cell c reads beyond the carried lower z face and edges
  T ek00, ek10, ek01, ek11, ei0, ei1, ej0, ej1, bi0, bi1, bj0, bj1, bk;  // e*0, e*1, bk: at the upper z face
  T qi0, qi1, qj0, qj1, qk;
  T u, v, w, r, p;
  __device__ __forceinline__ void load(const Dev<T>& d, int c, int px, int pl, bool comb, bool prim, bool dt) {
    const T *ei = d.E[0], *ej = d.E[1], *ek = d.E[2];
    ek00 = ek[c]; ek10 = ek[c + 1]; ek01 = ek[c + px]; ek11 = ek[c + 1 + px];
    ei0 = ei[c + pl]; ei1 = ei[c + px + pl];
    ej0 = ej[c + pl]; ej1 = ej[c + 1 + pl];
    bi0 = d.bi[c]; bi1 = d.bi[c + 1];
    bj0 = d.bj[c]; bj1 = d.bj[c + px];
    bk = d.bk[c + pl];
    if (comb) {
      qi0 = d.q[5][c]; qi1 = d.q[5][c + 1];
      qj0 = d.q[6][c]; qj1 = d.q[6][c + px];
      qk = d.q[7][c + pl];
    }
    if (prim) { u = d.ovx[c]; v = d.ovy[c]; w = d.ovz[c]; r = d.orho[c]; }
    if (dt) p = d.op[c];
  }
};
template <typename T, bool B>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 2 : 3) k_ct_fill(KArg<T, B> ka, int form, T cw, T den, int want_vf, int dt_next) {
  const int4 bb = ka.blk();
  const auto& d = ka.dev(bb);
  const Geom& g = d.g;
  const int i = g.ng + bb.y * 32 + (threadIdx.x & 31);
  const int j = g.ng + bb.z * 8 + (threadIdx.x >> 5);
  const int k0 = g.ng + bb.w * d.ctk, k1 = min(k0 + d.ctk, g.ng + g.nz0);
  const bool save = form == FORM_SAVE, want_dt = dt_next != 0;
  T m = T(INFINITY);
  unsigned st = 0;
  if (i < g.ng + g.nx0 && j < g.ng + g.ny0) {
    const int px = g.px, pl = (int)g.plane;
    int c = i + px * j + pl * k0;
    const T tau = step_tau<T>(d.sc);
    const T dx = d.wx[i], dy = d.wy[j];
    const T rx = d.rwx[i], ry = d.rwy[j];
    typedef Ops<T> O;
    // a face from its old value, U^n and the four edges around it (advance_bijk + combine)
    auto face = [&](T b, T q, T e1, T w1, T r1, T e2, T w2, T r2) {
      T n;
      if constexpr (std::is_same<T, float>::value)  // the contraction spelled out: a face has the same bits as a low and as a high one
        n = fmaf(-tau, fmaf(e1, r1, -(e2 * r2)), b);
      else
        n = b - tau * (O::dc(e1, w1, r1) - O::dc(e2, w2, r2));
      return form >= 0 ? comb(form, cw, q, n, den) : n;
    };
    const bool lx = i == g.ng + g.nx0 - 1, ly = j == g.ng + g.ny0 - 1;
    T ei0 = d.E[0][c], ei1 = d.E[0][c + px], ej0 = d.E[1][c], ej1 = d.E[1][c + 1], bk = d.bk[c];
    const T qk = form >= 0 ? d.q[7][c] : T(0);
    CtIn<T> a, nx;
    a.load(d, c, px, pl, form >= 0, want_vf || want_dt, want_dt);
    T bkl = face(bk, qk, ej1 - ej0, dx, rx, ei1 - ei0, dy, ry);
    for (int k = k0; k < k1; ++k, c += pl) {
      if (k + 1 < k1) nx.load(d, c + pl, px, pl, form >= 0, want_vf || want_dt, want_dt);
      const T dz = d.wz[k], rz = d.rwz[k];
      const bool lz = k == g.ng + g.nz0 - 1;
      if (save) {  // face B^n of the step (this first stage's input) for the later combines
        d.q[5][c] = a.bi0;
        d.q[6][c] = a.bj0;
        d.q[7][c] = bk;
        if (lx) d.q[5][c + 1] = a.bi1;
        if (ly) d.q[6][c + px] = a.bj1;
        if (lz) d.q[7][c + pl] = a.bk;
      }
      const T bil = face(a.bi0, a.qi0, a.ek01 - a.ek00, dy, ry, a.ej0 - ej0, dz, rz);
      const T bih = face(a.bi1, a.qi1, a.ek11 - a.ek10, dy, ry, a.ej1 - ej1, dz, rz);
      const T bjl = face(a.bj0, a.qj0, a.ei0 - ei0, dz, rz, a.ek10 - a.ek00, dx, rx);
      const T bjh = face(a.bj1, a.qj1, a.ei1 - ei1, dz, rz, a.ek11 - a.ek01, dx, rx);
      const T bkh = face(a.bk, a.qk, a.ej1 - a.ej0, dx, rx, a.ei1 - a.ei0, dy, ry);
      d.obi[c] = bil;
      d.obj[c] = bjl;
      d.obk[c] = bkl;
      if (lx) d.obi[c + 1] = bih;
      if (ly) d.obj[c + px] = bjh;
      if (lz) d.obk[c + pl] = bkh;
      const T bx = T(0.5) * add_rn(bih, bil);
      const T by = T(0.5) * add_rn(bjh, bjl);
      const T bz = T(0.5) * add_rn(bkh, bkl);
      d.bx[c] = bx;
      d.by[c] = by;
      d.bz[c] = bz;
      if (want_vf) d.vf[c] = vf_val(a.u, a.v, a.w, sq3(bx, by, bz), a.r);
      if (want_dt) {
        const T dt = cell_dt<T, false>(d, c, i, j, k, a.r, a.p, a.u, a.v, a.w, bx, by, bz, st);
        m = (dt < m) ? dt : m;
      }
      ei0 = a.ei0; ei1 = a.ei1; ej0 = a.ej0; ej1 = a.ej1;
      bk = a.bk;
      bkl = bkh;
      a = nx;
    }
  }
  if (want_dt) dt_next_accumulate(d.sc, m, st);
}

// ------------------------------------------------------------ diagnostics
// Double-double (Neumaier/TwoSum) accumulation of mass and energy, max |div B|
// (FP64), min rho incl. ghosts.  Deterministic: fixed per-thread order,
// fixed tree; partial results per block reduced by one block in order.
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e) {
  s = a + b;
  double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
struct DD { double s, c; };
__device__ __forceinline__ DD dd_add(DD x, DD y) {
  double s, e;
  two_sum(x.s, y.s, s, e);
  e += x.c + y.c;
  double s2, e2;
  two_sum(s, e, s2, e2);
  return DD{s2, e2};
}

template <typename T, bool M>
__global__ void k_diag_partial(Dev<T> d, double* part) {
  const Geom& g = d.g;
  long long n = (long long)g.nx0 * g.ny0 * g.nz0;
  DD ms{0, 0}, es{0, 0};
  double dmax = 0.0;
  const double gm1 = (double)d.gam - 1.0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    int i = (int)(t % g.nx0) + g.ng;
    long long r = t / g.nx0;
    int j = (int)(r % g.ny0) + g.ng;
    int k = (int)(r / g.ny0) + g.ng;
    long long c = idx3<T>(g, i, j, k);
    double dv = M ? d.m.vol64[c] : d.dx[i] * d.dy[j] * d.dz[k];
    double rr = d.rho[c], u = d.vx[c], v = d.vy[c], w = d.vz[c], pp = d.p[c];
    double a = d.bx[c], b = d.by[c], cc = d.bz[c];
    ms = dd_add(ms, DD{rr * dv, 0.0});
    double e = 0.5 * rr * (u * u + v * v + w * w) + pp / gm1 + 0.5 * (a * a + b * b + cc * cc);
    es = dd_add(es, DD{e * dv, 0.0});
    double db;
    if (M)  // net face flux out of the cell / V
      db = (((double)d.bi[c + 1] - (double)d.bi[c]) + ((double)d.bj[c + g.px] - (double)d.bj[c]) +
            ((double)d.bk[c + g.plane] - (double)d.bk[c])) / dv;
    else
      db = ((double)d.bi[c + 1] - (double)d.bi[c]) / d.dx[i] +
           ((double)d.bj[c + g.px] - (double)d.bj[c]) / d.dy[j] +
           ((double)d.bk[c + g.plane] - (double)d.bk[c]) / d.dz[k];
    db = fabs(db);
    dmax = db > dmax ? db : dmax;
  }
  __shared__ double sh[5][256];
  int tid = threadIdx.x;
  sh[0][tid] = ms.s; sh[1][tid] = ms.c; sh[2][tid] = es.s; sh[3][tid] = es.c; sh[4][tid] = dmax;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (tid < w) {
      DD a = dd_add(DD{sh[0][tid], sh[1][tid]}, DD{sh[0][tid + w], sh[1][tid + w]});
      DD b = dd_add(DD{sh[2][tid], sh[3][tid]}, DD{sh[2][tid + w], sh[3][tid + w]});
      sh[0][tid] = a.s; sh[1][tid] = a.c; sh[2][tid] = b.s; sh[3][tid] = b.c;
      sh[4][tid] = sh[4][tid] > sh[4][tid + w] ? sh[4][tid] : sh[4][tid + w];
    }
    __syncthreads();
  }
  if (tid == 0) {
    double* o = part + 5 * blockIdx.x;
    o[0] = sh[0][0]; o[1] = sh[1][0]; o[2] = sh[2][0]; o[3] = sh[3][0]; o[4] = sh[4][0];
  }
}

template <typename T>
__global__ void k_diag_final(Dev<T> d, const double* part, int nb, double* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  DD m{0, 0}, e{0, 0};
  double dm = 0;
  for (int b = 0; b < nb; ++b) {
    const double* o = part + 5 * b;
    m = dd_add(m, DD{o[0], o[1]});
    e = dd_add(e, DD{o[2], o[3]});
    dm = o[4] > dm ? o[4] : dm;
  }
  out[0] = m.s + m.c;
  out[1] = e.s + e.c;
  out[2] = dm;
}

template <typename T>
__global__ void k_min_rho(Dev<T> d, double* out) {
  const Geom& g = d.g;
  long long n = (long long)g.nx * g.ny * g.nz;
  double m = INFINITY;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    int i = (int)(t % g.nx);
    long long r = t / g.nx;
    int j = (int)(r % g.ny);
    int k = (int)(r / g.ny);
    double v = d.rho[idx3<T>(g, i, j, k)];
    m = v < m ? v : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    double y = __shfl_xor_sync(0xffffffffu, m, o);
    m = y < m ? y : m;
  }
  __shared__ double sm[32];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sm[wid] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = sm[w] < m ? sm[w] : m;
    m = sm[0] < m ? sm[0] : m;
    // single block launch: plain store
    out[3] = m;
  }
}

// ---------------------------------------------------------------- launchers

template <typename T>
Prm<T> prm_of(const Dev<T>& d) {
  Prm<T> P;
  P.pdmb = d.pdmb; P.eps = d.eps; P.alpha = d.alpha; P.beta = d.beta; P.tvd_shift = d.tvd_shift;
  return P;
}

template <typename T, bool M>
void Launch<T, M>::bxyz_vf(const Dev<T>& d, bool want_vf, cudaStream_t st) {
  dim3 b(64, 4, 1);
  k_bxyz_vf<T, M><<<grid3(d.g.nx, d.g.ny, d.g.nz, b), b, 0, st>>>(d, want_vf ? 1 : 0);
}

template <typename T, bool M>
void Launch<T, M>::fill_bxyz(const Dev<T>& d, bool want_vf, cudaStream_t st, bool dt_next) {
  const bool dt = dt_next && !M;
  if (dt) k_next_reset<<<1, 1, 0, st>>>(d.sc);
  k_fill_bxyz<T, M, false><<<FillShape(d.g).blocks(), 256, 0, st>>>(one(d), want_vf ? 1 : 0, 0, dt ? 1 : 0);
}

template <typename T, bool M>
void Launch<T, M>::ct_fill(const Dev<T>& d, int form, double c, double den, bool want_vf, cudaStream_t st,
                           bool dt_next) {
  if constexpr (M) {  // metric mode: CT, then the fill + bxyz pass of the new half
    ct(d, form, c, den, st);
    fill_bxyz(other_half(d), want_vf, st);
  } else {
    const FillShape fs(d.g);
    static PerDevice pref_ct, pref_fill;
    prefer_carveout(k_ct_fill<T, false>, 0, pref_ct);
    prefer_carveout(k_fill_bxyz<T, false, false>, 0, pref_fill);
    k_ct_fill<T, false><<<dim3(fs.nbx, fs.nby, (d.g.nz0 + d.ctk - 1) / d.ctk), 256, 0, st>>>(one(d), form, (T)c, (T)den,
                                                                        want_vf ? 1 : 0, dt_next ? 1 : 0);
    k_fill_bxyz<T, false, false><<<(fs.nshell + 255) / 256, 256, 0, st>>>(one(other_half(d)), want_vf ? 1 : 0, 1,
                                                                         dt_next ? 1 : 0);
  }
}

template <typename T, bool M>
void Launch<T, M>::cfl(const Dev<T>& d, int mode, cudaStream_t st, bool save) {
  dim3 grid((d.g.nx + 31) / 32, (d.g.ny + 7) / 8, (d.g.nz + 7) / 8);
  static PerDevice pref;
  prefer_carveout(k_cfl<T, M, false>, 0, pref);
  k_cfl<T, M, false><<<grid, 256, 0, st>>>(one(d), save ? 1 : 0, 0);
  k_cfl_final<T><<<1, 1, 0, st>>>(d, mode);
}

template <typename T, bool M>
void Launch<T, M>::cfl_folded(const Dev<T>& d, int mode, bool recompute, cudaStream_t st) {
  if (recompute) {
    k_next_reset<<<1, 1, 0, st>>>(d.sc);
    dim3 grid((d.g.nx + 31) / 32, (d.g.ny + 7) / 8, (d.g.nz + 7) / 8);
    k_cfl<T, M, false><<<grid, 256, 0, st>>>(one(d), 0, 1);
  }
  k_cfl_final<T><<<1, 1, 0, st>>>(d, mode | 4);
}

template <typename T, bool M>
void Launch<T, M>::predictor_ab(const Dev<T>& d, cudaStream_t st) {
  const int n = (d.g.nx + Vec16<T>::W) / Vec16<T>::W * d.g.py * d.g.pz;
  k_predictor_ab<T><<<(n + 255) / 256, 256, 0, st>>>(d);
}

template <typename T, int RECON, bool M>
void flux_r(const Dev<T>& d, const Inp<T>& in, cudaStream_t st) {
  Prm<T> P = prm_of(d);
  const Geom& g = d.g;
  const int n0 = (g.nx0 + 1) * g.ny0 * g.nz0, n1 = g.nx0 * (g.ny0 + 1) * g.nz0, n2 = g.nx0 * g.ny0 * (g.nz0 + 1);
  k_flux<T, RECON, 0, M, false><<<(n0 + 127) / 128, 128, 0, st>>>(one(d), in, P);
  k_flux<T, RECON, 1, M, false><<<(n1 + 127) / 128, 128, 0, st>>>(one(d), in, P);
  k_flux<T, RECON, 2, M, false><<<(n2 + 127) / 128, 128, 0, st>>>(one(d), in, P);
}

template <typename T, bool M>
void Launch<T, M>::fluxes(const Dev<T>& d, const Inp<T>& in, cudaStream_t st) {
  switch (d.recon) {
    case R_PDM: flux_r<T, R_PDM, M>(d, in, st); break;
    case R_PDMG: flux_r<T, R_PDMG, M>(d, in, st); break;
    case R_TVD: flux_r<T, R_TVD, M>(d, in, st); break;
    case R_WENO: flux_r<T, R_WENO, M>(d, in, st); break;
    case R_MPWENO: flux_r<T, R_MPWENO, M>(d, in, st); break;
    default: flux_r<T, R_TVDMC, M>(d, in, st); break;
  }
}

// Face tiles of axis D (1: y, 2: z) with tile length TDV along the sweep.
template <typename T, int RECON, int D, bool M, int TDV>
void launch_flux_t(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, int form, T c, T den, int ab,
                   cudaStream_t st) {
  constexpr size_t sm = flux_t_smem<T, TDV>();
  static PerDevice attr;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    cudaFuncSetAttribute(k_flux_t<T, RECON, D, M, false, TDV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    attr.mark(bit);
  }
  const Geom& g = d.g;
  const dim3 grid = (D == 1) ? dim3((g.nx0 + 31) / 32, (g.ny0 + TDV - 1) / TDV, g.nz0)
                             : dim3((g.nx0 + 31) / 32, (g.nz0 + TDV - 1) / TDV, g.ny0);
  k_flux_t<T, RECON, D, M, false, TDV><<<grid, dim3(32, TDV + 1), sm, st>>>(one(d), in, P, form, c, den, ab);
}

// Tile lengths compiled for a (precision, reconstruction, mode): 4, 8 and 16
// for the FP32 Cartesian PDM path (chosen by the autotuner), 8 elsewhere.
template <typename T, int RECON, bool M>
constexpr bool tunable() {
  return std::is_same<T, float>::value && is_pdm(RECON) && !M;
}

inline dim3 sweep_grid(int D, const Geom& g, int seg) {
  const int n0 = (D == 1) ? g.ny0 : g.nz0, no = (D == 1) ? g.nz0 : g.ny0;
  return dim3((g.nx0 * no + 127) / 128, (n0 + seg - 1) / seg);
}

template <typename T, int RECON, int D, bool M>
void flux_t_any(const Dev<T>& d, const Inp<T>& in, const Prm<T>& P, int form, T c, T den, int ab, cudaStream_t st) {
  if constexpr (std::is_same<T, float>::value && !M) {
    if (d.tile_td == kSweepTile) {  // column sweeps
      static PerDevice pref;  // 4 blocks of 20 (y) or 22 KB (z) static shared memory
      prefer_carveout(k_flux_sweep<T, D, false, RECON>, 50, pref);
      k_flux_sweep<T, D, false, RECON><<<sweep_grid(D, d.g, d.seg[D - 1]), dim3(32, 4), 0, st>>>(one(d), in, P, form, c, den);
      return;
    }
  }
  if constexpr (tunable<T, RECON, M>()) {
    if (d.tile_td == 4) return launch_flux_t<T, RECON, D, M, 4>(d, in, P, form, c, den, ab, st);
    if (d.tile_td == 16) return launch_flux_t<T, RECON, D, M, 16>(d, in, P, form, c, den, ab, st);
  }
  launch_flux_t<T, RECON, D, M, TD>(d, in, P, form, c, den, ab, st);
}

template <typename T, int RECON, bool M>
void hydro_r(const Dev<T>& d, const Inp<T>& in, int part, int form, double c, double den, bool ab,
             cudaStream_t st) {
  Prm<T> P = prm_of(d);
  const Geom& g = d.g;
  if constexpr (std::is_same<T, double>::value) {
    if (part == 0) {
      const unsigned n = (unsigned)((g.nx0 + 1) * g.ny0 * g.nz0) + g.nx0 * (g.ny0 + 1) * g.nz0 +
                         g.nx0 * g.ny0 * (g.nz0 + 1);
      const unsigned nt = n < 4 * 152 * 128 ? 64 : 128;
      k_faces<RECON, M><<<(n + nt - 1) / nt, nt, 0, st>>>(d, in, P);
    } else if (part == 2) {
      int tz = 1;
      while (tz < 32 && tz < g.nz0) tz *= 2;
      const dim3 b(128 / tz, tz);
      k_update_faces<M><<<(g.nx0 + b.x - 1) / b.x * g.ny0, b, 0, st>>>(d, form, c, den);
    }
  } else if (part == 0) {
    const int n0 = (g.nx0 + 1) * g.ny0 * g.nz0;
    static PerDevice pref;
    prefer_carveout(k_flux<T, RECON, 0, M, false>, 0, pref);
    k_flux<T, RECON, 0, M, false><<<(n0 + 127) / 128, 128, 0, st>>>(one(d), in, P);
  } else if (part == 1) {
    flux_t_any<T, RECON, 1, M>(d, in, P, -1, T(0), T(1), 0, st);
  } else if (part == 2) {
    flux_t_any<T, RECON, 2, M>(d, in, P, form, (T)c, (T)den, ab ? 1 : 0, st);
  }
}

template <typename T, bool M>
void Launch<T, M>::hydro(const Dev<T>& d, const Inp<T>& in, int part, int form, double c, double den, bool ab,
                         cudaStream_t st) {
  switch (d.recon) {
    case R_PDM: hydro_r<T, R_PDM, M>(d, in, part, form, c, den, ab, st); break;
    case R_PDMG: hydro_r<T, R_PDMG, M>(d, in, part, form, c, den, ab, st); break;
    case R_TVD: hydro_r<T, R_TVD, M>(d, in, part, form, c, den, ab, st); break;
    case R_WENO: hydro_r<T, R_WENO, M>(d, in, part, form, c, den, ab, st); break;
    case R_MPWENO: hydro_r<T, R_MPWENO, M>(d, in, part, form, c, den, ab, st); break;
    default: hydro_r<T, R_TVDMC, M>(d, in, part, form, c, den, ab, st); break;
  }
}

// ------------------------------------------------------------- Yee EMF
// get_eijk_Yee (mhd3d3.f90:1654-1752).  First the 12 split electric fields
// of every cell, ghosts included, from the Gaussian moments of get_v_center
// (2562-2592, the get_v_face element formula):
//   ez_ab = bx vx0a vy1b - by vx1a vy0b, ex_ab = by vy0a vz1b - bz vy1a vz0b,
//   ey_ab = bz vz0a vx1b - bx vz1a vx0b   (a, b = + / - moments),
// stored as ye[f * 4 + s], f = x, y, z edges, s = pp, np, pn, nn.
template <typename T>
__global__ void k_yee_split(Dev<T> d, Inp<T> in) {
  const Geom& g = d.g;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (i >= g.nx || j >= g.ny || k >= g.nz) return;
  const int c = i + g.px * (j + g.py * k);
  const T bxc = in.bx[c], byc = in.by[c], bzc = in.bz[c];
  const T bsq = bxc * bxc + byc * byc + bzc * bzc;
  const T lam = Ops<T>::dv(in.rho[c], T(2) * in.p[c] + bsq);
  T x0p, x0n, x1p, x1n, y0p, y0n, y1p, y1n, z0p, z0n, z1p, z1n;
  Moments<T>::hydro(lam, in.vx[c], true, x0p, x1p);
  Moments<T>::hydro(lam, in.vx[c], false, x0n, x1n);
  Moments<T>::hydro(lam, in.vy[c], true, y0p, y1p);
  Moments<T>::hydro(lam, in.vy[c], false, y0n, y1n);
  Moments<T>::hydro(lam, in.vz[c], true, z0p, z1p);
  Moments<T>::hydro(lam, in.vz[c], false, z0n, z1n);
  d.ye[0][c] = byc * y0p * z1p - bzc * y1p * z0p;
  d.ye[1][c] = byc * y0n * z1p - bzc * y1n * z0p;
  d.ye[2][c] = byc * y0p * z1n - bzc * y1p * z0n;
  d.ye[3][c] = byc * y0n * z1n - bzc * y1n * z0n;
  d.ye[4][c] = bzc * z0p * x1p - bxc * z1p * x0p;
  d.ye[5][c] = bzc * z0n * x1p - bxc * z1n * x0p;
  d.ye[6][c] = bzc * z0p * x1n - bxc * z1p * x0n;
  d.ye[7][c] = bzc * z0n * x1n - bxc * z1n * x0n;
  d.ye[8][c] = bxc * x0p * y1p - byc * x1p * y0p;
  d.ye[9][c] = bxc * x0n * y1p - byc * x1n * y0p;
  d.ye[10][c] = bxc * x0p * y1n - byc * x1p * y0n;
  d.ye[11][c] = bxc * x0n * y1n - byc * x1n * y0n;
}

// Then, per edge of family E, each split field is reconstructed to the edge
// in two passes -- along axis DA to the edge's DA face (first index of the
// field), at the rows of the DB stencil, then along DB to its DB face (second
// index) -- taking the left state for a + moment and the right one for a -
// moment; the edge EMF is epp + enp + epn + enn.  ei: y then z, ej: z then x,
// ek: x then y (reconstruct_3d dirs 5/6, 6/4, 4/5).  Only the rows the
// second pass reads are reconstructed in the first.
// PDM state of one side from 8 taps.  The other side does not enter the sum, so a NaN is kept
// to the states that have it in the reference's form: the left one of a NaN on either side of
// the face, the right one of a NaN in its own cell.
__device__ __forceinline__ bool nan_bits(double x) { return (__double2hiint(x) & 0x7fffffff) > 0x7ff00000; }
__device__ __forceinline__ bool nan_bits(float x) { return x != x; }
template <typename T>
__device__ __forceinline__ T pdm_one(const T* a, T pdmb, bool left) {
  const T lim = nan_bits(a[3]) ? a[4] : a[3];
  T l, r;
  if constexpr (std::is_same<T, double>::value)
    pdm_states_fused(a[2], a[3], a[4], a[5], tap8_fused(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]), pdmb, l, r, lim);
  else
    pdm_states(a[2], a[3], a[4], a[5], tap8(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]), pdmb, l, r, lim);
  return !left ? r : nan_bits(a[4]) ? a[4] : l;
}
template <typename T, int RECON, int E>
__global__ void k_emf_yee(Dev<T> d, Prm<T> P) {
  const Geom& g = d.g;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + g.ng;
  const int j = blockIdx.y * blockDim.y + threadIdx.y + g.ng;
  const int k = blockIdx.z + g.ng;
  const int ni = g.nx0 + (E != 0), nj = g.ny0 + (E != 1), nk = g.nz0 + (E != 2);
  if (i >= g.ng + ni || j >= g.ng + nj || k >= g.ng + nk) return;
  const int c = i + g.px * (j + g.py * k);
  const int st[3] = {1, g.px, (int)g.plane};
  constexpr int DA = (E == 0) ? 1 : (E == 1) ? 2 : 0;
  constexpr int DB = (E == 0) ? 2 : (E == 1) ? 0 : 1;
  const int sA = st[DA], sB = st[DB];
  constexpr bool TV = (RECON == R_TVD || RECON == R_TVDMC);
  constexpr int M0 = is_pdm(RECON) ? 0 : TV ? 2 : 1;
  constexpr int M1 = is_pdm(RECON) ? 7 : TV ? 5 : 6;
  T part[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {  // pp, np, pn, nn
    const T* f = d.ye[E * 4 + s];
    const bool left1 = (s == 0 || s == 2), left2 = (s < 2);
    T q[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      q[m] = T(0);
      if (m >= M0 && m <= M1) {
        const int e = c + (m - 4) * sB;
        if constexpr (RECON == R_PDM) {
          T a[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) a[t] = f[e + (t - 4) * sA];
          q[m] = pdm_one(a, P.pdmb, left1);
        } else {
          T l, r;
          recon_face<T, RECON>(f, e, sA, P, l, r);
          q[m] = left1 ? l : r;
        }
      }
    }
    if constexpr (RECON == R_PDM) {
      part[s] = pdm_one(q, P.pdmb, left2);
    } else {
      T l, r;
      recon_win<T, RECON, 0>(q, P, l, r);
      part[s] = left2 ? l : r;
    }
  }
  d.E[E][c] = part[0] + part[1] + part[2] + part[3];
}

template <typename T, int RECON>
void emf_yee_r(const Dev<T>& d, const Inp<T>& in, cudaStream_t st) {
  const Prm<T> P = prm_of(d);
  const Geom& g = d.g;
  const dim3 b(32, 4, 1);
  k_yee_split<T><<<grid3(g.nx, g.ny, g.nz, b), b, 0, st>>>(d, in);
  k_emf_yee<T, RECON, 0><<<grid3(g.nx0, g.ny0 + 1, g.nz0 + 1, b), b, 0, st>>>(d, P);
  k_emf_yee<T, RECON, 1><<<grid3(g.nx0 + 1, g.ny0, g.nz0 + 1, b), b, 0, st>>>(d, P);
  k_emf_yee<T, RECON, 2><<<grid3(g.nx0 + 1, g.ny0 + 1, g.nz0, b), b, 0, st>>>(d, P);
}

template <typename T>
void emf_yee(const Dev<T>& d, const Inp<T>& in, cudaStream_t st) {
  switch (d.recon) {
    case R_PDM: emf_yee_r<T, R_PDM>(d, in, st); break;
    case R_PDMG: emf_yee_r<T, R_PDMG>(d, in, st); break;
    case R_TVD: emf_yee_r<T, R_TVD>(d, in, st); break;
    case R_WENO: emf_yee_r<T, R_WENO>(d, in, st); break;
    case R_MPWENO: emf_yee_r<T, R_MPWENO>(d, in, st); break;
    default: emf_yee_r<T, R_TVDMC>(d, in, st); break;
  }
}

// FP32: ei tiles of 32 x 4 x 4 edges; ej, ek plane tiles of 32 x 8.
template <typename T, int RECON, bool M>
void emf_weno(const Dev<T>& d, const Inp<T>& in, cudaStream_t st) {
  const Prm<T> P = prm_of(d);
  if constexpr (std::is_same<T, double>::value) {
    launch_emf64<RECON, M>(d, in, P, st);
  } else {
    launch_emf_weno<T, RECON, 0, 32, 4, 4, 512, M>(d, in, P, st);
    launch_emf_weno<T, RECON, 1, 32, 1, 8, 256, M>(d, in, P, st);
    launch_emf_weno<T, RECON, 2, 32, 8, 1, 256, M>(d, in, P, st);
  }
}

template <typename T, int RECON, bool M>
void emf_r(const Dev<T>& d, const Inp<T>& in, cudaStream_t st) {
  Prm<T> P = prm_of(d);
  dim3 b(32, 4, 1);
  const Geom& g = d.g;
  k_emf<T, RECON, 0, M><<<grid3(g.nx0, g.ny0 + 1, g.nz0 + 1, b), b, 0, st>>>(d, in, P);
  k_emf<T, RECON, 1, M><<<grid3(g.nx0 + 1, g.ny0, g.nz0 + 1, b), b, 0, st>>>(d, in, P);
  k_emf<T, RECON, 2, M><<<grid3(g.nx0 + 1, g.ny0 + 1, g.nz0, b), b, 0, st>>>(d, in, P);
}

// ei tile cross-section: 8 x 8 edges in FP32, 4 x 4 in FP64 (batches); its length along
// the edge axis is ei_x() below.
#ifndef MHD_EI_TILE
#define MHD_EI_TILE 8
#endif
template <typename T> struct EiTile { static constexpr int Y = MHD_EI_TILE; };
// Edge-axis length of the 8 x 8 ei tile (the 4 x 4 tile stays 32 long): 16
// halves its 96 KB of shared memory, so 4 blocks (full occupancy) fit an SM;
// measured 2 % faster for the EMF family than 32 at 256^3.
#ifndef MHD_EI_X
#define MHD_EI_X 16
#endif
constexpr int ei_x(int y) { return y == 8 ? MHD_EI_X : 32; }
template <> struct EiTile<double> { static constexpr int Y = 4; };

template <typename T, int RECON, bool M>
void emf_pdm(const Dev<T>& d, const Inp<T>& in, cudaStream_t st) {
  Prm<T> P = prm_of(d);
  // (the metric mode keeps the tiles: beside the streams its face tiles ran a third slower)
  if constexpr (std::is_same<T, float>::value && !M) {
    if (d.tile_ey == kEmfStream) {
      emf_pdm_stream<T, RECON, M>(d, in, P, st);
      return;
    }
  }
  if constexpr (std::is_same<T, double>::value) {
    launch_emf64<RECON, M>(d, in, P, st);
  } else {
    if (!M && d.tile_ey == 4)
      launch_emf_pdm<T, RECON, 0, 32, 4, 4, 512, M>(d, in, P, st);
    else
      launch_emf_pdm<T, RECON, 0, ei_x(EiTile<T>::Y), EiTile<T>::Y, EiTile<T>::Y, 512, M>(d, in, P, st);
    launch_emf_pdm<T, RECON, 1, 32, 1, kPT, 32 * kPT, M>(d, in, P, st);
    launch_emf_pdm<T, RECON, 2, 32, kPT, 1, 32 * kPT, M>(d, in, P, st);
  }
}

template <typename T, bool M>
void Launch<T, M>::emf(const Dev<T>& d, const Inp<T>& in0, cudaStream_t st) {
  if constexpr (!M) {  // Yee: Cartesian only (checked at mhd_init)
    if (d.emf == EMF_YEE) {
      emf_yee<T>(d, in0, st);
      return;
    }
  }
  Inp<T> in = in0;
  if (M) {
    // normal velocities and face-normal field of the stage input, in the
    // places of v and bi/bj/bk
    dim3 b(64, 4, 1);
    k_metric_prep<T><<<grid3(d.g.nx + 1, d.g.ny + 1, d.g.nz + 1, b), b, 0, st>>>(d, in0);
    in.vx = d.mw[0]; in.vy = d.mw[1]; in.vz = d.mw[2];
    in.bi = d.mbn[0]; in.bj = d.mbn[1]; in.bk = d.mbn[2];
  }
  switch (d.recon) {
    case R_PDM: emf_pdm<T, R_PDM, M>(d, in, st); break;
    case R_PDMG: emf_pdm<T, R_PDMG, M>(d, in, st); break;
    case R_TVD: emf_r<T, R_TVD, M>(d, in, st); break;
    case R_WENO: emf_weno<T, R_WENO, M>(d, in, st); break;
    case R_MPWENO: emf_weno<T, R_MPWENO, M>(d, in, st); break;
    default: emf_r<T, R_TVDMC, M>(d, in, st); break;
  }
}

template <typename T, bool M>
void Launch<T, M>::ct(const Dev<T>& d, int form, double c, double den, cudaStream_t st) {
  dim3 b(32, 4, 1);
  const Geom& g = d.g;
  k_update_b<T, M, false><<<grid3(g.nx0 + 1, g.ny0 + 1, g.nz0 + 1, b), b, 0, st>>>(one(d), form, (T)c, (T)den);
}

template <typename T, bool M>
void Launch<T, M>::fill(const Dev<T>& d, cudaStream_t st) {
  dim3 b(64, 4, 1);
  k_fill<T><<<grid3(d.g.nx + 1, d.g.ny + 1, d.g.nz + 1, b), b, 0, st>>>(d);
}

// ------------------------------------------------------------ batched ensemble
template <typename T>
dim3 Batch<T>::dims(int fam, const Dev<T>& d, int td, int ey) {
  const Geom& g = d.g;
  const bool stream = std::is_same<T, float>::value && ey == kEmfStream;
  const int Y = std::is_same<T, float>::value && !stream ? ey : EiTile<T>::Y;
  if (!std::is_same<T, float>::value) td = TD;
  switch (fam) {
    case BF_CFL: return dim3((g.nx + 31) / 32, (g.ny + 7) / 8, (g.nz + 7) / 8);
    case BF_FLUX_X: return dim3(((g.nx0 + 1) * g.ny0 * g.nz0 + 127) / 128, 1, 1);
    case BF_FLUX_Y: return td == kSweepTile ? sweep_grid(1, g, d.seg[0]) : dim3((g.nx0 + 31) / 32, (g.ny0 + td - 1) / td, g.nz0);
    case BF_FLUX_Z: return td == kSweepTile ? sweep_grid(2, g, d.seg[1]) : dim3((g.nx0 + 31) / 32, (g.nz0 + td - 1) / td, g.ny0);
    case BF_EMF_I: return stream ? emf_stream_grid(0, g, d.eseg[0]) : emf_grid(0, g, ei_x(Y), Y, Y);
    case BF_EMF_J: return stream ? emf_stream_grid(1, g, d.eseg[1]) : emf_grid(1, g, 32, 1, kPT);
    case BF_EMF_K: return stream ? emf_stream_grid(2, g, d.eseg[2]) : emf_grid(2, g, 32, kPT, 1);
    case BF_EMF_R: return stream ? dim3(EmfRows(g).blocks(), 1, 1) : dim3(0, 0, 0);
    case BF_CT: {  // k_ct_fill: the fill's interior tiles
      const FillShape fs(g);
      return dim3(fs.nbx, fs.nby, (g.nz0 + d.ctk - 1) / d.ctk);
    }
    default: return dim3((FillShape(g).nshell + 255) / 256, 1, 1);  // BF_FILL: the shell of the new half
  }
}

template <typename T>
void Batch<T>::cfl(const BatchView& v, int sel, int mode, bool recompute, cudaStream_t st) {
  const Dev<T>* tab = (const Dev<T>*)v.tab[sel];
  const int nb = (v.ngrids + 127) / 128;
  if (recompute) {
    k_next_reset_batch<T><<<nb, 128, 0, st>>>(tab, v.ngrids);
    k_cfl<T, false, true><<<v.nblk[BF_CFL], 256, 0, st>>>(KArg<T, true>{tab, v.map[BF_CFL]}, 0, 1);
  }
  k_cfl_final_batch<T><<<nb, 128, 0, st>>>(tab, v.ngrids, mode | 4);
}

template <typename K>
void set_smem(K kernel, size_t bytes) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Batched EMF families with ei tile Y (edges along y and z per block).
template <typename T, int RECON, int Y>
void batch_emf(const BatchView& v, const Dev<T>* tab, const Prm<T>& P, cudaStream_t st) {
  constexpr int X = ei_x(Y);
  constexpr size_t si = emf_pdm_smem<T, 0, X, Y, Y>();
  constexpr size_t sj = emf_pdm_smem<T, 1, 32, 1, kPT>();
  constexpr size_t sk = emf_pdm_smem<T, 2, 32, kPT, 1>();
  static PerDevice attr;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    set_smem(k_emf_pdm<T, RECON, 0, X, Y, Y, 512, false, true>, si);
    set_smem(k_emf_pdm<T, RECON, 1, 32, 1, kPT, 32 * kPT, false, true>, sj);
    set_smem(k_emf_pdm<T, RECON, 2, 32, kPT, 1, 32 * kPT, false, true>, sk);
    attr.mark(bit);
  }
  const Inp<T> none{};
  k_emf_pdm<T, RECON, 0, X, Y, Y, 512, false, true><<<v.nblk[BF_EMF_I], 512, si, st>>>(
      KArg<T, true>{tab, v.map[BF_EMF_I]}, none, P);
  k_emf_pdm<T, RECON, 1, 32, 1, kPT, 32 * kPT, false, true><<<v.nblk[BF_EMF_J], 32 * kPT, sj, st>>>(
      KArg<T, true>{tab, v.map[BF_EMF_J]}, none, P);
  k_emf_pdm<T, RECON, 2, 32, kPT, 1, 32 * kPT, false, true><<<v.nblk[BF_EMF_K], 32 * kPT, sk, st>>>(
      KArg<T, true>{tab, v.map[BF_EMF_K]}, none, P);
}

// Batched slice-streamed EMF families and their boundary rows.
template <typename T, int RECON>
void batch_emf_stream(const BatchView& v, const Dev<T>* tab, const Prm<T>& P, cudaStream_t st) {
  stream_attr<T, RECON, 0, false, true>();
  stream_attr<T, RECON, 1, false, true>();
  stream_attr<T, RECON, 2, false, true>();
  const Inp<T> none{};
  constexpr int NT = 32 * MHD_EMF_NW;
  k_emf_stream<T, RECON, 0, MHD_EMF_NW, false, true><<<v.nblk[BF_EMF_I], NT, EmfStream<T, 0, MHD_EMF_NW>::smem, st>>>(
      KArg<T, true>{tab, v.map[BF_EMF_I]}, none, P);
  k_emf_stream<T, RECON, 1, MHD_EMF_NW, false, true><<<v.nblk[BF_EMF_J], NT, EmfStream<T, 1, MHD_EMF_NW>::smem, st>>>(
      KArg<T, true>{tab, v.map[BF_EMF_J]}, none, P);
  k_emf_stream<T, RECON, 2, MHD_EMF_NW, false, true><<<v.nblk[BF_EMF_K], NT, EmfStream<T, 2, MHD_EMF_NW>::smem, st>>>(
      KArg<T, true>{tab, v.map[BF_EMF_K]}, none, P);
  k_emf_rows<T, RECON, false, true><<<v.nblk[BF_EMF_R], 256, emf_rows_smem<T>(), st>>>(
      KArg<T, true>{tab, v.map[BF_EMF_R]}, none, P);
}

// Batched y / z face tiles of length TDV.
template <typename T, int RECON, int TDV>
void batch_flux_t(const BatchView& v, const Dev<T>* tab, const Prm<T>& P, int form, T c, T den, cudaStream_t st) {
  constexpr size_t sf = flux_t_smem<T, TDV>();
  static PerDevice attr;
  unsigned long long bit = 0;
  if (attr.need(bit)) {
    set_smem(k_flux_t<T, RECON, 1, false, true, TDV>, sf);
    set_smem(k_flux_t<T, RECON, 2, false, true, TDV>, sf);
    attr.mark(bit);
  }
  const Inp<T> none{};
  k_flux_t<T, RECON, 1, false, true, TDV><<<v.nblk[BF_FLUX_Y], dim3(32, TDV + 1), sf, st>>>(
      KArg<T, true>{tab, v.map[BF_FLUX_Y]}, none, P, -1, T(0), T(1), 0);
  k_flux_t<T, RECON, 2, false, true, TDV><<<v.nblk[BF_FLUX_Z], dim3(32, TDV + 1), sf, st>>>(
      KArg<T, true>{tab, v.map[BF_FLUX_Z]}, none, P, form, c, den, 0);
}

// Parts 1 (EMF families) and 2 (face fluxes and the conserved update) of Batch::parts.
template <typename T, int RECON>
void batch_emf_and_faces(const BatchView& v, const Dev<T>* tab, const Prm<T>& P, int which, int form, T c, T den,
                         cudaStream_t st) {
  constexpr bool F32 = std::is_same<T, float>::value;
  if (which & 1) {
    if constexpr (F32) {
      if (v.tile_ey == kEmfStream) batch_emf_stream<T, RECON>(v, tab, P, st);
      else if (v.tile_ey == 4) batch_emf<T, RECON, 4>(v, tab, P, st);
      else batch_emf<T, RECON, EiTile<T>::Y>(v, tab, P, st);
    } else {
      batch_emf<T, RECON, EiTile<T>::Y>(v, tab, P, st);
    }
  }
  if (which & 2) {
    const Inp<T> none{};
    k_flux<T, RECON, 0, false, true>
        <<<v.nblk[BF_FLUX_X], 128, 0, st>>>(KArg<T, true>{tab, v.map[BF_FLUX_X]}, none, P);
    if constexpr (F32) {
      if (v.tile_td == kSweepTile) {
        k_flux_sweep<T, 1, true, RECON><<<v.nblk[BF_FLUX_Y], dim3(32, 4), 0, st>>>(
            KArg<T, true>{tab, v.map[BF_FLUX_Y]}, none, P, -1, T(0), T(1));
        k_flux_sweep<T, 2, true, RECON><<<v.nblk[BF_FLUX_Z], dim3(32, 4), 0, st>>>(
            KArg<T, true>{tab, v.map[BF_FLUX_Z]}, none, P, form, c, den);
      } else if (v.tile_td == 4) {
        batch_flux_t<T, RECON, 4>(v, tab, P, form, c, den, st);
      } else if (v.tile_td == 16) {
        batch_flux_t<T, RECON, 16>(v, tab, P, form, c, den, st);
      } else {
        batch_flux_t<T, RECON, TD>(v, tab, P, form, c, den, st);
      }
    } else {
      batch_flux_t<T, RECON, TD>(v, tab, P, form, c, den, st);
    }
  }
}

template <typename T>
void Batch<T>::parts(const BatchView& v, int sel, int which, int form, double c, double den, cudaStream_t st) {
  const Dev<T>* tab = (const Dev<T>*)v.tab[sel];
  // the batch shares the deck's limiter constants (checked when it is built)
  Prm<T> P;
  P.pdmb = (T)v.pdmb; P.eps = (T)v.eps; P.alpha = (T)v.alpha; P.beta = (T)v.beta; P.tvd_shift = v.tvd_shift;
  if (pdm_signless(P.pdmb)) batch_emf_and_faces<T, R_PDM>(v, tab, P, which, form, (T)c, (T)den, st);
  else batch_emf_and_faces<T, R_PDMG>(v, tab, P, which, form, (T)c, (T)den, st);
  if (which & 4) {  // face-B update + bxyz + vf (interior), then the ghost shell of the half the stage wrote
    const int dt_next = (which & 8) ? 1 : 0;
    k_ct_fill<T, true><<<v.nblk[BF_CT], 256, 0, st>>>(KArg<T, true>{tab, v.map[BF_CT]}, form, (T)c, (T)den, 1, dt_next);
    KArg<T, true> fa{(const Dev<T>*)v.tab[sel ^ 1], v.map[BF_FILL]};
    k_fill_bxyz<T, false, true><<<v.nblk[BF_FILL], 256, 0, st>>>(fa, 1, 1, dt_next);
  }
}

template <typename T, bool M>
void Launch<T, M>::diagnostics(const Dev<T>& d, double* out, cudaStream_t st) {
  // out: device buffer of 5 + 5*nb doubles; out[4] (CFL dt) is filled by the caller
  const int nb = 152 * 2;
  double* part = out + 8;
  k_diag_partial<T, M><<<nb, 256, 0, st>>>(d, part);
  k_diag_final<T><<<1, 1, 0, st>>>(d, part, nb, out);
  k_min_rho<T><<<1, 1024, 0, st>>>(d, out);
}

}  // namespace mhd
