// cueva_mp.cuh -- MP5 / MP7 / MP9 monotonicity-preserving reconstruction
// (Suresh & Huynh 1997) as one interface pair per thread.
//
// The reference reconstructs whole grid lines (mp5.f95:2-278, mp7.f95:2-315,
// mp9.f95:2-320): for every cell k it forms the limited left value up(k) at
// k+1/2 and right value um(k) at k-1/2, and the interface between cells i and
// i+1 takes L = up(i), R = um(i+1) (16_hll_flow_mpx.f95:942-1036).  Every
// (cell, slot) value depends only on the cells k-R..k+R of its own slot, so a
// thread that owns interface i loads the 2R+2 cells i-R..i+1+R into registers
// and evaluates exactly the two values it needs.  Operation order follows the
// Fortran so the FP64 build without FMA contraction is bit-identical.
#pragma once
#include "cueva_common.cuh"

namespace cueva {

// The minmod functions of funciones.f95 are written with sign arithmetic,
//   DMM(x, y)      = 0.5 (sign(1,x) + sign(1,y)) min(|x|, |y|)          (:148-162)
//   DM4(w, x, y, z) = 0.125 (sign(1,w) + sign(1,x))
//                     |(sign(1,w) + sign(1,y)) (sign(1,w) + sign(1,z))| min(|w|,|x|,|y|,|z|)   (:165-185)
// Every factor in front of the minimum is exactly +-1 or a signed zero, so
// they equal a selection on the sign bits: +-min with the sign of the first
// argument where all signs agree; otherwise (+-0) * min, with -0 only where
// DM4's first pair agrees (0.125 (+-2) |0| = -0 for negative w).  The zero
// is still multiplied by the minimum so that an infinite or NaN minimum
// gives NaN as in the sign arithmetic.  Results are bit-identical, with a
// third of the FP64 operations (the MP limiters call these in every pair).
template <typename T>
__device__ __forceinline__ T DMM(T x, T y) {
  const T m = fmin2(fabs(x), fabs(y));
  return (signbit(x) == signbit(y)) ? copysign(m, x) : T(0) * m;
}
// DMM for the monotonicity tests, with a plain zero where the signs differ:
// the test's product is the same for finite arguments, and where an
// argument is infinite or NaN the value under test is not finite or equals
// an infinite u, so the test fails either way
template <typename T>
__device__ __forceinline__ T DMM_test(T x, T y) {
  const T m = fmin2(fabs(x), fabs(y));
  return (signbit(x) == signbit(y)) ? copysign(m, x) : T(0);
}
template <typename T>
__device__ __forceinline__ T DM4(T w, T xx, T y, T z) {
  // (w and x are NaN whenever y or z is, so the order of the minima is free)
  const T m = fmin2(fmin2(fabs(w), fabs(xx)), fmin2(fabs(y), fabs(z)));
  const bool sw = signbit(w);
  const bool first = signbit(xx) == sw;
  if (first && signbit(y) == sw && signbit(z) == sw) return copysign(m, w);
  return (first ? copysign(T(0), w) : T(0)) * m;
}

// stencil radius of the unlimited interface formula; RM = 3 is the
// second-order MC reconstruction of the MCL flux routines (radius 1)
template <int RM> struct MPR { static constexpr int R = RM + 2; };
template <> struct MPR<3> { static constexpr int R = 1; };

// monotonized-central slope (mcl with slop = 2, funciones.f95:56-95):
// 0.5 (sign(1,a) + sign(1,b)) min(2|a|, 2|b|, |a+b|/2), the sign factor
// taken as a selection on the sign bits as in DMM
template <typename T>
__device__ __forceinline__ T mc_slope(T fa, T fb) {
  const T m = fmin2(fmin2(T(2.0) * fabs(fa), T(2.0) * fabs(fb)), T(0.5) * fabs(fa + fb));
  return (signbit(fa) == signbit(fb)) ? copysign(m, fa) : T(0) * m;
}

// unlimited left value at k+1/2 (SH97 eq. 2.1 / 2.31) around register index C.
// A product with 2 or 4 is exact, so it is taken in one FMA with the
// neighbouring term: same rounding, one operation less (with DMM_test and
// the halves of the HLLC fluxes: 2048 x 4096 step 15.43 -> 14.89 ms, B200).
template <int RM, int C, typename T, int N>
__device__ __forceinline__ T mp_vorp(const T (&u)[N]) {
  if constexpr (RM == 0) {
    const T b1 = T(1.0 / 60.0);
    return b1 * (fma_rn(T(2.0), u[C - 2], -(T(13.0) * u[C - 1])) + T(47.0) * u[C] + T(27.0) * u[C + 1] -
                 T(3.0) * u[C + 2]);
  } else if constexpr (RM == 1) {
    const T b1 = T(1.0 / 420.0);
    return b1 * fma_rn(T(4.0), u[C + 3], -T(3.0) * u[C - 3] + T(25.0) * u[C - 2] - T(101.0) * u[C - 1] +
                                             T(319.0) * u[C] + T(214.0) * u[C + 1] - T(38.0) * u[C + 2]);
  } else {
    const T b1 = T(1.0 / 2520.0);
    return b1 * (fma_rn(T(4.0), u[C - 4], -(T(41.0) * u[C - 3])) + T(199.0) * u[C - 2] - T(641.0) * u[C - 1] +
                 T(1879.0) * u[C] + T(1375.0) * u[C + 1] - T(305.0) * u[C + 2] + T(55.0) * u[C + 3] -
                 T(5.0) * u[C + 4]);
  }
}
// unlimited right value at k-1/2 (mirror formulas, same term order as the Fortran)
template <int RM, int C, typename T, int N>
__device__ __forceinline__ T mp_vorm(const T (&u)[N]) {
  if constexpr (RM == 0) {
    const T b1 = T(1.0 / 60.0);
    return b1 * fma_rn(T(2.0), u[C + 2],
                       -T(3.0) * u[C - 2] + T(27.0) * u[C - 1] + T(47.0) * u[C] - T(13.0) * u[C + 1]);
  } else if constexpr (RM == 1) {
    const T b1 = T(1.0 / 420.0);
    return b1 * fma_rn(T(4.0), u[C - 3], -T(3.0) * u[C + 3] + T(25.0) * u[C + 2] - T(101.0) * u[C + 1] +
                                             T(319.0) * u[C] + T(214.0) * u[C - 1] - T(38.0) * u[C - 2]);
  } else {
    const T b1 = T(1.0 / 2520.0);
    return b1 * (fma_rn(T(4.0), u[C + 4], -(T(41.0) * u[C + 3])) + T(199.0) * u[C + 2] - T(641.0) * u[C + 1] +
                 T(1879.0) * u[C] + T(1375.0) * u[C - 1] - T(305.0) * u[C - 2] + T(55.0) * u[C - 3] -
                 T(5.0) * u[C - 4]);
  }
}

// up(k) for the cell at register index C (mp5.f95:104-136) in two steps:
// mp_up_fast gives the unlimited value vorp and whether it passes the
// monotonicity test (then vorp is up(k)).  The interface pairs below take all
// their tests first (independent chains for the scheduler) and limit only
// the values that failed, together.
template <int RM, int C, typename T, int N>
__device__ __forceinline__ T mp_up_fast(const T (&u)[N], bool& ok) {
  const T alpha = T(2.0), epsm = T(1.0e-10);
  const T du0 = u[C] - u[C - 1];
  const T du1 = u[C + 1] - u[C];
  const T vorp = mp_vorp<RM, C>(u);
  const T vmpp = u[C] + DMM_test(du1, alpha * du0);
  ok = (vorp - u[C]) * (vorp - vmpp) <= epsm;
  return vorp;
}
// um(k) for the cell at register index C (mp5.f95:142-167), same first step
template <int RM, int C, typename T, int N>
__device__ __forceinline__ T mp_um_fast(const T (&u)[N], bool& ok) {
  const T alpha = T(2.0), epsm = T(1.0e-10);
  const T du0 = u[C] - u[C - 1];
  const T du1 = u[C + 1] - u[C];
  const T vorm = mp_vorm<RM, C>(u);
  const T vmpm = u[C] + DMM_test(-du0, -alpha * du1);
  ok = (vorm - u[C]) * (vorm - vmpm) <= epsm;
  return vorm;
}
// the limited values of an interface pair, both sides in one go: their
// chains are independent (latency), and the curvature limiter in the middle
// of the face is the same number for both (DM4 is symmetric in what its
// arguments are permuted by)
template <int RM, int C, typename T, int N>
__device__ __forceinline__ void mp_lim_pair(const T (&u)[N], T& L, T& R, bool okL, bool okR) {
  const T alpha = T(2.0), b2 = T(4.0 / 3.0);
  const T duL = u[C] - u[C - 1], duR = u[C + 2] - u[C + 1];
  const T dA = u[C - 2] - T(2.0) * u[C - 1] + u[C];
  const T dB = u[C - 1] - T(2.0) * u[C] + u[C + 1];
  const T dC = u[C] - T(2.0) * u[C + 1] + u[C + 2];
  const T dD = u[C + 1] - T(2.0) * u[C + 2] + u[C + 3];
  const T dm4L = DM4(T(4.0) * dB - dA, T(4.0) * dA - dB, dB, dA);
  const T dm4M = DM4(T(4.0) * dB - dC, T(4.0) * dC - dB, dB, dC);
  const T dm4R = DM4(T(4.0) * dC - dD, T(4.0) * dD - dC, dC, dD);
  const T av = T(0.5) * (u[C] + u[C + 1]), md = av - T(0.5) * dm4M;
  const T lo = fmin2(u[C], u[C + 1]), hi = fmax2(u[C], u[C + 1]);   // u[C + 1], u[C] on the right: equal values
  const T ulL = u[C] + alpha * duL, lcL = u[C] + T(0.5) * duL + b2 * dm4L;
  const T ulR = u[C + 1] - alpha * duR, lcR = u[C + 1] - T(0.5) * duR + b2 * dm4R;
  const T mnL = fmax2(fmin2(lo, md), fmin2(fmin2(u[C], ulL), lcL));
  const T mxL = fmin2(fmax2(hi, md), fmax2(fmax2(u[C], ulL), lcL));
  const T mnR = fmax2(fmin2(lo, md), fmin2(fmin2(u[C + 1], ulR), lcR));
  const T mxR = fmin2(fmax2(hi, md), fmax2(fmax2(u[C + 1], ulR), lcR));
  if (!okL) L = L + DMM(mnL - L, mxL - L);
  if (!okR) R = R + DMM(mnR - R, mxR - R);
}

// interface pair: u holds cells i-R .. i+1+R; returns L = up(i), R = um(i+1)
// (both monotonicity tests first: two independent chains before the rare
// limiting steps)
template <int RM, typename T, int N>
__device__ __forceinline__ void mp_pair(const T (&u)[N], T& L, T& R) {
  constexpr int C = MPR<RM>::R;
  bool okL, okR;
  L = mp_up_fast<RM, C>(u, okL);
  R = mp_um_fast<RM, C + 1>(u, okR);
  if (!(okL && okR)) mp_lim_pair<RM, C>(u, L, R, okL, okR);
}
// up(k), um(k) of the cells at C and C + 1 (the positivity-fixed pairs), the
// four tests first, then the limited values of those that failed with the
// three curvature limiters they share
template <int RM, int C, typename T, int N>
__device__ __forceinline__ void mp_quad(const T (&u)[N], T& up0, T& um0, T& up1, T& um1) {
  bool o0, o1, o2, o3;
  up0 = mp_up_fast<RM, C>(u, o0);
  um0 = mp_um_fast<RM, C>(u, o1);
  up1 = mp_up_fast<RM, C + 1>(u, o2);
  um1 = mp_um_fast<RM, C + 1>(u, o3);
  if (o0 && o1 && o2 && o3) return;
  const T alpha = T(2.0), b2 = T(4.0 / 3.0);
  const T dA = u[C - 2] - T(2.0) * u[C - 1] + u[C];
  const T dB = u[C - 1] - T(2.0) * u[C] + u[C + 1];
  const T dC = u[C] - T(2.0) * u[C + 1] + u[C + 2];
  const T dD = u[C + 1] - T(2.0) * u[C + 2] + u[C + 3];
  const T dm4L = DM4(T(4.0) * dB - dA, T(4.0) * dA - dB, dB, dA);
  const T dm4M = DM4(T(4.0) * dB - dC, T(4.0) * dC - dB, dB, dC);
  const T dm4R = DM4(T(4.0) * dC - dD, T(4.0) * dD - dC, dC, dD);
  // value w of the cell value c towards its neighbour n: slope d on the far
  // side (signed towards n), curvatures near and far
  auto limit = [&](T w, T c, T n, T d, T nearc, T farc) {
    const T md = T(0.5) * (c + n) - T(0.5) * nearc;
    const T ul = c + alpha * d, lc = c + T(0.5) * d + b2 * farc;
    const T mn = fmax2(fmin2(fmin2(c, n), md), fmin2(fmin2(c, ul), lc));
    const T mx = fmin2(fmax2(fmax2(c, n), md), fmax2(fmax2(c, ul), lc));
    return w + DMM(mn - w, mx - w);
  };
  if (!o0) up0 = limit(up0, u[C], u[C + 1], u[C] - u[C - 1], dm4M, dm4L);
  if (!o1) um0 = limit(um0, u[C], u[C - 1], -(u[C + 1] - u[C]), dm4L, dm4M);
  if (!o2) up1 = limit(up1, u[C + 1], u[C + 2], u[C + 1] - u[C], dm4R, dm4M);
  if (!o3) um1 = limit(um1, u[C + 1], u[C], -(u[C + 2] - u[C + 1]), dm4M, dm4R);
}

// pair for the p / rho slots: the positivity fix-up of mp5.f95:177-216 makes
// the final up(k) depend on um(k) and the final um(k) on up(k)
template <typename T>
__device__ __forceinline__ void posfix_point(T uk, T duk, T duk1, T& up, T& um) {
  if (up < T(0.0)) { up = uk + T(0.50) * DMM(duk, duk1); um = uk; }
  if (um < T(0.0)) { um = uk - T(0.50) * DMM(duk, duk1); up = uk; }
}
template <int RM, typename T, int N>
__device__ __forceinline__ void mp_pair_pos(const T (&u)[N], T& L, T& R) {
  constexpr int C = MPR<RM>::R;
  T up0, um0, up1, um1;
  mp_quad<RM, C>(u, up0, um0, up1, um1);
  posfix_point(u[C], u[C] - u[C - 1], u[C + 1] - u[C], up0, um0);
  posfix_point(u[C + 1], u[C + 1] - u[C], u[C + 2] - u[C + 1], up1, um1);
  L = up0;
  R = um1;
}

// positivity-fixed pair on differences u - c0 (mixed precision): the same
// limiter (it is translation-equivariant) with the sign tests of the
// positivity fix taken on the FP64 value c0 + u
template <typename T>
__device__ __forceinline__ void posfix_point_delta(double c0, T uk, T duk, T duk1, T& up, T& um) {
  if (c0 + double(up) < 0.0) { up = uk + T(0.50) * DMM(duk, duk1); um = uk; }
  if (c0 + double(um) < 0.0) { um = uk - T(0.50) * DMM(duk, duk1); up = uk; }
}
template <int RM, typename T, int N>
__device__ __forceinline__ void mp_pair_pos_delta(const T (&u)[N], double c0, T& L, T& R) {
  constexpr int C = MPR<RM>::R;
  T up0, um0, up1, um1;
  mp_quad<RM, C>(u, up0, um0, up1, um1);
  posfix_point_delta(c0, u[C], u[C] - u[C - 1], u[C + 1] - u[C], up0, um0);
  posfix_point_delta(c0, u[C + 1], u[C + 1] - u[C], u[C + 2] - u[C + 1], up1, um1);
  L = up0;
  R = um1;
}

// two fields' pairs side by side: twice the independent chains of mp_pair,
// for kernels whose warps have nothing else to wait on
template <int RM, typename T, int N>
__device__ __forceinline__ void mp_pair2(const T (&u)[N], const T (&v)[N], T& uL, T& uR, T& vL, T& vR) {
  constexpr int C = MPR<RM>::R;
  bool a, b, c, d;
  uL = mp_up_fast<RM, C>(u, a);
  uR = mp_um_fast<RM, C + 1>(u, b);
  vL = mp_up_fast<RM, C>(v, c);
  vR = mp_um_fast<RM, C + 1>(v, d);
  if (!(a && b && c && d)) {
    mp_lim_pair<RM, C>(u, uL, uR, a, b);
    mp_lim_pair<RM, C>(v, vL, vR, c, d);
  }
}

// Out-of-line entry points.  A sweep thread reconstructs ~45 slots per grid
// point; inlining the limiter 45 times made the kernel larger than the
// instruction cache (ncu: "no instruction" was the top stall).  One copy of
// each limiter body is called with the stencil values in registers.
template <typename T> struct Pair { T L, R; };

template <typename T> struct Pair2 { T uL, uR, vL, vR; };

template <int RM, typename T> struct MPCall;
// two fields in one call (MP5 and MP7; the arguments of two MP9 stencils no
// longer fit the registers of a call)
template <int RM, typename T> struct MPCall2;
template <typename T> struct MPCall2<0, T> {
  static __device__ __noinline__ Pair2<T> pair(T a0, T a1, T a2, T a3, T a4, T a5, T b0, T b1, T b2, T b3, T b4, T b5) {
    const T u[6] = {a0, a1, a2, a3, a4, a5}, v[6] = {b0, b1, b2, b3, b4, b5};
    Pair2<T> p; mp_pair2<0>(u, v, p.uL, p.uR, p.vL, p.vR); return p;
  }
  static __device__ __forceinline__ Pair2<T> call(const T (&u)[6], const T (&v)[6]) {
    return pair(u[0], u[1], u[2], u[3], u[4], u[5], v[0], v[1], v[2], v[3], v[4], v[5]);
  }
};
template <typename T> struct MPCall2<1, T> {
  static __device__ __noinline__ Pair2<T> pair(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7, T b0, T b1, T b2, T b3,
                                               T b4, T b5, T b6, T b7) {
    const T u[8] = {a0, a1, a2, a3, a4, a5, a6, a7}, v[8] = {b0, b1, b2, b3, b4, b5, b6, b7};
    Pair2<T> p; mp_pair2<1>(u, v, p.uL, p.uR, p.vL, p.vR); return p;
  }
  static __device__ __forceinline__ Pair2<T> call(const T (&u)[8], const T (&v)[8]) {
    return pair(u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
  }
};
template <typename T> struct MPCall<0, T> {
  static __device__ __noinline__ Pair<T> pair(T a0, T a1, T a2, T a3, T a4, T a5) {
    const T u[6] = {a0, a1, a2, a3, a4, a5};
    Pair<T> p; mp_pair<0>(u, p.L, p.R); return p;
  }
  static __device__ __noinline__ Pair<T> pos(T a0, T a1, T a2, T a3, T a4, T a5) {
    const T u[6] = {a0, a1, a2, a3, a4, a5};
    Pair<T> p; mp_pair_pos<0>(u, p.L, p.R); return p;
  }
  static __device__ __noinline__ Pair<T> posd(T a0, T a1, T a2, T a3, T a4, T a5, double c0) {
    const T u[6] = {a0, a1, a2, a3, a4, a5};
    Pair<T> p; mp_pair_pos_delta<0>(u, c0, p.L, p.R); return p;
  }
  static __device__ __forceinline__ Pair<T> call_posd(const T (&u)[6], double c0) { return posd(u[0], u[1], u[2], u[3], u[4], u[5], c0); }
  template <bool POS> static __device__ __forceinline__ Pair<T> call(const T (&u)[6]) {
    return POS ? pos(u[0], u[1], u[2], u[3], u[4], u[5]) : pair(u[0], u[1], u[2], u[3], u[4], u[5]);
  }
};
template <typename T> struct MPCall<1, T> {
  static __device__ __noinline__ Pair<T> pair(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7) {
    const T u[8] = {a0, a1, a2, a3, a4, a5, a6, a7};
    Pair<T> p; mp_pair<1>(u, p.L, p.R); return p;
  }
  static __device__ __noinline__ Pair<T> pos(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7) {
    const T u[8] = {a0, a1, a2, a3, a4, a5, a6, a7};
    Pair<T> p; mp_pair_pos<1>(u, p.L, p.R); return p;
  }
  static __device__ __noinline__ Pair<T> posd(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7, double c0) {
    const T u[8] = {a0, a1, a2, a3, a4, a5, a6, a7};
    Pair<T> p; mp_pair_pos_delta<1>(u, c0, p.L, p.R); return p;
  }
  static __device__ __forceinline__ Pair<T> call_posd(const T (&u)[8], double c0) { return posd(u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], c0); }
  template <bool POS> static __device__ __forceinline__ Pair<T> call(const T (&u)[8]) {
    return POS ? pos(u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7])
               : pair(u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7]);
  }
};
template <typename T> struct MPCall<2, T> {
  static __device__ __noinline__ Pair<T> pair(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7, T a8, T a9) {
    const T u[10] = {a0, a1, a2, a3, a4, a5, a6, a7, a8, a9};
    Pair<T> p; mp_pair<2>(u, p.L, p.R); return p;
  }
  static __device__ __noinline__ Pair<T> pos(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7, T a8, T a9) {
    const T u[10] = {a0, a1, a2, a3, a4, a5, a6, a7, a8, a9};
    Pair<T> p; mp_pair_pos<2>(u, p.L, p.R); return p;
  }
  static __device__ __noinline__ Pair<T> posd(T a0, T a1, T a2, T a3, T a4, T a5, T a6, T a7, T a8, T a9, double c0) {
    const T u[10] = {a0, a1, a2, a3, a4, a5, a6, a7, a8, a9};
    Pair<T> p; mp_pair_pos_delta<2>(u, c0, p.L, p.R); return p;
  }
  static __device__ __forceinline__ Pair<T> call_posd(const T (&u)[10], double c0) { return posd(u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], u[8], u[9], c0); }
  template <bool POS> static __device__ __forceinline__ Pair<T> call(const T (&u)[10]) {
    return POS ? pos(u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], u[8], u[9])
               : pair(u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7], u[8], u[9]);
  }
};

// second-order MC pair of 16_hll_flow_mcl.f95:565-1112 (FAC = 0.5, no
// positivity fix): u holds cells i-1 .. i+2
template <typename T> struct MPCall<3, T> {
  template <bool POS> static __device__ __forceinline__ Pair<T> call(const T (&u)[4]) {
    Pair<T> p;
    p.L = u[1] + T(0.5) * mc_slope(u[2] - u[1], u[1] - u[0]);
    p.R = u[2] - T(0.5) * mc_slope(u[3] - u[2], u[2] - u[1]);
    return p;
  }
};

}  // namespace cueva
