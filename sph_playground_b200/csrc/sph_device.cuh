// sph_device.cuh — device-side building blocks of the SPH step engine:
// kernel shapes (M4/M6/Gauss), two-sum accumulators, packed pair-data
// layouts and the launch-parameter block shared by all kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "sph_abi.h"

namespace sph {

// ---- enums mirrored from playground/src/const.f90 --------------------------
enum : int { esd_fab = 400, esd_n2w = 401, esd_fw = 402, esd_2nw_ds = 403,
             esd_2nw_sd = 404 };
enum : int { ept_empty = 0, ept_real = 1, ept_fixed = 2, ept_fixedreal = 21,
             ept_fixedmirror = 22, ept_periodic = 3 };
// 0-based store columns (const.f90:69-103 minus one)
enum : int {
  es_rx = 0, es_ry, es_rz, es_vx, es_vy, es_vz, es_ax, es_ay, es_az, es_m,
  es_den, es_h, es_dh, es_p, es_u, es_du, es_t, es_kappa, es_dtdx, es_dtdy,
  es_dtdz, es_ddt, es_bx, es_by, es_bz, es_dbx, es_dby, es_dbz, es_c, es_om,
  es_type, es_vfld
};
constexpr int NCOL = SPH_ES_TOTAL;
constexpr double kLightspeed = 2.997924e10;  // const.f90:6
constexpr double kRg = 8.314e7;              // const.f90:7
constexpr double kSigmaB = 5.67051e-5;       // const.f90:8

// ---- kernel shapes ------------------------------------------------------------
// The reference evaluates f(q), f'(q), f''(q) piecewise (kernel/base_m6.f90:36-97,
// base_m4.f90:35-90, base_gauss.f90:39-82).  On the device the pieces are
// written branch-free with clamped terms t_k = max(k - q, 0): for q beyond a
// break point the clamped term is exactly zero, so the sum equals the
// reference's piece without divergent branches inside a warp.
enum KernelId : int { KM4 = SPH_KERNEL_M4, KM6 = SPH_KERNEL_M6, KGAUSS = SPH_KERNEL_GAUSS };

template <int K> struct KRad;
template <> struct KRad<KM4> { static constexpr double v = 2.0; };
template <> struct KRad<KM6> { static constexpr double v = 3.0; };
template <> struct KRad<KGAUSS> { static constexpr double v = 10.0; };

// max(x, 0).  FP64: cleared by its sign bit, three integer operations in
// place of a comparison on the FP64 pipe and two selects (a NaN with a clear
// sign passes; every sum that meets one is reported through q_bad).
template <class R> __device__ __forceinline__ R rmax0(R x) { return x > R(0) ? x : R(0); }
template <> __device__ __forceinline__ double rmax0<double>(double x) {
  const int hi = __double2hiint(x), m = ~(hi >> 31);
  return __hiloint2double(hi & m, __double2loint(x) & m);
}
// x where it is below 0, else 0, for a NaN too.  FP64: by its high word, for
// the same reason.
__device__ __forceinline__ float rmin0(float x) { return x < 0.f ? x : 0.f; }
__device__ __forceinline__ double rmin0(double x) {
  return unsigned(__double2hiint(x)) - 0x80000000u <= 0x7ff00000u ? x : 0.0;
}
// q = r / h is negative, NaN or, in FP64, infinite (its high word, as unsigned,
// is not below that of infinity): two records less than 1.5e-154 apart have
// no direction (their r^2 is subnormal)
__device__ __forceinline__ bool q_bad(float q) { return !(q >= 0.f); }
__device__ __forceinline__ bool q_bad(double q) { return unsigned(__double2hiint(q)) >= 0x7ff00000u; }

template <int K, class R>
__device__ __forceinline__ void kshape_f_df(R q, R& f, R& df) {
  if constexpr (K == KM6) {
    R t3 = rmax0(R(3) - q), t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    R s3 = t3 * t3, s2 = t2 * t2, s1 = t1 * t1;
    R q3 = s3 * s3, q2 = s2 * s2, q1 = s1 * s1;
    f = q3 * t3 - R(6) * (q2 * t2) + R(15) * (q1 * t1);
    df = R(-5) * q3 + R(30) * q2 - R(75) * q1;
  } else if constexpr (K == KM4) {
    R t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    R s2 = t2 * t2, s1 = t1 * t1;
    f = R(0.25) * (s2 * t2) - s1 * t1;
    df = R(-0.75) * s2 + R(3) * s1;
  } else {
    R e = exp(-q * q);
    f = e;
    df = R(-2) * e * q;
  }
}

template <int K, class R>
__device__ __forceinline__ R kshape_df(R q) {
  if constexpr (K == KM6) {
    R t3 = rmax0(R(3) - q), t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    R s3 = t3 * t3, s2 = t2 * t2, s1 = t1 * t1;
    return R(-5) * (s3 * s3) + R(30) * (s2 * s2) - R(75) * (s1 * s1);
  } else if constexpr (K == KM4) {
    R t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    return R(-0.75) * (t2 * t2) + R(3) * (t1 * t1);
  } else {
    return R(-2) * exp(-q * q) * q;
  }
}

// f'(q) / KDfScale<K>::v, for the force pass: the common factor of the
// pieces goes into wCv / h^(d+1) once per particle instead of into every
// pair (one product per kernel value fewer).
template <int K> struct KDfScale;
template <> struct KDfScale<KM4> { static constexpr double v = -0.75; };
template <> struct KDfScale<KM6> { static constexpr double v = -5.0; };
template <> struct KDfScale<KGAUSS> { static constexpr double v = -2.0; };
template <int K, class R>
__device__ __forceinline__ R kshape_df_scaled(R q) {
  if constexpr (K == KM6) {
    R t3 = rmax0(R(3) - q), t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    R s3 = t3 * t3, s2 = t2 * t2, s1 = t1 * t1;
    return s3 * s3 - R(6) * (s2 * s2) + R(15) * (s1 * s1);
  } else if constexpr (K == KM4) {
    R t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    return t2 * t2 - R(4) * (t1 * t1);
  } else {
    return exp(-q * q) * q;
  }
}

template <int K, class R>
__device__ __forceinline__ void kshape_all(R q, R& f, R& df, R& ddf) {
  if constexpr (K == KM6) {
    R t3 = rmax0(R(3) - q), t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    R s3 = t3 * t3, s2 = t2 * t2, s1 = t1 * t1;
    R c3 = s3 * t3, c2 = s2 * t2, c1 = s1 * t1;
    R q3 = s3 * s3, q2 = s2 * s2, q1 = s1 * s1;
    f = q3 * t3 - R(6) * (q2 * t2) + R(15) * (q1 * t1);
    df = R(-5) * q3 + R(30) * q2 - R(75) * q1;
    ddf = R(20) * c3 - R(120) * c2 + R(300) * c1;
  } else if constexpr (K == KM4) {
    R t2 = rmax0(R(2) - q), t1 = rmax0(R(1) - q);
    R s2 = t2 * t2, s1 = t1 * t1;
    f = R(0.25) * (s2 * t2) - s1 * t1;
    df = R(-0.75) * s2 + R(3) * s1;
    ddf = R(1.5) * t2 - R(6) * t1;
  } else {
    R e = exp(-q * q);
    f = e;
    df = R(-2) * e * q;
    ddf = R(-2) * e + R(4) * e * q * q;
  }
}

// ---- two FP32 values per instruction ----------------------------------------
// Blackwell's packed FP32 operations (PTX f32x2): one instruction for two
// independent multiply-adds, each rounded as the scalar one.  They halve the
// issue slots of FP32 arithmetic, not its time on the FMA pipe, so they pay
// where a kernel is bound by instruction issue.
struct F2 {
  unsigned long long v;
  F2() = default;
  __device__ __forceinline__ F2(float a, float b) {
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  }
  __device__ __forceinline__ explicit F2(float a) : F2(a, a) {}
  __device__ __forceinline__ float x() const {
    float a;
    asm("mov.b64 {%0, _}, %1;" : "=f"(a) : "l"(v));
    return a;
  }
  __device__ __forceinline__ float y() const {
    float b;
    asm("mov.b64 {_, %0}, %1;" : "=f"(b) : "l"(v));
    return b;
  }
};
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_fma(b, F2(-1.f), a); }  // (exact product)
__device__ __forceinline__ F2 f2_max0(F2 a) { return F2(fmaxf(a.x(), 0.f), fmaxf(a.y(), 0.f)); }

// FP32 f(q) that follows q below FP32 resolution, for the Newton iteration on
// h.  q_lo is the rounding residual of q = r/h.  q is split as qh + dq with
// qh on the 2^-21 grid (for q < 4, q + 4 carries an ulp of 2^-21, so the add
// rounds q to it and the subtraction back is exact), which makes every piece
// t_k = c_k - qh exact; dq = (q - qh) + q_lo (the first difference exact)
// enters f to first order, f(q) = f(qh) + f'(qh) dq, the second-order term
// being below 1e-12 of f.  The density sum then changes smoothly with h
// instead of in steps of one FP32 ulp of q, so the Newton iterates settle.
template <int K>
__device__ __forceinline__ void kshape_f_df_res(float q, float q_lo, float& f, float& df) {
  if constexpr (K == KM6 || K == KM4) {
    const float qh = __fsub_rn(__fadd_rn(q, 4.0f), 4.0f);
    const float dq = __fadd_rn(__fsub_rn(q, qh), q_lo);
    constexpr int NP = (K == KM6) ? 3 : 2;
    const float cs[3] = {K == KM6 ? 3.f : 2.f, K == KM6 ? 2.f : 1.f, 1.f};
    const float as[3] = {K == KM6 ? 1.f : 0.25f, K == KM6 ? -6.f : -1.f, 15.f};
    f = 0.f;
    df = 0.f;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const float th = fmaxf(cs[k] - qh, 0.f);  // exact: both on the 2^-21 grid
      const float s = th * th;
      if constexpr (K == KM6) {
        const float q4 = s * s;
        f = fmaf(as[k], q4 * th, f);
        df = fmaf(-5.f * as[k], q4, df);
      } else {
        f = fmaf(as[k], s * th, f);
        df = fmaf(-3.f * as[k], s, df);
      }
    }
    f = fmaf(df, dq, f);
  } else {
    float e = expf(-q * q);
    f = e;
    df = -2.f * e * q;
    f = fmaf(df, q_lo, f);
  }
}

// The same for two values, from q = r ih rounded and r, ih_lo: q_lo, the
// residual of q, is r ih_lo - (q - r ih), the bracket exact by FMA.  nqh is
// -qh.  (The Gauss kernel: one after the other.)
template <int K>
__device__ __forceinline__ void kshape_f_df_res2(F2 q, F2 r, F2 neg_ih, F2 ih_lo, F2& f, F2& df) {
  const F2 ne = f2_fma(r, neg_ih, q);
  if constexpr (K == KM6 || K == KM4) {
    const F2 nqh = f2_sub(F2(4.0f), f2_add(q, F2(4.0f)));
    const F2 dq = f2_fma(r, ih_lo, f2_sub(f2_add(q, nqh), ne));
    constexpr int NP = (K == KM6) ? 3 : 2;
    const float cs[3] = {K == KM6 ? 3.f : 2.f, K == KM6 ? 2.f : 1.f, 1.f};
    const float as[3] = {K == KM6 ? 1.f : 0.25f, K == KM6 ? -6.f : -1.f, 15.f};
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const F2 th = f2_max0(f2_add(F2(cs[k]), nqh));  // exact: both on the 2^-21 grid
      const F2 s = f2_mul(th, th);
      const F2 p = K == KM6 ? f2_mul(s, s) : s;
      const F2 pt = f2_mul(p, th);
      const float d = (K == KM6 ? -5.f : -3.f) * as[k];
      f = k == 0 ? (as[0] == 1.f ? pt : f2_mul(F2(as[0]), pt)) : f2_fma(F2(as[k]), pt, f);
      df = k == 0 ? f2_mul(F2(d), p) : f2_fma(F2(d), p, df);
    }
    f = f2_fma(df, dq, f);
  } else {
    const F2 q_lo = f2_sub(f2_mul(r, ih_lo), ne);
    float f0, d0, f1, d1;
    kshape_f_df_res<K>(q.x(), q_lo.x(), f0, d0);
    kshape_f_df_res<K>(q.y(), q_lo.y(), f1, d1);
    f = F2(f0, f1);
    df = F2(d0, d1);
  }
}

template <int K, class R>
__device__ __forceinline__ R kshape_f(R q) {
  R f, df;
  kshape_f_df<K, R>(q, f, df);
  return f;
}

// Reciprocal square root, square root and root of a quotient of the pair
// arithmetic.  FP32 uses the MUFU approximations (about 2 ulp), inside the
// FP32 path's error budget.  FP64 takes every root from the hardware's
// approximation y of 1 / sqrt(x) (PTX rsqrt.approx.ftz.f64, relative error
// below 2^-19) and a few FMAs: a pair of the force pass had two of CUDA's
// roots and two quotients, each a longer sequence with a branch (circuit2 of
// a 96^3 blast 2.03 -> 1.61 ms with this and the packed factors).
// Range: arguments, and for the ratio a and a b, from 2^-1010 (9e-305, so that
// residuals are normal numbers) to the largest number; below it fsqrt and
// froot_ratio give 0.  (The reference's own sums leave the range there: m_b P,
// rho^2.)  CUDA's root outside it, as a branch: 96^3 blast of 4 steps 9.6 ->
// 11.1 ms.  Errors: tests/test_pair_roots.py.
__device__ __forceinline__ double rsqrt_approx(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// x is not below 2^-1010 (by its high word; a NaN is not)
__device__ __forceinline__ bool root_range(double x) {
  return unsigned(__double2hiint(x)) >= unsigned(1023 - 1010) << 20;
}
template <class R> __device__ __forceinline__ R frsqrt(R x);
// With e = 1 - x y^2, 1/sqrt(x) = y (1 - e)^(-1/2) = y (1 + e/2 + 3 e^2 / 8 +
// O(e^3)), the binomial series, whose next term is below 2^-55: within 1.2
// ulp (1 / sqrt(x) of two correctly rounded operations: 1.5).  0 gives NaN,
// a subnormal x infinity.
template <> __device__ __forceinline__ double frsqrt<double>(double x) {
  const double y = rsqrt_approx(x);
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
template <> __device__ __forceinline__ float frsqrt<float>(float x) { return rsqrtf(x); }
template <class R> __device__ __forceinline__ R fsqrt(R x);
// Goldschmidt's step, g = x y towards sqrt(x) with h = y / 2 towards 1 / (2
// sqrt(x)), then Newton's from the exact residual x - g^2 (P. Markstein,
// Software Division and Square Root Using Goldschmidt's Algorithms, 2004):
// within 0.6 ulp.  (51^3 FP64 density pass: with the early return 683 us, with
// a selection at the end 700; x frsqrt(x), 2 ulp, 687.)
template <> __device__ __forceinline__ double fsqrt<double>(double x) {
  if (!root_range(x)) return 0.0;
  const double y = rsqrt_approx(x), h = 0.5 * y;
  double g = x * y;
  g = fma(g, fma(-g, h, 0.5), g);
  return fma(fma(-g, g, x), h, g);
}
template <> __device__ __forceinline__ float fsqrt<float>(float x) {
  return x > 0.f ? x * rsqrtf(x) : 0.f;
}
template <class R> __device__ __forceinline__ R fdiv(R a, R b);
template <> __device__ __forceinline__ double fdiv<double>(double a, double b) { return a / b; }
template <> __device__ __forceinline__ float fdiv<float>(float a, float b) { return __fdividef(a, b); }
// sqrt(a / b) for a >= 0, b > 0 (FP32: as the quotient's root, which
// measured faster there than one rsqrt of the product).  FP64: the same two
// steps for s = a y with y towards 1 / sqrt(a b) = 1 / (s b), the residual
// a - s (s b): within 1.1 ulp (root and quotient correctly rounded: 1).
// (96^3 blast of 4 steps: with the selection at the end 9.54 ms, with an early
// return 9.58; a frsqrt(a b), 2.5 ulp, 9.61.)
__device__ __forceinline__ float froot_ratio(float a, float b) { return fsqrt<float>(fdiv<float>(a, b)); }
__device__ __forceinline__ double froot_ratio(double a, double b) {
  const double x = a * b;
  const double y = rsqrt_approx(x), h = 0.5 * y;
  double s = a * y;
  s = fma(s, fma(-x * y, h, 0.5), s);
  s = fma(fma(-s, s * b, a), h, s);
  return root_range(x) && root_range(a) ? s : 0.0;
}
// (x, y, z) of square length b2 > 0 to length 1, also where b2 is subnormal
// or has overflowed
__device__ __forceinline__ void to_unit(float b2, float& x, float& y, float& z) {
  const float ib = frsqrt<float>(b2);
  x *= ib; y *= ib; z *= ib;
}
__device__ __forceinline__ void to_unit(double b2, double& x, double& y, double& z) {
  if (!root_range(b2) || b2 > 1.7976931348623157e308) {
    const double s = b2 < 1.0 ? 0x1p500 : 0x1p-500;
    x *= s; y *= s; z *= s;
    b2 = x * x + y * y + z * z;
  }
  const double ib = frsqrt<double>(b2);
  x *= ib; y *= ib; z *= ib;
}

// h^n for small non-negative n (the reference's h**dim, h**(dim+2)).
template <int N, class R>
__device__ __forceinline__ R ipow(R x) {
  if constexpr (N == 0) return R(1);
  else if constexpr (N == 1) return x;
  else if constexpr (N == 2) return x * x;
  else if constexpr (N == 3) return x * (x * x);
  else if constexpr (N == 4) { R s = x * x; return s * s; }
  else { R s = x * x; return (s * s) * x; }
}

// ---- compensated accumulation ---------------------------------------------------
// Two-sum (Knuth): s + e == a + b exactly.  The FP32 path keeps every
// per-particle sum as (s, c) so that summing ~200 pair terms loses no more
// than one rounding of the final value.
template <class R> struct Acc {
  R s, c;
  __device__ __forceinline__ void init() { s = R(0); c = R(0); }
  __device__ __forceinline__ void add(R x) {
    R t = s + x;
    R bp = t - s;
    R e = (s - (t - bp)) + (x - bp);
    s = t;
    c += e;
  }
  __device__ __forceinline__ R val() const { return s + c; }
  __device__ __forceinline__ double dval() const { return double(s) + double(c); }
};
// two of them side by side
struct Acc2 {
  F2 s, c;
  __device__ __forceinline__ void init() { s = F2(0.f); c = F2(0.f); }
  __device__ __forceinline__ void add(F2 x) {
    const F2 t = f2_add(s, x);
    const F2 bp = f2_sub(t, s);
    const F2 e = f2_add(f2_sub(s, f2_sub(t, bp)), f2_sub(x, bp));
    s = t;
    c = f2_add(c, e);
  }
  __device__ __forceinline__ double dval() const {
    return (double(s.x()) + double(c.x())) + (double(s.y()) + double(c.y()));
  }
};
// Plain running sum in R with the same interface: a lane's share of a pair
// loop (n terms) carries at most gamma_n * sum|t| of rounding, about 2e-6
// sum|t| in FP32 for the n ~ 30 terms of a force lane; the lanes are then
// added in FP64.
template <class R> struct SumAcc {
  R s;
  __device__ __forceinline__ void init() { s = R(0); }
  __device__ __forceinline__ void add(R x) { s += x; }
  __device__ __forceinline__ R val() const { return s; }
  __device__ __forceinline__ double dval() const { return double(s); }
};
// Plain FP64 accumulator with the same interface.
template <> struct Acc<double> {
  double s;
  __device__ __forceinline__ void init() { s = 0.0; }
  __device__ __forceinline__ void add(double x) { s += x; }
  __device__ __forceinline__ double val() const { return s; }
  __device__ __forceinline__ double dval() const { return s; }
};

// ---- packed pair data (sorted order; the streams are listed at PackBufs) ----------
// FP64 positions are the sorted records' own; the FP32 force pass takes a
// hi/lo float pair of (x - origin + 2^E), all in one binade, so hi_i - hi_j
// is exact and dx = (hi_i - hi_j) + (lo_i - lo_j) carries one FP32 rounding;
// the FP32 density pass takes 31-bit fixed point (FixPos).
template <class R> struct PairPos;  // position handle for dx computation
template <> struct PairPos<double> {
  double x, y, z;
};
template <> struct PairPos<float> {
  float xh, yh, zh, xl, yl, zl;
};

__device__ __forceinline__ void pos_delta(const PairPos<double>& a, const PairPos<double>& b,
                                          double& dx, double& dy, double& dz) {
  dx = a.x - b.x; dy = a.y - b.y; dz = a.z - b.z;
}
// the density pass's FP32 positions: 31-bit fixed point over the packing
// frame; a separation is an exact integer difference rounded once to FP32
// (the scaling by the power-of-two unit is exact)
struct FixPos {
  int32_t x, y, z;
};
__device__ __forceinline__ void pos_delta(const FixPos& a, const FixPos& b, float& dx, float& dy,
                                          float& dz, float unit) {
  dx = __int2float_rn(a.x - b.x) * unit;
  dy = __int2float_rn(a.y - b.y) * unit;
  dz = __int2float_rn(a.z - b.z) * unit;
}
__device__ __forceinline__ void pos_delta(const PairPos<double>& a, const PairPos<double>& b,
                                          double& dx, double& dy, double& dz, double) {
  pos_delta(a, b, dx, dy, dz);
}
__device__ __forceinline__ void pos_delta(const PairPos<float>& a, const PairPos<float>& b,
                                          float& dx, float& dy, float& dz) {
  dx = (a.xh - b.xh) + (a.xl - b.xl);
  dy = (a.yh - b.yh) + (a.yl - b.yl);
  dz = (a.zh - b.zh) + (a.zl - b.zl);
}

// ---- launch parameters -------------------------------------------------------------
struct Params {
  int dim;
  int kernel;
  double krad;
  double wCv;      // knorm(dim)
  double fwc;      // fwcl(dim)
  double hfac;
  double alpha, beta, au;
  double gamma;
  double muzero;
  double difcond;
  int difiso;
  int ddw;
  int full_tensor;
  int eq_hydro, eq_magneto, eq_diff, eq_fld;
  int adden, artts;
  double tol;
  int maxiter;
  int eos_kind;  // 0 none, 1 adiabatic, 2 isothermal
  double c_iso;  // c of row 1 for eos_isothermal
};

// Counters of a block: each v[k] summed (or, with is_max[k], maximised) over
// the block's threads into thread 0's v[k], through shared memory, so that
// a kernel issues its counter atomics once per block, not once per warp
// (hundreds of thousands of same-address atomics per launch otherwise).
// Every thread of the block must call it; blocks of at most 1024 threads.
template <int N>
__device__ __forceinline__ void block_counters(unsigned long long (&v)[N], const bool (&is_max)[N]) {
  __shared__ unsigned long long part[32][N];
#pragma unroll
  for (int k = 0; k < N; ++k)
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long t = __shfl_xor_sync(0xffffffffu, v[k], o);
      v[k] = is_max[k] ? (t > v[k] ? t : v[k]) : v[k] + t;
    }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < N; ++k) part[w][k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 1; i < int((blockDim.x + 31) >> 5); ++i)
      for (int k = 0; k < N; ++k)
        v[k] = is_max[k] ? (part[i][k] > v[k] ? part[i][k] : v[k]) : v[k] + part[i][k];
}

// ---- a record's place among its cell's members -------------------------------------
// The counting sorts leave a cell's members in the order the atomics came; its
// records go by increasing index, each behind the smaller ones.  Every thread
// of a block of TPB calls it, for TPB consecutive members, u = members[q] of
// the cell [s, e) each (on: there is one).  Up to kCrowd members each counts
// the smaller ones.  In a crowded cell (far outliers make the cells wide) that
// costs the square of the members: there the block sorts its own, finds for
// every member of the cell how many of them it is smaller than, and adds up.
// (320,000 records in eight cells: the whole sort 6.4 ms by counting, 0.6 so,
// beside a search of 6.2.)
constexpr int kCrowd = 128;
template <int TPB>
__device__ __forceinline__ int32_t place_in_cell(const int32_t* members, bool on, int32_t u, int32_t s,
                                                 int32_t e) {
  __shared__ int32_t own[TPB], hist[TPB], cell, cell_end;
  const int tid = threadIdx.x;
  bool crowded = on && e - s > kCrowd;
  int32_t k = s;
  if (on && !crowded)
    for (int32_t i = s; i < e; ++i) k += members[i] < u ? 1 : 0;
  while (__syncthreads_or(crowded)) {  // a crowded cell of these members after the other
    if (tid == 0) cell = INT32_MAX;
    __syncthreads();
    if (crowded) atomicMin(&cell, s);
    __syncthreads();
    const bool mine = crowded && s == cell;
    if (mine) cell_end = e;
    own[tid] = mine ? u : INT32_MAX;
    hist[tid] = 0;
    __syncthreads();
    for (int size = 2; size <= TPB; size <<= 1)
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        const int o = tid ^ stride;
        const int32_t x = own[tid], y = own[o];
        __syncthreads();
        if (o > tid && (x > y) == ((tid & size) == 0)) {
          own[tid] = y;
          own[o] = x;
        }
        __syncthreads();
      }
    // p: how many of its own are at most w
    auto at_most = [&](int32_t w) {
      int p = 0;
      for (int d = TPB / 2; d > 0; d >>= 1) p += own[p + d - 1] <= w ? d : 0;
      return p + (own[p] <= w ? 1 : 0);
    };
    for (int32_t i = cell + tid; i < cell_end; i += TPB) {
      const int p = at_most(members[i]);
      if (p < TPB) atomicAdd(&hist[p], 1);
    }
    __syncthreads();
    for (int d = 1; d < TPB; d <<= 1) {
      const int32_t v = tid >= d ? hist[tid - d] : 0;
      __syncthreads();
      hist[tid] += v;
      __syncthreads();
    }
    if (mine) {
      k += hist[at_most(u) - 1];
      crowded = false;
    }
  }
  return k;
}

// status word helper: first error wins
__device__ __forceinline__ void raise_status(int* status, int code) {
  atomicCAS(status, 0, code);
}

}  // namespace sph
