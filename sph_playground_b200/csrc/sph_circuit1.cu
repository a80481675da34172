// sph_circuit1.cu — circuit1 on the device: density summation, the Newton
// iteration on h with the grad-h term Omega (circuit1.f90:76-224), the
// direct-summation variant (circuit1.f90:227-305) and the temperature
// gradient used by the diffusion methods, with the adiabatic / isothermal EOS
// (eos.f90:21-45) fused into the epilogue.
//
// Two schedules give the reference's Jacobi iteration:
//  * k_c1_newton — without diffusion no particle reads another particle's
//    h, rho or Omega inside the loop (only positions and masses), so each
//    particle's sequence of iterates is independent of the others: one
//    thread runs its own Newton loop until |h_new - h|/h_0 <= tol or the
//    sweep cap, exactly the iterates the global loop gives it.
//  * k_c1_sweep — with a temperature gradient the sum reads the neighbours'
//    previous-sweep h, rho, Omega (circuit1.f90:163-179); one launch per
//    sweep over snapshot arrays, the host loops while any eps > tol.
#include "sph_internal.h"

namespace sph {
namespace {

constexpr int TPB = 128;

inline int nblocks(int64_t n, int tpb = TPB) {
  int64_t b = (n + tpb - 1) / tpb;
  return int(b < 1 ? 1 : b);
}

template <class R> struct PosAccess;
template <> struct PosAccess<double> {
  using Pos = PairPos<double>;
  static __device__ __forceinline__ double unit(const PackBufs&) { return 1.0; }
  static __device__ __forceinline__ PairPos<double> load(const PackBufs& pb, int64_t j, double& m) {
    const Rec64 a = ld_rec(&pb.d[0][j]);
    m = a.b.y;
    PairPos<double> r;
    r.x = a.a.x; r.y = a.a.y; r.z = a.b.x;
    return r;
  }
  static __device__ __forceinline__ double temp(const PackBufs& pb, int64_t j) {
    return __ldg(&pb.vt[j]).y;
  }
};
template <> struct PosAccess<float> {
  using Pos = FixPos;
  static __device__ __forceinline__ float unit(const PackBufs& pb) { return *pb.unit; }
  static __device__ __forceinline__ FixPos load(const PackBufs& pb, int64_t j, float& m) {
    const float4 a = __ldg(&pb.q[6][j]);
    m = a.w;
    FixPos r;
    r.x = __float_as_int(a.x); r.y = __float_as_int(a.y); r.z = __float_as_int(a.z);
    return r;
  }
  static __device__ __forceinline__ float temp(const PackBufs& pb, int64_t j) {
    return __ldg(&pb.q[4][j]).x;
  }
};

template <class R> __device__ __forceinline__ R rsq(R x) { return fsqrt<R>(x); }

// One Newton update from the summed density and dW/dh terms
// (circuit1.f90:191-206).  Returns eps; writes rho, Omega, h_new.
template <int DIM>
__device__ __forceinline__ double newton_update(double ha, double ha0, double ma, double hfac,
                                                double wsum, double osum, double& rho,
                                                double& om, double& hn) {
  rho = wsum;
  om = 1. - osum * (-ha / (DIM * rho));
  double dfdh = -DIM * rho * om / ha;
  double fh = ma * ipow<DIM>(hfac / ha) - rho;
  hn = ha - fh / dfdh;
  return fabs(hn - ha) / ha0;
}

__device__ __forceinline__ void eos_epilogue(double* cols, int64_t ld, int64_t p, double rho,
                                             const Params& P) {
  if (P.eos_kind == 1) {
    double pr = (P.gamma - 1.) * rho * cols[es_u * ld + p];
    cols[es_p * ld + p] = pr;
    cols[es_c * ld + p] = sqrt(P.gamma * pr / rho);
  } else if (P.eos_kind == 2) {
    cols[es_p * ld + p] = rho * P.c_iso * P.c_iso;
  }
}

// Sum a per-lane double over the G lanes of a group (all lanes get the sum).
template <int G>
__device__ __forceinline__ double group_sum(double v, unsigned gmask) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(gmask, v, o);
  return v;
}

template <int G>
__device__ __forceinline__ unsigned group_mask() {
  const int wl = threadIdx.x & 31;
  return (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (wl & ~(G - 1)));
}

// ---- fused Newton loop (no temperature gradient) ------------------------------------------
// G lanes per centre: each lane sums every G-th neighbour of the centre's
// row of the neighbour list (coalesced), the group adds its lanes' two-sum
// partials in FP64, and every lane takes the same FP64 Newton step.
// (FP64: 8 blocks per SM, 62 registers; a 96^3 blast of 4 steps took 9.66 ms,
// with 7 blocks 9.86, with 6 10.1.  FP32: 6 blocks per SM, 74 registers, no
// spill: 128^3, 4 lanes, density pass 3.22 ms, blast step 0.955; 7 blocks
// 3.39 / 0.936, 8 with 24 spilled bytes 3.46 / 1.026.)
template <int K, int DIM, class R, int G>
__global__ void __launch_bounds__(TPB, sizeof(R) == 4 ? 6 : 8)
k_c1_newton(C1Args a, PackBufs pb, Params P) {
  const int64_t c = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G;
  const int lane = threadIdx.x & (G - 1);
  const unsigned gmask = group_mask<G>();
  unsigned long long pairs = 0, sweeps = 0;
  int maxit = 0;
  if (c < a.nc) {
    const int64_t k = a.centre_k[c];
    const int64_t p = a.centre_p[c];
    double* cols = a.cols;
    const int64_t ld = a.ld;
    R mi;
    const typename PosAccess<R>::Pos pi = PosAccess<R>::load(pb, k, mi);
    const R punit = PosAccess<R>::unit(pb);
    const double ma = cols[es_m * ld + p];
    const double ha0 = cols[es_h * ld + p];
    const int n = a.ncnt[c];
    const int32_t* __restrict__ row = a.nl + a.rowoff[c];
    const double wcv = P.wCv;
    // kernel shape at q = 0 for the self term (circuit1.f90:191-194)
    R f0, df0;
    kshape_f_df<K, R>(R(0), f0, df0);
    double ha = ha0, rho = 0., om = 1., hn = ha0, eps_prev = 1e300;
    int it = 0;
    bool bad = false;
    for (;;) {
      ++it;
      // (the separations stay in fixed-point units: 1/h carries the unit, a
      // power of two, so q is the same as from physical separations)
      const double ihd_full = 1.0 / ha;
      const R ih0 = R(ihd_full);
      const R ih = ih0 * punit;
      const R ih_lo = R(ihd_full - double(ih0)) * punit;
      // the density sum keeps its two-sum partials (its smoothness in h is
      // what the Newton iteration needs); the d rho / dh sum only scales the
      // Newton step and Omega, so a plain per-lane sum suffices
      double sw_lane, so_lane;
      if constexpr (sizeof(R) == 4) {
        // U neighbours per lane per round: their pair data are all requested
        // before the first is used, so the gathers overlap; the list entries
        // of the next round are read one round ahead
        constexpr int U = 4;
        int32_t jn[U];
#pragma unroll
        for (int u = 0; u < U; ++u) jn[u] = (lane + u * G < n) ? row[lane + u * G] : -1;
        // FP32: two neighbours per packed instruction.  The kernel is bound
        // by instruction issue (79 % of the slots, FMA pipe 45 %, one pair at a time)
        // and has FMA time to spare.  An entry past the row's end is record
        // 0 with mass 0.  Separations are whole fixed-point units, so r2 is 0
        // or at least 1 and rsqrt(max(r2, 1)) serves both; q = r / h is NaN
        // or negative only if 1/h is.
        bad |= n > 0 && q_bad(float(ih));
        Acc2 sw;
        sw.init();
        F2 so(0.f);
        const F2 ih2(ih), nih2(-ih), ihl2(ih_lo);
        for (int l0 = lane; l0 < n; l0 += G * U) {
          FixPos pj[U];
          float mj[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            pj[u] = PosAccess<float>::load(pb, jn[u] >= 0 ? jn[u] : 0, mj[u]);
            if (jn[u] < 0) mj[u] = 0.f;
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int l = l0 + (U + u) * G;
            jn[u] = l < n ? row[l] : -1;
          }
#pragma unroll
          for (int u = 0; u < U; u += 2) {
            const F2 dx(__int2float_rn(pi.x - pj[u].x), __int2float_rn(pi.x - pj[u + 1].x));
            F2 r2 = f2_mul(dx, dx);
            if (DIM >= 2) {
              const F2 dy(__int2float_rn(pi.y - pj[u].y), __int2float_rn(pi.y - pj[u + 1].y));
              r2 = f2_fma(dy, dy, r2);
            }
            if (DIM == 3) {
              const F2 dz(__int2float_rn(pi.z - pj[u].z), __int2float_rn(pi.z - pj[u + 1].z));
              r2 = f2_fma(dz, dz, r2);
            }
            const F2 r = f2_mul(r2, F2(rsqrtf(fmaxf(r2.x(), 1.f)), rsqrtf(fmaxf(r2.y(), 1.f))));
            const F2 q = f2_mul(r, ih2);
            // q carries the FP32 rounding of r/h; its residual (exact via
            // FMA) and the residuals of the kernel pieces enter f to first
            // order, so the density sum varies smoothly with h below FP32
            // resolution and the Newton iterates converge instead of cycling
            // between neighbouring FP32 values (kshape_f_df_res).
            F2 f, df;
            kshape_f_df_res2<K>(q, r, nih2, ihl2, f, df);
            const F2 m2(mj[u], mj[u + 1]);
            sw.add(f2_mul(m2, f));
            so = f2_fma(m2, f2_fma(q, df, f2_mul(F2(float(DIM)), f)), so);
          }
        }
        sw_lane = sw.dval();
        so_lane = double(so.x()) + double(so.y());
      } else {
        Acc<R> sw;
        SumAcc<R> so;
        sw.init();
        so.init();
        // The next neighbour's record and the index after it are read ahead,
        // one neighbour per round (96^3, 4 lanes: 0.66 -> 0.57 ms; two per
        // round, their indices alone ahead, was the former).
        int32_t jnext = lane + G < n ? row[lane + G] : 0;
        R mn;
        typename PosAccess<R>::Pos pn = PosAccess<R>::load(pb, lane < n ? row[lane] : 0, mn);
        for (int l = lane; l < n; l += G) {
          const typename PosAccess<R>::Pos pj = pn;
          const R mj = mn;
          pn = PosAccess<R>::load(pb, jnext, mn);
          jnext = l + 2 * G < n ? row[l + 2 * G] : 0;
          R dx, dy, dz;
          pos_delta(pi, pj, dx, dy, dz, R(1));
          R r2 = dx * dx;
          if (DIM >= 2) r2 += dy * dy;
          if (DIM == 3) r2 += dz * dz;
          const R r = rsq<R>(r2);
          const R q = r * ih;
          bad |= q_bad(q);
          R f, df;
          kshape_f_df<K, R>(q, f, df);
          sw.add(mj * f);
          so.add(mj * (R(DIM) * f + q * df));
        }
        sw_lane = sw.dval();
        so_lane = so.dval();
      }
      const double swt = group_sum<G>(sw_lane, gmask);
      const double sot = group_sum<G>(so_lane, gmask);
      // W = wCv f / h^d; dW/dh = -wCv / h^(d+1) (d f + q f')  (kernel.f90:178-187, 239-249)
      const double ihd = 1.0 / ipow<DIM>(ha);
      const double wsum = wcv * ihd * (a.mref * swt + ma * double(f0));
      const double osum = -wcv * ihd / ha * (a.mref * sot + ma * (DIM * double(f0)));
      const double eps = newton_update<DIM>(ha, ha0, ma, P.hfac, wsum, osum, rho, om, hn);
      if (hn <= 0.) {
        if (lane == 0) raise_status(a.status, SPH_ERR_H_NEG);
        break;
      }
      if (!(eps > P.tol) || it >= P.maxiter) break;
      if constexpr (sizeof(R) == 4) {
        // FP32 sums carry a noise floor of a few 1e-9 in rho, i.e. ~1e-8 in
        // the Newton step, and the FP32 force pass moves a lattice at rest
        // by its rounding, so h drifts by ~1e-8 per step.  An eps below 1e-7
        // puts the stored rho within 3e-7 of the converged one, inside the
        // FP32 path's budget: stop there on the first sweep, and later once
        // eps no longer at least halves (further sweeps move h only within
        // that noise).  At 160^3 Sedov this keeps the sweeps per particle at
        // 1.00 instead of 1.4 (whole steps where every particle would take
        // a second sweep for an eps just above 1e-8).
        if (eps < 1e-7 && (it == 1 || eps >= 0.5 * eps_prev)) break;
      }
      eps_prev = eps;
      ha = hn;
    }
    if (bad) raise_status(a.status, (ha > 0.0) ? SPH_ERR_Q_NAN : SPH_ERR_Q_NEG);
    if (lane == 0) {
      pairs = (unsigned long long)n * it;
      sweeps = it;
      maxit = it;
      cols[es_h * ld + p] = hn;
      cols[es_den * ld + p] = rho;
      cols[es_om * ld + p] = om;
      cols[es_dtdx * ld + p] = 0.;
      cols[es_dtdy * ld + p] = 0.;
      cols[es_dtdz * ld + p] = 0.;
      eos_epilogue(cols, ld, p, rho, P);
    }
  }
  unsigned long long wp = pairs, ws = sweeps;
  for (int o = 16; o > 0; o >>= 1) {
    wp += __shfl_xor_sync(0xffffffffu, wp, o);
    ws += __shfl_xor_sync(0xffffffffu, ws, o);
    maxit = max(maxit, __shfl_xor_sync(0xffffffffu, maxit, o));
  }
  if ((threadIdx.x & 31) == 0) {
    if (wp) atomicAdd(&a.dcnt[DC_C1_PAIRS], wp);
    if (ws) atomicAdd(&a.dcnt[DC_C1_CENTRE_SWEEPS], ws);
    if (maxit) atomicMax(&a.dcnt[DC_C1_MAXSWEEPS], (unsigned long long)maxit);
  }
}

// ---- one Jacobi sweep (diffusion / FLD, and the direct summation) ------------------------
// Neighbours are read from the snapshot taken before the sweep, so the sweep
// stores its own rho, h, Omega and EOS in the table at once; h at the start
// of the iterate, which eps is relative to, waits in h0.  (Storing them
// apart cost four copies before the sweeps and a pass after: a 64^2
// diffusion iterate's circuit1 took 49 us for 8 us of sums, so 28.)
template <int K, int DIM, class R, int G>
__global__ void __launch_bounds__(TPB)
k_c1_sweep(C1Args a, PackBufs pb, Params P) {
  const int64_t c = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G;
  const int lane = threadIdx.x & (G - 1);
  const unsigned gmask = group_mask<G>();
  unsigned long long pairs = 0, sweeps = 0;
  int active_left = 0;
  if (c < a.nc) {
    const int64_t k = a.centre_k[c];
    const int64_t p = a.centre_p[c];
    double* cols = a.cols;
    const int64_t ld = a.ld;
    const bool first = a.iter_dev ? *a.iter_dev == 0 : a.first != 0;
    if (a.simple || first || a.eps[p] > P.tol) {
      R mi;
      const typename PosAccess<R>::Pos pi = PosAccess<R>::load(pb, k, mi);
      const R punit = PosAccess<R>::unit(pb);
      const double ma = cols[es_m * ld + p];
      const double ha = a.hk_s[k], rhoa = a.dk_s[k], oma = a.ok_s[k];
      const double ha0 = first ? ha : a.h0[p];
      const double ta = cols[es_t * ld + p];
      const int n = a.ncnt[c];
      const int32_t* __restrict__ row = a.nl + a.rowoff[c];
      const bool dT = a.simple ? (P.eq_diff && (P.ddw == esd_2nw_ds || P.ddw == esd_2nw_sd))
                               : (P.eq_diff || P.eq_fld);
      const R ih = R(1.0 / ha);
      const R ih_lo = R(1.0 / ha - double(ih));
      const double Ka = P.wCv / ipow<DIM + 1>(ha);  // wCv / h^(d+1)
      Acc<R> sw, so;
      sw.init();
      so.init();
      Acc<R> g[3];
      g[0].init(); g[1].init(); g[2].init();
      bool bad = false;
      const R rta = R(ta), rrhoa = R(rhoa), roma = R(oma);
      // the next neighbour's record and the index after it are read ahead
      // (256^2 FP32 diffusion 1.33 -> 1.30 ms a pass of 9 iterates, 64^2 FP64
      // 0.87 -> 0.83, against the index alone)
      int32_t j1 = lane < n ? row[lane] : 0, j2 = lane + G < n ? row[lane + G] : 0;
      R mn;
      typename PosAccess<R>::Pos pn = PosAccess<R>::load(pb, j1, mn);
      for (int l = lane; l < n; l += G) {
        const int64_t j = j1;
        const R mj = mn;
        const typename PosAccess<R>::Pos pj = pn;
        j1 = j2;
        pn = PosAccess<R>::load(pb, j1, mn);
        j2 = l + 2 * G < n ? row[l + 2 * G] : 0;
        R dx, dy, dz;
        pos_delta(pi, pj, dx, dy, dz, punit);
        R r2 = dx * dx;
        if (DIM >= 2) r2 += dy * dy;
        if (DIM == 3) r2 += dz * dz;
        const R r = rsq<R>(r2);
        const R q = r * ih;
        bad |= q_bad(q);
        R f, df;
        if constexpr (sizeof(R) == 4) kshape_f_df_res<K>(q, fmaf(r, ih, -q) + r * ih_lo, f, df);
        else kshape_f_df<K, R>(q, f, df);
        sw.add(mj * f);
        if (!a.simple) so.add(mj * (R(DIM) * f + q * df));
        if (dT) {
          const R tb = PosAccess<R>::temp(pb, j);
          // nabla W_a = wCv f'(q_a) r_ab / (h_a^(d+1) r)   (kernel.f90:189-197)
          const R ga = fdiv<R>(R(Ka) * df, r);
          R coef;
          if (P.ddw == esd_2nw_sd) {
            const double hb = a.hk_s[j], rhob = a.dk_s[j], omb = a.ok_s[j];
            const R qb = r * R(1.0 / hb);
            const R dfb = kshape_df<K, R>(qb);
            const R gb = fdiv<R>(R(P.wCv / ipow<DIM + 1>(hb)) * dfb, r);
            R ca, cb;
            if (a.simple) {  // circuit1.f90:289
              ca = rta / rrhoa / rrhoa;
              cb = tb / R(rhob) / R(rhob);
            } else {  // circuit1.f90:176
              ca = rta * rrhoa / roma / rrhoa / rrhoa;
              cb = tb * rrhoa / R(omb) / R(rhob) / R(rhob);
            }
            coef = mj * (ca * ga + cb * gb);
          } else if (a.simple) {  // 2nw_ds, circuit1.f90:284
            coef = mj / rrhoa * (tb - rta) * ga;
          } else {  // circuit1.f90:179
            const R rhob = R(a.dk_s[j]);
            coef = mj / rrhoa / roma * (tb * rhob - rta * rrhoa) * ga;
          }
          g[0].add(coef * dx);
          if (DIM >= 2) g[1].add(coef * dy);
          if (DIM == 3) g[2].add(coef * dz);
        }
      }
      pairs = (lane == 0) ? n : 0;
      sweeps = (lane == 0) ? 1 : 0;
      if (bad) raise_status(a.status, (ha > 0.0) ? SPH_ERR_Q_NAN : SPH_ERR_Q_NEG);
      const double swt = group_sum<G>(sw.dval(), gmask);
      const double sot = group_sum<G>(so.dval(), gmask);
      const double g0 = group_sum<G>(g[0].dval(), gmask);
      const double g1 = group_sum<G>(g[1].dval(), gmask);
      const double g2 = group_sum<G>(g[2].dval(), gmask);
      R f0, df0;
      kshape_f_df<K, R>(R(0), f0, df0);
      const double ihd = 1.0 / ipow<DIM>(ha);
      const double wsum = P.wCv * ihd * (a.mref * swt + ma * double(f0));
      if (lane == 0) {
        cols[es_dtdx * ld + p] = a.mref * g0;
        cols[es_dtdy * ld + p] = a.mref * g1;
        cols[es_dtdz * ld + p] = a.mref * g2;
        if (a.simple) {
          // circuit1.f90:293-301
          const double hnew = P.hfac * pow(ma / wsum, 1. / DIM);
          cols[es_den * ld + p] = wsum;
          cols[es_h * ld + p] = hnew;
          cols[es_om * ld + p] = 1.;
          eos_epilogue(cols, ld, p, wsum, P);
        } else {
          const double osum = -P.wCv * ihd / ha * (a.mref * sot + ma * (DIM * double(f0)));
          double rho, om, hn;
          double eps = newton_update<DIM>(ha, ha0, ma, P.hfac, wsum, osum, rho, om, hn);
          if (hn <= 0.) raise_status(a.status, SPH_ERR_H_NEG);
          if constexpr (sizeof(R) == 4) {
            // FP32 noise floor, as in k_c1_newton: an eps below 1e-7 on the
            // first sweep, or a stagnating one later, counts as converged
            // (a table at rest otherwise takes 2-3 sweeps per iterate that
            // move h only within the FP32 sums' noise)
            const double eps_prev = a.eps[p];
            if (eps > P.tol && eps < 1e-7 && (first || eps >= 0.5 * eps_prev)) eps = 0.0;
          }
          a.eps[p] = eps;
          if (first) a.h0[p] = ha;
          cols[es_den * ld + p] = rho;
          cols[es_om * ld + p] = om;
          cols[es_h * ld + p] = hn;
          eos_epilogue(cols, ld, p, rho, P);
          active_left = eps > P.tol ? 1 : 0;
        }
      }
    }
  }
  unsigned long long wp = pairs, ws = sweeps;
  for (int o = 16; o > 0; o >>= 1) {
    wp += __shfl_xor_sync(0xffffffffu, wp, o);
    ws += __shfl_xor_sync(0xffffffffu, ws, o);
    active_left |= __shfl_xor_sync(0xffffffffu, active_left, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (wp) atomicAdd(&a.dcnt[DC_C1_PAIRS], wp);
    if (ws) atomicAdd(&a.dcnt[DC_C1_CENTRE_SWEEPS], ws);
    if (active_left) atomicOr(&a.red[a.active_slot], 1ull);
  }
}

// h, rho and Omega of every record from its row; clears the word active[0]
// in which the sweep marks that a particle stays active, having counted in
// active[1] the sweeps before this one that left one
__global__ void k_c1_snapshot(int64_t n, const int32_t* __restrict__ ssrc,
                              const double* __restrict__ cols, int64_t ld,
                              double* __restrict__ hk_s, double* __restrict__ dk_s,
                              double* __restrict__ ok_s, unsigned long long* __restrict__ active, int first,
                              const DevPlan* __restrict__ plan) {
  int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (k == 0) {
    active[1] = first ? 0ull : active[1] + (active[0] ? 1ull : 0ull);
    active[0] = 0ull;
  }
  if (plan) n = plan->nall;  // launched over the capacity
  if (k >= n) return;
  int64_t p = ssrc[k];
  hk_s[k] = cols[es_h * ld + p];
  dk_s[k] = cols[es_den * ld + p];
  ok_s[k] = cols[es_om * ld + p];
}

// direct summation: Omega = 1 on the rows that are no centres (circuit1.f90:62)
__global__ void k_c1_simple_rest(int64_t nrows, int64_t nreal, double* __restrict__ cols,
                                 int64_t ld) {
  const int64_t p = nreal + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p < nrows) cols[es_om * ld + p] = 1.;
}

template <int K, int DIM, class R>
void dispatch_newton(int G, const C1Args& a, const PackBufs& pb, const Params& P, cudaStream_t s) {
  switch (G) {
    case 4: k_c1_newton<K, DIM, R, 4><<<nblocks(a.nc * 4), TPB, 0, s>>>(a, pb, P); break;
    case 8: k_c1_newton<K, DIM, R, 8><<<nblocks(a.nc * 8), TPB, 0, s>>>(a, pb, P); break;
    case 16: k_c1_newton<K, DIM, R, 16><<<nblocks(a.nc * 16), TPB, 0, s>>>(a, pb, P); break;
    default: k_c1_newton<K, DIM, R, 32><<<nblocks(a.nc * 32), TPB, 0, s>>>(a, pb, P); break;
  }
  note_launch();
}
template <int K, int DIM, class R>
void dispatch_sweep(int G, const C1Args& a, const PackBufs& pb, const Params& P, cudaStream_t s) {
  switch (G) {
    case 4: k_c1_sweep<K, DIM, R, 4><<<nblocks(a.nc * 4), TPB, 0, s>>>(a, pb, P); break;
    case 8: k_c1_sweep<K, DIM, R, 8><<<nblocks(a.nc * 8), TPB, 0, s>>>(a, pb, P); break;
    case 16: k_c1_sweep<K, DIM, R, 16><<<nblocks(a.nc * 16), TPB, 0, s>>>(a, pb, P); break;
    default: k_c1_sweep<K, DIM, R, 32><<<nblocks(a.nc * 32), TPB, 0, s>>>(a, pb, P); break;
  }
  note_launch();
}

#define SPH_DISPATCH(FN)                                                             \
  template <int K, int DIM>                                                          \
  void FN##_prec(int prec, const C1Args& a, const PackBufs& pb, const Params& P,    \
                 cudaStream_t s) {                                                   \
    if (prec == SPH_PREC_FP64) FN<K, DIM, double>(a.G, a, pb, P, s);                 \
    else FN<K, DIM, float>(a.G, a, pb, P, s);                                        \
  }                                                                                  \
  template <int K>                                                                   \
  void FN##_dim(int prec, int dim, const C1Args& a, const PackBufs& pb,             \
                const Params& P, cudaStream_t s) {                                   \
    if (dim == 3) FN##_prec<K, 3>(prec, a, pb, P, s);                                \
    else if (dim == 2) FN##_prec<K, 2>(prec, a, pb, P, s);                           \
    else FN##_prec<K, 1>(prec, a, pb, P, s);                                         \
  }                                                                                  \
  void FN##_all(int prec, int kernel, int dim, const C1Args& a, const PackBufs& pb, \
                const Params& P, cudaStream_t s) {                                   \
    if (kernel == KM6) FN##_dim<KM6>(prec, dim, a, pb, P, s);                        \
    else if (kernel == KM4) FN##_dim<KM4>(prec, dim, a, pb, P, s);                   \
    else FN##_dim<KGAUSS>(prec, dim, a, pb, P, s);                                   \
  }

SPH_DISPATCH(dispatch_newton)
SPH_DISPATCH(dispatch_sweep)

}  // namespace

void launch_c1_newton(int prec, int kernel, int dim, const C1Args& a, PackBufs pb, Params P,
                      cudaStream_t s) {
  dispatch_newton_all(prec, kernel, dim, a, pb, P, s);
}
void launch_c1_sweep(int prec, int kernel, int dim, const C1Args& a, PackBufs pb, Params P,
                     cudaStream_t s) {
  dispatch_sweep_all(prec, kernel, dim, a, pb, P, s);
}
void launch_c1_simple_rest(int64_t nrows, int64_t nreal, double* cols, cudaStream_t s) {
  if (nrows <= nreal) return;
  k_c1_simple_rest<<<nblocks(nrows - nreal, 256), 256, 0, s>>>(nrows, nreal, cols, nrows);
  note_launch();
}
void launch_c1_snapshot(int64_t n, const int32_t* ssrc, const double* cols, int64_t ld,
                        double* hk_s, double* dk_s, double* ok_s, unsigned long long* active,
                        int first, cudaStream_t s, const DevPlan* plan) {
  k_c1_snapshot<<<nblocks(n, 256), 256, 0, s>>>(n, ssrc, cols, ld, hk_s, dk_s, ok_s, active,
                                                first, plan);
  note_launch();
}

}  // namespace sph
