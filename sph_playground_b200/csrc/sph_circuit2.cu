// sph_circuit2.cu — circuit2 on the device: the per-pair forces of
// circuit2.f90:58-505 (hydro pressure force and energy, Monaghan artificial
// viscosity :558-575, artificial conductivity :520-529, dh/dt from the
// continuity term, anisotropic / isotropic / flux-limited diffusion with the
// run-time second-derivative method, ideal-MHD stress and induction).
//
// G lanes per centre walk its neighbour list (lane l takes entries l, l + G,
// ...); neighbour data come from the packed sorted-order streams.  All
// nabla W terms are written as g * r_ab with
//   g_a = wCv f'(q_a) / (h_a^(d+1) r)      (nw_cart, kernel.f90:189-197)
// and the reference's per-pair divisions by rho^2 Omega are the per-particle
// factor Pi = 1/(rho^2 Omega) computed once when the streams are packed.
// The "ddw device function table" of kernel.f90:19-23 (procedure pointers
// nw, fab, n2w, hessian) is the run-time switch on P.ddw below; the branch
// is uniform across a launch, so it does not diverge.
//
// One instance per kind of run (C2Mode): an instance that served every set of
// equations held the conductivity tensors, both fields and every sum at once
// and spilled 350 bytes (2D FP64) to 680 (3D FP64) per thread.
// (Per iterate, before and after: MHD 201^2 FP64 57 and 37 us, diffusion by two
// first derivatives 256^2 FP32 50 and 27.)
#include "sph_internal.h"

namespace sph {
namespace {

constexpr int TPB = 128;

inline int nblocks(int64_t n, int tpb = TPB) {
  int64_t b = (n + tpb - 1) / tpb;
  return int(b < 1 ? 1 : b);
}

enum C2Mode : int {
  C2_HYDRO,    // hydrodynamics alone
  C2_MHD,      // with the magnetic field
  C2_HESSIAN,  // diffusion alone, by a Hessian method (fab, fw, n2w)
  C2_TWO_NW,   // diffusion alone, by two first derivatives
  C2_GENERAL   // every other set: flux-limited diffusion, diffusion with hydrodynamics or field
};

template <class R> struct Part {
  PairPos<R> pos;
  // Pi of a neighbour is the record's wCv / (h^(d+1) rho^2 Omega), of the
  // centre 1 / (rho^2 Omega); hrho = rho / 2, ac = alpha c, u = au u
  R m, invh, rho, hrho, Pi, P, ac, u, vx, vy, vz;
};
template <class R> struct PartX {
  R T, kappa, gx, gy, gz, bx, by, bz;
};

template <class R> struct Loader;
template <> struct Loader<double> {
  static __device__ __forceinline__ void hydro(const PackBufs& pb, int64_t j, Part<double>& o) {
    hydro(pb, j, ahead(pb, j), o);
  }
  // the part of a neighbour's record that is read one round ahead (AHEAD)
  struct Ahead { Rec64 a; };
  static __device__ __forceinline__ Ahead ahead(const PackBufs& pb, int64_t j) {
    return {ld_rec(&pb.d[0][j])};
  }
  static __device__ __forceinline__ void hydro(const PackBufs& pb, int64_t j, const Ahead& h,
                                               Part<double>& o) {
    const Rec64 a = h.a, c = ld_rec(&pb.d[1][j]), e = ld_rec(&pb.d[2][j]);
    o.vz = __ldg(&pb.vt[j].x);
    o.pos.x = a.a.x; o.pos.y = a.a.y; o.pos.z = a.b.x; o.m = a.b.y;
    o.invh = c.a.x; o.hrho = c.a.y; o.rho = 2.0 * c.a.y; o.Pi = c.b.x; o.P = c.b.y;
    o.ac = e.a.x; o.u = e.a.y; o.vx = e.b.x; o.vy = e.b.y;
  }
  // (what a mode does not use is not read)
  template <int MODE>
  static __device__ __forceinline__ void extra(const PackBufs& pb, int64_t j, PartX<double>& o) {
    if constexpr (MODE != C2_MHD) o.T = __ldg(&pb.vt[j].y);
    if constexpr (MODE == C2_TWO_NW || MODE == C2_GENERAL) {
      const Rec64 h = ld_rec(&pb.d[3][j]);
      o.kappa = h.a.x; o.gx = h.a.y; o.gy = h.b.x; o.gz = h.b.y;
    }
    const Rec64 k = ld_rec(&pb.d[4][j]);
    o.bx = k.a.x; o.by = k.a.y; o.bz = k.b.x;
  }
};
template <> struct Loader<float> {
  struct Ahead {};
  static __device__ __forceinline__ Ahead ahead(const PackBufs&, int64_t) { return {}; }
  static __device__ __forceinline__ void hydro(const PackBufs& pb, int64_t j, const Ahead&,
                                               Part<float>& o) {
    hydro(pb, j, o);
  }
  static __device__ __forceinline__ void hydro(const PackBufs& pb, int64_t j, Part<float>& o) {
    float4 a = __ldg(&pb.q[0][j]), b = __ldg(&pb.q[1][j]), c = __ldg(&pb.q[2][j]),
           d = __ldg(&pb.q[3][j]);
    o.pos.xh = a.x; o.pos.yh = a.y; o.pos.zh = a.z; o.m = a.w;
    o.pos.xl = b.x; o.pos.yl = b.y; o.pos.zl = b.z; o.invh = b.w;
    o.hrho = c.x; o.rho = 2.f * c.x; o.Pi = c.y; o.P = c.z; o.ac = c.w;
    o.u = d.x; o.vx = d.y; o.vy = d.z; o.vz = d.w;
  }
  template <int MODE>
  static __device__ __forceinline__ void extra(const PackBufs& pb, int64_t j, PartX<float>& o) {
    float4 e = __ldg(&pb.q[4][j]), f = __ldg(&pb.q[5][j]);
    o.T = e.x; o.kappa = e.y; o.gx = e.z; o.gy = e.w;
    o.gz = f.x; o.bx = f.y; o.by = f.z; o.bz = f.w;
  }
};

template <class R> __device__ __forceinline__ R my_sqrt(R x);
template <> __device__ __forceinline__ double my_sqrt<double>(double x) { return sqrt(x); }
template <> __device__ __forceinline__ float my_sqrt<float>(float x) { return sqrtf(x); }

// Conductivity tensor of a particle (circuit2.f90:203-205, 371-373): isotropic
// s I, the diagonal form diag(w) with w = k_par b_x^2, ..., or the full
// k_par w w^T with w the unit vector; which of them is the run's (KKind).
enum KKind : int { K_ISO, K_DIAG, K_FULL };
template <class R>
struct Tensor {
  R s, w[3];
  __device__ __forceinline__ void init() { s = R(0); w[0] = w[1] = w[2] = R(0); }
  // from the unit vector of the field
  __device__ __forceinline__ void aniso(int kind, R k_par, R x, R y, R z) {
    s = k_par;
    w[0] = kind == K_FULL ? x : k_par * x * x;
    w[1] = kind == K_FULL ? y : k_par * y * y;
    w[2] = kind == K_FULL ? z : k_par * z * z;
  }
  template <int DIM>
  __device__ __forceinline__ R trace(int kind) const {
    if (kind == K_ISO) return R(DIM) * s;
    R t = R(0);
    for (int x = 0; x < DIM; ++x) t += kind == K_FULL ? s * w[x] * w[x] : w[x];
    return t;
  }
  // r . K r over the run's axes
  template <int DIM>
  __device__ __forceinline__ R form(int kind, const R* r) const {
    R t = R(0);
    if (kind == K_FULL) {
      for (int x = 0; x < DIM; ++x) t += w[x] * r[x];
      return s * t * t;
    }
    for (int x = 0; x < DIM; ++x) t += (kind == K_ISO ? s : w[x]) * r[x] * r[x];
    return t;
  }
  __device__ __forceinline__ void apply(int kind, const R* g, R* out) const {
    const R d = kind == K_FULL ? s * (w[0] * g[0] + w[1] * g[1] + w[2] * g[2]) : R(0);
    for (int x = 0; x < 3; ++x)
      out[x] = kind == K_FULL ? w[x] * d : (kind == K_ISO ? s : w[x]) * g[x];
  }
};

// flux-limited diffusion coefficient (circuit2.f90:180-183, 358-361)
template <class R>
__device__ __forceinline__ R fld_coef(R gnorm, R kappa, R rho, R T, R& lambda) {
  R fr = gnorm / (kappa * rho * rho * T);
  lambda = (R(2) + fr) / (R(6) + R(3) * fr + fr * fr);
  return R(kLightspeed) * lambda / kappa / rho;
}

template <int G>
__device__ __forceinline__ double group_sum(double v, unsigned gmask) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(gmask, v, o);
  return v;
}

// G lanes per centre: lane l takes neighbours l, l+G, ... of the centre's
// list row; per-lane partial sums are added over the group in FP64 and
// lane 0 stores the result.
// (FP32: 9 blocks of 128 threads per SM, 56 registers with a 4-byte spill,
// measured 2.01 -> 1.95 ms on the 128^3 Sedov step against 8 blocks at 64
// registers; 10 blocks spill 44 bytes and take 2.5 ms)
template <int K, int DIM, class R, int MODE, int G>
__global__ void __launch_bounds__(TPB, sizeof(R) == 8 ? 5 : MODE == C2_HYDRO ? 9 : 7)
k_c2(C2Args a, PackBufs pb, Params P) {
  // The next neighbour's position is read a round ahead, so that r, its root
  // and the kernel do not wait for memory at the head of every round: FP64
  // hydrodynamics alone, long-scoreboard stalls 4.2 of 9 cycles an
  // instruction before (96^3, with 20 warps per SM: 1.60 -> 1.42 ms; with 1/h
  // and P as well 1.51, or 1.45 at 4 blocks per SM; position alone at 4 blocks
  // 1.48).  FP32 has 36 warps per SM and no registers left: 1.98 -> 2.07 ms
  // at 128^3.  With the field or diffusion no gain.
  constexpr bool AHEAD = sizeof(R) == 8 && MODE == C2_HYDRO;
  constexpr bool HEAT = MODE == C2_HESSIAN || MODE == C2_TWO_NW || MODE == C2_GENERAL;
  constexpr bool FIELD = MODE == C2_MHD || MODE == C2_GENERAL;
  constexpr bool PRESSURE = MODE == C2_HYDRO || MODE == C2_MHD || MODE == C2_GENERAL;
  const int64_t c = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) / G;
  const int lane = threadIdx.x & (G - 1);
  const int wl = threadIdx.x & 31;
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (wl & ~(G - 1)));
  unsigned long long pairs = 0;
  if (c < a.nc) {
    const int64_t k = a.centre_k[c];
    const int64_t p = a.centre_p[c];
    double* cols = a.cols;
    const int64_t ld = a.ld;
    Part<R> A;
    Loader<R>::hydro(pb, k, A);
    {
      // the record's second rho field is wCv Pi / h^(d+1), the
      // neighbour-side product; the centre takes Pi itself
      const double rr = cols[es_den * ld + p], oo = cols[es_om * ld + p];
      A.Pi = R(1.0 / (rr * rr * oo));
    }
    R Kh = A.invh;
    for (int d = 0; d < DIM; ++d) Kh *= A.invh;
    Kh *= R(P.wCv);                      // wCv / h_a^(d+1)
    const R Ka = Kh * R(KDfScale<K>::v);  // with f'(q) as kshape_df_scaled
    const R beta = R(P.beta);
    const bool artts = PRESSURE && P.artts == 1, adden = P.adden == 1,
               hydro = PRESSURE && P.eq_hydro != 0;
    const bool heat = MODE == C2_GENERAL ? P.eq_diff != 0 : HEAT;
    const bool field = MODE == C2_GENERAL ? P.eq_magneto != 0 : FIELD;
    const bool fld = MODE == C2_GENERAL && P.eq_fld != 0;
    const bool hessian = MODE == C2_HESSIAN ||
                         (MODE == C2_GENERAL &&
                          (P.ddw == esd_fab || P.ddw == esd_fw || P.ddw == esd_n2w));
    // the artificial conductivity term (circuit2.f90:316-331) is scaled by
    // au: au = -1 switches it off in the reference, and au = 0 makes it
    // vanish, so it is skipped for both
    const bool use_au = P.au != -1.0 && P.au != 0.0;
    const R rPiA = A.rho * A.Pi;  // 1 / (rho_a Omega_a)
    const R alpha_ca = A.ac;
    const R hrhoa = R(-0.5) * A.rho, hrho_a = R(0.5) * A.rho, rPiA_h = R(0.5) * rPiA;
    const R PiPa = hydro ? A.Pi * A.P : R(0);  // Pi_a P_a
    // force-type sums: plain per lane (a few tens of terms), FP64 over lanes
    SumAcc<R> dv[3], du, drho, ddt, db[3];
    for (int d = 0; d < 3; ++d) { dv[d].init(); db[d].init(); }
    du.init(); drho.init(); ddt.init();

    // ---- per-centre set-up of the other equations ----
    PartX<R> AX;
    Tensor<R> kta, ktb;
    const int kind = fld || P.difiso == 1 ? K_ISO : P.full_tensor ? K_FULL : K_DIAG;
    R kga[3] = {R(0), R(0), R(0)};  // K_a grad T_a
    R halfB2a = R(0);
    const R mu0inv = R(1.0 / P.muzero);
    SumAcc<R> tension;  // sum of m_b (B_a . r) g_a Pi_a / mu0, which meets B_a
    tension.init();
    if constexpr (MODE != C2_HYDRO) {
      Loader<R>::template extra<MODE>(pb, k, AX);
      const R b2 = AX.bx * AX.bx + AX.by * AX.by + AX.bz * AX.bz;
      halfB2a = R(0.5) * b2;
      kta.init();
      ktb.init();
      if (heat) {
        if (fld) {
          R lam;
          R gn = my_sqrt<R>(AX.gx * AX.gx + AX.gy * AX.gy + AX.gz * AX.gz);
          R fd = fld_coef<R>(gn, AX.kappa, A.rho, AX.T, lam);
          kta.s = fd;
          if (lane == 0)
            cols[es_vfld * ld + p] = double(fd) / ((double(AX.T) * double(A.rho)) / double(gn));
        } else if (P.difiso == 1) {
          kta.s = ktb.s = R(P.difcond);
        } else {
          R ux = AX.bx, uy = AX.by, uz = AX.bz;
          if (b2 != R(0)) to_unit(b2, ux, uy, uz);
          else ux = uy = uz = R(0);
          kta.aniso(kind, R(P.difcond), ux, uy, uz);
        }
        if (!hessian) {
          const R ga3[3] = {AX.gx, AX.gy, AX.gz};
          kta.apply(kind, ga3, kga);
        }
      }
    }
    const R tra = MODE != C2_HYDRO && hessian ? kta.template trace<DIM>(kind) : R(0);

    bool bad = false;
    const int n = a.ncnt[c];
    const int32_t* __restrict__ row = a.nl + a.rowoff[c];
    // the next neighbour's index is read one round ahead, so that a round
    // waits on one dependent load (the neighbour's streams), not two
    int32_t jnext = lane < n ? row[lane] : 0, jnext2 = 0;
    typename Loader<R>::Ahead next;
    if constexpr (AHEAD) {
      jnext2 = lane + G < n ? row[lane + G] : 0;
      next = Loader<R>::ahead(pb, jnext);
    }
    for (int l0 = lane; l0 < n; l0 += G) {
    {
      const int64_t j = jnext;
      Part<R> B;
      if constexpr (AHEAD) {
        Loader<R>::hydro(pb, j, next, B);
        jnext = jnext2;
        next = Loader<R>::ahead(pb, jnext);
        if (l0 + 2 * G < n) jnext2 = row[l0 + 2 * G];
      } else {
        Loader<R>::hydro(pb, j, B);
        if (l0 + G < n) jnext = row[l0 + G];
      }
      R rab[3];
      pos_delta(A.pos, B.pos, rab[0], rab[1], rab[2]);
      R r2 = rab[0] * rab[0];
      if (DIM >= 2) r2 += rab[1] * rab[1];
      if (DIM == 3) r2 += rab[2] * rab[2];
      const R invr = frsqrt<R>(r2);
      const R r = r2 * invr;
      const R vab[3] = {A.vx - B.vx, A.vy - B.vy, A.vz - B.vz};
      R vr = vab[0] * rab[0];
      if (DIM >= 2) vr += vab[1] * rab[1];
      if (DIM == 3) vr += vab[2] * rab[2];
      const R qa = r * A.invh, qb = r * B.invh;
      bad |= q_bad(qa) || q_bad(qb);
      R fa = R(0), dfa, ddfa = R(0);
      if constexpr (HEAT) {
        if (heat && hessian && P.ddw != esd_fab) {
          R d1;
          kshape_all<K, R>(qa, fa, d1, ddfa);
        }
      }
      dfa = kshape_df_scaled<K, R>(qa);
      const R dfb = kshape_df_scaled<K, R>(qb);
      const R ga = (Ka * invr) * dfa;  // nabla W_a = ga * r_ab
      // nabla W_b = gb r_ab, which always meets Pi_b: gbPi = gb Pi_b, and
      // cbr = wCv f'_b rho_b Pi_b / (2 h_b^(d+1)) for the conductivity (its
      // 1/2 folded in).  The record carries wCv Pi_b / h_b^(d+1) with the
      // scale of f', a product formed in FP64 when packed.
      const R gbPi = (B.Pi * invr) * dfb;
      const R cbr = (B.Pi * dfb) * B.hrho;
      const R mb = B.m;
      const R mgv = mb * ga * vr;      // m_b nabla W_a . v_ab
      if (adden) drho.add(mgv);        // circuit2.f90:265-267
      // F = ga (Pi_a Fa) + gbPi Fb (dv -= mb F r_ab); du += mgv (Pi_a Da).
      // With faba = Ka f'_a = ga r the viscous heating
      // mb dvr qav faba / (rho_a Omega_a) of circuit2.f90:329-334 is
      // mgv Pi_a (qav rho_a), and the pressure work of :343-344 is
      // mgv Pi_a P_a.  Pi_a is folded into the centre's terms.
      R FaPi = PiPa, Fb = R(0), DaPi = PiPa;
      if (artts) {
        // circuit2.f90:294-336; the Monaghan switch dvr < 0 as a clamp
        // (the record carries rho_b / 2 and alpha c_b)
        const R dvr = vr * invr;
        const R dneg = rmin0(dvr);
        const R qav = hrhoa * (alpha_ca - beta * dneg) * dneg;
        const R qbv = (-B.hrho) * (B.ac - beta * dneg) * dneg;
        Fb = qbv;
        FaPi = A.Pi * qav + PiPa;
        DaPi = qav * rPiA + PiPa;
        if (use_au) {  // (u is au u)
          const R faba = Ka * dfa;
          const R vsigu = froot_ratio(R(fabs(A.P - B.P)), hrho_a + B.hrho);
          du.add(mb * (vsigu * (A.u - B.u) * (faba * rPiA_h + cbr)));
        }
      }
      if (hydro) Fb += B.P;  // circuit2.f90:338-345
      const R F = ga * FaPi + gbPi * Fb;
      du.add(mgv * DaPi);
      R Fr = F;  // the force's factor along r_ab
      if constexpr (MODE != C2_HYDRO) {
        PartX<R> BX;
        Loader<R>::template extra<MODE>(pb, j, BX);
        if (heat) {
          // circuit2.f90:347-425
          if (fld) {
            R lam;
            R gn = my_sqrt<R>(BX.gx * BX.gx + BX.gy * BX.gy + BX.gz * BX.gz);
            ktb.s = fld_coef<R>(gn, BX.kappa, B.rho, BX.T, lam);
          } else if (P.difiso == 0) {
            const R b2 = BX.bx * BX.bx + BX.by * BX.by + BX.bz * BX.bz;
            if (b2 != R(0)) {  // a zero B_b keeps the previous tensor (:220-224)
              R ux = BX.bx, uy = BX.by, uz = BX.bz;
              to_unit(b2, ux, uy, uz);
              ktb.aniso(kind, R(P.difcond), ux, uy, uz);
            }
          }
          if (hessian) {
            // K_bar : Hessian_a  (kernel.f90:377-539, circuit2.f90:390-397)
            const R tr = R(0.5) * (tra + ktb.template trace<DIM>(kind));
            const R rr = R(0.5) * (kta.template form<DIM>(kind, rab) + ktb.template form<DIM>(kind, rab)) *
                         (invr * invr);
            R contr;
            if (P.ddw == esd_n2w) {
              contr = Kh * A.invh * ddfa * rr + ga * (tr - rr);
            } else {
              const R f2 = (P.ddw == esd_fab) ? -ga : R(0.5) * R(P.fwc) * Kh * A.invh * fa;
              contr = f2 * (R(DIM + 2) * rr - tr);
            }
            ddt.add(fdiv<R>(mb, B.rho * A.rho) * (BX.T * B.rho - AX.T * A.rho) * contr);
          } else {
            R kgb[3];
            const R gb3[3] = {BX.gx, BX.gy, BX.gz};
            ktb.apply(kind, gb3, kgb);
            R ka_r = R(0), kb_r = R(0);
            for (int x = 0; x < DIM; ++x) { ka_r += kga[x] * rab[x]; kb_r += kgb[x] * rab[x]; }
            if (P.ddw == esd_2nw_ds) ddt.add(mb * (ga * ka_r * A.Pi + gbPi * kb_r));
            else ddt.add(mb * A.Pi * ga * (kb_r - ka_r));  // esd_2nw_sd
          }
        }
        if (field) {
          // circuit2.f90:427-462: the stress of a is (B_a^2 / 2 r_ab -
          // B_a (B_a . r_ab)) / mu0; its first part joins the pressure's
          // factor, its second meets the centre's own B_a after the loop
          const R Ba[3] = {AX.bx, AX.by, AX.bz}, Bb[3] = {BX.bx, BX.by, BX.bz};
          R Bar = R(0), Bbr = R(0);
          for (int x = 0; x < DIM; ++x) { Bar += Ba[x] * rab[x]; Bbr += Bb[x] * rab[x]; }
          const R halfB2b = R(0.5) * (Bb[0] * Bb[0] + Bb[1] * Bb[1] + Bb[2] * Bb[2]);
          const R gam = ga * A.Pi * mu0inv, gbm = gbPi * mu0inv;
          Fr += gam * halfB2a + gbm * halfB2b;
          tension.add(mb * (gam * Bar));
          const R tb = mb * (gbm * Bbr), mga = mb * ga;
          for (int x = 0; x < 3; ++x) {
            dv[x].add(tb * Bb[x]);
            db[x].add(mga * (Bb[x] * vr - vab[x] * Bar));
          }
        }
      }
      if constexpr (PRESSURE)
        for (int d = 0; d < DIM; ++d) dv[d].add(-mb * Fr * rab[d]);
    }
    }
    if (bad) raise_status(a.status, SPH_ERR_Q_NAN);
    const double mref = a.mref;
    double ax = 0.0, ay = 0.0, az = 0.0, dus = 0.0;
    if constexpr (PRESSURE) {
      ax = group_sum<G>(dv[0].dval(), gmask);
      if (DIM >= 2 || FIELD) ay = group_sum<G>(dv[1].dval(), gmask);
      if (DIM == 3 || FIELD) az = group_sum<G>(dv[2].dval(), gmask);
      dus = group_sum<G>(du.dval(), gmask);
    }
    const double drs = group_sum<G>(drho.dval(), gmask);
    double dts = 0.0, b0 = 0.0, b1 = 0.0, b2 = 0.0;
    if constexpr (HEAT) dts = group_sum<G>(ddt.dval(), gmask);
    if constexpr (FIELD) {
      const double t = group_sum<G>(tension.dval(), gmask), rp = double(rPiA);
      ax += t * double(AX.bx);
      ay += t * double(AX.by);
      az += t * double(AX.bz);
      b0 = rp * group_sum<G>(db[0].dval(), gmask);
      b1 = rp * group_sum<G>(db[1].dval(), gmask);
      b2 = rp * group_sum<G>(db[2].dval(), gmask);
    }
    if (lane == 0) {
      pairs = n;
      cols[es_ax * ld + p] = mref * ax;
      cols[es_ay * ld + p] = mref * ay;
      cols[es_az * ld + p] = mref * az;
      cols[es_du * ld + p] = mref * dus;
      double dh = 0.;
      if (adden) {  // circuit2.f90:468-470
        const double ha = cols[es_h * ld + p];
        dh = -double(DIM) * ha * double(A.rho) * double(A.Pi) * (mref * drs);
      }
      cols[es_dh * ld + p] = dh;
      cols[es_ddt * ld + p] = mref * dts;
      cols[es_dbx * ld + p] = mref * b0;
      cols[es_dby * ld + p] = mref * b1;
      cols[es_dbz * ld + p] = mref * b2;
    }
  }
  unsigned long long wp = pairs;
  for (int o = 16; o > 0; o >>= 1) wp += __shfl_xor_sync(0xffffffffu, wp, o);
  if (wl == 0 && wp) atomicAdd(&a.dcnt[DC_C2_PAIRS], wp);
}

template <int K, int DIM, class R, int MODE>
void run_g(const C2Args& a, const PackBufs& pb, const Params& P, cudaStream_t s) {
  switch (a.G) {
    case 4: k_c2<K, DIM, R, MODE, 4><<<nblocks(a.nc * 4), TPB, 0, s>>>(a, pb, P); break;
    case 8: k_c2<K, DIM, R, MODE, 8><<<nblocks(a.nc * 8), TPB, 0, s>>>(a, pb, P); break;
    case 16: k_c2<K, DIM, R, MODE, 16><<<nblocks(a.nc * 16), TPB, 0, s>>>(a, pb, P); break;
    default: k_c2<K, DIM, R, MODE, 32><<<nblocks(a.nc * 32), TPB, 0, s>>>(a, pb, P); break;
  }
}
template <int K, int DIM, class R>
void run(const C2Args& a, const PackBufs& pb, const Params& P, cudaStream_t s) {
  const bool alone = P.eq_diff && !P.eq_hydro && !P.eq_magneto && !P.eq_fld && P.artts != 1;
  if (!P.eq_diff && !P.eq_magneto) run_g<K, DIM, R, C2_HYDRO>(a, pb, P, s);
  else if (!P.eq_diff) run_g<K, DIM, R, C2_MHD>(a, pb, P, s);
  else if (!alone) run_g<K, DIM, R, C2_GENERAL>(a, pb, P, s);
  else if (P.ddw == esd_fab || P.ddw == esd_fw || P.ddw == esd_n2w)
    run_g<K, DIM, R, C2_HESSIAN>(a, pb, P, s);
  else run_g<K, DIM, R, C2_TWO_NW>(a, pb, P, s);
  note_launch();
}
template <int K, int DIM>
void run_prec(int prec, const C2Args& a, const PackBufs& pb, const Params& P, cudaStream_t s) {
  if (prec == SPH_PREC_FP64) run<K, DIM, double>(a, pb, P, s);
  else run<K, DIM, float>(a, pb, P, s);
}
template <int K>
void run_dim(int prec, int dim, const C2Args& a, const PackBufs& pb, const Params& P,
             cudaStream_t s) {
  if (dim == 3) run_prec<K, 3>(prec, a, pb, P, s);
  else if (dim == 2) run_prec<K, 2>(prec, a, pb, P, s);
  else run_prec<K, 1>(prec, a, pb, P, s);
}

}  // namespace

void launch_c2(int prec, int kernel, int dim, const C2Args& a, PackBufs pb, Params P,
               cudaStream_t s) {
  if (kernel == KM6) run_dim<KM6>(prec, dim, a, pb, P, s);
  else if (kernel == KM4) run_dim<KM4>(prec, dim, a, pb, P, s);
  else run_dim<KGAUSS>(prec, dim, a, pb, P, s);
}

}  // namespace sph
