// Warp-per-cell FP64 reaction step for mechanisms with NC+1 <= 32 equations.
//
// One warp integrates one cell.  Lane l owns ODE component l (species mass
// fraction l, lane NC owns T); reaction-parallel work (rate constants,
// products of concentrations) is spread over the 32 lanes.  Every quantity the
// reference accumulates sequentially (mixture sums, WRMS norms, L1 norms,
// formation rates, reaction enthalpies) is accumulated in the same order here,
// from shared memory (sum_shared), so with FMA contraction disabled this path reproduces the CPU
// algorithm operation for operation; the remaining differences come from the
// device exp/log/pow, which agree with the host's to about one ulp.
//
// Algorithm followed (paths relative to solvers/openSMOKEpp4laminarSMOKE):
//   RHS        solvers/laminarSMOKE/unsteady/BatchReactorHomogeneousConstantPressure.H:175-223
//   thermo     maps/ThermodynamicsMap_CHEMKIN.hpp:429-520
//   kinetics   maps/KineticsMap_CHEMKIN.hpp:271-297, 1181-1398, 1496-1550, 1683-1768, 1956-1964
//   stoich.    maps/StoichiometricMap.hpp:512-598, 656-729, 916-1001
//   BDF        math/native-ode-solvers/MultiValueSolver.hpp:367-1328
//   Gear       math/native-ode-solvers/MethodGear.hpp:79-536
//   dense      math/native-ode-solvers/KernelDense.hpp:90-245
#pragma once
#include "lsg_common.cuh"
#include "lsg_kernels.h"

namespace lsg {

// One copy per translation unit; the host uploads it with cudaMemcpyToSymbol.
static __constant__ GearConsts c_gear;

// Dynamic shared memory of the warp kernels: the mechanism (kStaged), then the warps' work spaces.  The out-of-line
// functions below address it from here, so that they load from shared memory and not through generic pointers.
extern __shared__ __align__(16) unsigned char warp_smem[];
__device__ __forceinline__ MechLayout& warp_layout() {
  __shared__ MechLayout l;
  return l;
}
struct MechPlace {   // the tables in global memory, where they do not fit in shared memory
  const unsigned char* gmem;
};
__device__ __forceinline__ MechPlace& warp_mech() {
  __shared__ MechPlace m;
  return m;
}
template <bool kStaged>
__device__ __forceinline__ MechView warp_tables(const MechLayout& L) {
  const unsigned char* base = kStaged ? (const unsigned char*)warp_smem : warp_mech().gmem;
  return MechView{(const double*)base, (const int*)(base + (size_t)(kStaged ? L.base_double : L.n_double) * sizeof(double))};
}

// Per-warp shared-memory workspace (all arrays lane- or index-addressed).
struct WarpWS {
  double* Z;      // [8][32] Nordsieck array z_
  double* V;      // [8][32] v_
  double* J;      // [ld][ld] Jacobian by columns, ld: n rounded up to 4
  double* G;      // [ld][ld] LU factors of G = I - h r0 J, by columns, the rows in pivoted order
  double* C;      // [32] concentrations, [nc] = 1
  double* H;      // [32] h/RT
  double* S;      // [32] s/R
  double* X;      // [3][33] terms of sums; the solve's vector
  double* R;      // [2][32] 1 / pivots and what they lack of it
  double* KARR;   // [NR] forward Arrhenius constants (cache)
  double* UKEQ;   // [NR] 1/Keq (thermo reversible) or k_rev (explicit)
  double* NET;    // [NR] net rates
  double* KINF;   // [NFO] k_inf (cache)
  double* FEXP;   // [NFO][3] exponentials of F_cent
  double* LOGF;   // [NFO] log10 Fcent (Troe) / SRI factor (cache)
  int* PIV;       // [32] row of each pivot
  double* SC;     // [6] scalars: cached kinetic T, QR of the last call, P0, energy flag, rho0 (> 0: constant volume), P0 / R
  unsigned char* DROP;   // [NR] DRG-reduced step only (drg_ws_doubles): 1 for a reaction the analysis dropped
};

__host__ __device__ inline int warp_ld(int n) { return (n + 3) & ~3; }
__host__ __device__ inline int warp_ws_doubles(const MechLayout& L) {
  const int ld = warp_ld(L.nc + 1);
  auto even = [](int x) { return (x + 1) & ~1; };
  return 8 * 32 * 2 + 2 * ld * ld + 32 * 3 + 100 + 64 + even(L.nr) * 3 + even(L.n_fo > 0 ? 5 * L.n_fo : 1) + 16 + 6;
}

// The DRG kernel's per-warp workspace: the above and the dropped-reaction mask after it.
__host__ __device__ inline int drg_ws_doubles(const MechLayout& L) {
  return warp_ws_doubles(L) + (((L.nr + 7) / 8 + 1 + 1) & ~1);
}

__device__ __forceinline__ WarpWS carve_ws(double* base, const MechLayout& L) {
  const int ld = warp_ld(L.nc + 1);
  auto even = [](int x) { return (x + 1) & ~1; };
  WarpWS w;
  double* p = base;
  w.Z = p; p += 8 * 32;
  w.V = p; p += 8 * 32;
  w.J = p; p += ld * ld;
  w.G = p; p += ld * ld;
  w.C = p; p += 32;
  w.H = p; p += 32;
  w.S = p; p += 32;
  w.X = p; p += 100;
  w.R = p; p += 64;
  w.PIV = (int*)p; p += 16;
  w.SC = p; p += 6;
  w.KARR = p; p += even(L.nr);
  w.UKEQ = p; p += even(L.nr);
  w.NET = p; p += even(L.nr);
  w.KINF = p;
  w.LOGF = p + L.n_fo;
  w.FEXP = p + 2 * L.n_fo;
  p += even(L.n_fo > 0 ? 5 * L.n_fo : 1);
  w.DROP = (unsigned char*)p;
  return w;
}

// One copy of each transcendental: with warps on their own ways through the code, instruction fetch is what the
// kernels wait for first, so code size comes first.
__device__ __noinline__ double exp_w(double x) { return exp(x); }
__device__ __noinline__ double log_w(double x) { return log(x); }
__device__ __noinline__ double log10_w(double x) { return log10(x); }
__device__ __noinline__ double pow_w(double x, double y) { return pow(x, y); }
__device__ __noinline__ double div_w(double a, double b) { return a / b; }

// num / den to the last bit, for numerators that are often exactly zero (absent species): the division of a zero
// leaves the fast path, so a zero is multiplied by 1 / den instead, which gives the same zero, NaN or sign.
__device__ __noinline__ double div0(double num, double den) {
  const bool z = num == 0.;
  const double q = (z ? 1. : num) / den;
  return z ? num * q : q;
}

__device__ __forceinline__ double contrib(double nu, double v) {
  if (nu == 1.) return v;
  if (nu == 2.) return v + v;
  if (nu == 3.) return v + v + v;
  if (nu == 0.5) return 0.5 * v;
  return nu * v;
}

__device__ __noinline__ double conc_factor(double nu, double c1) {
  if (nu == 1.) return c1;
  if (nu == 2.) return c1 * c1;
  if (nu == 3.) return c1 * c1 * c1;
  if (nu == 0.5) return sqrt(c1);
  return pow(c1, nu);
}

// p[0] + ... + p[n - 1] from the left; p 16-byte aligned, in shared memory: broadcast loads instead of shuffles
__device__ __forceinline__ double sum_shared(const double* p, int n) {
  double s = 0.;
  int i = 0;
#pragma unroll 1
  for (; i + 4 <= n; i += 4) {
    const double2 a = *(const double2*)(p + i), b = *(const double2*)(p + i + 2);
    s += a.x;
    s += a.y;
    s += b.x;
    s += b.y;
  }
#pragma unroll 1
  for (; i < n; ++i) s += p[i];
  return s;
}
// The lanes' v summed in lane order
__device__ __noinline__ double sum_warp(int x_at, double v, int n) {
  double* const X = (double*)warp_smem + x_at;
  __syncwarp();
  X[threadIdx.x & 31] = v;
  __syncwarp();
  return sum_shared(X, n);
}
// Root mean square of the lanes' c, whose squares are summed in lane order
__device__ __noinline__ double norm_warp(int x_at, double c, int n) {
  double* const X = (double*)warp_smem + x_at;
  __syncwarp();
  X[threadIdx.x & 31] = c * c;
  __syncwarp();
  return sqrt(sum_shared(X, n) / double(n));
}
// Three such sums at once: lane 0 receives a's, lane 1 b's, the others c's.
__device__ __noinline__ double sum3_warp(int x_at, double a, double b, double c, int n) {
  double* const X = (double*)warp_smem + x_at;
  const int lane = threadIdx.x & 31;
  __syncwarp();
  X[lane] = a;
  X[33 + lane] = b;
  X[66 + lane] = c;
  __syncwarp();
  const double* p = X + 33 * (lane < 2 ? lane : 2);
  double s = 0.;
#pragma unroll 4
  for (int i = 0; i < n; ++i) s += p[i];
  return s;
}

// Net rate of a reaction outside the packed form (mech.h bx_pack): any stoichiometry, FORD orders, explicit reverse
// parameters, PLOG, CHEB and the extended forms.
template <bool kStaged>
__device__ __noinline__ double general_rate_warp(int wofs, int j, double cTotSum, double T, double Pk);
template <bool kStaged>
__device__ __noinline__ double equilibrium_arg(int wofs, int j, double lP);

// Fall-off or CABR factor of reaction j's rate constant, slot fo (KineticsMap_CHEMKIN.hpp:1257-1290, 1496-1550,
// 1613-1660): k0 (1 / (1 + Pr)) F; k_inf (Pr / (1 + Pr)) F over kArr.
template <bool kStaged>
__device__ __noinline__ double falloff_warp(int wofs, int fo, double kArr, double cTotSum, double T) {
  const MechLayout& L = warp_layout();
  const MechView M = warp_tables<kStaged>(L);
  const WarpWS W = carve_ws((double*)warp_smem + wofs, L);
  double Mc;
  const int single = M.I(L.fo_single)[fo];
  if (single < 0) {
    Mc = cTotSum;
    const int* fp = M.I(L.fo_ptr);
    const int* fs = M.I(L.fo_sp);
    const double* fe = M.D(L.fo_eff);
#pragma unroll 1
    for (int q2 = fp[fo]; q2 < fp[fo + 1]; ++q2) Mc += W.C[fs[q2]] * fe[q2];
  } else {
    Mc = W.C[single] + 1.e-16;
  }
  const double kInf = W.KINF[fo];
  const double lF = W.LOGF[fo];
  const double Pr = div_w(kArr * Mc, kInf);
  const bool cabr = M.I(L.fo_cabr)[fo] != 0;
  double wF = 1.;
  const int ty = M.I(L.fo_type)[fo];
  if (ty == 1) {
    double qq = 1. / 0.14;
    if (Pr > 1.e-32 || cabr) {
      const double nTroe = 0.75 - 1.27 * lF;
      const double cTroe = -0.4 - 0.67 * lF;
      const double sTroe = log10_w(Pr) + cTroe;
      qq = div_w(sTroe, nTroe - 0.14 * sTroe);
    }
    wF = pow_w(10., div_w(lF, 1. + qq * qq));
  } else if (ty == 2) {
    const double l10 = log10_w(Pr);
    const double xSRI = div_w(1., 1. + l10 * l10);
    wF = pow_w(lF, xSRI) * M.D(L.fo_d)[fo];
    const double e = M.D(L.fo_e)[fo];
    if (e != 0.) wF *= pow_w(T, e);
  }
  const double s = div_w(cabr ? 1. : Pr, 1. + Pr);
  return cabr ? s * wF : div_w(kInf * s * wF, kArr);
}

// ---------------------------------------------------------------------------
// Right-hand side f(y), warp cooperative.  yl: this lane's component.  The cached temperature of the kinetic
// constants (the reference's T_old test), the last QR, P0 and the energy flag live in the work space's scalar
// slots.  One out-of-line body, no code twice: what bounds the kernels is instruction fetch and the latency of a
// warp's dependent chain.  So sums read shared memory in order instead of a shuffle a term, divisions and
// logarithms of scalars run in one go on different lanes, the exponentials of a call are dealt evenly over the
// lanes, and reactions of the common form come packed.
// ---------------------------------------------------------------------------
template <bool kDrg, bool kStaged>
__device__ __noinline__ double rhs_warp(int wofs, double yl, double T) {
  const MechLayout& L = warp_layout();
  const MechView M = warp_tables<kStaged>(L);
  const WarpWS W = carve_ws((double*)warp_smem + wofs, L);
  const bool energy = W.SC[3] != 0.;
  const double rho0 = W.SC[4];   // constant volume when > 0 (BatchReactorHomogeneousConstantVolume.H:148-199)
  const bool cv = rho0 > 0.;
  const int lane = threadIdx.x & 31;
  const int NC = L.nc, NR = L.nr;
  const bool sp = lane < NC;
  const double mwl = sp ? M.D(L.mw)[lane] : 1.;
  // mole fractions, concentrations, density
  const double u = sum_warp(wofs + (int)(W.X - ((double*)warp_smem + wofs)), sp ? div0(yl, mwl) : 0., NC);
  const double num = lane == 1 ? W.SC[5] : lane == 2 ? 101325. / kRgas : 1.;
  const double quo = div_w(num, lane == 3 ? u : T);
  const double uT = __shfl_sync(kFull, quo, 0), MWmix = __shfl_sync(kFull, quo, 3);
  const double Patm_over_RT = __shfl_sync(kFull, quo, 2);
  const double xl = sp ? div0(MWmix * yl, mwl) : 0.;
  double cTot = __shfl_sync(kFull, quo, 1);   // P0 / R / T
  if (cv) cTot = div_w(rho0, MWmix);
  const double cl = cTot * xl;
  const double rho = cv ? rho0 : cTot * MWmix;
  const double T2 = T * T, T3 = T2 * T, T4 = T3 * T;
  const bool high = sp && T > M.D(L.t_mid)[lane];
  double hl = 0.;
  if (sp) {
    const double* A = (high ? M.D(L.dh_ht) : M.D(L.dh_lt)) + 6 * lane;
    hl = A[0] + T * A[1] + T2 * A[2] + T3 * A[3] + T4 * A[4] + uT * A[5];
    W.C[lane] = cl;
    W.H[lane] = hl;
  } else if (lane == NC) {
    W.C[NC] = 1.;   // the packed reactions' absent second species
  }
  const double T_old = W.SC[0];
  const bool recalc = div_w(fabs(T - T_old), T) > 0.;
  const int4* bx = (const int4*)M.I(L.bx_pack);
  if (recalc) {
    const double lg = log_w(lane == 1 ? Patm_over_RT : T);
    const double logT = __shfl_sync(kFull, lg, 0), lP = __shfl_sync(kFull, lg, 1);
    if (sp) {
      const double* A = (high ? M.D(L.ds_ht) : M.D(L.ds_lt)) + 6 * lane;
      W.S[lane] = A[0] * logT + T * A[1] + T2 * A[2] + T3 * A[3] + T4 * A[4] + A[5];
    }
    __syncwarp();
    // one exponential a lane and turn: rate constants, equilibrium constants, k_inf, F_cent's three
    const int nf = L.n_fo, n = 2 * NR + 4 * nf;
#pragma unroll 1
    for (int e = lane; e - lane < n; e += 32) {
      double arg = 0.;
      double* to = nullptr;
      bool neg = false;
      if (e < NR) {
        arg = M.D(L.lnA)[e] + M.D(L.beta)[e] * logT - M.D(L.eor)[e] * uT;
        neg = M.I(L.a_sign)[e] < 0;
        to = W.KARR + e;
      } else if (e < 2 * NR) {
        const int j = e - NR, kind = M.I(L.rev_kind)[j];
        if (kind == 1) {
          to = W.UKEQ + j;
          if (bx[j].z & kRxSpecial) {
            arg = equilibrium_arg<kStaged>(wofs, j, lP);
          } else {
            // StoichiometricMap::ReactionEnthalpyAndEntropy: species order, reactant first; the coefficients are
            // +-1 and +-2, so the products are exact and the fused operations round as sums
            const int4 m = ((const int4*)M.I(L.bx_merge))[j];
            double dh = 0., ds = 0.;
            auto add = [&](int q) {
              const double c = __hiloint2double(q & ~0xffff, 0);
              dh = __fma_rn(c, W.H[q & 0xffff], dh);
              ds = __fma_rn(c, W.S[q & 0xffff], ds);
            };
            add(m.x);
            add(m.y);
            add(m.z);
            add(m.w);
            if (bx[j].z & kRxLong) {
              const int4 o = ((const int4*)M.I(L.bx_more))[j];
              add(o.x);
              add(o.y);
            }
            arg = -ds + dh - lP * M.D(L.dnu)[j];
          }
        } else if (kind == 2) {
          const int s = M.I(L.rev_slot)[j];
          to = W.UKEQ + j;
          arg = M.D(L.rev_lnA)[s] + M.D(L.rev_beta)[s] * logT - M.D(L.rev_eor)[s] * uT;
        }
      } else if (e < 2 * NR + nf) {
        const int k = e - 2 * NR;
        to = W.KINF + k;
        arg = M.D(L.fo_lnA)[k] + M.D(L.fo_beta)[k] * logT - M.D(L.fo_eor)[k] * uT;
      } else if (e < n) {
        const int q = e - 2 * NR - nf, k = q / 3, c = q - 3 * k, ty = M.I(L.fo_type)[k];
        to = W.FEXP + q;
        // Troe: -T / b, -T / c, -d / T; SRI: -b / T, -T / c
        const double v = M.D(c == 0 ? L.fo_b : c == 1 ? L.fo_c : L.fo_d)[k];
        const bool over = ty == 2 ? c == 0 : c == 2;
        if (ty == 1 || (ty == 2 && c < 2)) arg = div_w(over ? -v : -T, over ? T : v);
      }
      const double x = exp_w(arg);
      if (to) *to = neg ? x * -1. : x;
    }
    __syncwarp();
#pragma unroll 1
    for (int k = lane; k < nf; k += 32) {
      const int ty = M.I(L.fo_type)[k];
      const double a = M.D(L.fo_a)[k], d = M.D(L.fo_d)[k];
      const double* E = W.FEXP + 3 * k;
      double lf = 0.;
      if (ty == 1) {
        double v = (1. - a) * E[0] + a * E[1];
        if (d != 0.) v += E[2];
        lf = (v < 1.e-300) ? -300. : log10_w(v);
      } else if (ty == 2) {
        lf = a * E[0] + E[1];
      }
      W.LOGF[k] = lf;
    }
  }
  const double Pk = cv ? cTot * kRgas * T : W.SC[2];
  __syncwarp();
  if (lane == 0) W.SC[0] = T;
  if (L.n_plog > 0 || L.n_cheb > 0) {
    // pressure-logarithmic and Chebyshev reactions: k depends on P too, so every call
    // (KineticsMap_CHEMKIN.hpp:1332-1348)
    const double logTk = log_w(T);
    const int* prx = M.I(L.plog_rxn);
#pragma unroll 1
    for (int k = lane; k < L.n_plog; k += 32) W.KARR[prx[k]] = plog_k(M, L, k, T, logTk, Pk);
    const int* crx = M.I(L.cheb_rxn);
#pragma unroll 1
    for (int k = lane; k < L.n_cheb; k += 32) W.KARR[crx[k]] = cheb_k(M, L, k, T, Pk);
    __syncwarp();
  }
  const double cTotSum = sum_shared(W.C, NC);
  {
    // fall-off reactions first, then special forms and third bodies: the lanes of a warp mostly share a path
    const int* ord = M.I(L.bx_order);
#pragma unroll 1
    for (int e = lane; e < NR; e += 32) {
      const int j = ord[e];
      const int4 r = bx[j];
      double net;
      if (r.z & kRxSpecial) {
        net = general_rate_warp<kStaged>(wofs, j, cTotSum, T, Pk);
      } else {
        const double kArr = W.KARR[j];
        double kMod = kArr;
        const int tb = M.I(L.tb_slot)[j], fo = M.I(L.fo_slot)[j];
        if (tb >= 0) {
          double Mc = cTotSum;
          const int* tp = M.I(L.tb_ptr);
          const int* ts = M.I(L.tb_sp);
          const double* te = M.D(L.tb_eff);
#pragma unroll 1
          for (int q2 = tp[tb]; q2 < tp[tb + 1]; ++q2) Mc += W.C[ts[q2]] * te[q2];
          kMod *= Mc;
        }
        if (fo >= 0) kMod *= falloff_warp<kStaged>(wofs, fo, kArr, cTotSum, T);
        net = W.C[r.x & 0xffff] * W.C[r.x >> 16];
        if (r.z & kRxLong) net *= W.C[r.w & 0xffff];
        if (r.z & kRxReversible) {
          double rv = W.C[r.y & 0xffff] * W.C[r.y >> 16];
          if (r.z & kRxLong) rv *= W.C[r.w >> 16];
          rv *= W.UKEQ[j];
          net -= rv;
        }
        net *= kMod;
      }
      if constexpr (kDrg) {
        if (W.DROP[j]) net = 0.;   // DRG-reduced system: dropped reactions (chemistry_DRG.H)
      }
      W.NET[j] = net;
    }
  }
  __syncwarp();
  double Rl = 0.;
  if (sp) {
    const int* fp = M.I(L.fr_ptr);
    if (L.fe_len > 0) {   // coefficients +-1 and +-2: exact products
      const int2* fe = (const int2*)M.I(L.fe_ent) + lane;
      const int len = fp[lane + 1] - fp[lane];
#pragma unroll 4
      for (int q2 = 0; q2 < len; ++q2) {
        const int2 e = fe[q2 * NC];
        Rl = __fma_rn(__hiloint2double(e.y, 0), W.NET[e.x], Rl);
      }
    } else {
      const int* fr = M.I(L.fr_rxn);
      const double* fc = M.D(L.fr_coef);
#pragma unroll 1
      for (int q2 = fp[lane]; q2 < fp[lane + 1]; ++q2) {
        const double c = fc[q2];
        Rl += contrib(c < 0. ? -c : c, W.NET[fr[q2]]) * (c < 0. ? -1. : 1.);
      }
    }
  }
  double dyl = sp ? div0(mwl * Rl, rho) : 0.;
  double QR = W.SC[1];
  if (energy) {
    double cpl = 0.;
    if (sp) {
      const double* A = (high ? M.D(L.cp_ht) : M.D(L.cp_lt)) + 5 * lane;
      cpl = A[0] + T * A[1] + T2 * A[2] + T3 * A[3] + T4 * A[4];
    }
    const double s3 = sum3_warp(wofs + (int)(W.X - ((double*)warp_smem + wofs)), cpl * xl, Rl * hl, Rl, NC);
    const double cpm = __shfl_sync(kFull, s3, 0) * kRgas;
    const double d = __shfl_sync(kFull, s3, 1);
    QR = -d * kRgas * T;
    if (cv) {
      const double CvMixMass = div_w(cpm - kRgas, MWmix);
      const double sumR = __shfl_sync(kFull, s3, 2);
      if (lane == NC) dyl = div_w(QR + kRgas * T * sumR, rho0 * CvMixMass);
    } else {
      const double CpMixMass = div_w(cpm, MWmix);
      if (lane == NC) dyl = div_w(QR, rho * CpMixMass);
    }
  }
  __syncwarp();
  if (lane == 0) W.SC[1] = QR;
  __syncwarp();
  return dyl;
}

// -ds + dh - lP dnu of any stoichiometry (StoichiometricMap::ReactionEnthalpyAndEntropy: species order, reactant first)
template <bool kStaged>
__device__ __noinline__ double equilibrium_arg(int wofs, int j, double lP) {
  const MechLayout& L = warp_layout();
  const MechView M = warp_tables<kStaged>(L);
  const WarpWS W = carve_ws((double*)warp_smem + wofs, L);
  const int* rsp = M.I(L.reac_sp);
  const double* rnu = M.D(L.reac_nu);
  const int* psp = M.I(L.prod_sp);
  const double* pnu = M.D(L.prod_nu);
  double dh = 0., ds = 0.;
  int a = M.I(L.reac_ptr)[j], b = M.I(L.prod_ptr)[j];
  const int ae = M.I(L.reac_ptr)[j + 1], be = M.I(L.prod_ptr)[j + 1];
  while (a < ae || b < be) {
    const int sa = a < ae ? rsp[a] : (1 << 30);
    const int sb = b < be ? psp[b] : (1 << 30);
    if (sa <= sb) {
      dh -= contrib(rnu[a], W.H[sa]);
      ds -= contrib(rnu[a], W.S[sa]);
      ++a;
    } else {
      dh += contrib(pnu[b], W.H[sb]);
      ds += contrib(pnu[b], W.S[sb]);
      ++b;
    }
  }
  return -ds + dh - lP * M.D(L.dnu)[j];
}

template <bool kStaged>
__device__ __noinline__ double general_rate_warp(int wofs, int j, double cTotSum, double T, double Pk) {
  const MechLayout& L = warp_layout();
  const MechView M = warp_tables<kStaged>(L);
  const WarpWS W = carve_ws((double*)warp_smem + wofs, L);
  double kArr = W.KARR[j];
  if (L.n_xplog > 0) {   // extended PLOG, every call: k depends on the concentrations (KineticsMap_CHEMKIN.hpp:1662-1670)
    const int xs = M.I(L.xplog_slot)[j];
    if (xs >= 0) kArr = xplog_k(M, L, xs, T, log(T), Pk, cTotSum, [&](int k) { return W.C[k]; });
  }
  double kMod = kArr;
  const int tb = M.I(L.tb_slot)[j];
  if (tb >= 0) {
    double Mc = cTotSum;
    const int* tp = M.I(L.tb_ptr);
    const int* ts = M.I(L.tb_sp);
    const double* te = M.D(L.tb_eff);
#pragma unroll 1
    for (int q2 = tp[tb]; q2 < tp[tb + 1]; ++q2) Mc += W.C[ts[q2]] * te[q2];
    kMod *= Mc;
  }
  const int fo = M.I(L.fo_slot)[j];
  if (fo >= 0) kMod *= falloff_warp<kStaged>(wofs, fo, kArr, cTotSum, T);
  if (L.n_xfo > 0) {     // extended fall-off (KineticsMap_CHEMKIN.hpp:1672-1681)
    const int xs = M.I(L.xfo_slot)[j];
    if (xs >= 0) {
      kArr = xfo_k(M, L, xs, T, cTotSum, [&](int k) { return W.C[k]; });
      kMod = kArr;
    }
  }
  const int* op = M.I(L.ford_ptr);     // forward rate-law orders (FORD, else the coefficients)
  const int* osp = M.I(L.ford_sp);
  const double* onu = M.D(L.ford_val);
  double net = 1.;
#pragma unroll 1
  for (int q2 = op[j]; q2 < op[j + 1]; ++q2) net *= conc_factor(onu[q2], W.C[osp[q2]]);
  const int kind = M.I(L.rev_kind)[j];
  if (kind != 0) {
    const int* pp = M.I(L.prod_ptr);
    const int* psp = M.I(L.prod_sp);
    const double* pnu = M.D(L.prod_nu);
    double rv = 1.;
#pragma unroll 1
    for (int q2 = pp[j]; q2 < pp[j + 1]; ++q2) rv *= conc_factor(pnu[q2], W.C[psp[q2]]);
    if (kind == 1) rv *= W.UKEQ[j];
    else rv *= W.UKEQ[j] / kArr;
    net -= rv;
  }
  return net * kMod;
}

// G = I - hr0 J; partial-pivot LU (largest magnitude, first occurrence), the factors' rows in pivoted order and the
// pivots' reciprocals.  A row a lane; up to 16 rows the half warps share the columns.  Rows stay where they are
// until the end (pos: their place in the pivoted order, which decides ties).  Returns whether every pivot is far
// from overflow and underflow (solve_warp).
__device__ __noinline__ bool factorize_warp(int wofs, int n, double hr0) {
  const WarpWS W = carve_ws((double*)warp_smem + wofs, warp_layout());
  const int lane = threadIdx.x & 31, ld = warp_ld(n);
  const bool two = n <= 16;
  const int r = two ? lane & 15 : lane, c0 = two ? lane >> 4 : 0, cs = two ? 2 : 1;
  double* const G = W.G + r;
  __syncwarp();
#pragma unroll 1
  for (int j = c0; j < ld; j += cs) {
    if (r < ld) {
      double g = r == j ? 1. : 0.;
      if (r < n && j < n) {
        g = W.J[j * ld + r] * -hr0;
        if (r == j) g += 1.;
      }
      G[j * ld] = g;
    }
  }
  __syncwarp();
  int pos = r;
  bool done = r >= n;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const double p = done ? 0. : G[k * ld];
    const unsigned hi = done ? 0u : ((unsigned)__double2hiint(p) & 0x7fffffffu) + 1u;
    const unsigned mh = __reduce_max_sync(kFull, hi);
    unsigned cd = __ballot_sync(kFull, hi == mh && lane == r);
    if (cd & (cd - 1u)) {   // the same high word: the low word decides, then the first place
      const unsigned lo = (unsigned)__double2loint(p);
      const unsigned ml = __reduce_max_sync(kFull, hi == mh ? lo : 0u);
      const bool eq = hi == mh && lo == ml;
      const int pm = __reduce_min_sync(kFull, eq ? pos : 64);
      cd = __ballot_sync(kFull, eq && pos == pm && lane == r);
    }
    const int pr = __ffs(cd) - 1;
    const double d = __shfl_sync(kFull, p, pr);
    const int at = __shfl_sync(kFull, pos, pr);
    if (lane == 0) W.PIV[k] = pr;
    if (!done && pos == k) pos = at;
    if (r == pr) {
      pos = k;
      done = true;
    }
    double l = p;
    if (d != 0.) l = div0(p, d);
    if (!done) {
      G[k * ld] = l;
      const double* u = W.G + pr;
      int j = k + 1;
      if (two && (j & 1) != c0) ++j;
#pragma unroll 1
      for (; j + 3 * cs < n; j += 4 * cs) {
        double g[4], v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          g[q] = G[(j + q * cs) * ld];
          v[q] = u[(j + q * cs) * ld];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) G[(j + q * cs) * ld] = g[q] - l * v[q];
      }
#pragma unroll 1
      for (; j < n; j += cs) G[j * ld] -= l * u[j * ld];
    }
    __syncwarp();
  }
  const int row = r < n ? W.PIV[r] : r;
#pragma unroll 1
  for (int j = c0; j - c0 < n; j += 4 * cs) {
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (j + q * cs < n && r < n) v[q] = W.G[(j + q * cs) * ld + row];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (j + q * cs < n && r < n) G[(j + q * cs) * ld] = v[q];
    __syncwarp();
  }
  double rd = 1., rl = 0.;
  bool far = true;
  if (lane < n) {
    const double d = W.G[lane * ld + lane], m = fabs(d);
    rd = div_w(1., d);
    rl = __fma_rn(-d, rd, 1.) * rd;
    far = m > 1.e-100 && m < 1.e100;
  }
  W.R[lane] = rd;
  W.R[32 + lane] = rl;
  far = __all_sync(kFull, far);
  __syncwarp();
  return far;
}

// x / d.  By 1 / d = r + rl (r rounded to nearest, rl the rest) the first estimate is within one unit in the last
// place, so the correction by the exact remainder gives the division's own value (Markstein, IBM J. Res. Dev. 34,
// 1990) as long as nothing comes near underflow or overflow, which solve_warp checks afterwards.
__device__ __forceinline__ double quotient_warp(bool recip, double x, double d, double r, double rl) {
  if (!recip) return div_w(x, d);
  const double q = __fma_rn(x, r, x * rl);
  return __fma_rn(__fma_rn(-q, d, x), r, q);
}

// KernelDense::SolveLinearSystem: the substitutions, lane = row.  Four columns at a time: their rows' values are
// broadcast, every lane solves the 4 x 4 triangle for itself and applies the four columns in order; rows whose unknown
// is out already go on being updated, which is harmless: the unknowns are kept in X.
__device__ __noinline__ double substitute_warp(int wofs, int n, bool recip, double x) {
  const WarpWS W = carve_ws((double*)warp_smem + wofs, warp_layout());
  const int lane = threadIdx.x & 31, ld = warp_ld(n);
  const double* const G = W.G;
#pragma unroll 1
  for (int k = 0; k < ld; k += 4) {
    const double* Gk = G + k * ld;
    double v0 = __shfl_sync(kFull, x, k), v1 = __shfl_sync(kFull, x, k + 1), v2 = __shfl_sync(kFull, x, k + 2),
           v3 = __shfl_sync(kFull, x, k + 3);
    const double2 a = *(const double2*)(Gk + k), b = *(const double2*)(Gk + k + 2);
    const double2 c = *(const double2*)(Gk + ld + k + 2), d = *(const double2*)(Gk + 2 * ld + k + 2);
    v1 -= a.y * v0;
    v2 -= b.x * v0;
    v3 -= b.y * v0;
    x -= Gk[lane] * v0;
    v2 -= c.x * v1;
    v3 -= c.y * v1;
    x -= Gk[ld + lane] * v1;
    v3 -= d.y * v2;
    x -= Gk[2 * ld + lane] * v2;
    x -= Gk[3 * ld + lane] * v3;
    if (lane == 0) {
      *(double2*)(W.X + k) = make_double2(v0, v1);
      *(double2*)(W.X + k + 2) = make_double2(v2, v3);
    }
  }
  __syncwarp();
  x = W.X[lane];
  __syncwarp();
#pragma unroll 1
  for (int k = ld - 4; k >= 0; k -= 4) {
    const double* Gk = G + k * ld;
    double v0 = __shfl_sync(kFull, x, k), v1 = __shfl_sync(kFull, x, k + 1), v2 = __shfl_sync(kFull, x, k + 2),
           v3 = __shfl_sync(kFull, x, k + 3);
    const double2 a = *(const double2*)(Gk + 3 * ld + k), b = *(const double2*)(Gk + 3 * ld + k + 2);
    const double2 c = *(const double2*)(Gk + 2 * ld + k), d = *(const double2*)(Gk + 2 * ld + k + 2);
    const double2 e = *(const double2*)(Gk + ld + k);
    const double2 r0 = *(const double2*)(W.R + k), r1 = *(const double2*)(W.R + k + 2);
    const double2 s0 = *(const double2*)(W.R + 32 + k), s1 = *(const double2*)(W.R + 32 + k + 2);
    v3 = quotient_warp(recip, v3, b.y, r1.y, s1.y);
    v2 -= b.x * v3;
    v1 -= a.y * v3;
    v0 -= a.x * v3;
    x -= Gk[3 * ld + lane] * v3;
    v2 = quotient_warp(recip, v2, d.x, r1.x, s1.x);
    v1 -= c.y * v2;
    v0 -= c.x * v2;
    x -= Gk[2 * ld + lane] * v2;
    v1 = quotient_warp(recip, v1, e.y, r0.y, s0.y);
    v0 -= e.x * v1;
    x -= Gk[ld + lane] * v1;
    v0 = quotient_warp(recip, v0, Gk[k], r0.x, s0.x);
    x -= Gk[lane] * v0;
    if (lane == 0) {
      *(double2*)(W.X + k) = make_double2(v0, v1);
      *(double2*)(W.X + k + 2) = make_double2(v2, v3);
    }
  }
  __syncwarp();
  return W.X[lane];
}
__device__ __noinline__ double solve_warp(int wofs, int n, bool recip, double xl) {
  const WarpWS W = carve_ws((double*)warp_smem + wofs, warp_layout());
  const int lane = threadIdx.x & 31;
  double x = __shfl_sync(kFull, xl, lane < n ? W.PIV[lane] : 0);
  if (lane >= n) x = 0.;
  __syncwarp();
  double y = substitute_warp(wofs, n, recip, x);
  // the quotients are exact if neither they nor the products behind them left the range
  const double m = lane < n ? fabs(y) : 0.;
  if (recip && !__all_sync(kFull, m == 0. || (m > 1.e-160 && m < 1.e160))) y = substitute_warp(wofs, n, false, x);
  return lane < n ? y : 0.;
}

// (J v)_lane, columns in order
__device__ __noinline__ double jacobian_times_warp(int wofs, int n, double v) {
  const WarpWS W = carve_ws((double*)warp_smem + wofs, warp_layout());
  const int lane = threadIdx.x & 31, ld = warp_ld(n);
  __syncwarp();
  W.X[lane] = v;
  __syncwarp();
  double s = 0.;
#pragma unroll 4
  for (int j = 0; j < n; ++j) s += W.J[j * ld + lane] * W.X[j];
  return s;
}

// ---------------------------------------------------------------------------
// Gear / multivalue BDF integrator state for one warp (one cell).  Vectors are
// held one component per lane (registers) or in the per-warp shared arrays.
// ---------------------------------------------------------------------------
// kDrg: the DRG-reduced system (chemistry_DRG.H) instead of the full reactor.
template <bool kDrg, bool kStaged>
struct GearWarpT {
  static constexpr int MAX_ORDER = 5, MIN_ORDER = 1;
  enum { H_DEC, H_CONST, H_INC };
  enum { O_DEC, O_CONST, O_INC };
  enum { JAC_CHANGE, JAC_MODIFIED };
  enum { M_TO_FACT, M_FACT };
  enum { CONV_FAIL, CONV_OK };

  WarpWS W;
  int wofs;           // the work space in the dynamic shared memory, in doubles
  int lane, ne;
  bool active;        // lane < ne
  // per-lane vector components
  double b, deltab, f, va, vb, y, y0, eps, minv, maxv;
  // scalar state (replicated in all lanes)
  double alfa2_4, alfa2_5;   // alfa2[4], alfa2[5]; alfa2[0..3] stay 0.8
  __device__ __forceinline__ double alfa2(unsigned k) const { return k == 4 ? alfa2_4 : (k == 5 ? alfa2_5 : .8); }
  double abs_tol, rel_tol;
  unsigned maximum_order, max_number_steps;
  double t, t0, tOut, tInMeshPoint, tStabilize;
  double hPreviousStep, hNordsieck, hScaleMax, h, hNextStep, hScale;
  bool fixedOrderMin;
  unsigned iterConstSteps, iterMinimumOrder;
  unsigned p, iterOrder, orderInNextStep, maxConvergenceIterations, maxIterationsJacobian;
  int odeHStatus, odeOrderStatus, status, factorizationStatus, jacobianStatus, convergenceStatus;
  unsigned numberOfSteps, iterConvergence, iterConvergenceRate, iterConvergenceFailure, iterErrorFailure;
  unsigned numberOfConvergenceFailuresForOrderMax, stepOfLastJacobian;
  unsigned cnt[NCNT];
  bool recip;         // factorize_warp's result
  // DRG-reduced system (BatchReactorHomogeneousConstantPressure.H:253-320): lane l < drg_ni owns species
  // drg_sp (the l-th important one), lane drg_ni owns T; as a lane of the full layout (species `lane`),
  // drg_pos is that species' reduced index or -1, drg_omega its fixed mass fraction.
  bool unconstrained = false;   // no minimum/maximum constraints: KernelDense's unconstrained increments
  int drg_ni = 0, drg_sp = 0, drg_pos = -1, drg_nc = 0;
  double drg_omega = 0.;

  __device__ __forceinline__ int x_at() const { return (int)(W.X - (double*)warp_smem); }
  __device__ __forceinline__ double& Z(int i) { return W.Z[i * 32 + lane]; }
  __device__ __forceinline__ double& V(int i) { return W.V[i * 32 + lane]; }

  // f(y) of the system being integrated: the full reactor, or the DRG-reduced one evaluated through the
  // full layout (kept species fixed, dropped reactions at zero rate) and gathered back to the reduced lanes
  __device__ __forceinline__ double eval(double yl) {
    if constexpr (!kDrg) {
      return rhs_warp<false, kStaged>(wofs, yl, __shfl_sync(kFull, yl, ne - 1));
    } else {
      const double T = __shfl_sync(kFull, yl, drg_ni);
      const double v = __shfl_sync(kFull, yl, drg_pos >= 0 ? drg_pos : 0);
      const double yf = lane < drg_nc ? (drg_pos >= 0 ? v : drg_omega) : T;
      const double df = rhs_warp<true, kStaged>(wofs, yf, T);
      return __shfl_sync(kFull, df, drg_sp);
    }
  }

  __device__ __forceinline__ double rhs(double yl) {
    ++cnt[CNT_RHS];
    return eval(yl);
  }

  __device__ __forceinline__ double error_control(double w, double e) {   // OpenSMOKEUtilities.hpp:689-701
    const double c = active ? w * e : 0.;
    return norm_warp(x_at(), c, ne);
  }

  __device__ __forceinline__ void check_constraints(double& yl) {
    if (active) {
      if (yl < minv) yl = minv;
      if (yl > maxv) yl = maxv;
    }
  }

  __device__ __forceinline__ void one_over_epsilon(double w) {
    if (active) {
      eps = abs_tol + rel_tol * fabs(w);
      eps = div_w(1., eps);
    }
  }

  // KernelDense::NumericalJacobian, constrained branch (max constraints are on)
  __device__ __forceinline__ void numerical_jacobian(double& yl, double fl) {
    const double ZERO_DER = sqrt(kTinyFloat);
    const double ETA2 = sqrt(kMachEpsDouble);
    const double BETA = 1.e+3 * kMachEpsDouble;
    double hf = BETA * fabs(h) * error_control(fl, eps) * double(ne);
    if (hf < 1.e-10) hf = 1.;
    const int n = ne, ld = warp_ld(n);
    // every lane its own component's increment
    const double ie = div_w(1., eps), he = div_w(hf, eps);
    double hJ;
    if (kDrg && unconstrained) {   // KernelDense.hpp:111-193 without maximum constraints
      hJ = ETA2 * fabs(fmax(yl, ie));
      hJ = fmax(hJ, he);
      hJ = fmax(hJ, ZERO_DER);
      hJ = fmin(hJ, 0.001 + 0.001 * fabs(yl));
    } else {
      const double a = fabs(yl), bb = fabs(ie);
      hJ = ETA2 * (a > bb ? a : bb);
      hJ = fmax(hJ, he);
      hJ = fmax(hJ, ZERO_DER);
      if (yl + hJ > maxv) hJ = -hJ;
    }
    const double hInv = div_w(1., hJ);
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
      const double aux = eval(lane == j ? yl + hJ : yl);
      const double hi = __shfl_sync(kFull, hInv, j);
      if (active) W.J[j * ld + lane] = hi * (aux - fl);
    }
    cnt[CNT_JAC_RHS] += (unsigned)n;
    __syncwarp();
  }

  __device__ __forceinline__ void build_and_factorize(double hr0) {
    recip = factorize_warp(wofs, ne, hr0);
    ++cnt[CNT_FACT];
  }

  __device__ __forceinline__ void solve(double& xl) {
    xl = solve_warp(wofs, ne, recip, xl);
    ++cnt[CNT_SOLVE];
  }

  __device__ __forceinline__ void set_initial_conditions(double tstart, double y0l) {
    tOut = t = t0 = tInMeshPoint = tStabilize = tstart;
    p = 1; iterOrder = 0; orderInNextStep = 1; maxConvergenceIterations = 4;
    maxIterationsJacobian = 20 + 5 * (unsigned)(ne - 3);
    if (maxIterationsJacobian > 50u && ne < 80) maxIterationsJacobian = 50u;
    odeHStatus = H_CONST; odeOrderStatus = O_CONST; status = 1;
    factorizationStatus = M_TO_FACT; jacobianStatus = JAC_CHANGE; convergenceStatus = CONV_OK;
    h = 0.; hNextStep = 0.; hScale = 0.;
    numberOfSteps = 0; numberOfConvergenceFailuresForOrderMax = 0;
    iterConvergence = 0; iterConvergenceRate = 0; iterConvergenceFailure = 0; iterErrorFailure = 0;
    stepOfLastJacobian = 0;
    y0 = y0l;
    hPreviousStep = 0.; hNordsieck = 0.; hScaleMax = 1000.;
    fixedOrderMin = false; iterConstSteps = 0; iterMinimumOrder = 0;
    for (int k = 0; k < NCNT; ++k) cnt[k] = 0;
    f = rhs(y0);
  }

  __device__ __forceinline__ unsigned find_correction() {
    vb = active ? V(0) : 0.;
    check_constraints(vb);
    f = rhs(vb);
    if (numberOfSteps >= stepOfLastJacobian + maxIterationsJacobian) jacobianStatus = JAC_CHANGE;
    if (jacobianStatus == JAC_CHANGE) {
      stepOfLastJacobian = numberOfSteps;
      jacobianStatus = JAC_MODIFIED;
      numerical_jacobian(vb, f);
      ++cnt[CNT_JAC];
      factorizationStatus = M_TO_FACT;
    }
    const double r0 = c_gear.r[0][p - 1];
    const double hr0 = h * r0;
    if (factorizationStatus == M_FACT && iterOrder == 0) factorizationStatus = M_TO_FACT;
    if (factorizationStatus == M_TO_FACT) {
      build_and_factorize(hr0);
      factorizationStatus = M_FACT;
    }
    deltab = f * h;
    deltab -= active ? V(1) : 0.;
    solve(deltab);
    b = deltab;
    double oldCC = 0.;
#pragma unroll 1
    for (unsigned k = 1; k <= maxConvergenceIterations; ++k) {
      const double cc = r0 * error_control(deltab, eps);
      if (cc < 1.) { convergenceStatus = CONV_OK; return k; }
      if (k > 1 && cc > 2. * oldCC) { convergenceStatus = CONV_FAIL; return k; }
      oldCC = cc;
      va = b * r0;
      va += active ? V(0) : 0.;
      if (active) {
        if (va < minv) { va = minv; b = div_w(minv - Z(0), r0); }
        if (va > maxv) { va = maxv; b = div_w(maxv - Z(0), r0); }
      }
      f = rhs(va);
      deltab = f * h;
      deltab -= active ? V(1) : 0.;
      deltab -= b;
      solve(deltab);
      b += deltab;
    }
    convergenceStatus = CONV_FAIL;
    return maxConvergenceIterations;
  }

  __device__ __forceinline__ void convergence_failure_recovery() {
    hScale = 0.25;
    if (numberOfSteps < 10) hScale = 0.1;
    hScale = fmax(hScale, div_w(0., fabs(h)));
    odeHStatus = H_DEC;
    if (p > (unsigned)MIN_ORDER) { p -= 1; odeOrderStatus = O_DEC; }
    alfa2_4 -= 0.01;
    alfa2_5 -= 0.02;
    if (alfa2_4 < 0.) { alfa2_4 = 0.; maximum_order = 3; if (p > 3) { p = 3; odeOrderStatus = O_DEC; } }
    if (alfa2_5 < 0.) { alfa2_5 = 0.; maximum_order = 4; if (p > 4) { p = 4; odeOrderStatus = O_DEC; } }
    if (numberOfSteps > 5) {
      numberOfConvergenceFailuresForOrderMax++;
      if (numberOfConvergenceFailuresForOrderMax % 5 == 0) {
        if (p != (unsigned)MIN_ORDER) { p = MIN_ORDER; odeOrderStatus = O_DEC; }
      }
      if (numberOfConvergenceFailuresForOrderMax % 10 == 0 && tStabilize != tInMeshPoint) {
        va = rhs(active ? Z(0) : 0.);
        if (active) Z(1) = va * h;
        tStabilize = tInMeshPoint;
      }
    }
    if (numberOfSteps > stepOfLastJacobian + 5u) jacobianStatus = JAC_CHANGE;
    if (numberOfSteps != stepOfLastJacobian && iterConvergenceFailure == 50u) jacobianStatus = JAC_CHANGE;
    hNextStep *= hScale;
  }

  __device__ __forceinline__ void convergence_rate() {
    if (iterErrorFailure > 0 || iterConvergenceFailure > 0) iterConvergenceRate = 0;
    if (iterConvergence <= 1) return;
    vb = active ? V(0) - Z(0) : 0.;
    const double s = jacobian_times_warp(wofs, ne, vb);
    va = active ? s : 0.;
    va *= h;
    va += active ? Z(1) : 0.;
    va = (active ? V(1) : 0.) - va;
    const double s2 = sum3_warp(x_at(), active ? fabs(va) : 0., active ? fabs(V(1)) : 0., 0., ne);
    const double normd = __shfl_sync(kFull, s2, 0), normf = __shfl_sync(kFull, s2, 1);
    if (normd > 3. * normf + .1 && iterConvergence > 2) {
      if (numberOfSteps > stepOfLastJacobian + 5u) jacobianStatus = JAC_CHANGE;
      hScale = 0.5; odeHStatus = H_DEC; hNextStep = h * hScale;
      if (p > 1) { orderInNextStep = p - 1; odeOrderStatus = O_DEC; }
      iterConvergenceRate = 0; iterConvergenceFailure = 1;
      return;
    }
    if (normd > normf + 0.1) {
      iterConvergenceRate++;
      if (iterConvergenceRate >= 5) {
        hScale = 0.8; odeHStatus = H_DEC; hNextStep = h * hScale;
        iterConvergenceRate = 0; iterConvergenceFailure = 1;
      }
      if (numberOfSteps > stepOfLastJacobian + 5u && iterConvergence > 2) {
        jacobianStatus = JAC_CHANGE;
        iterConvergenceRate = 0; iterConvergenceFailure = 1;
      }
    }
  }

  __device__ __forceinline__ void multi_value_step() {
    if (active) {
      // the prediction v = D z in registers; the rows above p are zero, so the whole triangle may run
      double w[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) w[i] = i <= (int)p ? Z(i) : 0.;
      const double z0 = w[0];
#pragma unroll
      for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = 4; j >= i; --j) w[j] += w[j + 1];
      if (w[0] < minv && fabs(w[0] - minv) * eps < double(ne)) {
        w[0] = minv;
        w[1] = minv - z0;
#pragma unroll
        for (int i = 2; i < 6; ++i) w[i] = 0.;
      }
      if (w[0] > maxv && fabs(w[0] - maxv) * eps < double(ne)) {
        w[0] = maxv;
        w[1] = maxv - z0;
#pragma unroll
        for (int i = 2; i < 6; ++i) w[i] = 0.;
      }
#pragma unroll
      for (int i = 0; i < 6; ++i)
        if (i <= (int)p) V(i) = w[i];
    }
    __syncwarp();
    iterConvergence = find_correction();
    if (convergenceStatus == CONV_FAIL) return;
    const double r0 = c_gear.r[0][p - 1];
    if (active) {
      va = b * r0;
      if (V(0) + va < minv) {
        b = minv - Z(0) - V(1);
        V(0) = minv - va;
        if (V(0) < minv) V(0) = minv;
      }
      if (V(0) + va > maxv) {
        b = maxv - Z(0) - V(1);
        V(0) = maxv - va;
        if (V(0) > maxv) V(0) = maxv;
      }
      V(0) += va;
      V(1) += b;
#pragma unroll 1
      for (unsigned i = 2; i <= p; ++i) {
        va = b * c_gear.r[i][p - 1];
        V(i) += va;
      }
      va = V(p) - Z(p);
      V(p + 1) = div0(va, double(p) + 1.);
      if (iterOrder >= p) {
        va = V(p + 1) - Z(p + 1);
        V(p + 2) = div0(va, double(p) + 2.);
      }
    }
    __syncwarp();
  }

  __device__ __forceinline__ void new_order_new_h() {
    // candidates for p - 1, p, p + 1: their norms in one go, their powers on three lanes
    double hMinus = 0., hPlus = 0., alfa1 = 0., alfa3 = 0.;
    const bool lower = p > (unsigned)MIN_ORDER && odeOrderStatus != O_INC;
    const bool higher = p < maximum_order && odeOrderStatus != O_DEC;
    const double c0 = active ? V(p) * eps : 0., c1 = active ? V(p + 1) * eps : 0.;
    const double c2 = active && higher ? V(p + 2) * eps : 0.;
    const double s3 = sum3_warp(x_at(), c0 * c0, c1 * c1, c2 * c2, ne);
    const unsigned k = lane < 2 ? lane : 2, po = p - 1 + k;
    double hq = c_gear.Ep[po < 6u ? po : 5u] * sqrt(s3 / double(ne)) + kMachEpsFloat;
    hq = pow_w(div_w(1., hq), div_w(1., double(p + k)));
    const double q0 = __shfl_sync(kFull, hq, 0), q1 = __shfl_sync(kFull, hq, 1), q2 = __shfl_sync(kFull, hq, 2);
    if (lower) {
      alfa1 = alfa2(p - 1) - .05;
      hMinus = alfa1 * q0;
    }
    const double hCur = alfa2(p) * q1;
    if (higher) {
      alfa3 = alfa2(p + 1) - .25;
      hPlus = alfa3 * q2;
    }
    if (hMinus > hCur && hMinus > hPlus) {
      hScale = div_w(.75, alfa1) * hMinus; orderInNextStep = p - 1; odeOrderStatus = O_DEC;
    } else if (hCur > hMinus && hCur > hPlus) {
      hScale = div_w(.75, alfa2(p)) * hCur; orderInNextStep = p; odeOrderStatus = O_CONST;
    } else {
      hScale = div_w(.75, alfa3) * hPlus; orderInNextStep = p + 1; odeOrderStatus = O_INC;
    }
    if (fixedOrderMin) {
      iterMinimumOrder++;
      if (iterMinimumOrder < 2000) {
        hScale = div_w(.75, alfa2(p)) * hCur; orderInNextStep = p; odeOrderStatus = O_CONST;
      } else {
        fixedOrderMin = false;
      }
    }
    if (hScale < 1.2) {
      iterConstSteps++;
      hScale = 1.; odeHStatus = H_CONST; orderInNextStep = p; odeOrderStatus = O_CONST; hNextStep = h;
    } else {
      iterConstSteps = 0;
      hScale = fmin(hScale, hScaleMax);
      odeHStatus = H_INC;
      hNextStep = h * hScale;
    }
    if (iterConstSteps > 500 ||
        (numberOfSteps % 1000 == 0 && numberOfSteps != 0 && (fabs(h) < 1.e-7 || fabs(h) < 1.e-5 * t))) {
      if (p > (unsigned)MIN_ORDER) {
        fixedOrderMin = true; iterMinimumOrder = 0;
        orderInNextStep = MIN_ORDER; odeOrderStatus = O_DEC;
        hScale = 0.5; hNextStep = h * hScale; odeHStatus = H_DEC;
      }
    }
  }

  __device__ __forceinline__ void driver_step() {
    iterConvergenceFailure = 0; iterErrorFailure = 0; convergenceStatus = CONV_OK;
    if (odeOrderStatus != O_CONST || odeHStatus != H_CONST) iterOrder = 0;
    p = orderInNextStep;
    odeOrderStatus = O_CONST;
    hScaleMax = 2.;
    if (numberOfSteps < 10) hScaleMax = 1000.;
    else if (numberOfSteps > 10 && numberOfSteps < 20) hScaleMax = 10.;
#pragma unroll 1
    for (int guard = 0; guard < 1000000; ++guard) {
      if (odeHStatus != H_CONST) {
        hScale = div_w(hNextStep, hNordsieck);
        double hr = 1.;
#pragma unroll 1
        for (unsigned i = 1; i <= p; ++i) {
          hr *= hScale;
          if (active) Z(i) *= hr;
        }
        if (active) { double z0 = Z(0); check_constraints(z0); Z(0) = z0; }
        iterOrder = 0;
        odeHStatus = H_CONST;
      }
      h = hNextStep;
      hNordsieck = hNextStep;
      t = tInMeshPoint + h;
      if (t == tInMeshPoint) { status = -6; return; }
      __syncwarp();
      multi_value_step();
      if (convergenceStatus == CONV_FAIL) {
        iterConvergenceFailure++;
        ++cnt[CNT_CONVFAIL];
        if (iterConvergenceFailure >= 50u) { status = -5; return; }
        if (fabs(h - 0.) <= kMachEpsDouble * 0.) { status = -6; return; }
        convergence_failure_recovery();
      } else {
        double hCur = c_gear.Ep[p] * error_control(active ? V(p + 1) : 0., eps);
        if (hCur > 1.) {
          iterErrorFailure++;
          ++cnt[CNT_ERRFAIL];
          if (iterErrorFailure >= 50u) { status = -4; return; }
          if (fabs(h - 0.) <= kMachEpsDouble * 0.) { status = -6; return; }
          hScaleMax = 1.;
          hCur = 0.8 * pow_w(div_w(1., hCur), div_w(1., double(p + 1)));
          hScale = hCur;
          if (p > (unsigned)MIN_ORDER) {
            double hMinus = c_gear.Ep[p - 1] * error_control(active ? V(p) : 0., eps);
            hMinus = div_w(1., hMinus + kMachEpsFloat);
            hMinus = 0.8 * pow_w(hMinus, div_w(1., double(p)));
            if (hMinus > hCur) { hScale = hMinus; p -= 1; odeOrderStatus = O_DEC; }
          }
          hScale = fmin(hScale, 0.5);
          hScale = fmax(hScale, div_w(0., fabs(h)));
          hScale = fmax(hScale, 1.e-3);
          if (p == 1 && hScale < 0.1 && numberOfSteps > 10 && tInMeshPoint != tStabilize) {
            va = rhs(active ? Z(0) : 0.);
            if (active) Z(1) = va * h;
            tStabilize = tInMeshPoint;
          }
          odeHStatus = H_DEC;
          hNextStep *= hScale;
        } else {
          hNordsieck = h; hPreviousStep = h; hNextStep = h;
          orderInNextStep = p; odeOrderStatus = O_CONST; odeHStatus = H_CONST;
          convergence_rate();
          if (iterErrorFailure > 0 || iterConvergenceFailure > 0) {
            iterErrorFailure = 0; iterConvergenceFailure = 0;
          } else {
            iterOrder++;
            if (iterOrder > p + 1) new_order_new_h();
          }
          if (active) {
#pragma unroll 1
            for (unsigned i = 0; i <= p + 2; ++i) Z(i) = V(i);
            double z0 = Z(0); check_constraints(z0); Z(0) = z0;
          }
          __syncwarp();
          return;
        }
      }
      __syncwarp();
    }
    status = -5;
  }

  // MultiValueSolver::Solve from a fresh initial condition.  On failure y holds
  // the last accepted state.
  __device__ __forceinline__ int solve_to(double tEnd) {
    tOut = tEnd;
    const bool illegal = active && (y0 < minv || y0 > maxv);
    if (__any_sync(kFull, illegal)) { status = -9; y = y0; return status; }
    one_over_epsilon(y0);
    double lo, hi;
    if (t0 != 0.) { lo = 100. * kMachEpsDouble * fabs(t0); hi = fabs(t0); }
    else { lo = kMachEpsDouble; hi = 1.e-4; }
    double h0 = div_w(0.5, error_control(f, eps) + kMachEpsFloat);
    if (h0 < lo) h0 = lo;
    if (h0 > hi) h0 = hi;
    h0 *= div_w(fabs(tOut - t0), tOut - t0);
    if (active) { Z(0) = y0; Z(1) = f * h0; }
    hPreviousStep = h0; hNordsieck = h0; hNextStep = h0;
    status = 2;
    __syncwarp();
#pragma unroll 1
    for (unsigned k = 1; k <= max_number_steps; ++k) {
      one_over_epsilon(active ? Z(0) : 0.);
      const double tolSafe = kMachEpsDouble * error_control(active ? Z(0) : 0., eps);
      if (tolSafe > 1.) { status = -2; y = active ? Z(0) : 0.; return status; }
      tInMeshPoint = t;
      driver_step();
      if (status <= 0) { t = tInMeshPoint; y = active ? Z(0) : 0.; return status; }
      numberOfSteps++;
      ++cnt[CNT_STEPS];
      if (tOut == t) { y = active ? Z(0) : 0.; return status; }
      if (tOut < t) {
        // Interpolation (:687-706) + the extra RHS call that sets QR at tOut
        const double hp = div_w(tOut - t, hNordsieck);
        double hr = 1.;
        y = active ? Z(0) : 0.;
        if (hp != 0.) {
#pragma unroll 1
          for (unsigned i = 1; i <= p; ++i) {
            hr *= hp;
            if (active) { va = Z(i) * hr; y += va; }
          }
          check_constraints(y);
        }
        va = rhs(y);
        return status;
      }
    }
    status = -1;
    y = active ? Z(0) : 0.;
    return status;
  }
};

}  // namespace lsg
