// Per-cell property update after the reaction step: laminarSMOKE's loop over
// the cells in solvers/laminarSMOKE/properties.H:40-190, with the mixture
// rules of OpenSMOKE++'s maps:
//
// * x_i = MWmix Y_i / MW_i, MWmix = 1 / sum Y_i / MW_i
//   (ThermodynamicsMap_CHEMKIN.hpp:429-434);
// * cTot = p / (R T), psi = cTot MWmix / p, h = R T sum x_i (h/RT)_i / MWmix
//   (properties.H:93-96, ThermodynamicsMap_CHEMKIN.hpp:514-520);
// * mu: Wilke's rule over the fitted species viscosities, pairs k < j in the
//   reference's order (TransportPropertiesMap_CHEMKIN.hpp:729-766, 959-1001);
// * lambda: Mathur-Saxena, 0.5 (sum x lambda + 1 / sum x / lambda) (:947-957);
//   cp = sum x cp_i / MWmix, cv = (cp_molar - R) / MWmix, species cp_i / MW_i
//   (properties.H:103-122), evaluated when the energy equation is solved or
//   the Lewis-number diffusivities need them;
// * the simplified transport option mu0 (T/T0)^beta0, mu cp / Pr0 (:124-133);
// * Dmix: mixture-averaged, (MW~ - x~_k M_k) / (MW~ sum_j x~_j / D_kj) with
//   x~ = (x + 1e-14) / (1 + 1e-14 nc) and D_kj from the binary fits at the
//   cell's pressure (gamma :798-859, gammaMix :1032-1059); or
//   lambda / (p psi cp Le_k) with Lewis numbers (properties.H:152-162);
// * Dsoret_i = Dmix_i theta_i MW_i / MWmix, theta_i = sum_j theta_ij x_i x_j
//   for the light species (teta :768-796, tetaMix :1103-1117;
//   properties.H:177-189).
//
// One thread per cell.  Species rows are species-major with the cells of a
// warp in consecutive lanes, so every row read and written is coalesced.  The
// per-species work arrays of a cell sit in shared memory laid out
// [array][species][thread], so the lanes of a warp touch consecutive doubles;
// tables of up to 40 KB are copied into shared memory by each block, larger
// ones read as warp-uniform 16-byte loads through L1, which the streamed rows
// bypass.
//
// What a cell costs is arithmetic, not HBM: nc (nc - 1) / 2 binary fits, each an
// exponential, then nc^2 Wilke terms.  The FP64 pipe is 50 % busy; the rest are
// dependent chains in the 8 to 24 warps of an SM and, in Wilke's loop, shared
// memory (two work array entries and two table entries for every two pairs).  So the exponentials of the
// fits are a range reduction and a Taylor polynomial inline (exp_fit: 20
// instructions against some 60 of the library's), no pair divides (1 / D by the
// negated fit, sqrt(eta) and its reciprocal by half the fit's exponent), and a
// pair's Wilke terms use sqrt(phi) from the host.  Contraction is off: the sums
// whose terms cancel (h, the Soret terms) round like the host arithmetic, the others are written
// with fma.  1,048,576 H2/CO cells with
// every field: 1,510 us with divisions and the library's exponentials, 630 us now
// (the bytes alone: 92 us); 39,999 CH4 cells: 245 and 127 us.
#include "lsg_common.cuh"
#include "lsg_kernels.h"

namespace lsg {

namespace {
constexpr size_t kPropSmemMax = 200 * 1024;
constexpr size_t kPropTableMax = 40 * 1024;   // tables up to this size are copied into each block's shared memory
constexpr double kThreshold = 1.e-14;       // TransportPropertiesMap_CHEMKIN.hpp:47
constexpr double kMu0 = 1.8405e-5, kT0 = 300., kBeta0 = 0.6759, kPr0 = 0.7;   // properties.H:126-129

// e^x for the fits: x = k ln 2 + r with |r| <= ln 2 / 2 (ln 2 as an unevaluated sum of two doubles) and the Taylor
// polynomial of degree 13, whose remainder is below 4e-18, without a branch, so that several run interleaved.  It
// holds for |x| <= 690; a cell whose temperature lets a fit's exponent come near that (TransportLayout::T_min: far
// outside the fits, or NaN) is evaluated with the library's exp (kFast false).  The constants are held in registers through
// volatile asm: left to itself the compiler rebuilds each with two moves before every use.
struct ExpConst {
  double c[13];   // 1 / 13!, 1 / 12!, ..., 1 / 3!, then log2(e), ln 2
  __device__ __forceinline__ ExpConst() {
    const double v[13] = {1. / 6227020800., 1. / 479001600., 1. / 39916800., 1. / 3628800., 1. / 362880., 1. / 40320.,
                          1. / 5040., 1. / 720., 1. / 120., 1. / 24., 1. / 6., 1.4426950408889634, 0.6931471805599453};
#pragma unroll
    for (int i = 0; i < 13; ++i) asm volatile("mov.f64 %0, %1;" : "=d"(c[i]) : "d"(v[i]));
  }
};
template <bool kFast>
__device__ __forceinline__ double exp_fit(const ExpConst& e, double x) {
  if constexpr (!kFast) return exp(x);
  constexpr double kRound = 6755399441055744.;   // 1.5 * 2^52: adding it rounds to an integer
  const double t = fma(x, e.c[11], kRound), k = t - kRound;
  double r = fma(-k, e.c[12], x);
  r = fma(-k, 2.3190468138462996e-17, r);
  double p = e.c[0];
#pragma unroll
  for (int i = 1; i < 11; ++i) p = fma(p, r, e.c[i]);
  p = fma(p, r, .5);
  p = fma(p, r, 1.);
  p = fma(p, r, 1.);
  return __hiloint2double(__double2hiint(p) + (__double2loint(t) << 20), __double2loint(p));
}

// num / den with the zero numerators of absent species kept off the division's slow path; the same value.
__device__ __forceinline__ double div_z(double num, double den) {
  const bool z = num == 0.;
  const double q = (z ? 1. : num) / den;
  return z ? num * q : q;
}

// f[0] + f[1] x + f[2] x^2 + f[3] x^3 from a table row (16-byte aligned, the same in every lane)
__device__ __forceinline__ double cubic(const double* f, double x) {
  const double2 lo = *(const double2*)f, hi = *((const double2*)f + 1);
  return fma(fma(fma(hi.y, x, hi.x), x, lo.y), x, lo.x);
}

// work arrays of a block: two per thread and species (x; 1 / sqrt(eta), then the shifted mole fractions' sums)
size_t prop_smem(int nc, int bd) { return (size_t)2 * nc * bd * sizeof(double); }

// The block size that keeps most threads resident beside `tables` bytes of tables (0: none fits).
int pick_block(int nc, size_t tables) {
  int best = 0, most = 0;
  for (int bd : {128, 64, 32}) {
    const size_t per = prop_smem(nc, bd) + tables + 1024;
    if (prop_smem(nc, bd) + tables > kPropSmemMax) continue;
    long blocks = (long)(227 * 1024 / per);
    if (blocks * bd > 768) blocks = 768 / bd;   // what the registers allow
    if (blocks * bd > most) { most = (int)(blocks * bd); best = bd; }
  }
  return best;
}

size_t table_bytes(const MechLayout& L, const TransportLayout& TL) {
  const size_t b = sizeof(double) * ((size_t)TL.n_double + L.ds_ht + L.nc + 1);
  return b <= kPropTableMax ? b : 0;
}
}  // namespace

constexpr int kPropMaxSpecies = 266;
int properties_block(int nc) { return nc <= kPropMaxSpecies ? pick_block(nc, 0) : 0; }

// The tables of a block: the mechanism's and the transport doubles, the species' middle temperatures, the light
// species' indices.
struct Tables {
  const double *MD, *TD, *TM;
  const int* TI;
};

// What a cell reads: its mass fractions go to xs.  All of it is read before anything is written, so that a field may
// take the place of an input.
struct CellInputs {
  double T, p, u;   // temperature, pressure, sum Y_i / MW_i
};
template <int BD>
__device__ __forceinline__ CellInputs cell_inputs(const PropArgs& a, const double* MW, int nc, double* xs, long c) {
  CellInputs in;
  in.T = __ldcs(a.T + c);
  in.p = a.p ? __ldcs(a.p + c) : a.p_scalar;
  double u = 0.;
#pragma unroll 4
  for (int s = 0; s < nc; ++s) {
    const double y = __ldcs(a.Y + s * a.ld + c);
    xs[s * BD] = y;
    u += div_z(y, MW[s]);
  }
  in.u = u;
  return in;
}

// One cell.
template <int BD, bool kFast>
__device__ __forceinline__ void cell_properties(const MechLayout& L, const TransportLayout& TL, const PropArgs& a,
                                                const Tables& tb, double* xs, double* us, long c, const CellInputs& in) {
  const int nc = L.nc;
  const double *MD = tb.MD, *TD = tb.TD, *TM = tb.TM;
  const double* MW = MD + L.mw;
  const long lo = a.ld_out;
  const ExpConst E;
  const double T = in.T, p = in.p;
  const double MWm = 1. / in.u;
  const double cTot = p / kRgas / T;
  const double psi = cTot * MWm / p;
  if (a.MWmix) __stcs(a.MWmix + c, MWm);
  if (a.cTot) __stcs(a.cTot + c, cTot);
  if (a.psi) __stcs(a.psi + c, psi);

  const bool lewis = a.lewis != nullptr, thermal = a.energy || lewis;
  const double T2 = T * T, T3 = T2 * T, T4 = T3 * T, uT = 1. / T, lT = log(T);
  double hmix = 0., cpm = 0., l1 = 0., l2 = 0.;
  for (int s = 0; s < nc; ++s) {
    const double x = div_z(MWm * xs[s * BD], MW[s]);
    xs[s * BD] = x;
    if (a.X) __stcs(a.X + s * lo + c, x);
    const bool hi = T > TM[s];
    if (a.h) {
      const double* d = (hi ? MD + L.dh_ht : MD + L.dh_lt) + 6 * s;
      hmix += (d[0] + T * d[1] + T2 * d[2] + T3 * d[3] + T4 * d[4] + uT * d[5]) * x;
    }
    const double half = 0.5 * cubic(TD + TL.eta + 4 * s, lT);
    us[s * BD] = exp_fit<kFast>(E, -half);
    if (thermal) {
      const double ll = cubic(TD + TL.lam + 4 * s, lT);
      l1 = fma(x, exp_fit<kFast>(E, ll), l1);
      l2 = fma(x, exp_fit<kFast>(E, -ll), l2);
      const double* q = (hi ? MD + L.cp_ht : MD + L.cp_lt) + 5 * s;
      const double cpr = q[0] + T * q[1] + T2 * q[2] + T3 * q[3] + T4 * q[4];
      cpm += cpr * x;
      if (a.cp_species) __stcs(a.cp_species + s * lo + c, (cpr * kRgas) / MW[s]);
    }
  }
  if (a.h) __stcs(a.h + c, hmix * (kRgas * T) / MWm);
  double lambda = 0., cp = 0.;
  if (thermal) {
    lambda = 0.50 * (l1 + 1. / l2);
    cpm *= kRgas;
    if (a.cv) __stcs(a.cv + c, (cpm - kRgas) / MWm);
    cp = cpm / MWm;
    if (a.cp) __stcs(a.cp + c, cp);
  }
  double mu = 0.;
  if (a.simplified) {
    mu = kMu0 * pow(T / kT0, kBeta0);
    lambda = mu * cp / kPr0;
  } else if (a.mu) {
    // Wilke's rule (etaMix): mu = sum_k x_k eta_k / sum_j x_j phi_kj (1 + sqrt(eta_k / eta_j) (M_j / M_k)^(1/4))^2,
    // two k a turn so that a cell's x_j and 1 / sqrt(eta_j) are read half as often; the pair's table entry holds
    // sqrt(phi) and sqrt(phi) (M_j / M_k)^(1/4)
    const double2* W = (const double2*)(TD + TL.wilke);
    for (int k = 0; k < nc; k += 2) {
      const int k1 = k + 1 < nc ? k + 1 : k;
      const double u0 = us[k * BD], u1 = us[k1 * BD], s0 = 1. / u0, s1 = 1. / u1;
      const double2 *w0 = W + k * nc, *w1 = W + k1 * nc;
      double a0 = 0., a1 = 0.;
#pragma unroll 4
      for (int j = 0; j < nc; ++j) {
        const double x = xs[j * BD], v = us[j * BD];
        const double2 f0 = w0[j], f1 = w1[j];
        const double d0 = fma(f0.y, s0 * v, f0.x), d1 = fma(f1.y, s1 * v, f1.x);
        a0 = fma(x, d0 * d0, a0);
        a1 = fma(x, d1 * d1, a1);
      }
      mu += div_z(xs[k * BD], u0 * u0 * a0);
      if (k + 1 < nc) mu += div_z(xs[k1 * BD], u1 * u1 * a1);
    }
  }
  if (a.mu) __stcs(a.mu + c, mu);
  if (thermal && a.lambda) __stcs(a.lambda + c, lambda);

  if (!a.Dmix) return;
  const int* it = tb.TI;
  if (a.Dsoret) {   // the thermal-diffusion ratios, while x is at hand; scaled by Dmix below
    const double* ft = TD + TL.teta;
    for (int m = 0; m < TL.n_teta; ++m) {
      const double xi = xs[it[m] * BD];
      double th = 0.;
#pragma unroll 4
      for (int j = 0; j < nc; ++j, ft += 4) {   // terms of both signs: uncontracted, as the host
        const double2 f0 = *(const double2*)ft, f1 = *((const double2*)ft + 1);
        th += (f0.x + f0.y * T + f1.x * T2 + f1.y * T3) * xi * xs[j * BD];
      }
      a.Dsoret[m * lo + c] = th;
    }
  }
  double* acc = us;
  if (lewis) {
    const double coef = lambda / (p * psi) / cp;
    for (int s = 0; s < nc; ++s) {
      const double D = coef / a.lewis[s];
      acc[s * BD] = D;
      __stcs(a.Dmix + s * lo + c, D);
    }
  } else {
    const double pbar = p / 100000.;
    const double sum_thr = 1. + kThreshold * (double)nc;
    double MWc = 0.;
    for (int s = 0; s < nc; ++s) {   // the shifted mole fractions replace x
      const double x = (xs[s * BD] + kThreshold) / sum_thr;
      xs[s * BD] = x;
      MWc += x * MW[s];
      acc[s * BD] = 0.;
    }
    // sums over the pairs of x / D at 1 bar, 1 / D by the negated fit
    const double* fg = TD + TL.gam;
    for (int k = 0; k < nc; ++k) {
      const double xk = xs[k * BD];
      double sk = acc[k * BD];
      int j = k + 1;
      for (; j + 4 <= nc; j += 4, fg += 16) {   // four pairs interleaved
        double g[4], v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          g[q] = -cubic(fg + 4 * q, lT);
          v[q] = acc[(j + q) * BD];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) g[q] = exp_fit<kFast>(E, g[q]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          sk = fma(xs[(j + q) * BD], g[q], sk);
          acc[(j + q) * BD] = fma(xk, g[q], v[q]);
        }
      }
      for (; j < nc; ++j, fg += 4) {
        const double g = exp_fit<kFast>(E, -cubic(fg, lT));
        sk = fma(xs[j * BD], g, sk);
        acc[j * BD] = fma(xk, g, acc[j * BD]);
      }
      const double D = (MWc - xk * MW[k]) / (MWc * (pbar * sk));
      acc[k * BD] = D;
      __stcs(a.Dmix + k * lo + c, D);
    }
  }
  if (!a.Dsoret) return;
  for (int m = 0; m < TL.n_teta; ++m) {
    const int i = it[m];
    a.Dsoret[m * lo + c] = acc[i * BD] * a.Dsoret[m * lo + c] * MW[i] / MWm;
  }
}

// The same cell with the library's exponentials.
template <int BD>
__device__ __noinline__ void cell_properties_slow(const MechLayout& L, const TransportLayout& TL, const PropArgs& a,
                                                  const Tables& tb, double* xs, double* us, long c, const CellInputs in) {
  cell_properties<BD, false>(L, TL, a, tb, xs, us, c, in);
}

// BD threads a block; STAGED: the tables are in shared memory (the mechanism's doubles up to the entropy fits and the
// species' middle temperatures, the whole transport table), else read through L1.
template <int BD, bool STAGED>
__global__ void __launch_bounds__(BD) properties_kernel(const __grid_constant__ MechLayout L,
                                                        const unsigned char* __restrict__ mech_gmem,
                                                        const __grid_constant__ TransportLayout TL,
                                                        const unsigned char* __restrict__ tr_gmem,
                                                        const __grid_constant__ PropArgs a) {
  extern __shared__ __align__(16) double sm[];
  const int nc = L.nc;
  Tables tb{(const double*)mech_gmem, (const double*)tr_gmem, (const double*)mech_gmem + L.t_mid,
            (const int*)(tr_gmem + (size_t)TL.n_double * sizeof(double)) + TL.iteta};
  double* xs = sm + threadIdx.x;             // xs[s * BD]
  double* us = xs + nc * BD;
  if constexpr (STAGED) {
    double2* t = (double2*)(sm + 2 * nc * BD);
    const int nt = TL.n_double / 2, nm = (L.ds_ht + 1) / 2;
    for (int i = threadIdx.x; i < nt; i += BD) t[i] = ((const double2*)tr_gmem)[i];
    for (int i = threadIdx.x; i < nm; i += BD) t[nt + i] = ((const double2*)mech_gmem)[i];
    double* tm = (double*)(t + nt + nm);
    for (int i = threadIdx.x; i < nc; i += BD) tm[i] = tb.TM[i];
    __syncthreads();
    tb.TD = sm + 2 * nc * BD;
    tb.MD = tb.TD + 2 * nt;
    tb.TM = tm;
  }
  const long c = blockIdx.x * (long)BD + threadIdx.x;
  if (c >= a.ncells) return;   // no block barriers below
  const CellInputs in = cell_inputs<BD>(a, tb.MD + L.mw, nc, xs, c);
  if (in.T >= TL.T_min && in.T <= TL.T_max) cell_properties<BD, true>(L, TL, a, tb, xs, us, c, in);
  else cell_properties_slow<BD>(L, TL, a, tb, xs, us, c, in);
}

namespace {
template <int BD, bool STAGED>
cudaError_t props(const MechLayout& L, const unsigned char* mech_gmem, const TransportLayout& TL,
                  const unsigned char* tr_gmem, const PropArgs& a, size_t smem, cudaStream_t stream) {
  // the same value at every call: another thread may launch the kernel with another size at the same time
  const cudaError_t e = cudaFuncSetAttribute(properties_kernel<BD, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kPropSmemMax);
  if (e != cudaSuccess) return e;
  const long grid = (a.ncells + BD - 1) / BD;
  properties_kernel<BD, STAGED><<<(unsigned)grid, BD, smem, stream>>>(L, mech_gmem, TL, tr_gmem, a);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_properties(const MechLayout& L, const unsigned char* mech_gmem, const TransportLayout& TL,
                              const unsigned char* tr_gmem, const PropArgs& a, cudaStream_t stream) {
  if (a.ncells <= 0) return cudaSuccess;
  const size_t tables = table_bytes(L, TL);
  const int bd = pick_block(L.nc, tables);
  if (bd == 0) return cudaErrorInvalidValue;
  const size_t smem = prop_smem(L.nc, bd) + tables;
  if (tables == 0) {
    if (bd == 128) return props<128, false>(L, mech_gmem, TL, tr_gmem, a, smem, stream);
    if (bd == 64) return props<64, false>(L, mech_gmem, TL, tr_gmem, a, smem, stream);
    return props<32, false>(L, mech_gmem, TL, tr_gmem, a, smem, stream);
  }
  if (bd == 128) return props<128, true>(L, mech_gmem, TL, tr_gmem, a, smem, stream);
  if (bd == 64) return props<64, true>(L, mech_gmem, TL, tr_gmem, a, smem, stream);
  return props<32, true>(L, mech_gmem, TL, tr_gmem, a, smem, stream);
}

}  // namespace lsg
