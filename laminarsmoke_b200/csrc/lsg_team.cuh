// Resident form of the batched step: a block keeps up to 32 cells -- their whole
// solver state, Jacobian and inverse -- in shared memory from the pending
// request to the end of the step, and runs the round scheme's solver with the
// round scheme's arithmetic, operation by operation, so a cell's result does not
// depend on which of the two integrates it.  Every turn of a block
//
//   1. hands its 32 evaluation slots to the cells' requests: one for a plain
//      request, the columns of a finite-difference Jacobian to what is free;
//   2. evaluates the right-hand sides of all slots (rhs_slots): lane = slot,
//      warp = species or reaction, so that a warp runs one reaction's code for
//      all cells without divergence; every sum in rhs_cell's order;
//   3. advances the cells whose request is complete (advance_team): a team of
//      W lanes a cell (16, two cells a warp, or a whole warp), lane =
//      component, through the Gear state machine to the next request.
//
// The barriers between the stages also keep the warps on the same code: with
// every warp on its own the kernel spent 60 % of its time on instruction fetch.
// What bounds it now: the longest dependent FP64 chain of a turn; 47 % of a warp's
// time is at the turn's barriers, where the others wait for it.  There is no HBM traffic between a cell's load and its store; the mechanism tables
// are read through L1 at warp-uniform addresses.
#pragma once

namespace lsg {
namespace {

constexpr int kTeamThreads = 512;   // one block per SM: 16 warps of up to 128 registers
constexpr int kTeamWarps = kTeamThreads / 32;
constexpr int kSlots = 32;          // right-hand sides of a turn, one per lane

// Shared memory of one team, in doubles: the record's head and vectors (rec_layout's offsets), the Jacobian and
// the inverse (FP64 whatever the precision of the factorisation) by rows of ld, scratch for a vector and the
// elimination's pivot row and interchanges; an odd total, so that a component of 32 teams falls on 32 banks.
struct TeamLayout {
  int oj, ox, osc, total, ld;
};
__host__ __device__ inline TeamLayout team_layout(int n) {
  TeamLayout t{};
  t.ld = row_ld(n);
  t.oj = ND_ + NI_ / 2 + 22 * n;
  t.ox = t.oj + n * t.ld;
  t.osc = t.ox + n * t.ld;
  t.total = (t.osc + 2 * n) | 1;
  return t;
}

// Shared memory of the evaluation slots, in doubles [row][kSlots]: per species (C, g) pairs, an absent species
// (1, 0) and (R, h/RT) pairs; per reaction the rate constant, then the net rate; per fall-off slot k_inf and
// log10 F_cent; scalars.
enum : int { SS_T = 0, SS_LOGT, SS_UT, SS_LP, SS_MW, SS_CTOT, SS_RHO, SS_HJ, SS_HINV, SS_N };
struct SlotLayout {
  int cg, rh, net, fo, sc, total;
};
// Start of a team block's dynamic shared memory: everything the out-of-line functions read, so that they address
// it as shared memory (through pointers they would load by generic address).
struct TeamHead {
  MechLayout L;
  TeamLayout T;
  RecLayout R;
  SlotLayout S;
  StepOptions o;
  StepArgs a;
  const double* Md;
  const int* Mi;
};
constexpr int kHeadDoubles = (int)((sizeof(TeamHead) + 15) / 16 * 2);
extern __shared__ __align__(16) double team_smem[];
__device__ __forceinline__ const TeamHead& team_head() { return *(const TeamHead*)team_smem; }

__host__ __device__ inline SlotLayout slot_layout(const MechLayout& L) {
  SlotLayout s{};
  s.cg = kHeadDoubles;
  s.rh = s.cg + 2 * (L.nc + 1) * kSlots;
  s.net = s.rh + 2 * L.nc * kSlots;
  s.fo = s.net + L.nr * kSlots;
  s.sc = s.fo + 2 * L.n_fo * kSlots;
  s.total = s.sc + SS_N * kSlots;
  return s;
}

// One copy of each transcendental: the team kernels are bound by instruction fetch before anything else (with
// every call site inlined, 15 of the 21 cycles between a warp's instructions went to it), so code size comes first.
__device__ __noinline__ double exp_o(double x) { return exp(x); }
__device__ __noinline__ double log_o(double x) { return log(x); }
__device__ __noinline__ double log10_o(double x) { return log10(x); }
__device__ __noinline__ double exp10_o(double x) { return exp10(x); }

// num / den to the last bit, for numerators that are often exactly zero (absent species): the division of a zero
// leaves the fast path (some 100 instructions instead of 10), so a zero is multiplied by 1 / den instead, which
// gives the same zero, NaN or sign.
__device__ __forceinline__ double div0(double num, double den) {
  const bool z = num == 0.;
  const double q = (z ? 1. : num) / den;
  return z ? num * q : q;
}

// The evaluation slots as the rate functions see them: this lane's column.
struct Slot {
  int cg;   // (C, h/RT - s/R) of species k at team_smem[cg + 2 kSlots k]
  __device__ __forceinline__ double C(int k) const { return team_smem[cg + 2 * kSlots * k]; }
  __device__ __forceinline__ double G(int k) const { return team_smem[cg + 2 * kSlots * k + 1]; }
  __device__ __forceinline__ double total(int nc) const {   // the concentrations' sum, in species order
    double s = 0.;
#pragma unroll 4
    for (int i = 0; i < nc; ++i) s += C(i);
    return s;
  }
};

// Third-body concentration of slot s of a (pointer, species, efficiency - 1) list.
__device__ __forceinline__ double third_body(const int* ptr, const int* sp, const double* eff, int s, double cTotSum,
                                             const Slot& S) {
  double Mc = cTotSum;
  const int qe = ptr[s + 1];
#pragma unroll 2
  for (int q = ptr[s]; q < qe; ++q) Mc += S.C(sp[q]) * eff[q];
  return Mc;
}

// log10 F of the Troe form at the reduced pressure Pr (KineticsMap_CHEMKIN.hpp:1496-1550)
__device__ __forceinline__ double troe_f(double lF, double Pr, bool cabr) {
  double qq;
  if (Pr > 1.e-32 || cabr) {
    const double nTroe = 0.75 - 1.27 * lF;
    const double cTroe = -0.4 - 0.67 * lF;
    const double sTroe = log10_o(Pr) + cTroe;
    qq = sTroe / (nTroe - 0.14 * sTroe);
  } else {
    qq = 1. / 0.14;
  }
  return exp10_o(lF / (1. + qq * qq));
}

// Fall-off / CABR factor applied to kMod (KineticsMap_CHEMKIN.hpp:1257-1290, 1496-1550, 1613-1660), as in
// rhs_cell; the SRI form keeps its calls inline, where the compiler rounds them as there.
__device__ __noinline__ double falloff_mod(int fo, double kArr, double kMod, double Mc,
                                           double T, double logT, double uT) {
  const MechLayout& L = team_head().L;
  const MechView M{team_head().Md, team_head().Mi};
  const double kInf = exp_o(M.D(L.fo_lnA)[fo] + M.D(L.fo_beta)[fo] * logT - M.D(L.fo_eor)[fo] * uT);
  const double a = M.D(L.fo_a)[fo], b = M.D(L.fo_b)[fo], c = M.D(L.fo_c)[fo], d = M.D(L.fo_d)[fo];
  const int ty = M.I(L.fo_type)[fo];
  const double Pr = kArr * Mc / kInf;
  const bool cabr = M.I(L.fo_cabr)[fo] != 0;
  double wF = 1.;
  if (ty == 1) {
    double v = (1. - a) * exp_o(-T / b) + a * exp_o(-T / c);
    if (d != 0.) v += exp_o(-d / T);
    wF = troe_f((v < 1.e-300) ? -300. : log10_o(v), Pr, cabr);
  } else if (ty == 2) {
    const double lF = a * exp(-b / T) + exp(-T / c);
    const double l10 = log10(Pr);
    const double xSRI = 1. / (1. + l10 * l10);
    wF = pow(lF, xSRI) * d;
    const double e = M.D(L.fo_e)[fo];
    if (e != 0.) wF *= pow(T, e);
  }
  if (cabr) kMod *= (1. / (1. + Pr)) * wF;
  else kMod *= kInf * (Pr / (1. + Pr)) * wF / kArr;
  return kMod;
}

// Net rate of a reaction outside the packed form (mech.h rx_pack): any stoichiometry, FORD orders, explicit
// reverse parameters, PLOG, CHEB and the extended forms; rhs_cell's text.
__device__ __noinline__ double special_rate(int j, const Slot S, double cTotSum, double T,
                                            double logT, double uT, double lP, double Pk) {
  const MechLayout& L = team_head().L;
  const MechView M{team_head().Md, team_head().Mi};
  double kArr = exp(M.D(L.lnA)[j] + M.D(L.beta)[j] * logT - M.D(L.eor)[j] * uT);
  if (M.I(L.a_sign)[j] < 0) kArr *= -1.;
  if (L.n_plog > 0) {
    const int ps = M.I(L.plog_slot)[j];
    if (ps >= 0) kArr = plog_k(M, L, ps, T, logT, Pk);
  }
  if (L.n_cheb > 0) {
    const int cs = M.I(L.cheb_slot)[j];
    if (cs >= 0) kArr = cheb_k(M, L, cs, T, Pk);
  }
  if (L.n_xplog > 0) {
    const int xs = M.I(L.xplog_slot)[j];
    if (xs >= 0) kArr = xplog_k(M, L, xs, T, logT, Pk, cTotSum, [&](int k) { return S.C(k); });
  }
  double kMod = kArr;
  const int tb = M.I(L.tb_slot)[j];
  if (tb >= 0) kMod *= third_body(M.I(L.tb_ptr), M.I(L.tb_sp), M.D(L.tb_eff), tb, cTotSum, S);
  const int fo = M.I(L.fo_slot)[j];
  if (fo >= 0) {
    const int single = M.I(L.fo_single)[fo];
    const double Mc = single < 0 ? third_body(M.I(L.fo_ptr), M.I(L.fo_sp), M.D(L.fo_eff), fo, cTotSum, S)
                                 : S.C(single) + 1.e-16;
    kMod = falloff_mod(fo, kArr, kMod, Mc, T, logT, uT);
  }
  if (L.n_xfo > 0) {
    const int xs = M.I(L.xfo_slot)[j];
    if (xs >= 0) {
      kArr = xfo_k(M, L, xs, T, cTotSum, [&](int k) { return S.C(k); });
      kMod = kArr;
    }
  }
  const int* rp = M.I(L.reac_ptr);
  const int* rsp = M.I(L.reac_sp);
  const double* rnu = M.D(L.reac_nu);
  const int* op = M.I(L.ford_ptr);
  const int* osp = M.I(L.ford_sp);
  const double* onu = M.D(L.ford_val);
  const int* pp = M.I(L.prod_ptr);
  const int* psp = M.I(L.prod_sp);
  const double* pnu = M.D(L.prod_nu);
  double fwd = 1.;
  for (int q = op[j]; q < op[j + 1]; ++q) fwd *= conc_factor_r(onu[q], S.C(osp[q]));
  double net = fwd;
  const int kind = M.I(L.rev_kind)[j];
  if (kind != 0) {
    double rv = 1.;
    for (int q = pp[j]; q < pp[j + 1]; ++q) rv *= conc_factor_r(pnu[q], S.C(psp[q]));
    double rf;
    if (kind == 1) {
      double dg = 0.;
      for (int q = pp[j]; q < pp[j + 1]; ++q) dg += contrib_r(pnu[q], S.G(psp[q]));
      for (int q = rp[j]; q < rp[j + 1]; ++q) dg -= contrib_r(rnu[q], S.G(rsp[q]));
      rf = exp(dg - lP * M.D(L.dnu)[j]);
    } else {
      const int sr = M.I(L.rev_slot)[j];
      rf = exp(M.D(L.rev_lnA)[sr] + M.D(L.rev_beta)[sr] * logT - M.D(L.rev_eor)[sr] * uT) / kArr;
    }
    rv *= rf;
    net -= rv;
  }
  return net * kMod;
}

// Static split of a stage's items over nw warps: `big` items that weigh wt small ones are dealt out in turn, then
// the small ones in rounds, the warps that hold one big item more joining after wt rounds.  The small item of
// warp w in round r (w its number among the nw):
__device__ __forceinline__ int small_item(int r, int w, int nw, int big, int wt) {
  const int x = big % nw;
  if (r < wt) return w < x ? -1 : r * (nw - x) + w - x;
  return wt * (nw - x) + (r - wt) * nw + w;
}

// What a slot evaluates, as places in team_smem: the input vector y (component col replaced by y + hj), the
// destination of the derivatives (stride ds), and for a Jacobian column f0 (negative: a plain request).
struct Eval {
  int y, dst, f0, ds, col;
};

// The right-hand sides of a block's slots, lane = slot; called by every thread of the block, with a barrier
// before (the slots' SS_HJ and SS_HINV are set) and after.  Bit for bit rhs_cell's values: the sums over
// species and the formation rates run in its order, and its divisions and logarithms are the same operations.
// Returns QR in warp 0.
__device__ __noinline__ double rhs_slots(const Eval ev, bool live, double P0, int energy, double rho0) {
  const MechLayout& L = team_head().L;
  const SlotLayout& SL = team_head().S;
  const MechView M{team_head().Md, team_head().Mi};
  const int NC = L.nc, NR = L.nr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2* const CG = (double2*)(team_smem + SL.cg) + lane;
  double2* const RH = (double2*)(team_smem + SL.rh) + lane;
  double* const NET = team_smem + SL.net + lane;
  double* const FO = team_smem + SL.fo + lane;
  double* const SS = team_smem + SL.sc + lane;
  const Slot S{SL.cg + 2 * lane};
  const bool cv = rho0 > 0.;
  auto y = [&](int i) {
    const double v = team_smem[ev.y + i];
    return i == ev.col ? v + SS[SS_HJ * kSlots] : v;
  };
  const double* MW = M.D(L.mw);
  // ---- Y_i / MW_i; the functions of T alone
  for (int e = warp; e < NC + 2; e += kTeamWarps) {
    if (e == 0) {
      const double T = y(NC);
      SS[SS_T * kSlots] = T;
      SS[SS_UT * kSlots] = 1. / T;
      SS[SS_LOGT * kSlots] = log_o(T);
    } else if (e == 1) {
      SS[SS_LP * kSlots] = log_o(101325. / kRgas / y(NC));
      CG[NC * kSlots] = make_double2(1., 0.);
    } else {
      CG[(e - 2) * kSlots].x = div0(y(e - 2), MW[e - 2]);
    }
  }
  __syncthreads();
  const double T = SS[SS_T * kSlots], logT = SS[SS_LOGT * kSlots], uT = SS[SS_UT * kSlots];
  const double T2 = T * T, T3 = T2 * T, T4 = T3 * T;
  // ---- warp 0: mixture molecular weight, total concentration; the others: k_inf and F_cent of the fall-off
  // reactions, Arrhenius constants and species free energies
  if (warp == 0) {
    double u = 0.;
#pragma unroll 4
    for (int i = 0; i < NC; ++i) u += CG[i * kSlots].x;
    const double MWmix = 1. / u;
    const double cTot = cv ? rho0 / MWmix : P0 / kRgas / T;
    SS[SS_MW * kSlots] = MWmix;
    SS[SS_CTOT * kSlots] = cTot;
    SS[SS_RHO * kSlots] = cv ? rho0 : cTot * MWmix;
  } else {
    for (int k = warp - 1; k < L.n_fo; k += kTeamWarps - 1) {
      const int ty = M.I(L.fo_type)[k];
      if (ty == 2) continue;   // SRI: evaluated with the reaction
      FO[2 * k * kSlots] = exp_o(M.D(L.fo_lnA)[k] + M.D(L.fo_beta)[k] * logT - M.D(L.fo_eor)[k] * uT);
      if (ty == 1) {
        const double a = M.D(L.fo_a)[k], b = M.D(L.fo_b)[k], c = M.D(L.fo_c)[k], d = M.D(L.fo_d)[k];
        double v = (1. - a) * exp_o(-T / b) + a * exp_o(-T / c);
        if (d != 0.) v += exp_o(-d / T);
        FO[(2 * k + 1) * kSlots] = (v < 1.e-300) ? -300. : log10_o(v);
      }
    }
    const int4* rx = (const int4*)M.I(L.rx_pack);
    const double4* rd = (const double4*)M.D(L.rx_dat);
    for (int r = 0, e; (e = small_item(r, warp - 1, kTeamWarps - 1, L.n_fo, 5)) < NR + NC; ++r) {
      if (e < 0) continue;
      if (e < NR) {
        if (rx[e].y & kRxSpecial) continue;
        const double4 d = rd[e];   // lnA, beta, E/R, dnu
        double kArr = exp_o(d.x + d.y * logT - d.z * uT);
        if (rx[e].y & kRxNegative) kArr *= -1.;
        NET[e * kSlots] = kArr;
      } else {
        const int i = e - NR;
        const bool hi = T > M.D(L.t_mid)[i];
        const double* A = (hi ? M.D(L.dh_ht) : M.D(L.dh_lt)) + 6 * i;
        const double hrt = A[0] + T * A[1] + T2 * A[2] + T3 * A[3] + T4 * A[4] + uT * A[5];
        const double* B = (hi ? M.D(L.ds_ht) : M.D(L.ds_lt)) + 6 * i;
        CG[i * kSlots].y = hrt - (B[0] * logT + T * B[1] + T2 * B[2] + T3 * B[3] + T4 * B[4] + B[5]);
        RH[i * kSlots].y = hrt;
      }
    }
  }
  __syncthreads();
  const double MWmix = SS[SS_MW * kSlots], cTot = SS[SS_CTOT * kSlots], rho = SS[SS_RHO * kSlots];
  for (int i = warp; i < NC; i += kTeamWarps) {
    double x = MWmix * y(i);
    x = div0(x, MW[i]);
    CG[i * kSlots].x = cTot * x;
  }
  __syncthreads();
  // ---- net rates, fall-off reactions first
  {
    const int4* rx = (const int4*)M.I(L.rx_pack);
    const double4* rd = (const double4*)M.D(L.rx_dat);
    const int* ord = M.I(L.rx_order);
    const double lP = SS[SS_LP * kSlots];
    // the warp's fall-off reactions, then its share of the others
    const int NF = L.n_fo < NR ? L.n_fo : NR;
    const int nb = (NF + kTeamWarps - 1 - warp) / kTeamWarps;
    for (int k = -nb;; ++k) {
      int e = k < 0 ? (k + nb) * kTeamWarps + warp : small_item(k, warp, kTeamWarps, NF, 4);
      if (k >= 0) {
        if (e >= NR - NF) break;
        if (e < 0) continue;
        e += NF;
      }
      const int j = ord[e];
      const int4 r = rx[j];
      double net;
      if (r.y & kRxSpecial) {
        net = special_rate(j, S, S.total(NC), T, logT, uT, lP, cv ? cTot * kRgas * T : P0);
      } else {
        const double kArr = NET[j * kSlots];
        double kMod = kArr;
        if (r.z >= 0) kMod *= third_body(M.I(L.tb_ptr), M.I(L.tb_sp), M.D(L.tb_eff), r.z, S.total(NC), S);
        if (r.w >= 0) {
          const int single = M.I(L.fo_single)[r.w], ty = M.I(L.fo_type)[r.w];
          const double Mc = single < 0 ? third_body(M.I(L.fo_ptr), M.I(L.fo_sp), M.D(L.fo_eff), r.w, S.total(NC), S)
                                       : S.C(single) + 1.e-16;
          if (ty == 2) {
            kMod = falloff_mod(r.w, kArr, kMod, Mc, T, logT, uT);
          } else {
            const double kInf = FO[2 * r.w * kSlots];
            const double Pr = kArr * Mc / kInf;
            const bool cabr = M.I(L.fo_cabr)[r.w] != 0;
            const double wF = ty == 1 ? troe_f(FO[(2 * r.w + 1) * kSlots], Pr, cabr) : 1.;
            if (cabr) kMod *= (1. / (1. + Pr)) * wF;
            else kMod *= kInf * (Pr / (1. + Pr)) * wF / kArr;
          }
        }
        const double2 a0 = CG[(r.x & 255) * kSlots], a1 = CG[((r.x >> 8) & 255) * kSlots];
        net = a0.x * a1.x;
        if (r.y & kRxReversible) {
          const double2 b0 = CG[((r.x >> 16) & 255) * kSlots], b1 = CG[((r.x >> 24) & 255) * kSlots];
          double rv = b0.x * b1.x;
          double dg = b0.y + b1.y;
          if (r.y & kRxTwice) {
            dg -= a0.y + a0.y;
          } else {
            dg -= a0.y;
            dg -= a1.y;
          }
          const double rf = exp_o(dg - lP * rd[j].w);
          rv *= rf;
          net -= rv;
        }
        net *= kMod;
      }
      NET[j * kSlots] = net;
    }
  }
  __syncthreads();
  // ---- formation rates in reaction order (rhs_cell's accumulation), derivatives, terms of the two sums
  const double hinv = SS[SS_HINV * kSlots];
  for (int i = warp; i < NC; i += kTeamWarps) {
    const double2* fg = (const double2*)M.D(L.fg_ent);   // (coefficient, reaction): +-1 and +-2 make exact products
    const int qe = M.I(L.fg_ptr)[i + 1];
    double Rl = 0.;
    if (L.fg_exact) {
#pragma unroll 4
      for (int q = M.I(L.fg_ptr)[i]; q < qe; ++q) {
        const double2 e = fg[q];
        Rl = __fma_rn(e.x, NET[__double2loint(e.y) * kSlots], Rl);
      }
    } else {
      for (int q = M.I(L.fg_ptr)[i]; q < qe; ++q) {
        const double2 e = fg[q];
        const double v = NET[__double2loint(e.y) * kSlots];
        if (e.x < 0.) Rl -= contrib_r(-e.x, v);
        else Rl += contrib_r(e.x, v);
      }
    }
    const double f = div0(MW[i] * Rl, rho);
    if (live) team_smem[ev.dst + i * ev.ds] = ev.f0 >= 0 ? hinv * (f - team_smem[ev.f0 + i]) : f;
    if (energy) {
      const double* A = (T > M.D(L.t_mid)[i] ? M.D(L.cp_ht) : M.D(L.cp_lt)) + 5 * i;
      CG[i * kSlots] = make_double2(A[0] + T * A[1] + T2 * A[2] + T3 * A[3] + T4 * A[4], div0(CG[i * kSlots].x, cTot));
    }
    RH[i * kSlots].x = Rl;
  }
  __syncthreads();
  double QR = 0.;
  if (warp == 0) {
    double dT = 0.;
    if (energy) {
      double cpm = 0., dsum = 0.;
#pragma unroll 2
      for (int i = 0; i < NC; ++i) {
        const double2 c = CG[i * kSlots], r = RH[i * kSlots];
        cpm += c.x * c.y;
        dsum += r.x * r.y;
      }
      cpm *= kRgas;
      QR = -dsum * kRgas * T;
      if (cv) {
        const double CvMixMass = (cpm - kRgas) / MWmix;
        double sumR = 0.;
        for (int i = 0; i < NC; ++i) sumR += RH[i * kSlots].x;
        dT = (QR + kRgas * T * sumR) / (rho0 * CvMixMass);
      } else {
        const double CpMixMass = cpm / MWmix;
        dT = QR / (rho * CpMixMass);
      }
    }
    if (live) team_smem[ev.dst + NC * ev.ds] = ev.f0 >= 0 ? hinv * (dT - team_smem[ev.f0 + NC]) : dT;
  }
  return QR;
}

// G^-1, G = I - hr0 J, by Gauss-Jordan elimination in place with the pivots and the operations of gj_inverse:
// its right half [I] only ever holds non-trivial entries in the columns already eliminated on the left, so
// those columns hold them.  X receives G^-1 (rows of ld) and is the working matrix.  scr: n words for the pivot row, n
// ints for the interchanges.  The whole warp calls it; a
// team with on false passes through without a store.
template <int W>
__device__ __noinline__ void gj_team(int oj, int ox, int osc, double hr0, int n, int lane, bool on) {
  const double* J = team_smem + oj;
  double* X = team_smem + ox;
  double* K = team_smem + osc;
  const int ld = row_ld(n);
  int* perm = (int*)(K + n);
  const bool al = on && lane < n;
  double* Xi = X + (lane < n ? lane : 0) * ld;
  __syncwarp();
  if (al) {
    const double* Ji = J + lane * ld;
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
      double g = -hr0 * Ji[j];
      if (j == lane) g += 1.;
      Xi[j] = g;
    }
    perm[lane] = lane;
  }
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    double vv = (lane >= k && lane < n) ? fabs(Xi[k]) : -1.;
    int r = lane;
#pragma unroll
    for (int off = W / 2; off > 0; off >>= 1) {
      const double ov = __shfl_xor_sync(kFull, vv, off, W);
      const int orr = __shfl_xor_sync(kFull, r, off, W);
      if (ov > vv || (ov == vv && orr < r)) { vv = ov; r = orr; }
    }
    r = __shfl_sync(kFull, r, 0, W);
    if (r < k || r >= n) r = k;   // a NaN column cannot send the pivot outside rows k..n-1
    const double pv = X[r * ld + k];
    const double ipv = pv != 0. ? 1. / pv : 0.;
    __syncwarp();                 // every lane has the pivot before its row moves
    if (al) {
      const double ak = X[k * ld + lane], ar = X[r * ld + lane];
      K[lane] = lane == k ? ipv : ar * ipv;
      if (r != k) X[r * ld + lane] = ak;
      if (lane == 0) {
        const int t = perm[k];
        perm[k] = perm[r];
        perm[r] = t;
      }
    }
    __syncwarp();
    if (al && lane != k) {
      const double fct = Xi[k];
      Xi[k] = 0.;
      int j = 0;
#pragma unroll 1
      for (; j + 4 <= n; j += 4) {
        const double a0 = Xi[j], a1 = Xi[j + 1], a2 = Xi[j + 2], a3 = Xi[j + 3];
        const double k0 = K[j], k1 = K[j + 1], k2 = K[j + 2], k3 = K[j + 3];
        Xi[j] = a0 - fct * k0;
        Xi[j + 1] = a1 - fct * k1;
        Xi[j + 2] = a2 - fct * k2;
        Xi[j + 3] = a3 - fct * k3;
      }
#pragma unroll 1
      for (; j < n; ++j) Xi[j] = Xi[j] - fct * K[j];
    }
    __syncwarp();
    if (al) X[k * ld + lane] = K[lane];
    __syncwarp();
  }
  const int pc = al ? perm[lane] : 0;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const double g = al ? X[i * ld + lane] : 0.;
    __syncwarp();
    if (al) X[i * ld + pc] = g;
    __syncwarp();
  }
}

// gj_team's FP32 counterpart with the lane's row in registers, padded with zero columns to W: the column being eliminated is
// always a[0] and the row moves down by one with each pivot, so that every index is static; rows stay in their
// lanes and `pos` holds their place in the pivoted order (the interchanges move places, not data).
template <int W>
__device__ __noinline__ void gj_reg(int oj, int ox, double hr0, int n, int lane, unsigned gm, bool on) {
  __shared__ __align__(16) float pivot[kTeamThreads];
  float* K = pivot + (int)threadIdx.x / W * W;
  const double* J = team_smem + oj;
  double* X = team_smem + ox;
  const int ld = row_ld(n);
  const bool al = lane < n;
  float a[W];
  const double* Jr = J + (al ? lane : 0) * ld;
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const double g = j < n ? -hr0 * Jr[j] : 0.;
    a[j] = (float)(j == lane ? g + 1. : g);
  }
  int pos = lane, order = 0;       // order: lane k holds the row chosen as pivot k
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    // largest magnitude among the rows not yet pivoted, the first place on ties
    const unsigned key = al && pos >= k ? (__float_as_uint(a[0]) & 0x7fffffffu) + 1u : 0u;
    unsigned mx = key;
#pragma unroll
    for (int off = W / 2; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, off, W));
    unsigned cand = __ballot_sync(kFull, key == mx) & gm;
    if (__any_sync(kFull, (cand & (cand - 1u)) != 0u)) {
      int pm = key == mx ? pos : W;
#pragma unroll
      for (int off = W / 2; off > 0; off >>= 1) pm = min(pm, __shfl_xor_sync(kFull, pm, off, W));
      cand = __ballot_sync(kFull, al && pos == pm) & gm;
    }
    const int r = (__ffs(cand) - 1) & (W - 1);
    const int pr = __shfl_sync(kFull, pos, r, W);
    const bool piv = lane == r;
    if (pos == k) pos = pr;
    if (piv) pos = k;
    if (lane == k) order = r;
    const float fct = a[0];
    __syncwarp();                  // the last pivot row has been read
    if (piv) {
      const float ipv = fct != 0.f ? 1.f / fct : 0.f;
      a[0] = ipv;
#pragma unroll
      for (int j = 1; j < W; ++j) a[j] = a[j] * ipv;
#pragma unroll
      for (int j = 0; j < W; j += 4) *(float4*)(K + j) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
    }
    __syncwarp();
    if (piv) {
      const float c0 = a[0];
#pragma unroll
      for (int j = 0; j + 1 < W; ++j) a[j] = a[j + 1];
      a[W - 1] = c0;
    } else {
      const float k0 = K[0];
#pragma unroll
      for (int j = 0; j + 1 < W; ++j) a[j] = a[j + 1] - fct * K[j + 1];
      a[W - 1] = 0.f - fct * k0;
    }
  }
  // column c is now a[W - n + c]
#pragma unroll
  for (int j = 0; j < W; ++j)
    if (j >= W - n) {
      const int c = __shfl_sync(kFull, order, j - (W - n), W);
      if (on && al) X[pos * ld + c] = (double)a[j];
    }
  __syncwarp();
}

// (M x)_lane with rowdot_ol's two partial sums; M by rows of ld in shared memory, v the lane's x, xs scratch for
// n words.  The whole warp calls it.  Unrolled for W columns so that the loads overlap.
template <int W>
__device__ __noinline__ double rowdot_team(int om, int oxs, double v, int n, int lane) {
  const double* Ml = team_smem + om;
  double* xs = team_smem + oxs;
  __syncwarp();
  if (lane < n) xs[lane] = v;
  __syncwarp();
  double s0 = 0., s1 = 0.;
#pragma unroll
  for (int j = 0; j < W; j += 2) {
    if (j + 1 < n) {
      s0 = __fma_rn(Ml[j], xs[j], s0);
      s1 = __fma_rn(Ml[j + 1], xs[j + 1], s1);
    } else if (j < n) {
      s0 = __fma_rn(Ml[j], xs[j], s0);
    }
  }
  return s0 + s1;
}

// Weighted RMS norms (wrms_ol) of three vectors at once; lane 0 receives the first, lane 1 the second, the others
// the third.
template <int W>
__device__ __noinline__ double wrms3(double x0, double x1, double x2, double e, bool al, int n, int lane) {
  double c0 = al ? x0 * e : 0., c1 = al ? x1 * e : 0., c2 = al ? x2 * e : 0.;
  c0 = __dmul_rn(c0, c0);
  c1 = __dmul_rn(c1, c1);
  c2 = __dmul_rn(c2, c2);
#pragma unroll
  for (int off = W / 2; off > 0; off >>= 1) {
    c0 = __dadd_rn(c0, __shfl_xor_sync(kFull, c0, off, W));
    c1 = __dadd_rn(c1, __shfl_xor_sync(kFull, c1, off, W));
    c2 = __dadd_rn(c2, __shfl_xor_sync(kFull, c2, off, W));
  }
  return sqrt((lane == 0 ? c0 : lane == 1 ? c1 : c2) / double(n));
}

// The solver from a finished request to the next one: the state machine of rounds_advance_kernel on a cell
// whose state R (record layout RL up to the vectors), Jacobian and inverse are in shared memory.  The stages
// run in the machine's order, which never goes back within one visit, each for the teams of the warp that
// reached it, so that two cells on the same path share its instructions; the reductions are the whole warp's.
// Scalars used on every visit are loaded once, the rest read and written in place between barriers.  The
// expressions whose contraction decides the last bit are written out (__fma_rn, __dadd_rn) as the round
// scheme's kernel evaluates them.  act: the team has a finished request.  Returns the next phase.
template <typename LUT, int W>
__device__ __noinline__ int advance_team(int ro, int cell, int lane, unsigned gm, int phase, bool act) {
  const TeamHead& H = team_head();
  const RecLayout& RL = H.R;
  const TeamLayout& TL = H.T;
  const StepOptions& o = H.o;
  const StepArgs& a = H.a;
  const int NC = H.L.nc;
  double* const R = team_smem + ro;
  int* RI = (int*)(R + ND_);
  const int n = NC + 1;
  const bool al = lane < n;
  const double lo = lane < NC ? 0. : o.y_min_T, hi = lane < NC ? 1. : o.y_max_T;
  const int Jr = ro + TL.oj + (al ? lane * TL.ld : 0), Xr = ro + TL.ox + (al ? lane * TL.ld : 0), sc = ro + TL.osc;
  double* const zr = R + RL.oz + lane;   // row i of the lane's column: zr[i * n]
  double* const vr = R + RL.ov + lane;
  double t = R[D_T], tIn = R[D_TMESH], h = R[D_H], hNextStep = R[D_HNEXT], hNordsieck = R[D_HNORD];
  double hScale = R[D_HSCALE];
  unsigned p = RI[I_P], iterOrder = RI[I_ITORDER], orderNext = RI[I_ORDNEXT];
  int hStat = RI[I_HSTAT], oStat = RI[I_OSTAT], status = RI[I_STATUS];
  unsigned nsteps = RI[I_NSTEPS], itConvFail = RI[I_ITCONVFAIL], itErrFail = RI[I_ITERRFAIL];
  unsigned stepJ = RI[I_STEPLASTJ], newtonK = RI[I_NEWTONK];
  int jacChange = RI[I_JACCHANGE];
  double b = al ? R[RL.ob + lane] : 0., va = al ? R[RL.ova + lane] : 0., eps = al ? R[RL.oeps + lane] : 0.;
  enum : int { H_DEC = 0, H_CONST = 1, H_INC = 2 };
  enum : int { O_DEC = 0, O_CONST = 1, O_INC = 2 };
  auto any = [](bool v) { return __any_sync(kFull, v); };
  auto alfa2 = [&](unsigned k) { return k == 4 ? R[D_A24] : (k == 5 ? R[D_A25] : .8); };
  auto Z = [&](unsigned i) { return al ? zr[i * n] : 0.; };
  auto V = [&](unsigned i) { return al ? vr[i * n] : 0.; };
  auto setZ = [&](unsigned i, double v) { if (al) zr[i * n] = v; };
  auto setV = [&](unsigned i, double v) { if (al) vr[i * n] = v; };
  auto wrms = [&](double xv) { return wrms_ol<W>(xv, eps, al, n, kFull); };
  auto clamp = [&](double y) {
    if (al) {
      if (y < lo) y = lo;
      if (y > hi) y = hi;
    }
    return y;
  };
  bool start = false, drive = false, fin = false;
  auto stop = [&](int st) {   // the step ends with the last accepted state
    status = st;
    va = Z(0);
    fin = true;
  };
  __syncwarp();   // every lane has the scalars

  const bool init = act && phase == PH_INIT;
  if (any(init)) {
    // MultiValueSolver::Solve, first call (:445-469)
    const double f = al ? R[RL.of + lane] : 0.;
    const unsigned bad = __ballot_sync(kFull, init && al && (va < lo || va > hi)) & gm;
    if (init) eps = al ? 1. / (o.atol + o.rtol * fabs(va)) : 0.;
    const double wf = wrms(f);
    if (init) {
      if (bad) {
        status = -9;
        fin = true;
      } else {
        const double t0 = a.t0;
        double lo0, hi0;
        if (t0 != 0.) { lo0 = 100. * kMachEpsDouble * fabs(t0); hi0 = fabs(t0); }
        else { lo0 = kMachEpsDouble; hi0 = 1.e-4; }
        double h0 = 0.5 / (wf + kMachEpsFloat);
        if (h0 < lo0) h0 = lo0;
        if (h0 > hi0) h0 = hi0;
        const double tOut = t0 + (a.dt ? a.dt[cell] : a.dt_scalar);
        h0 *= fabs(tOut - t0) / (tOut - t0);
        setZ(0, va);
        setZ(1, f * h0);
        hNordsieck = h0; hNextStep = h0;
        R[D_TOUT] = tOut;
        status = 2;
        start = true;
      }
    }
  }
  if (act && (phase == PH_STAB_CONV || phase == PH_STAB_ERR)) {
    const double f = al ? R[RL.of + lane] : 0.;
    setZ(1, f * h);
    R[D_TSTAB] = tIn;
    if (phase == PH_STAB_CONV) {
      if (nsteps > stepJ + 5u) jacChange = 1;
      if (nsteps != stepJ && itConvFail == 50u) jacChange = 1;
      hNextStep *= R[D_PENDHS];
    } else {
      hStat = H_DEC;
      hNextStep *= hScale;
    }
    drive = true;
  }
  if (act && phase == PH_FINAL) fin = true;

  const bool newton = act && phase == PH_NEWTON;
  bool pred = act && phase == PH_PRED;
  if (any(act && (phase == PH_PRED || phase == PH_JAC || phase == PH_NEWTON))) {
    // MethodGear::FindCorrection after f(vb) (:205-262)
    if (pred) {
      if (nsteps >= stepJ + (unsigned)RI[I_MAXITJ]) jacChange = 1;
    }
    const bool want_j = pred && jacChange;
    if (any(want_j)) {
      const double wf = wrms(al ? R[RL.of0 + lane] : 0.);
      if (want_j) {
        stepJ = nsteps;
        jacChange = 0;
        double hf = 1.e+3 * kMachEpsDouble * fabs(h) * wf * double(n);
        if (hf < 1.e-10) hf = 1.;
        R[D_HF] = hf;
        phase = PH_JAC;   // KernelDense::NumericalJacobian: the n perturbed states next
        pred = false;
      }
    }
    const bool jac = act && phase == PH_JAC && !want_j;
    bool factor = false;
    double hr0f = R[D_HR0];
    if (pred || jac) {
      int factorized = jac ? 0 : RI[I_FACTORIZED];
      if (factorized && iterOrder == 0) factorized = 0;
      factor = !factorized;
      if (factor) hr0f = h * c_gear_r.r[0][p - 1];
    }
    if (any(factor)) {
      if constexpr (sizeof(LUT) == 4) gj_reg<W>(ro + TL.oj, ro + TL.ox, hr0f, n, lane, gm, factor);
      else gj_team<W>(ro + TL.oj, ro + TL.ox, sc, hr0f, n, lane, factor);
      if (factor) {
        const int c = RI[I_CNT0 + CNT_FACT], cj = RI[I_CNT0 + CNT_JAC];
        __syncwarp(gm);
        RI[I_CNT0 + CNT_FACT] = c + 1;
        if (jac) RI[I_CNT0 + CNT_JAC] = cj + 1;
        R[D_HR0] = hr0f;
        RI[I_FACTORIZED] = 1;
      }
    }
    const bool sol = pred || jac || newton;
    bool conv = false, fail = false;
    if (any(sol)) {
      // x = G^-1 rhs; with FP32 factors refined on the FP64 residual (solve_ol)
      const double fl = al ? R[(newton ? RL.of : RL.of0) + lane] : 0.;
      double rhs = al ? __fma_rn(fl, h, -V(1)) : 0.;
      if (newton) rhs -= b;
      double x = rowdot_team<W>(Xr, sc, rhs, n, lane);
      if (sizeof(LUT) == sizeof(float)) {
#pragma unroll 1
        for (int it = 0; it < kRefineR; ++it) {
          const double s = rowdot_team<W>(Jr, sc, x, n, lane);
          const double res = al ? rhs - __fma_rn(-hr0f, s, x) : 0.;
          x += rowdot_team<W>(Xr, sc, res, n, lane);
        }
      }
      if (!al) x = 0.;
      const double r0 = c_gear_r.r[0][p - 1];
      const double cc = r0 * wrms(x);
      if (sol) {
        const int c = RI[I_CNT0 + CNT_SOLVE];
        const double oldCC = R[D_OLDCC];
        if (newton) { b += x; ++newtonK; }
        else { b = x; newtonK = 1; }
        __syncwarp(gm);
        RI[I_CNT0 + CNT_SOLVE] = c + 1;
        if (newtonK > 4u) {
          fail = true;
          newtonK = 4u;   // iterConvergence
        } else if (cc < 1.) {
          conv = true;
        } else if (newtonK > 1 && cc > 2. * oldCC) {
          fail = true;
        } else {
          R[D_OLDCC] = cc;
          double vn = __fma_rn(b, r0, V(0));
          if (al) {
            if (vn < lo) { vn = lo; b = (lo - Z(0)) / r0; }
            if (vn > hi) { vn = hi; b = (hi - Z(0)) / r0; }
          }
          va = vn;
          phase = PH_NEWTON;
        }
      }
    }
    if (fail) {
      // DriverStep convergence-failure branch (:822-847) + recovery (MethodGear.hpp:343-423)
      itConvFail++;
      const int cf = RI[I_CNT0 + CNT_CONVFAIL];
      double alfa2_4 = R[D_A24] - 0.01, alfa2_5 = R[D_A25] - 0.02;
      unsigned ncf = RI[I_NCFOM];
      __syncwarp(gm);
      RI[I_CNT0 + CNT_CONVFAIL] = cf + 1;
      if (itConvFail >= 50u || fabs(h) <= 0.) {
        stop(itConvFail >= 50u ? -5 : -6);
        t = tIn;
      } else {
        double hs = 0.25;
        if (nsteps < 10) hs = 0.1;
        hs = fmax(hs, 0. / fabs(h));
        hStat = H_DEC;
        if (p > 1u) { p -= 1; oStat = O_DEC; }
        if (alfa2_4 < 0.) { alfa2_4 = 0.; RI[I_MAXORD] = 3; if (p > 3) { p = 3; oStat = O_DEC; } }
        if (alfa2_5 < 0.) { alfa2_5 = 0.; RI[I_MAXORD] = 4; if (p > 4) { p = 4; oStat = O_DEC; } }
        R[D_A24] = alfa2_4;
        R[D_A25] = alfa2_5;
        hScale = hs;
        R[D_PENDHS] = hs;
        bool stab = false;
        if (nsteps > 5) {
          ++ncf;
          RI[I_NCFOM] = (int)ncf;
          if (ncf % 5 == 0 && p != 1u) { p = 1; oStat = O_DEC; }
          stab = ncf % 10 == 0 && R[D_TSTAB] != tIn;
        }
        if (stab) {
          phase = PH_STAB_CONV;
        } else {
          if (nsteps > stepJ + 5u) jacChange = 1;
          if (nsteps != stepJ && itConvFail == 50u) jacChange = 1;
          hNextStep *= hs;
          drive = true;
        }
      }
    }
    if (any(conv)) {
      if (conv) {
        // MultiValueStep tail (:1271-1327)
        const double r0 = c_gear_r.r[0][p - 1];
        double bb = b;
        const double vrr = __dmul_rn(bb, r0);
        double x0 = V(0);
        const double x1 = V(1);
        if (al) {
          if (__dadd_rn(x0, vrr) < lo) { bb = lo - Z(0) - x1; x0 = lo - vrr; if (x0 < lo) x0 = lo; }
          if (__dadd_rn(x0, vrr) > hi) { bb = hi - Z(0) - x1; x0 = hi - vrr; if (x0 > hi) x0 = hi; }
        }
        setV(0, __dadd_rn(x0, vrr));
        setV(1, x1 + bb);
        b = bb;
#pragma unroll 1
        for (unsigned i = 2; i <= p; ++i) setV(i, __fma_rn(b, c_gear_r.r[i][p - 1], V(i)));
        const double v1 = div0(V(p) - Z(p), double(p) + 1.);
        setV(p + 1, v1);
        if (iterOrder >= p) setV(p + 2, div0(v1 - Z(p + 1), double(p) + 2.));
      }
      // error test (:876-962)
      double hCur = c_gear_r.Ep[p] * wrms(V(p + 1));
      const bool rej = conv && hCur > 1., acc = conv && !rej;
      if (any(rej)) {
        const double wm = wrms(V(p));
        if (rej) {
          itErrFail++;
          const int ce = RI[I_CNT0 + CNT_ERRFAIL];
          __syncwarp(gm);
          RI[I_CNT0 + CNT_ERRFAIL] = ce + 1;
          if (itErrFail >= 50u || fabs(h) <= 0.) {
            stop(itErrFail >= 50u ? -4 : -6);
            t = tIn;
          } else {
            R[D_HSCALEMAX] = 1.;
            hCur = 0.8 * pow_ol(1. / hCur, 1. / double(p + 1));
            hScale = hCur;
            if (p > 1u) {
              double hMinus = c_gear_r.Ep[p - 1] * wm;
              hMinus = 1. / (hMinus + kMachEpsFloat);
              hMinus = 0.8 * pow_ol(hMinus, 1. / double(p));
              if (hMinus > hCur) { hScale = hMinus; p -= 1; oStat = O_DEC; }
            }
            hScale = fmin(hScale, 0.5);
            hScale = fmax(hScale, 0. / fabs(h));
            hScale = fmax(hScale, 1.e-3);
            if (p == 1u && hScale < 0.1 && nsteps > 10 && tIn != R[D_TSTAB]) {
              phase = PH_STAB_ERR;
            } else {
              hStat = H_DEC;
              hNextStep *= hScale;
              drive = true;
            }
          }
        }
      }
      if (any(acc)) {
        // accepted step (:963-1037)
        if (acc) {
          hNordsieck = h; hNextStep = h;
          orderNext = p; oStat = O_CONST; hStat = H_CONST;
        }
        // MethodGear::ConvergenceRate (:425-516) with the stored Jacobian
        int rate = RI[I_ITCONVRATE];
        if (itErrFail > 0 || itConvFail > 0) rate = 0;
        const bool crt = acc && newtonK > 1;   // newtonK is iterConvergence here
        if (any(crt)) {
          const double s = rowdot_team<W>(Jr, sc, V(0) - Z(0), n, lane);
          const double vq = V(1) - (s * h + Z(1));
          const double normd = wsum_g<W>(kFull, al ? fabs(vq) : 0.);
          const double normf = wsum_g<W>(kFull, al ? fabs(V(1)) : 0.);
          if (crt) {
            if (normd > 3. * normf + .1 && newtonK > 2) {
              if (nsteps > stepJ + 5u) jacChange = 1;
              hScale = 0.5; hStat = H_DEC; hNextStep = h * hScale;
              if (p > 1) { orderNext = p - 1; oStat = O_DEC; }
              rate = 0; itConvFail = 1;
            } else if (normd > normf + 0.1) {
              rate++;
              if (rate >= 5) {
                hScale = 0.8; hStat = H_DEC; hNextStep = h * hScale;
                rate = 0; itConvFail = 1;
              }
              if (nsteps > stepJ + 5u && newtonK > 2) {
                jacChange = 1;
                rate = 0; itConvFail = 1;
              }
            }
          }
        }
        bool ord = false;
        if (acc) {
          if (itErrFail > 0 || itConvFail > 0) {
            itErrFail = 0; itConvFail = 0;
          } else {
            iterOrder++;
            ord = iterOrder > p + 1;
          }
        }
        __syncwarp();
        if (acc) RI[I_ITCONVRATE] = rate;
        if (any(ord)) {
          // NewOrderNewH (:1042-1210): candidates for p - 1, p, p + 1, their powers on three lanes
          const bool lower = p > 1u && oStat != O_INC;
          const bool higher = p < (unsigned)RI[I_MAXORD] && oStat != O_DEC;
          const unsigned pu = p + 2u < 8u ? p + 2u : 7u;
          const double wk = wrms3<W>(V(p), V(p + 1), V(pu), eps, al, n, lane);
          const int k = lane < 2 ? lane : 2;   // 0: p - 1, 1: p, 2: p + 1
          const unsigned po = p - 1u + (unsigned)k;
          double hq = __fma_rn(c_gear_r.Ep[po < 6u ? po : 5u], wk, kMachEpsFloat);
          hq = pow_ol(1. / hq, 1. / double(p + (unsigned)k));
          const double qm = __shfl_sync(kFull, hq, 0, W), qc = __shfl_sync(kFull, hq, 1, W);
          const double qp = __shfl_sync(kFull, hq, 2, W);
          if (ord) {
            const double alfa1 = lower ? alfa2(p - 1) - .05 : 0., alfa3 = higher ? alfa2(p + 1) - .25 : 0.;
            const double a2 = alfa2(p);
            const double hMinus = lower ? alfa1 * qm : 0., hC = a2 * qc, hPlus = higher ? alfa3 * qp : 0.;
            double ar = a2, hw = hC;
            orderNext = p;
            oStat = O_CONST;
            if (hMinus > hC && hMinus > hPlus) {
              ar = alfa1; hw = hMinus; orderNext = p - 1; oStat = O_DEC;
            } else if (!(hC > hMinus && hC > hPlus)) {
              ar = alfa3; hw = hPlus; orderNext = p + 1; oStat = O_INC;
            }
            const int fixedMin = RI[I_FIXEDMIN], im = RI[I_ITMINORD] + 1;
            int consts = RI[I_ITCONST] + 1;
            const double hsm = R[D_HSCALEMAX];
            __syncwarp(gm);
            if (fixedMin) {
              RI[I_ITMINORD] = im;
              if (im < 2000) { ar = a2; hw = hC; orderNext = p; oStat = O_CONST; }
              else RI[I_FIXEDMIN] = 0;
            }
            hScale = (.75 / ar) * hw;
            if (hScale < 1.2) {
              hScale = 1.; hStat = H_CONST; orderNext = p; oStat = O_CONST; hNextStep = h;
            } else {
              consts = 0;
              hScale = fmin(hScale, hsm);
              hStat = H_INC;
              hNextStep = h * hScale;
            }
            RI[I_ITCONST] = consts;
            if (consts > 500 || (nsteps % 1000 == 0 && nsteps != 0 && (fabs(h) < 1.e-7 || fabs(h) < 1.e-5 * t))) {
              if (p > 1u) {
                RI[I_FIXEDMIN] = 1;
                RI[I_ITMINORD] = 0;
                orderNext = 1; oStat = O_DEC;
                hScale = 0.5; hNextStep = h * hScale; hStat = H_DEC;
              }
            }
          }
        }
        if (acc) {
#pragma unroll 1
          for (unsigned i = 1; i <= p + 2; ++i) setZ(i, V(i));
          setZ(0, clamp(V(0)));
          nsteps++;
          const double tOut = R[D_TOUT];
          if (tOut == t) {
            va = Z(0);
            fin = true;
          } else if (tOut < t) {
            // Interpolation (:687-706); the RHS at tOut then sets QR (:599-611)
            const double hp = (tOut - t) / hNordsieck;
            double yv = Z(0);
            if (hp != 0.) {
              double hr = 1.;
#pragma unroll 1
              for (unsigned i = 1; i <= p; ++i) {
                hr *= hp;
                yv = __fma_rn(Z(i), hr, yv);
              }
              yv = clamp(yv);
            }
            va = yv;
            phase = PH_FINAL;
          } else {
            start = true;
          }
        }
      }
    }
  }
  // MultiValueSolver::Solve loop (:532-560) + DriverStep prologue (:753-776)
  if (start && nsteps >= (unsigned)o.max_steps) { stop(-1); start = false; }
  if (start) eps = al ? 1. / (o.atol + o.rtol * fabs(Z(0))) : 0.;
  // |z0| eps <= 1 / rtol: the test for a too small tolerance (MachEps wrms(z0) > 1) cannot hold above this rtol
  if (!(o.rtol > 1.e-14)) {
    const double w0 = wrms(Z(0));
    if (start && kMachEpsDouble * w0 > 1.) { stop(-2); start = false; }
  }
  if (start) {
    tIn = t;
    itConvFail = 0; itErrFail = 0;
    if (oStat != O_CONST || hStat != H_CONST) iterOrder = 0;
    p = orderNext;
    oStat = O_CONST;
    R[D_HSCALEMAX] = nsteps < 10 ? 1000. : (nsteps > 10 && nsteps < 20) ? 10. : 2.;
    drive = true;
  }
  if (drive) {
    // DriverStep while(1) body up to FindCorrection (:778-820, :1212-1266)
    if (hStat != H_CONST) {
      hScale = hNextStep / hNordsieck;
      double hr = 1.;
#pragma unroll 1
      for (unsigned i = 1; i <= p; ++i) {
        hr *= hScale;
        setZ(i, Z(i) * hr);
      }
      setZ(0, clamp(Z(0)));
      iterOrder = 0;
      hStat = H_CONST;
    }
    h = hNextStep;
    hNordsieck = hNextStep;
    t = tIn + h;
    if (t == tIn) {
      stop(-6);
    } else {
      // MultiValueStep prediction v = D z with min/max handling, then vb = CheckConstraints(v0); the rows
      // above p are zero, so the whole triangle may run
      double wv[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) wv[i] = (i <= (int)p) ? Z(i) : 0.;
      const double z0 = wv[0];
#pragma unroll
      for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = 4; j >= 0; --j)
          if (j >= i) wv[j] += wv[j + 1];
      if (al) {
        if (wv[0] < lo && fabs(wv[0] - lo) * eps < double(n)) {
          wv[1] = lo - z0;
          wv[0] = lo;
#pragma unroll
          for (int i = 2; i < 6; ++i) wv[i] = 0.;
        }
        if (wv[0] > hi && fabs(wv[0] - hi) * eps < double(n)) {
          wv[1] = hi - z0;
          wv[0] = hi;
#pragma unroll
          for (int i = 2; i < 6; ++i) wv[i] = 0.;
        }
      }
#pragma unroll
      for (int i = 0; i < 6; ++i)
        if (i <= (int)p) setV(i, wv[i]);
      if (al) R[RL.ovb + lane] = clamp(wv[0]);
      phase = PH_PRED;
    }
  }
  if (any(fin)) {
    // utilities.H:153-200 and the scatter of chemistry_DI.H:221-235
    const double s = wsum_g<W>(kFull, lane < NC ? va : 0.);
    if (fin) {
      if (lane < NC) a.Y[(long)lane * a.ld + cell] = va / s;
      if (o.energy && lane == NC) a.T[cell] = va;
      if (lane == 0) {
        if (a.Q) a.Q[cell] = R[D_QR];
        if (a.status) a.status[cell] = status;
        if (a.nsteps) a.nsteps[cell] = (int)nsteps;
      }
      phase = PH_DONE;
    }
  }
  __syncwarp();
  if (act) {   // the state back: every lane writes the same scalars
    if (al) {
      R[RL.ob + lane] = b;
      R[RL.ova + lane] = va;
      R[RL.oeps + lane] = eps;
    }
    R[D_T] = t; R[D_TMESH] = tIn; R[D_H] = h; R[D_HNEXT] = hNextStep; R[D_HNORD] = hNordsieck;
    R[D_HSCALE] = hScale;
    RI[I_STATUS] = status; RI[I_P] = (int)p; RI[I_ITORDER] = (int)iterOrder; RI[I_ORDNEXT] = (int)orderNext;
    RI[I_HSTAT] = hStat; RI[I_OSTAT] = oStat; RI[I_JACCHANGE] = jacChange; RI[I_NSTEPS] = (int)nsteps;
    RI[I_ITCONVFAIL] = (int)itConvFail; RI[I_ITERRFAIL] = (int)itErrFail;
    RI[I_STEPLASTJ] = (int)stepJ; RI[I_NEWTONK] = (int)newtonK; RI[I_CNT0 + CNT_STEPS] = (int)nsteps;
  }
  __syncwarp();
  return phase;
}

}  // namespace

// The reaction step of a.ncells cells.  Teams take their first cell by index, spread over the SMs, and the next
// ones from the queue.
template <typename LUT, int W>
__global__ void __launch_bounds__(kTeamThreads, 1)
    team_kernel(const __grid_constant__ MechLayout Lp, const unsigned char* __restrict__ mech_gmem,
                const __grid_constant__ StepOptions o, const __grid_constant__ StepArgs a, int teams, int* queue) {
  __shared__ int t_phase[kSlots], t_jcol[kSlots], t_next[kSlots], s_code[kSlots];
  __shared__ double t_rho[kSlots];
  const int NC = Lp.nc, n = NC + 1;
  const int wl = threadIdx.x & 31, lane = threadIdx.x & (W - 1);
  const int team = threadIdx.x / W;
  const bool own = team < teams;   // warps beyond the teams only evaluate
  if (threadIdx.x == 0) {
    TeamHead& H = *(TeamHead*)team_smem;
    H.L = Lp;
    H.T = team_layout(n);
    H.R = rec_layout(n, sizeof(LUT) == 8);
    H.S = slot_layout(Lp);
    H.o = o;
    H.a = a;
    H.Md = (const double*)mech_gmem;
    H.Mi = (const int*)(mech_gmem + (size_t)Lp.n_double * sizeof(double));
  }
  if (threadIdx.x < kSlots) {
    t_phase[threadIdx.x] = PH_DONE;
    t_jcol[threadIdx.x] = t_next[threadIdx.x] = 0;
    t_rho[threadIdx.x] = 0.;
  }
  __syncthreads();
  const TeamLayout& sT = team_head().T;
  const RecLayout& sR = team_head().R;
  const int base = team_head().S.total, ro = base + (own ? team : 0) * sT.total;
  double* const R = team_smem + ro;
  int* const RI = (int*)(R + ND_);
  const unsigned gm = W == 32 ? kFull : (0xffffu << (threadIdx.x & 16));
  const bool al = lane < n;
  // a team that never gets a cell passes through its warp's visits: valid state, order 1
  if (own) {
    for (int i = lane; i < sT.total; i += W) R[i] = 0.;
    __syncwarp();
    RI[I_P] = 1;
    if (lane == NC) R[sR.ova + lane] = 1000.;
  }
  __syncwarp();
  const int total = (int)a.ncells;
  const int stride = teams * (int)gridDim.x;
  const long max_requests = 4L * (long)o.max_steps * (NC + 10) + 64;
  int w = team * gridDim.x + blockIdx.x, cell = 0, phase = PH_DONE, crhs = 0;
  long req = 0;
  bool idle = !own;
  for (;;) {
    // ---- a finished team takes its next cell ----
    while (phase == PH_DONE && !idle) {
      if (w >= total) {
        idle = true;
        break;
      }
      cell = w;
      req = 0;
      crhs = 0;
      if (lane == 0) t_rho[team] = a.rho ? a.rho[cell] : 0.;
      const double Tc = a.T[cell];
      double y = lane < NC ? a.Y[(long)lane * a.ld + cell] : 0.;
      const bool skip = !(Tc > o.tmin_chem);   // chemistry_DI.H:92-96: the cell is skipped, its Y renormalised
      if (!skip && y < 0.) y = 0.;
      __syncwarp(gm);
      if (lane < NC) R[sT.osc + lane] = y;
      __syncwarp(gm);
      double s = 0.;
      for (int i = 0; i < NC; ++i) s += R[sT.osc + i];
      if (skip) {
        if (lane < NC) a.Y[(long)lane * a.ld + cell] = y / s;
        if (lane == 0) {
          if (a.status) a.status[cell] = 0;
          if (a.nsteps) a.nsteps[cell] = 0;
        }
        if (a.counters && lane < NCNT) a.counters[(long)cell * NCNT + lane] = 0;
      } else {
        if (lane < NC) R[sR.ova + lane] = y / s;
        if (lane == NC) R[sR.ova + lane] = Tc;
        // solver reset (MultiValueSolver.hpp:367-420), as rounds_init_kernel
        R[D_T] = a.t0; R[D_T0] = a.t0; R[D_TOUT] = a.t0; R[D_TMESH] = a.t0; R[D_TSTAB] = a.t0;
        R[D_H] = 0.; R[D_HNEXT] = 0.; R[D_HNORD] = 0.; R[D_HSCALE] = 0.; R[D_HSCALEMAX] = 1000.;
        R[D_A24] = o.alfa2_4; R[D_A25] = o.alfa2_5; R[D_QR] = 0.; R[D_OLDCC] = 0.; R[D_HF] = 0.;
        R[D_PENDHS] = 0.; R[D_HR0] = 0.;
        unsigned mij = 20u + 5u * (unsigned)(n - 3);
        if (mij > 50u && n < 80) mij = 50u;
        for (int i = 0; i < NI_; ++i) RI[i] = 0;
        RI[I_STATUS] = 1; RI[I_P] = 1; RI[I_ORDNEXT] = 1; RI[I_MAXITJ] = (int)mij; RI[I_HSTAT] = 1;
        RI[I_OSTAT] = 1; RI[I_JACCHANGE] = 1; RI[I_MAXORD] = o.maximum_order;
        phase = PH_INIT;
      }
      __syncwarp(gm);
      if (phase == PH_DONE) {
        if (lane == 0) w = atomicAdd(queue, 1);
        w = __shfl_sync(gm, w, 0, W) + stride;
      }
    }
    if (own && lane == 0) t_phase[team] = phase;
    if (__syncthreads_and(idle)) break;
    // ---- the evaluation slots: plain requests, then Jacobian columns (warp 0, lane = team, then lane = slot) ----
    if (threadIdx.x < kSlots) {
      const int ph = t_phase[wl];
      const bool jac = ph == PH_JAC, plain = ph != PH_DONE && !jac;
      const unsigned mp = __ballot_sync(kFull, plain);
      const int np = __popc(mp);
      s_code[wl] = -1;
      __syncwarp();
      if (plain) s_code[__popc(mp & ((1u << wl) - 1u))] = wl | 255 << 8;
      const int first = t_jcol[wl], rem = jac ? n - first : 0;
      int pre = rem;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(kFull, pre, off);
        if (wl >= off) pre += v;
      }
      pre += np - rem;             // the first slot of this team's columns
      int take = kSlots - pre;
      take = take < 0 ? 0 : take < rem ? take : rem;
      for (int c = 0; c < take; ++c) s_code[pre + c] = wl | (first + c) << 8;
      t_next[wl] = first + take;
      __syncwarp();
      const int code = s_code[wl];
      double hj = 0.;
      if (code >= 0 && (code >> 8) != 255) {
        // KernelDense::NumericalJacobian, constrained branch (KernelDense.hpp:111-193), as jacobian_column
        const double* Rb = team_smem + base + (code & 255) * sT.total;
        const int col = code >> 8;
        const double yh = Rb[sR.ovb + col], ej = Rb[sR.oeps + col], hf = Rb[D_HF];
        const double aa = fabs(yh), bb = fabs(1. / ej);
        hj = sqrt(kMachEpsDouble) * (aa > bb ? aa : bb);
        hj = fmax(hj, hf / ej);
        hj = fmax(hj, sqrt(kTinyFloat));
        if (yh + hj > (col < n - 1 ? 1. : o.y_max_T)) hj = -hj;
      }
      double* SS = team_smem + team_head().S.sc + wl;
      SS[SS_HJ * kSlots] = hj;
      SS[SS_HINV * kSlots] = 1. / hj;
    }
    __syncthreads();
    // ---- right-hand sides; an empty slot repeats slot 0 without a store (some slot is always taken) ----
    {
      const int code = s_code[wl];
      const int use = code >= 0 ? code : (s_code[0] | 255 << 8);
      const int tm = use & 255, col = use >> 8, ph = t_phase[tm];
      const int Rb = base + tm * sT.total;
      const bool jc = code >= 0 && col != 255;
      Eval ev;
      ev.y = Rb + (ph == PH_PRED || ph == PH_JAC ? sR.ovb : ph == PH_STAB_CONV || ph == PH_STAB_ERR ? sR.oz : sR.ova);
      ev.col = col;
      ev.dst = jc ? Rb + sT.oj + col : Rb + (ph == PH_PRED ? sR.of0 : sR.of);
      ev.ds = jc ? sT.ld : 1;
      ev.f0 = jc ? Rb + sR.of0 : -1;
      const double q = rhs_slots(ev, code >= 0, a.p, o.energy, t_rho[tm]);
      if (threadIdx.x < kSlots && code >= 0 && (!jc || col == n - 1)) team_smem[Rb + D_QR] = q;   // the last column's, as there
    }
    __syncthreads();
    // ---- the solver ----
    if (own) {   // whole warps: a warp's teams are both owned or the second passes through
      bool act = phase != PH_DONE && !idle;
      if (act) {
        if (phase == PH_JAC) {
          const int next = t_next[team];
          act = next == n;
          if (lane == 0) t_jcol[team] = act ? 0 : next;
          if (act) {
            const int c = RI[I_CNT0 + CNT_JAC_RHS];
            __syncwarp(gm);
            RI[I_CNT0 + CNT_JAC_RHS] = c + n;
          }
        } else {
          ++crhs;
        }
      }
      __syncwarp();
      const int was = phase;
      phase = advance_team<LUT, W>(ro, cell, lane, gm, phase, act);
      if (act && ++req > max_requests && phase != PH_DONE) {   // as the round limit: status -1, the last accepted state
        const double va = al ? R[sR.oz + lane] : 0.;
        const double s = wsum_g<W>(gm, lane < NC ? va : 0.);
        if (lane < NC) a.Y[(long)lane * a.ld + cell] = va / s;
        if (o.energy && lane == NC) a.T[cell] = va;
        if (lane == 0) {
          if (a.Q) a.Q[cell] = R[D_QR];
          if (a.status) a.status[cell] = -1;
          if (a.nsteps) a.nsteps[cell] = RI[I_NSTEPS];
        }
        phase = PH_DONE;
      }
      if (phase == PH_DONE && was != PH_DONE) {
        if (a.counters && lane < NCNT)
          a.counters[(long)cell * NCNT + lane] = lane == CNT_RHS ? crhs : RI[I_CNT0 + lane];
        if (lane == 0) w = atomicAdd(queue, 1);
        w = __shfl_sync(gm, w, 0, W) + stride;
      }
      __syncwarp();
    }
  }
}

namespace {

constexpr size_t kTeamSmem = 222 * 1024;   // of 227 KB: the static arrays and the layouts take the rest

// Teams of a block: what the SM's shared memory holds beside the slots, whole warps, at most one per slot and
// per W threads; 0 when not even one warp's teams fit.
inline int team_count(const MechLayout& L, int w) {
  const size_t slots = (size_t)slot_layout(L).total * sizeof(double), per = (size_t)team_layout(L.nc + 1).total * sizeof(double);
  if (slots + per * (32 / w) > kTeamSmem) return 0;
  long k = (long)((kTeamSmem - slots) / per);
  if (k > kSlots) k = kSlots;
  if (k > kTeamThreads / w) k = kTeamThreads / w;
  return (int)(k - k % (32 / w));
}

template <typename LUT, int W>
cudaError_t team_launch(const MechLayout& L, const unsigned char* mech_gmem, const StepOptions& o, const StepArgs& a,
                        int* queue, int sm_count, cudaStream_t stream) {
  int teams = team_count(L, W);
  if (teams <= 0) return cudaErrorInvalidValue;
  const long grid = a.ncells < sm_count ? a.ncells : sm_count;
  const long need = (a.ncells + grid - 1) / grid;   // cells a block
  if (need < teams) teams = (int)((need + 32 / W - 1) / (32 / W) * (32 / W));
  const size_t smem = sizeof(double) * ((size_t)slot_layout(L).total + (size_t)teams * team_layout(L.nc + 1).total);
  // the same value at every call: another thread may launch the kernel with another size at the same time
  cudaError_t e =
      cudaFuncSetAttribute(team_kernel<LUT, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTeamSmem);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(queue, 0, sizeof(int), stream);
  if (e != cudaSuccess) return e;
  team_kernel<LUT, W><<<(unsigned)grid, kTeamThreads, smem, stream>>>(L, mech_gmem, o, a, teams, queue);
  return cudaGetLastError();
}

}  // namespace
}  // namespace lsg
