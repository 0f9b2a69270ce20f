// Plain FP64 reaction step: warp per cell, the reference's algorithm operation
// for operation.  This translation unit is compiled with FMA contraction off
// (-fmad=false) so products and sums round exactly as the CPU code does.
#include "lsg_kernels.h"
#include "lsg_warp_fp64.cuh"

#include <math_constants.h>

namespace lsg {
namespace {

// One block an SM, which shares the staged mechanism: up to 16 warps of 128 registers, or up to 8 of 255, whose solver
// keeps its state in registers (plan_warps).
constexpr int kPlainWarps = 16, kPlainFew = 8;

// Layout, tables and the block's cell counter; false after a staging time-out.
__device__ __forceinline__ int& warp_next() {
  __shared__ int next;
  return next;
}
template <bool kStaged>
__device__ __forceinline__ bool warp_setup(const MechLayout& L, const unsigned char* mech_gmem, int* err) {
  __shared__ __align__(8) uint64_t mbar;
  if (threadIdx.x == 0) {
    warp_layout() = L;
    warp_mech().gmem = mech_gmem;
    warp_next() = 0;
  }
  if constexpr (kStaged) return stage_tables(warp_smem, mech_gmem, L, L.warp_int, &mbar, err);
  __syncthreads();
  return true;
}
// The warp's work space (in doubles) in the dynamic shared memory
template <bool kStaged>
__device__ __forceinline__ int warp_wofs(const MechLayout& L, int ws_doubles) {
  return (kStaged ? (int)(staged_bytes(L, L.warp_int) / 8u) : 0) + (int)(threadIdx.x >> 5) * ws_doubles;
}
// The warp's next cell: a block owns one cell of every gridDim in a row, its warps take them in turn.  Which one of the
// row changes from row to row without a pattern, for the cells' cost has one: with the same place in every row, a mesh
// whose lines are a multiple of gridDim long put the hot columns on a few blocks (296 x 40 H2/CO cells, ten hot columns,
// 26.0 ms then, 10.2 now, 8.8 for the same cells shuffled).  A counter in global memory would do it too, but calls on
// several streams, captured ones among them, could not share one.
__device__ __forceinline__ long warp_cell() {
  int k = 0;
  if ((threadIdx.x & 31) == 0) k = atomicAdd(&warp_next(), 1);
  k = __shfl_sync(kFull, k, 0);
  unsigned h = (unsigned)k * 0x9e3779b9u;   // bits of k mixed; 0 for the first row
  h = (h ^ (h >> 15)) * 0x2c1b3c6du;
  h ^= h >> 13;
  unsigned b = blockIdx.x + __umulhi(h, gridDim.x);
  if (b >= gridDim.x) b -= gridDim.x;
  return (long)gridDim.x * k + b;
}
}  // namespace

// solvers/laminarSMOKE/unsteady/chemistry_DI.H:92-235: gather, clip and
// renormalise, integrate, renormalise, scatter; Q is the reactor's QR after
// the solve (chemistry_DI.H:168).
template <bool kStaged, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, 1)
plain_warp_kernel(MechLayout L, const unsigned char* __restrict__ mech_gmem, StepOptions o, StepArgs a,
                  int* err) {
  if (!warp_setup<kStaged>(L, mech_gmem, err)) return;
  const int lane = threadIdx.x & 31;
  const int wofs = warp_wofs<kStaged>(L, warp_ws_doubles(L));
  const WarpWS W = carve_ws((double*)warp_smem + wofs, L);
#pragma unroll 1
  for (long cell; (cell = warp_cell()) < a.ncells;) {
  __syncwarp();
  if (lane == 0) {
    W.SC[0] = 0.; W.SC[1] = 0.; W.SC[2] = a.p; W.SC[3] = o.energy ? 1. : 0.;
    W.SC[4] = a.rho ? a.rho[cell] : 0.;
    W.SC[5] = div_w(a.p, kRgas);
  }
  __syncwarp();

  const int NC = L.nc;
  const int ne = NC + 1;
  double yl = 0.;
  if (lane < NC) yl = a.Y[(size_t)lane * a.ld + cell];
  const double Tc = a.T[cell];
  if (lane == NC) yl = Tc;
  double yf = yl;
  int st = 0;
  long long nsteps = 0;
  if (Tc > o.tmin_chem) {
    double y0 = yl;
    if (lane < NC && y0 < 0.) y0 = 0.;
    const double sum = sum_warp((int)(W.X - (double*)warp_smem), lane < NC ? y0 : 0., NC);
    if (lane < NC) y0 = div_w(y0, sum);
    GearWarpT<false, kStaged> g;
    g.W = W;
    g.wofs = wofs;
    g.lane = lane;
    g.ne = ne;
    g.active = lane < ne;
    g.alfa2_4 = o.alfa2_4;
    g.alfa2_5 = o.alfa2_5;
    g.maximum_order = (unsigned)o.maximum_order;
    g.max_number_steps = (unsigned)o.max_steps;
    g.abs_tol = o.atol;
    g.rel_tol = o.rtol;
    g.minv = lane < NC ? 0. : o.y_min_T;
    g.maxv = lane < NC ? 1. : o.y_max_T;
    g.b = g.deltab = g.f = g.va = g.vb = g.y = 0.;
    g.eps = 0.;
    g.set_initial_conditions(a.t0, y0);
    const double dtc = a.dt ? a.dt[cell] : a.dt_scalar;
    st = g.solve_to(a.t0 + dtc);
    yf = g.y;
    nsteps = g.cnt[CNT_STEPS];
    if (lane == 0) {
      if (a.Q) a.Q[cell] = g.W.SC[1];
      if (a.counters)
        for (int k = 0; k < NCNT; ++k) a.counters[(size_t)cell * NCNT + k] = g.cnt[k];
    }
  } else if (lane == 0 && a.counters) {
    for (int k = 0; k < NCNT; ++k) a.counters[(size_t)cell * NCNT + k] = 0;
  }
  // solvers/laminarSMOKE/utilities.H:153-200
  const double s = sum_warp((int)(W.X - (double*)warp_smem), lane < NC ? yf : 0., NC);
  if (lane < NC) {
    yf = div_w(yf, s);
    a.Y[(size_t)lane * a.ld + cell] = yf;
  }
  if (lane == NC && o.energy) a.T[cell] = yf;
  if (lane == 0) {
    if (a.status) a.status[cell] = st;
    if (a.nsteps) a.nsteps[cell] = (int)nsteps;
  }
  }
}

// ---------------------------------------------------------------------------
// DRG-reduced reaction step (solvers/laminarSMOKE/unsteady/chemistry_DRG.H with
// DRG.hpp), one warp per cell.  Per cell above min_T: the directed-relation-graph
// analysis at the cell's state, then the reduced system (the important species
// and T; the other species keep their mass fractions, the dropped reactions have
// zero rate) integrated by a fresh solver from t0 to t0 + dt, the mass fractions
// normalised after the step.
// ---------------------------------------------------------------------------

// Each cell's epsilon: the first band whose temperature is above the cell's; a
// cell above every band keeps the previous analysed cell's epsilon, and cells at
// or below min_T are not analysed (chemistry_DRG.H).  The carry-over runs in cell
// order, so one thread scans the batch.
__global__ void drg_eps_kernel(long ncells, const double* __restrict__ T, DrgArgs d) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  double eps = d.epsilon0;
  for (long i = 0; i < ncells; ++i) {
    const double t = T[i];
    if (t > d.min_T)
      for (int b = 0; b < d.nbands; ++b)
        if (t < d.band_T[b]) {
          eps = d.band_eps[b];
          break;
        }
    d.eps[i] = eps;
  }
}

template <bool kStaged, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, 1)
drg_warp_kernel(MechLayout L, const unsigned char* __restrict__ mech_gmem, StepOptions o, StepArgs a, DrgArgs d,
                int* err) {
  if (!warp_setup<kStaged>(L, mech_gmem, err)) return;
  const MechLayout& sL = warp_layout();
  const MechView M = warp_tables<kStaged>(sL);
  const int lane = threadIdx.x & 31;
  const int wofs = warp_wofs<kStaged>(L, drg_ws_doubles(L));
  const WarpWS W = carve_ws((double*)warp_smem + wofs, L);
#pragma unroll 1
  for (long cell; (cell = warp_cell()) < a.ncells;) {
  __syncwarp();
  if (lane == 0) {
    W.SC[0] = 0.; W.SC[1] = 0.; W.SC[2] = a.p; W.SC[3] = o.energy ? 1. : 0.; W.SC[4] = 0.; W.SC[5] = div_w(a.p, kRgas);
  }
  __syncwarp();
  const int NC = L.nc, NR = L.nr;
  const double Tc = a.T[cell];
  const double om = lane < NC ? a.Y[(size_t)lane * a.ld + cell] : 0.;
  int st = 0, nsp = 0, nrx = 0;
  if (Tc > d.min_T) {
    // ---- analysis (DRG.hpp:150-273): rates at the cell's state, then the search from the key species ----
    rhs_warp<false, kStaged>(wofs, lane < NC ? om : Tc, Tc);   // W.NET: net rates of progress
    __syncwarp();
    const double eps = d.eps[cell];
    double den = 0.;   // sum_k |nu_ki r_k|, reactions in ascending order
    for (int k = 0; k < NR; ++k) {
      const double nki = lane < NC ? drg_net_nu(M, sL, k, lane) : 0.;
      if (nki != 0.) den += fabs(nki * W.NET[k]);
    }
    int* Qu = (int*)W.J;   // the queue (at most nkey + NC entries; J and G are free until the solve)
    unsigned imp = 0u;
    int qlen = 0;
    for (int t = 0; t < d.nkey; ++t) {
      if (lane == 0) Qu[qlen] = d.key[t];
      ++qlen;
      imp |= 1u << d.key[t];
    }
    __syncwarp();
    for (int head = 0; head < qlen; ++head) {
      const int q = Qu[head];
      const double denq = __shfl_sync(kFull, den, q);
      double num = 0.;
      for (int k = 0; k < NR; ++k) {
        const double nq = drg_net_nu(M, sL, k, q);
        if (nq == 0.) continue;
        const double nkj = lane < NC ? drg_net_nu(M, sL, k, lane) : 0.;
        if (nkj != 0.) num += fabs(nq * W.NET[k]);
      }
      const bool add = lane < NC && !((imp >> lane) & 1u) && num / (1.e-64 + denq) > eps;
      const unsigned m = __ballot_sync(kFull, add);
      if (add) Qu[qlen + __popc(m & ((1u << lane) - 1u))] = lane;   // appended in ascending species order
      qlen += __popc(m);
      imp |= m;
      __syncwarp();
    }
    // a reaction is dropped when one of its species (non-zero net coefficient) was not reached
    int ndrop = 0;
    for (int k = lane; k < NR; k += 32) {
      bool keep = true;
      const int* pp = M.I(L.prod_ptr);
      const int* psp = M.I(L.prod_sp);
      const int* rpp = M.I(L.reac_ptr);
      const int* rsp = M.I(L.reac_sp);
      for (int q = pp[k]; q < pp[k + 1]; ++q) {
        const int s = psp[q];
        if (!((imp >> s) & 1u) && drg_net_nu(M, sL, k, s) != 0.) keep = false;
      }
      for (int q = rpp[k]; q < rpp[k + 1]; ++q) {
        const int s = rsp[q];
        if (!((imp >> s) & 1u) && drg_net_nu(M, sL, k, s) != 0.) keep = false;
      }
      W.DROP[k] = keep ? 0 : 1;
      ndrop += keep ? 0 : 1;
    }
    for (int off = 16; off > 0; off >>= 1) ndrop += __shfl_xor_sync(kFull, ndrop, off);
    __syncwarp();   // the mask is complete before the reduced system reads it
    // ---- the reduced system: lane l < ni owns the l-th important species, lane ni owns T ----
    const int ni = __popc(imp);
    int sp = NC;
    if (lane < ni) {
      unsigned mm = imp;
      for (int t = 0; t < lane; ++t) mm &= mm - 1u;
      sp = __ffs(mm) - 1;
    }
    const int pos = (lane < NC && ((imp >> lane) & 1u)) ? __popc(imp & ((1u << lane) - 1u)) : -1;
    const double ys = __shfl_sync(kFull, om, sp < NC ? sp : 0);
    const double y0 = lane < ni ? ys : (lane == ni ? Tc : 0.);
    GearWarpT<true, kStaged> g;
    g.W = W;
    g.wofs = wofs;
    g.lane = lane;
    g.ne = ni + 1;
    g.active = lane < ni + 1;
    g.drg_ni = ni;
    g.drg_nc = NC;
    g.drg_sp = sp;
    g.drg_pos = pos;
    g.drg_omega = om;
    // a fresh solver object per cell (chemistry_DRG.H): its own order-selection state and step limit
    g.alfa2_4 = 0.8;
    g.alfa2_5 = 0.8;
    g.maximum_order = 5u;
    g.max_number_steps = 500000u;
    if (cell == 0 || !d.first_cell_options_only) {
      g.abs_tol = o.atol;
      g.rel_tol = o.rtol;
      g.minv = lane < ni ? 0. : 200.;
      g.maxv = lane < ni ? 1. : 6000.;
      g.unconstrained = false;
    } else {   // the solver's own defaults (MultiValueSolver.hpp:41-43), no constraints
      g.abs_tol = 1.e-10;
      g.rel_tol = 100. * kMachEpsFloat;
      g.minv = -CUDART_INF;
      g.maxv = CUDART_INF;
      g.unconstrained = true;
    }
    g.b = g.deltab = g.f = g.va = g.vb = g.y = 0.;
    g.eps = 0.;
    g.set_initial_conditions(a.t0, y0);
    const double dtc = a.dt ? a.dt[cell] : a.dt_scalar;
    st = g.solve_to(a.t0 + dtc);
    // ---- scatter: the kept species' start values, the integrated ones, T; normalised ----
    const double yv = __shfl_sync(kFull, g.y, pos >= 0 ? pos : 0);
    const double Tf = __shfl_sync(kFull, g.y, ni);
    double yf = pos >= 0 ? yv : om;
    const double sum = sum_warp((int)(W.X - (double*)warp_smem), lane < NC ? yf : 0., NC);
    if (lane < NC) {
      yf = div_w(yf, sum);
      a.Y[(size_t)lane * a.ld + cell] = yf;
    }
    if (lane == 0) {
      if (o.energy) a.T[cell] = Tf;
      if (a.Q) a.Q[cell] = W.SC[1];
      if (a.counters)
        for (int k = 0; k < NCNT; ++k) a.counters[(size_t)cell * NCNT + k] = g.cnt[k];
      if (a.nsteps) a.nsteps[cell] = (int)g.cnt[CNT_STEPS];
    }
    nsp = ni;
    nrx = NR - ndrop;
  } else if (lane == 0) {
    if (a.counters)
      for (int k = 0; k < NCNT; ++k) a.counters[(size_t)cell * NCNT + k] = 0;
    if (a.nsteps) a.nsteps[cell] = 0;
  }
  if (lane == 0) {
    if (a.status) a.status[cell] = st;
    if (d.n_species) d.n_species[cell] = nsp;
    if (d.n_reactions) d.n_reactions[cell] = nrx;
  }
  }
}

// Standalone right-hand side, one warp per state (same arithmetic as inside the step).
template <bool kStaged, int kWarps>
__global__ void __launch_bounds__(kWarps * 32, 1)
rhs_warp_kernel(MechLayout L, const unsigned char* __restrict__ mech_gmem, long ncells, const double* __restrict__ y,
                double* __restrict__ dy, long ld, double p, int energy, double* qr, int* err) {
  if (!warp_setup<kStaged>(L, mech_gmem, err)) return;
  const int lane = threadIdx.x & 31;
  const int wofs = warp_wofs<kStaged>(L, warp_ws_doubles(L));
  const WarpWS W = carve_ws((double*)warp_smem + wofs, L);
  const int NC = L.nc;
#pragma unroll 1
  for (long cell; (cell = warp_cell()) < ncells;) {
    __syncwarp();
    if (lane == 0) {
      W.SC[0] = 0.; W.SC[1] = 0.; W.SC[2] = p; W.SC[3] = energy ? 1. : 0.; W.SC[4] = 0.; W.SC[5] = div_w(p, kRgas);
    }
    __syncwarp();
    const double yl = lane <= NC ? y[(size_t)lane * ld + cell] : 0.;
    const double T = __shfl_sync(kFull, yl, NC);
    const double d = rhs_warp<false, kStaged>(wofs, yl, T);
    if (lane <= NC) dy[(size_t)lane * ld + cell] = d;
    if (lane == 0 && qr) qr[cell] = W.SC[1];
  }
}

namespace {
// Largest dynamic shared memory of the kernels above beside their static one
constexpr size_t kPlainSmem = 227 * 1024 - 1024;

// The form takes a mechanism when the tables without the packed copies leave room for four work spaces.
size_t form_bytes(const MechLayout& L, size_t extra) {
  const int n = L.nc + 1;
  auto even = [](size_t x) { return (x + 1) & ~(size_t)1; };
  const size_t ws = 8 * 32 * 2 + even((size_t)n * (n + 1)) * 2 + 32 * 3 + even(L.nr) * 3 +
                    even(L.n_fo > 0 ? L.n_fo : 1) * 2 + 16 + 6 + extra;
  return staged_bytes(L, L.base_int) + 4 * ws * sizeof(double);
}

// Warps a block, and whether the tables are staged beside their work spaces.  They are unless fewer than four warps
// would be left, as with some 500 reactions: those read them from global memory.
int plan_warps(const MechLayout& L, int ws_doubles, bool* staged, size_t* smem, long cells_per_sm) {
  const size_t mech = staged_bytes(L, L.warp_int), ws = (size_t)ws_doubles * sizeof(double);
  size_t w = mech < kPlainSmem ? (kPlainSmem - mech) / ws : 0;
  *staged = w >= 4;
  if (!*staged) w = kPlainSmem / ws;
  if (w > (size_t)kPlainWarps) w = kPlainWarps;
  if (w > (size_t)cells_per_sm) w = (size_t)cells_per_sm;
  *smem = (*staged ? mech : 0) + w * ws;
  return (int)w;
}

// One block an SM, a small batch a cell an SM.  Where no more than 8 warps fit or have a cell, the kernel of 8, which
// does not spill: CH4, 300 cells 14.5 to 12.2 ms, H2/CO, 67 cells 8.7 to 7.5 ms; with more cells the warps count, H2/CO, 4096 cells
// 26.1 ms at 16 and 27.0 at 12.
template <typename K, typename... A>
cudaError_t launch_warps(const MechLayout& L, int ws_doubles, long ncells, K* const (&kernels)[2][2],
                         cudaStream_t stream, A... args) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const long blocks = ncells < sms ? ncells : sms;
  if (blocks <= 0) return cudaErrorInvalidConfiguration;
  bool staged = false;
  size_t smem = 0;
  const int warps = plan_warps(L, ws_doubles, &staged, &smem, (ncells + blocks - 1) / blocks);
  if (warps < 1) return cudaErrorInvalidValue;
  K* k = kernels[staged ? 1 : 0][warps <= kPlainFew ? 0 : 1];
  // the same value at every call: another thread may launch the kernel with another size at the same time
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlainSmem);
  if (e != cudaSuccess) return e;
  k<<<(unsigned)blocks, warps * 32, smem, stream>>>(args...);
  return cudaGetLastError();
}
#define LSG_WARP_KERNELS(k)                                       \
  {                                                               \
    {k<false, kPlainFew>, k<false, kPlainWarps>}, { k<true, kPlainFew>, k<true, kPlainWarps> } \
  }
}  // namespace

size_t plain_smem_bytes(const MechLayout& L) { return form_bytes(L, 0); }

size_t drg_smem_bytes(const MechLayout& L) { return form_bytes(L, (size_t)((L.nr + 7) / 8 + 1)); }

cudaError_t launch_rhs_warp(const MechLayout& L, const unsigned char* mech_gmem, long ncells, const double* y,
                            double* dy, long ld, double p, int energy, double* qr, int* err, cudaStream_t stream) {
  if (plain_smem_bytes(L) > 227 * 1024) return cudaErrorInvalidValue;
  using K = decltype(rhs_warp_kernel<true, kPlainFew>);
  static K* const kernels[2][2] = LSG_WARP_KERNELS(rhs_warp_kernel);
  return launch_warps<K>(L, warp_ws_doubles(L), ncells, kernels, stream, L, mech_gmem, ncells, y, dy, ld, p, energy, qr, err);
}

cudaError_t upload_gear_plain(const GearConsts& gc) {
  return cudaMemcpyToSymbol(c_gear, &gc, sizeof(GearConsts));
}

cudaError_t launch_plain(const MechLayout& L, const unsigned char* mech_gmem, const StepOptions& o,
                         const StepArgs& a, int* err, cudaStream_t stream) {
  if (a.ncells <= 0) return cudaSuccess;
  using K = decltype(plain_warp_kernel<true, kPlainFew>);
  static K* const kernels[2][2] = LSG_WARP_KERNELS(plain_warp_kernel);
  return launch_warps<K>(L, warp_ws_doubles(L), a.ncells, kernels, stream, L, mech_gmem, o, a, err);
}

cudaError_t launch_drg_eps(long ncells, const double* T, const DrgArgs& d, cudaStream_t stream) {
  if (ncells <= 0) return cudaSuccess;
  drg_eps_kernel<<<1, 32, 0, stream>>>(ncells, T, d);
  return cudaGetLastError();
}

cudaError_t launch_drg_plain(const MechLayout& L, const unsigned char* mech_gmem, const StepOptions& o,
                             const StepArgs& a, const DrgArgs& d, int* err, cudaStream_t stream) {
  if (a.ncells <= 0) return cudaSuccess;
  const cudaError_t e = launch_drg_eps(a.ncells, a.T, d, stream);
  if (e != cudaSuccess) return e;
  using K = decltype(drg_warp_kernel<true, kPlainFew>);
  static K* const kernels[2][2] = LSG_WARP_KERNELS(drg_warp_kernel);
  return launch_warps<K>(L, drg_ws_doubles(L), a.ncells, kernels, stream, L, mech_gmem, o, a, d, err);
}

}  // namespace lsg
