// poisson.cu -- FP64 Poisson solve on the reference's assembled operator.
//
// Host side: the operator is assembled row by row exactly as
// FiniteDifferenceMethod/src/generalized_poisson.jl does it
// (create_generalized_poisson_solver :34-68, apply_dirichlet :205-215,
// add_new_dof :217-230, apply_neumann :235-269, apply_periodic :286-324),
// kept in a 7-slot row form per node: self, (i-1,j), (i+1,j), (i,j-1),
// (i,j+1), x-periodic partner, y-periodic partner; plus σ columns.
//
// Device side, per solve of A ϕ = b (b[ρ] = -ρ/ε0, b[Dirichlet] = ϕ0):
//   * rows that are identity (Dirichlet, σ) are fixed values;
//   * the remaining rows are scaled by D so that S = -D A_ff is symmetric
//     positive (semi)definite (Neumann rows of apply_neumann have a different
//     scale than stencil rows);
//   * when S separates into (tridiagonal in x) + (periodic ring in y) -- true
//     for every problem of the reference that uses apply_periodic(solver, 1)
//     with column electrodes -- it is solved exactly by a real FFT along y, one
//     tridiagonal (Thomas / Sherman-Morrison for x-periodic) solve per Fourier
//     mode along x, and an inverse FFT; the residual is then re-evaluated in
//     FP64 and the correction repeated until ||res|| <= rtol ||rhs||
//     (every ny up to 4096; the odd factor of ny by dense DFTs);
//   * otherwise CG iterates to the same tolerance, preconditioned by a multigrid
//     V-cycle (multigrid.cu) or, for singular operators, by Jacobi scaling;
//   * small grids run a step's whole field part as one block (k_field_block).
// All-periodic / all-open operators are singular; the solve then uses the
// mean-zero gauge with the right-hand side projected onto the range (the
// reference's dense A\b has no defined answer there; E = -∇ϕ is unaffected).
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <map>
#include <tuple>
#include <vector>

#include "internal.cuh"
#include "multigrid.cuh"

namespace iskra {

struct RowClass {
  double c0, cW, cE, cS, cN;  // original (unscaled) coefficients
  double d;                   // symmetrising row scale
  double inv_d;               // 1 / d
  double sig_coef;            // coefficient of the σ column
  int sig_dof;                // -1: none
  int fixed;                  // identity row
  int rho;                    // b = -ρ/ε0 (ρ dof) else b = bfix
  float nd32;                 // -d in FP32 (scaling of the FP32 residual)
  float2 c0f, cWf, cEf, cSf, cNf;  // the coefficients as double-float pairs
  double s0, sW, sE, sS, sN;  // the scaled row -d c (the symmetric operator of CG), 0 on identity rows
};

struct DriveGroup {
  std::vector<int> nodes;
  double amp, freq, phase, dc;
};

struct PoissonScal {           // device-resident solver scalars
  double lambda;               // singular case: range projection shift
  double relres;
  double rhs2, res2;
  int iters;
  int done;
  int sweeps;
  unsigned ticket;             // blocks of the running k_residual that have finished
  double rz, rz_new, pap;
  int hist;                    // xh holds the previous step solve's ϕ (warm start)
  int e_pending;               // the first residual pass met rtol but wrote no E
  unsigned hticket;            // blocks of the running k_extrapolate that have finished
};

struct Poisson {
  // ---- host assembly (generalized_poisson.jl) ----
  int nx = 0, ny = 0, nn = 0;
  double dx = 0, dy = 0, eps0 = 0;
  std::vector<double> C;        // nn*7
  std::vector<double> bfix;     // b for non-ρ rows
  std::vector<uint8_t> rho_dof;
  std::vector<std::vector<double>> sig_cols;  // per σ dof: nn column
  std::vector<double> sig_b;
  std::vector<DriveGroup> drives;
  std::vector<double> er;       // (nx+1)*(ny+1) ones
  bool dirty = true;
  int method = 0;               // 0 auto, 1 CG (Jacobi), 2 CG with the multigrid preconditioner
  Mg *mg = nullptr;             // multigrid hierarchy of a non-separable operator (multigrid.cu)
  cudaGraphExec_t pcg_graph = nullptr;  // one multigrid-CG iteration (9 to 13 kernels), replayed
  double pcg_graph_rtol = 0;
  // ---- device representation ----
  bool separable = false, singular = false, cyclic = false;
  bool sep_form = false;        // the operator separates (direct_solve decides whether it is solved so)
  double stalled = 0;           // largest tolerance at which a direct solve stalled
  int nclass = 0;
  uint16_t *cls = nullptr;      // nn
  RowClass *classes = nullptr;
  double *bfix_d = nullptr;     // nn
  double *sigma_d = nullptr;    // nsig
  int nsig = 0;
  double *x = nullptr;          // ϕ (nn); for separable operators a view refreshed from xd on demand
  float2 *xd = nullptr;         // ϕ as double-float pairs (separable operators: the solver's state)
  float2 *bd = nullptr;         // b of the free rows as double-float pairs (first residual pass)
  void *xh = nullptr;           // previous step solve's ϕ in the state's representation (8 B per node)
  int warm_mode = 1;            // step solves start from 0: ϕ_n, 1: 2 ϕ_n - ϕ_(n-1)
  bool df_mode = false;         // the solver's state is xd (double-float), x a view
  bool x_stale = false;         // (df_mode) x lags xd
  double *r = nullptr, *z = nullptr, *p = nullptr, *ap = nullptr;  // nn
  double *p2 = nullptr;         // second direction buffer of the multigrid CG
  PcgScal *pcg = nullptr;       // its scalars
  double *part = nullptr;       // reduction partials (kPartials * 4)
  PoissonScal *scal = nullptr;
  PoissonScal *scal_h = nullptr;  // pinned
  double dsum = 0;              // Σ d over free rows (singular projection)
  // separable solver
  int N = 0, K = 0, log2p = 0, odd = 1;  // N = ny = 2^log2p odd, K = N/2+1
  // (FP32 correction: factors computed in FP64 on the host, stored rounded)
  float *r32 = nullptr;         // nn scaled residual, input of the correction
  float2 *spec = nullptr;       // nx*K
  float2 *tw = nullptr;         // N/2 twiddles exp(-2πi m/N), then the odd factor's exp(-2πi m/odd)
  float *low = nullptr, *up = nullptr;        // nx
  float *inv = nullptr, *cp = nullptr, *q = nullptr;  // nx*K
  float *gk = nullptr;          // 2K: 1/(1+v.q) and β/γ per mode (x-periodic)
  int cr_levels = 0;            // cyclic reduction: L = floor(log2 nx)
  int cr_nf = 0, cr_nb = 0;     // updated / eliminated rows over all levels
  float2 *cr_fwd = nullptr;     // (α, γ) per mode and updated row
  float2 *cr_back = nullptr;    // (a/b, c/b) per mode and eliminated row
  float *cr_backb = nullptr;    // 1/b per mode and eliminated row
  float *cr_top = nullptr;      // 1/b of the last row per mode
  int pin_k0 = -1;              // pinned column of mode 0 (singular)
  // drives on device
  int ndrive_nodes = 0;
  int *drive_node = nullptr;
  int *drive_group = nullptr;
  double *drive_par = nullptr;  // 4 per group
  int ndrive = 0;
  int blocks = 0;
  int cg_blocks = 0;            // blocks of the multigrid-PCG vector kernels (more per SM: latency bound)
  bool rho_fixed = false;       // some identity row takes its value from ρ (rewritten every solve)
  int last_iters = 0;
  double last_relres = 0;
  // FP64 Thomas factors of the separable operator (host copy; uploaded on
  // demand for the ensemble field solve)
  // FP64 cyclic-reduction coefficients of the ensemble field solve, packed:
  // fwd (K nf pairs), back (K nb pairs), backb (K nb), top (K)
  std::vector<double> cr64;
  double *cr64_d = nullptr;
};

constexpr int kPartials = 1024;
// blocks per SM of the node passes (residuals, conversions): they are latency bound;
// 20 steps of a 512 x 512 slab took 3764 us at 2, 3748 at 3, 3727 at 4, 3757 at 5 and
// 3872 at 6
#ifndef ISKRA_RES_BLOCKS_PER_SM
#define ISKRA_RES_BLOCKS_PER_SM 4
#endif

void poisson_destroy(Poisson *p) {
  if (!p) return;
  mg_destroy(p->mg);
  if (p->pcg_graph) cudaGraphExecDestroy(p->pcg_graph);
  cudaFree(p->cls);
  cudaFree(p->classes);
  cudaFree(p->bfix_d);
  cudaFree(p->sigma_d);
  cudaFree(p->x);
  cudaFree(p->xd);
  cudaFree(p->bd);
  cudaFree(p->xh);
  cudaFree(p->r);
  cudaFree(p->z);
  cudaFree(p->p);
  cudaFree(p->ap);
  cudaFree(p->p2);
  cudaFree(p->pcg);
  cudaFree(p->part);
  cudaFree(p->scal);
  if (p->scal_h) cudaFreeHost(p->scal_h);
  cudaFree(p->cr64_d);
  cudaFree(p->r32);
  cudaFree(p->spec);
  cudaFree(p->tw);
  cudaFree(p->low);
  cudaFree(p->up);
  cudaFree(p->inv);
  cudaFree(p->cp);
  cudaFree(p->q);
  cudaFree(p->gk);
  cudaFree(p->cr_fwd);
  cudaFree(p->cr_back);
  cudaFree(p->cr_backb);
  cudaFree(p->cr_top);
  cudaFree(p->drive_node);
  cudaFree(p->drive_group);
  cudaFree(p->drive_par);
  delete p;
}

// ===========================================================================
// device kernels
// ===========================================================================
// cls[k] = row class id of node k, with kFixedBit set on identity (fixed) rows
constexpr unsigned kFixedBit = 0x8000u;
constexpr unsigned kClassMask = 0x7fffu;

// (double-float arithmetic: df_* in internal.cuh)

struct OpView {
  const uint16_t *cls;
  const RowClass *classes;
  const double *bfix;
  const double *sigma;
  int nx, ny;
  int nclass;
};

__device__ __forceinline__ void nbr(int k, int nx, int ny, int &w, int &e, int &s, int &n) {
  const int i = k % nx, j = k / nx;
  w = i > 0 ? k - 1 : k + nx - 1;
  e = i < nx - 1 ? k + 1 : k - nx + 1;
  s = j > 0 ? k - nx : k + nx * (ny - 1);
  n = j < ny - 1 ? k + nx : k - nx * (ny - 1);
}

__device__ __forceinline__ double drive_value(const double *par, double t) {
  return par[0] * sin(2.0 * M_PI * par[1] * t + par[2]) + par[3];
}

// fixed-row values: Dirichlet / driven
__global__ void k_set_fixed(OpView op, const int *__restrict__ dnode, const int *__restrict__ dgroup,
                            const double *__restrict__ dpar, int ndn, const unsigned long long *__restrict__ step,
                            double dt, double *__restrict__ bfix_mut, double *__restrict__ x, float2 *__restrict__ xd,
                            const double *__restrict__ rho, double eps0, int nn) {
  pdl_wait();
  // driven groups update bfix (solve of step n uses V((n-2)Δt), n >= 2)
  const unsigned long long n_step = step ? *step : 0ull;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ndn; t += gridDim.x * blockDim.x) {
    const int k = dnode[t];
    if (n_step >= 2) {
      double tt = (double)(n_step - 2) * dt;
      bfix_mut[k] = drive_value(dpar + 4 * dgroup[t], tt);
    }
    x[k] = bfix_mut[k];
    if (xd) xd[k] = df_from(bfix_mut[k]);
  }
}

__global__ void k_fixed_to_x(OpView op, double *__restrict__ x, float2 *__restrict__ xd,
                             const double *__restrict__ rho, double neg_inv_eps0, int nn) {
  pdl_wait();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const unsigned ck = op.cls[k];
    if (ck & kFixedBit) {
      const double v = op.classes[ck & kClassMask].rho ? rho[k] * neg_inv_eps0 : op.bfix[k];
      x[k] = v;
      if (xd) xd[k] = df_from(v);
    }
  }
}

// ϕ conversions between the FP64 view and the double-float state
__global__ void k_df_to_x(const float2 *__restrict__ xd, double *__restrict__ x, int nn) {
  pdl_wait();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) x[k] = df_value(xd[k]);
}
__global__ void k_x_to_df(const double *__restrict__ x, float2 *__restrict__ xd, int nn) {
  pdl_wait();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) xd[k] = df_from(x[k]);
}

// Warm start of a step's solve: the free rows of ϕ extrapolated linearly in
// time from the last two step solutions, ϕ <- 2 ϕ_n - ϕ_(n-1) (a better
// initial guess than ϕ_n while the charge moves smoothly: fewer corrections
// reach the tolerance, which is still tested on the residual); xh <- ϕ_n.
// With no valid history (sc->hist == 0) it only records ϕ_n; the last block
// to finish marks the history valid (every block has read the flag by then).
template <bool DF>
__global__ void k_extrapolate(const uint16_t *__restrict__ cls, void *__restrict__ xv, void *__restrict__ xhv,
                              int nn, PoissonScal *sc) {
  pdl_wait();
  __shared__ int last;
  const bool h = sc->hist != 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const bool upd = h && !(cls[k] & kFixedBit);
    if (DF) {
      float2 *x = (float2 *)xv, *xh = (float2 *)xhv;
      const float2 a = x[k];
      if (upd) x[k] = df_add(make_float2(2.f * a.x, 2.f * a.y), df_neg(xh[k]));
      xh[k] = a;
    } else {
      double *x = (double *)xv, *xh = (double *)xhv;
      const double a = x[k];
      if (upd) x[k] = 2.0 * a - xh[k];
      xh[k] = a;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&sc->hticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    sc->hticket = 0u;
    sc->hist = 1;
  }
}

// Σ d_k b_k over free rows (singular case only: no fixed rows exist)
__global__ void k_sum_db(OpView op, const double *__restrict__ rho, double neg_inv_eps0, int nn,
                         double *__restrict__ part) {
  pdl_wait();
  __shared__ double sh[40];
  double v = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const RowClass &C = op.classes[op.cls[k] & kClassMask];
    if (!C.fixed) {
      double b = C.rho ? rho[k] * neg_inv_eps0 : op.bfix[k];
      if (C.sig_dof >= 0) b -= C.sig_coef * op.sigma[C.sig_dof];
      v += C.d * b;
    }
  }
  double t = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

__global__ void k_lambda(const double *__restrict__ part, int nparts, double dsum, PoissonScal *sc) {
  pdl_wait();
  __shared__ double sh[40];
  double s = sum_partials(part, nparts, sh);
  if (threadIdx.x == 0) sc->lambda = dsum > 0 ? s / dsum : 0.0;
}

static bool power_of_two(int n) { return (n & (n - 1)) == 0; }

// Optional E = -∇ϕ output of k_residual (generalized_poisson.jl:398-410):
// FP32 node values: the MCC target term and, staged per tile, the gather.
// The node differences are taken in FP64 (ϕ is ~10^2-10^3 V while neighbour
// differences are ~10^-1 V) and scaled in FP32, or wholly in FP64 (exact).
struct EOut {
  float2 *E32;
  float idx2, idx1, idy2, idy1;  // 1/(2Δx), 1/Δx, 1/(2Δy), 1/Δy
  int exact = 0;                 // FP64 down to the last rounding, as k_efield
  double dx2 = 0, dx1 = 0, dy2 = 0, dy1 = 0;  // (exact) the same
};

__device__ __forceinline__ void efield_at(const double *__restrict__ x, int k, int i, int j, int nx, int ny,
                                          const EOut &eo) {
  if (eo.exact) {
    const double ex = i == 0 ? (x[k] - x[k + 1]) * eo.dx1
                             : i == nx - 1 ? (x[k - 1] - x[k]) * eo.dx1 : (x[k - 1] - x[k + 1]) * eo.dx2;
    const double ey = j == 0 ? (x[k] - x[k + nx]) * eo.dy1
                             : j == ny - 1 ? (x[k - nx] - x[k]) * eo.dy1 : (x[k - nx] - x[k + nx]) * eo.dy2;
    eo.E32[k] = make_float2((float)ex, (float)ey);
    return;
  }
  float ex, ey;
  if (i == 0) ex = (float)(x[k] - x[k + 1]) * eo.idx1;
  else if (i == nx - 1) ex = (float)(x[k - 1] - x[k]) * eo.idx1;
  else ex = (float)(x[k - 1] - x[k + 1]) * eo.idx2;
  if (j == 0) ey = (float)(x[k] - x[k + nx]) * eo.idy1;
  else if (j == ny - 1) ey = (float)(x[k - nx] - x[k]) * eo.idy1;
  else ey = (float)(x[k - nx] - x[k + nx]) * eo.idy2;
  eo.E32[k] = make_float2(ex, ey);
}

constexpr int kSmemClasses = 128;  // row-class table held in shared memory up to this size

// res = b - λ - A x over free rows, stored scaled as r = -d * res (FP64 in
// r64 for CG, FP32 in r32 as the input of the FP32 separable correction).
// Block partials of ||res||² (and, in the FIRST pass of a solve, of
// ||rhs_eff||², rhs_eff = b - λ - A_fixed x_fixed) are summed by the last
// block to finish, in block order (deterministic), which updates
// relres/iters and sets sc->done when ||res|| <= rtol ||rhs_eff||.  With
// EOUT, E = -∇ϕ of x is written too.  Passes after the first return at once
// when sc->done is set and count one sweep each.
//
// GB300 runs FP64 at ~1/64 of the FP32 rate, so this pass is built to use few
// FP64 instructions: the sweep form sums the whole stencil in one FMA chain.
// In a step graph the residual of the last sweep flags DERR_NOTCONV (in
// *notconv) when the solve stops above tolerance.
struct SweepLoop {
  int *notconv;        // the last pass of a step graph: where an unmet tolerance is flagged
  StepStatus *status;  // where the pass that ends the solve reports to the host, or nullptr
  const int *err;      // (status) the error flag
};

// The step's error flag to the host, by one thread, when every kernel or phase that
// may set it has ended.
__device__ __forceinline__ void report_step(StepStatus *status, const int *err) {
  status->err = *(const volatile int *)err;
  __threadfence_system();
  *(volatile int *)&status->there = 1;
}

// Residual of free row k: res = b - λ - A x, returned scaled as -d res in
// FP32 (r64 != nullptr also receives it in FP64); 0 on fixed rows.  The
// FIRST pass of a solve also accumulates ||rhs_eff||² (rhs_eff = b - λ -
// A_fixed x_fixed).
template <bool FIRST>
__device__ __forceinline__ float residual_node(const OpView &op, const RowClass *__restrict__ CT,
                                               const double *__restrict__ x, const double *__restrict__ rho,
                                               double neg_inv_eps0, double lam, int singular, int k, int i, int j,
                                               double *__restrict__ r64, double &a2, double &b2) {
  const int nx = op.nx, ny = op.ny;
  const unsigned ck = op.cls[k];
  if (ck & kFixedBit) {
    if (r64) r64[k] = 0.0;
    return 0.f;
  }
  const RowClass &C = CT[ck];
  const int w = i > 0 ? k - 1 : k + nx - 1;
  const int e = i < nx - 1 ? k + 1 : k - nx + 1;
  const int s = j > 0 ? k - nx : k + nx * (ny - 1);
  const int n = j < ny - 1 ? k + nx : k - nx * (ny - 1);
  double b = C.rho ? rho[k] * neg_inv_eps0 : op.bfix[k];
  if (singular) b -= lam;
  if (C.sig_dof >= 0) b -= C.sig_coef * op.sigma[C.sig_dof];
  double res;
  if (FIRST) {
    double afix = 0, afree = C.c0 * x[k];
    double t;
    t = C.cW * x[w];
    if (op.cls[w] & kFixedBit) afix += t; else afree += t;
    t = C.cE * x[e];
    if (op.cls[e] & kFixedBit) afix += t; else afree += t;
    t = C.cS * x[s];
    if (op.cls[s] & kFixedBit) afix += t; else afree += t;
    t = C.cN * x[n];
    if (op.cls[n] & kFixedBit) afix += t; else afree += t;
    const double rhs = b - afix;
    res = rhs - afree;
    b2 = fma(rhs, rhs, b2);
  } else {
    // GB300 runs FP64 at ~1/64 of the FP32 rate: one FMA chain over the stencil
    double ax = C.c0 * x[k];
    ax = fma(C.cW, x[w], ax);
    ax = fma(C.cE, x[e], ax);
    ax = fma(C.cS, x[s], ax);
    ax = fma(C.cN, x[n], ax);
    res = b - ax;
  }
  a2 = fma(res, res, a2);
  if (r64) r64[k] = -C.d * res;
  return (float)res * C.nd32;
}

// Block partials of the norms, then the last block to finish sums them in
// block order (deterministic), updates relres/iters and sets sc->done when
// ||res|| <= rtol ||rhs_eff||.  Ends the kernel for every other block.  (256
// threads; block_sums instead of a shuffle tree in every warp.)
template <bool FIRST>
__device__ __forceinline__ void finish_norms(PoissonScal *sc, double *__restrict__ part, double a2, double b2,
                                             double rtol2, SweepLoop loop) {
  constexpr int K = FIRST ? 2 : 1;
  __shared__ double buf[K * 256];
  __shared__ int last;
  double v[K], t[K];
  v[0] = a2;
  if (FIRST) v[K - 1] = b2;
  block_sums<K>(v, buf, t);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < K; q++) part[q * kPartials + blockIdx.x] = t[q];
    __threadfence();
    last = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int q = 0; q < K; q++) {
    v[q] = 0;
    for (int k = threadIdx.x; k < gridDim.x; k += 256) v[q] += __ldcg(part + q * kPartials + k);
  }
  block_sums<K>(v, buf, t);
  const double a = t[0], bb = FIRST ? t[K - 1] : 0.0;
  if (threadIdx.x == 0) {
    sc->ticket = 0u;
    const double rhs2 = FIRST ? bb : sc->rhs2;
    if (FIRST) {
      sc->rhs2 = bb;
      sc->iters = 0;
    } else {
      sc->iters += 1;
    }
    sc->res2 = a;
    sc->relres = rhs2 > 0 ? sqrt(a / rhs2) : sqrt(a);
    const int done = (rhs2 > 0 && a <= rtol2 * rhs2) || a == 0.0;
    sc->done = done;
    if (FIRST) sc->e_pending = done;
    if (loop.notconv && !done) atomicOr(loop.notconv, DERR_NOTCONV);
    if (loop.status && (done || loop.notconv)) report_step(loop.status, loop.err);
  }
}

// The row classes in shared memory when they fit, copied 8 bytes a thread (a whole
// class per thread is a chain of 16-byte copies: 1 us more in every residual pass).
// They are written by the operator build: callable before pdl_wait.  The caller's
// next block barrier makes them readable.
__device__ __forceinline__ const RowClass *stage_classes(const OpView &op, RowClass *cls_sh) {
  if (op.nclass > kSmemClasses) return op.classes;
  static_assert(sizeof(RowClass) % 8 == 0, "copied in words of 8 bytes");
  const double *__restrict__ src = reinterpret_cast<const double *>(op.classes);
  double *dst = reinterpret_cast<double *>(cls_sh);
  for (int t = threadIdx.x; t < op.nclass * (int)(sizeof(RowClass) / 8); t += blockDim.x) dst[t] = __ldg(src + t);
  return cls_sh;
}

// Residual pass over all nodes (scaled residual to r32 or r64), optionally
// with E = -∇ϕ, and the convergence test.  Passes after the first return at
// once when sc->done is set and count one sweep each.
template <bool FIRST, bool EOUT>
__global__ void __launch_bounds__(256) k_residual(OpView op, const double *__restrict__ x,
                                                  const double *__restrict__ rho, double neg_inv_eps0,
                                                  PoissonScal *sc, double *__restrict__ r64, float *__restrict__ r32,
                                                  double *__restrict__ part, int nn, int singular, double rtol2,
                                                  EOut eo, SweepLoop loop) {
  __shared__ RowClass cls_sh[kSmemClasses];
  const RowClass *__restrict__ CT = stage_classes(op, cls_sh);
  pdl_wait();
  if (!FIRST && sc->done) return;
  __syncthreads();
  const double lam = singular ? sc->lambda : 0.0;
  const int nx = op.nx, ny = op.ny;
  double a2 = 0, b2 = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const int j = k / nx, i = k - j * nx;
    if (EOUT) efield_at(x, k, i, j, nx, ny, eo);
    const float v = residual_node<FIRST>(op, CT, x, rho, neg_inv_eps0, lam, singular, k, i, j, r64, a2, b2);
    if (r32) r32[k] = v;
  }
  finish_norms<FIRST>(sc, part, a2, b2, rtol2, loop);
}

// E = -∇ϕ at node k from ϕ at the node and its four stencil neighbours
// (double-float pairs, differenced in FP32: the hi parts of neighbours
// subtract exactly when within a factor 2; one-sided at the walls as efield_at)
__device__ __forceinline__ void efield_df5(float2 xk, float2 xw, float2 xe, float2 xs, float2 xn, int k, int i, int j,
                                           int nx, int ny, const EOut &eo) {
  auto dif = [](float2 p, float2 q) { return (p.x - q.x) + (p.y - q.y); };
  float ex, ey;
  if (i == 0) ex = dif(xk, xe) * eo.idx1;
  else if (i == nx - 1) ex = dif(xw, xk) * eo.idx1;
  else ex = dif(xw, xe) * eo.idx2;
  if (j == 0) ey = dif(xk, xn) * eo.idy1;
  else if (j == ny - 1) ey = dif(xs, xk) * eo.idy1;
  else ey = dif(xs, xn) * eo.idy2;
  eo.E32[k] = make_float2(ex, ey);
}

// Residual pass of the separable solver on the double-float ϕ: the stencil
// A x is summed in double-float arithmetic (FP32 pipes); the FIRST pass forms
// b (FP64, then split) for the free rows into bd and the rhs norm, later
// passes reuse bd.  Scaled FP32 residual to r32, E (EOUT), convergence test
// as k_residual (norms in FP64).  A node's loads (its row class, ϕ at the
// five stencil nodes, b) are all issued before its branch on the row class:
// the pass is bound by memory latency, not bandwidth.  In a step graph the
// FIRST pass writes no E (a correction nearly always follows); when it meets
// rtol already, the next pass, otherwise skipped, writes E instead.
// The node loop of k_residual_df over nodes k0, k0 + stride, ... < nn
// (partial norms in a2, b2).
template <bool FIRST, bool EOUT>
__device__ __forceinline__ void residual_df_nodes(const OpView &op, const RowClass *__restrict__ CT,
                                                  const float2 *__restrict__ x, const double *__restrict__ rho,
                                                  const float2 *__restrict__ rho_df, float2 nie_df,
                                                  double neg_inv_eps0, float2 *__restrict__ bd,
                                                  float *__restrict__ r32, int nn, int singular, double lam,
                                                  const EOut &eo, int k0, int stride, double &a2, double &b2) {
  const int nx = op.nx, ny = op.ny;
  for (int k = k0; k < nn; k += stride) {
    const int j = k / nx, i = k - j * nx;
    const int w = i > 0 ? k - 1 : k + nx - 1;
    const int e = i < nx - 1 ? k + 1 : k - nx + 1;
    const int s = j > 0 ? k - nx : k + nx * (ny - 1);
    const int n = j < ny - 1 ? k + nx : k - nx * (ny - 1);
    const unsigned ck = op.cls[k];
    const float2 xk = x[k], xw = x[w], xe = x[e], xs = x[s], xn = x[n];
    double rk = 0.0, fk = 0.0;
    float2 rdk = make_float2(0.f, 0.f);
    unsigned cw = 0, ce = 0, cs = 0, cn = 0;
    float2 b = make_float2(0.f, 0.f);
    if (FIRST) {
      if (rho_df) rdk = rho_df[k];
      else rk = rho[k];
      fk = op.bfix[k];
      cw = op.cls[w];
      ce = op.cls[e];
      cs = op.cls[s];
      cn = op.cls[n];
    } else {
      b = bd[k];
    }
    if (EOUT) efield_df5(xk, xw, xe, xs, xn, k, i, j, nx, ny, eo);
    if (ck & kFixedBit) {
      r32[k] = 0.f;
      continue;
    }
    const RowClass &C = CT[ck];
    float2 res;
    if (FIRST) {
      if (rho_df && C.rho) {  // ρ formed in double-float (no λ, no σ dofs then)
        b = df_mul(rdk, nie_df);
      } else {
        double bv = C.rho ? rk * neg_inv_eps0 : fk;
        if (singular) bv -= lam;
        if (C.sig_dof >= 0) bv -= C.sig_coef * op.sigma[C.sig_dof];
        b = df_from(bv);
      }
      bd[k] = b;
      float2 afix = make_float2(0.f, 0.f), afree = df_mul(C.c0f, xk);
      const float2 t[4] = {df_mul(C.cWf, xw), df_mul(C.cEf, xe), df_mul(C.cSf, xs), df_mul(C.cNf, xn)};
      const unsigned cq[4] = {cw, ce, cs, cn};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (cq[q] & kFixedBit) afix = df_add(afix, t[q]);
        else afree = df_add(afree, t[q]);
      }
      const float2 rhs = df_add(b, df_neg(afix));
      res = df_add(rhs, df_neg(afree));
      // the norms decide convergence to ~1e-7 relative at most: the FP32
      // value of the pair, squared in FP64 (no overflow)
      const double rh = (double)(rhs.x + rhs.y);
      b2 = fma(rh, rh, b2);
    } else {
      float2 ax = df_mul(C.c0f, xk);
      ax = df_add(ax, df_mul(C.cWf, xw));
      ax = df_add(ax, df_mul(C.cEf, xe));
      ax = df_add(ax, df_mul(C.cSf, xs));
      ax = df_add(ax, df_mul(C.cNf, xn));
      res = df_add(b, df_neg(ax));
    }
    const float resf = res.x + res.y;
    r32[k] = resf * C.nd32;
    const double rv = (double)resf;
    a2 = fma(rv, rv, a2);
  }
}

// E = -∇ϕ of the double-float ϕ at every node (a converged first residual
// wrote none)
__device__ __forceinline__ void efield_df_nodes(const float2 *__restrict__ x, int nx, int ny, int nn,
                                                const EOut &eo, int k0, int stride) {
  for (int k = k0; k < nn; k += stride) {
    const int j = k / nx, i = k - j * nx;
    const int w = i > 0 ? k - 1 : k + nx - 1, e = i < nx - 1 ? k + 1 : k - nx + 1;
    const int s = j > 0 ? k - nx : k + nx * (ny - 1), n = j < ny - 1 ? k + nx : k - nx * (ny - 1);
    efield_df5(x[k], x[w], x[e], x[s], x[n], k, i, j, nx, ny, eo);
  }
}

// Residual pass of the separable solver on the double-float ϕ: the stencil
// A x is summed in double-float arithmetic (FP32 pipes); the FIRST pass forms
// b (FP64, then split) for the free rows into bd and the rhs norm, later
// passes reuse bd.  Scaled FP32 residual to r32, E (EOUT), convergence test
// as k_residual (norms in FP64).  A node's loads (its row class, ϕ at the
// five stencil nodes, b) are all issued before its branch on the row class:
// the pass is bound by memory latency, not bandwidth.  In a step graph the
// FIRST pass writes no E (a correction nearly always follows); when it meets
// rtol already, the next pass, otherwise skipped, writes E instead.
template <bool FIRST, bool EOUT>
__global__ void __launch_bounds__(256) k_residual_df(OpView op, const float2 *__restrict__ x,
                                                     const double *__restrict__ rho, const float2 *__restrict__ rho_df,
                                                     float2 nie_df, double neg_inv_eps0,
                                                     float2 *__restrict__ bd, PoissonScal *sc, float *__restrict__ r32,
                                                     double *__restrict__ part, int nn, int singular, double rtol2,
                                                     EOut eo, SweepLoop loop) {
  __shared__ RowClass cls_sh[kSmemClasses];
  const RowClass *__restrict__ CT = stage_classes(op, cls_sh);
  pdl_wait();
  const int k0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  if (!FIRST && sc->done) {
    if (EOUT && sc->e_pending) efield_df_nodes(x, op.nx, op.ny, nn, eo, k0, stride);
    return;
  }
  __syncthreads();
  const double lam = singular ? sc->lambda : 0.0;
  double a2 = 0, b2 = 0;
  residual_df_nodes<FIRST, EOUT>(op, CT, x, rho, rho_df, nie_df, neg_inv_eps0, bd, r32, nn, singular, lam, eo, k0,
                                 stride, a2, b2);
  finish_norms<FIRST>(sc, part, a2, b2, rtol2, loop);
}

// mean-zero projection of the double-float ϕ (singular operators)
__global__ void k_sum_xd(const float2 *__restrict__ x, int nn, double *__restrict__ part) {
  pdl_wait();
  __shared__ double sh[40];
  double v = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) v += df_value(x[k]);
  double t = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}
__global__ void k_shift_xd(float2 *__restrict__ x, int nn, const double *__restrict__ part, int nparts) {
  pdl_wait();
  __shared__ double sh[40];
  double s = sum_partials(part, nparts, sh);
  const float2 m = df_neg(df_from(s / nn));
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) x[k] = df_add(x[k], m);
}

// ---------------- separable correction: FFT(y) x tridiagonal(x), FP32 ----------------
// One sweep computes δ ≈ S^-1 r in FP32 and adds it to the FP64 ϕ; the FP64
// residual pass that follows decides convergence (iterative refinement), so
// the converged ϕ meets the FP64 tolerance while the transform and the
// tridiagonal solves run on the FP32 pipes.  Two real columns share one
// complex FFT: z = a + i b, A_k = (Z_k + conj Z_{N-k})/2,
// B_k = (Z_k - conj Z_{N-k})/(2i).
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ unsigned bitrev(unsigned v, int bits) { return __brev(v) >> (32 - bits); }

// Transform length N = 2^log2p odd.  A power of two (odd == 1) is radix-2
// butterflies alone; any other ny takes its odd factor as dense DFTs first
// (ODD instantiations of the kernels), so that operators of every ny are
// solved directly instead of by multigrid CG (35 iterations of ~33 launches
// on a 301 x 97 slab: 3.6 ms per step).
struct FftPlan {
  int N, log2p, odd;
  const float2 *tw;   // N/2 twiddles exp(-2 pi i p / N)
  const float2 *twm;  // odd twiddles exp(-2 pi i p / odd) (odd > 1)
};

// position of input j in the buffer: subsequence j mod 2^log2p (bit-reversed),
// its elements contiguous
template <bool ODD>
__device__ __forceinline__ int fft_pos(int j, const FftPlan &F) {
  if (!ODD) return (int)bitrev((unsigned)j, F.log2p);
  const int r = F.log2p ? (int)bitrev((unsigned)(j & ((1 << F.log2p) - 1)), F.log2p) : 0;
  return r * F.odd + (j >> F.log2p);
}

// Dense DFTs of length m = odd over the m-element runs of TP columns (column
// stride S), src -> dst.  Outputs q and m - q share their products: with
// s_t = z_t + z_(m-t), d_t = z_t - z_(m-t),
//   Z_q, Z_(m-q) = z_0 + sum_t s_t cos(2 pi t q / m) -+ i d_t sin(2 pi t q / m)
// (four FMAs per t for the two).  m^2/4 terms per run: at the m of real grids
// (up to a few hundred) a few microseconds for the whole grid, bound by the
// shared-memory reads of the twiddle at (t q) mod m.
__device__ void dft_runs(const float2 *__restrict__ src, float2 *__restrict__ dst, int TP, const FftPlan &F, int S,
                         const float2 *twm, bool inverse) {
  const int m = F.odd, hm = (m - 1) >> 1, runs = 1 << F.log2p;
  const int per = runs * (hm + 1);
  for (int b = threadIdx.x; b < TP * per; b += blockDim.x) {
    const int col = b / per, r = (b - col * per) / (hm + 1), q = b - col * per - r * (hm + 1);
    const float2 *z = src + col * S + r * m;
    float2 *o = dst + col * S + r * m;
    float ar = z[0].x, ai = z[0].y, br = 0.f, bi = 0.f;
    int at = 0;
    for (int t = 1; t <= hm; t++) {
      at += q;
      if (at >= m) at -= m;
      const float2 w = twm[at];  // cos, -sin
      const float2 u = z[t], v = z[m - t];
      ar = fmaf(u.x + v.x, w.x, ar);
      ai = fmaf(u.y + v.y, w.x, ai);
      br = fmaf(u.x - v.x, w.y, br);
      bi = fmaf(u.y - v.y, w.y, bi);
    }
    // Z_q = a + i b for the forward transform (w.y = -sin), conjugated twiddles inverse
    const float sg = inverse ? -1.f : 1.f;
    o[q] = make_float2(ar - sg * bi, ai + sg * br);
    if (q) o[m - q] = make_float2(ar + sg * bi, ai - sg * br);
  }
  __syncthreads();
}

// FFT of TP length-N columns held in shared memory with column stride S
// (input at fft_pos): dense DFTs of the odd factor (buf -> alt), then radix-2
// DIT stages in place, twiddles tw (N/2, shared); the inverse uses conjugate
// twiddles and leaves the 1/N to the caller.  Returns the buffer that holds
// the result.
template <bool ODD>
__device__ float2 *fft_columns(float2 *buf, float2 *alt, int TP, const FftPlan &F, int S, const float2 *tw,
                               const float2 *twm, bool inverse) {
  const int N = F.N, logN = F.log2p;
  if (ODD) {
    dft_runs(buf, alt, TP, F, S, twm, inverse);
    buf = alt;
  }
  const int hlog = logN - 1, hn = N >> 1;
  const int total = logN > 0 ? TP * hn : 0;
  for (int s = 1; s <= logN; s++) {
    const int half = ODD ? F.odd << (s - 1) : 1 << (s - 1);
    const int tws = logN - s;  // twiddle index = pos << tws
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
      int col, kk, pos, i1;
      if (ODD) {
        col = b / hn;
        kk = b - col * hn;
        const int g = kk / half;
        pos = kk - g * half;
        i1 = 2 * g * half + pos;
      } else {
        col = b >> hlog;
        kk = b & (hn - 1);
        pos = kk & (half - 1);
        i1 = ((kk >> (s - 1)) << s) + pos;
      }
      const int i2 = i1 + half;
      float2 w = tw[pos << tws];
      if (inverse) w.y = -w.y;
      float2 *c = buf + col * S;
      const float2 t = cmulf(w, c[i2]);
      const float2 u = c[i1];
      c[i1] = make_float2(u.x + t.x, u.y + t.y);
      c[i2] = make_float2(u.x - t.x, u.y - t.y);
    }
    __syncthreads();
  }
  return buf;
}

// shared memory of a transform block: TP columns of stride N + 1, N/2
// twiddles and, with an odd factor, as many columns again and its twiddles
struct FftShared {
  float2 *buf, *tw, *alt, *twm;
};
template <bool ODD>
__device__ __forceinline__ FftShared fft_shared(float2 *base, int TP, const FftPlan &F) {
  FftShared q;
  const int cols = TP * (F.N + 1);
  q.buf = base;
  q.tw = base + cols;
  q.alt = ODD ? q.tw + (F.N >> 1) : nullptr;
  q.twm = ODD ? q.alt + cols : nullptr;
  for (int t = threadIdx.x; t < (F.N >> 1); t += blockDim.x) q.tw[t] = __ldg(F.tw + t);
  if (ODD)
    for (int t = threadIdx.x; t < F.odd; t += blockDim.x) q.twm[t] = __ldg(F.twm + t);
  return q;
}

// r (nx, ny) -> spec[i K + k], k = 0..N/2: forward FFT along y of the 2 TP
// columns of work item `item` (columns 2 TP item ...), two per complex
// transform.
template <bool ODD>
__device__ __forceinline__ void fft_fwd_item(int item, const float *__restrict__ r, int nx, const FftPlan &F, int TP,
                                             float2 *__restrict__ spec, float2 *base) {
  const int N = F.N, S = N + 1, W = 2 * TP, K = (N >> 1) + 1;
  const int i0 = item * W;
  const FftShared q = fft_shared<ODD>(base, TP, F);
  for (int t = threadIdx.x; t < W * N; t += blockDim.x) {
    const int j = t / W, c = t - j * W;
    const int i = i0 + c;
    const float v = i < nx ? r[i + (size_t)nx * j] : 0.f;
    reinterpret_cast<float *>(q.buf + (c >> 1) * S + fft_pos<ODD>(j, F))[c & 1] = v;
  }
  __syncthreads();
  const float2 *z = fft_columns<ODD>(q.buf, q.alt, TP, F, S, q.tw, q.twm, false);
  for (int t = threadIdx.x; t < TP * K; t += blockDim.x) {
    const int p = t / K, k = t - p * K;
    const float2 zk = z[p * S + k];
    const float2 zm = z[p * S + (k ? N - k : 0)];
    const int ia = i0 + 2 * p;
    if (ia < nx) spec[(size_t)ia * K + k] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    if (ia + 1 < nx) spec[(size_t)(ia + 1) * K + k] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
  }
}

template <bool ODD>
__global__ void __launch_bounds__(256) k_fft_fwd(const float *__restrict__ r, int nx, FftPlan F, int TP,
                                                 float2 *__restrict__ spec, const PoissonScal *__restrict__ sc) {
  pdl_wait();
  extern __shared__ float2 fbuf[];
  if (sc->done) return;
  fft_fwd_item<ODD>(blockIdx.x, r, nx, F, TP, spec, fbuf);
}

// Per Fourier mode and real/imaginary part (one thread each): Thomas forward
// elimination and back substitution along x with the precomputed factors, in
// place in spec; Sherman-Morrison correction for x-periodic operators.  Used
// when a mode's column does not fit in shared memory for cyclic reduction.
// Rows are fetched in chunks of kTriChunk so that the chunk's loads are in
// flight together instead of one L2 round trip per row of the recurrence.
constexpr int kTriChunk = 16;

__global__ void __launch_bounds__(64) k_tridiag(float *__restrict__ spec, int nx, int K,
                                                const float *__restrict__ low, const float *__restrict__ inv,
                                                const float *__restrict__ cp, const float *__restrict__ q,
                                                const float *__restrict__ gk, int cyclic, int pin0,
                                                const PoissonScal *__restrict__ sc) {
  pdl_wait();
  if (sc->done) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = t >> 1, part = t & 1;
  if (k >= K) return;
  const size_t K2 = 2 * (size_t)K;
  float *__restrict__ col = spec + 2 * (size_t)k + part;  // row i at col[i * K2]
  if (pin0 >= 0 && k == 0) col[(size_t)pin0 * K2] = 0.f;  // pinned row of the singular mode
  float y = 0.f;
  for (int i0 = 0; i0 < nx; i0 += kTriChunk) {
    float r[kTriChunk], iv[kTriChunk], a[kTriChunk];
#pragma unroll
    for (int c = 0; c < kTriChunk; c++) {
      const int i = i0 + c;
      if (i < nx) {
        r[c] = col[i * K2];
        iv[c] = inv[(size_t)i * K + k];
        a[c] = i > 0 ? __ldg(low + i) : 0.f;
      }
    }
#pragma unroll
    for (int c = 0; c < kTriChunk; c++) {
      const int i = i0 + c;
      if (i < nx) {
        y = (r[c] - a[c] * y) * iv[c];
        col[i * K2] = y;
      }
    }
  }
  float xn = y;
  for (int i1 = nx - 2; i1 >= 0; i1 -= kTriChunk) {
    float yv[kTriChunk], cv[kTriChunk];
#pragma unroll
    for (int c = 0; c < kTriChunk; c++) {
      const int i = i1 - c;
      if (i >= 0) {
        yv[c] = col[i * K2];
        cv[c] = cp[(size_t)i * K + k];
      }
    }
#pragma unroll
    for (int c = 0; c < kTriChunk; c++) {
      const int i = i1 - c;
      if (i >= 0) {
        xn = yv[c] - cv[c] * xn;
        col[i * K2] = xn;
      }
    }
  }
  if (cyclic && !(k == 0 && pin0 >= 0)) {
    const float x0 = col[0], xl = col[(size_t)(nx - 1) * K2];
    const float f = (x0 + gk[K + k] * xl) * gk[k];
    for (int i = 0; i < nx; i++) col[i * K2] -= f * q[(size_t)i * K + k];
  }
}

// Cyclic reduction along x for G Fourier modes (2G real columns) held in
// shared memory.  The host factorisation stores each mode's coefficients
// contiguously (fwd: nf (α, γ) pairs, back: nb (a/b, c/b) pairs, backb: nb
// 1/b, then 1/b of the last row), and the block stages them in shared memory
// with the data in one pass, so the 2L dependent levels run on shared memory
// only.  A block takes modes G blockIdx.x ...
struct CrArgs {
  float *spec;
  int nx, K, G, L, nf, nb;
  const float2 *fwd, *back;
  const float *backb, *top, *q, *gk;
  int cyclic, pin0;
};

// shared-memory layout of a block's modes: data of 2G columns, then per mode the
// coefficients
struct CrShared {
  float *d;            // [col][nx]
  float2 *cf, *cb;     // [g][nf], [g][nb]
  float *cbb;          // [g][nb]
};
__device__ __forceinline__ CrShared cr_shared(const CrArgs &A, float *fsh) {
  CrShared q;
  q.d = fsh;
  q.cf = reinterpret_cast<float2 *>(fsh + 2 * A.G * A.nx);
  q.cb = q.cf + (size_t)A.G * A.nf;
  q.cbb = reinterpret_cast<float *>(q.cb + (size_t)A.G * A.nb);
  return q;
}
// coefficients of modes k0 .. k0 + g - 1 (no barrier)
__device__ __forceinline__ void cr_stage(const CrArgs &A, const CrShared &q, int k0, int g) {
  const int nf = A.nf, nb = A.nb;
  for (int t = threadIdx.x; t < g * nf; t += blockDim.x) q.cf[t] = __ldg(A.fwd + (size_t)k0 * nf + t);
  for (int t = threadIdx.x; t < g * nb; t += blockDim.x) {
    q.cb[t] = __ldg(A.back + (size_t)k0 * nb + t);
    q.cbb[t] = __ldg(A.backb + (size_t)k0 * nb + t);
  }
}
// The 2L levels on the staged columns; REAL: one real column per mode (ny = 2),
// else its real and imaginary parts.  Ends with a block barrier.
template <bool REAL>
__device__ __forceinline__ void cr_levels(const CrArgs &A, const CrShared &q, int k0, int ncol) {
  const int nx = A.nx, L = A.L, nf = A.nf, nb = A.nb;
  constexpr int sh = REAL ? 0 : 1;  // column -> mode
  if (REAL) ncol = 2;
  int F = 0, B = 0;
  for (int l = 0; l < L; l++) {
    const int s = 1 << l, cnt = nx >> (l + 1);
    for (int t = threadIdx.x; t < cnt * ncol; t += blockDim.x) {
      const int m = t / ncol, col = t - m * ncol;
      const int i = (m + 1) * 2 * s - 1;
      const float2 ag = q.cf[(col >> sh) * nf + F + m];
      float *dc = q.d + col * nx;
      float v = dc[i] - ag.x * dc[i - s];
      if (i + s < nx) v -= ag.y * dc[i + s];
      dc[i] = v;
    }
    F += cnt;
    B += ((nx >> l) + 1) >> 1;
    __syncthreads();
  }
  const int topr = (1 << L) - 1;
  for (int col = threadIdx.x; col < ncol; col += blockDim.x) q.d[col * nx + topr] *= __ldg(A.top + k0 + (col >> sh));
  __syncthreads();
  for (int l = L - 1; l >= 0; l--) {
    const int s = 1 << l, ecnt = ((nx >> l) + 1) >> 1;
    B -= ecnt;
    for (int t = threadIdx.x; t < ecnt * ncol; t += blockDim.x) {
      const int m = t / ncol, col = t - m * ncol;
      const int j = (2 * m + 1) * s - 1;
      const int o = (col >> sh) * nb + B + m;
      const float2 r = q.cb[o];
      float *dc = q.d + col * nx;
      float x = q.cbb[o] * dc[j];
      if (j - s >= 0) x -= r.x * dc[j - s];
      if (j + s < nx) x -= r.y * dc[j + s];
      dc[j] = x;
    }
    __syncthreads();
  }
}
// solution of mode k at row i from its solved column (Sherman-Morrison for
// x-periodic operators)
__device__ __forceinline__ float cr_value(const CrArgs &A, const float *dc, int k, int i) {
  float v = dc[i];
  if (A.cyclic && !(k == 0 && A.pin0 >= 0))
    v -= (dc[0] + A.gk[A.K + k] * dc[A.nx - 1]) * A.gk[k] * A.q[(size_t)i * A.K + k];
  return v;
}

// spec -> spec for the modes of work item `item` (staged coefficients, data in
// q.d).  Ends with a block barrier.
__device__ __forceinline__ void cr_solve(const CrArgs &A, const CrShared &q, float *__restrict__ spec, int k0, int g) {
  const int nx = A.nx, K = A.K, ncol = 2 * g;
  for (int t = threadIdx.x; t < nx * ncol; t += blockDim.x) {
    const int i = t / ncol, col = t - i * ncol;
    const int k = k0 + (col >> 1);
    float v = spec[((size_t)i * K + k) * 2 + (col & 1)];
    if (A.pin0 >= 0 && k == 0 && i == A.pin0) v = 0.f;  // pinned row of the singular mode
    q.d[col * nx + i] = v;
  }
  __syncthreads();
  cr_levels<false>(A, q, k0, ncol);
  for (int t = threadIdx.x; t < nx * ncol; t += blockDim.x) {
    const int i = t / ncol, col = t - i * ncol;
    const int k = k0 + (col >> 1);
    spec[((size_t)i * K + k) * 2 + (col & 1)] = cr_value(A, q.d + col * nx, k, i);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) k_tridiag_cr(CrArgs A, const PoissonScal *__restrict__ sc) {
  pdl_wait();
  extern __shared__ float fsh[];  // CrShared (column = 2 (k - k0) + part)
  if (sc->done) return;
  const int k0 = blockIdx.x * A.G, g = min(A.G, A.K - k0);
  const CrShared q = cr_shared(A, fsh);
  cr_stage(A, q, k0, g);
  cr_solve(A, q, A.spec, k0, g);
}

// spec -> δ (nx, ny) by the inverse of k_fft_fwd for work item `item`; x +=
// δ on free rows.
template <bool DF, bool ODD>
__device__ __forceinline__ void fft_inv_item(int item, const float2 *__restrict__ spec, int nx, const FftPlan &F,
                                             int TP, const uint16_t *__restrict__ cls, float2 *__restrict__ xd,
                                             double *__restrict__ x64, float2 *base) {
  const int N = F.N, S = N + 1, W = 2 * TP, K = (N >> 1) + 1;
  const int i0 = item * W;
  const FftShared q = fft_shared<ODD>(base, TP, F);
  // the update's ϕ values and row classes, fetched before the transform
  constexpr int kPre = 8;
  float2 xp[kPre];
  double xq[kPre];
  bool freep[kPre];
#pragma unroll
  for (int u = 0; u < kPre; u++) {
    const int t = threadIdx.x + u * blockDim.x;
    const int j = t / W, c = t - j * W;
    const int i = i0 + c;
    freep[u] = false;
    xp[u] = make_float2(0.f, 0.f);
    xq[u] = 0.0;
    if (t < W * N && i < nx) {
      const size_t kk = i + (size_t)nx * j;
      freep[u] = !(cls[kk] & kFixedBit);
      if (freep[u]) {
        if (DF) xp[u] = xd[kk];
        else xq[u] = x64[kk];
      }
    }
  }
  for (int t = threadIdx.x; t < TP * N; t += blockDim.x) {
    const int p = ODD ? t / N : t >> F.log2p, k = ODD ? t - p * N : t & (N - 1);
    const int ia = i0 + 2 * p;
    const bool hi = k >= K;
    const int kk = hi ? N - k : k;
    float2 a = make_float2(0.f, 0.f), b = a;
    if (ia < nx) a = spec[(size_t)ia * K + kk];
    if (ia + 1 < nx) b = spec[(size_t)(ia + 1) * K + kk];
    if (hi) {
      a.y = -a.y;
      b.y = -b.y;
    }
    q.buf[p * S + fft_pos<ODD>(k, F)] = make_float2(a.x - b.y, a.y + b.x);
  }
  __syncthreads();
  const float2 *zb = fft_columns<ODD>(q.buf, q.alt, TP, F, S, q.tw, q.twm, true);
  const float invN = 1.f / (float)N;  // (exact for a power of two)
#pragma unroll
  for (int u = 0; u < kPre; u++) {
    const int t = threadIdx.x + u * blockDim.x;
    const int j = t / W, c = t - j * W;
    const int i = i0 + c;
    if (freep[u]) {
      const float2 z = zb[(c >> 1) * S + j];
      const float dz = (c & 1 ? z.y : z.x) * invN;
      if (DF) xd[i + (size_t)nx * j] = df_add_f(xp[u], dz);
      else x64[i + (size_t)nx * j] = xq[u] + (double)dz;
    }
  }
  for (int t = threadIdx.x + kPre * blockDim.x; t < W * N; t += blockDim.x) {
    const int j = t / W, c = t - j * W;
    const int i = i0 + c;
    if (i < nx) {
      const size_t kk = i + (size_t)nx * j;
      if (!(cls[kk] & kFixedBit)) {
        const float2 z = zb[(c >> 1) * S + j];
        const float dz = (c & 1 ? z.y : z.x) * invN;
        if (DF) xd[kk] = df_add_f(xd[kk], dz);
        else x64[kk] += (double)dz;
      }
    }
  }
}

template <bool DF, bool ODD>
__global__ void __launch_bounds__(256) k_fft_inv_update(const float2 *__restrict__ spec, int nx, FftPlan F, int TP,
                                                        const uint16_t *__restrict__ cls, float2 *__restrict__ xd,
                                                        double *__restrict__ x64, const PoissonScal *__restrict__ sc) {
  pdl_wait();
  extern __shared__ float2 fbuf[];
  if (sc->done) return;
  fft_inv_item<DF, ODD>(blockIdx.x, spec, nx, F, TP, cls, xd, x64, fbuf);
}

// mean-zero projection of x over nodes (singular case)
__global__ void k_sum_x(const double *__restrict__ x, int nn, double *__restrict__ part) {
  pdl_wait();
  __shared__ double sh[40];
  double v = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) v += x[k];
  double t = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}
__global__ void k_shift_x(double *__restrict__ x, int nn, const double *__restrict__ part, int nparts) {
  pdl_wait();
  __shared__ double sh[40];
  double s = sum_partials(part, nparts, sh);
  const double m = s / nn;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) x[k] -= m;
}

// ---------------- Jacobi-preconditioned CG ----------------
// S p on free rows (p = 0 on fixed rows)
__device__ __forceinline__ double apply_S(const OpView &op, const RowClass &C, const double *__restrict__ v, int k) {
  int w, e, s, n;
  nbr(k, op.nx, op.ny, w, e, s, n);
  double a = C.c0 * v[k] + C.cW * v[w] + C.cE * v[e] + C.cS * v[s] + C.cN * v[n];
  return -C.d * a;
}

__global__ void k_cg_init(OpView op, const double *__restrict__ r, double *__restrict__ z, double *__restrict__ p,
                          double *__restrict__ part, int nn) {
  __shared__ double sh[40];
  double v = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const RowClass &C = op.classes[op.cls[k] & kClassMask];
    double zz = C.fixed ? 0.0 : r[k] / (-C.d * C.c0);
    z[k] = zz;
    p[k] = zz;
    v += r[k] * zz;
  }
  double t = block_sum(v, sh);
  if (threadIdx.x == 0) part[2 * kPartials + blockIdx.x] = t;  // summed by k_cg_rz0
}

// rz of the iteration is held in sc->rz; the kernel that forms the next one
// stores it in sc->rz_new and this kernel (one per iteration, which reads
// neither) moves it to sc->rz: no block of a kernel reads a scalar another
// block of the same kernel writes.
__global__ void k_cg_ap(OpView op, const double *__restrict__ p, double *__restrict__ ap, double *__restrict__ part,
                        int nn, PoissonScal *__restrict__ sc) {
  __shared__ double sh[40];
  if (sc->done) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->rz = sc->rz_new;
  double v = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const RowClass &C = op.classes[op.cls[k] & kClassMask];
    double a = C.fixed ? 0.0 : apply_S(op, C, p, k);
    ap[k] = a;
    v += p[k] * a;
  }
  double t = block_sum(v, sh);
  if (threadIdx.x == 0) part[kPartials + blockIdx.x] = t;
}

// α = rz/pAp; x += αp; r -= αAp; z = r/diag; partial rz_new and ||res||²
__global__ void k_cg_update(OpView op, double *__restrict__ x, double *__restrict__ r, double *__restrict__ z,
                            const double *__restrict__ p, const double *__restrict__ ap, double *__restrict__ part,
                            int nparts, int nn, const PoissonScal *__restrict__ sc) {
  __shared__ double sh[40];
  if (sc->done) return;
  const double rz = sc->rz;
  const double pap = sum_partials(part + kPartials, nparts, sh);
  const double alpha = pap != 0 ? rz / pap : 0.0;
  double v = 0, w2 = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const RowClass &C = op.classes[op.cls[k] & kClassMask];
    if (C.fixed) {
      z[k] = 0.0;
      continue;
    }
    x[k] += alpha * p[k];
    double rr = r[k] - alpha * ap[k];
    r[k] = rr;
    double zz = rr / (-C.d * C.c0);
    z[k] = zz;
    v += rr * zz;
    double res = rr / C.d;
    w2 += res * res;
  }
  double t = block_sum(v, sh);
  double t2 = block_sum(w2, sh);
  if (threadIdx.x == 0) {
    part[2 * kPartials + blockIdx.x] = t;
    part[3 * kPartials + blockIdx.x] = t2;
  }
}

// β = rz_new/rz; p = z + βp; convergence on the unscaled residual
__global__ void k_cg_dir(OpView op, const double *__restrict__ z, double *__restrict__ p, double *__restrict__ part,
                         int nparts, int nn, PoissonScal *sc, double rtol2) {
  __shared__ double sh[40];
  if (sc->done) return;
  const double rz = sc->rz;
  const double rzn = sum_partials(part + 2 * kPartials, nparts, sh);
  const double res2 = sum_partials(part + 3 * kPartials, nparts, sh);
  const double beta = rz != 0 ? rzn / rz : 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) p[k] = z[k] + beta * p[k];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->rz_new = rzn;  // moved to sc->rz by the next k_cg_ap
    sc->res2 = res2;
    sc->relres = sc->rhs2 > 0 ? sqrt(res2 / sc->rhs2) : sqrt(res2);
    sc->iters += 1;
    if ((sc->rhs2 > 0 && res2 <= rtol2 * sc->rhs2) || res2 == 0.0) sc->done = 1;
  }
}

// rz of the first iteration (partials of k_cg_init / k_pcg_init in part[2K..])
__global__ void k_cg_rz0(const double *__restrict__ part, int nparts, PoissonScal *sc) {
  __shared__ double sh[40];
  const double t = sum_partials(part + 2 * kPartials, nparts, sh);
  if (threadIdx.x == 0) sc->rz_new = t;
}

// ---- flexible PCG with the multigrid preconditioner (multigrid.cu) ----
// Iteration: k_pcg_ap (direction, S p, alpha), k_pcg_update (x, r, the
// convergence test), the cycle z = M^-1 r, whose last kernel also forms z.r and
// z.Sp and beta (pcg_finish_dots).  A converged iteration runs no cycle.

// p = z + beta p, ap = S p, alpha = rz / p.Sp.  A block forms p on a 32 x 16 tile
// and a halo of one node in shared memory, one thread per node (1.2x the
// additions), so that the direction update costs no pass of its own; p
// alternates between two buffers (s->par), since neighbouring blocks read the
// old one.  Bound by GB300's FP64 rate (~7 FP64 instructions per node, 12 us at
// 1024 x 1024) and its memory traffic: 26 us there with cold caches, where the
// direction and S p kernels it replaces took 43 us.
constexpr int kApX = 32, kApY = 16, kApW = kApX + 2, kApH = kApY + 2;
constexpr int kApThreads = (kApW * kApH + 31) / 32 * 32;
__global__ void __launch_bounds__(kApThreads) k_pcg_ap(OpView op, const double *__restrict__ z,
                                                       double *__restrict__ pa, double *__restrict__ pb,
                                                       double *__restrict__ ap, double *__restrict__ part,
                                                       const int *skip, PcgScal *s) {
  __shared__ double sp[kApThreads];
  __shared__ double red[kApThreads];
  const int nx = op.nx, ny = op.ny;
  const int l = threadIdx.x, ly = l / kApW, lx = l - kApW * ly;
  const int tiles_x = (nx + kApX - 1) / kApX, tiles = tiles_x * ((ny + kApY - 1) / kApY);
  pdl_wait();
  if (*skip) return;
  const double beta = s->beta;
  const int par = s->par;
  const double *po = par ? pb : pa;
  double *pn = par ? pa : pb;
  double v = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int ty = tile / tiles_x;
    const int gx = (tile - ty * tiles_x) * kApX - 1 + lx, gy = ty * kApY - 1 + ly;
    const int k = wrap_any(gx, nx) + nx * wrap_any(gy, ny);
    const bool own = lx >= 1 && lx <= kApX && ly >= 1 && ly <= kApY && gx < nx && gy < ny;
    const RowClass &C = op.classes[op.cls[k] & kClassMask];
    double p = z[k];
    if (beta != 0) p = fma(beta, po[k], p);
    sp[l] = p;
    __syncthreads();
    if (own) {
      double a = C.s0 * p;  // (zeros on identity rows)
      a = fma(C.sW, sp[l - 1], a);
      a = fma(C.sE, sp[l + 1], a);
      a = fma(C.sS, sp[l - kApW], a);
      a = fma(C.sN, sp[l + kApW], a);
      pn[k] = p;
      ap[k] = a;
      v = fma(p, a, v);
    }
    __syncthreads();
  }
  const double part_v[1] = {v};
  double pap[1];
  if (grid_sums<1>(part_v, red, part, &s->tick_ap, pap) && threadIdx.x == 0)
    s->alpha = pap[0] != 0 ? s->rz / pap[0] : 0.0;
}

// x += alpha p; r -= alpha S p; the convergence test on the unscaled residual.
// A thread takes four nodes with all their loads in flight together.
__global__ void __launch_bounds__(256) k_pcg_update(OpView op, double *__restrict__ x, double *__restrict__ r,
                                                    const double *__restrict__ pa, const double *__restrict__ pb,
                                                    const double *__restrict__ ap, double *__restrict__ part, int nn,
                                                    PoissonScal *sc, PcgScal *s, double rtol2) {
  pdl_wait();
  if (sc->done) return;
  __shared__ double red[256];
  const double alpha = s->alpha;
  const double *p = s->par ? pa : pb;  // the buffer k_pcg_ap wrote
  double w2 = 0;
  constexpr int U = 4;
  const int stride = gridDim.x * blockDim.x;
  for (int k0 = blockIdx.x * blockDim.x + threadIdx.x; k0 < nn; k0 += U * stride) {
    double xk[U], rk[U], pk[U], ak[U], dk[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * stride;
      dk[u] = 0.0;
      if (k < nn) {
        const unsigned ck = op.cls[k];
        xk[u] = x[k];
        rk[u] = r[k];
        pk[u] = p[k];
        ak[u] = ap[k];
        if (!(ck & kFixedBit)) dk[u] = op.classes[ck & kClassMask].inv_d;
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = k0 + u * stride;
      if (dk[u] != 0.0) {  // a free row
        x[k] = fma(alpha, pk[u], xk[u]);
        const double rr = fma(-alpha, ak[u], rk[u]);
        r[k] = rr;
        const double res = rr * dk[u];
        w2 = fma(res, res, w2);
      }
    }
  }
  const double part_w[1] = {w2};
  double res[1];
  if (grid_sums<1>(part_w, red, part, &s->tick_up, res) && threadIdx.x == 0) {
    const double res2 = res[0];
    s->par ^= 1;
    sc->res2 = res2;
    sc->relres = sc->rhs2 > 0 ? sqrt(res2 / sc->rhs2) : sqrt(res2);
    sc->iters += 1;
    if ((sc->rhs2 > 0 && res2 <= rtol2 * sc->rhs2) || res2 == 0.0) sc->done = 1;
  }
}

// z.r and z.Sp of a hierarchy of one level (its coarsest solve forms no sums)
__global__ void __launch_bounds__(256) k_pcg_dots(const double *__restrict__ r, const double *__restrict__ z, int nn,
                                                  const int *skip, PcgDots D) {
  pdl_wait();
  if (*skip) return;
  __shared__ double red[512];
  double a = 0, b = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    a = fma(z[k], r[k], a);
    if (!D.init) b = fma(z[k], D.ap[k], b);
  }
  pcg_finish_dots(D, a, b, red);
}

// ===========================================================================
// host: assembly
// ===========================================================================
static Poisson *poisson_new(Ctx *c, double eps0) {
  Poisson *P = new Poisson();
  P->nx = c->nx;
  P->ny = c->ny;
  P->nn = c->nn;
  P->dx = c->g.dx;
  P->dy = c->g.dy;
  P->eps0 = eps0;
  const int nx = P->nx, ny = P->ny;
  P->C.assign((size_t)P->nn * 7, 0.0);
  P->bfix.assign(P->nn, 0.0);
  P->rho_dof.assign(P->nn, 1);
  P->er.assign((size_t)(nx + 1) * (ny + 1), 1.0);
  // create_generalized_poisson_solver (:42-61)
  for (int j = 0; j < ny; j++)
    for (int i = 0; i < nx; i++) {
      double *R = &P->C[(size_t)(i + nx * j) * 7];
      if (i < nx - 1) { R[0] -= 1.0; R[2] += 1.0; }
      if (i > 0) { R[0] -= 1.0; R[1] += 1.0; }
      if (j < ny - 1) { R[0] -= 1.0; R[4] += 1.0; }
      if (j > 0) { R[0] -= 1.0; R[3] += 1.0; }
    }
  const double h2 = P->dx * P->dx;  // A ./= grid.Δh[1]^2 (:65)
  for (auto &v : P->C) v /= h2;
  return P;
}

static double ER(const Poisson *P, int i1, int j1) {  // εr[i,j] with 1-based indices
  return P->er[(size_t)(i1 - 1) + (size_t)(P->nx + 1) * (j1 - 1)];
}

static void assemble_periodic(Poisson *P, int axis) {
  const int nx = P->nx, ny = P->ny;
  if (axis == 1) {
    const int js[2] = {1, ny};  // Julia iterates the tuple (1, ny)
    for (int t = 0; t < 2; t++) {
      const int j = js[t];
      for (int i = 1; i <= nx; i++) {
        double *R = &P->C[(size_t)((i - 1) + nx * (j - 1)) * 7];
        if (j == ny) {
          double cc = (0.5 * ER(P, i + 1, j + 1) + 0.5 * ER(P, i, j + 1)) / (P->dx * P->dx);
          R[0] -= cc;
          R[6] += cc;
        }
        if (j == 1) {
          double cc = (0.5 * ER(P, i + 1, j) + 0.5 * ER(P, i, j)) / (P->dx * P->dx);
          R[0] -= cc;
          R[6] += cc;
        }
      }
    }
  } else {
    for (int j = 1; j <= ny; j++) {
      const int is[2] = {1, nx};
      for (int t = 0; t < 2; t++) {
        const int i = is[t];
        double *R = &P->C[(size_t)((i - 1) + nx * (j - 1)) * 7];
        if (i == nx) {
          double cc = (0.5 * ER(P, i + 1, j + 1) + 0.5 * ER(P, i + 1, j)) / (P->dy * P->dy);
          R[0] -= cc;
          R[5] += cc;
        }
        if (i == 1) {
          double cc = (0.5 * ER(P, i, j) + 0.5 * ER(P, i, j + 1)) / (P->dy * P->dy);
          R[0] -= cc;
          R[5] += cc;
        }
      }
    }
  }
}

static void assemble_dirichlet(Poisson *P, const uint8_t *nodes, double phi0) {
  for (int r = 0; r < P->nn; r++) {
    if (!nodes[r]) continue;
    double *R = &P->C[(size_t)r * 7];
    for (int s = 0; s < 7; s++) R[s] = 0.0;
    for (auto &col : P->sig_cols) col[r] = 0.0;
    R[0] = 1.0;
    P->bfix[r] = phi0;
    P->rho_dof[r] = 0;
  }
}

// apply_neumann (generalized_poisson.jl:235-269).  gauss = false: the
// reference's rows exactly.  gauss = true: the same rows in the units of the
// stencil rows, i.e. the Gauss law of the electrode node's half (edge) or
// quarter (corner) cell with σ in C/m^2: the edge row is the reference's row
// divided by Δx with the σ coefficient 2/(ε0 Δx) (the reference's 2/Δx
// gradient row against a -ρ/ε0 right-hand side and an undivided σ mixes
// units), the corner row keeps its 1/Δ^2 coefficients and divides the σ
// coefficient by ε0.
static void assemble_neumann(Poisson *P, const uint8_t *nodes, int dof, bool gauss) {
  const int nx = P->nx, ny = P->ny;
  const double dx = P->dx, dy = P->dy;
  // edge-row ϕ divisor: Δx (reference), Δx Δx (Gauss form: 2 εr/(Δx Δx)
  // rounds like the stencil rows' 1/(Δx Δx), so the symmetrising scales stay
  // exact)
  const double ge = gauss ? dx * dx : dx;
  const double gs = gauss ? 1.0 / (P->eps0 * dx) : 1.0;   // edge-row σ scale
  const double gc = gauss ? 1.0 / P->eps0 : 1.0;          // corner-row σ scale
  auto N = [&](int i, int j) { return nodes[i + nx * j] != 0; };  // 0-based
  for (int j = 0; j < ny; j++)
    for (int i = 0; i < nx; i++) {
      if (!N(i, j)) continue;
      const bool a = i > 0 ? N(i - 1, j) : false;
      const bool b = i < nx - 1 ? N(i + 1, j) : false;
      const bool cc = j > 0 ? N(i, j - 1) : true;
      const bool d = j < ny - 1 ? N(i, j + 1) : true;
      const int r = i + nx * j;
      double *R = &P->C[(size_t)r * 7];
      std::vector<double> &S = P->sig_cols[dof - 1];
      if (cc == d && d == true && a == b && b == false) {
        const int ip = i == 0 ? i + 1 : i - 1;
        for (int s = 0; s < 7; s++) R[s] = 0.0;
        for (auto &col : P->sig_cols) col[r] = 0.0;
        R[0] -= 2 * ER(P, i + 1, j + 1) / ge;
        R[ip == i + 1 ? 2 : 1] += 2 * ER(P, ip + 1, j + 1) / ge;
        S[r] += 2 * gs;
      }
      if (cc != d) {
        const int ip = i == 0 ? i + 1 : i - 1;
        const int jp = cc ? j + 1 : j - 1;
        for (int s = 0; s < 7; s++) R[s] = 0.0;
        for (auto &col : P->sig_cols) col[r] = 0.0;
        const double e = ER(P, i + 1, j + 1);
        R[0] -= 4 * e / (3 * dx * dx);
        R[0] -= 4 * e / (3 * dy * dy);
        R[ip == i + 1 ? 2 : 1] += 4 * e / (3 * dx * dx);
        R[jp == j + 1 ? 4 : 3] += 4 * e / (3 * dy * dy);
        S[r] += (2.0 / 3.0) * (dx + dy) / (dx * dy) * gc;
      }
    }
}

// ===========================================================================
// host: device representation, symmetrisation, separable factorisation
// ===========================================================================
struct RowEff {
  double c0, cW, cE, cS, cN;
  int sig_dof;
  double sig_coef;
  bool fixed, rho;
};

static RowEff effective_row(const Poisson *P, int r) {
  const int nx = P->nx, ny = P->ny, i = r % nx, j = r / nx;
  const double *R = &P->C[(size_t)r * 7];
  RowEff e{};
  e.c0 = R[0];
  e.cW = R[1] + (i == 0 ? R[5] : 0.0);
  e.cE = R[2] + (i == nx - 1 ? R[5] : 0.0);
  e.cS = R[3] + (j == 0 ? R[6] : 0.0);
  e.cN = R[4] + (j == ny - 1 ? R[6] : 0.0);
  // nx == 1 / ny == 1 cannot occur (nx, ny >= 2)
  e.sig_dof = -1;
  e.sig_coef = 0;
  int nsig_here = 0;
  for (size_t k = 0; k < P->sig_cols.size(); k++)
    if (P->sig_cols[k][r] != 0.0) {
      e.sig_dof = (int)k;
      e.sig_coef = P->sig_cols[k][r];
      nsig_here++;
    }
  if (nsig_here > 1) e.sig_dof = -2;  // unsupported: flagged by the caller
  e.fixed = e.c0 == 1.0 && e.cW == 0 && e.cE == 0 && e.cS == 0 && e.cN == 0 && e.sig_dof == -1;
  e.rho = P->rho_dof[r] != 0;
  return e;
}

static int fft_smem_attr(Ctx *c);

// Largest odd factor of ny solved directly: its dense DFTs cost the square.  Steps
// at 1e-8, 200 k particles, µs direct (corrections) / multigrid CG: nx = 301: 74 (1)
// / 482 at ny = 255, 200 (2) / 580 at 1023, 349 (1) / 719 at 1533, 478 (1) / 768 at
// 2039, 1558 (1) / 1184 at 4093; nx = 2048: 246 (2) / 834, 1286 (2) / 1804, 2098 (1)
// / 2617, 2748 (1) / 2653.  A second correction would cost more than CG from about
// 1500 on.  Singular operators, whose CG has no multigrid, win at any factor (ny =
// 4093: 3.3-20 ms a solve against 117-1450).
constexpr int kMaxOdd = 1024;
static int odd_factor(int n) {
  while (n % 2 == 0) n /= 2;
  return n;
}

constexpr double kReportRtol = 1e-8;  // stands for a tolerance that is not known yet: the default one

// Whether a separable operator is solved directly (FFT along y, cyclic
// reduction along x) for tolerance rtol.  A power-of-two ny always is.  Any
// other ny is down to a tolerance of 1e-9 (301 x 97 slab: a step took
// 3.66 ms with multigrid CG, 0.10 ms directly); tighter ones keep CG, whose
// recursively updated residual reaches tolerances below the rounding floor
// of the recomputed one, and so does a context with a learned warm start,
// which works on CG solves, and an operator whose direct solve has stalled at this
// tolerance (solve_sync): the floor of the recomputed residual grows with nx^2 for a
// smooth ρ (uniform ρ: 6e-10 at 4096 columns, 4.6e-9 at 12000).
static bool direct_solve(Ctx *c, const Poisson *P, double rtol) {
  return P->sep_form && (power_of_two(P->ny) || (!c->lws && rtol >= 1e-9 && rtol > P->stalled));
}

// Effective rows and the symmetrising scale d of the free rows (breadth-first
// propagation); *any_fixed: some row is an identity row.
static int scaled_rows(Ctx *c, const Poisson *P, std::vector<RowEff> &rows, std::vector<double> &d, bool *any_fixed) {
  const int nx = P->nx, ny = P->ny, nn = P->nn;
  rows.resize(nn);
  for (int r = 0; r < nn; r++) {
    rows[r] = effective_row(P, r);
    if (rows[r].sig_dof == -2) return set_err(c, ISKRA_EINVAL, "a row couples to more than one σ dof");
  }
  // neighbor indices (wrapped) for the effective coefficients
  auto nb = [&](int r, int which) {
    const int i = r % nx, j = r / nx;
    switch (which) {
      case 0: return i > 0 ? r - 1 : r + nx - 1;
      case 1: return i < nx - 1 ? r + 1 : r - nx + 1;
      case 2: return j > 0 ? r - nx : r + nx * (ny - 1);
      default: return j < ny - 1 ? r + nx : r - nx * (ny - 1);
    }
  };
  auto coef_to = [&](int r, int col) {  // A[r, col] for a neighbor column
    const RowEff &e = rows[r];
    double a = 0;
    if (nb(r, 0) == col) a += e.cW;
    if (nb(r, 1) == col) a += e.cE;
    if (nb(r, 2) == col) a += e.cS;
    if (nb(r, 3) == col) a += e.cN;
    return a;
  };
  d.assign(nn, 0.0);
  std::vector<int> queue;
  queue.reserve(nn);
  *any_fixed = false;
  for (int r = 0; r < nn; r++) *any_fixed |= rows[r].fixed;
  for (int r0 = 0; r0 < nn; r0++) {
    if (rows[r0].fixed || d[r0] != 0.0) continue;
    d[r0] = 1.0;
    queue.clear();
    queue.push_back(r0);
    for (size_t h = 0; h < queue.size(); h++) {
      const int r = queue[h];
      for (int w = 0; w < 4; w++) {
        const int cidx = nb(r, w);
        if (cidx == r || rows[cidx].fixed) continue;
        const double arc = coef_to(r, cidx), acr = coef_to(cidx, r);
        if (arc == 0.0 && acr == 0.0) continue;
        if (arc == 0.0 || acr == 0.0)
          return set_err(c, ISKRA_EINVAL, "boundary setup gives a non-symmetrizable operator");
        const double want = d[r] * arc / acr;
        if (d[cidx] == 0.0) {
          d[cidx] = want;
          queue.push_back(cidx);
        } else if (std::fabs(d[cidx] - want) > 1e-9 * std::fabs(want)) {
          return set_err(c, ISKRA_EINVAL, "boundary setup gives a non-symmetrizable operator");
        }
      }
    }
  }
  return ISKRA_OK;
}

// The multigrid hierarchy of the CG path, from the scaled rows (host work).
static int build_mg(Ctx *c, Poisson *P, const std::vector<RowEff> &rows, const std::vector<double> &d) {
  const int nn = P->nn;
  std::vector<double> s0(nn, 0.0), sW(nn, 0.0), sE(nn, 0.0), sS(nn, 0.0), sN(nn, 0.0);
  std::vector<char> free_row(nn, 0);
  int per_x = 0, per_y = 0;
  for (int r = 0; r < nn; r++) {
    per_x |= P->C[(size_t)r * 7 + 5] != 0.0;
    per_y |= P->C[(size_t)r * 7 + 6] != 0.0;
    const RowEff &e = rows[r];
    if (e.fixed) continue;
    free_row[r] = 1;
    s0[r] = -d[r] * e.c0;
    sW[r] = -d[r] * e.cW;
    sE[r] = -d[r] * e.cE;
    sS[r] = -d[r] * e.cS;
    sN[r] = -d[r] * e.cN;
  }
  return mg_build(c, P->nx, P->ny, s0, sW, sE, sS, sN, free_row, per_x, per_y, &P->mg);
}

static int build_device(Ctx *c, Poisson *P) {
  const int nx = P->nx, ny = P->ny, nn = P->nn;
  std::vector<RowEff> rows;
  std::vector<double> d;
  bool any_fixed = false;
  {
    const int rc = scaled_rows(c, P, rows, d, &any_fixed);
    if (rc) return rc;
  }
  for (int r = 0; r < nn; r++)
    if (!rows[r].fixed && (!(d[r] > 0) || !(-d[r] * rows[r].c0 > 0)))
      return set_err(c, ISKRA_EINVAL, "assembled operator is not definite on its free rows");
  // singular: no fixed row and every free row sums to zero
  bool singular = !any_fixed;
  if (singular) {
    double mx = 0;
    for (int r = 0; r < nn; r++) mx = std::max(mx, std::fabs(rows[r].c0));
    for (int r = 0; r < nn && singular; r++) {
      const RowEff &e = rows[r];
      if (std::fabs(e.c0 + e.cW + e.cE + e.cS + e.cN) > 1e-12 * mx) singular = false;
    }
  }
  P->singular = singular;
  P->dsum = 0;
  for (int r = 0; r < nn; r++)
    if (!rows[r].fixed) P->dsum += d[r];
  // classes
  bool rho_fixed = false;
  // (a row mostly repeats the one before it: the table is searched only where it
  // does not.  Searched for every row, a 512 x 512 operator's first step took 29.5 ms
  // instead of 23.8.)
  typedef std::array<double, 10> RowKey;
  std::map<RowKey, int> cmap;
  std::vector<RowClass> classes;
  std::vector<uint16_t> cls(nn);
  RowKey prev{};
  int prev_id = -1;
  for (int r = 0; r < nn; r++) {
    const RowEff &e = rows[r];
    const RowKey key = {e.c0, e.cW, e.cE, e.cS, e.cN, e.fixed ? 1.0 : 0.0, e.rho ? 1.0 : 0.0,
                               (double)e.sig_dof, e.sig_coef, e.fixed ? 0.0 : d[r]};
    int id = prev_id;
    const bool repeats = prev_id >= 0 && key == prev;
    auto it = repeats ? cmap.end() : cmap.find(key);
    if (repeats) {
    } else if (it == cmap.end()) {
      id = (int)classes.size();
      if (id > (int)kClassMask) return set_err(c, ISKRA_EINVAL, "too many distinct operator rows");
      cmap[key] = id;
      RowClass rc{};
      rc.c0 = e.c0;
      rc.cW = e.cW;
      rc.cE = e.cE;
      rc.cS = e.cS;
      rc.cN = e.cN;
      rc.d = e.fixed ? 1.0 : d[r];
      rc.inv_d = 1.0 / rc.d;
      rc.nd32 = (float)(-rc.d);
      auto split = [](double v) {
        const float h = (float)v;
        return make_float2(h, (float)(v - (double)h));
      };
      rc.c0f = split(e.c0);
      rc.cWf = split(e.cW);
      rc.cEf = split(e.cE);
      rc.cSf = split(e.cS);
      rc.cNf = split(e.cN);
      if (!e.fixed) {
        rc.s0 = -rc.d * e.c0;
        rc.sW = -rc.d * e.cW;
        rc.sE = -rc.d * e.cE;
        rc.sS = -rc.d * e.cS;
        rc.sN = -rc.d * e.cN;
      }
      rc.sig_coef = e.sig_coef;
      rc.sig_dof = e.sig_dof;
      rc.fixed = e.fixed;
      rc.rho = e.rho;
      classes.push_back(rc);
    } else {
      id = it->second;
    }
    prev = key;
    prev_id = id;
    cls[r] = (uint16_t)(id | (e.fixed ? kFixedBit : 0u));
    rho_fixed |= e.fixed && e.rho;
  }
  P->nclass = (int)classes.size();
  P->rho_fixed = rho_fixed;
  // ---- separability: per column i, every j gives the same scaled row ----
  bool sep = P->method == 0 && ny >= 2 && ny <= 4096 && (singular || odd_factor(ny) <= kMaxOdd);
  std::vector<double> s0(nx), sW(nx), sE(nx), ey(nx);
  std::vector<int> colfixed(nx);
  for (int i = 0; i < nx && sep; i++) {
    const RowEff &e0 = rows[i];
    colfixed[i] = e0.fixed;
    for (int j = 1; j < ny && sep; j++) {
      const RowEff &e = rows[i + nx * j];
      if (e.fixed != e0.fixed) sep = false;
      if (!e.fixed && (e.c0 != e0.c0 || e.cW != e0.cW || e.cE != e0.cE || e.cS != e0.cS || e.cN != e0.cN ||
                       d[i + nx * j] != d[i]))
        sep = false;
    }
    if (!sep) break;
    if (!e0.fixed) {
      if (e0.cS != e0.cN) sep = false;
      s0[i] = -d[i] * e0.c0;
      sW[i] = -d[i] * e0.cW;
      sE[i] = -d[i] * e0.cE;
      ey[i] = -d[i] * e0.cS;
    }
  }
  P->sep_form = sep;
  P->stalled = 0;
  P->separable = direct_solve(c, P, kReportRtol);
  // ---- multigrid preconditioner of the CG path ----
  mg_destroy(P->mg);
  P->mg = nullptr;
  if (P->pcg_graph) cudaGraphExecDestroy(P->pcg_graph);
  P->pcg_graph = nullptr;
  if (!P->separable && !singular && P->method != 1) {
    const int rc = build_mg(c, P, rows, d);
    if (rc) return rc;
  }
  // ---- device upload ----
  cudaStream_t st = c->stream;
  ISKRA_CUDA(c, cudaStreamSynchronize(st));
  cudaFree(P->cls);
  cudaFree(P->classes);
  P->cls = nullptr;
  P->classes = nullptr;
  ISKRA_CUDA(c, cudaMalloc(&P->cls, nn * sizeof(uint16_t)));
  ISKRA_CUDA(c, cudaMalloc(&P->classes, classes.size() * sizeof(RowClass)));
  ISKRA_CUDA(c, cudaMemcpy(P->cls, cls.data(), nn * sizeof(uint16_t), cudaMemcpyHostToDevice));
  ISKRA_CUDA(c, cudaMemcpy(P->classes, classes.data(), classes.size() * sizeof(RowClass), cudaMemcpyHostToDevice));
  if (!P->bfix_d) ISKRA_CUDA(c, cudaMalloc(&P->bfix_d, nn * sizeof(double)));
  ISKRA_CUDA(c, cudaMemcpy(P->bfix_d, P->bfix.data(), nn * sizeof(double), cudaMemcpyHostToDevice));
  const int nsig = (int)P->sig_b.size();
  if (P->sigma_d && P->nsig > 0) {
    // the device σ values are authoritative (the circuit kernel updates them)
    ISKRA_CUDA(c, cudaMemcpy(P->sig_b.data(), P->sigma_d, std::min(nsig, P->nsig) * sizeof(double),
                             cudaMemcpyDeviceToHost));
  }
  if (nsig != P->nsig) {
    cudaFree(P->sigma_d);
    P->sigma_d = nullptr;
    P->nsig = nsig;
  }
  if (!P->sigma_d) ISKRA_CUDA(c, cudaMalloc(&P->sigma_d, (nsig > 0 ? nsig : 1) * sizeof(double)));
  if (nsig) ISKRA_CUDA(c, cudaMemcpy(P->sigma_d, P->sig_b.data(), nsig * sizeof(double), cudaMemcpyHostToDevice));
  if (P->df_mode && P->x_stale) {  // the FP64 view takes over the double-float state before a rebuild
    k_df_to_x<<<std::max(1, std::min(c->num_sms * 2, (nn + 255) / 256)), 256, 0, c->stream>>>(P->xd, P->x, nn);
    ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  P->df_mode = false;
  P->x_stale = false;
  if (!P->x) {
    ISKRA_CUDA(c, cudaMalloc(&P->x, nn * sizeof(double)));
    ISKRA_CUDA(c, cudaMemset(P->x, 0, nn * sizeof(double)));
    ISKRA_CUDA(c, cudaMalloc(&P->r, nn * sizeof(double)));
    ISKRA_CUDA(c, cudaMalloc(&P->z, nn * sizeof(double)));
    ISKRA_CUDA(c, cudaMalloc(&P->p, nn * sizeof(double)));
    ISKRA_CUDA(c, cudaMalloc(&P->ap, nn * sizeof(double)));
    ISKRA_CUDA(c, cudaMalloc(&P->p2, nn * sizeof(double)));
    ISKRA_CUDA(c, cudaMalloc(&P->pcg, sizeof(PcgScal)));
    ISKRA_CUDA(c, cudaMemset(P->pcg, 0, sizeof(PcgScal)));
    ISKRA_CUDA(c, cudaMalloc(&P->part, 4 * kPartials * sizeof(double)));
    ISKRA_CUDA(c, cudaMalloc(&P->scal, sizeof(PoissonScal)));
    ISKRA_CUDA(c, cudaMallocHost(&P->scal_h, sizeof(PoissonScal)));
    ISKRA_CUDA(c, cudaMemset(P->scal, 0, sizeof(PoissonScal)));
  }
  // drives
  cudaFree(P->drive_node);
  cudaFree(P->drive_group);
  cudaFree(P->drive_par);
  P->drive_node = nullptr;
  P->drive_group = nullptr;
  P->drive_par = nullptr;
  {
    std::vector<int> dn, dg;
    std::vector<double> dp;
    for (size_t g = 0; g < P->drives.size(); g++) {
      for (int n : P->drives[g].nodes) {
        dn.push_back(n);
        dg.push_back((int)g);
      }
      dp.insert(dp.end(), {P->drives[g].amp, P->drives[g].freq, P->drives[g].phase, P->drives[g].dc});
    }
    P->ndrive_nodes = (int)dn.size();
    P->ndrive = (int)P->drives.size();
    if (!dn.empty()) {
      ISKRA_CUDA(c, cudaMalloc(&P->drive_node, dn.size() * sizeof(int)));
      ISKRA_CUDA(c, cudaMalloc(&P->drive_group, dg.size() * sizeof(int)));
      ISKRA_CUDA(c, cudaMalloc(&P->drive_par, dp.size() * sizeof(double)));
      ISKRA_CUDA(c, cudaMemcpy(P->drive_node, dn.data(), dn.size() * sizeof(int), cudaMemcpyHostToDevice));
      ISKRA_CUDA(c, cudaMemcpy(P->drive_group, dg.data(), dg.size() * sizeof(int), cudaMemcpyHostToDevice));
      ISKRA_CUDA(c, cudaMemcpy(P->drive_par, dp.data(), dp.size() * sizeof(double), cudaMemcpyHostToDevice));
    }
  }
  P->blocks = std::min(kPartials, std::max(1, std::min(c->num_sms * ISKRA_RES_BLOCKS_PER_SM, (nn + 255) / 256)));
  P->cg_blocks = std::min(kPartials, std::max(1, std::min(c->num_sms * 6, (nn + 255) / 256)));
  // ---- separable factorisation ----
  cudaFree(P->r32);
  cudaFree(P->spec);
  cudaFree(P->tw);
  cudaFree(P->low);
  cudaFree(P->up);
  cudaFree(P->inv);
  cudaFree(P->cp);
  cudaFree(P->q);
  cudaFree(P->gk);
  cudaFree(P->cr_fwd);
  cudaFree(P->cr_back);
  cudaFree(P->cr_backb);
  cudaFree(P->cr_top);
  P->cr_fwd = P->cr_back = nullptr;
  P->cr_backb = P->cr_top = nullptr;
  P->r32 = nullptr;
  P->spec = nullptr;
  P->tw = nullptr;
  P->low = P->up = P->inv = P->cp = P->q = P->gk = nullptr;
  if (sep) {
    const int N = ny, K = N / 2 + 1;
    P->N = N;
    P->K = K;
    P->log2p = 0;
    P->odd = N;
    while (P->odd % 2 == 0) {
      P->odd /= 2;
      P->log2p++;
    }
    // tridiagonal couplings per column (k-independent); fixed columns decouple
    std::vector<double> lo(nx, 0.0), upv(nx, 0.0);
    double corner_lo = 0.0, corner_up = 0.0;  // T[0][nx-1], T[nx-1][0]
    for (int i = 0; i < nx; i++) {
      if (colfixed[i]) continue;
      const int iw = i > 0 ? i - 1 : nx - 1, ie = i < nx - 1 ? i + 1 : 0;
      double w = colfixed[iw] ? 0.0 : sW[i];
      double e = colfixed[ie] ? 0.0 : sE[i];
      if (i == 0) {
        if (iw == ie) { e += w; w = 0; }  // nx == 2: wrap partner is the east neighbour
        corner_lo = w;
      } else {
        lo[i] = w;
      }
      if (i == nx - 1) {
        if (iw == ie) { lo[i] += e; e = 0; }
        corner_up = e;
      } else {
        upv[i] = e;
      }
    }
    const bool cyclic = corner_lo != 0.0 || corner_up != 0.0;
    P->cyclic = cyclic;
    const int pin = singular ? 0 : -1;  // singular => no fixed column, pin column 0 of mode 0
    P->pin_k0 = pin;
    std::vector<double> inv((size_t)nx * K), cpv((size_t)nx * K), qv(cyclic ? (size_t)nx * K : 1), gkv(2 * K, 0.0);
    int cr_levels = 0;
    while ((2 << cr_levels) <= nx) cr_levels++;  // L = floor(log2 nx)
    size_t cr_nf = 0, cr_nb = 0;
    for (int l = 0; l < cr_levels; l++) {
      cr_nf += nx >> (l + 1);
      cr_nb += ((nx >> l) + 1) >> 1;
    }
    std::vector<double2> cr_fwd(cr_nf * K), cr_back(cr_nb * K);
    std::vector<double> cr_backb(cr_nb * K), cr_top(K);
    for (int k = 0; k < K; k++) {
      double vfac = 0;
      const double ck = std::cos(2.0 * M_PI * k / N);
      std::vector<double> diag(nx), lk(lo), uk(upv);
      for (int i = 0; i < nx; i++) diag[i] = colfixed[i] ? 1.0 : s0[i] + 2.0 * ey[i] * ck;
      const bool pinned = (k == 0 && pin >= 0);
      const bool cyc = cyclic && !pinned;
      double gamma = 0;
      if (cyc) {
        gamma = -diag[0];
        vfac = corner_lo / gamma;  // v = [1, 0, ..., 0, β/γ], β = T[0][nx-1]
        gkv[K + k] = vfac;
        diag[0] -= gamma;
        diag[nx - 1] -= corner_up * corner_lo / gamma;
      }
      // Thomas factors (host: the Sherman-Morrison vector q below)
      double cprev = 0;
      for (int i = 0; i < nx; i++) {
        const size_t o = (size_t)i * K + k;
        if (pinned && i == pin) {
          inv[o] = 0.0;  // y_pin = 0
          cpv[o] = 0.0;
          cprev = 0.0;
          continue;
        }
        const double a = i > 0 ? lk[i] : 0.0;
        const double den = diag[i] - a * cprev;
        if (den == 0.0) return set_err(c, ISKRA_EINVAL, "singular tridiagonal mode in the Poisson factorisation");
        inv[o] = 1.0 / den;
        cprev = (i < nx - 1 ? uk[i] : 0.0) / den;
        cpv[o] = cprev;
      }
      // cyclic-reduction coefficients of T' (device solve).  Level l (stride
      // s = 2^l) updates rows i = (m+1)2s-1 from rows i-s, i+s and eliminates
      // rows j = (2m+1)s-1, which the back substitution recovers from rows j-s,
      // j+s; the last row left is 2^L-1, L = floor(log2 nx).
      {
        std::vector<double> a(nx), b(diag), cc(nx);
        for (int i = 0; i < nx; i++) {
          a[i] = i > 0 ? lk[i] : 0.0;
          cc[i] = i < nx - 1 ? uk[i] : 0.0;
        }
        if (pinned) {  // identity row; the kernel zeroes its right-hand side
          a[pin] = 0.0;
          cc[pin] = 0.0;
          b[pin] = 1.0;
        }
        size_t F = 0, B = 0;
        for (int l = 0; l < cr_levels; l++) {
          const int s = 1 << l;
          const int ecnt = ((nx >> l) + 1) >> 1, cnt = nx >> (l + 1);
          for (int m = 0; m < ecnt; m++) {
            const int j = (2 * m + 1) * s - 1;
            if (b[j] == 0.0) return set_err(c, ISKRA_EINVAL, "singular tridiagonal mode in the Poisson factorisation");
            const size_t o = (size_t)k * cr_nb + B + m;
            cr_back[o] = make_double2(a[j] / b[j], cc[j] / b[j]);
            cr_backb[o] = 1.0 / b[j];
          }
          for (int m = 0; m < cnt; m++) {
            const int i = (m + 1) * 2 * s - 1, im = i - s, ip = i + s;
            const double al = a[i] / b[im];
            const double ga = ip < nx ? cc[i] / b[ip] : 0.0;
            cr_fwd[(size_t)k * cr_nf + F + m] = make_double2(al, ga);
            b[i] = b[i] - al * cc[im] - (ip < nx ? ga * a[ip] : 0.0);
            a[i] = -al * a[im];
            cc[i] = ip < nx ? -ga * cc[ip] : 0.0;
          }
          F += cnt;
          B += ecnt;
        }
        const int top = (1 << cr_levels) - 1;
        if (b[top] == 0.0) return set_err(c, ISKRA_EINVAL, "singular tridiagonal mode in the Poisson factorisation");
        cr_top[k] = 1.0 / b[top];
      }
      if (cyc) {
        // q = T'^{-1} u, u = [γ, 0, ..., 0, α], α = T[nx-1][0]
        std::vector<double> y(nx), u(nx, 0.0);
        u[0] = gamma;
        u[nx - 1] += corner_up;
        for (int i = 0; i < nx; i++) {
          const size_t o = (size_t)i * K + k;
          const double a = i > 0 ? lk[i] : 0.0;
          y[i] = (u[i] - a * (i > 0 ? y[i - 1] : 0.0)) * inv[o];
        }
        for (int i = nx - 2; i >= 0; i--) y[i] -= cpv[(size_t)i * K + k] * y[i + 1];
        for (int i = 0; i < nx; i++) qv[(size_t)i * K + k] = y[i];
        gkv[k] = 1.0 / (1.0 + y[0] + vfac * y[nx - 1]);
      }
    }
    // device tables in FP32 (the correction runs in FP32)
    auto f32 = [](const std::vector<double> &v) { return std::vector<float>(v.begin(), v.end()); };
    auto f32x2 = [](const std::vector<double2> &v) {
      std::vector<float2> o(v.size());
      for (size_t n = 0; n < v.size(); n++) o[n] = make_float2((float)v[n].x, (float)v[n].y);
      return o;
    };
    std::vector<float2> tw(N / 2 + P->odd);
    for (int m = 0; m < N / 2; m++) {
      const double ang = -2.0 * M_PI * m / N;
      tw[m] = make_float2((float)std::cos(ang), (float)std::sin(ang));
    }
    for (int m = 0; m < P->odd; m++) {
      const double ang = -2.0 * M_PI * m / P->odd;
      tw[N / 2 + m] = make_float2((float)std::cos(ang), (float)std::sin(ang));
    }
    P->cr64.clear();
    for (const double2 &v : cr_fwd) P->cr64.insert(P->cr64.end(), {v.x, v.y});
    for (const double2 &v : cr_back) P->cr64.insert(P->cr64.end(), {v.x, v.y});
    P->cr64.insert(P->cr64.end(), cr_backb.begin(), cr_backb.end());
    P->cr64.insert(P->cr64.end(), cr_top.begin(), cr_top.end());
    cudaFree(P->cr64_d);
    P->cr64_d = nullptr;
    const std::vector<float> lo32 = f32(lo), up32 = f32(upv), inv32 = f32(inv), cp32 = f32(cpv), gk32 = f32(gkv),
                             q32 = f32(qv), backb32 = f32(cr_backb), top32 = f32(cr_top);
    const std::vector<float2> fwd32 = f32x2(cr_fwd), back32 = f32x2(cr_back);
    ISKRA_CUDA(c, cudaMalloc(&P->r32, nn * sizeof(float)));
    ISKRA_CUDA(c, cudaMalloc(&P->spec, (size_t)nx * K * sizeof(float2)));
    ISKRA_CUDA(c, cudaMalloc(&P->tw, tw.size() * sizeof(float2)));
    ISKRA_CUDA(c, cudaMalloc(&P->low, nx * sizeof(float)));
    ISKRA_CUDA(c, cudaMalloc(&P->up, nx * sizeof(float)));
    ISKRA_CUDA(c, cudaMalloc(&P->inv, (size_t)nx * K * sizeof(float)));
    ISKRA_CUDA(c, cudaMalloc(&P->cp, (size_t)nx * K * sizeof(float)));
    ISKRA_CUDA(c, cudaMalloc(&P->gk, 2 * K * sizeof(float)));
    ISKRA_CUDA(c, cudaMemcpy(P->tw, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice));
    ISKRA_CUDA(c, cudaMemcpy(P->low, lo32.data(), nx * sizeof(float), cudaMemcpyHostToDevice));
    ISKRA_CUDA(c, cudaMemcpy(P->up, up32.data(), nx * sizeof(float), cudaMemcpyHostToDevice));
    ISKRA_CUDA(c, cudaMemcpy(P->inv, inv32.data(), inv32.size() * sizeof(float), cudaMemcpyHostToDevice));
    ISKRA_CUDA(c, cudaMemcpy(P->cp, cp32.data(), cp32.size() * sizeof(float), cudaMemcpyHostToDevice));
    ISKRA_CUDA(c, cudaMemcpy(P->gk, gk32.data(), 2 * K * sizeof(float), cudaMemcpyHostToDevice));
    P->cr_levels = cr_levels;
    P->cr_nf = (int)cr_nf;
    P->cr_nb = (int)cr_nb;
    ISKRA_CUDA(c, cudaMalloc(&P->cr_fwd, std::max<size_t>(1, fwd32.size()) * sizeof(float2)));
    ISKRA_CUDA(c, cudaMalloc(&P->cr_back, std::max<size_t>(1, back32.size()) * sizeof(float2)));
    ISKRA_CUDA(c, cudaMalloc(&P->cr_backb, std::max<size_t>(1, backb32.size()) * sizeof(float)));
    ISKRA_CUDA(c, cudaMalloc(&P->cr_top, K * sizeof(float)));
    if (!fwd32.empty())
      ISKRA_CUDA(c, cudaMemcpy(P->cr_fwd, fwd32.data(), fwd32.size() * sizeof(float2), cudaMemcpyHostToDevice));
    if (!back32.empty()) {
      ISKRA_CUDA(c, cudaMemcpy(P->cr_back, back32.data(), back32.size() * sizeof(float2), cudaMemcpyHostToDevice));
      ISKRA_CUDA(c, cudaMemcpy(P->cr_backb, backb32.data(), backb32.size() * sizeof(float), cudaMemcpyHostToDevice));
    }
    ISKRA_CUDA(c, cudaMemcpy(P->cr_top, top32.data(), K * sizeof(float), cudaMemcpyHostToDevice));
    if (cyclic) {
      ISKRA_CUDA(c, cudaMalloc(&P->q, q32.size() * sizeof(float)));
      ISKRA_CUDA(c, cudaMemcpy(P->q, q32.data(), q32.size() * sizeof(float), cudaMemcpyHostToDevice));
    }
  }
  if (sep) {
    int rc = fft_smem_attr(c);
    if (rc) return rc;
    if (!P->xd) ISKRA_CUDA(c, cudaMalloc(&P->xd, nn * sizeof(float2)));
    if (!P->bd) ISKRA_CUDA(c, cudaMalloc(&P->bd, nn * sizeof(float2)));
  }
  if (!P->xh) ISKRA_CUDA(c, cudaMalloc(&P->xh, nn * sizeof(double)));
  // a new operator: the next step solve starts from ϕ itself
  ISKRA_CUDA(c, cudaMemset(&P->scal->hist, 0, sizeof(int)));
  ISKRA_CUDA(c, setup_copies_done());
  P->dirty = false;
  return ISKRA_OK;
}

static int fixed_to_x_now(Ctx *c);

int poisson_prepare(Ctx *c) {
  Poisson *P = c->ps;
  if (!P) return set_err(c, ISKRA_EINVAL, "no Poisson solver: call iskra_poisson_create");
  if (!P->dirty) return ISKRA_OK;
  invalidate_graphs(c);
  int rc = build_device(c, P);
  if (rc) return rc;
  return fixed_to_x_now(c);
}

static OpView opview(Poisson *P) {
  OpView o;
  o.cls = P->cls;
  o.classes = P->classes;
  o.bfix = P->bfix_d;
  o.sigma = P->sigma_d;
  o.nx = P->nx;
  o.ny = P->ny;
  o.nclass = P->nclass;
  return o;
}

static EOut eout(Ctx *c, bool on) {
  EOut e{};
  if (!on) return e;
  e.E32 = c->E32;
  e.idx2 = (float)(1.0 / (2 * c->g.dx));
  e.idx1 = (float)(1.0 / c->g.dx);
  e.idy2 = (float)(1.0 / (2 * c->g.dy));
  e.idy1 = (float)(1.0 / c->g.dy);
  e.exact = !c->ps->separable || !power_of_two(c->ny);
  e.dx2 = 1.0 / (2 * c->g.dx);
  e.dx1 = 1.0 / c->g.dx;
  e.dy2 = 1.0 / (2 * c->g.dy);
  e.dy1 = 1.0 / c->g.dy;
  return e;
}

// x at the fixed rows from the fixed values.  Solves rewrite only rows whose
// value can change between solves (driven rows, ρ-valued rows); the others are
// written here, after an operator build or a host update of Dirichlet values.
static int fixed_to_x_now(Ctx *c) {
  Poisson *P = c->ps;
  int rc = sync_rho64(c);  // ρ-valued fixed rows read the FP64 ρ
  if (rc) return rc;
  k_fixed_to_x<<<P->blocks, 256, 0, c->stream>>>(opview(P), P->x, P->xd, c->rho,
                                                  -1.0 / P->eps0, P->nn);
  ISKRA_CUDA(c, cudaGetLastError());
  return ISKRA_OK;
}

// Column pairs per FFT block: about two blocks per SM (at least one pair),
// at most 64 KB of float2 per block.
static int fft_tp(int N, int odd, int nx, int sms) {
  int tp = nx / (4 * sms);
  const int fixed = N / 2 + (odd > 1 ? odd : 0);
  const int cap = (65536 / (int)sizeof(float2) - fixed) / ((odd > 1 ? 2 : 1) * (N + 1));
  if (tp > cap) tp = cap;
  if (tp > 16) tp = 16;
  if (tp < 1) tp = 1;
  return tp;
}

static size_t fft_smem(int N, int odd, int tp) {
  return ((size_t)(odd > 1 ? 2 : 1) * tp * (N + 1) + N / 2 + (odd > 1 ? odd : 0)) * sizeof(float2);
}

// Shared memory of one cyclic-reduction mode: 2 columns of nx floats and its
// coefficients (nf + nb float2, nb float; nf, nb < nx).
static size_t cr_mode_bytes(int nx) { return (size_t)nx * (2 * sizeof(float) + 2 * sizeof(float2) + sizeof(float)); }

// Fourier modes per cyclic-reduction block, about one block per mode up to
// K = 2 x SMs; 0 when one mode does not fit in shared memory (the chunked
// Thomas kernel is used then).
static int cr_modes_per_block(int nx, int K, int sms) {
  if (cr_mode_bytes(nx) > 160 * 1024) return 0;
  int g = K / (2 * sms);
  const int cap = (int)(160 * 1024 / cr_mode_bytes(nx));
  if (g > cap) g = cap;
  if (g > 8) g = 8;
  return g < 1 ? 1 : g;
}

static size_t cr_smem(const Poisson *P, int G) {
  return (size_t)G * (2 * P->nx * sizeof(float) + (P->cr_nf + P->cr_nb) * sizeof(float2) + P->cr_nb * sizeof(float));
}

static int fft_smem_attr(Ctx *c) {
  Poisson *P = c->ps;
  const int smem = (int)fft_smem(P->N, P->odd, fft_tp(P->N, P->odd, P->nx, c->num_sms));
  constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  if (P->odd > 1) {
    ISKRA_CUDA(c, cudaFuncSetAttribute(k_fft_fwd<true>, kAttr, smem));
    ISKRA_CUDA(c, cudaFuncSetAttribute(k_fft_inv_update<false, true>, kAttr, smem));
  } else {
    ISKRA_CUDA(c, cudaFuncSetAttribute(k_fft_fwd<false>, kAttr, smem));
    ISKRA_CUDA(c, cudaFuncSetAttribute(k_fft_inv_update<true, false>, kAttr, smem));
    ISKRA_CUDA(c, cudaFuncSetAttribute(k_fft_inv_update<false, false>, kAttr, smem));
  }
  const int G = cr_modes_per_block(c->ps->nx, c->ps->K, c->num_sms);
  const int crsm = (int)cr_smem(c->ps, G);
  if (G && crsm > 48 * 1024)
    ISKRA_CUDA(c, cudaFuncSetAttribute(k_tridiag_cr, cudaFuncAttributeMaxDynamicSharedMemorySize, crsm));
  return ISKRA_OK;
}

static CrArgs cr_args(Poisson *P, int G) {
  CrArgs A;
  A.spec = (float *)P->spec;
  A.nx = P->nx;
  A.K = P->K;
  A.G = G;
  A.L = P->cr_levels;
  A.nf = P->cr_nf;
  A.nb = P->cr_nb;
  A.fwd = P->cr_fwd;
  A.back = P->cr_back;
  A.backb = P->cr_backb;
  A.top = P->cr_top;
  A.q = P->q;
  A.gk = P->gk;
  A.cyclic = (int)P->cyclic;
  A.pin0 = P->pin_k0;
  return A;
}

// Launch shape of the separable correction.
struct SepShape {
  int TP, fb, G;
  size_t smem;
};

static SepShape sep_shape(Ctx *c) {
  Poisson *P = c->ps;
  SepShape sh;
  sh.TP = fft_tp(P->N, P->odd, P->nx, c->num_sms);
  sh.fb = (P->nx + 2 * sh.TP - 1) / (2 * sh.TP);
  sh.smem = fft_smem(P->N, P->odd, sh.TP);
  sh.G = cr_modes_per_block(P->nx, P->K, c->num_sms);
  return sh;
}

// First part of a solve: the warm start (step solves of separable
// operators), fixed rows, the singular-case shift and the first residual
// (with E for separable operators), which resets the solver scalars.
static int queue_prologue(Ctx *c, double rtol, double dt_for_drive, SweepLoop loop, bool warm) {
  Poisson *P = c->ps;
  const int nn = P->nn, B = P->blocks, T = 256;
  OpView op = opview(P);
  const double nie = -1.0 / P->eps0;
  const float2 nie_df = df_host(nie);
  cudaStream_t st = c->stream;
  // the first residual takes ρ in double-float when it was formed so; every
  // other reader takes the FP64 copy
  const float2 *rdf = (P->separable && P->df_mode && !P->singular && !P->rho_fixed && c->rho_df_valid)
                          ? c->rho_df : nullptr;
  if (!rdf) {
    int rc = sync_rho64(c);
    if (rc) return rc;
  }
  if (warm && P->separable && P->warm_mode == 1 && c->warm_fused) {
    c->warm_fused = false;  // the step's ρ pass ran it
  } else if (warm && P->separable && P->warm_mode == 1) {
    if (P->df_mode)
      ISKRA_CUDA(c, launch_pdl(k_extrapolate<true>, B, T, 0, st, (const uint16_t *)P->cls, (void *)P->xd, P->xh,
                               nn, P->scal));
    else
      ISKRA_CUDA(c, launch_pdl(k_extrapolate<false>, B, T, 0, st, (const uint16_t *)P->cls, (void *)P->x, P->xh,
                               nn, P->scal));
  }
  if (P->ndrive_nodes)
    ISKRA_CUDA(c, launch_pdl(k_set_fixed, (P->ndrive_nodes + 255) / 256, 256, 0, st, op,
                             (const int *)P->drive_node, (const int *)P->drive_group, (const double *)P->drive_par,
                             P->ndrive_nodes, (const unsigned long long *)c->d_step, dt_for_drive, P->bfix_d, P->x,
                             P->xd, (const double *)c->rho, P->eps0, nn));
  // k_set_fixed wrote the driven rows; ρ-valued identity rows follow ρ
  if (P->rho_fixed)
    ISKRA_CUDA(c, launch_pdl(k_fixed_to_x, B, T, 0, st, op, P->x, P->xd,
                             (const double *)c->rho, nie, nn));
  if (P->singular) {
    ISKRA_CUDA(c, launch_pdl(k_sum_db, B, T, 0, st, op, (const double *)c->rho, nie, nn, P->part));
    ISKRA_CUDA(c, launch_pdl(k_lambda, 1, T, 0, st, (const double *)P->part, B, P->dsum, P->scal));
  }
  if (P->separable && P->df_mode) {
    // (step graphs: E comes from the following pass)
    if (warm)
      ISKRA_CUDA(c, launch_pdl(k_residual_df<true, false>, B, T, 0, st, op, (const float2 *)P->xd,
                               (const double *)c->rho, rdf, nie_df, nie, P->bd, P->scal, P->r32, P->part, nn,
                               (int)P->singular, rtol * rtol, eout(c, false), loop));
    else
      ISKRA_CUDA(c, launch_pdl(k_residual_df<true, true>, B, T, 0, st, op, (const float2 *)P->xd,
                               (const double *)c->rho, rdf, nie_df, nie, P->bd, P->scal, P->r32, P->part, nn,
                               (int)P->singular, rtol * rtol, eout(c, true), loop));
  } else if (P->separable) {
    ISKRA_CUDA(c, launch_pdl(k_residual<true, true>, B, T, 0, st, op, (const double *)P->x, (const double *)c->rho,
                             nie, P->scal, (double *)nullptr, P->r32, P->part, nn, (int)P->singular, rtol * rtol,
                             eout(c, true), loop));
  } else {
    ISKRA_CUDA(c, launch_pdl(k_residual<true, false>, B, T, 0, st, op, (const double *)P->x, (const double *)c->rho,
                             nie, P->scal, P->r, (float *)nullptr, P->part, nn, (int)P->singular, rtol * rtol,
                             eout(c, false), loop));
  }
  ISKRA_CUDA(c, cudaGetLastError());
  return ISKRA_OK;
}

// `count` corrections: separable operators run the FP32 FFT, tridiagonal
// solve and inverse FFT, then the FP64 residual (each skipped on the device
// once converged); other operators run CG iterations (the caller loops for
// more).  `loop` applies to the last residual only.
static int queue_sweeps(Ctx *c, double rtol, int count, bool reset_cg, SweepLoop loop) {
  Poisson *P = c->ps;
  const int nn = P->nn, B = P->blocks, T = 256;
  OpView op = opview(P);
  const double nie = -1.0 / P->eps0;
  const double rtol2 = rtol * rtol;
  cudaStream_t st = c->stream;
  SweepLoop mid = loop;  // all but the last pass
  mid.notconv = nullptr;
  if (P->separable) {
    const SepShape sh = sep_shape(c);
    const int K = P->K;
    const FftPlan F{P->N, P->log2p, P->odd, P->tw, P->tw + P->N / 2};
    const bool odd = P->odd > 1;
    for (int s = 0; s < count; s++) {
      const bool last = s == count - 1;
      const PoissonScal *sc = P->scal;
      ISKRA_CUDA(c, launch_pdl(odd ? k_fft_fwd<true> : k_fft_fwd<false>, sh.fb, 256, sh.smem, st,
                               (const float *)P->r32, P->nx, F, sh.TP, P->spec, sc));
      if (sh.G) {
        ISKRA_CUDA(c, launch_pdl(k_tridiag_cr, (K + sh.G - 1) / sh.G, 256, cr_smem(P, sh.G), st, cr_args(P, sh.G),
                                 sc));
      } else {
        ISKRA_CUDA(c, launch_pdl(k_tridiag, (2 * K + 63) / 64, 64, 0, st, (float *)P->spec, P->nx, K,
                                 (const float *)P->low, (const float *)P->inv, (const float *)P->cp,
                                 (const float *)P->q, (const float *)P->gk, (int)P->cyclic, P->pin_k0, sc));
      }
      if (P->df_mode) {
        ISKRA_CUDA(c, launch_pdl(k_fft_inv_update<true, false>, sh.fb, 256, sh.smem, st, (const float2 *)P->spec,
                                 P->nx, F, sh.TP, (const uint16_t *)P->cls, P->xd, (double *)nullptr, sc));
        ISKRA_CUDA(c, launch_pdl(k_residual_df<false, true>, B, T, 0, st, op, (const float2 *)P->xd,
                                 (const double *)nullptr, (const float2 *)nullptr, make_float2(0.f, 0.f), nie,
                                 P->bd, P->scal, P->r32, P->part, nn,
                                 (int)P->singular, rtol2, eout(c, true), last ? loop : mid));
      } else {
        ISKRA_CUDA(c, launch_pdl(odd ? k_fft_inv_update<false, true> : k_fft_inv_update<false, false>, sh.fb, 256,
                                 sh.smem, st, (const float2 *)P->spec, P->nx, F, sh.TP, (const uint16_t *)P->cls,
                                 (float2 *)nullptr, P->x, sc));
        ISKRA_CUDA(c, launch_pdl(k_residual<false, true>, B, T, 0, st, op, (const double *)P->x,
                                 (const double *)c->rho, nie, P->scal, (double *)nullptr, P->r32, P->part, nn,
                                 (int)P->singular, rtol2, eout(c, true), last ? loop : mid));
      }
    }
  } else if (P->mg) {  // flexible PCG, one multigrid V-cycle per iteration
    const int *skip = &P->scal->done;
    const int G = P->cg_blocks;
    const int tiles = ((P->nx + kApX - 1) / kApX) * ((P->ny + kApY - 1) / kApY);
    PcgDots D;
    D.ap = P->ap;
    D.part = P->part;
    D.s = P->pcg;
    auto cycle = [&](int init) {
      D.init = init;
      bool dots = false;
      const int rc = mg_queue_cycle(c, P->mg, P->r, P->z, skip, D, &dots);
      if (rc || dots) return rc;
      ISKRA_CUDA(c, launch_pdl(k_pcg_dots, std::min(G, kPcgPartials), T, 0, st, (const double *)P->r,
                               (const double *)P->z, nn, skip, D));
      return (int)ISKRA_OK;
    };
    if (reset_cg) {  // rhs2 is already in scal
      const int rc = cycle(1);
      if (rc) return rc;
    }
    for (int s = 0; s < count; s++) {
      ISKRA_CUDA(c, launch_pdl(k_pcg_ap, std::min(tiles, std::min(kPcgPartials, c->num_sms * 3)), kApThreads, 0, st, op, (const double *)P->z, P->p, P->p2,
                               P->ap, P->part, skip, P->pcg));
      ISKRA_CUDA(c, launch_pdl(k_pcg_update, G, T, 0, st, op, P->x, P->r, (const double *)P->p, (const double *)P->p2,
                               (const double *)P->ap, P->part, nn, P->scal, P->pcg, rtol2));
      const int rc = cycle(0);
      if (rc) return rc;
    }
  } else {
    if (reset_cg) {  // rhs2 is already in scal
      k_cg_init<<<B, T, 0, st>>>(op, P->r, P->z, P->p, P->part, nn);
      k_cg_rz0<<<1, T, 0, st>>>(P->part, B, P->scal);
    }
    for (int s = 0; s < count; s++) {
      k_cg_ap<<<B, T, 0, st>>>(op, P->p, P->ap, P->part, nn, P->scal);
      k_cg_update<<<B, T, 0, st>>>(op, P->x, P->r, P->z, P->p, P->ap, P->part, B, nn, P->scal);
      k_cg_dir<<<B, T, 0, st>>>(op, P->z, P->p, P->part, B, nn, P->scal, rtol2);
    }
  }
  ISKRA_CUDA(c, cudaGetLastError());
  return ISKRA_OK;
}

// Sweeps a step graph runs per solve (each skipped on the device once the
// residual meets rtol): one FP32 correction reduces the residual by about
// 10^-5 (cold start) and the step starts from the previous potential.  (ny with
// an odd factor: the host goes on with the solve where these are not enough.)
static int graph_sweeps(double rtol) {
  const int n = (int)std::ceil(std::log(rtol) / std::log(1e-5));
  return std::max(2, std::min(8, n));
}

static int finish_solve(Ctx *c) {
  Poisson *P = c->ps;
  if (P->singular && P->df_mode) {
    ISKRA_CUDA(c, launch_pdl(k_sum_xd, P->blocks, 256, 0, c->stream, (const float2 *)P->xd, P->nn, P->part));
    ISKRA_CUDA(c, launch_pdl(k_shift_xd, P->blocks, 256, 0, c->stream, P->xd, P->nn, (const double *)P->part,
                             P->blocks));
  } else if (P->singular) {
    ISKRA_CUDA(c, launch_pdl(k_sum_x, P->blocks, 256, 0, c->stream, (const double *)P->x, P->nn, P->part));
    ISKRA_CUDA(c, launch_pdl(k_shift_x, P->blocks, 256, 0, c->stream, P->x, P->nn, (const double *)P->part,
                             P->blocks));
  }
  // the separable path wrote E in its residual passes (the mean shift of the
  // singular case leaves E unchanged); CG computes it here
  c->e_from_phi = true;
  if (P->df_mode) P->x_stale = true;
  if (P->separable) return ISKRA_OK;
  return launch_efield_from(c, P->x);
}

// Whether the host looks at a step's errors before it launches the next one: CG
// operators, and the direct solves of other ny, which were CG solves.
bool poisson_step_checked(Ctx *c) { return !c->ps->separable || !power_of_two(c->ps->ny); }

// Solve queued inside a step capture (separable operators).
int poisson_solve_graph(Ctx *c, double rtol) {
  int rc = poisson_prepare(c);
  if (rc) return rc;
  Poisson *P = c->ps;
  if (!P->separable) return set_err(c, ISKRA_EINVAL, "graph solve needs a separable operator");
  const int n = graph_sweeps(rtol);
  StepStatus *status = poisson_step_checked(c) ? c->h_status : nullptr;
  rc = queue_prologue(c, rtol, c->graph_dt, SweepLoop{nullptr, status, c->d_err}, true);
  if (rc) return rc;
  rc = queue_sweeps(c, rtol, n, false, SweepLoop{c->d_err, status, c->d_err});
  if (rc) return rc;
  return finish_solve(c);
}

// ---- a step's field part in one block ------------------------------------------
// On grids of up to kFieldBlockNodes nodes the circuit, the density pass, the warm
// start, the driven rows, the residuals and corrections (or the whole multigrid
// CG, up to ~1300 nodes), and E run as phases of one 512-thread block with ϕ, the
// right-hand side, the residual and the spectrum in shared memory: at these sizes each of the 9 (double-float) to 18 (FP64,
// singular) launches they took costs 3-10 us of launch and memory latency for
// well under a microsecond of work.  The phases are the multi-launch path's own
// node and line functions, so ϕ, ρ and E are the same bits; only the norms'
// summation order differs.  At ny = 2 (the quasi-1D grids) the transform is a sum
// and a difference, taken while the lines are loaded and stored.  Whole steps:
// 257 x 2 discharge 103 -> 85 us, 128 x 2 periodic beams 94 -> 68 us with their
// record (the block itself 17 and 25 us with warm caches).  A cluster of eight
// such blocks did not pay: its barriers cost 2-3 us each (128 x 2: no gain over
// the launches, 128 x 64: 56 against 50 us).
struct FieldBlock {
  FinalizeArgs A;
  FinalizeDfArgs D;
  CircuitArgs cir;             // cir.cd == nullptr: none
  unsigned long long *cir_seen;
  const double *vol_inv, *bg;
  const float2 *vol_inv_df, *bg_df;
  double *rho;
  float2 *rho_df;
  int warm;                    // ϕ <- 2 ϕ_n - ϕ_(n-1) once the history is valid
  OpView op;
  double *x;
  float2 *xd;
  void *xh;
  PoissonScal *sc;
  const int *dnode, *dgroup;
  const double *dpar;
  int ndn;
  const unsigned long long *step;
  double dt, nie, rtol2, dsum;
  float2 nie_df;
  double *bfix;
  int singular, rho_fixed, sweeps, nn;
  FftPlan F;
  CrArgs C;
  EOut eo;
  MgBlock mg;
  int *err;
  StepStatus *status;          // for the host, which waits for it, or nullptr
};
constexpr int kFieldThreads = 512, kFieldMgIterations = 10000;
// MODE: 0 ny = 2, 1 ny another power of two, 2 any other ny (direct solves); 3
// multigrid CG (FP64 state)
template <bool DF, int MODE>
__global__ void __launch_bounds__(kFieldThreads) k_field_block(FieldBlock P) {
  extern __shared__ __align__(16) unsigned char field_smem[];
  __shared__ double red[2 * kFieldThreads];
  __shared__ RowClass cls_sh[kSmemClasses];
  const int tid = threadIdx.x, T = kFieldThreads, nn = P.nn, nx = P.op.nx, ny = P.op.ny;
  constexpr bool TWO = MODE == 0, ODD = MODE == 2, MG = MODE == 3;
  // shared memory: ϕ, b or ρ (8 B a node), residual, spectrum, then the
  // transform's columns or the lines of the cyclic reduction
  float2 *xd = reinterpret_cast<float2 *>(field_smem), *bd = xd + nn;
  double *x64 = reinterpret_cast<double *>(field_smem), *rho64 = x64 + nn;
  float *r32 = reinterpret_cast<float *>(bd + nn);
  float2 *spec = reinterpret_cast<float2 *>(r32 + (nn + (nn & 1)));
  float2 *fbuf = spec + (TWO ? 0 : (size_t)nx * P.C.K);
  // coefficients of the lines: written by the operator build, read before the wait
  const size_t fft_n = TWO ? 0 : (ODD ? 2 : 1) * (size_t)((nx + 1) / 2) * (P.F.N + 1) + P.F.N / 2 + (ODD ? P.F.odd : 0);
  CrShared cr{};
  // multigrid CG: r, p, S p after ϕ and ρ, then the levels
  double *r64 = rho64 + nn, *p64 = r64 + nn, *ap64 = p64 + nn;
  float *lev = reinterpret_cast<float *>(ap64 + nn);
  const float *ci = P.mg.cinv;
  if (MG) {
    const float *staged = mg_bottom_stage(lev, P.mg.lv, 0, P.mg.L, P.mg.cinv, P.mg.cinv_shared);
    if (P.mg.cinv_shared) ci = staged;
  } else {
    cr = cr_shared(P.C, reinterpret_cast<float *>(fbuf + fft_n));
    cr_stage(P.C, cr, 0, P.C.K);
  }
  const RowClass *CT = stage_classes(P.op, cls_sh);
  PoissonScal *sc = P.sc;
  pdl_wait();
  const bool rho_df = DF && !P.singular && !P.rho_fixed;  // ρ formed in double-float
  const bool hist = P.warm && sc->hist != 0;
  // The last warp: circuit (it reads ϕ of the last step in global memory, which
  // is rewritten at the end) and driven values (a sine each in FP64) beside the
  // density pass.
  if (P.cir.cd && tid == T - 1) circuit_advance(P.cir, P.dt, P.cir_seen);
  // driven rows (the solve of step n uses V((n-2)Δt), n >= 2)
  for (int t = tid - (T - 32); t >= 0 && t < P.ndn; t += 32) {
    const unsigned long long n_step = *P.step;
    if (n_step >= 2) P.bfix[P.dnode[t]] = drive_value(P.dpar + 4 * P.dgroup[t], (double)(n_step - 2) * P.dt);
  }
  {
    int flags = 0;
    for (int k = tid; k < nn; k += T) {
      if (rho_df) {
        finalize_df_node(P.D, P.vol_inv_df, P.bg_df, P.rho_df, k, flags);
      } else {
        finalize_node(P.A, P.vol_inv, P.bg, P.rho, k, flags);
        if (!DF) rho64[k] = P.rho[k];
      }
      const bool upd = hist && !(P.op.cls[k] & kFixedBit);
      if (DF) {
        const float2 a = P.xd[k];
        xd[k] = upd ? df_add(make_float2(2.f * a.x, 2.f * a.y), df_neg(((float2 *)P.xh)[k])) : a;
        if (P.warm) ((float2 *)P.xh)[k] = a;
      } else {
        const double a = P.x[k];
        x64[k] = upd ? 2.0 * a - ((double *)P.xh)[k] : a;
        if (P.warm) ((double *)P.xh)[k] = a;
      }
    }
    if (flags) atomicOr(P.err, flags);
  }
  __syncthreads();
  if (P.warm && tid == 0) sc->hist = 1;
  if (P.ndn) {
    for (int t = tid; t < P.ndn; t += T) {
      const int k = P.dnode[t];
      if (DF) xd[k] = df_from(P.bfix[k]);
      else x64[k] = P.bfix[k];
    }
    __syncthreads();
  }
  if (P.rho_fixed) {  // ρ-valued identity rows
    for (int k = tid; k < nn; k += T) {
      const unsigned ck = P.op.cls[k];
      if (ck & kFixedBit) {
        const double v = CT[ck & kClassMask].rho ? P.rho[k] * P.nie : P.op.bfix[k];
        if (DF) xd[k] = df_from(v);
        else x64[k] = v;
      }
    }
    __syncthreads();
  }
  const double *rho = DF ? P.rho : rho64;
  double lam = 0.0;
  if (P.singular) {  // projection of the right-hand side onto the range
    double v[1] = {0}, t[1];
    for (int k = tid; k < nn; k += T) {
      const RowClass &C = CT[P.op.cls[k] & kClassMask];
      if (!C.fixed) {
        double b = C.rho ? rho[k] * P.nie : P.op.bfix[k];
        if (C.sig_dof >= 0) b -= C.sig_coef * P.op.sigma[C.sig_dof];
        v[0] += C.d * b;
      }
    }
    block_sums<1>(v, red, t);
    lam = P.dsum > 0 ? t[0] / P.dsum : 0.0;
    if (tid == 0) sc->lambda = lam;
  }
  double rhs2 = 0;
  if (MG) {
    // flexible PCG as in k_pcg_ap, k_pcg_update and the cycle, the whole solve
    // without a launch or a host check
    double v2[2] = {0, 0}, t2[2];
    for (int k = tid; k < nn; k += T)
      residual_node<true>(P.op, CT, x64, rho, P.nie, 0.0, 0, k, k % nx, k / nx, r64, v2[0], v2[1]);
    asm volatile("cp.async.wait_group 0;" ::: "memory");  // the staged levels (a barrier follows)
    block_sums<2>(v2, red, t2);
    rhs2 = t2[1];
    double res2 = t2[0], rz = 0, alpha = 0;
    int it = 0;
    bool done = (rhs2 > 0 && res2 <= P.rtol2 * rhs2) || res2 == 0.0;
    const MgSh q = mg_sh(lev, P.mg.lv[0]);
    // (a residual that is no number, or a direction without energy, stays so: the
    // rest of the iterations would only hold the device)
    bool stuck = !isfinite(res2);
    while (!done && !stuck && it < kFieldMgIterations) {
      for (int k = tid; k < nn; k += T) q.b[k] = (float)r64[k];
      __syncthreads();
      mg_bottom_cycle(lev, P.mg.lv, 0, P.mg.L, ci);
      v2[0] = v2[1] = 0;
      for (int k = tid; k < nn; k += T) {
        const double z = (double)q.x[k];
        v2[0] = fma(z, r64[k], v2[0]);
        if (it) v2[1] = fma(z, ap64[k], v2[1]);
      }
      block_sums<2>(v2, red, t2);
      const double beta = it && rz != 0 ? -alpha * t2[1] / rz : 0.0;
      rz = t2[0];
      for (int k = tid; k < nn; k += T) {
        double p = (double)q.x[k];
        if (beta != 0) p = fma(beta, p64[k], p);
        p64[k] = p;
      }
      __syncthreads();
      double v1[1] = {0}, t1[1];
      for (int k = tid; k < nn; k += T) {
        const RowClass &C = CT[P.op.cls[k] & kClassMask];
        int w, e, so, no;
        nbr(k, nx, ny, w, e, so, no);
        double a = C.s0 * p64[k];
        a = fma(C.sW, p64[w], a);
        a = fma(C.sE, p64[e], a);
        a = fma(C.sS, p64[so], a);
        a = fma(C.sN, p64[no], a);
        ap64[k] = a;
        v1[0] = fma(p64[k], a, v1[0]);
      }
      block_sums<1>(v1, red, t1);
      alpha = t1[0] != 0 ? rz / t1[0] : 0.0;
      v1[0] = 0;
      for (int k = tid; k < nn; k += T) {
        const unsigned ck = P.op.cls[k];
        if (ck & kFixedBit) continue;
        x64[k] = fma(alpha, p64[k], x64[k]);
        const double rr = fma(-alpha, ap64[k], r64[k]);
        r64[k] = rr;
        const double res = rr * CT[ck & kClassMask].inv_d;
        v1[0] = fma(res, res, v1[0]);
      }
      block_sums<1>(v1, red, t1);
      res2 = t1[0];
      it++;
      done = (rhs2 > 0 && res2 <= P.rtol2 * rhs2) || res2 == 0.0;
      stuck = alpha == 0 || !isfinite(res2);
    }
    if (tid == 0) {
      sc->rhs2 = rhs2;
      sc->res2 = res2;
      sc->relres = rhs2 > 0 ? sqrt(res2 / rhs2) : sqrt(res2);
      sc->iters = it;
      sc->done = done;
      sc->e_pending = 0;
      if (!done) atomicOr(P.err, DERR_NOTCONV);
    }
  }
  for (int s = 0; !MG; s++) {
    double a2 = 0, b2 = 0;
    if (DF) {
      if (s == 0)
        residual_df_nodes<true, false>(P.op, CT, xd, rho, rho_df ? P.rho_df : nullptr, P.nie_df, P.nie, bd, r32, nn,
                                       P.singular, lam, P.eo, tid, T, a2, b2);
      else
        residual_df_nodes<false, false>(P.op, CT, xd, nullptr, nullptr, P.nie_df, P.nie, bd, r32, nn, P.singular, lam,
                                        P.eo, tid, T, a2, b2);
    } else {
      for (int k = tid; k < nn; k += T) {
        const int j = k / nx, i = k - j * nx;
        r32[k] = s == 0 ? residual_node<true>(P.op, CT, x64, rho, P.nie, lam, P.singular, k, i, j, nullptr, a2, b2)
                        : residual_node<false>(P.op, CT, x64, rho, P.nie, lam, P.singular, k, i, j, nullptr, a2, b2);
      }
    }
    const double v[2] = {a2, b2};
    double t[2];
    block_sums<2>(v, red, t);
    if (s == 0) rhs2 = t[1];
    const bool done = (rhs2 > 0 && t[0] <= P.rtol2 * rhs2) || t[0] == 0.0;
    if (done || s == P.sweeps) {
      if (tid == 0) {
        sc->rhs2 = rhs2;
        sc->res2 = t[0];
        sc->relres = rhs2 > 0 ? sqrt(t[0] / rhs2) : sqrt(t[0]);
        sc->iters = s;
        sc->done = done;
        sc->e_pending = 0;
        if (!done) atomicOr(P.err, DERR_NOTCONV);
      }
      break;
    }
    // one FP32 correction
    if (TWO) {
      for (int i = tid; i < nx; i += T) {
        const float a = r32[i], b = r32[i + nx];
        cr.d[i] = P.C.pin0 == i ? 0.f : a + b;
        cr.d[nx + i] = a - b;
      }
      __syncthreads();
      cr_levels<true>(P.C, cr, 0, 2);
      for (int i = tid; i < nx; i += T) {
        const float a = cr_value(P.C, cr.d, 0, i), b = cr_value(P.C, cr.d + nx, 1, i);
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const int k = i + nx * j;
          if (P.op.cls[k] & kFixedBit) continue;
          const float dz = (j ? a - b : a + b) * 0.5f;
          if (DF) xd[k] = df_add_f(xd[k], dz);
          else x64[k] += (double)dz;
        }
      }
    } else {
      const int TP = (nx + 1) / 2;
      fft_fwd_item<ODD>(0, r32, nx, P.F, TP, spec, fbuf);
      __syncthreads();
      cr_solve(P.C, cr, reinterpret_cast<float *>(spec), 0, P.C.K);
      fft_inv_item<DF, ODD>(0, spec, nx, P.F, TP, P.op.cls, xd, x64, fbuf);
    }
    __syncthreads();
  }
  // Every flag of the step is set: its kernels ended before this one, and the
  // block's own flags were set before barriers above or by this thread.
  if (P.status && tid == 0) report_step(P.status, P.err);
  // E, and ϕ to memory
  for (int k = tid; k < nn; k += T) {
    const int j = k / nx, i = k - j * nx;
    if (DF) {
      const int w = i > 0 ? k - 1 : k + nx - 1, e = i < nx - 1 ? k + 1 : k - nx + 1;
      const int so = j > 0 ? k - nx : k + nx * (ny - 1), no = j < ny - 1 ? k + nx : k - nx * (ny - 1);
      efield_df5(xd[k], xd[w], xd[e], xd[so], xd[no], k, i, j, nx, ny, P.eo);
      if (!P.singular) P.xd[k] = xd[k];
    } else {
      efield_at(x64, k, i, j, nx, ny, P.eo);
      if (!P.singular) P.x[k] = x64[k];
    }
  }
  if (P.singular) {  // mean-zero ϕ
    double v[1] = {0}, t[1];
    for (int k = tid; k < nn; k += T) v[0] += DF ? df_value(xd[k]) : x64[k];
    block_sums<1>(v, red, t);
    const double m = t[0] / nn;
    for (int k = tid; k < nn; k += T) {
      if (DF) P.xd[k] = df_add(xd[k], df_neg(df_from(m)));
      else P.x[k] = x64[k] - m;
    }
  }
}

// Largest grids whose field part runs as one block: the crossing with the
// multi-launch path (whole steps: 33 x 32 36 against 43 us, 48 x 32 45 against 47,
// 65 x 32 51 against 49; ny = 2: 1000 x 2 90 against 104, 2000 x 2 105 against
// 109, 3000 x 2 equal).
constexpr int kFieldBlockNodes = 1536, kFieldBlockNodes1D = 4096;
constexpr size_t kFieldSmem = 192 * 1024;  // beside 28 KB of static arrays

static size_t field_block_bytes(const Poisson *P) {
  const size_t nn = P->nn;
  size_t b = 20 * (nn + 1) + cr_smem(P, P->K);
  if (P->N > 2) b += (size_t)P->nx * P->K * sizeof(float2) + fft_smem(P->N, P->odd, (P->nx + 1) / 2);
  return b;
}

bool poisson_one_block(Ctx *c) {
  const Poisson *P = c->ps;
  if (!P || P->dirty) return false;
  if (!P->separable) {  // multigrid CG without a learned warm start, levels and vectors in shared memory
    MgBlock v;
    return mg_block_view(P->mg, &v) && !lws_active(c) && 40 * (size_t)P->nn + v.bytes <= kFieldSmem;
  }
  return P->separable && P->nn <= (P->N == 2 ? kFieldBlockNodes1D : kFieldBlockNodes) &&
         field_block_bytes(P) <= kFieldSmem;
}

int launch_field_block(Ctx *c, double rtol) {
  Poisson *P = c->ps;
  const bool df = P->df_mode, rho_df = poisson_df_rho(c);
  FieldBlock B{};
  int rc = ISKRA_OK;
  if (c->cir_d) {
    rc = circuit_args(c, B.cir);
    B.cir_seen = c->cir_seen;
  }
  if (!rc) rc = step_density_args(c, rho_df, B.A, B.D);
  if (rc) return rc;
  B.vol_inv = c->vol_inv;
  B.bg = c->rho_bg;
  B.vol_inv_df = c->vol_inv_df;
  B.bg_df = c->bg_df;
  B.rho = c->rho;
  B.rho_df = c->rho_df;
  B.warm = P->warm_mode == 1;
  B.op = opview(P);
  B.x = P->x;
  B.xd = P->xd;
  B.xh = P->xh;
  B.sc = P->scal;
  B.dnode = P->drive_node;
  B.dgroup = P->drive_group;
  B.dpar = P->drive_par;
  B.ndn = P->ndrive_nodes;
  B.step = c->d_step;
  B.dt = c->graph_dt;
  B.nie = -1.0 / P->eps0;
  B.nie_df = df_host(B.nie);
  B.rtol2 = rtol * rtol;
  B.dsum = P->dsum;
  B.bfix = P->bfix_d;
  B.singular = P->singular;
  B.rho_fixed = P->rho_fixed;
  B.sweeps = std::min(8, graph_sweeps(rtol) + 2);  // (sweeps not needed cost nothing here)
  B.nn = P->nn;
  B.eo = eout(c, true);
  B.err = c->d_err;
  B.status = poisson_step_checked(c) ? c->h_status : nullptr;
  if (!P->separable) {
    mg_block_view(P->mg, &B.mg);
    ISKRA_CUDA(c, cudaFuncSetAttribute(k_field_block<false, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kFieldSmem));
    ISKRA_CUDA(c, launch_pdl(k_field_block<false, 3>, 1, kFieldThreads, 40 * (size_t)P->nn + B.mg.bytes, c->stream, B));
    c->e_from_phi = true;
    return ISKRA_OK;
  }
  B.F = FftPlan{P->N, P->log2p, P->odd, P->tw, P->tw + P->N / 2};
  B.C = cr_args(P, P->K);
  const int mode = P->N == 2 ? 0 : P->odd > 1 ? 2 : 1;
  auto kern = df ? (mode == 0 ? k_field_block<true, 0> : k_field_block<true, 1>)
                 : (mode == 0 ? k_field_block<false, 0> : mode == 1 ? k_field_block<false, 1> : k_field_block<false, 2>);
  ISKRA_CUDA(c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFieldSmem));
  ISKRA_CUDA(c, launch_pdl(kern, 1, kFieldThreads, field_block_bytes(P), c->stream, B));
  c->e_from_phi = true;
  if (df) P->x_stale = true;
  return ISKRA_OK;
}

// Learned warm start of a CG solve: δ = scale y on the free rows (the
// network's predicted correction), applied as ϕ += α δ with the exact line
// search α = δ·r / δ·Sδ in the energy norm of the scaled system S ϕ = c
// (r = c - S ϕ the scaled residual), so the CG error never grows.  Every
// scalar stays on the device: no host round trip inside the solve.
__global__ void k_lws_dir(OpView op, const float *__restrict__ y, const double *__restrict__ scale,
                          const double *__restrict__ r, double *__restrict__ p, double *__restrict__ part, int nn) {
  __shared__ double sh[40];
  const double sc = *scale;
  double v = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
    const RowClass &C = op.classes[op.cls[k] & kClassMask];
    const double d = C.fixed ? 0.0 : sc * (double)y[k];
    p[k] = d;
    v += d * r[k];
  }
  const double t = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// α from the block partials of δ·r (part) and δ·Sδ (part + kPartials); no
// step when the first residual already met the tolerance or α is not a
// positive number
__global__ void __launch_bounds__(256) k_lws_alpha(const double *__restrict__ part, int nb, LwsScal *ls,
                                                   const PoissonScal *sc) {
  __shared__ double sh[40];
  double dr = 0, dsd = 0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    dr += part[b];
    dsd += part[kPartials + b];
  }
  dr = block_sum(dr, sh);
  __syncthreads();
  dsd = block_sum(dsd, sh);
  if (threadIdx.x == 0) {
    double a = dsd > 0 ? dr / dsd : 0.0;
    if (!(a > 0) || !isfinite(a) || sc->done) a = 0.0;
    ls->alpha = a;
    ls->res2_before = sc->res2;
  }
}

__global__ void k_lws_axpy(double *__restrict__ x, const double *__restrict__ p, const LwsScal *__restrict__ ls,
                           int nn) {
  const double alpha = ls->alpha;
  if (alpha == 0.0) return;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) x[k] += alpha * p[k];
}

// after the residual of the corrected ϕ: statistics of the applied step
__global__ void k_lws_stats(LwsScal *ls, const PoissonScal *sc) {
  if (ls->alpha > 0) {
    ls->warm_solves++;
    ls->alpha_sum += ls->alpha;
    ls->ratio_sum += ls->res2_before > 0 ? sqrt(sc->res2 / ls->res2_before) : 0.0;
  }
}

static int lws_line_search(Ctx *c, const float *y, const double *scale) {
  Poisson *P = c->ps;
  const int B = P->blocks, T = 256, nn = P->nn;
  OpView op = opview(P);
  LwsScal *ls = lws_scal(c);
  k_lws_dir<<<B, T, 0, c->stream>>>(op, y, scale, P->r, P->p, P->part, nn);
  k_cg_ap<<<B, T, 0, c->stream>>>(op, P->p, P->ap, P->part, nn, P->scal);
  k_lws_alpha<<<1, 256, 0, c->stream>>>(P->part, B, ls, P->scal);
  k_lws_axpy<<<B, T, 0, c->stream>>>(P->x, P->p, ls, nn);
  ISKRA_CUDA(c, cudaGetLastError());
  return ISKRA_OK;
}

// A solve with host convergence checks (CG; the separable solver outside
// step graphs).  step: the solve of an iskra_step (CG operators), which
// starts from ϕ extrapolated in time like the graph path; other solves
// start from ϕ and end the extrapolation history.
static int choose_solver(Ctx *c, double rtol);
static int solve_sync(Ctx *c, double rtol, int maxit, int *iters, double *relres, bool step = false) {
  int rc = poisson_prepare(c);
  if (rc) return rc;
  rc = poisson_set_precision(c, rtol);
  if (rc) return rc;
  Poisson *P = c->ps;
  if (step && !P->separable && P->warm_mode == 1)
    ISKRA_CUDA(c, launch_pdl(k_extrapolate<false>, P->blocks, 256, 0, c->stream, (const uint16_t *)P->cls,
                             (void *)P->x, P->xh, P->nn, P->scal));
  bool first = true, lws_pending = false;
  int done_it = 0;
  double last_relres = INFINITY;
  const SweepLoop none{};
  for (;;) {
    // (multigrid CG: as many iterations as the last solve took before the
    // first host check, then two at a time; converged ones return at once)
    const int mg_chunk = first ? std::max(4, std::min(P->last_iters, 32)) : 2;
    const int chunk = std::min(P->separable ? 2 : (P->mg ? mg_chunk : 32), maxit - done_it);
    if (first) {
      rc = queue_prologue(c, rtol, c->graph_dt, none, false);
      if (rc) return rc;
      if (!P->separable && lws_active(c)) {
        // learned warm start: the network's correction from the first
        // residual, then the residual again (CG restarts from the corrected
        // ϕ).  Harvesting reads the first residual's convergence on the host
        // (a solve that needs no iteration gives no training pair); in use
        // mode the device skips the step of an already converged solve.
        bool run = true;
        if (lws_harvesting(c)) {
          ISKRA_CUDA(c, cudaMemcpyAsync(P->scal_h, P->scal, sizeof(PoissonScal), cudaMemcpyDeviceToHost,
                                        c->stream));
          ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
          run = !P->scal_h->done;
        }
        if (run) {
          const float *y = nullptr;
          const double *scale = nullptr;
          lws_pending = true;
          rc = lws_begin(c, P->r, &y, &scale);
          if (rc) return rc;
          rc = lws_mark_start(c, P->x);
          if (rc) return rc;
          if (y) {
            rc = lws_line_search(c, y, scale);
            if (rc) return rc;
            rc = queue_prologue(c, rtol, c->graph_dt, none, false);
            if (rc) return rc;
            k_lws_stats<<<1, 1, 0, c->stream>>>(lws_scal(c), P->scal);
            ISKRA_CUDA(c, cudaGetLastError());
          }
        }
      }
    }
    if (P->mg && !P->separable) {
      // multigrid CG: the start (V-cycle of the first residual) queued, then
      // the iteration's kernels replayed as one graph
      if (first) {
        rc = queue_sweeps(c, rtol, 0, true, none);
        if (rc) return rc;
      }
      if (!P->pcg_graph || P->pcg_graph_rtol != rtol) {
        if (P->pcg_graph) cudaGraphExecDestroy(P->pcg_graph);
        P->pcg_graph = nullptr;
        cudaGraph_t g;
        ISKRA_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        const int qrc = queue_sweeps(c, rtol, 1, false, none);
        const cudaError_t ce = cudaStreamEndCapture(c->stream, &g);
        if (qrc) {
          if (ce == cudaSuccess) cudaGraphDestroy(g);
          return qrc;
        }
        ISKRA_CUDA(c, ce);
        const cudaError_t ie = cudaGraphInstantiate(&P->pcg_graph, g, 0);
        cudaGraphDestroy(g);
        ISKRA_CUDA(c, ie);
        P->pcg_graph_rtol = rtol;
      }
      for (int s = 0; s < chunk; s++) ISKRA_CUDA(c, cudaGraphLaunch(P->pcg_graph, c->stream));
    } else {
      rc = queue_sweeps(c, rtol, chunk, first, none);
      if (rc) return rc;
    }
    first = false;
    ISKRA_CUDA(c, cudaMemcpyAsync(P->scal_h, P->scal, sizeof(PoissonScal), cudaMemcpyDeviceToHost, c->stream));
    ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
    done_it = P->scal_h->iters;
    if (P->scal_h->done || done_it >= maxit) break;
    if (P->separable && !power_of_two(P->ny)) {
      // two corrections that gain less than a factor of 10: the rounding floor is
      // above the tolerance, which CG, as it was before these operators were solved
      // directly, meets with its updated residual
      const double now = P->scal_h->relres;
      if (!std::isfinite(now)) break;
      if (!(now < 0.1 * last_relres)) {
        P->stalled = rtol;
        rc = choose_solver(c, rtol);
        if (rc) return rc;
        first = true;
        done_it = 0;
      }
      last_relres = now;
    }
  }
  rc = finish_solve(c);
  if (rc) return rc;
  if (lws_pending) {
    rc = lws_end(c, P->x, P->scal_h->done != 0);
    if (rc) return rc;
  }
  // ϕ moved outside the step sequence: the next step solve starts from it
  if (!step) ISKRA_CUDA(c, cudaMemsetAsync(&P->scal->hist, 0, sizeof(int), c->stream));
  ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  P->last_iters = P->scal_h->iters;
  P->last_relres = P->scal_h->relres;
  if (iters) *iters = P->scal_h->iters;
  if (relres) *relres = P->scal_h->relres;
  if (!P->scal_h->done) return set_err(c, ISKRA_ENOTCONV, "Poisson solve did not reach the tolerance");
  return collect_device_errors(c);
}

double *poisson_sigma_ptr(Ctx *c) { return c->ps ? c->ps->sigma_d : nullptr; }
// the device σ values with the operator built (outside stream capture a
// pending rebuild runs first; a captured step has prepared it already)
double *poisson_sigma_prepared(Ctx *c) {
  if (!c->ps) return nullptr;
  if (c->ps->dirty && poisson_prepare(c) != ISKRA_OK) return nullptr;
  return c->ps->nsig > 0 ? c->ps->sigma_d : nullptr;
}
const double *poisson_x_ptr(Ctx *c) { return c->ps ? c->ps->x : nullptr; }
const float2 *poisson_xd_ptr(Ctx *c) { return c->ps && c->ps->df_mode ? c->ps->xd : nullptr; }
bool poisson_warm_args(Ctx *c, WarmArgs *w) {
  Poisson *P = c->ps;
  if (!P || !P->separable || !P->df_mode || P->warm_mode != 1 || !P->xh || !P->xd) return false;
  w->cls = P->cls;
  w->xd = P->xd;
  w->xh = (float2 *)P->xh;
  w->hist = &P->scal->hist;
  w->ticket = &P->scal->hticket;
  w->fixed_bit = kFixedBit;
  return true;
}

bool poisson_df_rho(Ctx *c) {
  const Poisson *P = c->ps;
  return P && !P->dirty && P->separable && P->df_mode && !P->singular && !P->rho_fixed;
}
void poisson_mark_x_stale(Ctx *c) {
  if (c->ps && c->ps->df_mode) c->ps->x_stale = true;
}

// FP64 view of ϕ brought up to date with the double-float state (stream-ordered)
int poisson_sync_x(Ctx *c) {
  Poisson *P = c->ps;
  if (!P || !P->df_mode || !P->x_stale) return ISKRA_OK;
  k_df_to_x<<<P->blocks, 256, 0, c->stream>>>(P->xd, P->x, P->nn);
  ISKRA_CUDA(c, cudaGetLastError());
  P->x_stale = false;
  return ISKRA_OK;
}

// Precision of the separable solver's state for a tolerance.  Double-float
// keeps ϕ to ~48 bits; its residual floor (~2^-47 |A||x| / ||rhs||, 5e-13
// measured at 512^2) is far below 1e-9, so tolerances from 1e-9 up run on
// the FP32 pipes.  Tighter tolerances and operators with σ dofs (whose rows
// mix 1/Δx and 1/Δx^2 scales) keep the FP64 state, and so do operators whose ny
// is no power of two: they were CG solves, in FP64.
static bool want_df(const Poisson *P, double rtol) {
  return P->separable && power_of_two(P->ny) && P->nsig == 0 && rtol >= 1e-9;
}

// Puts the solver that direct_solve picks in effect (outside stream capture);
// the multigrid hierarchy is built when CG first needs it.
static int choose_solver(Ctx *c, double rtol) {
  Poisson *P = c->ps;
  const bool direct = direct_solve(c, P, rtol);
  if (P->dirty || direct == P->separable) return ISKRA_OK;
  int rc = poisson_sync_x(c);
  if (rc) return rc;
  if (!direct && !P->mg && !P->singular) {
    std::vector<RowEff> rows;
    std::vector<double> d;
    bool any_fixed = false;
    rc = scaled_rows(c, P, rows, d, &any_fixed);
    if (!rc) rc = build_mg(c, P, rows, d);
    if (rc) return rc;
  }
  ISKRA_CUDA(c, cudaMemsetAsync(&P->scal->hist, 0, sizeof(int), c->stream));
  P->separable = direct;
  invalidate_graphs(c);
  return ISKRA_OK;
}

// Switches the authoritative state (outside stream capture; stream-ordered).
int poisson_set_precision(Ctx *c, double rtol) {
  Poisson *P = c->ps;
  if (!P) return ISKRA_OK;
  const int rc = choose_solver(c, rtol);
  if (rc) return rc;
  const bool df = want_df(P, rtol);
  if (df == P->df_mode) return ISKRA_OK;
  if (df) {
    k_x_to_df<<<P->blocks, 256, 0, c->stream>>>(P->x, P->xd, P->nn);
    P->x_stale = false;
  } else {
    if (P->x_stale) k_df_to_x<<<P->blocks, 256, 0, c->stream>>>(P->xd, P->x, P->nn);
    P->x_stale = false;
  }
  ISKRA_CUDA(c, cudaMemsetAsync(&P->scal->hist, 0, sizeof(int), c->stream));  // history in the other representation
  ISKRA_CUDA(c, cudaGetLastError());
  P->df_mode = df;
  invalidate_graphs(c);
  return ISKRA_OK;
}
bool poisson_separable(Ctx *c) { return c->ps && c->ps->separable; }
int poisson_solve_blocking(Ctx *c, double rtol, int maxit) {
  return solve_sync(c, rtol, maxit, nullptr, nullptr, true);
}

// ---------------------------------------------------------------------------
// Ensemble field solve: one block per run forms ρ from the run's deposit,
// sets the fixed rows (drive amplitudes per run), and solves the separable
// operator directly in FP64 -- residual of the previous potential, DFT along
// y (N <= 16, direct), cyclic reduction along x per Fourier mode with the
// host's FP64 coefficients (the single-run solver's, staged in shared memory
// while ρ is formed), inverse DFT -- then writes E.  The same operator as one
// FP64 sweep of the single-run solver, exact to rounding.  Cyclic reduction
// takes 2 log2(nx) dependent levels where a Thomas sweep takes 2 nx dependent
// FP64 steps on one thread per mode (on GB300, whose FP64 rate is ~1/64 of
// FP32, that chain was 2/3 of the kernel).
// ---------------------------------------------------------------------------
struct FieldRuns {
  int ns;
  unsigned long long *acc[kMaxSpecies];  // run 0; run stride nn
  unsigned *cnt[kMaxSpecies];
  double scale[kMaxSpecies];             // w0 2^-48
  double q[kMaxSpecies];
  const double *vol_inv, *bg;
  double *rho, *x;                       // R x nn
  float2 *E32;                           // R x nn
  const double *amp;                     // R x ngroups drive amplitudes
  int ngroups;
  const int *drive_node, *drive_group;
  const double *drive_par;               // 4 per group; par[0] replaced by amp[r][g]
  int ndrive_nodes;
  const unsigned long long *d_step;
  double dt, neg_inv_eps0;
  const double *cr;                      // packed FP64 cyclic-reduction coefficients
  int ncr, L, nf, nb, pin0;              // their count, levels, rows per mode; pinned row of mode 0 (or -1)
  int N, K;
  float idx2, idx1, idy2, idy1;
  int *err;
};

__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

__global__ void __launch_bounds__(256) k_field_runs(OpView op, FieldRuns F) {
  extern __shared__ __align__(16) double fsm[];
  __shared__ RowClass cls_sh[kSmemClasses];
  __shared__ double twc[16], tws[16];  // cos, sin of 2π m/N
  const int nx = op.nx, ny = op.ny, nn = nx * ny, N = F.N, K = F.K, ncol = 2 * K;
  // xs, rs: nn each; dsp: column col = 2 k + part of the spectrum (nx each);
  // crs: the coefficients (2 nn + 2 nx K is even: 16-byte aligned pairs)
  double *xs = fsm, *rs = xs + nn, *dsp = rs + nn, *crs = dsp + (size_t)ncol * nx;
  // the coefficients do not depend on the previous kernel: staged before it ends
  for (int t = threadIdx.x; t < F.ncr; t += blockDim.x) cp_async8(crs + t, F.cr + t);
  asm volatile("cp.async.commit_group;" ::: "memory");
  pdl_wait();
  if (threadIdx.x < N) sincospi(2.0 * threadIdx.x / N, &tws[threadIdx.x], &twc[threadIdx.x]);
  const int r = blockIdx.x;
  const size_t o = (size_t)r * nn;
  const RowClass *__restrict__ CT = stage_classes(op, cls_sh);
  int flags = 0;
  // ρ from the run's deposit (consumed); ϕ of the previous step
  for (int k = threadIdx.x; k < nn; k += blockDim.x) {
    const double vi = F.vol_inv[k];
    double rho = 0.0;
    for (int s = 0; s < F.ns; s++) {
      const unsigned long long a = F.acc[s][o + k];
      if (F.cnt[s][o + k] > kMaxCell) flags |= DERR_OVERFLOW;
      F.acc[s][o + k] = 0ull;
      F.cnt[s][o + k] = 0u;
      rho += ((double)a * F.scale[s] * vi) * F.q[s];
    }
    if (F.bg) rho += F.bg[k];
    F.rho[o + k] = rho;
    xs[k] = F.x[o + k];
  }
  __syncthreads();
  // driven rows: V((n-2)Δt) with this run's amplitude, as k_set_fixed
  const unsigned long long n_step = *F.d_step;
  for (int t = threadIdx.x; t < F.ndrive_nodes; t += blockDim.x) {
    const int k = F.drive_node[t], g = F.drive_group[t];
    const double *par = F.drive_par + 4 * g;
    if (n_step >= 2) {
      const double tt = (double)(n_step - 2) * F.dt;
      xs[k] = F.amp[(size_t)r * F.ngroups + g] * sin(2.0 * M_PI * par[1] * tt + par[2]) + par[3];
    } else {
      xs[k] = op.bfix[k];
    }
  }
  __syncthreads();
  // scaled residual of the free rows
  for (int k = threadIdx.x; k < nn; k += blockDim.x) {
    const int j = k / nx, i = k - j * nx;
    const double rhoc = F.rho[o + k];
    const unsigned ck = op.cls[k];
    if (ck & kFixedBit) {
      rs[k] = 0.0;
      continue;
    }
    const RowClass &C = CT[ck];
    const int w = i > 0 ? k - 1 : k + nx - 1;
    const int e = i < nx - 1 ? k + 1 : k - nx + 1;
    const int s = j > 0 ? k - nx : k + nx * (ny - 1);
    const int n = j < ny - 1 ? k + nx : k - nx * (ny - 1);
    const double b = C.rho ? rhoc * F.neg_inv_eps0 : op.bfix[k];
    double ax = C.c0 * xs[k];
    ax = fma(C.cW, xs[w], ax);
    ax = fma(C.cE, xs[e], ax);
    ax = fma(C.cS, xs[s], ax);
    ax = fma(C.cN, xs[n], ax);
    rs[k] = -C.d * (b - ax);
  }
  __syncthreads();
  // DFT along y: column 2k (real) and 2k+1 (imaginary) of mode k,
  // Σ_j r[i, j] e^{-2πi jk/N}; the pinned row of mode 0 is zero
  for (int t = threadIdx.x; t < nx * K; t += blockDim.x) {
    const int i = t / K, k = t - i * K;
    double re = 0, im = 0;
    for (int j = 0; j < N; j++) {
      const int m = (j * k) % N;  // e^{-2πi jk/N}
      const double v = rs[i + nx * j];
      re += v * twc[m];
      im -= v * tws[m];
    }
    if (k == 0 && i == F.pin0) re = im = 0.0;
    dsp[(2 * k) * nx + i] = re;
    dsp[(2 * k + 1) * nx + i] = im;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // cyclic reduction (the single-run solver's levels, in FP64)
  const double2 *fwd = reinterpret_cast<const double2 *>(crs);
  const double2 *back = fwd + (size_t)K * F.nf;
  const double *backb = reinterpret_cast<const double *>(back + (size_t)K * F.nb);
  const double *top = backb + (size_t)K * F.nb;
  int Fo = 0, Bo = 0;
  for (int l = 0; l < F.L; l++) {
    const int s = 1 << l, cnt = nx >> (l + 1);
    for (int t = threadIdx.x; t < cnt * ncol; t += blockDim.x) {
      const int m = t / ncol, col = t - m * ncol;
      const int i = (m + 1) * 2 * s - 1;
      const double2 ag = fwd[(size_t)(col >> 1) * F.nf + Fo + m];
      double *dc = dsp + (size_t)col * nx;
      double v = dc[i] - ag.x * dc[i - s];
      if (i + s < nx) v -= ag.y * dc[i + s];
      dc[i] = v;
    }
    Fo += cnt;
    Bo += ((nx >> l) + 1) >> 1;
    __syncthreads();
  }
  const int topr = (1 << F.L) - 1;
  for (int col = threadIdx.x; col < ncol; col += blockDim.x) dsp[(size_t)col * nx + topr] *= top[col >> 1];
  __syncthreads();
  for (int l = F.L - 1; l >= 0; l--) {
    const int s = 1 << l, ecnt = ((nx >> l) + 1) >> 1;
    Bo -= ecnt;
    for (int t = threadIdx.x; t < ecnt * ncol; t += blockDim.x) {
      const int m = t / ncol, col = t - m * ncol;
      const int j = (2 * m + 1) * s - 1;
      const size_t q = (size_t)(col >> 1) * F.nb + Bo + m;
      const double2 rr = back[q];
      double *dc = dsp + (size_t)col * nx;
      double x = backb[q] * dc[j];
      if (j - s >= 0) x -= rr.x * dc[j - s];
      if (j + s < nx) x -= rr.y * dc[j + s];
      dc[j] = x;
    }
    __syncthreads();
  }
  // inverse DFT (Hermitian spectrum) and update of the free rows
  const bool pow2N = (N & (N - 1)) == 0;
  const double invN = 1.0 / N;
  for (int k = threadIdx.x; k < nn; k += blockDim.x) {
    if (op.cls[k] & kFixedBit) continue;
    const int j = k / nx, i = k - j * nx;
    double v = 0;
    for (int m = 0; m < N; m++) {
      const int mm = m < K ? m : N - m;
      const double re = dsp[(2 * mm) * nx + i];
      const double im = m < K ? dsp[(2 * mm + 1) * nx + i] : -dsp[(2 * mm + 1) * nx + i];
      const int q = (j * m) % N;
      v += re * twc[q] - im * tws[q];
    }
    xs[k] += pow2N ? v * invN : v / N;  // 1/N exact for a power of two
  }
  __syncthreads();
  // ϕ and E = -∇ϕ
  EOut eo;
  eo.E32 = F.E32 + o;
  eo.idx2 = F.idx2;
  eo.idx1 = F.idx1;
  eo.idy2 = F.idy2;
  eo.idy1 = F.idy1;
  for (int k = threadIdx.x; k < nn; k += blockDim.x) {
    const int j = k / nx, i = k - j * nx;
    F.x[o + k] = xs[k];
    efield_at(xs, k, i, j, nx, ny, eo);
  }
  if (flags) atomicOr(F.err, flags);
}

// Ensemble field solve over R runs (separable, non-cyclic, non-singular
// operators with N = ny <= 16 and no σ dof).
int launch_field_runs(Ctx *c, int R, FieldRunsHost &H, cudaStream_t st) {
  int rc = poisson_prepare(c);
  if (rc) return rc;
  Poisson *P = c->ps;
  if (!P->separable || P->odd > 1 || P->cyclic || P->singular || P->N > 16 || P->nsig > 0 || P->rho_fixed)
    return set_err(c, ISKRA_EINVAL, "ensemble field solve needs a separable, non-periodic-x operator with ny <= 16, "
                                    "a power of two");
  const int nx = P->nx, K = P->K, nn = P->nn;
  if (!P->cr64_d) return set_err(c, ISKRA_EINVAL, "FP64 factors not uploaded (poisson_upload_fp64)");
  FieldRuns F{};
  F.ns = H.ns;
  for (int s = 0; s < H.ns; s++) {
    F.acc[s] = H.acc[s];
    F.cnt[s] = H.cnt[s];
    F.scale[s] = H.scale[s];
    F.q[s] = H.q[s];
  }
  F.vol_inv = c->vol_inv;
  F.bg = c->rho_bg;
  F.rho = H.rho;
  F.x = H.x;
  F.E32 = H.E32;
  F.amp = H.amp;
  F.ngroups = P->ndrive;
  F.drive_node = P->drive_node;
  F.drive_group = P->drive_group;
  F.drive_par = P->drive_par;
  F.ndrive_nodes = P->ndrive_nodes;
  F.d_step = H.d_step;
  F.dt = H.dt;
  F.neg_inv_eps0 = -1.0 / P->eps0;
  F.cr = P->cr64_d;
  F.ncr = (int)P->cr64.size();
  F.L = P->cr_levels;
  F.nf = P->cr_nf;
  F.nb = P->cr_nb;
  F.pin0 = P->pin_k0;
  F.N = P->N;
  F.K = K;
  const EOut e = eout(c, true);
  F.idx2 = e.idx2;
  F.idx1 = e.idx1;
  F.idy2 = e.idy2;
  F.idy1 = e.idy1;
  F.err = H.err;
  const size_t smem = (2 * (size_t)nn + 2 * (size_t)nx * K + P->cr64.size()) * sizeof(double);
  if (smem > 200 * 1024) return set_err(c, ISKRA_EINVAL, "ensemble grid too large for the per-run field solve");
  ISKRA_CUDA(c, cudaFuncSetAttribute(k_field_runs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  ISKRA_CUDA(c, launch_pdl(k_field_runs, R, 256, smem, st, opview(P), F));
  return ISKRA_OK;
}

// FP64 Thomas factors on the device (outside any stream capture)
int poisson_upload_fp64(Ctx *c) {
  int rc = poisson_prepare(c);
  if (rc) return rc;
  Poisson *P = c->ps;
  if (!P->separable || P->odd > 1)
    return set_err(c, ISKRA_EINVAL, "ensemble field solve needs a separable operator with ny a power of two");
  if (P->cr64_d) return ISKRA_OK;
  ISKRA_CUDA(c, cudaMalloc(&P->cr64_d, std::max<size_t>(1, P->cr64.size()) * sizeof(double)));
  ISKRA_CUDA(c, cudaMemcpy(P->cr64_d, P->cr64.data(), P->cr64.size() * sizeof(double), cudaMemcpyHostToDevice));
  ISKRA_CUDA(c, setup_copies_done());
  return ISKRA_OK;
}

int poisson_ndrive(Ctx *c) { return c->ps ? c->ps->ndrive : 0; }
double poisson_drive_amp(Ctx *c, int g) { return c->ps ? c->ps->drives[g].amp : 0.0; }

}  // namespace iskra

using namespace iskra;

extern "C" {

int iskra_poisson_create(iskra_ctx *h, double eps0) {
  if (!h || !(eps0 > 0)) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (c->ps) poisson_destroy(c->ps);
  c->ps = poisson_new(c, eps0);
  return ISKRA_OK;
}

int iskra_poisson_apply_dirichlet(iskra_ctx *h, const uint8_t *nodes, double phi0) {
  if (!h || !nodes) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  Poisson *P = c->ps;
  // value-only update of rows that are already identity rows: no rebuild
  bool structural = false;
  for (int r = 0; r < P->nn && !structural; r++) {
    if (!nodes[r]) continue;
    const double *R = &P->C[(size_t)r * 7];
    bool ident = R[0] == 1.0;
    for (int s = 1; s < 7; s++) ident &= R[s] == 0.0;
    for (auto &col : P->sig_cols) ident &= col[r] == 0.0;
    if (!ident || P->rho_dof[r]) structural = true;
  }
  assemble_dirichlet(P, nodes, phi0);
  if (structural || P->dirty) {
    P->dirty = true;
    return ISKRA_OK;
  }
  ISKRA_CUDA(c, cudaMemcpyAsync(P->bfix_d, P->bfix.data(), P->nn * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  return fixed_to_x_now(c);
}

int iskra_poisson_apply_periodic(iskra_ctx *h, int axis) {
  if (!h) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  if (axis != 1 && axis != 2) return set_err(c, ISKRA_EINVAL, "axis must be 1 or 2");
  assemble_periodic(c->ps, axis);
  c->ps->dirty = true;
  return ISKRA_OK;
}

int iskra_poisson_add_dof(iskra_ctx *h, int *dof) {
  if (!h || !dof) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  c->ps->sig_cols.emplace_back(c->ps->nn, 0.0);
  c->ps->sig_b.push_back(0.0);
  *dof = (int)c->ps->sig_b.size();
  c->ps->dirty = true;
  return ISKRA_OK;
}

int iskra_poisson_apply_neumann(iskra_ctx *h, const uint8_t *nodes, int dof) {
  if (!h || !nodes) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  if (dof < 1 || dof > (int)c->ps->sig_b.size()) return set_err(c, ISKRA_EINVAL, "bad σ dof");
  assemble_neumann(c->ps, nodes, dof, false);
  c->ps->dirty = true;
  return ISKRA_OK;
}

int iskra_poisson_apply_neumann_gauss(iskra_ctx *h, const uint8_t *nodes, int dof) {
  if (!h || !nodes) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  if (dof < 1 || dof > (int)c->ps->sig_b.size()) return set_err(c, ISKRA_EINVAL, "bad σ dof");
  assemble_neumann(c->ps, nodes, dof, true);
  c->ps->dirty = true;
  return ISKRA_OK;
}

int iskra_poisson_set_sigma(iskra_ctx *h, int dof, double value) {
  if (!h) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps || dof < 1 || dof > (int)c->ps->sig_b.size()) return set_err(c, ISKRA_EINVAL, "bad σ dof");
  c->ps->sig_b[dof - 1] = value;
  if (c->ps->sigma_d && dof <= c->ps->nsig) {
    ISKRA_CUDA(c, cudaMemcpyAsync(c->ps->sigma_d + (dof - 1), &c->ps->sig_b[dof - 1], sizeof(double),
                                  cudaMemcpyHostToDevice, c->stream));
    ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  return ISKRA_OK;
}

int iskra_poisson_get_sigma(iskra_ctx *h, int dof, double *value) {
  if (!h || !value) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps || dof < 1 || dof > (int)c->ps->sig_b.size()) return set_err(c, ISKRA_EINVAL, "bad σ dof");
  if (c->ps->sigma_d && dof <= c->ps->nsig) {
    ISKRA_CUDA(c, cudaMemcpyAsync(&c->ps->sig_b[dof - 1], c->ps->sigma_d + (dof - 1), sizeof(double),
                                  cudaMemcpyDeviceToHost, c->stream));
    ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  *value = c->ps->sig_b[dof - 1];
  return ISKRA_OK;
}

int iskra_poisson_drive_dirichlet(iskra_ctx *h, const uint8_t *nodes, double amp, double freq, double phase,
                                  double dc) {
  if (!h || !nodes) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  DriveGroup g;
  for (int r = 0; r < c->ps->nn; r++) {
    if (!nodes[r]) continue;
    const double *R = &c->ps->C[(size_t)r * 7];
    bool ident = R[0] == 1.0 && !c->ps->rho_dof[r];
    for (int s = 1; s < 7; s++) ident &= R[s] == 0.0;
    if (!ident) return set_err(c, ISKRA_EINVAL, "driven nodes must be Dirichlet rows (apply_dirichlet first)");
    g.nodes.push_back(r);
  }
  g.amp = amp;
  g.freq = freq;
  g.phase = phase;
  g.dc = dc;
  c->ps->drives.push_back(g);
  c->ps->dirty = true;
  return ISKRA_OK;
}

int iskra_poisson_set_method(iskra_ctx *h, int method, int *active) {
  if (!h) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  if (method < 0 || method > 2) return set_err(c, ISKRA_EINVAL, "method must be 0, 1 or 2");
  if (c->ps->method != method) {
    c->ps->method = method;
    c->ps->dirty = true;
  }
  const int rc = poisson_prepare(c);
  if (rc) return rc;
  // (the solver itself changes with the next solve, whose tolerance decides; the
  // hierarchy of an operator solved directly so far is built when CG first needs it)
  const Poisson *P = c->ps;
  if (active) *active = direct_solve(c, P, kReportRtol) ? 0 : (P->method != 1 && !P->singular ? 2 : 1);
  return ISKRA_OK;
}

int iskra_poisson_set_warm_start(iskra_ctx *h, int mode) {
  if (!h) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  if (mode != 0 && mode != 1) return set_err(c, ISKRA_EINVAL, "warm-start mode must be 0 or 1");
  if (c->ps->warm_mode != mode) {
    c->ps->warm_mode = mode;
    invalidate_graphs(c);
    if (c->ps->scal) ISKRA_CUDA(c, cudaMemsetAsync(&c->ps->scal->hist, 0, sizeof(int), c->stream));
  }
  return ISKRA_OK;
}

int iskra_poisson_solve(iskra_ctx *h, double rtol, int maxit, int *iters, double *relres) {
  if (!h) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!(rtol > 0) || maxit < 1) return set_err(c, ISKRA_EINVAL, "bad tolerance / iteration limit");
  int rc = launch_charge_density(c);
  if (rc) return rc;
  return solve_sync(c, rtol, maxit, iters, relres);
}

int iskra_poisson_solve_host(iskra_ctx *h, const double *f, double rtol, int maxit, double *phi_out, int *iters,
                             double *relres) {
  if (!h || !f) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!(rtol > 0) || maxit < 1) return set_err(c, ISKRA_EINVAL, "bad tolerance / iteration limit");
  // the device ρ holds -f: b[ρ] = f/ε0 = -ρ/ε0
  std::vector<double> negf(c->nn);
  for (int k = 0; k < c->nn; k++) negf[k] = -f[k];
  // on the stream of the solve: a cudaMemcpy of up to 64 KB can return before
  // the device has the data, and the solve then read the previous ρ
  ISKRA_CUDA(c, cudaMemcpyAsync(c->rho, negf.data(), c->nn * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  c->rho64_valid = true;
  c->rho_df_valid = false;
  int rc = solve_sync(c, rtol, maxit, iters, relres);
  if (rc && rc != ISKRA_ENOTCONV) return rc;
  if (phi_out) {
    int rs = poisson_sync_x(c);
    if (rs) return rs;
    ISKRA_CUDA(c, cudaMemcpyAsync(phi_out, c->ps->x, c->nn * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  }
  return rc;
}

int iskra_solve_info(iskra_ctx *h, int *iters, double *relres) {
  if (!h) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps || !c->ps->scal) return set_err(c, ISKRA_EINVAL, "no solve yet");
  ISKRA_CUDA(c, cudaMemcpyAsync(c->ps->scal_h, c->ps->scal, sizeof(PoissonScal), cudaMemcpyDeviceToHost, c->stream));
  ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  if (iters) *iters = c->ps->scal_h->iters;
  if (relres) *relres = c->ps->scal_h->relres;
  return ISKRA_OK;
}

int iskra_poisson_residual(iskra_ctx *h, const double *f, const double *phi, double *relres) {
  if (!h || !f || !phi || !relres) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  if (!c->ps) return set_err(c, ISKRA_EINVAL, "no Poisson solver");
  int rc = poisson_prepare(c);
  if (rc) return rc;
  Poisson *P = c->ps;
  const int nx = P->nx, ny = P->ny, nn = P->nn;
  // the device copies of the fixed values (driven rows are rewritten there)
  // and of σ (the circuit and the tracker update it) are authoritative
  std::vector<double> bfix(nn), sig(P->sig_b.size());
  ISKRA_CUDA(c, cudaMemcpyAsync(bfix.data(), P->bfix_d, nn * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  if (!sig.empty() && P->sigma_d)
    ISKRA_CUDA(c, cudaMemcpyAsync(sig.data(), P->sigma_d, std::min<size_t>(sig.size(), P->nsig) * sizeof(double),
                                  cudaMemcpyDeviceToHost, c->stream));
  ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  // identity rows (Dirichlet values, driven rows): known values, moved to
  // the right-hand side as the solver does; the norms run over the others
  auto identity = [&](int r) {
    const double *R = &P->C[(size_t)r * 7];
    if (R[0] != 1.0) return false;
    for (int q = 1; q < 7; q++)
      if (R[q] != 0.0) return false;
    for (const auto &col : P->sig_cols)
      if (col[r] != 0.0) return false;
    return true;
  };
  std::vector<char> fixed(nn);
  for (int r = 0; r < nn; r++) fixed[r] = identity(r);
  double r2 = 0, b2 = 0;
  for (int r = 0; r < nn; r++) {
    if (fixed[r]) continue;
    const int i = r % nx, j = r / nx;
    const double *R = &P->C[(size_t)r * 7];
    const int col[7] = {r, i > 0 ? r - 1 : r, i < nx - 1 ? r + 1 : r, j > 0 ? r - nx : r, j < ny - 1 ? r + nx : r,
                        i == 0 ? r + nx - 1 : (i == nx - 1 ? r - nx + 1 : r),
                        j == 0 ? r + nx * (ny - 1) : (j == ny - 1 ? r - nx * (ny - 1) : r)};
    double afree = 0, known = 0;
    for (int q = 0; q < 7; q++) {
      if (R[q] == 0.0) continue;
      if (fixed[col[q]]) known += R[q] * phi[col[q]];
      else afree += R[q] * phi[col[q]];
    }
    for (size_t k = 0; k < P->sig_cols.size(); k++)
      if (P->sig_cols[k][r] != 0.0) known += P->sig_cols[k][r] * sig[k];
    const double b = (P->rho_dof[r] ? f[r] / P->eps0 : bfix[r]) - known;
    r2 += (b - afree) * (b - afree);
    b2 += b * b;
  }
  *relres = b2 > 0 ? std::sqrt(r2 / b2) : std::sqrt(r2);
  return ISKRA_OK;
}

}  // extern "C"

// device source of a field download (bringing ϕ and E up to date)
static int field_source(Ctx *c, int which, const double **src, size_t *n) {
  *n = (size_t)c->nn;
  if (which == ISKRA_FIELD_RHO) {
    int rs = sync_rho64(c);
    if (rs) return rs;
    *src = c->rho;
  } else if (which == ISKRA_FIELD_PHI) {
    if (!c->ps || !c->ps->x) return set_err(c, ISKRA_EINVAL, "no potential yet");
    int rs = poisson_sync_x(c);
    if (rs) return rs;
    *src = c->ps->x;
  } else if (which == ISKRA_FIELD_E) {
    if (c->e_from_phi && c->ps && c->ps->x) {
      int rs = poisson_sync_x(c);
      if (rs) return rs;
      int rc = launch_efield64(c, c->ps->x);
      if (rc) return rc;
    }
    *src = c->E64;
    *n *= 3;
  } else {
    return set_err(c, ISKRA_EINVAL, "bad field selector");
  }
  return ISKRA_OK;
}

extern "C" {

int iskra_field_download(iskra_ctx *h, int which, double *out) {
  if (!h || !out) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  const double *src = nullptr;
  size_t n = 0;
  int rc = field_source(c, which, &src, &n);
  if (rc) return rc;
  ISKRA_CUDA(c, cudaMemcpyAsync(out, src, n * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  ISKRA_CUDA(c, cudaStreamSynchronize(c->stream));
  return collect_device_errors(c);
}

// Non-blocking download: the field as the work queued so far leaves it is
// written to a device staging buffer on the context stream (ϕ of the
// double-float state converted straight into it), then copied to `out` on a
// second stream, so the copy overlaps the next queued steps.  Two staging
// buffers alternate: a download waits only for the copy of the one before
// last.  `out` (pinned host memory for a true overlap) holds the values after
// the next synchronising call.
int iskra_field_download_async(iskra_ctx *h, int which, double *out) {
  if (!h || !out) return ISKRA_EINVAL;
  Ctx *c = &h->c;
  const size_t cap = (size_t)c->nn * 3;
  if (!c->dl_stage) {
    ISKRA_CUDA(c, cudaMalloc(&c->dl_stage, 2 * cap * sizeof(double)));
    ISKRA_CUDA(c, cudaStreamCreateWithFlags(&c->dl_stream, cudaStreamNonBlocking));
    ISKRA_CUDA(c, cudaEventCreateWithFlags(&c->dl_ready, cudaEventDisableTiming));
    for (int b = 0; b < 2; b++) ISKRA_CUDA(c, cudaEventCreateWithFlags(&c->dl_done[b], cudaEventDisableTiming));
  }
  const int b = c->dl_next;
  double *stage = c->dl_stage + (size_t)b * cap;
  size_t n = 0;
  Poisson *P = c->ps;
  if (which == ISKRA_FIELD_PHI && P && P->x && P->df_mode && P->x_stale) {
    if (c->dl_used[b]) ISKRA_CUDA(c, cudaStreamWaitEvent(c->stream, c->dl_done[b], 0));
    k_df_to_x<<<P->blocks, 256, 0, c->stream>>>(P->xd, stage, P->nn);
    ISKRA_CUDA(c, cudaGetLastError());
    n = (size_t)P->nn;
  } else {
    const double *src = nullptr;
    int rc = field_source(c, which, &src, &n);
    if (rc) return rc;
    if (c->dl_used[b]) ISKRA_CUDA(c, cudaStreamWaitEvent(c->stream, c->dl_done[b], 0));
    ISKRA_CUDA(c, cudaMemcpyAsync(stage, src, n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  }
  ISKRA_CUDA(c, cudaEventRecord(c->dl_ready, c->stream));
  ISKRA_CUDA(c, cudaStreamWaitEvent(c->dl_stream, c->dl_ready, 0));
  ISKRA_CUDA(c, cudaMemcpyAsync(out, stage, n * sizeof(double), cudaMemcpyDeviceToHost, c->dl_stream));
  ISKRA_CUDA(c, cudaEventRecord(c->dl_done[b], c->dl_stream));
  c->dl_used[b] = true;
  c->dl_next = b ^ 1;
  c->dl_pending = true;
  return ISKRA_OK;
}

}  // extern "C"
