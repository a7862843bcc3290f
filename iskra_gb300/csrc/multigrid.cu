// multigrid.cu -- geometric multigrid V-cycle, the preconditioner of the CG
// Poisson solve for operators the FFT/tridiagonal solve cannot take (internal
// electrodes, non-column boundaries, Neumann rows that break separability).
//
// Replaces the reference's dense A\b (FiniteDifferenceMethod/src/
// generalized_poisson.jl:201-203,372-378) for those operators together with
// the FP64 conjugate-gradient iteration in poisson.cu: CG runs in FP64 on the
// symmetrised operator S = -D A over the free rows and is iterated to the
// requested relative residual; this file supplies z = M^-1 r, one V(2,2)
// cycle in FP32 (the preconditioner needs no FP64 accuracy; GB300 runs FP32
// at ~64x its FP64 rate, and the FP64 residual of the CG iteration decides
// convergence).  CG uses the flexible (Polak-Ribiere) direction update, so
// the FP32 rounding of the cycle does not stall it.
//
// Hierarchy: level 0 is S on the node grid (5-point, periodic wraps as the
// assembled operator has them; identity rows removed: the correction is zero
// there).  Coarser levels halve each axis that has at least 3 nodes (6 when
// periodic): coarse node I sits on fine node 2I, odd fine nodes interpolate
// linearly from their two coarse neighbours (one at an open far end; the seam of
// an odd periodic axis is at axis_parents), so
// P = Px (x) Py is bilinear; the coarse operator is the Galerkin product
// P^T S P (9-point), formed on the host in FP64.  Smoother: damped Jacobi
// (omega = 0.7), 2 sweeps before and after the coarse correction; the
// coarsest level (at most kMgCoarsest nodes) is solved exactly with its
// dense inverse.  The cycle is symmetric (same smoother before and after,
// restriction = P^T, exact coarsest solve), so it is a fixed SPD
// preconditioner up to FP32 rounding.
//
// Launches: one per level and leg.  k_mg_down does a level's two sweeps from
// zero, its residual and the restriction on shared-memory tiles with a halo;
// k_mg_up the prolongation and two sweeps; the smallest levels and the
// coarsest solve are one block (k_mg_bottom).
#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.cuh"
#include "multigrid.cuh"

namespace iskra {

constexpr float kMgOmega = 0.7f;

struct Mg {
  std::vector<MgLevel> lv;
  MgLevel *dlv = nullptr;      // device copy of lv (the single-block bottom reads it)
  int bottom = 0;              // first level of the single-block bottom (0: none)
  size_t bottom_smem = 0;      // its shared memory
  float *cinv = nullptr;       // dense inverse of the coarsest level (n x n)
};

void mg_destroy(Mg *m) {
  if (!m) return;
  for (auto &l : m->lv) {
    cudaFree(l.coef);
    cudaFree(l.dinv);
    cudaFree(l.x);
    cudaFree(l.x2);
    cudaFree(l.b);
  }
  cudaFree(m->cinv);
  cudaFree(m->dlv);
  delete m;
}

// ---- interpolation weights along one axis ----------------------------------
// The seam of a coarsened axis (MgXfer::seam_x, seam_y):
//   kSeamOpen    no coupling, or an odd periodic axis of 2m + 1 nodes, m odd: fine
//                nodes 2m and 0 are coarse nodes both, m + 1 in all
//   kSeamEven    an even periodic axis: the last odd node lies between coarse
//                nodes nc - 1 and 0
//   kSeamJump    an odd periodic axis of 2m + 1 nodes, m even: m coarse nodes, fine
//                node 2m - 1 takes the value of coarse node m - 1, fine node 2m that
//                of coarse node 0
// Both odd forms leave an even number of coarse nodes, so that the next coarsening
// closes the uneven interval at the seam again: the spacings of a level stay within
// a factor of 4, and point Jacobi goes on smoothing.  (Stopping at the odd axis and
// coarsening the other alone, as the hierarchy first did, makes the operator
// anisotropic: 257 x 257 nodes, y-periodic, took 48 iterations.)
static int coarse_nodes(int n, int per) {
  if (!per || n % 2 == 0) return (n + 1) / 2;
  const int m = n / 2;
  return m % 2 ? m + 1 : m;
}
static int seam(int n, int per) { return !per ? kSeamOpen : n % 2 == 0 ? kSeamEven : n / 2 % 2 ? kSeamOpen : kSeamJump; }

// fine index i -> up to two coarse parents with weights (n fine / nc coarse nodes):
// even i -> i/2 (1); odd i -> (i-1)/2 and (i+1)/2 (1/2 each), past the last coarse
// node as the seam has it.  Not coarsened: i -> i (1).
static int axis_parents(int i, int n, int nc, int coarsened, int per, int *c, float *w) {
  const int sm = seam(n, per);
  w[0] = 1.f;
  c[0] = coarsened ? i >> 1 : i;
  if (!coarsened) return 1;
  if (c[0] >= nc) c[0] = 0;  // kSeamJump's last node
  if ((i & 1) == 0) return 1;
  int hi = (i + 1) >> 1;
  if (hi >= nc) {
    if (sm != kSeamEven) return 1;
    hi = 0;
  }
  w[0] = w[1] = 0.5f;
  c[1] = hi;
  return 2;
}

// ---- downward leg of a level: two sweeps from zero, residual, restriction ----
// A block takes 16 x 8 coarse nodes.  On a shared-memory tile of the fine nodes
// under them: x0 = dinv b (the first sweep from x = 0 is pointwise) with a halo
// of 3, the second sweep x1 with a halo of 2, the residual with a halo of 1,
// then the coarse b.  One thread per tile node keeps the node's coefficients and
// b in registers through both stencil passes, and all its loads are issued at
// once: a level costs one memory latency and four barriers.  (A first version
// with 256 threads looping over the tile took 13 us on every level, the latency
// of its nine dependent rounds of loads.)  x1 of the tile's own fine nodes goes
// to memory for the upward leg.  At 1024 x 1024 16 us where the three kernels it
// replaces took 30, on levels of a few thousand nodes 4-5 us against 15.  r64 given: level 0, b = (float) r64 (the FP64
// scaled residual of the CG iteration).
constexpr int kDownCx = 16, kDownCy = 8;
constexpr int kDownW = 2 * kDownCx + 5, kDownH = 2 * kDownCy + 5;  // x0 region of a doubly coarsened level
constexpr int kDownThreads = (kDownW * kDownH + 31) / 32 * 32;

template <bool FIVE>
__global__ void __launch_bounds__(kDownThreads) k_mg_down(const float *__restrict__ coef,
                                                            const float *__restrict__ dinv, float *__restrict__ x,
                                                            const float *__restrict__ b, float *__restrict__ bc,
                                                            MgXfer T, const int *skip,
                                                            const double *__restrict__ r64) {
  __shared__ float s0[kDownThreads], s1[kDownThreads];
  const int nx = T.nx, ny = T.ny, n = nx * ny;
  const int l = threadIdx.x, ly = l / kDownW, lx = l - kDownW * ly;
  const int I0 = blockIdx.x * kDownCx, J0 = blockIdx.y * kDownCy;
  const int fx = T.cx ? 2 * I0 : I0, fy = T.cy ? 2 * J0 : J0;  // first own fine node
  const int ox = T.cx ? 2 * kDownCx : kDownCx, oy = T.cy ? 2 * kDownCy : kDownCy;  // own fine nodes per axis
  const int gx = fx - T.cx - 2, gy = fy - T.cy - 2;            // node of tile position (0, 0)
  const int W = (T.cx ? 2 * kDownCx + 1 : kDownCx) + 4, H = (T.cy ? 2 * kDownCy + 1 : kDownCy) + 4;
  const int k = wrap_any(gx + lx, nx) + nx * wrap_any(gy + ly, ny);
  // coefficients: written by the operator build, read before the wait
  const MgStencil<FIVE> S = mg_stencil<FIVE>(coef, k, n);
  const float dk = __ldg(dinv + k);
  pdl_wait();
  if (*skip) return;
  const float bk = r64 ? (float)r64[k] : b[k];
  const float x0 = __fmul_rn(dk, bk);
  s0[l] = x0;
  __syncthreads();
  if (lx >= 1 && lx < W - 1 && ly >= 1 && ly < H - 1) {
    const float v = dk != 0.f ? fmaf(dk, bk - apply9t(S, s0 + l, kDownW), x0) : 0.f;
    s1[l] = v;
    const int ux = gx + lx - fx, uy = gy + ly - fy;
    if ((unsigned)ux < (unsigned)ox && (unsigned)uy < (unsigned)oy && fx + ux < nx && fy + uy < ny) x[k] = v;
  }
  __syncthreads();
  if (lx >= 2 && lx < W - 2 && ly >= 2 && ly < H - 2)
    s0[l] = dk != 0.f ? bk - apply9t(S, s1 + l, kDownW) : 0.f;  // (x0 is used up)
  __syncthreads();
  const int I = I0 + lx, J = J0 + ly;
  if (lx < kDownCx && ly < kDownCy && I < T.ncx && J < T.ncy)
    bc[I + T.ncx * J] = restrict_at([&](int fi, int fj) { return s0[fi - gx + kDownW * (fj - gy)]; }, T, I, J);
}

// ---- upward leg of a level: prolongation and two sweeps ----
// A block takes 32 x 16 nodes, one thread per node of the tile and its halo of
// two: x + P xc, the first sweep with a halo of 1, the second into xo (another
// array than x: neighbouring blocks read x); coefficients and b in registers for
// both sweeps (four to five us on small levels against 12 in three launches).
// Level 0 (r64, z64 given) reads b = (float) r64, writes the result
// in FP64 and adds up z.r and z.Sp of the CG iteration (pcg_finish_dots).
constexpr int kUpX = 32, kUpY = 16, kUpW = kUpX + 4, kUpH = kUpY + 4;
constexpr int kUpThreads = (kUpW * kUpH + 31) / 32 * 32;

template <bool FIVE>
__global__ void __launch_bounds__(kUpThreads) k_mg_up(const float *__restrict__ coef, const float *__restrict__ dinv,
                                                      const float *__restrict__ x, const float *__restrict__ b,
                                                      const float *__restrict__ xc, float *__restrict__ xo, MgXfer T,
                                                      const int *skip, const double *__restrict__ r64,
                                                      double *__restrict__ z64, PcgDots D) {
  __shared__ float sa[kUpThreads], sx[kUpThreads];
  __shared__ double red[2 * kUpThreads];
  const int nx = T.nx, ny = T.ny, n = nx * ny;
  const int tiles_x = (nx + kUpX - 1) / kUpX, tiles = tiles_x * ((ny + kUpY - 1) / kUpY);
  const int l = threadIdx.x, ly = l / kUpW, lx = l - kUpW * ly;
  double zr = 0, za = 0;
  bool waited = false;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int ty = tile / tiles_x;
    const int gx = (tile - ty * tiles_x) * kUpX - 2 + lx, gy = ty * kUpY - 2 + ly;
    const int i = wrap_any(gx, nx), j = wrap_any(gy, ny), k = i + nx * j;
    const bool own = lx >= 2 && lx < kUpX + 2 && ly >= 2 && ly < kUpY + 2 && gx < nx && gy < ny;
    const MgStencil<FIVE> S = mg_stencil<FIVE>(coef, k, n);
    const float dk = __ldg(dinv + k);
    if (!waited) {
      pdl_wait();
      if (*skip) return;
      waited = true;
    }
    const double rk = r64 ? r64[k] : 0.0;
    const double apk = own && z64 && !D.init ? D.ap[k] : 0.0;
    const float bk = r64 ? (float)rk : b[k];
    float v = x[k];
    if (dk != 0.f) v += prolong_at(xc, T, i, j);
    sa[l] = v;
    __syncthreads();
    if (lx >= 1 && lx < kUpW - 1 && ly >= 1 && ly < kUpH - 1) {
      v = dk != 0.f ? v + dk * (bk - apply9t(S, sa + l, kUpW)) : 0.f;
      sx[l] = v;
    }
    __syncthreads();
    if (own) {
      v = dk != 0.f ? v + dk * (bk - apply9t(S, sx + l, kUpW)) : 0.f;
      if (z64) {
        const double z = (double)v;
        z64[k] = z;
        zr = fma(z, rk, zr);
        za = fma(z, apk, za);
      } else {
        xo[k] = v;
      }
    }
  }
  if (z64) pcg_finish_dots(D, zr, za, red);
}

// coarsest level: x = Ainv b (one warp per row)
// (a hierarchy of one level reads r64 and writes z64, the FP64 vectors of the
// CG iteration, directly)
__global__ void __launch_bounds__(256) k_mg_coarse(const float *__restrict__ inv, const float *__restrict__ b,
                                                   float *__restrict__ x, int n, const int *skip,
                                                   const double *__restrict__ r64, double *__restrict__ z64) {
  pdl_wait();
  if (*skip) return;
  const int lane = threadIdx.x & 31;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < n; row += (gridDim.x * blockDim.x) >> 5) {
    float s = 0.f;
    for (int c = lane; c < n; c += 32) s = fmaf(inv[(size_t)row * n + c], r64 ? (float)r64[c] : b[c], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
      if (z64) z64[row] = (double)s;
      else x[row] = s;
    }
  }
}

__global__ void __launch_bounds__(kMgBottomThreads) k_mg_bottom(const MgLevel *__restrict__ lv, int l0, int L,
                                                                const float *__restrict__ cinv, const int *skip) {
  extern __shared__ float mg_smem[];
  const float *ci = mg_bottom_stage(mg_smem, lv, l0, L, cinv);  // (written by the operator build)
  pdl_wait();
  if (*skip) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");  // no copy is in flight when the block ends
    return;
  }
  const MgLevel &D = lv[l0];
  for (int k = threadIdx.x; k < D.n; k += blockDim.x) mg_smem[10 * D.n + k] = D.b[k];
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  mg_bottom_cycle(mg_smem, lv, l0, L, ci);
  for (int k = threadIdx.x; k < D.n; k += blockDim.x) D.x[k] = mg_smem[11 * D.n + k];
}

// ---- host: hierarchy --------------------------------------------------------
struct HostLevel {
  int nx, ny, per_x, per_y;
  std::vector<double> coef;  // 9 x n (node-major per offset)
  std::vector<char> active;  // node takes part in the correction
};

static bool can_coarsen(int n, int per) { return n >= (per ? 6 : 3); }

// Galerkin P^T A P of a level onto its coarsening
static HostLevel galerkin(const HostLevel &F, int cx, int cy) {
  HostLevel C;
  C.nx = cx ? coarse_nodes(F.nx, F.per_x) : F.nx;
  C.ny = cy ? coarse_nodes(F.ny, F.per_y) : F.ny;
  C.per_x = F.per_x;
  C.per_y = F.per_y;
  const int nf = F.nx * F.ny, nc = C.nx * C.ny;
  C.coef.assign((size_t)9 * nc, 0.0);
  auto cdelta = [](int a, int b, int n, int per) {  // b - a in {-1, 0, 1}
    int d = b - a;
    if (per && n > 2) {
      if (d > 1) d -= n;
      if (d < -1) d += n;
    }
    return d;
  };
  for (int k = 0; k < nf; k++) {
    if (!F.active[k]) continue;
    const int j = k / F.nx, i = k - j * F.nx;
    int fci[2], fcj[2];
    float fwi[2], fwj[2];
    const int fpi = axis_parents(i, F.nx, C.nx, cx, F.per_x, fci, fwi);
    const int fpj = axis_parents(j, F.ny, C.ny, cy, C.per_y, fcj, fwj);
    for (int dy = -1; dy <= 1; dy++)
      for (int dx = -1; dx <= 1; dx++) {
        const double a = F.coef[(size_t)((dy + 1) * 3 + dx + 1) * nf + k];
        if (a == 0.0) continue;
        int gi = i + dx, gj = j + dy;
        gi = gi < 0 ? gi + F.nx : (gi >= F.nx ? gi - F.nx : gi);
        gj = gj < 0 ? gj + F.ny : (gj >= F.ny ? gj - F.ny : gj);
        if (!F.active[gi + F.nx * gj]) continue;
        int gci[2], gcj[2];
        float gwi[2], gwj[2];
        const int gpi = axis_parents(gi, F.nx, C.nx, cx, C.per_x, gci, gwi);
        const int gpj = axis_parents(gj, F.ny, C.ny, cy, C.per_y, gcj, gwj);
        for (int p1 = 0; p1 < fpj; p1++)
          for (int p0 = 0; p0 < fpi; p0++) {
            const int I = fci[p0], J = fcj[p1];
            const double wf = (double)fwi[p0] * (double)fwj[p1];
            for (int q1 = 0; q1 < gpj; q1++)
              for (int q0 = 0; q0 < gpi; q0++) {
                const int ddx = cdelta(I, gci[q0], C.nx, C.per_x), ddy = cdelta(J, gcj[q1], C.ny, C.per_y);
                const double v = wf * a * (double)gwi[q0] * (double)gwj[q1];
                C.coef[(size_t)((ddy + 1) * 3 + ddx + 1) * nc + I + C.nx * J] += v;
              }
          }
      }
  }
  C.active.assign(nc, 0);
  double mx = 0;
  for (int K = 0; K < nc; K++) mx = std::max(mx, std::fabs(C.coef[(size_t)4 * nc + K]));
  for (int K = 0; K < nc; K++) C.active[K] = C.coef[(size_t)4 * nc + K] > 1e-12 * mx;
  for (int K = 0; K < nc; K++)
    if (!C.active[K])
      for (int o = 0; o < 9; o++) C.coef[(size_t)o * nc + K] = 0.0;
  return C;
}

// inverse of the active part of a small SPD level (Gauss-Jordan, FP64)
static std::vector<float> dense_inverse(const HostLevel &L) {
  const int n = L.nx * L.ny;
  std::vector<double> A((size_t)n * n, 0.0), Inv((size_t)n * n, 0.0);
  for (int k = 0; k < n; k++) {
    Inv[(size_t)k * n + k] = 1.0;
    if (!L.active[k]) {
      A[(size_t)k * n + k] = 1.0;
      continue;
    }
    const int j = k / L.nx, i = k - j * L.nx;
    for (int dy = -1; dy <= 1; dy++)
      for (int dx = -1; dx <= 1; dx++) {
        const double a = L.coef[(size_t)((dy + 1) * 3 + dx + 1) * n + k];
        if (a == 0.0) continue;
        int gi = i + dx, gj = j + dy;
        gi = gi < 0 ? gi + L.nx : (gi >= L.nx ? gi - L.nx : gi);
        gj = gj < 0 ? gj + L.ny : (gj >= L.ny ? gj - L.ny : gj);
        const int g = gi + L.nx * gj;
        if (L.active[g]) A[(size_t)k * n + g] += a;
      }
  }
  for (int c = 0; c < n; c++) {
    int piv = c;
    for (int r = c + 1; r < n; r++)
      if (std::fabs(A[(size_t)r * n + c]) > std::fabs(A[(size_t)piv * n + c])) piv = r;
    if (piv != c)
      for (int q = 0; q < n; q++) {
        std::swap(A[(size_t)c * n + q], A[(size_t)piv * n + q]);
        std::swap(Inv[(size_t)c * n + q], Inv[(size_t)piv * n + q]);
      }
    const double d = A[(size_t)c * n + c];
    const double id = d != 0.0 ? 1.0 / d : 0.0;
    for (int q = 0; q < n; q++) {
      A[(size_t)c * n + q] *= id;
      Inv[(size_t)c * n + q] *= id;
    }
    for (int r = 0; r < n; r++) {
      if (r == c) continue;
      const double f = A[(size_t)r * n + c];
      if (f == 0.0) continue;
      for (int q = 0; q < n; q++) {
        A[(size_t)r * n + q] -= f * A[(size_t)c * n + q];
        Inv[(size_t)r * n + q] -= f * Inv[(size_t)c * n + q];
      }
    }
  }
  std::vector<float> out((size_t)n * n);
  for (int r = 0; r < n; r++)
    for (int q = 0; q < n; q++)
      out[(size_t)r * n + q] = (L.active[r] && L.active[q]) ? (float)Inv[(size_t)r * n + q] : 0.f;
  return out;
}

// Builds the hierarchy of the scaled operator S: per node its five
// coefficients s0 (diagonal), sW, sE, sS, sN (to the wrapped neighbours;
// zero where the assembled operator has no coupling) and whether the node is
// free (identity rows are not).  per_x / per_y: some row couples across the
// x / y seam.
int mg_build(Ctx *c, int nx, int ny, const std::vector<double> &s0, const std::vector<double> &sW,
             const std::vector<double> &sE, const std::vector<double> &sS, const std::vector<double> &sN,
             const std::vector<char> &free_row, int per_x, int per_y, Mg **out) {
  *out = nullptr;
  std::vector<HostLevel> H(1);
  HostLevel &L0 = H[0];
  L0.nx = nx;
  L0.ny = ny;
  L0.per_x = per_x;
  L0.per_y = per_y;
  const int n0 = nx * ny;
  L0.coef.assign((size_t)9 * n0, 0.0);
  L0.active = free_row;
  for (int k = 0; k < n0; k++) {
    if (!free_row[k]) continue;
    const int j = k / nx, i = k - j * nx;
    const int w = i > 0 ? k - 1 : k + nx - 1, e = i < nx - 1 ? k + 1 : k - nx + 1;
    const int s = j > 0 ? k - nx : k + nx * (ny - 1), nn_ = j < ny - 1 ? k + nx : k - nx * (ny - 1);
    L0.coef[(size_t)4 * n0 + k] = s0[k];
    if (free_row[w]) L0.coef[(size_t)3 * n0 + k] += sW[k];
    if (free_row[e]) L0.coef[(size_t)5 * n0 + k] += sE[k];
    if (free_row[s]) L0.coef[(size_t)1 * n0 + k] += sS[k];
    if (free_row[nn_]) L0.coef[(size_t)7 * n0 + k] += sN[k];
  }
  std::vector<int> cxs, cys;
  while (H.back().nx * H.back().ny > (H.size() == 1 ? kMgSingle : kMgCoarsest)) {
    const HostLevel &F = H.back();
    const int cx = can_coarsen(F.nx, F.per_x), cy = can_coarsen(F.ny, F.per_y);
    if (!cx && !cy) break;
    cxs.push_back(cx);
    cys.push_back(cy);
    H.push_back(galerkin(F, cx, cy));
  }
  if (H.back().nx * H.back().ny > 4096) return set_err(c, ISKRA_EINVAL, "multigrid: coarsest level too large");
  Mg *m = new Mg();
  m->lv.resize(H.size());
  for (size_t l = 0; l < H.size(); l++) {
    MgLevel &D = m->lv[l];
    const HostLevel &S = H[l];
    D.nx = S.nx;
    D.ny = S.ny;
    D.n = S.nx * S.ny;
    D.seam_x = seam(S.nx, S.per_x);
    D.seam_y = seam(S.ny, S.per_y);
    D.cx = l + 1 < H.size() ? cxs[l] : 0;
    D.cy = l + 1 < H.size() ? cys[l] : 0;
    D.five = 1;
    for (int o : {0, 2, 6, 8})
      for (int k = 0; k < D.n && D.five; k++)
        if (S.coef[(size_t)o * D.n + k] != 0.0) D.five = 0;
    std::vector<float> cf(S.coef.begin(), S.coef.end()), dinv(D.n, 0.f);
    for (int k = 0; k < D.n; k++)
      if (S.active[k] && S.coef[(size_t)4 * D.n + k] > 0) dinv[k] = kMgOmega / (float)S.coef[(size_t)4 * D.n + k];
    bool ok = cudaMalloc(&D.coef, cf.size() * sizeof(float)) == cudaSuccess &&
              cudaMalloc(&D.dinv, D.n * sizeof(float)) == cudaSuccess &&
              cudaMalloc(&D.x, D.n * sizeof(float)) == cudaSuccess &&
              cudaMalloc(&D.x2, D.n * sizeof(float)) == cudaSuccess &&
              cudaMalloc(&D.b, D.n * sizeof(float)) == cudaSuccess;
    if (!ok) {
      mg_destroy(m);
      return set_err(c, ISKRA_ENOMEM, "multigrid levels");
    }
    cudaMemcpy(D.coef, cf.data(), cf.size() * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemcpy(D.dinv, dinv.data(), D.n * sizeof(float), cudaMemcpyHostToDevice);
  }
  const std::vector<float> inv = dense_inverse(H.back());
  if (cudaMalloc(&m->cinv, inv.size() * sizeof(float)) != cudaSuccess) {
    mg_destroy(m);
    return set_err(c, ISKRA_ENOMEM, "multigrid coarsest inverse");
  }
  cudaMemcpy(m->cinv, inv.data(), inv.size() * sizeof(float), cudaMemcpyHostToDevice);
  // the single-block bottom: the smallest levels (from level 1 on, so that
  // level 0's FP64 conversions stay in its own kernels) that fit its shared
  // memory together
  const int L = (int)m->lv.size();
  if (cudaMalloc(&m->dlv, L * sizeof(MgLevel)) != cudaSuccess) {
    mg_destroy(m);
    return set_err(c, ISKRA_ENOMEM, "multigrid level table");
  }
  cudaMemcpy(m->dlv, m->lv.data(), L * sizeof(MgLevel), cudaMemcpyHostToDevice);
  if (L > 1) {
    int l0 = L, nodes = 0;
    const int nc = m->lv[L - 1].n;
    if (nc <= kMgCoarsest)
      while (l0 > 1 && nodes + m->lv[l0 - 1].n <= kMgBottomNodes) nodes += m->lv[--l0].n;
    if (l0 < L) {
      m->bottom = l0;
      m->bottom_smem = ((size_t)nodes * kMgBottomWords + (size_t)nc * nc) * sizeof(float);
      cudaFuncSetAttribute(k_mg_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (kMgBottomNodes * kMgBottomWords + kMgCoarsest * kMgCoarsest) * (int)sizeof(float));
    }
  }
  setup_copies_done();
  *out = m;
  return ISKRA_OK;
}

// The hierarchy for a one-block solve (poisson.cu): every level and, when it has
// one, the coarsest inverse at most 128 x 128, in shared memory.
bool mg_block_view(const Mg *m, MgBlock *v) {
  if (!m || !m->dlv) return false;
  *v = MgBlock{};
  v->lv = m->dlv;
  v->L = (int)m->lv.size();
  v->cinv = m->cinv;
  size_t words = 0;
  for (const auto &l : m->lv) words += (size_t)kMgBottomWords * l.n;
  const int nc = m->lv.back().n;
  v->cinv_shared = nc <= kMgCoarsest;
  v->bytes = (words + (v->cinv_shared ? (size_t)nc * nc : 0)) * sizeof(float);
  return true;
}

int mg_levels(const Mg *m) { return m ? (int)m->lv.size() : 0; }

// z = M^-1 r: one V(2,2) cycle on the scaled residual r (FP64, free rows);
// every kernel returns at once while *skip is set (a converged solve).  Level
// 0 reads r in FP64 and writes z in FP64 with the dot products of D; a
// hierarchy of one level leaves those to the caller (*dots_done = false).
int mg_queue_cycle(Ctx *c, Mg *m, const double *r, double *z, const int *skip, const PcgDots &D, bool *dots_done) {
  cudaStream_t st = c->stream;
  const int L = (int)m->lv.size();
  *dots_done = L > 1;
  auto xfer = [&](int l) {
    const MgLevel &F = m->lv[l], &C = m->lv[l + 1];
    return MgXfer{F.nx, F.ny, C.nx, C.ny, F.cx, F.cy, F.seam_x, F.seam_y};
  };
  const int lb = m->bottom ? m->bottom : L - 1;  // first level not run by per-level kernels
  for (int l = 0; l < lb; l++) {
    MgLevel &F = m->lv[l], &C = m->lv[l + 1];
    // tiles over the fine nodes (kSeamJump has one beyond the last coarse node's two)
    const int ox = F.cx ? 2 * kDownCx : kDownCx, oy = F.cy ? 2 * kDownCy : kDownCy;
    const dim3 g((F.nx + ox - 1) / ox, (F.ny + oy - 1) / oy);
    ISKRA_CUDA(c, launch_pdl(F.five ? k_mg_down<true> : k_mg_down<false>, g, kDownThreads, 0, st,
                             (const float *)F.coef, (const float *)F.dinv, F.x, (const float *)F.b, C.b, xfer(l), skip,
                             l == 0 ? r : nullptr));
  }
  if (m->bottom) {
    ISKRA_CUDA(c, launch_pdl(k_mg_bottom, 1, kMgBottomThreads, m->bottom_smem, st, (const MgLevel *)m->dlv, m->bottom,
                             L, (const float *)m->cinv, skip));
  } else {
    MgLevel &C = m->lv[L - 1];
    ISKRA_CUDA(c, launch_pdl(k_mg_coarse, std::max(1, std::min(c->num_sms * 2, (C.n + 7) / 8)), 256, 0, st,
                             (const float *)m->cinv, (const float *)C.b, C.x, C.n, skip, L == 1 ? r : nullptr,
                             L == 1 ? z : nullptr));
  }
  for (int l = lb - 1; l >= 0; l--) {
    MgLevel &F = m->lv[l];
    // the coarser level's correction: in x2 from its own k_mg_up, in x from the bottom
    const float *xc = l + 1 < lb ? m->lv[l + 1].x2 : m->lv[l + 1].x;
    const int tiles = ((F.nx + kUpX - 1) / kUpX) * ((F.ny + kUpY - 1) / kUpY);
    const int g = l == 0 ? std::min(tiles, std::min(kPcgPartials, c->num_sms * 2)) : tiles;  // 736 threads: 2 per SM
    ISKRA_CUDA(c, launch_pdl(F.five ? k_mg_up<true> : k_mg_up<false>, g, kUpThreads, 0, st, (const float *)F.coef,
                             (const float *)F.dinv, (const float *)F.x, (const float *)F.b, xc, F.x2, xfer(l), skip,
                             l == 0 ? r : nullptr, l == 0 ? z : nullptr, D));
  }
  ISKRA_CUDA(c, cudaGetLastError());
  return ISKRA_OK;
}

}  // namespace iskra
