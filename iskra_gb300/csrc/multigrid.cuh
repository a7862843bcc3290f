// multigrid.cuh -- the V-cycle's levels and the device code that works on them
// in shared memory: the cycle's kernels (multigrid.cu) and the one-block solve of
// small grids (poisson.cu).
#pragma once
#include "internal.cuh"

namespace iskra {

// Nodes of the level solved by its dense inverse: a grid of up to 400 nodes as
// it is (its inverse then makes the whole cycle exact), the coarsest of several
// levels at most 128, so that its inverse fits the bottom block's shared memory
// (64 KB) beside the levels above it.
constexpr int kMgCoarsest = 128, kMgSingle = 400;

struct MgLevel {
  int nx = 0, ny = 0, n = 0;
  int seam_x = 0, seam_y = 0;  // kSeam* of the axis
  int cx = 0, cy = 0;          // x / y coarsened towards the next level
  int five = 0;                // no corner couplings (5-point stencil)
  float *coef = nullptr;       // 9 x n: offset o = (dy + 1) 3 + (dx + 1), node-major
  float *dinv = nullptr;       // omega / diagonal, 0 on nodes outside the correction
  float *x = nullptr, *x2 = nullptr, *b = nullptr;
};

// ---- kernels (FP32) ----------------------------------------------------------
// Every stencil load is issued unconditionally (a zero coefficient multiplies a
// finite x) so that the loads of a node overlap.  FIVE: the level has no corner
// couplings (level 0, the 5-point operator): the four corner planes are neither
// read nor multiplied.
__device__ __forceinline__ int wrap_idx(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
// any position of a tile and its halo to its node (tiles may be wider than the grid)
__device__ __forceinline__ int wrap_any(int i, int n) {
  if ((unsigned)i < (unsigned)n) return i;
  const int m = i % n;
  return m < 0 ? m + n : m;
}

// a node's stencil coefficients in registers
template <bool FIVE>
struct MgStencil {
  float c[FIVE ? 5 : 9];
};
template <bool FIVE>
__device__ __forceinline__ MgStencil<FIVE> mg_stencil(const float *__restrict__ coef, int k, int n) {
  MgStencil<FIVE> S;
  constexpr int o[9] = {4, 1, 3, 5, 7, 0, 2, 6, 8};
#pragma unroll
  for (int q = 0; q < (FIVE ? 5 : 9); q++) S.c[q] = __ldg(coef + (size_t)o[q] * n + k);
  return S;
}
// (A x) at a node from shared memory: x points at the node's value, rows W apart
template <bool FIVE>
__device__ __forceinline__ float apply9t(const MgStencil<FIVE> &S, const float *x, int W) {
  float a = S.c[0] * x[0];
  a = fmaf(S.c[1], x[-W], a);
  a = fmaf(S.c[2], x[-1], a);
  a = fmaf(S.c[3], x[1], a);
  a = fmaf(S.c[4], x[W], a);
  if (!FIVE) {
    a = fmaf(S.c[FIVE ? 0 : 5], x[-W - 1], a);
    a = fmaf(S.c[FIVE ? 0 : 6], x[-W + 1], a);
    a = fmaf(S.c[FIVE ? 0 : 7], x[W - 1], a);
    a = fmaf(S.c[FIVE ? 0 : 8], x[W + 1], a);
  }
  return a;
}

enum { kSeamOpen = 0, kSeamEven = 1, kSeamJump = 2 };  // (multigrid.cu, interpolation weights)
struct MgXfer {
  int nx, ny, ncx, ncy, cx, cy, seam_x, seam_y;
};

// Weight along one axis of fine index f = 2I + d in coarse index I's restriction
// (axis_parents transposed): 1 at d = 0, 1/2 beside it, 1 on the last odd node
// when it has one parent and on kSeamJump's last node (f = -1), 0 outside the axis.
__device__ __forceinline__ float restrict_weight(int f, int d, int n, int nc, int seam) {
  if (d == 0) return 1.f;
  if (seam == kSeamEven) return 0.5f;
  if (f < 0) return seam == kSeamJump ? 1.f : 0.f;
  if (f >= n) return 0.f;
  return d > 0 && (f + 1) >> 1 >= nc ? 1.f : 0.5f;
}

// coarse b = P^T r at coarse node (I, J), gathered from its fine candidates
// 2I-1, 2I, 2I+1 (I itself on an axis that is not coarsened); r(fi, fj) takes
// the candidates as formed, wrapping at a periodic end is the caller's
template <class R>
__device__ __forceinline__ float restrict_at(R r, const MgXfer &T, int I, int J) {
  float s = 0.f;
#pragma unroll
  for (int dj = -1; dj <= 1; dj++) {
    if (!T.cy && dj) continue;
    const int fj = T.cy ? 2 * J + dj : J;
    const float wy = restrict_weight(fj, dj, T.ny, T.ncy, T.seam_y);
    if (wy == 0.f) continue;
#pragma unroll
    for (int di = -1; di <= 1; di++) {
      if (!T.cx && di) continue;
      const int fi = T.cx ? 2 * I + di : I;
      const float wx = restrict_weight(fi, di, T.nx, T.ncx, T.seam_x);
      if (wx != 0.f) s = fmaf(wx * wy, r(fi, fj), s);
    }
  }
  return s;
}

// the parents of fine index i along one axis (axis_parents): c0, and c1 >= 0
// when two share it equally
__device__ __forceinline__ void prolong_parents(int i, int nc, int coarsened, int seam, int &c0, int &c1) {
  c0 = coarsened ? i >> 1 : i;
  c1 = -1;
  if (coarsened && c0 >= nc) c0 = 0;  // kSeamJump's last node
  if (coarsened && (i & 1)) {
    const int hi = (i + 1) >> 1;
    c1 = hi < nc ? hi : seam == kSeamEven ? 0 : -1;
  }
}

// (P xc) at fine node (i, j)
__device__ __forceinline__ float prolong_at(const float *xc, const MgXfer &T, int i, int j) {
  int i0, i1, j0, j1;
  prolong_parents(i, T.ncx, T.cx, T.seam_x, i0, i1);
  prolong_parents(j, T.ncy, T.cy, T.seam_y, j0, j1);
  const float w = (i1 >= 0 ? 0.5f : 1.f) * (j1 >= 0 ? 0.5f : 1.f);
  float v = w * xc[i0 + T.ncx * j0];
  if (i1 >= 0) v = fmaf(w, xc[i1 + T.ncx * j0], v);
  if (j1 >= 0) {
    v = fmaf(w, xc[i0 + T.ncx * j1], v);
    if (i1 >= 0) v = fmaf(w, xc[i1 + T.ncx * j1], v);
  }
  return v;
}

// The smallest levels of the cycle in one block: levels l0 .. L-1 (together at
// most kMgBottomNodes nodes) get the same sweeps, residuals, transfers and
// coarsest solve as the per-level kernels, separated by block barriers
// instead of launches -- at a few thousand nodes a launch costs more than the
// level's work.  The levels' coefficients and vectors and the coarsest inverse
// live in shared memory (14 words a node, staged once, before the kernel waits
// for its predecessor): read from L2 in each of the cycle's phases they made the
// block 18 us (1024 + 256 nodes) to 30 us (1075 + 300) of dependent loads; now 12
// and 14.
// Leaves the correction in lv[l0].x.
constexpr int kMgBottomNodes = 2400;
constexpr int kMgBottomWords = 14;  // per node: 9 coefficients, dinv, b, x, x2, r
constexpr int kMgBottomThreads = 1024;

// shared-memory view of one bottom level
struct MgSh {
  float *coef, *dinv, *b, *x, *x2, *r;
  int nx, ny, n;
};
__device__ __forceinline__ MgSh mg_sh(float *base, const MgLevel &D) {
  MgSh q;
  q.nx = D.nx;
  q.ny = D.ny;
  q.n = D.n;
  q.coef = base;
  q.dinv = base + 9 * D.n;
  q.b = base + 10 * D.n;
  q.x = base + 11 * D.n;
  q.x2 = base + 12 * D.n;
  q.r = base + 13 * D.n;
  return q;
}
__device__ __forceinline__ float mg_apply(const MgSh &q, const float *x, int i, int j) {
  const int iw = wrap_idx(i - 1, q.nx), ie = wrap_idx(i + 1, q.nx), k = i + q.nx * j, n = q.n;
  const float *xs = x + q.nx * wrap_idx(j - 1, q.ny), *x0 = x + q.nx * j, *xn = x + q.nx * wrap_idx(j + 1, q.ny);
  float a = q.coef[4 * n + k] * x0[i];
  a = fmaf(q.coef[1 * n + k], xs[i], a);
  a = fmaf(q.coef[3 * n + k], x0[iw], a);
  a = fmaf(q.coef[5 * n + k], x0[ie], a);
  a = fmaf(q.coef[7 * n + k], xn[i], a);
  a = fmaf(q.coef[0 * n + k], xs[iw], a);
  a = fmaf(q.coef[2 * n + k], xs[ie], a);
  a = fmaf(q.coef[6 * n + k], xn[iw], a);
  return fmaf(q.coef[8 * n + k], xn[ie], a);
}
// f(i, j, k) for every node of a level: thread (x, y) of a 32-wide block takes
// nodes (x + 32 a, y + rows b)
template <class F>
__device__ __forceinline__ void mg_nodes(int nx, int ny, F f) {
  for (int j = threadIdx.x >> 5; j < ny; j += blockDim.x >> 5)
    for (int i = threadIdx.x & 31; i < nx; i += 32) f(i, j, i + nx * j);
}

// One cycle on the levels l0 .. L-1 held in shared memory (base), the
// right-hand side in the first one's b; cinv: the coarsest inverse (shared or
// global memory).  Ends with a block barrier.
__device__ __forceinline__ void mg_bottom_cycle(float *base, const MgLevel *__restrict__ lv, int l0, int L,
                                                const float *cinv) {
  auto xfer = [&](int l) {
    const MgLevel &F = lv[l], &C = lv[l + 1];
    return MgXfer{F.nx, F.ny, C.nx, C.ny, F.cx, F.cy, F.seam_x, F.seam_y};
  };
  float *at = base;
  for (int l = l0; l + 1 < L; l++) {
    const MgSh q = mg_sh(at, lv[l]);
    at += kMgBottomWords * q.n;
    const MgSh C = mg_sh(at, lv[l + 1]);
    mg_nodes(q.nx, q.ny, [&](int, int, int k) { q.x2[k] = __fmul_rn(q.dinv[k], q.b[k]); });
    __syncthreads();
    mg_nodes(q.nx, q.ny, [&](int i, int j, int k) {
      q.x[k] = q.dinv[k] != 0.f ? fmaf(q.dinv[k], q.b[k] - mg_apply(q, q.x2, i, j), q.x2[k]) : 0.f;
    });
    __syncthreads();
    mg_nodes(q.nx, q.ny, [&](int i, int j, int k) {
      q.r[k] = q.dinv[k] != 0.f ? q.b[k] - mg_apply(q, q.x, i, j) : 0.f;
    });
    __syncthreads();
    const MgXfer T = xfer(l);
    mg_nodes(C.nx, C.ny, [&](int I, int J, int k) {
      C.b[k] = restrict_at([&](int fi, int fj) { return q.r[wrap_idx(fi, T.nx) + T.nx * wrap_idx(fj, T.ny)]; }, T, I,
                           J);
    });
    __syncthreads();
  }
  {
    // eight lanes per row
    const MgSh C = mg_sh(at, lv[L - 1]);
    const int sub = threadIdx.x & 7;
    for (int row0 = 0; row0 < C.n; row0 += blockDim.x >> 3) {
      const int row = row0 + (threadIdx.x >> 3);
      float acc = 0.f;
      if (row < C.n)
        for (int c = sub; c < C.n; c += 8) acc = fmaf(cinv[row * C.n + c], C.b[c], acc);
      for (int o = 4; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, 8);
      if (sub == 0 && row < C.n) C.x[row] = acc;
    }
    __syncthreads();
  }
  for (int l = L - 2; l >= l0; l--) {
    at -= kMgBottomWords * lv[l].n;
    const MgSh q = mg_sh(at, lv[l]);
    const MgSh C = mg_sh(at + kMgBottomWords * q.n, lv[l + 1]);
    const MgXfer T = xfer(l);
    mg_nodes(q.nx, q.ny, [&](int i, int j, int k) {
      if (q.dinv[k] != 0.f) q.x[k] += prolong_at(C.x, T, i, j);
    });
    __syncthreads();
    mg_nodes(q.nx, q.ny, [&](int i, int j, int k) {
      q.x2[k] = q.dinv[k] != 0.f ? q.x[k] + q.dinv[k] * (q.b[k] - mg_apply(q, q.x, i, j)) : 0.f;
    });
    __syncthreads();
    mg_nodes(q.nx, q.ny, [&](int i, int j, int k) {
      q.x[k] = q.dinv[k] != 0.f ? q.x2[k] + q.dinv[k] * (q.b[k] - mg_apply(q, q.x2, i, j)) : 0.f;
    });
    __syncthreads();
  }
}

// coefficients of the levels l0 .. L-1 and the coarsest inverse into shared
// memory (one cp.async group, for the caller to wait for); returns the inverse's
// place
__device__ __forceinline__ float *mg_bottom_stage(float *base, const MgLevel *__restrict__ lv, int l0, int L,
                                                  const float *__restrict__ cinv, bool with_inverse = true) {
  // asynchronous 4-byte copies: all in flight together (the planes of odd-sized
  // levels have no common 16-byte alignment)
  auto copy = [](float *dst, const float *src, int n) {
    for (int t = threadIdx.x; t < n; t += blockDim.x)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst + t)),
                   "l"(src + t)
                   : "memory");
  };
  float *at = base;
  for (int l = l0; l < L; l++) {
    const MgLevel &D = lv[l];
    copy(at, D.coef, 9 * D.n);
    copy(at + 9 * D.n, D.dinv, D.n);
    at += kMgBottomWords * D.n;
  }
  const int nc = lv[L - 1].n;
  if (with_inverse) copy(at, cinv, nc * nc);
  asm volatile("cp.async.commit_group;" ::: "memory");
  return at;
}

// What a one-block solve needs of a hierarchy (mg_block_view).
struct MgBlock {
  const MgLevel *lv = nullptr;  // device table of the levels
  int L = 0;
  const float *cinv = nullptr;
  int cinv_shared = 0;          // the coarsest inverse is staged in shared memory too
  size_t bytes = 0;             // shared memory of the levels (and the inverse)
};
bool mg_block_view(const Mg *m, MgBlock *v);

}  // namespace iskra
