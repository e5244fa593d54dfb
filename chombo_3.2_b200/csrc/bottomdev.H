// The bottom solve's device code (BiCGStab and relaxation), written once over
// a context that says where the vectors live and how threads synchronise and
// sum: one thread block, a whole cooperative grid (kernels.cu), or a
// thread-block cluster holding the level in shared memory (coarse.cu).
#ifndef CMG_BOTTOMDEV_H
#define CMG_BOTTOMDEV_H

#include <cooperative_groups.h>

#include "cellops.H"
#include "kernels.H"

namespace cmg {
namespace cg = cooperative_groups;

// ---------------------------------------------------------------- bottom
// BiCGStabSolver<T>::solve (AMRElliptic/BiCGStabSolver.H:199-515) and
// RelaxSolver<T>::solve (RelaxSolver.H:128-186) on the deepest multigrid
// level, every dot product and norm summed in the reference's order: per box
// in x-fastest order (FArrayBox::dotProduct, FArrayBox.cpp:260-280;
// FArrayBox::sumPow pencil order, FArrayBox.cpp:168-209), then box by box
// from zero.  The vectors live in the bottom level's compact slot space (its
// valid cells, BottomPlan).  A stencil read of a face ghost goes straight to
// the valid cell that the level's exchange or boundary condition copies
// there (nbv: the source slot, or -(slot + 1) for a homogeneous Dirichlet
// ghost, read as 0 - value the way the BC writes it).  A ghost is only read
// while its source is not written (a colour pass reads the other colour; an
// operator apply writes another vector), so the value read is the one an
// exchange just before the pass would have left there.
// Three ways to run: in shared memory across a thread-block cluster
// (ClusterCtx, coarse.cu: every level that fits), one thread block per
// hierarchy on global vectors (BlkCtx), or the whole grid of one cooperative
// launch for one hierarchy with a large bottom level (GridCtx), its phases
// separated by grid barriers and its sums folded by block 0 from shared memory.
struct BottomArgs {
  BottomWork W;
  const BoxDesc* boxes;
  Scal sc;
  int vc;
  double* phiFab;
  const double* rhsFab;
  double *phi, *rhs, *r, *rt, *e, *p, *pt, *st, *t, *v;
  double eps, reps, hang, small, mult;
  const double* metric;  // device scalar: the solve's initial residual norm
  int imax, numRestarts;
  BottomConfig cfg;
  const double* epsPer;  // per block (hierarchy) tolerance of a BiCGStab bottom, or null
};

constexpr int kBottomGridThreads = 256;
constexpr int kBottomStage = 2048;  // doubles per fold chunk staged in shared memory (grid)

// In-order fold of p[0..n): a sum from zero, or a NaN-keeping max from zero.
__device__ __forceinline__ double foldRun(double acc, const double* p, int n, bool mx) {
  if (mx) {
    for (int b = 0; b < n; ++b) acc = nanMax(acc, p[b]);
  } else {
    for (int b = 0; b < n; ++b) acc += p[b];
  }
  return acc;
}

struct BlkCtx {
  static constexpr bool kGrid = false;
  static constexpr bool kCluster = false;
  double* part;   // per-box partials (dynamic shared memory)
  double* part2;  // a second set, for two sums folded together
  double* scal;   // 8 rotating broadcast slots (shared)
  int k;
  __device__ int tid() const { return threadIdx.x; }
  __device__ int nthr() const { return blockDim.x; }
  __device__ bool lead() const { return threadIdx.x == 0; }
  __device__ void sync() const { __syncthreads(); }
  // Folds part[0..n) (and part2 when two) once every thread has written its
  // partials; every thread gets the results.  A broadcast slot is written
  // again only four folds later, after every thread has read it.
  __device__ void reduce(int n, bool two, bool mx, double& r1, double& r2) {
    __syncthreads();
    const int s = k;
    k = (k + 2) & 7;
    if (threadIdx.x == 0) scal[s] = foldRun(0.0, part, n, mx);
    if (two && threadIdx.x == 32) scal[s + 1] = foldRun(0.0, part2, n, mx);
    __syncthreads();
    r1 = scal[s];
    if (two) r2 = scal[s + 1];
  }
};

struct GridCtx {
  static constexpr bool kGrid = true;
  static constexpr bool kCluster = false;
  double* part;   // per-box partials (global)
  double* part2;
  double* scal;   // 8 rotating broadcast slots (global)
  double* stage;  // 2 x kBottomStage doubles of shared memory
  int k;
  __device__ int tid() const { return blockIdx.x * blockDim.x + threadIdx.x; }
  __device__ int nthr() const { return gridDim.x * blockDim.x; }
  __device__ bool lead() const { return tid() == 0; }
  __device__ void sync() const { cg::this_grid().sync(); }
  __device__ void reduce(int n, bool two, bool mx, double& r1, double& r2) {
    cg::this_grid().sync();
    const int s = k;
    k = (k + 2) & 7;
    if (blockIdx.x == 0) {
      double a1 = 0.0, a2 = 0.0;
      for (int base = 0; base < n; base += kBottomStage) {
        const int m = min(kBottomStage, n - base);
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
          stage[i] = __ldcg(part + base + i);
          if (two) stage[kBottomStage + i] = __ldcg(part2 + base + i);
        }
        __syncthreads();
        if (threadIdx.x == 0) a1 = foldRun(a1, stage, m, mx);
        if (two && threadIdx.x == 32) a2 = foldRun(a2, stage + kBottomStage, m, mx);
        __syncthreads();
      }
      if (threadIdx.x == 0) scal[s] = a1;
      if (two && threadIdx.x == 32) scal[s + 1] = a2;
    }
    cg::this_grid().sync();
    r1 = __ldcg(scal + s);
    if (two) r2 = __ldcg(scal + s + 1);
  }
};

template <class C, class F>
__device__ __forceinline__ void bCells(C& c, int n, F fn) {
  for (int q = c.tid(); q < n; q += c.nthr()) fn(q);
  c.sync();
}

// The same writing the vector x, whose neighbours a stencil reads next.
template <class C, class F>
__device__ __forceinline__ void bCellsOf(C& c, int n, double* x, F fn) {
  for (int q = c.tid(); q < n; q += c.nthr()) fn(q);
  if constexpr (C::kCluster)
    c.publish(x);
  else
    c.sync();
}

// A face neighbour's value: the slot itself, or 0 - the source of a
// homogeneous Dirichlet ghost.
__device__ __forceinline__ double gval(const double* f, int v) { return v >= 0 ? f[v] : 0.0 - f[-v - 1]; }

// The partial sum of box b: x.y in x-fastest order, or sumPow(2) of x.
inline __device__ double boxPartial(const BottomArgs& A, int b, const double* x, const double* y, bool pencil) {
  const BoxDesc bd = A.boxes[b];
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1, nz = bd.hi[2] - bd.lo[2] + 1;
  const int s0 = A.W.boxStart[b];
  double s = 0.0;
  if (!pencil) {
    for (int q = s0; q < s0 + nx * ny * nz; ++q) s += x[q] * y[q];
  } else {
    // sumPow(p=2): per-x accumulation over pencils, then across x.
    for (int i = 0; i < nx; ++i) {
      double acc = 0.0;
      bool first = true;
      for (int k = 0; k < nz; ++k)
        for (int j = 0; j < ny; ++j) {
          double v = x[s0 + i + nx * (j + ny * k)];
          acc = first ? v * v : acc + v * v;
          first = false;
        }
      s = (i == 0) ? acc : s + acc;
    }
  }
  return s;
}

template <class C>
__device__ double bDot(C& c, const BottomArgs& A, const double* x, const double* y, bool pencil) {
  if constexpr (C::kCluster) {
    double r, unused;
    if (pencil)
      c.norm2(A, x, nullptr, nullptr, r, unused);
    else
      c.dots(A, x, y, nullptr, nullptr, r, unused);
    return r;
  } else {
  for (int b = c.tid(); b < A.W.nbox; b += c.nthr()) c.part[b] = boxPartial(A, b, x, y, pencil);
  double r, unused;
  c.reduce(A.W.nbox, false, false, r, unused);
  return r;
  }
}

// x1.y1 and x2.y2, each in the reference's order, folded side by side.
template <class C>
__device__ void bDot2(C& c, const BottomArgs& A, const double* x1, const double* y1, const double* x2,
                      const double* y2, double& r1, double& r2) {
  if constexpr (C::kCluster) {
    c.dots(A, x1, y1, x2, y2, r1, r2);
  } else {
  for (int b = c.tid(); b < A.W.nbox; b += c.nthr()) {
    c.part[b] = boxPartial(A, b, x1, y1, false);
    c.part2[b] = boxPartial(A, b, x2, y2, false);
  }
  c.reduce(A.W.nbox, true, false, r1, r2);
  }
}

// The norm of type A.cfg.normType: 2 the reference-ordered sqrt(sumPow),
// 0 the largest |x| (a max, so its order does not matter; NaN propagates).
template <class C>
__device__ double bNormType(C& c, const BottomArgs& A, const double* x) {
  if (A.cfg.normType == 2) return sqrt(bDot(c, A, x, x, true));
  if constexpr (C::kCluster) {
    return c.normMax(A, x);
  } else {
  double v = 0.0;
  for (int q = c.tid(); q < A.W.nv; q += c.nthr()) v = nanMax(v, fabs(x[q]));
  for (int o = 16; o > 0; o >>= 1) v = nanMax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) c.part[c.tid() >> 5] = v;
  double r, unused;
  c.reduce(c.nthr() >> 5, false, true, r, unused);
  return r;
  }
}

// One colour of levelGSRB, face ghosts read from their sources.
template <class C>
__device__ void bGsrb(C& c, const BottomArgs& A, double* phi, const double* rhs, int color) {
  const BottomWork& W = A.W;
  const int* list = W.col[color];
  const double dxinv = A.sc.dxinv;
  for (int idx = c.tid(); idx < W.ncol[color]; idx += c.nthr()) {
    const int q = list[idx];
    const int* n = W.nbv + 6 * q;
    const double pxp = gval(phi, n[0]), pxm = gval(phi, n[1]), pyp = gval(phi, n[2]), pym = gval(phi, n[3]),
                 pzp = gval(phi, n[4]), pzm = gval(phi, n[5]);
    const double pc = phi[q];
    if (A.vc) {
      const int* o = W.nb + 6 * q;
      const double div = W.b[0][o[0]] * (pxp - pc) - W.b[0][q] * (pc - pxm) + W.b[1][o[2]] * (pyp - pc) -
                         W.b[1][q] * (pc - pym) + W.b[2][o[4]] * (pzp - pc) - W.b[2][q] * (pc - pzm);
      const double lofphi = A.sc.alpha * W.a[q] * pc - A.sc.beta * div * dxinv;
      phi[q] = pc - W.lam[q] * (lofphi - rhs[q]);
    } else if (A.sc.laplacian) {
      const double lphi = (pxp + pxm + pyp + pym + pzp + pzm) * dxinv;
      phi[q] = A.sc.lambda * (rhs[q] - lphi);
    } else {
      const double lphi = (pxp + pxm + pyp + pym + pzp + pzm - 2.0 * 3 * pc) * dxinv;
      const double helmop = A.sc.alpha * pc + A.sc.beta * lphi;
      phi[q] = pc + A.sc.lambda * (helmop - rhs[q]);
    }
  }
  c.sync();
}

template <class C>
__device__ void bRelax(C& c, const BottomArgs& A, double* phi, const double* rhs, int nit) {
  if constexpr (C::kCluster) {
    c.sweeps(phi, rhs, nit);
  } else {
    for (int it = 0; it < nit; ++it)
      for (int color = 0; color <= 1; ++color) bGsrb(c, A, phi, rhs, color);
  }
}

// residual (mode 0) or applyOp (mode 1) into every valid slot of r.
template <class C>
__device__ void bOp(C& c, const BottomArgs& A, double* r, const double* phi, const double* rhs, int mode) {
  if constexpr (C::kCluster) {
    c.op(r, phi, rhs, mode);
    return;
  } else {
  const double dxinv = A.sc.dxinv;
  const BottomWork& W = A.W;
  bCells(c, W.nv, [&](int q) {
    const int* n = W.nbv + 6 * q;
    const double pxp = gval(phi, n[0]), pxm = gval(phi, n[1]), pyp = gval(phi, n[2]), pym = gval(phi, n[3]),
                 pzp = gval(phi, n[4]), pzm = gval(phi, n[5]);
    const double pc = phi[q];
    if (A.vc) {
      const int* o = W.nb + 6 * q;
      const double div = W.b[0][o[0]] * (pxp - pc) - W.b[0][q] * (pc - pxm) + W.b[1][o[2]] * (pyp - pc) -
                         W.b[1][q] * (pc - pym) + W.b[2][o[4]] * (pzp - pc) - W.b[2][q] * (pc - pzm);
      const double lofphi = A.sc.alpha * W.a[q] * pc - A.sc.beta * div * dxinv;
      r[q] = mode == 0 ? rhs[q] - lofphi : lofphi;
    } else {
      const double lap = (pxp + pxm + pyp + pym + pzp + pzm - 6.0 * pc) * dxinv;
      r[q] = mode == 0 ? -(A.sc.alpha * pc) - A.sc.beta * lap + rhs[q] : A.sc.alpha * pc + A.sc.beta * lap;
    }
  });
  }
}

template <class C>
__device__ void bPrecond(C& c, const BottomArgs& A, double* out, const double* in) {
  bCellsOf(c, A.W.nv, out, [&](int q) { out[q] = A.vc ? in[q] * A.W.lam[q] : in[q] * A.mult; });
  bRelax(c, A, out, in, 2);
}

// RelaxSolver<T>::solve (AMRElliptic/RelaxSolver.H:128-186): repeated
// preconditioner corrections e = preCond(r), phi += e, until the residual
// norm falls below eps times the initial one, imax iterations or a hang.
template <class C>
__device__ void bRelaxSolve(C& c, const BottomArgs& A) {
  const BottomWork& W = A.W;
  bOp(c, A, A.r, A.phi, A.rhs, 0);
  double norm = bNormType(c, A, A.r);
  double minNorm = norm;
  int iter = 0;
  if (norm > 0.) {
    const double initialNorm = norm;
    while (iter < A.cfg.imax) {
      bPrecond(c, A, A.e, A.r);
      bCellsOf(c, W.nv, A.phi, [&](int q) { A.phi[q] = A.phi[q] + A.e[q] * 1.0; });
      bOp(c, A, A.r, A.phi, A.rhs, 0);
      norm = bNormType(c, A, A.r);
      iter++;
      if (norm < A.cfg.eps * initialNorm) break;
      if (norm < minNorm)
        minNorm = norm;
      else if (norm * A.cfg.hang > minNorm)
        break;
    }
  }
  if (c.lead()) W.status[0] = 0, W.status[1] = iter;
}

// On the grid, boxes of at most this many cells have their element-wise
// updates and their partial sums done by one thread each, with no barrier in
// between (in one block a barrier costs less than the serialised updates).
constexpr int kBoxWiseCells = 64;

// r += v * sv and e += w * sw on every valid slot, then the norm of r (and,
// with rtr, the reference-ordered rt.r, folded beside it): the two sums a
// BiCGStab half step ends with.
template <class C>
__device__ double bUpdateNorm(C& c, const BottomArgs& A, const double* v, double sv, const double* w, double sw,
                              double* rtr) {
  const BottomWork& W = A.W;
  if constexpr (C::kCluster) {
    // the sums read the rank's own cells only, so its threads' barrier is enough
    for (int q = c.tid(); q < W.nv; q += c.nthr()) {
      A.r[q] = A.r[q] + v[q] * sv;
      A.e[q] = A.e[q] + w[q] * sw;
    }
    __syncthreads();
    if (A.cfg.normType == 2) {
      double n2, d = 0.0;
      c.norm2(A, A.r, rtr ? A.rt : nullptr, A.r, n2, d);
      if (rtr) *rtr = d;
      return sqrt(n2);
    }
    const double n = bNormType(c, A, A.r);
    if (rtr) *rtr = bDot(c, A, A.rt, A.r, false);
    return n;
  } else {
    if (C::kGrid && A.cfg.normType == 2 && W.maxBoxCells <= kBoxWiseCells) {
      for (int b = c.tid(); b < W.nbox; b += c.nthr()) {
        for (int q = W.boxStart[b]; q < W.boxStart[b + 1]; ++q) {
          A.r[q] = A.r[q] + v[q] * sv;
          A.e[q] = A.e[q] + w[q] * sw;
        }
        c.part[b] = boxPartial(A, b, A.r, A.r, true);
        if (rtr) c.part2[b] = boxPartial(A, b, A.rt, A.r, false);
      }
      double n2, d = 0.0;
      c.reduce(W.nbox, rtr != nullptr, false, n2, d);
      if (rtr) *rtr = d;
      return sqrt(n2);
    }
    bCells(c, W.nv, [&](int q) {
      A.r[q] = A.r[q] + v[q] * sv;
      A.e[q] = A.e[q] + w[q] * sw;
    });
    const double n = bNormType(c, A, A.r);
    if (rtr) *rtr = bDot(c, A, A.rt, A.r, false);
    return n;
  }
}

// p from r (init) or p = (p beta + v (-beta omega)) + r, then the
// preconditioner pt = preCond(p): the two share their first pass.
template <class C>
__device__ void bDirection(C& c, const BottomArgs& A, bool init, double b1, double bo) {
  const BottomWork& W = A.W;
  bCellsOf(c, W.nv, A.pt, [&](int q) {
    double x;
    if (init) {
      x = A.r[q];
    } else {
      x = A.p[q] * b1;
      x = x + A.v[q] * bo;
      x = x + A.r[q] * 1.0;
    }
    A.p[q] = x;
    A.pt[q] = A.vc ? x * W.lam[q] : x * A.mult;
  });
  bRelax(c, A, A.pt, A.p, 2);
}

template <class C>
__device__ void bBicgstab(C& c, const BottomArgs& A) {
  const BottomWork& W = A.W;
  const int nv = W.nv;
  auto zeroV = [&](double* x) { bCells(c, nv, [&](int q) { x[q] = 0.0; }); };
  auto incrPhi = [&]() { bCellsOf(c, nv, A.phi, [&](int q) { A.phi[q] = A.phi[q] + A.e[q] * 1.0; }); };
  // rt = r, e = 0 in one pass
  auto restartVectors = [&]() {
    bCells(c, nv, [&](int q) {
      A.rt[q] = A.r[q];
      A.e[q] = 0.0;
    });
  };
  bOp(c, A, A.r, A.phi, A.rhs, 0);
  restartVectors();
  int iter = 0, recount = 0, restarts = 0, status = 0;
  double rho[4] = {0, 0, 0, 0};
  double norm[2];
  norm[0] = bNormType(c, A, A.r);
  double initial_norm = norm[0];
  const double initial_residual = norm[0];
  norm[1] = norm[0];
  double alpha[2] = {0, 0}, beta[2] = {0, 0}, omega[2] = {0, 0};
  bool init = true;
  // rt.r of the current r when the last half step folded it beside its norm
  bool haveRho = false;
  double rhoNext = 0.0;
  const double metric = *A.metric;
  if (metric > 0) initial_norm = metric;
  while ((iter < A.imax && norm[0] > A.eps * norm[1]) && (norm[1] > 0)) {
    iter++;
    norm[1] = norm[0];
    alpha[1] = alpha[0];
    beta[1] = beta[0];
    omega[1] = omega[0];
    rho[3] = rho[2];
    rho[2] = rho[1];
    rho[1] = haveRho ? rhoNext : bDot(c, A, A.rt, A.r, false);
    haveRho = false;
    if (rho[1] == 0.0) {
      incrPhi();
      if (c.lead()) W.status[0] = 2, W.status[1] = iter;
      return;
    }
    double b1 = 0.0, bo = 0.0;
    if (!init) {
      beta[1] = (rho[1] / rho[2]) * (alpha[1] / omega[1]);
      b1 = beta[1];
      bo = -beta[1] * omega[1];
    }
    bDirection(c, A, init, b1, bo);
    init = false;
    bOp(c, A, A.v, A.pt, nullptr, 1);
    double m = bDot(c, A, A.rt, A.v, false);
    alpha[0] = rho[1] / m;
    if (fabs(m) > A.small * fabs(rho[1])) {
      const double a0 = alpha[0];
      norm[0] = bUpdateNorm(c, A, A.v, -a0, A.pt, a0, nullptr);
    } else {
      zeroV(A.r);
      norm[0] = 0.0;
    }
    if (norm[0] > A.eps * initial_norm && norm[0] > A.reps * initial_residual) {
      bPrecond(c, A, A.st, A.r);
      bOp(c, A, A.t, A.st, nullptr, 1);
      double tr, tt;
      bDot2(c, A, A.t, A.r, A.t, A.t, tr, tt);
      omega[0] = tr / tt;
      const double w0 = omega[0];
      norm[0] = bUpdateNorm(c, A, A.t, -w0, A.st, w0, &rhoNext);
      haveRho = true;
    }
    if (norm[0] <= A.eps * initial_norm || norm[0] <= A.reps * initial_residual) {
      status = 1;
      break;
    }
    if (omega[0] == 0.0 || norm[0] > (1 - A.hang) * norm[1]) {
      if (recount == 0) {
        recount = 1;
      } else {
        recount = 0;
        incrPhi();
        if (restarts == A.numRestarts) {
          if (c.lead()) W.status[0] = 3, W.status[1] = iter;
          return;
        }
        bOp(c, A, A.r, A.phi, A.rhs, 0);
        norm[0] = bNormType(c, A, A.r);
        rho[1] = 0.0;
        rho[2] = 0.0;
        rho[3] = 0.0;
        alpha[0] = 0;
        beta[0] = 0;
        omega[0] = 0;
        restartVectors();
        haveRho = false;
        restarts++;
        init = true;
      }
    }
  }
  incrPhi();
  if (c.lead()) W.status[0] = status, W.status[1] = iter;
}

template <class C>
__device__ void bottomRun(C& c, BottomArgs& A) {
  const BottomWork& W = A.W;
  A.r = W.v[0];
  A.rt = W.v[1];
  A.e = W.v[2];
  A.p = W.v[3];
  A.pt = W.v[4];
  A.st = W.v[5];
  A.t = W.v[6];
  A.v = W.v[7];
  A.phi = W.v[8];
  A.rhs = W.v[9];
  bCells(c, W.nv, [&](int q) {
    A.phi[q] = A.phiFab[W.fab[q]];
    A.rhs[q] = A.rhsFab[W.fab[q]];
  });
  if (A.cfg.kind == 1)
    bRelaxSolve(c, A);
  else
    bBicgstab(c, A);
  c.sync();
  for (int q = c.tid(); q < W.nv; q += c.nthr()) A.phiFab[W.fab[q]] = A.phi[q];
}

}  // namespace cmg

#endif
