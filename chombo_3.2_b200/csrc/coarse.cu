// The coarse part of the multigrid cycle in one cluster launch (coarse.H).
#include "coarse.H"

#include <algorithm>
#include <cstdio>
#include <functional>
#include <stdexcept>

#include "bottomdev.H"
#include "hostpool.H"

namespace cmg {

namespace {

constexpr int kCoarseThreads = 256;
// Depths of more cells than this, but for the bottom one, run as launches over
// the whole device: a 32^3 pass takes 2400 cycles here, as a launch 2 us.  As
// launches against here, ms: Poisson solves with a 32^3 level 0 0.77, 0.82
// (boxes of 16) and 0.76, 0.89 (one box), 36^3 2.46, 2.71, 48^3 0.93, 1.51; 64^3
// 1.06, 1.11; a forest of 12 two-level 32^3 mixed 3.22, 3.59.  Below 32^3 by the
// boxes: alike ones, which a launch reads across, 24^3 0.85, 0.87 as level 0 and
// 2.02, 1.94 as a depth of two-level 48^3; others 24^3 0.85, 0.77 as level 0 and
// 1.13, 1.03 as a depth of 48^3, 28^3 2.56, 2.52.  16^3 0.56, 0.50.  (The tables
// of a 32^3 depth took 1 ms of every new hierarchy's preparation besides.)
constexpr int64_t kCoarseMaxCells = 25000;
// With variable coefficients, eight more values a cell come from the second-level
// cache in every pass (7600 cycles for 32^3): 32^3 in alike boxes 1.27, 1.77, 24^3
// 1.53, 1.71 as level 0 and 3.28, 3.42 as a depth, in others 1.51, 1.51 and 2.05,
// 2.05; 28^3 4.91, 5.11; 20^3 3.93, 3.82.  Two-level 64^3, with 16^3 cells and
// fewer here against 32^3 and fewer: 4.15, 4.61.
constexpr int64_t kCoarseMaxCellsVC = 12000;
// The bottom depth is taken up to this size, for its solve.
constexpr int64_t kCoarseMaxBottomCells = 40000;
// Depths of at most this many cells stay on rank 0: an 8^3 pass takes 520
// cycles there, less than the cluster barrier and halo stores alone; a 16^3 one
// (2048 cells a pass) is no faster in one block than over 16.
constexpr int kSoloCells = 1536;
// Up to this many boxes every rank folds all box sums itself, which spares the
// second barrier; beyond, the folds dominate (8.2 cycles per dependent add,
// 8.7 measured) and one copy of the sums leaves room for the vectors.
constexpr int kAllRanksBoxes = 512;

inline void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    char buf[256];
    std::snprintf(buf, sizeof(buf), "cmg: %s: %s", what, cudaGetErrorString(e));
    throw std::runtime_error(buf);
  }
}

template <class T>
struct Args {
  const CoarseHier* hier;
  T* corr;
  const T* res;
  int ranks, pre, post, bottom, numMG, oneCell, fromZero;
  BottomConfig cfg;
  double eps, mult;
  const double *metrics, *epsPer;
  // An argument and not in the tables: new coefficients then change no device
  // memory (setting alpha and beta 14 -> 8 us).
  Scal sc[kCoarseMaxDepths];
};

__device__ __forceinline__ unsigned smemAddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned mapRank(unsigned a, int r) {
  unsigned o;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(r));
  return o;
}
__device__ __forceinline__ double ldRemote(unsigned a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ldRemote(unsigned a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void stRemote(unsigned a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void stRemote(unsigned a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void clusterSync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The block's fields.
extern __shared__ __align__(16) char coarseSmem[];

// Cell v (rank << shift | element) of a field every rank holds at f.
template <class T>
__device__ __forceinline__ T cellOn(const T* f, int v, int rank) {
  const int r = v >> kCoarseRankShift, i = v & ((1 << kCoarseRankShift) - 1);
  if (r == rank) return f[i];
  return ldRemote(mapRank(smemAddr(f + i), r), T(0));
}

// An entry's neighbours (CoarseDepth::nb): element i of f, or 0 - it where the
// high bit marks a Dirichlet ghost.
template <class T>
__device__ __forceinline__ T element(const T* f, unsigned n) {
  const T x = f[n & 0x7fff];
  return n & 0x8000 ? T(0) - x : x;
}
template <class T>
__device__ __forceinline__ void neighbours(const T* f, const uint4& w, T* v) {
  v[0] = element(f, w.x & 0xffff);
  v[1] = element(f, w.x >> 16);
  v[2] = element(f, w.y & 0xffff);
  v[3] = element(f, w.y >> 16);
  v[4] = element(f, w.z & 0xffff);
  v[5] = element(f, w.z >> 16);
}

// This rank's part of a depth's tables.  Entries c0 .. c1 - 1 are its colour-0
// cells, c1 .. c2 - 1 its colour-1 cells; p0, p1, p2 the same for the cells it
// sends (all equal where one rank holds the depth).
struct Range {
  const uint4* nb;
  const unsigned* push;
  int n, c0, c1, c2, p0, p1, p2;
};

// Sends the cells of push entries [p0, p1) to the halos that hold them.
template <class T>
__device__ __forceinline__ void pushCells(const unsigned* push, int p0, int p1, T* f) {
  const unsigned base = smemAddr(f);
  for (int p = p0 + threadIdx.x; p < p1; p += kCoarseThreads) {
    const unsigned v = __ldg(push + p);
    stRemote(mapRank(base + (v & 0x7fff) * (unsigned)sizeof(T), v >> 15 & 15), f[v >> 19]);
  }
}

template <class T, int VC>
__device__ __forceinline__ void loadCoef(const T* coef, int n, int e, T& av, T& lv, T* f) {
  av = lv = T(0);
  if (VC) {
    av = __ldg(coef + e);
    lv = __ldg(coef + n + e);
#pragma unroll
    for (int d = 0; d < 6; ++d) f[d] = __ldg(coef + (2 + d) * n + e);
  }
}

// The update of one entry of a colour pass, from its loaded tables.
template <class T, int VC>
__device__ __forceinline__ void updateCell(const uint4& w, const Scal& sc, T* phi, T rh, T av, T lv, const T* f) {
  T v[6];
  const T pc = phi[w.w];
  neighbours(phi, w, v);
  phi[w.w] = gsrbValue<T, VC>(sc, pc, rh, v, av, lv, f);
}

__device__ __forceinline__ void rankSync(int nc) {
  if (nc > 1)
    clusterSync();
  else
    __syncthreads();
}

// What the bottom solve's loops share (one copy per block, in shared memory;
// the loops below are calls, not inlined copies, to stay in the instruction
// cache).
struct BottomShared {
  Range R;
  const double* coef;
  Scal sc;
  int rank, nc;  // nc: ranks of the solve (1 when one rank holds it all)
  int box0, nb, nbox, maxNx, allRanks;
  uint64_t mNx;  // divMagic of maxNx
  const int4* box;
  double* part;  // allRanks: 2 buffers x 2 sums x nbox; else nbox
  double* pen;
};

// Sweeps of one depth, colour 0 first; after every pass the cells other ranks
// read are sent and the ranks meet.  Up to E entries of a colour per thread
// keep their tables and right-hand sides (and for E = 1 their coefficients) in
// registers over the sweeps; E = 0 reads them in every pass.
template <class T, int VC, int E>
__device__ __noinline__ void sweepsOf(const Range& R0, const T* coef, const Scal& sc0, T* phi, const T* rhs,
                                      int sweeps, int nc) {
  const Range R = R0;
  const Scal sc = sc0;
  constexpr bool kCoef = VC && E == 1;
  // The first kHeld cells a thread sends in either colour's passes, kept over
  // the sweeps too.
  constexpr int kHeld = E == 0 ? 1 : 2;
  unsigned sent[2][kHeld];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int u = 0; u < kHeld; ++u) {
      const int p = (c ? R.p1 : R.p0) + threadIdx.x + u * kCoarseThreads;
      sent[c][u] = p < (c ? R.p2 : R.p1) ? __ldg(R.push + p) : 0xffffffffu;
    }
  const unsigned base = smemAddr(phi);
  auto meet = [&](int c) {
    __syncthreads();
    if (nc > 1) {
#pragma unroll
      for (int u = 0; u < kHeld; ++u) {
        const unsigned v = sent[c][u];
        if (v != 0xffffffffu)
          stRemote(mapRank(base + (v & 0x7fff) * (unsigned)sizeof(T), v >> 15 & 15), phi[v >> 19]);
      }
      pushCells(R.push, (c ? R.p1 : R.p0) + kHeld * kCoarseThreads, c ? R.p2 : R.p1, phi);
      clusterSync();
    }
  };
  if constexpr (E > 0) {
    uint4 w[2][E];
    T rh[2][E], av[2][kCoef ? E : 1], lv[2][kCoef ? E : 1], f[2][kCoef ? E : 1][6];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int u = 0; u < E; ++u) {
        const int e = (c ? R.c1 : R.c0) + threadIdx.x + u * kCoarseThreads;
        w[c][u].w = 0xffffffffu;
        if (e >= (c ? R.c2 : R.c1)) continue;
        w[c][u] = __ldg(R.nb + e);
        rh[c][u] = rhs[w[c][u].w];
        if (kCoef) loadCoef<T, VC>(coef, R.n, e, av[c][u], lv[c][u], f[c][u]);
      }
    for (int it = 0; it < sweeps; ++it)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int u = 0; u < E; ++u) {
          if (w[c][u].w == 0xffffffffu) continue;
          if (VC && !kCoef) {
            T a1, l1, f1[6];
            loadCoef<T, VC>(coef, R.n, (c ? R.c1 : R.c0) + threadIdx.x + u * kCoarseThreads, a1, l1, f1);
            updateCell<T, VC>(w[c][u], sc, phi, rh[c][u], a1, l1, f1);
          } else {
            updateCell<T, VC>(w[c][u], sc, phi, rh[c][u], av[c][kCoef ? u : 0], lv[c][kCoef ? u : 0],
                              f[c][kCoef ? u : 0]);
          }
        }
        meet(c);
      }
  } else {
    for (int it = 0; it < 2 * sweeps; ++it) {
      const int e1 = it & 1 ? R.c2 : R.c1;
      for (int e = (it & 1 ? R.c1 : R.c0) + threadIdx.x; e < e1; e += kCoarseThreads) {
        const uint4 w = __ldg(R.nb + e);
        T av, lv, f[6];
        loadCoef<T, VC>(coef, R.n, e, av, lv, f);
        updateCell<T, VC>(w, sc, phi, rhs[w.w], av, lv, f);
      }
      if (it & 1)
        meet(1);
      else
        meet(0);
    }
  }
}
template <class T, int VC>
__device__ __forceinline__ void sweepsAll(const Range& R, const T* coef, const Scal& sc, T* phi, const T* rhs, int sweeps,
                                       int nc) {
  const int most = max(R.c1 - R.c0, R.c2 - R.c1);
  if (most <= kCoarseThreads)
    sweepsOf<T, VC, 1>(R, coef, sc, phi, rhs, sweeps, nc);
  else if (most <= 2 * kCoarseThreads)
    sweepsOf<T, VC, 2>(R, coef, sc, phi, rhs, sweeps, nc);
  else if (most <= 4 * kCoarseThreads)
    sweepsOf<T, VC, 4>(R, coef, sc, phi, rhs, sweeps, nc);
  else
    sweepsOf<T, VC, 0>(R, coef, sc, phi, rhs, sweeps, nc);
}

template <int VC>
__device__ __noinline__ void bottomSweeps(const BottomShared& S, double* phi, const double* rhs, int n) {
  sweepsAll<double, VC>(S.R, S.coef, S.sc, phi, rhs, n, S.nc);
}

template <int VC>
__device__ __noinline__ void bottomOp(const BottomShared& S, double* r, const double* phi, const double* rhs, int mode) {
  const Range R = S.R;
  const Scal sc = S.sc;
  for (int e = R.c0 + threadIdx.x; e < R.c2; e += kCoarseThreads) {
    const uint4 w = __ldg(R.nb + e);
    double av, lv, f[6], v[6];
    loadCoef<double, VC>(S.coef, R.n, e, av, lv, f);
    const int q = w.w;
    const double pc = phi[q];
    neighbours(phi, w, v);
    r[q] = mode == 0 ? opValue<double, VC, 0>(sc, pc, rhs[q], v, av, f) : opValue<double, VC, 1>(sc, pc, 0.0, v, av, f);
  }
  // the result is read on its own rank only
  __syncthreads();
}

// Sends a vector's cells, just written by this rank's threads, to the halos
// that hold them.
template <class T>
__device__ __noinline__ void publishCells(const Range& R, T* f, int nc) {
  __syncthreads();
  if (nc == 1) return;
  pushCells(R.push, R.p0, R.p2, f);
  clusterSync();
}

// term(0) + term(1) + ... in order from zero, read eight ahead of the chain of
// adds.
template <class F>
__device__ __forceinline__ double chainSum(int n, F term) {
  double s = 0.0, cur[8], nxt[8];
  const int full = n & ~7;
  if (full) {
#pragma unroll
    for (int u = 0; u < 8; ++u) cur[u] = term(u);
    for (int b = 8; b < full; b += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) nxt[u] = term(b + u);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += cur[u];
#pragma unroll
      for (int u = 0; u < 8; ++u) cur[u] = nxt[u];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) s += cur[u];
  }
  for (int b = full; b < n; ++b) s += term(b);
  return s;
}

// The sum of box b (of this rank) goes to the ranks that fold sum w.
__device__ __forceinline__ void pushSum(const BottomShared& S, int buf, int w, int b, double s) {
  if (S.allRanks) {
    double* p = S.part + (2 * buf + w) * S.nbox + S.box0 + b;
    if (S.nc == 1) {
      *p = s;
    } else {
      const unsigned a = smemAddr(p);
      for (int r = 0; r < S.nc; ++r) stRemote(mapRank(a, r), s);
    }
  } else {
    stRemote(mapRank(smemAddr(S.part + S.box0 + b), w), s);
  }
}

__device__ __forceinline__ double boxDot(const BottomShared& S, int b, const double* x, const double* y) {
  const int4 g = __ldg(S.box + S.box0 + b);
  const int n = g.y * g.z * g.w;
  const double *px = x + g.x, *py = y + g.x;
  return chainSum(n, [&](int q) { return px[q] * py[q]; });
}

// x1.y1 (and x2.y2 when x2): every box's products added x fastest.
__device__ __noinline__ void pushDots(const BottomShared& S, int buf, const double* x1, const double* y1,
                                      const double* x2, const double* y2) {
  const int nb = S.nb, tasks = x2 ? 2 * nb : nb;
  for (int t = threadIdx.x; t < tasks; t += kCoarseThreads) {
    const bool second = t >= nb;
    const int b = second ? t - nb : t;
    pushSum(S, buf, second, b, boxDot(S, b, second ? x2 : x1, second ? y2 : y1));
  }
}

// sumPow(2) of x (per box: one running sum per x over k and j, those added in
// x order, so each x is a thread's), and dx.dy beside it when dx.
__device__ __noinline__ void pushNorm2(const BottomShared& S, int buf, const double* x, const double* dx,
                                       const double* dy) {
  double* pen = S.pen;
  const int nb = S.nb, np = nb * S.maxNx, npr = (np + 31) & ~31, tasks = npr + (dx ? nb : 0);
  for (int t = threadIdx.x; t < tasks; t += kCoarseThreads) {
    if (t < np) {
      const int b = fastDiv(t, S.maxNx, S.mNx), i = t - b * S.maxNx;
      const int4 g = __ldg(S.box + S.box0 + b);
      if (i < g.y) {
        const int n = g.z * g.w;
        const double* p = x + g.x + i;
        // from +0, which a first square leaves as it is
        pen[t] = chainSum(n, [&](int q) { return p[q * g.y] * p[q * g.y]; });
      }
    } else if (t >= npr) {
      pushSum(S, buf, 1, t - npr, boxDot(S, t - npr, dx, dy));
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nb; b += kCoarseThreads) {
    const int nx = __ldg(S.box + S.box0 + b).y;
    const double* p = pen + b * S.maxNx;
    double s = p[0];
    for (int i = 1; i < nx; ++i) s = s + p[i];
    pushSum(S, buf, 0, b, s);
  }
}

// The pushed box sums added in box order.
__device__ __noinline__ double foldSums(const double* p, int n) {
  return chainSum(n, [&](int b) { return p[b]; });
}

// The largest |x| over every rank (a NaN stays).  red: 2 buffers of 16 ranks,
// then this rank's warps.
__device__ __noinline__ double maxOver(int n, const double* x, double* red, int buf, int rank, int nc) {
  double v = 0.0;
  for (int q = threadIdx.x; q < n; q += kCoarseThreads) v = nanMax(v, fabs(x[q]));
  for (int o = 16; o > 0; o >>= 1) v = nanMax(v, __shfl_xor_sync(0xffffffffu, v, o));
  double* warps = red + 32;
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 0; w < kCoarseThreads / 32; ++w) v = nanMax(v, warps[w]);
    if (nc == 1)
      red[16 * buf] = v;
    else
      for (int r = 0; r < nc; ++r) stRemote(mapRank(smemAddr(red + 16 * buf + rank), r), v);
  }
  rankSync(nc);
  v = 0.0;
  for (int r = 0; r < nc; ++r) v = nanMax(v, red[16 * buf + r]);
  return v;
}

// The bottom solve's context (bottomdev.H): this rank's part of the vectors in
// shared memory, box sums pushed to the ranks that fold them.
template <int VC>
struct ClusterCtx {
  static constexpr bool kCluster = true;
  const BottomShared* S;
  double *scal, *red;
  int rank, nc, k, buf;
  __device__ int tid() const { return threadIdx.x; }
  __device__ int nthr() const { return kCoarseThreads; }
  __device__ bool lead() const { return rank == 0 && threadIdx.x == 0; }
  __device__ void sync() const { rankSync(nc); }
  __device__ void sweeps(double* phi, const double* rhs, int n) { bottomSweeps<VC>(*S, phi, rhs, n); }
  __device__ void publish(double* f) { publishCells(S->R, f, nc); }
  __device__ void op(double* r, const double* phi, const double* rhs, int mode) { bottomOp<VC>(*S, r, phi, rhs, mode); }
  // Folds the pushed box sums in box order; every thread gets the results.
  // The two buffers of the all-ranks form keep a rank's next sums out of the
  // way of one still folding (a rank pushes into a buffer again only after a
  // barrier every rank passed with that fold done); the other form ends with a
  // barrier of its own.
  __device__ __forceinline__ void finish(bool two, double& r1, double& r2) {
    sync();
    const int s = k;
    k = (k + 2) & 7;
    if (S->allRanks) {
      const double* p = S->part + 2 * buf * S->nbox;
      if (threadIdx.x == 0) scal[s] = foldSums(p, S->nbox);
      if (two && threadIdx.x == 32) scal[s + 1] = foldSums(p + S->nbox, S->nbox);
      buf ^= 1;
      __syncthreads();
    } else {
      if (threadIdx.x == 0 && (rank == 0 || (two && rank == 1))) {
        const double v = foldSums(S->part, S->nbox);
        for (int r = 0; r < nc; ++r) stRemote(mapRank(smemAddr(scal + s + rank), r), v);
      }
      sync();
    }
    r1 = scal[s];
    if (two) r2 = scal[s + 1];
  }
  __device__ void dots(const BottomArgs&, const double* x1, const double* y1, const double* x2, const double* y2,
                       double& r1, double& r2) {
    pushDots(*S, buf, x1, y1, x2, y2);
    finish(x2 != nullptr, r1, r2);
  }
  __device__ void norm2(const BottomArgs&, const double* x, const double* dx, const double* dy, double& r1,
                        double& r2) {
    pushNorm2(*S, buf, x, dx, dy);
    finish(dx != nullptr, r1, r2);
  }
  __device__ double normMax(const BottomArgs& A, const double* x) {
    const double v = maxOver(A.W.nv, x, red, buf, rank, nc);
    buf ^= 1;
    return v;
  }
};

// What a block keeps in shared memory beside the fields (one copy: per-thread
// copies would not fit the first-level cache).
struct Block {
  CoarseHier H;
  Scal sc[kCoarseMaxDepths];
  BottomShared S;
  BottomArgs B;
  double scal[8], red[32 + kCoarseThreads / 32];
  int rank, nc;
};

// The pieces of the cycle, one call each (T: the cycle's precision).
template <class T, int VC>
struct Cycle {
  static constexpr int F = sizeof(T) == 8 ? 0 : 1;
  Block& K;
  const CoarseHier& H;
  int rank, nc;
  __device__ Cycle(Block& k) : K(k), H(k.H), rank(k.rank), nc(k.nc) {}
  __device__ T* phi(int d) const { return reinterpret_cast<T*>(coarseSmem + H.d[d].phi[F]); }
  __device__ T* rhs(int d) const { return reinterpret_cast<T*>(coarseSmem + H.d[d].rhs[F]); }
  __device__ const T* coef(int d) const {
    return F == 0 ? reinterpret_cast<const T*>(H.d[d].coefD) : reinterpret_cast<const T*>(H.d[d].coefF);
  }
  __device__ Range range(int d) const {
    const CoarseDepth& D = H.d[d];
    const int *c = D.colStart + 2 * rank, *p = D.pushStart + 2 * rank;
    return Range{D.nb, D.push, D.n, __ldg(c), __ldg(c + 1), __ldg(c + 2), __ldg(p), __ldg(p + 1), __ldg(p + 2)};
  }
  // Barrier of a depth's ranks: the cluster, or rank 0 alone.
  __device__ void sync(bool solo) const { rankSync(solo ? 1 : nc); }
};

template <class T, int VC>
__device__ __noinline__ void relaxDepth(Block& K, int d, int sweeps) {
  const Cycle<T, VC> Y(K);
  sweepsAll<T, VC>(Y.range(d), Y.coef(d), K.sc[d], Y.phi(d), Y.rhs(d), sweeps, Y.H.d[d].solo ? 1 : Y.nc);
}

// RESTRICTRES(VC3D): an eighth of the residual of every cell of depth d, then
// the sum over each coarse cell's eight, k, j, i order, from zero; the coarse
// correction starts at zero.
template <class T, int VC>
__device__ __noinline__ void restrictDepth(Block& K, int d) {
  const Cycle<T, VC> Y(K);
  constexpr int F = Cycle<T, VC>::F;
  const CoarseDepth& D = Y.H.d[d];
  T* tmp = reinterpret_cast<T*>(coarseSmem + Y.H.tmp[F]);
  {
    const Range R = Y.range(d);
    const T* coef = Y.coef(d);
    const Scal sc = K.sc[d];
    const T dxinv = T(sc.dxinv);
    const T* phi = Y.phi(d);
    const T* rhs = Y.rhs(d);
    for (int e = R.c0 + threadIdx.x; e < R.c2; e += kCoarseThreads) {
      const uint4 w = __ldg(R.nb + e);
      const int q = w.w;
      T av, lv, f[6], v[6];
      loadCoef<T, VC>(coef, R.n, e, av, lv, f);
      const T pc = phi[q];
      neighbours(phi, w, v);
      T lofphi;
      if (VC) {
        const T div = f[0] * (v[0] - pc) - f[1] * (pc - v[1]) + f[2] * (v[2] - pc) - f[3] * (pc - v[3]) +
                      f[4] * (v[4] - pc) - f[5] * (pc - v[5]);
        lofphi = T(sc.alpha) * av * pc - T(sc.beta) * div * dxinv;
      } else {
        lofphi = T(sc.alpha) * pc + T(sc.beta) * ((v[0] + v[1] + v[2] + v[3] + v[4] + v[5]) - pc * T(2) * T(3)) * dxinv;
      }
      tmp[q] = (rhs[q] - lofphi) / T(8);
    }
  }
  Y.sync(D.solo);
  const CoarseDepth& C = Y.H.d[d + 1];
  const Range R = Y.range(d + 1);
  T* phi = Y.phi(d + 1);
  T* rhs = Y.rhs(d + 1);
  const int rank = Y.rank;
  for (int e = R.c0 + threadIdx.x; e < R.c2; e += kCoarseThreads) {
    const int4 a = __ldg(C.child + 2 * e), b = __ldg(C.child + 2 * e + 1);
    const int q = __ldg(&R.nb[e].w), c[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    T t[8];
    int other = 0;
#pragma unroll
    for (int n = 0; n < 8; ++n) other |= (c[n] >> kCoarseRankShift) ^ rank;
    if (other == 0) {
#pragma unroll
      for (int n = 0; n < 8; ++n) t[n] = tmp[c[n] & ((1 << kCoarseRankShift) - 1)];
    } else {
#pragma unroll
      for (int n = 0; n < 8; ++n) t[n] = cellOn(tmp, c[n], rank);
    }
    T acc = T(0);
#pragma unroll
    for (int n = 0; n < 8; ++n) acc = acc + t[n];
    rhs[q] = acc;
  }
  if (R.c2 > R.c0)  // the correction, halo included
    for (int q = threadIdx.x; q < C.nField; q += kCoarseThreads) phi[q] = T(0);
  Y.sync(D.solo);
}

// PROLONG: phi += the coarse correction above each cell.
template <class T, int VC>
__device__ __noinline__ void prolongDepth(Block& K, int d) {
  const Cycle<T, VC> Y(K);
  const CoarseDepth& D = Y.H.d[d];
  const Range R = Y.range(d);
  T* phi = Y.phi(d);
  const T* corrC = Y.phi(d + 1);
  const int rank = Y.rank;
  for (int e0 = R.c0 + threadIdx.x; e0 < R.c2; e0 += 4 * kCoarseThreads) {
    // four entries' loads before their stores
    T x[4];
    int q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u * kCoarseThreads;
      if (e >= R.c2) continue;
      q[u] = __ldg(&R.nb[e].w);
      x[u] = phi[q[u]] + cellOn(corrC, __ldg(D.par + e), rank);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (e0 + u * kCoarseThreads < R.c2) phi[q[u]] = x[u];
  }
  publishCells(R, phi, D.solo ? 1 : Y.nc);
}

template <class T, int VC>
__device__ __noinline__ void bottomDepth(Block& K, const Args<T>& A, int h) {
  const Cycle<T, VC> Y(K);
  constexpr int F = Cycle<T, VC>::F;
  const CoarseHier& H = K.H;
  const int d = H.nd - 1, rank = K.rank;
  const CoarseDepth& D = H.d[d];
  if (A.oneCell) {
    relaxDepth<T, VC>(K, d, 1);
    return;
  }
  const int nc = D.solo ? 1 : K.nc;
  BottomArgs& B = K.B;
  if (threadIdx.x == 0) {
    BottomShared& S = K.S;
    S.R = Y.range(d);
    S.coef = D.coefD;
    S.sc = K.sc[d];
    S.rank = rank;
    S.nc = nc;
    S.box0 = D.solo ? 0 : H.boxRank[rank];
    S.nb = (D.solo ? H.nbox : H.boxRank[rank + 1]) - S.box0;
    S.nbox = H.nbox;
    S.maxNx = H.maxNx;
    S.mNx = divMagic(H.maxNx, (int64_t)S.nb * H.maxNx);
    S.allRanks = H.allRanks;
    S.box = H.box;
    S.part = reinterpret_cast<double*>(coarseSmem + H.part);
    S.pen = reinterpret_cast<double*>(coarseSmem + H.pen);
    const int s0 = D.solo ? 0 : H.rankSlot[rank], s1 = D.solo ? D.n : H.rankSlot[rank + 1];
    B.W.nv = s1 - s0;
    B.W.lam = VC ? const_cast<double*>(H.lamSlot) + s0 : nullptr;
    B.W.status = H.status;
    B.sc = K.sc[d];
    B.vc = VC;
    B.cfg = A.cfg;
    B.eps = A.cfg.kind == 1 ? A.cfg.eps : A.eps;  // RelaxSolver keeps its own tolerance
    if (A.epsPer && A.cfg.kind == 0) B.eps = A.epsPer[h];
    B.reps = A.cfg.reps;
    B.hang = A.cfg.hang;
    B.small = A.cfg.small;
    B.imax = A.cfg.imax;
    B.numRestarts = A.cfg.numRestarts;
    B.mult = A.mult;
    B.metric = A.metrics + h;
    // Vectors the operator reads hold a halo: pt (with st, whose life starts
    // after pt's ends, and the relaxation's e) and phi.
    double* v = reinterpret_cast<double*>(coarseSmem + H.vec[F]);
    const int nl = H.nLoc;
    B.pt = B.st = v;
    v += D.nField;
    B.r = v;
    B.rt = v + nl;
    B.e = A.cfg.kind == 1 ? B.pt : v + 2 * nl;
    B.p = v + 3 * nl;
    B.t = v + 4 * nl;
    B.v = v + 5 * nl;
    if constexpr (F == 0) {
      B.phi = Y.phi(d);
      B.rhs = Y.rhs(d);
    } else {
      // the bottom solve is FP64 whatever the cycle's precision
      B.rhs = v + 6 * nl;
      B.phi = v + 7 * nl;
    }
  }
  relaxDepth<T, VC>(K, d, A.bottom);
  rankSync(nc);
  if constexpr (F == 1) {
    for (int q = threadIdx.x; q < B.W.nv; q += kCoarseThreads) {
      B.phi[q] = Y.phi(d)[q];
      B.rhs[q] = Y.rhs(d)[q];
    }
    publishCells(K.S.R, B.phi, nc);
  }
  ClusterCtx<VC> c;
  c.S = &K.S;
  c.scal = K.scal;
  c.red = K.red;
  c.rank = rank;
  c.nc = nc;
  c.k = 0;
  c.buf = 0;
  if (A.cfg.kind == 1)
    bRelaxSolve(c, B);
  else
    bBicgstab(c, B);
  rankSync(nc);
  if constexpr (F == 1) {
    for (int q = threadIdx.x; q < B.W.nv; q += kCoarseThreads) Y.phi(d)[q] = (T)B.phi[q];
  }
  // a second visit (numMG > 1) relaxes phi again from its halos
  publishCells(K.S.R, Y.phi(d), nc);
}

// One cluster per hierarchy: MultiGrid::cycle from the top depth to the
// bottom and back, numMG visits of each coarser depth.  Depths from dSolo on
// are rank 0's; the other ranks wait where it comes back up.  Bound by latency:
// a colour pass is a table-held set of shared-memory reads, the update's chain
// of FP64 operations (8 cycles each), the stores to the halos of other blocks
// and a cluster barrier (480 cycles), 1270 cycles on a 16^3 depth over 16
// blocks and 2400 on 32^3 (520 for 8^3 in one block, with __syncthreads), where
// a launch over the device took about 4000; a BiCGStab iteration on 64 cells
// about 20,000 cycles.  Solves, launches before and this kernel after (it then
// held 32^3 depths too, see kCoarseMaxCells): 32^3 Poisson 1.63 -> 0.80 ms, 96^3 with a 24^3 bottom 22.8 -> 5.9 ms, 64^3 2.39 ->
// 1.44 ms, three-level 32^3 heat steps 14.6 -> 12.2 ms.
template <class T, int VC>
__global__ void __launch_bounds__(kCoarseThreads, 1) k_coarse(const __grid_constant__ Args<T> A) {
  __shared__ Block K;
  const int nc = A.ranks, h = blockIdx.x / nc, rank = blockIdx.x - h * nc;
  for (int i = threadIdx.x; i < (int)(sizeof(CoarseHier) / 4); i += kCoarseThreads)
    reinterpret_cast<int*>(&K.H)[i] = reinterpret_cast<const int*>(A.hier + h)[i];
  if (threadIdx.x < kCoarseMaxDepths) K.sc[threadIdx.x] = A.sc[threadIdx.x];
  if (threadIdx.x == 0) {
    K.rank = rank;
    K.nc = nc;
  }
  // the tables are fixed; corr and res are the previous kernels' (launchNext)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __syncthreads();
  const CoarseHier& H = K.H;
  const Cycle<T, VC> Y(K);
  const Range R0 = Y.range(0);
  T* phi0 = Y.phi(0);
  for (int e = R0.c0 + threadIdx.x; e < R0.c2; e += kCoarseThreads) {
    const int q = __ldg(&R0.nb[e].w), f = __ldg(H.fab + e);
    if (!A.fromZero) phi0[q] = A.corr[f];
    Y.rhs(0)[q] = A.res[f];
  }
  // every rank's block runs before another writes into it
  Y.sync(false);
  if (A.fromZero) {
    for (int q = threadIdx.x; q < H.d[0].nField; q += kCoarseThreads) phi0[q] = T(0);
    Y.sync(false);
  } else {
    publishCells(R0, phi0, nc);
  }
  const int bottom = H.nd - 1, dSolo = H.dSolo, last = rank == 0 ? bottom : min(dSolo, bottom);
  int visits[kCoarseMaxDepths];
  int d = 0;
  bool enter = true;
  while (true) {
    if (enter) {
      if (d < last) {
        relaxDepth<T, VC>(K, d, A.pre);
        restrictDepth<T, VC>(K, d);
        visits[d] = 0;
        ++d;
        continue;
      }
      if (rank == 0 || d < dSolo) bottomDepth<T, VC>(K, A, h);
      enter = false;
    } else if (++visits[d] < A.numMG) {
      ++d;
      enter = true;
      continue;
    } else {
      prolongDepth<T, VC>(K, d);
      relaxDepth<T, VC>(K, d, A.post);
    }
    if (d == dSolo) Y.sync(false);
    if (d == 0) break;
    --d;
  }
  for (int e = R0.c0 + threadIdx.x; e < R0.c2; e += kCoarseThreads)
    A.corr[__ldg(H.fab + e)] = phi0[__ldg(&R0.nb[e].w)];
  Y.sync(false);  // no rank leaves while another may still read its cells
}

// One depth per blockIdx.y, after the depths the bottom's slots.
template <class T>
__global__ void k_coarse_coef(const __grid_constant__ CoarseCoefs<T> C, int lamOnly) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  const auto& D = C.d[min(i, C.nd - 1)];
  const int n = D.n;
  if (e >= n) return;
  if (i == C.nd) {
    C.lamSlot[e] = D.lambda[C.slotFab[e]];
    return;
  }
  const int c = D.fab[e];
  T* out = D.out;
  out[n + e] = T(D.lambda[c]);
  if (lamOnly) return;
  out[e] = T(D.a[c]);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    out[(2 + 2 * d) * n + e] = T(D.b[d][D.fh[d * n + e]]);
    out[(3 + 2 * d) * n + e] = T(D.b[d][c]);
  }
}

template <class T>
auto kernelOf(int vc) {
  return vc ? k_coarse<T, 1> : k_coarse<T, 0>;
}

template <class K>
void configure(K kern) {
  check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoarseSmem), "coarse shared memory");
  check(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "coarse cluster size");
}

// Attributes at[0..2].  The block's shared memory is all the carve-out needs
// to hold (one block per SM): the rest stays first-level cache for the tables.
void launchConfig(cudaLaunchConfig_t& lc, cudaLaunchAttribute* at, int nh, int ranks, int bytes, cudaStream_t s) {
  lc = cudaLaunchConfig_t{};
  lc.gridDim = dim3(nh * ranks);
  lc.blockDim = dim3(kCoarseThreads);
  lc.dynamicSmemBytes = bytes;
  lc.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ranks;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  at[1].val.sharedMemCarveout = std::min(100, (bytes + 5 * 1024) * 100 / (228 * 1024) + 1);
  at[2].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[2].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = 3;
}

// ------------------------------------------------------------------- plans
int64_t domainCells(const LevelPlan& L) { return L.domain.numPts(); }
bool covers(const LevelPlan& L) {
  int64_t n = 0;
  for (const Box& b : L.grids.boxes) {
    for (int d = 0; d < 3; ++d)
      if (b.lo[d] < L.domain.lo[d] || b.hi[d] > L.domain.hi[d]) return false;
    n += b.numPts();
  }
  return n == domainCells(L);
}

// First box of each rank: consecutive boxes, about the same cells on each.
std::vector<int> boxRanks(const Layout& g, int ranks) {
  std::vector<int> first(ranks + 1, (int)g.size());
  const int64_t total = g.numCells();
  int64_t before = 0;
  int b = 0;
  for (int r = 0; r < ranks; ++r) {
    first[r] = b;
    const int64_t end = total * (r + 1) / ranks;
    while (b < (int)g.size() && before + g[b].numPts() / 2 < end) before += g[b++].numPts();
  }
  first[0] = 0;
  return first;
}

// Shared-memory offsets of a plan whose cell splits and halos are set.
void layOut(CoarsePlan& P) {
  auto pad = [](int64_t b) { return (b + 15) & ~int64_t(15); };
  int64_t top = 0;
  const int nd = (int)P.d.size();
  P.part = (int)top;
  top += pad((P.allRanks ? 4 : 1) * (int64_t)P.nbox * 8);
  P.pen = (int)top;
  top += pad((int64_t)P.nPen * 8);
  for (int f = 0; f < 2; ++f) {
    const int w = f == 0 ? 8 : 4;
    int64_t o = top, tmp = 0;
    for (int i = 0; i < nd; ++i) {
      P.phi[i][f] = (int)std::min<int64_t>(o, 1 << 30);
      o += pad((int64_t)P.d[i].nField * w);
      P.rhs[i][f] = (int)std::min<int64_t>(o, 1 << 30);
      o += pad((int64_t)P.d[i].nLoc * w);
      if (i + 1 < nd) tmp = std::max<int64_t>(tmp, P.d[i].nLoc);
    }
    // the restriction scratch and the bottom vectors are never live together
    P.tmp[f] = P.vec[f] = (int)std::min<int64_t>(o, 1 << 30);
    const int64_t nl = P.d.back().nLoc, nf = P.d.back().nField;
    o += std::max(pad(tmp * w), pad((f == 0 ? nf + 6 * nl : 2 * nf + 7 * nl) * 8));
    P.bytes[f] = (int)std::min<int64_t>(o, 1 << 30);
  }
}

// Splits the cells of every depth over the ranks.
void split(const std::vector<const LevelPlan*>& levels, int top, int ranks, CoarsePlan& P) {
  P = CoarsePlan();
  const int nd = (int)levels.size() - top;
  P.d.resize(nd);
  const Layout& bg = levels.back()->grids;
  P.nbox = (int)bg.size();
  P.dSolo = nd;
  for (int i = 0; i < nd; ++i) {
    CoarsePlan::Depth& D = P.d[i];
    D.n = (int)levels[top + i]->grids.numCells();
    D.dx = levels[top + i]->dx;
    D.solo = ranks == 1 || (D.n <= kSoloCells && P.nbox <= kAllRanksBoxes);
    if (D.solo && P.dSolo == nd) P.dSolo = i;
    D.per = D.solo ? D.n : (D.n + ranks - 1) / ranks;
    D.rankSlot.assign(ranks + 1, D.n);
    for (int r = 0; r <= ranks; ++r) D.rankSlot[r] = (int)std::min<int64_t>(D.n, (int64_t)r * D.per);
  }
  CoarsePlan::Depth& B = P.d.back();
  P.allRanks = P.nbox <= kAllRanksBoxes || ranks == 1;
  P.boxRank.assign(ranks + 1, P.nbox);
  P.boxRank[0] = 0;
  if (!B.solo) {
    P.boxRank = boxRanks(bg, ranks);
    int b = 0, s = 0;
    for (int r = 0; r <= ranks; ++r) {
      while (b < P.boxRank[r]) s += (int)bg[b++].numPts();
      B.rankSlot[r] = s;
    }
  }
  for (CoarsePlan::Depth& D : P.d)
    for (int r = 0; r < ranks; ++r) D.nLoc = std::max(D.nLoc, D.rankSlot[r + 1] - D.rankSlot[r]);
  for (const Box& b : bg.boxes) P.maxNx = std::max(P.maxNx, b.size(0));
  for (int r = 0; r < ranks; ++r) P.nPen = std::max(P.nPen, (P.boxRank[r + 1] - P.boxRank[r]) * P.maxNx);
}

}  // namespace

// Tables of one hierarchy from depth `top` on; false when a rank holds more
// cells than the indices do.
static bool buildTables(const std::vector<const LevelPlan*>& levels, int top, int ranks, const int* bc,
                        const bool* periodic, CoarsePlan& P) {
  split(levels, top, ranks, P);
  const int nd = (int)P.d.size();
  std::vector<std::vector<int>> enc(nd), slot0(nd);  // slot -> rank << shift | cell; first slot of each box
  const int mask = (1 << kCoarseRankShift) - 1;
  std::vector<std::vector<int>> entryOf(nd);  // slot -> entry: rank by rank, colour 0 first
  for (int i = 0; i < nd; ++i) {
    const LevelPlan& L = *levels[top + i];
    CoarsePlan::Depth& D = P.d[i];
    std::vector<char> colour;
    colour.reserve(D.n);
    for (const Box& x : L.grids.boxes) {
      slot0[i].push_back((int)colour.size());
      for (int k = x.lo[2]; k <= x.hi[2]; ++k)
        for (int j = x.lo[1]; j <= x.hi[1]; ++j)
          for (int q = x.lo[0]; q <= x.hi[0]; ++q) colour.push_back((q + j + k) & 1);
    }
    enc[i].resize(D.n);
    entryOf[i].resize(D.n);
    D.colStart.assign(2 * ranks + 1, D.n);
    int e = 0;
    for (int r = 0; r < ranks; ++r)
      for (int c = 0; c < 2; ++c) {
        D.colStart[2 * r + c] = e;
        for (int t = D.rankSlot[r]; t < D.rankSlot[r + 1]; ++t)
          if (colour[t] == c) {
            // the bottom's sums run over its boxes in order, the other depths'
            // passes over one colour at a time
            const int at = i + 1 == nd ? t - D.rankSlot[r] : e - D.colStart[2 * r];
            enc[i][t] = (r << kCoarseRankShift) | at;
            entryOf[i][t] = e++;
          }
      }
  }
  std::vector<char> fits(nd, 1);
  // Depths, their z-planes and their ranks are items of the host pool: a bottom of
  // 26^3 cells takes 2.0 ms of every new hierarchy's preparation on one thread,
  // 0.87 on 8 (1.3 with lists of the remote neighbours kept per plane and rank), a
  // depth of 20^3 0.78 and 0.71.  Below 16^3 cells waking the pool costs more than
  // it saves (0.3 ms on one thread).
  auto each = [](int cells, size_t items, const std::function<void(size_t)>& fn) {
    if (cells > 4096) return hostParallel(items, fn);
    for (size_t i = 0; i < items; ++i) fn(i);
  };
  each(P.d[0].n, nd, [&](size_t item) {
    const int i = (int)item;
    const LevelPlan& L = *levels[top + i];
    CoarsePlan::Depth& D = P.d[i];
    const Box& dom = L.domain;
    const int n = D.n, ext[3] = {dom.size(0), dom.size(1), dom.size(2)};
    PlanVec<int> owner(n);  // slot of each domain cell
    const std::vector<int>& entry = entryOf[i];
    auto cell = [&](int q, int j, int k) {
      return (q - dom.lo[0]) + (size_t)ext[0] * ((j - dom.lo[1]) + (size_t)ext[1] * (k - dom.lo[2]));
    };
    int s = 0;
    for (const Box& x : L.grids.boxes)
      for (int k = x.lo[2]; k <= x.hi[2]; ++k)
        for (int j = x.lo[1]; j <= x.hi[1]; ++j)
          for (int q = x.lo[0]; q <= x.hi[0]; ++q) owner[cell(q, j, k)] = s++;
    D.nb.resize(4 * (size_t)n);  // every entry of these tables is written below
    D.fab.resize(n);
    D.fh.resize(3 * (size_t)n);
    if (i + 1 < nd) D.par.resize(n);
    if (i > 0) D.child.resize(8 * (size_t)n);
    std::vector<std::pair<int, int>> planes;
    for (size_t b = 0; b < L.grids.size(); ++b)
      for (int k = L.grids[b].lo[2]; k <= L.grids[b].hi[2]; ++k) planes.push_back({(int)b, k});
    const size_t group = std::max<size_t>(1, 2048 * planes.size() / n);  // planes of about 2048 cells per item
    const size_t items = (planes.size() + group - 1) / group;
    PlanVec<int> near(6 * (size_t)n);  // per slot: its neighbours' slots (+x, -x, +y, ...), -1 beyond a wall
    each(n, items, [&](size_t g) {
      for (size_t pl = g * group; pl < std::min(planes.size(), (g + 1) * group); ++pl) {
        const int b = planes[pl].first, k = planes[pl].second;
        const Box& x = L.grids[b];
        const int step[3] = {1, x.size(0), x.size(0) * x.size(1)};
        int s = slot0[i][b] + step[2] * (k - x.lo[2]);
        const Box* coarse = i + 1 < nd ? &levels[top + i + 1]->grids[b] : nullptr;
        const Box* fine = i > 0 ? &levels[top + i - 1]->grids[b] : nullptr;
        for (int j = x.lo[1]; j <= x.hi[1]; ++j)
          for (int q = x.lo[0]; q <= x.hi[0]; ++q, ++s) {
            const int at = entry[s], p[3] = {q, j, k};
            const int me = enc[i][s], rank = me >> kCoarseRankShift;
            unsigned id[6];
            D.fab[at] = (int)cellIndex(L.boxes[b], q, j, k);
            for (int d = 0; d < 3; ++d) {
              D.fh[(size_t)d * n + at] = (int)cellIndex(L.boxes[b], q + (d == 0), j + (d == 1), k + (d == 2));
              for (int side = 0; side < 2; ++side) {  // + then -
                unsigned& v = id[2 * d + side];
                int& f = near[6 * (size_t)s + 2 * d + side];
                if (side == 0 ? p[d] < x.hi[d] : p[d] > x.lo[d]) {
                  f = s + (side == 0 ? step[d] : -step[d]);
                } else {
                  int m[3] = {q, j, k};
                  m[d] += side == 0 ? 1 : -1;
                  if (m[d] < dom.lo[d] || m[d] > dom.hi[d]) {
                    if (!(periodic && periodic[d])) {
                      f = -1;
                      v = (unsigned)(me & mask) | (bc && bc[2 * d + (side == 0 ? 1 : 0)] == 1 ? 0u : 0x8000u);
                      continue;
                    }
                    m[d] += side == 0 ? -ext[d] : ext[d];
                  }
                  f = owner[cell(m[0], m[1], m[2])];
                }
                const int e = enc[i][f];
                v = (e >> kCoarseRankShift) == rank ? (unsigned)(e & mask) : 0;  // else its halo element, below
              }
            }
            int* w = &D.nb[4 * (size_t)at];
            for (int d = 0; d < 3; ++d) w[d] = (int)(id[2 * d] | (id[2 * d + 1] << 16));
            w[3] = me & mask;
            auto half = [](int a) { return a < 0 ? -((1 - a) / 2) : a / 2; };  // floor(a / 2)
            if (coarse) {
              const int cs = slot0[i + 1][b] + (half(q) - coarse->lo[0]) +
                             coarse->size(0) * ((half(j) - coarse->lo[1]) + coarse->size(1) * (half(k) - coarse->lo[2]));
              D.par[at] = enc[i + 1][cs];
            }
            if (fine) {
              const int base = slot0[i - 1][b] + (2 * q - fine->lo[0]) +
                               fine->size(0) * ((2 * j - fine->lo[1]) + fine->size(1) * (2 * k - fine->lo[2]));
              for (int c = 0; c < 8; ++c)
                D.child[8 * (size_t)at + c] =
                    enc[i - 1][base + (c & 1) + fine->size(0) * (((c >> 1) & 1) + fine->size(1) * (c >> 2))];
            }
          }
      }
    });
    // Halos: the other ranks' cells a rank reads, by rank, colour and slot, so
    // that the cells a rank sends in one pass land next to each other.
    std::vector<int> nHalo(ranks);
    std::vector<std::vector<std::pair<int, unsigned>>> sent(ranks);  // by receiver: sender and colour, copy
    if (ranks > 1 && !D.solo) {
      PlanVec<int> slotOfEntry(n);
      for (int t = 0; t < n; ++t) slotOfEntry[entry[t]] = t;
      each(n, ranks, [&](size_t rank) {
        const int r = (int)rank;
        // the remote neighbours of this rank's cells
        auto remote = [&](auto fn) {
          for (int t = D.rankSlot[r]; t < D.rankSlot[r + 1]; ++t)
            for (int d = 0; d < 6; ++d) {
              const int f = near[6 * (size_t)t + d];
              if (f >= 0 && (enc[i][f] >> kCoarseRankShift) != r) fn(entry[t], d, entry[f]);
            }
        };
        std::vector<uint64_t> read(n / 64 + 1);  // by entry
        remote([&](int, int, int e) { read[e >> 6] |= uint64_t(1) << (e & 63); });
        PlanVec<unsigned short> where(n);  // halo element of each entry read
        for (size_t w = 0; w < read.size(); ++w)
          for (uint64_t left = read[w]; left; left &= left - 1) {
            const int e = (int)(64 * w) + __builtin_ctzll(left);
            const int from = enc[i][slotOfEntry[e]], owner = from >> kCoarseRankShift, src = from & mask;
            const int dst = D.nLoc + nHalo[r]++;
            if (src >= 1 << 13 || dst > 0x7fff || r > 15) {
              nHalo[r] = -1;
              return;
            }
            where[e] = (unsigned short)dst;
            sent[r].push_back({2 * owner + (e >= D.colStart[2 * owner + 1]),
                               (unsigned)src << 19 | (unsigned)r << 15 | (unsigned)dst});
          }
        remote([&](int at, int d, int e) {
          D.nb[4 * (size_t)at + (d >> 1)] |= (int)((unsigned)where[e] << (16 * (d & 1)));
        });
      });
    }
    D.nHalo = 0;
    for (int r = 0; r < ranks; ++r) {
      if (nHalo[r] < 0) fits[i] = 0;
      D.nHalo = std::max(D.nHalo, nHalo[r]);
    }
    D.pushStart.assign(2 * ranks + 1, 0);
    for (const auto& v : sent)
      for (const auto& p : v) ++D.pushStart[p.first + 1];
    for (int q = 0; q < 2 * ranks; ++q) D.pushStart[q + 1] += D.pushStart[q];
    D.push.resize(D.pushStart.back());
    std::vector<int> next(D.pushStart.begin(), D.pushStart.end() - 1);
    for (const auto& v : sent)
      for (const auto& p : v) D.push[next[p.first]++] = p.second;
    D.nField = D.nLoc + D.nHalo;
    if (D.nField > 0x8000) fits[i] = 0;
  });
  if (std::find(fits.begin(), fits.end(), 0) != fits.end()) return false;
  const LevelPlan& B = *levels.back();
  const CoarsePlan::Depth& DB = P.d.back();
  int r = 0;
  for (size_t b = 0; b < B.grids.size(); ++b) {
    while (r + 1 < ranks && (int)b >= P.boxRank[r + 1]) ++r;
    const Box& x = B.grids[b];
    for (int v : {slot0[nd - 1][b] - DB.rankSlot[r], x.size(0), x.size(1), x.size(2)}) P.box.push_back(v);
    for (int k = x.lo[2]; k <= x.hi[2]; ++k)
      for (int j = x.lo[1]; j <= x.hi[1]; ++j)
        for (int q = x.lo[0]; q <= x.hi[0]; ++q) P.bottomFab.push_back((int)cellIndex(B.boxes[b], q, j, k));
  }
  layOut(P);
  return true;
}

bool buildCoarse(const std::vector<const LevelPlan*>& levels, int top, int ranks, const int* bc, const bool* periodic,
                 CoarsePlan& P) {
  for (size_t t = top; t < levels.size(); ++t) {
    if (!covers(*levels[t])) return false;
    // across an odd periodic extent a cell's neighbour has its own colour
    for (int d = 0; d < 3; ++d)
      if (periodic && periodic[d] && levels[t]->domain.size(d) % 2) return false;
  }
  return buildTables(levels, top, ranks, bc, periodic, P) && P.bytes[0] <= kCoarseSmem;
}

bool planCoarse(const std::vector<std::vector<const LevelPlan*>>& levels, const int* bc, const bool* periodic, bool vc,
                int* top, int* ranks, std::vector<CoarsePlan>& plans) {
  const int D = (int)levels[0].size();
  // Sixteen ranks for one hierarchy; eight each when several share the device.
  const int most = levels.size() == 1 ? 16 : 8;
  for (int t = std::max(0, D - kCoarseMaxDepths); t < D; ++t) {
    int64_t cells = 0;
    for (const auto& h : levels) cells = std::max(cells, h[t]->grids.numCells());
    if (cells > (t + 1 == D ? kCoarseMaxBottomCells : vc ? kCoarseMaxCellsVC : kCoarseMaxCells)) continue;
    for (int r = cells <= kSoloCells ? 1 : most; r == 1 || r >= 8; r /= 2) {
      plans.assign(levels.size(), CoarsePlan());
      std::vector<char> ok(levels.size(), 0);
      hostParallel(levels.size(), [&](size_t k) { ok[k] = buildCoarse(levels[k], t, r, bc, periodic, plans[k]); });
      int bytes = 0;
      for (const CoarsePlan& P : plans)
        for (int f = 0; f < 2; ++f)
          if (P.bytes[f] <= kCoarseSmem) bytes = std::max(bytes, P.bytes[f]);
      if (std::find(ok.begin(), ok.end(), 0) == ok.end() && coarseFits(r, bytes)) {
        *top = t;
        *ranks = r;
        return true;
      }
      if (r == 1) break;
    }
  }
  plans.clear();
  return false;
}

template <class T>
void gatherCoarse(const CoarseCoefs<T>& C, bool lamOnly, cudaStream_t s) {
  int most = 0;
  for (int i = 0; i < C.nd; ++i) most = std::max(most, C.d[i].n);
  if (most == 0) return;
  k_coarse_coef<T><<<dim3((most + 255) / 256, C.nd + (C.lamSlot ? 1 : 0)), 256, 0, s>>>(C, lamOnly);
  addLaunches(1);
  check(cudaGetLastError(), "coarse coefficients");
}
template void gatherCoarse<double>(const CoarseCoefs<double>&, bool, cudaStream_t);
template void gatherCoarse<float>(const CoarseCoefs<float>&, bool, cudaStream_t);

bool coarseFits(int ranks, int bytes) {
  for (int vc = 0; vc < 2; ++vc)
    for (int f = 0; f < 2; ++f) {
      cudaLaunchConfig_t lc;
      cudaLaunchAttribute at[3];
      launchConfig(lc, at, 1, ranks, bytes, nullptr);
      int n = 0;
      cudaError_t e;
      if (f == 0) {
        configure(kernelOf<double>(vc));
        e = cudaOccupancyMaxActiveClusters(&n, kernelOf<double>(vc), &lc);
      } else {
        configure(kernelOf<float>(vc));
        e = cudaOccupancyMaxActiveClusters(&n, kernelOf<float>(vc), &lc);
      }
      if (e != cudaSuccess) {
        cudaGetLastError();  // an unsupported cluster size is an answer, not a failure
        return false;
      }
      if (n < 1) return false;
    }
  return true;
}

template <class T>
void coarseCycle(const CoarseHier* hier, int nh, int ranks, int bytes, const std::vector<Scal>& sc, T* corr, const T* res,
                 int vc, int pre, int post, int bottomSweeps, int numMG, bool oneCell, bool fromZero,
                 const BottomConfig& cfg, double eps, double mult, const double* metrics, const double* epsPer,
                 cudaStream_t s) {
  Args<T> A;
  A.hier = hier;
  A.corr = corr;
  A.res = res;
  A.ranks = ranks;
  A.pre = pre;
  A.post = post;
  A.bottom = bottomSweeps;
  A.numMG = numMG;
  A.oneCell = oneCell;
  A.fromZero = fromZero;
  A.cfg = cfg;
  A.eps = eps;
  A.mult = mult;
  A.metrics = metrics;
  A.epsPer = epsPer;
  for (int i = 0; i < kCoarseMaxDepths; ++i) A.sc[i] = sc[std::min<size_t>(i, sc.size() - 1)];
  cudaLaunchConfig_t lc;
  cudaLaunchAttribute at[3];
  launchConfig(lc, at, nh, ranks, bytes, s);
  check(cudaLaunchKernelEx(&lc, kernelOf<T>(vc), A), "coarse cycle");
  addLaunches(1);
  check(cudaGetLastError(), "coarse cycle");
}
#define CMG_INST(T)                                                                                                  \
  template void coarseCycle<T>(const CoarseHier*, int, int, int, const std::vector<Scal>&, T*, const T*, int, int,   \
                               int, int, int, bool, bool, const BottomConfig&, double, double, const double*,        \
                               const double*, cudaStream_t);
CMG_INST(double)
CMG_INST(float)

}  // namespace cmg
