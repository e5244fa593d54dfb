// Device kernels of the AMR multigrid V-cycle.  Each kernel states the
// reference operation (ChF kernel or C++ routine, paths relative to the
// Chombo lib/src tree) whose arithmetic it reproduces term for term, so the
// FP64 build (compiled with --fmad=false) rounds exactly like the reference.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <stdexcept>

#include <cooperative_groups.h>

#include "bottomdev.H"
#include "cellops.H"
#include "kernels.H"
#include "synthdev.H"
#include "plan.H"
#include "synthetic.H"

namespace cg = cooperative_groups;

namespace cmg {

namespace {

inline void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    char buf[256];
    std::snprintf(buf, sizeof(buf), "cmg: %s: %s", what, cudaGetErrorString(e));
    throw std::runtime_error(buf);
  }
}
std::atomic<long long> g_launches{0};
#define CMG_LAUNCHED(name) (g_launches.fetch_add(1, std::memory_order_relaxed), check(cudaGetLastError(), name))

// Launches a kernel that may start while the previous one of the stream still
// runs: its blocks are put on the device and read their tables (fixed since the
// set-up) early, and touch fields after beginAfterPrevious, which waits until
// the previous kernel has finished and its writes are visible.  Every kernel
// launched so calls it in every thread before anything else than table loads
// (before any return: a kernel that ended without waiting would let the next
// one pass it).  It lets the next launch begin only then, so at most one kernel
// waits on the device.  The launch latency of a chain of small kernels
// hides behind the kernel before: two-level 64^3 VC solve 4.44 -> 4.11 ms,
// 64^3 Poisson 1.20 -> 1.12, BiCGStab with three levels 50.1 -> 46.3, heat
// steps 9.84 -> 9.38, forest of 12 mixed 22.6 -> 21.9; large levels the same.
__device__ __forceinline__ void beginAfterPrevious() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
void launchNext(void (*kern)(P...), dim3 grid, int block, cudaStream_t s, A... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = grid;
  lc.blockDim = dim3(block);
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  check(cudaLaunchKernelEx(&lc, kern, static_cast<P>(args)...), "launch");
}

// Cell q of box b in x-fastest order.
__device__ __forceinline__ bool allCell(const BoxDesc& b, int q, int& i, int& j, int& k) {
  int nx = b.hi[0] - b.lo[0] + 1, ny = b.hi[1] - b.lo[1] + 1, nz = b.hi[2] - b.lo[2] + 1;
  if (q >= nx * ny * nz) return false;
  const int r = fastDiv(q, nx, b.mNx);
  const int kk = fastDiv(r, ny, b.mNy);
  i = b.lo[0] + (q - r * nx);
  j = b.lo[1] + (r - kk * ny);
  k = b.lo[2] + kk;
  return true;
}

// q-th cell of colour `color` (cells with i+j+k = color mod 2), the cells the
// GSRB kernels visit for redBlack = color (AMRPoissonOpF.ChF:151-158).
__device__ __forceinline__ bool colorCell(const BoxDesc& b, int q, int color, int& i, int& j, int& k) {
  int nx = b.hi[0] - b.lo[0] + 1, ny = b.hi[1] - b.lo[1] + 1, nz = b.hi[2] - b.lo[2] + 1;
  int half = (nx + 1) / 2;
  const int r = fastDiv(q, half, b.mHalf);
  if (r >= ny * nz) return false;
  const int kk = fastDiv(r, ny, b.mNy);
  j = b.lo[1] + (r - kk * ny);
  k = b.lo[2] + kk;
  const int par = (b.lo[0] + j + k + color) & 1;
  i = b.lo[0] + par + 2 * (q - r * half);
  return i <= b.hi[0];
}

// ---------------------------------------------------------------- ghosts
// Exchange copies (BoxLayoutData local copy), homogeneous Dirichlet faces
// (BCFunc.cpp:25-32,294-354: ghost = 2*0 - near), homogeneous quadratic and
// linear coarse-fine ghosts (InterpF.ChF:435-494) and zeroing.
// Each thread takes GHOST_PER_THREAD ghost cells of its block's range; the
// task of cell g is found by binary search in the cumulative cell counts,
// between the tasks holding the first cells of this block and of the next
// (blockTask).  The cells' target and source indices are resolved first and
// their loads issued together.  par >= 0 fills only the ghost cells of colour
// par ((i+j+k) & 1 == par): a colour pass reads no ghost of its own colour,
// so the fill before it needs only the other one; then a task offers
// colourSlots() slots, stepping by two along its parity axis.
template <class T>
__global__ void __launch_bounds__(GHOST_THREADS) k_ghost(const GhostTaskDev* tasks, const int* start,
                                                         const int* blockTask, int ntask, int ncell, int par, T* f,
                                                         T c1, T c2, T flin) {
  beginAfterPrevious();
  const int b0 = blockTask[blockIdx.x], b1 = min(blockTask[blockIdx.x + 1], ntask - 1);
  int64_t dst[GHOST_PER_THREAD], s1[GHOST_PER_THREAD], s2[GHOST_PER_THREAD];
  int kind[GHOST_PER_THREAD];
#pragma unroll
  for (int u = 0; u < GHOST_PER_THREAD; ++u) {
    kind[u] = -1;
    dst[u] = s1[u] = s2[u] = 0;
    const int g0 = blockIdx.x * GHOST_PER_BLOCK + u * GHOST_THREADS + threadIdx.x;
    if (g0 >= ncell) continue;
    int lo = b0, hi = b1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (start[mid] <= g0)
        lo = mid;
      else
        hi = mid - 1;
    }
    const GhostTaskDev& t = tasks[lo];
    int q = g0 - start[lo], c[3];
    if (par < 0) {
      const int nx = t.hi[0] - t.lo[0] + 1, ny = t.hi[1] - t.lo[1] + 1;
      c[0] = t.lo[0] + q % nx;
      int r = q / nx;
      c[1] = t.lo[1] + r % ny;
      c[2] = t.lo[2] + r / ny;
    } else {
      const int a = t.ax, d1 = a == 0 ? 1 : 0, d2 = a == 2 ? 1 : 2;
      const int ha = (t.hi[a] - t.lo[a] + 2) >> 1, n1 = t.hi[d1] - t.lo[d1] + 1;
      int r = q / ha;
      c[d1] = t.lo[d1] + r % n1;
      c[d2] = t.lo[d2] + r / n1;
      c[a] = t.lo[a] + ((par - t.lo[a] - c[d1] - c[d2]) & 1) + 2 * (q % ha);
      if (c[a] > t.hi[a]) continue;
    }
    kind[u] = t.kind;
    dst[u] = cellIndex(t.dst, c[0], c[1], c[2]);
    if (t.kind == G_COPY) {
      s1[u] = cellIndex(t.src, c[0] - t.shift[0], c[1] - t.shift[1], c[2] - t.shift[2]);
    } else if (t.kind != G_ZERO) {
      int e[3] = {0, 0, 0};
      e[t.dir] = -t.side;  // one cell inward
      s1[u] = cellIndex(t.dst, c[0] + e[0], c[1] + e[1], c[2] + e[2]);
      s2[u] = t.kind == G_CFQUAD ? cellIndex(t.dst, c[0] + 2 * e[0], c[1] + 2 * e[1], c[2] + 2 * e[2]) : s1[u];
    }
  }
  T v1[GHOST_PER_THREAD], v2[GHOST_PER_THREAD];
#pragma unroll
  for (int u = 0; u < GHOST_PER_THREAD; ++u) {
    if (kind[u] > 0 && kind[u] != G_ZERO) v2[u] = f[s2[u]];
    if (kind[u] >= 0 && kind[u] != G_ZERO) v1[u] = f[s1[u]];
  }
#pragma unroll
  for (int u = 0; u < GHOST_PER_THREAD; ++u) {
    const int k = kind[u];
    if (k < 0) continue;
    T out;
    if (k == G_COPY) {
      out = v1[u];
    } else if (k == G_ZERO) {
      out = T(0);
    } else if (k == G_BC) {
      T zero = T(0);
      out = T(2) * zero - v1[u];
    } else if (k == G_NEU) {
      out = v1[u];
    } else if (k == G_CFLIN) {
      out = flin * v1[u];
    } else {
      out = c1 * v1[u] + c2 * v2[u];
    }
    f[dst[u]] = out;
  }
}

// Ghost fill from the flat per-cell lists: entries [a0, a1) then [b0, b1),
// U per thread (GHOST_THREADS apart, so each batch of loads is coalesced),
// no table walk between a thread and its data.  A fill's sources are valid
// cells and its destinations ghost cells, so all loads of a thread are
// issued before its stores: the list and source latencies of its U entries
// overlap instead of adding up.
template <class T, int U>
__global__ void __launch_bounds__(GHOST_THREADS) k_ghostcells(const GhostCell* __restrict__ e, int a0, int a1,
                                                              int b0, int b1, T* f, T c1, T c2, T flin) {
  const int na = a1 - a0, n = na + (b1 - b0);
  const int base = blockIdx.x * (GHOST_THREADS * U) + threadIdx.x;
  GhostCell g[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int q = base + u * GHOST_THREADS;
    g[u] = q < n ? e[q < na ? a0 + q : b0 + (q - na)] : GhostCell{-1, 0, -1};
  }
  beginAfterPrevious();
  T v1[U], v2[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    v1[u] = g[u].dst >= 0 ? f[g[u].s1] : T(0);
    v2[u] = g[u].dst >= 0 && g[u].s2 >= 0 ? f[g[u].s2] : T(0);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (g[u].dst < 0) continue;
    T out;
    if (g[u].s2 == -1) {
      out = v1[u];
    } else if (g[u].s2 == -2) {
      T zero = T(0);
      out = T(2) * zero - v1[u];
    } else if (g[u].s2 == -3) {
      out = flin * v1[u];
    } else {
      out = c1 * v1[u] + c2 * v2[u];
    }
    f[g[u].dst] = out;
  }
}

// ---------------------------------------------------------------- stencils
// Sum of the six neighbours in the ChF order (+x, -x, +y, -y, +z, -z).
template <class T>
__device__ __forceinline__ T nbrSum(const T* p, const Stencil& st) {
  return p[st.xp] + p[st.xm] + p[st.yp] + p[st.ym] + p[st.zp] + p[st.zm];
}

// Variable-coefficient divergence term of VCAMRPoissonOpF.ChF:93-111 (the
// face above the cell in direction d is stored at the neighbour's index).
template <class T>
__device__ __forceinline__ T vcDiv(const T* p, const T* b0, const T* b1, const T* b2, const Stencil& st) {
  T pc = p[st.c];
  return b0[st.xp] * (p[st.xp] - pc) - b0[st.c] * (pc - p[st.xm]) + b1[st.yp] * (p[st.yp] - pc) -
         b1[st.c] * (pc - p[st.ym]) + b2[st.zp] * (p[st.zp] - pc) - b2[st.c] * (pc - p[st.zm]);
}

// Factors of the homogeneous coarse-fine ghost values.
struct GhostCoef {
  double c1, c2, flin;
};

// Value of one ghost-fill entry (GhostCell) from the current field: the
// arithmetic of k_ghostcells.
template <class T>
__device__ __forceinline__ T ghostCellValue(const GhostCell& g, const T* f, const GhostCoef& gc) {
  const T v1 = f[g.s1];
  if (g.s2 == -1) return v1;
  if (g.s2 == -2) {
    T zero = T(0);
    return T(2) * zero - v1;
  }
  if (g.s2 == -3) return T(gc.flin) * v1;
  return T(gc.c1) * v1 + T(gc.c2) * f[g.s2];
}

// GSRBLAPLACIAN / GSRBHELMHOLTZ (AMRPoissonOpF.ChF:51-198) and
// GSRBHELMHOLTZVC3D (VCAMRPoissonOpF.ChF:57-125), one colour, without a fill: the
// block first writes the face ghosts its own cells read (the chunk's entries
// of the fill that would precede the pass, pre[preStart[chunk] ..
// preStart[chunk + 1])).  Those ghosts belong to the other colour, so no other
// block writes their sources during the pass, and each is read only by the
// one valid cell next to it, updated by this block after the barrier: the
// values are the fill's.  The first entry of every thread is read before the
// wait for the previous kernel, and the cell's own values before the barrier:
// heat steps 8.12 -> 7.82 ms, two-level 64^3 VC solve 3.91 -> 3.84.  (The face
// coefficients before the barrier too: VC 4% slower.  Two cells per thread, as
// k_gsrb_pair: 2.5% slower on all, half the threads are in flight.)
template <class T, int VC>
__global__ void __launch_bounds__(CHUNK) k_gsrb(const BoxDesc* boxes, const Chunk* chunks, T* phi, const T* rhs,
                                                int color, Scal sc, const T* a, const T* b0, const T* b1, const T* b2,
                                                const T* lam, const GhostCell* __restrict__ pre,
                                                const int* __restrict__ preStart, GhostCoef gc) {
  const Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  int g0 = preStart[blockIdx.x] + threadIdx.x;
  const int g1 = preStart[blockIdx.x + 1];
  GhostCell g = {};
  if (g0 < g1) g = pre[g0];
  int i = 0, j = 0, k = 0;
  const bool in = colorCell(bd, ch.start + threadIdx.x, color, i, j, k);
  const Stencil st = stencil(bd, i, j, k);
  const int64_t c = st.c;
  beginAfterPrevious();
  T pc = T(0), rh = T(0), av = T(0), lv = T(0), f[6];
  if (in) {
    pc = phi[c];
    rh = rhs[c];
  }
  if (g0 < g1) phi[g.dst] = ghostCellValue(g, phi, gc);
  for (g0 += blockDim.x; g0 < g1; g0 += blockDim.x) {
    g = pre[g0];
    phi[g.dst] = ghostCellValue(g, phi, gc);
  }
  __syncthreads();
  if (!in) return;
  if (VC) {
    av = a[c];
    lv = lam[c];
    f[0] = b0[st.xp];
    f[1] = b0[c];
    f[2] = b1[st.yp];
    f[3] = b1[c];
    f[4] = b2[st.zp];
    f[5] = b2[c];
  }
  const T v[6] = {phi[st.xp], phi[st.xm], phi[st.yp], phi[st.ym], phi[st.zp], phi[st.zm]};
  phi[c] = gsrbValue<T, VC>(sc, pc, rh, v, av, lv, f);
}

// One cell of a colour pass whose ghosts are filled: k_gsrb's update.
template <class T, int VC>
__device__ __forceinline__ void gsrbOne(const BoxDesc& bd, int i, int j, int k, T* phi, const T* rhs, const Scal& sc,
                                        const T* a, const T* b0, const T* b1, const T* b2, const T* lam) {
  const Stencil s = stencil(bd, i, j, k);
  const T v[6] = {phi[s.xp], phi[s.xm], phi[s.yp], phi[s.ym], phi[s.zp], phi[s.zm]};
  T f[6], av = T(0), lv = T(0);
  if (VC) {
    av = a[s.c];
    lv = lam[s.c];
    f[0] = b0[s.xp];
    f[1] = b0[s.c];
    f[2] = b1[s.yp];
    f[3] = b1[s.c];
    f[4] = b2[s.zp];
    f[5] = b2[s.c];
  }
  phi[s.c] = gsrbValue<T, VC>(sc, phi[s.c], rhs[s.c], v, av, lv, f);
}

// The one-colour pass of k_gsrb (ghosts filled before the pass) with two
// cells per thread: colour indices q and q + 1 of the chunk, which for an
// even number of colour cells per row are neighbours in one row (i and
// i + 2), sharing the enumeration, the index arithmetic and the x-neighbour
// between them (phi[oth + xo] is +x of the first and -x of the second).  A
// pair split across rows (odd rows) updates its cells one by one.  All loads
// of a pair come before its stores (cells of one colour read only the other
// colour and themselves), so the updates are those of k_gsrb.
template <class T, int VC>
__global__ void __launch_bounds__(CHUNK / 2) k_gsrb_pair(const BoxDesc* boxes, const Chunk* chunks, T* phi,
                                                         const T* rhs, int color, Scal sc, const T* a, const T* b0,
                                                         const T* b1, const T* b2, const T* lam) {
  const Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  beginAfterPrevious();
  const int q = ch.start + 2 * threadIdx.x;
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1, nz = bd.hi[2] - bd.lo[2] + 1;
  const int half = (nx + 1) / 2;
  const int r = fastDiv(q, half, bd.mHalf);
  if (r >= ny * nz) return;
  const int kk = fastDiv(r, ny, bd.mNy);
  const int j = bd.lo[1] + (r - kk * ny), k = bd.lo[2] + kk;
  const int m = q - r * half;
  const int i = bd.lo[0] + ((bd.lo[0] + j + k + color) & 1) + 2 * m;
  if (m + 1 < half && i + 2 <= bd.hi[0]) {
    // both cells in this row
    const Stencil st = stencil(bd, i, j, k);
    const int c = st.c;
    const T pc0 = phi[c], pc1 = phi[c + 1];
    const T rh0 = rhs[c], rh1 = rhs[c + 1];
    const T xm = phi[st.xm], xc = phi[st.xp], xp = phi[st.xp + 1];
    const T v0[6] = {xc, xm, phi[st.yp], phi[st.ym], phi[st.zp], phi[st.zm]};
    const T v1[6] = {xp, xc, phi[st.yp + 1], phi[st.ym + 1], phi[st.zp + 1], phi[st.zm + 1]};
    T av0 = T(0), av1 = T(0), lv0 = T(0), lv1 = T(0), f0[6], f1[6];
    if (VC) {
      av0 = a[c];
      av1 = a[c + 1];
      lv0 = lam[c];
      lv1 = lam[c + 1];
      f0[0] = b0[st.xp];
      f0[1] = b0[c];
      f0[2] = b1[st.yp];
      f0[3] = b1[c];
      f0[4] = b2[st.zp];
      f0[5] = b2[c];
      f1[0] = b0[st.xp + 1];
      f1[1] = b0[c + 1];
      f1[2] = b1[st.yp + 1];
      f1[3] = b1[c + 1];
      f1[4] = b2[st.zp + 1];
      f1[5] = b2[c + 1];
    }
    const T n0 = gsrbValue<T, VC>(sc, pc0, rh0, v0, av0, lv0, f0);
    const T n1 = gsrbValue<T, VC>(sc, pc1, rh1, v1, av1, lv1, f1);
    phi[c] = n0;
    phi[c + 1] = n1;
    return;
  }
  if (i <= bd.hi[0]) gsrbOne<T, VC>(bd, i, j, k, phi, rhs, sc, a, b0, b1, b2, lam);
  int i1, j1, k1;
  if (colorCell(bd, q + 1, color, i1, j1, k1)) gsrbOne<T, VC>(bd, i1, j1, k1, phi, rhs, sc, a, b0, b1, b2, lam);
}

// Two same-row cells of one colour on a uniform level: the element of the
// first cell and of its neighbours, those beyond a face where their value is
// (UniformFaces), and which faces the pair touches.
struct UniformPair {
  int c, xp, xm, xe, yp, ym, zp, zm;  // xe: +x of the second cell
  int on;                             // bit f: the pair lies on face f
  // element indices of the face coefficients at +x, +y, +z (the box's own)
  int bx, by, bz;
};
__device__ __forceinline__ bool uniformPair(const BoxDesc& bd, const UniformFaces& uf, int q, int color,
                                            UniformPair& p) {
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1, nz = bd.hi[2] - bd.lo[2] + 1;
  const int half = nx >> 1;
  const int r = fastDiv(q, half, bd.mHalf);
  if (r >= ny * nz) return false;
  const int kk = fastDiv(r, ny, bd.mNy), jj = r - kk * ny, m = q - r * half;
  const int ii = ((bd.lo[0] + bd.lo[1] + bd.lo[2] + jj + kk + color) & 1) + 2 * m;  // x of the first cell in its box
  const int sy = bd.px >> 1, sz = sy * bd.py;
  const int slot = ((ii + 1) >> 1) + sy * (jj + 1) + sz * (kk + 1);
  const int own = (int)bd.off + color * (int)bd.half, oth = (int)bd.off + (1 - color) * (int)bd.half + slot;
  const int xo = (ii + 1) & 1;
  p.c = own + slot;
  const bool lx = ii == 0, hx = ii + 3 == nx, ly = jj == 0, hy = jj + 1 == ny, lz = kk == 0, hz = kk + 1 == nz;
  p.on = (lx ? 1 : 0) | (hx ? 2 : 0) | (ly ? 4 : 0) | (hy ? 8 : 0) | (lz ? 16 : 0) | (hz ? 32 : 0);
  p.bx = oth + xo;
  p.by = oth + sy;
  p.bz = oth + sz;
  p.xm = oth + xo - 1 + (lx ? uf.d[0] : 0);
  p.xp = oth + xo;
  p.xe = oth + xo + 1 + (hx ? uf.d[1] : 0);
  p.ym = oth - sy + (ly ? uf.d[2] : 0);
  p.yp = oth + sy + (hy ? uf.d[3] : 0);
  p.zm = oth - sz + (lz ? uf.d[4] : 0);
  p.zp = oth + sz + (hz ? uf.d[5] : 0);
  return true;
}

// The pair's values, neighbours (v0, v1 as gsrbValue takes them) and face
// coefficients.
template <class T, int VC>
__device__ __forceinline__ void uniformLoad(const UniformPair& p, const UniformFaces& uf, const T* phi, const T* b0,
                                            const T* b1, const T* b2, T* pc, T* v0, T* v1, T* f0, T* f1) {
  pc[0] = phi[p.c];
  pc[1] = phi[p.c + 1];
  v0[0] = phi[p.xp];
  v0[1] = phi[p.xm];
  v1[0] = phi[p.xe];
  v0[2] = phi[p.yp];
  v1[2] = phi[p.yp + 1];
  v0[3] = phi[p.ym];
  v1[3] = phi[p.ym + 1];
  v0[4] = phi[p.zp];
  v1[4] = phi[p.zp + 1];
  v0[5] = phi[p.zm];
  v1[5] = phi[p.zm + 1];
  if (VC) {
    f0[0] = b0[p.bx];
    f0[1] = b0[p.c];
    f0[2] = b1[p.by];
    f0[3] = b1[p.c];
    f0[4] = b2[p.bz];
    f0[5] = b2[p.c];
    f1[0] = b0[p.bx + 1];
    f1[1] = b0[p.c + 1];
    f1[2] = b1[p.by + 1];
    f1[3] = b1[p.c + 1];
    f1[4] = b2[p.bz + 1];
    f1[5] = b2[p.c + 1];
  }
  v1[1] = v0[0];
  if (uf.kind) {  // a box on the domain boundary
    auto wall = [&](int face, T& v, T x) {
      const int k = uf.kind >> (2 * face) & 3;
      if (k && (p.on >> face & 1)) v = k == 1 ? T(0) - x : x;
    };
    wall(0, v0[1], pc[0]);
    wall(1, v1[0], pc[1]);
    wall(2, v0[3], pc[0]);
    wall(2, v1[3], pc[1]);
    wall(3, v0[2], pc[0]);
    wall(3, v1[2], pc[1]);
    wall(4, v0[5], pc[0]);
    wall(4, v1[5], pc[1]);
    wall(5, v0[4], pc[0]);
    wall(5, v1[4], pc[1]);
  }
}

// The one-colour pass of k_gsrb_pair on a uniform level: neighbours beyond a
// face are read from the box beside it (they have the other colour, so the
// pass does not change them), so no ghost fill precedes it.  A block takes
// `per` consecutive chunks, so that the chain of table loads before its data is
// paid once for several chunks of the same box.  Bound by memory latency: 512^3
// periodic in 32^3 boxes, 460 us a pass (4.7 TB/s of 16 bytes per cell) against
// 442 us and a 207 us fill; its solve, with the residual and the restriction
// below, 115.4 -> 89.3 ms.
template <class T, int VC>
__global__ void __launch_bounds__(CHUNK / 2) k_gsrb_uniform(const BoxDesc* boxes, const UniformFaces* faces,
                                                            const Chunk* chunks, int n, int per, T* phi, const T* rhs,
                                                            int color, Scal sc, const T* a, const T* b0, const T* b1,
                                                            const T* b2, const T* lam) {
  const int end = min(n, (int)(blockIdx.x + 1) * per);
  for (int ci = blockIdx.x * per; ci < end; ++ci) {
    const Chunk ch = chunks[ci];
    const BoxDesc bd = boxes[ch.box];
    const UniformFaces uf = faces[ch.box];
    if (ci == (int)blockIdx.x * per) beginAfterPrevious();
    UniformPair p;
    if (!uniformPair(bd, uf, ch.start + 2 * threadIdx.x, color, p)) continue;
    T pc[2], v0[6], v1[6], f0[6], f1[6], av0 = T(0), av1 = T(0), lv0 = T(0), lv1 = T(0);
    const T rh0 = rhs[p.c], rh1 = rhs[p.c + 1];
    if (VC) {
      av0 = a[p.c];
      av1 = a[p.c + 1];
      lv0 = lam[p.c];
      lv1 = lam[p.c + 1];
    }
    uniformLoad<T, VC>(p, uf, phi, b0, b1, b2, pc, v0, v1, f0, f1);
    const T x0 = gsrbValue<T, VC>(sc, pc[0], rh0, v0, av0, lv0, f0);
    const T x1 = gsrbValue<T, VC>(sc, pc[1], rh1, v1, av1, lv1, f1);
    phi[p.c] = x0;
    phi[p.c + 1] = x1;
  }
}

// The first colour pass (colour 0) of a relaxation whose field is zero: the
// update of k_gsrb from zero values, in which the operator term vanishes, so
// neither phi, its ghosts nor the other coefficients are read, and the other
// colour's zeros are written on the way (no memset before the pass and no fill
// of colour-1 ghosts).  Two cells of each colour of a row per thread, as
// k_gsrb_pair enumerates them.  Bound by DRAM: 16 bytes per cell (rhs and
// lambda read on half the cells, phi written) against 8 for the memset, the
// fill and 48 for the full VC pass.  With the fused norm and the prolongation
// below: three-level 128^3 VC solve 73.1 -> 66.0 ms, mixed 49.2 -> 44.6 ms,
// 512^3 periodic 133.7 -> 115.4 ms.
template <class T, int VC>
__global__ void __launch_bounds__(CHUNK / 2) k_gsrb_first(const BoxDesc* boxes, const Chunk* chunks, T* phi,
                                                          const T* rhs, Scal sc, const T* lam) {
  const Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  beginAfterPrevious();
  const int q0 = ch.start + 2 * threadIdx.x;
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1, nz = bd.hi[2] - bd.lo[2] + 1;
  const int half = (nx + 1) / 2;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int q = q0 + u, r = fastDiv(q, half, bd.mHalf);
    if (r >= ny * nz) return;
    const int kk = fastDiv(r, ny, bd.mNy);
    const int j = r - kk * ny, m = q - r * half;
    const int par = (bd.lo[0] + bd.lo[1] + j + bd.lo[2] + kk) & 1;  // colour of the row's first cell
    const int row = (bd.px >> 1) * (j + 1 + bd.py * (kk + 1));      // its slots (px is even)
    const int own = 2 * m + par, oth = 2 * m + 1 - par;             // x of the colour-0 and colour-1 cell
    if (own < nx) {
      const int c = (int)bd.off + row + ((own + 1) >> 1);
      if (VC)
        phi[c] = T(0) - lam[c] * (T(0) - rhs[c]);
      else if (sc.laplacian)
        phi[c] = T(sc.lambda) * (rhs[c] - T(0));
      else
        phi[c] = T(0) + T(sc.lambda) * (T(0) - rhs[c]);
    }
    if (oth < nx) phi[(int)bd.off + (int)bd.half + row + ((oth + 1) >> 1)] = T(0);
  }
}

// Neighbour value across a box face from its fill rule (the value the ghost
// fill before the colour pass would have written, as in ghostValue).
template <class T>
__device__ __forceinline__ T ruleValue(const FaceRule& r, T pc, const T* phi, const GhostCoef& gc) {
  if (r.kind == FR_COPY || r.kind == FR_FAB) return phi[r.src];
  if (r.kind == FR_NEU) return pc;
  if (r.kind == FR_BC) {
    T zero = T(0);
    return T(2) * zero - pc;
  }
  if (r.kind == FR_CFLIN) return T(gc.flin) * pc;
  return T(gc.c1) * pc + T(gc.c2) * phi[r.src];
}

// One cell of a red-black sweep with the neighbours beyond its box taken from
// the face rules: the arithmetic of k_gsrb (GSRBHELMHOLTZVC3D,
// GSRBLAPLACIAN, GSRBHELMHOLTZ).  With deferCopy, a cell with an exchange-copy
// face ghost is left alone (its source box may not be done yet).
template <class T, int VC>
__device__ __forceinline__ void gsrbCell(const BoxDesc& bd, int b, int i, int j, int k, T* phi, const T* rhs,
                                         const Scal& sc, const T* a, const T* b0, const T* b1, const T* b2,
                                         const T* lam, const FaceRule* __restrict__ rules,
                                         const int* __restrict__ faceOff, const GhostCoef& gc, bool deferCopy) {
  const Stencil st = stencil(bd, i, j, k);
  const int64_t c = st.c;
  const int p[3] = {i, j, k};
  const int nb[6] = {st.xp, st.xm, st.yp, st.ym, st.zp, st.zm};
  FaceRule fr[6];
  bool onFace[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const int d = f >> 1, side = (f & 1) ? 0 : 1;  // +d then -d
    onFace[f] = side ? p[d] == bd.hi[d] : p[d] == bd.lo[d];
    if (onFace[f]) {
      const int t0 = d == 0 ? 1 : 0, t1 = d == 2 ? 1 : 2;
      fr[f] = rules[faceOff[6 * b + 2 * d + side] + (p[t0] - bd.lo[t0]) + (bd.hi[t0] - bd.lo[t0] + 1) * (p[t1] - bd.lo[t1])];
      if (deferCopy && fr[f].kind == FR_COPY) return;
    }
  }
  const T pc = phi[c];
  T v[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) v[f] = onFace[f] ? ruleValue(fr[f], pc, phi, gc) : phi[nb[f]];
  const T dxinv = T(sc.dxinv);
  if (VC) {
    T div = b0[st.xp] * (v[0] - pc) - b0[c] * (pc - v[1]) + b1[st.yp] * (v[2] - pc) - b1[c] * (pc - v[3]) +
            b2[st.zp] * (v[4] - pc) - b2[c] * (pc - v[5]);
    T lofphi = T(sc.alpha) * a[c] * pc - T(sc.beta) * div * dxinv;
    phi[c] = pc - lam[c] * (lofphi - rhs[c]);
  } else if (sc.laplacian) {
    T lphi = (v[0] + v[1] + v[2] + v[3] + v[4] + v[5]) * dxinv;
    phi[c] = T(sc.lambda) * (rhs[c] - lphi);
  } else {
    T lphi = ((v[0] + v[1] + v[2] + v[3] + v[4] + v[5]) - T(2.0) * T(3) * pc) * dxinv;
    T helmop = T(sc.alpha) * pc + T(sc.beta) * lphi;
    phi[c] = pc + T(sc.lambda) * (helmop - rhs[c]);
  }
}

// The fused sweep (gsrbSweepFused), first launch: one block per box marching
// through its z slabs.  Step s updates the colour-0 cells of slab s, then
// (after a barrier) the colour-1 cells of slab s - 1 except those with an
// exchange-copy face ghost.  Every read is the value the reference's two
// passes read: a colour-0 cell sees colour-1 neighbours not yet updated (slab
// s - 1 is updated after the barrier, slabs s and s + 1 in later steps, the
// other boxes' face cells only in the second launch), and a colour-1 cell sees
// the new colour-0 values of slabs s - 2 .. s of its own box; its coarse-fine
// and boundary ghosts use only its own box.  Part 2 of a step and part 1 of
// the next touch disjoint cells (slab s - 1 colour 1 against slab s + 1 colour
// 0 and its colour-1 neighbours in slabs s .. s + 2), so one barrier per step
// suffices.  The face coefficients and phi of a slab are read by both colours
// one step apart, from cache.
template <class T, int VC>
__global__ void __launch_bounds__(256) k_gsrb_march(const BoxDesc* boxes, T* phi, const T* rhs, Scal sc,
                                                    const T* a, const T* b0, const T* b1, const T* b2,
                                                    const T* lam, const FaceRule* __restrict__ rules,
                                                    const int* __restrict__ faceOff, GhostCoef gc) {
  const int b = blockIdx.x;
  const BoxDesc bd = boxes[b];
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1, nz = bd.hi[2] - bd.lo[2] + 1;
  const int half = (nx + 1) / 2;
  const int perSlab = half * ny;
  for (int s = 0; s <= nz; ++s) {
    if (s < nz) {
      const int k = bd.lo[2] + s;
      for (int q = threadIdx.x; q < perSlab; q += blockDim.x) {
        const int r = fastDiv(q, half, bd.mHalf);
        const int j = bd.lo[1] + r;
        const int i = bd.lo[0] + ((bd.lo[0] + j + k) & 1) + 2 * (q - r * half);
        if (i <= bd.hi[0]) gsrbCell<T, VC>(bd, b, i, j, k, phi, rhs, sc, a, b0, b1, b2, lam, rules, faceOff, gc, false);
      }
    }
    __syncthreads();
    if (s > 0) {
      const int k = bd.lo[2] + s - 1;
      for (int q = threadIdx.x; q < perSlab; q += blockDim.x) {
        const int r = fastDiv(q, half, bd.mHalf);
        const int j = bd.lo[1] + r;
        const int i = bd.lo[0] + ((bd.lo[0] + j + k + 1) & 1) + 2 * (q - r * half);
        if (i <= bd.hi[0]) gsrbCell<T, VC>(bd, b, i, j, k, phi, rhs, sc, a, b0, b1, b2, lam, rules, faceOff, gc, true);
      }
    }
  }
}

// The fused sweep, second launch: the colour-1 cells with an exchange-copy
// face ghost, now that every box has its new colour-0 values.
template <class T, int VC>
__global__ void __launch_bounds__(256) k_gsrb_deferred(const BoxDesc* boxes, const DeferredCell* cells, int n,
                                                       T* phi, const T* rhs, Scal sc, const T* a, const T* b0,
                                                       const T* b1, const T* b2, const T* lam,
                                                       const FaceRule* __restrict__ rules,
                                                       const int* __restrict__ faceOff, GhostCoef gc) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const DeferredCell dc = cells[t];
  const BoxDesc bd = boxes[dc.box];
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1;
  const int r = fastDiv(dc.q, nx, bd.mNx);
  const int kk = fastDiv(r, ny, bd.mNy);
  gsrbCell<T, VC>(bd, dc.box, bd.lo[0] + (dc.q - r * nx), bd.lo[1] + (r - kk * ny), bd.lo[2] + kk, phi, rhs, sc, a,
                  b0, b1, b2, lam, rules, faceOff, gc, false);
}

template <class T, int VC, int MODE, class O>
__device__ __forceinline__ T opOne(const BoxDesc& bd, int i, int j, int k, O* r, const T* phi, const T* rhs,
                                   const Scal& sc, const T* a, const T* b0, const T* b1, const T* b2) {
  const Stencil s = stencil(bd, i, j, k);
  const T v[6] = {phi[s.xp], phi[s.xm], phi[s.yp], phi[s.ym], phi[s.zp], phi[s.zm]};
  T f[6], av = T(0);
  if (VC) {
    av = a[s.c];
    f[0] = b0[s.xp];
    f[1] = b0[s.c];
    f[2] = b1[s.yp];
    f[3] = b1[s.c];
    f[4] = b2[s.zp];
    f[5] = b2[s.c];
  }
  const T out = opValue<T, VC, MODE>(sc, phi[s.c], MODE == 0 ? rhs[s.c] : T(0), v, av, f);
  r[s.c] = O(out);
  return fabs(out);
}

// v >= 0 or a NaN of either sign (fabs need not clear a NaN's sign bit): the
// IEEE bit pattern of a non-negative double orders like an unsigned integer, so
// an integer max is a floating max, and any NaN (exponent all ones, mantissa
// non-zero) is above every number, infinity included: a NaN anywhere wins.
__device__ __forceinline__ unsigned long long maxBits(double v) { return (unsigned long long)__double_as_longlong(v); }
__device__ __forceinline__ void atomicMaxPos(double* addr, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(addr), maxBits(v));
}

// The largest of a block's values (CHUNK threads) into *out, a running maximum.
// A block that does not exceed it sends no atomic; the comparison is the
// atomic's own (maxBits: as signed integers a NaN whose sign bit is set, such as
// infinity minus infinity gives, would be below every number), so a stale
// running value only costs an atomic.
__device__ __forceinline__ void blockMaxInto(double v, double* out) {
  for (int o = 16; o > 0; o >>= 1) v = nanMax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __shared__ double red[CHUNK / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < CHUNK / 32; ++w) v = nanMax(v, red[w]);
  if (maxBits(v) > maxBits(__ldcg(out))) atomicMaxPos(out, v);
}

// The operator / residual over both colours with two same-row cells per
// thread (as k_gsrb_pair): threads 0-127 take the colour-0 cells of one
// colour chunk, threads 128-255 the colour-1 cells of the chunk with the same
// boundaries, so a block reads both colour halves of the same slots and each
// half finds its neighbours in the other's lines.  opPair returns the largest
// |value| the thread wrote (for the residual's max-norm).
template <class T, int VC, int MODE, class O>
__device__ __forceinline__ T opPair(const BoxDesc* boxes, const Chunk* ch0, const Chunk* ch1, O* r, const T* phi,
                                    const T* rhs, const Scal& sc, const T* a, const T* b0, const T* b1, const T* b2) {
  const int color = threadIdx.x >= CHUNK / 2;
  const Chunk ch = (color ? ch1 : ch0)[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  beginAfterPrevious();
  const int q = ch.start + 2 * (threadIdx.x & (CHUNK / 2 - 1));
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1, nz = bd.hi[2] - bd.lo[2] + 1;
  const int half = (nx + 1) / 2;
  const int rr = fastDiv(q, half, bd.mHalf);
  if (rr >= ny * nz) return T(0);
  const int kk = fastDiv(rr, ny, bd.mNy);
  const int j = bd.lo[1] + (rr - kk * ny), k = bd.lo[2] + kk;
  const int m = q - rr * half;
  const int i = bd.lo[0] + ((bd.lo[0] + j + k + color) & 1) + 2 * m;
  if (m + 1 < half && i + 2 <= bd.hi[0]) {
    const Stencil st = stencil(bd, i, j, k);
    const int c = st.c;
    const T pc0 = phi[c], pc1 = phi[c + 1];
    T rh0 = T(0), rh1 = T(0);
    if (MODE == 0) {
      rh0 = rhs[c];
      rh1 = rhs[c + 1];
    }
    const T xm = phi[st.xm], xc = phi[st.xp], xp = phi[st.xp + 1];
    const T v0[6] = {xc, xm, phi[st.yp], phi[st.ym], phi[st.zp], phi[st.zm]};
    const T v1[6] = {xp, xc, phi[st.yp + 1], phi[st.ym + 1], phi[st.zp + 1], phi[st.zm + 1]};
    T av0 = T(0), av1 = T(0), f0[6], f1[6];
    if (VC) {
      av0 = a[c];
      av1 = a[c + 1];
      f0[0] = b0[st.xp];
      f0[1] = b0[c];
      f0[2] = b1[st.yp];
      f0[3] = b1[c];
      f0[4] = b2[st.zp];
      f0[5] = b2[c];
      f1[0] = b0[st.xp + 1];
      f1[1] = b0[c + 1];
      f1[2] = b1[st.yp + 1];
      f1[3] = b1[c + 1];
      f1[4] = b2[st.zp + 1];
      f1[5] = b2[c + 1];
    }
    const T r0 = opValue<T, VC, MODE>(sc, pc0, rh0, v0, av0, f0), r1 = opValue<T, VC, MODE>(sc, pc1, rh1, v1, av1, f1);
    r[c] = O(r0);
    r[c + 1] = O(r1);
    return nanMax(fabs(r0), fabs(r1));
  }
  T big = T(0);
  if (i <= bd.hi[0]) big = opOne<T, VC, MODE, O>(bd, i, j, k, r, phi, rhs, sc, a, b0, b1, b2);
  int i1, j1, k1;
  if (colorCell(bd, q + 1, color, i1, j1, k1))
    big = nanMax(big, opOne<T, VC, MODE, O>(bd, i1, j1, k1, r, phi, rhs, sc, a, b0, b1, b2));
  return big;
}

template <class T, int VC, int MODE>
__global__ void __launch_bounds__(CHUNK) k_op_pair(const BoxDesc* boxes, const Chunk* ch0, const Chunk* ch1, T* r,
                                                   const T* phi, const T* rhs, Scal sc, const T* a, const T* b0,
                                                   const T* b1, const T* b2) {
  opPair<T, VC, MODE, T>(boxes, ch0, ch1, r, phi, rhs, sc, a, b0, b1, b2);
}

// The residual and its max-norm (k_maxnorm's, over every cell it writes) in one
// pass, which saves reading the residual back: 8 of 32 bytes per cell with
// constant coefficients.  norm[boxHier[box]] in a forest.  O: the type the
// residual is stored in (FP32 for an FP32 cycle; the norm is the unrounded
// values').
template <class T, int VC, class O>
__global__ void __launch_bounds__(CHUNK) k_residual_norm(const BoxDesc* boxes, const Chunk* ch0, const Chunk* ch1, O* r,
                                                         const T* phi, const T* rhs, Scal sc, const T* a, const T* b0,
                                                         const T* b1, const T* b2, const int* boxHier, double* norm) {
  const double v = opPair<T, VC, 0, O>(boxes, ch0, ch1, r, phi, rhs, sc, a, b0, b1, b2);
  blockMaxInto(v, boxHier ? norm + boxHier[ch0[blockIdx.x].box] : norm);
}

// The residual (and NORM: its max-norm, as k_residual_norm) on a uniform level,
// no ghost fill before it: threads 0-127 take colour 0, threads 128-255 colour
// 1 of the same chunk.
template <class T, int VC, bool NORM, class O>
__global__ void __launch_bounds__(CHUNK) k_residual_uniform(const BoxDesc* boxes, const UniformFaces* faces,
                                                            const Chunk* chunks, int n, int per, O* r, const T* phi,
                                                            const T* rhs, Scal sc, const T* a, const T* b0, const T* b1,
                                                            const T* b2, const int* boxHier, double* norm) {
  const int color = threadIdx.x >= CHUNK / 2;
  const int end = min(n, (int)(blockIdx.x + 1) * per);
  double big = 0.0;
  for (int ci = blockIdx.x * per; ci < end; ++ci) {
    const Chunk ch = chunks[ci];
    const BoxDesc bd = boxes[ch.box];
    const UniformFaces uf = faces[ch.box];
    if (ci == (int)blockIdx.x * per) beginAfterPrevious();
    UniformPair p;
    if (!uniformPair(bd, uf, ch.start + 2 * (threadIdx.x & (CHUNK / 2 - 1)), color, p)) continue;
    T pc[2], v0[6], v1[6], f0[6], f1[6], av0 = T(0), av1 = T(0);
    const T rh0 = rhs[p.c], rh1 = rhs[p.c + 1];
    if (VC) {
      av0 = a[p.c];
      av1 = a[p.c + 1];
    }
    uniformLoad<T, VC>(p, uf, phi, b0, b1, b2, pc, v0, v1, f0, f1);
    const T x0 = opValue<T, VC, 0>(sc, pc[0], rh0, v0, av0, f0), x1 = opValue<T, VC, 0>(sc, pc[1], rh1, v1, av1, f1);
    r[p.c] = O(x0);
    r[p.c + 1] = O(x1);
    if (NORM) big = nanMax(big, nanMax((double)fabs(x0), (double)fabs(x1)));
  }
  if (NORM) {
    // forests: one chunk per block, so one hierarchy
    double* out = boxHier ? norm + boxHier[chunks[blockIdx.x * per].box] : norm;
    blockMaxInto(big, out);
  }
}

template <class T>
__global__ void k_negadd(const BoxDesc* boxes, const Chunk* chunks, T* r, const T* lofphi, const T* rhs) {
  Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  int i, j, k;
  if (!allCell(bd, ch.start + threadIdx.x, i, j, k)) return;
  int64_t c = cellIndex(bd, i, j, k);
  r[c] = lofphi[c] * T(-1) + rhs[c] * T(1);
}

template <class T, class X>
__global__ void k_incr(const BoxDesc* boxes, const Chunk* chunks, T* lhs, const X* x, T scale) {
  Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  int i, j, k;
  if (!allCell(bd, ch.start + threadIdx.x, i, j, k)) return;
  int64_t c = cellIndex(bd, i, j, k);
  lhs[c] = lhs[c] + T(x[c]) * scale;
}

// lhs += x * scale and r = -lofphi + rhs over whole level arrays, ghost and
// padding slots included: the valid cells get exactly the reference's
// values, the ghost slots of these fields are rewritten by a ghost fill or
// coarse-fine interpolation before anything reads them, and one flat,
// perfectly coalesced loop beats walking the valid cells box by box.
template <class T, class X>
__global__ void k_incr_flat(T* lhs, const X* x, T scale, int64_t n) {
  beginAfterPrevious();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    lhs[q] = lhs[q] + T(x[q]) * scale;
}
template <class T>
__global__ void k_negadd_flat(T* r, const T* lofphi, const T* rhs, int64_t n) {
  beginAfterPrevious();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    r[q] = lofphi[q] * T(-1) + rhs[q] * T(1);
}
// Chunks per block on a uniform level: more once the grid holds several waves
// of blocks anyway.
inline int uniformPer(int chunks) { return std::max(1, std::min(4, chunks / (148 * 32))); }

inline int flatBlocks(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 148 * 16); }

// x *= s over a whole level array (LevelDataOps::scale -> FArrayBox::mult).
__global__ void k_scale_flat(double* x, double s, int64_t n) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    x[q] = x[q] * s;
}

// Per-box dot products in the reference's order: FArrayBox::dotProduct
// (BoxTools/FArrayBox.cpp:260-280) accumulates x*y over the valid box k, j, i
// with i fastest into one running sum; the sum over boxes and levels is left
// to the caller (LevelDataOps::dotProduct, MultilevelLinearOp::dotProduct).
// One block per box of every level, one or two products at a time (x1.y1 and
// x2.y2): the block's threads load and multiply a chunk of DOT_CHUNK cells
// into shared memory (a product rounds the same whoever forms it) while one
// thread per product adds the chunk before, in order.  Cells whose mask is 0
// (under a finer level) count as zero, as in the reference's zeroed copies.
// Bound by the chain of dependent adds of the largest box (32,768 adds of a
// 32^3 box): the adding threads read ahead of the chain in registers, which
// takes DOT_ADD adds per 16-byte-load group, and all levels and both products
// run side by side.  A dependent FP64 add takes 8.2 cycles here, so a 32^3
// box cannot take less than 0.14 ms; one warp per box, one level and one
// product per launch took 0.36 ms each.  Three-level 64^3 BiCGStab solve: 93.5
// -> 61.6 ms.  A chunk's tail is filled with +0 products, added up to the next
// multiple of DOT_ADD: a sum that starts at +0 is never -0, so adding +0 leaves it
// as it is.  (Adding whole chunks cost boxes of a few cells 4 us a product.)
enum { DOT_THREADS = 128, DOT_PER_THREAD = 8, DOT_CHUNK = DOT_THREADS * DOT_PER_THREAD, DOT_ADD = 16 };

__device__ __forceinline__ double addChunk(double s, const double* p, int m) {
  const double2* v = reinterpret_cast<const double2*>(p);
  double2 cur[DOT_ADD / 2], nxt[DOT_ADD / 2];
#pragma unroll
  for (int u = 0; u < DOT_ADD / 2; ++u) cur[u] = v[u];
  for (int base = 0; base < m; base += DOT_ADD) {
    const int n = base + DOT_ADD < m ? base + DOT_ADD : 0;  // the last read-ahead is not used
#pragma unroll
    for (int u = 0; u < DOT_ADD / 2; ++u) nxt[u] = v[n / 2 + u];
#pragma unroll
    for (int u = 0; u < DOT_ADD / 2; ++u) {
      s += cur[u].x;
      s += cur[u].y;
    }
#pragma unroll
    for (int u = 0; u < DOT_ADD / 2; ++u) cur[u] = nxt[u];
  }
  return s;
}

template <bool TWO>
__global__ void __launch_bounds__(DOT_THREADS) k_box_dot(DotLevels D, double* out1, double* out2) {
  __shared__ __align__(16) double prod[2][TWO ? 2 : 1][DOT_CHUNK];
  int l = 0;
  while (l + 1 < D.n && (int)blockIdx.x >= D.lev[l + 1].first) ++l;
  const DotLevel& L = D.lev[l];
  const BoxDesc bd = L.boxes[blockIdx.x - L.first];
  const double *x1 = L.x1, *y1 = L.y1, *x2 = L.x2, *y2 = L.y2;
  const unsigned char* mask = L.mask;
  const int nx = bd.hi[0] - bd.lo[0] + 1, ny = bd.hi[1] - bd.lo[1] + 1, nz = bd.hi[2] - bd.lo[2] + 1;
  const int n = nx * ny * nz, tid = threadIdx.x;
  double a1[DOT_PER_THREAD], b1[DOT_PER_THREAD], a2[DOT_PER_THREAD], b2[DOT_PER_THREAD];
  unsigned char on[DOT_PER_THREAD];
  // Loads of one chunk into registers (issued, not waited for).
  auto issue = [&](int base) {
#pragma unroll
    for (int u = 0; u < DOT_PER_THREAD; ++u) {
      const int q = base + tid + DOT_THREADS * u;
      on[u] = 0;
      a1[u] = b1[u] = a2[u] = b2[u] = 0.0;
      int i, j, k;
      if (q < n && allCell(bd, q, i, j, k)) {
        const int64_t c = cellIndex(bd, i, j, k);
        on[u] = mask ? mask[c] : 1;
        a1[u] = x1[c];
        b1[u] = y1[c];
        if (TWO) {
          a2[u] = x2[c];
          b2[u] = y2[c];
        }
      }
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int u = 0; u < DOT_PER_THREAD; ++u) {
      prod[buf][0][tid + DOT_THREADS * u] = on[u] ? a1[u] * b1[u] : 0.0;
      if (TWO) prod[buf][TWO ? 1 : 0][tid + DOT_THREADS * u] = on[u] ? a2[u] * b2[u] : 0.0;
    }
  };
  double s = 0.0;
  issue(0);
  store(0);
  __syncthreads();
  for (int base = 0, buf = 0; base < n; base += DOT_CHUNK, buf ^= 1) {
    // the next chunk's loads are in flight while this one is added
    const bool more = base + DOT_CHUNK < n;
    if (more) issue(base + DOT_CHUNK);
    const int m = min(n - base, (int)DOT_CHUNK);
    if (tid == 0) s = addChunk(s, prod[buf][0], m);
    if (TWO && tid == 32) s = addChunk(s, prod[buf][TWO ? 1 : 0], m);
    if (more) store(buf ^ 1);
    __syncthreads();
  }
  if (tid == 0) out1[blockIdx.x] = s;
  if (TWO && tid == 32) out2[blockIdx.x] = s;
}

// dst = src over whole arrays (ghosts included), converting the type.
template <class D, class S>
__global__ void k_convert(D* dst, const S* src, int64_t n) {
  beginAfterPrevious();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    dst[q] = D(src[q]);
}

template <class T>
__global__ void k_maxnorm(const BoxDesc* boxes, const Chunk* chunks, int nchunks, const T* f,
                          const unsigned char* mask, double* out) {
  beginAfterPrevious();
  // Blocks stride over the chunks (one chunk each when the grid covers
  // them), so a large level sends one atomic per block, not per chunk.
  // Up to four chunks per step, their table loads and values issued
  // together (the max does not depend on the order).
  double v = 0.0;
  for (int c0 = blockIdx.x; c0 < nchunks; c0 += 4 * gridDim.x) {
    int64_t at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      at[u] = -1;
      const int cix = c0 + u * gridDim.x;
      if (cix >= nchunks) continue;
      const Chunk ch = chunks[cix];
      const BoxDesc bd = boxes[ch.box];
      int i, j, k;
      if (allCell(bd, ch.start + threadIdx.x, i, j, k)) {
        const int64_t c = cellIndex(bd, i, j, k);
        if (!mask || mask[c]) at[u] = c;
      }
    }
    double x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = at[u] >= 0 ? fabs((double)f[at[u]]) : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u) v = nanMax(v, x[u]);
  }
  for (int o = 16; o > 0; o >>= 1) v = nanMax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __shared__ double red[CHUNK / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < CHUNK / 32 ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v = nanMax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) atomicMaxPos(out, fabs(v));
  }
}

// The max-norm of a forest level, one chunk per block, folded into the
// norm of the chunk's hierarchy.
template <class T>
__global__ void k_maxnorm_hier(const BoxDesc* boxes, const Chunk* chunks, const int* boxHier, const T* f,
                               double* out) {
  const Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  beginAfterPrevious();
  double v = 0.0;
  int i, j, k;
  if (allCell(bd, ch.start + threadIdx.x, i, j, k)) v = fabs((double)f[cellIndex(bd, i, j, k)]);
  for (int o = 16; o > 0; o >>= 1) v = nanMax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __shared__ double red[CHUNK / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < CHUNK / 32 ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v = nanMax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) atomicMaxPos(out + boxHier[ch.box], fabs(v));
  }
}

// lhs += x over hierarchy blockIdx.y's element range of a forest level, if
// that hierarchy is still iterating (k_incr_flat's arithmetic).
template <class T, class X>
__global__ void k_incr_active(T* lhs, const X* x, const int64_t* hierStart, const int* active) {
  beginAfterPrevious();
  const int h = blockIdx.y;
  if (!active[h]) return;
  const int64_t a = hierStart[h], b = hierStart[h + 1];
  for (int64_t q = a + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < b; q += (int64_t)gridDim.x * blockDim.x)
    lhs[q] = lhs[q] + T(x[q]) * T(1.0);
}

// RESTRICTRES / RESTRICTRESVC3D (AMRPoissonOpF.ChF:394-438,
// VCAMRPoissonOpF.ChF:337-413): res_c accumulates (rhs - L phi)/8 over its 8
// fine cells in fine k-j-i order, starting from zero.
template <class T, int VC>
__global__ void k_restrictmg(const BoxDesc* fboxes, const BoxDesc* cboxes, const Chunk* chunks, T* resC,
                             const T* phi, const T* rhs, Scal sc, const T* a, const T* b0, const T* b1,
                             const T* b2) {
  Chunk ch = chunks[blockIdx.x];
  const BoxDesc cb = cboxes[ch.box];
  beginAfterPrevious();
  int I, J, K;
  if (!allCell(cb, ch.start + threadIdx.x, I, J, K)) return;
  const BoxDesc fb = fboxes[ch.box];
  const T dxinv = T(sc.dxinv);
  const T denom = T(8);
  T acc = T(0);
  for (int kk = 0; kk < 2; ++kk)
    for (int jj = 0; jj < 2; ++jj)
      for (int ii = 0; ii < 2; ++ii) {
        const Stencil st = stencil(fb, 2 * I + ii, 2 * J + jj, 2 * K + kk);
        const int64_t c = st.c;
        T pc = phi[c];
        T lofphi;
        if (VC)
          lofphi = T(sc.alpha) * a[c] * pc - T(sc.beta) * vcDiv(phi, b0, b1, b2, st) * dxinv;
        else
          lofphi = T(sc.alpha) * pc + T(sc.beta) * (nbrSum(phi, st) - pc * T(2) * T(3)) * dxinv;
        acc = acc + (rhs[c] - lofphi) / denom;
      }
  resC[cellIndex(cb, I, J, K)] = acc;
}

// k_restrictmg on a uniform level, no ghost fill before it: a thread's eight
// fine cells and the 24 around them are each read once (56 reads cell by cell),
// those beyond a face where their value is (UniformFaces).
template <class T, int VC>
__global__ void __launch_bounds__(CHUNK) k_restrict_uniform(const BoxDesc* fboxes, const UniformFaces* faces,
                                                            const BoxDesc* cboxes, const Chunk* chunks, T* resC,
                                                            const T* phi, const T* rhs, Scal sc, const T* a, const T* b0,
                                                            const T* b1, const T* b2) {
  const Chunk ch = chunks[blockIdx.x];
  const BoxDesc cb = cboxes[ch.box], fb = fboxes[ch.box];
  const UniformFaces uf = faces[ch.box];
  beginAfterPrevious();
  int I, J, K;
  if (!allCell(cb, ch.start + threadIdx.x, I, J, K)) return;
  const int x0 = 2 * I - fb.lo[0], y0 = 2 * J - fb.lo[1], z0 = 2 * K - fb.lo[2];  // the first fine cell in its box
  const int nx = fb.hi[0] - fb.lo[0] + 1, ny = fb.hi[1] - fb.lo[1] + 1, nz = fb.hi[2] - fb.lo[2] + 1;
  const int sy = fb.px >> 1, sz = sy * fb.py, par = fb.lo[0] + fb.lo[1] + fb.lo[2] + x0 + y0 + z0;
  // element of cell (x0 + x, y0 + y, z0 + z)
  auto at = [&](int x, int y, int z) {
    return (int)fb.off + ((par + x + y + z) & 1) * (int)fb.half + ((x0 + x + 1) >> 1) + sy * (y0 + y + 1) +
           sz * (z0 + z + 1);
  };
  const bool lx = x0 == 0, hx = x0 + 2 == nx, ly = y0 == 0, hy = y0 + 2 == ny, lz = z0 == 0, hz = z0 + 2 == nz;
  T in[2][2][2], xm[2][2], xp[2][2], ym[2][2], yp[2][2], zm[2][2], zp[2][2];  // [z][y][x], outer ones [.][.]
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int u = q & 1, v = q >> 1;
    in[v][u][0] = phi[at(0, u, v)];
    in[v][u][1] = phi[at(1, u, v)];
    xm[v][u] = phi[at(-1, u, v) + (lx ? uf.d[0] : 0)];
    xp[v][u] = phi[at(2, u, v) + (hx ? uf.d[1] : 0)];
    ym[v][u] = phi[at(u, -1, v) + (ly ? uf.d[2] : 0)];
    yp[v][u] = phi[at(u, 2, v) + (hy ? uf.d[3] : 0)];
    zm[v][u] = phi[at(u, v, -1) + (lz ? uf.d[4] : 0)];
    zp[v][u] = phi[at(u, v, 2) + (hz ? uf.d[5] : 0)];
  }
  if (uf.kind) {
    auto wall = [&](bool on, int face, T& v, T x) {
      const int k = uf.kind >> (2 * face) & 3;
      if (on && k) v = k == 1 ? T(0) - x : x;
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int u = q & 1, v = q >> 1;
      wall(lx, 0, xm[v][u], in[v][u][0]);
      wall(hx, 1, xp[v][u], in[v][u][1]);
      wall(ly, 2, ym[v][u], in[v][0][u]);
      wall(hy, 3, yp[v][u], in[v][1][u]);
      wall(lz, 4, zm[v][u], in[0][v][u]);
      wall(hz, 5, zp[v][u], in[1][v][u]);
    }
  }
  const T dxinv = T(sc.dxinv);
  T acc = T(0);
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const int x = n & 1, y = (n >> 1) & 1, z = n >> 2;
    const T pc = in[z][y][x];
    const T v[6] = {x ? xp[z][y] : in[z][y][1], x ? in[z][y][0] : xm[z][y], y ? yp[z][x] : in[z][1][x],
                    y ? in[z][0][x] : ym[z][x], z ? zp[y][x] : in[1][y][x], z ? in[0][y][x] : zm[y][x]};
    const int c = at(x, y, z);
    T lofphi;
    if (VC) {
      const T div = b0[at(x + 1, y, z)] * (v[0] - pc) - b0[c] * (pc - v[1]) + b1[at(x, y + 1, z)] * (v[2] - pc) -
                    b1[c] * (pc - v[3]) + b2[at(x, y, z + 1)] * (v[4] - pc) - b2[c] * (pc - v[5]);
      lofphi = T(sc.alpha) * a[c] * pc - T(sc.beta) * div * dxinv;
    } else {
      lofphi = T(sc.alpha) * pc + T(sc.beta) * ((v[0] + v[1] + v[2] + v[3] + v[4] + v[5]) - pc * T(2) * T(3)) * dxinv;
    }
    acc = acc + (rhs[c] - lofphi) / T(8);
  }
  resC[cellIndex(cb, I, J, K)] = acc;
}

// PROLONG (AMRPoissonOpF.ChF:453-478): phi += coarse(i/2), same box index.  One
// thread per coarse cell updates its eight fine cells, as k_prolongamr does.
template <class T>
__global__ void k_prolongmg(const BoxDesc* fboxes, const BoxDesc* cboxes, const Chunk* chunks, T* phi,
                            const T* corrC) {
  Chunk ch = chunks[blockIdx.x];
  const BoxDesc cb = cboxes[ch.box], fb = fboxes[ch.box];
  beginAfterPrevious();
  int I, J, K;
  if (!allCell(cb, ch.start + threadIdx.x, I, J, K)) return;
  const T c = corrC[cellIndex(cb, I, J, K)];
  int f[8];
  T v[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) f[n] = (int)cellIndex(fb, 2 * I + (n & 1), 2 * J + ((n >> 1) & 1), 2 * K + (n >> 2));
#pragma unroll
  for (int n = 0; n < 8; ++n) v[n] = phi[f[n]];
#pragma unroll
  for (int n = 0; n < 8; ++n) phi[f[n]] = v[n] + c;
}

// AVERAGE with refRatio 2 (AverageF.ChF:36-55) written straight into the
// coarse level through the coarsened-fine -> coarse copy items.
template <class T>
__global__ void k_average(const BoxDesc* fboxes, const BoxDesc* cboxes, const CoarseFineItem* items,
                          const Chunk* chunks, T* coarse, const T* fine) {
  Chunk ch = chunks[blockIdx.x];
  const CoarseFineItem it = items[ch.box];
  const BoxDesc fb = fboxes[it.fbox], cb = cboxes[it.cbox];
  int q = ch.start + threadIdx.x;
  int nx = it.hi[0] - it.lo[0] + 1, ny = it.hi[1] - it.lo[1] + 1, nz = it.hi[2] - it.lo[2] + 1;
  int I = it.lo[0] + q % nx, r = q / nx, J = it.lo[1] + r % ny, K = it.lo[2] + r / ny;
  beginAfterPrevious();
  if (q >= nx * ny * nz) return;
  const int i = 2 * I, j = 2 * J, k = 2 * K;
  T sum = fine[cellIndex(fb, i, j, k)] + fine[cellIndex(fb, i + 1, j, k)] + fine[cellIndex(fb, i, j + 1, k)] +
          fine[cellIndex(fb, i + 1, j + 1, k)] + fine[cellIndex(fb, i, j, k + 1)] +
          fine[cellIndex(fb, i + 1, j, k + 1)] + fine[cellIndex(fb, i, j + 1, k + 1)] +
          fine[cellIndex(fb, i + 1, j + 1, k + 1)];
  coarse[cellIndex(cb, I, J, K)] = T(0.125) * sum;
}

// AMRProlongS (AMRPoissonOp.cpp:959-990): fine += coarse(i/2).  One thread
// per coarse cell of an item (chunks over the items' coarse cells, x
// fastest) updates its eight fine cells: the coarse value is read once, the
// eight fine loads are independent, and for each of the eight child offsets
// a warp's threads touch consecutive slots of one colour half.
template <class T>
__global__ void k_prolongamr(const BoxDesc* fboxes, const BoxDesc* cboxes, const CoarseFineItem* items,
                             const Chunk* chunks, T* fine, const T* coarse) {
  Chunk ch = chunks[blockIdx.x];
  const CoarseFineItem it = items[ch.box];
  const BoxDesc fb = fboxes[it.fbox], cb = cboxes[it.cbox];
  const int q = ch.start + threadIdx.x;
  const int nx = it.hi[0] - it.lo[0] + 1, ny = it.hi[1] - it.lo[1] + 1, nz = it.hi[2] - it.lo[2] + 1;
  const int r = q / nx, kk = r / ny;
  const int I = it.lo[0] + (q - r * nx), J = it.lo[1] + (r - kk * ny), K = it.lo[2] + kk;
  beginAfterPrevious();
  if (q >= nx * ny * nz) return;
  const T c = coarse[cellIndex(cb, I, J, K)];
  int64_t f[8];
  T v[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) f[n] = cellIndex(fb, 2 * I + (n & 1), 2 * J + ((n >> 1) & 1), 2 * K + (n >> 2));
#pragma unroll
  for (int n = 0; n < 8; ++n) v[n] = fine[f[n]];
#pragma unroll
  for (int n = 0; n < 8; ++n) fine[f[n]] = v[n] + c;
}

// lhs = lhs + x * 1 (k_incr_flat's arithmetic), then x = the new lhs: the
// increment followed by a copy back, in one pass.
template <class T>
__global__ void k_incr_copy_flat(T* lhs, T* x, int64_t n) {
  beginAfterPrevious();
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    const T v = lhs[q] + x[q] * T(1.0);
    lhs[q] = v;
    x[q] = v;
  }
}

// lhs += x + y (k_incr_copy_flat's sum, then k_incr_flat's) over hierarchy
// blockIdx.y's elements, if it is still iterating (hierStart null: every one).
// Bound by DRAM: four arrays touched once, where the copy and the increment it
// stands for touch seven.
template <class T, class X>
__global__ void k_incr_sum(T* lhs, const X* x, const X* y, int64_t n, const int64_t* hierStart, const int* active) {
  beginAfterPrevious();
  int64_t a = 0, b = n;
  if (hierStart) {
    if (!active[blockIdx.y]) return;
    a = hierStart[blockIdx.y];
    b = hierStart[blockIdx.y + 1];
  }
  for (int64_t q = a + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < b; q += (int64_t)gridDim.x * blockDim.x)
    lhs[q] = lhs[q] + T(x[q] + y[q] * X(1.0)) * T(1.0);
}

// QuadCFStencil derivatives (AMRTools/QuadCFStencil.cpp:33-260).
template <class T>
__device__ __forceinline__ T cfFirst(const CFDeriv& d, const double* w, const int64_t* off, const T* pc, T dxc) {
  if (d.kind == 1) return (pc[off[d.start + 1]] - pc[off[d.start]]) / (T(2.0) * dxc);
  if (d.kind == 0) return T(0);
  T v = T(0);
  for (int n = 0; n < d.n; ++n) v += T(w[d.start + n]) * pc[off[d.start + n]];
  return v / dxc;
}
template <class T>
__device__ __forceinline__ T cfSecond(const CFDeriv& d, const double* w, const int64_t* off, const T* pc, T dxc) {
  if (d.kind == 1)
    return (pc[off[d.start + 1]] + pc[off[d.start]] - T(2.0) * pc[off[d.start + 2]]) / (dxc * dxc);
  if (d.kind == 0) return T(0);
  T v = T(0);
  for (int n = 0; n < d.n; ++n) v += T(w[d.start + n]) * pc[off[d.start + n]];
  return v / (dxc * dxc);
}
template <class T>
__device__ __forceinline__ T cfMixed(const CFDeriv& d, const double* w, const int64_t* off, const T* pc, T dxc) {
  if (d.kind == 1) {
    const int64_t* o = off + d.start;  // ur, ul, lr, ll
    return (pc[o[0]] + pc[o[3]] - pc[o[2]] - pc[o[1]]) / (T(4.) * dxc * dxc);
  }
  if (d.kind == 0) return T(0);
  T v = T(0);
  for (int n = 0; n < d.n; ++n) v += T(w[d.start + n]) * pc[off[d.start + n]];
  return v / (dxc * dxc);
}

// QuadCFInterp::getPhiStar + interpOnIVS (AMRTools/QuadCFInterp.cpp:569-839),
// in two launches.  First, per coarse cell under a coarse-fine face: the
// tangential first and second derivatives, the mixed derivative and the
// coarse value (six values into tmp); every fine ghost over that coarse cell
// (four on a face) reads them instead of gathering the stencils again.  A warp
// takes one of the six values of 32 coarse cells: each is a chain of three
// dependent loads (stencil, offsets, cells), and one thread for all six paid the
// chains one after the other.  The stencil is read before the wait for the
// previous kernel, as are the tables of the interpolation, the flux correction,
// the average and the prolongation below: heat steps 8.84 -> 8.10 ms, two-level
// 64^3 VC solve 3.90 -> 3.66, BiCGStab with three levels 46.8 -> 44.4.
template <class T>
__global__ void __launch_bounds__(192) k_cf_coarse(const CFCoarse* __restrict__ coarse, int n,
                                                   const double* __restrict__ w, const int64_t* __restrict__ off,
                                                   const T* phiC, T h, T* tmp) {
  const int t = blockIdx.x * 32 + (threadIdx.x & 31), v = threadIdx.x >> 5;
  const bool in = t < n;
  CFDeriv d = {};
  int64_t cc = 0;
  if (in && v < 5) d = v == 4 ? coarse[t].mx : (v & 1) ? coarse[t].d2[v >> 1] : coarse[t].d1[v >> 1];
  if (in && v == 5) cc = coarse[t].cc;
  beginAfterPrevious();
  if (!in) return;
  const T dxc = T(2) * h;
  T x;
  if (v == 5)
    x = phiC[cc];
  else if (v == 4)
    x = cfMixed(d, w, off, phiC, dxc);
  else if (v & 1)
    x = cfSecond(d, w, off, phiC, dxc);
  else
    x = cfFirst(d, w, off, phiC, dxc);
  tmp[6 * (int64_t)t + v] = x;
}

// Second, per fine ghost: phistar from the coarse Taylor expansion, then the
// quadratic through phistar and two fine cells, in the Fortran (packed face,
// QuadCFInterpF.ChF:9-48) or C++ (unpacked face) arithmetic.
// tmp == nullptr: the coarse data are zero (six zeros per coarse cell).
template <class T>
__global__ void k_quadcf(const CFFine* __restrict__ fine, int n, const T* tmp, T* phiF, T h) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  CFFine e = {};
  if (t < n) e = fine[t];
  beginAfterPrevious();
  if (t >= n) return;
  T s1 = T(0), c1 = T(0), s2 = T(0), c2 = T(0), mx = T(0), pc = T(0);
  if (tmp) {
    const T* c = tmp + 6 * (int64_t)e.coarse;
    s1 = c[0], c1 = c[1], s2 = c[2], c2 = c[3], mx = c[4], pc = c[5];
  }
  const T x1 = T(e.x1), x2 = T(e.x2);
  T update1 = x1 * s1 + T(0.5) * x1 * x1 * c1;
  T update2 = x2 * s2 + T(0.5) * x2 * x2 * c2;
  T update3 = x1 * x2 * mx;
  T ps = pc + update1 + update2 + update3;
  T pa = phiF[e.pa], pb = phiF[e.pb];
  T r;
  if (e.packed) {
    T frac = T(2.0) / (h * h);
    T denom = T(2 * 2 + 4 * 2 + 3);
    T mult = frac / denom;
    T invh = T(1.0) / h;
    T x = T(2.0) * h;
    T xsq = T(4.0) * h * h;
    T a = mult * (T(2.0) * ps + T(2 + 1) * pa - T(2 + 3) * pb);
    T b = (pb - pa) * invh - a * h;
    r = xsq * a + b * x + pa;
  } else {
    T a = (T(2.) / h / h) * (T(2.) * ps + pa * (T(2) + T(1.0)) - pb * (T(2) + T(3.0))) / (T(2 * 2 + 4 * 2) + T(3.0));
    T b = (pb - pa) / h - a * h;
    T x = T(2.) * h;
    r = a * x * x + b * x + pa;
  }
  phiF[e.g] = r;
}

// Flux-register correction (AMRPoissonOp::reflux, VCAMRPoissonOp2::reflux
// and LevelFluxRegister incrementCoarse/incrementFine/reflux).  phiC null: the
// coarse field is zero and lofphi holds a right-hand side, which becomes the
// residual: the corrected L(0) times -1 plus it, as k_negadd adds them.
template <class T, int VC>
__global__ void k_reflux(const RefluxCell* __restrict__ cells, int n, const RefluxCoarseTerm* __restrict__ cterms,
                         const RefluxFineGroup* __restrict__ fgroups,
                         T* lofphi, const T* phiC, const T* phiF, const T* bc0, const T* bc1, const T* bc2,
                         const T* bf0, const T* bf1, const T* bf2, T sc, T sf, T negs) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  RefluxCell rc = {};
  RefluxCoarseTerm ct = {};
  RefluxFineGroup g = {};
  if (t < n) {
    rc = cells[t];
    if (phiC && rc.nco > 0) ct = cterms[rc.start];
    if (rc.nfi > 0) g = fgroups[rc.fstart];
  }
  beginAfterPrevious();
  if (t >= n) return;
  auto dirOf = [](int d, const T* x, const T* y, const T* z) { return d == 0 ? x : d == 1 ? y : z; };
  T u = phiC ? lofphi[rc.c] : T(0);
  T coar = T(0);
  for (int m = 0; phiC && m < rc.nco; ++m) {
    if (m > 0) ct = cterms[rc.start + m];
    T flux;
    if (VC)
      flux = -dirOf(ct.dir, bc0, bc1, bc2)[ct.bface] * ((phiC[ct.hi] - phiC[ct.lo]) * sc);
    else
      flux = (phiC[ct.hi] - phiC[ct.lo]) * sc;
    coar = coar + flux * T(ct.sgn);
  }
  u = u + coar * negs;
  for (int m = 0; m < rc.nfi; ++m) {
    if (m > 0) g = fgroups[rc.fstart + m];
    T ff[4], reg = T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (VC)
        ff[q] = -dirOf(g.dir, bf0, bf1, bf2)[g.bface[q]] * ((phiF[g.hi[q]] - phiF[g.lo[q]]) * sf);
      else
        ff[q] = (phiF[g.hi[q]] - phiF[g.lo[q]]) * sf;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) reg = reg + T(g.scale) * ff[q];
    u = u + reg * negs;
  }
  lofphi[rc.c] = phiC ? u : u * T(-1) + lofphi[rc.c] * T(1);
}

// One block per hierarchy of the level: block k solves with works[k] and
// metrics[k], the rest of the arguments shared.
__global__ void __launch_bounds__(1024) k_bottom(BottomArgs A0, const BottomWork* works, const double* metrics) {
  extern __shared__ double spart[];
  __shared__ double scal[8];
  BottomArgs A = A0;
  A.W = works[blockIdx.x];
  A.metric = metrics + blockIdx.x;
  if (A0.epsPer && A0.cfg.kind == 0) A.eps = A0.epsPer[blockIdx.x];
  BlkCtx c;
  c.part = spart;
  c.part2 = spart + max(A.W.nbox, 32);
  c.scal = scal;
  c.k = 0;
  bottomRun(c, A);
}

// One hierarchy, the whole grid (cooperative launch).
__global__ void __launch_bounds__(kBottomGridThreads) k_bottom_grid(BottomArgs A, const BottomWork* works,
                                                                    const double* metrics) {
  __shared__ double stage[2 * kBottomStage];
  A.W = works[0];
  A.metric = metrics;
  if (A.epsPer && A.cfg.kind == 0) A.eps = A.epsPer[0];
  GridCtx c;
  c.part = A.W.gpart;
  c.part2 = A.W.gpart2;
  c.scal = A.W.gscal;
  c.stage = stage;
  c.k = 0;
  bottomRun(c, A);
}

__global__ void k_gather_slots(const int* fab, int n, const double* src, double* dst) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) dst[q] = src[fab[q]];
}

}  // namespace

}  // namespace cmg

namespace cmg {

template <class T>
void ghostFill(const LevelDev& L, T* f, bool withCF, cudaStream_t s, int par) {
  auto range = [&](int p, int& r0, int& r1) {
    r0 = L.gcStart[p];
    r1 = r0 + L.gcExch[p] + (withCF ? L.gcCF[p] : 0);
  };
  int a0, a1, b0 = 0, b1 = 0;
  range(par >= 0 ? par : 0, a0, a1);
  if (par < 0) range(1, b0, b1);
  const int n = (a1 - a0) + (b1 - b0);
  if (n == 0) return;
  const double dx = L.dx, dxc = L.dxCrse;
  T c1 = T(2 * (dxc - dx) / (dxc + dx));
  T c2 = T(-(dxc - dx) / (dxc + 3 * dx));
  T flin = T(1 - 2 * dx / (dx + dxc));
  // Four entries per thread once the fill exceeds one wave of resident
  // threads (148 SMs x 2048), one per thread below that.
  if (n > 148 * 2048) {
    constexpr int U = 4;
    launchNext(k_ghostcells<T, U>, (n + GHOST_THREADS * U - 1) / (GHOST_THREADS * U), GHOST_THREADS, s, L.gcells, a0,
               a1, b0, b1, f, c1, c2, flin);
  } else {
    launchNext(k_ghostcells<T, 1>, (n + GHOST_THREADS - 1) / GHOST_THREADS, GHOST_THREADS, s, L.gcells, a0, a1, b0, b1,
               f, c1, c2, flin);
  }
  CMG_LAUNCHED("ghostFill");
}

// BackwardEuler::createEulerRHS (BackwardEuler.cpp:190-226) over whole
// arrays: rhs = ((0 + phi) * a) + ((0 + src) * dt), a omitted for the
// constant-coefficient operator (its diagonalScale is a no-op).
__global__ void k_euler_rhs(double* rhs, const double* phi, const double* a, const double* src, double dt,
                            int64_t n) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double v = 0.0 + phi[q];
    if (a) v = v * a[q];
    double w = 0.0 + src[q];
    w = w * dt;
    rhs[q] = v + w;
  }
}

// AMRTGA::oneStep's source term: (0 + src * 1) / a (setToZero, incr,
// divideByIdentityCoef; no division for the constant-coefficient operator).
__global__ void k_tga_source(double* out, const double* src, const double* a, int64_t n) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
    double v = 0.0 + src[q] * 1.0;
    if (a) v = v / a[q];
    out[q] = v;
  }
}

// x *= a (FArrayBox::mult by a FAB: the VC operator's diagonalScale).
__global__ void k_mult_field(double* x, const double* a, int64_t n) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    x[q] = x[q] * a[q];
}

void tgaSource(double* out, const double* src, const double* a, int64_t n, cudaStream_t s) {
  if (n == 0) return;
  k_tga_source<<<flatBlocks(n), 256, 0, s>>>(out, src, a, n);
  CMG_LAUNCHED("tgaSource");
}

void multField(double* x, const double* a, int64_t n, cudaStream_t s) {
  if (n == 0) return;
  k_mult_field<<<flatBlocks(n), 256, 0, s>>>(x, a, n);
  CMG_LAUNCHED("multField");
}

void eulerRHS(double* rhs, const double* phi, const double* a, const double* src, double dt, int64_t n,
              cudaStream_t s) {
  if (n == 0) return;
  k_euler_rhs<<<flatBlocks(n), 256, 0, s>>>(rhs, phi, a, src, dt, n);
  CMG_LAUNCHED("eulerRHS");
}

void scaleField(double* x, double scale, int64_t n, cudaStream_t s) {
  if (n == 0) return;
  k_scale_flat<<<flatBlocks(n), 256, 0, s>>>(x, scale, n);
  CMG_LAUNCHED("scale");
}

void boxDots(const DotLevel* lev, int nlev, int nbox, bool two, double* out1, double* out2, cudaStream_t s) {
  // kernel arguments hold kDotLevels levels; deeper hierarchies take more launches
  for (int l0 = 0; l0 < nlev; l0 += kDotLevels) {
    DotLevels D;
    D.n = std::min(nlev - l0, (int)kDotLevels);
    const int b0 = lev[l0].first, b1 = l0 + D.n < nlev ? lev[l0 + D.n].first : nbox;
    if (b1 == b0) continue;
    for (int l = 0; l < D.n; ++l) {
      D.lev[l] = lev[l0 + l];
      D.lev[l].first -= b0;
    }
    if (two)
      k_box_dot<true><<<b1 - b0, DOT_THREADS, 0, s>>>(D, out1 + b0, out2 + b0);
    else
      k_box_dot<false><<<b1 - b0, DOT_THREADS, 0, s>>>(D, out1 + b0, nullptr);
    CMG_LAUNCHED("boxDots");
  }
}

void boxDots(const LevelDev& L, const double* x, const double* y, double* out, cudaStream_t s) {
  const DotLevel one{L.boxes, x, y, nullptr, nullptr, nullptr, 0};
  boxDots(&one, 1, L.nbox, false, out, nullptr, s);
}

void coveredMask(const LevelDev& L, unsigned char* mask, cudaStream_t s) {
  check(cudaMemsetAsync(mask, 1, L.nelem, s), "mask");
  if (L.nZero == 0) return;
  launchNext(k_ghost<unsigned char>, (L.nCellsZero + GHOST_PER_BLOCK - 1) / GHOST_PER_BLOCK, GHOST_THREADS, s, L.zero,
             L.zeroStart, L.zeroBlock, L.nZero, L.nCellsZero, -1, mask, 0, 0, 0);
  CMG_LAUNCHED("coveredMask");
}

template <class T>
void zeroCovered(const LevelDev& L, T* f, cudaStream_t s) {
  if (L.nZero == 0) return;
  launchNext(k_ghost<T>, (L.nCellsZero + GHOST_PER_BLOCK - 1) / GHOST_PER_BLOCK, GHOST_THREADS, s, L.zero, L.zeroStart,
             L.zeroBlock, L.nZero, L.nCellsZero, -1, f, T(0), T(0), T(0));
  CMG_LAUNCHED("zeroCovered");
}

template <class T>
void gsrb(const LevelDev& L, T* phi, const T* rhs, const Coef<T>& c, int color, cudaStream_t s, bool inlineGhosts) {
  int n = L.nColor[color];
  if (n == 0) return;
  Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  const double dx = L.dx, dxc = L.dxCrse;
  GhostCoef gc{2 * (dxc - dx) / (dxc + dx), -(dxc - dx) / (dxc + 3 * dx), 1 - 2 * dx / (dx + dxc)};
  auto launch = [&](auto kern, const T* a, const T* b0, const T* b1, const T* b2, const T* lam) {
    launchNext(kern, n, CHUNK, s, L.boxes, L.chColor[color], phi, rhs, color, sc, a, b0, b1, b2, lam,
               L.chGhost[color], L.chGhostStart[color], gc);
  };
  auto launchPair = [&](auto kern, const T* a, const T* b0, const T* b1, const T* b2, const T* lam) {
    launchNext(kern, n, CHUNK / 2, s, L.boxes, L.chColor[color], phi, rhs, color, sc, a, b0, b1, b2, lam);
  };
  if (c.vc) {
    if (inlineGhosts)
      launch(k_gsrb<T, 1>, c.a, c.b[0], c.b[1], c.b[2], c.lambda);
    else
      launchPair(k_gsrb_pair<T, 1>, c.a, c.b[0], c.b[1], c.b[2], c.lambda);
  } else {
    if (inlineGhosts)
      launch(k_gsrb<T, 0>, nullptr, nullptr, nullptr, nullptr, nullptr);
    else
      launchPair(k_gsrb_pair<T, 0>, nullptr, nullptr, nullptr, nullptr, nullptr);
  }
  CMG_LAUNCHED("gsrb");
}

template <class T>
void gsrbUniform(const LevelDev& L, T* phi, const T* rhs, const Coef<T>& c, int color, cudaStream_t s) {
  const int n = L.nColor[color];
  if (n == 0) return;
  const Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  const int per = uniformPer(n);
  auto kern = c.vc ? k_gsrb_uniform<T, 1> : k_gsrb_uniform<T, 0>;
  launchNext(kern, (n + per - 1) / per, CHUNK / 2, s, L.boxes, L.uniform, L.chColor[color], n, per, phi, rhs, color,
             sc, c.a, c.b[0], c.b[1], c.b[2], c.lambda);
  CMG_LAUNCHED("gsrbUniform");
}

template <class T>
void residualUniform(const LevelDev& L, T* r, const T* phi, const T* rhs, const Coef<T>& c, cudaStream_t s,
                     double* norm) {
  const int n = L.nColor[0];
  if (n == 0) return;
  const Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  const int per = norm && L.boxHier ? 1 : uniformPer(n);
  auto kern = norm ? (c.vc ? k_residual_uniform<T, 1, true, T> : k_residual_uniform<T, 0, true, T>)
                   : (c.vc ? k_residual_uniform<T, 1, false, T> : k_residual_uniform<T, 0, false, T>);
  launchNext(kern, (n + per - 1) / per, CHUNK, s, L.boxes, L.uniform, L.chColor[0], n, per, r, phi, rhs, sc, c.a,
             c.b[0], c.b[1], c.b[2], L.boxHier, norm);
  CMG_LAUNCHED("residualUniform");
}

template <class T>
void gsrbFirst(const LevelDev& L, T* phi, const T* rhs, const Coef<T>& c, cudaStream_t s) {
  const int n = L.nColor[0];
  if (n == 0) return;
  const Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  if (c.vc)
    launchNext(k_gsrb_first<T, 1>, n, CHUNK / 2, s, L.boxes, L.chColor[0], phi, rhs, sc, c.lambda);
  else
    launchNext(k_gsrb_first<T, 0>, n, CHUNK / 2, s, L.boxes, L.chColor[0], phi, rhs, sc, nullptr);
  CMG_LAUNCHED("gsrbFirst");
}

template <class T>
void gsrbSweepFused(const LevelDev& L, T* phi, const T* rhs, const Coef<T>& c, cudaStream_t s) {
  if (L.nbox == 0) return;
  Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  const double dx = L.dx, dxc = L.dxCrse;
  GhostCoef gc{2 * (dxc - dx) / (dxc + dx), -(dxc - dx) / (dxc + 3 * dx), 1 - 2 * dx / (dx + dxc)};
  const int nd = L.nDeferred, db = (nd + 255) / 256;
  if (c.vc) {
    k_gsrb_march<T, 1><<<L.nbox, 256, 0, s>>>(L.boxes, phi, rhs, sc, c.a, c.b[0], c.b[1], c.b[2], c.lambda,
                                              L.faceRules, L.faceOff, gc);
    CMG_LAUNCHED("gsrbMarch");
    if (nd > 0) {
      k_gsrb_deferred<T, 1><<<db, 256, 0, s>>>(L.boxes, L.deferred, nd, phi, rhs, sc, c.a, c.b[0], c.b[1], c.b[2],
                                               c.lambda, L.faceRules, L.faceOff, gc);
      CMG_LAUNCHED("gsrbDeferred");
    }
  } else {
    k_gsrb_march<T, 0><<<L.nbox, 256, 0, s>>>(L.boxes, phi, rhs, sc, nullptr, nullptr, nullptr, nullptr, nullptr,
                                              L.faceRules, L.faceOff, gc);
    CMG_LAUNCHED("gsrbMarch");
    if (nd > 0) {
      k_gsrb_deferred<T, 0><<<db, 256, 0, s>>>(L.boxes, L.deferred, nd, phi, rhs, sc, nullptr, nullptr, nullptr,
                                               nullptr, nullptr, L.faceRules, L.faceOff, gc);
      CMG_LAUNCHED("gsrbDeferred");
    }
  }
}

template <class T>
void residual(const LevelDev& L, T* r, const T* phi, const T* rhs, const Coef<T>& c, cudaStream_t s, double* norm) {
  if (L.nAll == 0) return;
  Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  const int n = L.nColor[0];
  const T *a = c.vc ? c.a : nullptr, *b0 = c.vc ? c.b[0] : nullptr, *b1 = c.vc ? c.b[1] : nullptr,
          *b2 = c.vc ? c.b[2] : nullptr;
  if (norm) {
    auto kern = c.vc ? k_residual_norm<T, 1, T> : k_residual_norm<T, 0, T>;
    launchNext(kern, n, CHUNK, s, L.boxes, L.chColor[0], L.chColor[1], r, phi, rhs, sc, a, b0, b1, b2, L.boxHier, norm);
  } else {
    auto kern = c.vc ? k_op_pair<T, 1, 0> : k_op_pair<T, 0, 0>;
    launchNext(kern, n, CHUNK, s, L.boxes, L.chColor[0], L.chColor[1], r, phi, rhs, sc, a, b0, b1, b2);
  }
  CMG_LAUNCHED("residual");
}

void residual32(const LevelDev& L, float* r, const double* phi, const double* rhs, const Coef<double>& c,
                cudaStream_t s, double* norm, bool acrossFaces) {
  const int n = L.nColor[0];
  if (n == 0) return;
  const Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  if (acrossFaces) {
    const int per = L.boxHier ? 1 : uniformPer(n);
    auto kern = c.vc ? k_residual_uniform<double, 1, true, float> : k_residual_uniform<double, 0, true, float>;
    launchNext(kern, (n + per - 1) / per, CHUNK, s, L.boxes, L.uniform, L.chColor[0], n, per, r, phi, rhs, sc, c.a,
               c.b[0], c.b[1], c.b[2], L.boxHier, norm);
  } else {
    auto kern = c.vc ? k_residual_norm<double, 1, float> : k_residual_norm<double, 0, float>;
    launchNext(kern, n, CHUNK, s, L.boxes, L.chColor[0], L.chColor[1], r, phi, rhs, sc, c.a, c.b[0], c.b[1], c.b[2],
               L.boxHier, norm);
  }
  CMG_LAUNCHED("residual32");
}

template <class T>
void applyOp(const LevelDev& L, T* lofphi, const T* phi, const Coef<T>& c, cudaStream_t s) {
  if (L.nAll == 0) return;
  Scal sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  const int n = L.nColor[0];
  if (c.vc)
    launchNext(k_op_pair<T, 1, 1>, n, CHUNK, s, L.boxes, L.chColor[0], L.chColor[1], lofphi, phi, nullptr, sc, c.a,
               c.b[0], c.b[1], c.b[2]);
  else
    launchNext(k_op_pair<T, 0, 1>, n, CHUNK, s, L.boxes, L.chColor[0], L.chColor[1], lofphi, phi, nullptr, sc, nullptr,
               nullptr, nullptr, nullptr);
  CMG_LAUNCHED("applyOp");
}

template <class T>
void negAdd(const LevelDev& L, T* r, const T* lofphi, const T* rhs, cudaStream_t s) {
  if (L.nelem == 0) return;
  launchNext(k_negadd_flat<T>, flatBlocks(L.nelem), 256, s, r, lofphi, rhs, L.nelem);
  CMG_LAUNCHED("negAdd");
}

template <class T>
void restrictMG(const LevelDev& F, const LevelDev& C, T* resC, const T* phi, const T* rhs, const Coef<T>& c,
                cudaStream_t s) {
  if (C.nAll == 0) return;
  Scal sc = scalars(F.dx, c.alpha, c.beta, c.vc);
  if (c.vc)
    launchNext(k_restrictmg<T, 1>, C.nAll, CHUNK, s, F.boxes, C.boxes, C.chAll, resC, phi, rhs, sc, c.a, c.b[0], c.b[1],
               c.b[2]);
  else
    launchNext(k_restrictmg<T, 0>, C.nAll, CHUNK, s, F.boxes, C.boxes, C.chAll, resC, phi, rhs, sc, nullptr, nullptr,
               nullptr, nullptr);
  CMG_LAUNCHED("restrictMG");
}

template <class T>
void restrictUniform(const LevelDev& F, const LevelDev& C, T* resC, const T* phi, const T* rhs, const Coef<T>& c,
                     cudaStream_t s) {
  if (C.nAll == 0) return;
  const Scal sc = scalars(F.dx, c.alpha, c.beta, c.vc);
  auto kern = c.vc ? k_restrict_uniform<T, 1> : k_restrict_uniform<T, 0>;
  launchNext(kern, C.nAll, CHUNK, s, F.boxes, F.uniform, C.boxes, C.chAll, resC, phi, rhs, sc, c.a, c.b[0], c.b[1],
             c.b[2]);
  CMG_LAUNCHED("restrictUniform");
}

template <class T>
void prolongMG(const LevelDev& F, const LevelDev& C, T* phi, const T* corrC, cudaStream_t s) {
  if (C.nAll == 0) return;
  launchNext(k_prolongmg<T>, C.nAll, CHUNK, s, F.boxes, C.boxes, C.chAll, phi, corrC);
  CMG_LAUNCHED("prolongMG");
}

template <class T>
void averageAMR(const LevelDev& F, const LevelDev& C, T* coarse, const T* fine, cudaStream_t s) {
  if (F.nItemChC == 0) return;
  launchNext(k_average<T>, F.nItemChC, CHUNK, s, F.boxes, C.boxes, F.items, F.itemChC, coarse, fine);
  CMG_LAUNCHED("averageAMR");
}

template <class T>
void prolongAMR(const LevelDev& F, const LevelDev& C, T* fine, const T* coarse, cudaStream_t s) {
  if (F.nItemChF == 0) return;
  launchNext(k_prolongamr<T>, F.nItemChC, CHUNK, s, F.boxes, C.boxes, F.items, F.itemChC, fine, coarse);
  CMG_LAUNCHED("prolongAMR");
}

template <class T>
void quadCF(const LevelDev& F, T* phiF, const T* phiC, cudaStream_t s) {
  if (F.nCfF == 0) return;
  T* tmp = nullptr;
  if (phiC) {
    tmp = reinterpret_cast<T*>(F.cfTmp);
    launchNext(k_cf_coarse<T>, (F.nCfC + 31) / 32, 192, s, F.cfC, F.nCfC, F.cfW, F.cfOff, phiC, T(F.dx), tmp);
    CMG_LAUNCHED("quadCFCoarse");
  }
  launchNext(k_quadcf<T>, (F.nCfF + 127) / 128, 128, s, F.cfF, F.nCfF, tmp, phiF, T(F.dx));
  CMG_LAUNCHED("quadCF");
}

template <class T>
void reflux(const LevelDev& C, T* lofphiC, const T* phiC, const T* phiF, const Coef<T>& cc, const Coef<T>& cf,
            cudaStream_t s) {
  if (C.nRf == 0) return;
  int nb = (C.nRf + 127) / 128;
  // getFlux scale beta * ref / dx with the coarse dx (AMRPoissonOp.cpp:1797-1851).
  T sc = T(cc.beta * 1 / C.dx);
  T sf = T(cc.beta * 2 / C.dx);
  T negs = T(-(1.0 / C.dx));
  if (cc.vc)
    launchNext(k_reflux<T, 1>, nb, 128, s, C.rfCells, C.nRf, C.rfC, C.rfF, lofphiC, phiC, phiF, cc.b[0], cc.b[1],
               cc.b[2], cf.b[0], cf.b[1], cf.b[2], sc, sf, negs);
  else
    launchNext(k_reflux<T, 0>, nb, 128, s, C.rfCells, C.nRf, C.rfC, C.rfF, lofphiC, phiC, phiF, nullptr, nullptr,
               nullptr, nullptr, nullptr, nullptr, sc, sf, negs);
  CMG_LAUNCHED("reflux");
}

template <class T>
void incr(const LevelDev& L, T* lhs, const T* x, double scale, cudaStream_t s) {
  if (L.nelem == 0) return;
  launchNext(k_incr_flat<T, T>, flatBlocks(L.nelem), 256, s, lhs, x, T(scale), L.nelem);
  CMG_LAUNCHED("incr");
}

template <class T>
void incrCopy(const LevelDev& L, T* lhs, T* x, cudaStream_t s) {
  if (L.nelem == 0) return;
  launchNext(k_incr_copy_flat<T>, flatBlocks(L.nelem), 256, s, lhs, x, L.nelem);
  CMG_LAUNCHED("incrCopy");
}

template <class T>
void maxNorm(const LevelDev& L, const T* f, double* out, cudaStream_t s, const unsigned char* mask) {
  if (L.nAll == 0) return;
  if (L.boxHier) {  // forests pass no mask
    launchNext(k_maxnorm_hier<T>, L.nAll, CHUNK, s, L.boxes, L.chAll, L.boxHier, f, out);
    CMG_LAUNCHED("maxNorm");
    return;
  }
  // One chunk per block (lowest latency) up to 4096 chunks; beyond, a
  // grid of 4096 blocks striding over them.
  const int blocks = std::min(L.nAll, 4096);
  launchNext(k_maxnorm<T>, blocks, CHUNK, s, L.boxes, L.chAll, L.nAll, f, mask, out);
  CMG_LAUNCHED("maxNorm");
}


long long launchCount() { return g_launches.load(std::memory_order_relaxed); }
void addLaunches(long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

void bottomSolve(const LevelDev& L, double* phi, const double* rhs, const Coef<double>& c, const BottomWork* works,
                 int nworks, int maxBoxes, const BottomConfig& cfg, double eps, const double* metrics,
                 cudaStream_t s, const double* epsPer, int gridBlocks) {
  if (nworks == 0) return;
  BottomArgs A;
  A.boxes = L.boxes;
  A.sc = scalars(L.dx, c.alpha, c.beta, c.vc);
  A.vc = c.vc;
  A.phiFab = phi;
  A.rhsFab = rhs;
  A.cfg = cfg;
  A.eps = cfg.kind == 1 ? cfg.eps : eps;  // RelaxSolver keeps its own tolerance
  A.epsPer = epsPer;
  A.reps = cfg.reps;
  A.hang = cfg.hang;
  A.small = cfg.small;
  A.imax = cfg.imax;
  A.numRestarts = cfg.numRestarts;
  // AMRPoissonOp::preCond multiplier (AMRPoissonOp.cpp:304-329).
  A.mult = 1.0 / (c.alpha - 2.0 * 3 * c.beta / (L.dx * L.dx));
  if (gridBlocks > 0) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(gridBlocks);
    lc.blockDim = dim3(kBottomGridThreads);
    lc.dynamicSmemBytes = 0;
    lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    check(cudaLaunchKernelEx(&lc, k_bottom_grid, A, works, metrics), "bottomSolve (grid)");
    CMG_LAUNCHED("bottomSolve");
    return;
  }
  const size_t smem = 2 * (size_t)std::max(maxBoxes, 32) * sizeof(double);
  if (smem > 48 * 1024) {
    if (smem > 200 * 1024) throw std::runtime_error("cmg: bottom level with too many boxes for one block");
    check(cudaFuncSetAttribute(k_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "bottom smem");
  }
  k_bottom<<<nworks, 1024, smem, s>>>(A, works, metrics);
  CMG_LAUNCHED("bottomSolve");
}

int bottomGridBlocks(int nv) {
  int dev = 0, sms = 0, occ = 0;
  check(cudaGetDevice(&dev), "device");
  check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
  check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_bottom_grid, kBottomGridThreads, 0), "occupancy");
  const int want = (nv + kBottomGridThreads - 1) / kBottomGridThreads;
  return std::max(1, std::min(want, sms * std::max(occ, 1)));
}

int bottomGridThreads() { return kBottomGridThreads; }

void gatherSlots(const BottomWork& w, const double* fab, double* dst, cudaStream_t s) {
  const int n = w.nv + w.ng;
  if (n == 0) return;
  k_gather_slots<<<(n + 255) / 256, 256, 0, s>>>(w.fab, n, fab, dst);
  CMG_LAUNCHED("gatherSlots");
}

void incrMixed(const LevelDev& L, double* lhs, const float* x, cudaStream_t s) {
  if (L.nelem == 0) return;
  launchNext(k_incr_flat<double, float>, flatBlocks(L.nelem), 256, s, lhs, x, 1.0, L.nelem);
  CMG_LAUNCHED("incrMixed");
}

template <class T, class X>
void incrActive(const LevelDev& L, T* lhs, const X* x, const int* active, cudaStream_t s) {
  if (L.nelem == 0) return;
  const int64_t per = (L.nelem + L.nh - 1) / L.nh;
  const int bx = (int)std::max<int64_t>(1, std::min<int64_t>((per + 255) / 256, 64));
  launchNext(k_incr_active<T, X>, dim3(bx, L.nh), 256, s, lhs, x, L.hierStart, active);
  CMG_LAUNCHED("incrActive");
}
template void incrActive<double, double>(const LevelDev&, double*, const double*, const int*, cudaStream_t);
template void incrActive<double, float>(const LevelDev&, double*, const float*, const int*, cudaStream_t);

template <class X>
void incrSum(const LevelDev& L, double* lhs, const X* x, const X* y, const int* active, cudaStream_t s) {
  if (L.nelem == 0) return;
  const int nh = active ? L.nh : 1;
  const int64_t per = (L.nelem + nh - 1) / nh;
  const int bx = active ? (int)std::max<int64_t>(1, std::min<int64_t>((per + 255) / 256, 64)) : flatBlocks(L.nelem);
  launchNext(k_incr_sum<double, X>, dim3(bx, nh), 256, s, lhs, x, y, L.nelem, active ? L.hierStart : nullptr, active);
  CMG_LAUNCHED("incrSum");
}

template <class D, class S>
void convert(D* dst, const S* src, int64_t n, cudaStream_t s) {
  if (n == 0) return;
  int blocks = (int)std::min<int64_t>((n + 255) / 256, 148 * 16);
  launchNext(k_convert<D, S>, blocks, 256, s, dst, src, n);
  CMG_LAUNCHED("convert");
}
template void convert<float, double>(float*, const double*, int64_t, cudaStream_t);
template void convert<double, float>(double*, const float*, int64_t, cudaStream_t);

// ------------------------------------------------ synthetic inputs, device
// The seeded fields of synthetic.H evaluated on the device (same formulas and
// operation order; exp and cos of the CUDA math library, so values agree with
// the host generator to within their last bits), and the coefficient set-up
// of finalizeCoefficients (resetLambda with SUMFACES, MG coefficient
// averages) with the host code's operation order.
namespace {

__global__ void k_fill_cells(const BoxDesc* boxes, const Chunk* chunks, double dx, cmg_synth::Bumps bumps,
                             cmg_synth::Modes am, double* rhs, double* a) {
  Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  int i, j, k;
  if (!allCell(bd, ch.start + threadIdx.x, i, j, k)) return;
  const double x = (i + 0.5) * dx, y = (j + 0.5) * dx, z = (k + 0.5) * dx;
  const int64_t c = cellIndex(bd, i, j, k);
  rhs[c] = devBumps(bumps, x, y, z);
  if (a) a[c] = devModes(am, x, y, z);
}

// One block per box: faces lo..hi+1 in direction d.
__global__ void k_fill_faces(const BoxDesc* boxes, double dx, int d, cmg_synth::Modes bm, double* b) {
  const BoxDesc bd = boxes[blockIdx.x];
  int n[3];
  for (int e = 0; e < 3; ++e) n[e] = bd.hi[e] - bd.lo[e] + 1 + (e == d);
  const int total = n[0] * n[1] * n[2];
  for (int q = threadIdx.x; q < total; q += blockDim.x) {
    int iv[3] = {bd.lo[0] + q % n[0], bd.lo[1] + (q / n[0]) % n[1], bd.lo[2] + q / (n[0] * n[1])};
    double x[3];
    for (int e = 0; e < 3; ++e) x[e] = (e == d) ? iv[e] * dx : (iv[e] + 0.5) * dx;
    b[cellIndex(bd, iv[0], iv[1], iv[2])] = devModes(bm, x[0], x[1], x[2]);
  }
}

// lambda = 1 / (alpha a + sum_d scale beta (b_hi + b_lo)) (computeLambda).
__global__ void k_lambda(const BoxDesc* boxes, const Chunk* chunks, const double* a, const double* b0,
                         const double* b1, const double* b2, double alpha, double beta, double dx, double* lam) {
  Chunk ch = chunks[blockIdx.x];
  const BoxDesc bd = boxes[ch.box];
  int i, j, k;
  if (!allCell(bd, ch.start + threadIdx.x, i, j, k)) return;
  const Stencil st = stencil(bd, i, j, k);
  const double scale = 1.0 / (dx * dx);
  double l = a[st.c] * alpha;
  l = l + scale * beta * (b0[st.xp] + b0[st.c]);
  l = l + scale * beta * (b1[st.yp] + b1[st.c]);
  l = l + scale * beta * (b2[st.zp] + b2[st.c]);
  lam[st.c] = 1.0 / l;
}

// averageCells: coarse(i) = refScale * sum of its r^3 fine values in k-j-i order.
__global__ void k_avg_cells(const BoxDesc* fboxes, const BoxDesc* cboxes, const Chunk* chunks, int r,
                            const double* f, double* out) {
  Chunk ch = chunks[blockIdx.x];
  const BoxDesc cb = cboxes[ch.box];
  int i, j, k;
  if (!allCell(cb, ch.start + threadIdx.x, i, j, k)) return;
  const BoxDesc fb = fboxes[ch.box];
  const double refScale = 1.0 / (double)(r * r * r);
  double s = 0.0;
  bool first = true;
  for (int c = 0; c < r; ++c)
    for (int bb = 0; bb < r; ++bb)
      for (int aa = 0; aa < r; ++aa) {
        double v = f[cellIndex(fb, i * r + aa, j * r + bb, k * r + c)];
        s = first ? v : s + v;
        first = false;
      }
  out[cellIndex(cb, i, j, k)] = refScale * s;
}

// averageFaces: coarse face = refScale * sum over the r^2 fine faces.
__global__ void k_avg_faces(const BoxDesc* fboxes, const BoxDesc* cboxes, int r, int d, const double* f,
                            double* out) {
  const BoxDesc cb = cboxes[blockIdx.x];
  const BoxDesc fb = fboxes[blockIdx.x];
  int n[3], ext[3] = {r, r, r};
  ext[d] = 1;
  for (int e = 0; e < 3; ++e) n[e] = cb.hi[e] - cb.lo[e] + 1 + (e == d);
  const double base = 1.0 / (double)r;
  const double refScale = base * base;
  const int total = n[0] * n[1] * n[2];
  for (int q = threadIdx.x; q < total; q += blockDim.x) {
    int i = cb.lo[0] + q % n[0], j = cb.lo[1] + (q / n[0]) % n[1], k = cb.lo[2] + q / (n[0] * n[1]);
    double s = 0;
    for (int c = 0; c < ext[2]; ++c)
      for (int bb = 0; bb < ext[1]; ++bb)
        for (int aa = 0; aa < ext[0]; ++aa) s = s + f[cellIndex(fb, i * r + aa, j * r + bb, k * r + c)];
    out[cellIndex(cb, i, j, k)] = refScale * s;
  }
}

}  // namespace

void fillSyntheticLevel(const LevelDev& L, uint64_t seed, double* rhs, double* a, double* const b[3],
                        cudaStream_t s) {
  fillSyntheticBoxes(L, seed, rhs, a, b, 0, L.nbox, 0, L.nAll, s);
}

void fillSyntheticBoxes(const LevelDev& L, uint64_t seed, double* rhs, double* a, double* const b[3], int box0,
                        int box1, int ch0, int ch1, cudaStream_t s) {
  cmg_synth::Problem prob(seed);
  if (ch1 <= ch0) return;
  k_fill_cells<<<ch1 - ch0, CHUNK, 0, s>>>(L.boxes, L.chAll + ch0, L.dx, prob.bumps, prob.acoef, rhs, a);
  CMG_LAUNCHED("fillCells");
  if (!b || box1 <= box0) return;
  for (int d = 0; d < 3; ++d) {
    k_fill_faces<<<box1 - box0, 256, 0, s>>>(L.boxes + box0, L.dx, d, prob.bcoef, b[d]);
    CMG_LAUNCHED("fillFaces");
  }
}

void lambdaLevel(const LevelDev& L, const double* a, const double* const b[3], double alpha, double beta,
                 double* lam, cudaStream_t s) {
  if (L.nAll == 0) return;
  k_lambda<<<L.nAll, CHUNK, 0, s>>>(L.boxes, L.chAll, a, b[0], b[1], b[2], alpha, beta, L.dx, lam);
  CMG_LAUNCHED("lambda");
}

void averageCoefficients(const LevelDev& F, const LevelDev& C, int r, const double* fa, const double* const fb[3],
                         double* ca, double* const cbf[3], cudaStream_t s) {
  if (C.nAll == 0) return;
  k_avg_cells<<<C.nAll, CHUNK, 0, s>>>(F.boxes, C.boxes, C.chAll, r, fa, ca);
  CMG_LAUNCHED("averageCells");
  for (int d = 0; d < 3; ++d) {
    k_avg_faces<<<C.nbox, 256, 0, s>>>(F.boxes, C.boxes, r, d, fb[d], cbf[d]);
    CMG_LAUNCHED("averageFaces");
  }
}

#define CMG_INST(T)                                                                                       \
  template void ghostFill<T>(const LevelDev&, T*, bool, cudaStream_t, int);                                \
  template void zeroCovered<T>(const LevelDev&, T*, cudaStream_t);                                         \
  template void gsrb<T>(const LevelDev&, T*, const T*, const Coef<T>&, int, cudaStream_t, bool);           \
  template void gsrbUniform<T>(const LevelDev&, T*, const T*, const Coef<T>&, int, cudaStream_t);           \
  template void residualUniform<T>(const LevelDev&, T*, const T*, const T*, const Coef<T>&, cudaStream_t,  \
                                   double*);                                                               \
  template void restrictUniform<T>(const LevelDev&, const LevelDev&, T*, const T*, const T*,               \
                                   const Coef<T>&, cudaStream_t);                                          \
  template void gsrbFirst<T>(const LevelDev&, T*, const T*, const Coef<T>&, cudaStream_t);                 \
  template void gsrbSweepFused<T>(const LevelDev&, T*, const T*, const Coef<T>&, cudaStream_t);            \
  template void residual<T>(const LevelDev&, T*, const T*, const T*, const Coef<T>&, cudaStream_t, double*); \
  template void applyOp<T>(const LevelDev&, T*, const T*, const Coef<T>&, cudaStream_t);                   \
  template void negAdd<T>(const LevelDev&, T*, const T*, const T*, cudaStream_t);                          \
  template void restrictMG<T>(const LevelDev&, const LevelDev&, T*, const T*, const T*, const Coef<T>&,    \
                              cudaStream_t);                                                               \
  template void prolongMG<T>(const LevelDev&, const LevelDev&, T*, const T*, cudaStream_t);                \
  template void averageAMR<T>(const LevelDev&, const LevelDev&, T*, const T*, cudaStream_t);               \
  template void prolongAMR<T>(const LevelDev&, const LevelDev&, T*, const T*, cudaStream_t);               \
  template void quadCF<T>(const LevelDev&, T*, const T*, cudaStream_t);                                    \
  template void reflux<T>(const LevelDev&, T*, const T*, const T*, const Coef<T>&, const Coef<T>&,         \
                          cudaStream_t);                                                                   \
  template void incrCopy<T>(const LevelDev&, T*, T*, cudaStream_t);                                         \
  template void incrSum<T>(const LevelDev&, double*, const T*, const T*, const int*, cudaStream_t);        \
  template void incr<T>(const LevelDev&, T*, const T*, double, cudaStream_t);                              \
  template void maxNorm<T>(const LevelDev&, const T*, double*, cudaStream_t, const unsigned char*);

CMG_INST(double)
CMG_INST(float)

}  // namespace cmg
