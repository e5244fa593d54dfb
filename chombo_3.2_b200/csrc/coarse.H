// The coarse part of the multigrid cycle below level 0 as one launch: every
// depth from a top depth down to the bottom solve, relaxed, restricted, solved
// and prolonged by one thread-block cluster per hierarchy that holds the
// depths' corrections and residuals in its shared memory (coarse.cu).
#ifndef CMG_COARSE_H
#define CMG_COARSE_H

#include <vector>

#include "cellops.H"
#include "kernels.H"
#include "plan.H"

namespace cmg {

enum {
  kCoarseMaxDepths = 16,
  kCoarseRankShift = 20,
  kCoarseSmem = 220 * 1024  // shared memory of the fields, of the 227 KB a block may hold
};

// One depth's tables.  A cell's slot counts the depth's cells box by box, x
// fastest; consecutive slots go to consecutive ranks (blocks of the cluster).
// Every rank's field holds its own cells (nLoc at most) and then its halo: the
// cells of other ranks its stencils read, sent by their owners when they
// change, so that a pass reads only its own shared memory.  Entries list the
// cells rank by rank, colour 0 first.  nb: the entry's neighbours (+x, -x, +y,
// -y, +z, -z) as 16-bit elements of the field, the high bit marking a
// homogeneous Dirichlet ghost (0 - the element named; exchange copies, periodic
// images and Neumann ghosts name the cell their value is copied from), and in
// w its own cell.  push: the cells a rank sends, by rank and colour, each as
// own element << 19 | receiving rank << 15 | its halo element there.
struct CoarseDepth {
  int n;               // cells
  int solo;            // every cell on rank 0
  int nField;          // elements of a field with its halo
  const int* colStart; // 2 per rank + 1: first entry of each rank and colour
  const uint4* nb;
  const unsigned* push;
  const int* pushStart; // 2 per rank + 1
  const int* par;      // the coarse cell above each entry (rank << shift | cell); not on the bottom depth
  const int4* child;   // per entry, its eight fine cells in k, j, i order (rank << shift | cell); not on the top depth
  const double* coefD; // VC: a, lambda, b at +x, -x, +y, -y, +z, -z; each n values in entry order
  const float* coefF;
  int phi[2], rhs[2];  // byte offsets in shared memory of the correction and residual, FP64 [0] and FP32 [1] cycles
};

struct CoarseHier {
  int nd;                 // depths
  int dSolo;              // first depth kept on rank 0 (nd: none)
  CoarseDepth d[kCoarseMaxDepths];
  const int *fab;         // top depth: FAB element of each entry
  // bottom
  int nbox, maxNx;
  int allRanks;           // sums folded by every rank (else by ranks 0 and 1, then broadcast)
  const int* boxRank;     // first box of each rank (ranks + 1)
  const int4* box;        // per box: first cell on its rank, nx, ny, nz
  const double* lamSlot;  // VC: lambda in slot order
  const int* rankSlot;    // first slot of each rank
  int nLoc;               // most cells of a rank on the bottom depth
  int tmp[2], vec[2];     // byte offsets: restriction scratch, bottom vectors
  int part, pen;          // byte offsets: box sums, pencil sums
  int* status;
};

// Host plan of one hierarchy's coarse part.
struct CoarsePlan {
  struct Depth {
    int n = 0, per = 0, solo = 0, nLoc = 0, nHalo = 0, nField = 0;
    double dx = 0;
    std::vector<int> rankSlot, colStart, pushStart;
    PlanVec<int> nb, par, child, fab, fh;  // fh: FAB elements of the high x, y, z faces
    std::vector<unsigned> push;
  };
  std::vector<Depth> d;
  int dSolo = 0, nbox = 0, maxNx = 0, nPen = 0, allRanks = 1;
  std::vector<int> boxRank, box, bottomFab;  // box: 4 per box
  int phi[kCoarseMaxDepths][2], rhs[kCoarseMaxDepths][2], tmp[2], vec[2], part = 0, pen = 0;
  int bytes[2] = {0, 0};  // shared memory of FP64 and FP32 cycles
};

// Tables of one hierarchy (levels: depth 0 = level 0, 1.. the multigrid depths)
// from depth `top` on, over `ranks` blocks; false when an FP64 cycle does not fit
// (an FP32 one also holds the FP64 bottom vectors and may be the larger).  bc and
// periodic as buildLevel's.
bool buildCoarse(const std::vector<const LevelPlan*>& levels, int top, int ranks, const int* bc, const bool* periodic,
                 CoarsePlan& P);
// The first depth the coarse launch can take, its ranks and the plans of every
// hierarchy; false when no depth fits.
bool planCoarse(const std::vector<std::vector<const LevelPlan*>>& levels, const int* bc, const bool* periodic, bool vc,
                int* top, int* ranks, std::vector<CoarsePlan>& plans);

// Gathers the depths' coefficients into entry order (CoarseDepth::coefD, coefF)
// and lambda on the bottom into slot order (lamSlot, may be null), in one launch.
// lamOnly: lambda alone, after alpha or beta changed.
template <class T>
struct CoarseCoefs {
  int nd;
  struct Depth {
    int n;
    const int *fab, *fh;
    const double *a, *b[3], *lambda;
    T* out;
  } d[kCoarseMaxDepths];
  const int* slotFab;
  double* lamSlot;
};
template <class T>
void gatherCoarse(const CoarseCoefs<T>& C, bool lamOnly, cudaStream_t s);

// Whether the device can hold a cluster of that size with that much shared memory.
bool coarseFits(int ranks, int bytes);

// The coarse cycle of every hierarchy on corr (zero at first when fromZero,
// whatever its memory holds) and res (the top depth's FAB fields): relaxations, restrictions, bottom solve and prolongations as
// Solver::mgCycle launches them one by one, the same values bit for bit.
// sc: the operator's scalars of each depth.
template <class T>
void coarseCycle(const CoarseHier* hier, int nh, int ranks, int bytes, const std::vector<Scal>& sc, T* corr, const T* res,
                 int vc, int pre, int post, int bottomSweeps, int numMG, bool oneCell, bool fromZero,
                 const BottomConfig& cfg, double eps, double mult, const double* metrics, const double* epsPer,
                 cudaStream_t s);

}  // namespace cmg

#endif
