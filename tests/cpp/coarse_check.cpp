// The coarse launch's tables (coarse.H) of a hierarchy's multigrid depths,
// checked cell by cell against the layouts: every cell is one entry of one
// rank, its neighbours, parent and children are the cells the exchange, the
// boundary conditions, PROLONG and RESTRICTRES name, and no two regions of
// shared memory overlap.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "../../chombo_3.2_b200/csrc/coarse.H"

using namespace cmg;

#define REQUIRE(c)                                                     \
  do {                                                                 \
    if (!(c)) {                                                        \
      std::printf("line %d: %s\n", __LINE__, #c);                      \
      std::exit(1);                                                    \
    }                                                                  \
  } while (0)

static int check(int n0, int maxBox, int block, const int* bc, const bool* per, int ranks, int topSkip) {
  const Box dom(IV{0, 0, 0}, IV{n0 - 1, n0 - 1, n0 - 1});
  std::vector<Box> boxes = domainSplit(dom, maxBox, block);
  const Layout g0(boxes);
  std::vector<LevelPlan> lev(1);
  buildLevel(lev[0], g0, dom, 1.0 / n0, 0.0, bc, per);
  for (int c = 2; g0.coarsenable(c * 2); c *= 2) {
    lev.emplace_back();
    buildLevel(lev.back(), g0.coarsen(c), dom.coarsen(c), 1.0 / n0 * c, 0.0, bc, per);
  }
  const int D = (int)lev.size(), top = std::min(topSkip, D - 1);
  std::vector<const LevelPlan*> levels;
  for (const LevelPlan& l : lev) levels.push_back(&l);
  CoarsePlan P;
  REQUIRE(buildCoarse(levels, top, ranks, bc, per, P));
  const int nd = (int)P.d.size();
  REQUIRE(nd == D - top);
  const int mask = (1 << kCoarseRankShift) - 1;
  std::vector<std::vector<int>> slots;                  // per depth: slot of each entry
  std::vector<std::vector<std::vector<int>>> entries;   // per depth and rank: entry of each element
  std::vector<std::pair<int, int>> finer;               // the finer depth's (parent, slot it must be)
  for (int i = 0; i < nd; ++i) {
    std::vector<std::pair<int, int>> parent;
    const LevelPlan& L = lev[top + i];
    const CoarsePlan::Depth& Q = P.d[i];
    REQUIRE(Q.n == (int)L.grids.numCells());
    // entry of each (rank, cell)
    std::vector<std::vector<int>> entry(ranks);
    for (int r = 0; r < ranks; ++r) entry[r].assign(Q.rankSlot[r + 1] - Q.rankSlot[r], -1);
    std::vector<int> rankOf(Q.n), colOf(Q.n);
    for (int r = 0; r < ranks; ++r)
      for (int c = 0; c < 2; ++c)
        for (int e = Q.colStart[2 * r + c]; e < Q.colStart[2 * r + c + 1]; ++e) {
          const int q = Q.nb[4 * (size_t)e + 3];
          REQUIRE(q >= 0 && q < (int)entry[r].size() && q < Q.nLoc && entry[r][q] < 0);
          entry[r][q] = e;
          rankOf[e] = r;
          colOf[e] = c;
        }
    // what each rank's halo elements hold: the entry pushed there
    REQUIRE(Q.nField >= Q.nLoc && Q.nField <= 0x8000);
    std::vector<std::vector<int>> halo(ranks, std::vector<int>(Q.nField, -1));
    REQUIRE((int)Q.pushStart.size() == 2 * ranks + 1 && Q.pushStart.back() == (int)Q.push.size());
    for (int r = 0; r < ranks; ++r)
      for (int c = 0; c < 2; ++c)
        for (int p = Q.pushStart[2 * r + c]; p < Q.pushStart[2 * r + c + 1]; ++p) {
          const unsigned v = Q.push[p];
          const int src = v >> 19, to = v >> 15 & 15, dst = v & 0x7fff;
          REQUIRE(to < ranks && to != r && dst >= Q.nLoc && dst < Q.nField && halo[to][dst] < 0);
          REQUIRE(src < (int)entry[r].size() && colOf[entry[r][src]] == c);
          halo[to][dst] = entry[r][src];
        }
    // slot of each entry: rank by rank, colour by colour in slot order
    std::vector<int> slot(Q.n);
    std::vector<IV> pos;       // by slot
    std::vector<int> boxOf;
    for (size_t b = 0; b < L.grids.size(); ++b) {
      const Box& x = L.grids[b];
      for (int k = x.lo[2]; k <= x.hi[2]; ++k)
        for (int j = x.lo[1]; j <= x.hi[1]; ++j)
          for (int q = x.lo[0]; q <= x.hi[0]; ++q) {
            pos.push_back(IV{q, j, k});
            boxOf.push_back((int)b);
          }
    }
    for (int r = 0, e = 0; r < ranks; ++r)
      for (int c = 0; c < 2; ++c)
        for (int t = Q.rankSlot[r]; t < Q.rankSlot[r + 1]; ++t)
          if (((pos[t][0] + pos[t][1] + pos[t][2]) & 1) == c) slot[e++] = t;
    auto slotOf = [&](int e) { return slot[e]; };
    if (i + 1 == nd)
      for (int e = 0; e < Q.n; ++e) REQUIRE(Q.nb[4 * (size_t)e + 3] == slot[e] - Q.rankSlot[rankOf[e]]);
    slots.push_back(slot);
    entries.push_back(entry);
    auto slotAt = [&](const IV& p) {
      const int b = ownerOf(L, p);
      REQUIRE(b >= 0);
      int s = 0;
      for (int x = 0; x < b; ++x) s += (int)L.grids[x].numPts();
      const Box& x = L.grids[b];
      return s + (p[0] - x.lo[0]) + x.size(0) * ((p[1] - x.lo[1]) + x.size(1) * (p[2] - x.lo[2]));
    };
    for (int e = 0; e < Q.n; ++e) {
      const int s = slotOf(e);
      const IV p = pos[s];
      const BoxDesc& bd = L.boxes[boxOf[s]];
      REQUIRE(colOf[e] == ((p[0] + p[1] + p[2]) & 1));
      REQUIRE(Q.fab[e] == (int)cellIndex(bd, p[0], p[1], p[2]));
      for (int d = 0; d < 3; ++d) {
        REQUIRE(Q.fh[(size_t)d * Q.n + e] == (int)cellIndex(bd, p[0] + (d == 0), p[1] + (d == 1), p[2] + (d == 2)));
        for (int side = 0; side < 2; ++side) {
          IV m = p;
          m[d] += side == 0 ? 1 : -1;
          const unsigned w = (unsigned)Q.nb[4 * (size_t)e + d] >> (16 * side) & 0xffff;
          const int el = w & 0x7fff;
          // the slot the element holds on this rank
          REQUIRE(el < Q.nLoc ? el < (int)entry[rankOf[e]].size() : halo[rankOf[e]][el] >= 0);
          const int src = slotOf(el < Q.nLoc ? entry[rankOf[e]][el] : halo[rankOf[e]][el]);
          const bool out = m[d] < L.domain.lo[d] || m[d] > L.domain.hi[d];
          if (out && per[d]) m[d] += side == 0 ? -L.domain.size(d) : L.domain.size(d);
          if (out && !per[d]) {
            const bool neumann = bc[2 * d + (side == 0)] == 1;
            REQUIRE((w >> 15) == (neumann ? 0u : 1u));
            REQUIRE(src == s);
          } else {
            REQUIRE((w >> 15) == 0 && src == slotAt(m));
          }
        }
      }
      if (i + 1 < nd) {
        const LevelPlan& LC = lev[top + i + 1];
        int s2 = 0;
        for (int x = 0; x < boxOf[s]; ++x) s2 += (int)LC.grids[x].numPts();
        const Box& x = LC.grids[boxOf[s]];
        s2 += (p[0] / 2 - x.lo[0]) + x.size(0) * ((p[1] / 2 - x.lo[1]) + x.size(1) * (p[2] / 2 - x.lo[2]));
        parent.push_back({Q.par[e], s2});
      }
      if (i > 0) {
        const LevelPlan& LF = lev[top + i - 1];
        int s2 = 0;
        for (int x = 0; x < boxOf[s]; ++x) s2 += (int)LF.grids[x].numPts();
        const Box& x = LF.grids[boxOf[s]];
        for (int n = 0; n < 8; ++n) {
          const int a = 2 * p[0] + (n & 1), b = 2 * p[1] + ((n >> 1) & 1), c = 2 * p[2] + (n >> 2);
          const int want = s2 + (a - x.lo[0]) + x.size(0) * ((b - x.lo[1]) + x.size(1) * (c - x.lo[2]));
          const int got = Q.child[8 * (size_t)e + n], r = got >> kCoarseRankShift, q = got & mask;
          REQUIRE(r < ranks && q < (int)entries[i - 1][r].size());
          REQUIRE(slots[i - 1][entries[i - 1][r][q]] == want);
        }
      }
    }
    // the finer depth's parents (this depth's cells)
    for (const auto& v : finer) {
      const int r = v.first >> kCoarseRankShift, q = v.first & mask;
      REQUIRE(r < ranks && q < (int)entry[r].size() && slotOf(entry[r][q]) == v.second);
    }
    finer = parent;
  }
  // bottom boxes on one rank each
  const CoarsePlan::Depth& B = P.d.back();
  int s = 0, r = 0;
  for (int b = 0; b < P.nbox; ++b) {
    while (r + 1 < ranks && b >= P.boxRank[r + 1]) ++r;
    const int n = P.box[4 * b + 1] * P.box[4 * b + 2] * P.box[4 * b + 3];
    REQUIRE(B.rankSlot[r] + P.box[4 * b] == s && s + n <= B.rankSlot[r + 1] && P.box[4 * b + 1] <= P.maxNx);
    s += n;
  }
  REQUIRE(s == B.n);
  for (int q = 0; q < ranks; ++q) {
    REQUIRE(B.rankSlot[q + 1] - B.rankSlot[q] <= B.nLoc);
    REQUIRE((P.boxRank[q + 1] - P.boxRank[q]) * P.maxNx <= P.nPen);
  }
  // regions in order, none overlapping the next, all inside the block's bytes
  for (int f = 0; f < 2; ++f) {
    const int w = f == 0 ? 8 : 4;
    int64_t end = (int64_t)(P.allRanks ? 4 : 1) * P.nbox * 8;
    REQUIRE(P.part == 0 && P.pen >= end);
    end = P.pen + (int64_t)P.nPen * 8;
    int64_t most = 0;
    for (int i = 0; i < nd; ++i) {
      for (int q = 0; q < ranks; ++q) REQUIRE(P.d[i].rankSlot[q + 1] - P.d[i].rankSlot[q] <= P.d[i].nLoc);
      REQUIRE(P.phi[i][f] >= end && P.phi[i][f] % 16 == 0);
      REQUIRE(P.rhs[i][f] >= P.phi[i][f] + (int64_t)P.d[i].nField * w);
      end = P.rhs[i][f] + (int64_t)P.d[i].nLoc * w;
      if (i + 1 < nd) most = std::max<int64_t>(most, P.d[i].nLoc);
    }
    REQUIRE(P.tmp[f] >= end && P.vec[f] >= end && P.vec[f] % 16 == 0);
    // vectors: pt with its halo and six more; FP32 cycles add the FP64 right-hand side and phi
    REQUIRE(P.tmp[f] + most * w <= P.bytes[f]);
    REQUIRE(P.vec[f] + (int64_t)(f == 0 ? B.nField + 6 * B.nLoc : 2 * B.nField + 7 * B.nLoc) * 8 <= P.bytes[f]);
  }
  std::printf("%d/%d/%d ranks %d: %d depths, %d boxes, solo from %d, %d bytes\n", n0, maxBox, block, ranks, nd, P.nbox,
              P.dSolo, P.bytes[0]);
  return 0;
}

int main() {
  const int dir[6] = {0, 0, 0, 0, 0, 0}, mix[6] = {0, 0, 1, 1, 0, 1};
  const bool none[3] = {false, false, false}, px[3] = {true, false, false}, all[3] = {true, true, true};
  check(32, 16, 8, dir, none, 16, 0);
  check(32, 32, 8, mix, none, 16, 0);
  check(24, 24, 8, mix, px, 8, 0);
  check(24, 12, 4, dir, all, 16, 0);
  check(40, 32, 8, mix, none, 16, 1);
  check(64, 4, 4, dir, all, 16, 1);
  check(16, 8, 8, mix, px, 1, 0);
  check(20, 20, 4, dir, none, 8, 0);
  check(48, 24, 8, dir, px, 8, 1);
  std::puts("ok");
}
