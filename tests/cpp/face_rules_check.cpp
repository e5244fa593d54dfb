// A level's face rules are made when something that reads them asks: not with
// the plan, whatever the level's size, and then for every face cell.
#include <cstdio>
#include <cstdlib>

#include "../../chombo_3.2_b200/csrc/plan.H"

using namespace cmg;

#define REQUIRE(c)                                                     \
  do {                                                                 \
    if (!(c)) {                                                        \
      std::printf("line %d: %s\n", __LINE__, #c);                      \
      std::exit(1);                                                    \
    }                                                                  \
  } while (0)

int main() {
  for (int n : {8, 32, 64}) {  // 32^3 cells were the most that had them with the plan
    const Box dom(IV{0, 0, 0}, IV{n - 1, n - 1, n - 1});
    LevelPlan L;
    buildLevel(L, Layout(domainSplit(dom, 16, 8)), dom, 1.0 / n, 0.0);
    REQUIRE(L.faceOff.empty() && L.faceRules.empty());
    int64_t faces = 0;
    for (const Box& b : L.grids.boxes)
      for (int d = 0; d < 3; ++d) faces += 2 * b.numPts() / b.size(d);
    REQUIRE(ensureChunkGhosts(L));
    REQUIRE((int64_t)L.faceRules.size() == faces && L.faceOff.back() == faces);
    REQUIRE(!L.chunkGhost[0].empty() && !ensureFaceRules(L) && !ensureChunkGhosts(L));
  }
  std::puts("ok");
}
