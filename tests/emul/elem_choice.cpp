// Prints 1 where the tiled engine is to run a permutation below the element kernel's
// size limits, 0 where the element kernel runs, -1 where its plan declines.
// Input (stdin): cases "es add rank dims perm in_align".
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../../exatensor_b200/csrc/tb_perm_plan.h"

using namespace tb;

int main() {
  int es, add, rank, align;
  while (std::scanf("%d %d %d", &es, &add, &rank) == 3) {
    std::vector<int> dims(rank), perm(rank);
    for (auto& x : dims) if (std::scanf("%d", &x) != 1) return 2;
    for (auto& x : perm) if (std::scanf("%d", &x) != 1) return 2;
    if (std::scanf("%d", &align) != 1) return 2;
    ElemPermParams E;
    if (!build_elem_plan(es, rank, dims.data(), perm.data(), (int64_t)1 << 40, &E)) { std::puts("-1"); continue; }
    std::printf("%d\n", (int)tiled_is_ahead(E, es, add != 0, rank, dims.data(), perm.data(), align));
  }
  return 0;
}
