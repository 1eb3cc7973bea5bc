// Replays the element permutation's order on the CPU: every element moved once,
// from the right place, all offsets inside the tensor.  Input (stdin): cases "es
// rank dims perm"; output: OK, DECLINED or BAD per case.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../../exatensor_b200/csrc/tb_perm_plan.h"

using namespace tb;

int main() {
  int es, rank;
  while (std::scanf("%d %d", &es, &rank) == 2) {
    std::vector<int> dims(rank), perm(rank);
    for (auto& x : dims) if (std::scanf("%d", &x) != 1) return 2;
    for (auto& x : perm) if (std::scanf("%d", &x) != 1) return 2;
    ElemPermParams P;
    if (!build_elem_plan(es, rank, dims.data(), perm.data(), (int64_t)1 << 40, &P)) { std::puts("DECLINED"); continue; }
    int64_t vol = 1;
    std::vector<int64_t> so(rank);
    for (int x : dims) vol *= x;
    {
      std::vector<int64_t> oe(rank);
      for (int i = 0; i < rank; ++i) oe[perm[i] - 1] = dims[i];
      int64_t s = 1;
      std::vector<int64_t> pos(rank);
      for (int q = 0; q < rank; ++q) { pos[q] = s; s *= oe[q]; }
      for (int i = 0; i < rank; ++i) so[i] = pos[perm[i] - 1];
    }
    std::vector<int64_t> want(vol);
    for (int64_t i = 0; i < vol; ++i) {
      int64_t r = i, o = 0;
      for (int k = 0; k < rank; ++k) { o += r % dims[k] * so[k]; r /= dims[k]; }
      want[i] = o;
    }
    std::vector<char> seen(vol, 0);
    bool ok = P.vol == (uint64_t)vol;
    for (uint32_t i = 0; ok && i < P.vol; ++i) {
      uint32_t rest = i, a = 0;
      for (int d = 0; d < P.rank - 1; ++d) elem_digit(P, d, &rest, &a);
      a += rest * P.sin[P.rank - 1];
      if (a >= vol || seen[a]++ || want[a] != (int64_t)i) ok = false;
    }
    std::puts(ok ? "OK" : "BAD");
  }
  return 0;
}
