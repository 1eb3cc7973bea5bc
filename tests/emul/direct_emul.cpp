// Replays the one-kernel contraction's plan and index arithmetic on the CPU:
// every tile, row, column and contracted index that the kernel would visit, in
// exact integers, against a contraction by plain loops over the index digits.
// Input (stdin): cases "drank lrank rrank  ddims  ldims  rdims  cptrn  es cplx
// variant split box"; output: one line per case, "OK ..." or "BAD ...", or
// "DECLINED".
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../exatensor_b200/csrc/tb_direct_plan.h"
#include "../../include/talsh_b200.h"

namespace tb { void set_error(const char*, ...) {} }
using namespace tb;
using namespace tb::direct;

// the kernels' tile shapes (rows, columns, contracted indices, threads, CTAs per SM)
static const std::vector<TileShape> kReal = {{32, 32, 32, 128, 3}, {64, 64, 16, 128, 3}, {128, 32, 16, 128, 3},
                                             {32, 128, 16, 128, 3}, {128, 64, 16, 256, 2}, {128, 16, 16, 128, 3},
                                             {16, 128, 16, 128, 3}};
static const std::vector<TileShape> kCplx = {{32, 32, 16, 128, 3}, {64, 32, 8, 128, 3}, {128, 16, 8, 128, 3},
                                             {16, 128, 8, 128, 3}, {64, 64, 8, 256, 1}, {128, 32, 8, 256, 1}};

int main() {
  int dr, lr, rr;
  while (std::scanf("%d %d %d", &dr, &lr, &rr) == 3) {
    std::vector<int> dd(dr), ld(lr), rd(rr), cp(lr + rr);
    for (auto* v : {&dd, &ld, &rd, &cp})
      for (auto& x : *v)
        if (std::scanf("%d", &x) != 1) return 2;
    int es, cplx, variant, split, box;
    if (std::scanf("%d %d %d %d %d", &es, &cplx, &variant, &split, &box) != 5) return 2;
    Matricization Z;
    if (matricize(cp.data(), dr, dd.data(), lr, ld.data(), rr, rd.data(), &Z)) { std::puts("BAD pattern"); continue; }
    const int64_t nd = Z.M * Z.N, nl = Z.M * Z.K, nr = Z.N * Z.K;
    std::vector<int64_t> L(nl), R(nr), D(nd), ref(nd);
    for (int64_t i = 0; i < nl; ++i) L[i] = (i * 2654435761u >> 7) % 211 - 105;
    for (int64_t i = 0; i < nr; ++i) R[i] = (i * 40503u >> 3) % 197 - 98;
    // plain loops over the groups' digits
    auto at = [](const std::vector<MGroup>& g, int64_t i, bool second) {
      int64_t o = 0;
      for (auto& x : g) { o += (i % x.ext) * (second ? x.s2 : x.s1); i /= x.ext; }
      return o;
    };
    for (int64_t m = 0; m < Z.M; ++m)
      for (int64_t n = 0; n < Z.N; ++n) {
        int64_t s = 0;
        for (int64_t k = 0; k < Z.K; ++k)
          s += L[at(Z.m, m, false) + at(Z.k, k, false)] * R[at(Z.n, n, false) + at(Z.k, k, true)];
        ref[at(Z.m, m, true) + at(Z.n, n, true)] = s;
      }
    DirectPlan pl;
    const std::vector<TileShape>& sh = cplx ? kCplx : kReal;
    const int e = plan_direct(Z, es, cplx != 0, (void*)0x100000000000, (void*)0x200000000000, (void*)0x300000000000, sh,
                              148, &pl, variant, split, box);
    if (e == TB_ERR_NOT_IMPLEMENTED) { std::puts("DECLINED"); continue; }
    if (e) { std::puts("BAD plan"); continue; }
    const Params& P = pl.P;
    const TileShape& T = sh[pl.variant];
    const std::vector<int64_t>& A = pl.swap ? R : L;
    const std::vector<int64_t>& B = pl.swap ? L : R;
    std::vector<int> written(nd, 0);
    const char* bad = nullptr;
    const int ktiles = (int)((P.K + T.bkt - 1) / T.bkt);
    if (pl.ctas != (int64_t)P.m.tiles * P.n.tiles * P.split) bad = "grid";
    for (int64_t cta = 0; cta < pl.ctas / P.split && !bad; ++cta) {
      uint32_t mt, nt;
      if (P.n_fast) { mt = cta / P.n.tiles; nt = cta % P.n.tiles; } else { nt = cta / P.m.tiles; mt = cta % P.m.tiles; }
      std::vector<int64_t> ra(T.bm), rb(T.bn), dm(T.bm), dn(T.bn);
      for (int i = 0; i < T.bm; ++i) side_offsets(P.m, mt, T.bm, i, ra[i], dm[i]);
      for (int i = 0; i < T.bn; ++i) side_offsets(P.n, nt, T.bn, i, rb[i], dn[i]);
      std::vector<int64_t> acc((size_t)T.bm * T.bn, 0);
      for (int rank = 0; rank < P.split; ++rank) {
        const int k0 = (int)((int64_t)ktiles * rank / P.split), k1 = (int)((int64_t)ktiles * (rank + 1) / P.split);
        for (int64_t k = (int64_t)k0 * T.bkt; k < (int64_t)k1 * T.bkt && k < P.K; ++k) {
          int64_t oa = 0, ob = 0;
          digits(P.k, P.ngk, (uint32_t)k, oa, ob);
          for (int i = 0; i < T.bm; ++i) {
            if (ra[i] < 0) continue;
            if (ra[i] + oa >= (int64_t)A.size()) { bad = "A offset"; break; }
            for (int j = 0; j < T.bn; ++j) {
              if (rb[j] < 0) continue;
              if (rb[j] + ob >= (int64_t)B.size()) { bad = "B offset"; break; }
              acc[(size_t)j * T.bm + i] += A[ra[i] + oa] * B[rb[j] + ob];
            }
          }
        }
      }
      // a staged box tile: every row of the box at a position of its own inside
      // the skewed pitch, and gathered by one lane
      if (P.m.box) {
        std::vector<int> used(T.bm + 16, 0), lane(T.bm, 0);
        for (int i = 0; i < T.bm; ++i) {
          const int p = small_div(i, P.m.tq_inv);
          if (p != i / P.m.tq || small_div(i, P.m.tp_inv) != i / P.m.tp) bad = "small_div";
          if (p >= P.m.tp) { if (ra[i] >= 0) bad = "row past the box"; continue; }
          const int pos = box_position(p, i - p * P.m.tq, P.m.tq);
          if (pos < 0 || pos >= T.bm + 16 || used[pos]++) bad = "box position";
        }
        for (int r = 0; r < T.bm; ++r) {
          const int q = small_div(r, P.m.tp_inv), p = r - q * P.m.tp;
          if (q < P.m.tq) ++lane[q + p * P.m.tq];
        }
        for (int i = 0; i < P.m.tp * P.m.tq; ++i) if (lane[i] != 1) bad = "box lanes";
        if (P.m.tp * P.m.tq > T.bm) bad = "box size";
      }
      for (int j = 0; j < T.bn && !bad; ++j)
        for (int i = 0; i < T.bm; ++i) {
          if (dm[i] < 0 || dn[j] < 0) continue;
          const int64_t o = dm[i] + dn[j];
          if (o >= nd) { bad = "D offset"; break; }
          ++written[o];
          D[o] = acc[(size_t)j * T.bm + i];
        }
    }
    for (int64_t o = 0; o < nd && !bad; ++o) {
      if (written[o] != 1) bad = "D written";
      else if (D[o] != ref[o]) bad = "D value";
    }
    if (bad) std::printf("BAD %s\n", bad);
    else std::printf("OK variant=%d split=%d box=%d swap=%d a_on_k=%d b_on_k=%d\n", pl.variant, P.split, P.m.box, (int)pl.swap, P.a_on_k, P.b_on_k);
  }
  return 0;
}
