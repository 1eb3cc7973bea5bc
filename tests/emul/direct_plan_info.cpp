// Prints which tile shape, K split and row box the one-kernel contraction's planner
// (tb_direct_plan.cpp) takes, and the time it predicts.
// Input (stdin): cases "drank lrank rrank  ddims  ldims  rdims  cptrn  es cplx";
// output: "variant split box a_on_k b_on_k us" per case, or "DECLINED".
#define main emul_main  // the tile shapes are the emulation's
#include "direct_emul.cpp"
#undef main

int main() {
  int dr, lr, rr;
  while (std::scanf("%d %d %d", &dr, &lr, &rr) == 3) {
    std::vector<int> dd(dr), ld(lr), rd(rr), cp(lr + rr);
    for (auto* v : {&dd, &ld, &rd, &cp})
      for (auto& x : *v)
        if (std::scanf("%d", &x) != 1) return 2;
    int es, cplx;
    if (std::scanf("%d %d", &es, &cplx) != 2) return 2;
    Matricization Z;
    DirectPlan pl;
    if (matricize(cp.data(), dr, dd.data(), lr, ld.data(), rr, rd.data(), &Z) ||
        plan_direct(Z, es, cplx != 0, (void*)0x100000000000, (void*)0x200000000000, (void*)0x300000000000,
                    cplx ? kCplx : kReal, 148, &pl)) {
      std::puts("DECLINED");
      continue;
    }
    std::printf("%d %d %d %d %d %.1f\n", pl.variant, pl.P.split, pl.P.m.box, pl.P.a_on_k, pl.P.b_on_k, pl.us);
  }
  return 0;
}
