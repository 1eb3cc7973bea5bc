// tb_direct_plan.cpp -- plans of the one-kernel contraction (host code, no CUDA).
#include "tb_direct_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "../../include/talsh_b200.h"

namespace tb {
namespace {

using namespace direct;

int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

void set_group(Group* o, const MGroup& g) {
  o->ext = (uint32_t)g.ext;
  magic32((uint32_t)g.ext, &o->magic, &o->shift);
  o->s1 = g.s1;
  o->s2 = g.s2;
}

// Drops unit extents and merges neighbours that are contiguous in both strides.
std::vector<MGroup> merged(const std::vector<MGroup>& in) {
  std::vector<MGroup> out;
  for (const MGroup& g : in) {
    if (g.ext == 1) continue;
    if (!out.empty() && g.s1 == out.back().s1 * out.back().ext && g.s2 == out.back().s2 * out.back().ext)
      out.back().ext *= g.ext;
    else
      out.push_back(g);
  }
  return out;
}

int64_t volume(const std::vector<MGroup>& g) {
  int64_t v = 1;
  for (auto& x : g) v *= x.ext;
  return v;
}

int find_unit(const std::vector<MGroup>& g, bool second) {
  for (size_t i = 0; i < g.size(); ++i)
    if ((second ? g[i].s2 : g[i].s1) == 1) return (int)i;
  return -1;
}

// The rows (columns) of one operand for tiles of b of them.
void linear_side(const std::vector<MGroup>& g, int b, Side* S) {
  std::memset(S, 0, sizeof(*S));
  S->ng = (int)g.size();
  for (int i = 0; i < S->ng; ++i) set_group(&S->g[i], g[i]);
  S->count = (uint32_t)volume(g);
  S->tiles = (uint32_t)cdiv(S->count, b);
  S->tp = S->tq = 1;
}
// p: the operand's contiguous group; g[0]: D's fastest.
void box_side(const std::vector<MGroup>& g, int p, int tp, int tq, Side* S) {
  std::memset(S, 0, sizeof(*S));
  const MGroup &P = g[p], &Q = g[0];
  S->box = 1;
  S->tp = tp;
  S->tq = tq;
  S->tp_inv = (65536 + tp - 1) / tp;
  S->tq_inv = (65536 + tq - 1) / tq;
  S->pext = (uint32_t)P.ext;
  S->qext = (uint32_t)Q.ext;
  S->p1 = P.s1; S->p2 = P.s2;
  S->q1 = Q.s1; S->q2 = Q.s2;
  MGroup nq = Q, np = P;
  nq.ext = cdiv(Q.ext, tq);
  np.ext = cdiv(P.ext, tp);
  set_group(&S->nq, nq);
  set_group(&S->np, np);
  int64_t tiles = nq.ext * np.ext;
  for (size_t i = 1; i < g.size(); ++i) {
    if ((int)i == p) continue;
    set_group(&S->g[S->ng++], g[i]);
    tiles *= g[i].ext;
  }
  S->count = (uint32_t)volume(g);
  S->tiles = (uint32_t)std::min<int64_t>(tiles, INT32_MAX);
}

bool overlap(const void* a, int64_t an, const void* b, int64_t bn) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y + (uintptr_t)bn && y < x + (uintptr_t)an;
}

}  // namespace

// The cost model.  Fitted to measured times of every tile shape over random
// contractions; per shape, the share of the FP64 tensor rate (64 multiply-adds
// per clock and SM) that its warps reach with the SM full.
namespace {
constexpr double kEffReal[] = {0.56, 0.60, 0.67, 0.63, 0.67, 0.65, 0.46};
constexpr double kEffCplx[] = {0.97, 0.97, 0.65, 0.68, 0.83, 0.76};
constexpr double kFmaPerUs = 64 * 1900.0;  // per SM
constexpr double kHbmPerUs = 4.4e6;        // bytes
constexpr double kL2PerUs = 8.4e6;
constexpr double kFixedUs = 7.5;           // launch, offset tables and write-out of one round of CTAs
constexpr double kRoundUs = 3.0;           // each further round
constexpr double kKTileUs = 1.05;          // latency of one K tile
// CTAs per SM that fit, by data kind (R4, R8, C4, C8) and shape; and CTAs resident at
// once in clusters of 2, 4 and 8, at one to five per SM: a cluster stays within a GPC,
// so that the larger ones leave SMs empty (cudaOccupancyMaxActiveClusters on B200).
constexpr int kFit[4][7] = {{3, 3, 3, 3, 2, 5, 4}, {3, 3, 3, 3, 2, 3, 2}, {4, 3, 3, 3, 1, 1, 0}, {3, 3, 2, 2, 1, 1, 0}};
constexpr int kResident[3][5] = {{148, 296, 444, 592, 740}, {132, 284, 416, 568, 700}, {120, 264, 384, 568, 688}};
}  // namespace

int plan_direct(const Matricization& Z, int es, bool cplx, const void* d, const void* l, const void* r,
                const std::vector<TileShape>& V, int sms, DirectPlan* out, int force_variant, int force_split,
                int force_box) {
  const int64_t lim = (int64_t)1 << 30;
  if (Z.M > lim || Z.N > lim || Z.K > lim) return TB_ERR_NOT_IMPLEMENTED;
  // an output that overlaps an operand is multiplied from copies (TTGT)
  if (overlap(d, Z.M * Z.N * es, l, Z.M * Z.K * es) || overlap(d, Z.M * Z.N * es, r, Z.N * Z.K * es))
    return TB_ERR_NOT_IMPLEMENTED;
  auto by_d = [](const MGroup& x, const MGroup& y) { return x.s2 < y.s2; };
  std::vector<MGroup> m, n, k;
  for (auto& g : Z.m) if (g.ext > 1) m.push_back(g);
  for (auto& g : Z.n) if (g.ext > 1) n.push_back(g);
  for (auto& g : Z.k) if (g.ext > 1) k.push_back(g);
  std::stable_sort(m.begin(), m.end(), by_d);
  std::stable_sort(n.begin(), n.end(), by_d);
  const bool swap = !n.empty() && (m.empty() || n[0].s2 < m[0].s2);  // the rows hold D's fastest dimension
  if (swap) {
    std::swap(m, n);
    for (auto& g : k) std::swap(g.s1, g.s2);
  }
  const int64_t M = volume(m), N = volume(n), K = volume(k);
  // contracted order: the index that is contiguous in an operand comes first
  // (the larger operand's where both have one), then that operand's order
  {
    const int ka = find_unit(k, false), kb = find_unit(k, true);
    const bool by_b = ka < 0 || (kb >= 0 && N > M);
    std::stable_sort(k.begin(), k.end(), [&](const MGroup& x, const MGroup& y) {
      return by_b && kb >= 0 ? x.s2 < y.s2 : x.s1 < y.s1;
    });
  }
  // columns: the right operand's contiguous group first (each column of D is a run of its own)
  {
    const int u = find_unit(n, false);
    if (u > 0) std::rotate(n.begin(), n.begin() + u, n.begin() + u + 1);
  }
  m = merged(m);
  n = merged(n);
  k = merged(k);
  if (m.size() > kMaxGroups || n.size() > kMaxGroups || k.size() > kMaxGroups) return TB_ERR_NOT_IMPLEMENTED;
  Params& P = out->P;
  std::memset(&P, 0, sizeof(P));
  P.ngk = (int)k.size();
  for (int i = 0; i < P.ngk; ++i) set_group(&P.k[i], k[i]);
  P.K = (uint32_t)K;
  P.a_on_k = !k.empty() && k[0].s1 == 1;
  P.b_on_k = !k.empty() && k[0].s2 == 1;
  const int pm = P.a_on_k ? -1 : find_unit(m, false);  // the rows' contiguous group (0: D's fastest as well)
  const bool b_seq = P.b_on_k || find_unit(n, false) == 0 || N == 1;
  const double sector = 32.0 / es;
  const double dbytes = 2.0 * M * N * es, abytes = (double)M * K * es, bbytes = (double)N * K * es;
  out->us = 1e30;
  for (size_t v = 0; v < V.size(); ++v) {
    if (force_variant >= 0 && (int)v != force_variant) continue;
    const TileShape& sh = V[v];
    for (int box = 0; box < 2; ++box) {
      if (force_box >= 0 && box != force_box) continue;
      int tp = 1, tq = 1;
      double mrows = (double)cdiv(M, sh.bm) * sh.bm, amp = 1.0;
      if (pm > 0) {
        // linear rows still hold runs of the contiguous group when few rows of
        // the groups before it fill less than a tile; L1 serves their sectors
        double before = 1.0;
        for (int i = 0; i < pm; ++i) before *= (double)m[i].ext;
        const double run = std::max(1.0, std::min((double)m[pm].ext, sh.bm / before));
        amp = std::min(sector, (run * es + 32.0 - es) / (run * es));
      } else if (pm < 0 && !P.a_on_k && M > 1) {
        amp = sector;
      }
      if (box) {
        if (pm <= 0 || sh.bm < 32) continue;
        // the box with the least traffic: runs of tp (operand) and tq (D)
        // elements touch about one sector more than they fill
        double best = 1e300;
        const int64_t pe = m[pm].ext, qe = m[0].ext;
        for (int c = 2; c <= 16; ++c) {
          const int64_t p0 = cdiv(pe, cdiv(pe, c)), q0 = cdiv(qe, cdiv(qe, std::max<int64_t>(1, sh.bm / p0)));
          const double ap = (p0 * es + 32.0 - es) / (p0 * es), aq = (q0 * es + 32.0 - es) / (q0 * es);
          const double rows = (double)M / pe / qe * cdiv(pe, p0) * cdiv(qe, q0) * sh.bm;
          const double w = rows * (1.0 + 0.25 * ap + 0.25 * aq);
          if (w < best) { best = w; tp = (int)p0; tq = (int)q0; mrows = rows; amp = ap; }
        }
      }
      const double mt = mrows / sh.bm, nt = (double)cdiv(N, sh.bn);
      const double ktiles = (double)cdiv(K, sh.bkt);
      for (int split = 1; split <= 8; split *= 2) {
        if (force_split > 0 && split != force_split) continue;
        if (split > 1 && (ktiles < 2 * split || mt * nt * (split / 2) >= 2.0 * sms)) continue;
        const double ctas = mt * nt * split;
        if (ctas > 2e9) continue;
        const double kt = std::ceil(ktiles / split);
        const double kk = std::min(kt * sh.bkt, (double)cdiv(K, 4) * 4);
        const double per_sm = std::ceil(ctas / sms);
        const double eff = cplx ? kEffCplx[v] : kEffReal[v];
        const double fma = per_sm * sh.bm * sh.bn * kk * (cplx ? 4 : 1) / (kFmaPerUs * eff);
        const double lat = std::ceil(per_sm / sh.occ) * (kRoundUs + kKTileUs * kt);
        // clusters that do not fit wait for a whole round of the others and then run
        // nearly alone: 416 CTAs in clusters of 8 took 1.5 times their work's time
        double stretch = 1.0;
        if (split > 1) {
          const int fit = kFit[(cplx ? 2 : 0) + (es == (cplx ? 16 : 8) ? 1 : 0)][v], lg = split == 2 ? 0 : split == 4 ? 1 : 2;
          const double full = ctas / kResident[lg][fit - 1] * 148.0 / sms, part = full - std::floor(full);
          if (full > 1.0) stretch = (std::floor(full) + (part > 0.0 ? std::max(0.5, part) : 0.0)) / full;
        }
        const double hbm = (dbytes + abytes + bbytes) / kHbmPerUs;
        const double l2 = (abytes * amp * nt + bbytes * (b_seq ? 1.0 : sector) * mt + dbytes) / kL2PerUs;
        const double us = kFixedUs + std::sqrt(stretch * stretch * (fma * fma + lat * lat) + hbm * hbm + l2 * l2) + 0.5 * (split - 1);
        if (us < out->us) {
          out->us = us;
          out->variant = (int)v;
          out->tp = box ? tp : 0;
          out->tq = tq;
          P.split = split;
        }
      }
    }
  }
  if (out->us >= 1e30) return TB_ERR_NOT_IMPLEMENTED;
  const TileShape& sh = V[out->variant];
  if (out->tp) box_side(m, pm, out->tp, out->tq, &P.m);
  else linear_side(m, sh.bm, &P.m);
  linear_side(n, sh.bn, &P.n);
  const int64_t ctas = (int64_t)P.m.tiles * P.n.tiles * P.split;
  if (ctas > INT32_MAX) return TB_ERR_NOT_IMPLEMENTED;
  out->ctas = ctas;
  P.n_fast = M >= N;
  P.A = swap ? r : l;
  P.B = swap ? l : r;
  P.D = const_cast<void*>(d);
  out->swap = swap;
  return 0;
}

}  // namespace tb
