// tb_direct_plan.h -- plans of the one-kernel contraction (tb_direct.cuh): which
// index groups run along a tile's rows, columns and contracted values, and the
// offsets of a tile's indices.  Host code without CUDA, shared with the kernel
// and with the CPU test of its index arithmetic.
#pragma once
#include <cstdint>
#include <vector>

#include "tb_fastdiv.h"
#include "tb_pattern.h"

namespace tb {
namespace direct {

constexpr int kMaxGroups = 12;  // index groups per side after merging; more go to TTGT

struct Group {
  uint32_t ext, magic;  // extent and its 32-bit magic divisor (fdiv32)
  int shift;
  int64_t s1, s2;       // strides: operand and D (rows, columns); A and B (contracted)
};

// Rows (columns) of one operand.  Linear: index i of tile t is t * tile + i,
// digits taken group by group.  Box: the operand's contiguous group p and D's
// fastest group q are different, and a tile is a box of tp x tq of them (i = q +
// tq * p; rows from tp * tq up to the tile's size stay empty), so that both the gather and the
// writes of D run along contiguous elements; the tile number takes the box's position and the
// remaining groups.
struct Side {
  int ng, box;
  uint32_t count;            // linear: rows in all
  uint32_t tiles;
  int tp, tq;
  uint32_t tp_inv, tq_inv;   // small_div magics
  uint32_t pext, qext;
  int64_t p1, p2, q1, q2;    // strides of p and q: operand, D
  Group nq, np;              // boxes along q and p (ext, divisor)
  Group g[kMaxGroups];
};

struct Params {
  const void* A;
  const void* B;
  void* D;
  Side m, n;
  int ngk;
  uint32_t K;
  Group k[kMaxGroups];
  int a_on_k, b_on_k;        // gather lanes run along the contracted index (else along rows / columns)
  int n_fast;                // consecutive CTAs step along columns (else along rows)
  int split;                 // CTAs of a cluster that share a tile's contracted range
  double ar, ai, br, bi;
  int aconj, bconj;
};

TB_HD void digits(const Group* g, int ng, uint32_t i, int64_t& o1, int64_t& o2) {
  for (int j = 0; j < ng; ++j) {
    const uint32_t q = fdiv32(i, g[j].magic, g[j].shift);
    const int64_t x = (int64_t)(i - q * g[j].ext);
    o1 += x * g[j].s1;
    o2 += x * g[j].s2;
    i = q;
  }
}

// i / d for 0 <= i < 256, 1 <= d <= 128, inv = ceil(2^16 / d).
TB_HD int small_div(int i, uint32_t inv) { return (int)(((uint32_t)i * inv) >> 16); }

// Where row (p, q) of a box tile sits in a staged [k][row] tile: a skew of one
// element per p spreads the gather's writes along p over the banks.
TB_HD int box_position(int p, int q, int tq) { return q + p * (tq + 1); }

// Offsets of index i of a tile in the operand and in D (both -1 past the edge).
TB_HD void side_offsets(const Side& S, uint32_t tile, int bsize, int i, int64_t& o1, int64_t& o2) {
  o1 = o2 = 0;
  if (S.box) {
    uint32_t r = tile;
    uint32_t t = fdiv32(r, S.nq.magic, S.nq.shift);
    const int ip = small_div(i, S.tq_inv);
    const uint32_t q = (r - t * S.nq.ext) * (uint32_t)S.tq + (uint32_t)(i - ip * S.tq);
    r = t;
    t = fdiv32(r, S.np.magic, S.np.shift);
    const uint32_t p = (r - t * S.np.ext) * (uint32_t)S.tp + (uint32_t)ip;
    digits(S.g, S.ng, t, o1, o2);
    o1 += (int64_t)p * S.p1 + (int64_t)q * S.q1;
    o2 += (int64_t)p * S.p2 + (int64_t)q * S.q2;
    if (ip >= S.tp || p >= S.pext || q >= S.qext) o1 = o2 = -1;
  } else {
    const uint32_t m = tile * (uint32_t)bsize + (uint32_t)i;
    if (m < S.count) digits(S.g, S.ng, m, o1, o2);
    else o1 = o2 = -1;
  }
}

}  // namespace direct

// A tile shape: rows, columns, contracted indices per K tile, threads, CTAs
// per SM that its registers and shared memory allow.
struct TileShape { int bm, bn, bkt, threads, occ; };

struct DirectPlan {
  direct::Params P;
  int64_t ctas;
  int variant, tp, tq;  // tp: 0 without a box
  bool swap;   // the rows come from R
  double us;   // predicted time
};

// Plans the one-kernel form of a contraction over the given tile shapes.
// Returns TB_ERR_NOT_IMPLEMENTED for what it leaves to the other methods: more
// than 2^30 rows, columns or contracted values, more index groups than its
// parameter block holds, or an output that overlaps an operand.  The forced
// values (>= 0; split > 0) pin the tile shape, K split and row boxes (the CPU
// replay of the index arithmetic goes through all of them).
int plan_direct(const Matricization& Z, int es, bool cplx, const void* d, const void* l, const void* r,
                const std::vector<TileShape>& shapes, int sms, DirectPlan* out, int force_variant = -1,
                int force_split = 0, int force_box = -1);

}  // namespace tb
