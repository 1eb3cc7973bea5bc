// tb_direct.cuh -- contractions in one kernel, in the tensors' own layouts.
//
//   D[dm(m) + dn(n)] = beta D + alpha sum_k op(A)[am(m) + ak(k)] op(B)[bn(n) + bk(k)]
//
// The plain (TTGT) method permutes both operands into matrices, multiplies, and
// permutes the product into D: up to four kernels, three scratch matrices and,
// for a product with a short contracted index, four passes over D instead of
// two.  Here a CTA computes the offsets of its tile's rows, columns and
// contracted indices itself, gathers the operand tiles with cp.async straight
// into the multiplication's shared-memory layout, and writes D through its
// offsets.  What bounds it: D's traffic for short contracted indices, FP64
// tensor throughput (by mma.sync m8n8k4; the larger FP64 shapes are not tried) for
// long ones, and the launch for small ones.  Measured, us, TTGT / this: 121 x 25 x
// 121 R8 54 / 12; 324 x 325 x 104 R8 49 / 13; 6859 x 6859 x 19 R8 (752 MB of D traffic)
// 520 / 239; R4 index transform 373248 x 24 x 72 245 / 117.  Staging every product in
// shared memory before writing D cost the third 352.
//
// All data kinds accumulate in FP64 (R4 and C4 are widened when fragments are
// read, which costs a conversion per 16 multiply-adds), so no sum is less exact
// than the tensor's own type gives.
#pragma once
#include <cooperative_groups.h>

#include <type_traits>

#include "tb_async.cuh"
#include "tb_common.cuh"
#include "tb_direct_plan.h"

namespace tb {
namespace direct {

template <typename E>
struct Elem {
  static constexpr bool CPLX = std::is_same<E, float2>::value || std::is_same<E, double2>::value;
  static constexpr bool F32 = std::is_same<E, float>::value || std::is_same<E, float2>::value;
  using R = typename std::conditional<F32, float, double>::type;
  using Acc = typename std::conditional<CPLX, double2, double>::type;
};

// Shared-memory pitches that keep both the gathers' writes and the fragment
// reads (8 rows x 4 contracted indices per warp) free of bank conflicts:
// [row][k] rows of BK + 4 elements, [k][row] rows of rows + a pad; the left
// side's pad also holds a box's skew of one element per p (box_position).
template <typename E>
constexpr int pad_b() { return sizeof(E) == 4 ? 8 : (sizeof(E) == 8 ? 4 : 2); }
template <typename E>
constexpr int pad_a() { return 16 + pad_b<E>(); }
constexpr int tile_elems(int rows, int bk, int pad) {
  return rows * (bk + 4) > bk * (rows + pad) ? rows * (bk + 4) : bk * (rows + pad);
}
constexpr int kStagePad = 2;  // staged product columns: rows + 2 (mod 8 = 2: conflict-free fragment writes)

// WM x WN warps of (8 MI) x (8 NI) tiles, KW warp groups sharing each K tile of
// KW * BK indices (their sums are added in group order), ST pipeline stages.
template <typename E, int WM, int WN, int KW, int MI, int NI, int BK, int ST>
struct Shape {
  static constexpr int BM = WM * MI * 8, BN = WN * NI * 8, BKT = BK * KW, T = WM * WN * KW * 32;
  static constexpr int SA = tile_elems(BM, BKT, pad_a<E>()), SB = tile_elems(BN, BKT, pad_b<E>());
  static constexpr size_t table_bytes() { return (size_t)(2 * (BM + BN) + 2 * (ST + 1) * BKT) * 8; }
  static constexpr size_t smem(bool staged) {
    const size_t pipe = (size_t)ST * (SA + SB) * sizeof(E);
    const size_t stage = (size_t)KW * BN * (BM + kStagePad) * sizeof(typename Elem<E>::Acc);
    return table_bytes() + (staged && stage > pipe ? stage : pipe);
  }
};

template <typename E, typename R>
__device__ __forceinline__ void update(const Params& P, bool read_d, E* d, const double& v, const E& old) {
  const double x = P.ar * v;
  *d = (E)(read_d ? fma(P.br, (double)old, x) : x);
}
template <typename E, typename R>
__device__ __forceinline__ void update(const Params& P, bool read_d, E* d, const double2& v, const E& old) {
  double x = P.ar * v.x - P.ai * v.y, y = P.ar * v.y + P.ai * v.x;
  if (read_d) {
    x += P.br * (double)old.x - P.bi * (double)old.y;
    y += P.br * (double)old.y + P.bi * (double)old.x;
  }
  E w;
  w.x = (R)x;
  w.y = (R)y;
  *d = w;
}

// Word: nothing, or the address of a word without which set the kernel does nothing (a
// kernel of its own, since waiting for one parameter before all others costs every
// launch 0.4 us).
template <typename E, int WM, int WN, int KW, int MI, int NI, int BK, int ST, int OCC, class... Word>
__global__ void __launch_bounds__(WM* WN* KW * 32, OCC) direct_kernel(const __grid_constant__ Params P, Word... when) {
  using S = Shape<E, WM, WN, KW, MI, NI, BK, ST>;
  using R = typename Elem<E>::R;
  using Acc = typename Elem<E>::Acc;
  constexpr bool CPLX = Elem<E>::CPLX;
  constexpr int BM = S::BM, BN = S::BN, BKT = S::BKT, T = S::T, NC = CPLX ? 2 : 1;
  if constexpr (sizeof...(Word) > 0) {
    if ((!*when || ...)) return;
  }
  extern __shared__ __align__(16) unsigned char direct_smem[];
  int64_t* row_a = reinterpret_cast<int64_t*>(direct_smem);
  int64_t* row_b = row_a + BM;
  int64_t* dm = row_b + BN;
  int64_t* dn = dm + BM;
  int64_t* koff = dn + BN;  // [ST + 1][2][BKT]: A and B offsets of a K tile's indices
  E* pipe = reinterpret_cast<E*>(direct_smem + S::table_bytes());
  Acc* stage = reinterpret_cast<Acc*>(direct_smem + S::table_bytes());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kw = warp / (WM * WN), wm = (warp / WN) % WM, wn = warp % WN;
  const int g = lane >> 2, t = lane & 3;
  const uint32_t split = (uint32_t)P.split;
  const uint32_t rank = split > 1 ? blockIdx.x % split : 0u;
  const uint32_t tile = split > 1 ? blockIdx.x / split : blockIdx.x;
  uint32_t mt, nt;
  if (P.n_fast) { mt = tile / P.n.tiles; nt = tile - mt * P.n.tiles; }
  else { nt = tile / P.m.tiles; mt = tile - nt * P.m.tiles; }
  const int ktiles_all = (int)((P.K + BKT - 1) / BKT);
  const int kt0 = (int)((int64_t)ktiles_all * rank / split), kt1 = (int)((int64_t)ktiles_all * (rank + 1) / split);

  for (int i = tid; i < BM + BN; i += T) {
    int64_t o1, o2;
    if (i < BM) { side_offsets(P.m, mt, BM, i, o1, o2); row_a[i] = o1; dm[i] = o2; }
    else { side_offsets(P.n, nt, BN, i - BM, o1, o2); row_b[i - BM] = o1; dn[i - BM] = o2; }
  }
  auto k_offsets = [&](int kt, int i) {  // entry i of K tile kt
    const uint32_t k = (uint32_t)kt * BKT + (uint32_t)i;
    int64_t oa = 0, ob = 0;
    if (k < P.K) digits(P.k, P.ngk, k, oa, ob);
    else oa = ob = -1;
    int64_t* s = koff + (size_t)(kt % (ST + 1)) * 2 * BKT;
    s[i] = oa;
    s[BKT + i] = ob;
  };
  for (int e = tid; e < ST * BKT; e += T) {
    const int kt = kt0 + e / BKT;
    if (kt < kt1) k_offsets(kt, e % BKT);
  }
  // strides of (row, k) in a staged tile
  const int am = P.a_on_k ? BKT + 4 : 1, ak = P.a_on_k ? 1 : BM + pad_a<E>();
  const int bm = P.b_on_k ? BKT + 4 : 1, bk = P.b_on_k ? 1 : BN + pad_b<E>();
  const bool box = P.m.box != 0;
  const int tp = P.m.tp, tq = P.m.tq;
  auto issue = [&](int kt) {
    const int st = kt % ST;
    const int64_t* ko = koff + (size_t)(kt % (ST + 1)) * 2 * BKT;
    const int kend = ((int)P.K - kt * BKT + 3) & ~3;  // the multiplication reads whole groups of four
    E* sa = pipe + (size_t)st * (S::SA + S::SB);
    E* sb = sa + S::SA;
    // A thread's copies share one contracted index (lanes along k) or one row
    // (lanes along rows); the other index steps by a constant, so a copy costs a
    // table read, an addition and two predicates.
    auto side = [&](auto rows_c, const E* src, E* dst, const int64_t* row, const int64_t* kof, bool on_k, bool bx, int pitch) {
      constexpr int ROWS = decltype(rows_c)::value;
      static_assert(T % ROWS == 0 && T % BKT == 0 && ROWS * BKT % T == 0, "whole gather rounds");
      constexpr int IT = ROWS * BKT / T;
      if (on_k) {
        const int kk = tid % BKT, r0 = tid / BKT;
        if (kk >= kend) return;
        const int64_t kf = kof[kk];
        const E* base = src + (kf < 0 ? 0 : kf);
        E* d = dst + r0 * pitch + kk;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
          const int64_t ro = row[r0 + it * (T / BKT)];
          const bool ok = (ro | kf) >= 0;
          cp_async_elem<(int)sizeof(E)>(d + it * (T / BKT) * pitch, base + (ok ? ro : 0), ok);
        }
      } else {
        int r = tid % ROWS, pos = r;
        const int k0 = tid / ROWS;
        if (bx) {  // lanes along the operand's contiguous group p
          const int q = small_div(r, P.m.tp_inv), p = r - q * tp;
          if (q >= tq) return;
          r = q + p * tq;
          pos = box_position(p, q, tq);
        }
        const int64_t ro = row[r];
        const E* base = src + (ro < 0 ? 0 : ro);
        E* d = dst + pos + k0 * pitch;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
          const int kk = k0 + it * (T / ROWS);
          if (kk >= kend) break;
          const int64_t kf = kof[kk];
          const bool ok = (ro | kf) >= 0;
          cp_async_elem<(int)sizeof(E)>(d + it * (T / ROWS) * pitch, base + (ok ? kf : 0), ok);
        }
      }
    };
    side(std::integral_constant<int, BM>{}, (const E*)P.A, sa, row_a, ko, P.a_on_k != 0, box, P.a_on_k ? am : ak);
    side(std::integral_constant<int, BN>{}, (const E*)P.B, sb, row_b, ko + BKT, P.b_on_k != 0, false, P.b_on_k ? bm : bk);
  };
  double acc[NC][MI][NI][2];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j) acc[c][i][j][0] = acc[c][i][j][1] = 0.0;
  __syncthreads();
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) {
    if (kt0 + s < kt1) issue(kt0 + s);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  // D's elements of this thread: rows wm * 8 MI + 8 i + g, columns wn * 8 NI +
  // 8 j + 2 t + h.  Those of the first half of the rows are read while the
  // operands arrive, so that a short contracted range does not wait for them
  // afterwards.
  const bool read_d = P.br != 0.0 || P.bi != 0.0;
  const bool staged = KW > 1 || split > 1;
  constexpr int H = MI / 2;
  E* D = (E*)P.D;
  E old[H][NI][2];
  auto d_offset = [&](int i, int j, int h) -> int64_t {
    const int64_t om = dm[wm * MI * 8 + i * 8 + g], on = dn[wn * NI * 8 + j * 8 + 2 * t + h];
    return (om | on) < 0 ? -1 : om + on;
  };
  auto read_old = [&](int i0) {
#pragma unroll
    for (int i = 0; i < H; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int64_t o = d_offset(i0 + i, j, h);
          if (o >= 0) old[i][j][h] = D[o];
        }
  };
  if (KW == 1 && !staged && read_d) read_old(0);
  int arow[MI];  // this thread's fragment rows in a staged left tile
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = wm * MI * 8 + i * 8 + g;
    const int p = small_div(r, P.m.tq_inv);
    arow[i] = !box ? r * am : p < tp ? box_position(p, r - p * tq, tq) : 0;
  }
  const double sga = P.aconj ? -1.0 : 1.0, sgb = P.bconj ? -1.0 : 1.0;
  for (int kt = kt0; kt < kt1; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(ST - 2) : "memory");
    __syncthreads();
    if (kt + ST - 1 < kt1) issue(kt + ST - 1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (kt + ST < kt1 && tid < BKT) k_offsets(kt + ST, tid);
    const E* sa = pipe + (size_t)(kt % ST) * (S::SA + S::SB);
    const E* pa = sa + (kw * BK + t) * ak;
    const E* pb = sa + S::SA + (wn * NI * 8 + g) * bm + (kw * BK + t) * bk;
    const int kleft = (int)P.K - kt * BKT - kw * BK;  // this group's indices left
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      if (kk >= kleft) break;
      if constexpr (!CPLX) {
        double a[MI], b[NI];
#pragma unroll
        for (int i = 0; i < MI; ++i) a[i] = (double)pa[arow[i] + kk * ak];
#pragma unroll
        for (int j = 0; j < NI; ++j) b[j] = (double)pb[j * 8 * bm + kk * bk];
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < NI; ++j) dmma(acc[0][i][j][0], acc[0][i][j][1], a[i], b[j]);
      } else {
        double ax[MI], ay[MI], bx[NI], by[NI];
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          const E v = pa[arow[i] + kk * ak];
          ax[i] = (double)v.x;
          ay[i] = sga * (double)v.y;
        }
#pragma unroll
        for (int j = 0; j < NI; ++j) {
          const E v = pb[j * 8 * bm + kk * bk];
          bx[j] = (double)v.x;
          by[j] = sgb * (double)v.y;
        }
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < NI; ++j) {
            dmma(acc[0][i][j][0], acc[0][i][j][1], ax[i], bx[j]);
            dmma(acc[0][i][j][0], acc[0][i][j][1], -ay[i], by[j]);
            dmma(acc[NC - 1][i][j][0], acc[NC - 1][i][j][1], ax[i], by[j]);
            dmma(acc[NC - 1][i][j][0], acc[NC - 1][i][j][1], ay[i], bx[j]);
          }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if constexpr (KW == 1) {
    if (!staged) {
#pragma unroll
      for (int i0 = 0; i0 < MI; i0 += H) {
        if (i0 && read_d) read_old(i0);
#pragma unroll
        for (int i = 0; i < H; ++i)
#pragma unroll
          for (int j = 0; j < NI; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int64_t o = d_offset(i0 + i, j, h);
              if (o < 0) continue;
              if constexpr (CPLX)
                update<E, R>(P, read_d, D + o, make_double2(acc[0][i0 + i][j][h], acc[NC - 1][i0 + i][j][h]), old[i][j][h]);
              else
                update<E, R>(P, read_d, D + o, acc[0][i0 + i][j][h], old[i][j][h]);
            }
      }
      return;
    }
  }
  __syncthreads();  // the pipeline's buffers become the staging area
  // staged product: [kw][column][row]
  constexpr int SP = BM + kStagePad;
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = wm * MI * 8 + i * 8 + g, n = wn * NI * 8 + j * 8 + 2 * t + h;
        Acc* s = stage + ((size_t)kw * BN + n) * SP + r;
        if constexpr (CPLX) *s = make_double2(acc[0][i][j][h], acc[NC - 1][i][j][h]);
        else *s = acc[0][i][j][h];
      }
  namespace cg = cooperative_groups;
  if (split > 1) cg::this_cluster().sync();
  else __syncthreads();
  // each CTA of a cluster finishes its share of the tile's columns, adding the
  // CTAs' and warp groups' sums in order
  const int c0 = (int)(BN * rank / split), c1 = (int)(BN * (rank + 1) / split);
  constexpr int U = 8;
  for (int e0 = tid + c0 * BM; e0 < c1 * BM; e0 += U * T) {
    int64_t off[U];
    E prev[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * T;
      off[u] = -1;
      if (e >= c1 * BM) continue;
      const int64_t om = dm[e % BM], on = dn[e / BM];
      if ((om | on) < 0) continue;
      off[u] = om + on;
      if (read_d) prev[u] = D[off[u]];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (off[u] < 0) continue;
      const int e = e0 + u * T;
      Acc v;
      if constexpr (CPLX) v = make_double2(0.0, 0.0);
      else v = 0.0;
      for (uint32_t r = 0; r < split; ++r) {
        const Acc* s = split > 1 ? cg::this_cluster().map_shared_rank(stage, r) : stage;
#pragma unroll
        for (int w = 0; w < KW; ++w) {
          const Acc y = s[((size_t)w * BN + e / BM) * SP + e % BM];
          if constexpr (CPLX) { v.x += y.x; v.y += y.y; }
          else v += y;
        }
      }
      update<E, R>(P, read_d, D + off[u], v, prev[u]);
    }
  }
  if (split > 1) cg::this_cluster().sync();  // no CTA leaves while another reads its staged sums
}

}  // namespace direct
}  // namespace tb
