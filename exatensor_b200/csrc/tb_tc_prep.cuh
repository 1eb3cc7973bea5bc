// tb_tc_prep.cuh -- operand preparation for the tensor-core contractions:
// TMA tensor maps over operand planes, offset tables, row exponent maxima, and
// the gathers that convert operands (read through offset tables, so that the
// input permutation is fused) into INT8 slice planes or BF16 parts.  Each
// kernel exists in a dense form (one operand per launch) and a grouped form
// (a table of operand jobs per launch, for block-sparse contractions).
#pragma once
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include "tb_async.cuh"
#include "tb_common.cuh"
#include "tb_pattern.h"
#include "tb_tc_gemm.cuh"

namespace tb {
namespace {

// ---- TMA tensor maps (driver entry point, no libcuda link) --------------------
PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  });
  return fn;
}

// 3-D map over planes of [rows][kpad] K-major operands, 128-byte rows per box.
int make_operand_map(CUtensorMap* map, const void* base, bool i8, int64_t kpad, int64_t rows, int planes,
                     int box_rows) {
  auto enc = get_encode();
  if (!enc) { set_error("cuTensorMapEncodeTiled is unavailable"); return TB_ERR_CUDA; }
  const int es = i8 ? 1 : 2;
  cuuint64_t dims[3] = {(cuuint64_t)kpad, (cuuint64_t)rows, (cuuint64_t)planes};
  cuuint64_t strides[2] = {(cuuint64_t)(kpad * es), (cuuint64_t)(kpad * es * rows)};
  cuuint32_t box[3] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                   const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d)", (int)r); return TB_ERR_CUDA; }
  return 0;
}

// ---- offset tables ----------------------------------------------------------------
// o1[i] = sum_g digit_g(i) s1_g and o2[i] with s2_g, first group fastest.  Rows
// whose operand is contiguous along another group than D run in blocks of eight
// of that group (group 0, with its remaining positions the last group): i counts
// whole blocks first, then the `tail` positions left over, so that no row is
// padding and both the gathers (eight elements in a row) and the writes of D
// (rows eight apart) stay coalesced.
struct TableJob {
  int ng;
  int64_t count, full;        // rows; rows in whole blocks (= count without a tail)
  int64_t base1, base2;       // offsets of the tail
  int64_t tail;               // extent of group 0 in the tail
  FastDiv tail_div;
  int64_t* o1;
  int64_t* o2;
  int64_t ext[kMaxRank], s1[kMaxRank], s2[kMaxRank];
  FastDiv div[kMaxRank];
};
struct TableParams {
  TableJob job[3];            // rows of A, rows of B, contracted indices
  unsigned first[3];          // first CTA of each job
  unsigned zero_cta;          // first CTA that clears words
  uint32_t* zero;
  int64_t zero_words;
};

__device__ __forceinline__ void table_job(const TableJob& J, int64_t cta, int64_t ctas) {
  for (int64_t i = cta * blockDim.x + threadIdx.x; i < J.count; i += ctas * blockDim.x) {
    const bool tail = i >= J.full;
    uint64_t r = (uint64_t)(tail ? i - J.full : i);
    int64_t a = tail ? J.base1 : 0, b = tail ? J.base2 : 0;
    for (int g = 0; g < J.ng; ++g) {
      const bool t0 = tail && g == 0;
      const uint64_t q = t0 ? J.tail_div.div(r) : J.div[g].div(r);
      const int64_t x = (int64_t)(r - q * (uint64_t)(t0 ? J.tail : J.ext[g]));
      a += x * J.s1[g];
      b += x * J.s2[g];
      r = q;
    }
    J.o1[i] = a;
    J.o2[i] = b;
  }
}

// All offset tables of a contraction, and the words that its other kernels
// expect cleared (row maxima, counters), in one launch.
__global__ void __launch_bounds__(256) tables_kernel(const __grid_constant__ TableParams P) {
  const unsigned x = blockIdx.x;
  if (x >= P.zero_cta) {
    for (int64_t i = (x - P.zero_cta) * 256 + threadIdx.x; i < P.zero_words; i += (int64_t)(gridDim.x - P.zero_cta) * 256)
      P.zero[i] = 0;
  } else if (x >= P.first[2]) {
    table_job(P.job[2], x - P.first[2], P.zero_cta - P.first[2]);
  } else if (x >= P.first[1]) {
    table_job(P.job[1], x - P.first[1], P.first[2] - P.first[1]);
  } else {
    table_job(P.job[0], x, P.first[1]);
  }
}

void set_table_job(TableJob* J, const std::vector<MGroup>& groups, int64_t* o1, int64_t* o2) {
  J->ng = (int)groups.size();
  J->count = 1;
  for (int g = 0; g < J->ng; ++g) {
    J->ext[g] = groups[g].ext;
    J->div[g].init((uint64_t)groups[g].ext);
    J->s1[g] = groups[g].s1;
    J->s2[g] = groups[g].s2;
    J->count *= groups[g].ext;
  }
  J->full = J->count;
  J->tail = 1;
  J->tail_div.init(1);
  J->o1 = o1;
  J->o2 = o2;
}

// Rows in blocks of `block` of group p (see TableJob).
void set_blocked_job(TableJob* J, const std::vector<MGroup>& groups, int p, int64_t block, int64_t* o1, int64_t* o2) {
  const MGroup P = groups[p];
  const int64_t b = std::min(block, P.ext), whole = P.ext / b, rest = P.ext % b;
  std::vector<MGroup> g;
  g.push_back({b, P.s1, P.s2, P.dpos, P.src});
  for (size_t i = 0; i < groups.size(); ++i)
    if ((int)i != p) g.push_back(groups[i]);
  g.push_back({whole, P.s1 * b, P.s2 * b, P.dpos, P.src});
  set_table_job(J, g, o1, o2);
  if (rest) {
    J->tail = rest;
    J->tail_div.init((uint64_t)rest);
    J->base1 = whole * b * P.s1;
    J->base2 = whole * b * P.s2;
    J->count += J->full / b / whole * rest;
  }
}

int run_tables(TableParams& P, cudaStream_t s) {
  unsigned at = 0;
  for (int j = 0; j < 3; ++j) {
    P.first[j] = at;
    at += (unsigned)std::max<int64_t>(1, std::min<int64_t>((P.job[j].count + 255) / 256, num_sms() * 4));
  }
  P.zero_cta = at;
  at += (unsigned)std::max<int64_t>(1, std::min<int64_t>((P.zero_words + 255) / 256, num_sms()));
  tables_kernel<<<at, 256, 0, s>>>(P);
  TB_CHECK_LAUNCH();
  return 0;
}

// ---- operand conversion helpers --------------------------------------------------
__device__ __forceinline__ unsigned exp_field(double x) {
  return (unsigned)((__double_as_longlong(x) >> 52) & 0x7FF);
}

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(x);
  lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

// ---- operand gather: 64 x 64 tiles through source offset tables ----------------
// Element (m, k) of a matricized operand lives at src[lm[m] + lk[k]].  A tile
// is read with lanes along whichever index is contiguous in the source, staged
// in shared memory, and converted with lanes along k so that every thread
// writes 4 consecutive K positions of each output plane in one store.
// Tiles cover [0, rows_pad) x [0, kpad_src): padding is written as zeros.
constexpr int kGThreads = 256;
constexpr int kMaxSlicesDev = 7;
template <typename E> constexpr int gather_rows() { return sizeof(E) == 16 ? 32 : 64; }  // 32-34 KB tiles
constexpr int kGK = 64;

enum GatherMode { G_SLICE_R8, G_SLICE_C8A, G_SLICE_C8B, G_SPLIT_R4, G_SPLIT_C4A, G_SPLIT_C4B,
                  G_RESID_R8, G_RESID_C8A, G_RESID_C8B };

// Ozaki scheme II operands: each scaled value x in (-1/2, 1/2) becomes the
// integer X = floor(x 2^(p+1)) (|X| <= 2^p, exact in FP64), stored as its
// residues modulo the pairwise coprime moduli m_i <= 256 in the symmetric
// range (signed 8 bits), one plane per modulus.  The moduli are the first n
// entries of one fixed table, so the gathers see them as compile-time
// constants.
constexpr int kMaxModuli = 15;
TB_HD constexpr int residue_modulus(int i) {
  return i == 0 ? 256 : i == 1 ? 255 : i == 2 ? 253 : i == 3 ? 251 : i == 4 ? 247 : i == 5 ? 241 : i == 6 ? 239
       : i == 7 ? 233 : i == 8 ? 229 : i == 9 ? 227 : i == 10 ? 223 : i == 11 ? 211 : i == 12 ? 199 : i == 13 ? 197
       : 193;
}
// 2^e mod m
TB_HD constexpr int pow2_mod(int e, int m) {
  int r = 1 % m;
  for (int i = 0; i < e; ++i) r = (2 * r) % m;
  return r;
}
// 2^e mod m_i in the symmetric range [-(m-1)/2, m/2]
TB_HD constexpr int residue_cdig(int i, int e) {
  const int m = residue_modulus(i), c = pow2_mod(e, m);
  return c > (m - 1) / 2 ? c - m : c;
}

struct ResidueSpec {
  int n;                    // moduli: residue_modulus(0 .. n-1)
  int p;                    // operand bits: |X| <= 2^p
  double pscale;            // 2^(p+1)
  int ndig;                 // balanced 16-bit digits of X: 3 (p <= 46) or 4
};

// How a row's values spread below its largest: bits 16 j .. 16 j + 15 of `bins` count
// the values with exponent field e - j, j = 0..3 (of use for e > 3 only: field 0 holds
// zeros and subnormal values); e is 0 only for a row of zeros.
struct __align__(16) RowSpread {
  unsigned long long bins;
  unsigned e, pad_;
};
__device__ __forceinline__ void spread_add(RowSpread& S, double x) {
  const unsigned f = exp_field(x);
  if (f > S.e || S.e == 0) {  // seldom, but for the first values
    const unsigned g = f ? f : (x != 0.0 ? 1u : 0u), up = g - S.e;
    S.bins = up > 3 ? 0ull : S.bins << (16 * up);
    S.e = g;
  }
  const unsigned j = S.e - f;
  S.bins += j <= 3 ? 1ull << (16 * j) : 0ull;
}
__device__ __forceinline__ void spread_merge(RowSpread& S, const RowSpread& o) {
  const unsigned e = max(S.e, o.e), a = e - S.e, b = e - o.e;
  S.bins = (a > 3 ? 0ull : S.bins << (16 * a)) + (b > 3 ? 0ull : o.bins << (16 * b));
  S.e = e;
}

struct GatherParams {
  const void* src;
  const int64_t* lm;   // source offset of row m (m < rows)
  const int64_t* lk;   // source offset of contracted index k (k < K)
  int64_t rows, K;     // valid extents
  int64_t kpad;        // real row length of the output planes (elements)
  int64_t pstride;     // elements per plane
  void* planes;
  unsigned* rowE;      // per row: largest exponent field (slice modes read it; the
                       // split modes set it to 2047 for rows with a NaN or an infinity)
  RowSpread* spread;   // row maxima that also count: [row][K split]; else null
  int slices;
  int lanes_on_k;      // 1: consecutive k are contiguous in the source
  int vec;             // 1 (lanes_on_k): aligned 16-byte groups of k are contiguous and aligned in the source
  double isign;        // -1 conjugates the imaginary part
  ResidueSpec rs;      // residue modes: the moduli
};

// Residues of integers |X| <= 2^p (p <= 52).  X is split once into digits D_j of
// weight w_j, so that for every modulus the residue is
//   raw = sum_j D_j c_j   (c_j = w_j mod m in the symmetric range, c_0 = 1),
// exact in FP32 (|raw| < 2^24), then r = raw - m rint(raw / m) in [-m/2, m/2] --
// exact, the quotient rounded by the 1.5 * 2^23 trick (right since raw / m is
// never within 1/(2m) of a half integer for odd m, and the product's error is
// far below that).  The low byte of r, read off the bit pattern of r + 1.5 *
// 2^23, is r in signed 8 bits (for m = 256, r = 128 gives -128, the same
// residue).  For m = 256 the residue is D_0's low byte.
//
// The digits come without conversions, for two values at a time.  Adding 1.5 *
// 2^52 + B to v rounds v to the nearest integer X (one rounding: the sum lies in
// [2^52, 2^53)) and leaves X + B in the sum's low mantissa bits; a 16-bit field u
// placed under the bit pattern of 1.5 * 2^23 (one byte permute) is the float 1.5
// * 2^23 + u, and one subtraction removes it with the field's bias.
//   NDIG = 3 (p <= 46): B = 2^15 (1 + 2^16 + 2^32), digits u_j - 2^15 of weight 2^(16 j).
//   NDIG = 4: X = 2^24 H + L with H = rint(v / 2^24) (|H| <= 2^28) and L = rint
//   of the exact remainder (|L| <= 2^23); L + 2^23 + 2^15 and H + 2^28 + 2^15 give
//   digits of weight 1, 2^16, 2^24 and 2^40.
TB_HD constexpr int digit_weight(int ndig, int j) { return ndig == 3 ? 16 * j : (j == 0 ? 0 : j == 1 ? 16 : j == 2 ? 24 : 40); }

__device__ __forceinline__ float field_lo(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B400000u, 0x7610)); }
__device__ __forceinline__ float field_hi(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B400000u, 0x7632)); }

// Digits of two operand values: X = rint(x 2^(se + p + 1)) with sc = 2^(se + p +
// 1), or 0 when that is not a double (rows of tiny values, scaled in two steps).
template <int NDIG>
__device__ __forceinline__ void digits2(double x0, int se0, double sc0, double x1, int se1, double sc1, double pscale,
                                        float2 (&d)[4]) {
  constexpr float kM = 12582912.0f;  // 1.5 * 2^23
  constexpr double kM52 = 6755399441055744.0;  // 1.5 * 2^52
  if constexpr (NDIG == 3) {
    constexpr double kB = kM52 + 140739635871744.0;  // + 2^15 + 2^31 + 2^47
    const double y0 = sc0 != 0.0 ? fma(x0, sc0, kB) : fma(scale2(x0, se0), pscale, kB);
    const double y1 = sc1 != 0.0 ? fma(x1, sc1, kB) : fma(scale2(x1, se1), pscale, kB);
    const uint32_t l0 = (uint32_t)__double2loint(y0), h0 = (uint32_t)__double2hiint(y0);
    const uint32_t l1 = (uint32_t)__double2loint(y1), h1 = (uint32_t)__double2hiint(y1);
    const float2 bias = make_float2(-(kM + 32768.0f), -(kM + 32768.0f));
    d[0] = __fadd2_rn(make_float2(field_lo(l0), field_lo(l1)), bias);
    d[1] = __fadd2_rn(make_float2(field_hi(l0), field_hi(l1)), bias);
    d[2] = __fadd2_rn(make_float2(field_lo(h0), field_lo(h1)), bias);
  } else {
    constexpr double kBH = kM52 + 268468224.0, kBL = kM52 + 8421376.0;  // + 2^28 + 2^15; + 2^23 + 2^15
    const double v0 = sc0 != 0.0 ? x0 * sc0 : scale2(x0, se0) * pscale, v1 = sc1 != 0.0 ? x1 * sc1 : scale2(x1, se1) * pscale;
    const double h0 = fma(v0, 0x1p-24, kBH), h1 = fma(v1, 0x1p-24, kBH);
    const double l0 = fma(kBH - h0, 0x1p24, v0) + kBL, l1 = fma(kBH - h1, 0x1p24, v1) + kBL;
    const uint32_t wl0 = (uint32_t)__double2loint(l0), wl1 = (uint32_t)__double2loint(l1);
    const uint32_t wh0 = (uint32_t)__double2loint(h0), wh1 = (uint32_t)__double2loint(h1);
    const float2 b16 = make_float2(-(kM + 32768.0f), -(kM + 32768.0f)), b7 = make_float2(-(kM + 128.0f), -(kM + 128.0f)),
                 b12 = make_float2(-(kM + 4096.0f), -(kM + 4096.0f));
    d[0] = __fadd2_rn(make_float2(field_lo(wl0), field_lo(wl1)), b16);
    d[1] = __fadd2_rn(make_float2(field_hi(wl0), field_hi(wl1)), b7);
    d[2] = __fadd2_rn(make_float2(field_lo(wh0), field_lo(wh1)), b16);
    d[3] = __fadd2_rn(make_float2(field_hi(wh0), field_hi(wh1)), b12);
  }
}

// r + 1.5 * 2^23 for modulus I of two values at once (packed FP32 pairs,
// each component rounded as fmaf / __fadd_rn): the low byte of each
// component's bit pattern is its residue
template <int NDIG, int I>
__device__ __forceinline__ float2 residue_shifted2(const float2 (&d)[4]) {
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
  constexpr int m = residue_modulus(I);
  const float2 magic = make_float2(kMagic, kMagic);
  if constexpr (m == 256) {
    return __fadd2_rn(d[0], magic);
  } else {
    constexpr float negm = -(float)m, inv = 1.0f / (float)m;
    constexpr float c1 = (float)residue_cdig(I, digit_weight(NDIG, 1)), c2 = (float)residue_cdig(I, digit_weight(NDIG, 2)),
                    c3 = (float)residue_cdig(I, digit_weight(NDIG, NDIG > 3 ? 3 : 2));
    float2 raw = __ffma2_rn(d[1], make_float2(c1, c1), d[0]);
    raw = __ffma2_rn(d[2], make_float2(c2, c2), raw);
    if constexpr (NDIG > 3) raw = __ffma2_rn(d[3], make_float2(c3, c3), raw);
    const float2 q = __fadd2_rn(__ffma2_rn(raw, make_float2(inv, inv), magic), make_float2(-kMagic, -kMagic));
    return __fadd2_rn(__ffma2_rn(q, make_float2(negm, negm), raw), magic);
  }
}

// low bytes of four words, packed little-endian
__device__ __forceinline__ uint32_t pack_low_bytes(float a, float b, float c, float d) {
  const uint32_t lo = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x0040);
  const uint32_t hi = __byte_perm(__float_as_uint(c), __float_as_uint(d), 0x0040);
  return __byte_perm(lo, hi, 0x5410);
}

// Residue I of four values (two pairs), packed little-endian.
template <int NDIG, int I>
__device__ __forceinline__ uint32_t residue4(const float2 (&a)[4], const float2 (&b)[4]) {
  const float2 ra = residue_shifted2<NDIG, I>(a), rb = residue_shifted2<NDIG, I>(b);
  return pack_low_bytes(ra.x, ra.y, rb.x, rb.y);
}

// f(integral_constant<int, I>) for I = I0 .. min(n, N) - 1 (n uniform)
template <int I, int N, class F>
__device__ __forceinline__ void for_moduli(int n, F&& f) {
  if constexpr (I < N) {
    if (I < n) {
      f(std::integral_constant<int, I>{});
      for_moduli<I + 1, N>(n, f);
    }
  }
}

// Slices of x in (-1/2, 1/2): balanced signed base-256 digits of the fixed-point
// value X = floor(x * 2^55) = sum_i d_i 2^(48-8i), d_i in [-128, 127] for
// i >= 1 and |d_0| <= 64.  With Y = X + 0x808080808080 the low bytes of Y are
// d_i + 128 and Y >> 48 = d_0, so each slice is one byte of Y (bit 7 flipped
// for i >= 1).  Digit i has weight 2^-(8i+7); the digits are centred on zero,
// so the parts dropped by keeping s slices or slice pairs do not accumulate a
// bias over K.  The scaling by 2^55 is exact and the conversion rounds toward
// minus infinity.
__device__ __forceinline__ long long fixed55(double x) {
  return __double2ll_rd(x * 36028797018963968.0) + 0x808080808080ll;  // 2^55; Y
}
// Slice i of four consecutive values, packed little-endian into one word.
__device__ __forceinline__ uint32_t slice4(long long y0, long long y1, long long y2, long long y3, int i) {
  const int sh = 48 - 8 * i;
  const uint32_t flip = i == 0 ? 0u : 0x80808080u;
  return ((uint32_t)((y0 >> sh) & 255) | ((uint32_t)((y1 >> sh) & 255) << 8) |
          ((uint32_t)((y2 >> sh) & 255) << 16) | ((uint32_t)((y3 >> sh) & 255) << 24)) ^
         flip;
}

// Operand element type of a gather mode.
template <int MODE>
struct GatherElem {
  static constexpr bool CPLX = MODE == G_SLICE_C8A || MODE == G_SLICE_C8B || MODE == G_SPLIT_C4A ||
                               MODE == G_SPLIT_C4B || MODE == G_RESID_C8A || MODE == G_RESID_C8B;
  static constexpr bool F32 = MODE == G_SPLIT_R4 || MODE == G_SPLIT_C4A || MODE == G_SPLIT_C4B;
  using R = typename std::conditional<F32, float, double>::type;
  using E = typename std::conditional<CPLX, typename std::conditional<F32, float2, double2>::type, R>::type;
};
// Tile of a gather mode: TM rows x TK contracted values in two buffers, rows of
// CH 16-byte chunks and one chunk of padding.  A conversion thread takes KPT
// consecutive k of a row (G chunks); chunk c of a row sits at c ^ ((c / G) & 7),
// so that the eight threads of a quarter warp read eight different 16-byte
// banks, and copies along k or along rows write without conflicts beyond two.
template <int MODE>
struct GatherTile {
  using E = typename GatherElem<MODE>::E;
  static constexpr int ES = (int)sizeof(E), TM = gather_rows<E>(), TK = kGK;
  static constexpr int KPT = MODE == G_RESID_R8 || MODE == G_SPLIT_R4 ? 8 : 4;
  static constexpr int G = KPT * ES / 16, CH = TK * ES / 16, PITCH = (CH + 1) * 16;
  static constexpr int BUF = TM * PITCH;
  static __device__ __forceinline__ int chunk(int c) { return (c ^ ((c / G) & 7)) * 16; }
  static __device__ __forceinline__ int at(int k) {
    const int byte = k * ES;
    return chunk(byte >> 4) + (byte & 15);
  }
};
// Dynamic shared memory of a gather CTA: two tile buffers, a ring of three
// tiles' K offsets, the row offsets and the row scale exponents.
template <int MODE>
constexpr int gather_smem_bytes() {
  using T = GatherTile<MODE>;
  return 2 * T::BUF + 3 * T::TK * 8 + T::TM * 20;
}

// Bound by instruction issue, not by HBM: the conversion costs about 5 packed
// instructions per value pair and modulus.  A thread's copies therefore share
// one row or one k (a table read and an addition per copy, or one 16-byte copy
// per two or four values where `vec` allows), and its conversions share the
// digits of eight values and store 8 bytes per plane.
template <int MODE, int NDIG = 3>
__device__ __forceinline__ void gather_body(const GatherParams& P, int64_t rowtile, int ky, int kstep) {
  constexpr bool CPLX = GatherElem<MODE>::CPLX;
  constexpr bool F32 = GatherElem<MODE>::F32;
  using E = typename GatherElem<MODE>::E;
  using T = GatherTile<MODE>;
  constexpr int TM = T::TM, TK = T::TK, ES = T::ES, KPT = T::KPT;
  // Tiles move global -> shared with cp.async, double-buffered: tile i+1 is in
  // flight while tile i converts, without passing through registers.  Its
  // source addresses need the K offsets of tile i+1, which sit in shared
  // memory: they were read from global memory (into a register, by one thread
  // per k) during tile i-1's conversion and stored at its end.
  extern __shared__ __align__(16) unsigned char gather_smem[];
  int64_t* lkbuf = reinterpret_cast<int64_t*>(gather_smem + 2 * T::BUF);  // [3][TK]
  int64_t* sm_lm = lkbuf + 3 * TK;                                         // [TM]
  double* sm_sc = reinterpret_cast<double*>(sm_lm + TM);  // residue modes: 2^(se + p + 1), or 0
  int* sm_se = reinterpret_cast<int*>(sm_sc + TM);  // slice and residue modes: the row's scale exponent
  const int64_t m0 = rowtile * TM;
  const int tid = threadIdx.x;
  const E* src = (const E*)P.src;
  const int64_t ntiles = (P.kpad / (CPLX ? 2 : 1)) / TK;  // conversion also writes the padding
  if (ky >= ntiles) return;  // uniform: no tile for this CTA
  if (tid < TM) {
    sm_lm[tid] = (m0 + tid < P.rows) ? P.lm[m0 + tid] : -1;
    if constexpr (!F32) {
      const int se = 1021 - (int)(m0 + tid < P.rows ? P.rowE[m0 + tid] : 1021u);
      sm_se[tid] = se;
      sm_sc[tid] = se + P.rs.p + 1 <= 1023 ? pow2d(se + P.rs.p + 1) : 0.0;
    }
  }
  if (tid < TK) {
    for (int j = 0; j < 2; ++j) {
      const int64_t k = ((int64_t)ky + (int64_t)j * kstep) * TK + tid;
      lkbuf[j * TK + tid] = k < P.K ? P.lk[k] : 0;
    }
  }
  auto issue_tile = [&](int64_t k0, int buf, const int64_t* lkt) {
    unsigned char* t = gather_smem + (size_t)buf * T::BUF;
    const int64_t kleft = P.K - k0;
    if (P.lanes_on_k && (P.vec || ES == 16)) {
      constexpr int VW = 16 / ES, RS = kGThreads / T::CH;  // values per copy, rows per round
      static_assert(kGThreads % T::CH == 0 && TM % RS == 0, "whole rounds");
      const int ch = tid % T::CH, r0 = tid / T::CH;
      const bool kv = ch * VW < kleft;
      const E* base = src + (kv ? lkt[ch * VW] : 0);
      unsigned char* d = t + r0 * T::PITCH + T::chunk(ch);
#pragma unroll
      for (int it = 0; it < TM / RS; ++it) {
        const int64_t lm = sm_lm[r0 + it * RS];
        const bool ok = kv && lm >= 0;
        cp_async_elem<16>(d + it * RS * T::PITCH, base + (ok ? lm : 0), ok);
      }
    } else if (P.lanes_on_k) {
      constexpr int RS = kGThreads / TK;
      const int kk = tid % TK, r0 = tid / TK;
      const bool kv = kk < kleft;
      const E* base = src + (kv ? lkt[kk] : 0);
      unsigned char* d = t + r0 * T::PITCH + T::at(kk);
#pragma unroll
      for (int it = 0; it < TM / RS; ++it) {
        const int64_t lm = sm_lm[r0 + it * RS];
        const bool ok = kv && lm >= 0;
        cp_async_elem<ES>(d + it * RS * T::PITCH, base + (ok ? lm : 0), ok);
      }
    } else {
      constexpr int KS = kGThreads / TM;
      const int r = tid % TM, kk0 = tid / TM;
      const int64_t lm = sm_lm[r];
      const E* base = src + (lm >= 0 ? lm : 0);
      unsigned char* d = t + r * T::PITCH;
#pragma unroll
      for (int it = 0; it < TK / KS; ++it) {
        const int kk = kk0 + it * KS;
        const bool ok = lm >= 0 && kk < kleft;
        cp_async_elem<ES>(d + T::at(kk), base + (ok ? lkt[kk] : 0), ok);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  __syncthreads();  // sm_lm and the first two tiles' K offsets ready
  issue_tile((int64_t)ky * TK, 0, lkbuf);
  int i = 0;
  for (int64_t kt = ky; kt < ntiles; kt += kstep, ++i) {
    const int64_t k0 = kt * TK;
    __syncthreads();  // buffer (i+1) & 1 consumed; K offsets of tile i+1 visible
    if (kt + kstep < ntiles)
      issue_tile((kt + kstep) * TK, (i + 1) & 1, lkbuf + ((i + 1) % 3) * TK);
    else
      asm volatile("cp.async.commit_group;\n" ::: "memory");  // empty group: keeps the count
    int64_t lk2 = 0;  // K offset of tile i+2 (one per thread < TK), stored after the conversion
    {
      const int64_t k = (kt + 2 * (int64_t)kstep) * TK + tid;
      if (tid < TK && kt + 2 * (int64_t)kstep < ntiles && k < P.K) lk2 = P.lk[k];
    }
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this thread's copies of tile i
    __syncthreads();                                          // everyone's
    const unsigned char* tile = gather_smem + (size_t)(i & 1) * T::BUF;
    {
      // convert: thread -> (row mm, KPT consecutive k)
      for (int idx = tid; idx < TM * (TK / KPT); idx += kGThreads) {
        const int mm = idx / (TK / KPT), kj = idx % (TK / KPT), kq = kj * KPT;
        const int64_t m = m0 + mm, k = k0 + kq;
        union { uint4 q[T::G]; E v[KPT]; } in;
#pragma unroll
        for (int u = 0; u < T::G; ++u)
          in.q[u] = *reinterpret_cast<const uint4*>(tile + mm * T::PITCH + (((kj * T::G + u) ^ (kj & 7)) * 16));
        if constexpr (MODE == G_RESID_R8) {
          const int se = sm_se[mm];
          const double sc = sm_sc[mm];
          float2 g[4][4];
#pragma unroll
          for (int t = 0; t < 4; ++t) digits2<NDIG>(in.v[2 * t], se, sc, in.v[2 * t + 1], se, sc, P.rs.pscale, g[t]);
          int8_t* base = (int8_t*)P.planes + m * P.kpad + k;
          for_moduli<0, kMaxModuli>(P.rs.n, [&](auto ic) {
            constexpr int I = decltype(ic)::value;
            *reinterpret_cast<uint2*>(base) = make_uint2(residue4<NDIG, I>(g[0], g[1]), residue4<NDIG, I>(g[2], g[3]));
            base += P.pstride;
          });
        } else if constexpr (MODE == G_RESID_C8A) {
          // A' row m: (re, im) interleaved along K
          const int se = sm_se[mm];
          const double sc = sm_sc[mm];
          float2 g[4][4];
#pragma unroll
          for (int t = 0; t < 4; ++t)
            digits2<NDIG>(in.v[t].x, se, sc, P.isign * in.v[t].y, se, sc, P.rs.pscale, g[t]);
          int8_t* base = (int8_t*)P.planes + m * P.kpad + 2 * k;
          for_moduli<0, kMaxModuli>(P.rs.n, [&](auto ic) {
            constexpr int I = decltype(ic)::value;
            *reinterpret_cast<uint2*>(base) = make_uint2(residue4<NDIG, I>(g[0], g[1]), residue4<NDIG, I>(g[2], g[3]));
            base += P.pstride;
          });
        } else if constexpr (MODE == G_RESID_C8B) {
          // B' rows 2n = (re, -im), 2n+1 = (im, re) interleaved along K; the
          // residues of -im are those of im, negated byte by byte
          const int se = sm_se[mm];
          const double sc = sm_sc[mm];
          float2 R[2][4], I[2][4];
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            digits2<NDIG>(in.v[2 * t].x, se, sc, in.v[2 * t + 1].x, se, sc, P.rs.pscale, R[t]);
            digits2<NDIG>(P.isign * in.v[2 * t].y, se, sc, P.isign * in.v[2 * t + 1].y, se, sc, P.rs.pscale, I[t]);
          }
          int8_t* b0 = (int8_t*)P.planes + (2 * m) * P.kpad + 2 * k;
          for_moduli<0, kMaxModuli>(P.rs.n, [&](auto ic) {
            constexpr int J = decltype(ic)::value;
            const uint32_t re = residue4<NDIG, J>(R[0], R[1]), im = residue4<NDIG, J>(I[0], I[1]);
            const uint32_t ni = __vsub4(0u, im);
            *reinterpret_cast<uint2*>(b0) = make_uint2(__byte_perm(re, ni, 0x5140), __byte_perm(re, ni, 0x7362));
            *reinterpret_cast<uint2*>(b0 + P.kpad) = make_uint2(__byte_perm(im, re, 0x5140), __byte_perm(im, re, 0x7362));
            b0 += P.pstride;
          });
        } else if constexpr (MODE == G_SLICE_R8) {
          const int se = sm_se[mm];
          long long X[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) X[t] = fixed55(scale2(in.v[t], se));
          int8_t* base = (int8_t*)P.planes + m * P.kpad + k;
#pragma unroll
          for (int i = 0; i < kMaxSlicesDev; ++i)
            if (i < P.slices) *reinterpret_cast<uint32_t*>(base + i * P.pstride) = slice4(X[0], X[1], X[2], X[3], i);
        } else if constexpr (MODE == G_SLICE_C8A) {
          // A' row m: (re, im) interleaved along K
          const int se = sm_se[mm];
          long long R[4], I[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const E v = in.v[t];
            R[t] = fixed55(scale2(v.x, se));
            I[t] = fixed55(scale2(P.isign * v.y, se));
          }
          int8_t* base = (int8_t*)P.planes + m * P.kpad + 2 * k;
#pragma unroll
          for (int i = 0; i < kMaxSlicesDev; ++i)
            if (i < P.slices) {
              uint2 w = make_uint2(slice4(R[0], I[0], R[1], I[1], i), slice4(R[2], I[2], R[3], I[3], i));
              *reinterpret_cast<uint2*>(base + i * P.pstride) = w;
            }
        } else if constexpr (MODE == G_SLICE_C8B) {
          // B' rows 2n = (re, -im), 2n+1 = (im, re) interleaved along K
          const int se = sm_se[mm];
          long long R[4], I[4], NI[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const E v = in.v[t];
            const double im = scale2(P.isign * v.y, se);
            R[t] = fixed55(scale2(v.x, se));
            I[t] = fixed55(im);
            NI[t] = fixed55(-im);
          }
          int8_t* b0 = (int8_t*)P.planes + (2 * m) * P.kpad + 2 * k;
          int8_t* b1 = b0 + P.kpad;
#pragma unroll
          for (int i = 0; i < kMaxSlicesDev; ++i)
            if (i < P.slices) {
              *reinterpret_cast<uint2*>(b0 + i * P.pstride) =
                  make_uint2(slice4(R[0], NI[0], R[1], NI[1], i), slice4(R[2], NI[2], R[3], NI[3], i));
              *reinterpret_cast<uint2*>(b1 + i * P.pstride) =
                  make_uint2(slice4(I[0], R[0], I[1], R[1], i), slice4(I[2], R[2], I[3], R[3], i));
            }
        } else if constexpr (MODE == G_SPLIT_R4) {
          __nv_bfloat16 h[8], l[8];
          bool nf = false;
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            split_bf16(in.v[t], h[t], l[t]);
            nf |= !isfinite(in.v[t]);
          }
          if (nf && P.rowE && m < P.rows) atomicMax(&P.rowE[m], 2047u);  // row left to the non-finite fix-up
          __nv_bfloat16* base = (__nv_bfloat16*)P.planes + m * P.kpad + k;
          __nv_bfloat162 hh[4] = {{h[0], h[1]}, {h[2], h[3]}, {h[4], h[5]}, {h[6], h[7]}};
          __nv_bfloat162 ll[4] = {{l[0], l[1]}, {l[2], l[3]}, {l[4], l[5]}, {l[6], l[7]}};
          *reinterpret_cast<uint4*>(base) = *reinterpret_cast<uint4*>(hh);
          *reinterpret_cast<uint4*>(base + P.pstride) = *reinterpret_cast<uint4*>(ll);
        } else {
          // complex FP32: A' rows (re, im); B' rows 2n (re, -im), 2n+1 (im, re)
          __nv_bfloat16 hr[4], lr[4], hi[4], li[4], nhi[4], nli[4];
          bool nf = false;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const E v = in.v[t];
            const float im = (float)P.isign * v.y;
            split_bf16(v.x, hr[t], lr[t]);
            split_bf16(im, hi[t], li[t]);
            split_bf16(-im, nhi[t], nli[t]);
            nf |= !isfinite(v.x) || !isfinite(v.y);
          }
          if (nf && P.rowE && m < P.rows) atomicMax(&P.rowE[m], 2047u);  // row left to the non-finite fix-up
          if constexpr (MODE == G_SPLIT_C4A) {
            __nv_bfloat16* base = (__nv_bfloat16*)P.planes + m * P.kpad + 2 * k;
            __nv_bfloat162 H[4] = {{hr[0], hi[0]}, {hr[1], hi[1]}, {hr[2], hi[2]}, {hr[3], hi[3]}};
            __nv_bfloat162 L[4] = {{lr[0], li[0]}, {lr[1], li[1]}, {lr[2], li[2]}, {lr[3], li[3]}};
            *reinterpret_cast<uint4*>(base) = *reinterpret_cast<uint4*>(H);
            *reinterpret_cast<uint4*>(base + P.pstride) = *reinterpret_cast<uint4*>(L);
          } else {
            __nv_bfloat16* b0 = (__nv_bfloat16*)P.planes + (2 * m) * P.kpad + 2 * k;
            __nv_bfloat16* b1 = b0 + P.kpad;
            __nv_bfloat162 H0[4] = {{hr[0], nhi[0]}, {hr[1], nhi[1]}, {hr[2], nhi[2]}, {hr[3], nhi[3]}};
            __nv_bfloat162 L0[4] = {{lr[0], nli[0]}, {lr[1], nli[1]}, {lr[2], nli[2]}, {lr[3], nli[3]}};
            __nv_bfloat162 H1[4] = {{hi[0], hr[0]}, {hi[1], hr[1]}, {hi[2], hr[2]}, {hi[3], hr[3]}};
            __nv_bfloat162 L1[4] = {{li[0], lr[0]}, {li[1], lr[1]}, {li[2], lr[2]}, {li[3], lr[3]}};
            *reinterpret_cast<uint4*>(b0) = *reinterpret_cast<uint4*>(H0);
            *reinterpret_cast<uint4*>(b0 + P.pstride) = *reinterpret_cast<uint4*>(L0);
            *reinterpret_cast<uint4*>(b1) = *reinterpret_cast<uint4*>(H1);
            *reinterpret_cast<uint4*>(b1 + P.pstride) = *reinterpret_cast<uint4*>(L1);
          }
        }
      }
    }
    if (tid < TK) lkbuf[((i + 2) % 3) * TK + tid] = lk2;
  }
}

// Both operands of a contraction in one launch: CTAs from ctas_a on work on B.
// CTA x of an operand takes row tile x % rows and every gy-th K tile from x / rows.
struct GatherPair {
  GatherParams a, b;
  unsigned ctas_a, rows_a, rows_b;
  int gy_a, gy_b;
  const unsigned* refused;  // nothing to do if this word is set (null: never)
};

// (the complex residue modes leave two CTAs per SM registers enough not to spill)
template <int MODEA, int MODEB, int NDIG = 3>
__global__ void __launch_bounds__(kGThreads, MODEB == G_RESID_C8B ? 2 : 3)
    gather_kernel(const __grid_constant__ GatherPair Q) {
  if (Q.refused && *Q.refused) return;
  const bool second = blockIdx.x >= Q.ctas_a;
  const unsigned x = second ? blockIdx.x - Q.ctas_a : blockIdx.x, rows = second ? Q.rows_b : Q.rows_a;
  const unsigned ky = x / rows, rt = x - ky * rows;
  if constexpr (MODEA == MODEB) {
    const GatherParams P = second ? Q.b : Q.a;
    gather_body<MODEA, NDIG>(P, rt, (int)ky, second ? Q.gy_b : Q.gy_a);
  } else {
    if (second) gather_body<MODEB, NDIG>(Q.b, rt, (int)ky, Q.gy_b);
    else gather_body<MODEA, NDIG>(Q.a, rt, (int)ky, Q.gy_a);
  }
}

// Grouped form: CTA x works on row tile map[x].y of job map[x].x.
template <int MODE>
__global__ void __launch_bounds__(kGThreads, 3) gather_grouped_kernel(const GatherParams* __restrict__ jobs,
                                                                   const int2* __restrict__ map) {
  const int2 jm = map[blockIdx.x];
  const GatherParams P = jobs[jm.x];
  gather_body<MODE>(P, jm.y, blockIdx.y, gridDim.y);
}

// Sets the grouped gather's dynamic shared-memory limit on the current device
// (once per device; call it before any stream capture).
template <int MODE>
cudaError_t gather_grouped_prepare() {
  static DeviceOnce once;
  return smem_limit_once(once, gather_grouped_kernel<MODE>, gather_smem_bytes<MODE>());
}

// exponents: rowexp[r] = rowE[r] - 1021
__global__ void exps_kernel(const unsigned* __restrict__ rowE, int* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (int)rowE[i] - 1021;
}

// Whether residues may stand for FP64 sums, decided from the operands.  With p
// operand bits a residue product is off by at most K 2^(a + b + 2 - p), 2^a and 2^b the
// binades of the row's and the column's largest values.  If at least C of the K pairs
// hold two values within s binades of those, the sum of |products| is at least C 2^(a +
// b - 2 s), so that bound is K 2^(2 + 2 s - p) / C of it, and no larger than the K 2^-53
// of a sum of K FP64 terms where C >= 2^(55 + 2 s - p).  C is at least K minus the
// values of the worst row and of the worst column that are not within s binades;
// C >= K / 4 is asked for as well.  Rows and columns with a NaN or an infinity (the
// fix-up multiplies them in FP64) and rows of zeros do not count.
struct GuardParams {
  const RowSpread* a;        // [row][K split] of both operands
  const RowSpread* b;
  int64_t m, n;              // rows, columns
  int gy_a, gy_b;            // K splits
  int kr;                    // values per row
  int need[3];               // C for s = 1, 2, 3
  unsigned* words;           // zeroed: [0..2], [3..5] values missing in the worst row and column, [6]
                             // CTAs done, [7] the verdict: 1 where residues are refused
};

// Both operands' exponents in one launch: rowx[r] = rowE[r] - 1021, colx likewise
// (rep = 2 for complex B' rows).  Rows and columns flagged 2047 (a NaN or an
// infinity) are also appended to the bad lists (in no particular order; nbad[0..1]
// count them).  GUARD: the last CTA writes the verdict.
template <bool GUARD>
__global__ void __launch_bounds__(256) exps_pair_kernel(const unsigned* __restrict__ rowE, int* __restrict__ rowx, int64_t m,
                                 int* __restrict__ badrows, const unsigned* __restrict__ colE, int* __restrict__ colx,
                                 int64_t n, int rep, int* __restrict__ badcols, int* __restrict__ nbad,
                                 const __grid_constant__ GuardParams G) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m + n; i += (int64_t)gridDim.x * blockDim.x) {
    const bool col = i >= m;
    const int64_t j = col ? i - m : i;
    const unsigned e = col ? colE[j / rep] : rowE[j];
    (col ? colx : rowx)[j] = (int)e - 1021;
    if (e >= 2047u) {
      if (!col) badrows[atomicAdd(nbad, 1)] = (int)j;
      else if (j % rep == 0) badcols[atomicAdd(nbad + 1, 1)] = (int)(j / rep);
    }
  }
  if constexpr (GUARD) {
    // eight lanes merge a row's records
    unsigned miss[2][3] = {{0, 0, 0}, {0, 0, 0}};
    __shared__ unsigned sm_miss[6];
    if (threadIdx.x < 6) sm_miss[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, sub = lane & 7;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); 4 * w < G.m + G.n; w += warps) {
      const int64_t i = 4 * w + (lane >> 3);
      const bool in = i < G.m + G.n, col = i >= G.m;
      const int splits = col ? G.gy_b : G.gy_a;
      const RowSpread* rec = col ? G.b + (i - G.m) * splits : G.a + i * splits;
      RowSpread S{0ull, 0u, 0u};
      if (in)
#pragma unroll 4
        for (int y = sub; y < splits; y += 8) spread_merge(S, rec[y]);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        const RowSpread T{__shfl_xor_sync(0xffffffffu, S.bins, o), __shfl_xor_sync(0xffffffffu, S.e, o), 0u};
        spread_merge(S, T);
      }
      if (S.e == 0 || S.e >= 2047u) continue;
      if (S.e <= 3) S.bins = 0;
      int c = G.kr - (int)(S.bins & 0xFFFF);
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        c -= (int)((S.bins >> (16 * (s + 1))) & 0xFFFF);
        if (col) miss[1][s] = max(miss[1][s], (unsigned)c);
        else miss[0][s] = max(miss[0][s], (unsigned)c);
      }
    }
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const unsigned v = __reduce_max_sync(0xffffffffu, miss[o][s]);
        if (lane == 0 && v) atomicMax(&sm_miss[3 * o + s], v);
      }
    __syncthreads();
    if (threadIdx.x < 6 && sm_miss[threadIdx.x]) {
      atomicMax(&G.words[threadIdx.x], sm_miss[threadIdx.x]);
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&G.words[6], 1u) == gridDim.x - 1) {
      __threadfence();
      bool ok = false;
      for (int s = 0; s < 3; ++s)
        ok = ok || G.kr - (int)atomicAdd(&G.words[s], 0u) - (int)atomicAdd(&G.words[3 + s], 0u) >= G.need[s];
      G.words[7] = ok ? 0u : 1u;
    }
  }
}

// ---- non-finite fix-up -----------------------------------------------------------
// D entries whose row of A or column of B holds a NaN or an infinity are left
// untouched by the GEMM epilogue (nf_skip) and computed here as plain dot
// products in FP64 (FP32 data too, rounded once at the end), so that
// non-finite values propagate the way an IEEE GEMM propagates them: a NaN
// term, an infinity times zero, or infinities of both signs give NaN; other
// infinities give an infinity of their sign.  Work: one warp per entry, the
// entries of the flagged rows (all columns) and then of the flagged columns
// (the rows that are not flagged).  With nothing flagged every CTA returns at
// once.
struct NfParams {
  const void* srcA;
  const void* srcB;
  const int64_t *lmA, *lkA, *lmB, *lkB;  // operand offsets (rows, contracted index)
  const int64_t *dm, *dn;                 // D offsets of rows of A and columns of B
  void* D;
  int64_t M, N, K;                        // rows of A, columns of B (complex: pairs), contracted extent
  const unsigned* rowE;                   // 2047: the row holds a non-finite value
  const int* badrows;                     // flagged rows of A, count nbad[0]
  const int* badcols;                     // flagged columns of B, count nbad[1]
  const int* nbad;
  double isignA, isignB;                  // -1: conjugate the operand
  double ar, ai, br, bi;                  // alpha, beta (beta 0: D is not read)
  const unsigned* refused;                // nothing to do if this word is set (null: never)
};

template <typename R, bool CPLX>
__global__ void __launch_bounds__(256) nonfinite_fixup_kernel(const __grid_constant__ NfParams P) {
  const int nbr = P.nbad[0], nbc = P.nbad[1];
  if (nbr == 0 && nbc == 0) return;
  if (P.refused && *P.refused) return;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t total = (int64_t)nbr * P.N + (int64_t)nbc * P.M;
  for (int64_t e = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); e < total; e += warps) {
    int64_t m, n;
    if (e < (int64_t)nbr * P.N) {
      m = P.badrows[e / P.N];
      n = e % P.N;
    } else {
      const int64_t f = e - (int64_t)nbr * P.N;
      n = P.badcols[f / P.M];
      m = f % P.M;
      if (P.rowE[m] >= 2047u) continue;  // done with the flagged rows
    }
    const int64_t a0 = P.lmA[m], b0 = P.lmB[n];
    double sr = 0.0, si = 0.0;
    if constexpr (!CPLX) {
      const R* A = (const R*)P.srcA;
      const R* B = (const R*)P.srcB;
      for (int64_t k = lane; k < P.K; k += 32) sr += (double)A[a0 + P.lkA[k]] * (double)B[b0 + P.lkB[k]];
    } else {
      using C2 = typename std::conditional<sizeof(R) == 8, double2, float2>::type;
      const C2* A = (const C2*)P.srcA;
      const C2* B = (const C2*)P.srcB;
      for (int64_t k = lane; k < P.K; k += 32) {
        const C2 x = A[a0 + P.lkA[k]], y = B[b0 + P.lkB[k]];
        const double xr = x.x, xi = P.isignA * (double)x.y, yr = y.x, yi = P.isignB * (double)y.y;
        sr += xr * yr - xi * yi;
        si += xr * yi + xi * yr;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      if (CPLX) si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (lane != 0) continue;
    const int64_t off = P.dm[m] + P.dn[n];
    if constexpr (!CPLX) {
      R* D = (R*)P.D;
      const double v = P.ar * sr;
      D[off] = (R)(P.br == 0.0 ? v : P.br * (double)D[off] + v);
    } else {
      using C2 = typename std::conditional<sizeof(R) == 8, double2, float2>::type;
      C2* D = (C2*)P.D;
      double vr = P.ar * sr - P.ai * si, vi = P.ar * si + P.ai * sr;
      if (P.br != 0.0 || P.bi != 0.0) {
        const C2 d = D[off];
        vr += P.br * (double)d.x - P.bi * (double)d.y;
        vi += P.br * (double)d.y + P.bi * (double)d.x;
      }
      C2 w;
      w.x = (R)vr;
      w.y = (R)vi;
      D[off] = w;
    }
  }
}


// ---- Ozaki scheme II reconstruction (Chinese remainder theorem) ------------------
// With M = prod m_i, M_i = M / m_i, y_i = M_i^-1 mod m_i and s_i = y_i M_i, the
// exact integer dot product is C = sum_i r_i s_i - Q M, |C| < M / 2 by the choice
// of p.  s_i and M are cut into three parts of at most 41 bits of 2^b > M, so
// that each part's sum over r_i < 2^8 and 15 terms, and its difference with Q
// times M's part, is exact in FP64; the three differences are added with one
// error term, so C comes out within about one rounding whatever cancels.  Q =
// rint(first sum / M) is right because |C| stays a part in 2^20 below M / 2
// (residue_bits) and the dropped parts are below 2^-28 M.  C is scaled by 2^(e_m
// + f_n - 2(p+1)) exactly, and D = beta D + alpha C through the offset tables.
// Rows and columns flagged as holding a NaN or an infinity are left to the
// fix-up kernel.  Bound by the bytes of the planes and D and by the FP64 units
// (four operations per residue) about alike, and for small outputs by its memory
// latencies: 40 us for 1600^2 x 15 moduli, 68 us for 9216 x 576 x 15.  A 60 KB
// shared-memory table of 128-bit multiples, one random 16-byte read per residue, took
// 80 and 161 us.
struct CrtView {               // one output
  const uint8_t* res;          // residue planes [i][row][column], bytes
  int64_t res_ld, res_plane;
  int64_t rows, cols;          // rows of A; columns of B (complex: column pairs)
  int row_step;                // rows between a warp's lanes (blocked rows: the block, see TableJob)
  int leave_flagged;           // 1: flagged rows and columns are the fix-up's; 0: they become NaN
  const int64_t* dm;
  const int64_t* dn;
  void* D;
  const int* rowexp;
  const int* colexp;
};
struct CrtParams {
  CrtView v;                   // (dense form)
  int n;
  int mod[kMaxModuli];
  double s1[kMaxModuli], s2[kMaxModuli], s3[kMaxModuli];
  double M1, M2, M3, invM;
  int shift;                   // 2 (p + 1)
  double ar, ai, br, bi;
  const unsigned* refused;     // nothing to do if this word is set (null: never)
};

// A warp takes 32 rows (lanes; D's fastest) and a thread kCrtCols residue
// columns of its row, one 16-byte load per plane; the warps of a CTA take
// neighbouring columns, so that together they use whole lines of the planes.
constexpr int kCrtCols = 16, kCrtWarps = 4;

template <bool CPLX>
__device__ __forceinline__ void crt_body(const CrtParams& P, const CrtView& V, unsigned block) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned rs = (unsigned)V.row_step;
  const unsigned row_blocks = (unsigned)((V.rows + 32 * rs - 1) / (32 * rs)) * rs;
  const unsigned cb = block / row_blocks, rb = block - cb * row_blocks;
  const int64_t m = ((int64_t)(rb / rs) * 32 + lane) * rs + rb % rs;
  constexpr int RC = CPLX ? 2 : 1, DC = kCrtCols / RC;  // residue columns per D column; D columns per thread
  const int64_t c0 = ((int64_t)cb * kCrtWarps + warp) * kCrtCols;
  if (c0 >= V.cols * RC) return;
  const bool mok = m < V.rows;
  // Everything that depends on nothing is loaded at once, so that a warp waits for
  // two memory latencies, not five: its row's exponent and D offset, its columns'
  // (one column per lane, handed around by shuffles), its residues; then D.
  const int re = mok ? V.rowexp[m] : kNonFiniteExp;
  const int64_t dmo = mok ? V.dm[m] : 0;
  const int64_t nl = c0 / RC + (lane < DC ? lane : 0);
  const bool lok = nl < V.cols;
  const int ce_l = lok ? V.colexp[nl * RC] : kNonFiniteExp;
  const int64_t dn_l = lok ? V.dn[nl] : 0;
  const uint8_t* rp = V.res + (mok ? m : 0) * V.res_ld + c0;  // rows are padded to whole column tiles: always inside the plane
  uint4 w[kMaxModuli];
#pragma unroll
  for (int i = 0; i < kMaxModuli; ++i)
    w[i] = i < P.n ? *reinterpret_cast<const uint4*>(rp + i * V.res_plane) : make_uint4(0, 0, 0, 0);
  const bool read_d = P.br != 0.0 || P.bi != 0.0;
  using E = typename std::conditional<CPLX, double2, double>::type;
  E* D = (E*)V.D;
  constexpr int G = 8, H = G / RC, NG = kCrtCols / G;  // residue columns and D columns of one group
  // column j of D: its offset (-1: not written here) and exponent
  auto column = [&](int j, int64_t& o, int& ce) {
    ce = __shfl_sync(0xffffffffu, ce_l, j);
    const int64_t dn = __shfl_sync(0xffffffffu, dn_l, j);
    const bool in = mok && c0 / RC + j < V.cols;
    const bool flagged = re >= kNonFiniteExp || ce >= kNonFiniteExp;
    o = in && !(flagged && V.leave_flagged) ? dmo + dn : -1;
  };
  E old[NG][H];
#pragma unroll
  for (int g = 0; g < NG; ++g)
#pragma unroll
    for (int j = 0; j < H; ++j) {
      int64_t o;
      int ce;
      column(g * H + j, o, ce);
      if (read_d && o >= 0) old[g][j] = D[o];
    }
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    double a[G], b[G], c[G];
#pragma unroll
    for (int j = 0; j < G; ++j) a[j] = b[j] = c[j] = 0.0;
#pragma unroll
    for (int i = 0; i < kMaxModuli; ++i) {
      if (i >= P.n) break;
      const double s1 = P.s1[i], s2 = P.s2[i], s3 = P.s3[i];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const uint32_t q = g == 0 ? (j < 4 ? w[i].x : w[i].y) : (j < 4 ? w[i].z : w[i].w);
        // r as a double: 2^52 + r by its bits, minus 2^52
        const double r = __hiloint2double(0x43300000, (int)__byte_perm(q, 0u, 0x4440 + (j & 3))) - 4503599627370496.0;
        a[j] = fma(r, s1, a[j]);
        b[j] = fma(r, s2, b[j]);
        c[j] = fma(r, s3, c[j]);
      }
    }
    auto combine = [&](int j, int cexp) {
      const double Q = rint(a[j] * P.invM);
      const double x = fma(-Q, P.M1, a[j]), y = fma(-Q, P.M2, b[j]), z = fma(-Q, P.M3, c[j]);  // exact
      const double t = x + y, yy = t - x;
      const double err = (x - (t - yy)) + (y - yy);  // x + y = t + err exactly
      if (re >= kNonFiniteExp || cexp >= kNonFiniteExp) return __longlong_as_double(0x7FF8000000000000ll);
      return scale2(t + (err + z), re + cexp - P.shift);
    };
#pragma unroll
    for (int j = 0; j < H; ++j) {
      int64_t o;
      int ce;
      column(g * H + j, o, ce);
      if (o < 0) continue;
      if constexpr (!CPLX) {
        const double v = P.ar * combine(j, ce);
        D[o] = P.br == 0.0 ? v : fma(P.br, old[g][j], v);
      } else {
        const double xr = combine(2 * j, ce), xi = combine(2 * j + 1, ce);
        double2 v;
        v.x = P.ar * xr - P.ai * xi;
        v.y = P.ar * xi + P.ai * xr;
        if (read_d) {
          v.x += P.br * old[g][j].x - P.bi * old[g][j].y;
          v.y += P.br * old[g][j].y + P.bi * old[g][j].x;
        }
        D[o] = v;
      }
    }
  }
}

template <bool CPLX>
__global__ void __launch_bounds__(32 * kCrtWarps, 3) crt_kernel(const __grid_constant__ CrtParams P) {
  if (P.refused && *P.refused) return;
  crt_body<CPLX>(P, P.v, blockIdx.x);
}

// Grouped form: CTA x works on block map[x].y of output map[x].x.
__global__ void __launch_bounds__(32 * kCrtWarps, 3) crt_grouped_kernel(const __grid_constant__ CrtParams P,
                                                                       const CrtView* __restrict__ outputs,
                                                                       const int2* __restrict__ map) {
  const int2 jm = map[blockIdx.x];
  const CrtView V = outputs[jm.x];
  crt_body<false>(P, V, (unsigned)jm.y);
}

// CTAs of one output.
int64_t crt_blocks(int64_t rows, int64_t residue_cols, int row_step) {
  return (rows + 32 * row_step - 1) / (32 * row_step) * row_step *
         ((residue_cols + kCrtCols * kCrtWarps - 1) / (kCrtCols * kCrtWarps));
}

// ---- Ozaki scheme II: the plan ------------------------------------------------------
// Pairwise coprime moduli <= 256, largest first (their residues in the
// symmetric range are signed 8-bit).  With n of them, M = prod m_i and the
// operands scaled to integers |X| <= 2^p, an exact INT32 GEMM per modulus and
// the Chinese remainder theorem give the exact integer product as long as
// M > 2 Kr 2^(2p) (Kr: the real contraction length).
constexpr int kModuliTable[kMaxModuli] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193};
constexpr bool moduli_table_matches() {
  for (int i = 0; i < kMaxModuli; ++i)
    if (kModuliTable[i] != residue_modulus(i)) return false;
  return true;
}
static_assert(moduli_table_matches(), "the gathers' compile-time moduli must be the plan's table");
constexpr int kMinModuli = 8;
constexpr int kMaxPassBlocks = 1023;  // K blocks of one exact INT32 pass (128^3 each, below 2^31)
constexpr int kResidueBitsTarget = 46;  // the default choice: |X| <= 2^46, operands within 2^-48 as by six INT8 slices

using u128 = unsigned __int128;

u128 moduli_product(int n) {
  u128 M = 1;
  for (int i = 0; i < n; ++i) M *= (u128)kModuliTable[i];
  return M;
}

// The largest p with M (1 - 2^-20) > 2 Kr 2^(2p) for n moduli (checked in exact
// integer arithmetic; the 2^-20 is the room that crt_kernel's quotient needs).
int residue_bits(int n, int64_t Kr) {
  const u128 Mf = moduli_product(n), M = Mf - (Mf >> 20);
  int p = 0;
  while (p < 60 && (M >> (2 * (p + 1))) > (u128)(2 * Kr)) ++p;
  return p;
}

struct ResiduePlan {
  ResidueSpec rs;
  int p;
  CrtParams crt;  // constants only; pointers and sizes are filled by the caller
};

// Moduli count and constants for a contraction of real length Kr: `want` > 0
// asks for that many moduli, else the fewest with p >= kResidueBitsTarget.
// Returns false when no allowed count reaches kResidueBitsTarget bits.
bool plan_residues(int64_t Kr, int want, ResiduePlan* out) {
  int n = want;
  if (n <= 0) {
    for (n = kMinModuli; n <= kMaxModuli && residue_bits(n, Kr) < kResidueBitsTarget; ++n) {}
    if (n > kMaxModuli) return false;
  }
  if (n < kMinModuli || n > kMaxModuli) return false;
  // at most 52 bits: X = x 2^(p+1) rounded to an integer must be exact in
  // FP64; the automatic choice keeps the 46-bit target (three 16-bit digits
  // per operand in the gathers), an explicit moduli count all its bits
  const int p = std::min(residue_bits(n, Kr), want > 0 ? 52 : kResidueBitsTarget);
  if (p < 20) return false;
  ResiduePlan& R = *out;
  std::memset(&R, 0, sizeof(R));
  R.p = p;
  R.rs.n = n;
  R.rs.pscale = std::ldexp(1.0, p + 1);
  const u128 M = moduli_product(n);
  R.crt.n = n;
  R.crt.shift = 2 * (p + 1);
  R.rs.p = p;
  R.rs.ndig = p <= 46 ? 3 : 4;
  int b = 0;
  while (b < 127 && (M >> b) != 0) ++b;
  // bits [b - 41 (k + 1), b - 41 k) of x, k = 0..2, as a double (exact)
  auto part = [&](u128 x, int k) {
    const int lo = std::max(0, b - 41 * (k + 1)), hi = std::max(0, b - 41 * k);
    return std::ldexp((double)(uint64_t)((x >> lo) & (((u128)1 << (hi - lo)) - 1)), lo);
  };
  for (int i = 0; i < n; ++i) {
    const int m = kModuliTable[i];
    const u128 Mi = M / (u128)m;
    const int mi_mod = (int)(Mi % (u128)m);
    int y = 0;
    for (int c = 1; c < m; ++c)
      if ((mi_mod * c) % m == 1) { y = c; break; }
    R.crt.mod[i] = m;
    const u128 s = Mi * (u128)y;
    R.crt.s1[i] = part(s, 0);
    R.crt.s2[i] = part(s, 1);
    R.crt.s3[i] = part(s, 2);
  }
  R.crt.M1 = part(M, 0);
  R.crt.M2 = part(M, 1);
  R.crt.M3 = part(M, 2);
  R.crt.invM = 1.0 / (double)M;
  return true;
}

// Row maxima of the FP64 exponent fields (the slice scales), streamed without
// shared-memory staging: each thread keeps the running maximum of the rows it
// touches in registers over all K tiles of its CTA, and the CTA merges them once
// at the end.  Thread -> (row, k) mapping as in gather_kernel.  SPREAD: the same
// for a RowSpread per row, written per CTA (P.spread).
template <bool CPLX, bool SPREAD>
__device__ __forceinline__ void rowmax_body(const GatherParams& P, int64_t rowtile, int ky, int kstep) {
  using E = typename std::conditional<CPLX, double2, double>::type;
  constexpr int TM = gather_rows<E>(), TK = kGK, IT = TM * TK / kGThreads;
  __shared__ unsigned sm_max[TM];
  __shared__ RowSpread sm_spread[SPREAD ? kGThreads : 1];
  const int tid = threadIdx.x;
  if (tid < TM) sm_max[tid] = 0;
  const int64_t m0 = rowtile * TM;
  const E* src = (const E*)P.src;
  const int64_t nkt = (P.K + TK - 1) / TK;
  auto take = [](unsigned& e, RowSpread& S, const E& v) {
    if constexpr (SPREAD) {
      if constexpr (CPLX) { spread_add(S, v.x); spread_add(S, v.y); }
      else spread_add(S, v);
    } else {
      if constexpr (CPLX) e = max(e, max(exp_field(v.x), exp_field(v.y)));
      else e = max(e, exp_field(v));
    }
  };
  if (!P.lanes_on_k) {
    // rows contiguous in the source: each thread keeps one row (tid % TM) and
    // walks k = tid / TM + j * (threads / TM) -- one offset, one maximum
    constexpr int KS = kGThreads / TM;
    const int mm = tid % TM;
    const int64_t lm = m0 + mm < P.rows ? P.lm[m0 + mm] : -1;
    unsigned e = 0;
    RowSpread S{0ull, 0u, 0u};
    if (lm >= 0) {
      for (int64_t kt = ky; kt < nkt; kt += kstep) {
        const int64_t k0 = kt * TK + tid / TM;
        E v[TK / KS];  // all loads before the first is used
#pragma unroll
        for (int it = 0; it < TK / KS; ++it) {
          const int64_t k = k0 + it * KS;
          v[it] = k < P.K ? src[lm + P.lk[k]] : E{};
        }
#pragma unroll
        for (int it = 0; it < TK / KS; ++it) take(e, S, v[it]);
      }
    }
    if constexpr (SPREAD) { e = S.e; sm_spread[tid] = S; }
    __syncthreads();
    if (e) atomicMax(&sm_max[mm], e);
    __syncthreads();
    if (tid < TM && m0 + tid < P.rows) {
      if (sm_max[tid]) atomicMax(&P.rowE[m0 + tid], sm_max[tid]);
      if constexpr (SPREAD) {
#pragma unroll
        for (int i = 1; i < KS; ++i) spread_merge(S, sm_spread[tid + i * TM]);
        P.spread[(m0 + tid) * kstep + ky] = S;
      }
    }
    return;
  }
  if constexpr (SPREAD) {
    // half a warp per row: a thread counts in TM / 16 rows only (16 rows a thread, as
    // below, take 128 registers: 200 against 131 us for the 96/24 ladder)
    constexpr int KL = 16, RR = TM * KL / kGThreads, KR = TK / KL;
    const int kl = tid % KL, r0 = tid / KL;
    int64_t lmv[RR];
    RowSpread S[RR];
#pragma unroll
    for (int i = 0; i < RR; ++i) {
      const int64_t m = m0 + r0 + i * (kGThreads / KL);
      lmv[i] = m < P.rows ? P.lm[m] : -1;
      S[i] = {0ull, 0u, 0u};
    }
    for (int64_t kt = ky; kt < nkt; kt += kstep) {
      E v[RR][KR];  // all loads before the first is used
#pragma unroll
      for (int j = 0; j < KR; ++j) {
        const int64_t k = kt * TK + kl + j * KL;
        const int64_t lk = k < P.K ? P.lk[k] : 0;
#pragma unroll
        for (int i = 0; i < RR; ++i) v[i][j] = lmv[i] >= 0 && k < P.K ? src[lmv[i] + lk] : E{};
      }
#pragma unroll
      for (int i = 0; i < RR; ++i)
#pragma unroll
        for (int j = 0; j < KR; ++j) {
          if constexpr (CPLX) { spread_add(S[i], v[i][j].x); spread_add(S[i], v[i][j].y); }
          else spread_add(S[i], v[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < RR; ++i) {
      RowSpread T = S[i];
#pragma unroll
      for (int o = KL / 2; o > 0; o >>= 1)
        spread_merge(T, RowSpread{__shfl_xor_sync(0xffffffffu, T.bins, o), __shfl_xor_sync(0xffffffffu, T.e, o), 0u});
      const int64_t m = m0 + r0 + i * (kGThreads / KL);
      if (kl == 0 && m < P.rows) {
        if (T.e) atomicMax(&P.rowE[m], T.e);
        P.spread[m * kstep + ky] = T;
      }
    }
    return;
  }
  int64_t lmv[IT];
  unsigned emax[IT];
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int idx = tid + it * kGThreads;
    const int mm = idx / TK;
    lmv[it] = m0 + mm < P.rows ? P.lm[m0 + mm] : -1;
    emax[it] = 0;
  }
  for (int64_t kt = ky; kt < nkt; kt += kstep) {
    const int64_t k0 = kt * TK;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int idx = tid + it * kGThreads;
      const int kk = idx % TK;
      if (lmv[it] >= 0 && k0 + kk < P.K) {
        const E v = src[lmv[it] + P.lk[k0 + kk]];
        if constexpr (CPLX) emax[it] = max(emax[it], max(exp_field(v.x), exp_field(v.y)));
        else emax[it] = max(emax[it], exp_field(v));
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int it = 0; it < IT; ++it) {
    const int idx = tid + it * kGThreads;
    const int mm = idx / TK;
    // the lanes of a warp hold one row: one atomic per warp and row instead of 32 on
    // one shared word (the 40^6 product's row maxima: 36 -> 27 us)
    const unsigned e = __reduce_max_sync(0xffffffffu, emax[it]);
    if ((tid & 31) == 0 && e) atomicMax(&sm_max[mm], e);
  }
  __syncthreads();
  if (tid < TM && sm_max[tid] && m0 + tid < P.rows) atomicMax(&P.rowE[m0 + tid], sm_max[tid]);
}

template <bool CPLX, bool SPREAD>
__global__ void __launch_bounds__(kGThreads) rowmax_kernel(const __grid_constant__ GatherPair Q) {
  const bool second = blockIdx.x >= Q.ctas_a;
  const unsigned x = second ? blockIdx.x - Q.ctas_a : blockIdx.x, rows = second ? Q.rows_b : Q.rows_a;
  const unsigned ky = x / rows, rt = x - ky * rows;
  const GatherParams P = second ? Q.b : Q.a;
  rowmax_body<CPLX, SPREAD>(P, rt, (int)ky, second ? Q.gy_b : Q.gy_a);
}

template <bool CPLX>
__global__ void __launch_bounds__(kGThreads) rowmax_grouped_kernel(const GatherParams* __restrict__ jobs,
                                                                   const int2* __restrict__ map) {
  const int2 jm = map[blockIdx.x];
  const GatherParams P = jobs[jm.x];
  rowmax_body<CPLX, false>(P, jm.y, blockIdx.y, gridDim.y);
}

// CTAs per row tile of one operand: enough to fill the GPU several times over, each
// walking a strided set of K tiles.
int64_t k_splits(int64_t rows, int64_t kt) {
  return std::max<int64_t>(1, std::min<int64_t>(kt, (int64_t)num_sms() * 16 / std::max<int64_t>(1, rows)));
}
template <bool CPLX>
int rowmax_splits(int64_t rows, int64_t K) {
  constexpr int64_t TM = CPLX ? gather_rows<double2>() : gather_rows<double>();
  return (int)k_splits((rows + TM - 1) / TM, (K + kGK - 1) / kGK);
}

// Grid of a launch over both operands.
int pair_grid(GatherPair* Q, const GatherParams& a, const GatherParams& b, int64_t rows_a, int64_t kt_a, int64_t rows_b,
              int64_t kt_b, unsigned* grid) {
  const int64_t ga = k_splits(rows_a, kt_a), gb = k_splits(rows_b, kt_b);
  if (rows_a * ga + rows_b * gb > INT32_MAX) { set_error("gather grid too large"); return TB_ERR_LIMIT; }
  Q->a = a;
  Q->b = b;
  Q->refused = nullptr;
  Q->rows_a = (unsigned)rows_a;
  Q->rows_b = (unsigned)rows_b;
  Q->gy_a = (int)ga;
  Q->gy_b = (int)gb;
  Q->ctas_a = (unsigned)(rows_a * ga);
  *grid = (unsigned)(rows_a * ga + rows_b * gb);
  return 0;
}

template <bool CPLX>
int run_rowmax(const GatherParams& a, const GatherParams& b, cudaStream_t s) {
  constexpr int64_t TM = CPLX ? gather_rows<double2>() : gather_rows<double>();
  GatherPair Q;
  unsigned grid;
  if (int e = pair_grid(&Q, a, b, (a.rows + TM - 1) / TM, (a.K + kGK - 1) / kGK, (b.rows + TM - 1) / TM,
                        (b.K + kGK - 1) / kGK, &grid))
    return e;
  if (a.spread) rowmax_kernel<CPLX, true><<<grid, kGThreads, 0, s>>>(Q);
  else rowmax_kernel<CPLX, false><<<grid, kGThreads, 0, s>>>(Q);
  TB_CHECK_LAUNCH();
  return 0;
}

template <int MODEA, int MODEB>
int run_gather(const GatherParams& a, const GatherParams& b, int64_t rows_a, int64_t rows_b, int64_t ktiles,
               const unsigned* refused, cudaStream_t s) {
  GatherPair Q;
  unsigned grid;
  if (int e = pair_grid(&Q, a, b, rows_a, ktiles, rows_b, ktiles, &grid)) return e;
  Q.refused = refused;
  constexpr int smem = std::max(gather_smem_bytes<MODEA>(), gather_smem_bytes<MODEB>());
  auto launch = [&](auto kern, DeviceOnce& once) -> int {
    const cudaError_t e = smem_limit_once(once, kern, smem);
    if (e != cudaSuccess) { set_error("gather smem attribute: %s", cudaGetErrorString(e)); return TB_ERR_CUDA; }
    kern<<<grid, kGThreads, smem, s>>>(Q);
    return 0;
  };
  static DeviceOnce once3, once4;
  int err = 0;
  if constexpr (MODEA == G_RESID_R8 || MODEA == G_RESID_C8A) {
    err = a.rs.ndig > 3 ? launch(gather_kernel<MODEA, MODEB, 4>, once4) : launch(gather_kernel<MODEA, MODEB, 3>, once3);
  } else {
    err = launch(gather_kernel<MODEA, MODEB>, once3);
  }
  if (err) return err;
  TB_CHECK_LAUNCH();
  return 0;
}


}  // namespace
}  // namespace tb
