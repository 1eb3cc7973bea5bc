// tb_tc.cu -- the tensor-core contraction path (TB_METHOD_FUSED).
//
// FP64 (R8, C8): Ozaki-style splitting into 8-bit slices.  Each row m of the
// matricized left operand is scaled by 2^-e_m (e_m from the row's largest
// exponent) into (-1/2, 1/2) and cut into s balanced signed 8-bit digits of
// weight 2^-(8i+7), i = 0..s-1 (exact in FP64; see fixed55); the right
// operand likewise per column.  The tcgen05 GEMM (tb_tc_gemm.cuh) multiplies
// slice pairs (i, j) with i + j <= s - 1 exactly in INT32 (kind::i8),
// grouping pairs of equal i + j, split along K where needed, into one TMEM
// accumulator while no INT32 overflow is possible, and the epilogue adds
// 2^(e_m + f_n - 8(i+j) - 14) * acc in FP64 into D.
// FP32 (R4, C4): each value splits into BF16 high and low parts; the three
// products hi*hi + hi*lo + lo*hi accumulate in FP32 in TMEM.
// Complex data runs as a real GEMM of twice the size: A' = [Ar Ai] interleaved
// along K, B' rows (2n, 2n+1) = ([Br, -Bi], [Bi, Br]), so that columns (2n,
// 2n+1) of the product hold the real and imaginary parts of C(m, n).
//
// The operand preparation reads the tensors in their own layouts through
// per-row and per-index offset tables (the input permutations are fused into
// the conversion to slices or BF16 parts),
// and the epilogue writes D through per-row and per-column offset tables (the
// output permutation) with alpha and beta applied.
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "tb_common.cuh"
#include "tb_contract.h"
#include "tb_direct.h"
#include "tb_permute.cuh"
#include "tb_tc_gemm.cuh"
#include "tb_tc_prep.cuh"

namespace tb {

namespace {

// ---- driver ----------------------------------------------------------------------
constexpr int kDefaultSlices = 6;
constexpr int kMaxSlices = 7;  // 7 slices hold all 55 bits of the fixed-point value
constexpr int kBf16PassKBlocks = 32;  // split-BF16: K blocks (64 values each) per accumulator pass

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// One operand of the GEMM: a source tensor, its row groups and its contracted
// dims (Z.k order), each with strides in this tensor (s1) and in D (s2).
struct Operand {
  const void* ptr;
  std::vector<MGroup> rows;   // uncontracted groups: s1 = stride in this tensor, s2 = stride in D
  std::vector<MGroup> ks;     // contracted groups: s1 = stride in this tensor
  bool conj;
};

template <int BN, bool I8, int EPI>
int launch_tc(const TcGemmParams& P, cudaStream_t s) {
  constexpr size_t smem = tc_smem_bytes<BN>();
  static DeviceOnce attr;
  const cudaError_t e = smem_limit_once(attr, tc_gemm_kernel<BN, I8, EPI>, (int)smem);
  if (e != cudaSuccess) { set_error("tcgen05 GEMM smem attribute: %s", cudaGetErrorString(e)); return TB_ERR_CUDA; }
  const int grid = std::max(1, std::min(gemm_units<EPI>(P), num_sms()));
  tc_gemm_kernel<BN, I8, EPI><<<grid, kTcThreads, smem, s>>>(P);
  TB_CHECK_LAUNCH();
  return 0;
}

// CTA-pair kernel: grid = 2 x (pairs that can be resident at once, capped by the tiles).
template <int BN, bool I8, int EPI>
int launch_tc2(const TcGemmParams& P, cudaStream_t s) {
  constexpr size_t smem = tc2_smem_bytes<BN>();
  // per device: the shared-memory limit and the pairs resident at once
  static std::atomic<int> max_pairs_of[64];
  const int dev = current_device();
  int max_pairs = max_pairs_of[dev].load(std::memory_order_relaxed);
  if (!max_pairs) {
    cudaError_t e = cudaFuncSetAttribute(tc_gemm2_kernel<BN, I8, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) { set_error("tcgen05 pair GEMM smem attribute: %s", cudaGetErrorString(e)); return TB_ERR_CUDA; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)num_sms(), 1, 1);
    cfg.blockDim = dim3(kTcThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, tc_gemm2_kernel<BN, I8, EPI>, &cfg);
    if (e != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = num_sms() / 2;
    }
    max_pairs = n;
    max_pairs_of[dev].store(n, std::memory_order_relaxed);
  }
  const int pairs = std::max(1, std::min(gemm_units<EPI>(P), max_pairs));
  tc_gemm2_kernel<BN, I8, EPI><<<2 * pairs, kTcThreads, smem, s>>>(P);
  TB_CHECK_LAUNCH();
  return 0;
}

template <int BN>
int launch_tc_epi(const TcGemmParams& P, int epi, bool pair, cudaStream_t s) {
  if (pair) {
    switch (epi) {
      case EPI_RESID: return launch_tc2<BN, true, EPI_RESID>(P, s);
      case EPI_OZAKI_R: return launch_tc2<BN, true, EPI_OZAKI_R>(P, s);
      case EPI_OZAKI_C: return launch_tc2<BN, true, EPI_OZAKI_C>(P, s);
      case EPI_BF16_R: return launch_tc2<BN, false, EPI_BF16_R>(P, s);
      default: return launch_tc2<BN, false, EPI_BF16_C>(P, s);
    }
  }
  switch (epi) {
    case EPI_RESID: return launch_tc<BN, true, EPI_RESID>(P, s);
    case EPI_OZAKI_R: return launch_tc<BN, true, EPI_OZAKI_R>(P, s);
    case EPI_OZAKI_C: return launch_tc<BN, true, EPI_OZAKI_C>(P, s);
    case EPI_BF16_R: return launch_tc<BN, false, EPI_BF16_R>(P, s);
    default: return launch_tc<BN, false, EPI_BF16_C>(P, s);
  }
}

}  // namespace

int select_method(int dtk, const Matricization& Z, const tb_plan_t* plan) {
  (void)dtk;
  if (plan && plan->method != TB_METHOD_AUTO) return plan->method;
  // tensor cores pay off once the GEMM is large enough to fill the GPU
  const double flops = 2.0 * (double)Z.M * (double)Z.N * (double)Z.K;
  if (Z.M >= 64 && Z.N >= 32 && Z.K >= 64 && flops >= 4e9) return TB_METHOD_FUSED;
  return TB_METHOD_TTGT;
}

// Fixed launches, operand bytes read and plane bytes written (MB), MMA work of
// whole rounds of work units (10^6 operations), output bytes (MB) and rounds,
// weighted by a fit to 212 random contractions on B200 (5% rms for R8, 8% for
// R4): a round of units costs its MMAs plus about 3 us, D's bytes run at 2.6 to
// 4.4 TB/s, operands at 4 to 7 TB/s.  Products that take 192-wide tiles are predicted
// as by 256-wide ones: three tiles of 192 columns took 7% less than three of 256.
double predicted_fused_us(const Matricization& Z, int dtk, int n) {
  const bool cplx = is_complex(dtk), f64 = is_double(dtk);
  bool swap = false;  // rows: the operand holding D's fastest dimension
  {
    int64_t lm = INT64_MAX, ln = INT64_MAX;
    for (auto& g : Z.m) if (g.ext > 1) lm = std::min(lm, g.s2);
    for (auto& g : Z.n) if (g.ext > 1) ln = std::min(ln, g.s2);
    swap = ln < lm;
  }
  const double M = (double)(swap ? Z.N : Z.M), N = (double)(swap ? Z.M : Z.N), K = (double)Z.K, es = elem_bytes(dtk);
  const double Kr = cplx ? 2 * K : K, Nr = cplx ? 2 * N : N;
  const double bn = Nr >= 192 ? 256 : 128;
  const double mt = std::ceil(M / 128), nt = std::ceil(Nr / bn), kp = std::ceil(Kr / 128) * 128;
  const double reads = f64 ? 2 : 1, plane = f64 ? n : 4;  // row maxima read FP64 operands a second time
  const double gather = ((M + N) * K * es * reads + (mt * 128 + nt * bn) * kp * plane) * 1e-6;
  const double sms = 148;
  if (f64) {
    const double rounds = std::ceil(n * mt * nt / sms);
    const double work = rounds * sms * 128 * bn * kp * 2e-6, out = M * Nr * (n + 16) * 1e-6;
    return cplx ? 41.3 + 0.23 * gather + 0.000275 * work + 0.271 * out + 3.53 * rounds
                : 44.4 + 0.271 * gather + 0.000293 * work + 0.384 * out + 3.33 * rounds;
  }
  const double passes = std::ceil(std::ceil(Kr * 2 / 128) / 32), rounds = std::ceil(mt * nt / sms);
  const double work = rounds * sms * 128 * bn * kp * 6e-6, out = M * Nr * 8 * passes * 1e-6;
  return cplx ? 27.0 + 0.135 * gather + 0.000448 * work + 0.144 * out + 9.19 * rounds * passes
              : 30.5 + 0.224 * gather + 0.000437 * work + 0.331 * out + 14.8 * rounds * passes;
}

int contract_fused(const Matricization& Z0, int dtk, const int* ddims, void* d, const int* ldims, const void* l,
                   const int* rdims, const void* r, double ar, double ai, bool accumulate, int lconj, int rconj,
                   const tb_plan_t* plan, cudaStream_t s, tb_contract_stats_t* stats, const DirectPlan* otherwise) {
  (void)ddims;
  if (Z0.K < 1 || Z0.M < 1 || Z0.N < 1 || Z0.k.empty()) return TB_ERR_NOT_IMPLEMENTED;
  Matricization Z = Z0;
  // unit extents carry no index; rows in D-stride order so that consecutive
  // epilogue lanes write consecutive D
  auto by_d = [](const MGroup& x, const MGroup& y) { return x.s2 < y.s2; };
  auto no_units = [](std::vector<MGroup>& g) {
    g.erase(std::remove_if(g.begin(), g.end(), [](const MGroup& x) { return x.ext == 1; }), g.end());
  };
  auto unit_of = [](const std::vector<MGroup>& g, bool second) {
    for (size_t i = 0; i < g.size(); ++i)
      if ((second ? g[i].s2 : g[i].s1) == 1) return (int)i;
    return -1;
  };
  no_units(Z.m);
  no_units(Z.n);
  no_units(Z.k);
  std::stable_sort(Z.m.begin(), Z.m.end(), by_d);
  std::stable_sort(Z.n.begin(), Z.n.end(), by_d);
  // the operand holding D's fastest dimension plays the row (M) role
  const bool swap = !Z.n.empty() && (Z.m.empty() || Z.n[0].s2 < Z.m[0].s2);
  // contracted order: an index that is contiguous in an operand comes first (the
  // larger operand's where both have one), so that its gather runs along it
  {
    const int kl = unit_of(Z.k, false), kr = unit_of(Z.k, true);
    const bool by_r = kl < 0 || (kr >= 0 && Z.N > Z.M);
    std::stable_sort(Z.k.begin(), Z.k.end(), [&](const MGroup& x, const MGroup& y) {
      return by_r && kr >= 0 ? x.s2 < y.s2 : x.s1 < y.s1;
    });
  }
  Operand Lop{l, Z.m, {}, lconj != 0}, Rop{r, Z.n, {}, rconj != 0};
  for (auto g : Z.k) {
    Lop.ks.push_back(g);                       // s1 = L stride
    MGroup h = g; h.s1 = g.s2; Rop.ks.push_back(h);  // R stride
  }
  (void)ldims; (void)rdims;
  const Operand& A = swap ? Rop : Lop;
  Operand& B = swap ? Lop : Rop;
  // columns: the operand's contiguous group first (a column's place among the
  // others matters to no write of D)
  if (const int u = unit_of(B.rows, false); u > 0) std::rotate(B.rows.begin(), B.rows.begin() + u, B.rows.begin() + u + 1);
  const bool cplx = is_complex(dtk), i8 = is_double(dtk);
  int64_t M = 1, Nc = 1;
  for (auto& g : A.rows) M *= g.ext;
  for (auto& g : B.rows) Nc *= g.ext;
  const int64_t K = Z.K;
  const int64_t Kr = cplx ? 2 * K : K, Nr = cplx ? 2 * Nc : Nc;
  const int64_t Kpad = round_up(Kr, 128);
  // N tile: what the plan asks for, else 256 (128 for narrow products).  Without a
  // request residue products take 192 where the tiles then read a twelfth less (128 +
  // BN rows of 128 bytes per K block), which is where fewer of their columns are
  // padding: N = 576 in three tiles of 192 instead of three of 256 (9216 x 576 x 9216
  // by 15 moduli: GEMM 642 -> 597 us, 1589 -> 1553 us in all).
  const bool asks_tile = plan && (plan->tile_n == 128 || plan->tile_n == 256);
  int BN = asks_tile ? plan->tile_n : Nr >= 192 ? 256 : 128;
  if (!asks_tile && i8 && !(plan && (plan->slices > 0 || plan->moduli < 0 || plan->tile_m == 256)) && Nr > 128 &&
      12 * ((Nr + 191) / 192) * (128 + 192) <= 11 * ((Nr + 255) / 256) * (128 + 256))
    BN = 192;
  // M tile: one SM per 128-row tile unless the plan asks for SM pairs (256
  // rows); the pair kernel halves the B traffic per SM but measured no faster
  // on the CCSD-like shapes, whose GEMMs run at the power cap.
  const bool pair = plan && plan->tile_m == 256;
  const int TM = pair ? 256 : 128;
  const int64_t Mpad = round_up(M, TM);
  // products and passes: an entry multiplies plane a of A by plane b of B over
  // a K-block range; the entries of a pass share one exact INT32 accumulator.
  struct Entry { int a, b, kb0, kb1; };
  std::vector<std::vector<Entry>> passes;
  std::vector<int> shifts;
  const int kblocks = (int)(Kpad * (i8 ? 1 : 2) / 128);  // 128-byte K blocks
  int S = 0, npa = 2, npb = 2;
  // R8/C8: modular residues (one exact INT8 GEMM per modulus, fewer than the
  // slice pairs) unless the plan asks for INT8 slices or the contraction
  // needs more moduli; K ranges longer than one exact INT32 pass (1023 K
  // blocks) are cut into equal chunks whose residues the epilogue adds mod m.
  ResiduePlan RP;
  const int res_nch = (kblocks + kMaxPassBlocks - 1) / kMaxPassBlocks;
  const bool resid = i8 && !(plan && (plan->slices > 0 || plan->moduli < 0)) &&
                     plan_residues(Kr, plan ? plan->moduli : 0, &RP) && RP.rs.n * res_nch <= kMaxProducts;
  if (i8 && plan && plan->moduli > 0 && !resid) {
    set_error("modular residues: %d moduli do not fit this contraction (K = %lld)", plan->moduli, (long long)Kr);
    return TB_ERR_INVALID_ARGS;
  }
  if (otherwise && (!resid || RP.p < 51 || Kr > 65535)) return TB_ERR_NOT_IMPLEMENTED;
  if (!resid && BN == 192) BN = 256;  // residues only
  const int64_t Npad = round_up(Nr, BN);
  if (Mpad / 128 * (Npad / BN) > INT32_MAX || M > INT32_MAX || Nr > INT32_MAX) return TB_ERR_LIMIT;
  if (resid) {
    const int chunk = (kblocks + res_nch - 1) / res_nch;
    for (int i = 0; i < RP.rs.n; ++i)
      for (int kb = 0; kb < kblocks; kb += chunk) {
        passes.push_back({{i, i, kb, std::min(kblocks, kb + chunk)}});
        shifts.push_back(RP.crt.mod[i]);  // the epilogue's modulus
      }
    npa = npb = RP.rs.n;
  } else if (i8) {
    S = (plan && plan->slices > 0) ? plan->slices : kDefaultSlices;
    if (S < 2 || S > kMaxSlices) { set_error("slice count %d outside 2..%d", S, kMaxSlices); return TB_ERR_INVALID_ARGS; }
    // |slice| <= 128, so one K block (128 products) adds at most 128^3.
    const int64_t cap = INT32_MAX;
    // The products of one i + j share a pass while the sum stays exact
    // (at most cap / 128^3 = 1023 K blocks per pass).  A group that needs
    // several passes gets passes of equal size, so that each pass's MMAs are
    // long enough to hide the previous pass's epilogue (1152 blocks: 576 +
    // 576, not 1023 + 129).
    const int64_t per_block = (int64_t)128 * 128 * 128;
    const int64_t max_blocks = cap / per_block;
    for (int dsum = 2; dsum <= S + 1; ++dsum) {   // 1-based slice indices with i + j = dsum
      int64_t total = 0;
      for (int i = 1; i < dsum; ++i)
        if (i <= S && dsum - i <= S) total += kblocks;
      if (total == 0) continue;
      const int64_t npass = (total + max_blocks - 1) / max_blocks;
      const int64_t room_max = (total + npass - 1) / npass;  // <= max_blocks
      std::vector<Entry> cur;
      int64_t load = 0;
      for (int i = 1; i < dsum; ++i) {
        const int j = dsum - i;
        if (i > S || j > S) continue;
        for (int kb = 0; kb < kblocks;) {
          if (load >= room_max) { passes.push_back(cur); shifts.push_back(8 * dsum - 2); cur.clear(); load = 0; }
          const int n = (int)std::min<int64_t>(room_max - load, kblocks - kb);
          cur.push_back({i - 1, j - 1, kb, kb + n});
          load += n;
          kb += n;
        }
      }
      if (!cur.empty()) { passes.push_back(cur); shifts.push_back(8 * dsum - 2); }
    }
    npa = npb = S;
  } else {
    // The FP32 accumulation of the tensor cores loses accuracy about linearly
    // with K (R4 CCSD-like, K = 36864: 1.8e-4 relative in one pass), so the K
    // range is cut into passes of kBf16PassKBlocks blocks (longer where the
    // entry limit requires) that the epilogue adds into D, one rounding each.
    static const int pass_kb = [] {
      const char* e = getenv("TB_BF16_PASS_KB");  // tuning knob
      const int v = e ? atoi(e) : 0;
      return v > 0 ? v : kBf16PassKBlocks;
    }();
    const int terms = (plan && plan->bf16_terms == 4) ? 4 : 3;
    const int max_passes = kMaxProducts / terms;  // the parameter block holds kMaxProducts entries
    const int step = std::max(pass_kb, (kblocks + max_passes - 1) / max_passes);
    for (int kb = 0; kb < kblocks; kb += step) {
      const int k1 = std::min(kblocks, kb + step);
      std::vector<Entry> p3 = {{0, 0, kb, k1}, {0, 1, kb, k1}, {1, 0, kb, k1}};
      if (terms == 4) p3.push_back({1, 1, kb, k1});
      passes.push_back(p3);
      shifts.push_back(0);
    }
  }
  int nprod = 0, nplane_products = 0;
  for (auto& p : passes) {
    nprod += (int)p.size();
    for (auto& e : p) nplane_products += (e.kb0 == 0);  // count each plane pair once
  }
  if (nprod > kMaxProducts || (int)passes.size() > kMaxProducts) {
    set_error("tensor-core plan needs %d GEMM entries in %d passes (limit %d)", nprod, (int)passes.size(),
              kMaxProducts);
    return TB_ERR_NOT_IMPLEMENTED;
  }
  // scratch: operand planes, offset tables, exponents
  const int oes = i8 ? 1 : 2;
  const size_t bytesA = (size_t)npa * Mpad * Kpad * oes, bytesB = (size_t)npb * Npad * Kpad * oes;
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t offA = 0, offB = al(bytesA), offDm = offB + al(bytesB), offDn = offDm + al(M * 8),
               offLA = offDn + al(Nc * 8), offLB = offLA + al(M * 8), offKA = offLB + al(Nc * 8),
               offKB = offKA + al(K * 8), offRE = offKB + al(K * 8), offCE = offRE + al(M * 4),
               offNB = offCE + al(Nc * 4), offRX = offNB + 256, offCX = offRX + al(M * 4), offBR = offCX + al(Nr * 4),
               offBC = offBR + al(M * 4), offRES = offBC + al(Nc * 4),
               offSA = offRES + (resid ? al((size_t)RP.rs.n * Npad * Mpad) : 0);
  const int splitsA = !otherwise ? 0 : cplx ? rowmax_splits<true>(M, K) : rowmax_splits<false>(M, K);
  const int splitsB = !otherwise ? 0 : cplx ? rowmax_splits<true>(Nc, K) : rowmax_splits<false>(Nc, K);
  const size_t offSB = offSA + al(sizeof(RowSpread) * splitsA * M), total = offSB + al(sizeof(RowSpread) * splitsB * Nc);
  unsigned char* ws = nullptr;
  if (int e = scratch_alloc((void**)&ws, total, s)) return e;
  int err = 0;
  int8_t* Ap = (int8_t*)(ws + offA);
  int8_t* Bp = (int8_t*)(ws + offB);
  int64_t* dm = (int64_t*)(ws + offDm);
  int64_t* dn = (int64_t*)(ws + offDn);
  int64_t* lmA = (int64_t*)(ws + offLA);
  int64_t* lmB = (int64_t*)(ws + offLB);
  int64_t* lkA = (int64_t*)(ws + offKA);
  int64_t* lkB = (int64_t*)(ws + offKB);
  unsigned* rowE = (unsigned*)(ws + offRE);
  unsigned* colE = (unsigned*)(ws + offCE);
  int* rowx = (int*)(ws + offRX);
  int* colx = (int*)(ws + offCX);
  int* badrows = (int*)(ws + offBR);  // rows of A / columns of B holding a NaN or an infinity
  int* badcols = (int*)(ws + offBC);
  int* nbad = (int*)(ws + offNB);     // counts of both, the GEMM's work-unit counter, GuardParams::words from nbad[8] on
  const unsigned* refused = otherwise ? (const unsigned*)nbad + 15 : nullptr;
  const int64_t ksrc_pad = cplx ? Kpad / 2 : Kpad;  // padded K in source elements
  do {
    // Offset tables and cleared words (row maxima, counters) in one launch.  A's
    // rows run in blocks of its contiguous group where that is not D's fastest
    // one: the gathers then read 64 bytes at a time instead of single elements
    // (40^6 R8: row maxima and gathers 132 -> 60 us).  The residue path's
    // reconstruction steps over the blocks; the epilogues that write D directly
    // write runs of four instead, once per accumulator pass, so they take blocks
    // only where the operand's bytes outweigh that.
    const int pa = !A.ks.empty() && A.ks[0].s1 == 1 ? -1 : unit_of(A.rows, false);
    const bool blocked = pa > 0 && (resid || 32.0 * (double)K > 8.0 * (double)Nr * (double)passes.size());
    const int kRowBlock = 8;
    TableParams TP;
    std::memset(&TP, 0, sizeof(TP));
    if (blocked) set_blocked_job(&TP.job[0], A.rows, pa, kRowBlock, lmA, dm);
    else set_table_job(&TP.job[0], A.rows, lmA, dm);
    set_table_job(&TP.job[1], B.rows, lmB, dn);
    {
      std::vector<MGroup> ks = A.ks;  // s1: A's stride, s2: B's
      for (size_t i = 0; i < ks.size(); ++i) ks[i].s2 = B.ks[i].s1;
      set_table_job(&TP.job[2], ks, lkA, lkB);
    }
    TP.zero = (uint32_t*)rowE;
    TP.zero_words = (int64_t)(offRX - offRE) / 4;
    if ((err = run_tables(TP, s))) break;
    GatherParams GA{}, GB{};
    GA.src = A.ptr; GA.lm = lmA; GA.lk = lkA; GA.rows = M; GA.K = K; GA.kpad = Kpad; GA.pstride = Mpad * Kpad;
    GA.planes = Ap; GA.rowE = rowE; GA.slices = S; GA.isign = A.conj ? -1.0 : 1.0;
    // 16-byte copies: whole groups of k that are contiguous and aligned in the operand
    auto lanes = [&](GatherParams& G, const Operand& O, bool rows_run) {
      const int64_t vw = 16 / elem_bytes(dtk);
      G.lanes_on_k = (!O.ks.empty() && O.ks[0].s1 == 1) || !rows_run ? 1 : 0;
      bool vec = !O.ks.empty() && O.ks[0].s1 == 1 && O.ks[0].ext % vw == 0 && (uintptr_t)O.ptr % 16 == 0;
      for (size_t i = 1; i < O.ks.size(); ++i) vec = vec && O.ks[i].s1 % vw == 0;
      for (auto& g : O.rows) vec = vec && g.s1 % vw == 0;
      G.vec = vec ? 1 : 0;
    };
    lanes(GA, A, blocked || pa == 0);
    if (resid) GA.rs = RP.rs;
    GB.src = B.ptr; GB.lm = lmB; GB.lk = lkB; GB.rows = Nc; GB.K = K; GB.kpad = Kpad; GB.pstride = Npad * Kpad;
    GB.planes = Bp; GB.rowE = colE; GB.slices = S; GB.isign = B.conj ? -1.0 : 1.0;
    lanes(GB, B, !B.rows.empty() && B.rows[0].s1 == 1);
    if (resid) GB.rs = RP.rs;
    const int tmr = i8 && cplx ? 32 : 64;               // gather tile rows (16-byte elements: 32)
    const int64_t gA = Mpad / tmr, gB = (cplx ? Npad / 2 : Npad) / tmr, gk = ksrc_pad / kGK;
    // row / column exponents and the lists of rows and columns flagged as
    // holding a NaN or an infinity (exponent field 2047): the epilogue leaves
    // their D entries to nonfinite_fixup_kernel.  nbad[0..1]: flagged row /
    // column counts; nbad[2]: the GEMM's work-unit counter.
    GuardParams GP{};
    if (otherwise) {
      GA.spread = (RowSpread*)(ws + offSA);
      GB.spread = (RowSpread*)(ws + offSB);
      GP.a = GA.spread; GP.b = GB.spread;
      GP.m = M; GP.n = Nc;
      GP.gy_a = splitsA; GP.gy_b = splitsB;
      GP.kr = (int)Kr;
      for (int i = 1; i <= 3; ++i) GP.need[i - 1] = std::max(1 << (55 + 2 * i - RP.p), (int)((Kr + 3) / 4));
      GP.words = (unsigned*)nbad + 8;
    }
    auto run_exps = [&]() -> int {
      // GUARD: eight lanes per row
      const int64_t items = otherwise ? 8 * (M + Nc) : M + Nr;
      const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((items + 255) / 256, otherwise ? 4 * num_sms() : 4096));
      if (otherwise)
        exps_pair_kernel<true><<<grid, 256, 0, s>>>(rowE, rowx, M, badrows, colE, colx, Nr, cplx ? 2 : 1, badcols, nbad, GP);
      else
        exps_pair_kernel<false><<<grid, 256, 0, s>>>(rowE, rowx, M, badrows, colE, colx, Nr, cplx ? 2 : 1, badcols, nbad, GP);
      TB_CHECK_LAUNCH();
      return 0;
    };
    if (i8) {
      if ((err = cplx ? run_rowmax<true>(GA, GB, s) : run_rowmax<false>(GA, GB, s))) break;
      if ((err = run_exps())) break;
      if (resid) err = cplx ? run_gather<G_RESID_C8A, G_RESID_C8B>(GA, GB, gA, gB, gk, refused, s)
                            : run_gather<G_RESID_R8, G_RESID_R8>(GA, GB, gA, gB, gk, refused, s);
      else err = cplx ? run_gather<G_SLICE_C8A, G_SLICE_C8B>(GA, GB, gA, gB, gk, refused, s)
                      : run_gather<G_SLICE_R8, G_SLICE_R8>(GA, GB, gA, gB, gk, refused, s);
      if (err) break;
    } else {
      if ((err = cplx ? run_gather<G_SPLIT_C4A, G_SPLIT_C4B>(GA, GB, gA, gB, gk, refused, s)
                      : run_gather<G_SPLIT_R4, G_SPLIT_R4>(GA, GB, gA, gB, gk, refused, s)))
        break;
      if ((err = run_exps())) break;  // the split gathers flag non-finite rows
    }
    // GEMM parameters
    // per call (about 2 KB), so that host threads contracting on different
    // streams never share a parameter block
    TcGemmParams P;
    std::memset(&P, 0, sizeof(P));
    if ((err = make_operand_map(&P.tmA, Ap, i8, Kpad, Mpad, npa, 128))) break;
    if ((err = make_operand_map(&P.tmB, Bp, i8, Kpad, Npad, npb, pair ? BN / 2 : BN))) break;
    P.M = (int)M; P.N = (int)Nr;
    P.mtiles = (int)(Mpad / TM); P.ntiles = (int)(Npad / BN);
    P.kblocks = (int)(Kpad * oes / 128);
    P.npass = (int)passes.size();
    P.res_nch = resid ? res_nch : 1;
    int q = 0;
    for (size_t p = 0; p < passes.size(); ++p) {
      P.pass_first[p] = q;
      P.pass_shift[p] = shifts[p];
      P.pass_magic[p] = resid ? (int)(4294967296ull / (unsigned long long)shifts[p]) : 0;
      for (auto& e : passes[p]) {
        P.prod_a[q] = e.a; P.prod_b[q] = e.b; P.prod_kb0[q] = e.kb0; P.prod_kb1[q] = e.kb1;
        ++q;
      }
    }
    P.pass_first[passes.size()] = q;
    P.D = d; P.dm = dm; P.dn = dn; P.rowexp = rowx; P.colexp = colx;
    const double realpha = cplx ? ar : (ar != 0.0 ? std::hypot(ar, ai) * (ar > 0 ? 1.0 : -1.0) : ai);
    P.ar = realpha; P.ai = cplx ? ai : 0.0;
    P.br = accumulate ? 1.0 : 0.0; P.bi = 0.0;
    P.err = device_error_word();
    P.refused = refused;
    P.nf_skip = resid ? 0 : 1;  // residues: crt_kernel leaves the flagged entries to the fix-up
    if (resid) {
      P.res = (uint8_t*)(ws + offRES);
      P.res_ld = Npad;
      P.res_plane = Npad * Mpad;
    }
    // Work units: dynamic (a counter) unless TB_TC_SCHED=0.  L2 policy: with
    // residues every unit reads one modulus's planes, and all m-tiles re-read
    // that modulus's B plane -- when it fits in about three quarters of L2, B
    // is kept (evict-last) and A streamed (evict-first).  TB_TC_L2HINT=0 / 1
    // turns the policy off / on regardless.
    static const int sched_env = [] { const char* e = getenv("TB_TC_SCHED"); return e ? atoi(e) : 1; }();
    static const int hint_env = [] { const char* e = getenv("TB_TC_L2HINT"); return e ? atoi(e) : -1; }();
    P.sched = sched_env ? (unsigned*)(nbad + 2) : nullptr;
    const size_t bplane = (size_t)Npad * Kpad * oes;
    P.l2hint = hint_env >= 0 ? (hint_env ? 1 : 0) : (resid && bplane <= (size_t)96 << 20 ? 1 : 0);
    const int epi = resid ? EPI_RESID : i8 ? (cplx ? EPI_OZAKI_C : EPI_OZAKI_R) : (cplx ? EPI_BF16_C : EPI_BF16_R);
    const int ts = timed_begin(s);
    err = BN == 256   ? launch_tc_epi<256>(P, epi, pair, s)
          : BN == 192 ? launch_tc<192, true, EPI_RESID>(P, s)
                      : launch_tc_epi<128>(P, epi, pair, s);
    timed_end(ts, s);
    if (err) break;
    if (resid) {
      // Chinese remainder reconstruction of the exact products into D
      CrtParams C = RP.crt;
      C.v = {(const uint8_t*)(ws + offRES), Npad, Npad * Mpad, M, Nc, blocked ? kRowBlock : 1, 1, dm, dn, d, rowx, colx};
      C.ar = realpha; C.ai = cplx ? ai : 0.0; C.br = P.br; C.bi = 0.0;
      C.refused = refused;
      const int64_t cg = crt_blocks(M, Nr, C.v.row_step);
      if (cg > INT32_MAX) { set_error("residue reconstruction grid too large"); err = TB_ERR_LIMIT; break; }
      if (cplx) crt_kernel<true><<<(unsigned)cg, 32 * kCrtWarps, 0, s>>>(C);
      else crt_kernel<false><<<(unsigned)cg, 32 * kCrtWarps, 0, s>>>(C);
      count_launch();
      if (cudaError_t e = cudaGetLastError()) {
        set_error("residue reconstruction launch: %s", cudaGetErrorString(e));
        err = TB_ERR_CUDA;
        break;
      }
    }
    // entries of rows / columns with a NaN or an infinity (returns at once without)
    NfParams F;
    F.srcA = A.ptr; F.srcB = B.ptr;
    F.lmA = lmA; F.lkA = lkA; F.lmB = lmB; F.lkB = lkB;
    F.dm = dm; F.dn = dn; F.D = d;
    F.M = M; F.N = Nc; F.K = K;
    F.rowE = rowE; F.badrows = badrows; F.badcols = badcols; F.nbad = nbad;
    F.isignA = A.conj ? -1.0 : 1.0; F.isignB = B.conj ? -1.0 : 1.0;
    F.ar = realpha; F.ai = cplx ? ai : 0.0; F.br = P.br; F.bi = 0.0;
    F.refused = refused;
    const unsigned fgrid = (unsigned)(2 * num_sms());
    if (dtk == kR8) nonfinite_fixup_kernel<double, false><<<fgrid, 256, 0, s>>>(F);
    else if (dtk == kC8) nonfinite_fixup_kernel<double, true><<<fgrid, 256, 0, s>>>(F);
    else if (dtk == kR4) nonfinite_fixup_kernel<float, false><<<fgrid, 256, 0, s>>>(F);
    else nonfinite_fixup_kernel<float, true><<<fgrid, 256, 0, s>>>(F);
    count_launch();
    if (cudaError_t e = cudaGetLastError()) {
      set_error("non-finite fix-up launch: %s", cudaGetErrorString(e));
      err = TB_ERR_CUDA;
      break;
    }
    if (otherwise && (err = run_direct(*otherwise, dtk, realpha, cplx ? ai : 0.0, accumulate, lconj, rconj, s, refused))) break;
    if (stats) {
      stats->slices = S;
      stats->passes = (int)passes.size();
      stats->products = nplane_products;
      stats->tile_n = BN;
      stats->tile_m = TM;
      stats->gemm_launches = 1;
      stats->m = M; stats->n = Nr; stats->k = Kr;
      stats->moduli = resid ? RP.rs.n : 0;
      stats->residue_bits = resid ? RP.p : 0;
    }
  } while (false);
  scratch_free(ws, s);
  return err;
}

}  // namespace tb
