// tb_direct.cu -- launches of the one-kernel contraction (tb_direct.cuh).
#include "tb_direct.h"
#include "tb_direct.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "tb_contract.h"
#include "tb_pattern.h"

namespace tb {
namespace {

using namespace direct;

template <typename E, int WM, int WN, int KW, int MI, int NI, int BK, int ST, int OCC>
struct Variant {
  using S = Shape<E, WM, WN, KW, MI, NI, BK, ST>;
  static TileShape shape() { return {S::BM, S::BN, S::BKT, S::T, OCC}; }
  static int launch(const Params& P, int64_t ctas, cudaStream_t s, const unsigned* when) {
    if constexpr (!Elem<E>::F32) {  // conditional launches: FP64 data only
      if (when) return launch_as(P, ctas, s, when);
    }
    return launch_as(P, ctas, s);
  }
  template <class... Word>
  static int launch_as(const Params& P, int64_t ctas, cudaStream_t s, Word... when) {
    static DeviceOnce attr;
    auto kern = direct_kernel<E, WM, WN, KW, MI, NI, BK, ST, OCC, Word...>;
    const size_t smem = S::smem(P.split > 1 || KW > 1);
    cudaError_t e = smem_limit_once(attr, kern, (int)S::smem(true));
    if (e != cudaSuccess) { set_error("direct contraction smem attribute: %s", cudaGetErrorString(e)); return TB_ERR_CUDA; }
    if (P.split == 1) {
      kern<<<(unsigned)ctas, S::T, smem, s>>>(P, when...);
    } else {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)ctas, 1, 1);
      cfg.blockDim = dim3(S::T, 1, 1);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = s;
      cudaLaunchAttribute a;
      a.id = cudaLaunchAttributeClusterDimension;
      a.val.clusterDim.x = (unsigned)P.split;
      a.val.clusterDim.y = a.val.clusterDim.z = 1;
      cfg.attrs = &a;
      cfg.numAttrs = 1;
      e = cudaLaunchKernelEx(&cfg, kern, P, when...);
      if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("direct contraction cluster launch: %s", cudaGetErrorString(e));
        return TB_ERR_CUDA;
      }
    }
    TB_CHECK_LAUNCH();
    return 0;
  }
};

struct VariantRef {
  TileShape sh;
  int (*launch)(const Params&, int64_t, cudaStream_t, const unsigned*);
};
template <class V>
VariantRef ref() { return {V::shape(), &V::launch}; }

// Real kinds: 32 x 32 warp tiles (16 accumulators per fragment load of 8).
// Small products use one 32 x 32 tile whose four warps share each K tile;
// narrow sides have 16- and 32-wide shapes so that padding is not multiplied.
template <typename E>
const std::vector<VariantRef>& variants_real() {
  static const std::vector<VariantRef> v = {
      ref<Variant<E, 1, 1, 4, 4, 4, 8, 3, 3>>(),  ref<Variant<E, 2, 2, 1, 4, 4, 16, 3, 3>>(),
      ref<Variant<E, 4, 1, 1, 4, 4, 16, 2, 3>>(), ref<Variant<E, 1, 4, 1, 4, 4, 16, 2, 3>>(),
      ref<Variant<E, 4, 2, 1, 4, 4, 16, 3, 2>>(), ref<Variant<E, 4, 1, 1, 4, 2, 16, 3, 3>>(),
      ref<Variant<E, 1, 4, 1, 2, 4, 16, 3, 3>>(),
  };
  return v;
}
// Complex kinds: four real products per element, 32 x 16 warp tiles.
template <typename E>
const std::vector<VariantRef>& variants_cplx() {
  static const std::vector<VariantRef> v = {
      ref<Variant<E, 1, 2, 2, 4, 2, 8, 3, 3>>(), ref<Variant<E, 2, 2, 1, 4, 2, 8, 3, 3>>(),
      ref<Variant<E, 4, 1, 1, 4, 2, 8, 3, 3>>(), ref<Variant<E, 1, 4, 1, 2, 4, 8, 3, 3>>(),
      ref<Variant<E, 2, 4, 1, 4, 2, 8, 3, 1>>(), ref<Variant<E, 4, 2, 1, 4, 2, 8, 3, 1>>(),
  };
  return v;
}
const std::vector<VariantRef>& variants(int dtk) {
  switch (dtk) {
    case kR4: return variants_real<float>();
    case kR8: return variants_real<double>();
    case kC4: return variants_cplx<float2>();
    default: return variants_cplx<double2>();
  }
}

// The tile shapes of a data kind, for the planner.
const std::vector<TileShape>& shapes(int dtk) {
  auto of = [](const std::vector<VariantRef>& v) {
    std::vector<TileShape> s;
    for (auto& x : v) s.push_back(x.sh);
    return s;
  };
  static const std::vector<TileShape> real = of(variants(kR8)), cplx = of(variants(kC8));
  return is_complex(dtk) ? cplx : real;
}

}  // namespace

int direct_plan(const Matricization& Z, int dtk, const void* d, const void* l, const void* r, DirectPlan* out) {
  return plan_direct(Z, elem_bytes(dtk), is_complex(dtk), d, l, r, shapes(dtk), num_sms(), out);
}

int run_direct(const DirectPlan& plan, int dtk, double ar, double ai, bool accumulate, int lconj, int rconj,
               cudaStream_t s, const unsigned* when) {
  Params P = plan.P;
  P.ar = ar;
  P.ai = ai;
  P.br = accumulate ? 1.0 : 0.0;
  P.bi = 0.0;
  P.aconj = plan.swap ? rconj : lconj;
  P.bconj = plan.swap ? lconj : rconj;
  const int ts = timed_begin(s);
  const int e = variants(dtk)[plan.variant].launch(P, plan.ctas, s, when);
  timed_end(ts, s);
  return e;
}

}  // namespace tb
