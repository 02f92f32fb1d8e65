// Instantiations of the tensor-core GEMM for one element type and two weight formats, selected at
// compile time (-DINST_BF16={0,1} -DINST_F0=.. -DINST_F1=..) so that the units build in parallel.
#include "gemm_tc.cuh"

#ifndef INST_BF16
#error "compile with -DINST_BF16=0|1 -DINST_F0=<format> -DINST_F1=<format>"
#endif

namespace b200q {
namespace tc {

#if INST_BF16
using InstT = __nv_bfloat16;
#else
using InstT = half;
#endif

template <typename T, int F, int CG, int TOK, bool SUMS = false>
static int launch_one(const TcMaps& maps, const TcParams& p, bool pdl, cudaStream_t stream) {
  using Cfg = TcCfg<F, CG, TOK, SUMS>;
  static_assert(Cfg::kWD >= 2, "weight ring too shallow");
  auto kernel = gemm_tc_kernel<T, F, CG, TOK, SUMS>;
  static bool attr_done[64] = {};  // per device; benign race: the call is idempotent
  int dev = 0;
  B200Q_CUDA_OK(cudaGetDevice(&dev));
  if (!attr_done[dev & 63]) {
    B200Q_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    attr_done[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.workers * CG));
  cfg.blockDim = dim3(Cfg::kThreads);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n_attr = 0;
  if (CG == 2) {
    attr[n_attr].id = cudaLaunchAttributeClusterDimension;
    attr[n_attr].val.clusterDim.x = 2;
    attr[n_attr].val.clusterDim.y = 1;
    attr[n_attr].val.clusterDim.z = 1;
    ++n_attr;
  }
  if (pdl) {
    attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
    ++n_attr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n_attr;
  B200Q_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, maps, p));
  note_launch();
  return B200Q_OK;
}

template <typename T, int F>
int launch_format(const TcMaps& maps, const TcParams& p, int cg, bool sums, bool pdl, cudaStream_t stream);

template <typename T, int F>
static int launch_sums(const TcMaps& maps, const TcParams& p, int cg, bool pdl, cudaStream_t stream) {
  if constexpr (F == kU4B8 || F == kU4Z || F == kU8B128 || F == kU8Z) {
    if (p.tn <= group_sums_tokens(cg))
      return cg == 2 ? launch_one<T, F, 2, 80, true>(maps, p, pdl, stream) : launch_one<T, F, 1, 64, true>(maps, p, pdl, stream);
  }
  set_error("group scales on the sums: weight format %d, %d tokens per tile", F, p.tn);
  return B200Q_EUNSUPPORTED;
}

#define B200Q_TC_FORMAT(F)                                                                                           \
  template <>                                                                                                        \
  int launch_format<InstT, F>(const TcMaps& maps, const TcParams& p, int cg, bool sums, bool pdl, cudaStream_t stream) { \
    if (sums) return launch_sums<InstT, F>(maps, p, cg, pdl, stream);                                                \
    if (cg == 2)                                                                                                     \
      return p.box <= 64   ? launch_one<InstT, F, 2, 64>(maps, p, pdl, stream)                                       \
             : p.box <= 80 ? launch_one<InstT, F, 2, 80>(maps, p, pdl, stream)                                       \
             : p.box <= 96 ? launch_one<InstT, F, 2, 96>(maps, p, pdl, stream)                                       \
                           : launch_one<InstT, F, 2, 128>(maps, p, pdl, stream);                                     \
    return p.box <= 64 ? launch_one<InstT, F, 1, 64>(maps, p, pdl, stream)                                           \
                       : launch_one<InstT, F, 1, 128>(maps, p, pdl, stream);                                         \
  }

B200Q_TC_FORMAT(INST_F0)
#if INST_F1 != INST_F0
B200Q_TC_FORMAT(INST_F1)
#endif

}  // namespace tc
}  // namespace b200q
