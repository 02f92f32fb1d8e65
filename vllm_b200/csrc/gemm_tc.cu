// Host side of the tensor-core GEMM (gemm_tc.cuh): tensor maps, tile plan, dispatch by format.
#include "gemm_tc.cuh"

#include <mutex>
#include <unordered_map>

namespace b200q {
namespace tc {

__device__ int g_tc_error;

// Arrival counters of shared tiles, zero between kernels.  One row per stream (calls on one stream are
// ordered, calls on different streams may overlap); a process with more streams than rows runs its
// further streams without shared tiles.
constexpr int kCounterRows = 1024, kCounterLen = 256;
__device__ int32_t g_tc_counters[kCounterRows][kCounterLen];

// one definition per (type, format), in the gemm_tc_inst.cu units
template <typename T, int F>
int launch_format(const TcMaps& maps, const TcParams& p, int cg, bool pdl, cudaStream_t stream);

static int format_bits(int fmt) { return (fmt == kU8B128 || fmt == kU8Z || fmt == kF8 || fmt == kU8ZF) ? 8 : 4; }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// Device addresses of the error word and of the stream's counters (null when there are no rows left).
static int device_words(cudaStream_t stream, int** error, int32_t** counters) {
  static std::mutex mu;
  static struct { int* error; int32_t* counters; std::unordered_map<cudaStream_t, int> rows; } per_device[64];
  int dev = 0;
  B200Q_CUDA_OK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  auto& d = per_device[dev & 63];
  if (!d.error) {
    void *e = nullptr, *c = nullptr;
    B200Q_CUDA_OK(cudaGetSymbolAddress(&c, g_tc_counters));
    B200Q_CUDA_OK(cudaGetSymbolAddress(&e, g_tc_error));
    d.counters = static_cast<int32_t*>(c);
    d.error = static_cast<int*>(e);
  }
  *error = d.error;
  auto it = d.rows.find(stream);
  if (it == d.rows.end() && (int)d.rows.size() < kCounterRows) it = d.rows.emplace(stream, (int)d.rows.size()).first;
  *counters = it == d.rows.end() ? nullptr : d.counters + (size_t)it->second * kCounterLen;
  return B200Q_OK;
}

// A plain 2-D map: `rows` rows of `cols` elements, box of box_rows x box_cols.
static int make_map(CUtensorMap* map, const void* base, CUtensorMapDataType type, int elem_bytes, int64_t cols,
                    int64_t rows, int box_cols, int box_rows) {
  const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t gstride[1] = {(cuuint64_t)cols * elem_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estride[2] = {1, 1};
  const CUresult r = get_encode_fn()(map, type, 2, const_cast<void*>(base), gdim, gstride, box, estride,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200Q_REQUIRE(r == CUDA_SUCCESS, B200Q_ECUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
  return B200Q_OK;
}

// Scale rows that eight consecutive k-tiles, starting at a multiple of eight, can touch.
static int rows_per_round(int gb) {
  return gb % 8 == 0 ? 1 : 8 % gb == 0 ? 8 / gb : (kRoundTiles + gb - 2) / gb + 1;
}

// Maps of one layer's weights (of all experts: `experts` matrices one below the other).
static int make_weight_maps(TcMaps* m, TcParams* p, const void* b, const void* scales, const void* zeros, int fmt,
                            int64_t n, int64_t k, int64_t experts) {
  const int bits = format_bits(fmt);
  // packed weights as rows of k-tiles of 8-byte elements; box = a round x 128 columns
  int rc = make_map(&m->b, b, CU_TENSOR_MAP_DATA_TYPE_UINT64, 8, n * bits / 4, experts * (k / 16), 32 * bits, kRoundTiles);
  if (rc != B200Q_OK) return rc;
  p->groups = (int)(k / 16 / p->group_blocks);
  p->group_rows = rows_per_round(p->group_blocks);
  if (fmt == kNV4 || fmt == kMX4) {
    // bytes: a pair of groups is a row of 2 N; elements of 8 bytes
    rc = make_map(&m->s, scales, CU_TENSOR_MAP_DATA_TYPE_UINT64, 8, n / 4, p->groups / 2, 32, fmt == kNV4 ? 4 : 2);
  } else if (!p->channelwise) {
    rc = make_map(&m->s, scales, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, n, experts * p->groups, 128, p->group_rows);
  }
  if (rc != B200Q_OK) return rc;
  if (fmt == kU4Z || fmt == kU8Z)
    rc = make_map(&m->z, zeros, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, n * bits / 32, experts * p->groups, 4 * bits, p->group_rows);
  else if (fmt == kU4ZF || fmt == kU8ZF)
    rc = make_map(&m->z, zeros, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, n, experts * p->groups, 128, p->group_rows);
  return rc;
}

// Rows of A, 64 columns x `box_rows` rows, 128-byte swizzle.
static int make_a_map(CUtensorMap* map, const void* a, int64_t lda, int64_t m, int64_t k, int box_rows, int a_dtype) {
  const cuuint64_t gdim[2] = {(cuuint64_t)k, (cuuint64_t)m};
  const cuuint64_t gstride[1] = {(cuuint64_t)lda * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t estride[2] = {1, 1};
  const CUresult r = get_encode_fn()(
      map, a_dtype == B200Q_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
      const_cast<void*>(a), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200Q_REQUIRE(r == CUDA_SUCCESS, B200Q_ECUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
  return B200Q_OK;
}

// Sums of tiles that are all shared: one thread per token and four columns, contributors in k order.
template <typename T>
__global__ void __launch_bounds__(256) tc_reduce_kernel(const TcParams p, int cg) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int n4 = p.n / 4;
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
  if (idx >= (long long)p.m * n4) return;
  const int tok = (int)(idx / n4), n = (int)(idx - (long long)tok * n4) * 4;
  const int rounds = (p.k / kBK + 1) / 2;
  const long long units = (long long)p.sk_tiles * rounds;
  const int cols = cg * kBN, tok_tile = tok / p.tn;
  const long long unit0 = ((long long)(n / cols) * p.tok_tiles + tok_tile) * rounds;
  const int first = share_of(unit0, p.workers, units);
  const int count = share_of(unit0 + rounds - 1, p.workers, units) - first + 1;
  const float* src = p.partials + ((size_t)((n / kBN) % cg) * p.tn + (tok - tok_tile * p.tn)) * kBN + n % kBN;
  const size_t slot_floats = (size_t)cg * p.tn * kBN;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  for (int i0 = 0; i0 < count; i0 += 4) {
    float4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i0 + i < count)
        // the first contributor's piece begins the tile (slot 1 of its worker)
        x[i] = __ldcg(reinterpret_cast<const float4*>(src + (2 * (first + i0 + i) + (i0 + i == 0 ? 1 : 0)) * slot_floats));
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i0 + i < count) { v[0] += x[i].x; v[1] += x[i].y; v[2] += x[i].z; v[3] += x[i].w; }
  }
  uint16_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float cs = 1.f;
    if (p.channelwise) cs = Pair<T>::to_float(static_cast<const uint16_t*>(p.scales)[single_perm_pos(n + e)]) * p.chan_factor;
    if (p.global_scale) cs = Pair<T>::to_float(*static_cast<const uint16_t*>(p.global_scale));
    const float bs = p.bias ? Pair<T>::to_float(static_cast<const uint16_t*>(p.bias)[single_perm_pos(n + e)]) : 0.f;
    o[e] = Pair<T>::from_float(v[e] * cs + bs);
  }
  *reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.c) + (size_t)tok * p.n + n) =
      make_uint2((uint32_t)o[0] | ((uint32_t)o[1] << 16), (uint32_t)o[2] | ((uint32_t)o[3] << 16));
}

template <typename T>
static int launch_reduce(const TcParams& p, int cg, cudaStream_t stream) {
  const long long threads = (long long)p.m * (p.n / 4);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((threads + 255) / 256));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  B200Q_CUDA_OK(cudaLaunchKernelEx(&cfg, tc_reduce_kernel<T>, p, cg));
  note_launch();
  return B200Q_OK;
}

struct TcPlan {
  int cg, tn, box, tok_tiles, workers, sk_tiles, reduce_later;
  int64_t partial_bytes;
};

// Tile and work split by estimated time (microseconds; the constants are measured on B200).  Candidates:
// single CTAs with token tiles of up to 128 rows, CTA pairs with up to 256; whole tiles only, the ragged
// last wave shared by k-range, or, with fewer tiles than workers, all tiles shared and added up by the
// reduce kernel.
static TcPlan plan_tiles(int64_t m, int64_t n, int64_t k, int sms, int64_t scratch_bytes) {
  const int64_t rounds = (k / kBK + 1) / 2;
  TcPlan best = {};
  double best_cost = 1e300;
  for (int cg = 1; cg <= 2; ++cg) {
    if (cg == 2 && m <= 128) break;
    const int64_t most = 128 * cg, grain = 16 * cg;
    TcPlan pl = {};
    pl.cg = cg;
    const int64_t want = (m + most - 1) / most;
    pl.tn = (int)(((m + want - 1) / want + grain - 1) / grain * grain);
    pl.tok_tiles = (int)((m + pl.tn - 1) / pl.tn);
    pl.box = pl.tn / cg;
    const int64_t cols = kBN * cg, most_workers = sms / cg;
    const int64_t tiles = (n + cols - 1) / cols * pl.tok_tiles;
    // a round: bound by the conversion, or by the MMAs of a full pair tile
    const double round = cg == 2 ? 0.47 + 0.13 * pl.tn / 256 : 0.47 + 0.08 * pl.tn / 128;
    const int64_t slot_bytes = (int64_t)cg * pl.tn * kBN * 4;
    // whole tiles
    {
      pl.workers = (int)(tiles < most_workers ? tiles : most_workers);
      const double cost = (double)((tiles + most_workers - 1) / most_workers * rounds) * round;
      if (cost < best_cost) { best_cost = cost; best = pl; }
    }
    const int64_t rem = tiles % most_workers;
    if (rem == 0 || most_workers * cg > kCounterLen) continue;
    if (tiles > most_workers) {
      // the ragged wave together with one whole wave, so that no worker's share is a sliver; the additions
      // hide behind a further whole wave where there is one
      pl.workers = (int)most_workers;
      pl.sk_tiles = (int)(rem + most_workers);
      pl.partial_bytes = 2 * most_workers * slot_bytes;
      const double cost = (double)(tiles * rounds) / (double)most_workers * round +
                          (tiles >= 2 * most_workers ? 1.5 : 2.0 + 8.0 * pl.tn / (128 * cg));
      if (pl.partial_bytes <= scratch_bytes && cost < best_cost) { best_cost = cost; best = pl; }
    } else {
      // at least two rounds for every worker
      int64_t workers = tiles * rounds / 2;
      if (workers > most_workers) workers = most_workers;
      if (workers <= tiles) continue;
      pl.workers = (int)workers;
      pl.sk_tiles = (int)tiles;
      pl.reduce_later = 1;
      pl.partial_bytes = 2 * workers * slot_bytes;
      const double cost = (double)((tiles * rounds + workers - 1) / workers) * round + 2.5 +
                          2.0 * (double)((workers + tiles) * slot_bytes) / 4e6;
      if (pl.partial_bytes <= scratch_bytes && cost < best_cost) { best_cost = cost; best = pl; }
    }
  }
  return best;
}

template <typename T>
static int launch_type(const TcMaps& maps, const TcParams& p, int fmt, int cg, bool pdl, cudaStream_t stream) {
  switch (fmt) {
    case kU4B8: return launch_format<T, kU4B8>(maps, p, cg, pdl, stream);
    case kU4Z: return launch_format<T, kU4Z>(maps, p, cg, pdl, stream);
    case kU8B128: return launch_format<T, kU8B128>(maps, p, cg, pdl, stream);
    case kU8Z: return launch_format<T, kU8Z>(maps, p, cg, pdl, stream);
    case kF8: return launch_format<T, kF8>(maps, p, cg, pdl, stream);
    case kNV4: return launch_format<T, kNV4>(maps, p, cg, pdl, stream);
  }
  if constexpr (std::is_same<T, half>::value) {
    if (fmt == kU4ZF) return launch_format<T, kU4ZF>(maps, p, cg, pdl, stream);
    if (fmt == kU8ZF) return launch_format<T, kU8ZF>(maps, p, cg, pdl, stream);
  } else {
    if (fmt == kMX4) return launch_format<T, kMX4>(maps, p, cg, pdl, stream);
  }
  set_error("weight format %d is not available for this activation type", fmt);
  return B200Q_EUNSUPPORTED;
}

}  // namespace tc

// True when the tensor-core kernel can take this problem.
bool tc_gemm_supported(int64_t size_n, int64_t size_k, int gm) {
  return size_k % tc::kBK == 0 && size_n % 64 == 0 && gm != kLookup && tc::get_encode_fn() != nullptr;
}

// a: [M, K] 16-bit row-major with row stride lda (already gathered for act-order).
int launch_tc_gemm(const void* a, int64_t lda, const uint32_t* b, const void* scales, const uint32_t* zeros,
                   const void* bias, const void* global_scale, void* c, int a_dtype, int fmt, int64_t size_m,
                   int64_t size_n, int64_t size_k, int group_blocks, int channelwise, void* scratch,
                   int64_t scratch_bytes, cudaStream_t stream) {
  tc::TcParams p = {};
  int rc = tc::device_words(stream, &p.error, &p.counters);
  if (rc != B200Q_OK) return rc;
  const tc::TcPlan plan = tc::plan_tiles(size_m, size_n, size_k, device_sm_count(), p.counters ? scratch_bytes : 0);
  tc::TcMaps maps = {};
  p.group_blocks = group_blocks; p.channelwise = channelwise;
  rc = tc::make_a_map(&maps.a, a, lda, size_m, size_k, plan.box, a_dtype);
  if (rc == B200Q_OK) rc = tc::make_weight_maps(&maps, &p, b, scales, zeros, fmt, size_n, size_k, 1);
  if (rc != B200Q_OK) return rc;
  p.scales = scales; p.bias = bias; p.global_scale = global_scale; p.c = c;
  p.m = (int)size_m; p.n = (int)size_n; p.k = (int)size_k;
  p.tn = plan.tn; p.box = plan.box; p.tok_tiles = plan.tok_tiles; p.workers = plan.workers;
  p.sk_tiles = plan.sk_tiles; p.reduce_later = plan.reduce_later;
  p.chan_factor = fmt != tc::kF8 ? 1.f : a_dtype == B200Q_F16 ? Fp8Cvt<half>::kRebiasInv : Fp8Cvt<__nv_bfloat16>::kRebiasInv;
  p.partials = static_cast<float*>(scratch);
  // early launch only where this kernel's fixed costs matter: with many rows the waiting CTAs would take
  // the SMs from an act-order gather still running in front
  const bool pdl = pdl_enabled() && size_m <= 128;
  rc = a_dtype == B200Q_F16 ? tc::launch_type<half>(maps, p, fmt, plan.cg, pdl, stream)
                            : tc::launch_type<__nv_bfloat16>(maps, p, fmt, plan.cg, pdl, stream);
  if (rc != B200Q_OK || !plan.reduce_later) return rc;
  return a_dtype == B200Q_F16 ? tc::launch_reduce<half>(p, plan.cg, stream)
                              : tc::launch_reduce<__nv_bfloat16>(p, plan.cg, stream);
}

// Scratch the tensor-core kernel would like for this problem (fp32 partials of shared tiles).
int64_t tc_gemm_scratch_bytes(int64_t size_m, int64_t size_n, int64_t size_k) {
  if (size_k % tc::kBK != 0 || size_n % 64 != 0) return 0;
  return tc::plan_tiles(size_m, size_n, size_k, device_sm_count(), int64_t(1) << 40).partial_bytes;
}

int tc_error_flag(bool reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, tc::g_tc_error, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v != 0) {
    int zero = 0;
    cudaMemcpyToSymbol(tc::g_tc_error, &zero, sizeof(int));
    // a kernel that gave up may have left arrivals behind
    void* c = nullptr;
    if (cudaGetSymbolAddress(&c, tc::g_tc_counters) == cudaSuccess) cudaMemset(c, 0, sizeof(tc::g_tc_counters));
  }
  return v;
}

}  // namespace b200q
