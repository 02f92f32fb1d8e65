// Host side of the tensor-core GEMM (gemm_tc.cuh): tensor maps, tile plan, dispatch by format.
#include "gemm_tc.cuh"

namespace b200q {
namespace tc {

__device__ int g_tc_error;

// one definition per (type, format), in the gemm_tc_inst.cu units
template <typename T, int F>
int launch_format(const TcMaps& maps, const TcParams& p, int cg, bool sums, bool pdl, cudaStream_t stream);

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

static int error_word(int** out) {
  static int* addr[64] = {};  // per device; benign race: the same value every time
  int dev = 0;
  B200Q_CUDA_OK(cudaGetDevice(&dev));
  if (!addr[dev & 63]) {
    void* a = nullptr;
    B200Q_CUDA_OK(cudaGetSymbolAddress(&a, g_tc_error));
    addr[dev & 63] = static_cast<int*>(a);
  }
  *out = addr[dev & 63];
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
  // packed weights: k-tiles of pieces of 128 bytes; box = a round x 128 columns, swizzled piece by piece
  const cuuint64_t gdim[3] = {16, (cuuint64_t)(n * bits / 64), (cuuint64_t)(experts * (k / 16))};
  const cuuint64_t gstride[2] = {128, (cuuint64_t)(n * 2 * bits)};
  const cuuint32_t box[3] = {16, (cuuint32_t)(2 * bits), (cuuint32_t)kRoundTiles};
  const cuuint32_t estride[3] = {1, 1, 1};
  const CUresult r = get_encode_fn()(&m->b, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<uint32_t*>(static_cast<const uint32_t*>(b)),
                                     gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200Q_REQUIRE(r == CUDA_SUCCESS, B200Q_ECUDA, "cuTensorMapEncodeTiled failed with %d", (int)r);
  int rc = B200Q_OK;
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

// Sums of the shared tiles: blockIdx.y = tile, one thread per token and four columns, contributors in k
// order.
template <typename T>
__global__ void __launch_bounds__(256) tc_reduce_kernel(const TcParams p, int cg) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int cols4 = cg * kBN / 4;
  const int idx = blockIdx.x * 256 + threadIdx.x, tile = blockIdx.y;
  const int tt = idx / cols4, col = (idx - tt * cols4) * 4;  // inside the tile
  const int n_tile = tile / p.tok_tiles;
  const int tok = (tile - n_tile * p.tok_tiles) * p.tn + tt;
  const int n = n_tile * cg * kBN + col;
  if (tt >= p.tn || tok >= p.m || n >= p.n) return;
  const int rounds = (p.k / kBK + 1) / 2;
  const long long units = (long long)p.sk_tiles * rounds, unit0 = (long long)tile * rounds;
  const int first = share_of(unit0, p.workers, units);
  const int count = share_of(unit0 + rounds - 1, p.workers, units) - first + 1;
  const float* src = p.partials + ((size_t)(col / kBN) * p.tn + tt) * kBN + col % kBN;
  const size_t slot_floats = (size_t)cg * p.tn * kBN;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  for (int i0 = 0; i0 < count; i0 += 4) {
    float4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i0 + i < count)
        // a piece that begins the tile is in slot 1 of its worker, any other in slot 0
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
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.tn * cg * kBN / 4 + 255) / 256), (unsigned)p.sk_tiles);
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
  int cg, tn, box, tok_tiles, workers, sk_tiles;
  int64_t partial_bytes;
  double us;         // estimate that the plans are compared by
  double rounds_us;  // the part of it that is rounds
  int rounds;        // of the busiest worker
};

// Microseconds of a round (128 deep in k) of one tile: the table that plans are compared by, measured on B200 for 4-bit
// weights while all operands went through shared memory.  It is too high for the kernel as it is, and not by one factor.
// Table / now, 4-bit at 1965 MHz: single CTAs of 48 tokens 0.45 / 0.36, of 128 0.58 / 0.35, pairs of 160 0.57 / 0.40, of 192
// 0.64 / 0.43, of 256 0.78 / 0.52; 8-bit per column 160 0.36, 8-bit groups of 128 256 0.73.  So whole waves look longer
// against shared ones than they are (fp8 24 x 4096 x 28672: 28.8 against 28.4 by the table, 21.6 against 22.8 by the time of
// a round now), wide single CTAs longer against pairs, and 8 bits are planned as if they were 4.
static double round_us(int cg, int tn) {
  if (cg == 1) return tn <= 64 ? 0.45 : 0.46 + 0.00096 * tn;
  const double t = 0.22 + 0.00217 * tn;
  return t < 0.5 ? 0.5 : t;
}

// Tile and work split by estimated time.  Candidates: single CTAs with token tiles of up to 128 rows, CTA
// pairs with up to 256, a few tile widths each; whole tiles only, or the ragged last wave shared by
// k-range (its partial sums are written and read once, and cost a launch).
static TcPlan plan_tiles(int64_t m, int64_t n, int64_t k, int sms, int64_t scratch_bytes) {
  const int64_t rounds = (k / kBK + 1) / 2;
  TcPlan best = {};
  best.us = 1e300;
  for (int cg = 1; cg <= 2; ++cg) {
    if (cg == 2 && m <= 64) break;
    const int64_t most = 128 * cg, grain = 16 * cg;
    const int64_t want = (m + most - 1) / most;
    int last_tn = 0;
    for (int64_t more = 0; more < 4; ++more) {
      TcPlan pl = {};
      pl.cg = cg;
      pl.tn = (int)(((m + want + more - 1) / (want + more) + grain - 1) / grain * grain);
      if (pl.tn == last_tn) continue;
      last_tn = pl.tn;
      pl.tok_tiles = (int)((m + pl.tn - 1) / pl.tn);
      pl.box = pl.tn / cg;
      const int64_t cols = kBN * cg, most_workers = sms / cg;
      const int64_t tiles = (n + cols - 1) / cols * pl.tok_tiles;
      const double round = round_us(cg, pl.tn);
      const int64_t waves = tiles / most_workers, rem = tiles % most_workers;
      pl.workers = (int)(tiles < most_workers ? tiles : most_workers);
      pl.rounds = (int)((waves + (rem > 0)) * rounds);
      const double cost = pl.rounds * round;
      pl.us = pl.rounds_us = cost;
      if (cost < best.us) best = pl;
      if (rem == 0) continue;
      // at least two rounds for every worker
      const int64_t by_work = rem * rounds / 2;
      int64_t workers = by_work < most_workers ? by_work : most_workers;
      if (waves > 0) workers = most_workers;
      if (workers <= rem || rem * rounds < workers) continue;  // every worker has a round: the sums are taken over all
      pl.workers = (int)workers;
      pl.sk_tiles = (int)rem;
      const int64_t slot_bytes = (int64_t)cg * pl.tn * kBN * 4;
      pl.partial_bytes = 2 * workers * slot_bytes;
      pl.rounds = (int)(waves * rounds + (rem * rounds + workers - 1) / workers);
      pl.rounds_us = pl.rounds * round;
      // (fixed costs for the choice between plans; tc_gemm_estimate_us has its own, fitted to whole calls.  The
      // two put sharing up to 1.5 us apart, and fp8 at 24 x 4096 x 28672 is shared by a margin of 0.4 us.)
      // a second segment behind whole tiles: its own pipeline fill and drain (1152 x 19392, 152 tiles of nine
      // rounds: 15.2 us with the last four shared, 11.0 in two waves)
      pl.us = pl.rounds_us + 2.5 + (waves > 0 ? 2.0 : 0.0) + 2.0 * (double)((workers + rem) * slot_bytes) / 4e6;
      if (pl.partial_bytes <= scratch_bytes && pl.us < best.us) best = pl;
    }
  }
  return best;
}

template <typename T>
static int launch_type(const TcMaps& maps, const TcParams& p, int fmt, int cg, bool sums, bool pdl, cudaStream_t stream) {
  switch (fmt) {
    case kU4B8: return launch_format<T, kU4B8>(maps, p, cg, sums, pdl, stream);
    case kU4Z: return launch_format<T, kU4Z>(maps, p, cg, sums, pdl, stream);
    case kU8B128: return launch_format<T, kU8B128>(maps, p, cg, sums, pdl, stream);
    case kU8Z: return launch_format<T, kU8Z>(maps, p, cg, sums, pdl, stream);
    case kF8: return launch_format<T, kF8>(maps, p, cg, sums, pdl, stream);
    case kNV4: return launch_format<T, kNV4>(maps, p, cg, sums, pdl, stream);
  }
  if constexpr (std::is_same<T, half>::value) {
    if (fmt == kU4ZF) return launch_format<T, kU4ZF>(maps, p, cg, sums, pdl, stream);
    if (fmt == kU8ZF) return launch_format<T, kU8ZF>(maps, p, cg, sums, pdl, stream);
  } else {
    if (fmt == kMX4) return launch_format<T, kMX4>(maps, p, cg, sums, pdl, stream);
  }
  set_error("weight format %d is not available for this activation type", fmt);
  return B200Q_EUNSUPPORTED;
}

}  // namespace tc

// True when the tensor-core kernel can take this problem.
bool tc_gemm_supported(int64_t size_n, int64_t size_k, int gm) {
  return size_k % tc::kBK == 0 && size_n % 64 == 0 && gm != kLookup && tc::get_encode_fn() != nullptr;
}

// True when the tensor-core kernel can apply these group scales to fp32 sums: groups of a step or of whole rounds.
bool tc_group_sums_supported(int64_t group_size) { return group_size == tc::kBK || (group_size > 0 && group_size % (2 * tc::kBK) == 0); }
// rows of a tile at most in that form (cg = 1: single CTAs, 2: pairs)
int tc_group_sums_rows(int cg) { return tc::group_sums_tokens(cg); }

// a: [M, K] 16-bit row-major with row stride lda (already gathered for act-order: `gathered`).  sums: group scales on the fp32
// sums (up to 64 rows).
int launch_tc_gemm(const void* a, int64_t lda, const uint32_t* b, const void* scales, const uint32_t* zeros,
                   const void* bias, const void* global_scale, void* c, int a_dtype, int fmt, int64_t size_m,
                   int64_t size_n, int64_t size_k, int group_blocks, int channelwise, bool sums, bool gathered, void* scratch,
                   int64_t scratch_bytes, cudaStream_t stream) {
  tc::TcParams p = {};
  int rc = tc::error_word(&p.error);
  if (rc != B200Q_OK) return rc;
  const tc::TcPlan plan = tc::plan_tiles(size_m, size_n, size_k, device_sm_count(), scratch_bytes);
  tc::TcMaps maps = {};
  p.group_blocks = group_blocks; p.channelwise = channelwise;
  rc = tc::make_a_map(&maps.a, a, lda, size_m, size_k, plan.box, a_dtype);
  if (rc == B200Q_OK) rc = tc::make_weight_maps(&maps, &p, b, scales, zeros, fmt, size_n, size_k, 1);
  if (rc != B200Q_OK) return rc;
  p.scales = scales; p.bias = bias; p.global_scale = global_scale; p.c = c;
  p.m = (int)size_m; p.n = (int)size_n; p.k = (int)size_k;
  p.tn = plan.tn; p.box = plan.box; p.tok_tiles = plan.tok_tiles; p.workers = plan.workers;
  p.sk_tiles = plan.sk_tiles;
  p.chan_factor = fmt != tc::kF8 ? 1.f : a_dtype == B200Q_F16 ? Fp8Cvt<half>::kRebiasInv : Fp8Cvt<__nv_bfloat16>::kRebiasInv;
  p.partials = static_cast<float*>(scratch);
  // early launch, but not of many rows behind their act-order gather: the waiting CTAs would take the SMs from it
  const bool pdl = pdl_enabled() && (size_m <= tc::kAheadRows || !gathered);
  rc = a_dtype == B200Q_F16 ? tc::launch_type<half>(maps, p, fmt, plan.cg, sums, pdl, stream)
                            : tc::launch_type<__nv_bfloat16>(maps, p, fmt, plan.cg, sums, pdl, stream);
  if (rc != B200Q_OK || plan.sk_tiles == 0) return rc;
  return a_dtype == B200Q_F16 ? tc::launch_reduce<half>(p, plan.cg, stream)
                              : tc::launch_reduce<__nv_bfloat16>(p, plan.cg, stream);
}

// Mixture of experts: rows of A in sorted order, tiles {expert, first row, rows} in device memory, written by
// a kernel in front.  `box`: token rows a CTA stages; a tile has at most that many rows (pairs: twice).  Group scales
// go on the fp32 sums, as in the decode kernel that the same layer runs at fewer rows.
int launch_tc_moe(const void* a, int64_t rows, const uint32_t* b, const void* scales, const uint32_t* zeros,
                  const void* bias, void* c, int a_dtype, int fmt, int64_t experts, int64_t size_n, int64_t size_k,
                  int64_t num_groups, int pairs, int box, const int4* tile_list, const int32_t* tile_count,
                  const int32_t* ids, int scatter, const float* row_weights, cudaStream_t stream) {
  tc::TcParams p = {};
  int rc = tc::error_word(&p.error);
  if (rc != B200Q_OK) return rc;
  B200Q_REQUIRE(size_k % num_groups == 0 && (size_k / num_groups) % 16 == 0, B200Q_EINVAL,
                "size_k = %lld does not split into %lld groups", (long long)size_k, (long long)num_groups);
  tc::TcMaps maps = {};
  p.group_blocks = (int)(size_k / num_groups / 16); p.channelwise = num_groups == 1;
  rc = tc::make_a_map(&maps.a, a, size_k, rows, size_k, box, a_dtype);
  if (rc == B200Q_OK) rc = tc::make_weight_maps(&maps, &p, b, scales, zeros, fmt, size_n, size_k, experts);
  if (rc != B200Q_OK) return rc;
  const int cg = pairs ? 2 : 1;
  p.scales = scales; p.bias = bias; p.c = c; p.chan_factor = 1.f;
  p.m = (int)rows; p.n = (int)size_n; p.k = (int)size_k;
  p.tn = box * cg; p.box = box; p.tok_tiles = 1; p.workers = device_sm_count() / cg;
  p.tile_list = tile_list; p.tile_count = tile_count;
  p.ids = row_weights || scatter ? ids : nullptr; p.scatter = scatter; p.row_weights = row_weights; p.out_rows = (int)rows;
  p.s_stride = num_groups * size_n; p.bias_stride = size_n;
  const bool pdl = pdl_enabled(), sums = !p.channelwise;
  return a_dtype == B200Q_F16 ? tc::launch_type<half>(maps, p, fmt, cg, sums, pdl, stream)
                              : tc::launch_type<__nv_bfloat16>(maps, p, fmt, cg, sums, pdl, stream);
}

// Scratch the tensor-core kernel would like for this problem (fp32 partials of shared tiles).
int64_t tc_gemm_scratch_bytes(int64_t size_m, int64_t size_n, int64_t size_k) {
  if (size_k % tc::kBK != 0 || size_n % 64 != 0 || device_sm_count() < 2) return 0;  // (0: no device to plan for)
  return tc::plan_tiles(size_m, size_n, size_k, device_sm_count(), int64_t(1) << 40).partial_bytes;
}

TcSplit tc_gemm_split(int64_t size_m, int64_t size_n, int64_t size_k) {
  const tc::TcPlan pl = tc::plan_tiles(size_m, size_n, size_k, device_sm_count(), int64_t(1) << 40);
  return {pl.rounds, pl.workers, pl.sk_tiles > 0};
}

// Estimated time of the kernel (and its reduce kernel) in us, fitted to whole calls of up to 16 rows; `factor`: time
// of a round against the table.
double tc_gemm_estimate_us(int64_t size_m, int64_t size_n, int64_t size_k, double factor) {
  const tc::TcPlan pl = tc::plan_tiles(size_m, size_n, size_k, device_sm_count(), int64_t(1) << 40);
  const double us = factor * pl.rounds_us;
  if (pl.sk_tiles == 0) return 3.0 + us;
  // the exchange of sums: more of it with more tokens, less where there are only a few rounds to exchange
  const bool behind_whole_tiles = (size_n + tc::kBN * pl.cg - 1) / (tc::kBN * pl.cg) * pl.tok_tiles > pl.sk_tiles;
  return 5.0 + (us < 2.7 ? 0.55 * us : 1.5) + 0.02 * (double)size_m + (behind_whole_tiles ? 1.0 : 0.0) + us;
}

int tc_error_flag(bool reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, tc::g_tc_error, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v != 0) {
    int zero = 0;
    cudaMemcpyToSymbol(tc::g_tc_error, &zero, sizeof(int));
  }
  return v;
}

}  // namespace b200q
