// Mixture-of-experts layer: routing (sort of the (token, slot) pairs by expert), row gather, sum over the
// slots, and the sequence of launches of one layer.  The GEMMs are the decode kernel (gemm_stream.cuh,
// blocks of sorted ids) for few rows per expert and the tensor-core kernel (gemm_tc.cuh, tile list) above.
#include "common.cuh"
#include "gemm_params.cuh"

namespace b200q {

int launch_tc_moe(const void* a, int64_t rows, const uint32_t* b, const void* scales, const uint32_t* zeros,
                  const void* bias, void* c, int a_dtype, int fmt, int64_t experts, int64_t size_n, int64_t size_k,
                  int64_t num_groups, int pairs, int box, const int4* tile_list, const int32_t* tile_count,
                  const int32_t* ids, int scatter, const float* row_weights, cudaStream_t stream);
bool tc_gemm_supported(int64_t size_n, int64_t size_k, int gm);
bool tc_group_sums_supported(int64_t group_size);
int tc_group_sums_rows(int cg);

namespace moe {

constexpr int kSortThreads = 1024;
constexpr int kSortWarps = kSortThreads / 32;

struct SortParams {
  const void* topk_ids;       // [numel] int32 or int64
  int ids64;
  const int32_t* expert_map;  // [experts]: local expert, -1 = on another rank; or null
  int numel, experts;
  int block;                  // > 0: runs are padded to a multiple of `block`; 0: not padded, tile list
  int max_rows;               // tile list: rows per tile at most
  int32_t* sorted_ids;        // padding = numel
  int sorted_len;
  int32_t* block_experts;     // padded form: expert of every block
  int blocks;
  int32_t* total;             // rows in use (padded form), tiles (tile list)
  int4* tiles;                // tile list {expert, first row, rows}
};

// One CTA, stable: every warp counts a contiguous share of the ids, prefix sums over (expert, warp) give
// each warp its first position per expert, and the warps place their ids.  The torch formulation of the
// same took some twenty launches (300 us of host time per layer).
__global__ void __launch_bounds__(kSortThreads, 1) moe_sort_kernel(const SortParams p) {
  extern __shared__ int32_t counts[];  // [experts][kSortWarps], then [experts + 1] run starts
  int32_t* starts = counts + p.experts * kSortWarps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  for (int i = threadIdx.x; i < p.experts * kSortWarps; i += kSortThreads) counts[i] = 0;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  __syncthreads();
  const int per = ((p.numel + kSortWarps - 1) / kSortWarps + 31) / 32 * 32;
  const int i0 = warp * per, i1 = min(p.numel, i0 + per);
  // expert of id i, -1 outside the range of this warp (or of the experts)
  auto expert_of = [&](int i) {
    if (i >= i1) return -1;
    const long long e = p.ids64 ? static_cast<const long long*>(p.topk_ids)[i]
                                : (long long)static_cast<const int32_t*>(p.topk_ids)[i];
    return e >= 0 && e < p.experts ? (int)e : -1;
  };
  for (int i = i0; i < i1; i += 32) {
    const int e = expert_of(i + lane);
    const uint32_t peers = __match_any_sync(~0u, e);
    if (e >= 0 && lane == __ffs(peers) - 1) counts[e * kSortWarps + warp] += __popc(peers);
  }
  __syncthreads();
  // per expert: exclusive prefix over the warps; the run length goes to starts[e]
  for (int e = warp; e < p.experts; e += kSortWarps) {
    const int c = counts[e * kSortWarps + lane];
    int incl = c;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int v = __shfl_up_sync(~0u, incl, d);
      if (lane >= d) incl += v;
    }
    counts[e * kSortWarps + lane] = incl - c;
    if (lane == 31) starts[e] = incl;
  }
  __syncthreads();
  // run starts: exclusive prefix over the experts (padded runs), by one warp
  if (warp == 0) {
    int base = 0, tiles = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      const int run = e < p.experts ? starts[e] : 0;
      const int padded = p.block > 0 ? (run + p.block - 1) / p.block * p.block : run;
      int local = e;
      if (p.expert_map && e < p.experts) local = p.expert_map[e];
      // tile list: the run in equal parts of at most max_rows; experts of other ranks have none
      const int parts = p.block > 0 || local < 0 ? 0 : (run + p.max_rows - 1) / p.max_rows;
      int incl = padded, tincl = parts;
#pragma unroll
      for (int d = 1; d < 32; d *= 2) {
        const int v = __shfl_up_sync(~0u, incl, d), t = __shfl_up_sync(~0u, tincl, d);
        if (lane >= d) { incl += v; tincl += t; }
      }
      const int start = base + incl - padded;
      if (e < p.experts) {
        if (p.block > 0) {
          for (int b = start / p.block; b < (start + padded) / p.block; ++b) p.block_experts[b] = local;
        } else {
          for (int j = 0; j < parts; ++j) {
            const int r0 = (int)((long long)run * j / parts), r1 = (int)((long long)run * (j + 1) / parts);
            p.tiles[tiles + tincl - parts + j] = make_int4(local, start + r0, r1 - r0, 0);
          }
        }
      }
      __syncwarp();
      if (e < p.experts) starts[e] = start;
      base += __shfl_sync(~0u, incl, 31);
      tiles += __shfl_sync(~0u, tincl, 31);
    }
    if (lane == 0) {
      starts[p.experts] = base;
      *p.total = p.block > 0 ? base : tiles;
    }
  }
  // padding everywhere first; the ids overwrite their places
  if (p.block > 0)
    for (int i = threadIdx.x; i < p.sorted_len; i += kSortThreads) p.sorted_ids[i] = p.numel;
  __syncthreads();
  const int used = starts[p.experts];
  if (p.block > 0) {
    // blocks past the end belong to expert 0 (mapped), as the block list always has been filled
    const int rest = p.expert_map ? p.expert_map[0] : 0;
    for (int b = used / p.block + threadIdx.x; b < p.blocks; b += kSortThreads) p.block_experts[b] = rest;
  }
  for (int i = i0; i < i1; i += 32) {
    const int e = expert_of(i + lane);
    const uint32_t peers = __match_any_sync(~0u, e);
    if (e >= 0) {
      const int at = starts[e] + counts[e * kSortWarps + warp] + __popc(peers & ((1u << lane) - 1));
      p.sorted_ids[at] = i + lane;
    }
    __syncwarp();
    if (e >= 0 && lane == __ffs(peers) - 1) counts[e * kSortWarps + warp] += __popc(peers);
    __syncwarp();
  }
}

static int launch_sort(const SortParams& p, cudaStream_t stream) {
  const size_t smem = (size_t)(p.experts * kSortWarps + p.experts + 1) * 4;
  B200Q_REQUIRE(smem <= (size_t)device_max_smem_optin(), B200Q_EUNSUPPORTED, "moe: too many experts (%d)", p.experts);
  if (smem > 48 * 1024)
    B200Q_CUDA_OK(cudaFuncSetAttribute(moe_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(kSortThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  B200Q_CUDA_OK(cudaLaunchKernelEx(&cfg, moe_sort_kernel, p));
  note_launch();
  return B200Q_OK;
}

// out[i] = a[ids[i] / top_k], rows of k 16-bit values; one block per row
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint16_t* __restrict__ a, int64_t lda,
                                                          const int32_t* __restrict__ ids, uint16_t* __restrict__ out,
                                                          int numel, int k, int top_k) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int id = ids[blockIdx.x];
  if (id < 0 || id >= numel) return;
  const uint4* src = reinterpret_cast<const uint4*>(a + (size_t)(id / top_k) * lda);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)blockIdx.x * k);
  for (int i = threadIdx.x; i < k / 8; i += 256) dst[i] = src[i];
}

// out[m] = sum over the slots j of in[m * top_k + j] whose expert is on this rank: fp32 sum in slot order,
// one rounding.  A thread handles eight columns.
template <typename T>
__global__ void __launch_bounds__(256) sum_slots_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out,
                                                        const void* topk_ids, int ids64, const int32_t* expert_map,
                                                        int experts, int m, int top_k, int k) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
  const int k8 = k / 8;
  if (idx >= (long long)m * k8) return;
  const int row = (int)(idx / k8), v = (int)(idx - (long long)row * k8);
  float s[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) s[e] = 0.f;
  for (int j = 0; j < top_k; ++j) {
    const size_t r = (size_t)row * top_k + j;
    const long long ex = ids64 ? static_cast<const long long*>(topk_ids)[r]
                               : (long long)static_cast<const int32_t*>(topk_ids)[r];
    // a row no expert of this rank has written
    if (ex < 0 || ex >= experts || (expert_map && expert_map[ex] < 0)) continue;
    const uint4 x = reinterpret_cast<const uint4*>(in + r * k)[v];
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      s[2 * e] += Pair<T>::to_float((uint16_t)(w[e] & 0xffffu));
      s[2 * e + 1] += Pair<T>::to_float((uint16_t)(w[e] >> 16));
    }
  }
  reinterpret_cast<uint4*>(out + (size_t)row * k)[v] = make_uint4(Pair<T>::pack(s[0], s[1]), Pair<T>::pack(s[2], s[3]),
                                                                  Pair<T>::pack(s[4], s[5]), Pair<T>::pack(s[6], s[7]));
}

template <typename K, typename... Args>
static int launch_pdl(K kernel, dim3 grid, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  B200Q_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, args...));
  note_launch();
  return B200Q_OK;
}

inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// How a layer runs, from sizes known on the host.
struct Plan {
  bool tc;         // tensor-core kernel over a tile list; else the decode kernel over padded blocks
  int pairs;       // tc: CTA pairs
  int box;         // tc: token rows a CTA stages
  int max_rows;    // tc: rows per tile
  int block;       // decode kernel: block size
  int64_t len;     // sorted ids (with padding: a whole number of blocks)
};

// Whether the tensor-core kernel takes the GEMMs, by rows per expert on average.  `group`: the smaller group size of
// the two matrices, 0 when both have a scale per column.  Lines and times (us, a layer of eight experts, top-2,
// decode kernel / tensor cores; 4096 / 14336 unless stated):
//   scales per column    4-bit from 7 rows, 8-bit always
//   groups of 128, up    4-bit from 14 rows (12 rows 323 / 362, 14 rows 370 / 362, 16 rows 530 / 362), 8-bit from two
//                        (two rows 404 / 340, four 424 / 357; 2048 / 1408, two rows 43.3 / 44.3)
//   groups of 64         two buffers of group sums a round: 4-bit above 14.4, where the decode kernel's blocks get wider (14
//                        rows 384 / 449, 16 rows 569 / 447), with zero-points or 8 bits from 14 (8-bit 14 rows 581 / 448;
//                        2048 / 1408 58.0 / 56.7, 12 rows 52.2 / 56.0)
//   other groups         never: the group sums come in whole steps
// The lines hold on other layers: groups of 64, 4-bit, decode kernel / tensor cores at 14 and at 15 rows: 64 experts top-6 2048
// / 1408 205 / 199 and 304 / 198, 128 top-8 2048 / 768 243 / 232 and 377 / 232, 16 top-4 4096 / 2048 135 / 156 and 185 / 156,
// 32 top-4 2880 / 2880 242 / 258 and 365 / 258, 8 top-2 2048 / 1408 43 / 50 and 53 / 50.  Farthest off: 8-bit at 12 to 13
// rows in groups of 64 (577 / 462), 8-bit groups of 128 at three rows of 8 top-2 2048 / 1408 (41 / 46), zero-points in groups of
// 128 at 8 to 13 rows of 128 experts (254 / 213 at 13).
static bool on_tensor_cores(int64_t rows, int64_t experts, int64_t k, int64_t n, int bits, bool zp, int64_t group) {
  if (!tc_gemm_supported(2 * n, k, kChannel) || !tc_gemm_supported(k, n, kChannel)) return false;
  const double avg = (double)rows / (double)experts;
  if (group == 0) return bits == 8 || avg > 7.0;
  if (!tc_group_sums_supported(group)) return false;
  if (group < 128) return avg >= (bits == 4 && !zp ? 14.5 : 14.0);
  return avg >= (bits == 4 ? 14.0 : 2.0);
}

static Plan make_plan(bool tc, int64_t rows, int64_t experts, int64_t global_experts, int64_t group) {
  Plan pl = {};
  const double avg = (double)rows / (double)experts;
  pl.tc = tc;
  if (pl.tc) {
    // pairs where a tile is wide enough for the MMAs to matter
    pl.pairs = avg > 40.0;
    pl.box = group > 0 ? tc_group_sums_rows(pl.pairs ? 2 : 1) / (pl.pairs ? 2 : 1) : !pl.pairs ? 64 : avg > 160.0 ? 128 : 96;
    pl.max_rows = pl.box * (pl.pairs ? 2 : 1);
    pl.len = rows;
  } else {
    // the block sizes of the decode kernel (fused_marlin_moe.py:286-288 walks further, to 64)
    pl.block = rows < 0.9 * 8 * experts ? 8 : rows < 0.9 * 16 * experts ? 16 : 32;
    pl.len = align_up(rows + global_experts * (pl.block - 1), pl.block);
  }
  return pl;
}

struct Layout {
  int64_t sorted, blocks, total, tiles, rows, gate_up, act, down, bytes;
};
static Layout make_layout(const Plan& pl, int64_t rows, int64_t experts, int64_t k, int64_t n) {
  Layout l = {};
  int64_t at = 0;
  auto take = [&](int64_t bytes) { const int64_t o = at; at += align_up(bytes, 256); return o; };
  l.total = take(4);
  l.sorted = take(pl.len * 4);
  l.blocks = take(pl.tc ? 4 : (pl.len / pl.block + 1) * 4);
  l.tiles = take(pl.tc ? (experts + rows / pl.max_rows + 1) * 16 : 16);
  // gathered input rows share their place with the activation output (used one after the other)
  l.rows = l.act = take(rows * (k > n ? k : n) * 2);
  l.gate_up = take(rows * 2 * n * 2);
  l.down = take(rows * k * 2);
  l.bytes = at;
  return l;
}

}  // namespace moe
}  // namespace b200q

using namespace b200q;

extern "C" int b200q_moe_align_block_size(const void* topk_ids, int ids64, const int32_t* expert_map, int64_t numel,
                                          int64_t block_size, int64_t num_experts, int32_t* sorted_token_ids,
                                          int64_t sorted_len, int32_t* expert_ids, int64_t num_blocks,
                                          int32_t* num_tokens_post_padded, b200q_stream_t stream) {
  B200Q_REQUIRE(numel >= 0 && numel < (1ll << 30) && block_size >= 1 && num_experts >= 1, B200Q_EINVAL,
                "moe_align_block_size: invalid size");
  B200Q_REQUIRE(sorted_token_ids && expert_ids && num_tokens_post_padded && (topk_ids || numel == 0), B200Q_EINVAL,
                "null tensor pointer");
  B200Q_REQUIRE(sorted_len >= numel + num_experts * (block_size - 1) && num_blocks * block_size >= sorted_len &&
                    sorted_len < (1ll << 31), B200Q_EINVAL,
                "moe_align_block_size: outputs too small");
  moe::SortParams p = {};
  p.topk_ids = topk_ids; p.ids64 = ids64; p.expert_map = expert_map;
  p.numel = (int)numel; p.experts = (int)num_experts; p.block = (int)block_size;
  p.sorted_ids = sorted_token_ids; p.sorted_len = (int)sorted_len;
  p.block_experts = expert_ids; p.blocks = (int)num_blocks; p.total = num_tokens_post_padded;
  return moe::launch_sort(p, static_cast<cudaStream_t>(stream));
}

extern "C" size_t b200q_fused_marlin_moe_scratch_bytes(int64_t size_m, int64_t top_k, int64_t num_experts,
                                                       int64_t global_experts, int64_t size_k, int64_t size_n, int bits) {
  if (size_m <= 0 || top_k <= 0 || num_experts <= 0) return 256;
  const int64_t rows = size_m * top_k;
  // either kernel may be taken (alignment and the groups decide, too); a tile list is longest with the smallest tiles
  (void)bits;
  size_t most = 0;
  for (int tc = 0; tc < 3; ++tc) {
    const moe::Plan pl = moe::make_plan(tc != 0, rows, num_experts, global_experts, tc == 2 ? 64 : 0);
    const size_t b = (size_t)moe::make_layout(pl, rows, global_experts, size_k, size_n).bytes;
    if (b > most) most = b;
  }
  return most;
}

// One layer: see include/b200q.h
extern "C" int b200q_fused_marlin_moe(
    const void* hidden, int64_t lda, const uint32_t* w1, const uint32_t* w2, const void* w1_scale, const void* w2_scale,
    const uint32_t* w1_zeros, const uint32_t* w2_zeros, const void* bias1, const void* bias2, const float* topk_weights,
    const void* topk_ids, int ids64, const int32_t* expert_map, void* out, void* scratch, size_t scratch_bytes,
    int64_t b_q_type_id, int a_dtype, int64_t size_m, int64_t top_k, int64_t size_k, int64_t size_n,
    int64_t num_experts, int64_t global_experts, int64_t groups1, int64_t groups2, int weight_on_input,
    b200q_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int bits = b_q_type_id == kTypeU8B128 || b_q_type_id == kTypeU8 ? 8 : 4;
  const bool zp = w1_zeros != nullptr;
  B200Q_REQUIRE((b_q_type_id == kTypeU4B8 || b_q_type_id == kTypeU8B128) ? !zp
                : (b_q_type_id == kTypeU4 || b_q_type_id == kTypeU8) && zp, B200Q_EINVAL,
                "moe: b_q_type must be u4 or u8 with zero-points, uint4b8 or uint8b128 without");
  B200Q_REQUIRE((w2_zeros != nullptr) == zp, B200Q_EINVAL, "moe: zero-points of only one of the matrices");
  B200Q_REQUIRE(a_dtype == B200Q_F16 || a_dtype == B200Q_BF16, B200Q_EINVAL, "moe: only bfloat16 and float16");
  B200Q_REQUIRE(size_m >= 0 && top_k >= 1 && num_experts >= 1 && global_experts >= 1 && size_k > 0 && size_n > 0 &&
                    size_k % 64 == 0 && size_n % 32 == 0, B200Q_EINVAL,
                "moe: invalid sizes (M = %lld, K = %lld, N = %lld)", (long long)size_m, (long long)size_k, (long long)size_n);
  if (size_m == 0) return B200Q_OK;
  B200Q_REQUIRE(hidden && w1 && w2 && w1_scale && w2_scale && topk_weights && topk_ids && out && scratch, B200Q_EINVAL,
                "null tensor pointer");
  B200Q_REQUIRE(lda >= size_k && lda % 8 == 0 && (reinterpret_cast<uintptr_t>(hidden) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(out) & 15) == 0, B200Q_EINVAL,
                "moe: activations must be aligned to 16 bytes with a row stride divisible by 8");
  const int64_t rows = size_m * top_k;
  B200Q_REQUIRE(rows < (1ll << 30), B200Q_EINVAL, "moe: too many rows");
  const bool aligned = ((reinterpret_cast<uintptr_t>(w1) | reinterpret_cast<uintptr_t>(w2) | reinterpret_cast<uintptr_t>(w1_scale) |
                         reinterpret_cast<uintptr_t>(w2_scale) | reinterpret_cast<uintptr_t>(w1_zeros) |
                         reinterpret_cast<uintptr_t>(w2_zeros)) & 15) == 0;
  B200Q_REQUIRE(groups1 >= 1 && groups2 >= 1 && size_k % groups1 == 0 && size_n % groups2 == 0, B200Q_EINVAL,
                "moe: invalid number of groups (%lld, %lld)", (long long)groups1, (long long)groups2);
  const int64_t group1 = groups1 > 1 ? size_k / groups1 : 0, group2 = groups2 > 1 ? size_n / groups2 : 0;
  const bool groups_fit = (group1 == 0 || tc_group_sums_supported(group1)) && (group2 == 0 || tc_group_sums_supported(group2));
  const int64_t group = group1 == 0 ? group2 : group2 == 0 ? group1 : group1 < group2 ? group1 : group2;
  const bool tc = aligned && groups_fit && moe::on_tensor_cores(rows, num_experts, size_k, size_n, bits, zp, group);
  const moe::Plan pl = moe::make_plan(tc, rows, num_experts, global_experts, group);
  const moe::Layout l = moe::make_layout(pl, rows, global_experts, size_k, size_n);
  B200Q_REQUIRE((int64_t)scratch_bytes >= l.bytes && (reinterpret_cast<uintptr_t>(scratch) & 255) == 0, B200Q_ESCRATCH,
                "moe: scratch of %zu bytes is below the required %lld", scratch_bytes, (long long)l.bytes);
  char* s = static_cast<char*>(scratch);
  int32_t* sorted = reinterpret_cast<int32_t*>(s + l.sorted);
  int32_t* total = reinterpret_cast<int32_t*>(s + l.total);
  int32_t* block_experts = reinterpret_cast<int32_t*>(s + l.blocks);
  int4* tiles = reinterpret_cast<int4*>(s + l.tiles);
  void *gathered = s + l.rows, *act = s + l.act, *gate_up = s + l.gate_up, *down = s + l.down;

  moe::SortParams sp = {};
  sp.topk_ids = topk_ids; sp.ids64 = ids64; sp.expert_map = expert_map;
  sp.numel = (int)rows; sp.experts = (int)global_experts;
  sp.block = pl.block; sp.max_rows = pl.max_rows;
  sp.sorted_ids = sorted; sp.sorted_len = (int)pl.len;
  sp.block_experts = block_experts; sp.blocks = pl.tc ? 0 : (int)(pl.len / pl.block);
  sp.total = total; sp.tiles = tiles;
  int rc = moe::launch_sort(sp, stream);
  if (rc != B200Q_OK) return rc;
  if (pl.tc) {
    const int fmt = bits == 4 ? (zp ? 1 : 0) : (zp ? 3 : 2);  // the Fmt enum of gemm_tc.cuh
    rc = moe::launch_pdl(moe::gather_rows_kernel, dim3((unsigned)rows), stream, static_cast<const uint16_t*>(hidden), lda,
                         (const int32_t*)sorted, static_cast<uint16_t*>(gathered), (int)rows, (int)size_k, (int)top_k);
    if (rc != B200Q_OK) return rc;
    rc = launch_tc_moe(gathered, rows, w1, w1_scale, w1_zeros, bias1, gate_up, a_dtype, fmt, num_experts, 2 * size_n, size_k,
                       groups1, pl.pairs, pl.box, tiles, total, sorted, 0, weight_on_input ? topk_weights : nullptr, stream);
    if (rc != B200Q_OK) return rc;
    rc = b200q_silu_and_mul(act, gate_up, rows, size_n, a_dtype, stream_);
    if (rc != B200Q_OK) return rc;
    rc = launch_tc_moe(act, rows, w2, w2_scale, w2_zeros, bias2, down, a_dtype, fmt, num_experts, size_k, size_n, groups2,
                       pl.pairs, pl.box, tiles, total, sorted, 1, weight_on_input ? nullptr : topk_weights, stream);
  } else {
    rc = b200q_moe_wna16_marlin_gemm(hidden, lda, w1, w1_scale, w1_zeros, bias1, gate_up, sorted, block_experts, total,
                                     topk_weights, pl.len, pl.block, top_k, weight_on_input, num_experts, b_q_type_id, a_dtype,
                                     size_m, 2 * size_n, size_k, groups1, stream_);
    if (rc != B200Q_OK) return rc;
    rc = b200q_silu_and_mul(act, gate_up, rows, size_n, a_dtype, stream_);
    if (rc != B200Q_OK) return rc;
    rc = b200q_moe_wna16_marlin_gemm(act, size_n, w2, w2_scale, w2_zeros, bias2, down, sorted, block_experts, total,
                                     topk_weights, pl.len, pl.block, 1, !weight_on_input, num_experts, b_q_type_id, a_dtype,
                                     rows, size_k, size_n, groups2, stream_);
  }
  if (rc != B200Q_OK) return rc;
  const dim3 grid((unsigned)((size_m * (size_k / 8) + 255) / 256));
  auto sum = a_dtype == B200Q_F16 ? moe::sum_slots_kernel<half> : moe::sum_slots_kernel<__nv_bfloat16>;
  return moe::launch_pdl(sum, grid, stream, static_cast<const uint16_t*>(down), static_cast<uint16_t*>(out), topk_ids, ids64,
                         expert_map, (int)global_experts, (int)size_m, (int)top_k, (int)size_k);
}
