// Mixed-precision GEMM on the 5th-generation tensor cores: C[M,N] = A[M,K] * dequant(B), tcgen05.mma
// with TMEM accumulators.  The kernel computes C^T = B^T A^T: the weights are the 128-row (CTA pair:
// 256-row) operand, the rows of A ("tokens") are the MMA's N dimension, so that a tile fits any token
// count in steps of 16 (32), a lane of the accumulator is one output column (its channel scale and bias
// are one register), and every CTA converts each weight of its tile once.
//
// One persistent CTA per SM, or (more than 128 tokens) one CTA pair per two SMs: with cta_group::2 a
// 256 x 256 tile is computed by two CTAs that each convert 128 of the 256 weight columns and stage half
// of the tokens; the tensor cores read the other half from the peer.  A single-CTA 256 x 256 tile needs
// 96 B per clock of shared memory for the MMA operands alone, and 176 of the 128 there are together with
// the conversion; the pair needs 64 for the operands and leaves room for two accumulators.
//
// Converted weights go to TMEM, where tcgen05.mma takes its 128-lane operand from as well: a thread converts one
// column, which is a lane there, and shared memory carries neither the store nor the MMAs' reads of them.  Only tiles
// of more than 192 tokens, whose accumulators fill TMEM, keep them in shared memory.  A round (below), cycles, with the
// operand in shared memory / in TMEM: single CTAs 4-bit 48 tokens 822 / 709, 128 tokens 811 / 696, 8-bit 48 tokens 835 /
// 620 (then HBM), fp8 24 tokens 870 / 662; pairs 4-bit 160 tokens 869 / 781, 192 tokens 872 / 839, 8-bit 160 tokens 1039 /
// 699, 192 tokens 1032 / 795.  What bounds it now: instruction issue (60 to 66 % with one or two warps of a kind on a
// scheduler), of which eight instructions a packed word are the conversion; pairs in long runs the power limit.
//
// Roles, hand-offs through mbarriers; a step is 64 deep in k, two steps make a round:
//   16 dequant warps  packed words -> exact 16-bit codes -> scaled -> MMA operand.  Four groups of four take rounds in
//                     turn (weights in shared memory: two groups of eight), so that one waits and fetches while others
//                     convert
//   producer warp     packed weights, scales and zero-points of a round into a ring of kWD slots (four or eight,
//                     what the operands leave room for), one copy each (with a copy per step and per scale
//                     row the issuing thread was the bottleneck at 925 cycles a step; a division in its loop cost 300)
//   token warp        token rows of a round (TMA, 128B swizzle) into kTokRing slots
//   MMA warp          one elected thread issues tcgen05.mma, eight per round, and commits the slots; in the
//                     second CTA of a pair it tells the leader that the CTA's weights are converted
//   4 epilogue warps  TMEM -> registers -> scale and bias -> C, overlapped with the next tile's MMAs (two
//   (8, see SUMS)     accumulator buffers); where K is split, fp32 partial sums -> scratch
//
// Work is cut into (tile, k-range) segments.  Whole waves of tiles run one tile per CTA (pair); what
// would be a ragged last wave (or the only one) is cut into equal k-ranges instead: the workers of such a
// "shared" tile leave fp32 partial tiles in the scratch and tc_reduce_kernel adds them in k order on the
// whole GPU.  (The last worker to arrive adding them in place was slower: four warps of one CTA in three
// took 80 of 107 us at M = 256, 4096 x 4096.)
//
// Every wait is bounded: after kSpinLimit polls a role records a code in *p.error, stops, and the
// kernel drains (TMEM is freed), so a broken hand-off can not hang the GPU.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "gemm_params.cuh"

namespace b200q {
namespace tc {

// weight formats
enum Fmt : int {
  kU4B8 = 0,   // uint4, built-in offset 8
  kU4Z = 1,    // uint4 with packed zero-points
  kU8B128 = 2,
  kU8Z = 3,
  kF8 = 4,     // float8_e4m3fn
  kNV4 = 5,    // float4_e2m1f, fp8 (S0E5M3) scales per 16, global scale
  kMX4 = 6,    // float4_e2m1f, e8m0 scales per 32
  kU4ZF = 7,   // uint4 with 16-bit float zero-points (HQQ)
  kU8ZF = 8,
};
template <int F>
struct FmtInfo {
  static constexpr int kBits = (F == kU8B128 || F == kU8Z || F == kF8 || F == kU8ZF) ? 8 : 4;
  static constexpr bool kFp4 = F == kNV4 || F == kMX4;
  static constexpr bool kZp = F == kU4Z || F == kU8Z;      // packed integer zero-points
  static constexpr bool kZpF = F == kU4ZF || F == kU8ZF;   // float zero-points
};

constexpr int kBK = 64;            // k per step: one 128-byte swizzle row of 16-bit values
constexpr int kRoundTiles = 8;     // k-tiles (16 rows) per round of two steps
constexpr int kBN = 128;           // weight columns per CTA
// epilogue warps: TMEM lane quadrant = warp % 4; with group scales on the sums two share a quadrant
constexpr int epi_warps(bool sums) { return sums ? 8 : 4; }
constexpr uint32_t kSpinLimit = 1u << 24;
// Rows up to which a call fetches packed weights, scales and zero-points before the kernels in front are through, as
// include/b200q.h says: what such a kernel writes is visible after the wait alone.  Captured, us, fetched ahead / behind the
// wait / no early launch: 200 x 2048 x 2048 8.4 / 10.3 / 11.8, 256 x 4096 x 4096 16.3 / 17.0 / 19.0, 1000 x 4096 x 6144
// 41.9 / 42.0 / 43.1.  (Asked for in L2 before the wait: 17.3, 340 x 4096 x 14336 38.5 instead of 37.9.)
constexpr int kAheadRows = 128;

struct TcParams {
  int* error;                // device word: 0 = ok; else (role << 8) | barrier id of the first wait that timed out
  const void* scales;        // [G, N] permuted (fp4: bytes, regrouped)
  const void* bias;          // [N] permuted or null
  const void* global_scale;  // NVFP4
  void* c;                   // [M, N]
  int m, n, k;
  int group_blocks;          // k-tiles (16 rows) per scale group; K/16 when there is one group
  int groups;                // scale groups of one expert
  int group_rows;            // scale rows copied per round
  int channelwise;           // one scale per column: applied to the fp32 sums
  int tn;                    // tokens per tile (multiple of 16, of 32 for a CTA pair)
  int box;                   // token rows a CTA stages per step
  int tok_tiles;             // token tiles
  int workers;               // CTAs, or CTA pairs, of the grid
  int sk_tiles;              // the first tiles are shared out by k-range among all workers
  float chan_factor;         // of the channel-wise scales (fp8: takes the exponent re-bias out)
  float* partials;           // [worker][2][CG][tn][128] fp32
  // mixture of experts: tiles come from a list in device memory {expert, first row, rows}; the rows of A
  // are in sorted order, output row = ids[row] (scatter) or row, scaled by row_weights[ids[row]]
  const int4* tile_list;
  const int32_t* tile_count;
  const int32_t* ids;
  int scatter;               // 0: output rows stay in sorted order
  const float* row_weights;
  int out_rows;
  long long s_stride, bias_stride;  // per expert, elements
};

// A: rows of A; B: packed weights; S: scales; Z: zero-points (the last two only where the format has them)
struct TcMaps {
  CUtensorMap a, b, s, z;
};

// ---- PTX wrappers ------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
// One arrival of a converged warp: by lane 0, as a predicate (a branch costs a dozen instructions with what joins the
// lanes again).
__device__ __forceinline__ void mbar_arrive(uint32_t bar, int lane) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}\n" ::"r"(bar),
               "r"(lane)
               : "memory");
}
// arrive on a barrier of the other CTA, given by its cluster address (mapa), as a release at cluster scope of what
// this thread has written or seen written in its own CTA's shared memory: that is all the waiter (acquire at
// cluster scope) reads.  (An arrival's default scope is its own CTA; arrive.release.cluster took 1350 cycles, the
// fence limited to shared memory costs a layer 0 to 1 %, 3 % at 200 tokens.)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n" ::: "memory");
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
               : "memory");
}
// Bounded wait on a phase parity.  Returns false (and records `what`) on time-out.  CLUSTER: the
// barrier is also arrived on by the peer CTA (acquire at cluster scope).  SLEEP_NS: back off between
// polls (roles with long waits leave the issue slots to the others).
template <bool CLUSTER>
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  if (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  return done != 0;
}
template <bool CLUSTER, int SLEEP_NS = 0>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int what, volatile int* cta_abort,
                                          int* error) {
  if (__builtin_expect(mbar_try<CLUSTER>(bar, parity), 1)) return true;
  for (uint32_t spin = 1; spin < kSpinLimit; ++spin) {
    if (SLEEP_NS > 0) __nanosleep(SLEEP_NS);
    if (mbar_try<CLUSTER>(bar, parity)) return true;
    // now and then: stop early if another role of this CTA has already given up
    if ((spin & 1023u) == 1023u && *cta_abort != 0) return false;
  }
  *cta_abort = 1;
  atomicCAS(error, 0, what);
  return false;
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];\n" ::"l"(map) : "memory");
}
// CG == 2: the barrier may be the peer's (its cluster address is given)
template <int CG>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  if (CG == 2)
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
  else
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
  if (CG == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  if (CG == 2)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(cols) : "memory");
  else
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// D[tmem] (+)= A * B, 16-bit inputs, fp32 accumulate.  B in shared memory (b: low word of its descriptor, hi: the high
// word), A there too, or (TA) in TMEM: 128 lanes of each CTA, two k per column.
#define B200Q_UMMA(G, A_DECL, A_OP)                                                                                    \
  asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\t" A_DECL                           \
               "mov.b64 db, {%2, %3};\n\ttcgen05.mma.cta_group::" G ".kind::f16 [%0], " A_OP ", db, %4, p;\n\t}\n" ::"r"( \
                   d_tmem),                                                                                            \
               "r"(a), "r"(b), "r"(hi), "r"(idesc), "r"(accumulate)                                                    \
               : "memory")
template <int CG, bool TA>
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint32_t a, uint32_t b, uint32_t hi, uint32_t idesc,
                                         uint32_t accumulate) {
  if constexpr (TA) {
    if constexpr (CG == 2) B200Q_UMMA("2", "", "[%1]");
    else B200Q_UMMA("1", "", "[%1]");
  } else {
    if constexpr (CG == 2) B200Q_UMMA("2", "mov.b64 da, {%1, %3};\n\t", "da");
    else B200Q_UMMA("1", "mov.b64 da, {%1, %3};\n\t", "da");
  }
}
// arrive on an mbarrier (CG == 2: the same one of both CTAs) when all MMAs issued so far have completed
template <int CG>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  if (CG == 2)
    asm volatile(
        "{\n\t.reg .b16 mask;\n\tmov.u16 mask, 3;\n\t"
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], mask;\n\t}\n" ::
            "r"(bar)
        : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// 32 lanes x 16 consecutive fp32 columns of TMEM -> 16 registers per thread
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// 32 lanes x 32 consecutive fp32 columns of TMEM -> 32 registers per thread
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// true in one lane of a converged warp; unlike a lane test it keeps the operands of the tensor-core
// instructions in uniform registers
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(pred));
  return pred != 0;
}

// four 8 x 8 matrices of 16-bit values in the MMA fragment layout; lane 8 i + r gives row r of matrix i
template <int OFF>
__device__ __forceinline__ void stmatrix_x4_off(uint32_t addr, const uint32_t (&f)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0+%5], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(f[0]), "r"(f[1]),
               "r"(f[2]), "r"(f[3]), "n"(OFF)
               : "memory");
}

// Shared-memory matrix descriptor: K-major tile, 128-byte swizzle, rows 128 B apart, 8-row atoms 1024 B
// apart (version 1 = sm_100 format): low word (16-byte address, leading offset 1), high word.
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
constexpr uint32_t kDescHi = 64u | (1u << 14) | (2u << 29);
// instruction descriptor: fp32 accumulate, A and B K-major
template <typename T>
__device__ __forceinline__ uint32_t make_idesc(int m, int n) {
  const uint32_t f = std::is_same<T, half>::value ? 0u : 1u;
  return (1u << 4) | (f << 7) | (f << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Tokens of a tile at most, where group scales are applied to the sums (two buffers of group sums beside the weights
// in TMEM; the tile's running sums in registers).
__host__ __device__ constexpr int group_sums_tokens(int cg) { return cg == 1 ? 64 : 160; }

// Shared-memory and TMEM plan.  TOK: token rows a CTA can stage per step.  SUMS: group scales stay out of the weight
// ring.
template <int F, int CG, int TOK, bool SUMS>
struct TcCfg {
  using I = FmtInfo<F>;
  static constexpr int kTileBytes = 16 * 64 * I::kBits / 8;    // one packed 16 x 64 weight tile
  static constexpr int kWBytes = kRoundTiles * 2 * kTileBytes;  // 8 k-tiles x 2 column tiles
  // rows of scales (fp4: of byte pairs) a round can touch
  static constexpr int kSRow = 2 * kBN;
  static constexpr int kSBytes = SUMS ? 0 : (F == kNV4 ? 4 : F == kMX4 ? 2 : kRoundTiles) * kSRow;
  static constexpr int kZRow = I::kZpF ? 2 * kBN : I::kZp ? kBN * I::kBits / 8 : 0;
  static constexpr int kSZBytes = kSBytes + kRoundTiles * kZRow;  // scales and zero-points of a round: a multiple of 128
  static constexpr int kWSlot = kWBytes + kSZBytes;
  // Converted weights: in TMEM (two k per column, a round 64 columns), where the accumulators leave room; else in
  // shared memory behind the token rows of the slot.
  static constexpr int kBufCols = SUMS ? group_sums_tokens(CG) : CG * (TOK <= 64 ? 64 : TOK);
  static constexpr int kBufs = SUMS && CG == 1 ? 4 : 2;
  static constexpr int kTmemSlots = (512 - kBufs * kBufCols) / 64;
  static constexpr bool kInTmem = kTmemSlots >= 2;
  static constexpr int kTmemCols = kInTmem ? 512 : kBufs * kBufCols;
  static constexpr int kACol = 512 - kTmemSlots * 64;  // first column of the weights
  static constexpr int kTokBytes = TOK * 128;                // token rows of a step
  static constexpr int kABytes = kInTmem ? 0 : kBN * 128;    // converted weights of a step in shared memory
  static constexpr int kBarBytes = 1024;
  // SUMS: scales of sixteen groups for each epilogue warp, the 64 columns that its 32 are stored among
  static constexpr int kEpiWarpBytes = SUMS ? 16 * 128 : 0;
  static constexpr int kEpiBytes = epi_warps(SUMS) * kEpiWarpBytes;
  static constexpr int kRoom = 226 * 1024 - kBarBytes - kEpiBytes - 1024;  // - alignment slack
  // Rings: token rows of kTokRing rounds, converted weights of kARing.  A token row asked for takes up to 1800 cycles
  // to arrive, so with weights in TMEM four rounds of them (six were no faster; 192 tokens with two 938 cycles a round,
  // 800 with four), beside eight slots of packed weights where these fit, else four.  Weights in shared memory: three
  // slots of both where two slots of packed weights still fit: with two, the chain conversion -> MMAs -> next conversion
  // of a slot (2540 cycles at 256 tokens) is longer than the MMAs of two rounds.
  static constexpr int kBoth = 2 * (kTokBytes + kABytes);
  static constexpr int kARing = !kInTmem ? (3 * kBoth + 2 * kWSlot <= kRoom ? 3 : 2) : kTmemSlots > 4 ? 4 : kTmemSlots;
  static constexpr int kTokFit8 = (kRoom - 8 * kWSlot) / (2 * kTokBytes), kTokFit4 = (kRoom - 4 * kWSlot) / (2 * kTokBytes);
  static constexpr int kTokFit = kTokFit8 >= 4 ? kTokFit8 : kTokFit4;
  static constexpr int kTokRing = !kInTmem ? kARing : kTokFit > 4 ? 4 : kTokFit;
  static constexpr int kRingBytes = kTokRing * 2 * kTokBytes + kARing * 2 * kABytes;
  // Dequant warps: groups that take rounds in turn.  In TMEM four groups of four, a warp both steps of a round; else
  // two groups of eight, a warp one step.
  static constexpr int kGroupWarps = kInTmem ? 4 : 8;
  static constexpr int kGroups = kInTmem ? 4 : 2;
  static_assert(kTokRing >= kGroups && kTokRing >= kARing, "parities of the dequant warps' waits");
  static constexpr int kFit = (kRoom - kRingBytes) / kWSlot;
  static constexpr int kWD = (kFit > 8 ? 8 : kFit) / kGroups * kGroups;  // a slot always belongs to the same group
  // Roles by warp (one stays idle: they begin at a multiple of four, the unit of a register split and of the TMEM
  // quadrants)
  static constexpr int kDequantWarps = kGroups * kGroupWarps;
  static constexpr int kProducerWarp = kDequantWarps;
  static constexpr int kTokenWarp = kProducerWarp + 1;
  static constexpr int kMmaWarp = kTokenWarp + 1;
  static constexpr int kEpiWarp0 = kMmaWarp + 2;
  static constexpr int kThreads = 32 * (kEpiWarp0 + epi_warps(SUMS));
  // With few places in TMEM (pairs) a dequant warp holds the whole round in registers before it asks for one: with
  // half of the conversion done on the place, it went round in 2500 cycles (160 tokens, three places).
  static constexpr bool kHoldRound = kInTmem && !SUMS && kARing < 4;
  // Registers a thread of the roles (SUMS: the epilogue holds up to 80 sums); what the launch has is an upper limit.  The
  // forms with a split spill 52 to 224 bytes, outside the rounds: warp-level loads and stores of local memory are 22200 and
  // 18500 a launch at 160 tokens, 7400 and 7104 at 192, 15984 and 12284 for SUMS in single CTAs, at K = 4096 as at 16384;
  // 0.2 % of the instructions of a layer of eight experts at 500 tokens.  (56 registers instead of 40 for the other roles
  // leave them as they are.)
  static constexpr bool kSplitRegs = SUMS || kHoldRound;
  static constexpr int kDequantRegs = kHoldRound ? 88 : CG == 1 ? 64 : 56, kOtherRegs = kHoldRound ? 48 : 40,
                       kEpiRegs = kHoldRound ? 80 : CG == 1 ? 96 : 120;
  static_assert(!kSplitRegs || 32 * (kDequantWarps * kDequantRegs + 4 * kOtherRegs + epi_warps(SUMS) * kEpiRegs) <=
                                   kThreads * (65536 / kThreads / 8 * 8), "registers");
  static constexpr int kSmemBytes = kRingBytes + kWD * kWSlot + kBarBytes + kEpiBytes + 1024;  // + alignment slack
};

// Position in a ring of N slots and the parity of the current pass over it.
template <int N>
struct Ring {
  int i = 0;
  uint32_t ph = 0;
  template <int BY = 1>
  __device__ __forceinline__ void next() {
    i += BY % N;
    if (BY / N % 2 != 0) ph ^= 1;
    if (BY % N != 0 && i >= N) { i -= N; ph ^= 1; }
  }
};

// ---- schedule ------------------------------------------------------------------------
struct Segment {
  int n_tile;        // tile along N, in units of CG * 128 columns
  int tok0, rows;    // first token row, valid rows
  int expert;
  int r0, r1;        // rounds
  bool shared;       // a k-range of a shared tile
  int slot;          // shared: where the partial sums go
};

// Which of `workers` equal shares of `units` holds `unit`.
__device__ __forceinline__ int share_of(long long unit, int workers, long long units) {
  return (int)(((unit + 1) * workers - 1) / units);
}

// All roles of a worker walk the same sequence of segments.
struct Schedule {
  const TcParams& p;
  int worker, rounds;      // rounds per tile
  long long u, u1, units;  // shared region: range of (tile, round) units
  int tile, tiles;         // whole tiles
  __device__ Schedule(const TcParams& p_, int worker_, int cols_per_tile)
      : p(p_), worker(worker_), rounds((p_.k / kBK + 1) / 2) {
    const int n_tiles = (p.n + cols_per_tile - 1) / cols_per_tile;
    tiles = n_tiles * (p.tile_list ? *p.tile_count : p.tok_tiles);
    units = (long long)p.sk_tiles * rounds;
    u = units * worker / p.workers;
    u1 = units * (worker + 1) / p.workers;
    tile = p.sk_tiles + worker;
  }
  __device__ __forceinline__ void place(Segment& s, int t) const {
    if (p.tile_list) {
      const int count = *p.tile_count;
      const int4 e = __ldg(p.tile_list + t % count);
      s.n_tile = t / count;
      s.expert = e.x; s.tok0 = e.y; s.rows = e.z;
    } else {
      s.n_tile = t / p.tok_tiles;
      s.expert = 0;
      s.tok0 = (t - s.n_tile * p.tok_tiles) * p.tn;
      s.rows = min(p.tn, p.m - s.tok0);
    }
  }
  __device__ __forceinline__ bool next(Segment& s) {
    if (u < u1) {
      const int t = (int)(u / rounds);
      s.r0 = (int)(u - (long long)t * rounds);
      s.r1 = (int)min((long long)rounds, s.r0 + (u1 - u));
      u += s.r1 - s.r0;
      place(s, t);
      s.shared = true;
      s.slot = 2 * worker + (s.r0 > 0 ? 0 : 1);
      return true;
    }
    if (tile < tiles) {
      s.r0 = 0;
      s.r1 = rounds;
      s.shared = false;
      place(s, tile);
      tile += p.workers;
      return true;
    }
    return false;
  }
  // tokens of the MMA for this segment: a narrow last tile leaves MMAs out (by itself worth up to 1 %: captured, 340 x 14336 x
  // 4096 39.2 -> 38.9 us, 8-bit 333 x 3584 x 37888 76.25 -> 76.2)
  template <int CG>
  __device__ __forceinline__ int mma_n(const Segment& s) const {
    constexpr int g = 16 * CG;
    return (s.rows + g - 1) / g * g;
  }
};

// ---- conversion ------------------------------------------------------------------------
// A thread converts one column: of a k-tile it takes four packed words (q = 0..3), each with the codes of rows 2q,
// 2q + 1 (pair `lo`) and 2q + 8, 2q + 9 (pair `hi`) of its column.  4-bit words hold those of column c8 + 8, too, one
// byte further up (`h8` = 8 in the threads of those columns).
//
// What is subtracted from the code, made once per group: the format's own offset, or the zero-point.
template <typename T, int F>
struct Offset {
  uint32_t lo, hi;  // operands of the subtraction (fp16 4-bit `hi`: of the fma)
};
template <typename T, int F>
__device__ __forceinline__ Offset<T, F> make_offset(uint32_t z) {  // z: packed zero-point of the column
  constexpr bool kHalf = std::is_same<T, half>::value;
  using I = FmtInfo<F>;
  Offset<T, F> o;
  if constexpr (I::kFp4 || F == kF8) {
    o.lo = o.hi = 0;
  } else if constexpr (I::kBits == 4) {
    const uint32_t zz = F == kU4Z ? z | (z << 16) : F == kU4B8 ? 0x00080008u : 0u;
    if constexpr (kHalf) {
      o.lo = 0x64006400u + zz;         // 1024 + z
      o.hi = 0xd400d400u + (zz << 4);  // -(64 + z)
    } else {
      o.lo = o.hi = 0x43004300u + zz;  // 128 + z
    }
  } else if constexpr (kHalf) {
    o.lo = o.hi = 0x64006400u + (F == kU8Z ? z | (z << 16) : F == kU8B128 ? 0x00800080u : 0u);
  } else {
    // codes come as code - 128 (see below): z - 128, an exact small integer
    o.lo = o.hi = F == kU8Z ? (uint32_t)Pair<T>::from_float((float)((int)z - 128)) * 0x10001u : 0u;
  }
  return o;
}
template <typename T, int F>
__device__ __forceinline__ void convert_word(uint32_t w, uint32_t h8, const Offset<T, F>& o, uint32_t& lo, uint32_t& hi) {
  constexpr bool kHalf = std::is_same<T, half>::value;
  using I = FmtInfo<F>;
  if constexpr (I::kFp4) {
    // sign, two exponent bits, one mantissa bit into the fields of the 16-bit format
    constexpr int kShift = kHalf ? 3 : 6;
    const uint32_t a = w << (12 - h8), b = w << (8 - h8);
    lo = (a & 0x80008000u) | ((a & 0x70007000u) >> kShift);
    hi = (b & 0x80008000u) | ((b & 0x70007000u) >> kShift);
    if constexpr (F == kMX4) {  // exact re-bias, 2^126
      lo = Pair<T>::mul(lo, 0x7e807e80u);
      hi = Pair<T>::mul(hi, 0x7e807e80u);
    }
  } else if constexpr (I::kBits == 4) {
    const uint32_t x = w >> h8;
    if constexpr (kHalf) {
      lo = Pair<T>::sub(mask_or(x, reg_const<0x000f000fu>(), reg_const<0x64006400u>()), o.lo);
      hi = Pair<T>::fma(mask_or(x, reg_const<0x00f000f0u>(), reg_const<0x64006400u>()), 0x2c002c00u, o.hi);
    } else {
      lo = Pair<T>::sub(mask_or(x, reg_const<0x000f000fu>(), reg_const<0x43004300u>()), o.lo);
      hi = Pair<T>::sub(mask_or(x >> 4, reg_const<0x000f000fu>(), reg_const<0x43004300u>()), o.hi);
    }
  } else if constexpr (F == kF8) {
    uint32_t t[2];
    dequant_fp8<T>(w, t);
    lo = t[0];
    hi = t[1];
  } else if constexpr (kHalf) {
    lo = Pair<T>::sub(__byte_perm(w, 0x64646464u, 0x4240), o.lo);
    hi = Pair<T>::sub(__byte_perm(w, 0x64646464u, 0x4341), o.hi);
  } else {
    // The low seven bits fit bf16's mantissa: (128 + low) - (128 or 256, by the eighth bit) = code - 128.
    static_assert(F != kU8ZF, "float zero-points are fp16's alone");
    const uint32_t m = reg_const<0x007f007fu>(), e = reg_const<0x43004300u>(), t = 0x00800080u, f = 0x43804380u;
    const uint32_t w8 = w >> 8;
    lo = Pair<T>::sub(mask_or(w, m, e), (w & t) ^ f);
    hi = Pair<T>::sub(mask_or(w8, m, e), (w8 & t) ^ f);
    if constexpr (F == kU8Z) {
      lo = Pair<T>::sub(lo, o.lo);
      hi = Pair<T>::sub(hi, o.hi);
    }
  }
}

// fp4: a scale byte, given in both halves of a word, as a 16-bit pair
template <typename T, int F>
__device__ __forceinline__ uint32_t fp4_scale(uint32_t b) {
  if constexpr (F == kMX4 || std::is_same<T, half>::value) {
    return b << 7;  // e8m0 -> bf16 exponent; S0E5M3 -> fp16 bits 14..7
  } else {
    const uint32_t t = b << 4;  // -> bf16: top exponent bit, then the seven lower bits
    return (t & 0x07f007f0u) | ((t & 0x08000800u) << 3);
  }
}

// SUMS: group scales are applied to fp32 sums, as in the decode kernel, so that calls which either kernel may take
// give results of one precision.  The MMAs take the exact codes, a group of k at a time into one of a ring of TMEM
// buffers; the epilogue warps add scale x buffer to the tile's running sums in registers while the next group is
// computed.  Groups of one step or of whole rounds only.  fp16 results that are not the correctly rounded ones: 0.03 to
// 0.13 % over 2048 .. 8192 deep layers of every integer type (decode kernel 0.8 to 6 %, scaled weights rounded to 16 bits
// 39 %).
// What bounds it: the hand-overs, and instruction issue (58 to 64 %) with the conversion beside it.  Cycles a round, with
// the operand in shared memory and the running sums of pairs in TMEM / now: single CTAs 4-bit 32 rows 1084 / 890, 8-bit 16
// rows 1056 / 959; pairs at 125 rows (eight experts, 4096 / 14336, 500 tokens) 1320 / 1190.  Two terms per weight, the
// rounded product and the rest, are as exact but take the MMAs twice; with four epilogue warps, or a wait for every
// buffer, a round took 0.78 us.
template <typename T, int F, int CG, int TOK, bool SUMS>
__global__ void __launch_bounds__(TcCfg<F, CG, TOK, SUMS>::kThreads, 1)
gemm_tc_kernel(const __grid_constant__ TcMaps maps, const TcParams p) {
  using Cfg = TcCfg<F, CG, TOK, SUMS>;
  using I = FmtInfo<F>;
  static_assert(!SUMS || (!I::kFp4 && !I::kZpF && F != kF8), "sums of exact integer codes");
  constexpr int RING = Cfg::kTokRing, ARING = Cfg::kARing, WD = Cfg::kWD, BITS = I::kBits;
  constexpr bool kPair = CG == 2;
  constexpr int kDequantWarps = Cfg::kDequantWarps, kProducerWarp = Cfg::kProducerWarp, kTokenWarp = Cfg::kTokenWarp,
                kMmaWarp = Cfg::kMmaWarp, kEpiWarp0 = Cfg::kEpiWarp0;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t a_base = smem_base + RING * 2 * Cfg::kTokBytes;
  const uint32_t w_base = smem_base + Cfg::kRingBytes;
  const uint32_t sz_base = w_base + WD * Cfg::kWBytes;  // scales and zero-points of the rounds
  const uint32_t bars = sz_base + WD * Cfg::kSZBytes;
  auto tok_slot = [&](int i) { return smem_base + i * 2 * Cfg::kTokBytes; };
  // barriers (8 bytes each).  full (token rows landed and weights converted) and tmem_empty of the
  // leader CTA serve the pair; full of the other CTA counts its own conversion.
  auto full = [&](int i) { return bars + 8 * i; };
  auto empty = [&](int i) { return bars + 8 * (RING + i); };
  auto full_w = [&](int w) { return bars + 8 * (2 * RING + w); };
  auto empty_w = [&](int w) { return bars + 8 * (2 * RING + WD + w); };
  const uint32_t bars2 = bars + 8 * (2 * RING + 2 * WD);
  // TMEM: accumulator buffers, then the converted weights.  Buffers are given back REL at a time, so that the MMA
  // warp rarely waits for one.
  constexpr int BUFS = Cfg::kBufs, REL = BUFS / 2;
  constexpr uint32_t kBufCols = Cfg::kBufCols, kTmemCols = Cfg::kTmemCols;
  static_assert(BUFS * kBufCols + (Cfg::kInTmem ? ARING * 64 : 0) <= kTmemCols, "TMEM");
  auto tmem_full = [&](int b) { return bars2 + 8 * b; };
  auto tmem_empty = [&](int b) { return bars2 + 8 * (BUFS + b); };
  const uint32_t tmem_slot = bars2 + 8 * (BUFS + 2);

  if (threadIdx.x == 32 * kProducerWarp) {
    prefetch_map(&maps.b);
    prefetch_map(&maps.a);
    if (I::kFp4 || (!SUMS && !p.channelwise)) prefetch_map(&maps.s);
    if (I::kZp || I::kZpF) prefetch_map(&maps.z);
  }
  // the next kernel in the stream may be scheduled while this one runs (it waits for completion itself)
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  __shared__ int s_abort;
  volatile int* cta_abort = &s_abort;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = kPair ? (blockIdx.x & 1) : 0;
  const int worker = kPair ? blockIdx.x >> 1 : blockIdx.x;
  const int NT = p.n / 64;
  const int gb = p.group_blocks;
  const int steps = p.k / kBK;
  const int group_steps = gb / 4;  // SUMS: 1 or even

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < RING; ++i) {
      // conversion of this CTA; the leader's also the token rows and the other CTA's conversion
      mbar_init(full(i), Cfg::kGroupWarps + (rank == 0 ? CG : 0));
      mbar_init(empty(i), 1);
    }
    for (int w = 0; w < WD; ++w) {
      mbar_init(full_w(w), 1);
      mbar_init(empty_w(w), Cfg::kGroupWarps);
    }
    for (int b = 0; b < BUFS; ++b) mbar_init(tmem_full(b), 1);
    for (int b = 0; b < 2; ++b) mbar_init(tmem_empty(b), epi_warps(SUMS) * CG);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kMmaWarp) tmem_alloc<CG>(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  if (kPair) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot));
  // the tile list of a mixture-of-experts call is written by the kernel in front
  if (p.tile_list) asm volatile("griddepcontrol.wait;\n" ::: "memory");
  Schedule sched(p, worker, CG * kBN);
  Segment sg;
  if (warp >= kDequantWarps && warp < kEpiWarp0) {
    if constexpr (Cfg::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(Cfg::kOtherRegs));
    if (warp == kProducerWarp) {
      // ================= producer =========================================================
      // Packed weights run ahead of the kernel in front, up to kAheadRows rows.  (The line itself costs calls below that 0 to
      // 0.1 us, wherever it stands: 48 x 14336 x 4096 17.6 -> 17.7.  With the scales on the sums a call has few rows or has
      // waited for its tile list: expert layers were 1 % slower with the line.)
      if constexpr (!SUMS)
        if (p.m > kAheadRows) asm volatile("griddepcontrol.wait;\n" ::: "memory");
      Ring<WD> wr;
      bool ok = true;
      const int kt_all = p.k / 16;
      const int g_step = kRoundTiles / gb, g_step_rest = kRoundTiles - g_step * gb;  // groups in a round
      const bool scales = I::kFp4 || (!SUMS && !p.channelwise);
      const uint32_t bytes = Cfg::kWBytes + (scales ? (I::kFp4 ? Cfg::kSBytes : p.group_rows * Cfg::kSRow) : 0) +
                             p.group_rows * Cfg::kZRow;
      while (ok && sched.next(sg)) {
        const int nt0 = (sg.n_tile * CG + (int)rank) * 2;
        // first row of scales of a round; everything past the end of a matrix is zero-filled and counted
        int g0 = sg.r0 * kRoundTiles / gb, g_rest = sg.r0 * kRoundTiles - g0 * gb;
        g0 += sg.expert * p.groups;
        for (int r = sg.r0; r < sg.r1; ++r) {
          if (!(ok = mbar_wait<false>(empty_w(wr.i), wr.ph ^ 1, (1 << 8) | 3, cta_abort, p.error))) break;
          const uint32_t dst = w_base + wr.i * Cfg::kWBytes, dst_sz = sz_base + wr.i * Cfg::kSZBytes, bar = full_w(wr.i);
          if (elect_one()) {
            mbar_expect_tx(bar, bytes);
            tma_load_3d(dst, &maps.b, 0, nt0 * BITS, sg.expert * kt_all + r * kRoundTiles, bar);
            if (I::kFp4)
              tma_load_2d<1>(dst_sz, &maps.s, nt0 * 16, r * (Cfg::kSBytes / Cfg::kSRow), bar);
            else if (scales)
              tma_load_2d<1>(dst_sz, &maps.s, nt0 * 64, g0, bar);
            if (I::kZp || I::kZpF)
              tma_load_2d<1>(dst_sz + Cfg::kSBytes, &maps.z, I::kZp ? nt0 * 2 * BITS : nt0 * 64, g0, bar);
          }
          __syncwarp();
          wr.next();
          g0 += g_step;
          g_rest += g_step_rest;
          if (g_rest >= gb) {
            g_rest -= gb;
            ++g0;
          }
        }
      }
    } else if (warp == kTokenWarp) {
      // ================= token rows =======================================================
      Ring<RING> ring;
      bool ok = true;
      const uint32_t ft0 = kPair ? mapa(full(0), 0) : full(0);  // the leader's
      // the rows of A come from the kernel in front (programmatic dependent launch)
      asm volatile("griddepcontrol.wait;\n" ::: "memory");
      while (ok && sched.next(sg)) {
        const int row = sg.tok0 + (kPair ? (int)rank * (sched.template mma_n<CG>(sg) / 2) : 0);
        for (int r = sg.r0; r < sg.r1; ++r) {
          if (!(ok = mbar_wait<kPair>(empty(ring.i), ring.ph ^ 1, (1 << 8) | 4, cta_abort, p.error))) break;
          const bool two = 2 * r + 1 < steps;  // a K of an odd number of steps ends with a round of one
          if (elect_one()) {
            if (rank == 0) mbar_expect_tx(full(ring.i), CG * p.box * (two ? 256 : 128));
            tma_load_2d<CG>(tok_slot(ring.i), &maps.a, 2 * r * kBK, row, ft0 + 8 * ring.i);
            if (two) tma_load_2d<CG>(tok_slot(ring.i) + Cfg::kTokBytes, &maps.a, (2 * r + 1) * kBK, row, ft0 + 8 * ring.i);
          }
          __syncwarp();
          ring.next();
        }
      }
    } else if (warp == kMmaWarp) {
      // ================= MMA issuer (leader CTA), relay (the other CTA of a pair) ==========
      // the whole warp walks the loop, one elected lane issues
      if (rank == 0) {
        Ring<RING> ring;
        Ring<ARING> a_ring;
        int acc_i = 0;  // buffers filled so far
        bool ok = true;
        // the ring stays below 256 KB: slot offsets add up in the address field of the descriptors
        const uint32_t da0 = Cfg::kInTmem ? tmem_base + Cfg::kACol : smem_desc_lo(a_base), db0 = smem_desc_lo(tok_slot(0));
        while (ok && sched.next(sg)) {
          const uint32_t idesc = make_idesc<T>(CG * 128, sched.template mma_n<CG>(sg));
          // a commit hands one buffer to the epilogue: the sums of the segment, or (SUMS) of each of its groups
          uint32_t d = 0;
          auto open = [&]() {
            if (acc_i % REL == 0) {
              if (!(ok = mbar_wait<kPair>(tmem_empty((acc_i / REL) & 1), ((acc_i / BUFS) & 1) ^ 1, (2 << 8) | 5, cta_abort, p.error)))
                return;
              tc_fence_after();
            }
            d = tmem_base + acc_i % BUFS * kBufCols;
          };
          // MMAs of a step; `fresh`: they begin a buffer
          auto issue = [&](uint32_t a, uint32_t b, bool fresh) {
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16) {
              umma_f16<CG, Cfg::kInTmem>(d, a + (Cfg::kInTmem ? 8 : 2) * k16, b + 2 * k16, kDescHi, idesc, k16 > 0 || !fresh);
            }
          };
          // the second step of a slot; the next slot
          constexpr uint32_t kA1 = Cfg::kInTmem ? 32 : Cfg::kABytes / 16, kB1 = Cfg::kTokBytes / 16;
          constexpr uint32_t kASlot = Cfg::kInTmem ? 64 : 2 * Cfg::kABytes / 16;
          // rounds until the buffer is handed over (SUMS with groups of a single step: two buffers per round)
          const int rounds_per_buf = SUMS ? group_steps / 2 : sg.r1 - sg.r0;
          int left = SUMS && rounds_per_buf > 0 ? rounds_per_buf - sg.r0 % rounds_per_buf : sg.r1 - sg.r0;
          bool fresh = true;
          for (int r = sg.r0; r < sg.r1; ++r) {
            if (!(ok = mbar_wait<kPair>(full(ring.i), ring.ph, (2 << 8) | 0, cta_abort, p.error))) break;
            if (fresh) {
              open();
              if (!ok) break;
            }
            tc_fence_after();
            const uint32_t da = da0 + a_ring.i * kASlot, db = db0 + ring.i * (2 * Cfg::kTokBytes / 16);
            const bool second = 2 * r + 1 < steps;
            if (!SUMS || rounds_per_buf > 0) {
              const bool last = --left == 0 || r + 1 == sg.r1;
              if (elect_one()) {
                issue(da, db, fresh);
                if (second) issue(da + kA1, db + kB1, false);
                umma_commit<CG>(empty(ring.i));  // slot reusable once these MMAs have read it
                if (last) umma_commit<CG>(tmem_full(acc_i % BUFS));
              }
              fresh = last;
              if (last) {
                ++acc_i;
                left = rounds_per_buf;
              }
            } else {
              if (elect_one()) {
                issue(da, db, true);
                umma_commit<CG>(tmem_full(acc_i % BUFS));
                if (!second) umma_commit<CG>(empty(ring.i));
              }
              __syncwarp();
              ++acc_i;
              if (second) {
                open();
                if (!ok) break;
                if (elect_one()) {
                  issue(da + kA1, db + kB1, true);
                  umma_commit<CG>(tmem_full(acc_i % BUFS));
                  umma_commit<CG>(empty(ring.i));
                }
                ++acc_i;
              }
            }
            __syncwarp();
            ring.next();
            a_ring.next();
          }
        }
      } else {
        Ring<RING> ring;
        bool ok = true;
        const uint32_t leader = mapa(full(0), 0);
        while (ok && sched.next(sg)) {
          for (int r = sg.r0; r < sg.r1; ++r) {
            if (!(ok = mbar_wait<false>(full(ring.i), ring.ph, (2 << 8) | 6, cta_abort, p.error))) break;
            if constexpr (Cfg::kInTmem) {  // passes on that the weights are in this CTA's TMEM
              tc_fence_after();
              tc_fence_before();
            }
            if (elect_one()) mbar_arrive_cluster(leader + 8 * ring.i);
            __syncwarp();
            ring.next();
          }
        }
      }
    }
  } else if (warp < kDequantWarps) {
    if constexpr (Cfg::kHoldRound) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(Cfg::kDequantRegs));
    else if constexpr (Cfg::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(Cfg::kDequantRegs));
    // ================= dequant warps ====================================================
    // A thread is a column, and as such a lane of TMEM; a group of warps takes every kGroups-th round, a warp one step
    // or both.  Four packed words of a k-tile at a time: the copy's 128-byte swizzle puts the words of a warp's columns
    // in different banks.
    constexpr int GROUPS = Cfg::kGroups;
    const int quad = warp & 3, group = warp / Cfg::kGroupWarps;
    const int col = quad * 32 + lane, nt = col >> 6, sub = (col >> 4) & 3, h = (col >> 3) & 1, c8 = col & 7;
    const uint32_t h8 = BITS == 4 ? 8 * h : 0;
    // word q of k-tile i: w_rel + i * 2 kTileBytes, its 16-byte chunk (4-bit: 4 (c8 % 2) + q, 8-bit: 2 q + sub / 2)
    // within the 128-byte row (4-bit: 4 nt + c8 / 2, 8-bit: 8 nt + c8) exchanged with the row's number
    const uint32_t w_row = BITS == 4 ? 4 * nt + (c8 >> 1) : 8 * nt + c8;
    const uint32_t w_chunk = (BITS == 4 ? 4 * (c8 & 1) : sub >> 1) ^ (w_row & 7);
    const uint32_t w_rel = w_row * 128 + w_chunk * 16 + (BITS == 4 ? sub * 4 : (sub & 1) * 8 + h * 4);
    constexpr uint32_t kQ = BITS == 4 ? 16 : 32;  // distance of the words, by exclusive or
    const uint32_t s_rel = I::kFp4 ? nt * 128 + c8 * 16 + 4 * (sub >> 1) + 2 * h + (sub & 1)
                                   : nt * 128 + c8 * 16 + (2 * sub + h) * 2;
    const uint32_t z_rel = Cfg::kSBytes + (I::kZpF ? nt * 128 + c8 * 16 + (2 * sub + h) * 2 : nt * 8 * BITS + c8 * BITS);
    // of the zero-point within its word(s): column c8 + 8 (2 sub + h)
    const uint32_t z_shift = BITS == 4 ? 4 * (sub + 4 * h) : 8 * (2 * h + (sub & 1));
    const uint32_t a_tmem = tmem_base + ((uint32_t)(quad * 32) << 16) + Cfg::kACol;
    // scale rows of this warp's four k-tiles within the round's copy
    const bool one_row = (gb & 3) == 0;  // the same for all four (a step begins at a multiple of four)
    const bool fixed_row = (gb & 7) == 0 || (8 % gb) == 0;  // the same in every round: gb a multiple of 8, or 1, 2, 4
    const int row_shift = min(__ffs(gb) - 1, 3);
    // A round's place for converted weights is free once the MMAs of the round kARing before have retired: `gone`
    // walks the barriers that say so, starting before the first pass (parity 1).  Parities are never ambiguous: the
    // MMAs retire in order, and with no more groups than kTokRing a group has waited before for the MMAs of the pass
    // before.
    Ring<WD> wr;
    Ring<RING> ring, gone;
    Ring<ARING> a_ring;
    wr.i = ring.i = group;
    a_ring.i = group % ARING;
    gone.i = group < ARING ? group - ARING + RING : group - ARING;
    gone.ph = group < ARING ? 1 : 0;
    int first = group;  // rounds of the next segment before this group's first one
    bool ok = true;
    while (ok && sched.next(sg)) {
      const bool live = (sg.n_tile * CG + (int)rank) * 2 + nt < NT;
      int r = sg.r0 + first;
      for (; r < sg.r1; r += GROUPS) {
        const uint32_t szslot = sz_base + wr.i * Cfg::kSZBytes;
        if (!(ok = mbar_wait<false>(full_w(wr.i), wr.ph, (3 << 8) | 1, cta_abort, p.error))) break;
        // k-tile i of a step: pairs of rows (0, 1) (2, 3) .. (14, 15)
        auto convert_step = [&](int st, uint32_t (&f)[32], auto scaled_c) {
          constexpr bool kScaled = decltype(scaled_c)::value;
          const uint32_t wslot = w_base + wr.i * Cfg::kWBytes + st * (8 * Cfg::kTileBytes) + w_rel;
          uint32_t w[16], sc[4], zr[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) w[4 * i + q] = lds32((wslot ^ (q * kQ)) + i * (2 * Cfg::kTileBytes));
          auto load_row = [&](int i) {
            const int rkt = 4 * st + i;
            if constexpr (I::kFp4) {
              // 16 bytes per (tile, c8) of a pair of groups; this k-tile's group is half of them
              const uint32_t pair = F == kNV4 ? rkt >> 1 : st, half = F == kNV4 ? rkt & 1 : (rkt >> 1) & 1;
              sc[i] = lds8(szslot + s_rel + pair * 256 + half * 8);
            } else {
              const int row = fixed_row ? rkt >> row_shift : (r * kRoundTiles + rkt) / gb - (r * kRoundTiles) / gb;
              if constexpr (kScaled) sc[i] = lds16(szslot + s_rel + row * Cfg::kSRow);
              if constexpr (I::kZpF) zr[i] = lds16(szslot + z_rel + row * Cfg::kZRow);
              if constexpr (I::kZp) zr[i] = lds32(szslot + z_rel + row * Cfg::kZRow + (BITS == 8 ? (sub >> 1) * 4 : 0));
            }
          };
          if constexpr (I::kFp4) {
#pragma unroll
            for (int i = 0; i < 4; ++i) load_row(i);
          } else if constexpr (kScaled || I::kZp || I::kZpF) {
            load_row(0);
            if (one_row) {
#pragma unroll
              for (int i = 1; i < 4; ++i) { sc[i] = sc[0]; zr[i] = zr[0]; }
            } else {
#pragma unroll
              for (int i = 1; i < 4; ++i) load_row(i);
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint32_t z = 0, s = 0, zs = 0;
            if constexpr (I::kZp) z = (zr[i] >> z_shift) & (BITS == 4 ? 15u : 255u);
            const Offset<T, F> off = make_offset<T, F>(z);
            if constexpr (kScaled) {
              if constexpr (I::kFp4) s = fp4_scale<T, F>(sc[i] | (sc[i] << 16));
              else s = dup_lo(sc[i]);
              // q * s - zp * s with the product zp * s rounded, one fma per pair (as gemm_lookup.cuh)
              if constexpr (I::kZpF) zs = Pair<T>::mul(dup_lo(zr[i]), s) ^ 0x80008000u;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t lo, hi;
              convert_word<T, F>(w[4 * i + q], h8, off, lo, hi);
              if constexpr (kScaled) {
                lo = I::kZpF ? Pair<T>::fma(lo, s, zs) : Pair<T>::mul(lo, s);
                hi = I::kZpF ? Pair<T>::fma(hi, s, zs) : Pair<T>::mul(hi, s);
              } else if constexpr (F == kF8) {
                // true magnitude before the MMA (exact); the epilogue takes the factor out of the scale
                lo = Pair<T>::mul(lo, Fp8Cvt<T>::kRebias);
                hi = Pair<T>::mul(hi, Fp8Cvt<T>::kRebias);
              }
              f[8 * i + q] = lo;
              f[8 * i + 4 + q] = hi;
            }
          }
        };
        auto convert = [&](int st, uint32_t (&f)[32]) {
          if constexpr (I::kFp4 || I::kZpF) {
            convert_step(st, f, std::true_type{});
          } else if constexpr (SUMS) {
            convert_step(st, f, std::false_type{});
          } else {
            if (p.channelwise) convert_step(st, f, std::false_type{});
            else convert_step(st, f, std::true_type{});
          }
        };
        // The slot of the packed words goes back once every lane has read its words: the fence orders a lane's reads
        // before the copy that refills the slot (generic and async proxy), the warp barrier and the release of the
        // arrival carry that from all lanes to the producer, whose wait acquires it.
        auto give_back = [&]() {
          fence_proxy_async_smem();
          __syncwarp();
          mbar_arrive(empty_w(wr.i), lane);
        };
        // converted words wait in registers until the MMAs have read what was in their place
        auto wait_empty = [&]() { return mbar_wait<kPair>(empty(gone.i), gone.ph, (3 << 8) | 4, cta_abort, p.error); };
        auto have = [&](int st) { return live && 2 * r + st < steps; };  // a K of an odd number of steps ends with a round of one
        if constexpr (Cfg::kHoldRound) {
          uint32_t f0[32], f1[32];
          const bool mine0 = have(0), mine1 = have(1);
          if (mine0) convert(0, f0);
          if (mine1) convert(1, f1);
          give_back();
          if (!(ok = wait_empty())) break;
          tc_fence_after();
          if (mine0) tmem_st32(a_tmem + a_ring.i * 64, f0);
          if (mine1) tmem_st32(a_tmem + a_ring.i * 64 + 32, f1);
          tmem_st_wait();
          tc_fence_before();
        } else if constexpr (Cfg::kInTmem) {
#pragma unroll 1
          for (int st = 0; st < 2; ++st) {
            uint32_t f[32];
            const bool mine = have(st);
            if (mine) convert(st, f);
            if (st == 1) {
              give_back();
            } else {
              if (!(ok = wait_empty())) break;
              tc_fence_after();
            }
            if (mine) tmem_st32(a_tmem + a_ring.i * 64 + st * 32, f);
          }
          if (!ok) break;
          tmem_st_wait();
          tc_fence_before();
        } else {
          // By fragments: a thread takes the words of a lane of the packed layout, k-tile `kt` of both steps, column tile
          // `fnt`, and a warp stores a 16 x 16 sub-tile with one stmatrix: half the reads and a quarter of the stores of the
          // form by columns, which made 256 tokens 1200 cycles a round instead of 1035.
          constexpr int NW = BITS == 4 ? 4 : 8;
          const int fc8 = lane >> 2, kt = warp & 3, fnt = (warp >> 2) & 1;
          const bool flive = (sg.n_tile * CG + (int)rank) * 2 + fnt < NT;
          // The fragments of a 16 x 16 sub-tile are four 8 x 8 matrices (k lo and hi of columns 0-7, of columns 8-15):
          // one stmatrix.  This lane's row of it: matrix lane / 8, column lane % 8, a 16-byte chunk of a 128 B row.
          const uint32_t b_rel = (fnt * 64 + (lane & 7) + 8 * (lane >> 4)) * 128 + (((2 * kt + ((lane >> 3) & 1)) ^ (lane & 7)) << 4);
          // the lane's words within the k-tile's rows of 128 bytes, 16-byte chunks exchanged with the row's number
          const uint32_t f_row = fnt * (Cfg::kTileBytes / 128) + lane * BITS / 32;
          const uint32_t f_chunk = (BITS == 4 ? lane & 7 : (lane & 3) * 2) ^ (f_row & 7);
          const uint32_t fw_rel = kt * (2 * Cfg::kTileBytes) + f_row * 128 + f_chunk * 16;
          // packed words of the lane, [sub] (4-bit) or [2 sub + block] (8-bit), scales and zero-points of the
          // two tiles
          uint32_t w2[2][NW], sc2[2][4] = {}, zr2[2][4] = {};
#pragma unroll
          for (int st = 0; st < 2; ++st) {
#pragma unroll
            for (int v = 0; v < BITS / 4; ++v) {
              const uint4 w4 = lds128((w_base + wr.i * Cfg::kWBytes + fw_rel + st * (8 * Cfg::kTileBytes)) ^ (v * 16));
              w2[st][4 * v] = w4.x; w2[st][4 * v + 1] = w4.y; w2[st][4 * v + 2] = w4.z; w2[st][4 * v + 3] = w4.w;
            }
            const int rkt = 4 * st + kt;
            if constexpr (I::kFp4) {
              // 16 bytes per (tile, c8) of a pair of groups; this k-tile's group is half of them
              const uint32_t pair = F == kNV4 ? rkt >> 1 : st, half = F == kNV4 ? rkt & 1 : (rkt >> 1) & 1;
              const uint32_t src = szslot + pair * 256 + fnt * 128 + fc8 * 16 + half * 8;
              sc2[st][0] = lds32(src);
              sc2[st][1] = lds32(src + 4);
            } else {
              const int row = fixed_row ? rkt >> row_shift : (r * kRoundTiles + rkt) / gb - (r * kRoundTiles) / gb;
              if (!SUMS && !p.channelwise) {
                const uint4 s4 = lds128(szslot + row * Cfg::kSRow + fnt * 128 + fc8 * 16);
                sc2[st][0] = s4.x; sc2[st][1] = s4.y; sc2[st][2] = s4.z; sc2[st][3] = s4.w;
              }
              if constexpr (I::kZp) {
                const uint32_t zsrc = szslot + Cfg::kSBytes + row * Cfg::kZRow + fnt * (8 * BITS) + fc8 * BITS;
                zr2[st][0] = lds32(zsrc);
                if (BITS == 8) zr2[st][1] = lds32(zsrc + 4);
              }
              if constexpr (I::kZpF) {
                const uint4 z4 = lds128(szslot + Cfg::kSBytes + row * Cfg::kZRow + fnt * 128 + fc8 * 16);
                zr2[st][0] = z4.x; zr2[st][1] = z4.y; zr2[st][2] = z4.z; zr2[st][3] = z4.w;
              }
            }
          }
          give_back();
          if (!(ok = wait_empty())) break;
          if (flive) {
            const uint32_t b0 = a_base + a_ring.i * 2 * Cfg::kABytes + b_rel;
#pragma unroll
            for (int st = 0; st < 2; ++st) {
              if (2 * r + st >= steps) break;  // the last round of an odd number of steps
              const uint32_t b = b0 + st * Cfg::kABytes;
              const uint32_t (&w)[NW] = w2[st];
              const uint32_t (&sc)[4] = sc2[st];
              const uint32_t (&zr)[4] = zr2[st];
              auto convert = [&](auto sub_c, auto scaled_c) {
                constexpr int sub = decltype(sub_c)::value;
                // columns c8 + 16 sub (f[0], f[1]: k lo and hi) and + 8 (f[2], f[3])
                uint32_t f[4], z[2] = {0, 0};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  if constexpr (I::kZp) z[h] = BITS == 4 ? (zr[0] >> (4 * (sub + 4 * h))) & 15u
                                                         : (zr[sub >> 1] >> (8 * (2 * h + (sub & 1)))) & 255u;
                  convert_word<T, F>(BITS == 4 ? w[sub] : w[2 * sub + h], BITS == 4 ? 8 * h : 0, make_offset<T, F>(z[h]),
                                     f[2 * h], f[2 * h + 1]);
                }
                if constexpr (decltype(scaled_c)::value) {
                  uint32_t s_lo, s_hi;
                  if constexpr (I::kFp4) {
                    // byte 4 (sub / 2) + 2 h + sub % 2 of the lane's eight belongs to column c8 + 16 sub + 8 h
                    s_lo = fp4_scale<T, F>(__byte_perm(sc[sub >> 1], 0, sub & 1 ? 0x4141 : 0x4040));
                    s_hi = fp4_scale<T, F>(__byte_perm(sc[sub >> 1], 0, sub & 1 ? 0x4343 : 0x4242));
                  } else {
                    s_lo = dup_lo(sc[sub]);
                    s_hi = dup_hi(sc[sub]);
                  }
                  if constexpr (I::kZpF) {
                    // q * s - zp * s with the product zp * s rounded, one fma per pair (as gemm_lookup.cuh)
                    const uint32_t z_lo = Pair<T>::mul(dup_lo(zr[sub]), s_lo) ^ 0x80008000u;
                    const uint32_t z_hi = Pair<T>::mul(dup_hi(zr[sub]), s_hi) ^ 0x80008000u;
                    f[0] = Pair<T>::fma(f[0], s_lo, z_lo);
                    f[1] = Pair<T>::fma(f[1], s_lo, z_lo);
                    f[2] = Pair<T>::fma(f[2], s_hi, z_hi);
                    f[3] = Pair<T>::fma(f[3], s_hi, z_hi);
                  } else {
                    f[0] = Pair<T>::mul(f[0], s_lo);
                    f[1] = Pair<T>::mul(f[1], s_lo);
                    f[2] = Pair<T>::mul(f[2], s_hi);
                    f[3] = Pair<T>::mul(f[3], s_hi);
                  }
                } else if constexpr (F == kF8) {
                  // true magnitude before the MMA (exact); the epilogue takes the factor out of the scale
#pragma unroll
                  for (int i = 0; i < 4; ++i) f[i] = Pair<T>::mul(f[i], Fp8Cvt<T>::kRebias);
                }
                stmatrix_x4_off<sub * 2048>(b, f);
              };
              auto convert_all = [&](auto scaled_c) {
                convert(std::integral_constant<int, 0>{}, scaled_c);
                convert(std::integral_constant<int, 1>{}, scaled_c);
                convert(std::integral_constant<int, 2>{}, scaled_c);
                convert(std::integral_constant<int, 3>{}, scaled_c);
              };
              if constexpr (I::kFp4 || I::kZpF) {
                convert_all(std::true_type{});
              } else {
                if (p.channelwise) convert_all(std::false_type{});
                else convert_all(std::true_type{});
              }
            }
          }
          fence_proxy_async_smem();  // generic-proxy stores -> visible to the tensor core
        }
        __syncwarp();
        mbar_arrive(full(ring.i), lane);
        wr.template next<GROUPS>();
        ring.template next<GROUPS>();
        gone.template next<GROUPS>();
        a_ring.template next<GROUPS>();
      }
      first = r - sg.r1;
    }
  } else {
    if constexpr (SUMS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(Cfg::kEpiRegs));
    else if constexpr (Cfg::kSplitRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(Cfg::kEpiRegs));
    // ================= epilogue: TMEM -> registers -> C ==================================
    const int quad = warp & 3;  // TMEM lanes 32 quad .. 32 quad + 31
    const uint32_t te0 = kPair ? mapa(tmem_empty(0), 0) : tmem_empty(0);
    uint16_t* C = static_cast<uint16_t*>(p.c);
    int acc_i = 0;  // buffers read so far
    bool ok = true;
    // C, the partial sums and the counters may still be in use by the kernel in front
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    while (ok && sched.next(sg)) {
      const int n = (sg.n_tile * CG + (int)rank) * kBN + quad * 32 + lane;  // this lane's output column
      const bool n_ok = n < p.n;                                            // uniform per warp: N % 64 == 0
      const uint32_t lanes = tmem_base + ((uint32_t)(quad * 32) << 16);
      uint32_t taddr = 0;
      // wait for the next buffer
      auto take = [&]() {
        const int buf = acc_i % BUFS;
        if (!(ok = mbar_wait<kPair, SUMS ? 0 : 100>(tmem_full(buf), (acc_i / BUFS) & 1, (4 << 8) | 4, cta_abort, p.error))) return;
        ++acc_i;
        tc_fence_after();
        taddr = lanes + buf * kBufCols;
      };
      float cs = 1.f, bs = 0.f;
      if (n_ok) {
        if (!SUMS && p.channelwise)
          cs = Pair<T>::to_float(static_cast<const uint16_t*>(p.scales)[(size_t)sg.expert * p.s_stride + single_perm_pos(n)]) *
               p.chan_factor;
        if (F == kNV4) cs = Pair<T>::to_float(*static_cast<const uint16_t*>(p.global_scale));
        if (p.bias)
          bs = Pair<T>::to_float(static_cast<const uint16_t*>(p.bias)[(size_t)sg.expert * p.bias_stride + single_perm_pos(n)]);
      }
      // Scale, bias, rounding and store of COUNT (16 or 32) consecutive tokens of the warp's 32 columns.  Lanes pair
      // up: of two neighbouring tokens the even lane stores the first for both lanes' columns, the odd
      // lane the second, so that a store instruction writes 64 B of two rows.
      // (No test inside the loops: with one per token 32 tokens took 1160 cycles, and the last tile's are exposed.)
      auto store = [&](int t0, auto& v, auto count_c) {
        constexpr int COUNT = decltype(count_c)::value;
        int my_id = 0;
        float my_w = 1.f;
#pragma unroll
        for (int t = 0; t < COUNT; ++t) v[t] = v[t] * cs + bs;
        if (p.ids) {
          my_id = lane < COUNT && t0 + lane < sg.rows ? p.ids[sg.tok0 + t0 + lane] : p.out_rows;
          if (p.row_weights && my_id < p.out_rows) my_w = p.row_weights[my_id];
#pragma unroll
          for (int t = 0; t < COUNT; ++t) v[t] *= __shfl_sync(~0u, my_w, t);
        }
        const bool odd = lane & 1;
        uint32_t word[COUNT / 2];
#pragma unroll
        for (int t = 0; t < COUNT / 2; ++t) word[t] = Pair<T>::pack(v[2 * t], v[2 * t + 1]);
        const uint32_t pick = odd ? 0x3276u : 0x5410u;
#pragma unroll
        for (int t = 0; t < COUNT / 2; ++t) word[t] = __byte_perm(word[t], __shfl_xor_sync(~0u, word[t], 1), pick);
        const int t1 = t0 + (odd ? 1 : 0);
        if (!p.scatter) {
          uint16_t* dst = C + (size_t)(sg.tok0 + t1) * p.n + (n & ~1);
          const size_t step2 = (size_t)2 * p.n;
          if (t0 + COUNT <= sg.rows) {
#pragma unroll
            for (int t = 0; t < COUNT; t += 2, dst += step2) *reinterpret_cast<uint32_t*>(dst) = word[t / 2];
          } else {
#pragma unroll
            for (int t = 0; t < COUNT; t += 2, dst += step2)
              if (t1 + t < sg.rows) *reinterpret_cast<uint32_t*>(dst) = word[t / 2];
          }
        } else {
#pragma unroll
          for (int t = 0; t < COUNT; t += 2) {
            const int id = __shfl_sync(~0u, my_id, t + (odd ? 1 : 0));
            if (t1 + t < sg.rows && id < p.out_rows)
              *reinterpret_cast<uint32_t*>(C + (size_t)id * p.n + (n & ~1)) = word[t / 2];
          }
        }
      };
      auto release = [&]() {  // the buffer taken last, with the REL - 1 before it
        if (acc_i % REL != 0) return;
        const int half = (acc_i / REL - 1) & 1;
        tc_fence_before();
        __syncwarp();
        if (!kPair || rank == 0) {
          mbar_arrive(tmem_empty(half), lane);
        } else if (lane == 0) {
          mbar_arrive_cluster(te0 + 8 * half);
        }
      };
      const size_t slot_floats = (size_t)p.tn * kBN;  // partial sums, token-major: a warp writes 128 B per token
      float* mine = p.partials + ((size_t)sg.slot * CG + rank) * slot_floats + quad * 32 + lane;
      if constexpr (!SUMS) {
        take();
        if (!ok) break;
        for (int t0 = 0; t0 < sg.rows; t0 += 32) {
          uint32_t r[32];
          tmem_ld32(taddr + t0, r);
          tmem_ld_wait();
          if (!sg.shared) {
            if (n_ok) {
              float v[32];
#pragma unroll
              for (int t = 0; t < 32; ++t) v[t] = __uint_as_float(r[t]);
              store(t0, v, std::integral_constant<int, 32>{});
            }
          } else {
#pragma unroll
            for (int t = 0; t < 32; ++t)
              if (t0 + t < sg.rows) __stcg(mine + (size_t)(t0 + t) * kBN, __uint_as_float(r[t]));
          }
        }
        release();
      } else {
        // scale x group sums into the running sums, a group at a time.  The two warps of a quadrant take the lower
        // and the upper tokens.  The scales come four groups at a time through a ring of sixteen groups in shared
        // memory: registers that wait for a load are not to spare here (one spilled costs the load's latency).
        const int step0 = 2 * sg.r0, step1 = min(steps, 2 * sg.r1);
        const int g0 = step0 / group_steps, groups = (step1 - 1) / group_steps + 1 - g0;
        const uint32_t s_ring = bars + Cfg::kBarBytes + (warp - kEpiWarp0) * Cfg::kEpiWarpBytes;
        const uint32_t s_mine = s_ring + ((n & 7) * 8 + ((n >> 3) & 7)) * 2;  // this lane's column in a row
        auto fetch = [&](int c0) {  // groups c0 .. c0 + 3, a lane 16 bytes
          const int c = c0 + (lane >> 3);
          if (n_ok && c < groups)
            cp_async16(s_ring + (c & 15) * 128 + (lane & 7) * 16,
                       static_cast<const uint16_t*>(p.scales) + ((size_t)sg.expert * p.groups + g0 + c) * p.n + (n & ~63) + (lane & 7) * 8);
          cp_async_commit();
        };
        const int half = (sg.rows + 31) / 32 * 16;
        const int t_lo = warp >= kEpiWarp0 + 4 ? half : 0, t_hi = min(sg.rows, t_lo + half);
        constexpr int BLOCKS = CG == 1 ? 2 : 5;  // of 16 tokens
        static_assert(BLOCKS * 32 >= (int)kBufCols, "tokens of a warp");
        float2 acc[8 * BLOCKS];  // the running sums, two tokens each
#pragma unroll
        for (int t = 0; t < 8 * BLOCKS; ++t) acc[t] = make_float2(0.f, 0.f);
        // NB: blocks of 16 tokens, a constant so that a block's load runs while the block before is added (with a test
        // per block eight experts at 500 tokens took 578 us, 514 without).  The buffer goes back as soon as its last
        // values are in registers.
        auto all_groups = [&](auto nb_c) {
          constexpr int NB = decltype(nb_c)::value;
          for (int c = 0; c < groups; ++c) {
            if (c % 4 == 0) {
              fetch(c + 12);  // (their places were last read four groups ago)
              cp_async_wait<3>();
              __syncwarp();
            }
            const uint32_t code = lds16(s_mine + (c & 15) * 128);
            take();
            if (!ok) return;
            const float scale = Pair<T>::to_float((uint16_t)code);
            const float2 s2 = make_float2(scale, scale);
            uint32_t r[2][16];
            if constexpr (NB > 0) tmem_ld16(taddr + t_lo, r[0]);
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              tmem_ld_wait();
              if (b + 1 < NB) tmem_ld16(taddr + t_lo + 16 * (b + 1), r[(b + 1) & 1]);
              else release();
#pragma unroll
              for (int t = 0; t < 8; ++t) acc[8 * b + t] = __ffma2_rn(s2, make_float2(__uint_as_float(r[b & 1][2 * t]), __uint_as_float(r[b & 1][2 * t + 1])),
                                             acc[8 * b + t]);
            }
            if constexpr (NB == 0) release();
          }
        };
        fetch(0);
        fetch(4);
        fetch(8);
        switch (t_hi > t_lo ? (t_hi - t_lo + 15) >> 4 : 0) {
          case 0: all_groups(std::integral_constant<int, 0>{}); break;
          case 1: all_groups(std::integral_constant<int, 1>{}); break;
          case 2: all_groups(std::integral_constant<int, 2>{}); break;
          case 3: all_groups(std::integral_constant<int, BLOCKS < 3 ? BLOCKS : 3>{}); break;
          case 4: all_groups(std::integral_constant<int, BLOCKS < 4 ? BLOCKS : 4>{}); break;
          default: all_groups(std::integral_constant<int, BLOCKS>{});
        }
        cp_async_wait<0>();
        __syncwarp();
        if (!ok) break;
        auto finish16 = [&](int t0, float (&v)[16]) {
          if (!sg.shared) {
            if (n_ok) store(t0, v, std::integral_constant<int, 16>{});
          } else {
#pragma unroll
            for (int t = 0; t < 16; ++t)
              if (t0 + t < sg.rows) __stcg(mine + (size_t)(t0 + t) * kBN, v[t]);
          }
        };
#pragma unroll
        for (int b = 0; b < BLOCKS; ++b) {
          if (t_lo + 16 * b >= t_hi) break;
          float v[16];
#pragma unroll
          for (int t = 0; t < 16; ++t) v[t] = t & 1 ? acc[8 * b + t / 2].y : acc[8 * b + t / 2].x;
          finish16(t_lo + 16 * b, v);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  // no CTA of the pair may leave while the other may still arrive on its barriers or read its memory
  if (kPair) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc<CG>(tmem_base, kTmemCols);
  }
}

}  // namespace tc
}  // namespace b200q
