// Checkpoint-format -> Marlin tile layout re-tiling, and the activation column
// gather used by act-order.  Pure integer / byte movement: HBM-bound.
//
// Output layout (int32 [K/16, N*16/pf]): for k-tile kt and 64-column tile nt the
// tile's words are contiguous at ((kt * N/64) + nt) * W, W = 128 (4-bit) or 256
// (8-bit).  Inside a tile, lane = 4*c + q (c = 0..7, q = 0..3) owns column c
// (+8 for block 1) of each 16-column sub-tile `sub` and rows 2q + {0,1,8,9}:
//   4-bit: word lane*4 + sub, nibble t holds (row, block) =
//          t:0 (2q,0) 1 (2q+8,0) 2 (2q,1) 3 (2q+8,1) 4 (2q+1,0) 5 (2q+9,0) 6 (2q+1,1) 7 (2q+9,1)
//   8-bit: word lane*8 + sub*2 + block, byte t holds row 2q + {0, 8, 1, 9}[t]
#include "common.cuh"

namespace b200q {

namespace {

constexpr int kRepackThreads = 256;

// N neighbouring words; one vector store where the base allows it (`vec`: 16-byte aligned buffer)
template <int N>
__device__ __forceinline__ void store_words(uint32_t* dst, const uint32_t* v, bool vec) {
  if (vec) {
    if constexpr (N == 4) *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
    else *reinterpret_cast<uint2*>(dst) = make_uint2(v[0], v[1]);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) dst[i] = v[i];
  }
}
__device__ __forceinline__ bool aligned16(const void* p) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// ---- one k-tile, one column per lane --------------------------------------------------------
// A lane that owns column n of a k-tile (16 rows) contributes to the four q-words of that
// column.  Row r = 2q + e + 8h sits at bit kPos(r): the code is rotated there and merged with
// one and-or, so a code costs two instructions once its packed word is in a register.
template <int BITS>
__device__ __forceinline__ constexpr int row_pos(int r) {
  return 16 * (r & 1) + BITS * (r >> 3);  // 4-bit: nibble 4e + h; 8-bit: byte 2e + h
}
template <int BITS>
__device__ __forceinline__ void merge_row(uint32_t (&acc)[4], int r, uint32_t word, uint32_t rot) {
  const uint32_t mask = ((1u << BITS) - 1) << row_pos<BITS>(r);
  acc[(r & 7) >> 1] |= __funnelshift_r(word, word, rot) & mask;
}

// Lanes hold 32 neighbouring columns (lane = c + 8 block + 16 s): 4 x 4 exchange between the
// lanes of a column c, after which lane (block, s) owns the words of q = 2 block + s.
// 4-bit: out[0..1] = words of sub-tiles (0, 1) of the 32 columns (both blocks merged);
// 8-bit: out[0..3] = words (sub 0 block 0), (0, 1), (1, 0), (1, 1).
template <int BITS>
__device__ __forceinline__ void exchange32(const uint32_t (&acc)[4], int lane,
                                           uint32_t (&out)[BITS == 4 ? 2 : 4]) {
  const bool b = lane & 8, s = lane & 16;
  const uint32_t k0 = b ? acc[2] : acc[0], k1 = b ? acc[3] : acc[1];
  const uint32_t r0 = __shfl_xor_sync(~0u, b ? acc[0] : acc[2], 8);
  const uint32_t r1 = __shfl_xor_sync(~0u, b ? acc[1] : acc[3], 8);
  if constexpr (BITS == 4) {
    // the other column block's nibbles: block 1 sits 8 bits above block 0
    const uint32_t f0 = b ? (k0 << 8) | r0 : k0 | (r0 << 8);
    const uint32_t f1 = b ? (k1 << 8) | r1 : k1 | (r1 << 8);
    const uint32_t keep = s ? f1 : f0;
    const uint32_t recv = __shfl_xor_sync(~0u, s ? f0 : f1, 16);
    out[0] = s ? recv : keep;
    out[1] = s ? keep : recv;
  } else {
    // (block 0, block 1) words of this lane's sub-tile for q = 2b and 2b + 1
    const uint32_t q0[2] = {b ? r0 : k0, b ? k0 : r0}, q1[2] = {b ? r1 : k1, b ? k1 : r1};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t keep = s ? q1[i] : q0[i];
      const uint32_t recv = __shfl_xor_sync(~0u, s ? q0[i] : q1[i], 16);
      out[i] = s ? recv : keep;
      out[2 + i] = s ? keep : recv;
    }
  }
}

// GPTQ layout without a permutation: a warp takes a (k-tile, 64-column tile) at a time, lane =
// column (and column + 32).  Loads are 128 B rows, stores the tile's contiguous 512 B / 1 KB.
// Bound by HBM.
template <int BITS>
__global__ void __launch_bounds__(kRepackThreads)
gptq_repack_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int n_tiles,
                   long long units) {
  constexpr int PF = 32 / BITS;
  constexpr int ROWS = 16 / PF;  // packed rows of a k-tile
  constexpr int U = 4;           // units in flight per warp
  const int lane = threadIdx.x & 31;
  const int size_n = n_tiles * 64;
  const long long u0 = ((long long)blockIdx.x * (kRepackThreads / 32) + (threadIdx.x >> 5)) * U;
  uint32_t w[U][ROWS][2];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u0 + u >= units) break;
    const long long kt = (u0 + u) / n_tiles;
    const uint32_t* src = in + kt * ROWS * size_n + ((u0 + u) - kt * n_tiles) * 64 + lane;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      w[u][r][0] = __ldcs(src + (size_t)r * size_n);
      w[u][r][1] = __ldcs(src + (size_t)r * size_n + 32);
    }
  }
  const int c = lane & 7, q = 2 * ((lane >> 3) & 1) + (lane >> 4);
  const bool vec = aligned16(out);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u0 + u >= units) break;
    uint32_t o[2][BITS == 4 ? 2 : 4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t acc[4] = {0, 0, 0, 0};
#pragma unroll
      for (int r = 0; r < 16; ++r)
        merge_row<BITS>(acc, r, w[u][r / PF][half], ((r % PF) * BITS - row_pos<BITS>(r)) & 31);
      exchange32<BITS>(acc, lane, o[half]);
    }
    uint32_t* dst = out + (u0 + u) * (16 * 64 / PF) + (4 * c + q) * BITS;
#pragma unroll
    for (int j = 0; j < BITS / 4; ++j) store_words<4>(dst + 4 * j, &o[0][0] + 4 * j, vec);
  }
}

// words of an 8 x 8 nibble (4 x 4 byte) block -> its transpose: w'[i] element j = w[j] element i
template <int BITS>
__device__ __forceinline__ void transpose_codes(uint32_t (&w)[32 / BITS]) {
  constexpr int N = 32 / BITS;
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {  // 16-bit halves
    const uint32_t a = w[i], b = w[i + N / 2];
    w[i] = __byte_perm(a, b, 0x5410);
    w[i + N / 2] = __byte_perm(a, b, 0x7632);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {  // bytes
    if (i & (N / 4)) continue;
    const uint32_t a = w[i], b = w[i + N / 4];
    w[i] = __byte_perm(a, b, 0x6240);
    w[i + N / 4] = __byte_perm(a, b, 0x7351);
  }
  if constexpr (BITS == 4) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {  // nibbles
      const uint32_t a = w[i], b = w[i + 1], m = 0x0f0f0f0fu;
      w[i] = (a & m) | ((b << 4) & ~m);
      w[i + 1] = ((a >> 4) & m) | (b & ~m);
    }
  }
}

// GPTQ layout with the rows in act-order: output row k comes from packed row perm[k] / PF, so
// every packed row is needed by as many k-tiles as it holds codes (fetching it from L2 each time:
// 248 us for 4096 x 28672 4-bit on B200).  A CTA brings all packed rows of C columns on chip
// once, transposes blocks of PF rows x PF columns so that a word holds PF neighbouring columns of
// ONE row, and keeps that row-major panel in shared memory; thread (k-tile, q) then fetches its
// four rows in whole vectors and a second transpose yields the words of the eight columns c.
// Two transposes cost one instruction per code; picking single codes out of the packed words
// (ten instructions per code with addresses) made the same traffic issue-bound at 55 us.
// blockIdx.x = panel, blockIdx.y = share of the k-tiles (more than one only when there are
// too few panels to fill the GPU).
template <int BITS, int C>
struct PanelCfg {
  static constexpr int PF = 32 / BITS;
  static constexpr int kRowWords = C / PF;
  // one row's worth of padding per PF rows: the stores of a transposed block hit distinct banks
  static __host__ __device__ constexpr long long words(long long k) { return (k + k / PF) * kRowWords; }
};
template <int BITS, int C>
__global__ void __launch_bounds__(kRepackThreads)
gptq_repack_perm_kernel(const uint32_t* __restrict__ in, const int32_t* __restrict__ perm,
                        uint32_t* __restrict__ out, int size_k, int size_n) {
  constexpr int PF = 32 / BITS;
  constexpr int W = 16 * 64 / PF;
  constexpr int RW = PanelCfg<BITS, C>::kRowWords;  // words of a panel row = column groups
  constexpr int SUBS = C / 16;
  extern __shared__ __align__(16) uint32_t panel[];
  const int KT = size_k / 16;
  const int n0 = blockIdx.x * C;
  {
    const int items = size_k / PF * RW;
    const bool vec_in = aligned16(in);
    constexpr int U = 4;  // items in flight per thread
    for (int i0 = threadIdx.x; i0 < items; i0 += U * kRepackThreads) {
      uint32_t w[U][PF];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * kRepackThreads;
        if (i >= items) break;
        const uint32_t* src = in + (size_t)(i / RW) * size_n + n0 + (i % RW) * PF;
#pragma unroll
        for (int j = 0; j < PF; j += 4) {
          const uint4 v = vec_in ? __ldcs(reinterpret_cast<const uint4*>(src + j))
                                 : make_uint4(src[j], src[j + 1], src[j + 2], src[j + 3]);
          w[u][j] = v.x; w[u][j + 1] = v.y; w[u][j + 2] = v.z; w[u][j + 3] = v.w;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * kRepackThreads;
        if (i >= items) break;
        transpose_codes<BITS>(w[u]);
        uint32_t* dst = panel + (i / RW) * ((PF + 1) * RW) + i % RW;
#pragma unroll
        for (int j = 0; j < PF; ++j) dst[j * RW] = w[u][j];
      }
    }
  }
  __syncthreads();

  const int kt0 = (int)((long long)KT * blockIdx.y / gridDim.y);
  const int kt1 = (int)((long long)KT * (blockIdx.y + 1) / gridDim.y);
  const bool vec = aligned16(out);
  uint32_t* tile0 = out + (size_t)(n0 / 64) * W;
  for (int i = threadIdx.x; i < (kt1 - kt0) * 4; i += kRepackThreads) {
    const int kt = kt0 + (i >> 2), q = i & 3;
    uint32_t rows[4][RW];  // rows 2q, 2q + 8, 2q + 1, 2q + 9: the order of the bytes / nibble pairs
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t k = (uint32_t)__ldg(perm + kt * 16 + 2 * q + (r >> 1) + 8 * (r & 1));
      const uint32_t* src = panel + (k + k / PF) * RW;
      if constexpr (RW == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(src);
        rows[r][0] = v.x; rows[r][1] = v.y;
      } else {
#pragma unroll
        for (int j = 0; j < RW; j += 4) {
          const uint4 v = *reinterpret_cast<const uint4*>(src + j);
          rows[r][j] = v.x; rows[r][j + 1] = v.y; rows[r][j + 2] = v.z; rows[r][j + 3] = v.w;
        }
      }
    }
    uint32_t* tile = tile0 + (size_t)kt * (size_n / 64) * W;
    const int sub0 = (n0 >> 4) & 3;
    if constexpr (BITS == 4) {
      // nibble t of a word: row (t & 1) + 2 (t >> 2) of `rows`, column block (t >> 1) & 1
      uint32_t o[SUBS][8];
#pragma unroll
      for (int s = 0; s < SUBS; ++s) {
#pragma unroll
        for (int t = 0; t < 8; ++t) o[s][t] = rows[(t & 1) + 2 * (t >> 2)][2 * s + ((t >> 1) & 1)];
        transpose_codes<4>(o[s]);
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint32_t* dst = tile + (4 * c + q) * 4 + sub0;
        if constexpr (SUBS == 2) {
          const uint32_t v[2] = {o[0][c], o[1][c]};
          store_words<2>(dst, v, vec);
        } else {
          *dst = o[0][c];
        }
      }
    } else {
      // byte t of a word: row t of `rows`; word group 4 sub + 2 block + c / 4 of a row
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        uint32_t o[2 * SUBS][4];
#pragma unroll
        for (int sb = 0; sb < 2 * SUBS; ++sb) {
#pragma unroll
          for (int t = 0; t < 4; ++t) o[sb][t] = rows[t][2 * sb + ch];
          transpose_codes<8>(o[sb]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t v[2 * SUBS];
#pragma unroll
          for (int sb = 0; sb < 2 * SUBS; ++sb) v[sb] = o[sb][c];
          store_words<2 * SUBS>(tile + (4 * (4 * ch + c) + q) * 8 + 2 * sub0, v, vec);
        }
      }
    }
  }
}

// The same for a K whose panel does not fit on chip (4-bit beyond 25824 rows, 8-bit beyond 11616):
// lane = column, 128 B row pieces gathered from global memory / L2 for every k-tile.
template <int BITS>
__global__ void __launch_bounds__(kRepackThreads)
gptq_repack_perm_large_kernel(const uint32_t* __restrict__ in, const int32_t* __restrict__ perm,
                              uint32_t* __restrict__ out, int size_k, int size_n) {
  constexpr int PF = 32 / BITS;
  constexpr int W = 16 * 64 / PF;
  const int lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * 32;
  const bool vec = aligned16(out);
  const int c = lane & 7, q = 2 * ((lane >> 3) & 1) + (lane >> 4), half = (n0 >> 5) & 1;
  for (int kt = blockIdx.y * (kRepackThreads / 32) + (threadIdx.x >> 5); kt < size_k / 16;
       kt += gridDim.y * (kRepackThreads / 32)) {
    uint32_t acc[4] = {0, 0, 0, 0};
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const uint32_t k = (uint32_t)__ldg(perm + kt * 16 + r);
      merge_row<BITS>(acc, r, in[(size_t)(k / PF) * size_n + n0 + lane],
                      ((k % PF) * BITS - row_pos<BITS>(r)) & 31);
    }
    uint32_t o[BITS == 4 ? 2 : 4];
    exchange32<BITS>(acc, lane, o);
    uint32_t* tile = out + ((size_t)kt * (size_n / 64) + n0 / 64) * W;
    store_words<BITS / 2>(tile + (4 * c + q) * BITS + half * (BITS / 2), o, vec);
  }
}

// AWQ layout: a word holds 8 (4) neighbouring columns of one row, interleaved.  A warp stages
// 16 rows x 32 words (128 B rows) in its own piece of shared memory; lane (c, q) then picks the
// codes of its column residue from its four rows (the eight lanes of a q read the same
// addresses).  Column 8w+i of a 4-bit word sits at nibble [0,4,1,5,2,6,3,7][i] (the inverse of
// the format's [0,2,4,6,1,3,5,7] interleave); 8-bit: byte [0,2,1,3][i].  Bound by HBM.
template <int BITS>
__global__ void __launch_bounds__(kRepackThreads)
awq_repack_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int k_tiles,
                  int n_tiles) {
  constexpr int PF = 32 / BITS;
  constexpr int W = 16 * 64 / PF;
  constexpr int TW = 64 / PF;        // words of a row of one 64-column tile: 8, 16
  constexpr int TPW = 32 / TW;       // tiles a warp stages at a time: 4, 2
  constexpr int STRIDE = 36;         // words; keeps 16 B alignment and spreads the four q rows
  __shared__ __align__(16) uint32_t staged[kRepackThreads / 32][16 * STRIDE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (n_tiles + TPW - 1) / TPW;
  const long long unit = (long long)blockIdx.x * (kRepackThreads / 32) + warp;
  if (unit >= (long long)groups * k_tiles) return;
  const int kt = (int)(unit / groups);
  const int nt0 = (int)(unit - (long long)kt * groups) * TPW;
  const int tiles = min(TPW, n_tiles - nt0);
  uint32_t* st = staged[warp];
  {
    // 8 lanes per row, 4 rows per step; a row's tail past the last tile is not read
    const int chunk = lane & 7;
    const uint4* src = reinterpret_cast<const uint4*>(in + (size_t)(kt * 16 + (lane >> 3)) * (n_tiles * TW) +
                                                      nt0 * TW) + chunk;
    uint4 v[4];
    const bool live = chunk * 4 < tiles * TW;
    const bool vec_in = aligned16(in);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (live && vec_in) v[i] = __ldcs(src + (size_t)i * n_tiles * TW);
    if (live && !vec_in) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(src) + (size_t)i * 4 * n_tiles * TW;
        v[i] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (live) *reinterpret_cast<uint4*>(st + (4 * i + (lane >> 3)) * STRIDE + chunk * 4) = v[i];
  }
  __syncwarp();
  const int c = lane >> 2, q = lane & 3;
  const int i = c % PF;
  const uint32_t src_bit = BITS * ((BITS == 4) ? ((i >> 1) + 4 * (i & 1)) : (((i & 1) << 1) | (i >> 1)));
  for (int t = 0; t < tiles; ++t) {
    uint32_t o[BITS];  // the lane's words of the tile: 4 (4-bit), 8
#pragma unroll
    for (int j = 0; j < BITS; ++j) o[j] = 0;
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
      const int e = rr & 1, h = rr >> 1;  // row 2q + e + 8h
      const uint32_t* row = st + (2 * q + e + 8 * h) * STRIDE + t * TW;
      const uint32_t rot = (src_bit - (16 * e + BITS * h)) & 31;
      if constexpr (BITS == 4) {
        const uint4 lo = *reinterpret_cast<const uint4*>(row), hi = *reinterpret_cast<const uint4*>(row + 4);
        const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};  // word 2 sub + block
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int pos = 16 * e + 4 * h + 8 * (j & 1);
          o[j >> 1] |= __funnelshift_r(w[j], w[j], (j & 1) ? rot - 8 : rot) & (0xfu << pos);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {  // word 4 sub + 2 block + c / 4
          const uint32_t w = row[2 * j + (c >> 2)];
          o[j] |= __funnelshift_r(w, w, rot) & (0xffu << (16 * e + 8 * h));
        }
      }
    }
    uint32_t* dst = out + ((size_t)kt * n_tiles + nt0 + t) * W + lane * BITS;
#pragma unroll
    for (int j = 0; j < BITS / 4; ++j) store_words<4>(dst + 4 * j, o + 4 * j, aligned16(out));
  }
}

template <int BITS>
int launch_gptq_repack(const uint32_t* in, const int32_t* perm, uint32_t* out, int64_t size_k,
                       int64_t size_n, cudaStream_t stream) {
  const int n_tiles = (int)(size_n / 64);
  const int64_t k_tiles = size_k / 16;
  if (!perm) {
    const long long units = (long long)k_tiles * n_tiles;
    const long long per_block = kRepackThreads / 32 * 4;
    gptq_repack_kernel<BITS><<<(unsigned)((units + per_block - 1) / per_block), kRepackThreads, 0, stream>>>(
        in, out, n_tiles, units);
    return B200Q_OK;
  }
  const int64_t bytes32 = PanelCfg<BITS, 32>::words(size_k) * 4, bytes16 = PanelCfg<BITS, 16>::words(size_k) * 4;
  // 32 columns while they fit: 128 B row pieces and half as many partial output sectors (K = 8192,
  // 4-bit: 82 us against 113 us with 16 columns, although only one CTA fits an SM)
  const int64_t limit = device_max_smem_optin();
  const int c = bytes32 <= limit ? 32 : bytes16 <= limit ? 16 : 0;
  if (c == 0) {
    const dim3 grid((unsigned)(size_n / 32), (unsigned)((k_tiles + 63) / 64));
    gptq_repack_perm_large_kernel<BITS><<<grid, kRepackThreads, 0, stream>>>(in, perm, out, (int)size_k, (int)size_n);
    return B200Q_OK;
  }
  const int64_t panels = size_n / c;
  // each further share of the k-tiles stages the whole panel again: only while SMs would idle
  int64_t shares = device_sm_count() / panels;
  shares = shares < 1 ? 1 : shares > 8 ? 8 : shares;
  const dim3 grid((unsigned)panels, (unsigned)(shares < k_tiles ? shares : k_tiles));
  const int64_t smem = c == 32 ? bytes32 : bytes16;
  auto kernel = c == 32 ? gptq_repack_perm_kernel<BITS, 32> : gptq_repack_perm_kernel<BITS, 16>;
  if (smem > 48 * 1024)
    B200Q_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kernel<<<grid, kRepackThreads, smem, stream>>>(in, perm, out, (int)size_k, (int)size_n);
  return B200Q_OK;
}

// out[m, k] = a[m, perm[k]].  One block per row (grid-stride); the row is staged
// in shared memory with coalesced 16-byte loads when it fits, so both the read
// and the write of every row are coalesced.
__global__ void __launch_bounds__(256)
permute_cols_kernel(const uint16_t* __restrict__ a, int64_t lda, const int32_t* __restrict__ perm,
                    uint16_t* __restrict__ out, int size_m, int size_k, int stage_in_smem) {
  extern __shared__ __align__(16) uint16_t row_buf[];
  // 16-byte stores and permutation loads need K % 8 == 0 and aligned bases
  const bool vec_out = (size_k % 8 == 0) && ((reinterpret_cast<uintptr_t>(perm) & 15) == 0) &&
                       ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
  // the GEMM that follows may start prefetching its weights right away
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  for (int m = blockIdx.x; m < size_m; m += gridDim.x) {
    const uint16_t* src = a + (size_t)m * lda;
    uint16_t* dst = out + (size_t)m * size_k;
    if (stage_in_smem) {
      // lda % 8 == 0 and a 16 B aligned base make every row 16 B aligned
      const int vecs = size_k / 8;
      for (int i = threadIdx.x; i < vecs; i += blockDim.x)
        reinterpret_cast<uint4*>(row_buf)[i] = reinterpret_cast<const uint4*>(src)[i];
      for (int i = vecs * 8 + threadIdx.x; i < size_k; i += blockDim.x) row_buf[i] = src[i];
      __syncthreads();
      if (vec_out) {
        // eight outputs per thread: two 16-byte loads of the permutation, one 16-byte store
        for (int i = threadIdx.x; i < vecs; i += blockDim.x) {
          const int4 p0 = __ldg(reinterpret_cast<const int4*>(perm) + 2 * i);
          const int4 p1 = __ldg(reinterpret_cast<const int4*>(perm) + 2 * i + 1);
          uint4 v;
          v.x = (uint32_t)row_buf[p0.x] | ((uint32_t)row_buf[p0.y] << 16);
          v.y = (uint32_t)row_buf[p0.z] | ((uint32_t)row_buf[p0.w] << 16);
          v.z = (uint32_t)row_buf[p1.x] | ((uint32_t)row_buf[p1.y] << 16);
          v.w = (uint32_t)row_buf[p1.z] | ((uint32_t)row_buf[p1.w] << 16);
          reinterpret_cast<uint4*>(dst)[i] = v;
        }
      } else {
        for (int k = threadIdx.x; k < size_k; k += blockDim.x) dst[k] = row_buf[perm[k]];
      }
      __syncthreads();
    } else {
      for (int k = threadIdx.x; k < size_k; k += blockDim.x) dst[k] = src[perm[k]];
    }
  }
}

// Few rows (decode): one thread per 8 output elements, many blocks per row, so
// that the gather is spread over the whole GPU; the reads hit L2.
__global__ void __launch_bounds__(256)
permute_cols_small_kernel(const uint16_t* __restrict__ a, int64_t lda,
                          const int32_t* __restrict__ perm, uint16_t* __restrict__ out, int size_k) {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const int m = blockIdx.y;
  const int k0 = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (k0 >= size_k) return;
  const uint16_t* src = a + (size_t)m * lda;
  // the permutation is a constant of the layer: fetch it while the kernel before this one
  // in the stream drains, then wait for that kernel (it produced `a` and may still read `out`)
  const int4 p0 = *reinterpret_cast<const int4*>(perm + k0);
  const int4 p1 = *reinterpret_cast<const int4*>(perm + k0 + 4);
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  uint4 v;
  v.x = (uint32_t)src[p0.x] | ((uint32_t)src[p0.y] << 16);
  v.y = (uint32_t)src[p0.z] | ((uint32_t)src[p0.w] << 16);
  v.z = (uint32_t)src[p1.x] | ((uint32_t)src[p1.y] << 16);
  v.w = (uint32_t)src[p1.z] | ((uint32_t)src[p1.w] << 16);
  *reinterpret_cast<uint4*>(out + (size_t)m * size_k + k0) = v;
}

}  // namespace

int launch_permute_cols(const void* a, int64_t lda, const int32_t* perm, void* out, int64_t size_m,
                        int64_t size_k, cudaStream_t stream) {
  if (size_m == 0 || size_k == 0) return B200Q_OK;
  if (size_m <= 64 && size_k % 8 == 0 && (reinterpret_cast<uintptr_t>(perm) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    dim3 grid((unsigned)((size_k / 8 + 255) / 256), (unsigned)size_m);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    B200Q_CUDA_OK(cudaLaunchKernelEx(&cfg, permute_cols_small_kernel, static_cast<const uint16_t*>(a),
                                     lda, perm, static_cast<uint16_t*>(out), (int)size_k));
    note_launch();
    return B200Q_OK;
  }
  const size_t row_bytes = (size_t)size_k * 2;
  const bool aligned = (lda % 8 == 0) && ((reinterpret_cast<uintptr_t>(a) & 15) == 0);
  int stage = aligned && row_bytes <= (size_t)device_max_smem_optin() - 1024;
  size_t smem = stage ? row_bytes : 0;
  if (smem > 48 * 1024)
    B200Q_CUDA_OK(cudaFuncSetAttribute(permute_cols_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int blocks = (int)(size_m < 4 * (int64_t)device_sm_count() ? size_m : 4 * device_sm_count());
  permute_cols_kernel<<<blocks, 256, smem, stream>>>(
      static_cast<const uint16_t*>(a), lda, perm, static_cast<uint16_t*>(out), (int)size_m,
      (int)size_k, stage);
  note_launch();
  B200Q_CUDA_OK(cudaGetLastError());
  return B200Q_OK;
}

}  // namespace b200q

using namespace b200q;

extern "C" int b200q_gptq_marlin_repack(const uint32_t* b_q_weight, const int32_t* perm,
                                        uint32_t* out, int64_t size_k, int64_t size_n, int num_bits,
                                        b200q_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  B200Q_REQUIRE(num_bits == 4 || num_bits == 8, B200Q_EINVAL, "num_bits must be 4 or 8. Got = %d",
                num_bits);
  B200Q_REQUIRE(size_k >= 0 && size_k % 16 == 0, B200Q_EINVAL,
                "size_k = %lld is not divisible by tile_k_size = 16", (long long)size_k);
  B200Q_REQUIRE(size_n >= 0 && size_n % 64 == 0, B200Q_EINVAL,
                "size_n = %lld is not divisible by tile_n_size = 64", (long long)size_n);
  B200Q_REQUIRE(size_k / 16 <= 65535, B200Q_EUNSUPPORTED, "size_k = %lld too large",
                (long long)size_k);
  if (size_k == 0 || size_n == 0) return B200Q_OK;
  B200Q_REQUIRE(b_q_weight && out, B200Q_EINVAL, "null tensor pointer");
  const int rc = num_bits == 4 ? launch_gptq_repack<4>(b_q_weight, perm, out, size_k, size_n, stream)
                               : launch_gptq_repack<8>(b_q_weight, perm, out, size_k, size_n, stream);
  if (rc != B200Q_OK) return rc;
  note_launch();
  B200Q_CUDA_OK(cudaGetLastError());
  return B200Q_OK;
}

extern "C" int b200q_awq_marlin_repack(const uint32_t* b_q_weight, uint32_t* out, int64_t size_k,
                                       int64_t size_n, int num_bits, b200q_stream_t stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  B200Q_REQUIRE(num_bits == 4 || num_bits == 8, B200Q_EINVAL, "num_bits must be 4 or 8. Got = %d",
                num_bits);
  B200Q_REQUIRE(size_k >= 0 && size_k % 16 == 0, B200Q_EINVAL,
                "size_k = %lld is not divisible by tile_k_size = 16", (long long)size_k);
  B200Q_REQUIRE(size_n >= 0 && size_n % 64 == 0, B200Q_EINVAL,
                "size_n = %lld is not divisible by tile_n_size = 64", (long long)size_n);
  B200Q_REQUIRE(size_k / 16 <= 65535, B200Q_EUNSUPPORTED, "size_k = %lld too large",
                (long long)size_k);
  if (size_k == 0 || size_n == 0) return B200Q_OK;
  B200Q_REQUIRE(b_q_weight && out, B200Q_EINVAL, "null tensor pointer");
  const int n_tiles = (int)(size_n / 64), k_tiles = (int)(size_k / 16);
  const int tiles_per_warp = num_bits == 4 ? 4 : 2;
  const long long warps = (long long)((n_tiles + tiles_per_warp - 1) / tiles_per_warp) * k_tiles;
  const unsigned blocks = (unsigned)((warps + kRepackThreads / 32 - 1) / (kRepackThreads / 32));
  if (num_bits == 4)
    awq_repack_kernel<4><<<blocks, kRepackThreads, 0, stream>>>(b_q_weight, out, k_tiles, n_tiles);
  else
    awq_repack_kernel<8><<<blocks, kRepackThreads, 0, stream>>>(b_q_weight, out, k_tiles, n_tiles);
  note_launch();
  B200Q_CUDA_OK(cudaGetLastError());
  return B200Q_OK;
}

extern "C" int b200q_permute_cols(const void* a, int64_t lda, const int32_t* perm, void* out,
                                  int64_t size_m, int64_t size_k, b200q_stream_t stream) {
  B200Q_REQUIRE(size_m >= 0 && size_k >= 0, B200Q_EINVAL, "negative size");
  if (size_m == 0 || size_k == 0) return B200Q_OK;
  B200Q_REQUIRE(a && perm && out, B200Q_EINVAL, "null tensor pointer");
  B200Q_REQUIRE(lda >= size_k, B200Q_EINVAL, "lda = %lld < size_k = %lld", (long long)lda,
                (long long)size_k);
  return launch_permute_cols(a, lda, perm, out, size_m, size_k, static_cast<cudaStream_t>(stream));
}
