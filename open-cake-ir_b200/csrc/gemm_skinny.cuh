// Block-scaled FP8 (e4m3) GEMM for few rows per group on sm_100a: weights stream through, a handful of tokens stays.
//
// The same products as gemm_fp8.cuh, C[m, n] = sum_kb (sum_{k in kb} A[m, k] B[n, k]) sfa[kb, m] sfb[n/128, kb], for decode
// steps whose groups (experts, or the whole dense problem) have a handful of rows and are few themselves.  What bounds it is
// the weight stream: 2 x 16 rows of products per weight byte at most.  The tcgen05 core takes a tile's K blocks one after
// another (0.25 to 0.4 us each) and 256 columns to a CTA, so a small problem occupies a few SMs for long; from about a tile to an SM
// on its narrow row tiles are the faster ones.  Here every warp is on its own: it streams 32 weight rows
// through a ring of its own (cp.async, one 128-wide K block of weights, token rows and scales per slot, several slots in
// flight, no CTA-wide barrier in the main loop), multiplies with mma.m16n8k32 (weights are the 16 rows, tokens the 8
// columns; exact products, fp32 sums, 1.06 clocks per instruction and SM) into a fresh partial sum per K block and
// promotes that with the block's scales in registers.
//
// A CTA of eight warps covers WM = 8 / WK sub-tiles of 32 weight rows, each by WK warps that take every WK-th K block and
// meet once per item in shared memory (in warp order).  WK = 1 for many groups (a whole 128-feature quantisation group
// of the gate/up product lies in one CTA and is quantised here); WK = 4, 8 where items would not fill the GPU, the
// gate/up result then leaves as fp32 for quantize_kernel.
// K order inside a block is free as long as both operands use the same: lane quad q takes bytes [32 q, 32 q + 32) of a row,
// so that fragments of all four k-steps are two 16-byte shared-memory reads per row instead of eight 4-byte ones.
#pragma once
#include "gemm_fp8.cuh"
#include <climits>
#include <type_traits>

namespace cake {
namespace skinny {

using gemm::kDense;
using gemm::kDown;
using gemm::kGateUp;
constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int kSubRows = 32;                       // weight rows of a warp: two MMA tiles (gate/up: 16 of x1, 16 of x2)
constexpr int kWeightBytes = kSubRows * 128;       // of one K block
constexpr int kMaxGroups = gemm::kMaxGroups;

struct Params {
  const uint8_t* w;            // [groups, w_rows, 128 * k_blocks]
  const float* sw;             // [groups, w_rows / 128, k_blocks]
  const uint8_t* x;            // rows of x_stride bytes
  const float* sx;             // [k_blocks * TERMS, sx_stride]
  const int* row_map;          // sorted row -> pair, token = pair / map_div, which names the row of x and sx (null: the sorted row does)
  const int* offsets;          // [groups + 1] rows before a group (null: one group of dense_rows rows)
  const float* row_weight;     // kDown: route weight of a pair (by row_map_weight)
  const int* weight_map;       // kDown: sorted row -> pair
  void* out;                   // kGateUp: e4m3 [rows, n * terms] (WK = 1) or fp32 [rows, n]; else bf16 [rows, n]
  float* out_scale;            // kGateUp, WK = 1: [n / 128 * terms, row_capacity]
  int* status;                 // status word to clear (null: someone else does); nothing here waits, so nothing ever sets it
  int max_rows;                // groups of more rows are the tcgen05 core's where that pays (0: none are)
  const int* core;             // max_rows > 0: device word that says whether it does
  int n, k_blocks, w_rows, groups, dense_rows, x_stride, sx_stride, map_div, row_capacity, terms;
};

// TERMS: e4m3 terms of a token row (value, residual), one row of k_blocks after the other; a weight block meets both.
template <int NT, int WK, int TERMS>
struct Shape {
  static constexpr int kTokens = NT * 8;
  static constexpr int kTermBytes = kTokens * 128;
  static constexpr int kScaleOffset = kWeightBytes + TERMS * kTermBytes;        // 128 bytes of sx per term, then sw
  static constexpr int kSlotBytes = kScaleOffset + TERMS * 128 + 128;
  static constexpr int kReduceBytes = WK > 1 ? kWarps * NT * 4 * 32 * 4 : 0;    // one MMA tile's sums of every warp
  static constexpr int kSlots = (232448 - 8192 - kReduceBytes) / (kWarps * kSlotBytes) > 6 ? 6 : (232448 - 8192 - kReduceBytes) / (kWarps * kSlotBytes);
  static constexpr int kSmemBytes = kSlots * kWarps * kSlotBytes + kReduceBytes;
};

__device__ __forceinline__ void cp_async_16_hint(uint32_t dst, const void* src, uint64_t policy) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_16_zfill(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_4_zfill(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ float2 lds64f(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ void mma_e4m3(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct Item {
  int group, feature0, row0, rows;                 // first feature of the CTA's sub-tiles; first sorted row; rows of it (<= 8 NT)
};

template <int MODE, int NT, int WK, int TERMS>
__global__ void __launch_bounds__(kThreads, 1)
skinny_kernel(const Params p) {
  using S = Shape<NT, WK, TERMS>;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int tile_prefix[kMaxGroups + 1];      // row tiles before a group
  __shared__ float group_amax[2][kWarps][S::kTokens];
  constexpr int WM = kWarps / WK;
  constexpr int kSubFeatures = MODE == kGateUp ? 16 : 32;
  constexpr int kItemFeatures = WM * kSubFeatures;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp / WK, wk = warp % WK;
  const int g8 = lane >> 2, q = lane & 3;
  const uint32_t ring = smem_u32(smem) + warp * (S::kSlots * S::kSlotBytes);
  float* reduce = reinterpret_cast<float*>(smem + S::kSlots * kWarps * S::kSlotBytes);
  const uint64_t stream = l2_policy_evict_first();
  // Everything before this overlaps the kernel in front: with groups the set-up, in the dense form, whose one group lies in the parameters, all up to the first
  // load (launches in turn: 8 x 4096 x 7168 8.5 and 7.5 us, 16 x 1024 x 1152 4.2 and 3.1).
  auto behind_grid = [&]() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (p.status && blockIdx.x == 0 && threadIdx.x == 0) *p.status = 0;
  };
  if (MODE != kDense) behind_grid();

  if (warp == 0) {
    int max_rows = INT_MAX;
    if (MODE != kDense && p.max_rows && *p.core) max_rows = p.max_rows;
    int running = 0;
    for (int base = 0; base < p.groups; base += 32) {
      const int g = base + lane;
      const int count = g < p.groups ? (p.offsets ? p.offsets[g + 1] - p.offsets[g] : p.dense_rows) : 0;
      const int tiles = MODE != kDense && count > max_rows ? 0 : (count + S::kTokens - 1) / S::kTokens;
      int incl = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (g < p.groups) tile_prefix[g] = running + incl - tiles;
      running += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) tile_prefix[p.groups] = running;
  }
  __syncthreads();
  const int n_tiles = (p.n + kItemFeatures - 1) / kItemFeatures;
  const int items = tile_prefix[p.groups] * n_tiles;
  // item i: groups in order, feature tiles of a group in order, row tiles of a feature tile next to each other (the second
  // one finds the weights in L2)
  auto locate = [&](int i, Item* it) {
    int lo = 0, hi = p.groups;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tile_prefix[mid] * n_tiles <= i) lo = mid; else hi = mid;
    }
    const int m_tiles = tile_prefix[lo + 1] - tile_prefix[lo], idx = i - tile_prefix[lo] * n_tiles;
    const int begin = p.offsets ? p.offsets[lo] : 0, end = p.offsets ? p.offsets[lo + 1] : p.dense_rows;
    it->group = lo;
    it->feature0 = idx / m_tiles * kItemFeatures;
    it->row0 = begin + idx % m_tiles * S::kTokens;
    it->rows = min(S::kTokens, end - it->row0);
  };
  // a warp whose features lie past n (n is a multiple of 128, an item may cover 256) streams the last ones again, to no effect
  auto sub_feature = [&](const Item& it) { return min(it.feature0 + wm * kSubFeatures, p.n - kSubFeatures); };

  // ---- load side: the stream of (item, K block) pairs of this warp, some slots ahead of the compute side
  int load_item = blockIdx.x, load_kb = wk, load_slot = 0;
  const uint8_t *w_lo = nullptr, *w_hi = nullptr;  // this lane's first weight row of each MMA tile, at its 16-byte chunk
  const float* sw_ptr = nullptr;                   // lanes 0, 1: the scale row of each MMA tile
  const uint8_t* x_ptr[2 * NT];                    // this lane's token rows (null: no such row)
  const float* sx_ptr = nullptr;                   // this lane's token's scales
  int load_tiles = 0;                              // token tiles of eight in the item
  const size_t w_stride = size_t(p.k_blocks) * 128;
  auto open_item = [&]() {
    if (load_item >= items) return;
    Item it;
    locate(load_item, &it);
    const int f = sub_feature(it);
    const uint8_t* w = p.w + (size_t(it.group) * p.w_rows + f + (lane >> 3)) * w_stride + (lane & 7) * 16;
    w_lo = w;
    w_hi = w + size_t(MODE == kGateUp ? p.n : 16) * w_stride;
    sw_ptr = p.sw + (size_t(it.group) * (p.w_rows / 128) + f / 128 + (MODE == kGateUp ? (lane & 1) * (p.n / 128) : 0)) * p.k_blocks;
    load_tiles = (it.rows + 7) >> 3;
#pragma unroll
    for (int i = 0; i < 2 * NT; ++i) {
      const int r = i * 4 + (lane >> 3);
      x_ptr[i] = nullptr;
      if (r < it.rows) {
        const int row = p.row_map ? __ldg(p.row_map + it.row0 + r) / p.map_div : it.row0 + r;
        x_ptr[i] = p.x + size_t(row) * p.x_stride + (lane & 7) * 16;
      }
    }
    sx_ptr = nullptr;
    if (lane < it.rows) sx_ptr = p.sx + (p.row_map ? __ldg(p.row_map + it.row0 + lane) / p.map_div : it.row0 + lane);
  };
  auto load_next = [&]() {                         // one slot; an empty copy group past the end, so that the group count stays
    if (load_item < items) {
      const uint32_t dst = ring + load_slot * S::kSlotBytes + (lane >> 3) * 128;
#pragma unroll
      for (int i = 0; i < 8; ++i) {                // four rows of 128 bytes per instruction
        const uint8_t* src = (i < 4 ? w_lo : w_hi) + size_t(load_kb) * 128 + size_t(i & 3) * 4 * w_stride;
        cp_async_16_hint(dst + i * 512 + (((lane & 7) ^ ((i * 4 + (lane >> 3)) & 7)) << 4), src, stream);
      }
      const uint32_t scales = ring + load_slot * S::kSlotBytes + S::kScaleOffset;
#pragma unroll
      for (int term = 0; term < TERMS; ++term) {
        const int x_col = term * p.k_blocks + load_kb;
#pragma unroll
        for (int i = 0; i < 2 * NT; ++i)
          if (i < 2 * load_tiles)
            cp_async_16_zfill(dst + kWeightBytes + term * S::kTermBytes + i * 512 + (((lane & 7) ^ ((i * 4 + (lane >> 3)) & 7)) << 4),
                              x_ptr[i] ? x_ptr[i] + size_t(x_col) * 128 : p.x, x_ptr[i] != nullptr);
        if (lane < S::kTokens) cp_async_4_zfill(scales + term * 128 + lane * 4, sx_ptr ? sx_ptr + size_t(x_col) * p.sx_stride : p.sx, sx_ptr != nullptr);
      }
      if (lane < 2) cp_async_4_zfill(scales + TERMS * 128 + lane * 4, sw_ptr + load_kb, true);
      load_kb += WK;
      if (load_kb >= p.k_blocks) { load_kb = wk; load_item += gridDim.x; open_item(); }
      load_slot = load_slot + 1 == S::kSlots ? 0 : load_slot + 1;
    }
    cp_async_commit();
  };
  // a warp without a K block of its own (fewer K blocks than warps share) has nothing to load
  if (wk >= p.k_blocks) load_item = items;
  open_item();
  if (MODE == kDense) behind_grid();
#pragma unroll
  for (int s = 0; s < S::kSlots - 1; ++s) load_next();

  int slot = 0, flip = 0;
  for (int i = blockIdx.x; i < items; i += gridDim.x) {
    Item it;
    locate(i, &it);
    const int tiles = (it.rows + 7) >> 3;
    // the route weight of token `lane`, asked for before the products: asked for where it is used, its two dependent loads
    // took longer than the products of a short K
    float token_weight = 0.f;
    if (MODE == kDown && lane < it.rows) token_weight = __ldg(p.row_weight + __ldg(p.weight_map + it.row0 + lane));
    float acc[2][NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[0][n][e] = acc[1][n][e] = 0.f;
    for (int kb = wk; kb < p.k_blocks; kb += WK) {
      cp_async_wait<S::kSlots - 2>();
      __syncwarp();                                // the slot has landed for every lane; every lane is done with the one before
      load_next();
      const uint32_t s = ring + slot * S::kSlotBytes, scales = s + S::kScaleOffset;
      uint32_t a[2][2][8];                         // [MMA tile][row g / g + 8][k-step pair words]
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = t * 16 + h * 8 + g8;
          const uint4 lo = lds128(s + r * 128 + (((2 * q) ^ g8) << 4)), hi = lds128(s + r * 128 + (((2 * q + 1) ^ g8) << 4));
          a[t][h][0] = lo.x; a[t][h][1] = lo.y; a[t][h][2] = lo.z; a[t][h][3] = lo.w;
          a[t][h][4] = hi.x; a[t][h][5] = hi.y; a[t][h][6] = hi.z; a[t][h][7] = hi.w;
        }
      const float2 sw = lds64f(scales + TERMS * 128);
#pragma unroll
      for (int m = 0; m < NT * TERMS; ++m) {
        const int n = m / TERMS, term = m % TERMS;
        if (n >= tiles) break;
        const uint32_t xr = s + kWeightBytes + term * S::kTermBytes + (n * 8 + g8) * 128;
        const uint4 lo = lds128(xr + (((2 * q) ^ g8) << 4)), hi = lds128(xr + (((2 * q + 1) ^ g8) << 4));
        const uint32_t b[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        const float2 sx = lds64f(scales + term * 128 + (n * 8 + q * 2) * 4);
        float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
          for (int t = 0; t < 2; ++t)
            mma_e4m3(d[t], a[t][0][2 * ks], a[t][1][2 * ks], a[t][0][2 * ks + 1], a[t][1][2 * ks + 1], b[2 * ks], b[2 * ks + 1]);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const float w = t == 0 ? sw.x : sw.y, s0 = w * sx.x, s1 = w * sx.y;
          acc[t][n][0] = fmaf(d[t][0], s0, acc[t][n][0]); acc[t][n][1] = fmaf(d[t][1], s1, acc[t][n][1]);
          acc[t][n][2] = fmaf(d[t][2], s0, acc[t][n][2]); acc[t][n][3] = fmaf(d[t][3], s1, acc[t][n][3]);
        }
      }
      slot = slot + 1 == S::kSlots ? 0 : slot + 1;
    }

    const bool exists = it.feature0 + wm * kSubFeatures < p.n;
    const int f = sub_feature(it);
    // One accumulator of each MMA tile: token 8 n + 2 q + (e & 1) of the item, feature f + g + 8 (e >> 1) (+ 16 in tile 1)
    auto emit = [&](int n, int e, float v0, float v1) {
      const int token = n * 8 + q * 2 + (e & 1);
      const float w = MODE == kDown ? __shfl_sync(0xffffffffu, token_weight, token) : 1.f;
      if (!exists || token >= it.rows) return;
      const size_t at = size_t(it.row0 + token) * p.n + f + g8 + 8 * (e >> 1);
      if (MODE == kGateUp) {
        reinterpret_cast<float*>(p.out)[at] = v0 * silu(v1);
      } else {
        reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(v0 * w);
        reinterpret_cast<__nv_bfloat16*>(p.out)[at + 16] = __float2bfloat16_rn(v1 * w);
      }
    };
    if (WK > 1) {
      // the sub-tile's warps add their sums in warp order; each of them finishes a share of the accumulators
      constexpr int kMine = (NT * 4 + WK - 1) / WK;
      float sum[2][kMine];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int j = 0; j < NT * 4; ++j) reduce[(warp * NT * 4 + j) * 32 + lane] = acc[t][j >> 2][j & 3];
        __syncthreads();
#pragma unroll
        for (int m = 0; m < kMine; ++m) {
          const int j = wk + m * WK;
          float v = 0.f;
          if (j < NT * 4) {
#pragma unroll
            for (int k = 0; k < WK; ++k) v += reduce[((wm * WK + k) * NT * 4 + j) * 32 + lane];
          }
          sum[t][m] = v;
        }
        __syncthreads();
      }
#pragma unroll
      for (int m = 0; m < kMine; ++m) {
        const int j = wk + m * WK;
        if (j < NT * 4) emit(j >> 2, j & 3, sum[0][m], sum[1][m]);
      }
    } else if (MODE != kGateUp) {
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) emit(n, e, acc[0][n][e], acc[1][n][e]);
    } else {
      // SwiGLU, then e4m3 quantisation over the item's 128 features (16 of each warp): the warps' maxima meet in shared memory
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        if (n >= tiles) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[0][n][e] *= silu(acc[1][n][e]);
      }
      for (int term = 0; term < p.terms; ++term, flip ^= 1) {
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          if (n >= tiles) break;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float m = fmaxf(fabsf(acc[0][n][e]), fabsf(acc[0][n][e + 2]));
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (g8 == 0) group_amax[flip][warp][n * 8 + q * 2 + e] = m;
          }
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          if (n >= tiles) break;
          float scale[2], inv[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float m = 0.f;
#pragma unroll
            for (int k = 0; k < kWarps; ++k) m = fmaxf(m, group_amax[flip][k][n * 8 + q * 2 + e]);
            scale[e] = m > 0.f ? m / 448.f : 1.f;
            inv[e] = 1.f / scale[e];
          }
          const uint32_t packed = pack_e4m3x4(acc[0][n][0] * inv[0], acc[0][n][1] * inv[1], acc[0][n][2] * inv[0], acc[0][n][3] * inv[1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int token = n * 8 + q * 2 + (e & 1);
            const uint8_t byte = uint8_t(packed >> (8 * e));
            if (token < it.rows) {
              reinterpret_cast<uint8_t*>(p.out)[size_t(it.row0 + token) * (size_t(p.n) * p.terms) + size_t(term) * p.n + f + g8 + 8 * (e >> 1)] = byte;
              if (warp == 0 && g8 == 0 && e < 2) p.out_scale[size_t(term * (p.n / 128) + it.feature0 / 128) * p.row_capacity + it.row0 + token] = scale[e];
            }
            acc[0][n][e] -= e4m3_to_float(byte) * scale[e & 1];      // what a second term has to carry
          }
        }
      }
    }
  }
  cp_async_wait<0>();
}

// fp32 [rows, n] -> e4m3 [rows, n * terms] + scales [n / 128 * terms, row_capacity]: one warp per (row, 128 features).
static __global__ void __launch_bounds__(256)
quantize_kernel(const float* __restrict__ in, const int* __restrict__ rows_ptr, uint8_t* __restrict__ out, float* __restrict__ out_scale,
                int n, int terms, int row_capacity) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, blocks = n / 128;
  const int total = *rows_ptr * blocks;
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < total; i += gridDim.x * 8) {
    const int row = i / blocks, b = i - row * blocks;
    float4 v = *reinterpret_cast<const float4*>(in + size_t(row) * n + b * 128 + lane * 4);
    for (int term = 0; term < terms; ++term) {
      const float m = warp_max(fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
      const float scale = m > 0.f ? m / 448.f : 1.f, inv = 1.f / scale;
      const uint32_t packed = pack_e4m3x4(v.x * inv, v.y * inv, v.z * inv, v.w * inv);
      reinterpret_cast<uint32_t*>(out + size_t(row) * (size_t(n) * terms) + size_t(term) * n + b * 128)[lane] = packed;
      if (lane == 0) out_scale[size_t(term * blocks + b) * row_capacity + row] = scale;
      v.x -= e4m3_to_float(uint8_t(packed)) * scale; v.y -= e4m3_to_float(uint8_t(packed >> 8)) * scale;
      v.z -= e4m3_to_float(uint8_t(packed >> 16)) * scale; v.w -= e4m3_to_float(uint8_t(packed >> 24)) * scale;
    }
  }
}

// A kernel's entry points by run-time numbers: token tiles of eight (one or two), K split, terms (two in the down mode only).
template <int MODE, typename F>
inline int with_shape(int nt, int wk, int terms, F f) {
  auto by_terms = [&](auto tiles, auto split) {
    if constexpr (MODE == kDown) { if (terms == 2) return f(tiles, split, std::integral_constant<int, 2>()); }
    return f(tiles, split, std::integral_constant<int, 1>());
  };
  auto by_split = [&](auto tiles) {
    if (wk == 1) return by_terms(tiles, std::integral_constant<int, 1>());
    if constexpr (MODE != kGateUp) { if (wk == 4) return by_terms(tiles, std::integral_constant<int, 4>()); }
    return by_terms(tiles, std::integral_constant<int, 8>());
  };
  return nt == 1 ? by_split(std::integral_constant<int, 1>()) : by_split(std::integral_constant<int, 2>());
}
template <int MODE>
inline int launch_any(int nt, int wk, int terms, const Params& p, int grid, cudaStream_t s) {
  return with_shape<MODE>(nt, wk, terms, [&](auto tiles, auto split, auto t) {
    return launch_dependent(skinny_kernel<MODE, tiles(), split(), t()>, dim3(grid), dim3(kThreads), Shape<tiles(), split(), t()>::kSmemBytes, s, p);
  });
}
template <int MODE>
inline int prepare_any(int nt, int wk, int terms) {
  return with_shape<MODE>(nt, wk, terms, [](auto tiles, auto split, auto t) {
    return int(cudaFuncSetAttribute(skinny_kernel<MODE, tiles(), split(), t()>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<tiles(), split(), t()>::kSmemBytes));
  });
}

// Time of a launch in units of a warp's K block (32 weight rows x 128): rounds of the GPU times an item's K blocks and what
// it costs beside them.  `features`: of an item, `row_tiles`: row tiles of all groups together.
inline double cost(double row_tiles, int n, int features, int k_blocks, int wk, int sms) {
  const double items = row_tiles * ((n + features - 1) / features);
  const double rounds = items <= sms ? 1 : items > 8 * sms ? items / sms : double((long long)(items / sms + 0.999));
  return rounds * ((k_blocks + wk - 1) / wk + 3);
}
// How many warps share a sub-tile's K blocks; on a tie the smaller split, which meets less often.
inline int choose_split(double row_tiles, int n, int k_blocks, int sms) {
  int best = 1;
  for (int wk : {4, 8})
    if (wk <= k_blocks && cost(row_tiles, n, 32 * (kWarps / wk), k_blocks, wk, sms) < 0.999 * cost(row_tiles, n, 32 * (kWarps / best), k_blocks, best, sms)) best = wk;
  return best;
}
// The same for the gate/up product (16 features to a sub-tile), where a split means that quantize_kernel runs after it.
inline int choose_split_gate_up(double row_tiles, int n, int k_blocks, int sms) {
  return k_blocks >= 8 && cost(row_tiles, n, 16, k_blocks, 8, sms) + 5 < cost(row_tiles, n, 128, k_blocks, 1, sms) ? 8 : 1;
}

}  // namespace skinny
}  // namespace cake
