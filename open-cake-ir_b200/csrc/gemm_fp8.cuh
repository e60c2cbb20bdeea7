// Block-scaled FP8 (e4m3) GEMM core for sm_100a: one persistent, warp-specialised kernel
// shared by the dense block-scaled GEMM and the two grouped GEMMs of the MoE expert layer.
//
//   C[m, n] = sum_kb ( sum_{k in kb} A[m, k] * B[n, k] ) * sfa[kb, m] * sfb[n/128, kb]
//
// Layout contract (reference: docs/adr/0023-block-scales-are-axis-relations.md:21-27,
// src/open_cake_ir/tasks/solx_fib/moe.py:13-20): A e4m3 [rows, K] row-major with fp32 scales
// stored K-block-major [K/128, rows]; B e4m3 [N, K] row-major ("N-K weights") with fp32 scales
// [N/128, K/128]; grouped problems stack B as [G, N, K] and A as expert-contiguous row
// segments described by `offsets[G+1]`.
//
// Mapping to the hardware.  A CTA owns a 128-row x 256-column output tile per work item.
// Rows are TMEM lanes (UMMA M = 128), columns are TMEM columns (UMMA N = 256).  For every
// 128-wide K block, four tcgen05.mma.kind::f8f6f4 (K = 32 each) write a FRESH partial product
// into one of two TMEM accumulator stages; eight epilogue warps read that stage back
// (tcgen05.ld), multiply it by the block's scales and add it to fp32 registers ("promotion"),
// which is what arbitrary fp32 1x128 / 128x128 scales need -- the hardware block-scaled kinds
// only take power-of-two scales per 32 elements.  While the epilogue promotes block kb the
// tensor core already works on block kb+1 in the other stage.  A group's last row tile may be one of
// 64 or 32 rows (tile_rows).  Operands arrive through a TMA ring of four stages, six where CTAs share K (128-byte swizzle, one elected producer thread); the MMA is issued by one
// elected thread of a second warp.  Work items are (group, n tile, m tile) with the m tile
// fastest, so CTAs that share a weight tile run at the same time and the second reader hits L2.
// Items either go round the CTAs in turn or are drawn from a device counter by the TMA warp, which
// hands them to the other roles through a four-slot ring (Params::queue).
#pragma once
#include "common.cuh"
#include <type_traits>

namespace cake {
namespace gemm {

constexpr int kBM = 128;          // rows per tile = UMMA M = TMEM lanes
constexpr int kBN = 256;          // columns per tile = UMMA N
constexpr int kBK = 128;          // e4m3 elements (= bytes) per K block = scale granularity
constexpr int kUmmaK = 32;        // K of one tcgen05.mma for 8-bit operands
constexpr int kTmemColumns = 512;                 // all of an SM's tensor memory
constexpr int kBytesA = kBM * kBK;                // 16 KiB
constexpr int kBytesB = kBN * kBK;                // 32 KiB
// The rings: tiles of 256 columns, and of 128 where CTAs share K (see the kernel).  The latter have few K blocks to a CTA and wait for HBM
// on all of them, so every stage more is a block sooner (64 x 4096 x 7168, 14 blocks to a CTA: 11.5 us with four stages of 48 KB and two
// accumulators, 10.7 with six of 32 KB and four; 48 x 9472 x 7168 19.7 and 18.4).
template <bool SPLIT>
struct Ring {
  static constexpr int kCols = SPLIT ? 128 : kBN;
  static constexpr int kStageBytes = kBytesA + kCols * kBK;
  static constexpr int kStages = SPLIT ? 6 : 4;            // 192 KiB of shared memory
  static constexpr int kTmemStages = kTmemColumns / kCols;
};
// Where an index of the operand ring lies.  Six is not a power of two: stepped, since a division by it takes some 20 clocks of a K block.
template <bool SPLIT>
struct At {
  uint32_t index = 0, slot_ = 0, phase_ = 0;
  __device__ __forceinline__ void next() {
    if (!SPLIT) ++index;
    else if (++slot_ == uint32_t(Ring<true>::kStages)) { slot_ = 0; phase_ ^= 1; }
  }
  __device__ __forceinline__ uint32_t slot() const { return SPLIT ? slot_ : index % Ring<false>::kStages; }
  __device__ __forceinline__ uint32_t phase() const { return SPLIT ? phase_ : (index / Ring<false>::kStages) & 1; }
};
constexpr int kRingBytes = Ring<false>::kStages * Ring<false>::kStageBytes, kMaxStages = Ring<true>::kStages, kMaxTmemStages = Ring<true>::kTmemStages;
static_assert(Ring<true>::kStages * Ring<true>::kStageBytes <= kRingBytes && kMaxStages >= Ring<false>::kStages, "the narrow ring does not fit");
constexpr int kTailRows = 32;                    // box rows of the small A map
constexpr int kControlWarps = 4;                  // one warpgroup: warp 0 TMA, warp 1 MMA, warp 2 scales, warp 3 idle
constexpr int kEpilogueWarps = 8;                 // two warpgroups: 2 column groups x 4 TMEM lane quadrants
constexpr int kThreads = (kControlWarps + kEpilogueWarps) * 32;
// Register budget moved between the warpgroups once the roles split.  The pool setmaxnreg draws on
// is what the launch allocated, 168 registers x 384 threads = 64512, not the SM's 65536: an
// increase that asks for more than the pool ever holds blocks for good.  128 x 56 + 256 x 224 = 64512 (at 40 and 232 the kernel spilled
// a few registers: the MoE layer 2 % slower).
constexpr int kControlRegs = 56;
constexpr int kEpilogueRegs = 224;
static_assert(kControlWarps * 32 * kControlRegs + kEpilogueWarps * 32 * kEpilogueRegs <= (65536 / kThreads / 8 * 8) * kThreads,
              "setmaxnreg budget exceeds the registers the launch allocates");
constexpr int kMaxGroups = 512;
constexpr int kMaxSplit = 4;      // CTAs that share a tile's K
constexpr int kItemSlots = 4;
// The scales of block it + kScaleAhead are announced with the operands of block it, so that the epilogue can read a
// block's scales from shared memory while it still works on the block before.  A slot is refilled when the shared-memory
// stage of block it is handed back, i.e. when the MMAs of block it - kStages are done; those were issued after the epilogue
// had read the scales of block it - kStages - kTmemStages.
constexpr int kScaleAhead = 2;
constexpr int kScaleSlots = 16;
static_assert(kScaleSlots >= kMaxStages + kMaxTmemStages + kScaleAhead, "a slot's scales could be overwritten before they are read");

enum Mode : int {
  kDense = 0,        // C bf16 [M, N]
  kGateUp = 1,       // grouped GEMM1: x1 = cols [0,128), x2 = cols [128,256) of the tile;
                     // out = e4m3(x1 * silu(x2)) + per-(row,128) scale  (optionally hi+lo split)
  kDown = 2,         // grouped GEMM2: out bf16 [rows, N] = acc * route weight of the row
};

struct Params {
  int n;                       // output columns per group (dense N; GEMM1: I; GEMM2: H)
  int k_blocks;                // K / 128 of the A operand
  int b_k_blocks;              // K / 128 of the B operand (== k_blocks unless A is hi/lo split)
  int b_rows_per_group;        // rows of B per group (dense N; GEMM1: 2I; GEMM2: H)
  int groups;                  // 1 for dense
  int row_capacity;            // rows the A buffer (and its scale rows) is allocated for
  int interleave_hi_lo;        // 1: A K-block kb -> A column block (kb&1)*(k_blocks/2) + kb/2, B block kb/2
  const int* offsets;          // [groups+1] device row offsets into A; null = one group of dense_rows rows
  int dense_rows;
  const int* enabled;          // grouped modes: device word, 0 = there is nothing to do here (null: there is)
  int min_rows;                // groups of at most so many rows are left out: another kernel's (0: none are)
  const float* sfa;            // [k_blocks, row_capacity]
  const float* sfb;            // [groups, b_rows_per_group/128, b_k_blocks]
  void* out;                   // see Mode
  float* out_scale;            // kGateUp: [out_k_blocks, row_capacity]
  const float* row_weight;     // kDown: [row_capacity] route weight per sorted row
  int split_act;               // kGateUp: 1 = also write the residual (lo) term
  int* status;                 // device status word (0 = ok)
  int* queue;                  // device counter, 0 at launch: work items are drawn from it (null: item i goes to CTA i mod grid)
  int* drawn_out;              // device counter, 0 at launch, of CTAs that have drawn their last item: the last one clears both (null: the caller does)
  int wait_kiloclocks;         // budget of a bounded wait in units of 1024 clocks (0: the default, about a second)
  int skip_load;               // test hook: CTA 0's producer leaves out the loads of its second K block, once
};

struct Shared {
  uint4 out_rows[kEpilogueWarps][128];                      // per epilogue warp: 32 rows of 64 bytes on their way out
  int4 item[kItemSlots];                                    // group (-1: no further item), first row, rows, n tile
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t tmem_full[kMaxTmemStages];
  uint64_t tmem_empty[kMaxTmemStages];
  uint64_t exchange_done;                                   // kGateUp: all epilogue warps have published their amax
  uint64_t item_full[kItemSlots], item_empty[kItemSlots];   // hand-over of work items from the TMA warp to the other roles
  float scale_a[kScaleSlots][kBM];                          // sfa of the tile's rows for one K block
  float scale_b[kScaleSlots][2];                            // sfb of the tile's two 128-column halves
  uint32_t tmem_base;
  WaitControl wait;
  int tile_prefix[kMaxGroups + 1];     // m tiles before group g
  float exchange[2][2][2 * kBM];       // [item parity][term][part of the row's 128 features][row] amax exchange for kGateUp
};

// A warp's 32 rows of 64 bytes (lane i holds row i) to global memory.  Through shared memory, so that a store instruction
// writes whole 64-byte runs of eight rows: written straight from the registers it touches 16 bytes of each of 32 rows,
// and the output of a tile then cost 110 clocks per K block (8192 x 4096 x 7168), 13 % of the whole.  The 16-byte chunk
// index is XORed with the row pair, which keeps both sides free of bank conflicts.
__device__ __forceinline__ void warp_store_64(uint4* scratch, const uint4 (&v)[4], uint8_t* dst, size_t stride, int rows, int lane) {
#pragma unroll
  for (int c = 0; c < 4; ++c) scratch[lane * 4 + (c ^ ((lane >> 1) & 3))] = v[c];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i * 8 + (lane >> 2), c = lane & 3;
    const uint4 x = scratch[r * 4 + (c ^ ((r >> 1) & 3))];
    if (r < rows) *reinterpret_cast<uint4*>(dst + size_t(r) * stride + c * 16) = x;
  }
  __syncwarp();
}

struct Item {
  int group, row0, rows_valid, n_tile;
};

// Rows of the product that a tile takes.  Groups seldom end on 128 rows: an expert of 128 rows on average has a few in a second
// tile half of the time, and in a step of some hundred tokens it has ten or thirty in all.  A tile of 32 or 64 rows (the
// weight-stationary products) takes 307 or 323 clocks of tensor pipe a K block (429 or 449 with the two commits behind each) instead of 512, a quarter or half of the
// promotion and less of A; under the power cap what it does not do is time for the others (hidden 7168, 256 experts of 2048, all
// with as many rows: 2380 -> 1830 us at 32, 2566 -> 2090 at 64, 4116 -> 3660 at 137; at 128 there is nothing to gain).
template <int MODE>
__host__ __device__ constexpr int tile_rows(int rows_valid) {
  return MODE == kDense ? kBM : rows_valid <= 32 ? 32 : rows_valid <= 64 ? 64 : kBM;
}

// Work item `g` -> (group, m tile, n tile); items of one group are ordered n tile major,
// m tile minor.  Returns false past the end.
__device__ __forceinline__ bool locate(const Shared* sh, const Params& p, int n_tiles, int g, Item* it) {
  const int total = sh->tile_prefix[p.groups] * n_tiles;
  if (g >= total) return false;
  int lo = 0, hi = p.groups;            // largest group with prefix*n_tiles <= g
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (sh->tile_prefix[mid] * n_tiles <= g) lo = mid; else hi = mid;
  }
  const int m_tiles = sh->tile_prefix[lo + 1] - sh->tile_prefix[lo];
  const int idx = g - sh->tile_prefix[lo] * n_tiles;
  const int begin = p.offsets ? p.offsets[lo] : 0;
  const int end = p.offsets ? p.offsets[lo + 1] : p.dense_rows;
  const int mt = idx % m_tiles;
  it->group = lo;
  it->n_tile = idx / m_tiles;
  it->row0 = begin + mt * kBM;
  it->rows_valid = min(kBM, end - it->row0);
  return true;
}

__device__ __forceinline__ float4 load_cluster(uint32_t local_addr, uint32_t rank) {
  float4 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(local_addr), "r"(rank) : "memory");
  return v;
}

// SPLIT (dense only): tiles of 128 columns, each shared by the CTAs of a cluster (two or four), a part of K to each.  A
// problem of few tiles otherwise runs its K blocks, about 0.45 us each, one after another on a handful of SMs (64 x 4096 x
// 7168: 16 SMs).  The parts meet through distributed shared memory: CTA r finishes columns [128 r / S, 128 (r + 1) / S).
template <int MODE>
struct Maps { CUtensorMap a, a_tail, b; };
template <>
struct Maps<kGateUp> { CUtensorMap a, a_tail, b, b_narrow; };        // b_narrow: boxes of 32 rows
template <int MODE, bool SPLIT = false>
__global__ void __launch_bounds__(kThreads, 1)
gemm_fp8_kernel(const __grid_constant__ Maps<MODE> maps, const Params p) {
  if (MODE != kDense && p.enabled) {               // the usual case is to leave, so before anything is set up
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (*p.enabled == 0) return;
  }
  constexpr int kStages = Ring<SPLIT>::kStages, kTmemStages = Ring<SPLIT>::kTmemStages, kStageBytes = Ring<SPLIT>::kStageBytes;
  constexpr int kCols = Ring<SPLIT>::kCols;        // columns of a tile
  extern __shared__ uint8_t smem_raw[];
  // by an offset, not by rounding the pointer as an integer: the compiler then still knows that it is shared memory
  uint8_t* tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  Shared* sh = reinterpret_cast<Shared*>(tiles + kRingBytes);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  uint32_t rank = 0, split = 1;
  if (SPLIT) {
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(split));
  }
  const int first_item = SPLIT ? blockIdx.x / split : blockIdx.x;
  const int k_begin = SPLIT ? int(rank * uint32_t(p.k_blocks) / split) : 0;                  // this CTA's K blocks
  const int k_count = SPLIT ? int((rank + 1) * uint32_t(p.k_blocks) / split) - k_begin : p.k_blocks;
  const int n_tiles = (MODE == kGateUp) ? p.n / 128 : (p.n + kCols - 1) / kCols;

  if (threadIdx.x == 0) {                          // (one after another: only those that the form has)
    for (int s = 0; s < kStages; ++s) { mbar_init(&sh->full[s], 1 + 32); mbar_init(&sh->empty[s], 1); }
    for (int s = 0; s < kTmemStages; ++s) { mbar_init(&sh->tmem_full[s], 1); mbar_init(&sh->tmem_empty[s], kEpilogueWarps); }
    for (int s = 0; !SPLIT && s < kItemSlots; ++s) { mbar_init(&sh->item_full[s], 1); mbar_init(&sh->item_empty[s], 2 + kEpilogueWarps); }
    if (MODE == kGateUp) mbar_init(&sh->exchange_done, kEpilogueWarps);
    sh->wait.abort_flag = 0;
    sh->wait.budget_kiloclocks = p.wait_kiloclocks;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sh->tmem_base, kTmemColumns);
    tmem_relinquish();
  }
  if (threadIdx.x == 96) {
    tma_prefetch_descriptor(&maps.a);
    tma_prefetch_descriptor(&maps.a_tail);
    tma_prefetch_descriptor(&maps.b);
    if constexpr (MODE == kGateUp) tma_prefetch_descriptor(&maps.b_narrow);
  }
  // Launched as a programmatic dependent: what comes before this overlaps the kernel in front.  The dense form's items lie in the parameters, so there
  // the roles are set up and the first item found by then as well, and each waits where it begins (its bounded waits among them; the first load
  // came 1.2 us behind that kernel's end with the wait here; launches in turn: 64 x 4096 x 7168 11.7 and 11.0 us, 32 x 2048 x 2048 6.5 and 6.0).
  auto behind_grid = []() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  };
  if (MODE != kDense) behind_grid();
  if (warp == kControlWarps) {   // m-tile prefix over groups (serial per lane chunk, then a warp scan)
    int running = 0;
    for (int base = 0; base < p.groups; base += 32) {
      int g = base + lane;
      int tiles_g = 0;
      if (g < p.groups) {
        int cnt = p.offsets ? p.offsets[g + 1] - p.offsets[g] : p.dense_rows;
        tiles_g = cnt > p.min_rows ? (cnt + kBM - 1) / kBM : 0;
      }
      int incl = tiles_g;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (g < p.groups) sh->tile_prefix[g] = running + incl - tiles_g;
      running += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) sh->tile_prefix[p.groups] = running;
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  volatile int* abort_flag = &sh->wait.abort_flag;
  // With groups, or where items are drawn, the TMA warp, which is ahead of the others, finds an item's group and rows and
  // hands them on: the search of the prefix and the two offsets behind it cost the epilogue 1400 clocks an item (a K block
  // takes it 800), in which no product was taken up.  One group without a queue has nothing to search.
  const bool handed = p.queue || p.offsets;

  if (warp < kControlWarps) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kControlRegs));
  if (warp == 0) {
    // ------------------------------ TMA producer --------------------------------------
    if (elect_one()) {
      const uint64_t keep = l2_policy_evict_last();    // activations: re-read by every n tile
      // Work items.  With a queue, this thread draws them (the first is the CTA's index, every later
      // one comes from the device counter, asked for one item ahead) and hands each to the other
      // roles through a small ring, so that an SM that runs slower simply takes fewer
      // items; without one, item i belongs to CTA i mod grid.  The next item is found and handed on
      // half-way through the K blocks of the one before, while this thread is ahead of the ring anyway
      // (found between two items it delays the next one's first loads; second GEMM of 2500 tokens, two terms, hidden 2048, 128
      // experts of 768: 137 us then, 128 now).
      uint32_t it = 0, k = 0;
      At<SPLIT> at;
      bool ok = true, valid;
      Item item;
      int g = first_item;
      auto find = [&](int index, uint32_t nth) {         // item `index`, the nth of this CTA
        valid = locate(sh, p, n_tiles, index, &item);
        if (!handed) return;
        const int slot = nth % kItemSlots;
        ok = mbar_wait(&sh->item_empty[slot], ((nth / kItemSlots) & 1) ^ 1, abort_flag, p.status, kStatusWaitFlag);
        if (!ok) return;
        sh->item[slot] = valid ? make_int4(item.group, item.row0, item.rows_valid, item.n_tile) : make_int4(-1, 0, 0, 0);
        mbar_arrive(&sh->item_full[slot]);
      };
      find(g, 0);
      if (MODE == kDense) {
        behind_grid();
        // Long before any wait can run out, as the grid fits the GPU and its CTAs start together.  (Were the SMs of CTA 0 held by other work for the second that
        // a wait takes to run out, its report would be lost; a kernel in front that clears the word takes 0.4 us of 7 to 21, 0.7 to 1.2 launched from the host.)
        if (!p.queue && blockIdx.x == 0) *p.status = 0;
      }
      const int find_at = (k_count - 1) / 2;
      while (ok && valid) {
        g = p.queue ? int(gridDim.x) + atomicAdd(p.queue, 1) : g + int(gridDim.x);
        const int b_row0 = item.group * p.b_rows_per_group;
        const int m = MODE == kDense ? (item.rows_valid <= kTailRows ? kTailRows : kBM) : tile_rows<MODE>(item.rows_valid);       // rows of A to bring in
        const uint32_t stage_tx = uint32_t(m * kBK + kCols * kBK);
        const int a_row0 = item.row0, n_tile = item.n_tile;
        for (int kb = 0; kb < k_count; ++kb, ++it, at.next()) {
          const int s = at.slot();
          ok = mbar_wait(&sh->empty[s], at.phase() ^ 1, abort_flag, p.status, kStatusWaitSmemEmpty);
          if (!ok) break;
          if (kb == find_at) find(g, k + 1);                            // (this item is in the variables above)
          if (!ok) break;
          if (p.skip_load && blockIdx.x == 0 && it == 1) continue;      // test hook: this ring slot is never filled
          uint8_t* a_dst = tiles + s * kStageBytes;
          uint8_t* b_dst = a_dst + kBytesA;
          int a_col = k_begin + kb, b_col = k_begin + kb;
          if (p.interleave_hi_lo) { a_col = (kb & 1) * (p.k_blocks >> 1) + (kb >> 1); b_col = kb >> 1; }
          mbar_arrive_expect_tx(&sh->full[s], stage_tx);
          tma_load_2d_hint(a_dst, m < kBM ? &maps.a_tail : &maps.a, a_col * kBK, a_row0, &sh->full[s], keep);
          if (MODE != kDense && m == 64) tma_load_2d_hint(a_dst + kTailRows * kBK, &maps.a_tail, a_col * kBK, a_row0 + kTailRows, &sh->full[s], keep);
          if constexpr (MODE == kGateUp) {
            if (m < kBM) {
              // 32 rows of x1, the matching 32 of x2, the next 32 of x1, ...: an epilogue thread of a narrow tile holds both of a feature
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                tma_load_2d(b_dst + (2 * i) * 32 * kBK, &maps.b_narrow, b_col * kBK, b_row0 + n_tile * 128 + 32 * i, &sh->full[s]);
                tma_load_2d(b_dst + (2 * i + 1) * 32 * kBK, &maps.b_narrow, b_col * kBK, b_row0 + p.n + n_tile * 128 + 32 * i, &sh->full[s]);
              }
            } else {
              // 128 rows of the first half (x1) and the matching 128 rows of the second half (x2)
              tma_load_2d(b_dst, &maps.b, b_col * kBK, b_row0 + n_tile * 128, &sh->full[s]);
              tma_load_2d(b_dst + 128 * kBK, &maps.b, b_col * kBK, b_row0 + p.n + n_tile * 128, &sh->full[s]);
            }
          } else {
            tma_load_2d(b_dst, &maps.b, b_col * kBK, b_row0 + n_tile * kCols, &sh->full[s]);
          }
        }
        ++k;
      }
      if (p.drawn_out && atomicAdd(p.drawn_out, 1) == int(gridDim.x) - 1) { *p.queue = 0; *p.drawn_out = 0; }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ----------------------------------------
    if (elect_one()) {
      if (MODE == kDense) asm volatile("griddepcontrol.wait;" ::: "memory");
      uint32_t it = 0, k = 0;
      At<SPLIT> at;
      bool ok = true;
      Item item;
      for (int g = first_item; ok; g += gridDim.x, ++k) {
        if (handed) {                  // the k-th item of this CTA, from the TMA warp
          const int slot = k % kItemSlots;
          ok = mbar_wait(&sh->item_full[slot], (k / kItemSlots) & 1, abort_flag, p.status, kStatusWaitFlag);
          if (!ok) break;
          const int4 v = sh->item[slot];
          mbar_arrive(&sh->item_empty[slot]);
          if (v.x < 0) break;
          item.rows_valid = v.z;
        } else if (!locate(sh, p, n_tiles, g, &item)) {
          break;
        }
        auto products = [&](auto narrow, uint32_t idesc) {
          for (int kb = 0; kb < k_count; ++kb, ++it, at.next()) {
            const int s = at.slot();
            const int t = it % kTmemStages;
            ok = mbar_wait_both(&sh->full[s], at.phase(), kStatusWaitSmemFull, &sh->tmem_empty[t],
                                ((it / kTmemStages) & 1) ^ 1, kStatusWaitTmemEmpty, abort_flag, p.status);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t a_addr = smem_u32(tiles + s * kStageBytes);
            const uint64_t a_desc = umma_desc_sw128(a_addr);
            const uint64_t b_desc = umma_desc_sw128(a_addr + kBytesA);
            const uint32_t d = tmem_base + t * kCols;
#pragma unroll
            for (int j = 0; j < kBK / kUmmaK; ++j) {
              // advancing K inside the 128-byte swizzle row: +32 bytes = +2 in the 16-byte address field
              const uint64_t step = j * (kUmmaK >> 4);
              if constexpr (decltype(narrow)::value) umma_f8f6f4_ws(d, a_desc + step, b_desc + step, idesc, j > 0);
              else umma_f8f6f4(d, a_desc + step, b_desc + step, idesc, j > 0);
            }
            tcgen05_commit(&sh->empty[s]);       // the ring slot is free once these MMAs have read it
            tcgen05_commit(&sh->tmem_full[t]);   // and the partial product is complete
          }
        };
        const int m = tile_rows<MODE>(item.rows_valid);
        if (MODE != kDense && m < kBM) products(std::true_type(), umma_idesc(0 /* e4m3 */, m, kCols));
        else products(std::false_type(), umma_idesc(0 /* e4m3 */, kBM, kCols));
      }
    }
  } else if (warp == 2) {
    // ------------------------------ scale loader --------------------------------------
    // Brings the scales of a K block (one per row of the tile, one per 128 columns) into a shared-memory ring and
    // announces them with the operands of the block kScaleAhead before it: a complete partial product implies that the
    // scales of the next one are there, so the epilogue waits once per block and reads them a block ahead.  (Each epilogue
    // thread loading its own scales a few blocks ahead into registers paid one round trip to L2 per block, because handing
    // a register on from block to block waits for the load behind it; a barrier of their own cost 150 clocks per block,
    // and reading them when they are needed 75 to 170, since the reads queue behind the tensor core's operand reads.)
    if (MODE == kDense) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int sfb_rows = p.b_rows_per_group / 128;
    uint32_t it = 0, k = 0;
    At<SPLIT> at;                        // of block it - kScaleAhead
    bool ok = true;
    Item item;
    for (int g = first_item; ok; g += gridDim.x, ++k) {
      if (handed) {                    // the k-th item of this CTA, from the TMA warp
        const int slot = k % kItemSlots;
        ok = mbar_wait(&sh->item_full[slot], (k / kItemSlots) & 1, abort_flag, p.status, kStatusWaitFlag);
        if (!ok) break;
        const int4 v = sh->item[slot];
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->item_empty[slot]);
        if (v.x < 0) break;
        item.group = v.x; item.row0 = v.y; item.rows_valid = v.z; item.n_tile = v.w;
      } else if (!locate(sh, p, n_tiles, g, &item)) {
        break;
      }
      // lanes 0 and 1 also fetch sfb: of x1 and x2 in the gate/up mode, else of the tile's two 128-column halves
      const int sfb_row = MODE == kGateUp ? item.n_tile + (lane & 1) * (p.n / 128) : SPLIT ? item.n_tile : min(item.n_tile * 2 + (lane & 1), sfb_rows - 1);
      const float* sfb = p.sfb + (size_t(item.group) * sfb_rows + sfb_row) * p.b_k_blocks;
      for (int kb = 0; ok && kb < k_count; ++kb, ++it) {
        ok = it < kScaleAhead || mbar_wait(&sh->empty[at.slot()], at.phase() ^ 1, abort_flag, p.status, kStatusWaitSmemEmpty);
        if (!ok) break;
        int a_col = k_begin + kb, b_col = k_begin + kb;
        if (p.interleave_hi_lo) { a_col = (kb & 1) * (p.k_blocks >> 1) + (kb >> 1); b_col = kb >> 1; }
        const float* sfa = p.sfa + size_t(a_col) * p.row_capacity;
        const int slot = it % kScaleSlots;
#pragma unroll
        for (int j = 0; j < kBM; j += 32)
          if (MODE == kDense || j < item.rows_valid) cp_async_4(&sh->scale_a[slot][j + lane], sfa + min(item.row0 + j + lane, p.row_capacity - 1));
        if (lane < 2) cp_async_4(&sh->scale_b[slot][lane], sfb + b_col);
        if (it >= kScaleAhead) { cp_async_arrive_noinc(&sh->full[at.slot()]); at.next(); }
      }
    }
    for (uint32_t j = it < kScaleAhead ? 0 : it - kScaleAhead; ok && j < it; ++j, at.next()) {       // the last blocks announce no further scales
      ok = mbar_wait(&sh->empty[at.slot()], at.phase() ^ 1, abort_flag, p.status, kStatusWaitSmemEmpty);
      if (ok) cp_async_arrive_noinc(&sh->full[at.slot()]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  if (SPLIT) { cluster_sync(); cluster_sync(); }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
    // ------------------------------ epilogue / promotion ------------------------------
    if (MODE == kDense) asm volatile("griddepcontrol.wait;" ::: "memory");
    const int ew = warp - kControlWarps;
    const int quad = warp & 3;                 // TMEM lanes a warp may read: 32*(warp id % 4)
    const int cg = ew >> 2;                    // column group 0..1
    const uint32_t lane_base = tmem_base + (uint32_t(quad * 32) << 16);
    uint32_t it = 0, k = 0;
    uint32_t exchanges = 0;                    // amax exchanges so far (phase of Shared::exchange_done)
    int parity = 0;
    bool ok = true, met = false;               // met: SPLIT, this thread has been at the cluster's barriers
    Item item;
    // One item of a tile of R rows.  256 / R threads share a row, R columns each: thread `part` has the tile's columns
    // [part R, part R + R), or, gate/up, x1 and x2 of features [part R / 2, part R / 2 + R / 2).
    auto run_item = [&](auto rows_tag) {
      constexpr int R = decltype(rows_tag)::value;
      const int r = R == 128 ? quad * 32 + lane : R == 64 ? (quad & 1) * 32 + lane : lane;       // row inside the tile
      const int part = R == 128 ? cg : R == 64 ? (quad >> 1) * 2 + cg : quad * 2 + cg;
      const int first_r = r - lane;            // the warp's first row
      const int row = item.row0 + r;
      float w = 1.f;                            // asked for here, a round trip to L2 before the K blocks end
      if (MODE == kDown && r < item.rows_valid) w = __ldg(p.row_weight + row);
      uint64_t acc2[R / 2];                     // R fp32 accumulators as packed pairs
#pragma unroll
      for (int i = 0; i < R / 2; ++i) acc2[i] = 0;
      float sa = 0.f, sb0 = 0.f, sb1 = 0.f;    // scales of the coming block
      auto read_scales = [&](uint32_t block) {
        sa = sh->scale_a[block % kScaleSlots][r];
        sb0 = sh->scale_b[block % kScaleSlots][MODE == kGateUp || SPLIT ? 0 : part * R / 128];
        if (MODE == kGateUp) sb1 = sh->scale_b[block % kScaleSlots][1];
      };
      if (it > 0) read_scales(it);
      for (int kb = 0; kb < k_count; ++kb, ++it) {
        const int t = it % kTmemStages;
        ok = mbar_wait(&sh->tmem_full[t], (it / kTmemStages) & 1, abort_flag, p.status, kStatusWaitTmemFull);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t stage_addr = lane_base + t * kCols;
        if (it == 0) read_scales(0);
        const float s0 = sa * sb0, s1 = MODE == kGateUp ? sa * sb1 : s0;
        const uint64_t s0p = pack_f32x2(s0, s0), s1p = pack_f32x2(s1, s1);
        if constexpr (R == 128) {
          // two round trips to tensor memory per K block, 64 columns each: gate/up takes 64 x1 columns and the matching 64 x2
          // columns; the other modes take 128 consecutive columns (64 where CTAs share K)
          const int seg_col0 = MODE == kGateUp || SPLIT ? cg * 64 : cg * 128;
          const int seg_col1 = MODE == kGateUp ? 128 + cg * 64 : cg * 128 + 64;
          uint64_t v[32];
          tmem_ld_wait_64(stage_addr + seg_col0, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) acc2[i] = fma_f32x2(v[i], s0p, acc2[i]);
          if (!SPLIT) tmem_ld_wait_64(stage_addr + seg_col1, v);
          tcgen05_fence_before();            // everything this warp needs has left tensor memory
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->tmem_empty[t]);
          if (kb + 1 < k_count) read_scales(it + 1);
          if (SPLIT) continue;                   // 64 columns to a thread
#pragma unroll
          for (int i = 0; i < 32; ++i) acc2[32 + i] = fma_f32x2(v[i], s1p, acc2[32 + i]);
        } else {
          uint64_t v[R / 2];
          if constexpr (R == 64) tmem_ld_wait_64(stage_addr + cg * 64, v);
          else tmem_ld_wait_2x16(stage_addr + cg * (MODE == kGateUp ? 16 : 32), stage_addr + (MODE == kGateUp ? 32 + cg * 16 : cg * 32 + 16), v);
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->tmem_empty[t]);
          if (kb + 1 < k_count) read_scales(it + 1);
#pragma unroll
          for (int i = 0; i < R / 2; ++i) acc2[i] = fma_f32x2(v[i], i < R / 4 ? s0p : s1p, acc2[i]);
        }
      }
      if (SPLIT) {
        // This CTA's products are done, so its operand ring is idle: the sums go there, [chunk of 4 columns][row], and every
        // CTA reads its own columns of all of them.  Each starts with its own part and goes round from there, so that the
        // CTAs of a cluster read from different ones at a time (pushed to their owners, all in the same order, the sums took
        // 14 us at eight CTAs).
        const int chunks = 32 / int(split);
        float4* sums = reinterpret_cast<float4*>(tiles);
        if (ok) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float4 v;
            unpack_f32x2(acc2[2 * i], v.x, v.y);
            unpack_f32x2(acc2[2 * i + 1], v.z, v.w);
            sums[(cg * 16 + i) * kBM + r] = v;
          }
        }
        cluster_sync();
        if (ok) {
          const int rows = (item.rows_valid + 31) & ~31, column0 = item.n_tile * kCols + int(rank) * chunks * 4;
          for (int i = threadIdx.x - kControlWarps * 32; i < rows * chunks / 2; i += kEpilogueWarps * 32) {
            const int row_i = i % rows, c = i / rows * 2;
            const uint32_t from = smem_u32(sums + (int(rank) * chunks + c) * kBM + row_i);
            float4 v[kMaxSplit][2];
#pragma unroll
            for (int k = 0; k < kMaxSplit; ++k)
              if (k < int(split)) {
                const uint32_t peer = (rank + k) & (split - 1);
                v[k][0] = load_cluster(from, peer);
                v[k][1] = load_cluster(from + kBM * 16, peer);
              }
            float4 sum[2] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int k = 0; k < kMaxSplit; ++k)
              if (k < int(split))
#pragma unroll
                for (int h = 0; h < 2; ++h) { sum[h].x += v[k][h].x; sum[h].y += v[k][h].y; sum[h].z += v[k][h].z; sum[h].w += v[k][h].w; }
            if (row_i < item.rows_valid && column0 + c * 4 < p.n)
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + size_t(item.row0 + row_i) * p.n + column0 + c * 4) =
                  make_uint4(pack_bf16x2(sum[0].x, sum[0].y), pack_bf16x2(sum[0].z, sum[0].w), pack_bf16x2(sum[1].x, sum[1].y), pack_bf16x2(sum[1].z, sum[1].w));
          }
        }
        cluster_sync();                          // the sums stay until every CTA of the cluster has read them
        met = true;
        return;
      }
      if (!ok) return;
      float acc[R];
#pragma unroll
      for (int i = 0; i < R / 2; ++i) unpack_f32x2(acc2[i], acc[2 * i], acc[2 * i + 1]);
      if (MODE == kDense || MODE == kDown) {
        uint8_t* out = reinterpret_cast<uint8_t*>(reinterpret_cast<__nv_bfloat16*>(p.out) + size_t(item.row0 + first_r) * p.n + item.n_tile * kBN + part * R);
        // rows past the group's end and, where N is an odd multiple of 128, the tile's second 128 columns hold nothing
        const int rows = item.n_tile * kBN + part * R < p.n ? item.rows_valid - first_r : 0;
#pragma unroll
        for (int c = 0; c < R / 32; ++c) {       // 32 columns = 64 bytes of each row at a time
          uint4 v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float* a = acc + c * 32 + i * 8;
            v[i].x = pack_bf16x2(a[0] * w, a[1] * w); v[i].y = pack_bf16x2(a[2] * w, a[3] * w);
            v[i].z = pack_bf16x2(a[4] * w, a[5] * w); v[i].w = pack_bf16x2(a[6] * w, a[7] * w);
          }
          warp_store_64(sh->out_rows[ew], v, out + c * 64, size_t(p.n) * 2, rows, lane);
        }
      } else {
        // SwiGLU on the R / 2 (x1, x2) pairs this thread holds, then e4m3 quantisation of the 128-wide
        // group it shares with the other threads of the same row.
        // Nothing overlaps it but the two blocks the tensor core is ahead, so its length counts in full: 8700 clocks (11100
        // with the second term) with the gate's quotient by `/` and one e4m3 value taken back at a time, against 900 a K
        // block.  The first GEMM of 2500 tokens, hidden 2048, 128 experts of 768, two terms: 204 us then, 163 now.
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
          acc[i] *= silu(acc[R / 2 + i]);
          amax = fmaxf(amax, fabsf(acc[i]));
        }
        const int out_kb = p.n / 128;                      // K blocks of one term of the output
        const int terms = p.split_act ? 2 : 1;
        const size_t out_stride = size_t(p.n) * terms;
        uint8_t* out = reinterpret_cast<uint8_t*>(p.out) + size_t(item.row0 + first_r) * out_stride + item.n_tile * 128 + part * (R / 2);
        for (int term = 0; term < terms; ++term, ++exchanges) {
          // The threads of a row meet through shared memory.  The hand-over is an mbarrier wait like
          // every other wait of the kernel: bounded, and given up when another role has raised the abort flag.
          float* const exchange = sh->exchange[parity][term];
          exchange[part * R + r] = amax;
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->exchange_done);
          ok = mbar_wait(&sh->exchange_done, exchanges & 1, abort_flag, p.status, kStatusWaitFlag);
          if (!ok) break;
          float group_amax = amax;
#pragma unroll
          for (int i = 0; i < 256 / R; ++i) group_amax = fmaxf(group_amax, exchange[i * R + r]);
          const float scale = group_amax > 0.f ? group_amax / 448.f : 1.f;
          const float inv = 1.f / scale;
          uint32_t packed[R / 8];
#pragma unroll
          for (int i = 0; i < R / 2; i += 4) packed[i >> 2] = pack_e4m3x4(acc[i] * inv, acc[i + 1] * inv, acc[i + 2] * inv, acc[i + 3] * inv);
          uint4 v[R / 32];
#pragma unroll
          for (int i = 0; i < R / 32; ++i) v[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
          uint8_t* const dst = out + size_t(term) * p.n;
          if constexpr (R == 128) {
            warp_store_64(sh->out_rows[ew], v, dst, out_stride, item.rows_valid - first_r, lane);
          } else if (r < item.rows_valid) {
#pragma unroll
            for (int i = 0; i < R / 32; ++i) reinterpret_cast<uint4*>(dst + size_t(lane) * out_stride)[i] = v[i];
          }
          if (r < item.rows_valid && part == 0) p.out_scale[size_t(term * out_kb + item.n_tile) * p.row_capacity + row] = scale;
          if (term + 1 < terms) {        // residual after the first term becomes the value to quantise
            amax = 0.f;
#pragma unroll
            for (int i = 0; i < R / 2; i += 2) {
              const float2 first = e4m3x2_to_float2(uint16_t(packed[i >> 2] >> ((i & 2) * 8)));
              acc[i] -= first.x * scale;
              acc[i + 1] -= first.y * scale;
              amax = fmaxf(amax, fmaxf(fabsf(acc[i]), fabsf(acc[i + 1])));
            }
          }
        }
      }
    };
    for (int g = first_item; ok && !met; g += gridDim.x, parity ^= 1, ++k) {
      if (handed) {                    // the k-th item of this CTA, from the TMA warp
        const int slot = k % kItemSlots;
        ok = mbar_wait(&sh->item_full[slot], (k / kItemSlots) & 1, abort_flag, p.status, kStatusWaitFlag);
        if (!ok) break;
        const int4 v = sh->item[slot];
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->item_empty[slot]);
        if (v.x < 0) break;
        item.group = v.x; item.row0 = v.y; item.rows_valid = v.z; item.n_tile = v.w;
      } else if (!locate(sh, p, n_tiles, g, &item)) {
        break;
      }
      const int m = tile_rows<MODE>(item.rows_valid);
      if (m == kBM) run_item(std::integral_constant<int, 128>());
      if constexpr (MODE != kDense) {
        if (m == 64) run_item(std::integral_constant<int, 64>());
        if (m == 32) run_item(std::integral_constant<int, 32>());
      }
    }
    if (SPLIT && !met) { cluster_sync(); cluster_sync(); }
  }

  // ------------------------------ teardown ---------------------------------------------
  tcgen05_fence_before();
  __syncthreads();
  if (sh->wait.abort_flag) {
    settle_after_abort();
    __syncthreads();
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kTmemColumns);
  }
}

constexpr size_t kSmemBytes = size_t(kRingBytes) + sizeof(Shared) + 1024;
static_assert(kSmemBytes <= 232448, "the kernel's shared memory exceeds what a CTA may have on sm_100");

}  // namespace gemm
}  // namespace cake
