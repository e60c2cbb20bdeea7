// Causal GQA prefill for sm_100a: query tiles against shared KV tiles on tcgen05 (flash attention).
//
// Operator: the prefill branches of src/open_cake_ir/tasks/solx_fib/attention.py:132-183 (attention_specs.py:85-248), see
// prefill.cuh for the masking rules.  A unit of work is one KV head and a tile of consecutive query tokens of one segment; the
// G = Hq/Hkv query heads that share the KV head are packed beside the tokens as rows, 128 / G tokens to an M = 128 tile,
// two such tiles (A and B) to a CTA, so a 128-token K/V tile brought into shared memory serves 256 rows.
//   S[128 x 128]  = Q . K^T      both from shared memory, K-major
//   O[128 x 128] += P . V        P from tensor memory, V read MN-major (as it lies)
// Tensor memory: S_A, S_B, O_A, O_B, 128 columns each.  P is two bf16 terms (value + rounding residual: one term alone is
// not accurate enough for the contract's tolerance), 64 + 64 columns, and overwrites the logits it was made from.
//
// What bounds it: the tensor pipe.  A 128 x 128 tile of (row, KV row) pairs costs about 870 clocks for S (operands from
// shared memory) and 1060 for the two terms of P V; the softmax of a tile needs 1024 clocks of the special-function unit
// and about 750 issue slots per warp.  Two row tiles with a softmax warpgroup each keep the pipe busy: the products of
// one run while the other's softmax does ([P V of A(j), S of A(j+1)], [P V of B(j), S of B(j+1)], ...).
// Running each query token as a decode sequence of its own read every KV row once per query token instead.
// A unit goes through its KV tiles one after another (2 to 3 us each), so a unit that alone would take longer than an even share of
// the launch's KV tiles, a few query rows behind a long prefix, is cut into pieces of consecutive KV tiles; these leave partial results,
// which merge_kernel puts together.
// Roles: warp 0 issues the products, warps 4..7 gather Q, K and V rows (cp.async through the page table, any page size; the
// copies announce themselves on the stage's barrier), warps 8..11 and 12..15 are the softmax of tiles A and B.  Every wait
// is bounded and reports through the status word.
#pragma once
#include "common.cuh"
#include <climits>

namespace cake {
namespace gqa_prefill {

constexpr int kD = 128;                          // head dimension
constexpr int kRows = 128;                       // rows of a query tile = TMEM lanes
constexpr int kTile = 128;                       // KV rows per tile
constexpr int kStages = 2;                       // K and V ring depth (each)
constexpr int kSlabBytes = 128 * 128;            // 128 rows x 64 elements
constexpr int kTileBytes = 2 * kSlabBytes;       // 32 KiB: 128 rows of 128 bf16
constexpr int kLoaderWarp0 = 4, kLoaderWarps = 4;      // warp 0 issues the products; warps 1..3 only take part in the barriers
constexpr int kSoftmaxWarp0 = 8;                 // two warpgroups: warp % 4 = TMEM lane quadrant
constexpr int kThreads = 512;
constexpr int kControlRegs = 72, kSoftmaxRegs = 184;
static_assert(256 * kControlRegs + 256 * kSoftmaxRegs <= (65536 / kThreads / 8 * 8) * kThreads, "setmaxnreg budget exceeds the launch's registers");
constexpr uint32_t kColS = 0, kColO = 256, kTmemColumns = 512;        // tile X: S at kColS + 128 X, O at kColO + 128 X
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleThreshold = 8.f;         // log2 units: O is rescaled when the running maximum grows by more
constexpr int kCostBuckets = 1024;
// KV tiles of a piece at least, and by how many a piece has to be shorter than its tile: the merge takes 5 us and more.
constexpr int kMinPiece = 2, kMinGain = 4;
constexpr int kMaxSms = 192;                     // what the workspace is sized for

struct Params {
  const __nv_bfloat16 *q, *k, *v;                // [total_q, Hq, D], [rows, Hkv, D]
  const int *qo_indptr, *kv_indptr, *kv_indices, *last_page_len;      // kv_indices null: ragged; last_page_len null: pages full
  const float* sm_scale;
  __nv_bfloat16* out;
  float* lse;
  int4* tiles;                                   // [capacity] {first query row, rows, KV rows the first one sees (may be < 1), KV rows of the segment}
  int4* spans;                                   // [capacity] {where the segment's page list starts, first KV tile, KV tile behind the last, slot of the partial result (-1: whole)}
  int4* cuts;                                    // [2 * cut_capacity] tiles that are cut: {as in `tiles`}, {first slot, pieces}
  int* tile_count;                               // [2] entries of `tiles`, cut tiles
  float *part_o, *part_lse;                      // [cut_capacity, Hkv, part_rows, D] normalised, [cut_capacity, Hkv, part_rows] base 2
  int* prefix;                                   // [segments + 3] tiles before a segment
  int* status;
  int total_q, segments, hq, hkv, group, page_size, nan_for_masked, capacity, wait_kiloclocks;
  int sms, cut_capacity, part_rows;              // cut_capacity: pieces of cut tiles at most (0: nothing is cut)
  int skip_load;                                 // test hook: CTA 0's loader warps leave out the second K tile of their first unit
};

struct Shared {
  uint64_t k_full[kStages], k_empty[kStages], v_full[kStages], v_empty[kStages];
  uint64_t q_full[2], q_empty[2], s_full[2], p_ready[2][2], o_done[2];     // per query tile; p_ready: per half of P
  uint32_t tmem_base;
  WaitControl wait;
};
constexpr int kOutBytes = 8 * 32 * 128;          // per softmax warp: 32 rows of 128 bytes on their way out
constexpr size_t kSmemBytes = size_t(2 + 2 * kStages) * kTileBytes + kOutBytes + sizeof(Shared) + 1024;
static_assert(kSmemBytes <= 232448, "the kernel's shared memory exceeds what a CTA may have on sm_100");

inline int tokens_per_tile(int group) { return 2 * (kRows / group); }
inline int tile_capacity(int64_t total_q, int64_t segments, int group, int cuts) { return int(total_q / tokens_per_tile(group) + segments + 3) + cuts; }
inline int part_rows(int64_t total_q, int group) { return total_q <= kRows / group ? int(total_q) * group : 2 * kRows; }      // one query tile or two

// One CTA: cuts the query rows of every segment into tiles and lists them, most KV tiles first, so that the CTAs that start
// last are the short ones.  Rows outside every segment form two more segments without KV rows (they become zeros).  With `sms`
// CTAs and N KV tiles in all, for each KV head, a tile of n goes to floor(n sms / (N Hkv)) pieces, about an even share each, where that
// is shorter by enough to pay for the merge; no more pieces than sms / Hkv in all.
static __global__ void __launch_bounds__(1024)
plan_kernel(const Params p) {
  __shared__ int sums[32];
  __shared__ int bucket[kCostBuckets];
  __shared__ int cut_tile[kMaxSms], cut_first[kMaxSms], cut_size[kMaxSms], cut_count;      // cut_count: cut tiles << 16 | their pieces
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tid = threadIdx.x;
  const int per = 2 * (kRows / p.group);
  const int rows_end = p.qo_indptr[p.segments];
  auto segment = [&](int b, int* qs, int* qe) {
    if (b < p.segments) { *qs = p.qo_indptr[b]; *qe = p.qo_indptr[b + 1]; }
    else if (b == p.segments) { *qs = rows_end; *qe = p.total_q; }
    else { *qs = 0; *qe = p.qo_indptr[0]; }
  };
  const int count = p.segments + 2;
  bucket[tid] = 0;
  if (tid == 0) cut_count = 0;
  int before = 0;
  for (int base = 0; base < count; base += 1024) {
    const int b = base + tid;
    int qs = 0, qe = 0, all;
    if (b < count) segment(b, &qs, &qe);
    const int n = qe > qs ? (qe - qs + per - 1) / per : 0;
    const int mine = before + cta_exclusive_scan<32>(n, sums, all);
    if (b < count) p.prefix[b] = mine;
    before += all;
  }
  const int total = min(before, p.capacity - p.cut_capacity);
  __syncthreads();
  auto describe = [&](int t, int4* tile, int* page) {      // returns the tile's KV tiles
    int lo = 0, hi = count;                      // largest b with prefix[b] <= t
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (p.prefix[mid] <= t) lo = mid; else hi = mid;
    }
    int qs, qe;
    segment(lo, &qs, &qe);
    const int i = (t - p.prefix[lo]) * per;
    int kv_len = 0;
    *page = 0;
    if (lo < p.segments) {
      *page = p.kv_indptr[lo];
      const int units = p.kv_indptr[lo + 1] - *page;
      kv_len = units <= 0 ? 0 : p.last_page_len ? (units - 1) * p.page_size + p.last_page_len[lo] : units * p.page_size;
    }
    *tile = make_int4(qs + i, min(per, qe - qs - i), i + 1 + kv_len - (qe - qs), kv_len);
    const int last = min(kv_len, tile->z + tile->y - 1);
    return last > 0 ? (last + kTile - 1) / kTile : 0;
  };
  int4 tile, tile0;
  int page, page0;
  const int n0 = tid < total ? describe(tid, &tile0, &page0) : 0;      // the first 1024 tiles stay in registers
  float share = 0;                               // KV tiles of the launch, over all heads, to an SM
  if (p.cut_capacity) {
    int mine = n0, all;
    for (int t = tid + 1024; t < total; t += 1024) mine += describe(t, &tile, &page);
    cta_exclusive_scan<32>(mine, sums, all);
    share = float(all) * float(p.hkv) / float(p.sms) * 1.0001f;        // (rounding may leave a piece out, never make one more)
  }
  auto size_of = [&](int n) {                    // KV tiles of a tile's pieces
    if (share == 0.f || float(n) < 2.f * share) return n;
    const int k = min(int(float(n) / share), n / kMinPiece), size = (n + k - 1) / k;
    return n - size >= kMinGain ? size : n;
  };
  auto bucket_of = [&](int n) { return kCostBuckets - 1 - min(kCostBuckets - 1, n); };
  auto count_tile = [&](int t, int n, const int4& tile) {
    const int size = size_of(n), pieces = n > size ? (n + size - 1) / size : 1;
    atomicAdd(bucket + bucket_of(size), pieces);
    if (pieces > 1) {
      const int at = atomicAdd(&cut_count, (1 << 16) + pieces), c = at >> 16;
      cut_tile[c] = t; cut_first[c] = at & 0xffff; cut_size[c] = size;
      p.cuts[2 * c] = tile;
      p.cuts[2 * c + 1] = make_int4(at & 0xffff, pieces, 0, 0);
    }
  };
  if (tid < total) count_tile(tid, n0, tile0);
  for (int t = tid + 1024; t < total; t += 1024) { const int n = describe(t, &tile, &page); count_tile(t, n, tile); }
  __syncthreads();
  int all;
  const int mine = bucket[tid];
  const int start = cta_exclusive_scan<32>(mine, sums, all);
  bucket[tid] = start;
  __syncthreads();
  auto list_tile = [&](int n, const int4& tile, int page) {
    if (size_of(n) < n) return;
    const int at = atomicAdd(bucket + bucket_of(n), 1);
    p.tiles[at] = tile;
    p.spans[at] = make_int4(page, 0, n, -1);
  };
  if (tid < total) list_tile(n0, tile0, page0);
  for (int t = tid + 1024; t < total; t += 1024) { const int n = describe(t, &tile, &page); list_tile(n, tile, page); }
  const int cuts = cut_count >> 16, pieces = cut_count & 0xffff;
  for (int e = tid; e < pieces; e += 1024) {     // the pieces of the cut tiles, a thread each
    int lo = 0, hi = cuts;                       // largest c with cut_first[c] <= e
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (cut_first[mid] <= e) lo = mid; else hi = mid;
    }
    const int n = describe(cut_tile[lo], &tile, &page), size = cut_size[lo], first = (e - cut_first[lo]) * size;
    const int at = atomicAdd(bucket + bucket_of(size), 1);
    p.tiles[at] = tile;
    p.spans[at] = make_int4(page, first, min(n, first + size), e);
  }
  if (tid == 0) { p.tile_count[0] = all; p.tile_count[1] = cuts; *p.status = 0; }
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;              // 0 source bytes = zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// Byte offset of 16-byte chunk `chunk` (0..15) of row `row`: two slabs of 64 columns with the 128-byte swizzle.
__device__ __forceinline__ uint32_t row_off(int row, int chunk) {
  return uint32_t((chunk >> 3) * kSlabBytes + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
}

// One unit of work as every role reads it from the list.
struct Work {
  int q0, rows, first_visible, kv_len, page_base, kvh;
  int begin, slot;                                 // first KV tile; where a piece of a cut tile leaves its result (-1: whole)
  int n_kv[2], n;                                  // KV tiles of it that each query tile sees; the larger of the two
};
// The k-th unit of this CTA, false past the end.  CTA c takes entries c, 2g-1-c, 2g+c, ... of the (tile, KV head) list, which
// is sorted by length: turning round every other time evens out what a CTA gets.
template <bool CUT>
__device__ __forceinline__ bool get_work(const Params& p, int units, int k, Work* w) {
  const int g = gridDim.x;
  const int u = k * g + ((k & 1) ? g - 1 - int(blockIdx.x) : int(blockIdx.x));
  if (u >= units) return false;
  const int index = u / p.hkv;
  w->kvh = u - index * p.hkv;
  const int4 tile = __ldg(p.tiles + index);
  int4 span = make_int4(0, 0, INT_MAX, -1);
  if (CUT) span = __ldg(p.spans + index);
  else span.x = __ldg(&p.spans[index].x);
  w->page_base = span.x; w->begin = span.y; w->slot = span.w;
  w->q0 = tile.x; w->rows = tile.y; w->first_visible = tile.z; w->kv_len = tile.w;
  const int per_half = kRows / p.group;
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int mine = min(w->rows - x * per_half, per_half);
    const int last = mine > 0 ? min(w->kv_len, w->first_visible + x * per_half + mine - 1) : 0;
    w->n_kv[x] = last > 0 ? (last + kTile - 1) / kTile : 0;
    if (CUT) w->n_kv[x] = max(0, min(span.z, w->n_kv[x]) - span.y);
  }
  w->n = max(w->n_kv[0], w->n_kv[1]);
  return true;
}

// The tensor core multiplies every V row of a tile with a weight, the masked ones with 0, and 0 times an infinity or a NaN is
// NaN.  For a row whose O is not finite this looks at the V rows that its tiles hold and it does not see, [visible, loaded),
// and where one of them is not finite, writes the row again from the KV rows that it does see, [begin, visible), with the same maximum
// (to `part` where it is a piece's).  By a whole warp: lane i has dims [4 i, 4 i + 4).  Rare, and out of line for the registers of the loop.
static __device__ __noinline__ void without_masked_rows(const Params& p, int q_row, int head, int kvh, int page_base, int begin, int visible, int loaded,
                                                        float scale2, float m, float by, float* part) {
  const int lane = threadIdx.x & 31;
  auto row4 = [&](const __nv_bfloat16* rows, size_t row) {
    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(rows + row * kD) + lane);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
  };
  auto kv_row = [&](int t) {
    return size_t(p.kv_indices ? __ldg(p.kv_indices + page_base + t / p.page_size) * p.page_size + t % p.page_size : page_base + t) * p.hkv + kvh;
  };
  float spread = 0.f;                              // NaN once an element is not finite
  for (int t = visible; t < loaded; ++t) {
    const float4 v = row4(p.v, kv_row(t));
    spread = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, spread))));
  }
  if (!__any_sync(0xffffffffu, spread != spread)) return;
  const float4 q = row4(p.q, size_t(q_row) * p.hq + head);
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int t = begin; t < visible; ++t) {
    const size_t at = kv_row(t);
    const float4 k = row4(p.k, at), v = row4(p.v, at);
    const float w = ex2(fmaf(warp_sum(q.x * k.x + q.y * k.y + q.z * k.z + q.w * k.w), scale2, -m));
    o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w);
  }
  if (part) reinterpret_cast<float4*>(part)[lane] = make_float4(o.x * by, o.y * by, o.z * by, o.w * by);
  else reinterpret_cast<uint2*>(p.out + (size_t(q_row) * p.hq + head) * kD)[lane] = make_uint2(pack_bf16x2(o.x * by, o.y * by), pack_bf16x2(o.z * by, o.w * by));
}

// The sum of 32 values on top of a pair of sums: not finite once a value is not.
__device__ __forceinline__ uint64_t sum_32(const float (&o)[32], uint64_t sum) {
  uint64_t s[4] = {sum, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 16; ++i) s[i & 3] = add_f32x2(s[i & 3], pack_f32x2(o[2 * i], o[2 * i + 1]));
  return add_f32x2(add_f32x2(s[0], s[1]), add_f32x2(s[2], s[3]));
}

// The rows of a cut tile's piece, each lane its own (null: no such row); returns the sum as sum_32 does.  Out of line: most units are whole.
static __device__ __noinline__ uint64_t write_part(uint32_t o_col, int tiles, float* part, float inv) {
  uint64_t sum = 0;
#pragma unroll 1
  for (int c = 0; c < kD; c += 32) {
    float o[32];
    if (tiles > 0) {
      tmem_ld_32x32b_x32(o_col + c, o);
      tcgen05_wait_ld();
    }
    sum = sum_32(o, sum);
    if (part) {
#pragma unroll
      for (int i = 0; i < 32; i += 4)
        *reinterpret_cast<float4*>(part + c + i) = inv == 0.f ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
    }
    __syncwarp();
  }
  return sum;
}

// CUT: some tiles may be cut.
template <bool CUT>
__global__ void __launch_bounds__(kThreads, 1)
prefill_kernel(const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t q_addr = smem_u32(base), k_addr = q_addr + 2 * kTileBytes, v_addr = k_addr + kStages * kTileBytes;
  uint8_t* out_rows = base + (2 + 2 * kStages) * kTileBytes;
  Shared* sh = reinterpret_cast<Shared*>(out_rows + kOutBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&sh->k_full[s], kLoaderWarps * 32); mbar_init(&sh->k_empty[s], 1);
      mbar_init(&sh->v_full[s], kLoaderWarps * 32); mbar_init(&sh->v_empty[s], 1);
    }
    for (int x = 0; x < 2; ++x) {
      mbar_init(&sh->q_full[x], kLoaderWarps * 32); mbar_init(&sh->q_empty[x], 1);
      mbar_init(&sh->s_full[x], 1); mbar_init(&sh->o_done[x], 1);
      mbar_init(&sh->p_ready[x][0], 4); mbar_init(&sh->p_ready[x][1], 4);
    }
    sh->wait.abort_flag = 0;
    sh->wait.budget_kiloclocks = p.wait_kiloclocks;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&sh->tmem_base, kTmemColumns);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  volatile int* abort_flag = &sh->wait.abort_flag;
  const int per_half = kRows / p.group;            // query tokens per M tile
  // launched as a programmatic dependent of the plan kernel: the list is read only after that grid has completed
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int units = *p.tile_count * p.hkv;

  if (warp < kSoftmaxWarp0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kControlRegs));
    if (warp == 0) {
      // ------------------------------ MMA issuer --------------------------------------
      if (elect_one()) {
        constexpr uint32_t idesc_qk = umma_idesc_ex(1 /* bf16 */, kRows, kTile, 0, 0);
        constexpr uint32_t idesc_pv = umma_idesc_ex(1 /* bf16 */, kRows, kD, 0, 1 /* V is MN-major */);
        bool ok = true;
        uint32_t it = 0;                           // KV tiles so far
        uint32_t products[2] = {0, 0}, loads[2] = {0, 0};      // per query tile: KV tiles and Q blocks so far
        Work w;
        auto issue_qk = [&](int x, uint32_t i) {
          const uint64_t a = umma_desc_sw128(q_addr + x * kTileBytes), b = umma_desc_sw128(k_addr + (i % kStages) * kTileBytes);
#pragma unroll
          for (int step = 0; step < kD / 16; ++step) {
            const uint64_t off = uint64_t(((step >> 2) * kSlabBytes + (step & 3) * 32) >> 4);
            umma_f16(tmem_base + kColS + x * kTile, a + off, b + off, idesc_qk, step != 0);
          }
          tcgen05_commit(&sh->s_full[x]);
        };
        auto k_ready = [&](uint32_t i) {
          ok = mbar_wait(&sh->k_full[i % kStages], (i / kStages) & 1, abort_flag, p.status, kStatusWaitSmemFull);
          fence_proxy_async_smem();                // the rows were written through the generic proxy
          tcgen05_fence_after();
        };
        for (int k = 0; ok && get_work<CUT>(p, units, k, &w); ++k) {
          if (w.n == 0) continue;
          k_ready(it);
#pragma unroll 1
          for (int x = 0; ok && x < 2; ++x) {
            if (w.n_kv[x] == 0) continue;
            ok = mbar_wait(&sh->q_full[x], loads[x]++ & 1, abort_flag, p.status, kStatusWaitSmemFull);
            if (!ok) break;
            fence_proxy_async_smem();
            issue_qk(x, it);
            if (w.n_kv[x] == 1) tcgen05_commit(&sh->q_empty[x]);
          }
          if (!ok) break;
          tcgen05_commit(&sh->k_empty[it % kStages]);
          for (int j = 0; ok && j < w.n; ++j, ++it) {
            const int s = it % kStages;
            ok = mbar_wait(&sh->v_full[s], (it / kStages) & 1, abort_flag, p.status, kStatusWaitSmemFull);
            if (!ok) break;
            fence_proxy_async_smem();
            const uint64_t v_base = umma_desc_sw128_ex(v_addr + s * kTileBytes, kSlabBytes, 1024);
            bool k_waited = false;
#pragma unroll 1
            for (int x = 0; ok && x < 2; ++x) {
              if (j >= w.n_kv[x]) continue;
              // P comes in two halves of 64 KV rows, so that the product starts while the second half is being made
#pragma unroll
              for (int half = 0; half < 2; ++half) {
                ok = ok && mbar_wait(&sh->p_ready[x][half], products[x] & 1, abort_flag, p.status, kStatusWaitFlag);
                if (!ok) break;
                tcgen05_fence_after();
#pragma unroll
                for (int term = 0; term < 2; ++term)
#pragma unroll
                  for (int ks = half * 4; ks < half * 4 + 4; ++ks)
                    umma_f16_a_tmem(tmem_base + kColO + x * kD, tmem_base + kColS + x * kTile + (ks >> 1) * 32 + term * 16 + (ks & 1) * 8,
                                    v_base + uint64_t((ks * 2048) >> 4), idesc_pv, (j | half | term | (ks & 3)) != 0);
              }
              if (!ok) break;
              ++products[x];
              tcgen05_commit(&sh->o_done[x]);
              // The logits of the next tile go where P of this one lies: the pipe runs one thread's products in order
              if (j + 1 < w.n_kv[x]) {
                if (!k_waited) { k_ready(it + 1); k_waited = true; }
                if (ok) issue_qk(x, it + 1);
                if (ok && j + 2 == w.n_kv[x]) tcgen05_commit(&sh->q_empty[x]);
              }
            }
            if (!ok) break;
            tcgen05_commit(&sh->v_empty[s]);
            if (k_waited) tcgen05_commit(&sh->k_empty[(it + 1) % kStages]);
          }
        }
      }
    } else if (warp >= kLoaderWarp0) {
      // ------------------------------ loader ------------------------------------------
      // Row pairs (two rows of 256 bytes per instruction): a warp takes 32 of a tile's rows, whose pages its lanes look up a
      // tile ahead of their use and hand round by shuffle.
      const int lw = warp - kLoaderWarp0, chunk = lane & 15;
      bool ok = true;
      uint32_t it = 0, loads[2] = {0, 0};
      Work w;
      for (int k = 0; ok && get_work<CUT>(p, units, k, &w); ++k) {
        if (w.n == 0) continue;
        struct Lookup { int page, offset; };       // offset -1: no such token
        auto lookup = [&](int j) -> Lookup {
          const int token = (w.begin + j) * kTile + lw * 32 + lane;
          if (token >= w.kv_len) return {0, -1};
          if (!p.kv_indices) return {0, w.page_base + token};
          const int page = token / p.page_size;
          return {__ldg(p.kv_indices + w.page_base + page), token - page * p.page_size};
        };
        auto resolve = [&](Lookup l) {
          asm volatile("" : "+r"(l.page));         // the page number is not worked on before this point, so the lookup is not waited for
          return l.offset < 0 ? -1 : l.page * p.page_size + l.offset;      // < 2^31 rows
        };
        Lookup ahead = lookup(0);
        // Q rows: token q0 + x * per_half + r / G, head kvh * G + r % G; rows without a token are zeros
        for (int x = 0; ok && x < 2; ++x) {
          if (w.n_kv[x] == 0) continue;
          ok = mbar_wait(&sh->q_empty[x], (loads[x]++ & 1) ^ 1, abort_flag, p.status, kStatusWaitSmemEmpty);
          if (!ok) break;
#pragma unroll 4
          for (int pair = lw * 16; pair < lw * 16 + 16; ++pair) {
            const int r = pair * 2 + (lane >> 4), token = x * per_half + r / p.group;
            const bool valid = r < per_half * p.group && token < w.rows;
            cp_async_16(q_addr + x * kTileBytes + row_off(r, chunk),
                        p.q + (size_t(w.q0 + (valid ? token : 0)) * p.hq + w.kvh * p.group + r % p.group) * kD + chunk * 8, valid);
          }
          cp_async_arrive_noinc(&sh->q_full[x]);
        }
        for (int j = 0; ok && j < w.n; ++j, ++it) {
          const int s = it % kStages;
          const int row = resolve(ahead);
          ahead = j + 1 < w.n ? lookup(j + 1) : Lookup{0, -1};
#pragma unroll
          for (int kv = 0; kv < 2; ++kv) {
            ok = mbar_wait(kv ? &sh->v_empty[s] : &sh->k_empty[s], ((it / kStages) & 1) ^ 1, abort_flag, p.status, kStatusWaitSmemEmpty);
            if (!ok) break;
            if (p.skip_load && blockIdx.x == 0 && it == 1 && kv == 0) continue;      // test hook: never filled
            const __nv_bfloat16* src = (kv ? p.v : p.k) + size_t(w.kvh) * kD + chunk * 8;
            const uint32_t dst = (kv ? v_addr : k_addr) + s * kTileBytes;
#pragma unroll
            for (int pair = 0; pair < 16; ++pair) {
              const int r = pair * 2 + (lane >> 4);
              const int at = __shfl_sync(0xffffffffu, row, r);
              cp_async_16(dst + row_off(lw * 32 + r, chunk), src + size_t(at < 0 ? 0 : at) * p.hkv * kD, at >= 0);
            }
            cp_async_arrive_noinc(kv ? &sh->v_full[s] : &sh->k_full[s]);
          }
          if (!ok) break;
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
    // ------------------------------ softmax / output -------------------------------------
    const int x = (warp - kSoftmaxWarp0) >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;                // row of the query tile = TMEM lane
    const uint32_t lane_base = tmem_base + (uint32_t(quad * 32) << 16);
    const uint32_t s_col = lane_base + kColS + x * kTile, o_col = lane_base + kColO + x * kD;
    const float scale2 = __ldg(p.sm_scale) * kLog2e;
    const bool scale_positive = scale2 > 0.f;      // the contract's scales are; any other is applied to the logits first
    const float pre = scale_positive ? 1.f : scale2, post = scale_positive ? scale2 : 1.f;
    const int token = x * per_half + r / p.group, head_in_group = r % p.group;
    const bool slot = r < per_half * p.group;
    const bool out_aligned = !(reinterpret_cast<uintptr_t>(p.out) & 15);      // the caller's output may lie on any 8-byte boundary
    uint4* scratch = reinterpret_cast<uint4*>(out_rows + (warp - kSoftmaxWarp0) * (32 * 128));
    bool ok = true;
    uint32_t done = 0;                             // KV tiles so far
    Work w;
    for (int k = 0; ok && get_work<CUT>(p, units, k, &w); ++k) {
      const bool exists = slot && token < w.rows;
      const int visible = exists ? min(w.kv_len, w.first_visible + token) : 0;      // KV rows this row sees
      const int seen = visible - w.begin * kTile;  // of the unit's
      const int tiles = x ? w.n_kv[1] : w.n_kv[0];
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < tiles; ++j, ++done) {
        ok = mbar_wait(&sh->s_full[x], done & 1, abort_flag, p.status, kStatusWaitTmemFull);
        if (!ok) break;
        tcgen05_fence_after();
        // The logits are read twice, once for the maximum and once for the weights, 32 columns at a time: all 128 in
        // registers spill.  P of 32 KV rows (16 columns of values, 16 of residuals) goes over the logits it comes from.
        const int limit = seen - j * kTile;        // columns at and past it are masked
        const bool plain = !__any_sync(0xffffffffu, limit < kTile) && scale_positive;
        float t4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < kTile; c += 64) {
          float sc[64];
          tmem_ld_32x32b_x32(s_col + c, sc);
          tmem_ld_32x32b_x32(s_col + c + 32, sc + 32);
          tcgen05_wait_ld();
          if (!plain) {
#pragma unroll
            for (int i = 0; i < 64; ++i) sc[i] = c + i < limit ? sc[i] * pre : -INFINITY;
          }
#pragma unroll
          for (int i = 0; i < 64; i += 8) {
#pragma unroll
            for (int q = 0; q < 4; ++q) t4[q] = max3(t4[q], sc[i + q], sc[i + 4 + q]);
          }
        }
        const float tmax = fmaxf(fmaxf(t4[0], t4[1]), fmaxf(t4[2], t4[3])) * post;
        if (j == 0) {
          m_ref = tmax;
        } else {
          const bool need = tmax > m_ref + kRescaleThreshold;
          if (__any_sync(0xffffffffu, need)) {     // O is about to be rescaled in tensor memory: the product before must have landed
            ok = mbar_wait(&sh->o_done[x], (done - 1) & 1, abort_flag, p.status, kStatusWaitFlag);
            if (!ok) break;
            tcgen05_fence_after();
            const float alpha = need ? exp2f(m_ref - tmax) : 1.f;
            if (need) { m_ref = tmax; l *= alpha; }
#pragma unroll 1
            for (int c = 0; c < kD; c += 16) {
              float o[16];
              tmem_ld_32x32b_x16(o_col + c, o);
              tcgen05_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] *= alpha;
              tmem_st_32x32b_x16(o_col + c, reinterpret_cast<const uint32_t*>(o));
            }
          }
        }
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;       // a row that sees nothing: weights 0, not NaN
        const uint64_t post2 = pack_f32x2(post, post), minus_m = pack_f32x2(-m_use, -m_use), minus_one = pack_f32x2(-1.f, -1.f);
        uint64_t sum2[2] = {0, 0};
#pragma unroll
        for (int c = 0; c < kTile; c += 32) {
          float sc[32];
          tmem_ld_32x32b_x32(s_col + c, sc);
          tcgen05_wait_ld();
          if (!plain) {
#pragma unroll
            for (int i = 0; i < 32; ++i) sc[i] = c + i < limit ? sc[i] * pre : -INFINITY;
          }
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float a, b;
            unpack_f32x2(fma_f32x2(pack_f32x2(sc[2 * i], sc[2 * i + 1]), post2, minus_m), a, b);
            a = ex2(a); b = ex2(b);
            const uint64_t pair = pack_f32x2(a, b);
            sum2[i & 1] = add_f32x2(sum2[i & 1], pair);
            hi[i] = pack_bf16x2(a, b);
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(hi[i] << 16), __uint_as_float(hi[i] & 0xffff0000u)), minus_one, pair), a, b);
            lo[i] = pack_bf16x2(a, b);
          }
          tmem_st_32x32b_x16(s_col + c, hi);
          tmem_st_32x32b_x16(s_col + c + 16, lo);
          if (c & 32) {                            // 64 KV rows of P are complete
            tcgen05_wait_st();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh->p_ready[x][c >> 6]);
          }
        }
        float a, b;
        unpack_f32x2(add_f32x2(sum2[0], sum2[1]), a, b);
        l += a + b;
      }
      if (ok && tiles > 0) ok = mbar_wait(&sh->o_done[x], (done - 1) & 1, abort_flag, p.status, kStatusWaitFlag);
      if (!ok) break;
      tcgen05_fence_after();
      // A sum that is NaN (a NaN, or infinities that met, in what the row sees) goes on as one.  A row that sees KV rows has a
      // weight of at least 2^-8, unless every logit is -inf: 0 / 0, as in the decode form.  Else a zero sum means that it sees nothing (of this piece).
      if (visible > 0 && l == 0.f && w.slot < 0) l = __int_as_float(0x7fc00000);
      // rows leave through shared memory, 128 bytes of a row at a time
      const float inv = l == 0.f ? 0.f : 1.f / l;
      const bool nan = p.nan_for_masked && w.kv_len > 0 && visible <= 0;
      float* part = nullptr;                       // where the row of a cut tile's piece goes
      if (CUT && w.slot >= 0) {
        const size_t row = (size_t(w.slot) * p.hkv + w.kvh) * p.part_rows + x * kRows + r;
        part = p.part_o + row * kD;
        if (exists) p.part_lse[row] = l == 0.f ? -INFINITY : m_ref + log2f(l);
      } else if (exists) {
        p.lse[size_t(w.q0 + token) * p.hq + w.kvh * p.group + head_in_group] = l == 0.f ? -INFINITY : m_ref + log2f(l);
      }
      uint64_t sum = 0;                            // of the row's O, as a pair: not finite once an element is not
      if (CUT && part) sum = write_part(o_col, tiles, exists ? part : nullptr, inv);
#pragma unroll 1
      for (int h = CUT && part ? kD : 0; h < kD; h += 64) {
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          float o[32];
          if (tiles > 0) {
            tmem_ld_32x32b_x32(o_col + h + c, o);
            tcgen05_wait_ld();
          }
          sum = sum_32(o, sum);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 v;
            v.x = pack_bf16x2(o[8 * i] * inv, o[8 * i + 1] * inv); v.y = pack_bf16x2(o[8 * i + 2] * inv, o[8 * i + 3] * inv);
            v.z = pack_bf16x2(o[8 * i + 4] * inv, o[8 * i + 5] * inv); v.w = pack_bf16x2(o[8 * i + 6] * inv, o[8 * i + 7] * inv);
            if (l == 0.f) v = nan ? make_uint4(0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u) : make_uint4(0u, 0u, 0u, 0u);
            scratch[lane * 8 + ((c / 8 + i) ^ (lane & 7))] = v;
          }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = i * 4 + (lane >> 3), chunk = lane & 7;
          const int row_r = quad * 32 + rr, row_token = x * per_half + row_r / p.group;
          if (row_r < per_half * p.group && row_token < w.rows) {
            const uint4 v = scratch[rr * 8 + (chunk ^ (rr & 7))];
            __nv_bfloat16* dst = p.out + (size_t(w.q0 + row_token) * p.hq + w.kvh * p.group + row_r % p.group) * kD + h + chunk * 8;
            if (out_aligned) {
              *reinterpret_cast<uint4*>(dst) = v;
            } else {
              reinterpret_cast<uint2*>(dst)[0] = make_uint2(v.x, v.y);
              reinterpret_cast<uint2*>(dst)[1] = make_uint2(v.z, v.w);
            }
          }
        }
        __syncwarp();
      }
      const int loaded = min(w.kv_len, (w.begin + tiles) * kTile);      // KV row behind the last in the row's products
      float sum_a, sum_b;
      unpack_f32x2(sum, sum_a, sum_b);
      uint32_t again = __ballot_sync(0xffffffffu, seen > 0 && visible < loaded && l == l && !(fabsf(sum_a + sum_b) <= 3.4e38f));
      while (again) {                              // (the row's first result has been written, by this warp)
        const int src = __ffs(again) - 1, row_r = quad * 32 + src, q_row = w.q0 + x * per_half + row_r / p.group, head = w.kvh * p.group + row_r % p.group;
        again &= again - 1;
        without_masked_rows(p, q_row, head, w.kvh, w.page_base, w.begin * kTile, __shfl_sync(0xffffffffu, visible, src), loaded, scale2,
                            __shfl_sync(0xffffffffu, m_ref, src), __shfl_sync(0xffffffffu, inv, src), part ? part + (src - lane) * kD : nullptr);
      }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (sh->wait.abort_flag) {
    settle_after_abort();
    __syncthreads();
  }
  if (warp == 0) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kTmemColumns);
  }
}

// Puts the pieces of cut tiles together: a warp to a row of a (tile, KV head), four dims to a lane, the results of four pieces in flight.
constexpr int kMergeWarps = 8;
static __global__ void __launch_bounds__(kMergeWarps * 32)
merge_kernel(const Params p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, per_half = kRows / p.group;
  const int rows = p.tile_count[1] * p.hkv * p.part_rows;       // <= (sms / Hkv) Hkv 256
  for (int i = blockIdx.x * kMergeWarps + (threadIdx.x >> 5); i < rows; i += gridDim.x * kMergeWarps) {
    const int row = i % p.part_rows, kvh = i / p.part_rows % p.hkv, cut = i / p.part_rows / p.hkv;
    const int4 tile = p.cuts[2 * cut], pieces = p.cuts[2 * cut + 1];
    const int r = row % kRows, token = row / kRows * per_half + r / p.group;
    if (r >= per_half * p.group || token >= tile.y) continue;
    const size_t first = (size_t(pieces.x) * p.hkv + kvh) * p.part_rows + row, stride = size_t(p.hkv) * p.part_rows;
    float mm = -INFINITY, weight = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 < pieces.y; k0 += 4) {
      float ls[4];
      float4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const size_t at = first + size_t(min(k0 + k, pieces.y - 1)) * stride;
        ls[k] = k0 + k < pieces.y ? __ldcg(p.part_lse + at) : -INFINITY;
        v[k] = __ldcg(reinterpret_cast<const float4*>(p.part_o + at * kD) + lane);
      }
      const float m_new = fmaxf(fmaxf(fmaxf(ls[0], ls[1]), fmaxf(ls[2], ls[3])), mm);
      const float rescale = mm == m_new ? 1.f : exp2f(mm - m_new);
      mm = m_new;
      weight *= rescale;
      acc.x *= rescale; acc.y *= rescale; acc.z *= rescale; acc.w *= rescale;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float w = ls[k] == -INFINITY ? 0.f : exp2f(ls[k] - mm);      // -inf: the row sees nothing of the piece; NaN goes on as one
        weight += w;
        acc.x = fmaf(w, v[k].x, acc.x); acc.y = fmaf(w, v[k].y, acc.y); acc.z = fmaf(w, v[k].z, acc.z); acc.w = fmaf(w, v[k].w, acc.w);
      }
    }
    const size_t out_row = size_t(tile.x + token) * p.hq + kvh * p.group + r % p.group;
    const bool sees = min(tile.w, tile.z + token) > 0;
    uint2 packed = make_uint2(0u, 0u);
    float lse = -INFINITY;
    if (weight != 0.f) {
      const float inv = 1.f / weight;
      packed = make_uint2(pack_bf16x2(acc.x * inv, acc.y * inv), pack_bf16x2(acc.z * inv, acc.w * inv));
      lse = mm + log2f(weight);
    } else if (sees || (p.nan_for_masked && tile.w > 0)) {                 // every logit is -inf; or the row sees nothing
      packed = make_uint2(0x7fc07fc0u, 0x7fc07fc0u);
      if (sees) lse = __int_as_float(0x7fc00000);
    }
    reinterpret_cast<uint2*>(p.out + out_row * kD)[lane] = packed;
    if (lane == 0) p.lse[out_row] = lse;
  }
}

}  // namespace gqa_prefill
}  // namespace cake
