// Dense block-scaled FP8 GEMM entry points (C ABI) on top of the shared tcgen05 core.
#include "gemm_fp8.cuh"
#include "gemm_skinny.cuh"
#include "../../include/cake_b200.h"
#include <new>

namespace cake {
namespace {

struct DenseHandle {
  int device;
  CUtensorMap map_a, map_a_tail, map_b;
  gemm::Params params;
  int grid, split;                     // CTAs that share a tile of 128 columns (0: tiles of 256, the whole of K to a CTA)
  int* status;
  int skinny_grid, skinny_tiles, skinny_split;      // few rows: token tiles of eight and K split of skinny_kernel (0: the tcgen05 core)
  skinny::Params skinny;
};

}  // namespace
}  // namespace cake

void cake::gemm_launch_facts(int* threads, int* dynamic_shared_bytes) {
  *threads = cake::gemm::kThreads;
  *dynamic_shared_bytes = int(cake::gemm::kSmemBytes);
}

extern "C" size_t cake_b200_block_scaled_gemm_workspace_bytes(const cake_b200_gemm_config*) { return 256; }

extern "C" int cake_b200_block_scaled_gemm_create(void** buffers, const cake_b200_gemm_config* config,
                                                  void** handle_out) {
  using namespace cake;
  if (!buffers || !config || !handle_out) return kErrBadArgument;
  *handle_out = nullptr;
  int device = 0;
  if (int rc = require_blackwell(&device)) return rc;
  for (int i = 0; i < 6; ++i)
    if (!buffers[i] || (reinterpret_cast<uintptr_t>(buffers[i]) & 15)) return kErrBadArgument;
  const int64_t m = config->m, n = config->n, k = config->k;
  if (m <= 0 || n <= 0 || k <= 0 || (k % gemm::kBK) || (n % 128) || m > INT32_MAX / 2 || n > INT32_MAX / 2)
    return kErrBadArgument;
  auto* h = new (std::nothrow) DenseHandle;
  if (!h) return int(cudaErrorMemoryAllocation);
  h->device = device;
  int rc = make_tensor_map_u8_sw128(&h->map_a, buffers[0], uint64_t(m), uint64_t(k), gemm::kBM);
  if (!rc) rc = make_tensor_map_u8_sw128(&h->map_a_tail, buffers[0], uint64_t(m), uint64_t(k), gemm::kTailRows);
  // Where tiles of 128 columns leave SMs idle, two or four CTAs of a cluster share a tile's K, at least four K blocks each
  // (64 x 4096 x 7168: 28.7 us as 16 tiles of 256 columns, 15.5 at four CTAs to each of them, 12.1 at four CTAs to each of 32
  // tiles of 128; clusters of eight do not all fit the GPU at a time).
  const int sms = sm_count(device), row_tiles = int((m + gemm::kBM - 1) / gemm::kBM);
  const int64_t narrow = row_tiles * (n / 128);
  h->split = 0;
  for (int s = gemm::kMaxSplit; s > 1 && !h->split; s >>= 1)
    if (narrow * s <= sms && k / gemm::kBK >= 4 * s) h->split = s;
  if (!rc) rc = make_tensor_map_u8_sw128(&h->map_b, buffers[2], uint64_t(n), uint64_t(k), h->split ? 128 : gemm::kBN);
  if (!rc) rc = int(cudaFuncSetAttribute(gemm::gemm_fp8_kernel<gemm::kDense>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, int(gemm::kSmemBytes)));
  if (rc) { delete h; return rc; }
  gemm::Params& p = h->params;
  p = gemm::Params{};
  p.n = int(n);
  p.k_blocks = p.b_k_blocks = int(k / gemm::kBK);
  p.b_rows_per_group = int(n);
  p.groups = 1;
  p.row_capacity = int(m);
  p.offsets = nullptr;
  p.dense_rows = int(m);
  p.sfa = static_cast<const float*>(buffers[1]);
  p.sfb = static_cast<const float*>(buffers[3]);
  p.out = buffers[4];
  h->status = static_cast<int*>(buffers[5]);
  p.status = h->status;
  p.queue = h->status + 4;               // work-item counter, inside the 256-byte status block
  const long long items = row_tiles * ((n + gemm::kBN - 1) / gemm::kBN);
  // Drawing items from a counter evens out SMs of different speed, 2 % of a long launch, but the counter has to be cleared in
  // front of the kernel, 4 us: not for a few rounds of the GPU (346 x 6272 x 640, one round: 12.3 -> 7.5 us).
  if (items <= 6 * sms) p.queue = nullptr;
  if (h->split) {
    rc = int(cudaFuncSetAttribute(gemm::gemm_fp8_kernel<gemm::kDense, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gemm::kSmemBytes)));
    if (rc) { delete h; return rc; }
  }
  h->grid = h->split ? int(narrow) * h->split : int(items < sms ? items : sms);
  // At most 16 rows go through the weight-streaming kernel (4096 x 7168: 8.9 us at 1 row, 10.5 at 16; 12.1 for a split tile
  // of the core).  Beyond, its second tile of 16 rows reads the weights again.
  h->skinny_tiles = m > 16 ? 0 : m <= 8 ? 1 : 2;
  h->skinny_split = skinny::choose_split(1.0, int(n), p.k_blocks, sms);
  const int64_t skinny_items = (n + 32 * (8 / h->skinny_split) - 1) / (32 * (8 / h->skinny_split));
  if (h->skinny_tiles) {
    skinny::Params& q = h->skinny;
    q = skinny::Params{};
    q.w = static_cast<const uint8_t*>(buffers[2]);
    q.sw = p.sfb;
    q.x = static_cast<const uint8_t*>(buffers[0]);
    q.sx = p.sfa;
    q.out = p.out;
    q.status = h->status;
    q.n = int(n);
    q.k_blocks = p.k_blocks;
    q.w_rows = int(n);
    q.groups = 1;
    q.dense_rows = int(m);
    q.x_stride = int(k);
    q.sx_stride = int(m);
    q.terms = 1;
    h->skinny_grid = int(skinny_items < sms ? skinny_items : sms);
    rc = skinny::prepare_any<gemm::kDense>(h->skinny_tiles, h->skinny_split, 1);
    if (rc) { delete h; return rc; }
  }
  *handle_out = h;
  return 0;
}

extern "C" int cake_b200_block_scaled_gemm_launch(void* handle, void* cuda_stream) {
  using namespace cake;
  if (!handle) return kErrBadArgument;
  auto* h = static_cast<DenseHandle*>(handle);
  int device = -1;
  CAKE_CUDA_OK(cudaGetDevice(&device));
  if (device != h->device) return kErrWrongDevice;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(cuda_stream);
  if (h->skinny_tiles && !test_hooks().skip_load)
    return skinny::launch_any<gemm::kDense>(h->skinny_tiles, h->skinny_split, 1, h->skinny, h->skinny_grid, stream);
  gemm::Params p = h->params;
  p.wait_kiloclocks = test_hooks().budget_kiloclocks;
  p.skip_load = test_hooks().skip_load;
  if (h->split)
    return launch_dependent_cluster(h->split, gemm::gemm_fp8_kernel<gemm::kDense, true>, dim3(h->grid), dim3(gemm::kThreads), gemm::kSmemBytes,
                                    stream, gemm::Maps<gemm::kDense>{h->map_a, h->map_a_tail, h->map_b}, p);
  if (p.queue) CAKE_CUDA_OK(cudaMemsetAsync(h->status, 0, 8 * sizeof(int), stream));     // status word and work-item counter
  return launch_dependent(gemm::gemm_fp8_kernel<gemm::kDense>, dim3(h->grid), dim3(gemm::kThreads), gemm::kSmemBytes, stream, gemm::Maps<gemm::kDense>{h->map_a, h->map_a_tail, h->map_b}, p);
}

extern "C" int cake_b200_block_scaled_gemm_destroy(void* handle) {
  delete static_cast<cake::DenseHandle*>(handle);
  return 0;
}
