// Host side of the Hamming shortlist entries (catalog_api.cu, ctx.cu) on a stand-in for the
// CUDA runtime and a launch_topk that does what the scenario says: built and run by
// test_topk_host_cpu.py.
#include <vector>

#include "fake_cuda.h"
#include "psift_internal.cuh"

// ---- the kernels' launchers
static int g_launches = 0, g_block = 0;
static bool g_time_out = false;
namespace psift {
cudaError_t launch_quantize(const float*, int, uint64_t*, uint8_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_popc_probe(int, int, uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_dequantize(const uint8_t*, int, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_votes(const uint64_t*, int, const uint64_t*, const long long*, int, int, uint32_t*, cudaStream_t) {
  return cudaSuccess;
}
size_t topk_scratch(int nq, int block) { return (size_t)(nq < block ? nq : block) * 8448; }
cudaError_t launch_topk(const uint64_t*, int, const uint64_t*, long long, int, int block, uint8_t*, uint32_t*,
                        uint32_t*, int, uint32_t* err, uint64_t*, cudaStream_t) {
  ++g_launches;
  g_block = block;
  if (g_time_out) *err |= kErrTimeout;
  return cudaSuccess;
}
cudaError_t launch_l2_rerank(const float*, int, const float*, const uint32_t*, int, uint32_t*, float*, cudaStream_t) {
  return cudaSuccess;
}
}  // namespace psift

// A wait that gives up in the shortlist kernel is reported, once, by the entry that read
// the lists back or, after the device entry, by the next synchronisation.
static int timeout_reported(psift_ctx* ctx) {
  uint64_t q[2] = {1, 2}, c[4] = {3, 4, 5, 6};
  uint32_t idx[1], dist[1];
  CHECK(psift_hamming_topk(ctx, q, 1, c, 2, 1, idx, dist) == PSIFT_OK);
  g_time_out = true;
  CHECK(psift_hamming_topk(ctx, q, 1, c, 2, 1, idx, dist) == PSIFT_ERR_TIMEOUT);
  g_time_out = false;
  CHECK(psift_ctx_synchronize(ctx) == PSIFT_OK);
  CHECK(psift_hamming_topk(ctx, q, 1, c, 2, 1, idx, dist) == PSIFT_OK);
  CHECK(psift_hamming_topk_dev(ctx, q, 1, c, 2, 1, idx, dist) == PSIFT_OK);
  CHECK(psift_ctx_synchronize(ctx) == PSIFT_OK);
  g_time_out = true;
  CHECK(psift_hamming_topk_dev(ctx, q, 1, c, 2, 1, idx, dist) == PSIFT_OK);
  g_time_out = false;
  CHECK(psift_hamming_topk_dev(ctx, q, 1, c, 2, 1, idx, dist) == PSIFT_OK);
  std::memset(ctx->d_error, 0, 4);  // as every other host entry does before its own work
  CHECK(psift_ctx_synchronize(ctx) == PSIFT_ERR_TIMEOUT);
  CHECK(psift_ctx_synchronize(ctx) == PSIFT_OK);
  return 0;
}

// Queries are taken in smaller blocks when the device is short of memory, and only then.
static int smaller_blocks(psift_ctx* ctx) {
  std::vector<uint64_t> q(2 * 8192);
  std::vector<uint32_t> idx(8192), dist(8192);
  uint64_t c[2] = {3, 4};
  g_malloc_limit = 32u << 20;
  CHECK(psift_hamming_topk_dev(ctx, q.data(), 8192, c, 1, 1, idx.data(), dist.data()) == PSIFT_OK);
  CHECK(g_launches == 1 && g_block == 1024);
  g_malloc_limit = 4u << 20;
  psift_ctx* fresh = nullptr;
  CHECK(psift_ctx_create(0, &fresh) == PSIFT_OK);
  CHECK(psift_hamming_topk_dev(fresh, q.data(), 8192, c, 1, 1, idx.data(), dist.data()) == PSIFT_OK);
  CHECK(g_launches == 2 && g_block == 128);
  psift_ctx_destroy(fresh);
  g_malloc_limit = 1u << 20;
  CHECK(psift_ctx_create(0, &fresh) == PSIFT_OK);
  CHECK(psift_hamming_topk_dev(fresh, q.data(), 8192, c, 1, 1, idx.data(), dist.data()) == PSIFT_ERR_OUT_OF_MEMORY);
  // any other failure is returned at once
  g_malloc_limit = ~(size_t)0;
  g_sync_result = cudaErrorLaunchFailure;
  const int before = g_syncs;
  CHECK(psift_hamming_topk_dev(fresh, q.data(), 8192, c, 1, 1, idx.data(), dist.data()) == PSIFT_ERR_CUDA);
  CHECK(g_syncs == before + 1 && g_launches == 2);
  g_sync_result = cudaSuccess;
  psift_ctx_destroy(fresh);
  return 0;
}

int main(int argc, char** argv) {
  psift_ctx* ctx = nullptr;
  CHECK(psift_ctx_create(0, &ctx) == PSIFT_OK);
  CHECK(argc == 2);
  int rc = 2;
  if (!std::strcmp(argv[1], "timeout")) rc = timeout_reported(ctx);
  if (!std::strcmp(argv[1], "memory")) rc = smaller_blocks(ctx);
  psift_ctx_destroy(ctx);
  return rc;
}
