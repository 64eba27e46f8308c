// Host side of the RANSAC entries (ransac_api.cu, ctx.cu) on a stand-in for the CUDA runtime:
// built and run by test_ransac_host_cpu.py.
#include "fake_cuda.h"
#include "psift_internal.cuh"
#include "ransac_common.cuh"

static int g_max_n = -1, g_n_sim = -1;
static double g_mean_n = -1;
namespace psift {
cudaError_t launch_ransac(const RansacJob* jobs, int n_jobs, int n_sim, int max_n, double mean_n, int, cudaStream_t) {
  g_max_n = max_n;
  g_n_sim = n_sim;
  g_mean_n = mean_n;
  for (int i = 0; i < n_jobs; ++i) {  // every array of a set is there, and in the workspace
    std::memset(jobs[i].cdf, 1, sizeof(double) * (size_t)jobs[i].n);
    std::memset(jobs[i].list, 1, sizeof(int) * (size_t)jobs[i].n);
    std::memset(jobs[i].xy, 1, sizeof(float4) * (size_t)jobs[i].n);
  }
  return cudaSuccess;
}
}  // namespace psift

// A match set's workspace: 28 bytes a match (cumulative weights, inlier list, coordinates).
int main() {
  constexpr uint32_t n = 1000000;
  psift_ctx* ctx = nullptr;
  CHECK(psift_ctx_create(0, &ctx) == PSIFT_OK);
  psift_match* m = (psift_match*)std::calloc(n, sizeof(psift_match));
  uint8_t* mask = (uint8_t*)std::calloc(n, 1);
  float model[9];
  int32_t has;
  uint32_t count;
  psift_ransac_options opt;
  psift_ransac_options_default(&opt);
  const psift_ransac_job job{m, n, mask, model, &has, &count, nullptr, nullptr};
  g_malloc_limit = 28u * n + (2u << 20);
  for (int homography = 0; homography < 2; ++homography)
    CHECK(psift_ransac_batch_dev(ctx, &job, 1, &opt, homography) == PSIFT_OK);
  CHECK(g_max_n == (int)n);  // what the CTAs' size goes by
  psift_ransac_job two[2] = {job, job};
  two[0].n = 33;
  two[1].n = 2;
  CHECK(psift_ransac_batch_dev(ctx, two, 2, &opt, 0) == PSIFT_OK && g_max_n == 33);
  CHECK(g_n_sim == 2 && g_mean_n == 17.5);
  CHECK(psift_ransac_batch_dev(ctx, two, 2, &opt, 1) == PSIFT_OK && g_n_sim == 0);
  two[0].n = two[1].n = n;
  g_malloc_limit = 1u << 20;
  CHECK(psift_ransac_batch_dev(ctx, two, 2, &opt, 1) == PSIFT_ERR_OUT_OF_MEMORY);
  psift_ctx_destroy(ctx);
  std::free(m);
  std::free(mask);
  return 0;
}
