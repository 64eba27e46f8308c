// Host side of the strip level blur (blur_strip.cuh): work items and launch.
#include <algorithm>

#include "blur_strip.cuh"

namespace psift {
namespace {

template <int R, bool FUSED>
cudaError_t launch_strip_r(const ImagePlan* plans, const ImagePlan* h_plans, int n, int octave, int level,
                           int down_level, int zrev, const Taps2& taps, int max_h, int max_w, cudaStream_t st) {
  using G = StripGeom<R>;
  constexpr int W = G::W;
  const bool down = level == down_level;
  auto* const kernel = down ? blur_strip_kernel<R, FUSED, true> : blur_strip_kernel<R, FUSED, false>;
  const void* fn = (const void*)kernel;
  const size_t smem = (size_t)G::SMEM_BYTES * W;
  cudaError_t e = ensure_smem_attr(fn, smem);
  if (e != cudaSuccess) return e;
  const int seg = kStripChunks * G::CR - 2 * R;  // output rows per segment
  TileMap tm;
  tm.n = 0;
  tm.prefix[0] = 0;
  dim3 grid(((max_w + kStripW - 1) / kStripW + W - 1) / W, (max_h + seg - 1) / seg, n);
  if (h_plans && n <= kTileMapMax) {
    for (int i = 0; i < n; ++i) {
      const bool has = octave < h_plans[i].n_oct;
      const int tx = has ? (h_plans[i].oct[octave].w + kStripW - 1) / kStripW : 0;
      const int ty = has ? (h_plans[i].oct[octave].h + seg - 1) / seg : 0;
      tm.tiles_x[i] = std::max(tx, 1);
      tm.prefix[i + 1] = tm.prefix[i] + tx * ty;
    }
    tm.n = n;
    grid = dim3((unsigned)(tm.prefix[n] + W - 1) / W, 1, 1);
  }
  if (grid.x == 0 || grid.y == 0) return cudaSuccess;
  kernel<<<grid, 32 * W, smem, st>>>(plans, octave, level, zrev, seg, taps, tm);
  return cudaGetLastError();
}

}  // namespace

// The level blur of images [0, n): h_plans (the plans' host copy) sizes the work
// items; without it, or above kTileMapMax images, they cover max_h x max_w of
// every image.
cudaError_t launch_blur_strip(int radius, bool fused, const ImagePlan* plans, const ImagePlan* h_plans, int n,
                              int octave, int level, int down_level, int zrev, const Taps2& taps, int max_h,
                              int max_w, cudaStream_t st) {
  switch (radius) {
#define PSIFT_SR(RR)                                                                                                \
  case RR:                                                                                                          \
    return fused ? launch_strip_r<RR, true>(plans, h_plans, n, octave, level, down_level, zrev, taps, max_h, max_w, \
                                            st)                                                                \
                 : launch_strip_r<RR, false>(plans, h_plans, n, octave, level, down_level, zrev, taps, max_h,       \
                                             max_w, st);
    PSIFT_SR(1) PSIFT_SR(2) PSIFT_SR(3) PSIFT_SR(4) PSIFT_SR(5) PSIFT_SR(6) PSIFT_SR(7) PSIFT_SR(8)
    PSIFT_SR(9) PSIFT_SR(10)
#undef PSIFT_SR
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace psift
