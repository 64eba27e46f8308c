// K1-K3 host dispatch: octave base and level blurs (the kernel template lives in
// blur_kernel.cuh; this file instantiates the reference-rounding blur over a
// (tiles x, tiles y, images) grid, pyramid_fused.cu the single-rounding one, and
// pyramid_tiled*.cu both over a tile work list).
#include "blur_kernel.cuh"

namespace psift {

// Host entry: mode 0 = level blur (octave, level >= 1); modes 1..4 = octave-0 base.
// variant (level blur only) picks the default (0: strips for large launches,
// blur_strip.cuh, else 4 x 8 outputs per thread), other outputs per thread (1, 2,
// see blur_kernel.cuh), the TMA-tile kernel (3, blur_tma.cuh; needs the host copy
// of the plans for its tensor maps) or 128 x 64 tiles of 512 threads (4: half
// the horizontal pass's halo rows per output); every variant computes the same
// values.  fused: the single-rounding blur
// (one fused multiply-add per tap; not the reference's rounding).
cudaError_t launch_blur_tma(int radius, bool fused, const ImagePlan* d_plans, const ImagePlan* h_plans, int n,
                            int octave, int level, int down_level, int zrev, const Taps2& taps, uint32_t* err,
                            cudaStream_t st);

cudaError_t launch_blur_strip(int radius, bool fused, const ImagePlan* plans, const ImagePlan* h_plans, int n,
                              int octave, int level, int down_level, int zrev, const Taps2& taps, int max_h,
                              int max_w, cudaStream_t st);
constexpr int kStripMaxR = 10;                    // largest radius of the strip kernel
constexpr long long kStripMinPixels = 6000000;

cudaError_t launch_blur(int mode, const float* taps_host, int radius, const ImagePlan* plans, int n, int octave,
                        int level, int down_level, int max_h, int max_w, cudaStream_t st, int variant, bool fused,
                        const TileMap* tiles, const ImagePlan* h_plans, uint32_t* err) {
  Taps2 t;
  for (int i = 0; i < kMaxTaps; ++i) {
    const float v = i <= 2 * radius ? taps_host[i] : 0.0f;
    t.w[i] = make_float2(v, v);
  }
  t.one = make_float2(1.0f, 1.0f);
  const int zrev = (octave * 8 + level) & 1;
  // Variant 0: strips from kStripMinPixels output pixels per launch, else tiles.  A
  // strip's warp needs 6 to 10 us for its chunk however small the launch is, a tile
  // CTA 5 to 7 us (640 x 480, R = 4 / 10: strips 8.4 / 13.2 us, tiles 7.4 / 11.6);
  // two 1920 x 1080 planes take the same time either way (13.9 .. 30 against 15.2
  // .. 24 us), one 3840 x 2160 plane 19.4 / 25 / 30 / 25 / 41 us as strips and 25.3
  // / 28 / 31 / 35 / 41 as tiles.
  if (mode == MODE_LEVEL && variant == 0 && radius <= kStripMaxR) {
    long long pixels = 0;
    for (int i = 0; i < n; ++i) {
      if (!h_plans) pixels += (long long)max_h * max_w;
      else if (octave < h_plans[i].n_oct) pixels += (long long)h_plans[i].oct[octave].h * h_plans[i].oct[octave].w;
    }
    if (pixels >= kStripMinPixels)
      return launch_blur_strip(radius, fused, plans, h_plans, n, octave, level, down_level, zrev, t, max_h, max_w, st);
  }
  // variant 3: TMA tiles, persistent CTAs (blur_tma.cuh), either rounding
  if (mode == MODE_LEVEL && variant == 3)
    return launch_blur_tma(radius, fused, plans, h_plans, n, octave, level, down_level, zrev, t, err, st);
  // images of different sizes: one CTA per listed tile (4 x 8 outputs per thread)
  if (tiles && tiles->n > 0)
    return launch_blur_tiled(mode, fused, radius, plans, n, octave, level, down_level, zrev, t, *tiles, st);
  if (fused) return launch_blur_fused(mode, radius, plans, n, octave, level, down_level, zrev, t, max_h, max_w, st);
  switch (mode) {
    case MODE_LEVEL:
      switch (variant) {
        case 0: return launch_blur_mode<MODE_LEVEL, 4, 8, false>(radius, plans, n, octave, level, down_level, zrev, t, nullptr, max_h, max_w, st);
        case 1: return launch_blur_mode<MODE_LEVEL, 8, 8, false>(radius, plans, n, octave, level, down_level, zrev, t, nullptr, max_h, max_w, st);
        case 2: return launch_blur_mode<MODE_LEVEL, 4, 4, false>(radius, plans, n, octave, level, down_level, zrev, t, nullptr, max_h, max_w, st);
        case 4:  // 128-row tiles, 512 threads
          return launch_blur_mode<MODE_LEVEL, 4, 8, false, false, 128, 512>(radius, plans, n, octave, level, down_level,
                                                                            zrev, t, nullptr, max_h, max_w, st);
        default: return cudaErrorInvalidValue;
      }
    case MODE_INIT_F32: return launch_blur_mode<MODE_INIT_F32, 4, 8, false>(radius, plans, n, octave, level, down_level, zrev, t, nullptr, max_h, max_w, st);
    case MODE_INIT_U8: return launch_blur_mode<MODE_INIT_U8, 4, 8, false>(radius, plans, n, octave, level, down_level, zrev, t, nullptr, max_h, max_w, st);
    case MODE_INIT_F32_UP: return launch_blur_mode<MODE_INIT_F32_UP, 4, 8, false>(radius, plans, n, octave, level, down_level, zrev, t, nullptr, max_h, max_w, st);
    case MODE_INIT_U8_UP: return launch_blur_mode<MODE_INIT_U8_UP, 4, 8, false>(radius, plans, n, octave, level, down_level, zrev, t, nullptr, max_h, max_w, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace psift
