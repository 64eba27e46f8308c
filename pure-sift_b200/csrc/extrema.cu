// K4: 26-neighbour DoG extrema + Hessian edge test + 3D Taylor refinement, with
// ordered compaction, and the 4096-feature cap (stable top-K by |response|).
//
// Reference: passes_hessian_edge_test (src/pipeline.rs:664-687),
// refine_extremum_3d (:697-770), is_greater/less_than_patch3x3 (:775-808),
// extract_extrema_in_octave_slices (:810-916), Pyramid::extract_extrema
// (:535-547), the cap in extract_sift_features_with_kind (:1643-1651).
//
// Order: the reference emits keypoints octave by octave, slice by slice, row by
// row, column by column.  extrema_mark writes one bit per pixel plus a count per
// (octave, slice, row); row_scan turns the counts into exclusive offsets; and
// extrema_emit (one warp per row) writes each keypoint at its rank, so the list
// is identical in content and order to the reference's.
//
// Every arithmetic step repeats the reference's f32 expression in order
// (no FMA: the library is built with -fmad=false).  The single transcendental,
// k^ds, is evaluated in double and rounded once to f32.
#include "detect_plan.cuh"
#include "psift_internal.cuh"

namespace psift {

// The 3x3x3 DoG values around pixel (x, y) of slice s, each the rounded difference
// D[i] = G[i+1] - G[i] the pyramid defines (build_scale_space_pyramid_with_options,
// src/pipeline.rs:550-638), formed here from the four Gaussian planes it spans
// instead of being stored: the blur then writes one plane per level, not two
// (20 of 64 bytes per octave pixel at 3 scales).  Entries are row-major, [4] the centre.
struct Dog27 {
  float p[9], c[9], n[9];
};

// g: G[s-1] at (x, y); every load is issued before the first use.
__device__ __forceinline__ void load_dog27(const float* __restrict__ g, long long ps, long long pitch, Dog27& d) {
  float v[4][9];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) v[i][3 * r + k] = __ldg(g + i * ps + (r - 1) * pitch + (k - 1));
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    d.p[k] = v[1][k] - v[0][k];
    d.c[k] = v[2][k] - v[1][k];
    d.n[k] = v[3][k] - v[2][k];
  }
}

// refine_extremum_3d (src/pipeline.rs:697-770).
__device__ __forceinline__ void refine3d(const Dog27& d, float& ox_o, float& oy_o, float& os_o, float& interp_o) {
  const float center = d.c[4];
  const float gx = 0.5f * (d.c[5] - d.c[3]);
  const float gy = 0.5f * (d.c[7] - d.c[1]);
  const float gs = 0.5f * (d.n[4] - d.p[4]);
  const float dxx = d.c[5] - 2.0f * center + d.c[3];
  const float dyy = d.c[7] - 2.0f * center + d.c[1];
  const float dss = d.n[4] - 2.0f * center + d.p[4];
  const float dxy = 0.25f * ((d.c[8] - d.c[6]) - (d.c[2] - d.c[0]));
  const float dxs = 0.25f * ((d.n[5] - d.n[3]) - (d.p[5] - d.p[3]));
  const float dys = 0.25f * ((d.n[7] - d.n[1]) - (d.p[7] - d.p[1]));
  const float c00 = dyy * dss - dys * dys;
  const float c01 = dys * dxs - dxy * dss;
  const float c02 = dxy * dys - dyy * dxs;
  const float c11 = dxx * dss - dxs * dxs;
  const float c12 = dxy * dxs - dxx * dys;
  const float c22 = dxx * dyy - dxy * dxy;
  const float det3 = dxx * c00 + dxy * c01 + dxs * c02;
  if (fabsf(det3) > 1e-9f) {
    const float inv_det = -1.0f / det3;
    const float ox = (c00 * gx + c01 * gy + c02 * gs) * inv_det;
    const float oy = (c01 * gx + c11 * gy + c12 * gs) * inv_det;
    const float os = (c02 * gx + c12 * gy + c22 * gs) * inv_det;
    if (fabsf(ox) <= 0.5f && fabsf(oy) <= 0.5f && fabsf(os) <= 0.5f) {
      ox_o = ox;
      oy_o = oy;
      os_o = os;
      interp_o = center + 0.5f * (gx * ox + gy * oy + gs * os);
      return;
    }
  }
  if (fabsf(c22) > 1e-9f) {
    const float inv_det2 = -1.0f / c22;
    float ox = (dyy * gx - dxy * gy) * inv_det2;
    float oy = (-dxy * gx + dxx * gy) * inv_det2;
    ox = ox < -0.5f ? -0.5f : (ox > 0.5f ? 0.5f : ox);
    oy = oy < -0.5f ? -0.5f : (oy > 0.5f ? 0.5f : oy);
    float os = 0.0f;
    if (fabsf(dss) > 1e-6f) {
      os = -gs / dss;
      os = os < -0.5f ? -0.5f : (os > 0.5f ? 0.5f : os);
    }
    ox_o = ox;
    oy_o = oy;
    os_o = os;
    interp_o = center + 0.5f * (gx * ox + gy * oy + gs * os);
    return;
  }
  ox_o = oy_o = os_o = 0.0f;
  interp_o = center;
}

// Full acceptance test for the pixel whose neighbourhood is d: the reference's
// comparison chain (is_greater/less_than_patch3x3 over the current, previous and
// next slices), its edge test and its refinement.  Short-circuiting does not
// change the outcome (all must hold).
__device__ __forceinline__ bool accept_pixel(const Dog27& d, float thr) {
  const float v = d.c[4];
  if (fabsf(v) <= thr) return false;
  const bool pos = v > 0.0f;
  bool ext = true;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    if (k != 4) ext = ext && (pos ? v > d.c[k] : v < d.c[k]);
    ext = ext && (pos ? v > d.p[k] : v < d.p[k]);
    ext = ext && (pos ? v > d.n[k] : v < d.n[k]);
  }
  if (!ext) return false;
  // passes_hessian_edge_test (src/pipeline.rs:664-687)
  {
    const float dxx = d.c[5] - 2.0f * v + d.c[3];
    const float dyy = d.c[7] - 2.0f * v + d.c[1];
    const float dxy = 0.25f * ((d.c[8] - d.c[6]) - (d.c[2] - d.c[0]));
    const float trace = dxx + dyy;
    const float det = dxx * dyy - dxy * dxy;
    const float ratio = (11.0f * 11.0f) / 10.0f;
    if (!(det > 1e-9f && (trace * trace) < ratio * det)) return false;
  }
  float ox, oy, os, interp;
  refine3d(d, ox, oy, os, interp);
  return fabsf(interp) > thr;
}

// 128 threads per CTA; WPR warps share a row (all S slices), 4 / WPR rows per CTA.
// A warp walks every WPR-th 128-pixel span of its row (a lane reads 4 pixels of
// each of the planes G[1..S+1] as 128-bit loads; the next span's loads are issued
// before the current span is processed).
//   A. streaming: a pixel of slice s stays a candidate if its D is above the
//      threshold and above every neighbour at hand, or below the negated threshold
//      and below every neighbour at hand: left and right (inside the span) and
//      slices s - 1, s + 1 where they are among the loaded ones.  Each of these
//      comparisons is part of the full test, so nothing is lost, and the survivors
//      are a few per row instead of every pixel of a blob.
//   B. survivors queue up in shared memory and take the full 26-neighbour /
//      Hessian / refinement test 32 at a time; accepted ones set their bit of the
//      row's mask words (zeroed first).
// Bound by HBM latency and the comparisons' issue: 4 (S + 1) bytes per pixel read
// once, 57 us for two 3840 x 2160 octaves at 3 scales (4.7 TB/s, 78 us with a warp
// per row: four warps per row keep the last wave of a launch short).
constexpr int kMarkWarps = 4;
constexpr int kMarkSpan = 128;  // pixels per warp step

template <int S>
__device__ __forceinline__ void mark_load_span(const float* __restrict__ g1, long long ps, int x0, int w,
                                               float4 (&v)[S + 1]) {
#pragma unroll
  for (int i = 0; i <= S; ++i) {
    const float* g = g1 + i * ps + x0;
    if (x0 + 3 < w) {
      v[i] = __ldg(reinterpret_cast<const float4*>(g));
    } else {
      v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (x0 + 0 < w) v[i].x = g[0];
      if (x0 + 1 < w) v[i].y = g[1];
      if (x0 + 2 < w) v[i].z = g[2];
    }
  }
}

template <int S, int WPR>
__global__ void __launch_bounds__(kMarkWarps * 32) extrema_mark_kernel(const ImagePlan* __restrict__ plans,
                                                                       int octave, ExtremaParams prm) {
  constexpr int ROWS = kMarkWarps / WPR;
  __shared__ uint32_t s_q[kMarkWarps][31 + S * kMarkSpan];  // (s - 1) << 16 | x
  __shared__ uint32_t s_cnt[ROWS][S];
  const ImagePlan& P = plans[blockIdx.y];
  if (octave >= P.n_oct) return;
  const OctaveDev& O = P.oct[octave];
  if ((int)blockIdx.x * ROWS >= O.h) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = warp / WPR, part = warp % WPR;
  const int y = blockIdx.x * ROWS + row;
  const long long ps = O.plane_stride, pitch = O.pitch;
  const int w = O.w, words = O.words;
  const long long slice_words = (long long)O.h * words;
  uint32_t* mrow = O.masks + (long long)y * words;  // slice 1's; slice s: + (s - 1) * slice_words
  const int tid = threadIdx.x % (32 * WPR);         // thread of the row
  if (tid < S) s_cnt[row][tid] = 0;
  if (y < O.h)
    for (int s = 0; s < S; ++s)
      for (int i = tid; i < words; i += 32 * WPR) mrow[s * slice_words + i] = 0;
  __syncthreads();  // the zeroed words and counts before the bits set in them
  if (y >= 1 && y < O.h - 1) {
    const float* g0 = O.g + (long long)y * pitch;  // G[0], row y
    const float* g1 = g0 + ps;
    const float thr = prm.threshold;
    const float none = __int_as_float(0x7fffffff);  // NaN: ignored by fmaxf / fminf
    uint32_t* q = s_q[warp];
    int queued = 0;
    auto test = [&](int i) {
      const uint32_t e = q[i];
      const int s = (int)(e >> 16), x = (int)(e & 0xFFFFu);
      if (x < 1 || x >= w - 1) return;
      Dog27 d;
      load_dog27(g0 + s * ps + x, ps, pitch, d);  // G[s-1] of slice s (e holds s - 1)
      if (accept_pixel(d, thr)) {
        atomicOr(mrow + s * slice_words + (x >> 5), 1u << (x & 31));
        atomicAdd(&s_cnt[row][s], 1u);
      }
    };

    float4 cur[S + 1], nxt[S + 1];
    mark_load_span<S>(g1, ps, part * kMarkSpan + 4 * lane, w, cur);
    for (int xb = part * kMarkSpan; xb < w; xb += WPR * kMarkSpan) {
      if (xb + WPR * kMarkSpan < w) mark_load_span<S>(g1, ps, xb + WPR * kMarkSpan + 4 * lane, w, nxt);
      float D[S][4];
#pragma unroll
      for (int s = 0; s < S; ++s) {
        D[s][0] = cur[s + 1].x - cur[s].x;
        D[s][1] = cur[s + 1].y - cur[s].y;
        D[s][2] = cur[s + 1].z - cur[s].z;
        D[s][3] = cur[s + 1].w - cur[s].w;
      }
      unsigned long long m = 0;  // bit 4 (s - 1) + i: pixel xb + 4 lane + i of slice s
#pragma unroll
      for (int s = 0; s < S; ++s) {
        float left = __shfl_up_sync(0xffffffffu, D[s][3], 1), right = __shfl_down_sync(0xffffffffu, D[s][0], 1);
        if (lane == 0) left = none;
        if (lane == 31) right = none;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float v = D[s][i];
          const float l = i > 0 ? D[s][i > 0 ? i - 1 : 0] : left, r = i < 3 ? D[s][i < 3 ? i + 1 : 3] : right;
          float hi = fmaxf(fmaxf(thr, l), r), lo = fminf(fminf(-thr, l), r);
          if (s > 0) hi = fmaxf(hi, D[s > 0 ? s - 1 : 0][i]), lo = fminf(lo, D[s > 0 ? s - 1 : 0][i]);
          if (s + 1 < S) hi = fmaxf(hi, D[s + 1 < S ? s + 1 : s][i]), lo = fminf(lo, D[s + 1 < S ? s + 1 : s][i]);
          if (v > hi || v < lo) m |= 1ull << (4 * s + i);
        }
      }
      if (__any_sync(0xffffffffu, m != 0)) {
        const int c = __popcll(m);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        int pos = queued + incl - c;
        while (m) {
          const int b = __ffsll((long long)m) - 1;
          m &= m - 1;
          q[pos++] = (uint32_t)(b >> 2) << 16 | (uint32_t)(xb + 4 * lane + (b & 3));
        }
        queued += __shfl_sync(0xffffffffu, incl, 31);
        __syncwarp();
        while (queued >= 32) {
          queued -= 32;
          test(queued + lane);
        }
        __syncwarp();
      }
#pragma unroll
      for (int i = 0; i <= S; ++i) cur[i] = nxt[i];
    }
    if (lane < queued) test(lane);
  }
  __syncthreads();
  if (y < O.h && tid < S) P.row_counts[O.row_base + tid * O.h + y] = s_cnt[row][tid];
}

// Block-wide exclusive scan helper for 1024 threads; returns the block total.
__device__ __forceinline__ uint32_t block_exclusive_scan_1024(uint32_t v, uint32_t& excl, uint32_t* s_warp) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) s_warp[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = s_warp[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    s_warp[lane] = w;  // inclusive warp totals
  }
  __syncthreads();
  const uint32_t warp_prefix = wid > 0 ? s_warp[wid - 1] : 0u;
  excl = warp_prefix + x - v;
  const uint32_t total = s_warp[31];
  __syncthreads();
  return total;
}

// One block (1024 threads) per image: exclusive offsets over all (octave, slice, row),
// kScanRows consecutive rows per thread: bound by the latency of a turn's loads and
// barriers, so a turn takes 16,384 rows (12,150 rows of a 1920 x 1080 image at 3 scales
// and 4 octaves), all loads issued at once.  With the one launch of extrema_emit_kernel:
// a 640 x 480 image on the host 306 -> 291 us, a device batch of four 1920 x 1080 1094 ->
// 1072 us.
constexpr int kScanRows = 16;
__global__ void __launch_bounds__(1024) row_scan_kernel(const ImagePlan* __restrict__ plans, uint32_t kp_cap,
                                                        uint32_t* err) {
  const ImagePlan& P = plans[blockIdx.x];
  __shared__ uint32_t s_warp[32];
  const int rows = P.total_rows;
  uint32_t carry = 0;
  for (int base = 0; base < rows; base += 1024 * kScanRows) {
    const int i = base + (int)threadIdx.x * kScanRows;
    uint32_t v[kScanRows], sum = 0;
    if (i + kScanRows <= rows) {
#pragma unroll
      for (int q = 0; q < kScanRows; q += 4) {
        const uint4 c = *reinterpret_cast<const uint4*>(P.row_counts + i + q);
        v[q] = c.x, v[q + 1] = c.y, v[q + 2] = c.z, v[q + 3] = c.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < kScanRows; ++q) v[q] = i + q < rows ? P.row_counts[i + q] : 0u;
    }
#pragma unroll
    for (int q = 0; q < kScanRows; ++q) sum += v[q];
    uint32_t excl;
    const uint32_t tot = block_exclusive_scan_1024(sum, excl, s_warp);
    uint32_t at = carry + excl;
#pragma unroll
    for (int q = 0; q < kScanRows; ++q) {
      const uint32_t c = v[q];
      v[q] = at;
      at += c;
    }
    if (i + kScanRows <= rows) {
#pragma unroll
      for (int q = 0; q < kScanRows; q += 4)
        *reinterpret_cast<uint4*>(P.row_offsets + i + q) = make_uint4(v[q], v[q + 1], v[q + 2], v[q + 3]);
    } else {
#pragma unroll
      for (int q = 0; q < kScanRows; ++q)
        if (i + q < rows) P.row_offsets[i + q] = v[q];
    }
    carry += tot;
  }
  if (threadIdx.x == 0) {
    *P.kp_count = carry;
    if (carry > kp_cap) atomicOr(err, kErrKeypointCapacity);
  }
}

// Grid (ceil(rows / 8), images), 256 threads: one warp per (octave, slice, row), the
// octaves in one launch (each is a few microseconds of latency, not work).
__global__ void __launch_bounds__(256) extrema_emit_kernel(const ImagePlan* __restrict__ plans, ExtremaParams prm,
                                                           uint32_t kp_cap) {
  const ImagePlan& P = plans[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= P.total_rows || P.row_counts[r] == 0) return;
  int octave = 0;
  while (octave + 1 < P.n_oct && r >= P.oct[octave + 1].row_base) ++octave;
  const OctaveDev& O = P.oct[octave];
  const int row_local = r - O.row_base;
  const int s = 1 + row_local / O.h;
  const int y = row_local - (s - 1) * O.h;
  uint32_t pos_base = P.row_offsets[r];
  const long long ps = O.plane_stride;
  const float* g = O.g + (long long)(s - 1) * ps + (long long)y * O.pitch;  // G[s-1], row y
  const uint32_t* mrow = O.masks + ((long long)(s - 1) * O.h + y) * O.words;
  const float mult = O.scale_factor;
  const float eff = prm.eff_scale[octave][s];
  for (int wb = 0; wb < O.words; wb += 32) {
    uint32_t word = (wb + lane < O.words) ? mrow[wb + lane] : 0u;
    const uint32_t c = __popc(word);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    uint32_t pos = pos_base + incl - c;
    while (word) {
      const int b = __ffs(word) - 1;
      word &= word - 1;
      const int x = (wb + lane) * 32 + b;
      float dx, dy, ds, interp;
      Dog27 d;
      load_dog27(g + x, ps, O.pitch, d);
      refine3d(d, dx, dy, ds, interp);
      if (pos < kp_cap) {
        psift_keypoint kp;
        const float kds = (float)pow((double)prm.k, (double)ds);
        const float refined_scale = eff * kds;
        float lf = roundf((float)s + ds);
        lf = lf < 1.0f ? 1.0f : (lf > (float)prm.scales ? (float)prm.scales : lf);
        kp.x = ((float)x + dx) * mult;
        kp.y = ((float)y + dy) * mult;
        kp.scale = fmaxf(refined_scale, 0.25f * kBaseSigma);
        kp.response = interp;
        kp.octave = (uint32_t)octave;
        kp.layer = (uint32_t)lf;
        P.kps[pos] = kp;
      }
      ++pos;
    }
    pos_base += __shfl_sync(0xffffffffu, incl, 31);
  }
}

// Stable top-K by |response| (descending; ties keep keypoint order), then
// sorted -- exactly `sort_by(|b| b.response.abs() ...)` + `truncate(K)`.
// One block (1024 threads) per image.  The K selected sort keys live in
// dynamic shared memory (next_pow2(K) x 8 bytes).
__global__ void __launch_bounds__(1024) select_topk_kernel(const ImagePlan* __restrict__ plans, uint32_t kp_cap,
                                                           uint32_t max_features, uint32_t* err) {
  const ImagePlan& P = plans[blockIdx.x];
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_hist[256];
  __shared__ uint32_t s_sel[4];
  extern __shared__ unsigned long long s_keys[];
  const uint32_t found = *P.kp_count;
  const uint32_t N = found < kp_cap ? found : kp_cap;
  const uint32_t K = max_features;
  if (K == 0 || N <= K) {
    for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) P.sel[i] = P.kps[i];
    if (threadIdx.x == 0) *P.sel_count = N;
    return;
  }
  // Radix select of the K-th largest key, most significant byte first.
  uint32_t prefix = 0, mask = 0, need = K;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) {
      const uint32_t key = __float_as_uint(fabsf(P.kps[i].response));
      if ((key & mask) == prefix) atomicAdd(&s_hist[(key >> shift) & 0xFF], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t above = 0;
      int b = 255;
      for (; b > 0; --b) {
        if (above + s_hist[b] >= need) break;
        above += s_hist[b];
      }
      s_sel[0] = (uint32_t)b;
      s_sel[1] = need - above;
    }
    __syncthreads();
    prefix |= s_sel[0] << shift;
    mask |= 0xFFu << shift;
    need = s_sel[1];
    __syncthreads();
  }
  const uint32_t T = prefix;  // K-th largest key; take all keys > T and the first `need` keys == T
  uint32_t n_sel = 0, n_eq = 0;
  for (uint32_t base = 0; base < N; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    uint32_t key = 0;
    if (i < N) key = __float_as_uint(fabsf(P.kps[i].response));
    const uint32_t is_eq = (i < N && key == T) ? 1u : 0u;
    uint32_t eq_excl;
    const uint32_t eq_tot = block_exclusive_scan_1024(is_eq, eq_excl, s_warp);
    const uint32_t take = (i < N) && (key > T || (is_eq && n_eq + eq_excl < need)) ? 1u : 0u;
    uint32_t sel_excl;
    const uint32_t sel_tot = block_exclusive_scan_1024(take, sel_excl, s_warp);
    if (take) {
      const uint32_t slot = n_sel + sel_excl;
      if (slot < K) s_keys[slot] = ((unsigned long long)(~key) << 32) | (unsigned long long)i;
    }
    n_eq += eq_tot;
    n_sel += sel_tot;
  }
  uint32_t n2 = 1;
  while (n2 < K) n2 <<= 1;
  for (uint32_t i = K + threadIdx.x; i < n2; i += blockDim.x) s_keys[i] = ~0ull;
  if (threadIdx.x == 0 && n_sel != K) atomicOr(err, kErrSortCapacity);
  __syncthreads();
  // Bitonic sort ascending on (~|response|, index).
  for (uint32_t k = 2; k <= n2; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < n2; i += blockDim.x) {
        const uint32_t ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long a = s_keys[i], b = s_keys[ixj];
          const bool up = (i & k) == 0;
          if ((a > b) == up) {
            s_keys[i] = b;
            s_keys[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = threadIdx.x; i < K; i += blockDim.x) P.sel[i] = P.kps[(uint32_t)(s_keys[i] & 0xFFFFFFFFu)];
  if (threadIdx.x == 0) *P.sel_count = K;
}

template <int S>
static void launch_mark_s(const ImagePlan* plans, int n, int octave, int max_h, int max_w, const ExtremaParams& prm,
                          cudaStream_t st) {
  // at least two spans per warp of a row
  if (max_w > 6 * kMarkSpan)
    extrema_mark_kernel<S, 4><<<dim3(max_h, n), kMarkWarps * 32, 0, st>>>(plans, octave, prm);
  else if (max_w > 3 * kMarkSpan)
    extrema_mark_kernel<S, 2><<<dim3((max_h + 1) / 2, n), kMarkWarps * 32, 0, st>>>(plans, octave, prm);
  else
    extrema_mark_kernel<S, 1><<<dim3((max_h + 3) / 4, n), kMarkWarps * 32, 0, st>>>(plans, octave, prm);
}

cudaError_t launch_extrema_mark(const ImagePlan* plans, int n, int octave, int max_h, int max_w,
                                const ExtremaParams& prm, cudaStream_t st) {
  switch (prm.scales) {
#define PSIFT_MARK(SS)                                              \
  case SS:                                                          \
    launch_mark_s<SS>(plans, n, octave, max_h, max_w, prm, st);     \
    break;
    PSIFT_MARK(3) PSIFT_MARK(4) PSIFT_MARK(5) PSIFT_MARK(6) PSIFT_MARK(7) PSIFT_MARK(8) PSIFT_MARK(9) PSIFT_MARK(10)
#undef PSIFT_MARK
    default:
      return cudaErrorInvalidValue;  // scales is validated to 3..10
  }
  return cudaGetLastError();
}

// An octave's DoG slices G[i+1] - G[i], i = blockIdx.y, dense one after the other
// (psift_build_pyramid hands them to the caller).
__global__ void dog_planes_kernel(const float* __restrict__ g, long long plane_stride, long long pitch, int h, int w,
                                  float* __restrict__ out) {
  const float* lower = g + blockIdx.y * plane_stride;
  const float* upper = lower + plane_stride;
  out += (long long)blockIdx.y * h * w;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)h * w;
       i += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(i / w), x = (int)(i - (long long)y * w);
    out[i] = upper[y * pitch + x] - lower[y * pitch + x];
  }
}

cudaError_t launch_dog_planes(const float* g, long long plane_stride, int slices, long long pitch, int h, int w,
                              float* out, cudaStream_t st) {
  const long long blocks = ((long long)h * w + 255) / 256;
  dog_planes_kernel<<<dim3((unsigned)(blocks < 148 * 32 ? blocks : 148 * 32), slices), 256, 0, st>>>(g, plane_stride,
                                                                                                 pitch, h, w, out);
  return cudaGetLastError();
}

cudaError_t launch_row_scan(const ImagePlan* plans, int n, uint32_t kp_cap, uint32_t* err, cudaStream_t st) {
  row_scan_kernel<<<n, 1024, 0, st>>>(plans, kp_cap, err);
  return cudaGetLastError();
}

// max_rows: the most rows (octave, slice, row) of an image.
cudaError_t launch_extrema_emit(const ImagePlan* plans, int n, int max_rows, const ExtremaParams& prm, uint32_t kp_cap,
                                cudaStream_t st) {
  extrema_emit_kernel<<<dim3((max_rows + 7) / 8, n), 256, 0, st>>>(plans, prm, kp_cap);
  return cudaGetLastError();
}

cudaError_t launch_select_topk(const ImagePlan* plans, int n, uint32_t kp_cap, uint32_t max_features, uint32_t* err,
                               cudaStream_t st) {
  uint32_t n2 = 1;
  while (n2 < max_features) n2 <<= 1;
  const size_t smem = max_features ? n2 * sizeof(unsigned long long) : 0;
  cudaError_t e = ensure_smem_attr((const void*)select_topk_kernel, 128 * 1024);
  if (e != cudaSuccess) return e;
  select_topk_kernel<<<n, 1024, smem, st>>>(plans, kp_cap, max_features, err);
  return cudaGetLastError();
}

}  // namespace psift
