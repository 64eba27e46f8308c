// The level blur of large launches: one warp per 64-column strip segment, both
// passes in registers as transposed FIR filters.
//
// Reference: gaussian_blur (src/pipeline.rs:314-425); same taps, order, borders
// and roundings as blur_kernel.cuh (see there), so the planes are the same.
//
// A warp owns 64 columns x a segment of rows and walks down it CR (54 to 64) input
// rows at a time, alone (no block barriers):
//   1. the chunk's rows (64 + 2R' columns each) arrive in shared memory by 16-byte
//      asynchronous copies; a row's source index is clamped to the plane, columns
//      outside it are filled in afterwards (first and last strips only);
//   2. horizontal pass, in place: a lane walks a whole row, adjacent columns packed
//      (f32x2); two rows per lane;
//   3. vertical pass: lane l owns columns 2l, 2l + 1 and walks the rows; its 2R
//      pending sums stay in registers from chunk to chunk, so a segment recomputes
//      only its first 2R rows.
//
// Transposed FIR: the outputs that an input still has to reach are held as partial
// sums, in a ring of registers indexed by the output modulo 2R (the loops are
// unrolled by that period, so the sums never move).  A step forms each distinct
// product w_k x once (the taps are symmetric: outputs R before and R after share
// one) and adds it where it belongs.  Every output still accumulates its taps in
// input order, k = 0..2R, each a rounded product and a rounded addition.  Products
// are fma(x, w_k, +0): the rounded product, up to the sign of a zero, which no
// sum that starts at +0 shows; the first product is the reference's 0 + x w_0.
//
// What bounds it: packed operations of the FP32 pipe at R >= 6, HBM below (8 bytes
// per pixel).  Per output pair a pass takes 2R + 1 additions and about 1.3 R
// products instead of 2R + 1 of each, and the horizontal pass has no halo rows
// except a segment's first 2R.  Adjacent columns as the packed pair (rather than
// two rows) leave the operands where the loads put them: pairs across rows cost a
// register move per operation (measured: 12 % to 24 % of all instructions).
// Four 3840 x 2160 planes, R = 4 / 5 / 6 / 8 / 10, us per launch: 57.6 / 67 / 79 /
// 88 / 112 against 84.6 / 94 / 107 / 121 / 141 of the 64 x 64-tile kernel.
// Segments of two chunks: one chunk 58 / 69 / 83 / 95 / 129 (more rows recomputed),
// three 61 / 69 / 81 / 88 / 111 (longer last wave on smaller launches).
// From R = 7 four warps share a CTA, one per scheduler (R = 8 / 10: 93 / 121 us as
// single-warp CTAs, nine or ten per SM on four schedulers); below, single warps
// leave room for eleven per SM (R = 4: 63 us with four).
#pragma once
#include "blur_kernel.cuh"

namespace psift {

constexpr int kStripW = 64;      // columns per strip
constexpr int kStripChunks = 2;  // chunks per segment (see above)

template <int R>
struct StripGeom {
  static constexpr int W = R >= 7 ? 4 : 1;    // warps per CTA
  static constexpr int RP = (R + 3) / 4 * 4;  // column halo in whole 16-byte units
  static constexpr int IN_W = kStripW + 2 * RP;
  // floats per staged row: an odd number of 16-byte units, so that a quarter-warp's
  // 8 rows fall into 8 different bank groups
  static constexpr int P = (IN_W / 4) % 2 ? IN_W : IN_W + 4;
  // input rows per chunk: whole periods of the 2R pending vertical sums, two per lane
  static constexpr int CR = 64 / (2 * R) * (2 * R);
  static constexpr int SMEM_BYTES = CR * P * 4;  // per warp
};

// ---- packed f32x2
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\t"
      "mov.b64 x, {%2, %3};\n\t"
      "mov.b64 y, {%4, %5};\n\t"
      "mov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ void st_global_if(bool p, float* a, float2 v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p st.global.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(a),
               "f"(v.x), "f"(v.y), "r"((uint32_t)p)
               : "memory");
}
__device__ __forceinline__ void st_global_if(bool p, float* a, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(a), "f"(v),
               "r"((uint32_t)p)
               : "memory");
}

template <int R>
struct StripTaps {
  float2 w[R + 1];  // {w_k, w_k}, k = 0..R
  float2 one;       // {1, 1} from the kernel parameters (see mul_add2_rn)
  float2 zero;
};

template <int R, bool FUSED>
__device__ __forceinline__ float2 fir_add(const float2* p, float2 x, float2 acc, const StripTaps<R>& t, int k) {
  const int i = k <= R ? k : 2 * R - k;
  if constexpr (FUSED) return fma2(x, t.w[i], acc);
  else return fma2(p[i], t.one, acc);
}

// Vertical step, input row c (static modulo 2R): slot s of a holds the pending
// output row j = s (mod 2R); row c reaches outputs c - 2R .. c.  Returns output
// c - 2R, complete.
template <int R, bool FUSED>
__device__ __forceinline__ float2 fir_row(float2 (&a)[2 * R], float2 x, const StripTaps<R>& t, int c) {
  constexpr int N = 2 * R;
  float2 p[R + 1];
#pragma unroll
  for (int k = 0; k <= R; ++k) p[k] = fma2(x, t.w[k], t.zero);
  const float2 out = fir_add<R, FUSED>(p, x, a[c % N], t, N);
#pragma unroll
  for (int k = N - 1; k >= 1; --k) a[(c + N - k) % N] = fir_add<R, FUSED>(p, x, a[(c + N - k) % N], t, k);
  a[c % N] = p[0];
  return out;
}

// Horizontal step, input column c of a row, x = {in[c], in[c + 1]}: slot s of a
// holds the pending output pair (2s, 2s + 1) (s modulo R), which column c reaches
// with tap k = c - 2s.  Pairs outside [0, 62] (unless all: every pair exists) are
// left alone.  Returns pair c - 2R, complete when c is even.
template <int R, bool FUSED>
__device__ __forceinline__ float2 fir_col(float2 (&a)[R], float2 x, const StripTaps<R>& t, int c, bool all) {
  constexpr int N = 2 * R;
  float2 p[R + 1], out = t.zero;
#pragma unroll
  for (int k = c & 1; k <= R; k += 2) p[k] = fma2(x, t.w[k], t.zero);
#pragma unroll
  for (int k = N - (c & 1); k >= (c & 1); k -= 2) {
    const int j = c - k;
    if (!all && (j < 0 || j >= kStripW)) continue;
    const int s = ((j / 2) % R + R) % R;
    if (k == N) out = fir_add<R, FUSED>(p, x, a[s], t, k);
    else if (k == 0) a[s] = p[0];
    else a[s] = fir_add<R, FUSED>(p, x, a[s], t, k);
  }
  return out;
}

// Horizontal pass of one row in place: outputs 0..63 overwrite columns 0..63 of the
// staged row (a pair is complete 2R columns after its first input).  Pairs of
// adjacent columns are operands as they lie in memory; the odd ones in between
// cost two moves.  The first and last 2R inputs touch only the pairs that exist
// (unrolled); the rest repeat with the sums' period.
template <int R, bool FUSED>
__device__ __forceinline__ void strip_row(float* __restrict__ row, const StripTaps<R>& t) {
  using G = StripGeom<R>;
  constexpr int N = 2 * R;
  constexpr int OFF = G::RP - R;  // staged column of input 0
  constexpr int ITER = (kStripW - N) / N;
  constexpr int C1 = N + ITER * N, CE = kStripW - 1 + N;
  float2 a[R];
  auto pair_at = [&](int c) { return *reinterpret_cast<const float2*>(row + c + OFF); };  // c + OFF even
  float2 nat = pair_at(-(OFF % 2));  // the aligned pair reaching column 0
  auto column = [&](int c, bool all) {
    float2 x;
    if ((c + OFF) % 2 == 0) {
      x = nat;
    } else {
      const float2 next = pair_at(c + 1);
      x = make_float2(nat.y, next.x);
      nat = next;
    }
    const float2 v = fir_col<R, FUSED>(a, x, t, c, all);
    if (c % 2 == 0 && (all || c >= N)) *reinterpret_cast<float2*>(row + c - N) = v;
  };
#pragma unroll
  for (int c = 0; c < N; ++c) column(c, false);
#pragma unroll 1
  for (int i = 0; i < ITER; ++i, row += N) {
#pragma unroll
    for (int c = N; c < 2 * N; ++c) column(c, true);
  }
  row -= ITER * N;
#pragma unroll
  for (int c = C1; c < CE; ++c) column(c, false);
}

// Items: (strip, segment of seg_rows output rows, image), strips fastest;
// reversed when zrev, so that a level starts with what the one before wrote last.
template <int R, bool FUSED, bool DOWN>
__global__ void __launch_bounds__(32 * StripGeom<R>::W, StripGeom<R>::W == 4 ? 2 : 9)
    blur_strip_kernel(const ImagePlan* __restrict__ plans, int octave, int level, int zrev, int seg_rows, const __grid_constant__ Taps2 taps, const __grid_constant__ TileMap tiles) {
  using G = StripGeom<R>;
  constexpr int N = 2 * R, W = G::W;
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* buf = reinterpret_cast<float*>(smem4) + warp * (G::SMEM_BYTES / 4);
  int z, bx, by;
  if (tiles.n > 0) {
    if (!tile_of(tiles, (long long)blockIdx.x * W + warp, zrev, z, bx, by)) return;
  } else {
    bx = blockIdx.x * W + warp;
    by = zrev ? (int)gridDim.y - 1 - (int)blockIdx.y : (int)blockIdx.y;
    z = zrev ? (int)gridDim.z - 1 - (int)blockIdx.z : (int)blockIdx.z;
  }
  const ImagePlan& P = plans[z];
  if (octave >= P.n_oct) return;
  const OctaveDev& O = P.oct[octave];
  const int h = O.h, w = O.w;
  const int x0 = bx * kStripW, y0 = by * seg_rows;
  if (x0 >= w || y0 >= h) return;
  const int y1 = min(y0 + seg_rows, h);
  const int rows_total = y1 - y0 + N;
  const long long pitch = O.pitch;
  const float* src = O.g + (long long)(level - 1) * O.plane_stride;

  // columns [gx0, gx1) exist (the row pitch is a multiple of 32 floats, so the
  // copy may end in the row's padding); the rest is filled in after the copy
  const int gx0 = max(x0 - G::RP, 0), gx1 = min(x0 + kStripW + G::RP, (w + 3) & ~3);
  const int lead = gx0 - (x0 - G::RP);                       // columns left of the plane
  const int last = min(w - 1 - (x0 - G::RP), G::IN_W - 1);   // last column inside it
  const bool patch = lead > 0 || last < G::IN_W - 1;
  // lane u copies the 16-byte unit u of every row
  const bool has_unit = 4 * lane < gx1 - gx0;
  const float* unit_src = src + gx0 + 4 * lane;
  const uint32_t unit_dst = (uint32_t)__cvta_generic_to_shared(buf + lead + 4 * lane);
  auto issue = [&](int c0) {
    if (has_unit) {
      const int ya = y0 - R + c0, nr = min(G::CR, rows_total - c0);
      const float* s = unit_src + (long long)clampi(ya, 0, h - 1) * pitch;
      if (ya >= 0 && ya + G::CR <= h && nr == G::CR) {
#pragma unroll 4
        for (int r = 0; r < G::CR; ++r, s += pitch)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(unit_dst + r * G::P * 4), "l"(s) : "memory");
      } else {
#pragma unroll 1
        for (int r = 0; r < nr; ++r) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(unit_dst + r * G::P * 4), "l"(s) : "memory");
          if (ya + r >= 0 && ya + r < h - 1) s += pitch;
        }
      }
    }
  };
  issue(0);

  StripTaps<R> t;
#pragma unroll
  for (int k = 0; k <= R; ++k) t.w[k] = taps.w[k];
  t.one = taps.one;
  t.zero = make_float2(0.0f, 0.0f);
  const int gx = x0 + 2 * lane;
  const bool col_ok = gx < w;  // a pair's second column may lie in the row's padding
  // DOWN: the level's even rows and columns are the next octave's base
  const bool do_down = DOWN && octave + 1 < P.n_oct;
  const OctaveDev& Nx = P.oct[do_down ? octave + 1 : octave];
  const int down_h = min(Nx.h, (y1 + 1) >> 1);
  const long long down_pitch = Nx.pitch;
  const bool down_ok = do_down && (gx >> 1) < Nx.w;
  float* down = Nx.g + (gx >> 1);
  float* gout = O.g + (long long)level * O.plane_stride + gx;
  float2 va[N];  // the vertical pass's pending sums
#pragma unroll
  for (int m = 0; m < N; ++m) va[m] = t.zero;

  for (int c0 = 0; c0 < rows_total; c0 += G::CR) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    const int nr = min(G::CR, rows_total - c0);
#pragma unroll 1
    for (int r = lane; r < nr; r += 32) {
      float* row = buf + r * G::P;
      if (patch) {
        const float v0 = row[lead], v1 = row[last];
        for (int c = 0; c < lead; ++c) row[c] = v0;
        for (int c = last + 1; c < G::IN_W; ++c) row[c] = v1;
      }
      strip_row<R, FUSED>(row, t);
    }
    __syncwarp();
    const float* colp = buf + 2 * lane;
#pragma unroll 1
    for (int b = 0; b < G::CR; b += N, colp += N * G::P) {
      // output row completed by the block's first input row: y0 - 2R (a whole block
      // of rows above the segment, discarded), y0, y0 + 2R, ...  All are even.
      const int yb = y0 + c0 + b - N;
      if (yb >= y1) break;
      const int rows = col_ok && yb >= y0 ? y1 - yb : 0;
      const int rows_down = down_ok && yb >= y0 ? 2 * down_h - yb : 0;
      float* grow = gout + (long long)yb * pitch;
      float* drow = down + (long long)(yb >> 1) * down_pitch;
#pragma unroll
      for (int r = 0; r < N; ++r) {
        const float2 v = fir_row<R, FUSED>(va, *reinterpret_cast<const float2*>(colp + r * G::P), t, r);
        st_global_if(r < rows, grow, v);
        grow += pitch;
        if (DOWN && r % 2 == 0) {
          st_global_if(r < rows_down, drow, v.x);
          drow += down_pitch;
        }
      }
    }
    __syncwarp();
    if (c0 + G::CR < rows_total) issue(c0 + G::CR);
  }
}

}  // namespace psift
