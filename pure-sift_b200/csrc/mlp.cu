// K11: the learned correspondence scorer that drives guided RANSAC sampling.
// No counterpart in the reference (its sampler weights matches by 1/ratio,
// src/pipeline.rs:2006-2036).
//
// Network 8 -> 64 -> 64 -> 1, ReLU, ReLU, sigmoid.  Parameters are f32 masters;
// the forward pass rounds weights and activations to bf16 (round to nearest even)
// and accumulates in f32.  The backward pass is f32 on the same bf16-rounded
// operands (straight-through rounding).  Training is deterministic:
//   mlp_step_kernel    a cluster of CTAs per chunk of samples: forward, dL/dz for every layer,
//                      per-parameter sums over the chunk's samples in order;
//   mlp_update_kernel  sums over the chunks in order, Adam update of the f32 masters,
//                      the minibatch loss.
// Loss: mean binary cross-entropy over the minibatch.
#include <cooperative_groups.h>

#include <algorithm>

#include "psift_internal.cuh"

namespace cg = cooperative_groups;

namespace psift {

constexpr int kF = 8, kH = 64;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kH * kF, kOffW2 = kOffB1 + kH, kOffB2 = kOffW2 + kH * kH,
              kOffW3 = kOffB2 + kH, kOffB3 = kOffW3 + kH, kNP = kOffB3 + 1;  // 4801

__device__ __forceinline__ float bf16r(float x) {
  const uint32_t u = __float_as_uint(x);
  if ((u & 0x7f800000u) == 0x7f800000u) return x;  // inf / nan unchanged
  const uint32_t r = u + 0x7FFFu + ((u >> 16) & 1u);
  return __uint_as_float(r & 0xFFFF0000u);
}

struct MlpSmem {
  float w1[kH][kF];
  float b1[kH];
  float w2[kH][kH];
  float b2[kH];
  float w3[kH];
  float b3;
};

__device__ void load_params(const float* __restrict__ p, MlpSmem& s) {
  for (int i = threadIdx.x; i < kH * kF; i += blockDim.x) (&s.w1[0][0])[i] = bf16r(p[kOffW1 + i]);
  for (int i = threadIdx.x; i < kH * kH; i += blockDim.x) (&s.w2[0][0])[i] = bf16r(p[kOffW2 + i]);
  for (int i = threadIdx.x; i < kH; i += blockDim.x) {
    s.b1[i] = p[kOffB1 + i];
    s.b2[i] = p[kOffB2 + i];
    s.w3[i] = bf16r(p[kOffW3 + i]);
  }
  if (threadIdx.x == 0) s.b3 = p[kOffB3];
  __syncthreads();
}

// Forward of one sample; returns z3.
__device__ __forceinline__ float forward1(const MlpSmem& s, const float* __restrict__ x) {
  float xb[kF], h1b[kH];
#pragma unroll
  for (int k = 0; k < kF; ++k) xb[k] = bf16r(x[k]);
#pragma unroll
  for (int j = 0; j < kH; ++j) {
    float z = s.b1[j];
#pragma unroll
    for (int k = 0; k < kF; ++k) z = __fmaf_rn(s.w1[j][k], xb[k], z);
    h1b[j] = bf16r(z > 0.0f ? z : 0.0f);
  }
  float z3 = s.b3;
#pragma unroll 4
  for (int j = 0; j < kH; ++j) {
    float z = s.b2[j];
#pragma unroll
    for (int k = 0; k < kH; ++k) z = __fmaf_rn(s.w2[j][k], h1b[k], z);
    z3 = __fmaf_rn(s.w3[j], bf16r(z > 0.0f ? z : 0.0f), z3);
  }
  return z3;
}

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }

__global__ void __launch_bounds__(256) mlp_infer_kernel(const float* __restrict__ params, const float* __restrict__ X,
                                                        int n, float* __restrict__ prob) {
  __shared__ MlpSmem s;
  load_params(params, s);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    prob[i] = sigmoidf_(forward1(s, X + (size_t)i * kF));
  }
}

// One training step's samples, forward and backward, and their gradient sums: a cluster
// of kStepCtas CTAs per chunk of kGradChunk samples, everything in shared memory.  For
// the samples' passes each CTA takes a quarter of the chunk; for the sums over the
// chunk's samples each takes a quarter of the units and fetches its columns of the
// others' activations and derivatives through distributed shared memory.  The products
// (layer 2, its transpose, the W2 gradient) are register-tiled: a thread holds 4 x 2
// results and takes one step of the inner index at a time, so every result is the same
// chain of fused multiply-adds, in the same order, as one thread per sample (or per
// parameter) would compute.  Deterministic: parameter sums run over the chunk's samples
// in order, the chunks are added in order by mlp_update_kernel.
// Bound by shared-memory loads (a 4 x 2 tile loads 6 values for 8 multiply-adds) and by
// the latency of the phases, which depend on one another.
// A step of 4096 samples, its update included: 65.5 us as one-thread-per-sample and
// one-thread-per-parameter kernels through global memory, 41 with one CTA per chunk, 18.9
// like this; of 128 samples 61.8 -> 15.5, of 65,536 samples 266 -> 146 us.
constexpr int kGradChunk = 128;
constexpr int kStepCtas = 4;
constexpr int kStepThreads = 256;
constexpr int kCtaSamples = kGradChunk / kStepCtas;
constexpr int kCtaUnits = kH / kStepCtas;
constexpr int kSS = kCtaSamples + 4;  // row stride of [unit][sample] arrays
constexpr int kHS = kH + 4;           // row stride of [sample][unit] arrays and of w2
constexpr int kTS = kH + 2;           // row stride of w2t: two-way conflicts at most in its transposing stores

struct StepSmem {
  union {
    struct {
      float w2[kH][kHS];   // [j][k]
      float w2t[kH][kTS];  // [k][j]
    };
    float h1_all[kGradChunk][kH];  // after the passes: the chunk's layer-1 activations
  };
  union {
    float t[kH][kSS];  // h1 [k][sample], then dz2 [j][sample]
    float dz2_all[kGradChunk][kCtaUnits];  // after the passes: this CTA's units, as the next two
  };
  float dz1_all[kGradChunk][kCtaUnits];
  float h2_all[kGradChunk][kCtaUnits];
  float x_all[kGradChunk][kF];
  // this CTA's samples; read by the cluster
  float h1[kCtaSamples][kHS];  // activations: +0 where z <= 0, never elsewhere (see relu_bf16)
  float h2[kCtaSamples][kHS];
  float dz2[kCtaSamples][kHS];
  float dz1[kCtaSamples][kHS];
  float x[kCtaSamples][kF];
  float dz3[kCtaSamples];
  float w1[kH][kF];
  float b1[kH], b2[kH], w3[kH];
  float dz3_all[kGradChunk];
  float b3;
};

// bf16(max(z, 0)), with -0 for a positive z that rounds to zero: the bits are zero
// exactly where the ReLU is inactive.
__device__ __forceinline__ float relu_bf16(float z) {
  if (!(z > 0.0f)) return 0.0f;
  const float h = bf16r(z);
  return h == 0.0f ? -0.0f : h;
}
__device__ __forceinline__ bool active(float h) { return __float_as_uint(h) != 0u; }

// A step's two kernels and the next step's follow one another without a gap
// (programmatic dependent launch): a kernel's CTAs start while the previous kernel's run
// and wait here for it to complete; before that they only read what no kernel of the
// training loop writes (samples, labels, indices).  The loop's first kernel waits for
// everything before it.
__device__ __forceinline__ void next_kernel_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__global__ void __cluster_dims__(kStepCtas, 1, 1) __launch_bounds__(kStepThreads, 2)
    mlp_step_kernel(const float* __restrict__ params, const float* __restrict__ X, const float* __restrict__ Y,
                    const int* __restrict__ idx, int B, float* __restrict__ loss_o, float* __restrict__ partial) {
  extern __shared__ __align__(16) uint8_t step_smem[];
  StepSmem& s = *reinterpret_cast<StepSmem*>(step_smem);
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = (int)cluster.block_rank(), chunk = blockIdx.x / kStepCtas;
  const int nb = min(kGradChunk, B - chunk * kGradChunk);             // the chunk's samples
  const int s0 = chunk * kGradChunk + rank * kCtaSamples;             // this CTA's first
  const int ns = min(kCtaSamples, max(nb - rank * kCtaSamples, 0));   // and how many (the rest count as zeros)
  {  // features, a value per thread
    const int r = tid / kF, k = tid % kF;
    s.x[r][k] = r < ns ? bf16r(X[(size_t)(idx ? idx[s0 + r] : s0 + r) * kF + k]) : 0.0f;
  }
  next_kernel_may_start();
  wait_for_previous_kernel();
  // parameters, the weights rounded to bf16
  for (int i = tid; i < kH * kF; i += kStepThreads) (&s.w1[0][0])[i] = bf16r(params[kOffW1 + i]);
#pragma unroll
  for (int q = 0; q < kH * kH / kStepThreads; ++q) {
    const int i = tid + q * kStepThreads;
    const float w = bf16r(params[kOffW2 + i]);
    s.w2[i / kH][i % kH] = w;
    s.w2t[i % kH][i / kH] = w;
  }
  if (tid < kH) {
    s.b1[tid] = params[kOffB1 + tid];
    s.b2[tid] = params[kOffB2 + tid];
    s.w3[tid] = bf16r(params[kOffW3 + tid]);
  }
  if (tid == 0) s.b3 = params[kOffB3];
  __syncthreads();
  const int v0 = 8 * warp;  // lane: a sample, warp: 8 units
  {                         // layer 1
    float x[kF], h[8];
#pragma unroll
    for (int k = 0; k < kF; ++k) x[k] = s.x[lane][k];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      float z = s.b1[v0 + q];
#pragma unroll
      for (int k = 0; k < kF; ++k) z = __fmaf_rn(s.w1[v0 + q][k], x[k], z);
      h[q] = relu_bf16(z);
      s.t[v0 + q][lane] = h[q];
    }
    *reinterpret_cast<float4*>(&s.h1[lane][v0]) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(&s.h1[lane][v0 + 4]) = make_float4(h[4], h[5], h[6], h[7]);
  }
  __syncthreads();
  // 4 (samples) x 2 (units) tiles: a warp covers the 32 samples x 8 units, lanes 8 x 4
  // tiles (two loads without conflicts per step)
  const int r0 = 4 * (lane & 7), u0 = 8 * warp + 2 * (lane >> 3);
  {  // layer 2
    float acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[i][0] = s.b2[u0];
      acc[i][1] = s.b2[u0 + 1];
    }
#pragma unroll 8
    for (int k = 0; k < kH; ++k) {
      const float4 h = *reinterpret_cast<const float4*>(&s.t[k][r0]);
      const float2 w = *reinterpret_cast<const float2*>(&s.w2t[k][u0]);
      const float hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][0] = __fmaf_rn(w.x, hv[i], acc[i][0]);
        acc[i][1] = __fmaf_rn(w.y, hv[i], acc[i][1]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float2*>(&s.h2[r0 + i][u0]) = make_float2(relu_bf16(acc[i][0]), relu_bf16(acc[i][1]));
  }
  __syncthreads();
  // layer 3, loss and its derivative: a thread per sample
  if (tid < kCtaSamples) {
    float z3 = s.b3;
#pragma unroll
    for (int j = 0; j < kH; j += 4) {
      const float4 h = *reinterpret_cast<const float4*>(&s.h2[tid][j]);
      z3 = __fmaf_rn(s.w3[j], h.x, z3);
      z3 = __fmaf_rn(s.w3[j + 1], h.y, z3);
      z3 = __fmaf_rn(s.w3[j + 2], h.z, z3);
      z3 = __fmaf_rn(s.w3[j + 3], h.w, z3);
    }
    float dz3 = 0.0f;
    if (tid < ns) {
      const float y = Y[idx ? idx[s0 + tid] : s0 + tid];
      const float p = sigmoidf_(z3);
      // BCE with logits: softplus(z) - y z, numerically stable form
      loss_o[s0 + tid] = fmaxf(z3, 0.0f) - z3 * y + log1pf(expf(-fabsf(z3)));
      dz3 = (p - y) * (1.0f / (float)B);
    }
    s.dz3[tid] = dz3;
  }
  __syncthreads();
  {
    const float4 ha = *reinterpret_cast<const float4*>(&s.h2[lane][v0]), hb = *reinterpret_cast<const float4*>(&s.h2[lane][v0 + 4]);
    const float h[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
    const float dz3 = s.dz3[lane];
    float d[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      d[q] = active(h[q]) ? dz3 * s.w3[v0 + q] : 0.0f;
      s.t[v0 + q][lane] = d[q];
    }
    *reinterpret_cast<float4*>(&s.dz2[lane][v0]) = make_float4(d[0], d[1], d[2], d[3]);
    *reinterpret_cast<float4*>(&s.dz2[lane][v0 + 4]) = make_float4(d[4], d[5], d[6], d[7]);
  }
  __syncthreads();
  {  // back through layer 2
    float acc[4][2] = {};
#pragma unroll 8
    for (int j = 0; j < kH; ++j) {
      const float4 d = *reinterpret_cast<const float4*>(&s.t[j][r0]);
      const float2 w = *reinterpret_cast<const float2*>(&s.w2[j][u0]);
      const float dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][0] = __fmaf_rn(w.x, dv[i], acc[i][0]);
        acc[i][1] = __fmaf_rn(w.y, dv[i], acc[i][1]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 h = *reinterpret_cast<const float2*>(&s.h1[r0 + i][u0]);
      *reinterpret_cast<float2*>(&s.dz1[r0 + i][u0]) =
          make_float2(active(h.x) ? acc[i][0] : 0.0f, active(h.y) ? acc[i][1] : 0.0f);
    }
  }
  cluster.sync();
  // the chunk's layer-1 activations and features, and this CTA's units of the rest
  const int c0 = kCtaUnits * rank;
#pragma unroll
  for (int q = 0; q < kGradChunk * kH / 4 / kStepThreads; ++q) {
    const int i = tid + q * kStepThreads, b = i / (kH / 4), c = 4 * (i % (kH / 4));
    const StepSmem* o = cluster.map_shared_rank(&s, (unsigned)(b / kCtaSamples));
    *reinterpret_cast<float4*>(&s.h1_all[b][c]) = *reinterpret_cast<const float4*>(&o->h1[b % kCtaSamples][c]);
  }
#pragma unroll
  for (int q = 0; q < kGradChunk * kCtaUnits / 4 / kStepThreads; ++q) {
    const int i = tid + q * kStepThreads, b = i / (kCtaUnits / 4), c = 4 * (i % (kCtaUnits / 4)), r = b % kCtaSamples;
    const StepSmem* o = cluster.map_shared_rank(&s, (unsigned)(b / kCtaSamples));
    *reinterpret_cast<float4*>(&s.dz2_all[b][c]) = *reinterpret_cast<const float4*>(&o->dz2[r][c0 + c]);
    *reinterpret_cast<float4*>(&s.dz1_all[b][c]) = *reinterpret_cast<const float4*>(&o->dz1[r][c0 + c]);
    *reinterpret_cast<float4*>(&s.h2_all[b][c]) = *reinterpret_cast<const float4*>(&o->h2[r][c0 + c]);
  }
  {
    const int b = tid / 2, c = 4 * (tid % 2);
    const StepSmem* o = cluster.map_shared_rank(&s, (unsigned)(b / kCtaSamples));
    *reinterpret_cast<float4*>(&s.x_all[b][c]) = *reinterpret_cast<const float4*>(&o->x[b % kCtaSamples][c]);
    if (c == 0) s.dz3_all[b] = o->dz3[b % kCtaSamples];
  }
  cluster.sync();  // also: nobody reads this CTA's arrays any more
  float* part = partial + (size_t)chunk * kNP;
  if (warp < 4) {  // W2: 4 (j) x 2 (k) per thread, lanes 4 x 8 tiles
    const int j0 = 4 * (lane & 3), k0 = 16 * warp + 2 * (lane >> 2);
    float acc[4][2] = {};
#pragma unroll 8
    for (int b = 0; b < nb; ++b) {
      const float4 d = *reinterpret_cast<const float4*>(&s.dz2_all[b][j0]);
      const float2 h = *reinterpret_cast<const float2*>(&s.h1_all[b][k0]);
      const float dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[j][0] = __fmaf_rn(dv[j], h.x, acc[j][0]);
        acc[j][1] = __fmaf_rn(dv[j], h.y, acc[j][1]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 2; ++k) part[kOffW2 + (c0 + j0 + j) * kH + k0 + k] = acc[j][k];
  } else if (warp < 6) {  // W1: 1 (j) x 2 (k)
    const int j = (tid - 128) / (kF / 2), k = 2 * (tid % (kF / 2));
    float g0 = 0.0f, g1 = 0.0f;
#pragma unroll 8
    for (int b = 0; b < nb; ++b) {
      const float d = s.dz1_all[b][j];
      const float2 x = *reinterpret_cast<const float2*>(&s.x_all[b][k]);
      g0 = __fmaf_rn(d, x.x, g0);
      g1 = __fmaf_rn(d, x.y, g1);
    }
    part[kOffW1 + (c0 + j) * kF + k] = g0;
    part[kOffW1 + (c0 + j) * kF + k + 1] = g1;
  } else {  // biases and W3
    const int q = tid - 192, j = q % kCtaUnits;
    float g = 0.0f;
    if (q < kCtaUnits) {
#pragma unroll 8
      for (int b = 0; b < nb; ++b) g += s.dz1_all[b][j];
      part[kOffB1 + c0 + j] = g;
    } else if (q < 2 * kCtaUnits) {
#pragma unroll 8
      for (int b = 0; b < nb; ++b) g += s.dz2_all[b][j];
      part[kOffB2 + c0 + j] = g;
    } else if (q < 3 * kCtaUnits) {
#pragma unroll 8
      for (int b = 0; b < nb; ++b) g = __fmaf_rn(s.dz3_all[b], s.h2_all[b][j], g);
      part[kOffW3 + c0 + j] = g;
    } else if (q == 3 * kCtaUnits && rank == 0) {
#pragma unroll 8
      for (int b = 0; b < nb; ++b) g += s.dz3_all[b];
      part[kOffB3] = g;
    }
  }
}
static_assert(2 * (sizeof(StepSmem) + 1024) <= 228 * 1024, "two CTAs per SM");
static_assert(kCtaSamples == 32 && kCtaUnits == 16 && kStepThreads == kCtaSamples * kF && kH == 8 * (kStepThreads / 32),
              "tiles cover the chunk");

// Adds the chunks' gradient sums in chunk order and, with `update`, takes the Adam step
// on the f32 masters; the last CTA writes the mean of the per-sample losses, in a fixed
// order: thread t sums samples t, t + 256, t + 512, ..., then a fixed pairwise tree.
// Bound by the latency of its loads: a CTA takes 32 parameters, its 8 warps fetch the
// rows of up to kUpdateTile chunks at once and the first one adds them in order.
// With the overlapped launches a step of 4096 samples takes 18.9 us, 20.5 with a thread
// per parameter reading 16 chunks ahead and the kernels one after the other.
constexpr int kUpdateThreads = 256;
constexpr int kUpdateParams = 32;
constexpr int kUpdateTile = 128;  // chunks in shared memory at a time
__global__ void __launch_bounds__(kUpdateThreads) mlp_update_kernel(
    int chunks, const float* __restrict__ partial, float* __restrict__ grad, float* __restrict__ params,
    float* __restrict__ m, float* __restrict__ v, bool update, float lr, float beta1, float beta2, float eps, float bc1,
    float bc2, const float* __restrict__ l, int B, float* __restrict__ loss_out) {
  __shared__ float part[kUpdateTile][kUpdateParams];
  const int t = threadIdx.x;
  wait_for_previous_kernel();
  next_kernel_may_start();  // not sooner: its clusters would share SMs that the last step's still hold
  if (blockIdx.x == gridDim.x - 1) {
    if (!loss_out) return;
    float* sums = &part[0][0];
    float sum = 0.0f;
#pragma unroll 32
    for (int b = t; b < B; b += kUpdateThreads) sum += l[b];
    sums[t] = sum;
    __syncthreads();
    for (int h = kUpdateThreads / 2; h > 0; h >>= 1) {
      if (t < h) sums[t] += sums[t + h];
      __syncthreads();
    }
    if (t == 0) *loss_out = sums[0] / (float)B;
    return;
  }
  constexpr int kRows = kUpdateThreads / kUpdateParams;
  const int lane = t % kUpdateParams, row = t / kUpdateParams, p = blockIdx.x * kUpdateParams + lane;
  const bool own = row == 0 && p < kNP, adam = own && update;
  const float m0 = adam ? m[p] : 0.0f, v0 = adam ? v[p] : 0.0f, w0 = adam ? params[p] : 0.0f;
  float g = 0.0f;
  for (int c0 = 0; c0 < chunks; c0 += kUpdateTile) {
    const int n = min(kUpdateTile, chunks - c0);
    float x[kUpdateTile / kRows];
#pragma unroll
    for (int q = 0; q < kUpdateTile / kRows; ++q) {
      const int c = row + q * kRows;
      x[q] = c < n && p < kNP ? partial[(size_t)(c0 + c) * kNP + p] : 0.0f;
    }
    __syncthreads();  // the previous tile is added
#pragma unroll
    for (int q = 0; q < kUpdateTile / kRows; ++q) part[row + q * kRows][lane] = x[q];
    __syncthreads();
    if (own) {
#pragma unroll 16
      for (int c = 0; c < n; ++c) g += part[c][lane];
    }
  }
  if (!own) return;
  grad[p] = g;
  if (update) {
    const float mm = beta1 * m0 + (1.0f - beta1) * g;
    const float vv = beta2 * v0 + (1.0f - beta2) * g * g;
    m[p] = mm;
    v[p] = vv;
    params[p] = w0 - lr * (mm / bc1) / (sqrtf(vv / bc2) + eps);
  }
}

// ------------------------------------------------------------ tensor-core inference
// mlp_infer_tc_kernel: the same network on bf16 tensor-core tiles
// (mma.sync m16n8k16, f32 accumulation).  A warp evaluates 16 samples per tile:
// layer 1 (K = 8 features, padded to 16) and layer 2 (K = 64) are MMAs whose f32
// accumulators start at the biases; the layer-1 accumulator fragment, ReLU'd and
// rounded to bf16, is exactly the layer-2 A fragment (rows g / g + 8, columns
// 2t, 2t + 1 of consecutive 8-column tiles), so activations never leave the
// registers; layer 3 is a per-row dot product reduced over the 4 lanes of a
// quad.  The bf16-rounded weights live in registers for the whole kernel.
// Operand rounding is the scalar kernel's (bf16, round to nearest even); only
// the f32 summation order inside a product differs.
//
// Input staging: persistent CTAs (one per SM) take chunks of kMlpChunk samples
// (32 KB) round-robin; thread 0 streams them into a kMlpStages-deep shared-memory
// ring with 1-D bulk async copies (cp.async.bulk, mbarrier completion), so the
// HBM reads run ahead of the tensor work.  Every wait is bounded: on timeout the
// CTA records kErrTimeout in err and returns once its issued copies have landed.
constexpr int kMlpThreads = 256;
constexpr int kMlpWarps = kMlpThreads / 32;
constexpr int kMlpChunk = 1024;  // samples per ring stage
constexpr int kMlpStages = 4;
constexpr uint32_t kMlpSpin = 1u << 24;
constexpr size_t kMlpSmem = (size_t)kMlpStages * kMlpChunk * kF * sizeof(float) + 128;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// {lo, hi} -> bf16x2 (round to nearest even), lo in the low half.
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ bool mlp_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < kMlpSpin; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__global__ void __launch_bounds__(kMlpThreads, 1) mlp_infer_tc_kernel(const float* __restrict__ params,
                                                                      const float* __restrict__ X, int n,
                                                                      float* __restrict__ prob, uint32_t* err) {
  extern __shared__ __align__(128) uint8_t mlp_smem[];
  float* xs = reinterpret_cast<float*>(mlp_smem);
  uint64_t* full = reinterpret_cast<uint64_t*>(mlp_smem + (size_t)kMlpStages * kMlpChunk * kF * sizeof(float));
  uint64_t* empty = full + kMlpStages;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int n_chunks = (n + kMlpChunk - 1) / kMlpChunk;
  if ((int)blockIdx.x >= n_chunks) return;
  const int my_chunks = (n_chunks - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  auto chunk_samples = [&](int i) {
    const int base = ((int)blockIdx.x + i * (int)gridDim.x) * kMlpChunk;
    return min(kMlpChunk, n - base);
  };
  auto issue = [&](int i) {  // thread 0: chunk i of this CTA into stage i % kMlpStages
    const int s = i % kMlpStages;
    const long long base = ((long long)blockIdx.x + (long long)i * gridDim.x) * kMlpChunk;
    const uint32_t bytes = (uint32_t)chunk_samples(i) * kF * sizeof(float);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&full[s])), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(xs + (size_t)s * kMlpChunk * kF)),
        "l"(X + base * kF), "r"(bytes), "r"(smem_addr(&full[s]))
        : "memory");
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMlpStages; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&empty[s])), "r"(kMlpWarps) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int i = 0; i < kMlpStages && i < my_chunks; ++i) issue(i);
  }
  // bf16 weight fragments (B operands: column n = output g of the 8-column tile,
  // rows k = 2t, 2t + 1 and 2t + 8, 2t + 9 of the 16-deep K step) and biases for
  // the accumulator columns 2t, 2t + 1 of each 8-column tile
  uint32_t w1r[8], w2r[4][8][2];
  float b1v[8][2], b2v[8][2], w3v[8][2];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    const int j = nt * 8 + g;
    w1r[nt] = pack_bf16(params[kOffW1 + j * kF + 2 * t], params[kOffW1 + j * kF + 2 * t + 1]);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const float* w = params + kOffW2 + j * kH + kk * 16 + 2 * t;
      w2r[kk][nt][0] = pack_bf16(w[0], w[1]);
      w2r[kk][nt][1] = pack_bf16(w[8], w[9]);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      b1v[nt][c] = params[kOffB1 + nt * 8 + 2 * t + c];
      b2v[nt][c] = params[kOffB2 + nt * 8 + 2 * t + c];
      w3v[nt][c] = bf16r(params[kOffW3 + nt * 8 + 2 * t + c]);
    }
  }
  const float b3 = params[kOffB3];
  __syncthreads();  // barriers initialised
  bool ok = true;
  for (int i = 0; i < my_chunks; ++i) {
    const int s = i % kMlpStages;
    const uint32_t par = (uint32_t)(i / kMlpStages) & 1u;
    if (!mlp_wait(&full[s], par)) {
      ok = false;
      break;
    }
    const float* xc = xs + (size_t)s * kMlpChunk * kF;
    const int cnt = chunk_samples(i);
    const long long base = ((long long)blockIdx.x + (long long)i * gridDim.x) * kMlpChunk;
    for (int tile = warp; tile * 16 < cnt; tile += kMlpWarps) {
      // layer 1: A = the tile's 16 x 8 features (K padded with zeros)
      const float2 xa = *reinterpret_cast<const float2*>(xc + (tile * 16 + g) * kF + 2 * t);
      const float2 xb = *reinterpret_cast<const float2*>(xc + (tile * 16 + g + 8) * kF + 2 * t);
      const uint32_t a1[4] = {pack_bf16(xa.x, xa.y), pack_bf16(xb.x, xb.y), 0u, 0u};
      uint32_t a2[4][4];
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        float c[4] = {b1v[nt][0], b1v[nt][1], b1v[nt][0], b1v[nt][1]};
        mma_bf16_16816(c, a1, w1r[nt], 0u);
        // ReLU, bf16: this tile is K columns 8 (nt & 1) .. of layer 2's K step nt / 2
        a2[nt >> 1][(nt & 1) * 2 + 0] = pack_bf16(fmaxf(c[0], 0.0f), fmaxf(c[1], 0.0f));
        a2[nt >> 1][(nt & 1) * 2 + 1] = pack_bf16(fmaxf(c[2], 0.0f), fmaxf(c[3], 0.0f));
      }
      // layer 2 and the layer-3 dot products of rows g and g + 8
      float z_lo = 0.0f, z_hi = 0.0f;
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        float c[4] = {b2v[nt][0], b2v[nt][1], b2v[nt][0], b2v[nt][1]};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) mma_bf16_16816(c, a2[kk], w2r[kk][nt][0], w2r[kk][nt][1]);
        z_lo = __fmaf_rn(w3v[nt][0], bf16r(fmaxf(c[0], 0.0f)), z_lo);
        z_lo = __fmaf_rn(w3v[nt][1], bf16r(fmaxf(c[1], 0.0f)), z_lo);
        z_hi = __fmaf_rn(w3v[nt][0], bf16r(fmaxf(c[2], 0.0f)), z_hi);
        z_hi = __fmaf_rn(w3v[nt][1], bf16r(fmaxf(c[3], 0.0f)), z_hi);
      }
      z_lo += __shfl_xor_sync(0xffffffffu, z_lo, 1);
      z_hi += __shfl_xor_sync(0xffffffffu, z_hi, 1);
      z_lo += __shfl_xor_sync(0xffffffffu, z_lo, 2);
      z_hi += __shfl_xor_sync(0xffffffffu, z_hi, 2);
      if (t == 0) {
        const int r0 = tile * 16 + g, r1 = r0 + 8;
        if (r0 < cnt) prob[base + r0] = sigmoidf_(b3 + z_lo);
        if (r1 < cnt) prob[base + r1] = sigmoidf_(b3 + z_hi);
      }
    }
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&empty[s])) : "memory");
    if (threadIdx.x == 0 && i + kMlpStages < my_chunks) {
      // refill this stage once every warp is done with it
      if (!mlp_wait(&empty[s], par)) {
        ok = false;
        break;
      }
      issue(i + kMlpStages);
    }
  }
  if (!ok) {
    atomicOr(err, kErrTimeout);
    // wait (bounded) for this CTA's copies still in flight before the CTA exits
    if (threadIdx.x == 0) {
      const int issued = min(my_chunks, kMlpStages);
      for (int i = 0; i < issued; ++i) mlp_wait(&full[i % kMlpStages], (uint32_t)(i / kMlpStages) & 1u);
    }
  }
}

cudaError_t launch_mlp_infer(const float* params, const float* X, int n, float* prob, int num_sms, uint32_t* err,
                             cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if ((reinterpret_cast<uintptr_t>(X) & 15u) == 0) {
    // tensor-core path: the bulk copies need 16-byte aligned rows (32 B per sample)
    cudaError_t e = ensure_smem_attr((const void*)mlp_infer_tc_kernel, kMlpSmem);
    if (e != cudaSuccess) return e;
    const int chunks = (n + kMlpChunk - 1) / kMlpChunk;
    mlp_infer_tc_kernel<<<std::min(chunks, num_sms), kMlpThreads, kMlpSmem, st>>>(params, X, n, prob, err);
    return cudaGetLastError();
  }
  const int blocks = std::min((n + 255) / 256, num_sms * 8);
  mlp_infer_kernel<<<blocks, 256, 0, st>>>(params, X, n, prob);
  return cudaGetLastError();
}

// Workspace for a minibatch of B: the per-sample losses, then one row of kNP partial
// gradient sums per kGradChunk samples.
size_t mlp_batch_floats(int B) { return (size_t)B + (size_t)((B + kGradChunk - 1) / kGradChunk) * kNP; }

cudaError_t launch_mlp_step(float* params, const float* X, const float* Y, const int* idx, int B, float* work,
                            float* grad, float* m, float* v, float lr, int t, float* loss_out, bool update,
                            cudaStream_t st) {
  float* lb = work;
  float* partial = lb + B;
  const int chunks = (B + kGradChunk - 1) / kGradChunk;
  cudaError_t e = ensure_smem_attr((const void*)mlp_step_kernel, sizeof(StepSmem));
  if (e != cudaSuccess) return e;
  const float b1 = 0.9f, b2 = 0.999f;
  const float bc1 = 1.0f - powf(b1, (float)t), bc2 = 1.0f - powf(b2, (float)t);
  cudaLaunchAttribute overlap;
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(chunks * kStepCtas));
  cfg.blockDim = dim3(kStepThreads);
  cfg.dynamicSmemBytes = sizeof(StepSmem);
  cfg.stream = st;
  cfg.attrs = &overlap;
  cfg.numAttrs = t > 1 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, mlp_step_kernel, (const float*)params, X, Y, idx, B, lb, partial);
  if (e != cudaSuccess) return e;
  cfg.gridDim = dim3((unsigned)((kNP + kUpdateParams - 1) / kUpdateParams + 1));
  cfg.blockDim = dim3(kUpdateThreads);
  cfg.dynamicSmemBytes = 0;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, mlp_update_kernel, chunks, (const float*)partial, grad, params, m, v, update, lr, b1, b2,
                            1e-8f, bc1, bc2, (const float*)lb, B, loss_out);
}

}  // namespace psift
