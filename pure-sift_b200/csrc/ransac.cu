// K10: similarity RANSAC and homography LO-RANSAC on the GPU, one CTA per match set.
//
// Reference (src/pipeline.rs): splitmix64_next (:1862-1868),
// evaluate_similarity_hypothesis (:1873-1897), fit_procrustes_similarity
// (:1900-1975), adaptive_ransac_iters (:1979-2002), build_ratio_weighted_cdf /
// sample_weighted_index (:2006-2036), filter_matches_ransac_with_seed
// (:2055-2191), smallest_eigenvector_9x9 (:2276-2353), has_degenerate_triangle /
// is_degenerate_quad (:2357-2404), fit_homography_dlt_f64 (:2408-2528),
// evaluate_homography_hypothesis_f64 / collect (:2550-2601),
// local_optimize_homography (:2605-2631), estimate_homography_ransac_with_seeds
// (:2663-2755).
//
// Identical results for the same seed.  The random stream does not depend on
// the data except through the CDF, so samples are drawn ahead: splitmix64's
// state advances by a constant, draw t is a pure function of (seed, t).
// Hypotheses are generated and fitted a batch (a quarter of the CTA's threads) at a
// time: a quad of lanes per homography fit (f64 DLT; the cyclic Jacobi's rotations shared by the quad in
// shared memory, each lane updating rows ql, ql + 4, ql + 8, so every value is
// the sequential solver's), then counted by warps (two hypotheses per pass over
// the packed match coordinates, no block barrier), and the reference's loop is
// replayed in order by every thread on identical shared values: every decision
// (count, tie on the sequential error sum, adaptive iteration budget, LO
// refinement) is taken exactly as the reference takes it.  Error sums are needed
// only to break a tie on the count, so they are computed when a tie occurs (for
// the incumbent too, if its sum is not known yet): an error sum is a function of
// the model alone, so the deferred value is the one the reference computed.
// Error sums are the reference's sequential sums over the matches in input order
// (terms computed in parallel, summed serially); LO refits accumulate A^T A per
// entry sequentially over the inliers in order (45 threads) and solve it with one
// quad.
#include <stdint.h>

#include "psift_internal.cuh"
#include "ransac_common.cuh"

namespace psift {

template <int N>
struct Int {
  static constexpr int value = N;
};

// ---- packed f32x2
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "mul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// Offsets i * 9 + j, i < j, of a 9 x 9 matrix's strict upper triangle.
static __constant__ uint8_t kStrictUpper[36] = {1,  2,  3,  4,  5,  6,  7,  8,  11, 12, 13, 14, 15, 16, 17, 21, 22, 23,
                                                24, 25, 26, 31, 32, 33, 34, 35, 41, 42, 43, 44, 51, 52, 53, 61, 62, 71};

// A CTA's threads, by the match sets of a launch (see launch_ransac).  512 threads fit and
// count the most hypotheses at a time, which is what a set with many outliers spends its
// time on, and take a whole SM; the serial parts (replay, sequential sums, the Jacobi of a
// refit) leave most of them idle, so once there are several sets per SM two CTAs of 256
// threads side by side (128 registers, ~100 KB of shared memory) or four of 128 get more done.
template <int THREADS>
struct RansacCta {
static constexpr int kRThreads = THREADS;
static constexpr int kRWarps = kRThreads / 32;
static constexpr int kBatch = kRThreads / 4;  // a quad of lanes per hypothesis fit
// the weight sums are taken by 128 threads whatever the CTA's size, so that a set's
// sums (and its iteration budget) do not depend on the launch it is part of
static constexpr int kMassThreads = 128;
static constexpr int kDrawChunk = kBatch * 16;
// Jacobi matrix and eigenvectors (81 doubles each) of every hypothesis of a batch
static constexpr size_t kJacSmem = sizeof(double) * 162 * kBatch;
// LO refits stage row values (10 doubles per point) in the same buffer
static constexpr int kRowChunk = (int)(kJacSmem / (sizeof(double) * 10));
// sequential sums over an inlier list stage its points (float4) there
static constexpr int kPtChunk = (int)(kJacSmem / sizeof(float4));
// and the counts the first matches' coordinates, as four float arrays of kStage; the
// last eighth is left to ordered_sum, which breaks ties while they are staged
static constexpr size_t kSumOff = kJacSmem / 8 * 7 / 16 * 16;
static constexpr int kStage = (int)(kSumOff / sizeof(float4)) / 64 * 64;

struct RShared {
  int n;
  float tsq_f;
  double tsq_d;
  int top32[32];
  // batch of hypotheses
  float ha[kBatch], hb[kBatch], htx[kBatch], hty[kBatch];
  double H[kBatch][9];
  float4 hband[kBatch];  // the f32 test's bounds (see h_band)
  double BH[9], Hc[9];   // the incumbent homography, the candidate being refined
  unsigned coord_max[3];  // bits of max |query x|, |query y|, |target x or y| over the matches
  int hvalid[kBatch];
  int hcnt[kBatch];
  int quad[kBatch][4];
  // scratch scalars
  unsigned long long key_min;
  int flag;
  float fres[8];
  double dres[16];
  double ata[9][9];
  int draw_ptr, draws_ready, dup;
  int draws_s[2 * kDrawChunk];  // draw t lives at [t % (2 * kDrawChunk)]
  int sim_count;
  float sim_model[6];
  int has_sim;
  uint32_t red_u[32];
  double red_d[32];
};

// build_ratio_weighted_cdf: weights in parallel, the running sum sequentially.
static __device__ void build_cdf(const RansacJob& J, RShared& S) {
  const int n = S.n;
  for (int i = threadIdx.x; i < n; i += kRThreads) {
    double w;
    if (J.weights) {
      w = (double)J.weights[i];
    } else {
      const float r = J.m[i].ratio;
      double rd = 1.0;
      if (isfinite(r)) {
        rd = (double)r;
        rd = rd < 0.05 ? 0.05 : (rd > 1.0 ? 1.0 : rd);
      }
      w = 1.0 / rd;
    }
    J.cdf[i] = w;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // running sum in order; 16 weights are loaded ahead of the dependent additions
    double acc = 0.0;
    int i = 0;
    for (; i + 16 <= n; i += 16) {
      double w[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) w[u] = J.cdf[i + u];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        acc += w[u];
        J.cdf[i + u] = acc;
      }
    }
    for (; i < n; ++i) {
      acc += J.cdf[i];
      J.cdf[i] = acc;
    }
    S.dres[0] = acc;
  }
  __syncthreads();
  const double acc = S.dres[0];
  if (acc > 0.0) {
    const double inv = 1.0 / acc;
    for (int i = threadIdx.x; i < n; i += kRThreads) J.cdf[i] *= inv;
  }
  __syncthreads();
  if (threadIdx.x == 0 && n > 0) J.cdf[n - 1] = 1.0;
  __syncthreads();
}

// adaptive_ransac_iters (src/pipeline.rs:1979-2002).
static __device__ int adaptive_iters(int inl, int total, int ss, int min_it, int cap) {
  if (total == 0 || inl == 0) return cap;
  double w = (double)inl / (double)total;
  w = w < 1e-3 ? 1e-3 : (w > 1.0 - 1e-6 ? 1.0 - 1e-6 : w);
  double p = w * w;  // powi(w, 2) / powi(w, 4) as the compiler runtime evaluates them
  if (ss == 4) p = p * p;
  p = p < 1e-12 ? 1e-12 : (p > 1.0 - 1e-9 ? 1.0 - 1e-9 : p);
  const double num = log(1.0 - 0.999);
  const double den = log(1.0 - p);
  if (fabs(den) < 1e-12) return min_it;
  const double est = ceil(num / den);
  if (!isfinite(est)) return cap;
  double c = est;
  if (c < (double)min_it) c = (double)min_it;
  if (c > (double)cap) c = (double)cap;
  return (int)c;
}

// ---------------------------------------------------------- block reductions
static __device__ __forceinline__ int block_sum_int(int v, RShared& S) {
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) S.red_u[threadIdx.x >> 5] = (uint32_t)v;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < kRWarps; ++w) t += (int)S.red_u[w];
  __syncthreads();
  return t;
}

static __device__ __forceinline__ double block_sum_double(double v, RShared& S) {
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) S.red_d[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < kRWarps; ++w) t += S.red_d[w];
  __syncthreads();
  return t;
}

// Guided sampling stops on the sampled inlier mass: the probability that one
// draw hits an inlier of the current model is w = sum over its inliers of the
// sampling weight / total weight (the reference's count / n when the weights are
// uniform).  Same formula as adaptive_ransac_iters otherwise.
static __device__ int adaptive_iters_w(double w, int ss, int min_it, int cap) {
  if (!(w > 0.0)) return cap;
  w = w < 1e-3 ? 1e-3 : (w > 1.0 - 1e-6 ? 1.0 - 1e-6 : w);
  double p = w * w;
  if (ss == 4) p = p * p;
  p = p < 1e-12 ? 1e-12 : (p > 1.0 - 1e-9 ? 1.0 - 1e-9 : p);
  const double num = log(1.0 - 0.999);
  const double den = log(1.0 - p);
  if (fabs(den) < 1e-12) return min_it;
  const double est = ceil(num / den);
  if (!isfinite(est)) return cap;
  double c = est;
  if (c < (double)min_it) c = (double)min_it;
  if (c > (double)cap) c = (double)cap;
  return (int)c;
}

// Sequential sum, in match order, of term(i) for i < n: the CTA computes the
// terms of a chunk into shared memory (the end of the batch's Jacobi space, free
// whenever a sum is taken), thread 0 adds them in order with its loads issued ahead of the
// dependent additions; the result is returned to every thread.  Terms of matches
// that are not inliers are zero, which leaves the running sum unchanged (x + 0 ==
// x for the finite, non-negative partial sums), so this equals the reference's
// sum over the inliers alone.
template <typename T, typename Term>
static __device__ T ordered_sum(RShared& S, int n, Term term) {
  extern __shared__ double jac[];
  T* buf = reinterpret_cast<T*>(reinterpret_cast<uint8_t*>(jac) + kSumOff);
  constexpr int cap = (int)((kJacSmem - kSumOff) / sizeof(T));
  T s = T(0);
  for (int c0 = 0; c0 < n; c0 += cap) {
    const int cn = min(cap, n - c0);
    for (int j = threadIdx.x; j < cn; j += kRThreads) buf[j] = term(c0 + j);
    __syncthreads();
    if (threadIdx.x == 0) {
      int j = 0;
      for (; j + 16 <= cn; j += 16) {
        T e[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) e[u] = buf[j + u];
#pragma unroll
        for (int u = 0; u < 16; ++u) s += e[u];
      }
      for (; j < cn; ++j) s += buf[j];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) S.dres[15] = (double)s;  // exact for float too
  __syncthreads();
  const T r = (T)S.dres[15];
  __syncthreads();
  return r;
}

// ------------------------------------------------------------- similarity
// evaluate_similarity_hypothesis's per-match test (src/pipeline.rs:1884-1893).
static __device__ __forceinline__ bool sim_inlier(const float4 p, float a, float b, float tx, float ty, float tsq, float& e) {
  const float px = a * p.x - b * p.y + tx;
  const float py = b * p.x + a * p.y + ty;
  const float dx = px - p.z;
  const float dy = py - p.w;
  e = dx * dx + dy * dy;
  return e <= tsq;
}

// Whether a warp's hypothesis, counted so far to c (per lane) with `rest` matches to go,
// can still reach `best`, the incumbent's count.  The replay only asks whether a count
// is at least that, and the incumbent's never falls, so a count may stop short once it
// cannot.
static constexpr int kCheck = 16;  // matches per lane between checks
static __device__ __forceinline__ bool can_reach(bool valid, int c, int rest, int best) {
  const int s = (int)__reduce_add_sync(0xffffffffu, (unsigned)c);
  return valid && s + rest >= best;
}

// The first matches' coordinates to shared memory, as four arrays: a lane then reads
// two matches as packed pairs, and 16 warps re-reading every match for every pass
// don't go through L2.  Returns how many are staged (a multiple of 64).
static __device__ int stage_coords(const RansacJob& J, RShared& S) {
  extern __shared__ double jac[];
  float* c = reinterpret_cast<float*>(jac);
  const int ns = min(S.n / 64 * 64, kStage);
  for (int i = threadIdx.x; i < ns; i += kRThreads) {
    const float4 p = J.xy[i];
    c[i] = p.x;
    c[kStage + i] = p.y;
    c[2 * kStage + i] = p.z;
    c[3 * kStage + i] = p.w;
  }
  __syncthreads();
  return ns;
}

// Inlier counts of the similarity hypotheses h < nh of the batch (S.ha.. /
// S.hvalid -> S.hcnt): warp w takes h = w, w + kRWarps, ..., four per pass over the
// matches.  The staged ones (ns) are taken two per lane in packed arithmetic, with the
// roundings of sim_inlier: `one` = 1 comes from the kernel's parameters, so that no
// multiplication and addition become one operation.  Ends with a block barrier.
// 1000 hypotheses on 5650 matches: 1.71 M cycles with the coordinates read from L2 and
// scalar arithmetic, 1.18 M like this.
static __device__ void sim_count_batch(const RansacJob& J, RShared& S, int nh, int best, int ns, float one) {
  extern __shared__ double jac[];
  const float* xs = reinterpret_cast<const float*>(jac);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float tsq = S.tsq_f;
  const float2 p1 = make_float2(one, one), m1 = make_float2(-one, -one);
  constexpr int kPass = 4;
  for (int h0 = warp; h0 < nh; h0 += kPass * kRWarps) {
    float2 a[kPass], b[kPass], tx[kPass], ty[kPass];
    bool v[kPass], go = false;
    int c[kPass];
#pragma unroll
    for (int u = 0; u < kPass; ++u) {
      const int h = h0 + u * kRWarps;
      v[u] = h < nh && S.hvalid[h] != 0;
      const float av = v[u] ? S.ha[h] : 0.0f, bv = v[u] ? S.hb[h] : 0.0f;
      const float xv = v[u] ? S.htx[h] : 0.0f, yv = v[u] ? S.hty[h] : 0.0f;
      a[u] = make_float2(av, av);
      b[u] = make_float2(bv, bv);
      tx[u] = make_float2(xv, xv);
      ty[u] = make_float2(yv, yv);
      c[u] = 0;
      go |= v[u];
    }
    auto reach = [&](int rest) {
      bool any = false;
#pragma unroll
      for (int u = 0; u < kPass; ++u) any |= can_reach(v[u], c[u], rest, best);
      return any;
    };
    for (int i0 = 0; go && i0 < ns; i0 += 32 * kCheck) {
      const int i1 = min(i0 + 32 * kCheck, ns);
#pragma unroll 2
      for (int i = i0 + 2 * lane; i < i1; i += 64) {
        const float2 x = *reinterpret_cast<const float2*>(xs + i), y = *reinterpret_cast<const float2*>(xs + kStage + i);
        const float2 z = *reinterpret_cast<const float2*>(xs + 2 * kStage + i), w = *reinterpret_cast<const float2*>(xs + 3 * kStage + i);
#pragma unroll
        for (int u = 0; u < kPass; ++u) {
          const float2 dx = fma2(z, m1, add2(fma2(mul2(b[u], y), m1, mul2(a[u], x)), tx[u]));
          const float2 dy = fma2(w, m1, add2(fma2(mul2(b[u], x), p1, mul2(a[u], y)), ty[u]));
          const float2 e = fma2(mul2(dx, dx), p1, mul2(dy, dy));
          c[u] += e.x <= tsq ? 1 : 0;
          c[u] += e.y <= tsq ? 1 : 0;
        }
      }
      go = reach(S.n - i1);
    }
    for (int i0 = ns; go && i0 < S.n; i0 += 32 * kCheck) {
      const int i1 = min(i0 + 32 * kCheck, S.n);
      for (int i = i0 + lane; i < i1; i += 32) {
        const float4 p = J.xy[i];
#pragma unroll
        for (int u = 0; u < kPass; ++u) {
          float e;
          c[u] += sim_inlier(p, a[u].x, b[u].x, tx[u].x, ty[u].x, tsq, e) ? 1 : 0;
        }
      }
      go = reach(S.n - i1);
    }
#pragma unroll
    for (int u = 0; u < kPass; ++u) {
      const int h = h0 + u * kRWarps;
      const int sum = (int)__reduce_add_sync(0xffffffffu, (unsigned)c[u]);
      if (lane == 0 && h < nh) S.hcnt[h] = sum;
    }
  }
  __syncthreads();
}

static __device__ double weight_total(const RansacJob& J, RShared& S) {
  double t = 0.0;
  for (int i = threadIdx.x; i < S.n && threadIdx.x < kMassThreads; i += kMassThreads) t += (double)J.weights[i];
  return block_sum_double(t, S);
}

static __device__ double sim_mass(const RansacJob& J, RShared& S, float a, float b, float tx, float ty) {
  double t = 0.0;
  for (int i = threadIdx.x; i < S.n && threadIdx.x < kMassThreads; i += kMassThreads) {
    float e;
    if (sim_inlier(J.xy[i], a, b, tx, ty, S.tsq_f, e)) t += (double)J.weights[i];
  }
  return block_sum_double(t, S);
}

// Sequential f32 error sum over inliers in input order (whole CTA; result broadcast).
static __device__ float sim_err(const RansacJob& J, RShared& S, float a, float b, float tx, float ty) {
  const float tsq = S.tsq_f;
  return ordered_sum<float>(S, S.n, [&](int i) {
    float e;
    return sim_inlier(J.xy[i], a, b, tx, ty, tsq, e) ? e : 0.0f;
  });
}

// Ordered inlier list of a similarity model into J.list; returns its length.
static __device__ int sim_collect(const RansacJob& J, RShared& S, float a, float b, float tx, float ty) {
  int base = 0;
  for (int c0 = 0; c0 < S.n; c0 += kRThreads) {
    const int i = c0 + threadIdx.x;
    bool in = false;
    if (i < S.n) {
      const float4 p = J.xy[i];
      // the collection expression of src/pipeline.rs:2161-2166 / :2172-2178
      const float dx = (a * p.x - b * p.y + tx) - p.z;
      const float dy = (b * p.x + a * p.y + ty) - p.w;
      in = dx * dx + dy * dy <= S.tsq_f;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, in);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) S.red_u[threadIdx.x >> 5] = __popc(bal);
    __syncthreads();
    int pre = 0, tot = 0;
    for (int w = 0; w < kRWarps; ++w) {
      if (w < (int)(threadIdx.x >> 5)) pre += (int)S.red_u[w];
      tot += (int)S.red_u[w];
    }
    if (in) J.list[base + pre + __popc(bal & ((1u << (threadIdx.x & 31)) - 1u))] = i;
    base += tot;
    __syncthreads();
  }
  return base;
}

// fit_procrustes_similarity over J.list[0..k) (sequential sums; threads 0..6).
static __device__ bool procrustes(const RansacJob& J, RShared& S, float* jac, int k, float* out6) {
  if (k == 0) return false;
  if (k == 1) {
    if (threadIdx.x == 0) {
      const psift_match& m = J.m[J.list[0]];
      S.fres[0] = 1.0f;
      S.fres[1] = 0.0f;
      S.fres[2] = m.displacement_x;
      S.fres[3] = m.displacement_y;
      S.fres[4] = 1.0f;
      S.fres[5] = 0.0f;
    }
    __syncthreads();
    for (int i = 0; i < 6; ++i) out6[i] = S.fres[i];
    __syncthreads();
    return true;
  }
  const float inv_n = 1.0f / (float)k;
  // The inliers' points (list order) staged in shared memory a chunk at a time;
  // the sums stay sequential in list order (threads 0..3, then 0..2), their
  // terms read at shared-memory latency.  One chunk is staged once for both.
  float4* st = reinterpret_cast<float4*>(jac);
  auto stage = [&](int c0, int cn) {
    for (int j = threadIdx.x; j < cn; j += kRThreads) st[j] = J.xy[J.list[c0 + j]];
  };
  float s = 0.0f;
  for (int c0 = 0; c0 < k; c0 += kPtChunk) {
    const int cn = min(kPtChunk, k - c0);
    stage(c0, cn);
    __syncthreads();
    if (threadIdx.x < 4) {
      const float* col = reinterpret_cast<const float*>(st) + threadIdx.x;
#pragma unroll 8
      for (int j = 0; j < cn; ++j) s += col[4 * j];
    }
    __syncthreads();
  }
  if (threadIdx.x < 4) S.fres[threadIdx.x] = s * inv_n;
  __syncthreads();
  const float mqx = S.fres[0], mqy = S.fres[1], mtx = S.fres[2], mty = S.fres[3];
  s = 0.0f;
  for (int c0 = 0; c0 < k; c0 += kPtChunk) {
    const int cn = min(kPtChunk, k - c0);
    if (k > kPtChunk) {
      stage(c0, cn);
      __syncthreads();
    }
    if (threadIdx.x < 3) {
#pragma unroll 8
      for (int j = 0; j < cn; ++j) {
        const float4 p = st[j];
        const float qx = p.x - mqx, qy = p.y - mqy, tx = p.z - mtx, ty = p.w - mty;
        const float v = threadIdx.x == 0 ? qx * qx + qy * qy : threadIdx.x == 1 ? qx * tx + qy * ty : qx * ty - qy * tx;
        s += v;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < 3) S.fres[4 + threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    const float sqq = S.fres[4], na = S.fres[5], nb = S.fres[6];
    float a = 1.0f, b = 0.0f;
    if (sqq > 1e-5f) {
      const float af = na / sqq, bf = nb / sqq;
      const float s2 = af * af + bf * bf;
      if (s2 >= 0.04f && s2 <= 25.0f) {
        a = af;
        b = bf;
      }
    }
    S.dres[0] = a;  // staging through doubles is exact for f32 values
    S.dres[1] = b;
    S.dres[2] = mtx - (a * mqx - b * mqy);
    S.dres[3] = mty - (b * mqx + a * mqy);
    S.dres[4] = sqrtf(a * a + b * b);
    S.dres[5] = atan2f(b, a) * 57.2957795130823208767981548141051703f;
  }
  __syncthreads();
  for (int i = 0; i < 6; ++i) out6[i] = (float)S.dres[i];
  __syncthreads();
  return true;
}

// The incumbent of a replay: every thread holds the same copy (the replay reads
// only shared values that stay fixed while it runs, so every thread takes the
// same decisions); err is valid when err_known.
struct SimBest {
  float a, b, tx, ty;
  int count;
  float err;
  bool err_known;
};

// Replays hypothesis h of the batch against the incumbent (count first, the
// sequential error sum on a tie): true if it replaces the incumbent.
static __device__ bool sim_consider(const RansacJob& J, RShared& S, SimBest& B, int h) {
  const int c = S.hcnt[h];
  if (c < B.count) return false;
  const float a = S.ha[h], b = S.hb[h], tx = S.htx[h], ty = S.hty[h];
  if (c > B.count) {
    B.count = c;
    B.err_known = false;
  } else {
    // the same parameters as the incumbent give the same error sum: not below it
    if (__float_as_uint(a) == __float_as_uint(B.a) && __float_as_uint(b) == __float_as_uint(B.b) &&
        __float_as_uint(tx) == __float_as_uint(B.tx) && __float_as_uint(ty) == __float_as_uint(B.ty))
      return false;
    if (!B.err_known) {
      B.err = sim_err(J, S, B.a, B.b, B.tx, B.ty);
      B.err_known = true;
    }
    const float e = sim_err(J, S, a, b, tx, ty);
    if (!(e < B.err)) return false;
    B.err = e;
  }
  B.a = a;
  B.b = b;
  B.tx = tx;
  B.ty = ty;
  return true;
}

// filter_matches_ransac_with_seed (src/pipeline.rs:2055-2191).  Writes the
// inlier list (J.list, length S.sim_count) and S.sim_model / S.has_sim.
static __device__ void similarity_ransac(const RansacJob& J, RShared& S, double* jac, uint64_t seed, float thr,
                                         float one) {
  const int n = S.n;
  if (threadIdx.x == 0) {
    S.has_sim = 0;
    S.sim_count = 0;
  }
  __syncthreads();
  if (n == 0) return;
  if (n == 1) {
    if (threadIdx.x == 0) J.list[0] = 0;
    __syncthreads();
    float m6[6];
    procrustes(J, S, reinterpret_cast<float*>(jac), 1, m6);
    if (threadIdx.x == 0) {
      for (int i = 0; i < 6; ++i) S.sim_model[i] = m6[i];
      S.has_sim = 1;
      S.sim_count = 1;
    }
    __syncthreads();
    return;
  }
  const float thresh = fmaxf(thr, 0.5f);
  if (threadIdx.x == 0) {
    S.tsq_f = thresh * thresh;
    S.key_min = 0;
  }
  __syncthreads();
  // the 32 lowest-ratio matches in stable order: keys (ratio bits, index) ascending
  const int ntop = n < 32 ? n : 32;
  for (int r = 0; r < ntop; ++r) {
    unsigned long long best = ~0ull;
    const unsigned long long floor_key = r == 0 ? 0ull : S.key_min;
    for (int i = threadIdx.x; i < n; i += kRThreads) {
      const float ratio = J.m[i].ratio;
      const uint32_t rb = __float_as_uint(ratio) ^ ((__float_as_uint(ratio) >> 31) ? 0xFFFFFFFFu : 0x80000000u);
      const unsigned long long key = ((unsigned long long)rb << 32) | (uint32_t)i;
      if ((r == 0 || key > floor_key) && key < best) best = key;
    }
    for (int o = 16; o >= 1; o >>= 1) {
      const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
      best = t < best ? t : best;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) S.dres[threadIdx.x >> 5] = __longlong_as_double((long long)best);
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long b = ~0ull;
      for (int w = 0; w < kRWarps; ++w) {
        const unsigned long long v = (unsigned long long)__double_as_longlong(S.dres[w]);
        b = v < b ? v : b;
      }
      S.key_min = b;
      S.top32[r] = (int)(b & 0xFFFFFFFFu);
    }
    __syncthreads();
  }
  // Phase A: the initial model (translation of the lowest-ratio match) and the 32
  // one-point translations, counted together, replayed in order.  The initial
  // model is translation 0: its evaluation is hypothesis 0's.
  if (threadIdx.x < ntop) {
    const psift_match& mr = J.m[S.top32[threadIdx.x]];
    S.ha[threadIdx.x] = 1.0f;
    S.hb[threadIdx.x] = 0.0f;
    S.htx[threadIdx.x] = mr.displacement_x;
    S.hty[threadIdx.x] = mr.displacement_y;
    S.hvalid[threadIdx.x] = 1;
  }
  const int ns = stage_coords(J, S);  // also: the batch is complete
  sim_count_batch(J, S, ntop, 0, ns, one);
  SimBest B{1.0f, 0.0f, S.htx[0], S.hty[0], S.hcnt[0], 0.0f, false};
  for (int r = 0; r < ntop; ++r) sim_consider(J, S, B, r);
  __syncthreads();  // the batch slots are rewritten below
  // Phase B: adaptive 2-point hypotheses
  build_cdf(J, S);
  const bool guided = J.weights != nullptr;
  const double wtot = guided ? weight_total(J, S) : 1.0;
  int max_iters = guided ? adaptive_iters_w(sim_mass(J, S, B.a, B.b, B.tx, B.ty) / wtot, 2, 64, 1000)
                         : adaptive_iters(B.count, n, 2, 64, 1000);
  int iters_done = 0;
  bool stop = false;
  for (int base = 0, nh = 0; !stop && base < 1000; base += nh) {
    if (base >= max_iters) break;
    nh = min(kBatch, max_iters - base);
    const int t = threadIdx.x;
    if (t < nh) {
      const int it = base + t;  // 0-based iteration; draws 2it, 2it+1
      int i1 = sample_at(J.cdf, n, seed, 2ull * it);
      int i2 = sample_at(J.cdf, n, seed, 2ull * it + 1ull);
      if (i2 == i1) i2 = (i1 + 1) % n;
      const float4 m1 = J.xy[i1];
      const float4 m2 = J.xy[i2];
      const float dxq = m2.x - m1.x, dyq = m2.y - m1.y;
      const float dq = dxq * dxq + dyq * dyq;
      int valid = 0;
      float a = 0.f, b = 0.f, tx = 0.f, ty = 0.f;
      if (!(dq < 16.0f)) {
        const float dxt = m2.z - m1.z, dyt = m2.w - m1.w;
        a = (dxq * dxt + dyq * dyt) / dq;
        b = (dxq * dyt - dyq * dxt) / dq;
        const float s2 = a * a + b * b;
        if (s2 >= 0.04f && s2 <= 25.0f) {
          tx = m1.z - (a * m1.x - b * m1.y);
          ty = m1.w - (b * m1.x + a * m1.y);
          valid = 1;
        }
      }
      S.ha[t] = a;
      S.hb[t] = b;
      S.htx[t] = tx;
      S.hty[t] = ty;
      S.hvalid[t] = valid;
    }
    __syncthreads();
    sim_count_batch(J, S, nh, B.count, ns, one);
    // replay in order
    for (int h = 0; h < nh; ++h) {
      const int it = base + h;
      if (it >= max_iters) {
        stop = true;
        break;
      }
      iters_done = it + 1;
      if (!S.hvalid[h]) continue;
      if (sim_consider(J, S, B, h))
        max_iters = guided ? adaptive_iters_w(sim_mass(J, S, B.a, B.b, B.tx, B.ty) / wtot, 2, 64, 1000)
                           : adaptive_iters(B.count, n, 2, 64, 1000);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && J.iters) J.iters[0] = iters_done;
  // consensus, Procrustes refit, re-collection
  int k = sim_collect(J, S, B.a, B.b, B.tx, B.ty);
  float refined[6];
  const bool has_ref = procrustes(J, S, reinterpret_cast<float*>(jac), k, refined);
  if (has_ref) {
    // count of the refined model's consensus (same expression as the collection)
    int c = 0;
    for (int i = threadIdx.x; i < n; i += kRThreads) {
      const float4 p = J.xy[i];
      const float dx = (refined[0] * p.x - refined[1] * p.y + refined[2]) - p.z;
      const float dy = (refined[1] * p.x + refined[0] * p.y + refined[3]) - p.w;
      c += dx * dx + dy * dy <= S.tsq_f ? 1 : 0;
    }
    c = block_sum_int(c, S);
    if (c >= k) k = sim_collect(J, S, refined[0], refined[1], refined[2], refined[3]);
  }
  float fin[6];
  const bool has_fin = procrustes(J, S, reinterpret_cast<float*>(jac), k, fin);
  if (threadIdx.x == 0) {
    S.sim_count = k;
    if (has_fin) {
      for (int i = 0; i < 6; ++i) S.sim_model[i] = fin[i];
      S.has_sim = 1;
    } else if (has_ref) {
      for (int i = 0; i < 6; ++i) S.sim_model[i] = refined[i];
      S.has_sim = 1;
    }
  }
  __syncthreads();
}

// ------------------------------------------------------------- homography
// evaluate_homography_hypothesis_f64's per-match test (src/pipeline.rs:2557-2573).
static __device__ __forceinline__ bool h_inlier(const float4 p, const double* H, double tsq, double& e) {
  const double qx = p.x, qy = p.y;
  const double w = H[6] * qx + H[7] * qy + H[8];
  if (fabs(w) < 1e-9) return false;
  const double iw = 1.0 / w;
  const double px = (H[0] * qx + H[1] * qy + H[2]) * iw;
  const double py = (H[3] * qx + H[4] * qy + H[5]) * iw;
  const double dx = px - (double)p.z, dy = py - (double)p.w;
  e = dx * dx + dy * dy;
  return e <= tsq;
}

// The f32 test of h_count_batch.  With M = max(Bx, By) + T Bw, where Bx = |h0| Qx + |h1|
// Qy + |h2| bounds the terms of the numerator X over the set's matches (By, Bw alike) and
// T the target coordinates, the f32 values of w and of U = X - tx w, V = Y - ty w are off
// by at most 3.1 2^-24 Bw and 4.2 2^-24 M (H rounded, two fused steps each, one more for
// U); the reference's f64 value of e is off from (U^2 + V^2) / w^2 by far less.  So with
// G = thr (3.1 2^-24 Bw + 2e-9) + 6 2^-24 M (the 2e-9 keeps |w| >= 1e-9 certain) e <= thr^2
// is certain for |(U, V)| <= thr |w| - G and excluded for |(U, V)| >= thr |w| + G, and
// 2 thr |w| G <= k (thr w)^2 + G^2 / k, for any k, turns both into
//   U^2 + V^2 <= w^2 lo.x + lo.y    and    U^2 + V^2 >= w^2 hi.x + hi.y.
// In between, for values too large and for NaN the f64 test decides: there lo is (-1, -1),
// below every sum of squares (also of w = U = V = 0, which f32 rounding does give), and hi
// is NaN.
static __device__ float4 h_band(const RShared& S, const double* H) {
  const double Qx = __uint_as_float(S.coord_max[0]), Qy = __uint_as_float(S.coord_max[1]), T = __uint_as_float(S.coord_max[2]);
  const double Bx = fabs(H[0]) * Qx + fabs(H[1]) * Qy + fabs(H[2]);
  const double By = fabs(H[3]) * Qx + fabs(H[4]) * Qy + fabs(H[5]);
  const double Bw = fabs(H[6]) * Qx + fabs(H[7]) * Qy + fabs(H[8]);
  const double M = Bx + By + T * Bw, thr2 = S.tsq_d;  // Bx + By >= max(Bx, By), and holds a NaN
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  if (!(M < 1e15) || !(Bw < 1e15) || !(Qx < 1e15) || !(Qy < 1e15) || !(T < 1e15) || !(thr2 < 1e7))
    return make_float4(-1.0f, -1.0f, (float)nan, 0.0f);
  const double thr = sqrt(thr2);
  const double G = 1.01 * (thr * (3.1 * 0x1p-24 * Bw + 2e-9) + 6.0 * 0x1p-24 * M);
  const double k = fmin(fmax(G / thr, 0x1p-20), 0.5), s = 0x1p-20;  // s: the f32 roundings of the test itself
  return make_float4((float)(thr2 * (1.0 - k) * (1.0 - s)), (float)(-G * G * (1.0 / k - 1.0) * (1.0 + s)),
                     (float)(thr2 * (1.0 + k) * (1.0 + s)), (float)(G * G * (1.0 / k + 1.0) * (1.0 + s)));
}

// Inlier counts of the homographies h < nh of the batch (S.H / S.hband / S.hvalid ->
// S.hcnt): warp w takes h = w, w + kRWarps, ..., two per pass over the matches.  The
// staged matches (ns) are tested in packed f32, two per lane, the undecided ones in f64
// (see h_band).  Ends with a barrier.
// 88 hypotheses on 5650 matches: 606 k cycles in f64 (a division each, coordinates from
// L2), 161 k like this.
static __device__ void h_count_batch(const RansacJob& J, RShared& S, int nh, int best, int ns) {
  extern __shared__ double jac[];
  const float* xs = reinterpret_cast<const float*>(jac);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double tsq = S.tsq_d;
  constexpr int kPass = 2;
  for (int h0 = warp; h0 < nh; h0 += kPass * kRWarps) {
    bool v[kPass], go = false;
    int c[kPass];
    float2 H[kPass][9];
    float4 band[kPass];
#pragma unroll
    for (int u = 0; u < kPass; ++u) {
      const int h = h0 + u * kRWarps;
      v[u] = h < nh && S.hvalid[h] != 0;
      c[u] = 0;
      go |= v[u];
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const float f = v[u] ? (float)S.H[h][i] : 0.0f;
        H[u][i] = i < 6 ? make_float2(-f, -f) : make_float2(f, f);
      }
      band[u] = v[u] ? S.hband[h] : make_float4(-1.0f, -1.0f, 0.0f, 0.0f);  // an absent one: never in, always decided
    }
    auto exact = [&](int u, float4 p) {
      double e;
      return h_inlier(p, S.H[h0 + u * kRWarps], tsq, e);
    };
    auto reach = [&](int rest) {
      bool any = false;
#pragma unroll
      for (int u = 0; u < kPass; ++u) any |= can_reach(v[u], c[u], rest, best);
      return any;
    };
    for (int i0 = 0; go && i0 < ns; i0 += 32 * kCheck) {
      const int i1 = min(i0 + 32 * kCheck, ns);
      for (int i = i0 + 2 * lane; i < i1; i += 64) {
        const float2 x = *reinterpret_cast<const float2*>(xs + i), y = *reinterpret_cast<const float2*>(xs + kStage + i);
        const float2 z = *reinterpret_cast<const float2*>(xs + 2 * kStage + i), t = *reinterpret_cast<const float2*>(xs + 3 * kStage + i);
        unsigned open = 0;  // bit 2 u + k: match k of the pair is undecided for u
#pragma unroll
        for (int u = 0; u < kPass; ++u) {
          const float2 w = fma2(H[u][6], x, fma2(H[u][7], y, H[u][8]));
          const float2 U = fma2(z, w, fma2(H[u][0], x, fma2(H[u][1], y, H[u][2])));  // minus the numerators
          const float2 V = fma2(t, w, fma2(H[u][3], x, fma2(H[u][4], y, H[u][5])));
          const float2 e = fma2(U, U, mul2(V, V)), w2 = mul2(w, w);
          const float2 lo = fma2(w2, make_float2(band[u].x, band[u].x), make_float2(band[u].y, band[u].y));
          const float2 hi = fma2(w2, make_float2(band[u].z, band[u].z), make_float2(band[u].w, band[u].w));
          const bool in0 = e.x <= lo.x, in1 = e.y <= lo.y;
          c[u] += in0 ? 1 : 0;
          c[u] += in1 ? 1 : 0;
          if (!in0 && !(e.x >= hi.x)) open |= 1u << (2 * u);
          if (!in1 && !(e.y >= hi.y)) open |= 2u << (2 * u);
        }
        while (open) {
          const int k = __ffs(open) - 1;
          open &= open - 1;
          const float4 p = k & 1 ? make_float4(x.y, y.y, z.y, t.y) : make_float4(x.x, y.x, z.x, t.x);
          const int in = exact(k >> 1, p) ? 1 : 0;
#pragma unroll
          for (int u = 0; u < kPass; ++u) c[u] += k >> 1 == u ? in : 0;
        }
      }
      go = reach(S.n - i1);
    }
    for (int i0 = ns; go && i0 < S.n; i0 += 32 * kCheck) {
      const int i1 = min(i0 + 32 * kCheck, S.n);
      for (int i = i0 + lane; i < i1; i += 32) {
        const float4 p = J.xy[i];
#pragma unroll
        for (int u = 0; u < kPass; ++u) c[u] += v[u] && exact(u, p) ? 1 : 0;
      }
      go = reach(S.n - i1);
    }
#pragma unroll
    for (int u = 0; u < kPass; ++u) {
      const int h = h0 + u * kRWarps;
      const int sum = (int)__reduce_add_sync(0xffffffffu, (unsigned)c[u]);
      if (lane == 0 && h < nh) S.hcnt[h] = sum;
    }
  }
  __syncthreads();
}

static __device__ int h_count(const RansacJob& J, RShared& S, const double* Hs) {
  double H[9];
  for (int i = 0; i < 9; ++i) H[i] = Hs[i];
  int c = 0;
  for (int i = threadIdx.x; i < S.n; i += kRThreads) {
    double e;
    c += h_inlier(J.xy[i], H, S.tsq_d, e) ? 1 : 0;
  }
  return block_sum_int(c, S);
}

static __device__ double h_mass(const RansacJob& J, RShared& S, const double* Hs) {
  double H[9];
  for (int i = 0; i < 9; ++i) H[i] = Hs[i];
  double t = 0.0;
  for (int i = threadIdx.x; i < S.n && threadIdx.x < kMassThreads; i += kMassThreads) {
    double e;
    if (h_inlier(J.xy[i], H, S.tsq_d, e)) t += (double)J.weights[i];
  }
  return block_sum_double(t, S);
}

// Sequential f64 error sum over the inliers in input order (whole CTA).
static __device__ double h_err(const RansacJob& J, RShared& S, const double* H) {
  const double tsq = S.tsq_d;
  double Hl[9];
  for (int i = 0; i < 9; ++i) Hl[i] = H[i];
  return ordered_sum<double>(S, S.n, [&](int i) {
    double e;
    return h_inlier(J.xy[i], Hl, tsq, e) ? e : 0.0;
  });
}

static __device__ int h_collect(const RansacJob& J, RShared& S, const double* Hs) {
  double H[9];
  for (int i = 0; i < 9; ++i) H[i] = Hs[i];
  int base = 0;
  for (int c0 = 0; c0 < S.n; c0 += kRThreads) {
    const int i = c0 + threadIdx.x;
    bool in = false;
    if (i < S.n) {
      double e;
      in = h_inlier(J.xy[i], H, S.tsq_d, e);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, in);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) S.red_u[threadIdx.x >> 5] = __popc(bal);
    __syncthreads();
    int pre = 0, tot = 0;
    for (int w = 0; w < kRWarps; ++w) {
      if (w < (int)(threadIdx.x >> 5)) pre += (int)S.red_u[w];
      tot += (int)S.red_u[w];
    }
    if (in) J.list[base + pre + __popc(bal & ((1u << (threadIdx.x & 31)) - 1u))] = i;
    base += tot;
    __syncthreads();
  }
  return base;
}

// (a, b), a <= b, of upper-triangle entry e (row-major, 45 entries).
static __device__ __forceinline__ void upper_entry(int e, int& a, int& b) {
  a = 0;
  while (e >= 9 - a) {
    e -= 9 - a;
    ++a;
  }
  b = a + e;
}

// smallest_eigenvector_9x9 (src/pipeline.rs:2276-2353), the cyclic Jacobi shared
// by a quad of lanes (ql = 0..3, converged, qmask their lane mask).  A (81
// doubles, shared memory, the upper triangle complete) is diagonalised in place; V
// (81 doubles) receives the eigenvectors, a row each.  Returns the column of the
// smallest diagonal entry (the first on ties), or -1 if that eigenvector is not
// finite.  A's diagonal and V are complete and visible to the quad on return.
// V must be A + 81 with A on a 16-byte boundary.
//
// A sweep's 36 rotations are a serial chain in the reference, and the chain of one
// rotation's parameters (division, two square roots, two reciprocals in f64) is what
// a fit takes its time for.  Two rotations without a common index do not read each
// other's pivots, so rotation (p, r) runs at step p + r, up to four per step, one per
// lane: 15 steps instead of 36.  Rounding does not commute, so every entry still sees
// its updates in the reference's order:
//   - a rotation (p, q) reaches column r > q when (p, r) is about to run (then every
//     earlier rotation of index r has), so the lane of p first applies (p, p+1) ..
//     (p, r-1) to column r, takes its pivot, and applies (p, r) to columns p+1 .. r-1;
//   - what is left of a sweep touches rows whose own rotations are over (row i of A
//     right of the diagonal, by rotations of indices above i) and the rows of V; these
//     rows are independent of one another and are rotated once the sweep's parameters
//     are known.
// Every value and decision is the sequential solver's, bit by bit.  Bound by the latency
// of a step (parameters 550 cycles).  Against the rotations one after the other, their
// row updates shared by the lanes: 128 fits of a CTA 486 -> 293 k cycles, one fit (a
// refit, 6 sweeps) 205 -> 141 k.
// Volatile, or the compiler loads all of a sweep's parameters first, and spills.
static __device__ __forceinline__ double2 rot_params(const double2* cs) {
  double2 r;
  asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];" : "=d"(r.x), "=d"(r.y) : "r"((uint32_t)__cvta_generic_to_shared(cs)) : "memory");
  return r;
}
static constexpr int kSkipHi = 0x40000000;  // c = 2: the rotation was skipped (a cosine is at most 1)
static __device__ __noinline__ int quad_cyclic_jacobi(double* A, double* V, int ql, unsigned qmask) {
  double2* CS = reinterpret_cast<double2*>(V + 1);  // (c, s) of the sweep's rotations, row-major
  double va[9], vb[9];  // rows ql and ql + 4 of V; row 8 lives below A's diagonal
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    va[c] = c == ql ? 1.0 : 0.0;
    vb[c] = c == ql + 4 ? 1.0 : 0.0;
  }
  if (ql == 0) {
#pragma unroll
    for (int c = 0; c < 8; ++c) A[72 + c] = 0.0;
    A[63] = 1.0;
  }
  for (int sweep = 0; sweep < 20; ++sweep) {
    double mx = 0.0;
#pragma unroll
    for (int s = 0; s < 9; ++s) {
      const double v = fabs(A[kStrictUpper[ql + 4 * s]]);
      if (v > mx) mx = v;
    }
    mx = fmax(mx, __shfl_xor_sync(qmask, mx, 1));
    mx = fmax(mx, __shfl_xor_sync(qmask, mx, 2));
    if (mx < 1e-13) break;
    // the rotations' parameters and the entries they depend on
#pragma unroll 1
    for (int step = 1; step <= 15; ++step) {
      int p = ql, r = step - ql;
      if (r > 8) {
        p += 4;
        r -= 4;
      }
      const int longest = step <= 8 ? step - 1 : 15 - step;  // of the step's columns, above the pivots
      if (p < r && r <= 8) {
        const int cnt = r - p - 1;
        double* const row = A + p * 9 + p + 1;    // A[p][p + 1 + k] at [k]
        double* const col = A + (p + 1) * 9 + r;  // A[p + 1 + k][r] at [9 k]
        double2* const cs = CS + (p * (17 - p) >> 1);
        double x = A[p * 9 + r];
        double y[7];
        // all seven slots at once or the first three, by the step's longest column; what
        // lies beyond cnt is loaded (it is in the quad's memory) and not used
        auto column = [&](auto first, auto last) {
          constexpr int k0 = decltype(first)::value, k1 = decltype(last)::value;
          double2 rot[k1];
#pragma unroll
          for (int k = k0; k < k1; ++k) {
            rot[k] = cs[min(k, cnt)];
            y[k] = col[9 * k];
          }
#pragma unroll
          for (int k = k0; k < k1; ++k) {
            const bool on = k < cnt && __double2hiint(rot[k].x) != kSkipHi;
            const double nx = rot[k].x * x - rot[k].y * y[k], ny = rot[k].y * x + rot[k].x * y[k];
            x = on ? nx : x;
            y[k] = on ? ny : y[k];
          }
        };
        if (longest > 0) column(Int<0>(), Int<3>());
        if (longest > 3) column(Int<3>(), Int<7>());
        const double apq = x;
        const bool rotate = !(fabs(apq) < 1e-15);
        double c = 2.0, s = 0.0;
        if (rotate) {
          const double app = A[p * 10], aqq = A[r * 10];
          const double tau = (aqq - app) / (2.0 * apq);
          // __drcp_rn(x) is 1.0 / x: both are IEEE round-to-nearest, the reciprocal is the cheaper sequence
          const double m = __drcp_rn(fabs(tau) + sqrt(1.0 + tau * tau)), t = tau >= 0.0 ? m : -m;
          c = __drcp_rn(sqrt(1.0 + t * t));
          s = t * c;
          A[p * 10] = app - t * apq;
          A[r * 10] = aqq + t * apq;
        }
        cs[cnt] = make_double2(c, s);
        row[cnt] = rotate ? 0.0 : apq;
        auto rest = [&](auto first, auto last) {
          constexpr int k0 = decltype(first)::value, k1 = decltype(last)::value;
          double a[k1];
#pragma unroll
          for (int k = k0; k < k1; ++k) a[k] = row[k];
#pragma unroll
          for (int k = k0; k < k1; ++k) {
            const double na = c * a[k] - s * y[k], ny = s * a[k] + c * y[k];
            if (k < cnt && rotate) row[k] = na;
            if (k < cnt) col[9 * k] = rotate ? ny : y[k];
          }
        };
        if (longest > 0) rest(Int<0>(), Int<3>());
        if (longest > 3) rest(Int<3>(), Int<7>());
      }
      __syncwarp(qmask);
    }
    // V's rows ql and ql + 4
#pragma unroll
    for (int p = 0; p < 8; ++p) {
#pragma unroll
      for (int q = p + 1; q < 9; ++q) {
        const double2 rot = rot_params(CS + p * (17 - p) / 2 + q - p - 1);
        if (__double2hiint(rot.x) != kSkipHi) {
          const double ap = va[p], aq = va[q], bp = vb[p], bq = vb[q];
          va[p] = rot.x * ap - rot.y * aq;
          va[q] = rot.y * ap + rot.x * aq;
          vb[p] = rot.x * bp - rot.y * bq;
          vb[q] = rot.y * bp + rot.x * bq;
        }
      }
    }
    {  // row 8 of V (lane 0), rows 0, 1, 2 of A right of the diagonal
      double* const base = ql == 0 ? A + 72 : A + (ql - 1) * 9;
      double* const last = ql == 0 ? A + 63 : base + 8;
      double x[9];
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c] = base[c];
      x[8] = *last;
#pragma unroll
      for (int p = 0; p < 8; ++p) {
#pragma unroll
        for (int q = p + 1; q < 9; ++q) {
          const double2 rot = rot_params(CS + p * (17 - p) / 2 + q - p - 1);
          if (p >= ql && __double2hiint(rot.x) != kSkipHi) {
            const double xp = x[p], xq = x[q];
            x[p] = rot.x * xp - rot.y * xq;
            x[q] = rot.y * xp + rot.x * xq;
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c >= ql) base[c] = x[c];
      *last = x[8];
    }
    {  // rows 3 .. 6 of A
      double* const base = A + (3 + ql) * 9;
      double x[9];
#pragma unroll
      for (int c = 4; c < 9; ++c) x[c] = base[c];
#pragma unroll
      for (int p = 4; p < 8; ++p)
#pragma unroll
        for (int q = p + 1; q < 9; ++q) {
          const double2 rot = rot_params(CS + p * (17 - p) / 2 + q - p - 1);
          if (p > 3 + ql && __double2hiint(rot.x) != kSkipHi) {
            const double xp = x[p], xq = x[q];
            x[p] = rot.x * xp - rot.y * xq;
            x[q] = rot.y * xp + rot.x * xq;
          }
        }
#pragma unroll
      for (int c = 4; c < 9; ++c)
        if (c > 3 + ql) base[c] = x[c];
    }
    __syncwarp(qmask);
  }
  __syncwarp(qmask);  // V takes the place of the parameters
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    V[ql * 9 + c] = va[c];
    V[(ql + 4) * 9 + c] = vb[c];
  }
  if (ql == 0) {
#pragma unroll
    for (int c = 0; c < 8; ++c) V[72 + c] = A[72 + c];
    V[80] = A[63];
  }
  __syncwarp(qmask);
  int mi = 0;
  double me = A[0];
  for (int i = 1; i < 9; ++i)
    if (A[i * 10] < me) {
      me = A[i * 10];
      mi = i;
    }
  for (int r = 0; r < 9; ++r)
    if (!isfinite(V[r * 9 + mi])) return -1;
  return mi;
}

// De-normalisation of the null vector hv (src/pipeline.rs:2500-2528).
static __device__ void denormalise(const double* hv, double sq, double st, double cxq, double cyq, double cxt, double cyt,
                            double* H) {
  const double hn[3][3] = {{hv[0], hv[1], hv[2]}, {hv[3], hv[4], hv[5]}, {hv[6], hv[7], hv[8]}};
  const double tq[3][3] = {{sq, 0.0, -sq * cxq}, {0.0, sq, -sq * cyq}, {0.0, 0.0, 1.0}};
  const double ist = 1.0 / st;
  const double tti[3][3] = {{ist, 0.0, cxt}, {0.0, ist, cyt}, {0.0, 0.0, 1.0}};
  double tmp[3][3];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) tmp[r][c] = hn[r][0] * tq[0][c] + hn[r][1] * tq[1][c] + hn[r][2] * tq[2][c];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) H[3 * r + c] = tti[r][0] * tmp[0][c] + tti[r][1] * tmp[1][c] + tti[r][2] * tmp[2][c];
  if (fabs(H[8]) > 1e-12) {
    const double inv = 1.0 / H[8];
    for (int i = 0; i < 9; ++i) H[i] *= inv;
  }
}

// The two A^T A rows of one normalised correspondence (x, y) -> (x', y')
// (src/pipeline.rs:2466-2479) take 10 distinct values, kept as one row:
//   [-x, -y, -1, 0, x x', y x', x', x y', y y', y']
// Row 1's entry a is row[(kSlot1 >> 4a) & 15], row 2's row[(kSlot2 >> 4a) & 15];
// every value is the reference's (negation is exact, the products are the same
// rounded products), so a sum of r1[a] r1[b] + r2[a] r2[b] terms is unchanged.
static constexpr int kRowVals = 10;
static constexpr unsigned long long kSlot1 = 0x654333210ull;  // -x -y -1 0 0 0 xx' yx' x'
static constexpr unsigned long long kSlot2 = 0x987210333ull;  // 0 0 0 -x -y -1 xy' yy' y'

static __device__ __forceinline__ void dlt_row_values(double x, double y, double xp, double yp, double* r) {
  r[0] = -x, r[1] = -y, r[2] = -1.0, r[3] = 0.0, r[4] = x * xp, r[5] = y * xp, r[6] = xp, r[7] = x * yp,
  r[8] = y * yp, r[9] = yp;
}

// fit_homography_dlt_f64 on 4 correspondences by a quad of lanes: every lane
// normalises; lane i writes point i's row values (in V, free until the Jacobi
// starts); the 45 A^T A entries are split over the lanes, each summed over the 4
// points in order; the quad runs the Jacobi.  The result (H, return value) is
// the leader's (ql == 0).
static __device__ bool quad_fit4(const float4* __restrict__ xy, const int* idx, double* A, double* V, int ql,
                          unsigned qmask, double* H) {
  double qx[4], qy[4], tx[4], ty[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 p = xy[idx[i]];
    qx[i] = p.x, qy[i] = p.y, tx[i] = p.z, ty[i] = p.w;
  }
  const double inv_n = 1.0 / 4.0;
  double cxq = 0, cyq = 0, cxt = 0, cyt = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (!isfinite(qx[i]) || !isfinite(qy[i]) || !isfinite(tx[i]) || !isfinite(ty[i])) return false;
    cxq += qx[i];
    cyq += qy[i];
    cxt += tx[i];
    cyt += ty[i];
  }
  cxq *= inv_n;
  cyq *= inv_n;
  cxt *= inv_n;
  cyt *= inv_n;
  double mdq = 0, mdt = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double dxq = qx[i] - cxq, dyq = qy[i] - cyq;
    const double dxt = tx[i] - cxt, dyt = ty[i] - cyt;
    mdq += sqrt(dxq * dxq + dyq * dyq);
    mdt += sqrt(dxt * dxt + dyt * dyt);
  }
  mdq *= inv_n;
  mdt *= inv_n;
  if (!isfinite(mdq) || !isfinite(mdt) || mdq < 1e-6 || mdt < 1e-6) return false;
  const double sq = 1.41421356237309504880 / mdq, st = 1.41421356237309504880 / mdt;
  {
    const float4 p = xy[idx[ql]];
    dlt_row_values(((double)p.x - cxq) * sq, ((double)p.y - cyq) * sq, ((double)p.z - cxt) * st,
                   ((double)p.w - cyt) * st, V + ql * kRowVals);
  }
  __syncwarp(qmask);
  for (int e = ql; e < 45; e += 4) {
    int a, b;
    upper_entry(e, a, b);
    const int s1a = (int)(kSlot1 >> (4 * a)) & 15, s1b = (int)(kSlot1 >> (4 * b)) & 15;
    const int s2a = (int)(kSlot2 >> (4 * a)) & 15, s2b = (int)(kSlot2 >> (4 * b)) & 15;
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double* r = V + i * kRowVals;
      s += r[s1a] * r[s1b] + r[s2a] * r[s2b];
    }
    A[a * 9 + b] = s;
    A[b * 9 + a] = s;
  }
  __syncwarp(qmask);  // rows read, A complete
  const int mi = quad_cyclic_jacobi(A, V, ql, qmask);
  if (mi < 0 || ql != 0) return mi >= 0;
  double hv[9];
#pragma unroll
  for (int r = 0; r < 9; ++r) hv[r] = V[r * 9 + mi];
  denormalise(hv, sq, st, cxq, cyq, cxt, cyt, H);
  return true;
}

// fit_homography_dlt_f64 over J.list[0..k) (k >= 4), whole CTA; jac holds one
// free A / V pair.  Result in S.dres[0 .. 8]; false if the fit fails.
static __device__ bool fit_dlt_list(const RansacJob& J, RShared& S, double* jac, int k) {
  const double inv_n = 1.0 / (double)k;
  // The inliers' points (list order) staged in shared memory a chunk at a time;
  // every sum below stays sequential in list order, its terms read at
  // shared-memory latency (the centroids by threads 0..3, the mean distances'
  // terms computed by the CTA and added by threads 0, 1).
  constexpr int kChunk = (int)(kJacSmem / (sizeof(float4) + 2 * sizeof(double)));
  float4* st = reinterpret_cast<float4*>(jac);
  double* dq = reinterpret_cast<double*>(st + kChunk);
  double* dt = dq + kChunk;
  auto stage = [&](int c0, int cn) {
    for (int j = threadIdx.x; j < cn; j += kRThreads) st[j] = J.xy[J.list[c0 + j]];
  };
  if (threadIdx.x == 0) S.flag = 1;
  double s = 0.0;
  for (int c0 = 0; c0 < k; c0 += kChunk) {
    const int cn = min(kChunk, k - c0);
    stage(c0, cn);
    __syncthreads();
    for (int j = threadIdx.x; j < cn; j += kRThreads) {
      const float4 p = st[j];
      if (!isfinite(p.x) || !isfinite(p.y) || !isfinite(p.z) || !isfinite(p.w)) S.flag = 0;
    }
    if (threadIdx.x < 4) {
      const float* col = reinterpret_cast<const float*>(st) + threadIdx.x;
#pragma unroll 8
      for (int j = 0; j < cn; ++j) s += (double)col[4 * j];
    }
    __syncthreads();
  }
  if (threadIdx.x < 4) S.dres[threadIdx.x] = s * inv_n;
  __syncthreads();
  const bool finite = S.flag != 0;
  const double cxq = S.dres[0], cyq = S.dres[1], cxt = S.dres[2], cyt = S.dres[3];
  __syncthreads();
  if (!finite) return false;
  s = 0.0;
  for (int c0 = 0; c0 < k; c0 += kChunk) {
    const int cn = min(kChunk, k - c0);
    if (k > kChunk) {
      stage(c0, cn);
      __syncthreads();
    }
    for (int j = threadIdx.x; j < cn; j += kRThreads) {
      const float4 p = st[j];
      const double ax = (double)p.x - cxq, ay = (double)p.y - cyq;
      const double bx = (double)p.z - cxt, by = (double)p.w - cyt;
      dq[j] = sqrt(ax * ax + ay * ay);
      dt[j] = sqrt(bx * bx + by * by);
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      const double* d = threadIdx.x == 0 ? dq : dt;
      int j = 0;
      for (; j + 16 <= cn; j += 16) {
        double e[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) e[u] = d[j + u];
#pragma unroll
        for (int u = 0; u < 16; ++u) s += e[u];
      }
      for (; j < cn; ++j) s += d[j];
    }
    __syncthreads();
  }
  if (threadIdx.x < 2) S.dres[4 + threadIdx.x] = s * inv_n;
  __syncthreads();
  const double mdq = S.dres[4], mdt = S.dres[5];
  __syncthreads();
  if (!isfinite(mdq) || !isfinite(mdt) || mdq < 1e-6 || mdt < 1e-6) return false;
  const double sq = 1.41421356237309504880 / mdq, st_ = 1.41421356237309504880 / mdt;
  // upper triangle of A^T A: entry (a, b), a <= b, one thread each, sequential
  // over the list; the points' normalised row values staged through jac a chunk
  // at a time
  {
    int a = 0, b = 0;
    if (threadIdx.x < 45) upper_entry(threadIdx.x, a, b);
    const int s1a = (int)(kSlot1 >> (4 * a)) & 15, s1b = (int)(kSlot1 >> (4 * b)) & 15;
    const int s2a = (int)(kSlot2 >> (4 * a)) & 15, s2b = (int)(kSlot2 >> (4 * b)) & 15;
    double sum = 0.0;
    for (int c0 = 0; c0 < k; c0 += kRowChunk) {
      const int cn = min(kRowChunk, k - c0);
      for (int j = threadIdx.x; j < cn; j += kRThreads) {
        const float4 p = J.xy[J.list[c0 + j]];
        dlt_row_values(((double)p.x - cxq) * sq, ((double)p.y - cyq) * sq, ((double)p.z - cxt) * st_,
                       ((double)p.w - cyt) * st_, jac + j * kRowVals);
      }
      __syncthreads();
      if (threadIdx.x < 45) {
#pragma unroll 8
        for (int j = 0; j < cn; ++j) {
          const double* r = jac + j * kRowVals;
          sum += r[s1a] * r[s1b] + r[s2a] * r[s2b];
        }
      }
      __syncthreads();
    }
    if (threadIdx.x < 45) {
      S.ata[a][b] = sum;
      S.ata[b][a] = sum;
    }
  }
  __syncthreads();
  if (threadIdx.x < 4) {  // the eigen-decomposition by the first quad
    const int ql = threadIdx.x;
    double* A = jac;
    double* V = jac + 81;
    for (int e = ql; e < 81; e += 4) A[e] = S.ata[e / 9][e % 9];
    __syncwarp(0xFu);
    const int mi = quad_cyclic_jacobi(A, V, ql, 0xFu);
    if (ql == 0) {
      S.flag = mi >= 0 ? 1 : 0;
      if (mi >= 0) {
        double hv[9], Hl[9];
        for (int r = 0; r < 9; ++r) hv[r] = V[r * 9 + mi];
        denormalise(hv, sq, st_, cxq, cyq, cxt, cyt, Hl);
        for (int i = 0; i < 9; ++i) S.dres[i] = Hl[i];
      }
    }
  }
  __syncthreads();
  const bool ok = S.flag != 0;
  __syncthreads();
  return ok;
}

// has_degenerate_triangle (src/pipeline.rs:2357-2388)
static __device__ bool degenerate4(const double (&p)[4][2]) {
  const int T[4][3] = {{0, 1, 2}, {0, 1, 3}, {0, 2, 3}, {1, 2, 3}};
  for (int t = 0; t < 4; ++t) {
    const double xi = p[T[t][0]][0], yi = p[T[t][0]][1], xj = p[T[t][1]][0], yj = p[T[t][1]][1];
    const double xk = p[T[t][2]][0], yk = p[T[t][2]][1];
    if (!isfinite(xi) || !isfinite(yi) || !isfinite(xj) || !isfinite(yj) || !isfinite(xk) || !isfinite(yk)) return true;
    const double dx1 = xj - xi, dy1 = yj - yi, dx2 = xk - xi, dy2 = yk - yi, dx3 = xk - xj, dy3 = yk - yj;
    const double cross = fabs(dx1 * dy2 - dy1 * dx2);
    const double me = fmax(fmax(dx1 * dx1 + dy1 * dy1, dx2 * dx2 + dy2 * dy2), dx3 * dx3 + dy3 * dy3);
    if (cross < 4.0 || cross < 1e-3 * me) return true;
  }
  return false;
}

// local_optimize_homography (src/pipeline.rs:2605-2631); updates H (shared memory) /
// count / err in place (err valid when err_known; computed only for a tie).
static __device__ void local_optimize(const RansacJob& J, RShared& S, double* jac, double* H, int& count, double& err,
                               bool& err_known) {
  for (int round = 0; round < 2; ++round) {
    const int k = h_collect(J, S, H);
    if (k < 4) break;
    if (!fit_dlt_list(J, S, jac, k)) break;
    const int rc = h_count(J, S, S.dres);
    if (rc < count) break;
    if (rc == count) {
      if (!err_known) {
        err = h_err(J, S, H);
        err_known = true;
      }
      const double re = h_err(J, S, S.dres);
      if (!(re < err)) break;
      err = re;
    } else {
      err_known = false;
    }
    if (threadIdx.x < 9) H[threadIdx.x] = S.dres[threadIdx.x];
    __syncthreads();
    count = rc;
  }
}

static __device__ void run(const RansacJob& J, RShared& S, float one) {
  extern __shared__ double jac[];
  const int n = J.n;
  if (threadIdx.x == 0) S.n = n;
  if (threadIdx.x < 3) S.coord_max[threadIdx.x] = 0;
  __syncthreads();
  unsigned mx[3] = {0, 0, 0};  // as bits: a NaN exceeds every number
  for (int i = threadIdx.x; i < n; i += kRThreads) {
    J.mask[i] = 0;
    const psift_match& m = J.m[i];
    const float4 p = make_float4(m.query_x, m.query_y, m.target_x, m.target_y);
    J.xy[i] = p;
    mx[0] = max(mx[0], __float_as_uint(fabsf(p.x)));
    mx[1] = max(mx[1], __float_as_uint(fabsf(p.y)));
    mx[2] = max(mx[2], max(__float_as_uint(fabsf(p.z)), __float_as_uint(fabsf(p.w))));
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const unsigned w = __reduce_max_sync(0xffffffffu, mx[k]);
    if ((threadIdx.x & 31) == 0) atomicMax(&S.coord_max[k], w);
  }
  __syncthreads();
  similarity_ransac(J, S, jac, J.sim_seed, J.thr, one);
  if (!J.homography) {
    const int k = S.sim_count;
    for (int j = threadIdx.x; j < k; j += kRThreads) J.mask[J.list[j]] = 1;
    if (threadIdx.x == 0) {
      *J.count = k;
      *J.has_model = S.has_sim;
      for (int i = 0; i < 6; ++i) J.model[i] = S.has_sim ? S.sim_model[i] : 0.0f;
    }
    return;
  }
  // ---- homography (src/pipeline.rs:2663-2755)
  const double thresh = (double)fmaxf(J.thr, 0.5f);
  if (threadIdx.x == 0) S.tsq_d = thresh * thresh;
  __syncthreads();
  // The incumbent, held identically by every thread.
  bool has_bh = S.has_sim != 0;
  double* const BH = S.BH;
  if (threadIdx.x == 0) {
    const double a = S.sim_model[0], b = S.sim_model[1];
    BH[0] = a, BH[1] = -b, BH[2] = S.sim_model[2];
    BH[3] = b, BH[4] = a, BH[5] = S.sim_model[3];
    BH[6] = 0.0, BH[7] = 0.0, BH[8] = 1.0;
  }
  __syncthreads();
  int best_count = 0;
  double best_err = __longlong_as_double(0x7ff0000000000000ll);
  bool err_known = true;
  if (has_bh) {
    best_count = h_count(J, S, BH);
    err_known = false;
  }
  auto finish_sim = [&]() {
    const int k = S.sim_count;
    for (int j = threadIdx.x; j < k; j += kRThreads) J.mask[J.list[j]] = 1;
    if (threadIdx.x == 0) {
      *J.count = k;
      *J.has_model = has_bh ? 1 : 0;
      for (int i = 0; i < 9; ++i) J.model[i] = has_bh ? (float)BH[i] : 0.0f;
    }
  };
  if (n < 4) {
    finish_sim();
    return;
  }
  // J.cdf is the similarity stage's: the same matches and weights
  const bool guided = J.weights != nullptr;
  const double wtot = guided ? weight_total(J, S) : 1.0;
  int max_iters = guided ? adaptive_iters_w((has_bh ? h_mass(J, S, BH) : 0.0) / wtot, 4, 64, 2000)
                         : adaptive_iters(best_count, n, 4, 64, 2000);
  if (threadIdx.x == 0) {
    S.draw_ptr = 0;
    S.draws_ready = 0;
  }
  __syncthreads();
  const uint64_t seed = J.hom_seed;
  const int draw_cap = 2000 * 16;  // at most 16 draws per iteration
  int iters_done = 0;
  bool stop = false;
  for (int base = 0, nh = 0; !stop && base < 2000; base += nh) {
    if (base >= max_iters) break;
    nh = min(kBatch, max_iters - base);
    // draws for this batch: at most 16 per iteration
    {
      const int need = S.draw_ptr + kDrawChunk;
      for (int t0 = S.draws_ready; t0 < need && t0 < draw_cap; t0 += kRThreads) {
        const int t = t0 + threadIdx.x;
        if (t < need && t < draw_cap) S.draws_s[t % (2 * kDrawChunk)] = sample_at(J.cdf, n, seed, (uint64_t)t);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        S.draws_ready = need < draw_cap ? need : draw_cap;
        S.dup = kBatch;
      }
      __syncthreads();
      // Almost every sample's first 4 draws are distinct: sample done + k then uses draws
      // p + 4 k .. p + 4 k + 3 up to the first one with a repeat, which thread 0 takes as
      // the reference does; the rest follow in the next turn.
      for (int done = 0; done < nh;) {
        const int p = S.draw_ptr, h = done + (int)threadIdx.x;
        if (h < nh) {
          int q[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) q[k] = S.draws_s[(p + 4 * (int)threadIdx.x + k) % (2 * kDrawChunk)];
          const bool dup = q[0] == q[1] || q[0] == q[2] || q[0] == q[3] || q[1] == q[2] || q[1] == q[3] || q[2] == q[3];
          if (dup) atomicMin(&S.dup, h);
#pragma unroll
          for (int k = 0; k < 4; ++k) S.quad[h][k] = q[k];
          S.hvalid[h] = 1;
        }
        __syncthreads();
        const int first = min(S.dup, nh);
        __syncthreads();
        if (threadIdx.x == 0) {
          int p0 = p + 4 * (first - done);
          if (first < nh) {
            // distinct draws in order, held in registers (q0 first)
            int chosen = 0, attempts = 0;
            int q0 = 0, q1 = 0, q2 = 0, q3 = 0;
            while (chosen < 4 && attempts < 16) {
              ++attempts;
              const int c = S.draws_s[(p0++) % (2 * kDrawChunk)];
              const bool dup = (chosen > 0 && q0 == c) || (chosen > 1 && q1 == c) || (chosen > 2 && q2 == c);
              if (!dup) {
                if (chosen == 0) q0 = c;
                else if (chosen == 1) q1 = c;
                else if (chosen == 2) q2 = c;
                else q3 = c;
                ++chosen;
              }
            }
            S.quad[first][0] = q0;
            S.quad[first][1] = q1;
            S.quad[first][2] = q2;
            S.quad[first][3] = q3;
            S.hvalid[first] = chosen == 4 ? 1 : 0;
            S.dup = kBatch;
          }
          S.draw_ptr = p0;
        }
        __syncthreads();
        done = min(first + 1, nh);
      }
    }
    // fits: a quad of lanes per hypothesis
    {
      const int h = threadIdx.x >> 2, ql = threadIdx.x & 3;
      const unsigned qmask = 0xFu << (threadIdx.x & 28);
      bool valid = h < nh && S.hvalid[h] != 0;
      if (valid) {
        double qp[4][2], tp[4][2];
        for (int i = 0; i < 4; ++i) {
          const float4 p = J.xy[S.quad[h][i]];
          qp[i][0] = p.x;
          qp[i][1] = p.y;
          tp[i][0] = p.z;
          tp[i][1] = p.w;
        }
        if (degenerate4(qp) || degenerate4(tp)) {
          valid = false;
        } else {
          double Hh[9];
          valid = quad_fit4(J.xy, S.quad[h], jac + h * 162, jac + h * 162 + 81, ql, qmask, Hh);
          if (valid && ql == 0) {
            for (int i = 0; i < 9; ++i) S.H[h][i] = Hh[i];
            S.hband[h] = h_band(S, Hh);
          }
        }
      }
      __syncwarp();  // every lane of the quad has read S.hvalid[h]
      if (ql == 0) S.hvalid[h] = valid ? 1 : 0;
    }
    __syncthreads();
    const int ns = stage_coords(J, S);
    h_count_batch(J, S, nh, best_count, ns);
    // replay in order
    for (int h = 0; h < nh; ++h) {
      const int it = base + h;
      if (it >= max_iters) {
        stop = true;
        break;
      }
      iters_done = it + 1;
      if (!S.hvalid[h]) continue;
      int c = S.hcnt[h];
      if (c < best_count) continue;
      double e = 0.0;
      bool e_known = false;
      if (c == best_count) {
        if (!err_known) {
          best_err = h_err(J, S, BH);
          err_known = true;
        }
        e = h_err(J, S, S.H[h]);
        e_known = true;
        if (!(e < best_err)) continue;
      }
      if (threadIdx.x < 9) S.Hc[threadIdx.x] = S.H[h][threadIdx.x];
      __syncthreads();
      local_optimize(J, S, jac, S.Hc, c, e, e_known);
      best_count = c;
      best_err = e;
      err_known = e_known;
      __syncthreads();
      if (threadIdx.x < 9) BH[threadIdx.x] = S.Hc[threadIdx.x];
      __syncthreads();
      has_bh = true;
      max_iters = guided ? adaptive_iters_w(h_mass(J, S, BH) / wtot, 4, 64, 2000)
                         : adaptive_iters(best_count, n, 4, 64, 2000);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && J.iters) J.iters[1] = iters_done;
  if (!has_bh) {
    // no model at all: no hypothesis was accepted, so no LO ran and J.list still
    // holds the similarity inliers
    finish_sim();
    return;
  }
  local_optimize(J, S, jac, BH, best_count, best_err, err_known);
  const int k = h_collect(J, S, BH);
  for (int j = threadIdx.x; j < k; j += kRThreads) J.mask[J.list[j]] = 1;
  if (threadIdx.x == 0) {
    *J.count = k;
    *J.has_model = 1;
    for (int i = 0; i < 9; ++i) J.model[i] = (float)BH[i];
  }
}
};

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) ransac_kernel(const RansacJob* __restrict__ jobs, float one) {
  __shared__ typename RansacCta<THREADS>::RShared S;
  RansacCta<THREADS>::run(jobs[blockIdx.x], S, one);
}

template <int THREADS>
static cudaError_t launch_ransac_t(const RansacJob* jobs, int n_jobs, cudaStream_t st) {
  constexpr size_t smem = RansacCta<THREADS>::kJacSmem;
  cudaError_t e = ensure_smem_attr((const void*)ransac_kernel<THREADS>, smem);
  if (e != cudaSuccess) return e;
  ransac_kernel<THREADS><<<n_jobs, THREADS, smem, st>>>(jobs, 1.0f);
  return cudaGetLastError();
}

// How many threads a set gets.  Microseconds with 512 / 256 / 128 threads:
// - up to one set per SM, 512: 148 homographies of 100 to 200 matches, outliers 10 to 70 %,
//   2834 / 3924 / 6407, of 3800 to 7600 3342 / 5264 / 12124.  But a set of up to 32 matches
//   gives 512 threads nothing to do but wait for one another: 148 of 12 at 10 % outliers 646 /
//   571 / 665 (one similarity of 6 on the host 84 us, 73 with 256).
// - up to two sets per SM, 256, so that all run at once: 296 homographies of 100 matches, 10 %,
//   1079 / 534 / 613; 296 of 1000 to 2000, 10 to 70 %, 3340 / 2961 / 4366.  Where sets differ
//   much, the longest ones set the time and 512 would still be better (of 100 to 200, 10 to
//   70 %, 3354 / 4133 / 6560), but half the speed for sets that are alike is worse.
// - beyond, similarities, which have little for many threads to share, 128, four sets per SM:
//   444 of 100 matches, 10 %, 238 / 156 / 92, of 1000 to 2000, 10 to 70 %, 1223 / 1017 / 977;
//   256 for larger sets (592 of 2000 to 4000 2235 / 1744 / 1959).
// - beyond, homographies 256: 444 of 100 matches, 10 %, 1609 / 1032 / 656, but of 100 to 200, 10
//   to 70 %, 3996 / 4482 / 6606; 1200 of those 7782 / 6715 / 8076, of 400 to 800 7844 / 6013 /
//   6527.  Of up to 32 matches 128 from three sets per SM: 1000 of 12, 10 %, 4058 / 2101 / 1449.
cudaError_t launch_ransac(const RansacJob* jobs, int n_jobs, int n_sim, int max_n, double mean_n, int num_sms,
                          cudaStream_t st) {
  if (n_jobs <= 0) return cudaSuccess;
  const bool few = max_n <= 32;
  if (n_jobs <= num_sms && !few) return launch_ransac_t<512>(jobs, n_jobs, st);
  const bool small = n_sim == n_jobs ? n_jobs > 2 * num_sms && mean_n <= 2000.0 : n_jobs > 3 * num_sms && few;
  return small ? launch_ransac_t<128>(jobs, n_jobs, st) : launch_ransac_t<256>(jobs, n_jobs, st);
}

}  // namespace psift
