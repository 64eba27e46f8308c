// K9: 128-bit binary signatures and the catalog's Hamming stages.
//
// Reference: quantize_descriptor_u128 (src/catalog.rs:37-45),
// FeatureCatalog::search_features coarse voting (src/catalog.rs:588-641) with the
// multi-index-hashing tables (:291-321) and count_coarse_hamming_votes
// (:707-728); quantize_descriptor_u8 / dequantize_descriptor_u8
// (src/pipeline.rs:1024-1044).
//
// Signatures are two little-endian u64 words (bit i of the u128 = bit i%64 of
// word i/64).  All comparisons are integer: results are bit-exact.
//
// Votes.  The exhaustive path counts the queries whose nearest signature in the
// entry is within 24 bits.  The MIH path (more than 32 entries) only reaches a
// signature through one of its 16 byte bands, i.e. when some byte of q ^ s is
// zero; a (query, entry) pair votes iff some signature of the entry has
// popcount(q ^ s) <= 24 AND a zero byte in q ^ s.  Both are evaluated directly,
// without the inverted tables.
//
// Top-k shortlist (no reference counterpart; the catalog search at scale): the k
// codes nearest to each query by (Hamming distance, catalog index), in hamming_tc.cu;
// the exact f32 re-rank of a shortlist is here.
#include <algorithm>

#include "psift_internal.cuh"

namespace psift {

constexpr int kTopKMax = 64;  // shortlist length upper bound

// popc(x0) + popc(x1) + popc(x2) + popc(x3) with three popcounts: a carry-save
// step gives, bit by bit, x0 + x1 + x2 = s + 2c (s = x0 ^ x1 ^ x2, c = majority),
// so the sum is popc(s) + 2 popc(c) + popc(x3), the same integer.  The popcount
// pipe bounds the Hamming scans; s and c are one LOP3 each on the ALU pipe.
__device__ __forceinline__ int popc4(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
  const uint32_t s = x0 ^ x1 ^ x2;
  const uint32_t c = (x0 & x1) | (x2 & (x0 ^ x1));
  return __popc(s) + 2 * __popc(c) + __popc(x3);
}

__device__ __forceinline__ int ham128(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint4 c) {
  return popc4(a0 ^ c.x, a1 ^ c.y, a2 ^ c.z, a3 ^ c.w);
}

__device__ __forceinline__ bool has_zero_byte(uint32_t x) { return ((x - 0x01010101u) & ~x & 0x80808080u) != 0; }

// quantize_descriptor_u128 (src/catalog.rs:37-45): bit d = desc[d] > 0.065.
// A warp handles kQDesc descriptors; lane l reads dims l, l + 32, l + 64, l + 96
// of each (coalesced 128-byte rows, all loads issued first) and the ballot of
// "dim 32 w + l > 0.065" over the lanes is code word w, bit l.
constexpr int kQDesc = 4;
__global__ void __launch_bounds__(256) quantize_codes_kernel(const float* __restrict__ desc, int n,
                                                             uint64_t* __restrict__ codes) {
  const int lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kQDesc;
  float v[kQDesc][4];
#pragma unroll
  for (int d = 0; d < kQDesc; ++d)
#pragma unroll
    for (int w = 0; w < 4; ++w) v[d][w] = row0 + d < n ? __ldcs(desc + (size_t)(row0 + d) * 128 + 32 * w + lane) : 0.0f;
#pragma unroll
  for (int d = 0; d < kQDesc; ++d) {
    uint32_t word[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) word[w] = __ballot_sync(0xffffffffu, v[d][w] > 0.065f);
    const uint32_t lo = lane ? word[2] : word[0], hi = lane ? word[3] : word[1];  // no indexed local array
    if (lane < 2 && row0 + d < n) codes[2 * (size_t)(row0 + d) + lane] = (uint64_t)lo | ((uint64_t)hi << 32);
  }
}

// quantize_descriptor_u128 + quantize_descriptor_u8: one warp per descriptor.
__global__ void quantize_kernel(const float* __restrict__ desc, int n, uint64_t* __restrict__ codes,
                                uint8_t* __restrict__ u8) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  const float4 v = reinterpret_cast<const float4*>(desc + (size_t)row * 128)[lane];
  const float e[4] = {v.x, v.y, v.z, v.w};
  if (codes) {
    // element 4*lane + j -> bit (4*lane + j)
    uint32_t nib = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) nib |= (e[j] > 0.065f ? 1u : 0u) << j;
    uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      const uint32_t x = __shfl_sync(0xffffffffu, nib, l);
      w[l >> 3] |= x << (4 * (l & 7));
    }
    if (lane == 0) {
      codes[2 * (size_t)row] = (uint64_t)w[0] | ((uint64_t)w[1] << 32);
      codes[2 * (size_t)row + 1] = (uint64_t)w[2] | ((uint64_t)w[3] << 32);
    }
  }
  if (u8) {
    uint32_t packed = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float q = roundf(e[j] * 512.0f);
      q = q < 0.0f ? 0.0f : (q > 255.0f ? 255.0f : q);
      packed |= (uint32_t)q << (8 * j);
    }
    reinterpret_cast<uint32_t*>(u8 + (size_t)row * 128)[lane] = packed;
  }
}

// dequantize_descriptor_u8: v/512 then L2 renormalisation (sequential sum).  A
// warp per 32 rows: the u8 rows are copied into shared memory (16-byte
// asynchronous copies, all in flight together), lane j adds up row j's squared
// norm sequentially from there, and the scaled rows are written back coalesced
// (a float4 per lane and row).
constexpr int kDqWarps = 4;
constexpr int kDqStride = 144;  // bytes per staged row: lanes reading 16 B of different rows hit distinct banks

__device__ __forceinline__ float4 dq4(uint32_t p) {
  return make_float4((float)(p & 0xFF) * (1.0f / 512.0f), (float)((p >> 8) & 0xFF) * (1.0f / 512.0f),
                     (float)((p >> 16) & 0xFF) * (1.0f / 512.0f), (float)(p >> 24) * (1.0f / 512.0f));
}

__global__ void __launch_bounds__(32 * kDqWarps) dequantize_kernel(const uint8_t* __restrict__ q, int n,
                                                                   float* __restrict__ out) {
  __shared__ __align__(16) uint8_t stage[kDqWarps][32 * kDqStride];
  __shared__ float inv_s[kDqWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * kDqWarps + warp) * 32;
  if (row0 >= n) return;
  const int nr = min(32, n - row0);
  uint8_t* st = stage[warp];
  // the warp's rows as 16-byte pieces: piece t of the block is row t / 8, bytes 16 (t % 8)
  for (int t = lane; t < nr * 8; t += 32) {
    const int r = t >> 3, c = (t & 7) * 16;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(st + r * kDqStride + c)),
                 "l"(q + (size_t)(row0 + r) * 128 + c)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  if (lane < nr) {
    const uint8_t* rr = st + lane * kDqStride;
    float s = 0.0f;
#pragma unroll 2
    for (int c = 0; c < 8; ++c) {
      const uint4 w = *reinterpret_cast<const uint4*>(rr + 16 * c);
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 v = dq4(ws[k]);
        s += v.x * v.x;
        s += v.y * v.y;
        s += v.z * v.z;
        s += v.w * v.w;
      }
    }
    const float norm = sqrtf(s);
    inv_s[warp][lane] = norm > 1e-7f ? 1.0f / norm : 1.0f;  // 1: the row is kept as it is
  }
  __syncwarp();
  for (int r = 0; r < nr; ++r) {
    float4 v = dq4(*reinterpret_cast<const uint32_t*>(st + r * kDqStride + 4 * lane));
    const float inv = inv_s[warp][r];
    if (inv != 1.0f) {
      v.x *= inv;
      v.y *= inv;
      v.z *= inv;
      v.w *= inv;
    }
    reinterpret_cast<float4*>(out + (size_t)(row0 + r) * 128)[lane] = v;
  }
}

// Votes: one block per entry, each thread owns queries tid, tid+blockDim, ...
// The entry's signatures are read in the same order by every lane (broadcast
// loads from L1); a query stops at its first qualifying signature.
__global__ void __launch_bounds__(256) votes_kernel(const uint4* __restrict__ q, int nq, const uint4* __restrict__ cat,
                                                     const long long* __restrict__ offsets, int mih,
                                                     uint32_t* __restrict__ votes) {
  const int e = blockIdx.x;
  const long long s0 = offsets[e], s1 = offsets[e + 1];
  uint32_t hits = 0;
  for (int qi = threadIdx.x; qi < nq; qi += blockDim.x) {
    const uint4 qq = q[qi];
    for (long long s = s0; s < s1; ++s) {
      const uint4 c = cat[s];
      const uint32_t x0 = qq.x ^ c.x, x1 = qq.y ^ c.y, x2 = qq.z ^ c.z, x3 = qq.w ^ c.w;
      const int d = popc4(x0, x1, x2, x3);
      if (d <= 24 && (!mih || has_zero_byte(x0) || has_zero_byte(x1) || has_zero_byte(x2) || has_zero_byte(x3))) {
        ++hits;
        break;
      }
    }
  }
  __shared__ uint32_t s_sum[8];
  for (int o = 16; o >= 1; o >>= 1) hits += __shfl_xor_sync(0xffffffffu, hits, o);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = hits;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_sum[w];
    votes[e] = t;
  }
}

// Exact FP32 L2^2 re-rank of each query's k candidates (reference summation
// order), sorted by (d2, index).  One warp per query; its candidates' rows come into
// shared memory `turn` at a time, k in equal turns of at most kRerankRows (a row is one
// coalesced 512-byte asynchronous copy), where lane c sums candidate c; no more shared
// memory than the turns need, so that few candidates leave room for more warps.  Bound by
// the random 512-byte rows: 4096 x 64 of a 2M-row catalog (134 MB) 50 us, 147 with a lane
// walking each row in global memory; 16384 x 1 / 17 / 64 of 500,000 rows 37 / 65 / 124 us
// (47 / 80 / 128 with 16 rows' memory and turns for every k; 39 / 77 / 256 by walking).
constexpr int kRerankRows = 16;
constexpr int kRerankStride = 132;  // floats per staged row: lanes of different rows hit distinct banks
constexpr int kRerankWarps = 8;
__global__ void __launch_bounds__(32 * kRerankWarps) l2_rerank_kernel(const float* __restrict__ qd, int nq,
                                                                      const float* __restrict__ cd,
                                                                      const uint32_t* __restrict__ cand, int k, int turn,
                                                                      uint32_t* __restrict__ out_idx,
                                                                      float* __restrict__ out_d2) {
  __shared__ unsigned long long s_keys[kRerankWarps][kTopKMax];
  extern __shared__ float4 s_rows[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qi = blockIdx.x * kRerankWarps + warp;
  if (qi >= nq) return;
  unsigned long long* keys = s_keys[warp];
  float* rows = reinterpret_cast<float*>(s_rows) + warp * turn * kRerankStride;
  const float* a = qd + (size_t)qi * 128;
  for (int t = lane; t < kTopKMax; t += 32) keys[t] = ~0ull;
  for (int t0 = 0; t0 < k; t0 += turn) {
    const int nr = min(turn, k - t0);
    const uint32_t mine = lane < nr ? cand[(long long)qi * k + t0 + lane] : 0xFFFFFFFFu;
    __syncwarp();  // the previous rows are read
    for (int r = 0; r < nr; ++r) {
      const uint32_t c = __shfl_sync(0xffffffffu, mine, r);
      if (c != 0xFFFFFFFFu)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(rows + r * kRerankStride + 4 * lane)),
                     "l"(cd + (size_t)c * 128 + 4 * lane)
                     : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (mine != 0xFFFFFFFFu) {
      const float* b = rows + lane * kRerankStride;
      float s = 0.0f;
#pragma unroll 8
      for (int i = 0; i < 128; i += 4) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(a + i));
        const float4 y = *reinterpret_cast<const float4*>(b + i);
        float d = x.x - y.x;
        s += d * d;
        d = x.y - y.y;
        s += d * d;
        d = x.z - y.z;
        s += d * d;
        d = x.w - y.w;
        s += d * d;
      }
      // non-negative floats order like their bit patterns
      keys[t0 + lane] = ((unsigned long long)__float_as_uint(s) << 32) | mine;
    }
  }
  __syncwarp();
  for (int kk = 2; kk <= kTopKMax; kk <<= 1) {
    for (int j = kk >> 1; j > 0; j >>= 1) {
      for (int i = lane; i < kTopKMax; i += 32) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long x = keys[i], y = keys[ixj];
          const bool up = (i & kk) == 0;
          if ((x > y) == up) {
            keys[i] = y;
            keys[ixj] = x;
          }
        }
      }
      __syncwarp();
    }
  }
  for (int t = lane; t < k; t += 32) {
    const unsigned long long key = keys[t];
    const bool ok = key != ~0ull;
    out_idx[(long long)qi * k + t] = ok ? (uint32_t)(key & 0xFFFFFFFFu) : 0xFFFFFFFFu;
    out_d2[(long long)qi * k + t] = ok ? __uint_as_float((uint32_t)(key >> 32)) : __int_as_float(0x7f800000);
  }
}

cudaError_t launch_quantize(const float* desc, int n, uint64_t* codes, uint8_t* u8, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (codes) quantize_codes_kernel<<<(n + 8 * kQDesc - 1) / (8 * kQDesc), 256, 0, st>>>(desc, n, codes);
  if (u8) quantize_kernel<<<(n + 7) / 8, 256, 0, st>>>(desc, n, nullptr, u8);
  return cudaGetLastError();
}

cudaError_t launch_dequantize(const uint8_t* q, int n, float* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  dequantize_kernel<<<(n + 32 * kDqWarps - 1) / (32 * kDqWarps), 32 * kDqWarps, 0, st>>>(q, n, out);
  return cudaGetLastError();
}

cudaError_t launch_votes(const uint64_t* q, int nq, const uint64_t* cat, const long long* offsets, int n_entries,
                         int mih, uint32_t* votes, cudaStream_t st) {
  if (n_entries <= 0) return cudaSuccess;
  votes_kernel<<<n_entries, 256, 0, st>>>((const uint4*)q, nq, (const uint4*)cat, offsets, mih, votes);
  return cudaGetLastError();
}

// Throughput probe for the INT roofline of the Hamming kernels: every thread
// keeps 8 independent 32-bit popcount chains in registers (no memory traffic in
// the loop); the sum is stored so nothing is dead code.
__global__ void __launch_bounds__(256) popc_probe_kernel(uint32_t seed, int iters, uint32_t* out) {
  uint32_t v[8], acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = seed * (threadIdx.x + 1u) + 0x9E3779B9u * (uint32_t)(j + 1) + blockIdx.x;
    acc[j] = 0;
  }
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      acc[j] += __popc(v[j]);
      v[j] ^= acc[j];
    }
  }
  uint32_t t = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) t += acc[j];
  out[blockIdx.x * blockDim.x + threadIdx.x] = t;
}

cudaError_t launch_popc_probe(int blocks, int iters, uint32_t* out, cudaStream_t st) {
  popc_probe_kernel<<<blocks, 256, 0, st>>>(12345u, iters, out);
  return cudaGetLastError();
}

cudaError_t launch_l2_rerank(const float* qd, int nq, const float* cd, const uint32_t* cand, int k,
                             uint32_t* out_idx, float* out_d2, cudaStream_t st) {
  if (nq <= 0) return cudaSuccess;
  const int turns = (k + kRerankRows - 1) / kRerankRows, turn = (k + turns - 1) / turns;
  const size_t smem = sizeof(float) * kRerankWarps * turn * kRerankStride;
  cudaError_t e = ensure_smem_attr((const void*)l2_rerank_kernel, smem);
  if (e != cudaSuccess) return e;
  l2_rerank_kernel<<<(nq + kRerankWarps - 1) / kRerankWarps, 32 * kRerankWarps, smem, st>>>(qd, nq, cd, cand, k, turn,
                                                                                          out_idx, out_d2);
  return cudaGetLastError();
}

}  // namespace psift
