// K9b: the top-k Hamming shortlist of a large catalog on the tensor cores.
//
// No reference counterpart (see hamming.cu).  With bits as +-1, the dot product of two
// 128-bit codes is 128 - 2 d: the distances of a 128-query tile to 256 codes are one
// M = 128, N = 256, K = 128 product of e4m3 values, exact in the f32 accumulators.
// Popcounts bound the scan of hamming.cu at 0.46 of their rate; the product costs four
// tcgen05.mma and the selection a maximum per 8 values, because only codes that beat a
// query's k-th distance so far can enter its list.
//
// The catalog is taken in ranges: topk_chunk_kernel lists the first one; then, range by
// range, each up to eight times as long as all before it,
//   hamming_tc_kernel     appends every code with d < T (the query's k-th distance so
//                         far) to the query's candidates: about 7 k of them;
//   hamming_select_kernel merges them with the list (distance, index order).
// A later code at distance T cannot displace a listed one (its index is larger), so the
// strict comparison loses nothing.  A query whose candidates overflow (its near codes
// are bunched late in the catalog) is scanned exactly by the select kernel.
//
// 2,000,000 codes x 4096 queries, top 64: see launch_topk_tc.
#include <cuda.h>

#include <algorithm>

#include "psift_internal.cuh"
#include "tc_ptx.cuh"

namespace psift {

cudaError_t launch_topk(const uint64_t* q, int nq, const uint64_t* cat, long long ncat, int k, int n_chunks,
                        unsigned long long* part, uint32_t* out_idx, uint32_t* out_dist, cudaStream_t st);

namespace {

constexpr int kHM = 128;                 // queries per A tile
constexpr int kHN = 256;                 // codes per MMA (N) = columns per accumulator
constexpr int kHSuper = 512;             // codes expanded to shared memory at a time
constexpr int kHHalves = kHSuper / kHN;
constexpr int kHParts = 4;               // epilogue warps per TMEM lane quarter (64 columns each)
constexpr int kHEpiWarps = 4 * kHParts;
constexpr int kHExpWarps = 2;
constexpr int kHThreads = 32 * (2 + kHEpiWarps + kHExpWarps);  // A copies, MMA, epilogue, code expansion
constexpr int kHAStages = 3;
constexpr uint32_t kHABytes = kHM * 128u;
constexpr uint32_t kHBBytes = kHSuper * 128u;
constexpr uint32_t kHSmB = kHAStages * kHABytes;
constexpr uint32_t kHSmBar = kHSmB + 2 * kHBBytes;
constexpr uint32_t kHSmTotal = kHSmBar + 256 + 1024;  // + alignment slack
static_assert(kHSmTotal <= 227 * 1024, "shared memory per CTA");
// kind::f8f6f4 instruction descriptor: D f32, A/B e4m3, both K-major, M = 128, N = 256
constexpr uint32_t kHIdesc = (1u << 4) | ((uint32_t)(kHN >> 3) << 17) | ((uint32_t)(kHM >> 4) << 24);
constexpr int kHCap = 2048;              // candidates kept per query and range
constexpr int kHQueryBlock = 8192;       // queries per pass (64 MB of candidates)

// 16 code bits -> 16 e4m3 bytes, +1 (0x38) where a bit is set, -1 (0xB8) elsewhere.
__device__ __forceinline__ uint4 expand16(uint32_t bits) {
  auto four = [](uint32_t n) { return 0xB8B8B8B8u ^ (((n & 15u) * 0x00204081u & 0x01010101u) << 7); };
  return make_uint4(four(bits), four(bits >> 4), four(bits >> 8), four(bits >> 12));
}

// Byte offset of 16-byte piece c of row r in a K-major, 128-byte-swizzled tile.
__device__ __forceinline__ uint32_t sw128_offset(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

__device__ __forceinline__ void umma_e4m3(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z)
      : "memory");
}

// The queries as swizzled e4m3 tiles (kHABytes each), and their counters cleared.
__global__ void hamming_expand_queries_kernel(const uint16_t* __restrict__ q, int nq, int tiles,
                                              uint8_t* __restrict__ image, uint32_t* __restrict__ cnt) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;  // (row, piece)
  if (u >= tiles * kHM * 8) return;
  const int row = u >> 3, c = u & 7;
  const uint32_t bits = row < nq ? q[(size_t)row * 8 + c] : 0u;
  const int tile = row / kHM, r = row % kHM;
  *reinterpret_cast<uint4*>(image + (size_t)tile * kHABytes + sw128_offset(r, c)) = expand16(bits);
  if (c == 0 && row < nq) cnt[row] = 0;
}

// One range [lo, hi) of the catalog against every query tile.  Persistent, one CTA per
// SM, each taking every gridDim.x-th block of kHSuper codes: two warps expand the next
// block into shared memory while the current one is multiplied with the query tiles
// (pre-swizzled, copied in through a ring); the accumulators are double-buffered in
// TMEM; 16 epilogue warps compare 64 columns each.  Waits are bounded as in
// match_tc_kernel.
__global__ void __launch_bounds__(kHThreads, 1)
    hamming_tc_kernel(const uint8_t* __restrict__ image, int q_tiles, int nq, const uint16_t* __restrict__ cat,
                      long long lo, long long hi, const uint32_t* __restrict__ list_dist, int k,
                      uint32_t* __restrict__ cnt, uint32_t* __restrict__ cand, uint32_t* err) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* afull = reinterpret_cast<uint64_t*>(smem + kHSmBar);  // [kHAStages] query tile landed
  uint64_t* aempty = afull + kHAStages;                           // [kHAStages] its MMAs done
  uint64_t* bfull = aempty + kHAStages;                           // [2] codes expanded
  uint64_t* bempty = bfull + 2;                                   // [2] their MMAs done
  uint64_t* accf = bempty + 2;                                    // [2] accumulator ready
  uint64_t* acce = accf + 2;                                      // [2] accumulator read out
  volatile uint32_t* taddr_slot = reinterpret_cast<volatile uint32_t*>(acce + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(acce + 3);
  const long long n_super = (hi - lo + kHSuper - 1) / kHSuper;
  if ((long long)blockIdx.x >= n_super) return;
  const int my = (int)((n_super - blockIdx.x + gridDim.x - 1) / gridDim.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kHAStages; ++i) {
      mbar_init(&afull[i], 1);
      mbar_init(&aempty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bfull[i], kHExpWarps * 32);
      mbar_init(&bempty[i], 1);
      mbar_init(&accf[i], 1);
      mbar_init(&acce[i], kHEpiWarps);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32((const void*)taddr_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *taddr_slot;
  const int tiles = my * q_tiles;  // query tiles to stream in all

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int issued = 0;
      for (; issued < tiles; ++issued) {
        const int as = issued % kHAStages;
        if (!mbar_wait(&aempty[as], (((uint32_t)(issued / kHAStages)) & 1u) ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&afull[as], kHABytes);
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                smem_u32(smem + as * kHABytes)),
            "l"(image + (size_t)(issued % q_tiles) * kHABytes), "r"(kHABytes), "r"(smem_u32(&afull[as]))
            : "memory");
      }
      if (!ok) {
        atomicOr(err, kErrTimeout);
        *abort_flag = 1;
        if (issued > 0)  // drain: the copies already issued land before the CTA leaves (bounded)
          for (int b = issued > kHAStages ? issued - kHAStages : 0; b < issued; ++b)
            for (uint32_t i = 0; i < kSpinLimit && !mbar_try_wait(&afull[b % kHAStages], ((uint32_t)(b / kHAStages)) & 1u);
                 ++i) {
            }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      bool ok = true;
      int t = 0, acc = 0;
      uint64_t* last_bar = nullptr;
      uint32_t last_par = 0;
      for (int s = 0; ok && s < my; ++s) {
        const int sb = s & 1;
        if (!mbar_wait(&bfull[sb], ((uint32_t)(s >> 1)) & 1u, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t b_base = smem_u32(smem + kHSmB + sb * kHBBytes);
        for (int qt = 0; ok && qt < q_tiles; ++qt, ++t) {
          const int as = t % kHAStages;
          if (!mbar_wait(&afull[as], ((uint32_t)(t / kHAStages)) & 1u, abort_flag)) {
            ok = false;
            break;
          }
          const uint32_t a_base = smem_u32(smem + as * kHABytes);
          for (int half = 0; half < kHHalves; ++half, ++acc) {
            const int st = acc & 1;
            const uint32_t ph = ((uint32_t)(acc >> 1)) & 1u;
            if (!mbar_wait(&acce[st], ph ^ 1u, abort_flag)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(st * kHN);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)  // 32 bytes of K each
              umma_e4m3(d, sw128_desc(a_base + kk * 32u), sw128_desc(b_base + half * (kHN * 128u) + kk * 32u), kHIdesc,
                        kk > 0 ? 1u : 0u);
            umma_commit(&accf[st]);
            last_bar = &accf[st];
            last_par = ph;
          }
          if (ok) umma_commit(&aempty[as]);
        }
        if (ok) umma_commit(&bempty[sb]);
      }
      if (!ok) {
        atomicOr(err, kErrTimeout);
        *abort_flag = 1;
        if (last_bar)  // drain (bounded): the last issued MMA group
          for (uint32_t i = 0; i < kSpinLimit && !mbar_try_wait(last_bar, last_par); ++i) {
          }
      }
    }
  } else if (warp < 2 + kHEpiWarps) {
    // epilogue: TMEM lane quarter warp % 4, 64-column part (warp - 2) / 4
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const float inf = __int_as_float(0x7f800000);
    bool live = true;
    int acc = 0;
    for (int s = 0; s < my; ++s) {
      const long long c0 = lo + ((long long)blockIdx.x + (long long)s * gridDim.x) * kHSuper;
      for (int qt = 0; qt < q_tiles; ++qt) {
        const int q = qt * kHM + quarter * 32 + lane;
        // d < T  <=>  dot = 128 - 2 d > 128 - 2 T
        const float thr = q < nq ? 128.0f - 2.0f * (float)list_dist[(size_t)q * k + (k - 1)] : inf;
        for (int half = 0; half < kHHalves; ++half, ++acc) {
          const int st = acc & 1;
          if (live && !__all_sync(0xffffffffu, mbar_wait(&accf[st], ((uint32_t)(acc >> 1)) & 1u, abort_flag))) {
            live = false;
            atomicOr(err, kErrTimeout);
            *abort_flag = 1;
          }
          if (!live) continue;
          tc_fence_after();
          __syncwarp();
          uint32_t r[2][32];
          const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(st * kHN + part * 64);
          tmem_ld32_nowait(ta, r[0]);
          tmem_ld32_nowait(ta + 32u, r[1]);
          tmem_wait32(r[0]);
          tmem_wait32(r[1]);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acce[st]);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float m = -inf;
#pragma unroll
            for (int c = 0; c < 32; c += 2) m = max3f(m, __uint_as_float(r[h][c]), __uint_as_float(r[h][c + 1]));
            if (m > thr) {  // few lanes: the columns that beat the threshold
              uint32_t hit = 0;
#pragma unroll
              for (int c = 0; c < 32; ++c) hit |= (__uint_as_float(r[h][c]) > thr ? 1u : 0u) << c;
              const long long base = c0 + half * kHN + part * 64 + h * 32;
              if (base + 32 > hi) hit &= base >= hi ? 0u : (1u << (int)(hi - base)) - 1u;  // codes past the range
              if (hit) {
                uint32_t pos = atomicAdd(&cnt[q], (uint32_t)__popc(hit));
                uint32_t* dst = cand + (size_t)q * kHCap;
                while (hit) {
                  const int c = __ffs(hit) - 1;
                  hit &= hit - 1;
                  if (pos < (uint32_t)kHCap) dst[pos] = (uint32_t)(base + c);
                  ++pos;
                }
              }
            }
          }
        }
      }
    }
  } else {
    // code expansion: 16 bits (one 16-byte piece) per thread and step
    const int t0 = threadIdx.x - 32 * (2 + kHEpiWarps);
    for (int s = 0; s < my; ++s) {
      const int sb = s & 1;
      if (!mbar_wait(&bempty[sb], (((uint32_t)(s >> 1)) & 1u) ^ 1u, abort_flag)) {
        atomicOr(err, kErrTimeout);
        *abort_flag = 1;
        break;
      }
      const long long c0 = lo + ((long long)blockIdx.x + (long long)s * gridDim.x) * kHSuper;
      uint8_t* dst = smem + kHSmB + sb * kHBBytes;
#pragma unroll 8
      for (int u = t0; u < kHSuper * 8; u += 32 * kHExpWarps) {
        const long long code = c0 + (u >> 3);
        const uint32_t bits = code < hi ? cat[code * 8 + (u & 7)] : 0u;
        *reinterpret_cast<uint4*>(dst + sw128_offset(u >> 3, u & 7)) = expand16(bits);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the stores before the MMAs' reads
      mbar_arrive(&bfull[sb]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

__device__ __forceinline__ uint32_t ham4(const uint4 a, const uint4 b) {
  return __popc(a.x ^ b.x) + __popc(a.y ^ b.y) + __popc(a.z ^ b.z) + __popc(a.w ^ b.w);
}

// Ascending bitonic sort of a[0..m), m a power of two, by the block.
__device__ __forceinline__ void block_sort(unsigned long long* a, int m) {
  for (int kk = 2; kk <= m; kk <<= 1)
    for (int j = kk >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int i = threadIdx.x; i < m / 2; i += blockDim.x) {
        const int lo = 2 * i - (i & (j - 1)), hi = lo + j;
        const unsigned long long x = a[lo], y = a[hi];
        if ((x > y) == ((lo & kk) == 0)) {
          a[lo] = y;
          a[hi] = x;
        }
      }
    }
  __syncthreads();
}

// One block per query: the k smallest (distance, index) keys of its list and its
// candidates of the range [lo, hi), written back to the list (sorted); the candidate
// count is cleared for the next range.  Overflowed candidates: the range is scanned
// twice, for the histogram of its distances and for the keys under (and, in index
// order, at) the k-th distance.
constexpr int kHSelThreads = 256;
__global__ void __launch_bounds__(kHSelThreads) hamming_select_kernel(const uint4* __restrict__ q,
                                                                      const uint4* __restrict__ cat, long long lo,
                                                                      long long hi, int k, uint32_t* __restrict__ cnt,
                                                                      const uint32_t* __restrict__ cand,
                                                                      uint32_t* __restrict__ list_idx,
                                                                      uint32_t* __restrict__ list_dist) {
  __shared__ unsigned long long keys[2 * kHCap];
  __shared__ uint32_t hist[129 + 1];
  __shared__ int s_d, s_need, s_low, s_scan[kHSelThreads / 32];
  const int qi = blockIdx.x, t = threadIdx.x;
  const uint32_t n = cnt[qi];
  if (n == 0) return;  // nothing in the range comes before the k-th entry
  __syncthreads();
  if (t == 0) cnt[qi] = 0;
  const uint4 qc = q[qi];
  uint32_t* li = list_idx + (size_t)qi * k;
  uint32_t* ld = list_dist + (size_t)qi * k;
  auto key_of = [](uint32_t d, uint32_t i) { return ((unsigned long long)d << 32) | i; };
  int total;
  if (n <= (uint32_t)kHCap) {
    for (int i = t; i < k; i += kHSelThreads) keys[i] = key_of(ld[i], li[i]);
    for (int i = t; i < (int)n; i += kHSelThreads) {
      const uint32_t c = cand[(size_t)qi * kHCap + i];
      keys[k + i] = key_of(ham4(qc, cat[c]), c);
    }
    total = k + (int)n;
  } else {
    for (int i = t; i < 130; i += kHSelThreads) hist[i] = 0;
    __syncthreads();
    for (int i = t; i < k; i += kHSelThreads) atomicAdd(&hist[ld[i]], 1u);
    for (long long c = lo + t; c < hi; c += kHSelThreads) atomicAdd(&hist[ham4(qc, cat[c])], 1u);
    __syncthreads();
    if (t == 0) {
      int run = 0, d = 0;
      while (run + (int)hist[d] < k) run += (int)hist[d++];
      s_d = d;           // the k-th distance
      s_need = k - run;  // keys taken at it
      s_low = 0;
    }
    __syncthreads();
    const uint32_t D = (uint32_t)s_d;
    // keys under D in any order at [0, k), then keys at D in index order
    int at = 0;
    for (int i = t; i < k; i += kHSelThreads)
      if (ld[i] < D) keys[atomicAdd(&s_low, 1)] = key_of(ld[i], li[i]);
    for (int i = 0; i < k; ++i)  // the list's entries at D: smaller indices than the range's
      if (ld[i] == D) {
        if (at < s_need && t == 0) keys[k + at] = key_of(D, li[i]);
        ++at;
      }
    for (long long c0 = lo; c0 < hi; c0 += kHSelThreads) {
      const long long c = c0 + t;
      const uint32_t d = c < hi ? ham4(qc, cat[c]) : 0xFFFFFFFFu;
      if (d < D) keys[atomicAdd(&s_low, 1)] = key_of(d, (uint32_t)c);
      const unsigned bal = __ballot_sync(0xffffffffu, d == D);
      if ((t & 31) == 0) s_scan[t >> 5] = __popc(bal);
      __syncthreads();
      int pos = at;
      for (int w = 0; w < kHSelThreads / 32; ++w) {
        if (w < (t >> 5)) pos += s_scan[w];
        at += s_scan[w];
      }
      pos += __popc(bal & ((1u << (t & 31)) - 1u));
      if (d == D && pos < s_need) keys[k + pos] = key_of(D, (uint32_t)c);
      __syncthreads();
    }
    __syncthreads();
    const int low = s_low;  // k - s_need
    for (int i = t; i < s_need; i += kHSelThreads) keys[low + i] = keys[k + i];
    total = k;
  }
  int m = 1;
  while (m < total) m <<= 1;
  for (int i = total + t; i < m; i += kHSelThreads) keys[i] = ~0ull;
  block_sort(keys, m);
  for (int i = t; i < k; i += kHSelThreads) {
    li[i] = (uint32_t)keys[i];
    ld[i] = (uint32_t)(keys[i] >> 32);
  }
}

size_t query_tiles(int nq) { return ((size_t)nq + kHM - 1) / kHM; }

}  // namespace

// Whether the tensor-core scan takes a shortlist of k over ncat codes for nq queries.
bool topk_tc_applies(int nq, long long ncat) { return nq >= 64 && ncat >= 65536; }

// The codes that topk_chunk_kernel lists first.
long long topk_tc_first(long long ncat) { return std::max<long long>(ncat / 64, 4096); }

size_t topk_tc_scratch(int nq) {
  const size_t b = (size_t)std::min(nq, kHQueryBlock);
  return query_tiles((int)b) * kHABytes + b * 4 + b * kHCap * 4 + 3 * 256;
}

cudaError_t launch_topk_tc(const uint64_t* q, int nq, const uint64_t* cat, long long ncat, int k, int first_chunks,
                           unsigned long long* part, uint8_t* scratch, uint32_t* out_idx, uint32_t* out_dist,
                           int num_sms, uint32_t* err, uint64_t* launches, cudaStream_t st) {
  cudaError_t e = ensure_smem_attr((const void*)hamming_tc_kernel, kHSmTotal);
  if (e != cudaSuccess) return e;
  const long long first = topk_tc_first(ncat);
  e = launch_topk(q, nq, cat, first, k, first_chunks, part, out_idx, out_dist, st);
  *launches += 2;
  for (int q0 = 0; q0 < nq && e == cudaSuccess; q0 += kHQueryBlock) {
    const int n = std::min(kHQueryBlock, nq - q0), tiles = (int)query_tiles(n);
    uint8_t* image = scratch;
    uint32_t* cnt = reinterpret_cast<uint32_t*>(scratch + align_up((size_t)tiles * kHABytes, 256));
    uint32_t* cand = cnt + align_up((size_t)n, 64);
    const uint64_t* qb = q + 2 * (size_t)q0;
    uint32_t *li = out_idx + (size_t)q0 * k, *ld = out_dist + (size_t)q0 * k;
    hamming_expand_queries_kernel<<<(tiles * kHM * 8 + 255) / 256, 256, 0, st>>>((const uint16_t*)qb, n, tiles, image,
                                                                               cnt);
    ++*launches;
    for (long long lo = first; lo < ncat;) {
      const long long hi = std::min(ncat, 8 * lo);
      const long long blocks = (hi - lo + kHSuper - 1) / kHSuper;
      hamming_tc_kernel<<<(unsigned)std::min<long long>(blocks, num_sms), kHThreads, kHSmTotal, st>>>(
          image, tiles, n, (const uint16_t*)cat, lo, hi, ld, k, cnt, cand, err);
      hamming_select_kernel<<<n, kHSelThreads, 0, st>>>((const uint4*)qb, (const uint4*)cat, lo, hi, k, cnt, cand, li,
                                                        ld);
      *launches += 2;
      lo = hi;
    }
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace psift
