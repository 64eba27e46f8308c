// K9b: the top-k Hamming shortlist of a large catalog on the tensor cores.
//
// No reference counterpart (see hamming.cu).  With bits as +-1, the dot product of two
// 128-bit codes is 128 - 2 d: the distances of a 128-query tile to 256 codes are one
// M = 128, N = 256, K = 128 product of e4m3 values, exact in the f32 accumulators.
// A popcount scan reached 0.46 of the popcount rate; the product costs four tcgen05.mma and the selection a maximum per 8 values, because only codes that beat a
// query's k-th distance so far can enter its list.
//
// The catalog is taken in ranges: hamming_select_kernel lists the first 2048 codes;
// then, range by range, each up to eight times as long as all before it,
//   hamming_tc_kernel     appends every code with d < T (the query's k-th distance so
//                         far) to the query's candidates: at most about 7 k of them;
//   hamming_select_kernel merges them with the list (distance, index order).
// A later code at distance T cannot displace a listed one (its index is larger), so the
// strict comparison loses nothing.  A query whose candidates overflow (its near codes
// are bunched late in the catalog) is scanned exactly by the select kernel.
//
// The last range of 2,000,000 codes x 4096 queries (950,000 codes) runs at 7.8 T code pairs/s,
// 2.0 PFLOP/s of e4m3 products; what bounds it is the epilogue (the maxima of 32,768
// accumulators per tile by 16 warps), not the tensor pipe.
#include <cuda.h>

#include <algorithm>

#include "psift_internal.cuh"
#include "tc_ptx.cuh"

namespace psift {

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
constexpr int kHQueryBlock = 8192;       // most queries per pass (64 MB of candidates)
constexpr int kHQueue = 96;              // hits a warp gathers before it appends them
constexpr uint32_t kHSmBar = kHSmB + 2 * kHBBytes;
constexpr uint32_t kHSmThr = kHSmBar + 256;
constexpr uint32_t kHSmQueue = kHSmThr + 4 * kHQueryBlock;
constexpr uint32_t kHSmTotal = kHSmQueue + kHEpiWarps * (kHQueue * 8 + 8) + 1024;  // + alignment slack
static_assert(kHSmTotal <= 227 * 1024, "shared memory per CTA");
// kind::f8f6f4 instruction descriptor: D f32, A/B e4m3, both K-major, M = 128, N = 256
constexpr uint32_t kHIdesc = (1u << 4) | ((uint32_t)(kHN >> 3) << 17) | ((uint32_t)(kHM >> 4) << 24);
constexpr int kHCap = 2048;              // candidates kept per query and range
constexpr int kHFirst = 2048;            // codes listed before the first range

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
    hamming_tc_kernel(const uint8_t* __restrict__ image, int all_tiles, int nq, const uint16_t* __restrict__ cat,
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
  // the query tiles of this CTA: all of them, or a share when the range has fewer code
  // blocks than there are SMs
  const int qt0 = (int)((long long)all_tiles * blockIdx.y / gridDim.y);
  const int q_tiles = (int)((long long)all_tiles * (blockIdx.y + 1) / gridDim.y) - qt0;
  const long long n_super = (hi - lo + kHSuper - 1) / kHSuper;
  if ((long long)blockIdx.x >= n_super || q_tiles == 0) return;
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
  // dot = 128 - 2 d: d < T <=> dot > 128 - 2 T
  float* thr_s = reinterpret_cast<float*>(smem + kHSmThr);
  for (int i = threadIdx.x; i < q_tiles * kHM; i += kHThreads)
    thr_s[i] = qt0 * kHM + i < nq ? 128.0f - 2.0f * (float)list_dist[(size_t)(qt0 * kHM + i) * k + (k - 1)]
                                  : __int_as_float(0x7f800000);
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
            "l"(image + (size_t)(qt0 + issued % q_tiles) * kHABytes), "r"(kHABytes), "r"(smem_u32(&afull[as]))
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
    // epilogue: TMEM lane quarter warp % 4, 64-column part (warp - 2) / 4.  Hits go to
    // the warp's queue in shared memory and on to the queries' candidates kHQueue or so
    // at a time: one global atomic's latency per batch, not per hit.
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    uint2* queue = reinterpret_cast<uint2*>(smem + kHSmQueue) + (warp - 2) * kHQueue;
    uint32_t* queued = reinterpret_cast<uint32_t*>(smem + kHSmQueue + kHEpiWarps * kHQueue * 8) + 2 * (warp - 2);
    const float inf = __int_as_float(0x7f800000);
    bool live = true;
    int acc = 0;
    auto append = [&](uint32_t q, uint32_t code) {
      const uint32_t pos = atomicAdd(&cnt[q], 1u);
      if (pos < (uint32_t)kHCap) cand[(size_t)q * kHCap + pos] = code;
    };
    auto flush = [&](int n) {
      for (int i = lane; i < n; i += 32) append(queue[i].x, queue[i].y);
      __syncwarp();
      if (lane == 0) *queued = 0;
      __syncwarp();
    };
    if (lane == 0) *queued = 0;
    __syncwarp();
    for (int s = 0; s < my; ++s) {
      const long long c0 = lo + ((long long)blockIdx.x + (long long)s * gridDim.x) * kHSuper + part * 64;
      const bool tail = c0 + kHSuper > hi;
      for (int qt = 0; qt < q_tiles; ++qt) {
        const int q = (qt0 + qt) * kHM + quarter * 32 + lane;
        const float thr = thr_s[qt * kHM + quarter * 32 + lane];
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
          float m[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float m0 = -inf, m1 = -inf;
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
              m0 = max3f(m0, __uint_as_float(r[h][c]), __uint_as_float(r[h][c + 1]));
              m1 = max3f(m1, __uint_as_float(r[h][c + 2]), __uint_as_float(r[h][c + 3]));
            }
            m[h] = fmaxf(m0, m1);
          }
          if (!__any_sync(0xffffffffu, fmaxf(m[0], m[1]) > thr)) continue;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (m[h] > thr) {  // few lanes: the columns that beat the threshold
              uint32_t hit = 0;
#pragma unroll
              for (int c = 0; c < 32; ++c) hit |= (__uint_as_float(r[h][c]) > thr ? 1u : 0u) << c;
              const long long base = c0 + half * kHN + h * 32;
              if (tail && base + 32 > hi) hit &= base >= hi ? 0u : (1u << (int)(hi - base)) - 1u;  // codes past the range
              uint32_t pos = hit ? atomicAdd(queued, (uint32_t)__popc(hit)) : 0u;
              while (hit) {
                const uint32_t code = (uint32_t)(base + __ffs(hit) - 1);
                hit &= hit - 1;
                if (pos < (uint32_t)kHQueue) queue[pos] = make_uint2((uint32_t)q, code);
                else append((uint32_t)q, code);
                ++pos;
              }
            }
          }
          __syncwarp();
          const uint32_t n = *reinterpret_cast<volatile uint32_t*>(queued);
          if (n >= (uint32_t)kHQueue / 2) flush(min((int)n, kHQueue));
        }
      }
    }
    flush(min((int)*reinterpret_cast<volatile uint32_t*>(queued), kHQueue));
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
// count is cleared for the next range.  FIRST: no list yet, the candidates are all the
// range's codes (at most kHCap).  A histogram of the distances gives the k-th one, D;
// only the keys up to D are sorted.  Overflowed candidates: the range is scanned twice,
// for the histogram and for the keys under (and, in index order, at) D.
constexpr int kHSelThreads = 256;
template <bool FIRST>
__global__ void __launch_bounds__(kHSelThreads) hamming_select_kernel(const uint4* __restrict__ q,
                                                                      const uint4* __restrict__ cat, long long lo,
                                                                      long long hi, int k, uint32_t* __restrict__ cnt,
                                                                      const uint32_t* __restrict__ cand,
                                                                      uint32_t* __restrict__ list_idx,
                                                                      uint32_t* __restrict__ list_dist) {
  __shared__ unsigned long long keys[kHCap + 64], out[kHCap + 64];
  __shared__ uint32_t hist[129];
  __shared__ int s_d, s_need, s_low, s_scan[kHSelThreads / 32];
  const int qi = blockIdx.x, t = threadIdx.x;
  const uint32_t n = FIRST ? (uint32_t)(hi - lo) : cnt[qi];
  if (!FIRST && n == 0) return;  // nothing in the range comes before the k-th entry
  for (int i = t; i < 129; i += kHSelThreads) hist[i] = 0;
  if (t == 0) s_low = 0, s_d = 128, s_need = k;  // fewer than k codes in all: every one is taken
  __syncthreads();
  if (!FIRST && t == 0) cnt[qi] = 0;
  const uint4 qc = q[qi];
  uint32_t* li = list_idx + (size_t)qi * k;
  uint32_t* ld = list_dist + (size_t)qi * k;
  auto key_of = [](uint32_t d, uint32_t i) { return ((unsigned long long)d << 32) | i; };
  const int kl = FIRST ? 0 : k;  // listed so far
  const bool gathered = n <= (uint32_t)kHCap;
  for (int i = t; i < kl; i += kHSelThreads) {
    keys[i] = key_of(ld[i], li[i]);
    atomicAdd(&hist[ld[i]], 1u);
  }
  if (gathered) {
    for (int i = t; i < (int)n; i += kHSelThreads) {
      const uint32_t c = FIRST ? (uint32_t)(lo + i) : cand[(size_t)qi * kHCap + i];
      const uint32_t d = ham4(qc, cat[c]);
      keys[kl + i] = key_of(d, c);
      atomicAdd(&hist[d], 1u);
    }
  } else {
    for (long long c = lo + t; c < hi; c += kHSelThreads) atomicAdd(&hist[ham4(qc, cat[c])], 1u);
  }
  __syncthreads();
  if (t < 32) {  // D: the bin where the running count reaches k (lane l scans bins 5l .. 5l + 4)
    int local = 0;
#pragma unroll
    for (int b = 0; b < 5; ++b) local += 5 * t + b < 129 ? (int)hist[5 * t + b] : 0;
    int incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (t >= o) incl += v;
    }
    int run = incl - local;
    if (run < k && incl >= k) {
      int d = 5 * t;
      while (run + (int)hist[d] < k) run += (int)hist[d++];
      s_d = d;
      s_need = k - run;  // keys taken at it
    }
  }
  __syncthreads();
  const uint32_t D = (uint32_t)s_d;
  int total;
  if (gathered) {  // every key up to D, in any order
    for (int i = t; i < kl + (int)n; i += kHSelThreads)
      if ((uint32_t)(keys[i] >> 32) <= D) out[atomicAdd(&s_low, 1)] = keys[i];
    __syncthreads();
    total = s_low;
  } else {
    // keys under D in any order at [0, k - need); the keys at D follow in index order,
    // the list's first (smaller indices than the range's), need of them
    const int need = s_need;
    int at = 0;
    for (int i = t; i < k; i += kHSelThreads)
      if ((uint32_t)(keys[i] >> 32) < D) out[atomicAdd(&s_low, 1)] = keys[i];
    for (int i = 0; i < k; ++i)
      if ((uint32_t)(keys[i] >> 32) == D) {
        if (at < need && t == 0) out[k - need + at] = keys[i];
        ++at;
      }
    for (long long c0 = lo; c0 < hi; c0 += kHSelThreads) {
      const long long c = c0 + t;
      const uint32_t d = c < hi ? ham4(qc, cat[c]) : 0xFFFFFFFFu;
      if (d < D) out[atomicAdd(&s_low, 1)] = key_of(d, (uint32_t)c);
      const unsigned bal = __ballot_sync(0xffffffffu, d == D);
      if ((t & 31) == 0) s_scan[t >> 5] = __popc(bal);
      __syncthreads();
      int pos = at;
      for (int w = 0; w < kHSelThreads / 32; ++w) {
        if (w < (t >> 5)) pos += s_scan[w];
        at += s_scan[w];
      }
      pos += __popc(bal & ((1u << (t & 31)) - 1u));
      if (d == D && pos < need) out[k - need + pos] = key_of(D, (uint32_t)c);
      __syncthreads();
    }
    total = k;
  }
  int m = 1;
  while (m < total) m <<= 1;
  unsigned long long* dst = out;
  if (m <= kHCap) {
    for (int i = total + t; i < m; i += kHSelThreads) dst[i] = ~0ull;
    block_sort(dst, m);
  } else {
    // a crowd of ties that cannot be padded in place: rank each key by counting
    __syncthreads();
    for (int i = t; i < total; i += kHSelThreads) {
      const unsigned long long x = out[i];
      int rank = 0;
      for (int j = 0; j < total; ++j) rank += out[j] < x;
      if (rank < k) keys[rank] = x;
    }
    __syncthreads();
    dst = keys;
  }
  for (int i = t; i < k; i += kHSelThreads) {  // places without a code: ~0
    li[i] = i < total ? (uint32_t)dst[i] : 0xFFFFFFFFu;
    ld[i] = i < total ? (uint32_t)(dst[i] >> 32) : 0xFFFFFFFFu;
  }
}

size_t query_tiles(int nq) { return ((size_t)nq + kHM - 1) / kHM; }

}  // namespace

// Device scratch for a query block (the queries are taken `block` at a time).
size_t topk_scratch(int nq, int block) {
  const size_t b = (size_t)std::min(nq, block);
  return query_tiles((int)b) * kHABytes + b * 4 + b * kHCap * 4 + 3 * 256;
}

// 2M codes x 4096 queries: 1.69 ms (11.9 as a popcount scan with per-chunk lists merged
// at the end); 65536 x 512: 81 us (742); 16384 x 64: 37 us (301); 4096 x 1: 32 us (304).
cudaError_t launch_topk(const uint64_t* q, int nq, const uint64_t* cat, long long ncat, int k, int block,
                        uint8_t* scratch, uint32_t* out_idx, uint32_t* out_dist, int num_sms, uint32_t* err,
                        uint64_t* launches, cudaStream_t st) {
  cudaError_t e = ensure_smem_attr((const void*)hamming_tc_kernel, kHSmTotal);
  if (e != cudaSuccess) return e;
  for (int q0 = 0; q0 < nq; q0 += block) {
    const int n = std::min(block, nq - q0), tiles = (int)query_tiles(n);
    uint8_t* image = scratch;
    uint32_t* cnt = reinterpret_cast<uint32_t*>(scratch + align_up((size_t)tiles * kHABytes, 256));
    uint32_t* cand = cnt + align_up((size_t)n, 64);
    const uint64_t* qb = q + 2 * (size_t)q0;
    uint32_t *li = out_idx + (size_t)q0 * k, *ld = out_dist + (size_t)q0 * k;
    const long long first = std::min<long long>(ncat, kHFirst);
    hamming_select_kernel<true><<<n, kHSelThreads, 0, st>>>((const uint4*)qb, (const uint4*)cat, 0, first, k, cnt,
                                                            cand, li, ld);
    ++*launches;
    if (first == ncat) continue;
    hamming_expand_queries_kernel<<<(tiles * kHM * 8 + 255) / 256, 256, 0, st>>>((const uint16_t*)qb, n, tiles, image,
                                                                               cnt);
    ++*launches;
    for (long long lo = first; lo < ncat;) {
      const long long hi = std::min(ncat, 8 * lo);
      const long long blocks = (hi - lo + kHSuper - 1) / kHSuper;
      const int share = blocks < num_sms ? std::min(tiles, (int)(num_sms / blocks)) : 1;
      hamming_tc_kernel<<<dim3((unsigned)std::min<long long>(blocks, num_sms), share), kHThreads, kHSmTotal, st>>>(
          image, tiles, n, (const uint16_t*)cat, lo, hi, ld, k, cnt, cand, err);
      hamming_select_kernel<false><<<n, kHSelThreads, 0, st>>>((const uint4*)qb, (const uint4*)cat, lo, hi, k, cnt,
                                                               cand, li, ld);
      *launches += 2;
      lo = hi;
    }
  }
  return cudaGetLastError();
}

}  // namespace psift
