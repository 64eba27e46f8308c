// K9b: the top-k Hamming shortlist of a large catalog on the tensor cores.
//
// No reference counterpart (see hamming.cu).  With bits as +-1, the dot product of two
// 128-bit codes is 128 - 2 d: the distances of a 128-query tile to 256 codes are one
// M = 128, N = 256, K = 128 product of e4m3 values, exact in the f32 accumulators.
// A popcount scan reached 0.46 of the popcount rate; the product costs four tcgen05.mma and
// the selection a maximum of every accumulator, because only codes that beat a query's k-th
// entry so far can enter its list.
//
// The catalog is taken in parts, each a sample of all of it (hamming_order.cuh):
// hamming_first_kernel lists the smallest (at most 8192 codes); then, part by part, each
// up to seven times as long as all before it,
//   hamming_tc_kernel     appends every code that comes before the query's k-th entry so
//                         far (T, iT) in (distance, index) order to the query's
//                         candidates: about 7 k of them, in whatever order the catalog is;
//   hamming_select_kernel merges them with the list.
// The last part of 2,000,000 codes x 4096 queries (1.5 M codes) runs at 7.2 T code pairs/s,
// 1.9 PFLOP/s of e4m3 products; what bounds it is the epilogue (the maxima of 32,768
// accumulators per tile by 16 warps, and the lookup of those that are candidates: ALU pipe 57
// to 60 %), not the tensor pipe (43 %).
// Codes at distance T are told apart by their index in steps of 256 (the few too many fall
// out at the merge), so a catalog of many equal codes does not flood the candidates either.
// A query whose candidates overflow all the same is scanned exactly by the select kernel.
#include <cuda.h>

#include <algorithm>

#include "hamming_order.cuh"
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
static_assert(kHExpWarps == 2 && HammingOrder::kUnit == 8 && kHSuper == kHExpWarps * 32 * HammingOrder::kUnit,
              "a unit per lane of the expansion warps");
// kind::f8f6f4 instruction descriptor: D f32, A/B e4m3, both K-major, M = 128, N = 256
constexpr uint32_t kHIdesc = (1u << 4) | ((uint32_t)(kHN >> 3) << 17) | ((uint32_t)(kHM >> 4) << 24);
constexpr int kHCap = 2048;              // candidates kept per query and part

// A query's k-th entry as one word: the index in steps of 256 | distance + 1 (0: no code
// comes before it).
__device__ __forceinline__ uint32_t pack_kth(uint32_t dist, uint32_t index) { return (index & ~255u) | (dist + 1u); }

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

// One part of the catalog (`n` places, 8 per unit) against every query tile.  Persistent, one
// CTA per SM, each taking every gridDim.x-th block of kHSuper codes: two warps expand the next
// block into shared memory while the current one is multiplied with the query tiles
// (pre-swizzled, copied in through a ring); the accumulators are double-buffered in
// TMEM; 16 epilogue warps compare 64 columns each.  Waits are bounded as in
// match_tc_kernel.
__global__ void __launch_bounds__(kHThreads, 1)
    hamming_tc_kernel(const uint8_t* __restrict__ image, int all_tiles, int nq, const uint4* __restrict__ cat,
                      long long ncat, const __grid_constant__ HammingOrder order, int part_i, long long n,
                      const uint32_t* __restrict__ kth, uint32_t* __restrict__ cnt, uint32_t* __restrict__ cand,
                      uint32_t* err) {
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
  // the query tiles of this CTA: all of them, or a share when the part has fewer code
  // blocks than there are SMs
  const int qt0 = (int)((long long)all_tiles * blockIdx.y / gridDim.y);
  const int q_tiles = (int)((long long)all_tiles * (blockIdx.y + 1) / gridDim.y) - qt0;
  const long long n_super = (n + kHSuper - 1) / kHSuper;
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
  uint32_t* kth_s = reinterpret_cast<uint32_t*>(smem + kHSmThr);
  for (int i = threadIdx.x; i < q_tiles * kHM; i += kHThreads) kth_s[i] = qt0 * kHM + i < nq ? kth[qt0 * kHM + i] : 0u;
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
    auto append = [&](uint32_t q, uint32_t place) {
      const uint32_t pos = atomicAdd(&cnt[q], 1u);
      if (pos < (uint32_t)kHCap) cand[(size_t)q * kHCap + pos] = place;
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
      const long long p0 = ((long long)blockIdx.x + (long long)s * gridDim.x) * kHSuper;
      const long long c0 = p0 + part * 64;
      const bool tail = c0 + kHSuper > n;
      // the first code of either half, rounded down to a step of 256: what the index of a
      // query's k-th entry is compared with
      uint32_t first = 0;
      if (lane < kHHalves && p0 + lane * kHN < n)
        first = order.unit(part_i, (uint32_t)((p0 + lane * kHN) / HammingOrder::kUnit)) * HammingOrder::kUnit & ~255u;
      const uint32_t first0 = __shfl_sync(0xffffffffu, first, 0), first1 = __shfl_sync(0xffffffffu, first, 1);
      for (int qt = 0; qt < q_tiles; ++qt) {
        const int q = (qt0 + qt) * kHM + quarter * 32 + lane;
        const uint32_t e = kth_s[qt * kHM + quarter * 32 + lane];
        // dot = 128 - 2 d is even: d < T <=> dot > 128 - 2 T, d <= T <=> dot > 127 - 2 T
        const float thr0 = __fmaf_rn(-2.0f, __uint_as_float(0x4B000000u | (e & 255u)), 16777346.0f);
        for (int half = 0; half < kHHalves; ++half, ++acc) {
          const float thr = (half ? first1 : first0) <= e ? thr0 - 1.0f : thr0;
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
              uint32_t hit = 0;  // bit c: the sign of thr - column c (half of it off the pipe that takes the maxima)
#pragma unroll
              for (int c = 31; c >= 0; --c)
                hit = __funnelshift_l(__float_as_uint(__fsub_rn(thr, __uint_as_float(r[h][c]))), hit, 1);
              const long long base = c0 + half * kHN + h * 32;
              if (tail && base + 32 > n) hit &= base >= n ? 0u : (1u << (int)(n - base)) - 1u;  // past the part
              uint32_t pos = hit ? atomicAdd(queued, (uint32_t)__popc(hit)) : 0u;
              while (hit) {
                const uint32_t place = (uint32_t)(base + __ffs(hit) - 1);
                hit &= hit - 1;
                if (pos < (uint32_t)kHQueue) queue[pos] = make_uint2((uint32_t)q, place);
                else append((uint32_t)q, place);
                ++pos;
              }
            }
          }
          __syncwarp();
          const uint32_t held = *reinterpret_cast<volatile uint32_t*>(queued);
          if (held >= (uint32_t)kHQueue / 2) flush(min((int)held, kHQueue));
        }
      }
    }
    flush(min((int)*reinterpret_cast<volatile uint32_t*>(queued), kHQueue));
  } else {
    // code expansion: a warp takes half of a block's units, a lane 8 of their codes, all
    // loaded at once before the wait for the buffer
    const int half = warp - (2 + kHEpiWarps);
    for (int s = 0; s < my; ++s) {
      const int sb = s & 1;
      const long long place =
          ((long long)blockIdx.x + (long long)s * gridDim.x) * kHSuper + (half * 32 + lane) * HammingOrder::kUnit;
      const uint32_t unit = place < n ? order.unit(part_i, (uint32_t)(place / HammingOrder::kUnit)) : 0xFFFFFFFFu;
      uint4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const long long code = (long long)__shfl_sync(0xffffffffu, unit, 4 * j + (lane >> 3)) * 8 + (lane & 7);
        v[j] = code < ncat ? cat[code] : make_uint4(0, 0, 0, 0);
      }
      if (!mbar_wait(&bempty[sb], (((uint32_t)(s >> 1)) & 1u) ^ 1u, abort_flag)) {
        atomicOr(err, kErrTimeout);
        *abort_flag = 1;
        break;
      }
      uint8_t* dst = smem + kHSmB + sb * kHBBytes;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = half * (kHSuper / 2) + 32 * j + lane;
        const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(dst + sw128_offset(row, c)) = expand16(w[c >> 1] >> (16 * (c & 1)));
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
  // three popcounts: x + y + z = s + 2 c, bit by bit (see ham128 in hamming.cu)
  const uint32_t x = a.x ^ b.x, y = a.y ^ b.y, z = a.z ^ b.z;
  return __popc(x ^ y ^ z) + 2 * __popc((x & y) | (x & z) | (y & z)) + __popc(a.w ^ b.w);
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

constexpr int kHSelThreads = 256;

// A block for QB queries: the k smallest (distance, index) keys of the first part, `part_i`,
// to the list (sorted) and the k-th of them to `kth`.  Distances go to shared memory as
// bytes; the k-th one, D, is found by halving its range, four bytes at a time; then
// every thread looks through a run of consecutive places, and a sum over the threads tells
// where its keys under D and its first ones at D (places are in index order) belong.
// Bound by the codes' way from L2 to the SMs with one query a block, by popcounts with two.
template <int UNITS, int QB>
__global__ void __launch_bounds__(kHSelThreads)
    hamming_first_kernel(const uint4* __restrict__ q, int nq, const uint4* __restrict__ cat, long long ncat,
                         const __grid_constant__ HammingOrder order, int part_i, int k,
                         uint32_t* __restrict__ list_idx, uint32_t* __restrict__ list_dist, uint32_t* __restrict__ kth) {
  constexpr int kPlaces = UNITS * HammingOrder::kUnit;  // most places of the part
  constexpr int kRun = kPlaces / kHSelThreads;          // of a thread's run
  static_assert(kRun % 4 == 0 && kPlaces < 65536, "whole words, sums in 16 bits");
  constexpr int kWarps = kHSelThreads / 32;
  __shared__ __align__(16) uint8_t dist[QB][kPlaces];
  __shared__ uint32_t units[UNITS], sums[2][kWarps];
  __shared__ unsigned long long keys[64];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int n_units = (int)order.part_units(part_i);
  for (int u = t; u < n_units; u += kHSelThreads) units[u] = order.unit(part_i, (uint32_t)u);
  __syncthreads();
  auto code_at = [&](int p) {  // the code at place p; ncat or more: none
    const int u = p / HammingOrder::kUnit;
    return u < n_units ? (long long)units[u] * HammingOrder::kUnit + p % HammingOrder::kUnit : ncat;
  };
  uint4 qc[QB];
#pragma unroll
  for (int b = 0; b < QB; ++b) qc[b] = q[min((int)blockIdx.x * QB + b, nq - 1)];
  int valid = 0;
#pragma unroll 8
  for (int p = t; p < kPlaces; p += kHSelThreads) {
    const long long c = code_at(p);
    const bool ok = c < ncat;
    const uint4 code = ok ? cat[c] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int b = 0; b < QB; ++b) dist[b][p] = ok ? (uint8_t)ham4(qc[b], code) : (uint8_t)128;
    valid += ok;
  }
  int turn = 0;
  auto block_sum = [&](uint32_t v) {  // also: what was written to shared memory before is visible
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) sums[turn & 1][warp] = v;
    __syncthreads();
    uint32_t r = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) r += sums[turn & 1][w];
    ++turn;
    return r;
  };
  const int listed = min(k, (int)block_sum((uint32_t)valid));
#pragma unroll 1
  for (int b = 0; b < QB; ++b) {
    const int qi = blockIdx.x * QB + b;
    if (qi >= nq) break;
    uint32_t run[kRun / 4];  // places kRun t .. kRun t + kRun - 1
#pragma unroll
    for (int i = 0; i < kRun / 4; ++i) run[i] = reinterpret_cast<const uint32_t*>(dist[b])[t * (kRun / 4) + i];
    // bytes (at most 128) of the run up to m <= 127: 128 + m - byte does not borrow
    auto count = [&](int m) {
      const uint32_t m4 = (uint32_t)(128 + m) * 0x01010101u;
      uint32_t c = 0;
#pragma unroll
      for (int i = 0; i < kRun / 4; ++i) c += (m4 - run[i]) >> 7 & 0x01010101u;
      return c * 0x01010101u >> 24;
    };
    int lo = 0, hi = 128;  // D in [lo, hi]: the smallest with `listed` distances up to it
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if ((int)block_sum(count(mid)) >= listed) hi = mid;
      else lo = mid + 1;
    }
    const int D = lo;
    // the top bits of a word's bytes that hold distances up to D (128: also where no code is)
    auto upto = [&](int i) {
      if (D < 128) return ((uint32_t)(128 + D) * 0x01010101u - run[i]) & 0x80808080u;
      uint32_t m = 0;
      for (int j = 0; j < 4; ++j) m |= code_at(t * kRun + 4 * i + j) < ncat ? 0x80u << 8 * j : 0u;
      return m;
    };
    // keys under D | keys at D << 16, of the threads before this one and in all
    const uint32_t under = D > 0 ? count(D - 1) : 0u;
    uint32_t mine = 0;
#pragma unroll
    for (int i = 0; i < kRun / 4; ++i) mine += __popc(upto(i));
    mine = under | (mine - under) << 16;
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) sums[turn & 1][warp] = incl;
    __syncthreads();
    uint32_t before = incl - mine, all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t v = sums[turn & 1][w];
      if (w < warp) before += v;
      all += v;
    }
    ++turn;
    const int below = (int)(all & 0xffffu);
    int at_low = (int)(before & 0xffffu), at_tie = below + (int)(before >> 16);
    if ((mine & 0xffffu) || (mine && at_tie < listed)) {
#pragma unroll
      for (int i = 0; i < kRun / 4; ++i) {
        for (uint32_t m = upto(i); m; m &= m - 1) {
          const int byte = (__ffs(m) - 1) / 8, d = (int)(run[i] >> 8 * byte & 0xffu);
          int& at = d < D ? at_low : at_tie;
          if (at < listed) keys[at] = (unsigned long long)d << 32 | (uint32_t)code_at(t * kRun + 4 * i + byte);
          ++at;
        }
      }
    }
    __syncthreads();
    uint32_t* li = list_idx + (size_t)qi * k;
    uint32_t* ld = list_dist + (size_t)qi * k;
    if (t < listed) {  // a key's place is the number of smaller ones
      const unsigned long long x = keys[t];
      int rank = 0;
      for (int j = 0; j < listed; ++j) rank += keys[j] < x;
      li[rank] = (uint32_t)x;
      ld[rank] = (uint32_t)(x >> 32);
      if (rank == k - 1) kth[qi] = pack_kth((uint32_t)(x >> 32), (uint32_t)x);
    } else if (t < k) {  // places without a code: ~0
      li[t] = 0xFFFFFFFFu;
      ld[t] = 0xFFFFFFFFu;
    }
    // the next query's keys are written behind the barriers of its sums
  }
}

template <int UNITS>
void launch_first(const uint4* q, int nq, const uint4* cat, long long ncat, const HammingOrder& order, int part, int k,
                  uint32_t* li, uint32_t* ld, uint32_t* kth, int num_sms, cudaStream_t st) {
  if (nq >= 8 * num_sms)
    hamming_first_kernel<UNITS, 2><<<(nq + 1) / 2, kHSelThreads, 0, st>>>(q, nq, cat, ncat, order, part, k, li, ld, kth);
  else
    hamming_first_kernel<UNITS, 1><<<nq, kHSelThreads, 0, st>>>(q, nq, cat, ncat, order, part, k, li, ld, kth);
}

// One block per query: the k smallest (distance, index) keys of its list and its
// candidates of part `part_i`, written back to the list (sorted) with the k-th of them to
// `kth`; the candidate count is cleared for the next part.  A histogram of the distances
// gives the k-th one, D; only the keys up to D are sorted.  Overflowed candidates: the part
// is scanned twice, for the histogram and for the keys under (and, the first ones, at) D.
__global__ void __launch_bounds__(kHSelThreads)
    hamming_select_kernel(const uint4* __restrict__ q, const uint4* __restrict__ cat, long long ncat,
                          const __grid_constant__ HammingOrder order, int part_i, int k, uint32_t* __restrict__ cnt,
                          const uint32_t* __restrict__ cand, uint32_t* __restrict__ list_idx,
                          uint32_t* __restrict__ list_dist, uint32_t* __restrict__ kth) {
  __shared__ unsigned long long keys[kHCap + 64], out[kHCap + 64];
  __shared__ uint32_t hist[129];
  __shared__ int s_d, s_need, s_low, s_scan[kHSelThreads / 32];
  const int qi = blockIdx.x, t = threadIdx.x;
  const long long places = (long long)order.part_units(part_i) * HammingOrder::kUnit;
  const uint32_t n = cnt[qi];
  if (n == 0) return;  // nothing in the part comes before the k-th entry
  for (int i = t; i < 129; i += kHSelThreads) hist[i] = 0;
  if (t == 0) s_low = 0;
  __syncthreads();
  if (t == 0) cnt[qi] = 0;
  const uint4 qc = q[qi];
  uint32_t* li = list_idx + (size_t)qi * k;
  uint32_t* ld = list_dist + (size_t)qi * k;
  auto key_of = [](uint32_t d, uint32_t i) { return ((unsigned long long)d << 32) | i; };
  // the code at a place of the part; ncat or more: none (the catalog's last unit may be short)
  auto code_at = [&](uint32_t place) {
    return (long long)order.unit(part_i, place / HammingOrder::kUnit) * HammingOrder::kUnit + place % HammingOrder::kUnit;
  };
  const bool gathered = n <= (uint32_t)kHCap;
  for (int i = t; i < k; i += kHSelThreads) {
    keys[i] = key_of(ld[i], li[i]);
    atomicAdd(&hist[ld[i]], 1u);
  }
  if (gathered) {
    for (int i = t; i < (int)n; i += kHSelThreads) {
      const long long c = code_at(cand[(size_t)qi * kHCap + i]);
      if (c < ncat) {
        const uint32_t d = ham4(qc, cat[c]);
        keys[k + i] = key_of(d, (uint32_t)c);
        atomicAdd(&hist[d], 1u);
      } else {
        keys[k + i] = ~0ull;
      }
    }
  } else {
    for (long long p = t; p < places; p += kHSelThreads) {
      const long long c = code_at((uint32_t)p);
      if (c < ncat) atomicAdd(&hist[ham4(qc, cat[c])], 1u);
    }
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
    for (int i = t; i < k + (int)n; i += kHSelThreads)
      if ((uint32_t)(keys[i] >> 32) <= D) out[atomicAdd(&s_low, 1)] = keys[i];
    __syncthreads();
    total = s_low;
  } else {
    // keys under D in any order at [0, k - need), then the list's keys at D, then the part's
    // first `need` at D (its places are in index order): at most 2 k
    const int need = s_need;
    for (int i = t; i < k; i += kHSelThreads)
      if ((uint32_t)(keys[i] >> 32) < D) out[atomicAdd(&s_low, 1)] = keys[i];
    int tied = 0;
    for (int i = 0; i < k; ++i)
      if ((uint32_t)(keys[i] >> 32) == D) {
        if (t == 0) out[k - need + tied] = keys[i];
        ++tied;
      }
    int at = 0;  // the part's codes at D so far
    for (long long p0 = 0; p0 < places; p0 += kHSelThreads) {
      const long long p = p0 + t, c = p < places ? code_at((uint32_t)p) : ncat;
      const uint32_t d = c < ncat ? ham4(qc, cat[c]) : 0xFFFFFFFFu;
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
      if (d == D && pos < need) out[k - need + tied + pos] = key_of(D, (uint32_t)c);
      __syncthreads();
    }
    total = k - need + tied + min(at, need);
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
  for (int i = t; i < k; i += kHSelThreads) {
    li[i] = (uint32_t)dst[i];
    ld[i] = (uint32_t)(dst[i] >> 32);
  }
  if (t == 0) kth[qi] = pack_kth((uint32_t)(dst[k - 1] >> 32), (uint32_t)dst[k - 1]);
}

size_t query_tiles(int nq) { return ((size_t)nq + kHM - 1) / kHM; }

}  // namespace

// Device scratch for a query block (the queries are taken `block` at a time).
size_t topk_scratch(int nq, int block) {
  const size_t b = (size_t)std::min(nq, block);
  return query_tiles((int)b) * kHABytes + 2 * b * 4 + b * kHCap * 4 + 4 * 256;
}

// 2M codes x 4096 queries x 64: 1.63 ms (11.9 as a popcount scan with per-chunk lists merged
// at the end), 2.2 in scenes of 20,000 near codes; 65536 x 512: 80 us (742); 16384 x 64: 34 us
// (301); 4096 x 1: 17 us (304).
cudaError_t launch_topk(const uint64_t* q, int nq, const uint64_t* cat, long long ncat, int k, int block,
                        uint8_t* scratch, uint32_t* out_idx, uint32_t* out_dist, int num_sms, uint32_t* err,
                        uint64_t* launches, cudaStream_t st) {
  cudaError_t e = ensure_smem_attr((const void*)hamming_tc_kernel, kHSmTotal);
  if (e != cudaSuccess) return e;
  const HammingOrder order((uint64_t)ncat, (uint32_t)std::min(nq, block), (uint32_t)k, num_sms);
  for (int q0 = 0; q0 < nq; q0 += block) {
    const int n = std::min(block, nq - q0), tiles = (int)query_tiles(n);
    uint8_t* image = scratch;
    uint32_t* cnt = reinterpret_cast<uint32_t*>(scratch + align_up((size_t)tiles * kHABytes, 256));
    uint32_t* kth = cnt + align_up((size_t)n, 64);
    uint32_t* cand = kth + align_up((size_t)n, 64);
    const uint64_t* qb = q + 2 * (size_t)q0;
    uint32_t *li = out_idx + (size_t)q0 * k, *ld = out_dist + (size_t)q0 * k;
    int part = order.sets - 1;
    auto* const first =
        order.first == HammingOrder::kFirst[0] ? launch_first<HammingOrder::kFirst[0]> : launch_first<HammingOrder::kFirst[1]>;
    first((const uint4*)qb, n, (const uint4*)cat, ncat, order, part, k, li, ld, kth, num_sms, st);
    ++*launches;
    if (part == 0) continue;
    hamming_expand_queries_kernel<<<(tiles * kHM * 8 + 255) / 256, 256, 0, st>>>((const uint16_t*)qb, n, tiles, image,
                                                                               cnt);
    ++*launches;
    while (--part >= 0) {
      const long long places = (long long)order.part_units(part) * HammingOrder::kUnit;
      const long long blocks = (places + kHSuper - 1) / kHSuper;
      const int share = blocks < num_sms ? std::min(tiles, (int)(num_sms / blocks)) : 1;
      hamming_tc_kernel<<<dim3((unsigned)std::min<long long>(blocks, num_sms), share), kHThreads, kHSmTotal, st>>>(
          image, tiles, n, (const uint4*)cat, ncat, order, part, places, kth, cnt, cand, err);
      hamming_select_kernel<<<n, kHSelThreads, 0, st>>>((const uint4*)qb, (const uint4*)cat, ncat, order, part, k, cnt,
                                                        cand, li, ld, kth);
      *launches += 2;
    }
  }
  return cudaGetLastError();
}

}  // namespace psift
