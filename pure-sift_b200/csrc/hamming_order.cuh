// The order in which the Hamming shortlist (hamming_tc.cu) takes a catalog's codes.
//
// The shortlist compares a part of the catalog against each query's k-th entry so far, and
// what a part adds is about (its codes / codes before it) * k entries only if the codes
// before it are a fair sample.  Codes in catalog order are not: neighbours belong to one
// image or scene, and a scene near to a query comes all at once (2,000,000 codes in scenes
// of 20,000 x 4096 queries took 38.9 ms that way, 1.7 ms in random order; 2.2 and 1.6 like
// this).  So the parts are samples of the whole catalog, spread evenly and off any period:
// set 0 is all of the catalog's units (8 codes, one 128-byte line), set i + 1 holds one unit
// of every few consecutive ones of set i, picked by a hash; the smallest set is taken first,
// then, set by set, the units that the one before lacks.  Every part is in ascending code
// order.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <cmath>

#ifdef __CUDACC__
#define PSIFT_HD __host__ __device__ __forceinline__
#else
#define PSIFT_HD inline
#endif

namespace psift {

struct HammingOrder {
  static constexpr int kUnit = 8;               // codes per unit
  static constexpr uint32_t kMaxStep = 8;       // a query's candidates of a part: about 7 k of the 2048 kept
  static constexpr uint32_t kFirst[2] = {256, 1024};  // the last set's most units
  static constexpr uint32_t kLeast = 16;        // units before any other part: k <= 64 codes are listed by then
  static constexpr int kMaxSets = 9;            // 2^29 units / 8^7 = 256
  uint32_t size[kMaxSets];                      // units per set
  uint32_t step;                                // units of a set per unit of the next
  int sets;
  uint32_t first;                               // the smallest set's most units, of kFirst

  // For a search of `queries` x `k` on `sms` SMs: the first part and the number of further
  // ones with the least estimated time (see part_us).  Against all choices timed on random
  // codes, 4096 to 4 M x 1 to 16384 queries, its choice costs 0.3 % on average, 8 % at most;
  // e.g. 2 M x 4096 x 64 1636 us as 4 parts of step 4, 1732 as 3 of 7, 1676 as 5 of 4.
  HammingOrder(uint64_t codes, uint32_t queries, uint32_t k, int sms) : step(2), sets(1), first(kFirst[0]) {
    size[0] = (uint32_t)((codes + kUnit - 1) / kUnit);
    double best = 1e300;
    for (int f = 0; f < 2; ++f) {
      for (int parts = 0; parts < kMaxSets; ++parts) {
        HammingOrder o(size[0], kFirst[f], parts);
        if (o.step > kMaxStep || (parts > 0 && o.part_units(parts) < kLeast)) continue;
        double us = f ? 24 + 0.0156 * queries : 15 + 0.0094 * queries;
        for (int i = 0; i < parts; ++i) us += o.part_us(i, queries, k, sms);
        if (us < best) best = us, *this = o;
      }
    }
  }

  static uint64_t reach(uint64_t first, uint64_t step, int parts) {
    for (int i = 0; i < parts; ++i) first *= step;
    return first;
  }

  // `parts` further parts of a catalog's units, in the smallest step for that many.
  HammingOrder(uint32_t units, uint32_t first_units, int parts) : step(2), sets(parts + 1), first(first_units) {
    for (int i = 0; i < kMaxSets; ++i) size[i] = 0;
    size[0] = units;
    while (step <= kMaxStep && reach(first, step, parts) < units) ++step;
    for (int i = 1; i < sets; ++i) size[i] = (size[i - 1] + step - 1) / step;
  }

  // Estimated microseconds of part i: its two launches, and rounds of a block of 512 codes
  // against a CTA's query tiles, 1.06 us a tile (3.7 at least, to expand the codes), more by
  // the share of a warp's 32 x 64 products that hold candidates and by how many they hold.
  double part_us(int i, uint32_t queries, uint32_t k, int sms) const {
    const double codes = (double)kUnit * part_units(i), hits = (step - 1.0) * k * 2048 / (codes + 1);
    const long long blocks = ((long long)codes + 511) / 512, tiles = (queries + 127) / 128;
    const long long share = blocks < sms ? std::min(tiles, sms / std::max(blocks, 1LL)) : 1;
    const long long rounds = (blocks + sms - 1) / sms, turn = (tiles + share - 1) / share;
    return 12.5 + 0.006 * queries + rounds * std::max(3.7, turn * 1.06 * (1 + 1.5 * (1 - std::exp(-hits)) + 0.12 * hits));
  }

  // Units of a part: set `i`, without those of set i + 1 if there is one.
  PSIFT_HD uint32_t part_units(int i) const { return i + 1 < sets ? size[i] - size[i + 1] : size[i]; }

  // Which unit of group g (`step` consecutive ones) of set i is in set i + 1.
  PSIFT_HD uint32_t pick(int i, uint32_t g) const {
    const uint32_t left = size[i] - g * step, m = left < step ? left : step;
    uint32_t x = (g + 1u) * 0x9E3779B1u + (uint32_t)i * 0x85EBCA6Bu;
    x ^= x >> 15;
    x *= 0x2C1B3C6Du;
    x ^= x >> 12;
    return (uint32_t)(((uint64_t)x * m) >> 32);
  }

  // The catalog unit at place t < part_units(i) of part i.
  PSIFT_HD uint32_t unit(int i, uint32_t t) const {
    uint32_t e = t;
    if (i + 1 < sets) {
      const uint32_t g = t / (step - 1), r = t - g * (step - 1);
      e = g * step + r + (r >= pick(i, g) ? 1u : 0u);
    }
    for (int j = i - 1; j >= 0; --j) e = e * step + pick(j, e);
    return e;
  }
};

}  // namespace psift
