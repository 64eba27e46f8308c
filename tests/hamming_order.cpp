// hamming_order.cuh on the host, built by the tests:
//   hamming_order check SIZE...              the parts of catalogs of these sizes
//   hamming_order units SIZE QUERIES K SMS   the units of the last part
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "hamming_order.cuh"

using psift::HammingOrder;

static int check(const char* name, uint64_t codes, const HammingOrder& o) {
  const uint64_t units = (codes + 7) / 8;
  if (o.sets < 1 || o.sets > o.kMaxSets || o.step > o.kMaxStep || o.part_units(o.sets - 1) > o.first)
    return std::printf("%s: sets\n", name), 1;
  // more than one set: the first part has 64 codes or more whatever a short unit lacks
  if (o.sets > 1 && o.part_units(o.sets - 1) < o.kLeast) return std::printf("%s: first part\n", name), 1;
  uint64_t total = 0;
  std::vector<char> seen(units < (1u << 20) ? units : 0, 0);
  for (int i = o.sets - 1; i >= 0; --i) {
    const uint32_t n = o.part_units(i);
    if (i + 1 < o.sets && n > (o.step - 1ull) * o.size[i + 1]) return std::printf("%s: part %d\n", name, i), 1;
    total += n;
    uint64_t last = 0;
    const uint32_t step = seen.empty() ? n / 5000 + 1 : 1;  // of a huge catalog: some places
    for (uint64_t t = 0; t < n; t += step) {
      const uint64_t u = o.unit(i, (uint32_t)t);
      if (u >= units || (t && u <= last))
        return std::printf("%s: part %d place %llu\n", name, i, (unsigned long long)t), 1;
      last = u;
      if (!seen.empty() && seen[u]++) return std::printf("%s: unit %llu twice\n", name, (unsigned long long)u), 1;
    }
    if (n && o.unit(i, n - 1) >= units) return std::printf("%s: part %d end\n", name, i), 1;
  }
  if (total != units) return std::printf("%s: %llu units\n", name, (unsigned long long)total), 1;
  return 0;
}

int main(int argc, char** argv) {
  if (!std::strcmp(argv[1], "units")) {
    const HammingOrder o(std::strtoull(argv[2], nullptr, 10), std::atoi(argv[3]), std::atoi(argv[4]),
                         std::atoi(argv[5]));
    for (uint32_t t = 0; t < o.part_units(0); ++t) std::printf("%u\n", o.unit(0, t));
    return 0;
  }
  const uint32_t searches[][2] = {{1, 64}, {64, 1}, {512, 64}, {4096, 64}, {20000, 1}, {1u << 20, 64}};
  for (int a = 2; a < argc; ++a) {
    const uint64_t codes = std::strtoull(argv[a], nullptr, 10);
    for (auto& q : searches)
      if (check(argv[a], codes, HammingOrder(codes, q[0], q[1], 148))) return 1;
    for (int parts = 0; parts < HammingOrder::kMaxSets; ++parts)  // and every other choice
      for (uint32_t first : HammingOrder::kFirst) {
        const HammingOrder o((uint32_t)((codes + 7) / 8), first, parts);
        if (o.step <= o.kMaxStep && o.part_units(parts) >= o.kLeast && check(argv[a], codes, o)) return 1;
      }
  }
  return 0;
}
