// Row split of the passes over tall matrices (csrc/tall.hpp); no GPU calls.
#include <cstdio>
#include <cstdlib>

#include "../../pcaone_b200/csrc/tall.hpp"

#define CHECK(cond)                                                                                      \
  do {                                                                                                   \
    if (!(cond)) {                                                                                       \
      std::fprintf(stderr, "line %d: %s (n = %lld, cap = %d)\n", __LINE__, #cond, (long long)n, cap);    \
      std::exit(1);                                                                                      \
    }                                                                                                    \
  } while (0)

int main() {
  const int64_t sizes[] = {1, 63, 64, 65, 511, 512, 513, 5003, 20000, 500000, int64_t(1) << 33};
  for (const int64_t n : sizes)
    for (int cap = 0; cap <= pg::kTallMaxParts; ++cap) {
      const int clusters = pg::tall_clusters(n, cap);
      CHECK(clusters >= 1 && clusters <= (cap < 1 ? 1 : cap));
      const int64_t ctas = (int64_t)clusters * pg::kTallCluster;
      CHECK(ctas * pg::tall_rows_per_cta(n, ctas) >= n);
    }
  return 0;
}
