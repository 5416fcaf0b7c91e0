// Host-side checks of the work list of the kernel for small batches (no GPU
// needed): every point once, no batch left whole where it alone would set the
// launch's time, whatever the number of batches, and the choice between the two
// kernels.  Built and run by tests/test_small_items.py against libfrpa.so; prints
// "ok" or the first failure.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "frpa_internal.cuh"

using frpa::Rho1WorkItem;

#define CHECK(cond, ...)       \
  do {                         \
    if (!(cond)) {             \
      std::printf("FAIL line %d: ", __LINE__); \
      std::printf(__VA_ARGS__); \
      std::printf("\n");       \
      return 1;                \
    }                          \
  } while (0)

static std::vector<Rho1WorkItem> plan(int n, int nc_lo, int nc_hi, int np_lo, int np_hi, std::mt19937 &rng) {
  std::vector<Rho1WorkItem> b;
  for (int i = 0; i < n; ++i) {
    const int nc = nc_lo + (int)(rng() % (nc_hi - nc_lo + 1)), np = np_lo + (int)(rng() % (np_hi - np_lo + 1));
    b.push_back(Rho1WorkItem{i, nc, np, 0, np, 0, 0, (int)(rng() >> 1), 0});
  }
  return b;
}

int main() {
  constexpr int SMS = 148;
  std::mt19937 rng(5);
  std::vector<Rho1WorkItem> items;
  // points covered once, in whole 32-point steps
  for (int n : {1, 7, 148, 592, 593, 2000})
    for (int T : {1, 4})
      for (int order = 0; order < 3; ++order) {
        std::vector<Rho1WorkItem> b = plan(n, 1, 120, 0, 400, rng);
        frpa::rho1_small_build_items(b, T, SMS, order, 2, &items);
        std::vector<int> parts(n, 0), points(n, 0);
        for (const Rho1WorkItem &w : items) {
          CHECK(w.pn >= 1 && w.p0 % 32 == 0 && (w.pn % 32 == 0 || w.p0 + w.pn == w.np), "part %d+%d of %d", w.p0, w.pn,
                w.np);
          ++parts[w.batch];
          points[w.batch] += w.pn;
        }
        for (const Rho1WorkItem &w : b) CHECK(points[w.batch] == w.np, "batch %d: %d of %d points", w.batch,
                                              points[w.batch], w.np);
        if ((int)items.size() <= 4 * SMS)
          for (size_t i = 1; i < items.size(); ++i)
            CHECK((long long)items[i - 1].nc * items[i - 1].nc * items[i - 1].pn >=
                      (long long)items[i].nc * items[i].nc * items[i].pn, "few items not largest first");
        frpa::rho1_small_build_items(b, T, SMS, order, 1, &items);
        CHECK(items.empty(), "switched off, but %zu items", items.size());
      }
  // one batch of many points among n ordinary ones: cut, below and above four rounds of SMs
  for (int n : {200, 591, 592, 593, 600, 1000, 3000})
    for (int top : {2000, 20000}) {
      std::vector<Rho1WorkItem> b = plan(n, 60, 120, 100, 150, rng);
      b[n / 3].nc = 120;
      b[n / 3].np = b[n / 3].pn = top;
      frpa::rho1_small_build_items(b, 1, SMS, 2, 2, &items);
      long long total = 0;
      int longest = 0;
      for (const Rho1WorkItem &w : items) {
        total += w.pn;
        longest = std::max(longest, w.pn);
      }
      // no item above an SM's mean share of the points by more than one step
      CHECK(longest <= std::max<long long>(160, total / SMS) + 32, "%d batches, one of %d points: an item of %d", n, top,
            longest);
    }
  // the choice: measured far on one side or the other
  frpa::rho1_small_build_items(plan(64, 40, 120, 100, 200, rng), 1, SMS, 2, 0, &items);
  CHECK(!items.empty(), "64 ordinary batches not taken");
  frpa::rho1_small_build_items(plan(2000, 64, 72, 250, 400, rng), 1, SMS, 2, 0, &items);
  CHECK(!items.empty(), "2,000 batches of many points not taken");
  frpa::rho1_small_build_items(plan(6000, 110, 120, 60, 64, rng), 1, SMS, 2, 0, &items);
  CHECK(items.empty(), "6,000 batches of 64 points taken");
  frpa::rho1_small_build_items(plan(600, 16, 24, 250, 400, rng), 4, SMS, 2, 0, &items);
  CHECK(items.empty(), "600 batches of few functions, four perturbations taken");
  std::printf("ok\n");
  return 0;
}
