// Host check of which form of the sparse factor and solves a matrix takes (csrc/sparse.hpp): the side
// that was measured faster.
#include <cstdio>

#include "sparse.hpp"

static int failures = 0;
#define EXPECT(c) \
  do { \
    if (!(c)) { \
      ++failures; \
      std::printf("line %d: %s\n", __LINE__, #c); \
    } \
  } while (0)

int main() {
  using sov::factor_on_one_cta;
  using sov::solve_on_one_cta;
  // m rows in path blocks of b: b levels, an entry of L and an update term per row but a block's last
  auto factor = [](int m, int b) { return factor_on_one_cta(m, b, m - m / b); };
  auto solve = [](int m, int b) { return solve_on_one_cta(m, b, m - m / b); };
  for (int m : {500, 1000, 2000, 4000})
    for (int b : {4, 8, 16, 32}) EXPECT(factor(m, b) && solve(m, b));
  EXPECT(factor(4000, 1) && solve(4000, 1) && factor(4000, 2) && solve(4000, 2));
  // wide and shallow: the grid
  for (int m : {8000, 14000, 20000, 27000, 200000})
    for (int b : {1, 2}) EXPECT(!factor(m, b) && !solve(m, b));
  for (int m : {14000, 20000, 27000})
    for (int b : {4, 8, 16}) EXPECT(!factor(m, b));
  EXPECT(factor(8000, 8) && factor(20000, 32) && !factor(27000, 32));
  EXPECT(solve(8000, 8) && solve(14000, 8) && solve(20000, 32) && !solve(20000, 8) && !solve(27000, 16));
  // deep: by terms and entries
  EXPECT(factor_on_one_cta(16251, 64, 123845) && solve_on_one_cta(16251, 64, 44059));
  EXPECT(factor_on_one_cta(26001, 70, 198695) && solve_on_one_cta(26001, 70, 70585));
  EXPECT(!factor_on_one_cta(45501, 76, 347961) && !factor_on_one_cta(3600, 212, 1019338));
  EXPECT(factor_on_one_cta(2500, 171, 573704) && solve_on_one_cta(3600, 212, 55898));
  EXPECT(!solve_on_one_cta(3600, 10, 30001));
  // family solves: a CTA per LP but for many rows in few steps
  using sov::family_solve_on_one_cta;
  EXPECT(family_solve_on_one_cta(1800, 40) && family_solve_on_one_cta(2000, 2) && family_solve_on_one_cta(3600, 212));
  EXPECT(!family_solve_on_one_cta(6000, 8) && !family_solve_on_one_cta(6000, 1) && !family_solve_on_one_cta(14000, 8));
  std::printf("failures %d\n", failures);
  return failures != 0;
}
