// Checks the rules of multi_grid.h around their edges.
#include <cstdio>

#include "multi_grid.h"

using namespace rodv;

static int fails = 0;
#define CHECK(x)                               \
  do {                                         \
    if (!(x)) {                                \
      printf("line %d: %s\n", __LINE__, #x);   \
      ++fails;                                 \
    }                                          \
  } while (0)

int main() {
  for (int max_rounds : {1, 2, 3, 4}) {
    for (int resident : {1, 296, 444, 888})
      for (int items = 1; items <= 4 * resident + 3; ++items) {
        const int b = even_blocks(resident, items, max_rounds);
        CHECK(b >= 1 && b <= resident && b <= items);
        const int full = resident < items ? resident : items;
        const int rounds = (items + full - 1) / full;
        // never more rounds than the full grid takes, and full above max_rounds
        CHECK((items + b - 1) / b == rounds || b == full);
        if (rounds == 1 || rounds > max_rounds) CHECK(b == full);
      }
  }
  CHECK(even_blocks(444, 540, kEvenRoundsF32) == 270);
  // FP64: a block's warps hold all its items' passes, or the grid is full
  for (int w : {2, 4})
    for (int passes = 1; passes <= 9; ++passes) {
      const int r = even_rounds_f64(passes, w);
      CHECK(r >= 1 && (r == 1 || r * passes <= w));
    }
  CHECK(even_blocks(444, 460, even_rounds_f64(2, 4)) == 230);
  CHECK(even_blocks(444, 600, even_rounds_f64(8, 4)) == 444);
  CHECK(even_blocks(296, 300, even_rounds_f64(5, 4)) == 296);
  for (int sms : {1, 148})
    for (int w : {2, 4}) {
      CHECK(takes_few((long)8 * sms / w * w, sms));
      CHECK(!takes_few(((long)8 * sms / w + 1) * w, sms));
    }
  if (!fails) printf("OK\n");
  return fails != 0;
}
