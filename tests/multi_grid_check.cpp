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
  for (int resident : {1, 296, 444, 888})
    for (int items = 1; items <= 4 * resident + 3; ++items) {
      const int b = even_blocks(resident, items);
      CHECK(b >= 1 && b <= resident && b <= items);
      const int full = resident < items ? resident : items;
      const int rounds = (items + full - 1) / full;
      // never more rounds than the full grid takes, and full above three
      CHECK((items + b - 1) / b == rounds || b == full);
      if (rounds == 1 || rounds > 3) CHECK(b == full);
    }
  CHECK(even_blocks(444, 540) == 270);
  for (int sms : {1, 148})
    for (int w : {2, 4}) {
      CHECK(takes_few((long)8 * sms / w * w, sms));
      CHECK(!takes_few(((long)8 * sms / w + 1) * w, sms));
    }
  if (!fails) printf("OK\n");
  return fails != 0;
}
