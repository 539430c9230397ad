// Checks pack_rows / pack_codes (pack_rows.h): whatever form the host runs, a
// read's row words and a haplotype's codes are those of row_word and the code
// table, the padding words are 0, nothing past them is written, and a base
// outside A, C, G, T, N is reported wherever it stands.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "pack_rows.h"

using namespace rodv;

static int fails = 0;
#define CHECK(x)                                            \
  do {                                                      \
    if (!(x)) {                                             \
      printf("line %d: %s\n", __LINE__, #x);                \
      if (++fails > 5) exit(1);                             \
    }                                                       \
  } while (0)

static uint32_t code_of(uint8_t c) {
  switch (c) {
    case 'A': return kA;
    case 'C': return kC;
    case 'G': return kG;
    case 'T': return kT;
    default: return kN;
  }
}

int main() {
  std::mt19937 rng(5);
  for (uint32_t n = 1; n <= 131; ++n)
    for (int uniform = 0; uniform < 2; ++uniform)
      for (int shift = 0; shift < 3; ++shift) {  // unaligned inputs
        std::vector<uint8_t> f[5];
        for (auto& v : f) v.resize(n + 3);
        uint8_t* p[5];
        for (int k = 0; k < 5; ++k) p[k] = f[k].data() + shift;
        for (uint32_t k = 0; k < n; ++k) {
          p[0][k] = (uint8_t) "ACGTN"[rng() % 5];
          for (int q = 1; q < 5; ++q) p[q][k] = (uint8_t)rng();  // the high bit is masked
          if (uniform && k)
            for (int q = 2; q < 5; ++q) p[q][k] = p[q][0];
        }
        const ReadQuals z{p[1], p[2], p[3], p[4]};
        const uint32_t padded = (n + 3) & ~3u;
        uint32_t* dst = static_cast<uint32_t*>(aligned_alloc(16, 4 * (padded + 4)));
        for (uint32_t k = 0; k < padded + 4; ++k) dst[k] = 0xdeadbeef;
        int bad = -1;
        pack_rows(p[0], z, n, uniform != 0, shift == 1, dst, &bad);
        pack_fence();
        CHECK(bad == -1);
        for (uint32_t k = 0; k < n; ++k)
          CHECK(dst[k] == row_word(code_of(p[0][k]), p[1][k], p[2][k], p[3][k], p[4][k]));
        for (uint32_t k = n; k < padded; ++k) CHECK(dst[k] == 0);
        for (uint32_t k = padded; k < padded + 4; ++k) CHECK(dst[k] == 0xdeadbeef);
        std::vector<uint8_t> codes(n + 4, 77);
        pack_codes(p[0], n, codes.data() + 1, &bad);
        CHECK(bad == -1 && codes[0] == 77 && codes[n + 1] == 77);
        for (uint32_t k = 0; k < n; ++k) CHECK(codes[k + 1] == code_of(p[0][k]));
        // one base outside the domain, anywhere
        const uint32_t at = rng() % n;
        int other;
        do other = (int)(rng() & 255);
        while (code_table().v[other] != 0xff);
        p[0][at] = (uint8_t)other;
        bad = -1;
        pack_rows(p[0], z, n, uniform != 0, shift == 1, dst, &bad);
        CHECK(bad == other);
        bad = -1;
        pack_codes(p[0], n, codes.data() + 1, &bad);
        CHECK(bad == other);
        CHECK(!bases_valid(p[0], n) && bases_valid(p[0], at) &&
              bases_valid(p[0] + at + 1, n - at - 1));
        free(dst);
      }
  for (int c = 0; c < 256; ++c)  // every byte value through the 16-base form
  {
    std::vector<uint8_t> s(16, 'A'), codes(16);
    s[c & 15] = (uint8_t)c;
    int bad = -1;
    pack_codes(s.data(), 16, codes.data(), &bad);
    CHECK(bases_valid(s.data(), 16) == (bad == -1));
    const bool in = c == 'A' || c == 'C' || c == 'G' || c == 'T' || c == 'N';
    CHECK((bad == -1) == in);
    if (in) CHECK(codes[c & 15] == code_of((uint8_t)c));
  }
  if (!fails) printf("OK\n");
  return fails != 0;
}
