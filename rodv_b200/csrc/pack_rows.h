// pack_rows.h -- host conversion of bases and qualities to the packed layout
// (layout.h): base codes and row words.
//
// A read of n bases becomes n row words of 4 bytes, padded with zero words to a
// multiple of four.  The words are written once and read next by the copy
// engine, so the SSE2 form writes those of a large batch past the caches
// (streaming stores): out of lines that many cores had just written, the upload
// of an 8 MB batch ran at 7 GB/s (1.1 ms; 35 GB/s, 0.23 ms, with these).  A
// batch below kStreamBytes is written by one or a few cores and uploads as fast
// from the caches.  The scalar form is the same function for other hosts and
// for a read's last bases.
#pragma once
#include <cstdint>
#include <cstring>

#include "layout.h"

#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace rodv {

constexpr uint64_t kStreamBytes = 1u << 20;

// A0 C1 G2 T3 N4; 0xff marks a base outside the engine's domain.
struct CodeTable {
  uint8_t v[256];
  CodeTable() {
    std::memset(v, 0xff, sizeof(v));
    v['A'] = kA; v['C'] = kC; v['G'] = kG; v['T'] = kT; v['N'] = kN;
  }
};
inline const CodeTable& code_table() {
  static const CodeTable t;
  return t;
}

// One base's code; *bad takes a base outside the domain (else unchanged).
inline uint8_t base_code(uint8_t base, int* bad) {
  const uint8_t c = code_table().v[base];
  if (c == 0xff) *bad = (int)base;
  return c;
}

// The four quality arrays of a read.  Uniform reads' ins, del and gcp are those
// of the first base.
struct ReadQuals {
  const uint8_t *q, *ins, *del, *gcp;
};

inline void pack_rows_scalar(const uint8_t* base, const ReadQuals& z, uint32_t k, uint32_t n,
                             bool uniform, uint32_t* dst, int* bad) {
  for (; k < n; ++k) {
    const uint32_t j = uniform ? 0 : k;
    dst[k] = row_word(base_code(base[k], bad), z.q[k], z.ins[j], z.del[j], z.gcp[j]);
  }
  for (; k < ((n + 3) & ~3u); ++k) dst[k] = 0;
}

#if defined(__SSE2__)
// Codes of 16 bases: bits 1-2 of A, C, T, G count 0, 1, 2, 3, x ^ (x >> 1) swaps
// the last two.  *ok: bytes 0xff where the base is one of A, C, G, T, N.
inline __m128i codes16(__m128i c, __m128i* ok) {
  auto is = [&](char l) { return _mm_cmpeq_epi8(c, _mm_set1_epi8(l)); };
  const __m128i three = _mm_set1_epi8(3);
  const __m128i x = _mm_and_si128(_mm_srli_epi16(c, 1), three);
  const __m128i code = _mm_xor_si128(x, _mm_and_si128(_mm_srli_epi16(x, 1), three));
  const __m128i n = is('N');
  *ok = _mm_or_si128(_mm_or_si128(_mm_or_si128(is('A'), is('C')), _mm_or_si128(is('G'), is('T'))),
                     n);
  return _mm_or_si128(_mm_andnot_si128(n, code), _mm_and_si128(n, _mm_set1_epi8(kN)));
}
#endif

// Whether all n bases are A, C, G, T or N.
inline bool bases_valid(const uint8_t* base, uint32_t n) {
  uint32_t k = 0;
#if defined(__SSE2__)
  for (; k + 16 <= n; k += 16) {
    __m128i ok;
    codes16(_mm_loadu_si128(reinterpret_cast<const __m128i*>(base + k)), &ok);
    if (_mm_movemask_epi8(ok) != 0xffff) return false;
  }
#endif
  for (; k < n; ++k)
    if (code_table().v[base[k]] == 0xff) return false;
  return true;
}

// Row words of a read of n bases to dst (16-byte aligned, n rounded up to a
// multiple of four words); stream: with streaming stores (then pack_fence).
inline void pack_rows(const uint8_t* base, const ReadQuals& z, uint32_t n, bool uniform,
                      bool stream, uint32_t* dst, int* bad) {
  uint32_t k = 0;
#if defined(__SSE2__)
  const __m128i zero = _mm_setzero_si128(), low7 = _mm_set1_epi8(127);
  auto load = [&](const uint8_t* p) {
    return _mm_loadu_si128(reinterpret_cast<const __m128i*>(p));
  };
  const uint32_t gaps = uniform ? row_word(0, 0, z.ins[0], z.del[0], z.gcp[0]) : 0;
  const __m128i gap16[2] = {_mm_set1_epi16((short)(gaps & 0xffff)),
                            _mm_set1_epi16((short)(gaps >> 16))};
  for (; k + 16 <= n; k += 16) {
    __m128i ok;
    const __m128i code = codes16(load(base + k), &ok);
    if (_mm_movemask_epi8(ok) != 0xffff) break;  // the scalar form names the base
    const __m128i q = _mm_and_si128(load(z.q + k), low7);
    __m128i ins = zero, del = zero, gcp = zero;
    if (!uniform) {
      ins = _mm_and_si128(load(z.ins + k), low7);
      del = _mm_and_si128(load(z.del + k), low7);
      gcp = _mm_and_si128(load(z.gcp + k), low7);
    }
    for (int h = 0; h < 2; ++h) {  // 8 bases: the words' low and high halves
      auto wide = [&](__m128i v) {
        return h ? _mm_unpackhi_epi8(v, zero) : _mm_unpacklo_epi8(v, zero);
      };
      __m128i lo = _mm_or_si128(wide(code), _mm_slli_epi16(wide(q), 3)), hi;
      if (uniform) {
        lo = _mm_or_si128(lo, gap16[0]);
        hi = gap16[1];
      } else {
        const __m128i i16 = wide(ins);
        lo = _mm_or_si128(lo, _mm_slli_epi16(i16, 10));
        hi = _mm_or_si128(_mm_srli_epi16(i16, 6),
                          _mm_or_si128(_mm_slli_epi16(wide(del), 1), _mm_slli_epi16(wide(gcp), 8)));
      }
      __m128i* out = reinterpret_cast<__m128i*>(dst + k + 8 * h);
      const __m128i w0 = _mm_unpacklo_epi16(lo, hi), w1 = _mm_unpackhi_epi16(lo, hi);
      if (stream) {
        _mm_stream_si128(out, w0);
        _mm_stream_si128(out + 1, w1);
      } else {
        _mm_store_si128(out, w0);
        _mm_store_si128(out + 1, w1);
      }
    }
  }
#endif
  pack_rows_scalar(base, z, k, n, uniform, dst, bad);
}

// Codes of n haplotype bases.
inline void pack_codes(const uint8_t* base, uint32_t n, uint8_t* dst, int* bad) {
  uint32_t k = 0;
#if defined(__SSE2__)
  for (; k + 16 <= n; k += 16) {
    __m128i ok;
    const __m128i code =
        codes16(_mm_loadu_si128(reinterpret_cast<const __m128i*>(base + k)), &ok);
    if (_mm_movemask_epi8(ok) != 0xffff) break;
    _mm_storeu_si128(reinterpret_cast<__m128i*>(dst + k), code);
  }
#endif
  for (; k < n; ++k) dst[k] = base_code(base[k], bad);
}

// Ends a thread's streaming stores: they are visible to whoever the thread
// signals next.
inline void pack_fence() {
#if defined(__SSE2__)
  _mm_sfence();
#endif
}

}  // namespace rodv
