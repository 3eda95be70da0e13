// 32 code bytes, shifted and masked, squeezed to 4, 2 or 1 bits a code: element i of the run is bits [i*B, i*B + B) of the output,
// little-endian.  Two forms with the same bytes out: plain C++ for any host, and SSE2 (part of every x86-64), which packs a
// 14336 x 4096 Q4_K matrix in 10 ms on one thread where a code at a time took 66.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace qb {

namespace plain {
template <int B>
inline void squeeze(uint8_t const* src, int shift, uint8_t* dst) {
  for (int i = 0; i < 4 * B; ++i) {
    unsigned v = 0;
    for (int j = 0; j < 8 / B; ++j) v |= ((unsigned(src[i * (8 / B) + j]) >> shift) & ((1u << B) - 1u)) << (B * j);
    dst[i] = uint8_t(v);
  }
}
inline void squeeze4(uint8_t const* src, int shift, uint8_t* dst) { squeeze<4>(src, shift, dst); }   // 32 codes -> 16 bytes
inline void squeeze2(uint8_t const* src, int shift, uint8_t* dst) { squeeze<2>(src, shift, dst); }   // -> 8 bytes
inline void squeeze1(uint8_t const* src, int shift, uint8_t* dst) { squeeze<1>(src, shift, dst); }   // -> 4 bytes
}  // namespace plain

#if defined(__SSE2__)
namespace sse2 {
inline __m128i load16(uint8_t const* p) { return _mm_loadu_si128(reinterpret_cast<__m128i const*>(p)); }
inline __m128i pair4(__m128i v, int shift) {                              // 16-bit lanes: two 4-bit codes -> one byte
  v = _mm_srli_epi16(v, shift);
  return _mm_or_si128(_mm_and_si128(v, _mm_set1_epi16(0x0F)), _mm_and_si128(_mm_srli_epi16(v, 4), _mm_set1_epi16(0xF0)));
}
inline void squeeze4(uint8_t const* src, int shift, uint8_t* dst) {       // 32 codes of 4 bits -> 16 bytes
  _mm_storeu_si128(reinterpret_cast<__m128i*>(dst), _mm_packus_epi16(pair4(load16(src), shift), pair4(load16(src + 16), shift)));
}
inline __m128i quad2(__m128i v, int shift) {                              // 32-bit lanes: four 2-bit codes -> one byte
  v = _mm_and_si128(_mm_srli_epi32(v, shift), _mm_set1_epi8(3));
  v = _mm_or_si128(v, _mm_srli_epi32(v, 6));
  return _mm_and_si128(_mm_or_si128(v, _mm_srli_epi32(v, 12)), _mm_set1_epi32(0xFF));
}
inline void squeeze2(uint8_t const* src, int shift, uint8_t* dst) {       // 32 codes of 2 bits -> 8 bytes
  __m128i const w = _mm_packs_epi32(quad2(load16(src), shift), quad2(load16(src + 16), shift));
  _mm_storel_epi64(reinterpret_cast<__m128i*>(dst), _mm_packus_epi16(w, w));
}
inline void squeeze1(uint8_t const* src, int shift, uint8_t* dst) {       // 32 codes of 1 bit -> 4 bytes
  for (int i = 0; i < 2; ++i) {                                           // the bit moves to the top of its byte
    uint16_t const m = uint16_t(_mm_movemask_epi8(_mm_slli_epi16(load16(src + 16 * i), 7 - shift)));
    std::memcpy(dst + 2 * i, &m, 2);
  }
}
}  // namespace sse2
using namespace sse2;
#else
using namespace plain;
#endif

}  // namespace qb
