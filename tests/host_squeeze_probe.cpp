// Both forms of the code squeezer on random bytes and every shift: the bytes out are the same (exit code 0).
#include <cstdio>
#include <cstdlib>

#include "qb_host_squeeze.hpp"

int main() {
  uint8_t src[32], a[16], b[16];
  std::srand(7);
  for (int round = 0; round < 2000; ++round) {
    for (uint8_t& v : src) v = uint8_t(std::rand() >> 3);
    for (int shift = 0; shift < 8; ++shift) {
      if (shift <= 4) {
        qb::squeeze4(src, shift, a); qb::plain::squeeze4(src, shift, b);
        if (std::memcmp(a, b, 16)) return std::printf("4 bits, shift %d\n", shift), 1;
      }
      if (shift <= 6) {
        qb::squeeze2(src, shift, a); qb::plain::squeeze2(src, shift, b);
        if (std::memcmp(a, b, 8)) return std::printf("2 bits, shift %d\n", shift), 1;
      }
      qb::squeeze1(src, shift, a); qb::plain::squeeze1(src, shift, b);
      if (std::memcmp(a, b, 4)) return std::printf("1 bit, shift %d\n", shift), 1;
      for (int i = 0; i < 32; ++i)
        if (((b[i / 8] >> (i % 8)) & 1) != ((src[i] >> shift) & 1)) return std::printf("plain, shift %d\n", shift), 1;
    }
  }
  return 0;
}
