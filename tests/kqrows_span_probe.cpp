// Walks kr_span over every segment of a tensor: standard input holds  base bytes row_bytes segment_bytes  -- the copies must stay
// inside the tensor, cover the segment and stay below the pitch the kernel gives a row.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "qb_kqrows_units.hpp"

static int fail(char const* what, unsigned long long v) { std::printf("%s: %llu\n", what, v); return 1; }

int main() {
  unsigned long long base, bytes, row, seg, single = 0;
  if (std::scanf("%llu %llu %llu %llu", &base, &bytes, &row, &seg) != 4) return 2;
  for (unsigned long long r = 0; r < bytes; r += row)
    for (unsigned long long o = 0; o < row; o += seg) {
      uintptr_t const b = base + r + o;
      unsigned const len = unsigned(seg < row - o ? seg : row - o);
      qb::KrSpan const s = qb::kr_span(b, len, base, base + bytes);
      if (s.first > b || b - s.first > 15 || s.first % 16) return fail("destination", b);
      if (s.from % 16 || s.to % 16 || s.from > s.to) return fail("not whole units", b);
      if (s.from < base || s.to > base + bytes) return fail("outside the tensor", b);
      std::vector<char> got(len);
      for (uintptr_t p = s.from; p < s.to; ++p)
        if (p >= b && p < b + len) got[p - b] = 1;
      for (uintptr_t p = b; p < s.from; ++p) { ++got[p - b]; ++single; }
      for (uintptr_t p = s.to; p < b + len; ++p) { ++got[p - b]; ++single; }
      for (char c : got)
        if (c != 1) return fail("byte missing or copied twice", b);
    }
  std::printf("%llu\n", single);
  return 0;
}
