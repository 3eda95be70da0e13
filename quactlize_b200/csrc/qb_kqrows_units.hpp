// Index arithmetic of the several-row raw-block kernel (qb_gemv_kqrows.cu): which (expert, eight-row group, tile) units a launch
// has and how they are cut over the clusters, and which 16-byte units a row's copy takes.  Plain C++ as well as device code, so
// that a host test walks it for offsets that no launch may be given and for the ends of a tensor.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define QB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define QB_HOST_DEVICE inline
#endif

namespace qb {

constexpr int kKrCols = 8;                         // activation rows of a group
constexpr long long kKrMaxUnits = 1ll << 29;       // units of a launch, checked on the host: their numbers stay ints

// An offset as the kernel uses it: inside [0, rows] and never below the one before it, whatever memory holds.  The experts then
// share out at most `rows` rows, which is what kr_most_groups() counts on.
QB_HOST_DEVICE int kr_settle(int before, int raw, int rows) {
  int const v = raw < 0 ? 0 : raw > rows ? rows : raw;
  return v > before ? v : before;
}
QB_HOST_DEVICE int kr_groups(int rows) { return (rows + kKrCols - 1) / kKrCols; }
// Groups that `rows` rows dealt to `experts` experts make at most: one a row, and one a full eight plus one an expert.
QB_HOST_DEVICE int kr_most_groups(int rows, int experts) {
  long long const v = (long long)(rows / kKrCols) + experts;
  return v < rows ? int(v) : rows;
}
// First unit of share `part` out of `parts`.
QB_HOST_DEVICE int kr_cut(long long units, unsigned part, unsigned parts) { return int(units * part / parts); }

// The bulk copy of `len` bytes at address `b` that may start off a 16-byte boundary: the units from `first` on, those that reach
// outside the tensor [lo, hi) left out.  The bytes of the segment in a unit left out, [b, from) and [to, b + len), are copied
// one by one.  len is at least 32, so from <= to.
struct KrSpan { uintptr_t first, from, to; };
QB_HOST_DEVICE KrSpan kr_span(uintptr_t b, unsigned len, uintptr_t lo, uintptr_t hi) {
  KrSpan s;
  s.first = b & ~uintptr_t(15);
  s.from = s.first < lo ? s.first + 16 : s.first;
  s.to = (b + len + 15) & ~uintptr_t(15);
  if (s.to > hi) s.to -= 16;
  return s;
}

}  // namespace qb
