// Index arithmetic of the several-row raw-block kernel (qb_gemv_kqrows.cu): which (expert, eight-row group, tile) units a launch
// has and how they are cut over the clusters.  Plain C++ as well as device code, so that a host test walks it for offsets that
// no launch may be given.
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

}  // namespace qb
