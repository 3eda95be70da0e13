// Walks the unit arithmetic of the several-row raw-block kernel for offsets read from standard input:
//   rows experts tiles parts offset_0 .. offset_experts        -> "groups most" on success, a message and exit code 1 otherwise
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "qb_kqrows_units.hpp"

static int fail(char const* what, long long v) { std::printf("%s: %lld\n", what, v); return 1; }

int main() {
  int rows, experts, tiles, parts;
  if (std::scanf("%d %d %d %d", &rows, &experts, &tiles, &parts) != 4) return 2;
  std::vector<int> off(experts + 1), cum(experts);
  int top = 0, groups = 0;
  for (int& o : off) {
    if (std::scanf("%d", &o) != 1) return 2;
    o = qb::kr_settle(top, o, rows);
    if (o < top || o > rows) return fail("offset below the one before it or beyond the rows", o);
    top = o;
  }
  for (int e = 0; e < experts; ++e) cum[e] = groups += qb::kr_groups(off[e + 1] - off[e]);
  int const most = qb::kr_most_groups(rows, experts);
  if (groups > most) return fail("more groups than the host counted on", groups);
  if ((long long)most * tiles > qb::kKrMaxUnits) return fail("declined on the host", most);
  long long const units = (long long)groups * tiles;
  int last = 0;
  for (int p = 0; p < parts; ++p) {
    int const u = qb::kr_cut(units, p, parts), end = qb::kr_cut(units, p + 1, parts);
    if (u != last || end < u || end > units) return fail("bad share", u);
    last = end;
    if (u == end) continue;
    int const first = u / tiles, final = (end - 1) / tiles;     // the share's first and last group: whose rows are they?
    for (int gi : {first, final}) {
      int e = 0;
      while (e < experts && cum[e] <= gi) ++e;
      if (e == experts) return fail("group beyond the experts", gi);
      int const row = off[e] + (gi - (e ? cum[e - 1] : 0)) * qb::kKrCols;
      if (row < 0 || row >= off[e + 1]) return fail("row outside its expert", row);
    }
  }
  if (last != units) return fail("units left over", units - last);
  std::printf("%d %d\n", groups, most);
  return 0;
}
