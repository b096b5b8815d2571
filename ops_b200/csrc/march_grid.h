// How many rows a warp (or CTA) of a column march takes.
#pragma once
#include <algorithm>

namespace opsb {

// `columns` independent columns of n rows are cut into strips; a strip costs
// its rows and `halo` more that it reads for its neighbours. `resident` strips
// run at a time, so the time is that of ceil(strips / resident) waves: the
// strips that fill whole waves win, and of those the long ones. (CloverLeaf 2D
// at 3840^2 with strips of 64 rows ran 3.3 waves in the time of 4, the heat
// solver's 2048^2 direction kernel 1.4 waves in the time of 2.) At most
// `most` strips. The loop goes over the strip lengths, about 2 sqrt(n) of them:
// over every number of strips it took 0.2 ms of a solve on 5 x 40,000 cells.
inline int march_rows(long long columns, int n, int halo, long long resident, long long most = 1LL << 40) {
  int best = n;
  double cost = 1e300;
  for (int c = 1; c <= n;) {
    const int rows = (n + c - 1) / c;
    if (rows < 2 && n > 1) break;
    const long long strips = columns * ((n + rows - 1) / rows);
    if (strips > most && c > 1) break;
    const long long waves = (strips + resident - 1) / resident;
    if (waves > 16 && c > 1) break;
    const double t = (double)waves * (rows + halo);
    if (t < cost * 0.999) {
      cost = t;
      best = rows;
    }
    if (rows < 2) break;
    c = (n + rows - 2) / (rows - 1);  // the next number of strips that have fewer rows
  }
  return best;
}

}  // namespace opsb
