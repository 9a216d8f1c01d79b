// The number of tiles that a move between the orders takes, in closed form, against
// the tiles themselves; and that these hold every state once.
#include <cstdio>
#include <vector>

#include "../../manybody_gb300/csrc/mb_internal.h"

int main() {
  int bad = 0;
  for (int L = 1; L <= 12; ++L)
    for (int nu = 0; nu <= L; ++nu)
      for (int nd = 0; nd <= L; ++nd) {
        const mb::SpinSector up = mb::make_spin_sector(L, nu), dn = mb::make_spin_sector(L, nd);
        for (int slots : {37, 64, 512, 1016}) {
          const mb::OrderTiles t = mb::order_tiles(L, up, dn, slots);
          int64_t states = 0;
          for (const mb::OrderTile& x : t.tiles) states += (int64_t)x.n_rows * x.n_cols * x.k;
          if (states != up.D * dn.D || (int64_t)t.tiles.size() != mb::order_tile_count(L, nu, nd, slots)) {
            std::printf("%d sites %d+%d, %d slots: %zu tiles, %lld states\n", L, nu, nd, slots,
                        t.tiles.size(), (long long)states);
            ++bad;
          }
        }
      }
  return bad ? 1 : 0;
}
