// The room that a projector of n sinograms makes in the column walk's queue of
// bins covers what a pass over any shard of them may queue for a LOR.
#include <algorithm>
#include <cstdio>
#include "internal.h"

int main() {
  for (int whole = 1; whole <= apirl::kColWindow + 1; whole++)
    for (int shard = 1; shard <= whole; shard++)
      if (std::min(apirl::col_direct(shard), shard) > apirl::col_direct_room(whole)) {
        printf("a shard of %d of %d sinograms: %d bins a LOR, room %d\n", shard, whole,
               std::min(apirl::col_direct(shard), shard), apirl::col_direct_room(whole));
        return 1;
      }
  return 0;
}
