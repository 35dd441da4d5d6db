// Rules of the library that show in times only: a batch's item shapes.  One section per argument; prints
// "ok" or what differs.
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "batch.cu"

using namespace atc;

#define REQUIRE(cond)                                   \
  do {                                                  \
    if (!(cond)) {                                      \
      std::printf("line %d: %s\n", __LINE__, #cond);    \
      return 1;                                         \
    }                                                   \
  } while (0)

// ---- no device needed ----------------------------------------------------------------
static int shapes() {
  const ItemShape base = default_shape(32);
  atc_tuning rows{}, mixed{}, wide{};
  rows.group_by_source = 1;
  mixed.group_by_source = 2;
  wide.group_by_source = 1;
  wide.bisson_cutover = 64;
  wide.bisson_warp_chunk = 2048;
  // a batch tuned to rows items and then run in the other mode has that mode's items
  const ItemShape tuned = shape_from(&rows, base), then = shape_from(&mixed, tuned);
  REQUIRE(same_shape(then, shape_from(&mixed, base)));
  // what rows items do not use makes no other shape; what they use does
  REQUIRE(same_shape(rows_shape(tuned), rows_shape(shape_from(&wide, base))));
  rows.bisson_warp_chunk = 32;
  REQUIRE(!same_shape(rows_shape(tuned), rows_shape(shape_from(&rows, base))));
  return 0;
}

int main(int argc, char** argv) {
  const char* const what = argc > 1 ? argv[1] : "";
  int r = 2;
  if (!strcmp(what, "shapes")) r = shapes();
  if (r == 0) std::printf("ok\n");
  return r;
}
