// Host check of the rule that gives a lattice its stage kernel (stage_parts): no device code runs.
// A wave of 75,776 cells (148 SMs); each line is a size on one side of a border.
#include <stdio.h>

#include "gvh_stage_launch.cuh"

int main() {
  const long long wave = gvh::stage_wave_cells(148);
  const struct {
    long long cells;
    int ideal, shear, bulk;  // parts
  } want[] = {{1, 8, 8, 8},          {9472, 8, 8, 8},    {9473, 4, 4, 4},   {18944, 4, 4, 4},
              {18945, 2, 4, 4},      {20128, 2, 4, 4},   {20129, 2, 2, 4},  {24000, 2, 2, 4},
              {28416, 2, 2, 4},      {28417, 2, 2, 2},   {37888, 2, 2, 2},  {37889, 4, 4, 4},
              {56832, 4, 4, 4},      {56833, 1, 1, 1},   {1046821, 1, 1, 1}};
  int errors = wave != 75776;
  for (const auto &w : want) {
    const int got[3] = {gvh::stage_parts(w.cells, wave, 0, 0), gvh::stage_parts(w.cells, wave, 1, 0),
                        gvh::stage_parts(w.cells, wave, 1, 1)};
    if (got[0] != w.ideal || got[1] != w.shear || got[2] != w.bulk) {
      printf("%lld cells: %d %d %d\n", w.cells, got[0], got[1], got[2]);
      ++errors;
    }
  }
  printf("%d errors\n", errors);
  return errors ? 1 : 0;
}
