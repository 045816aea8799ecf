// Sizes of a block of decoder_rows.cuh: plain C++.
#pragma once

namespace spsattn {

struct RowsTiles {
  int bn, bm;                 // weight rows and input rows of a block
  long long blocks, cost;
};

// A block reads (bn + bm) rows of K columns, and 16 rows' worth of time goes by around them.  The cheapest sizes by
// that and the number of waves; ties go to the wider input tile, which reads the weights fewer times.
// bn in steps of `step` up to `most`.
inline RowsTiles rows_tiles(int weight_rows, int rows, int multiprocessors, int step, int most) {
  RowsTiles best{0, 0, 0, 0};
  for (int bm = (rows + 15) / 16 * 16; bm >= 16; bm -= 16)
    for (int bn = step; bn <= most; bn += step) {
      const long long blocks = ((long long)weight_rows + bn - 1) / bn * ((rows + bm - 1) / bm);
      const long long waves = (blocks + multiprocessors - 1) / multiprocessors, cost = waves * (bn + bm + 16);
      if (best.blocks == 0 || cost < best.cost) best = {bn, bm, blocks, cost};
    }
  return best;
}

}  // namespace spsattn
