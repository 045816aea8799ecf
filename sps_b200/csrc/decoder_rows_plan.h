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

// Whether a step of 1 to 16 rows that both could do goes by decoder_rows.cuh rather than decoder_step.cuh.  us per token,
// decoder_step.cuh / decoder_rows.cuh, one row per sequence, in a captured graph:
//   8 rows:  12 layers of 512 columns 224 / 237, 768 268 / 288, 1024 307 / 312, 6 of 2048 308 / 293 (4 rows 287 / 291)
//   9 rows:  4 layers of 64 to 256 columns (intermediate 192 to 2048) 77..82 / 78..87, 256 x 1024 84.2 / 83.4, 320 x 320 80.2 / 84.5,
//            384 x 512 86.7 / 83.5, 512 x 1024 88.6 / 86.7, 2048 x 2048 163 / 139; 12 layers of 768 301 / 289
//   16 rows: 192 x 512 80.2 / 83.3, 256 x 704 84.6 / 84.8, 320 x 320 84.6 / 83.8, 320 x 832 91.6 / 86.3, 512 x 1024 93.0 / 87.2
// (a second tile of 8 rows is what costs decoder_step.cuh more than the separate norm costs the other).  Launched one by
// one, every launch takes about 0.5 us more, and decoder_rows.cuh has two more of them per layer; 12 layers:
//   9 rows:  512 x 2048 291 / 299, 640 x 1728 297 / 312, 768 x 2048 321 / 328, 768 x 3072 348 / 337, 896 x 2432 342 / 332,
//            1024 x 1024 307 / 325, 1024 x 2816 352 / 351, 6 of 1536 x 4096 251 / 223
//   12 rows: 384 x 1024 263 / 276, 640 x 1728 308 / 314, 768 x 2048 331 / 331..338;  16 rows: 512 x 1024 274 / 283, 640 x 1728 336 / 317, 768 x 2048 355 / 328
inline bool rows_faster(int rows, int hidden, int intermediate, bool captured) {
  if (rows <= 8 || hidden < 384) return false;
  return captured || (long long)rows * hidden * (4LL * hidden + 3LL * intermediate) >= 90000000;     // rows x weights of a layer
}

}  // namespace spsattn
