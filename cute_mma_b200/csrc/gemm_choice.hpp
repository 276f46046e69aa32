// Which kernel a plain GEMM runs on: tiles of 128 x (16..128) with K in pieces (small_kernel), CTA-pair tiles of 256 x 256 (gemm2_kernel)
// or of 256 x 512 (gemm2w_kernel).  All three return the same bits as long as K is not cut.
#pragma once

namespace b200 {

// Tiles of 128 x 128 of an m x n result.
inline long long tiles_128(int m, int n) { return ((static_cast<long long>(m) + 127) / 128) * ((static_cast<long long>(n) + 127) / 128); }

// Whether small_kernel takes a plain m x n product of `steps` K steps (128 bytes of a row each).
// As long as its 128 x 128 tiles do not outnumber the SMs, always (fixed cost per launch 5 us against 7 to 9 us, and 256 x
// 256 tiles leave most SMs idle: 640 x 1280 x 1024 TF32 29 -> 10 us), and for n <= 128, of which a pair tile covers twice
// the columns at least (65536 x 120 x 4096 half 100 against 128 us, 131072 x 64 x 512 31 against 40).  Above, the two are
// compared by a model fitted to 649 random shapes of 149 to 1500 tiles: a K step of two tiles per SM costs 0.74 us for 128
// columns and half of that for the 128 rows of P alone (a narrow tile loads and multiplies those all the same), a last wave of one tile
// per SM 0.24 and of more 0.48; a round of pair tiles 0.34 us per step on 74 pairs, either size; plus fixed costs.  What it
// picks takes 0.9 % longer than the better of the two on average, at worst 31 % (23650 x 310 x 1485 NT half to float 50.0 us against
// 38.1).  Counted by its columns alone a narrow tile lost up to 55 % (7016 x 272 x 2536 half 29.5 against 21.0, 33475 x 147 x 2919 67.8
// against 47.9).  5936 x 776 x 5822 NT: 118 against 68 us; 2815 x 6280 x 163: 27 against 20; 11904 x 276 x 263 TF32: 9.9 against 15.7.
// With K whole (the GEMMs of oft_two_pass, n the rows of X) the model decides in the first range too, where a K step of an SM's only
// tile costs 0.4 us: 96 tiles of 64 steps 29.6 us against 36.9, 128 tiles of 226 steps 97.9 against 85; 280 tiles of 45
// steps 27.8 / 41.7, 1296 tiles of 4 steps 30.0 / 26.7.
inline bool small_wins(int m, int n, int steps, bool whole_k, long long sms) {
  const long long t128 = tiles_128(m, n), pairs = sms / 2;
  if (n <= 128 ? !whole_k || t128 > sms : !whole_k && t128 <= sms) return true;
  const long long t256 = ((static_cast<long long>(m) + 255) / 256) * ((static_cast<long long>(n) + 255) / 256);
  const long long waves = t128 / (2 * sms), rest = t128 % (2 * sms);
  const int tiles_n = (n + 127) / 128;
  const double step = (0.5 + 0.5 * ((n + tiles_n - 1) / tiles_n) / 128.0) * steps;  // K steps of 128 columns
  const double small = t128 <= sms ? 6.0 + 0.4 * step
                                   : 6.0 + step * (0.74 * waves + (rest == 0 ? 0.0 : rest <= sms ? 0.24 : 0.48)) + 1.8 * (waves + (rest > 0));
  const double pair = 8.0 + static_cast<double>((t256 + pairs - 1) / pairs) * (0.34 * steps + 1.7);
  return small < pair;
}

// Whether the plain GEMM of `steps` K steps runs on tiles of 256 x 512 (gemm2w_kernel).  Both kernels give the longest pair the
// same number of 256-column tiles, `rounds`; the wide one moves a quarter less between L2 and the SMs and starts with bigger
// loads, so it needs a second round to pair up and some work to make up for the start.  us on tiles of 256 / 512: 8192^3
// 864 / 842, 4690 x 9804 x 9607 NT 906 / 782, TF32 NT 5933 x 7743 x 6727 1331 / 1000; below the lines 1634 x 4191 x 725 TF32 TN (46 K
// steps in a row) 25 / 26.5, 3658 x 3972 x 551 NT half (36) 25.3 / 26.9, above them 3257 x 3051 x 1588 NT half (75) 38.8 / 37.2,
// 9304 x 808 x 1265 NT (40) 29.2 / 27.2.  Short tiles of TN products are bound by their stores, which come in bursts here:
// 13171 x 10088 x 256 98 / 138, 8192 x 8192 x 512 69 / 72.
// How much the quarter is worth depends on whether the operands' rows start on 128-byte lines (whole_lines).  Where they do not,
// every 128-byte piece of a tile touches two, and the wide tile takes 0.91 of the other's time on average (190 random shapes above
// the lines).  Where they do, NT products are level in short runs and 2 % faster in long ones, under the power cap; TN
// products are 3 % slower (216 shapes) up to 48 K steps, or 320 in a row, and beyond that (71) as the NT ones: 1600 x 3840 x 4928
// half to float 56 / 60, 3583 x 5376 x 448 TF32 39 / 42, 5117 x 9734 x 3328 269 / 274 (0.97 in long runs), 1600 x 12608 x 7680 327 / 313 (0.93).
// In between the two are level where whole wide tiles fill their rounds to five sixths (and 48 steps each): 2048 x 4096 x 3648 55.7 / 55.9,
// 4096 x 2048 x 4096 behind the rotation of the weight (A_RW) 77.0 / 75.6.  Two columns of tiles are one wide one, which reads A once
// for both: 0.96 over 16 shapes, 20480 x 331 x 6784 115 / 105, 21888 x 424 x 6272 121 / 111.
// And there a last column of 256 without a neighbour, which reads all of A once more, costs more than its neighbours
// save until they are eight or so: 49664 x 768 x 4672 NT 247 / 264, 12544 x 1792 x 2048 TF32 126 / 142, but 49664 x 1024 x 4672 343 / 337.
inline bool wide_wins(int m, int n, int steps, bool nt, bool whole_lines, long long sms) {
  const long long pairs = sms / 2, tiles_n = (n + 255ll) / 256, tiles = (m + 255ll) / 256 * tiles_n, rounds = (tiles + pairs - 1) / pairs;
  if (n <= 256 || rounds < 2 || rounds * steps < (nt ? 40 : 60) || (!nt && steps <= 8)) return false;
  if (!whole_lines) return true;
  const bool filled = tiles_n % 2 == 0 && 6 * tiles >= 5 * (rounds + rounds % 2) * pairs;
  return (tiles_n % 2 == 0 || tiles_n >= 8) && (nt || tiles_n == 2 || (steps >= 48 && (filled || rounds * steps >= 320)));
}

}  // namespace b200
