// Which form of the Lorenz '96 transition a launch takes.
#pragma once

namespace bpf {

// Blocks of the two-thread form on an SM for a launch of `blocks` blocks
// (128 particles each) of d components of esz bytes, or 0 for one thread per
// particle.  Microseconds per filter step on B200 (resampler included), one
// thread / two threads, 148 SMs:
//   FP32, d = 40: 25.3 / 21.2 at N = 4096, 31.7 / 27.1 at 18944, 37.6 / 30.3
//     at 37888 (two blocks on every SM; 36.6 compiled for three), 44.3 / 38.0
//     at 56832 (three), 44.4 / 46.7 at 65536 (a second wave); d = 8, 16, 32 at
//     37888: 24.8 / 23.1, 27.2 / 24.9, 35.7 / 29.4, at 56832: 29.5 / 24.7,
//     34.3 / 28.1, 41.7 / 35.2.
//   FP64, d = 40: 33.8 / 24.8 at 4096, 40.8 / 33.9 at 20011, 69.1 / 60.8 at
//     65536, 699 / 643 at 10^6, d = 32: 565 / 541 at 10^6: one thread's
//     registers leave an SM half the warps at any size.
//   FP64, d = 8, 16: 27.0 / 24.8, 32.8 / 28.7 at 37888, but 29.1 / 32.0, 36.7
//     / 36.4 at 47360, 34.5 / 38.4, 46.0 / 47.3 at 94720, 168 / 227, 279 / 325
//     at 10^6: there one thread has the registers it needs, and the halves'
//     exchange of three components a stage is dear beside four or eight.
inline int l96_pair_blocks(int d, int esz, int blocks) {
  if (d % 8 != 0) return 0;  // a Philox block's four components belong to one thread
  if (esz == 8) return d >= 32 || blocks <= 2 * 148 ? 2 : 0;
  return blocks <= 2 * 148 ? 2 : blocks <= 3 * 148 ? 3 : 0;
}

}  // namespace bpf
