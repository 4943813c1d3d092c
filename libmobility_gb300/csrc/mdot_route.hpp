// The kernel that an all-pairs product outside a solve takes.
//
// mdot_pairs_kernel computes a pair once for both particles and is the faster
// one nearly everywhere; where it is not, what it pays per tile pair (a copy
// to shared memory, two partial sums written, read and folded behind a grid
// barrier) outweighs the pairs saved.  All times below are of the kernels in a
// CUDA graph on a GB300, this library's, in microseconds.
#pragma once

namespace lmg {

enum class MdotRoute { tiled, symmetric, pairs };  // mdot_kernel, mdot_sym_kernel, mdot_pairs_kernel

// The symmetric open-space kernel (FP32 forces) against the pairs: tiles of 128
// particles, half of a diagonal tile's steps, four particles a slot, but
// padding to 128.  Batches of 384 and more take it always (500: 8.4 and 8.3,
// 4096: 18.9 and 20.2).  Smaller ones where its tiles cost no more steps than
// the pairs' slots, once the GPU is filled: 100 batches of 256 13.6 and 17.3,
// 234 of 96 13.1 and 16.3, 70 of 128 10.3 and 10.9, but 20 of 96 9.9 and 8.1;
// with more padding 100 of 320 20.5 and 20.7, 400 of 260 61 and 49.
inline bool mdot_symmetric_better(int N, int nper, int num_sms) {
  if (N > nper && nper % 4 != 0) return false;  // it loads four particles at once
  if (nper >= 384) return true;
  if (N < 48 * num_sms) return false;
  const int t = (nper + 127) / 128;
  const int tpb = (nper + 63) / 64, slots = ((nper + tpb - 1) / tpb + 1) / 2;
  // lane steps: 16 pairs each, 17 on a diagonal tile and 32 beside it; 4 pairs
  // each, one for every slot
  return 16 * (17 * t + 16 * t * (t - 1)) <= 4 * slots * tpb * (tpb + 1) / 2;
}

// one: forces or torques alone, with angular velocities (mdot_kernel leaves
// out the blocks of what is absent, the pairs do not).
inline MdotRoute mdot_route(bool fp64, bool wall, bool ang, bool one, int N, int nper,
                            int num_sms) {
  if (nper <= 0) return MdotRoute::tiled;
  const int nb = N / nper;
  // A handful of particles, one CTA: no barrier and no partial sums.  N = 10:
  // open with torques 5.3 and 6.9, wall 5.2 and 7.1; 2 x 17 open forces 5.4 and 6.3;
  // FP64 N = 5: open 9.5 and 12.2; N = 1: wall with torques 7.6 and 33.
  const int few = fp64 ? (wall ? (one ? 5 : 3) : (one ? 11 : 8))
                       : (wall ? (!ang ? 19 : one ? 24 : 16) : (ang && !one ? 24 : 34));
  if (N <= few) return MdotRoute::tiled;
  // particles that meet only themselves: 31 x 1 wall with torques 6.5 and 8.6, open
  // forces 5.1 and 6.2 (84 x 1 8.8 and 10.2, 6.2 and 7.0; but open with torques 9.6
  // and 8.8, wall forces 9.2 and 7.7); FP64 6 x 1 above a wall 15 and 21
  if (nper == 1 && N <= (fp64 ? 8 : wall == ang ? num_sms : 32)) return MdotRoute::tiled;
  if (!fp64 && !ang && !wall && mdot_symmetric_better(N, nper, num_sms))
    return MdotRoute::symmetric;
  // More tiny batches than SMs: each is a tile pair of its own, while a tile
  // of mdot_kernel holds many; it does best where 32 is a multiple of the
  // batch, so that a warp's targets meet 32 sources.
  if (nb > num_sms) {
    if (fp64) {
      // 100 000 x 1: open 236 and 901, wall 422 and 1520 (3000 x 1: 70 and 82);
      // open, 25 000 x 4 236 and 413, 3125 x 32 237 and 252, but 625 x 16 45 and
      // 38, 5000 x 20 356 and 269; wall, 25 000 x 4 956 and 744
      if (nper == 1) {
        if (N >= 16 * num_sms) return MdotRoute::tiled;
      } else if (!wall) {
        if (nper <= 4 && N >= 64 * num_sms) return MdotRoute::tiled;
        if ((nper <= 8 || 32 % nper == 0) && N >= 192 * num_sms) return MdotRoute::tiled;
      }
    } else {
      // 1000 x 2: wall with torques 16 and 41, forces 14 and 24; 18 750 x 16: 146
      // and 243, 100 and 120; 5000 x 20: 95 and 81, 68 and 43.  With torques the
      // pairs' partial sums are twice as many: 375 x 8 in open space 11.8 and 13.7
      // (forces 9.0 and 9.0), 625 x 16 11.9 and 14.3 (forces 9.1 and 9.7).  Above a
      // wall an evaluation is dearer, and where 32 is no multiple of the batch
      // mdot_kernel makes more: 655 x 12 24 and 19, 322 x 7 21 and 17 (forces alone
      // 988 x 6 18 and 25).
      if (nper <= (ang && (!wall || one) ? 8 : 4)) return MdotRoute::tiled;
      const bool whole = 32 % nper == 0;
      if (nper <= 16 && nb >= (ang && (!wall || whole) ? 4 : 8) * num_sms)
        return MdotRoute::tiled;
      // 937 x 32 with torques, open 12.7 and 21.3, wall 20.7 and 28.3
      if (nper == 32 && ang && nb >= 2 * num_sms) return MdotRoute::tiled;
      // open with torques: 1500 x 20 20.8 and 24.4, 4166 x 24 46 and 53; a batch a
      // tile, 234 x 128 16.6 and 26, 800 x 128 51 and 61
      if (!wall && ang && !one && ((nper <= 24 && nb >= 8 * num_sms) || nper == 128))
        return MdotRoute::tiled;
    }
  }
  // Forces or torques alone in open space: mdot_kernel does half the work of
  // either both, but loses much at the edges of batches that are no whole tiles.
  if (one && !wall) {
    if (fp64) {
      // 369 x 64 139 and 230, 400 x 33 115 and 156, 2000 x 100 2048 and 2658, but
      // 160 x 65 188 and 148, 200 x 48 142 and 113, 500 x 30 114 and 101; 320 x 1 53
      // and 69, 1427 x 8 55 and 105, 2591 x 3 66 and 101 (721 x 3 67 and 41); one batch
      // of 4096 1390 and 1275
      if (nb >= 2 * num_sms && (N >= 80 * num_sms || nper % 32 == 0 || nper == 1))
        return MdotRoute::tiled;
      if (nper <= 8 && nb >= 8 * num_sms) return MdotRoute::tiled;
    } else {
      // one batch: N = 16384 354 and 433, 6000 67 and 70, 4096 37.1 and 37.5 (but
      // 4 x 2500 76 and 55, 2 x 9001 293 and 269)
      if (nb == 1 && (double)N * N >= 2e7) return MdotRoute::tiled;
      // whole tiles: 10 x 512 15.4 and 18.4, 2 x 16384 698 and 862; 2 x 256 12.0 and
      // 11.5
      if (nper % 128 == 0 && nb > 1 && N >= 16 * num_sms) return MdotRoute::tiled;
      // whole warps: 400 x 64 14.3 and 17.6, 400 x 96 22 and 31, 1000 x 160 90 and 107
      // (267 x 160 50 and 39)
      if (nb > num_sms && (nper <= 16 || (nper % 32 == 0 && nper < 128)))
        return MdotRoute::tiled;
      if (nb >= 4 * num_sms && nper % 32 == 0) return MdotRoute::tiled;
      // batches that leave half of the pairs' second tile empty: 2000 x 72 60 and 95,
      // 2000 x 100 88 and 108, 2000 x 120 119 and 119, 800 x 72 46 and 44
      if (nb >= 10 * num_sms && nper > 64 && nper < 112) return MdotRoute::tiled;
    }
  }
  return MdotRoute::pairs;
}

}  // namespace lmg
