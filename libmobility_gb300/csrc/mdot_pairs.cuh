// M.[F;T] over unordered pairs: every geometry, precision and set of blocks.
//
// Same product as mdot_kernel (libMobility solvers/NBody/extra/
// NbodyRPY.cu:26-252).  The mobility matrix is symmetric, so the coefficients
// of a pair (pairwise.cuh) are computed once and give both particles'
// velocities: per ordered pair 73 multiply-add slots instead of 175 above a
// wall with torques, 33 instead of 100 with forces alone, and in FP64, where
// the pipe is 64 times narrower, the same saving and fewer operations in the
// reciprocal square roots.
//
// Work (per batch of nper particles, tiles of 32 slots; a slot is two
// particles in FP32, one in FP64):
//   * tile pairs (I, J), I <= J, are numbered row by row; each is S rotation
//     steps, S the slots of a tile in use (32, or as few as hold a batch in as
//     many tiles): at step k lane l < S pairs the particles of its slot of tile I
//     (in registers) with those of slot (l + k) mod S of tile J, staged in the
//     warp's shared memory beside that slot's sums.  No two lanes meet a slot
//     in a step, so the J side needs neither atomics nor reductions.  On a
//     diagonal tile (I, I) the S steps cover every ordered pair, and only the
//     I side is kept;
//   * the steps of all tile pairs are cut into equal contiguous ranges, one
//     per resident warp; the next tile is copied in while one is worked on.  A
//     warp keeps the I side across a row (two-sum in FP32) and writes one
//     partial when the row or its range ends; the J side is one partial per
//     tile pair.  (Ranges handed out from a counter, large ones first, were
//     slower up to N = 16384, 688 against 684 us, and 2 % faster at 65536: a
//     warp that runs behind gets the pipe to itself at the end, where it runs
//     at seven eighths of the rate, and shorter ranges mean more partials);
//   * partials have closed-form places: one slot per tile pair (J side), one
//     per row (I side), and one of each per warp, for a range that starts in
//     the middle of a tile pair or row.  Every slot that is read was written
//     in the same launch, so scratch needs no clearing;
//   * pairs closer than 2a take the fast form (r^2 clamped at 4); steps where a
//     lane met one are flagged and, after the tile pair's steps, those pairs
//     get (exact - fast);
//   * after a bounded grid barrier the partials are folded, one component of a
//     tile at a time by a warp, or by a block's four warps taking every fourth
//     partial, with the two-sum transformation in FP32; the order is fixed, so
//     results repeat bit for bit;
//   * the rows are done in passes when the partials of all of them would not
//     fit the scratch limit: whole batches, or bands of rows of one batch,
//     with the sums carried from pass to pass.
//
// What bounds it, measured (GB300, kernel times, mdot_kernel before): FP32 wall
// with torques N = 16384 678 us (1399): 393 cycles of a scheduler per 64
// unordered pairs, 146 packed instructions on the FMA pipe with 2.7 operand
// reads each; wall forces N = 16384 323 us (751), N = 100003 11.6 ms (27.0);
// open with torques N = 6001 70 us (103).  FP64 is the FP64 pipe itself (36
// operations an unordered pair in open space, 151 above a wall with torques):
// open forces N = 4096 560 us (1019), wall with torques N = 3001 1264 us
// (4974).  A few hundred particles cost 8 to 12 us (16 to 63), FP64 17 to 44
// (298 to 3167): launch, one tile's latency, barrier and fold; 64 batches of 333,
// open forces, 16.9 us, of which the steps take 7.
#pragma once
#include <cstddef>
#include <vector>

#include <cuda_runtime.h>

#include "pack2.cuh"
#include "pairwise.cuh"

namespace lmg {

constexpr int kPairsThreads = 128;  // four warps per block

// Particles of a lane's slot; a tile is 32 slots.
template <class R> constexpr int kPairsSlot = sizeof(R) == 4 ? 2 : 1;
template <class R> constexpr int kPairsTile = 32 * kPairsSlot<R>;

// One launch: global rows (tile I of batch b = b * tpb + I) [row0, row1).
struct PairsPass {
  int row0 = 0, row1 = 0;
  unsigned steps = 0;   // rotation steps of its tile pairs
  unsigned per_warp = 0;  // steps of a warp's range
  int warps = 0, grid = 0;
  size_t cut_off = 0;   // this pass's part of the tables below
};

struct PairsPlan {
  bool ok = false;      // false: use mdot_kernel
  int N = 0, nper = 0, tpb = 0;
  int slots = 32;       // of a tile in use (the same for all)
  bool wall = false, ang = false;
  std::vector<PairsPass> passes;
  size_t part_elems = 0;  // scratch (of R) of the largest pass
  size_t acc_elems = 0;   // sums carried between passes
  bool carries = false;   // a batch takes several passes (else nothing is carried)
  // per pass: for each tile, where its list of J-side partials of cut tile
  // pairs begins (tiles + 1 entries), then the warps that wrote them
  std::vector<int> cuts;
};

// Plans the launches for `resident` blocks on the GPU at once (no device
// needed).  force_warps > 0 caps the warps the steps are spread over,
// max_part > 0 the scratch elements (tests).
template <class R>
void mdot_pairs_plan_tables(int N, int nper, bool ang, long long resident, int force_warps,
                            size_t max_part, PairsPlan &p);

template <class R>
cudaError_t mdot_pairs_plan(int N, int nper, bool wall, bool ang, int num_sms, int force_warps,
                            size_t max_part, PairsPlan &p);

// U (and W with ang; either may be null) = M.[F;T]; F or T null: zero.
// `bar` is the grid barrier's arrival count, one per pass, zero before the
// plan's first launch; *err (device visible) is set if a barrier ran out.
template <class R>
cudaError_t mdot_pairs_launch(const PairsPlan &p, const int *cuts, const R *pos, const R *F,
                              const R *T, R *U, R *W, R inv_a, PairScale<R> k, R *part, R *acc,
                              unsigned long long *bar, int *err, cudaStream_t stream);

}  // namespace lmg
