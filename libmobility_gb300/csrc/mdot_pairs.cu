// All-pairs product over unordered pairs: kernel, plan and launch.  The scheme
// is described in mdot_pairs.cuh.  Compiled once per precision (LMG_REAL).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "bounds.cuh"
#include "grid_sync.cuh"
#include "launch_count.hpp"
#include "mdot_pairs.cuh"

#ifndef LMG_REAL
#define LMG_REAL float
#endif

namespace lmg {

namespace {

// Largest scratch for the tile pairs of a pass, in elements (1 GiB in FP32, 2 in
// FP64); the slots of the rows and warps come on top.  A handle keeps it.
constexpr size_t kPairsMaxPart = size_t(1) << 28;
// Tile pairs of a row whose I sums a lane adds up before the two-sum (in FP32
// the lanes of a packed sum then hold 128 terms each at most).
constexpr int kPairsHeld = 4;
// Fewest rotation steps a warp is given.
constexpr long long kPairsMinSteps = 4;
// Padding particles of a ragged tile: no force or torque, 4 radii apart on a
// line far from the origin (and one radius above a wall); their own sums are
// never read.
constexpr double kPadX = 1.0e6;
constexpr double kTooHigh = 1.152921504606846976e18;  // 2^60 radii

template <class R> struct LaneTypes;
template <> struct LaneTypes<float> { using V = F2; using L = float2; };
template <> struct LaneTypes<double> { using V = double; using L = double; };
__device__ __forceinline__ float lane_value(float2 v, int q) { return q ? v.y : v.x; }
__device__ __forceinline__ double lane_value(double v, int) { return v; }
__device__ __forceinline__ float lane_of(F2 v, int q) { return q ? v.v.y : v.v.x; }
__device__ __forceinline__ double lane_of(double v, int) { return v; }

__device__ __forceinline__ F2 splat(float x, F2) { return bc(x); }
__device__ __forceinline__ double splat(double x, double) { return x; }
// a slot's sums from those of its particles (each lane of an F2 holds half)
__device__ __forceinline__ F2 both(F2 a, F2 b) { return mk2(a.v.x + a.v.y, b.v.x + b.v.y); }
__device__ __forceinline__ double both(double a, double) { return a; }

// running sum (S, C): two-sum in FP32, plain in FP64
__device__ __forceinline__ void fold_in(float &S, float &C, float t) {
  const float s = S + t;
  const float bp = s - S;
  C += (S - (s - bp)) + (t - bp);
  S = s;
}
__device__ __forceinline__ void fold_in(double &S, double &, double t) { S += t; }
__device__ __forceinline__ void fold_in(F2 &S, F2 &C, F2 t) {
  const F2 s = S + t;
  const F2 bp = s - S;
  C = C + ((S - (s - bp)) + (t - bp));
  S = s;
}

template <class R> struct PairsArgs {
  const R *pos, *F, *T;
  R *U, *W;
  int N, nper, tpb;   // tpb: tiles per batch
  int slots;          // of a tile in use
  int row0, row1;
  int tiles;          // tiles of all batches
  unsigned steps, per_warp;
  int warps;
  bool first, last;   // of the passes
  bool wide;          // a slot of any tile is 8-byte aligned in pos, F and T
  int share;          // warps that fold a component of a tile together (1 or 4)
  R inv_a;
  PairScale<R> k;
  R *part;
  size_t part_elems;
  R *acc;
  const int *cuts;
  unsigned long long *bar;
  int spins;  // of the barrier
  int *err;
};

// Tile pairs before global row r (rows of a batch shrink by one tile each).
__host__ __device__ __forceinline__ long long pairs_before(int tpb, int r) {
  const long long b = r / tpb, I = r - b * tpb;
  return b * ((long long)tpb * (tpb + 1) / 2) + I * tpb - I * (I - 1) / 2;
}

// Tile pairs of a batch before local row I.
__host__ __device__ __forceinline__ int local_before(int tpb, int I) {
  return I * tpb - I * (I - 1) / 2;
}

template <int BYTES> __device__ __forceinline__ void copy_async(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES)
               : "memory");
}
__device__ __forceinline__ void copies_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Starts the copies of the lane's particles of tile t (of the batch that starts
// at particle b0) to raw[positions, F, T][3 * particle + component]; only that
// lane reads them back (scale_slot).
template <class R, bool ANG, int NA, int TE>
__device__ __forceinline__ void fetch_slot(const PairsArgs<R> &a, int S, int b0, int t, int lane,
                                           R (&raw)[NA][TE]) {
  constexpr int NS = kPairsSlot<R>;
  const int l = NS * (t * S + lane);
  if (lane >= S) return;
  const size_t g = 3 * (size_t)(b0 + l);
  const R *src[3] = {a.pos + g, a.F + g, a.T + g};
  const bool use[3] = {true, a.F != nullptr, ANG && a.T != nullptr};
  if (l + NS <= a.nper && (NS == 1 || a.wide) &&
      LMG_IN_BOUNDS(b0 + l + NS <= a.N, 21, b0 + l)) {
#pragma unroll
    for (int q = 0; q < NA; q++) {
      if (!use[q]) continue;
#pragma unroll
      for (int c = 0; c < 3; c++)  // 8 bytes each
        copy_async<8>(&raw[q][3 * NS * lane + NS * c], src[q] + NS * c);
    }
  } else if (NS > 1) {
#pragma unroll
    for (int q = 0; q < NA; q++) {
      if (!use[q]) continue;
#pragma unroll
      for (int c = 0; c < 3 * NS; c++)
        if (l + c / 3 < a.nper && LMG_IN_BOUNDS(b0 + l + c / 3 < a.N, 21, b0 + l))
          copy_async<sizeof(R)>(&raw[q][3 * NS * lane + c], src[q] + c);
    }
  }
}

// The lane's particles, scaled: out = x, y, z, F, T.
template <class R, bool WALL, bool ANG, int NA, int TE, int NV, int TS>
__device__ __forceinline__ void scale_slot(const PairsArgs<R> &a, int S, int t, int lane,
                                           const R (&raw)[NA][TE], R (&out)[NV][TS]) {
  constexpr int NS = kPairsSlot<R>;
  using L = typename LaneTypes<R>::L;
  R v[NS][9];
  R r[NA][3 * NS];
#pragma unroll
  for (int q = 0; q < NA; q++) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const L x = reinterpret_cast<const L *>(raw[q])[3 * lane + c];
#pragma unroll
      for (int h = 0; h < NS; h++) r[q][NS * c + h] = lane_value(x, h);
    }
  }
#pragma unroll
  for (int q = 0; q < NS; q++) {
    const bool in = lane < S && NS * (t * S + lane) + q < a.nper;
    // no contraction with the differences: a particle meets itself at d = 0
    v[q][0] = in ? mul_rn(r[0][3 * q], a.inv_a) : R(kPadX) + R(4 * (NS * lane + q));
    v[q][1] = in ? mul_rn(r[0][3 * q + 1], a.inv_a) : R(0);
    v[q][2] = in ? mul_rn(r[0][3 * q + 2], a.inv_a) : (WALL ? R(1) : R(0));
    R sF = a.k.sF, sT = a.k.sT;
    if (WALL) {
      const R z = v[q][2];
      const R b = z < R(0) ? R(0) : (z > R(1) ? R(1) : z);
      v[q][2] = z > R(1) ? z : R(1);
      // The product of two heights must not overflow (pairwise.cuh; it is
      // multiplied by a fifth power that is 0 by then): a particle 1e18 radii up,
      // which meets nobody to within rounding, goes no higher but further away.
      if (sizeof(R) == 4 && z > R(kTooHigh)) {
        v[q][2] = R(kTooHigh);
        v[q][0] += z - R(kTooHigh);
      }
      sF *= b;
      sT *= b;
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      v[q][3 + c] = in && a.F ? sF * r[1][3 * q + c] : R(0);
      if (ANG) v[q][6 + c] = in && a.T ? sT * r[ANG ? 2 : 0][3 * q + c] : R(0);
    }
  }
#pragma unroll
  for (int c = 0; c < NV; c++) {
    if constexpr (NS == 2)
      reinterpret_cast<float2 *>(out[c])[lane] = make_float2(v[0][c], v[NS - 1][c]);
    else
      out[c][lane] = v[0][c];
  }
}

// Resident blocks per SM the register budget is made for (no spills).  FP32 is
// bound by operand reads (pairwise.cuh), not by warps in flight: N = 16384
// with 1, 2, 3 (4) blocks: wall with torques 744, 695, 685 us, wall forces 385,
// 329, 324 (323) us.
template <class R, bool WALL, bool ANG> constexpr int pairs_min_blocks() {
  if (sizeof(R) == 8) return WALL && ANG ? 2 : 3;
  return ANG ? 3 : 4;
}
// With fewer than this many steps a warp, two blocks per SM are launched: the
// ranges are longer, their partials fewer, and a warp alone on its scheduler
// still runs at seven eighths of its rate (N = 2048 wall with torques, 9 steps
// a warp with three blocks: 23.4 us with three, 21.1 us with two; N = 3000 open
// with torques, 20 steps: 25.2 and 23.9 us; N = 6001, 78 steps: 69.6 and 71).
// The line is lower with torques in small batches, whose sums have few partials
// either way: 64 batches of 333 above a wall, 24 steps, 48.4 us with three and
// 51.0 with two, 32 of 500 in open space, 20 steps, 27.5 and 29.1 us (one batch
// of 3000, 20 steps, 25.2 and 23.9).  Not with forces alone: 64 batches of 333,
// 18 steps, 18.4 us with four blocks and 17.6 with two.
constexpr long long pairs_few_steps(bool ang, long long tpb) {
  return ang && tpb <= 32 ? 16 : 24;
}

// A warp's shared memory: tiles I and J, the next ones as they arrive, the J
// sums, the row's I sums (sum, compensation).
template <class R, bool ANG> struct PairsWarp {
  static constexpr int NC = ANG ? 6 : 3, NV = ANG ? 9 : 6, TS = kPairsTile<R>;
  R I[NV][TS], J[NV][TS], next_I[NV / 3][3 * TS], next_J[NV / 3][3 * TS], A[NC][TS], S[NC][TS],
      C[sizeof(R) == 4 ? NC : 1][TS];
};

// A warp's next piece of work: steps k .. k+n-1 of one tile pair.
struct Segment {
  int left;                // steps left of the warp's range (these included)
  int batch, I, J, p;      // row, column and number of the tile pair
  int k, n;
  bool new_row, new_tile;  // the row begins here; tile I is not the last segment's
};

// FULL: all 32 slots of a tile are in use.
template <class R, bool WALL, bool ANG, bool FULL>
__global__ void __launch_bounds__(kPairsThreads, (pairs_min_blocks<R, WALL, ANG>()))
mdot_pairs_kernel(const PairsArgs<R> a) {
  using V = typename LaneTypes<R>::V;
  constexpr int NS = kPairsSlot<R>, TS = kPairsTile<R>;
  constexpr int NC = ANG ? 6 : 3, NV = ANG ? 9 : 6;
  constexpr int EL = NC * TS;  // elements of a partial, [component][particle]
  constexpr int NW = kPairsThreads / 32;  // warps of a block

  using Warp = PairsWarp<R, ANG>;
  extern __shared__ __align__(16) unsigned char smem[];
  Warp *sm = reinterpret_cast<Warp *>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gw = blockIdx.x * NW + warp;
  Warp &w = sm[warp];
  const int nsl = FULL ? 32 : a.slots;

  const int ppb = a.tpb * (a.tpb + 1) / 2;
  const int P0 = (int)pairs_before(a.tpb, a.row0);
  const int npairs = (int)pairs_before(a.tpb, a.row1) - P0;
  const size_t slot_row = npairs, slot_irow = slot_row + (a.row1 - a.row0),
               slot_cut = slot_irow + a.warps;

  auto put = [&](size_t slot, const R (&src)[NC][TS]) {
    if (!LMG_IN_BOUNDS((slot + 1) * EL <= a.part_elems, 22, slot)) return;
    V *d = reinterpret_cast<V *>(a.part + slot * EL);
#pragma unroll
    for (int c = 0; c < NC; c++) {
      const V *s = reinterpret_cast<const V *>(src[c]);
      if constexpr (sizeof(R) == 4)
        __stcg(reinterpret_cast<float2 *>(d) + c * 32 + lane, s[lane].v);
      else
        __stcg(reinterpret_cast<double *>(d) + c * 32 + lane, s[lane]);
    }
  };

  // the warp's range, and in it the tile pair it begins with
  Segment cur;
  const unsigned x0 = (unsigned)gw * a.per_warp;
  cur.left = 0;
  if (gw < a.warps) {
    cur.left = (int)min(a.per_warp, a.steps - x0);
    cur.p = (int)(x0 / (unsigned)nsl);
    cur.k = (int)(x0 - (unsigned)cur.p * (unsigned)nsl);
    cur.n = min(nsl - cur.k, cur.left);
    const int g = P0 + cur.p;
    cur.batch = a.tpb == a.tiles ? 0 : g / ppb;
    const int rem = g - cur.batch * ppb;
    const float m = 2.0f * (float)a.tpb + 1.0f;
    int I = (int)(0.5f * (m - sqrtf(fmaxf(m * m - 8.0f * (float)rem, 0.0f))));
    I = max(0, min(I, a.tpb - 1));
    while (local_before(a.tpb, I) > rem) I--;
    while (local_before(a.tpb, I + 1) <= rem) I++;
    cur.I = I;
    cur.J = I + rem - local_before(a.tpb, I);
    cur.new_row = cur.k == 0 && cur.J == I;
    cur.new_tile = true;
  }
  auto follow = [&](const Segment &c) {
    Segment s = c;
    s.left = c.left - c.n;
    s.p++;
    s.J++;
    s.k = 0;
    s.n = min(nsl, s.left);
    s.new_row = s.new_tile = s.J == a.tpb;
    if (s.new_tile) {
      if (++s.I == a.tpb) {
        s.I = 0;
        s.batch++;
      }
      s.J = s.I;
    }
    return s;
  };
  auto fetch = [&](const Segment &s) {
    if (s.left == 0) return;
    const int b0 = s.batch * a.nper;
    if (s.new_tile) fetch_slot<R, ANG>(a, nsl, b0, s.I, lane, w.next_I);
    fetch_slot<R, ANG>(a, nsl, b0, s.J, lane, w.next_J);
  };

  fetch(cur);
  // the slot that a lane meets at step k; lanes past the slots keep to their own,
  // which is padding in every tile
  const bool idle = !FULL && lane >= nsl;
  auto met = [&](int k) {
    if (FULL) return (lane + k) & 31;
    const int s = lane + k;
    return idle ? lane : (s >= nsl ? s - nsl : s);
  };
  const V zero = splat(R(0), V());
  bool row_begun = false;  // the I sums are those of the row's first partial
  int held = 0;            // tile pairs whose I sums are still in registers
  V vi[NS][9];
  Vec6<V> ui[NS];
  while (cur.left > 0) {
    copies_done();
    if (cur.new_tile) {
      scale_slot<R, WALL, ANG>(a, nsl, cur.I, lane, w.next_I, w.I);
      row_begun = cur.new_row;
      held = 0;
#pragma unroll
      for (int c = 0; c < NC; c++) {
        reinterpret_cast<V *>(w.S[c])[lane] = zero;
        if (sizeof(R) == 4) reinterpret_cast<V *>(w.C[sizeof(R) == 4 ? c : 0])[lane] = zero;
      }
#pragma unroll
      for (int q = 0; q < NS; q++) {
#pragma unroll
        for (int c = 0; c < 9; c++)
          vi[q][c] = c < NV ? splat(w.I[c < NV ? c : 0][NS * lane + q], V()) : zero;
        ui[q] = {zero, zero, zero, zero, zero, zero};
      }
    }
    scale_slot<R, WALL, ANG>(a, nsl, cur.J, lane, w.next_J, w.J);
#pragma unroll
    for (int c = 0; c < NC; c++) reinterpret_cast<V *>(w.A[c])[lane] = zero;
    __syncwarp();
    const Segment nxt = follow(cur);
    fetch(nxt);
    const bool diag = cur.J == cur.I;
    const int k_end = cur.k + cur.n;
    unsigned near = 0u;  // steps with a pair closer than 2a
#pragma unroll 1
    for (int k = cur.k; k < k_end; k++) {
      const int s = met(k);
      V vj[9], A[6];
#pragma unroll
      for (int c = 0; c < 9; c++)
        vj[c] = c < NV ? reinterpret_cast<const V *>(w.J[c < NV ? c : 0])[s] : zero;
      // the slot's sums so far (a diagonal tile's are dropped)
#pragma unroll
      for (int c = 0; c < 6; c++)
        A[c] = c < NC ? reinterpret_cast<const V *>(w.A[c < NC ? c : 0])[s] : zero;
      Vec6<V> aj = {A[0], A[1], A[2], A[3], A[4], A[5]};
      bool close = false;
#pragma unroll
      for (int q = 0; q < NS; q++)
        close |= any_below4(pair_both<V, WALL, ANG>(vi[q], vj, ui[q], aj));
      near |= close && !idle ? 1u << k : 0u;
      if (!diag) {
        const V sum[6] = {aj.ux, aj.uy, aj.uz, aj.wx, aj.wy, aj.wz};
#pragma unroll
        for (int c = 0; c < NC; c++) reinterpret_cast<V *>(w.A[c])[s] = sum[c];
      }
      __syncwarp();  // the slot belongs to another lane at the next step
    }
    const bool flush = nxt.new_tile || nxt.left == 0;  // the last of this row or range
    if (++held == kPairsHeld || flush) {
      held = 0;
      V t[6];
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const V sum[2][6] = {{ui[0].ux, ui[0].uy, ui[0].uz, ui[0].wx, ui[0].wy, ui[0].wz},
                             {ui[NS - 1].ux, ui[NS - 1].uy, ui[NS - 1].uz, ui[NS - 1].wx,
                              ui[NS - 1].wy, ui[NS - 1].wz}};
        t[c] = both(sum[0][c], sum[1][c]);
        V S = reinterpret_cast<V *>(w.S[c])[lane];
        V C = reinterpret_cast<V *>(w.C[sizeof(R) == 4 ? c : 0])[lane];
        fold_in(S, C, t[c]);
        reinterpret_cast<V *>(w.S[c])[lane] = S;
        if (sizeof(R) == 4) reinterpret_cast<V *>(w.C[sizeof(R) == 4 ? c : 0])[lane] = C;
      }
#pragma unroll
      for (int q = 0; q < NS; q++) ui[q] = {zero, zero, zero, zero, zero, zero};
    }
    // exact - fast for the close pairs: usually no two flagged steps share a slot,
    // and each lane takes its own in turn, all side by side; else step by step.
    // Either way every sum gets its corrections in step order.  (Always step by
    // step: 500 batches of 60 13.3 us, 11.8 side by side; N = 200 in FP64 17.7,
    // 16.0.)
    unsigned st = __reduce_or_sync(0xffffffffu, near);
    const unsigned long long at = (unsigned long long)near << lane;  // bit k to k + lane
    const unsigned slots = (unsigned)at | (unsigned)(at >> nsl);
    const bool apart =
        st == 0u || diag ||
        (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(near)) ==
            __popc(__reduce_or_sync(0xffffffffu, slots & (0xffffffffu >> (32 - nsl))));
    while (st != 0u) {
      const unsigned from = apart ? near : st;
      const int k = __ffs(from) - 1;
      if (from != 0u && ((near >> k) & 1u)) {
        const int s = met(k);
        // which of the slots' pairs (NS q + h); FP32 takes the distances of all
        // four first, which spares most of the loads below
        unsigned which = (1u << (NS * NS)) - 1u;
        if constexpr (NS == 2) {
          which = 0u;
#pragma unroll
          for (int q = 0; q < NS; q++) {
            V d[3];
#pragma unroll
            for (int c = 0; c < 3; c++) d[c] = vi[q][c] - reinterpret_cast<const V *>(w.J[c])[s];
            const V r2 = vfma(d[2], d[2], vfma(d[0], d[0], d[1] * d[1]));
#pragma unroll
            for (int h = 0; h < NS; h++) which |= below4(lane_of(r2, h)) ? 1u << (NS * q + h) : 0u;
          }
        }
#pragma unroll 1
        for (; which != 0u; which &= which - 1u) {
          const int qh = __ffs(which) - 1;
          const int li = NS * lane + qh / NS, lj = NS * s + qh % NS;
          R pi[9], pj[9];
#pragma unroll
          for (int c = 0; c < 9; c++) {
            pi[c] = c < NV ? w.I[c < NV ? c : 0][li] : R(0);
            pj[c] = c < NV ? w.J[c < NV ? c : 0][lj] : R(0);
          }
          const R dx = pi[0] - pj[0], dy = pi[1] - pj[1], dz = pi[2] - pj[2];
          const R r2 = vfma(dz, dz, vfma(dx, dx, dy * dy));
          if (NS == 1 && !below4(r2)) continue;
          Vec6<R> o = {0, 0, 0, 0, 0, 0};
          pair_correct<R, WALL, ANG>(pi, pj, r2, o);
          const R ai[6] = {o.ux, o.uy, o.uz, o.wx, o.wy, o.wz};
#pragma unroll
          for (int c = 0; c < NC; c++)
            fold_in(w.S[c][li], w.C[sizeof(R) == 4 ? c : 0][li], ai[c]);
          if (!diag) {
            o = {0, 0, 0, 0, 0, 0};
            pair_correct<R, WALL, ANG>(pj, pi, r2, o);
            const R aj[6] = {o.ux, o.uy, o.uz, o.wx, o.wy, o.wz};
#pragma unroll
            for (int c = 0; c < NC; c++) w.A[c][lj] += aj[c];
          }
        }
      }
      if (apart) {
        near &= near - 1u;
        st = __any_sync(0xffffffffu, near != 0u) ? 1u : 0u;
      } else {
        st &= st - 1u;
        __syncwarp();
      }
    }
    __syncwarp();
    if (!diag) put(cur.k == 0 ? (size_t)cur.p : slot_cut + gw, w.A);
    if (flush) {
      if (sizeof(R) == 4) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
          V *S = reinterpret_cast<V *>(w.S[c]) + lane;
          *S = *S + reinterpret_cast<V *>(w.C[sizeof(R) == 4 ? c : 0])[lane];
        }
      }
      put(row_begun ? slot_row + (cur.batch * a.tpb + cur.I - a.row0) : slot_irow + gw,
          w.S);
    }
    __syncwarp();
    cur = nxt;
  }

  // After a wait that ran out the partials may be incomplete: what this block
  // would fold is NaN (for certain that part; it marks all of the pass), and the
  // host raises an error when it sees the flag.
  if (!grid_barrier_mono(a.bar, a.spins)) {
    if (threadIdx.x == 0) *a.err = 1;
    const int b_lo = a.row0 / a.tpb, b_hi = (a.row1 - 1) / a.tpb + 1;  // batches
    if (a.last) {
      for (size_t e = 3 * (size_t)b_lo * a.nper + threadIdx.x; e < 3 * (size_t)b_hi * a.nper;
           e += kPairsThreads) {
        if (!LMG_IN_BOUNDS(e < 3 * (size_t)a.N, 25, e)) continue;
        if (a.U) a.U[e] = R(NAN);
        if (ANG && a.W) a.W[e] = R(NAN);
      }
    } else {
      for (size_t e = 2 * (size_t)b_lo * a.tpb * EL + threadIdx.x;
           e < 2 * (size_t)b_hi * a.tpb * EL; e += kPairsThreads)
        a.acc[e] = R(NAN);
    }
    return;
  }

  // ---- fold the partials: one component of a tile at a time, by a warp or by
  // the block's four warps, each taking every fourth partial, sixteen loads ahead ----
  R (*red)[2][TS] = reinterpret_cast<R (*)[2][TS]>(&sm[0]);  // [warp][S, C][particle]
  using L = typename LaneTypes<R>::L;
  const int *cut_begin = a.cuts, *cut_warp = a.cuts + a.tiles + 1;
  // (a pass over a band of rows still touches every tile of its batch)
  const int t_lo = a.row0 / a.tpb * a.tpb, t_hi = ((a.row1 - 1) / a.tpb + 1) * a.tpb;
  auto fold_units = [&](auto share) {
    constexpr bool alone = decltype(share)::value == 1;
    constexpr int step = alone ? 1 : NW;
    const int sub = alone ? 0 : warp;
    const int stride = alone ? (int)gridDim.x * NW : (int)gridDim.x;
    for (int unit = alone ? gw : (int)blockIdx.x; unit < (t_hi - t_lo) * NC; unit += stride) {
      const int t = t_lo + unit / NC, comp = unit % NC;
      const int tb = t / a.tpb, tl = t - tb * a.tpb;  // batch, tile in it
      const L *src = reinterpret_cast<const L *>(a.part + comp * TS) + lane;
      R S[NS], C[NS];
#pragma unroll
      for (int q = 0; q < NS; q++) S[q] = C[q] = R(0);
      constexpr int UN = 16;
      // adds the partials slot(e), e = sub, sub + step, ... < n
      auto gather = [&](int n, auto slot) {
        for (int e0 = sub; e0 < n; e0 += UN * step) {
          L v[UN];
#pragma unroll
          for (int u = 0; u < UN; u++) {
            const int e = e0 + u * step;
            v[u] = L();
            if (e < n) {
              const size_t sl = slot(e);
              if (LMG_IN_BOUNDS((sl + 1) * EL <= a.part_elems, 23, sl))
                v[u] = __ldcg(src + sl * (EL / NS));
            }
          }
#pragma unroll
          for (int u = 0; u < UN; u++) {
#pragma unroll
            for (int q = 0; q < NS; q++) fold_in(S[q], C[q], lane_value(v[u], q));
          }
        }
      };
      // J side: rows I < tl of its batch in this pass
      const int I_lo = max(0, a.row0 - tb * a.tpb), I_hi = min(tl, a.row1 - tb * a.tpb);
      const int base = tb * ppb - P0 + tl;
      gather(I_hi - I_lo, [&](int e) {
        const int I = I_lo + e;
        return (size_t)(base + local_before(a.tpb, I) - I);
      });
      // I side: the row's own partial, then those of warps that began in it
      if (t >= a.row0 && t < a.row1) {
        const unsigned xs = (unsigned)nsl * (unsigned)(tb * ppb + local_before(a.tpb, tl) - P0);
        const unsigned xe = xs + (unsigned)nsl * (unsigned)(a.tpb - tl);
        const int w_lo = (int)(xs / a.per_warp), w_hi = (int)((xe - 1u) / a.per_warp);
        gather(w_hi - w_lo + 1, [&](int e) {
          return e == 0 ? slot_row + (t - a.row0) : slot_irow + w_lo + e;
        });
      }
      // J side of tile pairs that a warp began in
      const int q_lo = __ldg(cut_begin + t);
      gather(__ldg(cut_begin + t + 1) - q_lo,
             [&](int e) { return slot_cut + __ldg(cut_warp + q_lo + e); });
      auto finish = [&](int p, R s, R c) {
        const size_t o = ((size_t)t * NC + comp) * TS + p;
        if (!a.first) {
          fold_in(s, c, a.acc[2 * o]);
          c += a.acc[2 * o + 1];
        }
        if constexpr (!alone) {
#pragma unroll
          for (int q = 1; q < NW; q++) {
            fold_in(s, c, red[q][0][p]);
            c += red[q][1][p];
          }
        }
        if (!a.last) {
          a.acc[2 * o] = s;
          a.acc[2 * o + 1] = c;
          return;
        }
        const int l = tl * NS * nsl + p, i = tb * a.nper + l;
        if (p >= NS * nsl || l >= a.nper || !LMG_IN_BOUNDS(i < a.N, 24, i)) return;
        s += c;
        if (WALL) {
          const R z = mul_rn(a.pos[3 * (size_t)i + 2], a.inv_a);
          s *= z < R(0) ? R(0) : (z > R(1) ? R(1) : z);
        }
        if (comp < 3) {
          if (a.U) a.U[3 * (size_t)i + comp] = s;
        } else if (a.W) {
          a.W[3 * (size_t)i + (comp - 3)] = a.k.sW * s;
        }
      };
      if constexpr (alone) {
#pragma unroll
        for (int q = 0; q < NS; q++) finish(NS * lane + q, S[q], C[q]);
      } else {
#pragma unroll
        for (int q = 0; q < NS; q++) {
          red[warp][0][NS * lane + q] = S[q];
          red[warp][1][NS * lane + q] = C[q];
        }
        __syncthreads();
        for (int p = threadIdx.x; p < TS; p += kPairsThreads)
          finish(p, red[0][0][p], red[0][1][p]);
        __syncthreads();
      }
    }
  };
  if (a.share == 1) fold_units(std::integral_constant<int, 1>());
  else fold_units(std::integral_constant<int, NW>());
}

template <class R> size_t pairs_smem(bool ang) {
  return kPairsThreads / 32 * (ang ? sizeof(PairsWarp<R, true>) : sizeof(PairsWarp<R, false>));
}

template <class R, bool FULL> const void *pairs_kernel_of(bool wall, bool ang) {
  if (wall) return ang ? (const void *)mdot_pairs_kernel<R, true, true, FULL>
                       : (const void *)mdot_pairs_kernel<R, true, false, FULL>;
  return ang ? (const void *)mdot_pairs_kernel<R, false, true, FULL>
             : (const void *)mdot_pairs_kernel<R, false, false, FULL>;
}
template <class R> const void *pairs_kernel(bool wall, bool ang, bool full) {
  return full ? pairs_kernel_of<R, true>(wall, ang) : pairs_kernel_of<R, false>(wall, ang);
}

}  // namespace

template <class R>
void mdot_pairs_plan_tables(int N, int nper, bool ang, long long resident, int force_warps,
                            size_t max_part, PairsPlan &p) {
  p = PairsPlan{};
  if (N <= 0 || nper <= 0 || N % nper != 0 || resident < 1) return;
  constexpr int TS = kPairsTile<R>;
  const int EL = (ang ? 6 : 3) * TS;
  const int tpb = (nper + TS - 1) / TS, nb = N / nper;
  constexpr int NS = kPairsSlot<R>;
  const long long rows = (long long)nb * tpb;
  // 32-bit tile pair numbers; beyond a million particles a batch (FP32) the
  // passes' tables would grow past what they save
  if (tpb > 16384 || rows * (tpb + 1) / 2 >= (1LL << 30)) return;
  // The slots of a tile in use: where there is work for every warp, as few as
  // hold the batch in as many tiles, so that no tile is mostly padding (333
  // particles: 6 tiles of 28 slots of two).  64 batches of 333 17.7 -> 16.9 us,
  // above a wall with torques 48.0 -> 44.0; 64 of 100 in FP64 61 -> 52.  Where
  // there is not, ranges of four steps fit 32 better (30 batches of 100 8.0 us,
  // 8.8 with 25 slots).
  const long long wpb = kPairsThreads / 32;
  const int S = 16 * rows * (tpb + 1) > kPairsMinSteps * wpb * resident
                    ? ((nper + tpb - 1) / tpb + NS - 1) / NS
                    : 32;
  p.N = N;
  p.nper = nper;
  p.tpb = tpb;
  p.slots = S;
  p.ang = ang;
  const size_t cap = max_part > 0 ? max_part : kPairsMaxPart;
  // tile pairs of a pass: at least one row's, at most what the scratch holds
  // (the rows' and warps' slots come on top) and the steps' 31-bit count allows
  const long long max_pairs =
      std::min(std::max(1LL, (long long)(cap / EL)), 1LL << 25);
  for (int r = 0; r < rows;) {
    int r1 = r;
    long long n = 0;
    while (r1 < rows) {
      const long long len = tpb - r1 % tpb;
      if (r1 > r && n + len > max_pairs) break;
      n += len;
      r1++;
    }
    // a pass is whole batches or a band of one: it ends with the batch it
    // began inside, and otherwise not inside a later one
    if (r % tpb != 0) r1 = std::min(r1, (r / tpb + 1) * tpb);
    if (r1 < rows && r1 % tpb != 0 && r1 - r1 % tpb > r) r1 -= r1 % tpb;
    PairsPass q;
    q.row0 = r;
    q.row1 = r1;
    const long long pairs = pairs_before(tpb, r1) - pairs_before(tpb, r);
    const long long W = S * pairs;
    q.steps = (unsigned)W;
    long long nw = std::min(wpb * resident, (W + kPairsMinSteps - 1) / kPairsMinSteps);
    if (force_warps > 0) nw = std::min<long long>(nw, force_warps);
    q.per_warp = (unsigned)((W + nw - 1) / nw);
    q.warps = (int)((W + q.per_warp - 1) / q.per_warp);
    q.grid = (int)((q.warps + wpb - 1) / wpb);
    // warps that begin inside a tile pair off the diagonal, by its column
    q.cut_off = p.cuts.size();
    std::vector<int> col(q.warps, -1);
    std::vector<int> count(rows + 1, 0);
    int row = r;
    long long start = 0;  // first tile pair of `row` in this pass
    for (int w = 1; w < q.warps; w++) {
      const long long x = (long long)w * q.per_warp, pr = x / S;
      while (start + (tpb - row % tpb) <= pr) {
        start += tpb - row % tpb;
        row++;
      }
      const int J = row + (int)(pr - start);
      if (x % S != 0 && J != row) {
        col[w] = J;
        count[J + 1]++;
      }
    }
    for (long long t = 0; t < rows; t++) count[t + 1] += count[t];
    const size_t base = p.cuts.size();
    p.cuts.insert(p.cuts.end(), count.begin(), count.end());
    p.cuts.resize(base + rows + 1 + count[rows]);
    int *warps = p.cuts.data() + base + rows + 1;
    std::vector<int> fill(count.begin(), count.end() - 1);
    for (int w = 1; w < q.warps; w++)
      if (col[w] >= 0) warps[fill[col[w]]++] = w;
    p.part_elems = std::max(p.part_elems, (size_t)EL * (size_t)(pairs + (r1 - r) + 2 * q.warps));
    p.passes.push_back(q);
    p.carries = p.carries || r1 % tpb != 0;
    r = r1;
  }
  // bands of one batch carry their sums; passes of whole batches need not
  p.acc_elems = p.passes.size() > 1 ? 2 * (size_t)rows * EL : 0;
  p.ok = true;
}

template <class R>
cudaError_t mdot_pairs_plan(int N, int nper, bool wall, bool ang, int num_sms, int force_warps,
                            size_t max_part, PairsPlan &p) {
  int per_sm = 1 << 30;
  for (const bool full : {true, false}) {
    const void *k = pairs_kernel<R>(wall, ang, full);
    int n = 0;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)pairs_smem<R>(ang));
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kPairsThreads, pairs_smem<R>(ang));
    if (e != cudaSuccess) return e;
    per_sm = std::min(per_sm, n);
  }
  const long long tpb = (nper + kPairsTile<R> - 1) / kPairsTile<R>;
  const long long steps = 16 * tpb * (tpb + 1) * (N / nper);
  if (steps < pairs_few_steps(ang, tpb) * per_sm * num_sms * (kPairsThreads / 32)) per_sm = std::min(per_sm, 2);
  mdot_pairs_plan_tables<R>(N, nper, ang, (long long)per_sm * num_sms, force_warps, max_part, p);
  p.wall = wall;
  return cudaSuccess;
}

template <class R>
cudaError_t mdot_pairs_launch(const PairsPlan &p, const int *cuts, const R *pos, const R *F,
                              const R *T, R *U, R *W, R inv_a, PairScale<R> k, R *part, R *acc,
                              unsigned long long *bar, int *err, cudaStream_t stream) {
  if (!p.ok) return cudaErrorInvalidValue;
  for (size_t q = 0; q < p.passes.size(); q++) {
    const PairsPass &s = p.passes[q];
    PairsArgs<R> a{};
    a.pos = pos;
    a.F = F;
    a.T = T;
    a.U = U;
    a.W = W;
    a.N = p.N;
    a.nper = p.nper;
    a.tpb = p.tpb;
    a.slots = p.slots;
    a.row0 = s.row0;
    a.row1 = s.row1;
    a.tiles = p.N / p.nper * p.tpb;
    a.steps = s.steps;
    a.per_warp = s.per_warp;
    a.warps = s.warps;
    // a batch's first and last pass
    a.first = s.row0 % p.tpb == 0;
    a.last = s.row1 % p.tpb == 0;
    a.inv_a = inv_a;
    a.k = k;
    a.part = part;
    a.part_elems = p.part_elems;
    a.acc = acc;
    a.cuts = cuts + s.cut_off;
    a.wide = (p.nper % 2 == 0 || p.nper == p.N) &&
             ((reinterpret_cast<uintptr_t>(pos) | reinterpret_cast<uintptr_t>(F) |
               reinterpret_cast<uintptr_t>(T)) & 7) == 0;
    a.bar = bar + q;
    a.spins = g_barrier_spins.load() < 0 ? kMonoSpins : (int)g_barrier_spins.load();
    a.err = err;
    // Folding: rounds of loads one after the other (16 partials a warp, about
    // as much again to start and finish a component of a tile) with four warps
    // on each, or one.  64 batches of 333 (10 partials a tile): 24.0 us with
    // four, 17.9 with one, wall with torques 63.7 and 51.2.  With many partials
    // four are as good or better (N = 16384 wall forces, 272 a tile: 326.9
    // and 328.5 us).
    {
      const long long NW = kPairsThreads / 32, nc = p.ang ? 6 : 3;
      const long long tiles = ((s.row1 - 1) / p.tpb + 1 - s.row0 / p.tpb) * (long long)p.tpb;
      const long long n = p.tpb + 1 + 2LL * s.warps / tiles, units = tiles * nc;
      auto up = [](long long x, long long y) { return (x + y - 1) / y; };
      const long long four = up(units, s.grid) * (up(n, 16 * NW) + 1);
      const long long one = up(units, NW * s.grid) * (up(n, 16) + 1);
      a.share = n <= 64 && one < four ? 1 : (int)NW;
    }
    void *params[] = {(void *)&a};
    count_launch();
    const cudaError_t e =
        cudaLaunchCooperativeKernel(pairs_kernel<R>(p.wall, p.ang, p.slots == 32), dim3(s.grid),
                                    dim3(kPairsThreads), params, pairs_smem<R>(p.ang), stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// this translation unit's bounds status (the checked build; 0 otherwise)
#define LMG_STATUS_FN(tag) bounds_status_pairs_##tag
#define LMG_STATUS_NAME(tag) LMG_STATUS_FN(tag)
unsigned long long LMG_STATUS_NAME(LMG_REAL)(bool reset) { return bounds_status_here(reset); }

template void mdot_pairs_plan_tables<LMG_REAL>(int, int, bool, long long, int, size_t,
                                               PairsPlan &);
template cudaError_t mdot_pairs_plan<LMG_REAL>(int, int, bool, bool, int, int, size_t,
                                               PairsPlan &);
template cudaError_t mdot_pairs_launch<LMG_REAL>(const PairsPlan &, const int *, const LMG_REAL *,
                                                 const LMG_REAL *, const LMG_REAL *, LMG_REAL *,
                                                 LMG_REAL *, LMG_REAL, PairScale<LMG_REAL>,
                                                 LMG_REAL *, LMG_REAL *, unsigned long long *,
                                                 int *, cudaStream_t);

}  // namespace lmg
