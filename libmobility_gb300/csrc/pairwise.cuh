// Pair physics of the NBody Rotne-Prager-Yamakawa mobility, open boundary and
// single bottom wall, in the form the unordered-pair kernel uses
// (mdot_pairs.cuh): coefficients of a pair once, applied to both particles.
//
// Physics follows libMobility solvers/NBody/extra/hydrodynamicKernels.cuh:
//   RPY_UF :41-57, RPY_WT :63-86, RPY_UT/RPY_WF :89-118 (open-space blocks),
//   wallCorrection_UF :187-249, _WT :253-282, _UT :287-319, _WF :324-359,
//   BottomWall::dotProduct :362-441 (damping b_i b_j, heights clamped at a,
//   image vector r_ij + 2 h_j z, UT evaluated with -r_ij + 2 h_i z).
//
// Representation chosen here (not the reference's entry-by-entry matrices):
//   * lengths are divided by the hydrodynamic radius a when a source or a
//     target is loaded;
//   * forces are multiplied by 3/4 t0 and torques by rt0 when loaded, and
//     angular velocities by rt0 / (3/4 t0) when stored.  What is left between
//     them are the blocks with prefactors 4/3 (U from F) and 1 (the others,
//     r0 (3/4 t0) / rt0^2 = 1), so a pair's constants are numbers, and the
//     leading ones of U from F are 1;
//   * the wall damping b_i b_j is part of the same two factors (b_j at the
//     load of a source, b_i at the store of a target).
//
// Wall pairs.  With rho = (dx, dy), the plane through both particles and the
// wall normal z is a symmetry plane, so each block of a pair (direct part and
// image together) is one of two forms with five or four coefficients,
//
//   U from F, W from T:   al I_xy + be rho rho^T + ga rho z^T + de z rho^T + ep z z^T
//   W from F:             aj J + n (bj rho + cj z)^T + g z n^T
//
// where n = (dy, -dx) and J F = (Fy, -Fx).  Summing the reference's polynomials
// into these coefficients (with h_j = hh Rz, h_j h_i = hh (1 - hh) Rz^2) leaves
// no division, and collects the terms of the direct part and of the image
// before they meet a vector: 10 multiply-adds apply a translational block.
// The mobility is symmetric: for the pair taken the other way round (j the
// target) the blocks are the transposes, so the same coefficients serve both
// particles; U from T of (i, j) is the transpose of W from F of (j, i), whose
// coefficients (a -> -aj with X's sign, h_j -> h_i) are carried along.
//
// Cost.  In FP32 an instruction on the FMA pipe is bound by the registers it
// reads: measured per scheduler, a packed multiply-add of three different
// register pairs takes 3.1 cycles, one with a constant or with an operand the
// instruction before it read 2.1, a packed product or sum 2.1 (the pipe itself
// needs 2).  So constants are literals, signs are folded into operands (free),
// and fewer operations pay even where a multiply-add could absorb them.
#pragma once
#include <cuda_runtime.h>

#include "pack2.cuh"

namespace lmg {

// a b + c in one rounding, and a constant, for float, double and F2 (two pairs
// in packed FP32 instructions)
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) { return fma2(a, b, c); }
__device__ __forceinline__ F2 operator-(F2 a) { return neg2(a); }
template <class V> __device__ __forceinline__ V cst(double x);
template <> __device__ __forceinline__ float cst<float>(double x) { return (float)x; }
template <> __device__ __forceinline__ double cst<double>(double x) { return x; }
template <> __device__ __forceinline__ F2 cst<F2>(double x) { return bc((float)x); }

// Reciprocal square root of a normal number (squared distances clamped at 4).
// FP32: the hardware approximation without the subnormal handling.
__device__ __forceinline__ float rsq(float x) { return rsqrt_normal<float>(x); }
__device__ __forceinline__ F2 rsq(F2 x) { return mk2(rsq(x.v.x), rsq(x.v.y)); }
// FP64: the hardware's approximation y0 from the upper word, then one step of
// Householder's third-order method for y^-2 = x: with e = 1 - x y0^2,
// y = y0 (1 + e/2 + 3/8 e^2), relative error 5/16 e^3.  Five operations on the
// FP64 pipe, which bounds every FP64 pair kernel.
__device__ __forceinline__ double rsq(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  const double r = fma(y * e, fma(0.375, e, 0.5), y);
  return __double2hiint(y) == 0 ? 0.0 : r;  // 0 where x overflowed
}

// r^2 < 4 and max(r^2, 4).  FP64: by the upper word's bits (integer pipe; a
// comparison would take a slot of the FP64 pipe).
__device__ __forceinline__ bool below4(float r2) { return r2 < 4.0f; }
__device__ __forceinline__ bool below4(double r2) { return __double2hiint(r2) < 0x40100000; }
__device__ __forceinline__ float clamp4(float r2) { return fmaxf(r2, 4.0f); }
__device__ __forceinline__ double clamp4(double r2) { return below4(r2) ? 4.0 : r2; }
__device__ __forceinline__ F2 clamp4(F2 r2) { return mk2(clamp4(r2.v.x), clamp4(r2.v.y)); }
__device__ __forceinline__ bool any_below4(float r2) { return below4(r2); }
__device__ __forceinline__ bool any_below4(double r2) { return below4(r2); }
__device__ __forceinline__ bool any_below4(F2 r2) { return fminf(r2.v.x, r2.v.y) < 4.0f; }

// Factors of the loads and stores (see above): F times sF, T times sT, U as
// summed, W times sW.
template <class R> struct PairScale {
  R sF, sT, sW;
};
template <class R> inline PairScale<R> make_pair_scale(double t0, double rt0) {
  return {R(0.75 * t0), R(rt0), R(rt0 / (0.75 * t0))};
}

// Coefficients of one pair, both directions; the second and third group with
// angular velocities (ANG) only.
template <class V> struct PairCoef {
  V al, be, ga, de, ep;       // U from F
  V alw, bew, gaw, dew, epw;  // W from T
  // W from F of (i, j): aj, bj, ncj = -cj; of (j, i): mi = -ai, bi, nci = -ci
  V g, aj, bj, ncj, mi, bi, nci;
};

// Open space, separated pair (r >= 2a; the caller clamps r^2 at 4 and corrects
// closer pairs, near_diff): f I + G d d^T in al, be (U from F) and alw, bew
// (W from T), the coupling c (F x d) in g.
template <class V, bool ANG>
__device__ __forceinline__ void open_coeffs(V ir, PairCoef<V> &c) {
  const V ir2 = ir * ir;
  const V ir3 = ir2 * ir;
  const V ir5 = ir3 * ir2;
  c.al = vfma(cst<V>(2.0 / 3.0), ir3, ir);
  c.be = vfma(cst<V>(-2.0), ir5, ir3);
  if (ANG) {
    c.alw = cst<V>(-0.5) * ir3;
    c.bew = cst<V>(1.5) * ir5;
    c.g = ir3;
  }
}

// Bottom wall, separated pair: direct part and image (Swan & Brady 2007).
// ir = 1/|d| (clamped), i = 1/|R| with R = (dx, dy, Rz), Rz = hi + hj.
template <class V, bool ANG>
__device__ __forceinline__ void wall_coeffs(V dz, V Rz, V hi, V hj, V ir, V i, PairCoef<V> &c) {
  const V ir2 = ir * ir, ir3 = ir2 * ir, ir5 = ir3 * ir2;
  const V i2 = i * i, i3 = i2 * i, i5 = i3 * i2;
  const V ez = Rz * i, q = ez * ez;
  const V Rz5 = Rz * i5;
  const V g = ir3 - i3;
  {
    const V H = hi * hj;
    const V K = vfma(vfma(cst<V>(70.0 / 3.0), i2, cst<V>(-10.0)), q,
                     vfma(cst<V>(6.0), H, cst<V>(2.0)));
    const V y = vfma(cst<V>(-2.0), ir5, g);
    const V zy = dz * y;
    const V fa = vfma(cst<V>(2.0 / 3.0), ir3, ir - i);
    const V t = vfma(cst<V>(-2.0), H, cst<V>(-2.0 / 3.0));
    const V v = Rz5 * vfma(cst<V>(-10.0), i2, K);
    c.be = vfma(i5, vfma(cst<V>(-10.0 / 3.0), i2, K), y);
    c.ga = zy - v;
    c.de = zy + v;
    c.al = vfma(i3, vfma(cst<V>(2.0), q, t),
                vfma(i5, vfma(cst<V>(-10.0 / 3.0), q, cst<V>(2.0 / 3.0)), fa));
    c.ep = vfma(i3, vfma(-q, K + cst<V>(2.0), t),
                vfma(i5, vfma(cst<V>(20.0), q, cst<V>(-2.0)), vfma(dz, zy, fa)));
  }
  if (ANG) {
    const V Z = cst<V>(1.5) * ir5, Zd = Z * dz, s = cst<V>(-0.5) * ir3;
    c.alw = vfma(i3, vfma(cst<V>(-6.0), q, cst<V>(3.5)), s);
    c.bew = vfma(cst<V>(-4.5), i5, Z);
    c.gaw = vfma(cst<V>(-1.5), Rz5, Zd);
    c.dew = vfma(cst<V>(1.5), Rz5, Zd);
    c.epw = vfma(i3, vfma(cst<V>(-1.5), q, cst<V>(0.5)), vfma(Zd, dz, s));
    const V tt = dz * g;
    c.g = g;
    c.aj = vfma(cst<V>(-2.0), Rz5, tt);
    c.mi = vfma(cst<V>(2.0), Rz5, tt);
    const V N6 = cst<V>(-6.0) * i5, R10 = Rz5 * (cst<V>(10.0) * i2);
    c.bj = vfma(N6, hj, R10);
    c.bi = vfma(N6, hi, R10);
    const V m2 = vfma(cst<V>(-2.0), i5, g);
    c.nci = vfma(Rz, c.bi, m2);
    c.ncj = vfma(Rz, c.bj, m2);
  }
}

template <class V> struct Vec6 {
  V ux, uy, uz, wx, wy, wz;
};

// Adds to one particle of a wall pair, o, what the other one's force v[3..5]
// and torque v[6..8] give it.  The two directions differ in the arguments
// alone: ga and de, gaw and dew change places, and the couplings take the
// other set of coefficients (A: U from T, B: W from F).
template <class V, bool ANG>
__device__ __forceinline__ void wall_apply(const PairCoef<V> &c, V dx, V dy, V ga, V de, V gaw,
                                           V dew, V A, V At, V Ac, V Ag, V B, V Bt, V Bc, V Bg,
                                           const V (&v)[9], Vec6<V> &o) {
  const V s = vfma(dx, v[3], dy * v[4]);
  V tr = vfma(c.be, s, ga * v[5]);
  if constexpr (!ANG) {
    o.ux = vfma(c.al, v[3], vfma(tr, dx, o.ux));
    o.uy = vfma(c.al, v[4], vfma(tr, dy, o.uy));
    o.uz = vfma(de, s, vfma(c.ep, v[5], o.uz));
  } else {
    const V pT = vfma(dy, v[6], -(dx * v[7]));
    const V tz = Ag * v[8];
    tr = vfma(At, pT, tr);
    o.ux = vfma(tz, dy, vfma(A, v[7], vfma(c.al, v[3], vfma(tr, dx, o.ux))));
    o.uy = vfma(-tz, dx, vfma(-A, v[6], vfma(c.al, v[4], vfma(tr, dy, o.uy))));
    o.uz = vfma(Ac, pT, vfma(de, s, vfma(c.ep, v[5], o.uz)));
    const V sT = vfma(dx, v[6], dy * v[7]);
    const V p = vfma(dy, v[3], -(dx * v[4]));
    const V tw = vfma(c.bew, sT, gaw * v[8]);
    const V tn = vfma(Bt, s, Bc * v[5]);
    o.wx = vfma(tn, dy, vfma(B, v[4], vfma(c.alw, v[6], vfma(tw, dx, o.wx))));
    o.wy = vfma(-tn, dx, vfma(-B, v[3], vfma(c.alw, v[7], vfma(tw, dy, o.wy))));
    o.wz = vfma(Bg, p, vfma(dew, sT, vfma(c.epw, v[8], o.wz)));
  }
}

// Open space: f F + G (d.F) d and, with e = c d for particle i and -c d for j,
// the coupling F x e.
template <class V, bool ANG>
__device__ __forceinline__ void open_apply(const PairCoef<V> &c, V ex, V ey, V ez, V dx, V dy,
                                           V dz, const V (&v)[9], Vec6<V> &o) {
  const V s = c.be * vfma(dx, v[3], vfma(dy, v[4], dz * v[5]));
  o.ux = vfma(c.al, v[3], vfma(s, dx, o.ux));
  o.uy = vfma(c.al, v[4], vfma(s, dy, o.uy));
  o.uz = vfma(c.al, v[5], vfma(s, dz, o.uz));
  if constexpr (ANG) {
    const V t = c.bew * vfma(dx, v[6], vfma(dy, v[7], dz * v[8]));
    o.wx = vfma(c.alw, v[6], vfma(t, dx, o.wx));
    o.wy = vfma(c.alw, v[7], vfma(t, dy, o.wy));
    o.wz = vfma(c.alw, v[8], vfma(t, dz, o.wz));
    o.ux = vfma(v[7], ez, vfma(-v[8], ey, o.ux));
    o.uy = vfma(v[8], ex, vfma(-v[6], ez, o.uy));
    o.uz = vfma(v[6], ey, vfma(-v[7], ex, o.uz));
    o.wx = vfma(v[4], ez, vfma(-v[5], ey, o.wx));
    o.wy = vfma(v[5], ex, vfma(-v[3], ez, o.wy));
    o.wz = vfma(v[3], ey, vfma(-v[4], ex, o.wz));
  }
}

// Exact minus separated-form coefficients of the direct part of an overlapping
// pair, 0 < r < 2 (units of a), the separated form being the one at r = 2.
template <class R, bool ANG>
__device__ __forceinline__ void near_diff(R r2, R ir, PairCoef<R> &c) {
  const R r = r2 * ir;
  c.al = vfma(R(-3.0 / 8.0), r, R(0.75));  // 4/3 (1 - 9/32 r - 7/16)
  c.be = vfma(R(0.125), ir, R(-0.0625));   // 4/3 (3/32 / r - 3/64)
  if (ANG) {
    c.alw = vfma(r, vfma(R(5.0 / 64.0), r2, R(-27.0 / 32.0)), R(1.0625));
    c.bew = vfma(R(9.0 / 32.0), ir, vfma(R(-3.0 / 64.0), r, R(-3.0 / 64.0)));
    c.g = vfma(R(-3.0 / 16.0), r, R(0.5 - 0.125));
  }
}

// The self pair: self mobilities, and above a wall (WALL) the self terms B1,
// B2, B3 (:190-202, :256-261, :290-294, :327-331) at height h.
template <class R, bool WALL, bool ANG>
__device__ __forceinline__ void self_pair(R h, const R (&v)[9], Vec6<R> &o) {
  R fxy = R(4.0 / 3.0), fz = R(4.0 / 3.0), txy = R(1), tz = R(1), cc = R(0);
  if (WALL) {
    const R ih = R(1) / h;
    const R ih2 = ih * ih, ih3 = ih2 * ih, ih5 = ih3 * ih2;
    fxy += R(-1.0 / 12.0) * (R(9) * ih - R(2) * ih3 + ih5);
    fz += R(-1.0 / 6.0) * (R(9) * ih - R(4) * ih3 + ih5);
    txy += R(-5.0 / 16.0) * ih3;
    tz += R(-0.125) * ih3;
    cc = R(0.125) * (ih2 * ih2);
  }
  o.ux += fxy * v[3]; o.uy += fxy * v[4]; o.uz += fz * v[5];
  if (ANG) {
    o.wx += txy * v[6]; o.wy += txy * v[7]; o.wz += tz * v[8];
    o.ux += cc * v[7]; o.uy -= cc * v[6];
    o.wx -= cc * v[4]; o.wy += cc * v[3];
  }
}

// One unordered pair in the fast form: the separated formulas at max(r^2, 4),
// finite and O(1) for an overlapping pair, exact for r >= 2a.  Adds to oi what
// j's force and torque give particle i and to oj the converse; returns r^2.
// v = x, y, z, F, T (T unused without ANG).  V: float, double or F2.
template <class V, bool WALL, bool ANG>
__device__ __forceinline__ V pair_both(const V (&vi)[9], const V (&vj)[9], Vec6<V> &oi,
                                       Vec6<V> &oj) {
  const V dx = vi[0] - vj[0], dy = vi[1] - vj[1], dz = vi[2] - vj[2];
  PairCoef<V> c;
  V r2;
  if constexpr (WALL) {
    const V sxy = vfma(dx, dx, dy * dy);
    r2 = vfma(dz, dz, sxy);
    const V Rz = vi[2] + vj[2];
    wall_coeffs<V, ANG>(dz, Rz, vi[2], vj[2], rsq(clamp4(r2)), rsq(vfma(Rz, Rz, sxy)), c);
    wall_apply<V, ANG>(c, dx, dy, c.ga, c.de, c.gaw, c.dew, c.mi, c.bi, c.nci, -c.g, c.aj, c.bj,
                       -c.ncj, c.g, vj, oi);
    wall_apply<V, ANG>(c, dx, dy, c.de, c.ga, c.dew, c.gaw, -c.aj, c.bj, -c.ncj, c.g, -c.mi, c.bi,
                       c.nci, -c.g, vi, oj);
  } else {
    r2 = vfma(dx, dx, vfma(dy, dy, dz * dz));
    open_coeffs<V, ANG>(rsq(clamp4(r2)), c);
    V ex, ey, ez;
    if (ANG) { ex = c.g * dx; ey = c.g * dy; ez = c.g * dz; }
    open_apply<V, ANG>(c, ex, ey, ez, dx, dy, dz, vj, oi);
    if constexpr (ANG) open_apply<V, ANG>(c, -ex, -ey, -ez, dx, dy, dz, vi, oj);
    else open_apply<V, ANG>(c, ex, ey, ez, dx, dy, dz, vi, oj);
  }
  return r2;
}

// Exact minus fast, for target i of a pair with r^2 < 4 that was added in the
// fast form (both are O(1) there, so the difference is accurate); the image of
// an overlapping pair is the same in both.  A pair at r = 0 is the self pair
// (or a coincident one, taken as the reference takes it).
template <class R, bool WALL, bool ANG>
__device__ __forceinline__ void pair_correct(const R (&vi)[9], const R (&vj)[9], R r2,
                                             Vec6<R> &o) {
  if (r2 > R(0)) {
    const R dx = vi[0] - vj[0], dy = vi[1] - vj[1], dz = vi[2] - vj[2];
    PairCoef<R> c;
    near_diff<R, ANG>(r2, rsqrt(r2), c);
    open_apply<R, ANG>(c, ANG ? c.g * dx : R(0), ANG ? c.g * dy : R(0), ANG ? c.g * dz : R(0), dx,
                       dy, dz, vj, o);
  } else {
    Vec6<R> s = {0, 0, 0, 0, 0, 0}, f = {0, 0, 0, 0, 0, 0}, unused = {0, 0, 0, 0, 0, 0};
    self_pair<R, WALL, ANG>(vi[2], vj, s);
    pair_both<R, WALL, ANG>(vi, vj, f, unused);
    o.ux += s.ux - f.ux; o.uy += s.uy - f.uy; o.uz += s.uz - f.uz;
    o.wx += s.wx - f.wx; o.wy += s.wy - f.wy; o.wz += s.wz - f.wz;
  }
}

}  // namespace lmg
