// srt_wide.cuh — one ray traced by a whole warp, in FP64 or in double-float
// (dd) arithmetic: the re-trace of the MIXED form's flagged rays and the FP64
// form of small ray ranges (kernels in srt_retrace.cu).
//
// What bounds it: a warp's FP64 instruction takes 64 cycles on this GPU
// whether one lane or 32 are active, FP64 instructions of one warp do not
// overlap (a dependent chain and four independent ones both ran at 64.1 cycles
// per instruction), and an SM retires one warp instruction per 19 cycles
// however many warps it holds (measured with a DFMA loop, 1 to 8 warps per SM,
// 1 to 32 active lanes). So a short list's time is the number of FP64
// instructions on a warp's path, and a long list's their number per ray. The
// right-hand side (four tricubic interpolations and ~250 further operations)
// is therefore cut into phases in which every lane does the same operation on
// its own operands, taken from and left in a warp's scratch in shared memory:
//   positions and cells   6 lanes  one axis of the centred / staggered grid
//   tap loads             32 lanes 8 lanes per field, two rows of 4 taps each
//   weights               24 lanes one tap of one axis set: value, d, d2 by
//                                  Horner with the lane's coefficients (6 ops)
//   frame                 13 lanes the nine components of n, e1, e2 and the
//                                  dA > 1/2 branch's four quotients: one
//                                  square root and one division in all
//   x, y, z passes        32 lanes 6, 3 and 1-2 four-term chains per lane
//   right-hand side       six rounds of dot products and linear combinations
//   RK4                   lane j holds component j of the state
// ~104 FP64 instructions per stage against ~730 for the four-lane groups this
// replaces (one field per lane, the rest of the right-hand side repeated on
// each).
//
// Every value is formed by the operations rhs_fp64 (srt_scheme.cuh) uses, in
// the same order, written as explicit fused chains in both, so the FP64 maps
// are the one-lane form's bit for bit. The phases are plain functions of
// (lane, scratch), so the host builds and checks them lane by lane.
#pragma once
#include "srt_scheme.cuh"

namespace srt {

// ---------------------------------------------------------------- scratch

// Elements of R in a warp's scratch. Offsets below 256 fit the packed operand
// tables of the right-hand side's rounds.
enum {
  kWsU = 0,      // n, e1, e2
  kWsQuo = 9,    // the four quotients of the dA > 1/2 branch (0 where it is off)
  kWsOne = 13,   // 1, 1, 1
  kWsZero = 16,  // 0
  kWsNeg1 = 17,
  kWsNeg2 = 18,
  kWsTwo = 19,
  kWsFour = 20,
  kWsY = 22,       // stage state (19)
  kWsTri = 41,     // per field (B_x, B_y, B_z, phi): value, gradient, full Hessian (13)
  kWsTriStride = 13,
  kWsD1 = 93,      // round 1 (29)
  kWsD2 = 122,     // round 2 (16)
  kWsD3 = 138,     // round 3 (12)
  kWsD4 = 150,     // round 4 (3)
  kWsD5 = 153,     // round 5 (5)
  kWsT = 158,      // offsets in the cell: centred x, y, z, staggered x, y, z
  kWsW = 164,      // weights: 6 axis sets x (w, g, h) x 4 taps
  kWsX = 236,      // x pass: 4 fields x 16 rows x (value, d, d2)
  kWsYp = 428,     // y pass: 4 fields x 4 slices x (a, ay, ayy, ax, axy, axx)
  kWsSize = 524,
  // five warps per ray (FieldLane): each field's own weights and offsets
  kWsWf = 524,  // 4 fields x 3 axes x (w, g, h) x 4 taps
  kWsTf = 668,  // 4 fields x 3 axes
  kWsBlockSize = 680
};

// Operands of the rounds, one 32-bit word per lane and round.
//   dot rounds 1, 3, 4: A offset, A stride, B offset, B stride (three terms)
//   round 2: X, Y, Z, Z' of X + beta Y + gamma (Z + Z')
//   round 5: X, beta, Y, Z of X + beta Y + Z / 2 (Z = 0 but for P_perp:H)
//   round 6: A, B, C, D of A B + C D + E, with E and the signs in `e6`
struct WideTables {
  uint32_t r1[32], r2[32], r3[32], r4[32], r5[32], r6[32], e6[32];
};

constexpr uint32_t wide_pack(int a, int b, int c, int d) {
  return (uint32_t)a | ((uint32_t)b << 8) | ((uint32_t)c << 16) | ((uint32_t)d << 24);
}

constexpr int kWideNegB = 1, kWideNegD = 2, kWideNegE = 4;  // signs in e6, above bit 8

constexpr WideTables make_wide_tables() {
  WideTables t = {};
  const int n = kWsU, a = kWsU + 3, b = kWsU + 6;
  const int idle = wide_pack(kWsZero, 0, kWsZero, 0);
  const int phi = kWsTri + 3 * kWsTriStride;
  const int sym[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  for (int l = 0; l < 32; ++l) {
    t.r1[l] = t.r3[l] = t.r4[l] = idle;
    t.r2[l] = t.r5[l] = t.r6[l] = wide_pack(kWsZero, kWsZero, kWsZero, kWsZero);
    t.e6[l] = kWsZero;
  }
  // round 1. 0-2: grad B_c . n; 3-11: (Hess B_c n)_i; 12-14: (Hess phi n)_i;
  // 15: grad phi . n; 16-18: (n . grad B)_i; 19-24: sum_c n_c Hess B_c (xx xy
  // xz yy yz zz); 25-28: the four traces
  for (int c = 0; c < 3; ++c) {
    const int f = kWsTri + c * kWsTriStride;
    t.r1[c] = wide_pack(f + 1, 1, n, 1);
    for (int i = 0; i < 3; ++i) t.r1[3 + 3 * c + i] = wide_pack(f + 4 + 3 * i, 1, n, 1);
    t.r1[12 + c] = wide_pack(phi + 4 + 3 * c, 1, n, 1);
    t.r1[16 + c] = wide_pack(kWsTri + 1 + c, kWsTriStride, n, 1);
  }
  t.r1[15] = wide_pack(phi + 1, 1, n, 1);
  for (int i = 0; i < 3; ++i)
    for (int j = i; j < 3; ++j) t.r1[19 + sym[i][j]] = wide_pack(kWsTri + 4 + 3 * i + j, kWsTriStride, n, 1);
  for (int f = 0; f < 4; ++f) t.r1[25 + f] = wide_pack(kWsTri + f * kWsTriStride + 4, 4, kWsOne, 1);
  // round 2. 0-8: effective tidal matrix Hess phi + T / 2 (full);
  // 9-11: v = 2 grad phi + n . grad B; 12-14: w = 2 grad phi + (grad B n + n . grad B) / 2;
  // 15: 1 + 2 phi
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 3; ++j)
      t.r2[3 * i + j] = wide_pack(phi + 4 + 3 * i + j, kWsD1 + 19 + sym[i][j], kWsD1 + 3 + 3 * i + j, kWsD1 + 3 + 3 * j + i);
    t.r2[9 + i] = wide_pack(kWsD1 + 16 + i, phi + 1 + i, kWsZero, kWsZero);
    t.r2[12 + i] = wide_pack(kWsZero, phi + 1 + i, kWsD1 + i, kWsD1 + 16 + i);
  }
  t.r2[15] = wide_pack(kWsOne, phi, kWsZero, kWsZero);
  // round 3. 0: n . v; 1: e1 . w; 2: e2 . w; 3: n . (n . grad B); 4: n Hess phi n;
  // 5: n . Laplacian B; 6-8: He e1; 9-11: He e2
  t.r3[0] = wide_pack(n, 1, kWsD2 + 9, 1);
  t.r3[1] = wide_pack(a, 1, kWsD2 + 12, 1);
  t.r3[2] = wide_pack(b, 1, kWsD2 + 12, 1);
  t.r3[3] = wide_pack(n, 1, kWsD1 + 16, 1);
  t.r3[4] = wide_pack(n, 1, kWsD1 + 12, 1);
  t.r3[5] = wide_pack(n, 1, kWsD1 + 25, 1);
  for (int i = 0; i < 3; ++i) {
    t.r3[6 + i] = wide_pack(kWsD2 + 3 * i, 1, a, 1);
    t.r3[9 + i] = wide_pack(kWsD2 + 3 * i, 1, b, 1);
  }
  // round 4: e1 He e1, e2 He e2, e1 He e2
  t.r4[0] = wide_pack(a, 1, kWsD3 + 6, 1);
  t.r4[1] = wide_pack(b, 1, kWsD3 + 9, 1);
  t.r4[2] = wide_pack(a, 1, kWsD3 + 9, 1);
  // round 5: S1, S2, 4 L, -P_perp:Hess phi + n . Laplacian B / 2, dA^2
  t.r5[0] = wide_pack(kWsD4 + 0, kWsNeg1, kWsD4 + 1, kWsZero);
  t.r5[1] = wide_pack(kWsZero, kWsTwo, kWsD4 + 2, kWsZero);
  t.r5[2] = wide_pack(kWsD3 + 3, kWsFour, kWsD1 + 15, kWsZero);
  t.r5[3] = wide_pack(kWsD1 + 28, kWsNeg1, kWsD3 + 4, kWsD3 + 5);
  t.r5[4] = wide_pack(kWsZero, kWsY + 12, kWsY + 12, kWsZero);
  // round 6: the 19 derivatives
  for (int i = 0; i < 3; ++i) {
    t.r6[i] = wide_pack(n + i, kWsD2 + 15, kWsZero, kWsZero);
    t.e6[i] = (uint32_t)(kWsTri + i * kWsTriStride) | ((uint32_t)(kWideNegB | kWideNegE) << 8);
    t.r6[3 + i] = wide_pack(n + i, kWsD3 + 0, kWsZero, kWsZero);
    t.e6[3 + i] = (uint32_t)(kWsD2 + 9 + i) | ((uint32_t)kWideNegB << 8);
    t.r6[6 + i] = wide_pack(n + i, kWsD3 + 1, kWsZero, kWsZero);
    t.e6[6 + i] = (uint32_t)kWsZero | ((uint32_t)kWideNegB << 8);
    t.r6[9 + i] = wide_pack(n + i, kWsD3 + 2, kWsZero, kWsZero);
    t.e6[9 + i] = (uint32_t)kWsZero | ((uint32_t)kWideNegB << 8);
  }
  t.e6[12] = (uint32_t)(kWsY + 13) | ((uint32_t)kWideNegE << 8);
  t.r6[13] = wide_pack(kWsY + 12, kWsD5 + 3, kWsD5 + 2, kWsY + 13);
  t.e6[13] = (uint32_t)kWsQuo | ((uint32_t)kWideNegD << 8);
  t.r6[14] = wide_pack(kWsD5 + 0, kWsD5 + 4, kWsD5 + 2, kWsY + 14);
  t.r6[15] = wide_pack(kWsD5 + 1, kWsD5 + 4, kWsD5 + 2, kWsY + 15);
  t.r6[16] = wide_pack(kWsZero, kWsZero, kWsNeg2, kWsQuo + 1);
  t.r6[17] = wide_pack(kWsZero, kWsZero, kWsNeg2, kWsQuo + 2);
  t.e6[18] = (uint32_t)(kWsQuo + 3);
  return t;
}

// Catmull-Rom coefficients per tap: value c0..c3, derivative c0..c2, second
// derivative c0, c1 (cr_weights_fp64's, with the powers a tap lacks as zeros).
struct WideCoef {
  float v[4], g[3], h[2];
};

SRT_HD WideCoef wide_coef(int tap) {
  WideCoef c;
  c.v[0] = tap == 1 ? 1.f : 0.f;
  c.v[1] = tap == 0 ? -0.5f : (tap == 2 ? 0.5f : 0.f);
  c.v[2] = tap == 0 ? 1.f : (tap == 1 ? -2.5f : (tap == 2 ? 2.f : -0.5f));
  c.v[3] = tap == 0 ? -0.5f : (tap == 1 ? 1.5f : (tap == 2 ? -1.5f : 0.5f));
  c.g[0] = tap == 0 ? -0.5f : (tap == 2 ? 0.5f : 0.f);
  c.g[1] = tap == 0 ? 2.f : (tap == 1 ? -5.f : (tap == 2 ? 4.f : -1.f));
  c.g[2] = tap == 0 ? -1.5f : (tap == 1 ? 4.5f : (tap == 2 ? -4.5f : 1.5f));
  c.h[0] = tap == 0 ? 2.f : (tap == 1 ? -5.f : (tap == 2 ? 4.f : -1.f));
  c.h[1] = tap == 0 ? -3.f : (tap == 1 ? 9.f : (tap == 2 ? -9.f : 3.f));
  return c;
}

// Integer part of a floored position.
SRT_HD int64_t int_r(double f) { return (int64_t)f; }
SRT_HD int64_t int_r(const dd& f) { return (int64_t)f.hi + (int64_t)f.lo; }
SRT_HD double floor_r(double x) { return floor(x); }
SRT_HD dd floor_r(const dd& x) { return dd_floor(x); }
SRT_HD bool above_half(double x) { return x > 0.5; }
SRT_HD bool above_half(const dd& x) { return x > dd(0.5f); }

// A tap's three weights at w[0], w[4], w[8].
template <typename R>
SRT_HD void wide_weights(const WideCoef& cf, const R& t, R* w) {
  R v = fma_r(R(cf.v[3]), t, R(cf.v[2]));
  v = fma_r(v, t, R(cf.v[1]));
  w[0] = fma_r(v, t, R(cf.v[0]));
  const R g = fma_r(R(cf.g[2]), t, R(cf.g[1]));
  w[4] = fma_r(g, t, R(cf.g[0]));
  w[8] = fma_r(R(cf.h[1]), t, R(cf.h[0]));
}

// Output o of a slice's y pass (a, ay, ayy, ax, axy, axx) from the y weights and
// the slice's four rows of x pass results.
template <typename R>
SRT_HD void wide_y_output(const R* w, const R* x, R* out, int o) {
  const int wo = o == 1 || o == 4 ? 4 : (o == 2 ? 8 : 0), xo = o < 3 ? 0 : (o == 5 ? 2 : 1);
  Chain<R> s;
#pragma unroll
  for (int b = 0; b < 4; ++b) s.add(w[wo + b], x[3 * b + xo]);
  out[o] = s.value();
}

// ------------------------------------------------------------- lane phases

// What one lane keeps in registers through a ray: its operand words, its
// weights' coefficients, and its component of the state, the stage's k and the
// RK4 accumulator.
template <typename R>
struct WideLane {
  int lane;
  uint32_t r1, r2, r3, r4, r5, r6, e6;
  float beta2, gamma2;  // round 2
  WideCoef cf;
  R y, k, acc;
  float tap[8];

  SRT_HD void start(int l, const WideTables& t) {
    lane = l;
    r1 = t.r1[l], r2 = t.r2[l], r3 = t.r3[l], r4 = t.r4[l], r5 = t.r5[l], r6 = t.r6[l], e6 = t.e6[l];
    beta2 = l < 9 ? 0.5f : 2.f;
    gamma2 = l < 9 ? -0.25f : (l >= 12 && l < 15 ? 0.5f : 0.f);
    cf = wide_coef(l & 3);
  }

  // constants of the scratch (once per warp)
  SRT_HD void constants(R* S) const {
    if (lane < 3) S[kWsOne + lane] = R(1.f);
    if (lane == 3) S[kWsZero] = R(0.f);
    if (lane == 4) S[kWsNeg1] = R(-1.f);
    if (lane == 5) S[kWsNeg2] = R(-2.f);
    if (lane == 6) S[kWsTwo] = R(2.f);
    if (lane == 7) S[kWsFour] = R(4.f);
  }

  // stage input y + c k
  SRT_HD void stage(R* S, int st) {
    if (lane < 19) S[kWsY + lane] = st == 0 ? y : axpy_r(R(st == 3 ? 1.f : 0.5f), k, y);
  }

  // one axis of the centred (lanes 0-2) or staggered grid (3-5)
  SRT_HD void position(R* S, int* cell, const Geom& G) const {
    if (lane >= 6) return;
    const int a = lane < 3 ? lane : lane - 3;
    R x = S[kWsY + a];
    if (lane >= 3) x = x - R(0.5f);
    const R f = floor_r(x);
    S[kWsT + lane] = x - f;
    const int64_t c = int_r(f);
    cell[lane] = (uint64_t)c < (uint64_t)G.n[a] ? (int)c : wrap64(c, G.n[a]);
  }

  // taps of rows 2 sub and 2 sub + 1 (row = 4 slice + row in slice) of field lane / 8
  SRT_HD void load_taps(const int* cell, const FieldPtrs& F, const Geom& G) {
    const int f = lane >> 3, sub = lane & 7;
    const float* src = f == 3 ? F.phi : (f == 0 ? F.b[0] : (f == 1 ? F.b[1] : F.b[2]));
    const float* p = src + (cell_base(G, cell[f == 0 ? 3 : 0], cell[f == 1 ? 4 : 1], cell[f == 2 ? 5 : 2]) +
                            (sub >> 1) * G.pxy + 2 * (sub & 1) * G.px) * G.ts;
#pragma unroll
    for (int i = 0; i < 4; ++i) tap[i] = ldg(p + i * G.ts);
#pragma unroll
    for (int i = 0; i < 4; ++i) tap[4 + i] = ldg(p + (G.px + i) * G.ts);
  }

  SRT_HD void weights(R* S) const {
    if (lane >= 24) return;
    const int set = lane >> 2, i = lane & 3;
    wide_weights(cf, S[kWsT + set], S + kWsW + 12 * set + i);
  }

  // Lanes 0-8: component i of unit vector v. Lanes 9-12: the branch's
  // quotients (s1^2 + s2^2) / dA^3, s1 q / dA^2, s2 q / dA^2 and
  // -(s1 el2 - s2 el1) / (dA^2 (2 + q)), q = (4 + el1^2 + el2^2)^(1/2) formed
  // as the norm of (2, el1, el2), so one root and one division serve all.
  SRT_HD void frame(R* S) const {
    const int l = lane < 13 ? lane : 0;
    const bool vec = l < 9;
    const int j = l - 9;
    const R c0 = vec ? S[kWsY + 3 + 3 * (l / 3)] : S[kWsTwo];
    const R c1 = S[kWsY + (vec ? 4 + 3 * (l / 3) : 16)], c2 = S[kWsY + (vec ? 5 + 3 * (l / 3) : 17)];
    Chain<R> q2;
    q2.add(c0, c0);
    q2.add(c1, c1);
    q2.add(c2, c2);
    const R r = sqrt_r(q2.value());
    const R dA = S[kWsY + 12], s1 = S[kWsY + 14], s2 = S[kWsY + 15];
    const R zero(0.f), one(1.f);
    // numerator A B + C D, denominator dA^2 times F
    const R A = j == 1 ? s1 : s2, B = j == 0 ? s2 : (j == 3 ? c1 : r);
    const R C = (j == 0 || j == 3) ? s1 : zero, D = j == 0 ? s1 : (j == 3 ? -c2 : zero);
    Chain<R> nm;
    nm.add(C, D);
    nm.add(A, B);
    const R rp2 = r + R(2.f);
    const R F = j == 0 ? dA : (j == 3 ? rp2 : one);
    const R den = dA * dA * F;
    const R quo = (vec ? S[kWsY + 3 + l] : nm.value()) / (vec ? r : den);
    if (lane < 13) S[vec ? kWsU + l : kWsQuo + j] = (vec || above_half(dA)) ? quo : zero;
  }

  SRT_HD void x_pass(R* S) const {
    const int f = lane >> 3, sub = lane & 7;
    const R* w = S + kWsW + 12 * (f == 0 ? 3 : 0);
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      const R w0 = w[4 * o], w1 = w[4 * o + 1], w2 = w[4 * o + 2], w3 = w[4 * o + 3];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        Chain<R> c;
        c.add(w0, tap[4 * r]);
        c.add(w1, tap[4 * r + 1]);
        c.add(w2, tap[4 * r + 2]);
        c.add(w3, tap[4 * r + 3]);
        S[kWsX + 48 * f + 3 * (2 * sub + r) + o] = c.value();
      }
    }
  }

  // slice sub / 2: (a, ay, ayy) on the even lanes, (ax, axy, axx) on the odd
  SRT_HD void y_pass(R* S) const {
    const int f = lane >> 3, sub = lane & 7, c = sub >> 1, odd = sub & 1;
    const R* w = S + kWsW + 12 * (f == 1 ? 4 : 1);
    const R* x = S + kWsX + 48 * f + 12 * c;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      wide_y_output(w, x, S + kWsYp + 24 * f + 6 * c, 3 * odd + o);
    }
  }

  // outputs sub and, on the first two lanes of a field, 8 + sub
  SRT_HD void z_pass(R* S) const {
    const int f = lane >> 3, sub = lane & 7;
    const R* w = S + kWsW + 12 * (f == 2 ? 5 : 2);
    R* out = S + kWsTri + kWsTriStride * f;
    z_output(w, S + kWsYp + 24 * f, out, sub);
    if (sub < 2) z_output(w, S + kWsYp + 24 * f, out, 8 + sub);
  }

  SRT_HD static void z_output(const R* w, const R* ys, R* out, int m) {
    // m: v, gx, gy, gz, xx, xy, xz, yy, yz, zz; 4-bit source, order and places
    const int src = (int)((0x0123450130ull >> (4 * m)) & 15);
    const int ord = (int)((0x2101001000ull >> (4 * m)) & 15);
    Chain<R> s;
#pragma unroll
    for (int c = 0; c < 4; ++c) s.add(w[4 * ord + c], ys[6 * c + src]);
    const R v = s.value();
    // full Hessian rows at 4, 7, 10
    const int h = m < 4 ? 0 : m - 4;
    out[m < 4 ? m : (int)((0xC98654u >> (4 * h)) & 15)] = v;
    if (m >= 4) out[(0xCB8A74u >> (4 * h)) & 15] = v;
  }

  SRT_HD static R dot(const R* S, uint32_t t) {
    const R* a = S + (t & 255);
    const R* b = S + ((t >> 16) & 255);
    const int sa = (t >> 8) & 255, sb = t >> 24;
    Chain<R> c;
    c.add(a[0], b[0]);
    c.add(a[sa], b[sb]);
    c.add(a[2 * sa], b[2 * sb]);
    return c.value();
  }

  SRT_HD void round1(R* S) const {
    const R v = dot(S, r1);
    if (lane < 29) S[kWsD1 + lane] = v;
  }
  SRT_HD void round2(R* S) const {
    const R z = S[(r2 >> 16) & 255] + S[r2 >> 24];
    Chain<R> c(S[r2 & 255]);
    c.add(R(beta2), S[(r2 >> 8) & 255]);
    c.add(R(gamma2), z);
    if (lane < 16) S[kWsD2 + lane] = c.value();
  }
  SRT_HD void round3(R* S) const {
    const R v = dot(S, r3);
    if (lane < 12) S[kWsD3 + lane] = v;
  }
  SRT_HD void round4(R* S) const {
    const R v = dot(S, r4);
    if (lane < 3) S[kWsD4 + lane] = v;
  }
  SRT_HD void round5(R* S) const {
    Chain<R> c(S[r5 & 255]);
    c.add(S[(r5 >> 8) & 255], S[(r5 >> 16) & 255]);
    c.add(R(0.5f), S[r5 >> 24]);
    if (lane < 5) S[kWsD5 + lane] = c.value();
  }
  // this lane's derivative and its place in the RK4 accumulator
  SRT_HD void round6(const R* S, int st) {
    const int neg = e6 >> 8;
    const R E = S[e6 & 255], B = S[(r6 >> 8) & 255], D = S[r6 >> 24];
    Chain<R> c(neg & kWideNegE ? -E : E);
    c.add(S[(r6 >> 16) & 255], neg & kWideNegD ? -D : D);
    c.add(S[r6 & 255], neg & kWideNegB ? -B : B);
    k = c.value();
    if (st == 0)
      acc = k;
    else if (st < 3)
      acc = axpy_r(R(2.f), k, acc);
    else
      y = axpy_r(acc + k, R(1.0 / 6.0), y);
  }
};

// --------------------------------------------------- five warps per ray
//
// The same stage cut over warps: warps 0-3 interpolate one field each (FieldLane:
// positions, weights, passes; only warp barriers between them), warp 4 forms the
// frame (WideLane::frame) beside them, then warp 0 runs the rounds. ~24 FP64
// instructions on a field warp's path, ~26 on the frame's and 18 in the rounds
// against ~104 for one warp, and ~140 in all, so an SM's FP64 rate (19 cycles an
// instruction) still carries four rays at a time as fast as one warp each would.

template <typename R>
struct FieldLane {
  int lane, f;
  WideCoef cf;
  float tap[4];

  SRT_HD void start(int l, int field) {
    lane = l;
    f = field;
    cf = wide_coef(l & 3);
  }

  // offset and cell on one axis (lanes 0-2)
  SRT_HD void position(R* S, int* cell, const Geom& G) const {
    if (lane >= 3) return;
    R x = S[kWsY + lane];
    if (lane == f) x = x - R(0.5f);
    const R fl = floor_r(x);
    S[kWsTf + 3 * f + lane] = x - fl;
    const int64_t c = int_r(fl);
    cell[3 * f + lane] = (uint64_t)c < (uint64_t)G.n[lane] ? (int)c : wrap64(c, G.n[lane]);
  }

  // taps of row lane % 16 (4 slice + row in slice)
  SRT_HD void load_taps(const int* cell, const FieldPtrs& F, const Geom& G) {
    const int* c = cell + 3 * f;
    const int row = lane & 15;
    const float* src = f == 3 ? F.phi : (f == 0 ? F.b[0] : (f == 1 ? F.b[1] : F.b[2]));
    const float* p = src + (cell_base(G, c[0], c[1], c[2]) + (row >> 2) * G.pxy + (row & 3) * G.px) * G.ts;
#pragma unroll
    for (int i = 0; i < 4; ++i) tap[i] = ldg(p + i * G.ts);
  }

  SRT_HD void weights(R* S) const {
    if (lane >= 12) return;
    const R t = S[kWsTf + 3 * f + (lane >> 2)];
    wide_weights(cf, t, S + kWsWf + 36 * f + 12 * (lane >> 2) + (lane & 3));
  }

  // value (lanes 0-15) and first derivative (16-31), then the second (0-15)
  SRT_HD void x_pass(R* S) const {
    x_chain(S, lane >> 4);
    if (lane < 16) x_chain(S, 2);
  }
  SRT_HD void x_chain(R* S, int o) const {
    const R* w = S + kWsWf + 36 * f + 4 * o;
    Chain<R> c;
#pragma unroll
    for (int i = 0; i < 4; ++i) c.add(w[i], tap[i]);
    S[kWsX + 48 * f + 3 * (lane & 15) + o] = c.value();
  }

  // lane 6 slice + output
  SRT_HD void y_pass(R* S) const {
    if (lane >= 24) return;
    const int c = lane / 6, o = lane - 6 * c;
    wide_y_output(S + kWsWf + 36 * f + 12, S + kWsX + 48 * f + 12 * c, S + kWsYp + 24 * f + 6 * c, o);
  }

  SRT_HD void z_pass(R* S) const {
    if (lane >= 10) return;
    WideLane<R>::z_output(S + kWsWf + 36 * f + 24, S + kWsYp + 24 * f, S + kWsTri + kWsTriStride * f, lane);
  }
};

}  // namespace srt
