// srt_adjoint.cuh — reverse mode (vector-Jacobian product) of one evaluation of
// the tracer's right-hand side (snapshot-raytracer.cu:315-510), for the vjp of
// the maps with respect to the phi and B grids.
//
// The reverse sweep of an RK4 step (snapshot-raytracer.cu:524-549) needs, for
// each stage input u and output cotangent fb, ub = J(u)^T fb together with the
// cotangents of the grid values the stage read. Derived by hand from the
// forward computation in srt_scheme.cuh:
//   * every intermediate cotangent of the right-hand side (of L = n.g + n.ngB/4,
//     of P_perp:H, of the shear projections S1/S2, of the tidal matrix T, of
//     n.lap B, n.grad B and the e.n.grad B scalars, of phi, grad phi, Hess phi
//     and of the B values) depends on fb and on the state only, so each field's
//     cotangent (value, gradient, Hessian) is known before the field is read;
//   * one fused pass per field then interpolates value, gradient, Hessian and
//     the ten third derivatives (the position cotangent needs d/dx of the
//     Hessian), scatters the 64 tap cotangents into the gradient grid, and
//     adds the field's share of the state cotangents;
//   * the terms that need sums over fields (v = 2g + n.grad B, L, P_perp:H,
//     the effective tidal matrix) are added after the four passes.
// Catmull-Rom's third derivative is piecewise constant: weights (-3, 9, -9, 3).
#pragma once
#include <type_traits>
#include "srt_scheme.cuh"

namespace srt {

template <typename T>
struct CRW4 {  // Catmull-Rom weights for value and d/dt .. d3/dt3
  T w[4], g[4], h[4], k[4];
};

template <typename T>
SRT_HD void cr_weights4(T t, CRW4<T>& c) {
  CRW<T> b;
  cr_weights(t, b);
  for (int i = 0; i < 4; ++i) {
    c.w[i] = b.w[i];
    c.g[i] = b.g[i];
    c.h[i] = b.h[i];
  }
  c.k[0] = T(-3);
  c.k[1] = T(9);
  c.k[2] = T(-9);
  c.k[3] = T(3);
}

// ---------------------------------------------------------- accumulators

// Where the tap cotangents go. Three flavours:
//   AccF32    FP32 vector atomics into a grid of cells (float4 per padded
//             voxel): the cotangents of a voxel's value and of its second
//             differences along y, x and both, which fold_kernel gathers onto
//             the voxels; one 16-byte atomic carries a tap's four;
//   AccF64    FP64 atomics into a halo-padded grid (one per tap), one call per
//             4-tap x-row of a tricubic footprint (padded index `row` of its
//             first tap);
//   AccFixed  64-bit fixed point into a halo-padded grid (order-independent,
//             so repeated runs give identical bits), by rows too.
// A null grid (gradient not requested) ignores the contributions, and the
// passes skip forming them (active() is false).
// Near the observer every ray adds to the same few voxels, and atomics on one
// address run one after another: there each warp adds to one of kHotCopies
// copies of a kHotSide^3 region around the observer (behind the grid, merged
// into it afterwards), spreading them over as many addresses. 256^3 / nside 128:
// the first 12 of 128 steps took 9.0 ms against ~3.1 for the others.
constexpr int kHotSide = 32, kHotCopies = 16;

// Index in a copy of the footprint that starts at cell (cx, cy, cz), or -1 where
// it leaves the region (padded positions n / 2 - kHotSide / 2 on).
SRT_HD int hot_base(const Geom& G, const int* c) {
  const unsigned x = (unsigned)(c[0] - G.n[0] / 2 + kHotSide / 2), y = (unsigned)(c[1] - G.n[1] / 2 + kHotSide / 2),
                 z = (unsigned)(c[2] - G.n[2] / 2 + kHotSide / 2);
  const bool in = x <= kHotSide - 4 && y <= kHotSide - 4 && z <= kHotSide - 4;
  return in ? (int)(x + kHotSide * (y + kHotSide * z)) : -1;
}

// A sweep's atomics go to 32 lines an instruction and held its loads up behind
// them (64 a stage; long-scoreboard stalls 3.2 of 5.9 cycles an instruction), so
// the lanes work in pairs: the two cells of a grid row that a ray adds to are
// neighbours in memory, and each atomic instruction takes both cells of one of
// the pair's rays, half the lines (long-scoreboard stalls 0.7; a 512^3 / nside
// 256 / 256 steps gradient 389 -> 373 ms). All lanes of a warp call these
// together; a lane without a ray follows one with a zero cotangent.
// DISTANCE: lanes from one ray of a pair to the other (1, or 4 where four lanes
// share a ray and `mask` holds the lanes whose field takes part).
template <int DISTANCE>
struct AccPaired {
  float4* g;
  int64_t hot = 0;  // index of this warp's copy; 0: no copies
  unsigned mask = 0xffffffffu;
  SRT_HD bool active() const { return g != nullptr; }
  SRT_HD static int lane() {
#if defined(__CUDA_ARCH__)
    return (threadIdx.x / DISTANCE) & 1;
#else
    return 0;
#endif
  }
  // Where a field's footprint goes: entries of the pair's even and odd ray for
  // this lane's cell of the first slice's first inner row, and the strides.
  struct Place {
    float4 *even, *odd;
    int64_t px, pxy;
  };
  SRT_HD Place place(int64_t base, int hbase, const Geom& G) const {
    Place p{nullptr, nullptr, G.px, G.pxy};
#if defined(__CUDA_ARCH__)
    if (hot && __all_sync(mask, hbase >= 0)) {
#else
    if (hot && hbase >= 0) {
#endif
      base = hot + hbase;
      p.px = kHotSide;
      p.pxy = kHotSide * kHotSide;
    }
    int64_t other = base;
#if defined(__CUDA_ARCH__)
    other = __shfl_xor_sync(mask, base, DISTANCE);
#endif
    const int me = lane();
    p.even = g + (me ? other : base) + p.px + 1 + me;
    p.odd = g + (me ? base : other) + p.px + 1 + me;
    return p;
  }
  // A row's two cells: this lane's (me = lane(): tap 1 or 2) and the other.
  SRT_HD void add_row2(float4* even, float4* odd, float4 own, float4 other) const {
#if defined(__CUDA_ARCH__)
    const int me = lane();
    const float4 in =
        make_float4(__shfl_xor_sync(mask, other.x, DISTANCE), __shfl_xor_sync(mask, other.y, DISTANCE),
                    __shfl_xor_sync(mask, other.z, DISTANCE), __shfl_xor_sync(mask, other.w, DISTANCE));
    atomicAdd(even, me ? in : own);
    atomicAdd(odd, me ? own : in);
#else
    (void)odd;
    for (int e = 0; e < 2; ++e) {
      const float4 v = e ? other : own;
      even[e].x += v.x;
      even[e].y += v.y;
      even[e].z += v.z;
      even[e].w += v.w;
    }
#endif
  }
};

// Accumulators that take cells (add_row2) rather than rows of taps.
template <typename Acc>
struct TakesCells : std::false_type {};
typedef AccPaired<1> AccF32;
template <int D>
struct TakesCells<AccPaired<D>> : std::true_type {};

struct AccF64 {
  double* g;
  SRT_HD bool active() const { return g != nullptr; }
  SRT_HD void add(int64_t i, double v) const {
#if defined(__CUDA_ARCH__)
    atomicAdd(g + i, v);
#else
    g[i] += v;
#endif
  }
  SRT_HD void add_row(int64_t row, double c0, double c1, double c2, double c3) const {
    if (!g) return;
    add(row, c0);
    add(row + 1, c1);
    add(row + 2, c2);
    add(row + 3, c3);
  }
};

// Fixed point with kFixedScale = 2^32 units per unit of gradient; |gradient|
// per voxel must stay below 2^31. Contributions are rounded to the nearest
// unit before the integer addition, so the result does not depend on the
// order of the additions. A contribution of magnitude 2^30 or more (or one
// that is not finite) sets *ovf, where the integer sum may already have
// wrapped; the fold kernel sets it too for a folded |gradient| >= 2^30, and
// srt_vjp then fails with SRT_ERR_OVERFLOW instead of returning wrapped values.
constexpr double kFixedScale = 4294967296.0;
constexpr double kFixedLimit = 1073741824.0;  // 2^30 units of gradient

struct AccFixed {
  unsigned long long* g;
  unsigned* ovf = nullptr;
  SRT_HD bool active() const { return g != nullptr; }
  SRT_HD void add(int64_t i, double v) const {
    if (!(fabs(v) < kFixedLimit)) {
#if defined(__CUDA_ARCH__)
      if (ovf) atomicOr(ovf, 1u);
#else
      if (ovf) *ovf |= 1u;
#endif
      v = 0.0;  // llrint of it would be undefined
    }
    const long long q = llrint(v * kFixedScale);
#if defined(__CUDA_ARCH__)
    atomicAdd(g + i, (unsigned long long)q);
#else
    g[i] += (unsigned long long)q;
#endif
  }
  SRT_HD void add_row(int64_t row, double c0, double c1, double c2, double c3) const {
    if (!g) return;
    add(row, c0);
    add(row + 1, c1);
    add(row + 2, c2);
    add(row + 3, c3);
  }
};

// No accumulation: the B components' passes when only the phi gradient is
// wanted. active() is false at compile time, so those passes are compiled
// without their scatter (less code, fewer registers).
struct AccNone {
  SRT_HD constexpr bool active() const { return false; }
  template <typename V>
  SRT_HD void add_row(int64_t, V, V, V, V) const {}
};

// ------------------------------------------------- fused field pass (vjp)

// Interpolates one field (value, gradient, Hessian into Q; third derivatives
// used internally), adds qb . dQ/dposition to xb and scatters the cotangent of
// every tap, sum_q qb_q W_q(tap), through `acc`.
// qb: cotangents of (v, gx, gy, gz, hxx, hxy, hxz, hyy, hyz, hzz); the
// Hessian entries are the unique components (off-diagonal cotangents already
// hold both symmetric halves).
template <typename T, typename Acc>
SRT_HD void tricubic_vjp(const float* __restrict__ f, int64_t base, int64_t px, int64_t pxy, int ts, T tx, T ty, T tz,
                         const T* qb, Tri<T>& Q, T* xb, const Acc& acc) {
  CRW4<T> X, Y, Z;
  cr_weights4(tx, X);
  cr_weights4(ty, Y);
  cr_weights4(tz, Z);
  const bool scatter = acc.active();  // this field's gradient was requested
  // per-row scatter factors: the tap cotangent of row (b, c) is
  // wx_i Cw + gx_i Cg + hx_i Ch with Cw = wz_c Aw_b + gz_c Bw_b + hz_c Dw_b,
  // Cg = wz_c Ag_b + gz_c Bg_b, Ch = wz_c Ah_b.
  T Aw[4], Bw[4], Dw[4], Ag[4], Bg[4], Ah[4];
  for (int b = 0; b < 4; ++b) {
    Aw[b] = qb[0] * Y.w[b] + qb[2] * Y.g[b] + qb[7] * Y.h[b];
    Bw[b] = qb[3] * Y.w[b] + qb[8] * Y.g[b];
    Dw[b] = qb[9] * Y.w[b];
    Ag[b] = qb[1] * Y.w[b] + qb[5] * Y.g[b];
    Bg[b] = qb[6] * Y.w[b];
    Ah[b] = qb[4] * Y.w[b];
  }
  // 20 accumulators: derivative orders (x, y, z) with x + y + z <= 3
  T o000 = 0, o001 = 0, o002 = 0, o003 = 0, o010 = 0, o011 = 0, o012 = 0, o020 = 0, o021 = 0, o030 = 0;
  T o100 = 0, o101 = 0, o102 = 0, o110 = 0, o111 = 0, o120 = 0, o200 = 0, o201 = 0, o210 = 0, o300 = 0;
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    T s00 = 0, s01 = 0, s02 = 0, s03 = 0, s10 = 0, s11 = 0, s12 = 0, s20 = 0, s21 = 0, s30 = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int64_t row = base + c * pxy + b * px;
      const float* rp = f + row * ts;
      const T p0 = (T)ldg(rp), p1 = (T)ldg(rp + ts), p2 = (T)ldg(rp + 2 * ts), p3 = (T)ldg(rp + 3 * ts);
      const T r0 = X.w[0] * p0 + X.w[1] * p1 + X.w[2] * p2 + X.w[3] * p3;
      const T r1 = X.g[0] * p0 + X.g[1] * p1 + X.g[2] * p2 + X.g[3] * p3;
      const T r2 = X.h[0] * p0 + X.h[1] * p1 + X.h[2] * p2 + X.h[3] * p3;
      const T r3 = X.k[0] * p0 + X.k[1] * p1 + X.k[2] * p2 + X.k[3] * p3;
      s00 += Y.w[b] * r0;
      s01 += Y.g[b] * r0;
      s02 += Y.h[b] * r0;
      s03 += Y.k[b] * r0;
      s10 += Y.w[b] * r1;
      s11 += Y.g[b] * r1;
      s12 += Y.h[b] * r1;
      s20 += Y.w[b] * r2;
      s21 += Y.g[b] * r2;
      s30 += Y.w[b] * r3;
      if (scatter) {
        const T Cw = Z.w[c] * Aw[b] + Z.g[c] * Bw[b] + Z.h[c] * Dw[b];
        const T Cg = Z.w[c] * Ag[b] + Z.g[c] * Bg[b];
        const T Ch = Z.w[c] * Ah[b];
        acc.add_row(row, X.w[0] * Cw + X.g[0] * Cg + X.h[0] * Ch, X.w[1] * Cw + X.g[1] * Cg + X.h[1] * Ch,
                    X.w[2] * Cw + X.g[2] * Cg + X.h[2] * Ch, X.w[3] * Cw + X.g[3] * Cg + X.h[3] * Ch);
      }
    }
    const T zw = Z.w[c], zg = Z.g[c], zh = Z.h[c], zk = Z.k[c];
    o000 += zw * s00; o001 += zg * s00; o002 += zh * s00; o003 += zk * s00;
    o010 += zw * s01; o011 += zg * s01; o012 += zh * s01;
    o020 += zw * s02; o021 += zg * s02;
    o030 += zw * s03;
    o100 += zw * s10; o101 += zg * s10; o102 += zh * s10;
    o110 += zw * s11; o111 += zg * s11;
    o120 += zw * s12;
    o200 += zw * s20; o201 += zg * s20;
    o210 += zw * s21;
    o300 += zw * s30;
  }
  Q.v = o000;
  Q.g[0] = o100;
  Q.g[1] = o010;
  Q.g[2] = o001;
  Q.h[0] = o200;
  Q.h[1] = o110;
  Q.h[2] = o101;
  Q.h[3] = o020;
  Q.h[4] = o011;
  Q.h[5] = o002;
  // xb_j += qb . dQ/dx_j
  xb[0] += qb[0] * o100 + qb[1] * o200 + qb[2] * o110 + qb[3] * o101 + qb[4] * o300 + qb[5] * o210 +
           qb[6] * o201 + qb[7] * o120 + qb[8] * o111 + qb[9] * o102;
  xb[1] += qb[0] * o010 + qb[1] * o110 + qb[2] * o020 + qb[3] * o011 + qb[4] * o210 + qb[5] * o120 +
           qb[6] * o111 + qb[7] * o030 + qb[8] * o021 + qb[9] * o012;
  xb[2] += qb[0] * o001 + qb[1] * o101 + qb[2] * o011 + qb[3] * o002 + qb[4] * o201 + qb[5] * o111 +
           qb[6] * o102 + qb[7] * o021 + qb[8] * o012 + qb[9] * o003;
}

// Per order in x (w: value, g: first, h: second), the cotangents of a slice's row
// values and of their second differences along y at rows 1 and 2: (value,
// difference) pairs per row, for the slice's z weights.
struct SliceCotangents {
  float2 w[2], g[2], h[2];
};
SRT_HD SliceCotangents slice_cotangents(const float* qb, const CWD& Y, float zw, float zg, float zh) {
  const float a0 = fmaf(qb[0], zw, fmaf(qb[3], zg, qb[9] * zh)), a1 = fmaf(qb[2], zw, qb[8] * zg), a2 = qb[7] * zw;
  const float b0 = fmaf(qb[1], zw, qb[6] * zg), b1 = qb[5] * zw, c0 = qb[4] * zw;
  const float w2 = fmaf(Y.t, a0, a1), g2 = fmaf(Y.t, b0, b1), h2 = Y.t * c0;
  return SliceCotangents{{make_float2(a0 - w2, fmaf(Y.w0, a0, fmaf(Y.g0, a1, Y.h0 * a2))),
                          make_float2(w2, fmaf(Y.w3, a0, fmaf(Y.g3, a1, Y.h3 * a2)))},
                         {make_float2(b0 - g2, fmaf(Y.w0, b0, Y.g0 * b1)), make_float2(g2, fmaf(Y.w3, b0, Y.g3 * b1))},
                         {make_float2(c0 - h2, Y.w0 * c0), make_float2(h2, Y.w3 * c0)}};
}

// The same pass for the MIXED form, in FP32 on the second-difference form of
// the cubic (CWD): the x pass on packed pairs as in tricubic_mixed, with its
// third derivative (one packed subtraction a row), the y pass on scalars, the
// z pass on pairs of outputs, and the next slice's data loaded while the
// current one is processed.
// The tap cotangents are formed in the basis the passes read: per slice, for
// the four inner taps, the cotangents of the value and of the second
// differences along y, x and both (60 operations a slice against 72 plus the
// row factors on sixteen taps). AccF32 adds them as they are, one 16-byte
// vector atomic per inner tap, and fold_kernel applies the (symmetric) second
// differences once per voxel; the other accumulators get them expanded to taps.
// 332 lane operations without the scatter against 536 on four taps.
template <int UNROLL, typename Acc, typename Src>
SRT_HD void tricubic_vjp_mixed(const Src& src, int64_t base, int hbase, const Geom& G, const float* t, const float* qb,
                               Tri<float>& Q, float* xb, const Acc& acc) {
  CWD X, Y;
  CRW<float> Z;
  cr_weights_diff(t[0], X);
  cr_weights_diff(t[1], Y);
  cr_weights_mixed(t[2], Z);
  const XDup xd(X);
  const bool scatter = acc.active();  // this field's gradient was requested
  AccF32::Place at = {};
  int me = 0;
  float2 ow, og, oh, nw, ng, nh;  // difference weights of this lane's cell of a pair and the other
  if constexpr (TakesCells<Acc>::value) {
    if (scatter) {
      const auto p = acc.place(base, hbase, G);
      at = {p.even, p.odd, p.px, p.pxy};
    }
    me = Acc::lane();
    ow = me ? xd.w3 : xd.w0, og = me ? xd.g3 : xd.g0, oh = me ? xd.h3 : xd.h0;
    nw = me ? xd.w0 : xd.w3, ng = me ? xd.g0 : xd.g3, nh = me ? xd.h0 : xd.h3;
  }
  // outputs oXYZ by derivative order, as pairs (two orders of the same z weight);
  // x and y third derivatives are summed as thirds
  const float2 z0 = make_float2(0.f, 0.f);
  float2 W0 = z0, W1 = z0, W2 = z0, W3 = z0, W4 = z0, G0 = z0, G1 = z0, G2 = z0, H0 = z0;
  float o102 = 0.f, o003 = 0.f;
  SliceData nt = src.load(0);
#pragma unroll UNROLL
  for (int c = 0; c < 4; ++c) {
    // this slice's z weights by selection (an indexed read of Z would put
    // it in local memory)
    const float zw = c == 0 ? Z.w[0] : (c == 1 ? Z.w[1] : (c == 2 ? Z.w[2] : Z.w[3]));
    const float zg = c == 0 ? Z.g[0] : (c == 1 ? Z.g[1] : (c == 2 ? Z.g[2] : Z.g[3]));
    const float zh = c == 0 ? Z.h[0] : (c == 1 ? Z.h[1] : (c == 2 ? Z.h[2] : Z.h[3]));
    const float zk = c == 0 ? -3.f : (c == 1 ? 9.f : (c == 2 ? -9.f : 3.f));
    XRow x[2];
    {
      const SliceData ct = nt;
      nt = src.load(c < 3 ? c + 1 : 3);  // the last slice reloads itself: no branch in the loop
      Src::template x_pass<true>(ct, xd, x);
    }
    const YIn v = Src::at(x[0].v, x[1].v), g = Src::at(x[0].g, x[1].g), h = Src::at(x[0].h, x[1].h),
              k = Src::at(x[0].k, x[1].k);
    const float mv = v.v2 - v.v1, mg = g.v2 - g.v1, mh = h.v2 - h.v1, mk = k.v2 - k.v1;
    const float s00 = y_value(Y, v, mv), s01 = y_first(Y, v, mv), s02 = y_second(Y, v), s03 = v.e2 - v.e1;
    const float s10 = y_value(Y, g, mg), s11 = y_first(Y, g, mg), s12 = y_second(Y, g);
    const float s20 = y_value(Y, h, mh), s21 = y_first(Y, h, mh), s30 = y_value(Y, k, mk);
    const float2 P0 = make_float2(s00, s01), P1 = make_float2(s10, s11), P2 = make_float2(s02, s20);
    W0 = ffma2(dup2(zw), P0, W0);
    W1 = ffma2(dup2(zw), P1, W1);
    W2 = ffma2(dup2(zw), P2, W2);
    W3 = ffma2(dup2(zw), make_float2(s12, s21), W3);
    W4 = ffma2(dup2(zw), make_float2(s03, s30), W4);
    G0 = ffma2(dup2(zg), P0, G0);
    G1 = ffma2(dup2(zg), P1, G1);
    G2 = ffma2(dup2(zg), P2, G2);
    H0 = ffma2(dup2(zh), P0, H0);
    o102 = fmaf(zh, s10, o102);
    o003 = fmaf(zk, s00, o003);
    if (scatter) {
      const SliceCotangents sc = slice_cotangents(qb, Y, zw, zg, zh);
      const float2 *Cw = sc.w, *Cg = sc.g, *Ch = sc.h;
      if constexpr (TakesCells<Acc>::value) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 p2 = ffma2(xd.t, Cw[j], Cg[j]), p1 = fsub2(Cw[j], p2);
          const float2 po = me ? p2 : p1, pn = me ? p1 : p2;
          const float2 eo = ffma2(ow, Cw[j], ffma2(og, Cg[j], fmul2(oh, Ch[j])));
          const float2 en = ffma2(nw, Cw[j], ffma2(ng, Cg[j], fmul2(nh, Ch[j])));
          acc.add_row2(at.even + j * at.px, at.odd + j * at.px, make_float4(po.x, po.y, eo.x, eo.y),
                           make_float4(pn.x, pn.y, en.x, en.y));
        }
        at.even += at.pxy;
        at.odd += at.pxy;
      } else {
        const int64_t row = base + c * G.pxy, px = G.px;
        float2 p1[2], p2[2], e1[2], e2[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          p2[j] = ffma2(xd.t, Cw[j], Cg[j]);
          p1[j] = fsub2(Cw[j], p2[j]);
          e1[j] = ffma2(xd.w0, Cw[j], ffma2(xd.g0, Cg[j], fmul2(xd.h0, Ch[j])));
          e2[j] = ffma2(xd.w3, Cw[j], ffma2(xd.g3, Cg[j], fmul2(xd.h3, Ch[j])));
        }
        const float2 n2 = dup2(-2.f);
        float2 t[2][4];  // taps along x of (value, difference along y) at rows 1 and 2
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          t[j][0] = e1[j];
          t[j][1] = fadd2(ffma2(n2, e1[j], p1[j]), e2[j]);
          t[j][2] = fadd2(ffma2(n2, e2[j], p2[j]), e1[j]);
          t[j][3] = e2[j];
        }
        float r1[4], r2[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          r1[i] = fmaf(-2.f, t[0][i].y, t[0][i].x) + t[1][i].y;
          r2[i] = fmaf(-2.f, t[1][i].y, t[1][i].x) + t[0][i].y;
        }
        acc.add_row(row, t[0][0].y, t[0][1].y, t[0][2].y, t[0][3].y);
        acc.add_row(row + px, r1[0], r1[1], r1[2], r1[3]);
        acc.add_row(row + 2 * px, r2[0], r2[1], r2[2], r2[3]);
        acc.add_row(row + 3 * px, t[1][0].y, t[1][1].y, t[1][2].y, t[1][3].y);
      }
    }
  }
  const float o030 = 3.f * W4.x, o300 = 3.f * W4.y;
  Q.v = W0.x;
  Q.g[0] = W1.x;
  Q.g[1] = W0.y;
  Q.g[2] = G0.x;
  Q.h[0] = W2.y;
  Q.h[1] = W1.y;
  Q.h[2] = G1.x;
  Q.h[3] = W2.x;
  Q.h[4] = G0.y;
  Q.h[5] = H0.x;
  // o000 W0.x, o010 W0.y, o100 W1.x, o110 W1.y, o020 W2.x, o200 W2.y, o120 W3.x,
  // o210 W3.y, o001 G0.x, o011 G0.y, o101 G1.x, o111 G1.y, o021 G2.x, o201 G2.y,
  // o002 H0.x, o012 H0.y: xb_j += qb . dQ/dx_j
  xb[0] += qb[0] * W1.x + qb[1] * W2.y + qb[2] * W1.y + qb[3] * G1.x + qb[4] * o300 + qb[5] * W3.y + qb[6] * G2.y +
           qb[7] * W3.x + qb[8] * G1.y + qb[9] * o102;
  xb[1] += qb[0] * W0.y + qb[1] * W1.y + qb[2] * W2.x + qb[3] * G0.y + qb[4] * W3.y + qb[5] * W3.x + qb[6] * G1.y +
           qb[7] * o030 + qb[8] * G2.x + qb[9] * H0.y;
  xb[2] += qb[0] * G0.x + qb[1] * G1.x + qb[2] * G0.y + qb[3] * H0.x + qb[4] * G2.y + qb[5] * G1.y + qb[6] * o102 +
           qb[7] * G2.x + qb[8] * H0.y + qb[9] * o003;
}

// The scatter of two stages whose footprints are the same cell (AccF32): the tap
// cotangents of (ta, qa) and (tb, qb) are added before they go to memory.
struct ScatterWeights {
  float2 t, ow, og, oh, nw, ng, nh;  // x: difference weights of this lane's cell of a pair and the other
  CWD y;
  CRW<float> z;
  SRT_HD ScatterWeights(const float* tt, int me) {
    CWD X;
    cr_weights_diff(tt[0], X);
    cr_weights_diff(tt[1], y);
    cr_weights_mixed(tt[2], z);
    t = dup2(X.t);
    ow = dup2(me ? X.w3 : X.w0), og = dup2(me ? X.g3 : X.g0), oh = dup2(me ? X.h3 : X.h0);
    nw = dup2(me ? X.w0 : X.w3), ng = dup2(me ? X.g0 : X.g3), nh = dup2(me ? X.h0 : X.h3);
  }
};
SRT_HD float of_slice(const float* w, int c) { return c == 0 ? w[0] : (c == 1 ? w[1] : (c == 2 ? w[2] : w[3])); }
SRT_HD void scatter_two(const AccF32& acc, int64_t base, int hbase, const Geom& G, const float* ta, const float* qa,
                        const float* tb, const float* qb) {
  AccF32::Place at = acc.place(base, hbase, G);
  const int me = AccF32::lane();
  const ScatterWeights a(ta, me), b(tb, me);
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    const SliceCotangents ca =
        slice_cotangents(qa, a.y, of_slice(a.z.w, c), of_slice(a.z.g, c), of_slice(a.z.h, c));
    const SliceCotangents cb =
        slice_cotangents(qb, b.y, of_slice(b.z.w, c), of_slice(b.z.g, c), of_slice(b.z.h, c));
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 p2 = ffma2(a.t, ca.w[j], fadd2(ca.g[j], ffma2(b.t, cb.w[j], cb.g[j])));
      const float2 p1 = fsub2(fadd2(ca.w[j], cb.w[j]), p2);
      const float2 po = me ? p2 : p1, pn = me ? p1 : p2;
      const float2 eo =
          ffma2(a.ow, ca.w[j], ffma2(a.og, ca.g[j], ffma2(a.oh, ca.h[j],
          ffma2(b.ow, cb.w[j], ffma2(b.og, cb.g[j], fmul2(b.oh, cb.h[j]))))));
      const float2 en =
          ffma2(a.nw, ca.w[j], ffma2(a.ng, ca.g[j], ffma2(a.nh, ca.h[j],
          ffma2(b.nw, cb.w[j], ffma2(b.ng, cb.g[j], fmul2(b.nh, cb.h[j]))))));
      acc.add_row2(at.even + j * at.px, at.odd + j * at.px, make_float4(po.x, po.y, eo.x, eo.y),
                   make_float4(pn.x, pn.y, en.x, en.y));
    }
    at.even += at.pxy;
    at.odd += at.pxy;
  }
}

// -------------------------------------------------------- stage and core

// What the right-hand-side vjp needs about one stage input, independent of
// the state representation (FP64 full state or MIXED perturbation state).
template <typename T>
struct StageView {
  T n[3], a[3], b[3];  // unit vectors n, e1, e2
  T rn, ra, rb;        // 1 / |raw vector| (normalisation Jacobians)
  T A, Ap, s1, s2, e1, e2;
  bool branch;         // dA > 1/2
  int64_t base[4];     // padded base index per field: B_x, B_y, B_z, phi
  int64_t basep[4];    // the same cells in the row-pair and half-cell layouts
  int hbase[4];        // the same cells near the observer (hot_base; MIXED)
  T t[4][3];           // cell offsets per field and axis
};

// symmetric 3x3 as unique components xx xy xz yy yz zz
SRT_HD int sym_idx(int i, int j) {
  return (i == j) ? (i == 0 ? 0 : (i == 1 ? 3 : 5)) : ((i + j == 1) ? 1 : ((i + j == 2) ? 2 : 4));
}

// One field's pass: FP32 (MIXED) from the handle's layout; FP64 in the plain form.
template <int LAYOUT, int UNROLL, typename T, typename Acc>
SRT_HD void field_pass(const FieldPtrs& F, int f, const StageView<T>& V, const Geom& G, const T* qb, Tri<T>& Q, T* xb,
                       const Acc& acc) {
  const int64_t base = V.base[f], basep = V.basep[f];
  const T* t = V.t[f];
  if constexpr (sizeof(T) == sizeof(float))
    tricubic_vjp_mixed<UNROLL, Acc>(cell_source<LAYOUT>(F, G, f, base, basep), base, V.hbase[f], G, t, qb, Q, xb, acc);
  else
    tricubic_vjp<T, Acc>(f == 3 ? F.phi : F.b[f], base, G.px, G.pxy, G.ts, t[0], t[1], t[2], qb, Q, xb, acc);
}

SRT_HD float fm(float a, float b, float c) { return fmaf(a, b, c); }
SRT_HD double fm(double a, double b, double c) { return fma(a, b, c); }
template <typename T>
SRT_HD T vdot(const T* a, const T* b) { return fm(a[2], b[2], fm(a[1], b[1], a[0] * b[0])); }
// Row i of a symmetric matrix (xx xy xz yy yz zz) times v.
template <typename T>
SRT_HD T sym_row(const T* h, int i, const T* v) {
  return fm(h[sym_idx(i, 2)], v[2], fm(h[sym_idx(i, 1)], v[1], h[sym_idx(i, 0)] * v[0]));
}

// What the B components' passes share. Cotangents, known before any field is
// read: u = (n.grad B)bar + e1bar e1 / 2 + e2bar e2 / 2, h1 = e1bar / 2,
// h2 = e2bar / 2, Tb that of the tidal matrix and D its diagonal plus that of
// n . Laplacian B. Sums over the components as BSums64's (Gn = G n,
// ngB = G^T n, S = sum_C n_C H_C, K_ij = (H_i n)_j + (H_j n)_i).
template <typename T>
struct BVjp {
  T u[3], h1, h2, Tb[6], D[3];
  T Gn[3], ngB[3], S[6], K[6], nlap;
};

// B component C's cotangents (value, gradient, Hessian).
template <int C, typename T>
SRT_HD void b_cotangent(const StageView<T>& V, const T* fb, const BVjp<T>& B, T* qb) {
  const T* n = V.n;
  const T nc = n[C], n2 = T(2) * nc, kap = fm(B.h1, V.a[C], B.h2 * V.b[C]);
  const T Tc[3] = {B.Tb[sym_idx(C, 0)], B.Tb[sym_idx(C, 1)], B.Tb[sym_idx(C, 2)]};
  qb[0] = -fb[C];
  for (int i = 0; i < 3; ++i) qb[1 + i] = fm(nc, B.u[i], kap * n[i]);
  // Hessian cotangent n_c (Tb + nlapb I) - sym(Tb_c. (x) n), off-diagonals
  // holding both halves
  for (int i = 0; i < 3; ++i) {
    qb[4 + sym_idx(i, i)] = fm(nc, B.D[i], -(Tc[i] * n[i]));
    for (int j = i + 1; j < 3; ++j)
      qb[4 + sym_idx(i, j)] = fm(n2, B.Tb[sym_idx(i, j)], -fm(Tc[i], n[j], Tc[j] * n[i]));
  }
}

// Its interpolation Q folded into the sums and into nb, the cotangent of n
// (those of e1 and e2 follow from the sums).
template <int C, typename T>
SRT_HD void b_fold(const StageView<T>& V, const Tri<T>& Q, BVjp<T>& B, T* nb) {
  const T* n = V.n;
  const T nc = n[C], kap = fm(B.h1, V.a[C], B.h2 * V.b[C]);
  const T Tc[3] = {B.Tb[sym_idx(C, 0)], B.Tb[sym_idx(C, 1)], B.Tb[sym_idx(C, 2)]};
  for (int i = 0; i < 3; ++i) B.ngB[i] = fm(Q.g[i], nc, C == 0 ? T(0) : B.ngB[i]);
  B.Gn[C] = vdot(Q.g, n);
  B.nlap = fm(nc, Q.h[0] + Q.h[3] + Q.h[5], C == 0 ? T(0) : B.nlap);
  for (int k = 0; k < 6; ++k) B.S[k] = fm(nc, Q.h[k], C == 0 ? T(0) : B.S[k]);
  for (int i = 0; i < 3; ++i) {
    const T Hn = sym_row(Q.h, i, n);
    T& k = B.K[sym_idx(C, i)];  // met at component min(i, C) first, max(i, C) second
    k = i == C ? Hn + Hn : (i > C ? Hn : k + Hn);
  }
  // H_c : (Tb + nlapb I)
  const T HT = fm(Q.h[0], B.D[0], fm(Q.h[3], B.D[1], Q.h[5] * B.D[2])) +
               T(2) * fm(Q.h[1], B.Tb[1], fm(Q.h[2], B.Tb[2], Q.h[4] * B.Tb[4]));
  nb[C] += vdot(Q.g, B.u) + HT;
  for (int k = 0; k < 3; ++k) nb[k] += fm(kap, Q.g[k], -sym_row(Q.h, k, Tc));
}

// What phi's cotangents take from the state.
template <typename T>
struct PhiVjp {
  T nfx, e1b, e2b, Lb, PHb, vb[3], Heb[6];
};
template <typename T>
SRT_HD void phi_cotangent(const StageView<T>& V, const PhiVjp<T>& p, T* qb) {
  qb[0] = T(-2) * p.nfx;
  for (int i = 0; i < 3; ++i)
    qb[1 + i] = fm(T(2), fm(p.e1b, V.a[i], fm(p.e2b, V.b[i], p.vb[i])), V.n[i] * p.Lb);
  for (int i = 0; i < 3; ++i) {
    const T t = V.n[i] * p.PHb;
    qb[4 + sym_idx(i, i)] = fm(V.n[i], t, p.Heb[sym_idx(i, i)] - p.PHb);
    for (int j = i + 1; j < 3; ++j) qb[4 + sym_idx(i, j)] = T(2) * fm(t, V.n[j], p.Heb[sym_idx(i, j)]);
  }
}

// The four fused passes of a stage by one lane: the B sums and nb, the position
// cotangent xb and phi's interpolation P. The slice loops are unrolled where only
// phi's scatter follows them, loops with four scatters, where the code outgrows
// the instruction cache (SRT_DETERMINISTIC's sweep; the FP32 one scatters apart
// from the interpolations).
template <int LAYOUT, typename T, typename AccB, typename AccP>
struct OneLanePasses {
  const FieldPtrs& F;
  const Geom& G;
  const AccB* accb;
  const AccP& accp;
  static constexpr int kUnroll = std::is_same<AccB, AccNone>::value ? 4 : 1;
  template <int C>
  SRT_HD void component(const StageView<T>& V, const T* fb, BVjp<T>& B, T* nb, T* xb) const {
    T qb[10];
    b_cotangent<C>(V, fb, B, qb);
    Tri<T> Q;
    field_pass<LAYOUT, kUnroll, T, AccB>(F, C, V, G, qb, Q, xb, accb[C]);
    b_fold<C>(V, Q, B, nb);
  }
  SRT_HD void operator()(const StageView<T>& V, const T* fb, const PhiVjp<T>& p, BVjp<T>& B, T* nb, T* xb,
                         Tri<T>& P) const {
    // compile-time component index: no local-memory arrays
    component<0>(V, fb, B, nb, xb);
    component<1>(V, fb, B, nb, xb);
    component<2>(V, fb, B, nb, xb);
    T qb[10];
    phi_cotangent(V, p, qb);
    field_pass<LAYOUT, kUnroll, T, AccP>(F, 3, V, G, qb, P, xb, accp);
  }
};

// yb += J(u)^T fb for the stage described by V, its four passes by `passes`.
template <typename T, typename Passes>
SRT_HD void rhs_vjp_with(const StageView<T>& V, const T* fb, T* yb, const Passes& passes) {
  const T* n = V.n;
  const T* a = V.a;
  const T* b = V.b;
  // ---- intermediate cotangents (state only)
  const T nfx = vdot(n, fb), nfn = vdot(n, fb + 3);
  const T e1b = -vdot(n, fb + 6), e2b = -vdot(n, fb + 9);
  T vb[3];
  for (int i = 0; i < 3; ++i) vb[i] = fm(-n[i], nfn, fb[3 + i]);
  T Apb = -fb[12];
  const T Lb = T(4) * fm(V.s1, fb[14], fm(V.s2, fb[15], -(V.Ap * fb[13])));
  const T PHb = -V.A * fb[13], nlapb = T(0.5) * V.A * fb[13];
  const T A2 = V.A * V.A;
  const T S1b = A2 * fb[14], S2b = A2 * fb[15];
  // the dA > 1/2 branch's terms, formed either way and selected (no branch;
  // where dA = 0 they are not finite and not selected)
  T Ab = 0, s1b = 0, s2b = 0, el1b = 0, el2b = 0;
  {
    const T iA = T(1) / V.A, iA2 = iA * iA, iA3 = iA2 * iA;
    const T q = sqrt(fm(V.e2, V.e2, fm(V.e1, V.e1, T(4))));
    const T iD = T(1) / (A2 * (T(2) + q));  // of the rotation's quotient N / D
    const T N = fm(V.s1, V.e2, -(V.s2 * V.e1)), Nb = -fb[18] * iD, NN = N * Nb;  // D times D's cotangent is -NN
    const T sf = fm(V.s1, fb[16], V.s2 * fb[17]), c13 = T(2) * iA3 * fb[13], cq = T(-2) * q * iA2;
    const T bs1 = fm(V.s1, c13, fm(cq, fb[16], V.e2 * Nb)), bs2 = fm(V.s2, c13, fm(cq, fb[17], -(V.e1 * Nb)));
    const T bA = iA * (T(-1.5) * fm(V.s1, V.s1, V.s2 * V.s2) * c13 + T(-2) * fm(cq, sf, NN));
    const T qq = fm(T(-2) * iA2, sf, -(A2 * iD) * NN) / q;  // q's cotangent over q
    s1b = V.branch ? bs1 : T(0);
    s2b = V.branch ? bs2 : T(0);
    Ab = V.branch ? bA : T(0);
    el1b = V.branch ? fm(V.e1, qq, -(V.s2 * Nb)) : T(0);
    el2b = V.branch ? fm(V.e2, qq, V.s1 * Nb) : T(0);
  }
  // cotangent of the effective tidal matrix He = H + T/2:
  // (a a - b b) S1b + (a b + b a) S2b = a p + b r, symmetric
  T p[3], r[3], Heb[6];
  for (int i = 0; i < 3; ++i) {
    p[i] = fm(S1b, a[i], S2b * b[i]);
    r[i] = fm(S2b, a[i], -(S1b * b[i]));
  }
  for (int i = 0; i < 3; ++i)
    for (int j = i; j < 3; ++j) Heb[sym_idx(i, j)] = fm(a[i], p[j], b[i] * r[j]);
  BVjp<T> B;
  B.h1 = T(0.5) * e1b;
  B.h2 = T(0.5) * e2b;
  for (int k = 0; k < 6; ++k) B.Tb[k] = T(0.5) * Heb[k];
  for (int i = 0; i < 3; ++i) {
    B.D[i] = B.Tb[sym_idx(i, i)] + nlapb;
    const T ngBb = fm(T(0.25) * n[i], Lb, vb[i]);
    B.u[i] = fm(B.h1, a[i], fm(B.h2, b[i], ngBb));
  }
  PhiVjp<T> ph;
  ph.nfx = nfx, ph.e1b = e1b, ph.e2b = e2b, ph.Lb = Lb, ph.PHb = PHb;
  for (int i = 0; i < 3; ++i) ph.vb[i] = vb[i];
  for (int k = 0; k < 6; ++k) ph.Heb[k] = Heb[k];
  T nb[3] = {0, 0, 0}, xb[3] = {0, 0, 0};
  Tri<T> P;
  passes(V, fb, ph, B, nb, xb, P);
  const T* g = P.g;
  // ---- the rest of n's cotangent, and those of e1, e2 and the scalars
  T v[3], w[3], Hn[3];
  for (int i = 0; i < 3; ++i) {
    v[i] = fm(T(2), g[i], B.ngB[i]);
    w[i] = fm(T(0.5), B.Gn[i] + B.ngB[i], T(2) * g[i]);  // e.w = 2 e.grad phi + e.n.grad B
    Hn[i] = sym_row(P.h, i, n);
  }
  const T nv = vdot(n, v), sa = vdot(a, w), sb = vdot(b, w);
  const T L4 = fm(T(4), vdot(n, g), vdot(n, B.ngB)), phi1 = fm(T(2), P.v, T(1)), PH2 = T(2) * PHb;
  for (int i = 0; i < 3; ++i) {
    T t = fm(T(0.25), B.ngB[i], g[i]) * Lb;
    t = fm(PH2, Hn[i], t);
    t = fm(-phi1, fb[i], t);
    t = fm(-nv, fb[3 + i], t);
    t = fm(-v[i], nfn, t);
    t = fm(-sa, fb[6 + i], t);
    nb[i] += fm(-sb, fb[9 + i], t);
  }
  Apb = fm(-L4, fb[13], Apb);
  s1b = fm(L4, fb[14], s1b);
  s2b = fm(L4, fb[15], s2b);
  // -P_perp:H + n.Laplacian B / 2
  Ab = fm(fm(T(0.5), B.nlap, (P.h[0] + P.h[3] + P.h[5]) - vdot(n, Hn)), fb[13], Ab);
  T He[6], ab[3], bb[3], Hea[3], Heb3[3];
  for (int k = 0; k < 6; ++k) He[k] = fm(T(-0.25), B.K[k], fm(T(0.5), B.S[k], P.h[k]));
  for (int i = 0; i < 3; ++i) {
    Hea[i] = sym_row(He, i, a);
    Heb3[i] = sym_row(He, i, b);
  }
  const T S1 = vdot(a, Hea) - vdot(b, Heb3), S2 = T(2) * vdot(a, Heb3);
  Ab = fm(T(2) * V.A, fm(S1, fb[14], S2 * fb[15]), Ab);
  const T S1d = T(2) * S1b, S2d = T(2) * S2b;
  for (int i = 0; i < 3; ++i) {
    ab[i] = fm(e1b, w[i], fm(S1d, Hea[i], S2d * Heb3[i]));
    bb[i] = fm(e2b, w[i], fm(S2d, Hea[i], -(S1d * Heb3[i])));
  }

  // ---- through the normalisations, into the state cotangent
  const T nnb = vdot(n, nb), aab = vdot(a, ab), bbb = vdot(b, bb);
  for (int i = 0; i < 3; ++i) {
    yb[i] += xb[i];
    yb[3 + i] = fm(V.rn, fm(-n[i], nnb, nb[i]), yb[3 + i]);
    yb[6 + i] = fm(V.ra, fm(-a[i], aab, ab[i]), yb[6 + i]);
    yb[9 + i] = fm(V.rb, fm(-b[i], bbb, bb[i]), yb[9 + i]);
  }
  yb[12] += Ab;
  yb[13] += Apb;
  yb[14] += s1b;
  yb[15] += s2b;
  yb[16] += el1b;
  yb[17] += el2b;
}

// The same by one lane; tap cotangents go to accb[0..2] (B_x, B_y, B_z) and accp
// (phi).
template <typename T, typename AccB, typename AccP, int LAYOUT = kPlanes>
SRT_HD void rhs_vjp(const StageView<T>& V, const FieldPtrs& F, const Geom& G, const T* fb, T* yb, const AccB* accb,
                    const AccP& accp) {
  rhs_vjp_with(V, fb, yb, OneLanePasses<LAYOUT, T, AccB, AccP>{F, G, accb, accp});
}

// ------------------------------------------------------- stage views

// FP64 full state y (layout of rhs_std).
SRT_HD void stage_view_fp64(const double* y, const Geom& G, StageView<double>& V) {
  const double nr = sqrt(y[3] * y[3] + y[4] * y[4] + y[5] * y[5]);
  const double ar = sqrt(y[6] * y[6] + y[7] * y[7] + y[8] * y[8]);
  const double br = sqrt(y[9] * y[9] + y[10] * y[10] + y[11] * y[11]);
  V.rn = 1.0 / nr;
  V.ra = 1.0 / ar;
  V.rb = 1.0 / br;
  for (int i = 0; i < 3; ++i) {
    V.n[i] = y[3 + i] / nr;
    V.a[i] = y[6 + i] / ar;
    V.b[i] = y[9 + i] / br;
  }
  V.A = y[12];
  V.Ap = y[13];
  V.s1 = y[14];
  V.s2 = y[15];
  V.e1 = y[16];
  V.e2 = y[17];
  V.branch = y[12] > 0.5;
  for (int f = 0; f < 4; ++f) {
    int cell[3];
    for (int i = 0; i < 3; ++i) {
      const double x = y[i] - ((f == i) ? 0.5 : 0.0);
      const double fl = floor(x);
      V.t[f][i] = x - fl;
      cell[i] = wrap64((int64_t)fl, G.n[i]);
    }
    V.base[f] = cell_base(G, cell[0], cell[1], cell[2]);
    V.basep[f] = cell_base_pair(G, cell[0], cell[1], cell[2]);
  }
}

// MIXED perturbation state d at affine parameter s (layout of rhs_mixed).
SRT_HD void stage_view_mixed(const float* d, float s, const MixedRay& R, const Geom& G, const float* x0,
                             StageView<float>& V) {
  const float* v0s[3] = {R.n0, R.a0, R.b0};
  float* outs[3] = {V.n, V.a, V.b};
  float* rs[3] = {&V.rn, &V.ra, &V.rb};
  for (int k = 0; k < 3; ++k) {
    const float* v0 = v0s[k];
    const float* dv = d + 3 + 3 * k;
    const float q = R.eta[k] + 2.f * (v0[0] * dv[0] + v0[1] * dv[1] + v0[2] * dv[2]) +
                    (dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]);
    const float rm1 = rsqrt1p_m1(q);
    *rs[k] = 1.f + rm1;
    for (int i = 0; i < 3; ++i) outs[k][i] = v0[i] + (v0[i] * rm1 + dv[i] * (1.f + rm1));
  }
  V.A = s + d[12];
  V.Ap = d[13] - 1.f;
  V.s1 = d[14];
  V.s2 = d[15];
  V.e1 = d[16];
  V.e2 = d[17];
  V.branch = d[12] > 0.5f - s;
  int cc[3], cs[3];
  float tc[3], ts[3];
  for (int i = 0; i < 3; ++i) {
    const float p = s * R.n0[i];
    const float pe = fmaf(s, R.n0[i], -p);
    float th, tl;
    two_sum(x0[i], -p, th, tl);
    const float lo = (tl - pe) + d[i];
    float df;
    locate_mixed(th, lo, G.n[i], G.invn[i], cc[i], tc[i], cs[i], ts[i], df);
  }
  for (int f = 0; f < 4; ++f) {
    int cell[3];
    for (int i = 0; i < 3; ++i) {
      const bool stag = (f == i);
      cell[i] = stag ? cs[i] : cc[i];
      V.t[f][i] = stag ? ts[i] : tc[i];
    }
    V.base[f] = cell_base(G, cell[0], cell[1], cell[2]);
    V.basep[f] = cell_base_pair(G, cell[0], cell[1], cell[2]);
    V.hbase[f] = hot_base(G, cell);
  }
}

}  // namespace srt
