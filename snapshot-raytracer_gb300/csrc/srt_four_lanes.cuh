// srt_four_lanes.cuh — a MIXED stage by four lanes that hold the same ray, one
// field each: the kernels of small ranges, forward and adjoint (device code).
#pragma once
#include "srt_scheme.cuh"

namespace srt {

// The interpolation lane first + f of a group holds.
__device__ __forceinline__ void fetch_tri(const Tri<float>& own, int f, int first, Tri<float>& r) {
  const unsigned mask = 0xfu << first;
  r.v = __shfl_sync(mask, own.v, first + f);
#pragma unroll
  for (int i = 0; i < 3; ++i) r.g[i] = __shfl_sync(mask, own.g[i], first + f);
#pragma unroll
  for (int i = 0; i < 6; ++i) r.h[i] = __shfl_sync(mask, own.h[i], first + f);
}

// The stage's interpolations by a group of four lanes that hold the same ray,
// one field each (B_x, B_y, B_z, phi), exchanged by shuffles; every lane then
// folds them in OneLane's order, so the values are the same bits.
template <int LAYOUT>
struct FourLanes {
  int field, first;  // this lane's field; the group's first lane
  __device__ void operator()(const FieldPtrs& F, const Geom& G, const int* cc, const int* cs, const float* tc,
                             const float* ts, const float* n, BAcc& A, Tri<float>& p) const {
    Tri<float> own;
    {
      AxisWeights<LAYOUT> X, Y;
      CRW<float> Z;
      axis_weights(field == 0 ? ts[0] : tc[0], X);
      axis_weights(field == 1 ? ts[1] : tc[1], Y);
      cr_weights_mixed(field == 2 ? ts[2] : tc[2], Z);
      const int cx = field == 0 ? cs[0] : cc[0], cy = field == 1 ? cs[1] : cc[1], cz = field == 2 ? cs[2] : cc[2];
      tricubic_mixed(cell_source<LAYOUT>(F, G, field, cx, cy, cz), X, Y, Z, own);
    }
    Tri<float> r;
    fetch_tri(own, 0, first, r);
    add_b_component<0>(r, n, A);
    fetch_tri(own, 1, first, r);
    add_b_component<1>(r, n, A);
    fetch_tri(own, 2, first, r);
    add_b_component<2>(r, n, A);
    fetch_tri(own, 3, first, p);
  }
};

}  // namespace srt
