// srt_adjoint.cu — vjp of the six maps with respect to the phi and B grids
// (srt_vjp in include/srt.h). The reference has no derivatives; what is
// differentiated is its forward scheme, snapshot-raytracer.cu:315-583, as
// restated in srt_scheme.cuh.
//
// Kernels (rays in the forward's launch order):
//   ray_count_, ray_scan_,  Morton-ordered list of the RING pixels of the
//   ray_write_kernel        requested range
//   ckpt_kernel             forward trace storing the state every C steps (and
//                           the final state); of the last segments the tape too
//   near_ckpt_kernel        the same for the rays that came near a cell face, by
//                           the four-tap passes
//   final_cotangent_kernel  cotangent of the final state from the map weights
//   segment_kernel          per segment, backwards: recompute it from its
//                           checkpoint, writing every stage's input (the tape)
//   sweep_kernel            then its steps, backwards, by the RK4 adjoint,
//                           scattering the tap cotangents into halo-padded
//                           gradient grids (FP32 atomics on cells, or 64-bit
//                           fixed point for SRT_DETERMINISTIC)
//   reverse_kernel_fp64     both in one, FP64 (atomics, or fixed point)
//   *_small_kernel          ranges of few rays, four lanes per ray
//   merge_hot_kernel        adds the copies of the region around the observer
//   fold_kernel             sums the halo copies of each voxel back onto the
//                           periodic grid and writes the caller's layout
#include <algorithm>
#include <chrono>
#include <cstring>
#include <type_traits>
#include "srt_adjoint.cuh"
#include "srt_four_lanes.cuh"
#include "srt_internal.h"

namespace srt {

// ------------------------------------------------------------- ray list

struct RangeArgs {
  int64_t nside, pix_begin, pix_count, launch_rays;
  int log2p;
};

__device__ __forceinline__ int64_t ring_of_slot(const RangeArgs& a, int64_t t) {
  if (t >= a.launch_rays) return -1;
  const int64_t face = t >> (2 * a.log2p);
  int64_t ix, iy;
  hp_deinterleave(t & ((int64_t(1) << (2 * a.log2p)) - 1), &ix, &iy);
  if (ix >= a.nside || iy >= a.nside) return -1;
  const int64_t ring = hp_xyf2ring(a.nside, ix, iy, (int)face);
  return (ring >= a.pix_begin && ring < a.pix_begin + a.pix_count) ? ring : -1;
}

constexpr int kListBlock = 256;

__global__ void ray_count_kernel(const RangeArgs a, int* counts) {
  const int64_t t = (int64_t)blockIdx.x * kListBlock + threadIdx.x;
  const int in = ring_of_slot(a, t) >= 0;
  const int c = __syncthreads_count(in);
  if (threadIdx.x == 0) counts[blockIdx.x] = c;
}

// Exclusive sums of n block counts, by one block.
__global__ void __launch_bounds__(1024) ray_scan_kernel(const int* counts, int64_t n, int64_t* offsets) {
  __shared__ int warp_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t run = 0;
  for (int64_t q0 = 0; q0 < n; q0 += 1024) {
    const int64_t q = q0 + threadIdx.x;
    const int c = q < n ? counts[q] : 0;
    int sum = c;  // inclusive within the warp
    for (int d = 1; d < 32; d *= 2) {
      const int v = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += v;
    }
    if (lane == 31) warp_sum[warp] = sum;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      before += w < warp ? warp_sum[w] : 0;
      all += warp_sum[w];
    }
    if (q < n) offsets[q] = run + before + sum - c;
    run += all;
    __syncthreads();
  }
}

__global__ void ray_write_kernel(const RangeArgs a, const int64_t* offsets, int64_t* rays) {
  __shared__ int warp_tot[kListBlock / 32];
  const int64_t t = (int64_t)blockIdx.x * kListBlock + threadIdx.x;
  const int64_t ring = ring_of_slot(a, t);
  const unsigned mask = __ballot_sync(0xffffffffu, ring >= 0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) warp_tot[warp] = __popc(mask);
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += warp_tot[w];
  if (ring >= 0) rays[offsets[blockIdx.x] + before + __popc(mask & ((1u << lane) - 1u))] = ring;
}

// ------------------------------------------------------------ arguments

struct AdjArgs {
  FieldPtrs F;
  Geom G;
  int64_t nside, pix_begin, count;
  int64_t* rays;  // RING pixels, Morton order; kNearBit: near a cell face
  int64_t* near;  // [0] the number of marked rays, [1 ...] their slots
  float* bases;   // [12][count]: n0, e1, e2 and eta of the rays' MixedRay
  int n_steps, C, nseg;
  const float* w[6];  // map weights, indexed by ring - pix_begin
  void* ckpt;         // [nseg + 1][state][count]
  void* seg;          // [C][state + 57][count] (FP64); MIXED: the tape (kTapeStep)
  int tape_from;      // MIXED forward: steps from here on go to the tape at once
  void* acc[4];       // padded gradient accumulators B_x, B_y, B_z, phi (NULL: not wanted)
  // forward with a tape (srt_forward_tape): the maps, indexed by ring - pix_begin,
  // and the output slots of rays that came within the cell-face guard
  float* maps[6];
  int64_t* refine_list;
  unsigned long long* refine_count;
};

template <typename T>
__device__ __forceinline__ void store_vec(T* base, int64_t count, int64_t slot, const T* v, int n) {
  for (int j = 0; j < n; ++j) base[(int64_t)j * count + slot] = v[j];
}
template <typename T>
__device__ __forceinline__ void load_vec(const T* base, int64_t count, int64_t slot, T* v, int n) {
  for (int j = 0; j < n; ++j) v[j] = base[(int64_t)j * count + slot];
}

// ------------------------------------------------------------ MIXED mode


// Floats of one step of the MIXED tape: the four stage inputs.
constexpr int kTapeStep = 4 * 19;

// The rays' straight-ray bases, stored by the checkpointing forward: forming
// them takes ~150 FP64 instructions a ray, which every segment's two launches
// would repeat (3 % of a 512^3 / nside 256 / 256 steps gradient).
__device__ __forceinline__ void store_bases(const AdjArgs& A, int64_t slot, const MixedRay& R) {
  store_vec(A.bases, A.count, slot, R.n0, 3);
  store_vec(A.bases + 3 * A.count, A.count, slot, R.a0, 3);
  store_vec(A.bases + 6 * A.count, A.count, slot, R.b0, 3);
  store_vec(A.bases + 9 * A.count, A.count, slot, R.eta, 3);
}
__device__ __forceinline__ void load_bases(const AdjArgs& A, int64_t slot, MixedRay& R) {
  load_vec(A.bases, A.count, slot, R.n0, 3);
  load_vec(A.bases + 3 * A.count, A.count, slot, R.a0, 3);
  load_vec(A.bases + 6 * A.count, A.count, slot, R.b0, 3);
  load_vec(A.bases + 9 * A.count, A.count, slot, R.eta, 3);
}

// Rays whose trajectory comes within the cell-face guard (a few in 10,000) keep
// the four-tap passes' trajectory in the adjoint. Which side of a face FP32
// rounding puts such a ray on decides its Hessian weights there, and with them
// single voxels of the gradient (by up to 4e-3 of its rms at 512^3 / nside 256 /
// 256 steps), so the second-difference passes' rounding is not let decide it:
// ckpt_kernel_mixed marks and lists these rays, near_ckpt_kernel traces their
// checkpoints again, and the segment kernel's first blocks take them apart.
constexpr int64_t kNearBit = int64_t(1) << 62;

__device__ __forceinline__ int64_t ring_of(const AdjArgs& A, int64_t slot) { return A.rays[slot] & ~kNearBit; }
__device__ __forceinline__ bool is_near(const AdjArgs& A, int64_t slot) { return (A.rays[slot] & kNearBit) != 0; }

// f(slot, together) for each marked ray, by blocks 0 .. blocks - 1 of four warps: up
// to kNearPerWarp rays per warp of the first warp_blocks by a warp each (together: all
// 32 lanes hold the ray; 12 us a step), longer lists by a lane each in all blocks (~40
// us a step, 32 rays at a time). A warp per ray whatever the list made the gradient of
// strong fields slower than one without this pass: 256^3 / nside 128 / 128 steps, C =
// 12, 669 / 1,881 / 6,024 rays marked of 196,608: 46.6 / 59.6 / 99.2 ms, now 43.9 /
// 49.6 / 57.4, and 41.4 with 8.
constexpr int kNearPerWarp = 2;

template <typename Fn>
__device__ __forceinline__ void for_near_rays(const AdjArgs& A, int64_t blocks, int64_t warp_blocks, const Fn& f) {
  const int64_t n = A.near[0], warp = threadIdx.x >> 5;
  const bool together = n <= kNearPerWarp * warp_blocks * 4;
  if (together && blockIdx.x >= warp_blocks) return;
  // consecutive warps of rays in consecutive blocks
  const int64_t step = together ? warp_blocks * 4 : blocks * 128;
  const int64_t first = together ? warp * warp_blocks + blockIdx.x
                                 : (warp * blocks + blockIdx.x) * 32 + (threadIdx.x & 31);
#pragma unroll 1
  for (int64_t i = first; i < n; i += step) f(A.near[1 + i], together);
}

// Touches the footprints of the step after `step` along the straight ray, two
// rows of one field per lane, so that the ray's own loads find them in L1: a
// marked ray is traced by a warp whose lanes all hold it, with no neighbours
// to share taps with (38 -> 11 us a step).
__device__ __forceinline__ void prefetch_step(const AdjArgs& A, const MixedRay& R, const float* x0, const float* y,
                                              int step) {
  const int lane = threadIdx.x & 31, f = lane >> 3, sub = lane & 7;
  int cell[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float p = x0[i] - (float)(step + 1) * R.n0[i] + y[i] - (f == i ? 0.5f : 0.f);
    cell[i] = wrap32((int)floorf(p), A.G.n[i], A.G.invn[i]);
  }
  const float* v = (f == 3 ? A.F.phi : (f == 0 ? A.F.b[0] : (f == 1 ? A.F.b[1] : A.F.b[2]))) +
                   (cell_base(A.G, cell[0], cell[1], cell[2]) + (sub >> 1) * A.G.pxy + 2 * (sub & 1) * A.G.px) * A.G.ts;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float t;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(t) : "l"(v + ((e >> 1) * A.G.px + 3 * (e & 1)) * A.G.ts));
    (void)t;
  }
}

// Forward trace of one ray storing the state every C steps (and the final
// state); y holds the final state.
// TAPE: the stage inputs of steps tape_from on go to the tape (by lanes with
// `tape`), so that those segments are not recomputed. together: a marked ray that all
// lanes of the warp hold.
template <bool TAPE, typename Interp>
__device__ __forceinline__ void ckpt_ray(const Interp& interp, const AdjArgs& A, int64_t slot, const RayDir& d,
                                         MixedRay& R, float* y, Guard& gd, bool tape = true, bool together = false) {
  constexpr bool kNear = std::is_same<Interp, OneLane<kFourTaps>>::value;
  float x0[3];
  mixed_observer(A.G, x0);
  init_mixed(d, R, y);
  if (!kNear) store_bases(A, slot, R);
  float* ck = (float*)A.ckpt;
  store_vec(ck, A.count, slot, y, kMixedState);
#pragma unroll 1
  for (int st = 0; st < A.n_steps; ++st) {
    if (kNear && together) prefetch_step(A, R, x0, y, st);
    if (gd.m) gd.begin_step(y);
    float* us = TAPE && tape && st >= A.tape_from
                    ? (float*)A.seg + (int64_t)(st - A.tape_from) * kTapeStep * A.count + slot
                    : nullptr;
    step_mixed(interp, R, A.F, A.G, x0, st, y, us, A.count, gd);
    if (gd.m) gd.end_step(st);
    const int done = st + 1;
    if (done % A.C == 0 || done == A.n_steps) {
      const int k = (done + A.C - 1) / A.C;
      store_vec(ck + (int64_t)k * kMixedState * A.count, A.count, slot, y, kMixedState);
    }
  }
}

// The checkpoints of one ray, with the cell-face guard of the trace kernel; marks
// and lists it where the guard catches it. MAPS (srt_forward_tape): also its maps
// and the list of rays to re-trace; the arithmetic is the trace kernels', so the
// maps are srt_forward's. first: this lane writes what a ray has once.
template <bool MAPS, typename Interp>
__device__ __forceinline__ void ckpt_one(const Interp& interp, const AdjArgs& A, int64_t slot, bool first,
                                         float* guard_m) {
  const int64_t ring = ring_of(A, slot);
  MixedRay R;
  float y[kMixedState];
  Guard gd;
  gd.m = guard_m;
  gd.m[0] = 0.f;
  ckpt_ray<!MAPS>(interp, A, slot, ray_dir_pix(A.nside, ring), R, y, gd, first);
  if (!first) return;
  if (gd.near) {
    A.rays[slot] = ring | kNearBit;
    A.near[1 + atomicAdd((unsigned long long*)A.near, 1ull)] = slot;
  }
  if (MAPS) {
    const int64_t o = ring - A.pix_begin;
    float out[6];
    extract_mixed(R, A.n_steps, y, out);
#pragma unroll
    for (int m = 0; m < 6; ++m) A.maps[m][o] = out[m];
    if (gd.near && A.refine_list) {
      const unsigned long long k = atomicAdd(A.refine_count, 1ull);
      if (k < (unsigned long long)A.count) A.refine_list[k] = o;
    }
  }
}

template <int LAYOUT, bool MAPS>
__global__ void __launch_bounds__(128, 2) ckpt_kernel_mixed(const AdjArgs A) {
  const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= A.count) return;
  __shared__ float guard_m[128][2];
  ckpt_one<MAPS>(OneLane<LAYOUT>(), A, slot, true, guard_m[threadIdx.x]);
}

// Small ranges, forward and adjoint: four lanes per ray, one-warp blocks (at most four
// per SM, so the four taps get the registers that trace_small_kernel gives them).
template <int LAYOUT, bool MAPS>
__global__ void __launch_bounds__(32, by_four_taps(LAYOUT) ? 8 : 12) ckpt_small_kernel(const AdjArgs A) {
  const int lane = threadIdx.x;
  const int64_t slot = (int64_t)blockIdx.x * 8 + (lane >> 2);
  if (slot >= A.count) return;
  __shared__ float guard_m[32][2];
  ckpt_one<MAPS>(FourLanes<LAYOUT>{lane & 3, lane & ~3}, A, slot, (lane & 3) == 0, guard_m[lane]);
}

// The marked rays' checkpoints by the four-tap passes. Few rays: the launch is about
// one ray's latency.
template <bool TAPE>
__global__ void __launch_bounds__(128, 2) near_ckpt_kernel(const AdjArgs A) {
  for_near_rays(A, gridDim.x, gridDim.x, [&](int64_t slot, bool together) {
    MixedRay R;
    float y[kMixedState];
    Guard gd;  // disabled
    ckpt_ray<TAPE>(OneLane<kFourTaps>(), A, slot, ray_dir_pix(A.nside, ring_of(A, slot)), R, y, gd, true, together);
  });
}

// Cotangent of the final state from the map weights (the transpose of
// extract_mixed) -> lam [19][count].
__global__ void __launch_bounds__(128) final_cotangent_kernel_mixed(const AdjArgs A, float* lam) {
  const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= A.count) return;
  const int64_t ring = ring_of(A, slot);
  const int64_t o = ring - A.pix_begin;
  const RayDir d = ray_dir_pix(A.nside, ring);
  MixedRay R;
  float y[kMixedState];
  init_mixed(d, R, y);
  load_vec((const float*)A.ckpt + (int64_t)A.nseg * kMixedState * A.count, A.count, slot, y, kMixedState);
  float l[19];
  for (int j = 0; j < 19; ++j) l[j] = 0.f;
  float w[6];
  for (int m = 0; m < 6; ++m) w[m] = A.w[m][o];
  l[12] = w[0];
  l[16] = w[1];
  l[17] = w[2];
  l[18] = w[3];
  const float S = (float)A.n_steps;
  float u[3];
  for (int i = 0; i < 3; ++i) u[i] = (y[i] + y[19 + i]) / S;
  const float q = R.eta[0] - 2.f * (R.n0[0] * u[0] + R.n0[1] * u[1] + R.n0[2] * u[2]) +
                  (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
  const float c = rsqrt1p_m1(q);
  const float r3 = (1.f + c) * (1.f + c) * (1.f + c);  // (1 + q)^(-3/2)
  float Db[3], um[3];
  for (int i = 0; i < 3; ++i) {
    Db[i] = w[4] * R.a0[i] + w[5] * R.b0[i];
    um[i] = u[i] - R.n0[i];
  }
  const float dotv = um[0] * Db[0] + um[1] * Db[1] + um[2] * Db[2];
  for (int i = 0; i < 3; ++i) l[i] = ((1.f + c) * Db[i] - dotv * r3 * um[i]) / S;
  store_vec(lam, A.count, slot, l, 19);
}

// Recompute segment sgi of one ray from its checkpoint, storing the four stage
// inputs of every step: tape [C][4 x 19][count].
template <typename Interp>
__device__ __forceinline__ void segment_ray(const Interp& interp, const AdjArgs& A, int sgi, int64_t slot,
                                            bool first = true, bool together = false) {
  MixedRay R;
  float y[kMixedState], x0[3];
  mixed_observer(A.G, x0);
  load_bases(A, slot, R);
  const int s0 = sgi * A.C, s1 = min(s0 + A.C, A.n_steps);
  load_vec((const float*)A.ckpt + (int64_t)sgi * kMixedState * A.count, A.count, slot, y, kMixedState);
  float* tape = (float*)A.seg;
#pragma unroll 1
  for (int st = s0; st < s1; ++st) {
    Guard gd;  // disabled
    if (std::is_same<Interp, OneLane<kFourTaps>>::value && together) prefetch_step(A, R, x0, y, st);
    step_mixed(interp, R, A.F, A.G, x0, st, y,
               first ? tape + (int64_t)(st - s0) * kTapeStep * A.count + slot : nullptr, A.count, gd);
  }
}

// The first near_blocks blocks (one per SM) take the marked rays by the four-tap
// passes: first, so that their latency hides behind the other rays', and a short list
// in a quarter of them (with its warps in all of them the segment is 1-2 % longer).
template <int LAYOUT>
__global__ void __launch_bounds__(128, 2) segment_kernel_mixed(const AdjArgs A, int sgi, unsigned near_blocks) {
  if (blockIdx.x < near_blocks) {
    for_near_rays(A, near_blocks, (near_blocks + 3) / 4, [&](int64_t slot, bool together) {
      segment_ray(OneLane<kFourTaps>(), A, sgi, slot, true, together);
    });
    return;
  }
  const int64_t slot = (int64_t)(blockIdx.x - near_blocks) * 128 + threadIdx.x;
  if (slot < A.count && !is_near(A, slot)) segment_ray(OneLane<LAYOUT>(), A, sgi, slot);
}

// Marked rays by their four lanes too: the other groups of the warp wait for them (a
// launch of their own, 12 us a step after this one, was 3 us even with none marked).
template <int LAYOUT>
__global__ void __launch_bounds__(32, by_four_taps(LAYOUT) ? 8 : 12) segment_small_kernel(const AdjArgs A, int sgi) {
  constexpr bool kFour = by_four_taps(LAYOUT);  // all rays are traced so
  const int lane = threadIdx.x;
  const int64_t slot = (int64_t)blockIdx.x * 8 + (lane >> 2);
  if (slot >= A.count) return;
  if (kFour || !is_near(A, slot))
    segment_ray(FourLanes<LAYOUT>{lane & 3, lane & ~3}, A, sgi, slot, (lane & 3) == 0);
  else
    segment_ray(FourLanes<kFour ? LAYOUT : kFourTaps>{lane & 3, lane & ~3}, A, sgi, slot, (lane & 3) == 0);
}

// The four passes of a stage by one lane, FP32 accumulation: the interpolations,
// and every second stage one scatter for two. In the backward order the stages come
// in pairs (the midpoint stages of a step; a step's first stage and the last one of
// the step before) whose positions differ by ~1e-4 cells or less, so their 16 cells
// per field are the same unless a face lies between them, and adding their tap
// cotangents before they go to memory halves the atomics, whose way to L2 the sweep
// waited for with both gradients (61 % of its cycles). 256^3 / nside 128 / 128 steps:
// 46.9 -> 41.6 ms; 512^3 / nside 256 / 256 steps: 359.7 -> 317 ms, phi only (the
// backward half) 181 -> 171. The interpolations, with no scatter in them, are best
// unrolled (rolled: 47.7 and 361 ms), the scatter in a loop over its slices
// (unrolled: 43.4 and 329 ms, the code outgrows the instruction cache).
template <int LAYOUT, bool BGRAD>
struct DeferredPasses {
  // a pending stage per thread: 10 cotangents per field, the offsets on the centred
  // (and staggered) axes, the fields' cells (base, hot_base)
  static constexpr int kFields = BGRAD ? 4 : 1, kQ = 0, kT = 10 * kFields, kBase = kT + (BGRAD ? 6 : 3),
                       kHot = kBase + 2 * kFields, kWords = kHot + kFields;
  const FieldPtrs& F;
  const Geom& G;
  AccF32 acc[4];
  float (*pend)[128];
  bool second = false, pending = false;

  __device__ float& word(int w) const { return pend[w][threadIdx.x]; }
  template <int f>
  __device__ void load_pending(float* t, float* q, int64_t* base, int* hbase) const {
    constexpr int k = BGRAD ? f : 0;
    for (int i = 0; i < 10; ++i) q[i] = word(kQ + 10 * k + i);
    for (int i = 0; i < 3; ++i) t[i] = word(kT + i + (i == f ? 3 : 0));
    *base = (int64_t)(((unsigned long long)__float_as_uint(word(kBase + 2 * k + 1)) << 32) |
                      __float_as_uint(word(kBase + 2 * k)));
    *hbase = __float_as_int(word(kHot + k));
  }
  template <int f>
  __device__ void deposit(const StageView<float>& V, const float* qb) const {
    constexpr int k = BGRAD ? f : 0;
    if (BGRAD && f == 3 && !second)  // phi's axes serve the B components too
      for (int i = 0; i < 3; ++i) word(kT + i) = V.t[3][i];
    if (!acc[f].active()) return;
    if (!second) {
      for (int i = 0; i < 10; ++i) word(kQ + 10 * k + i) = qb[i];
      if (f != 3)
        word(kT + 3 + f) = V.t[f][f];
      else if (!BGRAD)
        for (int i = 0; i < 3; ++i) word(kT + i) = V.t[3][i];
      word(kBase + 2 * k) = __uint_as_float((unsigned)V.base[f]);
      word(kBase + 2 * k + 1) = __uint_as_float((unsigned)((unsigned long long)V.base[f] >> 32));
      word(kHot + k) = __int_as_float(V.hbase[f]);
      return;
    }
    float ta[3], tb[3], qa[10], q[10];
    int64_t base = V.base[f], base_a = base;
    int hbase = V.hbase[f], hbase_a = hbase;
    for (int i = 0; i < 10; ++i) q[i] = qb[i];
    for (int i = 0; i < 3; ++i) tb[i] = ta[i] = V.t[f][i];
    if (pending)
      load_pending<f>(ta, qa, &base_a, &hbase_a);
    else
      for (int i = 0; i < 10; ++i) qa[i] = 0.f;
    // the pending stage with this one where their cells agree, else (rarely) in a
    // round of its own
    bool same = base_a == base;
    float qs[10];
    for (int i = 0; i < 10; ++i) qs[i] = same ? qa[i] : 0.f;
#pragma unroll 1
    for (;;) {
      scatter_two(acc[f], base, hbase, G, ta, qs, tb, q);
      if (!__any_sync(0xffffffffu, !same)) break;
      for (int i = 0; i < 10; ++i) {
        q[i] = 0.f;
        qs[i] = same ? 0.f : qa[i];
      }
      base = base_a;
      hbase = hbase_a;
      same = true;
    }
  }
  // The last pending stage of a segment.
  template <int f>
  __device__ void flush_field() const {
    if (!acc[f].active()) return;
    float t[3], q[10], none[10];
    int64_t base;
    int hbase;
    load_pending<f>(t, q, &base, &hbase);
    for (int i = 0; i < 10; ++i) none[i] = 0.f;
    scatter_two(acc[f], base, hbase, G, t, q, t, none);
  }
  __device__ void flush() const {
    if constexpr (BGRAD) {
      flush_field<0>();
      flush_field<1>();
      flush_field<2>();
    }
    flush_field<3>();
  }
  template <int C>
  __device__ void component(const StageView<float>& V, const float* fb, BVjp<float>& B, float* nb, float* xb) const {
    float qb[10];
    b_cotangent<C>(V, fb, B, qb);
    Tri<float> Q;
    field_pass<LAYOUT, 4, float, AccNone>(F, C, V, G, qb, Q, xb, AccNone());
    if constexpr (BGRAD) deposit<C>(V, qb);
    b_fold<C>(V, Q, B, nb);
  }
  __device__ void operator()(const StageView<float>& V, const float* fb, const PhiVjp<float>& p, BVjp<float>& B,
                             float* nb, float* xb, Tri<float>& P) const {
    component<0>(V, fb, B, nb, xb);
    component<1>(V, fb, B, nb, xb);
    component<2>(V, fb, B, nb, xb);
    float qb[10];
    phi_cotangent(V, p, qb);
    field_pass<LAYOUT, 4, float, AccNone>(F, 3, V, G, qb, P, xb, AccNone());
    deposit<3>(V, qb);
  }
};
template <typename P>
struct IsDeferred : std::false_type {};
template <int LAYOUT, bool BGRAD>
struct IsDeferred<DeferredPasses<LAYOUT, BGRAD>> : std::true_type {};

// Backward sweep over segment sgi: per step, backwards, the RK4 adjoint
//   a4 = J(u4)^T l/6, a3 = J(u3)^T (l/3 + a4), a2 = J(u2)^T (l/3 + a3/2),
//   a1 = J(u1)^T (l/6 + a2/2), l <- l + a1 + a2 + a3 + a4,
// with the stage inputs u from the tape (the next stage's inputs are loaded
// while the current stage runs); l carried in lam between segments. l and the
// running sum of the a's live in shared memory (one column per thread) to keep
// registers for the field passes.
// live: this lane's ray counts; store: it writes the cotangent back.
template <int THREADS, typename Passes>
__device__ __forceinline__ void sweep_segment(const AdjArgs& A, int sgi, int64_t slot, bool live, bool store,
                                              const MixedRay& R, const float* x0, float* lam, Passes passes,
                                              float (*s_lam)[THREADS], float (*s_tot)[THREADS]) {
  const int t = threadIdx.x;
  for (int j = 0; j < 19; ++j) s_lam[j][t] = live ? lam[(int64_t)j * A.count + slot] : 0.f;
  const float* tape = (const float*)A.seg + slot;
  const int s0 = sgi * A.C, s1 = min(s0 + A.C, A.n_steps);
  // flattened (step, stage) index, descending; u holds the stage inputs of q
  int q = (s1 - s0) * 4 - 1;
  float u[19];
  for (int j = 0; j < 19; ++j) u[j] = ld_stream(tape + ((int64_t)(q >> 2) * kTapeStep + 19 * (q & 3) + j) * A.count);
  float an[19];  // a of the stage after this one (finite; its weight is 0 at stage 3)
  for (int j = 0; j < 19; ++j) an[j] = 0.f;
#pragma unroll 1
  for (; q >= 0; --q) {
    const int st = s0 + (q >> 2), stage = q & 3;
    const float c = (stage == 0) ? 0.f : ((stage == 3) ? 1.f : 0.5f);
    const float wl = (stage == 0 || stage == 3) ? (1.f / 6.f) : (1.f / 3.f);
    const float wa = (stage == 3) ? 0.f : ((stage == 2) ? 1.f : 0.5f);
    float fb[19];
    for (int j = 0; j < 19; ++j) fb[j] = wl * s_lam[j][t] + wa * an[j];
    StageView<float> V;
    stage_view_mixed(u, (float)st + c, R, A.G, x0, V);
    {  // prefetch the next (earlier) stage's inputs (the last stage reloads its own)
      const int qn = q > 0 ? q - 1 : 0;
      for (int j = 0; j < 19; ++j) u[j] = ld_stream(tape + ((int64_t)(qn >> 2) * kTapeStep + 19 * (qn & 3) + j) * A.count);
    }
    for (int j = 0; j < 19; ++j) an[j] = 0.f;
    if constexpr (IsDeferred<Passes>::value) passes.second = (q & 1) != 0;
    rhs_vjp_with(V, fb, an, passes);
    if constexpr (IsDeferred<Passes>::value) passes.pending = (q & 1) == 0;
    // the step's running sum of the a's restarts at its last stage
    for (int j = 0; j < 19; ++j) s_tot[j][t] = (stage == 3 ? 0.f : s_tot[j][t]) + an[j];
    if (stage == 0)
      for (int j = 0; j < 19; ++j) s_lam[j][t] += s_tot[j][t];
  }
  if constexpr (IsDeferred<Passes>::value) passes.flush();
  if (store)
    for (int j = 0; j < 19; ++j) lam[(int64_t)j * A.count + slot] = s_lam[j][t];
}

// Resident blocks of 128 threads per SM the sweep is compiled for (register
// budget 65536 / (128 * blocks)).
#ifndef SRT_SWEEP_MIN_BLOCKS
#define SRT_SWEEP_MIN_BLOCKS 2
#endif

// BGRAD: the B gradient is wanted (else the B passes are compiled without a
// scatter).
template <typename Acc, int LAYOUT, bool BGRAD>
__global__ void __launch_bounds__(128, SRT_SWEEP_MIN_BLOCKS)
    sweep_kernel_mixed(const AdjArgs A, int sgi, float* lam, Acc a0, Acc a1, Acc a2, Acc a3) {
  __shared__ float s_lam[19][128];
  __shared__ float s_tot[19][128];
  int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // the warp's lanes stay together for the paired atomics: one past the last ray
  // follows it with a zero cotangent and stores nothing
  const bool live = slot < A.count;
  if (!__any_sync(0xffffffffu, live)) return;
  if constexpr (TakesCells<Acc>::value) {
    // this warp's copy of the region around the observer
    const int64_t copy = ((slot >> 5) % kHotCopies) * (kHotSide * kHotSide * kHotSide);
    for (Acc* a : {&a0, &a1, &a2, &a3})
      if (a->hot) a->hot += copy;
  } else if (!live) {
    return;
  }
  if (!live) slot = A.count - 1;
  typedef typename std::conditional<BGRAD, Acc, AccNone>::type AccB;
  AccB accb[3];
  if constexpr (BGRAD) {
    accb[0] = a0;
    accb[1] = a1;
    accb[2] = a2;
  }
  MixedRay R;
  float x0[3];
  load_bases(A, slot, R);
  mixed_observer(A.G, x0);
  if constexpr (TakesCells<Acc>::value) {
    typedef DeferredPasses<LAYOUT, BGRAD> Passes;
    __shared__ float pend[Passes::kWords][128];
    sweep_segment<128>(A, sgi, slot, live, live, R, x0, lam, Passes{A.F, A.G, {a0, a1, a2, a3}, pend}, s_lam, s_tot);
    return;
  }
  sweep_segment<128>(A, sgi, slot, live, live, R, x0, lam, OneLanePasses<LAYOUT, float, AccB, Acc>{A.F, A.G, accb, a3},
                     s_lam, s_tot);
}

// The four passes of a stage by four lanes that hold the same ray, one field
// each; every lane then folds them.
template <int LAYOUT, typename Acc>
struct FourLanePasses {
  const FieldPtrs& F;
  const Geom& G;
  const Acc& acc;  // this lane's field's
  int field, first;
  __device__ void operator()(const StageView<float>& V, const float* fb, const PhiVjp<float>& p, BVjp<float>& B,
                             float* nb, float* xb, Tri<float>& P) const {
    float qb[10], q[10];
    phi_cotangent(V, p, qb);
    b_cotangent<0>(V, fb, B, q);
    for (int i = 0; i < 10; ++i) qb[i] = field == 0 ? q[i] : qb[i];
    b_cotangent<1>(V, fb, B, q);
    for (int i = 0; i < 10; ++i) qb[i] = field == 1 ? q[i] : qb[i];
    b_cotangent<2>(V, fb, B, q);
    for (int i = 0; i < 10; ++i) qb[i] = field == 2 ? q[i] : qb[i];
    StageView<float> W;  // this lane's field's cell in the place of all (selects, no indexed arrays)
    W.base[0] = field == 0 ? V.base[0] : (field == 1 ? V.base[1] : (field == 2 ? V.base[2] : V.base[3]));
    W.basep[0] = field == 0 ? V.basep[0] : (field == 1 ? V.basep[1] : (field == 2 ? V.basep[2] : V.basep[3]));
    W.hbase[0] = field == 0 ? V.hbase[0] : (field == 1 ? V.hbase[1] : (field == 2 ? V.hbase[2] : V.hbase[3]));
    for (int i = 0; i < 3; ++i)
      W.t[0][i] = field == 0 ? V.t[0][i] : (field == 1 ? V.t[1][i] : (field == 2 ? V.t[2][i] : V.t[3][i]));
    Tri<float> own;
    float x[3] = {0.f, 0.f, 0.f};
    tricubic_vjp_mixed<1, Acc>(cell_source<LAYOUT>(F, G, field, W.base[0], W.basep[0]), W.base[0], W.hbase[0], G, W.t[0],
                               qb, own, x, acc);
    const unsigned mask = 0xfu << first;
    for (int i = 0; i < 3; ++i) {
      float v = __shfl_sync(mask, x[i], first);
      for (int f = 1; f < 4; ++f) v += __shfl_sync(mask, x[i], first + f);
      xb[i] += v;
    }
    Tri<float> Q;
    fetch_tri(own, 0, first, Q);
    b_fold<0>(V, Q, B, nb);
    fetch_tri(own, 1, first, Q);
    b_fold<1>(V, Q, B, nb);
    fetch_tri(own, 2, first, Q);
    b_fold<2>(V, Q, B, nb);
    fetch_tri(own, 3, first, P);
  }
};

// The sweep of a small range: four lanes per ray, one-warp blocks.
template <typename Acc, int LAYOUT>
__global__ void __launch_bounds__(32, 8)
    sweep_small_kernel(const AdjArgs A, int sgi, float* lam, Acc a0, Acc a1, Acc a2, Acc a3) {
  __shared__ float s_lam[19][32];
  __shared__ float s_tot[19][32];
  const int lane = threadIdx.x, field = lane & 3;
  int64_t slot = (int64_t)blockIdx.x * 8 + (lane >> 2);
  const bool live = slot < A.count;  // lanes past the last ray follow it with a zero cotangent
  if (!live) slot = A.count - 1;
  Acc acc = field == 0 ? a0 : (field == 1 ? a1 : (field == 2 ? a2 : a3));
  if constexpr (TakesCells<Acc>::value) {
    if (acc.hot) acc.hot += (blockIdx.x % kHotCopies) * (kHotSide * kHotSide * kHotSide);
    acc.mask = __ballot_sync(0xffffffffu, acc.active());
  }
  MixedRay R;
  float x0[3];
  load_bases(A, slot, R);
  mixed_observer(A.G, x0);
  sweep_segment<32>(A, sgi, slot, live, live && field == 0, R, x0, lam,
                    FourLanePasses<LAYOUT, Acc>{A.F, A.G, acc, field, lane & ~3}, s_lam, s_tot);
}

// fn(std::integral_constant<int, LAYOUT>()) for the passes of a handle's forward:
// second differences or four taps.
template <typename Fn>
void with_forward_layout(const srt_fields* f, const Fn& fn) {
  const int layout = f->layout();
  if (layout == kCells)
    fn(std::integral_constant<int, kCells>());
  else if (layout == kHalf)
    fn(std::integral_constant<int, kHalf>());
  else if (layout == kPairs)
    fn(std::integral_constant<int, kFourPairs>());
  else if (f->four_taps)
    fn(std::integral_constant<int, kFourPlanes>());
  else
    fn(std::integral_constant<int, kPlanes>());
}

// The same for the sweep, which interpolates at positions it is given and takes the
// second differences in every layout.
template <typename Fn>
void with_sweep_layout(const srt_fields* f, const Fn& fn) {
  const int layout = f->layout();
  if (layout == kCells)
    fn(std::integral_constant<int, kCells>());
  else if (layout == kHalf)
    fn(std::integral_constant<int, kHalf>());
  else if (layout == kPairs)
    fn(std::integral_constant<int, kPairs>());
  else
    fn(std::integral_constant<int, kPlanes>());
}

// Blocks of the launches for the marked rays alone: all that are resident at once, and
// no more than give each ray a warp.
inline unsigned near_ckpt_blocks(unsigned blocks, int sms) { return std::min<unsigned>(blocks * 32, 2 * sms); }

template <int LAYOUT, bool MAPS>
void launch_ckpt(const AdjArgs& A, bool small, unsigned blocks, cudaStream_t s) {
  if (small)
    ckpt_small_kernel<LAYOUT, MAPS><<<(unsigned)((A.count + 7) / 8), 32, 0, s>>>(A);
  else
    ckpt_kernel_mixed<LAYOUT, MAPS><<<blocks, 128, 0, s>>>(A);
}
template <int LAYOUT>
void launch_segment(const AdjArgs& A, int sgi, bool small, unsigned blocks, unsigned near, cudaStream_t s) {
  if (small)
    segment_small_kernel<LAYOUT><<<(unsigned)((A.count + 7) / 8), 32, 0, s>>>(A, sgi);
  else
    segment_kernel_mixed<LAYOUT><<<blocks + near, 128, 0, s>>>(A, sgi, near);
}

inline void copy_extra(AccPaired<4>& to, const AccF32& from) { to.hot = from.hot; }
inline void copy_extra(AccFixed& to, const AccFixed& from) { to.ovf = from.ovf; }

template <typename Acc>
void launch_sweep(const AdjArgs& A, int sgi, float* lam, const Acc* a, const srt_fields* f, bool bgrad, bool small,
                  unsigned blocks, cudaStream_t s) {
  with_sweep_layout(f, [&](auto l) {
    constexpr int L = decltype(l)::value;
    if (small) {
      typedef typename std::conditional<TakesCells<Acc>::value, AccPaired<4>, Acc>::type AccS;
      AccS b[4];
      for (int f = 0; f < 4; ++f) {
        b[f].g = a[f].g;
        copy_extra(b[f], a[f]);
      }
      sweep_small_kernel<AccS, L><<<(unsigned)((A.count + 7) / 8), 32, 0, s>>>(A, sgi, lam, b[0], b[1], b[2], b[3]);
      return;
    }
    if (bgrad)
      sweep_kernel_mixed<Acc, L, true><<<blocks, 128, 0, s>>>(A, sgi, lam, a[0], a[1], a[2], a[3]);
    else
      sweep_kernel_mixed<Acc, L, false><<<blocks, 128, 0, s>>>(A, sgi, lam, a[0], a[1], a[2], a[3]);
  });
}

// ------------------------------------------------------------- FP64 mode

__global__ void __launch_bounds__(128) ckpt_kernel_fp64(const AdjArgs A) {
  const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= A.count) return;
  const RayDir d = ray_dir_pix(A.nside, ring_of(A, slot));
  double y[19];
  init_std(d, A.G, y);
  double* ck = (double*)A.ckpt;
  store_vec(ck, A.count, slot, y, 19);
#pragma unroll 1
  for (int st = 0; st < A.n_steps; ++st) {
    step_std<kFP64>(A.F, A.G, y, nullptr);
    const int done = st + 1;
    if (done % A.C == 0 || done == A.n_steps) {
      const int k = (done + A.C - 1) / A.C;
      store_vec(ck + (int64_t)k * 19 * A.count, A.count, slot, y, 19);
    }
  }
}

template <typename Acc>
__global__ void __launch_bounds__(128) reverse_kernel_fp64(const AdjArgs A, const Acc a0, const Acc a1,
                                                          const Acc a2, const Acc a3) {
  const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= A.count) return;
  const Acc acc[4] = {a0, a1, a2, a3};
  const int64_t ring = ring_of(A, slot);
  const int64_t o = ring - A.pix_begin;
  const RayDir d = ray_dir_pix(A.nside, ring);
  const double* ck = (const double*)A.ckpt;
  double* sg = (double*)A.seg;
  constexpr int kSeg = 19 + 57;
  double y[19], lam[19];
  {
    load_vec(ck + (int64_t)A.nseg * 19 * A.count, A.count, slot, y, 19);
    for (int j = 0; j < 19; ++j) lam[j] = 0.0;
    double w[6];
    for (int m = 0; m < 6; ++m) w[m] = A.w[m][o];
    lam[12] = w[0];
    lam[16] = w[1];
    lam[17] = w[2];
    lam[18] = w[3];
    // deflection = (X/|X| - r_hat) . (e_theta, e2): Xb = (I - X^ X^T) Db / |X|
    double X[3];
    for (int i = 0; i < 3; ++i) X[i] = y[i] - (double)A.G.n[i] * 0.5;
    const double nrm = sqrt(X[0] * X[0] + X[1] * X[1] + X[2] * X[2]);
    const double Db[3] = {w[4] * d.ct * d.cp + w[5] * d.sp, w[4] * d.ct * d.sp - w[5] * d.cp, -w[4] * d.st};
    const double xd = (X[0] * Db[0] + X[1] * Db[1] + X[2] * Db[2]) / nrm;
    for (int i = 0; i < 3; ++i) lam[i] = (Db[i] - X[i] / nrm * xd) / nrm;
  }
#pragma unroll 1
  for (int sgi = A.nseg - 1; sgi >= 0; --sgi) {
    const int s0 = sgi * A.C, s1 = min(s0 + A.C, A.n_steps);
    load_vec(ck + (int64_t)sgi * 19 * A.count, A.count, slot, y, 19);
#pragma unroll 1
    for (int st = s0; st < s1; ++st) {
      double* rec = sg + (int64_t)(st - s0) * kSeg * A.count;
      store_vec(rec, A.count, slot, y, 19);
      double ks[57];
      step_std<kFP64>(A.F, A.G, y, ks);
      store_vec(rec + (int64_t)19 * A.count, A.count, slot, ks, 57);
    }
#pragma unroll 1
    for (int st = s1 - 1; st >= s0; --st) {
      const double* rec = sg + (int64_t)(st - s0) * kSeg * A.count;
      double yi[19], anext[19], atot[19];
      load_vec(rec, A.count, slot, yi, 19);
      for (int j = 0; j < 19; ++j) atot[j] = 0.0;
#pragma unroll 1
      for (int stage = 3; stage >= 0; --stage) {
        double u[19], fb[19];
        const double c = (stage == 0) ? 0.0 : ((stage == 3) ? 1.0 : 0.5);
        if (stage == 0) {
          for (int j = 0; j < 19; ++j) u[j] = yi[j];
        } else {
          double kprev[19];
          load_vec(rec + (int64_t)(19 + 19 * (stage - 1)) * A.count, A.count, slot, kprev, 19);
          for (int j = 0; j < 19; ++j) u[j] = yi[j] + c * kprev[j];
        }
        const double wl = (stage == 0 || stage == 3) ? (1.0 / 6.0) : (1.0 / 3.0);
        const double wa = (stage == 3) ? 0.0 : ((stage == 2) ? 1.0 : 0.5);
        for (int j = 0; j < 19; ++j) fb[j] = wl * lam[j] + (stage == 3 ? 0.0 : wa * anext[j]);
        StageView<double> V;
        stage_view_fp64(u, A.G, V);
        double ub[19];
        for (int j = 0; j < 19; ++j) ub[j] = 0.0;
        rhs_vjp<double, Acc, Acc>(V, A.F, A.G, fb, ub, acc, acc[3]);
        for (int j = 0; j < 19; ++j) {
          anext[j] = ub[j];
          atot[j] += ub[j];
        }
      }
      for (int j = 0; j < 19; ++j) lam[j] += atot[j];
    }
  }
}

// ------------------------------------------------------------------ fold

// Value of padded index q of an accumulator grid.
template <typename G>
struct PadRead;
template <>
struct PadRead<double> {  // FP64 atomics: one entry per padded voxel
  typedef double T;
  const double* g;
  __device__ T operator()(int64_t q) const { return g[q]; }
  __device__ static double value(T s) { return s; }
};
template <>
struct PadRead<unsigned long long> {  // fixed point: exact integer sums
  typedef unsigned long long T;
  const unsigned long long* g;
  __device__ T operator()(int64_t q) const { return g[q]; }
  __device__ static double value(T s) { return (double)(long long)s / kFixedScale; }
};

// Value of padded position (i, j, k) of an accumulator grid; for cells, the
// transpose of cell_of: the second differences gather their neighbours'
// cotangents (symmetric stencils; only positions 1 .. n + 1 hold any).
// INSIDE: the neighbours are known to lie in the grid.
template <bool INSIDE, typename G>
__device__ __forceinline__ typename PadRead<G>::T pad_value(const PadRead<G>& rd, int64_t i, int64_t j, int64_t k,
                                                            int64_t p0, int64_t p1) {
  return rd(i + p0 * (j + p1 * k));
}
template <>
struct PadRead<float4> {
  typedef float T;
  const float4* g;
  __device__ static double value(T s) { return (double)s; }
};
template <bool INSIDE>
__device__ __forceinline__ float pad_value(const PadRead<float4>& rd, int64_t i, int64_t j, int64_t k, int64_t p0,
                                           int64_t p1) {
  float s = 0.f;
  const float4* at = rd.g + i + p0 * (j + p1 * k);
#pragma unroll
  for (int b = -1; b <= 1; ++b)
#pragma unroll
    for (int a = -1; a <= 1; ++a) {
      if (!INSIDE && (i + a < 0 || i + a >= p0 || j + b < 0 || j + b >= p1)) continue;
      const float4 c = __ldg(at + a + p0 * b);
      const float wx = a == 0 ? -2.f : 1.f, wy = b == 0 ? -2.f : 1.f;
      float v = wx * wy * c.w;
      if (a == 0) v += wy * c.y;
      if (b == 0) v += wx * c.z;
      if (a == 0 && b == 0) v += c.x;
      s += v;
    }
  return s;
}

// Adds the copies of the region around the observer (behind the grid's pvox
// entries) into the grid.
__global__ void __launch_bounds__(256) merge_hot_kernel(float4* g, int64_t pvox, const Geom G) {
  constexpr int kRegion = kHotSide * kHotSide * kHotSide;
  const int q = blockIdx.x * 256 + threadIdx.x;
  const int x = q % kHotSide + G.n[0] / 2 - kHotSide / 2, y = q / kHotSide % kHotSide + G.n[1] / 2 - kHotSide / 2,
            z = q / (kHotSide * kHotSide) + G.n[2] / 2 - kHotSide / 2;
  float4* dst = g + x + G.px * y + G.pxy * z;
  float4 s = *dst;
  for (int c = 0; c < kHotCopies; ++c) {
    const float4 v = g[pvox + (int64_t)c * kRegion + q];
    s.x += v.x;
    s.y += v.y;
    s.z += v.z;
    s.w += v.w;
  }
  *dst = s;
}

// For voxel (i, j, k): sum of the padded copies (the interior one and the
// halo copies) -> out[v * stride + comp] (+= when accumulate). Blocks of 32 x 8
// voxels of a plane (the cells' stencils share their neighbours in L1), looping
// where an axis is longer than the grid.
template <typename G>
__global__ void __launch_bounds__(256) fold_kernel(const G* __restrict__ padded, int64_t n0, int64_t n1, int64_t n2,
                                                   float* out, int stride, int comp, int accumulate, unsigned* ovf) {
  const int64_t i = (int64_t)blockIdx.x * 32 + threadIdx.x;
  if (i >= n0) return;
  const PadRead<G> rd{padded};
  const int64_t p0 = n0 + 3, p1 = n1 + 3;
  for (int64_t k = blockIdx.z; k < n2; k += gridDim.z) {
    for (int64_t j = (int64_t)blockIdx.y * 8 + threadIdx.y; j < n1; j += (int64_t)gridDim.y * 8) {
      typename PadRead<G>::T sum = 0;
      if (i > 1 && i < n0 - 1 && j > 1 && j < n1 - 1 && k > 1 && k < n2 - 1) {  // no halo copies
        sum = pad_value<true>(rd, i + 1, j + 1, k + 1, p0, p1);
      } else {
        int64_t pi[4], pj[4], pk[4];
        const int ni = padded_coords(i, n0, pi), nj = padded_coords(j, n1, pj), nk = padded_coords(k, n2, pk);
        for (int a = 0; a < nk; ++a)
          for (int b = 0; b < nj; ++b)
            for (int c = 0; c < ni; ++c) sum += pad_value<false>(rd, pi[c], pj[b], pk[a], p0, p1);
      }
      const double dval = PadRead<G>::value(sum);
      if (ovf && !(fabs(dval) < kFixedLimit)) atomicOr(ovf, 1u);  // fixed point near or past its range
      const float val = (float)dval;
      float* dst = out + (i + n0 * (j + n1 * k)) * stride + comp;
      *dst = accumulate ? *dst + val : val;
    }
  }
}

}  // namespace srt

using namespace srt;

namespace {

// Scratch, given back on the stream it was taken on: by release() before a call's
// last wait, with the handle's device current (a NULL stream is that device's).
struct DevBuf {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  ~DevBuf() { release(); }
  void release() {
    pool_free(p, s);
    p = nullptr;
  }
  cudaError_t alloc(size_t bytes, cudaStream_t stream) {
    s = stream;
    const cudaError_t e = scratch_alloc(&p, bytes, stream);
    if (e != cudaSuccess) p = nullptr;
    return e;
  }
};

template <typename Acc, typename E>
void make_acc(Acc* acc, void* const* bufs) {
  for (int f = 0; f < 4; ++f) acc[f].g = (E*)bufs[f];
}

}  // namespace

#define VJP_TRY(expr, what)          \
  do {                               \
    cudaError_t _e = (expr);         \
    if (_e != cudaSuccess) {         \
      rc = cuda_error(_e, what);     \
      goto done;                     \
    }                                \
  } while (0)

namespace {

// Morton-ordered list of the RING pixels in [pix_begin, pix_begin + pix_count)
// (the forward's launch order) -> rays.
int build_ray_list(int64_t nside, int64_t pix_begin, int64_t pix_count, cudaStream_t s, DevBuf& counts,
                   DevBuf& offsets, DevBuf& rays, int64_t* kernels) {
  int rc = SRT_OK;
  RangeArgs ra;
  ra.nside = nside;
  int l = 0;
  while ((int64_t(1) << l) < nside) ++l;
  ra.log2p = l;
  ra.launch_rays = 12 * (int64_t(1) << (2 * l));
  ra.pix_begin = pix_begin;
  ra.pix_count = pix_count;
  const int64_t nblk = (ra.launch_rays + kListBlock - 1) / kListBlock;
  VJP_TRY(counts.alloc(nblk * sizeof(int), s), "allocate ray counts");
  VJP_TRY(offsets.alloc(nblk * sizeof(int64_t), s), "allocate ray offsets");
  VJP_TRY(rays.alloc(pix_count * sizeof(int64_t), s), "allocate ray list");
  ray_count_kernel<<<(unsigned)nblk, kListBlock, 0, s>>>(ra, (int*)counts.p);
  ray_scan_kernel<<<1, 1024, 0, s>>>((const int*)counts.p, nblk, (int64_t*)offsets.p);
  ray_write_kernel<<<(unsigned)nblk, kListBlock, 0, s>>>(ra, (const int64_t*)offsets.p, (int64_t*)rays.p);
  *kernels += 3;
  VJP_TRY(cudaGetLastError(), "ray list kernels");
done:
  return rc;
}

}  // namespace

// Ranges the small kernels take: up to one of their warps per scheduler (128^3, 48
// steps, both gradients: 768 rays 3.22 -> 1.57 ms, 4,800 rays 2.82 -> 1.64, 12,288
// rays 3.41 against 4.18).
static bool small_adjoint(int64_t rays, int sms) { return rays <= (int64_t)sms * 4 * 8; }

// Segments whose tape srt_vjp's forward writes at once, the last ones, instead of
// a recompute (256^3 / nside 128 / 128 steps, C = 12: 5 of 11, 49.8 -> 46.9 ms): as many as
// 4 GiB hold; none where device memory is short (an eighth of what is free beside the
// outputs' staging), looked at above 256 MiB (where the query's microseconds no longer
// count). The caller goes back to one segment where the allocation fails.
static int kept_segments(int nseg, int64_t seg_bytes, int64_t out_bytes, int device) {
  const int64_t most = int64_t(4) << 30, few = int64_t(256) << 20;
  const int kept = (int)std::min<int64_t>(nseg, most / std::max<int64_t>(seg_bytes, 1));
  if (kept * seg_bytes > few) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess ||
        (int64_t)free_b + pool_reusable_bytes(device) < out_bytes + 8 * kept * seg_bytes)
      return 0;
  }
  return kept;
}

// Rays below which a gradient's scratch is not cut further.
constexpr int64_t kLeastPart = 4096;

// A forward trace's checkpoints (srt_forward_tape) for srt_vjp_tape.
struct srt_tape {
  const srt_fields* fields = nullptr;
  int device = 0;
  int64_t nside = 0, pix_begin = 0, pix_count = 0;
  int n_steps = 0, C = 0, nseg = 0;
  int64_t* rays = nullptr;  // Morton-ordered RING pixels (device), marked near a cell face
  int64_t* near = nullptr;  // their number and slots (device)
  float* bases = nullptr;   // [12][pix_count] (device)
  float* ckpt = nullptr;    // [nseg + 1][kMixedState][pix_count] (device)
  int64_t bytes = 0;
};

static int vjp_impl(const srt_fields* fields, int64_t nside, int64_t pix_begin, int64_t pix_count, int n_steps,
                    int precision, const float* const weights[SRT_NUM_MAPS], float* dphi, float* db_xyz,
                    int ckpt_every, unsigned flags, void* stream, srt_stats* stats, const srt_tape* tape);

extern "C" int srt_vjp(const srt_fields* fields, int64_t nside, int64_t pix_begin, int64_t pix_count, int n_steps,
                       int precision, const float* const weights[SRT_NUM_MAPS], float* dphi, float* db_xyz,
                       int ckpt_every, unsigned flags, void* stream, srt_stats* stats) {
  NvtxRange nvtx_("srt_vjp");
  return vjp_impl(fields, nside, pix_begin, pix_count, n_steps, precision, weights, dphi, db_xyz, ckpt_every, flags,
                  stream, stats, nullptr);
}

// srt_vjp; with a tape, the rays and checkpoints of srt_forward_tape replace
// the ray list and the checkpointing forward pass (MIXED only).
static int vjp_impl(const srt_fields* fields, int64_t nside, int64_t pix_begin, int64_t pix_count, int n_steps,
                    int precision, const float* const weights[SRT_NUM_MAPS], float* dphi, float* db_xyz,
                    int ckpt_every, unsigned flags, void* stream, srt_stats* stats, const srt_tape* tape) {
  const auto t_wall = std::chrono::steady_clock::now();
  if (!fields) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_vjp: fields is NULL");
  if (nside < 1 || nside > (int64_t(1) << 16))
    return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_vjp: invalid nside %lld", (long long)nside);
  const int64_t npix = 12 * nside * nside;
  if (pix_begin < 0 || pix_count < 0 || pix_begin > npix || pix_count > npix - pix_begin)
    return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_vjp: pixel range outside [0, %lld)", (long long)npix);
  if (n_steps < 1 || n_steps > (1 << 22)) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_vjp: invalid n_steps %d", n_steps);
  if (precision != SRT_PRECISION_FP64 && precision != SRT_PRECISION_MIXED)
    return set_error(precision == SRT_PRECISION_REF16 ? SRT_ERR_UNSUPPORTED : SRT_ERR_INVALID_ARGUMENT,
                     "srt_vjp: precision %d has no adjoint (use SRT_PRECISION_FP64 or SRT_PRECISION_MIXED)", precision);
  if (!weights) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_vjp: weights is NULL");
  for (int m = 0; m < 6; ++m)
    if (!weights[m] && pix_count > 0) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_vjp: weights[%d] is NULL", m);
  if (stats) memset(stats, 0, sizeof(*stats));
  const srt_fields* f = fields;
  const int64_t vox = f->n[0] * f->n[1] * f->n[2];
  const int64_t pvox = f->pn[0] * f->pn[1] * f->pn[2];
  const bool dev_io = (flags & SRT_OUTPUT_DEVICE) != 0;
  const bool accumulate = (flags & SRT_ACCUMULATE) != 0;
  const bool determ = (flags & SRT_DETERMINISTIC) != 0;
  const bool fp64 = precision == SRT_PRECISION_FP64;
  cudaStream_t s = (cudaStream_t)stream;
  int C = ckpt_every > 0 ? ckpt_every : (int)std::max(1.0, std::floor(std::sqrt((double)n_steps) + 0.5));
  if (C > n_steps) C = n_steps;
  if (tape) C = tape->C;
  const int nseg = (n_steps + C - 1) / C;
  int rc = SRT_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  if (prev != f->device) cudaSetDevice(f->device);
  DevBuf counts, offsets, rays, near, bases, wdev, ckpt, seg, lam, gacc[4], gout_phi, gout_b, ovf;
  const auto release = [&] {
    for (DevBuf* b : {&counts, &offsets, &rays, &near, &bases, &wdev, &ckpt, &seg, &lam, &gacc[0], &gacc[1], &gacc[2],
                      &gacc[3], &gout_phi, &gout_b, &ovf})
      b->release();
  };
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int64_t kernels = 0, h2d = 0, d2h = 0;
  {
    // padded accumulator entry: 8 B (FP64 / fixed point), 16 B (FP32: a cell's four cotangents)
    const size_t accsz = (determ || fp64) ? 8 : 16;
    if (!dev_io) {
      // host gradients: start from zero (or from the caller's values when accumulating)
      if (dphi) {
        VJP_TRY(gout_phi.alloc(vox * sizeof(float), s), "allocate dphi");
        if (accumulate) {
          VJP_TRY(cudaMemcpyAsync(gout_phi.p, dphi, vox * sizeof(float), cudaMemcpyHostToDevice, s), "copy dphi");
          h2d += vox * sizeof(float);
        }
      }
      if (db_xyz) {
        VJP_TRY(gout_b.alloc(3 * vox * sizeof(float), s), "allocate db");
        if (accumulate) {
          VJP_TRY(cudaMemcpyAsync(gout_b.p, db_xyz, 3 * vox * sizeof(float), cudaMemcpyHostToDevice, s), "copy db");
          h2d += 3 * vox * sizeof(float);
        }
      }
    }
    float* out_phi = dev_io ? dphi : (float*)gout_phi.p;
    float* out_b = dev_io ? db_xyz : (float*)gout_b.p;
    if (pix_count > 0 && (dphi || db_xyz)) {
      // ---- ray list (a tape brings its own)
      int64_t* ray_list = tape ? tape->rays : nullptr;
      if (!tape) {
        rc = build_ray_list(nside, pix_begin, pix_count, s, counts, offsets, rays, &kernels);
        if (rc != SRT_OK) goto done;
        ray_list = (int64_t*)rays.p;
      }

      // ---- weights on the device
      const float* wd[6];
      if (dev_io) {
        for (int m = 0; m < 6; ++m) wd[m] = weights[m];
      } else {
        VJP_TRY(wdev.alloc(6 * pix_count * sizeof(float), s), "allocate weights");
        for (int m = 0; m < 6; ++m) {
          VJP_TRY(cudaMemcpyAsync((float*)wdev.p + m * pix_count, weights[m], pix_count * sizeof(float),
                                  cudaMemcpyHostToDevice, s),
                  "copy weights");
          wd[m] = (const float*)wdev.p + m * pix_count;
        }
        h2d += 6 * pix_count * (int64_t)sizeof(float);
      }

      // ---- padded accumulators
      // copies of the region around the observer (FP32 accumulation), where the
      // grid holds the region
      const bool hot = !fp64 && !determ && std::min(f->n[0], std::min(f->n[1], f->n[2])) >= kHotSide;
      const int64_t acc_entries = pvox + (hot ? (int64_t)kHotCopies * kHotSide * kHotSide * kHotSide : 0);
      for (int fld = 0; fld < 4; ++fld) {
        const bool want = (fld == 3) ? (dphi != nullptr) : (db_xyz != nullptr);
        if (!want) continue;
        VJP_TRY(gacc[fld].alloc(acc_entries * accsz, s), "allocate gradient accumulators");
        VJP_TRY(cudaMemsetAsync(gacc[fld].p, 0, acc_entries * accsz, s), "clear accumulators");
      }
      if (determ) {  // fixed-point range flag
        VJP_TRY(ovf.alloc(sizeof(unsigned), s), "allocate overflow flag");
        VJP_TRY(cudaMemsetAsync(ovf.p, 0, sizeof(unsigned), s), "clear overflow flag");
      }

      // ---- the rays' scratch: checkpoints, the segments' records, cotangents; for
      // half the rays at a time, or a quarter, ..., where it finds no room for all
      const int state = fp64 ? 19 : kMixedState;
      const size_t esz = fp64 ? sizeof(double) : sizeof(float);
      int64_t part = pix_count, seg_bytes = 0;
      int kept = 0;
      for (;; part = (part + 1) / 2) {
        // per-step records of one segment: FP64 y, k1, k2, k3; MIXED the four stage inputs
        seg_bytes = (int64_t)C * (fp64 ? state + 57 : kTapeStep) * part * (int64_t)esz;
        kept = fp64 || tape ? 0 : kept_segments(nseg, seg_bytes, 32 * pvox, f->device);
        cudaError_t e = cudaSuccess;
        const char* what = "";
        const auto take = [&](DevBuf& b, size_t bytes, const char* name) {
          if (e == cudaSuccess) e = b.alloc(bytes, s), what = name;
        };
        if (!tape) take(ckpt, (size_t)(nseg + 1) * state * part * esz, "allocate checkpoints");
        if (!tape && !fp64) {
          take(near, (part + 1) * sizeof(int64_t), "allocate near rays");
          take(bases, (size_t)12 * part * sizeof(float), "allocate ray bases");
        }
        if (!fp64) take(lam, (size_t)19 * part * sizeof(float), "allocate state cotangents");
        if (e == cudaSuccess) {
          e = seg.alloc(std::max(kept, 1) * seg_bytes, s);
          if (e == cudaErrorMemoryAllocation && kept > 1) {  // one segment's records always do
            kept = 1;
            e = seg.alloc(seg_bytes, s);
          }
          what = "allocate segment records";
        }
        if (e == cudaSuccess) break;
        if (e != cudaErrorMemoryAllocation || tape || part <= kLeastPart) VJP_TRY(e, what);
        for (DevBuf* b : {&ckpt, &near, &bases, &lam}) b->release();
      }

      AdjArgs A;
      A.F = make_ptrs(f);
      A.G = make_geom(f);
      A.nside = nside;
      A.pix_begin = pix_begin;
      A.near = tape ? tape->near : (int64_t*)near.p;
      A.bases = tape ? tape->bases : (float*)bases.p;
      A.n_steps = n_steps;
      A.C = C;
      A.nseg = nseg;
      for (int m = 0; m < 6; ++m) A.w[m] = wd[m];
      A.ckpt = tape ? (void*)tape->ckpt : ckpt.p;
      A.seg = seg.p;
      A.tape_from = (nseg - kept) * C;
      for (int fld = 0; fld < 4; ++fld) A.acc[fld] = gacc[fld].p;
      for (int m = 0; m < 6; ++m) A.maps[m] = nullptr;
      A.refine_list = nullptr;
      A.refine_count = nullptr;

      int sms = 0;
      VJP_TRY(sm_count(&sms), "device attributes");
      VJP_TRY(cudaEventCreate(&e0), "cudaEventCreate");
      VJP_TRY(cudaEventCreate(&e1), "cudaEventCreate");
      VJP_TRY(cudaEventRecord(e0, s), "cudaEventRecord");
      for (int64_t first = 0; first < pix_count; first += part) {
        A.rays = ray_list + first;
        A.count = std::min(part, pix_count - first);
        A.seg = seg.p;
        const unsigned blocks = (unsigned)((A.count + 127) / 128);
        if (fp64) {
          ckpt_kernel_fp64<<<blocks, 128, 0, s>>>(A);
          if (determ) {
            AccFixed ac[4];
            make_acc<AccFixed, unsigned long long>(ac, A.acc);
            for (int fld = 0; fld < 4; ++fld) ac[fld].ovf = (unsigned*)ovf.p;
            reverse_kernel_fp64<AccFixed><<<blocks, 128, 0, s>>>(A, ac[0], ac[1], ac[2], ac[3]);
          } else {
            AccF64 ac[4];
            make_acc<AccF64, double>(ac, A.acc);
            reverse_kernel_fp64<AccF64><<<blocks, 128, 0, s>>>(A, ac[0], ac[1], ac[2], ac[3]);
          }
          kernels += 2;
        } else {
          // forward with checkpoints; then per segment, backwards: recompute
          // the segment's tape, sweep it
          const bool small = small_adjoint(A.count, sms);
          if (!tape) {  // else the checkpoints come from srt_forward_tape
            VJP_TRY(cudaMemsetAsync(near.p, 0, sizeof(int64_t), s), "clear near rays");
            with_forward_layout(f, [&](auto l) { launch_ckpt<decltype(l)::value, false>(A, small, blocks, s); });
            near_ckpt_kernel<true><<<near_ckpt_blocks(blocks, sms), 128, 0, s>>>(A);
          }
          final_cotangent_kernel_mixed<<<blocks, 128, 0, s>>>(A, (float*)lam.p);
          kernels += tape ? 1 : 3;
          AccF32 af[4];
          AccFixed ax[4];
          make_acc<AccF32, float4>(af, A.acc);
          for (int fld = 0; fld < 4; ++fld) af[fld].hot = hot ? pvox : 0;
          make_acc<AccFixed, unsigned long long>(ax, A.acc);
          for (int fld = 0; fld < 4; ++fld) ax[fld].ovf = (unsigned*)ovf.p;
          const bool bgrad = db_xyz != nullptr;
          const int kept_from = nseg - kept;  // segments from here on are on the tape already
          for (int sgi = nseg - 1; sgi >= 0; --sgi) {
            A.seg = seg.p;
            if (sgi >= kept_from) A.seg = (float*)seg.p + (int64_t)(sgi - kept_from) * C * kTapeStep * A.count;
            if (sgi < kept_from)
              with_forward_layout(f, [&](auto l) { launch_segment<decltype(l)::value>(A, sgi, small, blocks, sms, s); });
            if (determ)
              launch_sweep<AccFixed>(A, sgi, (float*)lam.p, ax, f, bgrad, small, blocks, s);
            else
              launch_sweep<AccF32>(A, sgi, (float*)lam.p, af, f, bgrad, small, blocks, s);
            kernels += sgi < kept_from ? 2 : 1;
          }
        }
      }
      for (int fld = 0; fld < 4 && hot; ++fld) {
        if (!gacc[fld].p) continue;
        merge_hot_kernel<<<kHotSide * kHotSide * kHotSide / 256, 256, 0, s>>>((float4*)gacc[fld].p, pvox, A.G);
        ++kernels;
      }
      VJP_TRY(cudaGetLastError(), "adjoint kernels");
      // ---- fold onto the periodic grid
      const dim3 fgrid((unsigned)((f->n[0] + 31) / 32), (unsigned)std::min<int64_t>((f->n[1] + 7) / 8, 65535),
                       (unsigned)std::min<int64_t>(f->n[2], 65535));
      const dim3 fblock(32, 8);
      for (int fld = 0; fld < 4; ++fld) {
        if (!gacc[fld].p) continue;
        float* dst = (fld == 3) ? out_phi : out_b;
        const int stride = (fld == 3) ? 1 : 3, comp = (fld == 3) ? 0 : fld;
        const int accum = accumulate ? 1 : 0;
        if (determ)
          fold_kernel<unsigned long long><<<fgrid, fblock, 0, s>>>((const unsigned long long*)gacc[fld].p, f->n[0],
                                                                 f->n[1], f->n[2], dst, stride, comp, accum,
                                                                 (unsigned*)ovf.p);
        else if (fp64)
          fold_kernel<double><<<fgrid, fblock, 0, s>>>((const double*)gacc[fld].p, f->n[0], f->n[1], f->n[2], dst,
                                                     stride, comp, accum, nullptr);
        else
          fold_kernel<float4><<<fgrid, fblock, 0, s>>>((const float4*)gacc[fld].p, f->n[0], f->n[1], f->n[2], dst,
                                                     stride, comp, accum, nullptr);
        ++kernels;
      }
      VJP_TRY(cudaGetLastError(), "fold kernel");
      VJP_TRY(cudaEventRecord(e1, s), "cudaEventRecord");
    } else if (!accumulate) {
      if (out_phi) VJP_TRY(cudaMemsetAsync(out_phi, 0, vox * sizeof(float), s), "clear dphi");
      if (out_b) VJP_TRY(cudaMemsetAsync(out_b, 0, 3 * vox * sizeof(float), s), "clear db");
    }
    if (!dev_io) {
      if (dphi) {
        VJP_TRY(cudaMemcpyAsync(dphi, out_phi, vox * sizeof(float), cudaMemcpyDeviceToHost, s), "copy dphi back");
        d2h += vox * sizeof(float);
      }
      if (db_xyz) {
        VJP_TRY(cudaMemcpyAsync(db_xyz, out_b, 3 * vox * sizeof(float), cudaMemcpyDeviceToHost, s), "copy db back");
        d2h += 3 * vox * sizeof(float);
      }
    }
    unsigned flag = 0;
    if (ovf.p)
      VJP_TRY(cudaMemcpyAsync(&flag, ovf.p, sizeof(flag), cudaMemcpyDeviceToHost, s), "read overflow flag");
    release();
    VJP_TRY(cudaStreamSynchronize(s), "srt_vjp");
    if (flag) {
      rc = set_error(SRT_ERR_OVERFLOW,
                     "srt_vjp: SRT_DETERMINISTIC gradient beyond the fixed-point range (|gradient| >= 2^30 per "
                     "voxel, or not finite); the gradients are not valid (use the FP32/FP64 accumulation)");
      goto done;
    }
    if (stats) {
      float ms = -1.f;
      if (e0 && e1) cudaEventElapsedTime(&ms, e0, e1);
      stats->trace_ms = ms;
      stats->rays = pix_count;
      stats->ray_steps = pix_count * (int64_t)n_steps;
      stats->kernels = kernels;
      stats->h2d_bytes = h2d;
      stats->d2h_bytes = d2h;
    }
  }
done:
  release();
  if (rc != SRT_OK) cudaStreamSynchronize(s);  // copies from or to the caller's buffers may be under way
  scratch_settle(f->device, s);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (prev != f->device) cudaSetDevice(prev);
  if (stats)
    stats->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_wall).count();
  return rc;
}

// ------------------------------------------------------------------ tape

extern "C" int srt_forward_tape(const srt_fields* fields, int64_t nside, int64_t pix_begin, int64_t pix_count,
                                int n_steps, int ckpt_every, float* const maps[SRT_NUM_MAPS], unsigned flags,
                                void* stream, srt_stats* stats, srt_tape** out) {
  NvtxRange nvtx_("srt_forward_tape");
  const auto t_wall = std::chrono::steady_clock::now();
  if (!out) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_forward_tape: out is NULL");
  *out = nullptr;
  if (!fields) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_forward_tape: fields is NULL");
  if (nside < 1 || nside > (int64_t(1) << 16))
    return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_forward_tape: invalid nside %lld", (long long)nside);
  const int64_t npix = 12 * nside * nside;
  if (pix_begin < 0 || pix_count < 1 || pix_begin > npix || pix_count > npix - pix_begin)
    return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_forward_tape: pixel range outside [0, %lld) or empty",
                     (long long)npix);
  if (n_steps < 1 || n_steps > (1 << 22))
    return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_forward_tape: invalid n_steps %d", n_steps);
  if (!maps) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_forward_tape: maps is NULL");
  for (int m = 0; m < 6; ++m)
    if (!maps[m]) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_forward_tape: maps[%d] is NULL", m);
  if (stats) memset(stats, 0, sizeof(*stats));
  const srt_fields* f = fields;
  cudaStream_t s = (cudaStream_t)stream;
  const bool dev_out = (flags & SRT_OUTPUT_DEVICE) != 0;
  int C = ckpt_every > 0 ? ckpt_every : (int)std::max(1.0, std::floor(std::sqrt((double)n_steps) + 0.5));
  if (C > n_steps) C = n_steps;
  const int nseg = (n_steps + C - 1) / C;
  int rc = SRT_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  if (prev != f->device) cudaSetDevice(f->device);
  srt_tape* t = new (std::nothrow) srt_tape();
  DevBuf counts, offsets, rays, near, bases, ckpt, dmaps, rlist, rcount;
  const auto release = [&] {  // all but what the tape takes over
    for (DevBuf* b : {&counts, &offsets, &dmaps, &rlist, &rcount}) b->release();
  };
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int64_t kernels = 0;
  if (!t) {
    rc = set_error(SRT_ERR_OUT_OF_MEMORY, "srt_forward_tape: host allocation failed");
    goto done;
  }
  {
    rc = build_ray_list(nside, pix_begin, pix_count, s, counts, offsets, rays, &kernels);
    if (rc != SRT_OK) goto done;
    VJP_TRY(ckpt.alloc((size_t)(nseg + 1) * kMixedState * pix_count * sizeof(float), s), "allocate checkpoints");
    VJP_TRY(near.alloc((pix_count + 1) * sizeof(int64_t), s), "allocate near rays");
    VJP_TRY(cudaMemsetAsync(near.p, 0, sizeof(int64_t), s), "clear near rays");
    VJP_TRY(bases.alloc((size_t)12 * pix_count * sizeof(float), s), "allocate ray bases");
    VJP_TRY(rlist.alloc(pix_count * sizeof(int64_t), s), "allocate refine list");
    VJP_TRY(rcount.alloc(sizeof(unsigned long long), s), "allocate refine count");
    VJP_TRY(cudaMemsetAsync(rcount.p, 0, sizeof(unsigned long long), s), "clear refine count");
    float* dm[6];
    if (dev_out) {
      for (int m = 0; m < 6; ++m) dm[m] = maps[m];
    } else {
      VJP_TRY(dmaps.alloc(6 * pix_count * sizeof(float), s), "allocate maps");
      for (int m = 0; m < 6; ++m) dm[m] = (float*)dmaps.p + m * pix_count;
    }
    AdjArgs A;
    memset(&A, 0, sizeof(A));
    A.F = make_ptrs(f);
    A.G = make_geom(f);
    A.nside = nside;
    A.pix_begin = pix_begin;
    A.count = pix_count;
    A.rays = (int64_t*)rays.p;
    A.near = (int64_t*)near.p;
    A.bases = (float*)bases.p;
    A.n_steps = n_steps;
    A.C = C;
    A.nseg = nseg;
    A.ckpt = ckpt.p;
    for (int m = 0; m < 6; ++m) A.maps[m] = dm[m];
    A.refine_list = (int64_t*)rlist.p;
    A.refine_count = (unsigned long long*)rcount.p;
    VJP_TRY(cudaEventCreate(&e0), "cudaEventCreate");
    VJP_TRY(cudaEventCreate(&e1), "cudaEventCreate");
    VJP_TRY(cudaEventRecord(e0, s), "cudaEventRecord");
    const unsigned blocks = (unsigned)((pix_count + 127) / 128);
    int sms = 0;
    VJP_TRY(sm_count(&sms), "device attributes");
    const bool small = small_adjoint(pix_count, sms);
    with_forward_layout(f, [&](auto l) { launch_ckpt<decltype(l)::value, true>(A, small, blocks, s); });
    near_ckpt_kernel<false><<<near_ckpt_blocks(blocks, sms), 128, 0, s>>>(A);
    kernels += 2;
    VJP_TRY(cudaGetLastError(), "checkpointing forward");
    TraceArgs ta;
    ta.F = A.F;
    ta.G = A.G;
    ta.nside = nside;
    ta.pix_begin = pix_begin;
    ta.pix_count = pix_count;
    ta.n_steps = n_steps;
    for (int m = 0; m < 6; ++m) ta.maps[m] = dm[m];
    ta.refine_list = A.refine_list;
    ta.refine_count = A.refine_count;
    VJP_TRY(launch_refine(ta, s, &kernels), "refine kernel launch");
    VJP_TRY(cudaEventRecord(e1, s), "cudaEventRecord");
    if (!dev_out)
      for (int m = 0; m < 6; ++m)
        VJP_TRY(cudaMemcpyAsync(maps[m], dm[m], pix_count * sizeof(float), cudaMemcpyDeviceToHost, s),
                "copy maps to host");
    unsigned long long refined = 0;
    VJP_TRY(cudaMemcpyAsync(&refined, rcount.p, sizeof(refined), cudaMemcpyDeviceToHost, s), "read refine count");
    release();
    VJP_TRY(cudaStreamSynchronize(s), "srt_forward_tape");
    if (stats) {
      float ms = -1.f;
      cudaEventElapsedTime(&ms, e0, e1);
      stats->trace_ms = ms;
      stats->rays = pix_count;
      stats->ray_steps = pix_count * (int64_t)n_steps;
      stats->kernels = kernels;
      stats->d2h_bytes = dev_out ? 0 : 6 * pix_count * (int64_t)sizeof(float);
      stats->refined_rays = (int64_t)refined;
    }
    t->fields = f;
    t->device = f->device;
    t->nside = nside;
    t->pix_begin = pix_begin;
    t->pix_count = pix_count;
    t->n_steps = n_steps;
    t->C = C;
    t->nseg = nseg;
    t->rays = (int64_t*)rays.p;
    t->near = (int64_t*)near.p;
    t->bases = (float*)bases.p;
    t->ckpt = (float*)ckpt.p;
    t->bytes = (2 * pix_count + 1) * (int64_t)sizeof(int64_t) + 48 * pix_count + (int64_t)(nseg + 1) * kMixedState * pix_count * 4;
    rays.p = nullptr;  // owned by the tape from here on
    near.p = nullptr;
    bases.p = nullptr;
    ckpt.p = nullptr;
    *out = t;
    t = nullptr;
  }
done:
  release();
  for (DevBuf* b : {&rays, &near, &bases, &ckpt}) b->release();  // of a failed call
  if (rc != SRT_OK) cudaStreamSynchronize(s);
  scratch_settle(f->device, s);
  delete t;
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (prev != f->device) cudaSetDevice(prev);
  if (stats)
    stats->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_wall).count();
  return rc;
}

extern "C" int srt_vjp_tape(const srt_tape* tape, const float* const weights[SRT_NUM_MAPS], float* dphi,
                            float* db_xyz, unsigned flags, void* stream, srt_stats* stats) {
  NvtxRange nvtx_("srt_vjp_tape");
  if (!tape) return set_error(SRT_ERR_INVALID_ARGUMENT, "srt_vjp_tape: tape is NULL");
  return vjp_impl(tape->fields, tape->nside, tape->pix_begin, tape->pix_count, tape->n_steps, SRT_PRECISION_MIXED,
                  weights, dphi, db_xyz, tape->C, flags, stream, stats, tape);
}

extern "C" int64_t srt_tape_bytes(const srt_tape* tape) { return tape ? tape->bytes : 0; }

extern "C" int srt_tape_destroy(srt_tape* tape) {
  if (!tape) return SRT_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  if (prev != tape->device) cudaSetDevice(tape->device);
  // the calls that used the tape have returned, and they are synchronous
  for (void* p : {(void*)tape->rays, (void*)tape->near, (void*)tape->bases, (void*)tape->ckpt}) pool_free(p, nullptr);
  scratch_settle(tape->device, nullptr);
  if (prev != tape->device) cudaSetDevice(prev);
  delete tape;
  return SRT_OK;
}
