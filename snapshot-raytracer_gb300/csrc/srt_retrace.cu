// srt_retrace.cu — warp-per-ray traces (srt_wide.cuh): the re-trace of the
// rays a MIXED trace flagged, and the FP64 form of small ray ranges.
#include <algorithm>
#include <cstdlib>
#include "srt_internal.h"
#include "srt_wide.cuh"

namespace srt {

__device__ const WideTables kWideTables = make_wide_tables();

// The rays of a launch: those a MIXED trace listed (LIST; the count read on the
// device, no host round trip, and nothing to do unless it lies in [min_count,
// max_count]: the kernels for short and for long lists are both queued), else the whole
// range.
template <bool LIST>
__device__ __forceinline__ int64_t ray_count(const TraceArgs& A, int64_t min_count, int64_t max_count) {
  if (!LIST) return A.pix_count;
  const int64_t n = min((int64_t)*A.refine_count, A.pix_count);
  return n < min_count || n > max_count ? 0 : n;
}
template <bool LIST>
__device__ __forceinline__ int64_t output_slot(const TraceArgs& A, int64_t i) { return LIST ? A.refine_list[i] : i; }
__device__ __forceinline__ RayDir slot_direction(const TraceArgs& A, int64_t o) {
  return ray_dir_pix(A.nside, A.nested ? hp_nest2ring(A.nside, A.pix_begin + o) : A.pix_begin + o);
}

// Lane j < 19 of a warp takes component j of the initial state.
template <typename R>
__device__ __forceinline__ void init_lane(WideLane<R>& L, const RayDir& d, const Geom& G) {
  double y[19];
  init_std(d, G, y);
#pragma unroll
  for (int j = 0; j < 19; ++j)
    if (L.lane == j) L.y = R(y[j]);
}

// The maps from the state the warp's lanes hold.
template <typename R>
__device__ __forceinline__ void write_maps(const WideLane<R>& L, R* S, const TraceArgs& A, const RayDir& d, int64_t o) {
  if (L.lane < 19) S[kWsY + L.lane] = L.y;
  __syncwarp();
  if (L.lane == 0) {
    double y[19];
    for (int j = 0; j < 19; ++j) y[j] = (double)S[kWsY + j];
    float out[6];
    extract_std(d, A.G, y, out);
#pragma unroll
    for (int m = 0; m < 6; ++m) A.maps[m][o] = out[m];
  }
  __syncwarp();
}

// The right-hand side from the interpolations and the frame in the scratch.
template <typename R>
__device__ __forceinline__ void run_rounds(WideLane<R>& L, R* S, int st) {
  L.round1(S);
  __syncwarp();
  L.round2(S);
  __syncwarp();
  L.round3(S);
  __syncwarp();
  L.round4(S);
  __syncwarp();
  L.round5(S);
  __syncwarp();
  L.round6(S, st);
  __syncwarp();
}

// One warp per ray: rays blockIdx.x, + gridDim.x, ... of the n, by one-warp blocks.
template <typename R, bool LIST>
__device__ __forceinline__ void wide_trace(const TraceArgs& A, R* S, int* cell, int64_t n) {
  WideLane<R> L;
  L.start((int)threadIdx.x, kWideTables);
  L.constants(S);
#pragma unroll 1
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t o = output_slot<LIST>(A, i);
    const RayDir d = slot_direction(A, o);
    init_lane(L, d, A.G);
    __syncwarp();
#pragma unroll 1
    for (int step = 0; step < A.n_steps; ++step) {
#pragma unroll 1
      for (int st = 0; st < 4; ++st) {
        L.stage(S, st);
        __syncwarp();
        L.position(S, cell, A.G);
        __syncwarp();
        L.load_taps(cell, A.F, A.G);  // in flight through the weights and the frame
        L.weights(S);
        L.frame(S);
        __syncwarp();
        L.x_pass(S);
        __syncwarp();
        L.y_pass(S);
        __syncwarp();
        L.z_pass(S);
        __syncwarp();
        run_rounds(L, S, st);
      }
    }
    write_maps(L, S, A, d, o);
  }
}

// A list of more than min_count - 1 rays: in FP64 up to fp64_max of them, else in
// double-float (one launch for both: an empty one takes 4 us, 0.8 % of a 128^3 sky).
__global__ void __launch_bounds__(32, 16) wide_list_kernel(const TraceArgs A, int64_t min_count, int64_t fp64_max) {
  // raw storage viewed as double or dd: dd has a constructor, which a shared array
  // of it would not run anyway
  __shared__ float2 scratch[kWsSize];
  __shared__ int cell[6];
  const int64_t n = ray_count<true>(A, min_count, A.pix_count);
  if (blockIdx.x >= n) return;
  if (n <= fp64_max)
    wide_trace<double, true>(A, reinterpret_cast<double*>(scratch), cell, n);
  else
    wide_trace<dd, true>(A, reinterpret_cast<dd*>(scratch), cell, n);
}

// The FP64 form of a range.
__global__ void __launch_bounds__(32, 16) wide_range_kernel(const TraceArgs A) {
  __shared__ double scratch[kWsSize];
  __shared__ int cell[6];
  wide_trace<double, false>(A, scratch, cell, A.pix_count);
}

// Five warps per ray in FP64 (FieldLane): the shortest way through a stage, for
// lists and ranges of at most kBlockRaysPerSM rays per SM.
constexpr int kBlockThreads = 160, kBlockRaysPerSM = 4;

template <bool LIST>
__global__ void __launch_bounds__(kBlockThreads, kBlockRaysPerSM)
    block_kernel(const TraceArgs A, int64_t min_count, int64_t max_count) {
  __shared__ double S[kWsBlockSize];
  __shared__ int cell[12];
  const int64_t n = ray_count<LIST>(A, min_count, max_count);
  if (blockIdx.x >= n) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WideLane<double> L;  // warp 0: the state and the rounds; warp 4: the frame
  FieldLane<double> I;
  L.start(lane, kWideTables);
  I.start(lane, warp < 4 ? warp : 0);
  if (warp == 0) L.constants(S);
#pragma unroll 1
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t o = output_slot<LIST>(A, i);
    RayDir d = {};
    if (warp == 0) {
      d = slot_direction(A, o);
      init_lane(L, d, A.G);
    }
#pragma unroll 1
    for (int step = 0; step < A.n_steps; ++step) {
#pragma unroll 1
      for (int st = 0; st < 4; ++st) {
        if (warp == 0) L.stage(S, st);
        __syncthreads();
        if (warp < 4) {
          I.position(S, cell, A.G);
          __syncwarp();
          I.load_taps(cell, A.F, A.G);
          I.weights(S);
          __syncwarp();
          I.x_pass(S);
          __syncwarp();
          I.y_pass(S);
          __syncwarp();
          I.z_pass(S);
        } else {
          L.frame(S);
        }
        __syncthreads();
        if (warp == 0) run_rounds(L, S, st);
      }
    }
    if (warp == 0) write_maps(L, S, A, d, o);
  }
}

constexpr int kWideBlocksPerSM = 16;

cudaError_t sm_count(int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  return e == cudaSuccess ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) : e;
}

// Lists of up to 64 rays per SM are re-traced in FP64 with the one-lane FP64 form's
// operations (bit-identical maps): by five warps per ray up to kBlockRaysPerSM rays
// per SM, where a stage's latency counts, by one warp per ray above, where the FP64
// unit's rate does. Longer lists run in double-float arithmetic on the FP32 pipes:
// maps within four float ulps of FP64 (tested), but for a ray within ~1e-12 cells of
// a face, which may take the other cell. Double-float is the faster from four rays
// per SM on already (256^3, 1024 steps: 2,813 rays 85 ms in FP64, 24.5 in
// double-float; 7,850 rays 212 and 56.6), so the line costs time: up to it a sky and
// the same sky in batches, whose lists are shorter, have the same bits. The
// environment variable SRT_REFINE_DD_MIN overrides dd_min (tests use it to reach
// both on small skies).
constexpr int kFp64ListRaysPerSM = 64;

cudaError_t launch_refine(const TraceArgs& a, cudaStream_t s, int64_t* kernels) {
  int sms = 0;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  int64_t dd_min = kFp64ListRaysPerSM * (int64_t)sms;
  if (const char* v = getenv("SRT_REFINE_DD_MIN")) dd_min = std::max(0LL, strtoll(v, nullptr, 10));
  if (a.pix_count < 1) return cudaSuccess;
  const int64_t block_max = std::min(dd_min, kBlockRaysPerSM * (int64_t)sms);
  const int64_t blocks = std::min(a.pix_count, kBlockRaysPerSM * (int64_t)sms);
  const int64_t warps = std::min(a.pix_count, kWideBlocksPerSM * (int64_t)sms);
  block_kernel<true><<<(unsigned)blocks, kBlockThreads, 0, s>>>(a, 1, block_max);
  if (kernels) ++*kernels;
  if (a.pix_count > block_max) {
    wide_list_kernel<<<(unsigned)warps, 32, 0, s>>>(a, block_max + 1, dd_min);
    if (kernels) ++*kernels;
  }
  return cudaGetLastError();
}

cudaError_t launch_wide_fp64(const TraceArgs& a, cudaStream_t s, int64_t* kernels) {
  int sms = 0;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  if (a.pix_count <= kBlockRaysPerSM * (int64_t)sms)
    block_kernel<false><<<(unsigned)a.pix_count, kBlockThreads, 0, s>>>(a, 0, 0);
  else
    wide_range_kernel<<<(unsigned)std::min(a.pix_count, kWideBlocksPerSM * (int64_t)sms), 32, 0, s>>>(a);
  if (kernels) ++*kernels;
  return cudaGetLastError();
}

}  // namespace srt
