// srt_retrace.cu — warp-per-ray traces (srt_wide.cuh): the re-trace of the
// rays a MIXED trace flagged, and the FP64 form of small ray ranges.
#include <algorithm>
#include <cstdlib>
#include "srt_internal.h"
#include "srt_wide.cuh"

namespace srt {

__device__ const WideTables kWideTables = make_wide_tables();

// One-warp blocks; each traces rays blockIdx.x, + gridDim.x, ... of its list.
// LIST: the rays a MIXED trace listed, count read on the device (no host round
// trip); the kernel whose range [min_count, max_count] holds the count runs,
// the other leaves at once. Otherwise every ray of the requested range.
template <typename R, bool LIST>
__global__ void __launch_bounds__(32, 16) wide_kernel(const TraceArgs A, int64_t min_count, int64_t max_count) {
  // raw storage viewed as R: dd has a constructor, which a shared array of it
  // would not run anyway
  __shared__ float2 scratch[kWsSize];
  __shared__ int cell[6];
  R* S = reinterpret_cast<R*>(scratch);
  int64_t n = A.pix_count;
  if (LIST) {
    n = min((int64_t)*A.refine_count, n);
    if (n < min_count || n > max_count) return;
  }
  WideLane<R> L;
  L.start((int)threadIdx.x, kWideTables);
  L.constants(S);
#pragma unroll 1
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t o = LIST ? A.refine_list[i] : i;  // output slot
    const int64_t ring = A.nested ? hp_nest2ring(A.nside, A.pix_begin + o) : A.pix_begin + o;
    const RayDir d = ray_dir_pix(A.nside, ring);
    {
      double y[19];
      init_std(d, A.G, y);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 19; ++j)
        if (L.lane == j) L.y = R(y[j]);
    }
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
    }
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
}

constexpr int kWideBlocksPerSM = 16;

namespace {
cudaError_t sm_count(int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  return e == cudaSuccess ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) : e;
}
}  // namespace

// Lists up to dd_min rays (two warps per SM sub-partition) are re-traced in
// FP64 with the one-lane FP64 form's operations (bit-identical maps), longer
// ones in double-float arithmetic on the FP32 pipes (maps within one float
// ulp). The environment variable SRT_REFINE_DD_MIN overrides dd_min (tests use
// it to reach both on small skies).
constexpr int64_t kRefineWarpsPerSubpartition = 1;

cudaError_t launch_refine(const TraceArgs& a, cudaStream_t s, int64_t* kernels) {
  int sms = 0;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  int64_t dd_min = kRefineWarpsPerSubpartition * 4 * (int64_t)sms;
  if (const char* v = getenv("SRT_REFINE_DD_MIN")) dd_min = strtoll(v, nullptr, 10);
  const int64_t blocks = std::min(a.pix_count, kWideBlocksPerSM * (int64_t)sms);
  if (blocks < 1) return cudaSuccess;
  wide_kernel<double, true><<<(unsigned)blocks, 32, 0, s>>>(a, 1, dd_min);
  wide_kernel<dd, true><<<(unsigned)blocks, 32, 0, s>>>(a, std::max<int64_t>(dd_min, 0) + 1, a.pix_count);
  if (kernels) *kernels += 2;
  return cudaGetLastError();
}

cudaError_t launch_wide_fp64(const TraceArgs& a, cudaStream_t s, int64_t* kernels) {
  int sms = 0;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::min(a.pix_count, kWideBlocksPerSM * (int64_t)sms);
  wide_kernel<double, false><<<(unsigned)blocks, 32, 0, s>>>(a, 0, 0);
  if (kernels) ++*kernels;
  return cudaGetLastError();
}

}  // namespace srt
