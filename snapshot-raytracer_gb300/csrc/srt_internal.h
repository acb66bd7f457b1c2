// srt_internal.h — shared declarations between the libsrt translation units.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <functional>
#include <string>
#include <nvtx3/nvToolsExt.h>
#include "srt.h"
#include "srt_scheme.cuh"

// Device memory of one set of laid-out fields (see srt_fields_create).
struct srt_fields {
  int device = 0;
  int64_t n[3] = {0, 0, 0};
  int64_t pn[3] = {0, 0, 0};  // padded extents n + 3
  // either cells (B_x, B_y, B_z, phi; 16 bytes per padded voxel), or padded FP32
  // planes and, where they fit, half cells or (four_taps) row pairs in the same order
  float4* cell[4] = {nullptr, nullptr, nullptr, nullptr};
  float* phi = nullptr;
  float* b[3] = {nullptr, nullptr, nullptr};
  float2* pr[4] = {nullptr, nullptr, nullptr, nullptr};
  // made on first REF16 use: padded half(B * 2^27), and phi as a plane where the
  // fields are cells
  __half* bh[3] = {nullptr, nullptr, nullptr};
  float* ref_phi = nullptr;
  int64_t bytes = 0;
  // The MIXED forward takes the four-tap passes (alloc_fields), else the second
  // differences, in every layout: MIXED's bits depend on the grid, the flags and the
  // device, not on what memory was free.
  bool four_taps = false;
  int layout() const {
    return cell[0] ? srt::kCells : (pr[0] ? (four_taps ? srt::kPairs : srt::kHalf) : srt::kPlanes);
  }
  // the MIXED trace kernel of this layout
  int mixed_mode() const {
    if (four_taps) return pr[0] ? srt::kMIXED_FOUR_PAIR : srt::kMIXED_FOUR;
    return cell[0] ? srt::kMIXED_CELL : (pr[0] ? srt::kMIXED_HALF : srt::kMIXED);
  }
  // the values of B component c (0-2) or phi (3), make_geom's ts floats apart
  const float* values(int c) const { return cell[c] ? &cell[c]->x : (c == 3 ? phi : b[c]); }
};

namespace srt {

// Device memory of fields: a per-device stream-ordered pool that keeps freed
// memory for reuse (srt_release_cached_memory trims it).
cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t s);
void pool_free(void* p, cudaStream_t s);
int64_t pool_reusable_bytes(int dev);
// A call's scratch, from a second pool that keeps a bounded amount; given back by
// pool_free on the stream of its last use. Both allocations go through the
// failure-injection hook (srt_debug_fail_alloc).
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s);
// Returns to the device what the scratch pool of `dev` holds unused above its bound
// (waits for s, where the scratch was given back, only if it holds more).
void scratch_settle(int dev, cudaStream_t s);

// NVTX range over a scope (the public entry points and their phases), for
// profilers' timelines and range filters; header-only, inert unless a tool
// is attached.
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

// Error reporting (thread-local last error message).
int set_error(int code, const char* fmt, ...);
int cuda_error(cudaError_t e, const char* what);

struct TraceArgs {
  FieldPtrs F;
  Geom G;
  int64_t nside = 0;
  int log2p = 0;            // launch order: Morton over a 2^log2p square per face
  int64_t launch_rays = 0;  // launch slots: 12 * 4^log2p (RING ranges) or pix_count (NESTED)
  int64_t pix_begin = 0, pix_count = 0;
  bool nested = false;      // [pix_begin, pix_begin + pix_count) is a NESTED range
  int n_steps = 0;
  float* maps[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  // MIXED: the output slots of rays that came within the cell-face guard are
  // appended here (NULL: no fallback) and re-traced by launch_refine.
  int64_t* refine_list = nullptr;
  unsigned long long* refine_count = nullptr;
};

Geom make_geom(const srt_fields* f);
FieldPtrs make_ptrs(const srt_fields* f);

// Field layout kernels.
// src: planes k0 .. k1-1 of phi (comps 1, dst[0]) or of the interleaved B
// (comps 3, dst[0..2]); device memory or mapped pinned host memory.
cudaError_t launch_pad_fields(const float* src, int comps, float* const dst[3], const int64_t n[3],
                              const int64_t pn[3], int64_t k0, int64_t k1, cudaStream_t s);
// src: device memory.
cudaError_t launch_cells(const float* src, int comps, float4* const dst[3], const int64_t n[3], int64_t k0, int64_t k1,
                         cudaStream_t s);
// count floats from mapped pinned host memory to device memory.
cudaError_t launch_fetch(const float* src, float* dst, int64_t count, cudaStream_t s);
cudaError_t launch_quantize_half(const float* src, int ts, __half* dst, int64_t count, cudaStream_t s);
// The same values as a plane.
cudaError_t launch_extract(const float* src, int ts, float* dst, int64_t count, cudaStream_t s);
// Row pairs or half cells of a padded plane array.
cudaError_t launch_pair_build(const float* src, float2* dst, const int64_t pn[3], bool half, cudaStream_t s);

// Trace kernel launch (mode = kFP64 / kREF16 / a handle's mixed_mode()).
cudaError_t launch_trace(int mode, const TraceArgs& a, cudaStream_t s, int64_t* kernels);
// Re-trace of the rays listed by a MIXED trace (count read on the device), in FP64 or,
// long lists, in double-float.
cudaError_t launch_refine(const TraceArgs& a, cudaStream_t s, int64_t* kernels);
// The FP64 form of a small range, five warps or one per ray (srt_retrace.cu):
// launch_trace takes it up to kWideFp64RaysPerSM rays per SM, where a lane per ray
// leaves the FP64 unit waiting (256^3, 16 steps, 152 SMs: 2,000 rays 0.89 against 4.88
// ms, 14,000 5.9 against 8.2, 20,000 8.4 against 9.3, 24,000 10.0 against 9.3).
constexpr int64_t kWideFp64RaysPerSM = 140;
cudaError_t launch_wide_fp64(const TraceArgs& a, cudaStream_t s, int64_t* kernels);

// Progressive reads of an HDF5 field (srt_io.cpp), for srt_fields_load_h5.
// h5_field_open reads the header and checks the dataset as
// srt_h5_read_scalar (vector3 false) or srt_h5_read_vector3 (true) do;
// h5_field_read fills `out` (all elements as floats, times `scale`) in order
// along the slowest axis and calls ready(n) once the first n floats are final;
// ready returning false stops the read (the call then returns
// SRT_ERR_CANCELLED).
struct H5Field;
int h5_field_open(const char* path, const char* dset, bool vector3, int64_t dims[8], int* rank, H5Field** out);
int h5_field_read(H5Field* h, float* out, double scale, const std::function<bool(int64_t)>& ready);
void h5_field_close(H5Field* h);

// Forgets srt_forward_noalloc's cached scratch addresses (srt_noalloc.cu).
void noalloc_forget_scratch();

// Number of SMs of the current device.
cudaError_t sm_count(int* sms);

// Peak issue-rate probes (FMA loop kernels); returns achieved FLOP/s.
cudaError_t probe_fma(int kind, double* flops_per_s);

}  // namespace srt
