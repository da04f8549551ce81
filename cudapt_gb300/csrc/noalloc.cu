// Allocation-free variant of the device-array bilateral filter, for callers
// that cannot allocate device memory when they call it: code that runs while a
// custom allocator or a pre-reserved memory pool owns the device heap, or on
// a latency-critical path.  The spatial weights reach the kernel as one of its
// arguments, so there is nothing to allocate, to copy or to share: calls on
// different streams or threads do not meet.
//
// The table holds 64 floats, so radius <= 31 (2*radius+1 weights); larger
// radii are rejected before any arithmetic on the radius.  Each call
// synchronizes the caller's stream (all work queued on it so far, not only the
// filter), so it is refused (GBPT_ERR_STATE) while that stream is captured.
#include <cuda_runtime.h>

#include <string>

#include "gbpt_internal.h"
#include "launch.h"

extern "C" gbpt_status gbpt_bilateral_noalloc(const float* color, const float* pos, const float* norm,
                                              const float* emit, uint32_t width, uint32_t height, float color_eud,
                                              float pos_eud, float norm_eud, float emit_eud, uint32_t radius,
                                              const float* g, float* out, void* stream) {
  if (!color || !pos || !norm || !g || !out) return gbpt::fail(GBPT_ERR_INVALID_ARG, "NULL argument");
  if (width == 0 || height == 0) return gbpt::fail(GBPT_ERR_INVALID_ARG, "empty image");
  // compared before any arithmetic on radius, which could wrap
  if (radius > (sizeof(gbpt::BilatTable) / sizeof(float) - 1) / 2)
    return gbpt::fail(GBPT_ERR_INVALID_ARG, "radius " + std::to_string(radius) +
                                                " exceeds the allocation-free limit of 31 (64-entry weight table)");
  cudaStream_t s = (cudaStream_t)stream;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(s, &cap);
  if (e != cudaSuccess || cap != cudaStreamCaptureStatusNone)
    return gbpt::fail(GBPT_ERR_STATE, "gbpt_bilateral_noalloc synchronizes its stream: it cannot be called while the "
                                      "stream is being captured");
  e = gbpt::launch_bilateral(color, pos, norm, emit, width, height, color_eud, pos_eud, norm_eud, emit_eud, radius, g,
                             out, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return gbpt::fail(GBPT_ERR_CUDA, std::string("bilateral_noalloc: ") + cudaGetErrorString(e));
  return GBPT_OK;
}
