// Shared definitions for the RBF attention kernels: tile geometry, argument blocks, status codes.
#pragma once

#include "ptx.cuh"

namespace rbf {

static constexpr int kTile = 128;       // rows of a query tile == keys of a key tile
static constexpr float kLog2e = 1.4426950408889634f;

// Status codes returned through the C ABI (0 = success).
enum Status : int {
  kOk = 0,
  kErrBadArgument = 1,     // null pointer, non-positive size, unsupported D / dtype
  kErrBadLayout = 2,       // stride or alignment the TMA engine cannot address
  kErrWorkspace = 3,       // workspace missing or too small
  kErrTensorMap = 4,       // cuTensorMapEncodeTiled failed or is unavailable
  kErrLaunch = 5,          // CUDA launch error
  kErrDevice = 6,          // a device-side bounded wait ran out (see rbf_b200_read_device_status)
};

// Sum of `count` floats `stride` apart (<= 0: none), four at a time: the loads of a thread do not wait for one another.
__device__ __forceinline__ float strided_sum(const float* p, int64_t stride, int count) {
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
  int i = 0;
  for (; i + 3 < count; i += 4, p += 4 * stride) {
    s0 += p[0];
    s1 += p[stride];
    s2 += p[2 * stride];
    s3 += p[3 * stride];
  }
  for (; i < count; ++i, p += stride) s0 += *p;
  return (s0 + s1) + (s2 + s3);
}

// Number of key/query rows after padding to whole tiles; the per-row fp32 side arrays
// (key norms, query norms, delta) use this as their row pitch so that every tile read is in bounds.
__host__ __device__ inline int padded_rows(int n) { return (n + kTile - 1) / kTile * kTile; }

}  // namespace rbf
