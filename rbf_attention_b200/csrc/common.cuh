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

// Order of the backward's items, (key tile, batch-head) pairs: head by head, which keeps a head's Q, dO and dQ in L2, except
// for the last heads of a causal launch. Their key tiles run heaviest first over all of them, so that the launch ends with its
// shortest items. They are as many as have the work that all SMs get through during a longest item, sms * n steps of
// n (n + 1) / 2 per head; what starts last then ends last by a step or two, not by n.
// Backward call, microseconds, against head by head throughout (in turn on one box, replayed back to back): B4 H8 N1024 D64
// 36.4 -> 30.7, B2 H12 N1500 D80 79.4 -> 59.9, B4 H8 N4100 D64 239 -> 225, B64 H8 N1028 D64 377 -> 371, B8 H16 N4096 D64
// 853 -> 833, B2 H32 N16384 D128 level. (All heads in such groups one after the other: the same within 1 %; groups of half the
// size 231-251 at N4100, of twice the size 418-436 at N1028.)
inline int item_group(int n_tiles, int heads, int causal, int sms) {
  const int group = causal ? (2 * sms + n_tiles) / (n_tiles + 1) : 0;
  return group < heads ? group : heads;
}
__device__ __forceinline__ void decode_item(int item, int n_tiles, int plain_heads, int group, int& bh, int& kt) {
  const int w = item - plain_heads * n_tiles;
  if (w < 0) {
    bh = item / n_tiles;
    kt = item - bh * n_tiles;
  } else {
    kt = w / group;
    bh = plain_heads + w - kt * group;
  }
}

// Number of key/query rows after padding to whole tiles; the per-row fp32 side arrays
// (key norms, query norms, delta) use this as their row pitch so that every tile read is in bounds.
__host__ __device__ inline int padded_rows(int n) { return (n + kTile - 1) / kTile * kTile; }

}  // namespace rbf
