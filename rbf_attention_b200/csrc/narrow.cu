// fp32 tensors on the fp16-operand kernels: narrowing of a call's inputs and widening of its gradients, one launch each.
// Roofline: HBM / launch latency. PyTorch took one launch per tensor and direction, and the check whether an input left
// fp16's range another five per tensor (an isinf, an any and an or, with temporaries): 40 launches and 157 us of device
// time in a training pass at B2 H8 N1024 D64, against 8 launches with these two kernels (the range flag's clearing is one of
// them; the narrowing's last block posts it). That pass: 426 us with PyTorch's launches, 276 us with these kernels and a
// posting launch of its own, 145-164 us now, with the calls prepared in the extension as well.
#include <cuda_fp16.h>

#include "launch.h"

namespace rbf {
namespace {

// One 16-byte store of eight halves per thread; blockIdx.y selects the tensor.
__global__ void __launch_bounds__(256) narrow_kernel(const NarrowArgs a) {
  const int t = blockIdx.y;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  bool bad = false;
  if (i < a.chunks) {
    const int per_row = a.D / 8;
    const int64_t row = i / per_row;
    const int ch = static_cast<int>(i - row * per_row);
    const int64_t bh = row / a.N, n = row - bh * a.N;
    const int64_t b = bh / a.H, h = bh - b * a.H;
    const float4* src = reinterpret_cast<const float4*>(a.src[t] + b * a.strides[t][0] + h * a.strides[t][1] +
                                                        n * a.strides[t][2] + ch * 8);
    const float4 x = src[0], y = src[1];
    const uint4 o = make_uint4(pack2<false>(x.x, x.y), pack2<false>(x.z, x.w), pack2<false>(y.x, y.y), pack2<false>(y.z, y.w));
    reinterpret_cast<uint4*>(a.dst[t])[i] = o;
    const uint32_t w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) bad |= (w[j] & 0x7fffu) == 0x7c00u || (w[j] & 0x7fff0000u) == 0x7c000000u;   // an infinity
  }
  if (t < a.checked && __any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *a.flag = 1u;
  if (a.status_slot == nullptr) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&a.flag[1], 1u) == gridDim.x * gridDim.y - 1) {
    __threadfence();
    post_status_word(reinterpret_cast<const DeviceStatus*>(a.flag), a.status_slot);
  }
}

__global__ void __launch_bounds__(256) widen_kernel(const WidenArgs a) {
  const int t = blockIdx.y;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= a.chunks) return;
  const uint4 v = reinterpret_cast<const uint4*>(a.src[t])[i];
  const float2 p0 = unpack2<false>(v.x), p1 = unpack2<false>(v.y), p2 = unpack2<false>(v.z), p3 = unpack2<false>(v.w);
  float4* dst = reinterpret_cast<float4*>(a.dst[t]) + 2 * i;
  dst[0] = make_float4(p0.x, p0.y, p1.x, p1.y);
  dst[1] = make_float4(p2.x, p2.y, p3.x, p3.y);
}

}  // namespace

cudaError_t launch_narrow(const NarrowArgs& a, cudaStream_t stream) {
  narrow_kernel<<<dim3(static_cast<unsigned>((a.chunks + 255) / 256), a.count), 256, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_widen(const WidenArgs& a, cudaStream_t stream) {
  widen_kernel<<<dim3(static_cast<unsigned>((a.chunks + 255) / 256), a.count), 256, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace rbf
