// GELU of the model's MLP (nn.GELU() between the two projections of every block, train_rbf_transformer.py:143: the
// exact, erf-based form) for 16-bit activations, forward and backward as streaming kernels. Roofline: HBM (forward:
// read h, write a; backward: read h and dy, write dh). The normal distribution function comes from the rational
// approximation 7.1.26 of Abramowitz & Stegun, erfc(z) = t (a1 + t (a2 + t (a3 + t (a4 + t a5)))) exp(-z^2) with
// t = 1 / (1 + p z), absolute error below 1.5e-7 - a thousandth of a bf16 rounding step - at one reciprocal and one
// exponential on the special-function unit; erff() costs as many instructions as the rest of the element and makes
// the kernel issue-bound. The backward also sums its output over the rows (the bias gradient of the projection that
// feeds the GELU) in the same pass, with the column-sum kernel's layout: a block owns 256 columns and a band of rows.
#include <cstdint>
#include <cuda_runtime.h>

#include "launch.h"

namespace rbf {
namespace {

template <bool kBf16>
__device__ __forceinline__ float2 g_unpack(uint32_t w) {
  if constexpr (kBf16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  return make_float2(__half2float(__ushort_as_half(static_cast<unsigned short>(w & 0xffffu))),
                     __half2float(__ushort_as_half(static_cast<unsigned short>(w >> 16))));
}
template <bool kBf16>
__device__ __forceinline__ uint32_t g_pack(float a, float b) {
  if constexpr (kBf16) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
  }
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ float g_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float g_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Phi(x) = P(N(0,1) <= x) and e = exp(-x^2 / 2) of two values. Two-wide multiplies and additions (the same roundings as
// one at a time; the coefficients carry the 0.5 of 0.5 erfc(z)).
__device__ __forceinline__ float2 normal_cdf2(float2 x, float2& e) {
  float t0 = g_rcp(fmaf(0.3275911f * 0.70710678f, fabsf(x.x), 1.0f));           // z = |x| / sqrt(2)
  float t1 = g_rcp(fmaf(0.3275911f * 0.70710678f, fabsf(x.y), 1.0f));
  float e0, e1;
  fmul2(e0, e1, x.x, x.y, x.x, x.y);
  fmul2(e0, e1, e0, e1, -0.5f * 1.4426950408889634f, -0.5f * 1.4426950408889634f);
  e = make_float2(g_ex2(e0), g_ex2(e1));
  float q0 = 0.5f * 1.061405429f, q1 = q0;
  ffma2v(q0, q1, t0, t1, q0, q1, 0.5f * -1.453152027f, 0.5f * -1.453152027f);
  ffma2v(q0, q1, t0, t1, q0, q1, 0.5f * 1.421413741f, 0.5f * 1.421413741f);
  ffma2v(q0, q1, t0, t1, q0, q1, 0.5f * -0.284496736f, 0.5f * -0.284496736f);
  ffma2v(q0, q1, t0, t1, q0, q1, 0.5f * 0.254829592f, 0.5f * 0.254829592f);
  fmul2(t0, t1, t0, t1, q0, q1);
  fmul2(q0, q1, t0, t1, e.x, e.y);                                               // 0.5 erfc(z)
  fadd2(t0, t1, 1.0f, 1.0f, -q0, -q1);
  return make_float2(x.x >= 0.f ? t0 : q0, x.y >= 0.f ? t1 : q1);
}

// Both grids are what is resident at once. Two values per instruction, two chunks (forward) or the next row (backward) in
// flight, five or six blocks per SM and one wave of them, against one value at a time and 16 or 8 blocks per SM of which 8 or
// 4 were resident (bf16, back to back, device and launches):
//   65792 x 2048: forward 95.7 -> 92.8 us (5.8 TB/s), backward with the bias sums 165.2 -> 129.0 us (6.3 TB/s)
//   16400 x 2048: 27.4 -> 27.3, 49.7 -> 38.7;  65792 x 512: 27.3 -> 27.5, 56.2 -> 41.7
// (backward two-wide alone 159.6, without unrolling 151.9, one wave of four blocks 136.7; two rows ahead with four blocks
// 136.7, with three 151.8.)
constexpr int kGeluFwdBlocks = 6;
constexpr int kGeluBwdBlocks = 5;

template <bool kBf16>
__global__ void __launch_bounds__(256, kGeluFwdBlocks) gelu_fwd_kernel(const uint4* __restrict__ h, uint4* __restrict__ out,
                                                                       int64_t n16) {
  for (int64_t i = blockIdx.x * 512ll + threadIdx.x; i < n16; i += gridDim.x * 512ll) {
    uint4 raw[2];                                 // two chunks' loads under way
    raw[0] = h[i];
    const bool both = i + 256 < n16;
    raw[1] = both ? h[i + 256] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 1 && !both) break;
      const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 x = g_unpack<kBf16>(w[j]);
        float2 e;
        const float2 c = normal_cdf2(x, e);
        o[j] = g_pack<kBf16>(x.x * c.x, x.y * c.y);
      }
      out[i + u * 256] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// dh = dy * (Phi(h) + h phi(h)); partials[band][c] = sum over the band's rows of dh[:, c] (when partials != nullptr)
template <bool kBf16>
__global__ void __launch_bounds__(256, kGeluBwdBlocks) gelu_bwd_kernel(const uint16_t* __restrict__ h,
                                                                       const uint16_t* __restrict__ dy,
                                                                       uint16_t* __restrict__ dh, int64_t rows, int cols,
                                                                       int64_t band, float* __restrict__ partials) {
  __shared__ float s_acc[8][256 + 8];
  grid_dependents_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = (blockIdx.x * 32 + lane) * 8;
  const int64_t r0 = blockIdx.y * band, r1 = min(r0 + band, rows);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < cols) {
    // the next row's loads are under way while a row is evaluated
    uint4 h_next = make_uint4(0u, 0u, 0u, 0u), g_next = h_next;
    if (r0 + warp < r1) {
      h_next = *reinterpret_cast<const uint4*>(h + (r0 + warp) * cols + col);
      g_next = *reinterpret_cast<const uint4*>(dy + (r0 + warp) * cols + col);
    }
#pragma unroll 1                                  // unrolled twice it takes 60 registers
    for (int64_t r = r0 + warp; r < r1; r += 8) {
      const int64_t at = r * cols + col;
      const uint4 hr = h_next, gr = g_next;
      if (r + 8 < r1) {
        h_next = *reinterpret_cast<const uint4*>(h + at + 8ll * cols);
        g_next = *reinterpret_cast<const uint4*>(dy + at + 8ll * cols);
      }
      const uint32_t hw[4] = {hr.x, hr.y, hr.z, hr.w}, gw[4] = {gr.x, gr.y, gr.z, gr.w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 x = g_unpack<kBf16>(hw[j]), g = g_unpack<kBf16>(gw[j]);
        float2 e;
        const float2 c = normal_cdf2(x, e);
        float d0, d1;
        fmul2(d0, d1, x.x, x.y, 0.3989422804f, 0.3989422804f);
        ffma2v(d0, d1, d0, d1, e.x, e.y, c.x, c.y);
        fmul2(d0, d1, d0, d1, g.x, g.y);
        o[j] = g_pack<kBf16>(d0, d1);
        // the sums take the rounded values: what a reduction over the stored dh would see
        const float2 rd = g_unpack<kBf16>(o[j]);
        fadd2(acc[2 * j], acc[2 * j + 1], acc[2 * j], acc[2 * j + 1], rd.x, rd.y);
      }
      *reinterpret_cast<uint4*>(dh + at) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (partials == nullptr) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) s_acc[warp][lane * 8 + j] = acc[j];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < cols) {
    float sum = 0.f;
#pragma unroll
    for (int wv = 0; wv < 8; ++wv) sum += s_acc[wv][threadIdx.x];
    partials[static_cast<int64_t>(blockIdx.y) * cols + c] = sum;
  }
}

}  // namespace

cudaError_t launch_gelu_fwd(const void* h, void* out, int64_t n, bool bf16, int sms, cudaStream_t stream) {
  const int64_t n16 = n / 8;
  if (n16 == 0) return cudaSuccess;
  const int64_t want = (n16 + 511) / 512, most = static_cast<int64_t>(sms) * kGeluFwdBlocks;
  const int grid = static_cast<int>(want < most ? want : most);
  if (bf16) gelu_fwd_kernel<true><<<grid, 256, 0, stream>>>(static_cast<const uint4*>(h), static_cast<uint4*>(out), n16);
  else gelu_fwd_kernel<false><<<grid, 256, 0, stream>>>(static_cast<const uint4*>(h), static_cast<uint4*>(out), n16);
  return cudaGetLastError();
}

cudaError_t launch_gelu_bwd(const void* h, const void* dy, void* dh, int64_t rows, int cols, bool bf16, float* partials,
                            float* dbias, int sms, cudaStream_t stream) {
  if (rows == 0) return dbias != nullptr ? cudaMemsetAsync(dbias, 0, cols * sizeof(float), stream) : cudaSuccess;
  const int col_blocks = (cols + 255) / 256;
  int bands = col_sums_bands(rows, cols, sms);
  const int one_wave = sms * kGeluBwdBlocks / col_blocks;      // (of few bands a wave may be far from full)
  if (one_wave >= 8 && bands > one_wave) bands = one_wave;
  const int64_t band = (rows + bands - 1) / bands;
  const dim3 grid(col_blocks, bands);
  const uint16_t* hp = static_cast<const uint16_t*>(h);
  const uint16_t* gp = static_cast<const uint16_t*>(dy);
  uint16_t* op = static_cast<uint16_t*>(dh);
  float* part = dbias != nullptr ? partials : nullptr;
  if (bf16) gelu_bwd_kernel<true><<<grid, 256, 0, stream>>>(hp, gp, op, rows, cols, band, part);
  else gelu_bwd_kernel<false><<<grid, 256, 0, stream>>>(hp, gp, op, rows, cols, band, part);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || dbias == nullptr) return e;
  return launch_col_sums_final(partials, bands, cols, dbias, stream);
}

}  // namespace rbf
