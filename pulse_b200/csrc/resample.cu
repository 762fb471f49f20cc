// resample.cu -- the upscaling hand-off: the accumulation target resampled to
// the view's resolution as RGBA16F (half4), headless.
//
// The reference draws a fullscreen triangle whose fragment shader samples the
// path-tracer target with wgpu's default sampler (nearest filtering, clamp to
// edge; src/path_tracer/pt_upscaling/pt_upscaling.wgsl:48-50,
// src/path_tracer/pt_upscaling/node.rs:70-77) into the Rgba16Float view
// target.  Here output texel (x, y) of an out_w x out_h image takes
//   u = (x + 0.5) / out_w,  v = (y + 0.5) / out_h       (the fragment centre)
//   nearest:  source texel (min(floor(u W), W-1), min(floor(v H), H-1))
//   bilinear: the four texels around (u W - 0.5, v H - 0.5), clamped to the edge,
//             mixed as (1-fx)(1-fy) a + fx(1-fy) b + (1-fx) fy c + fx fy d
// and converts each channel to half with round-to-nearest-even.
#include <cuda_fp16.h>

#include "kernels.h"

namespace pt {

namespace {

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
  return (uint32_t)__half_as_ushort(ha) | ((uint32_t)__half_as_ushort(hb) << 16);
}

__device__ __forceinline__ uint2 pack_half4(float4 c) {
  return make_uint2(pack_half2(c.x, c.y), pack_half2(c.z, c.w));
}

// Bound by the source texels a thread reads (four 16-byte loads a bilinear texel, from
// L1) and by the divisions of its position.  A block covers kRows rows, so that the
// columns' positions are worked out once, and a thread two neighbouring texels, one
// 16-byte store.  Bilinear 1080p -> 4K (99.5 MB, 15.0 us at the measured copy rate):
// 41 us with a thread per texel; 39.0 / 33.5 / 31.0 / 30.7 with two texels and
// 1 / 2 / 4 / 8 rows, 34.9 with one texel and 4 rows, 36.9 with four texels.  Keeping
// the lower source row in registers for the next output row took 39.
constexpr uint32_t kRows = 4;

template <bool BILINEAR, int PER>
__global__ void __launch_bounds__(256) k_resample(const float4* __restrict__ src, uint32_t W, uint32_t H,
                                                  uint2* __restrict__ dst, uint32_t out_w, uint32_t out_h) {
  const uint32_t x0 = (blockIdx.x * blockDim.x + threadIdx.x) * PER;
  if (x0 >= out_w) return;
  // the columns' sampling positions serve every row of the block
  uint32_t xa[PER], xb[PER];
  float fx[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const float u = (__uint2float_rn(x0 + k) + 0.5f) / __uint2float_rn(out_w);
    if (BILINEAR) {
      const float px = u * __uint2float_rn(W) - 0.5f, f = floorf(px);
      const int ix = (int)f;
      fx[k] = px - f;
      xa[k] = min((uint32_t)max(ix, 0), W - 1);
      xb[k] = (uint32_t)min(max(ix + 1, 0), (int)W - 1);
    } else {
      fx[k] = 0.0f;
      xa[k] = xb[k] = min((uint32_t)floorf(u * __uint2float_rn(W)), W - 1);
    }
  }
  for (uint32_t r = 0; r < kRows; ++r) {
    const uint32_t y = blockIdx.y * kRows + r;
    if (y >= out_h) return;
    const float v = (__uint2float_rn(y) + 0.5f) / __uint2float_rn(out_h);
    uint2 out[PER];
    if (BILINEAR) {
      const float py = v * __uint2float_rn(H) - 0.5f, f = floorf(py);
      const float fy = py - f;
      const int iy = (int)f;
      const size_t ya = (size_t)min((uint32_t)max(iy, 0), H - 1) * W;
      const size_t yb = (size_t)min(max(iy + 1, 0), (int)H - 1) * W;
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const float4 a = src[ya + xa[k]], b = src[ya + xb[k]], cc = src[yb + xa[k]], d = src[yb + xb[k]];
        const float w00 = (1.0f - fx[k]) * (1.0f - fy), w10 = fx[k] * (1.0f - fy), w01 = (1.0f - fx[k]) * fy,
                    w11 = fx[k] * fy;
        float4 c;
        c.x = ((a.x * w00 + b.x * w10) + cc.x * w01) + d.x * w11;
        c.y = ((a.y * w00 + b.y * w10) + cc.y * w01) + d.y * w11;
        c.z = ((a.z * w00 + b.z * w10) + cc.z * w01) + d.z * w11;
        c.w = ((a.w * w00 + b.w * w10) + cc.w * w01) + d.w * w11;
        out[k] = pack_half4(c);
      }
    } else {
      const size_t row = (size_t)min((uint32_t)floorf(v * __uint2float_rn(H)), H - 1) * W;
#pragma unroll
      for (int k = 0; k < PER; ++k) out[k] = pack_half4(src[row + xa[k]]);
    }
    uint2* o = dst + (size_t)y * out_w + x0;
    if (PER == 2) *reinterpret_cast<uint4*>(o) = make_uint4(out[0].x, out[0].y, out[PER - 1].x, out[PER - 1].y);
    else o[0] = out[0];
  }
}

}  // namespace

cudaError_t launch_resample(const float4* src, uint32_t W, uint32_t H, void* dst, uint32_t out_w, uint32_t out_h,
                            uint32_t filter, cudaStream_t st) {
  if (out_w == 0 || out_h == 0) return cudaSuccess;
  uint2* d = (uint2*)dst;
  // two texels a thread where every row starts on a 16-byte boundary (31 us for 1080p ->
  // 4K, one texel a thread 34.9); an odd width or an offset destination takes one
  const bool two = out_w % 2 == 0 && ((uintptr_t)dst & 15u) == 0;
  const uint32_t per = two ? 2 : 1;
  const dim3 grid((out_w + 256 * per - 1) / (256 * per), (out_h + kRows - 1) / kRows);
  const auto k = filter == 0 ? (two ? k_resample<false, 2> : k_resample<false, 1>)
                             : (two ? k_resample<true, 2> : k_resample<true, 1>);
  k<<<grid, 256, 0, st>>>(src, W, H, d, out_w, out_h);
  return cudaGetLastError();
}

}  // namespace pt
