// Passes over the heads of every token around the matrix-state recurrences, for bfloat16 rows that can be read four values at a
// time: what feeds a recurrence in float32, and the norm and gate of its read-outs.  A warp takes (token, head) pairs a grid apart;
// a block a token and four heads spent its time starting and ending
// (2048 tokens of 8 heads of 128, one value a lane and read against four: read-outs 9.9 and 8.3 us, the delta rule's inputs 15.0 and
// 13.1; linear attention's inputs with decays, 1800 tokens of 16 heads, 28.5 and 19.9 - the logarithms and exponentials of the
// decays are most of it).
#pragma once

#include "common.cuh"

namespace mi {

__device__ __forceinline__ float4 load_row4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_row4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void store_row4(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  uint2 raw;
  raw.x = *reinterpret_cast<const uint32_t*>(&lo);
  raw.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = raw;
}
// exp(x) for x <= 0, near 1 from the difference to 1: expf errs there by parts of an ulp to one side, which thousands of tokens of
// decays near 1 add up.
__device__ __forceinline__ float decay_exp(float x) { return x > -0.5f ? 1.f + expm1f(x) : expf(x); }
__device__ __forceinline__ float4 scaled4(float4 v, float f) { return make_float4(v.x * f, v.y * f, v.z * f, v.w * f); }

// Whether rows of `values` values a head, `stride` values a token, start on the boundaries of four values everywhere.
template <typename T>
inline bool rows4(const T* p, int values, long long stride) {
  return p == nullptr || (values % 4 == 0 && stride % 4 == 0 && ((uintptr_t)p % (4 * sizeof(T))) == 0);
}
inline dim3 head_rows_grid(long long units) {
  const long long blocks = (units + 7) / 8, most = 8ll * sm_count();      // eight warps a block, one round of blocks
  return dim3((unsigned)(blocks < most ? blocks : most));
}

// out[t, h] = o / sqrt(mean(o^2) + eps) * norm_w * act(gate[t, h]), o = raw[t, h]: norm_w [vdim] and gate optional.
static __global__ void __launch_bounds__(256)
head_output_kernel(__nv_bfloat16* __restrict__ out, int ldo, const float* __restrict__ raw, const __nv_bfloat16* __restrict__ gate, int ldg,
                   const float* __restrict__ norm_w, int T, int heads, int vdim, float eps, int gate_silu) {
  const int lane = threadIdx.x & 31, units = T * heads, step = gridDim.x * 8;
  grid_dependency_sync();
#pragma unroll 2
  for (int u = blockIdx.x * 8 + (threadIdx.x >> 5); u < units; u += step) {
    const int t = u / heads, h = u - t * heads;
    const float* o = raw + (size_t)u * vdim;
    float ss = 0.f;
    for (int j = 4 * lane; j < vdim; j += 128) {
      const float4 v = load_row4(o + j);
      ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
    }
    const float rstd = 1.f / sqrtf(warp_sum(ss) / (float)vdim + eps);
    for (int j = 4 * lane; j < vdim; j += 128) {
      float4 y = scaled4(load_row4(o + j), rstd);
      if (norm_w) {
        const float4 w = load_row4(norm_w + j);
        y.x *= w.x; y.y *= w.y; y.z *= w.z; y.w *= w.w;
      }
      if (gate) {
        const float4 g = load_row4(gate + (size_t)t * ldg + h * vdim + j);
        auto act = [&](float z) { const float s = 1.f / (1.f + expf(-z)); return gate_silu ? z * s : s; };
        y.x *= act(g.x); y.y *= act(g.y); y.z *= act(g.z); y.w *= act(g.w);
      }
      store_row4(out + (size_t)t * ldo + h * vdim + j, y);
    }
  }
}

}  // namespace mi
