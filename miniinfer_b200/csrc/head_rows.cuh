// Passes over the heads of every token around the matrix-state recurrences, for bfloat16 rows that can be read four values at a
// time: what feeds a recurrence in float32, and the norm and gate of its read-outs.  A warp takes (token, head) pairs a grid apart;
// a block a token and four heads spent its time starting and ending
// (2048 tokens of 8 heads of 128, one value a lane and read against four: the delta rule's inputs 15.0 and 13.1 us; linear attention's
// inputs with decays, 1800 tokens of 16 heads, 28.5 and 19.9 - the logarithms and exponentials of the decays are most of it).  Read-outs,
// behind another kernel, unrolled with a copy of the activation a value, and as below: 1800 tokens of 16 heads 13.1 and 11.5 us, 2048 of 32 28.6
// and 21.6 (9.7 and 18.2 by the hardware's exponential and reciprocal, which round some results to the other neighbour).
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

// 1 / (1 + exp(-z)).  A call, and not a copy for every value of a lane, of which a kernel this short would mostly wait for the fetching.
static __device__ __noinline__ float4 sigmoid4(float4 z) {
  return make_float4(1.f / (1.f + expf(-z.x)), 1.f / (1.f + expf(-z.y)), 1.f / (1.f + expf(-z.z)), 1.f / (1.f + expf(-z.w)));
}

// out[t, h] = o / sqrt(mean(o^2) + eps) * norm_w * act(gate[t, h]), o = raw[t, h]: norm_w [vdim] and gate optional.  A warp
// asks for the rows of UNITS (token, head) pairs before it works on the first; heads of more than 128 values take its lanes several times.
constexpr int OUTPUT_UNITS = 2;
template <bool WIDE>      // heads of more than 128 values
static __global__ void __launch_bounds__(256)
head_output_kernel(__nv_bfloat16* __restrict__ out, int ldo, const float* __restrict__ raw, const __nv_bfloat16* __restrict__ gate, int ldg,
                   const float* __restrict__ norm_w, int T, int heads, int vdim, float eps, int gate_silu) {
  const int lane = threadIdx.x & 31, units = T * heads, step = gridDim.x * 8, j0 = 4 * lane;
  const bool first = j0 < vdim;
  const float4 one = make_float4(1.f, 1.f, 1.f, 1.f), w0 = norm_w && first ? load_row4(norm_w + j0) : one;
  grid_dependency_sync();
#pragma unroll 1
  for (int u0 = blockIdx.x * 8 + (threadIdx.x >> 5); u0 < units; u0 += OUTPUT_UNITS * step) {
    float4 o[OUTPUT_UNITS], g[OUTPUT_UNITS];
#pragma unroll
    for (int i = 0; i < OUTPUT_UNITS; ++i) {
      const int u = u0 + i * step, t = u / heads, h = u - t * heads;
      const bool in = first && u < units;
      o[i] = in ? load_row4(raw + (size_t)u * vdim + j0) : make_float4(0.f, 0.f, 0.f, 0.f);
      g[i] = in && gate ? load_row4(gate + (size_t)t * ldg + h * vdim + j0) : one;
    }
    auto write = [&](int u, int j, float4 v, float4 z, float4 w, float rstd) {
      const int t = u / heads, h = u - t * heads;
      float4 y = scaled4(v, rstd);
      y.x *= w.x; y.y *= w.y; y.z *= w.z; y.w *= w.w;
      if (gate) {
        const float4 s = sigmoid4(z);
        y.x *= gate_silu ? z.x * s.x : s.x;
        y.y *= gate_silu ? z.y * s.y : s.y;
        y.z *= gate_silu ? z.z * s.z : s.z;
        y.w *= gate_silu ? z.w * s.w : s.w;
      }
      store_row4(out + (size_t)t * ldo + h * vdim + j, y);
    };
    float ss[OUTPUT_UNITS];
#pragma unroll
    for (int i = 0; i < OUTPUT_UNITS; ++i) {
      ss[i] = fmaf(o[i].x, o[i].x, fmaf(o[i].y, o[i].y, fmaf(o[i].z, o[i].z, o[i].w * o[i].w)));
      if (WIDE && u0 + i * step < units) {
#pragma unroll 1
        for (int j = j0 + 128; j < vdim; j += 128) {
          const float4 v = load_row4(raw + (size_t)(u0 + i * step) * vdim + j);
          ss[i] = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss[i]))));
        }
      }
    }
#pragma unroll
    for (int b = 16; b > 0; b >>= 1)
#pragma unroll
      for (int i = 0; i < OUTPUT_UNITS; ++i) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], b);
#pragma unroll
    for (int i = 0; i < OUTPUT_UNITS; ++i) {
      const int u = u0 + i * step;
      if (u >= units) break;
      const float rstd = 1.f / sqrtf(ss[i] / (float)vdim + eps);
      if (first) write(u, j0, o[i], g[i], w0, rstd);
#pragma unroll 1
      for (int j = j0 + 128; WIDE && j < vdim; j += 128) {
        const int t = u / heads, h = u - t * heads;
        write(u, j, load_row4(raw + (size_t)u * vdim + j), gate ? load_row4(gate + (size_t)t * ldg + h * vdim + j) : one, norm_w ? load_row4(norm_w + j) : one, rstd);
      }
    }
  }
}

}  // namespace mi
