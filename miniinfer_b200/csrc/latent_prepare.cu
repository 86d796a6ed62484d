// Attention through a latent: what stands between the down-projections and the attention kernels.
//
// Of a token only a latent c (C values, RMS-normed with a weight) and one rotated key part shared by all heads (R
// values) are kept.  Per head the unrotated key is W_uk c and the value W_uv c, so a head's score is
//   (W_uk^T q_plain) . c + q_rot . k_rot
// and its output W_uv (sum_j p_j c_j): the keys' and values' up-projections move to the query and to the output, and
// attention runs over one shared key/value head whose key row is [c | k_rot] and whose value row is c.
//
//   latent_down:  from the fused down-projection rows - the query latent (Q values at q_off) and the key/value row
//                 (C + R values at kv_off) - the normed query latent into a buffer of its own, the normed c and the
//                 rotated k_rot into the layer's pages (key row [c | k_rot | 0], value row [c | 0]);
//   latent_query: the rotated part of every query head, rotated, into its place behind the C values that the product
//                 with W_uk fills, in the packed query rows [token, head, cache head size].
//
// Norms, angles and rotations in float32; a table row holds cos of R / 2 angles, then their sines; value i pairs
// with value i + R / 2 (halves) or 2i with 2i + 1 (interleaved): (u, v) -> (u cos - v sin, v cos + u sin).
#include "common.cuh"

namespace {

__device__ __forceinline__ float rotated(const float* x, int d, int R, int interleaved, const float* cs) {
  const int half = R / 2;
  const bool first = interleaved ? !(d & 1) : d < half;
  const int pi = interleaved ? d >> 1 : (first ? d : d - half);
  const int partner = interleaved ? d ^ 1 : (first ? d + half : d - half);
  const float c = cs[pi], s = cs[half + pi];
  return first ? x[d] * c - x[partner] * s : x[d] * c + x[partner] * s;
}

// Sums of two values over a block, in an order that depends on blockDim only.
__device__ __forceinline__ float2 block_sum2(float2 v, float2* scratch /* >= 33 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v.x = mi::warp_sum(v.x);
  v.y = mi::warp_sum(v.y);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float2 t = lane < (int)(blockDim.x >> 5) ? scratch[lane] : make_float2(0.f, 0.f);
  t.x = mi::warp_sum(t.x);
  t.y = mi::warp_sum(t.y);
  return t;
}

// Latency is all there is to a decode step's few rows: both sums of squares at once, all loads of a row on their way together
// (8 tokens, query latent of 1536: 10.0 us with one sum after the other in 128 threads, 6.5 so).  Where tokens are more than the
// multiprocessors hold at once, the bigger block only keeps others out (2048 tokens: 9.4 us at 256 threads, 6.8 at 128).  The block's
// size is part of the order in which a row's squares are added: float32 rows, whose bits must not depend on how many tokens share
// their step, have the same block in every step.
constexpr int DOWN_THREADS = 256, DOWN_FEW_TOKENS = 1024;

template <typename T>
__global__ void __launch_bounds__(DOWN_THREADS)
latent_down_kernel(const T* __restrict__ down, int ld, int q_off, int kv_off, int Q, int C, int R, int hdp,
                   const float* __restrict__ q_w, const float* __restrict__ kv_w, float eps, T* __restrict__ cq_out,
                   const float* __restrict__ rope, const int* __restrict__ positions, int interleaved,
                   const int* __restrict__ slot_mapping, T* __restrict__ kv_layer, int page_size) {
  __shared__ float2 scratch[33];
  extern __shared__ float kr[];                  // the R unrotated values of the shared key part
  const int t = blockIdx.x;
  const int pos = positions[t];
  const int slot = slot_mapping ? slot_mapping[t] : -1;
  mi::grid_dependency_sync();
  const T* row = down + (size_t)t * ld;
  float2 ss = make_float2(0.f, 0.f);
  if (cq_out) {
#pragma unroll 8
    for (int i = threadIdx.x; i < Q; i += blockDim.x) {
      const float v = mi::to_float(row[q_off + i]);
      ss.x += v * v;
    }
  }
  if (slot >= 0) {
    for (int i = threadIdx.x; i < C; i += blockDim.x) {
      const float v = mi::to_float(row[kv_off + i]);
      ss.y += v * v;
    }
    for (int i = threadIdx.x; i < R; i += blockDim.x) kr[i] = mi::to_float(row[kv_off + C + i]);
  }
  ss = block_sum2(ss, scratch);                  // its barrier also publishes kr
  if (cq_out) {
    const float rstd = 1.f / sqrtf(ss.x / (float)Q + eps);
#pragma unroll 8
    for (int i = threadIdx.x; i < Q; i += blockDim.x)
      cq_out[(size_t)t * Q + i] = mi::from_float<T>(q_w[i] * (mi::to_float(row[q_off + i]) * rstd));
  }
  if (slot < 0) return;
  const float rstd = 1.f / sqrtf(ss.y / (float)C + eps);
  const int page = slot / page_size, off = slot % page_size;
  T* krow = kv_layer + (((size_t)page * 2 + 0) * page_size + off) * hdp;
  T* vrow = kv_layer + (((size_t)page * 2 + 1) * page_size + off) * hdp;
  const float* cs = rope + (size_t)pos * R;
  for (int i = threadIdx.x; i < hdp; i += blockDim.x) {
    float kval = 0.f, vval = 0.f;
    if (i < C) kval = vval = kv_w[i] * (mi::to_float(row[kv_off + i]) * rstd);
    else if (i < C + R) kval = rotated(kr, i - C, R, interleaved, cs);
    krow[i] = mi::from_float<T>(kval);
    vrow[i] = mi::from_float<T>(vval);
  }
}

// The same for bfloat16 rows whose parts are whole 16 bytes: a thread eight values of a row - of the query latent, of c, or of the key's
// rest -, their weights and angles read before the wait, one round trip behind it.  (A value a thread, unrolled eight times: 13 KB of
// instructions that come from L2 for one row a block; 8 tokens, query latent of 1536, behind another kernel 6.8 us, so 3.1; 2048 tokens, of 384,
// 6.6 and 5.8.)
struct Eight { float v[8]; };
__device__ __forceinline__ Eight load8(const __nv_bfloat16* p) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const uint32_t part[4] = {raw.x, raw.y, raw.z, raw.w};
  Eight e;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&part[i]));
    e.v[2 * i] = f.x;
    e.v[2 * i + 1] = f.y;
  }
  return e;
}
__device__ __forceinline__ Eight load8(const float* p) {
  Eight e;
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    const float4 f = *reinterpret_cast<const float4*>(p + i);
    e.v[i] = f.x; e.v[i + 1] = f.y; e.v[i + 2] = f.z; e.v[i + 3] = f.w;
  }
  return e;
}
__device__ __forceinline__ uint4 packed8(const Eight& e) {
  uint32_t r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(e.v[2 * i], e.v[2 * i + 1]);
    r[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(r[0], r[1], r[2], r[3]);
}
// Values d .. d + 7 of R rotated ones, from x (the R values unrotated, 16-byte aligned) and the position's row of the table: R a multiple of 8,
// for halves of 16.
struct Angles { Eight c, s; };
__device__ __forceinline__ Angles angles8(const float* cs, int d, int R, int interleaved) {
  Angles a;
  if (interleaved) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a.c.v[2 * i] = a.c.v[2 * i + 1] = cs[d / 2 + i];
      a.s.v[2 * i] = a.s.v[2 * i + 1] = cs[R / 2 + d / 2 + i];
    }
  } else {
    const int pi = d < R / 2 ? d : d - R / 2;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a.c.v[i] = cs[pi + i];
      a.s.v[i] = cs[R / 2 + pi + i];
    }
  }
  return a;
}
__device__ __forceinline__ Eight rotated8(const __nv_bfloat16* x, int d, int R, int interleaved, const Angles& a) {
  const bool first = d < R / 2;
  const Eight u = load8(x + d), w = load8(x + (interleaved ? d : first ? d + R / 2 : d - R / 2));
  Eight y;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float partner = interleaved ? u.v[i ^ 1] : w.v[i];
    const bool minus = interleaved ? !(i & 1) : first;
    y.v[i] = minus ? u.v[i] * a.c.v[i] - partner * a.s.v[i] : u.v[i] * a.c.v[i] + partner * a.s.v[i];
  }
  return y;
}

__global__ void __launch_bounds__(1024)
latent_down8_kernel(const __nv_bfloat16* __restrict__ down, int ld, int q_off, int kv_off, int Q, int C, int R, int hdp,
                    const float* __restrict__ q_w, const float* __restrict__ kv_w, float eps, __nv_bfloat16* __restrict__ cq_out,
                    const float* __restrict__ rope, const int* __restrict__ positions, int interleaved,
                    const int* __restrict__ slot_mapping, __nv_bfloat16* __restrict__ kv_layer, int page_size) {
  __shared__ float2 scratch[33];
  const int t = blockIdx.x, slot = slot_mapping ? slot_mapping[t] : -1;
  // this thread's eight values: of the query latent, of c, then of the key's rest (rotated values and zeros)
  int i = 8 * threadIdx.x;
  const bool of_q = i < Q;
  if (!of_q) i -= Q;
  const bool of_c = !of_q && slot >= 0 && i < C, of_rest = !of_q && slot >= 0 && i >= C && i < hdp, turned = of_rest && i < C + R;
  Eight w;
  Angles a;
  if (of_q || of_c) w = load8((of_q ? q_w : kv_w) + i);
  if (turned) a = angles8(rope + (size_t)positions[t] * R, i - C, R, interleaved);
  mi::grid_dependency_sync();
  const __nv_bfloat16* row = down + (size_t)t * ld;
  Eight x;
#pragma unroll
  for (int e = 0; e < 8; ++e) x.v[e] = 0.f;
  if (of_q || of_c) x = load8(row + (of_q ? q_off : kv_off) + i);
  else if (turned) x = rotated8(row + kv_off + C, i - C, R, interleaved, a);
  float sum = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) sum = fmaf(x.v[e], x.v[e], sum);
  const float2 ss = block_sum2(make_float2(of_q ? sum : 0.f, of_c ? sum : 0.f), scratch);
  if (of_q || of_c) {
    const float rstd = 1.f / sqrtf((of_q ? ss.x / (float)Q : ss.y / (float)C) + eps);
#pragma unroll
    for (int e = 0; e < 8; ++e) x.v[e] = w.v[e] * (x.v[e] * rstd);
  }
  const uint4 y = packed8(x);
  if (of_q) {
    *reinterpret_cast<uint4*>(cq_out + (size_t)t * Q + i) = y;
  } else if (of_c || of_rest) {
    const int page = slot / page_size, off = slot - page * page_size;
    __nv_bfloat16* krow = kv_layer + (((size_t)page * 2 + 0) * page_size + off) * hdp + i;
    *reinterpret_cast<uint4*>(krow) = y;
    *reinterpret_cast<uint4*>(krow + (size_t)page_size * hdp) = of_c ? y : make_uint4(0u, 0u, 0u, 0u);
  }
}

// Eight values a thread of the rotated part and of the zeros behind it.  (2048 tokens of 16 heads, 32 rotated: 7.3 us a value a lane, so 2.8.)
__global__ void __launch_bounds__(256)
latent_query8_kernel(const __nv_bfloat16* __restrict__ q, int ldq, int total, int H, int D, int R, int C, int hdp, __nv_bfloat16* __restrict__ q_out,
                     const float* __restrict__ rope, const int* __restrict__ positions, int interleaved) {
  const int idx = blockIdx.x * 256 + threadIdx.x, per = (hdp - C) / 8, u = idx / per, d = 8 * (idx - u * per), t = u / H, h = u - t * H;
  if (idx >= total) {
    mi::grid_dependency_sync();
    return;
  }
  Angles a;
  if (d < R) a = angles8(rope + (size_t)positions[t] * R, d, R, interleaved);
  mi::grid_dependency_sync();
  uint4 y = make_uint4(0u, 0u, 0u, 0u);
  if (d < R) y = packed8(rotated8(q + (size_t)t * ldq + (size_t)h * (D + R) + D, d, R, interleaved, a));
  *reinterpret_cast<uint4*>(q_out + (size_t)u * hdp + C + d) = y;
}

// A warp takes (token, head) pairs a grid apart: a block a token and four heads spent its time starting and ending (2048 tokens
// of 16 / 32 heads: 11.8 / 24.3 us, 7.3 / 14.5 so).
constexpr int QUERY_WARPS = 8;

template <typename T>
__global__ void __launch_bounds__(32 * QUERY_WARPS)
latent_query_kernel(const T* __restrict__ q, int ldq, int units, int H, int D, int R, int C, int hdp, T* __restrict__ q_out,
                    const float* __restrict__ rope, const int* __restrict__ positions, int interleaved) {
  const int lane = threadIdx.x & 31, half = R / 2;
  mi::grid_dependency_sync();
#pragma unroll 2
  for (int u = blockIdx.x * QUERY_WARPS + (threadIdx.x >> 5); u < units; u += gridDim.x * QUERY_WARPS) {
    const int t = u / H, h = u - t * H;
    const float* cs = rope + (size_t)positions[t] * R;
    const T* src = q + (size_t)t * ldq + (size_t)h * (D + R) + D;
    T* dst = q_out + (size_t)u * hdp + C;
    for (int i = lane; i < hdp - C; i += 32) {
      float v = 0.f;
      if (i < R) {
        const bool first = interleaved ? !(i & 1) : i < half;
        const int pi = interleaved ? i >> 1 : (first ? i : i - half), partner = interleaved ? i ^ 1 : (first ? i + half : i - half);
        const float c = cs[pi], s = cs[half + pi], x = mi::to_float(src[i]), y = mi::to_float(src[partner]);
        v = first ? x * c - y * s : x * c + y * s;
      }
      dst[i] = mi::from_float<T>(v);
    }
  }
}

}  // namespace

MI_API int mi_latent_down(const void* down, int dtype, int ld, int q_off, int kv_off, int T, int Q, int C, int R, int hdp,
                          const float* q_w, const float* kv_w, float eps, void* cq_out, const float* rope, const int* positions,
                          int interleaved, const int* slot_mapping, void* kv_layer, int page_size, cudaStream_t stream) {
  MI_REQUIRE(T >= 0 && Q > 0 && C > 0 && R > 0 && R % 2 == 0 && hdp >= C + R, "latent_down: bad sizes Q=%d C=%d R=%d cache head size %d", Q, C, R, hdp);
  MI_REQUIRE(rope != nullptr && positions != nullptr && eps > 0.f, "latent_down: the rotation table, positions and eps are needed");
  MI_REQUIRE(slot_mapping == nullptr || (kv_layer != nullptr && page_size > 0), "latent_down: a store needs the cache layer");
  MI_REQUIRE(R * sizeof(float) <= 32 * 1024, "latent_down: rotated part of %d values is too long", R);
  if (T == 0) return 0;
  // eight values a thread: whole 16 bytes everywhere, a row in one block
  const auto aligned = [](const void* q) { return ((uintptr_t)q % 16) == 0; };
  const int threads = ((cq_out ? Q : 0) + (slot_mapping ? hdp : 0)) / 8;
  if (dtype == MI_BF16 && cq_out && Q % 8 == 0 && C % 8 == 0 && R % (interleaved ? 8 : 16) == 0 && hdp % 8 == 0 && ld % 8 == 0 && q_off % 8 == 0 && kv_off % 8 == 0 &&
      aligned(down) && aligned(q_w) && aligned(kv_w) && aligned(cq_out) && aligned(rope) && aligned(kv_layer) && threads <= 1024) {
    mi::launch(latent_down8_kernel, dim3(T), dim3((threads + 31) / 32 * 32), 0, stream, (const __nv_bfloat16*)down, ld, q_off, kv_off, Q, C, R, hdp,
               q_w, kv_w, eps, (__nv_bfloat16*)cq_out, rope, positions, interleaved, slot_mapping, (__nv_bfloat16*)kv_layer, page_size);
    MI_LAUNCH_OK("latent_down");
    return 0;
  }
  const size_t smem = (size_t)R * sizeof(float);
  const dim3 block(dtype == MI_F32 || T <= DOWN_FEW_TOKENS ? DOWN_THREADS : DOWN_THREADS / 2);
  if (dtype == MI_BF16)
    mi::launch(latent_down_kernel<__nv_bfloat16>, dim3(T), block, smem, stream, (const __nv_bfloat16*)down, ld, q_off, kv_off, Q, C, R, hdp,
               q_w, kv_w, eps, (__nv_bfloat16*)cq_out, rope, positions, interleaved, slot_mapping, (__nv_bfloat16*)kv_layer, page_size);
  else if (dtype == MI_F32)
    mi::launch(latent_down_kernel<float>, dim3(T), block, smem, stream, (const float*)down, ld, q_off, kv_off, Q, C, R, hdp,
               q_w, kv_w, eps, (float*)cq_out, rope, positions, interleaved, slot_mapping, (float*)kv_layer, page_size);
  else return mi_fail("latent_down: unknown dtype %d", dtype);
  MI_LAUNCH_OK("latent_down");
  return 0;
}

MI_API int mi_latent_query(const void* q, int dtype, int ldq, int T, int H, int D, int R, int C, int hdp, void* q_out,
                           const float* rope, const int* positions, int interleaved, cudaStream_t stream) {
  MI_REQUIRE(T >= 0 && H > 0 && D > 0 && R > 0 && R % 2 == 0 && hdp >= C + R, "latent_query: bad sizes");
  MI_REQUIRE(R * 4 * sizeof(float) <= 32 * 1024, "latent_query: rotated part of %d values is too long", R);
  if (T == 0) return 0;
  MI_REQUIRE((long long)T * H <= 1 << 30, "latent_query: %d tokens of %d heads are too many for one launch", T, H);
  const long long eights = (long long)T * H * ((hdp - C) / 8);
  if (dtype == MI_BF16 && R % (interleaved ? 8 : 16) == 0 && C % 8 == 0 && hdp % 8 == 0 && D % 8 == 0 && ldq % 8 == 0 && ((uintptr_t)q % 16) == 0 &&
      ((uintptr_t)q_out % 16) == 0 && ((uintptr_t)rope % 16) == 0 && eights <= 1 << 30) {
    mi::launch(latent_query8_kernel, dim3((unsigned)((eights + 255) / 256)), dim3(256), 0, stream, (const __nv_bfloat16*)q, ldq, (int)eights, H, D, R, C, hdp,
               (__nv_bfloat16*)q_out, rope, positions, interleaved);
    MI_LAUNCH_OK("latent_query");
    return 0;
  }
  const int units = T * H, blocks = (units + QUERY_WARPS - 1) / QUERY_WARPS, most = 8 * mi::sm_count();
  const dim3 grid(blocks < most ? blocks : most), block(32 * QUERY_WARPS);
  if (dtype == MI_BF16)
    mi::launch(latent_query_kernel<__nv_bfloat16>, grid, block, 0, stream, (const __nv_bfloat16*)q, ldq, units, H, D, R, C, hdp,
               (__nv_bfloat16*)q_out, rope, positions, interleaved);
  else if (dtype == MI_F32)
    mi::launch(latent_query_kernel<float>, grid, block, 0, stream, (const float*)q, ldq, units, H, D, R, C, hdp, (float*)q_out,
               rope, positions, interleaved);
  else return mi_fail("latent_query: unknown dtype %d", dtype);
  MI_LAUNCH_OK("latent_query");
  return 0;
}
