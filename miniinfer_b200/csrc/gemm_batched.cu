// A batch of small matrix products over strided operands, for any sizes and alignments:
//
//   out[b][m, n] = act( sum_k x[b][m, k] * w[b][n, k]  (+ bias[n]) )  (* sigmoid(row_gate[m, b]) or * sigmoid(value_gate[m, b N + n]))
//
// x[b] starts at x + b * x_batch with rows lda apart, w[b] at w + b * w_batch with rows ldw apart, out[b] at
// out + b * o_batch with rows ldo apart - so the heads of a token's row (a batch stride of one head, a row stride of
// the whole row) are multiplied with a matrix per head without being repacked, and a column range of a row can be
// an operand.  Products and sums in float32, whatever the storage type - k ascending but for bfloat16 results on the tensor
// cores, which add up sixteen products at a time -: a row's result does not depend on the other rows.  act: 0 none, 1 softplus (log(1 + exp(z)), z itself above 20).  row_gate: one logit per
// (row, batch) at row_gate[m * gate_stride + b]; the output rows of batch b are multiplied with its sigmoid.  value_gate: one
// logit per output value instead, at value_gate[m * gate_stride + b * N + n].
//
// This is the product of per-head up- and down-projections of a latent attention, of the 32-bit path for batches of them and
// for rows whose values do not lie side by side, and the fallback of the bfloat16 path for inner sizes that are no multiple of 8.
// The general kernel: tiles of 64 x 64 through shared memory, 16 values of k at a time, 4 x 4 outputs a thread.
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16;

struct BatchedArgs {
  const void* x; const void* w; void* out;
  long long x_batch, w_batch, o_batch;
  int lda, ldw, ldo;
  int M, N, K;
  const float* bias;
  int act;
  const void* row_gate;
  int gate_stride;
  const void* value_gate;      // one logit per output value: row m at m * gate_stride, batch b's N values from column b * N on
  int w_fixed;                 // no kernel that may still be running writes w
};

template <typename T, typename TO>
__global__ void __launch_bounds__(256)
gemm_batched_kernel(BatchedArgs a) {
  mi::grid_dependency_sync();
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int b = blockIdx.z;
  const T* x = (const T*)a.x + (size_t)b * a.x_batch;
  const T* w = (const T*)a.w + (size_t)b * a.w_batch;
  TO* out = (TO*)a.out + (size_t)b * a.o_batch;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < a.K; k0 += BK) {
    for (int idx = threadIdx.x; idx < BM * BK; idx += 256) {
      const int r = idx / BK, c = idx % BK;
      const int m = m0 + r, k = k0 + c;
      xs[c][r] = (m < a.M && k < a.K) ? mi::to_float(x[(size_t)m * a.lda + k]) : 0.f;
      const int n = n0 + r;
      ws[c][r] = (n < a.N && k < a.K) ? mi::to_float(w[(size_t)n * a.ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < BK; ++c) {
      float xv[4], wv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) xv[i] = xs[c][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) wv[j] = ws[c][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= a.M) continue;
    float gate = 1.f;
    if (a.row_gate) gate = 1.f / (1.f + expf(-mi::to_float(((const T*)a.row_gate)[(size_t)m * a.gate_stride + b])));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= a.N) continue;
      float y = acc[i][j];
      if (a.bias) y += a.bias[n];
      if (a.act == 1) y = y > 20.f ? y : log1pf(expf(y));
      if (a.value_gate) y *= 1.f / (1.f + expf(-mi::to_float(((const T*)a.value_gate)[(size_t)m * a.gate_stride + (size_t)b * a.N + n])));
      out[(size_t)m * a.ldo + n] = mi::from_float<TO>(y * gate);
    }
  }
}

// Few rows (a decode step) in bfloat16: the tiled kernel would wait for global memory once per 16 values of k with one
// block a tile.  Here a warp takes one output column (batch, n): its lanes deal out k, every lane multiplies its values of
// the weight row with up to 16 rows of x, and the lanes' sums meet by shuffles.  The sum's order differs from the tiled
// kernel's, so the 32-bit path, whose results must not depend on how a request was cut, does not take this kernel.
constexpr int FEW_ROWS = 16;

template <typename TO>
__global__ void __launch_bounds__(128)
gemm_batched_few_rows_kernel(BatchedArgs a) {
  mi::grid_dependency_sync();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * 4 + warp;
  const int b = blockIdx.y;
  if (n >= a.N) return;
  const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + (size_t)b * a.x_batch;
  const __nv_bfloat16* w = (const __nv_bfloat16*)a.w + (size_t)b * a.w_batch + (size_t)n * a.ldw;
  float acc[FEW_ROWS];
#pragma unroll
  for (int m = 0; m < FEW_ROWS; ++m) acc[m] = 0.f;
  for (int k = lane; k < a.K; k += 32) {
    const float wv = __bfloat162float(w[k]);
#pragma unroll
    for (int m = 0; m < FEW_ROWS; ++m)
      if (m < a.M) acc[m] = fmaf(__bfloat162float(x[(size_t)m * a.lda + k]), wv, acc[m]);
  }
  TO* out = (TO*)a.out + (size_t)b * a.o_batch;
#pragma unroll
  for (int m = 0; m < FEW_ROWS; ++m) {
    if (m >= a.M) break;
    float y = mi::warp_sum(acc[m]);
    if (lane == 0) {
      if (a.bias) y += a.bias[n];
      if (a.act == 1) y = y > 20.f ? y : log1pf(expf(y));
      if (a.row_gate) y *= 1.f / (1.f + expf(-__bfloat162float(((const __nv_bfloat16*)a.row_gate)[(size_t)m * a.gate_stride + b])));
      if (a.value_gate) y *= 1.f / (1.f + expf(-__bfloat162float(((const __nv_bfloat16*)a.value_gate)[(size_t)m * a.gate_stride + (size_t)b * a.N + n])));
      out[(size_t)m * a.ldo + n] = mi::from_float<TO>(y);
    }
  }
}

// The same on the tensor cores (mma.sync), where the values of k can be fetched in pairs: a warp takes eight output columns
// of a batch and the whole of K, straight from global memory, so all of its loads are in flight together.  EIGHT: rows of whole 16
// bytes are fetched so, a thread of a quad eight values of k that two products share, in the same order for both operands, and fixed
// weights before the wait for the kernel before (with the weights behind it: 8 tokens of 32 heads, the two products of a layer, 0.6 us more).  GATES: with an activation or a gate a value; without them
// their code is not there to be jumped across (8 rows of 32 heads, 192 x 128 and 128 x 192, behind other kernels: 4.0 us each, so 3.4).
__device__ __forceinline__ uint32_t pair_at(const __nv_bfloat16* p, bool take) { return take ? *reinterpret_cast<const uint32_t*>(p) : 0u; }
__device__ __forceinline__ uint4 eight_at(const __nv_bfloat16* p, bool take) { return take ? *reinterpret_cast<const uint4*>(p) : make_uint4(0u, 0u, 0u, 0u); }
__device__ __forceinline__ void mma_onto(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t w0, uint32_t w1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(w0), "r"(w1));
}

template <typename TO, bool EIGHT, bool GATES>
__global__ void __launch_bounds__(128)
gemm_batched_mma_few_rows_kernel(BatchedArgs a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3, q = t * 2;
  const int n0 = (blockIdx.x * 4 + warp) * 8;
  const int b = blockIdx.y;
  const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + (size_t)b * a.x_batch;
  const __nv_bfloat16* w = (const __nv_bfloat16*)a.w + (size_t)b * a.w_batch + (size_t)min(n0 + g, a.N - 1) * a.ldw;
  const bool lo = g < a.M, hi = g + 8 < a.M;
  const __nv_bfloat16* x0 = x + (size_t)(lo ? g : 0) * a.lda;
  const __nv_bfloat16* x1 = x + (size_t)(hi ? g + 8 : 0) * a.lda;
  float c[4] = {0.f, 0.f, 0.f, 0.f};
  if constexpr (EIGHT) {
    constexpr int AHEAD = 8;      // 256 values of k
    uint4 wv[AHEAD];
    auto weights = [&](int k0) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) wv[i] = eight_at(w + k0 + 32 * i + 8 * t, k0 + 32 * i + 8 * t < a.K);
    };
    if (!a.w_fixed) mi::grid_dependency_sync();
    weights(0);
    if (a.w_fixed) mi::grid_dependency_sync();
#pragma unroll 1
    for (int k0 = 0; k0 < a.K; k0 += 32 * AHEAD) {
      if (k0 > 0) weights(k0);
      uint4 xa[AHEAD], xb[AHEAD];
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const int k = k0 + 32 * i + 8 * t;
        xa[i] = eight_at(x0 + k, lo && k < a.K);
        xb[i] = eight_at(x1 + k, hi && k < a.K);
      }
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        mma_onto(c, xa[i].x, xb[i].x, xa[i].y, xb[i].y, wv[i].x, wv[i].y);
        mma_onto(c, xa[i].z, xb[i].z, xa[i].w, xb[i].w, wv[i].z, wv[i].w);
      }
    }
    if (n0 >= a.N) return;
  } else {
    mi::grid_dependency_sync();
    if (n0 >= a.N) return;
#pragma unroll 8
    for (int k = 0; k < a.K; k += 16) {
      const int ka = k + q, kb = ka + 8;
      const bool ia = ka < a.K, ib = kb < a.K;
      mma_onto(c, pair_at(x0 + ka, ia && lo), pair_at(x1 + ka, ia && hi), pair_at(x0 + kb, ib && lo), pair_at(x1 + kb, ib && hi), pair_at(w + ka, ia), pair_at(w + kb, ib));
    }
  }
  TO* out = (TO*)a.out + (size_t)b * a.o_batch;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int m = g + 8 * h;
    if (m >= a.M) break;
    const float gate = a.row_gate ? 1.f / (1.f + expf(-__bfloat162float(((const __nv_bfloat16*)a.row_gate)[(size_t)m * a.gate_stride + b]))) : 1.f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int n = n0 + q + e;
      if (n >= a.N) continue;
      float y = c[2 * h + e];
      if (GATES) {
        if (a.bias) y += a.bias[n];
        if (a.act == 1) y = y > 20.f ? y : log1pf(expf(y));
        if (a.value_gate) y *= 1.f / (1.f + expf(-__bfloat162float(((const __nv_bfloat16*)a.value_gate)[(size_t)m * a.gate_stride + (size_t)b * a.N + n])));
      }
      out[(size_t)m * a.ldo + n] = mi::from_float<TO>(y * gate);
    }
  }
}

// Many rows in bfloat16 on the tensor cores (mma.sync), for operands whose rows can be fetched 16 bytes at a time: tiles of 64 x 64, a
// warp 32 x 32, K in stages of 64 by cp.async.  These products are small and read their rows once - 2048 rows of 16 heads,
// 64 x 192 each, move 17 MB - so the memory bounds them, where the FMA kernel above was bound by its arithmetic (50.6 us);
// a tcgen05 tile of 128 rows would wait for the same bytes.  The tensor core cuts off what its accumulator does not
// hold, always towards zero: every sixteen products start from zero and are added to the sum in a rounded addition.  bfloat16
// results only: in float32 the sums of sixteen would still err by more than the chain of FMAs (K = 4096, carried on in the
// accumulator: 4.4e-6 of the norm, by FMAs 6.1e-7).
constexpr int TK = 64, LDS = TK + 8, TSTAGES = 3, LDC = 64 + 4;

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

__global__ void __launch_bounds__(128)
gemm_batched_mma_kernel(BatchedArgs a) {
  extern __shared__ __align__(16) __nv_bfloat16 tiles[];      // [TSTAGES][x rows, w rows][64][LDS]
  const int b = blockIdx.z, m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
  const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + (size_t)b * a.x_batch;
  const __nv_bfloat16* w = (const __nv_bfloat16*)a.w + (size_t)b * a.w_batch;
  const int steps = (a.K + TK - 1) / TK;
  auto stage = [&](int s, bool weights) {
    if (s < steps) {
      __nv_bfloat16* dst = tiles + ((s % TSTAGES) * 2 + (weights ? 1 : 0)) * 64 * LDS;
#pragma unroll
      for (int i = threadIdx.x; i < 64 * TK / 8; i += 128) {
        const int r = i / (TK / 8), k = s * TK + i % (TK / 8) * 8, row = (weights ? n0 : m0) + r;
        const bool in = row < (weights ? a.N : a.M) && k < a.K;
        const __nv_bfloat16* src = weights ? w + (in ? (size_t)row * a.ldw + k : 0) : x + (in ? (size_t)row * a.lda + k : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * LDS + i % (TK / 8) * 8)),
                     "l"(src), "r"(in ? 16 : 0) : "memory");
      }
    }
    if (!weights) asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int s = 0; s < TSTAGES - 1; ++s) stage(s, true);      // the weights are written by no kernel: fetched before the wait
  mi::grid_dependency_sync();
  for (int s = 0; s < TSTAGES - 1; ++s) stage(s, false);
  float c[2][4][4] = {};
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(TSTAGES - 2) : "memory");
    __syncthreads();
    stage(s + TSTAGES - 1, true);
    stage(s + TSTAGES - 1, false);
    const __nv_bfloat16 *xs = tiles + (s % TSTAGES) * 2 * 64 * LDS, *ws = xs + 64 * LDS;
#pragma unroll
    for (int k = 0; k < TK; k += 16) {
      uint32_t xa[2][4], wb[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) ldmatrix4(xa[i], xs + (wm + 16 * i + (lane & 15)) * LDS + k + (lane >> 4) * 8);
#pragma unroll
      for (int j = 0; j < 2; ++j) ldmatrix4(wb[j], ws + (wn + 16 * j + (lane & 7) + (lane >> 4) * 8) * LDS + k + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float p[4];
          asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                       : "=f"(p[0]), "=f"(p[1]), "=f"(p[2]), "=f"(p[3])
                       : "r"(xa[i][0]), "r"(xa[i][1]), "r"(xa[i][2]), "r"(xa[i][3]), "r"(wb[j >> 1][(j & 1) * 2]), "r"(wb[j >> 1][(j & 1) * 2 + 1]),
                         "f"(0.f));
#pragma unroll
          for (int e = 0; e < 4; ++e) c[i][j][e] += p[e];
        }
    }
  }
  // Through shared memory, so that one loop serves all values of a thread and rows are written 16 bytes at a time.  Value by value from the
  // registers the activation and the gates stood there 32 times, 110 KB of instructions that nearly all calls only jump across, line by
  // line from L2: 2048 rows of 16 heads, 64 x 192, behind another kernel 16.8 us, so 9.7; 500 rows of 32 heads, 128 x 192, 18 and 9.2.
  float* cs = reinterpret_cast<float*>(tiles);      // [64][LDC]
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float2*>(cs + (wm + 16 * i + (lane >> 2) + 8 * h) * LDC + wn + 8 * j + (lane & 3) * 2) = make_float2(c[i][j][2 * h], c[i][j][2 * h + 1]);
  __syncthreads();
  if (a.bias || a.act || a.value_gate) {
#pragma unroll 1
    for (int i = threadIdx.x; i < 64 * 64; i += 128) {
      const int r = i >> 6, m = m0 + r, n = n0 + (i & 63);
      if (m >= a.M || n >= a.N) continue;
      float y = cs[r * LDC + (i & 63)];
      if (a.bias) y += a.bias[n];
      if (a.act == 1) y = y > 20.f ? y : log1pf(expf(y));
      if (a.value_gate) y *= 1.f / (1.f + expf(-__bfloat162float(((const __nv_bfloat16*)a.value_gate)[(size_t)m * a.gate_stride + (size_t)b * a.N + n])));
      cs[r * LDC + (i & 63)] = y;
    }
    __syncthreads();
  }
  __nv_bfloat16* out = (__nv_bfloat16*)a.out + (size_t)b * a.o_batch;
#pragma unroll 1
  for (int i = threadIdx.x; i < 64 * 8; i += 128) {
    const int r = i >> 3, m = m0 + r, n = n0 + (i & 7) * 8;
    if (m >= a.M || n >= a.N) continue;
    const float gate = a.row_gate ? 1.f / (1.f + expf(-__bfloat162float(((const __nv_bfloat16*)a.row_gate)[(size_t)m * a.gate_stride + b]))) : 1.f;
    const float* y = cs + r * LDC + (i & 7) * 8;
    __nv_bfloat16* o = out + (size_t)m * a.ldo + n;
    if (n + 8 <= a.N && ((uintptr_t)o % 16) == 0) {
      __nv_bfloat162 v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = __floats2bfloat162_rn(y[2 * e] * gate, y[2 * e + 1] * gate);
      *reinterpret_cast<uint4*>(o) = *reinterpret_cast<const uint4*>(v);
    } else {
#pragma unroll 1
      for (int e = 0; e < 8 && n + e < a.N; ++e) o[e] = __float2bfloat16_rn(y[e] * gate);
    }
  }
}

}  // namespace

MI_API int mi_gemm_batched_few_rows(void* out, int out_dtype, const void* x, const void* w, int dtype, int batch, int M, int N, int K,
                                    int lda, long long x_batch, int ldw, long long w_batch, int ldo, long long o_batch,
                                    const float* bias, int act, const void* row_gate, int gate_stride, const void* value_gate, int w_fixed, cudaStream_t stream) {
  MI_REQUIRE(batch > 0 && batch <= 65535 && M >= 0 && M <= FEW_ROWS && N > 0 && K > 0, "gemm_batched_few_rows: bad sizes batch=%d M=%d N=%d K=%d", batch, M, N, K);
  MI_REQUIRE(dtype == MI_BF16 && lda >= K && ldw >= K && ldo >= N && (act == 0 || act == 1), "gemm_batched_few_rows: bfloat16 operands, rows that do not overlap");
  if (M == 0) return 0;
  BatchedArgs a;
  a.x = x; a.w = w; a.out = out; a.x_batch = x_batch; a.w_batch = w_batch; a.o_batch = o_batch;
  a.lda = lda; a.ldw = ldw; a.ldo = ldo; a.M = M; a.N = N; a.K = K; a.bias = bias; a.act = act;
  a.row_gate = row_gate; a.gate_stride = gate_stride; a.value_gate = value_gate; a.w_fixed = w_fixed;
  const bool pairs = K % 2 == 0 && lda % 2 == 0 && ldw % 2 == 0 && x_batch % 2 == 0 && w_batch % 2 == 0 && ((uintptr_t)x % 4) == 0 && ((uintptr_t)w % 4) == 0;
  if (pairs && (out_dtype == MI_BF16 || out_dtype == MI_F32)) {
    const dim3 mgrid((N + 31) / 32, batch);
    const bool eight = K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && x_batch % 8 == 0 && w_batch % 8 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0;
    const bool gates = bias || act || value_gate;
#define MI_FEW(TO)                                                                                                                     \
  mi::launch(eight ? gates ? gemm_batched_mma_few_rows_kernel<TO, true, true> : gemm_batched_mma_few_rows_kernel<TO, true, false>       \
                   : gates ? gemm_batched_mma_few_rows_kernel<TO, false, true> : gemm_batched_mma_few_rows_kernel<TO, false, false>,    \
             mgrid, dim3(128), 0, stream, a)
    if (out_dtype == MI_BF16) MI_FEW(__nv_bfloat16);
    else MI_FEW(float);
#undef MI_FEW
    MI_LAUNCH_OK("gemm_batched_few_rows");
    return 0;
  }
  dim3 grid((N + 3) / 4, batch);
  if (out_dtype == MI_BF16) mi::launch(gemm_batched_few_rows_kernel<__nv_bfloat16>, grid, dim3(128), 0, stream, a);
  else if (out_dtype == MI_F32) mi::launch(gemm_batched_few_rows_kernel<float>, grid, dim3(128), 0, stream, a);
  else return mi_fail("gemm_batched_few_rows: unknown output dtype %d", out_dtype);
  MI_LAUNCH_OK("gemm_batched_few_rows");
  return 0;
}

MI_API int mi_gemm_batched(void* out, int out_dtype, const void* x, const void* w, int dtype, int batch, int M, int N, int K,
                           int lda, long long x_batch, int ldw, long long w_batch, int ldo, long long o_batch,
                           const float* bias, int act, const void* row_gate, int gate_stride, const void* value_gate, cudaStream_t stream) {
  MI_REQUIRE(batch > 0 && batch <= 65535 && M >= 0 && N > 0 && K > 0, "gemm_batched: bad sizes batch=%d M=%d N=%d K=%d", batch, M, N, K);
  MI_REQUIRE(lda >= K && ldw >= K && ldo >= N, "gemm_batched: rows overlap (lda=%d ldw=%d ldo=%d)", lda, ldw, ldo);
  MI_REQUIRE(act == 0 || act == 1, "gemm_batched: unknown activation %d", act);
  MI_REQUIRE(row_gate == nullptr || value_gate == nullptr, "gemm_batched: a gate a row or a gate a value, not both");
  if (M == 0) return 0;
  BatchedArgs a;
  a.x = x; a.w = w; a.out = out; a.x_batch = x_batch; a.w_batch = w_batch; a.o_batch = o_batch;
  a.lda = lda; a.ldw = ldw; a.ldo = ldo; a.M = M; a.N = N; a.K = K; a.bias = bias; a.act = act;
  a.row_gate = row_gate; a.gate_stride = gate_stride; a.value_gate = value_gate;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
  MI_REQUIRE(grid.y <= 65535, "gemm_batched: M=%d is too large for one launch", M);
  // rows that start on 16-byte boundaries and hold whole 16 bytes; the others keep the FMA kernel
  const bool whole = dtype == MI_BF16 && out_dtype == MI_BF16 && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && x_batch % 8 == 0 && w_batch % 8 == 0 &&
                     ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0;
  if (whole) {
    constexpr size_t smem = (size_t)TSTAGES * 2 * 64 * LDS * sizeof(__nv_bfloat16);
    if (cudaFuncSetAttribute(gemm_batched_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return mi_fail("gemm_batched: %zu bytes of shared memory were refused", smem);
    mi::launch(gemm_batched_mma_kernel, grid, dim3(128), smem, stream, a);
    MI_LAUNCH_OK("gemm_batched");
    return 0;
  }
  if (dtype == MI_F32 && out_dtype == MI_F32) mi::launch(gemm_batched_kernel<float, float>, grid, dim3(256), 0, stream, a);
  else if (dtype == MI_BF16 && out_dtype == MI_BF16) mi::launch(gemm_batched_kernel<__nv_bfloat16, __nv_bfloat16>, grid, dim3(256), 0, stream, a);
  else if (dtype == MI_BF16 && out_dtype == MI_F32) mi::launch(gemm_batched_kernel<__nv_bfloat16, float>, grid, dim3(256), 0, stream, a);
  else return mi_fail("gemm_batched: unsupported dtypes operands=%d out=%d", dtype, out_dtype);
  MI_LAUNCH_OK("gemm_batched");
  return 0;
}

namespace {
// x[m, i] *= sigmoid(gate[m, i]) over bfloat16 rows, 8 values a thread where the rows are 16-byte aligned.
template <int V>
__global__ void __launch_bounds__(256)
sigmoid_gate_kernel(__nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ gate, long long ldg, int N, size_t total) {
  mi::grid_dependency_sync();
  const int per_row = N / V;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const size_t m = idx / per_row;
    const int i = (int)(idx - m * per_row) * V;
    __nv_bfloat16* xp = x + m * ldx + i;
    const __nv_bfloat16* gp = gate + m * ldg + i;
    if (V == 8) {
      uint4 xv = *reinterpret_cast<const uint4*>(xp);
      const uint4 gv = *reinterpret_cast<const uint4*>(gp);
      __nv_bfloat162* xs = reinterpret_cast<__nv_bfloat162*>(&xv);
      const __nv_bfloat162* gs = reinterpret_cast<const __nv_bfloat162*>(&gv);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 a = __bfloat1622float2(xs[k]), g = __bfloat1622float2(gs[k]);
        xs[k] = __floats2bfloat162_rn(__fdividef(a.x, 1.f + __expf(-g.x)), __fdividef(a.y, 1.f + __expf(-g.y)));
      }
      *reinterpret_cast<uint4*>(xp) = xv;
    } else {
      *xp = __float2bfloat16_rn(__fdividef(__bfloat162float(*xp), 1.f + __expf(-__bfloat162float(*gp))));
    }
  }
}
}  // namespace

// x [M, N] *= sigmoid(gate [M, N]), bfloat16, in place; rows ldx and ldg values apart.
MI_API int mi_sigmoid_gate_bf16(void* x, long long ldx, const void* gate, long long ldg, int M, int N, cudaStream_t stream) {
  MI_REQUIRE(M >= 0 && N > 0 && ldx >= N && ldg >= N, "sigmoid_gate: bad sizes M=%d N=%d", M, N);
  if (M == 0) return 0;
  const bool vec = N % 8 == 0 && ldx % 8 == 0 && ldg % 8 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)gate % 16) == 0;
  const size_t total = (size_t)M * N / (vec ? 8 : 1), want = (total + 255) / 256, most = (size_t)mi::sm_count() * 16;
  const dim3 grid((unsigned)(want < most ? want : most));
  if (vec) mi::launch(sigmoid_gate_kernel<8>, grid, dim3(256), 0, stream, (__nv_bfloat16*)x, ldx, (const __nv_bfloat16*)gate, ldg, N, total);
  else mi::launch(sigmoid_gate_kernel<1>, grid, dim3(256), 0, stream, (__nv_bfloat16*)x, ldx, (const __nv_bfloat16*)gate, ldg, N, total);
  MI_LAUNCH_OK("sigmoid_gate");
  return 0;
}
