// Recurrences with a matrix state [dim, vdim] a head that decays, a chunk of 64 tokens at a time: the gated delta rule and
// linear attention, with one decay a key channel, a head, or a constant a head.
//
// With g_t the decays of a token, one a key channel (all equal where a head has one), P_t the product of g over the chunk up
// to and with token t, S_0 the state a chunk starts from, and rows k_t, q_t, v_t, the recurrence
//   S_t = diag(g_t) S_(t-1) + k_t u_t^T,   o_t = S_t^T q_t,   u_t = beta_t (v_t - (diag(g_t) S_(t-1))^T k_t)   (delta rule) or v_t
// is, over a chunk,
//   (I + L) U = diag(beta) (V - K~ S_0),   L[t, s] = beta_t sum_d k_t k_s (P_t / P_s)  for s < t,   K~_t = P_t k_t
//   O = Q~ S_0 + A U,                      A[t, s] = sum_d q_t k_s (P_t / P_s)         for s <= t,  Q~_t = P_t q_t
//   S_C = diag(P_C) S_0 + K^^T U,          K^_s = (P_C / P_s) k_s.
// The triangular system does not need the state if its right side is kept in two parts, U = U0 - W S_0 with
// U0 = (I + L)^-1 diag(beta) V and W = (I + L)^-1 diag(beta) K~.  A ratio P_t / P_s is never formed as a quotient: it is the
// product of the decays between the two tokens, each in 0 .. 1, so nothing overflows and a decay of zero is just that.
// Tokens go in blocks of eight.  With F_t the product from the start of t's block to t, E_s the one from behind s to the
// end of its block and B_b a block's whole product, P_t / P_s = F_t B_(I-1) .. B_(J+1) E_s for t in block I and s in an earlier
// block J; inside a block the product is walked.  Three kernels:
//   chunk_build  a block per (chunk, head), all at once: A, L, the inverse of I + L, W, U0, K^ and Q~;
//   chunk_state  a block per (request, head, group of value columns), the only one that walks the chunks in order: keeps S in
//                registers, leaves every chunk's S_0, U = U0 - W S_0 and the state behind the last chunk;
//   chunk_out    a block per (chunk, head, 64 value columns), all at once: O, written over the values.
// Chunks are counted over the items of at least min_tokens new tokens, in their order; a step whose chunks need more
// scratch than SLAB_FLOATS is worked through in slabs, the state row carrying over.
//
// Every product runs on the tensor cores (mma.sync m16n8k8) with each float32 operand as the sum of two tf32 numbers and
// three of the four partial products, added up in float32: as FMAs they were bound by the reads of shared memory that
// feed them.  tcgen05 has no use here: the chain of chunks is latency, and its operands are made in registers.  Against
// float64 the state errs, in parts of its norm, after 2048 tokens of 8 heads of 128 x 128 (in brackets what did these steps before:
// the walk in stretches, and for the delta rule with one decay a head chunks of FMAs): delta rule, decays a channel about 1 / 50 a
// token 1.9e-7 (3.5e-7), 1 / 3000 3.2e-7 (3.4e-6), stronger than 1 / 2 1.4e-7 (0.7e-7); a head 1.6e-7 (2.4e-7), 2.3e-7 (4.2e-7), 1.3e-7
// (0.9e-7); linear attention 1.3e-7 (1.7e-7), 4.7e-7 (1.3e-5), 0.65e-7 (0.3e-7).
// Measured on B200, one request of 2048 tokens, 8 / 16 / 32 heads of 128 x 128, the whole operation in microseconds: delta rule with
// one decay a key channel 193, 284, 494 (in stretches 1017, 1204, 1254), one a head 188, 270, 473 (chunks of FMAs 208, 296, 586), linear
// attention 126, 188, 345 (in stretches 173, 281, 476).
#include "chunked_state.cuh"

namespace mi {
namespace {

constexpr int C = CHUNK_TOKENS;
constexpr long long SLAB_FLOATS = 72ll << 20;      // 288 MiB: 87 chunks of 16 heads of 128 x 128 (delta rule)
constexpr int THREADS = 256;
constexpr int OB = 64;                 // value columns of a chunk_out block
constexpr int VT = 128;                // value columns that chunk_build takes at a time
constexpr int NB = C / 8;              // blocks of eight tokens

__host__ __device__ inline int pad(int x, int m) { return (x + m - 1) / m * m; }

struct Args : ChunkedStateArgs {
  int dp, vp;                          // dim padded to 32, vdim padded to 32
  // per (chunk, head): W [C][dp] and U0 / U [C][vp] (delta rule), A [C][C], K^ and Q~ [C][dp], S_0 [dp][vp], P_C and what its rounding leaves [2][dp]
  float *w, *u, *at, *kh, *qt, *s0, *pc;
  int c0, c1;                          // the slab's chunks
};

__host__ __device__ inline long long unit_floats(int dp, int vp, bool delta) {
  return (delta ? (long long)C * (dp + vp) : 0) + C * C + 2ll * C * dp + (long long)dp * vp + 2 * dp;
}

// The item that chunk number c (over the items that are long enough) belongs to and the chunk's place in it; item -1: none.
__device__ __forceinline__ void find_chunk(const Args& a, int c, int& item, int& place) {
  item = -1;
  for (int b = 0; b < a.items; ++b) {
    const int n = a.q_len[b];
    if (n < a.min_tokens) continue;
    const int nc = (n + C - 1) / C;
    if (c < nc) { item = b; place = c; return; }
    c -= nc;
  }
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st2(float* p, float x, float y) { *reinterpret_cast<float2*>(p) = make_float2(x, y); }
__device__ __forceinline__ void copy16(float* dst, const float* src, bool take) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = take ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_begun() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------------------------------------------------ products

// A float32 number as the sum of two tf32 ones, the upper rounded to nearest in the integer unit: three plain instructions, where
// two conversions cost the state kernel twice the instructions (of 1600 a warp and chunk, 110 us for 32 chunks).  The lower part
// keeps bits that the tensor core does not look at: at most one of its twelve, so cutting it off errs as much as rounding it.
// Rounding it in the integer unit is not open: the sum would carry a NaN of all ones, which is what arithmetic returns, into a
// zero - as it does in the upper part, where the lower one remains a NaN.
struct Two {
  uint32_t hi, lo;
  __device__ __forceinline__ Two() {}
  __device__ __forceinline__ explicit Two(float x) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
  }
};
// Whether some lane of the warp holds a number that is not finite.  A tile's product with a triangular matrix multiplies the zeros
// behind the diagonal too, and zero times such a number is a NaN in rows of earlier tokens: the warp then adds up its elements
// one by one, up to the diagonal.
template <int N>
__device__ __forceinline__ bool any_not_finite(const float (&v)[N]) {
  bool bad = false;
#pragma unroll
  for (int i = 0; i < N; ++i) bad |= !(fabsf(v[i]) <= 3.402823466e38f);
  return __any_sync(0xffffffffu, bad);
}
__device__ __forceinline__ void mma1(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// A sum of products in two parts: the products of the upper parts of the operands, and those with a lower part, which are 2^-11 of them.
struct Sum {
  float c[4], small[4];
  __device__ __forceinline__ Sum() {
#pragma unroll
    for (int e = 0; e < 4; ++e) c[e] = small[e] = 0.f;
  }
  __device__ __forceinline__ float at(int e) const { return c[e] + small[e]; }
};
// s += a b for a 16 x 8 operand (rows g and g + 8, columns t and t + 4) and an 8 x 8 one (rows t and t + 4, column g), g = lane / 4,
// t = lane % 4; s: row g columns 2 t and 2 t + 1, then row g + 8.  The tensor core cuts its accumulator off towards zero at every
// product, so only the small products are carried on in it: eight products of upper parts - 22 bits each, exact - start from zero and
// join the sum in a rounded addition.  (All carried on, read-outs of 2048 tokens erred by 1.1e-6 of their norm; so by 2.6e-7, and the walk
// in order by 2.5e-7.  The fourth product costs 10 % and takes 2 % off that.)
__device__ __forceinline__ void mma3(Sum& s, const Two (&a)[4], const Two (&b)[2]) {
  const float zero[4] = {0.f, 0.f, 0.f, 0.f};
  float p[4];
  mma1(s.small, a[0].lo, a[1].lo, a[2].lo, a[3].lo, b[0].hi, b[1].hi, s.small);
  mma1(s.small, a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].lo, b[1].lo, s.small);
  mma1(p, a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].hi, b[1].hi, zero);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    s.c[e] += p[e];
  }
}
// The 16 x 8 operand of a row-major tile.
__device__ __forceinline__ void load_a(Two (&a)[4], const float* p, int ld, int g, int t) {
  a[0] = Two(p[g * ld + t]);
  a[1] = Two(p[(g + 8) * ld + t]);
  a[2] = Two(p[g * ld + t + 4]);
  a[3] = Two(p[(g + 8) * ld + t + 4]);
}
// The same with two values a read: the inner index runs 0 2 4 6 1 3 5 7, so the 8 x 8 operand beside it has rows 2 t and 2 t + 1.
__device__ __forceinline__ void load_a_pairs(Two (&a)[4], const float* p, int ld, int g, int t) {
  const float2 x = *reinterpret_cast<const float2*>(p + g * ld + 2 * t), y = *reinterpret_cast<const float2*>(p + (g + 8) * ld + 2 * t);
  a[0] = Two(x.x);
  a[1] = Two(y.x);
  a[2] = Two(x.y);
  a[3] = Two(y.y);
}
// The transpose of a row-major 8 x 16 tile, rows 2 g and 2 g + 1 in the places of g and g + 8.
__device__ __forceinline__ void load_a_transposed(Two (&a)[4], const float* p, int ld, int g, int t) {
  const float2 x = *reinterpret_cast<const float2*>(p + t * ld + 2 * g), y = *reinterpret_cast<const float2*>(p + (t + 4) * ld + 2 * g);
  a[0] = Two(x.x);
  a[1] = Two(x.y);
  a[2] = Two(y.x);
  a[3] = Two(y.y);
}
__device__ __forceinline__ void load_b(Two (&b)[2], const float* p, int ld, int g, int t) {
  b[0] = Two(p[t * ld + g]);
  b[1] = Two(p[(t + 4) * ld + g]);
}
// Rows r0 and r1 of a tile of numbers already in two parts.
__device__ __forceinline__ void load_b(Two (&b)[2], const uint2* p, int ld, int g, int r0, int r1) {
  const uint2 x = p[r0 * ld + g], y = p[r1 * ld + g];
  b[0].hi = x.x; b[0].lo = x.y;
  b[1].hi = y.x; b[1].lo = y.y;
}

// -------------------------------------------------------------------------------------------------------------- build

constexpr int LDT = C + 4;             // a row of the inverse
struct BuildLayout {                   // float offsets
  int ld, k, q, g, total, diag, beta, rest, f, floats;
  __host__ __device__ explicit BuildLayout(int dp) {
    ld = dp + 4;
    k = 0;                                                            // [C][ld] keys; E k; then the values, VT columns at a time
    q = k + C * (dp > VT ? ld : VT + 4);                              // [C][ld] queries; F q; then L^T [C][C] and the inverse [C][LDT]
    g = q + (C * ld > C * C + C * LDT ? C * ld : C * C + C * LDT);    // [C][ld] decays; F k; then diag(beta) K~
    total = g + C * ld;                                               // [NB][dp] a block's whole product
    diag = total + NB * dp;                                           // [NB][64] products inside a block: 36 of q, 28 of k
    beta = diag + NB * 64;                                            // [C]
    rest = beta + C;                                                  // [NB][dp] one decay a channel: what the rounding of the block's product leaves
    f = rest + NB * dp;                                               // one decay a head: F [C], E [C], a block's product [NB], as doubles [NB]
    floats = f + 2 * C + 3 * NB;
  }
};

// Sums 64 values over the 32 lanes; lane l ends with the sums number 2 l and 2 l + 1 in v[0] and v[1].
__device__ __forceinline__ void reduce_scatter(float (&v)[64], int lane) {
#pragma unroll
  for (int n = 32, bit = 16; n >= 2; n /= 2, bit /= 2) {
    const bool upper = lane & bit;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if (i >= n) break;
      const float keep = upper ? v[i + n] : v[i], send = upper ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
}

template <bool DELTA>
__global__ void __launch_bounds__(THREADS, 2)
chunk_build_kernel(Args a) {
  extern __shared__ __align__(16) float sm[];
  const BuildLayout at(a.dp);
  const int ld = at.ld, dp = a.dp;
  float *ks = sm + at.k, *qs = sm + at.q, *gs = sm + at.g, *total = sm + at.total, *bt = sm + at.beta;
  __shared__ int found[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, head = blockIdx.y;
  if (tid == 0) find_chunk(a, a.c0 + blockIdx.x, found[0], found[1]);
  mi::grid_dependency_sync();
  __syncthreads();
  const int item = found[0];
  if (item < 0) return;
  const int first = found[1] * C, n = min(C, a.q_len[item] - first), row0 = a.q_start[item] + first;
  const int kvh = head / (a.heads / a.qk_heads);
  const size_t unit = (size_t)blockIdx.x * a.heads + head;
  {      // tokens behind the last and channels behind the last: zero keys and queries, decays of one
    const int per_row = dp / 4, rows = THREADS / per_row, t0 = tid / per_row, d = (tid - t0 * per_row) * 4;
#pragma unroll 4
    for (int t = t0; t < C && t0 < rows; t += rows) {
      const bool in = t < n && d < a.dim;
      const size_t from = in ? ((size_t)(row0 + t) * a.qk_heads + kvh) * a.dim + d : 0;
      copy16(ks + t * ld + d, a.kn + from, in);
      copy16(qs + t * ld + d, a.qn + from, in);
      float4 x = make_float4(1.f, 1.f, 1.f, 1.f);
      if (in) {
        if (a.decay == CHUNK_DECAY_CHANNEL) {
          x = ld4(a.g + ((size_t)(row0 + t) * a.heads + head) * a.dim + d);
        } else {
          const float y = a.decay == CHUNK_DECAY_HEAD ? expf(a.g[(size_t)(row0 + t) * a.heads + head]) : a.g[head];
          x = make_float4(y, y, y, y);
        }
      }
      st4(gs + t * ld + d, x);
    }
    if (DELTA && tid < C) bt[tid] = tid < n ? a.beta[(size_t)(row0 + tid) * a.heads + head] : 0.f;
  }
  copies_begun();
  // One decay a head: F, E and the blocks' products are sums of logarithms (a constant's: products) in double, rounded once.  A constant's
  // float products err alike in every chunk, and logarithms of decays near one hold digits that the decays do not.
  const bool per_head = a.decay != CHUNK_DECAY_CHANNEL, logs = a.decay == CHUNK_DECAY_HEAD;
  float* fs = sm + at.f;
  double* whole = reinterpret_cast<double*>(fs + 2 * C + NB);
  if (per_head && tid < NB) {
    double x[8], sum = logs ? 0. : 1.;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int t = 8 * tid + j;
      x[j] = t >= n ? sum : (double)a.g[logs ? (size_t)(row0 + t) * a.heads + head : head];
    }
    double f = sum;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      f = logs ? f + x[j] : f * x[j];
      fs[8 * tid + j] = logs ? expf((float)f) : (float)f;
    }
    whole[tid] = f;
    fs[2 * C + tid] = logs ? expf((float)f) : (float)f;
#pragma unroll
    for (int j = 7; j >= 0; --j) {
      fs[C + 8 * tid + j] = logs ? expf((float)sum) : (float)sum;
      sum = logs ? sum + x[j] : sum * x[j];
    }
  }
  copies_done<0>();
  __syncthreads();

  // Inside the blocks, a warp a block of eight tokens and a lane four key channels: products number p (p + 1) / 2 + s of q_p and
  // k_s for s <= p, then 36 + p (p - 1) / 2 + s of k_p and k_s for s < p, the decays between s and p walked.
  {
    float v[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = 0.f;
    if (4 * lane < dp) {
      const float* kr = ks + warp * 8 * ld + 4 * lane;
      const float *qr = qs + warp * 8 * ld + 4 * lane, *gr = gs + warp * 8 * ld + 4 * lane;
      float4 key[8];      // key s times the decays from behind s to the token at hand
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const float4 kp = ld4(kr + p * ld), qp = ld4(qr + p * ld), gp = ld4(gr + p * ld);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          if (s < p) {
            key[s].x *= gp.x; key[s].y *= gp.y; key[s].z *= gp.z; key[s].w *= gp.w;
            v[36 + p * (p - 1) / 2 + s] = fmaf(kp.x, key[s].x, fmaf(kp.y, key[s].y, fmaf(kp.z, key[s].z, kp.w * key[s].w)));
            v[p * (p + 1) / 2 + s] = fmaf(qp.x, key[s].x, fmaf(qp.y, key[s].y, fmaf(qp.z, key[s].z, qp.w * key[s].w)));
          }
        }
        key[p] = kp;
        v[p * (p + 1) / 2 + p] = fmaf(qp.x, kp.x, fmaf(qp.y, kp.y, fmaf(qp.z, kp.z, qp.w * kp.w)));
      }
    }
    reduce_scatter(v, lane);
    st2(sm + at.diag + warp * 64 + 2 * lane, v[0], v[1]);
  }
  __syncthreads();
  // E k, F q and F k over the keys, queries and decays, a thread eight tokens of a block in a channel
  for (int i = tid; i < NB * dp; i += THREADS) {
    const int b = i / dp, d = i % dp;
    float gv[8], kv[8], f = 1.f, rest = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) { gv[j] = gs[(8 * b + j) * ld + d]; kv[j] = ks[(8 * b + j) * ld + d]; }
    if (per_head) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        qs[(8 * b + j) * ld + d] *= fs[8 * b + j];
        gs[(8 * b + j) * ld + d] = fs[8 * b + j] * kv[j];
        ks[(8 * b + j) * ld + d] = fs[C + 8 * b + j] * kv[j];
      }
      total[b * dp + d] = fs[2 * C + b];
      continue;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float before = f;
      f *= gv[j];
      rest = fmaf(rest, gv[j], fmaf(before, gv[j], -f));
      qs[(8 * b + j) * ld + d] *= f;
      gs[(8 * b + j) * ld + d] = f * kv[j];
    }
    total[b * dp + d] = f;
    sm[at.rest + b * dp + d] = rest;
    f = 1.f;
#pragma unroll
    for (int j = 7; j >= 0; --j) {
      ks[(8 * b + j) * ld + d] = f * kv[j];
      f *= gv[j];
    }
  }
  __syncthreads();
  // Between blocks: warp I has the rows of its block - eight of F k above eight of F q - and every earlier block's E k, times the
  // products of the blocks between
  Sum acc[NB - 1];
  if (warp == 0 && per_head) {      // P_C and what its rounding leaves
    double p = logs ? 0. : 1.;
#pragma unroll
    for (int b = 0; b < NB; ++b) p = logs ? p + whole[b] : p * whole[b];
    if (logs) p = exp(p);
    const float high = (float)p, low = (float)(p - (double)high);
    for (int d = lane; d < dp; d += 32) {
      a.pc[unit * 2 * dp + d] = high;
      a.pc[unit * 2 * dp + dp + d] = low;
    }
  }
  if (warp > 0) {
    const float *fk = gs + (8 * warp + g) * ld, *fq = qs + (8 * warp + g) * ld;
    for (int d = 0; d < dp; d += 8) {
      Two x[4];
      x[0] = Two(fk[d + t4]);
      x[1] = Two(fq[d + t4]);
      x[2] = Two(fk[d + t4 + 4]);
      x[3] = Two(fq[d + t4 + 4]);
      float p0 = 1.f, p1 = 1.f;
#pragma unroll
      for (int j = NB - 2; j >= 0; --j) {
        if (j < warp) {
          if (j + 1 < warp) { p0 *= total[(j + 1) * dp + d + t4]; p1 *= total[(j + 1) * dp + d + t4 + 4]; }
          const float* ek = ks + (8 * j + g) * ld + d + t4;
          Two y[2];
          y[0] = Two(ek[0] * p0);
          y[1] = Two(ek[4] * p1);
          mma3(acc[j], x, y);
        }
      }
    }
  }
  // A, a row a token: zeros behind the diagonal
  {
    float* out = a.at + unit * C * C + (size_t)(8 * warp + g) * C + 2 * t4;
    const float* dq = sm + at.diag + warp * 64 + g * (g + 1) / 2;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      float x = 0.f, y = 0.f;
      if (j < warp) { x = acc[j < NB - 1 ? j : 0].at(2); y = acc[j < NB - 1 ? j : 0].at(3); }
      if (j == warp) {
        x = 2 * t4 <= g ? dq[2 * t4] : 0.f;
        y = 2 * t4 + 1 <= g ? dq[2 * t4 + 1] : 0.f;
      }
      st2(out + 8 * j, x, y);
    }
  }
  // K^ and Q~, and F k becomes diag(beta) K~
  for (int i = tid; i < NB * dp; i += THREADS) {
    const int b = i / dp, d = i % dp;
    float before = 1.f, behind = 1.f;
    for (int j = 0; j < b; ++j) before *= total[j * dp + d];
    for (int j = NB - 1; j > b; --j) behind *= total[j * dp + d];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int t = 8 * b + j;
      a.kh[(unit * C + t) * dp + d] = ks[t * ld + d] * behind;
      a.qt[(unit * C + t) * dp + d] = qs[t * ld + d] * before;
    }
    if (b == NB - 1 && !per_head) {
      double p = 1.;
      for (int j = 0; j < NB; ++j) p *= (double)total[j * dp + d] + (double)sm[at.rest + j * dp + d];
      a.pc[unit * 2 * dp + d] = (float)p;
      a.pc[unit * 2 * dp + dp + d] = (float)(p - (double)(float)p);
    }
  }
  if (!DELTA) return;
  __syncthreads();
  for (int i = tid; i < NB * dp; i += THREADS) {      // (a loop of its own: the warps above still read F k)
    const int b = i / dp, d = i % dp;
    float before = 1.f;
    for (int j = 0; j < b; ++j) before *= total[j * dp + d];
#pragma unroll
    for (int j = 0; j < 8; ++j) gs[(8 * b + j) * ld + d] *= bt[8 * b + j] * before;
  }
  auto fetch_values = [&](int v0) {
    for (int i = tid; i < C * VT / 4; i += THREADS) {
      const int t = i / (VT / 4), c = v0 + (i % (VT / 4)) * 4;
      const bool in = t < n && c < a.vdim;
      copy16(ks + t * (VT + 4) + c - v0, a.raw + (in ? (size_t)(row0 + t) * (a.heads * a.vdim) + head * a.vdim + c : 0), in);
    }
    copies_begun();
  };
  fetch_values(0);
  float *lt = qs, *inv = qs + C * C;
  {      // L^T, the part before the diagonal
    const int t = 8 * warp + g;
    const float* dk = sm + at.diag + warp * 64 + 36 + g * (g - 1) / 2;
#pragma unroll
    for (int j = 0; j < NB - 1; ++j) {
      if (j < warp) {
        lt[(8 * j + 2 * t4) * C + t] = bt[t] * acc[j].at(0);
        lt[(8 * j + 2 * t4 + 1) * C + t] = bt[t] * acc[j].at(1);
      }
    }
    if (2 * t4 < g) lt[(8 * warp + 2 * t4) * C + t] = bt[t] * dk[2 * t4];
    if (2 * t4 + 1 < g) lt[(8 * warp + 2 * t4 + 1) * C + t] = bt[t] * dk[2 * t4 + 1];
  }
  __syncthreads();
  // The inverse of I + L in halves of 32 tokens, [[A, 0], [B, D]]^-1 = [[A^-1, 0], [-D^-1 (B A^-1), D^-1]]: A and D by substitution, a
  // thread a column - an unknown that is final is taken off all later rows -, the rest as two products.  (One substitution over
  // 64 rows kept two warps busy and six waiting for a quarter of the kernel.)
  constexpr int HALF = C / 2;
  if (tid < C) {
    const int h0 = tid & HALF, col = tid - h0;
    float x[HALF];
#pragma unroll
    for (int t = 0; t < HALF; ++t) x[t] = t == col ? 1.f : 0.f;
#pragma unroll
    for (int s = 0; s < HALF - 1; ++s) {
#pragma unroll
      for (int q = (s + 1) / 4 * 4; q < HALF; q += 4) {
        const float4 l = ld4(lt + (h0 + s) * C + h0 + q);
        if (q > s) x[q] = fmaf(-l.x, x[s], x[q]);
        if (q + 1 > s) x[q + 1] = fmaf(-l.y, x[s], x[q + 1]);
        if (q + 2 > s) x[q + 2] = fmaf(-l.z, x[s], x[q + 2]);
        if (q + 3 > s) x[q + 3] = fmaf(-l.w, x[s], x[q + 3]);
      }
    }
#pragma unroll
    for (int t = 0; t < HALF; ++t) {
      inv[(h0 + t) * LDT + tid] = x[t];
      if (h0 == 0) inv[t * LDT + HALF + tid] = 0.f;
    }
  }
  __syncthreads();
  {
    const int m = (warp & 1) * 16, c = (warp >> 1) * 8;      // a warp 16 rows x 8 columns of the 32 x 32
    Sum ba;
#pragma unroll
    for (int k = 0; k < HALF; k += 8) {      // B A^-1, B being L's lower half (kept transposed)
      Two l[4], r[2];
      const float* p = lt + (k + t4) * C + HALF + m + g;
      l[0] = Two(p[0]);
      l[1] = Two(p[8]);
      l[2] = Two(p[4 * C]);
      l[3] = Two(p[4 * C + 8]);
      load_b(r, inv + k * LDT + c, LDT, g, t4);
      mma3(ba, l, r);
    }
    st2(inv + (HALF + m + g) * LDT + c + 2 * t4, ba.at(0), ba.at(1));
    st2(inv + (HALF + m + g + 8) * LDT + c + 2 * t4, ba.at(2), ba.at(3));
    __syncthreads();
    Sum dba;
#pragma unroll
    for (int k = 0; k < HALF; k += 8) {
      Two l[4], r[2];
      load_a(l, inv + (HALF + m) * LDT + HALF + k, LDT, g, t4);
      load_b(r, inv + (HALF + k) * LDT + c, LDT, g, t4);
      mma3(dba, l, r);
    }
    float x[4] = {dba.at(0), dba.at(1), dba.at(2), dba.at(3)};
    if (any_not_finite(x)) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = m + g + 8 * (e >> 1), col = c + 2 * t4 + (e & 1);
        x[e] = 0.f;
        for (int k = 0; k <= row; ++k) x[e] = fmaf(inv[(HALF + row) * LDT + HALF + k], inv[(HALF + k) * LDT + col], x[e]);
      }
    }
    __syncthreads();
    st2(inv + (HALF + m + g) * LDT + c + 2 * t4, -x[0], -x[1]);
    st2(inv + (HALF + m + g + 8) * LDT + c + 2 * t4, -x[2], -x[3]);
  }
  copies_done<0>();
  __syncthreads();
  // W and U0: a warp 16 rows (warp % 4) of every other group of 32 columns
  auto multiply = [&](const float* right, int ldr, int columns, const float* scale, float* out, int ldo) {
    const int m0 = (warp & 3) * 16;
    for (int n0 = (warp >> 2) * 32; n0 < columns; n0 += 64) {
      Sum sum[4];
      for (int k = 0; k < m0 + 16; k += 8) {      // (the inverse is zero behind its diagonal)
        Two x[4];
        load_a(x, inv + m0 * LDT + k, LDT, g, t4);
        const float s0 = scale ? scale[k + t4] : 1.f, s1 = scale ? scale[k + t4 + 4] : 1.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          Two y[2];
          y[0] = Two(right[(k + t4) * ldr + n0 + 8 * j + g] * s0);
          y[1] = Two(right[(k + t4 + 4) * ldr + n0 + 8 * j + g] * s1);
          mma3(sum[j], x, y);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float c[4] = {sum[j].at(0), sum[j].at(1), sum[j].at(2), sum[j].at(3)};
        if (any_not_finite(c)) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = m0 + g + 8 * (e >> 1), col = n0 + 8 * j + 2 * t4 + (e & 1);
            c[e] = 0.f;
            for (int k = 0; k <= t; ++k) c[e] = fmaf(inv[t * LDT + k], right[k * ldr + col] * (scale ? scale[k] : 1.f), c[e]);
          }
        }
        st2(out + (size_t)(m0 + g) * ldo + n0 + 8 * j + 2 * t4, c[0], c[1]);
        st2(out + (size_t)(m0 + g + 8) * ldo + n0 + 8 * j + 2 * t4, c[2], c[3]);
      }
    }
  };
  multiply(gs, ld, dp, nullptr, a.w + unit * C * dp, dp);
  for (int v0 = 0; v0 < a.vp; v0 += VT) {
    if (v0 > 0) {
      __syncthreads();
      fetch_values(v0);
      copies_done<0>();
      __syncthreads();
    }
    multiply(ks, VT + 4, min(VT, a.vp - v0), bt, a.u + unit * C * a.vp + v0, a.vp);
  }
}

// -------------------------------------------------------------------------------------------------------------- state

template <int CB>                      // value columns of a block
struct StateLayout {                   // float offsets
  // rows of S and U in two parts: strides at which the reads of a half warp, two rows apart (S) or one (U), fall into different banks
  static constexpr int LDU = CB + 8, LDS2 = CB + 2, LDU2 = CB + 4;
  int ld, k, u, p, stage, s2, u2, floats;
  __host__ __device__ StateLayout(int dp, bool delta) {
    ld = dp + 8;
    k = delta ? C * ld : 0;            // a stage: W [C][ld], K^ [C][ld], U0 or V [C][LDU], P_C [2][dp]
    u = k + C * ld;
    p = u + C * LDU;
    stage = p + 2 * dp;
    s2 = 2 * stage;                    // [dp][LDS2] pairs, [C][LDU2] pairs
    u2 = s2 + (delta ? 2 * dp * LDS2 : 0);
    floats = u2 + 2 * C * LDU2;
  }
};

template <int CB, bool DELTA>
__global__ void __launch_bounds__(THREADS, 1)
chunk_state_kernel(Args a) {
  using L = StateLayout<CB>;
  constexpr int LDU = L::LDU, LDS2 = L::LDS2, LDU2 = L::LDU2, NT = CB / 8;
  extern __shared__ __align__(16) float sm[];
  const L at(a.dp, DELTA);
  const int dp = a.dp, ld = at.ld, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int head = blockIdx.x, v0 = blockIdx.y * CB, item = blockIdx.z;
  const int n_new = a.q_len[item], row0 = a.q_start[item], slot = a.seq_slot[item];
  if (n_new < a.min_tokens) return;
  int base = 0;                        // the number of this item's first chunk
  for (int b = 0; b < item; ++b)
    if (a.q_len[b] >= a.min_tokens) base += (a.q_len[b] + C - 1) / C;
  const int from = max(a.c0, base), to = min(a.c1, base + (n_new + C - 1) / C);
  if (from >= to) return;
  uint2 *s2 = reinterpret_cast<uint2*>(sm + at.s2), *u2 = reinterpret_cast<uint2*>(sm + at.u2);
  mi::grid_dependency_sync();
  // which 16 bytes of a row of W and K^ this thread copies, of every k_rows-th row
  const int per_row = dp / 4, k_rows = THREADS / per_row, kt = tid / per_row, kd = (tid - kt * per_row) * 4;
  auto fetch = [&](int c, float* buf) {
    const size_t unit = (size_t)(c - a.c0) * a.heads + head;
    if (kt < k_rows) {
      const size_t from_row = (unit * C + kt) * dp + kd;
#pragma unroll 8
      for (int t = kt; t < C; t += k_rows) {
        if (DELTA) copy16(buf + t * ld + kd, a.w + from_row + (size_t)(t - kt) * dp, true);
        copy16(buf + at.k + t * ld + kd, a.kh + from_row + (size_t)(t - kt) * dp, true);
      }
    }
    const int first = (c - base) * C, n = min(C, n_new - first);
#pragma unroll
    for (int i = tid; i < C * CB / 4; i += THREADS) {
      const int t = i / (CB / 4), col = (i % (CB / 4)) * 4;
      if (DELTA) {
        copy16(buf + at.u + t * LDU + col, a.u + (unit * C + t) * a.vp + v0 + col, true);
      } else {
        const bool in = t < n && v0 + col < a.vdim;
        copy16(buf + at.u + t * LDU + col, a.raw + (in ? (size_t)(row0 + first + t) * (a.heads * a.vdim) + head * a.vdim + v0 + col : 0), in);
      }
    }
    if (tid < dp / 2) copy16(buf + at.p + 4 * tid, a.pc + unit * 2 * dp + 4 * tid, true);
    copies_begun();
  };
  fetch(from, sm);
  // this warp's rows of S: 16 key channels - a lane those numbered 2 g and 2 g + 1 -, all columns of the block
  const int d0 = 16 * warp + 2 * g;
  const bool holds = 16 * warp < dp;
  float* st = a.state + (size_t)slot * a.state_stride + (size_t)head * a.dim * a.vdim;
  float S[NT][4];
  auto keep = [&]() {
    if (DELTA && holds) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const Two x(S[j][2 * h]), y(S[j][2 * h + 1]);
          *reinterpret_cast<uint4*>(s2 + (d0 + h) * LDS2 + 8 * j + 2 * t4) = make_uint4(x.hi, x.lo, y.hi, y.lo);
        }
    }
  };
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1), c = v0 + 8 * j + 2 * t4 + (e & 1);
      S[j][e] = (holds && d < a.dim && c < a.vdim) ? st[(size_t)d * a.vdim + c] : 0.f;
    }
  keep();
  for (int c = from; c < to; ++c) {
    const float* cur = sm + ((c - from) & 1) * at.stage;
    const size_t unit = (size_t)(c - a.c0) * a.heads + head;
    if (c + 1 < to) {
      fetch(c + 1, sm + ((c + 1 - from) & 1) * at.stage);
      copies_done<1>();
    } else {
      copies_done<0>();
    }
    __syncthreads();
    if (holds) {
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) st2(a.s0 + (unit * dp + d0 + h) * a.vp + v0 + 8 * j + 2 * t4, S[j][2 * h], S[j][2 * h + 1]);
    }
    if (DELTA) {      // U = U0 - W S_0: a warp 16 tokens, half of the columns
      constexpr int HT = NT / 2;
      const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * (CB / 2);
      Sum x[HT];
#pragma unroll 4
      for (int k = 0; k < dp; k += 8) {
        Two w[4];
        load_a_pairs(w, cur + m0 * ld + k, ld, g, t4);
#pragma unroll
        for (int j = 0; j < HT; ++j) {
          Two s[2];
          load_b(s, s2 + k * LDS2 + n0 + 8 * j, LDS2, g, 2 * t4, 2 * t4 + 1);
          mma3(x[j], w, s);
        }
      }
#pragma unroll
      for (int j = 0; j < HT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int t = m0 + g + 8 * h, col = n0 + 8 * j + 2 * t4;
          const float2 u0 = *reinterpret_cast<const float2*>(cur + at.u + t * LDU + col);
          const float y0 = u0.x - x[j].at(2 * h), y1 = u0.y - x[j].at(2 * h + 1);
          st2(a.u + (unit * C + t) * a.vp + v0 + col, y0, y1);
          const Two p(y0), q(y1);
          *reinterpret_cast<uint4*>(u2 + t * LDU2 + col) = make_uint4(p.hi, p.lo, q.hi, q.lo);
        }
    } else {
#pragma unroll
      for (int i = tid; i < C * CB; i += THREADS) {
        const Two p(cur[at.u + i / CB * LDU + i % CB]);
        u2[i / CB * LDU2 + i % CB] = make_uint2(p.hi, p.lo);
      }
    }
    __syncthreads();
    if (holds) {      // S = diag(P_C) S_0 + K^^T U
      Sum more[NT];
#pragma unroll
      for (int k = 0; k < C; k += 8) {
        Two x[4];
        load_a_transposed(x, cur + at.k + k * ld + 16 * warp, ld, g, t4);
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          Two y[2];
          load_b(y, u2 + k * LDU2 + 8 * j, LDU2, g, t4, t4 + 4);
          mma3(more[j], x, y);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {      // (P_C in two parts: products of decays near one are all rounded to the same side, a constant's to the same value)
        const float p = cur[at.p + d0 + h], p_low = cur[at.p + dp + d0 + h];
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 2 * h; e < 2 * h + 2; ++e) {
            const float low = S[j][e] * p_low;
            S[j][e] = fmaf(S[j][e], p, more[j].at(e) + (fabsf(low) <= 3.402823466e38f ? low : 0.f));      // (an infinite state stays one)
          }
      }
      keep();
    }
    __syncthreads();      // everyone is done with this stage before the fetch after next fills it
  }
  if (holds) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = d0 + (e >> 1), c = v0 + 8 * j + 2 * t4 + (e & 1);
        if (d < a.dim && c < a.vdim) st[(size_t)d * a.vdim + c] = S[j][e];
      }
  }
}

// -------------------------------------------------------------------------------------------------------------- out

constexpr int LDA = C + 8, LDV = OB + 4, OUT_THREADS = 128;
__host__ __device__ inline size_t out_smem(int dp) { return (size_t)(C * (dp + 8) + C * LDA + dp * LDV + C * LDV) * sizeof(float); }

// A warp 32 tokens x 32 columns: four operand halves split in two parts serve 24 products; with 16 x 32 a warp the splitting took
// half of the instructions.
template <bool DELTA>
__global__ void __launch_bounds__(OUT_THREADS)
chunk_out_kernel(Args a) {
  extern __shared__ __align__(16) float sm[];
  const int dp = a.dp, ldq = dp + 8;
  float *qt = sm, *aa = qt + C * ldq, *s0 = aa + C * LDA, *us = s0 + dp * LDV;
  __shared__ int found[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, head = blockIdx.y, v0 = blockIdx.z * OB;
  if (tid == 0) find_chunk(a, a.c0 + blockIdx.x, found[0], found[1]);
  mi::grid_dependency_sync();
  __syncthreads();
  const int item = found[0];
  if (item < 0) return;
  const int first = found[1] * C, n = min(C, a.q_len[item] - first), row0 = a.q_start[item] + first;
  const size_t unit = (size_t)blockIdx.x * a.heads + head;
  {
    const int per_row = dp / 4, rows = OUT_THREADS / per_row, t0 = tid / per_row, d = (tid - t0 * per_row) * 4;
#pragma unroll 4
    for (int t = t0; t < C && t0 < rows; t += rows) copy16(qt + t * ldq + d, a.qt + (unit * C + t) * dp + d, true);
  }
#pragma unroll 4
  for (int i = tid; i < dp * (OB / 4); i += OUT_THREADS) {
    const int d = i / (OB / 4), c = (i % (OB / 4)) * 4;
    const bool in = v0 + c < a.vp;
    copy16(s0 + d * LDV + c, a.s0 + (in ? (unit * dp + d) * a.vp + v0 + c : 0), in);
  }
  copies_begun();
#pragma unroll 4
  for (int i = tid; i < C * (C / 4); i += OUT_THREADS) {
    const int t = i / (C / 4), s = (i % (C / 4)) * 4;
    copy16(aa + t * LDA + s, a.at + (unit * C + t) * C + s, true);
  }
#pragma unroll 4
  for (int i = tid; i < C * (OB / 4); i += OUT_THREADS) {
    const int t = i / (OB / 4), c = (i % (OB / 4)) * 4;
    const bool in = DELTA ? v0 + c < a.vp : t < n && v0 + c < a.vdim;
    const float* from = DELTA ? a.u + (in ? (unit * C + t) * a.vp + v0 + c : 0)
                              : a.raw + (in ? (size_t)(row0 + t) * (a.heads * a.vdim) + head * a.vdim + v0 + c : 0);
    copy16(us + t * LDV + c, from, in);
  }
  copies_begun();
  const int m0 = (warp & 1) * 32, n0 = (warp >> 1) * 32;
  Sum sum[2][4];
  auto multiply = [&](const float* left, int ldl, const float* right, int k) {      // eight inner values, in the order 0 2 4 6 1 3 5 7
    Two x[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) load_a_pairs(x[i], left + (m0 + 16 * i) * ldl + k, ldl, g, t4);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float* r = right + (k + 2 * t4) * LDV + n0 + 8 * j + g;
      Two y[2];
      y[0] = Two(r[0]);
      y[1] = Two(r[LDV]);
#pragma unroll
      for (int i = 0; i < 2; ++i) mma3(sum[i][j], x[i], y);
    }
  };
  copies_done<1>();
  __syncthreads();
#pragma unroll 2
  for (int k = 0; k < dp; k += 8) multiply(qt, ldq, s0, k);      // Q~ S_0
  copies_done<0>();
  __syncthreads();
#pragma unroll 2
  for (int k = 0; k < m0 + 32; k += 8) multiply(aa, LDA, us, k);      // A U: nothing behind the diagonal
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = sum[i][j].at(e);
      if (any_not_finite(acc[i][j])) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = m0 + 16 * i + g + 8 * (e >> 1), c = n0 + 8 * j + 2 * t4 + (e & 1);
          float y = 0.f, z = 0.f;
          for (int d = 0; d < a.dim; ++d) y = fmaf(qt[t * ldq + d], s0[d * LDV + c], y);
          for (int s = 0; s <= t; ++s) z = fmaf(aa[t * LDA + s], us[s * LDV + c], z);
          acc[i][j][e] = fabsf(z) <= 3.402823466e38f ? y + z : NAN;      // an infinite value: the recurrence adds it up over channels of both signs
        }
      }
    }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = m0 + 16 * i + g + 8 * h, c = v0 + n0 + 8 * j + 2 * t4;
        if (t < n && c < a.vdim) st2(a.raw + (size_t)(row0 + t) * (a.heads * a.vdim) + head * a.vdim + c, acc[i][j][2 * h], acc[i][j][2 * h + 1]);
      }
}

int most_chunks(int T, int items) { return T / C + items; }      // every item's last chunk may be a short one
int slab_chunks(int heads, int dim, int vdim, bool delta) {
  const long long n = SLAB_FLOATS / (heads * unit_floats(pad(dim, 32), pad(vdim, 32), delta));
  return n < 1 ? 1 : n < 65535 ? (int)n : 65535;
}

template <typename K>
bool allow(K kernel, size_t smem) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess; }

}  // namespace

long long chunked_state_scratch_floats(int T, int items, int heads, int dim, int vdim, bool delta) {
  const int slab = slab_chunks(heads, dim, vdim, delta);
  const long long chunks = most_chunks(T, items) < slab ? most_chunks(T, items) : slab;
  return chunks * heads * unit_floats(pad(dim, 32), pad(vdim, 32), delta);
}

int chunked_state_slabs(int T, int items, int heads, int dim, int vdim, bool delta) {
  const int slab = slab_chunks(heads, dim, vdim, delta);
  return (most_chunks(T, items) + slab - 1) / slab;
}

int chunked_state_run(const ChunkedStateArgs& in, int T, float* scratch, cudaStream_t stream) {
  MI_REQUIRE(chunked_state_takes(in.dim, in.vdim) && in.min_tokens > 0 && in.heads % in.qk_heads == 0,
             "chunked_state: dim=%d (a multiple of 4 up to %d), vdim=%d (a multiple of 4)", in.dim, CHUNK_MAX_DIM, in.vdim);
  MI_REQUIRE(((uintptr_t)scratch % 16) == 0 && ((uintptr_t)in.qn % 16) == 0 && ((uintptr_t)in.kn % 16) == 0 && ((uintptr_t)in.raw % 16) == 0 &&
             (in.decay != CHUNK_DECAY_CHANNEL || ((uintptr_t)in.g % 16) == 0), "chunked_state: buffers must be 16-byte aligned");
  const bool delta = in.beta != nullptr;
  Args a;
  static_cast<ChunkedStateArgs&>(a) = in;
  a.dp = pad(in.dim, 32);
  a.vp = pad(in.vdim, 32);
  const int total = most_chunks(T, in.items), most = slab_chunks(in.heads, in.dim, in.vdim, delta), slab = total < most ? total : most;
  const size_t units = (size_t)slab * in.heads;
  a.w = scratch;
  a.u = a.w + (delta ? units * C * a.dp : 0);
  a.at = a.u + (delta ? units * C * a.vp : 0);
  a.kh = a.at + units * C * C;
  a.qt = a.kh + units * C * a.dp;
  a.s0 = a.qt + units * C * a.dp;
  a.pc = a.s0 + units * a.dp * a.vp;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !configured[dev]) {
    const size_t build = BuildLayout(CHUNK_MAX_DIM).floats * sizeof(float), out = out_smem(CHUNK_MAX_DIM);
    if (!allow(chunk_build_kernel<true>, build) || !allow(chunk_build_kernel<false>, build) || !allow(chunk_out_kernel<true>, out) ||
        !allow(chunk_out_kernel<false>, out) || !allow(chunk_state_kernel<16, true>, StateLayout<16>(CHUNK_MAX_DIM, true).floats * sizeof(float)) ||
        !allow(chunk_state_kernel<32, true>, StateLayout<32>(CHUNK_MAX_DIM, true).floats * sizeof(float)) ||
        !allow(chunk_state_kernel<16, false>, StateLayout<16>(CHUNK_MAX_DIM, false).floats * sizeof(float)) ||
        !allow(chunk_state_kernel<32, false>, StateLayout<32>(CHUNK_MAX_DIM, false).floats * sizeof(float)))
      return mi_fail("chunked_state: the shared memory was refused");
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  // 16 value columns a block while such blocks fit the SMs in one round, 32 beyond: half as many chains, each a little longer
  const bool wide = (long long)in.heads * in.items * (a.vp / 16) > mi::sm_count();
  for (int c0 = 0; c0 < total; c0 += slab) {
    a.c0 = c0;
    a.c1 = c0 + slab < total ? c0 + slab : total;
    mi::launch(delta ? chunk_build_kernel<true> : chunk_build_kernel<false>, dim3(a.c1 - a.c0, in.heads), dim3(THREADS),
               BuildLayout(a.dp).floats * sizeof(float), stream, a);
    if (wide)
      mi::launch(delta ? chunk_state_kernel<32, true> : chunk_state_kernel<32, false>, dim3(in.heads, a.vp / 32, in.items), dim3(THREADS),
                 StateLayout<32>(a.dp, delta).floats * sizeof(float), stream, a);
    else
      mi::launch(delta ? chunk_state_kernel<16, true> : chunk_state_kernel<16, false>, dim3(in.heads, a.vp / 16, in.items), dim3(THREADS),
                 StateLayout<16>(a.dp, delta).floats * sizeof(float), stream, a);
    mi::launch(delta ? chunk_out_kernel<true> : chunk_out_kernel<false>, dim3(a.c1 - a.c0, in.heads, (a.vp + OB - 1) / OB), dim3(OUT_THREADS),
               out_smem(a.dp), stream, a);
  }
  MI_LAUNCH_OK("chunked_state");
  return 0;
}

}  // namespace mi
