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
// block J; inside a block the product is walked.  Kernels:
//   chunk_build  a block per (chunk, head), all at once: A and Q~; for the delta rule L, the inverse of I + L, W, U0 and K^; for linear
//                attention, where U = V, K^^T V;
//   chunk_state  (delta rule) a block per (request, head, group of value columns), the only one that walks the chunks in order: keeps S in
//                registers, leaves every chunk's S_0, U = U0 - W S_0 and the state behind the last chunk;
//   chunk_scan   (linear attention) the same walk without products, a thread four elements of S;
//   chunk_out    a block per (chunk, head, 64 value columns), all at once: O, written over the values.
// Chunks are counted over the items of at least min_tokens new tokens, in their order; a step whose chunks need more
// scratch than SLAB_FLOATS is worked through in slabs, the state row carrying over.
//
// Every product runs on the tensor cores (mma.sync m16n8k8) with each float32 operand as the sum of two tf32 numbers and
// three of the four partial products (two where one operand is the values, which come from bfloat16 and have no lower part), added up
// in float32: as FMAs they were bound by the reads of shared memory that feed them.  tcgen05 has no use here: the chain of chunks is
// latency, and its operands are made in registers.  Against float64 the state errs, in parts of its norm, after 2048 tokens of 8 heads of
// 128 x 128 (in brackets what did these steps before: the walk in stretches, and for the delta rule with one decay a head chunks of
// FMAs): delta rule, decays a channel about 1 / 50 a token 1.9e-7 (3.5e-7), 1 / 3000 3.2e-7 (3.4e-6), stronger than 1 / 2 1.2e-7
// (0.7e-7); a head 1.6e-7 (2.4e-7), 2.3e-7 (4.2e-7), 1.2e-7 (0.9e-7); linear attention 1.4e-7 (1.7e-7), 4.7e-7 (1.3e-5), 0.65e-7 (0.3e-7).
// Measured on B200, one request of 2048 tokens, 8 / 16 / 32 heads of 128 x 128, the whole operation in microseconds: delta rule with
// one decay a key channel 130, 229, 416 (without chunks 1034, 1203, 1261), one a head 123, 210, 379 (692, 1105, 1151), linear attention
// 82, 139, 249 (171, 270, 451), with a constant a head 75, 125, 226 (157, 231, 392).  What bounds them: build and out run through 60 to 80 and
// 20 KB of instructions once, which come from L2, and their products at a third of the tensor cores' rate - splitting the operands takes as many
// issue slots as the products -; the walk takes 2700 cycles a chunk with 8 columns a block, of which its two products' tensor cycles are 800.
#include "chunked_state.cuh"

#include <algorithm>
#include <type_traits>

namespace mi {
namespace {

constexpr int C = CHUNK_TOKENS;
constexpr long long SLAB_FLOATS = 72ll << 20;      // 288 MiB: 86 chunks of 16 heads of 128 x 128 (delta rule)
constexpr int THREADS = 256;
constexpr int OB = 64;                 // value columns of a chunk_out block
constexpr int VT = 128;                // value columns that chunk_build takes at a time
constexpr int NB = C / 8;              // blocks of eight tokens

__host__ __device__ inline int pad(int x, int m) { return (x + m - 1) / m * m; }

struct Args : ChunkedStateArgs {
  int dp, vp;                          // dim padded to 32, vdim padded to 32
  // per (chunk, head): A [C][C], Q~ [C][dp], S_0 [dp][vp], P_C and what its rounding leaves [2][dp]; the delta rule's W and K^ [C][row_floats(dp)] and
  // U0 / U [vp / 8][C][8], as chunk_state holds them in shared memory; linear attention's K^^T V in the place of S_0 at first
  float *w, *u, *at, *kh, *qt, *s0, *pc;
  int c0, c1;                          // the slab's chunks
};

__host__ __device__ inline int row_floats(int dp) { return dp + 8; }      // of W and K^: 8-byte reads of a quarter warp's rows fall into different banks
__host__ __device__ inline long long unit_floats(int dp, int vp, bool delta) {
  return (delta ? (long long)C * (2 * row_floats(dp) + vp) : 0) + C * C + (long long)C * dp + (long long)dp * vp + 2 * dp;
}

// The item that chunk number c (over the items that are long enough) belongs to and the chunk's place in it; item -1: none.
__device__ __forceinline__ void find_chunk(const Args& a, int c, int& item, int& place) {
  item = -1;
#pragma unroll 1
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
// Rows come by bulk copies, a thread a row: as 16-byte copies of all threads, with their addresses, they took 4400 cycles to ask for.
__device__ __forceinline__ unsigned shared_at(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_at(bar)) : "memory"); }
__device__ __forceinline__ void bars_ready() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void bar_expect(uint64_t* bar, int bytes) {      // by one thread; a copy may end before
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_at(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(float* to, const float* from, int floats, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(shared_at(to)), "l"(from), "r"(floats * 4), "r"(shared_at(bar)) : "memory");
}
// before a barrier behind which bulk copies go where this thread has read or written
__device__ __forceinline__ void bulk_may_follow() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// False if the block's own copies, the only thing ever waited for, have not come: what depends on them - the chunk's read-outs, the state and
// all later read-outs of the head - is then made NaN, and the status word is set.
constexpr int WAIT_LIMIT = 1 << 22;
__device__ __forceinline__ bool bar_wait(uint64_t* bar, int parity) {
  unsigned done = 0;
#pragma unroll 1
  for (int i = 0; i < WAIT_LIMIT && !done; ++i)
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(shared_at(bar)), "r"(parity) : "memory");
  return done;
}

__device__ __forceinline__ void say_late(bool late, int* status) {
  if (late && status != nullptr) atomicExch(status, CHUNK_STATUS_LATE);
}

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
// a += b, of two pairs in one instruction each: what limits these kernels is the number of instructions that can be issued
__device__ __forceinline__ void add2(float& a0, float& a1, float b0, float b1) {
  asm("{\n .reg .b64 a, b;\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n add.rn.f32x2 a, a, b;\n mov.b64 {%0, %1}, a;\n}\n" : "+f"(a0), "+f"(a1) : "f"(b0), "f"(b1));
}
// Two numbers at a time: the lower parts, x - hi, as one pair.
__device__ __forceinline__ void split2(Two& a, Two& b, float x, float y) {
  a.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  b.hi = (__float_as_uint(y) + 0x1000u) & 0xffffe000u;
  asm("{\n .reg .b64 h, m, v;\n mov.b64 h, {%2, %3};\n mov.b64 m, {%6, %6};\n mov.b64 v, {%4, %5};\n fma.rn.f32x2 v, h, m, v;\n mov.b64 {%0, %1}, v;\n}\n"
      : "=r"(a.lo), "=r"(b.lo) : "r"(a.hi), "r"(b.hi), "f"(x), "f"(y), "f"(-1.f));
}
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
  add2(s.c[0], s.c[1], p[0], p[1]);
  add2(s.c[2], s.c[3], p[2], p[3]);
}
// The same for an 8 x 8 operand of numbers that tf32 holds, as the values are, which come from bfloat16: no lower part.
__device__ __forceinline__ void mma2(Sum& s, const Two (&a)[4], float b0, float b1) {
  const float zero[4] = {0.f, 0.f, 0.f, 0.f};
  float p[4];
  mma1(s.small, a[0].lo, a[1].lo, a[2].lo, a[3].lo, __float_as_uint(b0), __float_as_uint(b1), s.small);
  mma1(p, a[0].hi, a[1].hi, a[2].hi, a[3].hi, __float_as_uint(b0), __float_as_uint(b1), zero);
  add2(s.c[0], s.c[1], p[0], p[1]);
  add2(s.c[2], s.c[3], p[2], p[3]);
}
// The 16 x 8 operand of a row-major tile.
__device__ __forceinline__ void load_a(Two (&a)[4], const float* p, int ld, int g, int t, float s0 = 1.f, float s1 = 1.f) {      // s0, s1: of its columns t and t + 4
  split2(a[0], a[1], p[g * ld + t] * s0, p[(g + 8) * ld + t] * s0);
  split2(a[2], a[3], p[g * ld + t + 4] * s1, p[(g + 8) * ld + t + 4] * s1);
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
  split2(a[0], a[1], x.x, x.y);
  split2(a[2], a[3], y.x, y.y);
}
__device__ __forceinline__ void load_b(Two (&b)[2], const float* p, int ld, int g, int t) {
  split2(b[0], b[1], p[t * ld + g], p[(t + 4) * ld + g]);
}
// -------------------------------------------------------------------------------------------------------------- build

constexpr int LDT = C + 4;             // a row of the inverse
constexpr int PAIRS = NB * (NB - 1) / 2;      // of blocks of eight tokens, an earlier one and a later one
struct BuildLayout {                   // float offsets
  int ld, k, q, g, total, diag, beta, rest, f, floats;
  __host__ __device__ explicit BuildLayout(int dp) {
    ld = dp + 4;
    const int rows = C * (dp > VT ? ld : VT + 4);      // of channels, then of values, VT columns at a time
    k = 0;                                                            // [C][ld] keys; E k; then delta: the values, linear: K^
    q = k + rows;                                                     // [C][ld] queries; F q; then L^T [C][C] and behind it half of the tiles' sums, then the inverse [C][LDT]
    g = q + (C * ld > C * C + C * LDT ? C * ld : C * C + C * LDT);    // [C][ld] decays; delta: F k, diag(beta) K~; linear: the values
    total = g + rows;                                                 // [NB][dp] a block's whole product
    diag = total + NB * dp;                                           // [NB][64] products inside a block: 36 of q, 28 of k
    beta = diag + NB * 64;                                            // [C]
    rest = beta + C;                                                  // [NB][dp] one decay a channel: what the rounding of the block's product leaves
    f = rest + NB * dp;                                               // one decay a head: F [C], E [C], a block's product [NB], as doubles [NB], the decays [C], what they are of [C]
    floats = f + 4 * C + 3 * NB;
  }
};
static_assert(PAIRS * 128 <= C * LDT, "half of the tiles' sums lie where the inverse will");

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

// Block I's rows - eight of F k above eight of F q - times every earlier block's E k and the products of the blocks between, over the
// channels d0 .. d1 - 1.  I is known to the compiler, so the reads of a step's tiles stand before its products.
template <int I, bool DELTA>
__device__ __forceinline__ void between_blocks(Sum (&acc)[NB - 1], const float* ks, const float* qs, const float* gs, const float* total, int ld, int dp,
                                               int d0, int d1, int g, int t4) {
  const float *fk = gs + (8 * I + g) * ld + t4, *fq = qs + (8 * I + g) * ld + t4;
#pragma unroll 1
  for (int d = d0; d < d1; d += 8) {
    float e0[I > 0 ? I : 1], e1[I > 0 ? I : 1], p0 = 1.f, p1 = 1.f;
#pragma unroll
    for (int j = I - 1; j >= 0; --j) {
      if (j + 1 < I) { p0 *= total[(j + 1) * dp + d + t4]; p1 *= total[(j + 1) * dp + d + t4 + 4]; }
      const float* ek = ks + (8 * j + g) * ld + d + t4;
      e0[j] = ek[0] * p0;
      e1[j] = ek[4] * p1;
    }
    Two x[4];
    split2(x[0], x[2], DELTA ? fk[d] : 0.f, DELTA ? fk[d + 4] : 0.f);
    split2(x[1], x[3], fq[d], fq[d + 4]);
#pragma unroll
    for (int j = I - 1; j >= 0; --j) {
      Two y[2];
      split2(y[0], y[1], e0[j], e1[j]);
      mma3(acc[j], x, y);
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
  __shared__ __align__(8) uint64_t bars[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, head = blockIdx.y;
  if (tid == 0) {
    find_chunk(a, a.c0 + blockIdx.x, found[0], found[1]);
    bar_init(bars);
    bar_init(bars + 1);
    bars_ready();
  }
  mi::grid_dependency_sync();
  __syncthreads();
  const int item = found[0];
  if (item < 0) return;
  const int first = found[1] * C, n = min(C, a.q_len[item] - first), row0 = a.q_start[item] + first;
  const int kvh = head / (a.heads / a.qk_heads);
  const size_t unit = (size_t)blockIdx.x * a.heads + head;
  const bool per_head = a.decay != CHUNK_DECAY_CHANNEL, logs = a.decay == CHUNK_DECAY_HEAD;
  float *fs = sm + at.f, *of_token = fs + 2 * C + 3 * NB, *step_of = of_token + C;
  double* whole = reinterpret_cast<double*>(fs + 2 * C + NB);
  // Rows of keys, queries and decays, a thread a row; tokens behind the last and channels behind the last: zero keys and queries, decays of one
  if (tid == 0) bar_expect(bars, n * (per_head ? 2 : 3) * a.dim * 4);
  {
    const int t = tid & (C - 1), which = tid / C;      // (a warp has one kind of rows)
    if (which < (per_head ? 2 : 3)) {
      float* to = (which == 0 ? ks : which == 1 ? qs : gs) + t * ld;
      const float fill = which == 2 ? 1.f : 0.f;
      if (t < n)
        bulk_copy(to, which == 2 ? a.g + ((size_t)(row0 + t) * a.heads + head) * a.dim
                                 : (which ? a.qn : a.kn) + ((size_t)(row0 + t) * a.qk_heads + kvh) * a.dim, a.dim, bars);
#pragma unroll 1
      for (int d = t < n ? a.dim : 0; d < dp; d += 4) st4(to + d, make_float4(fill, fill, fill, fill));
    } else if (tid >= 3 * C) {
      if (DELTA) bt[t] = t < n ? a.beta[(size_t)(row0 + t) * a.heads + head] : 0.f;
      if (per_head) {
        const float x = t < n ? a.g[logs ? (size_t)(row0 + t) * a.heads + head : head] : logs ? 0.f : 1.f;
        step_of[t] = x;
        of_token[t] = logs ? expf(x) : x;
      }
    }
  }
  // One decay a head: F, E and the blocks' products are sums of logarithms (a constant's: products) in double, rounded once.  A constant's
  // float products err alike in every chunk, and logarithms of decays near one hold digits that the decays do not.
  if (per_head) {
    __syncthreads();
    if (tid < 2 * C) {      // F of a token, then E of one
      const int t = tid & (C - 1), b = t & ~7;
      const bool forward = tid < C;
      double f = logs ? 0. : 1.;
#pragma unroll 1
      for (int j = forward ? b : b + 7; forward ? j <= t : j > t; j += forward ? 1 : -1) f = logs ? f + (double)step_of[j] : f * (double)step_of[j];
      const float r = logs ? expf((float)f) : (float)f;
      fs[tid] = r;
      if (forward && (t & 7) == 7) {
        whole[t >> 3] = f;
        fs[2 * C + (t >> 3)] = r;
      }
    }
  }
  bool late = __syncthreads_or(!bar_wait(bars, 0));
  // Inside the blocks, a warp a block of eight tokens, a lane two key channels at a time: products number p (p + 1) / 2 + s of q_p and
  // k_s for s <= p, then 36 + p (p - 1) / 2 + s of k_p and k_s for s < p, the decays between s and p walked.  A key that has
  // walked to the block's end is E k; F q and F k are left beside it, each in the place of what it was made from.
  {
    float v[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = 0.f;
    const float* table = fs + 8 * warp;      // (one decay a head)
#pragma unroll 1
    for (int d = 2 * lane; d < dp; d += 64) {
      float *kr = ks + warp * 8 * ld + d, *qr = qs + warp * 8 * ld + d, *gr = gs + warp * 8 * ld + d;
      const float* decays = per_head ? of_token + 8 * warp : gr;
      const int to_next = per_head ? 1 : ld, to_second = per_head ? 0 : 1;
      float2 key[8];      // key s times the decays from behind s to the token at hand
      float2 f = make_float2(1.f, 1.f), rest = make_float2(0.f, 0.f);
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const float2 kp = *reinterpret_cast<const float2*>(kr + p * ld), qp = *reinterpret_cast<const float2*>(qr + p * ld);
        const float2 gp = make_float2(decays[p * to_next], decays[p * to_next + to_second]);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          if (s < p) {
            key[s].x *= gp.x; key[s].y *= gp.y;
            const int i = p * (p + 1) / 2 + s;
            v[i] = fmaf(qp.x, key[s].x, fmaf(qp.y, key[s].y, v[i]));
            if (DELTA) {
              const int l = 36 + p * (p - 1) / 2 + s;
              v[l] = fmaf(kp.x, key[s].x, fmaf(kp.y, key[s].y, v[l]));
            }
          }
        }
        key[p] = kp;
        const int i = p * (p + 1) / 2 + p;
        v[i] = fmaf(qp.x, kp.x, fmaf(qp.y, kp.y, v[i]));
        const float2 before = f;
        f.x *= gp.x; f.y *= gp.y;
        rest.x = fmaf(rest.x, gp.x, fmaf(before.x, gp.x, -f.x));
        rest.y = fmaf(rest.y, gp.y, fmaf(before.y, gp.y, -f.y));
        if (per_head) f.x = f.y = table[p];
        st2(qr + p * ld, qp.x * f.x, qp.y * f.y);
        if (DELTA) st2(gr + p * ld, kp.x * f.x, kp.y * f.y);
      }
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const float2 k = *reinterpret_cast<const float2*>(kr + s * ld);
        const float e = table[C + s];
        st2(kr + s * ld, per_head ? k.x * e : key[s].x, per_head ? k.y * e : key[s].y);
      }
      if (per_head) f.x = f.y = fs[2 * C + warp];
      st2(total + warp * dp + d, f.x, f.y);
      st2(sm + at.rest + warp * dp + d, rest.x, rest.y);
    }
    reduce_scatter(v, lane);
    st2(sm + at.diag + warp * 64 + 2 * lane, v[0], v[1]);
  }
  bulk_may_follow();
  __syncthreads();
  int values_round = 0;
  auto fetch_values = [&](float* to, int v0) {      // VT columns from v0 on, zeros behind the last token; what lies behind the last column reaches only columns there
    const int columns = min(VT, a.vdim - v0);
    if (tid == 0) bar_expect(bars + 1, n * columns * 4);
    if (tid < C) {
      float* row = to + tid * (VT + 4);
      if (tid < n) bulk_copy(row, a.raw + (size_t)(row0 + tid) * (a.heads * a.vdim) + head * a.vdim + v0, columns, bars + 1);
#pragma unroll 1
      for (int c = tid < n ? columns : 0; c < VT; c += 4) st4(row + c, make_float4(0.f, 0.f, 0.f, 0.f));
    }
  };
  auto values_there = [&]() {      // for all threads
    late |= (bool)__syncthreads_or(!bar_wait(bars + 1, values_round & 1));
    ++values_round;
  };
  if (!DELTA) fetch_values(gs, 0);
  // Between blocks: warp I has block I over the lower half of the channels and block 7 - I over the upper, seven tiles each (all channels of
  // block I a warp, behind branches: 13000 cycles and more; so 7400).  The two warps of a pair share their code.  One body for all blocks, its
  // tiles behind branches, is a quarter of the instructions and 15000 cycles: the reads of a step's tiles no longer stand before its products.
  float own[NB - 1][4], other[NB - 1][4];
  switch (min(warp, NB - 1 - warp)) {
#define MI_BETWEEN(I)                                                                                                              \
  case I: {                                                                                                                        \
    constexpr int J = NB - 1 - I;                                                                                                  \
    const bool first_of_pair = warp == I;                                                                                          \
    Sum x[NB - 1], y[NB - 1];                                                                                                      \
    between_blocks<I, DELTA>(x, ks, qs, gs, total, ld, dp, first_of_pair ? 0 : dp / 2, first_of_pair ? dp / 2 : dp, g, t4);        \
    between_blocks<J, DELTA>(y, ks, qs, gs, total, ld, dp, first_of_pair ? dp / 2 : 0, first_of_pair ? dp : dp / 2, g, t4);        \
    _Pragma("unroll") for (int j = 0; j < J; ++j)                                                                                  \
      _Pragma("unroll") for (int e = 0; e < 4; ++e) {                                                                              \
        const float v = j < I ? x[j].at(e) : 0.f, w = y[j].at(e);                                                                  \
        own[j][e] = first_of_pair ? v : w;                                                                                         \
        other[j][e] = first_of_pair ? w : v;                                                                                       \
      }                                                                                                                            \
    break;                                                                                                                         \
  }
    MI_BETWEEN(0) MI_BETWEEN(1) MI_BETWEEN(2) MI_BETWEEN(3)
#undef MI_BETWEEN
  }
  if (warp == 0 && per_head) {      // P_C and what its rounding leaves
    double p = logs ? 0. : 1.;
#pragma unroll 1
    for (int b = 0; b < NB; ++b) p = logs ? p + whole[b] : p * whole[b];
    if (logs) p = exp(p);
    const float high = (float)p, low = (float)(p - (double)high);
    for (int d = lane; d < dp; d += 32) {
      a.pc[unit * 2 * dp + d] = high;
      a.pc[unit * 2 * dp + dp + d] = low;
    }
  }
  // Q~ and K^, a thread the blocks b0, b0 + step, ... of a channel, with the products of the blocks before and behind
  const int step = THREADS / dp, b0 = tid / dp, my_d = tid - b0 * dp, b_last = b0 + (NB - 1 - b0) / step * step;
  auto forward = [&](auto use) {
    float before = 1.f;
    int at_b = 0;
#pragma unroll 1
    for (int b = b0; b < NB && b0 < step; b += step) {
#pragma unroll 1
      for (; at_b < b; ++at_b) before *= total[at_b * dp + my_d];
      use(8 * b, before);
    }
  };
  auto backward = [&](auto use) {
    float behind = 1.f;
    int at_b = NB - 1;
#pragma unroll 1
    for (int b = b_last; b >= 0 && b0 < step; b -= step) {
#pragma unroll 1
      for (; at_b > b; --at_b) behind *= total[at_b * dp + my_d];
      use(8 * b, behind);
    }
  };
  forward([&](int row, float before) {
#pragma unroll
    for (int j = 0; j < 8; ++j) a.qt[(unit * C + row + j) * dp + my_d] = qs[(row + j) * ld + my_d] * before;
  });
  if (DELTA)
    backward([&](int row, float behind) {
#pragma unroll
      for (int j = 0; j < 8; ++j) a.kh[(unit * C + row + j) * row_floats(dp) + my_d] = ks[(row + j) * ld + my_d] * behind;
    });
  if (b0 == step - 1 && !per_head) {
    double p = 1.;
#pragma unroll 1
    for (int j = 0; j < NB; ++j) p *= (double)total[j * dp + my_d] + (double)sm[at.rest + j * dp + my_d];
    a.pc[unit * 2 * dp + my_d] = (float)p;
    a.pc[unit * 2 * dp + dp + my_d] = (float)(p - (double)(float)p);
  }
  bulk_may_follow();
  __syncthreads();      // everyone is done with E k, F q and F k
  float *lt = qs, *inv = qs + C * C;
#pragma unroll
  for (int j = 0; j < NB - 1; ++j)      // the other half of block 7 - warp's tiles, block I's from number I (I - 1) / 2 on
    if (j < NB - 1 - warp) st4(inv + (((NB - 1 - warp) * (NB - 2 - warp) / 2 + j) * 32 + lane) * 4, make_float4(other[j][0], other[j][1], other[j][2], other[j][3]));
  if (DELTA) {
    fetch_values(ks, 0);
    forward([&](int row, float before) {      // F k becomes K~
#pragma unroll
      for (int j = 0; j < 8; ++j) gs[(row + j) * ld + my_d] *= before;
    });
  } else {
    backward([&](int row, float behind) {      // E k becomes K^
#pragma unroll
      for (int j = 0; j < 8; ++j) ks[(row + j) * ld + my_d] *= behind;
    });
  }
  if (!DELTA) values_there();
  else __syncthreads();
  // A, a row a token: zeros behind the diagonal; and L^T, the part before the diagonal
  {
    const int t = 8 * warp + g;
    float* out = a.at + unit * C * C + (size_t)t * C + 2 * t4;
    const float *dq = sm + at.diag + warp * 64 + g * (g + 1) / 2, *dk = sm + at.diag + warp * 64 + 36 + g * (g - 1) / 2;
    const float* half = inv + (warp * (warp - 1) / 2 * 32 + lane) * 4;
    const float b = DELTA ? bt[t] : 0.f;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      float x = 0.f, y = 0.f;
      if (j < warp) {
        const int i = j < NB - 1 ? j : 0;
        const float4 h = ld4(half + j * 128);
        x = own[i][2] + h.z;
        y = own[i][3] + h.w;
        if (DELTA) {
          lt[(8 * j + 2 * t4) * C + t] = b * (own[i][0] + h.x);
          lt[(8 * j + 2 * t4 + 1) * C + t] = b * (own[i][1] + h.y);
        }
      }
      if (j == warp) {
        x = 2 * t4 <= g ? dq[2 * t4] : 0.f;
        y = 2 * t4 + 1 <= g ? dq[2 * t4 + 1] : 0.f;
        if (DELTA) {
          if (2 * t4 < g) lt[(8 * warp + 2 * t4) * C + t] = b * dk[2 * t4];
          if (2 * t4 + 1 < g) lt[(8 * warp + 2 * t4 + 1) * C + t] = b * dk[2 * t4 + 1];
        }
      }
      st2(out + 8 * j, late ? NAN : x, late ? NAN : y);
    }
  }
  if (!DELTA) {      // K^^T V: a warp 16 key channels - a lane those numbered 2 g and 2 g + 1 -, 32 value columns at a time
    for (int v0 = 0; v0 < a.vp; v0 += VT) {
      if (v0 > 0) {
        bulk_may_follow();
        __syncthreads();
        fetch_values(gs, v0);
        values_there();
      }
      if (16 * warp >= dp) continue;
#pragma unroll 1
      for (int c = 0; c < min(VT, a.vp - v0); c += 32) {
        Sum more[4];
#pragma unroll 1
        for (int k = 0; k < C; k += 8) {
          Two x[4];
          load_a_transposed(x, ks + k * ld + 16 * warp, ld, g, t4);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float* y = gs + (k + t4) * (VT + 4) + c + 8 * j + g;
            mma2(more[j], x, y[0], y[4 * (VT + 4)]);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            st2(a.s0 + (unit * dp + 16 * warp + 2 * g + h) * a.vp + v0 + c + 8 * j + 2 * t4, late ? NAN : more[j].at(2 * h), late ? NAN : more[j].at(2 * h + 1));
      }
    }
    if (tid == 0) say_late(late, a.status);
    return;
  }
  __syncthreads();
  // The inverse of I + L from blocks of 16 tokens on, [[A, 0], [B, D]]^-1 = [[A^-1, 0], [-D^-1 (B A^-1), D^-1]]: the blocks on the diagonal by
  // substitution, a thread a column - an unknown that is final is taken off all later rows -, then 32 and 64 as two products each.
  // (Substitution over 32 rows was 640 instructions in a row for two warps, 5700 cycles; so 1300 and 1100.)
  constexpr int HALF = C / 2, SUB = C / 4;
  if (tid < C) {
    const int h0 = tid & ~(SUB - 1), col = tid - h0;
    float x[SUB];
#pragma unroll
    for (int t = 0; t < SUB; ++t) x[t] = t == col ? 1.f : 0.f;
#pragma unroll
    for (int s = 0; s < SUB - 1; ++s) {
#pragma unroll
      for (int q = (s + 1) / 4 * 4; q < SUB; q += 4) {
        const float4 l = ld4(lt + (h0 + s) * C + h0 + q);
        if (q > s) x[q] = fmaf(-l.x, x[s], x[q]);
        if (q + 1 > s) x[q + 1] = fmaf(-l.y, x[s], x[q + 1]);
        if (q + 2 > s) x[q + 2] = fmaf(-l.z, x[s], x[q + 2]);
        if (q + 3 > s) x[q + 3] = fmaf(-l.w, x[s], x[q + 3]);
      }
    }
#pragma unroll
    for (int t = 0; t < SUB; ++t) {
      inv[(h0 + t) * LDT + tid] = x[t];
      if (h0 & SUB) inv[(h0 - SUB + t) * LDT + tid] = 0.f;
    }
  }
  __syncthreads();
  {      // 16 -> 32, twice, a thread two values of a column: as many rounded sums as the substitution had
    const int r0 = (tid >> 7) * HALF + SUB, row = r0 + (tid >> 3 & 15), c = r0 - SUB + 2 * (tid & 7);
    auto dot = [&](const float* left, int step, int k0) {      // sum over 16 k: left[k step] inv[k0 + k][c], [c + 1]
      float x = 0.f, y = 0.f;
#pragma unroll 4
      for (int k = 0; k < SUB; ++k) {
        const float2 r = *reinterpret_cast<const float2*>(inv + (k0 + k) * LDT + c);
        x = fmaf(left[k * step], r.x, x);
        y = fmaf(left[k * step], r.y, y);
      }
      return make_float2(x, y);
    };
    const float2 ba = dot(lt + (r0 - SUB) * C + row, C, r0 - SUB);      // B A^-1 (L is kept transposed)
    st2(inv + row * LDT + c, ba.x, ba.y);
    __syncthreads();
    float2 x = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int k = r0; k <= row; ++k) {
      const float2 r = *reinterpret_cast<const float2*>(inv + k * LDT + c);
      x.x = fmaf(inv[row * LDT + k], r.x, x.x);
      x.y = fmaf(inv[row * LDT + k], r.y, x.y);
    }
    __syncthreads();
    st2(inv + row * LDT + c, -x.x, -x.y);
    __syncthreads();
  }
  {      // 32 -> 64: a warp 16 rows x 8 columns
    const int m = HALF + (warp & 1) * 16, c = (warp >> 1) * 8;
    float* block = inv + (m + g) * LDT + c + 2 * t4;
    Sum ba;
#pragma unroll 1
    for (int k = 0; k < HALF; k += 8) {
      Two l[4], r[2];
      const float* p = lt + (k + t4) * C + m + g;
      split2(l[0], l[1], p[0], p[8]);
      split2(l[2], l[3], p[4 * C], p[4 * C + 8]);
      load_b(r, inv + k * LDT + c, LDT, g, t4);
      mma3(ba, l, r);
    }
    st2(block, ba.at(0), ba.at(1));
    st2(block + 8 * LDT, ba.at(2), ba.at(3));
    __syncthreads();
    Sum dba;
#pragma unroll 1
    for (int k = HALF; k < C; k += 8) {
      Two l[4], r[2];
      load_a(l, inv + m * LDT + k, LDT, g, t4);
      load_b(r, inv + k * LDT + c, LDT, g, t4);
      mma3(dba, l, r);
    }
    float x[4] = {dba.at(0), dba.at(1), dba.at(2), dba.at(3)};
    if (any_not_finite(x)) {      // element by element, and only up to the diagonal
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = m + g + 8 * (e >> 1), col = c + 2 * t4 + (e & 1);
        x[e] = 0.f;
#pragma unroll 1
        for (int k = HALF; k <= row; ++k) x[e] = fmaf(inv[row * LDT + k], inv[k * LDT + col], x[e]);
      }
    }
    __syncthreads();
    st2(block, -x[0], -x[1]);
    st2(block + 8 * LDT, -x[2], -x[3]);
  }
  values_there();
  // W and U0, the inverse times diag(beta) times K~ and times V side by side: a warp two tiles of 16 rows, one of the upper and one
  // of the lower half so that all have as much of the inverse before the diagonal, in 32 columns
  for (int v0 = 0; v0 < a.vp; v0 += VT) {
    if (v0 > 0) {
      bulk_may_follow();
      __syncthreads();
      fetch_values(ks, v0);
      values_there();
    }
    const int columns = dp + min(VT, a.vp - v0);
#pragma unroll 1
    for (int n0 = (v0 ? dp : 0) + (warp >> 1) * 32; n0 < columns; n0 += 128) {
      const bool keys = n0 < dp;
      const float* right = keys ? gs + n0 : ks + n0 - dp;
      const int ldr = keys ? ld : VT + 4;
      float* out = keys ? a.w + unit * C * row_floats(dp) + n0 : a.u + unit * C * a.vp + (size_t)(v0 + n0 - dp) * C;
      const int ldo = keys ? row_floats(dp) : 8, next = keys ? 8 : 8 * C;      // floats to the next token, to the next eight columns
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        const int m0 = 16 * (side ? 3 - (warp & 1) : warp & 1);
        Sum sum[4];
#pragma unroll 1
        for (int k = 0; k < m0 + 16; k += 8) {      // (the inverse is zero behind its diagonal)
          Two l[4];
          load_a(l, inv + m0 * LDT + k, LDT, g, t4, bt[k + t4], bt[k + t4 + 4]);
          const float* r = right + (k + t4) * ldr + g;
          if (keys) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              Two y[2];
              split2(y[0], y[1], r[8 * j], r[4 * ldr + 8 * j]);
              mma3(sum[j], l, y);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) mma2(sum[j], l, r[8 * j], r[4 * ldr + 8 * j]);
          }
        }
        float* o = out + (size_t)(m0 + g) * ldo + 2 * t4;
        unsigned bad = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float c[4] = {sum[j].at(0), sum[j].at(1), sum[j].at(2), sum[j].at(3)};
          st2(o + j * next, late ? NAN : c[0], late ? NAN : c[1]);
          st2(o + j * next + 8 * ldo, late ? NAN : c[2], late ? NAN : c[3]);
          bad |= any_not_finite(c) && !late ? 15u << 4 * j : 0;
        }
#pragma unroll 1
        for (; bad; bad &= bad - 1) {      // element by element, and only up to the diagonal
          const int j = __ffs(bad) - 1 >> 2, e = __ffs(bad) - 1 & 3, t = m0 + g + 8 * (e >> 1), col = 8 * j + 2 * t4 + (e & 1);
          float y = 0.f;
#pragma unroll 1
          for (int k = 0; k <= t; ++k) y = fmaf(inv[t * LDT + k] * bt[k], right[k * ldr + col], y);
          o[j * next + (e >> 1) * 8 * ldo + (e & 1)] = y;
        }
      }
    }
  }
  if (tid == 0) say_late(late, a.status);
}

// -------------------------------------------------------------------------------------------------------------- state

// The chunks that an item's walk of this slab covers, and the number of the item's first chunk; from >= to: none.
__device__ __forceinline__ void walk_of(const Args& a, int item, int& base, int& from, int& to) {
  base = from = to = 0;
  if (a.q_len[item] < a.min_tokens) return;
#pragma unroll 1
  for (int b = 0; b < item; ++b)
    if (a.q_len[b] >= a.min_tokens) base += (a.q_len[b] + C - 1) / C;
  from = max(a.c0, base);
  to = min(a.c1, base + (a.q_len[item] + C - 1) / C);
}
// P_C S_0 + K^^T U, P_C in two parts: products of decays near one are all rounded to the same side, a constant's to the same value.
__device__ __forceinline__ float decayed(float s, float p, float p_low, float more) {
  const float low = s * p_low;
  return fmaf(s, p, more + (fabsf(low) <= 3.402823466e38f ? low : 0.f));      // (an infinite state stays one)
}

// Linear attention: U = V does not need the state, so K^^T V of all chunks is there and only P_C S_0 + K^^T V is walked, a thread four
// elements of the state, their chunks' S_0 written over K^^T V.  (29 chunks of 16 heads of 128 x 128: 48 us with the products inside the
// walk; the scan takes 9, the products 16 more in chunk_build.)
constexpr int SCAN_THREADS = 256, SCAN_AHEAD = 4;
__global__ void __launch_bounds__(SCAN_THREADS)
chunk_scan_kernel(Args a) {
  const int dp = a.dp, head = blockIdx.y, item = blockIdx.z;
  const int i = (blockIdx.x * SCAN_THREADS + threadIdx.x) * 4, d = i / a.vp, c = i - d * a.vp;
  int base, from, to;
  walk_of(a, item, base, from, to);
  if (from >= to || d >= dp) return;
  const bool in = d < a.dim && c < a.vdim;
  float* st = a.state + (size_t)a.seq_slot[item] * a.state_stride + (size_t)head * a.dim * a.vdim + (size_t)d * a.vdim + c;
  mi::grid_dependency_sync();
  float S[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) S[e] = in ? st[e] : 0.f;      // (a state's row may start at any multiple of four bytes)
  float4 more[SCAN_AHEAD];
  float p[SCAN_AHEAD], low[SCAN_AHEAD];
  for (int c0 = from; c0 < to; c0 += SCAN_AHEAD) {
#pragma unroll
    for (int k = 0; k < SCAN_AHEAD; ++k) {
      if (c0 + k < to) {
        const size_t unit = (size_t)(c0 + k - a.c0) * a.heads + head;
        more[k] = ld4(a.s0 + unit * dp * a.vp + i);
        p[k] = a.pc[unit * 2 * dp + d];
        low[k] = a.pc[unit * 2 * dp + dp + d];
      }
    }
#pragma unroll
    for (int k = 0; k < SCAN_AHEAD; ++k) {
      if (c0 + k < to) {
        st4(a.s0 + ((size_t)(c0 + k - a.c0) * a.heads + head) * dp * a.vp + i, make_float4(S[0], S[1], S[2], S[3]));
        S[0] = decayed(S[0], p[k], low[k], more[k].x);
        S[1] = decayed(S[1], p[k], low[k], more[k].y);
        S[2] = decayed(S[2], p[k], low[k], more[k].z);
        S[3] = decayed(S[3], p[k], low[k], more[k].w);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (in) st[e] = S[e];
}

// The delta rule's walk.  A chunk is two products in a chain, W S_0 over the channels and K^^T U over the tokens, with the state in registers
// between them; sixteen warps split the first one's channels in quarters (of 32 columns: in halves) and add up the parts in shared memory, and
// a chunk's W, K^ and U0 come by four bulk copies one chunk ahead.  (32 chunks of 8 heads of 128 x 128: 100 us by eight warps that split no
// channels, 16 columns a block and 16-byte copies by all threads; so 50.)
constexpr int STATE_THREADS = 512;
template <int CB>                      // value columns of a block
struct StateLayout {                   // float offsets
  static constexpr int NT = CB / 8, PARTS = CB == 32 ? 2 : 4;
  // rows of S, of U and of the partial sums: strides at which a warp's reads, two rows apart (S) or one (U), fall into different banks
  static constexpr int LDS = CB + 4, LDU = CB == 8 ? 8 : CB + 8, LDX = CB + 2;
  int k, u, p, stage, s, ut, x, bars, floats;
  __host__ __device__ explicit StateLayout(int dp) {
    k = C * row_floats(dp);            // a stage: W, K^ [C][row_floats(dp)], U0 [NT][C][8], P_C [2][dp]
    u = 2 * k;
    p = u + C * CB;
    stage = p + 2 * dp;
    s = 2 * stage;                     // [dp][LDS]
    ut = s + dp * LDS;                 // [C][LDU]
    x = ut + C * LDU;                  // [PARTS][C][LDX]
    bars = x + PARTS * C * LDX;
    floats = bars + 4;
  }
  size_t bytes() const { return (size_t)floats * sizeof(float); }
};

template <int CB>
__global__ void __launch_bounds__(STATE_THREADS, 1)
chunk_state_kernel(Args a) {
  using L = StateLayout<CB>;
  constexpr int LDS = L::LDS, LDU = L::LDU, LDX = L::LDX, NT = L::NT, PARTS = L::PARTS;
  constexpr int ST = NT > 1 ? NT / 2 : 1;      // 8-column tiles of S that a warp holds
  extern __shared__ __align__(16) float sm[];
  const L at(a.dp);
  const int dp = a.dp, ld = row_floats(dp), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int head = blockIdx.x, v0 = blockIdx.y * CB, item = blockIdx.z;
  int base, from, to;
  walk_of(a, item, base, from, to);
  if (from >= to) return;
  float *ss = sm + at.s, *us = sm + at.ut;
  float* parts = sm + at.x;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + at.bars);
  if (tid == 0) {
    bar_init(full);
    bar_init(full + 1);
    bars_ready();
  }
  mi::grid_dependency_sync();
  __syncthreads();
  auto fetch = [&](int c) {      // by one thread, into a stage that everyone has left
    const size_t unit = (size_t)(c - a.c0) * a.heads + head;
    float* buf = sm + ((c - from) & 1) * at.stage;
    uint64_t* bar = full + ((c - from) & 1);
    bar_expect(bar, at.stage * 4);
    bulk_copy(buf, a.w + unit * C * ld, C * ld, bar);
    bulk_copy(buf + at.u, a.u + unit * C * a.vp + (size_t)v0 * C, C * CB, bar);
    bulk_copy(buf + at.k, a.kh + unit * C * ld, C * ld, bar);
    bulk_copy(buf + at.p, a.pc + unit * 2 * dp, 2 * dp, bar);
  };
  if (tid == 0) fetch(from);
  // this warp's part of S: 16 key channels - a lane those numbered 2 g and 2 g + 1 -, ST tiles of columns from j0 on.  With one
  // tile for all the upper eight warps hold none and have half of the tokens of K^^T U.
  const int d0 = 16 * (warp & 7) + 2 * g, j0 = NT > 1 ? (warp >> 3) * ST : 0;
  const bool adds = 16 * (warp & 7) < dp, holds = adds && (NT > 1 || warp < 8);
  float* st = a.state + (size_t)a.seq_slot[item] * a.state_stride + (size_t)head * a.dim * a.vdim;
  float S[ST][4];
  auto keep = [&]() {
#pragma unroll
    for (int j = 0; j < ST; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) st2(ss + (d0 + h) * LDS + 8 * (j0 + j) + 2 * t4, S[j][2 * h], S[j][2 * h + 1]);
  };
#pragma unroll
  for (int j = 0; j < ST; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1), c = v0 + 8 * (j0 + j) + 2 * t4 + (e & 1);
      S[j][e] = (holds && d < a.dim && c < a.vdim) ? st[(size_t)d * a.vdim + c] : 0.f;
    }
  if (holds) keep();
  __syncthreads();
  bool late = false;      // a wait for this block's own copies ran out: U becomes NaN, and with it the state and what is read from it
  for (int c = from; c < to; ++c) {
    const int stage = (c - from) & 1;
    const float* cur = sm + stage * at.stage;
    const size_t unit = (size_t)(c - a.c0) * a.heads + head;
    if (tid == 0 && c + 1 < to) fetch(c + 1);
    late |= !bar_wait(full + stage, ((c - from) >> 1) & 1);
    {      // W S_0: a warp 16 tokens and a part of the channels - all columns, or of 32 half
      constexpr int HT = CB == 32 ? 2 : NT;
      const int m0 = (warp & 3) * 16, part = (warp >> 2) % PARTS, n0 = CB == 32 ? (warp >> 3) * 16 : 0;
      const int k0 = part * (dp / PARTS), k1 = k0 + dp / PARTS;
      Sum x[HT];
#pragma unroll 4
      for (int k = k0; k < k1; k += 8) {
        Two w[4];
        load_a_pairs(w, cur + m0 * ld + k, ld, g, t4);
#pragma unroll
        for (int j = 0; j < HT; ++j) {
          Two s[2];
          const float* row = ss + (k + 2 * t4) * LDS + n0 + 8 * j + g;
          split2(s[0], s[1], row[0], row[LDS]);
          mma3(x[j], w, s);
        }
      }
#pragma unroll
      for (int j = 0; j < HT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) st2(parts + (part * C + m0 + g + 8 * h) * LDX + n0 + 8 * j + 2 * t4, x[j].at(2 * h), x[j].at(2 * h + 1));
    }
    if (holds) {
#pragma unroll
      for (int j = 0; j < ST; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) st2(a.s0 + (unit * dp + d0 + h) * a.vp + v0 + 8 * (j0 + j) + 2 * t4, S[j][2 * h], S[j][2 * h + 1]);
    }
    late = __syncthreads_or(late);
#pragma unroll
    for (int i = tid; i < C * CB; i += STATE_THREADS) {      // U = U0 - W S_0, element i of [NT][C][8]
      const int t = (i >> 3) & (C - 1), col = (i / (8 * C)) * 8 + (i & 7);
      float x = parts[t * LDX + col];
#pragma unroll
      for (int q = 1; q < PARTS; ++q) x += parts[(q * C + t) * LDX + col];
      const float y = late ? NAN : cur[at.u + i] - x;
      a.u[unit * C * a.vp + (size_t)v0 * C + i] = y;
      us[t * LDU + col] = y;
    }
    __syncthreads();
    Sum more[ST];
    if (adds) {      // S = diag(P_C) S_0 + K^^T U
      constexpr int KU = NT > 1 ? C : C / 2;
      const int k0 = NT > 1 ? 0 : (warp >> 3) * KU;
#pragma unroll
      for (int k = 0; k < KU; k += 8) {
        Two x[4];
        load_a_transposed(x, cur + at.k + (k0 + k) * ld + 16 * (warp & 7), ld, g, t4);
#pragma unroll
        for (int j = 0; j < ST; ++j) {
          Two y[2];
          load_b(y, us + (k0 + k) * LDU + 8 * (j0 + j), LDU, g, t4);
          mma3(more[j], x, y);
        }
      }
    }
    if (NT == 1) {
      if (warp >= 8) st4(parts + ((warp & 7) * 32 + lane) * 4, make_float4(more[0].at(0), more[0].at(1), more[0].at(2), more[0].at(3)));
      __syncthreads();
      if (warp < 8) {
        const float4 x = ld4(parts + (warp * 32 + lane) * 4);
        add2(more[0].c[0], more[0].c[1], x.x, x.y);
        add2(more[0].c[2], more[0].c[3], x.z, x.w);
      }
    }
    if (holds) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float p = cur[at.p + d0 + h], p_low = cur[at.p + dp + d0 + h];
#pragma unroll
        for (int j = 0; j < ST; ++j)
#pragma unroll
          for (int e = 2 * h; e < 2 * h + 2; ++e) S[j][e] = decayed(S[j][e], p, p_low, more[j].at(e));
      }
      keep();
    }
    __syncthreads();      // everyone is done with this stage before the fetch after next fills it
  }
  if (holds) {
#pragma unroll
    for (int j = 0; j < ST; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = d0 + (e >> 1), c = v0 + 8 * (j0 + j) + 2 * t4 + (e & 1);
        if (d < a.dim && c < a.vdim) st[(size_t)d * a.vdim + c] = late ? NAN : S[j][e];
      }
  }
  if (tid == 0) say_late(late, a.status);
}

// -------------------------------------------------------------------------------------------------------------- out

// Three sums of up to 64 inner values each, one after the other: Q~ S_0 over the lower half of the channels, over the upper, A U over the
// tokens.  Their operands take turns in two buffers, so three blocks share an SM (with all operands there at once two blocks did: linear
// attention, 29 chunks of 16 heads of 128 x 128, 37 us).
constexpr int LDL = C + 8, LDV = OB + 4, OUT_THREADS = 128;
constexpr int OUT_BUFFER = C * LDL + C * LDV;
static_assert(CHUNK_MAX_DIM / 2 <= C, "half of the channels fit a buffer");
constexpr size_t OUT_SMEM = 2 * OUT_BUFFER * sizeof(float);

// A warp 32 tokens x 32 columns: four operand halves split in two parts serve 24 products; with 16 x 32 a warp the splitting took
// half of the instructions.
template <bool DELTA>
__global__ void __launch_bounds__(OUT_THREADS, 3)
chunk_out_kernel(Args a) {
  extern __shared__ __align__(16) float sm[];
  const int dp = a.dp, half = dp / 2;
  __shared__ int found[2];
  __shared__ __align__(8) uint64_t bars[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3, head = blockIdx.y, v0 = blockIdx.z * OB;
  if (tid == 0) {
    find_chunk(a, a.c0 + blockIdx.x, found[0], found[1]);
    for (int b = 0; b < 3; ++b) bar_init(bars + b);
    bars_ready();
  }
  mi::grid_dependency_sync();
  __syncthreads();
  const int item = found[0];
  if (item < 0) return;
  const int first = found[1] * C, n = min(C, a.q_len[item] - first), row0 = a.q_start[item] + first;
  const size_t unit = (size_t)blockIdx.x * a.heads + head;
  // Three rounds of 64 rows of the left side and up to 64 of the right, a thread a row of one of them; no values behind the last token
  auto fetch = [&](int part) {
    float* buf = sm + (part & 1) * OUT_BUFFER;
    const int r = tid & (C - 1), columns = min(OB, (DELTA || part < 2 ? a.vp : a.vdim) - v0), rows = part < 2 ? half : DELTA ? C : n;
    if (tid == 0) bar_expect(bars + part, (C * (part < 2 ? half : C) + rows * columns) * 4);
    if (tid < C) {
      if (part < 2) bulk_copy(buf + r * LDL, a.qt + (unit * C + r) * dp + part * half, half, bars + part);
      else bulk_copy(buf + r * LDL, a.at + (unit * C + r) * C, C, bars + part);
    } else {
      float* to = buf + C * LDL + r * LDV;
      if (r >= rows) {
#pragma unroll 1
        for (int c = 0; c < OB; c += 4) st4(to + c, make_float4(0.f, 0.f, 0.f, 0.f));
      } else if (part < 2) {
        bulk_copy(to, a.s0 + (unit * dp + part * half + r) * a.vp + v0, columns, bars + part);
      } else if (!DELTA) {
        bulk_copy(to, a.raw + (size_t)(row0 + r) * (a.heads * a.vdim) + head * a.vdim + v0, columns, bars + part);
      } else if (8 * r < columns) {      // (groups of eight columns of all tokens)
        bulk_copy(buf + C * LDL + r * 8 * C, a.u + unit * C * a.vp + (size_t)(v0 + 8 * r) * C, 8 * C, bars + part);
      }
    }
  };
  const int m0 = (warp & 1) * 32, n0 = (warp >> 1) * 32;
  Sum sum[2][4];
  auto multiply = [&](const float* buf, int k_end, int ldr, int next, auto plain) {      // plain: the right side is what tf32 holds
#pragma unroll 1
    for (int k = 0; k < k_end; k += 8) {      // eight inner values, in the order 0 2 4 6 1 3 5 7
      Two x[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) load_a_pairs(x[i], buf + (m0 + 16 * i) * LDL + k, LDL, g, t4);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float* r = buf + C * LDL + (k + 2 * t4) * ldr + (n0 / 8 + j) * next + g;
        if (plain.value) {
#pragma unroll
          for (int i = 0; i < 2; ++i) mma2(sum[i][j], x[i], r[0], r[ldr]);
        } else {
          Two y[2];
          split2(y[0], y[1], r[0], r[ldr]);
#pragma unroll
          for (int i = 0; i < 2; ++i) mma3(sum[i][j], x[i], y);
        }
      }
    }
  };
  fetch(0);
  fetch(1);
  bool late = false;
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {
    late |= !bar_wait(bars + part, 0);
    multiply(sm + part * OUT_BUFFER, half, LDV, 8, std::false_type());
    if (part == 0) {
      bulk_may_follow();
      __syncthreads();
      fetch(2);
    }
  }
  late |= !bar_wait(bars + 2, 0);
  __syncthreads();      // (the zeros behind the last token)
  multiply(sm, m0 + 32, DELTA ? 8 : LDV, DELTA ? 8 * C : 8, std::integral_constant<bool, !DELTA>());      // A U: nothing behind the diagonal; linear attention's U are the values
  late = __any_sync(0xffffffffu, late);
  float* o = a.raw + (size_t)row0 * (a.heads * a.vdim) + head * a.vdim + v0;
  unsigned bad = 0;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float x[4] = {sum[i][j].at(0), sum[i][j].at(1), sum[i][j].at(2), sum[i][j].at(3)};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = m0 + 16 * i + g + 8 * h, c = n0 + 8 * j + 2 * t4;
        if (t < n && v0 + c < a.vdim) st2(o + (size_t)t * (a.heads * a.vdim) + c, late ? NAN : x[2 * h], late ? NAN : x[2 * h + 1]);
      }
      bad |= any_not_finite(x) && !late ? 15u << 4 * (4 * i + j) : 0;
    }
  const float *aa = sm, *us = sm + C * LDL;
#pragma unroll 1
  for (; bad; bad &= bad - 1) {
    const int b = __ffs(bad) - 1, e = b & 3, t = m0 + 16 * (b >> 4) + g + 8 * (e >> 1), c = n0 + 8 * (b >> 2 & 3) + 2 * t4 + (e & 1);
    if (t >= n || v0 + c >= a.vdim) continue;
    float y = 0.f, z = 0.f;
#pragma unroll 1
    for (int d = 0; d < a.dim; ++d) y = fmaf(a.qt[(unit * C + t) * dp + d], a.s0[(unit * dp + d) * a.vp + v0 + c], y);
#pragma unroll 1
    for (int s = 0; s <= t; ++s) z = fmaf(aa[t * LDL + s], DELTA ? us[(c / 8 * C + s) * 8 + (c & 7)] : us[s * LDV + c], z);
    o[(size_t)t * (a.heads * a.vdim) + c] = fabsf(z) <= 3.402823466e38f ? y + z : NAN;      // an infinite value: the recurrence adds it up over channels of both signs
  }
  if (lane == 0) say_late(late, a.status);
}

int most_chunks(int T, int items) { return T / C + items; }      // every item's last chunk may be a short one
int slab_chunks(int heads, int dim, int vdim, bool delta) {
  const long long n = SLAB_FLOATS / (heads * unit_floats(pad(dim, 32), pad(vdim, 32), delta));
  return n < 1 ? 1 : n < 65535 ? (int)n : 65535;
}

// Blocks of a kernel for which every SM has room twice are put two to an SM even where there are SMs for all, while the kernel before still has
// some, and the kernel then takes half as long again (chunk_build 24.7 us instead of 16.3): as many blocks as SMs or fewer ask for more shared memory
// than two of them find.  The operation, linear attention, a constant a head, one request, 8 heads of 160 tokens 45.0 -> 31.4 us, 16 of 64 42.4 -> 30.9,
// 32 of 160 49.2 -> 40.8; delta rule, a decay a channel, 16 heads of 112 58.1 -> 44.7.
constexpr size_t ALONE_SMEM = 115 * 1024;
size_t alone(size_t smem, long long blocks) { return blocks <= mi::sm_count() ? std::max(smem, ALONE_SMEM) : smem; }

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
  a.kh = a.w + (delta ? units * C * row_floats(a.dp) : 0);
  a.u = a.kh + (delta ? units * C * row_floats(a.dp) : 0);
  a.at = a.u + (delta ? units * C * a.vp : 0);
  a.qt = a.at + units * C * C;
  a.s0 = a.qt + units * C * a.dp;
  a.pc = a.s0 + units * a.dp * a.vp;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !configured[dev]) {
    const size_t build = std::max(BuildLayout(CHUNK_MAX_DIM).floats * sizeof(float), ALONE_SMEM), out = std::max(OUT_SMEM, ALONE_SMEM);
    if (!allow(chunk_build_kernel<true>, build) || !allow(chunk_build_kernel<false>, build) || !allow(chunk_out_kernel<true>, out) ||
        !allow(chunk_out_kernel<false>, out) || !allow(chunk_state_kernel<8>, StateLayout<8>(CHUNK_MAX_DIM).bytes()) ||
        !allow(chunk_state_kernel<16>, StateLayout<16>(CHUNK_MAX_DIM).bytes()) || !allow(chunk_state_kernel<32>, StateLayout<32>(CHUNK_MAX_DIM).bytes()))
      return mi_fail("chunked_state: the shared memory was refused");
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  // Value columns of a chunk_state block: as few as still put every block on an SM of its own, 32 where none does
  auto blocks = [&](int cb) { return (long long)in.heads * in.items * (a.vp / cb); };
  const int cb = blocks(8) <= mi::sm_count() ? 8 : blocks(16) <= mi::sm_count() ? 16 : 32;
  for (int c0 = 0; c0 < total; c0 += slab) {
    a.c0 = c0;
    a.c1 = c0 + slab < total ? c0 + slab : total;
    mi::launch(delta ? chunk_build_kernel<true> : chunk_build_kernel<false>, dim3(a.c1 - a.c0, in.heads), dim3(THREADS),
               alone(BuildLayout(a.dp).floats * sizeof(float), (long long)(a.c1 - a.c0) * in.heads), stream, a);
    const dim3 grid(in.heads, a.vp / cb, in.items);
    if (!delta)
      mi::launch(chunk_scan_kernel, dim3((a.dp * a.vp / 4 + SCAN_THREADS - 1) / SCAN_THREADS, in.heads, in.items), dim3(SCAN_THREADS), 0, stream, a);
    else if (cb == 8)
      mi::launch(chunk_state_kernel<8>, grid, dim3(STATE_THREADS), StateLayout<8>(a.dp).bytes(), stream, a);
    else if (cb == 16)
      mi::launch(chunk_state_kernel<16>, grid, dim3(STATE_THREADS), StateLayout<16>(a.dp).bytes(), stream, a);
    else
      mi::launch(chunk_state_kernel<32>, grid, dim3(STATE_THREADS), StateLayout<32>(a.dp).bytes(), stream, a);
    mi::launch(delta ? chunk_out_kernel<true> : chunk_out_kernel<false>, dim3(a.c1 - a.c0, in.heads, (a.vp + OB - 1) / OB), dim3(OUT_THREADS),
               alone(OUT_SMEM, (long long)(a.c1 - a.c0) * in.heads * ((a.vp + OB - 1) / OB)), stream, a);
  }
  MI_LAUNCH_OK("chunked_state");
  return 0;
}

}  // namespace mi
