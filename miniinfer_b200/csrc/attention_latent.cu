// Attention of many query heads over ONE shared key/value head whose values are the first columns of its keys - attention
// through a latent - in bf16 on the fifth-generation tensor cores (tcgen05), for key rows of 64 to 256 values.
//
// The query rows of the step lie behind one another, [token, head], so a piece of work is any 128 of them that belong to one
// request - 8 tokens of 16 heads -: all heads of a token see the same keys, so nearly no product is done above the
// diagonal, and a key tile is fetched once for 128 rows.  A tile is 128 keys; its rows serve the scores as they lie (K-major) and,
// their first out_hd columns, the weighted values (MN-major): one copy of a row where keys and values of their own are two, which
// is what lets two whole tiles of 64 KB wait in shared memory beside the 64 KB of the work's queries.
//
// Blocks are persistent, one per SM, works dealt out longest first in rounds that go back and forth; barrier phases run on across
// works.  Roles of a block: a producer thread (Q of a work, key tiles into two stages, by TMA in the 128-byte swizzle), a thread
// that issues all products, eight softmax warps.  Tensor memory: the output row (256 columns) and two buffers of scores, which
// take turns: the softmax leaves a tile's weights in the buffer that held its scores; scores are computed two tiles ahead.  Two threads
// share a row of scores, 64 each, and agree on its maximum through shared memory; the output row is rescaled when the maximum of one
// of a warp's 32 rows has moved.
//
// The weights are rounded to bf16 for P V, and that is what a row errs by beside its own last rounding.  The weight of the row's
// maximum is exactly 1 - a maximum that may lag by 2^8 would save most rescalings, and 2 us of 55, but rounds the heaviest
// weight too -, and the sum that divides the row is that of the rounded weights.  2048 tokens, scores of standard deviation 4: 1.72e-3
// of the norm (with a lagging maximum and unrounded sums 2.07e-3, the mma.sync kernel 1.72e-3).  A decode token, of whose tiles most is
// latency, takes its weights in two bf16 parts, P V twice: 1.66e-3 for 2048 keys (1.80e-3 in one part, the mma.sync kernel 1.74e-3).
//
// Rows that no row of a work may see - behind its last key, before its window: another request's, or never written - must not be
// multiplied, for a weight of zero times an infinity is a NaN: P V leaves out whole sixteens of such keys, and the softmax warps zero
// what is left of them in shared memory (at most 30 rows, in a work's first and last tile), once their registers are free: 51.2 us
// for 2048 tokens where reading them all took 50.6; before the exponentials the same lines took 53.0, in a warp of its own 52.8.
// Keys that some rows of a work see and others do not are multiplied for all: a number that is not finite there reaches up to 127
// rows before its own, as it reached the other rows of a tile of 64 tokens in the mma.sync kernel.
//
// What bounds it: a tile's stage is given back by its P V, so the copy of the tile after next and its S lie on a chain of about 6800
// cycles for two tiles, of which the products are 4600 (clock stamps).  Tiles of 64 keys in four stages are no faster: a product
// of 128 x 64 x 16 takes 81 cycles where one of 128 x 128 x 16 takes 95.  Neither the exponentials nor the copies from L2 matter (left
// out in turn: no change).  (Stamps and trials, 51 us, are of the form whose maximum lagged and that read all rows.)  Measured on B200, 2048
// tokens, latent 192 + 32: 16 heads 55 us, 232 by the mma.sync kernel; 1000 tokens of 32 heads of 192 + 64 with a window of 1024 35 us,
// 149 by that.
//
// (Pairs of values in one instruction - f32x2, a maximum of three - in the prompt's form: 55.1 -> 52.5 us at 2048 tokens.  The decode form is
// left at its registers: at 142 instead of 168 a block leaves room for the next kernels beside it, which then find the SMs unevenly
// taken, and a decode step of 8 tokens of 32 heads took 54 us instead of 48.)
//
// Decode tokens run through the same tiles: a work is one request's up to 128 heads and a piece of its keys, counted from key 0, and
// leaves sums that are not normalised for latent_merge_kernel.  Most of the 128 rows are padding, which costs nothing: a piece is bound
// by the latency of its one or two tiles and by bytes, and every key row is fetched once for all heads, as key and as value
// at once.  Measured on B200, 8 tokens of 32 heads of 192 + 64 over 2048 keys each: the layer around them 87.7 us with the
// mma.sync kernel of attention_decode.cu (16 heads a pass, keys and values fetched apart: 40.6 us, its merge 6.3), 51.2 so.
//
// (the mma.sync kernel of attention_prefill.cu takes the other forms: keys and values of their own, pages that are no multiple
// of 64, sizes of other alignment).
#include <cuda.h>
#include <string.h>

#include "attention_scores.cuh"
#include "common.cuh"

namespace {

constexpr int BM = 128, BN = 128;             // query rows of a work, keys of a tile
constexpr int STAGES = 2;                     // key tiles in shared memory, and buffers of scores in tensor memory
constexpr int BOX = 64;                       // columns of a TMA box: 128 bytes
constexpr int Q_COL_BYTES = BM * 128, K_COL_BYTES = BN * 128;      // the rows of one box of columns
constexpr int SOFTMAX_WARPS = 8, PRODUCER_WARP = 8, MMA_WARP = 9, THREADS = 320;
constexpr int TMEM_COLS = 512, O_COL = 0, S_COL = 256;      // scores of tile g at S_COL + BN (g % STAGES), its weights over the first half of them
constexpr int WAIT_LIMIT = 1 << 22;

struct Args {
  __nv_bfloat16* out;            // [T * nh, out_hd]
  const int* block_table; int bt_stride;
  const int* tiles;              // [n_tiles, 2]: item, first of 64 new tokens
  const int *q_start, *q_len, *ctx_len, *seq_slot;
  int* status;
  int n_tiles, nh, page_size, window;
  int boxes, steps, n_out, out_hd;      // boxes and 16s of columns of a row, columns of P V (whole boxes), of which out_hd are stored
  float scale_log2;              // scale * log2(e)
  const float* sink;             // [nh] or null
  // decode tokens: a piece of chunk keys (counted from key 0) of one request and up to 128 of its heads is a work
  const int* decode_items;       // [n_dec]: item of each decode entry
  float *part_o, *part_ml;       // [n_dec, max_splits, nh, out_hd] not normalised; [n_dec, max_splits, nh, 2]: base-2 maximum, sum
  int n_dec, chunk, max_splits;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait.  `abort` is a flag in shared memory: once any wait has run out, all waits return.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* status) {
  const uint32_t addr = smem_u32(bar);
  for (int i = 0; i < WAIT_LIMIT; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    if (done) return;
    if ((i & 63) == 63 && *abort) return;
  }
  *abort = 1;
  atomicExch(status, 2);
}
__device__ __forceinline__ void tma_load(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// The barrier gets an arrival when all products issued so far by this thread are done.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], and with A in tensor memory (lane = row, two bf16 of consecutive k to a column).
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 consecutive columns of this thread's lane, written.
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
// N consecutive columns of this thread's lane (lane = 32 * (warp % 4) + lane of the warp), read.
__device__ __forceinline__ void tmem_ld(float (&v)[32], uint32_t taddr) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld(float (&v)[64], uint32_t taddr) {
  uint32_t r[64];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}
// Shared-memory operand descriptor, 128-byte swizzle: start address, leading and stride byte offsets in 16-byte units,
// descriptor version 1 (bits 46..47), layout type 2 = 128-byte swizzle (bits 61..63).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor of kind::f16: float32 accumulator (bits 4..5 = 1), bf16 A and B (bits 7..9 and 10..12 = 1), B K-major or
// MN-major (bit 16), N / 8 at bits 17..22, M / 16 at bits 24..28.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// 128 query rows of one request and the key tiles that they see.
struct Work {
  int rows;                      // of the 128 that exist; 0: none
  int row0, first;               // first row in the step's [token, head] rows; the same counted from the item's first new token's
  int start, p_first, p_last, lo_first, lo_last, t_begin, n;
  int slot;                      // decode: entry and piece, entry * max_splits + piece
  const int* bt;
};

// Work number w of the step, longest first: the parts of the last 64 tokens, last to first, then of the 64 before, ...
__device__ __forceinline__ Work work_of(const Args& a, int w, int per_tile) {
  Work k;
  const int tile = a.n_tiles - 1 - w / per_tile, part = per_tile - 1 - w % per_tile;
  const int item = a.tiles[2 * tile], o = a.tiles[2 * tile + 1];
  const int q_len = a.q_len[item], ctx = a.ctx_len[item];
  k.rows = min(BM, min(64, q_len - o) * a.nh - part * BM);
  k.start = ctx - q_len;
  k.first = o * a.nh + part * BM;
  k.row0 = a.q_start[item] * a.nh + k.first;
  k.p_first = k.start + k.first / a.nh;
  k.p_last = k.start + (k.first + max(k.rows, 1) - 1) / a.nh;
  k.lo_last = mi::first_visible(k.p_last, a.window);
  k.lo_first = mi::first_visible(k.p_first, a.window);
  k.t_begin = k.lo_first / BN;
  k.n = k.p_last / BN - k.t_begin + 1;
  k.slot = 0;
  k.bt = a.block_table + (size_t)a.seq_slot[item] * a.bt_stride;
  return k;
}
// Of decode tokens: the first piece of every request, then the second, ...
__device__ __forceinline__ Work decode_work_of(const Args& a, int w, int parts) {
  Work k;
  const int part = w % parts, entry = w / parts % a.n_dec, split = w / parts / a.n_dec;
  const int item = a.decode_items[entry];
  const int p = a.ctx_len[item] - 1, lo = mi::first_visible(p, a.window), piece = lo / a.chunk + split;
  k.rows = p >= 0 && piece * a.chunk <= p ? min(BM, a.nh - part * BM) : 0;
  k.first = part * BM;
  k.row0 = a.q_start[item] * a.nh + k.first;
  k.start = k.p_first = k.p_last = p;
  k.lo_first = k.lo_last = lo;
  k.t_begin = max(lo, piece * a.chunk) / BN;
  k.n = min(p, (piece + 1) * a.chunk - 1) / BN - k.t_begin + 1;
  k.slot = entry * a.max_splits + split;
  k.bt = a.block_table + (size_t)a.seq_slot[item] * a.bt_stride;
  return k;
}
// The keys of the tile from key0 on that some row of the work sees: the first, and one past the last.
__device__ __forceinline__ int2 seen_keys(const Work& k, int key0) { return make_int2(max(k.lo_first - key0, 0), min(k.p_last + 1 - key0, BN)); }
// The i-th work of block b: rounds that go back and forth, so that the block with the longest work of one round gets the
// shortest of the next.  -1 past the end.
__device__ __forceinline__ int nth_work(int i, int b, int blocks, int total) {
  const int w = i * blocks + ((i & 1) ? blocks - 1 - b : b);
  return w < total ? w : -1;
}

template <bool DECODE>
__global__ void __launch_bounds__(THREADS, 1)
attention_latent_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map, Args a) {
  const int per_tile = ((DECODE ? 1 : 64) * a.nh + BM - 1) / BM, total = per_tile * (DECODE ? a.n_dec * a.max_splits : a.n_tiles);
  const int blocks = gridDim.x, me = blockIdx.x;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int q_bytes = a.boxes * Q_COL_BYTES, tile_bytes = a.boxes * K_COL_BYTES;
  unsigned char *q_s = smem, *k_s = smem + q_bytes;         // [STAGES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(k_s + STAGES * tile_bytes);
  uint64_t *q_full = bars, *q_empty = bars + 1, *o_free = bars + 2;
  uint64_t *k_full = bars + 3, *k_empty = k_full + STAGES;  // of a tile: copied; read by S and by P V
  uint64_t *s_full = k_empty + STAGES, *p_full = s_full + STAGES, *o_full = p_full + STAGES;      // of a tile: S computed, weights written and rows zeroed, P V added
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + STAGES);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* row_max = reinterpret_cast<float*>(bars + 32);     // [2 tiles][2 halves][BM]; at a work's end the halves' sums in [half][BM] behind
  float* row_sum = row_max + 4 * BM;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    mbar_init(o_free, SOFTMAX_WARPS);
    for (int b = 0; b < STAGES; ++b) {
      mbar_init(&k_full[b], 1);
      mbar_init(&k_empty[b], 1);
      mbar_init(&s_full[b], 1);
      mbar_init(&p_full[b], SOFTMAX_WARPS);
      mbar_init(&o_full[b], 1);
    }
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  mi::grid_dependency_sync();

  // Tiles are counted over the block's works: tile g has stage, score buffer and barriers g % STAGES, use g / STAGES of them.
  if (warp == PRODUCER_WARP) {
    if (lane == 0) {
      int g = 0, it = 0;
      for (int i = 0;; ++i) {
        const int w = nth_work(i, me, blocks, total);
        if (w < 0 || *abort) break;
        const Work k = DECODE ? decode_work_of(a, w, per_tile) : work_of(a, w, per_tile);
        if (k.rows <= 0) continue;
        mbar_wait(q_empty, (it & 1) ^ 1, abort, a.status);
        mbar_expect_tx(q_full, (uint32_t)q_bytes);
        for (int c = 0; c < a.boxes; ++c)
          for (int r = 0; r < 2; ++r) tma_load(q_s + c * Q_COL_BYTES + r * 64 * 128, &q_map, c * BOX, k.row0 + 64 * r, q_full);
        for (int j = 0; j < k.n && !*abort; ++j, ++g) {
          const int b = g % STAGES;
          mbar_wait(&k_empty[b], ((g / STAGES) & 1) ^ 1, abort, a.status);
          mbar_expect_tx(&k_full[b], (uint32_t)tile_bytes);
          for (int r = 0; r < BN; r += 64) {
            const int key = (k.t_begin + j) * BN + r;
            const int page = k.bt[min(key / a.page_size, a.bt_stride - 1)];      // past the context: the dummy page, masked below
            const int y = page * 2 * a.page_size + key % a.page_size;            // a page's keys, then its values
            for (int c = 0; c < a.boxes; ++c) tma_load(k_s + b * tile_bytes + c * K_COL_BYTES + r * 128, &kv_map, c * BOX, y, &k_full[b]);
          }
        }
        ++it;
      }
    }
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      constexpr uint32_t IDESC_S = instr_desc(BM, BN, false);
      const uint32_t idesc_pv = instr_desc(BM, a.n_out, true);
      const uint64_t q_desc = smem_desc(smem_u32(q_s), 16, 1024);
      const int steps = a.steps;
      int g0 = 0, it = 0;
      for (int i = 0;; ++i) {
        const int w = nth_work(i, me, blocks, total);
        if (w < 0 || *abort) break;
        const Work k = DECODE ? decode_work_of(a, w, per_tile) : work_of(a, w, per_tile);
        if (k.rows <= 0) continue;
        auto scores = [&](int j) {
          const int g = g0 + j, b = g % STAGES;
          mbar_wait(&k_full[b], (g / STAGES) & 1, abort, a.status);      // (the stage's last P V is done then, and with it the use of its scores)
          if (*abort) return;
          tc_fence_after();
          const uint64_t k_desc = smem_desc(smem_u32(k_s + b * tile_bytes), 16, 1024);
          for (int s = 0; s < steps; ++s) {
            const int in_box = (s & 3) * 2;      // 16 columns further: 32 bytes of a row of its box
            tc_mma(tmem + S_COL + BN * b, q_desc + (uint64_t)((s >> 2) * (Q_COL_BYTES >> 4) + in_box),
                   k_desc + (uint64_t)((s >> 2) * (K_COL_BYTES >> 4) + in_box), IDESC_S, s > 0 ? 1u : 0u);
          }
          tc_commit(&s_full[b]);
          if (j == k.n - 1) tc_commit(q_empty);
        };
        mbar_wait(q_full, it & 1, abort, a.status);
        for (int j = 0; j < min(k.n, STAGES) && !*abort; ++j) scores(j);      // scores run two tiles ahead
        for (int j = 0; j < k.n && !*abort; ++j) {
          const int g = g0 + j, b = g % STAGES;
          if (j == 0 && it > 0) mbar_wait(o_free, (it - 1) & 1, abort, a.status);      // the work before has its output row in registers
          mbar_wait(&p_full[b], (g / STAGES) & 1, abort, a.status);
          if (*abort) break;
          tc_fence_after();
          const uint64_t v_desc = smem_desc(smem_u32(k_s + b * tile_bytes), K_COL_BYTES, 1024);
          auto add = [&](int s, bool onto) {      // 16 keys further: 2048 bytes of every box
            tc_mma_ts(tmem + O_COL, tmem + S_COL + BN * b + 8 * s, v_desc + (uint64_t)(s * (2048 >> 4)), idesc_pv, onto ? 1u : 0u);
            if constexpr (DECODE)
              tc_mma_ts(tmem + O_COL, tmem + S_COL + BN * b + BN / 2 + 8 * s, v_desc + (uint64_t)(s * (2048 >> 4)), idesc_pv, 1u);
          };
          if (j == 0 || j == k.n - 1) {
            const int2 keys = seen_keys(k, (k.t_begin + j) * BN);
#pragma unroll 1
            for (int s = keys.x / 16; 16 * s < keys.y; ++s) add(s, j > 0 || s > keys.x / 16);
          } else {
            for (int s = 0; s < BN / 16; ++s) add(s, true);
          }
          tc_commit(&o_full[b]);
          tc_commit(&k_empty[b]);
          if (j + STAGES < k.n) scores(j + STAGES);
        }
        g0 += k.n;
        ++it;
      }
    }
  } else {
    // Warp w: tensor-memory lanes 32 (w % 4) .. + 31, half w / 4 of their rows of scores: 64 keys a thread.
    const int quarter = warp & 3, half = warp >> 2, r = quarter * 32 + lane;
    const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
    int seen[STAGES] = {};
    auto wait_o = [&](int g) {      // P V of tile g is added
#pragma unroll
      for (int b = 0; b < STAGES; ++b)
        if (b == g % STAGES) {
          while (seen[b] <= g / STAGES) {
            mbar_wait(&o_full[b], seen[b] & 1, abort, a.status);
            ++seen[b];
          }
        }
      tc_fence_after();
    };
    auto meet = [&]() {      // the two warps that share rows
      asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
    };
    int g = 0;
    for (int i = 0;; ++i) {
      const int w = nth_work(i, me, blocks, total);
      if (w < 0) break;
      const Work k = DECODE ? decode_work_of(a, w, per_tile) : work_of(a, w, per_tile);
      if (k.rows <= 0) continue;
      const bool valid = r < k.rows;
      const int f = k.first + r, pos = valid ? k.start + f / a.nh : k.p_last, lo = mi::first_visible(pos, a.window);
      float m_run = -INFINITY, l_run = 0.f;
      for (int j = 0; j < k.n; ++j, ++g) {
        const int b = g % STAGES, key0 = (k.t_begin + j) * BN;
        const uint32_t s_addr = t_lane + S_COL + BN * b;
        mbar_wait(&s_full[b], (g / STAGES) & 1, abort, a.status);
        tc_fence_after();
        float v[BN / 2];
        tmem_ld(v, s_addr + BN / 2 * half);
        if (!(key0 + BN - 1 <= k.p_first && key0 >= k.lo_last)) {      // a tile that the mask touches
          const int first = lo - key0 - BN / 2 * half, last = pos - key0 - BN / 2 * half;
#pragma unroll
          for (int e = 0; e < BN / 2; ++e) v[e] = (e >= first && e <= last) ? v[e] : -INFINITY;
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < BN / 2; e += 2) {
          if (DECODE) {
            mx4[e & 3] = fmaxf(mx4[e & 3], v[e]);
            mx4[(e & 3) + 1] = fmaxf(mx4[(e & 3) + 1], v[e + 1]);
          } else {
            mx4[e >> 1 & 3] = mi::max_of(mx4[e >> 1 & 3], v[e], v[e + 1]);
          }
        }
        float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        float* maxima = row_max + (g & 1) * 2 * BM;
        maxima[half * BM + r] = mx;
        tc_fence_before();
        meet();      // both halves of the scores are in registers: the weights may be written over them
        tc_fence_after();
        mx = fmaxf(mx, maxima[(half ^ 1) * BM + r]);
        const float m_new = fmaxf(m_run, mx * a.scale_log2);      // the scale is positive
        const bool move = m_new > m_run;
        if (__any_sync(0xffffffffu, move)) {
          const float alpha = move ? exp2f(m_run - m_new) : 1.f;
          if (j > 0) {
            wait_o(g - 1);
#pragma unroll 1
            for (int c = half; 32 * c < a.n_out; c += 2) {
              float o[32];
              uint32_t x[32];
              tmem_ld(o, t_lane + O_COL + 32 * c);
#pragma unroll
              for (int e = 0; e < 32; e += 2) {
                if (DECODE) {
                  o[e] *= alpha;
                  o[e + 1] *= alpha;
                } else {
                  mi::mul_pair(o[e], o[e + 1], o[e], o[e + 1], alpha);
                }
                x[e] = __float_as_uint(o[e]);
                x[e + 1] = __float_as_uint(o[e + 1]);
              }
              tmem_st(t_lane + O_COL + 32 * c, x);
            }
          }
          l_run *= alpha;
          if (move) m_run = m_new;
        }
        const float m_use = m_run == -INFINITY ? 0.f : m_run;
        float part[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t packed[BN / 4];
#pragma unroll
        for (int e = 0; e < BN / 2; e += 2)
          if (!DECODE) mi::fma_pair(v[e], v[e + 1], v[e], v[e + 1], a.scale_log2, -m_use);
#pragma unroll
        for (int e = 0; e < BN / 2; ++e) v[e] = mi::ex2_fast(DECODE ? fmaf(v[e], a.scale_log2, -m_use) : v[e]);      // nothing where the row may not see the key
        if constexpr (DECODE) {      // in two bf16 parts: P V twice
          uint32_t low[BN / 4];
#pragma unroll
          for (int e = 0; e < BN / 4; ++e) {
            packed[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
            low[e] = pack_bf16(v[2 * e] - __uint_as_float(packed[e] << 16), v[2 * e + 1] - __uint_as_float(packed[e] & 0xffff0000u));
            part[2 * e & 3] += v[2 * e];
            part[(2 * e + 1) & 3] += v[2 * e + 1];
          }
          tmem_st(s_addr + BN / 2 + BN / 4 * half, low);
        } else {
#pragma unroll
          for (int e = 0; e < BN / 4; ++e) {
            packed[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
            mi::add_pair(part[2 * e & 3], part[(2 * e + 1) & 3], __uint_as_float(packed[e] << 16), __uint_as_float(packed[e] & 0xffff0000u));
          }
        }
        tmem_st(s_addr + BN / 4 * half, packed);      // two keys to a column
        if (j == 0 || j == k.n - 1) {      // the rows that nobody sees in the sixteens at the edges (S has read them): zeros before P V reads them
          const int2 keys = seen_keys(k, key0);
          if ((keys.x | keys.y) & 15) {
            if (8 * lane < a.n_out) {
              unsigned char* column = k_s + b * tile_bytes + (lane >> 3) * K_COL_BYTES + (lane & 7) * 16;
              for (int row = (keys.x & ~15) + warp; row < keys.x; row += SOFTMAX_WARPS) *reinterpret_cast<uint4*>(column + row * 128) = make_uint4(0, 0, 0, 0);
              for (int row = keys.y + warp; row < ((keys.y + 15) & ~15); row += SOFTMAX_WARPS) *reinterpret_cast<uint4*>(column + row * 128) = make_uint4(0, 0, 0, 0);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          }
        }
        l_run += (part[0] + part[1]) + (part[2] + part[3]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        if (g >= STAGES) wait_o(g - STAGES);      // long done - S of this tile came behind it -: keeps this thread in step with the barrier
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[b]);
      }
#pragma unroll
      for (int back = STAGES; back > 0; --back)
        if (g >= back) wait_o(g - back);
      row_sum[half * BM + r] = l_run;
      meet();
      if constexpr (DECODE) {
        const size_t at = (size_t)k.slot * a.nh + f;      // (of a head that exists)
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const int c = 2 * n + half;
          if (32 * c < a.n_out && quarter * 32 < k.rows) {
            float o[32];
            tmem_ld(o, t_lane + O_COL + 32 * c);
            if (valid && !*abort) {
#pragma unroll
              for (int q = 0; q < 8; ++q)
                if (32 * c + 4 * q < a.out_hd)
                  *reinterpret_cast<float4*>(a.part_o + at * a.out_hd + 32 * c + 4 * q) = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
            }
          }
        }
        if (valid && half == 0 && !*abort) *reinterpret_cast<float2*>(a.part_ml + 2 * at) = make_float2(m_run, row_sum[r] + row_sum[BM + r]);
        tc_fence_before();
        meet();      // (the sums are read too: the next work may leave its own)
        if (lane == 0) mbar_arrive(o_free);
        continue;
      }
      const float sink2 = a.sink ? a.sink[f % a.nh] * 1.4426950408889634f : -INFINITY;      // base 2, like the scores
      const float m_all = fmaxf(m_run, sink2), weight = exp2f(m_run - m_all);
      const float factor = weight / ((row_sum[r] + row_sum[BM + r]) * weight + (a.sink ? exp2f(sink2 - m_all) : 0.f));
      uint32_t o2[4][16];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int c = 2 * n + half;
        if (32 * c < a.n_out) {
          float o[32];
          tmem_ld(o, t_lane + O_COL + 32 * c);
#pragma unroll
          for (int e = 0; e < 16; ++e) o2[n][e] = pack_bf16(o[2 * e] * factor, o[2 * e + 1] * factor);
        }
      }
      tc_fence_before();
      meet();      // (the sums are read too: the next work may leave its own)
      if (lane == 0) mbar_arrive(o_free);
      if (valid && !*abort) {
        __nv_bfloat16* dst = a.out + (size_t)(k.row0 + r) * a.out_hd;
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int d = 32 * (2 * n + half) + 8 * q;
            if (d < a.out_hd) *reinterpret_cast<uint4*>(dst + d) = make_uint4(o2[n][4 * q], o2[n][4 * q + 1], o2[n][4 * q + 2], o2[n][4 * q + 3]);
          }
      }
    }
  }
  // every tensor-memory access is done, then the columns go back
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
  }
}

// The pieces of a decode token added up, a block per (request, query head) and a thread per value; pieces in ascending order.
// An entry without keys (a padded one) gets zeros.
constexpr int MERGE_PIECES = 256;      // whose factors are made a thread each, at a time
__global__ void __launch_bounds__(256)
latent_merge_kernel(Args a) {
  __shared__ float s_f[MERGE_PIECES], s_l[MERGE_PIECES];
  const int head = blockIdx.x, entry = blockIdx.y, item = a.decode_items[entry];
  const int p = a.ctx_len[item] - 1, n = p < 0 ? 0 : p / a.chunk - mi::first_visible(p, a.window) / a.chunk + 1;
  const float sink2 = a.sink ? a.sink[head] * 1.4426950408889634f : -INFINITY;      // base 2, like the scores
  mi::grid_dependency_sync();
  const float* ml = a.part_ml + 2 * ((size_t)entry * a.max_splits * a.nh + head);
  const float* po = a.part_o + ((size_t)entry * a.max_splits * a.nh + head) * a.out_hd;
  // Up to 32 pieces: a lane a piece's maximum and sum, a thread its value of eight pieces at a time, the first eight on their way with the
  // maxima (8 tokens of 32 heads in 9 pieces, behind another kernel: 5.3 us by the loops below, so 4.8)
  if (n <= 32) {
    constexpr int AT_ONCE = 8;
    const int lane = threadIdx.x & 31;
    const bool live = threadIdx.x < a.out_hd;
    float2 mine = make_float2(-INFINITY, 0.f);
    if (lane < n) mine = *reinterpret_cast<const float2*>(ml + (size_t)2 * lane * a.nh);
    float f = 0.f, m = sink2, acc = 0.f;
#pragma unroll 1
    for (int s0 = 0; s0 < n; s0 += AT_ONCE) {
      float v[AT_ONCE];
#pragma unroll
      for (int s = 0; s < AT_ONCE; ++s) v[s] = live && s0 + s < n ? po[(size_t)(s0 + s) * a.nh * a.out_hd + threadIdx.x] : 0.f;
      if (s0 == 0) {
        m = fmaxf(m, mi::warp_max(mine.x));
        f = lane < n ? exp2f(mine.x - m) : 0.f;
      }
#pragma unroll
      for (int s = 0; s < AT_ONCE; ++s)
        if (s0 + s < n) acc = fmaf(v[s], __shfl_sync(0xffffffffu, f, s0 + s), acc);
    }
    const float l = mi::warp_sum(mine.y * f) + (a.sink ? exp2f(sink2 - m) : 0.f);
    if (live) a.out[((size_t)a.q_start[item] * a.nh + head) * a.out_hd + threadIdx.x] = __float2bfloat16_rn(n > 0 ? acc * (1.f / l) : 0.f);
    return;
  }
  float m = sink2;
  for (int s = threadIdx.x & 31; s < n; s += 32) m = fmaxf(m, ml[(size_t)2 * s * a.nh]);
  m = mi::warp_max(m);
  float l = a.sink ? exp2f(sink2 - m) : 0.f, acc = 0.f;
  for (int s0 = 0; s0 < n; s0 += MERGE_PIECES) {
    const int near = min(n - s0, MERGE_PIECES);
    __syncthreads();
    for (int s = threadIdx.x; s < near; s += blockDim.x) {
      const float2 v = *reinterpret_cast<const float2*>(ml + (size_t)2 * (s0 + s) * a.nh);
      s_f[s] = exp2f(v.x - m);
      s_l[s] = v.y;
    }
    __syncthreads();
    for (int s = 0; s < near; ++s) l = fmaf(s_l[s], s_f[s], l);
    if (threadIdx.x < a.out_hd) {
#pragma unroll 16
      for (int s = 0; s < near; ++s) acc = fmaf(po[(size_t)(s0 + s) * a.nh * a.out_hd + threadIdx.x], s_f[s], acc);
    }
  }
  if (threadIdx.x < a.out_hd)
    a.out[((size_t)a.q_start[item] * a.nh + head) * a.out_hd + threadIdx.x] = __float2bfloat16_rn(n > 0 ? acc * (1.f / l) : 0.f);
}

size_t smem_bytes(int boxes) { return 1024 + (size_t)boxes * (Q_COL_BYTES + STAGES * K_COL_BYTES) + 32 * 8 + 6 * BM * sizeof(float); }

}  // namespace

// Describes rows of bf16 - [rows, width], row-major, width a multiple of 8 - to the TMA engine: boxes of 64 rows x 64 columns, 128-byte swizzle,
// zeros past the last row and column.  `out_map` receives 128 bytes.
MI_API int mi_rows_tensor_map(void* out_map, const void* base, long long rows, long long width) {
  typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
    return mi_fail("rows_tensor_map: the driver does not offer cuTensorMapEncodeTiled");
  MI_REQUIRE(((uintptr_t)base % 16) == 0 && rows > 0 && width >= BOX && width % 8 == 0, "rows_tensor_map: rows=%lld, width=%lld or the address do not fit", rows, width);
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)width * 2};
  const cuuint32_t box[2] = {BOX, 64}, elem[2] = {1, 1};
  const CUresult r = ((EncodeFn)fn)(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return mi_fail("rows_tensor_map: cuTensorMapEncodeTiled failed with code %d", (int)r);
  memcpy(out_map, &map, sizeof(map));
  return 0;
}

// q_map, kv_map: mi_rows_tensor_map of the queries [T * nh, hd] and of the layer's cache [pages * 2 * page_size, hd] (one key/value head).
// out [T * nh, out_hd].  status: one word, set to 2 if a bounded wait ran out.
static int latent_launch(Args& a, const void* q_map, const void* kv_map, int hd, long long works, cudaStream_t stream) {
  a.boxes = (hd + BOX - 1) / BOX;
  a.steps = hd / 16;
  a.n_out = (a.out_hd + BOX - 1) / BOX * BOX;
  MI_REQUIRE(hd >= 64 && hd <= 256 && hd % 16 == 0 && a.out_hd > 0 && a.out_hd <= hd && a.out_hd % 8 == 0, "attention_latent: bad head sizes %d, %d", hd, a.out_hd);
  MI_REQUIRE(a.nh > 0 && a.page_size > 0 && a.page_size % 64 == 0 && a.scale_log2 > 0.f && ((uintptr_t)a.out % 16) == 0,
             "attention_latent: nh=%d, page_size=%d, the scale or the output do not fit", a.nh, a.page_size);
  MI_REQUIRE(works <= 1 << 30, "attention_latent: %lld works of %d heads are too many for one launch", works, a.nh);
  auto kernel = a.n_dec ? attention_latent_kernel<true> : attention_latent_kernel<false>;
  static bool ready[64][2] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !ready[dev][a.n_dec > 0]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(4)) != cudaSuccess)
      return mi_fail("attention_latent: %zu bytes of shared memory were refused", smem_bytes(4));
    if (dev >= 0 && dev < 64) ready[dev][a.n_dec > 0] = true;
  }
  CUtensorMap qm, km;
  memcpy(&qm, q_map, sizeof(qm));
  memcpy(&km, kv_map, sizeof(km));
  const int blocks = (int)(works < mi::sm_count() ? works : mi::sm_count());
  // the shared memory of four boxes at any size: a block then has its SM's tensor memory to itself
  if (mi::launch(kernel, dim3(blocks), dim3(THREADS), smem_bytes(4), stream, qm, km, a) != cudaSuccess)
    return mi_fail("attention_latent: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
  return 0;
}

MI_API int mi_attention_prefill_latent(void* out, const void* q_map, const void* kv_map, const int* block_table, int bt_stride, const int* tiles,
                                       int n_tiles, const int* q_start, const int* q_len, const int* ctx_len, const int* seq_slot, int* status,
                                       int nh, int hd, int out_hd, int page_size, float scale, int window, const float* sink, cudaStream_t stream) {
  MI_REQUIRE(n_tiles >= 0, "attention_prefill_latent: n_tiles=%d", n_tiles);
  if (n_tiles == 0) return 0;
  Args a{(__nv_bfloat16*)out, block_table, bt_stride, tiles, q_start, q_len, ctx_len, seq_slot, status, n_tiles, nh, page_size, window,
         0, 0, 0, out_hd, scale * 1.4426950408889634f, sink, nullptr, nullptr, nullptr, 0, 0, 0};
  const int code = latent_launch(a, q_map, kv_map, hd, (64ll * nh + BM - 1) / BM * n_tiles, stream);
  if (code != 0) return code;
  MI_LAUNCH_OK("attention_prefill_latent");
  return 0;
}

// One new token of each of the items decode_items[n_dec].  chunk: keys of a piece, a multiple of 128; max_splits: at least the pieces of any
// entry.  scratch: n_dec * max_splits * nh * (out_hd + 2) floats, 16-byte aligned.
MI_API int mi_attention_decode_latent(void* out, const void* q_map, const void* kv_map, const int* block_table, int bt_stride, const int* decode_items,
                                      int n_dec, const int* q_start, const int* ctx_len, const int* seq_slot, int* status, float* scratch, int nh,
                                      int hd, int out_hd, int page_size, float scale, int window, const float* sink, int chunk, int max_splits,
                                      cudaStream_t stream) {
  MI_REQUIRE(n_dec >= 0 && n_dec <= 65535 && max_splits > 0 && chunk > 0 && chunk % BN == 0 && ((uintptr_t)scratch % 16) == 0,
             "attention_decode_latent: %d entries, chunk %d, %d pieces or the scratch do not fit", n_dec, chunk, max_splits);
  if (n_dec == 0) return 0;
  Args a{(__nv_bfloat16*)out, block_table, bt_stride, nullptr, q_start, nullptr, ctx_len, seq_slot, status, 0, nh, page_size, window,
         0, 0, 0, out_hd, scale * 1.4426950408889634f, sink, decode_items, scratch, scratch + (size_t)n_dec * max_splits * nh * out_hd,
         n_dec, chunk, max_splits};
  const int code = latent_launch(a, q_map, kv_map, hd, (long long)(nh + BM - 1) / BM * n_dec * max_splits, stream);
  if (code != 0) return code;
  if (mi::launch(latent_merge_kernel, dim3(nh, n_dec), dim3((out_hd + 31) / 32 * 32), 0, stream, a) != cudaSuccess)
    return mi_fail("attention_decode_latent: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
  MI_LAUNCH_OK("attention_decode_latent");
  return 0;
}
