// Attention over the paged cache in true float32, for softmax weights (sink, output gate, window or chunks, kept first keys).
//
// What attention_generic.cu computes, for rows that share their keys: a block takes up to 32 (token, query head) rows of one
// key/value head, brings the keys and values 32 at a time into shared memory by cp.async (two stages) and uses them for all
// of its rows, where the generic kernel reads them from L2 again for every token and head.  A warp has eight rows: a lane
// is two keys of four of them while the scores are made, and four output columns (or eight) while the values are weighed.
//
// The order of the arithmetic of a row depends on its position, the window and keep_first alone.  Its visible keys are cut into segments of
// 256 keys at multiples of 256 (first those of the kept first keys, then those of the window or of all earlier keys); a
// segment is walked in chunks of 32 with an online softmax of its own, and the segments' results are merged in order.  So the
// blocks of a cluster can take the segments of a row side by side - eight at a time, each leaving its maxima, sums and output
// rows in its shared memory for the block that owns a row - and the result is bit-equal whatever the number of blocks, however
// the request was cut into steps and whatever else is in the batch.
//
// What bounds it: for prompt portions the reads of shared memory and two blocks an SM (six reads of 16 bytes a lane for 16 packed
// FMAs of scores, three for 32 FMAs of values), for single tokens, whose segments four warps walk together, the latency of a chunk's scores.
// Measured on B200, 16 / 8 heads of 128, microseconds in the generic kernel and here: 300 new tokens 179 -> 75 (85 with a key a
// lane for all eight rows), 400 behind 1600 others 2850 -> 551 (605), one token behind 700 248 -> 23, eight tokens behind 2000 each 1484 -> 62.
#include <cooperative_groups.h>

#include <type_traits>

#include "attention_scores.cuh"
#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int CHUNK = 32, SEG = 256;

struct F32Args {
  float* out; const float* q; int q_stride;
  const float* kv; const int* block_table; int bt_stride;
  const int* items;                     // prefill: (item, first row) pairs, one for `tile_rows` tokens; decode: items
  const int* q_start; const int* q_len; const int* ctx_len; const int* seq_slot;
  int subtiles, tile_rows, tokens;      // prefill: blocks a pair, its tokens, tokens of a block; decode: subtiles 0
  int nh, nkv, hd, page_size; float scale; int window, keep_first;
  const float* sink; const float* gate; int gate_stride, out_hd, gate_per_head;
  int cluster;
};

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// RW: rows of a warp.  NV: groups of 128 values that hold a head.
template <int WARPS, int RW, int NV>
struct Layout {
  static constexpr int ROWS = WARPS * RW;
  int ldk;
  __host__ __device__ explicit Layout(int hd) : ldk(hd + 4) {}
  // float offsets; the segment's results lie where its keys were staged
  __host__ __device__ int keys(int stage) const { return stage * CHUNK * ldk; }
  __host__ __device__ int values(int stage) const { return 2 * CHUNK * ldk + stage * CHUNK * (ldk - 4); }
  __host__ __device__ int queries() const { return 2 * CHUNK * (2 * ldk - 4); }
  __host__ __device__ int weights() const { return queries() + ROWS * ldk; }      // of a warp: [key][row], then the rows' factors
  __host__ __device__ int running() const { return weights() + WARPS * (CHUNK + 1) * 8; }
  __host__ __device__ int floats() const { return running() + ROWS * (ldk - 4) + 4 * ROWS; }
};

template <int WARPS, int RW, int NV>
__global__ void __launch_bounds__(32 * WARPS)
attention_f32_kernel(const F32Args a) {
  using L = Layout<WARPS, RW, NV>;
  constexpr int ROWS = L::ROWS, THREADS = 32 * WARPS, HALF = 4;
  static_assert(RW == 2 * HALF, "");
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const L at(a.hd);
  const int hd = a.hd, group = a.nh / a.nkv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int unit = blockIdx.x / a.cluster, rank = blockIdx.x % a.cluster, kvh = blockIdx.y;

  // the rows: row i is token tok0 + i / group of the item, query head kvh * group + i % group
  int item, tok0 = 0, ntok = 1;
  if (a.subtiles) {
    const int pair = unit / a.subtiles, sub = unit % a.subtiles;
    item = a.items[2 * pair];
    tok0 = a.items[2 * pair + 1] + sub * a.tokens;
    ntok = min(a.tokens, min(a.tile_rows - sub * a.tokens, a.q_len[item] - tok0));
  } else {
    item = a.items[unit];
  }
  const int row0 = a.q_start[item], p0 = a.ctx_len[item] - a.q_len[item] + tok0;
  const int* bt = a.block_table + (size_t)a.seq_slot[item] * a.bt_stride;
  mi::grid_dependency_sync();
  if (ntok <= 0) return;      // the whole cluster: beyond the item's end
  const int rows = ntok * group, p_max = p0 + ntok - 1;

  float* run_o = sm + at.running();
  float *run_m = run_o + ROWS * hd, *run_l = run_m + ROWS, *part_m = run_l + ROWS, *part_l = part_m + ROWS;
  float* part_o = sm;
  for (int i = threadIdx.x; i < ROWS * (hd / 4); i += THREADS) {
    const int r = i / (hd / 4), d = (i % (hd / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) v = *reinterpret_cast<const float4*>(a.q + (size_t)(row0 + tok0 + r / group) * a.q_stride + (size_t)(kvh * group + r % group) * hd + d);
    *reinterpret_cast<float4*>(sm + at.queries() + r * at.ldk + d) = v;
    *reinterpret_cast<float4*>(run_o + r * hd + d) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int r = threadIdx.x; r < ROWS; r += THREADS) {
    run_m[r] = a.sink && r < rows ? a.sink[kvh * group + r % group] : -INFINITY;
    run_l[r] = a.sink ? 1.f : 0.f;
  }

  // Of a chunk's scores a lane makes those of four of its warp's rows and two keys, sixteen apart.  Lanes i and i ^ 1 then read the same keys and lanes i and
  // i ^ 2 the same rows, and a 16-byte read of either takes two cycles of shared memory instead of four (with a key a lane for all eight rows
  // 16 packed FMAs needed 20 cycles of reads, now 12).
  const int wrow = warp * RW, half = lane & 1, slot = lane >> 1;
  int p[HALF], lo[HALF], kept[HALF];      // what its rows see
#pragma unroll
  for (int i = 0; i < HALF; ++i) {
    const int r = wrow + HALF * half + i;
    p[i] = r < rows ? p0 + r / group : -1;
    lo[i] = r < rows ? mi::first_visible(p[i], a.window) : 0;
    kept[i] = r < rows && a.window > 0 ? min(a.keep_first, lo[i]) : 0;
  }
  // the segments of the block's rows: those with kept keys, then those from the first row's first key to the last row's last
  const int lo_min = mi::first_visible(p0, a.window);
  const int kept_max = a.window > 0 ? min(a.keep_first, mi::first_visible(p_max, a.window)) : 0;
  const int kept_segs = (kept_max + SEG - 1) / SEG, seg0 = lo_min / SEG;
  const int segs = kept_segs + p_max / SEG - seg0 + 1;

  const size_t page_elems = (size_t)2 * a.nkv * a.page_size * hd, v_off = (size_t)a.nkv * a.page_size * hd;
  const float* kv = a.kv + (size_t)kvh * a.page_size * hd;

  for (int round = 0; round < segs; round += a.cluster) {
    const int seg = round + rank;
    float m[HALF], l[HALF], o[RW][4 * NV];
#pragma unroll
    for (int i = 0; i < HALF; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < RW; ++i)
#pragma unroll
      for (int d = 0; d < 4 * NV; ++d) o[i][d] = 0.f;
    if (seg < segs) {
      const bool first_keys = seg < kept_segs;
      const int base = first_keys ? seg * SEG : (seg0 + seg - kept_segs) * SEG;
      const int key_end = first_keys ? min(base + SEG, kept_max) : min(base + SEG, p_max + 1);      // one past the last key wanted
      const int key_lo = first_keys ? 0 : lo_min;
      const int c_begin = max(base, key_lo / CHUNK * CHUNK);
      auto stage = [&](int c, int s) {
        if (c < key_end) {
          const int j = c + lane;
          long long off = -1;
          if (j >= key_lo && j < key_end) off = (long long)((size_t)bt[j / a.page_size] * page_elems + (size_t)(j % a.page_size) * hd);
          for (int jj = warp; jj < CHUNK; jj += WARPS) {
            const long long ko = __shfl_sync(0xffffffffu, off, jj);
#pragma unroll
            for (int n = 0; n < NV; ++n) {
              const int d = 128 * n + 4 * lane;
              if (d < hd) {
                const float* src = ko < 0 ? kv : kv + ko + d;
                const uint32_t kd = (uint32_t)__cvta_generic_to_shared(sm + at.keys(s) + jj * at.ldk + d);
                const uint32_t vd = (uint32_t)__cvta_generic_to_shared(sm + at.values(s) + jj * hd + d);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(kd), "l"(src), "r"(ko < 0 ? 0 : 16) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(vd), "l"(ko < 0 ? kv : src + v_off), "r"(ko < 0 ? 0 : 16) : "memory");
              }
            }
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      stage(c_begin, 0);
      int s = 0;
      for (int c = c_begin; c < key_end; c += CHUNK, s ^= 1) {
        stage(c + CHUNK, s ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        // a row's key is visible in this stretch; a warp none of whose rows sees any key of the chunk has nothing to do
        bool seen[HALF][2], any = false, every = true;
#pragma unroll
        for (int i = 0; i < HALF; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = c + slot + 16 * e;
            seen[i][e] = first_keys ? j < kept[i] : j >= lo[i] && j <= p[i];
            any |= seen[i][e];
            every &= seen[i][e] || p[i] < 0;      // (a row that does not exist)
          }
        if (__any_sync(0xffffffffu, any)) {
          uint64_t acc[HALF][2];
#pragma unroll
          for (int i = 0; i < HALF; ++i) acc[i][0] = acc[i][1] = 0;
          const float* kr = sm + at.keys(s) + slot * at.ldk;
          const float* qr = sm + at.queries() + (wrow + HALF * half) * at.ldk;
#pragma unroll 4
          for (int d = 0; d < hd; d += 4) {
            const ulonglong2 k0 = *reinterpret_cast<const ulonglong2*>(kr + d), k1 = *reinterpret_cast<const ulonglong2*>(kr + 16 * at.ldk + d);
#pragma unroll
            for (int i = 0; i < HALF; ++i) {
              const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(qr + i * at.ldk + d);
              acc[i][0] = fma2(q4.y, k0.y, fma2(q4.x, k0.x, acc[i][0]));
              acc[i][1] = fma2(q4.y, k1.y, fma2(q4.x, k1.x, acc[i][1]));
            }
          }
          float pe[2][HALF], alpha[HALF];
#pragma unroll
          for (int i = 0; i < HALF; ++i) {
            float sc[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float x, y;
              asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(acc[i][e]));
              sc[e] = seen[i][e] ? a.scale * (x + y) : -INFINITY;
            }
            float m_new = fmaxf(sc[0], sc[1]);
#pragma unroll
            for (int k = 16; k > 1; k >>= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, k));
            m_new = fmaxf(m[i], m_new);
            const bool none = m_new == -INFINITY;      // no key of this segment seen yet, or none whose score weighs anything
            alpha[i] = none ? 1.f : expf(m[i] - m_new);
#pragma unroll
            for (int e = 0; e < 2; ++e) pe[e][i] = seen[i][e] ? expf(sc[e] - (none ? 0.f : m_new)) : 0.f;
            float sum = pe[0][i] + pe[1][i];      // (as the halves of a warp with a key a lane add up)
#pragma unroll
            for (int k = 16; k > 1; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
            l[i] = l[i] * alpha[i] + sum;
            m[i] = m_new;
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if (!seen[i][e]) pe[e][i] = -1.f;      // (no weight is)
          }
          float* pw = sm + at.weights() + warp * (CHUNK + 1) * RW;
#pragma unroll
          for (int e = 0; e < 2; ++e) *reinterpret_cast<float4*>(pw + (slot + 16 * e) * RW + HALF * half) = make_float4(pe[e][0], pe[e][1], pe[e][2], pe[e][3]);
          if (slot == 0) *reinterpret_cast<float4*>(pw + CHUNK * RW + HALF * half) = make_float4(alpha[0], alpha[1], alpha[2], alpha[3]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < RW; ++i) {
            const float f = pw[CHUNK * RW + i];
#pragma unroll
            for (int d = 0; d < 4 * NV; ++d) o[i][d] *= f;
          }
          const float* vr = sm + at.values(s);
          // MASKED: a row takes nothing from a key that it may not see, not even zero times its value, which may be no number
          auto weigh = [&](auto masked) {
            constexpr bool MASKED = decltype(masked)::value;
#pragma unroll(MASKED ? 1 : 4)
            for (int jj = 0; jj < CHUNK; ++jj) {
              float w[RW];
#pragma unroll
              for (int i = 0; i < RW; i += 2) {
                const float2 t = *reinterpret_cast<const float2*>(pw + jj * RW + i);
                w[i] = t.x;
                w[i + 1] = t.y;
              }
#pragma unroll
              for (int n = 0; n < NV; ++n) {
                const int d = 128 * n + 4 * lane;
                if (d < hd) {
                  const float4 v = *reinterpret_cast<const float4*>(vr + jj * hd + d);
#pragma unroll
                  for (int i = 0; i < RW; ++i) {
                    if (MASKED && w[i] < 0.f) continue;
                    o[i][4 * n] = fmaf(w[i], v.x, o[i][4 * n]);
                    o[i][4 * n + 1] = fmaf(w[i], v.y, o[i][4 * n + 1]);
                    o[i][4 * n + 2] = fmaf(w[i], v.z, o[i][4 * n + 2]);
                    o[i][4 * n + 3] = fmaf(w[i], v.w, o[i][4 * n + 3]);
                  }
                }
              }
            }
          };
          if (__all_sync(0xffffffffu, every)) weigh(std::false_type());
          else weigh(std::true_type());
        }
        __syncthreads();      // the stage may be filled again
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
    // this segment's results into shared memory; the owner of a row merges those of the round in the segments' order
#pragma unroll
    for (int i = 0; i < RW; ++i) {
      const int r = wrow + i;
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const int d = 128 * n + 4 * lane;
        if (d < hd) *reinterpret_cast<float4*>(part_o + r * hd + d) = make_float4(o[i][4 * n], o[i][4 * n + 1], o[i][4 * n + 2], o[i][4 * n + 3]);
      }
    }
    if (slot == 0) {
#pragma unroll
      for (int i = 0; i < HALF; ++i) {
        part_m[wrow + HALF * half + i] = m[i];
        part_l[wrow + HALF * half + i] = l[i];
      }
    }
    cluster.sync();
    for (int r = rank + a.cluster * warp; r < rows; r += a.cluster * WARPS) {
      float mm = run_m[r], ll = run_l[r], oo[4 * NV];
#pragma unroll
      for (int n = 0; n < NV; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) oo[4 * n + e] = 128 * n + 4 * lane < hd ? run_o[r * hd + 128 * n + 4 * lane + e] : 0.f;
      for (int b = 0; b < a.cluster && round + b < segs; ++b) {
        const float pm = *cluster.map_shared_rank(part_m + r, b), pl = *cluster.map_shared_rank(part_l + r, b);
        if (pm == -INFINITY && pl == 0.f) continue;      // no key of that segment is visible (scores that are no numbers leave a sum that is none)
        const float m_new = fmaxf(mm, pm), fa = expf(mm - m_new), fb = expf(pm - m_new);
        ll = ll * fa + pl * fb;
        mm = m_new;
        const float* po = cluster.map_shared_rank(part_o + r * hd, b);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const int d = 128 * n + 4 * lane;
          if (d < hd) {
            const float4 v = *reinterpret_cast<const float4*>(po + d);
            oo[4 * n] = oo[4 * n] * fa + v.x * fb;
            oo[4 * n + 1] = oo[4 * n + 1] * fa + v.y * fb;
            oo[4 * n + 2] = oo[4 * n + 2] * fa + v.z * fb;
            oo[4 * n + 3] = oo[4 * n + 3] * fa + v.w * fb;
          }
        }
      }
      __syncwarp();
      if (round + a.cluster < segs) {
        if (lane == 0) {
          run_m[r] = mm;
          run_l[r] = ll;
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const int d = 128 * n + 4 * lane;
          if (d < hd) *reinterpret_cast<float4*>(run_o + r * hd + d) = make_float4(oo[4 * n], oo[4 * n + 1], oo[4 * n + 2], oo[4 * n + 3]);
        }
      } else {
        const int token = row0 + tok0 + r / group, head = kvh * group + r % group;
        const float inv = 1.f / ll;
        float* dst = a.out + ((size_t)token * a.nh + head) * a.out_hd;
        const float* gt = a.gate ? a.gate + (size_t)token * a.gate_stride : nullptr;
#pragma unroll
        for (int n = 0; n < NV; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int d = 128 * n + 4 * lane + e;
            if (d < a.out_hd) {
              float y = oo[4 * n + e] * inv;
              if (gt) y = y / (1.f + expf(-gt[mi::gate_index(head, d, a.out_hd, a.gate_per_head)]));
              dst[d] = y;
            }
          }
      }
    }
    cluster.sync();      // nobody overwrites what a neighbour still reads, and nobody leaves
  }
}

// One new token: the same arithmetic, a block's four warps sharing a segment instead of one walking it (a lone warp took 9000 cycles a chunk
// of 32 keys).  A row's scores of a chunk, its maximum and its sum are one warp's, a key a lane; a thread then weighs the values of an output
// column, all rows of it, key after key.  While a chunk is weighed the next one's scores are made and the one behind it is copied: a barrier a chunk.
// RW: rows of a block, the query heads of a key/value head.  16 / 8 heads of 128, microseconds by one warp and by four: two tokens behind 1000
// 37 -> 23, eight behind 2000 each 77 -> 62, three behind 300 36 -> 23.  The scores' chain of 64 packed FMAs and its reads take two thirds of that.
// (With bulk copies, two a key, in place of 16-byte ones: 45, 100, 43; with the scores' loop unrolled further the same.)
// The merge of a round repeats that above: as one function for both the compiler gives this kernel other registers, and two tokens behind 1000 take 30 us.
template <int RW, int NV>
struct OneLayout {
  int hd, ldk;
  __host__ __device__ explicit OneLayout(int hd) : hd(hd), ldk(hd + 4) {}
  __host__ __device__ int keys(int stage) const { return stage * CHUNK * ldk; }
  __host__ __device__ int values(int stage) const { return 3 * CHUNK * ldk + stage * CHUNK * hd; }
  __host__ __device__ int queries() const { return 3 * CHUNK * (ldk + hd); }
  __host__ __device__ int weights(int stage) const { return queries() + RW * hd + stage * (CHUNK + 1) * RW; }      // [key][row], then the rows' factors
  __host__ __device__ int running() const { return queries() + RW * hd + 2 * (CHUNK + 1) * RW; }
  __host__ __device__ int floats() const { return running() + RW * hd + 4 * RW; }
};

template <int RW, int NV>
__global__ void __launch_bounds__(128)
attention_f32_one_kernel(const F32Args a) {
  constexpr int WARPS = 4, PER_WARP = (RW + WARPS - 1) / WARPS;
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const OneLayout<RW, NV> at(a.hd);
  const int hd = a.hd, ldk = at.ldk, rows = a.nh / a.nkv;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int item = a.items[blockIdx.x / a.cluster], rank = blockIdx.x % a.cluster, kvh = blockIdx.y;
  const int token = a.q_start[item], p = a.ctx_len[item] - 1;
  const int* bt = a.block_table + (size_t)a.seq_slot[item] * a.bt_stride;
  const int lo = mi::first_visible(p, a.window), kept = a.window > 0 ? min(a.keep_first, lo) : 0;
  const int kept_segs = (kept + SEG - 1) / SEG, seg0 = lo / SEG, segs = kept_segs + p / SEG - seg0 + 1;
  const size_t page_elems = (size_t)2 * a.nkv * a.page_size * hd, v_off = (size_t)a.nkv * a.page_size * hd;
  const float* kv = a.kv + (size_t)kvh * a.page_size * hd;
  float* run_o = sm + at.running();
  float *run_m = run_o + RW * hd, *run_l = run_m + RW, *part_m = run_l + RW, *part_l = part_m + RW;
  float* part_o = sm;
  mi::grid_dependency_sync();
  for (int i = 4 * tid; i < RW * hd; i += 512) {
    const int r = i / hd;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) v = *reinterpret_cast<const float4*>(a.q + (size_t)token * a.q_stride + (size_t)(kvh * rows) * hd + i);
    *reinterpret_cast<float4*>(sm + at.queries() + i) = v;
    *reinterpret_cast<float4*>(run_o + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (tid < RW) {
    run_m[tid] = a.sink && tid < rows ? a.sink[kvh * rows + tid] : -INFINITY;
    run_l[tid] = a.sink ? 1.f : 0.f;
  }
  for (int round = 0; round < segs; round += a.cluster) {
    const int seg = round + rank;
    float m[PER_WARP], l[PER_WARP], o[RW][NV];
#pragma unroll
    for (int i = 0; i < PER_WARP; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < RW; ++i)
#pragma unroll
      for (int n = 0; n < NV; ++n) o[i][n] = 0.f;
    if (seg < segs) {
      const bool first_keys = seg < kept_segs;
      const int base = first_keys ? seg * SEG : (seg0 + seg - kept_segs) * SEG;
      const int key_end = first_keys ? min(base + SEG, kept) : min(base + SEG, p + 1), key_lo = first_keys ? 0 : lo;
      const int c_begin = max(base, key_lo / CHUNK * CHUNK);
      // four threads a key; keys that are not seen are zeros.  A key's page is looked up a chunk ahead.
      const int jj = tid >> 2;
      auto seen_key = [&](int j) { return j >= key_lo && j < key_end; };
      int page = seen_key(c_begin + jj) ? bt[(c_begin + jj) / a.page_size] : 0;
      auto stage = [&](int c, int s) {
        const int j = c + jj;
        if (c < key_end) {
          const bool in = seen_key(j);
          const float* src = in ? kv + (size_t)page * page_elems + (size_t)(j % a.page_size) * hd : kv;
          const uint32_t kd = (uint32_t)__cvta_generic_to_shared(sm + at.keys(s) + jj * ldk), vd = (uint32_t)__cvta_generic_to_shared(sm + at.values(s) + jj * hd);
#pragma unroll 4
          for (int d = (tid & 3) * 4; d < hd; d += 16) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(kd + 4 * d), "l"(in ? src + d : kv), "r"(in ? 16 : 0) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(vd + 4 * d), "l"(in ? src + v_off + d : kv), "r"(in ? 16 : 0) : "memory");
          }
          page = seen_key(j + CHUNK) ? bt[(j + CHUNK) / a.page_size] : 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      // this warp's rows of a chunk: weights and the factor of what was added up before
      auto score = [&](int c, int s, int b) {
        if (c >= key_end || warp >= rows) return;
        const bool seen = c + lane >= key_lo && c + lane < key_end;
        uint64_t acc[PER_WARP];
#pragma unroll
        for (int i = 0; i < PER_WARP; ++i) acc[i] = 0;
        const float *kr = sm + at.keys(s) + lane * ldk, *qr = sm + at.queries() + warp * hd;
#pragma unroll 4
        for (int d = 0; d < hd; d += 4) {
          const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(kr + d);
#pragma unroll
          for (int i = 0; i < PER_WARP; ++i) {
            const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(qr + i * WARPS * hd + d);
            acc[i] = fma2(q4.y, k4.y, fma2(q4.x, k4.x, acc[i]));
          }
        }
        float* w = sm + at.weights(b);
#pragma unroll
        for (int i = 0; i < PER_WARP; ++i) {
          const int r = warp + i * WARPS;
          if (r >= rows) break;
          float x, y;
          asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(acc[i]));
          const float sc = seen ? a.scale * (x + y) : -INFINITY, m_new = fmaxf(m[i], mi::warp_max(sc));
          const bool none = m_new == -INFINITY;      // no key of this segment seen yet, or none whose score weighs anything
          const float alpha = none ? 1.f : expf(m[i] - m_new), pe = seen ? expf(sc - (none ? 0.f : m_new)) : 0.f;
          l[i] = l[i] * alpha + mi::warp_sum(pe);
          m[i] = m_new;
          w[lane * RW + r] = pe;
          if (lane == 0) w[CHUNK * RW + r] = alpha;
        }
      };
      auto weigh = [&](int s, int b) {
        const float *w = sm + at.weights(b), *v = sm + at.values(s) + tid;
#pragma unroll
        for (int i = 0; i < RW; ++i)
#pragma unroll
          for (int n = 0; n < NV; ++n) o[i][n] *= w[CHUNK * RW + i];
#pragma unroll 8
        for (int jj = 0; jj < CHUNK; ++jj) {
          float x[RW];
#pragma unroll
          for (int i = 0; i < RW; i += 2) {
            const float2 t = *reinterpret_cast<const float2*>(w + jj * RW + i);
            x[i] = t.x;
            x[i + 1] = t.y;
          }
#pragma unroll
          for (int n = 0; n < NV; ++n) {
            const float y = tid + 128 * n < hd ? v[jj * hd + 128 * n] : 0.f;
#pragma unroll
            for (int i = 0; i < RW; ++i) o[i][n] = fmaf(x[i], y, o[i][n]);
          }
        }
      };
      stage(c_begin, 0);
      stage(c_begin + CHUNK, 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      score(c_begin, 0, 0);
      int s = 0, b = 0;      // the chunk's stage and buffer of weights
#pragma unroll 1
      for (int c = c_begin; c < key_end; c += CHUNK, b ^= 1) {
        const int s1 = s == 2 ? 0 : s + 1, s2 = s1 == 2 ? 0 : s1 + 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();      // the next chunk has landed, this one's weights are there, and the one before is done with
        stage(c + 2 * CHUNK, s2);
        score(c + CHUNK, s1, b ^ 1);
        weigh(s, b);
        s = s1;
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
    // this segment's results into shared memory; the owner of a row merges those of the round in the segments' order
#pragma unroll
    for (int i = 0; i < RW; ++i)
#pragma unroll
      for (int n = 0; n < NV; ++n)
        if (tid + 128 * n < hd) part_o[i * hd + tid + 128 * n] = o[i][n];
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < PER_WARP; ++i)
        if (warp + i * WARPS < RW) {
          part_m[warp + i * WARPS] = m[i];
          part_l[warp + i * WARPS] = l[i];
        }
    }
    cluster.sync();
    for (int r = rank + a.cluster * warp; r < rows; r += a.cluster * WARPS) {
      float mm = run_m[r], ll = run_l[r], oo[4 * NV];
#pragma unroll
      for (int n = 0; n < NV; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) oo[4 * n + e] = 128 * n + 4 * lane < hd ? run_o[r * hd + 128 * n + 4 * lane + e] : 0.f;
#pragma unroll 1
      for (int b = 0; b < a.cluster && round + b < segs; ++b) {
        const float pm = *cluster.map_shared_rank(part_m + r, b), pl = *cluster.map_shared_rank(part_l + r, b);
        if (pm == -INFINITY && pl == 0.f) continue;      // no key of that segment is visible (scores that are no numbers leave a sum that is none)
        const float m_new = fmaxf(mm, pm), fa = expf(mm - m_new), fb = expf(pm - m_new);
        ll = ll * fa + pl * fb;
        mm = m_new;
        const float* po = cluster.map_shared_rank(part_o + r * hd, b);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const int d = 128 * n + 4 * lane;
          if (d < hd) {
            const float4 v = *reinterpret_cast<const float4*>(po + d);
            oo[4 * n] = oo[4 * n] * fa + v.x * fb;
            oo[4 * n + 1] = oo[4 * n + 1] * fa + v.y * fb;
            oo[4 * n + 2] = oo[4 * n + 2] * fa + v.z * fb;
            oo[4 * n + 3] = oo[4 * n + 3] * fa + v.w * fb;
          }
        }
      }
      __syncwarp();
      if (round + a.cluster < segs) {
        if (lane == 0) {
          run_m[r] = mm;
          run_l[r] = ll;
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const int d = 128 * n + 4 * lane;
          if (d < hd) *reinterpret_cast<float4*>(run_o + r * hd + d) = make_float4(oo[4 * n], oo[4 * n + 1], oo[4 * n + 2], oo[4 * n + 3]);
        }
      } else {
        const int head = kvh * rows + r;
        const float inv = 1.f / ll;
        float* dst = a.out + ((size_t)token * a.nh + head) * a.out_hd;
        const float* gt = a.gate ? a.gate + (size_t)token * a.gate_stride : nullptr;
#pragma unroll
        for (int n = 0; n < NV; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int d = 128 * n + 4 * lane + e;
            if (d < a.out_hd) {
              float y = oo[4 * n + e] * inv;
              if (gt) y = y / (1.f + expf(-gt[mi::gate_index(head, d, a.out_hd, a.gate_per_head)]));
              dst[d] = y;
            }
          }
      }
    }
    cluster.sync();      // nobody overwrites what a neighbour still reads, and nobody leaves
  }
}

// ONE: one new token's rows, RW of them, by four warps together.
template <int WARPS, int RW, int NV, bool ONE>
int launch_form(F32Args a, int units, cudaStream_t stream) {
  const size_t smem = sizeof(float) * (ONE ? OneLayout<RW, NV>(a.hd).floats() : Layout<WARPS, RW, NV>(a.hd).floats());
  void (*kernel)(const F32Args);
  if constexpr (ONE) kernel = attention_f32_one_kernel<RW, NV>;
  else kernel = attention_f32_kernel<WARPS, RW, NV>;
  static int ready[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || ready[dev] < (int)smem) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return mi_fail("attention_f32: %zu bytes of shared memory were refused", smem);
    if (dev >= 0 && dev < 64) ready[dev] = (int)smem;
  }
  // as many blocks a cluster as keep the grid within about four blocks a SM: more only shares a row's segments out further
  a.cluster = 1;
  while (a.cluster < 8 && 2ll * a.cluster * units * a.nkv <= 4ll * mi::sm_count()) a.cluster *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)units * a.cluster, a.nkv);
  cfg.blockDim = dim3(32 * WARPS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = a.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = mi::pdl_enabled() ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, a) != cudaSuccess) return mi_fail("attention_f32: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
  return 0;
}

template <int RW, bool ONE>
int launch_rows(const F32Args& a, int units, cudaStream_t stream) {
  return a.hd <= 128 ? launch_form<4, RW, 1, ONE>(a, units, stream) : launch_form<4, RW, 2, ONE>(a, units, stream);
}

}  // namespace

// tiles: [num_tiles, 2] (item, first row) for every tile_rows new tokens of the items that bring several; decode_items: the
// items that bring one.  q: the first nh * hd values of rows q_stride apart.
MI_API int mi_attention_f32(float* out, const float* q, int q_stride, const float* kv_layer, const int* block_table, int bt_stride,
                            const int* tiles, int num_tiles, int tile_rows, const int* decode_items, int num_decode,
                            const int* q_start, const int* q_len, const int* ctx_len, const int* seq_slot, int nh, int nkv, int hd,
                            int page_size, float scale, int window, const float* sink, const float* gate, int gate_stride, int out_hd,
                            int keep_first, int gate_per_head, cudaStream_t stream) {
  MI_REQUIRE(nh > 0 && nkv > 0 && nh % nkv == 0 && nh / nkv <= 32 && nkv <= 65535, "attention_f32: bad head counts nh=%d nkv=%d", nh, nkv);
  MI_REQUIRE(hd > 0 && hd % 4 == 0 && hd <= 256 && out_hd > 0 && out_hd <= hd, "attention_f32: bad head sizes %d, %d", hd, out_hd);
  MI_REQUIRE(page_size > 0 && q_stride % 4 == 0 && keep_first >= 0 && tile_rows > 0, "attention_f32: bad page_size=%d or q_stride=%d", page_size, q_stride);
  MI_REQUIRE(((uintptr_t)q % 16) == 0 && ((uintptr_t)kv_layer % 16) == 0, "attention_f32: rows must start on 16-byte boundaries");
  const int group = nh / nkv;
  F32Args a{out, q, q_stride, kv_layer, block_table, bt_stride, nullptr, q_start, q_len, ctx_len, seq_slot, 0, tile_rows, 1, nh, nkv, hd,
            page_size, scale, window, keep_first, sink, gate, gate_stride, out_hd, gate_per_head, 1};
  if (num_tiles > 0) {
    F32Args p = a;
    p.items = tiles;
    p.tokens = 32 / group;
    p.subtiles = (tile_rows + p.tokens - 1) / p.tokens;
    if (launch_rows<8, false>(p, num_tiles * p.subtiles, stream)) return 1;
  }
  if (num_decode > 0) {
    a.items = decode_items;
    if (group <= 2 ? launch_rows<2, true>(a, num_decode, stream) : group <= 8 ? launch_rows<8, true>(a, num_decode, stream) : launch_rows<8, false>(a, num_decode, stream))
      return 1;
  }
  return 0;
}
