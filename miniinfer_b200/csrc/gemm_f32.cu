// True float32 matrix product on the CUDA cores: out[M, N] = x[M, K] * w[N, K]^T.
//
// This is the matrix product of the engine's 32-bit path.  Every product and sum is an fp32 FMA (no TF32, no tensor cores).
// The order in which an output element adds its K products is a function of K alone: K is cut into sixteen parts of equal
// length (a multiple of the 32 columns that are staged at a time); within a part the products of even k and those of odd k
// are added in ascending k, each to a sum of its own - the two halves of a packed fma.rn.f32x2 -, and the two sums are added
// up; four parts after one another make a group, and the four groups the result.  So the value of an element does not
// depend on M, on the tile it falls in, on how many warps and blocks share it or on what else is in the batch: the 32-bit
// path gives bit-equal logits however the tokens are cut into steps.  The reference has no 32-bit path (it calls cuBLAS in
// fp16, miniinfer/layers/linear.py:30-32).
//
// What bounds it: the packed FMAs' own rate and the clusters' ends for many rows, latency for few.  A thread computes 8 x 4 elements (fewer for small
// M): rows are staged as they lie in memory, K fastest, so that cp.async brings them without a transposition and a 16-byte
// read of shared memory gives two packed operands; rows of 36 floats keep the eight rows that a warp reads at a time in
// different banks.  Two forms, both in three stages of 32 columns:
//   * more than 32 rows: four warps share a tile of 64 x 64 and walk the parts of a group, or of all four, one after the other;
//   * up to 32 rows: every warp has a tile of its rows x 32 and parts of its own, staged by itself, so that the weights come
//     in at many places at once; the warps' sums are added up in shared memory.
// The groups go to the four blocks of a cluster, whose sums are added up in each other's shared memory, in the order that
// one block would - for few rows only where the tiles alone leave SMs idle, for many from some hundred columns on.
// Measured on B200, weights in L2, in microseconds, against one form of 64 x 64 tiles, 4 x 4 elements a thread, staged one
// step at a time: 8 x 4096 x 1024 74 -> 9.1, 16 x 1024 x 2048 146 -> 8.9, 40 x 6144 x 1024 75 -> 27, 302 x 4096 x 1024 174 -> 78,
// 302 x 1024 x 2048 149 -> 48, 2048 x 4096 x 1024 583 -> 433 (40 of the 70 TFLOP/s that a loop of FMAs alone reaches),
// 8 x 151936 x 1024 727 -> 112 (5.6 TB/s).  (With lanes that share neither rows in pairs and copies that check and place each row
// by itself: 9.8, 9.0, 29, 88, 53, 491, 124.)  Sixteen partial sums also err less: 1.2e-7 against 5.7e-7 of the norm at K = 1024.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int BK = 32, LDS = BK + 4, STAGES = 3, GROUPS = 4, PARTS = 4;      // PARTS: of a group

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

template <bool VEC>
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool valid) {
  if (VEC)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float halves(uint64_t v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo + hi;
}

// Rows row0 .. of a matrix with `rows` rows, ld values apart, columns k0 .. k0 + 31, into ROWS staged rows, by THREADS threads of which this one
// is number `thread`.  A copy costs a minimum, a multiplication and itself: rows beyond the matrix are its last one again or what lay there, and nobody
// stores their sums (with a check of each row and an address of its own the copies took a tenth of the kernel's time).  Columns from K on are zeros.
template <int ROWS, int THREADS, bool VEC>
__device__ __forceinline__ void stage_rows(float* dst, const float* src, int row0, int rows, int ld, int k0, int K, int thread) {
  constexpr int W = VEC ? 4 : 1, PER_ROW = BK / W, AT_ONCE = THREADS / PER_ROW;
  static_assert(THREADS % PER_ROW == 0 && ROWS % AT_ONCE == 0, "");
  const int r = row0 + thread / PER_ROW, c = thread % PER_ROW * W;
  const bool valid = k0 + c < K;
  const char* column = reinterpret_cast<const char*>(src + (valid ? k0 + c : 0));
  dst += thread / PER_ROW * LDS + c;
#pragma unroll VEC ? 8 : 4
  for (int i = 0; i < ROWS; i += AT_ONCE)
    if (!VEC || row0 + i < rows) copy_async<VEC>(dst + i * LDS, reinterpret_cast<const float*>(column + (long long)min(r + i, rows - 1) * (4u * ld)), valid);
}

// TM: rows of a thread (a warp has 4 TM rows x 32 columns).  SHARED: four warps, 2 x 2, share a tile; else a warp has the
// block's whole tile and parts of its own.
template <int TM, bool SHARED>
struct Tile {
  static constexpr int TN = 4, BM = 4 * TM * (SHARED ? 2 : 1), BN = 8 * TN * (SHARED ? 2 : 1), STAGE = (BM + BN) * LDS;
  static constexpr int LDP = BN + 4, SUMS = BM * LDP;                                  // the sums of one warp or block
  static constexpr int STAGED = STAGES * STAGE * (SHARED ? 1 : 4), SUMMED = SUMS * (SHARED ? 1 : 4);
  static constexpr size_t SMEM = sizeof(float) * (STAGED > SUMMED ? STAGED : SUMMED);  // (the sums lie where the stages were)
};

// CLUSTER: the block's group is its rank in a cluster of GROUPS blocks.
template <int TM, bool SHARED, bool CLUSTER, bool VEC>
__device__ __forceinline__ void product(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w,
                                        int M, int N, int K, int ldx, int ldo, int m_tile, int n_tile, int rank) {
  using T = Tile<TM, SHARED>;
  constexpr int TN = T::TN, BM = T::BM, BN = T::BN, MOVERS = SHARED ? 128 : 32;
  extern __shared__ __align__(16) float sm[];
  const int m0 = m_tile * BM, n0 = n_tile * BN;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, thread = SHARED ? threadIdx.x : lane;
  // A 16-byte read of a warp takes two cycles of shared memory instead of four if the lanes i and i ^ 1, or i and i ^ 2, of all read the same
  // place: the rows of x are shared by the former and those of w by the latter
  const int row = (SHARED ? (warp & 1) * 4 * TM : 0) + (lane >> 1 & 1) + (lane >> 4) * 2, col = (SHARED ? (warp >> 1) * 8 * TN : 0) + (lane & 1) + (lane >> 2 & 3) * 2;
  float* stages = sm + (SHARED ? 0 : warp * STAGES * T::STAGE);
  const int len = ((K + GROUPS * PARTS - 1) / (GROUPS * PARTS) + BK - 1) / BK * BK;       // columns of a part
  const int per_part = len / BK;
  // parts that this warp walks: its block's group, or one part of that, or a group, or all
  constexpr bool ALL = SHARED && !CLUSTER;
  const int parts = ALL ? GROUPS * PARTS : SHARED || !CLUSTER ? PARTS : 1;
  const int first = ALL ? 0 : SHARED ? rank * PARTS : (CLUSTER ? rank * PARTS + warp : warp * PARTS);
  // a part without columns is +0 and left out (in another, columns beyond K are staged as zeros)
  const int begin = first * len, steps = per_part * min(parts, max(0, (K - begin + len - 1) / len));

  auto stage_w = [&](int s) {
    if (s < steps) stage_rows<BN, MOVERS, VEC>(stages + (s % STAGES) * T::STAGE + BM * LDS, w, n0, N, K, begin + s * BK, K, thread);
  };
  auto stage_x = [&](int s) {
    if (s < steps) stage_rows<BM, MOVERS, VEC>(stages + (s % STAGES) * T::STAGE, x, m0, M, ldx, begin + s * BK, K, thread);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) stage_w(s);      // the weights are written by no kernel: fetched before the wait
  mi::grid_dependency_sync();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) stage_x(s);

  uint64_t acc[TM][TN];
  float group[TM][TN], total[ALL ? TM : 1][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      acc[i][j] = 0;
      group[i][j] = 0.f;
      if (ALL) total[ALL ? i : 0][j] = 0.f;
    }

  int in_part = 0, part = 0;
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    if (SHARED) __syncthreads(); else __syncwarp();     // stage s has landed, and everybody is done with the one refilled now
    stage_w(s + STAGES - 1);
    stage_x(s + STAGES - 1);
    const float* xs = stages + (s % STAGES) * T::STAGE + row * LDS;
    const float* ws = stages + (s % STAGES) * T::STAGE + (BM + col) * LDS;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 b[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(ws + 8 * j * LDS + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xs + 4 * i * LDS + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma2(a.y, b[j].y, fma2(a.x, b[j].x, acc[i][j]));
      }
    }
    if (++in_part == per_part) {
      in_part = 0;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const float sum = halves(acc[i][j]);
          acc[i][j] = 0;
          group[i][j] = (ALL ? part % PARTS : part) == 0 ? sum : group[i][j] + sum;
          if (ALL && (part % PARTS == PARTS - 1 || s + 1 == steps)) total[ALL ? i : 0][j] = part < PARTS ? group[i][j] : total[ALL ? i : 0][j] + group[i][j];
        }
      ++part;
    }
  }

  // the warps' sums (SHARED: the block's) side by side in shared memory
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* mine = sm + (SHARED ? 0 : warp * T::SUMS);
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) mine[(row + 4 * i) * T::LDP + col + 8 * j] = ALL ? total[ALL ? i : 0][j] + 0.f : group[i][j];      // (+ 0: as groups without columns do)
  if (ALL) {
    __syncthreads();
    for (int i = threadIdx.x; i < BM * BN; i += 128) {
      const int r = i / BN, c = i % BN;
      if (m0 + r < M && n0 + c < N) out[(size_t)(m0 + r) * ldo + n0 + c] = sm[r * T::LDP + c];
    }
    return;
  }
  if (!CLUSTER) {      // a group a warp
    __syncthreads();
    for (int i = threadIdx.x; i < BM * BN; i += 128) {
      const int r = i / BN, c = i % BN;
      if (m0 + r >= M || n0 + c >= N) continue;
      float v = sm[r * T::LDP + c];
#pragma unroll
      for (int g = 1; g < GROUPS; ++g) v += sm[g * T::SUMS + r * T::LDP + c];
      out[(size_t)(m0 + r) * ldo + n0 + c] = v;
    }
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const float* sums[GROUPS];
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) sums[g] = cluster.map_shared_rank(sm, g);
  for (int i = threadIdx.x; i < BM / GROUPS * BN; i += 128) {      // this block's share of the rows
    const int r = rank * (BM / GROUPS) + i / BN, c = i % BN;
    if (m0 + r >= M || n0 + c >= N) continue;
    float v = 0.f;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      float one = sums[g][r * T::LDP + c];
      if (!SHARED) {      // a part a warp
#pragma unroll
        for (int p = 1; p < PARTS; ++p) one += sums[g][p * T::SUMS + r * T::LDP + c];
      }
      v = g == 0 ? one : v + one;
    }
    out[(size_t)(m0 + r) * ldo + n0 + c] = v;
  }
  cluster.sync();      // nobody leaves while its sums are read
}

template <int TM, bool SHARED, bool VEC>
__global__ void __launch_bounds__(128)
gemm_f32_kernel(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w, int M, int N, int K, int ldx, int ldo) {
  product<TM, SHARED, false, VEC>(out, x, w, M, N, K, ldx, ldo, blockIdx.y, blockIdx.x, 0);
}

template <int TM, bool SHARED, bool VEC>
__global__ void __cluster_dims__(GROUPS, 1, 1) __launch_bounds__(128, SHARED ? 3 : 1)      // (three, 168 registers a thread, of the four that shared memory holds; with two 302 x 4096 x 1024 takes 89 us)
gemm_f32_groups_kernel(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w, int M, int N, int K, int ldx, int ldo) {
  product<TM, SHARED, true, VEC>(out, x, w, M, N, K, ldx, ldo, blockIdx.y, blockIdx.x / GROUPS, blockIdx.x % GROUPS);
}

template <int TM, bool SHARED, bool VEC>
int launch_tiles(float* out, const float* x, const float* w, int M, int N, int K, int ldx, int ldo, cudaStream_t stream) {
  using T = Tile<TM, SHARED>;
  const int m_tiles = (M + T::BM - 1) / T::BM, n_tiles = (N + T::BN - 1) / T::BN;
  MI_REQUIRE(m_tiles <= 65535, "gemm_f32: M=%d is too large for one launch", M);
  auto whole = gemm_f32_kernel<TM, SHARED, VEC>;
  auto groups = gemm_f32_groups_kernel<TM, SHARED, VEC>;
  static bool ready[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !ready[dev]) {
    if (cudaFuncSetAttribute(whole, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(groups, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM) != cudaSuccess)
      return mi_fail("gemm_f32: %zu bytes of shared memory were refused", T::SMEM);
    if (dev >= 0 && dev < 64) ready[dev] = true;
  }
  // Few columns: a block walks all parts of a shared tile itself, for a cluster's blocks would wait longer for one another than
  // they work (`alone`, below).  In microseconds, walked / in clusters: 40 x 1024 x 128 8.8 / 9.1, x 192 10.0 / 9.0; 300 x 1024
  // x 64 8.7 / 10.2, x 256 12.8 / 15.7, x 384 18.0 / 16.0; 40 x 4096 x 256 13.0 / 15.6; 300 x 4096 x 384 41 / 45, x 512 54 / 45; 2048 x
  // 1024 x 384 54 / 66, x 512 70 / 66; 2048 x 4096 x 64 38 / 134, x 384 178 / 243.
  // Few rows: from a tile for every SM on, a block walks a tile's groups itself (24 x 6144 x 1024, 192 tiles: 17.8 us against
  // 20.2 with clusters; 8 x 151936 x 1024: 112 against 191).  Shared tiles of many columns are better off in clusters, whose smaller
  // blocks fill the SMs more evenly (302 x 4096 x 1024: 78 against 96); 2048 x 4096 x 1024 would take 421 instead of 433, but only while
  // the last round of blocks is nearly full.
  const long long tiles = (long long)m_tiles * n_tiles;
  const bool alone = K <= 128 || (K <= 256 && tiles >= 64) || (K <= 384 && tiles >= 320);
  if (SHARED ? alone : n_tiles >= mi::sm_count())
    mi::launch(whole, dim3(n_tiles, m_tiles), dim3(128), T::SMEM, stream, out, x, w, M, N, K, ldx, ldo);
  else
    mi::launch(groups, dim3(GROUPS * n_tiles, m_tiles), dim3(128), T::SMEM, stream, out, x, w, M, N, K, ldx, ldo);
  MI_LAUNCH_OK("gemm_f32");
  return 0;
}

template <bool VEC>
int launch_rows(float* out, const float* x, const float* w, int M, int N, int K, int ldx, int ldo, cudaStream_t stream) {
  // Few rows of few columns against many weights go by shared tiles too: 8 x 4096 x 64 4.6 us so and 5.8 by tiles of few rows, 24 x 4096
  // x 128 8.0 and 10.5 (8 x 4096 x 128 8.0 and 6.0; 8 x 1024 x 64 4.4 and 2.9, 24 x 1024 x 64 4.4 and 4.3)
  if (N >= 4096 && K <= (M > 16 ? 128 : 64)) return launch_tiles<8, true, VEC>(out, x, w, M, N, K, ldx, ldo, stream);
  if (M <= 8) return launch_tiles<2, false, VEC>(out, x, w, M, N, K, ldx, ldo, stream);
  if (M <= 16) return launch_tiles<4, false, VEC>(out, x, w, M, N, K, ldx, ldo, stream);
  if (M <= 32) return launch_tiles<8, false, VEC>(out, x, w, M, N, K, ldx, ldo, stream);
  return launch_tiles<8, true, VEC>(out, x, w, M, N, K, ldx, ldo, stream);
}

}  // namespace

// x: rows ldx values apart.
MI_API int mi_gemm_f32(float* out, const float* x, const float* w, int M, int N, int K, int ldx, int ldo,
                       cudaStream_t stream) {
  MI_REQUIRE(M >= 0 && N > 0 && K > 0 && ldx >= K && ldo >= N, "gemm_f32: bad sizes M=%d N=%d K=%d ldx=%d ldo=%d", M, N, K, ldx, ldo);
  if (M == 0) return 0;
  // rows that start on 16-byte boundaries are staged 16 bytes at a time, others value by value
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0;
  return vec ? launch_rows<true>(out, x, w, M, N, K, ldx, ldo, stream) : launch_rows<false>(out, x, w, M, N, K, ldx, ldo, stream);
}
