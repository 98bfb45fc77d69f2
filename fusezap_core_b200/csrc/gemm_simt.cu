// C[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) with plain 32-bit FMAs: the matrix product of the float32 path, and the
// general fallback of the bfloat16 path for sizes the tensor-core kernel refuses.
//
// Every output element is summed in one order that (N, K) alone fix, whatever M, the kernel, the tile or the thread it
// lands in: K is cut into at most 32 chunks of equal length, a chunk is one chain of fmaf in rising k from zero, a group
// of neighbouring chunks is added up in order, and the groups are added up in order. So a row's result has the same bits
// in every batch and every cutting of the work, and no reduced-precision mode is involved (the reference's CUDA "float32"
// product is a 3xTF32 tensor-core kernel, fusezap/device/cuda_kernels/tf32.py:1-12; its plain 32-bit product lives on its
// CPU device only). The cuts are what lets a few rows use the whole chip: with one chain over all of K (the order before)
// 4 x 4,864 -> 896 had 14 blocks to run in and took 215 us.
//
// Few rows (M <= 16): `gemm_simt_few_kernel`, bound by reading W. More rows: `gemm_simt_tile_kernel` and, where tiles are
// many, `gemm_simt_wide_kernel`, bound by the FMA pipes (a probe of independent fmaf chains reached 70 TFLOP/s, of packed
// pairs 71).
#include "common.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

namespace {
// The order of an output's sum. `chunk` k (a multiple of 32) per chunk, `chunks` <= 32 of them, `per_group` chunks to a
// group, `groups` <= 8 groups. A group is what one block of the tile kernel sums: at least 128 k, and the more groups the
// fewer columns there are, so that a few hundred rows of a narrow product still give every SM work.
struct Order { int chunk, chunks, per_group, groups; };
Order order_of(int N, int K) {
  Order o;
  o.chunk = 32 * ((K + 1023) / 1024);
  o.chunks = (K + o.chunk - 1) / o.chunk;
  int g = K / 128 < 8 ? K / 128 : 8;
  if (g > 16384 / N) g = 16384 / N;
  if (g < 1) g = 1;
  o.per_group = (o.chunks + g - 1) / g;
  o.groups = (o.chunks + o.per_group - 1) / o.per_group;
  return o;
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Four neighbouring k of one row into shared memory as float32; `k_end` is where the row's k stop, `row_ok` whether there
// is such a row. VEC: rows start on 16-byte boundaries and K is a multiple of 4 (asynchronous copy); else one by one.
template <typename T, bool VEC>
__device__ __forceinline__ void stage4(float* dst, const T* base, long long row, int K, int k, int k_end, bool row_ok) {
  if constexpr (VEC) {
    const bool ok = row_ok && k < k_end;
    fz_copy16(dst, ok ? base + row * K + k : base, ok);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = row_ok && k + i < k_end ? Cvt<T>::to_f(base[row * K + k + i]) : 0.f;
  }
}

__device__ __forceinline__ void fma4(float& acc, float4 a, float4 w) {
  acc = fmaf(a.x, w.x, acc);
  acc = fmaf(a.y, w.y, acc);
  acc = fmaf(a.z, w.z, acc);
  acc = fmaf(a.w, w.w, acc);
}

// ---- few rows
// A block owns 8 * RPL columns (rows of W) and all of K: warp w has chunks 4w .. 4w+3, eight lanes to a chunk, RPL
// columns to a lane, MR rows of A to each. So N * 32 / RPL chains run at once, and a warp waits for no other until the
// end: it streams its own 16 k of every (column, chunk) per stage through a ring of its own, 64 contiguous bytes each,
// whose 16-byte pieces stand in an order that changes every two rows (conflict-free reads without padding, so that three
// blocks share an SM at K = 896). Where the columns give every SM at most one block (DEEP) the ring takes all of its
// memory. The first stages of W, which no kernel of a step writes, are asked for ahead of the wait on the kernel before.
// Blocks that stay and walk several tiles with the ring running on measured slower at large N (896 -> 151,936 at 8 rows:
// 211 against 156 us): waiting at each tile's end for the slowest warp costs more than a new block. Measured at 4 rows,
// weights from HBM: 4,864 -> 896 7.1 us (rings two blocks could share: 10.1; one chain of fmaf over all of K: 215), 896
// -> 9,728 9.8 us (padded rows, two blocks per SM: 11.0; 75), 896 -> 151,936 113 us (132; 417), 4.8 TB/s; 4,096 -> 28,672
// 75 us, 6.3 TB/s.
constexpr int FEW_K = 16;
template <int MR, int RPL, bool DEEP> struct Few {
  static constexpr int W_FLOATS = 32 * RPL * FEW_K, A_SUB = MR * FEW_K + 4, STAGE = W_FLOATS + 4 * A_SUB;   // per warp
  static constexpr int FIT = (DEEP ? 220 : 112) * 1024 / (8 * STAGE * 4), MOST = DEEP ? 8 : 4;
  static constexpr int STAGES = FIT < 2 ? 2 : FIT > MOST ? MOST : FIT;      // two blocks per SM where that leaves two stages
};
// Where piece q (four k) of a stage's row lies within the row.
__device__ __forceinline__ int few_piece(int row, int q) { return (q ^ ((row >> 1) & 3)) * 4; }

template <typename TA, typename TC, int MR, int RPL, bool VEC, bool DEEP>
__global__ void __launch_bounds__(256)
gemm_simt_few_kernel(const TA* __restrict__ A, const TA* __restrict__ W, const float* __restrict__ bias,
                     TC* __restrict__ C, int M, int N, int K, Order o, int slots) {
  using F = Few<MR, RPL, DEEP>;
  constexpr int COLS = 8 * RPL;
  extern __shared__ float4 few_smem[];
  fz_grid_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane & 7, sub = lane >> 3;
  float* ring = reinterpret_cast<float*>(few_smem) + (size_t)warp * slots * F::STAGE;      // `slots`: STAGES, or the stages there are if fewer
  const int n0 = blockIdx.x * COLS;
  const int stages = o.chunk / FEW_K;

  auto load_w = [&](int s) {
    float* at = ring + (s % F::STAGES) * F::STAGE;
#pragma unroll
    for (int j = 0; j < 4 * RPL; ++j) {
      const int e = lane + 32 * j, stream = e >> 2, q = (e & 3) * 4;
      const int c = warp * 4 + stream / COLS, n = n0 + stream % COLS;
      const int k = c * o.chunk + s * FEW_K + q, end = min(K, (c + 1) * o.chunk);
      stage4<TA, VEC>(at + stream * FEW_K + few_piece(stream, e & 3), W, n, K, k, end, n < N && c < o.chunks);
    }
  };
  auto load_a = [&](int s) {
    float* at = ring + (s % F::STAGES) * F::STAGE + F::W_FLOATS;
#pragma unroll
    for (int j = 0; j < (16 * MR + 31) / 32; ++j) {
      const int e = lane + 32 * j;
      if (16 * MR % 32 == 0 || e < 16 * MR) {
        const int p = e / (4 * MR), m = e / 4 % MR, q = (e & 3) * 4, c = warp * 4 + p;
        const int k = c * o.chunk + s * FEW_K + q, end = min(K, (c + 1) * o.chunk);
        stage4<TA, VEC>(at + p * F::A_SUB + m * FEW_K + q, A, m, K, k, end, m < M && c < o.chunks);
      }
    }
  };

  float acc[RPL][MR];
#pragma unroll
  for (int i = 0; i < RPL; ++i)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[i][m] = 0.f;

#pragma unroll
  for (int s = 0; s < F::STAGES; ++s)
    if (s < stages) load_w(s);
  fz_grid_wait();
#pragma unroll
  for (int s = 0; s < F::STAGES; ++s) {
    if (s < stages) load_a(s);
    cp_commit();
  }
  for (int s = 0; s < stages; ++s) {
    cp_wait<F::STAGES - 1>();
    __syncwarp();
    const float* at = ring + (s % F::STAGES) * F::STAGE;
    const float* aw = at + F::W_FLOATS + sub * F::A_SUB;
#pragma unroll
    for (int q = 0; q < FEW_K / 4; ++q) {
      float4 w[RPL];
#pragma unroll
      for (int i = 0; i < RPL; ++i) w[i] = *reinterpret_cast<const float4*>(at + (sub * COLS + r + 8 * i) * FEW_K + few_piece(r, q));
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const float4 a = *reinterpret_cast<const float4*>(aw + m * FEW_K + 4 * q);
#pragma unroll
        for (int i = 0; i < RPL; ++i) fma4(acc[i][m], a, w[i]);
      }
    }
    __syncwarp();
    if (s + F::STAGES < stages) {
      load_w(s + F::STAGES);
      load_a(s + F::STAGES);
    }
    cp_commit();
  }
  cp_wait<0>();
  __syncthreads();      // the rings are done with: their memory takes the chunks' sums, [chunk][row of A][column]
  float* sums = reinterpret_cast<float*>(few_smem);
  const int c = warp * 4 + sub;
  if (c < o.chunks) {
#pragma unroll
    for (int m = 0; m < MR; ++m)
#pragma unroll
      for (int i = 0; i < RPL; ++i) sums[(c * MR + m) * COLS + r + 8 * i] = acc[i][m];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < COLS * M; e += blockDim.x) {
    const int n = n0 + e % COLS;
    if (n >= N) continue;
    float v = 0.f;
    for (int g = 0, ch = 0; g < o.groups; ++g) {
      float part = 0.f;
      for (const int end = min(o.chunks, ch + o.per_group); ch < end; ++ch) part += sums[ch * MR * COLS + e];
      v += part;
    }
    if (bias) v += bias[n];
    C[(size_t)(e / COLS) * N + n] = Cvt<TC>::from_f(v);
  }
}

// ---- more rows
// Tiles of (8 TM) x (16 TN) outputs, 128 threads with TM x TN outputs each, 32 k per stage, three stages of asynchronous
// copies; rows lie in shared memory as in memory, padded to 144 bytes, and are read 16 bytes (four k) at a time. With 8 x
// 4 outputs per thread 16 warps share an SM; 8 x 6 and 8 x 8 reach the same 40 TFLOP/s on large products and lose on
// small ones (300 rows, 896 -> 9,728: 160, 174 and 208 us). A block sums one group of chunks (`acc` the chunk's chain,
// `tot` the group) and the blocks of a tile's groups, a cluster, add their tiles up in order through distributed shared
// memory. Measured at 300 rows: 896 -> 9,728 265 -> 160 us, 4,864 -> 896 215 -> 78 us, 896 -> 151,936 3,364 -> 2,031 us
// (40 TFLOP/s).
constexpr int TN = 4, TILE_CTAS = 4, TILE_N = 16 * TN, TILE_K = 32, TILE_ROW = TILE_K + 4, TILE_STAGES = 3;
template <typename TA, typename TC, int TM, bool VEC>
__global__ void __launch_bounds__(128, TILE_CTAS)
gemm_simt_tile_kernel(const TA* __restrict__ A, const TA* __restrict__ W, const float* __restrict__ bias,
                      TC* __restrict__ C, int M, int N, int K, Order o, int m_tiles) {
  constexpr int BM = 8 * TM, STAGE = (BM + TILE_N) * TILE_ROW;
  extern __shared__ float4 tile_smem[];
  float* ring = reinterpret_cast<float*>(tile_smem);
  fz_grid_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);      // 16 x 8 threads, a warp 8 x 4 of them
  const int m0 = (blockIdx.x % m_tiles) * BM, n0 = (blockIdx.x / m_tiles) * TILE_N;
  const int k_first = blockIdx.z * o.per_group * o.chunk, k_end = min(K, k_first + o.per_group * o.chunk);
  const int stages = (k_end - k_first + TILE_K - 1) / TILE_K, per_chunk = o.chunk / TILE_K;

  auto load = [&](int s, bool w_rows) {
    float* at = ring + (s % TILE_STAGES) * STAGE + (w_rows ? BM * TILE_ROW : 0);
    const int k = k_first + s * TILE_K + (tid & 7) * 4;
    const int first = w_rows ? n0 : m0, limit = w_rows ? N : M;
#pragma unroll
    for (int i = 0; i < (w_rows ? TILE_N : BM) / 16; ++i) {
      const int row = (tid >> 3) + 16 * i;
      stage4<TA, VEC>(at + row * TILE_ROW + (tid & 7) * 4, w_rows ? W : A, first + row, K, k, k_end, first + row < limit);
    }
  };

  float acc[TM][TN], tot[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = tot[i][j] = 0.f;

#pragma unroll
  for (int s = 0; s < TILE_STAGES - 1; ++s)
    if (s < stages) load(s, true);
  fz_grid_wait();
#pragma unroll
  for (int s = 0; s < TILE_STAGES - 1; ++s) {
    if (s < stages) load(s, false);
    cp_commit();
  }
  int left = per_chunk;
  for (int s = 0; s < stages; ++s) {
    cp_wait<TILE_STAGES - 2>();
    __syncthreads();
    if (s + TILE_STAGES - 1 < stages) {
      load(s + TILE_STAGES - 1, true);
      load(s + TILE_STAGES - 1, false);
    }
    cp_commit();
    const float* as = ring + (s % TILE_STAGES) * STAGE + ty * TILE_ROW;
    const float* ws = ring + (s % TILE_STAGES) * STAGE + (BM + tx) * TILE_ROW;
#pragma unroll 2
    for (int q = 0; q < TILE_K / 4; ++q) {
      float4 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + 16 * j * TILE_ROW + 4 * q);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(as + 8 * i * TILE_ROW + 4 * q);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
      }
    }
    if (--left == 0 || s + 1 == stages) {
      left = per_chunk;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          tot[i][j] += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }
  cp_wait<0>();
  if (o.groups == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + ty + 8 * i;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int n = n0 + tx + 16 * j;
        if (n >= N) continue;
        float v = tot[i][j];
        if (bias) v += bias[n];
        C[(size_t)m * N + n] = Cvt<TC>::from_f(v);
      }
    }
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) ring[(ty + 8 * i) * TILE_N + tx + 16 * j] = tot[i][j];
  cluster.sync();
  for (int e = blockIdx.z * 128 + tid; e < BM * TILE_N; e += 128 * o.groups) {      // the blocks share the tile
    const int m = m0 + e / TILE_N, n = n0 + e % TILE_N;
    if (m >= M || n >= N) continue;
    float part[8];
#pragma unroll
    for (int g = 0; g < 8; ++g)
      if (g < o.groups) part[g] = cluster.map_shared_rank(ring, g)[e];
    float v = 0.f;
#pragma unroll
    for (int g = 0; g < 8; ++g)
      if (g < o.groups) v += part[g];
    if (bias) v += bias[n];
    C[(size_t)m * N + n] = Cvt<TC>::from_f(v);
  }
  cluster.sync();      // nobody leaves while its tile may still be read
}

// ---- many rows and columns
// Products of one group whose tiles of 64 x 128 outputs give every SM two blocks: 128 threads with 8 x 8 outputs each, 16 k
// per stage. A stage is fetched into registers while the one before is multiplied and then lies in shared memory k by k, so
// that a thread reads its 8 and 8 values of a k as 16-byte pieces and multiplies pairs of columns with `__ffma2_rn` (each
// half rounds as fmaf, so the bits are the tile kernel's): half as many instructions, and fewer that wait for a register
// bank, which held the tile kernel (0.39 cycles of dispatch stall per instruction) at 40 TFLOP/s. Measured: 300 x 896 ->
// 9,728 160 -> 137 us, 300 x 896 -> 151,936 2,031 -> 1,750 us (47 TFLOP/s), 64 rows of it 435 -> 390; with one block per
// SM (100 x 896 -> 9,728) it loses, 82 -> 92 us.
constexpr int WIDE_N = 128, WIDE_K = 16;
template <typename TA, typename TC, bool VEC>
__global__ void __launch_bounds__(128, 2)
gemm_simt_wide_kernel(const TA* __restrict__ A, const TA* __restrict__ W, const float* __restrict__ bias,
                      TC* __restrict__ C, int M, int N, int K, Order o, int m_tiles) {
  constexpr int TM = 8, BM = 8 * TM, STAGE = (BM + WIDE_N) * WIDE_K, A_PASSES = BM / 32, W_PASSES = WIDE_N / 32;
  __shared__ __align__(16) float buf[2 * STAGE];      // two stages of [k][64 rows of A], [k][128 rows of W]
  fz_grid_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);      // 16 x 8 threads, a warp 8 x 4 of them
  const int m0 = (blockIdx.x % m_tiles) * BM, n0 = (blockIdx.x / m_tiles) * WIDE_N;
  const int stages = (K + WIDE_K - 1) / WIDE_K, per_chunk = o.chunk / WIDE_K;
  // staging: four lanes to a row (four k each), 32 rows a pass. Row r, k lies at [k][r ^ 8 (k / 4)]: the four lanes' rows
  // then go to different banks, and pieces of eight rows stay whole.
  const int lrow = tid >> 2, lk = (tid & 3) * 4, lswz = (tid & 3) * 8;

  auto fetch = [&](const TA* base, int row, int limit, int s) {
    const int k = s * WIDE_K + lk;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < limit) {
      const TA* at = base + (long long)row * K + k;
      if constexpr (VEC) {
        if (k < K) v = *reinterpret_cast<const float4*>(at);
      } else {
        if (k < K) v.x = Cvt<TA>::to_f(at[0]);
        if (k + 1 < K) v.y = Cvt<TA>::to_f(at[1]);
        if (k + 2 < K) v.z = Cvt<TA>::to_f(at[2]);
        if (k + 3 < K) v.w = Cvt<TA>::to_f(at[3]);
      }
    }
    return v;
  };
  auto put = [&](float* at, int width, int row, float4 v) {
    at[lk * width + (row ^ lswz)] = v.x;
    at[(lk + 1) * width + (row ^ lswz)] = v.y;
    at[(lk + 2) * width + (row ^ lswz)] = v.z;
    at[(lk + 3) * width + (row ^ lswz)] = v.w;
  };
  float4 fa[A_PASSES], fw[W_PASSES];
  auto fetch_a = [&](int s) {
#pragma unroll
    for (int i = 0; i < A_PASSES; ++i) fa[i] = fetch(A, m0 + lrow + 32 * i, M, s);
  };
  auto fetch_w = [&](int s) {
#pragma unroll
    for (int i = 0; i < W_PASSES; ++i) fw[i] = fetch(W, n0 + lrow + 32 * i, N, s);
  };
  auto put_stage = [&](int which) {
    float* at = buf + which * STAGE;
#pragma unroll
    for (int i = 0; i < A_PASSES; ++i) put(at, BM, lrow + 32 * i, fa[i]);
#pragma unroll
    for (int i = 0; i < W_PASSES; ++i) put(at + BM * WIDE_K, WIDE_N, lrow + 32 * i, fw[i]);
  };

  float2 acc[TM][4], tot[TM][4];      // columns tx * 4 + 0, 1 | 2, 3 and the same 64 further on
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = tot[i][j] = make_float2(0.f, 0.f);

  fetch_w(0);      // (no kernel of a step writes weights)
  fz_grid_wait();
  fetch_a(0);
  put_stage(0);
  __syncthreads();
  int left = per_chunk;
  for (int s = 0; s < stages; ++s) {
    const bool more = s + 1 < stages;
    if (more) {
      fetch_w(s + 1);
      fetch_a(s + 1);
    }
    const float* as = buf + (s & 1) * STAGE;
    const float* ws = as + BM * WIDE_K;
#pragma unroll
    for (int k = 0; k < WIDE_K; ++k) {
      const int swz = (k >> 2) * 8;
      alignas(16) float a[TM];
#pragma unroll
      for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(a + i) = *reinterpret_cast<const float4*>(as + k * BM + ((ty * TM + i) ^ swz));
      alignas(16) float2 w[4];
      *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(ws + k * WIDE_N + ((tx * 4) ^ swz));
      *reinterpret_cast<float4*>(w + 2) = *reinterpret_cast<const float4*>(ws + k * WIDE_N + ((tx * 4 + 64) ^ swz));
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(aa, w[j], acc[i][j]);
      }
    }
    if (--left == 0 || !more) {
      left = per_chunk;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          tot[i][j] = __fadd2_rn(tot[i][j], acc[i][j]);
          acc[i][j] = make_float2(0.f, 0.f);
        }
    }
    if (more) put_stage((s + 1) & 1);      // (that buffer was last read a stage ago, before the barrier)
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n0 + tx * 4 + (j & 3) + (j >> 2) * 64;
      if (n >= N) continue;
      float v = j & 1 ? tot[i][j >> 1].y : tot[i][j >> 1].x;
      if (bias) v += bias[n];
      C[(size_t)m * N + n] = Cvt<TC>::from_f(v);
    }
  }
}

template <typename TA, typename TC, int MR, int RPL, bool VEC, bool DEEP>
int launch_few(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, Order o, cudaStream_t stream) {
  using F = Few<MR, RPL, DEEP>;
  const int warps = (o.chunks + 3) / 4, stages = o.chunk / FEW_K, slots = stages < F::STAGES ? stages : F::STAGES;
  const size_t ring = sizeof(float) * (size_t)warps * slots * F::STAGE, sums = sizeof(float) * (size_t)o.chunks * MR * 8 * RPL;
  const size_t smem = ring > sums ? ring : sums;
  auto kern = gemm_simt_few_kernel<TA, TC, MR, RPL, VEC, DEEP>;
  FZ_RAISE_SMEM(kern);
  fz_launch(kern, dim3((N + 8 * RPL - 1) / (8 * RPL)), dim3(32 * warps), smem, stream, (const TA*)A, (const TA*)W, bias, (TC*)C, M, N, K, o, slots);
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

template <typename TA, typename TC, int TM, bool VEC>
int launch_tile(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, Order o, cudaStream_t stream) {
  const long long m_tiles = (M + 8 * TM - 1) / (8 * TM), tiles = m_tiles * ((N + TILE_N - 1) / TILE_N);
  if (tiles > 2147483647LL) return FZ_TOO_LARGE;
  // Blocks of a cluster may be put on one SM while others idle: few blocks ask for enough shared memory to be spread out.
  const long long per_sm = (tiles * o.groups + 147) / 148;
  size_t smem = sizeof(float) * TILE_STAGES * (size_t)(8 * TM + TILE_N) * TILE_ROW;
  if (per_sm < TILE_CTAS && smem < 220 * 1024 / per_sm) smem = 220 * 1024 / per_sm / 1024 * 1024;
  auto kern = gemm_simt_tile_kernel<TA, TC, TM, VEC>;
  FZ_RAISE_SMEM(kern);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, 1, o.groups);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (o.groups > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = o.groups;
  }
  if (fz_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaLaunchKernelEx(&cfg, kern, (const TA*)A, (const TA*)W, bias, (TC*)C, M, N, K, o, (int)m_tiles);
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

template <typename TA, typename TC, bool VEC>
int launch_wide(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, Order o, cudaStream_t stream) {
  const int m_tiles = (M + 63) / 64;
  const long long tiles = (long long)m_tiles * ((N + WIDE_N - 1) / WIDE_N);
  if (tiles > 2147483647LL) return FZ_TOO_LARGE;
  fz_launch(gemm_simt_wide_kernel<TA, TC, VEC>, dim3((unsigned)tiles), dim3(128), 0, stream, (const TA*)A, (const TA*)W, bias, (TC*)C, M, N, K, o, m_tiles);
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

// Two columns per lane (every value of A read once for both) from 256 blocks on.
template <typename TA, typename TC, int MR, bool VEC>
int launch_few_n(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, Order o, cudaStream_t stream) {
  if (N >= 4096) return launch_few<TA, TC, MR, 2, VEC, false>(A, W, bias, C, M, N, K, o, stream);
  if constexpr (VEC)      // (asynchronous copies alone gain from depth)
    if ((N + 7) / 8 <= 148) return launch_few<TA, TC, MR, 1, VEC, true>(A, W, bias, C, M, N, K, o, stream);
  return launch_few<TA, TC, MR, 1, VEC, false>(A, W, bias, C, M, N, K, o, stream);
}

template <typename TA, typename TC, bool VEC>
int launch_rows(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, cudaStream_t stream) {
  const Order o = order_of(N, K);
  // Few rows read W at memory's pace up to 8 and still beat tiles at 16 (16 rows: 896 -> 9,728 26 us, tiles 42 at 17; 896 -> 151,936
  // 230 us, 251 at 17). Wide tiles from two blocks per SM on (see there).
  if (M <= 1) return launch_few_n<TA, TC, 1, VEC>(A, W, bias, C, M, N, K, o, stream);
  if (M <= 2) return launch_few_n<TA, TC, 2, VEC>(A, W, bias, C, M, N, K, o, stream);
  if (M <= 4) return launch_few_n<TA, TC, 4, VEC>(A, W, bias, C, M, N, K, o, stream);
  if (M <= 8) return launch_few_n<TA, TC, 8, VEC>(A, W, bias, C, M, N, K, o, stream);
  if (M <= 16) return launch_few_n<TA, TC, 16, VEC>(A, W, bias, C, M, N, K, o, stream);
  // Tiles of 32 rows waste less than tiles of 64 up to 32 (43 against 62 us) and are done in half the time where all of them
  // start at once: 200 x 97 -> 384 in bfloat16 6.9 us, 10.9 with 64 rows, 300 x 256 -> 96 6.5, 10.0; operands that are read one by
  // one gain up to three per SM (64 x 897 -> 9,728, 304 tiles, 92, 112; 128 x 897 -> 1,152, 504, loses 23, 30), the others lose
  // in places (64 x 4,864 -> 896, 224 tiles, 32, 29).
  const long long tiles32 = (long long)((M + 31) / 32) * ((N + TILE_N - 1) / TILE_N) * o.groups;
  if (M <= 32 || tiles32 <= (VEC ? 148 : 444)) return launch_tile<TA, TC, 4, VEC>(A, W, bias, C, M, N, K, o, stream);
  if (o.groups == 1 && (long long)((M + 63) / 64) * ((N + WIDE_N - 1) / WIDE_N) >= 296)
    return launch_wide<TA, TC, VEC>(A, W, bias, C, M, N, K, o, stream);
  return launch_tile<TA, TC, 8, VEC>(A, W, bias, C, M, N, K, o, stream);
}

template <typename TA, typename TC>
int launch(const void* A, const void* W, const float* bias, void* C, int M, int N, int K, cudaStream_t stream) {
  if constexpr (sizeof(TA) == 4)
    if (K % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0) return launch_rows<TA, TC, true>(A, W, bias, C, M, N, K, stream);
  return launch_rows<TA, TC, false>(A, W, bias, C, M, N, K, stream);
}
}  // namespace

// in_dtype: dtype of A and W; out_dtype: dtype of C. bias (float32) may be null.
FZ_API int fz_gemm_simt(const void* A, const void* W, const float* bias, void* C, int in_dtype, int out_dtype, int M,
                        int N, int K, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return FZ_OK;
  if (K <= 0) return FZ_BAD_SHAPE;
  if (M > 16 * 65535) return FZ_TOO_LARGE;      // (rows and their tiles are counted in int)
  if (in_dtype == FZ_F32 && out_dtype == FZ_F32) return launch<float, float>(A, W, bias, C, M, N, K, stream);
  if (in_dtype == FZ_BF16 && out_dtype == FZ_F32) return launch<__nv_bfloat16, float>(A, W, bias, C, M, N, K, stream);
  if (in_dtype == FZ_BF16 && out_dtype == FZ_BF16) return launch<__nv_bfloat16, __nv_bfloat16>(A, W, bias, C, M, N, K, stream);
  return FZ_BAD_DTYPE;
}

#ifdef FZ_TIMELINE
FZ_TIMELINE_READER(gemm_simt)
#endif
