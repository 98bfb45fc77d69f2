// Paged attention with 32-bit arithmetic on CUDA cores: the attention of the float32 path (prompt portions and decoded
// tokens alike), and the general fallback of the bfloat16 path.
//
// Keys are walked in chunks of 32 whose boundaries are multiples of 32 in absolute position: chunk c holds keys 32c ..
// 32c+31, lane j scores key 32c+j, and the running (max, sum, accumulator) is updated chunk by chunk in rising c. A row's
// chunks are cut into at most eight spans of equal length (two chunks at least); a span starts afresh, and the spans'
// results are merged in order. The order of every sum therefore depends only on the row's own position and window, never
// on the batch, the cut of the prompt or the pages used (the reference's general kernel stages 32-key chunks in shared
// memory the same way: fusezap/device/cuda_kernels/attention.py:330-436).
//
//   scores s_j = (q . k_j) * scale over keys max(0, p - window + 1) <= j <= p of the row's own request (window 0: all),
//   out = sum_j exp(s_j - max) v_j / sum_j exp(s_j - max)                       (fusezap/serve/kv_cache.py:258-274)
//
// A block has a few successive rows of one portion, one kv head and up to 32 (row, query head) pairs, which share every
// chunk's keys and values (copied to shared memory up to three chunks ahead); warp w has pairs w, w + W, ... Few rows: a row
// per block, and the spans of a row go to the eight blocks of a cluster, merged through distributed shared memory. Bound by
// latency at the path's sizes: a chain of chunks, each a copy, a dot product per lane and a walk over 32 values. Measured
// at 14 heads of 64 over 2 kv heads (one block per row and kv head, no spans, copies element by element): 4 rows of 250 to
// 500 keys 8.4 us (146 inside a step), 400 prompt rows 74 (118), 200 rows of 150 to 300 keys 43 (68).
#include "common.cuh"
#include <cooperative_groups.h>
#include <math.h>
namespace cg = cooperative_groups;

namespace {
constexpr int CHUNK = 32;
constexpr int MAX_WARPS = 8;
constexpr int MAX_HD = 512;
constexpr int SPANS = 8, SPAN_CHUNKS = 2;      // most spans of a row; fewest chunks of a span
constexpr int MAX_ROWS = 8;                    // rows of a block (a power of two, fewer than a warp's lanes)

// (row, head) pairs per warp: what fits in registers beside DPL output dimensions per lane, twice
template <int DPL> struct Pairs { static constexpr int PER_WARP = DPL <= 4 ? 4 : DPL <= 8 ? 2 : 1; };

__device__ __forceinline__ float4 four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}

// The merge of a span's (m, l, a) into what the spans before it gave; `keep` and `add` are the two weights.
__device__ __forceinline__ void span_weights(float& M, float m, float& keep, float& add) {
  const float mn = fmaxf(M, m);
  keep = expf(M - mn);
  add = expf(m - mn);
  M = mn;
}
__device__ __forceinline__ float span_add(float total, float part, float keep, float add) { return __fmaf_rn(total, keep, __fmul_rn(part, add)); }

__device__ __forceinline__ int span_length(int chunks) {
  const int len = (chunks + SPANS - 1) / SPANS;
  return len < SPAN_CHUNKS ? SPAN_CHUNKS : len;
}

struct Args {
  const int *pos, *seq_row, *table;
  long long page_stride;
  int mb, page_size, N, Hq, Hkv, hd, hdp, G_all, GS, slices, rows, window, buffers;
  float scale;
  int* err;
};

// Blocks of 256 threads per SM that the registers are to leave room for. (Left to itself the compiler keeps some of the kernels
// with four pairs per warp to 76 registers and others to 140, 20 % slower either way; with one pair 86 registers in place
// of 64 cost 100 rows of 64 20 %, 64 in place of 85 16 rows of 80 in bfloat16 24 %.)
template <int DPL, int PW> constexpr int per_sm() { return DPL > 8 ? 1 : DPL > 4 || PW > 2 ? 2 : DPL > 2 || PW > 1 ? 3 : 4; }

// VEC: rows of keys and values start on 16-byte boundaries and are whole 16-byte pieces (asynchronous copies).
// SPLIT: one row per block, the blocks of a cluster along z take a span each.
// PW: pairs per warp at most.
template <typename T, int DPL, int PW, bool VEC, bool SPLIT>
__global__ void __launch_bounds__(32 * MAX_WARPS, (per_sm<DPL, PW>()))
attn_simt_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool, T* __restrict__ out, Args A) {
  constexpr int PAD = 16 / sizeof(T);
  extern __shared__ float4 attn_smem[];
  fz_grid_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
  const int hd = A.hd, hdp = A.hdp, ks = hdp + PAD;
  // (a kv head's query heads beyond GS are another block's: slices along x, which has room for them beside any number of heads)
  const int kvh = blockIdx.y, g_base = (blockIdx.x % A.slices) * A.GS, G = min(A.GS, A.G_all - g_base);
  const int first = blockIdx.x / A.slices;
  const int head0 = kvh * A.G_all + g_base;
  // Positions, rows and block tables are the step's metadata, which the host wrote before its first kernel: they are read
  // ahead of the wait on the kernel before. Queries, keys and values are not.
  const int row = A.seq_row[first], p0 = A.pos[first];
  int rows = 1;
  if (!SPLIT && A.rows > 1 && row >= 0) {
    // The rows of the block: of the run of neighbouring rows of one request at successive positions that row `first` is in,
    // those up to the next position that is a multiple of A.rows. The block of a row in the middle has nothing to do.
    const int i = lane - 1, n = first + i;      // lane 0: is the row before this one in the same block? else: row first + i?
    const bool joined = i < A.rows && n >= 0 && n < A.N && A.seq_row[n] == row && A.pos[n] == p0 + i && (p0 + max(i, 0)) % A.rows != 0;
    const unsigned int run = __ballot_sync(0xffffffffu, joined || i == 0);
    if (run & 1u) {
      fz_grid_wait();
      return;
    }
    rows = __ffs(~(run >> 1)) - 1;
  }
  // shared memory: per buffer keys [32][hdp + PAD] and values [32][hdp], then queries [pair][hdp] and weights [warp][PW][32] in float32
  T* kv = reinterpret_cast<T*>(attn_smem);
  const int kv_size = CHUNK * (ks + hdp);
  float* Qs = reinterpret_cast<float*>(kv + A.buffers * kv_size);
  float* Ps = Qs + A.rows * G * hdp + warp * PW * CHUNK;

  if (row < 0) {      // a padding row gives zeros
    fz_grid_wait();
    if (!SPLIT || blockIdx.z == 0)
      for (int i = threadIdx.x; i < G * hd; i += blockDim.x) out[((size_t)first * A.Hq + head0) * hd + i] = Cvt<T>::from_f(0.f);
    return;
  }
  const int pairs = rows * G;
  int at[PW];      // where a pair's query lies (a warp without one computes the last pair's scores and drops them)
#pragma unroll
  for (int a = 0; a < PW; ++a) at[a] = min(warp + a * W, pairs - 1) * hdp;
  const int lo_min = A.window > 0 ? max(0, p0 - A.window + 1) : 0, p_max = p0 + rows - 1;
  int c_first = lo_min / CHUNK, c_last = p_max / CHUNK;
  int spans = 1;
  if constexpr (SPLIT) {
    const int chunks = c_last - c_first + 1, len = span_length(chunks);
    spans = (chunks + len - 1) / len;
    c_first += blockIdx.z * len;
    c_last = min(c_last, c_first + len - 1);
  }
  // per pair: the span being walked (m, l, acc), what the spans before it gave (M, L, tot), the chunk where the next span starts
  float m[PW], l[PW], acc[PW][DPL], M[PW], L[PW], tot[PW][DPL];
  int cut[PW];
#pragma unroll
  for (int a = 0; a < PW; ++a) {
    m[a] = M[a] = -INFINITY;
    l[a] = L[a] = 0.f;
    cut[a] = -1;
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[a][i] = tot[a][i] = 0.f;
  }
  const int* trow = A.table + (size_t)row * A.mb;
  const long long head_off = (long long)kvh * A.page_size * hd;

  // Where the chunk's keys lie, a lane each (-1: not seen by any row, or without a page): asked for one chunk before the
  // copies that need it.
  auto find = [&](int c) {
    const int key = c * CHUNK + lane;
    long long off = -1;
    if (c <= c_last && key >= lo_min && key <= p_max) {
      const int page = trow[key / A.page_size];
      if (page >= 0) off = (long long)page * A.page_stride + head_off + (long long)(key % A.page_size) * hd;
      else atomicOr(A.err, FZ_ERR_NO_PAGE);
    }
    return off;
  };
  auto load = [&](int c, long long where) {
    T* Ks = kv + (c & (A.buffers - 1)) * kv_size;
    T* Vs = Ks + CHUNK * ks;
    if constexpr (VEC) {
      for (int j = warp; c <= c_last && j < CHUNK; j += W) {
        long long off = __shfl_sync(0xffffffffu, where, j);
        const bool ok = off >= 0;
        if (!ok) off = 0;
        for (int e = lane * PAD; e < 2 * hd; e += 32 * PAD) {
          const bool is_k = e < hd;
          const int d = is_k ? e : e - hd;
          fz_copy16(is_k ? Ks + j * ks + d : Vs + j * hdp + d, (is_k ? k_pool : v_pool) + off + d, ok);
        }
      }
    } else if (c <= c_last) {
#pragma unroll DPL <= 2 ? 4 : 1
      for (int j = warp; j < CHUNK; j += W) {      // (a few keys' values on their way before the first is stored)
        const long long off = __shfl_sync(0xffffffffu, where, j);
        T k[DPL], v[DPL];
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
          const int d = lane + 32 * i;
          const bool in = off >= 0 && d < hd;
          k[i] = in ? k_pool[off + d] : Cvt<T>::from_f(0.f);
          v[i] = in ? v_pool[off + d] : Cvt<T>::from_f(0.f);
        }
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
          const int d = lane + 32 * i;
          if (d < hdp) {
            Ks[j * ks + d] = k[i];
            Vs[j * hdp + d] = v[i];
          }
        }
      }
    }
    if constexpr (VEC) asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // The ring of `buffers` chunks (1, 2 or 4): all but one are filled here, the last in the loop, a chunk ahead.
  const int ahead = A.buffers - 1;
  long long early[3], next = -1;
#pragma unroll
  for (int i = 0; i < 3; ++i) early[i] = i < ahead ? find(c_first + i) : -1;
  next = find(c_first + ahead);
  fz_grid_wait();
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < ahead) load(c_first + i, early[i]);
  for (int pair = warp; pair < pairs; pair += W) {
    const T* from = q + ((size_t)(first + pair / G) * A.Hq + head0 + pair % G) * hd;
    for (int d = lane; d < hdp; d += 32) Qs[pair * hdp + d] = d < hd ? Cvt<T>::to_f(from[d]) : 0.f;
  }
  for (int c = c_first; c <= c_last; ++c) {
    load(c + ahead, next);
    next = find(c + ahead + 1);
    if constexpr (VEC) {
      if (ahead == 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
      else if (ahead == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const T* Ks = kv + (c & (A.buffers - 1)) * kv_size;
    const T* Vs = Ks + CHUNK * ks;
    // scores of the warp's pairs: four partial sums over d mod 4 each, added up as (0 + 1) + (2 + 3)
    float s[PW][4];
#pragma unroll
    for (int a = 0; a < PW; ++a) s[a][0] = s[a][1] = s[a][2] = s[a][3] = 0.f;
#pragma unroll 4
    for (int d = 0; d < hdp; d += 4) {
      const float4 k4 = four(Ks + lane * ks + d);
#pragma unroll
      for (int a = 0; a < PW; ++a) {
        const float4 q4 = four(Qs + at[a] + d);
        s[a][0] = fmaf(q4.x, k4.x, s[a][0]);
        s[a][1] = fmaf(q4.y, k4.y, s[a][1]);
        s[a][2] = fmaf(q4.z, k4.z, s[a][2]);
        s[a][3] = fmaf(q4.w, k4.w, s[a][3]);
      }
    }
    // j_from .. j_to: the chunk's keys that a pair's row sees (none: the chunk lies outside its row's range, and the pair
    // stays as it is). The pairs' maxima, exponentials and sums run side by side.
    int j_from[PW], j_to[PW];
    float sc[PW], top[PW], sum[PW], corr[PW];
    bool whole = true;
#pragma unroll
    for (int a = 0; a < PW; ++a) {
      const int pair = warp + a * W;
      j_from[a] = 0;
      j_to[a] = -1;
      if (pair < pairs) {
        const int p = p0 + pair / G, lo = A.window > 0 ? max(0, p - A.window + 1) : 0;
        j_from[a] = max(lo - c * CHUNK, 0);
        j_to[a] = min(p - c * CHUNK, CHUNK - 1);
        whole = whole && j_from[a] == 0 && j_to[a] == CHUNK - 1;
        if constexpr (!SPLIT) {
          if (j_from[a] <= j_to[a]) {
            if (cut[a] < 0) cut[a] = lo / CHUNK + span_length(p / CHUNK - lo / CHUNK + 1);
            if (c == cut[a]) {      // a new span: the last one joins the total
              if (M[a] == -INFINITY && L[a] == 0.f) {
                M[a] = m[a];
                L[a] = l[a];
#pragma unroll
                for (int i = 0; i < DPL; ++i) tot[a][i] = acc[a][i];
              } else {
                float keep, add;
                span_weights(M[a], m[a], keep, add);
                L[a] = span_add(L[a], l[a], keep, add);
#pragma unroll
                for (int i = 0; i < DPL; ++i) tot[a][i] = span_add(tot[a][i], acc[a][i], keep, add);
              }
              cut[a] += span_length(p / CHUNK - lo / CHUNK + 1);
              m[a] = -INFINITY;
              l[a] = 0.f;
#pragma unroll
              for (int i = 0; i < DPL; ++i) acc[a][i] = 0.f;
            }
          }
        }
      }
      const bool valid = lane >= j_from[a] && lane <= j_to[a];
      sc[a] = valid ? __fmul_rn((s[a][0] + s[a][1]) + (s[a][2] + s[a][3]), A.scale) : -INFINITY;
      top[a] = sc[a];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int a = 0; a < PW; ++a) top[a] = fmaxf(top[a], __shfl_xor_sync(0xffffffffu, top[a], o));
#pragma unroll
    for (int a = 0; a < PW; ++a) {
      const bool live = j_from[a] <= j_to[a];
      top[a] = fmaxf(m[a], top[a]);       // finite where the pair's row sees a key of the chunk; else nothing below uses it
      const float pj = lane >= j_from[a] && lane <= j_to[a] ? expf(sc[a] - top[a]) : 0.f;
      corr[a] = live ? expf(m[a] - top[a]) : 1.f;               // 0 for the first chunk of a span (m = -inf)
      sum[a] = pj;
      Ps[a * CHUNK + lane] = pj;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int a = 0; a < PW; ++a) sum[a] += __shfl_xor_sync(0xffffffffu, sum[a], o);
#pragma unroll
    for (int a = 0; a < PW; ++a) {
      if (j_from[a] <= j_to[a]) {
        l[a] = __fmaf_rn(l[a], corr[a], sum[a]);
        m[a] = top[a];
      }
#pragma unroll
      for (int i = 0; i < DPL; ++i) acc[a][i] *= corr[a];
    }
    __syncwarp();
    for (int j = 0; j < CHUNK; j += 4) {
      float v[4][DPL];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < DPL; ++i) v[u][i] = lane + 32 * i < hdp ? Cvt<T>::to_f(Vs[(j + u) * hdp + lane + 32 * i]) : 0.f;
#pragma unroll
      for (int a = 0; a < PW; ++a) {
        const float4 p4 = four(Ps + a * CHUNK + j);
        const float pw[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          // (a key that the row does not see takes no part, whatever its value: 0 * inf)
          const bool seen = whole || (j + u >= j_from[a] && j + u <= j_to[a]);
#pragma unroll
          for (int i = 0; i < DPL; ++i) acc[a][i] = seen ? fmaf(pw[u], v[u][i], acc[a][i]) : acc[a][i];
        }
      }
    }
    __syncthreads();      // the chunk is consumed
  }

  if constexpr (SPLIT) {
    // a span's result per head: max, sum, accumulator; the cluster's blocks share the heads' values and merge in order
    cg::cluster_group cluster = cg::this_cluster();
    float* part = reinterpret_cast<float*>(kv);      // [head][2 + hd]
#pragma unroll
    for (int a = 0; a < PW; ++a) {
      const int g = warp + a * W;
      if (g >= G || (int)blockIdx.z >= spans) break;
      if (lane == 0) {
        part[g * (hd + 2)] = m[a];
        part[g * (hd + 2) + 1] = l[a];
      }
#pragma unroll
      for (int i = 0; i < DPL; ++i)
        if (lane + 32 * i < hd) part[g * (hd + 2) + 2 + lane + 32 * i] = acc[a][i];
    }
    cluster.sync();
    for (int e = blockIdx.z * blockDim.x + threadIdx.x; e < G * hd; e += gridDim.z * blockDim.x) {
      const int g = e / hd, d = e - g * hd;
      float sm[SPANS], sl[SPANS], sa[SPANS];
#pragma unroll
      for (int s = 0; s < SPANS; ++s) {
        if (s < spans) {
          const float* from = cluster.map_shared_rank(part, s) + g * (hd + 2);
          sm[s] = from[0];
          sl[s] = from[1];
          sa[s] = from[2 + d];
        }
      }
      float mm = sm[0], ll = sl[0], aa = sa[0];
#pragma unroll
      for (int s = 1; s < SPANS; ++s) {
        if (s < spans) {
          float keep, add;
          span_weights(mm, sm[s], keep, add);
          ll = span_add(ll, sl[s], keep, add);
          aa = span_add(aa, sa[s], keep, add);
        }
      }
      out[((size_t)first * A.Hq + head0) * hd + e] = Cvt<T>::from_f(aa * (1.0f / ll));
    }
    cluster.sync();      // nobody leaves while its results may still be read
  } else {
#pragma unroll
    for (int a = 0; a < PW; ++a) {
      const int pair = warp + a * W;
      if (pair >= pairs) break;
      if (M[a] == -INFINITY && L[a] == 0.f) {      // one span
        L[a] = l[a];
#pragma unroll
        for (int i = 0; i < DPL; ++i) tot[a][i] = acc[a][i];
      } else {
        float keep, add;
        span_weights(M[a], m[a], keep, add);
        L[a] = span_add(L[a], l[a], keep, add);
#pragma unroll
        for (int i = 0; i < DPL; ++i) tot[a][i] = span_add(tot[a][i], acc[a][i], keep, add);
      }
      const float inv = 1.0f / L[a];
      T* orow = out + ((size_t)(first + pair / G) * A.Hq + head0 + pair % G) * hd;
#pragma unroll
      for (int i = 0; i < DPL; ++i) {
        const int d = lane + 32 * i;
        if (d < hd) orow[d] = Cvt<T>::from_f(tot[a][i] * inv);
      }
    }
  }
}

// Warps, chunks in shared memory and bytes of a block with A.rows rows. A warp without a pair helps with the copies: eight where
// blocks are few (2 heads of 20, 8 rows of 4,000 keys 47 us with two warps, 33 with eight) and where values are copied one
// by one (4 heads of 31 over 2, 296 rows of 4,000 keys 1,229 and 512), else no more than there are pairs (32 heads of 128
// over 8, 4 rows of 4,000 keys 95 us with eight, 71 with four).
struct Block { int warps, buffers; size_t smem; };
template <typename T, int DPL, bool VEC>
Block block_of(const Args& A, int per_warp, bool split) {
  const int G = A.G_all < A.GS ? A.G_all : A.GS, pairs = A.rows * G;
  const long long blocks = (long long)A.N * A.Hkv * A.slices / A.rows * (split ? SPANS : 1);
  const int least = !VEC || blocks <= 148 ? MAX_WARPS : DPL > 4 ? 4 : 2;
  Block b = {pairs < least ? least : pairs < MAX_WARPS ? pairs : MAX_WARPS, 1, 0};
  const size_t kv = sizeof(T) * (size_t)CHUNK * (2 * A.hdp + 16 / sizeof(T)), rest = sizeof(float) * ((size_t)pairs * A.hdp + (size_t)b.warps * per_warp * CHUNK);
  for (int n = 4; n > 1 && b.buffers == 1; n /= 2)      // as many chunks as leave two blocks per SM, two if only one block fits
    if (n * kv + rest <= (size_t)(n > 2 ? 100 : 200) * 1024) b.buffers = n;
  b.smem = b.buffers * kv + rest;
  const size_t part = sizeof(float) * (size_t)G * (A.hd + 2);      // (the spans' results reuse the keys and values)
  if (split && b.smem < part) b.smem = part;
  return b;
}

template <typename T, int DPL, int PW, bool VEC, bool SPLIT>
int launch(const void* q, const void* k_pool, const void* v_pool, void* out, Args A, cudaStream_t stream) {
  const Block block = block_of<T, DPL, VEC>(A, PW, SPLIT);
  const size_t smem = block.smem;
  A.buffers = block.buffers;
  auto kern = attn_simt_kernel<T, DPL, PW, VEC, SPLIT>;
  if (smem > (size_t)FZ_MOST_SMEM) return FZ_TOO_LARGE;
  FZ_RAISE_SMEM(kern);
  cudaLaunchConfig_t cfg = {};
  const long long along_x = (long long)A.N * A.slices;
  if (along_x > 2147483647LL) return FZ_TOO_LARGE;
  cfg.gridDim = dim3((unsigned)along_x, A.Hkv, SPLIT ? SPANS : 1);
  cfg.blockDim = dim3(32 * block.warps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (SPLIT) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = SPANS;
  }
  if (fz_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaLaunchKernelEx(&cfg, kern, (const T*)q, (const T*)k_pool, (const T*)v_pool, (T*)out, A);
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

// A launch with as many pairs per warp as the block's pairs need.
template <typename T, int DPL, bool VEC, bool SPLIT>
int launch_pairs(const void* q, const void* k_pool, const void* v_pool, void* out, Args A, cudaStream_t stream) {
  constexpr int MOST = Pairs<DPL>::PER_WARP;
  const int pairs = A.rows * A.GS;
  if constexpr (MOST >= 4)
    if (pairs > 2 * MAX_WARPS) return launch<T, DPL, 4, VEC, SPLIT>(q, k_pool, v_pool, out, A, stream);
  if constexpr (MOST >= 2)
    if (pairs > MAX_WARPS) return launch<T, DPL, 2, VEC, SPLIT>(q, k_pool, v_pool, out, A, stream);
  return launch<T, DPL, 1, VEC, SPLIT>(q, k_pool, v_pool, out, A, stream);
}

// How a step is split: sets A.GS, A.slices and A.rows, returns whether a row's spans go to the blocks of a cluster.
template <typename T, int DPL, bool VEC>
bool split_step(Args& A, int max_context, int max_run) {
  constexpr int PAIRS = MAX_WARPS * Pairs<DPL>::PER_WARP;
  A.GS = A.G_all < PAIRS ? A.G_all : PAIRS;
  A.slices = (A.G_all + A.GS - 1) / A.GS;
  const long long blocks = (long long)A.N * A.Hkv * A.slices;
  // Spans of a row side by side while their blocks, eight to a row and kv head (or slice of its heads), start within 2.5 rounds,
  // within 6 where rows may have more than 512 keys, and within one where short rows could share keys instead: a short span
  // costs its block more than its keys. us with spans and without, 14 heads of 64 over 2 kv heads: 64 rows (2.3 rounds) of 150
  // to 300 keys 32, 30, 148 rows (5.3) 67, 41; 148 rows of 500 to 1,000 keys 107, 125, 200 rows (7.2) 141, 135. 32 heads of
  // 128 over 8: 16 rows of 300 36, 36, 32 rows of 1,000 (4.6) 105, 125, 64 rows (9.2) 201, 188. 4 heads of 256: 32 rows of 300
  // (1.7) 39, 53, 148 rows of 1,000 (8) 208, 167. A prompt of 200 on 2 heads of 20 36 with spans, 17 sharing.
  A.rows = 1;
  const int pw = (A.GS + MAX_WARPS - 1) / MAX_WARPS, regs = pw > 2 ? per_sm<DPL, 4>() : pw > 1 ? per_sm<DPL, 2>() : per_sm<DPL, 1>();
  const Block b = block_of<T, DPL, VEC>(A, pw, true);
  const int by_smem = (int)(227 * 1024 / (b.smem + 1024)), by_regs = regs * MAX_WARPS / b.warps;
  const long long at_once = 148LL * (by_smem < by_regs ? by_smem : by_regs);
  if (max_context > SPAN_CHUNKS * CHUNK && 2 * SPANS * blocks <= (max_context > 512 ? 12 : max_run < 8 ? 5 : 2) * at_once) return true;
  // Rows that share the keys of a block. Up to a pair per warp they cost nothing (8 heads of 64 over 8, 64 rows behind 3,000
  // keys: 568 us with a row per block, 310 with two, 345 with eight); more only while they leave two blocks per SM, or one
  // where no more fit (14 heads of 64 over 2, 400 rows: 74 us with two rows per block, 84 with four; 1,500 rows 558, 523).
  const int free_rows = MAX_WARPS / A.GS < 1 ? 1 : MAX_WARPS / A.GS;
  A.rows = PAIRS / A.GS < MAX_ROWS ? PAIRS / A.GS : MAX_ROWS;
  while (A.rows > free_rows && (blocks + A.rows - 1) / A.rows < (DPL <= 4 ? 296 : 148)) A.rows /= 2;
  if (A.rows < free_rows) A.rows = free_rows;
  if (A.rows > max_run) A.rows = max_run;
  return false;
}

template <typename T, int DPL, bool VEC>
int choose(const void* q, const void* k_pool, const void* v_pool, void* out, Args A, int max_context, int max_run, cudaStream_t stream) {
  if (split_step<T, DPL, VEC>(A, max_context, max_run)) return launch_pairs<T, DPL, VEC, true>(q, k_pool, v_pool, out, A, stream);
  return launch_pairs<T, DPL, VEC, false>(q, k_pool, v_pool, out, A, stream);
}

template <typename T>
int dispatch(const void* q, const void* k_pool, const void* v_pool, void* out, Args A, int max_context, int max_run, cudaStream_t stream) {
  const bool vec = A.hd * sizeof(T) % 16 == 0 && A.page_stride * sizeof(T) % 16 == 0 && (((uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0;
  const int dpl = (A.hd + 31) / 32;
#define FZ_GO(D)                                                                                        \
  return vec ? choose<T, D, true>(q, k_pool, v_pool, out, A, max_context, max_run, stream)              \
             : choose<T, D, false>(q, k_pool, v_pool, out, A, max_context, max_run, stream)
  if (dpl <= 1) FZ_GO(1);
  if (dpl <= 2) FZ_GO(2);
  if (dpl <= 4) FZ_GO(4);
  if (dpl <= 8) FZ_GO(8);
  if (dpl <= 16) FZ_GO(16);
#undef FZ_GO
  return FZ_BAD_SHAPE;
}
}  // namespace

// Sizes taken: any Hkv, Hq any multiple of Hkv, 0 < hd <= 512. Anything else returns FZ_BAD_SHAPE.
FZ_API int fz_attn_simt_check(int Hq, int Hkv, int hd) {
  if (Hq <= 0 || Hkv <= 0 || hd <= 0 || Hq % Hkv) return FZ_BAD_SHAPE;
  if (hd > MAX_HD || (Hq / Hkv + 31) / 32 > 65535) return FZ_BAD_SHAPE;
  return FZ_OK;
}

// max_context: the longest context among the rows, or more; max_run: the most rows of one portion, or more (they decide how the
// work is split, never the results).
FZ_API int fz_attn_simt(const void* q, const void* k_pool, const void* v_pool, const int* pos, const int* seq_row,
                        const int* table, int mb, long long page_stride, int page_size, void* out, int dtype, int N,
                        int Hq, int Hkv, int hd, float scale, int window, int max_context, int max_run, int* err,
                        cudaStream_t stream) {
  if (N <= 0) return FZ_OK;
  if (fz_attn_simt_check(Hq, Hkv, hd) != FZ_OK || page_size <= 0 || Hkv > 65535) return FZ_BAD_SHAPE;
  Args A = {};
  A.pos = pos;
  A.seq_row = seq_row;
  A.table = table;
  A.page_stride = page_stride;
  A.mb = mb;
  A.page_size = page_size;
  A.N = N;
  A.Hq = Hq;
  A.Hkv = Hkv;
  A.hd = hd;
  A.hdp = (hd + 3) / 4 * 4;
  if (dtype == FZ_BF16) A.hdp = (hd + 7) / 8 * 8;
  A.G_all = Hq / Hkv;
  A.window = window;
  A.scale = scale;
  A.err = err;
  if (dtype == FZ_F32) return dispatch<float>(q, k_pool, v_pool, out, A, max_context, max_run < 1 ? 1 : max_run, stream);
  if (dtype == FZ_BF16) return dispatch<__nv_bfloat16>(q, k_pool, v_pool, out, A, max_context, max_run < 1 ? 1 : max_run, stream);
  return FZ_BAD_DTYPE;
}

// How a step of N rows with 16-byte aligned keys and a head size of at most 64 is split in float32: the most rows of a block, 0 for
// the spans of a row in the blocks of a cluster.
FZ_API int fz_attn_simt_rows(int N, int Hq, int Hkv, int hd, int max_context, int max_run) {
  if (fz_attn_simt_check(Hq, Hkv, hd) != FZ_OK || hd % 4 || hd > 64) return -1;
  Args A = {};
  A.N = N;
  A.Hkv = Hkv;
  A.hd = A.hdp = hd;
  A.G_all = Hq / Hkv;
  const bool spans = hd <= 32 ? split_step<float, 1, true>(A, max_context, max_run) : split_step<float, 2, true>(A, max_context, max_run);
  return spans ? 0 : A.rows;
}

#ifdef FZ_TIMELINE
FZ_TIMELINE_READER(attn_simt)
#endif
