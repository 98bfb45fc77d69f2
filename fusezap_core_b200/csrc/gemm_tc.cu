// bf16 matrix product on the 5th-generation tensor cores: C[M, N] = X[M, K] . W[N, K]^T (+ bias), float32 accumulation.
//
// One kernel serves prompt portions and decoded tokens. Both operands are K-major in global memory, so either can be
// the 128-row operand of `tcgen05.mma`:
//   rows mode  (many tokens): the 128 TMEM lanes are token rows, the instruction's N (BN = 64..256) are output features;
//   swap mode  (few tokens):  the 128 TMEM lanes are output features (rows of W, the operand that has to be streamed
//                             from HBM once), the instruction's N (BN = 16..128) are the token rows; the tile is stored
//                             transposed. Nothing is padded to 128 tokens. (The reference's decode GEMM swaps operands the
//                             same way on sm_90a wgmma: fusezap/device/cuda_kernels/wgmma.py:182-317.)
// Rows mode is persistent: the output tiles are walked token tiles fastest (so the CTAs running at one time share a few
// weight tiles in L2), the MMA lane alternates between two TMEM accumulators, and the epilogue warps store one tile
// while the next one is being computed. Where the token rows fill them, a PAIR of CTAs (a cluster of two) works on each
// 256 x 256 tile with `tcgen05.mma.cta_group::2` (`gemm_tc_rows_pair_kernel`); else one CTA per SM walks 128 x 256 tiles
// (`gemm_tc_rows_kernel`). Products of a few hundred rows with too few tiles for the SMs have their tiles' K ranges cut
// over a cluster (`gemm_tc_rows_split_kernel`, in both forms). Swap mode: a CTA computes one 128 x BN tile over one
// range of K:
//   warp 0  one lane issues the TMA loads (cp.async.bulk.tensor.2d, 128-byte swizzle, 64 k per stage) into a ring of
//           shared-memory stages guarded by full/empty mbarriers; no multicast;
//   warp 1  allocates the TMEM accumulator; one lane issues tcgen05.mma (128 x BN x 16, 4 per stage) and commits each
//           stage's completion to its empty barrier, the last one to the accumulator-ready barrier;
//   warps 2-5  read the accumulator with tcgen05.ld (each warp its own 32 lanes), add the bias and store.
// Split K (swap mode; the count is chosen from N and K only, never from M): the splits of a tile form one thread-block
// cluster. The tokens go in groups of one or four to the CTAs of the cluster: every CTA sends each CTA its float32
// partial sums of that CTA's tokens (`st.async` from registers into the other's shared memory, the bytes counted on a
// barrier there), and each CTA adds the splits' partials of its own tokens in split order 0, 1, 2, ... and stores the
// result. The sum has one fixed order (as the reference's split-K has: wgmma.py:209-239) and no partial ever goes to
// global memory. Waits on this CTA's own mbarriers are bounded by a time limit after which the kernel sets an error bit
// and leaves; the cluster barriers are hardware barriers, not spins.
// Epilogues besides bias + store: SwiGLU over weight rows packed as [64 gate | 64 up] blocks and the rotation of the q and k
// heads with the write of k and v into the paged cache (both modes); for few tokens the residual add with the norm behind
// it, and a per-tile argmax that stores no products at all (the lm_head of a greedy step).
#include "umma.cuh"

namespace {
using namespace fztma;
using namespace fzumma;

constexpr int BM = 128;           // TMEM lanes = rows of the 128-row operand
constexpr int BK = 64;            // k per stage: 64 bf16 = 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
constexpr int NUM_THREADS = 192;  // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue

// ---------------------------------------------------------------------------------------------- cluster helpers
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// The cluster address of shared-memory address `addr` in the cluster's CTA `rank`
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  return remote;
}
// VW floats to a cluster address, their bytes counted on the barrier at `bar` of the same CTA.
template <int VW>
__device__ __forceinline__ void send_floats(uint32_t to, uint32_t bar, const float* v) {
  if constexpr (VW == 4)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(to), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar) : "memory");
  else
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];"
                 ::"r"(to), "f"(v[0]), "r"(bar) : "memory");
}
// `mbar_wait` for bytes that other CTAs of the cluster send. They send whatever happens to their own waits, at the latest
// when these have given up; this CTA waits longer than that, so that it is there when they do.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  unsigned long long t0 = 0;
  for (uint32_t spins = 0;; ++spins) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    if (done) return true;
    if ((spins & 1023u) == 1023u) {
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > 5 * WAIT_LIMIT_NS) return false;
    }
  }
}
// The gated activation of the fused gate/up product. kind 1: silu(g) * u; 2: the tanh form of gelu,
// 0.5 g (1 + tanh(sqrt(2 / pi) (g + 0.044715 g^3))) * u.
__device__ __noinline__ float gelu_mul(float g, float u) {
  return 0.5f * g * (1.0f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
}
__device__ __forceinline__ float glu_mul(float g, float u, int kind) {
  if (kind == 2) return gelu_mul(g, u);
  return g / (1.0f + __expf(-g)) * u;
}
// (value, index) order of numpy.argmax: a NaN is the maximum, among equals the lower index wins; index 0x7fffffff: none
__device__ __forceinline__ bool am_better(float v, int i, float bv, int bi) {
  if (i == 0x7fffffff) return false;
  if (bi == 0x7fffffff) return true;
  const bool vn = isnan(v), bn = isnan(bv);
  if (vn != bn) return vn;
  if (vn) return i < bi;
  if (v != bv) return v > bv;
  return i < bi;
}

struct Params {
  float* c_f32;            // exactly one of c_f32 / c_bf16 is set
  __nv_bfloat16* c_bf16;
  const float* bias;       // over output features, may be null
  int* err;
  int rows;                // token rows (M of the product)
  int feats;               // output features (N of the product)
  int K;
  int splits;
  int stages;
  int parts_in_ring;       // few tokens: the partial sums arrive in the ring's memory (after a cluster barrier), not in memory of their own
  int vec_ok;              // rows mode: C rows are 16-byte aligned, so full groups of 16 columns go out as vectors
  int swiglu;              // W holds [64 gate rows | 64 up rows] blocks: store silu(gate) * up as bf16 [rows, feats / 2]
  // rope != 0 (few tokens: hd divides 128; many: a share of a tile's columns holds whole heads): the features are [q heads | k heads | v heads] of size hd; q and k are rotated
  // by the token's position, q goes to c_bf16 [rows, Hq * hd], k and v to the token's slot of the paged pool
  int rope;
  const float* cos_t;      // [max_len, hd / 2]
  const float* sin_t;
  const int* pos;          // [rows]
  const int* seq_row;      // [rows], negative: padding (q zeros, nothing stored)
  const int* table;        // [requests, mb] block table of the layer's cache group
  int mb;
  __nv_bfloat16* k_pool;
  __nv_bfloat16* v_pool;
  long long page_stride;
  int page_size, write, Hq, Hkv, hd, max_len;
  // relu2 != 0: every output goes out as max(y, 0)^2 of the biased sum y
  int relu2;
  // argmax != 0 (few tokens, no split): nothing is stored but, per token row and 128-feature tile, the largest value
  // and its feature index (numpy's order: a NaN is the maximum, the lower index wins among equals)
  int argmax;
  float* am_val;           // [rows][tiles]
  int* am_idx;
  // x set (few tokens): the product ends in the residual stream and the norm that follows it: x[row] += product + bias (float32),
  // h = x * norm_w in bfloat16, and per row the sums of squares of the new x over the features that one warp finishes, as
  // `ss_parts` numbers. The row's factor 1 / sqrt(mean of squares + eps) is left to the products that read h. (A norm's kernel of
  // its own is 1.5 to 3 us of a chain of dependent kernels, two a layer; h has one rounding either way. Decode steps at
  // Llama-3.1-8B sizes, 1, 8 and 64 rows of 4,096 keys: 2,957 -> 2,847 us, 3,455 -> 3,392, 7,643 -> 7,631; at Qwen2.5-0.5B sizes,
  // 1 row of 300 and 32 of 1,280: 592 -> 545, 879 -> 843.)
  float* x;
  const void* norm_w;      // [feats], float32 or bfloat16 (norm_bf16)
  int norm_bf16;
  __nv_bfloat16* h;
  float* ss_out;           // [rows][ss_parts]
  // ss set: the rows of X are such an h; each output is the product times its row's factor, plus the bias
  const float* ss;         // [rows][ss_parts]
  int ss_parts;
  float ss_mean, ss_eps;   // 1 / the size of a row, and what is added to the mean
};

__device__ __forceinline__ float finished(const Params& p, float y) {
  if (!p.relu2) return y;
  y = fmaxf(y, 0.f);
  return y * y;
}

// ---------------------------------------------------------------------------------------------- few tokens
// Partial sums of a tile lie as [split][group of the receiving CTA][feature of the tile][token of the group]: group g of VW
// tokens goes to rank g % splits, as its (g / splits)-th; 32 lanes of a warp, one feature each, send 128 VW neighbouring bytes.
// Groups of four, of one where a cluster has a CTA for every token: the parts then take a quarter of the memory (with 16 KB of
// parts the O product's CTAs at Llama-3.1-8B sizes do not all fit the SMs at once: 7.8 -> 11.9 us at one row).
__host__ __device__ inline int parts_slots(int cols, int splits, int vw) { return ((cols + vw - 1) / vw + splits - 1) / splits; }
__device__ __forceinline__ int parts_mine(int cols, int splits, int vw, int rank) { return ((cols + vw - 1) / vw - rank + splits - 1) / splits; }

// Where a thread's pair of features of one token goes (null: nowhere) and the angle that it is turned by. `turn` 0: zeros, 1: as
// it is, 2: turned.
struct Place { __nv_bfloat16* dst; float cs, sn; int turn; };

// The sums over the splits, in split order, of one, two or four neighbouring tokens of a group at one feature
__device__ __forceinline__ void add(float& a, float b) { a += b; }
__device__ __forceinline__ void add(float2& a, float2 b) { a.x += b.x; a.y += b.y; }
__device__ __forceinline__ void add(float4& a, float4 b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
template <int NV> struct Vec;
template <> struct Vec<1> { typedef float type; };
template <> struct Vec<2> { typedef float2 type; };
template <> struct Vec<4> { typedef float4 type; };
template <int NV>
__device__ __forceinline__ void sum_parts(const float* at, int splits, int step, float* out) {
  typedef typename Vec<NV>::type V;
  V v[8], acc{};
#pragma unroll
  for (int sp = 0; sp < 8; ++sp)
    if (sp < splits) v[sp] = *(const V*)(at + sp * step);
#pragma unroll
  for (int sp = 0; sp < 8; ++sp)
    if (sp < splits) add(acc, v[sp]);
  *(V*)out = acc;
}

// The epilogue of a tile, as far as it is known when the kernel is compiled (a kernel that held all of them was 80 KB of
// code and took its instructions from L2 on every launch of a decode step).
enum { EP_PLAIN = 0, EP_GLU = 1, EP_ROPE = 2, EP_ARGMAX = 3, EP_NORM = 4 };      // EP_NORM: see Params::x

// (Three or four CTAs to an SM as far as registers go. With 160 a thread, two CTAs took all of an SM's registers and the blocks of
// the kernels after this one could not become resident beside them: a decode step of 64 rows at Llama-3.1-8B sizes 7,730 ->
// 8,090 us.)
template <int BN, int EP, int VW>
__global__ void __launch_bounds__(NUM_THREADS, 4)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  // stages of [A: 128 x 64 bf16][B: BN x 64 bf16], 1024-byte aligned for the swizzle; what the other CTAs send, unless it
  // goes into the stages; the barriers
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = BN < 32 ? 32 : BN;
  constexpr bool PAIRS = EP == EP_GLU || EP == EP_ROPE;      // two features of a tile are finished together
  const int cols = p.rows;      // token rows of the step: at most BN
  const int tile = blockIdx.x, split = blockIdx.z;      // (the splits are the cluster: this CTA's rank is its split)
  constexpr int PART_GROUP = BM * VW, CV = VW > 1 ? VW / 2 : 1;      // floats of a group; tokens of it that one of two threads finishes
  const int slots = parts_slots(cols, p.splits, VW), mine = parts_mine(cols, p.splits, VW, split), part_step = slots * PART_GROUP;
  float* parts = (float*)(smem + (p.parts_in_ring ? 0 : p.stages * STAGE_BYTES));
  uint64_t* full = (uint64_t*)(smem + p.stages * STAGE_BYTES + (p.parts_in_ring ? 0 : p.splits * part_step * 4));
  uint64_t* empty = full + p.stages;
  uint64_t* acc_ready = empty + p.stages;
  uint64_t* parts_here = acc_ready + 1;
  uint32_t* tmem_slot = (uint32_t*)(parts_here + 1);
  int* flag = (int*)(tmem_slot + 1);     // a wait gave up
  float* factor = (float*)(flag + 1);    // [BN] of the tokens that this CTA finishes

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kblocks = (p.K + BK - 1) / BK;
  const int kb0 = kblocks * split / p.splits, nkb = kblocks * (split + 1) / p.splits - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_ready, 1);
    mbar_init(parts_here, 1);
    flag[0] = 0;
    mbar_init_fence();
    if (p.splits > 1) mbar_expect_tx(parts_here, (uint32_t)(p.splits * mine * PART_GROUP * 4));
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_d = *tmem_slot;
  if (p.splits > 1) cluster_arrive();      // this CTA's barrier may be sent to; waited for before the first send
  fz_grid_launch_dependents();

  // An epilogue thread's lane of tensor memory is feature r of the tile. Where two features belong together (gate and up,
  // the two values of a rotated pair) threads r and r + 64 finish features f1 and f2, each for half of a group's tokens.
  const int r = (warp & 3) * 32 + lane, par = r >> 6, q = r & 63;
  const int half = EP == EP_ROPE ? p.hd >> 1 : 64;
  const int j = EP == EP_ROPE ? q % half : q, f1 = PAIRS ? (EP == EP_ROPE ? q / half * p.hd : 0) + j : r, f2 = f1 + half;
  const int feat = tile * BM + f1;
  const bool own = feat < p.feats;
  float nw = 0.f, b1 = 0.f, b2 = 0.f;      // what no kernel of a step writes is asked for ahead of the wait on the kernel before
  // The rotation needs, of every token this thread will finish, the request's row, the position, the page and the angles:
  // loads that depend on one another and on nothing a kernel before this one writes (the host packed the step's metadata
  // before the step began). They are asked for now, and the addresses computed, by the epilogue warps that would otherwise only
  // wait, for the first group of tokens; those of further groups in the loop at the end. (What
  // follows the sums then takes 0.1 us of the product at one row at Qwen2.5-0.5B sizes. One warp per scheduler walks two hundred
  // dependent instructions in a microsecond.)
  Place ahead[CV];
  const int head = EP == EP_ROPE ? feat / p.hd : 0;      // (a tile starts at a head's first feature: hd divides 128)
  auto place = [&](int m, Place& at) {
    at = Place{nullptr, 0.f, 0.f, 0};
    if (m >= cols || !own) return;
    const int row = p.seq_row[m], ps = p.pos[m];
    const bool in_range = ps >= 0 && ps < p.max_len, there = row >= 0 && in_range;
    if (row >= 0 && !in_range && q == 0) atomicOr(p.err, FZ_ERR_POS_RANGE);
    if (head < p.Hq) {
      at.dst = p.c_bf16 + ((size_t)m * p.Hq + head) * p.hd + j;
    } else if (there && p.write) {
      const int page = p.table[(size_t)row * p.mb + ps / p.page_size];
      if (page < 0) {
        if (j == 0 && head == p.Hq) atomicOr(p.err, FZ_ERR_NO_PAGE);
      } else {
        __nv_bfloat16* pool = head < p.Hq + p.Hkv ? p.k_pool : p.v_pool;
        const int h = head - p.Hq - (head < p.Hq + p.Hkv ? 0 : p.Hkv);
        at.dst = pool + (long long)page * p.page_stride + ((long long)h * p.page_size + ps % p.page_size) * p.hd + j;
      }
    }
    if (head >= p.Hq + p.Hkv) at.turn = 1;
    else if (there) {
      at.turn = 2;
      at.cs = p.cos_t[(size_t)ps * half + j];
      at.sn = p.sin_t[(size_t)ps * half + j];
    }
  };
  if (warp >= 2) {
    if (p.bias && own) {
      b1 = p.bias[feat];
      if constexpr (PAIRS) b2 = p.bias[feat + half];
    }
    if constexpr (EP == EP_NORM)
      if (own) nw = p.norm_bf16 ? __bfloat162float(((const __nv_bfloat16*)p.norm_w)[feat]) : ((const float*)p.norm_w)[feat];
    if constexpr (EP == EP_ROPE) {
#pragma unroll
      for (int e = 0; e < CV; ++e)
        if (VW > 1 || par == 0) place(split * VW + par * CV + e, ahead[e]);
    }
    // (Used here, so that the loads cannot be put off to the end: 0.9 us of the q/k/v product with a bias.)
    asm volatile("" ::"f"(b1), "f"(b2), "f"(nw) : "memory");
  }
  if (warp == 1) fz_grid_wait();      // (warp 0 waits after it has requested the first weight stages)
  if (warp == 0) {
    if (lane == 0) {
      // The weights (A) do not depend on the kernel before this one: their first stages are requested before the wait on
      // that kernel, so they stream in while it finishes. Every weight is read once per step: it should leave L2 before
      // the activations, which are read again.
      const uint64_t stream_once = l2_evict_first();
      auto load_weights = [&](int i, int s) {
        tma_load_2d_u32_hint(smem_u32(smem + s * STAGE_BYTES), &map_a, smem_u32(&full[s]), (kb0 + i) * BK, tile * BM, stream_once);
      };
      const int early = nkb < p.stages ? nkb : p.stages;
#pragma unroll 1
      for (int i = 0; i < early; ++i) {
        mbar_expect_tx(&full[i], STAGE_BYTES);
        load_weights(i, i);
      }
      fz_grid_wait();
#pragma unroll 1
      for (int i = 0, s = 0, round = 0; i < nkb; ++i) {
        if (round > 0) {
          if (!mbar_wait(&empty[s], (round - 1) & 1)) { flag[0] = 1; break; }
          mbar_expect_tx(&full[s], STAGE_BYTES);
          load_weights(i, s);
        }
        tma_load_2d(smem + s * STAGE_BYTES + A_BYTES, &map_b, &full[s], (kb0 + i) * BK, 0);
        if (++s == p.stages) { s = 0; ++round; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(BM, BN);
#pragma unroll 1
      for (int i = 0, s = 0, round = 0; i < nkb; ++i) {
        if (!mbar_wait(&full[s], round & 1)) { flag[0] = 1; break; }
        tc_fence_after();
        const uint8_t* sa = smem + s * STAGE_BYTES;
        const uint64_t da = desc_k_major(smem_u32(sa)), db = desc_k_major(smem_u32(sa + A_BYTES));
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)   // 32 bytes further along the swizzled row per 16 k
          umma_bf16(tmem_d, da + (uint64_t)(k * UMMA_K * 2 / 16), db + (uint64_t)(k * UMMA_K * 2 / 16), idesc,
                    (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty[s]);
        if (++s == p.stages) { s = 0; ++round; }
      }
      umma_commit(acc_ready);   // arrives when every MMA issued so far has finished (at once if none was issued)
    }
  }
  if (warp < 2) {
    if (p.splits > 1) {
      cluster_wait();
      if (p.parts_in_ring) cluster_sync_all();
    }
  } else {
    // The epilogue: 4 warps, warp w reads TMEM lanes 32 * (w % 4) ... With a token at most for each CTA of a cluster they walk
    // through what they will do once before they wait, with nothing loaded, sent or stored: its instructions then are in the SM's
    // cache instead of on their way from L2, line by line, at the end of a chain of a few microseconds. Decode steps at
    // Qwen2.5-0.5B sizes, 1 row of 300 keys and 8 of 224, 552 -> 535 us, 618 -> 595; at Llama-3.1-8B sizes, 8 rows of 4,096, 3,415 ->
    // 3,375. With groups of four tokens the code for both passes costs more than it saves (32 rows of 1,280 keys 832 -> 868 us).
    float xs[VW] = {};      // EP_NORM: the stream's values of the tokens that this thread finishes next
    int pass = 1;
    if constexpr (VW == 1) {
      pass = p.splits > 1 ? 0 : 1;
      asm volatile("" : "+r"(pass));      // (two passes through the same code, not two copies of it)
    }
#pragma unroll 1
    for (; pass < 2; ++pass) {
      const bool real = VW > 1 || pass == 1;
      bool ok = true;
      if (real) {
        fz_grid_wait();
        if constexpr (EP == EP_NORM) {
#pragma unroll
          for (int e = 0; e < VW; ++e)
            if (own && split * VW + e < cols) xs[e] = p.x[(size_t)(split * VW + e) * p.feats + feat];
        } else if (p.ss != nullptr) {      // (while the products are under way)
          const int tokens = p.splits > 1 ? mine * VW : cols;
#pragma unroll 4
          for (int t = warp & 3; t < tokens; t += 4) {
            const int m = p.splits > 1 ? (split + t / VW * p.splits) * VW + t % VW : t;
            float sum = 0.f;
            if (m < cols)
              for (int i = lane; i < p.ss_parts; i += 32) sum += p.ss[(size_t)m * p.ss_parts + i];
            sum = warp_sum(sum);
            if (lane == 0) factor[t] = 1.0f / sqrtf(sum * p.ss_mean + p.ss_eps);
          }
          asm volatile("bar.sync 1, 128;" ::: "memory");
        }
        ok = __all_sync(0xffffffffu, mbar_wait(acc_ready, 0));   // warp-uniform: tcgen05.ld is warp-wide
        if (!ok) flag[0] = 1;
        tc_fence_after();
        if (p.splits > 1) {
          // Every CTA sends, whatever became of its waits, and nobody leaves before all that it is sent has arrived: no CTA's
          // memory goes away under a sender. In the ring's memory the parts may arrive once every CTA of the cluster has consumed
          // its stages. (Against sums fetched column by column from the other CTAs' shared memory, with a cluster barrier before and
          // one behind: decode steps at Qwen2.5-0.5B sizes, 1 row of 300 keys 674 -> 592 us, 32 of 1,280 1,057 -> 879; at
          // Llama-3.1-8B sizes 1, 8 and 64 rows of 4,096 keys 3,085 -> 2,957, 3,604 -> 3,455, 7,752 -> 7,643. What follows the
          // accumulator takes 0.5 to 0.9 us of each of a layer's products at Qwen2.5-0.5B sizes at one row, 1.4 to 2.8 at 32.)
          cluster_wait();
          if (p.parts_in_ring) cluster_sync_all();
        }
      }
      const uint32_t taddr = tmem_d + ((uint32_t)((warp & 3) * 32) << 16);
      const bool live = ok && nkb > 0;
      const uint32_t bar = smem_u32(parts_here);
      uint32_t at = smem_u32(parts) + (uint32_t)(split * part_step + r * VW) * 4u, to = 0;
#pragma unroll 1
      for (int c = 0; c < cols; c += 16) {
        float v[16];
        if (live && real) tmem_ld16(taddr + (uint32_t)c, v);
        else {
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = 0.f;
        }
        if (p.splits > 1) {
#pragma unroll
          for (int e = 0; e < 16; e += VW) {
            if (c + e >= cols) break;
            if (real) send_floats<VW>(map_to_cta(at, to), map_to_cta(bar, to), v + e);
            if (++to == (uint32_t)p.splits) { to = 0; at += PART_GROUP * 4; }
          }
        } else if (EP == EP_ARGMAX) {
          // the tile's logits go to the (idle) stage buffers as [token][feature], rows one float apart from a multiple of
          // the bank count, and are searched below
#pragma unroll
          for (int e = 0; e < 16; ++e) ((float*)smem)[(c + e) * (BM + 1) + r] = v[e] + b1;
        } else if (EP == EP_GLU) {
#pragma unroll
          for (int e = 0; e < 16; ++e) ((float*)smem)[(c + e) * BM + r] = v[e];      // [token][feature]
        } else if (EP == EP_ROPE) {
#pragma unroll
          for (int e = 0; e < 16; e += 4) ((float4*)smem)[((c + e) >> 2) * BM + r] = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
        } else if (own) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int m = c + e;
            if (m < cols) {
              const float y = finished(p, fmaf(v[e], p.ss ? factor[m] : 1.f, b1));
              if (p.c_f32) p.c_f32[(size_t)m * p.feats + feat] = y;
              else p.c_bf16[(size_t)m * p.feats + feat] = __float2bfloat16_rn(y);
            }
          }
        }
      }
      bool summed = true;      // this thread's tokens are complete in `parts`
      if (p.splits > 1) {
        if (real) summed = mbar_wait_cluster(parts_here, 0);
        if (!summed) flag[0] = 1;
      } else if (EP != EP_PLAIN) asm volatile("bar.sync 1, 128;" ::: "memory");

      if (EP == EP_GLU && p.splits == 1) {
        // K not split: the tile is complete in this CTA's shared memory. A warp takes every fourth token, a lane two
        // neighbouring features of the 64.
        const int f = 2 * lane, g0 = tile * BM + f;
        if (ok && g0 < p.feats) {
          float2 bg = make_float2(0.f, 0.f), bu = bg;
          if (p.bias) { bg = make_float2(p.bias[g0], p.bias[g0 + 1]); bu = make_float2(p.bias[g0 + 64], p.bias[g0 + 65]); }
          const float* t = (const float*)smem + f;
          __nv_bfloat16* dst = p.c_bf16 + tile * 64 + f;
#pragma unroll 4
          for (int c = warp & 3; c < cols; c += 4) {
            const float2 g = *(const float2*)(t + c * BM), u = *(const float2*)(t + c * BM + 64);
            const float sc = p.ss ? factor[c] : 1.f;      // (times one: the sum's bits)
            const __nv_bfloat162 y = __floats2bfloat162_rn(glu_mul(fmaf(g.x, sc, bg.x), fmaf(u.x, sc, bu.x), p.swiglu), glu_mul(fmaf(g.y, sc, bg.y), fmaf(u.y, sc, bu.y), p.swiglu));
            *(__nv_bfloat162*)(dst + (size_t)c * (p.feats >> 1)) = y;
          }
        }
      } else if (EP == EP_ARGMAX) {
        // 128 / BN threads share a token: each scans its part of the tile's 128 features in rising order (so the lower
        // index wins among equals), then the parts are merged in rising order
        constexpr int TPC = BM / BN < 1 ? 1 : BM / BN;          // threads per token
        constexpr int SEG = BM / TPC;                            // features per thread
        const float* am = (const float*)smem;
        float* best_v = (float*)smem + BN * (BM + 1);            // [BN][TPC]
        int* best_i = (int*)(best_v + BN * TPC);
        const int col = r % BN, seg = r / BN;                    // (for BN = 128 every thread has a token of its own)
        float x = 0.f;
        int ix = 0x7fffffff;
        if (seg < TPC) {
#pragma unroll 4
          for (int i = 0; i < SEG; ++i) {
            const int f = seg * SEG + i, ft = tile * BM + f;
            if (ft < p.feats && am_better(am[col * (BM + 1) + f], ft, x, ix)) { x = am[col * (BM + 1) + f]; ix = ft; }
          }
          best_v[col * TPC + seg] = x;
          best_i[col * TPC + seg] = ix;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (seg == 0 && col < cols) {
#pragma unroll 1
          for (int sgm = 1; sgm < TPC; ++sgm)
            if (am_better(best_v[col * TPC + sgm], best_i[col * TPC + sgm], x, ix)) { x = best_v[col * TPC + sgm]; ix = best_i[col * TPC + sgm]; }
          p.am_val[(size_t)col * gridDim.x + tile] = x;
          p.am_idx[(size_t)col * gridDim.x + tile] = ix;
        }
      } else if constexpr (EP == EP_NORM) {
        summed = __all_sync(0xffffffffu, summed);
#pragma unroll 1
        for (int i = 0; i < mine && summed; ++i) {      // (a warp's lanes stay together: they add up their squares)
          alignas(16) float y[VW];
          float sq[VW], old[VW];
#pragma unroll
          for (int e = 0; e < VW; ++e) {
            old[e] = xs[e];
            const int m = (split + (i + 1) * p.splits) * VW + e;
            if (real && own && m < cols) xs[e] = p.x[(size_t)m * p.feats + feat];
          }
          sum_parts<VW>(parts + i * PART_GROUP + r * VW, p.splits, part_step, y);
#pragma unroll
          for (int e = 0; e < VW; ++e) {
            const int m = (split + i * p.splits) * VW + e;
            sq[e] = 0.f;
            if (own && m < cols) {
              const size_t at = (size_t)m * p.feats + feat;
              const float v = old[e] + (y[e] + b1);
              if (real) {
                p.x[at] = v;
                p.h[at] = __float2bfloat16_rn(v * nw);
              }
              sq[e] = v * v;
            }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int e = 0; e < VW; ++e) sq[e] += __shfl_xor_sync(0xffffffffu, sq[e], o);
#pragma unroll
          for (int e = 0; e < VW; ++e) {
            const int m = (split + i * p.splits) * VW + e;
            if (real && lane == e && m < cols) p.ss_out[(size_t)m * p.ss_parts + tile * 4 + (warp & 3)] = sq[e];
          }
        }
      } else if constexpr (EP == EP_PLAIN) {
        if (p.splits > 1 && summed && own) {
#pragma unroll 1
          for (int i = 0; i < mine; ++i) {
            alignas(16) float y[VW];
            sum_parts<VW>(parts + i * PART_GROUP + r * VW, p.splits, part_step, y);
#pragma unroll
            for (int e = 0; e < VW; ++e) {
              const int m = (split + i * p.splits) * VW + e;
              if (m >= cols) break;
              const float v = finished(p, fmaf(y[e], p.ss ? factor[i * VW + e] : 1.f, b1));
              if (!real) continue;
              if (p.c_f32) p.c_f32[(size_t)m * p.feats + feat] = v;
              else p.c_bf16[(size_t)m * p.feats + feat] = __float2bfloat16_rn(v);
            }
          }
        }
      } else if (summed && ok && own && (VW > 1 || par == 0)) {
#pragma unroll (EP == EP_GLU ? 2 : 1)
        for (int i = 0; i < mine; ++i) {
          const float* at = parts + i * PART_GROUP + par * CV;
          alignas(8) float s1[CV], s2[CV];
          sum_parts<CV>(at + f1 * VW, p.splits, part_step, s1);
          sum_parts<CV>(at + f2 * VW, p.splits, part_step, s2);
#pragma unroll
          for (int e = 0; e < CV; ++e) {
            const int m = (split + i * p.splits) * VW + par * CV + e;
            if (m >= cols) break;
            const float sc = p.ss ? factor[i * VW + par * CV + e] : 1.f;
            const float v1 = fmaf(s1[e], sc, b1), v2 = fmaf(s2[e], sc, b2);
            if constexpr (EP == EP_GLU) {
              const __nv_bfloat16 y = __float2bfloat16_rn(glu_mul(v1, v2, p.swiglu));
              if (real) p.c_bf16[(size_t)m * (p.feats >> 1) + tile * 64 + q] = y;
            } else {
              Place& at = ahead[e];
              if (VW > 1 && i > 0) place(m, at);
              float o1 = 0.f, o2 = 0.f;
              if (at.turn == 2) fz_rope_pair(v1, v2, at.cs, at.sn, o1, o2);
              else if (at.turn == 1) { o1 = v1; o2 = v2; }
              const __nv_bfloat16 y1 = __float2bfloat16_rn(o1), y2 = __float2bfloat16_rn(o2);
              if (real && at.dst != nullptr) {
                at.dst[0] = y1;
                at.dst[half] = y2;
              }
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_d, TMEM_COLS);
  }
  if (threadIdx.x == 0 && flag[0]) atomicOr(p.err, FZ_ERR_WAIT_TIMEOUT);
}

// Rows mode: one thread's lane (token row `row`) of a finished accumulator of BN columns at `taddr`, with the bias added,
// to the output's columns n0 .. n0 + BN - 1 (or, with the fused SwiGLU, to its packed half); of these the `part`-th of PARTS
// equal shares. Every lane of the warp takes part in the loads from tensor memory whether or not its row exists or is stored: the
// loads are warp-wide instructions, so no lane leaves an iteration early (what follows a load is guarded instead) and the lanes
// meet at the head of every iteration.
//
// With p.rope the columns are whole heads [q | k | v] (the head size divides a share): q and k are rotated by the row's position, q
// goes to c_bf16, k and v to the token's slot of the paged pools, as the rotation's kernel does from the product's float32 output,
// with the same roundings. `RowPlace`: what a row's rotation needs, looked up while the tile is being computed.
// (The rotation's kernel read the product from L2 and wrote half of it again: 16.8 us of a layer of 2,048 rows at Llama-3.1-8B sizes
// beside 93 of the product, 89 to 92 together; a layer 826 -> 783 to 805 us, a whole prompt 26.86 -> 26.63 ms, where the runs of one side
// differ by 1.5 %. 2,100 rows at Qwen2.5-0.5B sizes 13.7 + 3.8 -> 15.0. 507 rows at the former 31.5 + 12.3 -> 34.2, but 6 us of that
// come back in the attention of the decoded rows behind it, whose blocks find no room beside the pairs'.)
struct RowPlace { int there, ps; long long slot; };      // slot: of the row's key in a page's first head, negative: not stored
__device__ __forceinline__ RowPlace row_place(const Params& p, int row, bool first) {
  RowPlace at{0, 0, -1};
  if (!p.rope || row >= p.rows) return at;
  const int seq = p.seq_row[row];
  at.ps = p.pos[row];
  const bool in_range = at.ps >= 0 && at.ps < p.max_len;
  if (seq >= 0 && !in_range && first) atomicOr(p.err, FZ_ERR_POS_RANGE);
  at.there = seq >= 0 && in_range;
  if (at.there && p.write) {
    const int page = p.table[(size_t)seq * p.mb + at.ps / p.page_size];
    if (page >= 0) at.slot = (long long)page * p.page_stride + (long long)(at.ps % p.page_size) * p.hd;
    else if (first) atomicOr(p.err, FZ_ERR_NO_PAGE);
  }
  return at;
}
__device__ __forceinline__ void store16_bf16(__nv_bfloat16* dst, const float* v) {
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *(const uint32_t*)&h;
  }
  ((uint4*)dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
  ((uint4*)dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
}
template <int BN, int PARTS>
__device__ __forceinline__ void rows_store_tile(const Params& p, uint32_t taddr, int row, int n0, int part, const RowPlace& at) {
  float v[16];
  if (p.rope) {
    float u[16];
    const int half = p.hd >> 1, hq = p.Hq * p.hd, hk = hq + p.Hkv * p.hd;
    const float* cs = p.cos_t + (size_t)(at.there ? at.ps : 0) * half;
    const float* sn = p.sin_t + (size_t)(at.there ? at.ps : 0) * half;
#pragma unroll 1
    for (int c = part * (BN / PARTS); c < (part + 1) * (BN / PARTS); c += 16) {
      if ((c & (p.hd - 1)) >= half) continue;      // (the second values of the pairs go with the first)
      const int n = n0 + c, j = n & (p.hd - 1);
      const bool turn = at.there && n < hk && row < p.rows;
      float4 co[4], si[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        co[i] = turn ? *(const float4*)(cs + j + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
        si[i] = turn ? *(const float4*)(sn + j + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncwarp();
      tmem_ld16(taddr + (uint32_t)c, v);
      tmem_ld16(taddr + (uint32_t)(c + half), u);
      __nv_bfloat16* dst = nullptr;
      if (row < p.rows && n < p.feats) {
        const int head = (n - (n < hk ? hq : hk)) / p.hd;
        if (n < hq) dst = p.c_bf16 + (size_t)row * hq + n;
        else if (at.slot >= 0) dst = (n < hk ? p.k_pool : p.v_pool) + at.slot + (long long)head * p.page_size * p.hd + j;
      }
      if (dst != nullptr) {
        if (p.bias) {
#pragma unroll
          for (int i = 0; i < 16; ++i) { v[i] += p.bias[n + i]; u[i] += p.bias[n + half + i]; }
        }
        if (n < hk) {
          const float* cf = (const float*)co;
          const float* sf = (const float*)si;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float o1 = 0.f, o2 = 0.f;
            if (at.there) fz_rope_pair(v[i], u[i], cf[i], sf[i], o1, o2);
            v[i] = o1;
            u[i] = o2;
          }
        }
        store16_bf16(dst, v);
        store16_bf16(dst + half, u);
      }
    }
    return;
  }
  if (p.swiglu) {
    // columns [128 b, 128 b + 64) are gate, [128 b + 64, 128 b + 128) up of output features 64 (n0 / 128 + b) ..
    float u[16];
    constexpr int FEATS = BN / 2 / PARTS;        // features of a share
#pragma unroll 1
    for (int f = part * FEATS; f < (part + 1) * FEATS; f += 16) {
      const int c = (f >> 6) * 128 + (f & 63);
      __syncwarp();
      tmem_ld16(taddr + (uint32_t)c, v);
      tmem_ld16(taddr + (uint32_t)(c + 64), u);
      const int n = n0 + c;                       // packed index of the gate column
      if (row < p.rows && n < p.feats) {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float g0 = v[i] + (p.bias ? p.bias[n + i] : 0.f), g1 = v[i + 1] + (p.bias ? p.bias[n + i + 1] : 0.f);
          const float u0 = u[i] + (p.bias ? p.bias[n + 64 + i] : 0.f), u1 = u[i + 1] + (p.bias ? p.bias[n + 64 + i + 1] : 0.f);
          const __nv_bfloat162 h2 = __floats2bfloat162_rn(glu_mul(g0, u0, p.swiglu), glu_mul(g1, u1, p.swiglu));
          w[i >> 1] = *(const uint32_t*)&h2;
        }
        uint4* dst = (uint4*)(p.c_bf16 + (size_t)row * (p.feats >> 1) + (n >> 7) * 64 + (n & 63));
        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
    return;
  }
#pragma unroll 1
  for (int c = part * (BN / PARTS); c < (part + 1) * (BN / PARTS); c += 16) {
    __syncwarp();
    tmem_ld16(taddr + (uint32_t)c, v);
    const int n = n0 + c;
    if (row < p.rows && p.vec_ok && n + 16 <= p.feats) {
      if (p.bias) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] += p.bias[n + i];
      }
      if (p.relu2) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = finished(p, v[i]);
      }
      if (p.c_f32) {
        float4* dst = (float4*)(p.c_f32 + (size_t)row * p.feats + n);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      } else {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const __nv_bfloat162 h2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
          w[i] = *(const uint32_t*)&h2;
        }
        uint4* dst = (uint4*)(p.c_bf16 + (size_t)row * p.feats + n);
        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
    } else if (row < p.rows) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (n + i < p.feats) {
          const float y = finished(p, v[i] + (p.bias ? p.bias[n + i] : 0.f));
          if (p.c_f32) p.c_f32[(size_t)row * p.feats + n + i] = y;
          else p.c_bf16[(size_t)row * p.feats + n + i] = __float2bfloat16_rn(y);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------- rows mode, persistent
// C[rows, feats] = X . W^T (+ bias) for many token rows. grid = min(tiles, SMs); tile i of a CTA is tile number
// blockIdx.x + i * gridDim.x, token tile = number % tiles_m, feature tile = number / tiles_m.
template <int BN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tc_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Params p,
                    int tiles_m, int tiles_n) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = 2 * BN <= 32 ? 32 : 2 * BN <= 64 ? 64 : 2 * BN <= 128 ? 128 : 2 * BN <= 256 ? 256 : 512;   // two accumulators (a power of two)
  uint64_t* full = (uint64_t*)(smem + (size_t)p.stages * STAGE_BYTES);
  uint64_t* empty = full + p.stages;
  uint64_t* acc_full = empty + p.stages;     // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2]
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  int* flag = (int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kblocks = (p.K + BK - 1) / BK;
  const int total = tiles_m * tiles_n;
  const int my_tiles = total > (int)blockIdx.x ? (total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 128); }
    flag[0] = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  fz_grid_launch_dependents();
  if (warp != 0) fz_grid_wait();

  if (warp == 0) {
    if (lane == 0) {
      // weights of the first stages before the wait on the previous kernel (they do not depend on it)
      const int first = (int)blockIdx.x;
      const int early = my_tiles > 0 ? (kblocks < p.stages ? kblocks : p.stages) : 0;
      for (int i = 0; i < early; ++i) {
        mbar_expect_tx(&full[i], STAGE_BYTES);
        tma_load_2d(smem + (size_t)i * STAGE_BYTES + A_BYTES, &map_w, &full[i], i * BK, (first / tiles_m) * BN);
      }
      fz_grid_wait();
      // (the stage and its round are kept by counting: this one lane feeds the whole pipeline, and a division per
      // k-block would make it the slowest part)
      int it = 0, s = 0, round = 0;
      bool ok = true;
      for (int j = 0; j < my_tiles && ok; ++j) {
        const int tile = (int)blockIdx.x + j * (int)gridDim.x;
        const int tm = tile % tiles_m, tn = tile / tiles_m;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          uint8_t* sa = smem + (size_t)s * STAGE_BYTES;
          if (it >= early) {
            if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1)) { flag[0] = 1; ok = false; break; }
            mbar_expect_tx(&full[s], STAGE_BYTES);
            tma_load_2d(sa + A_BYTES, &map_w, &full[s], kb * BK, tn * BN);
          }
          tma_load_2d(sa, &map_x, &full[s], kb * BK, tm * BM);
          if (++s == p.stages) { s = 0; ++round; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(BM, BN);
      int s = 0, round = 0;
      bool ok = true;
      for (int j = 0; j < my_tiles && ok; ++j) {
        const int acc = j & 1;
        if (j >= 2 && !mbar_wait(&acc_empty[acc], ((j >> 1) - 1) & 1)) { flag[0] = 1; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full[s], round & 1)) { flag[0] = 1; ok = false; break; }
          tc_fence_after();
          const uint8_t* sa = smem + (size_t)s * STAGE_BYTES;
          const uint64_t da = desc_k_major(smem_u32(sa)), db = desc_k_major(smem_u32(sa + A_BYTES));
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16(tmem_d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit(&empty[s]);
          if (++s == p.stages) { s = 0; ++round; }
        }
        umma_commit(&acc_full[acc]);
      }
    }
  } else {
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    bool ok = true;
    for (int j = 0; j < my_tiles && ok; ++j) {
      const int tile = (int)blockIdx.x + j * (int)gridDim.x;
      const int tm = tile % tiles_m, tn = tile / tiles_m;
      const int acc = j & 1;
      const RowPlace at = row_place(p, tm * BM + r, tn == 0);
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (j >> 1) & 1));
      if (!ok) { flag[0] = 1; break; }
      tc_fence_after();
      // (Four epilogue warps here. Eight, as in the two-SM kernel's plain epilogue, were measured on this kernel and did not pay: the tiles
      // it gets are narrow or few, and 2,048 tokens at Qwen2.5-0.5B sizes took 3.94 ms with them against 3.77 ms.)
      const uint32_t taddr = tmem_base + (uint32_t)(acc * BN) + ((uint32_t)(quad * 32) << 16);
      rows_store_tile<BN, 1>(p, taddr, tm * BM + r, tn * BN, 0, at);
      tc_fence_before();
      mbar_arrive(&acc_empty[acc]);      // this thread has read its lane of the accumulator
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && flag[0]) atomicOr(p.err, FZ_ERR_WAIT_TIMEOUT);
}

template <int BN>
int launch_rows(const CUtensorMap& mx, const CUtensorMap& mw, const Params& p, int tiles_m, int tiles_n, cudaStream_t stream) {
  constexpr int STAGE_BYTES = (BM + BN) * BK * 2;
  const size_t smem = (size_t)p.stages * STAGE_BYTES + 1024 + 8 * (2 * p.stages + 4) + 16;
  FZ_RAISE_SMEM(gemm_tc_rows_kernel<BN>);
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  const int total = tiles_m * tiles_n;
  dim3 grid(total < sms ? total : sms);
  fz_launch(gemm_tc_rows_kernel<BN>, grid, dim3(NUM_THREADS), smem, stream, mx, mw, p, tiles_m, tiles_n);
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

// ---------------------------------------------------------------------------------------------- rows mode, two SMs per tile
// The same product with a pair of CTAs (a cluster of two, on the two SMs of one TPC) on every 256 x 256 output tile:
// `tcgen05.mma.cta_group::2` multiplies 256 token rows by 256 features per instruction, each CTA holding its 128 token
// rows of X and its 128 of the 256 features of W in its own shared memory, and its 128 rows of the accumulator in its own
// tensor memory. Per SM and k-block that is 32 KB of operands instead of 48 KB for the same 128 x 256 outputs: less L2
// and shared-memory traffic, more stages in the ring, half as many instructions to issue.
//
// Who signals whom: each CTA's producer lane loads its own two operand tiles (`cp.async.bulk.tensor ... .cta_group::2`,
// which may count its bytes on the other CTA's barrier; no multicast) and has them counted on the `full` barrier of the
// leader (cluster rank 0), whose producer expects both CTAs' bytes. The leader's MMA lane issues the instructions for
// the pair and commits them to the `empty` (and, per tile, `acc_full`) barriers of BOTH CTAs (`tcgen05.commit` with a CTA
// mask), so each producer refills its own ring and each CTA's epilogue warps read their own tensor memory. One lane of
// each epilogue warp of both CTAs then arrives on the leader's `acc_empty` barrier (count 16). Every wait is bounded;
// both CTAs pass a cluster barrier after the barriers' initialisation and before they leave.
constexpr int PAIR_BN = 256;

__device__ __forceinline__ uint32_t ld_dsmem_u32(uint32_t cluster_addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}
// A tile into this CTA's shared memory, its bytes counted on a barrier given by its cluster address (this CTA's or its
// pair's).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y) : "memory");
}
// D (256 rows over the pair's tensor memories) (+)= A (each CTA's 128 rows) * B (each CTA's half of the N columns)
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives on the barrier at this shared-memory offset in both CTAs of the pair (cluster ranks `first` and `first` + 1) when
// the MMAs issued so far are complete.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint32_t first = 0u) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)(3u << first)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// Tensor memory for a pair: allocated for the pair as one (`cta_group::2`, executed by a warp of each CTA), so that both
// CTAs hold the same columns whatever else is resident on their SMs (measured with two CTAs per SM: separate
// `cta_group::1` allocations gave the CTAs of a pair different columns, this gives them the same); the kernels still
// compare the two addresses before they compute anything.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

// PARTS epilogue warps (warps 2 and up) per quarter of the tensor-memory lanes, each with its share of the tile's columns, so
// that some compute while others wait: with one the epilogue of a tile took longer than the products of a tile with a short
// K, 13 us at K = 896, where the products take 5. The gated epilogue takes four (two: 2,048 x 896 -> 9,728 43.7 us, 34.2 with
// four; 1,024 x 4,096 -> 28,672 177, 172), the plain one, which mostly stores, two (4,096 x 256 -> 8,192 61.7 us, 66.9 with
// four; 2,048 x 512 -> 2,048 11.5, 12.0; others the same with both).
template <int PARTS>
__global__ void __launch_bounds__(64 + 128 * PARTS, 1)
gemm_tc_rows_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Params p,
                         int tiles_m, int tiles_n) {
  constexpr int BN = PAIR_BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int A_BYTES = BM * BK * 2, B_BYTES = (BN / 2) * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr int TMEM_COLS = 2 * BN;          // two accumulators of 256 columns
  uint64_t* full = (uint64_t*)(smem + (size_t)p.stages * STAGE_BYTES);      // used in the leader only
  uint64_t* empty = full + p.stages;
  uint64_t* acc_full = empty + p.stages;     // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2], used in the leader only
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  int* flag = (int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();      // 0: the leader
  const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
  const int kblocks = (p.K + BK - 1) / BK;
  const int total = tiles_m * tiles_n;
  const int my_tiles = total > pair ? (total - pair + pairs - 1) / pairs : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 8 * PARTS); }
    flag[0] = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // the pair's barriers exist and its tensor memory is allocated before anything crosses over
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // One instruction writes the same tensor-memory address in both CTAs: the pair's allocation gives both the same
  // columns; if the two addresses ever differed, nothing is computed and the error is reported.
  const bool same_base = ld_dsmem_u32(map_to_cta(smem_u32(tmem_slot), rank ^ 1u)) == tmem_base;
  fz_grid_launch_dependents();
  if (warp != 0) fz_grid_wait();

  if (!same_base) {
    if (threadIdx.x == 0) flag[0] = 1;
  } else if (warp == 0) {
    if (lane == 0) {
      const uint32_t full0 = map_to_cta(smem_u32(full), 0u);      // the leader's `full` barriers, 8 bytes apart
      const uint32_t s0 = smem_u32(smem);
      // weights of the first stages before the wait on the previous kernel (they do not depend on it)
      const int first = pair;
      const int early = my_tiles > 0 ? (kblocks < p.stages ? kblocks : p.stages) : 0;
      for (int i = 0; i < early; ++i) {
        if (rank == 0) mbar_expect_tx(&full[i], 2 * STAGE_BYTES);
        tma_load_2d_pair(s0 + (uint32_t)(i * STAGE_BYTES + A_BYTES), &map_w, full0 + 8u * (uint32_t)i, i * BK,
                         (first / tiles_m) * BN + (int)rank * (BN / 2));
      }
      fz_grid_wait();
      int it = 0, s = 0, round = 0;
      bool ok = true;
      for (int j = 0; j < my_tiles && ok; ++j) {
        const int tile = pair + j * pairs;
        const int tm = tile % tiles_m, tn = tile / tiles_m;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const uint32_t sa = s0 + (uint32_t)(s * STAGE_BYTES);
          if (it >= early) {
            if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1)) { flag[0] = 1; ok = false; break; }
            if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE_BYTES);
            tma_load_2d_pair(sa + A_BYTES, &map_w, full0 + 8u * (uint32_t)s, kb * BK, tn * BN + (int)rank * (BN / 2));
          }
          tma_load_2d_pair(sa, &map_x, full0 + 8u * (uint32_t)s, kb * BK, (2 * tm + (int)rank) * BM);
          if (++s == p.stages) { s = 0; ++round; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = make_idesc(2 * BM, BN);
      int s = 0, round = 0;
      bool ok = true;
      for (int j = 0; j < my_tiles && ok; ++j) {
        const int acc = j & 1;
        if (j >= 2 && !mbar_wait(&acc_empty[acc], ((j >> 1) - 1) & 1)) { flag[0] = 1; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&full[s], round & 1)) { flag[0] = 1; ok = false; break; }
          tc_fence_after();
          const uint8_t* sa = smem + (size_t)s * STAGE_BYTES;
          const uint64_t da = desc_k_major(smem_u32(sa)), db = desc_k_major(smem_u32(sa + A_BYTES));
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_pair(tmem_d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty[s]);
          if (++s == p.stages) { s = 0; ++round; }
        }
        umma_commit_pair(&acc_full[acc]);
      }
    }
  } else {
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t acc_empty0 = map_to_cta(smem_u32(acc_empty), 0u);
    bool ok = true;
    for (int j = 0; j < my_tiles && ok; ++j) {
      const int tile = pair + j * pairs;
      const int tm = tile % tiles_m, tn = tile / tiles_m;
      const int acc = j & 1;
      const RowPlace at = row_place(p, (2 * tm + (int)rank) * BM + r, tn == 0 && warp < 6);
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (j >> 1) & 1));
      if (!ok) { flag[0] = 1; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t)(acc * BN) + ((uint32_t)(quad * 32) << 16);
      rows_store_tile<BN, PARTS>(p, taddr, (2 * tm + (int)rank) * BM + r, tn * BN, (warp - 2) >> 2, at);
      tc_fence_before();
      __syncwarp();      // every lane of the warp has read its lane of the accumulator
      if (lane == 0) mbar_arrive_cluster(acc_empty0 + 8u * (uint32_t)acc);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // nobody leaves while the other CTA may still signal its barriers or write its tensor memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && flag[0]) atomicOr(p.err, FZ_ERR_WAIT_TIMEOUT);
}

template <int PARTS>
int launch_rows_pair(const CUtensorMap& mx, const CUtensorMap& mw, const Params& p, int tiles_m, int tiles_n, int sms, cudaStream_t stream) {
  constexpr int STAGE_BYTES = (BM + PAIR_BN / 2) * BK * 2;
  const size_t smem = (size_t)p.stages * STAGE_BYTES + 1024 + 8 * (2 * p.stages + 4) + 16;
  FZ_RAISE_SMEM(gemm_tc_rows_pair_kernel<PARTS>);
  const int total = tiles_m * tiles_n, most = sms / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (unsigned)(total < most ? total : most));
  cfg.blockDim = dim3(64 + 128 * PARTS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (fz_pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  attr[na].id = cudaLaunchAttributeClusterDimension;
  attr[na].val.clusterDim.x = 2;
  attr[na].val.clusterDim.y = 1;
  attr[na].val.clusterDim.z = 1;
  ++na;
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t le = cudaLaunchKernelEx(&cfg, gemm_tc_rows_pair_kernel<PARTS>, mx, mw, p, tiles_m, tiles_n);
  if (le != cudaSuccess) return (int)le;
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

// ---------------------------------------------------------------------------------------------- rows mode, K split
// C[rows, feats] = X . W^T (+ bias) for a few hundred token rows, where the 128 x 256 output tiles are far fewer than the
// SMs: a tile's range of K is cut into `splits` pieces, one CTA each, and the CTAs of a tile form a thread-block cluster.
// A CTA can draw operands from L2 / HBM only at the rate its shared-memory ring and the memory latency allow (about
// 90 GB/s), so a tile that walks a long K alone takes its bytes / that rate, whatever the tensor core could do; cut in
// pieces, more SMs draw at once. Every CTA leaves its float32 partial tile in its own shared memory (row-major, rows
// padded by four floats so that neither the writes nor the reads collide on the banks); after a cluster barrier CTA r
// adds, for its share of the tile's columns, the partials of all splits in split order through distributed shared
// memory, adds the bias and stores. No partial goes to global memory; the sum has one fixed order.
constexpr int SPLIT_BN = 256;
constexpr int SPLIT_LD = SPLIT_BN + 4;      // floats per row of the partial tile

__device__ __forceinline__ float4 ld_dsmem_v4(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote));
  return v;
}

// The reduction of the K-cut many-token kernel for one token row: the column groups g0 .. g1 - 1 (four columns each) of
// the tile, every group the sum over the S splits' partial tiles in split order (read through distributed shared
// memory; U groups' loads are in flight together), plus the bias, stored.
template <bool PAIR, int S, int U>
__device__ __forceinline__ void split_reduce_rows(const Params& p, uint32_t base, int g0, int g1, int n0, int row, uint32_t half) {
  for (int gb = g0; gb < g1; gb += U) {
    float4 v[U][S];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int sp = 0; sp < S; ++sp)      // the CTA of split sp that holds the same rows: cluster rank sp, or 2 sp + half
        v[u][sp] = gb + u < g1 ? ld_dsmem_v4(base + (uint32_t)(4 * (gb + u)) * 4u, PAIR ? 2u * (uint32_t)sp + half : (uint32_t)sp)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int g = gb + u;
      if (g >= g1) break;
      const int n = n0 + 4 * g;
      if (n >= p.feats) break;
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int sp = 0; sp < S; ++sp) { acc.x += v[u][sp].x; acc.y += v[u][sp].y; acc.z += v[u][sp].z; acc.w += v[u][sp].w; }
      float y[4] = {acc.x, acc.y, acc.z, acc.w};
      if (p.vec_ok && n + 4 <= p.feats) {
        if (p.bias) {
#pragma unroll
          for (int j = 0; j < 4; ++j) y[j] += p.bias[n + j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = finished(p, y[j]);
        if (p.c_f32) {
          *(float4*)(p.c_f32 + (size_t)row * p.feats + n) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(y[0], y[1]), hi = __floats2bfloat162_rn(y[2], y[3]);
          *(uint2*)(p.c_bf16 + (size_t)row * p.feats + n) = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (n + j < p.feats) {
            const float yj = finished(p, y[j] + (p.bias ? p.bias[n + j] : 0.f));
            if (p.c_f32) p.c_f32[(size_t)row * p.feats + n + j] = yj;
            else p.c_bf16[(size_t)row * p.feats + n + j] = __float2bfloat16_rn(yj);
          }
        }
      }
    }
  }
}

// PAIR: the tile is 256 token rows by 256 features on a pair of CTAs (`tcgen05.mma.cta_group::2`, as in
// `gemm_tc_rows_pair_kernel`: each CTA loads its 128 rows of X and 128 of the 256 features of W, so a CTA draws 32 KB per
// k-block instead of 48 KB), the cluster is (2, 1, splits) with the two CTAs of a pair at neighbouring ranks, and a CTA
// adds up the partial tiles of its own half of the rows.
template <bool PAIR>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tc_rows_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Params p) {
  constexpr int BN = SPLIT_BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int A_BYTES = BM * BK * 2, B_BYTES = (PAIR ? BN / 2 : BN) * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  uint64_t* full = (uint64_t*)(smem + (size_t)p.stages * STAGE_BYTES);      // PAIR: used in the pair's leader only
  uint64_t* empty = full + p.stages;
  uint64_t* acc_ready = empty + p.stages;
  uint32_t* tmem_slot = (uint32_t*)(acc_ready + 1);
  int* flag = (int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const uint32_t half = PAIR ? (rank & 1u) : 0u, leader = PAIR ? (rank & ~1u) : rank;      // which rows of the pair's tile; its first CTA
  const int tm = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, tn = blockIdx.y, split = blockIdx.z;
  const int row0 = PAIR ? (2 * tm + (int)half) * BM : tm * BM;
  const int w_row0 = tn * BN + (PAIR ? (int)half * (BN / 2) : 0);
  const int kblocks = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)kblocks * split / p.splits), kb1 = (int)((long long)kblocks * (split + 1) / p.splits);
  const int nkb = kb1 - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_ready, 1);
    flag[0] = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    if constexpr (PAIR) tmem_alloc_pair(tmem_slot, BN); else tmem_alloc(tmem_slot, BN);
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();      // the pair's barriers and tensor memory exist before anything crosses over
  tc_fence_after();
  const uint32_t tmem_d = *tmem_slot;
  bool same_base = true;      // (one instruction writes the same tensor-memory address in both CTAs of a pair)
  if constexpr (PAIR) same_base = ld_dsmem_u32(map_to_cta(smem_u32(tmem_slot), rank ^ 1u)) == tmem_d;
  fz_grid_launch_dependents();
  if (warp != 0) fz_grid_wait();

  if (!same_base) {
    if (threadIdx.x == 0) flag[0] = 1;
  } else if (warp == 0) {
    if (lane == 0) {
      const uint32_t s0 = smem_u32(smem);
      const uint32_t full0 = PAIR ? map_to_cta(smem_u32(full), leader) : smem_u32(full);      // barriers are 8 bytes apart
      const uint32_t expect = PAIR ? 2 * STAGE_BYTES : STAGE_BYTES;
      auto load = [&](uint32_t dst, const CUtensorMap* map, int stage, int x, int y) {
        if constexpr (PAIR) tma_load_2d_pair(dst, map, full0 + 8u * (uint32_t)stage, x, y);
        else tma_load_2d_u32(dst, map, full0 + 8u * (uint32_t)stage, x, y);
      };
      // the weights of the first stages before the wait on the previous kernel (they do not depend on it)
      const int early = nkb < p.stages ? nkb : p.stages;
      for (int i = 0; i < early; ++i) {
        if (half == 0) mbar_expect_tx(&full[i], expect);
        load(s0 + (uint32_t)(i * STAGE_BYTES + A_BYTES), &map_w, i, (kb0 + i) * BK, w_row0);
      }
      fz_grid_wait();
      for (int i = 0, s = 0, round = 0; i < nkb; ++i) {
        const uint32_t sa = s0 + (uint32_t)(s * STAGE_BYTES);
        if (round > 0) {
          if (!mbar_wait(&empty[s], (round - 1) & 1)) { flag[0] = 1; break; }
          if (half == 0) mbar_expect_tx(&full[s], expect);
          load(sa + A_BYTES, &map_w, s, (kb0 + i) * BK, w_row0);
        }
        load(sa, &map_x, s, (kb0 + i) * BK, row0);
        if (++s == p.stages) { s = 0; ++round; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && half == 0) {
      constexpr uint32_t idesc = make_idesc(PAIR ? 2 * BM : BM, BN);
      for (int i = 0, s = 0, round = 0; i < nkb; ++i) {
        if (!mbar_wait(&full[s], round & 1)) { flag[0] = 1; break; }
        tc_fence_after();
        const uint8_t* sa = smem + (size_t)s * STAGE_BYTES;
        const uint64_t da = desc_k_major(smem_u32(sa)), db = desc_k_major(smem_u32(sa + A_BYTES));
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          if constexpr (PAIR) umma_bf16_pair(tmem_d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (i > 0 || k > 0) ? 1u : 0u);
          else umma_bf16(tmem_d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        if constexpr (PAIR) umma_commit_pair(&empty[s], leader); else umma_commit(&empty[s]);
        if (++s == p.stages) { s = 0; ++round; }
      }
      if constexpr (PAIR) umma_commit_pair(acc_ready, leader); else umma_commit(acc_ready);
    }
  } else {
    // the accumulator -> this CTA's partial tile in shared memory (every stage has been consumed by now, in both CTAs
    // of a pair: the commit covers the pair's instructions, which read both)
    const int quad = warp & 3, r = quad * 32 + lane;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(acc_ready, 0));
    if (!ok) flag[0] = 1;
    tc_fence_after();
    const uint32_t taddr = tmem_d + ((uint32_t)(quad * 32) << 16);
    float* part = (float*)smem + (size_t)r * SPLIT_LD;
    float v[16];
#pragma unroll 1
    for (int c = 0; c < BN; c += 16) {
      if (ok && nkb > 0) tmem_ld16(taddr + (uint32_t)c, v);
      else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < 16; j += 4) *(float4*)(part + c + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
  }
  // every thread of every CTA of the cluster passes both cluster barriers; only the epilogue warps work between them
  cluster_sync_all();
  if (warp >= 2 && same_base) {
    const int r = (warp & 3) * 32 + lane;
    const int row = row0 + r;
    // this CTA's share of the tile's columns, in groups of four
    const int groups = BN / 4;
    const int g0 = (int)((long long)groups * split / p.splits), g1 = (int)((long long)groups * (split + 1) / p.splits);
    const uint32_t base = smem_u32(smem) + (uint32_t)r * (uint32_t)(SPLIT_LD * 4);
    if (row < p.rows) {
      // (with two splits a thread has 32 groups: eight groups' partial tiles are asked for at once, which took 1 to 2 us
      // off products of 28 to 61 us; with four splits and 16 groups the same was measured and lost a little)
      if (p.splits == 2) split_reduce_rows<PAIR, 2, 8>(p, base, g0, g1, tn * BN, row, half);
      else if (p.splits == 4) split_reduce_rows<PAIR, 4, 2>(p, base, g0, g1, tn * BN, row, half);
      else split_reduce_rows<PAIR, 8, 2>(p, base, g0, g1, tn * BN, row, half);
    }
  }
  cluster_sync_all();      // nobody leaves while its shared memory may still be read
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_d, BN); else tmem_dealloc(tmem_d, BN);
  }
  if (threadIdx.x == 0 && flag[0]) atomicOr(p.err, FZ_ERR_WAIT_TIMEOUT);
}

template <bool PAIR>
int launch_rows_split(const CUtensorMap& mx, const CUtensorMap& mw, const Params& p, int tiles_m, int tiles_n, cudaStream_t stream) {
  constexpr int STAGE_BYTES = (BM + (PAIR ? SPLIT_BN / 2 : SPLIT_BN)) * BK * 2;
  const size_t ring = (size_t)p.stages * STAGE_BYTES, partial = (size_t)BM * SPLIT_LD * 4;
  const size_t smem = (ring > partial ? ring : partial) + 1024 + 8 * (2 * p.stages + 1) + 16;
  FZ_RAISE_SMEM(gemm_tc_rows_split_kernel<PAIR>);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((PAIR ? 2 : 1) * tiles_m, tiles_n, p.splits);      // PAIR: tiles_m counts tiles of 256 rows
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (fz_pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  attr[na].id = cudaLaunchAttributeClusterDimension;
  attr[na].val.clusterDim.x = PAIR ? 2 : 1;
  attr[na].val.clusterDim.y = 1;
  attr[na].val.clusterDim.z = (unsigned)p.splits;
  ++na;
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t le = cudaLaunchKernelEx(&cfg, gemm_tc_rows_split_kernel<PAIR>, mx, mw, p);
  if (le != cudaSuccess) return (int)le;
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

// ---------------------------------------------------------------------------------------------- host side
int device_sms() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      sms = 148;
  }
  return sms;
}

template <int BN, int EP, int VW>
int launch_few(const CUtensorMap& ma, const CUtensorMap& mb, Params p, dim3 grid, cudaStream_t stream) {
  constexpr int STAGE_BYTES = (BM + BN) * BK * 2;
  const size_t region = (size_t)p.splits * parts_slots(p.rows, p.splits, VW) * VW * BM * 4;
  size_t smem = (size_t)p.stages * STAGE_BYTES + 1024 + 8 * (2 * p.stages + 2) + 16 + (p.ss ? BN * 4 : 0);
  p.parts_in_ring = 1;
  if (p.splits > 1) {
    // The parts have memory of their own where as many CTAs fit an SM with it as without, or there are no more CTAs than SMs.
    // (The O product at Llama-3.1-8B sizes, 256 CTAs in clusters of eight, three to an SM: with 4 KB more, two to an SM, the
    // last cluster started only when others had left, 7.8 -> 11.3 us.)
    constexpr size_t sm = 228 * 1024, reserved = 1024;
    if (smem + region <= FZ_MOST_SMEM && (sm / (smem + region + reserved) == sm / (smem + reserved) || (int)grid.x * p.splits <= device_sms())) {
      p.parts_in_ring = 0;
      smem += region;
    } else if (region > (size_t)p.stages * STAGE_BYTES) return FZ_BAD_SHAPE;
  }
  const auto kern = gemm_tc_kernel<BN, EP, VW>;
  FZ_RAISE_SMEM(kern);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (fz_pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (p.splits > 1) {      // the splits of one tile are one cluster (z dimension)
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = (unsigned)p.splits;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t le = cudaLaunchKernelEx(&cfg, kern, ma, mb, p);
  if (le != cudaSuccess) return (int)le;
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}
template <int BN, int VW>
int launch_few_ep(const CUtensorMap& ma, const CUtensorMap& mb, const Params& p, dim3 grid, cudaStream_t stream) {
  if (p.swiglu) return launch_few<BN, EP_GLU, VW>(ma, mb, p, grid, stream);
  if (p.x) return p.splits > 1 ? launch_few<BN, EP_NORM, VW>(ma, mb, p, grid, stream) : FZ_BAD_SHAPE;
  if constexpr (BN <= 32)
    if (p.rope) return launch_few<BN, EP_ROPE, VW>(ma, mb, p, grid, stream);
  return launch_few<BN, EP_PLAIN, VW>(ma, mb, p, grid, stream);
}
template <int BN>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, const Params& p, dim3 grid, cudaStream_t stream) {
  if (p.argmax) return launch_few<BN, EP_ARGMAX, 4>(ma, mb, p, grid, stream);
  if constexpr (BN == 16)
    if (p.rows <= p.splits && p.splits > 1) return launch_few_ep<16, 1>(ma, mb, p, grid, stream);
  return launch_few_ep<BN, 4>(ma, mb, p, grid, stream);
}

int pick_stages(int bn) {
  const int stage = (BM + bn) * BK * 2;
  int s = (200 * 1024) / stage;
  if (bn <= 128) s = (100 * 1024) / stage;  // few-token mode: leaves room for two CTAs per SM
  return s < 2 ? 2 : (s > 8 ? 8 : s);
}
}  // namespace

// Can this kernel take the product? K a multiple of 8 (16-byte rows for TMA), operands 16-byte aligned.
FZ_API int fz_gemm_tc_check(const void* x, const void* w, int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return FZ_BAD_SHAPE;
  if (K % 8) return FZ_BAD_SHAPE;
  if (((uintptr_t)x | (uintptr_t)w) & 15) return FZ_BAD_ALIGNMENT;
  return FZ_OK;
}

// The number of K splits for a product with these N and K in swap mode: from N and K only, so that a token row's sum
// order never depends on how many rows share the step.
FZ_API int fz_gemm_tc_splits(int N, int K) {
  const int tiles = (N + BM - 1) / BM, kblocks = (K + BK - 1) / BK;
  // Two CTAs fit each of the 148 SMs, but clusters do not pack the GPCs perfectly: measured on B200, 48 clusters of 6
  // (288 CTAs) need a second wave (19 us for the 6144 x 4096 product) where 48 of 5 (13 us) and 32 of 8 do not. So the
  // CTA count stays at or below 256.
  // (Down to one k-block of 64 per piece: small products are bound by the chain of a single CTA's loads and
  // instructions, not by bytes, and more pieces shorten it. Measured at Qwen2.5-0.5B sizes, batch 8, two engines
  // alternating in one process: at least 4 k-blocks per piece 1.040 ms per step, 3: 0.992, 2: 0.956, 1: 0.936.)
  int s = 256 / tiles;
  if (s > kblocks) s = kblocks;
  if (s > 8) s = 8;                  // a portable cluster holds at most 8 CTAs
  return s < 1 ? 1 : s;
}

// The number of K pieces a product of M > 128 token rows is cut into (1: not cut): only where the 128 x 256 tiles are at
// most half as many as the SMs, no piece shorter than 8 k-blocks of 64, and a power of two: with one CTA per SM, clusters
// of three do not pack the GPCs (measured: 48 clusters of 3 need a second wave, 45 us for the 256 x 6144 x 4096 product
// where 48 of 2 take 29), clusters of 4 and 8 do as long as they cover at most 128 SMs.
FZ_API int fz_gemm_tc_rows_splits(int M, int N, int K) {
  if (M <= BM || N < 256) return 1;
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      sms = 148;
  }
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + 255) / 256);
  const int kblocks = (K + BK - 1) / BK;
  if (2 * tiles > sms) return 1;
  for (int s = 8; s >= 2; s >>= 1)
    if (tiles * s <= (s == 2 ? sms : 128) && kblocks / 8 >= s) return s;
  return 1;
}

// Which many-token kernel takes a product: 0 by the rule below, 1 always one SM per tile, 2 a pair of SMs per tile
// wherever the tile is 256 wide (for measurements and tests; the results differ by nothing but the kernel).
static int g_rows_mode = 0;
FZ_API void fz_gemm_tc_rows_mode(int mode) { g_rows_mode = mode; }

// Does a pair of SMs work on each 256 x 256 tile of this product (M > 128 token rows, not cut along K)? Where the pairs
// have at least half a round of tiles, and the token rows fill the pairs' second halves: an even count of 128-row tiles,
// or so many that the one empty half costs less than the pair gains (measured: 10 to 14 % at 1,024 rows and more).
FZ_API int fz_gemm_tc_rows_pairs(int M, int N, int K) {
  if (M <= BM || N < 256 || g_rows_mode == 1) return 0;
  if (g_rows_mode == 2) return 1;
  const int t128 = (M + BM - 1) / BM;
  const long long tiles = (long long)((t128 + 1) / 2) * ((N + PAIR_BN - 1) / PAIR_BN);
  return ((t128 % 2 == 0 || t128 >= 9) && 4 * tiles >= device_sms()) ? 1 : 0;
}

// The number of K pieces when pairs of SMs work on 256 x 256 tiles of a product that is cut along K (1: not this way).
// Only where the one-SM rule cuts K in two and the 128-row tiles come in an even count (no pair's second half empty):
// the clusters are then (2, 1, 2), as many CTAs as before draw a third fewer bytes each (measured: 29.5 -> 27.6 us for
// 256 x 6144 x 4096, 62.6 -> 54.7 us for 512 x 4096 x 14336). Clusters of (2, 1, 4) do not pack the GPCs: 16 of them
// took 41 us for 256 x 4096 x 4096 where 32 clusters of four one-SM pieces take 24.
FZ_API int fz_gemm_tc_rows_pair_splits(int M, int N, int K) {
  if (g_rows_mode == 1 || fz_gemm_tc_rows_splits(M, N, K) != 2) return 1;
  const int t128 = (M + BM - 1) / BM;
  if (t128 % 2) return 1;
  const long long tiles = (long long)(t128 / 2) * ((N + SPLIT_BN - 1) / SPLIT_BN);
  return tiles * 4 <= 128 ? 2 : 1;
}

// Which kernel takes a product of M > 128 token rows, and in what tiles.
struct RowsPlan {
  enum Kernel { ROWS, PAIR, SPLIT, SPLIT_PAIR } kernel;
  int bn, splits, parts;      // width of a tile; pieces of K; PAIR: groups of four epilogue warps
};
static RowsPlan rows_plan(int M, int N, int K, bool swiglu, int hd = 0) {      // hd: the tile must hold whole heads
  int bn = N >= 256 ? 256 : N >= 128 ? 128 : 64;     // with the fused SwiGLU N = 2 I >= 128, so a tile holds whole blocks
  if (bn == 256 && !swiglu) {
    // So few 128 x 256 tiles that the SMs are not half used, and a K worth cutting: the tiles' K ranges are cut so that
    // about one CTA per SM works (see `gemm_tc_rows_split_kernel`). The count follows from (M, N, K) of the product.
    const int pair_splits = fz_gemm_tc_rows_pair_splits(M, N, K), splits = fz_gemm_tc_rows_splits(M, N, K);
    if (pair_splits > 1) return {RowsPlan::SPLIT_PAIR, SPLIT_BN, pair_splits, 1};
    if (splits > 1) return {RowsPlan::SPLIT, SPLIT_BN, splits, 1};
    // Few token rows: when the 256-wide tiles do not fill the SMs even once, the narrowest width that still fits one
    // round is the fastest (256 x 4096 x 4096 is 32 tiles of 256 columns for 148 SMs, but 52 of 160). Not below 160:
    // a 128-wide instruction reads its operands from shared memory at the rate the tensor core consumes them and runs
    // at about half speed. With more than one round the widest tile stays: measured at 2,048 rows, 160-wide tiles in
    // three rounds (60 -> 72 us) lose against 256-wide ones in two, whatever the count of rounds says.
    const long long tm = (M + BM - 1) / BM;
    if (tm * ((N + 255) / 256) < device_sms()) {
      for (int cand : {224, 192, 160})
        if (tm * ((N + cand - 1) / cand) <= device_sms() && (hd == 0 || cand % hd == 0)) bn = cand;
    }
  }
  // many token rows: a pair of SMs on every 256 x 256 tile (see `gemm_tc_rows_pair_kernel`)
  if (bn == 256 && fz_gemm_tc_rows_pairs(M, N, K)) return {RowsPlan::PAIR, PAIR_BN, 1, swiglu ? 4 : 2};
  return {RowsPlan::ROWS, bn, 1, 1};
}

// x: [M, K] bf16, w: [N, K] bf16, bias: [N] float32 or null, c: [M, N] float32 (out_dtype 0) or bf16 (1).
FZ_API int fz_gemm_tc_qkv_rope_rows(int M, int N, int K, int hd);
static int gemm_tc_impl(const void* x, const void* w, const float* bias, void* c, int out_dtype, int M, int N, int K,
                        const Params& fused, int* err, cudaStream_t stream);

FZ_API int fz_gemm_tc(const void* x, const void* w, const float* bias, void* c, int out_dtype, int M, int N, int K,
                      int* err, cudaStream_t stream) {
  return gemm_tc_impl(x, w, bias, c, out_dtype, M, N, K, Params{}, err, stream);
}

// How many partial sums of squares per row a product that ends in the residual stream and the norm behind it leaves (0: such
// a product is refused). Few rows alone, K cut (up to 16,384 features, K from 72 on), and rows that the next product can read: the sums of squares are 0.2 us beside
// the partial sums that are in shared memory anyway. With many rows a thread finishes a row's piece, 64 bytes here and there of
// the stream, and every tile of the next product needs its rows' factors: 2,048 rows at Llama-3.1-8B sizes 26.9 -> 29.7 ms, 2,100
// rows at Qwen2.5-0.5B sizes 2.96 -> 3.14, so those keep the norm's kernel.
FZ_API int fz_gemm_tc_norm_parts(int M, int N, int K) {
  if (M <= 0 || M > 128 || N <= 0 || N % 8 || K <= 0 || K % 8 || fz_gemm_tc_splits(N, K) == 1) return 0;
  return (N + BM - 1) / BM * 4;
}

// stream [M, N] float32 += x . w^T + bias; h [M, N] bf16 = the new stream * norm_w (float32 or bf16); ss [M, fz_gemm_tc_norm_parts(M, N, K)]: partial
// sums of the new stream's squares.
FZ_API int fz_gemm_tc_add_norm(const void* x, const void* w, const float* bias, float* stream_x, const void* norm_w, int norm_dtype, void* h, float* ss,
                               int M, int N, int K, int* err, cudaStream_t stream) {
  Params f{};
  f.ss_parts = fz_gemm_tc_norm_parts(M, N, K);
  if (f.ss_parts == 0) return FZ_BAD_SHAPE;
  if (norm_dtype != FZ_F32 && norm_dtype != FZ_BF16) return FZ_BAD_DTYPE;
  if ((uintptr_t)h & 15) return FZ_BAD_ALIGNMENT;      // (the next product reads it)
  f.x = stream_x; f.norm_w = norm_w; f.norm_bf16 = norm_dtype == FZ_BF16; f.h = (__nv_bfloat16*)h; f.ss_out = ss;
  return gemm_tc_impl(x, w, bias, h, FZ_BF16, M, N, K, f, err, stream);
}

static void set_factors(Params& f, const float* ss, int ss_parts, float eps, int K) {
  f.ss = ss; f.ss_parts = ss_parts; f.ss_mean = 1.0f / (float)K; f.ss_eps = eps;
}

// `fz_gemm_tc` and `fz_gemm_tc_swiglu` (kind 0, 1, 2) of rows that `fz_gemm_tc_add_norm` left: x is its h, ss and ss_parts its
// partial sums; each row of the product is multiplied by 1 / sqrt(mean of squares + eps).
FZ_API int fz_gemm_tc_normed(const void* x, const float* ss, int ss_parts, float eps, const void* w, const float* bias, void* c, int out_dtype,
                             int M, int N, int K, int kind, int* err, cudaStream_t stream) {
  if (ss == nullptr || ss_parts <= 0 || kind < 0 || kind > 2) return FZ_BAD_SHAPE;
  if (kind && (N % 128 || out_dtype != FZ_BF16)) return FZ_BAD_SHAPE;
  if (kind && ((uintptr_t)c & 15)) return FZ_BAD_ALIGNMENT;
  Params f{};
  f.swiglu = kind;
  set_factors(f, ss, ss_parts, eps, K);
  return gemm_tc_impl(x, w, bias, c, out_dtype, M, N, K, f, err, stream);
}

// Can the query/key/value product of M token rows with heads of size hd end in the rotation and the cache write?
// (a 128-feature tile must hold whole heads; up to 32 rows, where the separate rotation kernel costs more than its work:
// with more rows the epilogue's per-token lookups outweigh the launch they save)
FZ_API int fz_gemm_tc_qkv_rope_check(int M, int hd) {
  return (M >= 1 && M <= 32 && hd >= 2 && hd % 2 == 0 && 128 % hd == 0) ? FZ_OK : FZ_BAD_SHAPE;
}

// The same for many rows (1 or 0): heads of 64 or 128, three tiles of rows and more, and a product whose K is not cut.
FZ_API int fz_gemm_tc_qkv_rope_rows(int M, int N, int K, int hd) {
  if (M <= 2 * BM || N < 256 || (hd != 64 && hd != 128)) return 0;
  const RowsPlan plan = rows_plan(M, N, K, false, hd);
  return plan.splits == 1 && plan.bn / plan.parts % hd == 0 ? 1 : 0;
}

// x: [M, K] bf16; w: [(Hq + 2 Hkv) hd, K] bf16, rows [q heads | k heads | v heads]; bias float32 or null. Rotates the q
// and k heads of every token by its position (pairs j, j + hd / 2; angles from cos_t / sin_t [max_len, hd / 2]) and
// writes q to q_out [M, Hq hd] bf16 and, if `write`, k and v to the token's slot of the paged pools (as the separate
// rotation kernel does, with the same roundings). seq_row < 0: a padding row (q zeros, nothing stored). ss: null, or as in
// `fz_gemm_tc_normed`.
FZ_API int fz_gemm_tc_qkv_rope(const void* x, const float* ss, int ss_parts, float eps, const void* w, const float* bias, int M, int K, const float* cos_t,
                               const float* sin_t, const int* pos, const int* seq_row, const int* table, int mb,
                               void* k_pool, void* v_pool, long long page_stride, int page_size, int write, void* q_out,
                               int Hq, int Hkv, int hd, int max_len, int* err, cudaStream_t stream) {
  if (Hq <= 0 || Hkv <= 0 || page_size <= 0) return FZ_BAD_SHAPE;
  if (fz_gemm_tc_qkv_rope_check(M, hd) != FZ_OK) {
    if (ss || !fz_gemm_tc_qkv_rope_rows(M, (Hq + 2 * Hkv) * hd, K, hd)) return FZ_BAD_SHAPE;
    if (((uintptr_t)q_out | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)cos_t | (uintptr_t)sin_t) & 15 || page_stride % 8) return FZ_BAD_ALIGNMENT;
  }
  Params f{};
  if (ss) set_factors(f, ss, ss_parts, eps, K);
  f.rope = 1;
  f.cos_t = cos_t; f.sin_t = sin_t; f.pos = pos; f.seq_row = seq_row; f.table = table; f.mb = mb;
  f.k_pool = (__nv_bfloat16*)k_pool; f.v_pool = (__nv_bfloat16*)v_pool; f.page_stride = page_stride;
  f.page_size = page_size; f.write = write; f.Hq = Hq; f.Hkv = Hkv; f.hd = hd; f.max_len = max_len;
  return gemm_tc_impl(x, w, bias, q_out, FZ_BF16, M, (Hq + 2 * Hkv) * hd, K, f, err, stream);
}

// The best (value, index) of a row over its tiles' partial results, in tile order; out[r] = the index (0 if none).
__global__ void argmax_tiles_kernel(const float* __restrict__ val, const int* __restrict__ idx, int tiles, int* __restrict__ out) {
  fz_grid_launch_dependents();
  fz_grid_wait();
  __shared__ float s_v[32];
  __shared__ int s_i[32];
  const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float x = 0.f;
  int ix = 0x7fffffff;
  for (int t = threadIdx.x; t < tiles; t += blockDim.x) {
    const float v = val[(size_t)r * tiles + t];
    const int i = idx[(size_t)r * tiles + t];
    if (am_better(v, i, x, ix)) { x = v; ix = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ox = __shfl_xor_sync(0xffffffffu, x, o);
    const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
    if (am_better(ox, oi, x, ix)) { x = ox; ix = oi; }
  }
  if (lane == 0) { s_v[warp] = x; s_i[warp] = ix; }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    x = lane < nw ? s_v[lane] : 0.f;
    ix = lane < nw ? s_i[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ox = __shfl_xor_sync(0xffffffffu, x, o);
      const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
      if (am_better(ox, oi, x, ix)) { x = ox; ix = oi; }
    }
    if (lane == 0) out[r] = ix == 0x7fffffff ? 0 : ix;
  }
}

// Can `fz_gemm_tc_argmax` take the product? Few token rows, and so many output tiles that K is not split.
FZ_API int fz_gemm_tc_argmax_check(int M, int N, int K) {
  return (M >= 1 && M <= 128 && N >= 1 && K >= 8 && K % 8 == 0 && fz_gemm_tc_splits(N, K) == 1) ? FZ_OK : FZ_BAD_SHAPE;
}

// ids[m] = argmax_n (x[m] . w[n] + bias[n]), numpy's order, without writing the products out. scratch_val / scratch_idx:
// M * ceil(N / 128) elements each.
FZ_API int fz_gemm_tc_argmax(const void* x, const void* w, const float* bias, int M, int N, int K, float* scratch_val,
                             int* scratch_idx, int* ids, int* err, cudaStream_t stream) {
  if (fz_gemm_tc_argmax_check(M, N, K) != FZ_OK) return FZ_BAD_SHAPE;
  Params f{};
  f.argmax = 1;
  f.am_val = scratch_val;
  f.am_idx = scratch_idx;
  int st = gemm_tc_impl(x, w, bias, scratch_val, FZ_F32, M, N, K, f, err, stream);
  if (st != FZ_OK) return st;
  fz_launch(argmax_tiles_kernel, dim3(M), dim3(256), 0, stream, (const float*)scratch_val, (const int*)scratch_idx,
            (N + BM - 1) / BM, ids);
  FZ_LAUNCH_CHECK();
  return FZ_OK;
}

// Fused gate/up product and SwiGLU: w is [2 I, K] with rows in blocks of 128 = [64 gate rows | 64 up rows] of the same 64
// features (bias packed the same way, or null); out is bf16 [M, I] = silu(x . gate^T) * (x . up^T). I % 64 == 0.
// kind 1: silu, 2: the tanh form of gelu.
FZ_API int fz_gemm_tc_swiglu(const void* x, const void* w_packed, const float* bias_packed, void* out, int M, int I, int K,
                             int kind, int* err, cudaStream_t stream) {
  if (I <= 0 || I % 64 || (kind != 1 && kind != 2)) return FZ_BAD_SHAPE;
  if (((uintptr_t)out) & 15) return FZ_BAD_ALIGNMENT;
  Params f{};
  f.swiglu = kind;
  return gemm_tc_impl(x, w_packed, bias_packed, out, FZ_BF16, M, 2 * I, K, f, err, stream);
}

// c = max(x . w^T + bias, 0)^2, from the unrounded sums.
FZ_API int fz_gemm_tc_relu2(const void* x, const void* w, const float* bias, void* c, int out_dtype, int M, int N, int K,
                            int* err, cudaStream_t stream) {
  Params f{};
  f.relu2 = 1;
  return gemm_tc_impl(x, w, bias, c, out_dtype, M, N, K, f, err, stream);
}

static int gemm_tc_impl(const void* x, const void* w, const float* bias, void* c, int out_dtype, int M, int N, int K,
                        const Params& fused, int* err, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return FZ_OK;
  int st = fz_gemm_tc_check(x, w, M, N, K);
  if (st != FZ_OK) return st;
  if (out_dtype != FZ_F32 && out_dtype != FZ_BF16) return FZ_BAD_DTYPE;
  if (fused.rope && M > 32 && !fz_gemm_tc_qkv_rope_rows(M, N, K, fused.hd)) return FZ_BAD_SHAPE;
  Params p = fused;
  p.c_f32 = out_dtype == FZ_F32 ? (float*)c : nullptr;
  p.c_bf16 = out_dtype == FZ_BF16 ? (__nv_bfloat16*)c : nullptr;
  p.bias = bias; p.err = err; p.rows = M; p.feats = N; p.K = K;
  p.splits = 1;
  p.vec_ok = (N % 8 == 0 && ((uintptr_t)c & 15) == 0) ? 1 : 0;
  CUtensorMap ma, mb;
  if (M <= 128) {
    // swap mode: W rows are the 128 lanes, the token rows are the instruction's N
    const int bn = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
    p.stages = pick_stages(bn);
    const int tiles = (N + BM - 1) / BM;
    p.splits = fz_gemm_tc_splits(N, K);
    {
      // A CTA that walks few k-blocks gains nothing from a ring deeper than half of them, and the shared memory it
      // leaves free lets blocks of the kernel after this one become resident (and fetch their weights) earlier:
      // measured on the O product of a decode step (8 k-blocks per CTA, 5 -> 4 stages), two engines alternating in one
      // process: batch 1 3.249 -> 3.212 ms per step, batch 8 3.908 -> 3.898; the same on the down product (28 k-blocks
      // per CTA) or on the q/k/v product lost.
      const int per_cta = ((K + BK - 1) / BK + p.splits - 1) / p.splits, enough = per_cta / 2 < 3 ? 3 : per_cta / 2;
      if (p.stages > enough) p.stages = enough;
      // A matrix that the rings of all its CTAs hold whole (up to 24 MB of 148 x 227 KB): then every weight is on its way
      // before the wait on the kernel before, and what follows the wait is the activations, the sums and the store alone.
      // Qwen2.5-0.5B sizes, 300 keys: a decode step of one row 684 -> 668 us, of 8 726 -> 722, of 32 905 -> 900, of 64 the same.
      // Larger ones would only keep the next kernels' blocks off the SMs. (At least three stages: they also hold the parts of 128
      // tokens, 72 KB.)
      const long long ring = (long long)per_cta * (BM + bn) * BK * 2;
      // With up to 16 tokens only where two CTAs could share an SM: a CTA that takes an SM's whole memory starts when the kernel before
      // has left it, a smaller one beside that kernel, its first stages then on their way. (The down product at Qwen2.5-0.5B sizes,
      // 56 CTAs of ten k-blocks, in rings of 10, 7, 5 and 4: a decode step of 1 row of 300 keys 532, 535, 507, 517 us, of 8 of 224 593,
      // 584, 580, 585, of 32 of 1,280, where it gains nothing, 794, 798, 806, 812.)
      if (ring <= (bn == 16 ? 100 : 200) * 1024 && ring * tiles * p.splits <= 24 << 20) p.stages = per_cta < 3 ? 3 : per_cta;
    }
    if ((st = get_map_bf16(w, N, K, BM, &ma)) != FZ_OK) return st;
    if ((st = get_map_bf16(x, M, K, bn, &mb)) != FZ_OK) return st;
    dim3 grid(tiles, 1, p.splits);
    switch (bn) {
      case 16: return launch<16>(ma, mb, p, grid, stream);
      case 32: return launch<32>(ma, mb, p, grid, stream);
      case 64: return launch<64>(ma, mb, p, grid, stream);
      default: return launch<128>(ma, mb, p, grid, stream);
    }
  }
  // rows mode: token rows are the 128 lanes; persistent CTAs with two accumulators
  if (p.x || p.ss) return FZ_BAD_SHAPE;
  const RowsPlan plan = rows_plan(M, N, K, p.swiglu != 0, p.rope ? p.hd : 0);
  p.splits = plan.splits;
  const bool pair = plan.kernel == RowsPlan::PAIR || plan.kernel == RowsPlan::SPLIT_PAIR;
  const int box = pair ? plan.bn / 2 : plan.bn, st_n = (200 * 1024) / ((BM + box) * BK * 2);
  p.stages = st_n < 2 || pair ? st_n : st_n > 8 ? 8 : st_n;
  if (p.stages < 2) p.stages = 2;
  if ((st = get_map_bf16(x, M, K, BM, &ma)) != FZ_OK) return st;
  if ((st = get_map_bf16(w, N, K, box, &mb)) != FZ_OK) return st;
  const int tiles_m = (M + BM - 1) / BM, pairs_m = (M + 2 * BM - 1) / (2 * BM), tiles_n = (N + plan.bn - 1) / plan.bn;
  switch (plan.kernel) {
    case RowsPlan::SPLIT_PAIR: return launch_rows_split<true>(ma, mb, p, pairs_m, tiles_n, stream);
    case RowsPlan::SPLIT: return launch_rows_split<false>(ma, mb, p, tiles_m, tiles_n, stream);
    case RowsPlan::PAIR: return (plan.parts == 4 ? launch_rows_pair<4> : launch_rows_pair<2>)(ma, mb, p, pairs_m, tiles_n, device_sms(), stream);
    default: break;
  }
  switch (plan.bn) {
    case 256: return launch_rows<256>(ma, mb, p, tiles_m, tiles_n, stream);
    case 224: return launch_rows<224>(ma, mb, p, tiles_m, tiles_n, stream);
    case 192: return launch_rows<192>(ma, mb, p, tiles_m, tiles_n, stream);
    case 160: return launch_rows<160>(ma, mb, p, tiles_m, tiles_n, stream);
    case 128: return launch_rows<128>(ma, mb, p, tiles_m, tiles_n, stream);
    default: return launch_rows<64>(ma, mb, p, tiles_m, tiles_n, stream);
  }
}

#ifdef FZ_TIMELINE
FZ_TIMELINE_READER(gemm_tc)
#endif
