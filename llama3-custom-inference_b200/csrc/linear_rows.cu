// out[rows, N] = act(x[rows, K] w[N, K]^T) of few rows (a decode step's tokens), bf16 operands, fp32 accumulation
// (include/l3ci_b200.h, l3ci_linear).
//
// A product of up to 64 rows is bound by reading w once.  What kept the library's kernels from that rate inside a decode step was not
// the stream itself but its edges: each product began to read its weights only when the kernel before it had ended, and drained
// before the next one began.  Here
//   * the weights take the 128-row side of the tcgen05 product and the tokens the narrow one (8, 16, 32 or 64): a CTA moves
//     128 rows of w, 64 columns at a time, through a ring of bulk tensor copies, and the tensor cores keep up with a fraction of
//     their rate, so nothing but the copies is timed;
//   * w does not depend on the kernel before (`early`): the ring is filled before griddepcontrol.wait, and only the tokens are asked
//     for after it.
//     A CTA takes at most half of an SM's shared memory, so that it can start beside the CTAs of the kernel before;
//   * few rows of w: a cluster of 2, 4 or 8 CTAs shares a tile's columns, and adds its parts through distributed shared memory in
//     the order of the ranks (results do not depend on timing);
//   * the activation that follows is done on the fp32 sums: gelu, tanh, or silu(gate) * up (or its clamped form) of a stacked matrix, a tile then being
//     64 gate rows and the 64 up rows of the same outputs.
// Measured in chains on weights beyond L2, us (the library's product and its activation): one row, w 2048 x 2048 3.7 (8.1), 2048 x 8192
// 9.2 (20.2), gated 2 x 8192 x 2048 13.7 (15.3), 128256 x 2048 82 (81); 64 rows 6.8 (5.7), 12.3 (13.7), 16.3 (15.9), 88 (95): the
// extension leaves the shapes that lose to the library.  A step of the 1B model behind 4001 tokens: 696 us, 1103 to 1127 with the library's, and
// 668 with the rotation and the cache write in the projections' last step (a launch a layer less; figures at the kernel).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "host_common.h"
#include "linear_many.h"
#include "mixer_types.cuh"
#include "ptx_sm100.cuh"
#include "tcgen05.cuh"
#include "tensor_map.h"

namespace l3ci {
namespace {

constexpr int kTile = 128;                 // rows of w per tile
constexpr int kDeep = 64;                  // columns per stage: 128 bytes
constexpr int kThreads = 192;              // producer, MMA issue, four output warps
constexpr int kWBytes = kTile * kDeep * 2;
constexpr int kSwap = 8;                   // tokens whose up halves pass through shared memory at a time

// NP: tokens of the narrow side.  The product's least width is 16: of a tile of 8 tokens it reads 8 rows of what lies behind, into
// columns of the accumulator that nobody reads.
template <int NP>
struct LinShape {
  static constexpr int kXBytes = NP * kDeep * 2;
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = NP <= 16 ? 6 : NP == 32 ? 5 : 4;
  static constexpr int kCols = NP < 16 ? 16 : NP;    // of the accumulator
  static constexpr uint32_t kTmem = 2 * kCols;       // two accumulators
  static constexpr int kPartBytes = NP * kTile * 4;  // a tile's parts from the cluster's CTAs
  // the parts lie in the ring, behind one more meeting of the cluster, where a place of their own would cost a stage
  static constexpr bool kInRing = NP > 8;
  static constexpr int kExtraBytes = kInRing ? kSwap * (kTile / 2) * 4 : kPartBytes;
  static constexpr size_t kSmem = 1024 + (size_t)kStages * kStageBytes + kExtraBytes + (2 * kStages + 4) * 8 + 16;
  static_assert(kStages * kStageBytes >= kPartBytes && kExtraBytes >= kSwap * (kTile / 2) * 4, "room for parts and up halves");
  static_assert(2 * (kSmem + 1024) <= 233472, "two CTAs per SM");
};

// Where a wait that ran out is recorded by calls without a status word of their own, until l3ci_linear_poll reads it.
__device__ int g_wait_status = 0;

struct LinParams {
  l3ci_linear_args a;
  int tiles, steps;                        // tiles of w, stages of K
  int group_tiles;                         // tiles of one group
  float limit, alpha;                      // of a gated activation
  l3ci_linear_rope rope;                   // (kernels with ROPE)
};

__device__ __forceinline__ float lin_act(float z, int act) {
  if (act == L3CI_ACT_GELU) return 0.5f * z * (1.f + erff(z * 0.70710678118654752f));
  if (act == L3CI_ACT_TANH) return tanhf(z);
  return z;
}

__device__ __forceinline__ void store_out(const l3ci_linear_args& a, int grp, int t, int n, float v) {
  const long long at = grp * a.out_sg + t * a.out_st + n;
  if (a.out_f32) static_cast<float*>(a.out)[at] = v;
  else static_cast<__nv_bfloat16*>(a.out)[at] = __float2bfloat16_rn(v);
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Address, among the cluster's, of what lies at `addr` in the shared memory of CTA `rank`.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void output_warps_meet() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
// Whether all four output warps are well: they meet at barriers together or not at all.
__device__ __forceinline__ bool output_warps_agree(bool ok) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n" : "=r"(r) : "r"((uint32_t)ok) : "memory");
  return r != 0;
}

// S: CTAs of a cluster, which share a tile's columns of w.  GATE: 1 silu(gate) * up of w's N gate rows and N up rows, 2 its clamped form
// (a kernel of its own: both in one took a layer's step of 64 rows 1 us), 0 none.
// ROPE: the outputs are queries, keys and values, which the last step rotates and puts where l3ci_rot_embed_kv_cache_at does, with its
// bits.  That call took 2.4 us of a layer's 43 at one token and 4001 positions, nearly all of it a launch and a trip to memory each way;
// here the table and the positions come while the sums still run.  A step of one token 696 -> 668 us.
template <int NP, int S, int GATE, bool ROPE>
__global__ void __launch_bounds__(kThreads, 2)
linear_rows_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ LinParams p) {
  using Sh = LinShape<NP>;
  constexpr bool GATED = GATE > 0;
  constexpr int kStages = Sh::kStages;
  constexpr int kOuts = GATED ? kTile / 2 : kTile;     // outputs of a tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t ring = smem_u32(smem);
  float* swap = reinterpret_cast<float*>(smem + kStages * Sh::kStageBytes);     // S == 1: the up halves
  float* parts = Sh::kInRing ? reinterpret_cast<float*>(smem) : swap;           // S > 1: the cluster's parts
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Sh::kStageBytes + Sh::kExtraBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + kStages * 8, done0 = empty0 + kStages * 8, read0 = done0 + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const l3ci_linear_args& a = p.a;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full0 + i * 8, 1);
      mbar_init(empty0 + i * 8, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(done0 + i * 8, 1);
      mbar_init(read0 + i * 8, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&xmap)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&wmap)) : "memory");
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), Sh::kTmem);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // behind the allocation: a CTA of the next kernel must not hold the tensor memory that this one waits for
  pdl_launch_dependents();
  if constexpr (S > 1 && !Sh::kInRing) cluster_arrive();
  const uint32_t tmem = *tmem_slot;
  const int rank = S > 1 ? (int)cluster_rank() : 0;
  const int first = blockIdx.x / S, stride = gridDim.x / S;
  const int k0 = (int)((long long)p.steps * rank / S), steps = (int)((long long)p.steps * (rank + 1) / S) - k0;   // this CTA's stages of a tile
  bool ok = true;
  int asked = 0;                        // stages that this thread has asked for

  constexpr int kOwn = kOuts / S;       // outputs of a cluster's CTA
  // a pair of outputs that are rotated together, of the output warps' threads: the first one's place is looked up ahead of the sums
  struct Pair { int t, j, n; long long pos; float2 turn; };
  auto pair_at = [&](int e) {
    Pair x;
    x.t = e / (kOwn / 2);
    x.j = e % (kOwn / 2) * 2;
    x.n = first * kOuts + rank * kOwn + x.j;
    x.pos = -1;
    x.turn = make_float2(1.f, 0.f);
    if (ROPE && warp >= 2 && x.t < (int)a.rows && x.n < a.N) {
      const long long pos = (long long)p.rope.positions[x.t / p.rope.T] + x.t % p.rope.T;
      if (pos >= 0 && pos < p.rope.freq_rows && pos < p.rope.cache_len) {
        x.pos = pos;
        if (x.n < (p.rope.Hq + p.rope.Hkv) * p.rope.D) x.turn = *reinterpret_cast<const float2*>(p.rope.freq_table + pos * p.rope.D + x.n % p.rope.D);
      }
    }
    return x;
  };
  Pair pair{};

  if (warp == 0) {
    // ---- producer ----
    if (lane == 0) {
      const uint64_t policy_w = l2_evict_first_policy();
      uint64_t policy_x;
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy_x));
      // (one thread's instructions are all that a stage waits for: counters, no divisions, on the way to a copy)
      struct At { int tile, grp, row, k; };
      auto at_tile = [&](int tile) { return At{tile, tile / p.group_tiles, tile % p.group_tiles * kOuts, 0}; };
      auto advance = [&](At& t) {
        if (++t.k == steps) t = at_tile(t.tile + stride);
      };
      auto load_w = [&](int s, const At& t) {
        const uint32_t dst = ring + s * Sh::kStageBytes, bar = full0 + s * 8;
        ++asked;
        mbar_expect_tx(bar, Sh::kStageBytes);
        tma_load_4d(dst, &wmap, bar, (k0 + t.k) * kDeep, t.row, 0, t.grp, policy_w);
        if (GATED) tma_load_4d(dst + kWBytes / 2, &wmap, bar, (k0 + t.k) * kDeep, t.row, 1, t.grp, policy_w);
      };
      auto load_x = [&](int s, const At& t) {
        tma_load_4d(ring + s * Sh::kStageBytes + kWBytes, &xmap, full0 + s * 8, (k0 + t.k) * kDeep, 0, 0, t.grp, policy_x);
      };
      if (!a.early) pdl_wait();
      At w = at_tile(first), x = w;
      int filled = 0;
      for (; filled < kStages && w.tile < p.tiles; ++filled, advance(w)) load_w(filled, w);
      if (a.early) pdl_wait();
      for (int f = 0; f < filled; ++f, advance(x)) load_x(f, x);
      uint32_t parity = 0;
      for (int s = 0; w.tile < p.tiles; advance(w)) {
        if (!mbar_wait_bounded_one(empty0 + s * 8, parity)) { ok = false; break; }
        load_w(s, w);
        load_x(s, w);
        if (++s == kStages) { s = 0; parity ^= 1; }
      }
    }
    ok = __shfl_sync(kFullMask, ok, 0);
  } else if (warp == 1) {
    // ---- MMA issue: all lanes run the code, one elected lane predicates the instructions ----
    pdl_wait();                          // (the bounds of the waits below count from here, not through the kernels before)
    constexpr uint32_t idesc = instr_desc(kTile, Sh::kCols, false);
    const uint32_t elected = lane == 0 ? 1u : 0u;
    int s = 0, round = 0;
    uint32_t parity = 0;
    for (int tile = first; tile < p.tiles && ok; tile += stride, ++round) {
      const int acc = round & 1;
      if (round >= 2 && !mbar_wait_bounded(read0 + acc * 8, ((round >> 1) - 1) & 1)) { ok = false; break; }
      tc_fence_after();
      for (int k = 0; k < steps; ++k) {
        if (!mbar_wait_bounded(full0 + s * 8, parity)) { ok = false; break; }
        tc_fence_after();
        const uint64_t wd = smem_desc(ring + s * Sh::kStageBytes, 16, 1024);
        const uint64_t xd = smem_desc(ring + s * Sh::kStageBytes + kWBytes, 16, 1024);
#pragma unroll
        for (int i = 0; i < kDeep / 16; ++i) mma_ss(tmem + acc * Sh::kCols, wd + i * 2, xd + i * 2, idesc, (k > 0 || i > 0) ? 1u : 0u, elected);
        tc_commit(empty0 + s * 8, elected);
        if (++s == kStages) { s = 0; parity ^= 1; }
      }
      if (ok) tc_commit(done0 + acc * 8, elected);
    }
  } else {
    // ---- output: a thread owns row r of the tile ----
    pdl_wait();
    if constexpr (ROPE) pair = pair_at((int)threadIdx.x - 64);
    const int q4 = warp & 3, r = q4 * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(q4 * 32) << 16;
    const int rows = (int)a.rows;
    int round = 0;
    for (int tile = first; tile < p.tiles; tile += stride, ++round) {
      const int acc = round & 1;
      ok = mbar_wait_bounded(done0 + acc * 8, (round >> 1) & 1);
      if (GATED && S == 1) ok = output_warps_agree(ok);
      if (!ok) break;
      tc_fence_after();
      if constexpr (S == 1) {
        const int grp = tile / p.group_tiles, n = tile % p.group_tiles * kOuts + (GATED ? r & 63 : r);
#pragma unroll
        for (int c = 0; c < NP; c += 16) {
          if (c >= rows) break;
          uint32_t v[16];
          tmem_ld16(tmem + acc * Sh::kCols + lane_addr + c, v);
          tc_wait_ld();
          if constexpr (GATED) {
#pragma unroll
            for (int h = 0; h < 16; h += kSwap) {
              if (c + h >= NP || c + h >= rows) break;
              if (r >= 64)
#pragma unroll
                for (int i = 0; i < kSwap; ++i) swap[i * 64 + r - 64] = __uint_as_float(v[h + i]);
              output_warps_meet();
              if (r < 64 && n < a.N)
#pragma unroll
                for (int i = 0; i < kSwap; ++i)
                  if (c + h + i < rows) store_out(a, grp, c + h + i, n, gated_activation(__uint_as_float(v[h + i]), swap[i * 64 + r], GATE == 2 ? p.limit : 0.f, p.alpha));
              output_warps_meet();
            }
          } else if (n < a.N) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c + i < rows) store_out(a, grp, c + i, n, lin_act(__uint_as_float(v[i]), a.act));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(read0 + acc * 8);
      }
    }
  }
  if constexpr (S > 1) {
    // ---- one tile per cluster: every CTA has its part of the sums; CTA o adds up outputs o * kOuts / S onwards ----
    constexpr int kSlice = kTile / S;                     // rows of w of a CTA
    __syncwarp();
    if constexpr (Sh::kInRing) cluster_arrive();
    cluster_wait();                                       // the others' shared memory may be written: they have started, or are done with the ring
    if (warp >= 2 && ok) {
      const int q4 = warp & 3, r = q4 * 32 + lane, rows = (int)a.rows;
      const int j = GATED ? r & 63 : r;
      // [token][rank][row of the slice]: a warp's stores of one token are neighbours (16-byte stores of four tokens each, which are
      // not, were slower)
      const uint32_t at = cluster_addr(smem_u32(parts) + ((rank * kSlice + (GATED ? r / 64 * kOwn : 0) + j % kOwn) << 2), (uint32_t)(j / kOwn));
#pragma unroll
      for (int c = 0; c < NP; c += 16) {
        if (c >= rows) break;
        uint32_t v[16];
        tmem_ld16(tmem + ((uint32_t)(q4 * 32) << 16) + c, v);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (c + i < NP && c + i < rows) st_cluster(at + (uint32_t)(c + i) * kTile * 4, v[i]);
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if constexpr (ROPE) {
      const l3ci_linear_rope& rp = p.rope;
      const int q_cols = rp.Hq * rp.D, k_cols = rp.Hkv * rp.D;
      for (int e = (int)threadIdx.x - 64; e >= 0 && e < (int)a.rows * (kOwn / 2); e += 128, pair = pair_at(e)) {
        if (pair.pos < 0) continue;                       // (a position outside the table or the cache is skipped, not written)
        float x = 0.f, y = 0.f;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          x += parts[pair.t * kTile + s * kSlice + pair.j];
          y += parts[pair.t * kTile + s * kSlice + pair.j + 1];
        }
        x = __bfloat162float(__float2bfloat16_rn(x));     // (the projections are bf16 where they are two calls)
        y = __bfloat162float(__float2bfloat16_rn(y));
        const long long row = (long long)(pair.t / rp.T) * rp.cache_sb + pair.pos * rp.cache_st;
        __nv_bfloat16* to = pair.n < q_cols ? static_cast<__nv_bfloat16*>(a.out) + pair.t * a.out_st + pair.n
                            : pair.n < q_cols + k_cols ? static_cast<__nv_bfloat16*>(rp.cache_k) + row + pair.n - q_cols
                                                       : static_cast<__nv_bfloat16*>(rp.cache_v) + row + pair.n - q_cols - k_cols;
        const float c = pair.turn.x, sn = pair.turn.y;
        const bool turns = pair.n < q_cols + k_cols;      // (a value is copied: an infinite neighbour must not reach it)
        *reinterpret_cast<__nv_bfloat162*>(to) = __floats2bfloat162_rn(turns ? __fmaf_rn(x, c, -__fmul_rn(y, sn)) : x,
                                                                       turns ? __fmaf_rn(x, sn, __fmul_rn(y, c)) : y);
      }
    }
    for (int e = threadIdx.x; !ROPE && e < (int)a.rows * kOwn; e += kThreads) {
      const int t = e / kOwn, j = e % kOwn, n = first % p.group_tiles * kOuts + rank * kOwn + j;
      if (n >= a.N) continue;
      float y = 0.f, u = 0.f;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        y += parts[t * kTile + s * kSlice + j];
        if (GATED) u += parts[t * kTile + s * kSlice + kOwn + j];
      }
      store_out(a, first / p.group_tiles, t, n, GATED ? gated_activation(y, u, GATE == 2 ? p.limit : 0.f, p.alpha) : lin_act(y, a.act));
    }
  }
  if (!ok && lane == 0) atomicExch(a.status ? a.status : &g_wait_status, (int)L3CI_ERR_DEVICE_WAIT);
  __syncwarp();
  tc_fence_before();
  // a wait ran out: the copies still under way land before the shared memory is given back (or their own waits run out too)
  if (__syncthreads_or(!ok))
    for (int f = asked > kStages ? asked - kStages : 0; f < asked; ++f) (void)mbar_wait_bounded_one(full0 + f % kStages * 8, (uint32_t)(f / kStages) & 1u);
  if (warp == 1) tmem_dealloc(tmem, Sh::kTmem);
}

template <int NP, int S, int GATE, bool ROPE = false>
int launch(const l3ci_linear_args* a, float limit, float alpha, cudaStream_t stream, const l3ci_linear_rope* rope = nullptr) {
  using Sh = LinShape<NP>;
  constexpr bool GATED = GATE > 0;
  constexpr int kOuts = GATED ? kTile / 2 : kTile;
  LinParams p = {};
  p.a = *a;
  p.limit = limit;
  p.alpha = alpha;
  if (rope) p.rope = *rope;
  p.group_tiles = (a->N + kOuts - 1) / kOuts;
  p.tiles = p.group_tiles * a->groups;
  p.steps = (a->K + kDeep - 1) / kDeep;
  const long long one = (long long)a->N * a->K;
  CUtensorMap xmap, wmap;
  if (int st = make_rows_map(&xmap, a->x, a->K, (int)a->rows, 1, a->groups, a->x_st, 0, a->x_sg, NP)) return st;
  if (int st = make_rows_map(&wmap, a->w, a->K, a->N, GATED ? 2 : 1, a->groups, a->K, one, one * (GATED ? 2 : 1), kOuts)) return st;
  auto kernel = linear_rows_kernel<NP, S, GATE, ROPE>;
  static bool configured[64] = {false};
  int dev = 0;
  L3CI_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    L3CI_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::kSmem));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const int sms = sm_count() > 0 ? sm_count() : 148;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(S > 1 ? p.tiles * S : p.tiles < 2 * sms ? p.tiles : 2 * sms));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Sh::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (S > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = S;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (programmatic_launch_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, xmap, wmap, p);
  if (e != cudaSuccess) return fail(L3CI_ERR_CUDA, "launch of linear_rows_kernel failed: %s", cudaGetErrorString(e));
  return L3CI_OK;
}

template <int NP, int GATE>
int launch_split(const l3ci_linear_args* a, float limit, float alpha, cudaStream_t stream) {
  constexpr bool GATED = GATE > 0;
  const long long tiles = (a->N + (GATED ? kTile / 2 : kTile) - 1) / (GATED ? kTile / 2 : kTile) * (long long)a->groups;
  int split = a->split;
  if (split == 0) {
    // the most CTAs that still run at once, two per SM, each with two stages or more (one row, 2048 x 2048: 10.3, 5.9, 4.3, 3.6 us by
    // 1, 2, 4, 8; gated 2 x 8192 x 2048: 13.1, 13.0, 14.8, 20.5; one CTA per SM instead cost a step of the 1B model 40 us)
    const int sms = sm_count() > 0 ? sm_count() : 148, steps = (a->K + kDeep - 1) / kDeep;
    split = 1;
    while (split < 8 && tiles * split * 2 <= 2 * sms && steps >= 4 * split) split *= 2;
  }
  while (split > 1 && split > (a->K + kDeep - 1) / kDeep) split /= 2;   // every CTA has a stage
  switch (split) {
    case 1: return launch<NP, 1, GATE>(a, limit, alpha, stream);
    case 2: return launch<NP, 2, GATE>(a, limit, alpha, stream);
    case 4: return launch<NP, 4, GATE>(a, limit, alpha, stream);
    case 8: return launch<NP, 8, GATE>(a, limit, alpha, stream);
    default: return fail(L3CI_ERR_INVALID, "linear: split %d is not 1, 2, 4 or 8", split);
  }
}

}  // namespace
}  // namespace l3ci

extern "C" int64_t l3ci_row_stride(const int64_t* sizes, const int64_t* strides, int32_t dims) {
  if (dims < 1) return -1;
  const int64_t width = sizes[dims - 1];
  if (strides[dims - 1] != 1 && width > 1) return -1;
  int64_t stride = -1, reach = 0;          // of the axes seen so far: none yet
  for (int d = dims - 2; d >= 0; --d) {
    if (sizes[d] == 1) continue;
    if (stride < 0) {
      stride = strides[d];
      if (stride < width) return -1;       // a broadcast axis among them
    } else if (strides[d] != reach) {
      return -1;
    }
    reach = strides[d] * sizes[d];
  }
  return stride < 0 ? width : stride;
}

extern "C" int l3ci_linear_poll(l3ci_stream_t stream_) {
  using namespace l3ci;
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  void* own = nullptr;
  L3CI_CUDA_TRY(cudaGetSymbolAddress(&own, g_wait_status));
  int* words[2] = {static_cast<int*>(own), linear_many_wait_status()};
  int status[2] = {0, 0};
  for (int i = 0; i < 2; ++i)
    if (words[i]) L3CI_CUDA_TRY(cudaMemcpyAsync(&status[i], words[i], sizeof(int), cudaMemcpyDeviceToHost, stream));
  L3CI_CUDA_TRY(cudaStreamSynchronize(stream));
  if (status[0] == 0 && status[1] == 0) return L3CI_OK;
  for (int i = 0; i < 2; ++i)
    if (words[i]) L3CI_CUDA_TRY(cudaMemsetAsync(words[i], 0, sizeof(int), stream));
  L3CI_CUDA_TRY(cudaStreamSynchronize(stream));
  return fail(status[0] ? status[0] : status[1], "linear: a bounded wait ran out in an earlier launch");
}

extern "C" int l3ci_linear_gated(const l3ci_linear_args* a, float limit, float alpha) {
  using namespace l3ci;
  clear_error();
  if (a && limit != 0.f && (a->act != L3CI_ACT_SILU_GATE || !(limit > 0.f))) return fail(L3CI_ERR_INVALID, "linear: a limit of %g with activation %d", limit, a->act);
  if (!a) return fail(L3CI_ERR_INVALID, "linear: null arguments");
  if (a->rows < 0 || a->K <= 0 || a->N < 0 || a->act < L3CI_ACT_NONE || a->act > L3CI_ACT_SILU_GATE || a->split < 0 || a->split > 8 || a->groups < 0)
    return fail(L3CI_ERR_INVALID, "linear: rows=%lld K=%d N=%d groups=%d act=%d split=%d", (long long)a->rows, a->K, a->N, a->groups, a->act, a->split);
  if (a->rows == 0 || a->N == 0 || a->groups == 0) return L3CI_OK;
  if (a->rows > L3CI_LINEAR_MAX_ROWS) return fail(L3CI_ERR_UNSUPPORTED, "linear: %lld rows, at most %d", (long long)a->rows, L3CI_LINEAR_MAX_ROWS);
  if (!a->x || !a->w || !a->out) return fail(L3CI_ERR_INVALID, "linear: null pointer");
  if ((long long)a->groups * (a->N / (kTile / 2) + 1) > INT32_MAX / 16) return fail(L3CI_ERR_INVALID, "linear: %d groups of %d rows of w", a->groups, a->N);
  if (a->K % 8 || a->x_st % 8 || a->x_sg % 8 || !aligned16(a->x) || !aligned16(a->w))
    return fail(L3CI_ERR_ALIGNMENT, "linear: rows of x and w must be whole 16-byte vectors");
  if (a->rows > 1 && a->out_st < a->N && (a->groups == 1 || a->out_sg < a->N)) return fail(L3CI_ERR_INVALID, "linear: rows of the result overlap");
  if ((a->rows > 1 && a->x_st <= 0) || (a->groups > 1 && (a->x_sg <= 0 || a->out_sg <= 0)))
    return fail(L3CI_ERR_INVALID, "linear: rows or groups without a stride of their own");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(a->stream);
  const bool gated = a->act == L3CI_ACT_SILU_GATE;
  auto go = [&](auto np) {
    constexpr int NP = decltype(np)::value;
    return !gated ? launch_split<NP, 0>(a, limit, alpha, s) : limit > 0.f ? launch_split<NP, 2>(a, limit, alpha, s) : launch_split<NP, 1>(a, limit, alpha, s);
  };
  if (a->rows <= 8) return go(std::integral_constant<int, 8>{});
  if (a->rows <= 16) return go(std::integral_constant<int, 16>{});
  if (a->rows <= 32) return go(std::integral_constant<int, 32>{});
  return go(std::integral_constant<int, 64>{});
}

extern "C" int l3ci_linear(const l3ci_linear_args* a) { return l3ci_linear_gated(a, 0.f, 0.f); }

extern "C" int l3ci_linear_rot_embed_kv_cache(const l3ci_linear_args* a, const l3ci_linear_rope* rope) {
  using namespace l3ci;
  clear_error();
  if (!a || !rope) return fail(L3CI_ERR_INVALID, "linear_rot_embed_kv_cache: null arguments");
  if (a->rows < 0 || a->K <= 0 || a->N <= 0 || a->act != L3CI_ACT_NONE || a->groups != 1 || a->out_f32 || rope->T <= 0 || rope->Hq <= 0 || rope->Hkv <= 0 || rope->D <= 0 ||
      a->rows % rope->T || a->N != (rope->Hq + 2 * rope->Hkv) * rope->D || rope->freq_rows < 0 || rope->cache_len < 0)
    return fail(L3CI_ERR_INVALID, "linear_rot_embed_kv_cache: rows=%lld K=%d N=%d T=%d heads %d, %d of %d", (long long)a->rows, a->K, a->N, rope->T, rope->Hq, rope->Hkv, rope->D);
  if (a->rows == 0) return L3CI_OK;
  if (!a->x || !a->w || !a->out || !rope->freq_table || !rope->positions || !rope->cache_k || !rope->cache_v)
    return fail(L3CI_ERR_INVALID, "linear_rot_embed_kv_cache: null pointer");
  if (a->K % 8 || a->x_st % 8 || !aligned16(a->x) || !aligned16(a->w)) return fail(L3CI_ERR_ALIGNMENT, "linear: rows of x and w must be whole 16-byte vectors");
  auto on4 = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 3) == 0; };
  if (rope->D % 2 || !on4(a->out) || a->out_st % 2 || !on4(rope->cache_k) || !on4(rope->cache_v) || rope->cache_sb % 2 || rope->cache_st % 2 || !on4(rope->positions) ||
      (reinterpret_cast<uintptr_t>(rope->freq_table) & 7))
    return fail(L3CI_ERR_ALIGNMENT, "linear_rot_embed_kv_cache: pairs must start on 4 bytes, the table on 8");
  if (a->rows > 1 && (a->x_st <= 0 || a->out_st < rope->Hq * rope->D)) return fail(L3CI_ERR_INVALID, "linear_rot_embed_kv_cache: rows without a stride of their own");
  // clusters of 8 or 4 CTAs a tile, up to 32 rows (16 threads a row in the last step): a decode step's projections; others are two calls
  const int sms = sm_count() > 0 ? sm_count() : 148, steps = (a->K + kDeep - 1) / kDeep;
  const long long tiles = (a->N + kTile - 1) / kTile;
  const int split = tiles * 8 <= 2 * sms && steps >= 16 ? 8 : tiles * 4 <= 2 * sms && steps >= 8 ? 4 : 0;
  if (split == 0 || a->rows > 32) return fail(L3CI_ERR_UNSUPPORTED, "linear_rot_embed_kv_cache: %lld rows, K=%d, N=%d", (long long)a->rows, a->K, a->N);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(a->stream);
  auto go = [&](auto np) {
    constexpr int NP = decltype(np)::value;
    return split == 8 ? launch<NP, 8, 0, true>(a, 0.f, 0.f, s, rope) : launch<NP, 4, 0, true>(a, 0.f, 0.f, s, rope);
  };
  return a->rows <= 8 ? go(std::integral_constant<int, 8>{}) : a->rows <= 16 ? go(std::integral_constant<int, 16>{}) : go(std::integral_constant<int, 32>{});
}
