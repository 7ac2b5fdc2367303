// out[rows, N] = act(x[rows, K] w[N, K]^T) of many rows (prompts) with the activation on the fp32 sums (include/l3ci_b200.h,
// l3ci_linear_many): bf16 operands, gelu, tanh, or silu(gate) * up of a stacked matrix (or the same with silu_mul's roundings).
//
// The library's product writes twice the outputs of a gated product (268 MB a layer for 8192 tokens of the 1B model), and a pass of
// its own reads them again.  Here the activation is done on the way out, under the next tile's product.
//   * two SMs share a tile of 256 x 256 (cta_group::2): each brings 128 rows of x and 128 rows of w per 64 columns, and reads half of
//     the operand bytes that two tiles of 128 x 256 would; of a gated product one brings the gate rows and the other the up rows of the
//     same 128 outputs, so that each finds both in its own accumulator;
//   * a persistent pair walks its tiles; two accumulators of 256 columns fill the tensor memory, and sixteen warps per SM work on one while
//     the other fills;
//   * outputs leave through shared memory, as 64-byte pieces of rows.
// In turn with the library's product and the pass for its activation, us (the library's product alone): gated 2 x 8192 x 2048, 8192 rows 495 and
// 413 (411), 6001 rows 362 and 304 (303); gelu 8192 x 2048, 8192 rows 301 and 226 (198), 6001 rows 218 and 175 (146): 1.15 to 1.39 PFLOP/s under the
// power limit, which the activation's own instructions share with the tensor cores (by erff and the IEEE division 250 and 191 at gelu).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "bf16x8.cuh"
#include "host_common.h"
#include "linear_many.h"
#include "mixer_types.cuh"
#include "ptx_sm100.cuh"
#include "tcgen05.cuh"
#include "tensor_map.h"

namespace l3ci {
namespace {

constexpr int kHalf = 128;                 // rows of x, and of w, of one SM
constexpr int kDeep = 64;                  // columns per stage: 128 bytes
constexpr int kBox = kHalf * 128;          // bytes
constexpr int kStages = 5;
constexpr int kCols = 256;                 // of an accumulator
constexpr int kOutWarps = 16;              // four groups of four: an activation's instructions need that many to hide their latency
constexpr int kPieceCols = 32;             // columns that a group takes at a time
constexpr int kPieceBytes = kHalf * kPieceCols * 2;
constexpr int kThreads = 32 * (4 + kOutWarps);   // producer, MMA issue, allocation, none; outputs
constexpr size_t kSmem = 1024 + (size_t)kStages * 2 * kBox + kOutWarps / 4 * kPieceBytes;

__device__ int g_wait_status = 0;

struct ManyParams {
  long long m_tiles, tiles;
  int steps, N, rows;
  __nv_bfloat16* out;
  long long out_st;
};

typedef unsigned long long f2;             // two floats

__device__ __forceinline__ f2 f2_same(float v) { return f2_packf(v, v); }
__device__ __forceinline__ float rcp(float x) { return __fdividef(1.f, x); }

// x times the normal distribution's integral, two at a time: max(x, 0) - |x| erfc(|x| / sqrt 2) / 2 by the Chebyshev fit to erfc of Press et
// al., "Numerical Recipes", section 6.2 (erfcc; fractional error below 1.2e-7 everywhere).  No branch, a third of the instructions of 0.5 x (1 +
// erff(x / sqrt 2)), and no cancellation for negative x, where that form loses 4e-4 of the value at -4 and all of it below -5.6; of every
// finite bf16 x with a normal result the rounded result is the nearest bf16.
__device__ __forceinline__ void gelu(float& x, float& y) {
  constexpr float kLog2e = 1.4426950408889634f, kRoot = 0.70710678118654752f;
  const f2 m = f2_packf(fminf(fabsf(x), 30.f), fminf(fabsf(y), 30.f));        // (erfc is 0 from 15 on; an infinity keeps its sign)
  float u, v;
  f2_unpack(f2_fma(m, f2_same(0.5f * kRoot), f2_same(1.f)), u, v);
  const f2 t = f2_packf(rcp(u), rcp(v));
  f2 e = f2_fma(t, f2_same(0.17087277f * kLog2e), f2_same(-0.82215223f * kLog2e));
  e = f2_fma(t, e, f2_same(1.48851587f * kLog2e));
  e = f2_fma(t, e, f2_same(-1.13520398f * kLog2e));
  e = f2_fma(t, e, f2_same(0.27886807f * kLog2e));
  e = f2_fma(t, e, f2_same(-0.18628806f * kLog2e));
  e = f2_fma(t, e, f2_same(0.09678418f * kLog2e));
  e = f2_fma(t, e, f2_same(0.37409196f * kLog2e));
  e = f2_fma(t, e, f2_same(1.00002368f * kLog2e));
  e = f2_fma(t, e, f2_same(-1.26551223f * kLog2e));
  f2_unpack(f2_fma(f2_mul(m, f2_same(-0.5f * kLog2e)), m, e), u, v);
  const f2 over = f2_mul(f2_packf(x, y), f2_packf(x < 0.f ? 0.f : 1.f, y < 0.f ? 0.f : 1.f));   // max(x, 0); NaN for -infinity, as 0.5 x (1 + erff) gives
  f2_unpack(f2_fma(f2_mul(m, f2_same(-0.5f)), f2_mul(t, f2_packf(fast_exp2(u), fast_exp2(v))), over), x, y);
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t first_cta(uint32_t addr) {   // what lies there in the pair's first CTA
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(0));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// A copy into this CTA's memory that is counted on a barrier of the pair's first CTA.
__device__ __forceinline__ void pair_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(0) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u), "r"(elected) : "memory");
}
// Arrives on the barrier of both CTAs once every MMA issued so far has completed.
__device__ __forceinline__ void pair_commit(uint32_t bar, uint32_t elected) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
               "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t}\n"
               ::"r"(bar), "r"(elected), "h"((uint16_t)3) : "memory");
}

// A pair of gate and up sums as a bf16 product has them, and silu's own rounding: l3ci_silu_mul's bits, by its short form of silu, whose error grows
// with |z| but which rounds to the same bf16 for all the gates there are (rms_norm.cu).  The gate of unrounded sums is by expf and the full
// division: of z between -85 and 0 the short form rounds some to another bf16 (2 x 8192 x 2048, 6001 rows: 276 us, by the short form 271).
__device__ __forceinline__ float bf16_of(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float silu_mul(float z, float u) {
  z = bf16_of(z);
  return bf16_of(__fdividef(z * 0.0625f, fmaf(__expf(-z), 0.0625f, 0.0625f))) * bf16_of(u);
}

template <int ACT>
__global__ void __launch_bounds__(kThreads, 1)
linear_many_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ ManyParams p) {
  constexpr bool GATED = ACT == L3CI_ACT_SILU_GATE || ACT == L3CI_ACT_SILU_MUL;
  constexpr int kOuts = GATED ? kHalf : 2 * kHalf;       // output columns of a tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_box = smem + kStages * 2 * kBox;
  __shared__ __align__(8) uint64_t bars[2 * kStages + 4];
  __shared__ uint32_t tmem_slot;
  const uint32_t ring = smem_u32(smem), full0 = smem_u32(bars), empty0 = full0 + kStages * 8, done0 = empty0 + kStages * 8, read0 = done0 + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const long long pair = blockIdx.x / 2, pairs = gridDim.x / 2;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full0 + i * 8, 1);
      mbar_init(empty0 + i * 8, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(done0 + i * 8, 1);
      mbar_init(read0 + i * 8, 2 * kOutWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(2 * kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_meet();                          // the other CTA's barriers stand, and its tensor memory is there
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_launch_dependents();
  pdl_wait();
  bool ok = true;
  int asked = 0;

  if (warp == 0) {
    // ---- producer: this CTA's halves ----
    if (lane == 0) {
      int s = 0;
      uint32_t parity = 1;
      for (long long tile = pair; tile < p.tiles && ok; tile += pairs) {
        const int row = (int)(tile % p.m_tiles) * 2 * kHalf + (int)rank * kHalf;
        const int col = (int)(tile / p.m_tiles) * kOuts + (GATED ? 0 : (int)rank * kHalf);
        for (int k = 0; k < p.steps; ++k) {
          if (!mbar_wait_bounded_one(empty0 + s * 8, parity)) { ok = false; break; }
          const uint32_t dst = ring + s * 2 * kBox, bar = first_cta(full0 + s * 8);
          ++asked;
          if (rank == 0) mbar_expect_tx(full0 + s * 8, 4 * kBox);
          pair_load(dst, &xmap, bar, k * kDeep, row, 0);
          pair_load(dst + kBox, &wmap, bar, k * kDeep, col, GATED ? (int)rank : 0);
          if (++s == kStages) { s = 0; parity ^= 1; }
        }
      }
      // (the stages' last arrivals come from the pair's products: this CTA must not leave ahead of them)
      for (int i = 0; i < kStages && i < asked && ok; ++i) {
        if (asked < kStages && i == 0) { s = 0; parity = 0; }
        ok = mbar_wait_bounded_one(empty0 + s * 8, parity);
        if (++s == kStages) { s = 0; parity ^= 1; }
      }
    }
    ok = __shfl_sync(kFullMask, ok, 0);
  } else if (warp == 1 && rank == 0) {
    // ---- MMA issue, for both: all lanes run the code, one elected lane predicates the instructions ----
    constexpr uint32_t idesc = instr_desc(2 * kHalf, kCols, false);
    const uint32_t elected = lane == 0 ? 1u : 0u;
    int s = 0, round = 0;
    uint32_t parity = 0;
    for (long long tile = pair; tile < p.tiles && ok; tile += pairs, ++round) {
      const int acc = round & 1;
      if (round >= 2 && !mbar_wait_bounded(read0 + acc * 8, ((round >> 1) - 1) & 1)) { ok = false; break; }
      tc_fence_after();
      for (int k = 0; k < p.steps; ++k) {
        if (!mbar_wait_bounded(full0 + s * 8, parity)) { ok = false; break; }
        tc_fence_after();
        const uint64_t xd = smem_desc(ring + s * 2 * kBox, 16, 1024), wd = smem_desc(ring + s * 2 * kBox + kBox, 16, 1024);
#pragma unroll
        for (int i = 0; i < kDeep / 16; ++i) pair_mma(tmem + acc * kCols, xd + i * 2, wd + i * 2, idesc, (k > 0 || i > 0) ? 1u : 0u, elected);
        pair_commit(empty0 + s * 8, elected);
        if (++s == kStages) { s = 0; parity ^= 1; }
      }
      if (ok) pair_commit(done0 + acc * 8, elected);
    }
  } else if (warp >= 4) {
    // ---- outputs: a thread owns a row; each group of four warps takes a quarter of the columns, 32 at a time through its box ----
    const int q4 = warp & 3, part = (warp - 4) >> 2, r = q4 * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(q4 * 32) << 16;
    uint8_t* box = out_box + part * kPieceBytes;
    constexpr int kShare = kOuts / (kOutWarps / 4);
    auto meet = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory"); };
    int round = 0;
    for (long long tile = pair; tile < p.tiles && ok; tile += pairs, ++round) {
      const int acc = round & 1;
      const int row = (int)(tile % p.m_tiles) * 2 * kHalf + (int)rank * kHalf, col = (int)(tile / p.m_tiles) * kOuts;
      ok = mbar_wait_bounded(done0 + acc * 8, (round >> 1) & 1);
      {   // (the four warps go on together or not at all)
        uint32_t all;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n" : "=r"(all) : "r"((uint32_t)ok), "r"(1 + part) : "memory");
        ok = all != 0;
      }
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int c0 = part * kShare; c0 < (part + 1) * kShare; c0 += kPieceCols) {
        meet();                                // the box has been read
        // (16 columns at a time, not unrolled: the activations of 64 did not fit the instruction cache)
#pragma unroll 1
        for (int c = 0; c < kPieceCols; c += 16) {
          uint32_t y[16], z[16];
          tmem_ld16(tmem + acc * kCols + lane_addr + c0 + c, y);
          if (GATED) tmem_ld16(tmem + acc * kCols + lane_addr + kHalf + c0 + c, z);
          tc_wait_ld();
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            float f[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              f[i] = __uint_as_float(y[v * 8 + i]);
              if (ACT == L3CI_ACT_SILU_MUL) f[i] = silu_mul(f[i], __uint_as_float(z[v * 8 + i]));
              else if (GATED) f[i] = gated_activation(f[i], __uint_as_float(z[v * 8 + i]), 0.f, 0.f);
              else if (ACT == L3CI_ACT_TANH) f[i] = tanhf(f[i]);
            }
            if (ACT == L3CI_ACT_GELU)
#pragma unroll
              for (int i = 0; i < 8; i += 2) gelu(f[i], f[i + 1]);
            *reinterpret_cast<uint4*>(box + r * 64 + (((c / 8 + v) ^ (r >> 1 & 3)) << 4)) = pack8(f);
          }
        }
        if (c0 + kPieceCols == (part + 1) * kShare) {        // the accumulator has been read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) arrive_cluster(first_cta(read0 + acc * 8));
        }
        meet();
        // pieces of 64 bytes of rows, four lanes each
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int at = i * 128 + q4 * 32 + lane, y = at >> 2, c = at & 3;
          if (row + y < p.rows && col + c0 + c * 8 < p.N)
            *reinterpret_cast<uint4*>(p.out + (long long)(row + y) * p.out_st + col + c0 + c * 8) = *reinterpret_cast<const uint4*>(box + y * 64 + ((c ^ (y >> 1 & 3)) << 4));
        }
      }
    }
  }
  if (!ok && lane == 0) atomicExch(&g_wait_status, (int)L3CI_ERR_DEVICE_WAIT);
  __syncwarp();
  tc_fence_before();
  // a wait ran out: the copies still under way land before the shared memory is given back (or their own waits run out too)
  if (__syncthreads_or(!ok) && rank == 0)
    for (int f = asked > kStages ? asked - kStages : 0; f < asked; ++f) (void)mbar_wait_bounded_one(full0 + f % kStages * 8, (uint32_t)(f / kStages) & 1u);
  __syncwarp();
  cluster_meet();                          // neither CTA leaves, nor frees, while the other still counts on its memory
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kCols) : "memory");
}

template <int ACT>
int launch(const l3ci_linear_args* a) {
  constexpr bool GATED = ACT == L3CI_ACT_SILU_GATE || ACT == L3CI_ACT_SILU_MUL;
  ManyParams p = {};
  const int outs = GATED ? kHalf : 2 * kHalf;
  p.m_tiles = (a->rows + 2 * kHalf - 1) / (2 * kHalf);
  p.tiles = p.m_tiles * ((a->N + outs - 1) / outs);
  p.steps = (a->K + kDeep - 1) / kDeep;
  p.N = a->N;
  const long long one = (long long)a->N * a->K;
  CUtensorMap xmap, wmap;
  if (int st = make_rows_map(&xmap, a->x, a->K, (int)a->rows, 1, 1, a->x_st, 0, 0, kHalf)) return st;
  if (int st = make_rows_map(&wmap, a->w, a->K, a->N, GATED ? 2 : 1, 1, a->K, one, one * 2, kHalf)) return st;
  p.out = static_cast<__nv_bfloat16*>(a->out);
  p.out_st = a->rows > 1 ? a->out_st : a->N;
  p.rows = (int)a->rows;
  auto kernel = linear_many_kernel<ACT>;
  static bool configured[64] = {false};
  int dev = 0;
  L3CI_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    L3CI_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const int sms = sm_count() > 0 ? sm_count() : 148;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (p.tiles < sms / 2 ? p.tiles : sms / 2)));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = reinterpret_cast<cudaStream_t>(a->stream);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = programmatic_launch_enabled() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, xmap, wmap, p);
  if (e != cudaSuccess) return fail(L3CI_ERR_CUDA, "launch of linear_many_kernel failed: %s", cudaGetErrorString(e));
  return L3CI_OK;
}

}  // namespace

int* linear_many_wait_status() {
  void* at = nullptr;
  return cudaGetSymbolAddress(&at, g_wait_status) == cudaSuccess ? static_cast<int*>(at) : nullptr;
}

}  // namespace l3ci

extern "C" int l3ci_linear_many(const l3ci_linear_args* a) {
  using namespace l3ci;
  clear_error();
  if (!a) return fail(L3CI_ERR_INVALID, "linear_many: null arguments");
  if (a->rows < 0 || a->rows > INT32_MAX || a->K <= 0 || a->N < 0 || a->act < L3CI_ACT_NONE || a->act > L3CI_ACT_SILU_MUL || a->groups != 1 || a->out_f32)
    return fail(L3CI_ERR_INVALID, "linear_many: rows=%lld K=%d N=%d groups=%d act=%d", (long long)a->rows, a->K, a->N, a->groups, a->act);
  if (a->rows == 0 || a->N == 0) return L3CI_OK;
  if (!a->x || !a->w || !a->out) return fail(L3CI_ERR_INVALID, "linear_many: null pointer");
  if (a->K % 8 || a->N % 8 || a->x_st % 8 || a->out_st % 8 || !aligned16(a->x) || !aligned16(a->w) || !aligned16(a->out))
    return fail(L3CI_ERR_ALIGNMENT, "linear_many: rows must be whole 16-byte vectors");
  if (a->rows > 1 && (a->x_st <= 0 || a->out_st < a->N)) return fail(L3CI_ERR_INVALID, "linear_many: rows without a stride of their own");
  switch (a->act) {
    case L3CI_ACT_GELU: return launch<L3CI_ACT_GELU>(a);
    case L3CI_ACT_TANH: return launch<L3CI_ACT_TANH>(a);
    case L3CI_ACT_SILU_GATE: return launch<L3CI_ACT_SILU_GATE>(a);
    case L3CI_ACT_SILU_MUL: return launch<L3CI_ACT_SILU_MUL>(a);
    default: return launch<L3CI_ACT_NONE>(a);
  }
}
