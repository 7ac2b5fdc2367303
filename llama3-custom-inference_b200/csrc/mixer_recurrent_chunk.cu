// The linear recurrences of prompts by chunks of 16 tokens (include/l3ci_mixers.h, l3ci_recurrent_scan_chunks).
//
// Token by token every step of the state waits for the sums over it (850 cycles a token at 48 heads of 128 x 128, mixer_recurrent.cu).  Over a
// chunk whose first token finds the state S,
//   gated delta rule:  u_i = beta_i (v_i - (k_i G_i)^T S - sum_{j<i} L_ij u_j),   o_i = (q_i G_i)^T S + sum_{j<=i} M_ij u_j,
//                      S <- diag(G) S + sum_j (k_j G_{>j}) u_j^T,
// with G_i the product of the decays up to token i, L_ij and M_ij the products of k_i, q_i with k_j decayed from j to i.  With T the inverse of
// (1 + beta L) times beta, U = T (V - (k G) S), and all but the terms with S is known ahead, for all chunks at once.  Time mixing is the same with
// U = V, decays up to i - 1 and the bonus on the diagonal of M.  (The chunked delta rule: Yang et al., "Parallelizing Linear Transformers with the
// Delta Rule over Sequence Length".)
//   chunk_inputs_kernel  a warp per head and chunk, lanes over channels: the decayed keys of the chunk's tokens stay in registers and are
//     multiplied on from token to token, so that every decay is a product of factors at most 1 and none is divided by; L's and M's rows are the
//     lanes' sums, T's columns a lane's each.
//   chunk_scan_kernel    a warp per 8 columns of the state, in its registers: sixteen lanes share four columns, four neighbouring rows of every
//     64 a lane.  Per chunk the sums W S and Q S, four tokens at a time over the sixteen lanes; U and the outputs, a token's column by one lane;
//     the new state.  Chunks come through a ring of bulk copies.
// All in 32-bit multiply-adds, a sum over the tokens up to its own only.  Products on the tensor cores, of operands in two or three tf32
// parts, were as fast for the delta rule and a quarter faster for time mixing, but their accumulators are cut off, not rounded: states that
// decay within a few tokens were twice as far from 64 bits as token by token.  And 0 times a later token's NaN is NaN.
// States against 64 bits, of their norm, in 1e-8 (40 to 4000 tokens, 64 and 128 channels; in brackets token by token): delta rule without
// decay 14 to 36 (14 to 35), decays of about e^-0.0008 a token 17 to 39 (19 to 43), e^-0.08 9.6 to 10.2 (9.5 to 10.0), e^-0.8 4.8 to
// 5.4 (4.9 to 5.6), e^-8 3.4 to 4.5 (4.2 to 4.5); time mixing, decays of about e^-e^-5 a token 18 to 41 (18 to 41), e^-e^-3 12.4 to 13.3
// (12.1 to 12.9), e^-e^-1 5.6 to 6.2 (5.5 to 6.1), e^-e 3.0 to 3.2 (3.0 to 3.2).  Outputs: the same, but for their rounding to bf16.
// us, by chunks and token by token: delta rule, 1777 tokens of 3 x 16 heads of 128 x 128 445 and 740; time mixing, 3 x 32 heads of 64 x 64
// 298 and 370.  Bound by shared memory: of the scan's 6.8 thousand cycles a chunk (128 x 128) the rows of W, Q and K, which every warp reads,
// and the shuffles take 4 to 5.  Eight columns a lane instead of four and four warps instead of eight (half of those rows): 577 and 484 us, one
// warp a scheduler waits out its own instructions.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mixer_recurrent.h"
#include "ptx_sm100.cuh"
#include "tcgen05.cuh"

namespace l3ci {
namespace {

__device__ int g_wait_status = 0;   // of calls without a status word of their own

constexpr int kChunk = 16;
constexpr int kDelta = 0, kTimeMix = 1;
constexpr int kOwn = 4;                           // a lane's columns
constexpr int kCols = 2 * kOwn;                   // a warp's: sixteen lanes share kOwn of them
constexpr int kTogether = 16 / kOwn;              // tokens whose sums over the state are taken together: one for each of the lanes
constexpr int kPatch = kChunk + 4;                // floats of a column's tokens in a patch: neighbours on other banks
constexpr int kMaxWarps = 8;
constexpr int kMaxCols = kMaxWarps * kCols;       // of a CTA
constexpr int kVPitch = kMaxCols * 2 + 16;        // bytes of a token's values in a stage
constexpr int kStages = 4;

// A chunk's block of D channels, in floats: W = k G (delta rule) and Q = q G, K decayed to the chunk's end, 16 tokens each, M, T (delta
// rule), the chunk's decays.
template <int KIND, int D>
struct ChunkShape {
  static constexpr int kRows = kChunk * D, kSquare = kChunk * kChunk;
  static constexpr int kAtQ = KIND == kDelta ? kRows : 0, kAtK = kAtQ + kRows, kAtM = kAtK + kRows, kAtT = kAtM + kSquare,
                       kAtG = kAtT + (KIND == kDelta ? kSquare : 0);
  static constexpr int kFloats = kAtG + D;
  static constexpr int kStage = kFloats * 4 + kChunk * kVPitch;      // bytes in the scan: the block and the values
  static_assert(kFloats % 4 == 0, "bulk copies of whole 16-byte vectors");
};

struct ChunkParams {
  l3ci_recurrent_scan_args a;
  float* blocks;                 // [B * H][chunks]
  int t0, tokens, chunks;        // of this segment
  int col_blocks, warps, last;
};

// ---- the chunks' inputs -----------------------------------------------------------------------------------------------------------
constexpr int kInputWarps = 4;

template <typename Q, int KIND, int D>
__global__ void __launch_bounds__(32 * kInputWarps)
chunk_inputs_kernel(const __grid_constant__ ChunkParams p, long long units) {
  using Sh = ChunkShape<KIND, D>;
  constexpr int CH = D / 32, P2 = CH / 2;         // a lane's neighbouring channels; pairs of them
  typedef unsigned long long f2;
  pdl_begin();
  const l3ci_recurrent_scan_args& a = p.a;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long unit = (long long)blockIdx.x * kInputWarps + warp;
  if (unit >= units) return;
  const int c = (int)(unit % p.chunks), bh = (int)(unit / p.chunks), h = bh % a.H, b = bh / a.H, R = a.H / a.G;
  const int d0 = lane * CH, n = min(kChunk, p.tokens - c * kChunk);
  const long long row0 = (long long)b * a.T + p.t0 + c * kChunk;
  float* block = p.blocks + (long long)(bh * (long long)p.chunks + c) * Sh::kFloats;
  auto pair_of = [](float x, float y) { return f2_packf(x, y); };
  auto dot = [&](const f2 (&x)[P2], const f2 (&y)[P2]) {
    f2 s = f2_mul(x[0], y[0]);
#pragma unroll
    for (int j = 1; j < P2; ++j) s = f2_fma(x[j], y[j], s);
    float u, v;
    f2_unpack(s, u, v);
    return u + v;
  };
  f2 t[kChunk][P2], run[P2], rest[P2], gb[P2], bonus[P2];   // decayed keys; product of the decays so far, what its roundings left
  auto put = [&](float* row, int j, f2 v) { *reinterpret_cast<f2*>(row + d0 + 2 * j) = v; };
  float t_col[kChunk];                            // column lane % 16 of T
#pragma unroll
  for (int j = 0; j < kChunk; ++j) t_col[j] = 0.f;
#pragma unroll
  for (int j = 0; j < P2; ++j) {
    run[j] = pair_of(1.f, 1.f);
    rest[j] = gb[j] = bonus[j] = 0ull;
    if (KIND == kTimeMix) {
      gb[j] = pair_of(a.g_bias[h * D + d0 + 2 * j], a.g_bias[h * D + d0 + 2 * j + 1]);
      bonus[j] = pair_of(a.bonus[h * D + d0 + 2 * j], a.bonus[h * D + d0 + 2 * j + 1]);
    }
  }
#pragma unroll
  for (int i = 0; i < kChunk; ++i)
#pragma unroll
    for (int j = 0; j < P2; ++j) t[i][j] = 0ull;
  // the next token's rows are under way while one is worked on
  float fq[CH], fk[CH], fg[CH], beta_next = 0.f;
  auto fetch = [&](int i) {
    const long long row = row0 + (i < n ? i : 0);
    load_vec<Q, CH>(static_cast<const Q*>(a.q) + row * a.qk_st + (h / R) * a.qk_sh + d0, fq);
    load_vec<Q, CH>(static_cast<const Q*>(a.k) + row * a.qk_st + (h / R) * a.qk_sh + d0, fk);
    load_vec<Q, CH>(static_cast<const Q*>(a.g) + row * a.g_st + h * a.g_sh + d0, fg);
    if (KIND == kDelta) beta_next = i < n ? a.beta[row * a.H + h] : 0.f;
  };
  fetch(0);
#pragma unroll 1
  for (int i = 0; i < kChunk; ++i) {
    const bool real = i < n;
    f2 q[P2], k[P2], g[P2];
    const float beta = beta_next;
    {
#pragma unroll
      for (int j = 0; j < P2; ++j) {
        q[j] = real ? pair_of(fq[2 * j], fq[2 * j + 1]) : 0ull;
        k[j] = real ? pair_of(fk[2 * j], fk[2 * j + 1]) : 0ull;
        if (KIND == kTimeMix) {
          float x, y;
          f2_unpack(f2_add(pair_of(fg[2 * j], fg[2 * j + 1]), gb[j]), x, y);
          fg[2 * j] = expf(-expf(x));
          fg[2 * j + 1] = expf(-expf(y));
        }
        g[j] = real ? pair_of(fg[2 * j], fg[2 * j + 1]) : pair_of(1.f, 1.f);   // (a token behind the last one changes nothing)
      }
    }
    fetch(i + 1 < kChunk ? i + 1 : i);
    f2 qg[P2], kg[P2];
#pragma unroll
    for (int j = 0; j < P2; ++j) {
      if (KIND == kDelta) {
        run[j] = f2_mul(run[j], g[j]);
        qg[j] = f2_mul(q[j], run[j]);
        kg[j] = f2_mul(k[j], run[j]);
      } else {
        // (without the rest states of slow decays were 1.06 times as far from 64 bits as token by token; of the delta rule they are nearer anyway)
        qg[j] = f2_mul(q[j], f2_add(run[j], rest[j]));
        kg[j] = f2_mul(bonus[j], k[j]);
        const f2 product = f2_mul(run[j], g[j]);
        rest[j] = f2_fma(rest[j], g[j], f2_fma(run[j], g[j], product ^ 0x8000000080000000ull));
        run[j] = product;
      }
      put(block + Sh::kAtQ + i * D, j, qg[j]);
      if (KIND == kDelta) put(block + i * D, j, kg[j]);
    }
    float sums[32];
#pragma unroll
    for (int x0 = 0; x0 < kChunk; x0 += 4) {
      if (x0 > i) {                               // keys of later tokens
#pragma unroll
        for (int x = x0; x < x0 + 4; ++x) sums[x] = sums[kChunk + x] = 0.f;
        continue;
      }
#pragma unroll
      for (int x = x0; x < x0 + 4; ++x) {
        if (KIND == kDelta) {
#pragma unroll
          for (int j = 0; j < P2; ++j) t[x][j] = x == i ? k[j] : f2_mul(t[x][j], g[j]);
          sums[x] = dot(k, t[x]);
          sums[kChunk + x] = dot(q, t[x]);
        } else {
#pragma unroll
          for (int j = 0; j < P2; ++j) t[x][j] = x == i ? kg[j] : t[x][j];
          sums[x] = 0.f;
          sums[kChunk + x] = dot(q, t[x]);
#pragma unroll
          for (int j = 0; j < P2; ++j) t[x][j] = x == i ? k[j] : f2_mul(t[x][j], g[j]);
        }
      }
    }
    // lane x: L_ix; lane 16 + x: M_ix
#pragma unroll
    for (int m = 16; m >= 1; m /= 2) {
      const bool upper = lane & m;
#pragma unroll
      for (int x = 0; x < m; ++x) {
        const float send = upper ? sums[x] : sums[x + m], mine = upper ? sums[x + m] : sums[x];
        sums[x] = mine + __shfl_xor_sync(kFullMask, send, m);
      }
    }
    if (lane >= kChunk) block[Sh::kAtM + i * kChunk + lane - kChunk] = sums[0];   // (those of later tokens are not read)
    if (KIND == kDelta) {
      const float row_l = lane < i ? -sums[0] : 0.f;
      float col = lane % kChunk == i ? 1.f : 0.f;
#pragma unroll
      for (int j0 = 0; j0 < kChunk; j0 += 4) {
        if (j0 >= i) break;
#pragma unroll
        for (int j = j0; j < j0 + 4; ++j) col = fmaf(__shfl_sync(kFullMask, row_l, j), t_col[j], col);
      }
      col *= beta;
#pragma unroll
      for (int j = 0; j < kChunk; ++j) t_col[j] = j == i ? col : t_col[j];
      if (lane < kChunk) block[Sh::kAtT + i * kChunk + lane] = col;
    }
  }
#pragma unroll
  for (int i = 0; i < kChunk; ++i)
#pragma unroll
    for (int j = 0; j < P2; ++j) put(block + Sh::kAtK + i * D, j, t[i][j]);
#pragma unroll
  for (int j = 0; j < P2; ++j) put(block + Sh::kAtG, j, f2_add(run[j], rest[j]));
}

// ---- the scan ----------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

template <int KIND, int D>
__global__ void __launch_bounds__(32 * (kMaxWarps + 1), 1)
chunk_scan_kernel(const __grid_constant__ ChunkParams p) {
  using Sh = ChunkShape<KIND, D>;
  typedef unsigned long long f2;
  constexpr int kRuns = D / 64;                   // a lane's rows: 4 neighbours of every 64
  extern __shared__ __align__(128) uint8_t ring_smem[];
  __shared__ __align__(16) float patches[kMaxWarps][2][kCols * kPatch];      // of a warp, by column: V - W S, U
  __shared__ __align__(8) uint64_t bars[2 * kStages];
  const l3ci_recurrent_scan_args& a = p.a;
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + kStages * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vb = blockIdx.x % p.col_blocks, bh = blockIdx.x / p.col_blocks, h = bh % a.H, b = bh / a.H;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full0 + i * 8, 1);
      mbar_init(empty0 + i * 8, p.warps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  pdl_begin();
  const bool fresh = a.positions[b] == 0 && p.t0 == 0;
  bool ok = true;
  int asked = 0;
  const int col0 = vb * p.warps * kCols;
  if (warp == p.warps) {
    // ---- producer: a chunk's block, and a token's values by each of 16 lanes ----
    const float* block = p.blocks + (long long)bh * p.chunks * Sh::kFloats;
    const __nv_bfloat16* v = static_cast<const __nv_bfloat16*>(a.v) + ((long long)b * a.T + p.t0) * a.v_st + h * a.v_sh + col0;
    const uint32_t v_bytes = min(p.warps * kCols, a.V - col0) * 2;
    for (int i = 0, s = 0, parity = 1; i < p.chunks; ++i) {
      if (!mbar_wait_bounded(empty0 + s * 8, parity)) { ok = false; break; }
      const uint32_t dst = smem_u32(ring_smem + s * Sh::kStage), bar = full0 + s * 8;
      if (lane == 0) {
        ++asked;
        mbar_expect_tx(bar, Sh::kFloats * 4 + kChunk * v_bytes);
        bulk_load(dst, block + (long long)i * Sh::kFloats, Sh::kFloats * 4, bar);
      }
      __syncwarp();
      if (lane < kChunk)    // (a token behind the last one has no share in anything: the last one's values again)
        bulk_load(dst + Sh::kFloats * 4 + lane * kVPitch, v + (long long)min(i * kChunk + lane, p.tokens - 1) * a.v_st, v_bytes, bar);
      if (++s == kStages) { s = 0; parity ^= 1; }
    }
    __syncwarp();
    if (a.tail && p.last && vb == 0) move_tails<__nv_bfloat16>(a, b, h, lane, 32, a.positions[b] == 0);
  } else {
    // Sixteen lanes share kOwn columns of all rows.  A lane's column c is column c ^ me of them, and token x of those taken together token
    // x ^ mine, so that the lanes' sums are added up without choosing what to send: a lane ends with column `me` of token `mine`.
    const int r = lane & 15, group = lane >> 4, me = r % kOwn, mine = r / kOwn, col = group * kOwn + me;
    const int c0 = col0 + warp * kCols + group * kOwn;
    const bool real = c0 < a.V;                   // (of a group all columns are, or none)
    float* state = a.state + b * a.state_sb + (long long)h * D * a.V + c0;
    auto row_of = [&](int j) { return j / 2 * 64 + 4 * r + j % 2 * 2; };                        // first row of pair j
    f2 S[kOwn][2 * kRuns];
#pragma unroll
    for (int c = 0; c < kOwn; ++c)
#pragma unroll
      for (int j = 0; j < 2 * kRuns; ++j) {
        const float* at = state + (long long)row_of(j) * a.V + (c ^ me);
        S[c][j] = !fresh && real ? f2_packf(at[0], at[a.V]) : 0ull;
      }
    float *seen = patches[warp][0], *u = patches[warp][1];
    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + ((long long)b * a.T + p.t0) * a.out_st + h * a.out_sh + c0 + me;
    auto load4 = [](const float* x, f2 (&y)[2]) {
      const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(x);
      y[0] = z.x;
      y[1] = z.y;
    };
    for (int i = 0, s = 0, parity = 0; i < p.chunks; ++i) {
      if (!mbar_wait_bounded(full0 + s * 8, parity)) { ok = false; break; }
      const float* st = reinterpret_cast<const float*>(ring_smem + s * Sh::kStage);
      const uint8_t* values = ring_smem + s * Sh::kStage + Sh::kFloats * 4 + (warp * kCols + col) * 2;
      const int n = min(kChunk, p.tokens - i * kChunk);
      float v[kChunk / kTogether];
#pragma unroll
      for (int i2 = 0; i2 < kChunk / kTogether; ++i2)
        v[i2] = real ? to_f32(*reinterpret_cast<const __nv_bfloat16*>(values + (i2 * kTogether + mine) * kVPitch)) : 0.f;
      auto put = [&](float* of, int i2, float y) { of[col * kPatch + i2 * kTogether + mine] = y; };
      if (KIND == kTimeMix) {                     // (U = V)
#pragma unroll
        for (int i2 = 0; i2 < kChunk / kTogether; ++i2) put(u, i2, v[i2]);
        __syncwarp();
      }
      // ---- sums over the state: W S of the delta rule, Q S ----
      constexpr int kSums = KIND == kDelta ? 2 : 1;
      float sums[kChunk / kTogether][kSums];
#pragma unroll
      for (int i2 = 0; i2 < kChunk / kTogether; ++i2)
#pragma unroll
        for (int k = 0; k < kSums; ++k) {
          f2 part[kTogether][kOwn];
#pragma unroll
          for (int x = 0; x < kTogether; ++x)
#pragma unroll
            for (int j = 0; j < kRuns; ++j) {
              f2 y[2];
              load4(st + (k == kSums - 1 ? Sh::kAtQ : 0) + (i2 * kTogether + (x ^ mine)) * D + j * 64 + 4 * r, y);
#pragma unroll
              for (int c = 0; c < kOwn; ++c) {
                part[x][c] = j == 0 ? f2_mul(y[0], S[c][0]) : f2_fma(y[0], S[c][2 * j], part[x][c]);
                part[x][c] = f2_fma(y[1], S[c][2 * j + 1], part[x][c]);
              }
            }
          float sum[kTogether][kOwn];
#pragma unroll
          for (int x = 0; x < kTogether; ++x)
#pragma unroll
            for (int c = 0; c < kOwn; ++c) {
              float y, z;
              f2_unpack(part[x][c], y, z);
              sum[x][c] = y + z;
            }
#pragma unroll
          for (int m = kTogether / 2; m >= 1; m /= 2)
#pragma unroll
            for (int x = 0; x < m; ++x)
#pragma unroll
              for (int c = 0; c < kOwn; ++c) sum[x][c] += __shfl_xor_sync(kFullMask, sum[x + m][c], m * kOwn);
#pragma unroll
          for (int m = kOwn / 2; m >= 1; m /= 2)
#pragma unroll
            for (int c = 0; c < m; ++c) sum[0][c] += __shfl_xor_sync(kFullMask, sum[0][c + m], m);
          sums[i2][k] = sum[0][0];
        }
      // ---- U, and the outputs with it: this lane's column and tokens, sums over the tokens up to them only ----
      float x[kChunk];
      auto column = [&](const float* of) {
#pragma unroll
        for (int j = 0; j < kChunk; j += 4) {
          const float4 f = *reinterpret_cast<const float4*>(of + col * kPatch + j);
          x[j] = f.x; x[j + 1] = f.y; x[j + 2] = f.z; x[j + 3] = f.w;
        }
      };
      auto over_tokens = [&](const float* square, int i2, float sum) {            // of token i2 * kTogether + mine
        const float* row = square + (i2 * kTogether + mine) * kChunk;
#pragma unroll
        for (int j = 0; j < (i2 + 1) * kTogether; j += 4) {
          const float4 f = *reinterpret_cast<const float4*>(row + j);
          const float y[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (j + e - i2 * kTogether <= mine) sum = fmaf(y[e], x[j + e], sum);
        }
        return sum;
      };
      if (KIND == kDelta) {
#pragma unroll
        for (int i2 = 0; i2 < kChunk / kTogether; ++i2) put(seen, i2, v[i2] - sums[i2][0]);
        __syncwarp();
        column(seen);
#pragma unroll
        for (int i2 = 0; i2 < kChunk / kTogether; ++i2) put(u, i2, over_tokens(st + Sh::kAtT, i2, 0.f));
        __syncwarp();
      }
      column(u);
#pragma unroll
      for (int i2 = 0; i2 < kChunk / kTogether; ++i2) {
        const int t = i2 * kTogether + mine;
        const float o = over_tokens(st + Sh::kAtM, i2, sums[i2][kSums - 1]);
        if (t < n && real) out[(long long)(i * kChunk + t) * a.out_st] = __float2bfloat16_rn(o);
      }
      // ---- the state: decayed, and the chunk's keys times U ----
#pragma unroll
      for (int j = 0; j < kRuns; ++j) {
        f2 g[2];
        load4(st + Sh::kAtG + j * 64 + 4 * r, g);
#pragma unroll
        for (int c = 0; c < kOwn; ++c) {
          S[c][2 * j] = f2_mul(S[c][2 * j], g[0]);
          S[c][2 * j + 1] = f2_mul(S[c][2 * j + 1], g[1]);
        }
      }
      auto add = [&](int t, const float (&y)[kOwn]) {
        f2 k[kRuns][2];
#pragma unroll
        for (int j = 0; j < kRuns; ++j) load4(st + Sh::kAtK + t * D + j * 64 + 4 * r, k[j]);
#pragma unroll
        for (int c = 0; c < kOwn; ++c) {
          const f2 y2 = f2_packf(y[c], y[c]);
#pragma unroll
          for (int j = 0; j < 2 * kRuns; ++j) S[c][j] = f2_fma(k[j / 2][j % 2], y2, S[c][j]);
        }
      };
      const float* own_u = u + group * kOwn * kPatch;
      if (n == kChunk) {
#pragma unroll
        for (int t = 0; t < kChunk; t += 4) {
          float y[4][kOwn];
#pragma unroll
          for (int c = 0; c < kOwn; ++c) {
            const float4 f = *reinterpret_cast<const float4*>(own_u + (c ^ me) * kPatch + t);
            y[0][c] = f.x; y[1][c] = f.y; y[2][c] = f.z; y[3][c] = f.w;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) add(t + e, y[e]);
        }
      } else {                                    // (what stands behind the last token may be no number)
#pragma unroll 1
        for (int t = 0; t < n; ++t) {
          float y[kOwn];
#pragma unroll
          for (int c = 0; c < kOwn; ++c) y[c] = own_u[(c ^ me) * kPatch + t];
          add(t, y);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + s * 8);
      if (++s == kStages) { s = 0; parity ^= 1; }
    }
    if (ok && real)
#pragma unroll
      for (int c = 0; c < kOwn; ++c)
#pragma unroll
        for (int j = 0; j < 2 * kRuns; ++j) {
          float* at = state + (long long)row_of(j) * a.V + (c ^ me);
          f2_unpack(S[c][j], at[0], at[a.V]);
        }
  }
  if (!ok && lane == 0) atomicExch(a.status ? a.status : &g_wait_status, (int)L3CI_ERR_DEVICE_WAIT);
  // a wait ran out: the copies still under way land before the shared memory is given back
  if (__syncthreads_or(!ok))
    for (int f = asked > kStages ? asked - kStages : 0; f < asked; ++f) (void)mbar_wait_bounded_one(full0 + f % kStages * 8, (uint32_t)(f / kStages) & 1u);
}

// Scratch of a chunk of all heads.
size_t chunk_bytes(const l3ci_recurrent_scan_args* a) {
  const size_t floats = a->kind == kDelta ? (a->D == 64 ? ChunkShape<kDelta, 64>::kFloats : ChunkShape<kDelta, 128>::kFloats)
                                          : (a->D == 64 ? ChunkShape<kTimeMix, 64>::kFloats : ChunkShape<kTimeMix, 128>::kFloats);
  return (size_t)a->B * a->H * floats * 4;
}
constexpr size_t kMaxScratch = 256ull << 20;      // longer prompts go in segments

// Warps of a CTA of the scan, eight columns each: the fewest columns for the busiest SM (96 heads' blocks of 64 columns leave a third of the SMs
// idle; 48 heads of 128 x 128, 132 tokens of 32 heads: 6 and 4 warps 431 and 36.2 us, 8 warps 440 and 52.3).
int scan_warps(const l3ci_recurrent_scan_args* a) {
  const long long sms = sm_count() > 0 ? sm_count() : 148, heads = (long long)a->B * a->H;
  long long least = -1;
  int best = kMaxWarps;
  for (int w = kMaxWarps; w >= kMaxWarps / 2; --w) {
    const long long ctas = heads * ((a->V + w * kCols - 1) / (w * kCols)), load = (ctas + sms - 1) / sms * w;
    if (least < 0 || load < least) { least = load; best = w; }
  }
  return best;
}

template <typename Q, int KIND, int D>
int launch(const l3ci_recurrent_scan_args* a, void* scratch, size_t bytes) {
  using Sh = ChunkShape<KIND, D>;
  const size_t one = chunk_bytes(a);
  const int all = (a->T + kChunk - 1) / kChunk;
  const int most = (int)(bytes / one < (size_t)all ? bytes / one : (size_t)all);
  if (!scratch || most < 1 || !aligned16(scratch)) return fail(L3CI_ERR_SCRATCH, "recurrent_scan: %zu bytes of scratch needed at least, %zu given", one, bytes);
  const int segments = (all + most - 1) / most, per = (all + segments - 1) / segments;
  const int warps = scan_warps(a);
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(a->stream);
  auto inputs = chunk_inputs_kernel<Q, KIND, D>;
  auto scan = chunk_scan_kernel<KIND, D>;
  static bool configured[64] = {false};
  int dev = 0;
  L3CI_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    L3CI_CUDA_TRY(cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * Sh::kStage));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  for (int c = 0; c < all; c += per) {
    ChunkParams p = {};
    p.a = *a;
    p.warps = warps;
    p.col_blocks = (a->V + warps * kCols - 1) / (warps * kCols);
    p.t0 = c * kChunk;
    p.chunks = per < all - c ? per : all - c;
    p.tokens = a->T - p.t0 < p.chunks * kChunk ? a->T - p.t0 : p.chunks * kChunk;
    p.last = c + per >= all;
    const long long heads = (long long)a->B * a->H, units = heads * p.chunks;
    p.blocks = static_cast<float*>(scratch);
    L3CI_LAUNCH("chunk_inputs_kernel", inputs, dim3((unsigned)((units + kInputWarps - 1) / kInputWarps)), dim3(32 * kInputWarps), 0, stream, p, units);
    L3CI_LAUNCH("chunk_scan_kernel", scan, dim3((unsigned)(heads * p.col_blocks)), dim3(32 * (p.warps + 1)), (size_t)kStages * Sh::kStage, stream, p);
  }
  return L3CI_OK;
}

bool applies(const l3ci_recurrent_scan_args* a) {
  const int qs = a->kind == kDelta ? 4 : 2;       // bytes of an element of q, k, g
  auto rows = [&](const void* x, int64_t st, int64_t sh) { return reinterpret_cast<uintptr_t>(x) % (4 * qs) == 0 && st % 4 == 0 && sh % 4 == 0; };
  return a->dtype == L3CI_BF16 && (a->D == 64 || a->D == 128) && (long long)a->B * a->H * ((a->T + kChunk - 1) / kChunk) <= 0x3fffffffLL &&
         rows(a->q, a->qk_st, a->qk_sh) && rows(a->k, a->qk_st, a->qk_sh) && rows(a->g, a->g_st, a->g_sh) && aligned16(a->v) && a->V % 8 == 0 && a->v_st % 8 == 0 && a->v_sh % 8 == 0;
}

}  // namespace

int* scan_chunks_wait_status() {
  void* at = nullptr;
  return cudaGetSymbolAddress(&at, g_wait_status) == cudaSuccess ? static_cast<int*>(at) : nullptr;
}

size_t scan_chunks_scratch(const l3ci_recurrent_scan_args* a) {
  // From where on the chunks are the faster, in CTAs of 64 columns and tokens; us by tokens and by chunks, heads of 128 x 128 and of 64 x 64.
  //   delta rule   32 CTAs, 1000 tokens 187 and 171, 138 and 178;   64 CTAs, 132 tokens 46.3 and 37.4, 43.2 and 40.1;
  //                96, 56 tokens 30.3 and 30.2;   128, 56 tokens 30.8 and 32.4, 64 tokens 33.9 and 32.4;   320, 56 tokens 72.5 and 79.5
  //                64 x 64: 128 CTAs, 112 tokens 39.8 and 41.6, 128 tokens 44.7 and 43.9;   96, 128 tokens 44.7 and 40.0
  //   time mixing  64 CTAs, 300 tokens 68.1 and 70.4, 400 tokens 87.5 and 81.6, 64 x 64 2000 tokens 269 and 352;
  //                128 x 128: 96 CTAs, 64 tokens 27.0 and 25.5;   128, 64 tokens 27.5 and 27.5
  //                64 x 64: 96 CTAs, 200 tokens 47.0 and 47.4, 240 tokens 55.0 and 50.6;   448, 240 tokens 108 and 88.8
  const long long ctas = (long long)a->B * a->H * ((a->V + kMaxCols - 1) / kMaxCols);
  if (!applies(a) || ctas < 64) return 0;
  const bool some = ctas >= 96, wide = a->D == 128;
  if (a->kind == kDelta && wide ? ctas < 128 ? a->T * ctas * ctas < 540000 : a->T < 80
      : a->kind == kDelta       ? a->T < (some ? 128 : 132)
      : wide                    ? a->T < (some ? 64 : 400)
                                : !some || a->T < 240)
    return 0;
  const size_t one = chunk_bytes(a), all = (size_t)((a->T + kChunk - 1) / kChunk);
  return one * all <= kMaxScratch ? one * all : one > kMaxScratch ? one : kMaxScratch / one * one;
}

int scan_chunks_launch(const l3ci_recurrent_scan_args* a, void* scratch, size_t bytes) {
  if (!applies(a)) return fail(L3CI_ERR_UNSUPPORTED, "recurrent_scan: these sizes are not scanned by chunks");
  if (a->kind == kDelta) return a->D == 64 ? launch<float, kDelta, 64>(a, scratch, bytes) : launch<float, kDelta, 128>(a, scratch, bytes);
  return a->D == 64 ? launch<__nv_bfloat16, kTimeMix, 64>(a, scratch, bytes) : launch<__nv_bfloat16, kTimeMix, 128>(a, scratch, bytes);
}

}  // namespace l3ci
