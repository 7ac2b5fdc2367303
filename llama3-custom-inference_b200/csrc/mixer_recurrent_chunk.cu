// The linear recurrences of prompts by chunks of 16 tokens (include/l3ci_mixers.h, l3ci_recurrent_scan_chunks).
//
// Token by token every step of the state waits for the sums over it (850 cycles a token at 48 heads of 128 x 128, mixer_recurrent.cu).  Over a
// chunk whose first token finds the state S,
//   gated delta rule:  u_i = beta_i (v_i - (k_i G_i)^T S - sum_{j<i} L_ij u_j),   o_i = (q_i G_i)^T S + sum_{j<=i} M_ij u_j,
//                      S <- diag(G) S + sum_j (k_j G_{>j}) u_j^T,
// with G_i the product of the decays up to token i, L_ij and M_ij the products of k_i, q_i with k_j decayed from j to i.  With T the inverse of
// (1 + beta L) times beta, U = T (V - (k G) S), and all but the terms with S is known ahead, for all chunks at once.  Time mixing is the same with
// U = V, decays up to i - 1 and the bonus on the diagonal of M.
//   chunk_inputs_kernel  a warp per head and chunk, lanes over channels: the decayed keys of the chunk's tokens stay in registers and are
//     multiplied on from token to token, so that every decay is a product of factors at most 1 and none is divided by; L's and M's rows are the
//     lanes' sums, T's columns a lane's each.
//   chunk_scan_kernel    a warp per 16 columns of the state, whose transpose it keeps in accumulators of m16n8k8 products: per chunk U, the
//     outputs and the new state are 312 of them (128 rows).  Operands are 32-bit, split into tf32 parts: two and three
//     products for the sums over the state, three and six (all but what lies below 2^-33) for U and the new state.  An accumulator's columns are the next product's depth, taken in the order in which they lie.  Chunks come through a ring of bulk
//     copies.
// 1777 tokens of 3 x 16 heads of 128 x 128 (delta rule): 429 us, token by token 741; 3 x 32 heads of 64 x 64 (time mixing): 231, 374.  Most of it is the
// scan, a warp per scheduler, of which the products alone are 3300 cycles a chunk.  With U and W instead of T in the chunks the rows of
// the forward substitution took longer than the scan; with the values read by the scan's lanes themselves a chunk took 1.4 times as long.
// Errors against 64 bits: outputs the same (their rounding to bf16); states after such prompts, of their norm, delta rule of four layers 1.43,
// 1.29, 1.27, 1.76 e-7, token by token 1.52, 1.24, 1.24, 2.34, time mixing 1.76 to 1.97 e-7 and 1.86 to 2.02.  By three products throughout (346
// us) it was 1.6 to 2.1 e-7: the bit that two parts leave out, and the product of the small parts.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mixer_recurrent.h"
#include "ptx_sm100.cuh"
#include "tcgen05.cuh"

namespace l3ci {
namespace {

constexpr int kChunk = 16;
constexpr int kDelta = 0, kTimeMix = 1;
constexpr int kScanWarps = 4;
constexpr int kBlockCols = 16 * kScanWarps;       // state columns of a CTA
constexpr int kVPitch = kBlockCols * 2 + 16;      // bytes of a token's values in a stage
constexpr int kMPitch = 20;                       // floats; pitches: neighbouring rows on other banks

// A chunk's block of D channels, in floats: W = k G (delta rule) and Q = q G, K decayed to the chunk's end, M, T (delta rule), the chunk's decays.  W,
// Q and K lie as the scan's lanes take them, 16 bytes each, split into their tf32 parts: of a token, hi and lo of two channels; of K, of a channel,
// hi and lo of two tokens.
template <int KIND, int D>
struct ChunkShape {
  static constexpr int kWPitch = 2 * D + 16, kKPitch = 4 * D + 8;    // of a token, of two tokens
  static constexpr int kW = KIND == kDelta ? kChunk * kWPitch : 0;
  static constexpr int kQ = kChunk * kWPitch, kK = kChunk / 2 * kKPitch, kM = kChunk * kMPitch;
  static constexpr int kAtQ = kW, kAtK = kAtQ + kQ, kAtM = kAtK + kK, kAtT = kAtM + kM, kAtG = kAtT + (KIND == kDelta ? kM : 0);
  static constexpr int kFloats = kAtG + D;
  static constexpr int kStage = kFloats * 4 + kChunk * kVPitch;      // bytes in the scan: the block and the values
  static_assert(kFloats % 4 == 0, "bulk copies of whole 16-byte vectors");
};

// A 32-bit number as two of the 11 bits that a tf32 product takes.  (Integer instructions: the conversion's own runs at an eighth of their rate.)
struct Split { uint32_t hi, lo; };
__device__ __forceinline__ Split split(float x) {
  Split s;
  s.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  s.lo = __float_as_uint(x - __uint_as_float(s.hi)) + 0x1000u;
  return s;
}

// The same without loss: lo as it is, of which a product takes the first 11 bits; the rest of it is a third part.
__device__ __forceinline__ Split split_whole(float x) {
  Split s;
  s.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  s.lo = __float_as_uint(x - __uint_as_float(s.hi));
  return s;
}
__device__ __forceinline__ uint32_t rest(uint32_t lo) { return __float_as_uint(__uint_as_float(lo) - __uint_as_float(lo & 0xffffe000u)); }

struct ChunkParams {
  l3ci_recurrent_scan_args a;
  float* blocks;                 // [B * H][chunks]
  int t0, tokens, chunks;        // of this segment
  int col_blocks, last, ring;
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
  f2 t[kChunk][P2], run[P2], gb[P2], bonus[P2];   // decayed keys; product of the decays so far
  // a pair of channels of a token, of W or Q
  auto put = [&](float* row, int j, f2 v) {
    float x, y;
    f2_unpack(v, x, y);
    const Split sx = split(x), sy = split(y);
    *reinterpret_cast<uint4*>(row + 2 * (d0 + 2 * j)) = make_uint4(sx.hi, sy.hi, sx.lo, sy.lo);
  };
  float t_col[kChunk];                            // column lane % 16 of T
#pragma unroll
  for (int j = 0; j < kChunk; ++j) t_col[j] = 0.f;
#pragma unroll
  for (int j = 0; j < P2; ++j) {
    run[j] = pair_of(1.f, 1.f);
    gb[j] = bonus[j] = 0ull;
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
        qg[j] = f2_mul(q[j], run[j]);
        kg[j] = f2_mul(bonus[j], k[j]);
        run[j] = f2_mul(run[j], g[j]);
      }
      put(block + Sh::kAtQ + i * Sh::kWPitch, j, qg[j]);
      if (KIND == kDelta) put(block + i * Sh::kWPitch, j, kg[j]);
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
    if (lane >= kChunk) block[Sh::kAtM + i * kMPitch + lane - kChunk] = lane - kChunk <= i ? sums[0] : 0.f;
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
      if (lane < kChunk) block[Sh::kAtT + i * kMPitch + lane] = col;
    }
  }
#pragma unroll
  for (int i = 0; i < kChunk; i += 2)
#pragma unroll
    for (int j = 0; j < P2; ++j) {
      float x[2], y[2];
      f2_unpack(t[i][j], x[0], x[1]);
      f2_unpack(t[i + 1][j], y[0], y[1]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const Split sx = split_whole(x[e]), sy = split_whole(y[e]);
        *reinterpret_cast<uint4*>(block + Sh::kAtK + i / 2 * Sh::kKPitch + 4 * (d0 + 2 * j + e)) = make_uint4(sx.hi, sy.hi, sx.lo, sy.lo);
      }
    }
#pragma unroll
  for (int j = 0; j < P2; ++j) *reinterpret_cast<f2*>(block + Sh::kAtG + d0 + 2 * j) = run[j];
}

// ---- the scan ----------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// An accumulator as the left operand of the next product, in two parts: its columns 2 t and 2 t + 1 are the depths t and t + 4.
struct Left { uint32_t hi[4], lo[4]; };
template <bool WHOLE = false>
__device__ __forceinline__ Left left(const float (&c)[4]) {
  Left l;
  const int from[4] = {0, 2, 1, 3};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const Split s = WHOLE ? split_whole(c[from[i]]) : split(c[from[i]]);
    l.hi[i] = s.hi;
    l.lo[i] = s.lo;
  }
  return l;
}
struct Right { Split x, y; };
// c (large products: their accumulator is cut off, not rounded) and d (small ones) += l r of split_whole's parts, all but what lies below 2^-33; EXACT: l has no small parts
template <bool EXACT>
__device__ __forceinline__ void mma_whole(float (&c)[4], float (&d)[4], const Left& l, const Right& r) {
  const uint32_t rx = rest(r.x.lo), ry = rest(r.y.lo);
  mma_tf32(d, l.hi, rx, ry);
  mma_tf32(d, l.hi, r.x.lo, r.y.lo);
  if (!EXACT) {
    uint32_t lr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) lr[i] = rest(l.lo[i]);
    mma_tf32(d, lr, r.x.hi, r.y.hi);
    mma_tf32(d, l.lo, r.x.lo, r.y.lo);
    mma_tf32(d, l.lo, r.x.hi, r.y.hi);
  }
  mma_tf32(c, l.hi, r.x.hi, r.y.hi);
}

__device__ __forceinline__ Right right(const float* p) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  return {{v.x, v.z}, {v.y, v.w}};
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

constexpr int kMaxStages = 4;

template <int KIND, int D>
__global__ void __launch_bounds__(32 * (kScanWarps + 1), 1)
chunk_scan_kernel(const __grid_constant__ ChunkParams p) {
  using Sh = ChunkShape<KIND, D>;
  constexpr int NT = D / 8;                       // accumulators of 8 state rows
  extern __shared__ __align__(128) uint8_t ring_smem[];
  __shared__ __align__(8) uint64_t bars[2 * kMaxStages];
  const l3ci_recurrent_scan_args& a = p.a;
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + kMaxStages * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int vb = blockIdx.x % p.col_blocks, bh = blockIdx.x / p.col_blocks, h = bh % a.H, b = bh / a.H;
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.ring; ++i) {
      mbar_init(full0 + i * 8, 1);
      mbar_init(empty0 + i * 8, kScanWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  pdl_begin();
  const bool fresh = a.positions[b] == 0 && p.t0 == 0;
  bool ok = true;
  int asked = 0;
  if (warp == kScanWarps) {
    // ---- producer: a chunk's block, and a token's values by each of 16 lanes ----
    const float* block = p.blocks + (long long)bh * p.chunks * Sh::kFloats;
    const __nv_bfloat16* v = static_cast<const __nv_bfloat16*>(a.v) + ((long long)b * a.T + p.t0) * a.v_st + h * a.v_sh + vb * kBlockCols;
    const uint32_t v_bytes = min(kBlockCols, a.V - vb * kBlockCols) * 2;
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
      if (++s == p.ring) { s = 0; parity ^= 1; }
    }
    __syncwarp();
    if (a.tail && p.last && vb == 0) move_tails<__nv_bfloat16>(a, b, h, lane, 32, a.positions[b] == 0);
  } else {
    const int c0 = vb * kBlockCols + warp * 16;
    float* state = a.state + b * a.state_sb + (long long)h * D * a.V + c0;
    float S[NT][4];
#pragma unroll
    for (int x = 0; x < NT; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = 8 * x + 2 * t4 + (e & 1), col = g + (e >> 1) * 8;
        S[x][e] = !fresh && c0 + col < a.V ? state[(long long)d * a.V + col] : 0.f;
      }
    __nv_bfloat16* out = static_cast<__nv_bfloat16*>(a.out) + ((long long)b * a.T + p.t0) * a.out_st + h * a.out_sh + c0;
    for (int i = 0, s = 0, parity = 0; i < p.chunks; ++i) {
      if (!mbar_wait_bounded(full0 + s * 8, parity)) { ok = false; break; }
      const float* st = reinterpret_cast<const float*>(ring_smem + s * Sh::kStage);
      const uint8_t* vs = ring_smem + s * Sh::kStage + Sh::kFloats * 4 + (warp * 16 + g) * 2;
      // (W S)^T and (Q S)^T, by token tiles of 8; the large products in two runs, the small ones in a third: an accumulator is cut off, not
      // rounded, at every step
      float ws[3][2][4] = {}, os[3][2][4] = {};
#pragma unroll
      for (int x = 0; x < NT; ++x) {
        const Left l = left<>(S[x]);
        Right w[2], q[2];
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          const int at = (8 * tt + g) * Sh::kWPitch + 16 * x + 4 * t4;
          q[tt] = right(st + Sh::kAtQ + at);
          if (KIND == kDelta) w[tt] = right(st + at);
        }
#pragma unroll
        for (int part = 0; part < 3; ++part)
#pragma unroll
          for (int tt = 0; tt < 2; ++tt) {
            const int run = part == 0 ? x % 2 : 2;
            if (KIND == kDelta) mma_tf32(ws[run][tt], part == 2 ? l.lo : l.hi, part == 1 ? w[tt].x.lo : w[tt].x.hi, part == 1 ? w[tt].y.lo : w[tt].y.hi);
            mma_tf32(os[run][tt], part == 2 ? l.lo : l.hi, part == 1 ? q[tt].x.lo : q[tt].x.hi, part == 1 ? q[tt].y.lo : q[tt].y.hi);
          }
      }
      // U^T, and the outputs with it: sums over the chunk's tokens j, rows i of T and of M
      Left u[2];
      auto by_rows = [&](const float* rows, const Left (&l)[2], float (&c)[3][2][4], bool exact, bool whole) {   // exact: l has no small part
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          Right m[2];
#pragma unroll
          for (int ti = 0; ti < 2; ++ti) {
            const float2 f = *reinterpret_cast<const float2*>(rows + (8 * ti + g) * kMPitch + 8 * tt + 2 * t4);
            m[ti] = whole ? Right{split_whole(f.x), split_whole(f.y)} : Right{split(f.x), split(f.y)};
          }
          if (whole) {
#pragma unroll
            for (int ti = 0; ti < 2; ++ti) mma_whole<false>(c[tt][ti], c[2][ti], l[tt], m[ti]);
            continue;
          }
#pragma unroll
          for (int part = 0; part < (exact ? 2 : 3); ++part)
#pragma unroll
            for (int ti = 0; ti < 2; ++ti)
              mma_tf32(c[part == 0 ? tt : 2][ti], part == 2 ? l[tt].lo : l[tt].hi, part == 1 ? m[ti].x.lo : m[ti].x.hi, part == 1 ? m[ti].y.lo : m[ti].y.hi);
        }
      };
#pragma unroll
      for (int tt = 0; tt < 2; ++tt) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[e] = to_f32(*reinterpret_cast<const __nv_bfloat16*>(vs + (8 * tt + 2 * t4 + (e & 1)) * kVPitch + (e >> 1) * 16));
          if (KIND == kDelta) v[e] -= ws[0][tt][e] + ws[1][tt][e] + ws[2][tt][e];
        }
        u[tt] = left<true>(v);
      }
      if (KIND == kDelta) {
        float us[3][2][4] = {};
        by_rows(st + Sh::kAtT, u, us, false, true);
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
#pragma unroll
          for (int e = 0; e < 4; ++e) us[0][tt][e] += us[1][tt][e] + us[2][tt][e];
          u[tt] = left<true>(us[0][tt]);
        }
      }
      by_rows(st + Sh::kAtM, u, os, KIND == kTimeMix, false);      // (time mixing's U are bf16)
      const int n = min(kChunk, p.tokens - i * kChunk);
#pragma unroll
      for (int ti = 0; ti < 2; ++ti)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int tok = 8 * ti + 2 * t4 + (e & 1), col = g + (e >> 1) * 8;
          if (tok < n && c0 + col < a.V) out[(long long)(i * kChunk + tok) * a.out_st + col] = __float2bfloat16_rn(os[0][ti][e] + os[1][ti][e] + os[2][ti][e]);
        }
      // the state: decayed, and the chunk's keys times U
      constexpr int kTogether = 4;
#pragma unroll
      for (int x0 = 0; x0 < NT; x0 += kTogether) {
        Right k[kTogether][2];
        float add[kTogether][4] = {}, small[kTogether][4] = {}, odd[kTogether][4] = {};
#pragma unroll
        for (int x = 0; x < kTogether; ++x)
#pragma unroll
          for (int tt = 0; tt < 2; ++tt) k[x][tt] = right(st + Sh::kAtK + (4 * tt + t4) * Sh::kKPitch + 4 * (8 * (x0 + x) + g));
#pragma unroll
        for (int tt = 0; tt < 2; ++tt)
#pragma unroll
          for (int x = 0; x < kTogether; ++x) mma_whole<KIND == kTimeMix>(tt > 0 ? odd[x] : add[x], small[x], u[tt], k[x][tt]);
#pragma unroll
        for (int x = 0; x < kTogether; ++x) {
          const float2 f = *reinterpret_cast<const float2*>(st + Sh::kAtG + 8 * (x0 + x) + 2 * t4);
#pragma unroll
          for (int e = 0; e < 4; ++e) S[x0 + x][e] = fmaf(S[x0 + x][e], e & 1 ? f.y : f.x, add[x][e] + (odd[x][e] + small[x][e]));
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + s * 8);
      if (++s == p.ring) { s = 0; parity ^= 1; }
    }
    if (ok)
#pragma unroll
      for (int x = 0; x < NT; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int d = 8 * x + 2 * t4 + (e & 1), col = g + (e >> 1) * 8;
          if (c0 + col < a.V) state[(long long)d * a.V + col] = S[x][e];
        }
  }
  if (!ok && lane == 0 && a.status) atomicExch(a.status, (int)L3CI_ERR_DEVICE_WAIT);
  // a wait ran out: the copies still under way land before the shared memory is given back
  if (__syncthreads_or(!ok))
    for (int f = asked > p.ring ? asked - p.ring : 0; f < asked; ++f) (void)mbar_wait_bounded_one(full0 + f % p.ring * 8, (uint32_t)(f / p.ring) & 1u);
}

// Scratch of the chunks of `tokens` tokens of all heads.
size_t chunk_bytes(const l3ci_recurrent_scan_args* a) {
  const size_t floats = a->kind == kDelta ? (a->D == 64 ? ChunkShape<kDelta, 64>::kFloats : ChunkShape<kDelta, 128>::kFloats)
                                          : (a->D == 64 ? ChunkShape<kTimeMix, 64>::kFloats : ChunkShape<kTimeMix, 128>::kFloats);
  return (size_t)a->B * a->H * floats * 4;
}
constexpr size_t kMaxScratch = 256ull << 20;      // longer prompts go in segments

template <typename Q, int KIND, int D>
int launch(const l3ci_recurrent_scan_args* a, void* scratch, size_t bytes) {
  using Sh = ChunkShape<KIND, D>;
  const size_t one = chunk_bytes(a);
  const int all = (a->T + kChunk - 1) / kChunk;
  const int most = (int)(bytes / one < (size_t)all ? bytes / one : (size_t)all);
  if (!scratch || most < 1 || !aligned16(scratch)) return fail(L3CI_ERR_SCRATCH, "recurrent_scan: %zu bytes of scratch needed at least, %zu given", one, bytes);
  const int segments = (all + most - 1) / most, per = (all + segments - 1) / segments;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(a->stream);
  auto inputs = chunk_inputs_kernel<Q, KIND, D>;
  auto scan = chunk_scan_kernel<KIND, D>;
  static bool configured[64] = {false};
  int dev = 0;
  L3CI_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    L3CI_CUDA_TRY(cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem_optin() - 1024));
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  for (int c = 0; c < all; c += per) {
    ChunkParams p = {};
    p.a = *a;
    p.col_blocks = (a->V + kBlockCols - 1) / kBlockCols;
    p.t0 = c * kChunk;
    p.chunks = per < all - c ? per : all - c;
    p.tokens = a->T - p.t0 < p.chunks * kChunk ? a->T - p.t0 : p.chunks * kChunk;
    p.last = c + per >= all;
    const long long heads = (long long)a->B * a->H, units = heads * p.chunks;
    p.blocks = static_cast<float*>(scratch);
    const int stage = Sh::kStage, room = max_smem_optin() - 1024;
    p.ring = room / stage < kMaxStages ? room / stage : kMaxStages;
    L3CI_LAUNCH("chunk_inputs_kernel", inputs, dim3((unsigned)((units + kInputWarps - 1) / kInputWarps)), dim3(32 * kInputWarps), 0, stream, p, units);
    L3CI_LAUNCH("chunk_scan_kernel", scan, dim3((unsigned)(heads * p.col_blocks)), dim3(32 * (kScanWarps + 1)), (size_t)p.ring * stage, stream, p);
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

size_t scan_chunks_scratch(const l3ci_recurrent_scan_args* a) {
  // From where the chunks are the faster, in CTAs of the scan and tokens (us by tokens and by chunks): 32 CTAs of the delta rule 384 tokens 79.5 and
  // 87.0, of time mixing 40.2 and 44.3, and a token more costs both the same; 64 CTAs 96 tokens 38.9 and 37.9, time mixing 128 25.5 and 25.6; 96
  // CTAs 48 tokens 30.7 and 30.0, 64 24.1 and 22.2; 256 CTAs 48 tokens 54.8 and 43.6, 33.9 and 28.1.
  const long long ctas = (long long)a->B * a->H * ((a->V + kBlockCols - 1) / kBlockCols);
  if (!applies(a) || ctas < 64 || a->T < 40 || a->T * ctas * ctas < 540000) return 0;
  const size_t one = chunk_bytes(a), all = (size_t)((a->T + kChunk - 1) / kChunk);
  return one * all <= kMaxScratch ? one * all : one > kMaxScratch ? one : kMaxScratch / one * one;
}

int scan_chunks_launch(const l3ci_recurrent_scan_args* a, void* scratch, size_t bytes) {
  if (!applies(a)) return fail(L3CI_ERR_UNSUPPORTED, "recurrent_scan: these sizes are not scanned by chunks");
  if (a->kind == kDelta) return a->D == 64 ? launch<float, kDelta, 64>(a, scratch, bytes) : launch<float, kDelta, 128>(a, scratch, bytes);
  return a->D == 64 ? launch<__nv_bfloat16, kTimeMix, 64>(a, scratch, bytes) : launch<__nv_bfloat16, kTimeMix, 128>(a, scratch, bytes);
}

}  // namespace l3ci
