// Nucleus (top-p) sampling step of a decode loop as one kernel: per sequence, the temperature softmax of its logits
// row, the nucleus of probability mass p, one draw from it, and the token bookkeeping that follows.
//
// The reference's sampling branch (model.py:367-369 `probs = softmax(logits / temperature)`, `sample_top_p`,
// model.py:400-423) sorts the whole vocabulary (128 256 entries) in descending order, takes the cumulative sum, drops
// every entry whose PRECEDING mass exceeds p, renormalises, draws with torch.multinomial and maps the draw back
// through the sort permutation: half a dozen full-vocabulary kernels per generated token.  The nucleus does not need
// the order, only its boundary: entry i is kept iff the mass of the entries that sort strictly before it is <= p.
// The weight e_i = exp((x_i - max) / T) is a function of the bf16 LOGIT, monotone, and a bf16 logit has only 65 536 patterns.
//
// top_p_count_kernel (rows of up to 8 x 65 528 logits, but for short ones of one CTA): a cluster of 8, 4 or 2 CTAs per row in small
// batches, one CTA in larger ones,
//   1. counts the keys (order-preserving patterns) of the row in shared memory in one pass,
//   2. finds the boundary of the nucleus digit by digit of the key from count x weight (2^-40 fixed point, exact sums); entries whose
//      logit equals the boundary pattern tie exactly and are kept in index order as long as the mass before them is <= p * sum (a
//      stable descending sort puts them in that order),
//   3. draws u in [0, 1) from a Philox4x32-10 stream keyed by (seed; row, step) and finds the entry where the mass of the nucleus in
//      INDEX order passes u * nucleus mass: the warp, the entry of its list.  Any fixed order gives the multinomial
//      distribution; index order needs no permutation.
// top_p_step_kernel (longer rows, and short ones of one CTA): the same integers by masses.  Each level of the search is a pass over
// the row that histograms the MASS per byte value in shared memory (integer atomics); weights are recomputed from the logits in every
// pass (same expression, same bits; the row stays in L2).
// Either writes the token exactly as l3ci_greedy_step does; nothing is sorted and nothing leaves the SMs.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include "bf16x8.cuh"
#include "host_common.h"
#include "ptx_sm100.cuh"
#include "warp_reduce.cuh"

namespace l3ci {
namespace {

constexpr int kTopPBlock = 1024;
constexpr int kTopPWarps = kTopPBlock / kWarp;

// Philox4x32-10 (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3", SC'11): first word of the block.
__device__ __forceinline__ uint32_t philox_first(uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c0;
}

// Block-wide exclusive prefix sum over the threads in index order, and the total.
template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* red, T& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T inc = v;
#pragma unroll
  for (int d = 1; d < kWarp; d <<= 1) {
    const T o = __shfl_up_sync(kFullMask, inc, d);
    if (lane >= d) inc += o;
  }
  __syncthreads();
  if (lane == kWarp - 1) red[warp] = inc;
  __syncthreads();
  T w = red[lane], winc = w;
#pragma unroll
  for (int d = 1; d < kWarp; d <<= 1) {
    const T o = __shfl_up_sync(kFullMask, winc, d);
    if (lane >= d) winc += o;
  }
  total = __shfl_sync(kFullMask, winc, kWarp - 1);
  const T before_warp = __shfl_sync(kFullMask, winc - w, warp);
  return before_warp + inc - v;
}

typedef unsigned long long u64;

// Several CTAs per row (a cluster of 2, 4 or 8 while rows x CTAs fit the device): each walks its share of the row in
// every pass, and the few numbers a pass yields (maximum, histogram, totals of the scans) are read from the peers'
// shared memory.  All CTAs then hold the same values and take the same decisions; sums are integers, so the split
// changes no bit.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier() {
  cluster_arrive();
  cluster_wait();
}
template <typename T>
__device__ __forceinline__ T ld_peer(const T* mine, uint32_t peer) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "32- or 64-bit values");
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(peer));
  if constexpr (sizeof(T) == 4) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
    return *reinterpret_cast<T*>(&v);
  } else {
    u64 v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
    return *reinterpret_cast<T*>(&v);
  }
}
// The CTAs' values of one quantity: each writes its own to a slot (no slot is used twice in a launch, so one cluster
// barrier per exchange is enough) and reads the others' after the barrier.  `before`: the sum over the CTAs in front
// of this one (the first CTA takes the front of the row); returns the sum over all.
template <int kCtas, typename T>
__device__ __forceinline__ T peer_sum(T mine, T* slot, uint32_t rank, T& before) {
  before = T(0);
  if constexpr (kCtas == 1) return mine;
  if (threadIdx.x == 0) *slot = mine;
  cluster_barrier();
  T all = T(0);
#pragma unroll
  for (uint32_t c = 0; c < (uint32_t)kCtas; ++c) {
    const T v = c == rank ? mine : ld_peer(slot, c);
    if (c < rank) before += v;
    all += v;
  }
  return all;
}
template <int kCtas>
__device__ __forceinline__ float peer_max(float mine, float* slot, uint32_t rank) {
  if constexpr (kCtas == 1) return mine;
  if (threadIdx.x == 0) *slot = mine;
  cluster_barrier();
  float m = mine;
#pragma unroll
  for (uint32_t c = 0; c < (uint32_t)kCtas; ++c)
    if (c != rank) m = fmaxf(m, ld_peer(slot, c));
  return m;
}

struct RowView {
  const __nv_bfloat16* row;
  long long vocab, nvec;   // nvec 16-byte vectors, then vocab - 8 * nvec scalars
  long long v_begin, v_end, s_begin;   // this CTA's vectors and where its scalars start (vocab: none)
  float scale, shift;      // weight of logit x: exp2(x * scale - shift), at most 1
  // The weight as a 2^-40 fixed-point integer.  (The hardware exponential, one instruction: a row is walked four
  // times and an SM has to evaluate 128 256 weights per pass; the same instruction on the same input gives the same
  // bits in every pass.)  All masses below are sums of these integers: exact, the same in whatever order they are
  // added (thousands of float additions of equal small terms into one accumulator all round the same way: torch's
  // own fp32 softmax is 7e-5 off on such rows), and addable with the integer atomics of shared memory — a float add
  // there is a compare-and-swap loop, which with 32 lanes on a few dozen hot bins retried ten times per add.
  __device__ __forceinline__ u64 weight(float x) const { return __float2ull_rn(fast_exp2(fmaf(x, scale, -shift)) * 1099511627776.f); }
};

// Order-preserving 16-bit key of a bf16 logit given as fp32 (larger logit, larger key; -0 and +0 share a key).  The
// weight is a monotone function of the logit and a bf16 logit has 65 536 patterns, so the nucleus boundary can be
// searched on the logit's own bits: two levels of 8 bits, and entries tie exactly when their logits are equal.
__device__ __forceinline__ uint32_t logit_key(float x) {
  const uint32_t u = __float_as_uint(x) >> 16;
  if (u == 0x8000u) return 0x8000u;                      // -0 -> +0
  return (u & 0x8000u) ? (~u & 0xffffu) : (u | 0x8000u);
}

constexpr int kCopies = 8;   // histogram copies (warp w adds to copy w % 8): spreads the adds over more banks and keeps a
                             // 16-bit limb's sum below 2^32 (a copy sees at most 4 warps x 4096 entries)

// One level of the search: among all entries (level 0) or those whose key has `prefix` in its high byte (level 1), the
// byte value in which the mass of the strictly larger keys crosses `budget`.  Masses are histogrammed per byte value as
// three 16-bit limbs of the fixed-point weight (integer atomics), summed exactly, and a block-wide suffix scan over the
// 256 values finds the crossing.  Returns the byte (0xffffffff: the candidates all fit the budget) and subtracts the
// mass above it from `budget`.  On level 0 the budget is not known yet: the pass yields the sum of all weights
// (`total_out`) and the budget becomes top_p times it.  All threads take part and get the same answer.
template <int kCtas>
__device__ __forceinline__ uint32_t search_level(const RowView& rv, int level, uint32_t prefix, float top_p, u64& total_out,
                                                 u64& budget, uint32_t* limbs, u64* red, int* s_pick, u64* s_above, uint32_t rank) {
  for (int i = threadIdx.x; i < kCopies * 3 * 256; i += kTopPBlock) limbs[i] = 0u;
  __syncthreads();
  uint32_t* mine = limbs + ((threadIdx.x >> 5) % kCopies) * 3 * 256;
  // a thread adds up consecutive entries that fall into the same bin and issues the atomics once per run
  int run_bin = -1;
  u64 run_q = 0;
  auto flush = [&]() {
    if (run_bin >= 0) {
      atomicAdd(mine + run_bin, (uint32_t)(run_q & 0xffffu));
      atomicAdd(mine + 256 + run_bin, (uint32_t)((run_q >> 16) & 0xffffu));
      atomicAdd(mine + 512 + run_bin, (uint32_t)(run_q >> 32));
    }
  };
  auto visit = [&](float x) {
    const uint32_t key = logit_key(x);
    if (level != 0 && (key >> 8) != prefix) return;
    const int bin = level == 0 ? (int)(key >> 8) : (int)(key & 255u);
    const u64 q = rv.weight(x);
    if (bin == run_bin) run_q += q;
    else { flush(); run_bin = bin; run_q = q; }
  };
  for (long long v = rv.v_begin + threadIdx.x; v < rv.v_end; v += kTopPBlock) {
    float f[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(rv.row) + v), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) visit(f[j]);
  }
  for (long long i = rv.s_begin + threadIdx.x; i < rv.vocab; i += kTopPBlock) visit(__bfloat162float(rv.row[i]));
  flush();
  __syncthreads();
  if constexpr (kCtas > 1) cluster_barrier();   // the peers' histograms are complete too
  // thread t < 256 owns byte value d = 255 - t (a prefix scan over threads is then a suffix scan over byte values):
  // the wanted value is the largest d whose inclusive suffix sum exceeds the budget, i.e. the mass strictly above it
  // is still within the budget and the mass down to it is not
  u64 h = 0;
  const int d = 255 - (int)threadIdx.x;
  if (threadIdx.x < 256) {
#pragma unroll
    for (int c = 0; c < kCopies; ++c) {
      const uint32_t* l = limbs + c * 3 * 256;
      h += (u64)l[d] + ((u64)l[256 + d] << 16) + ((u64)l[512 + d] << 32);
      if constexpr (kCtas > 1) {
#pragma unroll
        for (uint32_t pc = 0; pc < (uint32_t)kCtas; ++pc)
          if (pc != rank) h += (u64)ld_peer(l + d, pc) + ((u64)ld_peer(l + 256 + d, pc) << 16) + ((u64)ld_peer(l + 512 + d, pc) << 32);
      }
    }
  }
  if constexpr (kCtas > 1) cluster_barrier();   // all have read: the histograms may be cleared for the next level
  u64 total;
  const u64 before = block_exclusive_scan<u64>(h, red, total);   // mass of the byte values above d
  total_out = total;
  if (level == 0) budget = (u64)((double)top_p * (double)total);
  if (threadIdx.x == 0) { *s_pick = -1; *s_above = total; }
  __syncthreads();
  if (threadIdx.x < 256 && before <= budget && before + h > budget) { *s_pick = d; *s_above = before; }
  __syncthreads();
  const int pick = *s_pick;
  if (pick < 0) return 0xffffffffu;
  budget -= *s_above;
  return (uint32_t)pick;
}

template <int kCtas>
__global__ void __launch_bounds__(kTopPBlock)
top_p_step_kernel(const __nv_bfloat16* __restrict__ logits, long long vocab, long long row_stride, float inv_temperature,
                  float top_p, unsigned long long seed, long long* __restrict__ out_tokens, long long out_stride,
                  long long out_cols, long long* __restrict__ steps, long long* __restrict__ next_input,
                  int* __restrict__ positions, int* __restrict__ seq_lens, int* __restrict__ nucleus_count,
                  float* __restrict__ nucleus_mass) {
  __shared__ uint32_t limbs[kCopies * 3 * 256];
  __shared__ float redf[kTopPWarps];
  __shared__ u64 red[kTopPWarps];
  __shared__ long long redl[kTopPWarps];
  __shared__ int s_pick;
  __shared__ u64 s_above;
  __shared__ int s_owner;
  __shared__ long long s_token;
  __shared__ u64 s_slots[8];     // values for the peer CTA, one slot per exchange
  pdl_launch_dependents();  // the next one may be set up while this one runs
  pdl_wait();               // the previous kernel of the stream has completed; its writes are visible
  const long long b = blockIdx.x / kCtas;
  const uint32_t rank = kCtas > 1 ? cluster_rank() : 0u;
  RowView rv;
  rv.row = logits + b * row_stride;
  rv.vocab = vocab;
  rv.nvec = (reinterpret_cast<uintptr_t>(rv.row) & 15u) == 0 ? vocab / kVecElems : 0;
  rv.scale = inv_temperature * 1.4426950408889634f;
  // this CTA's share of the row in the passes that take it in any order: half of the vectors each, the scalars
  // behind them with the last CTA
  rv.v_begin = rv.nvec * rank / kCtas;
  rv.v_end = rv.nvec * (rank + 1) / kCtas;
  rv.s_begin = rank == kCtas - 1 ? rv.nvec * kVecElems : vocab;

  // ---- 1. maximum of the row (the sum of the weights falls out of the first histogram) ----
  float m = -INFINITY;
  for (long long v = rv.v_begin + threadIdx.x; v < rv.v_end; v += kTopPBlock) {
    float f[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(rv.row) + v), f);
    m = fmaxf(m, fmaxf(fmaxf(fmaxf(f[0], f[1]), fmaxf(f[2], f[3])), fmaxf(fmaxf(f[4], f[5]), fmaxf(f[6], f[7]))));
  }
  for (long long i = rv.s_begin + threadIdx.x; i < vocab; i += kTopPBlock) m = fmaxf(m, __bfloat162float(rv.row[i]));
  m = group_max<kWarp>(m);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) redf[threadIdx.x >> 5] = m;
  __syncthreads();
  float row_max = group_max<kWarp>(redf[threadIdx.x & 31]);
  row_max = peer_max<kCtas>(row_max, reinterpret_cast<float*>(&s_slots[0]), rank);
  rv.shift = row_max * rv.scale;

  // ---- 2. boundary of the nucleus: the largest logit pattern k* whose strictly-larger mass is still <= p * Z ----
  uint32_t key_star = 0u;
  bool all_kept = false;
  u64 Z = 0, budget = 0, bud = 0;
  {
    const uint32_t hi = search_level<kCtas>(rv, 0, 0u, top_p, Z, bud, limbs, red, &s_pick, &s_above, rank);
    budget = (u64)((double)top_p * (double)Z);
    if (hi == 0xffffffffu) {
      all_kept = true;   // top_p >= 1
    } else {
      u64 unused;
      const uint32_t lo = search_level<kCtas>(rv, 1, hi, 0.f, unused, bud, limbs, red, &s_pick, &s_above, rank);
      key_star = (hi << 8) | (lo == 0xffffffffu ? 0u : lo);   // (the sums are exact, so the second level finds its byte)
    }
  }
  const u64 above = budget - bud;   // mass of the entries whose logit is strictly above the boundary pattern
  // weight of the boundary pattern: the bf16 logit it stands for, through the same expression as every entry
  const uint32_t bits_star = (key_star & 0x8000u) ? (key_star & 0x7fffu) : (~key_star & 0xffffu);
  const u64 w_star = rv.weight(__uint_as_float(bits_star << 16));

  // ---- 3. nucleus mass per thread over a CONTIGUOUS run of the row (index order), ties at the boundary counted ----
  // runs of a multiple of 8 entries, so that an aligned row is walked with 16-byte loads
  constexpr long long kRowThreads = (long long)kTopPBlock * kCtas;   // the first CTA takes the front of the row
  const long long per = ((vocab + kRowThreads - 1) / kRowThreads + kVecElems - 1) / kVecElems * kVecElems;
  const long long row_thread = (long long)rank * kTopPBlock + threadIdx.x;
  const long long i_begin = row_thread * per < vocab ? row_thread * per : vocab;
  const long long i_end = i_begin + per < vocab ? i_begin + per : vocab;
  // calls fn(index, logit) for the entries of this thread's run in increasing order until fn returns true
  auto walk = [&](auto&& fn) {
    long long i = i_begin;
    if (rv.nvec > 0) {
      for (; i + kVecElems <= i_end; i += kVecElems) {
        float f[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(rv.row) + i / kVecElems), f);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (fn(i + j, f[j])) return;
      }
    }
    for (; i < i_end; ++i)
      if (fn(i, __bfloat162float(rv.row[i]))) return;
  };
  u64 w_mine = 0;
  long long n_eq = 0, n_above = 0;
  walk([&](long long, float x) {
    const uint32_t key = logit_key(x);
    if (all_kept || key > key_star) { w_mine += rv.weight(x); ++n_above; }
    else if (key == key_star) ++n_eq;
    return false;
  });
  long long eq_total;
  long long eq_before = block_exclusive_scan<long long>(n_eq, redl, eq_total);
  {   // index order over the CTAs: a CTA's entries come after all of those in front of it
    long long front;
    eq_total = peer_sum<kCtas>(eq_total, reinterpret_cast<long long*>(&s_slots[1]), rank, front);
    eq_before += front;
  }
  // entries equal to the boundary pattern, in index order: the j-th is kept while above + j * w* <= budget
  long long eq_kept = 0;
  if (!all_kept && eq_total > 0) {
    eq_kept = w_star > 0 ? (long long)((budget > above ? budget - above : 0) / w_star) + 1 : eq_total;
    if (eq_kept > eq_total) eq_kept = eq_total;
  }
  long long eq_mine = eq_kept - eq_before;
  eq_mine = eq_mine < 0 ? 0 : (eq_mine > n_eq ? n_eq : eq_mine);
  const u64 mass_mine = w_mine + (u64)eq_mine * w_star;
  u64 mass_total;
  u64 mass_before = block_exclusive_scan<u64>(mass_mine, red, mass_total);
  {
    u64 front;
    mass_total = peer_sum<kCtas>(mass_total, &s_slots[2], rank, front);
    mass_before += front;
  }

  // ---- 4. the draw: u in [0, 1) with 32 bits, target = floor(u * nucleus mass) < nucleus mass ----
  const long long step = steps ? steps[b] : 0;
  const uint32_t r = philox_first((uint32_t)seed, (uint32_t)(seed >> 32), (uint32_t)b, (uint32_t)(b >> 32), (uint32_t)step,
                                  (uint32_t)(step >> 32));
  const u64 target = __umul64hi(mass_total, (u64)r << 32);
  if (threadIdx.x == 0) s_owner = kTopPBlock;
  __syncthreads();
  if (mass_mine > 0 && mass_before <= target && target < mass_before + mass_mine) s_owner = (int)threadIdx.x;   // exactly one thread
  __syncthreads();
  // The thread whose run holds the target sits in one of the CTAs; that CTA writes the token.  An empty nucleus (a
  // row of NaNs) has no such thread: the first CTA's first thread stands in.
  const bool mine = s_owner < kTopPBlock || (mass_total == 0 && rank == 0);
  const int owner = s_owner < kTopPBlock ? s_owner : 0;
  if (mine && (int)threadIdx.x == owner) {
    u64 run = mass_before;
    long long eq_seen = eq_before, tok = -1, last = -1;
    walk([&](long long i, float x) {
      const uint32_t key = logit_key(x);
      bool in = all_kept || key > key_star;
      if (!in && key == key_star) { in = eq_seen < eq_kept; ++eq_seen; }
      if (!in) return false;
      last = i;
      run += rv.weight(x);
      if (run > target) { tok = i; return true; }
      return false;
    });
    if (tok < 0) tok = last >= 0 ? last : (i_begin < vocab ? i_begin : 0);
    s_token = tok;
  }
  __syncthreads();
  if (mine && threadIdx.x == 0) {
    const long long tok = s_token;
    if (out_tokens && steps) {
      if (step >= 0 && step < out_cols) out_tokens[b * out_stride + step] = tok;
      steps[b] = step + 1;
    } else if (out_tokens) {
      out_tokens[b * out_stride] = tok;
    }
    if (next_input) next_input[b] = tok;
    if (positions) positions[b] += 1;
    if (seq_lens) seq_lens[b] += 1;
    if (nucleus_mass) nucleus_mass[b] = Z > 0 ? (float)((double)mass_total / (double)Z) : 0.f;
  }
  if (nucleus_count) {
    long long total;
    block_exclusive_scan<long long>(n_above + eq_mine, redl, total);
    long long front;
    total = peer_sum<kCtas>(total, reinterpret_cast<long long*>(&s_slots[3]), rank, front);
    if (threadIdx.x == 0 && rank == 0) nucleus_count[b] = (int)total;
  }
  if constexpr (kCtas > 1) cluster_barrier();   // no CTA leaves while a peer may still read its shared memory
}


// ---- the same step by counts ---------------------------------------------------------------------------------------------------
// The weight is a function of the logit's key, so the mass of a key is its count times its weight, exactly: the row needs one
// histogram of counts over all 65 536 keys (16 bits each, 128 KB of shared memory) instead of a pass of three 64-bit-mass atomics
// per search level, and the weights are evaluated once per key that occurs.  A second pass over the row (from L2) lists the few entries of
// the nucleus.  All sums are the integers of the kernel above: same boundary, same ties, same draw, bit for bit.
//   64 rows of 128 256 logits: 22.1 us; 82 with the masses' histograms, whose atomics met on a few dozen bins; 34.3 with the row in
// registers, every lane weighing its own entries in unrolled loops: instruction fetch, and warps that waited for the lane with the most.
// Left is the counting: 14 of 43 thousand cycles, shared-memory atomics of 32 lanes on 32 random banks.
constexpr int kKeyWords = 32768;                  // two keys' counts each
constexpr int kGroup = 16;                        // neighbouring entries of a lane, at most
constexpr int kListed = kWarp * kGroup;           // entries of a warp's list
constexpr int kDense = 256;                       // of a round's 512, beyond which they are weighed without a list
constexpr int kCountSmem = (kKeyWords + kTopPWarps * kListed) * 4;
constexpr long long kMaxShare = 8191;             // groups of a CTA: a count of all its entries fits 16 bits
constexpr long long kFewLogits = 4096;            // logits of a one-CTA row that are few
// A weight is about 2^40 at most, except that of a logit without a number for one (NaN; an infinity or a value whose scaled
// difference to the maximum overflows): 2^63 or more, so that masses wrap.  Masses of weights below 2^44 do not, over the 524 224
// logits of the longest row.  A row with a larger weight is marked by this bit of its count.
constexpr uint32_t kOddWeight = 1u << 12;         // in a weight's high word
constexpr u64 kOddRow = 1u << 24;                 // above the entries of the longest row, with room for eight CTAs' marks

__device__ __forceinline__ uint32_t bits_key(uint32_t u) {   // logit_key of a bf16 pattern
  if (u == 0x8000u) return 0x8000u;
  return (u & 0x8000u) ? (~u & 0xffffu) : (u | 0x8000u);
}
__device__ __forceinline__ float key_logit(uint32_t key) { return __uint_as_float(((key & 0x8000u) ? (key & 0x7fffu) : (~key & 0xffffu)) << 16); }

// Sum over the warp's lanes in front of this one, and over all.
template <typename T>
__device__ __forceinline__ T warp_exclusive_scan(T v, T& total) {
  const int lane = threadIdx.x & 31;
  T inc = v;
#pragma unroll
  for (int d = 1; d < kWarp; d <<= 1) {
    const T o = __shfl_up_sync(kFullMask, inc, d);
    if (lane >= d) inc += o;
  }
  total = __shfl_sync(kFullMask, inc, kWarp - 1);
  return inc - v;
}
// Writes a value into the place of `mine` in a peer's shared memory.  (Of the few values of a meeting, which the CTAs then read from their
// own memory: a read of a peer's takes as long as the barrier once more.  The masses of the digits are read: 256 of them took longer to write.)
template <typename T>
__device__ __forceinline__ void st_peer(T* mine, uint32_t peer, T v) {
  static_assert(sizeof(T) == 4 || sizeof(T) == 8, "32- or 64-bit values");
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(peer));
  if constexpr (sizeof(T) == 4) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(*reinterpret_cast<uint32_t*>(&v)) : "memory");
  else asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(*reinterpret_cast<u64*>(&v)) : "memory");
}
// Sum of the CTAs' values, one per lane from slot 0 on, and of those in front of this CTA.
template <int kCtas, typename T>
__device__ __forceinline__ T slots_sum(const T* slots, uint32_t rank, T& front) {
  const uint32_t lane = threadIdx.x & 31;
  const T v = lane < (uint32_t)kCtas ? slots[lane] : T(0);
  T all;
  front = __shfl_sync(kFullMask, warp_exclusive_scan<T>(v, all), (int)rank);
  return all;
}

// Of 256 digits' masses (shared memory, digit d at digit_place(d)), by one warp: the largest digit whose mass together with that of
// the larger ones exceeds the budget, -1 if there is none; `above`: the mass of the larger ones; `total`: of all.
__device__ __forceinline__ int digit_place(int d) { return (255 - d) % 8 * 32 + (255 - d) / 8; }   // neighbouring lanes' digits on neighbouring banks
template <typename F>
__device__ __forceinline__ int digit_crossing(const u64* mass, F&& budget_of, u64& above, u64& total) {
  const int lane = threadIdx.x & 31;
  u64 h[8], sum = 0;                     // lane l: digits 255 - 8 l downwards
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    h[i] = mass[i * 32 + lane];
    sum += h[i];
  }
  u64 before = warp_exclusive_scan<u64>(sum, total);
  const u64 budget = budget_of(total);
  int pick = -1;
  u64 at = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (pick < 0 && before <= budget && before + h[i] > budget) {
      pick = 255 - 8 * lane - i;
      at = before;
    }
    before += h[i];
  }
  const unsigned who = __ballot_sync(kFullMask, pick >= 0);
  if (who == 0) return -1;
  const int src = __ffs(who) - 1;
  above = __shfl_sync(kFullMask, at, src);
  return __shfl_sync(kFullMask, pick, src);
}

template <int kCtas>
__global__ void __launch_bounds__(kTopPBlock, 1)
top_p_count_kernel(const __nv_bfloat16* __restrict__ logits, long long vocab, long long row_stride, float inv_temperature,
                   float top_p, unsigned long long seed, long long* __restrict__ out_tokens, long long out_stride,
                   long long out_cols, long long* __restrict__ steps, long long* __restrict__ next_input,
                   int* __restrict__ positions, int* __restrict__ seq_lens, int* __restrict__ nucleus_count,
                   float* __restrict__ nucleus_mass, long long stand_in_run) {
  extern __shared__ __align__(16) uint32_t counts[];   // word k / 2 holds the counts of keys k (even: low half)
  __shared__ float redf[kTopPWarps];
  __shared__ u64 own_mass[256], digit_mass[256];   // of this CTA, of all
  __shared__ u64 warp_ties[kTopPWarps];          // ties << 32 | entries above them
  __shared__ u64 warp_mass[kTopPWarps];
  uint32_t* s_list = counts + kKeyWords;         // entries of the nucleus, by warp
  __shared__ float s_max[kCtas];
  __shared__ u64 s_mass[kCtas], s_ties[kCtas];   // the CTAs'; of s_ties bit 24 onwards: CTAs with an odd row
  // what the first warp finds for all
  __shared__ int s_pick[2], s_odd, s_first;
  __shared__ u64 s_above[2], s_total, s_budget, s_mass_front, s_mass_total;
  __shared__ long long s_eq_front, s_eq_kept, s_over_total;
  __shared__ int s_any_odd;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = kCtas > 1 ? cluster_rank() : 0u;
  for (int i = tid; i < kKeyWords / 4; i += kTopPBlock) reinterpret_cast<uint4*>(counts)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    s_odd = 0;
    s_first = kTopPWarps;
  }
  if constexpr (kCtas > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // (waited for ahead of the first write to a peer: all of them have started)
  pdl_launch_dependents();  // the next one may be set up while this one runs
  pdl_wait();               // the previous kernel of the stream has completed; its writes are visible
  const long long b = blockIdx.x / kCtas;
  const __nv_bfloat16* row = logits + b * row_stride;
  const unsigned short* row_bits = reinterpret_cast<const unsigned short*>(row);
  const long long step = steps ? steps[b] : 0;            // (barriers of all CTAs follow before one of them writes it)
  const bool vectors = (reinterpret_cast<uintptr_t>(row) & 15u) == 0;
  // vectors of 8 entries: the CTA's run, in it the warp's, an even number; there a round of 32 neighbouring groups at a time
  const long long vecs = (vocab + kVecElems - 1) / kVecElems;
  const long long v_end = vecs * (rank + 1) / kCtas, v_cta = vecs * rank / kCtas;
  const int per_warp = (int)((v_end - v_cta + 2 * kTopPWarps - 1) / (2 * kTopPWarps)) * 2;
  const long long v_warp = v_cta + (long long)warp * per_warp, first = v_warp * kVecElems;
  const int n_warp = (int)max(0ll, min(min((long long)per_warp, v_end - v_warp) * kVecElems, vocab - first));   // entries of this warp
  // (short runs: half a group each, so that all lanes have some)
  const int group = per_warp <= kWarp ? kGroup / 2 : kGroup, round = kWarp * group;
  auto entries = [&](int it) { return max(0, min(group, n_warp - it * round - lane * group)); };   // of this lane's group of round `it`
  struct Group { uint4 v[2]; };
  auto load = [&](int it) {                               // zeros where the lane has none
    Group g;
    const int n = entries(it);
    const unsigned short* at = row_bits + first + it * round + lane * group;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      g.v[i] = make_uint4(0u, 0u, 0u, 0u);
      const int left = n - i * kVecElems;
      if (vectors && left >= kVecElems) {
        g.v[i] = __ldg(reinterpret_cast<const uint4*>(at) + i);
      } else if (left > 0) {
        uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int j = 0; j < kVecElems; ++j)
          if (j < left) w[j / 2] |= (uint32_t)__ldg(at + i * kVecElems + j) << (16 * (j & 1));
        g.v[i] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    return g;
  };
  // Calls visit(round, group) for the warp's rounds, the next group under way.  (Loops that are not unrolled: a launch meets a cold
  // instruction cache, and unrolled by rounds, with the row in registers, fetching the kernel took a third of its time.)
  auto rounds = [&](auto&& visit) {
    Group next = {};
#pragma unroll 1
    for (int it = -1; it * round < n_warp; ++it) {
      const Group g = next;
      next = load(it + 1);
      if (it >= 0) visit(it, g);
    }
  };
  const uint32_t r = philox_first((uint32_t)seed, (uint32_t)(seed >> 32), (uint32_t)b, (uint32_t)(b >> 32), (uint32_t)step,
                                  (uint32_t)(step >> 32));
  auto bits_of = [&](const Group& g, int j) {
    const uint4 v = j < kVecElems ? g.v[0] : g.v[1];
    const uint32_t w = (j & 4) ? (j & 2) ? v.w : v.z : (j & 2) ? v.y : v.x;
    return (j & 1) ? w >> 16 : w & 0xffffu;
  };
  __syncthreads();                                        // the counts are cleared

  // ---- 1. counts of the keys and the maximum ----
  float m = -INFINITY;
  rounds([&](int it, const Group& g) {
    const int n = entries(it);
    const uint4 v = g.v[0], u = g.v[1];
    if (n == kGroup && v.x == v.y && v.y == v.z && v.z == v.w && v.x >> 16 == (v.x & 0xffffu) && u.x == v.x && u.y == v.x && u.z == v.x && u.w == v.x) {
      const uint32_t key = bits_key(v.x & 0xffffu);       // a flat row's lanes would queue at one word
      m = fmaxf(m, __uint_as_float(v.x << 16));
      atomicAdd(counts + (key >> 1), (uint32_t)kGroup << (16 * (key & 1)));
      return;
    }
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      if (j >= n) break;
      const uint32_t u = bits_of(g, j), key = bits_key(u);
      m = fmaxf(m, __uint_as_float(u << 16));
      atomicAdd(counts + (key >> 1), 1u << (16 * (key & 1)));
    }
  });
  m = group_max<kWarp>(m);
  if (lane == 0) redf[warp] = m;
  __syncthreads();
  m = group_max<kWarp>(redf[lane]);
  if constexpr (kCtas > 1) {
    cluster_wait();
    if (tid < kCtas) st_peer(&s_max[rank], (uint32_t)tid, m);
    cluster_barrier();
#pragma unroll
    for (int c = 0; c < kCtas; ++c) m = fmaxf(m, s_max[c]);
  }
  RowView rv;
  rv.scale = inv_temperature * 1.4426950408889634f;
  rv.shift = m * rv.scale;

  // ---- 2. boundary of the nucleus, digit by digit of the key: the masses of this CTA's entries, then of all ----
  // (a digit by a warp, neighbours to different ones: those that occur are neighbours)
  uint32_t any = 0;                                       // high words of the weights
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    const int d = i * kTopPWarps + warp;
    const uint4 c = reinterpret_cast<const uint4*>(counts + d * 128)[lane];
    u64 q = 0;
    if (__any_sync(kFullMask, (c.x | c.y | c.z | c.w) != 0u)) {
      const uint32_t w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) {     // (no branches: the eight are under way together)
        const uint32_t n = (k & 1) ? w[k / 2] >> 16 : w[k / 2] & 0xffffu;
        const u64 each = rv.weight(key_logit((uint32_t)(d * 256 + lane * 8 + k)));
        any |= n ? (uint32_t)(each >> 32) : 0u;
        q += (u64)n * each;
      }
#pragma unroll
      for (int k = 16; k >= 1; k /= 2) q += __shfl_xor_sync(kFullMask, q, k);
    }
    if (lane == 0) own_mass[d] = q;
  }
  if (any >= kOddWeight) s_odd = 1;
  if constexpr (kCtas > 1) cluster_barrier();
  else __syncthreads();
  if (tid < 256) {
    u64 h = own_mass[tid];
#pragma unroll
    for (uint32_t pc = 0; pc < (uint32_t)kCtas; ++pc)
      if (pc != rank) h += ld_peer(own_mass + tid, pc);
    digit_mass[digit_place(tid)] = h;
  }
  __syncthreads();
  // (the scans by the first warp alone: 32 warps' shuffles took longer than the barriers)
  if (warp == 0) {
    u64 total, over = 0, limit = 0;
    const int pick = digit_crossing(digit_mass, [&](u64 all) { return limit = (u64)((double)top_p * (double)all); }, over, total);
    if (lane == 0) { s_pick[0] = pick; s_above[0] = over; s_total = total; s_budget = limit; }
  }
  __syncthreads();
  const int hi = s_pick[0];
  const u64 Z = s_total, budget = s_budget;
  const bool all_kept = hi < 0;                           // top_p >= 1
  uint32_t key_star = 0u;
  u64 bud = budget;
  if (!all_kept) {
    bud -= s_above[0];
    u64 h = 0;
    if (tid < 256) {
      const uint32_t key = ((uint32_t)hi << 8) | (uint32_t)tid;
      uint32_t n = (counts[key >> 1] >> (16 * (key & 1))) & 0xffffu;
#pragma unroll
      for (uint32_t pc = 0; pc < (uint32_t)kCtas; ++pc)
        if (pc != rank) n += (ld_peer(counts + (key >> 1), pc) >> (16 * (key & 1))) & 0xffffu;
      if (n) h = (u64)n * rv.weight(key_logit(key));
    }
    if (tid < 256) digit_mass[digit_place(tid)] = h;      // (the first digit's have been read)
    __syncthreads();
    if (warp == 0) {
      u64 total, over = 0;
      const int pick = digit_crossing(digit_mass, [&](u64) { return bud; }, over, total);
      if (lane == 0) { s_pick[1] = pick; s_above[1] = over; }
    }
    __syncthreads();
    const int lo = s_pick[1];
    if (lo >= 0) bud -= s_above[1];
    key_star = ((uint32_t)hi << 8) | (lo < 0 ? 0u : (uint32_t)lo);   // (the sums are exact: the second digit is found)
  }
  const u64 above = budget - bud;                         // mass of the entries strictly above the boundary
  const u64 w_star = rv.weight(key_logit(key_star));

  // ---- 3. the nucleus in index order: per warp, ties at the boundary counted ----
  // Few entries are in it: packed compares build masks, the entries of their bits go into the warp's list, and its lanes weigh one each.
  // A round that has more than half of its entries in it is weighed as it is (rows of 128256 logits of one size: 32 us; by lists 59).
  // order(u): signed, -0 just below +0; at a boundary of 0 both tie
  auto order = [](uint32_t u) { const int t = (int)(short)u; return t ^ ((t >> 31) & 0x7fff); };
  const int star = all_kept ? -40000 : (int)key_star - 0x8000;
  const int star_low = star == 0 ? -1 : star;
  // every entry here and the boundary (which may be another share's entry) has a number: bf16's own compare orders them (and ties -0 and +0)
  const float boundary = key_logit(key_star);
  const bool plain = !s_odd && !all_kept && boundary == boundary;
  auto at_least = [&](int it, const Group& g) {           // bit j: entry j of the group is in the nucleus or ties
    const int n = entries(it);
    uint32_t in = 0u;
    if (plain) {
      const uint32_t star2 = ((key_star & 0x8000u) ? (key_star & 0x7fffu) : (~key_star & 0xffffu)) * 0x10001u;
      const __nv_bfloat162 limit = *reinterpret_cast<const __nv_bfloat162*>(&star2);
      uint32_t in_high = 0u;                              // of the words' high halves, 16 bits up
#pragma unroll
      for (int k = 0; k < kGroup / 2; ++k) {
        const uint4 v = g.v[k / 4];
        const uint32_t w = k % 4 == 0 ? v.x : k % 4 == 1 ? v.y : k % 4 == 2 ? v.z : v.w;
        const uint32_t mask = __hge2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w), limit);
        in |= mask & (1u << (2 * k));
        in_high |= mask & (0x20000u << (2 * k));
      }
      in = (in | in_high >> 16) & ((1u << n) - 1u);
    } else {
#pragma unroll 1
      for (int j = 0; j < n; ++j) in |= (order(bits_of(g, j)) >= star_low ? 1u : 0u) << j;
    }
    return in;
  };
  auto weigh = [&](const Group& g, uint32_t in, u64& w, int& ties) {   // entry by entry
    w = 0;
    ties = 0;
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      const uint32_t u = bits_of(g, j);
      const bool tie = order(u) <= star, mine = in >> j & 1u;
      const u64 each = rv.weight(__uint_as_float(u << 16));
      w += mine && !tie ? each : 0;
      ties += mine && tie;
    }
  };
  uint32_t* list = s_list + warp * kListed;               // in index order: pattern, place in the warp's run << 16
  auto entry = [&](int i, int n, bool& tie) {             // entry i of the list's n, and whether it ties at the boundary
    const uint32_t e = i < n ? list[i] : 0u;
    tie = i < n && order(e & 0xffffu) <= star;
    return e;
  };
  u64 w_warp = 0;
  int eq_warp = 0, over_warp = 0, listed = 0;
  bool whole = true;                                      // the list has them all
  rounds([&](int it, const Group& g) {
    uint32_t in = at_least(it, g);
    int all;
    int at = warp_exclusive_scan<int>(__popc(in), all);
    if (all > kDense || listed + all > kListed) {
      u64 w;
      int ties;
      weigh(g, in, w, ties);
      w_warp += w;
      ties = __reduce_add_sync(kFullMask, ties);
      eq_warp += ties;
      over_warp += all - ties;
      whole = false;
      return;
    }
    at += listed;
    listed += all;
#pragma unroll 1
    for (; in; in &= in - 1) {
      const int j = __ffs(in) - 1;
      list[at++] = bits_of(g, j) | (uint32_t)(it * round + lane * group + j) << 16;
    }
  });
  __syncwarp();
#pragma unroll 1
  for (int i = 0; i < listed; i += kWarp) {
    bool tie;
    const uint32_t e = entry(i + lane, listed, tie);
    const u64 w = rv.weight(__uint_as_float(e << 16));
    w_warp += i + lane < listed && !tie ? w : 0;
    const int ties = __popc(__ballot_sync(kFullMask, tie));
    eq_warp += ties;
    over_warp += min(listed - i, kWarp) - ties;
  }
#pragma unroll
  for (int k = 16; k >= 1; k /= 2) w_warp += __shfl_xor_sync(kFullMask, w_warp, k);
  if (lane == 0) {
    warp_ties[warp] = (u64)eq_warp << 32 | (u64)over_warp;
    warp_mass[warp] = w_warp;
  }
  __syncthreads();
  if (warp == 0) {
    u64 ties_all, mass_all;
    const u64 ties = warp_exclusive_scan<u64>(warp_ties[lane], ties_all);
    const u64 mass = warp_exclusive_scan<u64>(warp_mass[lane], mass_all);
    warp_ties[lane] = ties;                               // from here on: of the warps in front
    warp_mass[lane] = mass;
    if (s_odd) ties_all |= kOddRow;
    if (lane < kCtas) {
      if constexpr (kCtas > 1) {
        st_peer(&s_ties[rank], (uint32_t)lane, ties_all);
        st_peer(&s_mass[rank], (uint32_t)lane, mass_all);
      } else {
        s_ties[0] = ties_all;
        s_mass[0] = mass_all;
      }
    }
  }
  __syncwarp();
  if constexpr (kCtas > 1) cluster_barrier();
  if (warp == 0) {
    u64 ties_in_front, mass_in_front;
    const u64 ties_all = slots_sum<kCtas>(s_ties, rank, ties_in_front);
    const u64 mass_all = slots_sum<kCtas>(s_mass, rank, mass_in_front);
    const long long eq_all = (long long)(ties_all >> 32), eq_in_front = (long long)(ties_in_front >> 32);
    const int over_all = (int)(ties_all & (kOddRow - 1));
    // entries equal to the boundary, in index order: the j-th is kept while above + j * w* <= budget
    long long kept = 0;
    if (!all_kept && eq_all > 0) {
      kept = eq_all;
      if (w_star > 0) {
        const u64 room = budget > above ? budget - above : 0;
        // (a division of 64 bits only where not all are kept)
        if (__umul64hi(w_star, (u64)(eq_all - 1)) != 0 || w_star * (u64)(eq_all - 1) > room) kept = (long long)(room / w_star) + 1;
      }
      if (kept > eq_all) kept = eq_all;
    }
    if (lane == 0) {
      s_eq_kept = kept; s_eq_front = eq_in_front; s_over_total = over_all; s_any_odd = (ties_all & 0xffffffffu) >= kOddRow;
      s_mass_total = mass_all; s_mass_front = mass_in_front;
    }
  }
  __syncthreads();
  const long long eq_kept = s_eq_kept, eq_before = (long long)(warp_ties[warp] >> 32) + s_eq_front;
  auto kept_of = [&](long long n_eq, long long seen) {    // of n_eq ties behind `seen` others
    const long long k = eq_kept - seen;
    return k < 0 ? 0 : k > n_eq ? n_eq : k;
  };
  const u64 mass_total = s_mass_total + (u64)eq_kept * w_star;
  const u64 mass_before = warp_mass[warp] + s_mass_front + (u64)kept_of(eq_before, 0) * w_star;
  const u64 mass_warp = w_warp + (u64)kept_of(eq_warp, eq_before) * w_star;

  // ---- 4. the draw: u in [0, 1) with 32 bits, target = floor(u * nucleus mass) < nucleus mass ----
  const u64 target = __umul64hi(mass_total, (u64)r << 32);
  // one warp of one CTA has the target in its run; an empty nucleus has no such warp: the first one stands in
  bool found = mass_warp > 0 && mass_before <= target && target < mass_before + mass_warp;
  bool stand_in = mass_total == 0 && rank == 0 && warp == 0;
  if (s_any_odd) {                          // masses may have wrapped: any number of warps may have it, the first takes it
    if (found && lane == 0) atomicMin(&s_first, warp);
    __syncthreads();
    if constexpr (kCtas > 1) cluster_barrier();
    const int first = lane >= kCtas ? kTopPWarps : kCtas == 1 || lane == (int)rank ? s_first : ld_peer(&s_first, (uint32_t)lane);
    const unsigned ctas = __ballot_sync(kFullMask, first < kTopPWarps);
    const int cta = ctas ? __ffs(ctas) - 1 : 0, its = __shfl_sync(kFullMask, first, cta);
    found = ctas && cta == (int)rank && its == warp;
    stand_in = !ctas && rank == 0 && warp == 0;
  }
  if (found || stand_in) {
    long long tok = -1;
    if (found) {
      u64 run = mass_before;
      long long seen = eq_before;
      if (whole) {
#pragma unroll 1
        for (int i = 0; i < listed && !__any_sync(kFullMask, tok >= 0); i += kWarp) {
          bool tie;
          const uint32_t e = entry(i + lane, listed, tie);
          const unsigned ties = __ballot_sync(kFullMask, tie);
          u64 w = rv.weight(__uint_as_float(e << 16)), w_all;
          if (tie) w = seen + __popc(ties & ((1u << lane) - 1u)) < eq_kept ? w_star : 0;
          if (i + lane >= listed) w = 0;
          const u64 mine = run + warp_exclusive_scan<u64>(w, w_all);
          if (w > 0 && mine <= target && target < mine + w) tok = first + (e >> 16);
          run += w_all;
          seen += __popc(ties);
        }
      } else {
        rounds([&](int it, const Group& g) {
          if (__any_sync(kFullMask, tok >= 0)) return;
          const uint32_t in = at_least(it, g);
          u64 w, w_all;
          int ties, ties_all;
          weigh(g, in, w, ties);
          const int ties_front = warp_exclusive_scan<int>(ties, ties_all);
          w += (u64)kept_of(ties, seen + ties_front) * w_star;
          u64 mine = run + warp_exclusive_scan<u64>(w, w_all);
          if (w > 0 && mine <= target && target < mine + w) {
            long long eq_seen = seen + ties_front;
#pragma unroll 1
            for (int j = 0; j < kGroup && tok < 0; ++j) {
              const uint32_t u = bits_of(g, j);
              bool mine_too = in >> j & 1u;
              if (mine_too && order(u) <= star) { mine_too = eq_seen < eq_kept; ++eq_seen; }
              if (mine_too) {
                mine += rv.weight(__uint_as_float(u << 16));
                if (mine > target) tok = first + it * round + lane * group + j;
              }
            }
          }
          run += w_all;
          seen += ties_all;
        });
      }
      // one lane has it (of an odd row any number: the first of them, or the first entry of the warp)
      const unsigned who = __ballot_sync(kFullMask, tok >= 0);
      if (who == 0 && lane == 0) tok = first;
      if (who != 0 && lane != __ffs(who) - 1) tok = -1;
    } else if (lane == 0) {
      // of the first entries of the row, as many as a thread of the kernel above walks: the one that passes the target, or the last
      // of the nucleus
      tok = 0;
      long long eq_seen = 0;
      u64 run = 0;
#pragma unroll 1
      for (long long i = 0; i < stand_in_run && i < vocab; ++i) {
        const uint32_t u = row_bits[i], key = bits_key(u);
        bool in = all_kept || key > key_star;
        if (!in && key == key_star) { in = eq_seen < eq_kept; ++eq_seen; }
        if (!in) continue;
        tok = i;
        run += rv.weight(__uint_as_float(u << 16));
        if (run > target) break;
      }
    }
    if (tok >= 0) {                                       // one lane
      if (out_tokens && steps) {
        if (step >= 0 && step < out_cols) out_tokens[b * out_stride + step] = tok;
        steps[b] = step + 1;
      } else if (out_tokens) {
        out_tokens[b * out_stride] = tok;
      }
      if (next_input) next_input[b] = tok;
      if (positions) positions[b] += 1;
      if (seq_lens) seq_lens[b] += 1;
      if (nucleus_mass) nucleus_mass[b] = Z > 0 ? (float)((double)mass_total / (double)Z) : 0.f;
    }
  }
  if (nucleus_count && tid == 0 && rank == 0) nucleus_count[b] = (int)(s_over_total + eq_kept);
  if constexpr (kCtas > 1) cluster_barrier();   // no CTA leaves while a peer may still read its shared memory
}

// CTAs per row, and whether keys are counted.
struct TopPForm { int ctas; bool counts; int mass_ctas; };
TopPForm top_p_form(long long rows, long long vocab) {
  const int sms = sm_count();
  // Small batches: a cluster of CTAs per row, as many (8, 4, 2) as still run all at once, so that the batch covers
  // the device (64 rows: 128 SMs; one row: 8).  A 148-SM part holds 15 clusters of 8, 33 of 4 or 74 of 2 of these
  // CTAs at a time (cudaOccupancyMaxActiveClusters); the bounds scale with the SM count.
  const int mass_ctas = sms <= 0 ? 1 : rows * 148 <= 15LL * sms ? 8 : rows * 148 <= 33LL * sms ? 4 : 2 * rows <= sms ? 2 : 1;
  // By counts while the counts of a CTA's share of the row fit 16 bits: more CTAs per row where that takes more of them.  Longer rows
  // yet, or a device without the shared memory: by masses.  So are short rows of one CTA each: clearing and summing 65 536 counts took longer than
  // the passes over the row before the nucleus was listed (75 rows, by masses and by counts: 1000 logits 11.4 and 13.8 us, 4096 13.5 and
  // 13.8).  In chains, with the lists: 500 logits 10.6 and 9.8, 1000 9.9 and 9.8, 2000 10.5 and 9.8, 4096 12.0 and 10.0, 8000 15.2 and 9.9: the line
  // is kept, and could be 0.
  const long long groups = (vocab + kVecElems - 1) / kVecElems;
  int ctas = mass_ctas;
  while (ctas < 8 && (groups + ctas - 1) / ctas > kMaxShare) ctas *= 2;
  const bool counts = (groups + ctas - 1) / ctas <= kMaxShare && (ctas > 1 || vocab > kFewLogits) && (sms <= 0 || max_smem_optin() >= kCountSmem + 8192);
  return {counts ? ctas : mass_ctas, counts, mass_ctas};
}
// Errors of a launch whose cluster (or CTA) the device, or the part of it that this process has, cannot hold.
bool not_placed(cudaError_t e) {
  return e == cudaErrorInvalidClusterSize || e == cudaErrorLaunchOutOfResources || e == cudaErrorInvalidConfiguration;
}

}  // namespace
}  // namespace l3ci

extern "C" int l3ci_top_p_kernel_choice(int64_t rows, int64_t vocab) {
  if (rows <= 0 || vocab <= 0) return -1;
  const l3ci::TopPForm f = l3ci::top_p_form(rows, vocab);
  return f.ctas + (f.counts ? 16 : 0);
}

extern "C" int l3ci_top_p_step(const void* logits, int64_t rows, int64_t vocab, int64_t row_stride, float temperature,
                               float top_p, uint64_t seed, int64_t* out_tokens, int64_t out_stride, int64_t out_cols,
                               int64_t* steps, int64_t* next_input, int32_t* positions, int32_t* seq_lens,
                               int32_t* nucleus_count, float* nucleus_mass, l3ci_stream_t stream_) {
  using namespace l3ci;
  clear_error();
  if (rows < 0 || vocab <= 0 || row_stride < vocab) return fail(L3CI_ERR_INVALID, "top_p_step: bad size");
  if (!(temperature > 0.f)) return fail(L3CI_ERR_INVALID, "top_p_step: temperature must be positive (use l3ci_greedy_step for 0)");
  if (!(top_p > 0.f)) return fail(L3CI_ERR_INVALID, "top_p_step: top_p must be positive");
  if (rows == 0) return L3CI_OK;
  if (!logits || (!out_tokens && !next_input)) return fail(L3CI_ERR_INVALID, "top_p_step: null logits or no output");
  if (rows > 0x7fffffffLL) return fail(L3CI_ERR_INVALID, "top_p_step: too many rows");
  if (steps && (!out_tokens || out_cols <= 0)) return fail(L3CI_ERR_INVALID, "top_p_step: steps needs out_tokens and its width");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  const auto lp = static_cast<const __nv_bfloat16*>(logits);
  const float inv_t = 1.0f / temperature;
  auto launch = [&](auto kernel, int c, int smem, auto... more) {
    static bool configured[64][9] = {};   // by device and CTAs per row
    int dev = 0;
    if (smem > 0 && (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !configured[dev][c])) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) configured[dev][c] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(c * rows));
    cfg.blockDim = dim3(kTopPBlock);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (c > 1) {
      attr[n].id = cudaLaunchAttributeClusterDimension;
      attr[n].val.clusterDim.x = (unsigned)c;
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
    return cudaLaunchKernelEx(&cfg, kernel, lp, (long long)vocab, (long long)row_stride, inv_t, top_p, (unsigned long long)seed,
                              reinterpret_cast<long long*>(out_tokens), (long long)out_stride, (long long)out_cols,
                              reinterpret_cast<long long*>(steps), reinterpret_cast<long long*>(next_input), positions, seq_lens,
                              nucleus_count, nucleus_mass, more...);
  };
  const TopPForm form = top_p_form(rows, vocab);
  auto failed = [](cudaError_t e) { return fail(L3CI_ERR_CUDA, "launch of the top_p_step kernel failed: %s", cudaGetErrorString(e)); };
  if (form.counts) {
    const long long walkers = (long long)kTopPBlock * form.mass_ctas, run = ((vocab + walkers - 1) / walkers + kVecElems - 1) / kVecElems * kVecElems;
    auto counts = [&](auto kernel) { return launch(kernel, form.ctas, kCountSmem, run); };
    const cudaError_t e = form.ctas == 8 ? counts(top_p_count_kernel<8>) : form.ctas == 4 ? counts(top_p_count_kernel<4>)
                          : form.ctas == 2 ? counts(top_p_count_kernel<2>) : counts(top_p_count_kernel<1>);
    if (e == cudaSuccess) return L3CI_OK;
    (void)cudaGetLastError();
    if (!not_placed(e)) return failed(e);
  }
  // (a cluster size the device or its partition cannot place falls back to the next smaller one)
  for (int c = form.mass_ctas; c > 1; c /= 2) {
    const cudaError_t e = c == 8 ? launch(top_p_step_kernel<8>, 8, 0) : c == 4 ? launch(top_p_step_kernel<4>, 4, 0) : launch(top_p_step_kernel<2>, 2, 0);
    if (e == cudaSuccess) return L3CI_OK;
    (void)cudaGetLastError();
    if (!not_placed(e)) return failed(e);
  }
  L3CI_LAUNCH("top_p_step_kernel", top_p_step_kernel<1>, dim3((unsigned)rows), dim3(kTopPBlock), 0, stream,
              lp, (long long)vocab, (long long)row_stride, inv_t, top_p, (unsigned long long)seed,
              reinterpret_cast<long long*>(out_tokens), (long long)out_stride, (long long)out_cols, reinterpret_cast<long long*>(steps),
              reinterpret_cast<long long*>(next_input), positions, seq_lens, nucleus_count, nucleus_mass);
  return L3CI_OK;
}
