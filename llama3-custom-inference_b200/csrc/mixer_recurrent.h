// Shared by the kernels of the linear recurrences.
#pragma once

#include "../../include/l3ci_mixers.h"
#include "host_common.h"
#include "mixer_types.cuh"

namespace l3ci {

// The scan by chunks of 16 tokens (mixer_recurrent_chunk.cu): bytes of scratch that it takes for these arguments (already validated), 0 where
// it does not apply or the scan token by token is the faster; its launch, without the heads' norm and gate.
size_t scan_chunks_scratch(const l3ci_recurrent_scan_args* a);
int scan_chunks_launch(const l3ci_recurrent_scan_args* a, void* scratch, size_t bytes);
// The device word where its waits that ran out are recorded (of the current device); null without a device.
int* scan_chunks_wait_status();

#if defined(__CUDACC__)
// The convolution's carried inputs: row r of the tail becomes the input of token T - (taps - 1) + r.  Channel c of a sequence,
// by one thread.
template <typename S>
__device__ __forceinline__ void move_tail(const l3ci_recurrent_scan_args& a, S* tail, const S* in, long long channels, long long c, bool fresh) {
  const int rows = a.taps - 1;
  for (int r = 0; r < rows; ++r) {
    const int t = a.T - rows + r;
    tail[r * channels + c] = t >= 0 ? in[t * a.conv_st + c] : fresh ? from_f32<S>(0.f) : tail[(r + a.T) * channels + c];
  }
}

// Those of head h's values and, by the first head that reads them, of its queries and keys; `i` of `n` threads.
template <typename S>
__device__ __forceinline__ void move_tails(const l3ci_recurrent_scan_args& a, int b, int h, int i, int n, bool fresh) {
  const int GD = a.G * a.D, R = a.H / a.G;
  const long long channels = 2LL * GD + (long long)a.H * a.V;
  S* tail = static_cast<S*>(a.tail) + b * a.tail_sb;
  const S* in = static_cast<const S*>(a.conv_in) + (long long)b * a.T * a.conv_st;
  for (int c = i; c < a.V; c += n) move_tail<S>(a, tail, in, channels, 2LL * GD + (long long)h * a.V + c, fresh);
  if (h % R == 0)
    for (int c = i; c < 2 * a.D; c += n) move_tail<S>(a, tail, in, channels, c < a.D ? (h / R) * a.D + c : GD + (h / R) * a.D + c - a.D, fresh);
}
#endif

}  // namespace l3ci
