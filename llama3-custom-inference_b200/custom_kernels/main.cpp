// Torch extension module `custom_kernels_extension`: the drop-in boundary.
//
// Exports the three functions the reference binds in custom_kernels/main.cpp:2-8
//   flash_attention_decode(query, keys, values) -> Tensor      (model.py:118, benchmark_kernel.py:25)
//   rms_norm(input, weight, eps) -> Tensor                     (model.py:71)
//   rot_embed(input, freq) -> Tensor                           (model.py:100-101)
// with the same positional signatures, return conventions (a freshly allocated tensor shaped
// like the input) and error type (RuntimeError through TORCH_CHECK), and adds keyword-only
// extras plus new functions; nothing here computes: every call validates its tensors, takes the
// device of the input and torch's current stream (the reference launches on the legacy default
// stream of whatever device is current, custom_kernels/custom_kernels.cu:274-275,386,439) and
// forwards raw pointers to the C ABI of include/l3ci_b200.h.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContextLight.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <map>
#include <mutex>
#include <optional>
#include <tuple>
#include <utility>

#include "l3ci_b200.h"

namespace {

using torch::Tensor;

l3ci_stream_t current_stream() {
  return reinterpret_cast<l3ci_stream_t>(c10::cuda::getCurrentCUDAStream().stream());
}

void check_status(int status, const char* what) {
  TORCH_CHECK(status == L3CI_OK, what, ": ", l3ci_status_string(status), " (", l3ci_last_error(), ")");
}

void check_bf16_cuda(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(t.scalar_type() == torch::kBFloat16, name, " must be bfloat16, got ", t.scalar_type());
}

// Scratch of the flash-decode kernel, one buffer per (device, stream), zero-filled when it is
// created and reused by later calls (the kernel leaves it ready).  The reference allocates its
// three scratch tensors on every call (custom_kernels/custom_kernels.cu:269-271).
struct Workspace {
  Tensor buf;
};
std::mutex g_ws_mutex;
std::map<std::pair<int, int64_t>, Workspace>& workspaces() {
  static auto* m = new std::map<std::pair<int, int64_t>, Workspace>();  // never destroyed: outlives CUDA teardown
  return *m;
}

Tensor& workspace_for(const Tensor& like, size_t bytes) {
  const auto stream = c10::cuda::getCurrentCUDAStream();
  const auto key = std::make_pair((int)like.get_device(), (int64_t)stream.id());
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  auto& all = workspaces();
  if (all.size() >= 16 && all.find(key) == all.end()) {
    // streams come and go (graph captures, side streams): the buffers of other streams are dropped rather than
    // kept for the life of the process; a stream that comes back gets a fresh zero-filled one
    for (auto it = all.begin(); it != all.end();) it = it->first.first == key.first ? all.erase(it) : std::next(it);
  }
  Workspace& ws = all[key];
  if (!ws.buf.defined() || (size_t)ws.buf.numel() < bytes) {
    ws.buf = torch::zeros({(int64_t)bytes}, torch::dtype(torch::kUInt8).device(like.device()));
  }
  return ws.buf;
}

struct DecodeShapes {
  int B, Hq, Hkv, D, n_seq;
};

DecodeShapes check_decode_inputs(const Tensor& q, const Tensor& k, const Tensor& v,
                                 const std::optional<Tensor>& seq_lens) {
  check_bf16_cuda(q, "query");
  check_bf16_cuda(k, "keys");
  check_bf16_cuda(v, "values");
  TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && v.dim() == 4, "query, keys, values must be 4-D [B, H, T, D]");
  TORCH_CHECK(q.size(2) == 1, "flash_attention_decode takes one query token per sequence, got ", q.size(2));
  TORCH_CHECK(k.sizes() == v.sizes(), "keys and values must have the same shape");
  TORCH_CHECK(k.size(0) == q.size(0) && k.size(3) == q.size(3), "batch / head size of query and keys differ");
  TORCH_CHECK(k.get_device() == q.get_device() && v.get_device() == q.get_device(), "inputs on different devices");
  TORCH_CHECK(q.stride(3) == 1 && k.stride(3) == 1 && v.stride(3) == 1, "last dimension must be contiguous");
  if (seq_lens) {
    TORCH_CHECK(seq_lens->is_cuda() && seq_lens->scalar_type() == torch::kInt32 && seq_lens->dim() == 1 &&
                    seq_lens->size(0) == q.size(0) && seq_lens->is_contiguous(),
                "seq_lens must be a contiguous int32 CUDA tensor of shape [B]");
  }
  DecodeShapes s;
  s.B = (int)q.size(0);
  s.Hq = (int)q.size(1);
  s.Hkv = (int)k.size(1);
  s.n_seq = (int)k.size(2);
  s.D = (int)q.size(3);
  TORCH_CHECK(s.D == 64 || s.D == 128, "Unsupported head size for splitkv kernel: ", s.D);
  TORCH_CHECK(s.Hkv > 0 && s.Hq % s.Hkv == 0 && s.Hq / s.Hkv <= 16,
              "Unsupported QKV head ratio for splitkv kernel: ", s.Hq, "/", s.Hkv);
  return s;
}

void run_decode(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& seq_lens,
                Tensor* out, Tensor* o_partial, Tensor* lse, double scale, int64_t max_ctas,
                const DecodeShapes& s) {
  l3ci_flash_decode_args a{};
  a.q = q.data_ptr();
  a.k = k.data_ptr();
  a.v = v.data_ptr();
  a.out = out ? out->data_ptr() : nullptr;
  a.o_partial = o_partial ? o_partial->data_ptr<float>() : nullptr;
  a.lse = lse ? lse->data_ptr<float>() : nullptr;
  a.seq_lens = seq_lens ? seq_lens->data_ptr<int32_t>() : nullptr;
  a.B = s.B; a.Hq = s.Hq; a.Hkv = s.Hkv; a.D = s.D; a.n_seq = s.n_seq;
  a.q_sb = q.stride(0); a.q_sh = q.stride(1);
  a.k_sb = k.stride(0); a.k_sh = k.stride(1); a.k_st = k.stride(2);
  a.v_sb = v.stride(0); a.v_sh = v.stride(1); a.v_st = v.stride(2);
  if (out) { a.o_sb = out->stride(0); a.o_sh = out->stride(1); }
  a.scale = (float)scale;
  a.max_ctas = (int32_t)max_ctas;
  a.stream = current_stream();
  const size_t need = l3ci_flash_decode_scratch_bytes(s.B, s.Hq, s.Hkv, s.D);
  Tensor& ws = workspace_for(q, need);
  a.scratch = ws.data_ptr();
  a.scratch_bytes = (size_t)ws.numel();
  check_status(l3ci_flash_decode(&a), "flash_attention_decode");
}

// reference: custom_kernels/custom_kernels.cu:233-338
Tensor flash_attention_decode(Tensor query, Tensor keys, Tensor values, std::optional<Tensor> seq_lens,
                              std::optional<Tensor> out, double scale, int64_t max_ctas) {
  const DecodeShapes s = check_decode_inputs(query, keys, values, seq_lens);
  const c10::cuda::CUDAGuard guard(query.device());
  Tensor result = out ? *out : torch::empty_like(query);
  if (out) {
    check_bf16_cuda(result, "out");
    TORCH_CHECK(result.sizes() == query.sizes() && result.stride(3) == 1, "out must be shaped like query");
  }
  if (s.B == 0) return result;
  run_decode(query, keys, values, seq_lens, &result, nullptr, nullptr, scale, max_ctas, s);
  return result;
}

// Attention over a slice of the cached sequence, returned as fp32 (o, lse) for lse_merge.
// `out_o` / `out_lse` (contiguous fp32 [B,Hq,D] / [B,Hq]) let the caller choose where the result lands, e.g. in
// its slot of an exchange buffer that peers can address.
std::tuple<Tensor, Tensor> flash_attention_decode_partial(Tensor query, Tensor keys, Tensor values,
                                                          std::optional<Tensor> seq_lens, double scale,
                                                          int64_t max_ctas, std::optional<Tensor> out_o,
                                                          std::optional<Tensor> out_lse) {
  const DecodeShapes s = check_decode_inputs(query, keys, values, seq_lens);
  const c10::cuda::CUDAGuard guard(query.device());
  auto f32 = torch::dtype(torch::kFloat32).device(query.device());
  TORCH_CHECK(out_o.has_value() == out_lse.has_value(), "out_o and out_lse go together");
  if (out_o) {
    TORCH_CHECK(out_o->is_cuda() && out_o->scalar_type() == torch::kFloat32 && out_o->is_contiguous() &&
                    out_o->numel() == (int64_t)s.B * s.Hq * s.D && out_lse->is_cuda() &&
                    out_lse->scalar_type() == torch::kFloat32 && out_lse->is_contiguous() &&
                    out_lse->numel() == (int64_t)s.B * s.Hq && out_o->get_device() == query.get_device() &&
                    out_lse->get_device() == query.get_device(),
                "out_o / out_lse must be contiguous fp32 CUDA tensors of B*Hq*D / B*Hq elements");
  }
  Tensor o = out_o ? *out_o : torch::empty({s.B, s.Hq, s.D}, f32);
  Tensor lse = out_lse ? *out_lse : torch::empty({s.B, s.Hq}, f32);
  if (s.B == 0) return {o, lse};
  run_decode(query, keys, values, seq_lens, nullptr, &o, &lse, scale, max_ctas, s);
  return {o, lse};
}

// Causal attention for T > 1 new tokens (model.py:114-116 sends this case to torch's SDPA): query [B,Hq,T,D],
// keys / values [B,Hkv,S,D] (views of the cache are fine), query t sees keys j <= start_pos + t.  Returns a tensor
// laid out like `query`.
Tensor prefill_attention(Tensor query, Tensor keys, Tensor values, int64_t start_pos, double scale, int64_t variant) {
  check_bf16_cuda(query, "query");
  check_bf16_cuda(keys, "keys");
  check_bf16_cuda(values, "values");
  TORCH_CHECK(query.dim() == 4 && keys.dim() == 4 && values.dim() == 4, "query, keys, values must be 4-D");
  TORCH_CHECK(keys.sizes() == values.sizes() && keys.size(0) == query.size(0) && keys.size(3) == query.size(3),
              "shape mismatch between query, keys and values");
  TORCH_CHECK(query.stride(3) == 1 && keys.stride(3) == 1 && values.stride(3) == 1, "last axis must be contiguous");
  TORCH_CHECK(keys.get_device() == query.get_device() && values.get_device() == query.get_device(), "tensors on different devices");
  const int64_t B = query.size(0), Hq = query.size(1), T = query.size(2), D = query.size(3), Hkv = keys.size(1), S = keys.size(2);
  TORCH_CHECK(D == 64 || D == 128, "Unsupported head size for prefill_attention kernel: ", D);
  TORCH_CHECK(Hkv > 0 && Hq % Hkv == 0, "query heads must be a multiple of kv heads");
  TORCH_CHECK(start_pos >= 0 && start_pos + T <= S, "start_pos + T must not exceed the keys given");
  const c10::cuda::CUDAGuard guard(query.device());
  Tensor out = torch::empty_strided(query.sizes(), query.strides(), query.options());
  if (B == 0 || T == 0) return out;
  l3ci_prefill_args a{};
  a.q = query.data_ptr(); a.k = keys.data_ptr(); a.v = values.data_ptr(); a.out = out.data_ptr(); a.status = nullptr;
  a.B = (int32_t)B; a.Hq = (int32_t)Hq; a.Hkv = (int32_t)Hkv; a.D = (int32_t)D;
  a.T = (int32_t)T; a.n_keys = (int32_t)S; a.start_pos = (int32_t)start_pos;
  a.q_sb = query.stride(0); a.q_sh = query.stride(1); a.q_st = query.stride(2);
  a.k_sb = keys.stride(0); a.k_sh = keys.stride(1); a.k_st = keys.stride(2);
  a.v_sb = values.stride(0); a.v_sh = values.stride(1); a.v_st = values.stride(2);
  a.o_sb = out.stride(0); a.o_sh = out.stride(1); a.o_st = out.stride(2);
  a.scale = (float)scale;
  a.variant = (int32_t)variant;
  a.stream = current_stream();
  check_status(l3ci_prefill_attention(&a), "prefill_attention");
  return out;
}

// out[b, h, 0, :] = sum_p softmax_p(lse[p, b, h]) * o[p, b, h, :]
Tensor lse_merge(Tensor o_parts, Tensor lse_parts) {
  TORCH_CHECK(o_parts.is_cuda() && o_parts.scalar_type() == torch::kFloat32 && o_parts.dim() == 4 &&
                  o_parts.is_contiguous(),
              "o_parts must be a contiguous fp32 CUDA tensor [parts, B, Hq, D]");
  TORCH_CHECK(lse_parts.is_cuda() && lse_parts.scalar_type() == torch::kFloat32 && lse_parts.dim() == 3 &&
                  lse_parts.is_contiguous() && lse_parts.size(0) == o_parts.size(0) &&
                  lse_parts.size(1) == o_parts.size(1) && lse_parts.size(2) == o_parts.size(2),
              "lse_parts must be a contiguous fp32 CUDA tensor [parts, B, Hq]");
  const c10::cuda::CUDAGuard guard(o_parts.device());
  const int parts = (int)o_parts.size(0), B = (int)o_parts.size(1), Hq = (int)o_parts.size(2), D = (int)o_parts.size(3);
  // Same memory layout as the reference's result for a [B, 1, Hq, D].transpose(1, 2) query.
  Tensor out = torch::empty({B, 1, Hq, D}, torch::dtype(torch::kBFloat16).device(o_parts.device())).transpose(1, 2);
  check_status(l3ci_lse_merge(o_parts.data_ptr<float>(), lse_parts.data_ptr<float>(), out.data_ptr(), parts, B, Hq,
                              D, out.stride(0), out.stride(1), current_stream()),
               "lse_merge");
  return out;
}

// Exchange of shard results over peer memory fused with their merge (l3ci_lse_exchange_merge).  `bufs` is an
// int64 CUDA tensor [ranks] holding the base addresses of every rank's exchange buffer as this process sees
// them; this rank's own result must already be in its slot of parity epoch & 1.
Tensor lse_exchange_merge(Tensor bufs, int64_t rank, int64_t epoch, int64_t B, int64_t Hq, int64_t D,
                          std::optional<Tensor> status) {
  TORCH_CHECK(bufs.is_cuda() && bufs.scalar_type() == torch::kInt64 && bufs.dim() == 1 && bufs.is_contiguous(),
              "bufs must be a contiguous int64 CUDA tensor of buffer addresses");
  if (status)
    TORCH_CHECK(status->is_cuda() && status->scalar_type() == torch::kInt32 && status->numel() >= 1 &&
                    status->get_device() == bufs.get_device(),
                "status must be an int32 CUDA tensor");
  const c10::cuda::CUDAGuard guard(bufs.device());
  Tensor out = torch::empty({B, 1, Hq, D}, torch::dtype(torch::kBFloat16).device(bufs.device())).transpose(1, 2);
  check_status(l3ci_lse_exchange_merge(reinterpret_cast<void* const*>(bufs.data_ptr<int64_t>()), (int32_t)rank,
                                       (int32_t)bufs.size(0), (uint32_t)epoch, out.data_ptr(), (int32_t)B, (int32_t)Hq,
                                       (int32_t)D, out.stride(0), out.stride(1),
                                       status ? status->data_ptr<int32_t>() : nullptr, current_stream()),
               "lse_exchange_merge");
  return out;
}

// Decode attention over this rank's slice of a sequence-sharded cache, merged with the other ranks' results in the
// same launch (l3ci_flash_decode_exchange).  `bufs`: int64 CUDA tensor [ranks] of the ranks' exchange buffers as this
// process addresses them.  Returns false-y (None) when the sizes go to the kernel without a fused exchange, so that
// the caller can take the two-launch path.
std::optional<Tensor> flash_attention_decode_exchange(Tensor query, Tensor keys, Tensor values, Tensor bufs, int64_t rank,
                                                      int64_t epoch, std::optional<Tensor> seq_lens, std::optional<Tensor> out,
                                                      std::optional<Tensor> status, double scale, int64_t max_ctas) {
  const DecodeShapes s = check_decode_inputs(query, keys, values, seq_lens);
  TORCH_CHECK(bufs.is_cuda() && bufs.scalar_type() == torch::kInt64 && bufs.dim() == 1 && bufs.is_contiguous() &&
                  bufs.get_device() == query.get_device(),
              "bufs must be a contiguous int64 CUDA tensor of buffer addresses on the device of the inputs");
  if (status)
    TORCH_CHECK(status->is_cuda() && status->scalar_type() == torch::kInt32 && status->numel() >= 1 &&
                    status->get_device() == query.get_device(),
                "status must be an int32 CUDA tensor");
  const c10::cuda::CUDAGuard guard(query.device());
  Tensor result = out ? *out : torch::empty_like(query);
  if (out) {
    check_bf16_cuda(result, "out");
    TORCH_CHECK(result.sizes() == query.sizes() && result.stride(3) == 1, "out must be shaped like query");
  }
  if (s.B == 0) return result;
  l3ci_flash_decode_args a{};
  a.q = query.data_ptr(); a.k = keys.data_ptr(); a.v = values.data_ptr(); a.out = result.data_ptr();
  a.seq_lens = seq_lens ? seq_lens->data_ptr<int32_t>() : nullptr;
  a.B = s.B; a.Hq = s.Hq; a.Hkv = s.Hkv; a.D = s.D; a.n_seq = s.n_seq;
  a.q_sb = query.stride(0); a.q_sh = query.stride(1);
  a.k_sb = keys.stride(0); a.k_sh = keys.stride(1); a.k_st = keys.stride(2);
  a.v_sb = values.stride(0); a.v_sh = values.stride(1); a.v_st = values.stride(2);
  a.o_sb = result.stride(0); a.o_sh = result.stride(1);
  a.scale = (float)scale;
  a.max_ctas = (int32_t)max_ctas;
  a.stream = current_stream();
  const int st = l3ci_flash_decode_exchange(&a, reinterpret_cast<void* const*>(bufs.data_ptr<int64_t>()), (int32_t)rank,
                                            (int32_t)bufs.size(0), (uint32_t)epoch, status ? status->data_ptr<int32_t>() : nullptr);
  if (st == L3CI_ERR_UNSUPPORTED) return std::nullopt;
  check_status(st, "flash_attention_decode_exchange");
  return result;
}

// reference: custom_kernels/custom_kernels.cu:369-389
Tensor rms_norm(Tensor input, Tensor weight, double eps) {
  check_bf16_cuda(input, "input");
  check_bf16_cuda(weight, "weight");
  TORCH_CHECK(input.dim() >= 1 && weight.dim() == 1 && weight.size(0) == input.size(-1),
              "weight must have the size of the last input dimension");
  TORCH_CHECK(weight.get_device() == input.get_device(), "input and weight on different devices");
  const c10::cuda::CUDAGuard guard(input.device());
  const int64_t E = input.size(-1);
  Tensor x = input.is_contiguous() ? input : input.contiguous();
  Tensor w = weight.is_contiguous() ? weight : weight.contiguous();
  Tensor out = torch::empty_like(x);
  const int64_t rows = E ? x.numel() / E : 0;
  check_status(l3ci_rms_norm(x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, E, E, E, (float)eps, current_stream()),
               "rms_norm");
  return out;
}

// (x + residual) and its RMSNorm in one pass: returns (sum, normed).  model.py:147-148 as one kernel.
std::tuple<Tensor, Tensor> add_rms_norm(Tensor x, Tensor residual, Tensor weight, double eps) {
  check_bf16_cuda(x, "x");
  check_bf16_cuda(residual, "residual");
  check_bf16_cuda(weight, "weight");
  TORCH_CHECK(x.sizes() == residual.sizes() && weight.dim() == 1 && weight.size(0) == x.size(-1), "shape mismatch");
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor xc = x.contiguous(), rc = residual.contiguous(), w = weight.contiguous();
  Tensor sum = torch::empty_like(xc), out = torch::empty_like(xc);
  const int64_t E = xc.size(-1);
  check_status(l3ci_add_rms_norm(xc.data_ptr(), rc.data_ptr(), w.data_ptr(), sum.data_ptr(), out.data_ptr(),
                                 E ? xc.numel() / E : 0, E, (float)eps, current_stream()),
               "add_rms_norm");
  return {sum, out};
}

// silu(gate) * up with the roundings of the two bf16 tensor ops it replaces (model.py:134).
Tensor silu_mul(Tensor gate, Tensor up) {
  check_bf16_cuda(gate, "gate");
  check_bf16_cuda(up, "up");
  TORCH_CHECK(gate.sizes() == up.sizes(), "gate and up must have the same shape");
  TORCH_CHECK(gate.dim() >= 1, "gate must have at least one dimension");
  const c10::cuda::CUDAGuard guard(gate.device());
  // rows of a [..., 2F] GEMM result split in halves stay in place: only the last axis must be contiguous
  const int64_t cols = gate.size(-1);
  auto rows2d = [&](const Tensor& t) {
    Tensor f = t.dim() == 2 ? t : t.reshape({-1, cols});  // a view whenever the leading axes collapse
    return f.stride(-1) == 1 ? f : f.contiguous();
  };
  Tensor g = rows2d(gate), u = rows2d(up);
  Tensor out = torch::empty(gate.sizes(), gate.options());
  check_status(l3ci_silu_mul(g.data_ptr(), u.data_ptr(), out.data_ptr(), g.size(0), cols, g.stride(0), u.stride(0),
                             current_stream()),
               "silu_mul");
  return out;
}

// Whether the kernel for few rows is taken where torch's product could be.  A CTA reads its rows of x anew for every tile of w and
// writes the results token by token, so it falls behind as rows / K grows.  Measured in chains, us (torch's) at 16, 32, 48, 64 rows: w
// 2048 x 2048 4.6 (5.6), 5.3 (5.6), 6.0 (5.7), 6.8 (5.7); 2048 x 8192 9.9 (13.4), 10.6 (13.3), 11.6 (13.5), 12.3 (13.7); 2048 x 128
// 3.2 (2.4), 5.3 (2.4), 6.7 (2.4), 7.9 (2.6).  Without `early` it is about 1 us slower.  Few outputs (4 x 2048: 5.2 (12.2) at 64 rows)
// and very many (128256 x 2048: 88 (95)) are its own at any number of rows, and so are fused activations, which it applies to sums
// that are not rounded to bf16: gated 2 x 8192 x 2048 14.1 (15.8), 15.0 (15.6), 15.6 (16.3), 16.3 (15.9); gelu 8192 x 2048 8.8 (10.7),
// 9.9 (10.9), 11.0 (11.4), 12.1 (11.5).
bool few_rows_pay(int64_t rows, int64_t K, int64_t N, int64_t groups, int64_t act, bool early) {
  return act != L3CI_ACT_NONE || rows <= (early ? 16 : 8) || rows <= K / (early ? 64 : 128) || N * groups <= 256 || N >= 32768;
}

// act(x w^T) of few rows in one kernel (l3ci_linear): x [..., K] with w [N, K] (gated: [2 N, K], gate rows, then up rows), or groups
// of products, x [groups, rows, K] with w [groups, N, K].  Nothing where that kernel does not apply (more rows, other types, layouts
// or alignments) or torch's product is the faster on the device (few_rows_pay).  `early`: the kernel may read w ahead of the stream's previous kernels; for a w that was complete before the last
// one of them that waits for its predecessors ahead of letting others start.  f32: an fp32 result.  `into`: where the result goes.
// `always`: wherever the kernel applies; for passes that wait for the host, which a launch of it costs about 4 us less than torch's
// product (a prompt of 64 tokens, 16 layers: 1.0 ms instead of 1.4).  `limit`, `alpha`: of a gated activation's clamped form.
std::optional<Tensor> few_rows(const Tensor& x, const Tensor& w, int64_t act, bool early, bool f32, const std::optional<Tensor>& into, bool always,
                               double limit, double alpha) {
  if (!x.is_cuda() || !w.is_cuda() || x.scalar_type() != torch::kBFloat16 || w.scalar_type() != torch::kBFloat16 ||
      w.get_device() != x.get_device() || x.dim() < 1)
    return std::nullopt;
  const bool grouped = w.dim() == 3, gated = act == L3CI_ACT_SILU_GATE;
  const int64_t K = x.size(-1);
  if ((w.dim() != 2 && !grouped) || w.size(-1) != K || (grouped && (x.dim() != 3 || x.size(0) != w.size(0)))) return std::nullopt;
  const int64_t groups = grouped ? w.size(0) : 1, rows = K * groups ? x.numel() / (K * groups) : 0;
  if (rows == 0 || rows > L3CI_LINEAR_MAX_ROWS || K % 8 || (gated && w.size(-2) % 2)) return std::nullopt;
  const int64_t N = gated ? w.size(-2) / 2 : w.size(-2);
  if (!always && !few_rows_pay(rows, K, N, groups, act, early)) return std::nullopt;
  auto at16 = [](const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; };
  if (N == 0 || K > INT32_MAX || w.size(-2) > INT32_MAX || groups > INT32_MAX || !w.is_contiguous() || !at16(x) || !at16(w)) return std::nullopt;
  auto row_stride = [&](const Tensor& t) {
    const int64_t* sizes = t.sizes().data() + (grouped ? 1 : 0);
    return l3ci_row_stride(sizes, t.strides().data() + (grouped ? 1 : 0), (int32_t)t.dim() - (grouped ? 1 : 0));
  };
  const int64_t stride = row_stride(x), group_stride = grouped ? x.stride(0) : 0;
  if (stride < 0 || stride % 8 || group_stride % 8 || (groups > 1 && group_stride <= 0)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(x.device());
  auto sizes = x.sizes().vec();
  sizes.back() = N;
  Tensor out;
  if (into) {
    out = *into;
    TORCH_CHECK(out.is_cuda() && out.get_device() == x.get_device() && out.sizes() == torch::IntArrayRef(sizes) &&
                    (out.scalar_type() == torch::kBFloat16 || out.scalar_type() == torch::kFloat) && row_stride(out) > 0 &&
                    (groups == 1 || out.stride(0) > 0),
                "the result's type, shape, device or strides");
  } else {
    out = torch::empty(sizes, x.options().dtype(f32 ? torch::kFloat : torch::kBFloat16));
  }
  l3ci_linear_args a{};
  a.x = x.data_ptr(); a.w = w.data_ptr(); a.out = out.data_ptr();
  a.rows = rows; a.x_st = stride; a.out_st = row_stride(out); a.x_sg = group_stride; a.out_sg = grouped ? out.stride(0) : 0;
  a.K = (int32_t)K; a.N = (int32_t)N; a.groups = (int32_t)groups; a.act = (int32_t)act;
  a.out_f32 = out.scalar_type() == torch::kFloat;
  a.early = early;
  a.stream = current_stream();
  check_status(l3ci_linear_gated(&a, (float)limit, (float)alpha), "linear");
  return out;
}

// Whether a product of many rows with its activation is the faster by l3ci_linear_many, tiles of 256 x 256 on pairs of SMs, than by torch's
// product and a pass for the activation: where there are tiles for more than one wave of pairs and the last wave is not nearly empty.  Both
// in turn, us: gated 2 x 8192 x 2048, rows 256 19.9 and 19.5, 512 30.8 and 29.0, 2048 128 and 98.6, 6001 362 and 304, 8192 495 and 413; gelu
// 8192 x 2048, rows 512 21.5 and 22.9, 1024 48.2 and 44.2, 2048 69.3 and 59.5, 8192 301 and 226.  (Without an activation it is the library's
// equal at best: 8192 rows 215 and 208, 2048 rows 48.7 and 51.3.)
bool many_rows_pay(int64_t rows, int64_t N, bool gated, int sms) {
  const int64_t outs = gated ? 128 : 256, tiles = (rows + 255) / 256 * ((N + outs - 1) / outs), pairs = sms / 2;
  const int64_t waves = (tiles + pairs - 1) / pairs;
  return pairs > 0 && 2 * tiles >= 3 * pairs && 20 * tiles >= 17 * waves * pairs;
}

// act(x w^T) of many rows in one kernel (l3ci_linear_many); nothing where it does not apply or does not pay.
std::optional<Tensor> many_rows(const Tensor& x, const Tensor& w, int64_t act) {
  if (!x.is_cuda() || !w.is_cuda() || x.scalar_type() != torch::kBFloat16 || w.scalar_type() != torch::kBFloat16 ||
      w.get_device() != x.get_device() || x.dim() < 1 || w.dim() != 2 || act == L3CI_ACT_NONE)
    return std::nullopt;
  const bool gated = act == L3CI_ACT_SILU_GATE || act == L3CI_ACT_SILU_MUL;
  const int64_t K = x.size(-1), N = gated ? w.size(0) / 2 : w.size(0), rows = K ? x.numel() / K : 0;
  if (w.size(1) != K || K % 8 || N == 0 || N % 8 || (gated && w.size(0) % 2) || !w.is_contiguous() || rows > INT32_MAX || K > INT32_MAX || w.size(0) > INT32_MAX ||
      !many_rows_pay(rows, N, gated, at::cuda::getDeviceProperties(x.get_device())->multiProcessorCount))
    return std::nullopt;
  auto at16 = [](const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; };
  const int64_t stride = l3ci_row_stride(x.sizes().data(), x.strides().data(), (int32_t)x.dim());
  if (stride < 0 || stride % 8 || !at16(x) || !at16(w)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(x.device());
  auto sizes = x.sizes().vec();
  sizes.back() = N;
  Tensor out = torch::empty(sizes, x.options());
  l3ci_linear_args a{};
  a.x = x.data_ptr(); a.w = w.data_ptr(); a.out = out.data_ptr();
  a.rows = rows; a.x_st = stride; a.out_st = N;
  a.K = (int32_t)K; a.N = (int32_t)N; a.groups = 1; a.act = (int32_t)act;
  a.stream = current_stream();
  check_status(l3ci_linear_many(&a), "linear_many");
  return out;
}

// act(x w^T) of any number of rows: few in one kernel (few_rows), many gated ones in another (many_rows), else torch's product and, gated,
// silu_mul.
Tensor linear(Tensor x, Tensor w, bool gated, bool early, bool always) {
  check_bf16_cuda(x, "x");
  check_bf16_cuda(w, "w");
  TORCH_CHECK(x.dim() >= 1 && w.dim() == 2 && w.size(1) == x.size(-1), "w must be [N, K] with K the last axis of x");
  TORCH_CHECK(w.get_device() == x.get_device(), "x and w on different devices");
  TORCH_CHECK(!gated || w.size(0) % 2 == 0, "a gated product takes an even number of rows of w");
  if (auto y = few_rows(x, w, gated ? L3CI_ACT_SILU_GATE : L3CI_ACT_NONE, early, false, std::nullopt, always, 0.0, 0.0)) return *y;
  if (gated)
    if (auto y = many_rows(x, w, L3CI_ACT_SILU_MUL)) return *y;     // (silu_mul's bits)
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y = at::linear(x, w);
  if (!gated) return y;
  const int64_t N = w.size(0) / 2;
  const Tensor gate = y.narrow(-1, 0, N), up = y.narrow(-1, N, N);
  return N > 0 && N % 8 == 0 ? silu_mul(gate, up) : at::mul(at::silu(gate), up);   // (silu_mul takes rows of whole 16-byte vectors)
}

// Greedy decode step in place: argmax of logits [B, vocab] (bf16) per row, token written to out_tokens[b, steps[b]]
// and next_input[b], steps / positions / seq_lens advanced by one.  model.py:370-381 as one kernel.
void greedy_step(Tensor logits, Tensor out_tokens, Tensor steps, Tensor next_input, Tensor positions, Tensor seq_lens) {
  check_bf16_cuda(logits, "logits");
  TORCH_CHECK(logits.dim() == 2 && logits.stride(1) == 1, "logits must be [B, vocab] with a contiguous last axis");
  const int64_t B = logits.size(0);
  auto check = [&](const Tensor& t, at::ScalarType ty, const char* name) {
    TORCH_CHECK(t.is_cuda() && t.device() == logits.device() && t.scalar_type() == ty, name, ": wrong device or dtype");
  };
  check(out_tokens, at::kLong, "out_tokens");
  check(steps, at::kLong, "steps");
  check(next_input, at::kLong, "next_input");
  check(positions, at::kInt, "positions");
  check(seq_lens, at::kInt, "seq_lens");
  TORCH_CHECK(out_tokens.dim() == 2 && out_tokens.size(0) == B && out_tokens.stride(1) == 1, "out_tokens must be [B, G]");
  TORCH_CHECK(steps.numel() == B && next_input.numel() == B && positions.numel() >= B && seq_lens.numel() >= B &&
                  steps.is_contiguous() && next_input.is_contiguous() && positions.is_contiguous() && seq_lens.is_contiguous(),
              "per-sequence state must be contiguous with one entry per row");
  const c10::cuda::CUDAGuard guard(logits.device());
  check_status(l3ci_greedy_step(logits.data_ptr(), B, logits.size(1), logits.stride(0), out_tokens.data_ptr<int64_t>(),
                                out_tokens.stride(0), out_tokens.size(1), steps.data_ptr<int64_t>(),
                                next_input.data_ptr<int64_t>(), positions.data_ptr<int32_t>(), seq_lens.data_ptr<int32_t>(),
                                current_stream()),
               "greedy_step");
}

// Nucleus sampling step in place (model.py:367-369 + sample_top_p, model.py:400-423, + the bookkeeping of
// model.py:373-381): one token per row of logits [B, vocab] (bf16) drawn from the top-p nucleus of
// softmax(logits / temperature); written like greedy_step writes its argmax.
void top_p_step(Tensor logits, Tensor out_tokens, Tensor steps, Tensor next_input, Tensor positions, Tensor seq_lens,
                double temperature, double top_p, int64_t seed) {
  check_bf16_cuda(logits, "logits");
  TORCH_CHECK(logits.dim() == 2 && logits.stride(1) == 1, "logits must be [B, vocab] with a contiguous last axis");
  TORCH_CHECK(temperature > 0 && top_p > 0, "temperature and top_p must be positive (temperature 0: greedy_step)");
  const int64_t B = logits.size(0);
  auto check = [&](const Tensor& t, at::ScalarType ty, const char* name) {
    TORCH_CHECK(t.is_cuda() && t.device() == logits.device() && t.scalar_type() == ty, name, ": wrong device or dtype");
  };
  check(out_tokens, at::kLong, "out_tokens");
  check(steps, at::kLong, "steps");
  check(next_input, at::kLong, "next_input");
  check(positions, at::kInt, "positions");
  check(seq_lens, at::kInt, "seq_lens");
  TORCH_CHECK(out_tokens.dim() == 2 && out_tokens.size(0) == B && out_tokens.stride(1) == 1, "out_tokens must be [B, G]");
  TORCH_CHECK(steps.numel() == B && next_input.numel() == B && positions.numel() >= B && seq_lens.numel() >= B &&
                  steps.is_contiguous() && next_input.is_contiguous() && positions.is_contiguous() && seq_lens.is_contiguous(),
              "per-sequence state must be contiguous with one entry per row");
  const c10::cuda::CUDAGuard guard(logits.device());
  check_status(l3ci_top_p_step(logits.data_ptr(), B, logits.size(1), logits.stride(0), (float)temperature, (float)top_p,
                               (uint64_t)seed, out_tokens.data_ptr<int64_t>(), out_tokens.stride(0), out_tokens.size(1),
                               steps.data_ptr<int64_t>(), next_input.data_ptr<int64_t>(), positions.data_ptr<int32_t>(),
                               seq_lens.data_ptr<int32_t>(), nullptr, nullptr, current_stream()),
               "top_p_step");
}

// reference: custom_kernels/custom_kernels.cu:418-442
Tensor rot_embed(Tensor input, Tensor freq) {
  check_bf16_cuda(input, "input");
  TORCH_CHECK(input.dim() == 4, "input must be [B, S, H, D]");
  TORCH_CHECK(freq.is_cuda() && freq.scalar_type() == torch::kFloat32, "freq must be a float32 CUDA tensor");
  TORCH_CHECK(freq.get_device() == input.get_device(), "input and freq on different devices");
  TORCH_CHECK(freq.numel() >= input.size(1) * input.size(3), "freq must hold [S, D] values");
  TORCH_CHECK(input.stride(3) == 1, "last dimension must be contiguous");
  const c10::cuda::CUDAGuard guard(input.device());
  Tensor f = freq.is_contiguous() ? freq : freq.contiguous();
  Tensor out = torch::empty(input.sizes(), input.options());
  check_status(l3ci_rot_embed(input.data_ptr(), f.data_ptr<float>(), out.data_ptr(), input.size(0), input.size(1),
                              input.size(2), input.size(3), input.stride(0), input.stride(1), input.stride(2),
                              current_stream()),
               "rot_embed");
  return out;
}

// Rotary embedding of q and k plus the cache write of k and v in one pass (model.py:100-108).
// qkv: [B, T, (n_head + 2*n_kv_head) * D]; caches: [maxB, maxLen, n_kv_head, D].  Returns rotated
// q as [B, T, n_head, D]; cache_k / cache_v are updated in place at [:, start_pos : start_pos + T].
//
// With `positions` (int32 [B] on the device) every sequence has its own position: token t of sequence b
// is at positions[b] + t, `freq` is then the WHOLE table and `start_pos` is ignored.  Nothing on the host
// depends on the positions, so a decode step written this way can be captured in a CUDA graph.
Tensor rot_embed_kv_cache(Tensor qkv, Tensor freq, Tensor cache_k, Tensor cache_v, int64_t start_pos,
                          int64_t n_head, int64_t n_kv_head, std::optional<Tensor> positions) {
  check_bf16_cuda(qkv, "qkv");
  check_bf16_cuda(cache_k, "cache_k");
  check_bf16_cuda(cache_v, "cache_v");
  TORCH_CHECK(qkv.dim() == 3 && qkv.stride(2) == 1, "qkv must be [B, T, (n_head + 2*n_kv_head) * D] with a contiguous last dimension");
  TORCH_CHECK(n_head > 0 && n_kv_head > 0 && qkv.size(2) % (n_head + 2 * n_kv_head) == 0, "qkv width does not match the head counts");
  const int64_t B = qkv.size(0), T = qkv.size(1), D = qkv.size(2) / (n_head + 2 * n_kv_head);
  TORCH_CHECK(cache_k.dim() == 4 && cache_k.sizes() == cache_v.sizes() && cache_k.strides() == cache_v.strides(),
              "cache_k and cache_v must be [maxB, maxLen, n_kv_head, D] with equal layout");
  TORCH_CHECK(cache_k.size(2) == n_kv_head && cache_k.size(3) == D && cache_k.stride(3) == 1 && cache_k.stride(2) == D,
              "cache rows must be [n_kv_head, D] contiguous");
  TORCH_CHECK(B <= cache_k.size(0), "batch does not fit the cache");
  TORCH_CHECK(freq.is_cuda() && freq.scalar_type() == torch::kFloat32 && freq.numel() >= T * D, "freq must be float32 [T, D]");
  if (positions) {
    TORCH_CHECK(positions->is_cuda() && positions->scalar_type() == torch::kInt32 && positions->dim() == 1 &&
                    positions->size(0) == B && positions->is_contiguous() && positions->get_device() == qkv.get_device(),
                "positions must be a contiguous int32 CUDA tensor of shape [B]");
    TORCH_CHECK(freq.dim() == 2 && freq.size(1) == D, "with positions, freq must be the whole [rows, D] table");
  } else {
    TORCH_CHECK(start_pos >= 0 && start_pos + T <= cache_k.size(1), "step does not fit the cache");
  }
  TORCH_CHECK(cache_k.get_device() == qkv.get_device() && cache_v.get_device() == qkv.get_device() &&
                  freq.get_device() == qkv.get_device(),
              "tensors on different devices");
  const c10::cuda::CUDAGuard guard(qkv.device());
  Tensor f = freq.is_contiguous() ? freq : freq.contiguous();
  Tensor q_out = torch::empty({B, T, n_head, D}, qkv.options());
  if (positions) {
    check_status(l3ci_rot_embed_kv_cache_at(qkv.data_ptr(), f.data_ptr<float>(), f.size(0), q_out.data_ptr(),
                                            cache_k.data_ptr(), cache_v.data_ptr(), positions->data_ptr<int32_t>(), B, T,
                                            n_head, n_kv_head, D, qkv.stride(0), qkv.stride(1), cache_k.stride(0),
                                            cache_k.stride(1), cache_k.size(1), current_stream()),
                 "rot_embed_kv_cache");
    return q_out;
  }
  check_status(l3ci_rot_embed_kv_cache(qkv.data_ptr(), f.data_ptr<float>(), q_out.data_ptr(), cache_k.data_ptr(),
                                       cache_v.data_ptr(), B, T, n_head, n_kv_head, D, qkv.stride(0), qkv.stride(1),
                                       cache_k.stride(0), cache_k.stride(1), start_pos, current_stream()),
               "rot_embed_kv_cache");
  return q_out;
}

// linear(x, w) of few rows, then rot_embed_kv_cache of its rows, in one kernel: the rotated queries; nothing where that kernel does not apply or
// does not pay (the rule of `linear`; more than 32 rows).  `early`, `always`: as in `linear`.
std::optional<Tensor> linear_rot_embed_kv_cache(Tensor x, Tensor w, Tensor freq, Tensor cache_k, Tensor cache_v, int64_t n_head, int64_t n_kv_head,
                                                Tensor positions, bool early, bool always) {
  check_bf16_cuda(x, "x");
  check_bf16_cuda(w, "w");
  check_bf16_cuda(cache_k, "cache_k");
  check_bf16_cuda(cache_v, "cache_v");
  TORCH_CHECK(x.dim() == 3 && w.dim() == 2 && w.size(1) == x.size(2), "x must be [B, T, K], w [N, K]");
  TORCH_CHECK(n_head > 0 && n_kv_head > 0 && w.size(0) % (n_head + 2 * n_kv_head) == 0, "w's rows do not match the head counts");
  const int64_t B = x.size(0), T = x.size(1), K = x.size(2), N = w.size(0), D = N / (n_head + 2 * n_kv_head);
  TORCH_CHECK(cache_k.dim() == 4 && cache_k.sizes() == cache_v.sizes() && cache_k.strides() == cache_v.strides(),
              "cache_k and cache_v must be [maxB, maxLen, n_kv_head, D] with equal layout");
  TORCH_CHECK(cache_k.size(2) == n_kv_head && cache_k.size(3) == D && cache_k.stride(3) == 1 && cache_k.stride(2) == D,
              "cache rows must be [n_kv_head, D] contiguous");
  TORCH_CHECK(B <= cache_k.size(0), "batch does not fit the cache");
  TORCH_CHECK(freq.is_cuda() && freq.scalar_type() == torch::kFloat32 && freq.dim() == 2 && freq.size(1) == D, "freq must be the whole float32 [rows, D] table");
  TORCH_CHECK(positions.is_cuda() && positions.scalar_type() == torch::kInt32 && positions.dim() == 1 && positions.size(0) == B && positions.is_contiguous(),
              "positions must be a contiguous int32 CUDA tensor of shape [B]");
  for (const Tensor& t : {w, cache_k, cache_v, freq, positions}) TORCH_CHECK(t.get_device() == x.get_device(), "tensors on different devices");
  const int64_t rows = B * T;
  if (rows == 0 || rows > 32 || K % 8 || !w.is_contiguous() || !freq.is_contiguous() ||
      (!always && !few_rows_pay(rows, K, N, 1, L3CI_ACT_NONE, early)))
    return std::nullopt;
  const int64_t stride = l3ci_row_stride(x.sizes().data(), x.strides().data(), 3);
  if (stride < 0 || stride % 8) return std::nullopt;
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor q = torch::empty({B, T, n_head, D}, x.options());
  l3ci_linear_args a{};
  a.x = x.data_ptr(); a.w = w.data_ptr(); a.out = q.data_ptr();
  a.rows = rows; a.x_st = stride; a.out_st = n_head * D;
  a.K = (int32_t)K; a.N = (int32_t)N; a.groups = 1; a.act = L3CI_ACT_NONE; a.early = early;
  a.stream = current_stream();
  l3ci_linear_rope r{};
  r.freq_table = freq.data_ptr<float>(); r.positions = positions.data_ptr<int32_t>();
  r.cache_k = cache_k.data_ptr(); r.cache_v = cache_v.data_ptr();
  r.freq_rows = freq.size(0); r.cache_sb = cache_k.stride(0); r.cache_st = cache_k.stride(1); r.cache_len = cache_k.size(1);
  r.T = (int32_t)T; r.Hq = (int32_t)n_head; r.Hkv = (int32_t)n_kv_head; r.D = (int32_t)D;
  const int status = l3ci_linear_rot_embed_kv_cache(&a, &r);
  if (status == L3CI_ERR_UNSUPPORTED || status == L3CI_ERR_ALIGNMENT) return std::nullopt;
  check_status(status, "linear_rot_embed_kv_cache");
  return q;
}

// Status of the few-row products on the current stream of `like`'s device: 0, or 6 once after a device-side wait ran out.
int64_t linear_status(Tensor like) {
  TORCH_CHECK(like.is_cuda(), "like must be a CUDA tensor");
  const c10::cuda::CUDAGuard guard(like.device());
  const int status = l3ci_linear_poll(current_stream());
  TORCH_CHECK(status != L3CI_ERR_CUDA, "linear_status: ", l3ci_last_error());
  return status;
}

// Synchronises the current stream of `like`'s device and reports whether a device-side bounded
// wait ran out in an earlier flash_attention_decode call on it (0 = fine).
int64_t flash_decode_status(Tensor like) {
  TORCH_CHECK(like.is_cuda(), "pass any tensor on the device to query");
  const c10::cuda::CUDAGuard guard(like.device());
  const auto stream = c10::cuda::getCurrentCUDAStream();
  const auto key = std::make_pair((int)like.get_device(), (int64_t)stream.id());
  Tensor buf;
  {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    auto it = workspaces().find(key);
    if (it == workspaces().end() || !it->second.buf.defined()) return 0;
    buf = it->second.buf;
  }
  return l3ci_flash_decode_poll(buf.data_ptr(), (size_t)buf.numel(), current_stream());
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  m.def("flash_attention_decode", torch::wrap_pybind_function(flash_attention_decode), "flash_attention_decode",
        py::arg("query"), py::arg("keys"), py::arg("values"), py::kw_only(), py::arg("seq_lens") = py::none(),
        py::arg("out") = py::none(), py::arg("scale") = 0.0, py::arg("max_ctas") = 0);
  m.def("rms_norm", torch::wrap_pybind_function(rms_norm), "rms_norm", py::arg("input"), py::arg("weight"),
        py::arg("eps"));
  m.def("add_rms_norm", torch::wrap_pybind_function(add_rms_norm), "add_rms_norm", py::arg("x"), py::arg("residual"),
        py::arg("weight"), py::arg("eps"));
  m.def("silu_mul", torch::wrap_pybind_function(silu_mul), "silu_mul", py::arg("gate"), py::arg("up"));
  m.def("linear", torch::wrap_pybind_function(linear), "linear", py::arg("x"), py::arg("w"), py::arg("gated") = false,
        py::arg("early") = false, py::arg("always") = false);
  m.def("few_rows", torch::wrap_pybind_function(few_rows), "few_rows", py::arg("x"), py::arg("w"), py::arg("act") = (int64_t)L3CI_ACT_NONE,
        py::arg("early") = false, py::arg("f32") = false, py::arg("into") = py::none(),
        py::arg("always") = false, py::arg("limit") = 0.0, py::arg("alpha") = 0.0);
  m.def("linear_rot_embed_kv_cache", torch::wrap_pybind_function(linear_rot_embed_kv_cache), "linear_rot_embed_kv_cache", py::arg("x"), py::arg("w"), py::arg("freq"),
        py::arg("cache_k"), py::arg("cache_v"), py::arg("n_head"), py::arg("n_kv_head"), py::arg("positions"), py::arg("early") = false, py::arg("always") = false);
  m.def("many_rows", torch::wrap_pybind_function(many_rows), "many_rows", py::arg("x"), py::arg("w"), py::arg("act"));
  m.def("greedy_step", torch::wrap_pybind_function(greedy_step), "greedy_step", py::arg("logits"), py::arg("out_tokens"),
        py::arg("steps"), py::arg("next_input"), py::arg("positions"), py::arg("seq_lens"));
  m.def("top_p_step", torch::wrap_pybind_function(top_p_step), "top_p_step", py::arg("logits"), py::arg("out_tokens"),
        py::arg("steps"), py::arg("next_input"), py::arg("positions"), py::arg("seq_lens"), py::arg("temperature"),
        py::arg("top_p"), py::arg("seed"));
  m.def("rot_embed", torch::wrap_pybind_function(rot_embed), "rot_embed", py::arg("input"), py::arg("freq"));
  m.def("rot_embed_kv_cache", torch::wrap_pybind_function(rot_embed_kv_cache), "rot_embed_kv_cache",
        py::arg("qkv"), py::arg("freq"), py::arg("cache_k"), py::arg("cache_v"), py::arg("start_pos"),
        py::arg("n_head"), py::arg("n_kv_head"), py::kw_only(), py::arg("positions") = py::none());
  m.def("flash_attention_decode_partial", torch::wrap_pybind_function(flash_attention_decode_partial),
        "flash_attention_decode_partial", py::arg("query"), py::arg("keys"), py::arg("values"), py::kw_only(),
        py::arg("seq_lens") = py::none(), py::arg("scale") = 0.0, py::arg("max_ctas") = 0,
        py::arg("out_o") = py::none(), py::arg("out_lse") = py::none());
  m.def("lse_exchange_merge", torch::wrap_pybind_function(lse_exchange_merge), "lse_exchange_merge", py::arg("bufs"),
        py::arg("rank"), py::arg("epoch"), py::arg("B"), py::arg("Hq"), py::arg("D"), py::kw_only(),
        py::arg("status") = py::none());
  // which decode kernel a call of these sizes takes on `device` (0 = persistent grid, else 16*C + W of the static deal)
  m.def("flash_decode_kernel_choice", [](int64_t device, int64_t B, int64_t Hq, int64_t Hkv, int64_t D, int64_t n_seq, bool ragged) {
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
    return (int64_t)l3ci_flash_decode_kernel_choice((int32_t)B, (int32_t)Hq, (int32_t)Hkv, (int32_t)D, (int32_t)n_seq,
                                                    ragged ? 1 : 0);
  }, py::arg("device"), py::arg("B"), py::arg("Hq"), py::arg("Hkv"), py::arg("D"), py::arg("n_seq"), py::arg("ragged") = false);
  m.def("flash_attention_decode_exchange", torch::wrap_pybind_function(flash_attention_decode_exchange),
        "flash_attention_decode_exchange", py::arg("query"), py::arg("keys"), py::arg("values"), py::arg("bufs"),
        py::arg("rank"), py::arg("epoch") = 0, py::kw_only(), py::arg("seq_lens") = py::none(), py::arg("out") = py::none(),
        py::arg("status") = py::none(), py::arg("scale") = 0.0, py::arg("max_ctas") = 0);
  m.def("flash_decode_exchange_bytes", [](int64_t ranks, int64_t B, int64_t Hq, int64_t D) {
    return (int64_t)l3ci_flash_decode_exchange_bytes((int32_t)ranks, (int32_t)B, (int32_t)Hq, (int32_t)D);
  });
  m.def("lse_exchange_bytes", [](int64_t ranks, int64_t B, int64_t Hq, int64_t D) {
    return (int64_t)l3ci_lse_exchange_bytes((int32_t)ranks, (int32_t)B, (int32_t)Hq, (int32_t)D);
  });
  m.def("lse_merge", torch::wrap_pybind_function(lse_merge), "lse_merge", py::arg("o_parts"), py::arg("lse_parts"));
  m.def("prefill_attention", torch::wrap_pybind_function(prefill_attention), "prefill_attention", py::arg("query"),
        py::arg("keys"), py::arg("values"), py::kw_only(), py::arg("start_pos") = 0, py::arg("scale") = 0.0,
        py::arg("variant") = 0);
  m.def("linear_status", torch::wrap_pybind_function(linear_status), "linear_status", py::arg("like"));
  m.def("flash_decode_status", torch::wrap_pybind_function(flash_decode_status), "flash_decode_status",
        py::arg("like"));
  m.def("c_abi_version", [] { return std::string(l3ci_version()); });
}
