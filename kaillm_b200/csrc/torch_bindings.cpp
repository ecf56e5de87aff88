// `_C_gguf` PyTorch extension: the same op schemas the reference registers
// (vllm_gguf_plugin/csrc/torch_bindings.cpp:22-61), implemented by calling the libkq C ABI
// (include/kq_gguf.h).  torch supplies device memory, the current stream and the dispatcher; all
// arithmetic happens behind the C ABI.
//
// Differences from the reference bindings, on purpose:
//   - outputs come from at::empty (the kernels write every element; the reference memsets with new_zeros);
//   - an unsupported GGML type raises instead of silently returning zeros
//     (reference: switch without default, csrc/gguf/gguf_kernel.cu:119-215);
//   - ops of this library's own beside the reference's six: ggml_dequant_mul_mat, ggml_dequantize_rows,
//     ggml_mul_mat_merged, fused_moe_swiglu (no derivative: kaillm_b200/linear.py calls them for plain tensors only).
#include <Python.h>

#include <algorithm>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/library.h>

#include "../../include/kq_gguf.h"

namespace {

int kq_dtype_of(at::ScalarType t, const char* what) {
  switch (t) {
    case at::kFloat: return KQ_F32;
    case at::kHalf: return KQ_F16;
    case at::kBFloat16: return KQ_BF16;
    default: TORCH_CHECK(false, what, ": dtype must be float32, float16 or bfloat16, got ", t);
  }
}

void check_weight(const at::Tensor& W, const char* fn) {
  TORCH_CHECK(W.is_cuda(), fn, ": W must be a CUDA tensor");
  TORCH_CHECK(W.scalar_type() == at::kByte, fn, ": W must be uint8 GGUF wire bytes");
  TORCH_CHECK(W.is_contiguous(), fn, ": W must be contiguous");
}

at::Tensor mul_mat_impl(bool mmq, const at::Tensor& W, const at::Tensor& X, int64_t type, int64_t row) {
  const char* fn = mmq ? "ggml_mul_mat_a8" : "ggml_mul_mat_vec_a8";
  check_weight(W, fn);
  TORCH_CHECK(X.is_cuda() && X.dim() == 2, fn, ": X must be a 2-D CUDA tensor");
  TORCH_CHECK(X.get_device() == W.get_device(), fn, ": W and X are on different devices");
  TORCH_CHECK(X.stride(1) == 1, fn, ": X must be contiguous along its last dimension");
  const int64_t m = X.size(0), k = X.size(1);
  const int xdt = kq_dtype_of(X.scalar_type(), fn);
  int blk = 0, bytes = 0;
  TORCH_CHECK(kq_block_geometry((int)type, &blk, &bytes) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(k % blk == 0, fn, ": X.size(1)=", k, " is not a multiple of the block size ", blk);
  TORCH_CHECK(row >= 0 && W.numel() >= row * (k / blk) * bytes, fn, ": W holds fewer than `row` rows of K=", k);
  const c10::cuda::CUDAGuard guard(X.device());
  at::Tensor Y = at::empty({m, row}, X.options());
  if (m == 0 || row == 0) return Y;
  const size_t ws = kq_workspace_bytes((int)type, m, row, k);
  at::Tensor scratch = at::empty({(int64_t)ws}, W.options());
  auto stream = at::cuda::getCurrentCUDAStream(X.get_device()).stream();
  auto fnp = mmq ? kq_mul_mat_a8 : kq_mul_mat_vec_a8;
  const int rc = fnp(W.data_ptr(), (int)type, row, k, X.data_ptr(), xdt, m, X.stride(0), Y.data_ptr(), xdt,
                     Y.stride(0), scratch.data_ptr(), ws, (void*)stream);
  TORCH_CHECK(rc == KQ_OK, fn, ": ", kq_last_error());
  return Y;
}

at::Tensor ggml_mul_mat_vec_a8(const at::Tensor& W, const at::Tensor& X, int64_t type, c10::SymInt row) {
  return mul_mat_impl(false, W, X, type, row.expect_int());
}

at::Tensor ggml_mul_mat_a8(const at::Tensor& W, const at::Tensor& X, int64_t type, c10::SymInt row) {
  return mul_mat_impl(true, W, X, type, row.expect_int());
}

// Projections of different types over the same activations (q/k/v of a mixed-type file): one quantization, every shard's
// kernel writes its own columns of the merged output.  mmq[i]: which of the two ops shard i is.
at::Tensor ggml_mul_mat_merged(at::TensorList Ws, const at::Tensor& X, at::IntArrayRef types, at::IntArrayRef mmq) {
  const char* fn = "ggml_mul_mat_merged";
  TORCH_CHECK(!Ws.empty() && Ws.size() == types.size() && Ws.size() == mmq.size(), fn, ": one type and flavour per shard");
  TORCH_CHECK(X.is_cuda() && X.dim() == 2 && X.stride(1) == 1, fn, ": X must be a 2-D CUDA tensor, contiguous along its last dimension");
  const int64_t m = X.size(0), k = X.size(1);
  const int xdt = kq_dtype_of(X.scalar_type(), fn);
  int64_t total = 0, widest = 0;
  size_t ws = 0;
  for (size_t i = 0; i < Ws.size(); ++i) {
    const at::Tensor& W = Ws[i];
    check_weight(W, fn);
    int blk = 0, bytes = 0;
    TORCH_CHECK(kq_block_geometry((int)types[i], &blk, &bytes) == KQ_OK, fn, ": ", kq_last_error());
    TORCH_CHECK(W.dim() == 2 && W.get_device() == X.get_device(), fn, ": W must be 2-D and on X's device");
    TORCH_CHECK(k % blk == 0 && W.size(1) == k / blk * bytes, fn, ": a shard does not hold rows of K=", k);
    total += W.size(0);
    widest = std::max(widest, W.size(0));
  }
  for (size_t i = 0; i < Ws.size(); ++i) ws = std::max(ws, kq_workspace_bytes((int)types[i], m, widest, k));
  const c10::cuda::CUDAGuard guard(X.device());
  at::Tensor Y = at::empty({m, total}, X.options());
  if (m == 0 || total == 0) return Y;
  at::Tensor scratch = at::empty({(int64_t)ws}, X.options().dtype(at::kByte));
  void* stream = (void*)at::cuda::getCurrentCUDAStream(X.get_device()).stream();
  TORCH_CHECK(kq_prepare_q8((int)types[0], widest, k, X.data_ptr(), xdt, m, X.stride(0), scratch.data_ptr(), ws, 0, stream) == KQ_OK, fn, ": ", kq_last_error());
  int64_t col = 0;
  for (size_t i = 0; i < Ws.size(); ++i) {
    const int64_t n = Ws[i].size(0);
    if (n == 0) continue;
    void* y = static_cast<char*>(Y.data_ptr()) + col * (int64_t)Y.element_size();
    TORCH_CHECK(kq_mul_mat_prepared(Ws[i].data_ptr(), (int)types[i], n, k, m, y, xdt, total, (int)mmq[i], scratch.data_ptr(), ws, stream) == KQ_OK,
                fn, ": ", kq_last_error());
    col += n;
  }
  return Y;
}

at::Tensor ggml_dequantize(const at::Tensor& W, int64_t type, c10::SymInt m_, c10::SymInt n_,
                           std::optional<at::ScalarType> dtype) {
  const char* fn = "ggml_dequantize";
  check_weight(W, fn);
  const int64_t m = m_.expect_int(), n = n_.expect_int();
  const at::ScalarType dt = dtype.value_or(at::kHalf);
  const int odt = kq_dtype_of(dt, fn);
  int blk = 0, bytes = 0;
  TORCH_CHECK(kq_block_geometry((int)type, &blk, &bytes) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(m >= 0 && n >= 0 && (m * n) % blk == 0, fn, ": m*n must be a multiple of the block size ", blk);
  TORCH_CHECK(W.numel() >= (m * n) / blk * bytes, fn, ": W holds fewer than m*n weights");
  const c10::cuda::CUDAGuard guard(W.device());
  at::Tensor DW = at::empty({m, n}, W.options().dtype(dt));
  if (m * n == 0) return DW;
  auto stream = at::cuda::getCurrentCUDAStream(W.get_device()).stream();
  const int rc = kq_dequantize(W.data_ptr(), (int)type, m * n, DW.data_ptr(), odt, (void*)stream);
  TORCH_CHECK(rc == KQ_OK, fn, ": ", kq_last_error());
  return DW;
}

// X @ dequantize(W)^T: one kernel where it covers the call, otherwise the two steps
at::Tensor ggml_dequant_mul_mat(const at::Tensor& W, const at::Tensor& X, int64_t type, c10::SymInt row_) {
  const char* fn = "ggml_dequant_mul_mat";
  const int64_t row = row_.expect_int();
  int blk = 0, bytes = 0;
  TORCH_CHECK(kq_block_geometry((int)type, &blk, &bytes) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(W.dim() == 2, fn, ": W must be 2-D");
  const bool half = X.scalar_type() == at::kHalf || X.scalar_type() == at::kBFloat16;
  if (half && W.is_cuda() && X.is_cuda() && W.get_device() == X.get_device() && W.scalar_type() == at::kByte && W.is_contiguous() &&
      X.dim() == 2 && X.stride(1) == 1 && W.size(0) == row && X.size(1) % blk == 0 && W.size(1) == X.size(1) / blk * bytes) {
    const int64_t m = X.size(0), k = X.size(1);
    const int xdt = kq_dtype_of(X.scalar_type(), fn);
    // short rows leave a second wave of tiles little to share its start-up with: 24576x1024 at 9 / 65 / 129 tokens, two steps / one kernel,
    // us: IQ4_NL 27 / 29 / 31 against 31 / 33 / 35, IQ4_XS 29 / 30 / 32 against 32 / 33 / 35; 32000x1024 33 / 33 / 35 against 31 / 31 / 35
    const bool short_rows = type != 21 && k < 2048 && row > 148 * 128 && row < 30000;   // IQ3_S: 31 against 29
    if (!short_rows && kq_dequant_mul_mat_preferred(row, m) && kq_dequant_mul_mat_supported(W.data_ptr(), (int)type, row, k, X.data_ptr(), xdt, m, X.stride(0))) {
      const c10::cuda::CUDAGuard guard(X.device());
      at::Tensor Y = at::empty({m, row}, X.options());
      auto stream = at::cuda::getCurrentCUDAStream(X.get_device()).stream();
      TORCH_CHECK(kq_dequant_mul_mat(W.data_ptr(), (int)type, row, k, X.data_ptr(), xdt, m, X.stride(0), Y.data_ptr(), Y.stride(0),
                                     (void*)stream) == KQ_OK, fn, ": ", kq_last_error());
      return Y;
    }
  }
  return at::matmul(X, ggml_dequantize(W, type, c10::SymInt(row), c10::SymInt(W.size(1) / bytes * blk), X.scalar_type()).t());
}

// rows `ids` (any shape) of the [n, row bytes] table W, dequantized: [*ids.shape, k]
at::Tensor ggml_dequantize_rows(const at::Tensor& W, const at::Tensor& ids, int64_t type, int64_t k, at::ScalarType dtype, bool f32_math) {
  const char* fn = "ggml_dequantize_rows";
  check_weight(W, fn);
  TORCH_CHECK(W.dim() == 2 && ids.is_cuda() && ids.get_device() == W.get_device(), fn, ": W must be 2-D and the ids on its device");
  const int odt = kq_dtype_of(dtype, fn);
  int blk = 0, bytes = 0;
  TORCH_CHECK(kq_block_geometry((int)type, &blk, &bytes) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(k > 0 && k % blk == 0 && W.size(1) == k / blk * bytes, fn, ": rows of W do not hold k=", k, " weights");
  const c10::cuda::CUDAGuard guard(W.device());
  const at::Tensor flat = ids.to(at::kLong).contiguous();
  auto shape = ids.sizes().vec();
  shape.push_back(k);
  at::Tensor out = at::empty(shape, W.options().dtype(dtype));
  const int rc = kq_dequantize_rows(W.data_ptr(), (int)type, W.size(0), k, flat.data_ptr<int64_t>(), flat.numel(), out.data_ptr(), odt,
                                    f32_math, (void*)at::cuda::getCurrentCUDAStream(W.get_device()).stream());
  TORCH_CHECK(rc == KQ_OK, fn, ": ", kq_last_error());
  return out;
}

// W: [E, row, row bytes] (or any contiguous uint8 tensor holding E matrices back to back)
at::Tensor moe_impl(bool block, const at::Tensor& X, const at::Tensor& W, const at::Tensor& ids, const at::Tensor* expert_ids,
                    const at::Tensor* num_post_padded, int64_t type, int64_t row, int64_t top_k, int64_t tokens) {
  const char* fn = block ? "ggml_moe_a8" : "ggml_moe_a8_vec";
  check_weight(W, fn);
  TORCH_CHECK(X.is_cuda() && X.dim() == 2, fn, ": X must be a 2-D CUDA tensor");
  TORCH_CHECK(X.get_device() == W.get_device(), fn, ": W and X are on different devices");
  TORCH_CHECK(X.stride(1) == 1, fn, ": X must be contiguous along its last dimension");
  TORCH_CHECK(tokens >= 0 && tokens <= X.size(0), fn, ": `tokens` exceeds X.size(0)");
  TORCH_CHECK(top_k > 0 && row >= 0, fn, ": top_k must be positive");
  const int64_t k = X.size(1);
  const int xdt = kq_dtype_of(X.scalar_type(), fn);
  int blk = 0, bytes = 0;
  TORCH_CHECK(kq_block_geometry((int)type, &blk, &bytes) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(k % blk == 0, fn, ": X.size(1)=", k, " is not a multiple of the block size ", blk);
  const int64_t per_expert = row * (k / blk) * bytes;
  TORCH_CHECK(per_expert > 0 && W.numel() % per_expert == 0, fn, ": W is not a whole number of [row, K] matrices");
  const int64_t experts = W.numel() / per_expert;
  auto as_i32 = [&](const at::Tensor& t, const char* name) {
    TORCH_CHECK(t.is_cuda() && t.get_device() == X.get_device(), fn, ": ", name, " must be on X's device");
    return t.scalar_type() == at::kInt && t.is_contiguous() ? t : t.to(at::kInt).contiguous();
  };
  const c10::cuda::CUDAGuard guard(X.device());
  at::Tensor Y = at::zeros({tokens * top_k, row}, X.options());   // rows nobody writes read as zero, as in the reference
  if (tokens == 0 || row == 0) return Y;
  const at::Tensor ids32 = as_i32(ids, block ? "sorted_token_ids" : "topk_ids");
  const size_t ws = kq_workspace_bytes((int)type, tokens, row, k);
  at::Tensor scratch = at::empty({(int64_t)ws}, W.options());
  auto stream = at::cuda::getCurrentCUDAStream(X.get_device()).stream();
  int rc;
  if (block) {
    const at::Tensor e32 = as_i32(*expert_ids, "expert_ids"), n32 = as_i32(*num_post_padded, "num_tokens_post_padded");
    TORCH_CHECK(n32.numel() >= 1, fn, ": num_tokens_post_padded is empty");
    TORCH_CHECK(e32.numel() * kq_moe_block_size((int)type) >= ids32.numel(), fn, ": expert_ids has fewer entries than blocks of sorted tokens");
    rc = kq_moe_a8(W.data_ptr(), (int)type, experts, row, k, X.data_ptr(), xdt, tokens, X.stride(0), ids32.data_ptr<int32_t>(),
                   ids32.numel(), e32.data_ptr<int32_t>(), n32.data_ptr<int32_t>(), (int)top_k, Y.data_ptr(), xdt, Y.stride(0),
                   scratch.data_ptr(), ws, (void*)stream);
  } else {
    TORCH_CHECK(ids32.numel() >= tokens * top_k, fn, ": topk_ids has fewer than tokens * top_k entries");
    rc = kq_moe_a8_vec(W.data_ptr(), (int)type, experts, row, k, X.data_ptr(), xdt, tokens, X.stride(0), ids32.data_ptr<int32_t>(),
                       (int)top_k, Y.data_ptr(), xdt, Y.stride(0), scratch.data_ptr(), ws, (void*)stream);
  }
  TORCH_CHECK(rc == KQ_OK, fn, ": ", kq_last_error());
  return Y;
}

at::Tensor ggml_moe_a8(const at::Tensor& X, const at::Tensor& W, const at::Tensor& sorted_token_ids, const at::Tensor& expert_ids,
                       const at::Tensor& num_tokens_post_padded, int64_t type, c10::SymInt row, c10::SymInt top_k,
                       c10::SymInt tokens) {
  return moe_impl(true, X, W, sorted_token_ids, &expert_ids, &num_tokens_post_padded, type, row.expect_int(), top_k.expect_int(),
                  tokens.expect_int());
}

at::Tensor ggml_moe_a8_vec(const at::Tensor& X, const at::Tensor& W, const at::Tensor& topk_ids, int64_t top_k, int64_t type,
                           c10::SymInt row, c10::SymInt tokens) {
  return moe_impl(false, X, W, topk_ids, nullptr, nullptr, type, row.expect_int(), top_k, tokens.expect_int());
}

// The whole SiLU feed-forward of linear.fused_moe_gguf: 5 launches (per-pair branch) or 6 (expert-sorted branch).
// W1 [E, 2 * inter, row bytes], W2 [E, hidden_out, row bytes], topk_ids [tokens, top_k], topk_weights of as many entries.
at::Tensor fused_moe_swiglu(const at::Tensor& X, const at::Tensor& W1, const at::Tensor& W2, const at::Tensor& topk_weights,
                            const at::Tensor& topk_ids, int64_t type1, int64_t type2, bool block) {
  const char* fn = "fused_moe_swiglu";
  check_weight(W1, fn);
  check_weight(W2, fn);
  TORCH_CHECK(W1.dim() == 3 && W2.dim() == 3 && X.dim() == 2 && topk_ids.dim() == 2, fn, ": bad dimensions");
  TORCH_CHECK(X.is_cuda() && X.stride(1) == 1, fn, ": X must be a CUDA tensor, contiguous along its last dimension");
  for (const at::Tensor* t : {&W1, &W2, &topk_weights, &topk_ids}) TORCH_CHECK(t->is_cuda() && t->get_device() == X.get_device(), fn, ": all tensors must be on X's device");
  const int64_t tokens = X.size(0), k1 = X.size(1), e = W1.size(0), n1 = W1.size(1), n2 = W2.size(1), top_k = topk_ids.size(1), pairs = tokens * top_k;
  const int64_t k2 = n1 / 2;
  int b1 = 0, s1 = 0, b2 = 0, s2 = 0;
  TORCH_CHECK(kq_block_geometry((int)type1, &b1, &s1) == KQ_OK && kq_block_geometry((int)type2, &b2, &s2) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(tokens > 0 && top_k > 0 && n1 % 2 == 0 && n1 > 0 && n2 > 0 && topk_ids.size(0) == tokens && topk_weights.numel() == pairs, fn, ": sizes do not match");
  TORCH_CHECK(k1 % b1 == 0 && W1.size(2) == k1 / b1 * s1 && k2 % b2 == 0 && W2.size(2) == k2 / b2 * s2 && W2.size(0) == e, fn, ": weight sizes do not match");
  const int xdt = kq_dtype_of(X.scalar_type(), fn), wdt = kq_dtype_of(topk_weights.scalar_type(), fn);
  const c10::cuda::CUDAGuard guard(X.device());
  auto stream = (void*)at::cuda::getCurrentCUDAStream(X.get_device()).stream();
  const at::Tensor ids = topk_ids.to(at::kInt).contiguous();
  const at::Tensor tw = topk_weights.contiguous();
  const auto iopt = X.options().dtype(at::kInt);
  at::Tensor sorted, eids, post, flag;
  at::cuda::CUDAEvent copied;
  if (block) {
    const int64_t bs = kq_moe_block_size((int)type1), nb = (pairs + e * (bs - 1) + bs - 1) / bs;
    sorted = at::empty({nb * bs}, iopt); eids = at::empty({nb}, iopt); post = at::empty({2}, iopt);
    TORCH_CHECK(kq_moe_align(ids.data_ptr<int32_t>(), pairs, e, sorted.data_ptr<int32_t>(), nb * bs, eids.data_ptr<int32_t>(), nb,
                             post.data_ptr<int32_t>(), stream) == KQ_OK, fn, ": ", kq_last_error());
    // an expert id outside [0, E) is an error in this branch: the flag travels to the host while the kernels below run, and the host
    // waits for it (so for all earlier work of the stream) at the end of the call; not capturable, as the chain of ops is not either
    flag = at::empty({2}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    flag.copy_(post, /*non_blocking=*/true);
    copied.record(at::cuda::getCurrentCUDAStream(X.get_device()));
  }
  const size_t ws1 = kq_workspace_bytes((int)type1, tokens, n1, k1), ws2 = kq_workspace_bytes((int)type2, pairs, n2, k2);
  at::Tensor scratch = at::empty({(int64_t)(ws1 > ws2 ? ws1 : ws2)}, W1.options());
  at::Tensor h = at::empty({pairs, n1}, X.options()), y = at::empty({pairs, n2}, X.options()), out = at::empty({tokens, n2}, X.options());
  const int32_t* idp = block ? sorted.data_ptr<int32_t>() : ids.data_ptr<int32_t>();
  const int32_t* ep = block ? eids.data_ptr<int32_t>() : nullptr;
  const int32_t* pp = block ? post.data_ptr<int32_t>() : nullptr;
  const int64_t nid = block ? sorted.numel() : pairs;
  TORCH_CHECK(kq_moe_project(0, W1.data_ptr(), (int)type1, e, n1, k1, X.data_ptr(), xdt, tokens, X.stride(0), idp, nid, ep, pp, (int)top_k,
                             h.data_ptr(), xdt, n1, scratch.data_ptr(), scratch.numel(), stream) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(kq_moe_project(1, W2.data_ptr(), (int)type2, e, n2, k2, h.data_ptr(), xdt, pairs, n1, idp, nid, ep, pp, 1, y.data_ptr(), xdt,
                             n2, scratch.data_ptr(), scratch.numel(), stream) == KQ_OK, fn, ": ", kq_last_error());
  TORCH_CHECK(kq_moe_combine(y.data_ptr(), xdt, tw.data_ptr(), wdt, tokens, n2, (int)top_k, out.data_ptr(), stream) == KQ_OK, fn, ": ", kq_last_error());
  if (block) {
    copied.synchronize();
    TORCH_CHECK(flag.data_ptr<int32_t>()[1] == 0, fn, ": topk_ids holds an expert id outside [0, ", e, ")");
  }
  return out;
}

int64_t ggml_moe_get_block_size(int64_t type) { return kq_moe_block_size((int)type); }

}  // namespace

TORCH_LIBRARY(_C_gguf, ops) {
  ops.def("ggml_dequantize(Tensor W, int type, SymInt m, SymInt n, ScalarType? dtype) -> Tensor");
  ops.def("ggml_mul_mat_vec_a8(Tensor W, Tensor X, int type, SymInt row) -> Tensor");
  ops.def("ggml_mul_mat_a8(Tensor W, Tensor X, int type, SymInt row) -> Tensor");
  ops.def("ggml_dequant_mul_mat(Tensor W, Tensor X, int type, SymInt row) -> Tensor");
  ops.def("ggml_dequantize_rows(Tensor W, Tensor ids, int type, int k, ScalarType dtype, bool f32_math) -> Tensor");
  ops.def("ggml_mul_mat_merged(Tensor[] W, Tensor X, int[] types, int[] mmq) -> Tensor");
  ops.def(
      "ggml_moe_a8(Tensor X, Tensor W, Tensor sorted_token_ids, Tensor expert_ids, Tensor "
      "num_tokens_post_padded, int type, SymInt row, SymInt top_k, SymInt tokens) -> Tensor");
  ops.def("ggml_moe_a8_vec(Tensor X, Tensor W, Tensor topk_ids, int top_k, int type, SymInt row, SymInt tokens) -> Tensor");
  ops.def(
      "fused_moe_swiglu(Tensor X, Tensor W1, Tensor W2, Tensor topk_weights, Tensor topk_ids, int type1, int type2, bool block) "
      "-> Tensor");
  ops.def("ggml_moe_get_block_size(int type) -> int");
}

TORCH_LIBRARY_IMPL(_C_gguf, CUDA, ops) {
  ops.impl("ggml_dequantize", &ggml_dequantize);
  ops.impl("ggml_mul_mat_vec_a8", &ggml_mul_mat_vec_a8);
  ops.impl("ggml_mul_mat_a8", &ggml_mul_mat_a8);
  ops.impl("ggml_dequant_mul_mat", &ggml_dequant_mul_mat);
  ops.impl("ggml_dequantize_rows", &ggml_dequantize_rows);
  ops.impl("ggml_mul_mat_merged", &ggml_mul_mat_merged);
  ops.impl("ggml_moe_a8", &ggml_moe_a8);
  ops.impl("ggml_moe_a8_vec", &ggml_moe_a8_vec);
  ops.impl("fused_moe_swiglu", &fused_moe_swiglu);
}

TORCH_LIBRARY_IMPL(_C_gguf, CompositeExplicitAutograd, ops) {
  ops.impl("ggml_moe_get_block_size", &ggml_moe_get_block_size);
}

static struct PyModuleDef kq_module_def = {PyModuleDef_HEAD_INIT, "_C_gguf", nullptr, -1, nullptr};

extern "C" PyObject* PyInit__C_gguf(void) { return PyModule_Create(&kq_module_def); }
