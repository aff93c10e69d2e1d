// Autograd functions of the hot single-GPU layers, in C++: linear (with bias, GELU and a residual), the LM head, layer norm, causal attention,
// cross-entropy, batch norm, convolution and the ResNet stem's convolution.  They make the checks of the Python functions that they
// stand for, and save the same tensors; only the host work around a launch is native.  A forward and backward of
// one layer took 100 - 160 us of Python (autograd.Function both ways, ctypes argument conversion, tensor bookkeeping)
// around 10 - 50 us of kernels, and a transformer block about as long as its kernels.
//
// Scratch memory is allocated per call from PyTorch's caching allocator on the calling stream; the buffers that are kept
// (KeptZeros) belong to one stream each.  A non-zero status is raised through torchmpi_b200._lib.check, so callers see the usual exceptions.
// The reference has no counterpart (its layers are Torch7's).
#include <torch/extension.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <atomic>
#include <cmath>
#include <map>
#include <mutex>
#include <string>
#include "tmpi_c_api.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

enum { LINEAR, LAYERNORM, ATTENTION, XENT, ATTENTION_BACKWARD, BATCHNORM, CONV, STEM, KINDS };
std::atomic<long long> g_launches[KINDS];      // attention: calls, and those of the backward alone
enum { EPI_BIAS = 1 };

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
void launched(int what, int n) { g_launches[what].fetch_add(n, std::memory_order_relaxed); }

void check(int status) {
  if (!status) return;
  pybind11::gil_scoped_acquire gil;
  pybind11::module_::import("torchmpi_b200._lib").attr("check")(status);
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return TMPI_F16;
    case at::kBFloat16: return TMPI_BF16;
    case at::kFloat: return TMPI_F32;
    case at::kDouble: return TMPI_F64;                           // what a kernel does not take, its entry point refuses
    case at::kByte: return TMPI_U8;
    case at::kChar: return TMPI_I8;
    case at::kShort: return TMPI_I16;
    case at::kInt: return TMPI_I32;
    case at::kLong: return TMPI_I64;
    default: throw pybind11::type_error(std::string("torchmpi_b200: unsupported dtype ") + c10::toString(t));
  }
}

// Contiguous and on a 16-byte boundary, which the elementwise kernels' loads need: a view into a larger buffer may start
// anywhere.
Tensor packed(const Tensor& t, at::MemoryFormat format = at::MemoryFormat::Contiguous) {
  if (t.is_contiguous(format) && (uintptr_t)t.data_ptr() % 16 == 0) return t;
  Tensor c = t.contiguous(format);
  if ((uintptr_t)c.data_ptr() % 16) c = c.clone(format);
  return c;
}

// A saved tensor as it was saved: hooks (torch.autograd.graph.save_on_cpu, say) may hand it back in another layout.
Tensor as_saved(const Tensor& t, at::MemoryFormat format = at::MemoryFormat::Contiguous) { return t.defined() ? packed(t, format) : t; }

// Buffers of arrival counters, which a kernel finds zero and leaves zero.  Two calls may share one only if one ends before the
// other starts, so there is one per stream, grown to the next power of two.  A call that is being captured gets its own, cleared
// inside the graph: the graph may be replayed on any stream, and has not run when the next eager call comes.  So does a call
// that needs a large one.  Buffers go back to the allocator, which hands them out on the stream they were used on.
struct KeptZeros {
  static constexpr size_t KEEP_BYTES = size_t(1) << 20, KEEP_STREAMS = 64;
  std::mutex lock;
  std::map<std::pair<int, void*>, Tensor> kept;
  int kept_at = 0;

  // failures: a number that grows when a kernel may have left a buffer behind that is not zero; all are dropped then.  It is odd as long as
  // a report of that waits to be read: further kernels may give up meanwhile without another change, so nothing is kept until then.
  Tensor get(const Tensor& like, size_t need, int failures = 0) {
    const auto bytes = like.options().dtype(at::kByte);
    if (need > KEEP_BYTES || failures % 2 || c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
      return at::zeros({(int64_t)need}, bytes);
    const std::pair<int, void*> key(like.get_device(), stream());
    std::map<std::pair<int, void*>, Tensor> old;                           // released outside the lock
    {
      std::lock_guard<std::mutex> hold(lock);
      if (failures != kept_at) {
        old.swap(kept);
        kept_at = failures;
      }
      const auto found = kept.find(key);
      if (found != kept.end() && (size_t)found->second.numel() >= need) return found->second;
    }
    size_t size = 4096;
    while (size < need) size *= 2;
    const Tensor fresh = at::zeros({(int64_t)size}, bytes);
    std::lock_guard<std::mutex> hold(lock);
    if (kept.size() >= KEEP_STREAMS) old.swap(kept);
    kept[key] = fresh;
    return fresh;
  }
};

bool pair_enabled() {
  int64_t v = 0;
  check(tmpi_get_tunable("gemm_pair", &v));
  return v != 0;
}

// ---------------------------------------------------------------- linear
Tensor matmul_nt(const Tensor& a_, const Tensor& b_, const Tensor& bias) {
  const Tensor a = a_.contiguous(), b = b_.contiguous(), c = bias.defined() ? bias.contiguous() : bias;
  const int M = (int)a.size(0), N = (int)b.size(0), K = (int)a.size(1), epi = c.defined() ? EPI_BIAS : 0;
  Tensor out = at::empty({M, N}, a.options());
  // few rows or columns: the pair kernel's narrow tiles, over more SMs
  if ((M < 256 || N < 256) && M >= 1 && N >= 1 && K >= 1 && N % 8 == 0 && K % 8 == 0 && pair_enabled())
    check(tmpi_gemm_bf16_any(a.data_ptr(), b.data_ptr(), out.data_ptr(), nullptr, c.defined() ? c.data_ptr() : nullptr, M, N, K, epi, stream()));
  else
    check(tmpi_gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), c.defined() ? c.data_ptr() : nullptr, M, N, K, epi, stream()));
  launched(LINEAR, 1);
  return out;
}

// a b^T + bias + residual, rounded once (linear_add of ops/gemm.py has made the checks)
Tensor matmul_nt_residual(const Tensor& a_, const Tensor& b_, const Tensor& bias, const Tensor& residual_) {
  const Tensor a = a_.contiguous(), b = b_.contiguous(), c = bias.defined() ? bias.contiguous() : bias, residual = packed(residual_);
  Tensor out = at::empty({a.size(0), b.size(0)}, a.options());
  check(tmpi_gemm_bf16_residual(a.data_ptr(), b.data_ptr(), out.data_ptr(), c.defined() ? c.data_ptr() : nullptr, residual.data_ptr(), (int)a.size(0),
                                (int)b.size(0), (int)a.size(1), stream()));
  launched(LINEAR, 1);
  return out;
}

Tensor gelu_pass(const Tensor& z) {
  if ((z.numel() * z.element_size()) % 16 || (uintptr_t)z.data_ptr() % 16) return at::gelu(z);
  Tensor y = at::empty_like(z);
  check(tmpi_gelu_fwd(z.data_ptr(), y.data_ptr(), (size_t)z.numel(), dtype_code(z.scalar_type()), stream()));
  launched(LINEAR, 1);
  return y;
}

// (z, gelu(z)); one kernel where the CTA-pair GEMM applies
std::pair<Tensor, Tensor> matmul_nt_gelu(const Tensor& a_, const Tensor& b_, const Tensor& bias) {
  const int64_t M = a_.size(0), N = b_.size(0), K = a_.size(1);
  if (!(M >= 1 && N >= 1 && K >= 1 && N % 8 == 0 && K % 8 == 0 && pair_enabled())) {
    Tensor z = matmul_nt(a_, b_, bias);
    return {z, gelu_pass(z)};
  }
  const Tensor a = a_.contiguous(), b = b_.contiguous(), c = bias.defined() ? bias.contiguous() : bias;
  Tensor z = at::empty({M, N}, a.options()), y = at::empty({M, N}, a.options());
  check(tmpi_gemm_bf16_any(a.data_ptr(), b.data_ptr(), z.data_ptr(), y.data_ptr(), c.defined() ? c.data_ptr() : nullptr, (int)M, (int)N,
                           (int)K, c.defined() ? EPI_BIAS : 0, stream()));
  launched(LINEAR, 1);
  return {z, y};
}

// a b and a^T b without the CTA-pair kernel: through transposed copies
Tensor matmul_nn(const Tensor& a, const Tensor& b) { return matmul_nt(a, b.t().contiguous(), Tensor()); }
Tensor matmul_tn(const Tensor& a, const Tensor& b) { return matmul_nt(a.t().contiguous(), b.t().contiguous(), Tensor()); }

// dz = dy * gelu'(z) (dy itself without z) and its column sum, in one pass where the kernel applies
std::pair<Tensor, Tensor> bias_grad(const Tensor& dy, const Tensor& z) {
  const int64_t rows = dy.size(0), C = dy.size(1);
  if (C % (128 * (16 / dy.element_size()))) {
    Tensor dz = z.defined() ? at::gelu_backward(dy, z) : dy;
    return {dz, dz.sum(0)};
  }
  Tensor scratch = at::empty({(int64_t)tmpi_bias_grad_scratch_bytes((int)C)}, dy.options().dtype(at::kByte));
  Tensor db = at::empty({C}, dy.options()), dz = z.defined() ? at::empty_like(dy) : dy;
  check(tmpi_bias_grad(dy.data_ptr(), z.defined() ? z.data_ptr() : nullptr, z.defined() ? dz.data_ptr() : nullptr, db.data_ptr(), (int)rows,
                       (int)C, dtype_code(dy.scalar_type()), scratch.data_ptr(), stream()));
  launched(LINEAR, 2);
  return {dz, db};
}

// Arrival counters for linear_bwd.cu
Tensor arrival_counters(const Tensor& like, int64_t counters) {
  static auto& kept = *new KeptZeros;
  return kept.get(like, sizeof(unsigned) * (size_t)counters, tmpi_gemm_failures());
}

// dX = dY W, dW = dY^T X and db = column sums of dY, those that are wanted, in one launch; dY may have a row pitch
void linear_gradients(const Tensor& dy, const Tensor& x, const Tensor& w, Tensor* dx, Tensor* dw, Tensor* db) {
  const int rows = (int)x.size(0), in = (int)x.size(1), out = (int)w.size(0), want = (dx ? 1 : 0) | (dw ? 2 : 0) | (db ? 4 : 0);
  size_t bytes = 0;
  int counters = 0;
  check(tmpi_linear_bwd_plan(rows, in, out, want, 0, &bytes, &counters));
  Tensor ws, arrivals;
  if (bytes) ws = at::empty({(int64_t)bytes}, dy.options().dtype(at::kByte));
  if (counters) arrivals = arrival_counters(dy, counters);
  if (dx) *dx = at::empty({rows, in}, dy.options());
  if (dw) *dw = at::empty({out, in}, dy.options());
  if (db) *db = at::empty({out}, dy.options());
  check(tmpi_linear_bwd(dy.data_ptr(), rows > 1 ? dy.stride(0) : 0, x.data_ptr(), w.data_ptr(), dx ? dx->data_ptr() : nullptr, dw ? dw->data_ptr() : nullptr,
                        db ? db->data_ptr() : nullptr, rows, in, out, 0, bytes ? ws.data_ptr() : nullptr, bytes,
                        counters ? arrivals.data_ptr() : nullptr, counters, stream()));
  launched(LINEAR, 1);
}

// dy * gelu'(z)
Tensor gelu_gradient(const Tensor& dy, const Tensor& z) {
  Tensor dz = at::empty_like(dy);
  check(tmpi_gelu_bwd(dy.data_ptr(), z.data_ptr(), dz.data_ptr(), (size_t)dy.numel(), dtype_code(dy.scalar_type()), stream()));
  launched(LINEAR, 1);
  return dz;
}

struct LinearFn : public torch::autograd::Function<LinearFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const c10::optional<Tensor>& bias_, bool with_gelu,
                        const c10::optional<Tensor>& residual) {
    const Tensor bias = bias_.has_value() ? *bias_ : Tensor();
    Tensor x2 = x.reshape({-1, x.size(-1)}), y, z;
    if (!(w.dim() == 2 && w.is_cuda() && w.size(1) == x2.size(1)))
      throw std::invalid_argument("matmul_nt expects bf16 CUDA matrices [M, K] and [N, K] with K a multiple of 8");
    if (with_gelu) std::tie(z, y) = matmul_nt_gelu(x2, w, bias);          // the pre-activation is needed by backward
    else if (residual.has_value()) y = matmul_nt_residual(x2, w, bias, residual->reshape({-1, w.size(0)}));
    else y = matmul_nt(x2, w, bias);
    ctx->save_for_backward({x2, w, z});
    ctx->saved_data["bias"] = bias.defined();
    ctx->saved_data["residual"] = residual.has_value();
    std::vector<int64_t> shape = x.sizes().vec();
    ctx->saved_data["shape"] = shape;
    shape.back() = w.size(0);
    return y.reshape(shape);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor x2 = as_saved(saved[0]), w = as_saved(saved[1]), z = as_saved(saved[2]);
    const Tensor& dy = grads[0];
    Tensor dy2 = packed(dy.reshape({-1, dy.size(-1)})), db, dx, dw;
    const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
    const Tensor dres = ctx->saved_data["residual"].toBool() ? dy : Tensor();               // the sum hands its gradient on as it is
    if ((need_x || need_w) && dy2.size(1) % 8 == 0 && pair_enabled()) {
      if (z.defined()) dy2 = gelu_gradient(dy2, z);
      const bool need_b = ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2);
      linear_gradients(dy2, x2, w, need_x ? &dx : nullptr, need_w ? &dw : nullptr, need_b ? &db : nullptr);
      if (need_x) dx = dx.view(ctx->saved_data["shape"].toIntVector());
      return {dx, dw, db, Tensor(), dres};
    }
    if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2)) std::tie(dy2, db) = bias_grad(dy2, z);
    else if (z.defined()) dy2 = at::gelu_backward(dy2, z);
    if (need_x) dx = matmul_nn(dy2, w).reshape(ctx->saved_data["shape"].toIntVector());
    if (need_w) dw = matmul_tn(dy2, x2);
    return {dx, dw, db, Tensor(), dres};
  }
};

// The head of ops/gemm.py (wide_head): x w^T for any number of outputs, in a buffer whose row pitch is the next multiple of 8, so that all
// three products run on the CTA-pair kernels with explicit pitches and no padding copies.
struct WideHeadFn : public torch::autograd::Function<WideHeadFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w) {
    const int64_t T = x.size(0), d = x.size(1), V = w.size(0), pitch = (V + 7) / 8 * 8;
    Tensor buf = at::empty({T, pitch}, x.options());
    check(tmpi_gemm_bf16_ex(x.data_ptr(), w.data_ptr(), buf.data_ptr(), nullptr, (int)T, (int)V, (int)d, d, d, pitch, 0, stream()));
    launched(LINEAR, 1);
    ctx->save_for_backward({x, w});
    return buf.narrow(1, 0, V);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor x = as_saved(saved[0]), w = as_saved(saved[1]);
    Tensor dl = grads[0], dx, dw;
    if (!(dl.stride(1) == 1 && dl.stride(0) % 8 == 0 && dl.stride(0) >= dl.size(1) && (uintptr_t)dl.data_ptr() % 16 == 0)) {
      Tensor padded = at::zeros({dl.size(0), (dl.size(1) + 7) / 8 * 8}, dl.options());
      dl = padded.narrow(1, 0, dl.size(1)).copy_(dl);
    }
    const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
    if (need_x || need_w) linear_gradients(dl, x, w, need_x ? &dx : nullptr, need_w ? &dw : nullptr, nullptr);
    return {dx, dw};
  }
};

// ---------------------------------------------------------------- layer norm
Tensor layer_norm_forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& bias, double eps) {
  const int64_t C = x.size(-1);
  const Tensor x2 = packed(x.reshape({-1, C})), g = packed(weight), b = packed(bias);
  const int64_t rows = x2.size(0);
  Tensor y = at::empty_like(x2), stats = at::empty({2, rows}, x.options().dtype(at::kFloat));      // mean, 1 / std
  float* mean = stats.data_ptr<float>();
  check(tmpi_layernorm_fwd(x2.data_ptr(), g.data_ptr(), b.data_ptr(), y.data_ptr(), mean, mean + rows, (int)rows, (int)C, (float)eps,
                           dtype_code(x.scalar_type()), stream()));
  launched(LAYERNORM, 1);
  ctx->save_for_backward({x2, g, stats});
  ctx->saved_data["shape"] = x.sizes().vec();
  return y.view(x.sizes());
}

// `add` (may be undefined): a gradient of x from elsewhere, added to dx
variable_list layer_norm_backward(AutogradContext* ctx, const Tensor& dy, const Tensor& add) {
  const auto saved = ctx->get_saved_variables();
  const Tensor x2 = as_saved(saved[0]), weight = as_saved(saved[1]), stats = as_saved(saved[2]);
  const int64_t rows = x2.size(0), C = x2.size(1);
  const Tensor dy2 = packed(dy.reshape({rows, C})), add2 = add.defined() ? packed(add.reshape({rows, C})) : add;
  Tensor dx = at::empty_like(x2), dgamma = at::empty_like(weight), dbeta = at::empty_like(weight);
  Tensor scratch = at::empty({(int64_t)tmpi_layernorm_scratch_bytes((int)C)}, x2.options().dtype(at::kByte));
  const float* mean = stats.data_ptr<float>();
  check(tmpi_layernorm_bwd_add(x2.data_ptr(), dy2.data_ptr(), add2.defined() ? add2.data_ptr() : nullptr, weight.data_ptr(), mean, mean + rows,
                               dx.data_ptr(), dgamma.data_ptr(), dbeta.data_ptr(), (int)rows, (int)C, dtype_code(x2.scalar_type()),
                               scratch.data_ptr(), stream()));
  launched(LAYERNORM, 2);
  return {dx.view(ctx->saved_data["shape"].toIntVector()), dgamma, dbeta, Tensor()};
}

struct LayerNormFn : public torch::autograd::Function<LayerNormFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& bias, double eps) {
    return layer_norm_forward(ctx, x, weight, bias, eps);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) { return layer_norm_backward(ctx, grads[0], Tensor()); }
};

// The layer norm of x and x itself, for a residual block whose identity takes the second output: the two gradients that reach x are
// added by the layer norm's kernel.
struct LayerNormForkFn : public torch::autograd::Function<LayerNormForkFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& bias, double eps) {
    ctx->set_materialize_grads(false);
    return {layer_norm_forward(ctx, x, weight, bias, eps), x};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (!grads[0].defined()) return {grads[1], Tensor(), Tensor(), Tensor()};
    return layer_norm_backward(ctx, grads[0], grads[1]);
  }
};

// ---------------------------------------------------------------- causal attention (head size 64, packed projection)
constexpr int64_t HEAD = 64;

struct AttentionFn : public torch::autograd::Function<AttentionFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, int64_t heads) {
    const int64_t B = qkv.size(0), T = qkv.size(1), C3 = qkv.size(2), C = C3 / 3;
    Tensor out = at::empty({B, T, C}, qkv.options()), lse = at::empty({B, heads, T}, qkv.options().dtype(at::kFloat));
    char* base = (char*)qkv.data_ptr();
    check(tmpi_attention_fwd(base, base + C * 2, base + 2 * C * 2, C3, out.data_ptr(), C, lse.data_ptr<float>(), (int)B, (int)T, (int)heads,
                             (float)(1.0 / std::sqrt((double)HEAD)), stream()));
    launched(ATTENTION, 1);
    ctx->save_for_backward({qkv, out, lse});
    ctx->saved_data["heads"] = heads;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor qkv = as_saved(saved[0]), out = as_saved(saved[1]), lse = as_saved(saved[2]);
    const int64_t heads = ctx->saved_data["heads"].toInt(), B = qkv.size(0), T = qkv.size(1), C3 = qkv.size(2), C = C3 / 3;
    const Tensor dout = grads[0].contiguous();
    Tensor dqkv = at::empty_like(qkv);
    Tensor dq_acc = at::empty({B * T, C}, lse.options()), delta = at::empty({B, heads, T}, lse.options());
    char *base = (char*)qkv.data_ptr(), *g = (char*)dqkv.data_ptr();
    check(tmpi_attention_bwd(base, base + C * 2, base + 2 * C * 2, C3, out.data_ptr(), C, dout.data_ptr(), C, lse.data_ptr<float>(),
                             delta.data_ptr<float>(), dq_acc.data_ptr<float>(), g, g + C * 2, g + 2 * C * 2, C3, (int)B, (int)T, (int)heads,
                             (float)(1.0 / std::sqrt((double)HEAD)), stream()));
    launched(ATTENTION, 1);
    launched(ATTENTION_BACKWARD, 1);
    return {dqkv, Tensor()};
  }
};

// ---------------------------------------------------------------- cross-entropy
// The arrival counter of the kernel's blocks and the row losses.  A call of very many rows clears a buffer of its own: the clearing
// costs nothing beside the pass and the buffer would be large to keep.
Tensor xent_scratch(const Tensor& x, int64_t rows) {
  static auto& kept = *new KeptZeros;                          // outlives the CUDA context: never destroyed
  return kept.get(x, tmpi_xent_scratch_bytes((int)rows));
}

// The gradient is computed with the loss and scaled in place by the incoming gradient, so backward runs once.
struct XentFn : public torch::autograd::Function<XentFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels, bool unit_grad) {
    const int64_t rows = logits.size(0), cols = logits.size(1);
    if (rows == 0) {                                            // the mean of no losses
      PyErr_SetString(PyExc_ZeroDivisionError, "cross_entropy: no rows");
      throw pybind11::error_already_set();
    }
    // rows may sit in a wider buffer: the kernel takes the pitch, and the gradient keeps it
    const bool pitched = logits.stride(1) == 1 && logits.stride(0) >= cols && rows > 1;
    const Tensor x = pitched ? logits : logits.contiguous();
    const int64_t ld = pitched ? logits.stride(0) : cols;
    const Tensor scratch = xent_scratch(x, rows);
    Tensor buf = at::empty({rows, ld}, x.options()), loss = at::empty({}, x.options().dtype(at::kFloat));
    check(tmpi_xent_mean_fwd_bwd_ld(x.data_ptr(), dtype_code(x.scalar_type()), labels.data_ptr<int64_t>(), (int)rows, (int)cols, (int)ld,
                                    loss.data_ptr<float>(), buf.data_ptr(), (float)(1.0 / (double)rows), scratch.data_ptr(), stream()));
    launched(XENT, 1);
    ctx->saved_data["buf"] = buf;
    ctx->saved_data["cols"] = cols;
    ctx->saved_data["unit"] = unit_grad;
    return loss;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    c10::IValue& kept = ctx->saved_data["buf"];
    TORCH_CHECK(kept.isTensor(), "cross_entropy: the gradient of this loss has been handed out already (backward runs once)");
    Tensor buf = kept.toTensor();
    kept = c10::IValue();
    if (!ctx->saved_data["unit"].toBool()) {
      check(tmpi_scale(buf.data_ptr(), (size_t)buf.numel(), dtype_code(buf.scalar_type()), grads[0].data_ptr<float>(), stream()));
      launched(XENT, 1);
    }
    return {buf.narrow(1, 0, ctx->saved_data["cols"].toInt()), Tensor(), Tensor()};
  }
};

// ---------------------------------------------------------------- batch norm and convolution of channels-last activations
// Sums the gradients that several consumers send into one activation inside their kernels: every consumer but the last parks its
// gradient here and returns none to autograd, the last one's kernel adds the parked sum.  A residual's gradient may be parked unwritten,
// as the incoming gradient and the ReLU's mask bits.  (GradFork of parallel/flat_buckets.py, for the functions below.)
struct Fork : torch::CustomClassHolder {
  int64_t consumers, seen = 0;
  Tensor parked, bits;
  explicit Fork(int64_t n) : consumers(n) {}
  bool parks_first() const { return seen == 0 && consumers > 1; }
  // make(add, bits): this consumer's gradient plus `add` (where its bit is set, if there are bits), when that is defined
  template <typename F> Tensor offer(F make) {
    ++seen;
    Tensor g = make(parked, bits);
    if (seen < consumers) {
      parked = g;
      bits = Tensor();
      return Tensor();
    }
    seen = 0;
    parked = bits = Tensor();
    return g;
  }
  void park_masked(const Tensor& grad, const Tensor& mask) {
    ++seen;
    parked = grad;
    bits = mask;
  }
};
using ForkPtr = c10::intrusive_ptr<Fork>;

c10::IValue keep_fork(const ForkPtr& f) { return f ? c10::IValue::make_capsule(f) : c10::IValue(); }
ForkPtr kept_fork(AutogradContext* ctx, const char* name) {
  const c10::IValue& v = ctx->saved_data[name];
  return v.isCapsule() ? c10::static_intrusive_pointer_cast<Fork>(v.toCapsule()) : ForkPtr();
}

Tensor channels_last(const Tensor& t) { return packed(t, at::MemoryFormat::ChannelsLast); }
Tensor empty_channels_last(at::IntArrayRef sizes, const Tensor& like) {
  return at::empty(sizes, like.options(), at::MemoryFormat::ChannelsLast);
}
const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
float* floats(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }

// the gradient where its mask bit is set
Tensor masked_tensor(const Tensor& grad, const Tensor& bits) {
  const int64_t per = grad.numel() / bits.numel(), N = grad.size(0), C = grad.size(1), H = grad.size(2), W = grad.size(3);      // elements of a byte
  const Tensor on = at::bitwise_and(at::bitwise_right_shift(bits.unsqueeze(1), at::arange(per, bits.options())), 1);
  return at::where(on.view({N, H, W, C}).permute({0, 3, 1, 2}).to(at::kBool), grad, at::zeros({}, grad.options()));
}

struct BnArgs { double eps, momentum; bool relu, training, keeps; int partial_rows; Tensor scratch; ForkPtr res_fork; };

struct BnFn : public torch::autograd::Function<BnFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const c10::optional<Tensor>& residual_, const Tensor& gamma, const Tensor& beta,
                        const c10::optional<Tensor>& running_mean, const c10::optional<Tensor>& running_var, const BnArgs& a) {
    const Tensor x = channels_last(x_), residual = residual_.has_value() ? channels_last(*residual_) : Tensor();
    const int64_t C = x.size(1), rows = x.size(0) * x.size(2) * x.size(3);
    Tensor y = empty_channels_last(x.sizes(), x), mean, invstd, bits;
    if (a.training) {
      mean = at::empty({2, C}, gamma.options());                       // and 1 / std behind it
      invstd = mean[1];
    } else {
      mean = running_mean->to(at::kFloat);
      invstd = at::rsqrt(running_var->to(at::kFloat) + a.eps);
    }
    // a ReLU layer with a residual keeps one mask bit per element for its backward (a sixteenth of y)
    if (a.relu && residual.defined() && a.keeps) bits = at::empty({rows * C / (16 / x.element_size())}, x.options().dtype(at::kByte));
    float *m = mean.data_ptr<float>(), *v = invstd.data_ptr<float>();
    const int type = dtype_code(x.scalar_type());
    float *rm = a.training && running_mean.has_value() ? floats(*running_mean) : nullptr, *rv = a.training && running_var.has_value() ? floats(*running_var) : nullptr;
    if (a.training && a.partial_rows > 0)
      check(tmpi_bn_relu_fwd_partials(x.data_ptr(), ptr(residual), y.data_ptr(), floats(gamma), floats(beta), rm, rv, m, v, rows, (int)C, (float)a.eps,
                                      (float)a.momentum, a.relu, type, (void*)ptr(bits), a.scratch.data_ptr(), a.partial_rows, stream()));
    else
      check(tmpi_bn_relu_fwd(x.data_ptr(), ptr(residual), y.data_ptr(), floats(gamma), floats(beta), rm, rv, m, v, rows, (int)C, (float)a.eps,
                             (float)a.momentum, a.relu, a.training, type, (void*)ptr(bits), a.scratch.data_ptr(), stream()));
    launched(BATCHNORM, !a.training ? 1 : a.partial_rows > 0 ? 2 : 3);
    // a ReLU layer without a residual rebuilds its mask from x in backward; neither kind reads y again
    const bool keep_y = a.relu && residual.defined() && !bits.defined();
    ctx->save_for_backward({x, keep_y ? y : Tensor(), gamma, beta, mean, a.training ? Tensor() : invstd, bits});
    ctx->saved_data["relu"] = a.relu;
    ctx->saved_data["residual"] = residual.defined();
    ctx->saved_data["fork"] = keep_fork(a.res_fork);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto cl = at::MemoryFormat::ChannelsLast;
    const Tensor x = as_saved(saved[0], cl), y = as_saved(saved[1], cl), mean = as_saved(saved[4]);
    const Tensor &gamma = saved[2], &beta = saved[3], &invstd = saved[5], &bits = saved[6];
    const Tensor dy = channels_last(grads[0]);
    const int64_t C = x.size(1), rows = x.size(0) * x.size(2) * x.size(3);
    const bool has_res = ctx->saved_data["residual"].toBool();
    const ForkPtr fork = kept_fork(ctx, "fork");
    // the first of several consumers of the residual parks its gradient for the last one's kernel: as dy and the mask bits
    const bool masked = has_res && bits.defined() && fork && fork->parks_first();
    Tensor dx = empty_channels_last(x.sizes(), x), dres = has_res && !masked ? empty_channels_last(x.sizes(), x) : Tensor();
    Tensor dgamma = at::empty({C}, gamma.options()), dbeta = at::empty({C}, gamma.options());
    const Tensor scratch = at::empty({(int64_t)tmpi_bn_scratch_bytes((int)C)}, x.options().dtype(at::kByte));
    check(tmpi_bn_relu_bwd_acc(x.data_ptr(), ptr(y), dy.data_ptr(), dx.data_ptr(), (void*)ptr(dres), floats(gamma), floats(beta), floats(mean),
                               invstd.defined() ? floats(invstd) : floats(mean) + C, floats(dgamma), floats(dbeta), rows, (int)C,
                               ctx->saved_data["relu"].toBool(), dtype_code(x.scalar_type()), ptr(bits), scratch.data_ptr(), nullptr, nullptr, stream()));
    launched(BATCHNORM, 3);
    if (masked) fork->park_masked(dy, bits);
    else if (dres.defined() && fork)
      dres = fork->offer([&](const Tensor& add, const Tensor& mask) { return add.defined() ? dres.add_(mask.defined() ? masked_tensor(add, mask) : add) : dres; });
    return {dx, dres, dgamma, dbeta, Tensor(), Tensor(), Tensor()};
  }
};

struct ConvArgs { int stride, pad; float* stats; int* rows; ForkPtr fork; };

struct ConvFn : public torch::autograd::Function<ConvFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x_, const Tensor& w_, const ConvArgs& a) {
    const Tensor x = channels_last(x_), w = channels_last(w_);
    const int64_t N = x.size(0), Cin = x.size(1), H = x.size(2), W = x.size(3), Cout = w.size(0), R = w.size(2), S = w.size(3);
    Tensor y = empty_channels_last({N, Cout, (H + 2 * a.pad - R) / a.stride + 1, (W + 2 * a.pad - S) / a.stride + 1}, x);
    int rows = 0;
    check(tmpi_conv_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), (int)N, (int)H, (int)W, (int)Cin, (int)Cout, (int)R, (int)S, a.stride, a.pad, a.stats,
                        &rows, stream()));
    launched(CONV, 1);
    if (a.rows) *a.rows = rows;
    ctx->save_for_backward({x, w});
    ctx->saved_data["stride"] = (int64_t)a.stride;
    ctx->saved_data["pad"] = (int64_t)a.pad;
    ctx->saved_data["fork"] = keep_fork(a.fork);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor x = channels_last(saved[0]), w = channels_last(saved[1]);
    const Tensor dy = channels_last(grads[0]);
    const int N = (int)x.size(0), Cin = (int)x.size(1), H = (int)x.size(2), W = (int)x.size(3), Cout = (int)w.size(0), R = (int)w.size(2), S = (int)w.size(3);
    const int stride = (int)ctx->saved_data["stride"].toInt(), pad = (int)ctx->saved_data["pad"].toInt();
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) {
      auto make = [&](Tensor add, Tensor bits) {
        if (bits.defined() && !(stride == 1 && add.sizes() == x.sizes() && add.scalar_type() == x.scalar_type() && (uintptr_t)add.data_ptr() % 16 == 0)) {
          add = masked_tensor(add, bits);
          bits = Tensor();
        }
        if (stride == 1) {
          if (add.defined()) add = channels_last(add);
          Tensor g = empty_channels_last(x.sizes(), dy);
          check(tmpi_conv_dgrad_masked(dy.data_ptr(), w.data_ptr(), g.data_ptr(), ptr(add), ptr(bits), N, H, W, Cin, Cout, R, S, 1, pad, stream()));
          launched(CONV, 1);
          return g;
        }
        Tensor g = std::get<0>(at::convolution_backward(dy, x, w, c10::nullopt, {stride, stride}, {pad, pad}, {1, 1}, false, {0, 0}, 1, {true, false, false}));
        return add.defined() ? g.add_(add) : g;                     // strided input gradients stay on the library
      };
      const ForkPtr fork = kept_fork(ctx, "fork");
      dx = fork ? fork->offer(make) : make(Tensor(), Tensor());
    }
    if (ctx->needs_input_grad(1)) {
      const size_t need = tmpi_conv_wgrad_workspace_bytes(N, H, W, Cin, Cout, R, S, stride, pad);
      const Tensor ws = at::empty({(int64_t)need}, x.options().dtype(at::kByte));
      dw = channels_last(at::empty(w.sizes(), x.options()));
      check(tmpi_conv_wgrad(dy.data_ptr(), x.data_ptr(), dw.data_ptr(), N, H, W, Cin, Cout, R, S, stride, pad, ws.data_ptr(), need, 0, stream()));
      launched(CONV, 2);
    }
    return {dx, dw, Tensor()};
  }
};

Tensor bn_relu(const Tensor& x, const c10::optional<Tensor>& residual, const Tensor& gamma, const Tensor& beta, const c10::optional<Tensor>& running_mean,
               const c10::optional<Tensor>& running_var, double eps, double momentum, bool relu, bool training, const ForkPtr& res_fork, int partial_rows,
               Tensor scratch) {
  auto wants = [](const Tensor& t) { return t.requires_grad(); };
  const bool keeps = at::GradMode::is_enabled() && (wants(x) || wants(gamma) || wants(beta) || (residual.has_value() && wants(*residual)));
  if (!scratch.defined()) scratch = at::empty({(int64_t)tmpi_bn_scratch_bytes((int)x.size(1))}, x.options().dtype(at::kByte));
  if (!training && !(running_mean.has_value() && running_var.has_value()))
    throw std::invalid_argument("batch norm: evaluation needs running statistics");
  return BnFn::apply(x, residual, gamma, beta, running_mean, running_var,
                     BnArgs{eps, momentum, relu, training, keeps, partial_rows, scratch, res_fork});
}

// ---------------------------------------------------------------- the ResNet stem's convolution
struct StemFn : public torch::autograd::Function<StemFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w) {
    const int64_t N = x.size(0), H = x.size(2), W = x.size(3);
    Tensor y = empty_channels_last({N, w.size(0), (H - 1) / 2 + 1, (W - 1) / 2 + 1}, x);
    check(tmpi_stem_conv_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), (int)N, (int)H, (int)W, (int)w.size(0), w.strides().data(), stream()));
    launched(STEM, 1);
    ctx->save_for_backward({x});                                 // nothing but the image is kept
    ctx->saved_data["shape"] = w.sizes().vec();
    ctx->saved_data["strides"] = w.strides().vec();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor x = channels_last(saved[0]);
    const Tensor dy = channels_last(grads[0]);
    const std::vector<int64_t> shape = ctx->saved_data["shape"].toIntVector(), strides = ctx->saved_data["strides"].toIntVector();
    Tensor dw = at::empty_strided(shape, strides, x.options());
    // partial sums of the CTAs (24 MB), from the allocator: calls on other streams, threads and in graphs have their own
    const size_t need = tmpi_stem_conv_wgrad_workspace_bytes();
    const Tensor ws = at::empty({(int64_t)need}, x.options().dtype(at::kByte));
    check(tmpi_stem_conv_wgrad(dy.data_ptr(), x.data_ptr(), dw.data_ptr(), (int)x.size(0), (int)x.size(2), (int)x.size(3), (int)shape[0], strides.data(),
                               ws.data_ptr(), need, stream()));
    launched(STEM, 2);
    return {Tensor(), dw};
  }
};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("linear", [](const Tensor& x, const Tensor& w, const c10::optional<Tensor>& bias, bool gelu) {
    return LinearFn::apply(x, w, bias, gelu, c10::optional<Tensor>());      // an input without a tensor has to be a nullopt: apply asks every Tensor for its device
  });
  m.def("linear_add", [](const Tensor& x, const Tensor& w, const c10::optional<Tensor>& bias, const Tensor& residual) {
    return LinearFn::apply(x, w, bias, false, c10::optional<Tensor>(residual));
  });
  m.def("wide_head", [](const Tensor& x, const Tensor& w) { return WideHeadFn::apply(x, w); });
  m.def("layer_norm_fork", [](const Tensor& x, const Tensor& w, const Tensor& b, double eps) { return LayerNormForkFn::apply(x, w, b, eps); });
  m.def("layer_norm", [](const Tensor& x, const Tensor& w, const Tensor& b, double eps) { return LayerNormFn::apply(x, w, b, eps); });
  m.def("causal_attention", [](const Tensor& qkv, int64_t heads) { return AttentionFn::apply(qkv, heads); });
  m.def("cross_entropy", [](const Tensor& logits, const Tensor& labels, bool unit_grad) {
    return XentFn::apply(logits, labels, unit_grad);
  });
  pybind11::class_<Fork, ForkPtr>(m, "Fork").def(pybind11::init([](int64_t n) { return c10::make_intrusive<Fork>(n); })).def_readwrite("consumers", &Fork::consumers);
  m.def("bn_relu", [](const Tensor& x, const c10::optional<Tensor>& residual, const Tensor& gamma, const Tensor& beta, const c10::optional<Tensor>& rm,
                      const c10::optional<Tensor>& rv, double eps, double momentum, bool relu, bool training, const ForkPtr& res_fork) {
    return bn_relu(x, residual, gamma, beta, rm, rv, eps, momentum, relu, training, res_fork, 0, Tensor());
  });
  m.def("stem_conv", [](const Tensor& x, const Tensor& w) { return StemFn::apply(x, w); });
  m.def("conv2d", [](const Tensor& x, const Tensor& w, int stride, int pad, const ForkPtr& fork) {
    return ConvFn::apply(x, w, ConvArgs{stride, pad, nullptr, nullptr, fork});
  });
  // bn(conv(x), residual) in training: the convolution's epilogue leaves the partial sums of its output's statistics
  m.def("conv_bn", [](const Tensor& x, const Tensor& w, int stride, int pad, const c10::optional<Tensor>& residual, const Tensor& gamma, const Tensor& beta,
                      const c10::optional<Tensor>& rm, const c10::optional<Tensor>& rv, double eps, double momentum, bool relu, const ForkPtr& fork,
                      const ForkPtr& res_fork) {
    const Tensor scratch = at::empty({(int64_t)tmpi_bn_scratch_bytes((int)w.size(0))}, x.options().dtype(at::kByte));
    int rows = 0;
    const Tensor y = ConvFn::apply(x, w, ConvArgs{stride, pad, (float*)scratch.data_ptr(), &rows, fork});
    return bn_relu(y, residual, gamma, beta, rm, rv, eps, momentum, relu, true, res_fork, rows, scratch);
  });
  m.def("cross_entropy_scratch", xent_scratch);
  m.def("arrival_counters", arrival_counters);
  m.def("launches", [](int what) { return g_launches[what].load(std::memory_order_relaxed); });
}
