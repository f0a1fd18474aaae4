// One GCN layer, forward and backward, and its autograd node.
//
// Reference math (src/graphcuda/cuda/gcn.cu:5-52, twin src/graphcuda/cpp/gcn.cpp:4-41):
//   forward   Y  = relu((A X) W)
//   backward  G  = dY * mask;  dW = (A X)^T G;  dX = A (G W^T)
// The reference always aggregates first and recomputes A X in the backward pass.  Here the aggregation runs on the
// narrower side -- (A X) W when in <= out, A (X W) when out < in and A is symmetric -- the intermediate is kept for
// the backward pass, ReLU / bias / mask are fused into the producing kernel, transposed operands are read in place,
// and dX is skipped when nobody needs it.  For a non-symmetric A the aggregate-first order is always used, so the
// results are the reference's (including its use of A rather than A^T for dX, gcn.cu:49).
#include <torch/csrc/autograd/custom_function.h>

#include "host.h"

namespace gch {

namespace {
// Transform-first layers with an output width that is not a multiple of 4 (47 classes) run on a zero-padded width so
// every row pitch is 16-byte aligned (vector gathers in the aggregation, TMA in the tensor-core GEMMs).  Small
// problems are not worth the copies.
constexpr int64_t kPadMinWork = int64_t(1) << 27;

struct PadEntry {
  void* ptr;
  c10::weak_intrusive_ptr<c10::StorageImpl> storage;
  int64_t rows, width;
};
std::mutex pad_mutex;
std::vector<PadEntry>& pad_entries() {
  static auto* v = new std::vector<PadEntry>();
  return *v;
}
void drop_expired() {
  auto& v = pad_entries();
  v.erase(std::remove_if(v.begin(), v.end(), [](const PadEntry& e) { return e.storage.expired(); }), v.end());
}

void check_args(const Tensor& X, const Adj& a, const Tensor& W) {
  require(X.dim() == 2 && W.dim() == 2, "Inputs must be 2D");
  require(X.is_cuda() && W.is_cuda(), "Inputs must be CUDA tensors");
  require(X.scalar_type() == at::kFloat && W.scalar_type() == at::kFloat, "Only float32 is supported here");
  require(a.K == X.size(0), "A.cols must match B.rows");
  require(X.size(1) == W.size(0), "A.cols must match B.rows");
  require(X.device() == a.device() && W.device() == X.device(), "A and B must be CUDA tensors on the same device");
}

Tensor pad_cols(const Tensor& t, int64_t width) {
  if (t.size(-1) == width) return t;
  if (OptTensor base = zero_padded_base(t, width)) return *base;
  if (t.dim() == 2 && t.scalar_type() == at::kFloat && t.stride(1) == 1 && t.stride(0) >= t.size(1) &&
      width % 4 == 0 && t.size(0) > 0) {
    const c10::cuda::CUDAGuard guard(t.device());
    Tensor out = empty_f32(t.size(0), width, t.device());  // one launch instead of a fill and a copy
    check(abi.gc_pad_rows_f32(t.const_data_ptr<float>(), ld_of(t), out.data_ptr<float>(), width, t.size(0), t.size(1),
                              stream_of(t.device())),
          "gc_pad_rows_f32");
    return out;
  }
  auto shape = t.sizes().vec();
  shape.back() = width;
  Tensor out = at::zeros(shape, t.options());
  out.narrow(-1, 0, t.size(-1)).copy_(t);
  return out;
}

// For a product that is aggregated next: rows on a 16-byte pitch, so that an odd width is still gathered in vectors.
Tensor product_to_gather(Tensor A, Tensor B, bool tb, int prec) {
  const Mat a = as_operand(A);
  Mat b = as_operand(B);
  if (tb) b = b.t();
  const int64_t n = b.cols, ld = (n + 3) / 4 * 4;
  Tensor out = empty_f32(a.rows, ld, A.device());
  gemm_into(a, b, out.data_ptr<float>(), std::max<int64_t>(ld, 1), Epi{}, false, prec, A.device());
  return ld == n ? out : out.narrow(1, 0, n);
}

Tensor product(Tensor A, Tensor B, bool ta, bool tb, int prec, const Epi& ep) {
  Mat a = as_operand(A), b = as_operand(B);
  if (ta) a = a.t();
  if (tb) b = b.t();
  Tensor out = empty_f32(a.rows, b.cols, A.device());
  gemm_into(a, b, out.data_ptr<float>(), std::max<int64_t>(b.cols, 1), ep, false, prec, A.device());
  return out;
}
}  // namespace

void register_zero_padded(const Tensor& buf) {
  std::lock_guard<std::mutex> lock(pad_mutex);
  drop_expired();
  pad_entries().push_back(PadEntry{buf.data_ptr(), buf.storage().getWeakStorageImpl(), buf.size(0), buf.size(1)});
}

OptTensor zero_padded_base(const Tensor& t, int64_t width) {
  if (t.dim() != 2 || t.stride(1) != 1 || t.stride(0) != width) return std::nullopt;
  std::lock_guard<std::mutex> lock(pad_mutex);
  for (const PadEntry& e : pad_entries()) {
    if (e.ptr != t.data_ptr() || e.rows != t.size(0) || e.width != width) continue;
    const auto s = e.storage.lock();
    if (s && s.get() == t.storage().unsafeGetStorageImpl()) return t.as_strided({e.rows, width}, {width, 1});
  }
  return std::nullopt;
}

int64_t zero_padded_count() {
  std::lock_guard<std::mutex> lock(pad_mutex);
  drop_expired();
  return int64_t(pad_entries().size());
}

int64_t padded_width(int64_t n_rows, int64_t in_dim, int64_t out_dim) {
  if (out_dim % 4 == 0 || n_rows * in_dim * out_dim < kPadMinWork) return out_dim;
  return (out_dim + 3) / 4 * 4;
}

// bf16 tier: whether the aggregation gathers a bf16 copy of H (half the bytes through the SM fill path, fp32 sums).  126 M
// non-zeros, F = 256: 5.9 ms + 0.6 ms for the copy against 8.7 ms.  Sparser matrices do not repay the conversion pass, and
// neither do small ones while fp32 has the mappings for few pieces that bf16 lacks (gc_spmm_csr_f32: up to 256 columns).
// Measured, time of copy and product over time of the fp32 product, at 17 to 80 non-zeros per row:
//   F = 128          2.6..1.4 to 20 K rows, 1.1..1.45 at 30 K, 0.9..1.5 at 40 K, 0.9..1.04 at 60 K, 0.8..1.05 above
//   F = 136 to 256   2.2..1.15 to 170 K non-zeros, 1.1..1.0 at 220..330 K, 0.8..1.05 at 340..510 K, 0.7..1.03 above
//   F = 264 to 384   1.25..1.0 to 820 K, 0.8..0.97 above
//   F = 448 to 1024  0.6..0.97 (1.05 at worst: 640 columns on 1 K rows, 40 K rows at 17 per row)
static bool bf16_gathers_pay(int64_t F, const Adj& a) {
  if (F < 128 || F % 8 != 0 || a.nnz < 16 * a.K) return false;
  if (F < 136) return a.M > 50000;
  if (F <= 256) return a.nnz >= 3 << 17;
  return F > 384 || a.nnz >= 13 << 16;
}

Tensor adj_matmul(Adj& a, Tensor H, int prec, const Epi& ep) {
  Tensor out = empty_f32(a.M, H.size(1), H.device());
  const int64_t F = H.size(1), ldy = std::max<int64_t>(F, 1);
  if (a.M == 0 || F == 0) return out;
  if (a.dense) {
    if (prec == GC_PREC_BF16 && !ep.mask) {
      // the adjacency does not change between calls: its owner keeps one bf16 copy of it (A16)
      const Tensor A16 = a.A16.defined() ? a.A16 : to_bf16(a.A, false);
      gemm_bf16_into(A16, to_bf16(H, true), out.data_ptr<float>(), ldy, ep, H.device());
    } else {
      Tensor A = a.A;
      const Mat ma = as_operand(A);
      gemm_into(ma, as_operand(H), out.data_ptr<float>(), ldy, ep, false, prec, H.device());
    }
    return out;
  }
  if (H.stride(1) != 1 || (H.size(0) > 1 && H.stride(0) < F)) H = H.contiguous();
  if (prec == GC_PREC_BF16 && bf16_gathers_pay(F, a)) {
    spmm_into(a, to_bf16(H, false), out.data_ptr<float>(), ldy, ep, false, 0);
  } else {
    spmm_into(a, H, out.data_ptr<float>(), ldy, ep, false, 0);
  }
  return out;
}

Forward layer_forward(const Tensor& X, Adj& a, const Tensor& W, const OptTensor& bias, bool relu, bool want_mask,
                      int prec) {
  check_args(X, a, W);
  const c10::cuda::CUDAGuard guard(X.device());
  const int64_t in = W.size(0), out_dim = W.size(1);
  Forward f;
  Epi ep;
  ep.relu = relu;
  Tensor b;
  if (bias && bias->defined()) {
    require(f32_on(*bias, X.device()) && bias->numel() == out_dim, "bias must be float32 [N] on the input's device");
    b = bias->contiguous();
    ep.bias = b.const_data_ptr<float>();
  }
  if (!(out_dim < in && a.is_symmetric())) {
    f.inter = adj_matmul(a, X, prec, Epi{});
    if (want_mask) {
      f.mask = empty_f32(a.M, out_dim, X.device());
      ep.mask = f.mask.data_ptr<float>();
    }
    f.Y = product(f.inter, W, false, false, prec, ep);
    return f;
  }
  const int64_t width = padded_width(X.size(0), in, out_dim);
  if (width != out_dim && b.defined()) {
    b = pad_cols(b, width);
    ep.bias = b.const_data_ptr<float>();
  }
  const Tensor H = product_to_gather(X, pad_cols(W, width), false, prec);
  if (want_mask) {
    f.mask = empty_f32(a.M, width, X.device());
    ep.mask = f.mask.data_ptr<float>();
  }
  f.Y = adj_matmul(a, H, prec, ep);
  if (width != out_dim) {  // views on the padded buffers; the pad columns hold zeros
    f.Y = f.Y.narrow(1, 0, out_dim);
    if (want_mask) f.mask = f.mask.narrow(1, 0, out_dim);
  }
  return f;
}

Tensor relu_backward(const Tensor& dYin, const Tensor& Yin) {
  require(dYin.dim() == 2 && dYin.sizes() == Yin.sizes() && dYin.is_cuda() && f32_on(dYin, Yin.device()) &&
              f32_on(Yin, dYin.device()),
          "relu_backward: two float32 CUDA matrices of one shape on one device expected");
  const Tensor dY = row_major(dYin), Y = row_major(Yin);
  const c10::cuda::CUDAGuard guard(dY.device());
  const int64_t M = dY.size(0), N = dY.size(1);
  Tensor G = empty_f32(M, N, dY.device());
  check(abi.gc_relu_backward_f32(dY.const_data_ptr<float>(), ld_of(dY), Y.const_data_ptr<float>(), ld_of(Y),
                                 G.data_ptr<float>(), std::max<int64_t>(N, 1), M, N, stream_of(dY.device())),
        "gc_relu_backward_f32");
  return G;
}

// The column sums of G; with Y, G is first multiplied by (Y > 0), in the same pass.
static Tensor bias_gradient(Tensor& G, const Tensor& Yin) {
  const int64_t M = G.size(0), N = G.size(1);
  const at::Device dev = G.device();
  Tensor db = at::empty({N}, at::TensorOptions().dtype(at::kFloat).device(dev));
  const Scratch ws = scratch(kSpmm, abi.gc_relu_bias_backward_workspace_bytes(M, N), dev);
  const Tensor dY = row_major(G);
  const bool masked = Yin.defined();
  const Tensor Y = masked ? row_major(Yin) : Tensor();
  Tensor out = masked ? empty_f32(M, N, dev) : Tensor();
  check(abi.gc_relu_bias_backward_f32(dY.const_data_ptr<float>(), ld_of(dY), masked ? Y.const_data_ptr<float>() : nullptr,
                                      masked ? ld_of(Y) : 0, masked ? out.data_ptr<float>() : nullptr,
                                      std::max<int64_t>(N, 1), M, N, db.data_ptr<float>(), ws.ptr, ws.bytes,
                                      stream_of(dev)),
        "gc_relu_bias_backward_f32");
  if (masked) G = out;
  return db;
}

Tensor mask_mul(const Tensor& dYin, const Tensor& maskin) {
  require(dYin.dim() == 2 && dYin.sizes() == maskin.sizes() && dYin.is_cuda() && f32_on(dYin, maskin.device()) &&
              f32_on(maskin, dYin.device()),
          "mask_mul: two float32 CUDA matrices of one shape on one device expected");
  const Tensor dY = row_major(dYin), mask = row_major(maskin);
  const c10::cuda::CUDAGuard guard(dY.device());
  const int64_t M = dY.size(0), N = dY.size(1);
  Tensor G = empty_f32(M, N, dY.device());
  check(abi.gc_mask_mul_f32(dY.const_data_ptr<float>(), ld_of(dY), mask.const_data_ptr<float>(), ld_of(mask),
                            G.data_ptr<float>(), std::max<int64_t>(N, 1), M, N, stream_of(dY.device())),
        "gc_mask_mul_f32");
  return G;
}

// Y is the saved activation (the ReLU mask is re-derived from it as Y > 0).
//
// Cross-layer fusion of the ReLU backward (reference gcn.cu:36): when this layer's input X is itself the ReLU output
// of the layer below (gate_dx), dX is multiplied by (X > 0) in the store of the kernel that produces it -- which is
// exactly the masking the layer below would do on its incoming gradient; that layer is then told its gradient arrives
// gated (grad_is_gated) and skips the separate pass.
Grads layer_backward(Tensor G, const Tensor& X, Adj& a, const Tensor& W, bool relu, const Tensor& Y,
                     const Tensor& inter, bool need_dX, bool need_dW, bool need_db, int prec, bool grad_is_gated,
                     bool gate_dx) {
  const c10::cuda::CUDAGuard guard(X.device());
  if (G.stride(1) != 1) G = G.contiguous();  // rows may keep a larger pitch (a padded gradient from the fused loss)
  Grads r;
  if (need_db) r.db = bias_gradient(G, relu && !grad_is_gated ? Y : Tensor());
  else if (relu && !grad_is_gated) G = relu_backward(G, Y);
  Epi gate;
  const bool fused_gate = gate_dx && need_dX && X.is_contiguous();
  if (fused_gate) gate.gate = X.const_data_ptr<float>();
  const int64_t out_dim = W.size(1);
  if (inter.defined()) {
    if (need_dW) r.dW = product(inter, G, true, false, prec, Epi{});
    // A, not A^T: reference gcn.cu:49
    if (need_dX) r.dX = adj_matmul(a, product_to_gather(G, W, true, prec), prec, gate);
  } else {
    // Y = A (X W), A symmetric: S = A^T G = A G
    const int64_t width = padded_width(X.size(0), W.size(0), out_dim);
    const Tensor S = adj_matmul(a, pad_cols(G, width), prec, Epi{});
    if (need_dW) {
      r.dW = product(X, S, true, false, prec, Epi{});
      if (width != out_dim) r.dW = r.dW.narrow(1, 0, out_dim);
    }
    if (need_dX) r.dX = product(S, pad_cols(W, width), false, true, prec, gate);
  }
  if (gate_dx && need_dX && !fused_gate) r.dX = relu_backward(r.dX, X);  // non-contiguous input: separate pass
  return r;
}

// Y = relu((adjm @ X) @ weights [+ bias]).  Unlike the reference (python/gcn.py:18) the fp32 mask is not materialised:
// the activation itself is saved and the mask re-derived as Y > 0; the aggregated features are saved instead of being
// recomputed (gcn.cu:40).
namespace {
struct ConvFunction : torch::autograd::Function<ConvFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& X, const Tensor& W, const OptTensor& bias,
                        const AdjPtr& a, int64_t flags, int64_t prec) {
    Forward f = layer_forward(X, *a, W, bias, flags & 1, false, int(prec));
    ctx->save_for_backward({X, W, f.Y, f.inter});
    ctx->saved_data["adj"] = c10::IValue::make_capsule(a);
    // bit 0: ReLU; bit 1: the incoming gradient is already gated; bit 2: gate dX by (X > 0); bit 3: bias
    ctx->saved_data["opt"] = (prec << 8) | flags | (bias && bias->defined() ? 8 : 0);
    return f.Y;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto adj = ctx->saved_data["adj"].toCapsule();
    const int64_t opt = ctx->saved_data["opt"].toInt();
    const bool has_bias = opt & 8;
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    Grads g = layer_backward(grads[0], saved[0], *static_cast<Adj*>(adj.get()), saved[1], opt & 1, saved[2], saved[3],
                             ctx->needs_input_grad(0), ctx->needs_input_grad(1),
                             has_bias && ctx->needs_input_grad(2), int(opt >> 8), opt & 2, opt & 4);
    return {g.dX, g.dW, g.db, Tensor(), Tensor(), Tensor()};
  }
};
}  // namespace

// fuse: bit 0 = the incoming gradient is already multiplied by this layer's ReLU mask;
//       bit 1 = X is the ReLU output of the layer below: gate dX by (X > 0) where it is produced
Tensor conv(const Tensor& X, const AdjPtr& a, const Tensor& W, const OptTensor& bias, bool relu, int64_t prec,
            int64_t fuse) {
  const bool has_bias = bias && bias->defined();
  // A tangent goes to the autograd node too: it has no forward-mode rule and says so, where the plain call below would
  // drop the tangent.
  const auto dual = [](const Tensor& t) { return t._fw_grad(0).defined(); };
  const bool record = (c10::GradMode::is_enabled() &&
                       (X.requires_grad() || W.requires_grad() || (has_bias && bias->requires_grad()))) ||
                      dual(X) || dual(W) || (has_bias && dual(*bias));
  if (!record) return layer_forward(X, *a, W, bias, relu, false, int(prec)).Y;
  return ConvFunction::apply(X, W, bias, a, (relu ? 1 : 0) | ((fuse & 3) << 1), prec);
}

}  // namespace gch
