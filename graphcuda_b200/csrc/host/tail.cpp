// The classification tail and the optimizers of the training scripts
// (reference tests/gcn/graphcuda_impl.py:24,45,55-56,63-68).
#include <torch/csrc/autograd/custom_function.h>

#include <vector>

#include "host.h"

namespace gch {

namespace {
// One byte per row, non-zero where the row counts; bool and uint8 selections are used as they are.
Tensor bytes_of(const Tensor& m) {
  if (m.scalar_type() == at::kBool || m.scalar_type() == at::kByte) return m.contiguous();
  return m.to(at::kByte).contiguous();
}
}  // namespace

NllForward nll_forward(const Tensor& Zin, const Tensor& labels, const OptTensor& row_mask, double scale) {
  require(Zin.dim() == 2 && Zin.is_cuda() && Zin.scalar_type() == at::kFloat, "logits must be a float32 CUDA matrix");
  require(labels.device() == Zin.device() && labels.scalar_type() == at::kLong && labels.numel() == Zin.size(0),
          "labels must be a CUDA int64 vector with one entry per row, on the logits' device");
  NllForward f;
  f.masked = row_mask && row_mask->defined();
  Tensor mask8;
  if (f.masked) {
    require(row_mask->device() == Zin.device() && row_mask->numel() == Zin.size(0),
            "row_mask must have one entry per row, on the logits' device");
    mask8 = bytes_of(*row_mask);
  }
  f.Z = Zin.stride(1) == 1 ? Zin : Zin.contiguous();
  f.labels = labels.contiguous();
  const int64_t M = f.Z.size(0), C = f.Z.size(1);
  const at::Device dev = f.Z.device();
  const c10::cuda::CUDAGuard guard(dev);
  const size_t wsb = std::max<size_t>(abi.gc_nll_workspace_bytes(M), 4);
  f.ws = at::empty({int64_t(wsb)}, at::TensorOptions().dtype(at::kByte).device(dev));
  f.loss = at::empty({}, at::TensorOptions().dtype(at::kFloat).device(dev));
  check(abi.gc_logsoftmax_nll_forward_f32(
            f.Z.const_data_ptr<float>(), M > 1 ? f.Z.stride(0) : std::max<int64_t>(C, 1),
            f.labels.const_data_ptr<int64_t>(), f.masked ? static_cast<const uint8_t*>(mask8.data_ptr()) : nullptr, M, C,
            float(scale), f.loss.data_ptr<float>(), f.ws.data_ptr(), wsb, stream_of(dev)),
        "gc_logsoftmax_nll_forward_f32");
  return f;
}

// masked: the rows are those of the forward pass's selection, of which the workspace holds a copy
Tensor nll_backward(const Tensor& grad, const Tensor& Z, const Tensor& labels, const Tensor& ws, bool masked,
                    double scale) {
  const int64_t M = Z.size(0), C = Z.size(1);
  const at::Device dev = Z.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t ldz = M > 1 ? Z.stride(0) : std::max<int64_t>(C, 1);
  int64_t lddz = std::max<int64_t>(C, 1);
  Tensor dZ;
  if (M > 1 && C < ldz && ldz <= C + 3 && ldz % 4 == 0 && reinterpret_cast<uintptr_t>(Z.data_ptr()) % 16 == 0) {
    // The logits are a view of a matrix padded to 16-byte rows (an odd class count): give the gradient the same
    // pitch with zero pad columns, so the layer below can aggregate it without re-padding a copy.
    lddz = ldz;
    Tensor buf = empty_f32(M, ldz, dev);
    register_zero_padded(buf);
    dZ = buf.narrow(1, 0, C);
  } else {
    dZ = empty_f32(M, C, dev);
  }
  const Tensor g = grad.to(at::kFloat).contiguous();
  const uint8_t* mask =
      masked ? static_cast<const uint8_t*>(ws.data_ptr()) + abi.gc_nll_workspace_bytes(M) - M : nullptr;
  check((lddz == C ? abi.gc_logsoftmax_nll_backward_f32 : abi.gc_logsoftmax_nll_backward_pad_f32)(
            Z.const_data_ptr<float>(), ldz, labels.const_data_ptr<int64_t>(), mask, M, C, float(scale),
            g.const_data_ptr<float>(), dZ.data_ptr<float>(), lddz, ws.data_ptr(), stream_of(dev)),
        "gc_logsoftmax_nll_backward_f32");
  return dZ;
}

namespace {
struct NllFunction : torch::autograd::Function<NllFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& Z, const Tensor& labels,
                        const OptTensor& row_mask, double scale) {
    const NllForward f = nll_forward(Z, labels, row_mask, scale);
    ctx->save_for_backward({f.Z, f.labels, f.ws});
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["masked"] = f.masked;
    return f.loss;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    return {nll_backward(grads[0], saved[0], saved[1], saved[2], ctx->saved_data["masked"].toBool(),
                         ctx->saved_data["scale"].toDouble()),
            Tensor(), Tensor(), Tensor()};
  }
};

}  // namespace

Tensor nll_loss(const Tensor& Z, const Tensor& labels, const OptTensor& row_mask, double scale) {
  return NllFunction::apply(Z, labels, row_mask, scale);
}

std::pair<Tensor, Tensor> argmax_accuracy(const Tensor& logits, const OptTensor& labels_in,
                                          const std::optional<std::vector<Tensor>>& masks, bool want_pred) {
  require(logits.is_cuda() && logits.dim() == 2 && logits.scalar_type() == at::kFloat,
          "argmax_accuracy: float32 CUDA matrix expected");
  const Tensor Z = (logits.stride(1) == 1 || logits.size(1) == 1) ? logits : logits.contiguous();
  const int64_t M = Z.size(0), C = Z.size(1);
  const at::Device dev = Z.device();
  const c10::cuda::CUDAGuard guard(dev);
  const bool labelled = labels_in && labels_in->defined();
  Tensor labels;
  std::vector<Tensor> rows;
  const uint8_t* list[8] = {};
  if (masks) {
    require(labelled, "argmax_accuracy: masks need labels");
    require(masks->size() >= 1 && masks->size() <= 8, "argmax_accuracy: between 1 and 8 row selections");
    for (const Tensor& m : *masks) {
      require(m.numel() == M && m.device() == dev,
              "argmax_accuracy: every selection needs one entry per row, on the logits' device");
      const bool bytes = m.scalar_type() == at::kBool || m.scalar_type() == at::kByte;
      rows.push_back((bytes ? m : m.ne(0)).contiguous());
      list[rows.size() - 1] = static_cast<const uint8_t*>(rows.back().data_ptr());
    }
  }
  const int n_masks = int(rows.size());
  if (labelled) {
    require(labels_in->scalar_type() == at::kLong && labels_in->numel() == M && labels_in->device() == dev,
            "argmax_accuracy: labels must be int64 [M] on the logits' device");
    labels = labels_in->contiguous();
  }
  Tensor pred, counts;
  const auto i64 = at::TensorOptions().dtype(at::kLong).device(dev);
  if (want_pred) pred = at::empty({M}, i64);
  if (labelled) counts = at::empty({std::max(n_masks, 1), 2}, i64);
  check(abi.gc_argmax_accuracy_masks_f32(Z.const_data_ptr<float>(), M > 1 ? Z.stride(0) : std::max<int64_t>(C, 1), M, C,
                                   labelled ? labels.const_data_ptr<int64_t>() : nullptr,
                                   list, n_masks,
                                   want_pred ? pred.data_ptr<int64_t>() : nullptr,
                                   labelled ? counts.data_ptr<int64_t>() : nullptr, stream_of(dev)),
        "gc_argmax_accuracy_f32");
  return {pred, counts};
}

// ------------------------------------------------------------------ optimizers
namespace {
struct Lists {
  std::vector<float*> p, m, v;
  std::vector<const float*> g;
  std::vector<int64_t> n;
  std::vector<Tensor> keep;
};
Lists lists(const std::vector<Tensor>& p, const std::vector<Tensor>& g) {
  Lists l;
  for (size_t i = 0; i < p.size(); ++i) {
    require(p[i].is_cuda() && p[i].scalar_type() == at::kFloat && p[i].is_contiguous(),
            "fused optimizers need contiguous float32 CUDA parameters");
    require(!g[i].is_sparse() && f32_on(g[i], p[i].device()) && g[i].numel() == p[i].numel(),
            "fused optimizers need dense float32 gradients on the parameter's device");
    require(p[i].device() == p[0].device(), "fused optimizers take the parameters of one device at a time");
    l.keep.push_back(g[i].contiguous());
    l.p.push_back(static_cast<float*>(p[i].data_ptr()));
    l.g.push_back(l.keep.back().const_data_ptr<float>());
    l.n.push_back(p[i].numel());
  }
  return l;
}
}  // namespace

void adam_step(const std::vector<Tensor>& p, const std::vector<Tensor>& g, const std::vector<Tensor>& m,
               const std::vector<Tensor>& v, double lr, double b1, double b2, double eps, double wd,
               const Tensor& state) {
  Lists l = lists(p, g);
  const auto moment = [](const Tensor& t, const Tensor& p) {
    return f32_on(t, p.device()) && t.is_contiguous() && t.numel() == p.numel();
  };
  require(p.empty() || p[0].device() == state.device(), "the optimizer state must be on the parameters' device");
  for (size_t i = 0; i < p.size(); ++i) {
    require(moment(m[i], p[i]) && moment(v[i], p[i]),
            "FusedAdam: exp_avg and exp_avg_sq must be contiguous float32 tensors of the parameter's size on its device");
    l.m.push_back(static_cast<float*>(m[i].data_ptr()));
    l.v.push_back(static_cast<float*>(v[i].data_ptr()));
  }
  const at::Device dev = state.device();
  const c10::cuda::CUDAGuard guard(dev);
  check(abi.gc_adam_step_f32(int(p.size()), l.p.data(), l.g.data(), l.m.data(), l.v.data(), l.n.data(), lr, b1, b2,
                             eps, wd, state.data_ptr(), stream_of(dev)),
        "gc_adam_step_f32");
}

void sgd_step(const std::vector<Tensor>& p, const std::vector<Tensor>& g, double lr, double wd) {
  if (p.empty()) return;
  Lists l = lists(p, g);
  const at::Device dev = p[0].device();
  const c10::cuda::CUDAGuard guard(dev);
  check(abi.gc_sgd_step_f32(int(p.size()), l.p.data(), l.g.data(), l.n.data(), lr, wd, stream_of(dev)),
        "gc_sgd_step_f32");
}

}  // namespace gch
