// Python module of the native host side.
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include "host.h"

namespace py = pybind11;
using namespace gch;

namespace {
using NoGil = py::call_guard<py::gil_scoped_release>;

// C = A B (+bias)(ReLU)(gate): checks, layouts, output allocation.
py::object gemm(const Tensor& Ain, const Tensor& Bin, const OptTensor& bias_in, bool relu, bool want_mask, int64_t prec,
                bool transposed_out, const OptTensor& out_in, const OptTensor& gate) {
  require(Ain.dim() == 2 && Bin.dim() == 2, "Inputs must be 2D");
  require(Ain.size(1) == Bin.size(0), "A.cols must match B.rows");
  require(Ain.is_cuda() && Bin.is_cuda(), "Inputs must be CUDA tensors");
  require(Ain.scalar_type() == at::kFloat && Bin.scalar_type() == at::kFloat, "Only float32 is supported here");
  require(Ain.device() == Bin.device(), "Inputs must be on the same device");
  Tensor out, mask;
  {
    const py::gil_scoped_release release;
    const at::Device dev = Ain.device();
    const c10::cuda::CUDAGuard guard(dev);
    Tensor A = Ain, B = Bin;
    const Mat a = as_operand(A), b = as_operand(B);
    const int64_t M = a.rows, N = b.cols, R = transposed_out ? N : M, Q = transposed_out ? M : N;
    if (out_in) {
      out = *out_in;
      require(f32_on(out, dev) && out.dim() == 2 && out.size(0) == R && out.size(1) == Q && out.is_contiguous(),
              "out has the wrong shape, dtype, layout or device");
    } else {
      out = empty_f32(R, Q, dev);
    }
    Epi ep;
    ep.relu = relu;
    Tensor bias;
    if (bias_in) {
      require(f32_on(*bias_in, dev) && bias_in->numel() == N, "bias must be float32 [N] on the operands' device");
      bias = bias_in->contiguous();
      ep.bias = bias.const_data_ptr<float>();
    }
    if (gate) {
      require(f32_on(*gate, dev) && gate->sizes() == out.sizes() && gate->is_contiguous(),
              "gate must be a contiguous float32 tensor of the result's shape, on its device");
      ep.gate = gate->const_data_ptr<float>();
    }
    if (want_mask) {
      mask = empty_f32(R, Q, dev);
      ep.mask = mask.data_ptr<float>();
    }
    gemm_into(a, b, static_cast<float*>(out.data_ptr()), std::max<int64_t>(Q, 1), ep, transposed_out, int(prec), dev);
  }
  return want_mask ? py::object(py::make_tuple(out, mask)) : py::cast(out);
}

Tensor gemm_bf16(const Tensor& A16, const Tensor& Bt16, const OptTensor& bias_in, bool relu, const OptTensor& out_in,
                 const OptTensor& gate) {
  require(A16.scalar_type() == at::kBFloat16 && Bt16.scalar_type() == at::kBFloat16 && A16.is_cuda() && Bt16.is_cuda(),
          "bf16 CUDA operands expected");
  require(A16.dim() == 2 && Bt16.dim() == 2 && A16.size(1) == Bt16.size(1), "A16 and Bt16 must share K");
  require(A16.device() == Bt16.device(), "Inputs must be on the same device");
  require(A16.stride(1) == 1 && Bt16.stride(1) == 1, "operands must have unit stride along K");
  const int64_t M = A16.size(0), N = Bt16.size(0);
  const at::Device dev = A16.device();
  const c10::cuda::CUDAGuard guard(dev);
  Tensor out;
  if (out_in) {
    out = *out_in;
    require(f32_on(out, dev) && out.dim() == 2 && out.size(0) == M && out.size(1) == N && out.is_contiguous(),
            "out has the wrong shape, dtype, layout or device");
  } else {
    out = empty_f32(M, N, dev);
  }
  Epi ep;
  ep.relu = relu;
  Tensor bias;
  if (bias_in) {
    require(f32_on(*bias_in, dev) && bias_in->numel() == N, "bias must be float32 [N] on the operands' device");
    bias = bias_in->contiguous();
    ep.bias = bias.const_data_ptr<float>();
  }
  if (gate) {
    require(f32_on(*gate, dev) && gate->sizes() == out.sizes() && gate->is_contiguous(),
            "gate must be a contiguous float32 tensor of the result's shape, on its device");
    ep.gate = gate->const_data_ptr<float>();
  }
  gemm_bf16_into(A16, Bt16, static_cast<float*>(out.data_ptr()), N, ep, dev);
  return out;
}

// Y = A H (+bias)(ReLU)(gate) on a CSR adjacency.
py::object spmm(const AdjPtr& adj, const Tensor& Hin, const OptTensor& bias_in, bool relu, bool want_mask,
                const OptTensor& accumulate_into, const OptTensor& out_in, int64_t panel_cols, const OptTensor& gate) {
  Adj& a = *adj;
  require(Hin.dim() == 2, "B must be 2D");
  require(Hin.size(0) == a.K, "A.cols must match B.rows");
  require(Hin.is_cuda() && Hin.device() == a.device(), "A and B must be CUDA tensors on the same device");
  const bool h16 = Hin.scalar_type() == at::kBFloat16;
  require(Hin.scalar_type() == at::kFloat || h16,
          "B must be float32 (or bfloat16 for the reduced-precision tier)");
  Tensor out, mask;
  {
    const py::gil_scoped_release release;
    Tensor H = Hin;
    const int64_t M = a.M, F = H.size(1);
    if (h16)
      require(H.stride(1) == 1 && F % 8 == 0 && (H.size(0) <= 1 || H.stride(0) % 8 == 0) &&
                  reinterpret_cast<uintptr_t>(H.data_ptr()) % 16 == 0,
              "a bfloat16 B needs a width and row pitch that are multiples of 8");
    else if (H.stride(1) != 1 || (H.size(0) > 1 && H.stride(0) < F))
      H = H.contiguous();
    const at::Device dev = a.device();
    const c10::cuda::CUDAGuard guard(dev);
    const bool accumulate = accumulate_into.has_value();
    if (accumulate) out = *accumulate_into;
    else if (out_in) out = *out_in;
    else out = empty_f32(M, F, dev);
    // `out` may be a column slice of a wider row-major matrix (unit column stride)
    require(f32_on(out, dev) && out.dim() == 2 && out.size(0) == M && out.size(1) == F && out.stride(1) == 1 &&
                (M <= 1 || out.stride(0) >= F),
            "out has the wrong shape, dtype, layout or device");
    const int64_t ldy = M > 1 ? out.stride(0) : std::max<int64_t>(F, 1);
    require(!want_mask || ldy == F, "a mask needs a contiguous output");
    Epi ep;
    ep.relu = relu;
    if (want_mask) {
      mask = empty_f32(M, F, dev);
      ep.mask = mask.data_ptr<float>();
    }
    Tensor bias;
    if (bias_in) {
      require(f32_on(*bias_in, dev) && bias_in->numel() == F, "bias must be float32 [F] on A's device");
      bias = bias_in->contiguous();
      ep.bias = bias.const_data_ptr<float>();
    }
    if (gate) {
      require(f32_on(*gate, dev) && gate->sizes() == out.sizes() && gate->is_contiguous() && ldy == F,
              "gate must be a contiguous float32 tensor of Y's shape, on its device");
      ep.gate = gate->const_data_ptr<float>();
    }
    if (M != 0 && F != 0)
      spmm_into(a, H, static_cast<float*>(out.data_ptr()), ldy, ep, accumulate, panel_cols);
  }
  return want_mask ? py::object(py::make_tuple(out, mask)) : py::cast(out);
}

AdjPtr make_csr(const Tensor& rowptr, const Tensor& col, const Tensor& val, int64_t M, int64_t K, int symmetric,
                bool use_plan) {
  require(rowptr.is_cuda() && col.is_cuda() && val.is_cuda(), "CSR arrays must be CUDA tensors");
  require(col.device() == rowptr.device() && val.device() == rowptr.device(), "CSR arrays must be on one device");
  require(rowptr.scalar_type() == at::kInt && col.scalar_type() == at::kInt, "rowptr/col must be int32");
  require(val.scalar_type() == at::kFloat, "CSR values must be float32");
  require(rowptr.numel() == M + 1, "rowptr must have M+1 entries");
  require(col.numel() == val.numel(), "col and val must have the same length");
  auto a = c10::make_intrusive<Adj>();
  a->rowptr = rowptr.contiguous();
  a->col = col.contiguous();
  a->val = val.contiguous();
  a->M = M;
  a->K = K;
  a->nnz = col.numel();
  a->symmetric = symmetric;
  a->use_plan = use_plan;
  return a;
}

// Other values on the same structure: the plans stay, the symmetry verdict does not.
void set_val(Adj& a, const Tensor& val) {
  require(!a.dense && val.is_cuda() && val.device() == a.device() && val.scalar_type() == at::kFloat &&
              val.numel() == a.nnz,
          "CSR values must be a float32 CUDA tensor with one entry per non-zero");
  a.val = val.contiguous();
  a.symmetric = -1;
}

AdjPtr make_dense(const Tensor& A, int symmetric) {
  require(A.dim() == 2 && A.is_cuda() && A.scalar_type() == at::kFloat,
          "dense adjacency must be a float32 CUDA matrix");
  auto a = c10::make_intrusive<Adj>();
  a->dense = true;
  a->A = A;
  a->M = A.size(0);
  a->K = A.size(1);
  a->symmetric = symmetric;
  return a;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("load_abi", &load_abi);
  m.def("gemm", &gemm);
  m.def("gemm_bf16", &gemm_bf16, NoGil());
  m.def("to_bf16", &to_bf16, NoGil());
  m.def("spmm", &spmm);
  m.def("relu_backward", &relu_backward, NoGil());
  m.def("mask_mul", &mask_mul, NoGil());
  m.def("scratch_clear", &scratch_clear, NoGil());

  py::class_<Plan, std::shared_ptr<Plan>>(m, "SpmmPlan")
      .def_readonly("buf", &Plan::buf)
      .def_readonly("n_pieces", &Plan::n_pieces)
      .def_readonly("n_slots", &Plan::n_slots)
      .def_readonly("n_cut", &Plan::n_cut)
      .def_readonly("panel_cols", &Plan::panel_cols);
  py::class_<Adj, AdjPtr>(m, "Adj")
      .def_readonly("rowptr", &Adj::rowptr)
      .def_readonly("col", &Adj::col)
      .def_readonly("val", &Adj::val)
      .def_readonly("A", &Adj::A)
      .def("set_val", &set_val)
      .def_readonly("M", &Adj::M)
      .def_readonly("K", &Adj::K)
      .def_readonly("nnz", &Adj::nnz)
      .def_readwrite("use_plan", &Adj::use_plan)
      .def_readwrite("segment", &Adj::segment)
      .def_readwrite("A16", &Adj::A16)
      .def_property("symmetric", [](const Adj& a) { return a.symmetric.load(); }, [](Adj& a, int v) { a.symmetric = v; })
      .def("is_symmetric", &Adj::is_symmetric, NoGil())
      .def("plan_for", &Adj::plan_for, py::arg("F"), py::arg("panel_cols") = 0, py::arg("segment") = 0, NoGil());
  m.def("csr", &make_csr);
  m.def("dense", &make_dense);

  m.def("degree_order", &degree_order, NoGil());
  m.def("edges_to_csr", &edges_to_csr, NoGil());

  m.def("padded_width", &padded_width);
  m.def("record_spmm", &record_spmm);
  m.def("take_spmm_records", &take_spmm_records, NoGil());
  m.def("zero_padded_base", &zero_padded_base);
  m.def("register_zero_padded", &register_zero_padded);
  m.def("zero_padded_count", &zero_padded_count);

  // None while a trace is being taken: the caller then goes through an autograd function in Python, which it records.
  m.def("conv", [](const Tensor& X, const AdjPtr& a, const Tensor& W, const OptTensor& bias, bool relu, int64_t prec,
                   int64_t fuse) -> OptTensor {
    if (torch::jit::tracer::isTracing()) return std::nullopt;
    return conv(X, a, W, bias, relu, prec, fuse);
  }, NoGil());
  m.def("layer_forward", [](const Tensor& X, const AdjPtr& a, const Tensor& W, const OptTensor& bias, bool relu,
                            bool want_mask, int64_t prec) {
    Forward f = layer_forward(X, *a, W, bias, relu, want_mask, int(prec));
    return std::make_tuple(f.Y, f.mask, f.inter);
  }, NoGil());
  m.def("layer_backward", [](const Tensor& G, const Tensor& X, const AdjPtr& a, const Tensor& W, bool relu, const Tensor& Y,
                             const OptTensor& inter, bool need_dX, bool need_dW, bool need_db, int64_t prec, int64_t fuse) {
    const Grads g = layer_backward(G, X, *a, W, relu, Y, inter ? *inter : Tensor(), need_dX, need_dW, need_db, int(prec),
                                   fuse & 1, fuse & 2);
    return std::make_tuple(g.dX, g.dW, g.db);
  }, NoGil());
  m.def("adj_matmul", [](const AdjPtr& a, const Tensor& H, int64_t prec) {
    require(H.dim() == 2 && H.size(0) == a->K, "A.cols must match B.rows");
    require(f32_on(H, a->device()), "B must be a float32 CUDA matrix on A's device");
    const c10::cuda::CUDAGuard guard(H.device());
    return adj_matmul(*a, H, int(prec), Epi{});
  }, NoGil());
  m.def("nll_loss", [](const Tensor& Z, const Tensor& labels, const OptTensor& row_mask, double scale) -> OptTensor {
    if (torch::jit::tracer::isTracing()) return std::nullopt;
    return nll_loss(Z, labels, row_mask, scale);
  }, NoGil());
  m.def("nll_forward", [](const Tensor& Z, const Tensor& labels, const OptTensor& row_mask, double scale) {
    const NllForward f = nll_forward(Z, labels, row_mask, scale);
    return std::make_tuple(f.loss, f.Z, f.labels, f.ws, f.masked);
  }, NoGil());
  m.def("nll_backward", &nll_backward, NoGil());
  m.def("argmax_accuracy", &argmax_accuracy, NoGil());
  m.def("adam_step", &adam_step, NoGil());
  m.def("sgd_step", &sgd_step, NoGil());
}
