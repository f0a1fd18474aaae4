// Native host side of the layer path: what sits between torch tensors and the C ABI.
//
// A step of a Cora-sized model is some 15 kernels of a few microseconds each; composing them in Python through ctypes
// cost 15-40 us of interpreter time per call (0.74 ms per eager training step for 0.13 ms of device work).  Allocation,
// shape checks, operand layout, the composition of a layer and its autograd node therefore live here; Python keeps the
// public signatures.  The C ABI library is reached through pointers resolved at import, so the same file serves both.
#pragma once

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/custom_class.h>

#include <atomic>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <stdexcept>
#include <string>

#include "../../../include/graphcuda_b200.h"

namespace gch {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

[[noreturn]] void raise(const std::string& msg);
inline void require(bool cond, const char* msg) {
  if (__builtin_expect(!cond, 0)) raise(msg);
}

// A float32 tensor whose memory a kernel on that device may be given (a host pointer would be a fault on the GPU).
inline bool f32_on(const Tensor& t, const at::Device& dev) {
  return t.device() == dev && t.scalar_type() == at::kFloat;
}

// ------------------------------------------------------------------ C ABI
#define GC_HOST_FUNCTIONS(X)                                                                                        \
  X(gc_last_error) X(gc_status_string) X(gc_spmm_default_panel_cols) X(gc_spmm_segment)                     \
  X(gc_spmm_plan_workspace_bytes) X(gc_spmm_plan_count) X(gc_spmm_plan_bytes) X(gc_spmm_plan_build)                 \
  X(gc_spmm_scratch_bytes) X(gc_spmm_csr_f32) X(gc_spmm_csr_bf16h_f32) X(gc_gemm_workspace_bytes) X(gc_gemm_f32)    \
  X(gc_convert_f32_bf16) X(gc_gemm_bf16_workspace_bytes) X(gc_gemm_bf16_f32) X(gc_relu_backward_f32)                \
  X(gc_mask_mul_f32) X(gc_nll_workspace_bytes) X(gc_logsoftmax_nll_forward_f32) X(gc_logsoftmax_nll_backward_f32)   \
  X(gc_argmax_accuracy_masks_f32) X(gc_logsoftmax_nll_backward_pad_f32) X(gc_adam_step_f32) X(gc_sgd_step_f32) X(gc_csr_is_symmetric) X(gc_pad_rows_f32)                         \
  X(gc_edges_workspace_bytes) X(gc_edges_sort) X(gc_edges_to_csr) X(gc_degree_order_workspace_bytes)                \
  X(gc_degree_order) X(gc_relu_bias_backward_workspace_bytes) X(gc_relu_bias_backward_f32)
struct Abi {
#define X(name) decltype(&::name) name = nullptr;
  GC_HOST_FUNCTIONS(X)
#undef X
};
extern Abi abi;
void load_abi(const std::string& path);
void check(int status, const char* what);

// ------------------------------------------------------------------ scratch
// Grow-only scratch, one buffer per (device, stream, tag).  Kernels of one stream run in order, so a buffer is never
// in use by two launches at once -- provided the launches of one call follow each other on the stream.  Several threads
// may issue on one stream, so a Scratch holds its buffer until it is destroyed: keep it until the call that uses it has
// returned, and take no second one of the same tag meanwhile.  While a stream is being captured the scratch is allocated for that call alone, from
// the graph's own pool: a buffer shared with eager launches could be outgrown and released while the graph still
// replays on it.  Nothing in a buffer outlives its call: what a tensor-core GEMM reports about a wait that ran out is
// read from the device's own word (gc_gemm_error_word).
enum Tag { kGemm = 0, kSpmm = 1, kTags = 2 };
struct Scratch {
  void* ptr = nullptr;
  size_t bytes = 0;
  Tensor keep;  // a per-call buffer, or one that another thread has outgrown by now
  std::unique_lock<std::mutex> turn;
};
Scratch scratch(Tag tag, size_t bytes, const at::Device& dev);
void scratch_clear();

inline void* stream_of(const at::Device& dev) { return at::cuda::getCurrentCUDAStream(dev.index()).stream(); }

// A row-major matrix as the kernels take it, or the transpose of one (trans: rows x cols is a view of a cols x rows
// matrix with leading dimension ld).
struct Mat {
  const float* p;
  int64_t rows, cols, ld;
  int trans;
  Mat t() const { return Mat{p, cols, rows, ld, !trans}; }
};
Mat as_operand(Tensor& t);       // copies (into t) only what has no unit stride
Tensor row_major(const Tensor& t);
inline int64_t ld_of(const Tensor& t) {
  return t.size(0) > 1 ? t.stride(0) : std::max<int64_t>({t.size(1), t.stride(0), 1});
}
Tensor empty_f32(int64_t rows, int64_t cols, const at::Device& dev);

// ------------------------------------------------------------------ products
struct Epi {
  const float* bias = nullptr;
  bool relu = false;
  float* mask = nullptr;
  const float* gate = nullptr;
};
void gemm_into(const Mat& A, const Mat& B, float* C, int64_t ldc, const Epi& ep, bool transposed_out, int prec,
               const at::Device& dev);
Tensor to_bf16(const Tensor& X, bool transpose);
void gemm_bf16_into(const Tensor& A16, const Tensor& Bt16, float* C, int64_t ldc, const Epi& ep,
                    const at::Device& dev);

struct Plan {
  Tensor buf;
  int64_t n_pieces, n_slots, n_cut, panel_cols;
};

// An adjacency: int32 CSR with its plans, or a dense matrix.
struct Adj : torch::CustomClassHolder {
  bool dense = false;
  int64_t M = 0, K = 0, nnz = 0;
  std::atomic<int> symmetric{-1};  // -1: not known yet
  // CSR
  Tensor rowptr, col, val;
  bool use_plan = true;
  int64_t segment = 0;  // longest piece; 0: the library's default
  // dense
  Tensor A, A16;

  at::Device device() const { return dense ? A.device() : val.device(); }
  std::shared_ptr<Plan> plan_for(int64_t F, int64_t panel_cols = 0, int64_t segment_len = 0);
  bool is_symmetric();

 private:
  std::mutex mutex_;           // the plans
  std::mutex symmetry_mutex_;  // held while the verdict is found, so that it is found once
  std::map<std::pair<int64_t, int64_t>, std::shared_ptr<Plan>> plans_;  // by panel width and segment
  std::map<int64_t, std::shared_ptr<Plan>> by_width_;  // by F, default panel width
};
using AdjPtr = c10::intrusive_ptr<Adj>;

// Y = A H (+bias)(ReLU)(mask)(gate); H is float32 (or bfloat16) with unit column stride.
void spmm_into(Adj& a, const Tensor& H, float* Y, int64_t ldy, const Epi& ep, bool accumulate, int64_t panel_cols);
void record_spmm(bool on);
std::vector<std::tuple<double, int64_t, int64_t, int64_t, int64_t>> take_spmm_records();
Tensor adj_matmul(Adj& a, Tensor H, int prec, const Epi& ep);

// ------------------------------------------------------------------ graphs
std::tuple<Tensor, Tensor, Tensor> degree_order(const Tensor& edge_index, int64_t n, bool want_relabel);
std::tuple<Tensor, Tensor, Tensor> edges_to_csr(const Tensor& edge_index, int64_t n, bool self_loops,
                                                const OptTensor& relabel);

// ------------------------------------------------------------------ layer, loss, optimizers (layer.cpp, tail.cpp)
struct Forward {
  Tensor Y, mask, inter;  // inter: A X when the aggregation came first, undefined otherwise
};
Forward layer_forward(const Tensor& X, Adj& a, const Tensor& W, const OptTensor& bias, bool relu, bool want_mask,
                      int prec);
struct Grads {
  Tensor dX, dW, db;
};
Grads layer_backward(Tensor G, const Tensor& X, Adj& a, const Tensor& W, bool relu, const Tensor& Y,
                     const Tensor& inter, bool need_dX, bool need_dW, bool need_db, int prec, bool grad_is_gated,
                     bool gate_dx);
Tensor conv(const Tensor& X, const AdjPtr& a, const Tensor& W, const OptTensor& bias, bool relu, int64_t prec,
            int64_t fuse);
Tensor relu_backward(const Tensor& dY, const Tensor& Y);
Tensor mask_mul(const Tensor& dY, const Tensor& mask);
int64_t padded_width(int64_t n_rows, int64_t in_dim, int64_t out_dim);

// Buffers this library produced with zero-filled pad columns: the loss backward writes the gradient of a padded logits
// matrix straight into one and hands out the unpadded view; the layer below finds the buffer again and uses it instead
// of zero-filling and copying a new one.
void register_zero_padded(const Tensor& buf);
OptTensor zero_padded_base(const Tensor& view, int64_t width);
int64_t zero_padded_count();

// The loss and what its backward pass needs: logits and labels as the kernels take them, and the workspace.
struct NllForward {
  Tensor loss, Z, labels, ws;
  bool masked;
};
NllForward nll_forward(const Tensor& Z, const Tensor& labels, const OptTensor& row_mask, double scale);
Tensor nll_backward(const Tensor& grad, const Tensor& Z, const Tensor& labels, const Tensor& ws, bool masked,
                    double scale);
Tensor nll_loss(const Tensor& Z, const Tensor& labels, const OptTensor& row_mask, double scale);
std::pair<Tensor, Tensor> argmax_accuracy(const Tensor& logits, const OptTensor& labels,
                                          const std::optional<std::vector<Tensor>>& masks, bool want_pred);
void adam_step(const std::vector<Tensor>& p, const std::vector<Tensor>& g, const std::vector<Tensor>& m,
               const std::vector<Tensor>& v, double lr, double b1, double b2, double eps, double wd, const Tensor& state);
void sgd_step(const std::vector<Tensor>& p, const std::vector<Tensor>& g, double lr, double wd);
}  // namespace gch
