// Library binding, scratch buffers and the single products (see host.h).
#include "host.h"

#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <ATen/cuda/CUDAEvent.h>
#include <dlfcn.h>

#include <atomic>

#include <unordered_map>

namespace gch {

void raise(const std::string& msg) { throw std::runtime_error(msg); }

Abi abi;

void load_abi(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) raise(std::string("cannot load ") + path + ": " + dlerror());
#define X(name)                                                                   \
  abi.name = reinterpret_cast<decltype(abi.name)>(dlsym(h, #name));               \
  if (!abi.name) raise(std::string(#name) + " is missing from " + path);
  GC_HOST_FUNCTIONS(X)
#undef X
}

void check(int status, const char* what) {
  if (__builtin_expect(status == 0, 1)) return;
  std::string msg = abi.gc_last_error();
  if (msg.empty()) msg = abi.gc_status_string(status);
  raise(std::string(what) + ": " + msg + " (status " + std::to_string(status) + ")");
}

// ------------------------------------------------------------------ scratch
namespace {
struct Key {
  int device;
  void* stream;
  bool operator==(const Key& o) const { return device == o.device && stream == o.stream; }
};
struct KeyHash {
  size_t operator()(const Key& k) const { return std::hash<void*>()(k.stream) * 31 + size_t(k.device); }
};
struct Buffer {
  std::mutex turn;  // held from the first launch that uses the buffer to the last of the same call
  Tensor mem;
};
struct Buffers {
  Buffer of[kTags];
};
std::mutex scratch_mutex;
// Never destroyed: the tensors must not outlive torch's allocator at process exit.  Entries stay when their memory is
// given back: another thread may be waiting for its turn.
std::unordered_map<Key, Buffers, KeyHash>& buffers() {
  static auto* m = new std::unordered_map<Key, Buffers, KeyHash>();
  return *m;
}
Tensor bytes_on(size_t n, const at::Device& dev) {
  return at::empty({int64_t(n)}, at::TensorOptions().dtype(at::kByte).device(dev));
}
}  // namespace

Scratch scratch(Tag tag, size_t bytes, const at::Device& dev) {
  Scratch s;
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
    s.keep = bytes_on(std::max<size_t>(256, bytes), dev);
  } else {
    Buffer* b;
    {
      std::lock_guard<std::mutex> lock(scratch_mutex);
      b = &buffers()[Key{dev.index(), at::cuda::getCurrentCUDAStream(dev.index()).stream()}].of[tag];
    }
    s.turn = std::unique_lock<std::mutex>(b->turn);
    if (!b->mem.defined() || size_t(b->mem.numel()) < bytes) {
      const size_t size = std::max<size_t>(256, (bytes + bytes / 4 + 255) & ~size_t(255));  // growth is rare
      b->mem = bytes_on(size, dev);
    }
    s.keep = b->mem;
  }
  s.ptr = s.keep.data_ptr();
  s.bytes = size_t(s.keep.numel());
  return s;
}

void scratch_clear() {
  std::lock_guard<std::mutex> lock(scratch_mutex);
  for (auto& entry : buffers())
    for (Buffer& b : entry.second.of) {
      std::lock_guard<std::mutex> turn(b.turn);
      b.mem = Tensor();
    }
}

// ------------------------------------------------------------------ layouts
Tensor empty_f32(int64_t rows, int64_t cols, const at::Device& dev) {
  return at::empty({rows, cols}, at::TensorOptions().dtype(at::kFloat).device(dev));
}

Tensor row_major(const Tensor& t) {
  if (t.stride(1) == 1 && t.stride(0) >= std::max<int64_t>(1, t.size(1))) return t;
  if (t.size(1) == 1 && t.stride(0) >= 1) return t;
  return t.contiguous();
}

Mat as_operand(Tensor& t) {
  if (t.stride(1) == 1 && (t.size(0) <= 1 || t.stride(0) >= t.size(1)))
    return Mat{t.const_data_ptr<float>(), t.size(0), t.size(1), ld_of(t), 0};
  if (t.stride(0) == 1 && (t.size(1) <= 1 || t.stride(1) >= t.size(0))) {
    const int64_t ld = t.size(1) > 1 ? t.stride(1) : std::max<int64_t>({t.size(0), t.stride(1), 1});
    return Mat{t.const_data_ptr<float>(), t.size(0), t.size(1), ld, 1};
  }
  t = t.contiguous();
  return Mat{t.const_data_ptr<float>(), t.size(0), t.size(1), ld_of(t), 0};
}

// ------------------------------------------------------------------ products
void gemm_into(const Mat& A, const Mat& B, float* C, int64_t ldc, const Epi& ep, bool transposed_out, int prec,
               const at::Device& dev) {
  const int64_t M = A.rows, K = A.cols, N = B.cols;
  if (M == 0 || N == 0) return;
  const size_t need = abi.gc_gemm_workspace_bytes(A.trans, B.trans, M, N, K, prec);
  const Scratch ws = scratch(kGemm, need, dev);
  const int epi = (ep.relu ? GC_EPI_RELU : 0) | (transposed_out ? GC_EPI_TRANSPOSED_OUT : 0);
  check(abi.gc_gemm_f32(A.trans, B.trans, M, N, K, A.p, A.ld, B.p, B.ld, C, ldc, ep.bias, epi, ep.mask, ep.gate, prec,
                        ws.ptr, ws.bytes, stream_of(dev)),
        "gc_gemm_f32");
}

Tensor to_bf16(const Tensor& Xin, bool transpose) {
  require(Xin.dim() == 2 && Xin.is_cuda() && Xin.scalar_type() == at::kFloat, "to_bf16: float32 CUDA matrix expected");
  const Tensor X = row_major(Xin);
  const int64_t rows = transpose ? X.size(1) : X.size(0), cols = transpose ? X.size(0) : X.size(1);
  const int64_t ld = (cols + 7) / 8 * 8;
  const c10::cuda::CUDAGuard guard(X.device());
  Tensor out = at::empty({rows, ld}, at::TensorOptions().dtype(at::kBFloat16).device(X.device()));
  check(abi.gc_convert_f32_bf16(X.const_data_ptr<float>(), ld_of(X), rows, cols,
                                static_cast<uint16_t*>(out.data_ptr()), ld, transpose ? 1 : 0, stream_of(X.device())),
        "gc_convert_f32_bf16");
  return ld == cols ? out : out.narrow(1, 0, cols);
}

void gemm_bf16_into(const Tensor& A16, const Tensor& Bt16, float* C, int64_t ldc, const Epi& ep,
                    const at::Device& dev) {
  const int64_t M = A16.size(0), K = A16.size(1), N = Bt16.size(0);
  if (M == 0 || N == 0) return;
  const Scratch ws = scratch(kGemm, abi.gc_gemm_bf16_workspace_bytes(M, N, K), dev);
  const int64_t k8 = (K + 7) / 8 * 8;
  check(abi.gc_gemm_bf16_f32(M, N, K, static_cast<const uint16_t*>(A16.data_ptr()), M > 1 ? A16.stride(0) : k8,
                             static_cast<const uint16_t*>(Bt16.data_ptr()), N > 1 ? Bt16.stride(0) : k8, C, ldc,
                             ep.bias, ep.relu ? GC_EPI_RELU : 0, ep.mask, ep.gate, ws.ptr, ws.bytes, stream_of(dev)),
        "gc_gemm_bf16_f32");
}

// ------------------------------------------------------------------ CSR
std::shared_ptr<Plan> Adj::plan_for(int64_t F, int64_t panel_cols, int64_t segment_len) {
  std::lock_guard<std::mutex> lock(mutex_);
  const bool standard = panel_cols <= 0 && segment_len <= 0;
  if (standard) {
    auto it = by_width_.find(F);
    if (it != by_width_.end()) return it->second;
  }
  if (panel_cols <= 0) panel_cols = abi.gc_spmm_default_panel_cols(K, std::max<int64_t>(F, 1));
  const int64_t seg = segment_len > 0 ? segment_len : segment > 0 ? segment : abi.gc_spmm_segment(nnz, F);
  const auto key = std::make_pair(panel_cols, seg);
  auto hit = plans_.find(key);
  std::shared_ptr<Plan> p = hit != plans_.end() ? hit->second : nullptr;
  if (!p) {
    const at::Device dev = device();
    const c10::cuda::CUDAGuard guard(dev);
    void* st = stream_of(dev);
    const int32_t* rp = rowptr.const_data_ptr<int32_t>();
    const int32_t* cp = col.const_data_ptr<int32_t>();
    Tensor counts = at::empty({3}, at::TensorOptions().dtype(at::kLong).device(dev));
    size_t wsb = abi.gc_spmm_plan_workspace_bytes(M, 0);
    Tensor ws = bytes_on(wsb, dev);
    check(abi.gc_spmm_plan_count(rp, cp, M, K, panel_cols, seg, counts.data_ptr<int64_t>(), ws.data_ptr(), wsb, st),
          "gc_spmm_plan_count");
    const Tensor host = counts.cpu();  // the one host read of plan building
    const int64_t* c = host.const_data_ptr<int64_t>();
    p = std::make_shared<Plan>();
    p->n_pieces = c[0];
    p->n_slots = c[1];
    p->n_cut = c[2];
    p->panel_cols = panel_cols;
    const size_t pb = abi.gc_spmm_plan_bytes(p->n_pieces, p->n_cut);
    p->buf = bytes_on(pb, dev);
    wsb = abi.gc_spmm_plan_workspace_bytes(M, p->n_pieces);
    ws = bytes_on(wsb, dev);
    check(abi.gc_spmm_plan_build(rp, cp, M, K, panel_cols, seg, p->n_pieces, p->n_slots, p->n_cut, p->buf.data_ptr(),
                                 pb, ws.data_ptr(), wsb, st),
          "gc_spmm_plan_build");
    // other streams may use the plan next
    C10_CUDA_CHECK(cudaStreamSynchronize(static_cast<cudaStream_t>(st)));
    plans_[key] = p;
  }
  if (standard) by_width_[F] = p;
  return p;
}

bool Adj::is_symmetric() {
  if (symmetric < 0) {
    std::lock_guard<std::mutex> lock(symmetry_mutex_);
    if (symmetric >= 0) return symmetric != 0;
    if (M != K) {
      symmetric = 0;
    } else if (dense) {
      symmetric = A.equal(A.t()) ? 1 : 0;
    } else {
      const c10::cuda::CUDAGuard guard(device());
      Tensor out = at::empty({1}, at::TensorOptions().dtype(at::kInt).device(device()));
      check(abi.gc_csr_is_symmetric(rowptr.const_data_ptr<int32_t>(), col.const_data_ptr<int32_t>(),
                                    val.const_data_ptr<float>(), M, out.data_ptr<int32_t>(), stream_of(device())),
            "gc_csr_is_symmetric");
      symmetric = out.item<int32_t>() ? 1 : 0;
    }
  }
  return symmetric != 0;
}

// Device times of the aggregations issued while recording is on: the layers call them without passing through Python,
// where a benchmark would otherwise put its events.
namespace {
struct SpmmRecord {
  at::cuda::CUDAEvent begin{cudaEventDefault}, end{cudaEventDefault};
  int64_t M, K, F, nnz;
};
std::atomic<bool> spmm_recording{false};
std::mutex spmm_records_mutex;
std::vector<SpmmRecord>& spmm_record_list() {
  static auto* v = new std::vector<SpmmRecord>();
  return *v;
}
}  // namespace

void record_spmm(bool on) { spmm_recording = on; }

// (ms, M, K, F, nnz) of every recorded aggregation, waiting for the last; clears the list.
std::vector<std::tuple<double, int64_t, int64_t, int64_t, int64_t>> take_spmm_records() {
  const std::lock_guard<std::mutex> lock(spmm_records_mutex);
  std::vector<std::tuple<double, int64_t, int64_t, int64_t, int64_t>> out;
  for (auto& r : spmm_record_list()) {
    r.end.synchronize();
    out.emplace_back(r.begin.elapsed_time(r.end), r.M, r.K, r.F, r.nnz);
  }
  spmm_record_list().clear();
  return out;
}

static void spmm_launch(Adj& a, const Tensor& Hin, float* Y, int64_t ldy, const Epi& ep, bool accumulate,
                        int64_t panel_cols);

void spmm_into(Adj& a, const Tensor& Hin, float* Y, int64_t ldy, const Epi& ep, bool accumulate, int64_t panel_cols) {
  if (!spmm_recording.load(std::memory_order_relaxed)) return spmm_launch(a, Hin, Y, ldy, ep, accumulate, panel_cols);
  const auto st = at::cuda::getCurrentCUDAStream(a.device().index());
  SpmmRecord r;
  r.M = a.M; r.K = a.K; r.F = Hin.size(1); r.nnz = a.nnz;
  r.begin.record(st);
  spmm_launch(a, Hin, Y, ldy, ep, accumulate, panel_cols);
  r.end.record(st);
  const std::lock_guard<std::mutex> lock(spmm_records_mutex);
  spmm_record_list().push_back(std::move(r));
}

// Whether gathering from a copy of H on an aligned pitch beats gathering H as it lies (rows that are not 16-byte aligned:
// one float per lane).  The copy costs 8 bytes per element, streamed, and scalar stores of Y stay; it pays where every row
// is gathered often enough, later for wider rows (a scalar gather of a wide row is whole lines too) and, on few rows,
// hardly where warps per piece serve scalar gathers as well.  Measured, time with the copy over time without, at rows /
// non-zeros per row: up to 16 columns 0.75 at 3 K..10 K rows, 1.4 / 1.3 / 0.9 at 40 K / 6, 10, 40, 1.2 / 0.9 at 80 K / 4.5,
// 10, 0.7 at 169 K; 17 to 32 0.4..0.9 throughout; 33 to 64 1.2 below 260 K non-zeros, 0.5..1.0 above; 65 to 208 1.2..1.5 on
// 20 K rows, 0.8..0.95 on 40 K and more from 650 K non-zeros; 255 to 256 1.2 / 1.0 / 0.95 at 169 K / 4.5, 13, 20; wider
// 0.7..1.0 on 6 K..20 K rows, and above at 6 / 10 / 13 / 20 per row 1.18 / 1.08 / 1.01 / 0.92 (F = 511, 169 K rows).
static bool copy_pays(int64_t F, int64_t K, int64_t nnz) {
  if (F <= 8 || nnz < 4 * K) return false;
  const int64_t some = 1 << 16, many = 5 << 17;
  if (F <= 16) return nnz >= some && (K <= 15000 || nnz >= 32 * K || (K > 75000 && nnz >= many));
  if (F <= 32) return nnz >= some;
  if (F <= 64) return nnz >= 4 * some;
  const bool large = K > 30000;
  if (F <= 256) return large && nnz >= many && (F <= 208 || nnz >= 12 * K);
  return nnz >= 2 * some && (!large || nnz >= 12 * K);
}

// Largest such copy at a time; wider matrices take it in slabs of columns.
constexpr int64_t kCopyBytes = int64_t(1) << 30;

static void spmm_launch(Adj& a, const Tensor& Hin, float* Y, int64_t ldy, const Epi& ep, bool accumulate, int64_t panel_cols) {
  const at::Device dev = a.device();
  const int64_t F = Hin.size(1);
  const bool h16 = Hin.scalar_type() == at::kBFloat16;
  std::shared_ptr<Plan> plan = a.use_plan ? a.plan_for(F, panel_cols) : nullptr;
  Scratch s;
  if (plan && plan->n_cut > 0) s = scratch(kSpmm, abi.gc_spmm_scratch_bytes(plan->n_slots, F), dev);
  const int epi = (ep.relu ? GC_EPI_RELU : 0) | (accumulate ? GC_EPI_ACCUMULATE : 0);
  const int32_t* rp = a.rowptr.const_data_ptr<int32_t>();
  const int32_t* cp = a.col.const_data_ptr<int32_t>();
  const float* vp = a.val.const_data_ptr<float>();
  const void* pb = plan ? plan->buf.data_ptr() : nullptr;
  const int64_t np = plan ? plan->n_pieces : 0, ns = plan ? plan->n_slots : 0, nc = plan ? plan->n_cut : 0;
  void* st = stream_of(dev);
  const int64_t ldh = Hin.size(0) > 1 ? Hin.stride(0) : std::max<int64_t>(F, 1);
  if (h16) {
    check(abi.gc_spmm_csr_bf16h_f32(rp, cp, vp, a.M, a.K, F, static_cast<const uint16_t*>(Hin.data_ptr()), ldh, ep.bias,
                                    epi, Y, ldy, ep.mask, ep.gate, pb, np, ns, nc, s.ptr, s.bytes, st),
          "gc_spmm_csr_f32");
    return;
  }
  // columns f0 .. f0 + n of Y from n columns at H
  const auto columns = [&](const float* H, int64_t ld, int64_t f0, int64_t n, int flags) {
    const auto at_f0 = [&](auto* p) { return p ? p + f0 : nullptr; };
    check(abi.gc_spmm_csr_f32(rp, cp, vp, a.M, a.K, n, H, ld, at_f0(ep.bias), epi | flags, Y + f0, ldy, at_f0(ep.mask),
                              at_f0(ep.gate), pb, np, ns, nc, s.ptr, s.bytes, st),
          "gc_spmm_csr_f32");
  };
  const float* H = Hin.const_data_ptr<float>();
  const bool aligned = ldh % 4 == 0 && reinterpret_cast<uintptr_t>(H) % 16 == 0;
  if (aligned && F % 4 == 0) return columns(H, ldh, 0, F, 0);
  const int64_t f4 = (F + 3) / 4 * 4;
  const int64_t last = (Hin.storage_offset() + (a.K - 1) * ldh + f4) * int64_t(sizeof(float));
  if (aligned && a.K > 0 && ldh >= f4 && last <= int64_t(Hin.storage().nbytes()))
    return columns(H, ldh, 0, F, GC_EPI_H_PADDED);  // a view of wider rows: what lies beyond the width may be read, and is not used
  if (!copy_pays(F, a.K, a.nnz)) return columns(H, ldh, 0, F, 0);
  const int64_t slabs = (a.K * f4 * int64_t(sizeof(float)) + kCopyBytes - 1) / kCopyBytes;
  const int64_t width = ((f4 / 4 + slabs - 1) / slabs) * 4;
  Tensor copy;
  try {
    copy = empty_f32(a.K, width, dev);
  } catch (const c10::OutOfMemoryError&) {
    return columns(H, ldh, 0, F, 0);
  }
  float* to = copy.data_ptr<float>();
  for (int64_t f0 = 0; f0 < F; f0 += width) {
    const int64_t n = std::min(width, F - f0);
    check(abi.gc_pad_rows_f32(H + f0, ldh, to, width, a.K, n, st), "gc_pad_rows_f32");
    columns(to, width, f0, n, GC_EPI_H_PADDED);
  }
}

// ------------------------------------------------------------------ graphs
// (perm, inv, int32 inv) of the order by decreasing number of incoming edges.
std::tuple<Tensor, Tensor, Tensor> degree_order(const Tensor& edge_index, int64_t n, bool want_relabel) {
  const at::Device dev = edge_index.device();
  const c10::cuda::CUDAGuard guard(dev);
  const Tensor target = edge_index.select(0, 1).contiguous();
  const auto i64 = at::TensorOptions().dtype(at::kLong).device(dev);
  Tensor perm = at::empty({n}, i64), inv = at::empty({n}, i64), relabel;
  if (want_relabel) relabel = at::empty({n}, i64.dtype(at::kInt));
  const size_t wsb = abi.gc_degree_order_workspace_bytes(n);
  Tensor ws = bytes_on(wsb, dev);
  check(abi.gc_degree_order(target.const_data_ptr<int64_t>(), target.numel(), n, perm.data_ptr<int64_t>(),
                            inv.data_ptr<int64_t>(), want_relabel ? relabel.data_ptr<int32_t>() : nullptr,
                            ws.data_ptr(), wsb, stream_of(dev)),
        "gc_degree_order");
  return {perm, inv, relabel};
}

// (rowptr, col, val) of the normalised adjacency of an int64 [2, E] edge list.
std::tuple<Tensor, Tensor, Tensor> edges_to_csr(const Tensor& edge_index, int64_t n, bool self_loops,
                                                const OptTensor& relabel) {
  const at::Device dev = edge_index.device();
  const c10::cuda::CUDAGuard guard(dev);
  const auto i32 = at::TensorOptions().dtype(at::kInt).device(dev);
  const int64_t E = edge_index.size(1);
  if (E + (self_loops ? n : 0) == 0)
    return {at::zeros({n + 1}, i32), at::empty({0}, i32), at::empty({0}, i32.dtype(at::kFloat))};
  const Tensor row = edge_index.select(0, 0).contiguous(), col = edge_index.select(0, 1).contiguous();
  const size_t wsb = abi.gc_edges_workspace_bytes(E, n, self_loops);
  Tensor ws = bytes_on(wsb, dev);
  void* st = stream_of(dev);
  int selector = 0;
  const int32_t* nnz_at = nullptr;
  check(abi.gc_edges_sort(row.const_data_ptr<int64_t>(), col.const_data_ptr<int64_t>(), E, n, self_loops,
                          relabel ? relabel->const_data_ptr<int32_t>() : nullptr, ws.data_ptr(), wsb, &selector,
                          &nnz_at, st),
        "gc_edges_sort");
  Tensor rowptr = at::empty({n + 1}, i32);
  const int64_t at = reinterpret_cast<const char*>(nnz_at) - static_cast<const char*>(ws.data_ptr());
  const Tensor sizes = ws.narrow(0, at, 8).cpu();  // the one host read
  const int64_t nnz = static_cast<const int32_t*>(sizes.data_ptr())[0];
  require(static_cast<const int32_t*>(sizes.data_ptr())[1] == 0,
          "edge_index names a vertex outside the graph (negative, or num_nodes and above)");
  Tensor c = at::empty({nnz}, i32), v = at::empty({nnz}, i32.dtype(at::kFloat));
  check(abi.gc_edges_to_csr(E, n, self_loops, selector, ws.data_ptr(), wsb, rowptr.data_ptr<int32_t>(),
                            c.data_ptr<int32_t>(), v.data_ptr<float>(), st),
        "gc_edges_to_csr");
  return {rowptr, c, v};
}

}  // namespace gch
