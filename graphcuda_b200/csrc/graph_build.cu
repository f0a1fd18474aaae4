// Adjacency construction on the GPU: GCN normalisation, COO -> CSR, symmetry
// test.  Takes over what the reference's scripts do with torch_geometric and
// torch sparse tensors before the layer is called
// (tests/gcn/graphcuda_impl.py:27-38: add_self_loops -> gcn_norm ->
// sparse_coo_tensor(...).coalesce()).
//
// Built WITHOUT fast-math: the normalisation must round exactly like torch's
// CPU kernels (1.0f / sqrtf(d), then two IEEE multiplications).
#include "common.cuh"

#include <algorithm>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

namespace {

__global__ void __launch_bounds__(256)
rows_to_rowptr_kernel(const int64_t* __restrict__ rows, int64_t nnz, int64_t M, int32_t* __restrict__ rowptr) {
  const int64_t stride = int64_t(gridDim.x) * 256;
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e <= nnz; e += stride) {
    // entry e opens every row in (rows[e-1], rows[e]]; e == nnz closes the tail
    const int64_t prev = e > 0 ? rows[e - 1] : -1;
    const int64_t cur = e < nnz ? rows[e] : M;
    for (int64_t r = prev + 1; r <= cur && r <= M; ++r) rowptr[r] = int32_t(e);
  }
}

__global__ void __launch_bounds__(256)
narrow_kernel(const int64_t* __restrict__ src, int32_t* __restrict__ dst, int64_t n) {
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < n; i += int64_t(gridDim.x) * 256)
    dst[i] = int32_t(src[i]);
}

// A vertex number of an edge list; the lists come from the caller, and one that names a vertex outside the graph must not
// be an access outside its arrays.
__device__ __forceinline__ bool is_vertex(int64_t v, int64_t N) { return v >= 0 && v < N; }

__global__ void __launch_bounds__(256)
degree_kernel(const int64_t* __restrict__ col, int64_t E, int64_t N, int32_t* __restrict__ deg) {
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e < E; e += int64_t(gridDim.x) * 256) {
    const int64_t c = col[e];
    if (is_vertex(c, N)) atomicAdd(deg + c, 1);  // integer counts: exact and order-independent
  }
}

__global__ void __launch_bounds__(256)
dinv_kernel(int32_t* __restrict__ deg_then_dinv, int64_t N) {
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < N; i += int64_t(gridDim.x) * 256) {
    const float d = float(deg_then_dinv[i]);
    // pow(d, -0.5) on torch CPU == 1.0f / sqrtf(d); isolated nodes: inf -> 0
    const float r = d > 0.f ? __fdiv_rn(1.0f, __fsqrt_rn(d)) : 0.f;
    reinterpret_cast<float*>(deg_then_dinv)[i] = r;
  }
}

__global__ void __launch_bounds__(256)
norm_weight_kernel(const int64_t* __restrict__ row, const int64_t* __restrict__ col, int64_t E, int64_t N,
                   const float* __restrict__ dinv, float* __restrict__ w) {
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e < E; e += int64_t(gridDim.x) * 256) {
    const int64_t r = row[e], c = col[e];
    if (!is_vertex(r, N) || !is_vertex(c, N)) {
      w[e] = __int_as_float(0x7fffffff);
      continue;
    }
    // dinv[row] * 1.0f * dinv[col], left to right
    const float a = __fmul_rn(dinv[r], 1.0f);
    w[e] = __fmul_rn(a, dinv[c]);
  }
}

__global__ void __launch_bounds__(256)
head_flag_kernel(const int64_t* __restrict__ row, const int64_t* __restrict__ col, int64_t E,
                 int32_t* __restrict__ head) {
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e < E; e += int64_t(gridDim.x) * 256)
    head[e] = (e == 0 || row[e] != row[e - 1] || col[e] != col[e - 1]) ? 1 : 0;
}

__global__ void total_kernel(const int64_t* __restrict__ row, const int64_t* __restrict__ col, int64_t E,
                             const int32_t* __restrict__ head_excl, int64_t* __restrict__ nnz_out) {
  if (E == 0) { *nnz_out = 0; return; }
  const int64_t e = E - 1;
  const int last = (e == 0 || row[e] != row[e - 1] || col[e] != col[e - 1]) ? 1 : 0;
  *nnz_out = int64_t(head_excl[e]) + last;
}

__global__ void __launch_bounds__(256)
csr_fill_kernel(const int64_t* __restrict__ row, const int64_t* __restrict__ col, const float* __restrict__ w,
                int64_t E, int64_t M, const int32_t* __restrict__ head_excl, int32_t* __restrict__ rowptr,
                int32_t* __restrict__ csr_col, float* __restrict__ csr_val) {
  const int64_t stride = int64_t(gridDim.x) * 256;
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e <= E; e += stride) {
    if (e == E) {
      // close the tail rows
      const int64_t prev = E > 0 ? row[E - 1] : -1;
      int32_t nnz = 0;
      if (E > 0) {
        const int64_t l = E - 1;
        nnz = head_excl[l] + ((l == 0 || row[l] != row[l - 1] || col[l] != col[l - 1]) ? 1 : 0);
      }
      for (int64_t r = prev + 1; r <= M; ++r) rowptr[r] = nnz;
      continue;
    }
    const bool new_row = (e == 0) || row[e] != row[e - 1];
    const bool is_head = new_row || col[e] != col[e - 1];
    if (!is_head) continue;
    const int32_t j = head_excl[e];
    if (new_row) {
      const int64_t prev = e > 0 ? row[e - 1] : -1;
      for (int64_t r = prev + 1; r <= row[e]; ++r) rowptr[r] = j;
    }
    // duplicates are added in input order
    float s = w[e];
    for (int64_t d = e + 1; d < E && row[d] == row[e] && col[d] == col[e]; ++d) s += w[d];
    csr_col[j] = int32_t(col[e]);
    csr_val[j] = s;
  }
}

// ---------------------------------------------------------------- edge list -> sorted keys
// The whole construction works on one integer per edge, row << bits | col with bits = ceil(log2 N): 32-bit keys up to
// 65536 vertices, 64-bit above.  The radix sort runs over the 2 * bits that are used (36 for 169 K vertices: 5 passes
// of 8 bytes instead of 8 of 16 for 64-bit keys with 64-bit permutations), the weights are computed from the degrees
// when the CSR is written instead of being carried along.
template <typename KEY>
__global__ void __launch_bounds__(256)
edge_key_kernel(const int64_t* __restrict__ row, const int64_t* __restrict__ col, int64_t E, int64_t N, int bits,
                const int32_t* __restrict__ relabel, KEY* __restrict__ keys, int32_t* __restrict__ deg,
                int32_t* __restrict__ outside, int64_t total) {
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e < total; e += int64_t(gridDim.x) * 256) {
    int64_t r = e - E, c = r;  // beyond the edges: the self-loops
    if (e < E) {
      r = row[e];
      c = col[e];
      if (!is_vertex(r, N) || !is_vertex(c, N)) {
        *outside = 1;  // the caller discards the result
        keys[e] = 0;
        continue;
      }
      if (relabel) {
        r = relabel[r];
        c = relabel[c];
      }
    }
    keys[e] = (KEY(r) << bits) | KEY(c);
    atomicAdd(deg + c, 1);  // integer counts: exact and order-independent
  }
}

template <typename KEY>
struct IsHead {  // entry e opens a new (row, col)
  const KEY* keys;
  __host__ __device__ int32_t operator()(int64_t e) const { return e == 0 || keys[e] != keys[e - 1] ? 1 : 0; }
};

// incl[e] = number of distinct (row, col) up to e, so the head of an entry writes element incl[e] - 1 of the CSR.
template <typename KEY>
__global__ void __launch_bounds__(256)
csr_from_keys_kernel(const KEY* __restrict__ keys, const int32_t* __restrict__ incl, int64_t E, int64_t N, int bits,
                     const float* __restrict__ dinv, int32_t* __restrict__ rowptr, int32_t* __restrict__ csr_col,
                     float* __restrict__ csr_val) {
  const KEY low = (KEY(1) << bits) - 1;
  for (int64_t e = int64_t(blockIdx.x) * 256 + threadIdx.x; e < E; e += int64_t(gridDim.x) * 256) {
    const KEY k = keys[e];
    const int64_t r = int64_t(k >> bits), c = int64_t(k & low);
    const bool first = e == 0;
    const KEY kp = first ? KEY(0) : keys[e - 1];
    if (first || kp != k) {
      const int32_t j = incl[e] - 1;
      for (int64_t q = first ? 0 : int64_t(kp >> bits) + 1; q <= r; ++q) rowptr[q] = j;
      // dinv[row] * 1.0f * dinv[col], left to right; duplicates are added in input order (they are equal)
      const float w = __fmul_rn(__fmul_rn(__ldg(dinv + r), 1.0f), __ldg(dinv + c));
      float s = w;
      for (int64_t d = e + 1; d < E && keys[d] == k; ++d) s = __fadd_rn(s, w);
      csr_col[j] = int32_t(c);
      csr_val[j] = s;
    }
    if (e == E - 1)
      for (int64_t q = r + 1; q <= N; ++q) rowptr[q] = incl[e];
  }
}

// Keys of the degree order: decreasing degree, ties by vertex (the sort is stable).
__global__ void __launch_bounds__(256)
degree_key_kernel(const int32_t* __restrict__ deg, uint32_t* __restrict__ keys, int32_t* __restrict__ ids, int64_t N) {
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < N; i += int64_t(gridDim.x) * 256) {
    keys[i] = ~uint32_t(deg[i]);
    ids[i] = int32_t(i);
  }
}
__global__ void __launch_bounds__(256)
degree_perm_kernel(const int32_t* __restrict__ ids, int64_t N, int64_t* __restrict__ perm, int64_t* __restrict__ inv,
                   int32_t* __restrict__ relabel) {
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < N; i += int64_t(gridDim.x) * 256) {
    const int32_t v = ids[i];
    perm[i] = v;
    inv[v] = i;
    if (relabel) relabel[v] = int32_t(i);
  }
}

__global__ void set_one_kernel(int32_t* out) { *out = 1; }

// One warp per row; every entry (i, j, v) looks for (j, i) by bisection of
// row j (columns sorted) and compares the value bits.
__global__ void __launch_bounds__(256)
symmetric_kernel(const int32_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                 const float* __restrict__ val, int M, int32_t* __restrict__ out) {
  const int lane = threadIdx.x % 32;
  const int64_t warps = int64_t(gridDim.x) * 8;
  for (int64_t i = int64_t(blockIdx.x) * 8 + threadIdx.x / 32; i < M; i += warps) {
    const int s = rowptr[i], e = rowptr[i + 1];
    for (int p = s + lane; p < e; p += 32) {
      const int j = col[p];
      bool found = false;
      if (j >= 0 && j < M) {
        int lo = rowptr[j], hi = rowptr[j + 1];
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          const int c = col[mid];
          if (c < int(i)) lo = mid + 1; else hi = mid;
        }
        if (lo < rowptr[j + 1] && col[lo] == int(i))
          found = __float_as_uint(val[lo]) == __float_as_uint(val[p]);
      }
      if (!found) *out = 0;
    }
  }
}

inline int id_bits(int64_t N) {
  int b = 1;
  while ((int64_t(1) << b) < N) ++b;
  return b;
}
inline size_t up256(size_t x) { return (x + 255) & ~size_t(255); }
// Temporary storage of the sorts and scans, by formula so that it is the same without a GPU.
inline size_t cub_bytes(int64_t n) { return (size_t(4) << 20) + size_t(n) / 4; }

inline unsigned grid_for(int64_t n) {
  return unsigned(std::max<int64_t>(1, std::min<int64_t>(gc::ceil_div(n, 256), gc::kNumSMs * 16)));
}

}  // namespace

extern "C" {

int gc_coo_rows_to_rowptr(const int64_t* rows, int64_t nnz, int64_t M, int32_t* rowptr, void* stream) {
  GC_REQUIRE(nnz >= 0 && M >= 0 && nnz < INT32_MAX && M < INT32_MAX, "gc_coo_rows_to_rowptr: size out of range");
  GC_REQUIRE(rowptr && (nnz == 0 || rows), "gc_coo_rows_to_rowptr: null pointer");
  rows_to_rowptr_kernel<<<grid_for(nnz + 1), 256, 0, gc::as_stream(stream)>>>(rows, nnz, M, rowptr);
  return gc::check_launch("gc_coo_rows_to_rowptr");
}

int gc_narrow_i64_i32(const int64_t* src, int32_t* dst, int64_t n, void* stream) {
  GC_REQUIRE(n >= 0, "gc_narrow_i64_i32: negative size");
  if (n == 0) return GC_OK;
  GC_REQUIRE(src && dst, "gc_narrow_i64_i32: null pointer");
  narrow_kernel<<<grid_for(n), 256, 0, gc::as_stream(stream)>>>(src, dst, n);
  return gc::check_launch("gc_narrow_i64_i32");
}

int gc_gcn_norm_f32(const int64_t* row, const int64_t* col, int64_t E, int64_t N, float* deg_scratch, float* w,
                    void* stream) {
  GC_REQUIRE(E >= 0 && N >= 0 && N < INT32_MAX, "gc_gcn_norm_f32: size out of range");
  if (E == 0 || N == 0) return GC_OK;
  GC_REQUIRE(row && col && deg_scratch && w, "gc_gcn_norm_f32: null pointer");
  cudaStream_t st = gc::as_stream(stream);
  cudaError_t e = cudaMemsetAsync(deg_scratch, 0, size_t(N) * 4, st);
  if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "gc_gcn_norm_f32: %s", cudaGetErrorString(e));
  int32_t* deg = reinterpret_cast<int32_t*>(deg_scratch);
  degree_kernel<<<grid_for(E), 256, 0, st>>>(col, E, N, deg);
  dinv_kernel<<<grid_for(N), 256, 0, st>>>(deg, N);
  norm_weight_kernel<<<grid_for(E), 256, 0, st>>>(row, col, E, N, deg_scratch, w);
  return gc::check_launch("gc_gcn_norm_f32", 3);
}

}  // extern "C"

namespace {
// Workspace: [keys][keys, other buffer][running counts, the word for vertices outside the graph, degrees (then their -1/2
// powers)][temporary storage].  The word lies between the last running count and the degrees: read with the one, cleared
// with the others.
struct EdgeWs {
  char *keys, *alt;
  int32_t *incl, *outside, *deg;
  void* cub;
  size_t cub_bytes, total;
};
EdgeWs edge_ws(void* ws, int64_t total, int64_t N) {
  EdgeWs w{};
  char* p = static_cast<char*>(ws);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = p ? p + off : nullptr;
    off += up256(bytes);
    return q;
  };
  const size_t kb = (2 * id_bits(N) <= 32 ? 4 : 8) * size_t(std::max<int64_t>(total, 1));
  w.keys = take(kb);
  w.alt = take(kb);
  w.incl = reinterpret_cast<int32_t*>(take(size_t(total + 1 + N) * 4));
  if (p) {
    w.outside = w.incl + total;
    w.deg = w.outside + 1;
  }
  w.cub_bytes = cub_bytes(total);
  w.cub = take(w.cub_bytes);
  w.total = off;
  return w;
}

template <typename KEY>
int sort_edges(const int64_t* row, const int64_t* col, int64_t E, int64_t N, int64_t total, const int32_t* relabel,
               const EdgeWs& w, int* selector, cudaStream_t st) {
  const int bits = id_bits(N);
  KEY *k0 = reinterpret_cast<KEY*>(w.keys), *k1 = reinterpret_cast<KEY*>(w.alt);
  edge_key_kernel<KEY><<<grid_for(total), 256, 0, st>>>(row, col, E, N, bits, relabel, k0, w.deg, w.outside, total);
  dinv_kernel<<<grid_for(N), 256, 0, st>>>(w.deg, N);
  cub::DoubleBuffer<KEY> db(k0, k1);
  size_t need = 0;
  cudaError_t e = cub::DeviceRadixSort::SortKeys(nullptr, need, db, int(total), 0, 2 * bits, st);
  if (e == cudaSuccess && need > w.cub_bytes)
    return gc::fail(GC_ERR_WORKSPACE, "gc_edges_sort: sort needs %zu bytes of temporary storage", need);
  need = w.cub_bytes;
  if (e == cudaSuccess) e = cub::DeviceRadixSort::SortKeys(w.cub, need, db, int(total), 0, 2 * bits, st);
  if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "gc_edges_sort: sort: %s", cudaGetErrorString(e));
  *selector = db.selector;
  auto heads = thrust::make_transform_iterator(thrust::counting_iterator<int64_t>(0), IsHead<KEY>{db.Current()});
  e = cub::DeviceScan::InclusiveSum(nullptr, need, heads, w.incl, int(total), st);
  if (e == cudaSuccess && need > w.cub_bytes)
    return gc::fail(GC_ERR_WORKSPACE, "gc_edges_sort: scan needs %zu bytes of temporary storage", need);
  need = w.cub_bytes;
  if (e == cudaSuccess) e = cub::DeviceScan::InclusiveSum(w.cub, need, heads, w.incl, int(total), st);
  if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "gc_edges_sort: scan: %s", cudaGetErrorString(e));
  return gc::check_launch("gc_edges_sort", 4);
}
}  // namespace

extern "C" {

size_t gc_edges_workspace_bytes(int64_t E, int64_t N, int self_loops) {
  if (E < 0 || N < 0) return 0;
  return edge_ws(nullptr, E + (self_loops ? N : 0), N).total;
}

int gc_edges_sort(const int64_t* row, const int64_t* col, int64_t E, int64_t N, int self_loops, const int32_t* relabel,
                  void* workspace, size_t workspace_bytes, int* selector, const int32_t** nnz_at, void* stream) {
  const int64_t total = E + (self_loops ? N : 0);
  GC_REQUIRE(E >= 0 && N >= 0 && total < INT32_MAX, "gc_edges_sort: size out of int32 range");
  GC_REQUIRE(total > 0 && (E == 0 || (row && col)) && workspace && selector && nnz_at, "gc_edges_sort: null pointer");
  const EdgeWs w = edge_ws(workspace, total, N);
  if (workspace_bytes < w.total) return gc::fail(GC_ERR_WORKSPACE, "gc_edges_sort: workspace too small");
  cudaStream_t st = gc::as_stream(stream);
  if (cudaMemsetAsync(w.outside, 0, size_t(N + 1) * 4, st) != cudaSuccess)
    return gc::fail(GC_ERR_CUDA, "gc_edges_sort: clearing the degrees failed");
  *nnz_at = w.incl + total - 1;
  return 2 * id_bits(N) <= 32 ? sort_edges<uint32_t>(row, col, E, N, total, relabel, w, selector, st)
                              : sort_edges<uint64_t>(row, col, E, N, total, relabel, w, selector, st);
}

int gc_edges_to_csr(int64_t E, int64_t N, int self_loops, int selector, const void* workspace, size_t workspace_bytes,
                    int32_t* rowptr, int32_t* csr_col, float* csr_val, void* stream) {
  const int64_t total = E + (self_loops ? N : 0);
  GC_REQUIRE(E >= 0 && N >= 0 && total > 0 && total < INT32_MAX, "gc_edges_to_csr: size out of range");
  GC_REQUIRE(workspace && rowptr && csr_col && csr_val, "gc_edges_to_csr: null pointer");
  const EdgeWs w = edge_ws(const_cast<void*>(workspace), total, N);
  if (workspace_bytes < w.total) return gc::fail(GC_ERR_WORKSPACE, "gc_edges_to_csr: workspace too small");
  cudaStream_t st = gc::as_stream(stream);
  const int bits = id_bits(N);
  const char* k = selector ? w.alt : w.keys;
  const float* dinv = reinterpret_cast<const float*>(w.deg);
  if (2 * bits <= 32)
    csr_from_keys_kernel<uint32_t><<<grid_for(total), 256, 0, st>>>(reinterpret_cast<const uint32_t*>(k), w.incl, total, N,
                                                                   bits, dinv, rowptr, csr_col, csr_val);
  else
    csr_from_keys_kernel<uint64_t><<<grid_for(total), 256, 0, st>>>(reinterpret_cast<const uint64_t*>(k), w.incl, total, N,
                                                                   bits, dinv, rowptr, csr_col, csr_val);
  return gc::check_launch("gc_edges_to_csr");
}

size_t gc_degree_order_workspace_bytes(int64_t N) {
  if (N < 0) return 0;
  return 5 * up256(size_t(std::max<int64_t>(N, 1)) * 4) + up256(cub_bytes(N));
}

int gc_degree_order(const int64_t* target, int64_t E, int64_t N, int64_t* perm, int64_t* inv, int32_t* relabel,
                    void* workspace, size_t workspace_bytes, void* stream) {
  GC_REQUIRE(E >= 0 && N >= 0 && N < INT32_MAX, "gc_degree_order: size out of range");
  if (N == 0) return GC_OK;
  GC_REQUIRE((E == 0 || target) && perm && inv && workspace, "gc_degree_order: null pointer");
  if (workspace_bytes < gc_degree_order_workspace_bytes(N))
    return gc::fail(GC_ERR_WORKSPACE, "gc_degree_order: workspace too small");
  cudaStream_t st = gc::as_stream(stream);
  const size_t b = up256(size_t(N) * 4);
  char* p = static_cast<char*>(workspace);
  int32_t* deg = reinterpret_cast<int32_t*>(p);
  cub::DoubleBuffer<uint32_t> dk(reinterpret_cast<uint32_t*>(p + b), reinterpret_cast<uint32_t*>(p + 2 * b));
  cub::DoubleBuffer<int32_t> dv(reinterpret_cast<int32_t*>(p + 3 * b), reinterpret_cast<int32_t*>(p + 4 * b));
  size_t have = cub_bytes(N), need = 0;
  if (cudaMemsetAsync(deg, 0, size_t(N) * 4, st) != cudaSuccess)
    return gc::fail(GC_ERR_CUDA, "gc_degree_order: clearing the degrees failed");
  if (E > 0) degree_kernel<<<grid_for(E), 256, 0, st>>>(target, E, N, deg);
  degree_key_kernel<<<grid_for(N), 256, 0, st>>>(deg, dk.Current(), dv.Current(), N);
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, need, dk, dv, int(N), 0, 32, st);
  if (e == cudaSuccess && need > have)
    return gc::fail(GC_ERR_WORKSPACE, "gc_degree_order: sort needs %zu bytes of temporary storage", need);
  if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(p + 5 * b, have, dk, dv, int(N), 0, 32, st);
  if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "gc_degree_order: sort: %s", cudaGetErrorString(e));
  degree_perm_kernel<<<grid_for(N), 256, 0, st>>>(dv.Current(), N, perm, inv, relabel);
  return gc::check_launch("gc_degree_order", 4);
}

size_t gc_csr_build_workspace_bytes(int64_t E) {
  if (E <= 0) return 256;
  size_t bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, bytes, static_cast<int32_t*>(nullptr), static_cast<int32_t*>(nullptr),
                                int(std::min<int64_t>(E, INT32_MAX)));
  return std::max<size_t>(bytes, 256);
}

int gc_csr_count_unique(const int64_t* row, const int64_t* col, int64_t E, int32_t* head, int64_t* nnz_out,
                        void* workspace, size_t workspace_bytes, void* stream) {
  GC_REQUIRE(E >= 0 && E < INT32_MAX, "gc_csr_count_unique: E out of int32 range");
  GC_REQUIRE(nnz_out, "gc_csr_count_unique: null nnz_out");
  cudaStream_t st = gc::as_stream(stream);
  if (E > 0) {
    GC_REQUIRE(row && col && head, "gc_csr_count_unique: null pointer");
    if (!workspace || workspace_bytes < gc_csr_build_workspace_bytes(E))
      return gc::fail(GC_ERR_WORKSPACE, "gc_csr_count_unique: workspace too small");
    head_flag_kernel<<<grid_for(E), 256, 0, st>>>(row, col, E, head);
    size_t bytes = workspace_bytes;
    cudaError_t e = cub::DeviceScan::ExclusiveSum(workspace, bytes, head, head, int(E), st);
    if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "gc_csr_count_unique: scan: %s", cudaGetErrorString(e));
  }
  total_kernel<<<1, 1, 0, st>>>(row, col, E, head, nnz_out);
  return gc::check_launch("gc_csr_count_unique", E > 0 ? 2 : 1);
}

int gc_csr_fill(const int64_t* row, const int64_t* col, const float* w, int64_t E, int64_t M, const int32_t* head,
                int32_t* rowptr, int32_t* csr_col, float* csr_val, void* stream) {
  GC_REQUIRE(E >= 0 && E < INT32_MAX && M >= 0 && M < INT32_MAX, "gc_csr_fill: size out of int32 range");
  GC_REQUIRE(rowptr, "gc_csr_fill: null rowptr");
  GC_REQUIRE(E == 0 || (row && col && w && head && csr_col && csr_val), "gc_csr_fill: null pointer");
  csr_fill_kernel<<<grid_for(E + 1), 256, 0, gc::as_stream(stream)>>>(row, col, w, E, M, head, rowptr, csr_col,
                                                                       csr_val);
  return gc::check_launch("gc_csr_fill");
}

int gc_csr_is_symmetric(const int32_t* rowptr, const int32_t* col, const float* val, int64_t M, int32_t* out,
                        void* stream) {
  GC_REQUIRE(M >= 0 && M < INT32_MAX, "gc_csr_is_symmetric: M out of range");
  GC_REQUIRE(out, "gc_csr_is_symmetric: null out");
  cudaStream_t st = gc::as_stream(stream);
  set_one_kernel<<<1, 1, 0, st>>>(out);
  if (M > 0) {
    GC_REQUIRE(rowptr, "gc_csr_is_symmetric: null rowptr");
    const unsigned grid = unsigned(std::min<int64_t>(gc::ceil_div(M, 8), gc::kNumSMs * 16));
    symmetric_kernel<<<grid, 256, 0, st>>>(rowptr, col, val, int(M), out);
  }
  return gc::check_launch("gc_csr_is_symmetric", M > 0 ? 2 : 1);
}

}  // extern "C"
