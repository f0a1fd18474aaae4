// Fused classification tail: log_softmax over the class dimension + negative
// log-likelihood of the labelled class, and its gradient with respect to the
// logits.  Takes over the PyTorch ops the reference's training script runs
// after the last layer (tests/gcn/graphcuda_impl.py:24 log_softmax,
// :55 F.nll_loss on the masked rows) -- four kernels and two N x C temporaries
// there, one pass here in each direction.
//
//   loss = scale * sum over selected rows r of ( logsumexp(Z[r, :]) - Z[r, y_r] )
//   dZ[r, c] = g * scale * ( exp(Z[r, c] - lse_r) - [c == y_r] )   for selected rows, 0 otherwise
//
// A group of lanes per row, shuffles for the max / sum; the loss is reduced per warp, per block and by a final single block in
// a fixed order (no atomics, bit-reproducible).
#include "common.cuh"

#include <algorithm>

namespace {

constexpr int kLossBlocks = gc::kNumSMs * 8;

// Rows of up to 128 classes are held in registers, NV vectors of four columns per lane, G = 4 lanes per row (8 above 64
// classes): every logit is read once, with 128-bit loads where the rows are aligned.  Few lanes per row, because the two
// reductions and the logarithm of a row cost each lane the same whatever it holds.  Columns beyond C read as -inf.
template <bool VEC>
__device__ __forceinline__ float4 load_logits(const float* __restrict__ z, int c, int C) {
  if (VEC && c + 4 <= C) return __ldcs(reinterpret_cast<const float4*>(z + c));
  float4 v;
  v.x = c < C ? __ldg(z + c) : -INFINITY;
  v.y = c + 1 < C ? __ldg(z + c + 1) : -INFINITY;
  v.z = c + 2 < C ? __ldg(z + c + 2) : -INFINITY;
  v.w = c + 3 < C ? __ldg(z + c + 3) : -INFINITY;
  return v;
}
template <int G>
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The lanes of a warp, then the 8 warps, in a fixed order.
__device__ __forceinline__ void store_block_loss(float acc, float* __restrict__ partials) {
  __shared__ float warp_loss[8];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) warp_loss[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float b = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) b += warp_loss[w];
    partials[blockIdx.x] = b;
  }
}

template <int G, int NV, bool VEC>
__global__ void __launch_bounds__(256)
lse_nll_forward_rows_kernel(const float* __restrict__ Z, int64_t ldz, const int64_t* __restrict__ labels,
                            const uint8_t* __restrict__ row_mask, int64_t M, int C, float* __restrict__ lse,
                            uint8_t* __restrict__ mask_copy, float* __restrict__ partials) {
  constexpr int R = 32 / G, U = NV >= 3 ? 2 : 4;  // rows per warp pass, passes in flight
  const int lane = threadIdx.x % 32, lg = lane % G, sub = lane / G;
  const int64_t stride = int64_t(gridDim.x) * 8 * R;
  float acc = 0.f;
  for (int64_t r0 = (int64_t(blockIdx.x) * 8 + threadIdx.x / 32) * R; r0 < M; r0 += stride * U) {  // uniform per warp
    float4 v[U][NV];
    int64_t y[U];
    uint8_t chosen[U];
    bool counts[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t r = min(r0 + u * stride + sub, M - 1);
#pragma unroll
      for (int k = 0; k < NV; ++k) v[u][k] = load_logits<VEC>(Z + r * ldz, (k * G + lg) * 4, C);
      y[u] = __ldg(labels + r);
      chosen[u] = row_mask ? __ldg(row_mask + r) : 1;
      counts[u] = r0 + u * stride + sub < M && chosen[u] && y[u] < C;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float mx = -INFINITY, s = 0.f;
#pragma unroll
      for (int k = 0; k < NV; ++k) mx = fmaxf(mx, fmaxf(fmaxf(v[u][k].x, v[u][k].y), fmaxf(v[u][k].z, v[u][k].w)));
      mx = group_max<G>(mx);
#pragma unroll
      for (int k = 0; k < NV; ++k)
        s += (expf(v[u][k].x - mx) + expf(v[u][k].y - mx)) + (expf(v[u][k].z - mx) + expf(v[u][k].w - mx));
      const float l = mx + logf(group_sum<G>(s));
      const int64_t r = r0 + u * stride + sub;
      if (lg == 0 && r < M) {
        lse[r] = l;
        if (row_mask) mask_copy[r] = chosen[u];
      }
#pragma unroll
      for (int k = 0; k < NV; ++k) {  // the lane that holds the label's logit adds the row's loss
        const int64_t at = y[u] - (k * G + lg) * 4;
        if (counts[u] && at >= 0 && at < 4)
          acc += l - (at == 0 ? v[u][k].x : at == 1 ? v[u][k].y : at == 2 ? v[u][k].z : v[u][k].w);
      }
    }
  }
  store_block_loss(acc, partials);
}

// More classes than that: a warp per row, its logits read twice.
__global__ void __launch_bounds__(256)
lse_nll_forward_kernel(const float* __restrict__ Z, int64_t ldz, const int64_t* __restrict__ labels,
                       const uint8_t* __restrict__ row_mask, int64_t M, int C, float* __restrict__ lse,
                       uint8_t* __restrict__ mask_copy, float* __restrict__ partials) {
  const int lane = threadIdx.x % 32;
  const int64_t stride = int64_t(gridDim.x) * 8;
  float acc = 0.f;
  for (int64_t r = int64_t(blockIdx.x) * 8 + threadIdx.x / 32; r < M; r += stride) {
    const float* z = Z + r * ldz;
    float mx = -INFINITY;
    for (int c = lane; c < C; c += 32) mx = fmaxf(mx, __ldg(z + c));
    mx = group_max<32>(mx);
    float s = 0.f;
    for (int c = lane; c < C; c += 32) s += expf(__ldg(z + c) - mx);
    s = group_sum<32>(s);
    if (lane == 0) {
      const float l = mx + logf(s);
      lse[r] = l;
      if (row_mask) mask_copy[r] = row_mask[r];
      if (!row_mask || row_mask[r]) {
        const int64_t y = labels[r];
        if (y >= 0 && y < C) acc += l - __ldg(z + y);
      }
    }
  }
  store_block_loss(acc, partials);
}

__global__ void __launch_bounds__(256)
loss_reduce_kernel(const float* __restrict__ partials, int n, float scale, float* __restrict__ loss) {
  __shared__ float sh[256];
  float a = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) a += partials[i];
  sh[threadIdx.x] = a;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = sh[0] * scale;
}

// One vector of four columns per thread.  PAD: rows of dZ end at the next multiple of 4 columns; zeros are written there.
template <bool VEC, bool PAD>
__global__ void __launch_bounds__(256)
lse_nll_backward_kernel(const float* __restrict__ Z, int64_t ldz, const int64_t* __restrict__ labels,
                        const uint8_t* __restrict__ row_mask, const float* __restrict__ lse,
                        const float* __restrict__ grad_loss, float scale, int64_t M, int C, float* __restrict__ dZ,
                        int64_t lddz) {
  const int quads = (C + 3) / 4;
  const int64_t total = M * quads;
  const float g = (grad_loss ? __ldg(grad_loss) : 1.f) * scale;
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < total; i += int64_t(gridDim.x) * 256) {
    const int64_t r = i / quads;
    const int c = int(i - r * quads) * 4;
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!row_mask || row_mask[r]) {
      const float4 v = load_logits<VEC>(Z + r * ldz, c, C);
      const float l = __ldg(lse + r);
      const int64_t y = __ldg(labels + r) - c;
      d.x = g * (expf(v.x - l) - (y == 0 ? 1.f : 0.f));
      d.y = g * (expf(v.y - l) - (y == 1 ? 1.f : 0.f));
      d.z = g * (expf(v.z - l) - (y == 2 ? 1.f : 0.f));
      d.w = g * (expf(v.w - l) - (y == 3 ? 1.f : 0.f));
    }
    float* p = dZ + r * lddz + c;
    if (PAD) {  // y may name a pad column only for a label that is out of range
      if (c + 1 >= C) d.y = 0.f;
      if (c + 2 >= C) d.z = 0.f;
      if (c + 3 >= C) d.w = 0.f;
    }
    if (VEC && (PAD || c + 4 <= C)) {
      *reinterpret_cast<float4*>(p) = d;
    } else {
      p[0] = d.x;
      if (c + 1 < C) p[1] = d.y;
      if (c + 2 < C) p[2] = d.z;
      if (c + 3 < C) p[3] = d.w;
    }
  }
}

struct MaskList {
  const uint8_t* p[8];  // one byte per row each
};

// Evaluation tail (reference tests/gcn/graphcuda_impl.py:63-68): row-wise
// argmax (lowest index among equal maxima) and, for each of n_masks row
// selections, how many selected rows were predicted right and how many were
// selected.  Integer atomics: the counts do not depend on the order.
// G lanes per row; up to 4 * G classes are read once, four columns per lane (VEC: with 128-bit loads).
template <int G, bool VEC>
__global__ void __launch_bounds__(256)
argmax_count_kernel(const float* __restrict__ Z, int64_t ldz, int64_t M, int C, const int64_t* __restrict__ labels,
                    const MaskList masks, int n_masks, int64_t* __restrict__ pred,
                    unsigned long long* __restrict__ counts) {
  __shared__ unsigned int sh[8][2 * 8];
  constexpr int R = 32 / G;  // rows per warp pass, G lanes each
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int lg = lane % G, sub = lane / G;
  const int64_t stride = int64_t(gridDim.x) * 8 * R;
  unsigned int right[8], chosen[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) right[m] = chosen[m] = 0;
  for (int64_t r0 = (int64_t(blockIdx.x) * 8 + warp) * R; r0 < M; r0 += stride) {  // uniform across the warp
    const int64_t r = r0 + sub;
    const bool valid = r < M;
    const float* z = Z + (valid ? r : 0) * ldz;
    float best = -INFINITY;
    int arg = C;  // no candidate seen yet
    if (valid)
      for (int c0 = lg * 4; c0 < C; c0 += G * 4) {
        const float4 q = load_logits<VEC>(z, c0, C);
        const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c0 + j < C && (v[j] > best || arg == C)) {
            best = v[j];
            arg = c0 + j;
          }
      }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
      if (oa < C && (arg == C || ob > best || (ob == best && oa < arg))) {
        best = ob;
        arg = oa;
      }
    }
    if (valid && lg == 0) {
      if (pred) pred[r] = arg;
      if (labels) {
        const bool hit = labels[r] == int64_t(arg);
        if (n_masks > 0) {
#pragma unroll
          for (int m = 0; m < 8; ++m)  // fixed trip count: the counters stay in registers
            if (m < n_masks && masks.p[m][r]) {
              chosen[m]++;
              right[m] += hit ? 1u : 0u;
            }
        } else {
          chosen[0]++;
          right[0] += hit ? 1u : 0u;
        }
      }
    }
  }
  if (!labels) return;
  const int nm = n_masks > 0 ? n_masks : 1;
  // the R row-slots of a warp (their leaders are lanes 0, G, 2G, ...), then the 8 warps
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    if (m < nm) {  // uniform
#pragma unroll
      for (int o = 16; o >= G; o >>= 1) {
        right[m] += __shfl_xor_sync(0xffffffffu, right[m], o);
        chosen[m] += __shfl_xor_sync(0xffffffffu, chosen[m], o);
      }
      if (lane == 0) {
        sh[warp][2 * m] = right[m];
        sh[warp][2 * m + 1] = chosen[m];
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 * nm) {
    unsigned long long t = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sh[w][threadIdx.x];
    if (t) atomicAdd(counts + threadIdx.x, t);
  }
}


int nll_backward(const float* Z, int64_t ldz, const int64_t* labels, const uint8_t* row_mask, int64_t M, int64_t C,
                 float scale, const float* grad_loss, float* dZ, int64_t lddz, bool pad, const void* workspace,
                 void* stream) {
  GC_REQUIRE(M >= 0 && C >= 1 && C < INT32_MAX, "gc_logsoftmax_nll_backward_f32: bad size");
  if (M == 0) return GC_OK;
  GC_REQUIRE(Z && labels && dZ && workspace, "gc_logsoftmax_nll_backward_f32: null pointer");
  GC_REQUIRE(ldz >= C && lddz >= C, "gc_logsoftmax_nll_backward_f32: leading dimension smaller than C");
  cudaStream_t st = gc::as_stream(stream);
  const float* lse = static_cast<const float*>(workspace) + kLossBlocks;
  const bool vec = ldz % 4 == 0 && lddz % 4 == 0 && gc::aligned16(Z) && gc::aligned16(dZ);
  GC_REQUIRE(!pad || (vec && lddz >= (C + 3) / 4 * 4), "gc_logsoftmax_nll_backward_f32: padded rows must be aligned");
  const unsigned grid = unsigned(std::min<int64_t>(gc::ceil_div(M * ((C + 3) / 4), 256), gc::kNumSMs * 32));
#define GC_BWD(V, P)                                                                                                 \
  lse_nll_backward_kernel<V, P><<<grid, 256, 0, st>>>(Z, ldz, labels, row_mask, lse, grad_loss, scale, M, int(C), dZ, lddz)
  if (vec && pad) GC_BWD(true, true);
  else if (vec) GC_BWD(true, false);
  else GC_BWD(false, false);
#undef GC_BWD
  return gc::check_launch("gc_logsoftmax_nll_backward_f32");
}

}  // namespace

extern "C" {

size_t gc_nll_workspace_bytes(int64_t M) {
  if (M < 0) return 0;
  return size_t(kLossBlocks) * sizeof(float) + size_t(M) * (sizeof(float) + 1);
}

int gc_logsoftmax_nll_forward_f32(const float* Z, int64_t ldz, const int64_t* labels, const uint8_t* row_mask,
                                  int64_t M, int64_t C, float scale, float* loss, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  GC_REQUIRE(M >= 0 && C >= 1 && C < INT32_MAX, "gc_logsoftmax_nll_forward_f32: bad size");
  GC_REQUIRE(loss && workspace, "gc_logsoftmax_nll_forward_f32: null pointer");
  GC_REQUIRE(M == 0 || (Z && labels), "gc_logsoftmax_nll_forward_f32: null pointer");
  GC_REQUIRE(ldz >= C, "gc_logsoftmax_nll_forward_f32: leading dimension smaller than C");
  if (workspace_bytes < gc_nll_workspace_bytes(M))
    return gc::fail(GC_ERR_WORKSPACE, "gc_logsoftmax_nll_forward_f32: workspace too small");
  cudaStream_t st = gc::as_stream(stream);
  float* partials = static_cast<float*>(workspace);
  float* lse = partials + kLossBlocks;
  uint8_t* copy = reinterpret_cast<uint8_t*>(lse + M);
  const int64_t rows_per_block = C <= 64 ? 64 : C <= 128 ? 32 : 8;
  const int blocks = int(std::max<int64_t>(1, std::min<int64_t>(gc::ceil_div(M, rows_per_block), kLossBlocks)));
  const bool vec = ldz % 4 == 0 && gc::aligned16(Z);
#define GC_ROWS(G, NV)                                                                                            \
  (vec ? lse_nll_forward_rows_kernel<G, NV, true><<<blocks, 256, 0, st>>>(Z, ldz, labels, row_mask, M, int(C), lse, \
                                                                         copy, partials)                          \
       : lse_nll_forward_rows_kernel<G, NV, false><<<blocks, 256, 0, st>>>(Z, ldz, labels, row_mask, M, int(C), lse, \
                                                                          copy, partials))
  if (M == 0) cudaMemsetAsync(partials, 0, sizeof(float) * size_t(blocks), st);
  else if (C <= 16) GC_ROWS(4, 1);
  else if (C <= 32) GC_ROWS(4, 2);
  else if (C <= 48) GC_ROWS(4, 3);
  else if (C <= 64) GC_ROWS(4, 4);
  else if (C <= 128) GC_ROWS(8, 4);
  else lse_nll_forward_kernel<<<blocks, 256, 0, st>>>(Z, ldz, labels, row_mask, M, int(C), lse, copy, partials);
#undef GC_ROWS
  loss_reduce_kernel<<<1, 256, 0, st>>>(partials, blocks, scale, loss);
  return gc::check_launch("gc_logsoftmax_nll_forward_f32", 2);
}

int gc_logsoftmax_nll_backward_f32(const float* Z, int64_t ldz, const int64_t* labels, const uint8_t* row_mask,
                                   int64_t M, int64_t C, float scale, const float* grad_loss, float* dZ,
                                   int64_t lddz, const void* workspace, void* stream) {
  return nll_backward(Z, ldz, labels, row_mask, M, C, scale, grad_loss, dZ, lddz, false, workspace, stream);
}

int gc_logsoftmax_nll_backward_pad_f32(const float* Z, int64_t ldz, const int64_t* labels, const uint8_t* row_mask,
                                       int64_t M, int64_t C, float scale, const float* grad_loss, float* dZ,
                                       int64_t lddz, const void* workspace, void* stream) {
  return nll_backward(Z, ldz, labels, row_mask, M, C, scale, grad_loss, dZ, lddz, true, workspace, stream);
}

int gc_argmax_accuracy_f32(const float* Z, int64_t ldz, int64_t M, int64_t C, const int64_t* labels,
                           const uint8_t* masks, int n_masks, int64_t* pred, int64_t* counts, void* stream) {
  GC_REQUIRE(!masks || n_masks >= 1, "gc_argmax_accuracy_f32: masks given with n_masks = 0");
  GC_REQUIRE(n_masks >= 0 && n_masks <= 8, "gc_argmax_accuracy_f32: at most 8 row selections");
  const uint8_t* list[8] = {};
  for (int m = 0; masks && m < n_masks; ++m) list[m] = masks + int64_t(m) * M;
  return gc_argmax_accuracy_masks_f32(Z, ldz, M, C, labels, list, masks ? n_masks : 0, pred, counts, stream);
}

int gc_argmax_accuracy_masks_f32(const float* Z, int64_t ldz, int64_t M, int64_t C, const int64_t* labels,
                                 const uint8_t* const* masks, int n_masks, int64_t* pred, int64_t* counts,
                                 void* stream) {
  GC_REQUIRE(M >= 0 && C >= 1 && C < INT32_MAX, "gc_argmax_accuracy_f32: bad size");
  GC_REQUIRE(ldz >= C, "gc_argmax_accuracy_f32: leading dimension smaller than C");
  GC_REQUIRE(n_masks >= 0 && n_masks <= 8, "gc_argmax_accuracy_f32: at most 8 row selections");
  GC_REQUIRE(n_masks == 0 || masks, "gc_argmax_accuracy_f32: null mask list");
  GC_REQUIRE(!labels || counts, "gc_argmax_accuracy_f32: labels given without counts");
  GC_REQUIRE(M == 0 || Z, "gc_argmax_accuracy_f32: null Z");
  MaskList list{};
  for (int m = 0; m < n_masks; ++m) {
    GC_REQUIRE(masks[m] || M == 0, "gc_argmax_accuracy_f32: null mask");
    list.p[m] = masks[m];
  }
  cudaStream_t st = gc::as_stream(stream);
  if (labels && cudaMemsetAsync(counts, 0, size_t(2 * std::max(n_masks, 1)) * sizeof(int64_t), st) != cudaSuccess)
    return gc::fail(GC_ERR_CUDA, "gc_argmax_accuracy_f32: clearing the counts failed");
  if (M == 0 || (!pred && !labels)) return GC_OK;
  const int group = C <= 16 ? 4 : C <= 64 ? 16 : 32;
  const int64_t rows_per_block = 8 * 32 / group;
  const unsigned blocks = unsigned(std::min<int64_t>(gc::ceil_div(M, rows_per_block), kLossBlocks));
  const bool vec = ldz % 4 == 0 && gc::aligned16(Z);
  auto* out = reinterpret_cast<unsigned long long*>(counts);
#define GC_ARGMAX(G)                                                                                              \
  (vec ? argmax_count_kernel<G, true><<<blocks, 256, 0, st>>>(Z, ldz, M, int(C), labels, list, n_masks, pred, out) \
       : argmax_count_kernel<G, false><<<blocks, 256, 0, st>>>(Z, ldz, M, int(C), labels, list, n_masks, pred, out))
  if (group == 4) GC_ARGMAX(4);
  else if (group == 16) GC_ARGMAX(16);
  else GC_ARGMAX(32);
#undef GC_ARGMAX
  return gc::check_launch("gc_argmax_accuracy_f32");
}

}  // extern "C"
