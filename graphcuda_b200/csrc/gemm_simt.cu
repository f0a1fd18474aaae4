// IEEE fp32 GEMM on CUDA cores with a fixed summation order.
//
// The bit-stable path behind gc_gemm_f32: it serves every shape and leading
// dimension (the tensor-core path needs 16-byte aligned rows), the small
// Cora-sized products where launch latency dominates, and it is the on-device
// cross-check for the tcgen05 kernels.  Takes over matmul1..4
// (src/graphcuda/cuda/matmul1.cu:5-23, matmul2.cu:3-62, matmul3.cu:8-191,
// matmul4.cu:44-206) and cublasSgemm as wrapped by
// src/graphcuda/cuda/gemm_cublas.cu:37-48; unlike matmul3/matmul4 it is
// correct for every M, N, K (no tile-shape or N%4 preconditions).
//
// Bound: FP32 FMA issue for square shapes, latency for the small ones.  A CTA
// computes BM x BN outputs with 256 threads; each stage of BK k-values is
// copied as it lies in memory (k-contiguous or m/n-contiguous, no transposition)
// by cp.async, ST stages deep: 16-byte copies where rows are aligned, 4-byte
// ones where they are not.  A thread takes four k-values at a time with 128-bit
// shared-memory reads of either layout and accumulates with packed FMAs
// (fma.rn.f32x2: two IEEE FMAs per issue slot), so the FMA pipe and not the
// issue slots or the shared-memory reads set the pace.  For narrow outputs the
// 256 threads split the k-values of a stage WK ways (a 64 x 16 tile alone would
// keep two warps busy).  K is split further over a cluster of up to 8 CTAs that
// add their tiles through distributed shared memory in rank order -- one launch,
// no workspace -- and, for long sums, over gridDim.z with partial tiles in the
// workspace and a second kernel.  Every order of additions is fixed.
#include "common.cuh"
#include "gemm_internal.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

__device__ __forceinline__ void copy16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One operand's stage.  KC: k is the contiguous direction (rows of X indices, pitch BK + 4: eight lanes reading
// 128 bits of eight consecutive rows hit distinct banks); else rows of k-values, pitch BX + 4.
template <int BX, int BK, bool KC>
struct Stage {
  static constexpr int kPitch = KC ? BK + 4 : BX + 4;
  static constexpr int kFloats = KC ? BX * kPitch : BK * kPitch;
  // A thread copies the elements (or quads) r + j * step of one column c of the stage, j = 0 .. kCopies - 1: addresses
  // advance by constants and the only per-stage work is the bound of the k direction.
  template <bool VEC>
  struct Copier {
    static constexpr int V = VEC ? 4 : 1;
    static constexpr int R = KC ? BX : BK, C = KC ? BK : BX;  // rows and contiguous elements of a stage
    static constexpr int kStep = 256 * V / C, kCopies = (R + kStep - 1) / kStep;
    const float* g;
    int64_t row_step;
    int r, c, x_left, ke;  // x_left: valid elements from this thread's first one in the X direction
    __device__ __forceinline__ Copier(const float* base, int64_t ld, int x0, int X, int k0, int ke_, int tid)
        : row_step(int64_t(kStep) * ld), r(tid / (C / V)), c((tid % (C / V)) * V), ke(ke_) {
      g = base + int64_t((KC ? x0 : k0) + r) * ld + (KC ? k0 : x0) + c;
      x_left = X - x0 - (KC ? r : c);
    }
    __device__ __forceinline__ void operator()(float* s, int64_t ld, int k, int kt) const {
      const float* p = g + (KC ? int64_t(kt) * BK : int64_t(kt) * BK * ld);
      const int k_left = ke - k - (KC ? c : r);
#pragma unroll
      for (int j = 0; j < kCopies; ++j, p += row_step) {
        if (R % kStep != 0 && r + j * kStep >= R) break;
        const int rows = KC ? x_left : k_left, cols = KC ? k_left : x_left;  // left of this thread's row / column
        const int n = j * kStep < rows ? (VEC ? max(0, min(4, cols)) : (cols > 0 ? 1 : 0)) : 0;
        float* d = s + (r + j * kStep) * kPitch + c;
        if (VEC) copy16(d, p, n * 4);
        else copy4(d, p, n * 4);
      }
    }
  };
  // Index within the tile of a thread's i-th row (t: its position among `threads` of this direction).
  template <int T>
  static __device__ __forceinline__ int index(int t, int i) {
    constexpr int kThreads = BX / T;
    return KC ? t + i * kThreads : (i / 4) * (kThreads * 4) + t * 4 + (i & 3);
  }
  // f[i][q] = element (index(t, i), k + q), q = 0..3
  template <int T>
  static __device__ __forceinline__ void frag(const float* s, int t, int k, float (&f)[T][4]) {
    if constexpr (KC) {
#pragma unroll
      for (int i = 0; i < T; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(s + index<T>(t, i) * kPitch + k);
        f[i][0] = v.x; f[i][1] = v.y; f[i][2] = v.z; f[i][3] = v.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int h = 0; h < T / 4; ++h) {
          const float4 v = *reinterpret_cast<const float4*>(s + (k + q) * kPitch + index<T>(t, h * 4));
          f[h * 4][q] = v.x; f[h * 4 + 1][q] = v.y; f[h * 4 + 2][q] = v.z; f[h * 4 + 3][q] = v.w;
        }
    }
  }
};

template <int BM, int BN, int TM, int TN, int WK, int BK, int ST, bool TA, bool TB>
struct Tile {
  using SA = Stage<BM, BK, !TA>;
  using SB = Stage<BN, BK, TB>;
  static constexpr int kStage = SA::kFloats + SB::kFloats;
  static constexpr int kRed = BM * BN * WK;  // the threads' sums, reusing the stages
  static constexpr int kFloats = ST * kStage > kRed ? ST * kStage : kRed;
  static constexpr int kBytes = kFloats * 4;
  static_assert((BM / TM) * (BN / TN) * WK == 256, "256 threads per CTA");
  static_assert(kBytes <= 227 * 1024, "shared memory");
};

struct Args {
  int M, N, K;
  const float* A;
  int64_t lda;
  const float* B;
  int64_t ldb;
  float* C;
  int64_t ldc;
  gc::GemmEpilogue ep;
  int k_per_split;
  float* partial;  // [gridDim.z][M][N] or null
};

template <int BM, int BN, int TM, int TN, int WK, int BK, int ST, bool TA, bool TB, bool VA, bool VB>
__global__ void __launch_bounds__(256, 2)
gemm_simt_kernel(const __grid_constant__ Args p) {
  using T = Tile<BM, BN, TM, TN, WK, BK, ST, TA, TB>;
  using SA = typename T::SA;
  using SB = typename T::SB;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int kb = blockIdx.z * p.k_per_split;
  const int ke = min(p.K, kb + p.k_per_split);
  // a warp covers 8 threads along M (where the tile has them) x 4 along N
  constexpr int NM = BM / TM, NN = BN / TN, GROUP = NM * NN;
  constexpr int LM = NM >= 8 ? 8 : NM, LN = 32 / LM < NN ? 32 / LM : NN, PW = LM * LN;
  const int wk = tid / GROUP, g = tid % GROUP;
  const int w = g / PW, l = g % PW;
  const int ty = (w % (NM / LM)) * LM + l % LM, tx = (w / (NM / LM)) * LN + l / LM;

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  const int nkt = (ke - kb + BK - 1) / BK;
  const typename SA::template Copier<VA> copy_a(p.A, p.lda, m0, p.M, kb, ke, tid);
  const typename SB::template Copier<VB> copy_b(p.B, p.ldb, n0, p.N, kb, ke, tid);
  auto issue = [&](int kt) {
    if (kt < nkt) {
      float* s = sm + (kt % ST) * T::kStage;
      copy_a(s, p.lda, kb + kt * BK, kt);
      copy_b(s + SA::kFloats, p.ldb, kb + kt * BK, kt);
    }
    copies_commit();
  };
#pragma unroll
  for (int s = 0; s < ST - 1; ++s) issue(s);
  for (int kt = 0; kt < nkt; ++kt) {
    copies_wait<ST - 2>();
    __syncthreads();
    issue(kt + ST - 1);
    const float* sa = sm + (kt % ST) * T::kStage;
    const float* sb = sa + SA::kFloats;
#pragma unroll
    for (int kk = 0; kk < BK / WK; kk += 4) {
      float a[TM][4], b[TN][4];
      SA::template frag<TM>(sa, ty, wk * (BK / WK) + kk, a);
      SB::template frag<TN>(sb, tx, wk * (BK / WK) + kk, b);
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i][q], b[j][q], acc[i][j]);
    }
  }
  copies_wait<0>();

  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = int(cluster.num_blocks());
  float* partial = p.partial ? p.partial + int64_t(blockIdx.z) * p.M * p.N : nullptr;
  if (WK == 1 && ranks == 1) {
    const bool vec = !TB && !p.ep.transposed && !partial && (p.ldc % 4 == 0) &&
                     (reinterpret_cast<uintptr_t>(p.C) & 15) == 0 && !p.ep.mask && !p.ep.gate;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + SA::template index<TM>(ty, i);
      if (gm >= p.M) continue;
#pragma unroll
      for (int h = 0; h < TN; h += 4) {
        float v[4] = {acc[i][h], acc[i][h + 1], acc[i][h + 2], acc[i][h + 3]};
        const int gn = n0 + SB::template index<TN>(tx, h);
        if (vec && gn + 4 <= p.N) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (p.ep.bias) v[j] += __ldg(p.ep.bias + gn + j);
            if (p.ep.relu) v[j] *= v[j] > 0.f ? 1.f : 0.f;
          }
          *reinterpret_cast<float4*>(p.C + int64_t(gm) * p.ldc + gn) = make_float4(v[0], v[1], v[2], v[3]);
          continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int n = n0 + SB::template index<TN>(tx, h + j);
          if (n >= p.N) continue;
          if (partial) partial[int64_t(gm) * p.N + n] = v[j];
          else gc::epilogue_store(v[j], gm, n, p.C, p.ldc, p.ep);
        }
      }
    }
    return;
  }

  // Sums of the WK groups, then of the cluster's CTAs, added in order.
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
      sm[wk * (BM * BN) + SA::template index<TM>(ty, i) * BN + SB::template index<TN>(tx, j)] = acc[i][j];
  __syncthreads();
  const bool last = ranks == 1;
  for (int e = tid; e < BM * BN; e += 256) {
    float s = sm[e];
#pragma unroll
    for (int q = 1; q < WK; ++q) s += sm[q * (BM * BN) + e];
    if (!last) {
      sm[e] = s;
      continue;
    }
    const int gm = m0 + e / BN, gn = n0 + e % BN;
    if (gm >= p.M || gn >= p.N) continue;
    if (partial) partial[int64_t(gm) * p.N + gn] = s;
    else gc::epilogue_store(s, gm, gn, p.C, p.ldc, p.ep);
  }
  if (last) return;
  cluster.sync();
  const int rank = int(cluster.block_rank());
  for (int e = rank * 256 + tid; e < BM * BN; e += ranks * 256) {
    const int gm = m0 + e / BN, gn = n0 + e % BN;
    if (gm >= p.M || gn >= p.N) continue;
    float s = 0.f;
    for (int r = 0; r < ranks; ++r) s += cluster.map_shared_rank(sm, r)[e];
    gc::epilogue_store(s, gm, gn, p.C, p.ldc, p.ep);
  }
  cluster.sync();  // the peers read this CTA's tile until here
}

// ------------------------------------------------------------------ host
struct Shape {
  int bm, bn, bk;
};
// Narrow tiles by the width of the output; 64 x 64 and 128 x 128 for the rest.
constexpr Shape kShapes[] = {{64, 8, 64}, {64, 16, 64}, {64, 32, 32}, {64, 64, 16}, {128, 128, 16}};

struct Choice {
  int shape, splits;
  bool cluster;  // the splits are one cluster (else partial tiles and a second kernel)
  int64_t k_per_split;
};

Choice choose(int64_t M, int64_t N, int64_t K) {
  using gc::ceil_div;
  using gc::kNumSMs;
  Choice best{};
  auto tiles = [&](int s) { return ceil_div(M, kShapes[s].bm) * ceil_div(N, kShapes[s].bn); };
  if (N <= 32) {
    best.shape = N <= 8 ? 0 : N <= 16 ? 1 : 2;
    // about two CTAs per SM; a split keeps at least two stages of k-values
    const int64_t want = ceil_div(2 * kNumSMs, std::max<int64_t>(tiles(best.shape), 1));
    const int64_t most = std::max<int64_t>(1, K / (2 * kShapes[best.shape].bk));
    int64_t s = std::min(want, most);
    if (s > 8 && K > 8192) {  // long sums: more splits than a cluster has CTAs, at least 512 k-values each
      best.splits = int(std::min<int64_t>({s, ceil_div(K, 512), 512}));
    } else {
      s = s >= 8 ? 8 : s >= 4 ? 4 : s >= 2 ? 2 : 1;
      best.splits = int(s);
      best.cluster = s > 1;
    }
  } else {
    // Time of the busiest SM in FMA clocks: CTAs on it x tile x k-values, the smaller tile at 0.8 of the larger one's
    // rate, plus the latency of a CTA's first stage and of the exchange of a split tile.
    double least = 0;
    for (int s = 3; s <= 4; ++s)
      for (int64_t z = 1; z <= 8; z *= 2) {
        if (z > 1 && K / z < 64) break;
        const double area = double(kShapes[s].bm) * kShapes[s].bn;
        const double per_sm = double(ceil_div(tiles(s) * z, kNumSMs));
        const double t = per_sm * (area * double(ceil_div(K, z)) / 128.0 * (s == 3 ? 1.25 : 1.0) +
                                   (z > 1 ? area / 4 : 0.0) + 1000.0);
        if (least == 0 || t < least) {
          least = t;
          best.shape = s;
          best.splits = int(z);
          best.cluster = z > 1;
        }
      }
    const int64_t t = tiles(best.shape);
    if (t * 8 < kNumSMs && K > 8192) {  // weight gradients: few tiles, long sums
      best.cluster = false;
      best.splits = int(std::min<int64_t>({ceil_div(2 * kNumSMs, t), ceil_div(K, 512), 512}));
    }
  }
  const int64_t bk = kShapes[best.shape].bk;
  best.k_per_split = std::max<int64_t>(bk, ceil_div(ceil_div(K, best.splits), bk) * bk);
  if (!best.cluster) best.splits = int(std::max<int64_t>(1, ceil_div(K, best.k_per_split)));
  return best;
}

template <int BM, int BN, int TM, int TN, int WK, int BK, int ST, bool TA, bool TB, bool VA, bool VB>
int launch_one(const Args& p, dim3 grid, int cluster, cudaStream_t st) {
  using T = Tile<BM, BN, TM, TN, WK, BK, ST, TA, TB>;
  auto kern = gemm_simt_kernel<BM, BN, TM, TN, WK, BK, ST, TA, TB, VA, VB>;
  if (T::kBytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kBytes);
    if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "gemm_simt: %s", cudaGetErrorString(e));
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = T::kBytes;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = unsigned(cluster);
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, p);
  return gc::check_launch("gemm_simt");
}

// A tile shape in the four layouts; aligned rows on both operands or on neither (one variant each).
template <int BM, int BN, int TM, int TN, int WK, int BK, int ST>
int launch(bool ta, bool tb, bool vec, const Args& p, dim3 grid, int cluster, cudaStream_t st) {
#define GC_L(TA_, TB_)                                                                                   \
  (vec ? launch_one<BM, BN, TM, TN, WK, BK, ST, TA_, TB_, true, true>(p, grid, cluster, st)              \
       : launch_one<BM, BN, TM, TN, WK, BK, ST, TA_, TB_, false, false>(p, grid, cluster, st))
  if (!ta && !tb) return GC_L(false, false);
  if (!ta) return GC_L(false, true);
  if (!tb) return GC_L(true, false);
  return GC_L(true, true);
#undef GC_L
}

}  // namespace

namespace gc {

// The first 256 bytes of every GEMM workspace hold the tensor-core path's
// sticky error word; split-K partials start behind it.
constexpr size_t kFlagBytes = 256;

size_t simt_workspace_bytes(bool ta, int64_t M, int64_t N, int64_t K) {
  if (narrow_supported(ta, M, N, K)) {
    const size_t b = narrow_partial_bytes(ta, M, N, K);
    return b ? kFlagBytes + b : 0;
  }
  const Choice c = choose(M, N, K);
  return c.splits > 1 && !c.cluster ? kFlagBytes + size_t(c.splits) * size_t(M) * size_t(N) * sizeof(float) : 0;
}

int gemm_simt(bool ta, bool tb, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B,
              int64_t ldb, float* C, int64_t ldc, const GemmEpilogue& ep, void* workspace, size_t workspace_bytes,
              cudaStream_t st) {
  if (narrow_supported(ta, M, N, K)) {
    const size_t need = narrow_partial_bytes(ta, M, N, K);
    const bool have = need && workspace && workspace_bytes >= kFlagBytes + need;
    return gemm_narrow(ta, tb, M, N, K, A, lda, B, ldb, C, ldc, ep,
                       have ? reinterpret_cast<float*>(static_cast<char*>(workspace) + kFlagBytes) : nullptr, st);
  }
  Choice c = choose(M, N, K);
  Args p{int(M), int(N), int(K), A, lda, B, ldb, C, ldc, ep, 0, nullptr};
  if (c.splits > 1 && !c.cluster) {
    if (!workspace || workspace_bytes < simt_workspace_bytes(ta, M, N, K)) {
      c.splits = 1;
      c.k_per_split = ceil_div(std::max<int64_t>(K, 1), kShapes[c.shape].bk) * kShapes[c.shape].bk;
    } else {
      p.partial = reinterpret_cast<float*>(static_cast<char*>(workspace) + kFlagBytes);
    }
  }
  p.k_per_split = int(std::min<int64_t>(c.k_per_split, INT32_MAX));
  const bool vec = lda % 4 == 0 && aligned16(A) && ldb % 4 == 0 && aligned16(B);
  const dim3 grid(unsigned(ceil_div(M, kShapes[c.shape].bm)), unsigned(ceil_div(N, kShapes[c.shape].bn)),
                  unsigned(c.splits));
  if (grid.y > 65535u) return fail(GC_ERR_UNSUPPORTED, "gemm_simt: N too large for this launch shape");
  const int cluster = c.cluster ? c.splits : 1;
  int rc;
  switch (c.shape) {
    case 0: rc = launch<64, 8, 4, 4, 8, 64, 3>(ta, tb, vec, p, grid, cluster, st); break;
    case 1: rc = launch<64, 16, 4, 4, 4, 64, 3>(ta, tb, vec, p, grid, cluster, st); break;
    case 2: rc = launch<64, 32, 4, 4, 2, 32, 3>(ta, tb, vec, p, grid, cluster, st); break;
    case 3: rc = launch<64, 64, 4, 4, 1, 16, 4>(ta, tb, vec, p, grid, cluster, st); break;
    default: rc = launch<128, 128, 8, 8, 1, 16, 3>(ta, tb, vec, p, grid, cluster, st); break;
  }
  if (rc != GC_OK || !p.partial) return rc;
  return splitk_reduce(int(M), int(N), c.splits, p.partial, C, ldc, ep, st);
}

}  // namespace gc
