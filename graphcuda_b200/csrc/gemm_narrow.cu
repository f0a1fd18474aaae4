// IEEE fp32 products with at most 16 output columns (the hidden layer and the
// classes of a Cora-sized model), CUDA cores, fixed summation order.
//
// A 64 x 16 tile staged through shared memory spends more instructions on
// staging than on the 16 FMAs an A element takes part in (2708 x 16 x 1433:
// 17 us, 3.7 instructions per FMA).  Both kernels here keep A out of shared
// memory and hold a register tile per warp:
//   lanes along k (A k-contiguous): a lane keeps its k's row of B in registers
//     and applies it to R rows of A, so 32 consecutive k of each row are one
//     coalesced load whatever the row pitch; the lanes' sums are folded by
//     shuffles, the 8 warps of a CTA (which split k) through shared memory;
//   lanes along m (A m-contiguous, the weight gradients): no folding across
//     lanes at all; the 8 warps of a CTA split k and add up through shared
//     memory, CTAs split k further (gridDim.y).
// Splits across CTAs are added in order, by a cluster through distributed
// shared memory when one cluster covers the output, else by a second kernel.
// Bound: latency of a few dependent loads, then instruction issue.  Measured:
// 2708 x 16 x 1433 19.8 -> 12.1 us, 1433 x 16 x 2708 24.9 -> 10.6 us,
// 16 x 7 x 2708 14.1 -> 5.3 us.
#include "common.cuh"
#include "gemm_internal.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

struct Args {
  int M, N, K;
  const float* A;
  int64_t lda;
  const float* B;
  int64_t ldb;
  float* C;
  int64_t ldc;
  gc::GemmEpilogue ep;
  float* partial;  // [splits][M][N] or null
};

// One k-block of 32: R rows' values in a[], the lane's row of B applied to them.
template <int R, int NP>
__device__ __forceinline__ void apply(float (&acc)[R * NP], const float (&a)[R], const float (&b)[NP]) {
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[r * NP + j] = fmaf(a[r], b[j], acc[r * NP + j]);
}

// A is M x K, k contiguous, any row pitch.  CTA: 8 / WK groups of R rows; the WK warps of a group take k-blocks of 32 in
// turn.  B passes through shared memory in chunks of kChunk rows (from L1 / L2 its latency was exposed once per block:
// 12.5 us for K = 1433 however few rows there were), A is requested PD blocks ahead in registers.
constexpr int kChunk = 1536;
template <int NP>
constexpr int chunk_bytes() { return kChunk * NP * 4; }

// Where 16-byte unit j of row k lies: the units are rotated so that the 8 rows that a quarter of a warp reads with one
// 128-bit access hit 8 distinct units of the 128 bytes of banks (unrotated rows of 64 bytes: 4-way conflicts).
template <int NP>
__device__ __forceinline__ int unit_of(int k, int j) {
  constexpr int CH = NP / 4;
  return k * CH + (j ^ ((k / (8 / CH)) & (CH - 1)));
}

template <int R, int NP, int WK, bool TB, bool VB>
__global__ void __launch_bounds__(256, 2)
narrow_k_kernel(const __grid_constant__ Args p) {
  constexpr int G = 8 / WK, PD = 4;
  extern __shared__ __align__(16) float bs[];  // [k of the chunk][NP]
  __shared__ float sums[8][R * NP];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int m0 = (int(blockIdx.x) * G + warp / WK) * R;
  float acc[R * NP];
#pragma unroll
  for (int i = 0; i < R * NP; ++i) acc[i] = 0.f;
  const float* a0[R];
#pragma unroll
  for (int r = 0; r < R; ++r)  // rows beyond M are not stored
    a0[r] = p.A + int64_t(min(m0 + r, p.M - 1)) * p.lda + (warp % WK) * 32 + lane;

  for (int c0 = 0; c0 < p.K; c0 += kChunk) {
    const int kc = min(kChunk, p.K - c0), kz = (kc + 31) & ~31;  // zeros up to whole blocks
    if (c0 > 0) __syncthreads();
    if (VB) {
      for (int i = threadIdx.x * 4; i < kz * NP; i += 1024) {
        const int k = i / NP, ok = k < kc;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         uint32_t(__cvta_generic_to_shared(bs + 4 * unit_of<NP>(k, i % NP / 4)))),
                     "l"(ok ? p.B + int64_t(c0 + k) * p.ldb + i % NP : p.B), "r"(ok ? 16 : 0) : "memory");
      }
    } else {
      for (int i = threadIdx.x; i < kz * NP; i += 256) {
        const int k = TB ? i % kz : i / NP, n = TB ? i / kz : i % NP;  // along B's contiguous direction
        const int ok = k < kc && n < p.N;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                         uint32_t(__cvta_generic_to_shared(bs + 4 * unit_of<NP>(k, n / 4) + n % 4))),
                     "l"(ok ? (TB ? p.B + int64_t(n) * p.ldb + c0 + k : p.B + int64_t(c0 + k) * p.ldb + n) : p.B),
                     "r"(ok ? 4 : 0) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int k_lane = (warp % WK) * 32 + lane;  // of this warp's first block
    float a[PD][R];
    auto fetch = [&](float (&v)[R], int kk) {  // kk: offset of the block from this warp's first one
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = k_lane + kk < kc ? __ldg(a0[r] + c0 + kk) : 0.f;
    };
#pragma unroll
    for (int u = 0; u < PD; ++u) fetch(a[u], u * 32 * WK);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int kk = 0; kk + (warp % WK) * 32 < kc; kk += PD * 32 * WK) {
#pragma unroll
      for (int u = 0; u < PD; ++u) {
        const int at = kk + u * 32 * WK;
        if (at + (warp % WK) * 32 < kc) {  // uniform across the warp
          float b[NP];
#pragma unroll
          for (int j = 0; j < NP; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(bs + 4 * unit_of<NP>(k_lane + at, j / 4));
            b[j] = v.x; b[j + 1] = v.y; b[j + 2] = v.z; b[j + 3] = v.w;
          }
          apply<R, NP>(acc, a[u], b);
          fetch(a[u], at + PD * 32 * WK);
        }
      }
    }
  }
  // Across the lanes: every step halves the values a lane keeps (R * NP values end up spread over 32 lanes).
  int base = 0;
#pragma unroll
  for (int o = 16, n = R * NP / 2; o > 0; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float give = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
    base += up ? n : 0;
  }
#pragma unroll
  for (int i = 0; i < R * NP / 32; ++i) sums[warp][base + i] = acc[i];
  __syncthreads();
  for (int e = threadIdx.x; e < G * R * NP; e += 256) {
    const int g = e / (R * NP), i = e % (R * NP);
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < WK; ++w) s += sums[g * WK + w][i];
    const int m = (int(blockIdx.x) * G + g) * R + i / NP, n = i % NP;
    if (m < p.M && n < p.N) gc::epilogue_store(s, m, n, p.C, p.ldc, p.ep);
  }
}

// A is K x M, m contiguous.  CTA: 32 * R rows of C and one of gridDim.y ranges of k, split over its 8 warps.
template <int R, int NP, bool TB>
__global__ void __launch_bounds__(256)
narrow_m_kernel(const __grid_constant__ Args p) {
  constexpr int BM = 32 * R, U = 16;
  __shared__ __align__(16) float sums[8][BM * (NP + 1)];  // and, while summing, each warp's rows of B
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int m0 = blockIdx.x * BM;
  const int per = (p.K + int(gridDim.y) * 8 - 1) / (int(gridDim.y) * 8);
  const int kb = (int(blockIdx.y) * 8 + warp) * per, ke = min(p.K, kb + per);
  float acc[R][NP];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[r][j] = 0.f;
  const float* a0 = p.A + m0 + lane;
  for (int k = kb; k < ke; k += U) {
    float a[U][R];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r)
        a[u][r] = (k + u < ke && m0 + lane + 32 * r < p.M) ? __ldg(a0 + int64_t(k + u) * p.lda + 32 * r) : 0.f;
    // The U rows of B, U * NP values, spread over the lanes by one load each and turned through shared memory.
    float* bs = &sums[warp][0];
#pragma unroll
    for (int i = lane; i < U * NP; i += 32) {
      const int u = i / NP, n = i % NP;
      bs[i] = (k + u < ke && n < p.N) ? __ldg(TB ? p.B + int64_t(n) * p.ldb + k + u : p.B + int64_t(k + u) * p.ldb + n) : 0.f;
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int j = 0; j < NP; j += 4) {
        const float4 b = *reinterpret_cast<const float4*>(bs + u * NP + j);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          acc[r][j] = fmaf(a[u][r], b.x, acc[r][j]);
          acc[r][j + 1] = fmaf(a[u][r], b.y, acc[r][j + 1]);
          acc[r][j + 2] = fmaf(a[u][r], b.z, acc[r][j + 2]);
          acc[r][j + 3] = fmaf(a[u][r], b.w, acc[r][j + 3]);
        }
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < NP; ++j) sums[warp][(32 * r + lane) * (NP + 1) + j] = acc[r][j];
  __syncthreads();
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = int(cluster.num_blocks());
  float* partial = p.partial ? p.partial + int64_t(blockIdx.y) * p.M * p.N : nullptr;
  for (int e = threadIdx.x; e < BM * NP; e += 256) {
    const int m = m0 + e / NP, n = e % NP, i = (e / NP) * (NP + 1) + n;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += sums[w][i];
    if (ranks > 1) {
      sums[0][i] = s;  // element i of row 0 is read by this thread alone
    } else if (m < p.M && n < p.N) {
      if (partial) partial[int64_t(m) * p.N + n] = s;
      else gc::epilogue_store(s, m, n, p.C, p.ldc, p.ep);
    }
  }
  if (ranks == 1) return;
  cluster.sync();
  for (int e = int(cluster.block_rank()) * 256 + threadIdx.x; e < BM * NP; e += ranks * 256) {
    const int m = m0 + e / NP, n = e % NP;
    if (m >= p.M || n >= p.N) continue;
    float s = 0.f;
    for (int r = 0; r < ranks; ++r) s += cluster.map_shared_rank(&sums[0][0], r)[(e / NP) * (NP + 1) + n];
    gc::epilogue_store(s, m, n, p.C, p.ldc, p.ep);
  }
  cluster.sync();  // the peers read this CTA's sums until here
}

struct MPlan {
  int r, splits;
  bool cluster;
};
MPlan m_plan(int64_t M, int64_t N, int64_t K) {
  using gc::ceil_div;
  MPlan pl{};
  pl.r = M <= 32 ? 1 : 2;
  const int64_t tiles = ceil_div(M, 32 * pl.r);
  // Two CTAs per SM and not one more (299 of them for 296 places: 1433 x 16 x 2708 12.7 us, 276 10.6; 3703 x 16 x 3327
  // 26.8 and 22.3), at least 16 k-values per warp.
  int64_t s = std::min<int64_t>(std::max<int64_t>(1, 2 * gc::kNumSMs / tiles), std::max<int64_t>(1, K / 128));
  // One cluster covers the output: at most 8 CTAs, no second kernel (16 x 7, cluster / splits over more CTAs: K = 1024 3.9 /
  // 4.8 us, 2048 4.9 / 5.2, 2708 5.9 / 5.9, 4096 6.7 / 4.9, 8192 10.3 / 5.4; 64 x 16 5.4 / 5.9 ... 15.4 / 6.5).
  pl.cluster = tiles == 1 && s > 1 && K <= 2816;
  if (pl.cluster) s = s >= 8 ? 8 : s >= 4 ? 4 : 2;
  pl.splits = int(s);
  return pl;
}

template <int NP, bool TB>
int launch_m(const Args& p, const MPlan& pl, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(gc::ceil_div(p.M, 32 * pl.r)), unsigned(pl.splits));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = unsigned(pl.splits);
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = pl.cluster ? 1 : 0;
  if (pl.r == 1) cudaLaunchKernelEx(&cfg, narrow_m_kernel<1, NP, TB>, p);
  else cudaLaunchKernelEx(&cfg, narrow_m_kernel<2, NP, TB>, p);
  return gc::check_launch("narrow_m_kernel");
}

template <int NP, bool TB, bool VB>
int launch_k(const Args& p, cudaStream_t st) {
  constexpr int R = 4;
  const int64_t groups = gc::ceil_div(p.M, R);
  const int bytes = int(std::min<int64_t>(kChunk, (p.K + 31) & ~31)) * NP * 4;
  auto go = [&](auto kern, int g) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, chunk_bytes<NP>());
    if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "narrow_k_kernel: %s", cudaGetErrorString(e));
    kern<<<unsigned(gc::ceil_div(groups, g)), 256, bytes, st>>>(p);
    return int(GC_OK);
  };
  // the least splitting of k that still gives every SM a CTA (2708 x 16 x 1433: 12.1 us at 2, 12.7 at 4, 14.8 at 8;
  // 148 rows: 8.6, 5.9, 4.7)
  int rc;
  if (groups >= 4 * gc::kNumSMs) rc = go(narrow_k_kernel<R, NP, 2, TB, VB>, 4);
  else if (groups >= 2 * gc::kNumSMs) rc = go(narrow_k_kernel<R, NP, 4, TB, VB>, 2);
  else rc = go(narrow_k_kernel<R, NP, 8, TB, VB>, 1);
  if (rc != GC_OK) return rc;
  return gc::check_launch("narrow_k_kernel");
}

}  // namespace

namespace gc {

// Where these kernels take the place of the tiled one.  Measured as time here over time there, 2500 sizes (M 256 to 20 K, or
// 7 to 16 K for the weight gradients, K 16 to 65 K, N 3 to 16), and as error against float64:
//   lanes along k: 0.4..1.0 while the rows fit the GPU at once (2 CTAs of 16 rows per SM: 4736) and B is one chunk of
//     k (1536; below K = 128 only with up to 8 columns, else up to 1.13), 1.0..1.5 at 5000 to 10,000 rows, 1.1..2.3 at
//     12 K to 20 K and at K = 2048 and above.  B given N x K is staged 4 bytes at a time by every CTA: N <= 8 as above to
//     K = 768, N = 16 to K = 512 and 1184 rows, 1.0..3.4 beyond.  Where the tiled kernel is the faster one its sums are the
//     longer ones (8192 x 16 x 512: 2.1e-7 against 0.9e-7, 16,384 x 16 x 1433: 3.4e-7 against 1.1e-7): such products
//     stay here.
//   lanes along m: 0.67..1.1 to K = 128 (no splitting); 0.44..1.2 to 4096 rows, 1.0..1.9 above.  One tile of up to 64
//     rows: 0.44..0.95 to K = 1536, 1.0..1.25 to 8192 except for 32 rows and 8 columns at most -- the tiled kernel is also
//     the more exact one there (64 x 16 x 8192: 1.3e-7 against 2.2e-7) -- and 0.5..0.75 above.
bool narrow_supported(bool ta, int64_t M, int64_t N, int64_t K) {
  if (N > 16 || K < 16 || M > 16384) return false;
  if (!ta) return K >= 128 || (N <= 8 && M <= 32 * kNumSMs);
  if (K <= 128) return N <= 8 || K >= 64;
  if (M <= 64 && (M > 32 || N > 8) && K > 1536 && K <= 8192) return false;
  return M <= 8192;
}

size_t narrow_partial_bytes(bool ta, int64_t M, int64_t N, int64_t K) {
  if (!ta) return 0;
  const MPlan pl = m_plan(M, N, K);
  return pl.splits > 1 && !pl.cluster ? size_t(pl.splits) * size_t(M) * size_t(N) * 4 : 0;
}

int gemm_narrow(bool ta, bool tb, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B,
                int64_t ldb, float* C, int64_t ldc, const GemmEpilogue& ep, float* partial, cudaStream_t st) {
  Args p{int(M), int(N), int(K), A, lda, B, ldb, C, ldc, ep, nullptr};
  const bool wide = N > 8;
  const bool vb = !tb && ldb % 4 == 0 && aligned16(B) && N == (wide ? 16 : 8);
  if (!ta) {
    if (wide) return tb ? launch_k<16, true, false>(p, st) : vb ? launch_k<16, false, true>(p, st) : launch_k<16, false, false>(p, st);
    return tb ? launch_k<8, true, false>(p, st) : vb ? launch_k<8, false, true>(p, st) : launch_k<8, false, false>(p, st);
  }
  MPlan pl = m_plan(M, N, K);
  if (pl.splits > 1 && !pl.cluster) {
    if (partial) p.partial = partial;
    else pl.splits = 1;
  }
  int rc;
  if (wide) rc = tb ? launch_m<16, true>(p, pl, st) : launch_m<16, false>(p, pl, st);
  else rc = tb ? launch_m<8, true>(p, pl, st) : launch_m<8, false>(p, pl, st);
  if (rc != GC_OK || !p.partial) return rc;
  return splitk_reduce(int(M), int(N), pl.splits, p.partial, C, ldc, ep, st);
}

}  // namespace gc
