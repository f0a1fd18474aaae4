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
// keep two warps busy).
//
// Work is the list of all (tile, stage of k) units, tile by tile, and a CTA takes
// a contiguous run of it: whole tiles when there are many, a share of one or the
// ends of two where tiles alone would leave SMs idle or a last wave nearly empty
// (2049 x 515 has 297 tiles of 64 x 64: one more than two per SM).  Sums of tiles
// that ended up in several CTAs go to the workspace and a second kernel adds them
// in CTA order.  Every order of additions is fixed.
#include "common.cuh"
#include "gemm_internal.cuh"

namespace {

using u64 = unsigned long long;
__device__ __forceinline__ u64 pack2(float a, float b) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
// (c0, c1) += a * b, both halves (fma.rn.f32x2: the rounding of two fmaf)
__device__ __forceinline__ void fma2(float& c0, float& c1, u64 a, u64 b) {
  u64 c = pack2(c0, c1);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(c));
}
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
  int tiles_n, stages;  // tiles along N; stages of k per tile
  int64_t units;        // tiles * stages
  int per_cta;          // units of a CTA
  float* partial;       // [2 * gridDim.x][BM * BN]: the first and the last tile of a CTA, where it has only a share of it
};

template <int BM, int BN, int TM, int TN, int WK, int BK, int ST, bool TA, bool TB, bool VA, bool VB>
__global__ void __launch_bounds__(256, TM == 8 ? 2 : 3)
gemm_simt_kernel(const __grid_constant__ Args p) {
  using T = Tile<BM, BN, TM, TN, WK, BK, ST, TA, TB>;
  using SA = typename T::SA;
  using SB = typename T::SB;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x;
  // a warp covers 8 threads along M (where the tile has them) x 4 along N
  constexpr int NM = BM / TM, NN = BN / TN, GROUP = NM * NN;
  constexpr int LM = NM >= 8 ? 8 : NM, LN = 32 / LM < NN ? 32 / LM : NN, PW = LM * LN;
  const int wk = tid / GROUP, g = tid % GROUP;
  const int w = g / PW, l = g % PW;
  const int ty = (w % (NM / LM)) * LM + l % LM, tx = (w / (NM / LM)) * LN + l / LM;

  int64_t unit = int64_t(blockIdx.x) * p.per_cta;
  const int64_t last_unit = min(p.units, unit + p.per_cta);
  for (int segment = 0; unit < last_unit; ++segment) {
    const int64_t tile = unit / p.stages;
    const int kt0 = int(unit - tile * p.stages);
    const int nkt = int(min(int64_t(p.stages - kt0), last_unit - unit));
    unit += nkt;
    const int m0 = int(tile / p.tiles_n) * BM, n0 = int(tile % p.tiles_n) * BN;
    const int kb = kt0 * BK, ke = min(p.K, kb + nkt * BK);

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
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
    __syncthreads();  // the previous tile's shared memory is free
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
        if constexpr (TB) {  // pairs of columns are not neighbours in registers: packing them costs more than it saves
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
              for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i][q], b[j][q], acc[i][j]);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            u64 bb[TN / 2];
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) bb[j] = pack2(b[2 * j][q], b[2 * j + 1][q]);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
              const u64 aa = pack2(a[i][q], a[i][q]);
#pragma unroll
              for (int j = 0; j < TN / 2; ++j) fma2(acc[i][2 * j], acc[i][2 * j + 1], aa, bb[j]);
            }
          }
        }
      }
    }
    copies_wait<0>();

    // a share of a tile: raw sums to the workspace, row-major BM x BN
    float* share = nkt < p.stages ? p.partial + (2 * int64_t(blockIdx.x) + (segment ? 1 : 0)) * (BM * BN) : nullptr;
    if (WK == 1) {
      const bool vec = !TB && !p.ep.transposed && (p.ldc % 4 == 0) && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0 &&
                       !p.ep.mask && !p.ep.gate;
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int mi = SA::template index<TM>(ty, i), gm = m0 + mi;
#pragma unroll
        for (int h = 0; h < TN; h += 4) {
          float v[4] = {acc[i][h], acc[i][h + 1], acc[i][h + 2], acc[i][h + 3]};
          if (share) {
#pragma unroll
            for (int j = 0; j < 4; ++j) share[mi * BN + SB::template index<TN>(tx, h + j)] = v[j];
            continue;
          }
          if (gm >= p.M) continue;
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
            if (n < p.N) gc::epilogue_store(v[j], gm, n, p.C, p.ldc, p.ep);
          }
        }
      }
      continue;
    }

    // the sums of the WK groups, added in order
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
        sm[wk * (BM * BN) + SA::template index<TM>(ty, i) * BN + SB::template index<TN>(tx, j)] = acc[i][j];
    __syncthreads();
    for (int e = tid; e < BM * BN; e += 256) {
      float s = sm[e];
#pragma unroll
      for (int q = 1; q < WK; ++q) s += sm[q * (BM * BN) + e];
      const int gm = m0 + e / BN, gn = n0 + e % BN;
      if (share) share[e] = s;
      else if (gm < p.M && gn < p.N) gc::epilogue_store(s, gm, gn, p.C, p.ldc, p.ep);
    }
  }
}

// Adds up the shares of the tiles that several CTAs worked on.  G = 1: four elements per thread, the shares in order
// (2049 x 515: two to four per tile).  G = 8, few tiles and long sums: 32 elements per CTA, eight contiguous groups of
// shares side by side, the group sums in order.
template <int BM, int BN, int G>
__global__ void __launch_bounds__(256)
gemm_shares_kernel(const __grid_constant__ Args p) {
  constexpr int E = G == 1 ? 1024 : 32, kPerTile = (BM * BN + E - 1) / E;
  const unsigned tile = blockIdx.x / kPerTile, chunk = blockIdx.x % kPerTile;
  const unsigned long long u0 = static_cast<unsigned long long>(tile) * p.stages;
  const int c0 = int(u0 / unsigned(p.per_cta)), c1 = int((u0 + p.stages - 1) / unsigned(p.per_cta));
  if (c0 == c1) return;  // one CTA had all of it
  const int m0 = int(tile / unsigned(p.tiles_n)) * BM, n0 = int(tile % unsigned(p.tiles_n)) * BN;
  // only the first contributor can have begun with an earlier tile; every later one began with this tile
  const bool first0 = static_cast<unsigned long long>(c0) * p.per_cta == u0;
  if constexpr (G == 1) {
    const int e = int(chunk) * E + int(threadIdx.x) * 4;
    if (e >= BM * BN) return;
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m >= p.M || n >= p.N) return;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c = c0; c <= c1; ++c) {
      const int slot = (c > c0 || first0) ? 0 : 1;
      const float4 v = __ldg(reinterpret_cast<const float4*>(p.partial + (2 * int64_t(c) + slot) * (BM * BN) + e));
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < p.N) gc::epilogue_store(v[j], m, n + j, p.C, p.ldc, p.ep);
  } else {
    __shared__ float sm[G][32];
    const int lane = threadIdx.x % 32, g = threadIdx.x / 32, e = int(chunk) * E + lane;
    const int per = (c1 - c0 + G) / G;
    float s = 0.f;
    for (int c = c0 + g * per; c <= min(c1, c0 + (g + 1) * per - 1); ++c)
      s += __ldg(p.partial + (2 * int64_t(c) + ((c > c0 || first0) ? 0 : 1)) * (BM * BN) + e);
    sm[g][lane] = s;
    __syncthreads();
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (g > 0 || m >= p.M || n >= p.N) return;
#pragma unroll
    for (int k = 1; k < G; ++k) s += sm[k][lane];
    gc::epilogue_store(s, m, n, p.C, p.ldc, p.ep);
  }
}

// ------------------------------------------------------------------ host
struct Shape {
  int bm, bn, bk;
  int resident;  // CTAs per SM (registers and shared memory)
  double rate;   // FMA rate of a full SM relative to the largest tile's
};
// Narrow tiles by the width of the output; 64 x 64 and 128 x 128 for the rest (4096 x 4096 x 1024: 41.8 and 52.0 TFLOP/s).
// 65,536 rows of K = 256 on the narrow ones: 8 columns 13.1, 16 21.3, 32 27.4 TFLOP/s; their rates only weigh whole tiles
// against shares.
constexpr Shape kShapes[] = {{64, 8, 64, 3, 0.3}, {64, 16, 64, 3, 0.5}, {64, 32, 32, 3, 0.7}, {64, 64, 32, 3, 0.8}, {128, 128, 32, 2, 1.0}};

struct Choice {
  int shape;
  int64_t tiles, stages, per_cta, ctas;
  bool shared() const { return per_cta % stages != 0; }
};

// Against all four of the choices for more than 32 columns (both tiles, whole or shared) at 239 sizes of 16 to 300 K rows,
// 17 to 6000 columns and K from 16 to 200 K: 3.8 % slower than the best of them on average, more than 5 % in 58 and more
// than 10 % in 32.  The worst are shares of large tiles where smaller shares (1576 x 80 x 1936 45.8 us against 32.7) or
// whole tiles (K near 100 and many rows: 119,390 x 80 x 102 130 against 98) would do; whole tiles sum in longer chains.
Choice choose(int64_t M, int64_t N, int64_t K) {
  using gc::ceil_div;
  Choice best{};
  double least = -1;
  const int lo = N <= 8 ? 0 : N <= 16 ? 1 : N <= 32 ? 2 : 3, hi = N <= 32 ? lo : 4;
  for (int s = lo; s <= hi; ++s) {
    const Shape& sh = kShapes[s];
    Choice c{};
    c.shape = s;
    c.tiles = ceil_div(M, sh.bm) * ceil_div(N, sh.bn);
    c.stages = std::max<int64_t>(1, ceil_div(K, sh.bk));
    const int64_t slots = int64_t(gc::kNumSMs) * sh.resident, units = c.tiles * c.stages;
    const double unit = double(sh.bm) * sh.bn * sh.bk / 128.0 / sh.rate;  // clocks of an SM
    // whole tiles: as long as the SM that gets the most of them
    c.per_cta = c.stages;
    c.ctas = c.tiles;
    double t = double(ceil_div(c.tiles, gc::kNumSMs)) * c.stages * unit + 1000.0;
    // or equal shares, at least 64 k-values each, plus a second kernel (4 to 7 us)
    const int64_t share = std::max<int64_t>(ceil_div(units, slots), std::min<int64_t>(c.stages, std::max(1, 64 / sh.bk)));
    const double shared_t = double(ceil_div(ceil_div(units, share), gc::kNumSMs)) * share * unit + 9000.0;
    if (c.stages > 1 && share != c.stages && shared_t < t) {
      c.per_cta = share;
      c.ctas = ceil_div(units, share);
      t = shared_t;
    }
    if (least < 0 || t < least) {
      least = t;
      best = c;
    }
  }
  return best;
}

template <int BM, int BN, int TM, int TN, int WK, int BK, int ST, bool TA, bool TB, bool VA, bool VB>
int launch_one(const Args& p, unsigned ctas, cudaStream_t st) {
  using T = Tile<BM, BN, TM, TN, WK, BK, ST, TA, TB>;
  auto kern = gemm_simt_kernel<BM, BN, TM, TN, WK, BK, ST, TA, TB, VA, VB>;
  if (T::kBytes > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kBytes);
    if (e != cudaSuccess) return gc::fail(GC_ERR_CUDA, "gemm_simt: %s", cudaGetErrorString(e));
  }
  kern<<<ctas, 256, T::kBytes, st>>>(p);
  return gc::check_launch("gemm_simt");
}

// A tile shape in the four layouts; aligned rows on both operands or on neither (one variant each).
template <int BM, int BN, int TM, int TN, int WK, int BK, int ST>
int launch(bool ta, bool tb, bool vec, const Args& p, const Choice& c, cudaStream_t st) {
  const unsigned n = unsigned(c.ctas);
  int rc;
#define GC_L(TA_, TB_)                                                                           \
  (vec ? launch_one<BM, BN, TM, TN, WK, BK, ST, TA_, TB_, true, true>(p, n, st)                  \
       : launch_one<BM, BN, TM, TN, WK, BK, ST, TA_, TB_, false, false>(p, n, st))
  if (!ta && !tb) rc = GC_L(false, false);
  else if (!ta) rc = GC_L(false, true);
  else if (!tb) rc = GC_L(true, false);
  else rc = GC_L(true, true);
#undef GC_L
  if (rc != GC_OK || !p.partial) return rc;
  if (c.stages > 16 * c.per_cta) gemm_shares_kernel<BM, BN, 8><<<unsigned(c.tiles * (BM * BN / 32)), 256, 0, st>>>(p);
  else gemm_shares_kernel<BM, BN, 1><<<unsigned(c.tiles * ((BM * BN + 1023) / 1024)), 256, 0, st>>>(p);
  return gc::check_launch("gemm_simt (shares)");
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
  return c.shared() ? kFlagBytes + size_t(2 * c.ctas) * kShapes[c.shape].bm * kShapes[c.shape].bn * sizeof(float) : 0;
}

int gemm_simt(bool ta, bool tb, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B,
              int64_t ldb, float* C, int64_t ldc, const GemmEpilogue& ep, void* workspace, size_t workspace_bytes,
              cudaStream_t st) {
  const size_t need = simt_workspace_bytes(ta, M, N, K);
  float* shares = need && workspace && workspace_bytes >= need
                      ? reinterpret_cast<float*>(static_cast<char*>(workspace) + kFlagBytes)
                      : nullptr;
  if (narrow_supported(ta, M, N, K)) return gemm_narrow(ta, tb, M, N, K, A, lda, B, ldb, C, ldc, ep, shares, st);
  Choice c = choose(M, N, K);
  if (c.shared() && !shares) {  // no workspace: whole tiles
    c.per_cta = c.stages;
    c.ctas = c.tiles;
  }
  if (c.ctas > INT32_MAX || c.tiles * (kShapes[c.shape].bm * kShapes[c.shape].bn / 32) > INT32_MAX)
    return fail(GC_ERR_UNSUPPORTED, "gemm_simt: too many tiles for one launch");
  const Args p{int(M), int(N), int(K), A, lda, B, ldb, C, ldc, ep, int(ceil_div(N, kShapes[c.shape].bn)), int(c.stages),
               c.tiles * c.stages, int(c.per_cta), c.shared() ? shares : nullptr};
  const bool vec = lda % 4 == 0 && aligned16(A) && ldb % 4 == 0 && aligned16(B);
  switch (c.shape) {
    case 0: return launch<64, 8, 4, 4, 8, 64, 3>(ta, tb, vec, p, c, st);
    case 1: return launch<64, 16, 4, 4, 4, 64, 3>(ta, tb, vec, p, c, st);
    case 2: return launch<64, 32, 4, 4, 2, 32, 3>(ta, tb, vec, p, c, st);
    case 3: return launch<64, 64, 4, 4, 1, 32, 3>(ta, tb, vec, p, c, st);
    default: return launch<128, 128, 8, 8, 1, 32, 3>(ta, tb, vec, p, c, st);
  }
}

}  // namespace gc
