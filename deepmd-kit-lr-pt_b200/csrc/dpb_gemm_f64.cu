// FP64 GEMM for the fitting network of the FP64 plain path (and the FP64
// training step), and its FP32 counterpart for the shapes the tensor-core
// GEMM does not take (N not a multiple of 80): C[M, N] = op(A) op(B) (+ bias[N])
// (+ C), row-major, with
// op(X) = X or X^T. The fitting layers are y = x W + b (forward, W [in, out]
// as stored), g_in = g W^T (input gradient) and gW += x^T g (weight
// gradient), the layer algebra of deepmd/dpmodel/utils/network.py:282-330.
// Any M, N, K and leading dimensions are accepted (edges are zero-filled).
//
// FP64: k_gemm_dmma, 64 x 80 tiles on the FP64 matrix instructions. FP32:
// k_gemm_small / k_gemm_big below on the FMA pipe.
#include <cooperative_groups.h>

#include <algorithm>

#include "dpb_common.cuh"

namespace dpb {
namespace {

constexpr int GB_M = 64, GB_N = 64, GB_K = 16, GB_T = 256;

// ------------------------------------------------- FP64 matrix instructions --
// mma.m16n8k4 runs at the rate of the FP64 FMA pipe (64 FMA per clock and SM,
// measured 18.5 T FMA/s against 17.2), but a warp tile of 32 x 40 reads 9
// operands per lane from shared memory for 80 FMAs, where the FMA form
// read 12 for 32 and stood at 5-6 T FMA/s, its shared-memory reads and its
// few CTAs the limit.
//
// CTA: 64 x 80 of C (three tiles cover the fitting width 240), 8 warps as 2 x 2
// warp tiles of 32 x 40 times two halves of every 16-wide k block; operands by
// 8-byte cp.async (any alignment, zero fill at the edges) through a ring of
// three stages, stored as they lie in memory with row strides of 4 modulo 16
// doubles, which makes every fragment read conflict-free. Few tiles (small
// M): a cluster of Z CTAs shares the tile's K range and adds the Z partial
// tiles through distributed shared memory in rank order, so the result does
// not depend on scheduling and no workspace is needed. Measured, the fitting
// GEMMs of one step: 3,993 atoms 1.63 -> 0.52 ms, a training step of 768 atoms
// (two streams) 4.0 -> 1.15 ms of kernel time.
constexpr int GD_M = 64, GD_N = 80, GD_K = 16, GD_ST = 3, GD_T = 256;
constexpr int GD_SK = GD_K + 4;                        // row stride of [m][k] / [n][k]
constexpr int GD_SM = GD_M + 4, GD_SN = GD_N + 4;      // of [k][m], [k][n]
constexpr int GD_AS = GD_M * GD_SK, GD_BS = GD_N * GD_SK;  // doubles per stage
static_assert(GD_K * GD_SM <= GD_AS && GD_K * GD_SN <= GD_BS, "stage sizes");
constexpr int GD_CS = GD_N + 2;                        // stride of the partial tile
constexpr int GD_SMEM = 8 * GD_ST * (GD_AS + GD_BS);
static_assert(GD_M * GD_CS <= GD_ST * (GD_AS + GD_BS), "the partial tile reuses the ring");

__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0)
               : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
      "{%0, %1, %2, %3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}

template <bool TA, bool TB>
__global__ void __launch_bounds__(GD_T, 2)
k_gemm_dmma(double* __restrict__ C, const double* __restrict__ A, const double* __restrict__ B,
            const double* __restrict__ bias, int M, int N, int K, int lda, int ldb, int ldc,
            int accumulate, int kchunk) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) double gsm[];
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int ntn = (N + GD_N - 1) / GD_N;  // tiles in one grid dimension: the others end at 65,535
  const int m0 = (int)(blockIdx.x / ntn) * GD_M, n0 = (int)(blockIdx.x % ntn) * GD_N;
  const int z = blockIdx.z, Z = gridDim.z;
  const int k0 = z * kchunk, k1 = min(K, k0 + kchunk);
  const int nk = k1 > k0 ? (k1 - k0 + GD_K - 1) / GD_K : 0;
  auto stage = [&](int b) { return gsm + (size_t)(b % GD_ST) * (GD_AS + GD_BS); };
  auto fetch = [&](int b) {
    double* sa = stage(b);
    double* sb = sa + GD_AS;
    const int kb = k0 + b * GD_K;
#pragma unroll
    for (int j = 0; j < GD_M * GD_K / GD_T; ++j) {
      const int q = tid + GD_T * j;
      const int m = TA ? q % GD_M : q / GD_K, k = TA ? q / GD_M : q % GD_K;
      const bool ok = m0 + m < M && kb + k < k1;
      const double* src = TA ? A + (size_t)(kb + k) * lda + m0 + m
                             : A + (size_t)(m0 + m) * lda + kb + k;
      cp_async8(sa + (TA ? k * GD_SM + m : m * GD_SK + k), ok ? src : A, ok);
    }
#pragma unroll
    for (int j = 0; j < GD_N * GD_K / GD_T; ++j) {
      const int q = tid + GD_T * j;
      const int n = TB ? q / GD_K : q % GD_N, k = TB ? q % GD_K : q / GD_N;
      const bool ok = n0 + n < N && kb + k < k1;
      const double* src = TB ? B + (size_t)(n0 + n) * ldb + kb + k
                             : B + (size_t)(kb + k) * ldb + n0 + n;
      cp_async8(sb + (TB ? n * GD_SK + k : k * GD_SN + n), ok ? src : B, ok);
    }
  };
  const int wm = (warp & 1) * 32, wn = ((warp >> 1) & 1) * 40, kg = (warp >> 2) * (GD_K / 2);
  double acc[2][5][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 5; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.;
#pragma unroll
  for (int b = 0; b < GD_ST - 1; ++b) {
    if (b < nk) fetch(b);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int b = 0; b < nk; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(GD_ST - 2) : "memory");
    __syncthreads();  // block b is here, and every warp is done with block b - 1
    if (b + GD_ST - 1 < nk) fetch(b + GD_ST - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double* sa = stage(b);
    const double* sb = sa + GD_AS;
#pragma unroll
    for (int ks = 0; ks < GD_K / 2; ks += 4) {
      const int k = kg + ks + t4;
      double a[2][2], bv[5];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m = wm + i * 16 + h * 8 + g;
          a[i][h] = TA ? sa[k * GD_SM + m] : sa[m * GD_SK + k];
        }
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const int n = wn + j * 8 + g;
        bv[j] = TB ? sb[n * GD_SK + k] : sb[k * GD_SN + n];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 5; ++j) dmma(acc[i][j], a[i][0], a[i][1], bv[j]);
    }
  }
  pdl_trigger();
  // the tile's sum over the two k halves, then over the cluster
  __syncthreads();
  double* part = gsm;
  auto at = [&](int i, int j, int c) {
    return part + (wm + i * 16 + (c >> 1) * 8 + g) * GD_CS + wn + j * 8 + 2 * t4 + (c & 1);
  };
  if (kg)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) *at(i, j, c) = acc[i][j][c];
  __syncthreads();
  if (!kg)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 5; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) *at(i, j, c) += acc[i][j][c];
  auto cluster = cg::this_cluster();
  if (Z > 1)
    cluster.sync();
  else
    __syncthreads();
  const int rows = (GD_M + Z - 1) / Z;
  for (int q = tid; q < rows * GD_N; q += GD_T) {
    const int rl = z * rows + q / GD_N, c = q % GD_N;
    if (rl >= GD_M || m0 + rl >= M || n0 + c >= N) continue;
    double v = 0.;
    for (int p = 0; p < Z; ++p)
      v += (Z > 1 ? cluster.map_shared_rank(part, p) : part)[rl * GD_CS + c];
    if (bias) v += bias[n0 + c];
    double* dst = C + (size_t)(m0 + rl) * ldc + n0 + c;
    if (accumulate) v += *dst;
    *dst = v;
  }
  if (Z > 1) cluster.sync();  // the partial tiles stay until everyone has read them
}

// element (r, c) of op(X) for an [rows, cols] operand with leading dim ld
template <bool TRANS, typename T>
__device__ __forceinline__ T ld_op(const T* __restrict__ X, int r, int c, int rows, int cols,
                                   int ld) {
  if (r >= rows || c >= cols) return (T)0;
  return TRANS ? X[(size_t)c * ld + r] : X[(size_t)r * ld + c];
}

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };

template <bool TA, bool TB, typename T>
__global__ void __launch_bounds__(GB_T)
k_gemm_small(T* __restrict__ C, const T* __restrict__ A, const T* __restrict__ B,
           const T* __restrict__ bias, int M, int N, int K, int lda, int ldb, int ldc,
           int accumulate) {
  using T2 = typename Vec2<T>::type;
  __shared__ __align__(16) T As[2][GB_K][GB_M + 2];
  __shared__ __align__(16) T Bs[2][GB_K][GB_N + 2];
  pdl_wait();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * GB_M, n0 = blockIdx.x * GB_N;
  const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, 4 x 4 outputs each
  // staging assignment: 64 x 16 = 1024 elements per operand, 4 per thread.
  // A (op(A) is M x K): element q = tid + 256 j -> (row, k); for a plain A
  // consecutive threads walk k (contiguous in memory), for A^T they walk m.
  T ra[4], rb[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = tid + GB_T * j;
      int r, k;
      if (TA) { r = q & 63; k = q >> 6; } else { k = q & 15; r = q >> 4; }
      ra[j] = TA ? ld_op<true, T>(A, m0 + r, k0 + k, M, K, lda)
                 : ld_op<false, T>(A, m0 + r, k0 + k, M, K, lda);
      int c, kk;
      if (TB) { kk = q & 15; c = q >> 4; } else { c = q & 63; kk = q >> 6; }
      rb[j] = TB ? ld_op<true, T>(B, k0 + kk, n0 + c, K, N, ldb)
                 : ld_op<false, T>(B, k0 + kk, n0 + c, K, N, ldb);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = tid + GB_T * j;
      int r, k;
      if (TA) { r = q & 63; k = q >> 6; } else { k = q & 15; r = q >> 4; }
      As[buf][k][r] = ra[j];
      int c, kk;
      if (TB) { kk = q & 15; c = q >> 4; } else { c = q & 63; kk = q >> 6; }
      Bs[buf][kk][c] = rb[j];
    }
  };
  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = (T)0;
  const int nk = (K + GB_K - 1) / GB_K;
  fetch(0);
  stash(0);
  __syncthreads();
  for (int t = 0; t < nk; ++t) {
    const int buf = t & 1;
    if (t + 1 < nk) fetch((t + 1) * GB_K);
#pragma unroll
    for (int k = 0; k < GB_K; ++k) {
      const T2 a01 = *reinterpret_cast<const T2*>(&As[buf][k][ty * 4]);
      const T2 a23 = *reinterpret_cast<const T2*>(&As[buf][k][ty * 4 + 2]);
      const T2 b01 = *reinterpret_cast<const T2*>(&Bs[buf][k][tx * 4]);
      const T2 b23 = *reinterpret_cast<const T2*>(&Bs[buf][k][tx * 4 + 2]);
      const T a[4] = {a01.x, a01.y, a23.x, a23.y};
      const T b[4] = {b01.x, b01.y, b23.x, b23.y};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    if (t + 1 < nk) {
      stash(buf ^ 1);
      __syncthreads();
    }
  }
  pdl_trigger();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = m0 + ty * 4 + i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tx * 4 + j;
      if (c >= N) continue;
      T v = acc[i][j];
      if (bias) v += bias[c];
      T* p = C + (size_t)r * ldc + c;
      if (accumulate) v += *p;
      *p = v;
    }
  }
}

// The large-M form: 128 x 64 tiles, K in steps of 8, each thread a block of
// 8 rows (ty * 4 + i and 64 + ty * 4 + i) by 4 columns, so every k step
// reads 6 shared-memory vectors for 32 FMAs (the 64 x 64 form above: 4 for
// 16).
constexpr int GL_M = 128, GL_N = 64, GL_K = 8;

template <bool TA, bool TB, typename T>
__global__ void __launch_bounds__(GB_T)
k_gemm_big(T* __restrict__ C, const T* __restrict__ A, const T* __restrict__ B,
           const T* __restrict__ bias, int M, int N, int K, int lda, int ldb, int ldc,
           int accumulate) {
  using T2 = typename Vec2<T>::type;
  __shared__ __align__(16) T As[2][GL_K][GL_M + 2];
  __shared__ __align__(16) T Bs[2][GL_K][GL_N + 2];
  pdl_wait();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * GL_M, n0 = blockIdx.x * GL_N;
  const int tx = tid & 15, ty = tid >> 4;
  T ra[4], rb[2];
  auto a_at = [&](int q, int& r, int& k) {
    if (TA) { r = q & 127; k = q >> 7; } else { k = q & 7; r = q >> 3; }
  };
  auto b_at = [&](int q, int& c, int& k) {
    if (TB) { k = q & 7; c = q >> 3; } else { c = q & 63; k = q >> 6; }
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int r, k;
      a_at(tid + GB_T * j, r, k);
      ra[j] = ld_op<TA, T>(A, m0 + r, k0 + k, M, K, lda);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      int c, k;
      b_at(tid + GB_T * j, c, k);
      rb[j] = ld_op<TB, T>(B, k0 + k, n0 + c, K, N, ldb);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int r, k;
      a_at(tid + GB_T * j, r, k);
      As[buf][k][r] = ra[j];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      int c, k;
      b_at(tid + GB_T * j, c, k);
      Bs[buf][k][c] = rb[j];
    }
  };
  T acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = (T)0;
  const int nk = (K + GL_K - 1) / GL_K;
  fetch(0);
  stash(0);
  __syncthreads();
  for (int t = 0; t < nk; ++t) {
    const int buf = t & 1;
    if (t + 1 < nk) fetch((t + 1) * GL_K);
#pragma unroll
    for (int k = 0; k < GL_K; ++k) {
      const T2 a0 = *reinterpret_cast<const T2*>(&As[buf][k][ty * 4]);
      const T2 a1 = *reinterpret_cast<const T2*>(&As[buf][k][ty * 4 + 2]);
      const T2 a2 = *reinterpret_cast<const T2*>(&As[buf][k][64 + ty * 4]);
      const T2 a3 = *reinterpret_cast<const T2*>(&As[buf][k][64 + ty * 4 + 2]);
      const T2 b0 = *reinterpret_cast<const T2*>(&Bs[buf][k][tx * 4]);
      const T2 b1 = *reinterpret_cast<const T2*>(&Bs[buf][k][tx * 4 + 2]);
      const T a[8] = {a0.x, a0.y, a1.x, a1.y, a2.x, a2.y, a3.x, a3.y};
      const T b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    if (t + 1 < nk) {
      stash(buf ^ 1);
      __syncthreads();
    }
  }
  pdl_trigger();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tx * 4 + j;
      if (c >= N) continue;
      T v = acc[i][j];
      if (bias) v += bias[c];
      T* p = C + (size_t)r * ldc + c;
      if (accumulate) v += *p;
      *p = v;
    }
  }
}

}  // namespace
}  // namespace dpb

using namespace dpb;

namespace {

// checks shared by the two precisions; 1 when there is nothing to do
template <typename T>
int gemm_args(const char* what, const T* C, const T* A, const T* B, int M, int N, int K, int lda,
              int ldb, int ldc, int trans_a, int trans_b) {
  if (M < 0 || N < 0 || K < 0 || (M > 0 && N > 0 && (!C || (K > 0 && (!A || !B))))) {
    set_error("%s: invalid arguments (M=%d N=%d K=%d)", what, M, N, K);
    return DPB_ERR_INVALID;
  }
  const int a_cols = trans_a ? M : K, b_cols = trans_b ? K : N;
  if (ldc < N || lda < a_cols || ldb < b_cols) {
    set_error("%s: leading dimensions too small (lda=%d ldb=%d ldc=%d)", what, lda, ldb, ldc);
    return DPB_ERR_INVALID;
  }
  return DPB_OK;
}

int grid_rows(const char* what, int M, int tile) {
  const int y = (M + tile - 1) / tile;
  if (y > 65535) {
    set_error("%s: M=%d needs more than 65535 row tiles", what, M);
    return -1;
  }
  return y;
}

}  // namespace

extern "C" int dpb_gemm_f64(double* C, const double* A, const double* B, const double* bias,
                            int M, int N, int K, int lda, int ldb, int ldc, int trans_a,
                            int trans_b, int accumulate, dpb_stream_t stream) {
  const int rc = gemm_args("gemm_f64", C, A, B, M, N, K, lda, ldb, ldc, trans_a, trans_b);
  if (rc || M == 0 || N == 0) return rc;
  if (grid_rows("gemm_f64", M, GL_M) < 0) return DPB_ERR_INVALID;
  const long long tiles = (long long)((M + GD_M - 1) / GD_M) * ((N + GD_N - 1) / GD_N);
  if (tiles > 0x7fffffff) {
    set_error("gemm_f64: M=%d N=%d need more than 2^31 - 1 tiles", M, N);
    return DPB_ERR_INVALID;
  }
  // K split over a cluster while the tiles leave SMs idle and each share keeps
  // four k blocks
  int Z = 1;
  while (Z < 8 && tiles * Z * 2 <= 2 * sm_count() && K >= 2 * Z * 4 * GD_K) Z *= 2;
  int kchunk = ((K + Z - 1) / Z + GD_K - 1) / GD_K * GD_K;
  if (kchunk == 0) kchunk = GD_K;
  auto run = [&](auto kern) -> int {
    DPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GD_SMEM),
             "gemm_f64");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles, 1, Z);
    cfg.blockDim = dim3(GD_T);
    cfg.dynamicSmemBytes = GD_SMEM;
    cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (Z > 1) {
      attr[n].id = cudaLaunchAttributeClusterDimension;
      attr[n].val.clusterDim.x = 1;
      attr[n].val.clusterDim.y = 1;
      attr[n].val.clusterDim.z = Z;
      ++n;
    }
    if (tune_value("pdl", 1) != 0) {
      attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[n].val.programmaticStreamSerializationAllowed = 1;
      ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    DPB_CUDA(cudaLaunchKernelEx(&cfg, kern, C, A, B, bias, M, N, K, lda, ldb, ldc, accumulate,
                                kchunk),
             "gemm_f64");
    return DPB_OK;
  };
  if (trans_a) return trans_b ? run(k_gemm_dmma<true, true>) : run(k_gemm_dmma<true, false>);
  return trans_b ? run(k_gemm_dmma<false, true>) : run(k_gemm_dmma<false, false>);
}

extern "C" int dpb_gemm_f32(float* C, const float* A, const float* B, const float* bias, int M,
                            int N, int K, int lda, int ldb, int ldc, int trans_a, int trans_b,
                            int accumulate, dpb_stream_t stream) {
  const int rc = gemm_args("gemm_f32", C, A, B, M, N, K, lda, ldb, ldc, trans_a, trans_b);
  if (rc || M == 0 || N == 0) return rc;
  const bool big = M >= GL_M && tune_value("gemm_simt_big", 1);
  const int gy = grid_rows("gemm_f32", M, big ? GL_M : GB_M);
  if (gy < 0) return DPB_ERR_INVALID;
  const dim3 grid((N + GB_N - 1) / GB_N, gy);
  auto run = [&](auto kern) -> int {
    DPB_CUDA(launch_pdl(kern, grid, dim3(GB_T), 0, as_stream(stream), C, A, B, bias, M, N, K, lda,
                        ldb, ldc, accumulate),
             "gemm_f32");
    return DPB_OK;
  };
  if (big) {
    if (trans_a)
      return trans_b ? run(k_gemm_big<true, true, float>) : run(k_gemm_big<true, false, float>);
    return trans_b ? run(k_gemm_big<false, true, float>) : run(k_gemm_big<false, false, float>);
  }
  if (trans_a)
    return trans_b ? run(k_gemm_small<true, true, float>) : run(k_gemm_small<true, false, float>);
  return trans_b ? run(k_gemm_small<false, true, float>) : run(k_gemm_small<false, false, float>);
}

// out[c * ld_out + r] = in[r * ld_in + c] for r < rows, c < cols, and zero for
// rows <= r < out_rows (a K padded to a multiple of 4 for the tensor-core
// GEMM's 16-byte rows, or one block of a concatenation along K)
__global__ void k_transpose_f32(float* __restrict__ out, const float* __restrict__ in, int rows,
                                int cols, int ld_in, int ld_out, int out_rows) {
  __shared__ float tile[32][33];
  pdl_wait();
  pdl_trigger();
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int r = r0 + k, c = c0 + threadIdx.x;
    tile[k][threadIdx.x] = (r < rows && c < cols) ? in[(size_t)r * ld_in + c] : 0.f;
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int c = c0 + k, r = r0 + threadIdx.x;
    if (c < cols && r < out_rows) out[(size_t)c * ld_out + r] = tile[threadIdx.x][k];
  }
}

extern "C" int dpb_transpose_f32(float* out, const float* in, int rows, int cols, int ld_in,
                                 int ld_out, int out_rows, dpb_stream_t stream) {
  if (rows < 0 || cols < 0 || out_rows < rows || ld_out < out_rows || ld_in < cols ||
      (out_rows > 0 && cols > 0 && (!out || (rows > 0 && !in)))) {
    set_error("transpose_f32: invalid arguments (rows=%d cols=%d ld_in=%d ld_out=%d "
              "out_rows=%d)", rows, cols, ld_in, ld_out, out_rows);
    return DPB_ERR_INVALID;
  }
  if (cols == 0 || out_rows == 0) return DPB_OK;
  const dim3 grid((cols + 31) / 32, (out_rows + 31) / 32);
  DPB_CUDA(launch_pdl(k_transpose_f32, grid, dim3(32, 8), 0, as_stream(stream), out, in, rows,
                      cols, ld_in, ld_out, out_rows),
           "transpose_f32");
  return DPB_OK;
}
