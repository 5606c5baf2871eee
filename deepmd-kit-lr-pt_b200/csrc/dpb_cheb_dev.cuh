// Device side of the descriptor passes on piecewise Chebyshev embeddings
// (dpb_se_a.cu): cheb_fwd_group / cheb_bwd_group, eight center atoms by eight
// warps. Used by the descriptor kernels and by the batched-frames step kernel.
//
// Over [lo, hi) of its table an embedding net is G(x)[m] = sum_k T_k(t) C[r][k][m]
// on interval r (t = (x - center_r) / halfwidth_r in [-1, 1), 16 polynomials),
// fitted to the table by the host. The sum over an atom's neighbor slots then
// separates from the channels:
//   xyz[d][m] = sum_r sum_k W[d][r, k] C[r][k][m],  W[d][r, k] = sum_{s in r} e_s[d] T_k(t_s)
// and, backward, with Z[d][r, k] = sum_m dxyz[d][m] C[r][k][m],
//   net_deriv_s[d] = sum_k T_k(t_s) Z[d][r, k]  (+ the slope's term for d = 0),
// so a slot costs 16 polynomials times 4 env columns instead of a gathered
// table row times every channel, and the channels become matrix products:
// [32 rows = 8 atoms x 4 env columns] x [16 k per touched interval] x [M]. 32
// rows are a quarter of a tcgen05 tile, and the K of the product is the set of
// intervals these atoms touch, so the products are warp-level MMAs
// (m16n8k16), the channel tiles spread over the warps.
//
// What bounds the passes: with one warp per four atoms (the same products,
// no barriers) they waited on loads, 0.26 issue per cycle; a warp per atom
// with the tiles shared keeps 24-32 warps per SM busy.
//
// FP32 operands are split into two FP16 terms, hi + lo, after scaling by a
// power of two (per atom and type from a bound of the row; per net for C), so
// that hi + lo holds 23 bits of every value down to 2^-16 of the largest and
// 2^-39 of the largest below that (dpb_f16split.cuh); the product is lo hi + hi lo + hi hi accumulated in FP32 from
// zero for each interval (16 k), and the intervals are added in FP32 outside
// the tensor cores, whose own accumulation truncates.
//
// Slots outside [lo, hi) (a pair closer than any in the model's statistics,
// the linear tails) are added from the table, a warp per slot.
#pragma once

#include "dpb_desc_dev.cuh"
#include "dpb_f16split.cuh"

namespace dpb {

constexpr int CHEB_K = 16;      // polynomials per interval (one MMA k step)
constexpr int CHEB_A = 8;       // atoms (and warps) per group: 32 MMA rows
constexpr int CHEB_MAXR = 16;   // intervals per net
constexpr int CHEB_TS = 20;     // staged polynomials of a slot: row stride (16-byte
                                // stores and the 16-lane reads both conflict-free)

struct ChebNet {
  const uint4* fw;            // [R][ceil(M / 8)][32 lanes]: B fragments of C (k x channels)
  const uint4* bw;            // [R][2][ceil(M / 16)][32]: B fragments of C^T (channels x k)
  const float2* iv;           // [R]: center, 1 / halfwidth
  const unsigned char* lut;   // interval of each cell of [lo, hi)
  float lo, hi, inv_cell, inv_scale;
  int ncell, R;
};

struct ChebTables {
  ChebNet net[PMAXT];
  int wstride;  // row stride of W: 16 R of the largest net + 8 (8 or 24 modulo 32:
                // the 8-byte reads of four rows and the two halves' adds are
                // conflict-free)
  int rmax;
};

__device__ __forceinline__ void mma_f16(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                        unsigned b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, "
      "{%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]),
        "f"(c[2]), "f"(c[3]));
}

// A B of one k step from the split operands, b = (hi k 0..7, hi k 8..15, lo, lo)
__device__ __forceinline__ void mma_split(float (&d)[4], const unsigned (&ah)[4],
                                          const unsigned (&al)[4], const uint4 b) {
  const float zero[4] = {0.f, 0.f, 0.f, 0.f};
  mma_f16(d, al, b.x, b.y, zero);
  mma_f16(d, ah, b.z, b.w, d);
  mma_f16(d, ah, b.x, b.y, d);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// one chunk of 32 slots of a type block: the lane's env row, how many slots
// of the chunk count (up to the fold slot, whose multiplicity goes to rep)
struct ChebSlots {
  float4 e;
  int n;        // slots [q0, q0 + n) count
  bool folded;  // the fold slot is the last of them
  float rep;    // this lane's multiplicity
};

template <bool COH>
__device__ __forceinline__ ChebSlots cheb_slots(const float4* erow, int q0, int nt, float last,
                                                int lane) {
  ChebSlots c;
  const int q = q0 + lane;
  c.e = q < nt ? (COH ? ld_cg4(erow + q) : ld_stream4(erow + q, l2_policy_first()))
               : make_float4(0.f, 0.f, 0.f, 0.f);
  const bool f = q < nt && c.e.x == last && c.e.y == 0.f && c.e.z == 0.f && c.e.w == 0.f;
  const unsigned b = __ballot_sync(0xffffffffu, f);
  c.n = min(32, nt - q0);
  c.folded = b != 0u;
  c.rep = 1.f;
  if (b) {
    const int s = __ffs(b) - 1;
    c.n = s + 1;
    if (lane == s) c.rep = (float)(nt - q0 - s);
  }
  return c;
}

// value of the last slot's first column (the fold test's reference)
template <bool COH>
__device__ __forceinline__ float cheb_last(const float4* erow, int nt) {
  return COH ? ld_cg4(erow + nt - 1).x : __ldg(&erow[nt - 1].x);
}

__device__ __forceinline__ bool cheb_locate(const ChebNet& c, float x, int& r, float& t,
                                            float& ih) {
  if (!(x >= c.lo && x < c.hi)) return false;
  const int cell = min((int)((x - c.lo) * c.inv_cell), c.ncell - 1);
  r = c.lut[cell];
  const float2 v = __ldg(c.iv + r);
  t = (x - v.x) * v.y;
  ih = v.y;
  return true;
}

// power of two that brings a descriptor row below 2^14, from its atom's x
// [4][M]: |D[m, a]| <= max_m sum_d x[d, m]^2
__device__ __forceinline__ float descriptor_scale(const float* x, int M, int lane) {
  float mx = 0.f;
  for (int m = lane; m < M; m += 32)
    mx = fmaxf(mx, x[m] * x[m] + x[M + m] * x[M + m] + x[2 * M + m] * x[2 * M + m] +
                       x[3 * M + m] * x[3 * M + m]);
  float inv;
  return f16_scale(warp_max(mx), inv);
}

// floats of shared memory per group of CHEB_A warps
static size_t cheb_fwd_floats(int M, int wstride) {
  const size_t w = (size_t)CHEB_A * 4 * wstride, x = (size_t)CHEB_A * 4 * M;
  return (w > x ? w : x) + 2 * CHEB_A + CHEB_A * (32 * CHEB_TS + 32 * 4);
}
static size_t cheb_bwd_floats(int M, int naxis, int rmax) {
  const size_t z = (size_t)CHEB_A * rmax * CHEB_K * 4;
  const size_t p = CHEB_A * ((size_t)4 * M + 4 * MAXAX + (size_t)M * naxis);
  return (z > p ? z : p) + 2 * CHEB_A + CHEB_A * 4 * ((size_t)(M + 15) / 16 * 16 + 8);
}

// barrier of the CHEB_A warps of a group
__device__ __forceinline__ void cheb_sync(int bar) {
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(32 * CHEB_A) : "memory");
}

// A fragments (rows g, g + 8 of 16; k pairs t4, t4 + 4) from rows of
// interleaved (hi pair, lo pair) words
__device__ __forceinline__ void frag_a(unsigned (&h)[4], unsigned (&l)[4], const float* p,
                                       int row8) {
  const uint2 v0 = *reinterpret_cast<const uint2*>(p);
  const uint2 v1 = *reinterpret_cast<const uint2*>(p + row8);
  const uint2 v2 = *reinterpret_cast<const uint2*>(p + 8);
  const uint2 v3 = *reinterpret_cast<const uint2*>(p + row8 + 8);
  h[0] = v0.x, h[1] = v1.x, h[2] = v2.x, h[3] = v3.x;
  l[0] = v0.y, l[1] = v1.y, l[2] = v2.y, l[3] = v3.y;
}

// Descriptor forward of atoms i0 .. i0 + 7 (those below nrow): warp w of the
// group sums atom i0 + w's slots into W, then all warps share the products.
// touched: the intervals that hold a slot of any of the eight, per type (may
// be NULL); row_scale: per descriptor row, the power of two that brings it
// below 2^14 (the operand scale of the FP16 fitting GEMM; may be NULL).
template <int CH, int NC, bool COH = false>
__device__ __forceinline__ void cheb_fwd_group(int i0, int nrow, int w, int lane, int bar,
                                               float* gsm, float* __restrict__ xyz_out,
                                               float* __restrict__ D,
                                               const int* __restrict__ drow,
                                               const float* __restrict__ em,
                                               const ChebTables& ct, const TypeTables& tt, int M,
                                               int naxis, float inv_nnei, unsigned* touched,
                                               float* row_scale) {
  constexpr int NTW = MAXM / 8 / CHEB_A;  // channel tiles per warp
  const int nnei = tt.nnei, wst = ct.wstride, ntile = (M + 7) / 8;
  const int i = i0 + w;
  const bool act = i < nrow;
  float* W = gsm;  // [32][wst], later x [32][M]
  float* s_inv = gsm + 4 * CHEB_A * (wst > M ? wst : M);  // [8] 1 / scale
  unsigned* s_mask = reinterpret_cast<unsigned*>(s_inv + CHEB_A);
  float* sT = s_inv + 2 * CHEB_A + w * (32 * CHEB_TS + 32 * 4);
  float* sE = sT + 32 * CHEB_TS;
  float* Wa = W + w * 4 * wst;  // this atom's rows
  const int g = lane >> 2, t4 = lane & 3;
  const int kk = lane & 15, dp = lane >> 4;  // W entries while summing: k, columns 2 dp, 2 dp + 1
  const int cd = lane >> 3, cp = lane & 7;   // while splitting: column, k pair
  float acc[2][NTW][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < NTW; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[m][j][k] = 0.f;
  bool outl = false;  // this atom has slots outside [lo, hi)
  for (int t = 0; t < tt.ntypes; ++t) {
    const int s0 = tt.sec[t], nt = tt.sec[t + 1] - s0;
    if (nt <= 0) {
      if (touched != nullptr && w == 0 && lane == 0)
        touched[(i0 / CHEB_A) * tt.ntypes + t] = 0u;
      continue;
    }
    const ChebNet& net = ct.net[t];
    for (int q = lane; q < wst; q += 32)
      reinterpret_cast<float4*>(Wa)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    unsigned mask = 0u;
    float inv = 0.f;
    if (act) {
      const float4* erow = reinterpret_cast<const float4*>(em + (size_t)i * nnei * 4) + s0;
      const float last = cheb_last<COH>(erow, nt);
      float* w0 = Wa + 2 * dp * wst + kk;
      float a0 = 0.f, a1 = 0.f, bound = 0.f;
      int cur = -1;
      bool done = false;
      for (int q0 = 0; q0 < nt && !done; q0 += 32) {
        ChebSlots c = cheb_slots<COH>(erow, q0, nt, last, lane);
        done = c.folded;
        const bool in = lane < c.n;
        int r = 0;
        float x = 0.f, ih = 0.f;
        const bool core = in && cheb_locate(net, c.e.x, r, x, ih);
        outl |= __ballot_sync(0xffffffffu, in && !core) != 0u;
        if (core) {
          c.e.x *= c.rep;  // the other columns of a fold slot are zero
        } else {
          c.e = make_float4(0.f, 0.f, 0.f, 0.f);
          x = 0.f;
        }
        bound += fmaxf(fmaxf(fabsf(c.e.x), fabsf(c.e.y)), fmaxf(fabsf(c.e.z), fabsf(c.e.w)));
        // this lane's slot: T_0 .. T_15
        float T[CHEB_K];
        T[0] = 1.f;
        T[1] = x;
#pragma unroll
        for (int k = 2; k < CHEB_K; ++k) T[k] = fmaf(2.f * x, T[k - 1], -T[k - 2]);
#pragma unroll
        for (int k = 0; k < CHEB_K; k += 4)
          *reinterpret_cast<float4*>(sT + lane * CHEB_TS + k) =
              make_float4(T[k], T[k + 1], T[k + 2], T[k + 3]);
        *reinterpret_cast<float4*>(sE + lane * 4) = c.e;
        const int up = __shfl_up_sync(0xffffffffu, r, 1);
        const unsigned chg =
            __ballot_sync(0xffffffffu, in && r != (lane == 0 ? cur : up));
        __syncwarp();
        // runs of slots of one interval (slots come nearest first, so an
        // interval is one run; any other order only makes more runs)
        int s = 0;
        while (s < c.n) {
          if ((chg >> s) & 1u) {
            if (cur >= 0) {
              w0[cur * CHEB_K] += a0;
              w0[wst + cur * CHEB_K] += a1;
            }
            cur = __shfl_sync(0xffffffffu, r, s);
            mask |= 1u << cur;
            a0 = a1 = 0.f;
          }
          const unsigned rest = chg & ~((2u << s) - 1u);
          const int end = rest ? __ffs(rest) - 1 : c.n;
#pragma unroll 4
          for (; s < end; ++s) {
            const float tv = sT[s * CHEB_TS + kk];
            const float2 ev = *reinterpret_cast<const float2*>(sE + s * 4 + 2 * dp);
            a0 = fmaf(tv, ev.x, a0);
            a1 = fmaf(tv, ev.y, a1);
          }
        }
        __syncwarp();  // the staging is rewritten by the next chunk
      }
      if (cur >= 0) {
        w0[cur * CHEB_K] += a0;
        w0[wst + cur * CHEB_K] += a1;
      }
      __syncwarp();
      // |T_k| <= 1 (to rounding), so sum |e| bounds every entry of W; the
      // touched entries become (hi pair, lo pair) words in place
      const float sc = f16_scale(warp_sum(bound), inv);
      for (unsigned m = mask; m; m &= m - 1u) {
        float2* p = reinterpret_cast<float2*>(Wa + cd * wst + (__ffs(m) - 1) * CHEB_K + 2 * cp);
        const float2 v = *p;
        uint2 o;
        split_f16(v.x * sc, v.y * sc, o.x, o.y);
        *reinterpret_cast<uint2*>(p) = o;
      }
    }
    if (lane == 0) {
      s_inv[w] = inv * net.inv_scale;
      s_mask[w] = mask;
    }
    cheb_sync(bar);
    unsigned all = 0u;
#pragma unroll
    for (int k = 0; k < CHEB_A; ++k) all |= s_mask[k];
    if (touched != nullptr && w == 0 && lane == 0) touched[(i0 / CHEB_A) * tt.ntypes + t] = all;
    const float in4[4] = {s_inv[g >> 2], s_inv[2 + (g >> 2)], s_inv[4 + (g >> 2)],
                          s_inv[6 + (g >> 2)]};
    const float* wa = W + g * wst + 2 * t4;
    const uint4* fr = net.fw + w * 32 + lane;
    auto load_b = [&](uint4 (&b)[NTW], int r) {
#pragma unroll
      for (int j = 0; j < NTW; ++j)
        if (w + CHEB_A * j < ntile) b[j] = __ldg(fr + (r * ntile + CHEB_A * j) * 32);
    };
    uint4 b[NTW], bn[NTW];
    if (all) load_b(b, __ffs(all) - 1);
    while (all) {
      const int r = __ffs(all) - 1;
      all &= all - 1u;
      if (all) load_b(bn, __ffs(all) - 1);  // the next interval's coefficients
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        unsigned ah[4], al[4];
        frag_a(ah, al, wa + m * 16 * wst + r * CHEB_K, 8 * wst);
#pragma unroll
        for (int j = 0; j < NTW; ++j) {
          if (w + CHEB_A * j >= ntile) break;
          float c[4];
          mma_split(c, ah, al, b[j]);
          acc[m][j][0] = fmaf(c[0], in4[2 * m], acc[m][j][0]);
          acc[m][j][1] = fmaf(c[1], in4[2 * m], acc[m][j][1]);
          acc[m][j][2] = fmaf(c[2], in4[2 * m + 1], acc[m][j][2]);
          acc[m][j][3] = fmaf(c[3], in4[2 * m + 1], acc[m][j][3]);
        }
      }
#pragma unroll
      for (int j = 0; j < NTW; ++j) b[j] = bn[j];
    }
    cheb_sync(bar);  // W is rebuilt by the next type
  }
  float* sx = gsm;  // x of the eight atoms, [4][M] each
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int j = 0; j < NTW; ++j) {
      const int col = (w + CHEB_A * j) * 8 + 2 * t4;
      if (col < M) {  // M is even
        *reinterpret_cast<float2*>(sx + (m * 16 + g) * M + col) =
            make_float2(acc[m][j][0] * inv_nnei, acc[m][j][1] * inv_nnei);
        *reinterpret_cast<float2*>(sx + (m * 16 + g + 8) * M + col) =
            make_float2(acc[m][j][2] * inv_nnei, acc[m][j][3] * inv_nnei);
      }
    }
  cheb_sync(bar);
  if (act) {
    float* xa = sx + w * 4 * M;
    if (outl) {  // slots outside the intervals, from the table
      const int m0 = 4 * lane;
      for (int t = 0; t < tt.ntypes; ++t) {
        const int s0 = tt.sec[t], nt = tt.sec[t + 1] - s0;
        if (nt <= 0) continue;
        const ChebNet& net = ct.net[t];
        const float4* erow = reinterpret_cast<const float4*>(em + (size_t)i * nnei * 4) + s0;
        const float last = cheb_last<COH>(erow, nt);
        bool done = false;
        for (int q0 = 0; q0 < nt && !done; q0 += 32) {
          const ChebSlots c = cheb_slots<COH>(erow, q0, nt, last, lane);
          done = c.folded;
          unsigned b = __ballot_sync(0xffffffffu,
                                     lane < c.n && !(c.e.x >= net.lo && c.e.x < net.hi));
          while (b) {
            const int s = __ffs(b) - 1;
            b &= b - 1u;
            const float4 e = make_float4(__shfl_sync(0xffffffffu, c.e.x, s),
                                         __shfl_sync(0xffffffffu, c.e.y, s),
                                         __shfl_sync(0xffffffffu, c.e.z, s),
                                         __shfl_sync(0xffffffffu, c.e.w, s));
            const float rep = __shfl_sync(0xffffffffu, c.rep, s) * inv_nnei;
            int idx;
            float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
            flocate(tt.info[t], e.x, idx, L.y, L.z);
            if (m0 < M) {
              const Coef4<NC> cf =
                  load_coef4<CH, NC>(tt.table[t] + m0 + (size_t)idx * M * NC, M);
              float2 a01[4], a23[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) a01[k] = a23[k] = make_float2(0.f, 0.f);
              fwd_slot<NC>(a01, a23, cf, e, L, 1.f);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                float4* p = reinterpret_cast<float4*>(xa + k * M + m0);
                float4 v = *p;
                v.x = fmaf(a01[k].x, rep, v.x);
                v.y = fmaf(a01[k].y, rep, v.y);
                v.z = fmaf(a23[k].x, rep, v.z);
                v.w = fmaf(a23[k].y, rep, v.w);
                *p = v;
              }
            }
          }
        }
      }
      __syncwarp();
    }
    float4* xo = reinterpret_cast<float4*>(xyz_out + (size_t)i * 4 * M);
    for (int q = lane; q < M; q += 32) xo[q] = reinterpret_cast<const float4*>(xa)[q];
    if (row_scale != nullptr) {
      const float sc = descriptor_scale(xa, M, lane);
      if (lane == 0) row_scale[drow[i]] = sc;
    }
    write_descriptor(D + (size_t)drow[i] * M * naxis, xa, M, naxis, lane);
  }
}

// Descriptor backward of atoms i0 .. i0 + 7: net_deriv rows, a warp per atom
// with the products shared. touched as written by cheb_fwd_group, or NULL
// (every interval is evaluated then).
template <int CH, int NC>
__device__ __forceinline__ void cheb_bwd_group(int i0, int nrow, int w, int lane, int bar,
                                               float* gsm, float* __restrict__ net_deriv,
                                               const float* __restrict__ dD,
                                               const int* __restrict__ drow,
                                               const float* __restrict__ xyz,
                                               const float* __restrict__ em,
                                               const ChebTables& ct, const TypeTables& tt, int M,
                                               int naxis, float inv_nnei,
                                               const unsigned* touched) {
  constexpr int KS = MAXM / 16;
  const int nnei = tt.nnei, ksteps = (M + 15) / 16, ys = ksteps * 16 + 8;
  const int i = i0 + w;
  const bool act = i < nrow;
  const int pw = 4 * M + 4 * MAXAX + M * naxis;
  float* s_x = gsm + w * pw;  // prologue, a warp each; later Z [8 atoms][interval][16 k][4]
  float* s_t = s_x + 4 * M;
  float* s_d = s_t + 4 * MAXAX;
  float* Z = gsm;
  const int zf = CHEB_A * ct.rmax * CHEB_K * 4;
  float* s_inv = gsm + (zf > CHEB_A * pw ? zf : CHEB_A * pw);
  float* Y = s_inv + 2 * CHEB_A;  // [32][ys]: dxyz as (hi pair, lo pair) words
  const int g = lane >> 2, t4 = lane & 3, m0 = 4 * lane;
  {
    float dyr[4][4];
    float inv = 0.f, sc = 0.f;
    if (act) {
      bwd_dyr(dyr, i, lane, s_x, s_t, s_d, dD, drow, xyz, M, naxis, inv_nnei);
      float mx = 0.f;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch)
#pragma unroll
        for (int k = 0; k < 4; ++k) mx = fmaxf(mx, fabsf(dyr[ch][k]));
      sc = f16_scale(warp_max(mx), inv);
    }
    if (m0 < ksteps * 16) {  // zero beyond M and for atoms beyond the last
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint4 o = make_uint4(0u, 0u, 0u, 0u);
        if (act) {
          split_f16(dyr[0][k] * sc, dyr[1][k] * sc, o.x, o.y);
          split_f16(dyr[2][k] * sc, dyr[3][k] * sc, o.z, o.w);
        }
        *reinterpret_cast<uint4*>(Y + (w * 4 + k) * ys + m0) = o;
      }
    }
    if (lane == 0) s_inv[w] = inv;
  }
  cheb_sync(bar);
  const float in4[4] = {s_inv[g >> 2], s_inv[2 + (g >> 2)], s_inv[4 + (g >> 2)],
                        s_inv[6 + (g >> 2)]};
  bool outl = false;
  for (int t = 0; t < tt.ntypes; ++t) {
    const int s0 = tt.sec[t], nt = tt.sec[t + 1] - s0;
    if (nt <= 0) continue;
    const ChebNet& net = ct.net[t];
    unsigned mask = (2u << (net.R - 1)) - 1u;
    if (touched != nullptr) mask = touched[(i0 / CHEB_A) * tt.ntypes + t];
    // Z of the touched intervals: the 8-wide k tiles (two per interval) in
    // turn over the warps
    for (int n = w; n < 2 * __popc(mask); n += CHEB_A) {
      unsigned m = mask;
      for (int k = n >> 1; k > 0; --k) m &= m - 1u;
      const int r = __ffs(m) - 1, h = n & 1;
      const uint4* fr = net.bw + (size_t)(r * 2 + h) * ksteps * 32 + lane;
      uint4 b[KS];
#pragma unroll
      for (int k = 0; k < KS; ++k)
        if (k < ksteps) b[k] = __ldg(fr + k * 32);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        float z[4] = {0.f, 0.f, 0.f, 0.f};
        const float* y = Y + (mt * 16 + g) * ys + 2 * t4;
#pragma unroll
        for (int k = 0; k < KS; ++k) {
          if (k >= ksteps) break;
          unsigned ah[4], al[4];
          frag_a(ah, al, y + k * 16, 8 * ys);
          float c[4];
          mma_split(c, ah, al, b[k]);
#pragma unroll
          for (int j = 0; j < 4; ++j) z[j] += c[j];
        }
        const float ia = in4[2 * mt] * net.inv_scale, ib = in4[2 * mt + 1] * net.inv_scale;
        float* zp =
            Z + (((mt * 4 + (g >> 2)) * net.R + r) * CHEB_K + h * 8 + 2 * t4) * 4 + (g & 3);
        float* zq = zp + 2 * net.R * CHEB_K * 4;
        zp[0] = z[0] * ia;
        zp[4] = z[1] * ia;
        zq[0] = z[2] * ib;
        zq[4] = z[3] * ib;
      }
    }
    cheb_sync(bar);
    if (act) {
      const size_t row = (size_t)i * nnei + s0;
      const float4* erow = reinterpret_cast<const float4*>(em) + row;
      float4* nrow_ = reinterpret_cast<float4*>(net_deriv) + row;
      const float last = cheb_last<false>(erow, nt);
      const float4* Za = reinterpret_cast<const float4*>(Z) + w * net.R * CHEB_K;
      bool done = false;
      for (int q0 = 0; q0 < nt; q0 += 32) {
        const int q = q0 + lane;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!done) {
          const ChebSlots c = cheb_slots<false>(erow, q0, nt, last, lane);
          done = c.folded;
          const bool in = lane < c.n;
          int r = 0;
          float x = 0.f, ih = 0.f;
          const bool core = in && cheb_locate(net, c.e.x, r, x, ih);
          outl |= __ballot_sync(0xffffffffu, in && !core) != 0u;
          if (core) {
            const float4* z = Za + r * CHEB_K;
            const float x2 = 2.f * x;
            float4 v = z[0];
            o = v;
            float T0 = 1.f, T1 = x, U0 = 0.f, U1 = 1.f, sl = 0.f;  // T_{k-1}, T_k, U_{k-2}, U_{k-1}
#pragma unroll
            for (int k = 1; k < CHEB_K; ++k) {
              v = z[k];
              o.x = fmaf(T1, v.x, o.x);
              o.y = fmaf(T1, v.y, o.y);
              o.z = fmaf(T1, v.z, o.z);
              o.w = fmaf(T1, v.w, o.w);
              const float ez = fmaf(c.e.x, v.x, fmaf(c.e.y, v.y, fmaf(c.e.z, v.z, c.e.w * v.w)));
              sl = fmaf((float)k * U1, ez, sl);  // T_k' = k U_{k-1}
              const float T2 = fmaf(x2, T1, -T0), U2 = fmaf(x2, U1, -U0);
              T0 = T1, T1 = T2, U0 = U1, U1 = U2;
            }
            o.x = fmaf(sl, ih, o.x);
            o.x *= c.rep, o.y *= c.rep, o.z *= c.rep, o.w *= c.rep;
          }
        }
        if (q < nt) nrow_[q] = o;
      }
    }
    cheb_sync(bar);  // Z is rebuilt by the next type (or the prologue's buffers reused)
  }
  if (act && outl) {  // slots outside the intervals, from the table
    float dyr[4][4];
    bwd_dyr(dyr, i, lane, s_x, s_t, s_d, dD, drow, xyz, M, naxis, inv_nnei);
    float2 dyr01[4], dyr23[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dyr01[k] = make_float2(dyr[0][k], dyr[1][k]);
      dyr23[k] = make_float2(dyr[2][k], dyr[3][k]);
    }
    for (int t = 0; t < tt.ntypes; ++t) {
      const int s0 = tt.sec[t], nt = tt.sec[t + 1] - s0;
      if (nt <= 0) continue;
      const ChebNet& net = ct.net[t];
      const size_t row = (size_t)i * nnei + s0;
      const float4* erow = reinterpret_cast<const float4*>(em) + row;
      const float last = cheb_last<false>(erow, nt);
      bool done = false;
      for (int q0 = 0; q0 < nt && !done; q0 += 32) {
        const ChebSlots c = cheb_slots<false>(erow, q0, nt, last, lane);
        done = c.folded;
        unsigned b = __ballot_sync(0xffffffffu,
                                   lane < c.n && !(c.e.x >= net.lo && c.e.x < net.hi));
        while (b) {
          const int s = __ffs(b) - 1;
          b &= b - 1u;
          const float4 e = make_float4(__shfl_sync(0xffffffffu, c.e.x, s),
                                       __shfl_sync(0xffffffffu, c.e.y, s),
                                       __shfl_sync(0xffffffffu, c.e.z, s),
                                       __shfl_sync(0xffffffffu, c.e.w, s));
          const float rep = __shfl_sync(0xffffffffu, c.rep, s);
          int idx;
          float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
          flocate(tt.info[t], e.x, idx, L.y, L.z);
          float P[4] = {0.f, 0.f, 0.f, 0.f};
          if (m0 < M) {
            const Coef4<NC> cf =
                load_coef4<CH, NC>(tt.table[t] + m0 + (size_t)idx * M * NC, M);
            bwd_slot<NC>(P, cf, e, L, rep, dyr01, dyr23);
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) P[k] = warp_sum(P[k]);
          if (lane == 0)
            reinterpret_cast<float4*>(net_deriv)[row + q0 + s] =
                make_float4(P[0], P[1], P[2], P[3]);
        }
      }
    }
  }
}

// checks the nets of a host description (one per neighbor type; a type
// without slots needs none)
static int make_cheb(ChebTables& ct, const dpb_cheb_net* nets, int ntypes, const int* sec) {
  if (nets == nullptr || ntypes < 1 || ntypes > PMAXT) {
    set_error("se_a cheb: one net per neighbor type (at most %d)", PMAXT);
    return DPB_ERR_INVALID;
  }
  ct.rmax = 1;
  for (int t = 0; t < ntypes; ++t) {
    const dpb_cheb_net& n = nets[t];
    ChebNet& c = ct.net[t];
    c = ChebNet{};
    c.R = 1;
    if (sec[t + 1] == sec[t]) continue;
    const uintptr_t al = (uintptr_t)n.fw | (uintptr_t)n.bw;
    if (n.fw == nullptr || n.bw == nullptr || n.iv == nullptr || n.lut == nullptr ||
        (al & 15) != 0 || ((uintptr_t)n.iv & 7) != 0 || n.nintervals < 1 ||
        n.nintervals > CHEB_MAXR || n.ncell < 1 || !(n.lo < n.hi) || !(n.inv_cell > 0.f) ||
        !(n.coef_scale > 0.f)) {
      set_error("se_a cheb: invalid net of neighbor type %d (1..%d intervals, aligned "
                "fragments)", t, CHEB_MAXR);
      return DPB_ERR_INVALID;
    }
    c.fw = static_cast<const uint4*>(n.fw);
    c.bw = static_cast<const uint4*>(n.bw);
    c.iv = reinterpret_cast<const float2*>(n.iv);
    c.lut = n.lut;
    c.lo = n.lo;
    c.hi = n.hi;
    c.inv_cell = n.inv_cell;
    c.inv_scale = 1.f / n.coef_scale;
    c.ncell = n.ncell;
    c.R = n.nintervals;
    if (c.R > ct.rmax) ct.rmax = c.R;
  }
  ct.wstride = CHEB_K * ct.rmax + 8;
  return DPB_OK;
}

}  // namespace dpb
