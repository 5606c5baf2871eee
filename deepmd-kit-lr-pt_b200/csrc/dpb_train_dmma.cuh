// The embedding passes of the standard net (1 -> 25 -> 50 -> 100) on the matrix
// instructions: in FP64 forward (G, xyz, D) and force backward (dE/d(em)), in
// FP64 and FP32 the tangent and the reverse pass over primal and tangent (weight
// gradients): the same quantities as k_tr_fwd / k_tr_bwd / k_tr_tan / k_tr_rev
// (dpb_train.cu, which includes this file).
//
// One warp takes one center atom and 16 neighbor rows at a time through the
// whole net as mma.m16n8k4 products. The FMA form held one channel per lane
// and read every operand from shared memory: 8 warps per SM, a third of the
// FP64 rate. Here the weights lie in shared memory in fragment order and
// the activations stay in registers between the layers, because the order of
// a product's k and of its columns is free: lane (g, t) = (lane / 4, lane % 4)
// owns the layer-1 channels s(j, t) = 4 j + t (j < 7) of rows g and g + 8, and
// column pair t of layer 2's tile j is the pair s(j, t), s(j, t) + 25, whose
// residual is that layer-1 channel and which is k = t of layer 3's steps
// (j, 0) and (j, 1). Layer 3 runs transposed (channels x rows), so its
// results feed the contraction over rows as A operands. What is left is the
// FP64 pipe itself: the products at 64 FMA per clock and SM, and 175 tanh per
// row (tanh_f64 below).
//
// Measured, 3,993 atoms: forward 1.17 -> 0.56 ms, backward 2.06 -> 0.91 ms.
#pragma once

namespace dpb {

constexpr int EM_S1 = 7;                       // layer-1 channels per lane and row
constexpr int EM_F2 = 7 * 7 * 32;              // fragment doubles: layer 2
constexpr int EM_F3 = 14 * (6 * 2 + 1) * 32;   // layer 3 (six 16-channel tiles, one of 8)
constexpr int EM_B3 = 25 * 7 * 32;             // layer 3 adjoint
constexpr int EM_B2 = 14 * 4 * 32;             // layer 2 adjoint
constexpr int EM_V = 28 + 28 + 52 + 100;       // W1, b1, b2, b3
constexpr int EM_FWD_T = EM_F2 + EM_F3 + EM_V;               // per type
constexpr int EM_BWD_T = EM_F2 + EM_F3 + EM_B3 + EM_B2 + EM_V;
constexpr int EM_H2S = 50;                     // row stride of the staged layer-2 outputs
constexpr int EM_TS = 20;                      // row stride of a staged 16 x 16 tile
constexpr int EM_FWD_W = 16 * 4 + 16 * EM_H2S;               // doubles per warp
constexpr int EM_BWD_W = 16 * 4 + 400 + 2 * 16 * EM_TS;
constexpr int EM_FWD_MAXW = 12, EM_BWD_MAXW = 8;

// tanh(x) = E / (E + 2), E = exp(2|x|) - 1 kept as 2^k (e^r - 1) + (2^k - 1),
// so small arguments keep their relative accuracy: 2|x| = k ln 2 + r, e^r - 1 by
// its Taylor series to r^13 (|r| <= 0.347: remainder 1e-17). The quotient: the
// hardware's estimate of the reciprocal (20 bits), one Newton-Raphson step on it
// (which squares its error; Muller et al., Handbook of Floating-Point Arithmetic,
// the chapter on division) and Markstein's correction by the residual (Computation
// of elementary functions on the IBM RISC System/6000 processor, 1990), the
// residual against E + 2 with its rounding (Dekker's fast two-sum). The roundings
// add up to less than 6 * 2^-53 of the result (r, the series and E 4.3 where E is
// smallest for its power of two, of which 0.83 reach the quotient, which adds one).
// Measured worst 2.21 * 2^-53 over 1e-300 .. 40 (CUDA's tanh 2.23). NaN stays NaN,
// beyond 20 the result is 1.
__device__ __forceinline__ double tanh_f64(double x) {
  const double ax = fabs(x);
  const double y = 2.0 * (ax > 20.0 ? 20.0 : ax);
  const double magic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low bits are the integer
  const double kd = fma(y, 1.4426950408889634, magic);
  const int k = __double2loint(kd);
  const double kf = kd - magic;
  // ln 2 as its 40 leading bits and the rest: k times the former is exact
  double r = fma(-kf, 0.6931471805601177, y);
  r = fma(-kf, -1.7239444525614835e-13, r);
  double p = 1.0 / 6227020800.0;  // 1 / 13!
  p = fma(p, r, 1.0 / 479001600.0);
  p = fma(p, r, 1.0 / 39916800.0);
  p = fma(p, r, 1.0 / 3628800.0);
  p = fma(p, r, 1.0 / 362880.0);
  p = fma(p, r, 1.0 / 40320.0);
  p = fma(p, r, 1.0 / 5040.0);
  p = fma(p, r, 1.0 / 720.0);
  p = fma(p, r, 1.0 / 120.0);
  p = fma(p, r, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(r * r, p, r);
  const double s = __hiloint2double((1023 + k) << 20, 0);
  const double E = fma(s, p, s - 1.0);
  const double d = E + 2.0;
  double q;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(q) : "d"(d));
  q = fma(q, fma(-d, q, 1.0), q);
  double v = E * q;
  const double dl = E - (d - 2.0);  // d + dl = E + 2
  v = fma(fma(-dl, v, fma(-d, v, E)), q, v);
  return copysign(v, x);
}

__device__ __forceinline__ void dmma16(double (&c)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, "
      "{%0, %1, %2, %3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}
__device__ __forceinline__ void dmma8(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// layer-2 channel of column / k pair member v owned by lane column u at step j,
// -1 when the slot is padding
__device__ __forceinline__ int em_c2(int j, int u, int v) {
  return 4 * j + u < 25 ? 4 * j + u + 25 * v : -1;
}

// zero in the padding of the layer-1 channels (an infinite input times its zero
// weight is none)
template <typename T>
__device__ __forceinline__ T em_pad(int s, int t4, T v) {
  return 4 * s + t4 < 25 ? v : (T)0;
}

// layer 2 and its adjoint in fragment order, W1 and b1 padded to 28
template <typename T>
__device__ inline void em_stage_f2(T* F2, const T* W2) {
  for (int e = threadIdx.x; e < EM_F2; e += blockDim.x) {
    const int lane = e & 31, j = (e >> 5) % 7, s = (e >> 5) / 7, g = lane >> 2;
    const int k = 4 * s + (lane & 3), c = em_c2(j, g >> 1, g & 1);
    F2[e] = k < 25 && c >= 0 ? W2[k * 50 + c] : (T)0;
  }
}
template <typename T>
__device__ inline void em_stage_b2(T* B2, const T* W2) {
  for (int e = threadIdx.x; e < EM_B2; e += blockDim.x) {
    const int lane = e & 31, q = (e >> 5) & 3, step = (e >> 5) >> 2, g = lane >> 2;
    const int c = em_c2(step >> 1, lane & 3, step & 1);
    const int k = 4 * (2 * q + (g & 1)) + (g >> 1);
    B2[e] = c >= 0 && k < 25 ? W2[k * 50 + c] : (T)0;
  }
}
template <typename T>
__device__ inline void em_stage_v(T* V, const TrNet<T>& net, int t) {
  for (int e = threadIdx.x; e < 28; e += blockDim.x) {
    V[e] = e < 25 ? net.W[t][0][e] : (T)0;
    V[28 + e] = e < 25 ? net.b[t][0][e] : (T)0;
  }
  for (int e = threadIdx.x; e < 50; e += blockDim.x) V[56 + e] = net.b[t][1][e];
}

// weights of net t into fragment order
__device__ inline void em_stage(double* w, const TrNet<double>& net, int t, bool bwd) {
  double* F2 = w;
  double* F3 = F2 + EM_F2;
  double* V = F3 + EM_F3 + (bwd ? EM_B3 + EM_B2 : 0);
  const double *W2 = net.W[t][1], *W3 = net.W[t][2];
  const int n = blockDim.x;
  em_stage_f2(F2, W2);
  for (int e = threadIdx.x; e < EM_F3; e += n) {
    // tiles 0..5: [tile][step][lane][row g, row g + 8]; tile 6: [step][lane]
    const bool last = e >= 6 * 14 * 64;
    const int f = last ? e - 6 * 14 * 64 : e;
    const int h = last ? 0 : f & 1, lane = last ? f & 31 : (f >> 1) & 31;
    const int q = last ? f >> 5 : f >> 6;
    const int step = q % 14, m = (last ? 96 : q / 14 * 16) + 8 * h + (lane >> 2);
    const int c = em_c2(step >> 1, lane & 3, step & 1);
    F3[e] = m < 100 && c >= 0 ? W3[c * 100 + m] : 0.;
  }
  em_stage_v(V, net, t);
  for (int e = threadIdx.x; e < 100; e += n) V[108 + e] = net.b[t][2][e];
  if (!bwd) return;
  double* B3 = F3 + EM_F3;
  for (int e = threadIdx.x; e < EM_B3; e += n) {
    const int lane = e & 31, j = (e >> 5) % 7, s = (e >> 5) / 7, g = lane >> 2;
    const int c = em_c2(j, g >> 1, g & 1);
    B3[e] = c >= 0 ? W3[c * 100 + 4 * s + (lane & 3)] : 0.;
  }
  em_stage_b2(B3 + EM_B3, W2);
}

// layers 1 and 2 of 16 rows: h1a / h1b the layer-1 outputs of rows g / g + 8 at
// the lane's channels, h2[j] the layer-2 outputs (row g: pair members 0, 1;
// row g + 8: 0, 1), with STAGE stored by row in hs as well
template <bool STAGE>
__device__ __forceinline__ void em_layers12(double (&h1a)[EM_S1], double (&h1b)[EM_S1],
                                            double (&h2)[7][4], double xa, double xb,
                                            const double* F2, const double* V, double* hs,
                                            int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int s = 0; s < EM_S1; ++s) {
    const double w = V[4 * s + t], b = V[28 + 4 * s + t];
    h1a[s] = em_pad(s, t, tanh_f64(fma(xa, w, b)));
    h1b[s] = em_pad(s, t, tanh_f64(fma(xb, w, b)));
  }
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const bool ok = 4 * j + t < 25;
    h2[j][0] = h2[j][2] = ok ? V[56 + 4 * j + t] : 0.;
    h2[j][1] = h2[j][3] = ok ? V[56 + 4 * j + t + 25] : 0.;
  }
#pragma unroll
  for (int s = 0; s < EM_S1; ++s)
#pragma unroll
    for (int j = 0; j < 7; ++j) dmma16(h2[j], h1a[s], h1b[s], F2[(s * 7 + j) * 32 + lane]);
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    h2[j][0] = tanh_f64(h2[j][0]) + h1a[j];
    h2[j][1] = tanh_f64(h2[j][1]) + h1a[j];
    h2[j][2] = tanh_f64(h2[j][2]) + h1b[j];
    h2[j][3] = tanh_f64(h2[j][3]) + h1b[j];
    if (STAGE && 4 * j + t < 25) {
      double* p = hs + g * EM_H2S + 4 * j + t;
      p[0] = h2[j][0];
      p[25] = h2[j][1];
      p[8 * EM_H2S] = h2[j][2];
      p[8 * EM_H2S + 25] = h2[j][3];
    }
  }
}

// layer 3 of channel tile m, transposed: z[n][..] rows 8 n + 2 t, + 1 of
// channels 16 m + g ([0], [1]) and + 8 ([2], [3]; absent in tile 6)
template <int LAST>
__device__ __forceinline__ void em_layer3(double (&z)[2][4], int m, const double (&h2)[7][4],
                                          const double* F3, const double* V, int lane) {
  const int g = lane >> 2, c = 16 * m + g;
  const double b0 = c < 100 ? V[108 + c] : 0., b1 = LAST ? 0. : V[108 + c + 8];
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    z[n][0] = z[n][1] = b0;
    z[n][2] = z[n][3] = b1;
  }
#pragma unroll
  for (int j = 0; j < 7; ++j)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int step = 2 * j + v;
      if (LAST) {
        const double a = F3[6 * 14 * 64 + step * 32 + lane];
        dmma8(z[0][0], z[0][1], a, h2[j][v]);
        dmma8(z[1][0], z[1][1], a, h2[j][2 + v]);
      } else {
        const double2 a = *reinterpret_cast<const double2*>(F3 + ((m * 14 + step) * 32 + lane) * 2);
        dmma16(z[0], a.x, a.y, h2[j][v]);
        dmma16(z[1], a.x, a.y, h2[j][2 + v]);
      }
    }
}

// 16 entries of the list from e0 on: env rows (times the multiplicity) to rr
// [16][4] and each row's x to this lane's rows g, g + 8
__device__ __forceinline__ void em_rows(double* rr, double& xa, double& xb, const int* ent,
                                        int e0, int ne, const double* em_row, bool mult,
                                        int lane) {
  double x = 0.;
  if (lane < 16) {
    double2 u = make_double2(0., 0.), v = u;
    if (lane < ne) {
      const int en = ent[e0 + lane];
      const double2* src = reinterpret_cast<const double2*>(em_row + (size_t)(en & 0xFFFF) * 4);
      u = src[0];
      v = src[1];
      x = u.x;
      if (mult) {
        const double mu = (double)(en >> 16);
        u.x *= mu, u.y *= mu, v.x *= mu, v.y *= mu;
      }
    }
    reinterpret_cast<double2*>(rr)[lane * 2] = u;
    reinterpret_cast<double2*>(rr)[lane * 2 + 1] = v;
  }
  xa = __shfl_sync(0xffffffffu, x, lane >> 2);
  xb = __shfl_sync(0xffffffffu, x, 8 + (lane >> 2));
  __syncwarp();
}

__global__ void __launch_bounds__(32 * EM_FWD_MAXW, 1)
k_emb_fwd_dmma(double* __restrict__ xyz_out, double* __restrict__ D_out,
               const double* __restrict__ em, TrNet<double> net, TrGeom g) {
  extern __shared__ __align__(16) double esm[];
  pdl_wait();
  pdl_trigger();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int gr = lane >> 2, t4 = lane & 3;
  for (int t = 0; t < g.ntypes; ++t) em_stage(esm + (size_t)t * EM_FWD_T, net, t, false);
  __syncthreads();
  double* ws = esm + (size_t)g.ntypes * EM_FWD_T + (size_t)w * EM_FWD_W;
  double* rr = ws;
  double* hs = ws + 64;
  int* ent = reinterpret_cast<int*>(esm + (size_t)g.ntypes * EM_FWD_T + (size_t)nw * EM_FWD_W) +
             (size_t)w * (g.nnei + TR_MAXT + 1);
  int* secn = ent + g.nnei;
  for (int row = blockIdx.x * nw + w; row < g.nrows; row += gridDim.x * nw) {
    tr_entries(ent, secn, g.nlist + (size_t)row * g.nnei, g, g.type[row], true, lane, 0,
               g.ntypes);
    double X[7][4];  // xyz: channels 16 m + g (+ 8), env columns 2 t, 2 t + 1 (t < 2)
#pragma unroll
    for (int m = 0; m < 7; ++m)
#pragma unroll
      for (int k = 0; k < 4; ++k) X[m][k] = 0.;
    for (int t = 0; t < g.ntypes; ++t) {
      const double* F2 = esm + (size_t)t * EM_FWD_T;
      const double* F3 = F2 + EM_F2;
      const double* V = F3 + EM_F3;
      for (int e0 = secn[t]; e0 < secn[t + 1]; e0 += 16) {
        double xa, xb;
        em_rows(rr, xa, xb, ent, e0, min(16, secn[t + 1] - e0),
                em + (size_t)row * g.nnei * 4, true, lane);
        double rb[2][2];  // env column g (< 4) of rows 8 n + 2 t + e
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) rb[n][e] = gr < 4 ? rr[(8 * n + 2 * t4 + e) * 4 + gr] : 0.;
        double h1a[EM_S1], h1b[EM_S1], h2[7][4];
        em_layers12<true>(h1a, h1b, h2, xa, xb, F2, V, hs, lane);
        __syncwarp();
        auto tile = [&](auto last, int m, double (&x)[4]) {
          constexpr int LAST = decltype(last)::value;
          double z[2][4];
          em_layer3<LAST>(z, m, h2, F3, V, lane);
          const int c = 16 * m + gr;
          const int ca = c < 50 ? c : c - 50, cb = c + 8 < 50 ? c + 8 : c - 42;
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const double* hrow = hs + (8 * n + 2 * t4 + e) * EM_H2S;
              if (LAST) {  // channels 96 .. 99: rows g < 4
                const double G = gr < 4 ? tanh_f64(z[n][e]) + hrow[gr < 4 ? ca : 0] : 0.;
                dmma8(x[0], x[1], G, rb[n][e]);
              } else {
                const double G0 = tanh_f64(z[n][e]) + hrow[ca];
                const double G1 = tanh_f64(z[n][2 + e]) + hrow[cb];
                dmma16(x, G0, G1, rb[n][e]);
              }
            }
        };
#pragma unroll
        for (int m = 0; m < 6; ++m) tile(std::integral_constant<int, 0>{}, m, X[m]);
        tile(std::integral_constant<int, 1>{}, 6, X[6]);
        __syncwarp();  // rr and hs are rewritten by the next rows
      }
    }
    // xyz / nnei (se_a.py:844), D = xyz^T xyz[:, :ax]
    const double nn = (double)g.nnei;
    double* S = hs;  // [4][100]
    if (t4 < 2)
#pragma unroll
      for (int m = 0; m < 7; ++m) {
        const int c = 16 * m + gr;
        if (c < 100) {
          S[(2 * t4) * 100 + c] = X[m][0] / nn;
          S[(2 * t4 + 1) * 100 + c] = X[m][1] / nn;
        }
        if (m < 6) {
          S[(2 * t4) * 100 + c + 8] = X[m][2] / nn;
          S[(2 * t4 + 1) * 100 + c + 8] = X[m][3] / nn;
        }
      }
    __syncwarp();
    for (int e = lane; e < 400; e += 32) xyz_out[(size_t)row * 400 + e] = S[e];
    double* Dr = D_out + (size_t)g.drow[row] * 100 * g.ax;
    for (int e = lane; e < 100 * g.ax; e += 32) {
      const int c = e / g.ax, k = e - c * g.ax;
      double d = 0.;
#pragma unroll
      for (int a = 0; a < 4; ++a) d = fma(S[a * 100 + c], S[a * 100 + k], d);
      Dr[e] = d;
    }
    __syncwarp();
  }
}

// CTAs [first[t], first[t + 1]) take neighbor type t (types are independent in
// the backward, and one net's fragments fill half of shared memory)
struct EmSplit {
  int first[TR_MAXT + 1];
};

__global__ void __launch_bounds__(32 * EM_BWD_MAXW, 1)
k_emb_bwd_dmma(double* __restrict__ gem, const double* __restrict__ em,
               const double* __restrict__ xbar, TrNet<double> net, TrGeom g, EmSplit split) {
  extern __shared__ __align__(16) double esm[];
  pdl_wait();
  pdl_trigger();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int gr = lane >> 2, t4 = lane & 3;
  int t = 0;
  while (t + 1 < g.ntypes && (int)blockIdx.x >= split.first[t + 1]) ++t;
  em_stage(esm, net, t, true);
  __syncthreads();
  const double* F2 = esm;
  const double* F3 = F2 + EM_F2;
  const double* B3 = F3 + EM_F3;
  const double* B2 = B3 + EM_B3;
  const double* V = B2 + EM_B2;
  double* ws = esm + EM_BWD_T + (size_t)w * EM_BWD_W;
  double* rr = ws;
  double* xs = rr + 64;              // xbar [4][100]
  double* zt = xs + 400;             // [16 rows][EM_TS]: zbar of the current channel tile
  double* yt = zt + 16 * EM_TS;      // its tanh
  int* ent = reinterpret_cast<int*>(esm + EM_BWD_T + (size_t)nw * EM_BWD_W) +
             (size_t)w * (g.nnei + TR_MAXT + 1);
  int* secn = ent + g.nnei;
  const int b0 = blockIdx.x - split.first[t], nb = split.first[t + 1] - split.first[t];
  for (int row = b0 * nw + w; row < g.nrows; row += nb * nw) {
    tr_entries(ent, secn, g.nlist + (size_t)row * g.nnei, g, g.type[row], false, lane, t, t + 1);
    const int total = secn[t + 1];
    if (total == 0) continue;
    for (int e = lane; e < 400; e += 32) xs[e] = xbar[(size_t)row * 400 + e];
    for (int e0 = 0; e0 < total; e0 += 16) {
      const int ne = min(16, total - e0);
      double xa, xb;
      em_rows(rr, xa, xb, ent, e0, ne, em + (size_t)row * g.nnei * 4, false, lane);
      double h1a[EM_S1], h1b[EM_S1], h2[7][4];
      em_layers12<false>(h1a, h1b, h2, xa, xb, F2, V, nullptr, lane);
      // hb2: adjoint of h2 (the layout of h2); the residual's share first:
      // sum_a R[row][a] (xbar[a][c] + xbar[a][c + 50])
      double hb2[7][4];
      const double ra = rr[gr * 4 + t4], rc = rr[(gr + 8) * 4 + t4];
#pragma unroll
      for (int j = 0; j < 7; ++j) {
#pragma unroll
        for (int k = 0; k < 4; ++k) hb2[j][k] = 0.;
        const int c = em_c2(j, gr >> 1, gr & 1);
        dmma16(hb2[j], ra, rc, c >= 0 ? xs[t4 * 100 + c] + xs[t4 * 100 + c + 50] : 0.);
      }
      // dE/dR of rows g, g + 8, columns 2 t, 2 t + 1: sum_c G[c] xbar[a][c], first
      // the residual's share of G
      double part[4] = {0., 0., 0., 0.};
#pragma unroll
      for (int j = 0; j < 7; ++j)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int c = em_c2(j, t4, v);
          dmma16(part, h2[j][v], h2[j][2 + v],
                 gr < 4 && c >= 0 ? xs[gr * 100 + c] + xs[gr * 100 + c + 50] : 0.);
        }
      auto tile = [&](auto last, int m) {
        constexpr int LAST = decltype(last)::value;
        const int c = 16 * m + gr;
        double z[2][4];
        em_layer3<LAST>(z, m, h2, F3, V, lane);
        double gb[2][4];  // gbar = sum_a R[row][a] xbar[a][channel]
        const bool in = !LAST || gr < 4;
        const double x0 = in ? xs[t4 * 100 + c] : 0., x1 = LAST ? 0. : xs[t4 * 100 + c + 8];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
#pragma unroll
          for (int k = 0; k < 4; ++k) gb[n][k] = 0.;
          const double rv = rr[(8 * n + gr) * 4 + t4];
          if (LAST)
            dmma8(gb[n][0], gb[n][1], x0, rv);
          else
            dmma16(gb[n], x0, x1, rv);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int r = 8 * n + 2 * t4 + e;
            if (in) {
              const double y = tanh_f64(z[n][e]);
              zt[r * EM_TS + gr] = gb[n][e] * (1. - y * y);
              yt[r * EM_TS + gr] = y;
            }
            if (!LAST) {
              const double y = tanh_f64(z[n][2 + e]);
              zt[r * EM_TS + gr + 8] = gb[n][2 + e] * (1. - y * y);
              yt[r * EM_TS + gr + 8] = y;
            }
          }
        __syncwarp();
#pragma unroll
        for (int s = 0; s < (LAST ? 1 : 4); ++s) {
          const int k = 4 * s + t4;
          const double a0 = zt[gr * EM_TS + k], a1 = zt[(gr + 8) * EM_TS + k];
          const double* bf = B3 + (size_t)((4 * m + s) * 7) * 32 + lane;
#pragma unroll
          for (int j = 0; j < 7; ++j) dmma16(hb2[j], a0, a1, bf[j * 32]);
          dmma16(part, yt[gr * EM_TS + k], yt[(gr + 8) * EM_TS + k],
                 gr < 4 ? xs[gr * 100 + 16 * m + k] : 0.);
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int m = 0; m < 6; ++m) tile(std::integral_constant<int, 0>{}, m);
      tile(std::integral_constant<int, 1>{}, 6);
      // layer 2 adjoint: zb2 in h2's place, then hb1 at the lane's channels
      double h1b_[8], h1d_[8];  // adjoints of h1, rows g and g + 8
      {
        double hb1[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int k = 0; k < 4; ++k) hb1[q][k] = 0.;
#pragma unroll
        for (int j = 0; j < 7; ++j) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double y = h2[j][k] - (k < 2 ? h1a[j] : h1b[j]);
            h2[j][k] = hb2[j][k] * (1. - y * y);
          }
#pragma unroll
          for (int v = 0; v < 2; ++v)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              dmma16(hb1[q], h2[j][v], h2[j][2 + v], B2[((2 * j + v) * 4 + q) * 32 + lane]);
        }
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          h1b_[s] = hb1[s >> 1][s & 1];
          h1d_[s] = hb1[s >> 1][2 + (s & 1)];
        }
      }
      double pa = 0., pb = 0.;
#pragma unroll
      for (int s = 0; s < EM_S1; ++s) {
        const double w1 = V[4 * s + t4];  // zero in padding
        pa = fma((h1b_[s] + hb2[s][0] + hb2[s][1]) * (1. - h1a[s] * h1a[s]), w1, pa);
        pb = fma((h1d_[s] + hb2[s][2] + hb2[s][3]) * (1. - h1b[s] * h1b[s]), w1, pb);
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        pa += __shfl_xor_sync(0xffffffffu, pa, o);
        pb += __shfl_xor_sync(0xffffffffu, pb, o);
      }
      if (t4 == 0) {
        part[0] += pa;
        part[2] += pb;
      }
      if (t4 < 2) {
        double* out = gem + (size_t)row * g.nnei * 4 + 2 * t4;
        if (gr < ne)
          *reinterpret_cast<double2*>(out + (size_t)(ent[e0 + gr] & 0xFFFF) * 4) =
              make_double2(part[0], part[1]);
        if (gr + 8 < ne)
          *reinterpret_cast<double2*>(out + (size_t)(ent[e0 + gr + 8] & 0xFFFF) * 4) =
              make_double2(part[2], part[3]);
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------- reverse over tangent --
// The weight gradients of J = sum Ebar E + <u, g> (k_tr_rev's) on the matrix
// instructions, FP64 and FP32. The FMA form adds every row group's share of the
// 6,250 weight gradients to shared memory: the atomics and the operand reads
// around them held it at a seventh of the FMA rate. Here the eight warps of a CTA
// take one 16-row tile each, of any atoms, and go through the net in step: layer
// 3 one 16-channel tile at a time, whose adjoints of all 128 rows meet in
// shared memory, and warp w adds their product with the rows' layer-2 outputs
// and tangents for 8 of the 50 units to registers that it keeps to the end.
//
// Shared memory holds one net (so a CTA stays with one neighbor type): W3
// once, rows of 100 with the second pair members 26 rows down, which makes the
// reads as layer-3 and as adjoint operand free of bank conflicts; row 25 is b3
// and meets the constant 1 at position 50 of the layer-2 outputs, which also
// collects the gradient of b3. Position 2 (c % 25) + c / 25 holds unit c.
//
// Tiles are numbered tile-in-atom first, so the empty ones (beyond an atom's
// neighbors) are the last and the rest come out even over the warps.
//
// Measured: FP64, 4 frames of 192 atoms 1666 -> 439 us (FP64 matrix pipe 49 % busy,
// the FMA pipe 10 %, issue slots 18 %); FP32, 16 frames 1584 -> 1033 us (matrix pipe
// 36 %, issue slots 45 %: splitting the operands takes three instructions per
// element). The rest is the latency of two warps per scheduler; the accumulators
// leave room for no more.
constexpr int EM_REV_NW = 8;
// Row strides that keep the operand reads free of (most) bank conflicts for
// 8-byte and 4-byte elements, in elements; W3's rows, staged layer-2 and
// layer-1 vectors. NJ: unit tiles per warp in the W3 gradient. Four-byte
// accumulators leave room for two, each warp then over half of the rows: an
// operand read serves twice as many products.
template <typename T>
struct EmRev {
  static constexpr bool F64 = sizeof(T) == 8;
  static constexpr int S3 = 100, P2S = F64 ? 52 : 56, P1S = F64 ? 28 : 40;
  static constexpr int NJ = F64 ? 1 : 2;
  static constexpr int W3 = 54 * S3 + 4;    // operand elements
  static constexpr int V = 28 + 28 + 52;
  static constexpr int H = 2 * 16 * P2S;    // per warp: layer-2 outputs, tangents
  static constexpr int Z = 2 * 16 * EM_TS;  // layer-3 adjoints of a channel tile
  static constexpr int R = 16 * 8;          // env rows and their tangents
  static constexpr int N = W3 * 8 / (int)sizeof(T) + EM_F2 + EM_B2 + V + EM_REV_NW * (H + Z + R + 56) +
                           EM_REV_NW * 4 / (int)sizeof(T);
};

// An operand element: FP64 as it is, FP32 as two TF32 terms (8 bytes either way).
struct EmTf {
  uint32_t hi, lo;
};
template <typename T>
struct EmOp {
  using type = T;
};
template <>
struct EmOp<float> {
  using type = EmTf;
};
__device__ __forceinline__ double em_op(double x) { return x; }
__device__ __forceinline__ EmTf em_op(float x) {
  EmTf r;
  r.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  r.lo = __float_as_uint(x - __uint_as_float(r.hi));
  return r;
}

// d = A B + c over eight k
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1, float c0, float c1, float c2, float c3) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%10, %11, %12, %13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2),
        "f"(c3));
}

// c += A B over eight k: a0, a1 rows g, g + 8 at k = t, a2, a3 at k = 4 + t, b0, b1
// column g at k = t, 4 + t; the same with rows 0 .. 7 only, and over four k.
__device__ __forceinline__ void em_mma(double (&c)[4], double a0, double a1, double a2, double a3,
                                       double b0, double b1) {
  dmma16(c, a0, a1, b0);
  dmma16(c, a2, a3, b1);
}
__device__ __forceinline__ void em_mma8(double (&c)[4], double a0, double a2, double b0,
                                        double b1) {
  dmma8(c[0], c[1], a0, b0);
  dmma8(c[0], c[1], a2, b1);
}
__device__ __forceinline__ void em_mma_k4(double (&c)[4], double a0, double a1, double b) {
  dmma16(c, a0, a1, b);
}
__device__ __forceinline__ void em_mma8_k4(double (&c)[4], double a, double b) {
  dmma8(c[0], c[1], a, b);
}
// FP32: three products (the fourth is below 2^-23 of the result). The matrix
// instruction truncates what it adds to its accumulator, which shows in sums
// that run on (five times the error of FP32 sums in the first layer's
// gradient): every eight k start from zero, the small products on their own, and
// the rounded FP32 add carries the sum. What each truncation takes off the large
// products, 2.3 to 3.3e-8 of their sum on average (measured over normal and
// one-signed operands; mean 2.7e-8), is given back: left out, every sum came out
// 3e-8 small, xyz' -3.3e-8 and the weight gradients -2.9 to -6.1e-8, and the
// gradients of a training step were 1 to 3 % further from 64 bits than with FP32
// sums. Rounding the lower terms, or the fourth product, changed neither. The
// reverse pass takes 3 % longer.
__device__ __forceinline__ void em_mma(float (&c)[4], EmTf a0, EmTf a1, EmTf a2, EmTf a3, EmTf b0,
                                       EmTf b1) {
  const uint32_t ah[4] = {a0.hi, a1.hi, a2.hi, a3.hi}, al[4] = {a0.lo, a1.lo, a2.lo, a3.lo};
  float d[4], e[4];
  mma_tf32(d, al, b0.hi, b1.hi, 0.f, 0.f, 0.f, 0.f);
  mma_tf32(e, ah, b0.hi, b1.hi, 0.f, 0.f, 0.f, 0.f);
  mma_tf32(d, ah, b0.lo, b1.lo, d[0], d[1], d[2], d[3]);
#pragma unroll
  for (int k = 0; k < 4; k += 2) {
    const float2 ek = make_float2(e[k], e[k + 1]);
    const float2 lost = make_float2(2.7e-8f, 2.7e-8f);
    const float2 v = __fadd2_rn(make_float2(c[k], c[k + 1]),
                                __fadd2_rn(__ffma2_rn(ek, lost, make_float2(d[k], d[k + 1])), ek));
    c[k] = v.x;
    c[k + 1] = v.y;
  }
}
__device__ __forceinline__ void em_mma8(float (&c)[4], EmTf a0, EmTf a2, EmTf b0, EmTf b1) {
  em_mma(c, a0, EmTf{0, 0}, a2, EmTf{0, 0}, b0, b1);
}
__device__ __forceinline__ void em_mma_k4(float (&c)[4], EmTf a0, EmTf a1, EmTf b) {
  em_mma(c, a0, a1, EmTf{0, 0}, EmTf{0, 0}, b, EmTf{0, 0});
}
__device__ __forceinline__ void em_mma8_k4(float (&c)[4], EmTf a, EmTf b) {
  em_mma(c, a, EmTf{0, 0}, EmTf{0, 0}, EmTf{0, 0}, b, EmTf{0, 0});
}
__device__ __forceinline__ double em_tanh(double x) { return tanh_f64(x); }
__device__ __forceinline__ float em_tanh(float x) { return tr_tanh(x); }

template <typename T>
struct EmPair;
template <>
struct EmPair<double> {
  using type = double2;
};
template <>
struct EmPair<float> {
  using type = float2;
};

// W3 (and b3 as row 25) of net t as operands
template <typename T>
__device__ inline void em_stage_w3(typename EmOp<T>::type* W3, const TrNet<T>& net, int t) {
  constexpr int S3 = EmRev<T>::S3;
  for (int e = threadIdx.x; e < EmRev<T>::W3; e += blockDim.x) {
    const int r = e / S3, c = e - r * S3;
    W3[e] = em_op(r < 25    ? net.W[t][2][e]
                  : r == 25 ? net.b[t][2][c]
                  : r < 51  ? net.W[t][2][e - S3]
                            : (T)0);
  }
}

// env rows and tangents of ne entries from e0 on (times the multiplicity) to rr
// [16][8], x and its tangent to this lane's rows g, g + 8
template <typename T>
__device__ __forceinline__ void em_env_rows(T* rr, T& x0, T& x1, T& d0, T& d1, const int* ent,
                                            int e0, int ne, int row, const TrGeom& g, const T* avg,
                                            const T* std_, const double* fbar, const double* vbar,
                                            int lane) {
  const int gr = lane >> 2;
  T x = (T)0, d = (T)0;
  if (lane < 16) {
    T Rv[4] = {(T)0, (T)0, (T)0, (T)0}, Rd[4] = {(T)0, (T)0, (T)0, (T)0}, mu = (T)0;
    if (lane < ne) {
      const TrAtom A = tr_atom(g, row);
      const int en = ent[e0 + lane];
      tr_env_tangent<T>(Rv, Rd, g, A, en & 0xFFFF, avg + (size_t)A.ti * g.nnei * 4,
                        std_ + (size_t)A.ti * g.nnei * 4, fbar, vbar);
      mu = (T)(en >> 16);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      rr[lane * 8 + a] = mu * Rv[a];
      rr[lane * 8 + 4 + a] = mu * Rd[a];
    }
    x = Rv[0];
    d = Rd[0];
  }
  x0 = __shfl_sync(0xffffffffu, x, gr);
  x1 = __shfl_sync(0xffffffffu, x, 8 + gr);
  d0 = __shfl_sync(0xffffffffu, d, gr);
  d1 = __shfl_sync(0xffffffffu, d, 8 + gr);
  __syncwarp();
}

// layer-1 outputs of rows g (ha) and g + 8 (hb) at the lane's channels
template <typename T>
__device__ __forceinline__ void em_layer1(T (&ha)[EM_S1], T (&hb)[EM_S1], T x0, T x1, const T* V,
                                          int t4) {
#pragma unroll
  for (int s = 0; s < EM_S1; ++s) {
    const T w1 = V[4 * s + t4], b1 = V[28 + 4 * s + t4];
    ha[s] = em_pad(s, t4, em_tanh(fma(x0, w1, b1)));
    hb[s] = em_pad(s, t4, em_tanh(fma(x1, w1, b1)));
  }
}

// layers 1 and 2 and their tangents, staged at their positions in hs and hd
template <typename T>
__device__ __forceinline__ void em_layers12_tan(T x0, T x1, T d0, T d1, const T* F2, const T* V,
                                                T* hs, T* hd, int lane) {
  using Op = typename EmOp<T>::type;
  using T2 = typename EmPair<T>::type;
  constexpr int P2S = EmRev<T>::P2S;
  const int gr = lane >> 2, t4 = lane & 3;
  T h1a[EM_S1], h1b[EM_S1], h2[7][4], ht[7][4];
  em_layer1(h1a, h1b, x0, x1, V, t4);
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const bool ok = 4 * j + t4 < 25;
    h2[j][0] = h2[j][2] = ok ? V[56 + 4 * j + t4] : (T)0;
    h2[j][1] = h2[j][3] = ok ? V[56 + 4 * j + t4 + 25] : (T)0;
#pragma unroll
    for (int k = 0; k < 4; ++k) ht[j][k] = (T)0;
  }
#pragma unroll
  for (int s = 0; s < EM_S1; s += 2) {
    Op ha[2], hb[2], ta[2], tb[2];
#pragma unroll
    for (int e = 0; e < 2 && s + e < EM_S1; ++e) {
      const T w1 = V[4 * (s + e) + t4];
      ta[e] = em_op(em_pad(s + e, t4, ((T)1 - h1a[s + e] * h1a[s + e]) * (d0 * w1)));
      tb[e] = em_op(em_pad(s + e, t4, ((T)1 - h1b[s + e] * h1b[s + e]) * (d1 * w1)));
      ha[e] = em_op(h1a[s + e]);
      hb[e] = em_op(h1b[s + e]);
    }
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      const Op b = em_op(F2[(s * 7 + j) * 32 + lane]);
      if (s + 1 < EM_S1) {
        const Op c = em_op(F2[((s + 1) * 7 + j) * 32 + lane]);
        em_mma(h2[j], ha[0], hb[0], ha[1], hb[1], b, c);
        em_mma(ht[j], ta[0], tb[0], ta[1], tb[1], b, c);
      } else {
        em_mma_k4(h2[j], ha[0], hb[0], b);
        em_mma_k4(ht[j], ta[0], tb[0], b);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    const T w1 = V[4 * j + t4];
    const T ta = ((T)1 - h1a[j] * h1a[j]) * (d0 * w1);
    const T tb = ((T)1 - h1b[j] * h1b[j]) * (d1 * w1);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T y = em_tanh(h2[j][k]);
      h2[j][k] = y + (k < 2 ? h1a[j] : h1b[j]);
      ht[j][k] = ((T)1 - y * y) * ht[j][k] + (k < 2 ? ta : tb);
    }
    if (j == 6 && t4 == 1) {  // positions 50 (the constant), 51
      h2[j][0] = h2[j][2] = (T)1;
      h2[j][1] = h2[j][3] = (T)0;
#pragma unroll
      for (int k = 0; k < 4; ++k) ht[j][k] = (T)0;
    }
    if (j < 6 || t4 < 2) {
      const int o = gr * P2S + 8 * j + 2 * t4;
      *reinterpret_cast<T2*>(hs + o) = T2{h2[j][0], h2[j][1]};
      *reinterpret_cast<T2*>(hs + o + 8 * P2S) = T2{h2[j][2], h2[j][3]};
      *reinterpret_cast<T2*>(hd + o) = T2{ht[j][0], ht[j][1]};
      *reinterpret_cast<T2*>(hd + o + 8 * P2S) = T2{ht[j][2], ht[j][3]};
    }
  }
}

// layer 3 (transposed, without its tanh) and its tangent: channels g, g + 8 of the
// tile that W3 points into, rows from hr (the lane's: layer-2 positions 2 t of row g)
template <int LAST, typename T>
__device__ __forceinline__ void em_layer3_tan(T (&z)[4], T (&zt)[4], const T* hr,
                                              const typename EmOp<T>::type* W3, int t4) {
  using Op = typename EmOp<T>::type;
  using T2 = typename EmPair<T>::type;
  constexpr int P2S = EmRev<T>::P2S, S3 = EmRev<T>::S3;
#pragma unroll
  for (int k = 0; k < 4; ++k) z[k] = zt[k] = (T)0;
#pragma unroll
  for (int j = 0; j < 7; ++j) {
    T2 h = *reinterpret_cast<const T2*>(hr + 8 * j);
    T2 q = *reinterpret_cast<const T2*>(hr + 16 * P2S + 8 * j);
    if (j == 6) {  // positions past 50: the next row's
      h.x = t4 < 2 ? h.x : (T)0;
      q.x = t4 < 2 ? q.x : (T)0;
      h.y = t4 < 1 ? h.y : (T)0;
      q.y = t4 < 1 ? q.y : (T)0;
    }
    const Op* a = W3 + 4 * j * S3;
    const Op* b = a + 26 * S3;
    if (LAST) {
      em_mma8(z, a[0], b[0], em_op(h.x), em_op(h.y));
      em_mma8(zt, a[0], b[0], em_op(q.x), em_op(q.y));
    } else {
      const Op a0 = a[0], a1 = a[8], b0 = b[0], b1 = b[8];
      em_mma(z, a0, a1, b0, b1, em_op(h.x), em_op(h.y));
      em_mma(zt, a0, a1, b0, b1, em_op(q.x), em_op(q.y));
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(32 * EM_REV_NW, 1)
k_emb_rev_mma(TrGrad<T> grad, const T* __restrict__ xbar,
               const T* __restrict__ xbard, const T* __restrict__ avg,
               const T* __restrict__ std_, const double* __restrict__ fbar,
               const double* __restrict__ vbar, TrNet<T> net, TrGeom g, EmSplit split) {
  using Ly = EmRev<T>;
  using T2 = typename EmPair<T>::type;
  constexpr int S3 = Ly::S3, P2S = Ly::P2S, P1S = Ly::P1S, NJ = Ly::NJ;
  extern __shared__ __align__(16) double esm[];
  pdl_wait();
  pdl_trigger();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gr = lane >> 2, t4 = lane & 3;
  int t = 0;
  while (t + 1 < g.ntypes && (int)blockIdx.x >= split.first[t + 1]) ++t;
  using Op = typename EmOp<T>::type;
  Op* W3 = reinterpret_cast<Op*>(esm);
  T* F2 = reinterpret_cast<T*>(W3 + Ly::W3);
  T* B2 = F2 + EM_F2;
  T* V = B2 + EM_B2;
  T* H = V + Ly::V;
  T* Z = H + EM_REV_NW * Ly::H;
  T* R = Z + EM_REV_NW * Ly::Z;
  T* G1 = R + EM_REV_NW * Ly::R;
  int* act = reinterpret_cast<int*>(G1 + EM_REV_NW * 56);
  em_stage_w3(W3, net, t);
  em_stage_f2(F2, net.W[t][1]);
  em_stage_b2(B2, net.W[t][1]);
  em_stage_v(V, net, t);
  for (int e = threadIdx.x; e < EM_REV_NW * 56; e += blockDim.x) G1[e] = (T)0;
  T* hs = H + w * Ly::H;
  T* hd = hs + 16 * P2S;
  T* zs = Z + w * Ly::Z;
  T* zd = zs + 16 * EM_TS;
  T* rr = R + w * Ly::R;
  T* g1 = G1 + w * 56;
  int* ent = reinterpret_cast<int*>(zs);  // read before the first adjoints are written
  int* secn = ent + g.nnei;
  T gw3[7][NJ][4], gw2[2][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    gw2[0][k] = gw2[1][k] = (T)0;
#pragma unroll
    for (int m = 0; m < 7; ++m)
#pragma unroll
      for (int n = 0; n < NJ; ++n) gw3[m][n][k] = (T)0;
  }
  const int nb = split.first[t + 1] - split.first[t];
  const long long ntile = (long long)g.nrows * ((g.sec[t + 1] - g.sec[t] + 15) / 16);
  long long idx = (long long)w * nb + (blockIdx.x - split.first[t]);
  bool any = false;
  for (;;) {
    __syncthreads();  // the previous round's last products have read Z
    int ne = 0, e0 = 0, row = 0;
    while (idx < ntile) {
      row = (int)(idx % g.nrows);
      e0 = 16 * (int)(idx / g.nrows);
      idx += (long long)nb * EM_REV_NW;
      tr_entries(ent, secn, g.nlist + (size_t)row * g.nnei, g, g.type[row], true, lane, t, t + 1);
      ne = max(0, min(16, secn[t + 1] - e0));
      if (ne > 0) break;
      __syncwarp();
    }
    if (lane == 0) act[w] = ne > 0;
    if (!__syncthreads_or(ne > 0)) break;
    any = true;
    const T* xb = xbar + (size_t)row * 400;
    const T* xd = xbard + (size_t)row * 400;
    T x0 = (T)0, x1 = (T)0, d0 = (T)0, d1 = (T)0;  // input and tangent of rows g, g + 8
    T hb2[7][4], hbd2[7][4];               // adjoints of layer 2's output and tangent
    if (ne > 0) {
      em_env_rows(rr, x0, x1, d0, d1, ent, e0, ne, row, g, avg, std_, fbar, vbar, lane);
      em_layers12_tan(x0, x1, d0, d1, F2, V, hs, hd, lane);
      // the layer-3 residual's share of the layer-2 adjoints
      const Op ra = em_op(rr[gr * 8 + t4]), rb = em_op(rr[(gr + 8) * 8 + t4]);
      const Op qa = em_op(rr[gr * 8 + 4 + t4]), qb = em_op(rr[(gr + 8) * 8 + 4 + t4]);
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        const int c = em_c2(j, gr >> 1, gr & 1), o = t4 * 100 + (c < 0 ? 0 : c);
        const Op u = em_op(c < 0 ? (T)0 : xb[o] + xb[o + 50]);
        const Op v = em_op(c < 0 ? (T)0 : xd[o] + xd[o + 50]);
#pragma unroll
        for (int k = 0; k < 4; ++k) hb2[j][k] = hbd2[j][k] = (T)0;
        em_mma(hb2[j], ra, rb, qa, qb, u, v);
        em_mma_k4(hbd2[j], ra, rb, v);
      }
      __syncwarp();
    }
    auto tile = [&](auto last, int m) {
      constexpr int LAST = decltype(last)::value;
      if (ne > 0) {
        const int c = 16 * m + gr;
        const bool in = !LAST || gr < 4;
        const int o = t4 * 100 + c;
        const Op xb0 = em_op(in ? xb[o] : (T)0), xb1 = em_op(LAST ? (T)0 : xb[o + 8]);
        const Op xd0 = em_op(in ? xd[o] : (T)0), xd1 = em_op(LAST ? (T)0 : xd[o + 8]);
#pragma unroll 1
        for (int n = 0; n < 2; ++n) {
          T z[4], zt[4];
          em_layer3_tan<LAST>(z, zt, hs + (8 * n + gr) * P2S + 2 * t4, W3 + t4 * S3 + c, t4);
          T gb[4] = {(T)0, (T)0, (T)0, (T)0}, gd[4] = {(T)0, (T)0, (T)0, (T)0};
          const Op rv = em_op(rr[(8 * n + gr) * 8 + t4]);
          const Op rd = em_op(rr[(8 * n + gr) * 8 + 4 + t4]);
          if (LAST) {
            em_mma8(gb, xb0, xd0, rv, rd);
            em_mma8_k4(gd, xd0, rv);
          } else {
            em_mma(gb, xb0, xb1, xd0, xd1, rv, rd);
            em_mma_k4(gd, xd0, xd1, rv);
          }
#pragma unroll
          for (int k = 0; k < (LAST ? 2 : 4); ++k)
            if (in) {
              const T y = em_tanh(z[k]), q = (T)1 - y * y;
              const int p = (8 * n + 2 * t4 + (k & 1)) * EM_TS + gr + 8 * (k >> 1);
              zs[p] = (gb[k] - (T)2 * y * zt[k] * gd[k]) * q;
              zd[p] = gd[k] * q;
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int s = 0; s < (LAST ? 1 : 2); ++s) {
          const int k = 8 * s + t4;
          const T *zp = zs + gr * EM_TS + k, *dp = zd + gr * EM_TS + k;
          const Op* bp = W3 + ((gr >> 1) + 26 * (gr & 1)) * S3 + 16 * m + k;
          const Op a0 = em_op(zp[0]), a1 = em_op(zp[8 * EM_TS]);
          const Op b0 = em_op(dp[0]), b1 = em_op(dp[8 * EM_TS]);
          if (LAST) {  // four channels
#pragma unroll
            for (int j = 0; j < 7; ++j) {
              em_mma_k4(hb2[j], a0, a1, bp[4 * S3 * j]);
              em_mma_k4(hbd2[j], b0, b1, bp[4 * S3 * j]);
            }
          } else {
            const Op a2 = em_op(zp[4]), a3 = em_op(zp[8 * EM_TS + 4]);
            const Op b2 = em_op(dp[4]), b3 = em_op(dp[8 * EM_TS + 4]);
#pragma unroll
            for (int j = 0; j < 7; ++j) {
              const Op c0 = bp[4 * S3 * j], c1 = bp[4 * S3 * j + 4];
              em_mma(hb2[j], a0, a1, a2, a3, c0, c1);
              em_mma(hbd2[j], b0, b1, b2, b3, c0, c1);
            }
          }
        }
      }
      __syncthreads();
      // W3 gradient of this tile's channels, units at positions 8 jt .. (+ 8)
      if (NJ == 2 || w < 7) {
        const int jt = NJ == 2 ? 2 * (w & 3) : w, v0 = NJ == 2 ? 4 * (w >> 2) : 0;
        T c[2][NJ][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int n = 0; n < NJ; ++n) c[0][n][k] = c[1][n][k] = (T)0;
#pragma unroll 1
        for (int v = v0; v < (NJ == 2 ? v0 + 4 : EM_REV_NW); ++v) {
          if (!act[v]) continue;
          const T* zp = Z + v * Ly::Z + t4 * EM_TS + gr;
          const T* hp = H + v * Ly::H + t4 * P2S + 8 * jt + gr;
#pragma unroll
          for (int s = 0; s < 4; ++s) {  // two steps of outputs, two of tangents
            const T *zq = zp + 8 * s * EM_TS, *zr = zq + 4 * EM_TS;
            const T *hq = hp + 8 * s * P2S, *hr = hq + 4 * P2S;
            if (LAST) {
              const Op a0 = em_op(zq[0]), a2 = em_op(zr[0]);
#pragma unroll
              for (int n = 0; n < NJ; ++n)
                em_mma8(c[s & 1][n], a0, a2, em_op(hq[8 * n]), em_op(hr[8 * n]));
            } else {
              const Op a0 = em_op(zq[0]), a1 = em_op(zq[8]), a2 = em_op(zr[0]), a3 = em_op(zr[8]);
#pragma unroll
              for (int n = 0; n < NJ; ++n)
                em_mma(c[s & 1][n], a0, a1, a2, a3, em_op(hq[8 * n]), em_op(hr[8 * n]));
            }
          }
        }
#pragma unroll
        for (int q = 0; q < 7; ++q)
          if (q == m)
#pragma unroll
            for (int n = 0; n < NJ; ++n)
#pragma unroll
              for (int k = 0; k < 4; ++k) gw3[q][n][k] += c[0][n][k] + c[1][n][k];
      }
      __syncthreads();
    };
#pragma unroll 1
    for (int m = 0; m < 6; ++m) tile(std::integral_constant<int, 0>{}, m);
    tile(std::integral_constant<int, 1>{}, 6);
    // layer 2's pre-activation adjoints take the place of its outputs and tangents
    T h1a[EM_S1], h1b[EM_S1];
    if (ne > 0) {
      em_layer1(h1a, h1b, x0, x1, V, t4);
      T u[4][4], v[4][4];  // layer 1's: channel 4 s + t of row g at [s / 2][s % 2]
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        u[j >> 1][j & 1] = hb2[j][0] + hb2[j][1];
        u[j >> 1][2 + (j & 1)] = hb2[j][2] + hb2[j][3];
        v[j >> 1][j & 1] = hbd2[j][0] + hbd2[j][1];
        v[j >> 1][2 + (j & 1)] = hbd2[j][2] + hbd2[j][3];
        if (j == 6 && t4 > 0) continue;
        const T w1 = V[4 * j + t4];
        T* ho = hs + gr * P2S + 8 * j + 2 * t4;
        T* po = hd + gr * P2S + 8 * j + 2 * t4;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int o = (k >> 1) * 8 * P2S + (k & 1);
          const T h = k < 2 ? h1a[j] : h1b[j];
          const T y = ho[o] - h, q = (T)1 - y * y;
          const T yt = po[o] - ((T)1 - h * h) * ((k < 2 ? d0 : d1) * w1);  // q times zdot
          ho[o] = hb2[j][k] * q - (T)2 * y * yt * hbd2[j][k];
          po[o] = hbd2[j][k] * q;
        }
      }
      u[3][1] = u[3][3] = v[3][1] = v[3][3] = (T)0;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 7; ++j) {
        const int o = gr * P2S + 8 * j + 2 * t4;
        const bool ok = j < 6 || t4 == 0;
        const T2 zero = T2{(T)0, (T)0};
        const T2 a0 = ok ? *reinterpret_cast<const T2*>(hs + o) : zero;
        const T2 a1 = ok ? *reinterpret_cast<const T2*>(hs + o + 8 * P2S) : zero;
        const T2 b0 = ok ? *reinterpret_cast<const T2*>(hd + o) : zero;
        const T2 b1 = ok ? *reinterpret_cast<const T2*>(hd + o + 8 * P2S) : zero;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const Op c0 = em_op(B2[((2 * j) * 4 + q) * 32 + lane]);
          const Op c1 = em_op(B2[((2 * j + 1) * 4 + q) * 32 + lane]);
          em_mma(u[q], em_op(a0.x), em_op(a1.x), em_op(a0.y), em_op(a1.y), c0, c1);
          em_mma(v[q], em_op(b0.x), em_op(b1.x), em_op(b0.y), em_op(b1.y), c0, c1);
        }
      }
#pragma unroll
      for (int s = 0; s < EM_S1; ++s) {
        const T w1 = V[4 * s + t4];
        const T qa = (T)1 - h1a[s] * h1a[s], qb = (T)1 - h1b[s] * h1b[s];
        const T ta = v[s >> 1][s & 1], tb = v[s >> 1][2 + (s & 1)];
        const T za = (u[s >> 1][s & 1] - (T)2 * h1a[s] * (d0 * w1) * ta) * qa;
        const T zb = (u[s >> 1][2 + (s & 1)] - (T)2 * h1b[s] * (d1 * w1) * tb) * qb;
        T gws = fma(x0, za, fma(d0, ta * qa, fma(x1, zb, d1 * (tb * qb)))), gbs = za + zb;
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          gws += __shfl_xor_sync(0xffffffffu, gws, o);
          gbs += __shfl_xor_sync(0xffffffffu, gbs, o);
        }
        if (gr == 0) {
          g1[4 * s + t4] += gws;
          g1[28 + 4 * s + t4] += gbs;
        }
      }
    }
    // W2 gradient: positions 16 (w / 2) .. of layer 2, channels 16 (w % 2) .. of
    // layer 1, whose outputs (and the constant 1 as channel 25, for b2), then
    // tangents, take the place of Z
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      if (half) __syncthreads();
      if (ne > 0) {
        T* p = Z + (w * 16 + gr) * P1S + t4;
#pragma unroll
        for (int s = 0; s < EM_S1; ++s) {
          const bool one = s == 6 && t4 == 1;
          const T w1 = V[4 * s + t4];
          p[4 * s] = half ? ((T)1 - h1a[s] * h1a[s]) * (d0 * w1) : one ? (T)1 : h1a[s];
          p[8 * P1S + 4 * s] = half ? ((T)1 - h1b[s] * h1b[s]) * (d1 * w1) : one ? (T)1 : h1b[s];
        }
      }
      __syncthreads();
      T c2[2][4];  // this half's sum: short chains
#pragma unroll
      for (int k = 0; k < 4; ++k) c2[0][k] = c2[1][k] = (T)0;
#pragma unroll 1
      for (int v = 0; v < EM_REV_NW; ++v) {
        if (!act[v]) continue;
        const T* ap = H + v * Ly::H + half * 16 * P2S + t4 * P2S + 16 * (w >> 1) + gr;
        const T* bp = Z + (v * 16 + t4) * P1S + 16 * (w & 1) + gr;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const T *aq = ap + 8 * s * P2S, *ar = aq + 4 * P2S;
          const T *bq = bp + 8 * s * P1S, *br = bq + 4 * P1S;
          const Op a0 = em_op(aq[0]), a1 = em_op(aq[8]), a2 = em_op(ar[0]), a3 = em_op(ar[8]);
          em_mma(c2[0], a0, a1, a2, a3, em_op(bq[0]), em_op(br[0]));
          em_mma(c2[1], a0, a1, a2, a3, em_op(bq[8]), em_op(br[8]));
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        gw2[0][k] += c2[0][k];
        gw2[1][k] += c2[1][k];
      }
    }
  }
  if (!any) return;
  if (NJ == 2 || w < 7)
#pragma unroll
    for (int m = 0; m < 7; ++m)
#pragma unroll
      for (int n = 0; n < NJ; ++n)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int c = 16 * m + gr + 8 * (k >> 1);
          const int p = 8 * (NJ == 2 ? 2 * (w & 3) + n : w) + 2 * t4 + (k & 1);
          if (c >= 100 || p > 50) continue;
          atomicAdd(p == 50 ? grad.b[t][2] + c
                            : grad.W[t][2] + ((p >> 1) + 25 * (p & 1)) * 100 + c,
                    gw3[m][n][k]);
        }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int p = 16 * (w >> 1) + gr + 8 * (k >> 1);
      const int i = 16 * (w & 1) + 8 * n + 2 * t4 + (k & 1);
      if (p >= 50 || i > 25) continue;
      const int c = (p >> 1) + 25 * (p & 1);
      atomicAdd(i == 25 ? grad.b[t][1] + c : grad.W[t][1] + i * 50 + c, gw2[n][k]);
    }
  for (int e = threadIdx.x; e < 56; e += blockDim.x) {
    const int i = e % 28;
    if (i >= 25) continue;
    T s = (T)0;
    for (int v = 0; v < EM_REV_NW; ++v) s += G1[v * 56 + e];
    atomicAdd((e < 28 ? grad.W[t][0] : grad.b[t][0]) + i, s);
  }
}

// --------------------------------------------------------------- tangent --
// xyz' and D' along u (k_tr_tan's) with the same products: a warp takes the
// neighbors of one type of an atom, 16 rows at a time, and adds its share of
// sum R' G + R G' to xyz' (cleared before; a launch takes two types, or one that
// adds to earlier ones, so the sum does not depend on the order). Nothing waits, so
// as many warps as fit: 12.
// Measured: FP64, 4 frames of 192 atoms 417 -> 182 us; FP32, 16 frames 404 -> 334.
constexpr int EM_TAN_NW = 12;
template <typename T>
constexpr int EM_TAN_N = EmRev<T>::W3 * 8 / (int)sizeof(T) + EM_F2 + EmRev<T>::V +
                         EM_TAN_NW * (EmRev<T>::H + EmRev<T>::R);

template <typename T>
__global__ void __launch_bounds__(32 * EM_TAN_NW, 1)
k_emb_tan_mma(T* __restrict__ xyz_t, const T* __restrict__ avg, const T* __restrict__ std_,
              const double* __restrict__ fbar, const double* __restrict__ vbar, TrNet<T> net,
              TrGeom g, EmSplit split) {
  using Ly = EmRev<T>;
  using Op = typename EmOp<T>::type;
  constexpr int S3 = Ly::S3, P2S = Ly::P2S;
  extern __shared__ __align__(16) double esm[];
  pdl_wait();
  pdl_trigger();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gr = lane >> 2, t4 = lane & 3;
  int t = 0;
  while (t + 1 < g.ntypes && (int)blockIdx.x >= split.first[t + 1]) ++t;
  Op* W3 = reinterpret_cast<Op*>(esm);
  T* F2 = reinterpret_cast<T*>(W3 + Ly::W3);
  T* V = F2 + EM_F2;
  T* hs = V + Ly::V + w * (Ly::H + Ly::R);
  T* hd = hs + 16 * P2S;
  T* rr = hs + Ly::H;
  em_stage_w3(W3, net, t);
  em_stage_f2(F2, net.W[t][1]);
  em_stage_v(V, net, t);
  __syncthreads();
  int* ent = reinterpret_cast<int*>(hs);  // rewritten for every tile: hs takes its place
  int* secn = ent + g.nnei;
  const int nb = split.first[t + 1] - split.first[t];
  for (int row = w * nb + (blockIdx.x - split.first[t]); row < g.nrows; row += nb * EM_TAN_NW) {
    const int* nl = g.nlist + (size_t)row * g.nnei;
    T X[7][4];  // channels 16 m + g (+ 8), env columns 2 t, 2 t + 1 (t < 2)
#pragma unroll
    for (int m = 0; m < 7; ++m)
#pragma unroll
      for (int k = 0; k < 4; ++k) X[m][k] = (T)0;
    int total = 1;
    for (int e0 = 0; e0 < total; e0 += 16) {
      tr_entries(ent, secn, nl, g, g.type[row], false, lane, t, t + 1);
      total = secn[t + 1];
      if (total == 0) break;
      T x0, x1, d0, d1;
      em_env_rows(rr, x0, x1, d0, d1, ent, e0, min(16, total - e0), row, g, avg, std_, fbar, vbar,
                  lane);
      em_layers12_tan(x0, x1, d0, d1, F2, V, hs, hd, lane);
      __syncwarp();
      auto tile = [&](auto last, int m, T (&x)[4]) {
        constexpr int LAST = decltype(last)::value;
        const int c = 16 * m + gr;
        const int ua = c < 50 ? c : LAST && gr >= 4 ? 0 : c - 50, ub = c + 8 < 50 ? c + 8 : c - 42;
        const int pa = ua < 25 ? 2 * ua : 2 * ua - 49, pb = ub < 25 ? 2 * ub : 2 * ub - 49;
#pragma unroll 1
        for (int n = 0; n < 2; ++n) {
          T z[4], zt[4];
          em_layer3_tan<LAST>(z, zt, hs + (8 * n + gr) * P2S + 2 * t4, W3 + t4 * S3 + c, t4);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int r = 8 * n + 2 * t4 + e;
            const Op rb = em_op(gr < 4 ? rr[r * 8 + gr] : (T)0);
            const Op rd = em_op(gr < 4 ? rr[r * 8 + 4 + gr] : (T)0);
            const T ya = em_tanh(z[e]);
            const T Ga = ya + hs[r * P2S + pa];
            const T Da = ((T)1 - ya * ya) * zt[e] + hd[r * P2S + pa];
            if (LAST) {
              em_mma8(x, em_op(gr < 4 ? Ga : (T)0), em_op(gr < 4 ? Da : (T)0), rd, rb);
            } else {
              const T yb = em_tanh(z[2 + e]);
              const T Gb = yb + hs[r * P2S + pb];
              const T Db = ((T)1 - yb * yb) * zt[2 + e] + hd[r * P2S + pb];
              em_mma(x, em_op(Ga), em_op(Gb), em_op(Da), em_op(Db), rd, rb);
            }
          }
        }
      };
#pragma unroll
      for (int m = 0; m < 6; ++m) tile(std::integral_constant<int, 0>{}, m, X[m]);
      tile(std::integral_constant<int, 1>{}, 6, X[6]);
      __syncwarp();  // hs and rr are rewritten by the next rows
    }
    if (total == 0 || t4 >= 2) continue;
    T* out = xyz_t + (size_t)row * 400 + 200 * t4 + gr;
#pragma unroll
    for (int m = 0; m < 7; ++m)
#pragma unroll
      for (int k = 0; k < (m == 6 ? 2 : 4); ++k)
        if (m < 6 || gr < 4) atomicAdd(out + 100 * (k & 1) + 16 * m + 8 * (k >> 1), X[m][k]);
  }
}

// xyz' / nnei, D' = xyz'^T xyz[:, :ax] + xyz^T xyz'[:, :ax]: a warp per atom
template <typename T>
__global__ void __launch_bounds__(128)
k_emb_tan_out(T* __restrict__ xyz_t, T* __restrict__ D_t, const T* __restrict__ xyz, TrGeom g) {
  __shared__ T sm[4][800];
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= g.nrows) return;
  T *X = sm[threadIdx.x >> 5], *Xd = X + 400;
  const T nn = (T)g.nnei;
  for (int e = lane; e < 400; e += 32) {
    X[e] = xyz[(size_t)row * 400 + e];
    Xd[e] = xyz_t[(size_t)row * 400 + e] / nn;
    xyz_t[(size_t)row * 400 + e] = Xd[e];
  }
  __syncwarp();
  T* Dr = D_t + (size_t)g.drow[row] * 100 * g.ax;
  for (int e = lane; e < 100 * g.ax; e += 32) {
    const int c = e / g.ax, k = e - c * g.ax;
    T d = (T)0;
#pragma unroll
    for (int a = 0; a < 4; ++a)
      d = fma(Xd[a * 100 + c], X[a * 100 + k], fma(X[a * 100 + c], Xd[a * 100 + k], d));
    Dr[e] = d;
  }
}

// most warps per CTA whose rows come out even: the smallest
// ceil(rows / (blocks * n)) * n, within shared memory
static int em_warps(int rows, int blocks, int maxw, size_t base, size_t per_warp) {
  int best = 0;
  long long cost = 0;
  for (int n = maxw; n >= 4; --n) {
    if (base + per_warp * n > 227 * 1024) continue;
    const long long c = (long long)ceil_div(rows, (long long)blocks * n) * n;
    if (best == 0 || c < cost) best = n, cost = c;
  }
  return best;
}

// The passes on the FP64 matrix instructions, for the standard net, 16-byte
// aligned env rows and at most three types (their fragments must fit in shared
// memory). em_try_* return -1 when the general kernels have to run.
static bool em_takes(const TrNet<double>& net, const TrGeom& g, const double* em,
                     const double* gem) {
  return net.n1 == 25 && net.n2 == 50 && net.n3 == 100 && g.ntypes <= 3 &&
         ((reinterpret_cast<uintptr_t>(em) | reinterpret_cast<uintptr_t>(gem)) & 15) == 0;
}

static int em_fwd(double* xyz, double* D, const double* em, const TrNet<double>& net,
                  const TrGeom& g, cudaStream_t st) {
  const size_t base = (size_t)g.ntypes * EM_FWD_T * 8;
  const size_t per = EM_FWD_W * 8 + (size_t)(g.nnei + TR_MAXT + 1) * 4;
  const int nw = em_warps(g.nrows, sm_count(), EM_FWD_MAXW, base, per);
  if (nw == 0) return -1;
  const size_t smem = base + per * nw;
  DPB_CUDA(cudaFuncSetAttribute(k_emb_fwd_dmma, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem),
           "se_a_train_fwd");
  const int grid = std::min(sm_count(), ceil_div(g.nrows, nw));
  DPB_CUDA(launch_pdl(k_emb_fwd_dmma, dim3(grid), dim3(32 * nw), smem, st, xyz, D, em, net, g),
           "se_a_train_fwd");
  return DPB_OK;
}

// CTAs per type of t0 .. t1 - 1 in proportion to its slots
static EmSplit em_split(const TrGeom& g, int& sms, int& used, int t0, int t1) {
  EmSplit sp{};
  sms = std::max(sm_count(), t1 - t0);
  used = 0;
  const int slots = std::max(1, g.sec[t1] - g.sec[t0]);
  for (int t = 0; t < g.ntypes; ++t) {
    sp.first[t] = used;
    if (t < t0 || t >= t1) continue;
    const int left = t1 - 1 - t;
    int n = (int)((long long)sms * (g.sec[t + 1] - g.sec[t]) / slots);
    n = t + 1 == t1 ? sms - used : std::max(1, std::min(n, sms - used - left));
    used += n;
  }
  sp.first[g.ntypes] = used;
  return sp;
}

static int em_bwd(double* gem, const double* em, const double* xbar, const TrNet<double>& net,
                  const TrGeom& g, cudaStream_t st) {
  int sms, used;
  const EmSplit sp = em_split(g, sms, used, 0, g.ntypes);
  const size_t base = (size_t)EM_BWD_T * 8;
  const size_t per = EM_BWD_W * 8 + (size_t)(g.nnei + TR_MAXT + 1) * 4;
  const int nw = em_warps(g.nrows, std::max(1, sms / g.ntypes), EM_BWD_MAXW, base, per);
  if (nw == 0) return -1;
  const size_t smem = base + per * nw;
  DPB_CUDA(cudaFuncSetAttribute(k_emb_bwd_dmma, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem),
           "se_a_train_bwd");
  DPB_CUDA(launch_pdl(k_emb_bwd_dmma, dim3(used), dim3(32 * nw), smem, st, gem, em, xbar, net, g,
                      sp),
           "se_a_train_bwd");
  return DPB_OK;
}

template <typename T>
static int em_rev(const TrGrad<T>& gr, const T* xb, const T* xbd, const T* avg, const T* std_,
                  const double* fbar, const double* vbar, const TrNet<T>& net, const TrGeom& g,
                  cudaStream_t st) {
  int sms, used;
  const EmSplit sp = em_split(g, sms, used, 0, g.ntypes);
  const size_t smem = (size_t)EmRev<T>::N * sizeof(T);
  auto kern = k_emb_rev_mma<T>;
  DPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
           "se_a_train_rev");
  DPB_CUDA(launch_pdl(kern, dim3(used), dim3(32 * EM_REV_NW), smem, st, gr, xb, xbd, avg, std_,
                      fbar, vbar, net, g, sp),
           "se_a_train_rev");
  return DPB_OK;
}

template <typename T>
static int em_try_fwd(T* xyz, T* D, const T* em, const TrNet<T>& net, const TrGeom& g,
                      cudaStream_t st) {
  if constexpr (std::is_same_v<T, double>)
    if (em_takes(net, g, em, nullptr)) return em_fwd(xyz, D, em, net, g, st);
  return -1;
}

template <typename T>
static int em_try_bwd(T* gem, const T* em, const T* xbar, const TrNet<T>& net, const TrGeom& g,
                      cudaStream_t st) {
  if constexpr (std::is_same_v<T, double>)
    if (em_takes(net, g, em, gem)) return em_bwd(gem, em, xbar, net, g, st);
  return -1;
}

// The tangent and the reverse pass keep one net per CTA, so any number of types;
// the entry list of an atom lies where a tile's layer outputs (adjoints) go later.
template <typename T>
static int em_try_tan(T* xyz_t, T* D_t, const T* xyz, const T* avg, const T* std_,
                      const double* fbar, const double* vbar, const TrNet<T>& net, const TrGeom& g,
                      cudaStream_t st) {
  static_assert((BT_NMAX + TR_MAXT + 1) * 4 <= EmRev<T>::H * (int)sizeof(T), "entry list");
  if (net.n1 != 25 || net.n2 != 50 || net.n3 != 100) return -1;
  const size_t smem = (size_t)EM_TAN_N<T> * sizeof(T);
  auto kern = k_emb_tan_mma<T>;
  DPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
           "se_a_train_tan");
  DPB_CUDA(cudaMemsetAsync(xyz_t, 0, (size_t)g.nrows * 400 * sizeof(T), st), "se_a_train_tan");
  // two types at a time, whose shares add up to the same in either order; every
  // further type by itself, after them
  for (int t0 = 0, t1; t0 < g.ntypes; t0 = t1) {
    t1 = std::min(g.ntypes, t0 == 0 ? 2 : t0 + 1);
    if (g.sec[t1] == g.sec[t0]) continue;
    int sms, used;
    const EmSplit sp = em_split(g, sms, used, t0, t1);
    DPB_CUDA(launch_pdl(kern, dim3(used), dim3(32 * EM_TAN_NW), smem, st, xyz_t, avg, std_, fbar,
                        vbar, net, g, sp),
             "se_a_train_tan");
  }
  DPB_CUDA(launch_pdl(k_emb_tan_out<T>, dim3(ceil_div(g.nrows, 4)), dim3(128), 0, st, xyz_t, D_t,
                      xyz, g),
           "se_a_train_tan");
  return DPB_OK;
}

template <typename T>
static int em_try_rev(const TrGrad<T>& gr, const T* xb, const T* xbd, const T* avg, const T* std_,
                      const double* fbar, const double* vbar, const TrNet<T>& net, const TrGeom& g,
                      cudaStream_t st) {
  static_assert((BT_NMAX + TR_MAXT + 1) * 4 <= EmRev<T>::Z * (int)sizeof(T), "entry list");
  if (net.n1 == 25 && net.n2 == 50 && net.n3 == 100)
    return em_rev<T>(gr, xb, xbd, avg, std_, fbar, vbar, net, g, st);
  return -1;
}

}  // namespace dpb
