// Compressed se_a embedding: the quintic table G_m(x) fused with the
// contraction over neighbors (tabulate_fusion_se_a and its two gradients).
//
// Layout: one warp per (center atom, block of 64 embedding channels; 32 of narrow
// nets, whose half-empty block would cost as much as a full one). The reference's table row holds a channel's six coefficients side by side; read
// per channel (24 or 48 bytes per lane) every line of the row went through L1
// three times, and one warp per atom left small systems waiting on each row.
// Here a row is read as it lies, 16 bytes per lane, and a lane works on
// coefficient pairs: pair q of the row belongs to channel q / 3 and powers
// 2 (q % 3), + 1, so its term is a.x t^k + a.y t^(k + 1), summed over slots per
// pair and over a channel's three pairs once at the end (forward), or multiplied
// by the channel's gradient at once (backward). Slots are located 32 at a time,
// one per lane, and the next slot's row is in flight while one is summed.
// Measured, 92 slots, M = 100, FP32: forward 192 atoms 94 -> 22 us, 12,288 atoms
// 317 -> 232 us (now L1 at 80 % and FP32 issue at 65 %), grad_grad 96 -> 23 and 338
// -> 316 us, gradient 101 -> 31 us at 192 atoms (k_tab_grad below; many
// atoms stay on k_tab_grad_channels, and some widths' grad_grad on
// k_tab_gg_channels).
//
// Semantics follow the CPU reference (source/lib/src/tabulate.cc): locate_xx
// (:45-73) with the nextafter upper bound (:21-30), linear extrapolation
// outside the table (:133-144), and the sorted-padding fold (:184-189): the
// first slot whose em_x equals the last slot's and whose em[1..3] are zero is
// weighted by (nnei - slot) and ends the loop.
#include <math.h>

#include "dpb_common.cuh"

namespace dpb {

template <typename T>
struct TabInfo {
  T lower, upper, max, s0, s1;
  int first;     // int((upper - lower) / stride0)
  int high_idx;  // locate_high_tail_xx
};

template <typename T>
static int make_info(TabInfo<T>& t, const T* info, int M) {
  if (info == nullptr) {
    set_error("table_info is required (host pointer, 6 values)");
    return DPB_ERR_INVALID;
  }
  if (M <= 0 || M > 1024) {
    set_error("last_layer_size must be between 1 and 1024 for GPU tabulation, but got %d", M);
    return DPB_ERR_INVALID;
  }
  t.lower = info[0];
  t.upper = info[1];
  t.max = info[2];
  t.s0 = info[3];
  t.s1 = info[4];
  t.first = (int)((t.upper - t.lower) / t.s0);
  T bxx = (sizeof(T) == 8) ? (T)nextafter((double)t.max, (double)t.lower)
                           : (T)nextafterf((float)t.max, (float)t.lower);
  t.high_idx = t.first + (int)((bxx - t.upper) / t.s1);
  return DPB_OK;
}

template <typename T>
__device__ __forceinline__ void locate(const TabInfo<T>& t, T x, int& idx, T& xx,
                                       T& delta) {
  delta = (T)0.;
  if (x < t.lower) {
    idx = 0;
    xx = (T)0.;
    delta = x - t.lower;
  } else if (x < t.upper) {
    idx = (int)((x - t.lower) / t.s0);
    xx = x - ((T)idx * t.s0 + t.lower);
  } else if (x < t.max) {
    idx = t.first + (int)((x - t.upper) / t.s1);
    xx = x - ((T)(idx - t.first) * t.s1 + t.upper);
  } else {
    idx = t.high_idx;
    xx = t.max - ((T)(idx - t.first) * t.s1 + t.upper);
    delta = x - t.max;
  }
}

// First slot of the sorted padding tail, or nnei when there is none.
template <typename T>
__device__ __forceinline__ int fold_start(const T* em_x, const T* em, int nnei, int lane) {
  const T last = em_x[nnei - 1];
  for (int base = 0; base < nnei; base += 32) {
    int jj = base + lane;
    bool c = false;
    if (jj < nnei) {
      const T* e = em + (size_t)jj * 4;
      c = em_x[jj] == last && e[1] == (T)0. && e[2] == (T)0. && e[3] == (T)0.;
    }
    unsigned b = __ballot_sync(0xffffffffu, c);
    if (b) return base + __ffs(b) - 1;
  }
  return nnei;
}

template <typename T>
struct Coef {
  T a0, a1, a2, a3, a4, a5;
};

__device__ __forceinline__ Coef<float> load_coef(const float* p) {
  const float2* q = reinterpret_cast<const float2*>(p);
  float2 x = __ldg(q), y = __ldg(q + 1), z = __ldg(q + 2);
  return {x.x, x.y, y.x, y.y, z.x, z.y};
}
__device__ __forceinline__ Coef<double> load_coef(const double* p) {
  const double2* q = reinterpret_cast<const double2*>(p);
  double2 x = __ldg(q), y = __ldg(q + 1), z = __ldg(q + 2);
  return {x.x, x.y, y.x, y.y, z.x, z.y};
}

// value (with extrapolation) and derivative of the quintic (tabulate.cc:116-144)
template <typename T>
__device__ __forceinline__ void poly(const Coef<T>& a, T xx, T delta, T& v, T& g) {
  g = a.a1 + ((T)2. * a.a2 + ((T)3. * a.a3 + ((T)4. * a.a4 + (T)5. * a.a5 * xx) * xx) * xx) * xx;
  v = a.a0 + (a.a1 + (a.a2 + (a.a3 + (a.a4 + a.a5 * xx) * xx) * xx) * xx) * xx;
  v = v + g * delta;
}

constexpr int TW = 4;     // warps per block
constexpr int TS = 12;    // staged values per slot: six weights of the value, six of
                          // the slope

template <typename T>
struct Pair;
template <>
struct Pair<float> {
  using type = float2;
};
template <>
struct Pair<double> {
  using type = double2;
};

// The pairs a lane owns. VW = 4: FP32 rows read as float4 (M even and the table
// 16-byte aligned), two neighboring pairs per load; VW = 2: one pair per load
// (float2 or double2).
template <int VW>
__device__ __forceinline__ int pair_index(int p, int lane) {
  return VW == 4 ? 2 * (lane + 32 * (p >> 1)) + (p & 1) : lane + 32 * p;
}
// acc[0..3] += u e[0..3]; FP32 two at a time
__device__ __forceinline__ void axpy4(float (&acc)[4], float u, const float (&e)[4]) {
  const float2 uu = make_float2(u, u);
  const float2 lo = __ffma2_rn(uu, make_float2(e[0], e[1]), make_float2(acc[0], acc[1]));
  const float2 hi = __ffma2_rn(uu, make_float2(e[2], e[3]), make_float2(acc[2], acc[3]));
  acc[0] = lo.x, acc[1] = lo.y, acc[2] = hi.x, acc[3] = hi.y;
}
__device__ __forceinline__ void axpy4(double (&acc)[4], double u, const double (&e)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) acc[k] = fma(u, e[k], acc[k]);
}

// four consecutive staged values (16-byte aligned)
template <typename T>
__device__ __forceinline__ void load4(T (&v)[4], const T* p) {
  using T2 = typename Pair<T>::type;
  if constexpr (sizeof(T) == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else {
    const T2 a = reinterpret_cast<const T2*>(p)[0], b = reinterpret_cast<const T2*>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  }
}

// which of the lane's three staged power pairs pair p uses: the staged pairs are
// rotated by the lane's class, pair_index(0, lane) % 3
template <int VW>
__host__ __device__ constexpr int pair_power(int p) {
  return VW == 4 ? (64 * (p >> 1) + (p & 1)) % 3 : (32 * p) % 3;
}

template <typename T, int VW, int TP>
__device__ __forceinline__ void load_row(typename Pair<T>::type (&a)[TP], const T* row, int npair,
                                         int lane) {
  using T2 = typename Pair<T>::type;
  if constexpr (VW == 4) {
#pragma unroll
    for (int i = 0; i < TP / 2; ++i) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (2 * (lane + 32 * i) < npair)  // M even: npair is even too
        v = __ldg(reinterpret_cast<const float4*>(row) + lane + 32 * i);
      a[2 * i] = make_float2(v.x, v.y);
      a[2 * i + 1] = make_float2(v.z, v.w);
    }
  } else {
#pragma unroll
    for (int p = 0; p < TP; ++p) {
      a[p].x = a[p].y = (T)0;
      if (lane + 32 * p < npair) a[p] = __ldg(reinterpret_cast<const T2*>(row) + lane + 32 * p);
    }
  }
}

// An extrapolation so long (or x so odd: infinite, NaN) that the weighted
// coefficients could overflow one by one, with signs of their own, where
// v + g delta does not
template <typename T>
__device__ __forceinline__ bool far_x(T x) {
  return !(fabs(x) <= (sizeof(T) == 4 ? (T)1e18 : (T)1e150));
}

// one slot per lane: its row and the weights w_k of the value (with the linear
// extrapolation, tabulate.cc:116-144: v + g delta) and dw_k of the slope; of a far
// slot, some finite ones
template <typename T>
__device__ __forceinline__ int stage_weights(T* sw, const TabInfo<T>& ti, T x, int lane) {
  int idx;
  T t, delta;
  locate(ti, far_x(x) ? ti.lower : x, idx, t, delta);
  T p = (T)1, d = (T)0;  // t^k, k t^(k - 1)
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    sw[lane * TS + k] = p + delta * d;
    sw[lane * TS + 6 + k] = d;
    d = (T)(k + 1) * p;
    p *= t;
  }
  return idx;
}

// The far slots of an atom, added to its finished results (all pointers at the
// atom's rows; o and tab at the block of nc channels). Apart from the loop over
// the slots, where a test cost 3 to 5 %; this way it costs up to 1 %.
template <typename T, bool GG>
__device__ __forceinline__ void fwd_far(T* o, const T* tab, TabInfo<T> ti, const T* ex, const T* ee,
                                     int nnei, int M, int nc, int brk, int last, const T* dzx,
                                     const T* dze, int lane) {
  for (int j = 0; j <= last; ++j) {
    int idx;
    T t, delta;
    if (!far_x(ex[j])) continue;
    locate(ti, ex[j], idx, t, delta);
    const T rep = j == brk ? (T)(nnei - j) : (T)1;
#pragma unroll 1
    for (int c = lane; c < nc; c += 32) {
      T v, g;
      poly(load_coef(tab + ((size_t)idx * M + c) * 6), t, delta, v, g);
      for (int k = 0; k < 4; ++k)
        o[k * M + c] += GG ? rep * (v * dze[j * 4 + k] + dzx[j] * g * ee[j * 4 + k])
                           : rep * v * ee[j * 4 + k];
    }
  }
}

template <typename T>
__device__ __noinline__ void grad_far(T* ox, T* oe, const T* table, TabInfo<T> ti, const T* ex,
                                      const T* ee, const T* dy, int nnei, int M, int brk, int last,
                                      int lane) {
  for (int j = 0; j <= last; ++j) {
    int idx;
    T t, delta;
    if (!far_x(ex[j])) continue;
    locate(ti, ex[j], idx, t, delta);
    T V[5] = {(T)0, (T)0, (T)0, (T)0, (T)0};
    for (int c = lane; c < M; c += 32) {
      T v, g;
      poly(load_coef(table + ((size_t)idx * M + c) * 6), t, delta, v, g);
      T s = (T)0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const T y = dy[k * M + c];
        s += ee[j * 4 + k] * y;
        V[k + 1] += v * y;
      }
      V[0] += g * s;
    }
    const T rep = j == brk ? (T)(nnei - j) : (T)1;
#pragma unroll
    for (int k = 0; k < 5; ++k) V[k] = rep * warp_sum(V[k]);
    __syncwarp();  // after what the kernel's loop stored here
    if (lane == 0) {
      ox[j] = V[0];
#pragma unroll
      for (int k = 0; k < 4; ++k) oe[j * 4 + k] = V[k + 1];
    }
  }
}

// out[i,k,m] = sum_jj w_jj * (G_m(x_jj) * em[jj,k])              (forward)
// out[i,k,m] = sum_jj w_jj * (G_m * dz_dem[jj,k] + dz_dem_x[jj] * G'_m * em[jj,k])
//                                                   (GG: grad_grad)
template <typename T, int VW, int TB, bool GG>
__global__ void __launch_bounds__(TW * 32)
k_tab_fwd(T* __restrict__ out, const T* __restrict__ table, TabInfo<T> ti,
          const T* __restrict__ em_x, const T* __restrict__ em, int nloc, int nnei, int M,
          const T* __restrict__ dz_dem_x, const T* __restrict__ dz_dem) {
  using T2 = typename Pair<T>::type;
  constexpr int TP = 3 * TB / 32;  // coefficient pairs per lane
  // per warp: weights [32][TS], env rows [32][4] (GG: and the two multipliers of
  // value and slope); the pair sums of one env column at the end
  __shared__ __align__(16) T s_w[TW][32 * TS];
  __shared__ __align__(16) T s_e[TW][32 * (GG ? 8 : 4)];
  __shared__ int s_row[TW][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * TW + w;
  if (i >= nloc) return;
  const int m0 = blockIdx.y * TB, npair = 3 * min(TB, M - m0);
  const int cls = pair_index<VW>(0, lane) % 3;
  const int off[3] = {2 * cls, 2 * ((cls + 1) % 3), 2 * ((cls + 2) % 3)};
  T acc[TP][4];
#pragma unroll
  for (int p = 0; p < TP; ++p)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[p][k] = (T)0;
  const T* ex = em_x + (size_t)i * nnei;
  const T* ee = em + (size_t)i * nnei * 4;
  const int brk = fold_start(ex, ee, nnei, lane);
  const int last = brk < nnei ? brk : nnei - 1;
  bool far = false;  // this lane has had a far slot
  for (int base = 0; base <= last; base += 32) {
    const int cnt = min(32, last + 1 - base), jj = base + lane;
    if (lane < cnt) {
      const T rep = jj == brk ? (T)(nnei - jj) : (T)1;
      far |= far_x(ex[jj]);
      s_row[w][lane] = stage_weights(s_w[w], ti, ex[jj], lane);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (GG) {
          const size_t at = (size_t)i * nnei + jj;
          s_e[w][lane * 8 + k] = rep * dz_dem[at * 4 + k];
          s_e[w][lane * 8 + 4 + k] = rep * dz_dem_x[at] * ee[jj * 4 + k];
        } else {
          s_e[w][lane * 4 + k] = rep * ee[jj * 4 + k];
        }
      }
      if (far_x(ex[jj]))
        for (int k = 0; k < (GG ? 8 : 4); ++k) s_e[w][lane * (GG ? 8 : 4) + k] = (T)0;
    }
    __syncwarp();
    const T* tab = table + (size_t)m0 * 6;
    const int rs = M * 6;
    T2 a[2][TP];  // two rows in turn: the next slot's is in flight
    auto fetch = [&](T2 (&v)[TP], int q) {
      load_row<T, VW, TP>(v, tab + (size_t)s_row[w][q] * rs, npair, lane);
    };
    auto slot = [&](const T2 (&v)[TP], int q) {
      T2 pw[3], dw[3];
      const T* sw = s_w[w] + q * TS;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        pw[j] = *reinterpret_cast<const T2*>(sw + off[j]);
        if (GG) dw[j] = *reinterpret_cast<const T2*>(sw + 6 + off[j]);
      }
      T e[4], f[4];
      load4(e, s_e[w] + q * (GG ? 8 : 4));
      if (GG) load4(f, s_e[w] + q * 8 + 4);
#pragma unroll
      for (int p = 0; p < TP; ++p) {
        const T2 z = pw[pair_power<VW>(p)];
        axpy4(acc[p], fma(v[p].x, z.x, v[p].y * z.y), e);
        if (GG) {
          const T2 dz = dw[pair_power<VW>(p)];
          axpy4(acc[p], fma(v[p].x, dz.x, v[p].y * dz.y), f);
        }
      }
    };
    fetch(a[0], 0);
    for (int q = 0; q < cnt; q += 2) {
      if (q + 1 < cnt) fetch(a[1], q + 1);
      slot(a[0], q);
      if (q + 2 < cnt) fetch(a[0], q + 2);
      if (q + 1 < cnt) slot(a[1], q + 1);
    }
    __syncwarp();
  }
  // a channel's three pairs, one env column at a time
  T* red = s_w[w];
  static_assert(32 * TS >= 3 * TB, "the pair sums reuse the staging");
  T* o = out + (size_t)i * 4 * M + m0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int p = 0; p < TP; ++p) red[pair_index<VW>(p, lane)] = acc[p][k];
    __syncwarp();
    for (int c = lane; 3 * c < npair; c += 32)
      o[k * M + c] = red[3 * c] + red[3 * c + 1] + red[3 * c + 2];
    __syncwarp();
  }
  if (__any_sync(0xffffffffu, far))
    fwd_far<T, GG>(o, table + (size_t)m0 * 6, ti, ex, ee, nnei, M, npair / 3, brk, last,
                   dz_dem_x + (size_t)i * nnei, dz_dem + (size_t)i * nnei * 4, lane);
}

// dy_dem_x[i,jj] = sum_m G'_m * sum_k em[jj,k] dy[k,m]
// dy_dem[i,jj,k] = sum_m G_m * dy[k,m]           (tabulate.cc:234-341)
// A CTA holds the nmb channel blocks of blockDim / (32 nmb) atoms; a warp's
// five sums per slot are reduced over its lanes in groups of four slots and
// over the blocks in shared memory.
template <typename T, int VW, int TB>
__global__ void __launch_bounds__(512)
k_tab_grad(T* __restrict__ dy_dem_x, T* __restrict__ dy_dem, const T* __restrict__ table,
           TabInfo<T> ti, const T* __restrict__ em_x, const T* __restrict__ em,
           const T* __restrict__ dy, int nloc, int nnei, int M, int nmb) {
  using T2 = typename Pair<T>::type;
  constexpr int TP = 3 * TB / 32;
  extern __shared__ __align__(16) unsigned char tab_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  T* s_w = reinterpret_cast<T*>(tab_smem) + (size_t)w * 32 * (TS + 4 + 5);
  T* s_e = s_w + 32 * TS;
  T* s_r = s_e + 32 * 4;  // [32][5]
  int* s_row = reinterpret_cast<int*>(reinterpret_cast<T*>(tab_smem) +
                                      (size_t)nw * 32 * (TS + 4 + 5)) + w * 32;
  const int mb = w % nmb;
  const int i = blockIdx.x * (nw / nmb) + w / nmb;
  const bool act = i < nloc;
  const int m0 = mb * TB, npair = 3 * min(TB, M - m0);
  const int cls = pair_index<VW>(0, lane) % 3;
  const int off[3] = {2 * cls, 2 * ((cls + 1) % 3), 2 * ((cls + 2) % 3)};
  const T* ex = em_x + (size_t)(act ? i : 0) * nnei;
  const T* ee = em + (size_t)(act ? i : 0) * nnei * 4;
  T dyr[TP][4];
#pragma unroll
  for (int p = 0; p < TP; ++p) {
    const int q = pair_index<VW>(p, lane);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      dyr[p][k] = act && q < npair ? dy[(size_t)i * 4 * M + k * M + m0 + q / 3] : (T)0;
  }
  const int brk = fold_start(ex, ee, nnei, lane);
  const int last = brk < nnei ? brk : nnei - 1;
  const int b4 = (lane >> 4) & 1, b3 = (lane >> 3) & 1;
  bool anyfar = false;
  for (int base = 0; base < nnei; base += 32) {
    const int cnt = act ? max(0, min(32, last + 1 - base)) : 0, jj = base + lane;
    if (lane < cnt) {
      s_row[lane] = stage_weights(s_w, ti, ex[jj], lane);
#pragma unroll
      for (int k = 0; k < 4; ++k) s_e[lane * 4 + k] = ee[jj * 4 + k];
    }
    anyfar |= __any_sync(0xffffffffu, lane < cnt && far_x(ex[jj])) != 0;
    __syncwarp();
    // two rows in turn, the next slot's in flight (FP64: one, the registers of a
    // second would not fit a 16-warp CTA)
    constexpr int NB = sizeof(T) == 4 ? 2 : 1;
    const T* tab = table + (size_t)m0 * 6;
    const int rs = M * 6;
    T2 a[NB][TP];
    auto fetch = [&](T2 (&v)[TP], int q) {
      load_row<T, VW, TP>(v, tab + (size_t)s_row[q] * rs, npair, lane);
    };
    if (NB == 2 && cnt > 0) fetch(a[0], 0);
    for (int q0 = 0; q0 < cnt; q0 += 4) {
      T S[4][5];  // per slot: the slope's sum, then the value's per env column
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = q0 + u;
        T V[4] = {(T)0, (T)0, (T)0, (T)0}, Q[4] = {(T)0, (T)0, (T)0, (T)0}, sl = (T)0;
        if (q < cnt) {
          if (NB == 1)
            fetch(a[0], q);
          else if (q + 1 < cnt)
            fetch(a[(u + 1) % NB], q + 1);
          const T2(&v)[TP] = a[u % NB];
          const T* sw = s_w + q * TS;
          T2 pw[3], dw[3];
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            pw[j] = *reinterpret_cast<const T2*>(sw + off[j]);
            dw[j] = *reinterpret_cast<const T2*>(sw + 6 + off[j]);
          }
#pragma unroll
          for (int p = 0; p < TP; ++p) {
            const T2 z = pw[pair_power<VW>(p)], dz = dw[pair_power<VW>(p)];
            axpy4(V, fma(v[p].x, z.x, v[p].y * z.y), dyr[p]);
            axpy4(Q, fma(v[p].x, dz.x, v[p].y * dz.y), dyr[p]);
          }
          T e[4];
          load4(e, s_e + q * 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) sl = fma(e[k], Q[k], sl);
        }
        S[u][0] = sl;
#pragma unroll
        for (int k = 0; k < 4; ++k) S[u][k + 1] = V[k];
      }
      // the xor-16 and -8 steps leave slot 2 b4 + b3 in a lane, summed over 8
      // lanes; xor-4, -2 and -1 finish the sum
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        T r0 = (b4 ? S[2][k] : S[0][k]) +
               __shfl_xor_sync(0xffffffffu, b4 ? S[0][k] : S[2][k], 16);
        T r1 = (b4 ? S[3][k] : S[1][k]) +
               __shfl_xor_sync(0xffffffffu, b4 ? S[1][k] : S[3][k], 16);
        T v = (b3 ? r1 : r0) + __shfl_xor_sync(0xffffffffu, b3 ? r0 : r1, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const int q = q0 + 2 * b4 + b3;
        if ((lane & 7) == 0 && q < cnt) s_r[q * 5 + k] = v;
      }
    }
    __syncthreads();
    // the atom's first warp adds the channel blocks; slots after the fold point
    // keep the zero of the reference's memset
    if (act && mb == 0 && jj < nnei) {
      T v[5] = {(T)0, (T)0, (T)0, (T)0, (T)0};
      if (lane < cnt) {
        for (int b = 0; b < nmb; ++b)
#pragma unroll
          for (int k = 0; k < 5; ++k) v[k] += s_r[(size_t)b * 32 * (TS + 4 + 5) + lane * 5 + k];
        const T rep = jj == brk ? (T)(nnei - jj) : (T)1;
#pragma unroll
        for (int k = 0; k < 5; ++k) v[k] *= rep;
      }
      dy_dem_x[(size_t)i * nnei + jj] = v[0];
#pragma unroll
      for (int k = 0; k < 4; ++k) dy_dem[((size_t)i * nnei + jj) * 4 + k] = v[k + 1];
    }
    __syncthreads();
  }
  if (act && mb == 0 && anyfar)
    grad_far(dy_dem_x + (size_t)i * nnei, dy_dem + (size_t)i * nnei * 4, table, ti, ex, ee,
             dy + (size_t)i * 4 * M, nnei, M, brk, last, lane);
}

// The gradient by channels, for many atoms: one warp per atom, lane l owns the
// channels mb + 32 c + l and reads a channel's six coefficients itself. With the
// chip full of atoms the smaller instruction count wins over the wide loads.
template <typename T, int MC>
__global__ void __launch_bounds__(TW * 32)
k_tab_grad_channels(T* __restrict__ dy_dem_x, T* __restrict__ dy_dem,
           const T* __restrict__ table, TabInfo<T> ti,
           const T* __restrict__ em_x, const T* __restrict__ em,
           const T* __restrict__ dy, int nloc, int nnei, int M) {
  // dy_dem_x[i,jj] = sum_m G'_m * sum_k em[jj,k] dy[k,m]
  // dy_dem[i,jj,k] = sum_m G_m * dy[k,m]           (tabulate.cc:234-341)
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * TW + w;
  if (i >= nloc) return;
  const T* ex = em_x + (size_t)i * nnei;
  const T* ee = em + (size_t)i * nnei * 4;
  const T* dyi = dy + (size_t)i * 4 * M;
  T* ox = dy_dem_x + (size_t)i * nnei;
  T* oe = dy_dem + (size_t)i * nnei * 4;
  const int brk = fold_start(ex, ee, nnei, lane);
  const int last = brk < nnei ? brk : nnei - 1;
  const int nmb = (M + 32 * MC - 1) / (32 * MC);
  for (int mb = 0; mb < nmb; ++mb) {
    const int m0 = mb * 32 * MC;
    T dyr[MC][4];
#pragma unroll
    for (int c = 0; c < MC; ++c) {
      const int m = m0 + c * 32 + lane;
#pragma unroll
      for (int k = 0; k < 4; ++k) dyr[c][k] = m < M ? dyi[k * M + m] : (T)0.;
    }
    for (int base = 0; base <= last; base += 32) {
      T kx = (T)0., kk4[4] = {(T)0., (T)0., (T)0., (T)0.};
      const int cnt = (last + 1 - base) < 32 ? (last + 1 - base) : 32;
      for (int q = 0; q < cnt; ++q) {
        const int jj = base + q;
        const T x = ex[jj];
        T e[4] = {ee[jj * 4 + 0], ee[jj * 4 + 1], ee[jj * 4 + 2], ee[jj * 4 + 3]};
        int idx;
        T xx, delta;
        locate(ti, x, idx, xx, delta);
        const T* row = table + (size_t)idx * M * 6;
        T px = (T)0., pk[4] = {(T)0., (T)0., (T)0., (T)0.};
#pragma unroll
        for (int c = 0; c < MC; ++c) {
          const int m = m0 + c * 32 + lane;
          if (m < M) {
            Coef<T> a = load_coef(row + (size_t)m * 6);
            T v, g;
            poly(a, xx, delta, v, g);
            T dot = e[0] * dyr[c][0] + e[1] * dyr[c][1] + e[2] * dyr[c][2] + e[3] * dyr[c][3];
            px += g * dot;
#pragma unroll
            for (int k = 0; k < 4; ++k) pk[k] += v * dyr[c][k];
          }
        }
        px = warp_sum(px);
#pragma unroll
        for (int k = 0; k < 4; ++k) pk[k] = warp_sum(pk[k]);
        const T rep = jj == brk ? (T)(nnei - jj) : (T)1.;
        if (lane == q) {
          kx = px * rep;
#pragma unroll
          for (int k = 0; k < 4; ++k) kk4[k] = pk[k] * rep;
        }
      }
      const int jj = base + lane;
      if (lane < cnt) {
        if (mb == 0) {
          ox[jj] = kx;
#pragma unroll
          for (int k = 0; k < 4; ++k) oe[jj * 4 + k] = kk4[k];
        } else {
          ox[jj] += kx;
#pragma unroll
          for (int k = 0; k < 4; ++k) oe[jj * 4 + k] += kk4[k];
        }
      }
    }
  }
  // slots after the fold point keep the zero of the reference's memset
  for (int jj = last + 1 + lane; jj < nnei; jj += 32) {
    ox[jj] = (T)0.;
#pragma unroll
    for (int k = 0; k < 4; ++k) oe[jj * 4 + k] = (T)0.;
  }
}

// grad_grad by channels in the same way
template <typename T, int MC>
__global__ void __launch_bounds__(TW * 32)
k_tab_gg_channels(T* __restrict__ out, const T* __restrict__ table, TabInfo<T> ti,
                  const T* __restrict__ em_x, const T* __restrict__ em, int nloc, int nnei, int M,
                  const T* __restrict__ dz_dem_x, const T* __restrict__ dz_dem) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * TW + w;
  if (i >= nloc) return;
  T acc[MC][4];
#pragma unroll
  for (int c = 0; c < MC; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[c][k] = (T)0;
  const size_t row0 = (size_t)i * nnei;
  const int brk = fold_start(em_x + row0, em + row0 * 4, nnei, lane);
  const int last = brk < nnei ? brk : nnei - 1;
  for (int jj = 0; jj <= last; ++jj) {
    const size_t at = row0 + jj;
    const T rep = jj == brk ? (T)(nnei - jj) : (T)1, dzx = dz_dem_x[at];
    T e[4], h[4], t, delta;
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = em[at * 4 + k], h[k] = dz_dem[at * 4 + k];
    int idx;
    locate(ti, em_x[at], idx, t, delta);
    const T* row = table + (size_t)idx * M * 6;
#pragma unroll
    for (int c = 0; c < MC; ++c) {
      const int m = c * 32 + lane;
      if (m >= M) continue;
      T v, g;
      poly(load_coef(row + (size_t)m * 6), t, delta, v, g);
      const T dg = dzx * g;
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[c][k] += rep * (v * h[k] + dg * e[k]);
    }
  }
  T* o = out + (size_t)i * 4 * M;
#pragma unroll
  for (int c = 0; c < MC; ++c) {
    const int m = c * 32 + lane;
    if (m < M)
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k * M + m] = acc[c][k];
  }
}

// 16-byte row loads need an even M (rows of 24 M bytes) and an aligned table;
// FP64 pairs are 16 bytes (as the reference's double2 loads, an aligned table is
// required)
template <typename T>
static bool wide_rows(const T* table, int M) {
  return sizeof(T) == 4 && (M & 1) == 0 && (reinterpret_cast<uintptr_t>(table) & 15) == 0;
}

template <typename T, int VW, int TB>
static void launch_fwd(T* out, const T* table, const TabInfo<T>& ti, const T* em_x,
                       const T* em, int nloc, int nnei, int M, const T* dzx,
                       const T* dze, cudaStream_t st) {
  const dim3 grid(ceil_div(nloc, TW), ceil_div(M, TB));
  auto kern = dze != nullptr ? k_tab_fwd<T, VW, TB, true> : k_tab_fwd<T, VW, TB, false>;
  kern<<<grid, TW * 32, 0, st>>>(out, table, ti, em_x, em, nloc, nnei, M, dzx, dze);
}

template <typename T, int MC>
static void launch_gg_channels(T* out, const T* table, const TabInfo<T>& ti, const T* em_x,
                               const T* em, int nloc, int nnei, int M, const T* dzx,
                               const T* dze, cudaStream_t st) {
  k_tab_gg_channels<T, MC><<<ceil_div(nloc, TW), TW * 32, 0, st>>>(out, table, ti, em_x, em, nloc,
                                                                  nnei, M, dzx, dze);
}

template <typename T>
static int tab_fwd(T* out, const T* table, const T* info, const T* em_x,
                   const T* em, int nloc, int nnei, int M, const T* dzx,
                   const T* dze, cudaStream_t st, const char* name) {
  TabInfo<T> ti;
  int rc = make_info(ti, info, M);
  if (rc) return rc;
  if (nloc < 0 || nnei < 0) {
    set_error("%s: negative sizes", name);
    return DPB_ERR_INVALID;
  }
  if (nloc == 0) return DPB_OK;
  if (nnei == 0) {
    // an empty neighbor axis is a valid empty reduction (tabulate.cc:173-179)
    DPB_CUDA(cudaMemsetAsync(out, 0, sizeof(T) * (size_t)nloc * 4 * M, st), name);
    return DPB_OK;
  }
  auto run = [&](auto launch) { launch(out, table, ti, em_x, em, nloc, nnei, M, dzx, dze, st); };
  // grad_grad of many atoms by channels where those fill their lanes better than
  // pairs fill their blocks: a third 32-channel share that would take a second block
  // of 64 (us at 12,288 atoms of 92 slots, M = 96, pairs against channels: FP32 307,
  // 259, FP64 598, 494; at 3,000 atoms about even in FP32, 160 and 190 in FP64), and
  // FP64 up to 32 channels (M = 32: 12,288 atoms 251, 189, 3,000 84, 60, 192 25, 45;
  // FP32 112, 137)
  const long long per_sm = nloc / sm_count();
  if (dze != nullptr && M > 64 && M <= 96 && per_sm >= 48)
    run(launch_gg_channels<T, 3>);
  else if (dze != nullptr && sizeof(T) == 8 && M <= 32 && per_sm >= 16)
    run(launch_gg_channels<T, 1>);
  else if (M <= 32)
    run(launch_fwd<T, 2, 32>);
  else if (wide_rows(table, M))
    run(launch_fwd<T, sizeof(T) == 4 ? 4 : 2, 64>);
  else
    run(launch_fwd<T, 2, 64>);
  DPB_CHECK_LAUNCH(name);
  return DPB_OK;
}

template <typename T>
static int tab_grad(T* dy_dem_x, T* dy_dem, const T* table, const T* info,
                    const T* em_x, const T* em, const T* dy, int nloc, int nnei,
                    int M, cudaStream_t st) {
  TabInfo<T> ti;
  int rc = make_info(ti, info, M);
  if (rc) return rc;
  if (nloc < 0 || nnei < 0) {
    set_error("tabulate_fusion_se_a_grad: negative sizes");
    return DPB_ERR_INVALID;
  }
  if (nloc == 0 || nnei == 0) return DPB_OK;  // tabulate.cc:251-256
  // Pairs or channels (us, 92 slots, M = 100, FP32 | FP64): 192 atoms 31 against 78
  // | 57 against 107, 3,000 atoms 108 against 108 | 211 against 207, 12,288 atoms 367
  // against 307 | 768 against 588
  if (nloc > 16 * sm_count()) {
    const dim3 grid(ceil_div(nloc, TW));
    auto by = [&](auto kern) {
      kern<<<grid, TW * 32, 0, st>>>(dy_dem_x, dy_dem, table, ti, em_x, em, dy, nloc, nnei, M);
    };
    if (M <= 32) by(k_tab_grad_channels<T, 1>);
    else if (M <= 64) by(k_tab_grad_channels<T, 2>);
    else if (M <= 96) by(k_tab_grad_channels<T, 3>);
    else by(k_tab_grad_channels<T, 4>);
    DPB_CHECK_LAUNCH("tabulate_fusion_se_a_grad");
    return DPB_OK;
  }
  const int nmb = ceil_div(M, M <= 32 ? 32 : 64);  // at most 16 warps per atom
  const int atoms = nmb < TW ? TW / nmb : 1, nw = atoms * nmb;
  const size_t smem = (size_t)nw * 32 * ((TS + 4 + 5) * sizeof(T) + sizeof(int));
  auto run = [&](auto kern) -> int {
    if (smem > 48 * 1024)
      DPB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
               "tabulate_fusion_se_a_grad");
    kern<<<ceil_div(nloc, atoms), nw * 32, smem, st>>>(dy_dem_x, dy_dem, table, ti, em_x, em, dy,
                                                       nloc, nnei, M, nmb);
    return DPB_OK;
  };
  if (M <= 32)
    rc = run(k_tab_grad<T, 2, 32>);
  else if (wide_rows(table, M))
    rc = run(k_tab_grad<T, sizeof(T) == 4 ? 4 : 2, 64>);
  else
    rc = run(k_tab_grad<T, 2, 64>);
  if (rc) return rc;
  DPB_CHECK_LAUNCH("tabulate_fusion_se_a_grad");
  return DPB_OK;
}

}  // namespace dpb

using namespace dpb;
extern "C" {

int dpb_tabulate_fusion_se_a_f64(double* out, const double* table,
                                 const double* table_info, const double* em_x,
                                 const double* em, int nloc, int nnei,
                                 int last_layer_size, dpb_stream_t stream) {
  return tab_fwd<double>(out, table, table_info, em_x, em, nloc, nnei,
                         last_layer_size, nullptr, nullptr, as_stream(stream),
                         "tabulate_fusion_se_a");
}

int dpb_tabulate_fusion_se_a_f32(float* out, const float* table,
                                 const float* table_info, const float* em_x,
                                 const float* em, int nloc, int nnei,
                                 int last_layer_size, dpb_stream_t stream) {
  return tab_fwd<float>(out, table, table_info, em_x, em, nloc, nnei,
                        last_layer_size, nullptr, nullptr, as_stream(stream),
                        "tabulate_fusion_se_a");
}

int dpb_tabulate_fusion_se_a_grad_f64(double* dy_dem_x, double* dy_dem,
                                      const double* table,
                                      const double* table_info,
                                      const double* em_x, const double* em,
                                      const double* dy, int nloc, int nnei,
                                      int last_layer_size,
                                      dpb_stream_t stream) {
  return tab_grad<double>(dy_dem_x, dy_dem, table, table_info, em_x, em, dy,
                          nloc, nnei, last_layer_size, as_stream(stream));
}

int dpb_tabulate_fusion_se_a_grad_f32(float* dy_dem_x, float* dy_dem,
                                      const float* table,
                                      const float* table_info,
                                      const float* em_x, const float* em,
                                      const float* dy, int nloc, int nnei,
                                      int last_layer_size,
                                      dpb_stream_t stream) {
  return tab_grad<float>(dy_dem_x, dy_dem, table, table_info, em_x, em, dy,
                         nloc, nnei, last_layer_size, as_stream(stream));
}

int dpb_tabulate_fusion_se_a_grad_grad_f64(
    double* dz_dy, const double* table, const double* table_info,
    const double* em_x, const double* em, const double* dz_dy_dem_x,
    const double* dz_dy_dem, int nloc, int nnei, int last_layer_size,
    dpb_stream_t stream) {
  if (dz_dy_dem_x == nullptr || dz_dy_dem == nullptr) {
    set_error("tabulate_fusion_se_a_grad_grad: dz_dy_dem_x and dz_dy_dem are required");
    return DPB_ERR_INVALID;
  }
  return tab_fwd<double>(dz_dy, table, table_info, em_x, em, nloc, nnei,
                         last_layer_size, dz_dy_dem_x, dz_dy_dem,
                         as_stream(stream), "tabulate_fusion_se_a_grad_grad");
}

int dpb_tabulate_fusion_se_a_grad_grad_f32(
    float* dz_dy, const float* table, const float* table_info,
    const float* em_x, const float* em, const float* dz_dy_dem_x,
    const float* dz_dy_dem, int nloc, int nnei, int last_layer_size,
    dpb_stream_t stream) {
  if (dz_dy_dem_x == nullptr || dz_dy_dem == nullptr) {
    set_error("tabulate_fusion_se_a_grad_grad: dz_dy_dem_x and dz_dy_dem are required");
    return DPB_ERR_INVALID;
  }
  return tab_fwd<float>(dz_dy, table, table_info, em_x, em, nloc, nnei,
                        last_layer_size, dz_dy_dem_x, dz_dy_dem,
                        as_stream(stream), "tabulate_fusion_se_a_grad_grad");
}

}  // extern "C"
