// The FP64 transform passes of fft_impl.cuh, forward and inverse, in fixed-grid limb arithmetic
// (limb.cuh): storage S = double, arithmetic T = lf3.
//
// What bounded them before: the FP64 pipe (0.63 T operations/s; a P1 of 10000^2 took 8.8 ms for
// 2.4 GB of traffic).  Each pass reads its inputs once into registers, sums |re| + |im| over
// every transform it holds (one exchange through shared memory beside the barrier that the
// twiddle tables need anyway), scales, transforms, and scales back on its stores.
//
// Measured at 10000^2, FP64 arithmetic and limbs: map rows 6.1 and 1.7 ms, column pass 2.5 and
// 0.70, P1 8.8 and 1.9 (four Gaussians of 100 to 600 rows), P3 5.9 and 1.5.
#pragma once

#include <cooperative_groups.h>

#include "fft_impl.cuh"
#include "limb.cuh"

namespace mlc {

template <typename T>
__device__ __forceinline__ C2<T> limb_zero() {
  return C2<T>{T(0.0), T(0.0)};
}

// ---------------------------------------------------------------- columns

// k_colpass2 (fft_impl.cuh) in limbs: the sums of a column's L1 inputs per thread are
// exchanged through red while the tables are being filled.  Strips wider than the pitch's
// 16-column granule mask the columns past it.
template <typename S, typename T, int CW, int L1, int L2, bool INV>
__global__ void __launch_bounds__((L1 > L2 ? L1 : L2) * CW, 2)
    k_limb_colpass2(C2<S>* __restrict__ buf, long pitch, long set_mul, long j_mul, LimbTab<T> twy, int tw_stride,
                    int post_tw) {
  constexpr int L = L1 * L2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const LimbArr<T> y = LimbArr<T>::at(smem_raw, L * CW);  // [L2][L1][CW]
  const LimbArr<T> wl = LimbArr<T>::at(smem_raw + LimbArr<T>::bytes(L * CW), L);                             // W_L^m
  const LimbArr<T> pw = LimbArr<T>::at(smem_raw + LimbArr<T>::bytes(L * CW) + LimbArr<T>::bytes(L), L);  // W_Ny^(set j)
  __shared__ LimbSum<S> red[L2][CW];
  const int set = blockIdx.y;
  const int c = threadIdx.x % CW, g = threadIdx.x / CW;
  const long col = (long)blockIdx.x * CW + c;
  const bool in = CW <= 16 || col < pitch;
  C2<S>* b = buf + (long)set * set_mul * pitch + col;
  C2<S> raw[L1];
  if (g < L2) {
#pragma unroll
    for (int n1 = 0; n1 < L1; n1++)
      raw[n1] = in ? b[(long)(L2 * n1 + g) * j_mul * pitch] : C2<S>{S(0.0), S(0.0)};
  }
  for (int m = threadIdx.x; m < L; m += blockDim.x) {
    wl.st(m, twy.ld((long)m * tw_stride));
    if (post_tw) pw.st(m, twy.ld((long)set * m));  // set*m < Ny
  }
  if (g < L2) red[g][c] = limb_sum<L1>(raw);
  __syncthreads();
  LimbSum<S> sum = red[0][c];
#pragma unroll
  for (int q = 1; q < L2; q++) sum = limb_sum_add(sum, red[q][c]);
  const LimbScale<T> sc = limb_scale(sum);
  if (g < L2) {
    C2<T> v[L1];
    const LimbScale<T> si = limb_lift<L1>(raw, sc);
#pragma unroll
    for (int n1 = 0; n1 < L1; n1++) v[n1] = limb_cin(raw[n1], si);
    Dft<T, L1, INV>::run(v);
#pragma unroll
    for (int k1 = 0; k1 < L1; k1++)
      y.st((g * L1 + k1) * CW + c, k1 == 0 ? limb_cnorm(v[0]) : limb_tw<INV>(v[k1], wl.ld(g * k1)));
  }
  __syncthreads();
  if (g < L1) {
    C2<T> u[L2];
#pragma unroll
    for (int n2 = 0; n2 < L2; n2++) u[n2] = y.ld((n2 * L1 + g) * CW + c);
    Dft<T, L2, INV>::run(u);
#pragma unroll
    for (int k2 = 0; k2 < L2; k2++) {
      const int j = g + L1 * k2;
      C2<T> val = u[k2];
      if (post_tw) val = limb_tw<INV>(val, pw.ld(j));
      if (in) b[(long)j * j_mul * pitch] = limb_cout<S>(val, sc);
    }
  }
}

// ---------------------------------------------------------------- P1

constexpr int LIMB_BAD = 0x7fffffff;  // the exponent of a column whose sum is not finite

// FP64: the profile's row spectra (P0, 2h rows) in limbs under one exponent per column, which
// every row block of P1 (N1 of them) then reads instead of scaling the rows anew: a CTA per
// strip, its threads over (row, column).
template <int CW>
__global__ void __launch_bounds__(256) k_limb_profile_columns(const C2<double>* __restrict__ kx, long pitch, int rows,
                                                              float4* __restrict__ la, float2* __restrict__ lb,
                                                              int* __restrict__ kexp) {
  constexpr int G = 256 / CW;
  __shared__ LimbSum<double> red[G][CW];
  const int c = threadIdx.x % CW, g = threadIdx.x / CW;
  const long col = (long)blockIdx.x * CW + c;
  LimbSum<double> sum{0, 0.f};
  for (int r = g; r < rows; r += G) {
    const C2<double> v = ldc(kx + r * pitch + col);
    sum = limb_sum_add(sum, limb_sum<1>(&v));
  }
  red[g][c] = sum;
  __syncthreads();
  sum = red[0][c];
#pragma unroll
  for (int q = 1; q < G; q++) sum = limb_sum_add(sum, red[q][c]);
  const LimbScale<lf3> sc = limb_scale(sum);
  if (g == 0) kexp[col] = sc.bad ? LIMB_BAD : sc.e;
  for (int r = g; r < rows; r += G) {
    const long i = r * pitch + col;
    C2<double> raw = ldc(kx + i);
    const LimbScale<lf3> si = limb_lift<1>(&raw, sc);
    const C2<lf3> v = limb_cin(raw, si);
    la[i] = make_float4(v.x.h, v.y.h, v.x.m, v.y.m);
    lb[i] = make_float2(v.x.l, v.y.l);
  }
}

// FP64 limbs in global memory: n complex values in two planes, then exponents.
struct LimbSpectrum {
  float4* a;
  float2* b;
  int* e;
  static size_t bytes(size_t n, size_t nexp) { return n * 24 + nexp * sizeof(int); }
  LimbSpectrum(void* p, size_t n) {
    a = (float4*)p;
    b = (float2*)((char*)p + n * 16);
    e = (int*)((char*)p + n * 24);
  }
  __device__ __forceinline__ C2<lf3> ld(long i) const { return LimbTab<lf3>{a, b}.ld(i); }
  __device__ __forceinline__ void st(long i, C2<lf3> v) const {
    a[i] = make_float4(v.x.h, v.y.h, v.x.m, v.y.m);
    b[i] = make_float2(v.x.l, v.y.l);
  }
};

// P1 of FP64 plans (k_conv_fused2's three modes: 0 the whole pass, 1 the profile's spectrum
// into ks, 2 from it).  The profile's spectrum stays in limbs, under the exponent of its
// column's rows, from its transform to the product (also in ks): no rounding to FP64 and no
// second scaling, so modes 1 + 2 equal mode 0 bit for bit.  1/(Nx Ny) = r 2^-rexp enters with
// the profile's first twiddles.  The map's column is scaled by its own sum, read once for the
// sum and once, out of L1 or L2, for the product (holding it in between took 40 registers).
// The products' sum is below the product of the two scales.
// Bound by the FP32 pipe and by instruction fetch: the unrolled code is some 60 KB, and strips
// of 32 columns (10 warps that run it together) fetch it half as often as 16.
template <int CW, int L1, int L2, int MODE>
__global__ void __launch_bounds__((L1 > L2 ? L1 : L2) * CW, 2)
    k_limb3_conv(const C2<double>* __restrict__ Fmap, C2<double>* __restrict__ out, long pitch, LimbSpectrum kx, int h,
                 int Ny, int N1, LimbTab<lf3> twy, lf3 r, int rexp, LimbSpectrum ks) {
  using T = lf3;
  constexpr int N2 = L1 * L2, G = L1 > L2 ? L1 : L2, NE = N2 / G;
  static_assert(N2 % G == 0, "rows per thread");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr size_t TB = LimbArr<T>::bytes(N2);
  const LimbArr<T> y = LimbArr<T>::at(smem_raw, N2 * CW);  // the profile's sub-pass, then the transposes
  unsigned char* tabs = smem_raw + LimbArr<T>::bytes(N2 * CW);
  const LimbArr<T> w2 = LimbArr<T>::at(tabs, N2);            // W_Ny^(n kk), n < N2
  const LimbArr<T> wl = LimbArr<T>::at(tabs + TB, N2);       // W_N2^m, m < N2
  const LimbArr<T> w2r = LimbArr<T>::at(tabs + 2 * TB, N2);  // r W_Ny^(n kk)
  const LimbArr<T> w1 = LimbArr<T>::at(tabs + 3 * TB, N1);   // W_N1^(n1 kk), n1 < N1
  __shared__ LimbSum<double> red[L1][CW];
  const int kk = blockIdx.y;
  const int c = threadIdx.x % CW, g = threadIdx.x / CW;
  const long col = (long)blockIdx.x * CW + c;
  const bool in = CW <= 16 || col < pitch;
  const C2<double>* f = Fmap + ((long)kk * N2 + g) * pitch + col;  // + L1 k2 rows
  if constexpr (MODE != 1) {
    if (g < L1) {
      C2<double> raw[L2];
#pragma unroll
      for (int k2 = 0; k2 < L2; k2++) raw[k2] = in ? f[(long)(L1 * k2) * pitch] : C2<double>{0.0, 0.0};
      red[g][c] = limb_sum<L2>(raw);
    }
  }
  for (int n = threadIdx.x; n < N2; n += blockDim.x) {
    const C2<T> w = twy.ld((long)n * kk);
    w2.st(n, w);
    wl.st(n, twy.ld((long)n * N1));
    if constexpr (MODE != 2) w2r.st(n, C2<T>{r * w.x, r * w.y});
  }
  int ke;  // the profile spectrum's exponent
  C2<T> u[L2];
  if constexpr (MODE != 2) {
    for (int n1 = threadIdx.x; n1 < N1; n1 += blockDim.x) w1.st(n1, twy.ld((long)((n1 * kk) % N1) * N2));
    ke = in ? kx.e[col] : 0;
    if (ke != LIMB_BAD) ke -= rexp;
    __syncthreads();
    // the profile's column sub-pass over its non-zero rows: kernel rows j < h (n1 from 0) and
    // j >= Ny - h (n1 up to N1 - 1; compacted row j - (Ny - 2h)), E elements at a time: their
    // loads of one term are in flight together, and the code stays short
    constexpr int E = NE % 2 == 0 ? 2 : 1;
#pragma unroll 1
    for (int i = 0; i < NE; i += E) {
      C2<T> acc[E];
      auto term = [&](int n1, bool high) {
        C2<T> v[E];
#pragma unroll
        for (int q = 0; q < E; q++) {
          const int j = n1 * N2 + g + G * (i + q);  // kernel row
          const bool on = in && (high ? j >= Ny - h : j < h);
          v[q] = on ? kx.ld((long)(high ? j - (Ny - 2 * h) : j) * pitch + col) : limb_zero<T>();
        }
        const C2<T> w = w1.ld(n1);
#pragma unroll
        for (int q = 0; q < E; q++) acc[q] = cadd(acc[q], limb_tw<false>(v[q], w));
      };
#pragma unroll
      for (int q = 0; q < E; q++) {
        const int j = g + G * (i + q);
        acc[q] = in && j < h ? kx.ld((long)j * pitch + col) : limb_zero<T>();  // weight W^0 = 1
      }
#pragma unroll 1
      for (int n1 = 1; n1 * N2 + g + G * i < h; n1++) term(n1, false);
#pragma unroll 1
      for (int n1 = max((Ny - h - g - G * (i + E - 1) + N2 - 1) / N2, 0); n1 < N1; n1++) term(n1, true);
#pragma unroll
      for (int q = 0; q < E; q++) {
        const int n2 = g + G * (i + q);
        y.st(n2 * CW + c, limb_tw<false>(acc[q], w2r.ld(n2)));
      }
    }
    __syncthreads();
    {
      C2<T> v[L1];
      if (g < L2) {
#pragma unroll
        for (int n1 = 0; n1 < L1; n1++) v[n1] = y.ld((L2 * n1 + g) * CW + c);
        Dft<T, L1, false>::run(v);
      }
      __syncthreads();
      if (g < L2) {
#pragma unroll
        for (int k1 = 0; k1 < L1; k1++)
          y.st((g * L1 + k1) * CW + c, k1 == 0 ? limb_cnorm(v[0]) : limb_tw<false>(v[k1], wl.ld(g * k1)));
      }
    }
    __syncthreads();
    if (g < L1) {
#pragma unroll
      for (int n2 = 0; n2 < L2; n2++) u[n2] = y.ld((n2 * L1 + g) * CW + c);
      Dft<T, L2, false>::run(u);
    }
    if constexpr (MODE == 1) {
      if (g < L1 && in) {
#pragma unroll
        for (int k2 = 0; k2 < L2; k2++) ks.st(((long)kk * N2 + g + L1 * k2) * pitch + col, limb_cnorm(u[k2]));
        if (g == 0) ks.e[(long)kk * pitch + col] = ke;
      }
      return;  // (every thread: no barrier follows)
    }
  } else {
    ke = in ? ks.e[(long)kk * pitch + col] : 0;
    if (g < L1) {
#pragma unroll
      for (int k2 = 0; k2 < L2; k2++)
        u[k2] = in ? ks.ld(((long)kk * N2 + g + L1 * k2) * pitch + col) : limb_zero<T>();
    }
    __syncthreads();
  }
  if constexpr (MODE != 1) {
    LimbSum<double> sum = red[0][c];
#pragma unroll
    for (int q = 1; q < L1; q++) sum = limb_sum_add(sum, red[q][c]);
    LimbScale<T> sc = limb_scale(sum);
    // product with the map spectrum: thread (k1 = g, c) holds frequencies k1 + L1 k2
    if (g < L1) {
#pragma unroll
      for (int k2 = 0; k2 < L2; k2++) {
        C2<double> raw = in ? f[(long)(L1 * k2) * pitch] : C2<double>{0.0, 0.0};
        const LimbScale<T> si = limb_lift<1>(&raw, sc);
        const C2<T> fl = limb_cin(raw, si);
        u[k2] = limb_tw<false>(fl, MODE == 0 ? limb_cnorm(u[k2]) : u[k2]);
      }
      Dft<T, L2, true>::run(u);  // over k2 -> n2
      // (the thread rewrites exactly the entries of y it read above: no other thread's data)
#pragma unroll
      for (int n2 = 0; n2 < L2; n2++)
        y.st((n2 * L1 + g) * CW + c, n2 == 0 ? limb_cnorm(u[0]) : limb_tw<true>(u[n2], wl.ld(g * n2)));
    }
    sc.bad |= ke == LIMB_BAD;  // the scales multiply: exponents add
    sc.e += sc.bad ? 0 : ke;
    __syncthreads();
    // inverse stage B: thread (n2 = g, c) over k1 -> rows n2 + L2 n1
    if (g < L2) {
      C2<T> v[L1];
#pragma unroll
      for (int k1 = 0; k1 < L1; k1++) v[k1] = y.ld((g * L1 + k1) * CW + c);
      Dft<T, L1, true>::run(v);
      if (in) {
#pragma unroll
        for (int n1 = 0; n1 < L1; n1++) {
          const int n = g + L2 * n1;
          out[((long)kk * N2 + n) * pitch + col] = limb_cout<double>(limb_tw<true>(v[n1], w2.ld(n)), sc);
        }
      }
    }
  }
}

// ---------------------------------------------------------------- rows

// An in-place transform of M = R0 R1 ... points in shared memory, one level per radix
// (decimation in frequency): level i works on blocks of B_i = M / (R0 ... R_{i-1}) points,
// item (block, m < B_i / R_i) transforms the R_i points m + q B_{i+1} and multiplies output q
// by W_{B_i}^(m q).  Output digit i of a result is index digit i of its place, so the last
// level, whose items each thread takes by their output index n0, leaves the CTA's
// registers in natural order: point n0 + q M / R_last.
// Blocks are padded to odd lengths (T_i in elements) where the next level's stride would
// put a warp's accesses in a few shared-memory banks.
template <int... R>
struct Levels;
template <int R0>
struct Levels<R0> {
  static constexpr int M = R0, T = R0, LAST = R0;
};
template <int R0, int R1, int... R>
struct Levels<R0, R1, R...> {
  using Next = Levels<R1, R...>;
  static constexpr int M = R0 * Next::M;
  static constexpr int TN = Next::T | 1;  // padded length of one sub-block
  static constexpr int T = R0 * TN;
  static constexpr int LAST = Next::LAST;
};

// place of point i of a block
template <typename LV>
struct LevelPlace;
template <int R0>
struct LevelPlace<Levels<R0>> {
  static __device__ __forceinline__ int of(int i) { return i; }
  static __device__ __forceinline__ int rev(int) { return 0; }
};
template <int R0, int R1, int... R>
struct LevelPlace<Levels<R0, R1, R...>> {
  using LV = Levels<R0, R1, R...>;
  using NP = LevelPlace<typename LV::Next>;
  static __device__ __forceinline__ int of(int i) {
    const int q = i / LV::Next::M;
    return q * LV::TN + NP::of(i - q * LV::Next::M);
  }
  // first point of the last level's item whose outputs start at index n (this block's digits)
  static __device__ __forceinline__ int rev(int n) {
    const int q = n / R0;
    return (n - q * R0) * LV::TN + NP::rev(q);
  }
};

// One level but the last: NB blocks of LV, whose places come from `outer`; tw(q, m) is
// W_{LV::M}^(m q).
// grow: the factor to the level's scale, 1 where it stays.
template <typename T, bool INV, int NT, typename LV, int R0, int NB, typename Place, typename Tw>
__device__ __forceinline__ void limb_level(const LimbArr<T>& s, float grow, Place outer, Tw tw) {
  constexpr int BN = LV::Next::M, TN = LV::TN;
  for (int it = threadIdx.x; it < NB * BN; it += NT) {
    const int blk = it / BN, m = it - blk * BN;
    const int p = outer(blk) + LevelPlace<typename LV::Next>::of(m);
    C2<T> u[R0];
#pragma unroll
    for (int q = 0; q < R0; q++) u[q] = s.ld(p + q * TN);
    if (grow != 1.f) {
#pragma unroll
      for (int q = 0; q < R0; q++) u[q] = cscale2(u[q], grow);
    }
    Dft<T, R0, INV>::run(u);
    s.st(p, limb_cnorm(u[0]));
#pragma unroll
    for (int q = 1; q < R0; q++) s.st(p + q * TN, limb_tw<INV>(u[q], tw(q, m)));
  }
  __syncthreads();
}

// Twiddles of the levels.  Level 0's (M points) come from global memory, tab0 in the order
// [q - 1][m] that a warp reads in whole lines (W_Nx at strides of 2 q entries cost a line per
// lane); the deeper levels' from shared memory in the same order, one table after another
// (level 1 in the order of W_{B1} at strides of q entries met a few banks).
template <typename LV>
struct DeepTwiddles {  // of the levels of LV but the last
  static constexpr int n = 0;
};
template <int R0, int R1, int... R>
struct DeepTwiddles<Levels<R0, R1, R...>> {
  using Next = typename Levels<R0, R1, R...>::Next;
  static constexpr int own = (R0 - 1) * Next::M;
  static constexpr int n = own + DeepTwiddles<Next>::n;
};
// f = M / LV::M: W_{LV::M}^e is entry 2 f e of the global table of W_Nx, Nx = 2 M.
template <typename T, int NT, int F, int R0>
__device__ __forceinline__ void limb_fill_deep(Levels<R0>, const LimbArr<T>&, int, const LimbTab<T>&) {}
template <typename T, int NT, int F, int R0, int R1, int... R>
__device__ __forceinline__ void limb_fill_deep(Levels<R0, R1, R...>, const LimbArr<T>& w, int at,
                                               const LimbTab<T>& twx) {
  using LV = Levels<R0, R1, R...>;
  constexpr int BN = LV::Next::M;
  for (int e = threadIdx.x; e < (R0 - 1) * BN; e += NT) {
    const int q = e / BN + 1, m = e - (q - 1) * BN;
    w.st(at + e, twx.ld(2L * F * q * m));
  }
  limb_fill_deep<T, NT, F * R0>(typename LV::Next{}, w, at + (R0 - 1) * BN, twx);
}

// All levels but the last, in order, from level DEPTH on; `at`: where the level's table starts
// in w.
template <typename T, bool INV, int NT, int DEPTH, int NB, typename Place, int R0>
__device__ __forceinline__ void limb_levels(Levels<R0>, const LimbArr<T>&, const LimbArr<T>&, int, const LimbTab<T>&,
                                            LimbGrow&, Place) {}
template <typename T, bool INV, int NT, int DEPTH, int NB, typename Place, int R0, int R1, int... R>
__device__ __forceinline__ void limb_levels(Levels<R0, R1, R...>, const LimbArr<T>& s, const LimbArr<T>& w, int at,
                                            const LimbTab<T>& tab0, LimbGrow& grow, Place outer) {
  using LV = Levels<R0, R1, R...>;
  constexpr int BN = LV::Next::M;
  limb_level<T, INV, NT, LV, R0, NB>(s, DEPTH == 0 ? 1.f : grow.next(R0), outer, [&](int q, int m) {
    if constexpr (DEPTH == 0) return tab0.ld((q - 1) * BN + m);
    else return w.ld(at + (q - 1) * BN + m);
  });
  limb_levels<T, INV, NT, DEPTH + 1, NB * R0>(
      typename LV::Next{}, s, w, DEPTH == 0 ? 0 : at + (R0 - 1) * BN, tab0, grow,
      [=](int blk) { return outer(blk / R0) + (blk % R0) * LV::TN; });
}

// The last level of a row transform from the padded places in s.  Its results go through cvt,
// then -- with BAR after a barrier, so that put may write over s -- to put(n, v).
template <typename T, bool INV, int NT, bool BAR, typename V, typename Cvt, typename Put, int R0, int... R>
__device__ __forceinline__ void limb_last_level(Levels<R0, R...>, const LimbArr<T>& s, float grow, Cvt cvt, Put put) {
  using LV = Levels<R0, R...>;
  constexpr int LAST = LV::LAST, NI = LV::M / LAST, PER = (NI + NT - 1) / NT;
  V out[PER][LAST];
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const int n0 = threadIdx.x + i * NT;
    if (n0 < NI) {
      const int p = LevelPlace<LV>::rev(n0);
      C2<T> u[LAST];
#pragma unroll
      for (int q = 0; q < LAST; q++) u[q] = s.ld(p + q);
      if (grow != 1.f) {
#pragma unroll
        for (int q = 0; q < LAST; q++) u[q] = cscale2(u[q], grow);
      }
      Dft<T, LAST, INV>::run(u);
#pragma unroll
      for (int q = 0; q < LAST; q++) out[i][q] = cvt(u[q]);
      if (!BAR) {
#pragma unroll
        for (int q = 0; q < LAST; q++) put(n0 + q * NI, out[i][q]);
      }
    }
  }
  if (BAR) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const int n0 = threadIdx.x + i * NT;
      if (n0 < NI) {
#pragma unroll
        for (int q = 0; q < LAST; q++) put(n0 + q * NI, out[i][q]);
      }
    }
  }
}

template <int NT>
__device__ __forceinline__ LimbPeak limb_block_peak(LimbPeak v, LimbPeak* red) {
  v = limb_peak_warp(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  LimbPeak all = red[0];
#pragma unroll
  for (int w = 1; w < NT / 32; w++) all = limb_peak_add(all, red[w]);
  return all;
}

template <typename T, typename LV>
constexpr size_t limb_row_smem() {
  return LimbArr<T>::bytes(LV::T) + LimbArr<T>::bytes(DeepTwiddles<typename LV::Next>::n);
}

// b[k] and its partner b[M-k] of the c2r input from xk = X[k], xm = conj X[M-k]:
// e' = conj e and, as W^-(M-k) = -conj W^-k, o' = conj o.
template <typename T>
__device__ __forceinline__ void limb_c2r_pair(C2<T> xk, C2<T> xm, C2<T> w, C2<T>& bk, C2<T>& bm) {
  const C2<T> e = cadd(xk, xm);
  const C2<T> o = limb_tw<true>(csub(xk, xm), w);  // (X - conj X') W^-k
  bk = C2<T>{e.x - o.y, e.y + o.x};
  bm = C2<T>{e.x + o.y, o.x - e.y};
}

// The inverse real transform of one spectrum row (as k_rows_c2r: the input
// b[k] = (X[k] + conj X[M-k]) + i (X[k] - conj X[M-k]) W_Nx^-k, then the inverse transform of
// M points).  The row is read once into registers, both partners k and M - k by one thread.
template <typename S, typename T, int NT, int R0, int... R>
__device__ __forceinline__ LimbGrow limb_c2r_first(Levels<R0, R...>, const C2<S>* __restrict__ a,
                                                       const LimbTab<T>& twx, const LimbTab<T>& tab0,
                                                       const LimbArr<T>& s, const LimbArr<T>& w, LimbPeak* red) {
  using LV = Levels<R0, R...>;
  constexpr int M = LV::M, NP = (M / 2 + 1 + NT - 1) / NT;
  const int tid = threadIdx.x;
  C2<S> x[2 * NP];
#pragma unroll
  for (int i = 0; i < NP; i++) {
    const int k = tid + i * NT;
    const bool in = k <= M / 2;
    x[2 * i] = in ? ldc(a + k) : C2<S>{S(0.0), S(0.0)};
    x[2 * i + 1] = in ? ldc(a + (M - k)) : C2<S>{S(0.0), S(0.0)};
  }
  limb_fill_deep<T, NT, R0>(typename LV::Next{}, w, 0, twx);
  // |b[k]| + |b[M-k]| <= 2 sqrt(2) (|X[k]| + |X[M-k]|), and each of them <= 2 (|X[k]| + |X[M-k]|)
  LimbGrow grow = LimbGrow::of(limb_block_peak<NT>(limb_peak<2 * NP, 2>(x), red), 2.82843f, 2.f);
  const LimbScale<T> sc = limb_lift<2 * NP>(x, grow.first(R0));
#pragma unroll
  for (int i = 0; i < NP; i++) {
    const int k = tid + i * NT;
    if (k <= M / 2) {
      C2<T> bk, bm;
      limb_c2r_pair(limb_cin(x[2 * i], sc), cconj(limb_cin(x[2 * i + 1], sc)), twx.ld(k), bk, bm);
      s.st(LevelPlace<LV>::of(k), bk);
      if (k > 0 && k != M - k) s.st(LevelPlace<LV>::of(M - k), bm);
    }
  }
  __syncthreads();
  limb_levels<T, true, NT, 0, 1>(LV{}, s, w, 0, tab0, grow, [](int) { return 0; });
  return grow;
}

template <typename S, typename T, typename TO, int NT, bool BAR, typename Put, typename LV>
__device__ __forceinline__ void limb_c2r_row(LV, const C2<S>* __restrict__ a, const LimbTab<T>& twx,
                                             const LimbTab<T>& tab0, unsigned char* smem, LimbPeak* red, Put put) {
  const LimbArr<T> s = LimbArr<T>::at(smem, LV::T);
  const LimbArr<T> w = LimbArr<T>::at(smem + LimbArr<T>::bytes(LV::T), DeepTwiddles<typename LV::Next>::n);
  LimbGrow grow = limb_c2r_first<S, T, NT>(LV{}, a, twx, tab0, s, w, red);
  const float last = grow.next(LV::LAST);
  const LimbScale<T> sc = grow.scale();
  limb_last_level<T, true, NT, BAR, C2<TO>>(
      LV{}, s, last, [&](C2<T> z) { return C2<TO>{limb_round(z.x, sc), limb_round(z.y, sc)}; }, put);
}

// P3: one row per CTA, the pixels written from registers in thread order.
template <typename S, typename T, typename TO, int NT, typename LV>
__global__ void __launch_bounds__(NT) k_limb_rows_c2r(const C2<S>* __restrict__ in, long pitch, TO* __restrict__ out,
                                                      long ldo, LimbTab<T> twx, LimbTab<T> tab0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LimbPeak red[NT / 32];
  C2<TO>* dst = reinterpret_cast<C2<TO>*>(out + (long)blockIdx.x * ldo);
  limb_c2r_row<S, T, TO, NT, false>(LV{}, in + (long)blockIdx.x * pitch, twx, tab0, smem_raw, red,
                                    [&](int n, C2<TO> z) { dst[n] = z; });
}

// P3 of four profiles with the interleave fused in, the cluster form of k_rows_c2r3_il
// (fft_impl.cuh): the row of pixels is left rounded to TO in each CTA's shared memory.
template <typename S, typename T, typename TO, int NT, typename LV>
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(NT)
    k_limb_rows_c2r_il(const C2<S>* __restrict__ specs, long spec_stride, long pitch, int nm, TO* __restrict__ out,
                       int S_, LimbTab<T> twx, LimbTab<T> tab0, unsigned planar) {
  constexpr int M = LV::M, NX = 2 * M;
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LimbPeak red[NT / 32];
  TO* px = reinterpret_cast<TO*>(smem_raw);
  C2<TO>* pz = reinterpret_cast<C2<TO>*>(smem_raw);
  const int row = blockIdx.y;
  const int k = (int)cl.block_rank(), quad = blockIdx.x >> 2, q = 4 * quad + k;
  if (q < nm && ((planar >> q) & 1u)) {  // the direct form's real map: copy its row
    const TO* src = reinterpret_cast<const TO*>(specs + (long)q * spec_stride) + (long)row * NX;
    for (int n = threadIdx.x; n < NX; n += NT) px[n] = src[n];
  } else if (q < nm) {
    limb_c2r_row<S, T, TO, NT, true>(LV{}, specs + (long)q * spec_stride + (long)row * pitch, twx, tab0, smem_raw, red,
                                     [&](int n, C2<TO> z) { pz[n] = z; });
  } else {
    for (int n = threadIdx.x; n < NX; n += NT) px[n] = TO(0);
  }
  cl.sync();  // every row of the cluster is in its CTA's shared memory
  const int W = S_ - 4 * quad < 4 ? S_ - 4 * quad : 4;  // values per pixel from this cluster
  constexpr int CH = (NX + 3) / 4;
  const int x0 = k * CH, x1 = x0 + CH < NX ? x0 + CH : NX;
  TO* dst = out + (long)row * NX * S_ + 4 * quad;
  if (W == 4) {
    const TO* src[4];
#pragma unroll
    for (int r = 0; r < 4; r++) src[r] = cl.map_shared_rank(px, r);
    for (int x = x0 + threadIdx.x; x < x1; x += NT) {
      TO v[4];
#pragma unroll
      for (int r = 0; r < 4; r++) v[r] = src[r][x];
      float4* d = reinterpret_cast<float4*>(dst + (long)x * S_);
      const float4* wv = reinterpret_cast<const float4*>(v);
#pragma unroll
      for (int i = 0; i < (int)(4 * sizeof(TO) / 16); i++) d[i] = wv[i];
    }
  } else {
    for (int r = 0; r < W; r++) {
      const TO* sr = cl.map_shared_rank(px, r);
      for (int x = x0 + threadIdx.x; x < x1; x += NT) dst[(long)x * S_ + r] = sr[x];
    }
  }
  // no CTA leaves while the others still read its shared memory (relaxed: see k_rows_c2r3_il)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// The forward real transform of one row per CTA (k_rows_r2c3's result): the levels, then
// X[k] and X[M-k] of each pair from Z[k] and Z[M-k].
template <typename S, typename T, int NT, typename LV, typename Loader>
__global__ void __launch_bounds__(NT)
    k_limb_rows_r2c(Loader ld, C2<S>* __restrict__ out, long pitch, LimbTab<T> twx, LimbTab<T> tab0) {
  constexpr int M = LV::M, NV = (M + NT - 1) / NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LimbPeak red[NT / 32];
  const LimbArr<T> s = LimbArr<T>::at(smem_raw, LV::T);
  const LimbArr<T> w = LimbArr<T>::at(smem_raw + LimbArr<T>::bytes(LV::T), DeepTwiddles<typename LV::Next>::n);
  const int tid = threadIdx.x, row = blockIdx.x;
  C2<S> x[NV];
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int n = tid + i * NT;
    x[i] = n < M ? ld.pair(row, n) : C2<S>{S(0.0), S(0.0)};
  }
  limb_fill_deep<T, NT, LV::M / LV::Next::M>(typename LV::Next{}, w, 0, twx);
  LimbGrow grow = LimbGrow::of(limb_block_peak<NT>(limb_peak<NV, 1>(x), red), 1.f, 1.f);
  const LimbScale<T> sc = limb_lift<NV>(x, grow.first(LV::M / LV::Next::M));
#pragma unroll
  for (int i = 0; i < NV; i++) {
    const int n = tid + i * NT;
    if (n < M) s.st(LevelPlace<LV>::of(n), limb_cin(x[i], sc));
  }
  __syncthreads();
  limb_levels<T, false, NT, 0, 1>(LV{}, s, w, 0, tab0, grow, [](int) { return 0; });
  limb_last_level<T, false, NT, true, C2<T>>(
      LV{}, s, grow.next(LV::LAST), [](C2<T> z) { return z; }, [&](int n, C2<T> z) { s.st(n, z); });
  __syncthreads();
  // X[k] = s - i W^k d with s = (Z[k] + conj Z[M-k]) / 2, d = (Z[k] - conj Z[M-k]) / 2, which the scale
  // of Z holds for; for M - k, s' = conj s and W^(M-k) d' = conj (W^k d): X[M-k] = conj s - i conj (W^k d)
  C2<S>* o = out + (long)row * pitch;
  const LimbScale<T> so = grow.scale();
  for (int k = tid; k <= M / 2; k += NT) {
    const C2<T> zk = cscale2(s.ld(k), 0.5f), zc = cconj(cscale2(s.ld(k == 0 ? 0 : M - k), 0.5f));
    const C2<T> a = cadd(zk, zc);
    const C2<T> wd = limb_tw<false>(csub(zk, zc), twx.ld(k));
    o[k] = limb_cout<S>(C2<T>{a.x + wd.y, a.y - wd.x}, so);
    if (k != M - k) o[M - k] = limb_cout<S>(C2<T>{a.x - wd.y, -wd.x - a.y}, so);
  }
  for (int k = M + 1 + tid; k < pitch; k += NT) o[k] = C2<S>{S(0.0), S(0.0)};
}

// ---------------------------------------------------------------- launches

template <typename T>
struct LimbTraits;
template <>
struct LimbTraits<lf3> {
  using S = double;
  using TO = double;
  // N entries: 16-byte plane, then the 8-byte plane
  static LimbTab<lf3> tab(const FftPlan2D&, const void*, const void* t3, int N) {
    return {(const float4*)t3, (const float2*)((const char*)t3 + (size_t)N * 16)};
  }
};
template <typename T>
static LimbTab<T> limb_twx(const FftPlan2D& p) { return LimbTraits<T>::tab(p, p.twx, p.twx3, p.Nx); }
template <typename T>
static LimbTab<T> limb_tab0(const FftPlan2D& p) {
  return LimbTraits<T>::tab(p, nullptr, p.twl3, limb_level0_entries(p.M));
}
template <typename T>
static LimbTab<T> limb_twy(const FftPlan2D& p) { return LimbTraits<T>::tab(p, p.twy, p.twy3, p.Ny); }

// Columns per CTA for factors whose larger one is g.  The passes are bound by the FP32 pipe and
// fetch long unrolled code: wide CTAs, two per SM.
constexpr int limb_cw(int g) { return g == 16 ? 16 : 32; }

// The same passes for other lengths (fft_limb_any.cu).
template <bool INV>
bool any_colpass_impl(mlc_ctx* ctx, const FftPlan2D& p, void* buf, char kind, int post_tw);
template <typename T>
bool any_rows_c2r_impl(mlc_ctx* ctx, const FftPlan2D& p, const void* in, void* out);
template <typename T, typename Loader>
bool any_rows_r2c_impl(mlc_ctx* ctx, const FftPlan2D& p, const Loader& ld, int nrows, void* out, const char* name);
bool any3_conv_fits(const FftPlan2D& p);
void any3_conv(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, void* out, const LimbSpectrum& rows, int h, lf3 r,
               int rexp);

template <typename T, bool INV>
bool limb_colpass_impl(mlc_ctx* ctx, const FftPlan2D& p, void* buf, char kind, int post_tw) {
  using S = typename LimbTraits<T>::S;
  const bool A = kind == 'A';
  const int L = A ? p.N1 : p.N2, nsets = A ? p.N2 : p.N1, tw_stride = A ? p.N2 : p.N1;
  const long set_mul = A ? 1 : p.N2, j_mul = A ? p.N2 : 1;
  using K = void (*)(C2<S>*, long, long, long, LimbTab<T>, int, int);
  K k = nullptr;
  int g = 0;
  switch (L) {
    case 100: k = k_limb_colpass2<S, T, limb_cw(10), 10, 10, INV>; g = 10; break;
    case 128: k = k_limb_colpass2<S, T, limb_cw(16), 8, 16, INV>; g = 16; break;
    case 64: k = k_limb_colpass2<S, T, limb_cw(8), 8, 8, INV>; g = 8; break;
    case 80: k = k_limb_colpass2<S, T, limb_cw(10), 8, 10, INV>; g = 10; break;
    case 50: k = k_limb_colpass2<S, T, limb_cw(10), 5, 10, INV>; g = 10; break;
    case 40: k = k_limb_colpass2<S, T, limb_cw(8), 5, 8, INV>; g = 8; break;
    default:
      return any_colpass_impl<INV>(ctx, p, buf, kind, post_tw);
  }
  const int cw = limb_cw(g);
  const size_t smem = LimbArr<T>::bytes(L * cw) + 2 * LimbArr<T>::bytes(L);
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, A ? "fft_col_A" : "fft_col_B");
    k<<<dim3(ceil_div(p.Wc, cw), nsets), g * cw, smem, ctx->stream>>>((C2<S>*)buf, p.Wp, set_mul, j_mul,
                                                                     limb_twy<T>(p), tw_stride, post_tw);
  }
  MLC_CHECK_LAUNCH();
  return true;
}

// P0's rows of an FP64 plan: the FP64 spectra, then their limbs (profile_rows_bytes).
inline LimbSpectrum limb3_profile_rows(const FftPlan2D& p, void* kx, int rows) {
  const size_t n = (size_t)rows * p.Wp;
  return LimbSpectrum((char*)kx + n * sizeof(C2<double>), n);
}

template <int MODE>
bool limb3_conv_impl(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, void* out, void* kx, int h, void* ks,
                     const char* name) {
  using K = void (*)(const C2<double>*, C2<double>*, long, LimbSpectrum, int, int, int, LimbTab<lf3>, lf3, int,
                     LimbSpectrum);
  K k = nullptr;
  int g = 0;
  switch (p.N2) {
    case 100: k = k_limb3_conv<limb_cw(10), 10, 10, MODE>; g = 10; break;
    case 128: k = k_limb3_conv<limb_cw(16), 8, 16, MODE>; g = 16; break;
    default: break;
  }
  if constexpr (MODE == 0) {
    switch (p.N2) {
      case 64: k = k_limb3_conv<limb_cw(8), 8, 8, MODE>; g = 8; break;
      case 80: k = k_limb3_conv<limb_cw(10), 8, 10, MODE>; g = 10; break;
      case 50: k = k_limb3_conv<limb_cw(10), 5, 10, MODE>; g = 10; break;
      case 40: k = k_limb3_conv<limb_cw(8), 5, 8, MODE>; g = 8; break;
      default: break;
    }
  }
  if (!k && !(MODE == 0 && any3_conv_fits(p))) return false;
  const LimbSpectrum rows = limb3_profile_rows(p, kx, 2 * h);
  if constexpr (MODE != 2) {
    MLC_KSCOPE(ctx, "conv_profile_columns");
    k_limb_profile_columns<16><<<ceil_div(p.Wc, 16), 256, 0, ctx->stream>>>((const C2<double>*)kx, p.Wp, 2 * h, rows.a,
                                                                           rows.b, rows.e);
  }
  MLC_CHECK_LAUNCH();
  // 1 / (Nx Ny) = r 2^-rexp with r in (1/2, 1]; its high limb a multiple of 2^-22, as a value's, for the
  // products with twiddles (both cut to 2^-24 only, their remainder had 25 bits: r W was off by 2^-49)
  const long double inv = 1.0L / ((long double)p.Nx * p.Ny);
  int e = 0;
  long double m = frexpl(inv, &e);
  const float a = (float)(rintl(m * 4194304.0L) / 4194304.0L);
  const float b = (float)(m - (long double)a);
  const lf3 r(a, b, (float)(m - (long double)a - (long double)b));
  if (!k) {
    any3_conv(ctx, p, Fmap, out, rows, h, r, -e);
    return true;
  }
  const int cw = limb_cw(g);
  const size_t smem = LimbArr<lf3>::bytes(p.N2 * cw) + 3 * LimbArr<lf3>::bytes(p.N2) + LimbArr<lf3>::bytes(p.N1);
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, name);
    k<<<dim3(ceil_div(p.Wc, cw), p.N1), g * cw, smem, ctx->stream>>>((const C2<double>*)Fmap, (C2<double>*)out, p.Wp,
                                                                    rows, h, p.Ny, p.N1, limb_twy<lf3>(p), r, -e,
                                                                    LimbSpectrum(ks, (size_t)p.Ny * p.Wp));
  }
  MLC_CHECK_LAUNCH();
  return true;
}

// Row lengths with a limb kernel (limb_first_radix lists them too), their radices and threads:
// f(levels, threads).
template <typename F>
static bool limb_row_dispatch(int M, F f) {
  using std::integral_constant;
  switch (M) {
    case 5000: f(Levels<10, 10, 10, 5>{}, integral_constant<int, 512>{}); return true;
    case 4096: f(Levels<8, 8, 8, 8>{}, integral_constant<int, 512>{}); return true;
    case 2000: f(Levels<8, 10, 5, 5>{}, integral_constant<int, 256>{}); return true;
    case 1000: f(Levels<10, 10, 10>{}, integral_constant<int, 128>{}); return true;
    default: return false;
  }
}

template <typename T>
bool limb_rows_c2r_impl(mlc_ctx* ctx, const FftPlan2D& p, const void* in, void* out) {
  using S = typename LimbTraits<T>::S;
  using TO = typename LimbTraits<T>::TO;
  const bool done = limb_row_dispatch(p.M, [&](auto lv, auto nt) {
    using LV = decltype(lv);
    auto k = k_limb_rows_c2r<S, T, TO, decltype(nt)::value, LV>;
    const size_t smem = limb_row_smem<T, LV>();
    set_max_smem((const void*)k, smem);
    {
      MLC_KSCOPE(ctx, "fft_rows_c2r");
      k<<<p.Ny, decltype(nt)::value, smem, ctx->stream>>>((const C2<S>*)in, p.Wp, (TO*)out, p.Nx, limb_twx<T>(p), limb_tab0<T>(p));
    }
    MLC_CHECK_LAUNCH();
  });
  return done || any_rows_c2r_impl<T>(ctx, p, in, out);
}

template <typename T>
bool limb_rows_c2r_il_impl(mlc_ctx* ctx, const FftPlan2D& p, const void* specs, long spec_stride, int nm, int S_,
                           void* out, unsigned planar) {
  using S = typename LimbTraits<T>::S;
  using TO = typename LimbTraits<T>::TO;
  return limb_row_dispatch(p.M, [&](auto lv, auto nt) {
    using LV = decltype(lv);
    auto k = k_limb_rows_c2r_il<S, T, TO, decltype(nt)::value, LV>;
    const size_t smem = limb_row_smem<T, LV>();
    set_max_smem((const void*)k, smem);
    {
      MLC_KSCOPE(ctx, "fft_rows_c2r_interleave");
      k<<<dim3(4 * ((nm + 3) / 4), p.Ny), decltype(nt)::value, smem, ctx->stream>>>(
          (const C2<S>*)specs, spec_stride, p.Wp, nm, (TO*)out, S_, limb_twx<T>(p), limb_tab0<T>(p), planar);
    }
    MLC_CHECK_LAUNCH();
  });
}

template <typename T, typename Loader>
bool limb_rows_r2c_impl(mlc_ctx* ctx, const FftPlan2D& p, const Loader& ld, int nrows, void* out, const char* name) {
  using S = typename LimbTraits<T>::S;
  const bool done = limb_row_dispatch(p.M, [&](auto lv, auto nt) {
    using LV = decltype(lv);
    auto k = k_limb_rows_r2c<S, T, decltype(nt)::value, LV, Loader>;
    const size_t smem = limb_row_smem<T, LV>();
    set_max_smem((const void*)k, smem);
    {
      MLC_KSCOPE(ctx, name);
      k<<<nrows, decltype(nt)::value, smem, ctx->stream>>>(ld, (C2<S>*)out, p.Wp, limb_twx<T>(p), limb_tab0<T>(p));
    }
    MLC_CHECK_LAUNCH();
  });
  return done || any_rows_r2c_impl<T>(ctx, p, ld, nrows, out, name);
}

}  // namespace mlc
