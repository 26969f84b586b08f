// FP32 and float-float passes of lengths without an unrolled kernel, by run-time radices
// (fft_any.cuh): the first level reads global memory, the last one writes it (rows, forward:
// the split's input in natural order), and only the levels between go through shared memory
// and back, in place.  The last level's items run in the order of their outputs, so that its
// stores are consecutive; the padded places keep its loads apart.
// Against the Stockham loop (a trip through shared memory per radix 2 to 8, twiddle powers by
// multiplication): FP32 convolutions of 4320^2 328 -> 269 us, 6000^2 391 -> 329, 9000^2 825 -> 583;
// FP64 maps in float-float 914 -> 774, 1436 -> 1191, 3321 -> 2478.
#pragma once

#include "fft_any.cuh"

namespace mlc {

template <bool INV, typename T>
__device__ __forceinline__ C2<T> any_tw(C2<T> v, C2<T> w) {
  return INV ? cmulc(v, w) : cmul(v, w);
}

// Level 0: load(index, column) for its inputs, results in place into s.
template <typename T, bool INV, int CW, typename Load>
__device__ __forceinline__ void any_first(C2<T>* s, const AnyLevels& lv, const C2<T>* __restrict__ tab, Load load) {
  any_radix(lv.r[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int bn = lv.bn[0], tn = lv.tn[0] * CW;
#pragma unroll 1
    for (int it = threadIdx.x; it < bn * CW; it += blockDim.x) {
      const int c = it % CW, m = it / CW;
      C2<T> u[R];
#pragma unroll
      for (int q = 0; q < R; q++) u[q] = load(m + bn * q, c);
      Dft<T, R, INV>::run(u);
      const int p = any_inner(lv, 1, m) * CW + c;
      s[p] = u[0];
#pragma unroll
      for (int q = 1; q < R; q++) s[p + q * tn] = any_tw<INV>(u[q], ldc(tab + (q - 1) * bn + m));
    }
  });
  __syncthreads();
}

// Levels 1 .. n - 2, in place.
template <typename T, bool INV, int CW>
__device__ __forceinline__ void any_middle(C2<T>* s, const AnyLevels& lv, const C2<T>* __restrict__ tab) {
#pragma unroll 1
  for (int i = 1; i < lv.n - 1; i++) {
    const C2<T>* t = tab + lv.tw[i];
    any_radix(lv.r[i], [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int bn = lv.bn[i], tn = lv.tn[i] * CW, items = lv.L / R * CW;
      const uint32_t mbn = lv.mbn[i];
#pragma unroll 1
      for (int it = threadIdx.x; it < items; it += blockDim.x) {
        const int c = it % CW, e = it / CW;
        const int blk = any_div(e, bn, mbn), m = e - blk * bn;
        C2<T>* x = s + (any_outer(lv, i, blk) + any_inner(lv, i + 1, m)) * CW + c;
        C2<T> u[R];
#pragma unroll
        for (int q = 0; q < R; q++) u[q] = x[q * tn];
        Dft<T, R, INV>::run(u);
        x[0] = u[0];
#pragma unroll
        for (int q = 1; q < R; q++) x[q * tn] = any_tw<INV>(u[q], ldc(t + (q - 1) * bn + m));
      }
    });
    __syncthreads();
  }
}

// The last level: put(index, column, value) with the outputs.
template <typename T, bool INV, int CW, typename Put>
__device__ __forceinline__ void any_last(const C2<T>* s, const AnyLevels& lv, Put put) {
  any_radix(lv.r[lv.n - 1], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int J = lv.L / R;
#pragma unroll 1
    for (int it = threadIdx.x; it < J * CW; it += blockDim.x) {
      const int c = it % CW, k = it / CW;
      const C2<T>* x = s + any_output(lv, k) * CW + c;
      C2<T> u[R];
#pragma unroll
      for (int q = 0; q < R; q++) u[q] = x[q * CW];
      Dft<T, R, INV>::run(u);
#pragma unroll
      for (int q = 0; q < R; q++) put(k + J * q, c, u[q]);
    }
  });
}

// Real transform of one row per CTA (k_rows_r2c's result).
template <typename T, typename Loader>
__global__ void __launch_bounds__(512) k_any_real_r2c(Loader ld, C2<T>* __restrict__ out, long pitch,
                                                      const C2<T>* __restrict__ twx,
                                                      const __grid_constant__ AnyLevels lv,
                                                      const C2<T>* __restrict__ tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* s = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* z = s + lv.places;
  const int M = lv.L, row = blockIdx.x;
  any_first<T, false, 1>(s, lv, tab, [&](int n, int) { return ld.pair(row, n); });
  any_middle<T, false, 1>(s, lv, tab);
  any_last<T, false, 1>(s, lv, [&](int k, int, C2<T> v) { z[k] = v; });
  __syncthreads();
  // X[M-k] of the pair has the conjugate sum and product: (conj s - i conj (W^k d)) / 2
  C2<T>* o = out + (long)row * pitch;
  for (int k = threadIdx.x; k <= M / 2; k += blockDim.x) {
    const C2<T> zk = z[k], zc = cconj(z[k == 0 ? 0 : M - k]);
    const C2<T> a = cadd(zk, zc);
    const C2<T> wd = cmul(ldc(twx + k), csub(zk, zc));
    o[k] = cfin(C2<T>{(T)0.5 * (a.x + wd.y), (T)0.5 * (a.y - wd.x)});
    if (k != M - k) o[M - k] = cfin(C2<T>{(T)0.5 * (a.x - wd.y), (T)0.5 * (-wd.x - a.y)});
  }
  for (int k = M + 1 + threadIdx.x; k < pitch; k += blockDim.x) o[k] = C2<T>{(T)0, (T)0};
}

// Inverse real transform of one row per CTA (k_rows_c2r's result).  The inputs of item j of
// level 0, k = j + J q, have their partners M - k in item J - j: a thread forms and transforms
// both.
template <typename T, typename TO>
__global__ void __launch_bounds__(512) k_any_real_c2r(const C2<T>* __restrict__ in, long pitch, TO* __restrict__ out,
                                                      long ldo, const C2<T>* __restrict__ twx,
                                                      const __grid_constant__ AnyLevels lv,
                                                      const C2<T>* __restrict__ tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* s = reinterpret_cast<C2<T>*>(smem_raw);
  const C2<T>* a = in + (long)blockIdx.x * pitch;
  any_radix(lv.r[0], [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int J = lv.bn[0], tn = lv.tn[0];
#pragma unroll 1
    for (int j = threadIdx.x; j <= J / 2; j += blockDim.x) {
      C2<T> u[R], v[R];
#pragma unroll
      for (int q = 0; q < R; q++) {
        const int k = j + J * q;
        const C2<T> xk = ldc(a + k), xm = cconj(ldc(a + (lv.L - k)));
        const C2<T> e = cadd(xk, xm), o = cmulc(csub(xk, xm), ldc(twx + k));  // (X - conj X') W^-k
        u[q] = C2<T>{e.x - o.y, e.y + o.x};
        v[R - 1 - q] = C2<T>{e.x + o.y, o.x - e.y};
      }
#pragma unroll
      for (int side = 0; side < 2; side++) {
        C2<T>* z = side ? v : u;
        const int m = side ? J - j : j;
        if (side && (j == 0 || 2 * j == J)) continue;  // items 0 and J / 2 are their own partners
        Dft<T, R, true>::run(z);
        const int p = any_inner(lv, 1, m);
        s[p] = z[0];
#pragma unroll
        for (int q = 1; q < R; q++) s[p + q * tn] = cmulc(z[q], ldc(tab + (q - 1) * J + m));
      }
    }
  });
  __syncthreads();
  any_middle<T, true, 1>(s, lv, tab);
  C2<TO>* dst = reinterpret_cast<C2<TO>*>(out + (long)blockIdx.x * ldo);
  any_last<T, true, 1>(s, lv, [&](int n, int, C2<T> z) { dst[n] = C2<TO>{out_cvt<TO>(z.x), out_cvt<TO>(z.y)}; });
}

// Column sub-pass (k_colpass): a strip of 16 columns per CTA.
constexpr int ANY_REAL_CW = 16;
template <typename T, bool INV>
__global__ void __launch_bounds__(256) k_any_real_colpass(C2<T>* __restrict__ buf, long pitch, long set_mul, long j_mul,
                                                          const C2<T>* __restrict__ twy, int post_tw,
                                                          const __grid_constant__ AnyLevels lv,
                                                          const C2<T>* __restrict__ tab) {
  constexpr int CW = ANY_REAL_CW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* s = reinterpret_cast<C2<T>*>(smem_raw);
  const int set = blockIdx.y;
  C2<T>* b = buf + (long)set * set_mul * pitch + (long)blockIdx.x * CW;
  any_first<T, INV, CW>(s, lv, tab, [&](int j, int c) { return b[(long)j * j_mul * pitch + c]; });
  any_middle<T, INV, CW>(s, lv, tab);
  any_last<T, INV, CW>(s, lv, [&](int j, int c, C2<T> v) {
    if (post_tw) v = any_tw<INV>(v, ldc(twy + (long)set * j));  // set*j < Ny
    b[(long)j * j_mul * pitch + c] = cfin(v);
  });
}

// ---------------------------------------------------------------- launches

template <typename T>
constexpr int any_real_resident() {  // threads an SM holds by their registers
  return std::is_same<T, float>::value ? 1024 : 512;
}

// Six CTAs or fewer per SM (the rows of a profile, small maps): the Stockham loops' short code and
// 512 threads a row finish first.  Float-float profile rows of 1500 and 4500 points 16 and 32 us
// against 42 and 54; six last passes of 810^2 174 against 208 us, of 1080^2 258 against 192; FP32
// is equal at 810^2, and 10 against 8 us a column pass at 1000^2.
static bool any_real_many(mlc_ctx* ctx, long ctas) { return ctas > 6L * ctx->sm_count; }

template <typename T, typename Loader>
bool any_real_r2c(mlc_ctx* ctx, const FftPlan2D& p, const Loader& ld, int nrows, void* out, const char* name) {
  const AnyLevels& lv = p.anyM;
  const size_t smem = ((size_t)lv.places + lv.L) * sizeof(C2<T>);
  if (lv.n < 2 || smem > ANY_SMEM || !any_real_many(ctx, nrows)) return false;
  auto k = k_any_real_r2c<T, Loader>;
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, name);
    k<<<nrows, any_row_threads(ctx, lv, smem, nrows, any_real_resident<T>()), smem, ctx->stream>>>(
        ld, (C2<T>*)out, p.Wp, (const C2<T>*)p.twx, lv, (const C2<T>*)p.anyM_tw);
  }
  MLC_CHECK_LAUNCH();
  return true;
}

template <typename T, typename TO>
bool any_real_c2r(mlc_ctx* ctx, const FftPlan2D& p, const void* in, void* out) {
  const AnyLevels& lv = p.anyM;
  const size_t smem = (size_t)lv.places * sizeof(C2<T>);
  if (lv.n < 2 || smem > ANY_SMEM || !any_real_many(ctx, p.Ny)) return false;
  auto k = k_any_real_c2r<T, TO>;
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, "fft_rows_c2r");
    k<<<p.Ny, any_row_threads(ctx, lv, smem, p.Ny, any_real_resident<T>()), smem, ctx->stream>>>(
        (const C2<T>*)in, p.Wp, (TO*)out, p.Nx, (const C2<T>*)p.twx, lv, (const C2<T>*)p.anyM_tw);
  }
  MLC_CHECK_LAUNCH();
  return true;
}

template <typename T, bool INV>
bool any_real_colpass(mlc_ctx* ctx, const FftPlan2D& p, void* buf, char kind, int post_tw) {
  const bool A = kind == 'A';
  const AnyLevels& lv = A ? p.any1 : p.any2;
  const size_t smem = (size_t)lv.L * ANY_REAL_CW * sizeof(C2<T>);
  const dim3 grid(ceil_div(p.Wc, ANY_REAL_CW), A ? p.N2 : p.N1);
  if (lv.n < 2 || smem > ANY_SMEM || !any_real_many(ctx, (long)grid.x * grid.y)) return false;
  auto k = k_any_real_colpass<T, INV>;
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, A ? "fft_col_A" : "fft_col_B");
    k<<<grid, any_col_threads(lv, ANY_REAL_CW, 256), smem, ctx->stream>>>(
        (C2<T>*)buf, p.Wp, A ? 1 : p.N2, A ? p.N2 : 1, (const C2<T>*)p.twy, post_tw, lv,
        (const C2<T>*)(A ? p.any1_tw : p.any2_tw));
  }
  MLC_CHECK_LAUNCH();
  return true;
}

}  // namespace mlc
