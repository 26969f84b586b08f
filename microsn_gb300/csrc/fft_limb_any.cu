// The limb passes (fft_limb.cuh) for lengths without an unrolled kernel: in-place transforms in
// shared memory by the radices of AnyLevels, chosen at run time, 2 to 10.  The small transforms
// are unrolled; the places of their points come from a few integer multiplications per item,
// little beside the arithmetic of its points.  Inputs wait in shared memory, as they were read,
// for the sum that scales them.
#include "fft_any.cuh"
#include "fft_limb.cuh"

namespace mlc {

// Level i, radix R, over CW interleaved columns.  DIT false: the small transform, then the
// twiddles; true (the way back, levels in the opposite order): conjugate twiddles, then it.
// grow: the factor to the level's scale (rows), 1 where it stays.
template <typename T, bool INV, bool DIT, int R, int CW, typename Tw>
__device__ __forceinline__ void any_level(const LimbArr<T>& s, const AnyLevels& lv, int i, float grow, Tw tw) {
  const int bn = lv.bn[i], tn = lv.tn[i] * CW, items = lv.L / R * CW;
  const bool last = i == lv.n - 1;
  const uint32_t mbn = lv.mbn[i];
#pragma unroll 1
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const int c = it % CW, e = it / CW;
    const int blk = any_div(e, bn, mbn), m = e - blk * bn;
    const int p = (any_outer(lv, i, blk) + any_inner(lv, i + 1, m)) * CW + c;
    C2<T> u[R];
#pragma unroll
    for (int q = 0; q < R; q++) u[q] = s.ld(p + q * tn);
    if (CW == 1 && grow != 1.f) {
#pragma unroll
      for (int q = 0; q < R; q++) u[q] = cscale2(u[q], grow);
    }
    if (DIT) {
      u[0] = limb_cnorm(u[0]);
      if (!last) {
#pragma unroll
        for (int q = 1; q < R; q++) u[q] = limb_tw<INV>(u[q], tw((q - 1) * bn + m));
      }
    }
    Dft<T, R, INV>::run(u);
    if (!DIT && !last) {
      s.st(p, limb_cnorm(u[0]));
#pragma unroll
      for (int q = 1; q < R; q++) s.st(p + q * tn, limb_tw<INV>(u[q], tw((q - 1) * bn + m)));
    } else {
#pragma unroll
      for (int q = 0; q < R; q++) s.st(p + q * tn, u[q]);
    }
  }
  __syncthreads();
}

template <typename T, bool INV, bool DIT, int CW, typename Tw>
__device__ __forceinline__ void any_level_r(const LimbArr<T>& s, const AnyLevels& lv, int i, float grow, Tw tw) {
  any_radix(lv.r[i], [&](auto r) { any_level<T, INV, DIT, decltype(r)::value, CW>(s, lv, i, grow, tw); });
}

// All levels: natural order in, digit order out (DIT: the other way round).  Level 0's twiddles
// straight from the table for rows (w holds the deeper levels'), else all from w.
template <typename T, bool INV>
__device__ __forceinline__ void any_row_transform(const LimbArr<T>& s, const AnyLevels& lv, const LimbTab<T>& tab,
                                                  const LimbArr<T>& w, LimbGrow& grow) {
  const int w0 = lv.n > 1 ? lv.tw[1] : 0;
#pragma unroll 1
  for (int i = 0; i < lv.n; i++) {
    const int at = lv.tw[i];
    if (i == 0) any_level_r<T, INV, false, 1>(s, lv, i, 1.f, [&](int e) { return tab.ld(e); });
    else any_level_r<T, INV, false, 1>(s, lv, i, grow.next(lv.r[i]), [&](int e) { return w.ld(at - w0 + e); });
  }
}
template <typename T, bool INV, bool DIT, int CW>
__device__ __forceinline__ void any_transform(const LimbArr<T>& s, const AnyLevels& lv, const LimbArr<T>& w) {
#pragma unroll 1
  for (int l = 0; l < lv.n; l++) {
    const int i = DIT ? lv.n - 1 - l : l;
    const int at = lv.tw[i];
    any_level_r<T, INV, DIT, CW>(s, lv, i, 1.f, [&](int e) { return w.ld(at + e); });
  }
}

// ---------------------------------------------------------------- rows

__device__ __forceinline__ LimbPeak any_block_peak(LimbPeak v, LimbPeak* red) {
  v = limb_peak_warp(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  LimbPeak all = red[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); w++) all = limb_peak_add(all, red[w]);
  return all;
}
template <typename S>
__device__ __forceinline__ LimbSum<S> limb_sum_zero();
template <>
__device__ __forceinline__ LimbSum<double> limb_sum_zero() { return LimbSum<double>{0, 0.f}; }

template <typename T>
__device__ __forceinline__ void any_fill_deep(const LimbArr<T>& w, const AnyLevels& lv, const LimbTab<T>& tab) {
  const int w0 = lv.n > 1 ? lv.tw[1] : 0, nw = lv.n > 1 ? lv.ntw - w0 : 0;
  for (int e = threadIdx.x; e < nw; e += blockDim.x) w.st(e, tab.ld(w0 + e));
}
template <typename T>
static size_t any_row_smem(const AnyLevels& lv) {
  return LimbArr<T>::bytes(lv.places) + LimbArr<T>::bytes(lv.n > 1 ? lv.ntw - lv.tw[1] : 0);
}

template <typename S, typename T, typename TO>
__global__ void __launch_bounds__(512)
    k_any_rows_c2r(const C2<S>* __restrict__ in, long pitch, TO* __restrict__ out, long ldo, LimbTab<T> twx,
                   const __grid_constant__ AnyLevels lv, LimbTab<T> tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LimbPeak red[512 / 32];
  const int M = lv.L, tid = threadIdx.x, NT = blockDim.x;
  const LimbArr<T> s = LimbArr<T>::at(smem_raw, lv.places);
  const LimbArr<T> w = LimbArr<T>::at(smem_raw + LimbArr<T>::bytes(lv.places), lv.n > 1 ? lv.ntw - lv.tw[1] : 0);
  const C2<S>* a = in + (long)blockIdx.x * pitch;
  LimbPeak peak{0, 0.f, 0.f};
  C2<S>* raw = reinterpret_cast<C2<S>*>(smem_raw);  // 16 bytes a value, as the limbs' first plane
  C2<S> top{S(0.0), S(0.0)};                        // X[M], beside X[0] of thread 0
  for (int k0 = tid; k0 <= M / 2; k0 += 2 * NT) {  // (the loads of a round are in flight together)
    C2<S> v[4];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int k = k0 + i * NT;
      v[2 * i] = k <= M / 2 ? ldc(a + k) : C2<S>{S(0.0), S(0.0)};
      v[2 * i + 1] = k <= M / 2 ? ldc(a + (M - k)) : C2<S>{S(0.0), S(0.0)};
    }
    peak = limb_peak_add(peak, limb_peak<4, 2>(v));
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int k = k0 + i * NT;
      if (k > M / 2) break;
      raw[any_inner(lv, 0, k)] = v[2 * i];
      if (k > 0) raw[any_inner(lv, 0, M - k)] = v[2 * i + 1];
      else top = v[2 * i + 1];
    }
  }
  any_fill_deep(w, lv, tab);
  // |b[k]| + |b[M-k]| <= 2 sqrt(2) (|X[k]| + |X[M-k]|), and each of them <= 2 (|X[k]| + |X[M-k]|)
  LimbGrow grow = LimbGrow::of(any_block_peak(peak, red), 2.82843f, 2.f);
  const LimbScale<T> sc = grow.first(lv.r[0]);
  for (int k = tid; k <= M / 2; k += NT) {
    C2<T> bk, bm;
    const int pk = any_inner(lv, 0, k), pm = k > 0 ? any_inner(lv, 0, M - k) : 0;
    C2<S> x[2] = {raw[pk], k > 0 ? raw[pm] : top};
    const LimbScale<T> si = limb_lift<2>(x, sc);
    limb_c2r_pair(limb_cin(x[0], si), cconj(limb_cin(x[1], si)), twx.ld(k), bk, bm);
    s.st(pk, bk);
    if (k > 0 && k != M - k) s.st(pm, bm);
  }
  __syncthreads();
  any_row_transform<T, true>(s, lv, tab, w, grow);
  const LimbScale<T> so = grow.scale();
  C2<TO>* dst = reinterpret_cast<C2<TO>*>(out + (long)blockIdx.x * ldo);
  for (int n = tid; n < M; n += NT) {
    const C2<T> z = s.ld(any_output(lv, n));
    dst[n] = C2<TO>{limb_round(z.x, so), limb_round(z.y, so)};
  }
}

template <typename S, typename T, typename Loader>
__global__ void __launch_bounds__(512)
    k_any_rows_r2c(Loader ld, C2<S>* __restrict__ out, long pitch, LimbTab<T> twx,
                   const __grid_constant__ AnyLevels lv, LimbTab<T> tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LimbPeak red[512 / 32];
  const int M = lv.L, tid = threadIdx.x, NT = blockDim.x, row = blockIdx.x;
  const LimbArr<T> s = LimbArr<T>::at(smem_raw, lv.places);
  const LimbArr<T> w = LimbArr<T>::at(smem_raw + LimbArr<T>::bytes(lv.places), lv.n > 1 ? lv.ntw - lv.tw[1] : 0);
  LimbPeak peak{0, 0.f, 0.f};
  C2<S>* raw = reinterpret_cast<C2<S>*>(smem_raw);
  for (int n0 = tid; n0 < M; n0 += 4 * NT) {  // (the loads of a round are in flight together)
    C2<S> v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = n0 + i * NT < M ? ld.pair(row, n0 + i * NT) : C2<S>{S(0.0), S(0.0)};
    peak = limb_peak_add(peak, limb_peak<4, 1>(v));
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (n0 + i * NT < M) raw[any_inner(lv, 0, n0 + i * NT)] = v[i];
  }
  any_fill_deep(w, lv, tab);
  LimbGrow grow = LimbGrow::of(any_block_peak(peak, red), 1.f, 1.f);
  const LimbScale<T> sc = grow.first(lv.r[0]);
  for (int n = tid; n < M; n += NT) {
    const int p = any_inner(lv, 0, n);
    C2<S> x = raw[p];
    const LimbScale<T> si = limb_lift<1>(&x, sc);
    s.st(p, limb_cin(x, si));
  }
  __syncthreads();
  any_row_transform<T, false>(s, lv, tab, w, grow);
  // the split of k_limb_rows_r2c
  C2<S>* o = out + (long)row * pitch;
  const LimbScale<T> so = grow.scale();
  for (int k = tid; k <= M / 2; k += NT) {
    const C2<T> zk = cscale2(s.ld(any_output(lv, k)), 0.5f);
    const C2<T> zc = cconj(cscale2(s.ld(k == 0 ? any_output(lv, 0) : any_output(lv, M - k)), 0.5f));
    const C2<T> a = cadd(zk, zc);
    const C2<T> wd = limb_tw<false>(csub(zk, zc), twx.ld(k));
    o[k] = limb_cout<S>(C2<T>{a.x + wd.y, a.y - wd.x}, so);
    if (k != M - k) o[M - k] = limb_cout<S>(C2<T>{a.x - wd.y, -wd.x - a.y}, so);
  }
  for (int k = M + 1 + tid; k < pitch; k += NT) o[k] = C2<S>{S(0.0), S(0.0)};
}

// ---------------------------------------------------------------- columns

constexpr int ANY_CW = 16, ANY_NT = 256, ANY_G = ANY_NT / ANY_CW;  // (threads at most)

// Sum of each column of a tile over the CTA: the threads of column c hold partial sums.
template <typename S>
__device__ __forceinline__ LimbSum<S> any_column_sum(LimbSum<S> v, LimbSum<S> (*red)[ANY_CW]) {
  const int c = threadIdx.x % ANY_CW, g = threadIdx.x / ANY_CW;
  red[g][c] = v;
  __syncthreads();
  LimbSum<S> sum = red[0][c];
  for (int q = 1; q < (int)blockDim.x / ANY_CW; q++) sum = limb_sum_add(sum, red[q][c]);
  return sum;
}

template <typename S, typename T, bool INV>
__global__ void __launch_bounds__(ANY_NT, 2)
    k_any_colpass(C2<S>* __restrict__ buf, long pitch, long set_mul, long j_mul, LimbTab<T> twy, int post_tw,
                  const __grid_constant__ AnyLevels lv, LimbTab<T> tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LimbSum<S> red[ANY_G][ANY_CW];
  const int L = lv.L, set = blockIdx.y;
  const int c = threadIdx.x % ANY_CW, g = threadIdx.x / ANY_CW, G = blockDim.x / ANY_CW;
  const LimbArr<T> s = LimbArr<T>::at(smem_raw, L * ANY_CW);
  const LimbArr<T> w = LimbArr<T>::at(smem_raw + LimbArr<T>::bytes(L * ANY_CW), lv.ntw);
  C2<S>* b = buf + (long)set * set_mul * pitch + (long)blockIdx.x * ANY_CW + c;
  LimbSum<S> sum = limb_sum_zero<S>();
  C2<S>* raw = reinterpret_cast<C2<S>*>(smem_raw);  // 16 bytes a value, as the limbs' first plane
  for (int j0 = g; j0 < L; j0 += 8 * G) {  // (the loads of a round are in flight together)
    C2<S> v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int j = j0 + i * G;
      v[i] = j < L ? b[(long)j * j_mul * pitch] : C2<S>{S(0.0), S(0.0)};
    }
    sum = limb_sum_add(sum, limb_sum<8>(v));
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (j0 + i * G < L) raw[(j0 + i * G) * ANY_CW + c] = v[i];
  }
  for (int e = threadIdx.x; e < lv.ntw; e += blockDim.x) w.st(e, tab.ld(e));
  const LimbScale<T> sc = limb_scale(any_column_sum(sum, red));
  for (int j = g; j < L; j += G) {
    C2<S> x = raw[j * ANY_CW + c];
    const LimbScale<T> si = limb_lift<1>(&x, sc);
    s.st(j * ANY_CW + c, limb_cin(x, si));
  }
  __syncthreads();
  any_transform<T, INV, false, ANY_CW>(s, lv, w);
  for (int j = g; j < L; j += G) {
    C2<T> v = s.ld(any_output(lv, j) * ANY_CW + c);
    if (post_tw) v = limb_tw<INV>(v, twy.ld((long)set * j));  // set*j < Ny
    b[(long)j * j_mul * pitch] = limb_cout<S>(v, sc);
  }
}

// P1 of FP64 plans (k_limb3_conv, mode 0): forward levels leave the profile's spectrum in digit
// order, where the product with the map's (read at the frequency of each place) is taken, and
// the levels in the opposite order lead back to rows in natural order.
__global__ void __launch_bounds__(ANY_NT, 2)
    k_any_conv(const C2<double>* __restrict__ Fmap, C2<double>* __restrict__ out, long pitch, LimbSpectrum kx, int h,
               int Ny, int N1, LimbTab<lf3> twy, lf3 r, int rexp, const __grid_constant__ AnyLevels lv,
               LimbTab<lf3> tab) {
  using T = lf3;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LimbSum<double> red[ANY_G][ANY_CW];
  const int N2 = lv.L, kk = blockIdx.y;
  const int c = threadIdx.x % ANY_CW, g = threadIdx.x / ANY_CW, G = blockDim.x / ANY_CW;
  const LimbArr<T> s = LimbArr<T>::at(smem_raw, N2 * ANY_CW);
  const LimbArr<T> w = LimbArr<T>::at(smem_raw + LimbArr<T>::bytes(N2 * ANY_CW), lv.ntw);
  const long col = (long)blockIdx.x * ANY_CW + c;
  const C2<double>* f = Fmap + (long)kk * N2 * pitch + col;
  LimbSum<double> sum = limb_sum_zero<double>();
#pragma unroll 4
  for (int k2 = g; k2 < N2; k2 += G) {
    const C2<double> v = ldc(f + (long)k2 * pitch);
    sum = limb_sum_add(sum, limb_sum<1>(&v));
  }
  for (int e = threadIdx.x; e < lv.ntw; e += blockDim.x) w.st(e, tab.ld(e));
  int ke = kx.e[col];
  if (ke != LIMB_BAD) ke -= rexp;
  // the profile's column sub-pass over its non-zero rows, then W_Ny^(n2 kk) r
  for (int n2 = g; n2 < N2; n2 += G) {
    C2<T> acc = n2 < h ? kx.ld((long)n2 * pitch + col) : limb_zero<T>();  // weight W^0 = 1
#pragma unroll 1
    for (int n1 = 1; n1 * N2 + n2 < h; n1++)
      acc = cadd(acc, limb_tw<false>(kx.ld((long)(n1 * N2 + n2) * pitch + col), twy.ld((long)((n1 * kk) % N1) * N2)));
#pragma unroll 1
    for (int n1 = max((Ny - h - n2 + N2 - 1) / N2, 0); n1 < N1; n1++)
      acc = cadd(acc, limb_tw<false>(kx.ld((n1 * N2 + n2 - (Ny - 2L * h)) * pitch + col),
                                           twy.ld((long)((n1 * kk) % N1) * N2)));
    const C2<T> t = twy.ld((long)n2 * kk);
    s.st(n2 * ANY_CW + c, limb_tw<false>(acc, limb_cnorm(C2<T>{r * t.x, r * t.y})));
  }
  const LimbScale<T> sf = limb_scale(any_column_sum(sum, red));  // (its barrier also ends the writes of s and w)
  any_transform<T, false, false, ANY_CW>(s, lv, w);
  for (int k2 = g; k2 < N2; k2 += G) {
    const int p = any_output(lv, k2) * ANY_CW + c;
    C2<double> x = ldc(f + (long)k2 * pitch);
    const LimbScale<T> si = limb_lift<1>(&x, sf);
    s.st(p, limb_tw<false>(limb_cin(x, si), limb_cnorm(s.ld(p))));
  }
  __syncthreads();
  any_transform<T, true, true, ANY_CW>(s, lv, w);
  LimbScale<T> sc = sf;
  sc.bad |= ke == LIMB_BAD;  // the scales multiply: exponents add
  sc.e += sc.bad ? 0 : ke;
  for (int n2 = g; n2 < N2; n2 += G)
    out[((long)kk * N2 + n2) * pitch + col] =
        limb_cout<double>(limb_tw<true>(s.ld(n2 * ANY_CW + c), twy.ld((long)n2 * kk)), sc);
}

// ---------------------------------------------------------------- launches

template <typename T>
static LimbTab<T> any_tab(const FftPlan2D& p, const AnyLevels& lv, const void* t) {
  return LimbTraits<T>::tab(p, t, t, lv.ntw);
}

template <typename T>
static int any_limb_row_threads(mlc_ctx* ctx, const AnyLevels& lv, size_t smem, int nrows) {
  return any_row_threads(ctx, lv, smem, nrows, 512);
}

template <typename T>
bool any_rows_c2r_impl(mlc_ctx* ctx, const FftPlan2D& p, const void* in, void* out) {
  using S = typename LimbTraits<T>::S;
  using TO = typename LimbTraits<T>::TO;
  const AnyLevels& lv = p.anyM;
  const size_t smem = any_row_smem<T>(lv);
  if (lv.n < 1 || smem > ANY_SMEM) return false;
  auto k = k_any_rows_c2r<S, T, TO>;
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, "fft_rows_c2r");
    k<<<p.Ny, any_limb_row_threads<T>(ctx, lv, smem, p.Ny), smem, ctx->stream>>>((const C2<S>*)in, p.Wp, (TO*)out, p.Nx, limb_twx<T>(p), lv,
                                                         any_tab<T>(p, lv, p.anyM_tw));
  }
  MLC_CHECK_LAUNCH();
  return true;
}

template <typename T, typename Loader>
bool any_rows_r2c_impl(mlc_ctx* ctx, const FftPlan2D& p, const Loader& ld, int nrows, void* out, const char* name) {
  using S = typename LimbTraits<T>::S;
  const AnyLevels& lv = p.anyM;
  const size_t smem = any_row_smem<T>(lv);
  if (lv.n < 1 || smem > ANY_SMEM) return false;
  // one row per SM at most (a profile's): the FP64 loop's short code finishes first up to here
  // (rows of 1200 points 30 us against 47, of 2160 points 55 either way, of 4500 points 102 against 70)
  if (nrows <= ctx->sm_count && p.M <= 2000) return false;
  auto k = k_any_rows_r2c<S, T, Loader>;
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, name);
    k<<<nrows, any_limb_row_threads<T>(ctx, lv, smem, nrows), smem, ctx->stream>>>(ld, (C2<S>*)out, p.Wp, limb_twx<T>(p), lv,
                                                          any_tab<T>(p, lv, p.anyM_tw));
  }
  MLC_CHECK_LAUNCH();
  return true;
}

template <bool INV>
bool any_colpass_impl(mlc_ctx* ctx, const FftPlan2D& p, void* buf, char kind, int post_tw) {
  using S = double;
  using T = lf3;
  const bool A = kind == 'A';
  const AnyLevels& lv = A ? p.any1 : p.any2;
  const size_t smem = LimbArr<T>::bytes((long)lv.L * ANY_CW) + LimbArr<T>::bytes(lv.ntw);
  if (lv.n < 1 || smem > ANY_SMEM) return false;
  auto k = k_any_colpass<S, T, INV>;
  set_max_smem((const void*)k, smem);
  {
    MLC_KSCOPE(ctx, A ? "fft_col_A" : "fft_col_B");
    k<<<dim3(ceil_div(p.Wc, ANY_CW), A ? p.N2 : p.N1), any_col_threads(lv, ANY_CW, ANY_NT), smem, ctx->stream>>>(
        (C2<S>*)buf, p.Wp, A ? 1 : p.N2, A ? p.N2 : 1, limb_twy<T>(p), post_tw, lv,
        any_tab<T>(p, lv, A ? p.any1_tw : p.any2_tw));
  }
  MLC_CHECK_LAUNCH();
  return true;
}

static size_t any3_conv_smem(const FftPlan2D& p) {
  return LimbArr<lf3>::bytes((long)p.N2 * ANY_CW) + LimbArr<lf3>::bytes(p.any2.ntw);
}
bool any3_conv_fits(const FftPlan2D& p) { return p.any2.n > 0 && any3_conv_smem(p) <= ANY_SMEM; }
void any3_conv(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, void* out, const LimbSpectrum& rows, int h, lf3 r,
               int rexp) {
  const AnyLevels& lv = p.any2;
  const size_t smem = any3_conv_smem(p);
  set_max_smem((const void*)k_any_conv, smem);
  {
    MLC_KSCOPE(ctx, "conv_fused_spectrum");
    k_any_conv<<<dim3(ceil_div(p.Wc, ANY_CW), p.N1), any_col_threads(lv, ANY_CW, ANY_NT), smem, ctx->stream>>>(
        (const C2<double>*)Fmap, (C2<double>*)out, p.Wp, rows, h, p.Ny, p.N1, limb_twy<lf3>(p), r, rexp, lv,
        any_tab<lf3>(p, lv, p.any2_tw));
  }
  MLC_CHECK_LAUNCH();
}

template bool any_colpass_impl<false>(mlc_ctx*, const FftPlan2D&, void*, char, int);
template bool any_colpass_impl<true>(mlc_ctx*, const FftPlan2D&, void*, char, int);
template bool any_rows_c2r_impl<lf3>(mlc_ctx*, const FftPlan2D&, const void*, void*);
template bool any_rows_r2c_impl<lf3, RealRows<double, double>>(mlc_ctx*, const FftPlan2D&,
                                                               const RealRows<double, double>&, int, void*, const char*);
template bool any_rows_r2c_impl<lf3, RealRows<double, float>>(mlc_ctx*, const FftPlan2D&,
                                                              const RealRows<double, float>&, int, void*, const char*);
template bool any_rows_r2c_impl<lf3, ProfileRows<double>>(mlc_ctx*, const FftPlan2D&, const ProfileRows<double>&, int,
                                                          void*, const char*);

}  // namespace mlc
