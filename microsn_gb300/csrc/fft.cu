// 2-D real FFTs and FFT convolution of a magnification map with a source profile.
//
// Replaces the reference's cuFFT D2Z/Z2D plans and kernel_multiplyFFTs
// (simulating_lcurves/src/gpu_functions.cu:150-200, 522-577) with hand-written passes:
//
//   forward(map):  R  rows, real FFT of length Nx (complex FFT of Nx/2 + split)
//                  A  columns, sub-pass over row sets {n1*N2 + n2}: length-N1 DFT, twiddle
//                  B  columns, sub-pass over row blocks {k1*N2 + n2}: length-N2 DFT
//     The spectrum is left in "digit-transposed" row order (row k1*N2 + k2 holds
//     frequency k1 + N1*k2); every consumer below works in that order, so no
//     reordering pass is ever made.
//
//   fused convolution per profile (MLC_CONV_FUSED):
//     P0  real FFT of the 2h non-zero rows of the wrapped profile only
//     P1  per (k1, strip): the profile's column spectrum for all k2 built in shared
//         memory (sub-pass A of the profile reduces to <= 2*ceil(h/N2) terms because
//         only rows [0,h) and [Ny-h,Ny) are non-zero), multiplied by the map spectrum
//         and by 1/(Nx Ny), then the inverse length-N2 sub-pass and its twiddle
//     P2  inverse sub-pass over row sets (length N1)
//     P3  inverse real FFT of each row (c2r)
//   plain convolution (MLC_CONV_PLAIN): full-size wrapped kernel, full forward,
//     pointwise multiply, full inverse -- one launch per stage, like the reference.
//
// This file holds the plans, the twiddle tables and the dispatch by precision; the
// kernels and launch sequences are in fft_impl.cuh.
#include <algorithm>
#include <cmath>
#include <functional>
#include <map>
#include <mutex>
#include <unordered_map>

#include "mlc_internal.h"

namespace mlc {

RadixList factor_radices(int L, int tw_stride) {
  RadixList rl{};
  rl.n = 0;
  rl.L = L;
  if (L < 1 || L > 65535) {
    rl.n = -1;
    return rl;
  }
  int n = L;
  while (n % 5 == 0) { rl.r[rl.n++] = 5; n /= 5; }
  while (n % 3 == 0) { rl.r[rl.n++] = 3; n /= 3; }
  int e2 = 0;
  while (n % 2 == 0) { e2++; n /= 2; }
  if (n != 1) {
    rl.n = -1;
    return rl;
  }
  int n8 = e2 / 3, rem = e2 % 3;
  if (rem == 1 && n8 > 0) {  // 8*2 -> 4*4
    n8--;
    rl.r[rl.n++] = 4;
    rl.r[rl.n++] = 4;
  } else if (rem == 1) {
    rl.r[rl.n++] = 2;
  } else if (rem == 2) {
    rl.r[rl.n++] = 4;
  }
  for (int i = 0; i < n8; i++) rl.r[rl.n++] = 8;
  int Ns = 1;
  rl.tlen = 0;
  for (int p = 0; p < rl.n; p++) {
    rl.Ns[p] = Ns;
    rl.toff[p] = rl.tlen;
    rl.tlen += p == 0 ? 0 : Ns * (rl.r[p] - 1);
    // exact j / Ns = umulhi(j, magic) for j * Ns < 2^32 (here j < L <= 65535)
    rl.magic[p] = Ns > 1 ? (uint32_t)((0x100000000ull + Ns - 1) / Ns) : 0u;
    rl.twstep[p] = (L / (Ns * rl.r[p])) * tw_stride;
    Ns *= rl.r[p];
  }
  return rl;
}

// Few and large radices: a level's twiddle products and its trip through shared memory cost more
// than the additions of a larger small transform.
AnyLevels any_levels(int L, bool pad) {
  AnyLevels lv;
  lv.L = L;
  if (L < 2 || L > 65535) return lv;
  int e2 = 0, e3 = 0, e5 = 0, n = L;
  while (n % 2 == 0) e2++, n /= 2;
  while (n % 3 == 0) e3++, n /= 3;
  while (n % 5 == 0) e5++, n /= 5;
  if (n != 1) return lv;
  std::vector<int> r;
  while (e2 > 0 && e5 > 0) r.push_back(10), e2--, e5--;
  while (e3 > 1) r.push_back(9), e3 -= 2;
  while (e2 > 2 && e2 != 4) r.push_back(8), e2 -= 3;
  while (e2 > 1) r.push_back(4), e2 -= 2;
  if (e2 > 0 && e3 > 0) r.push_back(6), e2--, e3--;
  for (; e5 > 0; e5--) r.push_back(5);
  for (; e3 > 0; e3--) r.push_back(3);
  for (; e2 > 0; e2--) r.push_back(2);
  std::sort(r.begin(), r.end(), std::greater<int>());
  if ((int)r.size() > AnyLevels::MAX) return lv;
  lv.n = (int)r.size();
  auto magic = [](int d) { return d > 1 ? (uint32_t)((0x100000000ull + d - 1) / d) : 0u; };
  int b = L;
  for (int i = 0; i < lv.n; i++) {
    lv.r[i] = r[i];
    b /= r[i];
    lv.bn[i] = b;
    lv.tw[i] = lv.ntw;
    if (i + 1 < lv.n) lv.ntw += (r[i] - 1) * b;
    lv.mr[i] = magic(r[i]);
    lv.mbn[i] = magic(b);
  }
  int t = 1;  // places of one sub-block, from the innermost outwards, odd where they are padded
  for (int i = lv.n - 1; i >= 0; i--) {
    lv.tn[i] = t;
    t *= r[i];
    if (pad && i > 0) t |= 1;
  }
  lv.places = t;
  return lv;
}

// The attribute belongs to the function on the current device: a process holding contexts
// on several GPUs sets it once per (device, function).
void set_max_smem(const void* func, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> done;
  int dev = 0;
  MLC_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(mu);
  const auto key = std::make_pair(dev, func);
  auto it = done.find(key);
  if (it != done.end() && it->second >= bytes) return;
  MLC_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  done[key] = bytes;
}

FftPlan2D::~FftPlan2D() {
  for (void* t : {twx, twy, twx3, twy3, twl3, twl, anyM_tw, any1_tw, any2_tw})
    if (t) cudaFree(t);
}

// exp(-2 pi i m / N), m in [0, N), evaluated in long double with the angle reduced to
// the first octant so that each entry is correctly rounded to FP64 in practice.
static void twiddle_table(int N, std::vector<long double>& re, std::vector<long double>& im) {
  re.resize(N);
  im.resize(N);
  const long double TWO_PI = 6.283185307179586476925286766559005768L;
  for (int m = 0; m < N; m++) {
    // reduce m/N to [0, 1/8] using the symmetries of cos/sin
    long q8 = (long)m * 8;  // octant index via integer arithmetic
    int oct = (int)(q8 / N);
    long double frac;  // angle fraction of a full turn within the octant frame
    long double c, s;
    // angle a = 2 pi m / N; write m/N = oct/8 + r with r in [0, 1/8)
    long double r = ((long double)m - (long double)oct * N / 8.0L) / N;
    (void)frac;
    long double a = TWO_PI * r;
    long double ca = cosl(a), sa = sinl(a);
    const long double h = 0.70710678118654752440084436210484903928L;
    // rotate by oct * 45 degrees
    switch (oct & 7) {
      case 0: c = ca; s = sa; break;
      case 1: c = h * (ca - sa); s = h * (ca + sa); break;
      case 2: c = -sa; s = ca; break;
      case 3: c = -h * (ca + sa); s = h * (ca - sa); break;
      case 4: c = -ca; s = -sa; break;
      case 5: c = -h * (ca - sa); s = -h * (ca + sa); break;
      case 6: c = sa; s = -ca; break;
      default: c = h * (ca + sa); s = -h * (ca - sa); break;
    }
    // exact values where they are known
    if ((long)m * 4 % N == 0) {
      long k = (long)m * 4 / N;
      c = (k == 0) ? 1 : (k == 2) ? -1 : 0;
      s = (k == 1) ? 1 : (k == 3) ? -1 : 0;
    }
    re[m] = c;
    im[m] = -s;  // forward sign
  }
}

template <typename T>
static void* upload_twiddles(int N) {
  std::vector<long double> re, im;
  twiddle_table(N, re, im);
  std::vector<C2<T>> h(N);
  for (int m = 0; m < N; m++) h[m] = C2<T>{(T)(double)re[m], (T)(double)im[m]};
  void* d = nullptr;
  MLC_CUDA(cudaMalloc(&d, sizeof(C2<T>) * N));
  MLC_CUDA(cudaMemcpy(d, h.data(), sizeof(C2<T>) * N, cudaMemcpyHostToDevice));
  return d;
}

// The same table in three limbs: a plane of (re, im) high and middle limbs, then one of low
// limbs.  The high limb is cut to multiples of 2^-24 (limb.cuh); the sum keeps what long
// double holds on this host (64 bits or more).
static void* upload_limbs3(const std::vector<long double>& re, const std::vector<long double>& im) {
  const size_t N = re.size();
  std::vector<float> h(N * 6);
  float* lo = h.data() + N * 4;
  for (size_t m = 0; m < N; m++)
    for (int k = 0; k < 2; k++) {
      const long double v = k ? im[m] : re[m];
      const float a = (float)(rintl(v * 16777216.0L) / 16777216.0L);
      const float b = (float)(v - (long double)a);
      h[m * 4 + k] = a;
      h[m * 4 + 2 + k] = b;
      lo[m * 2 + k] = (float)(v - (long double)a - (long double)b);
    }
  void* d = nullptr;
  MLC_CUDA(cudaMalloc(&d, h.size() * sizeof(float)));
  MLC_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(float), cudaMemcpyHostToDevice));
  return d;
}
static void* upload_twiddles3(int N) {
  std::vector<long double> re, im;
  twiddle_table(N, re, im);
  return upload_limbs3(re, im);
}
// Level 0 of the row transforms: W_M^(m q) for q = 1 .. R0 - 1, m < M / R0.
static void level0_table(int M, int R0, std::vector<long double>& lr, std::vector<long double>& li) {
  const int J = M / R0;
  std::vector<long double> re, im;
  twiddle_table(M, re, im);
  for (int q = 1; q < R0; q++)
    for (int m = 0; m < J; m++) {
      lr.push_back(re[(size_t)m * q]);
      li.push_back(im[(size_t)m * q]);
    }
}
static void* upload_level0_limbs3(int M) {
  std::vector<long double> lr, li;
  level0_table(M, limb_first_radix(M), lr, li);
  return upload_limbs3(lr, li);
}
static void* upload_level0_f32(int M) {
  std::vector<long double> lr, li;
  level0_table(M, row3_first_radix(M), lr, li);
  std::vector<C2<float>> h(lr.size());
  for (size_t i = 0; i < h.size(); i++) h[i] = C2<float>{(float)(double)lr[i], (float)(double)li[i]};
  void* d = nullptr;
  MLC_CUDA(cudaMalloc(&d, h.size() * sizeof(C2<float>)));
  MLC_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(C2<float>), cudaMemcpyHostToDevice));
  return d;
}

// The levels' twiddles W_{B_i}^(m q), [q - 1][m], one level after another, in the plan's own
// arithmetic (FP64: three limbs).
static void* upload_any(const AnyLevels& lv, int prec) {
  if (lv.n < 2) return nullptr;
  std::vector<long double> re, im, lr, li;
  twiddle_table(lv.L, re, im);
  int f = 1;  // W_{B_i} = W_L^f
  for (int i = 0; i + 1 < lv.n; i++) {
    for (int q = 1; q < lv.r[i]; q++)
      for (int m = 0; m < lv.bn[i]; m++) {
        lr.push_back(re[(size_t)m * q * f]);
        li.push_back(im[(size_t)m * q * f]);
      }
    f *= lv.r[i];
  }
  if (prec == MLC_F64) return upload_limbs3(lr, li);
  auto upload = [&](auto zero) {
    using T = decltype(zero);
    std::vector<C2<T>> h(lr.size());
    for (size_t i = 0; i < h.size(); i++) h[i] = C2<T>{T((double)lr[i]), T((double)li[i])};
    void* d = nullptr;
    MLC_CUDA(cudaMalloc(&d, h.size() * sizeof(C2<T>)));
    MLC_CUDA(cudaMemcpy(d, h.data(), h.size() * sizeof(C2<T>), cudaMemcpyHostToDevice));
    return d;
  };
  return prec_is_ff(prec) ? upload(ff(0.0)) : upload(0.f);
}

static void split_columns(int Ny, int& N1, int& N2) {
  int best = 1;
  for (int d = 1; (long)d * d <= Ny; d++)
    if (Ny % d == 0) best = d;
  N1 = best;
  N2 = Ny / best;
}

FftPlan2D* plan_get(mlc_ctx* ctx, int Nx, int Ny, int prec) {
  auto key = std::make_tuple(Nx, Ny, prec);
  auto it = ctx->plans.find(key);
  if (it != ctx->plans.end()) return it->second.get();
  MLC_REQUIRE(Nx >= 4 && Ny >= 2 && Nx % 2 == 0, MLC_ERR_ARG, "map sides must be even, Nx >= 4");
  std::unique_ptr<FftPlan2D> p(new FftPlan2D());
  p->Nx = Nx;
  p->Ny = Ny;
  p->prec = prec;
  p->M = Nx / 2;
  p->Wc = Nx / 2 + 1;
  p->Wp = (int)round_up(p->Wc, 16);
  p->elem = prec == MLC_F64 ? sizeof(C2<double>) : prec_is_ff(prec) ? sizeof(C2<ff>) : sizeof(C2<float>);
  p->CW = prec == MLC_F64 ? 8 : 16;  // as strip_width<T>() in fft_impl.cuh
  split_columns(Ny, p->N1, p->N2);
  p->rlM = factor_radices(p->M, 2);
  p->rlN1 = factor_radices(p->N1, p->N2);
  p->rlN2 = factor_radices(p->N2, p->N1);
  MLC_REQUIRE(p->rlM.n >= 0 && p->rlN1.n >= 0 && p->rlN2.n >= 0, MLC_ERR_ARG,
              "map sides must factor into 2, 3 and 5");
  size_t row_smem = 2 * (size_t)(p->M + 1) * p->elem;
  MLC_REQUIRE(row_smem <= 220 * 1024, MLC_ERR_LIMIT,
              "map row too long for one shared-memory row transform (Nx <= 13000 FP64, 26000 FP32)");
  MLC_REQUIRE(2 * (size_t)p->N2 * p->CW * p->elem <= 200 * 1024, MLC_ERR_LIMIT, "column length too large");
  if (prec == MLC_F64) {
    p->twx = upload_twiddles<double>(Nx);
    p->twy = upload_twiddles<double>(Ny);
    p->twx3 = upload_twiddles3(Nx);
    p->twy3 = upload_twiddles3(Ny);
    if (limb_first_radix(p->M)) p->twl3 = upload_level0_limbs3(p->M);
  } else if (prec_is_ff(prec)) {
    p->twx = upload_twiddles<ff>(Nx);
    p->twy = upload_twiddles<ff>(Ny);
  } else {
    p->twx = upload_twiddles<float>(Nx);
    p->twy = upload_twiddles<float>(Ny);
    if (row3_first_radix(p->M)) p->twl = upload_level0_f32(p->M);
  }
  p->anyM = any_levels(p->M, true);
  p->any1 = any_levels(p->N1, false);
  p->any2 = any_levels(p->N2, false);
  p->anyM_tw = upload_any(p->anyM, prec);
  p->any1_tw = upload_any(p->any1, prec);
  p->any2_tw = upload_any(p->any2, prec);
  // (the tables' copies went through the legacy default stream: they are there for any stream)
  MLC_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
  FftPlan2D* raw = p.get();
  ctx->plans[key] = std::move(p);
  return raw;
}

// ---------------------------------------------------------------- dispatch by precision

void fft2_forward(mlc_ctx* ctx, const FftPlan2D& p, const void* in, int in_dtype, void* spec) {
  if (prec_is_ff(p.prec)) forward_impl<ff>(ctx, p, in, in_dtype, spec);
  else if (p.prec == MLC_F64) forward_impl<double>(ctx, p, in, in_dtype, spec);
  else forward_impl<float>(ctx, p, in, in_dtype, spec);
}

void conv_fused(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, const double* prof, int pN, void* out) {
  if (p.prec == PREC_FFS) {  // P0-P2 to the half-spectrum, then P3 into FP32 pixels
    void* tmp = ws_get(ctx, WS_SPEC_TMP, p.spec_bytes());
    conv_fused_impl<ff>(ctx, p, Fmap, prof, pN, nullptr, tmp, WS_KX);
    rows_c2r_impl<ff, float>(ctx, p, tmp, out);
  } else if (p.prec == PREC_FF) conv_fused_impl<ff>(ctx, p, Fmap, prof, pN, out);
  else if (p.prec == MLC_F64) conv_fused_impl<double>(ctx, p, Fmap, prof, pN, out);
  else conv_fused_impl<float>(ctx, p, Fmap, prof, pN, out);
}

void conv_fused_spectrum(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, const double* prof, int pN,
                         void* spec_out, int kx_slot) {
  if (prec_is_ff(p.prec)) conv_fused_impl<ff>(ctx, p, Fmap, prof, pN, nullptr, spec_out, kx_slot);
  else if (p.prec == MLC_F64) conv_fused_impl<double>(ctx, p, Fmap, prof, pN, nullptr, spec_out, kx_slot);
  else conv_fused_impl<float>(ctx, p, Fmap, prof, pN, nullptr, spec_out, kx_slot);
}

bool profile_spectrum_supported(const FftPlan2D& p) {
  if (prec_is_ff(p.prec)) return profile_spectrum_supported_impl<ff>(p);
  if (p.prec == MLC_F64) return profile_spectrum_supported_impl<double>(p);
  return profile_spectrum_supported_impl<float>(p);
}

size_t profile_spectrum_bytes(const FftPlan2D& p) {
  return p.prec == MLC_F64 ? limb3_profile_spectrum_bytes(p) : p.spec_bytes();
}

void profile_spectrum(mlc_ctx* ctx, const FftPlan2D& p, const double* prof, int pN, void* ks) {
  if (prec_is_ff(p.prec)) profile_spectrum_impl<ff>(ctx, p, prof, pN, ks);
  else if (p.prec == MLC_F64) profile_spectrum_impl<double>(ctx, p, prof, pN, ks);
  else profile_spectrum_impl<float>(ctx, p, prof, pN, ks);
}

void conv_cached_spectrum(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, const void* ks, void* spec_out) {
  if (prec_is_ff(p.prec)) conv_cached_impl<ff>(ctx, p, Fmap, ks, spec_out);
  else if (p.prec == MLC_F64) conv_cached_impl<double>(ctx, p, Fmap, ks, spec_out);
  else conv_cached_impl<float>(ctx, p, Fmap, ks, spec_out);
}

void conv_cached(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, const void* ks, void* out) {
  if (p.prec == PREC_FFS) {
    void* tmp = ws_get(ctx, WS_SPEC_TMP, p.spec_bytes());
    conv_cached_impl<ff>(ctx, p, Fmap, ks, tmp);
    rows_c2r_impl<ff, float>(ctx, p, tmp, out);
  } else if (p.prec == PREC_FF) conv_cached_real_impl<ff>(ctx, p, Fmap, ks, out);
  else if (p.prec == MLC_F64) conv_cached_real_impl<double>(ctx, p, Fmap, ks, out);
  else conv_cached_real_impl<float>(ctx, p, Fmap, ks, out);
}

bool rows_c2r_interleave_supported(const FftPlan2D& p) {
  return (p.M == 5000 || p.M == 4096 || p.M == 2000 || p.M == 1000) && p.Ny <= 65535;  // rows on grid.y
}

bool rows_c2r_interleave(mlc_ctx* ctx, const FftPlan2D& p, const void* specs, long spec_stride, int nm, int S,
                         void* out, unsigned planar) {
  if (!rows_c2r_interleave_supported(p)) return false;
  if (p.prec == PREC_FFS) return c2r_interleave_impl<ff, float>(ctx, p, specs, spec_stride, nm, S, out, planar);
  if (p.prec == PREC_FF) return c2r_interleave_impl<ff>(ctx, p, specs, spec_stride, nm, S, out, planar);
  if (p.prec == MLC_F64) return limb3_rows_c2r_il(ctx, p, specs, spec_stride, nm, S, out, planar);
  return c2r_interleave_impl<float>(ctx, p, specs, spec_stride, nm, S, out, planar);
}

void conv_plain(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, const double* prof, int pN, void* out) {
  MLC_REQUIRE(!prec_is_ff(p.prec), MLC_ERR_ARG, "the plain form runs the map's own precision (map in float-float mode)");
  if (p.prec == MLC_F64) conv_plain_impl<double>(ctx, p, Fmap, prof, pN, out);
  else conv_plain_impl<float>(ctx, p, Fmap, prof, pN, out);
}

}  // namespace mlc
