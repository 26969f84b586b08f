// Column passes and P1 of FP64 transforms in three limbs (fft_limb.cuh).
#include "fft_limb.cuh"

namespace mlc {

bool limb3_colpass(mlc_ctx* ctx, const FftPlan2D& p, void* buf, char kind, bool inverse, int post_tw) {
  return inverse ? limb_colpass_impl<lf3, true>(ctx, p, buf, kind, post_tw)
                 : limb_colpass_impl<lf3, false>(ctx, p, buf, kind, post_tw);
}
bool limb3_conv(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, void* out, void* kx, int h) {
  return limb3_conv_impl<0>(ctx, p, Fmap, out, kx, h, nullptr, "conv_fused_spectrum");
}
bool limb3_conv_profile(mlc_ctx* ctx, const FftPlan2D& p, void* kx, int h, void* ks) {
  return limb3_conv_impl<1>(ctx, p, nullptr, nullptr, kx, h, ks, "conv_profile_spectrum");
}
bool limb3_conv_cached(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, void* out, const void* ks) {
  return limb3_conv_impl<2>(ctx, p, Fmap, out, nullptr, 0, (void*)ks, "conv_cached_spectrum");
}

size_t limb3_profile_spectrum_bytes(const FftPlan2D& p) {
  return LimbSpectrum::bytes((size_t)p.Ny * p.Wp, (size_t)p.N1 * p.Wp);
}

}  // namespace mlc
