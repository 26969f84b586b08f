// Inverse passes of FP32 maps with float-float transforms, in two limbs (fft_limb.cuh).
#include "fft_limb.cuh"

namespace mlc {

bool limb2_colpass_inverse(mlc_ctx* ctx, const FftPlan2D& p, void* buf, char kind, int post_tw) {
  return limb_colpass_impl<lf2, true>(ctx, p, buf, kind, post_tw);
}
bool limb2_conv(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, void* out, const void* kx, int h) {
  return limb2_conv_impl<0>(ctx, p, Fmap, out, kx, h, nullptr, "conv_fused_spectrum");
}
bool limb2_conv_cached(mlc_ctx* ctx, const FftPlan2D& p, const void* Fmap, void* out, const void* ks) {
  return limb2_conv_impl<2>(ctx, p, Fmap, out, nullptr, 0, ks, "conv_cached_spectrum");
}
bool limb2_rows_c2r(mlc_ctx* ctx, const FftPlan2D& p, const void* in, void* out) {
  return limb_rows_c2r_impl<lf2>(ctx, p, in, out);
}
bool limb2_rows_c2r_il(mlc_ctx* ctx, const FftPlan2D& p, const void* specs, long spec_stride, int nm, int S,
                       void* out, unsigned planar) {
  return limb_rows_c2r_il_impl<lf2>(ctx, p, specs, spec_stride, nm, S, out, planar);
}

}  // namespace mlc
