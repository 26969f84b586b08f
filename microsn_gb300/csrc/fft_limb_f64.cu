// Row passes of FP64 transforms in three limbs (fft_limb.cuh).
#include "fft_limb.cuh"

namespace mlc {

bool limb3_rows_r2c_map(mlc_ctx* ctx, const FftPlan2D& p, const void* in, int in_dtype, void* out) {
  if (in_dtype == MLC_F64)
    return limb_rows_r2c_impl<lf3>(ctx, p, RealRows<double, double>{(const double*)in, p.Nx}, p.Ny, out, "fft_rows_r2c");
  return limb_rows_r2c_impl<lf3>(ctx, p, RealRows<double, float>{(const float*)in, p.Nx}, p.Ny, out, "fft_rows_r2c");
}
bool limb3_rows_r2c_profile(mlc_ctx* ctx, const FftPlan2D& p, const double* prof, int pN, void* out) {
  if (pN < 2) return true;  // no rows
  return limb_rows_r2c_impl<lf3>(ctx, p, ProfileRows<double>{prof, pN, pN / 2, p.Nx}, 2 * (pN / 2), out,
                                 "fft_profile_rows");
}
bool limb3_rows_c2r(mlc_ctx* ctx, const FftPlan2D& p, const void* in, void* out) {
  return limb_rows_c2r_impl<lf3>(ctx, p, in, out);
}
bool limb3_rows_c2r_il(mlc_ctx* ctx, const FftPlan2D& p, const void* specs, long spec_stride, int nm, int S,
                       void* out, unsigned planar) {
  return limb_rows_c2r_il_impl<lf3>(ctx, p, specs, spec_stride, nm, S, out, planar);
}

}  // namespace mlc
