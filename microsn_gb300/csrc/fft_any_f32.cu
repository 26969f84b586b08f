// FP32 passes of lengths without an unrolled kernel (fft_any_real.cuh).
#include "fft_any_real.cuh"

namespace mlc {

template bool any_real_r2c<float, RealRows<float, double>>(mlc_ctx*, const FftPlan2D&, const RealRows<float, double>&, int,
                                                       void*, const char*);
template bool any_real_r2c<float, RealRows<float, float>>(mlc_ctx*, const FftPlan2D&, const RealRows<float, float>&, int,
                                                      void*, const char*);
template bool any_real_r2c<float, ProfileRows<float>>(mlc_ctx*, const FftPlan2D&, const ProfileRows<float>&, int, void*,
                                                  const char*);
template bool any_real_c2r<float, float>(mlc_ctx*, const FftPlan2D&, const void*, void*);
template bool any_real_colpass<float, false>(mlc_ctx*, const FftPlan2D&, void*, char, int);
template bool any_real_colpass<float, true>(mlc_ctx*, const FftPlan2D&, void*, char, int);

}  // namespace mlc
