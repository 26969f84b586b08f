// Float-float passes of lengths without an unrolled kernel (fft_any_real.cuh).
#include "fft_any_real.cuh"

namespace mlc {

template bool any_real_r2c<ff, RealRows<ff, double>>(mlc_ctx*, const FftPlan2D&, const RealRows<ff, double>&, int,
                                                       void*, const char*);
template bool any_real_r2c<ff, RealRows<ff, float>>(mlc_ctx*, const FftPlan2D&, const RealRows<ff, float>&, int,
                                                      void*, const char*);
template bool any_real_r2c<ff, ProfileRows<ff>>(mlc_ctx*, const FftPlan2D&, const ProfileRows<ff>&, int, void*,
                                                  const char*);
template bool any_real_c2r<ff, double>(mlc_ctx*, const FftPlan2D&, const void*, void*);
template bool any_real_c2r<ff, float>(mlc_ctx*, const FftPlan2D&, const void*, void*);
template bool any_real_colpass<ff, false>(mlc_ctx*, const FftPlan2D&, void*, char, int);
template bool any_real_colpass<ff, true>(mlc_ctx*, const FftPlan2D&, void*, char, int);

}  // namespace mlc
