// Float-float inverse row pass with FP32 outputs (FP32 maps with
// mlc_map_set_fft(map, MLC_FFT_F32X2)) of the row lengths without a limb kernel
// (fft_limb_ffs.cu).  The forward transform and P0 are the FP64 maps' float-float kernels
// (fft_ff.cu, fft_ff_conv.cu): they read and write float-float spectra whatever the pixels'
// type.
#include "fft_impl.cuh"

namespace mlc {

template void rows_c2r_impl<ff, float>(mlc_ctx*, const FftPlan2D&, const void*, void*);

}  // namespace mlc
