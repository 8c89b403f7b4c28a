// Internals shared by the two back-projectors (backproject.cu, bp_mma.cu).
#pragma once

#include <cstdint>

namespace atb {

// The gather back-projector behind atb_backproject (same arguments).  gate:
// null, or a device array of nslice words, the float bits of each slice's
// largest magnitude: the launch does its work only if one of them is not
// finite.  work: null, or scratch of bp_gather_workspace bytes, with which
// launches whose tiles do not fill the GPU split the angles over more CTAs.
int bp_gather(const void *sino, int sino_dtype, int64_t sino_row_stride, int64_t sino_slice_stride, int nrow,
              int nslice, int ncol, const double *trig, double center, int edge_pad, double mask_r2, float scale,
              float *out, int64_t out_row_stride, int64_t out_slice_stride, int flags, const unsigned *gate,
              void *work, void *stream);
long long bp_gather_workspace(int nrow, int nslice, int ncol);  // 0: none is used

// Status word of the tensor-core back-projector, as atb_backproject_status.
int bp_mma_status(int reset);

#ifdef __CUDACC__
// Power of two that scales a slice whose largest magnitude has these float
// bits to below 2^15 (and above 2^14 where the scale stays in range).
__host__ __device__ inline int bp_sample_exponent(unsigned maxbits) {
  const int e = 14 - ((int)(maxbits >> 23) - 127);
  return e < -126 ? -126 : (e > 126 ? 126 : e);
}
#endif

}  // namespace atb
