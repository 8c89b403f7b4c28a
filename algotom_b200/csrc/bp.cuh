// Internals shared by the two back-projectors (backproject.cu, bp_mma.cu).
#pragma once

#include <cstdint>

namespace atb {

// The gather back-projector behind atb_backproject (same arguments).  gate:
// null, or what bp_left_to_gather looks at for nslice slices: the launch does its
// work only if it holds.  work: null, or scratch of bp_gather_workspace bytes, with which
// launches whose tiles do not fill the GPU split the angles over more CTAs.
int bp_gather(const void *sino, int sino_dtype, int64_t sino_row_stride, int64_t sino_slice_stride, int nrow,
              int nslice, int ncol, const double *trig, double center, int edge_pad, double mask_r2, float scale,
              float *out, int64_t out_row_stride, int64_t out_slice_stride, int flags, const unsigned *gate,
              void *work, void *stream);
long long bp_gather_workspace(int nrow, int nslice, int ncol);  // 0: none is used

// atb_backproject_centers (same arguments); with interior >= 0 only the blocks
// of pixels that bp_interior does not hold for, unless the gate (for ngate
// slices, as above) leaves them all to this kernel.
int bp_gather_centers(const float *sino, int64_t sino_row_stride, int nrow, int ncol, const double *trig,
                      double center, int spacing, int ncenter, int edge_pad, double mask_r2, float scale, float *out,
                      int64_t out_row_stride, int64_t out_center_stride, int flags, const unsigned *gate, int ngate,
                      double interior, void *stream);

// Status word of the tensor-core back-projector, as atb_backproject_status.
int bp_mma_status(int reset);

#ifdef __CUDACC__
// Words of a gate: the float bits of each slice's largest magnitude, and from word
// kGatePairs on the slice's number of faint pairs: neighbouring samples, not both
// zero, of which the tensor cores' two float16 terms hold neither to 22 bits
// (below kFaint once scaled by bp_sample_exponent, about 2^-16 of the largest).
constexpr int kGatePairs = 64, kGateWords = 96;
constexpr float kFaint = 0.25f;

// Whether a stack is left to the gather kernel: a sample is not finite (0 times
// it must stay out of the pixels that do not read it), or a slice has more faint
// pairs than a sixteenth of its angles, so that some pixel may read little else:
// its sum would carry the rounding of samples 2^16 times as large (a pair has to
// be faint in nearly every angle for that; a filtered sinogram's zero crossings
// leave fewer than one per 1000 angles).  Every thread of the CTA calls it.
__device__ __forceinline__ bool bp_left_to_gather(const unsigned *gate, int ngate, int nrow) {
  const int t = threadIdx.x;
  return __syncthreads_or(t < ngate && (gate[t] >= 0x7f800000u || gate[kGatePairs + t] > (unsigned)nrow / 16u));
}

// Power of two that scales a slice whose largest magnitude has these float
// bits to below 2^15 (and above 2^14 where the scale stays in range).
__host__ __device__ inline int bp_sample_exponent(unsigned maxbits) {
  const int e = 14 - ((int)(maxbits >> 23) - 127);
  return e < -126 ? -126 : (e > 126 ? 126 : e);
}

// Whether every pixel of the 64 x 32 block (the gather kernel's tile of four
// slices) around pixel (x, y) lies within
// `radius` of the image centre, so that no position of it leaves a detector
// that reaches `radius` to both sides of the rotation axis.
__device__ __forceinline__ bool bp_interior(int x, int y, int ncol, double radius) {
  const double ic = 0.5 * (double)(ncol - 1);
  const int bx = x & ~63, by = y & ~31;
  const double dx = fmax(fabs((double)bx - ic), fabs((double)min(bx + 63, ncol - 1) - ic));
  const double dy = fmax(fabs((double)by - ic), fabs((double)min(by + 31, ncol - 1) - ic));
  return radius > 0.0 && dx * dx + dy * dy <= radius * radius;
}
#endif

}  // namespace atb
