// fvx_parts.cuh -- the FP32 value of an FP64 difference without the FP64 pipe, for the
// mixed-precision wake induction (fvx_flutter.cu); compiled for the host by its
// test too (without contraction).
#pragma once

#include <math.h>

#if defined(__CUDACC__)
#define FVX_PARTS __device__ __forceinline__
#else
#define FVX_PARTS static inline
#endif

namespace fvx {

// An FP64 number as three floats, exactly (24 + 24 + 5 bits).
struct Parts {
  float h, l, r;
};

FVX_PARTS Parts split_f32(double x) {
  Parts p;
  p.h = static_cast<float>(x);
  const double y = x - static_cast<double>(p.h);
  p.l = static_cast<float>(y);
  p.r = static_cast<float>(y - static_cast<double>(p.l));
  return p;
}

// float(x - y) of FP64 x and y in parts: the float of the rounded FP64
// difference, bit for bit, without the FP64 pipe (one subtraction and one
// conversion cost it about 130 FP32 issue slots).  x - y is h + l exactly, h the
// leading parts' rounded difference and l the error of that (Knuth's two_sum)
// plus the differences of the others; l rounds four times, by 2^-24 of at most
// |e| + |a| + |b| each, and FP64's own rounding is 2^-53 |h|.  Where adding and
// taking off that bound rounds to the same float, that float is the answer;
// else (about 2^-20 of the pairs) `same` is cleared and the caller takes the
// FP64 way.  Equal coordinates (particles on a point's span station) give zero
// bounds and a zero.
FVX_PARTS float diff_f32(const Parts& x, const Parts& y, bool& same) {
  const float h = x.h - y.h;
  const float bb = h - x.h;
  const float e = (x.h - (h - bb)) - (y.h + bb);
  const float a = x.l - y.l, b = x.r - y.r;
  const float l = e + (a + b);
  const float w = fmaf(fabsf(h), 2.220446049250313e-16f,                            // 2^-52
                       (fabsf(e) + (fabsf(a) + fabsf(b))) * 2.384185791015625e-07f);  // 2^-22
  const float r0 = h + (l - w);
  const float r1 = h + (l + w);
  same = same && r0 == r1;
  return r0;
}

}  // namespace fvx
