// pa_parity.cuh -- rounding of pass C's outputs to the nearest integer's parity (plain C++ outside nvcc).
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define PA_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PA_HOST_DEVICE inline
#endif

namespace pa {

// d - 1/2 with d the distance of v to the nearest even integer: positive where rint(v) is odd, and 1/2 minus its
// magnitude is v's distance to the nearest integer.  FP32 adds only (rint and the conversion to an integer run at an
// eighth of their rate): |v| is rounded to an even integer by adding 2^24, exact for |v| < 2^24 on either side of zero
// (without the magnitude, by v / 2 + 3 2^22, odd values below -2^23 came out even at a distance of zero).  From 2^24 on v is
// even; one that is not a multiple of the sum's spacing shows a distance of 1 or more.
PA_HOST_DEVICE float parity_half(float v) {
    const float magic = 16777216.0f, a = fabsf(v);
    const float even = (a + magic) - magic;
    return fabsf(a - even) - 0.5f;
}

}  // namespace pa
