// A float32 value as the sum of three bfloat16 ("planes", 24 significant bits in pieces of 8), for products on the tensor cores.
#pragma once
#include "common.cuh"

namespace ttie {
// 2 P values into their three planes, pairs of bfloat16 (the first value in the lower half): the nearest bfloat16 (ties away from zero), the
// rest's leading 8 bits, what is left (at most 7 bits, so nothing is lost above 2^-103).  Integer and add instructions, a step for all
// values at a time.  A NaN or an infinity leaves a NaN in the second plane.
template <int P>
__device__ __forceinline__ void split_values(float (&x)[2 * P], uint32_t (&p0)[P], uint32_t (&p1)[P], uint32_t (&p2)[P]) {
    uint32_t t[2 * P];
#pragma unroll
    for (int i = 0; i < 2 * P; ++i) t[i] = __float_as_uint(x[i]) + 0x8000u;
#pragma unroll
    for (int i = 0; i < P; ++i) p0[i] = __byte_perm(t[2 * i], t[2 * i + 1], 0x7632);
#pragma unroll
    for (int i = 0; i < 2 * P; ++i) x[i] -= __uint_as_float(t[i] & 0xffff0000u);
#pragma unroll
    for (int i = 0; i < P; ++i) p1[i] = __byte_perm(__float_as_uint(x[2 * i]), __float_as_uint(x[2 * i + 1]), 0x7632);
#pragma unroll
    for (int i = 0; i < 2 * P; ++i) x[i] -= __uint_as_float(__float_as_uint(x[i]) & 0xffff0000u);
#pragma unroll
    for (int i = 0; i < P; ++i) p2[i] = __byte_perm(__float_as_uint(x[2 * i]), __float_as_uint(x[2 * i + 1]), 0x7632);
}
}  // namespace ttie
