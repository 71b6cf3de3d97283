// IEEE double division on the integer and FP32 pipes, for devices with a slow FP64 pipe.  Plain C++, so
// that a host compiler can check it against its own division.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define F64_DIV_FN __host__ __device__ __forceinline__
#else
#include <math.h>
#define F64_DIV_FN static inline
#endif

namespace uc {

// a / b rounded to nearest even (IEEE double) by long division on the mantissas, radix 2^18: this part's
// FP64 pipe takes some 150 cycles for a warp's division, the integer and FP32 pipes about 20 for these
// instructions.  With ma, mb the mantissas scaled so that 1 <= ma / mb < 2, floor(2^53 ma / mb) has the
// 53 bits of the result and a rounding bit (a quotient of two doubles never lies halfway between two
// doubles, so that bit decides), in three digits d = rint(R 2^18 / mb) with the remainder R 2^18 - d mb
// between them: |d - R 2^18 / mb| < 0.75 (the reciprocal and the remainder are good to 2^-22 of the digit,
// 2^18), so a remainder stays below 0.75 mb in magnitude and only the last one needs a correction by mb.
// Returns false for zeros, infinities, NaNs, denormals and results outside the normal range.
F64_DIV_FN bool f64_div_bits(uint64_t a, uint64_t b, uint64_t *out)
{
    const uint32_t ea = (uint32_t)(a >> 52) & 0x7ff, eb = (uint32_t)(b >> 52) & 0x7ff;
    const int e = (int)ea - (int)eb + 1023;
    if (ea - 1 >= 0x7fe || eb - 1 >= 0x7fe || e < 2 || e > 2045) return false;
    uint64_t ma = (a & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    const uint64_t mb = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    const bool small = ma < mb;
    if (small) ma <<= 1;
    const float inv = 2097152.0f / (float)(uint32_t)(mb >> 21);    // 2^42 / mb
    int64_t rem = (int64_t)(ma - mb);                                                     // [0, mb)
    int64_t q = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int k = 0; k < 3; k++) {
        const int bits = k < 2 ? 18 : 17;
        const float f = (float)(int32_t)(rem >> 24) * (k < 2 ? inv : inv * 0.5f);
#ifdef __CUDA_ARCH__
        const int32_t d = __float2int_rn(f);
#else
        const int32_t d = (int32_t)rintf(f);
#endif
        q = (q << bits) + d;
        rem = (int64_t)(((uint64_t)rem << bits) - (uint64_t)(int64_t)d * mb);
    }
    if (rem < 0) q--;                                  // now the floor
    else if (rem >= (int64_t)mb) q++;
    q += 1ll << 53;
    // the exponent field is added to the mantissa with its leading one: a carry moves it up
    *out = ((a ^ b) & 0x8000000000000000ull) | (((uint64_t)(e - 1 - (small ? 1 : 0)) << 52) + (uint64_t)((q + 1) >> 1));
    return true;
}

}  // namespace uc
