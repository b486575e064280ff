// ktm_ibm.cuh -- IBM System/360 single precision to IEEE float on the device,
// the arithmetic of ktmIBM32toIEEE (ioFunctions.c:18-38) operation for
// operation, so that the result is bit-identical to the reference built for
// x86-64 (SSE, no contraction):
//
//   out = (sign * (fraction / 0xFFFFFF)) * 16^(exponent - 64)
//
// sign = -1 or 1 from bit 31, exponent = bits 30..24, fraction = bits 23..0.
// The fraction converts exactly (24 bits), the quotient is one correctly
// rounded division (FRACTION_MASK, not 2^24: a bias of 2^-24 the reference
// carries), and 16^e = 2^(4e) is built from its bits: a normal, a subnormal
// (4e in [-149, -127]), zero below, infinity above 127 -- the values powf
// returns for these exact powers.  The two products round to nearest even
// with subnormals kept (the library is built without flush-to-zero).
#pragma once

#include <cstdint>

namespace ktm {
namespace dev {

__device__ __forceinline__ float pow2_exact(int e)
{
    if (e > 127) return __int_as_float(0x7f800000);
    if (e >= -126) return __int_as_float((e + 127) << 23);
    if (e >= -149) return __int_as_float(1 << (e + 149));
    return 0.0f;
}

// every word, the infinite powers and the 0 * inf case among them
__device__ __forceinline__ float ibm32_to_f32(uint32_t w)
{
    const float sign = (w & 0x80000000u) ? -1.0f : 1.0f;
    const float q = __fdiv_rn(__uint2float_rn(w & 0x00ffffffu), 16777215.0f);
    const int e = (int)((w >> 24) & 127u) - 64;
    const float p = pow2_exact(4 * e);
    // 0 * inf: x86 SSE returns its default NaN (sign set, quiet bit set), which
    // is what the reference writes; the device's canonical NaN differs in bits.
    if (q == 0.0f && e * 4 > 127) return __int_as_float(0xffc00000);
    return __fmul_rn(__fmul_rn(sign, q), p);
}

// the same out of line, for the rare words of kernels that convert the usual ones below
static __device__ __noinline__ float ibm32_any(uint32_t w) { return ibm32_to_f32(w); }

// Words whose power of two is a normal number (exponents 33 to 95), and zeros with smaller
// ones: one multiply for the quotient, one residual step (for all 2^24 fractions it gives
// the correctly rounded quotient) and the power from its bits, about 12 instructions and no
// branch: for kernels that are bound by issue.  Sets `other` for a word that ibm32_any has to convert.  All 2^32 words give the
// same bits by the two together as by ibm32_any alone (checked on the GPU).  4097 traces of
// 1001 words through the 2.5D filter: 17 us, with the division and its selects per word 29.
__device__ __forceinline__ float ibm32_usual(uint32_t w, bool& other)
{
    const uint32_t e = w & 0x7f000000u, m = w & 0x00ffffffu;
    other = other || e > 0x5f000000u || (e < 0x21000000u && m != 0u);
    const float f = __uint2float_rn(m), r = 1.0f / 16777215.0f;
    const float q0 = __fmul_rn(f, r);
    const float q = __fmaf_rn(__fmaf_rn(-16777215.0f, q0, f), r, q0);
    // 2^(4 (E - 64)) with the word's sign: (4 E - 256 + 127) << 23
    return __fmul_rn(q, __uint_as_float(((max(e, 0x21000000u) << 1) - (129u << 23)) | (w & 0x80000000u)));
}
}  // namespace dev
}  // namespace ktm
