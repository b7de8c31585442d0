// Integer pieces of the exact bf16 slicing (tcgemm.cu), host and device.
//
// A row with exponent e (|x| < 2^e for every element) is scaled to the integer
// Y = round(x 2^(F - e)), |Y| <= 2^F, and cut into N balanced digits of radix 128,
// Y = sum_t d_t 2^(7 (N - 1 - t)), every digit an integer that bf16 holds exactly:
//   N = 6, F = 42: |d_0| <= 128, -64 <= d_t <= 63 below it (the mixed-precision path)
//   N = 9, F = 62: |d_0| <= 64, the same below (the plain FP64 path; 2^-62 of the row's scale)
// Digits are balanced rather than sign and magnitude for two reasons.  The sum over
// K of all digit products of one group i + j = t stays below 2^24, so FP32
// accumulation is exact for every input: N = 6: (2 128 64 + 4 64 64) K <= 2^24 for
// K <= 512; N = 9: 9 64 64 K < 2^24 for K <= 455.  And the products that are left
// out (i + j >= N) are half as large and of random sign: the error is about half
// that of 7-bit magnitudes at the same number of products.
//
// Adding the bias 64 (1 + 128 + ... ) (128 at the top of N = 6) to the two's
// complement Y turns the digits into plain bit fields u_t = d_t + bias.  The bf16
// pattern 0x4300 | u is the value 128 + u (u <= 128: a carry makes it 256), so one
// packed subtraction of 192 leaves two digits exactly.  GB300 runs 64-bit
// conversions and compares on its narrow FP64 pipe; everything here is 32-bit
// integer and bf16x2 arithmetic.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define HF_HD __host__ __device__ __forceinline__
#else
#define HF_HD inline
#endif

namespace hfgpu {

template <int NSL>
struct SliceFmt {
    static_assert(NSL == 6 || NSL == 9, "digit counts with a stated range");
    static constexpr int F = NSL == 6 ? 42 : 62;
    static constexpr int HALF = NSL == 6 ? 1 : 0;  // the biased value is kept doubled (one bit below the digits)
    static constexpr int KMAX = NSL == 6 ? 512 : 455;
    static constexpr uint64_t lower()  // 64 (1 + 128 + ... + 128^(NSL - 2))
    {
        uint64_t b = 0;
        for (int k = 0; k < NSL - 1; ++k) b |= 64ull << (7 * k);
        return b;
    }
    static constexpr uint64_t BIAS = (lower() + ((NSL == 6 ? 128ull : 64ull) << (7 * (NSL - 1)))) << HALF;
    // out = 2^(ea + eb - SHIFT) sum_t acc_t 2^(7 (NSL - 1 - t)): two scales F, less the
    // weights 7 (2 NSL - 2) - 7 (NSL - 1) taken by the recombination
    static constexpr int SHIFT = 2 * F - 7 * (NSL - 1);
};

// the biased digits of x (its bits), scaled by the row exponent e: U = Y + bias
// (doubled where HALF = 1).  Zero and subnormal x give Y = 0.
template <int NSL>
HF_HD uint64_t biased_digits(uint64_t bits, int e)
{
    using S = SliceFmt<NSL>;
    const int ex = (int)(bits >> 52) & 0x7FF;
    const uint64_t m = (bits << 11) | (1ull << 63);  // |x| = m 2^(ex - 1022 - 64)
    const int r = 63 - S::F + e + 1022 - ex;         // m >> r is |x| 2^(F + 1 - e)
    uint64_t t = 0;
    if (ex != 0 && r <= 63) t = (m >> r) + 1;        // + 1: round half up at the bit below the digits
    t = S::HALF ? t & ~1ull : t >> 1;
    const uint64_t sgn = (uint64_t)((int64_t)bits >> 63);
    return ((t ^ sgn) - sgn) + S::BIAS;
}

// the digit field of weight 128^(NSL - 1 - t) of U (biased)
template <int NSL>
HF_HD uint32_t digit_field(uint64_t U, int t)
{
    const uint32_t v = (uint32_t)(U >> (7 * (NSL - 1 - t) + SliceFmt<NSL>::HALF));
    return t == 0 ? v : v & 127u;
}

}  // namespace hfgpu
