// mpc_scale.h -- the exit pass's conversion to complex128 without the FP64 pipe.
//
// GB300 issues FP64 at 1/64 of its FP32 rate.  The product (double)a * scale of an FP32 value and a
// positive FP64 factor is formed on the integer pipe: the 24-bit by 53-bit product of the significands
// exactly (two 32 x 32 multiplications), rounded once to nearest even, so that it has the bits of the FP64
// multiplication.  Bound of the exit sweep with it: issue.  512x512x1024 2.12 ms (FP64 multiplication 3.15, a
// two-FP32 product good to 2^-47 1.86), 256x256x2048 1.35 ms (1.50, 1.25), 256x256x512 0.271 ms (0.406,
// 0.239).  The entry pass's conversion done the same way was slower: it waits on its loads.
// Host code as well, for its test.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define MPC_HD __host__ __device__ __forceinline__
#else
#define MPC_HD inline
#endif

namespace mpc {

// A factor as its significand (53 bits at the top of hi:lo), its exponent's part of the result's high word,
// and the number of FP32 exponents (from 1) that take the integer path: 254, or 0 where the factor is not
// positive or so small or large that a product with a normal float may leave the range of normal doubles.
struct IntScale {
    uint32_t lo, hi, eword, nexp;
};
MPC_HD IntScale int_scale(double scale) {
    uint64_t b;
    memcpy(&b, &scale, sizeof b);
    const uint32_t e = (uint32_t)(b >> 52);   // with the sign bit
    if (e < 129u || e > 1917u) return IntScale{0u, 0u, 0u, 0u};
    const uint64_t m = (b << 11) | 0x8000000000000000ull;
    return IntScale{(uint32_t)m, (uint32_t)(m >> 32), (e - 128u) << 20, 254u};
}

// (double)a * scale, s = int_scale(scale)
MPC_HD double scaled_double(float a, double scale, const IntScale& s) {
    uint32_t ab;
    memcpy(&ab, &a, sizeof ab);
    if (((ab >> 23) & 0xffu) - 1u >= s.nexp) {   // zero, denormal, infinity, NaN, or an unusual factor
        if ((ab << 1) != 0u || s.nexp == 0u) return (double)a * scale;
        const uint64_t z = (uint64_t)ab << 32;
        double d;
        memcpy(&d, &z, sizeof d);
        return d;
    }
    // the significands' product, 2^94 <= w2:w1:w0 < 2^96
    const uint32_t ma = (ab << 8) | 0x80000000u;
    const uint64_t t0 = (uint64_t)ma * s.lo;
    const uint64_t t1 = (uint64_t)ma * s.hi + (t0 >> 32);
    const uint32_t w0 = (uint32_t)t0, w1 = (uint32_t)t1, w2 = (uint32_t)(t1 >> 32);
    // its leading 53 bits, the next ones at the top of `rest`
    const uint32_t two = w2 >> 31, sh = 10u + two;
    const uint64_t m = t1 >> sh;
    const uint32_t rest = w1 << (32u - sh);
    // to nearest, a tie to even: a carry out of rest + (half - 1) + 1 where bits follow or the last bit is odd
    const uint32_t odd = ((uint32_t)m & 1u) | (w0 != 0u ? 1u : 0u);
    const uint32_t up = rest > 0x80000000u - odd ? 1u : 0u;
    // m's leading one adds 1 to the exponent
    const uint32_t e = ((ab >> 3) & 0x0ff00000u) + s.eword + (two << 20);
    const uint64_t r = (m + up + ((uint64_t)e << 32)) | (uint64_t)(ab & 0x80000000u) << 32;
    double d;
    memcpy(&d, &r, sizeof d);
    return d;
}

}  // namespace mpc
