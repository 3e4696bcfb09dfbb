// IEEE FP64 division a / b, rounded to nearest even, by 32-bit integer arithmetic.
//
// GB300 issues one FP64 warp instruction per ~19 cycles and SM (1.68 lane operations per
// clock) but an integer one per cycle or less, and its FP64 division is a sequence of
// dependent FP64 instructions: measured 562 cycles for a lone warp and 138 cycles of the SM
// per warp at 16 warps, against 206 and 31 for this routine.  It forms the 54-bit quotient
// from a 31-bit reciprocal in two digits of 29 and 24 bits with exact remainders, so its
// result is the correctly rounded one: the same bits as the `/` operator for every operand.
// Operands it does not cover (subnormal, infinite or NaN, zero divisor, a result outside
// the normal range) go to the hardware sequence.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FPDIV_HD __host__ __device__
#else
#define FPDIV_HD
#endif

namespace fpdiv {

FPDIV_HD inline uint64_t bits(double x)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}

FPDIV_HD inline double from_bits(uint32_t hi, uint32_t lo)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = (uint64_t)hi << 32 | lo;
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}

FPDIV_HD inline uint32_t mulhi(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)((uint64_t)a * b >> 32);
#endif
}

// high word of (hi:lo) << s, 0 < s < 32
FPDIV_HD inline uint32_t funnel(uint32_t hi, uint32_t lo, int s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return hi << s | lo >> (32 - s);
#endif
}

// 2^31 / f within 2^11 below, for f in [1, 2) given by its float bits: the approximate
// reciprocal (1 float ulp), lowered by 2^-20 and rounded to 22 bits so that it never
// exceeds the exact one
FPDIV_HD inline uint32_t seed(uint32_t fbits)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(fbits)));
    return __float_as_uint(__fmaf_rn(y, 0x1p22f - 4.0f, 0x1p23f)) << 9;
#else
    float f, y;
    memcpy(&f, &fbits, 4);
    y = 1.0f / f;
#ifdef FPDIV_SEED_ULPS   // tests: any reciprocal the device instruction may return
    uint32_t v;
    memcpy(&v, &y, 4);
    v += FPDIV_SEED_ULPS;
    memcpy(&y, &v, 4);
#endif
    y = (float)((double)y * (0x1p22 - 4.0) + 0x1p23);
    uint32_t u;
    memcpy(&u, &y, 4);
    return u << 9;
#endif
}

// Y with 2^83 / mb - 4 < Y <= 2^83 / mb for the 53-bit significand mb = (hi:lo)
FPDIV_HD inline uint32_t recip31(uint32_t hi, uint32_t lo)
{
    const uint32_t bt = funnel(hi, lo, 11);                              // mb >> 21
    const uint32_t y0 = seed((funnel(hi, lo, 3) & 0x007fffffu) | 0x3f800000u);
    const uint64_t e = (1ull << 62) - (uint64_t)bt * y0;                 // 2^62 (1 - b y0), < 2^43
    const uint32_t e50 = funnel((uint32_t)(e >> 32), (uint32_t)e, 20);   // e >> 12
    return y0 + (mulhi(y0, e50) >> 18) - 1u;
}

#ifdef __CUDACC__
// the hardware sequence, kept out of line: inlined, the compiler runs it for every operand
static __device__ __noinline__ double div_hw(double a, double b) { return a / b; }
#endif

// a / b for operands and result in the normal range, or a = +-0; *ok is false otherwise
FPDIV_HD inline double quotient(double a, double b, bool* ok)
{
    const uint64_t ua = bits(a), ub = bits(b);
    const uint32_t ah = (uint32_t)(ua >> 32), al = (uint32_t)ua, bh = (uint32_t)(ub >> 32), bl = (uint32_t)ub;
    const uint32_t ea = ah >> 20 & 0x7ffu, eb = bh >> 20 & 0x7ffu;
    const uint32_t mbh = (bh & 0xfffffu) | 0x100000u;
    const uint64_t mb = (uint64_t)mbh << 32 | bl;
    uint64_t ma = (uint64_t)((ah & 0xfffffu) | 0x100000u) << 32 | al;
    const bool lt = ma < mb;
    if (lt) ma += ma;                                                    // ma / mb in [1, 2)
    const uint32_t y = recip31(mbh, bl);
    // first digit: q1 = floor((ma / mb) 2^29) - (0 .. 4), r1 = ma 2^29 - q1 mb < 5 mb < 2^56
    const uint32_t at = funnel((uint32_t)(ma >> 32), (uint32_t)ma, 10);  // ma >> 22
    const uint32_t q1 = mulhi(at, y);
    const uint64_t r1 = (ma << 29) - (uint64_t)q1 * mb;
    // second digit: q2 = floor((r1 / mb) 2^24) - (0 or 1)
    const uint32_t q2 = mulhi((uint32_t)(r1 >> 24), y) >> 3;
    const uint64_t r2 = (r1 << 24) - (uint64_t)q2 * mb;
    // 54-bit quotient floor((ma / mb) 2^53); a quotient of two 53-bit significands is never
    // half way between two of 53 bits, so adding one to the 54th bit rounds to nearest
    uint64_t q = ((uint64_t)q1 << 24) + q2 + (r2 >= mb ? 2u : 1u);
    q >>= 1;
    const uint32_t e = ea - eb + 1022u - (lt ? 1u : 0u);                 // biased exponent - 1
    const uint32_t sign = (ah ^ bh) & 0x80000000u;
    const bool zero = (ah << 1 | al) == 0u;                              // +-0 / b: exact, and frequent
    *ok = (eb - 1u < 2046u) && (zero || ((ea - 1u < 2046u) && e < 2045u));
    return zero ? from_bits(sign, 0u) : from_bits(((uint32_t)(q >> 32) + (e << 20)) | sign, (uint32_t)q);
}

// a / b
FPDIV_HD inline double div(double a, double b)
{
#ifdef __CUDA_ARCH__
    bool ok;
    const double q = quotient(a, b, &ok);
    return ok ? q : div_hw(a, b);
#else
    return a / b;
#endif
}

}  // namespace fpdiv
