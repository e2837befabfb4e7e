// fast_exp.h -- exp(x) and a / b in FP64 on the integer pipe (shared by device and host code).
//
// GB300 issues one FP64 warp instruction every 19 cycles per SM (76 cycles for each of the four
// sub-partitions when all are busy, 64 when one warp runs alone) and runs 32-bit integer and FP32
// instructions beside it at 1 to 4 cycles: 16 32 x 32 + 64-bit multiply-adds hide behind one FP64 FMA.
// So both functions work on 64-bit fixed-point numbers, with no FP64 instruction in the common case.
//
// exp, after the table method of P. T. P. Tang, "Table-driven implementation of the exponential function in
// IEEE floating-point arithmetic", ACM TOMS 15(2):144-157, 1989, in base 2:
//   x log2(e) = k + j/256 + r,  0 <= r < 2^-8,  exp(x) = 2^k 2^(j/256) 2^r,
// 2^r by its Taylor polynomial of degree 5 (remainder below 2^-60).  The product x log2(e) is kept to 2^-64,
// the polynomial to about 2^-57, the table to 2^-64; the result is rounded once.
// The table (2 KB) is passed in: kernels keep it in shared memory, where lane-divergent indices do not
// serialise as constant-memory reads would.
// Accuracy: within 0.66 ulp of the exact value for 1 <= |x| <= 708, 1 ulp below (95% and 82% correctly
// rounded); +inf above, 0 below.
#pragma once
#ifndef __CUDACC_RTC__
#include <cstdint>
#include <cstring>
#else
typedef long long int64_t;
typedef unsigned long long uint64_t;
typedef int int32_t;
typedef unsigned int uint32_t;
#endif

#ifndef GDTK_HD
#ifdef __CUDACC__
#define GDTK_HD __host__ __device__ __forceinline__
#else
#define GDTK_HD inline
#endif
#endif

#ifndef GDTK_FN
#define GDTK_FN GDTK_HD
#endif

namespace gdtk {

// 2^(j/256) 2^63, j = 0..255, rounded to nearest: the significands with their leading bit.
#define GDTK_EXP2_TABLE_SIZE 256
#define GDTK_EXP2_TABLE_INIT { \
    0x8000000000000000ull, 0x8058d7d2d5e5f6b1ull, 0x80b1ed4fd999ab6cull, 0x810b40a1d81406d4ull, \
    0x8164d1f3bc030773ull, 0x81bea1708dde6056ull, 0x8218af4373fc25ecull, 0x8272fb97b2a5894cull, \
    0x82cd8698ac2ba1d7ull, 0x83285071e0fc4547ull, 0x8383594eefb6ee37ull, 0x83dea15b9541b132ull, \
    0x843a28c3acde4046ull, 0x8495efb3303efd30ull, 0x84f1f656379c1a29ull, 0x854e3cd8f9c8c95dull, \
    0x85aac367cc487b15ull, 0x86078a2f23642a9full, 0x8664915b923fba04ull, 0x86c1d919caef5c88ull, \
    0x871f61969e8d1010ull, 0x877d2afefd4e256cull, 0x87db357ff698d792ull, 0x88398146b919f1d4ull, \
    0x88980e8092da8527ull, 0x88f6dd5af155ac6bull, 0x8955ee03618e5fddull, 0x89b540a7902557a4ull, \
    0x8a14d575496efd9aull, 0x8a74ac9a79896e47ull, 0x8ad4c6452c728924ull, 0x8b3522a38e1e1032ull, \
    0x8b95c1e3ea8bd6e7ull, 0x8bf6a434adde0085ull, 0x8c57c9c4646f4ddeull, 0x8cb932c1bae97a95ull, \
    0x8d1adf5b7e5ba9e6ull, 0x8d7ccfc09c50e2f8ull, 0x8ddf042022e69cd6ull, 0x8e417ca940e35a01ull, \
    0x8ea4398b45cd53c0ull, 0x8f073af5a2013520ull, 0x8f6a8117e6c8e5c4ull, 0x8fce0c21c6726481ull, \
    0x9031dc431466b1dcull, 0x9095f1abc540ca6bull, 0x90fa4c8beee4b12bull, 0x915eed13c89689d3ull, \
    0x91c3d373ab11c336ull, 0x9228ffdc10a051adull, 0x928e727d9531f9acull, 0x92f42b88f673aa7cull, \
    0x935a2b2f13e6e92cull, 0x93c071a0eef94bc1ull, 0x9426ff0fab1c04b6ull, 0x948dd3ac8ddb7ed3ull, \
    0x94f4efa8fef70961ull, 0x955c5336887894d5ull, 0x95c3fe86d6cc7fefull, 0x962bf1cbb8d97560ull, \
    0x96942d3720185a00ull, 0x96fcb0fb20ac4ba3ull, 0x97657d49f17ab08eull, 0x97ce9255ec4357abull, \
    0x9837f0518db8a96full, 0x98a1976f7597e996ull, 0x990b87e266c189aaull, 0x9975c1dd47518c77ull, \
    0x99e0459320b7fa65ull, 0x9a4b13371fd166caull, 0x9ab62afc94ff864aull, 0x9b218d16f441d63dull, \
    0x9b8d39b9d54e5539ull, 0x9bf93118f3aa4cc1ull, 0x9c6573682ec32c2dull, 0x9cd200db8a0774cbull, \
    0x9d3ed9a72cffb751ull, 0x9dabfdff6367a2aaull, 0x9e196e189d472420ull, 0x9e872a276f0b98ffull, \
    0x9ef5326091a111aeull, 0x9f6386f8e28ba651ull, 0x9fd228256400dd06ull, 0xa041161b3d0121beull, \
    0xa0b0510fb9714fc2ull, 0xa11fd9384a344cf7ull, 0xa18faeca8544b6e4ull, 0xa1ffd1fc25cea188ull, \
    0xa27043030c496819ull, 0xa2e102153e918f9eull, 0xa3520f68e802bb93ull, 0xa3c36b345991b47cull, \
    0xa43515ae09e6809eull, 0xa4a70f0c95768ec5ull, 0xa5195786be9ef339ull, 0xa58bef536dbeb6eeull, \
    0xa5fed6a9b15138eaull, 0xa6720dc0be08a20cull, 0xa6e594cfeee86b1eull, 0xa7596c0ec55ff55bull, \
    0xa7cd93b4e965356aull, 0xa8420bfa298f70d1ull, 0xa8b6d5167b320e09ull, 0xa92bef41fa77771bull, \
    0xa9a15ab4ea7c0ef8ull, 0xaa1717a7b5693979ull, 0xaa8d2652ec907629ull, 0xab0386ef48868de1ull, \
    0xab7a39b5a93ed337ull, 0xabf13edf162675e9ull, 0xac6896a4be3fe929ull, 0xace0413ff83e5d04ull, \
    0xad583eea42a14ac6ull, 0xadd08fdd43d01491ull, 0xae493452ca35b80eull, 0xaec22c84cc5c9465ull, \
    0xaf3b78ad690a4375ull, 0xafb51906e75b8661ull, 0xb02f0dcbb6e04584ull, 0xb0a957366fb7a3c9ull, \
    0xb123f581d2ac2590ull, 0xb19ee8e8c94feb09ull, 0xb21a31a66618fe3bull, 0xb295cff5e47db4a4ull, \
    0xb311c412a9112489ull, 0xb38e0e38419fae18ull, 0xb40aaea2654b9841ull, 0xb487a58cf4a9c180ull, \
    0xb504f333f9de6484ull, 0xb58297d3a8b9f0d2ull, 0xb60093a85ed5f76cull, 0xb67ee6eea3b22b8full, \
    0xb6fd91e328d17791ull, 0xb77c94c2c9d725e9ull, 0xb7fbefca8ca41e7cull, 0xb87ba337a1743834ull, \
    0xb8fbaf4762fb9ee9ull, 0xb97c143756844dbfull, 0xb9fcd2452c0b9debull, 0xba7de9aebe5fea09ull, \
    0xbaff5ab2133e45fbull, 0xbb81258d5b704b6full, 0xbc034a7ef2e9fb0dull, 0xbc85c9c560e7b269ull, \
    0xbd08a39f580c36bfull, 0xbd8bd84bb67ed483ull, 0xbe0f6809860993e2ull, 0xbe935317fc378238ull, \
    0xbf1799b67a731083ull, 0xbf9c3c248e2486f8ull, 0xc0213aa1f0d08db0ull, 0xc0a6956e8836ca8dull, \
    0xc12c4cca66709456ull, 0xc1b260f5ca0fbb33ull, 0xc238d2311e3d6673ull, 0xc2bfa0bcfad907c9ull, \
    0xc346ccda24976407ull, 0xc3ce56c98d21b15dull, 0xc4563ecc5334cb33ull, 0xc4de8523c2c07baaull, \
    0xc5672a115506daddull, 0xc5f02dd6b0bbc3d9ull, 0xc67990b5aa245f79ull, 0xc70352f04336c51eull, \
    0xc78d74c8abb9b15dull, 0xc817f681416452b2ull, 0xc8a2d85c8ffe2c45ull, 0xc92e1a9d517f0eccull, \
    0xc9b9bd866e2f27a3ull, 0xca45c15afcc72624ull, 0xcad2265e4290774eull, 0xcb5eecd3b38597c9ull, \
    0xcbec14fef2727c5dull, 0xcc799f23d11510e5ull, 0xcd078b86503dcdd2ull, 0xcd95da6a9ff06445ull, \
    0xce248c151f8480e4ull, 0xceb3a0ca5dc6a55dull, 0xcf4318cf191918c1ull, 0xcfd2f4683f94eeb5ull, \
    0xd06333daef2b2595ull, 0xd0f3d76c75c5db8dull, 0xd184df6251699ac6ull, 0xd2164c023056bcabull, \
    0xd2a81d91f12ae45aull, 0xd33a5457a3029054ull, 0xd3ccf099859ac379ull, 0xd45ff29e0972c561ull, \
    0xd4f35aabcfedfa1full, 0xd5872909ab75d18aull, 0xd61b5dfe9f9bce07ull, 0xd6aff9d1e13ba2feull, \
    0xd744fccad69d6af4ull, 0xd7da67311797f56aull, 0xd870394c6db32c84ull, 0xd9067364d44a929cull, \
    0xd99d15c278afd7b6ull, 0xda3420adba4d8704ull, 0xdacb946f2ac9cc72ull, 0xdb63714f8e295255ull, \
    0xdbfbb797daf23755ull, 0xdc9467913a4f1c92ull, 0xdd2d818508324c20ull, 0xddc705bcd378f7f0ull, \
    0xde60f4825e0e9124ull, 0xdefb4e1f9d1037f2ull, 0xdf9612deb8f04420ull, 0xe031430a0d99e627ull, \
    0xe0ccdeec2a94e111ull, 0xe168e6cfd3295d23ull, 0xe2055afffe83d369ull, 0xe2a23bc7d7d91226ull, \
    0xe33f8972be8a5a51ull, 0xe3dd444c46499619ull, 0xe47b6ca0373da88dull, 0xe51a02ba8e26d681ull, \
    0xe5b906e77c8348a8ull, 0xe658797368b3a717ull, 0xe6f85aaaee1fce22ull, 0xe798aadadd5b9cbfull, \
    0xe8396a503c4bdc68ull, 0xe8da9958464b42abull, 0xe97c38406c4f8c57ull, 0xea1e4756550eb27bull, \
    0xeac0c6e7dd24392full, 0xeb63b74317369840ull, 0xec0718b64c1cbddcull, 0xecaaeb8ffb03ab41ull, \
    0xed4f301ed9942b84ull, 0xedf3e6b1d418a491ull, 0xee990f980da3025bull, 0xef3eab20e032bc6bull, \
    0xefe4b99bdcdaf5cbull, 0xf08b3b58cbe8b76aull, 0xf13230a7ad094509ull, 0xf1d999d8b7708cc1ull, \
    0xf281773c59ffb13aull, 0xf329c9233b6bae9cull, 0xf3d28fde3a641a5bull, 0xf47bcbbe6db9fddfull, \
    0xf5257d152486cc2cull, 0xf5cfa433e6537290ull, 0xf67a416c733f846eull, 0xf7255510c4288239ull, \
    0xf7d0df730ad13bb9ull, 0xf87ce0e5b2094d9cull, 0xf92959bb5dd4ba74ull, 0xf9d64a46eb939f35ull, \
    0xfa83b2db722a033aull, 0xfb3193cc4227c3f4ull, 0xfbdfed6ce5f09c49ull, 0xfc8ec01121e447bbull, \
    0xfd3e0c0cf486c175ull, 0xfdedd1b496a89f35ull, 0xfe9e115c7b8f884cull, 0xff4ecb59511ec8a5ull, \
}

GDTK_HD int64_t gdtk_bits(double x) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(x);
#else
    int64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif

}

GDTK_HD double gdtk_from_bits(int64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}

GDTK_HD double gdtk_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return __builtin_fma(a, b, c);
#endif
}

// ---------------------------------------------------------------- 64-bit products on the integer pipe
GDTK_HD uint64_t gdtk_mul32(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
GDTK_HD uint32_t gdtk_mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// High 64 bits of a b without the lowest partial product's carry: at most 3 below the exact value.
GDTK_HD uint64_t gdtk_mulhi64(uint64_t a, uint64_t b) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return gdtk_mul32(ah, bh) + gdtk_mulhi32(ah, bl) + gdtk_mulhi32(al, bh);
}

GDTK_FN double gdtk_exp(double x, const uint64_t* tab) {
    const uint64_t b = (uint64_t)gdtk_bits(x);
    const uint32_t hi = (uint32_t)(b >> 32), e = (hi >> 20) & 0x7ff;
    if (e >= 1033u) {   // |x| >= 1024, infinite or NaN
        if ((b & 0x7fffffffffffffffull) > 0x7ff0000000000000ull) return x;
        return (hi >> 31) ? 0.0 : gdtk_from_bits(0x7ff0000000000000LL);
    }
    // X = |x| 2^54 (bits below are dropped)
    const uint64_t m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 11;
    const uint32_t n = 1032u - e;
    const uint64_t X = n > 63u ? 0 : m >> n;
    // |x| log2(e) = k + f: X times log2(e) 2^63 to 96 bits, 2^117 standing for 1
    const uint32_t xh = (uint32_t)(X >> 32), xl = (uint32_t)X, ch = 0xb8aa3b29u, cl = 0x5c17f0bcu;
    const uint64_t p0 = gdtk_mul32(xl, cl);
    const uint64_t p1 = gdtk_mul32(xh, cl) + (p0 >> 32);
    const uint64_t p2 = gdtk_mul32(xl, ch) + (uint32_t)p1;
    const uint64_t p3 = gdtk_mul32(xh, ch) + (p1 >> 32) + (p2 >> 32);
    int k = (int)(p3 >> 53);
    uint64_t f = (p3 << 11) | ((uint32_t)p2 >> 21);   // fraction, 2^64 standing for 1
    if (hi >> 31) { k = -k - (f != 0); f = 0 - f; }
    // 2^(f - j/256) = 1 + 2^-8 u (c1 + u (c2 + u (c3 + u (c4 + u c5)))), u the fraction below j in units of
    // 2^-8, c_n = (ln 2)^n / n! 2^(-8 (n - 1)); c3..c5 and their products in units of 2^-51, the rest of 2^-64
    const uint64_t u = f << 8;
    const uint32_t u32 = (uint32_t)(u >> 32);
    const uint32_t v = 1907106652u + gdtk_mulhi32(u32, 1290923u + gdtk_mulhi32(u32, 699u));
    const uint64_t s = (2113054701612ull + gdtk_mulhi32(u32, v)) << 13;
    const uint64_t q = gdtk_mulhi64(u, 0xb17217f7d1cf79acull + gdtk_mulhi64(u, s));
    const uint64_t T = tab[(uint32_t)(f >> 56)];
    const uint64_t M = T + (gdtk_mulhi64(T, q) >> 8);
    const uint64_t r = (M >> 11) + ((M >> 10) & 1);   // 53 bits, rounded
    if (k > -1022 && k < 1023) return gdtk_from_bits((int64_t)(r + ((uint64_t)(uint32_t)(k + 1022) << 52)));
    if (k > 1023) return gdtk_from_bits(0x7ff0000000000000LL);
    if (k < -1080) return 0.0;
    // near the ends of the range: scale in two exact-power steps (the second may round
    // into the subnormal range, as the true result does)
    const double y = gdtk_from_bits((int64_t)(r + ((uint64_t)1022 << 52)));
    const int m1 = k / 2, m2 = k - m1;
    return (y * gdtk_from_bits((int64_t)(1023 + m1) << 52)) * gdtk_from_bits((int64_t)(1023 + m2) << 52);
}

#ifdef __CUDA_ARCH__
static __device__ __noinline__ double gdtk_div_ieee(double a, double b) { return a / b; }
#endif

// 2^64 / y for y = B / 2^63 in [1, 2), within a few units: the FP32 reciprocal of y's leading 24 bits
// (rcp.approx.ftz.f32, relative error below 2^-21 in all) as a 32-bit fraction R0, then
// R = R0 (1 + e + e^2) with e = 1 - y R0, whose error e^3 is below 2^-63.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint64_t gdtk_rcp64(uint64_t B) {
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__uint_as_float(0x3f800001u + ((uint32_t)(B >> 40) & 0x7fffffu))));
    // in [1/2, 1) whatever the approximation's last bit
    const uint32_t R0 = (min(max(__float_as_uint(rf), 0x3f000000u), 0x3f7fffffu) << 8) | 0x80000000u;
    const uint64_t T = gdtk_mul32((uint32_t)(B >> 32), R0) + gdtk_mulhi32((uint32_t)B, R0);
    int64_t E = (int64_t)(0x8000000000000000ull - T);   // e 2^63, below 2^43
    const int32_t E1 = (int32_t)(E >> 12);
    E += (int64_t)((uint64_t)((int64_t)E1 * E1) >> 39);
    const int32_t Eh = (int32_t)(E >> 11);
    const int64_t c = (int64_t)Eh * (int64_t)(uint64_t)R0 + gdtk_mulhi32(R0, (uint32_t)E << 21);
    return ((uint64_t)R0 << 32) + (uint64_t)(c >> 20);
}
#endif

// a / b within 0.51 ulp (99.9% correctly rounded) on the integer pipe: the 64-bit reciprocal of b's
// significand times a's, rounded once.  Operands and quotients that are not normal numbers (zero,
// subnormal, infinite, NaN) take one shared out-of-line IEEE division; a zero numerator over a normal
// divisor, which the rates of absent species give at every step, does not.
// An FP64 instruction holds an SM's FP64 pipe for 19 cycles (76 for each of the four sub-partitions'
// warps), so the reciprocal seed and 4 FP64 operations of a Newton-Raphson division took about 330
// cycles; this takes about 100 of the integer pipe's, which runs beside it.
GDTK_FN double gdtk_div(double a, double b) {
#ifdef __CUDA_ARCH__
    const uint64_t ua = (uint64_t)__double_as_longlong(a), ub = (uint64_t)__double_as_longlong(b);
    const uint32_t ha = (uint32_t)(ua >> 32), hb = (uint32_t)(ub >> 32);
    const uint32_t ea = (ha >> 20) & 0x7ff, eb = (hb >> 20) & 0x7ff;
    uint64_t q = gdtk_mulhi64((ua << 11) | 0x8000000000000000ull, gdtk_rcp64((ub << 11) | 0x8000000000000000ull));
    const uint32_t ge = (uint32_t)(q >> 63);      // the significands' quotient is in (1/2, 2), 2^63 standing for 1
    q <<= 1 - ge;
    const uint32_t ex = ea - eb + ge + 1021;      // exponent field less the leading bit's 1
    const uint64_t sign = (uint64_t)((ha ^ hb) & 0x80000000u) << 32;
    if (eb - 1u < 2046u) {
        if (ea - 1u < 2046u && ex < 2045u)
            return __longlong_as_double((long long)(((q >> 11) + ((q >> 10) & 1) + ((uint64_t)ex << 52)) | sign));
        if ((ua << 1) == 0) return __longlong_as_double((long long)sign);
    }
    return gdtk_div_ieee(a, b);
#else
    return a / b;
#endif
}

// 1 / b as gdtk_div, without the product.
GDTK_HD double gdtk_rcp(double b) {
#ifdef __CUDA_ARCH__
    const uint64_t ub = (uint64_t)__double_as_longlong(b);
    const uint32_t hb = (uint32_t)(ub >> 32), eb = (hb >> 20) & 0x7ff;
    uint64_t q = gdtk_rcp64((ub << 11) | 0x8000000000000000ull);   // 2^64 / y, in (2^63, 2^64), or 2^64 - few at y = 1
    if (eb - 1u < 2044u && (ub << 12) != 0)
        return __longlong_as_double((long long)((q >> 11) + ((q >> 10) & 1) + ((uint64_t)(2044u - eb) << 52)) |
                                    (long long)((uint64_t)(hb & 0x80000000u) << 32));
    return gdtk_div_ieee(1.0, b);
#else
    return 1.0 / b;
#endif
}

#ifdef __CUDACC__
// ln x on the integer pipe, after the same kind of table method (P. T. P. Tang, "Table-driven implementation of the
// logarithm function in IEEE floating-point arithmetic", ACM TOMS 16(4):378-400, 1990): x = 2^k z with z in
// [1/sqrt 2, sqrt 2), r = z inv_j - 1 with |r| < 2^-8.9 from a 32-bit reciprocal inv_j of z's interval,
//   ln x = k ln 2 - ln inv_j + r - r^2 (1/2 - r (1/3 - r (1/4 - r (1/5 - r/6)))),
// in 64-bit fixed point: 2^-62 for |k| <= 1, 2^-53 beyond, rounded once.  Within 1.2 ulp (99% correctly
// rounded; 0.13 ulp beyond the half for temperatures).  Within 1/16 of 1, where fixed point would lose
// relative accuracy, and for operands that are not positive normal numbers, the library's log runs.
// About 150 cycles of the integer pipe where the library's log takes 2,200 (its FP64 operations).
struct GdtkLogEntry { uint32_t inv, pad; int64_t L; };   // inv_j 2^31, -ln(inv_j) 2^62
static __device__ const __align__(16) GdtkLogEntry kGdtkLogTable[256] = {
    {0x7fc01ff0u, 0u, 8998414665322726ll}, {0x7f411e53u, 0u, 26942739767671375ll}, {0x7ec31843u, 0u, 44817515941805768ll}, {0x7e460adau, 0u, 62623274883990110ll},
    {0x7dc9f339u, 0u, 80360551694122604ll}, {0x7d4ece90u, 0u, 98029867128141961ll}, {0x7cd49a16u, 0u, 115631744678121797ll}, {0x7c5b5311u, 0u, 133166692686875710ll},
    {0x7be2f6ceu, 0u, 150635221558767311ll}, {0x7b6b82a7u, 0u, 168037830191025763ll}, {0x7af4f3feu, 0u, 185375016692622223ll}, {0x7a7f4841u, 0u, 202647269157614344ll},
    {0x7a0a7ce7u, 0u, 219855072001972700ll}, {0x79968f70u, 0u, 236998905667667615ll}, {0x79237d66u, 0u, 254079244056126874ll}, {0x78b1445cu, 0u, 271096556464898743ll},
    {0x783fe1f0u, 0u, 288051302715514983ll}, {0x77cf53c6u, 0u, 304943944239267715ll}, {0x775f978cu, 0u, 321774934689206548ll}, {0x76f0aafau, 0u, 338544719593703353ll},
    {0x76828bceu, 0u, 355253745286495101ll}, {0x761537d0u, 0u, 371902449414049796ll}, {0x75a8acd0u, 0u, 388491265257703956ll}, {0x753ce8a5u, 0u, 405020623810608869ll},
    {0x74d1e92fu, 0u, 421490948844782801ll}, {0x7467ac55u, 0u, 437902661321886349ll}, {0x73fe3007u, 0u, 454256174424373105ll}, {0x7395723bu, 0u, 470551900375692550ll},
    {0x732d70eeu, 0u, 486790247864139666ll}, {0x72c62a25u, 0u, 502971619415284002ll}, {0x725f9becu, 0u, 519096413519673428ll}, {0x71f9c457u, 0u, 535165021986376158ll},
    {0x7194a17fu, 0u, 551177836925622749ll}, {0x71303185u, 0u, 567135243310430132ll}, {0x70cc7290u, 0u, 583037623570703728ll}, {0x706962cdu, 0u, 598885357396484511ll},
    {0x70070070u, 0u, 614678819086588057ll}, {0x6fa549b4u, 0u, 630418377308047487ll}, {0x6f443cd9u, 0u, 646104399795544406ll}, {0x6ee3d826u, 0u, 661737248235284705ll},
    {0x6e8419e7u, 0u, 677317282996234308ll}, {0x6e25006eu, 0u, 692844860474337203ll}, {0x6dc68a14u, 0u, 708320330385570556ll}, {0x6d68b535u, 0u, 723744045569794039ll},
    {0x6d0b8037u, 0u, 739116344266583717ll}, {0x6caee980u, 0u, 754437575033772291ll}, {0x6c52ef7fu, 0u, 769708073955014501ll}, {0x6bf790a9u, 0u, 784928171944926363ll},
    {0x6b9ccb74u, 0u, 800098207313144792ll}, {0x6b429e60u, 0u, 815218502701246718ll}, {0x6ae907efu, 0u, 830289385274817177ll}, {0x6a9006a9u, 0u, 845311176363512741ll},
    {0x6a37991au, 0u, 860284196426430952ll}, {0x69dfbdd4u, 0u, 875208759732378773ll}, {0x6988736du, 0u, 890085179357474207ll}, {0x6931b880u, 0u, 904913764443615003ll},
    {0x68db8bacu, 0u, 919694822648866029ll}, {0x6885eb96u, 0u, 934428654758074857ll}, {0x6830d6e5u, 0u, 949115565021521522ll}, {0x67dc4c46u, 0u, 963755850521454019ll},
    {0x67884a6au, 0u, 978349806266680797ll}, {0x6734d006u, 0u, 992897725060488525ll}, {0x66e1dbd5u, 0u, 1007399892024455381ll}, {0x668f6c92u, 0u, 1021856600462332500ll},
    {0x663d8100u, 0u, 1036268130385690913ll}, {0x65ec17e3u, 0u, 1050634767090447204ll}, {0x659b3006u, 0u, 1064956784915951354ll}, {0x654ac836u, 0u, 1079234460552435617ll},
    {0x64fadf43u, 0u, 1093468070267000678ll}, {0x64ab7402u, 0u, 1107657884348286326ll}, {0x645c854bu, 0u, 1121804172405517996ll}, {0x640e11fbu, 0u, 1135907197778666113ll},
    {0x63c018f0u, 0u, 1149967228381423150ll}, {0x6372990eu, 0u, 1163984522868633405ll}, {0x6325913cu, 0u, 1177959338731095526ll}, {0x62d90063u, 0u, 1191891934979272455ll},
    {0x628ce570u, 0u, 1205782566509264075ll}, {0x62413f54u, 0u, 1219631483962893425ll}, {0x61f60d03u, 0u, 1233438936393365249ll}, {0x61ab4d73u, 0u, 1247205173980846614ll},
    {0x6160ff9fu, 0u, 1260930439506910557ll}, {0x61172283u, 0u, 1274614979495676078ll}, {0x60cdb521u, 0u, 1288259029999992381ll}, {0x6084b67bu, 0u, 1301862833462840222ll},
    {0x603c2597u, 0u, 1315426627317138432ll}, {0x5ff40180u, 0u, 1328950640977984829ll}, {0x5fac4940u, 0u, 1342435112895891728ll}, {0x5f64fbe7u, 0u, 1355880270452327193ll},
    {0x5f1e1886u, 0u, 1369286344181091286ll}, {0x5ed79e32u, 0u, 1382653559054895200ll}, {0x5e918c01u, 0u, 1395982143060524553ll}, {0x5e4be10fu, 0u, 1409272312604336304ll},
    {0x5e069c77u, 0u, 1422524292746930707ll}, {0x5dc1bd58u, 0u, 1435738302608003052ll}, {0x5d7d42d5u, 0u, 1448914555220258396ll}, {0x5d392c10u, 0u, 1462053272125995914ll},
    {0x5cf57831u, 0u, 1475154662741235988ll}, {0x5cb22662u, 0u, 1488218935986329459ll}, {0x5c6f35cdu, 0u, 1501246306170076965ll}, {0x5c2ca5a0u, 0u, 1514236981081322215ll},
    {0x5bea750du, 0u, 1527191161841090063ll}, {0x5ba8a344u, 0u, 1540109060748009884ll}, {0x5b672f7du, 0u, 1552990871308399167ll}, {0x5b2618ecu, 0u, 1565836804108261702ll},
    {0x5ae55ecdu, 0u, 1578647050710764020ll}, {0x5aa5005bu, 0u, 1591421810631588989ll}, {0xb4c9f9a5u, 0u, -1592415877503655658ll}, {0xb44aa6e9u, 0u, -1579711499949419975ll},
    {0xb3cc0706u, 0u, -1567042025113367036ll}, {0xb34e1884u, 0u, -1554407261444135171ll}, {0xb2d0d9efu, 0u, -1541807018798566496ll}, {0xb25449d7u, 0u, -1529241108508507520ll},
    {0xb1d866d1u, 0u, -1516709344993442917ll}, {0xb15d2f75u, 0u, -1504211542749137499ll}, {0xb0e2a260u, 0u, -1491747519502129740ll}, {0xb068be31u, 0u, -1479317091623858286ll},
    {0xafef818cu, 0u, -1466920078843777911ll}, {0xaf76eb18u, 0u, -1454556301205324177ll}, {0xaefef982u, 0u, -1442225583825591229ll}, {0xae87ab76u, 0u, -1429927745981102704ll},
    {0xae10ffa9u, 0u, -1417662616863268482ll}, {0xad9af4d0u, 0u, -1405430021502054851ll}, {0xad2589a3u, 0u, -1393229785513888461ll}, {0xacb0bce1u, 0u, -1381061741516990409ll},
    {0xac3c8d4au, 0u, -1368925719688238155ll}, {0xabc8f9a0u, 0u, -1356821549370109534ll}, {0xab5600abu, 0u, -1344749065515941710ll}, {0xaae3a136u, 0u, -1332708103976426703ll},
    {0xaa71da0du, 0u, -1320698498323498847ll}, {0xaa00aa01u, 0u, -1308720086325492472ll}, {0xa9900fe6u, 0u, -1296772706796545879ll}, {0xa9200a92u, 0u, -1284856198021137741ll},
    {0xa8b098e0u, 0u, -1272970402671574721ll}, {0xa841b9adu, 0u, -1261115162999054144ll}, {0xa7d36bd7u, 0u, -1249290319225144085ll}, {0xa765ae43u, 0u, -1237495719402748713ll},
    {0xa6f87fd6u, 0u, -1225731208026790920ll}, {0xa68bdf79u, 0u, -1213996632623935117ll}, {0xa61fcc16u, 0u, -1202291838860556536ll}, {0xa5b4449du, 0u, -1190616678846142292ll},
    {0xa54947fdu, 0u, -1178970999606172190ll}, {0xa4ded52cu, 0u, -1167354656387523200ll}, {0xa474eb1fu, 0u, -1155767499422462819ll}, {0xa40b88d0u, 0u, -1144209383950200553ll},
    {0xa3a2ad39u, 0u, -1132680161911568359ll}, {0xa33a575au, 0u, -1121179692042153787ll}, {0xa2d28634u, 0u, -1109707831546283239ll}, {0xa26b38c8u, 0u, -1098264434414916872ll},
    {0xa2046e1fu, 0u, -1086849364987873504ll}, {0xa19e253fu, 0u, -1075462479402497102ll}, {0xa1385d35u, 0u, -1064103642570303542ll}, {0xa0d3150cu, 0u, -1052772712931013228ll},
    {0xa06e4bd4u, 0u, -1041469554394186731ll}, {0xa00a00a0u, 0u, -1030194032999036460ll}, {0x9fa63284u, 0u, -1018946013524027557ll}, {0x9f42e095u, 0u, -1007725359498178428ll},
    {0x9ee009eeu, 0u, -996531941863230650ll}, {0x9e7dada9u, 0u, -985365626949627204ll}, {0x9e1bcae3u, 0u, -974226283400373018ll}, {0x9dba60bbu, 0u, -963113780482004585ll},
    {0x9d596e54u, 0u, -952027991611287314ll}, {0x9cf8f2d1u, 0u, -940968787425622140ll}, {0x9c98ed58u, 0u, -929936041040109964ll}, {0x9c395d10u, 0u, -918929624582666935ll},
    {0x9bda4124u, 0u, -907949414497436759ll}, {0x9b7b98c0u, 0u, -896995286316408663ll}, {0x9b1d6311u, 0u, -886067114671919769ll}, {0x9abf9f48u, 0u, -875164778638120800ll},
    {0x9a624c97u, 0u, -864288156465145665ll}, {0x9a056a31u, 0u, -853437125591909928ll}, {0x99a8f74cu, 0u, -842611566236746512ll}, {0x994cf320u, 0u, -831811359659272758ll},
    {0x98f15ce7u, 0u, -821036388194444172ll}, {0x989633dbu, 0u, -810286531683792990ll}, {0x983b773bu, 0u, -799561676495960865ll}, {0x97e12644u, 0u, -788861702955043965ll},
    {0x97874039u, 0u, -778186499803412671ll}, {0x972dc45bu, 0u, -767535949774252256ll}, {0x96d4b1efu, 0u, -756909940476813953ll}, {0x967c083bu, 0u, -746308358993170991ll},
    {0x9623c686u, 0u, -735731091892001635ll}, {0x95cbec1bu, 0u, -725178030747478488ll}, {0x95747844u, 0u, -714649063020117939ll}, {0x951d6a4du, 0u, -704144077559053380ll},
    {0x94c6c187u, 0u, -693662970179884809ll}, {0x94707d3fu, 0u, -683205627096681164ll}, {0x941a9cc8u, 0u, -672771943391177914ll}, {0x93c51f75u, 0u, -662361811970927450ll},
    {0x9370049cu, 0u, -651975129155842424ll}, {0x931b4b91u, 0u, -641611785391810809ll}, {0x92c6f3acu, 0u, -631271676438878673ll}, {0x9272fc48u, 0u, -620954701571842368ll},
    {0x921f64bfu, 0u, -610660756112309651ll}, {0x91cc2c6cu, 0u, -600389735172205242ll}, {0x917952aeu, 0u, -590141539337210897ll}, {0x9126d6e5u, 0u, -579916069063401419ll},
    {0x90d4b86fu, 0u, -569713218998450277ll}, {0x9082f6b0u, 0u, -559532893150689480ll}, {0x9031910au, 0u, -549374989758582671ll}, {0x8fe086e2u, 0u, -539239410795507244ll},
    {0x8f8fd7a0u, 0u, -529126062026930318ll}, {0x8f3f82a8u, 0u, -519034839635388937ll}, {0x8eef8766u, 0u, -508965653208050757ll}, {0x8e9fe542u, 0u, -498918402771541270ll},
    {0x8e509ba8u, 0u, -488892994154381331ll}, {0x8e01aa05u, 0u, -478889333258426590ll}, {0x8db30fc6u, 0u, -468907324134599449ll}, {0x8d64cc5cu, 0u, -458946876753812749ll},
    {0x8d16df35u, 0u, -449007893447817753ll}, {0x8cc947c5u, 0u, -439090286413124090ll}, {0x8c7c057du, 0u, -429193960221897251ll}, {0x8c2f17d2u, 0u, -419318825479812684ll},
    {0x8be27e39u, 0u, -409464791044779386ll}, {0x8b963829u, 0u, -399631767960408269ll}, {0x8b4a451au, 0u, -389819667519605085ll}, {0x8afea483u, 0u, -380028397325435527ll},
    {0x8ab355e0u, 0u, -370257873156179479ll}, {0x8a6858abu, 0u, -360508005163392945ll}, {0x8a1dac60u, 0u, -350778705786029316ll}, {0x89d3507du, 0u, -341069889787707457ll},
    {0x89894480u, 0u, -331381470296857181ll}, {0x893f87e8u, 0u, -321713360804922057ll}, {0x88f61a37u, 0u, -312065479196750375ll}, {0x88acfaeeu, 0u, -302437739764352437ll},
    {0x8864298fu, 0u, -292830057212219676ll}, {0x881ba59eu, 0u, -283242348693464148ll}, {0x87d36ea0u, 0u, -273674531823666025ll}, {0x878b841au, 0u, -264126522669600233ll},
    {0x8743e595u, 0u, -254598243873543112ll}, {0x86fc9296u, 0u, -245089608442271133ll}, {0x86b58aa8u, 0u, -235600540064296469ll}, {0x866ecd53u, 0u, -226130954829062788ll},
    {0x86285a23u, 0u, -216680775502370960ll}, {0x85e230a3u, 0u, -207249921340665572ll}, {0x859c5060u, 0u, -197838314237982453ll}, {0x8556b8e7u, 0u, -188445874640932310ll},
    {0x851169c7u, 0u, -179072525676171835ll}, {0x84cc6290u, 0u, -169718191118579122ll}, {0x8487a2d1u, 0u, -160382791260219186ll}, {0x84432a1bu, 0u, -151066249120404785ll},
    {0x83fef802u, 0u, -141768492566349147ll}, {0x83bb0c18u, 0u, -132489443939024929ll}, {0x837765f0u, 0u, -123229026280115809ll}, {0x83340520u, 0u, -113987167539447640ll},
    {0x82f0e93du, 0u, -104763792237292842ll}, {0x82ae11deu, 0u, -95558827750151755ll}, {0x826b7e99u, 0u, -86372198026240537ll}, {0x82292f08u, 0u, -77203834120173305ll},
    {0x81e722c2u, 0u, -68053659461191774ll}, {0x81a55963u, 0u, -58921606748578577ll}, {0x8163d283u, 0u, -49807598933376560ll}, {0x81228dbfu, 0u, -40711568288616261ll},
    {0x80e18ab3u, 0u, -31633443714015211ll}, {0x80a0c8fbu, 0u, -22573152848700295ll}, {0x80604836u, 0u, -13530628491512705ll}, {0x80200802u, 0u, -4505800079136905ll}};
static __device__ __noinline__ double gdtk_log(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const uint32_t e = (uint32_t)(b >> 52);
    if (e - 1u >= 2046u || b - 0x3fee000000000000ull < 0x3ff1000000000000ull - 0x3fee000000000000ull) return log(x);
    const uint32_t j = (uint32_t)(b >> 44) & 255u;
    const int up = j >= 106;                                              // significand above sqrt 2: z is its half
    const int k = (int)e - 1023 + up;
    const uint64_t z = ((b << 11) | 0x8000000000000000ull) >> up;         // 2^63
    const uint32_t inv = kGdtkLogTable[j].inv;
    const int64_t L = kGdtkLogTable[j].L;
    const int64_t r = (int64_t)(gdtk_mul32((uint32_t)(z >> 32), inv) + gdtk_mulhi32((uint32_t)z, inv) - 0x4000000000000000ull);   // 2^62
    const int r32 = (int)(r >> 23);                                       // 2^39
    int C = 429496730 - (__mulhi(r32, 357913941) >> 7);                   // 2^31: 1/5 - r/6
    C = 536870912 - (__mulhi(r32, C) >> 7);
    C = 715827883 - (__mulhi(r32, C) >> 7);                               // 1/3 - r (1/4 - ...)
    const uint64_t B = 0x2000000000000000ull - (uint64_t)(((int64_t)r32 * C) >> 8);   // 2^62: 1/2 - r C
    const uint64_t a = (uint64_t)(r < 0 ? -r : r) << 8;                   // 2^70
    const int64_t s = L + r - (int64_t)(gdtk_mulhi64(gdtk_mulhi64(a, a), B << 2) >> 14);
    int64_t v;
    uint32_t scale;
    if (k + 1u <= 2u) {
        v = s + (int64_t)k * 0x2c5c85fdf473de6bll;
        scale = 62;
    } else {
        v = (int64_t)k * 0x162e42fefa39efll + (((int64_t)k * 219028) >> 20) + ((s + 256) >> 9);
        scale = 53;
    }
    uint64_t u = (uint64_t)(v < 0 ? -v : v);
    const int c = __clzll((long long)u);
    u <<= c;
    const uint64_t m = (u >> 11) + ((u >> 10) & 1);
    return __longlong_as_double((long long)((m + ((uint64_t)(1085u - scale - (uint32_t)c) << 52)) |
                                            (v < 0 ? 0x8000000000000000ull : 0ull)));
}
#endif

}  // namespace gdtk
