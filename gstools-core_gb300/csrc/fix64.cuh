// fix64.cuh -- cosines of FP64 phases in 64-bit fixed point, on the integer
// pipes.
//
// GB300 issues an FP64 instruction at 1/64 of the FP32 rate (2 lanes per clock
// and SM; measured 1.7-2.0), a 32 x 32 -> 64 bit multiply-add at 30 and other
// integer instructions at about 60.  An FP64 sine or cosine of 11 to 13 FP64
// instructions therefore costs more than the same accuracy from some 25
// integer multiplies:
//
//   turn_fraction(ph)  |ph| < 2^32 as a fraction of a turn in units of 2^-64,
//                      whole turns dropped (the mantissa times 96 bits of
//                      2 / pi, shifted by the exponent), within 2^-60 turn;
//   turn_fraction_far(ph)  the same for |ph| < 2^44, from 128 bits of 2 / pi;
//   cos_fixed(theta)   the cosine of a turn fraction in units of 2^-62: one
//                      of 256 table entries and polynomials in the remainder.
//                      The error is 1.2e-16 RMS, 4.8e-16 the
//                      largest of 60,000 samples and 9e-16 at most (an FP64
//                      evaluation of the same degree, rounded at each step,
//                      has 7e-16 RMS).
//
// tests/test_fix64_cpu.py, test_fix64_far_cpu.py and test_fix64_products_cpu.py
// restate these and rn_product in exact integers, from the constants below.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gsc {

// cos(2 pi a / 256) in units of 2^-62, a = 0 .. 64
__device__ const uint64_t kQuarterCos[65] = {
    0x4000000000000000ull, 0x3ffb10c1099a1976ull, 0x3fec43c6f2dafbc7ull,
    0x3fd39b5a0310742aull, 0x3fb11b47a24a4b3cull, 0x3f84c8e1c33fa68full,
    0x3f4eaafe114a2d43ull, 0x3f0ec9f4e297526bull, 0x3ec52f9feeb96056ull,
    0x3e71e758c9cb118aull, 0x3e14fdf72461ae55ull, 0x3dae81ced092c67aull,
    0x3d3e82ad8c5bb4bbull, 0x3cc511d891c223ddull, 0x3c424209ed0dc97full,
    0x3bb6276d998478c2ull, 0x3b20d79e651a8c51ull, 0x3a8269a29b927359ull,
    0x39daf5e8798ee5e2ull, 0x392a96426823e9edull, 0x387165e3017b61a4ull,
    0x37af8158df2a533full, 0x36e5068a32dc7b22ull, 0x361214b02a03ff37ull,
    0x3536cc521d434606ull, 0x34534f408c4f03bbull, 0x3367c08fe70e8168ull,
    0x3274449324c7f69full, 0x317900d62a2e816aull, 0x30761c17ff2edba4ull,
    0x2f6bbe44d55f5dbcull, 0x2e5a106fdfff2c87ull, 0x2d413cccfe779921ull,
    0x2c216eaa3a59bdb7ull, 0x2afad26919d93f45ull, 0x29cd9577c7cbd228ull,
    0x2899e64a123bac30ull, 0x275ff45240a17279ull, 0x261feff9c2e069c2ull,
    0x24da0a99ba25bd51ull, 0x238e76735cd190d9ull, 0x223d66a836964508ull,
    0x20e70f3245ffdb2dull, 0x1f8ba4dbf89ab9fbull, 0x1e2b5d3806f63b1eull,
    0x1cc66e9931c45e17ull, 0x1b5d1009e15cc02bull, 0x19ef7943a8ed8a2eull,
    0x187de2a6aea962d2ull, 0x17088530fa459eafull, 0x158f9a75ab1fdcfeull,
    0x14135c9417660143ull, 0x1294062ed59f05a9ull, 0x1111d262b1f67761ull,
    0x0f8cfcbd90af8d58ull, 0x0e05c1353f27b17eull, 0x0c7c5c1e34d3055bull,
    0x0af10a22459fe32aull, 0x0964083747309d11ull, 0x07d59395aa5cc38dull,
    0x0645e9af0a6d0af8ull, 0x04b54824b3867d73ull, 0x0323ecbe21bb027dull,
    0x0192155f7a3667e0ull, 0x0000000000000000ull,
};

// With step = 2 pi / 256 and rho the remainder in table steps (|rho| <= 1/2):
//   1 - cos(step rho) = a1 rho^2 (1 - a2 rho^2)
//   sin(step rho)     = step rho (1 - s3 rho^2 + s5 rho^4)
// s3 = step^2 / 6, s5 = step^4 / 120 (Taylor); a1 and a2 are step^2 / 2 and
// step^2 / 12 with the sixth-order term, which would leave 4.8e-15, taken in
// by its minimax fit x^3 ~ 1.3923 x^2 - 0.4308 x on [0, 1] (1.8e-16 left).
constexpr uint64_t kStep69 = 0xc90fdaa22168c235ull;     // step 2^69
constexpr uint64_t kVersine75 = 0x9de9e64ddfc6dddbull;  // a1 2^75
constexpr uint32_t kVersineTwo = 1766222161u;          // a2 2^45
constexpr uint32_t kSineThree = 3532469012u;           // s3 2^45, half a unit up (see below)
constexpr uint32_t kSineFive = 53198u;                 // s5 2^44
// A phase offset is added to every turn fraction before the table look-up:
// half a table step (the index then rounds to nearest) less 2^-55 turn, the
// mean of what the truncated products in the sine's cubic term leave out.
constexpr uint64_t kCosOffset = (uint64_t(1) << 55) - (uint64_t(1) << 9);

// Table entries a = 0 .. 255 in shared memory: wide[a] = {cos low, cos high,
// step sin high, step sin low / 2}, narrow[a] = {a1 cos high, a1 cos low / 2},
// cos in units of 2^-62, the others of 2^-68.
struct CosTable {
    uint4 wide[256];
    uint2 narrow[256];
};

__device__ __forceinline__ int64_t quarter_cos(int a) {
    a &= 255;
    const int b = a & 127;
    const uint64_t v = kQuarterCos[b <= 64 ? b : 128 - b];
    // second and third quarters are negative
    return ((a + 64) & 128) ? -static_cast<int64_t>(v) : static_cast<int64_t>(v);
}

__device__ __forceinline__ void fill_cos_table(CosTable *t, int tid, int n) {
    for (int a = tid; a < 256; a += n) {
        const int64_t c = quarter_cos(a), s = quarter_cos(a - 64);
        int64_t ss = static_cast<int64_t>(__umul64hi(static_cast<uint64_t>(s < 0 ? -s : s), kStep69) << 1);
        int64_t cc = static_cast<int64_t>(__umul64hi(static_cast<uint64_t>(c < 0 ? -c : c), kVersine75) >> 5);
        if (s < 0) ss = -ss;
        if (c < 0) cc = -cc;
        t->wide[a] = make_uint4(static_cast<uint32_t>(c), static_cast<uint32_t>(c >> 32),
                                static_cast<uint32_t>(ss >> 32), static_cast<uint32_t>(ss) >> 1);
        t->narrow[a] = make_uint2(static_cast<uint32_t>(cc >> 32), static_cast<uint32_t>(cc) >> 1);
    }
}

// a >> n for n of 32 and more too (0), as the PTX instruction defines it
__device__ __forceinline__ uint32_t shr_clamp(uint32_t a, uint32_t n) {
    uint32_t r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(n));
    return r;
}

// ph / (2 pi) modulo one turn, in units of 2^-64, for |ph| < 2^32 (NaN and
// infinities give some value)
__device__ __forceinline__ uint64_t turn_fraction(double ph) {
    // the first 96 bits of 2 / pi
    constexpr uint32_t c2 = 0xA2F9836Eu, c1 = 0x4E441529u, c0 = 0xFC2757D1u;
    const uint32_t hi = static_cast<uint32_t>(__double2hiint(ph));
    const uint32_t lo = static_cast<uint32_t>(__double2loint(ph));
    uint32_t m1 = __funnelshift_l(lo, hi, 11) | 0x80000000u, m0 = lo << 11;   // 1.f, left-aligned
    // |ph| = m 2^(e - 63): the fraction is bits 97 - e .. 160 - e of m (2/pi 2^96),
    // taken by a left shift of t = e + 31 in 0 .. 63.  Phases below 2^-31 are
    // shifted down first (what that drops is below 2^-62 rad).
    const int t0 = static_cast<int>((hi >> 20) & 0x7ffu) - 992;
    const uint32_t down = static_cast<uint32_t>(max(-t0, 0));
    const uint32_t t = static_cast<uint32_t>(max(t0, 0));
    m0 = __funnelshift_rc(m0, m1, down);
    m1 = shr_clamp(m1, down);
    uint64_t w = static_cast<uint64_t>(__umulhi(m1, c0)) + __umulhi(m0, c1);
    w += static_cast<uint64_t>(m0) * c2;
    w += static_cast<uint64_t>(m1) * c1;                 // below 2^64: c1 + c2 < 2^32
    const uint32_t p2 = static_cast<uint32_t>(w);
    w = static_cast<uint64_t>(m1) * c2 + (w >> 32);
    const uint32_t p3 = static_cast<uint32_t>(w), p4 = static_cast<uint32_t>(w >> 32);
    const bool far = (t & 32u) != 0;
    const uint32_t a = far ? p4 : 0u, b = far ? p3 : p4, c = far ? p2 : p3;
    const uint32_t sign = static_cast<uint32_t>(static_cast<int32_t>(hi) >> 31);
    const uint32_t fh = __funnelshift_l(b, a, t) ^ sign, fl = __funnelshift_l(c, b, t) ^ sign;
    return (static_cast<uint64_t>(fh) << 32) | fl;
}

// As turn_fraction for |ph| < 2^44, within 2^-63 turn: the upper 128 bits of the
// mantissa times 2^128 2 / pi, shifted.
__device__ __forceinline__ uint64_t turn_fraction_far(double ph) {
    constexpr uint64_t ch = 0xA2F9836E4E441529ull, cl = 0xFC2757D1F534DDC0ull;
    const uint64_t bits = static_cast<uint64_t>(__double_as_longlong(ph));
    const uint64_t m = (bits << 11) | (uint64_t(1) << 63);                 // 1.f, left-aligned
    const uint64_t lo = m * ch, low = lo + __umul64hi(m, cl);              // bits 64..127 of the product
    const uint64_t high = __umul64hi(m, ch) + (low < lo ? 1u : 0u);        // 128..191
    // |ph| = m 2^(e - 63): the fraction starts at bit 129 - e of the product
    const int s = 1088 - static_cast<int>((bits >> 52) & 0x7ffu);          // 65 - e, at least 22
    const uint64_t f = s < 64 ? (high << (64 - s)) | (low >> s) : s < 128 ? high >> (s - 64) : 0u;
    return f ^ static_cast<uint64_t>(static_cast<int64_t>(bits) >> 63);
}

// cos(2 pi (theta - kCosOffset) / 2^64) in units of 2^-62
__device__ __forceinline__ int64_t cos_fixed(uint64_t theta, const CosTable *tab) {
    const uint32_t h = static_cast<uint32_t>(theta >> 32), l = static_cast<uint32_t>(theta);
    const uint32_t a = h >> 24;
    const uint4 e = tab->wide[a];
    const uint2 f = tab->narrow[a];
    // rho = (r1 + 2 r0 2^-32) 2^-32 table steps
    const int32_t r1 = static_cast<int32_t>(__funnelshift_l(l, h, 8) ^ 0x80000000u);
    const int32_t r0 = static_cast<int32_t>((l << 7) & 0x7fffffffu);
    // rho^2 in units of 2^-64 (+ 4: the truncated cross product never makes it negative)
    const int64_t sq = static_cast<int64_t>(r1) * r1 + 4 + (static_cast<int64_t>(__mulhi(r1, r0)) << 2);
    const uint32_t q = __funnelshift_l(static_cast<uint32_t>(sq),
                                       static_cast<uint32_t>(sq >> 32), 1);        // rho^2 2^33
    const uint32_t a2 = __umulhi(__umulhi(q, q), kVersineTwo);                     // a2 rho^4 2^47
    const int64_t v = sq - (static_cast<int64_t>(static_cast<int32_t>(a2)) << 17);
    const uint32_t s3 = __umulhi(q, kSineThree - __umulhi(q, kSineFive));          // 2^46
    const int64_t rho = (static_cast<int64_t>(r1) << 32) | (l << 8);
    const int64_t s = rho - (static_cast<int64_t>(__mulhi(r1, static_cast<int32_t>(s3))) << 18);
    const int32_t vh = static_cast<int32_t>(v >> 32), v0 = static_cast<int32_t>(static_cast<uint32_t>(v) >> 1);
    const int32_t sh = static_cast<int32_t>(s >> 32), s0 = static_cast<int32_t>(static_cast<uint32_t>(s) >> 1);
    const int32_t eh = static_cast<int32_t>(e.z), e0 = static_cast<int32_t>(e.w);
    const int32_t fh = static_cast<int32_t>(f.x), f0 = static_cast<int32_t>(f.y);
    // cos = cos_a - (a1 cos_a) v - (step sin_a) s, the products' low parts
    // from one-bit-short halves (their sum is doubled)
    int64_t p = static_cast<int64_t>(eh) * sh + static_cast<int64_t>(fh) * vh;
    p += static_cast<int64_t>(__mulhi(fh, v0) + __mulhi(f0, vh) + __mulhi(eh, s0)) << 1;
    p += static_cast<int64_t>(__mulhi(e0, sh)) << 1;
    const int64_t c = static_cast<int64_t>((static_cast<uint64_t>(e.y) << 32) | e.x);
    return c - (p >> 6);
}

// cos and sin of 2 pi (theta - kFineOffset) / 2^64 in units of 2^-62, within
// 1e-17: the same table steps with one more order of the cosine and 64-bit
// products, for factor tables, where an error is shared by many sums.
//   1 - cos(step rho) = f1 rho^2 (1 - f2 rho^2 + f3 rho^4)
//   sin(step rho)     = step rho (1 - f4 rho^2 + f5 rho^4)
// with the Taylor coefficients f1 = step^2 / 2, f2 = step^2 / 12, f3 =
// step^4 / 360, f4 = step^2 / 6, f5 = step^4 / 120 (the sine's next term is
// 8.4e-18).
constexpr uint64_t kFineOffset = uint64_t(1) << 55;
constexpr uint64_t kFine1 = 0x9de9e64df22ef2d2ull;     // f1 2^75
constexpr uint64_t kFine2 = 0x34a34cc4a60fa646ull;     // f2 2^76
constexpr uint64_t kFine3 = 0x000022a264558fb1ull;     // f3 2^75
constexpr uint64_t kFine4 = 0x34a34cc4a60fa646ull;     // f4 2^75
constexpr uint64_t kFine5 = 0x000033f396805789ull;     // f5 2^74
// (c, s: cos and sin of the table step theta >> 56)
__device__ __forceinline__ void cis_from(uint64_t theta, int64_t c, int64_t s, int64_t *cosine, int64_t *sine) {
    // rho 2^64 and rho^2 2^65 (at most 2^63)
    const int64_t rho = static_cast<int64_t>((theta << 8) ^ (uint64_t(1) << 63));
    const uint64_t q = static_cast<uint64_t>(__mul64hi(rho, rho)) << 1;
    // rho^2 (f2 - ..) in units of 2^-77, rho^2 (f4 - ..) of 2^-76
    const uint64_t lv = __umul64hi(q, kFine2 - __umul64hi(q, kFine3));
    const uint64_t ls = __umul64hi(q, kFine4 - __umul64hi(q, kFine5));
    // rho^2 (1 - ..) of 2^-65 and the versine of 2^-76; rho (1 - ..) of 2^-64 and the sine of 2^-68
    const uint64_t vq = q - (__umul64hi(q, lv) >> 13);
    const int64_t ver = static_cast<int64_t>(__umul64hi(vq, kFine1));
    const int64_t rs = rho - (__mul64hi(rho, static_cast<int64_t>(ls)) >> 12);
    const int64_t sn = __mul64hi(rs, static_cast<int64_t>(kStep69 >> 1));
    *cosine = c - (((__mul64hi(c, ver) >> 8) + __mul64hi(s, sn) + 8) >> 4);
    *sine = s - (((__mul64hi(s, ver) >> 8) - __mul64hi(c, sn) + 8) >> 4);
}
// No table in shared memory: for one value per thread, two reads of the quarter
// wave cost less than the table's set-up.
__device__ __forceinline__ void cis_fine(uint64_t theta, int64_t *cosine, int64_t *sine) {
    const int a = static_cast<int>(theta >> 56);
    cis_from(theta, quarter_cos(a), quarter_cos(a - 64), cosine, sine);
}

// An FP64 factor for rn_product: the mantissa left-aligned in 64 bits, and the
// sign and exponent field of the high word.  Zero becomes 2^-450, whose products
// with factors of exponents within 200 are too small to matter to a phase.
struct Factor {
    uint32_t m1, m0, e;
    // the number itself (not of a zero)
    __device__ __forceinline__ double value() const {
        return __hiloint2double(static_cast<int>(e | ((m1 << 1) >> 12)),
                                static_cast<int>(__funnelshift_r(m0, m1, 11)));
    }
};
// exponents that rn_product takes
__device__ __forceinline__ bool factor_in_range(double x) {
    const int e = static_cast<int>((static_cast<uint32_t>(__double2hiint(x)) >> 20) & 0x7ffu) - 1023;
    return x == 0.0 || (e >= -200 && e <= 200);
}
__device__ __forceinline__ Factor factor_of(double x) {
    const uint32_t hi = static_cast<uint32_t>(__double2hiint(x)), lo = static_cast<uint32_t>(__double2loint(x));
    if (x == 0.0) return Factor{0x80000000u, 0u, static_cast<uint32_t>(1023 - 450) << 20};
    return Factor{__funnelshift_l(lo, hi, 11) | 0x80000000u, lo << 11, hi & 0xfff00000u};
}

// x y rounded to nearest even, as the FP64 multiplier gives it, on the integer
// pipes: the 128-bit product of the mantissas, one bit of normalisation, the
// rounding added below the packed word, whose carry runs into the exponent.
// 4 wide multiplies and about 24 other instructions take the place of an FP64
// instruction, which holds its pipe four times as long as these hold theirs
// (77 clocks a warp against 50).
__device__ __forceinline__ double rn_product(const Factor &x, const Factor &y) {
    const uint64_t t = static_cast<uint64_t>(x.m0) * y.m0;
    const uint64_t u = static_cast<uint64_t>(x.m1) * y.m0 + (t >> 32);
    const uint64_t v = static_cast<uint64_t>(x.m0) * y.m1 + static_cast<uint32_t>(u);
    const uint64_t w = static_cast<uint64_t>(x.m1) * y.m1 + (u >> 32) + (v >> 32);
    const uint32_t h = static_cast<uint32_t>(w >> 32), l = static_cast<uint32_t>(w), m = static_cast<uint32_t>(v);
    const uint32_t up = (h >> 31) ^ 1u;                      // the product is below 2
    const uint32_t h2 = __funnelshift_l(l, h, up), l2 = __funnelshift_l(m, l, up);
    const uint32_t rest = min((m << up) | static_cast<uint32_t>(t), 1u);
    const uint32_t below = (l2 & 0x7ffu) | rest;             // what the mantissa leaves, sticky bit last
    const uint32_t lo = __funnelshift_r(l2, h2, 11);
    const uint32_t inc = (below + 0x3ffu + (lo & 1u)) >> 11;
    // sign and exponent fields add (mod 2^32); the mantissa's leading bit adds one
    const uint32_t e = x.e + y.e - (static_cast<uint32_t>(1023) << 20) - (up << 20);
    const uint64_t r = ((static_cast<uint64_t>(h2 >> 11) + e) << 32 | lo) + inc;
    return __longlong_as_double(static_cast<long long>(r));
}

// x = f 2^e with |f| in [1/2, 1) for finite x != 0, as frexp gives e (from the
// exponent field where x is normal; frexp is a long call)
__device__ __forceinline__ int exponent_of(double x) {
    const int field = static_cast<int>((static_cast<uint32_t>(__double2hiint(x)) >> 20) & 0x7ffu);
    if (field != 0) return field - 1022;
    int e;
    frexp(x, &e);
    return e;
}
// x 2^n as ldexp(x, n) gives it: a product with the power of two where that is a
// normal double
__device__ __forceinline__ double scale_pow2(double x, int n) {
    if (n >= -1022 && n <= 1023) return x * __hiloint2double((n + 1023) << 20, 0);
    return ldexp(x, n);
}

// Finite z1, z2 as z1 + i z2 = amp 2^ez e^{i beta} (amp in [1/2, sqrt 2), or
// 0): a first angle in FP32, its cosine and sine in 64 bits, then the remaining
// rotation d (1e-7 rad) from the cross product.  An FP64 atan2 and hypot would
// be a longer chain, and less exact.
__device__ __forceinline__ void mode_angle(double z1, double z2, double *amp,
                                           int *ez, uint64_t *beta) {
    *amp = 0.0;
    *ez = 0;
    *beta = 0;
    const double zm = fmax(fabs(z1), fabs(z2));
    if (zm == 0.0) return;
    *ez = exponent_of(zm);
    const int64_t f1 = __double2ll_rn(scale_pow2(z1, 62 - *ez)), f2 = __double2ll_rn(scale_pow2(z2, 62 - *ez));
    const float t = atan2f(static_cast<float>(f2), static_cast<float>(f1)) * 0.15915494f;   // turns
    const uint64_t b = static_cast<uint64_t>(__float2ll_rn(t * 1099511627776.0f)) << 24;
    int64_t c, s;
    cis_fine(b + kFineOffset, &c, &s);
    const double along = static_cast<double>(__mul64hi(f1, c) + __mul64hi(f2, s));    // units 2^-60
    const double across = static_cast<double>(__mul64hi(f2, c) - __mul64hi(f1, s));
    // across / along to 2^-45 of it: an FP32 reciprocal and one Newton step
    const double r0 = static_cast<double>(__frcp_rn(static_cast<float>(along)));
    const double d = across * fma(fma(-along, r0, 1.0), r0, r0);
    *amp = fma(along, 0.5 * d * d, along) * 0x1p-60;
    *beta = b + static_cast<uint64_t>(__double2ll_rn(d * 2.935890503282001e18));      // 2^64 / 2 pi
}

}  // namespace gsc
