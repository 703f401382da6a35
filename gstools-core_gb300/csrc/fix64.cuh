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
//   cos_fixed(theta)   the cosine of a turn fraction in units of 2^-62: one
//                      of 256 table entries and polynomials in the remainder.
//                      Over all phases the error is 1.2e-16 RMS, 4.2e-16 at
//                      most (an FP64 evaluation of the same degree, rounded
//                      at each step, has 7e-16 RMS).
//
// tests/test_fix64_cpu.py restates both in exact integers against 200-bit
// cosines, from the constants below.
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

}  // namespace gsc
