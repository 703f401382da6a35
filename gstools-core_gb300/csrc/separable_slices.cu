// separable_slices.cu -- the separable structured-grid contraction to FP64
// accuracy on the tcgen05 tensor cores (form GSC_FORM_SEP_F64), sm_103a.
//
// Same factorisation as separable_f64.cu (for each X_a one real GEMM with
// K = 2 modes: rows F[b, (2j, 2j+1)] = (Re, Im)(s_a[j] B[b, j]), columns
// G[c, (2j, 2j+1)] = (Re, -Im)(p_c C[c, j]); reference src/field.rs:37-65,
// :97-182 on the expanded grid).  GB300's FP64 MMA gives 1.1 TFLOP/s, its
// bf16 MMA 1,950, so F and G are held as 53-bit integers cut into six signed
// digits of 9 bits (Ozaki, Ogita, Oishi, Rump: error-free transformations of
// matrix products), each an exact bf16, and the 26 digit products whose
// weights are at least 2^-70 are summed on the tensor cores:
//
//   F = sum_i f_i 2^-(8 + 9 i),  G = sum_j g_j 2^-(8 + 9 j),  |f_i|, |g_j| <= 256
//   level l = i + j <= 6: all products have the unit 2^-(16 + 9 l)
//
//  * levels 0 to 3 each have a TMEM accumulator.  Its partial sums are
//    integers of its unit, and an FP32 accumulator adds integers exactly below
//    2^24, whatever the hardware's rounding.  The workers drain each
//    accumulator before any inputs could take it there: a k-block of 16 modes
//    adds at most 1.06, 2.98, 5.08 and 7.17 million units to level 0, 1, 2
//    and 3 (|F| and |G| of a mode are at most 1, the lower digits at most 256
//    each), so 12, 4, 3 and 2 k-blocks stay below 2^24 = 16.8 million.
//    Exactness needs no property of the inputs and no check;
//  * levels 4 to 6 share one accumulator, drained every 2 k-blocks: its
//    truncation is 2^-24 of sums that are 2^-36 of the field's;
//  * the drained sums are added in 64-bit integers of 2^-50 (finer for fewer
//    modes), which become FP64 at the end: one rounding.
// What is left is the representation (F and G to 2^-54), 1.3e-16 of the field,
// and the shared accumulator's truncation, 1.7e-16; the FP64 MMA's rounding
// grows with the modes, from 4e-16 (64 modes) to 2.2e-15 (2000).
//
// Small modes keep their precision: a mode's amplitude A_j and its column
// factor share its distance from the largest amplitude (s is scaled up and G
// down by 2^a_j, a_j half the exponents between them), and the columns of a
// vector component are scaled by its largest projector weight.  A_j is about what
// the mode adds to the field: without z2 where k = 0 (its sine is 0), and for a
// vector field with the exponent of its projector weights in it where all are
// weak, so that a mode along the first axis, which adds nothing, does not set the
// scale.
//
// Tables: phases k x in FP64 (as separable_f64.cu forms them), their cosines
// and sines in 64-bit fixed point (fix64.cuh), the products s B in 64-bit
// integers.  F's digits do not fit an SM's issue rate beside the drains, so a
// kernel of its own writes them in the layout the MMA reads (12 bytes per real
// element), for slabs of rows that bound the memory.
//
// Inputs that are not finite, phases of 2^32 and more and amplitudes beyond
// 2^+-900 set a word that stops the launches that follow; the FP64 MMA kernels
// queued behind run only then.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "fix64.cuh"
#include "internal.h"
#include "launch.cuh"
#include "sm100.cuh"

namespace gsc {
namespace {

using namespace sm100;

constexpr int kTileRows = 128;             // rows of F per tile
constexpr int kKbModes = 16;               // modes per k-block (K = 32)
constexpr int kSlices = 6;                 // digits per element
constexpr int kSliceF = kTileRows * 64;    // bytes of one slice of a k-block's F rows
constexpr int kSegModes = 4096;            // modes per integer total: |sum| <= 2^12, 2^62 units of 2^-50
constexpr int kFinest = 5;                 // bits of unit that fewer modes leave: down to 2^-55
constexpr int kAccs = 5;                   // levels 0-3 and the tail (4 to 6)
constexpr int kTail = 4;
constexpr int kAccCols = 96;               // TMEM columns between accumulators
constexpr int kTmem = 512;
constexpr int kThreads = 320;              // 8 worker warps, a copy warp, an MMA warp
constexpr int kCopyWarp = 8, kMmaWarp = 9;
constexpr float kPhaseLimit = 4.29e9f;     // turn_fraction's range, just below 2^32
// k-blocks between drains of each accumulator (see above)
__host__ __device__ constexpr int drain_period(int a) { return a == 0 ? 12 : a == 1 ? 4 : a == 2 ? 3 : 2; }

// Words the kernels share (zeroed before): [0] inputs outside this form,
// [1] 4000 + the largest amplitude's exponent, [2..4] 4000 + that of each
// component's projector weights (0 where all are zero).
constexpr int kWords = 8, kWordBias = 4000;

struct SlMode {
    double amp;        // A 2^-ez
    uint64_t beta;     // z1 - i z2 = A e^{-i beta}
    double w[3];       // projector weights (src/field.rs:138-152), over the power of two in A
    int32_t ez, ea;    // A <= 2^ea
};

struct SlTab {
    const double *cov, *z1, *z2;
    int dim, n_modes;              // n_modes: row length of cov
    int j0, nj, kb;                // this segment: modes [j0, j0 + nj), kb k-blocks
    const double *ax_b, *ax_m, *ax_n;
    int nb, nm, nn, ncomp, incompr;
    int nt, n_tiles;               // columns per tile
    SlMode *modes;
    longlong2 *svec;               // [nb or 1][16 kb]  s, units 2^-62
    longlong2 *btab;               // [nm][16 kb]       B, units 2^-62
    unsigned char *g;              // [tile][k-block][slice] images of nt rows x 64 bytes
    unsigned char *f;              // [row tile of the slab][k-block][slice] images of 128 rows x 64 bytes
    int64_t row0, rows_total;         // the slab's first row; rows of the output
    int *words;
};

// the least e with |x| <= 2^e, x != 0
__device__ __forceinline__ int ceil_exponent(double x) {
    const int e = exponent_of(x);
    return e - (fabs(x) == scale_pow2(0.5, e) ? 1 : 0);
}

// A mode whose projector weights are all weak (wmax the largest, 0: it adds nothing):
// their exponent goes into A.  Weights from kWeakWeight on stay: A is then at most
// 2^6 of what the mode adds.
constexpr double kWeakWeight = 0x1p-6;
__device__ __noinline__ void weak_mode(SlMode &m, double wmax) {
    if (wmax == 0.0) {
        m.amp = 0.0;
        m.ea = -kWordBias;
        return;
    }
    const int e = max(ceil_exponent(wmax), -200);
    m.ez += e;
    m.ea += e;
    for (int c = 0; c < 3; ++c) m.w[c] = scale_pow2(m.w[c], -e);
}

// z1 + i z2 of every mode as amplitude and angle, projector weights and the
// exponents of the largest.
__global__ void __launch_bounds__(128) sl_modes_kernel(SlTab t) {
    after_previous();
    const int j = blockIdx.x * 128 + threadIdx.x;
    const bool live = j < t.n_modes;
    int top[4] = {0, 0, 0, 0};
    bool bad = false;
    if (live) {
        SlMode m;
        const double z1 = t.z1[j], z2 = t.z2[j];
        double k[3] = {0.0, 0.0, 0.0};
        for (int d = 0; d < t.dim; ++d) k[d] = t.cov[static_cast<int64_t>(d) * t.n_modes + j];
        m.w[0] = m.w[1] = m.w[2] = 1.0;
        if (t.incompr) {   // projector as the reference forms it (src/field.rs:138-152)
            double kk = 0.0;
            for (int d = 0; d < t.dim; ++d) kk = __dadd_rn(kk, __dmul_rn(k[d], k[d]));
            const double k_2 = __ddiv_rn(k[0], kk);
            m.w[0] = __dadd_rn(1.0, -__dmul_rn(k[0], k_2));
            m.w[1] = -__dmul_rn(k[1], k_2);
            m.w[2] = -__dmul_rn(k[2], k_2);
        }
        bad = !(isfinite(z1) && isfinite(z2) && isfinite(k[0]) && isfinite(k[1]) && isfinite(k[2]) &&
                isfinite(m.w[0]) && isfinite(m.w[1]) && isfinite(m.w[2]));
        m.ez = 0;
        m.ea = -kWordBias;
        m.amp = 0.0;
        m.beta = 0;
        const double wmax = t.incompr ? fmax(fabs(m.w[0]), fmax(fabs(m.w[1]), t.dim == 3 ? fabs(m.w[2]) : 0.0)) : 1.0;
        const bool still = k[0] == 0.0 && k[1] == 0.0 && k[2] == 0.0;
        if (!bad) {
            mode_angle(z1, still ? 0.0 : z2, &m.amp, &m.ez, &m.beta);
            if (m.amp > 0.0) {
                m.ea = m.ez + ceil_exponent(m.amp);            // A <= 2^ea
                bad = m.ea < -900 || m.ea > 900;
            }
            if (wmax < kWeakWeight) weak_mode(m, wmax);
            if (m.amp > 0.0) top[0] = m.ea + kWordBias;
            for (int c = 0; c < t.ncomp; ++c)
                if (m.w[c] != 0.0) top[1 + c] = ceil_exponent(m.w[c]) + kWordBias;   // |w| <= 2^e
        }
        t.modes[j] = m;
    }
    if (bad) t.words[0] = 1;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int v = __reduce_max_sync(0xffffffffu, top[c]);
        if ((threadIdx.x & 31) == 0 && v > 0) atomicMax(t.words + 1 + c, v);
    }
}

__device__ __forceinline__ int top_exponent(int word) { return word > 0 ? word - kWordBias : 0; }

// half the exponents between this amplitude and the largest
__device__ __forceinline__ int mode_shift(const SlMode &m, int ew) { return m.amp > 0.0 ? (ew - m.ea) >> 1 : 0; }

// The six digits of a (re, im) pair in units of 2^-60, |re|, |im| <= 1, as
// packed bf16 pairs.  Offsets make every digit a plain bit field; a field under
// the exponent of 2^23 is its value as a float, one multiply-add takes the
// offset out and scales it, and the upper halves of two floats are the pair.
__device__ __forceinline__ void digits6(int64_t re, int64_t im, uint32_t (&w)[kSlices]) {
    // 256 in each digit (units 2^52, 2^43, 2^34, 2^25, 2^16, 2^7) and half a unit of the last
    constexpr int64_t off = (int64_t(256) << 52) + (int64_t(256) << 43) + (int64_t(256) << 34) + (int64_t(256) << 25) +
                            (int64_t(256) << 16) + (int64_t(256) << 7) + 64;
    const uint64_t a = static_cast<uint64_t>(re + off), b = static_cast<uint64_t>(im + off);
    const uint32_t ah = static_cast<uint32_t>(a >> 32), al = static_cast<uint32_t>(a);
    const uint32_t bh = static_cast<uint32_t>(b >> 32), bl = static_cast<uint32_t>(b);
    auto lift = [](uint32_t field, float unit) {
        return fmaf(__uint_as_float(0x4B000000u | field), unit, -8388864.0f * unit);   // (field - 256) unit
    };
    auto pack = [](float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); };
    w[0] = pack(lift(ah >> 20, 0x1p-8f), lift(bh >> 20, 0x1p-8f));
    w[1] = pack(lift((ah >> 11) & 511u, 0x1p-17f), lift((bh >> 11) & 511u, 0x1p-17f));
    w[2] = pack(lift((ah >> 2) & 511u, 0x1p-26f), lift((bh >> 2) & 511u, 0x1p-26f));
    w[3] = pack(lift(__funnelshift_r(al, ah, 25) & 511u, 0x1p-35f),
                lift(__funnelshift_r(bl, bh, 25) & 511u, 0x1p-35f));
    w[4] = pack(lift((al >> 16) & 511u, 0x1p-44f), lift((bl >> 16) & 511u, 0x1p-44f));
    w[5] = pack(lift((al >> 7) & 511u, 0x1p-53f), lift((bl >> 7) & 511u, 0x1p-53f));
}

// Byte offset of the 16-byte chunk c (modes 4c .. 4c+3) of row r in a slice
// image: 64-byte rows, 64-byte swizzle.
__device__ __forceinline__ uint32_t chunk_offset(int r, int c) {
    return static_cast<uint32_t>(r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
}

// Factor tables of a segment: G images (a thread per column row and chunk of
// four modes), then B and s (a thread per entry).
constexpr int kTabThreads = 256;
__global__ void __launch_bounds__(kTabThreads)
sl_tables_kernel(SlTab t, int64_t n_g, int64_t n_b, int64_t n_s) {
    after_previous();
    const int np = t.kb * kKbModes;
    const int ew = top_exponent(t.words[1]);
    bool bad = false;
    auto fraction = [&](int d, int j, double x) -> uint64_t {
        const double ph = __dmul_rn(t.cov[static_cast<int64_t>(d) * t.n_modes + j], x);
        bad = bad || !(fabs(ph) < static_cast<double>(kPhaseLimit));
        return turn_fraction(ph);
    };
    int64_t i = static_cast<int64_t>(blockIdx.x) * kTabThreads + threadIdx.x;
    const int64_t b_g = (n_g + kTabThreads - 1) / kTabThreads * kTabThreads;
    const int64_t b_b = (n_b + kTabThreads - 1) / kTabThreads * kTabThreads;
    if (i < b_g) {
        if (i < n_g) {
            const int c = static_cast<int>(i & 3);
            const int r = static_cast<int>((i >> 2) % t.nt);
            const int64_t blk = (i >> 2) / t.nt;                    // tile * kb + k-block
            const int kb = static_cast<int>(blk % t.kb), tile = static_cast<int>(blk / t.kb);
            const int col = tile * t.nt + r;
            const int comp = col / t.nn, n = col - comp * t.nn;
            uint32_t w[4][kSlices];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int jl = kb * kKbModes + 4 * c + u, j = t.j0 + jl;
                int64_t re = 0, im = 0;
                if (comp < t.ncomp && jl < t.nj) {
                    const SlMode &m = t.modes[j];
                    int64_t co, si;
                    cis_fine(fraction(t.dim - 1, j, t.ax_n[n]) + kFineOffset, &co, &si);
                    const int g = t.incompr ? top_exponent(t.words[2 + comp]) : 0;
                    const int64_t wf = __double2ll_rn(scale_pow2(m.w[comp], 62 - g - mode_shift(m, ew)));
                    re = __mul64hi(wf, co);
                    im = -__mul64hi(wf, si);
                }
                digits6(re, im, w[u]);
            }
            unsigned char *dst = t.g + blk * kSlices * (t.nt * 64) + chunk_offset(r, c);
#pragma unroll
            for (int s = 0; s < kSlices; ++s)
                *reinterpret_cast<uint4 *>(dst + static_cast<int64_t>(s) * (t.nt * 64)) =
                    make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]);
        }
    } else if (i < b_g + b_b) {
        i -= b_g;
        if (i < n_b) {
            const int jl = static_cast<int>(i % np), m = static_cast<int>(i / np);
            longlong2 v = make_longlong2(0, 0);
            if (jl < t.nj) {
                int64_t co, si;
                cis_fine(fraction(t.dim - 2, t.j0 + jl, t.ax_m[m]) + kFineOffset, &co, &si);
                v = make_longlong2(co, si);
            }
            t.btab[i] = v;
        }
    } else {
        i -= b_g + b_b;
        if (i < n_s) {
            const int jl = static_cast<int>(i % np), b = static_cast<int>(i / np);
            longlong2 v = make_longlong2(0, 0);
            if (jl < t.nj) {
                const int j = t.j0 + jl;
                const SlMode &m = t.modes[j];
                uint64_t th = kFineOffset - m.beta;
                if (t.dim == 3) th += fraction(0, j, t.ax_b[b]);
                int64_t co, si;
                cis_fine(th, &co, &si);
                const int64_t a = __double2ll_rn(scale_pow2(m.amp, m.ez - ew + mode_shift(m, ew) + 62));
                v = make_longlong2(__mul64hi(a, co) << 2, __mul64hi(a, si) << 2);
            }
            t.svec[i] = v;
        }
    }
    // set once or a few times: a store by every warp of a table whose phases are all too
    // large takes longer than the table (5000 x 1 points x 200 modes: 750 us a call,
    // 630 so)
    if (bad && *static_cast<volatile int *>(t.words) == 0) t.words[0] = 1;
}

// a b + c d of values in units of 2^-62 (|.| <= 1), in units of 2^-60; the
// low halves one bit short, their products' truncation made up on average
struct Word2 {
    int32_t h, l;
};
__device__ __forceinline__ Word2 word2(int64_t v) {
    return Word2{static_cast<int32_t>(v >> 32), static_cast<int32_t>(static_cast<uint32_t>(v) >> 1)};
}
__device__ __forceinline__ int64_t dot_fixed(Word2 a, Word2 b, Word2 c, Word2 d) {
    int64_t p = static_cast<int64_t>(a.h) * b.h + 4;
    p += static_cast<int64_t>(c.h) * d.h;
    const int32_t low = __mulhi(a.h, b.l) + __mulhi(a.l, b.h) + __mulhi(c.h, d.l) + __mulhi(c.l, d.h);
    return p + (static_cast<int64_t>(low) << 1);
}

// F digits of a slab: grid (2 * row tiles, k-blocks), a thread per row and
// chunk of four modes.  Bound by the integer pipes (about 550 instructions a
// thread) and by its stores, 12 bytes per real element.  Five blocks per SM
// (48 registers): with fewer registers it spills, with more it hides less (24,000
// rows x 1000 modes: 157 us unbounded, 135 at 5 blocks, 172 at 6; two rows per
// thread, which share s, 139).
constexpr int kSliceThreads = 256;
__global__ void __launch_bounds__(kSliceThreads, 5) sl_slice_kernel(SlTab t) {
    after_previous();
    if (t.words[0]) return;
    const int c = threadIdx.x & 3, r = (blockIdx.x & 1) * 64 + (threadIdx.x >> 2);
    const int kb = blockIdx.y;
    const int64_t tile = blockIdx.x >> 1;
    const int64_t row = t.row0 + tile * kTileRows + r;
    const int np = t.kb * kKbModes, j = kb * kKbModes + 4 * c;
    uint32_t w[4][kSlices];
    if (row < t.rows_total) {
        const int b = static_cast<int>(row / t.nm), m = static_cast<int>(row - static_cast<int64_t>(b) * t.nm);
        const longlong2 *sp = t.svec + static_cast<int64_t>(b) * np + j;
        const longlong2 *bp = t.btab + static_cast<int64_t>(m) * np + j;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const longlong2 s = sp[u], e = bp[u];
            const Word2 sx = word2(s.x), sy = word2(s.y), ny = word2(-s.y), bx = word2(e.x), by = word2(e.y);
            digits6(dot_fixed(sx, bx, ny, by), dot_fixed(sx, by, sy, bx), w[u]);
        }
    } else {
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int s = 0; s < kSlices; ++s) w[u][s] = 0u;
    }
    unsigned char *dst = t.f + (tile * t.kb + kb) * (kSlices * kSliceF) + chunk_offset(r, c);
#pragma unroll
    for (int s = 0; s < kSlices; ++s)
        *reinterpret_cast<uint4 *>(dst + s * kSliceF) = make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]);
}

struct SlGemm {
    const unsigned char *f, *g;
    int kb, n_tiles;               // k-blocks of the segment, column tiles
    int splits;                    // units per tile, each a share of the k-blocks
    int64_t units;
    int64_t row0, rows_total, P;   // slab's first row; rows of the output; points per component
    int nn, ncn;                   // columns per component, columns
    double *out;                   // (ncomp, rows, nn), whole tiles
    int64_t *part;                 // splits: the integer totals, split s at part + s * split_stride
    int64_t split_stride;
    int accumulate;                // add to the output (later segments)
    int finer;                     // integer totals in units of 2^-(50 + finer)
    const int *words;
    int *status;
};

// Shared memory: a ring of slots, one slice of F and of G each (the six slices
// of a k-block in order).  14 slots of 14 KB hold 2.3 k-blocks of 96 columns.
template <int NT>
struct SlLayout {
    static constexpr int G_BYTES = NT * 64;
    static constexpr int SLOT = kSliceF + G_BYTES;
    static constexpr int EPI_BYTES = 8 * 32 * 9 * 8;    // a worker warp's 32 rows x 8 columns, padded
    static constexpr int ROOM = 232448 - 1024 - 512 - EPI_BYTES;
    static constexpr int SLOTS = ROOM / SLOT < 24 ? ROOM / SLOT : 24;
    static constexpr int DATA = SLOTS * SLOT;           // the ring, then the epilogue's rows, then barriers
    static constexpr size_t SMEM = DATA + EPI_BYTES + 512 + 1024;
    static constexpr int HC = NT / 2;      // columns per worker half
    static_assert(SLOT % 1024 == 0, "slots keep the swizzle's alignment");
    // with at most 24 slots, k-block i + 4 is not copied before k-block i has been
    // multiplied, so four barriers tell the k-blocks in flight apart
    static_assert(SLOTS >= 12 && SLOTS <= 24, "two k-blocks at least, four at most");
    static_assert((8 + 2 * kAccs + 1) * 8 + 16 <= 512, "barriers");
    static_assert(NT % 16 == 0 && NT <= kAccCols && HC % 8 == 0, "tile width");
};

// What a unit of each accumulator counts in a 64-bit total of units 2^-(50 + finer).
struct Units {
    int32_t one, two, three;   // levels 1-3: 2^(25 + finer), 2^(16 + finer), 2^(7 + finer)
    int32_t zero;              // level 0: 2^(2 + finer) in the upper word
    float tail;                // 2^(50 + finer)
};

// a drained sum of accumulator A into the total
template <int A>
__device__ __forceinline__ void add_level(int64_t &acc, uint32_t bits, const Units &u) {
    const float v = __uint_as_float(bits);
    if constexpr (A == kTail) {
        acc += __float2int_rn(v * u.tail);
    } else {
        const int n = __float2int_rn(v * (A == 0 ? 0x1p16f : A == 1 ? 0x1p25f : A == 2 ? 0x1p34f : 0x1p43f));
        if constexpr (A == 0)
            acc += static_cast<int64_t>(static_cast<uint64_t>(static_cast<uint32_t>(n * u.zero)) << 32);
        else
            acc += static_cast<int64_t>(n) * (A == 1 ? u.one : A == 2 ? u.two : u.three);
    }
}

// columns [0, HC) of this warp's quarter and half of accumulator A, which
// starts at `taddr`
template <int A, int HC>
__device__ __forceinline__ void drain_acc(int64_t (&acc)[HC], uint32_t taddr, const Units &u) {
    constexpr int full = HC / 16 * 16;
#pragma unroll
    for (int c = 0; c < full; c += 16) {
        uint32_t v[16];
        tmem_ld16(taddr + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) add_level<A>(acc[c + i], v[i], u);
    }
    if constexpr (full < HC) {
        uint32_t v[8];
        tmem_ld8(taddr + full, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) add_level<A>(acc[full + i], v[i], u);
    }
}

__device__ __noinline__ double scaled_total_small(int64_t t, int e) { return ldexp(static_cast<double>(t), e); }

// t 2^e for an integer total, rounded to nearest even, by integer instructions (a
// conversion is an FP64 instruction: 16 clocks of an SM for a warp's).  The
// subnormal results' path is a call, so that it is not run in advance.
__device__ __forceinline__ double scaled_total(int64_t t, int e) {
    if (t == 0) return 0.0;
    const uint64_t mag = static_cast<uint64_t>(t < 0 ? -t : t);
    const int lz = __clzll(static_cast<long long>(mag));
    const uint64_t m = mag << lz;                    // leading bit at 63
    const int x = 63 - lz + e;                       // the value is 1.m 2^x
    if (x < -1020) return scaled_total_small(t, e);
    const uint64_t inc = ((m & 0x7ffu) + 0x3ffu + ((m >> 11) & 1u)) >> 11;
    // the leading bit adds one to the exponent field
    const uint64_t bits = (m >> 11) + inc + (static_cast<uint64_t>(x + 1022) << 52);
    return __longlong_as_double(static_cast<long long>(bits | (t < 0 ? uint64_t(1) << 63 : 0)));
}

// Tiles of 128 rows x NT columns.  One CTA per SM walks units (a tile, or one
// split of its k-blocks); the copies and MMAs of a unit follow those of the one
// before at once, while the workers still write that one out: its sums are in
// their registers.
//
// Per k-block 52 MMAs of 128 x NT x 16 beside 1.7 drained accumulators.  The
// products run in three groups, levels 0 to 2, level 3, tail, so that an
// accumulator that was just drained is needed again one group later at the
// earliest, and within a group by F slice, which the collector buffer keeps for
// its products (an MMA of 96 columns takes 56 clocks when it reads both operands
// and 48 when it keeps A; 52 and 41 for 80).
template <int NT>
__global__ void __launch_bounds__(kThreads, 1) sl_gemm_kernel(const SlGemm p) {
    using L = SlLayout<NT>;
    after_previous();
    if (p.words[0]) return;          // the same for every CTA
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::DATA + L::EPI_BYTES);   // [4] copies -> MMA
    uint64_t *kdone = full + 4;                  // [4] MMA commit of a k-block -> copies
    uint64_t *acc_full = kdone + 4;              // [5] MMA commit -> workers
    uint64_t *acc_empty = acc_full + kAccs;      // [5] workers -> MMA (8 arrivals)
    uint64_t *drain = acc_empty + kAccs;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // a unit's tile and k-blocks
    struct Unit {
        int nt, part, kbeg, kb;
        int64_t mt;
    };
    auto unit_at = [&](int64_t u) -> Unit {
        Unit x;
        x.part = static_cast<int>(u % p.splits);
        const int64_t tile = u / p.splits;
        x.nt = static_cast<int>(tile % p.n_tiles);
        x.mt = tile / p.n_tiles;
        x.kbeg = static_cast<int>(static_cast<int64_t>(x.part) * p.kb / p.splits);
        x.kb = static_cast<int>(static_cast<int64_t>(x.part + 1) * p.kb / p.splits) - x.kbeg;
        return x;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < 4; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&kdone[s], 1);
        }
        for (int a = 0; a < kAccs; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 8);
        }
        mbar_init(drain, 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tmem_alloc(tmem_slot, kTmem);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // k-blocks are counted through all units of the CTA: k-block `it` uses
    // barriers it % 4 and the ring slots from 6 it on
    if (warp == kCopyWarp) {
        if (elect_one()) {
            bool ok = true;
            int it = 0, slot = 0;
            for (int64_t u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
                const Unit x = unit_at(u);
                const unsigned char *fb = p.f + (x.mt * p.kb + x.kbeg) * (kSlices * kSliceF);
                const unsigned char *gb =
                    p.g + (static_cast<int64_t>(x.nt) * p.kb + x.kbeg) * (kSlices * L::G_BYTES);
                for (int i = 0; i < x.kb && ok; ++i, ++it) {
                    for (int s = 0; s < kSlices; ++s) {
                        const int q = it * kSlices + s - L::SLOTS;
                        if (q >= 0) {          // the k-block that last used the slot has been multiplied
                            const int k = q / kSlices;
                            ok = mbar_wait(&kdone[k & 3], (k >> 2) & 1, abort_flag, p.status, kErrTimeoutEmpty);
                            if (!ok) break;
                        }
                        if (s == 0) mbar_arrive_expect_tx(&full[it & 3], kSlices * L::SLOT);
                        unsigned char *dst = smem + slot * L::SLOT;
                        bulk_copy_g2s(dst, fb, kSliceF, &full[it & 3]);
                        bulk_copy_g2s(dst + kSliceF, gb, L::G_BYTES, &full[it & 3]);
                        fb += kSliceF;
                        gb += L::G_BYTES;
                        slot = slot + 1 == L::SLOTS ? 0 : slot + 1;
                    }
                }
            }
            // on abort the copies in flight land before the block ends; a k-block
            // that was cut short never completes its barrier, and that wait runs out
            if (*abort_flag)
                for (int i = it > 3 ? it - 3 : 0; i < it; ++i)
                    mbar_wait_drain(&full[i & 3], (i >> 2) & 1, p.status);
        }
    } else if (warp == kMmaWarp) {
        if (elect_one()) {
            // Little time may pass between two MMAs: the unit holds only a few
            // that were issued ahead.  So what a k-block needs is prepared between
            // the MMAs of the one before, a piece at a time, and accumulators are
            // waited for one by one, each right before its first product.
            constexpr uint32_t idesc = idesc_f16(kTileRows, NT, true);
            bool ok = true;
            int it = 0, slot = 0;
            uint32_t phase[kAccs] = {0, 0, 0, 0, 0};   // drains handed to the workers so far
            int left[kAccs];                           // k-blocks until the next drain
            uint32_t keep[kAccs];                      // 0: the accumulator starts again from zero
            uint64_t fd[kSlices], gd[kSlices], nf[kSlices], ng[kSlices];
            auto next_slot = [&](int s) {
                const uint32_t at = smem_u32(smem + slot * L::SLOT);
                nf[s] = desc_k_sw64(at);
                ng[s] = desc_k_sw64(at + kSliceF);
                slot = slot + 1 == L::SLOTS ? 0 : slot + 1;
            };
#pragma unroll
            for (int s = 0; s < kSlices; ++s) next_slot(s);
            bool ready = false;                        // the k-block's copies have been waited for
            int64_t u = blockIdx.x;
            int KB = u < p.units ? unit_at(u).kb : 0, i = 0;
            while (KB > 0) {
                if (!ready) ok = mbar_wait(&full[it & 3], (it >> 2) & 1, abort_flag, p.status, kErrTimeoutFull);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int s = 0; s < kSlices; ++s) {
                    fd[s] = nf[s];
                    gd[s] = ng[s];
                }
                if (i == 0) {
#pragma unroll
                    for (int a = 0; a < kAccs; ++a) {
                        left[a] = drain_period(a);
                        keep[a] = 0;
                    }
                }
                const bool last = i == KB - 1;
                // before an accumulator's first product: it may start again once the
                // workers have read it
                auto open = [&](int a) {
                    if (!keep[a] && phase[a] > 0 && ok) {
                        ok = mbar_wait(&acc_empty[a], (phase[a] - 1) & 1, abort_flag, p.status, kErrTimeoutAcc);
                        tc_fence_after();
                    }
                };
                // after its last product: drained when its period or the unit ends
                auto close = [&](int a) {
                    keep[a] = 1;
                    if (--left[a] == 0 || last) {
                        mma_commit(&acc_full[a]);
                        ++phase[a];
                        left[a] = drain_period(a);
                        keep[a] = 0;
                    }
                };
                // products (x, y) of F slice x with lo <= x + y <= hi into accumulator
                // min(x + y, tail); (the K step of 16 adds 32 bytes to an address, 2 in a
                // descriptor)
                auto group = [&](auto lo_, auto hi_, auto &&between) {
                    constexpr int lo = decltype(lo_)::value, hi = decltype(hi_)::value;
                    int n = 0;                         // a constant at every use once unrolled
#pragma unroll
                    for (int x = 0; x < kSlices; ++x)
#pragma unroll
                        for (int kk = 0; kk < 2; ++kk) {
                            bool filled = false;
#pragma unroll
                            for (int y = 0; y < kSlices; ++y) {
                                const int l = x + y;
                                if (l < lo || l > hi) continue;
                                const int a = l < kTail ? l : kTail;
                                const bool opens = x == 0 && kk == 0 && y == a;
                                if (opens) open(a);
                                const uint32_t d = tmem + a * kAccCols, acc = opens ? keep[a] : 1u;
                                if (filled) mma_f16_ss_keep<true>(d, fd[x] + 2 * kk, gd[y] + 2 * kk, idesc, acc);
                                else mma_f16_ss_keep<false>(d, fd[x] + 2 * kk, gd[y] + 2 * kk, idesc, acc);
                                filled = true;
                                between(n);
                                ++n;
                            }
                        }
                };
                group(std::integral_constant<int, 0>{}, std::integral_constant<int, 2>{}, [&](int n) {
                    if (n == 9) close(0);              // products 0, 3 are level 0's, 1, 4, 6, 8 level 1's
                    if (n == 10) close(1);
                });
                close(2);
                group(std::integral_constant<int, 3>{}, std::integral_constant<int, 3>{}, [](int) {});
                close(3);
                ready = false;
                group(std::integral_constant<int, kTail>{}, std::integral_constant<int, 6>{}, [&](int n) {
#pragma unroll
                    for (int s = 0; s < kSlices; ++s)
                        if (n == 3 + 2 * s) next_slot(s);
                    if (n == 20 && !last)
                        ready = mbar_test_wait(&full[(it + 1) & 3], ((it + 1) >> 2) & 1);
                });
                close(kTail);
                mma_commit(&kdone[it & 3]);
                ++it;
                ++i;
                if (last) {
                    u += gridDim.x;
                    KB = u < p.units ? unit_at(u).kb : 0;
                    i = 0;
                }
                if (!ok) break;
            }
            if (!ok) {
                mma_commit(drain);
                mbar_wait_drain(drain, 0, p.status);
            }
        }
    } else {
        // ---- workers ---------------------------------------------------------
        const int q = warp & 3, h = warp >> 2;
        const uint32_t taddr = tmem + (static_cast<uint32_t>(32 * q) << 16) + L::HC * h;
        int64_t *tr = reinterpret_cast<int64_t *>(smem + L::DATA) + warp * (32 * 9);
        Units units;
        units.zero = 1 << (2 + p.finer);
        units.one = 1 << (25 + p.finer);
        units.two = 1 << (16 + p.finer);
        units.three = 1 << (7 + p.finer);
        units.tail = ldexpf(1.0f, 50 + p.finer);
        const int ew = top_exponent(p.words[1]);
        int drains[kAccs] = {0, 0, 0, 0, 0};
        bool ok = true;
        for (int64_t u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
            const Unit x = unit_at(u);
            int64_t acc[L::HC];
#pragma unroll
            for (int c = 0; c < L::HC; ++c) acc[c] = 0;
            // a drain is taken by the whole warp: the barrier counts once every lane has passed it
            auto take = [&](auto level, int i) {
                constexpr int A = decltype(level)::value;
                if (!ok || !((i + 1) % drain_period(A) == 0 || i == x.kb - 1)) return;
                const bool got = mbar_wait(&acc_full[A], drains[A] & 1, abort_flag, p.status, kErrTimeoutAcc);
                ++drains[A];
                ok = __all_sync(0xffffffffu, got);
                if (!ok) return;
                tc_fence_after();
                drain_acc<A>(acc, taddr + A * kAccCols, units);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[A]);
            };
            for (int i = 0; i < x.kb && ok; ++i) {
                take(std::integral_constant<int, 0>{}, i);
                take(std::integral_constant<int, 1>{}, i);
                take(std::integral_constant<int, 2>{}, i);
                take(std::integral_constant<int, 3>{}, i);
                take(std::integral_constant<int, kTail>{}, i);
            }
            if (!ok) break;
            // ---- the unit's output: 8 columns at a time are turned around in
            // shared memory, so that a quarter of a warp writes 64 consecutive
            // bytes.  Splits leave their integers: their sum is exact, and the
            // conversion (an FP64 instruction) waits for it
            const int64_t rq = p.row0 + x.mt * kTileRows + 32 * q;
            const int rows = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(32), p.rows_total - rq)));
            const int n0 = x.nt * NT + L::HC * h;
#pragma unroll
            for (int c0 = 0; c0 < L::HC; c0 += 8) {
#pragma unroll
                for (int c = 0; c < 8; ++c) tr[lane * 9 + c] = acc[c0 + c];
                __syncwarp();
                const int c = lane & 7, col = n0 + c0 + c;
                if (col < p.ncn) {
                    const int comp = col / p.nn;
                    const int64_t at = comp * p.P + (col - comp * p.nn);
                    if (p.part) {
                        int64_t *o = p.part + x.part * p.split_stride + at + rq * p.nn;
                        for (int r = lane >> 3; r < rows; r += 4) o[static_cast<int64_t>(r) * p.nn] = tr[r * 9 + c];
                    } else {
                        const int e = ew + top_exponent(p.words[2 + comp]) - 50 - p.finer;
                        double *o = p.out + at + rq * p.nn;
                        for (int r = lane >> 3; r < rows; r += 4) {
                            const double v = scaled_total(tr[r * 9 + c], e);
                            double *dst = o + static_cast<int64_t>(r) * p.nn;
                            *dst = p.accumulate ? *dst + v : v;
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kMmaWarp) tmem_dealloc(tmem, kTmem);
}

// out = the splits' integer totals, added and converted: exact within a segment
// of modes (segments of `splits` totals each, the last of `last`), one rounding
// and for later segments one addition each
__global__ void __launch_bounds__(256)
sl_reduce_kernel(const int64_t *__restrict__ part, int segs, int splits, int last, int64_t P, int ncomp,
                 int finer, double *__restrict__ out, const int *__restrict__ words) {
    after_previous();
    if (words[0]) return;
    const int64_t q = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x, n = ncomp * P;
    if (q >= P) return;
    const int64_t i = blockIdx.y * P + q;
    const int e = top_exponent(words[1]) + top_exponent(words[2 + blockIdx.y]) - 50 - finer;
    double s = 0.0;
    for (int g = 0; g < segs; ++g) {
        const int k1 = g == segs - 1 ? last : splits;
        int64_t t = 0;
#pragma unroll 4
        for (int k = 0; k < k1; ++k) t += part[(static_cast<int64_t>(g) * splits + k) * n + i];
        const double v = scaled_total(t, e);
        if (g == 0) s = v;
        else s += v;
    }
    out[i] = s;
}

template <int NT>
int launch_gemm(const SlGemm &p, int64_t grid, cudaStream_t st) {
    GSC_TRY(smem_attr(reinterpret_cast<const void *>(sl_gemm_kernel<NT>), SlLayout<NT>::SMEM));
    GSC_CUDA(launch_after(sl_gemm_kernel<NT>, dim3(static_cast<unsigned>(grid)), dim3(kThreads),
                          SlLayout<NT>::SMEM, st, p));
    return GSC_OK;
}

size_t up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// clocks of a k-block's 52 MMAs of 128 x nt x 16: nt / 2 for the multiplies, and
// 128 bytes of shared memory per clock for the operands: 32 nt, and 4 KB more
// for the 26 that read F
double kblock_clocks(int nt) {
    return 26.0 * std::max(nt * 0.5, (4096.0 + 32.0 * nt) / 128.0) + 26.0 * nt * 0.5;
}

}  // namespace

// The launch plan of a grid: column tile, slabs of row tiles, splits.
struct SlPlan {
    int nt, n_tiles, splits;
    int64_t m_tiles, slab;         // row tiles, row tiles per slab
    int segs, kb;                  // mode segments, k-blocks of the longest
};
static SlPlan sl_plan(int64_t rows, int ncn, int64_t n_modes, int64_t out_bytes, int sms) {
    SlPlan s{};
    double best = 1e300;
    for (int nt : {96, 80, 64, 48, 32}) {
        const int tiles = (ncn + nt - 1) / nt;
        const double c = tiles * kblock_clocks(nt);
        if (c < best) {
            best = c;
            s.nt = nt;
            s.n_tiles = tiles;
        }
    }
    s.m_tiles = (rows + kTileRows - 1) / kTileRows;
    s.segs = static_cast<int>((n_modes + kSegModes - 1) / kSegModes);
    const int64_t seg_modes = std::min<int64_t>(n_modes, kSegModes);
    s.kb = static_cast<int>((seg_modes + kKbModes - 1) / kKbModes);
    // slabs of whole waves of tiles, about 1 GB of F digits each or one wave (one
    // column tile and 4096 modes: 1.9 GB), or all rows where those fit.  Shorter
    // mode segments, which would keep a wave in 1 GB, cost 5 to 7 % (200 x 120 x 60
    // x 4096 modes 1352 -> 1416 us).  The library keeps the scratch, as any other,
    // until gsc_release_buffers
    const int64_t tile_bytes = static_cast<int64_t>(s.kb) * kSlices * kSliceF;
    s.slab = s.m_tiles;
    if (s.m_tiles * tile_bytes > (int64_t(1) << 30)) {
        const int64_t most = std::max<int64_t>((int64_t(1) << 30) / tile_bytes, (sms + s.n_tiles - 1) / s.n_tiles);
        s.slab = std::min(s.m_tiles, most);
        for (int64_t waves = s.slab * s.n_tiles / sms; waves >= 1; --waves) {
            const int64_t m = waves * sms / s.n_tiles;       // fills `waves` waves but for less than n_tiles
            if (m >= 1 && m <= most && waves * sms - m * s.n_tiles < s.n_tiles) {
                s.slab = std::min(s.m_tiles, m);
                break;
            }
        }
    }
    // splits of the k-blocks where one slab's tiles leave SMs idle: the time of
    // the busiest SM, a fixed cost per part, and the partial fields' traffic
    s.splits = 1;
    if (s.slab == s.m_tiles) {
        const double kb_clocks = kblock_clocks(s.nt);
        double least = 1e300;
        const int64_t tiles = s.m_tiles * s.n_tiles;
        for (int k = 1; k <= 64 && s.kb / k >= 2; ++k) {
            if (k > 1 && static_cast<int64_t>(k) * s.segs * out_bytes > (int64_t(1) << 30)) break;
            double c = std::ceil(static_cast<double>(tiles * k) / sms) * (std::ceil(static_cast<double>(s.kb) / k) * kb_clocks + 4000.0);
            if (k > 1) c += 4000.0 + (k + 1.0) * out_bytes / 2500.0;
            if (c < least) {
                least = c;
                s.splits = k;
            }
        }
    }
    return s;
}

int sep_slices_run(DeviceCtx &ctx, const SepArgs &a, cudaStream_t st) {
    const int dim = static_cast<int>(a.dim);
    const int N = static_cast<int>(a.n_modes);
    const int ncomp = a.incompr ? dim : 1;
    const int nb = dim == 3 ? static_cast<int>(a.n[0]) : 1;
    const int nm = static_cast<int>(dim == 3 ? a.n[1] : a.n[0]);
    const int nn = static_cast<int>(dim == 3 ? a.n[2] : a.n[1]);
    const int64_t rows = static_cast<int64_t>(nb) * nm, P = rows * nn;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device) != cudaSuccess || sms <= 0) {
        cudaGetLastError();
        sms = 152;
    }
    const size_t out_bytes = sizeof(double) * static_cast<size_t>(ncomp) * P;
    SlPlan pl = sl_plan(rows, ncomp * nn, N, static_cast<int64_t>(out_bytes), sms);
    const int np = pl.kb * kKbModes;

    // scratch: words, modes, s, B, G images, F images of a slab, split fields;
    // the fallback's tables use the same memory behind the words
    const size_t off_modes = 256;
    const size_t off_s = up(off_modes + sizeof(SlMode) * static_cast<size_t>(N), 256);
    const size_t off_b = up(off_s + sizeof(longlong2) * static_cast<size_t>(nb) * np, 256);
    const size_t off_g = up(off_b + sizeof(longlong2) * static_cast<size_t>(nm) * np, 1024);
    const size_t g_bytes = static_cast<size_t>(pl.n_tiles) * pl.kb * kSlices * pl.nt * 64;
    const size_t off_f = up(off_g + g_bytes, 1024);
    size_t off_part = 0;
    int parts = 0;
    for (;;) {
        off_part = up(off_f + static_cast<size_t>(pl.slab) * pl.kb * kSlices * kSliceF, 1024);
        parts = pl.splits > 1 ? pl.splits * pl.segs : 0;
        const int rc = ensure_dev(ctx, ctx.scratch, std::max(off_part + parts * out_bytes, 256 + sep_f64_scratch(a)));
        if (rc == GSC_OK) break;
        if (rc != GSC_ERR_NOMEM) return rc;
        // no room: the digits of fewer rows at a time, then no splits, at last
        // the FP64 MMA kernels, which need neither
        if (pl.slab > 1) pl.slab = std::max<int64_t>(1, pl.slab / 4);
        else if (pl.splits > 1) pl.splits = 1;
        else return sep_f64_mma_run(ctx, a, st);
    }
    GSC_CUDA(cudaStreamWaitEvent(st, ctx.scratch_ready, 0));
    unsigned char *base = static_cast<unsigned char *>(ctx.scratch.ptr);

    SlTab t{};
    t.cov = a.cov;
    t.z1 = a.z1;
    t.z2 = a.z2;
    t.dim = dim;
    t.n_modes = N;
    t.ax_b = dim == 3 ? a.axis[0] : nullptr;
    t.ax_m = dim == 3 ? a.axis[1] : a.axis[0];
    t.ax_n = dim == 3 ? a.axis[2] : a.axis[1];
    t.nb = nb;
    t.nm = nm;
    t.nn = nn;
    t.ncomp = ncomp;
    t.incompr = a.incompr ? 1 : 0;
    t.nt = pl.nt;
    t.n_tiles = pl.n_tiles;
    t.words = reinterpret_cast<int *>(base);
    t.modes = reinterpret_cast<SlMode *>(base + off_modes);
    t.svec = reinterpret_cast<longlong2 *>(base + off_s);
    t.btab = reinterpret_cast<longlong2 *>(base + off_b);
    t.g = base + off_g;
    t.f = base + off_f;
    t.rows_total = rows;
    int64_t *part = reinterpret_cast<int64_t *>(base + off_part);

    // |total| <= the modes of a segment <= 2^(12 - finer)
    int finer = 0;
    while (finer < kFinest && N <= (kSegModes >> (finer + 1))) ++finer;

    GSC_CUDA(cudaMemsetAsync(t.words, 0, kWords * sizeof(int), st));
    {
        TimedLaunch tl(st);
        tl.begin(K_SEP_TABLES);
        sl_modes_kernel<<<static_cast<unsigned>((N + 127) / 128), 128, 0, st>>>(t);
        tl.end();
        GSC_CUDA(cudaGetLastError());
    }
    for (int seg = 0; seg < pl.segs; ++seg) {
        t.j0 = seg * kSegModes;
        t.nj = std::min(kSegModes, N - t.j0);
        t.kb = (t.nj + kKbModes - 1) / kKbModes;
        const int npj = t.kb * kKbModes;
        {
            TimedLaunch tl(st);
            tl.begin(K_SEP_TABLES);
            const int64_t n_g = static_cast<int64_t>(pl.n_tiles) * t.kb * pl.nt * 4;
            const int64_t n_b = static_cast<int64_t>(nm) * npj, n_s = static_cast<int64_t>(nb) * npj;
            const int64_t blocks = (n_g + kTabThreads - 1) / kTabThreads + (n_b + kTabThreads - 1) / kTabThreads +
                                   (n_s + kTabThreads - 1) / kTabThreads;
            if (blocks > 0x7fffffff) return set_error(GSC_ERR_INVALID, "tables too large");
            GSC_CUDA(launch_after(sl_tables_kernel, dim3(static_cast<unsigned>(blocks)), dim3(kTabThreads), 0, st,
                                  t, n_g, n_b, n_s));
            tl.end();
        }
        for (int64_t m0 = 0; m0 < pl.m_tiles; m0 += pl.slab) {
            const int64_t mts = std::min(pl.slab, pl.m_tiles - m0);
            t.row0 = m0 * kTileRows;
            {
                TimedLaunch tl(st);
                tl.begin(K_SEP_SPLIT);
                GSC_CUDA(launch_after(sl_slice_kernel, dim3(static_cast<unsigned>(2 * mts), static_cast<unsigned>(t.kb)),
                                      dim3(kSliceThreads), 0, st, t));
                tl.end();
            }
            SlGemm p{};
            p.f = t.f;
            p.g = t.g;
            p.kb = t.kb;
            p.n_tiles = pl.n_tiles;
            p.splits = std::min(pl.splits, t.kb);
            p.row0 = t.row0;
            p.rows_total = rows;
            p.P = P;
            p.nn = nn;
            p.ncn = ncomp * nn;
            p.words = t.words;
            p.status = a.status;
            p.out = a.out;
            p.accumulate = seg > 0;
            p.finer = finer;
            if (parts > 0) {
                p.part = part + static_cast<size_t>(seg) * pl.splits * ncomp * P;
                p.split_stride = static_cast<int64_t>(ncomp) * P;
            }
            p.units = mts * pl.n_tiles * p.splits;
            const int64_t grid = std::min<int64_t>(p.units, sms);
            TimedLaunch tl(st);
            tl.begin(K_SEP_F64_SLICES);
            if (pl.nt == 96) GSC_TRY(launch_gemm<96>(p, grid, st));
            else if (pl.nt == 80) GSC_TRY(launch_gemm<80>(p, grid, st));
            else if (pl.nt == 64) GSC_TRY(launch_gemm<64>(p, grid, st));
            else if (pl.nt == 48) GSC_TRY(launch_gemm<48>(p, grid, st));
            else GSC_TRY(launch_gemm<32>(p, grid, st));
            tl.end();
        }
    }
    if (parts > 0) {
        // the last segment may have fewer k-blocks than the splits
        const int kb_last = (N - (pl.segs - 1) * kSegModes + kKbModes - 1) / kKbModes;
        TimedLaunch tl(st);
        tl.begin(K_SPLIT_REDUCE);
        GSC_CUDA(launch_after(sl_reduce_kernel, dim3(static_cast<unsigned>((P + 255) / 256), ncomp), dim3(256), 0, st,
                              part, pl.segs, pl.splits, std::min(pl.splits, kb_last), P, ncomp, finer, a.out,
                              t.words));
        tl.end();
    }
    // inputs outside this form: the FP64 MMA kernels, which do nothing otherwise
    GSC_TRY(sep_f64_launch(a, base + 256, t.words, st));
    GSC_CUDA(cudaEventRecord(ctx.scratch_ready, st));
    return GSC_OK;
}

}  // namespace gsc
