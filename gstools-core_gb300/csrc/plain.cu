// plain.cu -- FP64 randomization-method summators for GB300 (sm_103a).
//
// Computes, to FP64 accuracy end to end,
//   scalar   u[p]    = sum_j z1_j cos(k_j.x_p) + z2_j sin(k_j.x_p)
//            (reference: src/field.rs:37-65)
//   incompr  u[i, p] = sum_j w_ij (z1_j cos(k_j.x_p) + z2_j sin(k_j.x_p)),
//            w_0j = 1 - k_0j k_0j/|k_j|^2, w_ij = -k_ij k_0j/|k_j|^2
//            (reference: src/field.rs:97-182)
//
// Design.  GB300's FP64 pipe issues 2 lanes per clock and SM, so only what
// needs its rounding stays on it; the rest runs on the integer pipes beside it:
//  * phase k.x with the reference's bits: ((k0*x0 + k1*x1) + k2*x2), no FMA
//    (src/field.rs:57, src/short_vec.rs:30-33).  The first product and the sums
//    are FP64 instructions; the other products are formed and rounded by
//    integer instructions (rn_product), which overlap them (in 2-D every
//    second point of a thread has its second product on the FP64 pipe too, so
//    that both kinds take about as long: 606 -> 598 us);
//  * z1 cos + z2 sin = A cos(phase - beta), A = |z1 + i z2| and beta its
//    angle, set up per mode (plain_rec_kernel); the phase becomes a 64-bit
//    fraction of a turn and its cosine a 64-bit integer (fix64.cuh: 1.2e-16
//    RMS), one integer multiply by A (scaled by the largest A of 32 modes, to
//    2^-57 of it) and a 64-bit sum over those 32 modes, which is exact; one
//    FP64 multiply-add per 32 modes adds it to the point's total.
//    An FP64 evaluation (phase, table look-up, polynomials, sum) is 18 FP64
//    instructions per point*mode for d = 3 and 16 for d = 2; this one has 3 and
//    2.  Integer issue bounds the kernel now (a mode's 110 to 190 integer
//    instructions against 77 clocks for each FP64 one): 100,000 2-D points x
//    1000 modes 3391 -> 577 us, 250,007 3-D points x 1999 modes 18.86 -> 3.49 ms
//    (4.89 with all products on the FP64 pipe), and the error against 64-bit
//    sums fell from 1.7e-15 to 7e-16;
//  * phases of 2^32 to 1e13 differ in how they are brought to a fraction of a
//    turn (100,000 2-D points x 500 modes 388 us, with sincos() 3000); larger
//    ones, and modes with a NaN or an infinity, take CUDA's sincos() and FP64
//    sums for that mode (the same tests for a whole warp);
//  * mode records (96 bytes) are staged 32 at a time into shared memory with
//    cp.async double buffering; each thread keeps R points in registers;
//  * when there are too few points to fill 152 SMs, the modes are split
//    across blockIdx.y and the partial sums are added in split order by a
//    second kernel (deterministic; no atomics).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>

#include "fix64.cuh"
#include "internal.h"
#include "launch.cuh"

namespace gsc {
namespace {

constexpr int kThreads = 128;                       // threads per block
constexpr int kGroup = kPlainGroupModes;            // modes per staged tile and integer sum
constexpr int64_t kChunkModes = 1 << 20;            // modes per record build
constexpr int64_t kLeastChunkModes = 1 << 16;       // the same where device memory is short
static_assert(kThreads == kBatchThreads, "batch units assume the plain block size");
static_assert(kGroup == 32, "a warp builds the records of a group");

// Mode record (8-byte words): what the sums read from shared memory, then the
// FP64 values of the exact path.
//   k0, k1 mantissa | k2 mantissa, k1 and k2 exponents | kCosOffset - beta, A0 |
//   A1 A2 | s0 s1 | s2, |k| bound (FP32)
//   z1 z2 | w0 w1 | w2 k1 | k2 -
// k1 and k2 as factors of rn_product (mantissas {high, low}).  A_i = A w_i (A
// alone for the scalar field) as an integer of units s_i 2^-8 held in two words
// {high, low / 2}; s_i = 2^(e_i - 56), 2^(e_i) above every |A_i| of the mode's
// group of 32.  The bound is infinite for a mode of the exact path.
constexpr int kRec = 20, kRecStaged = 12;
enum { R_K0 = 0, R_M1 = 1, R_M2 = 2, R_EXP = 3, R_BETA = 4, R_A0 = 5, R_S0 = 8, R_KABS = 11,
       R_Z1 = 12, R_Z2 = 13, R_W0 = 14, R_K1 = 17, R_K2 = 18 };
static_assert(kRec * 8 == kPlainRecBytesPerMode, "record layout");
constexpr float kFastPhase = 4.29e9f;               // |k| |x| bound of turn_fraction, below 2^32
constexpr float kFarPhase = 1e13f;                  // that of turn_fraction_far, below 2^44

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// ---------------------------------------------------------------------------
// Mode records.  One warp per group of 32 modes, lane = mode (live: it exists);
// all lanes call.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void rec_group(const double *__restrict__ cov, int64_t n_modes, int dim,
                                          int64_t j, bool live, double z1, double z2, int incompr,
                                          double *__restrict__ r) {
    double k[3] = {0.0, 0.0, 0.0}, w[3] = {0.0, 0.0, 0.0};
    if (live)
        for (int d = 0; d < dim && d < 3; ++d) k[d] = cov[d * n_modes + j];
    bool regular = isfinite(z1) && isfinite(z2) && isfinite(k[0]) && factor_in_range(k[1]) && factor_in_range(k[2]);
    if (incompr) {
        // src/field.rs:138: k_2 = k0 / k.k, ShortVec::dot order, no FMA
        double kk = 0.0;
        for (int d = 0; d < dim; ++d) kk = __dadd_rn(kk, __dmul_rn(k[d], k[d]));
        const double k_2 = __ddiv_rn(k[0], kk);
        w[0] = __dadd_rn(1.0, -__dmul_rn(k[0], k_2));          // :148
        w[1] = -__dmul_rn(k[1], k_2);                            // :150-152
        w[2] = -__dmul_rn(k[2], k_2);
        regular = regular && isfinite(w[0]) && isfinite(w[1]) && isfinite(w[2]);
    }
    uint64_t beta = 0;
    double amp = 0.0;                                            // A 2^-ez
    int ez = 0;
    // at k = 0 the sine is 0 everywhere: its weight must not count in A, whose
    // size sets the error
    const bool still = k[0] == 0.0 && k[1] == 0.0 && k[2] == 0.0;
    if (regular) mode_angle(z1, still ? 0.0 : z2, &amp, &ez, &beta);
    const int nout = incompr ? dim : 1;
    double a[3] = {incompr ? amp * w[0] : amp, amp * w[1], amp * w[2]};
    double scale[3] = {0.0, 0.0, 0.0};
    long long fix[3] = {0, 0, 0};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        if (i >= nout) continue;
        int e = -100000;
        if (regular && a[i] != 0.0) e = exponent_of(a[i]) + ez;
        const int eg = __reduce_max_sync(0xffffffffu, e);
        if (eg == -100000) continue;                             // all zero: scale 0
        if (eg < -900 || eg > 900) {
            regular = false;
            continue;
        }
        if (regular) fix[i] = __double2ll_rn(scale_pow2(a[i], ez - eg + 58));
        scale[i] = scale_pow2(1.0, eg - 56);
    }
    if (!live) return;
    const Factor f1 = factor_of(k[1]), f2 = factor_of(k[2]);
    r[R_K0] = k[0];
    r[R_M1] = __hiloint2double(static_cast<int>(f1.m0), static_cast<int>(f1.m1));
    r[R_M2] = __hiloint2double(static_cast<int>(f2.m0), static_cast<int>(f2.m1));
    r[R_EXP] = __hiloint2double(static_cast<int>(f2.e), static_cast<int>(f1.e));
    const float kabs = regular ? __double2float_ru(fabs(k[0]) + fabs(k[1]) + fabs(k[2]))
                               : __int_as_float(0x7f800000);
    r[R_KABS] = __hiloint2double(0, __float_as_int(kabs));
    r[R_BETA] = __longlong_as_double(static_cast<long long>(kCosOffset - beta));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        r[R_A0 + i] = __hiloint2double(static_cast<int>(static_cast<uint32_t>(fix[i]) >> 1),
                                       static_cast<int>(fix[i] >> 32));
        r[R_S0 + i] = scale[i];
        r[R_W0 + i] = w[i];
    }
    r[R_Z1] = z1;
    r[R_Z2] = z2;
    r[R_K1] = k[1];
    r[R_K2] = k[2];
    r[kRec - 1] = 0.0;
}

// Records of modes [j0, j0 + nc); grid ceil(nc / kThreads), j0 a multiple of 32.
__global__ void __launch_bounds__(kThreads)
plain_rec_kernel(const double *__restrict__ cov, const double *__restrict__ z1,
                 const double *__restrict__ z2, int dim, int64_t n_modes, int64_t j0, int64_t nc,
                 int incompr, double *__restrict__ rec, const int *__restrict__ run_if) {
    wait_previous();
    if (run_if && *run_if == 0) return;      // a predicated launch that is not wanted
    const int64_t jl = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x, j = j0 + jl;
    const bool live = jl < nc;
    const double a = live ? z1[j] : 0.0, b = live ? z2[j] : 0.0;
    rec_group(cov, n_modes, dim, j, live, a, b, incompr, rec + jl * kRec);
    next_may_start();
}

// Records of every item of a batch: the warps of column blockIdx.y walk the
// groups of item blockIdx.y.  The Fourier factor, where present, multiplies z1
// and z2 first.
__global__ void __launch_bounds__(kThreads)
batch_rec_kernel(const BatchItem *__restrict__ items, int64_t n_items, double *__restrict__ rec) {
    for (int64_t i = blockIdx.y; i < n_items; i += gridDim.y) {
        const BatchItem &it = items[i];
        const int64_t groups = (it.n_modes + kGroup - 1) / kGroup;
        for (int64_t g = static_cast<int64_t>(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5);
             g < groups; g += static_cast<int64_t>(gridDim.x) * (kThreads / 32)) {
            const int64_t j = g * kGroup + (threadIdx.x & 31);
            const bool live = j < it.n_modes;
            double a = live ? it.z1[j] : 0.0, b = live ? it.z2[j] : 0.0;
            if (live && it.sf) {
                const double f = it.sf[j];
                a = __dmul_rn(f, a);
                b = __dmul_rn(f, b);
            }
            rec_group(it.cov, it.n_modes, it.dim, j, live, a, b, it.incompr,
                      rec + (it.mode_off + j) * kRec);
        }
    }
}

// phase = k.x in the reference's order (ndarray dot on strided columns)
template <int D>
__device__ __forceinline__ double phase_of(const double *k, const double *x) {
    double ph = __dmul_rn(k[0], x[0]);
    if (D > 1) ph = __dadd_rn(ph, __dmul_rn(k[1], x[1]));
    if (D > 2) ph = __dadd_rn(ph, __dmul_rn(k[2], x[2]));
    return ph;
}

// The cosine of a phase of 2^32 and more, a call: inlined it cost the sums of
// ordinary phases 0.7 % (100,000 2-D points x 1000 modes 578.5 -> 582.7 us).
__device__ __noinline__ int64_t far_cos(double ph, uint64_t beta, const CosTable *tab) {
    return cos_fixed(turn_fraction_far(ph) + beta, tab);
}

struct PlainSmem {
    CosTable tab;
    __align__(16) double rec[2][kGroup * kRecStaged];
};

// ---------------------------------------------------------------------------
// One block's work: the kThreads*R points starting at p_first (thread t owns
// p_first + t + r*kThreads), modes [jb, je) of the records `rec` (indices
// relative to them; jb a multiple of kGroup).  The sums are written
// (accumulate=0) or added (accumulate=1) at dst + i*sd + p*sp.  sm.tab is
// filled by the caller (not read by LIBM, CUDA's sincos() for every mode).
// ---------------------------------------------------------------------------
template <int D, int R, bool INC, bool LIBM>
__device__ __forceinline__ void plain_block(const double *__restrict__ pos, int64_t P,
                                            int64_t p_first, const double *__restrict__ rec,
                                            int64_t jb, int64_t je, int accumulate,
                                            double *__restrict__ dst, int64_t sd, int64_t sp,
                                            PlainSmem &sm) {
    constexpr int NOUT = INC ? D : 1;
    const int tid = threadIdx.x;
    const int64_t p0 = p_first + tid;

    auto stage_tile = [&](int buf, int64_t t0) {
        const int chunks = static_cast<int>(min(static_cast<int64_t>(kGroup), je - t0)) * (kRecStaged / 2);
        const double *src = rec + t0 * kRec;
        for (int c = tid; c < chunks; c += kThreads) {
            const int m = c / (kRecStaged / 2), q = c - m * (kRecStaged / 2);
            cp_async16(&sm.rec[buf][m * kRecStaged + 2 * q], src + m * kRec + 2 * q);
        }
        cp_async_commit();
    };
    if (jb < je) stage_tile(0, jb);

    // x0 as FP64, the other coordinates as factors of integer products (LIBM:
    // read from pos where they are needed)
    double x0[R];
    Factor xf[R][D > 1 ? D - 1 : 1];
    double x1[R];                            // D == 2: the second coordinate of odd r
    double acc[R][NOUT];
    double xabs = 0.0;
    bool bad[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t p = p0 + r * kThreads;
        double s = 0.0;
        bad[r] = false;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double x = p < P ? pos[d * P + p] : 0.0;
            bad[r] = bad[r] || isnan(x);
            s += fabs(x);
            if (d == 0) {
                x0[r] = x;
            } else {
                xf[r][d - 1] = factor_of(x);
                x1[r] = x;
                if (!factor_in_range(x) && !isnan(x)) xabs = __longlong_as_double(0x7ff0000000000000ll);
            }
        }
        xabs = fmax(xabs, s);
#pragma unroll
        for (int i = 0; i < NOUT; ++i) acc[r][i] = 0.0;
    }
    // warp-uniform bound on |x| for the range test (NaN coordinates do not
    // count: their points end as NaN)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) xabs = fmax(xabs, __shfl_xor_sync(0xffffffffu, xabs, o));
    const float xbound = __double2float_ru(xabs);

    int buf = 0;
    for (int64_t t0 = jb; t0 < je; t0 += kGroup, buf ^= 1) {
        const int tm = static_cast<int>(min(static_cast<int64_t>(kGroup), je - t0));
        if (t0 + kGroup < je) {
            stage_tile(buf ^ 1, t0 + kGroup);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const double *rc = sm.rec[buf];
        // sums over the group in units s_i 2^-56 ...; the truncated products of
        // a term leave out two units on average
        long long sum[R][NOUT];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int i = 0; i < NOUT; ++i) sum[r][i] = 2 * tm;
        // a mode's amplitudes (R_A0 ...) times its cosine c at point r
        auto add_term = [&](int r, int64_t c, const double (&av)[3]) {
            const int32_t ch = static_cast<int32_t>(c >> 32);
            const int32_t c0 = static_cast<int32_t>(static_cast<uint32_t>(c) >> 1);
#pragma unroll
            for (int i = 0; i < NOUT; ++i) {
                const int32_t ah = __double2loint(av[i]), a0 = __double2hiint(av[i]);
                sum[r][i] += static_cast<int64_t>(ah) * ch;
                sum[r][i] += static_cast<int64_t>(__mulhi(ah, c0) + __mulhi(a0, ch)) << 1;
            }
        };
#pragma unroll 1
        for (int m = 0; m < tm; ++m) {
            const double2 *mr = reinterpret_cast<const double2 *>(rc + m * kRecStaged);
            const float kb = __int_as_float(__double2loint(rc[m * kRecStaged + R_KABS]));
            if (!LIBM && kb * xbound < kFastPhase) {
                const double2 q0 = mr[0], q2 = mr[2];
                double2 q1 = make_double2(0.0, 0.0);
                if (D > 1) q1 = mr[1];
                const Factor kf[2] = {{static_cast<uint32_t>(__double2loint(q0.y)), static_cast<uint32_t>(__double2hiint(q0.y)),
                                       static_cast<uint32_t>(__double2loint(q1.y))},
                                      {static_cast<uint32_t>(__double2loint(q1.x)), static_cast<uint32_t>(__double2hiint(q1.x)),
                                       static_cast<uint32_t>(__double2hiint(q1.y))}};
                const uint64_t beta = static_cast<uint64_t>(__double_as_longlong(q2.x));
                const double k1 = kf[0].value();
                double av[3] = {q2.y, 0.0, 0.0};
                if (INC) {
                    const double2 q3 = mr[3];
                    av[1] = q3.x;
                    av[2] = q3.y;
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    // as phase_of
                    double ph = __dmul_rn(q0.x, x0[r]);
#pragma unroll
                    for (int d = 1; d < D; ++d) {
                        const bool fp64 = D == 2 && (r & 1);
                        ph = __dadd_rn(ph, fp64 ? __dmul_rn(k1, x1[r]) : rn_product(kf[d - 1], xf[r][d - 1]));
                    }
                    add_term(r, cos_fixed(turn_fraction(ph) + beta, &sm.tab), av);
                }
            } else if (!LIBM && kb * xbound < kFarPhase) {
                const double *ex = rec + (t0 + m) * kRec;
                const double k[3] = {ex[R_K0], ex[R_K1], ex[R_K2]};
                const double av[3] = {ex[R_A0], ex[R_A0 + 1], ex[R_A0 + 2]};
                const uint64_t beta = static_cast<uint64_t>(__double_as_longlong(ex[R_BETA]));
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int64_t p = p0 + r * kThreads;
                    double x[D];
#pragma unroll
                    for (int d = 0; d < D; ++d) x[d] = p < P ? pos[d * P + p] : 0.0;
                    add_term(r, far_cos(phase_of<D>(k, x), beta, &sm.tab), av);
                }
            } else {
                const double *ex = rec + (t0 + m) * kRec;
                const double z1 = ex[R_Z1], z2 = ex[R_Z2];
                const double k[3] = {ex[R_K0], ex[R_K1], ex[R_K2]};
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int64_t p = p0 + r * kThreads;
                    double x[D];
#pragma unroll
                    for (int d = 0; d < D; ++d) x[d] = p < P ? pos[d * P + p] : 0.0;
                    double sn, cs;
                    sincos(phase_of<D>(k, x), &sn, &cs);
                    const double z12 = __dadd_rn(__dmul_rn(z1, cs), __dmul_rn(z2, sn));
#pragma unroll
                    for (int i = 0; i < NOUT; ++i) {
                        if (INC) acc[r][i] = fma(ex[R_W0 + i], z12, acc[r][i]);
                        else acc[r][i] = __dadd_rn(acc[r][i], z12);
                        if (!LIBM) sum[r][i] -= 2;
                    }
                }
            }
        }
        if (!LIBM) {
#pragma unroll
            for (int i = 0; i < NOUT; ++i) {
                const double s = rc[R_S0 + i];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r][i] = fma(static_cast<double>(sum[r][i]), s, acc[r][i]);
            }
        }
        __syncthreads();   // buffer `buf` is refilled two tiles later
    }

#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t p = p0 + r * kThreads;
        if (p >= P) continue;
#pragma unroll
        for (int i = 0; i < NOUT; ++i) {
            double v = acc[r][i];
            if (bad[r] && jb < je) v = __longlong_as_double(0x7ff8000000000000ll);
            double *o = dst + i * sd + p * sp;
            *o = accumulate ? *o + v : v;
        }
    }
}

// ---------------------------------------------------------------------------
// Main kernel.  grid (ceil(P / (T*R)), splits), block T.
// Split s handles modes [s*mps, min(nc, (s+1)*mps)) of the current chunk and
// writes (accumulate=0) or adds (accumulate=1) its sums at
// dst + s*split_stride + i*sd + p*sp.
// ---------------------------------------------------------------------------
template <int D, int R, bool INC, bool LIBM>
__device__ __forceinline__ void
plain_kernel_body(const double *__restrict__ pos, int64_t P, const double *__restrict__ rec, int64_t nc,
             int64_t mps, int accumulate, double *__restrict__ dst, int64_t sd, int64_t sp,
             int64_t split_stride, const int *__restrict__ run_if) {
    __shared__ PlainSmem sm;
    if (run_if) {
        after_previous();
        if (*run_if == 0) return;            // a predicated launch that is not wanted
    }
    if (!LIBM) fill_cos_table(&sm.tab, threadIdx.x, kThreads);   // read after the first tile's barrier
    after_previous();
    const int64_t jb = static_cast<int64_t>(blockIdx.y) * mps;
    const int64_t je = min(nc, jb + mps);
    plain_block<D, R, INC, LIBM>(pos, P, static_cast<int64_t>(blockIdx.x) * (kThreads * R), rec, jb, je,
                                 accumulate, dst + static_cast<int64_t>(blockIdx.y) * split_stride, sd,
                                 sp, sm);
}
template <int D, int R, bool INC, bool LIBM>
__global__ void __launch_bounds__(kThreads)
plain_kernel(const double *__restrict__ pos, int64_t P, const double *__restrict__ rec, int64_t nc,
             int64_t mps, int accumulate, double *__restrict__ dst, int64_t sd, int64_t sp,
             int64_t split_stride, const int *__restrict__ run_if) {
    plain_kernel_body<D, R, INC, LIBM>(pos, P, rec, nc, mps, accumulate, dst, sd, sp, split_stride, run_if);
}
// Scalar fields with two points per thread: registers for more blocks per SM, since
// more warps feed the FP64 pipe, up to where they spill.  100,000 2-D points x
// 1000 modes 598 us at 8 blocks, 577 at 10; 250,007 3-D points x 1999 modes 3.52
// ms at 7, 3.49 at 8, 3.52 at 9.
template <int D>
__global__ void __launch_bounds__(kThreads, D == 3 ? 8 : 10)
plain_pair_kernel(const double *__restrict__ pos, int64_t P, const double *__restrict__ rec, int64_t nc,
             int64_t mps, int accumulate, double *__restrict__ dst, int64_t sd, int64_t sp,
             int64_t split_stride, const int *__restrict__ run_if) {
    plain_kernel_body<D, 2, false, false>(pos, P, rec, nc, mps, accumulate, dst, sd, sp, split_stride, run_if);
}

// ---------------------------------------------------------------------------
// Persistent batch kernel: each block takes the next unit of the device work
// queue (atomic counter) until the queue is empty.  A unit is one point block
// of one item and one of its mode ranges; its sums go to the item's output,
// or to its split slot when the item's modes are split.
// ---------------------------------------------------------------------------
template <int R>
__global__ void __launch_bounds__(kThreads)
batch_plain_kernel(const BatchItem *__restrict__ items, const BatchUnit *__restrict__ units,
                   int64_t n_units, int *__restrict__ counter, const double *__restrict__ rec) {
    __shared__ PlainSmem sm;
    __shared__ int s_unit;
    fill_cos_table(&sm.tab, threadIdx.x, kThreads);
    for (;;) {
        __syncthreads();                     // s_unit of the previous unit is consumed
        if (threadIdx.x == 0) s_unit = atomicAdd(counter, 1);
        __syncthreads();
        const int64_t u = s_unit;
        if (u >= n_units) break;
        const BatchUnit w = units[u];
        const BatchItem &it = items[w.item];
        const int64_t P = it.n_points;
        const int64_t nout = it.incompr ? it.dim : 1;
        double *dst = it.splits > 1 ? it.part + static_cast<int64_t>(w.split) * nout * P : it.out;
        const double *rc = rec + it.mode_off * kRec;
        switch (it.dim * 2 + it.incompr) {
            case 2:
                plain_block<1, R, false, false>(it.pos, P, w.p_first, rc, w.jb, w.je, 0, dst, P, 1, sm);
                break;
            case 4:
                plain_block<2, R, false, false>(it.pos, P, w.p_first, rc, w.jb, w.je, 0, dst, P, 1, sm);
                break;
            case 5:
                plain_block<2, R, true, false>(it.pos, P, w.p_first, rc, w.jb, w.je, 0, dst, P, 1, sm);
                break;
            case 6:
                plain_block<3, R, false, false>(it.pos, P, w.p_first, rc, w.jb, w.je, 0, dst, P, 1, sm);
                break;
            case 7:
                plain_block<3, R, true, false>(it.pos, P, w.p_first, rc, w.jb, w.je, 0, dst, P, 1, sm);
                break;
            default:
                break;                       // rejected on the host
        }
    }
}

// out[i*sd + p*sp] = sum_s part[s][i][p], s ascending
__global__ void split_reduce_kernel(const double *__restrict__ part, int64_t S, int64_t nout,
                                    int64_t P, double *__restrict__ out, int64_t sd, int64_t sp,
                                    const int *__restrict__ run_if) {
    after_previous();
    if (run_if && *run_if == 0) return;      // a predicated launch that is not wanted
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= nout * P) return;
    const int64_t i = t / P, p = t - i * P;
    double s = 0.0;
    for (int64_t k = 0; k < S; ++k) s += part[k * nout * P + t];
    out[i * sd + p * sp] = s;
}

// Any dimension (0 or > 3), scalar field: one thread per point, CUDA sincos.
__global__ void generic_kernel(const double *__restrict__ cov, const double *__restrict__ z1,
                               const double *__restrict__ z2, const double *__restrict__ pos,
                               int64_t dim, int64_t N, int64_t P, double *__restrict__ out,
                               int64_t sp, const int *__restrict__ run_if) {
    if (run_if && *run_if == 0) return;      // a predicated launch that is not wanted
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= P) return;
    double sum = 0.0;
    for (int64_t j = 0; j < N; ++j) {
        double ph = 0.0;
        for (int64_t d = 0; d < dim; ++d) ph = __dadd_rn(ph, __dmul_rn(cov[d * N + j], pos[d * P + p]));
        double sn, cs;
        sincos(ph, &sn, &cs);
        sum = __dadd_rn(sum, __dadd_rn(__dmul_rn(z1[j], cs), __dmul_rn(z2[j], sn)));
    }
    out[p * sp] = sum;
}

// where a plain launch reads and writes; modes [0, nc) of rec in splits of mps
struct PlainLaunch {
    const double *pos;
    int64_t P;
    const double *rec;
    int64_t nc, mps;
    int accumulate;
    double *dst;
    int64_t sd, sp, split_stride;
    const int *run_if;
    bool after;            // overlaps the end of the record kernel
};

template <int R, bool INC, bool LIBM>
int dispatch_dim(int64_t dim, dim3 grid, cudaStream_t st, const PlainLaunch &l) {
    auto launch = [&](auto fn) -> int {
        if (l.after) {
            GSC_CUDA(launch_after(fn, grid, dim3(kThreads), 0, st, l.pos, l.P, l.rec, l.nc, l.mps, l.accumulate,
                                  l.dst, l.sd, l.sp, l.split_stride, l.run_if));
            return GSC_OK;
        }
        fn<<<grid, kThreads, 0, st>>>(l.pos, l.P, l.rec, l.nc, l.mps, l.accumulate, l.dst, l.sd, l.sp,
                                      l.split_stride, l.run_if);
        GSC_CUDA(cudaGetLastError());
        return GSC_OK;
    };
    if constexpr (!INC) {
        if (dim == 1) return launch(plain_kernel<1, R, INC, LIBM>);
    }
    if constexpr (R == 2 && !INC && !LIBM) {
        if (dim == 2) return launch(plain_pair_kernel<2>);
        if (dim == 3) return launch(plain_pair_kernel<3>);
    } else {
        if (dim == 2) return launch(plain_kernel<2, R, INC, LIBM>);
        if (dim == 3) return launch(plain_kernel<3, R, INC, LIBM>);
    }
    return set_error(GSC_ERR_DIM, "unsupported dimension for the plain kernel");
}

int dispatch_plain(int R, bool incompr, bool libm, int64_t dim, dim3 grid, cudaStream_t st,
                   const PlainLaunch &l) {
    if (libm && R == 1)
        return incompr ? dispatch_dim<1, true, true>(dim, grid, st, l)
                       : dispatch_dim<1, false, true>(dim, grid, st, l);
    if (libm)
        return incompr ? dispatch_dim<4, true, true>(dim, grid, st, l)
                       : dispatch_dim<4, false, true>(dim, grid, st, l);
    if (R == 1)
        return incompr ? dispatch_dim<1, true, false>(dim, grid, st, l)
                       : dispatch_dim<1, false, false>(dim, grid, st, l);
    if (R == 2)
        return incompr ? dispatch_dim<2, true, false>(dim, grid, st, l)
                       : dispatch_dim<2, false, false>(dim, grid, st, l);
    return incompr ? dispatch_dim<4, true, false>(dim, grid, st, l)
                   : dispatch_dim<4, false, false>(dim, grid, st, l);
}

// Launch shape: points per thread R and mode splits S (of mps modes, a
// multiple of the group of 32), by the time of the busiest SM.  Measured on
// GB300: a point*mode keeps a quarter of an SM for 195, 250 and 295 clocks a warp
// in 1, 2 and 3 dimensions (280 and 350 for vectors) at R = 2, 7 % more at R = 1
// and 3 % more at R = 4 (scalar fields at R = 2 were given more blocks per SM since,
// and take about 235 and 280 in 2 and 3 dimensions); a warp alone takes 2.2 times
// that per mode and point, so an SM wants more than two blocks.  Small calls want
// the splits that give them (1,000 2-D points x 1000 modes: 262 us with 2 splits at
// R = 2, 31 us with 32 at R = 1), large ones whole waves.  CUDA's sincos() form has
// R = 1 and 4: one 3-D point x 64 modes takes 52 and 169 us, 50,000 x 1000 modes
// 3157 and 3099.
//
// What splits smooth is part of one wave, a share that falls with the number of
// waves, while their partial sums grow with the points: 28.8 million 3-D
// vectors would gain 0.04 % from 2.8 GB of them.  They stop at
// kMostPartialBytes, above what any call of up to 2 million points wants.
constexpr int64_t kMostPartialBytes = int64_t(256) << 20;
struct PlainShape {
    int R;
    int64_t bx, S, mps;
};
PlainShape plain_shape(int64_t P, int64_t chunk, int64_t dim, int64_t nout, int sms, bool libm) {
    PlainShape best{4, (P + 4 * kThreads - 1) / (4 * kThreads), 1, (chunk + kGroup - 1) / kGroup * kGroup};
    double best_cost = 1e300;
    const double base = libm ? 2000.0 : nout > 1 ? (dim == 3 ? 350.0 : 280.0) : dim == 1 ? 195.0 : dim == 2 ? 250.0 : 295.0;
    const int64_t groups = std::max<int64_t>(1, (chunk + kGroup - 1) / kGroup);
    for (int R : {4, 2, 1}) {
        if (libm && R == 2) continue;
        const double pm = base * (libm ? (R == 1 ? 1.02 : 1.0) : R == 1 ? 1.07 : R == 2 ? 1.0 : 1.03);
        const int64_t bx = (P + kThreads * R - 1) / (kThreads * R);
        for (int64_t S = 1; S <= 64 && S <= groups; ++S) {
            const int64_t per = (groups + S - 1) / S;
            if (S > 1 && S * nout * P > kMostPartialBytes / static_cast<int64_t>(sizeof(double))) break;
            if ((groups + per - 1) / per != S) continue;       // fewer splits of the same share
            const double on_sm = std::ceil(static_cast<double>(bx) * S / sms);
            double cost = per * kGroup * std::max(on_sm, 2.2) * R * pm;
            if (S > 1) cost += 4000.0 + static_cast<double>(S) * nout * P * 8.0 / 2000.0;
            if (cost < best_cost) {
                best_cost = cost;
                best = PlainShape{R, bx, S, per * kGroup};
            }
        }
    }
    return best;
}

// The shape of a launch that mostly has nothing to do (run_if): few blocks, which
// each cost time only to look at the word (2,097,152 points x 4096 modes: 137 us
// of nothing in a real launch's shape, 8 us in 4,096 blocks).
PlainShape plain_shape_unlikely(int64_t P, int64_t chunk, int sms) {
    PlainShape s{4, (P + 4 * kThreads - 1) / (4 * kThreads), 1, 0};
    const int64_t groups = std::max<int64_t>(1, (chunk + kGroup - 1) / kGroup);
    const int64_t want = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(groups, 64), 4 * sms / s.bx));
    const int64_t per = (groups + want - 1) / want;
    s.S = (groups + per - 1) / per;
    s.mps = per * kGroup;
    return s;
}

int sm_count(int device) {
    static std::atomic<int> cached[64];   // zero-initialised (static storage)
    if (device >= 0 && device < 64) {
        const int c = cached[device].load(std::memory_order_relaxed);
        if (c) return c;
    }
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0)
        n = 152;
    if (device >= 0 && device < 64) cached[device].store(n, std::memory_order_relaxed);
    return n;
}

__global__ void grid_expand_kernel(const double *__restrict__ a0, const double *__restrict__ a1,
                                   const double *__restrict__ a2, int64_t n0, int64_t n1,
                                   int64_t n2, int dim, double *__restrict__ pos) {
    const int64_t P = n0 * n1 * n2;
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= P) return;
    const int64_t i2 = p % n2, i01 = p / n2, i1 = i01 % n1, i0 = i01 / n1;
    if (dim == 2) {
        // (n0, n1) grid: p = i0 * n1 + i1 with n2 == 1
        pos[p] = a0[i0];
        pos[P + p] = a1[i1];
    } else {
        pos[p] = a0[i0];
        pos[P + p] = a1[i1];
        pos[2 * P + p] = a2[i2];
    }
}

// (nout, P) rows -> (P, nout) for the points [p0, p0 + n): each thread moves
// one point's nout values (coalesced reads per component; a warp's nout
// stores cover one contiguous run of 32 * nout values).
__global__ void interleave_kernel(const double *__restrict__ src, int nout, int64_t P, int64_t p0,
                                  int64_t n, double *__restrict__ dst) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t p = p0 + i;
    for (int c = 0; c < nout; ++c) dst[p * nout + c] = src[c * P + p];
}

// Fourier method: the spectrum factor multiplies z1 cos + z2 sin of its mode
// (src/field.rs:241-242), so folding it into z1, z2 once per call lets every
// summator form compute the Fourier field unchanged.
__global__ void fourier_scale_kernel(const double *__restrict__ sf, const double *z1,
                                     const double *z2, int64_t n, double *z1s, double *z2s) {
    after_previous();
    const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double f = sf[j], a = z1[j], b = z2[j];
    z1s[j] = __dmul_rn(f, a);
    z2s[j] = __dmul_rn(f, b);
}

}  // namespace

int fourier_scale(const double *sf, const double *z1, const double *z2, int64_t n, double *z1s,
                  double *z2s, cudaStream_t st) {
    if (n == 0) return GSC_OK;
    TimedLaunch tl(st);
    tl.begin(K_FOURIER_SCALE);
    fourier_scale_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(sf, z1, z2, n, z1s,
                                                                                z2s);
    tl.end();
    GSC_CUDA(cudaGetLastError());
    return GSC_OK;
}

int split_reduce(const double *part, int64_t S, int64_t nout, int64_t P, double *out, int64_t sd,
                 int64_t sp, cudaStream_t st) {
    TimedLaunch tl(st);
    tl.begin(K_SPLIT_REDUCE);
    const int64_t tot = nout * P;
    GSC_CUDA(launch_after(split_reduce_kernel, dim3(static_cast<unsigned>((tot + 255) / 256)), dim3(256), 0, st,
                          part, S, nout, P, out, sd, sp, static_cast<const int *>(nullptr)));
    tl.end();
    return GSC_OK;
}

int grid_expand(const double *const *axis, const int64_t *n, int64_t dim, double *pos,
                cudaStream_t st) {
    const int64_t n2 = dim == 3 ? n[2] : 1;
    const int64_t P = n[0] * n[1] * n2;
    if (P == 0) return GSC_OK;
    grid_expand_kernel<<<static_cast<unsigned>((P + 255) / 256), 256, 0, st>>>(
        axis[0], axis[1], dim == 3 ? axis[2] : nullptr, n[0], n[1], n2, static_cast<int>(dim), pos);
    GSC_CUDA(cudaGetLastError());
    return GSC_OK;
}

int interleave_rows(const double *src, int64_t nout, int64_t P, int64_t p0, int64_t p1,
                    double *dst, cudaStream_t st) {
    const int64_t n = p1 - p0;
    if (n <= 0) return GSC_OK;
    TimedLaunch tl(st);
    tl.begin(K_INTERLEAVE);
    interleave_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
        src, static_cast<int>(nout), P, p0, n, dst);
    tl.end();
    GSC_CUDA(cudaGetLastError());
    return GSC_OK;
}

int plain_run(DeviceCtx &ctx, const PlainArgs &a, cudaStream_t st) {
    const int64_t P = a.n_points, N = a.n_modes, dim = a.dim;
    if (P == 0) return GSC_OK;
    const int64_t nout = a.incompr ? dim : 1;
    const bool libm = a.variant == 1;

    if (!a.incompr && (dim == 0 || dim > 3)) {
        TimedLaunch tl(st);
        tl.begin(K_GENERIC);
        const int tpb = 128;
        generic_kernel<<<static_cast<unsigned>((P + tpb - 1) / tpb), tpb, 0, st>>>(
            a.cov, a.z1, a.z2, a.pos, dim, N, P, a.out, a.out_sp, a.run_if);
        tl.end();
        GSC_CUDA(cudaGetLastError());
        return GSC_OK;
    }
    if (a.incompr && dim != 2 && dim != 3)
        return set_error(GSC_ERR_DIM, "Only two- and three-dimensional problems are supported.");

    // ---- launch geometry ---------------------------------------------------
    int64_t chunk = std::min<int64_t>(N, kChunkModes);
    PlainShape shp = a.run_if ? plain_shape_unlikely(P, chunk, sm_count(ctx.device))
                              : plain_shape(P, chunk, dim, nout, sm_count(ctx.device), libm);
    if (shp.bx > 0x7fffffff) return set_error(GSC_ERR_INVALID, "too many points for one launch");

    // ---- scratch: mode records of one chunk, split partials ------------------
    size_t off_part = 0;
    for (;;) {
        off_part = (static_cast<size_t>(chunk) * kPlainRecBytesPerMode + 255) / 256 * 256;
        const size_t part_bytes = shp.S > 1 ? static_cast<size_t>(shp.S) * nout * P * sizeof(double) : 0;
        const int rc = ensure_dev(ctx, ctx.scratch, off_part + part_bytes + 256);
        if (rc == GSC_OK) break;
        if (rc != GSC_ERR_NOMEM) return rc;
        // no room: no splits, then the records of fewer modes at a time
        if (shp.S > 1) shp.S = 1;
        else if (chunk > kLeastChunkModes) chunk = std::max<int64_t>(kLeastChunkModes, chunk / 4 / kGroup * kGroup);
        else return rc;
        if (shp.S == 1) shp.mps = (chunk + kGroup - 1) / kGroup * kGroup;
    }
    const int64_t S = shp.S;
    GSC_CUDA(cudaStreamWaitEvent(st, ctx.scratch_ready, 0));
    unsigned char *sbase = static_cast<unsigned char *>(ctx.scratch.ptr);
    double *rec = reinterpret_cast<double *>(sbase);
    double *part = reinterpret_cast<double *>(sbase + off_part);

    PlainLaunch l{};
    l.pos = a.pos;
    l.P = P;
    l.rec = rec;
    l.dst = S > 1 ? part : a.out;
    l.sd = S > 1 ? P : a.out_sd;
    l.sp = S > 1 ? 1 : a.out_sp;
    l.split_stride = S > 1 ? nout * P : 0;
    l.run_if = a.run_if;
    l.after = true;

    int64_t j0 = 0;
    do {
        const int64_t nc = std::min<int64_t>(N - j0, chunk);
        if (nc > 0) {
            TimedLaunch tl(st);
            tl.begin(K_MODE_TABLE);
            GSC_CUDA(launch_after(plain_rec_kernel, dim3(static_cast<unsigned>((nc + kThreads - 1) / kThreads)),
                                  dim3(kThreads), 0, st, a.cov, a.z1, a.z2, static_cast<int>(dim), N, j0, nc,
                                  a.incompr ? 1 : 0, rec, a.run_if));
            tl.end();
        }
        l.nc = nc;
        l.mps = shp.mps;
        l.accumulate = j0 > 0;
        // on later chunks, splits past the end of a short chunk are not
        // launched and keep their sums
        const int64_t s_used = (j0 == 0 || nc == 0) ? S : std::min<int64_t>(S, (nc + l.mps - 1) / l.mps);
        TimedLaunch tl(st);
        tl.begin(a.incompr ? K_PLAIN_INCOMPR : (libm ? K_PLAIN_LIBM : K_PLAIN_SCALAR));
        const int rc = dispatch_plain(shp.R, a.incompr, libm, dim,
                                      dim3(static_cast<unsigned>(shp.bx), static_cast<unsigned>(s_used)),
                                      st, l);
        tl.end();
        if (rc != GSC_OK) return rc;
        j0 += nc;
    } while (j0 < N);

    if (S > 1) {
        TimedLaunch tl(st);
        tl.begin(K_SPLIT_REDUCE);
        const int64_t tot = nout * P;
        GSC_CUDA(launch_after(split_reduce_kernel, dim3(static_cast<unsigned>((tot + 255) / 256)), dim3(256), 0, st,
                              part, S, nout, P, a.out, a.out_sd, a.out_sp, a.run_if));
        tl.end();
    }
    GSC_CUDA(cudaEventRecord(ctx.scratch_ready, st));
    return GSC_OK;
}

// ---- batched ensembles: records and the persistent kernel --------------------
int batch_plain_tables(const BatchItem *items, int64_t n_items, int64_t total_modes, double *rec,
                       cudaStream_t st) {
    if (total_modes == 0) return GSC_OK;
    TimedLaunch tl(st);
    tl.begin(K_BATCH_TABLES);
    // enough warps for the items' mean group count, the larger items striding
    const int64_t mean = (total_modes / kGroup + n_items) / n_items;
    const unsigned gx = static_cast<unsigned>(std::min<int64_t>(64, std::max<int64_t>(1, mean / (kThreads / 32))));
    batch_rec_kernel<<<dim3(gx, static_cast<unsigned>(std::min<int64_t>(n_items, 65535))), kThreads, 0, st>>>(
        items, n_items, rec);
    tl.end();
    GSC_CUDA(cudaGetLastError());
    return GSC_OK;
}

namespace {
using BatchPlainFn = void (*)(const BatchItem *, const BatchUnit *, int64_t, int *, const double *);
BatchPlainFn batch_plain_fn(int R) {
    if (R == 2) return batch_plain_kernel<2>;
    if (R == 4) return batch_plain_kernel<4>;
    if (R == 8) return batch_plain_kernel<8>;
    return nullptr;
}
}  // namespace

// The tile sizes that a caller may name (8 or 16 modes; 8 alone with 8 points
// per thread); the kernels stage 32 modes whatever it is.
bool batch_plain_config_ok(int R, int tile) {
    return batch_plain_fn(R) != nullptr && (tile == 8 || (tile == 16 && R != 8));
}

int batch_plain_occupancy(int R) {
    BatchPlainFn fn = batch_plain_fn(R);
    if (!fn) return 0;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kThreads, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int batch_plain_launch(int R, int blocks, const BatchItem *items, const BatchUnit *units,
                       int64_t n_units, int *counter, const double *rec, cudaStream_t st) {
    BatchPlainFn fn = batch_plain_fn(R);
    if (!fn) return set_error(GSC_ERR_INVALID, "unsupported batch configuration");
    TimedLaunch tl(st);
    tl.begin(K_BATCH_PLAIN);
    fn<<<blocks, kThreads, 0, st>>>(items, units, n_units, counter, rec);
    tl.end();
    GSC_CUDA(cudaGetLastError());
    return GSC_OK;
}

}  // namespace gsc

// ---------------------------------------------------------------------------
// Allocation-free variant of the scalar FP64 summator.
//
// Some callers must not let a library allocate device memory: a host whose
// framework allocator already owns the whole device (a cudaMalloc from the
// library would fail or fragment that pool), a real-time loop that cannot
// afford to block in the driver's allocator, or a plug-in host that only
// permits memory from its own arena.  For them the mode records of the
// plain kernel live in one fixed array compiled into the library, so a call
// allocates nothing; the caller passes the inputs and the output as usual.
//
// The array (160 KiB of mode records, enough for 1024 modes) is held on every GPU that loads the library until the process
// exits.  All calls share it and it keeps the last call's contents; every
// call rewrites the part it reads, so nothing has to start at zero.  Calls
// whose kernels overlap on the GPU (different streams, no ordering between
// them) race on the array.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char
    gsc_noalloc_scratch[gsc::kNoAllocModes * gsc::kPlainRecBytesPerMode];

namespace gsc {

static std::mutex g_noalloc_mu;
static void *g_noalloc_addr[64] = {nullptr};

// The device address of the fixed array on the current device, looked up
// once per device.  Host code cannot use the array's name as a device
// address: outside device code it names a host-side stand-in.
static int noalloc_address(int device, void **addr) {
    if (device < 0 || device >= 64) return set_error(GSC_ERR_INVALID, "device ordinal out of range");
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[device]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, gsc_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(fixed record array)");
        g_noalloc_addr[device] = p;
    }
    *addr = g_noalloc_addr[device];
    return GSC_OK;
}

int plain_noalloc_run(int device, const PlainArgs &a, cudaStream_t st) {
    constexpr int R = 4;
    const int64_t P = a.n_points, N = a.n_modes;
    if (N > kNoAllocModes)
        return set_error(GSC_ERR_INVALID, "gsc_summate_dev_noalloc takes at most " +
                                              std::to_string(kNoAllocModes) +
                                              " modes per call (its fixed record array holds "
                                              "that many); split the modes over several calls "
                                              "or use gsc_summate_dev");
    if (P == 0) return GSC_OK;
    void *scratch = nullptr;
    GSC_TRY(noalloc_address(device, &scratch));
    double *rec = static_cast<double *>(scratch);
    const int64_t bx = (P + kThreads * R - 1) / (kThreads * R);
    if (bx > 0x7fffffff) return set_error(GSC_ERR_INVALID, "too many points for one launch");
    if (N > 0) {
        plain_rec_kernel<<<static_cast<unsigned>((N + kThreads - 1) / kThreads), kThreads, 0, st>>>(
            a.cov, a.z1, a.z2, static_cast<int>(a.dim), N, 0, N, 0, rec, nullptr);
        GSC_CUDA(cudaGetLastError());
    }
    // one mode split: every point's modes are summed by one thread, in order
    PlainLaunch l{};
    l.pos = a.pos;
    l.P = P;
    l.rec = rec;
    l.nc = N;
    l.mps = N;
    l.dst = a.out;
    l.sd = P;
    l.sp = a.out_sp;
    return dispatch_plain(R, false, false, a.dim, dim3(static_cast<unsigned>(bx), 1), st, l);
}

}  // namespace gsc
