// separable_f64.cu -- the separable structured-grid contraction in FP64 on the
// double-precision MMA (mma.sync m8n8k4 f64), sm_103a.
//
// Same factorisation as separable_tc.cu (for each X_a one real GEMM with
// K = 2N: rows F[b, (2j, 2j+1)] = (Re, Im)(s_a[j] B[b, j]), columns
// G[c, (2j, 2j+1)] = (Re, -Im)(p_c C[c, j])), but every operand, product and
// sum is FP64, so the result agrees with the reference's summator
// (src/field.rs:37-65, :97-182 on the expanded grid) to FP64 round-off, for
// any inputs.  At 1.1 TFLOP/s it is the way out for what the sliced form
// (separable_slices.cu) does not take (values that are not finite, phases of
// 2^32 and more, calls without modes) and for grids that the x5 form flagged:
// both launches of a call are queued behind the fast form's and leave at once
// unless the word at run_if is set.  They run a fixed number of blocks, so that
// leaving costs the launches alone; a block takes the next tile when it is done
// with one (100^3 points x 1000 modes, 3 components, 1000 tiles: 16.7 ms, 19.1 when
// block b took tiles b, b + 608, ...).
//
// Tiles: one CTA per 64 x 64 output tile of one X_a, 4 warps of 32 x 32,
// K staged 32 at a time through shared memory (rows padded to 33 doubles to
// keep the fragment loads free of bank conflicts).  The F tile is formed in
// FP64 on the fly from the B table and s_a (4 FP64 operations per complex
// element, amortised over the 64 columns of the tile).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "internal.h"
#include "launch.cuh"

namespace gsc {
namespace {

constexpr int TM = 64, TN = 64, TK = 32;     // tile rows, columns, K per stage
constexpr int LDS = TK + 1;                  // padded shared-memory row (doubles)
constexpr int kF64Threads = 128;
constexpr int kF64TabGrid = 152 * 6;         // blocks of the tables that fit at once
// Blocks of the products on an SM: no more than it has tiles to compute, held to
// that by shared memory that they do not use.  They are launched while the tables
// still run, and where more of them fitted, they were placed several to an SM,
// beside idle ones, and shared its FP64 pipe to the end (40 x 80 x 100 x 2000
// modes, 160 tiles: 19.0 against 9.6 ms; 8 tiles took the time of 4).
constexpr int kF64Sms = 152, kF64MostPerSm = 4;
constexpr int kF64Smem[kF64MostPerSm] = {120 << 10, 80 << 10, 60 << 10, 0};   // of a block with 1, 2, 3, 4 on an SM

struct F64Tab {
    const double *cov, *z1, *z2;
    int dim, n_modes;
    const double *ax_b, *ax_m, *ax_n;
    int kb_dim, km_dim, kn_dim;
    int nb, nm, nn, ncomp, incompr;
    int k_pad, ncn_pad;
    double2 *svec;     // [nb][n_modes]
    double2 *btab;     // [n_modes][nm]
    double *g;         // [ncn_pad][k_pad]
    unsigned long long *next;   // sep_f64_kernel's next tile, set to 0 here
    const int *run_if; // null, or a device word: the launch does nothing while it is 0
};

__device__ void f64_svec_entry(const F64Tab &t, int64_t i) {
    const int b = static_cast<int>(i / t.n_modes), j = static_cast<int>(i % t.n_modes);
    double re = t.z1[j], im = -t.z2[j];
    if (t.dim == 3) {
        double s, c;
        sincos(t.cov[t.kb_dim * t.n_modes + j] * t.ax_b[b], &s, &c);
        const double r2 = re * c - im * s;
        im = re * s + im * c;
        re = r2;
    }
    t.svec[i] = make_double2(re, im);
}

__device__ void f64_btab_entry(const F64Tab &t, int64_t i) {
    const int j = static_cast<int>(i / t.nm), m = static_cast<int>(i % t.nm);
    double s, c;
    sincos(t.cov[t.km_dim * t.n_modes + j] * t.ax_m[m], &s, &c);
    t.btab[i] = make_double2(c, s);
}

__device__ void f64_gtab_entry(const F64Tab &t, int64_t i) {
    const int half_k = t.k_pad / 2;
    const int row = static_cast<int>(i / half_k), j = static_cast<int>(i % half_k);
    double re = 0.0, im = 0.0;
    if (row < t.ncomp * t.nn && j < t.n_modes) {
        const int c = row / t.nn, n = row - c * t.nn;
        double s, co;
        sincos(t.cov[t.kn_dim * t.n_modes + j] * t.ax_n[n], &s, &co);
        double pw = 1.0;
        if (t.incompr) {   // projector as the reference forms it (src/field.rs:138-152)
            double kk = 0.0;
            for (int d = 0; d < t.dim; ++d) {
                const double kd = t.cov[d * t.n_modes + j];
                kk = __dadd_rn(kk, __dmul_rn(kd, kd));
            }
            const double k0 = t.cov[j];
            const double k_2 = __ddiv_rn(k0, kk);
            pw = (c == 0) ? __dadd_rn(1.0, -__dmul_rn(k0, k_2))
                          : -__dmul_rn(t.cov[c * t.n_modes + j], k_2);
        }
        re = pw * co;
        im = -(pw * s);
    }
    t.g[static_cast<int64_t>(row) * t.k_pad + 2 * j] = re;
    t.g[static_cast<int64_t>(row) * t.k_pad + 2 * j + 1] = im;
}

// s, B and G tables: a fixed grid strides over all entries
__global__ void __launch_bounds__(256) f64_tables_kernel(F64Tab t) {
    after_previous();
    if (t.run_if && *t.run_if == 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) *t.next = 0;
    const int64_t n1 = static_cast<int64_t>(t.nb) * t.n_modes, n2 = static_cast<int64_t>(t.n_modes) * t.nm;
    const int64_t n3 = static_cast<int64_t>(t.ncn_pad) * (t.k_pad / 2);
    const int64_t step = static_cast<int64_t>(gridDim.x) * 256;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < n1 + n2 + n3; i += step) {
        if (i < n1) f64_svec_entry(t, i);
        else if (i < n1 + n2) f64_btab_entry(t, i - n1);
        else f64_gtab_entry(t, i - n1 - n2);
    }
}

__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

struct F64Params {
    const double2 *svec, *btab;
    const double *g;
    unsigned long long *next;
    int n_modes, nm, nn, ncn, k_pad;
    int m_tiles, n_tiles;
    int64_t tiles;       // nb * m_tiles * n_tiles
    double *out;
    int64_t comp_stride, batch_stride, row_stride;
    const int *run_if;   // as in F64Tab
};

__global__ void __launch_bounds__(kF64Threads)
sep_f64_kernel(const F64Params p) {
    after_previous();
    if (p.run_if && *p.run_if == 0) return;
    __shared__ double As[TM * LDS];
    __shared__ double Bs[TN * LDS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;   // warp's 32 x 32 sub-tile
    const int grp = lane >> 2, tig = lane & 3;

    __shared__ int64_t taken;
    for (;;) {
        if (tid == 0) taken = static_cast<int64_t>(atomicAdd(p.next, 1ull));
        __syncthreads();
        const int64_t tile = taken;          // every thread reads it before the barriers below
        if (tile >= p.tiles) break;
        const int nt = static_cast<int>(tile % p.n_tiles);
        const int64_t tm = tile / p.n_tiles;
        const int mt = static_cast<int>(tm % p.m_tiles), b = static_cast<int>(tm / p.m_tiles);
        const int m0 = mt * TM, n0 = nt * TN;

        double acc[4][4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

        const double2 *sv = p.svec + static_cast<int64_t>(b) * p.n_modes;
        for (int k0 = 0; k0 < p.k_pad; k0 += TK) {
            __syncthreads();
            // F tile: 64 rows x 16 modes, (Re, Im) interleaved along K
            for (int e = tid; e < TM * (TK / 2); e += kF64Threads) {
                const int r = e % TM, jl = e / TM;
                const int j = k0 / 2 + jl, m = m0 + r;
                double re = 0.0, im = 0.0;
                if (m < p.nm && j < p.n_modes) {
                    const double2 bt = p.btab[static_cast<int64_t>(j) * p.nm + m];
                    const double2 s = sv[j];
                    re = bt.x * s.x - bt.y * s.y;
                    im = bt.x * s.y + bt.y * s.x;
                }
                As[r * LDS + 2 * jl] = re;
                As[r * LDS + 2 * jl + 1] = im;
            }
            // G tile: 64 rows x 32 K
            for (int e = tid; e < TN * TK; e += kF64Threads) {
                const int r = e / TK, k = e % TK;
                Bs[r * LDS + k] = p.g[static_cast<int64_t>(n0 + r) * p.k_pad + k0 + k];
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < TK; kk += 4) {
                double a[4], bb[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = As[(wm + 8 * i + grp) * LDS + kk + tig];
#pragma unroll
                for (int j = 0; j < 4; ++j) bb[j] = Bs[(wn + 8 * j + grp) * LDS + kk + tig];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], bb[j]);
            }
        }

        double *ob = p.out + static_cast<int64_t>(b) * p.batch_stride;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int m = m0 + wm + 8 * i + grp;
            if (m >= p.nm) continue;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int gn = n0 + wn + 8 * j + 2 * tig + h;
                    if (gn >= p.ncn) continue;
                    const int comp = gn / p.nn;
                    ob[static_cast<int64_t>(m) * p.row_stride + comp * p.comp_stride + (gn - comp * p.nn)] =
                        acc[i][j][h];
                }
        }
    }
}

size_t up(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace

namespace {
struct F64Shape {
    int dim, N, ncomp, nb, nm, nn, k_pad, ncn, n_tiles, m_tiles, ncn_pad;
    int64_t P;
    size_t off_btab, off_g, off_next, total;     // s at 0
};
F64Shape f64_shape(const SepArgs &a) {
    F64Shape s;
    s.dim = static_cast<int>(a.dim);
    s.N = static_cast<int>(a.n_modes);
    s.ncomp = a.incompr ? s.dim : 1;
    s.nb = s.dim == 3 ? static_cast<int>(a.n[0]) : 1;
    s.nm = static_cast<int>(s.dim == 3 ? a.n[1] : a.n[0]);
    s.nn = static_cast<int>(s.dim == 3 ? a.n[2] : a.n[1]);
    s.P = static_cast<int64_t>(s.nb) * s.nm * s.nn;
    s.k_pad = std::max(TK, (2 * s.N + TK - 1) / TK * TK);
    s.ncn = s.ncomp * s.nn;
    s.n_tiles = (s.ncn + TN - 1) / TN;
    s.m_tiles = (s.nm + TM - 1) / TM;
    s.ncn_pad = s.n_tiles * TN;
    s.off_btab = up(sizeof(double2) * s.nb * static_cast<size_t>(s.N), 256);
    s.off_g = up(s.off_btab + sizeof(double2) * static_cast<size_t>(s.N) * s.nm, 256);
    s.off_next = up(s.off_g + sizeof(double) * static_cast<size_t>(s.ncn_pad) * s.k_pad, 256);
    s.total = s.off_next + sizeof(unsigned long long);
    return s;
}
}  // namespace

size_t sep_f64_scratch(const SepArgs &a) { return f64_shape(a).total; }

int sep_f64_launch(const SepArgs &a, unsigned char *base, const int *run_if, cudaStream_t st) {
    const F64Shape s = f64_shape(a);
    F64Tab t;
    t.cov = a.cov;
    t.z1 = a.z1;
    t.z2 = a.z2;
    t.dim = s.dim;
    t.n_modes = s.N;
    t.ax_b = s.dim == 3 ? a.axis[0] : nullptr;
    t.ax_m = s.dim == 3 ? a.axis[1] : a.axis[0];
    t.ax_n = s.dim == 3 ? a.axis[2] : a.axis[1];
    t.kb_dim = 0;
    t.km_dim = s.dim == 3 ? 1 : 0;
    t.kn_dim = s.dim == 3 ? 2 : 1;
    t.nb = s.nb;
    t.nm = s.nm;
    t.nn = s.nn;
    t.ncomp = s.ncomp;
    t.incompr = a.incompr ? 1 : 0;
    t.k_pad = s.k_pad;
    t.ncn_pad = s.ncn_pad;
    t.svec = reinterpret_cast<double2 *>(base);
    t.btab = reinterpret_cast<double2 *>(base + s.off_btab);
    t.g = reinterpret_cast<double *>(base + s.off_g);
    t.next = reinterpret_cast<unsigned long long *>(base + s.off_next);
    t.run_if = run_if;
    F64Params p;
    p.svec = t.svec;
    p.btab = t.btab;
    p.g = t.g;
    p.next = t.next;
    p.n_modes = s.N;
    p.nm = s.nm;
    p.nn = s.nn;
    p.ncn = s.ncn;
    p.k_pad = s.k_pad;
    p.m_tiles = s.m_tiles;
    p.n_tiles = s.n_tiles;
    p.tiles = static_cast<int64_t>(s.nb) * s.m_tiles * s.n_tiles;
    p.out = a.out;
    p.comp_stride = s.P;
    p.batch_stride = static_cast<int64_t>(s.nm) * s.nn;
    p.row_stride = s.nn;
    p.run_if = run_if;
    {
        TimedLaunch tl(st);
        tl.begin(K_SEP_TABLES);
        GSC_CUDA(launch_after(f64_tables_kernel, dim3(kF64TabGrid), dim3(256), 0, st, t));
        tl.end();
    }
    TimedLaunch tl(st);
    tl.begin(K_SEP_F64);
    const int per_sm = static_cast<int>(std::min<int64_t>(kF64MostPerSm, (p.tiles + kF64Sms - 1) / kF64Sms));
    const int own = (TM + TN) * LDS * static_cast<int>(sizeof(double));
    const size_t pad = static_cast<size_t>(std::max(0, kF64Smem[per_sm - 1] - own));
    GSC_TRY(smem_attr(reinterpret_cast<const void *>(sep_f64_kernel), kF64Smem[0]));
    GSC_CUDA(launch_after(sep_f64_kernel, dim3(static_cast<unsigned>(std::min<int64_t>(p.tiles, per_sm * kF64Sms))),
                          dim3(kF64Threads), pad, st, p));
    tl.end();
    return GSC_OK;
}

int sep_f64_run(DeviceCtx &ctx, const SepArgs &a, cudaStream_t st) {
    if (a.n[0] * a.n[1] * (a.dim == 3 ? a.n[2] : 1) == 0) return GSC_OK;
    if (!a.run_if && a.n_modes > 0) return sep_slices_run(ctx, a, st);
    return sep_f64_mma_run(ctx, a, st);
}

int sep_f64_mma_run(DeviceCtx &ctx, const SepArgs &a, cudaStream_t st) {
    GSC_TRY(ensure_dev(ctx, ctx.scratch, sep_f64_scratch(a)));
    GSC_CUDA(cudaStreamWaitEvent(st, ctx.scratch_ready, 0));
    GSC_TRY(sep_f64_launch(a, static_cast<unsigned char *>(ctx.scratch.ptr), a.run_if, st));
    GSC_CUDA(cudaEventRecord(ctx.scratch_ready, st));
    return GSC_OK;
}

}  // namespace gsc
