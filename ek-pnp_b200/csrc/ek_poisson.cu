// ek_poisson.cu -- spectral Poisson solve of the reference's discretisation.
//
// The reference (fast_Poisson, poisson.cu:180-306) odd-extends the interior
// rows to ne = 2(ny-1) rows, runs a 2D complex FFT (cuFFT), divides by
//     mu = kx^2 + (4/dy^2) sin^2(ky dy/2),  kx = 2 pi m/Lx,  ky = 2 pi n/(ne dy)
// and transforms back.  Along y the odd extension makes this a sine transform,
// and (4/dy^2) sin^2(n pi/(2(ny-1))) are exactly the eigenvalues of the
// three-point Dirichlet Laplacian on the ny-2 interior rows.  So, for every
// x-mode m, the reference solves the tridiagonal system
//     phi_{j-1} - (2 + kx_m^2 dy^2) phi_j + phi_{j+1} = dy^2 S_j,  phi_{-1} = phi_{n} = 0
// and this file solves it directly (Thomas recurrence with pivots computed
// once per channel), for any ny, with no FFT in y:
//   pass A  per pair of interior rows: real FFT in x (two rows packed as one
//           complex row; register-blocked radix-16 passes for powers of two
//           from 16 on, mixed radix otherwise, a direct sum for primes) -> spec[j][m], m = 0..nx/2
//   pass B  per x-mode m: Thomas sweeps down the column, partitioned into row
//           segments of at most 16 rows held in registers (one thread per
//           mode for columns taller than 8192 rows)
//   pass C  per pair of rows: inverse real FFT -> psi; wall rows = zeta(x)
// The result equals the reference's to rounding (the test suite compares).
#include <cuda_runtime.h>

#include "ek_fft16.cuh"
#include "ek_internal.h"

namespace ek {
namespace {

constexpr int PTPB = 256;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
template <typename C> __device__ __forceinline__ C cmake(double a, double b);
template <> __device__ __forceinline__ double2 cmake<double2>(double a, double b) { return make_double2(a, b); }
template <> __device__ __forceinline__ float2 cmake<float2>(double a, double b) { return make_float2((float)a, (float)b); }
__device__ __forceinline__ int brev(int i, int lg) { return (int)(__brev((unsigned)i) >> (32 - lg)); }

// ---- rows of any length (FP64): mixed radix --------------------------------
//
// nx = r_1 r_2 ... (Stockham, self-sorting, two buffers in shared memory).  With
// L = r_1 ... r_{i-1} the transforms of length L done so far, pass i takes the
// elements j + q nx/r (q < r), j < nx/r, to (j/L) L r + j mod L + q' L, with
// the twiddle exp(-2 pi i (j mod L) q / (L r)) and an r-point DFT.  Radices 4,
// 2, 3 and 5 are butterflies held by a thread; any other prime r is summed
// term by term, one output a thread: nx r products instead of the nx^2 of
// the direct transform, which took 211 us (inverse 263) at 1000 x 257 on B200
// against 10.4 (8.4) us here.  All roots are powers of the nx-th root from the table.
constexpr int MIXED_MAX_NX = 2048;  // longest (ek_create, ek_poisson_noalloc)
struct Radices {
    int n;
    int r[11];  // nx <= 2048 = 4^5 2
};

template <bool INV> __device__ __forceinline__ double2 root(const double2 *__restrict__ tw, int k) {
    const double2 w = __ldg(tw + k);
    return INV ? cconj(w) : w;
}
// z times -i (forward) or +i (inverse)
template <bool INV> __device__ __forceinline__ double2 rot90(double2 z) {
    return INV ? make_double2(-z.y, z.x) : make_double2(z.y, -z.x);
}

template <bool INV, int R>
__device__ __forceinline__ void radix_pass(const double2 *__restrict__ in, double2 *__restrict__ out, int nx, int L,
                                           const double2 *__restrict__ tw, int t, int T) {
    const int m = nx / R, ts = nx / (L * R);
    for (int j = t; j < m; j += T) {
        const int hi = j / L, k = j - hi * L;
        double2 x[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            x[q] = in[j + q * m];
            if (q > 0 && k > 0) x[q] = cmul(x[q], root<INV>(tw, k * q * ts));
        }
        double2 *o = out + hi * L * R + k;
        if constexpr (R == 2) {
            o[0] = cadd(x[0], x[1]);
            o[L] = csub(x[0], x[1]);
        } else if constexpr (R == 4) {
            const double2 s0 = cadd(x[0], x[2]), d0 = csub(x[0], x[2]), s1 = cadd(x[1], x[3]);
            const double2 d1 = rot90<INV>(csub(x[1], x[3]));
            o[0] = cadd(s0, s1);
            o[L] = cadd(d0, d1);
            o[2 * L] = csub(s0, s1);
            o[3 * L] = csub(d0, d1);
        } else if constexpr (R == 3) {
            constexpr double h = 0.86602540378443865;  // sin(pi/3)
            const double2 s = cadd(x[1], x[2]), d = rot90<INV>(csub(x[1], x[2]));
            const double2 c = make_double2(x[0].x - 0.5 * s.x, x[0].y - 0.5 * s.y);
            o[0] = cadd(x[0], s);
            o[L] = make_double2(c.x + h * d.x, c.y + h * d.y);
            o[2 * L] = make_double2(c.x - h * d.x, c.y - h * d.y);
        } else {
            static_assert(R == 5, "radices 2 to 5");
            constexpr double c1 = 0.30901699437494742, c2 = -0.80901699437494742;  // cos(2 pi/5), cos(4 pi/5)
            constexpr double s1 = 0.95105651629515357, s2 = 0.58778525229247313;   // sin(2 pi/5), sin(4 pi/5)
            const double2 a1 = cadd(x[1], x[4]), a2 = cadd(x[2], x[3]);
            const double2 b1 = rot90<INV>(csub(x[1], x[4])), b2 = rot90<INV>(csub(x[2], x[3]));
            const double2 e1 = make_double2(x[0].x + c1 * a1.x + c2 * a2.x, x[0].y + c1 * a1.y + c2 * a2.y);
            const double2 e2 = make_double2(x[0].x + c2 * a1.x + c1 * a2.x, x[0].y + c2 * a1.y + c1 * a2.y);
            const double2 f1 = make_double2(s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y);
            const double2 f2 = make_double2(s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y);
            o[0] = cadd(x[0], cadd(a1, a2));
            o[L] = cadd(e1, f1);
            o[2 * L] = cadd(e2, f2);
            o[3 * L] = csub(e2, f2);
            o[4 * L] = csub(e1, f1);
        }
    }
}

// A pass of prime radix r > 5: one output a thread, its r terms summed in order.
template <bool INV>
__device__ __forceinline__ void prime_pass(const double2 *__restrict__ in, double2 *__restrict__ out, int nx, int L,
                                           int r, const double2 *__restrict__ tw, int t, int T) {
    const int m = nx / r, ts = nx / (L * r);
    for (int e = t; e < nx; e += T) {
        const int qo = e / m, j = e - qo * m, hi = j / L, k = j - hi * L;
        // exponent of term q: q (k ts + qo m) mod nx
        int step = k * ts + qo * m;
        if (step >= nx) step -= nx;
        double2 acc = in[j];
        int idx = 0;
        for (int q = 1; q < r; ++q) {
            idx += step;
            if (idx >= nx) idx -= nx;
            acc = cadd(acc, cmul(in[j + q * m], root<INV>(tw, idx)));
        }
        out[hi * L * r + k + qo * L] = acc;
    }
}

// Transform of nx points in a (b: the other buffer) by threads t < T of a group,
// natural order in and out; returns the buffer that holds the result.  Every
// thread of the block calls it, with the same nx.
template <bool INV>
__device__ double2 *mixed_fft(double2 *a, double2 *b, int nx, const Radices &f, const double2 *__restrict__ tw, int t,
                              int T, int ns) {
    int L = 1;
    for (int i = 0; i < f.n; ++i) {
        const int r = f.r[i];
        fft16::rows_sync(ns);
        switch (r) {
            case 2: radix_pass<INV, 2>(a, b, nx, L, tw, t, T); break;
            case 3: radix_pass<INV, 3>(a, b, nx, L, tw, t, T); break;
            case 4: radix_pass<INV, 4>(a, b, nx, L, tw, t, T); break;
            case 5: radix_pass<INV, 5>(a, b, nx, L, tw, t, T); break;
            default: prime_pass<INV>(a, b, nx, L, r, tw, t, T); break;
        }
        double2 *swap = a;
        a = b;
        b = swap;
        L *= r;
    }
    fft16::rows_sync(ns);
    return a;
}

// The same for a prime nx by itself: the one pass of nx terms.  In the mixed form's
// kernel it took that kernel's registers (64 a thread against 40) and with them a
// second wave of blocks: 257 x 1200 237 us a step against 191 (B200).
template <bool INV>
__device__ __forceinline__ double2 *prime_fft(const double2 *in, double2 *out, int nx, const double2 *__restrict__ tw, int t,
                                              int T) {
    __syncthreads();
    for (int m = t; m < nx; m += T) {
        double2 acc = in[0];
        int idx = 0;
        for (int q = 1; q < nx; ++q) {
            idx += m;
            if (idx >= nx) idx -= nx;
            acc = cadd(acc, cmul(in[q], root<INV>(tw, idx)));
        }
        out[m] = acc;
    }
    __syncthreads();
    return out;
}
template <bool INV, bool PRIME>
__device__ __forceinline__ double2 *any_fft(double2 *a, double2 *b, int nx, const Radices &f, const double2 *__restrict__ tw,
                                            int t, int T, int ns) {
    if constexpr (PRIME) return prime_fft<INV>(a, b, nx, tw, t, T);
    else return mixed_fft<INV>(a, b, nx, f, tw, t, T, ns);
}

// Pass A of any length: row pair (2 pair + 1, 2 pair + 2) of the right-hand side
// -> spectra, by threads t < T of a group (z: 2 nx points of shared memory).
template <bool PRIME = false>
__device__ __forceinline__ void fwd_rows_any_len(const PoissonPlan &pp, const Radices &f, const double *rhs,
                                                 int nxp, int pair, bool live, double2 *z0, int t, int T, int ns = 0) {
    const int nx = pp.nx, j0 = 2 * pair, j1 = j0 + 1;
    const bool two = live && j1 < pp.n;
    const double *r0 = rhs + (size_t)(j0 + 1) * nxp;
    const double *r1 = rhs + (size_t)(j1 + 1) * nxp;
    for (int x = t; x < nx; x += T) z0[x] = make_double2(live ? ld_fresh(r0 + x) : 0.0, two ? ld_fresh(r1 + x) : 0.0);
    const double2 *z = any_fft<false, PRIME>(z0, z0 + nx, nx, f, pp.tw, t, T, ns);
    if (!live) return;
    // unpack the two real-input spectra: A = (Z[m] + conj Z[-m])/2, B = (Z[m] - conj Z[-m])/(2i)
    double2 *s0 = pp.spec + (size_t)j0 * pp.mp, *s1 = pp.spec + (size_t)j1 * pp.mp;
    for (int m = t; m <= nx / 2; m += T) {
        const double2 a = z[m], b = cconj(z[m == 0 ? 0 : nx - m]);
        s0[m] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y + b.y));
        if (two) s1[m] = make_double2(0.5 * (a.y - b.y), -0.5 * (a.x - b.x));
    }
}

template <bool PRIME>
__global__ void __launch_bounds__(PTPB)
fwd_rows(const PoissonPlan pp, const Radices f, const double *rhs, int nxp) {
    extern __shared__ double2 sm[];
    pdl_wait();
    fwd_rows_any_len<PRIME>(pp, f, rhs, nxp, blockIdx.x, true, sm, threadIdx.x, blockDim.x);
}

// Pass B: one thread per x-mode, Thomas sweep over the n interior rows.
// piv[j][m] = 1/(b_m - piv[j-1][m]) with b_m = -(2 + kx_m^2 dy^2).
__global__ void __launch_bounds__(PTPB) tridiag(const PoissonPlan pp) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_wait();
    if (m > pp.nx / 2) return;
    const size_t mp = pp.mp;
    double2 *col = pp.spec + m;
    const double *pv = pp.piv + m;
    const double dy2 = pp.dy2;
    double2 d = make_double2(0.0, 0.0);
    for (int j = 0; j < pp.n; ++j) {
        const double2 sj = col[j * mp];
        const double c = __ldg(pv + j * mp);
        d = make_double2((dy2 * sj.x - d.x) * c, (dy2 * sj.y - d.y) * c);
        col[j * mp] = d;
    }
    double2 xn = d;
    for (int j = pp.n - 2; j >= 0; --j) {
        const double2 dj = col[j * mp];
        const double c = __ldg(pv + j * mp);
        xn = make_double2(dj.x - c * xn.x, dj.y - c * xn.y);
        col[j * mp] = xn;
    }
}

// Wall rows psi[0] = zlo, psi[ny-1] = zhi (odd_extract, poisson.cu:297-304),
// spread over the nb blocks of one channel's inverse pass (lb = this block's
// index among them, bs threads a block) and issued at the start of the
// pass: one block writing both rows alone made a chain of dependent loads
// that outlasted the rest of the pass.
__device__ __forceinline__ void write_walls(double *__restrict__ psi, const double *__restrict__ zlo,
                                            const double *__restrict__ zhi, int nx, int ny, int nxp, int lb,
                                            int nb, int bs) {
    double *lo = psi, *hi = psi + (size_t)(ny - 1) * nxp;
    for (int g = lb * bs + (int)threadIdx.x; g < 2 * nx; g += nb * bs) {
        if (g < nx) lo[g] = __ldg(zlo + g);
        else hi[g - nx] = __ldg(zhi + g - nx);
    }
}

// Pass C of any length: spectra of a row pair -> psi rows.
template <bool PRIME = false>
__device__ __forceinline__ void inv_rows_any_len(const PoissonPlan &pp, const Radices &f, int nxp, double *__restrict__ psi,
                                                 int pair, bool live, double2 *z0, int t, int T, int ns = 0) {
    const int nx = pp.nx, j0 = 2 * pair, j1 = j0 + 1;
    const bool two = live && j1 < pp.n;
    const double2 *s0 = pp.spec + (size_t)j0 * pp.mp, *s1 = pp.spec + (size_t)j1 * pp.mp;
    for (int m = t; m <= nx / 2; m += T) {
        const double2 a = live ? s0[m] : make_double2(0.0, 0.0);
        const double2 b = two ? s1[m] : make_double2(0.0, 0.0);
        // Z[m] = A + iB, Z[-m] = conj(A) + i conj(B)
        z0[m] = make_double2(a.x - b.y, a.y + b.x);
        if (m != 0 && 2 * m != nx) z0[nx - m] = make_double2(a.x + b.y, -a.y + b.x);
    }
    const double2 *z = any_fft<true, PRIME>(z0, z0 + nx, nx, f, pp.tw, t, T, ns);
    if (!live) return;
    const double inv = 1.0 / (double)nx;
    double *p0 = psi + (size_t)(j0 + 1) * nxp, *p1 = psi + (size_t)(j1 + 1) * nxp;
    for (int x = t; x < nx; x += T) {
        p0[x] = z[x].x * inv;
        if (two) p1[x] = z[x].y * inv;
    }
}

template <bool PRIME>
__global__ void __launch_bounds__(PTPB)
inv_rows(const PoissonPlan pp, const Radices f, const Chan c, double *__restrict__ psi) {
    extern __shared__ double2 sm[];
    pdl_wait();
    write_walls(psi, c.zlo, c.zhi, pp.nx, c.ny, c.nxp, blockIdx.x, gridDim.x, blockDim.x);
    inv_rows_any_len<PRIME>(pp, f, c.nxp, psi, blockIdx.x, true, sm, threadIdx.x, blockDim.x);
}

// ---- radix-16 row transforms (power-of-two nx >= 16) -----------------------
//
// Compiled per size K = log2 nx (ek_fft16.cuh), T = nx/16 threads a row pair.
// Blocks are small -- 64 threads up to nx = 1024, else one row pair -- so that
// a channel of a hundred rows spreads over the GPU: with 256 threads a block,
// 256 x 128 ran on 4 SMs (FP64: 14 us forward, 11 us inverse) and 512 x 203 on
// 13 (FP32: 8.5 and 7.6 us).
// Shared memory asked for, in percent of the largest share: room for the blocks
// that the registers allow (128 KB at 4096 and 8192), the rest of the SM's memory
// left to L1 for the twiddles.  With all of it a pass of 10 steps took 2.5 % longer on
// B200 at 4096 x 1024 FP64 (4.45 ms against 4.33) and at 8192 x 2048 FP32 (9.13
// against 8.90).
constexpr int ROW_SMEM_PERCENT = 60;

template <int K> struct RowCfg {
    static constexpr int N = 1 << K, T = N >> 4;
    static constexpr int block = T <= 64 ? 64 : T;  // threads
    static constexpr int per = block / T;           // row pairs a block
};
#define EK_ROW_CASES(F) F(4) F(5) F(6) F(7) F(8) F(9) F(10) F(11) F(12) F(13)

// Pass A, FP64, of the row pairs pair_base + p (p: the transform's index in the
// block) below pair_end: right-hand side -> spectra.  The first radix-16 pass
// runs on the values as loaded.
template <int K>
__device__ __forceinline__ void fwd_rows_f64_k(const PoissonPlan &pp, const double *rhs, int nxp, int pair_base,
                                               int pair_end, double2 *sm, int ns = 0) {
    using S = fft16::Shape<K>;
    constexpr int N = S::N, T = S::T;
    const int p = threadIdx.x / T, t = threadIdx.x - p * T;
    double2 *s = sm + p * N;
    const int pair = pair_base + p, j0 = 2 * pair, j1 = j0 + 1;
    const bool live = pair < pair_end, two = live && j1 < pp.n;
    const double *r0 = rhs + (size_t)(j0 + 1) * nxp + t, *r1 = r0 + nxp;
    double2 x[16];
#pragma unroll
    for (int v = 0; v < 16; ++v) x[v] = make_double2(live ? ld_fresh(r0 + v * T) : 0.0, two ? ld_fresh(r1 + v * T) : 0.0);
    fft16::fwd_pass_store<K, 1>(x, s, t, p, pp.tw);
    fft16::rows_sync(ns);
    fft16::fwd_rest<K, 2>(s, t, p, pp.tw, ns);
    if (!live) return;
    double2 *s0 = pp.spec + (size_t)j0 * pp.mp, *s1 = pp.spec + (size_t)j1 * pp.mp;
    for (int m = t; m <= N / 2; m += T) {
        const double2 a = s[fft16::swz_base(brev(m, K), p)];
        const double2 b = cconj(s[fft16::swz_base(brev((N - m) & (N - 1), K), p)]);
        s0[m] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y + b.y));
        if (two) s1[m] = make_double2(0.5 * (a.y - b.y), -0.5 * (a.x - b.x));
    }
}

// Pass C, FP64: spectra -> psi rows (stored from registers by the last
// radix-16 pass).
template <int K>
__device__ __forceinline__ void inv_rows_f64_k(const PoissonPlan &pp, int nxp, double *__restrict__ psi, int pair_base,
                                               int pair_end, double2 *sm, int ns = 0) {
    using S = fft16::Shape<K>;
    constexpr int N = S::N, T = S::T;
    const int p = threadIdx.x / T, t = threadIdx.x - p * T;
    double2 *s = sm + p * N;
    const int pair = pair_base + p, j0 = 2 * pair, j1 = j0 + 1;
    const bool live = pair < pair_end, two = live && j1 < pp.n;
    const double2 *s0 = pp.spec + (size_t)j0 * pp.mp, *s1 = pp.spec + (size_t)j1 * pp.mp;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const int m = t + i * T;
        if (i == 8 && t != 0) break;
        const double2 a = live ? s0[m] : make_double2(0.0, 0.0), b = two ? s1[m] : make_double2(0.0, 0.0);
        s[fft16::swz_base(brev(m, K), p)] = make_double2(a.x - b.y, a.y + b.x);  // A + iB
        if (m != 0 && 2 * m != N) s[fft16::swz_base(brev(N - m, K), p)] = make_double2(a.x + b.y, -a.y + b.x);
    }
    fft16::rows_sync(ns);
    fft16::inv_partial<K>(s, t, p, ns);
    fft16::inv_full<K, S::NF>(s, t, p, pp.tw, ns);
    double2 x[16];
    fft16::inv_pass_load<K, 1>(x, s, t, p, pp.tw);
    if (!live) return;
    constexpr double inv = 1.0 / (double)N;
    double *p0 = psi + (size_t)(j0 + 1) * nxp + t, *p1 = p0 + nxp;
#pragma unroll
    for (int v = 0; v < 16; ++v) {
        p0[v * T] = x[v].x * inv;
        if (two) p1[v * T] = x[v].y * inv;
    }
}

template <int K>
__global__ void __launch_bounds__(RowCfg<K>::block, 512 / RowCfg<K>::block)
fwd_rows_f64(const PoissonPlan pp, const double *rhs, int nxp) {
    extern __shared__ double2 sm[];
    pdl_wait();
    fwd_rows_f64_k<K>(pp, rhs, nxp, blockIdx.x * RowCfg<K>::per, (pp.n + 1) / 2, sm);
}

template <int K>
__global__ void __launch_bounds__(RowCfg<K>::block, 512 / RowCfg<K>::block)
inv_rows_f64(const PoissonPlan pp, const Chan c, double *__restrict__ psi) {
    extern __shared__ double2 sm[];
    pdl_wait();
    write_walls(psi, c.zlo, c.zhi, pp.nx, c.ny, c.nxp, blockIdx.x, gridDim.x, blockDim.x);
    inv_rows_f64_k<K>(pp, c.nxp, psi, blockIdx.x * RowCfg<K>::per, (pp.n + 1) / 2, sm);
}

// ---- FP32 form of passes A and C ------------------------------------------
// The row is split into its mean (FP64: the zero mode) and the fluctuation
// about it, which is transformed in FP32.  The zero mode of every row is
// kept in column 0 of the FP64 spectrum; modes 1..nx/2 go to the FP32
// spectrum.

// Sum of v over the T threads of one transform group (T a power of two,
// groups contiguous in the block); every thread of the block calls it and
// gets the group's first lane's (or the block-level) value.
template <int BLOCK>
__device__ __forceinline__ double group_sum(double v, int T, double *red, int ns = 0) {
    const int w = T < 32 ? T : 32;
    for (int o = w >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (T < 32) return __shfl_sync(0xffffffffu, v, (threadIdx.x & 31) & ~(T - 1));
    v = __shfl_sync(0xffffffffu, v, 0);
    if (T == 32) return v;
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    fft16::rows_sync(ns);
    const int nw = T >> 5, g0 = (int)(threadIdx.x / T) * nw;
    double s = 0.0;
    for (int i = 0; i < nw; ++i) s += red[g0 + i];
    fft16::rows_sync(ns);
    return s;
}

// Pass A of the FP32 form for 2^K-point rows: the FP64 row sums (the zero
// mode) and the FP32 transform of the fluctuation about an offset (it only
// moves the unused FP32 zero bin; a close one keeps the rounding small).
// A row's right-hand side is rhsf plus, in FP64, the row constant: rhs_q
// (R+ - R-) of the row references and, on rows 1 and ny-2, the x-mean of the
// Dirichlet lifting -zeta/dy^2 (odd_extension, poisson.cu:228-241; its
// x-fluctuation is in rhsf).
// From the second solve on the offset is the previous solve's row mean and
// one pass over the row does both; the first solve takes two passes and the
// exact mean.  The first radix-16 pass runs on the values as loaded.
template <int BLOCK, int K>
__device__ __forceinline__ void fwd_rows_f32_k(const PoissonPlan &pp, const Chan &c, int pair_base, int pair_end,
                                               float2 *sm, double *red, int ns = 0) {
    using S = fft16::Shape<K>;
    constexpr int N = S::N, T = S::T;
    const int p = threadIdx.x / T, t = threadIdx.x - p * T;
    const int pair = pair_base + p;
    float2 *s = sm + p * N;
    const int j0 = 2 * pair, j1 = j0 + 1;
    const bool live = pair < pair_end, two = live && j1 < pp.n;
    const int nxp = c.nxp;
    // 32-bit offsets from the planes' base pointers (a plane is below 2^32
    // elements: one channel's planes fit device memory)
    const unsigned r0 = (unsigned)(j0 + 1) * (unsigned)nxp + (unsigned)t, r1 = r0 + (unsigned)nxp;
    const double k0 = live ? rhs_row_constant(pp, c, j0 + 1) : 0.0, k1 = two ? rhs_row_constant(pp, c, j1 + 1) : 0.0;
    const bool exact = *pp.rowmean_ok == 0;  // the same for every block of the launch
    // value - offset = rhsf + (row constant - offset), rounded once
    double d0 = (live && !exact) ? k0 - pp.rowmean[j0] : 0.0, d1 = (two && !exact) ? k1 - pp.rowmean[j1] : 0.0;
    double a0 = 0.0, a1 = 0.0;
    float2 x[16];
    if constexpr (T == 1) {  // a row a thread: 16 consecutive values
        const float4 *q0 = reinterpret_cast<const float4 *>(pp.rhsf + r0), *q1 = reinterpret_cast<const float4 *>(pp.rhsf + r1);
        const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const float4 u = live ? ld_fresh(q0 + v) : none, w = two ? ld_fresh(q1 + v) : none;
            x[4 * v] = make_float2(u.x, w.x);
            x[4 * v + 1] = make_float2(u.y, w.y);
            x[4 * v + 2] = make_float2(u.z, w.z);
            x[4 * v + 3] = make_float2(u.w, w.w);
        }
    } else {
#pragma unroll
        for (int v = 0; v < 16; ++v)
            x[v] = make_float2(live ? ld_fresh(pp.rhsf + (r0 + (unsigned)(v * T))) : 0.0f,
                               two ? ld_fresh(pp.rhsf + (r1 + (unsigned)(v * T))) : 0.0f);
    }
    auto less_offset = [&](bool sum) {
#pragma unroll
        for (int v = 0; v < 16; ++v) {
            const double f0 = (double)x[v].x, f1 = (double)x[v].y;
            if (sum) {
                a0 += f0;
                a1 += f1;
            }
            x[v] = make_float2((float)(f0 + d0), (float)(f1 + d1));
        }
    };
    if (exact) {
#pragma unroll
        for (int v = 0; v < 16; ++v) {
            a0 += (double)x[v].x;
            a1 += (double)x[v].y;
        }
    } else {
        less_offset(true);
    }
    a0 = group_sum<BLOCK>(a0, T, red, ns) + (double)N * k0;
    a1 = group_sum<BLOCK>(a1, T, red, ns) + (double)N * k1;
    if (exact) {
        d0 = live ? k0 - a0 / (double)N : 0.0;
        d1 = two ? k1 - a1 / (double)N : 0.0;
        less_offset(false);
    }
    if (t == 0 && live) {
        pp.spec[(size_t)j0 * pp.mp] = make_double2(a0, 0.0);
        pp.rowmean[j0] = a0 / (double)N;
        if (two) {
            pp.spec[(size_t)j1 * pp.mp] = make_double2(a1, 0.0);
            pp.rowmean[j1] = a1 / (double)N;
        }
    }
    fft16::fwd_pass_store<K, 1>(x, s, t, p, pp.twf);
    fft16::rows_sync(ns);
    fft16::fwd_rest<K, 2>(s, t, p, pp.twf, ns);
    if (!live) return;
    const unsigned q0 = (unsigned)j0 * (unsigned)pp.mp, q1 = q0 + (unsigned)pp.mp;
    auto mode = [&](int m, float2 *A, float2 *B) {
        const float2 a = s[fft16::swz_base(brev(m, K), p)], b = cconj(s[fft16::swz_base(brev(N - m, K), p)]);
        *A = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y + b.y));
        *B = make_float2(0.5f * (a.y - b.y), -0.5f * (a.x - b.x));
    };
    if constexpr (T == 1) {  // modes 0 (not used: zero) to 8 of a row, in 16-byte stores
        float2 A[9], B[9];
        A[0] = B[0] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int m = 1; m <= 8; ++m) mode(m, &A[m], &B[m]);
#pragma unroll
        for (int m = 0; m < 8; m += 2) {
            *reinterpret_cast<float4 *>(pp.specf + (q0 + m)) = make_float4(A[m].x, A[m].y, A[m + 1].x, A[m + 1].y);
            if (two) *reinterpret_cast<float4 *>(pp.specf + (q1 + m)) = make_float4(B[m].x, B[m].y, B[m + 1].x, B[m + 1].y);
        }
        pp.specf[q0 + 8] = A[8];
        if (two) pp.specf[q1 + 8] = B[8];
    } else {
        for (int m = t; m <= N / 2; m += T) {
            if (m == 0) continue;
            float2 A, B;
            mode(m, &A, &B);
            pp.specf[q0 + (unsigned)m] = A;
            if (two) pp.specf[q1 + (unsigned)m] = B;
        }
    }
}

// Wall rows of the FP32 form's psi: psim = the x-mean of the wall potential,
// psif = the potential minus it (zero for uniform walls), the FP64 plane's
// Dirichlet values too when write_f64; spread over the nb blocks of the pass.
__device__ __forceinline__ void write_walls_f32(const PoissonPlan &pp, const Chan &c, double *__restrict__ psi,
                                                bool write_f64, int lb, int nb, int bs) {
    const int nx = c.nx, ny = c.ny;
    float *flo = pp.psif, *fhi = pp.psif + (size_t)(ny - 1) * c.nxp;
    double *dlo = psi, *dhi = psi + (size_t)(ny - 1) * c.nxp;
    for (int g = lb * bs + (int)threadIdx.x; g < 2 * nx; g += nb * bs) {
        const bool low = g < nx;
        const int x = low ? g : g - nx;
        const double z = __ldg((low ? c.zlo : c.zhi) + x);
        (low ? flo : fhi)[x] = (float)(z - (low ? pp.zlo_mean : pp.zhi_mean));
        if (write_f64) (low ? dlo : dhi)[x] = z;
    }
    if (lb == 0 && threadIdx.x == 0) {
        pp.psim[0] = pp.zlo_mean;
        pp.psim[ny - 1] = pp.zhi_mean;
    }
}

// Pass C of the FP32 form: the two real rows' spectra packed as A + iB, the
// inverse transform; psif = the FP32 fluctuation / N (stored from registers by
// the last radix-16 pass), psim = the FP64 row mean, and the FP64 psi plane
// (mean + fluctuation) when write_f64.
template <int BLOCK, int K>
__device__ __forceinline__ void inv_rows_f32_k(const PoissonPlan &pp, const Chan &c, double *__restrict__ psi,
                                               bool write_f64, int pair_base, int pair_end, float2 *sm, int ns = 0) {
    using S = fft16::Shape<K>;
    constexpr int N = S::N, T = S::T;
    const int p = threadIdx.x / T, t = threadIdx.x - p * T;
    const int pair = pair_base + p;
    float2 *s = sm + p * N;
    const int j0 = 2 * pair, j1 = j0 + 1;
    const bool live = pair < pair_end, two = live && j1 < pp.n;
    const int nxp = c.nxp;
    // 32-bit offsets from the planes' base pointers (as in fwd_rows_f32_k)
    const unsigned q0 = (unsigned)j0 * (unsigned)pp.mp, q1 = q0 + (unsigned)pp.mp;
    // modes m = t + i T (i < 8) and, for t = 0, m = N/2: all loads first
    const float2 zero = make_float2(0.0f, 0.0f);
    float2 a[9], b[9];
    if constexpr (T == 1) {  // a row a thread: modes 0 (its slot holds zero) to 8
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 u = live ? *reinterpret_cast<const float4 *>(pp.specf + (q0 + i)) : none;
            const float4 w = two ? *reinterpret_cast<const float4 *>(pp.specf + (q1 + i)) : none;
            a[i] = i ? make_float2(u.x, u.y) : zero;
            a[i + 1] = make_float2(u.z, u.w);
            b[i] = i ? make_float2(w.x, w.y) : zero;
            b[i + 1] = make_float2(w.z, w.w);
        }
        a[8] = live ? pp.specf[q0 + 8] : zero;
        b[8] = two ? pp.specf[q1 + 8] : zero;
    } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const int m = t + i * T;
            const bool in = i < 8 || t == 0;
            a[i] = (live && in && m) ? pp.specf[q0 + (unsigned)m] : zero;
            b[i] = (two && in && m) ? pp.specf[q1 + (unsigned)m] : zero;
        }
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const int m = t + i * T;
        if (i == 8 && t != 0) break;
        s[fft16::swz_base(brev(m, K), p)] = make_float2(a[i].x - b[i].y, a[i].y + b[i].x);  // A + iB
        if (m != 0 && 2 * m != N)
            s[fft16::swz_base(brev(N - m, K), p)] = make_float2(a[i].x + b[i].y, -a[i].y + b[i].x);
    }
    fft16::rows_sync(ns);
    fft16::inv_partial<K>(s, t, p, ns);
    fft16::inv_full<K, S::NF>(s, t, p, pp.twf, ns);
    float2 x[16];
    fft16::inv_pass_load<K, 1>(x, s, t, p, pp.twf);
    const double inv = 1.0 / (double)N;
    const float invf = 1.0f / (float)N;  // a power of two: exact
    if (pair_base == 0 && threadIdx.x == 0) *pp.rowmean_ok = 1;
    if (live) {
        const double mean0 = pp.spec[(size_t)j0 * pp.mp].x * inv;
        const double mean1 = two ? pp.spec[(size_t)j1 * pp.mp].x * inv : 0.0;
        if (t == 0) {
            pp.psim[j0 + 1] = mean0;
            if (two) pp.psim[j1 + 1] = mean1;
        }
        const unsigned o0 = (unsigned)(j0 + 1) * (unsigned)nxp + (unsigned)t, o1 = o0 + (unsigned)nxp;
        if constexpr (T == 1) {
#pragma unroll
            for (int v = 0; v < 16; v += 4) {
                st_field_f4(pp.psif + (o0 + v), make_float4(x[v].x * invf, x[v + 1].x * invf, x[v + 2].x * invf, x[v + 3].x * invf),
                            pp.keep_l2);
                if (two)
                    st_field_f4(pp.psif + (o1 + v),
                                make_float4(x[v].y * invf, x[v + 1].y * invf, x[v + 2].y * invf, x[v + 3].y * invf), pp.keep_l2);
            }
        }
#pragma unroll
        for (int v = 0; v < 16; ++v) {
            const float y0 = x[v].x * invf, y1 = x[v].y * invf;
            const unsigned dv = (unsigned)(v * T);
            if constexpr (T > 1) {
                st_field_f(pp.psif + (o0 + dv), y0, pp.keep_l2);
                if (two) st_field_f(pp.psif + (o1 + dv), y1, pp.keep_l2);
            }
            if (write_f64) {
                psi[o0 + dv] = mean0 + (double)y0;
                if (two) psi[o1 + dv] = mean1 + (double)y1;
            }
        }
    }
}

// Pass A and C of a single channel, compiled per size; 1024 threads an SM (64
// registers a thread hold the 16 points of a transform).
template <int K>
__global__ void __launch_bounds__(RowCfg<K>::block, 1024 / RowCfg<K>::block)
fwd_rows_f32(const PoissonPlan pp, const Chan c) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[(RowCfg<K>::block + 31) / 32];
    pdl_wait();
    fwd_rows_f32_k<RowCfg<K>::block, K>(pp, c, blockIdx.x * RowCfg<K>::per, (pp.n + 1) / 2, (float2 *)smraw, red);
}

template <int K>
__global__ void __launch_bounds__(RowCfg<K>::block, 1024 / RowCfg<K>::block)
inv_rows_f32(const PoissonPlan pp, const Chan c, double *__restrict__ psi, bool write_f64) {
    extern __shared__ __align__(16) unsigned char smraw[];
    pdl_wait();
    write_walls_f32(pp, c, psi, write_f64, blockIdx.x, gridDim.x, blockDim.x);
    inv_rows_f32_k<RowCfg<K>::block, K>(pp, c, psi, write_f64, blockIdx.x * RowCfg<K>::per, (pp.n + 1) / 2, (float2 *)smraw);
}

// Sizes that a batch block of BLOCK threads runs, whole transforms only.
template <int BLOCK, int K> __host__ __device__ constexpr bool batch_fits() { return ((1 << K) >> 4) <= BLOCK && K <= 12; }

template <int BLOCK>
__device__ __forceinline__ void fwd_rows_any(const PoissonPlan &pp, const Chan &c, int pair_base, float2 *sm, double *red) {
    switch (pp.log2nx) {
#define EK_CASE(K)                                                                                     \
    case K:                                                                                            \
        if constexpr (batch_fits<BLOCK, K>()) fwd_rows_f32_k<BLOCK, K>(pp, c, pair_base, (pp.n + 1) / 2, sm, red); \
        break;
        EK_ROW_CASES(EK_CASE)
#undef EK_CASE
        default: break;
    }
}

template <int BLOCK>
__device__ __forceinline__ void inv_rows_any(const PoissonPlan &pp, const Chan &c, double *__restrict__ psi, bool write_f64,
                                             int pair_base, float2 *sm) {
    const int per = BLOCK / (pp.nx >> 4);
    write_walls_f32(pp, c, psi, write_f64, pair_base / per, ((pp.n + 1) / 2 + per - 1) / per, BLOCK);
    switch (pp.log2nx) {
#define EK_CASE(K)                                                                                                 \
    case K:                                                                                                        \
        if constexpr (batch_fits<BLOCK, K>())                                                                      \
            inv_rows_f32_k<BLOCK, K>(pp, c, psi, write_f64, pair_base, (pp.n + 1) / 2, sm);                        \
        break;
        EK_ROW_CASES(EK_CASE)
#undef EK_CASE
        default: break;
    }
}

// ---- pass B, partitioned Thomas solve ------------------------------------
//
// A block owns M consecutive x-modes; its 512 threads are S = 512/M row
// segments x M modes, each segment at most 16 rows (M is chosen so), held in
// registers with its pivots.  The forward recurrence
// d_j = (dy^2 S_j - d_{j-1}) piv_j is linear in the value entering a segment,
// so each segment first runs with a zero entry value while accumulating the
// product of (-piv); the true entry values follow from composing the
// segments' affine maps D -> e + f D in order (seg_carry), and each segment
// adds its correction.  The backward recurrence x_j = d_j - piv_j x_{j+1} is split the
// same way.  The result is the Thomas solution, reassociated.
constexpr int TB_THREADS = 512;
constexpr int TB_L = 16;

constexpr int TB_WARPS = TB_THREADS / 32;
constexpr int TB_MODES = 16;      // most modes a block, FP64
constexpr int TB_MODES_F32 = 8;   // FP32

// Shared memory of the carries.  FP64: composite maps of each warp's segments,
// per mode, one set for each sweep.  FP32: the segments' maps, two sets used in
// turn by the scan's rounds.
struct TridiagShared {
    double2 ends[2][TB_WARPS][TB_MODES];
    double mults[2][TB_WARPS][TB_MODES];
};
struct TridiagSharedF {
    float2 ends[2][TB_THREADS];
    float mults[2][TB_THREADS];
};
template <typename R> struct SharedOf;
template <> struct SharedOf<double> { using type = TridiagShared; };
template <> struct SharedOf<float> { using type = TridiagSharedF; };

__device__ __forceinline__ double2 shfl_c(double2 v, int lane) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}

// Value entering this thread's segment: the affine maps D -> e + f D of the
// segments of its mode (the block's threads are seg * M + mode) composed in
// order -- forward from segment 0 (FWD) or backward from segment S-1; the
// first segment in that order enters with 0.  A warp composes its 32/M
// segments by shuffles and leaves its total in shared memory; after one barrier
// each thread runs through the totals of the warps before its own (15 at most).
// (A Kogge-Stone scan of all segments in shared memory, two barriers a round:
// 6.7 us a launch at 256 x 128 FP64 on B200 against 5.6, 22.3 against 17.7 at
// 4096 x 1024.)  Every thread of the block calls it.
template <bool FWD>
__device__ __forceinline__ double2 seg_carry(double2 e, double f, int M, TridiagShared &sh) {
    using C = double2;
    using R = double;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, mode = lane & (M - 1);
    for (int off = M; off < 32; off <<= 1) {
        const int src = FWD ? lane - off : lane + off;
        const C e2 = shfl_c(e, src & 31);
        const R f2 = __shfl_sync(0xffffffffu, f, src & 31);
        if (FWD ? src >= 0 : src < 32) {
            e = cmake<C>(e.x + f * e2.x, e.y + f * e2.y);  // this segment after the earlier ones
            f = f * f2;
        }
    }
    constexpr int set = FWD ? 0 : 1;
    if (FWD ? lane >= 32 - M : lane < M) {
        sh.ends[set][warp][mode] = e;
        sh.mults[set][warp][mode] = f;
    }
    __syncthreads();
    C D = cmake<C>(0.0, 0.0);
    if (FWD) {
        for (int w = 0; w < warp; ++w) {
            const C ew = sh.ends[set][w][mode];
            const R fw = sh.mults[set][w][mode];
            D = cmake<C>(ew.x + fw * D.x, ew.y + fw * D.y);
        }
    } else {
        for (int w = TB_WARPS - 1; w > warp; --w) {
            const C ew = sh.ends[set][w][mode];
            const R fw = sh.mults[set][w][mode];
            D = cmake<C>(ew.x + fw * D.x, ew.y + fw * D.y);
        }
    }
    // through the segments of this warp before this thread's
    const int src = FWD ? lane - M : lane + M;
    const C ep = shfl_c(e, src & 31);
    const R fp = __shfl_sync(0xffffffffu, f, src & 31);
    if (FWD ? src >= 0 : src < 32) D = cmake<C>(ep.x + fp * D.x, ep.y + fp * D.y);
    return D;
}

// The same in FP32, by a Kogge-Stone scan over the S segments in shared memory,
// one barrier a round.  (The order of the products is part of a result's
// rounding: FP16 and FP32 runs repeat earlier ones bit for bit with this one.)
template <bool FWD>
__device__ __forceinline__ float2 seg_carry(float2 e, float f, int M, TridiagSharedF &sh) {
    const int tid = threadIdx.x, S = TB_THREADS / M, seg = tid / M, mode = tid & (M - 1);
    int set = 0;
    for (int off = 1; off < S; off <<= 1, set ^= 1) {
        sh.ends[set][tid] = e;
        sh.mults[set][tid] = f;
        __syncthreads();
        const int src = FWD ? seg - off : seg + off;
        if (FWD ? src >= 0 : src < S) {
            const float2 e2 = sh.ends[set][src * M + mode];
            const float f2 = sh.mults[set][src * M + mode];
            e = make_float2(e.x + f * e2.x, e.y + f * e2.y);  // this segment after the earlier ones
            f = f * f2;
        }
    }
    sh.ends[set][tid] = e;
    __syncthreads();
    const int prev = FWD ? seg - 1 : seg + 1;
    const float2 out = (FWD ? prev >= 0 : prev < S) ? sh.ends[set][prev * M + mode] : make_float2(0.0f, 0.0f);
    __syncthreads();  // sh is written again by the next call
    return out;
}

// (v - d) c with the difference and the product rounded (d, a product itself, is
// not fused into the difference: FP32 keeps the rounding of earlier runs).
__device__ __forceinline__ float2 rn_sub_mul(float2 v, float2 d, float c) {
    return make_float2(__fmul_rn(__fsub_rn(v.x, d.x), c), __fmul_rn(__fsub_rn(v.y, d.y), c));
}
__device__ __forceinline__ double2 rn_sub_mul(double2 v, double2 d, double c) {
    return make_double2((v.x - d.x) * c, (v.y - d.y) * c);
}

// One block of the partitioned solve on a spectrum of type C (pivots R), with
// segments of at most LMAX rows.  Rows past the end carry zero pivots and values,
// which pass zero on in either direction, so the sweeps need no row test.  spec, of
// the kernel before, is not __restrict__: the wait is in here.
template <int LMAX, typename R, typename C>
__device__ __forceinline__ void tridiag_part_len(const R *__restrict__ piv, C *spec, int n, int nx,
                                                 size_t mp, R dy2, int M, int m_base, typename SharedOf<R>::type &sh) {
    const int mlast = nx / 2;
    const int tid = threadIdx.x, mode = tid & (M - 1), S = TB_THREADS / M, seg = tid / M;
    const int m = m_base + mode;
    const bool mvalid = m <= mlast;
    const int L = (n + S - 1) / S, ja = seg * L, cnt = max(0, min(n, ja + L) - ja);
    const unsigned o = (unsigned)ja * (unsigned)mp + (unsigned)m;  // n mp < 2^32 (n <= 8192)
    R c[LMAX];
    C v[LMAX];
    pdl_wait();
#pragma unroll
    for (int q = 0; q < LMAX; ++q) {
        const bool on = mvalid && q < cnt;
        c[q] = on ? __ldg(piv + (o + q * (unsigned)mp)) : R(0);
        const C sv = on ? spec[o + q * (unsigned)mp] : cmake<C>(0.0, 0.0);
        v[q] = cmake<C>(dy2 * sv.x, dy2 * sv.y);
    }
    C d = cmake<C>(0.0, 0.0);
    R mu = R(1);
#pragma unroll
    for (int q = 0; q < LMAX; ++q) {
        d = rn_sub_mul(v[q], d, c[q]);
        mu = -c[q] * mu;
        v[q] = d;
        // the segment's own end, where L < LMAX (the same for every thread)
        if (LMAX > 1 && q + 1 == L) break;
    }
    {
        const C D = seg_carry<true>(d, mu, M, sh);  // true entry value of the segment
        mu = R(1);
#pragma unroll
        for (int q = 0; q < LMAX; ++q) {
            mu = -c[q] * mu;
            v[q].x += mu * D.x;
            v[q].y += mu * D.y;
        }
    }
    C x = cmake<C>(0.0, 0.0);
    R nu = R(1);
#pragma unroll
    for (int q = LMAX - 1; q >= 0; --q) {
        if (q >= L) continue;
        x = cmake<C>(v[q].x - c[q] * x.x, v[q].y - c[q] * x.y);
        nu = -c[q] * nu;
        v[q] = x;
    }
    const C X = seg_carry<false>(x, nu, M, sh);  // true exit value of the segment (x_n = 0)
    if (!mvalid) return;
    nu = R(1);
#pragma unroll
    for (int q = LMAX - 1; q >= 0; --q) {
        if (q < cnt) {
            nu = -c[q] * nu;
            spec[o + q * (unsigned)mp] = cmake<C>(v[q].x + nu * X.x, v[q].y + nu * X.y);
        }
    }
}

// The form for the segments' length: a sweep unrolled to 16 rows costs a channel
// of 7 rows a segment more than twice its arithmetic (FP64 most of all).
template <typename R, typename C>
__device__ __forceinline__ void tridiag_part_gen(const R *__restrict__ piv, C *spec, int n, int nx,
                                                 size_t mp, R dy2, int M, int m_base, typename SharedOf<R>::type &sh) {
    const int S = TB_THREADS / M, L = (n + S - 1) / S;
    if (L <= 4) tridiag_part_len<4, R, C>(piv, spec, n, nx, mp, dy2, M, m_base, sh);
    else if (L <= 8) tridiag_part_len<8, R, C>(piv, spec, n, nx, mp, dy2, M, m_base, sh);
    else tridiag_part_len<TB_L, R, C>(piv, spec, n, nx, mp, dy2, M, m_base, sh);
}

__device__ __forceinline__ void tridiag_part_dev(const PoissonPlan &pp, int M, int m_base, TridiagShared &sh) {
    tridiag_part_gen<double, double2>(pp.piv, pp.spec, pp.n, pp.nx, (size_t)pp.mp, pp.dy2, M, m_base, sh);
}

__global__ void __launch_bounds__(TB_THREADS) tridiag_part(const PoissonPlan pp, int M) {
    __shared__ TridiagShared sh;
    tridiag_part_dev(pp, M, blockIdx.x * M, sh);
}

// Shared memory of the FP32 form's column kernel: the FP32 modes' segment
// ends, or the zero mode's per-warp scan totals.
union ColumnShared {
    TridiagSharedF f;
    double wtot[TB_THREADS / 32];
};

// Inclusive sum of v over threads 0..threadIdx.x of the block (TB_THREADS
// threads): warp shuffles, then the warp totals in shared memory.  Every
// thread of the block calls it; *total gets the block's sum.
__device__ __forceinline__ double block_scan(double v, ColumnShared &sh, double *total) {
    constexpr int NW = TB_THREADS / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += t;
    }
    if (lane == 31) sh.wtot[w] = v;
    __syncthreads();
    if (w == 0) {
        double t = lane < NW ? sh.wtot[lane] : 0.0;
#pragma unroll
        for (int off = 1; off < NW; off <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, t, off);
            if (lane >= off) t += u;
        }
        if (lane < NW) sh.wtot[lane] = t;
    }
    __syncthreads();
    if (w > 0) v += sh.wtot[w - 1];
    *total = sh.wtot[NW - 1];
    __syncthreads();  // sh is written again by the next call
    return v;
}

// The zero mode (kx = 0) of the FP32 form's column solve in FP64, by one
// block.  Its system phi_{j-1} - 2 phi_j + phi_{j+1} = h_j, h_j = dy^2 S_j
// (S_j: the row sums in column 0 of the FP64 spectrum), phi_{-1} = phi_n = 0,
// is solved exactly by two prefix sums: with H_k = h_0 + ... + h_k,
//     phi_j = (j + 1) g_0 + (H_0 + ... + H_{j-1}),  g_0 = -(H_0 + ... + H_{n-1}) / (n + 1)
// (g_j = phi_j - phi_{j-1} steps by h_j).  Thread t owns rows [t L, t L + L),
// L = ceil(n / TB_THREADS), and reads them three times (the later reads hit
// L1), so the block holds no per-row registers and fits the FP32 kernel's
// budget; the two sums over the threads are block scans.
__device__ __forceinline__ void zero_mode_f64(const PoissonPlan &pp, ColumnShared &sh) {
    const int n = pp.n, L = (n + TB_THREADS - 1) / TB_THREADS;
    const int ja = (int)threadIdx.x * L, cnt = max(0, min(n, ja + L) - ja);
    const size_t stride = 2 * (size_t)pp.mp;  // element j of the column at col[j * stride]
    double *col = &pp.spec[0].x;
    const double dy2 = pp.dy2;
    pdl_wait();
    // segment sum of h, then H at the segment's start
    double s1 = 0.0;
    for (int q = 0; q < cnt; ++q) s1 += dy2 * col[(size_t)(ja + q) * stride];
    double tot;
    const double h0 = block_scan(s1, sh, &tot) - s1;  // H_{ja - 1}
    // segment sum of H, then the sum of H before the segment and over all rows
    double H = h0, s2 = 0.0;
    for (int q = 0; q < cnt; ++q) {
        H += dy2 * col[(size_t)(ja + q) * stride];
        s2 += H;
    }
    double S;
    const double G0 = block_scan(s2, sh, &S) - s2;  // H_0 + ... + H_{ja - 1}
    const double g0 = -S / (double)(n + 1);
    H = h0;
    double G = G0;
    for (int q = 0; q < cnt; ++q) {
        const int j = ja + q;
        const double hj = dy2 * col[(size_t)j * stride];
        col[(size_t)j * stride] = (double)(j + 1) * g0 + G;
        H += hj;
        G += H;
    }
}

// Pass B of the FP32 form in one kernel: block 0 solves the zero mode in
// FP64 (zero_mode_f64), blocks 1.. the modes 1..nx/2 in FP32, M per block,
// two blocks per SM.
__global__ void __launch_bounds__(TB_THREADS, 2) tridiag_modes_f32(const PoissonPlan pp, int M) {
    __shared__ ColumnShared sh;
    if (blockIdx.x == 0) {
        zero_mode_f64(pp, sh);
        return;
    }
    tridiag_part_gen<float, float2>(pp.pivf, pp.specf, pp.n, pp.nx, (size_t)pp.mp, (float)pp.dy2, M,
                                    1 + (blockIdx.x - 1) * M, sh.f);
}

// ---- a small channel's whole solve in one launch ------------------------------
//
// One cluster of up to 16 blocks runs passes A, B and C with the cluster's
// barrier between them: three launches' boundaries cost a channel of a thousand
// nodes more than the passes' work.  Each block takes an equal share of
// the row pairs, then every gridDim.x-th group of modes; the spectrum goes
// through L2.  The arithmetic is that of the separate passes, group for group, so
// the bits are theirs.  On larger channels 16 SMs are too few
// (poisson_cluster_blocks has the line and both sides).
constexpr int CL_THREADS = TB_THREADS;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

union ClusterShared {
    ColumnShared col;
    TridiagShared col64;
    double red[CL_THREADS / 32];
};

// Row pairs a block takes per round: as many as its threads hold, fewer where
// the channel's pairs then spread over all blocks.
__device__ __forceinline__ int cluster_share(int pairs, int per) {
    const int k = (pairs + (int)gridDim.x - 1) / (int)gridDim.x;
    return k < per ? k : per;
}

// Threads of the whole warps that `live` threads fill.
__device__ __forceinline__ int rows_threads(int live) { return (live + 31) & ~31; }

template <int K>
__global__ void __launch_bounds__(CL_THREADS, 1)
solve_cluster_f32(const PoissonPlan pp, const Chan c, double *__restrict__ psi, bool write_f64, int M) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ ClusterShared sh;
    float2 *sm = (float2 *)smraw;
    pdl_wait();
    const int b = blockIdx.x, nb = gridDim.x, pairs = (pp.n + 1) / 2;
    const int k = cluster_share(pairs, CL_THREADS / fft16::Shape<K>::T);
    const int ns = rows_threads(k * fft16::Shape<K>::T);  // warps without a row pair take no part
    if ((int)threadIdx.x < ns)
        for (int p0 = b * k; p0 < pairs; p0 += nb * k) {
            fwd_rows_f32_k<CL_THREADS, K>(pp, c, p0, min(pairs, p0 + k), sm, sh.red, ns);
            fft16::rows_sync(ns);
        }
    cluster_barrier();
    const int groups = 1 + (pp.nx / 2 + M - 1) / M;
    for (int g = b; g < groups; g += nb) {
        if (g == 0) zero_mode_f64(pp, sh.col);
        else
            tridiag_part_gen<float, float2>(pp.pivf, pp.specf, pp.n, pp.nx, (size_t)pp.mp, (float)pp.dy2, M, 1 + (g - 1) * M,
                                            sh.col.f);
        __syncthreads();
    }
    cluster_barrier();
    write_walls_f32(pp, c, psi, write_f64, b, nb, CL_THREADS);
    if ((int)threadIdx.x < ns)
        for (int p0 = b * k; p0 < pairs; p0 += nb * k) {
            inv_rows_f32_k<CL_THREADS, K>(pp, c, psi, write_f64, p0, min(pairs, p0 + k), sm, ns);
            fft16::rows_sync(ns);
        }
}

// FP64: K = 4 for nx = 16 (radix-16 transforms), 0 for the mixed lengths (T threads a
// row pair).
template <int K>
__global__ void __launch_bounds__(CL_THREADS, 1)
solve_cluster_f64(const PoissonPlan pp, const Radices f, int T, const Chan c, const double *rhs,
                  double *__restrict__ psi, int M) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ ClusterShared sh;
    double2 *sm = (double2 *)smraw;
    pdl_wait();
    const int b = blockIdx.x, nb = gridDim.x, pairs = (pp.n + 1) / 2;
    const int k = cluster_share(pairs, CL_THREADS / T), t = threadIdx.x % T, q = threadIdx.x / T;
    const int ns = rows_threads(k * T);  // warps without a row pair take no part
    if ((int)threadIdx.x < ns)
        for (int p0 = b * k; p0 < pairs; p0 += nb * k) {
            if constexpr (K > 0) fwd_rows_f64_k<K>(pp, rhs, c.nxp, p0, min(pairs, p0 + k), sm, ns);
            else fwd_rows_any_len(pp, f, rhs, c.nxp, p0 + q, q < k && p0 + q < pairs, sm + (size_t)q * 2 * pp.nx, t, T, ns);
            fft16::rows_sync(ns);
        }
    cluster_barrier();
    const int groups = (pp.nx / 2 + M) / M;
    for (int g = b; g < groups; g += nb) {
        tridiag_part_dev(pp, M, g * M, sh.col64);
        __syncthreads();
    }
    cluster_barrier();
    write_walls(psi, c.zlo, c.zhi, pp.nx, c.ny, c.nxp, b, nb, CL_THREADS);
    if ((int)threadIdx.x < ns)
        for (int p0 = b * k; p0 < pairs; p0 += nb * k) {
            if constexpr (K > 0) inv_rows_f64_k<K>(pp, c.nxp, psi, p0, min(pairs, p0 + k), sm, ns);
            else inv_rows_any_len(pp, f, c.nxp, psi, p0 + q, q < k && p0 + q < pairs, sm + (size_t)q * 2 * pp.nx, t, T, ns);
            fft16::rows_sync(ns);
        }
}

// ---- batched passes: one launch for many channels -------------------------
// A block's work item names its channel and its first row pair (passes A,
// C) or first x-mode (pass B); the channel's plan comes from a device table.
// Batches run the FP32 form.
// The channel's plan and constants are staged in shared memory (as a copy in
// registers they spilled 3.9 KB a thread of the forward pass).  BLOCK: 64
// threads where every channel's transform fits them (nx <= 1024), else 256.
struct RowItem {
    PoissonPlan pp;
    Chan c;
};
static_assert(sizeof(PoissonPlan) % 8 == 0 && sizeof(Chan) % 8 == 0, "copied by 8-byte words");
template <int BLOCK>
__device__ __forceinline__ void stage_item(RowItem &it, const PoissonPlan *__restrict__ plan, const Chan *__restrict__ chan) {
    for (int i = threadIdx.x; i < (int)(sizeof(PoissonPlan) / 8); i += BLOCK)
        ((unsigned long long *)&it.pp)[i] = __ldg((const unsigned long long *)plan + i);
    for (int i = threadIdx.x; i < (int)(sizeof(Chan) / 8); i += BLOCK)
        ((unsigned long long *)&it.c)[i] = __ldg((const unsigned long long *)chan + i);
    __syncthreads();
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK)
batch_fwd_rows_f32(const PoissonPlan *__restrict__ plans, const Chan *__restrict__ chans,
                   const int2 *__restrict__ items) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[BLOCK / 32];
    __shared__ __align__(16) RowItem ri;
    const int2 it = items[blockIdx.x];
    stage_item<BLOCK>(ri, plans + it.x, chans + it.x);
    fwd_rows_any<BLOCK>(ri.pp, ri.c, it.y, (float2 *)smraw, red);
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK)
batch_inv_rows_f32(const PoissonPlan *__restrict__ plans, const Chan *__restrict__ chans,
                   double *const *__restrict__ fields, const int2 *__restrict__ items, bool write_f64) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(16) RowItem ri;
    const int2 it = items[blockIdx.x];
    stage_item<BLOCK>(ri, plans + it.x, chans + it.x);
    inv_rows_any<BLOCK>(ri.pp, ri.c, fields[it.x] + F_PSI * ri.c.plane, write_f64, it.y, (float2 *)smraw);
}

// items {channel, first mode, modes per block}: FP32 mode blocks, and for
// modes per block == 0 the channel's FP64 zero mode (zero_mode_f64)
__global__ void __launch_bounds__(TB_THREADS, 2)
batch_tridiag_modes_f32(const PoissonPlan *__restrict__ plans, const int3 *__restrict__ items) {
    __shared__ ColumnShared sh;
    const int3 it = items[blockIdx.x];
    const PoissonPlan pp = plans[it.x];
    if (it.z == 0) {
        zero_mode_f64(pp, sh);
        return;
    }
    tridiag_part_gen<float, float2>(pp.pivf, pp.specf, pp.n, pp.nx, (size_t)pp.mp, (float)pp.dy2, it.z, it.y,
                                    sh.f);
}

// Modes per block of the partitioned solve for n rows, so that every segment
// has at most TB_L rows (0: too tall, use the one-thread-per-mode `tridiag`),
// and no more than a channel of nx columns has (rounded up to a power of two):
// a wide block reads longer runs of a row (256 x 128 FP64 on B200: 14.6 us a step
// with up to 16 modes, 14.7 with up to 8, 15.1 with up to 32: few blocks).  FP32
// keeps 8, and with it the segments and the rounding of earlier runs.
int tridiag_modes(int n, int nx, bool f32) {
    int most = f32 ? TB_MODES_F32 : TB_MODES;
    while (most > 1 && most / 2 > nx / 2) most /= 2;
    for (int M = most; M >= 1; M >>= 1)
        if ((n + TB_THREADS / M - 1) / (TB_THREADS / M) <= TB_L) return M;
    return 0;
}

bool use_r16(const PoissonPlan &pp) { return pp.pow2 && pp.nx >= 16; }

// nx as radices of the mixed form: fours, a two, threes, fives, other primes.
Radices radices(int nx) {
    Radices f{};
    const int small[4] = {4, 2, 3, 5};
    for (int r : small)
        while (nx % r == 0) {
            f.r[f.n++] = r;
            nx /= r;
        }
    for (int r = 7; nx > 1; r += 2)
        while (nx % r == 0) {
            f.r[f.n++] = r;
            nx /= r;
        }
    return f;
}
// A prime length above 5: the kernel of its own (prime_fft).
bool prime_length(const Radices &f) { return f.n == 1 && f.r[0] > 5; }
// Whether a length has a prime factor above 5, whose pass takes one thread an output.
bool prime_radix(int nx) {
    const Radices f = radices(nx);
    return f.n > 0 && f.r[f.n - 1] > 5;
}
// Threads of a mixed-form block: a butterfly of radix 4 a thread and pass; with a
// prime radix, whose pass outlasts the others, one output a thread (131 x 400 in 32
// threads 83 us a step on B200, in 160 41).
int mixed_threads(int nx) {
    const int t = ((prime_radix(nx) ? nx : nx / 4) + 31) / 32 * 32;
    return t < 32 ? 32 : (t > PTPB ? PTPB : t);
}

// Launches of one size of the row kernels.
template <int K> struct RowLaunch {
    static constexpr int block = RowCfg<K>::block;
    static int grid(const PoissonPlan &pp) { return ((pp.n + 1) / 2 + RowCfg<K>::per - 1) / RowCfg<K>::per; }
    template <typename C> static constexpr size_t smem() { return (size_t)RowCfg<K>::per * RowCfg<K>::N * sizeof(C); }
    static cudaError_t fwd64(const PoissonPlan &pp, const double *rhs, int nxp, bool chain, cudaStream_t s) {
        if (!chain) return launch_pdl(fwd_rows_f64<K>, dim3(grid(pp)), dim3(block), smem<double2>(), s, pp, rhs, nxp);
        return launch_chain(true, fwd_rows_f64<K>, dim3(grid(pp)), dim3(block), smem<double2>(), s, pp, rhs, nxp);
    }
    static cudaError_t inv64(const PoissonPlan &pp, const Chan &c, double *psi, bool pdl, cudaStream_t s) {
        return launch_chain(pdl, inv_rows_f64<K>, dim3(grid(pp)), dim3(block), smem<double2>(), s, pp, c, psi);
    }
    static cudaError_t fwd32(const PoissonPlan &pp, const Chan &c, bool chain, cudaStream_t s) {
        if (!chain) return launch_pdl(fwd_rows_f32<K>, dim3(grid(pp)), dim3(block), smem<float2>(), s, pp, c);
        return launch_chain(true, fwd_rows_f32<K>, dim3(grid(pp)), dim3(block), smem<float2>(), s, pp, c);
    }
    static cudaError_t inv32(const PoissonPlan &pp, const Chan &c, double *psi, bool write_f64, bool pdl, cudaStream_t s) {
        return launch_chain(pdl, inv_rows_f32<K>, dim3(grid(pp)), dim3(block), smem<float2>(), s, pp, c, psi, write_f64);
    }
    static cudaError_t limits(bool f32) {
        const void *fns[] = {(const void *)fwd_rows_f64<K>, (const void *)inv_rows_f64<K>, (const void *)fwd_rows_f32<K>,
                             (const void *)inv_rows_f32<K>};
        for (int i = 0; i < (f32 ? 4 : 2); ++i) {
            const size_t bytes = i < 2 ? smem<double2>() : smem<float2>();
            cudaError_t e = cudaFuncSetAttribute(fns[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(fns[i], cudaFuncAttributePreferredSharedMemoryCarveout, ROW_SMEM_PERCENT);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
};
#define EK_ROW_DISPATCH(lg, call)                       \
    switch (lg) {                                       \
        case 4: return RowLaunch<4>::call;              \
        case 5: return RowLaunch<5>::call;              \
        case 6: return RowLaunch<6>::call;              \
        case 7: return RowLaunch<7>::call;              \
        case 8: return RowLaunch<8>::call;              \
        case 9: return RowLaunch<9>::call;              \
        case 10: return RowLaunch<10>::call;            \
        case 11: return RowLaunch<11>::call;            \
        case 12: return RowLaunch<12>::call;            \
        case 13: return RowLaunch<13>::call;            \
        default: return cudaErrorInvalidValue;          \
    }

// Programmatic launch of passes B and C: where the passes are one wave of
// blocks it hides their launch latency; on channels of many nodes it made the
// step longer (4096 x 1024: 4.5 us a step), the waiting blocks taking the place
// of running ones.
bool small_channel(const PoissonPlan &pp) { return (size_t)pp.nx * pp.ny <= PDL_NODES; }

}  // namespace

size_t poisson_smem_bytes_f64(int nx) { return 2 * (size_t)nx * sizeof(double2); }

cudaError_t poisson_pass_f64(int pass, const PoissonPlan &pp, const Chan &c, double *fields, cudaStream_t s) {
    return poisson_pass_f64_at(pass, pp, c, fields + F_RHS * c.plane, fields + F_PSI * c.plane, s);
}

cudaError_t poisson_pass_f64_at(int pass, const PoissonPlan &pp, const Chan &c, const double *rhs, double *psi,
                                cudaStream_t s) {
    const bool pdl = small_channel(pp);
    if (pass == 1) {
        const int M = tridiag_modes(pp.n, pp.nx, false);
        if (M > 0) return launch_chain(pdl, tridiag_part, dim3((pp.nx / 2 + M) / M), dim3(TB_THREADS), 0, s, pp, M);
        return launch_chain(pdl, tridiag, dim3((pp.nx / 2 + 1 + PTPB - 1) / PTPB), dim3(PTPB), 0, s, pp);
    }
    if (use_r16(pp)) {
        if (pass == 0) EK_ROW_DISPATCH(pp.log2nx, fwd64(pp, rhs, c.nxp, pdl, s))
        EK_ROW_DISPATCH(pp.log2nx, inv64(pp, c, psi, pdl, s))
    }
    const Radices f = radices(pp.nx);
    const dim3 grid((pp.n + 1) / 2), block(mixed_threads(pp.nx));
    const size_t smem = poisson_smem_bytes_f64(pp.nx);
    if (prime_length(f)) {
        // Long blocks that fill the GPU are launched the ordinary way: scheduled early
        // they pile up on the SMs that the kernel before leaves first.  B200, us a
        // step, chained against ordinary: 131 x 200 27.6, 27.2; 131 x 400 38.8, 33.4;
        // 449 x 400 243, 181; but 131 x 101 22.1, 26.2 and 113 x 300 26.4, 29.2.
        const bool chain = pdl && !(pp.nx > 128 && (pp.n + 1) / 2 > 74);
        if (pass == 0) return launch_chain(chain, fwd_rows<true>, grid, block, smem, s, pp, f, rhs, c.nxp);
        return launch_chain(chain, inv_rows<true>, grid, block, smem, s, pp, f, c, psi);
    }
    if (pass == 0)
        return pdl ? launch_chain(true, fwd_rows<false>, grid, block, smem, s, pp, f, rhs, c.nxp)
                   : launch_pdl(fwd_rows<false>, grid, block, smem, s, pp, f, rhs, c.nxp);
    return launch_chain(pdl, inv_rows<false>, grid, block, smem, s, pp, f, c, psi);
}

int poisson_tridiag_modes(int n, int nx) { return tridiag_modes(n, nx, true); }

bool poisson_f32_supported(const PoissonPlan &pp) {
    return use_r16(pp) && tridiag_modes(pp.n, pp.nx, true) > 0 && pp.twf && pp.pivf && pp.specf && pp.rowmean && pp.rowmean_ok;
}

cudaError_t poisson_tridiag_f32(const PoissonPlan &pp, cudaStream_t s) {
    if (!poisson_f32_supported(pp)) return cudaErrorInvalidValue;
    const int M = tridiag_modes(pp.n, pp.nx, true);
    return launch_chain(small_channel(pp), tridiag_modes_f32, dim3(1 + (pp.nx / 2 + M - 1) / M), dim3(TB_THREADS), 0, s, pp,
                            M);
}

cudaError_t poisson_pass_f32(int pass, const PoissonPlan &pp, const Chan &c, double *psi, bool write_f64,
                             cudaStream_t s) {
    // pass B of this form runs through poisson_tridiag_f32
    if (!poisson_f32_supported(pp) || pass == 1) return cudaErrorInvalidValue;
    if (pass == 0) EK_ROW_DISPATCH(pp.log2nx, fwd32(pp, c, small_channel(pp), s))
    EK_ROW_DISPATCH(pp.log2nx, inv32(pp, c, psi, write_f64, small_channel(pp), s))
}

namespace {

// Threads a row pair and shared memory of the cluster's blocks.
int cluster_row_threads(const PoissonPlan &pp) {
    if (use_r16(pp)) return pp.nx >> 4;
    const int per = prime_radix(pp.nx) ? 1 : 4;  // points a thread (mixed_threads)
    int t = 32;
    while (t < CL_THREADS && per * t < pp.nx) t *= 2;
    return t;
}
// The most that any plan asks for: 512 threads of 16 FP64 points (two buffers of
// mixed length: 64 KB).  The kernels' limit, whatever plan sets it: one kernel
// serves all mixed lengths, several of which may be alive.
constexpr size_t CLUSTER_SMEM = (size_t)CL_THREADS * 16 * sizeof(double2);
size_t cluster_smem(const PoissonPlan &pp, bool f32) {
    const int per = CL_THREADS / cluster_row_threads(pp);
    return (size_t)per * pp.nx * (f32 ? sizeof(float2) : (use_r16(pp) ? 1 : 2) * sizeof(double2));
}
// The kernel of a plan (poisson_cluster_blocks): FP64 nx = 16 or a length of the mixed
// form, FP32 nx = 16 to 128.
const void *cluster_kernel(const PoissonPlan &pp, bool f32) {
    if (!f32) return use_r16(pp) ? (const void *)solve_cluster_f64<4> : (const void *)solve_cluster_f64<0>;
    switch (pp.log2nx) {
        case 4: return (const void *)solve_cluster_f32<4>;
        case 5: return (const void *)solve_cluster_f32<5>;
        case 6: return (const void *)solve_cluster_f32<6>;
        default: return (const void *)solve_cluster_f32<7>;
    }
}

}  // namespace

int poisson_cluster_blocks(const PoissonPlan &pp, bool f32) {
    // Time of a step with one launch over that with three, FP64 on B200 unless said
    // (44 lengths by 6 to 4000 rows, up to 20,000 nodes):
    // * each block holds its row pairs in one round: 2 x 400 0.89, 2 x 700 1.08, 2 x 4000
    //   1.58, 30 x 500 0.94, 27 x 700 1.22
    // * not with column segments of 5 to 8 rows: 10 x 256 0.91, 10 x 300 1.07; 50 x 128
    //   0.88, 50 x 200 1.07, 50 x 300 0.91; 64 x 200 FP32 1.00, 64 x 300 1.11
    // * powers of two: FP64 at 16 columns (16 x 128 0.84, 32 x 128 1.04, 64 x 128 1.07, 256
    //   x 64 1.06), FP32 up to 128 (16 x 128 0.93, 128 x 64 0.98, 256 x 33 1.04, 256 x 12
    //   1.12)
    // * other lengths up to 1024: 10 x 101 0.89, 300 x 48 0.88, 1000 x 12 0.98, 1500 x 6
    //   1.02, 2000 x 6 1.11
    // * a prime radix makes the row pairs the solve's bulk, which 16 SMs hold while each
    //   has one of them or 256 of their points: 113 x 64 0.91, 131 x 33 0.81, 131 x 48 1.05,
    //   251 x 64 1.46
    const int M = tridiag_modes(pp.n, pp.nx, f32);
    const size_t most = use_r16(pp) ? (size_t)8192 : (size_t)16384;
    if ((size_t)pp.nx * pp.ny > most || M == 0) return 0;
    const int share = ((pp.n + 1) / 2 + 15) / 16;  // row pairs a block
    const int L = (pp.n + TB_THREADS / M - 1) / (TB_THREADS / M);
    if (share > CL_THREADS / cluster_row_threads(pp) || (L > 4 && L <= 8)) return 0;
    if (pp.nx > (use_r16(pp) ? (f32 ? 128 : 16) : 1024)) return 0;
    if (!use_r16(pp) && prime_radix(pp.nx) && share > 1 && share * pp.nx > 256) return 0;
    const void *fn = cluster_kernel(pp, f32);
    const size_t smem = cluster_smem(pp, f32);
    if (smem > CLUSTER_SMEM) return 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLUSTER_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    for (int blocks = 16; blocks >= 8; blocks /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim = {(unsigned)blocks, 1, 1};
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0) return blocks;
        (void)cudaGetLastError();
    }
    return 0;
}

cudaError_t poisson_cluster(const PoissonPlan &pp, const Chan &c, bool f32, const double *rhs, double *psi, bool write_f64,
                            int blocks, cudaStream_t s) {
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim = {(unsigned)blocks, 1, 1};
    const dim3 g(blocks), t(CL_THREADS);
    const size_t smem = cluster_smem(pp, f32);
    const int M = tridiag_modes(pp.n, pp.nx, f32), T = cluster_row_threads(pp);
    const Radices f = use_r16(pp) ? Radices{} : radices(pp.nx);
    if (!f32)
        return launch_attrs(at, 2, use_r16(pp) ? solve_cluster_f64<4> : solve_cluster_f64<0>, g, t, smem, s, pp, f, T, c, rhs,
                            psi, M);
#define EK_CASE(K) \
    case K: return launch_attrs(at, 2, solve_cluster_f32<K>, g, t, smem, s, pp, c, psi, write_f64, M);
    switch (pp.log2nx) {
        EK_CASE(4) EK_CASE(5) EK_CASE(6) EK_CASE(7)
        default: return cudaErrorInvalidValue;
    }
#undef EK_CASE
}

int batch_row_block(int nx_max) { return nx_max <= 1024 ? 64 : 256; }

cudaError_t batch_poisson(int pass, const PoissonPlan *plans, const Chan *chans, double *const *fields,
                          const void *items, int nitems, int block, bool write_f64, cudaStream_t s) {
    if (nitems <= 0) return cudaSuccess;
    if (pass == 1) return cudaErrorInvalidValue;  // runs through batch_tridiag_f32
    const size_t smem = (size_t)block * 16 * sizeof(float2);
    const int2 *it = (const int2 *)items;
    if (block == 64) {
        if (pass == 0) batch_fwd_rows_f32<64><<<nitems, 64, smem, s>>>(plans, chans, it);
        else batch_inv_rows_f32<64><<<nitems, 64, smem, s>>>(plans, chans, fields, it, write_f64);
    } else {
        if (pass == 0) batch_fwd_rows_f32<256><<<nitems, 256, smem, s>>>(plans, chans, it);
        else batch_inv_rows_f32<256><<<nitems, 256, smem, s>>>(plans, chans, fields, it, write_f64);
    }
    return cudaGetLastError();
}

cudaError_t batch_tridiag_f32(const PoissonPlan *plans, const void *items, int nitems, cudaStream_t s) {
    if (nitems > 0) batch_tridiag_modes_f32<<<nitems, TB_THREADS, 0, s>>>(plans, (const int3 *)items);
    return cudaGetLastError();
}

namespace {
template <typename F>
cudaError_t row_limits(F *f, size_t smem) {
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, ROW_SMEM_PERCENT);
    return e;
}
template <bool PRIME>
cudaError_t mixed_limits() {
    const size_t most = poisson_smem_bytes_f64(MIXED_MAX_NX);
    const cudaError_t e = row_limits(fwd_rows<PRIME>, most);
    return e == cudaSuccess ? row_limits(inv_rows<PRIME>, most) : e;
}
}  // namespace

// Only the kernels of this length: an attribute call loads its kernel.  A limit
// belongs to the kernel, not to the plan: it is the same whatever plan sets it,
// so that plans of several lengths can be alive together (the mixed form's
// kernels serve all its lengths and take that of the longest).
cudaError_t poisson_set_smem_limits(const PoissonPlan &pp) {
    if (use_r16(pp)) EK_ROW_DISPATCH(pp.log2nx, limits(pp.specf != nullptr))
    return prime_length(radices(pp.nx)) ? mixed_limits<true>() : mixed_limits<false>();
}

// Every kernel of the FP64 passes, whatever the channel: loaded, limits set.
cudaError_t poisson_load_f64() {
    cudaError_t e = cudaSuccess;
#define EK_CASE(K) \
    if (e == cudaSuccess) e = RowLaunch<K>::limits(false);
    EK_ROW_CASES(EK_CASE)
#undef EK_CASE
    if (e == cudaSuccess) e = mixed_limits<false>();
    if (e == cudaSuccess) e = mixed_limits<true>();
    cudaFuncAttributes at;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, tridiag);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, tridiag_part);
    return e;
}

cudaError_t batch_set_smem_limits(int block) {
    const size_t smem = (size_t)block * 16 * sizeof(float2);
    cudaError_t e;
    if (block == 64) {
        e = row_limits(batch_fwd_rows_f32<64>, smem);
        return e == cudaSuccess ? row_limits(batch_inv_rows_f32<64>, smem) : e;
    }
    e = row_limits(batch_fwd_rows_f32<256>, smem);
    return e == cudaSuccess ? row_limits(batch_inv_rows_f32<256>, smem) : e;
}

}  // namespace ek
