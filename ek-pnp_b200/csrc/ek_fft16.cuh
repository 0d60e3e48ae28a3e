// ek_fft16.cuh -- complex transforms of 2^K points held by 2^(K-4) threads (16
// points a thread), FP32 (float2) and FP64 (double2), for the row passes of
// the Poisson solve.
//
// Forward: decimation in frequency, radix-16 passes from the top index bit
// down (bits [b, b+4), b = K-4, K-8, ...), then one radix-2^(K mod 4) pass on
// the lowest bits when K is not a multiple of 4.  A radix-16 pass is a
// 16-point DFT in registers (4 x 4 split, constant internal twiddles)
// followed by the 15 twiddles exp(-2 pi i kb f / 2^(b+4)); output digit f is
// stored at digit brev4(f), so the transform ends in bit-reversed order.
// Inverse: the adjoint passes in reverse order (conjugate twiddles before the
// inverse DFT), bit-reversed input to natural order.
//
// Shared memory holds transform p of a block at index
// i ^ (((i >> 4) ^ (i >> 8) ^ p) & 15), free of bank conflicts for the
// passes, natural-order and bit-reversed accesses.  The map is linear over
// XOR, so an element's address is its group base's address XOR a
// compile-time constant.  Every pass writes back onto the slots its group
// read, so one barrier per pass suffices.
// FP32 sums of complex values are packed instructions (one issue slot for
// both parts).  FP32 pass twiddles come from per-pass tables laid out f-major,
// kb-minor (the 32 lanes of a warp read consecutive entries); FP64 ones from
// the table of nx-th roots.
#pragma once
#include <cuda_runtime.h>

namespace ek {
namespace fft16 {

__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

template <typename C> struct RealOf;
template <> struct RealOf<float2> { using type = float; };
template <> struct RealOf<double2> { using type = double; };
template <typename C> using Real = typename RealOf<C>::type;
__device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }

constexpr double C1 = 0.92387953251128674;  // cos(pi/8)
constexpr double S1 = 0.38268343236508977;  // sin(pi/8)
constexpr double R2 = 0.70710678118654752;  // cos(pi/4)

__host__ __device__ constexpr int brev4(int f) { return ((f & 1) << 3) | ((f & 2) << 1) | ((f & 4) >> 1) | ((f & 8) >> 3); }
__host__ __device__ constexpr int brevq(int f, int q) { return brev4(f) >> (4 - q); }
// XOR-linear part of the shared-memory swizzle (without the transform term)
__host__ __device__ constexpr int lin(int v) { return v ^ (((v >> 4) ^ (v >> 8)) & 15); }

__device__ __forceinline__ int swz_base(int i, int p) { return i ^ (((i >> 4) ^ (i >> 8) ^ p) & 15); }

// z * exp(-/+ 2 pi i m/16) (forward: minus), m a compile-time constant
template <bool INV, int M, typename C>
__device__ __forceinline__ C w16(C z) {
    using R = Real<C>;
    constexpr int m = M & 15;
    if constexpr (m == 0) {
        return z;
    } else if constexpr (m == 8) {
        return mk(-z.x, -z.y);
    } else if constexpr (m == 4 || m == 12) {
        // forward m = 4: -i z; m = 12: +i z; inverse the other way round
        constexpr bool minus_i = (m == 4) != INV;
        return minus_i ? mk(z.y, -z.x) : mk(-z.y, z.x);
    } else {
        static_assert(m & 1, "the odd multiples of pi/4 are rot45's");
        constexpr double cs[8] = {1.0, C1, R2, S1, 0.0, -S1, -R2, -C1};   // cos(pi j/8), j < 8
        constexpr double sn[8] = {0.0, S1, R2, C1, 1.0, C1, R2, S1};      // sin(pi j/8), j < 8
        constexpr R c = (R)(m < 8 ? cs[m] : -cs[m - 8]);
        constexpr R s0 = (R)(m < 8 ? -sn[m] : sn[m - 8]);  // forward: -sin(pi m/8)
        constexpr R s = INV ? -s0 : s0;
        return mk(z.x * c - z.y * s, z.x * s + z.y * c);
    }
}

// z * exp(-/+ 2 pi i m/16) for m = 2, 6 (odd multiples of pi/4) is R45<m> times
// rot45<INV, m>(z): the factor is left to the sums that follow (one multiply-add
// each).
template <int M> __host__ __device__ constexpr double R45() { return M == 2 ? R2 : -R2; }
template <bool INV, int M, typename C>
__device__ __forceinline__ C rot45(C z) {
    static_assert(M == 2 || M == 6, "m = 2 or 6");
    // (c + i s) z with s = -c (forward m = 2, inverse m = 6) or s = c
    return ((M == 2) != INV) ? mk(z.x + z.y, z.y - z.x) : mk(z.x - z.y, z.x + z.y);
}
// a + c t for a constant c, rounded once
__device__ __forceinline__ float2 axpy(double c, float2 t, float2 a) { return __ffma2_rn(make_float2((float)c, (float)c), t, a); }
__device__ __forceinline__ double2 axpy(double c, double2 t, double2 a) { return make_double2(a.x + c * t.x, a.y + c * t.y); }
__device__ __forceinline__ float2 times(double c, float2 t) { return __fmul2_rn(make_float2((float)c, (float)c), t); }
__device__ __forceinline__ double2 times(double c, double2 t) { return make_double2(c * t.x, c * t.y); }

// Second half of a 4-point DFT: s0 = a + c, d0 = a - c, s1 = b + d, d1 = b - d
// -> X0, X1, X2, X3 in a, b, c, d.
template <bool INV, typename C>
__device__ __forceinline__ void dft4_end(C s0, C d0, C s1, C d1, C &a, C &b, C &c, C &d) {
    a = s0 + s1;
    c = s0 - s1;
    const C plus = mk(d0.x - d1.y, d0.y + d1.x), minus = mk(d0.x + d1.y, d0.y - d1.x);  // d0 +- i d1
    b = INV ? plus : minus;
    d = INV ? minus : plus;
}
// 4-point DFT in place: (a, b, c, d) -> (X0, X1, X2, X3)
template <bool INV, typename C>
__device__ __forceinline__ void dft4(C &a, C &b, C &c, C &d) {
    dft4_end<INV>(a + c, a - c, b + d, b - d, a, b, c, d);
}

// 16-point DFT in place; output f sits at x[out16(f)]
__host__ __device__ constexpr int out16(int f) { return 4 * (f & 3) + (f >> 2); }
template <bool INV, typename C>
__device__ __forceinline__ void dft16(C (&x)[16]) {
    // n = n1 + 4 n2, f = 4 f1 + f2: 4-point DFTs over n2, twiddles W16^(n1 f2),
    // 4-point DFTs over n1
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) dft4<INV>(x[n1], x[n1 + 4], x[n1 + 8], x[n1 + 12]);
    dft4<INV>(x[0], x[1], x[2], x[3]);
    {  // W^1, W^2, W^3
        const C b = w16<INV, 1>(x[5]), d = w16<INV, 3>(x[7]), t = rot45<INV, 2>(x[6]);
        dft4_end<INV>(axpy(R45<2>(), t, x[4]), axpy(-R45<2>(), t, x[4]), b + d, b - d, x[4], x[5], x[6], x[7]);
    }
    {  // W^2, W^4, W^6
        const C c = w16<INV, 4>(x[10]), t = rot45<INV, 2>(x[9]), d = times(R45<6>(), rot45<INV, 6>(x[11]));
        dft4_end<INV>(x[8] + c, x[8] - c, axpy(R45<2>(), t, d), axpy(R45<2>(), t, mk(-d.x, -d.y)), x[8], x[9], x[10], x[11]);
    }
    {  // W^3, W^6, W^9
        const C b = w16<INV, 3>(x[13]), d = w16<INV, 9>(x[15]), t = rot45<INV, 6>(x[14]);
        dft4_end<INV>(axpy(R45<6>(), t, x[12]), axpy(-R45<6>(), t, x[12]), b + d, b - d, x[12], x[13], x[14], x[15]);
    }
}

// 2^Q-point DFT (Q = 1..3) in place on x[o .. o + 2^Q); output f at x[o + outq<Q>(f)]
template <int Q> __host__ __device__ constexpr int outq(int f) { return Q == 3 ? 2 * (f & 3) + (f >> 2) : f; }
template <bool INV, int Q, typename C>
__device__ __forceinline__ void dftq(C *x) {
    if constexpr (Q == 1) {
        const C a = x[0], b = x[1];
        x[0] = a + b;
        x[1] = a - b;
    } else if constexpr (Q == 2) {
        dft4<INV>(x[0], x[1], x[2], x[3]);
    } else {
        // n = n1 + 2 n2, f = 4 f1 + f2: 4-point DFTs over n2, twiddles W8^(n1 f2),
        // 2-point DFTs over n1
        dft4<INV>(x[0], x[2], x[4], x[6]);
        dft4<INV>(x[1], x[3], x[5], x[7]);
        const C a0 = x[0], b0 = x[1], a2 = x[4], b2 = w16<INV, 4>(x[5]);
        const C t1 = rot45<INV, 2>(x[3]), t3 = rot45<INV, 6>(x[7]), a1 = x[2], a3 = x[6];
        x[0] = a0 + b0;
        x[1] = a0 - b0;
        x[2] = axpy(R45<2>(), t1, a1);
        x[3] = axpy(-R45<2>(), t1, a1);
        x[4] = a2 + b2;
        x[5] = a2 - b2;
        x[6] = axpy(R45<6>(), t3, a3);
        x[7] = axpy(-R45<6>(), t3, a3);
    }
}

template <int K>
struct Shape {
    static constexpr int N = 1 << K, T = N >> 4, NF = K >> 2, Q = K & 3;
    // full pass i = 1..NF works on bits [K - 4i, K - 4i + 4)
    __host__ __device__ static constexpr int bit(int i) { return K - 4 * i; }
    // offset of pass i's twiddle table (passes with bit >= 1 have one)
    __host__ __device__ static constexpr int off(int i) {
        int o = 0;
        for (int j = 1; j < i; ++j) o += 15 << (K - 4 * j);
        return o;
    }
};

// Pass twiddle of the table, loaded with an L2 evict_last policy: the tables
// (32 KB at nx = 4096) are read by every block of every solve, and between
// two solves the LBM step streams ~0.9 GB through L2; kept there, the
// inverse pass ran 19.8 us against 20.9 us at 4096 x 1024 (B200).
__device__ __forceinline__ float2 ldtw(const float2 *p) {
    float2 v;
    unsigned long long pol;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    asm volatile("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(v.x), "=f"(v.y) : "l"(p), "l"(pol));
    return v;
}

template <typename C> __device__ __forceinline__ C mulw(C a, C w) {
    return mk(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
template <typename C> __device__ __forceinline__ C mulw_conj(C a, C w) {
    return mk(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y);
}

// Twiddle exp(-2 pi i kb f / 2^(b+4)) of full pass I (b = Shape::bit(I)):
// FP32 from the pass tables, FP64 from the nx-th roots.
template <int K, int I> __device__ __forceinline__ float2 pass_tw(const float2 *__restrict__ t, int f, int kb) {
    return ldtw(t + Shape<K>::off(I) + ((f - 1) << Shape<K>::bit(I)) + kb);
}
template <int K, int I> __device__ __forceinline__ double2 pass_tw(const double2 *__restrict__ t, int f, int kb) {
    return __ldg(t + ((kb * f) << (K - 4 - Shape<K>::bit(I))));
}

// Barrier of the threads that run transforms: the whole block (n = 0), or its
// first n threads (whole warps) where the others have none.
__device__ __forceinline__ void rows_sync(int n) {
    if (n == 0) __syncthreads();
    else asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
}

// Thread t's group of full pass I: first element and in-group offset kb.
template <int K, int I>
__device__ __forceinline__ void group(int t, int &base, int &kb) {
    constexpr int b = Shape<K>::bit(I);
    kb = t & ((1 << b) - 1);
    base = kb | ((t >> b) << (b + 4));
}

// Forward full pass I on x (its group's elements, v = 0..15), result into s.
template <int K, int I, typename C>
__device__ __forceinline__ void fwd_pass_store(C (&x)[16], C *s, int t, int p,
                                               const C *__restrict__ twp) {
    constexpr int b = Shape<K>::bit(I);
    int base, kb;
    group<K, I>(t, base, kb);
    dft16<false>(x);
    const int sb = swz_base(base, p);
    if constexpr (b > 0) {
#pragma unroll
        for (int f = 1; f < 16; ++f) x[out16(f)] = mulw(x[out16(f)], pass_tw<K, I>(twp, f, kb));
    }
#pragma unroll
    for (int f = 0; f < 16; ++f) s[sb ^ lin(brev4(f) << b)] = x[out16(f)];
}

template <int K, int I, typename C>
__device__ __forceinline__ void fwd_pass_load(C (&x)[16], const C *s, int t, int p) {
    constexpr int b = Shape<K>::bit(I);
    int base, kb;
    group<K, I>(t, base, kb);
    const int sb = swz_base(base, p);
#pragma unroll
    for (int v = 0; v < 16; ++v) x[v] = s[sb ^ lin(v << b)];
}

// Forward passes 2..NF and the partial pass, after pass 1 stored into s.
template <int K, int I, typename C>
__device__ __forceinline__ void fwd_rest(C *s, int t, int p, const C *__restrict__ twp, int ns = 0) {
    if constexpr (I <= Shape<K>::NF) {
        C x[16];
        fwd_pass_load<K, I>(x, s, t, p);  // a pass writes back onto its group's own slots
        fwd_pass_store<K, I>(x, s, t, p, twp);
        rows_sync(ns);
        fwd_rest<K, I + 1>(s, t, p, twp, ns);
    } else if constexpr (Shape<K>::Q > 0) {
        constexpr int Q = Shape<K>::Q, R = 1 << Q;
        const int sb = swz_base(t << 4, p);
        C x[16];
#pragma unroll
        for (int v = 0; v < 16; ++v) x[v] = s[sb ^ v];
#pragma unroll
        for (int j = 0; j < 16; j += R) dftq<false, Q>(x + j);
#pragma unroll
        for (int j = 0; j < 16; j += R)
#pragma unroll
            for (int f = 0; f < R; ++f) s[sb ^ (j + brevq(f, Q))] = x[j + outq<Q>(f)];
        rows_sync(ns);
    }
}

// Inverse full pass I: conjugate twiddles, inverse DFT; x ends in natural
// order of v (element base | v << b).
template <int K, int I, typename C>
__device__ __forceinline__ void inv_pass_load(C (&x)[16], const C *s, int t, int p,
                                              const C *__restrict__ twp) {
    constexpr int b = Shape<K>::bit(I);
    int base, kb;
    group<K, I>(t, base, kb);
    const int sb = swz_base(base, p);
    C z[16];
#pragma unroll
    for (int f = 0; f < 16; ++f) z[f] = s[sb ^ lin(brev4(f) << b)];
    if constexpr (b > 0) {
#pragma unroll
        for (int f = 1; f < 16; ++f) z[f] = mulw_conj(z[f], pass_tw<K, I>(twp, f, kb));
    }
    dft16<true>(z);
#pragma unroll
    for (int v = 0; v < 16; ++v) x[v] = z[out16(v)];
}

template <int K, int I, typename C>
__device__ __forceinline__ void inv_pass_store(const C (&x)[16], C *s, int t, int p) {
    constexpr int b = Shape<K>::bit(I);
    int base, kb;
    group<K, I>(t, base, kb);
    const int sb = swz_base(base, p);
#pragma unroll
    for (int v = 0; v < 16; ++v) s[sb ^ lin(v << b)] = x[v];
}

// Inverse passes NF..2 (after the partial pass); pass 1 is left to the caller,
// which takes its output from registers.
template <int K, int I, typename C>
__device__ __forceinline__ void inv_full(C *s, int t, int p, const C *__restrict__ twp, int ns = 0) {
    if constexpr (I >= 2) {
        C x[16];
        inv_pass_load<K, I>(x, s, t, p, twp);
        inv_pass_store<K, I>(x, s, t, p);
        rows_sync(ns);
        inv_full<K, I - 1>(s, t, p, twp, ns);
    }
}

template <int K, typename C>
__device__ __forceinline__ void inv_partial(C *s, int t, int p, int ns = 0) {
    if constexpr (Shape<K>::Q > 0) {
        constexpr int Q = Shape<K>::Q, R = 1 << Q;
        const int sb = swz_base(t << 4, p);
        C x[16];
#pragma unroll
        for (int j = 0; j < 16; j += R)
#pragma unroll
            for (int f = 0; f < R; ++f) x[j + f] = s[sb ^ (j + brevq(f, Q))];
#pragma unroll
        for (int j = 0; j < 16; j += R) {
            dftq<true, Q>(x + j);
            C y[R];
#pragma unroll
            for (int v = 0; v < R; ++v) y[v] = x[j + outq<Q>(v)];
#pragma unroll
            for (int v = 0; v < R; ++v) s[sb ^ (j + v)] = y[v];
        }
        rows_sync(ns);
    }
}

}  // namespace fft16
}  // namespace ek
