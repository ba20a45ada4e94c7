// Single-element field inversion for the one-per-block inversions of the
// batch-invert and product kernels, the MSM's affine conversion and the Kate
// division.  A whole CTA or stream waits on one thread, so the dependent chain
// is what counts: the division steps of Bernstein and Yang ("Fast
// constant-time gcd computation and modular inversion", 2019) with delta
// starting at 1/2, 30 at a time on the low words of f and g alone (a 2 x 2
// matrix of 31-bit entries), then one pass that applies the matrix to f, g and
// to the cofactors d, e (reduced modulo m by a 30-bit Montgomery digit).  The
// start at 1/2, its bound of 590 steps for 256-bit inputs and the digit update
// of d and e follow Wuille's write-up of the algorithm for libsecp256k1
// (doc/safegcd_implementation.md there).  The loop ends when g is zero.
// d starts at 0 and e at R^2, so the result is (a R)^-1 R^2 = a^-1 R without a
// closing product.  |d| and |e| grow by at most m per pass (below 21 m; limbs
// and sums fit 64 bits).  Inverse of zero is zero.
#pragma once
#include "field.cuh"

namespace h2b {

// limb i of x in the 30-bit grid, x = 8 words (M modulus, Q R^2 mod m)
template <class C>
__host__ __device__ constexpr uint32_t qword(int w)
{
    return w == 0 ? C::Q0 : w == 1 ? C::Q1 : w == 2 ? C::Q2 : w == 3 ? C::Q3 : w == 4 ? C::Q4
         : w == 5 ? C::Q5 : w == 6 ? C::Q6 : w == 7 ? C::Q7 : 0u;
}
constexpr uint32_t M30 = (1u << 30) - 1;
template <class C>
__host__ __device__ constexpr int32_t m30(int i)
{
    return (int32_t)((((uint64_t)mword<C>((30 * i) / 32)) | ((uint64_t)mword<C>((30 * i) / 32 + 1) << 32)) >>
                     ((30 * i) % 32) & M30);
}
template <class C>
__host__ __device__ constexpr int32_t q30(int i)
{
    return (int32_t)((((uint64_t)qword<C>((30 * i) / 32)) | ((uint64_t)qword<C>((30 * i) / 32 + 1) << 32)) >>
                     ((30 * i) % 32) & M30);
}
template <class C>
struct Inv30 {
    static constexpr int32_t p0 = m30<C>(0), p1 = m30<C>(1), p2 = m30<C>(2), p3 = m30<C>(3), p4 = m30<C>(4),
                             p5 = m30<C>(5), p6 = m30<C>(6), p7 = m30<C>(7), p8 = m30<C>(8);
    static constexpr int32_t q0 = q30<C>(0), q1 = q30<C>(1), q2 = q30<C>(2), q3 = q30<C>(3), q4 = q30<C>(4),
                             q5 = q30<C>(5), q6 = q30<C>(6), q7 = q30<C>(7), q8 = q30<C>(8);
};

// d += c p for signed 30-bit limbs (the top limb keeps the sign)
template <class C>
H2B_DEV void inv30_add_mp(int32_t (&t)[9], const int32_t (&d)[9], int32_t c)
{
    using K = Inv30<C>;
    const int32_t p[9] = {K::p0, K::p1, K::p2, K::p3, K::p4, K::p5, K::p6, K::p7, K::p8};
    int64_t x = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        x += (int64_t)c * p[i] + d[i];
        t[i] = i < 8 ? (int32_t)((uint32_t)x & M30) : (int32_t)x;
        x >>= 30;
    }
}

template <class C>
__device__ __noinline__ Fp<C> finv_fast(const Fp<C> a)
{
    using K = Inv30<C>;
    if (a.is_zero()) return a;
    const int32_t p[9] = {K::p0, K::p1, K::p2, K::p3, K::p4, K::p5, K::p6, K::p7, K::p8};
    int32_t f[9], g[9], d[9], e[9] = {K::q0, K::q1, K::q2, K::q3, K::q4, K::q5, K::q6, K::q7, K::q8};
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const int w = (30 * i) / 32, o = (30 * i) % 32;
        f[i] = p[i];
        g[i] = (int32_t)(__funnelshift_r(a.v[w], w + 1 < 8 ? a.v[w + 1] : 0u, o) & M30);
        d[i] = 0;
    }
    int32_t k = 0;    // delta - 1/2
#pragma unroll 1
    for (int it = 0; it < 20; it++) {
        // 30 steps on the low words: 2^30 (f', g') = (u f + v g, q f + r g)
        int32_t u = 1, v = 0, q = 0, r = 1;
        uint32_t f0 = (uint32_t)f[0] | (uint32_t)f[1] << 30, g0 = (uint32_t)g[0] | (uint32_t)g[1] << 30;
#pragma unroll 6
        for (int s = 0; s < 30; s++) {
            const bool odd = g0 & 1u, sw = odd && k >= 0;
            const uint32_t nf = sw ? g0 : f0;
            const int32_t nu = sw ? q : u, nv = sw ? r : v;
            g0 += odd ? (sw ? 0u - f0 : f0) : 0u;
            q += odd ? (sw ? -u : u) : 0;
            r += odd ? (sw ? -v : v) : 0;
            k = sw ? -k : k + 1;
            g0 >>= 1;
            f0 = nf;
            u = nu << 1;
            v = nv << 1;
        }
        int64_t cf = (int64_t)u * f[0] + (int64_t)v * g[0], cg = (int64_t)q * f[0] + (int64_t)r * g[0];
        int64_t cd = (int64_t)u * d[0] + (int64_t)v * e[0], ce = (int64_t)q * d[0] + (int64_t)r * e[0];
        const int32_t md = (int32_t)(((uint32_t)cd * C::N0) & M30), me = (int32_t)(((uint32_t)ce * C::N0) & M30);
        cd += (int64_t)md * p[0];
        ce += (int64_t)me * p[0];
        cf >>= 30; cg >>= 30; cd >>= 30; ce >>= 30;
        uint32_t gz = 0;
#pragma unroll
        for (int i = 1; i < 9; i++) {
            cf += (int64_t)u * f[i] + (int64_t)v * g[i];
            cg += (int64_t)q * f[i] + (int64_t)r * g[i];
            cd += (int64_t)u * d[i] + (int64_t)v * e[i] + (int64_t)md * p[i];
            ce += (int64_t)q * d[i] + (int64_t)r * e[i] + (int64_t)me * p[i];
            f[i - 1] = (int32_t)((uint32_t)cf & M30); cf >>= 30;
            g[i - 1] = (int32_t)((uint32_t)cg & M30); cg >>= 30;
            d[i - 1] = (int32_t)((uint32_t)cd & M30); cd >>= 30;
            e[i - 1] = (int32_t)((uint32_t)ce & M30); ce >>= 30;
            gz |= (uint32_t)g[i - 1];
        }
        f[8] = (int32_t)cf; g[8] = (int32_t)cg; d[8] = (int32_t)cd; e[8] = (int32_t)ce;
        if ((gz | (uint32_t)g[8]) == 0) break;
    }
    // f = 1 or -1 (otherwise a was a multiple of m: zero, like the zero input)
    uint32_t pos = (uint32_t)f[0] ^ 1u, neg = ~(uint32_t)f[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        if (i) pos |= (uint32_t)f[i];
        neg |= (uint32_t)f[i] ^ M30;
    }
    pos |= (uint32_t)f[8];
    if (pos != 0 && neg != 0) return Fp<C>::zero();
    if (neg == 0) {
        int32_t x = 0;
#pragma unroll
        for (int i = 0; i < 9; i++) {
            x -= d[i];
            d[i] = i < 8 ? (int32_t)((uint32_t)x & M30) : x;
            x >>= 30;
        }
    }
    // |d| < 21 m -> [0, m)
    int32_t t[9];
    if (d[8] < 0) inv30_add_mp<C>(d, d, 32);
#pragma unroll 1
    for (int c = 16; c > 0; c >>= 1) {
        inv30_add_mp<C>(t, d, -c);
        const bool keep = t[8] < 0;
#pragma unroll
        for (int i = 0; i < 9; i++) d[i] = keep ? d[i] : t[i];
    }
    Fp<C> r;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int i0 = (32 * j) / 30, o = 32 * j - 30 * i0;
        uint64_t x = (uint64_t)(uint32_t)d[i0] >> o;
        x |= (uint64_t)(uint32_t)d[i0 + 1] << (30 - o);
        if (i0 + 2 < 9 && 60 - o < 32) x |= (uint64_t)(uint32_t)d[i0 + 2] << (60 - o);
        r.v[j] = (uint32_t)x;
    }
    return r;
}

} // namespace h2b
