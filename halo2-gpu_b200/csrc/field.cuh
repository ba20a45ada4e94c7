// BN254 prime-field arithmetic for sm_100a: 8 x 32-bit limbs, Montgomery form
// with R = 2^256, little-endian limb order.  Memory layout is byte-identical to
// halo2curves' `Fr` / `Fq` (4 x u64 little-endian, Montgomery form), which is
// what the reference's device type `fr_t` / `fp_t` stores
// (halo2_proofs/cuda/include/field/alt_bn128.hpp:15-43 pins the moduli,
// R^2 mod m, R mod m and n0' = -m^-1 mod 2^64).
//
// operator* is the Montgomery product in even and odd word rows
// (mont_mul_eo).  Four other forms stay for comparison (h2b_fr_mul_batch):
// word-serial CIOS with `mad.lo.cc` / `madc.hi.cc` chains (mont_mul_inline),
// the same recurrence with mad.wide products (mont_mul_wide), product
// scanning over 29-bit limbs with 64-bit column sums (mul29 / mont_mul_29),
// and product scanning over 52-bit limbs on the FP64 pipe (mont_mul_f64).
// Every value handed out of this header through Fp is fully
// reduced (canonical Montgomery residue), so outputs are bit-exact with any
// other correct implementation; Fl values (29-bit limbs) are below 2p until
// from_l() reduces them.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace h2b {

#define H2B_DEV __device__ __forceinline__

// Scalar field r (halo2curves bn256::Fr); constants from alt_bn128.hpp:30-43.
struct FrCfg {
    static constexpr uint32_t M0 = 0xf0000001u, M1 = 0x43e1f593u, M2 = 0x79b97091u, M3 = 0x2833e848u,
                              M4 = 0x8181585du, M5 = 0xb85045b6u, M6 = 0xe131a029u, M7 = 0x30644e72u;
    static constexpr uint32_t N0 = 0xefffffffu;  // low word of 0xc2e1f593efffffff
    static constexpr uint64_t NP52 = 0x1f593efffffffull;  // low 52 bits of the same n'
    static constexpr uint32_t O0 = 0x4ffffffbu, O1 = 0xac96341cu, O2 = 0x9f60cd29u, O3 = 0x36fc7695u,
                              O4 = 0x7879462eu, O5 = 0x666ea36fu, O6 = 0x9a07df2fu, O7 = 0x0e0a77c1u;
    static constexpr uint32_t Q0 = 0xae216da7u, Q1 = 0x1bb8e645u, Q2 = 0xe35c59e3u, Q3 = 0x53fe3ab1u,
                              Q4 = 0x53bb8085u, Q5 = 0x8c49833du, Q6 = 0x7f4e44a5u, Q7 = 0x0216d0b1u;
};

// Base field p (halo2curves bn256::Fq); constants from alt_bn128.hpp:15-29.
struct FqCfg {
    static constexpr uint32_t M0 = 0xd87cfd47u, M1 = 0x3c208c16u, M2 = 0x6871ca8du, M3 = 0x97816a91u,
                              M4 = 0x8181585du, M5 = 0xb85045b6u, M6 = 0xe131a029u, M7 = 0x30644e72u;
    static constexpr uint32_t N0 = 0xe4866389u;  // low word of 0x87d20782e4866389
    static constexpr uint64_t NP52 = 0x20782e4866389ull;  // low 52 bits of the same n'
    static constexpr uint32_t O0 = 0xc58f0d9du, O1 = 0xd35d438du, O2 = 0xf5c70b3du, O3 = 0x0a78eb28u,
                              O4 = 0x7879462cu, O5 = 0x666ea36fu, O6 = 0x9a07df2fu, O7 = 0x0e0a77c1u;
    static constexpr uint32_t Q0 = 0x538afa89u, Q1 = 0xf32cfc5bu, Q2 = 0xd44501fbu, Q3 = 0xb5e71911u,
                              Q4 = 0x0a417ff6u, Q5 = 0x47ab1effu, Q6 = 0xcab8351fu, Q7 = 0x06d89f71u;
};

template <class C>
struct Fp {
    uint32_t v[8];

    H2B_DEV static Fp zero()
    {
        Fp r;
#pragma unroll
        for (int i = 0; i < 8; i++) r.v[i] = 0;
        return r;
    }
    H2B_DEV static Fp one()
    {
        Fp r;
        r.v[0] = C::O0; r.v[1] = C::O1; r.v[2] = C::O2; r.v[3] = C::O3;
        r.v[4] = C::O4; r.v[5] = C::O5; r.v[6] = C::O6; r.v[7] = C::O7;
        return r;
    }
    H2B_DEV static Fp r2()
    {
        Fp r;
        r.v[0] = C::Q0; r.v[1] = C::Q1; r.v[2] = C::Q2; r.v[3] = C::Q3;
        r.v[4] = C::Q4; r.v[5] = C::Q5; r.v[6] = C::Q6; r.v[7] = C::Q7;
        return r;
    }
    H2B_DEV bool is_zero() const
    {
        uint32_t acc = v[0] | v[1] | v[2] | v[3] | v[4] | v[5] | v[6] | v[7];
        return acc == 0;
    }
    H2B_DEV bool operator==(const Fp& o) const
    {
        uint32_t acc = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) acc |= v[i] ^ o.v[i];
        return acc == 0;
    }
    H2B_DEV bool operator!=(const Fp& o) const { return !(*this == o); }
};

using Fr = Fp<FrCfg>;
using Fq = Fp<FqCfg>;

// One Montgomery word step: t (9 words, t < 2p on entry, t8 == 0) becomes
// (t + a*b + m*p) / 2^32 with m chosen so the low word vanishes.
template <class C>
H2B_DEV void mont_step(uint32_t (&t)[9], const uint32_t (&a)[8], uint32_t b)
{
    asm("{\n\t"
        ".reg .u32 m;\n\t"
        "mad.lo.cc.u32  %0, %9, %17, %0;\n\t"
        "madc.lo.cc.u32 %1, %10, %17, %1;\n\t"
        "madc.lo.cc.u32 %2, %11, %17, %2;\n\t"
        "madc.lo.cc.u32 %3, %12, %17, %3;\n\t"
        "madc.lo.cc.u32 %4, %13, %17, %4;\n\t"
        "madc.lo.cc.u32 %5, %14, %17, %5;\n\t"
        "madc.lo.cc.u32 %6, %15, %17, %6;\n\t"
        "madc.lo.cc.u32 %7, %16, %17, %7;\n\t"
        "addc.u32       %8, %8, 0;\n\t"
        "mad.hi.cc.u32  %1, %9, %17, %1;\n\t"
        "madc.hi.cc.u32 %2, %10, %17, %2;\n\t"
        "madc.hi.cc.u32 %3, %11, %17, %3;\n\t"
        "madc.hi.cc.u32 %4, %12, %17, %4;\n\t"
        "madc.hi.cc.u32 %5, %13, %17, %5;\n\t"
        "madc.hi.cc.u32 %6, %14, %17, %6;\n\t"
        "madc.hi.cc.u32 %7, %15, %17, %7;\n\t"
        "madc.hi.u32    %8, %16, %17, %8;\n\t"
        "mul.lo.u32     m, %0, %26;\n\t"
        "mad.lo.cc.u32  %0, m, %18, %0;\n\t"
        "madc.lo.cc.u32 %1, m, %19, %1;\n\t"
        "madc.lo.cc.u32 %2, m, %20, %2;\n\t"
        "madc.lo.cc.u32 %3, m, %21, %3;\n\t"
        "madc.lo.cc.u32 %4, m, %22, %4;\n\t"
        "madc.lo.cc.u32 %5, m, %23, %5;\n\t"
        "madc.lo.cc.u32 %6, m, %24, %6;\n\t"
        "madc.lo.cc.u32 %7, m, %25, %7;\n\t"
        "addc.u32       %8, %8, 0;\n\t"
        "mad.hi.cc.u32  %1, m, %18, %1;\n\t"
        "madc.hi.cc.u32 %2, m, %19, %2;\n\t"
        "madc.hi.cc.u32 %3, m, %20, %3;\n\t"
        "madc.hi.cc.u32 %4, m, %21, %4;\n\t"
        "madc.hi.cc.u32 %5, m, %22, %5;\n\t"
        "madc.hi.cc.u32 %6, m, %23, %6;\n\t"
        "madc.hi.cc.u32 %7, m, %24, %7;\n\t"
        "madc.hi.u32    %8, m, %25, %8;\n\t"
        "}"
        : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]), "+r"(t[7]),
          "+r"(t[8])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(b),
          "n"(C::M0), "n"(C::M1), "n"(C::M2), "n"(C::M3), "n"(C::M4), "n"(C::M5), "n"(C::M6), "n"(C::M7),
          "n"(C::N0));
    // t0 is now zero; shift one word down.
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = t[i + 1];
    t[8] = 0;
}

// r = t - m if t >= m else t  (t < 2m).
template <class C>
H2B_DEV void cond_sub(uint32_t (&r)[8], const uint32_t (&t)[8])
{
    uint32_t s[8], bw;
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]),
          "=r"(bw)
        : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
          "n"(C::M0), "n"(C::M1), "n"(C::M2), "n"(C::M3), "n"(C::M4), "n"(C::M5), "n"(C::M6), "n"(C::M7));
#pragma unroll
    for (int i = 0; i < 8; i++) r[i] = bw ? t[i] : s[i];
}

template <class C>
H2B_DEV Fp<C> mont_mul_inline(const Fp<C>& a, const Fp<C>& b)
{
    uint32_t t[9];
#pragma unroll
    for (int i = 0; i < 9; i++) t[i] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) mont_step<C>(t, a.v, b.v[i]);
    Fp<C> r;
    uint32_t lo[8];
#pragma unroll
    for (int i = 0; i < 8; i++) lo[i] = t[i];
    cond_sub<C>(r.v, lo);
    return r;
}

// Same CIOS recurrence with each limb product formed by one 32x32->64
// multiply-add (mad.wide.u32) and the 32-bit carry folded in with integer
// adds: on sm_100a mad.hi issues at half the rate of mad.lo, so a lo/hi pair
// costs three issue slots of the multiply pipe where one mad.wide costs about
// 1.5, and the adds go to the ALU pipe.  Every intermediate fits its word:
// a_j*b_i + t_j + c <= (2^32-1)^2 + 2(2^32-1) = 2^64 - 1.
template <class C>
H2B_DEV Fp<C> mont_mul_wide(const Fp<C>& a, const Fp<C>& b)
{
    const uint32_t P[8] = {C::M0, C::M1, C::M2, C::M3, C::M4, C::M5, C::M6, C::M7};
    uint32_t t[9];
#pragma unroll
    for (int i = 0; i < 9; i++) t[i] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t bi = b.v[i];
        uint32_t c = 0;
        uint64_t w;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            w = (uint64_t)a.v[j] * bi + t[j] + c;
            t[j] = (uint32_t)w;
            c = (uint32_t)(w >> 32);
        }
        t[8] += c;                         // t < 2p + p 2^32 < 2^287: no carry out
        const uint32_t m = t[0] * C::N0;
        w = (uint64_t)m * P[0] + t[0];     // low word becomes zero
        c = (uint32_t)(w >> 32);
#pragma unroll
        for (int j = 1; j < 8; j++) {
            w = (uint64_t)m * P[j] + t[j] + c;
            t[j - 1] = (uint32_t)w;
            c = (uint32_t)(w >> 32);
        }
        w = (uint64_t)t[8] + c;
        t[7] = (uint32_t)w;
        t[8] = (uint32_t)(w >> 32);        // zero: t < 2p after the shift
    }
    Fp<C> r;
    uint32_t lo[8];
#pragma unroll
    for (int i = 0; i < 8; i++) lo[i] = t[i];
    cond_sub<C>(r.v, lo);
    return r;
}

// Montgomery multiplication over 29-bit limbs with 64-bit column sums.
//
// A residue x R mod m (R = 2^256, the same Montgomery form as field.cuh) is
// re-sliced into nine limbs of 29 bits (the top limb holds bits 232..255).
// Each limb product is one 32x32->64 multiply-add (mad.wide.u32) into a
// 64-bit column sum; a column holds at most 18 products below 2^58 plus a
// carry below 2^35, so it never overflows and no per-product carry handling
// is needed.  On sm_100a mad.wide issues about twice as many full products per
// clock as a mad.lo/mad.hi pair, so the 162 products here (81 for a*b, 81 for
// m*p) cost fewer multiply-pipe cycles than the 264 lo/hi operations of 32-bit
// CIOS.
//
// Reduction is product-scanning Montgomery with eight 29-bit steps and a final
// 24-bit step (8*29 + 24 = 256), so R stays 2^256: m_k = (column_k * n') mod
// 2^w zeroes the low w bits of the running column.  The quotient then starts
// 5 bits into the 29-bit column grid (bit 261 - 256), and the result limbs are
// re-aligned with two shifts each.
//
// Bounds: inputs < 2p (limbs < 2^29) give a*b + M*p < 4p^2 + 2^256 p, so the
// result is < (4p/2^256 + 1) p < 2p; from_l() makes it canonical.

constexpr uint32_t M29 = (1u << 29) - 1;

template <class C>
__host__ __device__ constexpr uint32_t mword(int w)
{
    return w == 0 ? C::M0 : w == 1 ? C::M1 : w == 2 ? C::M2 : w == 3 ? C::M3 : w == 4 ? C::M4
         : w == 5 ? C::M5 : w == 6 ? C::M6 : w == 7 ? C::M7 : 0u;
}

// limb i of the modulus in the 29-bit grid
template <class C>
__host__ __device__ constexpr uint32_t p29(int i)
{
    return (uint32_t)((((uint64_t)mword<C>((29 * i) / 32)) | ((uint64_t)mword<C>((29 * i) / 32 + 1) << 32)) >>
                      ((29 * i) % 32)) & M29;
}

template <class C>
struct Fl {
    uint32_t l[9];
};

H2B_DEV uint64_t madw(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }

template <class C>
H2B_DEV Fl<C> to_l(const Fp<C>& a)
{
    Fl<C> r;
#pragma unroll
    for (int i = 0; i < 9; i++) {
        const int w = (29 * i) / 32, o = (29 * i) % 32;
        const uint32_t lo = a.v[w], hi = w + 1 < 8 ? a.v[w + 1] : 0u;
        r.l[i] = __funnelshift_r(lo, hi, o) & (i < 8 ? M29 : 0xffffffu);
    }
    return r;
}

// Packs normalised limbs (value < 2p) back to 8 x 32 and reduces below p.
template <class C>
H2B_DEV Fp<C> from_l(const Fl<C>& a)
{
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        // word j covers bits [32j, 32j + 32): limbs i0 = floor(32j/29) and i0 + 1 (and i0 + 2 for some j)
        const int i0 = (32 * j) / 29, o = 32 * j - 29 * i0;
        uint64_t x = (uint64_t)a.l[i0] >> o;
        x |= (uint64_t)(i0 + 1 < 9 ? a.l[i0 + 1] : 0u) << (29 - o);
        if (i0 + 2 < 9 && 58 - o < 32) x |= (uint64_t)a.l[i0 + 2] << (58 - o);
        w[j] = (uint32_t)x;
    }
    Fp<C> r;
    cond_sub<C>(r.v, w);
    return r;
}

template <class C>
H2B_DEV Fl<C> mul29(const Fl<C>& a, const Fl<C>& b)
{
    const uint32_t np = C::N0 & M29;
    uint32_t m[9];
    uint64_t acc = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
#pragma unroll
        for (int i = 0; i <= k; i++) acc = madw(a.l[i], b.l[k - i], acc);
#pragma unroll
        for (int i = 0; i < k; i++) acc = madw(m[i], p29<C>(k - i), acc);
        const uint32_t mk = ((uint32_t)acc * np) & (k < 8 ? M29 : 0xffffffu);
        m[k] = mk;
        acc = madw(mk, p29<C>(0), acc);
        if (k < 8) acc >>= 29;
    }
    // acc: column 8 with its low 24 bits zero; bit 24 of it is result bit 0
    const uint32_t low5 = (uint32_t)(acc >> 24) & 31u;
    acc >>= 29;
    uint32_t h[9];
#pragma unroll
    for (int k = 9; k < 17; k++) {
#pragma unroll
        for (int i = k - 8; i <= 8; i++) acc = madw(a.l[i], b.l[k - i], acc);
#pragma unroll
        for (int i = k - 8; i <= 8; i++) acc = madw(m[i], p29<C>(k - i), acc);
        h[k - 9] = (uint32_t)acc & M29;
        acc >>= 29;
    }
    h[8] = (uint32_t)acc;
    Fl<C> r;
    r.l[0] = (low5 | (h[0] << 5)) & M29;
#pragma unroll
    for (int j = 1; j < 9; j++) r.l[j] = ((h[j] << 5) | (h[j - 1] >> 24)) & M29;
    return r;
}

// Fp in, Fp out through the 29-bit product.
template <class C>
H2B_DEV Fp<C> mont_mul_29(const Fp<C>& a, const Fp<C>& b)
{
    return from_l(mul29(to_l(a), to_l(b)));
}

// Square through the same column grid: the cross products a_i a_j (i < j)
// appear twice, so they are formed once against d_i = 2 a_i (limbs < 2^30,
// products < 2^59, column sums still below 2^62): 45 products instead of 81.
template <class C>
H2B_DEV Fl<C> sqr29(const Fl<C>& a)
{
    const uint32_t np = C::N0 & M29;
    uint32_t d[9], m[9];
#pragma unroll
    for (int i = 0; i < 9; i++) d[i] = a.l[i] << 1;
    uint64_t acc = 0;
#pragma unroll
    for (int k = 0; k < 9; k++) {
#pragma unroll
        for (int i = 0; 2 * i < k; i++) acc = madw(d[i], a.l[k - i], acc);
        if ((k & 1) == 0) acc = madw(a.l[k / 2], a.l[k / 2], acc);
#pragma unroll
        for (int i = 0; i < k; i++) acc = madw(m[i], p29<C>(k - i), acc);
        const uint32_t mk = ((uint32_t)acc * np) & (k < 8 ? M29 : 0xffffffu);
        m[k] = mk;
        acc = madw(mk, p29<C>(0), acc);
        if (k < 8) acc >>= 29;
    }
    const uint32_t low5 = (uint32_t)(acc >> 24) & 31u;
    acc >>= 29;
    uint32_t h[9];
#pragma unroll
    for (int k = 9; k < 17; k++) {
#pragma unroll
        for (int i = k - 8; 2 * i < k; i++) acc = madw(d[i], a.l[k - i], acc);
        if ((k & 1) == 0) acc = madw(a.l[k / 2], a.l[k / 2], acc);
#pragma unroll
        for (int i = k - 8; i <= 8; i++) acc = madw(m[i], p29<C>(k - i), acc);
        h[k - 9] = (uint32_t)acc & M29;
        acc >>= 29;
    }
    h[8] = (uint32_t)acc;
    Fl<C> r;
    r.l[0] = (low5 | (h[0] << 5)) & M29;
#pragma unroll
    for (int j = 1; j < 9; j++) r.l[j] = ((h[j] << 5) | (h[j - 1] >> 24)) & M29;
    return r;
}

template <class C>
H2B_DEV Fp<C> mont_sqr_29(const Fp<C>& a)
{
    return from_l(sqr29(to_l(a)));
}

// ---- Montgomery product in even and odd word rows ---------------------------
//
// Word-serial Montgomery (R = 2^256) on two accumulators: e holds the limb
// products a_j b_i with j even at word j, o those with j odd at word j - 1 of
// a number that stands one word higher.  Every limb product's low and high
// word then land in the two words of one aligned pair, so a row of four
// products is one chain of 64-bit multiply-adds with carry (lo/hi pairs over
// the same operands), and no carry is handled by an instruction of its own but
// the last one of the chain.  After a reduction row e[0] is zero; dividing by
// 2^32 swaps the roles: o becomes the even words (e[1] joins its word 0) and
// e[2..7] the odd ones, which the next row's chains read as addends.  Keeping
// even and odd limb products apart is a known arrangement for GPU multiply-add
// chains (CGBN and sppark's Montgomery fields use it); the rows, the square and
// the two-product sum below are written out for eight words here.
//
// 128 wide multiply-adds and 8 digit products; about 205 instructions and 40
// registers.  Measured on B200 (one chain of products per thread, 16 warps per
// SM): 67.5 G products/s against 54.9 G for the FP64 form and 40 G for the
// 29-bit form; one warp alone takes 860 cycles per product against 1504.  The
// multiply pipe bounds it (a wide multiply-add with carry holds it about four
// cycles per warp); the ALU and FP64 pipes stay nearly idle, so additions and
// corrections beside it cost little.  The square forms 28 products above the
// diagonal, doubles them and adds 8 squares (36 wide multiply-adds instead of
// 64): 79.4 G/s.
//
// Bounds: between rows the value is below a + p, so a < 2^256 - p (4.29 p) and
// any b < 2^256 keep it inside nine words; the result is below a b / 2^256 + p:
// 1.19 p for a, b < p and 1.76 p for a, b < 2p.

// rows of the even/odd product: value = sum e[j] 2^(32 j) + 2^32 sum o[j] 2^(32 j)
template <class C>
H2B_DEV void eo_mul_first(uint32_t (&e)[8], uint32_t (&o)[8], const uint32_t (&a)[8], uint32_t b)
{
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=r"(e[j]), "=r"(e[j + 1]) : "r"(a[j]), "r"(b));
        asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=r"(o[j]), "=r"(o[j + 1]) : "r"(a[j + 1]), "r"(b));
    }
}
// (e, o) <- (e, o) / 2^32 + a b   (e[0] == 0): the new even words are o (+ e[1]), the new odd ones e[2..7]
template <class C>
H2B_DEV void eo_mad_shift(uint32_t (&e)[8], uint32_t (&o)[8], const uint32_t (&a)[8], uint32_t b)
{
    uint32_t n[8];
    asm("add.cc.u32 %0, %0, %9;\n\t"
        "madc.lo.cc.u32 %1, %16, %20, %10;\n\t"
        "madc.hi.cc.u32 %2, %16, %20, %11;\n\t"
        "madc.lo.cc.u32 %3, %17, %20, %12;\n\t"
        "madc.hi.cc.u32 %4, %17, %20, %13;\n\t"
        "madc.lo.cc.u32 %5, %18, %20, %14;\n\t"
        "madc.hi.cc.u32 %6, %18, %20, %15;\n\t"
        "madc.lo.cc.u32 %7, %19, %20, 0;\n\t"
        "madc.hi.u32 %8, %19, %20, 0;"
        : "+r"(o[0]), "=&r"(n[0]), "=&r"(n[1]), "=&r"(n[2]), "=&r"(n[3]), "=&r"(n[4]), "=&r"(n[5]), "=&r"(n[6]), "=&r"(n[7])
        : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(a[1]), "r"(a[3]), "r"(a[5]),
          "r"(a[7]), "r"(b));
    asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
        "addc.u32 %8, %8, 0;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(n[7])
        : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b));
#pragma unroll
    for (int j = 0; j < 8; j++) { e[j] = o[j]; o[j] = n[j]; }
}
// (e, o) += m p with m chosen so that e[0] becomes 0
template <class C>
H2B_DEV void eo_redc(uint32_t (&e)[8], uint32_t (&o)[8])
{
    const uint32_t m = e[0] * C::N0;
    asm("mad.lo.cc.u32 %0, %9, %8, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %8, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %8, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %8, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %8, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %8, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %8, %6;\n\t"
        "madc.hi.u32 %7, %12, %8, %7;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7])
        : "r"(m), "n"(C::M1), "n"(C::M3), "n"(C::M5), "n"(C::M7));
    asm("mad.lo.cc.u32 %0, %10, %9, %0;\n\t"
        "madc.hi.cc.u32 %1, %10, %9, %1;\n\t"
        "madc.lo.cc.u32 %2, %11, %9, %2;\n\t"
        "madc.hi.cc.u32 %3, %11, %9, %3;\n\t"
        "madc.lo.cc.u32 %4, %12, %9, %4;\n\t"
        "madc.hi.cc.u32 %5, %12, %9, %5;\n\t"
        "madc.lo.cc.u32 %6, %13, %9, %6;\n\t"
        "madc.hi.cc.u32 %7, %13, %9, %7;\n\t"
        "addc.u32 %8, %8, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(o[7])
        : "r"(m), "n"(C::M0), "n"(C::M2), "n"(C::M4), "n"(C::M6));
}
// the value (e[0] == 0) / 2^32, plus the number's last word at the top
H2B_DEV void eo_close(uint32_t (&w)[8], const uint32_t (&e)[8], const uint32_t (&o)[8], uint32_t top)
{
    asm("add.cc.u32 %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32 %7, %15, %23;"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(e[1]), "r"(e[2]),
          "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(top));
}

template <class C>
H2B_DEV void eo_mont(uint32_t (&w)[8], const uint32_t (&a)[8], const uint32_t (&b)[8])
{
    uint32_t e[8], o[8];
    eo_mul_first<C>(e, o, a, b[0]);
    eo_redc<C>(e, o);
#pragma unroll
    for (int i = 1; i < 8; i++) {
        eo_mad_shift<C>(e, o, a, b[i]);
        eo_redc<C>(e, o);
    }
    eo_close(w, e, o, 0u);
}

// a^2 in 16 words: 28 products above the diagonal in even and odd rows, doubled, and the 8 squares
template <class C>
H2B_DEV void eo_sqr16(uint32_t (&t)[16], const uint32_t (&a)[8])
{
    uint32_t ev[14], od[14];
    // row 0
#pragma unroll
    for (int j = 1; j < 8; j += 2)
        asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=r"(od[j - 1]), "=r"(od[j]) : "r"(a[0]), "r"(a[j]));
#pragma unroll
    for (int j = 2; j < 8; j += 2)
        asm("mul.lo.u32 %0, %2, %3;\n\tmul.hi.u32 %1, %2, %3;" : "=r"(ev[j]), "=r"(ev[j + 1]) : "r"(a[0]), "r"(a[j]));
    // row 1
    asm("mad.lo.cc.u32 %0, %7, %8, %0;\n\tmadc.hi.cc.u32 %1, %7, %8, %1;\n\t"
        "madc.lo.cc.u32 %2, %7, %9, %2;\n\tmadc.hi.cc.u32 %3, %7, %9, %3;\n\t"
        "madc.lo.cc.u32 %4, %7, %10, %4;\n\tmadc.hi.cc.u32 %5, %7, %10, %5;\n\taddc.u32 %6, 0, 0;"
        : "+r"(od[2]), "+r"(od[3]), "+r"(od[4]), "+r"(od[5]), "+r"(od[6]), "+r"(od[7]), "=r"(od[8])
        : "r"(a[1]), "r"(a[2]), "r"(a[4]), "r"(a[6]));
    asm("mad.lo.cc.u32 %0, %6, %7, %0;\n\tmadc.hi.cc.u32 %1, %6, %7, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %8, %2;\n\tmadc.hi.cc.u32 %3, %6, %8, %3;\n\t"
        "madc.lo.cc.u32 %4, %6, %9, 0;\n\tmadc.hi.u32 %5, %6, %9, 0;"
        : "+r"(ev[4]), "+r"(ev[5]), "+r"(ev[6]), "+r"(ev[7]), "=&r"(ev[8]), "=&r"(ev[9])
        : "r"(a[1]), "r"(a[3]), "r"(a[5]), "r"(a[7]));
    // row 2
    asm("mad.lo.cc.u32 %0, %6, %7, %0;\n\tmadc.hi.cc.u32 %1, %6, %7, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %8, %2;\n\tmadc.hi.cc.u32 %3, %6, %8, %3;\n\t"
        "madc.lo.cc.u32 %4, %6, %9, %4;\n\tmadc.hi.u32 %5, %6, %9, 0;"
        : "+r"(od[4]), "+r"(od[5]), "+r"(od[6]), "+r"(od[7]), "+r"(od[8]), "=&r"(od[9])
        : "r"(a[2]), "r"(a[3]), "r"(a[5]), "r"(a[7]));
    asm("mad.lo.cc.u32 %0, %5, %6, %0;\n\tmadc.hi.cc.u32 %1, %5, %6, %1;\n\t"
        "madc.lo.cc.u32 %2, %5, %7, %2;\n\tmadc.hi.cc.u32 %3, %5, %7, %3;\n\taddc.u32 %4, 0, 0;"
        : "+r"(ev[6]), "+r"(ev[7]), "+r"(ev[8]), "+r"(ev[9]), "=r"(ev[10])
        : "r"(a[2]), "r"(a[4]), "r"(a[6]));
    // row 3
    asm("mad.lo.cc.u32 %0, %5, %6, %0;\n\tmadc.hi.cc.u32 %1, %5, %6, %1;\n\t"
        "madc.lo.cc.u32 %2, %5, %7, %2;\n\tmadc.hi.cc.u32 %3, %5, %7, %3;\n\taddc.u32 %4, 0, 0;"
        : "+r"(od[6]), "+r"(od[7]), "+r"(od[8]), "+r"(od[9]), "=r"(od[10])
        : "r"(a[3]), "r"(a[4]), "r"(a[6]));
    asm("mad.lo.cc.u32 %0, %4, %5, %0;\n\tmadc.hi.cc.u32 %1, %4, %5, %1;\n\t"
        "madc.lo.cc.u32 %2, %4, %6, %2;\n\tmadc.hi.u32 %3, %4, %6, 0;"
        : "+r"(ev[8]), "+r"(ev[9]), "+r"(ev[10]), "=&r"(ev[11])
        : "r"(a[3]), "r"(a[5]), "r"(a[7]));
    // row 4
    asm("mad.lo.cc.u32 %0, %4, %5, %0;\n\tmadc.hi.cc.u32 %1, %4, %5, %1;\n\t"
        "madc.lo.cc.u32 %2, %4, %6, %2;\n\tmadc.hi.u32 %3, %4, %6, 0;"
        : "+r"(od[8]), "+r"(od[9]), "+r"(od[10]), "=&r"(od[11])
        : "r"(a[4]), "r"(a[5]), "r"(a[7]));
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\tmadc.hi.cc.u32 %1, %3, %4, %1;\n\taddc.u32 %2, 0, 0;"
        : "+r"(ev[10]), "+r"(ev[11]), "=r"(ev[12]) : "r"(a[4]), "r"(a[6]));
    // rows 5 and 6
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\tmadc.hi.cc.u32 %1, %3, %4, %1;\n\taddc.u32 %2, 0, 0;"
        : "+r"(od[10]), "+r"(od[11]), "=r"(od[12]) : "r"(a[5]), "r"(a[6]));
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.u32 %1, %2, %3, 0;" : "+r"(ev[12]), "=&r"(ev[13]) : "r"(a[5]), "r"(a[7]));
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.u32 %1, %2, %3, 0;" : "+r"(od[12]), "=&r"(od[13]) : "r"(a[6]), "r"(a[7]));
    // s = ev + 2^32 od (words 1..14)
    uint32_t s[15];
    s[1] = od[0];
    asm("add.cc.u32 %0, %13, %25;\n\taddc.cc.u32 %1, %14, %26;\n\taddc.cc.u32 %2, %15, %27;\n\t"
        "addc.cc.u32 %3, %16, %28;\n\taddc.cc.u32 %4, %17, %29;\n\taddc.cc.u32 %5, %18, %30;\n\t"
        "addc.cc.u32 %6, %19, %31;\n\taddc.cc.u32 %7, %20, %32;\n\taddc.cc.u32 %8, %21, %33;\n\t"
        "addc.cc.u32 %9, %22, %34;\n\taddc.cc.u32 %10, %23, %35;\n\taddc.cc.u32 %11, %24, %36;\n\taddc.u32 %12, %37, 0;"
        : "=&r"(s[2]), "=&r"(s[3]), "=&r"(s[4]), "=&r"(s[5]), "=&r"(s[6]), "=&r"(s[7]), "=&r"(s[8]), "=&r"(s[9]),
          "=&r"(s[10]), "=&r"(s[11]), "=&r"(s[12]), "=&r"(s[13]), "=&r"(s[14])
        : "r"(ev[2]), "r"(ev[3]), "r"(ev[4]), "r"(ev[5]), "r"(ev[6]), "r"(ev[7]), "r"(ev[8]), "r"(ev[9]), "r"(ev[10]),
          "r"(ev[11]), "r"(ev[12]), "r"(ev[13]), "r"(od[1]), "r"(od[2]), "r"(od[3]), "r"(od[4]), "r"(od[5]), "r"(od[6]),
          "r"(od[7]), "r"(od[8]), "r"(od[9]), "r"(od[10]), "r"(od[11]), "r"(od[12]), "r"(od[13]));
    // t = 2 s + the squares
    uint32_t d[16];
    d[0] = 0;
    d[1] = s[1] << 1;
#pragma unroll
    for (int j = 2; j < 15; j++) d[j] = __funnelshift_l(s[j - 1], s[j], 1);
    d[15] = s[14] >> 31;
    asm("mad.lo.cc.u32 %0, %16, %16, %24;\n\tmadc.hi.cc.u32 %1, %16, %16, %25;\n\t"
        "madc.lo.cc.u32 %2, %17, %17, %26;\n\tmadc.hi.cc.u32 %3, %17, %17, %27;\n\t"
        "madc.lo.cc.u32 %4, %18, %18, %28;\n\tmadc.hi.cc.u32 %5, %18, %18, %29;\n\t"
        "madc.lo.cc.u32 %6, %19, %19, %30;\n\tmadc.hi.cc.u32 %7, %19, %19, %31;\n\t"
        "madc.lo.cc.u32 %8, %20, %20, %32;\n\tmadc.hi.cc.u32 %9, %20, %20, %33;\n\t"
        "madc.lo.cc.u32 %10, %21, %21, %34;\n\tmadc.hi.cc.u32 %11, %21, %21, %35;\n\t"
        "madc.lo.cc.u32 %12, %22, %22, %36;\n\tmadc.hi.cc.u32 %13, %22, %22, %37;\n\t"
        "madc.lo.cc.u32 %14, %23, %23, %38;\n\tmadc.hi.u32 %15, %23, %23, %39;"
        : "=&r"(t[0]), "=&r"(t[1]), "=&r"(t[2]), "=&r"(t[3]), "=&r"(t[4]), "=&r"(t[5]), "=&r"(t[6]), "=&r"(t[7]),
          "=&r"(t[8]), "=&r"(t[9]), "=&r"(t[10]), "=&r"(t[11]), "=&r"(t[12]), "=&r"(t[13]), "=&r"(t[14]), "=&r"(t[15])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(d[0]), "r"(d[1]),
          "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]), "r"(d[8]), "r"(d[9]), "r"(d[10]), "r"(d[11]),
          "r"(d[12]), "r"(d[13]), "r"(d[14]), "r"(d[15]));
}

// (e, o) <- (e, o) / 2^32 + m p with the next word t of the reduced number at the top
template <class C>
H2B_DEV void eo_redc_shift(uint32_t (&e)[8], uint32_t (&o)[8], uint32_t t)
{
    uint32_t n[8], m;
    asm("add.cc.u32 %0, %0, %10;\n\t"
        "mul.lo.u32 %9, %0, %22;\n\t"
        "madc.lo.cc.u32 %1, %9, %18, %11;\n\t"
        "madc.hi.cc.u32 %2, %9, %18, %12;\n\t"
        "madc.lo.cc.u32 %3, %9, %19, %13;\n\t"
        "madc.hi.cc.u32 %4, %9, %19, %14;\n\t"
        "madc.lo.cc.u32 %5, %9, %20, %15;\n\t"
        "madc.hi.cc.u32 %6, %9, %20, %16;\n\t"
        "madc.lo.cc.u32 %7, %9, %21, %17;\n\t"
        "madc.hi.u32 %8, %9, %21, 0;"
        : "+r"(o[0]), "=&r"(n[0]), "=&r"(n[1]), "=&r"(n[2]), "=&r"(n[3]), "=&r"(n[4]), "=&r"(n[5]), "=&r"(n[6]),
          "=&r"(n[7]), "=&r"(m)
        : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(t), "n"(C::M1), "n"(C::M3),
          "n"(C::M5), "n"(C::M7), "n"(C::N0));
    asm("mad.lo.cc.u32 %0, %9, %10, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %10, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %11, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %11, %3;\n\t"
        "madc.lo.cc.u32 %4, %9, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %9, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %9, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %9, %13, %7;\n\t"
        "addc.u32 %8, %8, 0;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(n[7])
        : "r"(m), "n"(C::M0), "n"(C::M2), "n"(C::M4), "n"(C::M6));
#pragma unroll
    for (int j = 0; j < 8; j++) { e[j] = o[j]; o[j] = n[j]; }
}

template <class C>
H2B_DEV void eo_mont_sqr(uint32_t (&w)[8], const uint32_t (&a)[8])
{
    uint32_t t[16], e[8], o[8];
    eo_sqr16<C>(t, a);
#pragma unroll
    for (int j = 0; j < 8; j++) { e[j] = t[j]; o[j] = 0; }
    eo_redc<C>(e, o);
#pragma unroll
    for (int i = 8; i < 15; i++) eo_redc_shift<C>(e, o, t[i]);
    eo_close(w, e, o, t[15]);
}

// (e, o) += a b (no shift)
template <class C>
H2B_DEV void eo_mad(uint32_t (&e)[8], uint32_t (&o)[8], const uint32_t (&a)[8], uint32_t b)
{
    asm("mad.lo.cc.u32 %0, %8, %12, %0;\n\t"
        "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
        "madc.hi.u32 %7, %11, %12, %7;"
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7])
        : "r"(a[1]), "r"(a[3]), "r"(a[5]), "r"(a[7]), "r"(b));
    asm("mad.lo.cc.u32 %0, %9, %13, %0;\n\t"
        "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
        "addc.u32 %8, %8, 0;"
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(o[7])
        : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(a[6]), "r"(b));
}

// (a b + c d) 2^-256 mod p, below (a b + c d) / 2^256 + p, with one reduction
// (200 wide multiply-adds instead of 272).  Between rows the value is below
// a + c + p, so a + c < 2^256 - p (4.29 p).
template <class C>
H2B_DEV void eo_mont2(uint32_t (&w)[8], const uint32_t (&a)[8], const uint32_t (&b)[8], const uint32_t (&c)[8],
                      const uint32_t (&d)[8])
{
    uint32_t e[8], o[8];
    eo_mul_first<C>(e, o, a, b[0]);
    eo_mad<C>(e, o, c, d[0]);
    eo_redc<C>(e, o);
#pragma unroll
    for (int i = 1; i < 8; i++) {
        eo_mad_shift<C>(e, o, a, b[i]);
        eo_mad<C>(e, o, c, d[i]);
        eo_redc<C>(e, o);
    }
    eo_close(w, e, o, 0u);
}

template <class C>
H2B_DEV Fp<C> mont_mul_eo(const Fp<C>& a, const Fp<C>& b)
{
    uint32_t w[8];
    eo_mont<C>(w, a.v, b.v);
    Fp<C> r;
    cond_sub<C>(r.v, w);
    return r;
}
template <class C>
H2B_DEV Fp<C> mont_mul_eo_lazy(const Fp<C>& a, const Fp<C>& b)
{
    Fp<C> r;
    eo_mont<C>(r.v, a.v, b.v);
    return r;
}

template <class C>
H2B_DEV Fp<C> mont_sqr_eo(const Fp<C>& a)
{
    uint32_t w[8];
    eo_mont_sqr<C>(w, a.v);
    Fp<C> r;
    cond_sub<C>(r.v, w);
    return r;
}

template <class C>
H2B_DEV Fp<C> mont_sqr_eo_lazy(const Fp<C>& a)
{
    Fp<C> r;
    eo_mont_sqr<C>(r.v, a.v);
    return r;
}

// ---- Montgomery product on the FP64 pipe ---------------------------------
//
// Five 52-bit limbs held exactly in doubles.  A limb product a b < 2^104 is
// split into its high and low 52-bit halves by two FMAs and one subtraction
// (the exact-split technique of Emmart, Zheng and Weems, "Faster modular
// exponentiation using double precision floating point arithmetic on the
// GPU", ARITH 2018):
//   h = fma_rz(a, b, 2^104)            in [2^104, 2^105): ulp 2^52, so
//                                      h = 2^104 + floor(ab / 2^52) 2^52 exactly
//   l = fma(a, b, (2^104 + 2^52) - h)  = 2^52 + (ab mod 2^52), exact
// The bit patterns of h and l are then 0x467.. + hi and 0x433.. + lo, so
// column sums are plain 64-bit integer additions of the patterns; the
// exponent fields of every term that lands in a column are subtracted once,
// through the column's initial value.
//
// Montgomery reduction runs five 52-bit digit steps (R' = 2^260): q_i =
// (t_i mod 2^52) n' mod 2^52 on the integer multiply pipe, then q_i p added
// with the same splits.  The low half of q_i p_0 cancels t_i mod 2^52 by
// construction, so only its carry (1 unless t_i mod 2^52 is 0) is added.
// One operand enters as 16 a (still below 2^260), so the result is
// a b 2^-256 like the 29-bit product.  Bounds: 16 a b + Q p < 16 p^2 + 2^260 p,
// so the result is below (p / 2^256 + 1) p < 1.19 p; one conditional
// subtraction makes it canonical.  Column values stay below 2^57.
//
// Measured on B200: 55 G products/s at 64 to 72 registers (the even/odd form
// 67.5 G at 40).  A limb product with its split and sums takes 10.4 cycles per
// scheduler however many warps run, about what its 20 register words read take
// at two words a cycle, so neither fewer ALU instructions (the carry of a digit
// folded into the column's bias) nor a shorter digit chain (a multiple of p
// that is -1 mod 2^52) made it faster.  Kept as an independent second product
// for the tests of the first.

namespace f64 {
constexpr uint64_t M52 = (1ull << 52) - 1;
constexpr uint64_t EXP_LO = 0x4330000000000000ull;  // pattern of 2^52
constexpr uint64_t EXP_HI = 0x4670000000000000ull;  // pattern of 2^104
constexpr double C52 = 4503599627370496.0;
constexpr double C104 = 20282409603651670423947251286016.0;
constexpr double C104_52 = 20282409603651670423947251286016.0 + 4503599627370496.0;

// an integer below 2^52 as a double: the pattern of 2^52 + x, minus 2^52
H2B_DEV double u52d(uint64_t x) { return __dsub_rn(__longlong_as_double((long long)(x | EXP_LO)), C52); }
H2B_DEV uint64_t dbits(double x) { return (uint64_t)__double_as_longlong(x); }

// bits [S, S + 52) of the 256-bit value v (S < 0: zeros below bit 0)
template <int S>
H2B_DEV uint64_t bits52(const uint32_t (&v)[8])
{
    uint64_t r = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
        const int off = 32 * w - S;
        if (off >= 0 && off < 52) r |= (uint64_t)v[w] << off;
        else if (off < 0 && off > -32) r |= (uint64_t)(v[w] >> (-off));
    }
    return r & M52;
}

// limb i of the modulus in the 52-bit grid
template <class C>
__host__ __device__ constexpr uint64_t p52(int i)
{
    uint64_t r = 0;
    for (int w = 0; w < 8; w++) {
        const int off = 32 * w - 52 * i;
        if (off >= 0 && off < 52) r |= (uint64_t)mword<C>(w) << off;
        else if (off < 0 && off > -32) r |= (uint64_t)(mword<C>(w) >> (-off));
    }
    return r & M52;
}

// how many low and high halves land in column k (product and reduction)
__host__ __device__ constexpr uint64_t bias(int k)
{
    uint64_t nl = 0, nh = 0;
    for (int i = 0; i < 5; i++)
        for (int j = 0; j < 5; j++) {
            nl += (i + j == k);
            nh += (i + j + 1 == k) * 2;     // product hi, reduction hi (j = 0 included)
            nl += (j > 0 && i + j == k);    // reduction lo (j = 0 cancels)
        }
    return nl * EXP_LO + nh * EXP_HI;
}
}  // namespace f64

// The Montgomery core over 52-bit limbs: l = A B / 2^260 + (multiple of p
// absorbed), limbs normalised below 2^52 except the top one, which holds the
// rest.  A and B are limbs below 2^52 held exactly in doubles (any value
// below 2^260); the result is below A B / 2^260 + p.
namespace f64 {
template <class C>
H2B_DEV void mont52(const double (&A)[5], const double (&B)[5], uint64_t (&l)[5])
{
    // every constant below is a constexpr variable, so it is folded at
    // compile time (a constexpr call in a plain expression may be evaluated
    // on the device)
    constexpr uint64_t B0 = bias(0), B1 = bias(1), B2 = bias(2), B3 = bias(3), B4 = bias(4);
    constexpr uint64_t B5 = bias(5), B6 = bias(6), B7 = bias(7), B8 = bias(8), B9 = bias(9);
    constexpr double P0 = (double)p52<C>(0), P1 = (double)p52<C>(1), P2 = (double)p52<C>(2);
    constexpr double P3 = (double)p52<C>(3), P4 = (double)p52<C>(4);
    constexpr uint64_t NP = C::NP52;
    const double PD[5] = {P0, P1, P2, P3, P4};
    uint64_t col[10] = {0 - B0, 0 - B1, 0 - B2, 0 - B3, 0 - B4, 0 - B5, 0 - B6, 0 - B7, 0 - B8, 0 - B9};
#pragma unroll
    for (int i = 0; i < 5; i++) {
        uint64_t hp = 0;
#pragma unroll
        for (int j = 0; j < 5; j++) {
            const double h = __fma_rz(A[i], B[j], C104);
            const double lo = __fma_rn(A[i], B[j], __dsub_rn(C104_52, h));
            col[i + j] = j == 0 ? col[i + j] + dbits(lo) : col[i + j] + (dbits(lo) + hp);
            hp = dbits(h);
        }
        col[i + 5] += hp;
    }
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const uint64_t t = col[i];
        const uint64_t tl = t & M52;
        const double qd = u52d((tl * NP) & M52);
        uint64_t hp = dbits(__fma_rz(qd, PD[0], C104)) + (t >> 52) + (tl != 0 ? 1u : 0u);
#pragma unroll
        for (int j = 1; j < 5; j++) {
            const double pj = PD[j];
            const double h = __fma_rz(qd, pj, C104);
            const double lo = __fma_rn(qd, pj, __dsub_rn(C104_52, h));
            col[i + j] = col[i + j] + (dbits(lo) + hp);
            hp = dbits(h);
        }
        col[i + 5] += hp;
    }
    uint64_t c = 0;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const uint64_t x = col[5 + k] + c;
        l[k] = k < 4 ? (x & M52) : x;
        c = x >> 52;
    }
}
}  // namespace f64

template <class C>
H2B_DEV Fp<C> mont_mul_f64(const Fp<C>& a, const Fp<C>& b)
{
    using namespace f64;
    double A[5], B[5];
    A[0] = u52d(bits52<-4>(a.v)); A[1] = u52d(bits52<48>(a.v)); A[2] = u52d(bits52<100>(a.v));
    A[3] = u52d(bits52<152>(a.v)); A[4] = u52d(bits52<204>(a.v));
    B[0] = u52d(bits52<0>(b.v)); B[1] = u52d(bits52<52>(b.v)); B[2] = u52d(bits52<104>(b.v));
    B[3] = u52d(bits52<156>(b.v)); B[4] = u52d(bits52<208>(b.v));
    uint64_t l[5];
    mont52<C>(A, B, l);
    // 52-bit limbs -> 8 x 32 words
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int i0 = (32 * j) / 52, o = 32 * j - 52 * i0;
        uint64_t x = l[i0] >> o;
        if (i0 + 1 < 5) x |= l[i0 + 1] << (52 - o);
        w[j] = (uint32_t)x;
    }
    Fp<C> r;
    cond_sub<C>(r.v, w);
    return r;
}

// ---- residues in [0, 2p) ----------------------------------------------------
// A chain of products and sums (an NTT pass) can keep its values in [0, 2p)
// and make them canonical once at the end.  A product of a, b < 2p is below
// (4 p / 2^256 + 1) p < 1.76 p for both BN254 moduli (p < 2^253.6), so its
// closing subtraction can be left out; a sum below 4p (< 2^256) or a difference
// in (-2p, 2p) takes one correction by 2p.

// word w of 2m (8 x 32 grid)
template <class C>
__host__ __device__ constexpr uint32_t m2word(int w)
{
    return (mword<C>(w) << 1) | (w > 0 ? mword<C>(w - 1) >> 31 : 0u);
}

// (a + b) mod 2p in [0, 2p) for a, b < 2p
template <class C>
H2B_DEV Fp<C> add2p(const Fp<C>& a, const Fp<C>& b)
{
    uint32_t t[8], s[8], bw;
    asm("add.cc.u32  %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]),
          "=r"(bw)
        : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
          "n"(m2word<C>(0)), "n"(m2word<C>(1)), "n"(m2word<C>(2)), "n"(m2word<C>(3)), "n"(m2word<C>(4)),
          "n"(m2word<C>(5)), "n"(m2word<C>(6)), "n"(m2word<C>(7)));
    Fp<C> r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = bw ? t[i] : s[i];
    return r;
}

// (a - b) mod 2p in [0, 2p) for a, b < 2p
template <class C>
H2B_DEV Fp<C> sub2p(const Fp<C>& a, const Fp<C>& b)
{
    Fp<C> r;
    uint32_t bw;
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(bw)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    const uint32_t q0 = bw & m2word<C>(0), q1 = bw & m2word<C>(1), q2 = bw & m2word<C>(2), q3 = bw & m2word<C>(3);
    const uint32_t q4 = bw & m2word<C>(4), q5 = bw & m2word<C>(5), q6 = bw & m2word<C>(6), q7 = bw & m2word<C>(7);
    asm("add.cc.u32  %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, %9;\n\t"
        "addc.cc.u32 %2, %2, %10;\n\t"
        "addc.cc.u32 %3, %3, %11;\n\t"
        "addc.cc.u32 %4, %4, %12;\n\t"
        "addc.cc.u32 %5, %5, %13;\n\t"
        "addc.cc.u32 %6, %6, %14;\n\t"
        "addc.u32    %7, %7, %15;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]),
          "+r"(r.v[7])
        : "r"(q0), "r"(q1), "r"(q2), "r"(q3), "r"(q4), "r"(q5), "r"(q6), "r"(q7));
    return r;
}

// (a b + c d) 2^-256 mod p in [0, 2p) for a, b, c, d <= 2p: the sum's reduction
// leaves less than (8 p / 2^256 + 1) p < 2.52 p, one correction by 2p
template <class C>
H2B_DEV Fp<C> mont_mul_add_eo_lazy(const Fp<C>& a, const Fp<C>& b, const Fp<C>& c, const Fp<C>& d)
{
    uint32_t t[8], s[8], bw;
    eo_mont2<C>(t, a.v, b.v, c.v, d.v);
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]),
          "=r"(bw)
        : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]),
          "n"(m2word<C>(0)), "n"(m2word<C>(1)), "n"(m2word<C>(2)), "n"(m2word<C>(3)), "n"(m2word<C>(4)),
          "n"(m2word<C>(5)), "n"(m2word<C>(6)), "n"(m2word<C>(7)));
    Fp<C> r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = bw ? t[i] : s[i];
    return r;
}

// the canonical residue of a < 2p
template <class C>
H2B_DEV Fp<C> canon2p(const Fp<C>& a)
{
    Fp<C> r;
    cond_sub<C>(r.v, a.v);
    return r;
}

// operator* and fsqr.  The first factor must be below 2^256 - p (4.29 p; every
// canonical residue and every value below 2p is): beyond it a carry out of the
// ninth word is dropped.  The second may be any 256-bit value, and the product
// is canonical when the first is, so a value that comes from outside as it is
// (a caller's element, random words) stands second.
// One out-of-line body per field by default: kernels that chain many products
// (curve formulas) would inline two hundred instructions per product.
// H2B_INLINE_MUL=1 inlines them in a file.
#ifndef H2B_INLINE_MUL
#define H2B_INLINE_MUL 0
#endif
template <class C>
H2B_DEV Fp<C> mont_mul_sel(const Fp<C>& a, const Fp<C>& b)
{
    return mont_mul_eo<C>(a, b);
}

template <class C>
H2B_DEV Fp<C> mont_sqr_sel(const Fp<C>& a)
{
    return mont_sqr_eo<C>(a);
}

template <class C>
__device__ __noinline__ Fp<C> mont_mul_outline(const Fp<C> a, const Fp<C> b)
{
    return mont_mul_sel<C>(a, b);
}

template <class C>
__device__ __noinline__ Fp<C> mont_sqr_outline(const Fp<C> a)
{
    return mont_sqr_sel<C>(a);
}

// a b 2^-256 mod p in [0, 2p) for a, b < 2p, out of line (residues in [0, 2p) above)
template <class C>
__device__ __noinline__ Fp<C> mont_mul_lazy_outline(const Fp<C> a, const Fp<C> b)
{
    return mont_mul_eo_lazy<C>(a, b);
}

template <class C>
__device__ __noinline__ Fp<C> mont_sqr_lazy_outline(const Fp<C> a)
{
    return mont_sqr_eo_lazy<C>(a);
}

// a == 0 (mod p) for a < 2p: a is 0 or p
template <class C>
H2B_DEV bool is_zero2p(const Fp<C>& a)
{
    uint32_t z = 0, e = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        z |= a.v[i];
        e |= a.v[i] ^ mword<C>(i);
    }
    return z == 0 || e == 0;
}

template <class C>
H2B_DEV Fp<C> operator*(const Fp<C>& a, const Fp<C>& b)
{
#if H2B_INLINE_MUL
    return mont_mul_sel<C>(a, b);
#else
    return mont_mul_outline<C>(a, b);
#endif
}

template <class C>
H2B_DEV Fp<C> operator+(const Fp<C>& a, const Fp<C>& b)
{
    uint32_t t[8];
    asm("add.cc.u32  %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(t[0]), "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    Fp<C> r;
    cond_sub<C>(r.v, t);
    return r;
}

template <class C>
H2B_DEV Fp<C> operator-(const Fp<C>& a, const Fp<C>& b)
{
    Fp<C> r;
    uint32_t bw;
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7]), "=r"(bw)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    // On borrow add the modulus back (bw is 0 or all-ones).
    const uint32_t q0 = bw & C::M0, q1 = bw & C::M1, q2 = bw & C::M2, q3 = bw & C::M3;
    const uint32_t q4 = bw & C::M4, q5 = bw & C::M5, q6 = bw & C::M6, q7 = bw & C::M7;
    asm("add.cc.u32  %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, %9;\n\t"
        "addc.cc.u32 %2, %2, %10;\n\t"
        "addc.cc.u32 %3, %3, %11;\n\t"
        "addc.cc.u32 %4, %4, %12;\n\t"
        "addc.cc.u32 %5, %5, %13;\n\t"
        "addc.cc.u32 %6, %6, %14;\n\t"
        "addc.u32    %7, %7, %15;"
        : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]),
          "+r"(r.v[7])
        : "r"(q0), "r"(q1), "r"(q2), "r"(q3), "r"(q4), "r"(q5), "r"(q6), "r"(q7));
    return r;
}

template <class C>
H2B_DEV Fp<C>& operator*=(Fp<C>& a, const Fp<C>& b) { a = a * b; return a; }
template <class C>
H2B_DEV Fp<C>& operator+=(Fp<C>& a, const Fp<C>& b) { a = a + b; return a; }
template <class C>
H2B_DEV Fp<C>& operator-=(Fp<C>& a, const Fp<C>& b) { a = a - b; return a; }

template <class C>
H2B_DEV Fp<C> fneg(const Fp<C>& a) { return Fp<C>::zero() - a; }
template <class C>
H2B_DEV Fp<C> fdbl(const Fp<C>& a) { return a + a; }
template <class C>
H2B_DEV Fp<C> fsqr(const Fp<C>& a)
{
#if H2B_INLINE_MUL
    return mont_sqr_sel<C>(a);
#else
    return mont_sqr_outline<C>(a);
#endif
}

// Montgomery residue (any 256-bit value of its class) -> canonical integer (multiply by 1).
template <class C>
H2B_DEV Fp<C> from_mont(const Fp<C>& a)
{
    Fp<C> one_int = Fp<C>::zero();
    one_int.v[0] = 1;
    return one_int * a;
}
// any 256-bit integer -> its residue
template <class C>
H2B_DEV Fp<C> to_mont(const Fp<C>& a) { return Fp<C>::r2() * a; }

template <class C>
H2B_DEV Fp<C> ldg(const Fp<C>* p)
{
    Fp<C> r;
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 x = __ldg(q), y = __ldg(q + 1);
    r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w;
    r.v[4] = y.x; r.v[5] = y.y; r.v[6] = y.z; r.v[7] = y.w;
    return r;
}
template <class C>
H2B_DEV Fp<C> ld(const Fp<C>* p)
{
    Fp<C> r;
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 x = q[0], y = q[1];
    r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w;
    r.v[4] = y.x; r.v[5] = y.y; r.v[6] = y.z; r.v[7] = y.w;
    return r;
}
template <class C>
H2B_DEV void st(Fp<C>* p, const Fp<C>& a)
{
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
    q[1] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
}

} // namespace h2b
