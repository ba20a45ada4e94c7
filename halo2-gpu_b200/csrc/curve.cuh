// BN254 G1 (y^2 = x^3 + 3 over Fq) point arithmetic for the MSM.
//
// Affine points are 64 bytes {x, y} in Montgomery form with the point at
// infinity encoded as (0, 0) -- the halo2curves `G1Affine` memory image the
// reference passes to its MSM (halo2_proofs/cuda/include/curve/xyzz_t.hpp:49-50).
// Bucket accumulators use XYZZ coordinates (x = X/ZZ, y = Y/ZZZ, ZZ^3 = ZZZ^2,
// infinity <=> ZZ == 0) with the EFD formulas madd-2008-s (8M+2S),
// add-2008-s (12M+2S), mdbl-2008-s-1 and dbl-2008-s-1, written from the
// published formulas.  The MSM result leaves the device as the reference's
// 96-byte Jacobian image {X, Y, Z}: affine coordinates with Z = 1, or
// (0, 1, 0) for infinity (halo2_proofs/cuda/include/kernel/pippenger.h:659-668,
// halo2_proofs/cuda/include/curve/jacobian_t.hpp:64-83).
#pragma once
#include "field.cuh"
#include "inverse.cuh"
#include "lazy.cuh"

namespace h2b {

struct G1Affine {
    Fq x, y;
};

struct G1Xyzz {
    Fq X, Y, ZZ, ZZZ;
};

struct G1Jac {
    Fq X, Y, Z;
};

H2B_DEV bool is_inf(const G1Affine& p) { return p.x.is_zero() && p.y.is_zero(); }
H2B_DEV bool is_inf(const G1Xyzz& p) { return p.ZZ.is_zero(); }

H2B_DEV G1Xyzz xyzz_inf()
{
    G1Xyzz r;
    r.X = Fq::zero(); r.Y = Fq::zero(); r.ZZ = Fq::zero(); r.ZZZ = Fq::zero();
    return r;
}

H2B_DEV G1Affine ld_affine(const G1Affine* p)
{
    G1Affine r;
    r.x = ldg(&p->x);
    r.y = ldg(&p->y);
    return r;
}

H2B_DEV G1Xyzz ld_xyzz(const G1Xyzz* p)
{
    G1Xyzz r;
    r.X = ld(&p->X); r.Y = ld(&p->Y); r.ZZ = ld(&p->ZZ); r.ZZZ = ld(&p->ZZZ);
    return r;
}
H2B_DEV void st_xyzz(G1Xyzz* p, const G1Xyzz& a)
{
    st(&p->X, a.X); st(&p->Y, a.Y); st(&p->ZZ, a.ZZ); st(&p->ZZZ, a.ZZZ);
}

// mdbl-2008-s-1: double an affine point into XYZZ.
H2B_DEV G1Xyzz xyzz_dbl_affine(const G1Affine& p)
{
    if (is_inf(p) || p.y.is_zero()) return xyzz_inf();
    Fq U = fdbl(p.y);
    Fq V = fsqr(U);
    Fq W = U * V;
    Fq S = p.x * V;
    Fq xx = fsqr(p.x);
    Fq M = fdbl(xx) + xx;
    G1Xyzz r;
    r.X = fsqr(M) - fdbl(S);
    r.Y = M * (S - r.X) - W * p.y;
    r.ZZ = V;
    r.ZZZ = W;
    return r;
}

// dbl-2008-s-1 (a = 0).
H2B_DEV G1Xyzz xyzz_dbl(const G1Xyzz& p)
{
    if (is_inf(p) || p.Y.is_zero()) return xyzz_inf();
    Fq U = fdbl(p.Y);
    Fq V = fsqr(U);
    Fq W = U * V;
    Fq S = p.X * V;
    Fq xx = fsqr(p.X);
    Fq M = fdbl(xx) + xx;
    G1Xyzz r;
    r.X = fsqr(M) - fdbl(S);
    r.Y = M * (S - r.X) - W * p.Y;
    r.ZZ = V * p.ZZ;
    r.ZZZ = W * p.ZZZ;
    return r;
}

// madd-2008-s: acc += q (q affine), with the exceptional cases handled.
H2B_DEV void xyzz_madd(G1Xyzz& acc, const G1Affine& q)
{
    if (is_inf(q)) return;
    if (is_inf(acc)) {
        acc.X = q.x; acc.Y = q.y; acc.ZZ = Fq::one(); acc.ZZZ = Fq::one();
        return;
    }
    Fq U2 = q.x * acc.ZZ;
    Fq S2 = q.y * acc.ZZZ;
    Fq P = U2 - acc.X;
    Fq R = S2 - acc.Y;
    if (P.is_zero()) {
        if (R.is_zero()) acc = xyzz_dbl_affine(q);
        else acc = xyzz_inf();
        return;
    }
    Fq PP = fsqr(P);
    Fq PPP = P * PP;
    Fq Q = acc.X * PP;
    Fq X3 = fsqr(R) - PPP - fdbl(Q);
    acc.Y = R * (Q - X3) - acc.Y * PPP;
    acc.X = X3;
    acc.ZZ = acc.ZZ * PP;
    acc.ZZZ = acc.ZZZ * PPP;
}

// ---- XYZZ in the lazy form (R = 2^261), for the bucket accumulation -------
// Bounds (multiples of p) that every step relies on are written beside it;
// products follow (1 + 0.0059 a b) p (lazy.cuh).  The accumulator keeps
// X < 5.39p, Y < 3.34p, ZZ and ZZZ < 2p from one addition to the next;
// affine inputs are qx < 1.01p (canonical, or times beta) and qy < 2p
// (canonical, or negated as 2p - y).

typedef Fz<FqCfg> FqZ;

struct G1XyzzZ {
    FqZ X, Y, ZZ, ZZZ;
};

H2B_DEV G1XyzzZ xyzzz_inf()
{
    G1XyzzZ r;
    r.X = fz_zero<FqCfg>(); r.Y = fz_zero<FqCfg>(); r.ZZ = fz_zero<FqCfg>(); r.ZZZ = fz_zero<FqCfg>();
    return r;
}

// infinity is the explicit all-zero ZZ (no other path makes ZZ vanish)
H2B_DEV bool is_inf(const G1XyzzZ& p) { return fz_is_zero(p.ZZ); }

// 2 q for an affine q (qx < 1.01p, qy < 2p, qy != 0): dbl-2008-s-1 with Z = 1.
H2B_DEV G1XyzzZ xyzzz_dbl_affine(const FqZ& qx, const FqZ& qy)
{
    const FqZ U = fz_add(qy, qy);                              // < 4p
    const Fz2<FqCfg> vx = fz_sqr2(U, qx);                      // V < 1.094p, xx < 1.006p
    const Fz2<FqCfg> ws = fz_mul2(U, vx.a, qx, vx.a);          // W < 1.026p, S < 1.0065p
    const FqZ M = fz_add(fz_add(vx.b, vx.b), vx.b);            // < 3.02p
    const Fz2<FqCfg> mm = fz_mul2(M, M, ws.a, qy);             // MM < 1.054p, W y < 1.012p
    G1XyzzZ r;
    r.X = fz_sub<FqCfg, 3>(mm.a, fz_add(ws.b, ws.b));          // 2S < 2.013p; X3 < 4.054p
    const FqZ t1 = fz_mul_call(M, fz_sub<FqCfg, 5>(ws.b, r.X)); // S - X3 + 5p < 6.007p; t1 < 1.107p
    r.Y = fz_sub<FqCfg, 2>(t1, mm.b);                          // < 3.107p
    r.ZZ = vx.a;                                               // < 1.094p
    r.ZZZ = ws.a;                                              // < 1.026p
    return r;
}

// madd-2008-s: acc += (qx, qy), q affine and not infinity.  PP and R^2 are
// formed before the equal-x test (PP == 0 mod p exactly when P is).
H2B_DEV void xyzzz_madd(G1XyzzZ& acc, const FqZ& qx, const FqZ& qy, const FqZ& one)
{
    if (is_inf(acc)) {
        acc.X = qx; acc.Y = qy; acc.ZZ = one; acc.ZZZ = one;
        return;
    }
    const Fz2<FqCfg> us = fz_mul2(qx, acc.ZZ, qy, acc.ZZZ);   // U2 < 1.012p, S2 < 1.024p
    const FqZ P = fz_sub<FqCfg, 6>(us.a, acc.X);               // X1 < 5.39p; P < 7.01p
    const FqZ R = fz_sub<FqCfg, 4>(us.b, acc.Y);               // Y1 < 3.34p; R < 5.02p
    const Fz2<FqCfg> sq = fz_sqr2(P, R);                       // PP < 1.29p, RR < 1.149p
    if (fz_is_zero_mod(sq.a)) {
        acc = fz_is_zero_mod(sq.b) ? xyzzz_dbl_affine(qx, qy) : xyzzz_inf();
        return;
    }
    const Fz2<FqCfg> pq = fz_mul2(P, sq.a, acc.X, sq.a);       // PPP < 1.053p, Q < 1.041p
    const FqZ X3 = fz_sub<FqCfg, 4>(sq.b, fz_add(pq.a, fz_add(pq.b, pq.b)));  // PPP + 2Q < 3.135p; X3 < 5.149p
    const Fz2<FqCfg> yy = fz_mul2(R, fz_sub<FqCfg, 6>(pq.b, X3), acc.Y, pq.a); // Q - X3 + 6p < 7.041p;
                                                                              // < 1.209p, < 1.021p
    const Fz2<FqCfg> zz = fz_mul2(acc.ZZ, sq.a, acc.ZZZ, pq.a); // < 1.015p, < 1.012p
    acc.Y = fz_sub<FqCfg, 2>(yy.a, yy.b);                     // < 3.209p
    acc.X = X3;
    acc.ZZ = zz.a;
    acc.ZZZ = zz.b;
}

// Stores the canonical memory image of the accumulator (infinity stays
// ZZ = 0): four products by 2^256 mod p through the shared out-of-line
// product bodies, then the conditional subtractions.  Out of line itself, so
// the rarely taken store path does not crowd the addition loop's code.
static __device__ __noinline__ void st_xyzzz(G1Xyzz* dst, const G1XyzzZ p, const FqZ r256)
{
    const Fz2<FqCfg> a = fz_mul2(p.X, r256, p.Y, r256);    // X < 5.39p, Y < 3.34p: both < 1.032p
    const Fz2<FqCfg> b = fz_mul2(p.ZZ, r256, p.ZZZ, r256);  // < 1.012p
    G1Xyzz r;
    r.X = fz_canonical(a.a); r.Y = fz_canonical(a.b);
    r.ZZ = fz_canonical(b.a); r.ZZZ = fz_canonical(b.b);
    st_xyzz(dst, r);
}

// ---- XYZZ with coordinates in [0, 2p) ---------------------------------------
// The memory image with residues in [0, 2p): products without their closing
// subtraction (mont_mul_eo_lazy: 1.76p), sums and differences corrected by
// 2p.  Every function takes and returns coordinates below 2p; infinity is the
// all-zero ZZ (no product of nonzero residues is 0, and the exceptional cases
// write zeros).  INL: products inline (the bucket accumulation) or one shared
// out-of-line body per product (the tails, whose code must stay small).

template <bool INL>
H2B_DEV Fq qmul(const Fq& a, const Fq& b)
{
    return INL ? mont_mul_eo_lazy<FqCfg>(a, b) : mont_mul_lazy_outline<FqCfg>(a, b);
}

template <bool INL>
H2B_DEV Fq qsqr(const Fq& a)
{
    return INL ? mont_sqr_eo_lazy<FqCfg>(a) : mont_sqr_lazy_outline<FqCfg>(a);
}

H2B_DEV Fq qadd(const Fq& a, const Fq& b) { return add2p<FqCfg>(a, b); }
H2B_DEV Fq qsub(const Fq& a, const Fq& b) { return sub2p<FqCfg>(a, b); }

// 2p - a (a <= 2p): the complement that turns a subtraction into an addition
H2B_DEV Fq qneg2(const Fq& a)
{
    Fq r;
    asm("sub.cc.u32 %0, %16, %8;\n\tsubc.cc.u32 %1, %17, %9;\n\tsubc.cc.u32 %2, %18, %10;\n\t"
        "subc.cc.u32 %3, %19, %11;\n\tsubc.cc.u32 %4, %20, %12;\n\tsubc.cc.u32 %5, %21, %13;\n\t"
        "subc.cc.u32 %6, %22, %14;\n\tsubc.u32 %7, %23, %15;"
        : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]), "=&r"(r.v[6]),
          "=&r"(r.v[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "n"(m2word<FqCfg>(0)), "n"(m2word<FqCfg>(1)), "n"(m2word<FqCfg>(2)), "n"(m2word<FqCfg>(3)),
          "n"(m2word<FqCfg>(4)), "n"(m2word<FqCfg>(5)), "n"(m2word<FqCfg>(6)), "n"(m2word<FqCfg>(7)));
    return r;
}

// a b - c d, one reduction when the products are inline
template <bool INL>
H2B_DEV Fq qmulsub(const Fq& a, const Fq& b, const Fq& c, const Fq& d)
{
    return INL ? mont_mul_add_eo_lazy<FqCfg>(a, b, c, qneg2(d)) : qsub(qmul<INL>(a, b), qmul<INL>(c, d));
}

// the canonical memory image (infinity stays ZZ = 0)
H2B_DEV G1Xyzz xyzze_canonical(const G1Xyzz& a)
{
    G1Xyzz r;
    r.X = canon2p<FqCfg>(a.X); r.Y = canon2p<FqCfg>(a.Y);
    r.ZZ = canon2p<FqCfg>(a.ZZ); r.ZZZ = canon2p<FqCfg>(a.ZZZ);
    return r;
}
H2B_DEV void st_xyzze(G1Xyzz* p, const G1Xyzz& a) { st_xyzz(p, xyzze_canonical(a)); }

// 2 q for an affine q that is not infinity (y != 0 on this curve: the group order is odd)
template <bool INL>
__device__ __noinline__ G1Xyzz xyzze_dbl_affine(const Fq qx, const Fq qy)
{
    const Fq U = qadd(qy, qy), V = qsqr<INL>(U), xx = qsqr<INL>(qx);
    const Fq W = qmul<INL>(U, V), S = qmul<INL>(qx, V), M = qadd(qadd(xx, xx), xx);
    G1Xyzz r;
    r.X = qsub(qsqr<INL>(M), qadd(S, S));
    r.Y = qsub(qmul<INL>(M, qsub(S, r.X)), qmul<INL>(W, qy));
    r.ZZ = V;
    r.ZZZ = W;
    return r;
}

// dbl-2008-s-1 (a = 0)
template <bool INL>
H2B_DEV G1Xyzz xyzze_dbl(const G1Xyzz& p)
{
    if (is_inf(p)) return xyzz_inf();
    const Fq U = qadd(p.Y, p.Y), V = qsqr<INL>(U), xx = qsqr<INL>(p.X);
    const Fq W = qmul<INL>(U, V), S = qmul<INL>(p.X, V), M = qadd(qadd(xx, xx), xx);
    G1Xyzz r;
    r.ZZ = qmul<INL>(V, p.ZZ);
    r.ZZZ = qmul<INL>(W, p.ZZZ);
    r.X = qsub(qsqr<INL>(M), qadd(S, S));
    r.Y = qsub(qmul<INL>(M, qsub(S, r.X)), qmul<INL>(W, p.Y));
    return r;
}

// madd-2008-s: acc += (qx, qy), an affine point that is not infinity
template <bool INL>
H2B_DEV void xyzze_madd(G1Xyzz& acc, const Fq& qx, const Fq& qy)
{
    if (is_inf(acc)) {
        acc.X = qx; acc.Y = qy; acc.ZZ = Fq::one(); acc.ZZZ = Fq::one();
        return;
    }
    const Fq P = qsub(qmul<INL>(qx, acc.ZZ), acc.X);
    const Fq R = qsub(qmul<INL>(qy, acc.ZZZ), acc.Y);
    if (is_zero2p<FqCfg>(P)) {
        acc = is_zero2p<FqCfg>(R) ? xyzze_dbl_affine<false>(qx, qy) : xyzz_inf();
        return;
    }
    const Fq PP = qsqr<INL>(P);
    const Fq PPP = qmul<INL>(P, PP), Q = qmul<INL>(acc.X, PP);
    acc.ZZ = qmul<INL>(acc.ZZ, PP);
    acc.ZZZ = qmul<INL>(acc.ZZZ, PPP);
    acc.X = qsub(qsub(qsqr<INL>(R), PPP), qadd(Q, Q));
    acc.Y = qmulsub<INL>(R, qsub(Q, acc.X), acc.Y, PPP);
}

// add-2008-s: acc += q
template <bool INL>
H2B_DEV void xyzze_add(G1Xyzz& acc, const G1Xyzz& q)
{
    if (is_inf(q)) return;
    if (is_inf(acc)) { acc = q; return; }
    const Fq U1 = qmul<INL>(acc.X, q.ZZ), S1 = qmul<INL>(acc.Y, q.ZZZ);
    const Fq P = qsub(qmul<INL>(q.X, acc.ZZ), U1), R = qsub(qmul<INL>(q.Y, acc.ZZZ), S1);
    if (is_zero2p<FqCfg>(P)) {
        if (is_zero2p<FqCfg>(R)) acc = xyzze_dbl<INL>(acc);
        else acc = xyzz_inf();
        return;
    }
    const Fq PP = qsqr<INL>(P);
    const Fq PPP = qmul<INL>(P, PP), Q = qmul<INL>(U1, PP);
    acc.ZZ = qmul<INL>(qmul<INL>(acc.ZZ, q.ZZ), PP);
    acc.ZZZ = qmul<INL>(qmul<INL>(acc.ZZZ, q.ZZZ), PPP);
    acc.X = qsub(qsub(qsqr<INL>(R), PPP), qadd(Q, Q));
    acc.Y = qsub(qmul<INL>(R, qsub(Q, acc.X)), qmul<INL>(S1, PPP));
}

// ---- one warp per point: formulas over shared-memory slots --------------------
// A serial tail (doubling a window or bit sum many times, the sums of the
// results) is one dependent product after another.  Here a warp keeps its
// values in slots of shared memory; a level lets lane i take the i-th product
// of a formula (operands and result by slot number, five bits per lane in a
// literal), so a level costs one product's latency (860 cycles) and the
// exchange two 32-byte reads and one write per lane.  All values are below 2p.

H2B_DEV Fq sl_get(const Fq* sl, int i) { return ld(&sl[i]); }

// lane i < n: slot[(o >> 5 i) & 31] = slot[(a >> 5 i) & 31] * slot[(b >> 5 i) & 31]
H2B_DEV void sl_mul(Fq* sl, int n, uint32_t a, uint32_t b, uint32_t o)
{
    const int lane = (int)(threadIdx.x & 31);
    __syncwarp();
    Fq r;
    if (lane < n) r = mont_mul_eo_lazy<FqCfg>(sl[(a >> (5 * lane)) & 31], sl[(b >> (5 * lane)) & 31]);
    __syncwarp();
    if (lane < n) st(&sl[(o >> (5 * lane)) & 31], r);
    __syncwarp();
}

// (ca a + cb b + cc c) mod p, below 1.1p, for a, b, c <= 2p and ca + cb + cc <= 266:
// the sum stays below 2^264, and the quotient estimate from its bits above
// 2^248 is at most one short (2^280 / p rounded down is 88753990).
H2B_DEV Fq qlin(uint32_t ca, const Fq& a, uint32_t cb, const Fq& b, uint32_t cc, const Fq& c)
{
    // limb products first (independent), then one carry chain each way
    uint32_t lo[8], hi[8], w[9];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint64_t x = (uint64_t)ca * a.v[i] + (uint64_t)cb * b.v[i] + (uint64_t)cc * c.v[i];
        lo[i] = (uint32_t)x;
        hi[i] = (uint32_t)(x >> 32);
    }
    w[0] = lo[0];
    asm("add.cc.u32 %0, %8, %16;\n\taddc.cc.u32 %1, %9, %17;\n\taddc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\taddc.cc.u32 %4, %12, %20;\n\taddc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\taddc.u32 %7, %15, 0;"
        : "=&r"(w[1]), "=&r"(w[2]), "=&r"(w[3]), "=&r"(w[4]), "=&r"(w[5]), "=&r"(w[6]), "=&r"(w[7]), "=&r"(w[8])
        : "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]), "r"(hi[4]), "r"(hi[5]), "r"(hi[6]), "r"(hi[7]), "r"(lo[1]),
          "r"(lo[2]), "r"(lo[3]), "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7]));
    const uint32_t q = __umulhi((w[7] >> 24) | (w[8] << 8), 88753990u);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint64_t x = (uint64_t)q * mword<FqCfg>(i);
        lo[i] = (uint32_t)x;
        hi[i] = (uint32_t)(x >> 32);
    }
    asm("add.cc.u32 %0, %0, %7;\n\taddc.cc.u32 %1, %1, %8;\n\taddc.cc.u32 %2, %2, %9;\n\t"
        "addc.cc.u32 %3, %3, %10;\n\taddc.cc.u32 %4, %4, %11;\n\taddc.cc.u32 %5, %5, %12;\n\taddc.u32 %6, %6, %13;"
        : "+r"(lo[1]), "+r"(lo[2]), "+r"(lo[3]), "+r"(lo[4]), "+r"(lo[5]), "+r"(lo[6]), "+r"(lo[7])
        : "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]), "r"(hi[4]), "r"(hi[5]), "r"(hi[6]));
    Fq r;
    asm("sub.cc.u32 %0, %8, %16;\n\tsubc.cc.u32 %1, %9, %17;\n\tsubc.cc.u32 %2, %10, %18;\n\t"
        "subc.cc.u32 %3, %11, %19;\n\tsubc.cc.u32 %4, %12, %20;\n\tsubc.cc.u32 %5, %13, %21;\n\t"
        "subc.cc.u32 %6, %14, %22;\n\tsubc.u32 %7, %15, %23;"
        : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]), "=&r"(r.v[6]),
          "=&r"(r.v[7])
        : "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(lo[0]), "r"(lo[1]),
          "r"(lo[2]), "r"(lo[3]), "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7]));
    return r;
}

// 2^m times the XYZZ point in slots 0..3 (X, Y, ZZ, ZZZ; not infinity), in place.
// The x coordinate alone goes through the doublings: with x = X / Z,
//   X' = X^4 - 24 X Z^3,  Z' = 4 X^3 Z + 12 Z^4      (b = 3)
// which is two levels deep instead of the three of dbl-2008-s-1.  With
// C = X^3 Z and D = Z^4 the y coordinate is multiplied by
//   (2 C^2 + 120 C D - 144 D^2) / Z'^2
// at every doubling, whose numerators and denominators are collected by two
// further lanes one and two steps behind.  No point of this curve has order
// two (the group order is an odd prime), so Z never vanishes.
// Slots used: 0..15.
H2B_DEV void sl_dbl_many(Fq* sl, int m)
{
    if (m == 0) return;
    const int lane = (int)(threadIdx.x & 31);
    enum { X = 0, YN = 1, Z = 2, YD = 3, X2 = 4, Z2 = 5, XZ = 6, CC = 7, CD = 8, DD = 9, A = 10, B = 11, C = 12, D = 13,
           M = 14, ONE = 15 };
#define SL6(a, b, c, d, e, f) \
    ((uint32_t)(a) | (uint32_t)(b) << 5 | (uint32_t)(c) << 10 | (uint32_t)(d) << 15 | (uint32_t)(e) << 20 | (uint32_t)(f) << 25)
    if (lane == 0) st(&sl[M], Fq::one());
    if (lane == 1) st(&sl[ONE], Fq::one());
    if (lane == 2) st(&sl[C], Fq::one());
    if (lane == 3) st(&sl[D], Fq::one());
#pragma unroll 1
    for (int i = 0; i <= m; i++) {
        sl_mul(sl, 6, SL6(X, Z, X, C, C, D), SL6(X, Z, Z, C, D, D), SL6(X2, Z2, XZ, CC, CD, DD));
        sl_mul(sl, 6, SL6(X2, XZ, XZ, Z2, YN, YD), SL6(X2, Z2, X2, Z2, M, i ? Z2 : ONE), SL6(A, B, C, D, YN, YD));
        // lane 0: X' = A - 24 B; lane 1: Z' = 4 C + 12 D; lane 2: M = 2 CC + 120 CD - 144 DD of the step before
        if (lane < 3) {
            const Fq a = sl[lane == 0 ? A : lane == 1 ? C : CC];
            Fq b = sl[lane == 0 ? B : lane == 1 ? D : CD];
            const Fq c = qneg2(sl[DD]);
            if (lane == 0) b = qneg2(b);
            const Fq r = qlin(lane == 0 ? 1u : lane == 1 ? 4u : 2u, a, lane == 0 ? 24u : lane == 1 ? 12u : 120u, b,
                              lane == 2 ? 144u : 0u, c);
            if (lane == 2) { if (i) st(&sl[M], r); }
            else if (i < m) st(&sl[lane == 0 ? X : Z], r);
        }
        __syncwarp();
    }
    // x = X / Z, y = YN M / YD: with t = Z YD, ZZ = t^2, ZZZ = t^3, X' = X YD t, Y' = (YN M) Z t^2
    sl_mul(sl, 3, SL6(YN, Z, X, 0, 0, 0), SL6(M, YD, YD, 0, 0, 0), SL6(YN, A, B, 0, 0, 0));
    sl_mul(sl, 3, SL6(A, B, YN, 0, 0, 0), SL6(A, A, Z, 0, 0, 0), SL6(C, X, D, 0, 0, 0));
    sl_mul(sl, 2, SL6(C, D, 0, 0, 0, 0), SL6(A, C, 0, 0, 0, 0), SL6(YD, YN, 0, 0, 0, 0));
    if (lane == 0) st(&sl[Z], sl_get(sl, C));
    __syncwarp();
}

// slots 0..3 += slots 4..7 (XYZZ points, add-2008-s in four product levels).  Slots used: 0..19.
H2B_DEV void sl_add(Fq* sl)
{
    const int lane = (int)(threadIdx.x & 31);
    __syncwarp();
    if (sl_get(sl, 6).is_zero()) return;
    if (sl_get(sl, 2).is_zero()) {
        Fq t;
        if (lane < 4) t = sl_get(sl, 4 + lane);
        __syncwarp();
        if (lane < 4) st(&sl[lane], t);
        __syncwarp();
        return;
    }
    enum { X1 = 0, Y1 = 1, ZZ1 = 2, ZZZ1 = 3, XX2 = 4, YY2 = 5, ZZ2 = 6, ZZZ2 = 7, U1 = 8, U2 = 9, S1 = 10, S2 = 11,
           P = 12, RR = 13, PP = 14, R2 = 15, PPP = 16, QQ = 17, T = 18, W = 19 };
    sl_mul(sl, 6, SL6(X1, XX2, Y1, YY2, ZZ1, ZZZ1), SL6(ZZ2, ZZ1, ZZZ2, ZZZ1, ZZ2, ZZZ2), SL6(U1, U2, S1, S2, ZZ1, ZZZ1));
    if (lane < 2) st(&sl[lane ? RR : P], qsub(sl[lane ? S2 : U2], sl[lane ? S1 : U1]));
    __syncwarp();
    if (is_zero2p<FqCfg>(sl_get(sl, P))) {     // equal x: a doubling or P + (-P); slots 4..7 still hold the second point
        const bool dbl = is_zero2p<FqCfg>(sl_get(sl, RR));
        __syncwarp();
        if (lane == 0) {
            G1Xyzz q;
            q.X = sl[XX2]; q.Y = sl[YY2]; q.ZZ = sl[ZZ2]; q.ZZZ = sl[ZZZ2];
            q = dbl ? xyzze_dbl<false>(q) : xyzz_inf();
            st(&sl[X1], q.X); st(&sl[Y1], q.Y); st(&sl[ZZ1], q.ZZ); st(&sl[ZZZ1], q.ZZZ);
        }
        __syncwarp();
        return;
    }
    sl_mul(sl, 2, SL6(P, RR, 0, 0, 0, 0), SL6(P, RR, 0, 0, 0, 0), SL6(PP, R2, 0, 0, 0, 0));
    sl_mul(sl, 3, SL6(P, U1, ZZ1, 0, 0, 0), SL6(PP, PP, PP, 0, 0, 0), SL6(PPP, QQ, ZZ1, 0, 0, 0));
    if (lane == 0) {
        const Fq q = sl[QQ], x = qsub(qsub(sl[R2], sl[PPP]), qadd(q, q));
        st(&sl[X1], x);
        st(&sl[T], qsub(q, x));
    }
    sl_mul(sl, 3, SL6(RR, S1, ZZZ1, 0, 0, 0), SL6(T, PPP, PPP, 0, 0, 0), SL6(T, W, ZZZ1, 0, 0, 0));
    if (lane == 0) st(&sl[Y1], qsub(sl[T], sl[W]));
    __syncwarp();
}
#undef SL6

// XYZZ -> reference Jacobian image (affine with Z = 1; infinity = (0, 1, 0)).
H2B_DEV G1Jac xyzz_to_jac_affine(const G1Xyzz& p)
{
    G1Jac r;
    if (is_inf(p)) {
        r.X = Fq::zero(); r.Y = Fq::one(); r.Z = Fq::zero();
        return r;
    }
    Fq inv = finv_fast(p.ZZ * p.ZZZ); // 1 / (ZZ * ZZZ)
    Fq izz = inv * p.ZZZ;             // 1 / ZZ
    Fq izzz = inv * p.ZZ;             // 1 / ZZZ
    r.X = p.X * izz;
    r.Y = p.Y * izzz;
    r.Z = Fq::one();
    return r;
}

} // namespace h2b
