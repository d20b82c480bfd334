// curve.cuh -- BN254 point arithmetic for the MSM kernels: G1 (y^2 = x^3 + 3 over Fq)
// and G2 (the sextic twist y^2 = x^3 + 3/(9 + u) over Fq2 = Fq[u]/(u^2 + 1)).
//
// Bases are affine (x, y) in Montgomery form (64 bytes for G1, 128 for G2); the point at
// infinity is stored as all-zero coordinates, which is on neither curve. Bucket
// accumulators use XYZZ coordinates (x = X/ZZ, y = Y/ZZZ, ZZ^3 = ZZZ^2), infinity is
// ZZ == 0. The formulas are the published short-Weierstrass a = 0 XYZZ formulas
// (madd-2008-s, add-2008-s, dbl-2008-s-1, mdbl-2008-s-1 of the Explicit-Formulas
// Database); they do not involve b, so one generic version serves both groups. They are
// made complete by handling infinity, P == Q (doubling) and P == -Q (infinity)
// explicitly -- the same cases the reference's Jacobian code handles
// (runtime/metal/ecc_source.py:206-293; G2 in crypto/ecc/bn254.py via py_ecc).
#pragma once
#include "field.cuh"

namespace zk {

// ---- Fq2 = Fq[u] / (u^2 + 1) ------------------------------------------------------------
struct __align__(16) fq2 {
    fe c0, c1;  // c0 + c1 u
};

// ---- coordinate operations, overloaded for Fq (fe) and Fq2 (fq2) ------------------------
__device__ __forceinline__ fe c_add(const fe& a, const fe& b) { return fe_add<FqP>(a, b); }
__device__ __forceinline__ fe c_sub(const fe& a, const fe& b) { return fe_sub<FqP>(a, b); }
__device__ __forceinline__ fe c_dbl(const fe& a) { return fe_dbl<FqP>(a); }
__device__ __forceinline__ fe c_neg(const fe& a) { return fe_neg<FqP>(a); }
__device__ __forceinline__ fe c_mul(const fe& a, const fe& b) { return fe_mul<FqP>(a, b); }
__device__ __forceinline__ fe c_sqr(const fe& a) { return fe_sqr<FqP>(a); }
// a b - c d with one reduction (field.cuh, separated forms)
__device__ __forceinline__ fe c_mul_sub(const fe& a, const fe& b, const fe& c, const fe& d) {
    return fe_mul_sub<FqP>(a, b, c, d);
}
// zero mod q: the curve formulas keep Fq values lazy in [0, 2q) (field.cuh)
__device__ __forceinline__ bool c_is_zero(const fe& a) { return fe_is_zero_mod<FqP, true>(a); }
__device__ __forceinline__ void c_set_zero(fe& a) { a = fe_zero(); }
__device__ __forceinline__ void c_set_one(fe& a) { a = fe_one<FqP>(); }
__device__ __forceinline__ fe c_ldg(const fe* p) { return fe_ldg(p); }
__device__ __forceinline__ fe c_load(const fe* p) { return fe_load(p); }
__device__ __forceinline__ void c_store(fe* p, const fe& a) { fe_store(p, a); }

template <class T>
struct c_pair {
    T x, y;
};

// Two independent products.
__device__ __forceinline__ c_pair<fe> c_mul2(const fe& a, const fe& b, const fe& c, const fe& d) {
    return {c_mul(a, b), c_mul(c, d)};
}

__device__ __forceinline__ fq2 c_add(const fq2& a, const fq2& b) { return {c_add(a.c0, b.c0), c_add(a.c1, b.c1)}; }
__device__ __forceinline__ fq2 c_sub(const fq2& a, const fq2& b) { return {c_sub(a.c0, b.c0), c_sub(a.c1, b.c1)}; }
__device__ __forceinline__ fq2 c_dbl(const fq2& a) { return {c_dbl(a.c0), c_dbl(a.c1)}; }
__device__ __forceinline__ fq2 c_neg(const fq2& a) { return {c_neg(a.c0), c_neg(a.c1)}; }
// (a0 + a1 u)(b0 + b1 u) = (a0 b0 - a1 b1) + (a0 b1 + a1 b0) u, Karatsuba with lazy reduction: the u
// coefficient is (a0 + a1)(b0 + b1) - a0 b0 - a1 b1, 3 unreduced 512-bit products and 2 reductions.
// Measured, G2 MSM, lazy / 3 full products: 2^16 1.13 / 1.27 ms (accumulation 0.64 / 0.77), 2^18 3.16 /
// 3.46, 500000 points 5.02 / 5.52; a0 b0 - a1 b1, a0 b1 + a1 b0 (4 products, 2 reductions) was 15% slower
// than 3 full products in the accumulation when it was measured, with add-carry chains.
__device__ __forceinline__ fq2 c_mul(const fq2& a, const fq2& b) {
    const fe_pair r = fe2_mul_lazy_call<FqP>(a.c0, a.c1, b.c0, b.c1);
    return {r.c0, r.c1};
}
// (a0 + a1 u)^2 = (a0 + a1)(a0 - a1) + 2 a0 a1 u: 2 products
__device__ __forceinline__ fq2 c_sqr(const fq2& a) {
    const fe t0 = c_mul(c_add(a.c0, a.c1), c_sub(a.c0, a.c1));
    const fe t1 = c_mul(a.c0, a.c1);
    return {t0, c_dbl(t1)};
}
__device__ __forceinline__ bool c_is_zero(const fq2& a) {
    return fe_is_zero_mod<FqP>(a.c0) && fe_is_zero_mod<FqP>(a.c1);
}
__device__ __forceinline__ void c_set_zero(fq2& a) {
    a.c0 = fe_zero();
    a.c1 = fe_zero();
}
__device__ __forceinline__ void c_set_one(fq2& a) {
    a.c0 = fe_one<FqP>();
    a.c1 = fe_zero();
}
__device__ __forceinline__ fq2 c_ldg(const fq2* p) { return {fe_ldg(&p->c0), fe_ldg(&p->c1)}; }
__device__ __forceinline__ fq2 c_load(const fq2* p) { return {fe_load(&p->c0), fe_load(&p->c1)}; }
__device__ __forceinline__ void c_store(fq2* p, const fq2& a) {
    fe_store(&p->c0, a.c0);
    fe_store(&p->c1, a.c1);
}
__device__ __forceinline__ c_pair<fq2> c_mul2(const fq2& a, const fq2& b, const fq2& c, const fq2& d) {
    return {c_mul(a, b), c_mul(c, d)};
}

// Pairs with squares, {a^2, b^2} and {a^2, c d}: over Fq a square has its own product form
// (field.cuh); over Fq2 a square takes 2 Fq products instead of 3. c_mul_sub(a, b, c, d) = a b - c d, one reduction over Fq.
__device__ __forceinline__ c_pair<fe> c_sqr2(const fe& a, const fe& b) {
    return {c_sqr(a), c_sqr(b)};
}
__device__ __forceinline__ c_pair<fe> c_sqr_mul(const fe& a, const fe& c, const fe& d) {
    return {c_sqr(a), c_mul(c, d)};
}
__device__ __forceinline__ fq2 c_mul_sub(const fq2& a, const fq2& b, const fq2& c, const fq2& d) {
    return c_sub(c_mul(a, b), c_mul(c, d));
}
__device__ __forceinline__ c_pair<fq2> c_sqr2(const fq2& a, const fq2& b) { return {c_sqr(a), c_sqr(b)}; }
__device__ __forceinline__ c_pair<fq2> c_sqr_mul(const fq2& a, const fq2& c, const fq2& d) {
    return {c_sqr(a), c_mul(c, d)};
}

// ---- points -------------------------------------------------------------------------------
template <class T>
struct __align__(16) AffineT {
    T x, y;
};

template <class T>
struct __align__(16) XyzzT {
    T X, Y, ZZ, ZZZ;
};

using affine_t = AffineT<fe>;
using xyzz_t = XyzzT<fe>;
using affine2_t = AffineT<fq2>;
using xyzz2_t = XyzzT<fq2>;

template <class T>
__device__ __forceinline__ bool affine_is_inf(const AffineT<T>& p) {
    return c_is_zero(p.x) && c_is_zero(p.y);
}

// OR of every limb of a coordinate
__device__ __forceinline__ uint32_t c_bits_or(const fe& a) {
    return a.v[0] | a.v[1] | a.v[2] | a.v[3] | a.v[4] | a.v[5] | a.v[6] | a.v[7];
}
__device__ __forceinline__ uint32_t c_bits_or(const fq2& a) { return c_bits_or(a.c0) | c_bits_or(a.c1); }

// The stored form of infinity in a base array: all bits zero. Exact for stored bases: the
// Montgomery conversion keeps 0 at 0, and no point of either curve has x = y = 0.
template <class T>
__device__ __forceinline__ bool affine_is_zero_bits(const AffineT<T>& p) {
    return (c_bits_or(p.x) | c_bits_or(p.y)) == 0;
}

template <class T = fe>
__device__ __forceinline__ XyzzT<T> xyzz_inf() {
    XyzzT<T> r;
    c_set_zero(r.X);
    c_set_zero(r.Y);
    c_set_zero(r.ZZ);
    c_set_zero(r.ZZZ);
    return r;
}

template <class T>
__device__ __forceinline__ bool xyzz_is_inf(const XyzzT<T>& p) {
    return c_is_zero(p.ZZ);
}

template <class T>
__device__ __forceinline__ XyzzT<T> xyzz_neg(const XyzzT<T>& p) {
    XyzzT<T> r = p;
    r.Y = c_neg(p.Y);
    return r;
}

// The formulas below list their independent multiplications in pairs (c_mul2).

// 2 * (x, y) for an affine point that is not infinity (y != 0 on these curves).
template <class T>
__device__ __forceinline__ XyzzT<T> xyzz_dbl_affine(const T& x, const T& y) {
    const T U = c_dbl(y);
    const c_pair<T> vx = c_sqr2(U, x);              // V = U^2, x^2
    const c_pair<T> ws = c_mul2(U, vx.x, x, vx.x);  // W = U V, S = x V
    const T M = c_add(c_dbl(vx.y), vx.y);
    const T MM = c_sqr(M);
    XyzzT<T> r;
    r.X = c_sub(MM, c_dbl(ws.y));
    r.Y = c_mul_sub(M, c_sub(ws.y, r.X), ws.x, y);
    r.ZZ = vx.x;
    r.ZZZ = ws.x;
    return r;
}

template <class T>
__device__ __forceinline__ XyzzT<T> xyzz_dbl(const XyzzT<T>& p) {
    if (xyzz_is_inf(p)) return p;
    const T U = c_dbl(p.Y);
    const c_pair<T> vx = c_sqr2(U, p.X);              // V = U^2, X^2
    const c_pair<T> ws = c_mul2(U, vx.x, p.X, vx.x);  // W = U V, S = X V
    const T M = c_add(c_dbl(vx.y), vx.y);
    const c_pair<T> mz = c_sqr_mul(M, vx.x, p.ZZ);  // M^2, ZZ3 = V ZZ
    XyzzT<T> r;
    r.X = c_sub(mz.x, c_dbl(ws.y));
    r.Y = c_mul_sub(M, c_sub(ws.y, r.X), ws.x, p.Y);
    r.ZZ = mz.y;
    r.ZZZ = c_mul(ws.x, p.ZZZ);
    return r;
}

// The products of a formula: through the one non-inlined copy, or (Inline) inlined at every
// site, for a loop that holds one formula and runs it often enough to keep it in the
// instruction cache.
template <class T>
struct CallOps {
    static __device__ __forceinline__ T mul(const T& a, const T& b) { return c_mul(a, b); }
    static __device__ __forceinline__ T sqr(const T& a) { return c_sqr(a); }
    static __device__ __forceinline__ T mul_sub(const T& a, const T& b, const T& c, const T& d) {
        return c_mul_sub(a, b, c, d);
    }
};

template <class T>
struct InlineOps;
template <>
struct InlineOps<fe> {
    static __device__ __forceinline__ fe mul(const fe& a, const fe& b) { return mul_rows<FqP>(a, b); }
    static __device__ __forceinline__ fe sqr(const fe& a) { return fe_sqr_sos<FqP>(a); }
    static __device__ __forceinline__ fe mul_sub(const fe& a, const fe& b, const fe& c, const fe& d) {
        return fe_mul_sub_sos<FqP>(a, b, c, d);
    }
};
template <>
struct InlineOps<fq2> {
    static __device__ __forceinline__ fq2 mul(const fq2& a, const fq2& b) {
        const fe_pair r = fe2_mul_lazy<FqP>(a.c0, a.c1, b.c0, b.c1);
        return {r.c0, r.c1};
    }
    static __device__ __forceinline__ fq2 sqr(const fq2& a) {
        const fe t0 = mul_rows<FqP>(c_add(a.c0, a.c1), c_sub(a.c0, a.c1));
        return {t0, c_dbl(mul_rows<FqP>(a.c0, a.c1))};
    }
    static __device__ __forceinline__ fq2 mul_sub(const fq2& a, const fq2& b, const fq2& c, const fq2& d) {
        return c_sub(mul(a, b), mul(c, d));
    }
};

// acc + (x, y), (x, y) affine and not infinity.
template <class T, class Ops = CallOps<T>>
__device__ __forceinline__ XyzzT<T> xyzz_madd(const XyzzT<T>& acc, const T& x, const T& y) {
    if (xyzz_is_inf(acc)) {
        XyzzT<T> r;
        r.X = x;
        r.Y = y;
        c_set_one(r.ZZ);
        c_set_one(r.ZZZ);
        return r;
    }
    const T P = c_sub(Ops::mul(x, acc.ZZ), acc.X);   // U2 - X
    const T R = c_sub(Ops::mul(y, acc.ZZZ), acc.Y);  // S2 - Y
    if (c_is_zero(P)) {
        if (c_is_zero(R)) return xyzz_dbl_affine(x, y);
        return xyzz_inf<T>();
    }
    const T PP = Ops::sqr(P);
    XyzzT<T> r;
    r.ZZ = Ops::mul(acc.ZZ, PP);
    const T PPP = Ops::mul(P, PP);
    const T Q = Ops::mul(acc.X, PP);
    r.ZZZ = Ops::mul(acc.ZZZ, PPP);
    r.X = c_sub(c_sub(Ops::sqr(R), PPP), c_dbl(Q));
    r.Y = Ops::mul_sub(R, c_sub(Q, r.X), acc.Y, PPP);
    return r;
}

template <class T>
__device__ __forceinline__ XyzzT<T> xyzz_add(const XyzzT<T>& p, const XyzzT<T>& q) {
    if (xyzz_is_inf(p)) return q;
    if (xyzz_is_inf(q)) return p;
    const c_pair<T> u = c_mul2(p.X, q.ZZ, q.X, p.ZZ);    // U1, U2
    const c_pair<T> s = c_mul2(p.Y, q.ZZZ, q.Y, p.ZZZ);  // S1, S2
    const T P = c_sub(u.y, u.x);
    const T R = c_sub(s.y, s.x);
    if (c_is_zero(P)) {
        if (c_is_zero(R)) return xyzz_dbl(p);
        return xyzz_inf<T>();
    }
    const c_pair<T> pr = c_sqr2(P, R);                // PP, R^2
    const c_pair<T> pq = c_mul2(P, pr.x, u.x, pr.x);  // PPP, Q
    const c_pair<T> zz = c_mul2(p.ZZ, q.ZZ, p.ZZZ, q.ZZZ);
    XyzzT<T> r;
    r.X = c_sub(c_sub(pr.y, pq.x), c_dbl(pq.y));
    const c_pair<T> z3 = c_mul2(zz.x, pr.x, zz.y, pq.x);
    r.Y = c_mul_sub(R, c_sub(pq.y, r.X), s.x, pq.x);
    r.ZZ = z3.x;
    r.ZZZ = z3.y;
    return r;
}

template <class T>
__device__ __forceinline__ AffineT<T> affine_load(const AffineT<T>* p) {
    AffineT<T> r;
    r.x = c_ldg(&p->x);
    r.y = c_ldg(&p->y);
    return r;
}

template <class T>
__device__ __forceinline__ XyzzT<T> xyzz_load(const XyzzT<T>* p) {
    XyzzT<T> r;
    r.X = c_load(&p->X);
    r.Y = c_load(&p->Y);
    r.ZZ = c_load(&p->ZZ);
    r.ZZZ = c_load(&p->ZZZ);
    return r;
}

// The same through L2 only (points written earlier in the same launch by other CTAs).
__device__ __forceinline__ fe c_ldcg(const fe* p) { return fe_ldcg(p); }
__device__ __forceinline__ fq2 c_ldcg(const fq2* p) { return {fe_ldcg(&p->c0), fe_ldcg(&p->c1)}; }

template <class T>
__device__ __forceinline__ XyzzT<T> xyzz_ldcg(const XyzzT<T>* p) {
    XyzzT<T> r;
    r.X = c_ldcg(&p->X);
    r.Y = c_ldcg(&p->Y);
    r.ZZ = c_ldcg(&p->ZZ);
    r.ZZZ = c_ldcg(&p->ZZZ);
    return r;
}

// xyzz_load, or xyzz_ldcg when kL2 (inputs produced in the same launch)
template <bool kL2, class T>
__device__ __forceinline__ XyzzT<T> xyzz_get(const XyzzT<T>* p) {
    if constexpr (kL2) return xyzz_ldcg(p);
    else return xyzz_load(p);
}

template <class T>
__device__ __forceinline__ void xyzz_store(XyzzT<T>* p, const XyzzT<T>& a) {
    c_store(&p->X, a.X);
    c_store(&p->Y, a.Y);
    c_store(&p->ZZ, a.ZZ);
    c_store(&p->ZZZ, a.ZZZ);
}

// ---- points held by four lanes -------------------------------------------------------------
// A quad (lanes 4k .. 4k + 3 of a warp) holds one point, lane l its l-th coordinate (X, Y, ZZ,
// ZZZ), and adds two points with the four independent products of each step side by side: 4
// product times instead of 13, at 16 product slots instead of 13 products. For the trees and
// chains of the window reduction and the fixup, whose threads are too few to fill the chip:
// one addition takes a warp ~4.6 us alone with a point per thread, ~2 us with a point per
// quad. Every lane of the warp calls; quads without work pass infinity (all zero).
template <class T>
struct QuadOps {
    using Ops = InlineOps<T>;
};
template <>
struct QuadOps<fq2> {
    using Ops = CallOps<fq2>;  // four inlined Fq2 products would fill the instruction cache
};

__device__ __forceinline__ fe c_shfl(const fe& a, int src) {  // src: lane of the quad
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_sync(0xffffffffu, a.v[i], src, 4);
    return r;
}
__device__ __forceinline__ fe c_shfl_xor(const fe& a, int mask) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_xor_sync(0xffffffffu, a.v[i], mask);
    return r;
}
__device__ __forceinline__ fq2 c_shfl(const fq2& a, int src) { return {c_shfl(a.c0, src), c_shfl(a.c1, src)}; }
__device__ __forceinline__ fq2 c_shfl_xor(const fq2& a, int mask) {
    return {c_shfl_xor(a.c0, mask), c_shfl_xor(a.c1, mask)};
}
__device__ __forceinline__ fe c_sel(bool c, const fe& a, const fe& b) {  // c ? a : b
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = c ? a.v[i] : b.v[i];
    return r;
}
__device__ __forceinline__ fq2 c_sel(bool c, const fq2& a, const fq2& b) {
    return {c_sel(c, a.c0, b.c0), c_sel(c, a.c1, b.c1)};
}

// The lane's coordinate of 2 P (rare: a quad whose two points are equal): gathered, doubled by
// every lane, its own coordinate taken.
template <class T>
__device__ __noinline__ T quad_dbl(const T p) {
    const int l = threadIdx.x & 3;
    const XyzzT<T> d = xyzz_dbl(XyzzT<T>{c_shfl(p, 0), c_shfl(p, 1), c_shfl(p, 2), c_shfl(p, 3)});
    return c_sel(l < 2, c_sel(l == 0, d.X, d.Y), c_sel(l == 2, d.ZZ, d.ZZZ));
}

// The lane's coordinate of P + Q (the formula and cases of xyzz_add).
template <class T>
__device__ __forceinline__ T quad_add(const T& p, const T& q) {
    using Ops = typename QuadOps<T>::Ops;
    const int l = threadIdx.x & 3;
    const uint32_t inf = __shfl_sync(0xffffffffu, (c_is_zero(p) ? 1u : 0u) | (c_is_zero(q) ? 2u : 0u), 2, 4);
    const T m1 = Ops::mul(p, c_shfl_xor(q, 2));  // U1 = X1 ZZ2, S1 = Y1 ZZZ2, U2 = ZZ1 X2, S2 = ZZZ1 Y2
    const T o1 = c_shfl_xor(m1, 2);              // U2, S2, U1, S1
    const T d = c_sub(c_sel(l < 2, o1, m1), c_sel(l < 2, m1, o1));        // P, R, P, R
    const uint32_t dz = c_is_zero(d) ? 1u : 0u;
    const T m2 = Ops::mul(c_sel(l < 2, d, p), c_sel(l < 2, d, q));        // P^2, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
    const T PP = c_shfl(m2, 0);
    const T U1 = c_shfl(m1, 0);
    const T m3 = Ops::mul(c_sel(l == 0, d, c_sel(l == 1, U1, m2)), PP);   // PPP, Q, ZZ3, -
    const T PPP = c_shfl(m3, 0);
    const T S1 = c_shfl(m1, 1);
    const T X3 = c_sub(c_sub(m2, PPP), c_dbl(m3));                        // lane 1: R^2 - PPP - 2 Q
    const T m4 = Ops::mul(c_sel(l == 1, d, c_sel(l == 3, m2, S1)),        // S1 PPP, R (Q - X3), -, ZZZ3
                          c_sel(l == 1, c_sub(m3, X3), PPP));
    const T o4 = c_shfl_xor(c_sel(l == 1, X3, m4), 1);                    // lane 0: X3, lane 1: S1 PPP
    T r = c_sel(l < 2, c_sel(l == 0, o4, c_sub(m4, o4)), c_sel(l == 2, m3, m4));
    const uint32_t pz = __shfl_sync(0xffffffffu, dz, 0, 4), rz = __shfl_sync(0xffffffffu, dz, 1, 4);
    if (__any_sync(0xffffffffu, pz != 0 && inf == 0)) {  // the same x: twice the point, or infinity
        const T dbl = quad_dbl(p);
        T zero;
        c_set_zero(zero);
        r = c_sel(pz != 0, c_sel(rz != 0, dbl, zero), r);
    }
    r = c_sel((inf & 2u) != 0, p, r);
    return c_sel((inf & 1u) != 0, q, r);
}

// The lane's coordinate of a stored point.
template <bool kL2, class T>
__device__ __forceinline__ T quad_get(const XyzzT<T>* p) {
    const T* c = reinterpret_cast<const T*>(p) + (threadIdx.x & 3);
    if constexpr (kL2) return c_ldcg(c);
    else return c_load(c);
}

template <class T>
__device__ __forceinline__ void quad_put(XyzzT<T>* p, const T& v) {
    c_store(reinterpret_cast<T*>(p) + (threadIdx.x & 3), v);
}

// Sum of `terms` points by the warp: get(t) yields the lane's coordinate of term t; quad k
// takes the terms first + k, first + k + stride, ..., then the quads add up in a butterfly.
// Quad 0 ends with the sum. `first` and `stride` are multiples of 8.
template <class T, class Get>
__device__ __forceinline__ T warp_quad_sum(uint32_t terms, uint32_t first, uint32_t stride, Get&& get) {
    const uint32_t k = (threadIdx.x & 31) >> 2;
    T acc;
    c_set_zero(acc);
    if (first + k < terms) acc = get(first + k);
    for (uint32_t base = first + stride; base < terms; base += stride) {
        T v;
        c_set_zero(v);
        if (base + k < terms) v = get(base + k);
        acc = quad_add(acc, v);
    }
    const uint32_t width = first < terms ? terms - first : 0;  // quads that hold a term
    for (uint32_t off = 1; off < 8 && off < width; off <<= 1) acc = quad_add(acc, c_shfl_xor(acc, 4 * off));
    return acc;
}

// ... by the whole CTA (every thread calls): warps first, their sums through `red` (a point per
// warp). The sum is valid in quad 0.
template <class T, class Get>
__device__ __forceinline__ T cta_quad_sum(uint32_t terms, Get&& get, XyzzT<T>* red) {
    const uint32_t warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t used = min(nwarps, (terms + 7) / 8);  // warps with terms
    T acc;
    c_set_zero(acc);
    if (warp < used) acc = warp_quad_sum<T>(terms, 8 * warp, 8 * nwarps, get);
    if (used > 1) {
        if (warp < used && (threadIdx.x & 31) < 4) quad_put(red + warp, acc);
        __syncthreads();
        if (warp == 0) acc = warp_quad_sum<T>(used, 0, 8, [&](uint32_t t) { return quad_get<false>(red + t); });
        __syncthreads();  // red free again
    }
    return acc;
}

// The two groups as template arguments of the MSM kernels.
// Minimum resident 128-thread CTAs per SM asked of the G1 accumulation: 4 caps it at 128
// registers (no spills), 16 warps per SM; measured on GB300 at 2^20 with 3 / 4 / 5: 2.26 / 2.18 /
// 2.17 ms.
#ifndef ZK_ACC_MINB
#define ZK_ACC_MINB 4
#endif
// G2: 1 takes the registers it wants (2 CTAs per SM), 3 spill: 2^16 1.13 -> 1.25 ms, 2^18 3.16 -> 3.53.
#ifndef ZK_ACC_MINB_G2
#define ZK_ACC_MINB_G2 1
#endif
// Threads of the CTA that sums one long bucket's pieces (quads of lanes sum strided pieces, then a
// tree of the quads). G1 runs 128 threads with four CTAs per SM (a grid of as many): huge buckets
// are summed in chunks by many CTAs, so the CTA size serves the long buckets of small pipelines,
// whose few pieces leave most of a wide CTA idle (128 threads against 256 at two CTAs per SM: within
// 1% up to 2^18, 64 instances of 2^10 .. 2^20 27.95 / 28.0 ms, witness-like 2^19 1.16 / 1.12).
#ifndef ZK_FIXUP_LONG_G1
#define ZK_FIXUP_LONG_G1 128
#endif
// Minimum resident 128-thread CTAs per SM asked of the G1 merge and fixup kernels (G2 keeps
// 1: its points need the registers). 1 / 4: 2^20 2.89 / 2.89 ms, 64 instances 27.95 / 27.83.
#ifndef ZK_RED_MINB
#define ZK_RED_MINB 1
#endif
#ifndef ZK_FIXUP_LONG_MINB_G1
#define ZK_FIXUP_LONG_MINB_G1 4
#endif
struct CurveG1 {
    using T = fe;
    using A = affine_t;
    using P = xyzz_t;
    static constexpr int kAccMinBlocks = ZK_ACC_MINB;
    static constexpr int kFixupLongThreads = ZK_FIXUP_LONG_G1;
    static constexpr int kFixupLongMinBlocks = ZK_FIXUP_LONG_MINB_G1;
    static constexpr int kRedMinBlocks = ZK_RED_MINB;
};

struct CurveG2 {
    using T = fq2;
    using A = affine2_t;
    using P = xyzz2_t;
    static constexpr int kAccMinBlocks = ZK_ACC_MINB_G2;
    static constexpr int kFixupLongThreads = 128;
    static constexpr int kFixupLongMinBlocks = 1;
    static constexpr int kRedMinBlocks = 1;
};

}  // namespace zk
