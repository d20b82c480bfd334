// inverse.cuh -- the loop of the modular inverse of a field element, for the device and, as the
// product rows of field.cuh, for a host-side check.
#pragma once
#include "field.cuh"

namespace zk {

__host__ __device__ __forceinline__ uint32_t funnel_r(uint32_t lo, uint32_t hi, uint32_t z) {  // z < 32
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, z);
#else
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> z);
#endif
}
__host__ __device__ __forceinline__ uint32_t funnel_l(uint32_t lo, uint32_t hi, uint32_t z) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, z);
#else
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << z) >> 32);
#endif
}

// Trailing zeros of a limb, 31 for 0 (the caller shifts again).
__host__ __device__ __forceinline__ uint32_t low_zeros(uint32_t x) {
#ifdef __CUDA_ARCH__
    return x ? __ffs(x) - 1 : 31;
#else
    uint32_t z = 0;
    while (z < 31 && !((x >> z) & 1)) z++;
    return z;
#endif
}

// a >> z and a << z for z < 32 (no bit is lost to the left)
__host__ __device__ __forceinline__ void limbs_shr(fe& a, uint32_t z) {
#pragma unroll
    for (int i = 0; i < 7; i++) a.v[i] = funnel_r(a.v[i], a.v[i + 1], z);
    a.v[7] >>= z;
}
__host__ __device__ __forceinline__ void limbs_shl(fe& a, uint32_t z) {
#pragma unroll
    for (int i = 7; i > 0; i--) a.v[i] = funnel_l(a.v[i - 1], a.v[i], z);
    a.v[0] <<= z;
}
__host__ __device__ __forceinline__ fe limbs_add(const fe& a, const fe& b) {
    fe r;
    r.v[0] = u_add_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < 7; i++) r.v[i] = u_addc_cc(a.v[i], b.v[i]);
    r.v[7] = u_addc(a.v[7], b.v[7]);
    return r;
}
__host__ __device__ __forceinline__ fe limbs_sub(const fe& a, const fe& b, uint32_t* borrow) {
    fe r;
    r.v[0] = u_sub_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int i = 1; i < 8; i++) r.v[i] = u_subc_cc(a.v[i], b.v[i]);
    *borrow = u_subc(0u, 0u);
    return r;
}

// s = a^-1 2^k mod p for a != 0 (mod p), and false for a = 0. Binary extended Euclid without modular
// halvings (Kaliski's almost inverse): with u = p, v = a, r = 0, s = 1 the steps keep p = u s + v r
// and a s = v 2^k (mod p), k counting the halvings of u and v; at u = v = 1 s = a^-1 2^k.
//
// It ends for every a: 0 has no odd part and returns at once; otherwise u + v falls with every
// step, and u v, below 2^510 at first and at least 1, is halved k times, so k <= 510. For canonical
// a, 253 <= k <= 508 and s < p.
//
// What bounds it: ~180 steps of a subtraction, an addition and two shifts, chains of 8 limbs.
template <class F>
__host__ __device__ inline bool fe_almost_inverse(const fe& a, fe* s_out, uint32_t* k_out) {
    fe u, v = a, r = fe_zero(), s = fe_zero();
    if (fe_is_zero(a)) return false;
#pragma unroll
    for (int i = 0; i < 8; i++) u.v[i] = F::P(i);
    s.v[0] = 1;
    uint32_t k = 0;
    while (!(v.v[0] & 1)) {  // u stays odd until the first subtraction
        const uint32_t z = low_zeros(v.v[0]);
        limbs_shr(v, z);
        k += z;  // r = 0
    }
    for (;;) {  // u and v odd
        uint32_t less;
        fe d = limbs_sub(u, v, &less);
        if (fe_is_zero(d)) break;
        if (!less) {
            u = d;
            r = limbs_add(r, s);
            do {
                const uint32_t z = low_zeros(u.v[0]);
                limbs_shr(u, z);
                limbs_shl(s, z);
                k += z;
            } while (!(u.v[0] & 1));
        } else {
            v = limbs_sub(v, u, &less);
            s = limbs_add(s, r);
            do {
                const uint32_t z = low_zeros(v.v[0]);
                limbs_shr(v, z);
                limbs_shl(r, z);
                k += z;
            } while (!(v.v[0] & 1));
        }
    }
    *s_out = s;
    *k_out = k;
    return true;
}

}  // namespace zk
