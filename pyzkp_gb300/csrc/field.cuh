// field.cuh -- BN254 Fr / Fq arithmetic for sm_103a, 8 x 32-bit limbs, Montgomery R = 2^256.
//
// The Montgomery form uses R = 2^256, the same as the reference's 4 x u64 packing
// (runtime/kernels/cpu/kernels.py:46-50,135-141; runtime/metal/runtime.py:30-40 and
// runtime/metal/ecc_source.py:14-25 hold the same moduli), so the bytes of a device
// element are the bytes of the reference's "fr_mont_u64x4" element.
//
// Multiplication is CIOS (coarsely integrated operand scanning): per limb b_i of the
// multiplier, T += a b_i, then T += m p with m = t_0 (-p^-1), and one limb is shifted out.
// Both moduli are below 2^254, so the running value stays below 2^288 (9 limbs) and the
// result below 2p for inputs below 2p; one conditional subtraction yields the canonical
// representative in [0, p). How a row maps to wide multiply-adds, and what bounds it, is at
// the products below.
//
// Fr values are always fully reduced (equal values have equal bits: NTT outputs are
// stored and compared). Fq values inside the curve formulas are kept "lazy", in [0, 2p)
// (F::LAZY): since 4p < 2^256, a product of inputs below 2p is already below 2p without
// the final subtraction, sums subtract 2p when >= 2p, differences add 2p on a borrow, and
// zero tests accept 0 and p. fe_from_mont returns the canonical value; host code that
// reads device Fq values reduces them once more.
#pragma once
#include <cstdint>

namespace zk {

// Modulus, Montgomery one (2^256 mod p) and R^2 mod p as constexpr limb accessors, so
// unrolled code folds them into immediates.
struct FrP {
    __host__ __device__ static constexpr uint32_t P(int i) { return i == 0 ? 0xf0000001u : i == 1 ? 0x43e1f593u : i == 2 ? 0x79b97091u : i == 3 ? 0x2833e848u : i == 4 ? 0x8181585du : i == 5 ? 0xb85045b6u : i == 6 ? 0xe131a029u : 0x30644e72u; }
    static constexpr uint32_t INV = 0xefffffffu  /* -r^-1 mod 2^32 */;
    // (INV p + 1) / 2^32 (see the products below)
    __host__ __device__ static constexpr uint32_t NP(int i) { return i == 0 ? 0x6d1e0a6du : i == 1 ? 0xb5ea65a9u : i == 2 ? 0xc9e9f13fu : i == 3 ? 0xd42f5166u : i == 4 ? 0x6118fd20u : i == 5 ? 0x3b99a131u : i == 6 ? 0x82ba37b4u : 0x2d5e098bu; }
    static constexpr bool CALL_MUL = false;
    static constexpr bool LAZY = false;
    __host__ __device__ static constexpr uint32_t ONE(int i) { return i == 0 ? 0x4ffffffbu : i == 1 ? 0xac96341cu : i == 2 ? 0x9f60cd29u : i == 3 ? 0x36fc7695u : i == 4 ? 0x7879462eu : i == 5 ? 0x666ea36fu : i == 6 ? 0x9a07df2fu : 0x0e0a77c1u; }
    __host__ __device__ static constexpr uint32_t R2(int i) { return i == 0 ? 0xae216da7u : i == 1 ? 0x1bb8e645u : i == 2 ? 0xe35c59e3u : i == 3 ? 0x53fe3ab1u : i == 4 ? 0x53bb8085u : i == 5 ? 0x8c49833du : i == 6 ? 0x7f4e44a5u : 0x0216d0b1u; }
};

struct FqP {
    __host__ __device__ static constexpr uint32_t P(int i) { return i == 0 ? 0xd87cfd47u : i == 1 ? 0x3c208c16u : i == 2 ? 0x6871ca8du : i == 3 ? 0x97816a91u : i == 4 ? 0x8181585du : i == 5 ? 0xb85045b6u : i == 6 ? 0xe131a029u : 0x30644e72u; }
    static constexpr uint32_t INV = 0xe4866389u  /* -q^-1 mod 2^32 */;
    // (INV p + 1) / 2^32 (see the products below)
    __host__ __device__ static constexpr uint32_t NP(int i) { return i == 0 ? 0x705c70f2u : i == 1 ? 0xb5b479a3u : i == 2 ? 0x699a472au : i == 3 ? 0xef510c54u : i == 4 ? 0xb6c9df27u : i == 5 ? 0xb27cd0b5u : i == 6 ? 0x10b67b2fu : 0x2b32bd30u; }
    static constexpr bool CALL_MUL = true;
    static constexpr bool LAZY = true;
    __host__ __device__ static constexpr uint32_t ONE(int i) { return i == 0 ? 0xc58f0d9du : i == 1 ? 0xd35d438du : i == 2 ? 0xf5c70b3du : i == 3 ? 0x0a78eb28u : i == 4 ? 0x7879462cu : i == 5 ? 0x666ea36fu : i == 6 ? 0x9a07df2fu : 0x0e0a77c1u; }
    // 4 q^2 as 16 limbs (the offset that keeps a difference of two products below 4q^2 each
    // non-negative)
    __host__ __device__ static constexpr uint32_t FOUR_P_SQ(int i) {
        constexpr uint32_t v[16] = {0x9d75a6c4u, 0xed516288u, 0x27ab0404u, 0x98081cb4u, 0xb65b2b72u, 0x29406271u,
                                    0xe8490b21u, 0x11a27a55u, 0xd31ace34u, 0x9bb7e970u, 0x58dd5818u, 0xc02e1544u,
                                    0x0d234872u, 0x6669bdf0u, 0xd8f2fe71u, 0x249712e1u};
        return v[i];
    }
    __host__ __device__ static constexpr uint32_t R2(int i) { return i == 0 ? 0x538afa89u : i == 1 ? 0xf32cfc5bu : i == 2 ? 0xd44501fbu : i == 3 ? 0xb5e71911u : i == 4 ? 0x0a417ff6u : i == 5 ? 0x47ab1effu : i == 6 ? 0xcab8351fu : 0x06d89f71u; }
};

// Fr with lazy values in [0, 2r): for the NTT pass kernel only, whose last pass reduces
// every output once more (all other Fr code sees canonical values).
struct FrLazyP : FrP {
    static constexpr bool LAZY = true;
};

// Fr with one non-inlined copy of the product, for kernels whose loop bodies hold many
// products (inlined, they overflow the instruction cache).
struct FrCallP : FrP {
    static constexpr bool CALL_MUL = true;
};

// One field element: 8 little-endian 32-bit limbs (32 bytes, 32-byte aligned in memory).
struct __align__(16) fe {
    uint32_t v[8];
};

template <class F>
__device__ __forceinline__ fe fe_one() {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = F::ONE(i);
    return r;
}

__host__ __device__ __forceinline__ fe fe_zero() {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = 0;
    return r;
}

__host__ __device__ __forceinline__ bool fe_is_zero(const fe& a) {
    uint32_t x = a.v[0] | a.v[1] | a.v[2] | a.v[3] | a.v[4] | a.v[5] | a.v[6] | a.v[7];
    return x == 0;
}

__device__ __forceinline__ bool fe_eq(const fe& a, const fe& b) {
    uint32_t x = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) x |= a.v[i] ^ b.v[i];
    return x == 0;
}

// limb i of 2p
template <class F>
__host__ __device__ constexpr uint32_t p2_limb(int i) {
    return (F::P(i) << 1) | (i ? (F::P(i - 1) >> 31) : 0u);
}

// the modulus of the field's representation: 2p when lazy (values in [0, 2p)), else p
template <class F>
__host__ __device__ constexpr uint32_t mod_limb(int i) {
    return F::LAZY ? p2_limb<F>(i) : F::P(i);
}

// a == 0 mod p for a value of the field's representation ([0, p), or [0, 2p) when lazy).
// kEarly: limb 0 first (0 or p's limb 0 for either zero form): almost every value fails
// there, so a test costs a compare and a branch instead of 16 logic ops. Measured on GB300:
// G1 accumulation -0.4% / -0.6% at 2^20 / 2^22 with it, G2 +0.5% (its pairs of tests), so
// the G1 coordinates take it and the Fq2 ones do not.
template <class F, bool kEarly = false>
__device__ __forceinline__ bool fe_is_zero_mod(const fe& a) {
    if constexpr (kEarly) {
        if (a.v[0] != 0u && (!F::LAZY || a.v[0] != F::P(0))) return false;
    }
    if constexpr (F::LAZY) {
        uint32_t z = 0, e = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            z |= a.v[i];
            e |= a.v[i] ^ F::P(i);
        }
        return z == 0 || e == 0;
    } else {
        return fe_is_zero(a);
    }
}

// r = t - 2p if t >= 2p else t, for t < 4p (< 2^256).
template <class F>
__device__ __forceinline__ fe fe_reduce_2p(const fe& t) {
    fe s;
    uint32_t borrow;
    asm volatile("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s.v[0]), "=r"(s.v[1]), "=r"(s.v[2]), "=r"(s.v[3]), "=r"(s.v[4]), "=r"(s.v[5]), "=r"(s.v[6]),
          "=r"(s.v[7]), "=r"(borrow)
        : "r"(t.v[0]), "r"(t.v[1]), "r"(t.v[2]), "r"(t.v[3]), "r"(t.v[4]), "r"(t.v[5]), "r"(t.v[6]), "r"(t.v[7]),
          "n"(p2_limb<F>(0)), "n"(p2_limb<F>(1)), "n"(p2_limb<F>(2)), "n"(p2_limb<F>(3)), "n"(p2_limb<F>(4)),
          "n"(p2_limb<F>(5)), "n"(p2_limb<F>(6)), "n"(p2_limb<F>(7)));
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = borrow ? t.v[i] : s.v[i];
    return r;
}

// limb i of 4p (4p < 2^256 for both moduli)
template <class F>
__host__ __device__ constexpr uint32_t p4_limb(int i) {
    return (F::P(i) << 2) | (i ? (F::P(i - 1) >> 30) : 0u);
}

// r = t - 4p if t >= 4p else t, for any t < 2^256: r < 4p (2^256 < 6p), so fe_reduce_2p
// after it brings any 256-bit value into [0, 2p).
template <class F>
__device__ __forceinline__ fe fe_reduce_4p(const fe& t) {
    fe s;
    uint32_t borrow;
    asm volatile("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s.v[0]), "=r"(s.v[1]), "=r"(s.v[2]), "=r"(s.v[3]), "=r"(s.v[4]), "=r"(s.v[5]), "=r"(s.v[6]),
          "=r"(s.v[7]), "=r"(borrow)
        : "r"(t.v[0]), "r"(t.v[1]), "r"(t.v[2]), "r"(t.v[3]), "r"(t.v[4]), "r"(t.v[5]), "r"(t.v[6]), "r"(t.v[7]),
          "n"(p4_limb<F>(0)), "n"(p4_limb<F>(1)), "n"(p4_limb<F>(2)), "n"(p4_limb<F>(3)), "n"(p4_limb<F>(4)),
          "n"(p4_limb<F>(5)), "n"(p4_limb<F>(6)), "n"(p4_limb<F>(7)));
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = borrow ? t.v[i] : s.v[i];
    return r;
}

// r = t - p if t >= p else t, for t < 2p (< 2^255).
template <class F>
__device__ __forceinline__ fe fe_reduce_once(const fe& t) {
    fe s;
    uint32_t borrow;
    asm volatile("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s.v[0]), "=r"(s.v[1]), "=r"(s.v[2]), "=r"(s.v[3]), "=r"(s.v[4]), "=r"(s.v[5]), "=r"(s.v[6]),
          "=r"(s.v[7]), "=r"(borrow)
        : "r"(t.v[0]), "r"(t.v[1]), "r"(t.v[2]), "r"(t.v[3]), "r"(t.v[4]), "r"(t.v[5]), "r"(t.v[6]), "r"(t.v[7]),
          "n"(F::P(0)), "n"(F::P(1)), "n"(F::P(2)), "n"(F::P(3)), "n"(F::P(4)), "n"(F::P(5)), "n"(F::P(6)),
          "n"(F::P(7)));
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = borrow ? t.v[i] : s.v[i];
    return r;
}

template <class F>
__device__ __forceinline__ fe fe_add(const fe& a, const fe& b) {
    fe t;
    asm volatile("add.cc.u32  %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(t.v[0]), "=r"(t.v[1]), "=r"(t.v[2]), "=r"(t.v[3]), "=r"(t.v[4]), "=r"(t.v[5]), "=r"(t.v[6]),
          "=r"(t.v[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    if constexpr (F::LAZY) return fe_reduce_2p<F>(t);
    else return fe_reduce_once<F>(t);
}

template <class F>
__device__ __forceinline__ fe fe_sub(const fe& a, const fe& b) {
    fe t;
    uint32_t m;
    asm volatile("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(t.v[0]), "=r"(t.v[1]), "=r"(t.v[2]), "=r"(t.v[3]), "=r"(t.v[4]), "=r"(t.v[5]), "=r"(t.v[6]),
          "=r"(t.v[7]), "=r"(m)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    fe r;
    asm volatile("add.cc.u32  %0, %8, %16;\n\t"
        "addc.cc.u32 %1, %9, %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7])
        : "r"(t.v[0]), "r"(t.v[1]), "r"(t.v[2]), "r"(t.v[3]), "r"(t.v[4]), "r"(t.v[5]), "r"(t.v[6]), "r"(t.v[7]),
          "r"(mod_limb<F>(0) & m), "r"(mod_limb<F>(1) & m), "r"(mod_limb<F>(2) & m), "r"(mod_limb<F>(3) & m),
          "r"(mod_limb<F>(4) & m), "r"(mod_limb<F>(5) & m), "r"(mod_limb<F>(6) & m), "r"(mod_limb<F>(7) & m));
    return r;
}

template <class F>
__device__ __forceinline__ fe fe_neg(const fe& a) {
    return fe_sub<F>(fe_zero(), a);
}

template <class F>
__device__ __forceinline__ fe fe_dbl(const fe& a) {
    return fe_add<F>(a, a);
}

// ---- products -------------------------------------------------------------------------------
//
// The carry flag primitives are one PTX instruction each on the device (asm volatile keeps
// their order, so the flag flows from one to the next as in a single asm block; every other
// asm block that writes the flag is volatile too, or it could be moved in between); on the
// host they emulate the flag, so the same code runs in a host-side check of the arithmetic.
#ifndef __CUDA_ARCH__
inline uint32_t& host_carry_flag() {
    static thread_local uint32_t cc = 0;
    return cc;
}
#endif

__host__ __device__ __forceinline__ uint32_t u_add_cc(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
#else
    const uint64_t s = (uint64_t)a + b;
    host_carry_flag() = (uint32_t)(s >> 32);
    return (uint32_t)s;
#endif
}

__host__ __device__ __forceinline__ uint32_t u_addc_cc(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
#else
    const uint64_t s = (uint64_t)a + b + host_carry_flag();
    host_carry_flag() = (uint32_t)(s >> 32);
    return (uint32_t)s;
#endif
}

__host__ __device__ __forceinline__ uint32_t u_addc(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("addc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
#else
    return (uint32_t)((uint64_t)a + b + host_carry_flag());
#endif
}

__host__ __device__ __forceinline__ uint32_t u_sub_cc(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
#else
    host_carry_flag() = a < b ? 1u : 0u;
    return a - b;
#endif
}

__host__ __device__ __forceinline__ uint32_t u_subc_cc(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
#else
    const uint64_t d = (uint64_t)a - b - host_carry_flag();
    host_carry_flag() = (uint32_t)(d >> 63);
    return (uint32_t)d;
#endif
}

__host__ __device__ __forceinline__ uint32_t u_subc(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("subc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
#else
    return (uint32_t)((uint64_t)a - b - host_carry_flag());
#endif
}

// The 64-bit pair (lo, hi) += a * b, in two instructions that share a carry: lo and hi are
// the limbs of an even-aligned register pair, so one wide multiply-add does both. _cc
// leaves the carry out in the flag; kIn takes the flag's carry in.
template <bool kIn>
__host__ __device__ __forceinline__ void u_mad2_cc(uint32_t& lo, uint32_t& hi, uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    if constexpr (kIn)
        asm volatile("madc.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.cc.u32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(a), "r"(b));
    else
        asm volatile("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.cc.u32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(a), "r"(b));
#else
    const unsigned __int128 s = (unsigned __int128)((uint64_t)a * b) + (((uint64_t)hi << 32) | lo) + (kIn ? host_carry_flag() : 0u);
    lo = (uint32_t)s;
    hi = (uint32_t)(s >> 32);
    host_carry_flag() = (uint32_t)(s >> 64);
#endif
}

// ... and without a carry out (the caller's bound excludes one)
template <bool kIn>
__host__ __device__ __forceinline__ void u_mad2(uint32_t& lo, uint32_t& hi, uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    if constexpr (kIn)
        asm volatile("madc.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.u32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(a), "r"(b));
    else
        asm volatile("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.u32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(a), "r"(b));
#else
    const uint64_t s = (uint64_t)a * b + (((uint64_t)hi << 32) | lo) + (kIn ? host_carry_flag() : 0u);
    lo = (uint32_t)s;
    hi = (uint32_t)(s >> 32);
#endif
}

// The product rows keep a running value T (9 limbs) as two accumulators of four 64-bit
// columns each: e[0..7] at limbs 0..7 and o[0..7] at limbs 1..8, T = e + 2^32 o. A product
// a_j b_i belongs to the accumulator that its limb position is aligned with, so each of the
// 8 products of a row is ONE wide multiply-add with carry in and out (mad.lo.cc / madc.hi.cc
// on an aligned pair) and a row has two chains of four.
//
// What bounds it on GB300: the wide multiply-add. One takes 4 issue cycles of a scheduler's
// multiply pipe whether or not it adds and carries (measured: 10.1 T/s for the chip at
// 2070 MHz, 16 lanes a cycle a scheduler at two passes), and an add with carry 2 cycles of
// the other integer pipe. A product needs 128 of the former = 512 cycles a warp; this form
// adds 2 low multiplies and ~40 adds. Measured (independent chains, 64 warps per SM): 71.6 G
// products/s = 91% of the multiply pipe, against 47.8 G/s for full-width products folded in
// by separate add-with-carry chains (290 adds: the two pipes then take turns); 64-bit adds
// of full-width products 56.8 G/s.
//
// row_odd: o += {a_1, a_3, a_5, a_7} y, with the flag's carry into limb 1 when kIn. T stays
// below 2^288, so o (at most T / 2^32) never carries out.
template <bool kIn>
__host__ __device__ __forceinline__ void row_odd(uint32_t* o, const uint32_t* a, uint32_t y) {
    u_mad2_cc<kIn>(o[0], o[1], a[1], y);
    u_mad2_cc<true>(o[2], o[3], a[3], y);
    u_mad2_cc<true>(o[4], o[5], a[5], y);
    u_mad2<true>(o[6], o[7], a[7], y);
}

// row_even: e += {a_0, a_2, a_4, a_6} y, the carry out of limb 7 into o's top limb.
__host__ __device__ __forceinline__ void row_even(uint32_t* e, uint32_t* o, const uint32_t* a, uint32_t y) {
    u_mad2_cc<false>(e[0], e[1], a[0], y);
    u_mad2_cc<true>(e[2], e[3], a[2], y);
    u_mad2_cc<true>(e[4], e[5], a[4], y);
    u_mad2_cc<true>(e[6], e[7], a[6], y);
    o[7] = u_addc(o[7], 0u);
}

// The first row: e, o = a * y, nothing to add to.
__host__ __device__ __forceinline__ void row_first(uint32_t* e, uint32_t* o, const uint32_t* a, uint32_t y) {
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        const uint64_t p = (uint64_t)a[j] * y, q = (uint64_t)a[j + 1] * y;
        e[j] = (uint32_t)p;
        e[j + 1] = (uint32_t)(p >> 32);
        o[j] = (uint32_t)q;
        o[j + 1] = (uint32_t)(q >> 32);
    }
}

template <class F>
__host__ __device__ __forceinline__ void modulus_limbs(uint32_t* p) {
#pragma unroll
    for (int j = 0; j < 8; j++) p[j] = F::P(j);
}

// The modulus multiple N = (-p^-1 mod 2^32) p has N_0 = 2^32 - 1, so T + T_0 N is divisible by 2^32
// with the quotient floor(T / 2^32) + T_0 N', N' = (N + 1) / 2^32 < p: the row's multiplier is T's
// own low limb, without the multiplication by -p^-1 (and the wait for it). N has 286 bits, so
// a row leaves T up to 2^32 p larger than a row with p would; the last two rows use p (their
// multipliers computed), which brings the result to its bound: the rows before add at most
// 2^-32 p to it. Measured against 8 rows with p: 69.5 -> 71.6 G products/s, a lone product
// 878 -> 843 cycles.
static constexpr int kShortRows = 6;  // rows of a product that use N'

// T += m p with m = T_0 (-p^-1): limb 0 becomes 0.
template <class F>
__host__ __device__ __forceinline__ void row_reduce(uint32_t* e, uint32_t* o) {
    uint32_t p[8];
    modulus_limbs<F>(p);
    const uint32_t m = e[0] * F::INV;
    row_odd<false>(o, p, m);
    row_even(e, o, p, m);
}

// T / 2^32 once limb 0 is 0: o becomes the even accumulator, e without its limbs 0 and 1 the odd
// one with `top` at limb 7; limb 1 is added to the new even accumulator, its carry left in the
// flag for the odd row that follows.
__host__ __device__ __forceinline__ void row_shift(uint32_t* e, uint32_t* o, uint32_t top) {
    const uint32_t c = e[1];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const uint32_t x = j < 6 ? e[j + 2] : j == 6 ? top : 0u;
        e[j] = o[j];
        o[j] = x;
    }
    e[0] = u_add_cc(e[0], c);
}

// T = floor(T / 2^32) + m N' for m = T_0.
template <class F>
__host__ __device__ __forceinline__ void row_step(uint32_t* e, uint32_t* o, uint32_t top = 0u) {
    uint32_t n[8];
#pragma unroll
    for (int j = 0; j < 8; j++) n[j] = F::NP(j);
    const uint32_t m = e[0];
    row_shift(e, o, top);
    row_odd<true>(o, n, m);
    row_even(e, o, n, m);
}

// T / 2^32 (limb 0 being 0), then T += m p as in row_reduce.
template <class F>
__host__ __device__ __forceinline__ void row_shift_reduce(uint32_t* e, uint32_t* o, uint32_t top) {
    uint32_t p[8];
    modulus_limbs<F>(p);
    row_shift(e, o, top);
    const uint32_t m = e[0] * F::INV;
    row_odd<true>(o, p, m);
    row_even(e, o, p, m);
}

// (e + 2^32 o) / 2^32 as 8 limbs, limb 0 being 0 and the value below 2^288; `top` is added to
// limb 7 of the result.
__host__ __device__ __forceinline__ fe row_result(const uint32_t* e, const uint32_t* o, uint32_t top = 0u) {
    fe r;
    r.v[0] = u_add_cc(o[0], e[1]);
#pragma unroll
    for (int j = 1; j < 7; j++) r.v[j] = u_addc_cc(o[j], e[j + 1]);
    r.v[7] = u_addc(o[7], top);
    return r;
}

// a b 2^-256 mod p, below ab / 2^256 + (1 + 2^-31) p (CIOS rows): below 2p for a, b below 2p. T
// is largest in the first row with p, below 2^32 (a + N' + p) (1 + 2^-31), which has to stay below
// 2^288: for a below 3.35p (r; 3.39p for q). b may be any 256 bits. A value of a caller, which
// nothing has reduced, is therefore the second factor, or a factor of fe_mul_any.
template <class F>
__host__ __device__ __forceinline__ fe mul_rows(const fe& a, const fe& b) {
    uint32_t e[8], o[8];
    row_first(e, o, a.v, b.v[0]);
#pragma unroll
    for (int i = 1; i <= kShortRows; i++) {
        row_step<F>(e, o);
        row_odd<false>(o, a.v, b.v[i]);
        row_even(e, o, a.v, b.v[i]);
    }
#pragma unroll
    for (int i = kShortRows + 1; i < 8; i++) {
        row_reduce<F>(e, o);
        row_shift(e, o, 0u);
        row_odd<true>(o, a.v, b.v[i]);
        row_even(e, o, a.v, b.v[i]);
    }
    row_reduce<F>(e, o);
    return row_result(e, o);
}

// (a b + c d) 2^-256 mod p with one reduction, below (ab + cd) / 2^256 + p: below 2.52p for
// inputs up to 2p. T stays below 2^32 (a + c + p) <= 5p 2^32 < 2^288; rows with N' would leave no
// room for the last rows' m p beside both products, so every row uses p.
template <class F>
__host__ __device__ __forceinline__ fe mul_add_rows(const fe& a, const fe& b, const fe& c, const fe& d) {
    uint32_t e[8], o[8];
    row_first(e, o, a.v, b.v[0]);
    row_odd<false>(o, c.v, d.v[0]);
    row_even(e, o, c.v, d.v[0]);
    row_reduce<F>(e, o);
#pragma unroll
    for (int i = 1; i < 8; i++) {
        row_shift(e, o, 0u);
        row_odd<true>(o, a.v, b.v[i]);
        row_even(e, o, a.v, b.v[i]);
        row_odd<false>(o, c.v, d.v[i]);
        row_even(e, o, c.v, d.v[i]);
        row_reduce<F>(e, o);
    }
    return row_result(e, o);
}

// ---- products with a constant known beforehand ------------------------------------------------
//
// x w mod p for a constant w (a twiddle factor) held with w' = floor(w 2^256 / p) (Shoup): the
// quotient q = floor(x w' / 2^256) is at most 1 below floor(x w / p), so x w - q p, taken modulo
// 2^256, lies in [0, 2p). Only the upper columns of x w' and the lower halves of the other two
// products are needed: 99 wide and 16 low multiply-adds instead of 128 and 2, and half the
// carry additions. w is canonical, x any value below 4p.
//
// Bound: x w / p - x w' / 2^256 < x / 2^256 < 4p / 2^256 < 0.757, and leaving out the columns below
// limb 6 lowers the sum by less than 6 * 2^(64 + 160) = 6 * 2^-32 of q's unit, so the floor is
// lowered by at most 1.
struct fe_const {
    fe w, ws;  // w, floor(w 2^256 / p)
};

__host__ __device__ __forceinline__ uint32_t u_madc_lo(uint32_t a, uint32_t b, uint32_t c) {  // a b + c + carry in
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("madc.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
#else
    return a * b + c + host_carry_flag();
#endif
}

// c[0..2N-1] += {x_0, x_2, ..} y for N partial products (x strided by 2); kOut: the carry out
// becomes c[2N] (not yet written), else it is dropped or known to be none (a top pair that
// held at most a carry before: (2^32 - 1)^2 + 2 < 2^64).
template <int N, bool kOut>
__host__ __device__ __forceinline__ void col_chain(uint32_t* c, const uint32_t* x, uint32_t y) {
    if constexpr (N == 1) {
        if constexpr (kOut) u_mad2_cc<false>(c[0], c[1], x[0], y);
        else u_mad2<false>(c[0], c[1], x[0], y);
    } else {
        u_mad2_cc<false>(c[0], c[1], x[0], y);
#pragma unroll
        for (int k = 1; k + 1 < N; k++) u_mad2_cc<true>(c[2 * k], c[2 * k + 1], x[2 * k], y);
        if constexpr (kOut) u_mad2_cc<true>(c[2 * N - 2], c[2 * N - 1], x[2 * N - 2], y);
        else u_mad2<true>(c[2 * N - 2], c[2 * N - 1], x[2 * N - 2], y);
    }
    if constexpr (kOut) c[2 * N] = u_addc(0u, 0u);
}

// ... for N - 1 pairs and the low half of a last product at c[2N - 2] (modulo 2^32 there)
template <int N>
__host__ __device__ __forceinline__ void col_chain_low(uint32_t* c, const uint32_t* x, uint32_t y) {
    if constexpr (N == 1) {
        c[0] += x[0] * y;
    } else {
        u_mad2_cc<false>(c[0], c[1], x[0], y);
#pragma unroll
        for (int k = 1; k + 1 < N; k++) u_mad2_cc<true>(c[2 * k], c[2 * k + 1], x[2 * k], y);
        c[2 * N - 2] = u_madc_lo(x[2 * N - 2], y, c[2 * N - 2]);
    }
}

// (e + 2^32 o) += a x modulo 2^256, e at limbs 0..7, o at limbs 1..7
__host__ __device__ __forceinline__ void mul_low(uint32_t* e, uint32_t* o, const uint32_t* a, const uint32_t* x) {
    col_chain<4, false>(e, a, x[0]);
    col_chain_low<4>(o, a + 1, x[0]);
    col_chain<3, false>(e + 2, a + 1, x[1]);
    col_chain_low<4>(o, a, x[1]);
    col_chain<3, false>(e + 2, a, x[2]);
    col_chain_low<3>(o + 2, a + 1, x[2]);
    col_chain<2, false>(e + 4, a + 1, x[3]);
    col_chain_low<3>(o + 2, a, x[3]);
    col_chain<2, false>(e + 4, a, x[4]);
    col_chain_low<2>(o + 4, a + 1, x[4]);
    col_chain<1, false>(e + 6, a + 1, x[5]);
    col_chain_low<2>(o + 4, a, x[5]);
    col_chain<1, false>(e + 6, a, x[6]);
    col_chain_low<1>(o + 6, a + 1, x[6]);
    col_chain_low<1>(o + 6, a, x[7]);
}

// x w mod p in [0, 2p) for x below 4p
template <class F>
__host__ __device__ __forceinline__ fe fe_mul_const(const fe& x, const fe_const& c) {
    const uint32_t *a = c.ws.v, *y = x.v;
    // q: columns 6 .. 14 of x w', e at limbs 6 .. 15, o at limbs 7 .. 15
    uint32_t e[10], o[9], q[8];
#pragma unroll
    for (int j = 0; j < 10; j++) e[j] = 0u;
#pragma unroll
    for (int j = 0; j < 9; j++) o[j] = 0u;
    col_chain<1, false>(e, a + 6, y[0]);
    col_chain<1, false>(o, a + 7, y[0]);
    col_chain<2, false>(e, a + 5, y[1]);
    col_chain<1, true>(o, a + 6, y[1]);
    col_chain<2, true>(e, a + 4, y[2]);
    col_chain<2, false>(o, a + 5, y[2]);
    col_chain<3, false>(e, a + 3, y[3]);
    col_chain<2, true>(o, a + 4, y[3]);
    col_chain<3, true>(e, a + 2, y[4]);
    col_chain<3, false>(o, a + 3, y[4]);
    col_chain<4, false>(e, a + 1, y[5]);
    col_chain<3, true>(o, a + 2, y[5]);
    col_chain<4, true>(e, a, y[6]);
    col_chain<4, false>(o, a + 1, y[6]);
    col_chain<4, false>(e + 2, a + 1, y[7]);
    col_chain<4, true>(o, a, y[7]);
    (void)u_add_cc(e[1], o[0]);
#pragma unroll
    for (int j = 0; j < 7; j++) q[j] = u_addc_cc(e[j + 2], o[j + 1]);
    q[7] = u_addc(e[9], o[8]);
    // x w + q (2^256 - p) modulo 2^256
    uint32_t n[8];
#pragma unroll
    for (int j = 0; j < 8; j++) n[j] = j == 0 ? 0u - F::P(0) : ~F::P(j);
    uint32_t re[8], ro[7];
#pragma unroll
    for (int j = 0; j < 8; j++) re[j] = 0u;
#pragma unroll
    for (int j = 0; j < 7; j++) ro[j] = 0u;
    mul_low(re, ro, c.w.v, y);
    mul_low(re, ro, n, q);
    fe r;
    r.v[0] = re[0];
    r.v[1] = u_add_cc(re[1], ro[0]);
#pragma unroll
    for (int j = 2; j < 7; j++) r.v[j] = u_addc_cc(re[j], ro[j - 1]);
    r.v[7] = u_addc(re[7], ro[6]);
    return r;
}

// a - b + 2p for a, b below 2p: in (0, 4p), an operand of fe_mul_const
template <class F>
__host__ __device__ __forceinline__ fe fe_sub_4p(const fe& a, const fe& b) {
    fe t, r;
    t.v[0] = u_sub_cc(a.v[0], b.v[0]);
#pragma unroll
    for (int j = 1; j < 7; j++) t.v[j] = u_subc_cc(a.v[j], b.v[j]);
    t.v[7] = u_subc(a.v[7], b.v[7]);
    r.v[0] = u_add_cc(t.v[0], p2_limb<F>(0));
#pragma unroll
    for (int j = 1; j < 7; j++) r.v[j] = u_addc_cc(t.v[j], p2_limb<F>(j));
    r.v[7] = u_addc(t.v[7], p2_limb<F>(7));
    return r;
}

template <class F>
__device__ __noinline__ fe fe_mul_call(const fe a, const fe b) {
    return mul_rows<F>(a, b);
}

// r = a * b * 2^-256 mod p for a below 3.35p and any b (see mul_rows); in [0, p), or [0, 2p) when
// lazy, for a, b that are. F::CALL_MUL: one non-inlined copy of the product, called from
// every site. The curve formulas hold 10-14 products per loop body, so inlining them all
// overflows the instruction cache; the NTT butterflies hold one to four.
template <class F>
__device__ __forceinline__ fe fe_mul(const fe& a, const fe& b) {
    fe r;
    if constexpr (F::CALL_MUL) r = fe_mul_call<F>(a, b);
    else r = mul_rows<F>(a, b);
    if constexpr (F::LAZY) return r;
    else return fe_reduce_once<F>(r);
}

// ---- separated forms: a 512-bit product, then one Montgomery reduction -------------------
//
// Splitting the product from the reduction lets a square skip the 28 repeated cross
// products (100 wide multiply-adds instead of 128), and lets the Fq2 product reduce sums of
// products. They serve the lazy Fq of the curve formulas only.
//
// Reduction: (T + M p) / 2^256 row by row over a window of 9 limbs; T's limb 8 + i enters the
// window at its limb 7 after row i, so the window stays below 2^256 + 2^32 p before a shift
// and nothing carries out of it. The result is below T / 2^256 + p: below 2p for T < 4p^2 (a
// product of two values below 2p: T / 2^256 < 0.76 p), below 2.52 p for T < 8p^2, which one
// conditional subtraction of 2p brings below 2p (both moduli are below 0.19 * 2^256).

// t[0..15] = a * b for any 256-bit a, b, in even and odd columns (o[k] at limb k + 1). Rows 2k - 1
// and 2k end at the same even column and rows 2k and 2k + 1 at the same odd one, so only the
// second of each two can carry out.
__host__ __device__ __forceinline__ void sos_mul_wide(uint32_t* t, const uint32_t* a, const uint32_t* b) {
    uint32_t e[16], o[16];
#pragma unroll
    for (int j = 0; j < 16; j++) e[j] = o[j] = 0u;
    row_first(e, o, a, b[0]);
#pragma unroll
    for (int i = 1; i < 8; i += 2) {
        col_chain<4, true>(o + i - 1, a, b[i]);       // limbs i .. i + 7
        col_chain<4, false>(e + i + 1, a + 1, b[i]);  // limbs i + 1 .. i + 8
        if (i + 1 < 8) {
            col_chain<4, true>(e + i + 1, a, b[i + 1]);
            col_chain<4, false>(o + i + 1, a + 1, b[i + 1]);
        }
    }
    t[0] = e[0];
    t[1] = u_add_cc(e[1], o[0]);
#pragma unroll
    for (int j = 2; j < 15; j++) t[j] = u_addc_cc(e[j], o[j - 1]);
    t[15] = u_addc(e[15], o[14]);
}

// t[0..15] = a * a: the cross products a_i a_j (i < j) once, doubled, plus the squares a_i^2
// at limb 2i. Carries as in sos_mul_wide: of two rows that end at the same column the second.
__host__ __device__ __forceinline__ void sos_sqr_wide(uint32_t* t, const uint32_t* a) {
    uint32_t e[16], o[16];
#pragma unroll
    for (int j = 0; j < 16; j++) e[j] = o[j] = 0u;
    col_chain<4, false>(o, a + 1, a[0]);      // a_0 a_{1,3,5,7}: limbs 1 .. 8
    col_chain<3, false>(e + 2, a + 2, a[0]);  // a_0 a_{2,4,6}
    col_chain<3, true>(o + 2, a + 2, a[1]);
    col_chain<3, false>(e + 4, a + 3, a[1]);
    col_chain<3, false>(o + 4, a + 3, a[2]);
    col_chain<2, true>(e + 6, a + 4, a[2]);
    col_chain<2, true>(o + 6, a + 4, a[3]);
    col_chain<2, false>(e + 8, a + 5, a[3]);
    col_chain<2, false>(o + 8, a + 5, a[4]);
    col_chain<1, true>(e + 10, a + 6, a[4]);
    col_chain<1, true>(o + 10, a + 6, a[5]);
    col_chain<1, false>(e + 12, a + 7, a[5]);
    col_chain<1, false>(o + 12, a + 7, a[6]);
    // the cross sum x in limbs 1 .. 14 (below a^2 / 2 < 2^511)
    uint32_t x[15];
    x[1] = o[0];
    x[2] = u_add_cc(e[2], o[1]);
#pragma unroll
    for (int j = 3; j < 14; j++) x[j] = u_addc_cc(e[j], o[j - 1]);
    x[14] = u_addc(0u, o[13]);
    // doubled by shifting (no carry chain), then the squares
    t[0] = 0u;
    t[1] = x[1] << 1;
#pragma unroll
    for (int j = 2; j < 15; j++) t[j] = (x[j] << 1) | (x[j - 1] >> 31);
    t[15] = x[14] >> 31;
    u_mad2_cc<false>(t[0], t[1], a[0], a[0]);
#pragma unroll
    for (int i = 1; i < 7; i++) u_mad2_cc<true>(t[2 * i], t[2 * i + 1], a[i], a[i]);
    u_mad2<true>(t[14], t[15], a[7], a[7]);
}

// (T + M p) / 2^256 for t = T (16 limbs): T * 2^-256 mod p, below T / 2^256 + (1 + 2^-31) p.
template <class F>
__host__ __device__ __forceinline__ fe sos_redc(const uint32_t* t) {
    uint32_t e[8], o[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        e[j] = t[j];
        o[j] = 0u;
    }
#pragma unroll
    for (int i = 0; i < kShortRows; i++) row_step<F>(e, o, t[8 + i]);
    row_reduce<F>(e, o);
    row_shift_reduce<F>(e, o, t[14]);
    return row_result(e, o, t[15]);
}

// 2p - c for c in [0, 2p): in (0, 2p], congruent to -c
template <class F>
__host__ __device__ __forceinline__ fe sos_neg2p(const fe& c) {
    fe r;
    r.v[0] = u_sub_cc(p2_limb<F>(0), c.v[0]);
#pragma unroll
    for (int j = 1; j < 7; j++) r.v[j] = u_subc_cc(p2_limb<F>(j), c.v[j]);
    r.v[7] = u_subc(p2_limb<F>(7), c.v[7]);
    return r;
}

// r = t - 2p if t >= 2p else t, for t < 4p (the host-and-device twin of fe_reduce_2p)
template <class F>
__host__ __device__ __forceinline__ fe sos_reduce_2p(const fe& t) {
    fe s;
    s.v[0] = u_sub_cc(t.v[0], p2_limb<F>(0));
#pragma unroll
    for (int j = 1; j < 8; j++) s.v[j] = u_subc_cc(t.v[j], p2_limb<F>(j));
    const uint32_t borrow = u_subc(0u, 0u);
    fe r;
#pragma unroll
    for (int j = 0; j < 8; j++) r.v[j] = borrow ? t.v[j] : s.v[j];
    return r;
}

// A vector element of a caller as the first factor of a product: below 2p as it is (its top limb
// tells, and in earnest no thread of a warp goes on), else less 2p, below 2^256 - 2p < 3.3p.
template <class F>
__host__ __device__ __forceinline__ fe fe_first_factor(const fe& a) {
    if (a.v[7] < p2_limb<F>(7)) return a;
    return sos_reduce_2p<F>(a);
}

// The product rows for any 256-bit a and b.
template <class F>
__host__ __device__ __forceinline__ fe mul_rows_any(const fe& a, const fe& b) {
    return mul_rows<F>(fe_first_factor<F>(a), b);
}

// fe_mul for any 256-bit a and b (vectors of a caller)
template <class F>
__device__ __forceinline__ fe fe_mul_any(const fe& a, const fe& b) {
    return fe_mul<F>(fe_first_factor<F>(a), b);
}

// a^2 * 2^-256 mod p in [0, 2p) for a in [0, 2p)
template <class F>
__host__ __device__ __forceinline__ fe fe_sqr_sos(const fe& a) {
    static_assert(F::LAZY, "the separated forms keep lazy values");
    uint32_t t[16];
    sos_sqr_wide(t, a.v);
    return sos_redc<F>(t);
}

// a b * 2^-256 mod p in [0, 2p) for a, b in [0, 2p): product, then the reduction
template <class F>
__host__ __device__ __forceinline__ fe fe_mul_sos(const fe& a, const fe& b) {
    static_assert(F::LAZY, "the separated forms keep lazy values");
    uint32_t t[16];
    sos_mul_wide(t, a.v, b.v);
    return sos_redc<F>(t);
}

// (a b + c d) * 2^-256 mod p in [0, 2p) for inputs in [0, 2p] (one reduction, 192 wide
// multiply-adds instead of 256)
template <class F>
__host__ __device__ __forceinline__ fe fe_mul_add_sos(const fe& a, const fe& b, const fe& c, const fe& d) {
    static_assert(F::LAZY, "the separated forms keep lazy values");
    return sos_reduce_2p<F>(mul_add_rows<F>(a, b, c, d));
}

// (a b - c d) * 2^-256 mod p in [0, 2p) for inputs in [0, 2p): a b + (2p - c) d
template <class F>
__host__ __device__ __forceinline__ fe fe_mul_sub_sos(const fe& a, const fe& b, const fe& c, const fe& d) {
    return fe_mul_add_sos<F>(a, b, sos_neg2p<F>(c), d);
}

// Fq2 product with lazy reduction (Karatsuba): T0 = a0 b0, T1 = a1 b1, T2 = (a0 + a1)(b0 + b1)
// as 512-bit products, c0 = redc(T0 + (4q^2 - T1)), c1 = redc(T2 - T0 - T1) = redc(a0 b1 + a1 b0):
// 3 products and 2 reductions instead of 3 full products. Inputs in [0, 2q): the sums a0 + a1
// stay below 4q < 2^256 unreduced, both arguments of the reductions are below 8q^2, results in [0, 2q).
struct fe_pair {
    fe c0, c1;
};

template <class F>
__host__ __device__ __forceinline__ fe_pair fe2_mul_lazy(const fe& a0, const fe& a1, const fe& b0, const fe& b1) {
    static_assert(F::LAZY, "the separated forms keep lazy values");
    uint32_t t0[16], t1[16];
    sos_mul_wide(t0, a0.v, b0.v);
    sos_mul_wide(t1, a1.v, b1.v);
    // u = T0 + (4q^2 - T1) in (0, 8q^2); s = T0 + T1 (below 8q^2)
    uint32_t u[16], s[16];
    u[0] = u_sub_cc(F::FOUR_P_SQ(0), t1[0]);
#pragma unroll
    for (int j = 1; j < 15; j++) u[j] = u_subc_cc(F::FOUR_P_SQ(j), t1[j]);
    u[15] = u_subc(F::FOUR_P_SQ(15), t1[15]);
    u[0] = u_add_cc(u[0], t0[0]);
#pragma unroll
    for (int j = 1; j < 15; j++) u[j] = u_addc_cc(u[j], t0[j]);
    u[15] = u_addc(u[15], t0[15]);
    s[0] = u_add_cc(t0[0], t1[0]);
#pragma unroll
    for (int j = 1; j < 15; j++) s[j] = u_addc_cc(t0[j], t1[j]);
    s[15] = u_addc(t0[15], t1[15]);
    fe_pair r;
    r.c0 = sos_reduce_2p<F>(sos_redc<F>(u));
    // T2 - s with a0 + a1, b0 + b1 as plain 256-bit sums
    fe sa, sb;
    sa.v[0] = u_add_cc(a0.v[0], a1.v[0]);
#pragma unroll
    for (int j = 1; j < 7; j++) sa.v[j] = u_addc_cc(a0.v[j], a1.v[j]);
    sa.v[7] = u_addc(a0.v[7], a1.v[7]);
    sb.v[0] = u_add_cc(b0.v[0], b1.v[0]);
#pragma unroll
    for (int j = 1; j < 7; j++) sb.v[j] = u_addc_cc(b0.v[j], b1.v[j]);
    sb.v[7] = u_addc(b0.v[7], b1.v[7]);
    uint32_t t2[16];
    sos_mul_wide(t2, sa.v, sb.v);
    t2[0] = u_sub_cc(t2[0], s[0]);
#pragma unroll
    for (int j = 1; j < 15; j++) t2[j] = u_subc_cc(t2[j], s[j]);
    t2[15] = u_subc(t2[15], s[15]);
    r.c1 = sos_reduce_2p<F>(sos_redc<F>(t2));
    return r;
}

template <class F>
__device__ __noinline__ fe_pair fe2_mul_lazy_call(const fe a0, const fe a1, const fe b0, const fe b1) {
    return fe2_mul_lazy<F>(a0, a1, b0, b1);
}

template <class F>
__device__ __noinline__ fe fe_sqr_sos_call(const fe a) {
    return fe_sqr_sos<F>(a);
}

template <class F>
__device__ __noinline__ fe fe_mul_sub_sos_call(const fe a, const fe b, const fe c, const fe d) {
    return fe_mul_sub_sos<F>(a, b, c, d);
}

// The separated forms serve the lazy fields with the called multiplication: the curve
// formulas over Fq.
template <class F>
__device__ __forceinline__ constexpr bool use_sos() {
    return F::LAZY && F::CALL_MUL;
}

template <class F>
__device__ __forceinline__ fe fe_sqr(const fe& a) {
    if constexpr (use_sos<F>()) return fe_sqr_sos_call<F>(a);
    else return fe_mul<F>(a, a);
}

// a b - c d (inputs in the field's representation)
template <class F>
__device__ __forceinline__ fe fe_mul_sub(const fe& a, const fe& b, const fe& c, const fe& d) {
    if constexpr (use_sos<F>()) return fe_mul_sub_sos_call<F>(a, b, c, d);
    else return fe_sub<F>(fe_mul<F>(a, b), fe_mul<F>(c, d));
}

// canonical value (any 256-bit input, reduced mod p first) -> Montgomery form
template <class F>
__device__ __forceinline__ fe fe_to_mont(fe a) {
    // at most floor((2^256 - 1) / p) = 5 subtractions for both BN254 moduli
#pragma unroll 1
    for (int k = 0; k < 5; k++) {
        fe s;
        uint32_t br;
        asm volatile("sub.cc.u32  %0, %9, %17;\n\t"
            "subc.cc.u32 %1, %10, %18;\n\t"
            "subc.cc.u32 %2, %11, %19;\n\t"
            "subc.cc.u32 %3, %12, %20;\n\t"
            "subc.cc.u32 %4, %13, %21;\n\t"
            "subc.cc.u32 %5, %14, %22;\n\t"
            "subc.cc.u32 %6, %15, %23;\n\t"
            "subc.cc.u32 %7, %16, %24;\n\t"
            "subc.u32    %8, 0, 0;"
            : "=r"(s.v[0]), "=r"(s.v[1]), "=r"(s.v[2]), "=r"(s.v[3]), "=r"(s.v[4]), "=r"(s.v[5]), "=r"(s.v[6]),
              "=r"(s.v[7]), "=r"(br)
            : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
              "r"(a.v[7]), "n"(F::P(0)), "n"(F::P(1)), "n"(F::P(2)), "n"(F::P(3)), "n"(F::P(4)), "n"(F::P(5)),
              "n"(F::P(6)), "n"(F::P(7)));
        if (br) break;  // a < p
        a = s;
    }
    fe r2;
#pragma unroll
    for (int i = 0; i < 8; i++) r2.v[i] = F::R2(i);
    return fe_mul<F>(a, r2);
}

// Montgomery -> canonical in [0, p), for any 256-bit a: the product with 1 is below
// (1 + 2^-31) p + 1, one subtraction of p from its residue.
template <class F>
__device__ __forceinline__ fe fe_from_mont(const fe& a) {
    fe one;
#pragma unroll
    for (int i = 0; i < 8; i++) one.v[i] = i == 0 ? 1u : 0u;
    const fe r = fe_mul<F>(a, one);
    if constexpr (F::LAZY) return fe_reduce_once<F>(r);
    else return r;
}

// 32-byte element loads / stores as two 16-byte vector accesses
__device__ __forceinline__ fe fe_load(const fe* p) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 lo = q[0], hi = q[1];
    fe r;
    r.v[0] = lo.x;
    r.v[1] = lo.y;
    r.v[2] = lo.z;
    r.v[3] = lo.w;
    r.v[4] = hi.x;
    r.v[5] = hi.y;
    r.v[6] = hi.z;
    r.v[7] = hi.w;
    return r;
}

__device__ __forceinline__ fe fe_ldg(const fe* p) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 lo = __ldg(q), hi = __ldg(q + 1);
    fe r;
    r.v[0] = lo.x;
    r.v[1] = lo.y;
    r.v[2] = lo.z;
    r.v[3] = lo.w;
    r.v[4] = hi.x;
    r.v[5] = hi.y;
    r.v[6] = hi.z;
    r.v[7] = hi.w;
    return r;
}

__device__ __forceinline__ fe_const fe_ldg(const fe_const* p) { return {fe_ldg(&p->w), fe_ldg(&p->ws)}; }

// A 32-byte element through L2 only (ld.global.cg): for data that other CTAs wrote earlier
// in the same launch, which the non-coherent read-only path is not guaranteed to see.
__device__ __forceinline__ fe fe_ldcg(const fe* p) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 lo = __ldcg(q), hi = __ldcg(q + 1);
    fe r;
    r.v[0] = lo.x;
    r.v[1] = lo.y;
    r.v[2] = lo.z;
    r.v[3] = lo.w;
    r.v[4] = hi.x;
    r.v[5] = hi.y;
    r.v[6] = hi.z;
    r.v[7] = hi.w;
    return r;
}

__device__ __forceinline__ void fe_store(fe* p, const fe& a) {
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
    q[1] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
}

}  // namespace zk
