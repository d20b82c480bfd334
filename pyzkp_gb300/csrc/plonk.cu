// plonk.cu -- the PLONK quotient step on the device: BATCH_INV and the fused
// PLONK_T_QUOTIENT_EVALS op.
//
// BATCH_INV (runtime/kernels/cpu/kernels.py:_batch_inv -> crypto/field/batch.py:8-38):
// out[i] = in[i]^-1, and 0 where in[i] == 0, by Montgomery's trick: each lane takes kInvChunk
// elements (prefix products, a backward pass), the lanes' products are combined by the warp
// and inverted once, by every lane alike (binary extended Euclid: no divergence).
//
// PLONK_T_QUOTIENT_EVALS (runtime/kernels/cpu/kernels.py:_plonk_t_quotient_evals, used by
// protocols/plonk/prove.py:395-416): at x_i = shift * omega_m^i, i < m, from the
// extended-coset evaluations of a, b, c, z, pi, ql, qr, qm, qo, qc, s1, s2, s3, z(omega x)
// and L1, with u = omega_m^n:
//   gate  = ql a + qr b + qm a b + qo c + qc + pi
//   perm  = (a + beta x + gamma)(b + beta k1 x + gamma)(c + beta k2 x + gamma) z
//         - (a + beta s1 + gamma)(b + beta s2 + gamma)(c + beta s3 + gamma) z(omega x)
//   num_i = gate + alpha perm + alpha^2 (z - 1) L1
//   zh_i  = shift_n u^i - 1
// One thread per `chunk` points, 32 apart (a warp covers 32 * chunk consecutive points, so
// its loads are contiguous), the powers of omega_m and u carried from the thread's first
// point (from tables) in steps of omega_m^32 and u^32.
#include <cstring>
#include <vector>

#include "inverse.cuh"
#include "zk_internal.cuh"

namespace zk {

// (8 / 16 / 32 elements a lane: 86 / 66 / 78 us at 2^19, 260 / 188 / 185 at 2^21, 40 / 51 / 74 at 2^10)
static constexpr uint32_t kInvChunk = 16;
static constexpr uint32_t kInvWarp = 32 * kInvChunk;  // elements of a warp
// Points a thread takes at most: the starting powers cost it 7 products. Fewer while there are
// fewer than kQWarps warps per SM (a point is a chain of ~25
// products). Measured on GB300, 16 points always / so: the quotient step of 2^8 (m = 2^10) 316 -> 126
// us, 2^12 345 -> 148, 2^17 1576 -> 1498.
static constexpr uint32_t kQChunk = 16;
static constexpr uint32_t kQWarps = 32;

// The inverse of a Montgomery form a = x R (canonical): x^-1 R, and 0 for 0. s = a^-1 2^k =
// x^-1 R^-1 2^k from fe_almost_inverse, then x^-1 R = s 2^(512 - k), by a product with
// 2^(512 - k) / R and one with R^2. (a^(p - 2) takes 384 dependent products, ~150 us a thread.)
template <class F>
__device__ fe fe_inverse_binary(const fe& a) {
    fe s;
    uint32_t k;
    if (!fe_almost_inverse<F>(a, &s, &k)) return fe_zero();
    uint32_t j = 512 - k;
    while (j > 253) {  // 2^j below 2^254
        s = fe_add<F>(s, s);
        j--;
    }
    fe t = fe_zero(), r2;
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
        t.v[i] = i == j / 32 ? 1u << (j % 32) : 0u;
        r2.v[i] = F::R2(i);
    }
    return fe_mul<F>(fe_mul<F>(s, t), r2);
}

__device__ __forceinline__ fe fe_shfl_up(const fe& a, uint32_t d) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_up_sync(0xffffffffu, a.v[i], d);
    return r;
}
__device__ __forceinline__ fe fe_shfl_down(const fe& a, uint32_t d) {
    fe r;
#pragma unroll
    for (int i = 0; i < 8; i++) r.v[i] = __shfl_down_sync(0xffffffffu, a.v[i], d);
    return r;
}

// out must not alias in: the backward pass reads in[] again (out holds the prefixes). A lane's
// elements are 32 apart, so that the warp reads and writes whole lines. Measured at 2^19
// elements: 229 -> 66 us against a Fermat inversion per 32 consecutive elements (384 dependent
// products, and each lane's accesses a kilobyte from the next one's).
//
// An element counts as zero when it is a multiple of r, whatever its bits: when its product with
// a value that is not zero is (fe_mul takes any 256-bit second factor), so the running products
// stay non-zero.
__global__ void __launch_bounds__(128) fr_batch_inv_kernel(fe* __restrict__ out, const fe* __restrict__ in, size_t n) {
    if (!grid_enter()) return;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const size_t i0 = warp * kInvWarp + lane;
    if (warp * kInvWarp >= n) return;
    fe acc = fe_one<FrP>();
    for (uint32_t j = 0; j < kInvChunk; j++) {
        const size_t i = i0 + 32 * j;
        if (i >= n) break;
        fe_store(out + i, acc);  // product of the lane's non-zero inputs before i
        const fe t = fe_mul<FrP>(acc, fe_ldg(in + i));
        if (!fe_is_zero(t)) acc = t;
    }
    __syncwarp();
    // products of the lanes before (pre) and after (suf) this one
    fe pre = fe_shfl_up(acc, 1), suf = fe_shfl_down(acc, 1);
    if (lane == 0) pre = fe_one<FrP>();
    if (lane == 31) suf = fe_one<FrP>();
#pragma unroll 1
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const fe a = fe_shfl_up(pre, d), b = fe_shfl_down(suf, d);
        if (lane >= d) pre = fe_mul<FrP>(pre, a);
        if (lane + d < 32) suf = fe_mul<FrP>(suf, b);
        __syncwarp();
    }
    const fe others = fe_mul<FrP>(pre, suf);
    fe total = fe_mul<FrP>(others, acc);  // the same value in every lane, and not zero
    fe inv = fe_mul<FrP>(fe_inverse_binary<FrP>(total), others);
    for (uint32_t j = kInvChunk; j-- > 0;) {
        const size_t i = i0 + 32 * j;
        if (i >= n) continue;
        const fe t = fe_mul<FrP>(inv, fe_ldg(in + i));
        if (fe_is_zero(t)) {
            fe_store(out + i, fe_zero());
        } else {
            fe_store(out + i, fe_mul<FrP>(fe_load(out + i), inv));
            inv = t;
        }
    }
}

// The quotient kernel holds ~23 products per element: Fr with the non-inlined product
using FrQ = FrCallP;

struct QuotientIn {
    const fe* v[15];  // a b c z pi ql qr qm qo qc s1 s2 s3 zshift l1 (Montgomery)
};

struct QuotientK {  // Montgomery constants
    fe omega_m, u, shift, shift_n, alpha, alpha2, beta, gamma, beta_k1, beta_k2, one;
    fe omega_step, u_step;  // omega_m^32, u^32: a lane's step
};

// Starting powers of a lane, from tables (Montgomery): with i0 = w g + l (warp g of w = 32 chunk
// points, lane l), v^i0 = v^l * v^(w (g mod 64)) * v^(64 w (g / 64)) for v = omega_m and v = u:
//   pw[l], pw[32 + l]              omega_m^l, u^l                        (l < 32)
//   pw[64 + j], pw[128 + j]        omega_m^(w j), u^(w j)           (j < 64)
//   pw[192 + h], pw[192 + H + h]   omega_m^(64 w h), u^(64 w h)       (h < H)
// 4 products per thread instead of ~2 log2(i0) by square-and-multiply for each of the two.

__global__ void plonk_quotient_kernel(QuotientIn in, QuotientK K, size_t m, uint32_t chunk, const fe* __restrict__ pw,
                                      uint32_t H, fe* __restrict__ num, fe* __restrict__ zh) {
    if (!grid_enter()) return;
    // a warp covers 32 * chunk consecutive points, lane l the points base + l + 32 k (each
    // load of the warp reads 32 consecutive elements)
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t lane = t & 31;
    const size_t i0 = (t - lane) * chunk + lane;
    if (i0 >= m) return;
    const size_t g = t >> 5;
    const uint32_t glo = (uint32_t)(g & 63), ghi = (uint32_t)(g >> 6);
    fe x = fe_mul<FrQ>(fe_mul<FrQ>(fe_ldg(pw + lane), fe_ldg(pw + 64 + glo)), fe_ldg(pw + 192 + ghi));
    x = fe_mul<FrQ>(K.shift, x);
    fe un = fe_mul<FrQ>(fe_mul<FrQ>(fe_ldg(pw + 32 + lane), fe_ldg(pw + 128 + glo)), fe_ldg(pw + 192 + H + ghi));
    // the vectors of a caller that are first factors of products (see fe_mul)
    auto first = [](const fe* v) { return fe_first_factor<FrQ>(fe_ldg(v)); };
    for (size_t i = i0, k = 0; k < chunk && i < m; k++, i += 32) {
        const fe a = first(in.v[0] + i), b = first(in.v[1] + i), c = first(in.v[2] + i);
        const fe z = first(in.v[3] + i);
        fe gate = fe_add<FrQ>(fe_mul<FrQ>(a, fe_ldg(in.v[5] + i)), fe_mul<FrQ>(b, fe_ldg(in.v[6] + i)));
        gate = fe_add<FrQ>(gate, fe_mul<FrQ>(fe_mul<FrQ>(a, fe_ldg(in.v[7] + i)), b));
        gate = fe_add<FrQ>(gate, fe_mul<FrQ>(c, fe_ldg(in.v[8] + i)));
        gate = fe_add<FrQ>(gate, fe_add<FrQ>(fe_ldg(in.v[9] + i), fe_ldg(in.v[4] + i)));
        const fe t1 = fe_add<FrQ>(fe_add<FrQ>(a, fe_mul<FrQ>(K.beta, x)), K.gamma);
        const fe t2 = fe_add<FrQ>(fe_add<FrQ>(b, fe_mul<FrQ>(K.beta_k1, x)), K.gamma);
        const fe t3 = fe_add<FrQ>(fe_add<FrQ>(c, fe_mul<FrQ>(K.beta_k2, x)), K.gamma);
        const fe left = fe_mul<FrQ>(fe_mul<FrQ>(fe_mul<FrQ>(t1, t2), t3), z);
        const fe u1 = fe_add<FrQ>(fe_add<FrQ>(a, fe_mul<FrQ>(K.beta, fe_ldg(in.v[10] + i))), K.gamma);
        const fe u2 = fe_add<FrQ>(fe_add<FrQ>(b, fe_mul<FrQ>(K.beta, fe_ldg(in.v[11] + i))), K.gamma);
        const fe u3 = fe_add<FrQ>(fe_add<FrQ>(c, fe_mul<FrQ>(K.beta, fe_ldg(in.v[12] + i))), K.gamma);
        const fe right = fe_mul<FrQ>(fe_mul<FrQ>(fe_mul<FrQ>(u1, u2), u3), fe_ldg(in.v[13] + i));
        const fe perm = fe_sub<FrQ>(left, right);
        const fe boundary = fe_mul<FrQ>(fe_sub<FrQ>(z, K.one), fe_ldg(in.v[14] + i));
        const fe v = fe_add<FrQ>(gate, fe_add<FrQ>(fe_mul<FrQ>(K.alpha, perm), fe_mul<FrQ>(K.alpha2, boundary)));
        fe_store(num + i, v);
        fe_store(zh + i, fe_sub<FrQ>(fe_mul<FrQ>(K.shift_n, un), K.one));
        un = fe_mul<FrQ>(un, K.u_step);
        x = fe_mul<FrQ>(x, K.omega_step);
    }
}

static fe mont_fr(const uint8_t canonical[32]) {
    zkh::F4 v;
    std::memcpy(v.v, canonical, 32);
    const zkh::F4 m = zkh::to_mont(zkh::fr(), v);
    fe r;
    std::memcpy(r.v, m.v, 32);
    return r;
}

static fe mont_of(const zkh::F4& m) {
    fe r;
    std::memcpy(r.v, m.v, 32);
    return r;
}

}  // namespace zk

using zk::fe;

extern "C" {

int zk_fr_batch_inv(zk_ctx* ctx, void* out, const void* in, size_t n) {
    if (ctx == nullptr) {
        zk::set_error("null zk_ctx");
        return ZK_EINVAL;
    }
    if (n == 0) return ZK_OK;
    if (!out || !in) {
        zk::set_error("null buffer");
        return ZK_EINVAL;
    }
    ZK_TRY_CUDA(cudaSetDevice(ctx->impl.device));
    zk::Ctx* c = &ctx->impl;
    const fe* src = static_cast<const fe*>(in);
    void* copy = nullptr;
    if (out == in) {  // the kernel keeps its prefixes in out and re-reads in: copy the input
        int rc = zk::scratch_alloc(c, n * 32, &copy);
        if (rc != ZK_OK) return rc;
        ZK_TRY_CUDA(cudaMemcpyAsync(copy, in, n * 32, cudaMemcpyDeviceToDevice, c->stream));
        src = static_cast<const fe*>(copy);
    }
    const size_t warps = (n + zk::kInvWarp - 1) / zk::kInvWarp;
    ZK_LAUNCH_NEXT(c, "fr_batch_inv", zk::fr_batch_inv_kernel, (unsigned)((warps + 3) / 4), 128, 0,
              static_cast<fe*>(out), src, n);
    ZK_TRY_CUDA(cudaGetLastError());
    if (copy) zk::scratch_free(c, copy);
    return ZK_OK;
}

int zk_plonk_quotient_evals(zk_ctx* ctx, const void* const* inputs, size_t m, uint64_t n, const uint8_t omega_m[32],
                            const uint8_t shift[32], const uint8_t shift_n[32], const uint8_t alpha[32],
                            const uint8_t beta[32], const uint8_t gamma[32], const uint8_t k1[32],
                            const uint8_t k2[32], void* num_out, void* zh_out) {
    if (ctx == nullptr) {
        zk::set_error("null zk_ctx");
        return ZK_EINVAL;
    }
    if (m == 0) return ZK_OK;
    if (!inputs || !num_out || !zh_out || !omega_m || !shift || !shift_n || !alpha || !beta || !gamma || !k1 || !k2) {
        zk::set_error("null pointer");
        return ZK_EINVAL;
    }
    ZK_TRY_CUDA(cudaSetDevice(ctx->impl.device));
    zk::QuotientIn in;
    for (int i = 0; i < 15; i++) {
        if (inputs[i] == nullptr) {
            zk::set_error("null input vector");
            return ZK_EINVAL;
        }
        in.v[i] = static_cast<const fe*>(inputs[i]);
    }
    const zkh::Field& F = zkh::fr();
    zk::QuotientK K;
    K.omega_m = zk::mont_fr(omega_m);
    zkh::F4 om;
    std::memcpy(om.v, omega_m, 32);
    K.u = zk::mont_of(zkh::pow_u64(F, zkh::to_mont(F, om), n));
    K.shift = zk::mont_fr(shift);
    K.shift_n = zk::mont_fr(shift_n);
    K.alpha = zk::mont_fr(alpha);
    zkh::F4 a;
    std::memcpy(a.v, alpha, 32);
    const zkh::F4 am = zkh::to_mont(F, a);
    K.alpha2 = zk::mont_of(zkh::mul(F, am, am));
    K.beta = zk::mont_fr(beta);
    K.gamma = zk::mont_fr(gamma);
    zkh::F4 b, kk1, kk2;
    std::memcpy(b.v, beta, 32);
    std::memcpy(kk1.v, k1, 32);
    std::memcpy(kk2.v, k2, 32);
    const zkh::F4 bm = zkh::to_mont(F, b);
    K.beta_k1 = zk::mont_of(zkh::mul(F, bm, zkh::to_mont(F, kk1)));
    K.beta_k2 = zk::mont_of(zkh::mul(F, bm, zkh::to_mont(F, kk2)));
    K.one = zk::mont_of(zkh::one(F));
    K.omega_step = zk::mont_of(zkh::pow_u64(F, zkh::to_mont(F, om), 32));
    K.u_step = zk::mont_of(zkh::pow_u64(F, zkh::pow_u64(F, zkh::to_mont(F, om), n), 32));
    zk::Ctx* c = &ctx->impl;
    // the starting-power tables of the kernel (see plonk_quotient_kernel)
    uint32_t chunk = zk::kQChunk;
    while (chunk > 1 && m < 32ull * chunk * zk::kQWarps * c->num_sms) chunk /= 2;
    const uint64_t points = 32ull * chunk, warps = (m + points - 1) / points;
    const uint32_t H = (uint32_t)((warps + 63) / 64);
    std::vector<zkh::F4> pw(192 + 2 * (size_t)H);
    const zkh::F4 om_m = zkh::to_mont(F, om);
    const zkh::F4 u_m = zkh::pow_u64(F, om_m, n);
    struct Run {
        size_t at;
        zkh::F4 base;
        size_t count;
    };
    const Run runs[6] = {{0, om_m, 32},
                         {32, u_m, 32},
                         {64, zkh::pow_u64(F, om_m, points), 64},
                         {128, zkh::pow_u64(F, u_m, points), 64},
                         {192, zkh::pow_u64(F, om_m, 64 * points), H},
                         {192 + (size_t)H, zkh::pow_u64(F, u_m, 64 * points), H}};
    for (const Run& r : runs) {
        zkh::F4 cur = zkh::one(F);
        for (size_t i = 0; i < r.count; i++) {
            pw[r.at + i] = cur;
            cur = zkh::mul(F, cur, r.base);
        }
    }
    void* d_pw = nullptr;
    int rc = zk::scratch_alloc(c, pw.size() * 32, &d_pw);
    if (rc != ZK_OK) return rc;
    ZK_TRY_CUDA(cudaMemcpyAsync(d_pw, pw.data(), pw.size() * 32, cudaMemcpyHostToDevice, c->stream));
    ZK_LAUNCH_NEXT(c, "plonk_quotient", zk::plonk_quotient_kernel, (unsigned)((warps + 3) / 4), 128, 0, in, K, m, chunk,
              static_cast<const fe*>(d_pw), H, static_cast<fe*>(num_out), static_cast<fe*>(zh_out));
    ZK_TRY_CUDA(cudaGetLastError());
    zk::scratch_free(c, d_pw);
    return ZK_OK;
}

}  // extern "C"
