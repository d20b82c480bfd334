// Host build of the product rows of field.cuh (mul_rows, mul_add_rows, the square and the
// separated reduction): the template code the device runs, with the carry flag emulated on the
// host, against 128-bit host arithmetic (host_field.hpp). Operands are lazy values in [0, 2p)
// built from limbs of all zeros, all ones and random words, which drive the running value to
// the edges of its 9 limbs. argv[1]: the number of records; exit 0 when all agree. Built and run
// by tests/test_field_rows_host.py.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../pyzkp_gb300/csrc/field.cuh"
#include "../pyzkp_gb300/csrc/host_field.hpp"

using zk::fe;

static zkh::F4 words(const fe& a) {
    zkh::F4 r;
    std::memcpy(r.v, a.v, 32);
    return r;
}

static zkh::F4 canon(zkh::F4 a, const zkh::Field& F) {
    while (zkh::geq(a.v, F.p)) zkh::sub4(a.v, a.v, F.p);
    return a;
}

struct Gen {
    std::mt19937_64 g{20240607};
    fe lazy(const zkh::Field& F) {  // a value in [0, 2p); one in eight is 2p - 1 - (a small word)
        uint64_t p2[4];
        zkh::add4(p2, F.p, F.p);
        zkh::F4 t;
        if (g() % 8 == 0) {
            const uint64_t d[4] = {1 + g() % 4, 0, 0, 0};
            zkh::sub4(t.v, p2, d);
        } else {
            for (int j = 0; j < 4; j++) {
                uint64_t v = g();
                switch (g() % 8) {
                    case 0: v = 0; break;
                    case 1: v = ~0ull; break;
                    case 2: v &= 0xffffffffull; break;
                    case 3: v |= 0xffffffff00000000ull; break;
                }
                t.v[j] = v;
            }
            t.v[3] &= 0x7fffffffffffffffull;
            while (zkh::geq(t.v, p2)) zkh::sub4(t.v, t.v, p2);
        }
        fe x;
        std::memcpy(x.v, t.v, 32);
        return x;
    }
};

// floor(w 2^256 / p) by long division, bit by bit
static zkh::F4 quotient(const zkh::F4& w, const zkh::Field& F) {
    zkh::F4 rem = w, q = {{0, 0, 0, 0}};
    for (int i = 0; i < 256; i++) {
        zkh::add4(rem.v, rem.v, rem.v);  // rem < p < 2^254: no carry
        for (int j = 3; j > 0; j--) q.v[j] = (q.v[j] << 1) | (q.v[j - 1] >> 63);
        q.v[0] <<= 1;
        if (zkh::geq(rem.v, F.p)) {
            zkh::sub4(rem.v, rem.v, F.p);
            q.v[0] |= 1;
        }
    }
    return q;
}

static long bad = 0;

static void check(const char* what, const fe& got, const zkh::F4& want, const zkh::Field& F) {
    uint64_t p2[4];
    zkh::add4(p2, F.p, F.p);
    const zkh::F4 g = words(got), c = canon(g, F);
    if (zkh::geq(g.v, p2) || std::memcmp(&c, &want, 32) != 0) {
        if (bad++ < 5) std::printf("%s differs\n", what);
    }
}

int main(int argc, char** argv) {
    const long records = argc > 1 ? std::atol(argv[1]) : 1000;
    Gen gen;
    const zkh::Field &Q = zkh::fq(), &R = zkh::fr();
    for (long i = 0; i < records; i++) {
        const fe a = gen.lazy(Q), b = gen.lazy(Q), c = gen.lazy(Q), d = gen.lazy(Q);
        const zkh::F4 A = canon(words(a), Q), B = canon(words(b), Q), C = canon(words(c), Q), D = canon(words(d), Q);
        const zkh::F4 ab = zkh::mul(Q, A, B), cd = zkh::mul(Q, C, D);
        check("Fq product", zk::mul_rows<zk::FqP>(a, b), ab, Q);
        check("Fq separated product", zk::fe_mul_sos<zk::FqP>(a, b), ab, Q);
        check("Fq square", zk::fe_sqr_sos<zk::FqP>(a), zkh::mul(Q, A, A), Q);
        check("Fq a b + c d", zk::fe_mul_add_sos<zk::FqP>(a, b, c, d), zkh::add(Q, ab, cd), Q);
        check("Fq a b - c d", zk::fe_mul_sub_sos<zk::FqP>(a, b, c, d), zkh::sub(Q, ab, cd), Q);
        const zk::fe_pair f = zk::fe2_mul_lazy<zk::FqP>(a, b, c, d);  // (a + b u)(c + d u)
        check("Fq2 product, 1", f.c0, zkh::sub(Q, zkh::mul(Q, A, C), zkh::mul(Q, B, D)), Q);
        check("Fq2 product, u", f.c1, zkh::add(Q, zkh::mul(Q, A, D), zkh::mul(Q, B, C)), Q);
        const fe x = gen.lazy(R), y = gen.lazy(R);
        // x w for a constant w with floor(w 2^256 / r), x below 4r (a sum of two lazy values)
        zk::fe_const k;
        const zkh::F4 W = canon(words(gen.lazy(R)), R), ws = quotient(W, R);
        std::memcpy(k.w.v, W.v, 32);
        std::memcpy(k.ws.v, ws.v, 32);
        const fe u = gen.lazy(R), v = gen.lazy(R);
        zkh::F4 x4;
        zkh::add4(x4.v, words(u).v, words(v).v);
        fe xs;
        std::memcpy(xs.v, x4.v, 32);
        const zkh::F4 xw = zkh::mul(R, zkh::to_mont(R, canon(x4, R)), W);
        check("Fr product with a constant", zk::fe_mul_const<zk::FrLazyP>(xs, k), xw, R);
        const fe du = zk::fe_sub_4p<zk::FrLazyP>(u, v);
        const zkh::F4 duv = zkh::sub(R, canon(words(u), R), canon(words(v), R));
        check("Fr (u - v) w", zk::fe_mul_const<zk::FrLazyP>(du, k), zkh::mul(R, zkh::to_mont(R, duv), W), R);
        check("Fr product", zk::mul_rows<zk::FrLazyP>(x, y), zkh::mul(R, canon(words(x), R), canon(words(y), R)), R);
    }
    std::printf("%ld differ\n", bad);
    return bad != 0;
}
