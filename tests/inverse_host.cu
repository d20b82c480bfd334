// Host build of fe_almost_inverse (inverse.cuh): a s = 2^k mod p with 253 <= k <= 508 and s < p for
// canonical a, on edges and random words, and its end for the arguments outside that: 0, the
// multiples of p and 2^256 - 1. argv[1]: the number of random values; exit 0 when all hold. Built and
// run by tests/test_inverse_host.py under a time limit (an argument without an end would hang).
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../pyzkp_gb300/csrc/host_field.hpp"
#include "../pyzkp_gb300/csrc/inverse.cuh"

static long bad = 0;

static zk::fe limbs(const zkh::F4& a) {
    zk::fe r;
    std::memcpy(r.v, a.v, 32);
    return r;
}

static void check(const char* what, bool ok) {
    if (!ok && bad++ < 5) std::printf("%s\n", what);
}

template <class F>
static void canonical(const zkh::Field& P, const zkh::F4& a) {
    zk::fe s;
    uint32_t k = 0;
    if (zkh::is_zero(a)) {
        check("zero has an inverse", !zk::fe_almost_inverse<F>(limbs(a), &s, &k));
        return;
    }
    check("no inverse", zk::fe_almost_inverse<F>(limbs(a), &s, &k));
    check("k out of range", k >= 253 && k <= 508);
    zkh::F4 s4, two = {{1, 0, 0, 0}};
    std::memcpy(s4.v, s.v, 32);
    check("s not below p", !zkh::geq(s4.v, P.p));
    for (uint32_t i = 0; i < k; i++) two = zkh::add(P, two, two);
    check("a s differs from 2^k", zkh::eq(zkh::mul(P, zkh::to_mont(P, a), s4), two));
}

template <class F>
static void field(const zkh::Field& P, long records) {
    const zkh::F4 p = {{P.p[0], P.p[1], P.p[2], P.p[3]}};
    for (uint64_t e = 0; e < 4; e++) {
        canonical<F>(P, {{e, 0, 0, 0}});
        if (e) {
            const uint64_t d[4] = {e, 0, 0, 0};
            zkh::F4 t;
            zkh::sub4(t.v, P.p, d);
            canonical<F>(P, t);
        }
    }
    for (int b = 0; b < 254; b++) {
        zkh::F4 t = {{0, 0, 0, 0}};
        t.v[b / 64] = 1ull << (b % 64);
        if (!zkh::geq(t.v, P.p)) canonical<F>(P, t);
    }
    std::mt19937_64 g(7);
    for (long i = 0; i < records; i++) {
        zkh::F4 t = {{g(), g(), g(), g() >> 2}};
        while (zkh::geq(t.v, P.p)) zkh::sub4(t.v, t.v, P.p);
        canonical<F>(P, t);
    }
    zk::fe s;
    uint32_t k = 0;
    zkh::F4 m = p;
    for (int i = 1; i <= 5; i++) {  // p .. 5p < 2^256
        zk::fe_almost_inverse<F>(limbs(m), &s, &k);
        check("k above 510", k <= 510);
        zkh::add4(m.v, m.v, P.p);
    }
    zk::fe_almost_inverse<F>(limbs({{~0ull, ~0ull, ~0ull, ~0ull}}), &s, &k);
    check("k above 510", k <= 510);
}

int main(int argc, char** argv) {
    const long records = argc > 1 ? std::atol(argv[1]) : 1000;
    field<zk::FrP>(zkh::fr(), records);
    field<zk::FqP>(zkh::fq(), records);
    std::printf("%ld differ\n", bad);
    return bad != 0;
}
