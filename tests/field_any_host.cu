// Host build of the product for unreduced factors (mul_rows_any of field.cuh) and of mul_rows with an
// unreduced second factor, against 128-bit host arithmetic: residues of a b 2^-256 on words of all
// ones, all zeros and random bits, half of them just below 2^256, where the running value is
// largest. argv[1]: the number of records; exit 0 when all agree. Built and run by
// tests/test_field_any_host.py.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../pyzkp_gb300/csrc/field.cuh"
#include "../pyzkp_gb300/csrc/host_field.hpp"

using zk::fe;

static std::mt19937_64 g(20251);
static long bad = 0;

static fe any() {
    uint64_t w[4];
    for (uint64_t& x : w) {
        x = g();
        switch (g() % 6) {
            case 0: x = 0; break;
            case 1: x = ~0ull; break;
            case 2: x |= 0xffffffff00000000ull; break;
        }
    }
    if (g() % 2) w[3] |= 0xf000000000000000ull;
    fe r;
    std::memcpy(r.v, w, 32);
    return r;
}

static zkh::F4 residue(const fe& a, const zkh::Field& F) {
    zkh::F4 r;
    std::memcpy(r.v, a.v, 32);
    while (zkh::geq(r.v, F.p)) zkh::sub4(r.v, r.v, F.p);
    return r;
}

template <class P>
static void check(const char* what, const fe& got, const fe& a, const fe& b, const zkh::Field& F) {
    const zkh::F4 want = zkh::mul(F, residue(a, F), residue(b, F)), have = residue(got, F);
    if (!zkh::eq(have, want) && bad++ < 5) std::printf("%s differs\n", what);
}

template <class P>
static void field(const zkh::Field& F, long records) {
    for (long i = 0; i < records; i++) {
        const fe a = any(), b = any();
        check<P>("unreduced factors", zk::mul_rows_any<P>(a, b), a, b, F);
        fe c;
        const zkh::F4 r = residue(a, F);
        std::memcpy(c.v, r.v, 32);
        check<P>("unreduced second factor", zk::mul_rows<P>(c, b), c, b, F);
    }
}

int main(int argc, char** argv) {
    const long records = argc > 1 ? std::atol(argv[1]) : 1000;
    field<zk::FrP>(zkh::fr(), records);
    field<zk::FqP>(zkh::fq(), records);
    std::printf("%ld differ\n", bad);
    return bad != 0;
}
