// Host build of xyzz_mul (host_field.hpp) over a coordinate type that counts its products: the same
// point as double-and-add for small, sparse, dense and extreme scalars, for no more products. Exit 0
// when all hold. Built and run by tests/test_host_mul.py.
#include <cstdio>
#include <random>

#include "../pyzkp_gb300/csrc/host_field.hpp"

namespace counted {
struct C {
    zkh::F4 v;
};
static long products = 0;
inline C cadd(const C& a, const C& b) { return {zkh::cadd(a.v, b.v)}; }
inline C csub(const C& a, const C& b) { return {zkh::csub(a.v, b.v)}; }
inline C cmul(const C& a, const C& b) {
    products++;
    return {zkh::cmul(a.v, b.v)};
}
inline C csqr(const C& a) { return cmul(a, a); }
inline bool cis_zero(const C& a) { return zkh::cis_zero(a.v); }
}  // namespace counted

using counted::C;
using Point = zkh::XyzzT<C>;

static Point double_and_add(const Point& p, const zkh::F4& k) {
    Point acc = zkh::xyzz_inf<C>();
    for (int i = 255; i >= 0; i--) {
        acc = zkh::xyzz_dbl(acc);
        if ((k.v[i >> 6] >> (i & 63)) & 1) acc = zkh::xyzz_add(acc, p);
    }
    return acc;
}

static void affine(const Point& p, zkh::F4* x, zkh::F4* y) {
    const zkh::Xyzz q{p.X.v, p.Y.v, p.ZZ.v, p.ZZZ.v};
    zkh::xyzz_to_affine_canonical(q, x, y);
}

static long bad = 0;

static void check(const Point& p, const zkh::F4& k) {
    counted::products = 0;
    const Point want = double_and_add(p, k);
    const long most = counted::products;
    counted::products = 0;
    const Point got = zkh::xyzz_mul(p, k);
    const long used = counted::products;
    zkh::F4 x, y, u, v;
    affine(want, &x, &y);
    affine(got, &u, &v);
    if (!zkh::eq(x, u) || !zkh::eq(y, v) || used > most) {
        if (bad++ < 5)
            std::printf("k = %016llx%016llx%016llx%016llx: %ld products against %ld\n", (unsigned long long)k.v[3],
                        (unsigned long long)k.v[2], (unsigned long long)k.v[1], (unsigned long long)k.v[0], used, most);
    }
}

int main() {
    Point g;
    g.X = {zkh::cto_mont(zkh::F4{{1, 0, 0, 0}})};
    g.Y = {zkh::cto_mont(zkh::F4{{2, 0, 0, 0}})};
    g.ZZ = g.ZZZ = {zkh::one(zkh::fq())};
    std::mt19937_64 r(11);
    for (uint64_t k = 0; k < 300; k++) check(g, {{k, 0, 0, 0}});
    for (int b = 0; b < 254; b++) {
        zkh::F4 k{{0, 0, 0, 0}};
        k.v[b / 64] = 1ull << (b % 64);
        check(g, k);
        k.v[0] |= 1;
        check(g, k);
        for (int j = 0; j < b / 64; j++) k.v[j] = ~0ull;  // 2^b and every bit of the words below
        check(g, k);
        zkh::F4 d{{r(), r(), r(), r()}};  // random of b bits
        for (int j = 0; j < 4; j++) d.v[j] = j > b / 64 ? 0 : j < b / 64 ? d.v[j] : d.v[j] & ((1ull << (b % 64)) - 1);
        check(g, d);
    }
    for (uint64_t e = 1; e < 20; e++) {  // r - e
        zkh::F4 k;
        const uint64_t d[4] = {e, 0, 0, 0};
        zkh::sub4(k.v, zkh::fr().p, d);
        check(g, k);
    }
    std::printf("%ld differ\n", bad);
    return bad != 0;
}
