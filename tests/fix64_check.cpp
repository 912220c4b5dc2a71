// Host check of csrc/fix64.cuh against 128-bit integers and long double:
// fix64_check <count> <seed>.  Bounds: a complex product drops two terms of at most one unit per
// part, rounds once by a half and takes factors truncated by at most 2^-62 (operands of modulus
// 2^60.5: two times 0.71): 4 units; a quarter of it rounds by a half and drops a quarter of the
// rest, 2^62.5 in 4 units more of truncation: 3 units.  A 16-point transform sums 16 values
// with at most one product each: 16 * 4 units and the same again for an inverse.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "../qmctoolscl_gb300/csrc/fix64.cuh"

using namespace fx;

static u64 st;
static u64 rnd()
{
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st * 0x9E3779B97F4A7C15ull;
}
static i64 small(int bits) { return (i64)rnd() >> (64 - bits - 1); }

#define CHECK(c, ...)        \
    if (!(c)) {              \
        printf(__VA_ARGS__); \
        return 1;            \
    }

template <int NB>
static int check_dft()
{
    Cx x[16], y[16];
    for (int k = 0; k < 16; k++) x[k] = y[k] = Cx{small(57), small(57)};
    dft_regs<NB>(y);
    const int N = 1 << NB, G = 16 / N;
    for (int g = 0; g < G; g++)
        for (int p = 0; p < N; p++) {
            long double re = 0, im = 0;
            for (int j = 0; j < N; j++) {
                const Cx v = x[bitrev<NB>(j) * G + g];
                const long double a = -2 * M_PIl * ((j * p) % N) / N;
                re += v.r * cosl(a) - v.i * sinl(a);
                im += v.r * sinl(a) + v.i * cosl(a);
            }
            CHECK(fabsl(re - y[p * G + g].r) <= 128 && fabsl(im - y[p * G + g].i) <= 128, "dft%d %d\n", N, p);
        }
    Cx z[16];
    for (int k = 0; k < 16; k++) z[k] = Cx{y[k].r / N, y[k].i / N};
    idft_regs<NB>(z);
    for (int k = 0; k < 16; k++)
        CHECK(llabs(z[k].r - x[k].r) <= 256 && llabs(z[k].i - x[k].i) <= 256, "idft%d %d\n", N, k);
    return 0;
}

int main(int argc, char **argv)
{
    const long count = atol(argv[1]);
    st = 88172645463325252ull + (u64)atol(argv[2]) * 7919;
    const long double one62 = ldexpl(1, 62);
    for (long n = 0; n < count; n++) {
        // doubles in and out
        const u32 E = 300 + rnd() % 1200;
        u64 b = (rnd() & 0x800FFFFFFFFFFFFFull) | (u64)(E - rnd() % 70) << 52;
        if (n % 50 == 0) b &= 0x8000000000000000ull;
        const double v = of_bits(b);
        const i64 f = from_double<58>(v, E), f2 = from_double<60>(v, E);
        const long double unit = ldexpl(1, (int)E - 1080);
        CHECK(llabs(f) <= (1ll << 58) && fabsl((long double)f - v / unit) <= 0.5L, "from_double %.17g\n", v);
        CHECK(llabs(f2) <= (1ll << 60) && fabsl((long double)f2 - 4 * v / unit) <= 0.5L, "from_double %.17g\n", v);
        const i64 x = small(1 + rnd() % 61);
        const double d = to_double(x, (int)E - 1080);
        CHECK(fabsl(d / unit - x) <= fabsl((long double)x) * ldexpl(1, -53), "to_double %lld\n", x);
        if (llabs(x) < (1ll << 53)) CHECK(d / unit == (long double)x, "to_double exact %lld\n", x);
        for (int bits = 58; bits <= 60; bits += 2) {
            const int sh = excess(spread(x), bits);
            const i64 y = shift_by(x, sh > -28 ? sh : -28);
            CHECK(llabs(y) <= (1ll << bits) && (llabs(x) >> 32 == 0 || llabs(y) >= (1ll << (bits - 1)) - 1), "excess %lld\n", x);
        }
        // complex products
        const long double ang = 2 * M_PIl * (long double)rnd() / ldexpl(1, 64);
        const double c = n % 7 == 0 ? (double)(int)(rnd() % 3) - 1 : (double)cosl(ang);
        const double sn = n % 7 == 0 ? (c == 0 ? 1.0 : 0.0) : (double)sinl(ang);
        CHECK(fabsl(factor62(c) - c * one62) < 1, "factor62\n");
        const Tw w = make_tw(factor62(c), factor62(sn));
        const Cx a{small(60), small(60)};
        const Cx p = cmul<false, false>(a, w), q = cmul<true, false>(a, w);
        const long double ar = a.r, ai = a.i;
        CHECK(fabsl(p.r - (ar * c - ai * sn)) <= 4 && fabsl(p.i - (ar * sn + ai * c)) <= 4, "cmul\n");
        CHECK(fabsl(q.r - (ar * c + ai * sn)) <= 4 && fabsl(q.i - (ai * c - ar * sn)) <= 4, "cmul conj\n");
        const Cx g{a.r * 4, a.i * 4};  // up to 2^62 each
        const Cx u = cmul<false, true>(g, w);
        CHECK(fabsl(u.r - (ar * c - ai * sn)) <= 3 && fabsl(u.i - (ar * sn + ai * c)) <= 3, "cmul quarter\n");
        const Cx zero = cmul<false, false>(Cx{0, 0}, w), zero4 = cmul<false, true>(Cx{0, 0}, w);
        CHECK(zero.r == 0 && zero.i == 0 && zero4.r == 0 && zero4.i == 0, "cmul of zero\n");
        const Cx one = cmul<false, false>(a, make_tw(1ll << 62, 0));
        CHECK(one.r == a.r && one.i == a.i, "cmul by one\n");
        if (n % 16 == 0 && (check_dft<1>() || check_dft<2>() || check_dft<3>() || check_dft<4>())) return 1;
    }
    printf("ok %ld\n", count);
    return 0;
}
