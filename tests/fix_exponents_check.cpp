// Host check of the exponents in csrc/fix64.cuh: fix_exponents_check <count> <seed>.  Shifts against
// 128-bit integers, the exponent that a block is brought to, and 16-point transforms whose classes are lifted
// against long double: an output is off by at most 16 units of its own class (a rotation is off by 4
// at most, four stages of adds add four of them up).
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
static i64 upto(int bits) { return bits ? (i64)rnd() >> (63 - bits) : 0; }  // |.| <= 2^bits

#define CHECK(c, ...)        \
    if (!(c)) {              \
        printf(__VA_ARGS__); \
        return 1;            \
    }

// as the kernels do it, on an array
struct Lift {
    int room;
    template <bool FWD>
    void operator()(Cx (&x)[16], Lifts &out) const
    {
        if (!may_lift<FWD>(x)) return;
        for (int j = 1; j < 4; j++) {
            u64 mag = 0;
                for (int i = 0; i < 4; i++) mag |= mag64(x[FWD ? j + 4 * i : 4 * j + i]);
            const int s = lift_of(mag, room);
            out.s[j] = s;
                for (int i = 0; i < 4; i++) x[FWD ? j + 4 * i : 4 * j + i] = shift_any(x[FWD ? j + 4 * i : 4 * j + i], -s);
        }
    }
};

template <int NB, bool FWD>
static int check_lifted()
{
    constexpr int N = 1 << NB, G = 16 / N;
    const int deep = (int)(rnd() % 58);
    Cx x[16], y[16];
    for (int k = 0; k < 16; k++) {  // alike but for the lowest bits, in a random pattern of signs
        const i64 c = 1ll << 57, s = (rnd() & 1) ? 1 : -1;
        x[k] = y[k] = rnd() % 4 ? Cx{c + upto(deep), upto(deep)} : Cx{s * c + upto(deep), upto(deep)};
    }
    const Lifts l = FWD ? dft_regs<NB>(y, Lift{1000}) : idft_regs<NB>(y, Lift{1000});
    for (int g = 0; g < G; g++)
        for (int p = 0; p < N; p++) {
            long double re = 0, im = 0;
            for (int j = 0; j < N; j++) {
                const Cx v = x[(FWD ? bitrev<NB>(j) : j) * G + g];
                const int q = FWD ? p : bitrev<NB>(p);  // inverse: output bit-reversed
                const long double a = (FWD ? -2 : 2) * M_PIl * ((j * q) % N) / N;
                const long double c = (j * q) % N * 4 % N == 0 ? roundl(cosl(a)) : cosl(a), s = (j * q) % N * 4 % N == 0 ? roundl(sinl(a)) : sinl(a);
                re += v.r * c - v.i * s;
                im += v.r * s + v.i * c;
            }
            const int k = p * G + g, s = l.s[FWD ? dft_class<NB>(k) : idft_class<NB>(k)];
            CHECK(s >= 0 && llabs(y[k].r) < (1ll << 62) + (1ll << 61) && llabs(y[k].i) < (1ll << 62) + (1ll << 61), "range\n");
            // the sum itself is rounded to 64 bits in long double: 16 terms of 2^57, up to 2^61
            const long double tol = 16 * ldexpl(1, -s) + 4;
            CHECK(fabsl(re - ldexpl(y[k].r, -s)) <= tol && fabsl(im - ldexpl(y[k].i, -s)) <= tol, "lifted %d %d: %Lg\n", NB, k,
                  re - ldexpl(y[k].r, -s));
        }
    return 0;
}

int main(int argc, char **argv)
{
    const long count = atol(argv[1]);
    st = 88172645463325252ull + (u64)atol(argv[2]) * 7919;
    for (long n = 0; n < count; n++) {
        const i64 x = upto((int)(rnd() % 63));
        const int b = bits64(x);
        CHECK((x == 0) == (b == 0) && (x == 0 || ((__int128)llabs(x) <= (__int128)1 << b && llabs(x) >= (1ll << b >> 1))), "bits64 %lld\n", x);
        const int s = (int)(rnd() % 90) - (62 - b < 40 ? 62 - b : 40);
        const __int128 want = s <= 0 ? (__int128)x << -s : ((__int128)x + ((__int128)1 << (s - 1))) >> s;
        CHECK(shift_any(x, s) == (s < 63 ? (i64)want : 0), "shift_any %lld %d\n", x, s);
        if (s >= 0 && s < 32) CHECK(round_shift(x, (u32)s) == (i64)want, "round_shift %lld %d\n", x, s);
        // a block's common exponent: the largest value just below 2^58, the others no coarser than half its unit
        i64 v[16];
        int e[16], low = -1000 + (int)(rnd() % 200);
        for (int k = 0; k < 16; k++) {
            v[k] = rnd() % 5 ? upto((int)(rnd() % 62)) : 0;
            e[k] = v[k] ? (int)(rnd() % 80) - 700 : E_ZERO;
        }
        const int to = common_exponent(16, 58, low, [&](int k) { return v[k]; }, [&](int k) { return e[k]; });
        bool any = false;
        long double top = 0;
        for (int k = 0; k < 16; k++) {
            any = any || v[k];
            top = fmaxl(top, fabsl(ldexpl(v[k], e[k])));
            CHECK(fabsl(ldexpl(shift_any(v[k], to - e[k]), to) - ldexpl(v[k], e[k])) <= ldexpl(0.5L, to), "align %d\n", k);
        }
        CHECK(any ? to >= low && top <= ldexpl(1, to + 58) && (to == low || top >= ldexpl(1, to + 56)) : to == E_ZERO, "common_exponent\n");
        const u64 mag = (u64)upto((int)(rnd() % 62)) & 0x7FFFFFFFFFFFFFFFull;
        const int room = (int)(rnd() % 100) - 20, up = lift_of(mag, room);
        CHECK(up >= 0 && up <= (room > 0 ? room : 0) && (up == 0 || (mag << up >> up == mag && mag << up < 1ull << 60)), "lift_of\n");
        if (n % 4 == 0 && (check_lifted<4, true>() || check_lifted<3, true>() || check_lifted<2, true>() || check_lifted<1, true>() ||
                           check_lifted<4, false>() || check_lifted<3, false>() || check_lifted<2, false>() || check_lifted<1, false>()))
            return 1;
    }
    printf("ok %ld\n", count);
    return 0;
}
