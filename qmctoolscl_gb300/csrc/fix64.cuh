// fix64.cuh -- block fixed-point arithmetic of the FP64 transforms.
//
// GB300's FP64 unit takes two operations per SM and clock, its integer pipes
// about 64, so the transforms hold their values as 64-bit integers, value = x * 2^e.  The 16
// values that a thread takes through a group of four stages share an exponent, at most 2^58 in
// modulus on the way in: five bits more than a double's 53 for the largest of them.  Each stage at most
// doubles a value, so that no sum overflows.  Adds are exact; a twiddle product (factors in units of
// 2^-62) is off by about half a unit.  Between groups every thread collects 16 values of other
// threads, and where they are far smaller than the tile's they take an exponent of their own
// (common_exponent): what the stages before cancelled keeps the bits that it has, as in floating point.
// One exponent per tile lost them beside the tile's largest sums (constant data plus 1e-12 of noise: the
// outputs but the first had 5 digits).
//
// Everything here compiles for the host too (the CPU test holds it to 128-bit
// integer arithmetic).
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#define FX_UNROLL _Pragma("unroll")
#define FX_UNROLL2 _Pragma("unroll 2")
#else
#define FX_HD inline
#define FX_UNROLL
#define FX_UNROLL2
#endif

namespace fx {

typedef long long i64;
typedef unsigned long long u64;
typedef unsigned int u32;

constexpr int TOP = 58;        // a group of stages starts below 2^TOP: 16 times that, times sqrt 2, fits
constexpr int TOP_TW = 60;     // twiddle products that give a quarter start below 2^TOP_TW
// Blocks of 16 whose largest biased exponent is outside [E_MIN, E_MAX] (tiny, huge, inf, nan),
// before or after the scale, send their tile to FP64.
constexpr u32 E_MIN = 200;
constexpr u32 E_MAX = 1800;
constexpr int E_ZERO = -4000;  // the exponent of a block of zeros

FX_HD i64 make(u32 hi, u32 lo) { return (i64)(((u64)hi << 32) | lo); }
FX_HD u32 hi32(i64 x) { return (u32)((u64)x >> 32); }
FX_HD u32 lo32(i64 x) { return (u32)(u64)x; }

FX_HD u32 clz32(u32 v)
{
#ifdef __CUDA_ARCH__
    return (u32)__clz((int)v);
#else
    return v ? (u32)__builtin_clz(v) : 32u;
#endif
}

FX_HD u64 bits_of(double v)
{
    u64 b;
    memcpy(&b, &v, 8);
    return b;
}

FX_HD double of_bits(u64 b)
{
    double v;
    memcpy(&v, &b, 8);
    return v;
}

// v in units of 2^(E - 1022 - BITS), rounded (ties away from zero): |result| <= 2^BITS for
// every v whose biased exponent is at most E
template <int BITS>
FX_HD i64 from_double(double v, u32 E)
{
    const u64 b = bits_of(v);
    const u32 h = (u32)(b >> 32);
    u32 d = E - ((h >> 20) & 0x7FFu);
    d = d < 62u ? d : 62u;
    u64 m = (((u64)((h & 0xFFFFFu) | 0x100000u) << 32) | (u32)b) << (BITS - 53);
    m = (m + ((1ull << d) >> 1)) >> d;
    const u64 s = (u64)((i64)b >> 63);
    return (i64)((m ^ s) - s);
}

// x * 2^e rounded to a double (ties away from zero), 64 <= e + 1023 and the result normal
FX_HD double to_double(i64 x, int e)
{
    const u32 s = hi32(x) & 0x80000000u;
    const u64 u = s ? 0ull - (u64)x : (u64)x;
    u32 h = (u32)(u >> 32), l = (u32)u;
    if (h == 0) {
        if (l == 0) return 0.0;
        h = l;
        l = 0;
        e -= 32;
    }
    const u32 lz = clz32(h);
    const u64 n = (((u64)h << 32) | l) << lz;  // leading one at bit 63
    const u64 m = (n >> 11) + (((u32)n >> 10) & 1u);
    return of_bits(m + ((u64)(s + ((u32)(1085 + e - (int)lz) << 20)) << 32));
}

#ifdef __CUDACC__
// The same two conversions on the FP64 unit (values whose exponent is more than 63 below the
// tile's largest go to 0 either way; doubles that are zero or subnormal too).
template <int BITS>
__device__ __forceinline__ i64 from_double_hw(double v, u32 E)
{
    const u32 h = (u32)__double2hiint(v);
    const u32 low = (E > 64u ? E - 64u : 1u) << 20;
    const double s = __hiloint2double((int)(h + (((u32)(1022 + BITS) - E) << 20)), __double2loint(v));
    return (h & 0x7FFFFFFFu) < low ? 0ll : __double2ll_rn(s);
}

__device__ __forceinline__ double to_double_hw(i64 x, int e)
{
    const double d = __ll2double_rn(x);
    const int h = __double2hiint(d);
    return __hiloint2double(x ? h + (e << 20) : h, __double2loint(d));
}
#endif

// bits that tell how many a value needs: |x| < 2^(32 + 32 - clz32(spread(x)))
FX_HD u32 spread(i64 x) { return hi32(x) ^ (u32)((int)hi32(x) >> 31); }

// the right shift that brings the largest of values whose spreads have the union `acc` to
// [2^(bits-1), 2^bits) (negative: a left shift)
FX_HD int excess(u32 acc, int bits) { return 64 - bits - (int)clz32(acc); }

// x * 2^-s, rounded (ties up), -32 < s < 32
FX_HD i64 shift_by(i64 x, int s) { return s > 0 ? (x + (1ll << (s - 1))) >> s : (i64)((u64)x << -s); }

// the same for 0 <= s < 32, without a branch
FX_HD i64 round_shift(i64 x, u32 s) { return (x + (i64)((1u << s) >> 1)) >> s; }

// the same for any s; 0 from s = 63 on
FX_HD i64 shift_any(i64 x, int s)
{
    if (s <= 0) return (i64)((u64)x << (s > -63 ? -s : 63));
    return s < 63 ? (x + (1ll << (s - 1))) >> s : 0;
}

FX_HD int bits_of_word(u64 u)  // of an unsigned number, 0 for 0
{
    const u32 h = (u32)(u >> 32), l = (u32)u;
    return h ? 64 - (int)clz32(h) : 32 - (int)clz32(l);
}

// a word of as many bits as |x| has (or |x| - 1, for negative x), 0 only for 0; for several values the union
FX_HD u64 mag64(i64 x) { return (u64)(x ^ (x >> 63)) | (u64)x >> 63; }

struct Cx {
    i64 r, i;
};

FX_HD u32 spread(Cx x) { return spread(x.r) | spread(x.i); }
FX_HD u64 mag64(Cx x) { return mag64(x.r) | mag64(x.i); }
// b >= 1 with |x| <= 2^b; 0 for 0
template <class T>
FX_HD int bits64(T x) { return bits_of_word(mag64(x)); }
FX_HD Cx round_shift(Cx x, u32 s) { return Cx{round_shift(x.r, s), round_shift(x.i, s)}; }
FX_HD Cx shift_any(Cx x, int s)
{
    if (s <= 0) return Cx{(i64)((u64)x.r << (s > -63 ? -s : 63)), (i64)((u64)x.i << (s > -63 ? -s : 63))};
    const u32 r = s < 63 ? (u32)s : 63u;
    const i64 half = (i64)((1ull << r) >> 1);
    return s < 63 ? Cx{(x.r + half) >> r, (x.i + half) >> r} : Cx{0, 0};
}

// Register k's group where 16 registers hold G groups, numbered by the high or the low bits of k.
template <int G, bool HIGH>
FX_HD constexpr int group_of(int k) { return HIGH ? k / (16 / G) : k % G; }
template <int G, bool HIGH>
FX_HD constexpr int member_of(int g, int i) { return HIGH ? g * (16 / G) + i : i * G + g; }

// The exponent that N values x(i) of exponents e(i) are brought to: the largest just below 2^bits, in units
// of 2^low at least; E_ZERO where all are 0.
template <class X, class E>
FX_HD int common_exponent(int n, int bits, int low, X x, E e)
{
    int top = E_ZERO;
    FX_UNROLL2
    for (int i = 0; i < n; i++) {
        const int b = bits64(x(i));
        top = b && b + e(i) > top ? b + e(i) : top;
    }
    return top == E_ZERO ? E_ZERO : top - bits > low ? top - bits : low;
}

// A 64-bit integer as hi * 2^32 + lo with both halves signed.
struct Halves {
    int hi, lo;
};

FX_HD Halves halves(i64 v)
{
    Halves r;
    r.lo = (int)lo32(v);
    r.hi = (int)(hi32(v) + (lo32(v) >> 31));
    return r;
}

// f * 2^62, |f| <= 1, truncated towards zero
FX_HD i64 factor62(double f)
{
    const u64 b = bits_of(f);
    const u32 h = (u32)(b >> 32);
    const u32 d = 1023u - ((h >> 20) & 0x7FFu);
    u64 m = (((u64)((h & 0xFFFFFu) | 0x100000u) << 32) | (u32)b) << 10;
    m = d < 64u ? m >> d : 0ull;
    const u64 s = (u64)((i64)b >> 63);
    return (i64)((m ^ s) - s);
}

// x * f for f = w * 2^-62, |f| <= 1:
// (x.hi*w.hi) * 4 + (x.hi*w.lo + x.lo*w.hi) * 2^-30 + (x.lo*w.lo * 2^-62, at most one unit,
// of either sign: dropped).
FX_HD i64 mul_real(i64 x, Halves w)
{
    const Halves v = halves(x);
    const i64 h = (i64)v.hi * w.hi;
    i64 m = (i64)v.hi * w.lo + (1 << 29);
    m = (i64)v.lo * w.hi + m;
    return (i64)((u64)h << 2) + (m >> 30);
}

// A complex factor c + i d, with t = d and s = -d: the conjugate swaps the two.
struct Tw {
    Halves c, s, t;
};

FX_HD Tw make_tw(i64 c, i64 d)
{
    Tw w;
    w.c = halves(c);
    w.s = halves(-d);
    w.t = halves(d);
    return w;
}

// x1*w1 + x2*w2, or a quarter of it (QUARTER): the products' sum needs no shift then, only the
// upper word of the middle terms.  Operands up to 2^62.5 in modulus fit.
template <bool QUARTER>
FX_HD i64 dot(Halves x1, Halves w1, Halves x2, Halves w2)
{
    i64 m = (i64)x1.hi * w1.lo + (QUARTER ? 1ll << 31 : 1ll << 29);
    m = (i64)x1.lo * w1.hi + m;
    m = (i64)x2.hi * w2.lo + m;
    m = (i64)x2.lo * w2.hi + m;
    if (QUARTER) {
        const i64 h = (i64)x1.hi * w1.hi + (i64)(int)hi32(m);
        return (i64)x2.hi * w2.hi + h;
    }
    i64 h = (i64)x1.hi * w1.hi;
    h = (i64)x2.hi * w2.hi + h;
    return (i64)((u64)h << 2) + (m >> 30);
}

template <bool CONJ, bool QUARTER>
FX_HD Cx cmul(Cx x, const Tw &w)
{
    const Halves s = CONJ ? w.t : w.s, t = CONJ ? w.s : w.t;
    const Halves r = halves(x.r), i = halves(x.i);
    return Cx{dot<QUARTER>(r, w.c, i, s), dot<QUARTER>(r, t, i, w.c)};
}

// a quarter of x, for the values of a group whose factor is 1
FX_HD Cx quarter(Cx x) { return Cx{(x.r + 2) >> 2, (x.i + 2) >> 2}; }

// ------------------------------------------------ groups of stages in registers

// cos(pi/8), sin(pi/8) and sqrt(1/2), times 2^62
constexpr i64 COS8 = 0x3b20d79e651a8c51ll, SIN8 = 0x187de2a6aea962d2ll, HALF = 0x2d413cccfe779921ll;

// x times exp(-2 pi i K / 16) (CONJ: the conjugate), K = 1, 2, 3, 4, 6 or 9
template <int K, bool CONJ>
FX_HD Cx rot16(Cx x)
{
    if (K == 1) return cmul<CONJ, false>(x, make_tw(COS8, -SIN8));
    if (K == 3) return cmul<CONJ, false>(x, make_tw(SIN8, -COS8));
    if (K == 9) return cmul<CONJ, false>(x, make_tw(-COS8, SIN8));
    Cx y;
    if (K == 4) {  // -i (i)
        y.r = CONJ ? -x.i : x.i;
        y.i = CONJ ? x.r : -x.r;
        return y;
    }
    const Halves h = halves(HALF);
    if (K == 2) {  // (1 - i) / sqrt 2
        y.r = mul_real(CONJ ? x.r - x.i : x.r + x.i, h);
        y.i = mul_real(CONJ ? x.r + x.i : x.i - x.r, h);
    } else {  // K = 6: (-1 - i) / sqrt 2
        y.r = mul_real(CONJ ? -(x.r + x.i) : x.i - x.r, h);
        y.i = mul_real(CONJ ? x.r - x.i : -(x.r + x.i), h);
    }
    return y;
}

// 4-point DFT of a bit-reversed group (two decimation-in-time stages)
FX_HD void dft4(Cx &x0, Cx &x1, Cx &x2, Cx &x3)
{
    const Cx a{x0.r + x1.r, x0.i + x1.i}, b{x0.r - x1.r, x0.i - x1.i};
    const Cx c{x2.r + x3.r, x2.i + x3.i}, d{x2.r - x3.r, x2.i - x3.i};
    x0 = Cx{a.r + c.r, a.i + c.i};
    x2 = Cx{a.r - c.r, a.i - c.i};
    x1 = Cx{b.r + d.i, b.i - d.r};  // b - i d
    x3 = Cx{b.r - d.i, b.i + d.r};
}

// its inverse, bit-reversed output (two decimation-in-frequency stages)
FX_HD void idft4(Cx &x0, Cx &x1, Cx &x2, Cx &x3)
{
    const Cx a{x0.r + x2.r, x0.i + x2.i}, c{x0.r - x2.r, x0.i - x2.i};
    const Cx b{x1.r + x3.r, x1.i + x3.i}, d{x1.r - x3.r, x1.i - x3.i};
    x0 = Cx{a.r + b.r, a.i + b.i};
    x1 = Cx{a.r - b.r, a.i - b.i};
    x2 = Cx{c.r - d.i, c.i + d.r};  // c + i d
    x3 = Cx{c.r + d.i, c.i - d.r};
}

FX_HD void dft2(Cx &x0, Cx &x1)
{
    const Cx a = x0;
    x0 = Cx{a.r + x1.r, a.i + x1.i};
    x1 = Cx{a.r - x1.r, a.i - x1.i};
}

// Between its two halves a group's values fall into classes that do not mix again: the values of a class
// that the first half's adds have left small are shifted up, so that the rotations round beside
// them and not beside the group's largest.  Lifts has the shift of each class.
struct Lifts {
    int s[4];
};

// What a transform does between its halves, operator()<forward>(values, shifts): nothing, for blocks alike.
struct NoLift {
    template <bool FWD>
    FX_HD void operator()(Cx (&)[16], Lifts &) const
    {
    }
};

// Whether a class (registers k & 3 forward, k >> 2 inverse; class 0 takes no rotation) may need a lift: three
// of its four values are looked at, of which with data whose outputs are alike in size one is large
// enough but in one thread of a million.
template <bool FWD>
FX_HD bool may_lift(const Cx (&x)[16])
{
    bool small = false;
    FX_UNROLL
    for (int j = 1; j < 4; j++)
        small = small || !((FWD ? spread(x[j]) | spread(x[j + 4]) | spread(x[j + 8])
                                : spread(x[4 * j]) | spread(x[4 * j + 1]) | spread(x[4 * j + 2])) >> 21);
    return small;
}

// The shift that brings four values of magnitudes `mag` to below 2^60 (rotations and two more stages fit), where
// that is seven bits and more, `room` at most.
FX_HD int lift_of(u64 mag, int room)
{
    if (mag >> 53 || !mag) return 0;
    int s = 60 - bits_of_word(mag);
    s = s < room ? s : room;
    return s > 0 ? s : 0;
}

// The class of register k of a forward / inverse transform on NB bits.
template <int NB>
FX_HD constexpr int dft_class(int k) { return NB >= 3 ? k & 3 : 0; }
template <int NB>
FX_HD constexpr int idft_class(int k) { return NB >= 3 ? k >> 2 : 0; }

// The stages on the upper NB bits of a 4-bit register index (the lower 4 - NB bits
// number independent groups): forward, input bit-reversed.
template <int NB, class L>
FX_HD Lifts dft_regs(Cx (&x)[16], L lift)
{
    Lifts s{{0, 0, 0, 0}};
    if (NB == 1) {
        FX_UNROLL
        for (int k = 0; k < 8; k++) dft2(x[k], x[k + 8]);
    }
    if (NB == 4) {
        FX_UNROLL
        for (int k = 0; k < 16; k += 4) dft4(x[k], x[k + 1], x[k + 2], x[k + 3]);
        lift.template operator()<true>(x, s);
        x[5] = rot16<2, false>(x[5]);
        x[9] = rot16<1, false>(x[9]);
        x[13] = rot16<3, false>(x[13]);
        x[7] = rot16<6, false>(x[7]);
        x[11] = rot16<3, false>(x[11]);
        x[15] = rot16<9, false>(x[15]);
    }
    if (NB == 3) {
        FX_UNROLL
        for (int k = 0; k < 16; k += 4) {
            dft2(x[k], x[k + 2]);
            dft2(x[k + 1], x[k + 3]);
        }
        lift.template operator()<true>(x, s);
        x[7] = rot16<4, false>(x[7]);
        x[11] = rot16<2, false>(x[11]);
        x[15] = rot16<6, false>(x[15]);
    }
    if (NB >= 3) {
        x[6] = rot16<4, false>(x[6]);
        x[10] = rot16<2, false>(x[10]);
        x[14] = rot16<6, false>(x[14]);
    }
    if (NB >= 2) {
        FX_UNROLL
        for (int g = 0; g < 4; g++) dft4(x[g], x[g + 4], x[g + 8], x[g + 12]);
    }
    return s;
}
template <int NB>
FX_HD void dft_regs(Cx (&x)[16]) { dft_regs<NB>(x, NoLift{}); }

// the inverse, output bit-reversed
template <int NB, class L>
FX_HD Lifts idft_regs(Cx (&x)[16], L lift)
{
    Lifts s{{0, 0, 0, 0}};
    if (NB == 1) {
        FX_UNROLL
        for (int k = 0; k < 8; k++) dft2(x[k], x[k + 8]);
    }
    if (NB >= 2) {
        FX_UNROLL
        for (int g = 0; g < 4; g++) idft4(x[g], x[g + 4], x[g + 8], x[g + 12]);
    }
    if (NB >= 3) {
        lift.template operator()<false>(x, s);
        x[6] = rot16<4, true>(x[6]);
        x[10] = rot16<2, true>(x[10]);
        x[14] = rot16<6, true>(x[14]);
    }
    if (NB == 3) {
        x[7] = rot16<4, true>(x[7]);
        x[11] = rot16<2, true>(x[11]);
        x[15] = rot16<6, true>(x[15]);
        FX_UNROLL
        for (int k = 0; k < 16; k += 4) {
            dft2(x[k], x[k + 2]);
            dft2(x[k + 1], x[k + 3]);
        }
    }
    if (NB == 4) {
        x[5] = rot16<2, true>(x[5]);
        x[9] = rot16<1, true>(x[9]);
        x[13] = rot16<3, true>(x[13]);
        x[7] = rot16<6, true>(x[7]);
        x[11] = rot16<3, true>(x[11]);
        x[15] = rot16<9, true>(x[15]);
        FX_UNROLL
        for (int k = 0; k < 16; k += 4) idft4(x[k], x[k + 1], x[k + 2], x[k + 3]);
    }
    return s;
}
template <int NB>
FX_HD void idft_regs(Cx (&x)[16]) { idft_regs<NB>(x, NoLift{}); }

// Walsh-Hadamard stages on register bits LO .. HI-1
template <int LO, int HI>
FX_HD void wht_regs(i64 (&x)[16])
{
    FX_UNROLL
    for (int b = LO; b < HI; b++)
        FX_UNROLL
        for (int k = 0; k < 16; k++)
            if (!(k >> b & 1)) {
                const i64 u = x[k], v = x[k + (1 << b)];
                x[k] = u + v;
                x[k + (1 << b)] = u - v;
            }
}

// bit reversal of an NB-bit number
template <int NB>
FX_HD constexpr int bitrev(int v)
{
    int r = 0;
    FX_UNROLL
    for (int b = 0; b < NB; b++) r |= (v >> b & 1) << (NB - 1 - b);
    return r;
}

}  // namespace fx
