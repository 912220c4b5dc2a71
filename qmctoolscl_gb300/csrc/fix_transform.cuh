// fix_transform.cuh -- the passes of the FP64 transforms in block fixed point
// (fix64.cuh), included by transforms.cu.
//
// A pass takes groups of four index bits in registers: every thread holds 16 values
// whose indices differ in those four bits, runs the four stages on them, and the tile
// is re-dealt through shared memory (slots padded by one word per 16: no bank
// conflicts in any deal).  Two kinds of pass:
//   low   the lowest P = 9..12 index bits, a tile of 2^P consecutive values, 2^(P-4)
//         threads: three groups (bits 0-3, 4-7 and the window P-4..P-1);
//   high  the next S = 8 or 4 bits, 4096 / 2^S consecutive columns of 2^S strided
//         rows, 256 threads: two groups, or one that stays in registers.
// Exponents: a thread's 16 values have one of their own where their size asks for it (fix64.cuh), and the tile
// one in common where all blocks are alike, as random data's are.
// What bounds it: latency and the integer pipes together, with 14 warps of 16 per SM resident for complex data (issue 43-47 %,
// ALU 40-43 %, IMAD 46-56 %, stalls spread over waits, shared memory and the pipes), the ALU for real
// data (64 %, FP64 conversions 39-60 %); FFT of 32 x 2^20 in 0.55 + 0.56 ms, WHT of 300 x 2^16 in 89 + 60 us.  Sixteen complex values a thread (128 registers, 2 CTAs of 8 warps per SM) hold a
// radix-16 group: three exchanges for 12 bits where radix 4 in shared memory had six.
// Lengths below 2^9 keep the FP64 pass.  A tile that holds an inf or a nan, or blocks of values near the
// ends of the exponent range, is done by the FP64 stages.
#pragma once

#include "fix64.cuh"

namespace {

using fx::Cx;
using fx::i64;

constexpr int FIX_MIN_BITS = 9;  // shortest transform of the low pass

// Conversions: the idle FP64 unit takes all of those out and, of complex values, half of those
// in (whole registers, so without divergence).  32 vectors of 2^20, FFT: none on it 1180 us, all
// out 1155, and half in 1096, and all in 1106; 300 WHTs of 2^16: 166, 146, 155, 178.
template <int BITS>
__device__ __forceinline__ Cx take(Cx raw, int k, u32 E)
{
    const double r = as_double((u64)raw.r), i = as_double((u64)raw.i);
    return k < 8 ? Cx{fx::from_double_hw<BITS>(r, E), fx::from_double_hw<BITS>(i, E)}
                 : Cx{fx::from_double<BITS>(r, E), fx::from_double<BITS>(i, E)};
}

// exp(-2 pi i c j / 4096), j < 16, c < 256, and exp(-2 pi i c j / 256), j < 16, c < 16, as
// factors for cmul: [j][c].  Filled by every call's twiddle kernel ahead of its passes,
// always with the same values, so calls on other streams may fill them at the same time.
__device__ int4 fix_t12a[4096], fix_t8a[256];
__device__ int2 fix_t12b[4096], fix_t8b[256];

__device__ __forceinline__ void store_tw(int4 *pa, int2 *pb, double c, double d)
{
    const fx::Tw w = fx::make_tw(fx::factor62(c), fx::factor62(d));
    *pa = make_int4(w.c.hi, w.c.lo, w.s.hi, w.s.lo);
    *pb = make_int2(w.t.hi, w.t.lo);
}

__device__ __forceinline__ fx::Tw load_tw(const int4 *pa, const int2 *pb)
{
    const int4 u = *pa;
    const int2 v = *pb;
    fx::Tw w;
    w.c = fx::Halves{u.x, u.y};
    w.s = fx::Halves{u.z, u.w};
    w.t = fx::Halves{v.x, v.y};
    return w;
}

// entry t of the two tables, t < 4096 + 256
__device__ __forceinline__ void fill_fix_entry(u32 t)
{
    const bool big = t < 4096;
    const u32 i = big ? t : t - 4096;
    const u32 q = big ? ((i >> 8) * (i & 255u)) & 4095u : ((i >> 4) * (i & 15u)) & 255u;
    double sn, cs;
    sincospi((double)q * (big ? 1.0 / 2048 : 1.0 / 128), &sn, &cs);
    if (big)
        store_tw(&fix_t12a[i], &fix_t12b[i], cs, -sn);
    else
        store_tw(&fix_t8a[i], &fix_t8b[i], cs, -sn);
}

__device__ __forceinline__ u32 slot(u32 e) { return e + (e >> 4); }
constexpr u32 slots(u32 tile) { return tile + tile / 16; }

// A word per warp, combined by every thread after the next barrier.
template <int WARPS>
struct Warps {
    u32 w[WARPS];
};

template <int WARPS>
__device__ __forceinline__ void put_max(Warps<WARPS> &s, u32 v)
{
    v = __reduce_max_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31) == 0) s.w[threadIdx.x >> 5] = v;
}
template <int WARPS>
__device__ __forceinline__ u32 get_max(const Warps<WARPS> &s)
{
    u32 v = s.w[0];
#pragma unroll
    for (int i = 1; i < WARPS; i++) v = max(v, s.w[i]);
    return v;
}
template <int WARPS>
__device__ __forceinline__ void put_or(Warps<WARPS> &s, u32 v)
{
    v = __reduce_or_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31) == 0) s.w[threadIdx.x >> 5] = v;
}
template <int WARPS>
__device__ __forceinline__ u32 get_or(const Warps<WARPS> &s)
{
    u32 v = s.w[0];
#pragma unroll
    for (int i = 1; i < WARPS; i++) v |= s.w[i];
    return v;
}

__device__ __forceinline__ u32 mag_hi(i64 bits) { return (u32)((u64)bits >> 32) & 0x7FFFFFFFu; }
__device__ __forceinline__ u32 mag_hi(Cx bits) { return max(mag_hi(bits.r), mag_hi(bits.i)); }
__device__ __forceinline__ u64 nonzero(i64 bits) { return (u64)bits << 1; }
__device__ __forceinline__ u64 nonzero(Cx bits) { return nonzero(bits.r) | nonzero(bits.i); }

template <class V>
__device__ __forceinline__ u32 mag16(const V (&x)[16])
{
    u32 v = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) v = max(v, mag_hi(x[k]));
    return v;
}
template <class V>
__device__ __forceinline__ u32 spread16(const V (&x)[16])
{
    u32 acc = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) acc |= fx::spread(x[k]);
    return acc;
}

// ---- Exponents.  As long as every block of a tile has its largest value within NEAR bits of the tile's, the
// tile's threads have one exponent in common ("even"): data whose transform is alike in size stay
// there.  A thread that finds its block smaller, or lifts a class of it, takes exponents of its own ("odd"); from
// the next exchange on the tile's threads pass them along, a row of `exponent_row` words for each
// slot (group or class) of a source thread.  Five bits: a rounding beside the tile's largest value is then at most
// 2^-53 of the block's, a double's own.  FFT of 32 x 2^20 / WHT of 300 x 2^16, us: one exponent per tile, whatever the
// blocks, 1060 / 140; even tiles 1111 / 152 (the checks); a constant with a little noise 1399 / 203; exponents of their own
// throughout 1330 / 259; FP64 stages 4490 / 843.
constexpr int NEAR = 5;

__host__ __device__ constexpr u32 exponent_row(u32 T) { return T + 16; }  // rows half a line apart in the banks
template <u32 T, int SLOTS>
struct Exponents {
    int v[SLOTS][exponent_row(T)];
};

// slots of an inverse transform's group on NB bits: the classes of idft_regs and, below four bits, the
// independent groups (low register bits)
template <int NB>
__device__ __forceinline__ constexpr int idft_slot(int k)
{
    return NB == 4 ? k >> 2 : NB == 3 ? (k >> 2) * 2 + (k & 1) : k & ((1 << (4 - NB)) - 1);
}
template <int NB>
constexpr int idft_slots = NB == 1 || NB == 3 ? 8 : 4;

// whether values of largest biased exponent E, written back times 2^scale_exp, keep to fixed point
__device__ __forceinline__ bool fix_range(u32 E, int scale_exp)
{
    const int s = (int)E + scale_exp;
    return E >= fx::E_MIN && E <= fx::E_MAX && s >= (int)fx::E_MIN && s <= (int)fx::E_MAX;
}

// for the code of rare branches to be laid out of the way
__device__ __forceinline__ bool rare(bool v) { return __builtin_expect(v, 0); }

// What a thread knows of its tile's exponents.
struct State {
    bool even = true;  // the same for the tile's threads
    bool odd = false;  // this thread's differ
    bool bad = false;  // or cannot be: the tile is done in FP64
};

// Units are at least 2^low_exponent: results stay normal, their scale included.
__device__ __forceinline__ int low_exponent(const PassArgs &a) { return -1022 - min(a.scale_exp, 0); }

// bits that values of these exponents can be shifted up by
template <int G>
__device__ __forceinline__ int room(const int (&e)[G], int low)
{
    int v = e[0];
#pragma unroll
    for (int g = 1; g < G; g++) v = e[g] == fx::E_ZERO ? v : v == fx::E_ZERO ? e[g] : min(v, e[g]);
    return v - low;
}

// A thread's 16 places in a deal of the tile: `top` holds the tile's upper four bits in registers, `mid` bits 4-7,
// `low` bits 0-3.
template <class V>
struct Places;
template <>
struct Places<Cx> {
    i64 *sr, *si;
    u32 at, step;
    __device__ __forceinline__ Cx get(int k) const { return Cx{sr[at + k * step], si[at + k * step]}; }
    __device__ __forceinline__ void put(int k, Cx v) const
    {
        sr[at + k * step] = v.r;
        si[at + k * step] = v.i;
    }
};
template <>
struct Places<i64> {
    i64 *sr;
    u32 at, step;
    __device__ __forceinline__ i64 get(int k) const { return sr[at + k * step]; }
    __device__ __forceinline__ void put(int k, i64 v) const { sr[at + k * step] = v; }
};

template <int BITS>
__device__ __forceinline__ i64 take(i64 raw, int, u32 E) { return fx::from_double<BITS>(as_double((u64)raw), E); }

// The rare paths work on the thread's places, in calls with short loops: the registers and the instruction cache are left to
// the common ones (inline, the fused product of 100 x 2^16 took 740 us for 646).
// Doubles (as bits) to integers, one exponent per group, to out[g * blockDim.x]; true for values that have to
// stay in FP64.  A power of two that the results are multiplied by counts towards the range.
template <int BITS, int G, bool HIGH, class V>
__device__ __noinline__ bool enter_own(Places<V> at, int *out, int scale_exp)
{
    bool bad = false;
#pragma unroll 1
    for (int g = 0; g < G; g++) {
        u32 mx = 0;
        u64 any = 0;
#pragma unroll 1
        for (int i = 0; i < 16 / G; i++) {
            const V v = at.get(fx::member_of<G, HIGH>(g, i));
            mx = max(mx, mag_hi(v));
            any |= nonzero(v);
        }
        const u32 E = mx >> 20;
        const bool in = fix_range(E, scale_exp);
        bad = bad || (!in && any);
#pragma unroll 1
        for (int i = 0; i < 16 / G; i++) {
            const int k = fx::member_of<G, HIGH>(g, i);
            at.put(k, in ? take<BITS>(at.get(k), 8, E) : V{});
        }
        out[g * blockDim.x] = in ? (int)E - 1022 - BITS : fx::E_ZERO;
    }
    return bad;
}

// Values of exponents src(k) to one exponent per group.
template <int BITS, int G, bool HIGH, class V, class Src>
__device__ __noinline__ void align_own(Places<V> at, int *out, int low, Src src)
{
#pragma unroll 1
    for (int g = 0; g < G; g++) {
        const int e = fx::common_exponent(16 / G, BITS, low, [=](int i) { return at.get(fx::member_of<G, HIGH>(g, i)); },
                                          [=](int i) { return src(fx::member_of<G, HIGH>(g, i)); });
#pragma unroll 2
        for (int i = 0; i < 16 / G; i++) {
            const int k = fx::member_of<G, HIGH>(g, i);
            at.put(k, fx::shift_any(at.get(k), e - src(k)));
        }
        out[g * blockDim.x] = e;
    }
}

// The lift of a group's classes (fx::lift_of).
template <bool FWD>
__device__ __noinline__ void lift_own(Places<Cx> at, int *out, int room)
{
#pragma unroll 1
    for (int j = 1; j < 4; j++) {
        u64 mag = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) mag |= fx::mag64(at.get(FWD ? j + 4 * i : 4 * j + i));
        const int s = fx::lift_of(mag, room);
        out[j * blockDim.x] = s;
        if (s) {
#pragma unroll
            for (int i = 0; i < 4; i++) at.put(FWD ? j + 4 * i : 4 * j + i, fx::shift_any(at.get(FWD ? j + 4 * i : 4 * j + i), -s));
        }
    }
}

struct LiftOwn {
    State &st;
    Places<Cx> at;
    int *out, room;
    template <bool FWD>
    __device__ __forceinline__ void operator()(Cx (&x)[16], fx::Lifts &l) const
    {
        if (!rare(fx::may_lift<FWD>(x))) return;
#pragma unroll
        for (int k = 0; k < 16; k++) at.put(k, x[k]);
        lift_own<FWD>(at, out, room);
#pragma unroll
        for (int j = 1; j < 4; j++) l.s[j] = out[j * blockDim.x];
        st.odd |= (l.s[1] | l.s[2] | l.s[3]) != 0;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = at.get(k);
    }
};

// Values that are multiplied one by one after a group: those far below the others' size are shifted up, each by
// a count of its own, the thread's out[k * blockDim.x].
__device__ __noinline__ void lift_each_own(Places<Cx> at, int *out, int room)
{
#pragma unroll 1
    for (int k = 0; k < 16; k++) {
        const Cx v = at.get(k);
        const int b = fx::bits64(v), s = b ? max(min(62 - b, room), 0) : 0;
        at.put(k, fx::shift_any(v, -s));
        out[k * blockDim.x] = s;
    }
}

// an upper word of a block that is next to never far below its largest, with data alike in size
__device__ __forceinline__ u32 some_mag(const Cx (&x)[16])
{
    return max(max(max(mag_hi(x[0]), mag_hi(x[3])), max(mag_hi(x[5]), mag_hi(x[6]))), max(mag_hi(x[10]), mag_hi(x[13])));
}

// Doubles (as bits) to integers where the tile's largest upper word is `tile` and the thread's block has `mine`
// among its own; `at`: the places that its next exchange leaves the values in.
template <int BITS, int G, bool HIGH, class V>
__device__ __forceinline__ void enter(V (&x)[16], int (&e)[G], State &st, Places<V> at, int *out, u32 tile, u32 mine,
                                      int scale_exp)
{
    const u32 E = tile >> 20;
    if (!rare(!fix_range(E, scale_exp) || (mine >> 20) + NEAR < E)) {
#pragma unroll
        for (int g = 0; g < G; g++) e[g] = (int)E - 1022 - BITS;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = take<BITS>(x[k], k, E);
    } else {
#pragma unroll
        for (int k = 0; k < 16; k++) at.put(k, x[k]);
        st.bad |= enter_own<BITS, G, HIGH>(at, out, scale_exp);
        st.odd = true;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = at.get(k);
#pragma unroll
        for (int g = 0; g < G; g++) e[g] = out[g * blockDim.x];
    }
}

// The same for a block that is a tile of its own.
template <int BITS, class V>
__device__ __forceinline__ void enter_alone(V (&x)[16], int (&e)[1], State &st, Places<V> at, int *out, int scale_exp)
{
    const u32 mx = mag16(x);
    enter<BITS, 1, false>(x, e, st, at, out, mx, mx, scale_exp);
}

// whether none of eight words of a block reaches 2^bits: next to never in a block that does, with data alike in size.
__device__ __forceinline__ bool looks_small(const Places<Cx> &at, int bits)
{
    return !((fx::spread(at.get(0)) | fx::spread(at.get(3)) | fx::spread(at.get(6)) | fx::spread(at.get(13))) >> (bits - 32));
}
__device__ __forceinline__ bool looks_small(const Places<i64> &at, int bits)
{
    return !((fx::spread(at.get(0)) | fx::spread(at.get(3)) | fx::spread(at.get(5)) | fx::spread(at.get(6)) |
              fx::spread(at.get(9)) | fx::spread(at.get(10)) | fx::spread(at.get(12)) | fx::spread(at.get(15))) >> (bits - 32));
}

// Re-deal of the tile: every thread leaves its values where it last took them from and takes others, to
// one exponent per group: the tile's, or (src(k) the place of a value's exponent) their own.  False for every
// thread where one has found its values bad.
template <int BITS, int G, bool HIGH, int SLOTS, int WARPS, class V, class Src>
__device__ __forceinline__ bool redeal(V (&x)[16], int (&e)[G], const int (&own)[SLOTS], State &st, Warps<WARPS> &ws,
                                       u32 row, int *exps, int *out, int low, Places<V> from, Places<V> to, Src src)
{
    const int e0 = own[0];  // e and own may be the same
    if (st.even) put_or(ws, spread16(x));
#pragma unroll
    for (int k = 0; k < 16; k++) from.put(k, x[k]);
    bool alone = false;  // the thread's values are aligned on their own
    int right = 0;
    if (rare(!st.even || __syncthreads_or(st.odd || st.bad))) {
        st.even = false;
#pragma unroll
        for (int i = 0; i < SLOTS; i++) exps[i * row + threadIdx.x] = own[i];
        if (__syncthreads_or(st.bad)) return false;
        align_own<BITS, G, HIGH>(to, out, low, [=](int k) { return exps[src(k)]; });
        alone = true;
    } else {
        // a tile one bit below 2^BITS is left there
        const int s = fx::excess(get_or(ws), BITS);
        right = max(s, 0);
        alone = s < -1 || looks_small(to, BITS - NEAR + s);
        if (rare(alone)) {
            align_own<BITS, G, HIGH>(to, out, low, [=](int) { return e0; });
            st.odd = true;
        }
    }
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = to.get(k);
    if (right) {
        const u32 sh = alone ? 0u : (u32)right;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = fx::round_shift(x[k], sh);
    }
#pragma unroll
    for (int g = 0; g < G; g++) e[g] = e0 + right;
    if (rare(alone)) {
#pragma unroll
        for (int g = 0; g < G; g++) e[g] = out[g * blockDim.x];
    }
    return true;
}

// Values to doubles (as bits), x * 2^e, times sqrt(1/2) where `odd`: a product of its own, which rounds beside
// each value.
__device__ __forceinline__ i64 leave(i64 x, int e) { return (i64)as_bits(fx::to_double_hw(x, e)); }
__device__ __forceinline__ Cx leave(Cx x, int e) { return Cx{leave(x.r, e), leave(x.i, e)}; }
__device__ __forceinline__ i64 halve(i64 bits) { return (i64)as_bits(as_double((u64)bits) * 0.70710678118654752440); }
__device__ __forceinline__ Cx halve(Cx bits) { return Cx{halve(bits.r), halve(bits.i)}; }
template <class V>
__device__ __forceinline__ void leave16(V (&x)[16], const int (&e)[16], int scale_exp, bool odd)
{
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = leave(x[k], e[k] + scale_exp);
    if (rare(odd)) {
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = halve(x[k]);
    }
}

// The twiddles between two groups, w^(c j) / 4, are taken by the thread that has collected the values: rounding
// beside its own ones.  Forward, before the group on bits 4-7 of a tile (or of a high pass's rows): c the
// thread's, j the bit-reversed register index.  Inverse, before the group below it: the
// other way round (the table is symmetric).
template <bool CONJ>
__device__ __forceinline__ void twiddle_mid(Cx (&x)[16], u32 c)
{
    x[0] = fx::quarter(x[0]);
#pragma unroll
    for (int k = 1; k < 16; k++) {
        const int j = CONJ ? k : fx::bitrev<4>(k);
        x[k] = fx::cmul<CONJ, true>(x[k], load_tw(&fix_t8a[j * 16 + c], &fix_t8b[j * 16 + c]));
    }
}

// the twiddles below the low pass's top group of P - 8 stage bits: the register bits under them
// belong to the offset
template <int P>
__device__ __forceinline__ void twiddle_top(Cx (&x)[16], u32 t)
{
    constexpr int NB = P - 8;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const int j = fx::bitrev<NB>(k >> (4 - NB));
        if (j == 0) {
            x[k] = fx::quarter(x[k]);
            continue;
        }
        const u32 i = (u32)(j << (4 - NB)) * 256u + t + (u32)(k & ((1 << (4 - NB)) - 1)) * (1u << (P - 4));
        x[k] = fx::cmul<false, true>(x[k], load_tw(&fix_t12a[i], &fix_t12b[i]));
    }
}
template <int P>
__device__ __forceinline__ void untwiddle_top(Cx (&x)[16], u32 t)
{
    constexpr int NB = P - 8;
    const u32 i = ((__brev(t >> 4) >> (32 - NB)) << (4 - NB)) * 256u + (t & 15u);
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = fx::cmul<true, true>(x[k], load_tw(&fix_t12a[i + k * 16], &fix_t12b[i + k * 16]));
}

// Values that are multiplied one by one after a group: those that need 54 bits or less, where the others may take
// 62, are shifted up by eight, those that need 46 or less in a call by what they have.
__device__ __forceinline__ void lift_each(Cx (&x)[16], int (&e)[16], Places<Cx> at, int *out, int low)
{
    u32 all = 0xFFFFFFFFu;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const u32 m = fx::spread(x[k]);
        const int s = m >> 22 ? 0 : 8;
        x[k] = Cx{(i64)((u64)x[k].r << s), (i64)((u64)x[k].i << s)};
        e[k] -= s;
        all = min(all, m);
    }
    if (!rare(!(all >> 14))) return;
    int lo = e[0];
#pragma unroll
    for (int k = 0; k < 16; k++) {
        at.put(k, x[k]);
        lo = min(lo, e[k]);
    }
    lift_each_own(at, out, lo - low);
#pragma unroll
    for (int k = 0; k < 16; k++) {
        x[k] = at.get(k);
        e[k] -= out[k * 256];
    }
}

// A high pass's column twiddles w^(c br(row)), w = exp(-+2 pi i / 2^k1), c the column's offset
// below bit k0.  Eight row bits, row 16 q + k: br8 = 16 br4(k) + br4(q), a factor per thread
// (wa) and a table of 16 powers per column.
template <bool UNDO>
__device__ __forceinline__ void twiddle_columns(Cx (&x)[16], const fx::Tw &wa, const int4 *tba, const int2 *tbb,
                                                u32 col)
{
#pragma unroll
    for (int k = 0; k < 16; k++) {
        const int j = fx::bitrev<4>(k);
        x[k] = fx::cmul<UNDO, true>(x[k], wa);
        if (j) x[k] = fx::cmul<UNDO, false>(x[k], load_tw(&tba[j * 16 + col], &tbb[j * 16 + col]));
    }
}

// Four row bits: the powers 1, 2, 3 and then 4, 8, 12 of the column's w^c (24 products and six
// converted twiddles; 15 products would convert 15).  A quarter, as above.
template <bool CONJ, bool UNDO>
__device__ __forceinline__ void twiddle_powers(Cx (&x)[16], const PassArgs &a, u64 c, u32 sh)
{
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = fx::quarter(x[k]);  // j & 3 = 0: none of the first three
#pragma unroll
    for (int i = 1; i < 16; i = i < 3 ? i + 1 : (i == 3 ? 4 : i + 4)) {
        const u64 ip = (c * (u64)i) << sh;
        const fx::Tw w = fx::make_tw(fx::factor62(a.twr[ip]), fx::factor62(tw_im<CONJ>(a.twi[ip])));
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int j = fx::bitrev<4>(k);
            if (i < 4 ? (j & 3) == i : (j & 12) == i) x[k] = i < 4 ? fx::cmul<UNDO, true>(x[k], w) : fx::cmul<UNDO, false>(x[k], w);
        }
    }
}

// y * lam * f or y / lam * f (f = scale / n: the orthonormal factors of both transforms)
__device__ __forceinline__ void pointwise(const PassArgs &a, u64 gi, double &yr, double &yi)
{
    const u64 li = a.lam_all ? gi : (gi & ((1ull << a.m) - 1));
    const double lr = a.lr[li], lm = a.li[li], f = a.fix_lam_scale;
    if (f != 1.0) {
        yr *= f;
        yi *= f;
    }
    const double r = yr, i = yi;
    if (a.divide) {
        const double den = fma(lr, lr, lm * lm);
        yr = fma(r, lr, i * lm) / den;
        yi = fma(i, lr, -r * lm) / den;
    } else {
        yr = fma(r, lr, -i * lm);
        yi = fma(r, lm, i * lr);
    }
}

__device__ __forceinline__ double pointwise(const PassArgs &a, u64 gi, double y)
{
    const double l = a.lr[a.lam_all ? gi : (gi & ((1ull << a.m) - 1))], f = a.fix_lam_scale;
    if (f == 1.0) return a.divide ? y / l : y * l;
    return a.divide ? y * f / l : y * l * f;
}

// next tile's lines into L2 while this one is worked on
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

constexpr bool forward_kind(int kind) { return kind == FT_FFT || kind == FT_CONV; }
constexpr bool inverse_kind(int kind) { return kind == FT_IFFT || kind == FT_CONV; }

// ---- complex transforms, low pass: KIND FT_FFT, FT_IFFT or (n = 2^P) FT_CONV
template <int KIND, int P>
__global__ void __launch_bounds__(1 << (P - 4), P == 12 ? 2 : (P == 11 ? 4 : (P == 10 ? 8 : 16)))
    fix_low_kernel(PassArgs a)
{
    constexpr u32 T = 1u << (P - 4), TILE = 1u << P, ROW = exponent_row(T);
    constexpr int WARPS = (int)T / 32, NB = P - 8, G = 1 << (4 - NB), SLOTS = inverse_kind(KIND) ? idft_slots<NB> : 4;
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm, *si = sr + slots(TILE);
    __shared__ Warps<WARPS> ws[6];
    __shared__ Exponents<T, SLOTS> ex[2];
    __shared__ int eo[T < 64 ? 256 : 4 * T];  // what the rare paths return
    const u32 t = threadIdx.x;
    const Places<Cx> top{sr, si, slot(t), T + T / 16};
    const Places<Cx> mid{sr, si, (t & 15u) + 272u * (t >> 4), 17};
    const Places<Cx> low{sr, si, 17u * t, 1};
    const int lowest = low_exponent(a), lowest1 = KIND == FT_CONV ? -1022 : lowest;  // lowest1: of a fused pass's first half
    const u64 tiles = a.nvec << (a.m - P);
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const u64 base = tile << P;
        Cx x[16];
#pragma unroll
        for (int k = 0; k < 16; k++)
            x[k] = Cx{(i64)as_bits(a.xr[base + t + k * T]), (i64)as_bits(a.xi[base + t + k * T])};
        u32 mx = mag16(x);
        put_max(ws[0], mx);
        if (forward_kind(KIND)) {
#pragma unroll
            for (int k = 0; k < 16; k++) top.put(k, x[k]);
        }
        __syncthreads();
        const u64 next = tile + gridDim.x;
        if (next < tiles) {  // 16 values of 8 bytes a thread: one line of each array
            prefetch_l2(a.xr + (next << P) + t * 16);
            prefetch_l2(a.xi + (next << P) + t * 16);
        }
        State st;
        int e[1], et[G], own[16];  // et: the top group's exponents, own: those of the results
        if (forward_kind(KIND)) {
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = low.get(k);
            enter<fx::TOP, 1, false>(x, e, st, low, eo + t, get_max(ws[0]), some_mag(x), 0);
            fx::Lifts s = fx::dft_regs<4>(x, LiftOwn{st, low, eo + t, e[0] - lowest1});
            const int e1[4] = {e[0], e[0] - s.s[1], e[0] - s.s[2], e[0] - s.s[3]};
            if (!redeal<fx::TOP_TW, 1, false>(x, e, e1, st, ws[1], ROW, ex[0].v[0], eo + t, lowest1, low, mid,
                                              [=](int k) { return (t & 3u) * ROW + (t & ~15u) + k; })) {
                fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
                continue;
            }
            {
                twiddle_mid<false>(x, t & 15u);
                s = fx::dft_regs<4>(x, LiftOwn{st, mid, eo + t, e[0] + 2 - lowest1});
                const int e2[4] = {e[0] + 2, e[0] + 2 - s.s[1], e[0] + 2 - s.s[2], e[0] + 2 - s.s[3]};
                redeal<fx::TOP_TW, G, false>(x, et, e2, st, ws[2], ROW, ex[1].v[0], eo + t, lowest1, mid, top, [=](int k) {
                    return (((t >> 4) | (k * T / 16 & 15u)) & 3u) * ROW + ((k * T >> 8) << 4 | (t & 15u));
                });
                twiddle_top<P>(x, t);
                s = fx::dft_regs<NB>(x, LiftOwn{st, top, eo + t, room(et, lowest1)});
#pragma unroll
                for (int k = 0; k < 16; k++) own[k] = et[fx::group_of<G, false>(k)] + 2 - s.s[fx::dft_class<NB>(k)];
            }
        }
        if (KIND == FT_CONV) {
            leave16(x, own, 0, false);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                double yr = as_double((u64)x[k].r), yi = as_double((u64)x[k].i);
                pointwise(a, base + t + k * T, yr, yi);
                x[k] = Cx{(i64)as_bits(yr), (i64)as_bits(yi)};
            }
            mx = mag16(x);
            put_max(ws[3], mx);
            __syncthreads();
        }
        if (inverse_kind(KIND)) {
            st = State();
            enter<fx::TOP + 4 - NB, G, false>(x, et, st, top, eo + t, get_max(ws[KIND == FT_CONV ? 3 : 0]), mx, KIND == FT_CONV ? a.scale_exp : 0);
            fx::Lifts s = fx::idft_regs<NB>(x, LiftOwn{st, top, eo + t, room(et, lowest)});
            int e1[SLOTS];
#pragma unroll
            for (int k = 0; k < 16; k++) e1[idft_slot<NB>(k)] = et[fx::group_of<G, false>(k)] - s.s[fx::idft_class<NB>(k)];
            if (!redeal<fx::TOP_TW, 1, false>(x, e, e1, st, ws[4], ROW, ex[0].v[0], eo + t, lowest, top, mid, [=](int k) {
                return (u32)idft_slot<NB>((int)((t >> 4) * (256 / T)) + (k * 16 / (int)T)) * ROW + ((k * 16 + (t & 15u)) & (T - 1));
            })) {
                fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
                continue;
            }
            {
                untwiddle_top<P>(x, t);
                s = fx::idft_regs<4>(x, LiftOwn{st, mid, eo + t, e[0] + 2 - lowest});
                const int e2[4] = {e[0] + 2, e[0] + 2 - s.s[1], e[0] + 2 - s.s[2], e[0] + 2 - s.s[3]};
                redeal<fx::TOP_TW, 1, false>(x, e, e2, st, ws[5], ROW, ex[1].v[0], eo + t, lowest, mid, low,
                                             [=](int k) { return ((t & 15u) >> 2) * ROW + (t & ~15u) + k; });
                twiddle_mid<true>(x, __brev(t & 15u) >> 28);
                s = fx::idft_regs<4>(x, LiftOwn{st, low, eo + t, e[0] + 2 - lowest});
#pragma unroll
                for (int k = 0; k < 16; k++) own[k] = e[0] + 2 - s.s[fx::idft_class<4>(k)];
            }
        }
        leave16(x, own, a.scale_exp, a.scale_odd);
        if (inverse_kind(KIND)) {
#pragma unroll
            for (int k = 0; k < 16; k++) low.put(k, x[k]);
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = top.get(k);
        }
#pragma unroll
        for (int k = 0; k < 16; k++) {
            a.xr[base + t + k * T] = as_double((u64)x[k].r);
            a.xi[base + t + k * T] = as_double((u64)x[k].i);
        }
    }
}

// ---- complex transforms, high pass on bits k0 .. k0+S-1: KIND FT_FFT, FT_IFFT (CONJ: reading
// the forward table) or FT_CONV (the highest bits).  Four bits: a thread's block is a column of its own.
template <int KIND, bool CONJ, int S>
__global__ void __launch_bounds__(256, 2) fix_high_kernel(PassArgs a)
{
    constexpr u32 CT = 4096u >> S, ROW = exponent_row(256);
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm, *si = sr + slots(4096);
    __shared__ Warps<8> ws[4];
    __shared__ Exponents<256, S == 8 ? 4 : 1> ex[2];
    __shared__ int eo[inverse_kind(KIND) ? 16 * 256 : 4 * 256];  // what the rare paths return
    __shared__ int4 tba[256];
    __shared__ int2 tbb[256];
    const u32 t = threadIdx.x;
    const Places<Cx> top{sr, si, slot(t), 272};
    const Places<Cx> mid{sr, si, (t & 15u) + 272u * (t >> 4), 17};
    const int lowest = low_exponent(a), lowest1 = KIND == FT_CONV ? -1022 : lowest;  // lowest1: of a fused pass's first half
    const u64 chunks = (1ull << a.k0) / CT;
    const u64 tiles = (a.nvec << (a.m - a.k1)) * chunks;
    const u32 col = S == 8 ? (t & 15u) : t, q = S == 8 ? t >> 4 : 0u;
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const u64 c0 = (tile % chunks) * CT;
        const u64 base = ((tile / chunks) << a.k1) + c0;
        // rows of the first group (the lowest four row bits in registers) and of the last
        const u64 glow = base + col + (((u64)q * 16) << a.k0), gtop = base + col + ((u64)q << a.k0);
        const u64 slow = 1ull << a.k0, stop = 1ull << (a.k0 + (S == 8 ? 4 : 0));
        Cx x[16];
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const u64 gi = forward_kind(KIND) ? glow + k * slow : gtop + k * stop;
            x[k] = Cx{(i64)as_bits(a.xr[gi]), (i64)as_bits(a.xi[gi])};
        }
        u32 mx = mag16(x);
        const u64 c = c0 + col;
        const u32 sh = a.m - a.k1;
        fx::Tw wa;
        if (S == 8) {
            const u64 ia = (c * (__brev(q) >> 28)) << sh, ib = (c * q * 16) << sh;
            wa = fx::make_tw(fx::factor62(a.twr[ia]), fx::factor62(tw_im<CONJ>(a.twi[ia])));
            store_tw(&tba[q * 16 + col], &tbb[q * 16 + col], a.twr[ib], tw_im<CONJ>(a.twi[ib]));
            put_max(ws[0], mx);
            __syncthreads();
        }
        const u64 next = tile + gridDim.x;
        if (next < tiles) {
            const u64 nb = ((next / chunks) << a.k1) + (next % chunks) * CT +
                           (S == 8 ? (u64)t << a.k0 : ((u64)(t >> 4) << a.k0) + (t & 15u) * 16u);
            prefetch_l2(a.xr + nb);
            prefetch_l2(a.xi + nb);
        }
        constexpr int FIRST = forward_kind(KIND) ? fx::TOP_TW : fx::TOP;
        State st;
        int e[1], own[16];
        if (S == 8)
            enter<FIRST, 1, false>(x, e, st, forward_kind(KIND) ? mid : top, eo + t, get_max(ws[0]), mx, 0);
        else
            enter_alone<FIRST>(x, e, st, top, eo + t, 0);
        if (forward_kind(KIND)) {
            if (S == 8)
                twiddle_columns<false>(x, wa, tba, tbb, col);
            else
                twiddle_powers<CONJ, false>(x, a, c, sh);
            fx::Lifts s = fx::dft_regs<4>(x, LiftOwn{st, S == 8 ? mid : top, eo + t, e[0] + 2 - lowest1});
            if (S == 8) {
                const int e1[4] = {e[0] + 2, e[0] + 2 - s.s[1], e[0] + 2 - s.s[2], e[0] + 2 - s.s[3]};
                if (!redeal<fx::TOP_TW, 1, false>(x, e, e1, st, ws[1], ROW, ex[0].v[0], eo + t, lowest1, mid, top,
                                                  [=](int k) { return (q & 3u) * ROW + (k << 4 | (t & 15u)); })) {
                fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
                continue;
            }
                {
                    twiddle_mid<false>(x, q);
                    s = fx::dft_regs<4>(x, LiftOwn{st, top, eo + t, e[0] + 2 - lowest1});
                }
            }
#pragma unroll
            for (int k = 0; k < 16; k++) own[k] = e[0] + 2 - s.s[fx::dft_class<4>(k)];
        }
        if (KIND == FT_CONV) {
            leave16(x, own, 0, false);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                double yr = as_double((u64)x[k].r), yi = as_double((u64)x[k].i);
                pointwise(a, gtop + k * stop, yr, yi);
                x[k] = Cx{(i64)as_bits(yr), (i64)as_bits(yi)};
            }
            if (S == 8) {
                mx = mag16(x);
                put_max(ws[2], mx);
                __syncthreads();
                st = State();
                enter<fx::TOP, 1, false>(x, e, st, top, eo + t, get_max(ws[2]), mx, a.scale_exp);
            } else {
                enter_alone<fx::TOP>(x, e, st, top, eo + t, a.scale_exp);
            }
        }
        if (inverse_kind(KIND)) {
            // FT_CONV's inverse half undoes the same forward twiddles
            constexpr bool UNDO = KIND == FT_CONV;
            fx::Lifts s = fx::idft_regs<4>(x, LiftOwn{st, top, eo + t, e[0] - lowest});
            if (S == 8) {
                const int e1[4] = {e[0], e[0] - s.s[1], e[0] - s.s[2], e[0] - s.s[3]};
                if (!redeal<fx::TOP_TW, 1, false>(x, e, e1, st, ws[3], ROW, ex[1].v[0], eo + t, lowest, top, mid,
                                                  [=](int k) { return (q >> 2) * ROW + (k << 4 | (t & 15u)); })) {
                fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
                continue;
            }
                {
                    twiddle_mid<true>(x, __brev(q) >> 28);
                    e[0] += 2;
                    s = fx::idft_regs<4>(x, LiftOwn{st, mid, eo + t, e[0] - lowest});
                }
            }
#pragma unroll
            for (int k = 0; k < 16; k++) own[k] = e[0] + 2 - s.s[fx::idft_class<4>(k)];
            lift_each(x, own, S == 8 ? mid : top, eo + t, lowest);
            if (S == 8)
                twiddle_columns<UNDO>(x, wa, tba, tbb, col);
            else
                twiddle_powers<CONJ, UNDO>(x, a, c, sh);
        }
        if (S == 4 && rare(__syncthreads_or(st.bad))) {
            fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
            continue;
        }
        leave16(x, own, a.scale_exp, a.scale_odd);
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const u64 gi = inverse_kind(KIND) ? glow + k * slow : gtop + k * stop;
            a.xr[gi] = as_double((u64)x[k].r);
            a.xi[gi] = as_double((u64)x[k].i);
        }
        if (S == 8 && inverse_kind(KIND)) __syncthreads();  // all have read the table: the next tile's may be written
    }
}

// ---- Walsh-Hadamard transforms (the stages commute: the order of the groups is the one that
// loads and stores whole lines), low pass: KIND FT_FWHT or (n = 2^P) FT_WCONV
template <int KIND, int P>
__global__ void __launch_bounds__(1 << (P - 4), P == 12 ? 4 : (P == 11 ? 8 : (P == 10 ? 16 : 32)))
    fix_low_wht_kernel(PassArgs a)
{
    constexpr u32 T = 1u << (P - 4), TILE = 1u << P, ROW = exponent_row(T);
    constexpr int WARPS = (int)T / 32, G = 1 << (12 - P);  // groups of the middle deal: its upper register bits
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm;
    __shared__ Warps<WARPS> ws[6];
    __shared__ Exponents<T, KIND == FT_WCONV ? G : 1> ex[2];
    __shared__ int eo[256];  // what the rare paths return
    const u32 t = threadIdx.x;
    const Places<i64> top{sr, slot(t), T + T / 16};
    const Places<i64> mid{sr, (t & 15u) + 272u * (t >> 4), 17};
    const Places<i64> low{sr, 17u * t, 1};
    const int lowest = low_exponent(a), lowest1 = KIND == FT_WCONV ? -1022 : lowest;  // lowest1: of a fused pass's first half
    const u32 out = (t & 15u) + ((t >> 4) << 8);  // the middle deal's place in the tile, + 16 k
    const u64 tiles = a.nvec << (a.m - P);
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const u64 base = tile << P;
        i64 x[16];
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = (i64)as_bits(a.xr[base + t + k * T]);
        u32 mx = mag16(x);
        put_max(ws[0], mx);
        __syncthreads();
        const u64 next = tile + gridDim.x;
        if (next < tiles) prefetch_l2(a.xr + (next << P) + t * 16);
        State st;
        int e[1], eg[G], own[16];
        enter<fx::TOP, 1, false>(x, e, st, top, eo + t, get_max(ws[0]), mx, 0);
        fx::wht_regs<0, 4>(x);
        if (!redeal<fx::TOP, 1, false>(x, e, e, st, ws[1], ROW, ex[0].v[0], eo + t, lowest1, top, low,
                                       [=](int k) { return (16 * t + k) & (T - 1); })) {
                fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
                continue;
            }
        {
            fx::wht_regs<0, 4>(x);
            redeal<fx::TOP, G, true>(x, eg, e, st, ws[2], ROW, ex[1].v[0], eo + t, lowest1, low, mid,
                                     [=](int k) { return (t & ~15u) + k; });
            fx::wht_regs<0, P - 8>(x);
#pragma unroll
            for (int k = 0; k < 16; k++) own[k] = eg[fx::group_of<G, true>(k)];
        }
        if (KIND == FT_WCONV) {
            leave16(x, own, 0, false);
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = (i64)as_bits(pointwise(a, base + out + 16 * k, as_double((u64)x[k])));
            mx = mag16(x);
            put_max(ws[3], mx);
            __syncthreads();
            st = State();
            enter<fx::TOP, G, true>(x, eg, st, mid, eo + t, get_max(ws[3]), mx, a.scale_exp);
            fx::wht_regs<0, P - 8>(x);
            int e1[KIND == FT_WCONV ? G : 1];
#pragma unroll
            for (int g = 0; g < (KIND == FT_WCONV ? G : 1); g++) e1[g] = eg[g];
            if (!redeal<fx::TOP, 1, false>(x, e, e1, st, ws[4], ROW, ex[0].v[0], eo + t, lowest, mid, low,
                                           [=](int k) { return ((t & 15u) >> (P - 8)) * ROW + (t & ~15u) + k; })) {
                fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
                continue;
            }
            {
                fx::wht_regs<0, 4>(x);
                redeal<fx::TOP, 1, false>(x, e, e, st, ws[5], ROW, ex[1].v[0], eo + t, lowest, low, top,
                                          [=](int k) { return (t >> 4) + k * (T / 16); });
                fx::wht_regs<0, 4>(x);
#pragma unroll
                for (int k = 0; k < 16; k++) own[k] = e[0];
            }
        }
        leave16(x, own, a.scale_exp, a.scale_odd);
#pragma unroll
        for (int k = 0; k < 16; k++) a.xr[base + (KIND == FT_WCONV ? t + k * T : out + 16 * k)] = as_double((u64)x[k]);
    }
}

template <int KIND, int S>
__global__ void __launch_bounds__(256, 4) fix_high_wht_kernel(PassArgs a)
{
    constexpr u32 CT = 4096u >> S, ROW = exponent_row(256);
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm;
    __shared__ Warps<8> ws[4];
    __shared__ Exponents<256, 1> ex[2];
    __shared__ int eo[256];  // what the rare paths return
    const u32 t = threadIdx.x;
    const Places<i64> top{sr, slot(t), 272};
    const Places<i64> mid{sr, (t & 15u) + 272u * (t >> 4), 17};
    const int lowest = low_exponent(a), lowest1 = KIND == FT_WCONV ? -1022 : lowest;  // lowest1: of a fused pass's first half
    const u64 chunks = (1ull << a.k0) / CT;
    const u64 tiles = (a.nvec << (a.m - a.k1)) * chunks;
    const u32 col = S == 8 ? (t & 15u) : t, q = S == 8 ? t >> 4 : 0u;
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const u64 c0 = (tile % chunks) * CT;
        const u64 base = ((tile / chunks) << a.k1) + c0;
        const u64 glow = base + col + (((u64)q * 16) << a.k0), gtop = base + col + ((u64)q << a.k0);
        const u64 slow = 1ull << a.k0, stop = 1ull << (a.k0 + (S == 8 ? 4 : 0));
        i64 x[16];
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = (i64)as_bits(a.xr[glow + k * slow]);
        u32 mx = mag16(x);
        if (S == 8) {
            put_max(ws[0], mx);
            __syncthreads();
        }
        const u64 next = tile + gridDim.x;
        if (next < tiles)
            prefetch_l2(a.xr + ((next / chunks) << a.k1) + (next % chunks) * CT +
                        (S == 8 ? (u64)t << a.k0 : ((u64)(t >> 4) << a.k0) + (t & 15u) * 16u));
        State st;
        int e[1], own[16];
        if (S == 8)
            enter<fx::TOP, 1, false>(x, e, st, mid, eo + t, get_max(ws[0]), mx, 0);
        else
            enter_alone<fx::TOP>(x, e, st, mid, eo + t, 0);
        fx::wht_regs<0, 4>(x);
        if (S == 8) {
            if (!redeal<fx::TOP, 1, false>(x, e, e, st, ws[1], ROW, ex[0].v[0], eo + t, lowest1, mid, top,
                                           [=](int k) { return k << 4 | (t & 15u); })) {
                fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
                continue;
            }
            fx::wht_regs<0, 4>(x);
        }
#pragma unroll
        for (int k = 0; k < 16; k++) own[k] = e[0];
        if (KIND == FT_WCONV) {
            leave16(x, own, 0, false);
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = (i64)as_bits(pointwise(a, gtop + k * stop, as_double((u64)x[k])));
            if (S == 8) {
                mx = mag16(x);
                put_max(ws[2], mx);
                __syncthreads();
                st = State();
                enter<fx::TOP, 1, false>(x, e, st, top, eo + t, get_max(ws[2]), mx, a.scale_exp);
            } else {
                enter_alone<fx::TOP>(x, e, st, top, eo + t, a.scale_exp);
            }
            fx::wht_regs<0, 4>(x);
            if (S == 8) {
                if (!redeal<fx::TOP, 1, false>(x, e, e, st, ws[3], ROW, ex[1].v[0], eo + t, lowest, top, mid,
                                               [=](int k) { return k << 4 | (t & 15u); })) {
                fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
                continue;
            }
                fx::wht_regs<0, 4>(x);
            }
#pragma unroll
            for (int k = 0; k < 16; k++) own[k] = e[0];
        }
        if (S == 4 && rare(__syncthreads_or(st.bad))) {
            fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
            continue;
        }
        leave16(x, own, a.scale_exp, a.scale_odd);
#pragma unroll
        for (int k = 0; k < 16; k++)
            a.xr[KIND == FT_WCONV ? glow + k * slow : gtop + k * stop] = as_double((u64)x[k]);
    }
}

}  // namespace
