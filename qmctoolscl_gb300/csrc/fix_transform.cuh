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
// What bounds it: the ALU pipe (55-75 % busy over the pass, IMAD 20 %, HBM 24-50 %) and the
// barriers between the groups' phases; FFT of 32 x 2^20 in 0.53 + 0.52 ms, WHT of 300 x 2^16 in 73 +
// 71 us.  Sixteen complex values a thread (128 registers, 2 CTAs of 8 warps per SM) hold a
// radix-16 group: three exchanges for 12 bits where radix 4 in shared memory had six.
// Lengths below 2^9 keep the FP64 pass.  A tile that holds zeros only, an inf or a nan,
// or values near the ends of the exponent range is done by the FP64 stages.
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

// Deals of a tile over the threads: the place of register k's value.
struct DealTop {  // the tile's upper four bits in registers (T threads)
    u32 at, step;
    __device__ DealTop(u32 t, u32 T) : at(slot(t)), step(T + T / 16) {}
    __device__ u32 operator()(int k) const { return at + k * step; }
};
struct DealMid {  // bits 4-7
    u32 at;
    __device__ DealMid(u32 t) : at((t & 15u) + 272u * (t >> 4)) {}
    __device__ u32 operator()(int k) const { return at + k * 17; }
};
struct DealLow {  // bits 0-3
    u32 at;
    __device__ DealLow(u32 t) : at(17u * t) {}
    __device__ u32 operator()(int k) const { return at + k; }
};

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

__device__ __forceinline__ u32 mag_hi(double v) { return (u32)(as_bits(v) >> 32) & 0x7FFFFFFFu; }

__device__ __forceinline__ u32 spread16(const Cx (&x)[16])
{
    u32 acc = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) acc |= fx::spread(x[k].r) | fx::spread(x[k].i);
    return acc;
}
__device__ __forceinline__ u32 spread16(const i64 (&x)[16])
{
    u32 acc = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) acc |= fx::spread(x[k]);
    return acc;
}

// Re-deal of the tile from one deal to another: every thread leaves its values where it
// last took them from and takes others, with the tile's largest brought to 2^BITS.
template <int BITS, int WARPS, class From, class To>
__device__ __forceinline__ void redeal(Cx (&x)[16], int &e, i64 *sr, i64 *si, Warps<WARPS> &ws, From from, To to)
{
    put_or(ws, spread16(x));
#pragma unroll
    for (int k = 0; k < 16; k++) {
        sr[from(k)] = x[k].r;
        si[from(k)] = x[k].i;
    }
    __syncthreads();
    const int s = fx::excess(get_or(ws), BITS);
    e += s;
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = Cx{sr[to(k)], si[to(k)]};
    if (s > 0) {
        const i64 half = 1ll << (s - 1);
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = Cx{(x[k].r + half) >> s, (x[k].i + half) >> s};
    } else if (s < 0) {
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = Cx{fx::shift_by(x[k].r, s), fx::shift_by(x[k].i, s)};
    }
}

template <int BITS, int WARPS, class From, class To>
__device__ __forceinline__ void redeal(i64 (&x)[16], int &e, i64 *sr, Warps<WARPS> &ws, From from, To to)
{
    put_or(ws, spread16(x));
#pragma unroll
    for (int k = 0; k < 16; k++) sr[from(k)] = x[k];
    __syncthreads();
    const int s = fx::excess(get_or(ws), BITS);
    e += max(s, 0);
#pragma unroll
    for (int k = 0; k < 16; k++) x[k] = sr[to(k)];
    if (s > 0) {
        const i64 half = 1ll << (s - 1);
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = (x[k] + half) >> s;
    }
}

// the twiddles of the group on bits 4-7 of a tile (or of a high pass's rows): w^(c j) / 4, j
// the bit-reversed register index
template <bool CONJ>
__device__ __forceinline__ void twiddle_mid(Cx (&x)[16], u32 c)
{
    x[0] = fx::quarter(x[0]);
#pragma unroll
    for (int k = 1; k < 16; k++) {
        const int j = fx::bitrev<4>(k);
        x[k] = fx::cmul<CONJ, true>(x[k], load_tw(&fix_t8a[j * 16 + c], &fix_t8b[j * 16 + c]));
    }
}

// the twiddles of the low pass's top group: P - 8 stage bits above the register bits that
// still belong to the offset
template <int P, bool CONJ>
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
        x[k] = fx::cmul<CONJ, true>(x[k], load_tw(&fix_t12a[i], &fix_t12b[i]));
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

// values -> doubles: value * 2^e (times sqrt(1/2) for an odd number of stages in all)
template <class T>
__device__ __forceinline__ void halve_odd(T &x, bool odd)
{
    if (odd) x = fx::mul_real(x, fx::halves(fx::HALF));
}

// whether a tile of largest biased exponent E, written back times 2^scale_exp, keeps to fixed point
__device__ __forceinline__ bool fix_range(u32 E, int scale_exp)
{
    const int s = (int)E + scale_exp;
    return E >= fx::E_MIN && E <= fx::E_MAX && s >= (int)fx::E_MIN && s <= (int)fx::E_MAX;
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
    constexpr u32 T = 1u << (P - 4), TILE = 1u << P;
    constexpr int WARPS = (int)T / 32, NB = P - 8;
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm, *si = sr + slots(TILE);
    __shared__ Warps<WARPS> ws[6];
    const u32 t = threadIdx.x;
    const DealTop top(t, T);
    const DealMid mid(t);
    const DealLow low(t);
    const u64 tiles = a.nvec << (a.m - P);
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const u64 base = tile << P;
        Cx x[16];
        u32 mx = 0;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const double vr = a.xr[base + t + k * T], vi = a.xi[base + t + k * T];
            mx = max(mx, max(mag_hi(vr), mag_hi(vi)));
            x[k] = Cx{(i64)as_bits(vr), (i64)as_bits(vi)};
        }
        put_max(ws[0], mx);
        if (forward_kind(KIND)) {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                sr[top(k)] = x[k].r;
                si[top(k)] = x[k].i;
            }
        }
        __syncthreads();
        const u64 next = tile + gridDim.x;
        if (next < tiles) {  // 16 values of 8 bytes a thread: one line of each array
            prefetch_l2(a.xr + (next << P) + t * 16);
            prefetch_l2(a.xi + (next << P) + t * 16);
        }
        u32 E = get_max(ws[0]) >> 20;
        if (!fix_range(E, 0)) {
            fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
            continue;
        }
        if (forward_kind(KIND)) {
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = Cx{sr[low(k)], si[low(k)]};
        }
        int e = (int)E - 1022 - fx::TOP;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = take<fx::TOP>(x[k], k, E);
        if (forward_kind(KIND)) {
            fx::dft_regs<4>(x);
            redeal<fx::TOP_TW>(x, e, sr, si, ws[1], low, mid);
            twiddle_mid<false>(x, t & 15u);
            e += 2;
            fx::dft_regs<4>(x);
            redeal<fx::TOP_TW>(x, e, sr, si, ws[2], mid, top);
            twiddle_top<P, false>(x, t);
            e += 2;
            fx::dft_regs<NB>(x);
        }
        if (KIND == FT_CONV) {
            u32 m2 = 0;
#pragma unroll
            for (int k = 0; k < 16; k++) {
                double yr = fx::to_double_hw(x[k].r, e), yi = fx::to_double_hw(x[k].i, e);
                pointwise(a, base + t + k * T, yr, yi);
                m2 = max(m2, max(mag_hi(yr), mag_hi(yi)));
                x[k] = Cx{(i64)as_bits(yr), (i64)as_bits(yi)};
            }
            put_max(ws[3], m2);
            __syncthreads();
            E = get_max(ws[3]) >> 20;
            if (!fix_range(E, a.scale_exp)) {
                fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
                continue;
            }
            e = (int)E - 1022 - fx::TOP;
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = take<fx::TOP>(x[k], k, E);
        }
        if (inverse_kind(KIND)) {
            fx::idft_regs<NB>(x);
            twiddle_top<P, true>(x, t);
            e += 2;
            redeal<fx::TOP>(x, e, sr, si, ws[4], top, mid);
            fx::idft_regs<4>(x);
            twiddle_mid<true>(x, t & 15u);
            e += 2;
            redeal<fx::TOP>(x, e, sr, si, ws[5], mid, low);
            fx::idft_regs<4>(x);
        }
        e += a.scale_exp;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            halve_odd(x[k].r, a.scale_odd);
            halve_odd(x[k].i, a.scale_odd);
            x[k] = Cx{(i64)as_bits(fx::to_double_hw(x[k].r, e)), (i64)as_bits(fx::to_double_hw(x[k].i, e))};
        }
        if (inverse_kind(KIND)) {
#pragma unroll
            for (int k = 0; k < 16; k++) {
                sr[low(k)] = x[k].r;
                si[low(k)] = x[k].i;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = Cx{sr[top(k)], si[top(k)]};
        }
#pragma unroll
        for (int k = 0; k < 16; k++) {
            a.xr[base + t + k * T] = as_double((u64)x[k].r);
            a.xi[base + t + k * T] = as_double((u64)x[k].i);
        }
    }
}

// ---- complex transforms, high pass on bits k0 .. k0+S-1: KIND FT_FFT, FT_IFFT (CONJ: reading
// the forward table) or FT_CONV (the highest bits)
template <int KIND, bool CONJ, int S>
__global__ void __launch_bounds__(256, 2) fix_high_kernel(PassArgs a)
{
    constexpr u32 CT = 4096u >> S;
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm, *si = sr + slots(4096);
    __shared__ Warps<8> ws[4];
    __shared__ int4 tba[256];
    __shared__ int2 tbb[256];
    const u32 t = threadIdx.x;
    const DealTop top(t, 256);
    const DealMid mid(t);
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
        u32 mx = 0;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const u64 gi = forward_kind(KIND) ? glow + k * slow : gtop + k * stop;
            const double vr = a.xr[gi], vi = a.xi[gi];
            mx = max(mx, max(mag_hi(vr), mag_hi(vi)));
            x[k] = Cx{(i64)as_bits(vr), (i64)as_bits(vi)};
        }
        const u64 c = c0 + col;
        const u32 sh = a.m - a.k1;
        fx::Tw wa;
        if (S == 8) {
            const u64 ia = (c * (__brev(q) >> 28)) << sh, ib = (c * q * 16) << sh;
            wa = fx::make_tw(fx::factor62(a.twr[ia]), fx::factor62(tw_im<CONJ>(a.twi[ia])));
            store_tw(&tba[q * 16 + col], &tbb[q * 16 + col], a.twr[ib], tw_im<CONJ>(a.twi[ib]));
            put_max(ws[0], mx);
            __syncthreads();
            mx = get_max(ws[0]);
        }
        const u64 next = tile + gridDim.x;
        if (next < tiles) {
            const u64 nb = ((next / chunks) << a.k1) + (next % chunks) * CT +
                           (S == 8 ? (u64)t << a.k0 : ((u64)(t >> 4) << a.k0) + (t & 15u) * 16u);
            prefetch_l2(a.xr + nb);
            prefetch_l2(a.xi + nb);
        }
        u32 E = mx >> 20;
        bool bad = !fix_range(E, 0);
        if (S == 4) bad = __syncthreads_or(bad);
        if (bad) {
            fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
            continue;
        }
        constexpr int FIRST = forward_kind(KIND) ? fx::TOP_TW : fx::TOP;
        int e = (int)E - 1022 - FIRST;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = take<FIRST>(x[k], k, E);
        if (forward_kind(KIND)) {
            if (S == 8)
                twiddle_columns<false>(x, wa, tba, tbb, col);
            else
                twiddle_powers<CONJ, false>(x, a, c, sh);
            e += 2;
            fx::dft_regs<4>(x);
            if (S == 8) {
                redeal<fx::TOP_TW>(x, e, sr, si, ws[1], mid, top);
                twiddle_mid<false>(x, q);
                e += 2;
                fx::dft_regs<4>(x);
            }
        }
        if (KIND == FT_CONV) {
            u32 m2 = 0;
#pragma unroll
            for (int k = 0; k < 16; k++) {
                double yr = fx::to_double_hw(x[k].r, e), yi = fx::to_double_hw(x[k].i, e);
                pointwise(a, gtop + k * stop, yr, yi);
                m2 = max(m2, max(mag_hi(yr), mag_hi(yi)));
                x[k] = Cx{(i64)as_bits(yr), (i64)as_bits(yi)};
            }
            if (S == 8) {
                put_max(ws[2], m2);
                __syncthreads();
                m2 = get_max(ws[2]);
            }
            E = m2 >> 20;
            bad = !fix_range(E, a.scale_exp);
            if (S == 4) bad = __syncthreads_or(bad);
            if (bad) {
                fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
                continue;
            }
            e = (int)E - 1022 - fx::TOP;
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = take<fx::TOP>(x[k], k, E);
        }
        if (inverse_kind(KIND)) {
            // FT_CONV's inverse half undoes the same forward twiddles
            constexpr bool UNDO = KIND == FT_CONV;
            fx::idft_regs<4>(x);
            if (S == 8) {
                twiddle_mid<true>(x, q);
                e += 2;
                redeal<fx::TOP>(x, e, sr, si, ws[3], top, mid);
                fx::idft_regs<4>(x);
            }
            if (S == 8)
                twiddle_columns<UNDO>(x, wa, tba, tbb, col);
            else
                twiddle_powers<CONJ, UNDO>(x, a, c, sh);
            e += 2;
        }
        e += a.scale_exp;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            halve_odd(x[k].r, a.scale_odd);
            halve_odd(x[k].i, a.scale_odd);
            const u64 gi = inverse_kind(KIND) ? glow + k * slow : gtop + k * stop;
            a.xr[gi] = fx::to_double_hw(x[k].r, e);
            a.xi[gi] = fx::to_double_hw(x[k].i, e);
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
    constexpr u32 T = 1u << (P - 4), TILE = 1u << P;
    constexpr int WARPS = (int)T / 32;
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm;
    __shared__ Warps<WARPS> ws[6];
    const u32 t = threadIdx.x;
    const DealTop top(t, T);
    const DealMid mid(t);
    const DealLow low(t);
    const u32 out = (t & 15u) + ((t >> 4) << 8);  // the middle deal's place in the tile, + 16 k
    const u64 tiles = a.nvec << (a.m - P);
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const u64 base = tile << P;
        i64 x[16];
        u32 mx = 0;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const double v = a.xr[base + t + k * T];
            mx = max(mx, mag_hi(v));
            x[k] = (i64)as_bits(v);
        }
        put_max(ws[0], mx);
        __syncthreads();
        const u64 next = tile + gridDim.x;
        if (next < tiles) prefetch_l2(a.xr + (next << P) + t * 16);
        u32 E = get_max(ws[0]) >> 20;
        if (!fix_range(E, 0)) {
            fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
            continue;
        }
        int e = (int)E - 1022 - fx::TOP;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = fx::from_double<fx::TOP>(as_double((u64)x[k]), E);
        fx::wht_regs<0, 4>(x);
        redeal<fx::TOP>(x, e, sr, ws[1], top, low);
        fx::wht_regs<0, 4>(x);
        redeal<fx::TOP>(x, e, sr, ws[2], low, mid);
        fx::wht_regs<0, P - 8>(x);
        if (KIND == FT_WCONV) {
            u32 m2 = 0;
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const double y = pointwise(a, base + out + 16 * k, fx::to_double_hw(x[k], e));
                m2 = max(m2, mag_hi(y));
                x[k] = (i64)as_bits(y);
            }
            put_max(ws[3], m2);
            __syncthreads();
            E = get_max(ws[3]) >> 20;
            if (!fix_range(E, a.scale_exp)) {
                fp64_tile<KIND>(a, sm, base, 0, 0, 1, TILE);
                continue;
            }
            e = (int)E - 1022 - fx::TOP;
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = fx::from_double<fx::TOP>(as_double((u64)x[k]), E);
            fx::wht_regs<0, P - 8>(x);
            redeal<fx::TOP>(x, e, sr, ws[4], mid, low);
            fx::wht_regs<0, 4>(x);
            redeal<fx::TOP>(x, e, sr, ws[5], low, top);
            fx::wht_regs<0, 4>(x);
        }
        e += a.scale_exp;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            halve_odd(x[k], a.scale_odd);
            a.xr[base + (KIND == FT_WCONV ? t + k * T : out + 16 * k)] = fx::to_double_hw(x[k], e);
        }
    }
}

template <int KIND, int S>
__global__ void __launch_bounds__(256, 4) fix_high_wht_kernel(PassArgs a)
{
    constexpr u32 CT = 4096u >> S;
    extern __shared__ double sm[];
    i64 *sr = (i64 *)sm;
    __shared__ Warps<8> ws[4];
    const u32 t = threadIdx.x;
    const DealTop top(t, 256);
    const DealMid mid(t);
    const u64 chunks = (1ull << a.k0) / CT;
    const u64 tiles = (a.nvec << (a.m - a.k1)) * chunks;
    const u32 col = S == 8 ? (t & 15u) : t, q = S == 8 ? t >> 4 : 0u;
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const u64 c0 = (tile % chunks) * CT;
        const u64 base = ((tile / chunks) << a.k1) + c0;
        const u64 glow = base + col + (((u64)q * 16) << a.k0), gtop = base + col + ((u64)q << a.k0);
        const u64 slow = 1ull << a.k0, stop = 1ull << (a.k0 + (S == 8 ? 4 : 0));
        i64 x[16];
        u32 mx = 0;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const double v = a.xr[glow + k * slow];
            mx = max(mx, mag_hi(v));
            x[k] = (i64)as_bits(v);
        }
        if (S == 8) {
            put_max(ws[0], mx);
            __syncthreads();
            mx = get_max(ws[0]);
        }
        const u64 next = tile + gridDim.x;
        if (next < tiles)
            prefetch_l2(a.xr + ((next / chunks) << a.k1) + (next % chunks) * CT +
                        (S == 8 ? (u64)t << a.k0 : ((u64)(t >> 4) << a.k0) + (t & 15u) * 16u));
        u32 E = mx >> 20;
        bool bad = !fix_range(E, 0);
        if (S == 4) bad = __syncthreads_or(bad);
        if (bad) {
            fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
            continue;
        }
        int e = (int)E - 1022 - fx::TOP;
#pragma unroll
        for (int k = 0; k < 16; k++) x[k] = fx::from_double<fx::TOP>(as_double((u64)x[k]), E);
        fx::wht_regs<0, 4>(x);
        if (S == 8) {
            redeal<fx::TOP>(x, e, sr, ws[1], mid, top);
            fx::wht_regs<0, 4>(x);
        }
        if (KIND == FT_WCONV) {
            u32 m2 = 0;
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const double y = pointwise(a, gtop + k * stop, fx::to_double_hw(x[k], e));
                m2 = max(m2, mag_hi(y));
                x[k] = (i64)as_bits(y);
            }
            if (S == 8) {
                put_max(ws[2], m2);
                __syncthreads();
                m2 = get_max(ws[2]);
            }
            E = m2 >> 20;
            bad = !fix_range(E, a.scale_exp);
            if (S == 4) bad = __syncthreads_or(bad);
            if (bad) {
                fp64_tile<KIND>(a, sm, base, tile / chunks, c0, CT, 4096);
                continue;
            }
            e = (int)E - 1022 - fx::TOP;
#pragma unroll
            for (int k = 0; k < 16; k++) x[k] = fx::from_double<fx::TOP>(as_double((u64)x[k]), E);
            fx::wht_regs<0, 4>(x);
            if (S == 8) {
                redeal<fx::TOP>(x, e, sr, ws[3], top, mid);
                fx::wht_regs<0, 4>(x);
            }
        }
        e += a.scale_exp;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            halve_odd(x[k], a.scale_odd);
            a.xr[KIND == FT_WCONV ? glow + k * slow : gtop + k * stop] = fx::to_double_hw(x[k], e);
        }
    }
}

}  // namespace
