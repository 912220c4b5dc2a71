// transforms.cu -- FP64 radix-2 FFT (bit-reversed input, natural output),
// its inverse (natural input, bit-reversed output) and the Walsh-Hadamard
// transform, all orthonormal and in place along the last axis.
//
// Reference: qmctoolscl/c_funcs/fft_bro_1d_radix2.c:3-80 (decimation in
// time: stage k pairs i1, i1+2^k with twiddle tw[(i1 mod 2^k) * 2^(m-k-1)],
// tw[t] = exp(-2 pi i t/n)), ifft_bro_1d_radix2.c:3-81 (decimation in
// frequency: stage k pairs at distance 2^s, s = m-k-1, twiddle
// tw[(i1 mod 2^s) * 2^k] with the opposite sign), fwht_1d_radix2.c:3-53.
// Every stage of the reference divides by sqrt(2); here the stages are
// unscaled, run two at a time as radix-4 steps (three complex twiddle
// products per four values instead of four, half the shared-memory round
// trips), and the last pass multiplies by 2^(-m/2) once.  The results agree
// with the reference to FP64 rounding (not bit for bit).
//
// Passes.  Stages whose butterflies span the index bits [k0, k1) act on
// independent groups {h*2^k1 + q*2^k0 + c : q < 2^(k1-k0)}; a CTA loads one
// group for CT consecutive c (CT contiguous doubles per q, so loads and
// stores are coalesced runs), runs those stages in shared memory, and
// writes the tile back in place.  Up to 4096 complex (8192 real) values fit
// a tile, so lengths up to 2^12 (2^13 real) take one pass, up to 2^20 two,
// and so on.  The FFT runs the low-bit pass first, the inverse the high-bit
// pass first, matching the order of their stages.
//
// GB300 runs FP64 at about 1.25 TFLOP/s, so these FP64 stages (ft_pass_kernel) are bound by the
// FP64 unit.  From 2^9 values on the passes of fix_transform.cuh take their place: the same
// transform in 64-bit block fixed point on the integer and IMAD pipes, an exponent for every 16 values that
// go through four stages together.  Errors against long double, n = 2^9..2^16: 0.2-0.9 of the FP64
// stages' in L2 on normal, lognormal, smooth and nearly constant data and kernel columns, and no larger
// output by output (median and 90th percentile of |error| / |output|).  What is left of the block: a value
// that is 2^5 and more below another of its 16 keeps 58 bits below that one's size, which shows where the large ones
// cancel exactly and the small ones do not.  Device time, FP64 stages -> fixed point: FFT of
// 32 x 2^20 4490 -> 1111 us, IFFT of 111 x 2^10 17.2 -> 15.2, WHT of 300 x 2^16 843 -> 152.
// The tensor-core path (tc_fft.cu) is faster still at 1e-7, but for the WHT.
#include <cmath>

#include "common.cuh"

namespace {

constexpr int FT_THREADS = 256;
constexpr u32 TILE_COMPLEX = 4096;
constexpr u32 TILE_REAL = 8192;

enum FtKind { FT_FFT = 0, FT_IFFT = 1, FT_FWHT = 2, FT_CONV = 3, FT_WCONV = 4 };

__device__ void fill_fix_entry(u32 t);

// twiddles of an n-point transform, then (more = 4096 + 256) the tables of the fixed-point passes.
// From n = 8 on a thread takes one angle of the first eighth turn and writes its eight mirror
// images, an eighth of the FP64 work by the symmetry of the two functions: n = 2^20: 73 -> 15 us.
__global__ void twiddle_kernel(u64 n, double sign, double *twr, double *twi, u32 more)
{
    const u64 count = n >= 8 ? n / 8 + 1 : n;
    for (u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x; t < count + more; t += (u64)gridDim.x * blockDim.x) {
        if (t >= count) {
            fill_fix_entry((u32)(t - count));
            continue;
        }
        double sn, cs;
        // the angle 2*pi*t/n as a multiple of pi is exact for n a power of two
        sincospi(__ddiv_rn(__ull2double_rn(2 * t), __ull2double_rn(n)), &sn, &cs);
        if (n < 8) {
            twr[t] = cs;
            twi[t] = sign * sn;
            continue;
        }
        const u64 q = n / 4;
        if (8 * t == n) sn = cs;  // its own mirror image (sincospi's sine is a unit off there, its cosine is not)
        double c = cs, s = sn;  // of the angle t + k n / 4
#pragma unroll
        for (int k = 0; k < 4; k++) {
            twr[t + k * q] = c;
            twi[t + k * q] = sign * s;
            // the mirror image about the middle of the quarter: (k + 1) n / 4 - t
            const double mc = k & 1 ? -cs : sn, ms = k & 1 ? sn : cs;
            const u64 i = (k + 1) * q - t;
            if (t > 0 && t < n / 8) {
                twr[i] = k & 2 ? -mc : mc;
                twi[i] = sign * (k & 2 ? -ms : ms);
            }
            const double nc = 0.0 - s;  // turn by a quarter (a zero stays +0)
            s = c;
            c = nc;
        }
    }
}

struct PassArgs {
    u64 nvec;        // d1*d2 vectors
    u32 m;           // log2 n
    u32 k0, k1;      // index bits spanned by this pass
    u32 ct;          // consecutive c values per tile
    double *xr, *xi;
    const double *twr, *twi;
    double scale;    // applied on write-back when != 1
    // the fused forms: lam (lr, li; li unused for real data), n values shared by
    // the vectors (lam_all = 0) or one per element (lam_all = 1)
    const double *lr, *li;
    u32 lam_all, divide;
    double lam_scale;
    // the fixed-point passes: the write-back scale as 2^scale_exp (times sqrt(1/2)), and what of
    // lam_scale that leaves to the pointwise step; conj: the inverse steps read the forward
    // transform's table
    int scale_exp;
    double fix_lam_scale;
    bool scale_odd, conj;
};

// the imaginary part of a twiddle; conjugated when the inverse steps read the
// forward transform's table (the fused forms fill only that one)
template <bool CONJ>
__device__ __forceinline__ double tw_im(double v) { return CONJ ? -v : v; }

// The stages of one pass on a tile in shared memory (CT consecutive c per q):
// KIND's butterflies over the index bits [a.k0, a.k1) of group h, columns
// c0 .. c0+ct-1.
template <int KIND, bool CONJ>
__device__ __forceinline__ void ft_stages(const PassArgs &a, double *sr, double *si, u64 h, u64 c0, u32 ct,
                                          u32 tile_elems, u32 nt)
{
    const u32 nb = tile_elems / 2;
    const u32 nbits = a.k1 - a.k0;
    // stages in pairs (radix-4 steps), a single radix-2 stage for an odd bit count: the FFT
    // and WHT go up from bit k0 (the odd stage last), the inverse down from k1-1 (the odd
    // stage last as well, at bit k0)
    for (u32 done = 0; done < nbits;) {
        const u32 w = (nbits - done >= 2) ? 2u : 1u;
        const u32 bit = (KIND == FT_IFFT) ? (a.k1 - done - w) : (a.k0 + done);  // lowest bit of the step
        const u32 hb = bit - a.k0;
        done += w;
        if (w == 2) {
            const u32 S = (1u << hb) * ct;  // member stride in the tile
            // at bit 0 every twiddle is 1: the same step without the products (a separate loop,
            // so the FP64 multiplies are skipped rather than predicated off)
            if (KIND != FT_FWHT && bit == 0) {
                for (u32 b = threadIdx.x; b < tile_elems / 4; b += nt) {
                    const u32 p = b / ct, cc = b % ct;
                    const u32 e0 = (p << 2) * ct + cc, e1 = e0 + S, e2 = e1 + S, e3 = e2 + S;
                    const double x0r = sr[e0], x0i = si[e0], x1r = sr[e1], x1i = si[e1];
                    const double x2r = sr[e2], x2i = si[e2], x3r = sr[e3], x3i = si[e3];
                    if (KIND == FT_FFT) {
                        const double ar = x0r + x1r, ai = x0i + x1i, br = x0r - x1r, bi = x0i - x1i;
                        const double cr = x2r + x3r, ci = x2i + x3i, dr = x2r - x3r, di = x2i - x3i;
                        sr[e0] = ar + cr;
                        si[e0] = ai + ci;
                        sr[e2] = ar - cr;
                        si[e2] = ai - ci;
                        sr[e1] = br + di;
                        si[e1] = bi - dr;
                        sr[e3] = br - di;
                        si[e3] = bi + dr;
                    } else {
                        const double ar = x0r + x2r, ai = x0i + x2i, cr = x0r - x2r, ci = x0i - x2i;
                        const double br = x1r + x3r, bi = x1i + x3i, dr = x1r - x3r, di = x1i - x3i;
                        sr[e0] = ar + br;
                        si[e0] = ai + bi;
                        sr[e1] = ar - br;
                        si[e1] = ai - bi;
                        sr[e2] = cr - di;
                        si[e2] = ci + dr;
                        sr[e3] = cr + di;
                        si[e3] = ci - dr;
                    }
                }
                __syncthreads();
                continue;
            }
            for (u32 b = threadIdx.x; b < tile_elems / 4; b += nt) {
                const u32 p = b / ct, cc = b % ct;
                const u32 q0 = ((p >> hb) << (hb + 2)) | (p & ((1u << hb) - 1));
                const u32 e0 = q0 * ct + cc, e1 = e0 + S, e2 = e1 + S, e3 = e2 + S;
                if (KIND == FT_FWHT) {
                    const double x0 = sr[e0], x1 = sr[e1], x2 = sr[e2], x3 = sr[e3];
                    const double u0 = x0 + x1, u1 = x0 - x1, u2 = x2 + x3, u3 = x2 - x3;
                    sr[e0] = u0 + u2;
                    sr[e2] = u0 - u2;
                    sr[e1] = u1 + u3;
                    sr[e3] = u1 - u3;
                    continue;
                }
                // the group's offset below bit `bit`; w = tw[c * n / 2^(bit+2)] and its powers
                const u64 i0 = (h << a.k1) + ((u64)q0 << a.k0) + c0 + cc;
                const u64 c = i0 & ((1ull << bit) - 1);
                const u32 sh = a.m - bit - 2;
                const double w1r = a.twr[c << sh], w1i = tw_im<CONJ>(a.twi[c << sh]);
                const double w2r = a.twr[c << (sh + 1)], w2i = tw_im<CONJ>(a.twi[c << (sh + 1)]);
                const double w3r = a.twr[(3 * c) << sh], w3i = tw_im<CONJ>(a.twi[(3 * c) << sh]);
                const double x0r = sr[e0], x0i = si[e0], x1r = sr[e1], x1i = si[e1];
                const double x2r = sr[e2], x2i = si[e2], x3r = sr[e3], x3i = si[e3];
                if (KIND == FT_FFT) {
                    // two decimation-in-time stages: pre-twiddles w^br(p) (br: 0, 2, 1, 3) and the
                    // 4-point DFT of the bit-reversed group
                    const double y1r = fma(x1r, w2r, -x1i * w2i), y1i = fma(x1r, w2i, x1i * w2r);
                    const double y2r = fma(x2r, w1r, -x2i * w1i), y2i = fma(x2r, w1i, x2i * w1r);
                    const double y3r = fma(x3r, w3r, -x3i * w3i), y3i = fma(x3r, w3i, x3i * w3r);
                    const double ar = x0r + y1r, ai = x0i + y1i, br = x0r - y1r, bi = x0i - y1i;
                    const double cr = y2r + y3r, ci = y2i + y3i, dr = y2r - y3r, di = y2i - y3i;
                    sr[e0] = ar + cr;
                    si[e0] = ai + ci;
                    sr[e2] = ar - cr;
                    si[e2] = ai - ci;
                    sr[e1] = br + di;  // (x0 - x1) - i (x2 - x3)
                    si[e1] = bi - dr;
                    sr[e3] = br - di;  // (x0 - x1) + i (x2 - x3)
                    si[e3] = bi + dr;
                } else {
                    // two decimation-in-frequency stages (bits bit+1, then bit): the inverse
                    // 4-point DFT and post-twiddles v^(0, 2, 1, 3) (v = the + sign twiddle)
                    const double ar = x0r + x2r, ai = x0i + x2i, cr = x0r - x2r, ci = x0i - x2i;
                    const double br = x1r + x3r, bi = x1i + x3i, dr = x1r - x3r, di = x1i - x3i;
                    sr[e0] = ar + br;
                    si[e0] = ai + bi;
                    const double z1r = ar - br, z1i = ai - bi;
                    sr[e1] = fma(z1r, w2r, -z1i * w2i);
                    si[e1] = fma(z1r, w2i, z1i * w2r);
                    const double z2r = cr - di, z2i = ci + dr;  // (x0 - x2) + i (x1 - x3)
                    sr[e2] = fma(z2r, w1r, -z2i * w1i);
                    si[e2] = fma(z2r, w1i, z2i * w1r);
                    const double z3r = cr + di, z3i = ci - dr;  // (x0 - x2) - i (x1 - x3)
                    sr[e3] = fma(z3r, w3r, -z3i * w3i);
                    si[e3] = fma(z3r, w3i, z3i * w3r);
                }
            }
            __syncthreads();
            continue;
        }
        const u32 half = 1u << hb;
        for (u32 b = threadIdx.x; b < nb; b += nt) {
            const u32 p = b / ct, cc = b % ct;
            const u32 q1 = ((p >> hb) << (hb + 1)) | (p & (half - 1));
            const u32 e1 = q1 * ct + cc, e2 = e1 + half * ct;
            if (KIND == FT_FWHT) {
                const double x1 = sr[e1], x2 = sr[e2];
                sr[e1] = x1 + x2;
                sr[e2] = x1 - x2;
                continue;
            }
            // global index of the upper partner, for the twiddle
            const u64 i1 = (h << a.k1) + ((u64)q1 << a.k0) + c0 + cc;
            const u64 t = (i1 & ((1ull << bit) - 1)) << (a.m - bit - 1);
            const double wr = a.twr[t], wi = tw_im<CONJ>(a.twi[t]);
            const double ar = sr[e1], ai = si[e1], br = sr[e2], bi = si[e2];
            if (KIND == FT_FFT) {
                const double yr = fma(br, wr, -bi * wi), yi = fma(br, wi, bi * wr);
                sr[e1] = ar + yr;
                si[e1] = ai + yi;
                sr[e2] = ar - yr;
                si[e2] = ai - yi;
            } else {
                const double dr = ar - br, di = ai - bi;
                sr[e1] = ar + br;
                si[e1] = ai + bi;
                sr[e2] = fma(dr, wr, -di * wi);
                si[e2] = fma(dr, wi, di * wr);
            }
        }
        __syncthreads();
    }
}

// The stages of one pass on a tile in shared memory and, for the fused forms, the pointwise step
// between the forward and the inverse ones: y <- y * lam * f or y / lam * f (f = scale / n: the
// orthonormal factors of both transforms), lam n values shared by the vectors or one per element.
template <int KIND, bool CONJ>
__device__ __forceinline__ void ft_tile(const PassArgs &a, double *sr, double *si, u64 base, u64 h, u64 c0, u32 ct,
                                        u32 tile_elems, u32 nt)
{
    constexpr bool REAL = KIND == FT_FWHT || KIND == FT_WCONV;
    const u64 n = 1ull << a.m;
    if constexpr (KIND == FT_CONV || KIND == FT_WCONV) {
        ft_stages<KIND == FT_CONV ? (int)FT_FFT : (int)FT_FWHT, false>(a, sr, si, h, c0, ct, tile_elems, nt);
        const double f = a.lam_scale;
        for (u32 e = threadIdx.x; e < tile_elems; e += nt) {
            const u32 q = e / ct, cc = e % ct;
            const u64 gi = base + ((u64)q << a.k0) + cc;
            const u64 li = a.lam_all ? gi : (gi & (n - 1));
            const double lr = a.lr[li];
            if (REAL) {
                sr[e] = a.divide ? sr[e] * f / lr : sr[e] * lr * f;
            } else {
                const double lm = a.li[li], yr = sr[e] * f, yi = si[e] * f;
                if (a.divide) {
                    const double den = fma(lr, lr, lm * lm);
                    sr[e] = fma(yr, lr, yi * lm) / den;
                    si[e] = fma(yi, lr, -yr * lm) / den;
                } else {
                    sr[e] = fma(yr, lr, -yi * lm);
                    si[e] = fma(yr, lm, yi * lr);
                }
            }
        }
        __syncthreads();
        ft_stages<KIND == FT_CONV ? (int)FT_IFFT : (int)FT_FWHT, KIND == FT_CONV>(a, sr, si, h, c0, ct, tile_elems,
                                                                                 nt);
    } else {
        ft_stages<KIND, CONJ>(a, sr, si, h, c0, ct, tile_elems, nt);
    }
}

// One pass of a transform on tiles of the data.  KIND: FT_FFT, FT_IFFT
// (CONJ: reading the forward table), FT_FWHT, or the fused forms of the
// highest-bit pass: FT_CONV (forward FFT steps, the pointwise product or
// quotient by lam, inverse FFT steps) and FT_WCONV (WHT steps, pointwise,
// WHT steps).
template <int KIND, bool CONJ>
__global__ void __launch_bounds__(FT_THREADS) ft_pass_kernel(PassArgs a)
{
    constexpr bool REAL = KIND == FT_FWHT || KIND == FT_WCONV;
    extern __shared__ double sm[];
    const u32 Q = 1u << (a.k1 - a.k0);
    const u32 ct = a.ct;
    const u32 tile_elems = Q * ct;
    double *sr = sm;
    double *si = sm + tile_elems;  // unused for real data
    const u64 n = 1ull << a.m;
    const u64 H = n >> a.k1;                 // groups along the high bits
    const u64 cchunks = (1ull << a.k0) / ct;  // c chunks along the low bits
    const u64 tiles_per_vec = H * cchunks;
    const u64 total_tiles = a.nvec * tiles_per_vec;
    for (u64 tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
        const u64 v = tile / tiles_per_vec, rem = tile % tiles_per_vec;
        const u64 h = rem / cchunks, c0 = (rem % cchunks) * ct;
        const u64 base = v * n + (h << a.k1) + c0;
        for (u32 e = threadIdx.x; e < tile_elems; e += FT_THREADS) {
            const u32 q = e / ct, cc = e % ct;
            const u64 gi = base + ((u64)q << a.k0) + cc;
            sr[e] = a.xr[gi];
            if (!REAL) si[e] = a.xi[gi];
        }
        __syncthreads();
        ft_tile<KIND, CONJ>(a, sr, si, base, h, c0, ct, tile_elems, FT_THREADS);
        const double sc = a.scale;
        for (u32 e = threadIdx.x; e < tile_elems; e += FT_THREADS) {
            const u32 q = e / ct, cc = e % ct;
            const u64 gi = base + ((u64)q << a.k0) + cc;
            a.xr[gi] = sc != 1.0 ? sr[e] * sc : sr[e];
            if (!REAL) a.xi[gi] = sc != 1.0 ? si[e] * sc : si[e];
        }
        __syncthreads();
    }
}

// One tile of a fixed-point pass in FP64 (tiles that hold inf, nan or a block of values near the
// ends of the exponent range): starts from and ends with the data in global memory, and with
// a barrier.
template <int KIND>
__device__ __noinline__ void fp64_tile(const PassArgs &a, double *sm, u64 base, u64 h, u64 c0, u32 ct, u32 tile_elems)
{
    constexpr bool REAL = KIND == FT_FWHT || KIND == FT_WCONV;
    double *sr = sm, *si = sm + tile_elems;
    const u32 nt = blockDim.x;
    for (u32 e = threadIdx.x; e < tile_elems; e += nt) {
        const u64 gi = base + ((u64)(e / ct) << a.k0) + e % ct;
        sr[e] = a.xr[gi];
        if (!REAL) si[e] = a.xi[gi];
    }
    __syncthreads();
    if (KIND == FT_IFFT && a.conj)
        ft_tile<KIND, true>(a, sr, si, base, h, c0, ct, tile_elems, nt);
    else
        ft_tile<KIND, false>(a, sr, si, base, h, c0, ct, tile_elems, nt);
    for (u32 e = threadIdx.x; e < tile_elems; e += nt) {
        const u64 gi = base + ((u64)(e / ct) << a.k0) + e % ct;
        a.xr[gi] = sr[e] * a.scale;
        if (!REAL) a.xi[gi] = si[e] * a.scale;
    }
    __syncthreads();
}

}  // namespace

#include "fix_transform.cuh"

namespace {

struct Pass {
    u32 k0, k1, ct;
};

// Bit ranges covered by the passes, low bits first.
int plan_passes(u32 m, u32 tile, Pass *out)
{
    u32 lowbits = 0;
    while ((1u << (lowbits + 1)) <= tile) lowbits++;
    int np = 0;
    u32 k0 = 0;
    const u32 first = m < lowbits ? m : lowbits;
    out[np++] = Pass{0, first, 1};
    k0 = first;
    while (k0 < m) {
        const u32 ct = 16;  // 16 consecutive doubles = 128 bytes per run
        u32 span = 0;
        while ((ct << (span + 1)) <= tile) span++;
        const u32 k1 = (k0 + span < m) ? k0 + span : m;
        out[np++] = Pass{k0, k1, ct < (1u << k0) ? ct : (1u << k0)};
        k0 = k1;
    }
    return np;
}

template <int KIND, bool CONJ>
int launch_one(const PassArgs &a, unsigned grid, size_t smem, cudaStream_t s, const char *what)
{
    if (int rc = qmcgb::raise_smem_limit((const void *)ft_pass_kernel<KIND, CONJ>, smem, what)) return rc;
    ft_pass_kernel<KIND, CONJ><<<grid, FT_THREADS, smem, s>>>(a);
    return qmcgb::launch_status(what);
}

int launch_pass(int kind, bool conj, const PassArgs &a, unsigned grid, size_t smem, cudaStream_t s, const char *what)
{
    switch (kind) {
    case FT_FFT: return launch_one<FT_FFT, false>(a, grid, smem, s, what);
    case FT_IFFT: return conj ? launch_one<FT_IFFT, true>(a, grid, smem, s, what)
                              : launch_one<FT_IFFT, false>(a, grid, smem, s, what);
    case FT_FWHT: return launch_one<FT_FWHT, false>(a, grid, smem, s, what);
    case FT_CONV: return launch_one<FT_CONV, false>(a, grid, smem, s, what);
    default: return launch_one<FT_WCONV, false>(a, grid, smem, s, what);
    }
}

// ---- the fixed-point passes

// Few complex transforms of 2^9 are latency-bound, and the FP64 stages on 256 threads each
// answer sooner than one warp does, up to a vector per SM (FFT of 152 vectors: 12.6 us against
// 15.3; 200: 16.6 against 15.8; from 2^10 on fixed point wins from one vector, 15.0 against 17.4, but for
// data whose blocks take exponents of their own: 24, and from 2^11 on, 26 against 31).
bool use_fixed(bool real, u32 m, u64 nvec)
{
    return m > (u32)FIX_MIN_BITS || (m == (u32)FIX_MIN_BITS && (real || nvec > (u64)qmcgb::sm_count()));
}

// Bits of the low pass of an m-bit transform: what is left above it is a multiple of four.
u32 fix_low_bits(u32 m) { return m <= 12 ? m : 9 + (m - 9) % 4; }

// Passes, low bits first: the low pass, then eight bits at a time, four in the last one where
// eight do not remain.
int plan_fix_passes(u32 m, Pass *out)
{
    int np = 0;
    u32 k0 = fix_low_bits(m);
    out[np++] = Pass{0, k0, 1};
    while (k0 < m) {
        const u32 s = m - k0 >= 8 ? 8 : 4;
        out[np++] = Pass{k0, k0 + s, 4096u >> s};
        k0 += s;
    }
    return np;
}

template <class K>
int launch_fix(K kernel, const PassArgs &a, u64 tiles, unsigned threads, unsigned resident, size_t smem,
               cudaStream_t s, const char *what)
{
    if (int rc = qmcgb::raise_smem_limit((const void *)kernel, smem, what)) return rc;
    kernel<<<qmcgb::grid_for(tiles, 1, (unsigned)qmcgb::sm_count() * resident), threads, smem, s>>>(a);
    return qmcgb::launch_status(what);
}

template <int KIND, int P>
int launch_fix_low(const PassArgs &a, cudaStream_t s, const char *what)
{
    const u64 tiles = a.nvec << (a.m - P);
    const size_t words = slots(1u << P);
    if constexpr (KIND == FT_FWHT || KIND == FT_WCONV)
        return launch_fix(fix_low_wht_kernel<KIND, P>, a, tiles, 1u << (P - 4), P == 12 ? 4 : (P == 11 ? 8 : (P == 10 ? 16 : 32)),
                          words * 8, s, what);
    else
        return launch_fix(fix_low_kernel<KIND, P>, a, tiles, 1u << (P - 4), P == 12 ? 2 : (P == 11 ? 4 : (P == 10 ? 8 : 16)),
                          words * 16, s, what);
}

template <int KIND, bool CONJ>
int launch_fix_pass(const PassArgs &a, cudaStream_t s, const char *what)
{
    if (a.k0 == 0) {
        switch (a.k1) {
        case 9: return launch_fix_low<KIND, 9>(a, s, what);
        case 10: return launch_fix_low<KIND, 10>(a, s, what);
        case 11: return launch_fix_low<KIND, 11>(a, s, what);
        default: return launch_fix_low<KIND, 12>(a, s, what);
        }
    }
    const u64 tiles = (a.nvec << (a.m - a.k1)) * ((1ull << a.k0) / a.ct);
    const size_t words = slots(4096);
    const bool wide = a.k1 - a.k0 == 8;
    if constexpr (KIND == FT_FWHT || KIND == FT_WCONV)
        return wide ? launch_fix(fix_high_wht_kernel<KIND, 8>, a, tiles, 256, 4, words * 8, s, what)
                    : launch_fix(fix_high_wht_kernel<KIND, 4>, a, tiles, 256, 4, words * 8, s, what);
    else
        return wide ? launch_fix(fix_high_kernel<KIND, CONJ, 8>, a, tiles, 256, 2, words * 16, s, what)
                    : launch_fix(fix_high_kernel<KIND, CONJ, 4>, a, tiles, 256, 2, words * 16, s, what);
}

// one pass, in fixed point from 2^FIX_MIN_BITS values on
int launch_any(int kind, bool conj, bool fixed, PassArgs a, unsigned grid, size_t smem, cudaStream_t s,
               const char *what)
{
    if (!fixed) return launch_pass(kind, conj, a, grid, smem, s, what);
    a.conj = conj;
    switch (kind) {
    case FT_FFT: return launch_fix_pass<FT_FFT, false>(a, s, what);
    case FT_IFFT: return conj ? launch_fix_pass<FT_IFFT, true>(a, s, what) : launch_fix_pass<FT_IFFT, false>(a, s, what);
    case FT_FWHT: return launch_fix_pass<FT_FWHT, false>(a, s, what);
    case FT_CONV: return launch_fix_pass<FT_CONV, false>(a, s, what);
    default: return launch_fix_pass<FT_WCONV, false>(a, s, what);
    }
}

int run_transform(int kind, u64 d1, u64 d2, u64 n_half, double *twr, double *twi, double *xr, double *xi,
                  cudaStream_t s, const char *what)
{
    const u64 nvec = d1 * d2;
    QMC_REQUIRE_DOMAIN(n_half > 0 && (n_half & (n_half - 1)) == 0 && n_half <= (1ull << 40),
                       "%s: n = 2*n_half must be a power of two (n_half=%llu)", what,
                       (unsigned long long)n_half);
    const u64 n = 2 * n_half;
    u32 m = 0;
    while ((1ull << m) < n) m++;
    const bool fixed = use_fixed(kind == FT_FWHT || kind == FT_WCONV, m, nvec);
    if (kind != FT_FWHT) {
        QMC_REQUIRE(twr && twi, "%s: null twiddle pointer", what);
        twiddle_kernel<<<qmcgb::grid_for(n / 8 + 1 + (fixed ? 4096 + 256 : 8), 256, (unsigned)qmcgb::sm_count() * 8), 256, 0, s>>>(
            n, kind == FT_FFT ? -1.0 : 1.0, twr, twi, fixed ? 4096 + 256 : 0);
        if (int rc = qmcgb::launch_status(what)) return rc;
    }
    if (nvec == 0) return QMC_OK;
    QMC_REQUIRE(xr && (kind == FT_FWHT || xi), "%s: null data pointer", what);
    const u32 tile = kind == FT_FWHT ? TILE_REAL : TILE_COMPLEX;
    Pass passes[16];
    const int np = fixed ? plan_fix_passes(m, passes) : plan_passes(m, tile, passes);
    // orthonormal scaling 2^(-m/2), applied once by the last pass
    const double scale = (m % 2 == 0) ? ldexp(1.0, -(int)(m / 2)) : ldexp(1.0, -(int)(m / 2)) * 0.70710678118654752440;
    for (int pi = 0; pi < np; pi++) {
        const Pass p = (kind == FT_IFFT) ? passes[np - 1 - pi] : passes[pi];
        PassArgs a{};
        a.nvec = nvec;
        a.m = m;
        a.k0 = p.k0;
        a.k1 = p.k1;
        a.ct = p.ct;
        a.xr = xr;
        a.xi = xi;
        a.twr = twr;
        a.twi = twi;
        a.scale = (pi == np - 1) ? scale : 1.0;
        a.scale_exp = (pi == np - 1) ? -(int)(m / 2) : 0;
        a.scale_odd = (pi == np - 1) && m % 2;
        const u32 elems = (1u << (p.k1 - p.k0)) * p.ct;
        const size_t smem = (size_t)elems * sizeof(double) * (kind == FT_FWHT ? 1 : 2);
        const u64 tiles = nvec * (n >> p.k1) * ((1ull << p.k0) / p.ct);
        const unsigned grid = qmcgb::grid_for(tiles, 1, (unsigned)qmcgb::sm_count() * 8);
        if (int rc = launch_any(kind, false, fixed, a, grid, smem, s, what)) return rc;
    }
    return QMC_OK;
}

// y <- IFFT(FFT(y) * lam) * scale (or / lam), or the same with the WHT for real
// data: the forward passes but the last, one fused pass over the highest bits
// (forward steps, the pointwise step, inverse steps), the inverse passes but
// the first; FP64 throughout, the orthonormal factors folded into the
// pointwise scale.  The complex form fills the caller's twiddle arrays with
// the forward table and runs the inverse steps on its conjugates.
int run_fused(int kind, u64 d1, u64 d2, u64 n_half, double *twr, double *twi, const double *lr, const double *li,
              u64 lam_all, int divide, double scale, double *xr, double *xi, cudaStream_t s, const char *what)
{
    const bool real = kind == FT_WCONV;
    const u64 nvec = d1 * d2;
    QMC_REQUIRE_DOMAIN(n_half > 0 && (n_half & (n_half - 1)) == 0 && n_half <= (1ull << 40),
                       "%s: n = 2*n_half must be a power of two (n_half=%llu)", what,
                       (unsigned long long)n_half);
    QMC_REQUIRE(lam_all <= 1, "%s: lam_all is 0 (n values for every vector) or 1 (one per element)", what);
    const u64 n = 2 * n_half;
    u32 m = 0;
    while ((1ull << m) < n) m++;
    const bool fixed = use_fixed(kind == FT_FWHT || kind == FT_WCONV, m, nvec);
    if (!real) {
        QMC_REQUIRE(twr && twi, "%s: null twiddle pointer", what);
        twiddle_kernel<<<qmcgb::grid_for(n / 8 + 1 + (fixed ? 4096 + 256 : 8), 256, (unsigned)qmcgb::sm_count() * 8), 256, 0, s>>>(
            n, -1.0, twr, twi, fixed ? 4096 + 256 : 0);
        if (int rc = qmcgb::launch_status(what)) return rc;
    }
    if (nvec == 0) return QMC_OK;
    QMC_REQUIRE(xr && lr && (real || (xi && li)), "%s: null data or lam pointer", what);
    const u32 tile = real ? TILE_REAL : TILE_COMPLEX;
    Pass passes[16];
    const int np = fixed ? plan_fix_passes(m, passes) : plan_passes(m, tile, passes);
    // launch order: forward passes 0 .. np-2, the fused pass np-1, inverse passes np-2 .. 0
    for (int li_ = 0; li_ < 2 * np - 1; li_++) {
        const int pi = li_ < np ? li_ : 2 * np - 2 - li_;
        const int k = real ? (li_ == np - 1 ? FT_WCONV : FT_FWHT)
                           : (li_ < np - 1 ? FT_FFT : li_ == np - 1 ? FT_CONV : FT_IFFT);
        const Pass p = passes[pi];
        PassArgs a{};
        a.nvec = nvec;
        a.m = m;
        a.k0 = p.k0;
        a.k1 = p.k1;
        a.ct = p.ct;
        a.xr = xr;
        a.xi = xi;
        a.twr = twr;
        a.twi = twi;
        a.scale = 1.0;
        a.lr = lr;
        a.li = li;
        a.lam_all = (u32)lam_all;
        a.divide = divide ? 1u : 0u;
        a.lam_scale = scale / (double)n;
        a.fix_lam_scale = a.lam_scale;
        if (li_ == np - 1 && fixed) {
            // a factor that is a power of two goes into the exponent; tiles that it would take out of
            // the range (fix_range), and products that overflow without it, are done in FP64 with
            // the factor in the pointwise step
            int ex = 0;
            const double f = frexp(a.lam_scale, &ex);
            if (f == 0.5 && ex > -900 && ex < 900) {
                a.fix_lam_scale = 1.0;
                a.scale_exp = ex - 1;
            }
        }
        const u32 elems = (1u << (p.k1 - p.k0)) * p.ct;
        const size_t smem = (size_t)elems * sizeof(double) * (real ? 1 : 2);
        const u64 tiles = nvec * (n >> p.k1) * ((1ull << p.k0) / p.ct);
        const unsigned grid = qmcgb::grid_for(tiles, 1, (unsigned)qmcgb::sm_count() * 8);
        if (int rc = launch_any(k, k == FT_IFFT, fixed, a, grid, smem, s, what)) return rc;
    }
    return QMC_OK;
}

}  // namespace

extern "C" {

int qmc_fft_bro_1d_radix2(uint64_t d1, uint64_t d2, uint64_t n_half, double *twiddler, double *twiddlei, double *xr,
                          double *xi, qmc_stream_t s)
{
    return run_transform(FT_FFT, d1, d2, n_half, twiddler, twiddlei, xr, xi, QMC_STREAM(s), "fft_bro_1d_radix2");
}

int qmc_ifft_bro_1d_radix2(uint64_t d1, uint64_t d2, uint64_t n_half, double *twiddler, double *twiddlei, double *xr,
                           double *xi, qmc_stream_t s)
{
    return run_transform(FT_IFFT, d1, d2, n_half, twiddler, twiddlei, xr, xi, QMC_STREAM(s), "ifft_bro_1d_radix2");
}

int qmc_fwht_1d_radix2(uint64_t d1, uint64_t d2, uint64_t n_half, double *x, qmc_stream_t s)
{
    return run_transform(FT_FWHT, d1, d2, n_half, nullptr, nullptr, x, nullptr, QMC_STREAM(s), "fwht_1d_radix2");
}

int qmc_fft_mul_ifft(uint64_t d1, uint64_t d2, uint64_t n_half, double *twiddler, double *twiddlei, const double *lam_r,
                     const double *lam_i, uint64_t lam_per_element, int divide, double scale, double *xr, double *xi,
                     qmc_stream_t s)
{
    return run_fused(FT_CONV, d1, d2, n_half, twiddler, twiddlei, lam_r, lam_i, lam_per_element, divide, scale, xr,
                     xi, QMC_STREAM(s), "fft_mul_ifft");
}

int qmc_fwht_mul_fwht(uint64_t d1, uint64_t d2, uint64_t n_half, const double *lam, uint64_t lam_per_element,
                      int divide, double scale, double *x, qmc_stream_t s)
{
    return run_fused(FT_WCONV, d1, d2, n_half, nullptr, nullptr, lam, nullptr, lam_per_element, divide, scale, x,
                     nullptr, QMC_STREAM(s), "fwht_mul_fwht");
}

}  // extern "C"
