// halton_rows.cuh -- generation of the fused Halton plan with the term tables in shared
// memory and the digit sum mostly in integers, included by halton.cu.
//
// The sum of gdn_integer_to_float.c:33-39, v = RN(v + y_t), in three sections per (l, j):
//  * rows [0, t1), b^t1 >= 2^16: FP64 adds (the first is a load);
//  * the other rows: v's binade E is known now, and a term y becomes the integer
//    F = floor(y * 2^79).  While v stays in its binade, RN(v + y) adds y rounded to v's last
//    place 2^(E - 1075), whatever v is (ties aside), so the rounded terms are summed on their
//    own: acc = (acc + F + half) & ~(2^s - 1), s = 26 - (1022 - E): three integer
//    instructions a row where the FP64 add holds its narrow pipe for half a clock per SM.
//    The sum of the rounded terms is at last added to v's bits.  Rows [t1, tr), up to the last
//    one with a term that ties for some v of at least 2^-10 (terms above about 2^-25; every row of
//    base 2), round to even: seven instructions, with v's last bit in acc and a sticky bit in F.
// Points with v < 2^-10 after t1 rows (1 in 1000) or whose sum leaves the binade (v within 2^-16
// below a power of two) are redone by the plain FP64 chain.  Terms below half a last place of
// 2^-10 are left out.  A randomisation whose digits can reach their base (wide permutations)
// keeps FP64 for every row.
//
// Digits.  A raw digit is a sum mod b over the index digits.  The index splits as
// hi * b^K + x; the few hi of a warp's run of consecutive points have their sums H[hi][t] in
// shared memory.  Rows are renumbered by the inverse of the lowest digit's matrix entry (row t's table
// holds at g' the term of g = g' * C[0][t] mod b, the matrix is multiplied by the inverse), so
// with K = 1 a point's low part is its low digit itself in every row, and 32 consecutive points
// read consecutive table words: no bank conflicts, one add and one min per digit.  Rows whose
// entry has no inverse, and K > 1 (b < 32), read the low part from a table L[x][t].
//
// A CTA owns up to four consecutive dimensions of one randomisation (32 bytes of each output
// row, one store) and a range of points, in sections of a run per warp: no barrier after the tables, so
// that a warp with a point to redo holds up no other (with steps in common the barriers were
// two thirds of the time).  The term tables serve all sections of the CTA, the sums H one.
//
// What bounds it: issue (73 % of the slots), the shared-memory pipe (79 %: a table read is two
// wavefronts, a 32-byte piece of 32 rows up to 32) and the ALU (58 %).  First 100 primes, r = 32, n = 2^18: 6.67 ms
// (all FP64 adds 20.3; one section per CTA, and registers spilled for what the redone points need, 8.07).  The
// stores alone, a CTA after another in a column of 32 bytes, take 4.4 ms; with the CTAs of a row next
// to each other 2.6, but the whole no less (6.99: its CTAs differ in length).
#pragma once

namespace {

constexpr u32 HR_DIMS = 4;
constexpr u32 HR_PTS = 2;          // points of a lane: 32 apart
constexpr u32 HR_THREADS = 1024;   // 64 registers: 8.0 ms; 768 threads 8.8, 4 points on 640 threads 9.0 (first 100
                                   // primes, r=32, n=2^18, one section; 4 dimensions unrolled 8.9: instruction cache)
constexpr u32 HR_RUN = 16;         // most times 32 points in a warp's run (8: 7.21 ms, 16: 6.85, 32: 6.77, more memory)
constexpr u32 HR_STEPS = 64;       // most times HR_THREADS points of a CTA (16: 7.86 ms, 64: 6.92, 128: 7.02)
constexpr u32 HR_TINY = 9;         // integer rows need v >= 2^-(HR_TINY + 1)
constexpr int HR_UNIT = 79;        // F counts 2^-79: the integer rows' terms sum to 2^63 at most
constexpr u32 HR_HEAD_BITS = 16;   // b^t1 >= 2^16
// Below these the warp kernel, which has no tables to set up, finishes sooner.  us of preparation and run,
// warp kernel / this one, (r, n, d): (1, 20000, 20) 90 / 154, (4, 16384, 10) 121 / 157, (2, 30000, 50) 177 / 169,
// (16, 8192, 20) 197 / 181, (1, 10^6, 3) 647 / 339; of the run: (300, 1024, 100) 768 / 1386, (256, 2048, 100)
// 1267 / 1560, (32, 4096, 50) 211 / 185, (128, 4096, 100) 1266 / 979, (32, 262144, 100) 20320 / 6670, 64 uneven
// requests of 73 M coordinates 3027 / 1489.
constexpr double HR_MIN_COORDS = 2.4e6, HR_MIN_POINTS = 4000;
constexpr u32 HR_MAX_SMEM = 216 * 1024;  // and 6 KB of HConst, HSlow and output rows

// Up to four dimensions and the byte offsets of their tables in shared memory.
struct HGroup {
    u64 item0, span;      // its CTAs: r x splits from item0 on, span points each
    u32 req, splits;
    u32 j0, nd;
    u32 t_off[HR_DIMS], l_off[HR_DIMS], h_off[HR_DIMS], c_off[HR_DIMS];
    u32 h_size[HR_DIMS];  // per warp
};

// What this kernel needs of a dimension beyond HDim.
struct HRowDim {
    u32 t1, rows;  // FP64 rows at the front, rows that can change a sum of at least 2^-10
    u32 K2, bK2;   // low digits of its index split, b^K2
    u64 fdK2_M;
};

// 16-bit entries of a row of H or L: an even count, two digits to a word, an odd number of words
__host__ __device__ __forceinline__ u32 hr_pitch(u32 tmax) { return 2 * (((tmax + 1) / 2) | 1u); }

// what the preparation found about (l, j)
__device__ __forceinline__ u32 hr_info(u32 t1, u32 tr, u32 rows, bool low_table)
{
    return t1 | tr << 10 | rows << 20 | (low_table ? 1u << 31 : 0u);
}

// row flags: 1 a term that ties for some v in [2^-(HR_TINY+1), 1), 2 a digit at or above its base
__device__ __forceinline__ u32 hr_term_flags(u64 y, u64 dig, u64 b)
{
    u32 f = dig >= b ? 2u : 0u;
    if ((y >> 52) < 1023 - HR_HEAD_BITS) {
        bool exact;
        const u64 F = dsum::fixed_term(y, HR_UNIT, &exact);
        if (dsum::can_tie(F, exact, HR_UNIT, HR_TINY)) f |= 1u;
    } else {
        f |= 1u;  // too large for the integer rows
    }
    return f;
}

__device__ __forceinline__ u32 inverse_mod(u32 a, u32 b)  // 0 when there is none
{
    int r0 = (int)b, r1 = (int)a, x0 = 0, x1 = 1;
    while (r1) {
        const int q = r0 / r1, r = r0 - q * r1, x = x0 - q * x1;
        r0 = r1;
        r1 = r;
        x0 = x1;
        x1 = x;
    }
    if (r0 != 1) return 0;
    return (u32)(x0 < 0 ? x0 + (int)b : x0);
}

// One thread per (request, l, j, t): the row's multiplier (1 when the lowest digit's entry has no
// inverse) and the matrix column divided by it.
__global__ void halton_norm_kernel(HPlanDev P, const u32 *C, u32 *Cn, u32 *mul)
{
    for (u64 row = (u64)blockIdx.x * blockDim.x + threadIdx.x; row < P.rows; row += (u64)gridDim.x * blockDim.x) {
        const HReq &R = P.req[req_of(P.req, P.nreq, row, [](const HReq &q) { return q.t_base; })];
        const u64 loc = row - R.t_base, l = loc / R.s_per_l, off = loc % R.s_per_l;
        const HDim *dims = P.dims + R.dim0;
        const HDim &D = dims[dim_of(dims, R.d, off, [](const HDim &h) { return h.s_off; })];
        const u32 t = (u32)(off - D.s_off);
        if (t >= D.tmax) continue;
        const u64 base = R.c_base + l * R.c_per_l + D.c_off + t;
        const u32 c0 = C[base], q = inverse_mod(c0, D.b);
        mul[row] = q ? c0 : 1u;
        for (u32 k = 0; k < D.mmax; k++) {
            const u32 c = C[base + (u64)k * D.tmax];
            Cn[base + (u64)k * D.tmax] = q ? hmod(D.fd_M, D.b, c * q) : c;
        }
    }
}

// One thread per (request, l, j): the sections of its rows.
__global__ void halton_info_kernel(HPlanDev P, const u32 *flags, const u32 *Cn, u32 *info)
{
    for (u64 w = (u64)blockIdx.x * blockDim.x + threadIdx.x; w < P.titems; w += (u64)gridDim.x * blockDim.x) {
        const HReq &R = P.req[req_of(P.req, P.nreq, w, [](const HReq &q) { return q.tl_base; })];
        const u64 loc = w - R.tl_base, l = loc / R.d, j = loc % R.d;
        const HDim &D = P.dims[R.dim0 + j];
        const HRowDim &X = P.rdims[R.dim0 + j];
        const u32 *f = flags + R.t_base + l * R.s_per_l + D.s_off;
        const u32 *c0 = Cn + R.c_base + l * R.c_per_l + D.c_off;
        bool wide = false, low = X.K2 > 1;
        u32 tr = X.t1;
        for (u32 t = 0; t < D.tmax; t++) {
            wide = wide || (f[t] & 2u);
            if (t >= X.t1 && t < X.rows && (f[t] & 1u)) tr = t + 1;
            low = low || c0[t] != 1u;
        }
        info[w] = wide ? hr_info(D.tmax, D.tmax, D.tmax, low) : hr_info(X.t1, tr, X.rows, low);
    }
}

// Table reads by 32-bit shared-memory address.  hr_ld16, hr_ld32: T and L, which no one writes after the last
// barrier.  The sums H are written anew in every section: their reads (hr_sum16, hr_sum32) stay
// between the warp's barriers around the writes.
__device__ __forceinline__ u32 hr_ld16(u32 a)
{
    u32 v;
    asm("{.reg .u16 h; ld.shared.u16 h, [%1]; cvt.u32.u16 %0, h;}" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ u32 hr_ld32(u32 a)
{
    u32 v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ u64 hr_ld64(u32 a)
{
    u64 v;
    asm("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ u32 hr_sum16(u32 a)
{
    u32 v;
    asm volatile("{.reg .u16 h; ld.shared.u16 h, [%1]; cvt.u32.u16 %0, h;}" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ u32 hr_sum32(u32 a)
{
    u32 v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// What the steps of a warp need of a dimension, in shared memory.
struct HConst {
    u32 info, b8, bK2, pitch2;
    u64 M;            // direct-remainder constant of b^K2
    u32 T, H, L, h0;  // addresses of the tables; H, h0: this warp's and its first hi
};

// What the sections and the plain chain of a point need of a dimension, in shared memory (pointers
// kept in registers over the points' loop spilled others: 6.96 ms).
struct HSlow {
    const HDim *D;
    const HRowDim *X;
    const u64 *Y;
    const u32 *mul;
};

// The digits of one point: byte offsets in the rows of the term table.  LOW: the low part from
// the table row at `lp`, else the thread's own x8.
template <bool LOW>
struct HDigits {
    u32 hp, low;  // H[hi]; L[x] or the low part itself, times 8
    __device__ __forceinline__ u32 at(u32 t, u32 b8) const
    {
        const u32 s = hr_sum16(hp + 2 * t) + (LOW ? hr_ld16(low + 2 * t) : low);
        return __viaddmin_u32(s, 0u - b8, s);
    }
    // rows t (even) and t + 1 in the halves of a word, both sums below 2^15: a read, an add and a
    // conditional subtract for two digits (one each: 6.85 ms, 6.67 by pairs)
    __device__ __forceinline__ u32 pair(u32 t, u32 b8) const
    {
        const u32 s = hr_sum32(hp + 2 * t) + (LOW ? hr_ld32(low + 2 * t) : low * 0x10001u);
        return __viaddmin_u16x2(s, (0x10000u - b8) * 0x10001u, s);
    }
};

// The plain FP64 chain of one point, terms from the plan's table (mul: the rows' multipliers).
template <bool LOW>
__device__ __noinline__ double hr_point(const HDigits<LOW> W, const HSlow *slow)
{
    const HDim &D = *slow->D;
    const u64 *Y = slow->Y;
    const u32 *mul = slow->mul;
    const u32 b = D.b, tmax = D.tmax;
    const u64 M = D.fd_M;
    double v = 0.0;
#pragma unroll 4
    for (u32 t = 0; t < tmax; t++) v = __dadd_rn(v, as_double(Y[t * b + hmod(M, b, (W.at(t, 8 * b) >> 3) * mul[t])]));
    return v;
}

// The values of the lane's HR_PTS points; false in ok where a point has to be redone.
template <bool LOW>
__device__ __forceinline__ void hr_values(const HDigits<LOW> (&W)[HR_PTS], u32 T, u32 b8, u32 info,
                                          double (&v)[HR_PTS], bool (&ok)[HR_PTS])
{
    const u32 t1 = info & 1023u, tr = info >> 10 & 1023u, rows = info >> 20 & 1023u;
    u32 t = t1 > 1 ? 2 : 1;  // one row where there are no more digits
#pragma unroll
    for (u32 p = 0; p < HR_PTS; p++) {
        ok[p] = true;
        if (t == 2) {
            const u32 m = W[p].pair(0, b8);
            v[p] = __dadd_rn(as_double(hr_ld64(T + (m & 0xFFFFu))), as_double(hr_ld64(T + b8 + (m >> 16))));
        } else {
            v[p] = as_double(hr_ld64(T + W[p].at(0, b8)));
        }
    }
    T += (t - 1) * b8;
    for (; t < t1; t++) {
        T += b8;
#pragma unroll
        for (u32 p = 0; p < HR_PTS; p++) v[p] = __dadd_rn(v[p], as_double(hr_ld64(T + W[p].at(t, b8))));
    }
    if (t1 == rows) return;
    u64 acc[HR_PTS];
    u32 half[HR_PTS];
#pragma unroll
    for (u32 p = 0; p < HR_PTS; p++) {
        const u32 hi = (u32)__double2hiint(v[p]), tiny = 1022u - (hi >> 20);  // v < 1
        const u32 s = (HR_UNIT - 53) - (tiny <= HR_TINY ? tiny : 0u);
        half[p] = 1u << (s - 1);
        acc[p] = (u64)((u32)__double2loint(v[p]) & 1u) << s;
    }
    for (; t < tr; t++) {
        T += b8;
#pragma unroll
        for (u32 p = 0; p < HR_PTS; p++) acc[p] = dsum::add_even(acc[p], hr_ld64(T + W[p].at(t, b8)), half[p]);
    }
    auto plain_row = [&]() {
        T += b8;
#pragma unroll
        for (u32 p = 0; p < HR_PTS; p++) acc[p] = dsum::add_plain(acc[p], hr_ld64(T + W[p].at(t, b8)), half[p]);
        t++;
    };
    if ((t & 1u) && t < rows) plain_row();
#pragma unroll 1
    for (; t + 1 < rows; t += 2) {
        T += 2 * b8;
#pragma unroll
        for (u32 p = 0; p < HR_PTS; p++) {
            const u32 m = W[p].pair(t, b8);
            acc[p] = dsum::add_plain(acc[p], hr_ld64(T - b8 + (m & 0xFFFFu)), half[p]);
            acc[p] = dsum::add_plain(acc[p], hr_ld64(T + (m >> 16)), half[p]);
        }
    }
    if (t < rows) plain_row();
#pragma unroll
    for (u32 p = 0; p < HR_PTS; p++) {
        const u64 vb = as_bits(v[p]);
        const u32 E = (u32)(vb >> 52), s = 32u - __clz((int)half[p]);  // half = 2^(s - 1)
        const u64 r = (vb & ~1ull) + (acc[p] >> s);
        ok[p] = 1022u - E <= HR_TINY && (u32)(r >> 52) == E;
        v[p] = as_double(r);
    }
}

// One dimension of the lane's points.
template <bool LOW>
__device__ __forceinline__ void hr_dim(const HConst &c, const u32 (&index)[HR_PTS], const HSlow *slow,
                                       double (&v)[HR_PTS])
{
    HDigits<LOW> W[HR_PTS];
    bool ok[HR_PTS];
#pragma unroll
    for (u32 p = 0; p < HR_PTS; p++) {
        const u32 hi = hdiv(c.M, index[p]), x = index[p] - hi * c.bK2;
        W[p].hp = c.H + (hi - c.h0) * c.pitch2;
        W[p].low = LOW ? c.L + x * c.pitch2 : 8 * x;
    }
    hr_values<LOW>(W, c.T, c.b8, c.info, v, ok);
#pragma unroll
    for (u32 p = 0; p < HR_PTS; p++)
        if (!ok[p]) v[p] = hr_point<LOW>(W[p], slow);
}

__global__ void __launch_bounds__(HR_THREADS, 1) halton_rows_kernel(HPlanDev P)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ HConst consts[32][HR_DIMS];
    __shared__ HSlow slow[HR_DIMS];
    __shared__ double *outs[32];  // a warp's output row
    const u32 tid = threadIdx.x, nt = blockDim.x, warp = tid / 32, lane = tid % 32, nw = nt / 32;
    const u64 item = blockIdx.x;
    u32 glo = 0, ghi = P.ngroups - 1;  // the group whose CTAs hold this one
    while (glo < ghi) {
        const u32 mid = (glo + ghi + 1) >> 1;
        if (P.groups[mid].item0 <= item)
            glo = mid;
        else
            ghi = mid - 1;
    }
    const HGroup &G = P.groups[glo];
    const HReq &R = P.req[G.req];
    const u64 loc = item - G.item0, l = loc / G.splits, split = loc % G.splits;
    const HDim *dims = P.dims + R.dim0 + G.j0;
    const HRowDim *rdims = P.rdims + R.dim0 + G.j0;
    const u32 *Cnl = P.Cn + R.c_base + l * R.c_per_l;
    const u64 *Yl = P.Y + R.y_base + l * R.y_per_l;
    const u32 *mul_l = P.mul + R.t_base + l * R.s_per_l;
    const u32 *info_l = P.info + R.tl_base + l * R.d + G.j0;
    const u32 nd = G.nd;
    HConst *hc = consts[warp];
    const u32 sa = (u32)__cvta_generic_to_shared(sm);
    // the tables of the group's dimensions
    for (u32 q = 0; q < nd; q++) {
        const u32 info = info_l[q];
        const HDim &D = dims[q];
        const u32 t1 = info & 1023u, rows = info >> 20 & 1023u;
        const u32 b = D.b, tmax = D.tmax, nb = (b + 31) / 32;
        u64 *T = (u64 *)(sm + G.t_off[q]);
        const u64 *Y = Yl + D.y_off;
        const u32 *mul = mul_l + D.s_off;
        for (u32 u = warp; u < rows * nb; u += nw) {
            const u32 t = u / nb, g = (u % nb) * 32 + lane;
            if (g < b) {
                const u64 y = Y[t * b + hmod(D.fd_M, b, g * mul[t])];
                bool exact;
                const u64 F = dsum::fixed_term(y, HR_UNIT, &exact);
                T[t * b + g] = t >= t1 ? F | (exact ? 0u : 1u) : y;
            }
        }
        if (tid == 0) slow[q] = HSlow{&D, rdims + q, Y, mul};
        u32 *Cs = (u32 *)(sm + G.c_off[q]);
        for (u32 e = tid; e < D.mmax * tmax; e += nt) Cs[e] = Cnl[D.c_off + e];
    }
    __syncthreads();
    for (u32 q = 0; q < nd; q++) {
        if (!(info_l[q] >> 31)) continue;
        const HDim &D = dims[q];
        const HRowDim &X = rdims[q];
        const u32 pitch = hr_pitch(D.tmax);
        const u32 *Cs = (const u32 *)(sm + G.c_off[q]);
        u16 *L = (u16 *)(sm + G.l_off[q]);
        for (u32 x = warp; x < X.bK2; x += nw)
            for (u32 t = lane; t < D.tmax; t += 32) {
                u32 acc = 0, h = x;
                for (u32 k = 0; k < X.K2 && k < D.mmax; k++) {
                    const u32 d = hdiv(D.fd_M, h);
                    acc += (h - d * D.b) * Cs[k * D.tmax + t];
                    h = d;
                }
                L[x * pitch + t] = (u16)(8u * dim_mod(D, acc));
            }
    }
    __syncthreads();
    const u32 d = (u32)R.d;
    const bool v4 = nd == 4 && d % 4 == 0 && ((uintptr_t)R.x & 31u) == 0;
    // the CTA's points in sections, a run of each per warp: the tables above serve all of them, the
    // sums of the high digits one
    const u64 c0 = split * G.span, c_end = min(R.n, c0 + G.span);
    const u32 per = (u32)(G.span / nt), sections = (per + HR_RUN - 1) / HR_RUN;
    const u32 run = (per + sections - 1) / sections * 32;
    for (u64 i0 = c0 + warp * run; i0 < c_end; i0 += nw * run) {
        const u32 cnt = (u32)min((u64)run, c_end - i0);
        const u32 base = (u32)(R.n_start + i0);
        __syncwarp();  // the sums of the section before have been read
        if (lane == 0) outs[warp] = R.x + (l * R.n + i0) * R.d + G.j0;
        for (u32 q = 0; q < nd; q++) {
            const HDim &D = *slow[q].D;
            const HRowDim &X = *slow[q].X;
            const u32 tmax = D.tmax, pitch = hr_pitch(tmax), h0 = hdiv(X.fdK2_M, base);
            const u32 nh = hdiv(X.fdK2_M, base + cnt - 1) - h0 + 1;
            const u32 *Cs = (const u32 *)(sm + G.c_off[q]);
            u16 *H = (u16 *)(sm + G.h_off[q] + warp * G.h_size[q]);
            if (lane == 0)
                hc[q] = HConst{info_l[q], 8 * D.b, X.bK2, 2 * pitch, X.fdK2_M, sa + G.t_off[q],
                               sa + G.h_off[q] + warp * G.h_size[q], sa + G.l_off[q], h0};
            for (u32 e = lane; e < nh * tmax; e += 32) {
                const u32 u = e / tmax, t = e - u * tmax;
                u32 acc = 0, h = h0 + u;
                for (u32 k = X.K2; h && k < D.mmax; k++) {
                    const u32 d = hdiv(D.fd_M, h);
                    acc += (h - d * D.b) * Cs[k * tmax + t];
                    h = d;
                }
                H[u * pitch + t] = (u16)(8u * dim_mod(D, acc));
            }
        }
        __syncwarp();
        for (u32 i = lane; i < cnt; i += 32 * HR_PTS) {
            // a point past the end repeats the first: no branch around the shared work
            u32 index[HR_PTS];
#pragma unroll
            for (u32 p = 0; p < HR_PTS; p++) index[p] = base + (i + 32 * p < cnt ? i + 32 * p : i);
            double v[HR_DIMS][HR_PTS];
#pragma unroll 1
            for (u32 q = 0; q < HR_DIMS; q++) {
                if (q >= nd) break;
                const HConst c = hc[q];
                if (c.info >> 31)
                    hr_dim<true>(c, index, slow + q, v[q]);
                else
                    hr_dim<false>(c, index, slow + q, v[q]);
            }
#pragma unroll
            for (u32 p = 0; p < HR_PTS; p++) {
                if (i + 32 * p >= cnt) break;
                double *out = outs[warp] + (u64)(i + 32 * p) * d;
                if (v4) {
                    asm volatile("st.global.cs.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(out), "d"(v[0][p]), "d"(v[1][p]),
                                 "d"(v[2][p]), "d"(v[3][p])
                                 : "memory");
                } else {
#pragma unroll
                    for (u32 q = 0; q < HR_DIMS; q++)
                        if (q < nd) __stcs(out + q, v[q][p]);
                }
            }
        }
    }
}

}  // namespace
