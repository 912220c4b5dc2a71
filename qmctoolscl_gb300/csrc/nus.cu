// nus.cu -- nested uniform (Owen) scrambling of base-2 digital nets,
// bit for bit the reference's dnb2_nested_uniform_scramble
// (qmctoolscl/rand_funcs.py:155-253) with numpy's SFC64 generator streams.
//
// The reference walks one binary tree per generator (replication l,
// dimension j), point by point, and draws random bits whenever a point opens
// a new branch.  Its output is fixed by three facts:
//   * the root starts as a leaf for a phantom point with key 0 holding
//     tmax_new random bits, drawn first (rand_funcs.py:191-195);
//   * point v then draws tmax_new - L_v - 1 bits, where L_v is the longest
//     common prefix of v's key (xb << (tmax_new - tmax), tmax_new bits) with
//     any earlier point's key -- nothing when v repeats an earlier key;
//   * bit k (from the top) of a point's scramble comes from the draw of the
//     earliest point that shares the point's first k key bits.
// So per generator (all generators at once, in chunks that fit the caller's
// workspace):
//   1. keys in point order, the phantom (or the history of earlier calls)
//      first: transposed from xb's (r_x, n, d) layout;
//   2. stable LSD radix sort of (key, point) pairs, 8 bits per pass, over
//      the top log2(N) + 4 bits or so, each run of keys equal there finished
//      by an insertion sort (all 8-bit digits when a run is long);
//   3. bottom up, in one pass, the binary radix tree over the sorted pairs
//      (Apetrei's agglomerative construction; keys extended by the point
//      index so that equal keys split too) and each internal node's earliest
//      point; the later of its two children's earliest points first shares
//      a prefix of the node's length with an earlier point, which gives
//      every L_v;
//   4. the draws: how many outputs each takes from the generator (prefix
//      counts), the streams (the only serial step: numpy's SFC64), and the
//      draws' bits from them, by numpy's bounded-integer rule;
//   5. each node's part of the scramble (its earliest point's draw over the
//      depths the node spans) and each leaf's OR over its ancestors;
//   6. xrb = (xb << (tmax_new - tmax)) ^ scramble, transposed back.
#include "nus_dev.cuh"

namespace {

// ---- 1. keys ---------------------------------------------------------------

__global__ void nus_keys_kernel(NusDims m, const u64 *__restrict__ xb, const u64 *__restrict__ hist_keys,
                                const u64 *__restrict__ hist_draws, u64 *__restrict__ key, u64 *__restrict__ draw,
                                u64 *__restrict__ keys_out)
{
    __shared__ u64 tile[32][33];
    const u32 v0 = blockIdx.x * 32, g0 = blockIdx.y * 32;
    for (u32 k = threadIdx.y; k < 32; k += 8) {  // lanes along generators: xb's dimension axis
        const u32 v = v0 + k, g = g0 + threadIdx.x;
        u64 kv = 0;
        if (v < m.N && g < m.S) {
            const u64 s = m.s0 + g;
            if (v < m.H0) {
                kv = m.fresh ? 0 : hist_keys[s * m.h0 + v];
            } else {
                const u64 l = s / m.d, j = s - l * m.d, i = v - m.H0;
                const u64 w = xb[((l % m.r_x) * m.n + i) * m.d + j];
                kv = (m.td >= 64 ? 0 : w << m.td) & m.mask;
            }
        }
        tile[k][threadIdx.x] = kv;
    }
    __syncthreads();
    for (u32 k = threadIdx.y; k < 32; k += 8) {  // lanes along points
        const u32 g = g0 + k, v = v0 + threadIdx.x;
        if (g < m.S && v < m.N) {
            const u64 kv = tile[threadIdx.x][k];
            key[(u64)g * m.NP + v] = kv;
            if (keys_out) keys_out[(m.s0 + g) * m.N + v] = kv;
            if (!m.fresh && v < m.H0) draw[(u64)g * m.NP + v] = hist_draws[(m.s0 + g) * m.h0 + v];
        }
    }
}


// ---- 2-3. the radix sort and the bottom-up tree pass: nus_dev.cuh -------------------

// ---- 4. the draws ------------------------------------------------------------------
// Point v's draw of nb = T - 1 - L_v bits (the phantom's of T, first of all) is, by numpy's rules, the
// top nb bits of one 64-bit output (nb > 32), or of a 32-bit half (0 < nb <= 32): the high half kept
// from the last output that a half draw took, else the low half of a new output, whose high half is
// then kept.  So half draws alternate between a new output and the kept half, and the outputs taken
// before a draw are the full draws before it plus every other half draw: prefix counts.  The counts
// come first (one warp per 256 points, then a scan per generator); the stream itself, the only
// serial part, then runs without looking at the draws; and the draws take their bits from it, a
// thread per point.  With the draws formatted and stored inside the serial loop, a step took
// 68 cycles; the bare chain of 64-bit integer operations takes 24 on one warp (up to 32
// generators: the ALU).  r=4, d=8, n=200000: 7.15 ms for the draws before, 2.59 now (stream 2.53).

constexpr u32 DT = 256;  // points per warp of the counting and formatting passes: all loads in flight at once

// A tile's draws of more than 32 bits and of 1 to 32, with the full draws before its last two half
// draws; after the scan the prefix counts up to and including the tile, and in last1 the output
// that the last half draw with a new one took (NONE: no such draw).
struct DrawCount {
    u32 full, half, last1, last2;
};

// a generator's stream: outputs to run, and numpy's kept half at the start
struct DrawInfo {
    u32 outputs, has, half, pad;
};

__device__ __forceinline__ u32 tiles_of_draws(u32 N) { return (N + DT - 1) / DT; }

// bits that point v draws
__device__ __forceinline__ u32 draw_bits(const NusDims &m, u32 v, u32 L)
{
    if (v < m.H0) return m.fresh ? m.T : 0u;
    return L + 1 >= m.T ? 0u : m.T - 1 - L;
}

// the same for a lane's points v0, v0 + 32, .. of a tile; 0 past the end
__device__ __forceinline__ void tile_bits(const NusDims &m, const unsigned char *__restrict__ L, u32 v0,
                                          u32 (&nb)[DT / 32])
{
#pragma unroll
    for (u32 i = 0; i < DT / 32; i++) nb[i] = v0 + 32 * i < m.N && v0 + 32 * i >= m.H0 ? L[v0 + 32 * i] : 0;
#pragma unroll
    for (u32 i = 0; i < DT / 32; i++) nb[i] = v0 + 32 * i < m.N ? draw_bits(m, v0 + 32 * i, nb[i]) : 0;
}

// outputs that the first h half draws take, `has`: a half was kept at the start
__device__ __forceinline__ u32 half_outputs(u32 h, u32 has) { return (h + 1 - has) >> 1; }

__global__ void __launch_bounds__(256) nus_draw_count_kernel(NusDims m, const unsigned char *__restrict__ Lv,
                                                             DrawCount *__restrict__ counts)
{
    const u32 lane = threadIdx.x & 31, tile = blockIdx.x * 8 + (threadIdx.x >> 5), g = blockIdx.y;
    const u32 tiles = tiles_of_draws(m.N);
    if (tile >= tiles) return;
    u32 nb[DT / 32];
    tile_bits(m, Lv + (u64)g * m.NP, tile * DT + lane, nb);
    DrawCount c{0, 0, 0, 0};
#pragma unroll
    for (u32 i = 0; i < DT / 32; i++) {
        const u32 full = __ballot_sync(0xFFFFFFFFu, nb[i] > 32);
        const u32 half = __ballot_sync(0xFFFFFFFFu, nb[i] && nb[i] <= 32);
        if (half) {
            const u32 top = 1u << (31 - __clz(half)), rest = half ^ top;
            c.last2 = rest ? c.full + __popc(full & ((1u << (31 - __clz(rest))) - 1)) : c.last1;
            c.last1 = c.full + __popc(full & (top - 1));
        }
        c.full += __popc(full);
        c.half += __popc(half);
    }
    if (lane == 0) counts[(u64)g * tiles + tile] = c;
}

// one warp per generator: the scan over its tiles, the stream's length
__global__ void __launch_bounds__(32) nus_draw_scan_kernel(NusDims m, const u64 *__restrict__ states,
                                                           DrawCount *__restrict__ counts, DrawInfo *__restrict__ info)
{
    const u32 lane = threadIdx.x, g = blockIdx.x, tiles = tiles_of_draws(m.N);
    const u64 *st = states + (m.s0 + g) * 6;
    const u32 has = st[4] != 0;
    DrawCount *C = counts + (u64)g * tiles;
    u32 full = 0, half = 0, kept = NONE;
    for (u32 t0 = 0; t0 < tiles; t0 += 32) {
        const u32 t = t0 + lane;
        const DrawCount c = t < tiles ? C[t] : DrawCount{0, 0, 0, 0};
        u32 f = c.full, h = c.half;
#pragma unroll
        for (u32 o = 1; o < 32; o *= 2) {
            const u32 a = __shfl_up_sync(0xFFFFFFFFu, f, o), b = __shfl_up_sync(0xFFFFFFFFu, h, o);
            if (lane >= o) {
                f += a;
                h += b;
            }
        }
        // this tile's last half draw with a new output: its last one or the one before, by parity
        const u32 before = full + f - c.full, end = half + h;  // end: half draws up to and including the tile
        const u32 odd = (end - 1 + has) & 1u;                  // the last one took the kept half
        const bool any = c.half > odd;
        const u32 mine = before + (odd ? c.last2 : c.last1) + half_outputs(end - 1 - odd, has);
        const u32 with = __ballot_sync(0xFFFFFFFFu, any) & (0xFFFFFFFFu >> (31 - lane));
        const u32 from = __shfl_sync(0xFFFFFFFFu, mine, with ? 31 - __clz(with) : 0);
        const u32 k = with ? from : kept;
        if (t < tiles) C[t] = DrawCount{full + f, end, k, 0};
        full += __shfl_sync(0xFFFFFFFFu, f, 31);
        half += __shfl_sync(0xFFFFFFFFu, h, 31);
        kept = __shfl_sync(0xFFFFFFFFu, k, 31);
    }
    if (lane == 0) info[g] = DrawInfo{full + half_outputs(half, has), has, (u32)st[5], 0};
}

constexpr u32 STREAM_STEPS = 64;  // outputs per generator between two barriers (32: the whole call 4.80 ms, 64: 4.45)

// The streams of 32 generators: warp 0, alone on its quarter of the SM, steps them (a lane each) into
// shared memory, the other three warps write whole 256-byte row segments behind it.
__global__ void __launch_bounds__(128) nus_stream_kernel(NusDims m, u64 *__restrict__ states,
                                                         const DrawInfo *__restrict__ info, u64 *__restrict__ raw)
{
    __shared__ u64 buf[2][STREAM_STEPS][33];
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g0 = blockIdx.x * 32, g = g0 + lane;
    const u32 need = g < m.S ? info[g].outputs : 0;
    const u32 most = __reduce_max_sync(0xFFFFFFFFu, need);
    // lanes past the last generator step a stream of zeros along with the others, into a column that no one reads
    const u32 least = __reduce_min_sync(0xFFFFFFFFu, g < m.S ? need : NONE);
    u64 *st = states + (g < m.S ? m.s0 + g : 0) * 6;
    Sfc64 r{0, 0, 0, 0, 0, 0};
    if (warp == 0 && g < m.S) r = Sfc64{st[0], st[1], st[2], st[3], 0, 0};
    for (u32 i0 = 0, k = 0; i0 < most; i0 += STREAM_STEPS, k ^= 1) {
        if (warp == 0) {
            if (i0 + STREAM_STEPS <= least && __all_sync(0xFFFFFFFFu, (u32)r.w <= 0u - STREAM_STEPS)) {
                // the counter's upper half stands still: an instruction less of a step's thirteen on the ALU
                const u64 high = r.w & 0xFFFFFFFF00000000ull;
                const u32 low = (u32)r.w;
#pragma unroll
                for (u32 s = 0; s < STREAM_STEPS; s++) {
                    r.w = high | (low + s);
                    buf[k][s][lane] = r.next64();
                }
            } else {
                for (u32 s = 0; s < STREAM_STEPS && i0 + s < need; s++) buf[k][s][lane] = r.next64();
            }
        }
        __syncthreads();  // also: the other warps are done with the other buffer
        if (warp != 0) {
            // all reads ahead of all stores: row by row, three warps took longer than the 32 steps
#pragma unroll 1
            for (u32 h = 0; h < STREAM_STEPS; h += 32) {
                u64 x[11];
#pragma unroll
                for (u32 e = 0; e < 11; e++) x[e] = buf[k][h + lane][min(warp - 1 + 3 * e, 31u)];
                u64 *row = raw + (u64)(g0 + warp - 1) * m.NP + i0 + h + lane;
#pragma unroll
                for (u32 e = 0; e < 11; e++) {
                    const u32 q = warp - 1 + 3 * e, end = __shfl_sync(0xFFFFFFFFu, need, q & 31u);
                    if (q < 32 && i0 + h + lane < end) row[(u64)(3 * e) * m.NP] = x[e];
                }
            }
        }
    }
    if (warp == 0 && g < m.S) {
        st[0] = r.a;
        st[1] = r.b;
        st[2] = r.c;
        st[3] = r.w;
    }
}

// the draws of a tile from the stream; the last tile leaves numpy's kept half in the state
__global__ void __launch_bounds__(256) nus_draw_kernel(NusDims m, const unsigned char *__restrict__ Lv,
                                                       const DrawCount *__restrict__ counts,
                                                       const DrawInfo *__restrict__ info, const u64 *__restrict__ raw,
                                                       u64 *__restrict__ states, u64 *__restrict__ draw)
{
    const u32 lane = threadIdx.x & 31, tile = blockIdx.x * 8 + (threadIdx.x >> 5), g = blockIdx.y;
    const u32 tiles = tiles_of_draws(m.N);
    if (tile >= tiles) return;
    const u64 *R = raw + (u64)g * m.NP;
    u64 *D = draw + (u64)g * m.NP;
    const DrawInfo in = info[g];
    const u32 v0 = tile * DT + lane;
    u32 nb[DT / 32], at[DT / 32];  // at: the output, NONE for the state's half
    u32 high = 0;                  // bit i: draw i takes a kept half
    tile_bits(m, Lv + (u64)g * m.NP, v0, nb);
    DrawCount c{0, 0, NONE, 0};
    if (tile) c = counts[(u64)g * tiles + tile - 1];
    u32 kept = c.last1;  // the output whose high half is or was kept last (NONE: the state's own half)
    const u32 lt = (1u << lane) - 1;
#pragma unroll
    for (u32 i = 0; i < DT / 32; i++) {
        const bool is_half = nb[i] && nb[i] <= 32;
        const u32 full = __ballot_sync(0xFFFFFFFFu, nb[i] > 32), half = __ballot_sync(0xFFFFFFFFu, is_half);
        at[i] = c.full + __popc(full & lt);
        if (half) {  // the same for the warp
            const u32 h = c.half + __popc(half & lt);  // half draws before this point
            at[i] += half_outputs(h, in.has);
            const bool fresh = ((h + in.has) & 1u) == 0;
            const u32 news = __ballot_sync(0xFFFFFFFFu, is_half && fresh), before = news & lt;
            // the last new output of a half draw before each lane
            const u32 from = __shfl_sync(0xFFFFFFFFu, at[i], before ? 31 - __clz(before) : 0);
            const u32 last = __shfl_sync(0xFFFFFFFFu, at[i], news ? 31 - __clz(news) : 0);
            if (is_half && !fresh) {
                at[i] = before ? from : kept;
                high |= 1u << i;
            }
            if (news) kept = last;
        } else {
            at[i] += half_outputs(c.half, in.has);
        }
        c.full += __popc(full);
        c.half += __popc(half);
    }
    u64 x[DT / 32];
#pragma unroll
    for (u32 i = 0; i < DT / 32; i++) x[i] = nb[i] && at[i] != NONE ? R[at[i]] : (u64)in.half << 32;
#pragma unroll
    for (u32 i = 0; i < DT / 32; i++) {
        const u32 v = v0 + 32 * i;
        u64 y = 0;
        if (nb[i] > 32)
            y = nb[i] == 64 ? x[i] : x[i] >> (64 - nb[i]);
        else if (nb[i])
            y = ((high >> i) & 1u ? (u32)(x[i] >> 32) : (u32)x[i]) >> (32 - nb[i]);
        if (v < m.N && (v >= m.H0 || m.fresh)) D[v] = y;
    }
    if (tile == tiles - 1 && lane == 0) {
        u64 *st = states + (m.s0 + g) * 6;
        st[4] = (in.has + c.half) & 1u;
        st[5] = kept == NONE ? in.half : R[kept] >> 32;  // numpy keeps the last kept half here, used or not
    }
}

// ---- 5. scramble bits: each node's band, each leaf's ancestors -----------------
// A node spans the depths (parent's prefix length, own prefix length]; its
// bits there come from its earliest point's draw.  Depth k is bit T-1-k.

__device__ __forceinline__ u64 band_mask(int kmin, int kmax, int T)
{
    if (kmax > T - 1) kmax = T - 1;
    if (kmin > kmax) return 0;
    const u32 lo = (u32)(T - 1 - kmax), hi = (u32)(T - 1 - kmin);
    const u64 upto_hi = hi >= 63 ? ~0ull : ((2ull << hi) - 1ull);
    return upto_hi & ~((1ull << lo) - 1ull);
}

__global__ void __launch_bounds__(NUS_THREADS) nus_contrib_kernel(NusDims m, const unsigned char *__restrict__ lam,
                                                                  const u32 *__restrict__ pint,
                                                                  const u32 *__restrict__ minv,
                                                                  const u64 *__restrict__ draw,
                                                                  u64 *__restrict__ contrib)
{
    const u32 u = blockIdx.x * NUS_THREADS + threadIdx.x, g = blockIdx.y;
    if (u + 1 >= m.N) return;
    const u64 off = (u64)g * m.NP;
    const u32 P = pint[off + u];
    const int dP = P == NONE ? -1 : (int)lam[off + P];
    const u64 mask = band_mask(dP + 1, (int)lam[off + u], (int)m.T);
    contrib[off + u] = mask ? (draw[off + minv[off + u]] & mask) : 0;
}

__global__ void __launch_bounds__(NUS_THREADS) nus_walk_kernel(NusDims m, const u32 *__restrict__ val,
                                                               const unsigned char *__restrict__ lam,
                                                               const u32 *__restrict__ pleaf,
                                                               const u32 *__restrict__ pint,
                                                               const u64 *__restrict__ contrib,
                                                               const u64 *__restrict__ draw, u64 *__restrict__ shv,
                                                               unsigned int *err)
{
    const u32 p = blockIdx.x * NUS_THREADS + threadIdx.x, g = blockIdx.y;
    if (p >= m.N) return;
    const u64 off = (u64)g * m.NP;
    const u32 v = val[off + p];
    if (v < m.H0) return;  // the phantom and earlier calls' points are not output
    const u32 P = pleaf[off + p];
    const int dP = P == NONE ? -1 : (int)lam[off + P];
    u64 sh = draw[off + v] & band_mask(dP + 1, (int)m.T - 1, (int)m.T);
    int hop = 0;
    for (u32 u = P; u != NONE; u = pint[off + u]) {
        if (++hop > MAX_DEPTH) {
            atomicOr(err, 16u);
            break;
        }
        sh |= contrib[off + u];
    }
    shv[off + v] = sh;
}

// ---- 6. output, transposed back to (r, n, d) --------------------------------------

__global__ void nus_out_kernel(NusDims m, const u64 *__restrict__ xb, const u64 *__restrict__ shv,
                               u64 *__restrict__ xrb)
{
    __shared__ u64 tile[32][33];
    const u32 i0 = blockIdx.x * 32, g0 = blockIdx.y * 32;
    for (u32 k = threadIdx.y; k < 32; k += 8) {  // lanes along points
        const u32 g = g0 + k, i = i0 + threadIdx.x;
        tile[k][threadIdx.x] = (g < m.S && i < m.n) ? shv[(u64)g * m.NP + m.H0 + i] : 0;
    }
    __syncthreads();
    for (u32 k = threadIdx.y; k < 32; k += 8) {  // lanes along generators
        const u32 g = g0 + threadIdx.x, i = i0 + k;
        if (g < m.S && i < m.n) {
            const u64 s = m.s0 + g, l = s / m.d, j = s - l * m.d;
            const u64 w = xb[((l % m.r_x) * m.n + i) * m.d + j];
            xrb[(l * m.n + i) * m.d + j] = (m.td >= 64 ? 0 : w << m.td) ^ tile[threadIdx.x][k];
        }
    }
}

// ---- workspace -------------------------------------------------------------------

inline u64 al256(u64 b) { return (b + 255) & ~255ull; }

struct NusWork {
    u64 *keyA, *keyB, *draw, *shv;
    u32 *valA, *valB, *cnt, *pleaf, *pint, *ctl;
    unsigned long long *slot;
    unsigned char *lam, *Lv;
    u64 bytes;
};

// sub-arrays for `count` generators of N entries (stride NP), 256-byte aligned
NusWork nus_layout(char *base, u64 count, u64 NP, u64 NT)
{
    NusWork w{};
    u64 off = 0;
    auto take = [&](u64 bytes) {
        char *p = base ? base + off : nullptr;
        off += al256(bytes);
        return p;
    };
    const u64 e = count * NP;
    w.keyA = (u64 *)take(e * 8);
    w.keyB = (u64 *)take(e * 8);
    w.draw = (u64 *)take(e * 8);
    w.shv = (u64 *)take(e * 8);
    w.valA = (u32 *)take(e * 4);
    w.valB = (u32 *)take(e * 4);
    w.pleaf = (u32 *)take(e * 4);
    w.pint = (u32 *)take(e * 4);
    w.slot = (unsigned long long *)take(e * 8);
    w.cnt = (u32 *)take(count * 256 * NT * 4);
    w.lam = (unsigned char *)take(e);
    w.Lv = (unsigned char *)take(e);
    w.ctl = (u32 *)take(256);
    w.bytes = off;
    return w;
}

u64 entries_of(u64 n, u64 h0) { return (h0 ? h0 : 1) + n; }
u64 padded(u64 N) { return (N + 15) & ~15ull; }
u64 tiles_of(u64 N) { return (N + WT - 1) / WT; }

}  // namespace

extern "C" {

int qmc_dnb2_nus_workspace_size(uint64_t n, uint64_t h0, uint64_t generators, uint64_t *bytes)
{
    QMC_REQUIRE(bytes, "dnb2_nus_workspace_size: null output pointer");
    const u64 N = entries_of(n, h0);
    QMC_REQUIRE(N < MAX_ENTRIES, "dnb2_nested_uniform_scramble: %llu points and earlier entries per generator "
                "(at most 2^30 - 1)", (unsigned long long)N);
    *bytes = nus_layout(nullptr, generators ? generators : 1, padded(N), tiles_of(N)).bytes;
    return QMC_OK;
}

int qmc_dnb2_nested_uniform_scramble(uint64_t r, uint64_t n, uint64_t d, uint64_t r_x, uint64_t tmax,
                                     uint64_t tmax_new, uint64_t *states, uint64_t h0, const uint64_t *hist_keys,
                                     const uint64_t *hist_draws, const uint64_t *xb, uint64_t *xrb,
                                     uint64_t *keys_out, uint64_t *draws_out, void *work, uint64_t work_bytes,
                                     qmc_stream_t s)
{
    if (r == 0 || d == 0) return QMC_OK;
    QMC_REQUIRE_DOMAIN(tmax_new <= 64, "dnb2_nested_uniform_scramble: tmax_new = %llu (t must be between 0 and 64)",
                       (unsigned long long)tmax_new);
    QMC_REQUIRE(r_x >= 1, "dnb2_nested_uniform_scramble: r_x = 0");
    QMC_REQUIRE(states && work, "dnb2_nested_uniform_scramble: null states or workspace");
    QMC_REQUIRE(n == 0 || (xb && xrb), "dnb2_nested_uniform_scramble: null xb or xrb");
    QMC_REQUIRE(h0 == 0 || (hist_keys && hist_draws), "dnb2_nested_uniform_scramble: null history arrays");
    QMC_REQUIRE(((uintptr_t)work & 255) == 0, "dnb2_nested_uniform_scramble: workspace not 256-byte aligned");
    const u64 N = entries_of(n, h0);
    QMC_REQUIRE(N < MAX_ENTRIES, "dnb2_nested_uniform_scramble: %llu points and earlier entries per generator "
                "(at most 2^30 - 1)", (unsigned long long)N);
    const u64 NP = padded(N), NT = tiles_of(N), G = r * d;
    const u64 per = nus_layout(nullptr, 1, NP, NT).bytes;
    QMC_REQUIRE(work_bytes >= per, "dnb2_nested_uniform_scramble: workspace of %llu bytes, one generator needs %llu",
                (unsigned long long)work_bytes, (unsigned long long)per);
    // the most generators whose sub-arrays fit; work_bytes / per alone comes out one short for
    // a workspace sized for exactly that many, as the fixed words count once in any layout
    const u64 cap = G < 65535 ? G : 65535;
    u64 count = work_bytes / per;
    if (count > cap) count = cap;
    while (count < cap && nus_layout(nullptr, count + 1, NP, NT).bytes <= work_bytes) count++;
    while (count > 1 && nus_layout(nullptr, count, NP, NT).bytes > work_bytes) count--;
    NusWork w = nus_layout((char *)work, count, NP, NT);
    cudaStream_t st = QMC_STREAM(s);
    const u64 *xb_ = (const u64 *)xb, *hk_ = (const u64 *)hist_keys, *hd_ = (const u64 *)hist_draws;
    u64 *xrb_ = (u64 *)xrb, *ko_ = (u64 *)keys_out, *do_ = (u64 *)draws_out, *st_ = (u64 *)states;

    NusDims m{};
    m.n = n;
    m.d = d;
    m.r_x = r_x;
    m.td = tmax_new - tmax;  // wraps when tmax > tmax_new: numpy shifts by >= 64 give 0
    m.T = (u32)tmax_new;
    m.mask = tmax_new >= 64 ? ~0ull : ((1ull << tmax_new) - 1);
    m.h0 = h0;
    m.fresh = h0 == 0;
    m.N = (u32)N;
    m.NP = (u32)NP;
    m.H0 = (u32)(h0 ? h0 : 1);
    m.NT = (u32)NT;
    const u32 passes = m.T ? (m.T + 7) / 8 : 1;
    unsigned int *err = qmcgb::device_error_ptr();
    QMC_REQUIRE(err, "device error word unavailable");

    for (u64 s0 = 0; s0 < G; s0 += count) {
        m.s0 = s0;
        m.S = (u32)(G - s0 < count ? G - s0 : count);
        const u64 e = (u64)m.S * NP;
        nus_keys_kernel<<<dim3((unsigned)((N + 31) / 32), (m.S + 31) / 32), dim3(32, 8), 0, st>>>(
            m, xb_, hk_, hd_, w.keyA, w.draw, ko_);
        int rc = qmcgb::launch_status("dnb2_nus keys");
        if (rc) return rc;
        const u32 *vfin = nullptr;
        const u64 *kfin = nullptr;
        u64 *kfree = nullptr;
        u32 *vfree = nullptr;
        if (n > 0) {
            const dim3 tg((unsigned)((NT + NUS_WARPS - 1) / NUS_WARPS), m.S);
            if (int rc2 = qmcgb::raise_smem_limit((const void *)nus_scatter_kernel, NUS_SCATTER_SMEM, "dnb2_nus sort"))
                return rc2;
            auto pass = [&](const u64 *kin, const u32 *vin, u32 digit, u64 *kout, u32 *vout) {
                nus_hist_kernel<<<tg, NUS_THREADS, 0, st>>>(m, kin, 8 * digit, w.cnt);
                nus_scan_kernel<<<m.S, 1024, 0, st>>>(m, w.cnt);
                nus_scatter_kernel<<<tg, NUS_THREADS, NUS_SCATTER_SMEM, st>>>(m, kin, vin, 8 * digit, w.cnt, kout, vout);
                return qmcgb::launch_status("dnb2_nus sort");
            };
            // the top digits only: enough for keys that differ in their
            // first log2(N) + 4 bits, finished by the run fixup
            const u32 need_bits = (u32)(64 - __builtin_clzll((unsigned long long)(N - 1) | 1ull)) + 4;
            const u32 top = passes < (need_bits + 7) / 8 ? passes : (need_bits + 7) / 8;
            const u64 *kin = w.keyA;
            const u32 *vin = nullptr;
            for (u32 q = 0; q < top; q++) {
                u64 *kout = (q & 1) ? w.keyA : w.keyB;
                u32 *vout = (q & 1) ? w.valA : w.valB;
                rc = pass(kin, vin, passes - top + q, kout, vout);
                if (rc) return rc;
                kin = kout;
                vin = vout;
            }
            u64 *kf = (top & 1) ? w.keyB : w.keyA, *ko = (top & 1) ? w.keyA : w.keyB;
            u32 *vf = (top & 1) ? w.valB : w.valA, *vo = (top & 1) ? w.valA : w.valB;
            if (top < passes) {
                const dim3 ng((unsigned)((N + NUS_THREADS - 1) / NUS_THREADS), m.S);
                rc = qmcgb::cuda_status(cudaMemsetAsync(w.ctl, 0, 4, st), "dnb2_nus run flag");
                if (rc) return rc;
                nus_fixup_kernel<<<ng, NUS_THREADS, 0, st>>>(m, 8 * (passes - top), kf, vf, w.ctl);
                u32 longrun = 0;
                rc = qmcgb::cuda_status(cudaMemcpyAsync(&longrun, w.ctl, 4, cudaMemcpyDeviceToHost, st),
                                        "dnb2_nus run flag");
                if (rc) return rc;
                rc = qmcgb::cuda_status(cudaStreamSynchronize(st), "dnb2_nus run flag");
                if (rc) return rc;
                if (longrun) {  // every digit, from point order, ending in kf / vf
                    nus_unsort_kernel<<<ng, NUS_THREADS, 0, st>>>(m, kf, vf, w.shv);
                    const u64 *ki = w.shv;
                    const u32 *vi = nullptr;
                    for (u32 q = 0; q < passes; q++) {
                        const bool to_f = ((passes - 1 - q) & 1) == 0;
                        rc = pass(ki, vi, q, to_f ? kf : ko, to_f ? vf : vo);
                        if (rc) return rc;
                        ki = to_f ? kf : ko;
                        vi = to_f ? vf : vo;
                    }
                }
            }
            kfin = kf;
            vfin = vf;
            kfree = ko;
            vfree = vo;
            const dim3 ng((unsigned)((N + NUS_THREADS - 1) / NUS_THREADS), m.S);
            nus_lcp_kernel<<<ng, NUS_THREADS, 0, st>>>(m, kfin, vfin, w.lam);
            rc = qmcgb::cuda_status(cudaMemsetAsync(w.slot, 0xFF, e * 8, st), "dnb2_nus slots");
            if (rc) return rc;
            nus_build_kernel<<<ng, NUS_THREADS, 0, st>>>(m, vfin, w.lam, w.slot, w.pleaf, w.pint, vfree, w.Lv, err);
            rc = qmcgb::launch_status("dnb2_nus tree");
            if (rc) return rc;
        }
        // the counts and stream lengths in the sort's count array, the outputs in the array that the
        // scrambles take later
        const u32 dt = (m.N + DT - 1) / DT;
        DrawInfo *info = (DrawInfo *)w.cnt;
        DrawCount *counts = (DrawCount *)w.cnt + m.S;
        const dim3 dg((dt + 7) / 8, m.S);
        nus_draw_count_kernel<<<dg, 256, 0, st>>>(m, w.Lv, counts);
        nus_draw_scan_kernel<<<m.S, 32, 0, st>>>(m, st_, counts, info);
        nus_stream_kernel<<<(m.S + 31) / 32, 128, 0, st>>>(m, st_, info, w.shv);
        nus_draw_kernel<<<dg, 256, 0, st>>>(m, w.Lv, counts, info, w.shv, st_, w.draw);
        rc = qmcgb::launch_status("dnb2_nus draws");
        if (rc) return rc;
        if (draws_out) {
            rc = qmcgb::cuda_status(cudaMemcpy2DAsync(do_ + s0 * N, N * 8, w.draw, NP * 8, N * 8, m.S,
                                                      cudaMemcpyDeviceToDevice, st),
                                    "dnb2_nus draws out");
            if (rc) return rc;
        }
        if (n > 0) {
            const dim3 ng((unsigned)((N + NUS_THREADS - 1) / NUS_THREADS), m.S);
            u64 *contrib = kfree;
            nus_contrib_kernel<<<ng, NUS_THREADS, 0, st>>>(m, w.lam, w.pint, vfree, w.draw, contrib);
            nus_walk_kernel<<<ng, NUS_THREADS, 0, st>>>(m, vfin, w.lam, w.pleaf, w.pint, contrib, w.draw, w.shv, err);
            nus_out_kernel<<<dim3((unsigned)((n + 31) / 32), (m.S + 31) / 32), dim3(32, 8), 0, st>>>(m, xb_, w.shv, xrb_);
            rc = qmcgb::launch_status("dnb2_nus scramble");
            if (rc) return rc;
        }
    }
    return QMC_OK;
}

}  // extern "C"
