// Kernel A for bf16 gradients, second form: a warp owns a contiguous run of the tile from load to codes.
//
// A bf16 tile (29 056 values, 58 KB) and 15 KB of selection scratch sit in shared memory; three CTAs of 256 threads fit an
// SM.  The tile is cut into slots of 512 elements (a multiple of every aligned quant_block_size), and each of the eight
// warps owns seven or eight consecutive slots: the copy engine brings their gradient while the code words of the first ones
// travel into registers, and the warp decodes a = bf16(g + Qinv(e)) in place, lists the 16-element units that reach a bound
// carried over from the tile before, and later writes statistics and codes of its own blocks and asks for the next tile's
// gradient, without waiting for the other warps.  Only two things cross warps, and they cost the tile's only two barriers: the
// histogram that gives the k-th magnitude, and the number of selected values in the warps before, from which every selected value
// has its place in the ascending I / V row.
//
// Shared memory holds a with the eight octets of every 128-byte row permuted by the row number (octet o sits at
// o ^ ((o >> 3) & 7)): the decode writes two neighbouring octets per lane, the encode reads whole blocks per lane, both
// without bank conflicts.
//
// Selection: the values that reach the bound (a bf16 magnitude, `guess`) are counted in a histogram with one bin per bf16
// magnitude above it, so the bin of the k-th value is the k-th magnitude itself; among equal ones the lower positions win,
// and the units of a warp are listed in ascending order, so ranks and ties are prefix counts.  The next tile's bound lies
// a few magnitudes below this tile's k-th value.  A bound that was too high (fewer than k values reach it) is found anew from
// the histogram of the octet maxima; tiles that defeat this as well (fewer than k values that are not zero, k beyond the octets)
// fall back to a bisection on the key bits.
//
// Bound by instruction issue (25 instructions per element at 1965 MHz, 62 % of the cycles issue, the ALU pipe 54 % busy): the codec's half
// of them runs at the rate of the integer and FMA pipes, the rest is the selection and what every warp does once a tile.  us a
// launch, and the form for launches of fewer than ten tiles per SM: 215 M elements 255 (295), 133 M 165 (188), 43 M 63 (72), 12.9 M 20.3 (20.0).  Against a form of
// that design for all block sizes, with the quotient it had: blocks of 32, 29 M 53 (89), of 128 with k = 5 % 70 (113); loose blocks,
// 215 M 291 (331).  More registers than 80 a thread would cost the third CTA, and what the compiler spills costs more than it seems: 92
// bytes in the inner loops cost 20 us at 218 M.
//
// Results are bit-identical to those of the fp32 kernels' arithmetic (ef_topk_quant_f32.cu, ef_topk_quant.cu; same tie rule).
#include "common.cuh"
#include "select.cuh"
#include "codec_fast.cuh"
#include "async_copy.cuh"
#include "fused.cuh"

namespace mab {
namespace warps {

constexpr int S_WARPS = 8;
constexpr int S_NT = S_WARPS * 32;
constexpr int S_CTAS = 3;                    // resident CTAs per SM the shared memory and the registers are sized for
constexpr int S_SLOT = 512;                  // elements per slot: a unit of 16 per lane
constexpr int S_MAX_SLOTS = (SEL_MAX_TILE / S_SLOT + S_WARPS - 1) / S_WARPS;   // slots of a warp
constexpr int S_RING = 2;                    // slots whose code words are in flight
constexpr int S_UNITS = S_MAX_SLOTS * 32;    // 16-element units of a warp
constexpr int S_TABS = S_MAX_SLOTS / 4;
constexpr int S_QTAB = 32 * S_TABS;          // quantisation blocks of a warp whose constants are kept in a table: all with
                                             // 64 elements or more, loose ones (72 or more) included
constexpr int S_CAND = 4 * S_QTAB + 32;      // candidates a warp lists: k = 5 % of a tile has some 220
constexpr int S_BINS = 128;                  // bf16 magnitudes above the bound that are told apart: one octave
constexpr int S_WPT = SEL_WORDS / S_NT;      // bitmap words per thread of the bisection
static_assert(SEL_WORDS % S_NT == 0 && S_MAX_SLOTS % 4 == 0 && S_BINS <= S_NT, "whole shares");
static_assert(S_MAX_SLOTS * S_SLOT / 72 + 2 <= S_QTAB, "loose blocks a warp touches");

// Set when a wait on the copy engine gave up; read through mab_device_error() together with the other kernels' flags.
__device__ int g_copy_timeout;

// What a tile needs of its tensor's descriptor; filled in by one lane while the tile before is worked on.
struct TileInfo {
    uint16_t* g;                 // gradient (only loose tiles are written: the residual)
    uint8_t*  ef;
    uint16_t* mn;
    uint16_t* mx;
    int16_t*  i_out;
    uint16_t* v_out;
    uint16_t* qe;                // alpha == -2: where the residual goes
    int64_t   qb_at;             // loose: first touched block in the scratch arrays
    int n, k, ti, lrem0;         // lrem0: loose: where the tile starts inside its first block
};

struct __align__(16) SmemSel {
    union {
        struct {                                 // per warp:
            struct {
                uint16_t list[S_UNITS];          //   units that reach the bound, ascending
                union {                          //   in turn:
                float4   mu[S_QTAB];             //     (min, min, u, u) of its quantisation blocks
                uint32_t cand[S_CAND];           //     values that reach the bound, ascending positions: value << 16 | position
                uint32_t ext[2][S_QTAB];         //     extremes of the loose blocks it touches
                };
            } w[S_WARPS];
        };
        struct {                                 // bisection
            uint32_t sel_bm[SEL_WORDS];          // selected positions
            uint16_t sel_before[SEL_WORDS];      // selected positions in lower words
        };
    };
    int      hist[2][S_BINS];                    // of this tile and the next one, like counts
    uint32_t counts[2][S_WARPS];                 // values of a warp above | (at the k-th magnitude) << 16
    int      cold_hist[256];                     // of the octet maxima
    int      kmax[2];
    TileInfo info[3];                            // of the tiles before, now and next
    int      counters[40];
    int      scan[36];
};

// Where element `pos` of the tile sits.
__device__ __forceinline__ int phys_oct(int o) { return o ^ ((o >> 3) & 7); }
__device__ __forceinline__ int phys_pos(int pos) { return (phys_oct(pos >> 3) << 3) | (pos & 7); }

__device__ __forceinline__ void unpack8(const uint4& a, float (&v)[8]) {
    v[0] = __uint_as_float(a.x << 16); v[1] = __uint_as_float(a.x & 0xFFFF0000u);
    v[2] = __uint_as_float(a.y << 16); v[3] = __uint_as_float(a.y & 0xFFFF0000u);
    v[4] = __uint_as_float(a.z << 16); v[5] = __uint_as_float(a.z & 0xFFFF0000u);
    v[6] = __uint_as_float(a.w << 16); v[7] = __uint_as_float(a.w & 0xFFFF0000u);
}

// 0xFFFF in every half whose |value| reaches the bound (a NaN reaches none).
__device__ __forceinline__ uint32_t reach_mask(uint32_t w, uint32_t bound2) {
    uint32_t d;
    asm("set.ge.u32.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(w & 0x7FFF7FFFu), "r"(bound2));
    return d;
}

// The values of unit u (16 elements) that reach the bound, as bits.
__device__ __forceinline__ uint32_t unit_mask(const uint4* tile4, int u, uint32_t bound2) {
    const int at = phys_oct(2 * u);
    const uint4 a = tile4[at], b = tile4[at ^ 1];
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t m = 0u;                                         // even elements in the low half, odd ones in the high half
#pragma unroll
    for (int p = 0; p < 8; ++p) m |= reach_mask(w[p], bound2) & (0x00020001u << (2 * p));
    return (m | (m >> 16)) & 0xFFFFu;
}

// Slots [s0, s0 + ns) of the tile belong to this warp.  Which warps take one more than the others changes from CTA to CTA
// (`rot`), so that the schedulers of an SM get the same share.
struct Segment { int s0, ns; };
__device__ __forceinline__ Segment warp_segment(int n, int rot, int warp) {
    const int slots = (n + S_SLOT - 1) / S_SLOT, q = slots / S_WARPS, rem = slots % S_WARPS;
    uint32_t more = (1u << rem) - 1u;
    more = ((more << rot) | (more >> (S_WARPS - rot))) & ((1u << S_WARPS) - 1u);
    Segment s;
    s.s0 = warp * q + __popc(more & ((1u << warp) - 1u));
    s.ns = q + (int)((more >> warp) & 1u);
    return s;
}

// ---------------------------------------------------------------------------------------------- bisection route
// Number of tile elements with key >= thr (key bits), every thread of the CTA calling.
__device__ __forceinline__ int tile_count_ge(const uint4* tile4, int n_oct, int thr, int* counter) {
    const float thr_f = __int_as_float(thr);
    int c = 0;
    for (int o = threadIdx.x; o < n_oct; o += S_NT) {
        float v[8];
        unpack8(tile4[phys_oct(o)], v);
#pragma unroll
        for (int e = 0; e < 8; ++e) c += (fabsf(v[e]) >= thr_f) ? 1 : 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane_id() == 0 && c) atomicAdd(counter, c);
    __syncthreads();
    return *reinterpret_cast<volatile int*>(counter);
}

// sel_bm = gt | (the need_ties lowest positions of tie), sel_before = prefix popcount, from the
// thread's own four words of both masks.  Starts and ends with a barrier.
__device__ __forceinline__ void resolve_selection_regs(const uint32_t (&gt)[S_WPT], uint32_t (&tw)[S_WPT], int need_ties, SmemSel& ss) {
    __syncthreads();
    const int w0 = threadIdx.x * S_WPT;
    uint32_t sel[S_WPT];
    int total;
#pragma unroll
    for (int i = 0; i < S_WPT; ++i) sel[i] = gt[i];
    if (need_ties > 0) {
        int cnt = 0;
#pragma unroll
        for (int i = 0; i < S_WPT; ++i) cnt += __popc(tw[i]);
        int before = block_exclusive_scan(cnt, ss.scan, total);
#pragma unroll
        for (int i = 0; i < S_WPT; ++i) {
            const int keep = need_ties - before;
            before += __popc(tw[i]);
            if (keep <= 0) tw[i] = 0;
            else while (__popc(tw[i]) > keep) tw[i] &= ~(0x80000000u >> __clz(tw[i]));
            sel[i] |= tw[i];
        }
        __syncthreads();
    }
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < S_WPT; ++i) cnt += __popc(sel[i]);
    int before = block_exclusive_scan(cnt, ss.scan, total);
#pragma unroll
    for (int i = 0; i < S_WPT; ++i) { ss.sel_bm[w0 + i] = sel[i]; ss.sel_before[w0 + i] = (uint16_t)before; before += __popc(sel[i]); }
    __syncthreads();
}

// The whole selection of a tile at a cost that does not depend on the data: bisection on the key bits (all_zero: every key
// is zero, the k lowest positions win the ties), row written, selected values zeroed.  The caller has met at a barrier; ends with one.
// In line: as a function of its own it read the tile through generic addresses (loose blocks, k = 20 %, 12.9 M elements: this kernel
// 95 us, in line 89), and the registers saved around the call were spilled.
__device__ __forceinline__ void select_by_bisection(uint16_t* tile, SmemSel& ss, int n, int k, bool all_zero, int16_t* i_out, uint16_t* v_out) {
    const uint4* tile4 = reinterpret_cast<const uint4*>(tile);
    const int t = threadIdx.x, n_oct = (n + 7) >> 3;
    uint32_t gt[S_WPT], tw[S_WPT];
    int need = 0;
    if (all_zero) {
#pragma unroll
        for (int i = 0; i < S_WPT; ++i) {
            const int lo = (t * S_WPT + i) * 32;
            gt[i] = (lo + 32 <= k) ? 0xFFFFFFFFu : (lo < k ? ((1u << (k - lo)) - 1u) : 0u);
            tw[i] = 0u;
        }
    } else {
        if (t < 40) ss.counters[t] = 0;
        __syncthreads();
        int Tk = 0;
        for (int bit = 30; bit >= 16; --bit) {               // bf16 keys have 16 zero bits below
            const int cand = Tk | (1 << bit);
            if (tile_count_ge(tile4, n_oct, cand, &ss.counters[bit]) >= k) Tk = cand;
        }
        need = k - tile_count_ge(tile4, n_oct, Tk + 0x10000, &ss.counters[32]);
        const float Tf = __int_as_float(Tk);
#pragma unroll
        for (int i = 0; i < S_WPT; ++i) {                    // the thread's 128 positions = 16 octets
            gt[i] = 0u; tw[i] = 0u;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int o = (t * S_WPT + i) * 4 + b;
                if (o < n_oct) {
                    float v[8];
                    unpack8(tile4[phys_oct(o)], v);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const bool valid = o * 8 + e < n;     // padding never competes, whatever the threshold
                        gt[i] |= (valid && fabsf(v[e]) > Tf) ? (1u << (8 * b + e)) : 0u;
                        tw[i] |= (valid && fabsf(v[e]) == Tf) ? (1u << (8 * b + e)) : 0u;
                    }
                }
            }
        }
    }
    resolve_selection_regs(gt, tw, need, ss);
    const int w0 = t * S_WPT;
    for (int i = 0; i < S_WPT; ++i) {
        uint32_t sel = ss.sel_bm[w0 + i];
        int p = ss.sel_before[w0 + i];
        while (sel) {
            const int b = __ffs(sel) - 1;
            sel &= sel - 1;
            const int q = (w0 + i) * 32 + b;
            const int at = phys_pos(q);
            i_out[p] = (int16_t)q;
            v_out[p++] = tile[at];
            tile[at] = 0;
        }
    }
    __syncthreads();
}

// A bound from the tile itself, and the warp's units that reach it: the histogram of the octet maxima over the eight octaves
// below the largest, in bins of 1/32 octave, gives the largest bound that at least k octets reach.  0: every value is zero; -1: no bound (fewer than k octets lie in that range).  Needs cold_hist and kmax at zero.
// A launch whose CTAs work on a tile or two each spends much of its time here: two barriers, one pass over the tile.
struct Bound { int bound, n_w; };
__device__ __forceinline__ Bound bound_from_octets(const uint4* tile4, SmemSel& ss, int p, uint16_t* list, int s0, int ns, int n, int k) {
    const int lane = lane_id(), n_unit = (n + 15) >> 4;
    uint32_t m2[S_MAX_SLOTS], top = 0u;                      // the maxima of a unit's two octets
#pragma unroll
    for (int s = 0; s < S_MAX_SLOTS; ++s) {
        const int u = (s0 + s) * 32 + lane;
        m2[s] = 0u;
        if (s < ns && u < n_unit) {
            const int at = phys_oct(2 * u);
            const uint4 v = tile4[at], w = tile4[at ^ 1];
            const uint32_t x = maxabs_bf16x2(maxabs_bf16x2(v.x, v.y), maxabs_bf16x2(v.z, v.w));
            const uint32_t y = maxabs_bf16x2(maxabs_bf16x2(w.x, w.y), maxabs_bf16x2(w.z, w.w));
            m2[s] = max_bf16x2(maxabs_bf16x2(__byte_perm(x, y, 0x5410), __byte_perm(x, y, 0x7632)) & 0x7FFF7FFFu, 0u);   // (nothing but NaN: 0)
            top = max_bf16x2(top, m2[s]);
        }
    }
    top = __reduce_max_sync(0xffffffffu, max(top & 0xFFFFu, top >> 16));
    if (lane == 0 && top) atomicMax(&ss.kmax[p], (int)top);
    __syncthreads();
    const int kmax = ss.kmax[p];
    if (kmax == 0) return {0, 0};
#pragma unroll
    for (int s = 0; s < S_MAX_SLOTS; ++s) {
        const int a = (int)(m2[s] & 0xFFFFu), b = (int)(m2[s] >> 16);
        if (a > 0 && kmax - a < (256 << 2)) atomicAdd(&ss.cold_hist[(kmax - a) >> 2], 1);
        if (b > 0 && kmax - b < (256 << 2)) atomicAdd(&ss.cold_hist[(kmax - b) >> 2], 1);
    }
    __syncthreads();
    int h[8], sum = 0;
    {
        const int4 ha = reinterpret_cast<const int4*>(ss.cold_hist)[lane * 2], hb = reinterpret_cast<const int4*>(ss.cold_hist)[lane * 2 + 1];
        h[0] = ha.x; h[1] = ha.y; h[2] = ha.z; h[3] = ha.w; h[4] = hb.x; h[5] = hb.y; h[6] = hb.z; h[7] = hb.w;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) sum += h[i];
    int upto = sum;                                          // maxima in the bins of lanes <= this one
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const int v = __shfl_up_sync(0xffffffffu, upto, d); if (lane >= d) upto += v; }
    const unsigned ok = __ballot_sync(0xffffffffu, upto >= k);
    if (ok == 0u) return {-1, 0};
    const int owner = __ffs(ok) - 1;
    int c = upto - sum, bin = 0;
    bool found = false;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if (!found) { c += h[i]; bin = i; found = c >= k; }
    bin = __shfl_sync(0xffffffffu, bin, owner) + owner * 8;
    const int bound = max(1, kmax - (bin << 2) - 3);
    int n_w = 0;
#pragma unroll
    for (int s = 0; s < S_MAX_SLOTS; ++s) {
        const bool hit = max((int)(m2[s] & 0xFFFFu), (int)(m2[s] >> 16)) >= bound;
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        if (hit) list[n_w + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)((s0 + s) * 32 + lane);
        n_w += __popc(bal);
    }
    __syncwarp();
    return {bound, n_w};
}

// The warp's units with a value that reaches the bound, listed anew.
__device__ __noinline__ int relist(const uint4* tile4, uint16_t* list, int s0, int ns, int n, uint32_t bound2) {
    const int lane = lane_id(), n_unit = (n + 15) >> 4;
    int n_w = 0;
    for (int s = s0; s < s0 + ns; ++s) {
        const int u = s * 32 + lane;
        const bool hit = u < n_unit && unit_mask(tile4, u, bound2) != 0u;
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        if (hit) list[n_w + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)u;
        n_w += __popc(bal);
    }
    __syncwarp();
    return n_w;
}

// Exclusive prefix over the lanes' numbers of bits.  All 32 lanes call.
__device__ __forceinline__ int mask_prefix(uint32_t m, int& total) {
    const int cnt = __popc(m);
    int inc = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const int v = __shfl_up_sync(0xffffffffu, inc, d); if (lane_id() >= d) inc += v; }
    total = __shfl_sync(0xffffffffu, inc, 31);
    return inc - cnt;
}

// Row entries and zeros of a warp whose values did not fit the list: straight from its units.  `ties`: values equal to the
// k-th magnitude in the warps before, `rank`: the warp's first place in the row.
__device__ __noinline__ void select_from_units(uint16_t* tile, const uint16_t* list, int n_w, int kth, int need, int ties, int rank, int16_t* i_out,
                                               uint16_t* v_out) {
    const uint4* tile4 = reinterpret_cast<const uint4*>(tile);
    const int lane = lane_id();
    for (int q0 = 0; q0 < n_w; q0 += 32) {
        uint32_t gt = 0u, eq = 0u;
        int u = 0;
        if (q0 + lane < n_w) {
            u = list[q0 + lane];
            gt = unit_mask(tile4, u, (uint32_t)(kth + 1) * 0x10001u); eq = unit_mask(tile4, u, (uint32_t)kth * 0x10001u) ^ gt;
        }
        int total;
        const int keep = max(0, need - ties - mask_prefix(eq, total));   // the lowest positions among the equal ones
        ties += total;
        while (__popc(eq) > keep) eq &= ~(0x80000000u >> __clz(eq));
        uint32_t sel = gt | eq;
        int to = rank + mask_prefix(sel, total);
        rank += total;
        for (; sel; sel &= sel - 1, ++to) {
            const int pos = u * 16 + __ffs(sel) - 1, where = phys_pos(pos);
            i_out[to] = (int16_t)pos;
            v_out[to] = tile[where];
            tile[where] = 0;
        }
    }
}

// ---------------------------------------------------------------------------------------------- loads
// 8 bf16 values from any address: both aligned 16-byte pieces that hold some of them must be readable.
__device__ __forceinline__ uint4 load_octet_anywhere(const uint16_t* p) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    const uint4* piece = reinterpret_cast<const uint4*>(at & ~(uintptr_t)15);
    const uint4 x = __ldg(piece), y = (at & 15) ? __ldg(piece + 1) : make_uint4(0u, 0u, 0u, 0u);
    uint32_t w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    if (at & 8) { w[0] = w[2]; w[1] = w[3]; w[2] = w[4]; w[3] = w[5]; w[4] = w[6]; w[5] = w[7]; }
    if (at & 4) { w[0] = w[1]; w[1] = w[2]; w[2] = w[3]; w[3] = w[4]; w[4] = w[5]; }
    const int sh = (int)(at & 2) * 8;
    return make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh), __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
}

// The whole octets [o, o1) of a gradient that is not 16-byte aligned into their places in the tile, in order and not permuted
// (a slot's octets stay within its own eight rows, so the decode of a slot can permute them in place): from the two aligned
// pieces they lie in, but for the tile's first and last two octets, whose pieces may reach out of the buffer.
__device__ __noinline__ void stage_anywhere(uint16_t* tile, const uint16_t* g, int o, int o1, int n_oct) {
    auto edge = [&](int i) { return i == 0 || i >= n_oct - 2; };
#pragma unroll 1
    for (; o < o1; o += 4 * 32) {                            // four octets' loads in flight
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int at = o + i * 32;
            if (at < o1 && !edge(at)) v[i] = load_octet_anywhere(g + at * 8);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int at = o + i * 32;
            if (at >= o1) continue;
            if (!edge(at)) reinterpret_cast<uint4*>(tile)[at] = v[i];
            else for (int e = 0; e < 8; ++e) tile[at * 8 + e] = g[at * 8 + e];
        }
    }
}

__device__ __forceinline__ void store_code_word(uint8_t* ef_g, bool aligned4, int o, int n, uint32_t w) {
    if (aligned4 && o * 8 + 8 <= n) { reinterpret_cast<uint32_t*>(ef_g)[o] = w; return; }
    for (int b = 0; b < 4; ++b) if (o * 8 + 2 * b < n) ef_g[o * 4 + b] = (uint8_t)(w >> (8 * b));
}

// 8 bytes, if `on`.
__device__ __forceinline__ void ld_global_8(const void* p, bool on, uint2& a) {
    asm volatile("{.reg .pred q; setp.ne.b32 q, %3, 0; @q ld.global.v2.b32 {%0,%1}, [%2];}" : "+r"(a.x), "+r"(a.y) : "l"(p), "r"((int)on));
}
// 32 bytes in one access (sm_100).
__device__ __forceinline__ void st_global_32(void* p, const uint32_t* w) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}

// N code words of one quantisation block; `al`: what the address is aligned to (at most 32).
template <int N>
__device__ __forceinline__ void store_codes(uint8_t* dst, const uint32_t (&w)[N], int al) {
    if (N >= 8 && al >= 32) {
#pragma unroll
        for (int i = 0; i < N / 8; ++i) st_global_32(dst + 32 * i, w + 8 * i);
    } else if (N >= 4 && al >= 16) {
#pragma unroll
        for (int i = 0; i < N / 4; ++i) reinterpret_cast<uint4*>(dst)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
    } else if (al >= 4) {
#pragma unroll
        for (int i = 0; i < N; ++i) reinterpret_cast<uint32_t*>(dst)[i] = w[i];
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
            for (int b = 0; b < 4; ++b) dst[4 * i + b] = (uint8_t)(w[i] >> (8 * b));
    }
}

// ---------------------------------------------------------------------------------------------- decode
// Both halves of a packed instruction work on elements of one kind, even (high nibbles, low bf16 halves) or odd, so that its
// constants are pairs of equal values: with (even, odd) pairs the compiler spends seven more instructions an octet.
struct Pairs { float2 a, b, c, d; };                         // elements (0, 2), (1, 3), (4, 6), (5, 7) of an octet
__device__ __forceinline__ Pairs unpack_pairs(const uint4& v) {
    Pairs p;
    p.a = make_float2(__uint_as_float(v.x << 16), __uint_as_float(v.y << 16));
    p.b = make_float2(__uint_as_float(v.x & 0xFFFF0000u), __uint_as_float(v.y & 0xFFFF0000u));
    p.c = make_float2(__uint_as_float(v.z << 16), __uint_as_float(v.w << 16));
    p.d = make_float2(__uint_as_float(v.z & 0xFFFF0000u), __uint_as_float(v.w & 0xFFFF0000u));
    return p;
}

// Qinv(code) = RN(RN(code * u) + mn) as in decode_octet_fast, with the high nibbles left where they are: 2^23 + 16 code times
// u / 16 is the same product.  Needs a u that is zero or at least 2^-100 (u / 16 exact) and below 2^100.
struct UnitConsts { float2 ue, uo, ne, no, mn; };
__device__ __forceinline__ UnitConsts unit_consts(const float4& mu) {   // (mn, mn, u, u)
    const float2 u = make_float2(mu.z, mu.w);
    UnitConsts c;
    c.uo = u;
    c.ue = __fmul2_rn(u, make_float2(0.0625f, 0.0625f));
    c.ne = __fmul2_rn(u, make_float2(-524288.0f, -524288.0f));
    c.no = __fmul2_rn(u, make_float2(-8388608.0f, -8388608.0f));
    c.mn = make_float2(mu.x, mu.y);
    return c;
}

// A block's decode constants from the bits of its statistics as floats, as qparams() gives them where max - min is zero or in
// [2^-96, 2^100]; `slow` is raised elsewhere.
__device__ __forceinline__ QParams block_params(uint32_t mn_bits, uint32_t mx_bits, bool& slow) {
    QParams q;
    q.mn = __uint_as_float(mn_bits);
    const float d = __fsub_rn(__uint_as_float(mx_bits), q.mn), c = 0.0666666701436042785644531f;   // RN(1 / 15): see div15_rn
    const float p = __fmul_rn(d, c);
    q.u = __fmaf_rn(__fmaf_rn(-15.0f, p, d), c, p);
    slow |= !(d == 0.0f || (d >= 1.2621774e-29f && d <= CODEC_U_MAX));
    return q;
}

// a = bf16(g + Qinv(e)) of one octet.
__device__ __forceinline__ uint4 decode_add(const uint4& g, uint32_t codes, const UnitConsts& c) {
    const uint32_t hi = codes & 0xF0F0F0F0u, lo = codes & 0x0F0F0F0Fu;
    const Pairs p = unpack_pairs(g);
    const float2 a = __fadd2_rn(__fadd2_rn(__ffma2_rn(make_float2(magic_byte<0>(hi), magic_byte<1>(hi)), c.ue, c.ne), c.mn), p.a);
    const float2 b = __fadd2_rn(__fadd2_rn(__ffma2_rn(make_float2(magic_byte<0>(lo), magic_byte<1>(lo)), c.uo, c.no), c.mn), p.b);
    const float2 d = __fadd2_rn(__fadd2_rn(__ffma2_rn(make_float2(magic_byte<2>(hi), magic_byte<3>(hi)), c.ue, c.ne), c.mn), p.c);
    const float2 e = __fadd2_rn(__fadd2_rn(__ffma2_rn(make_float2(magic_byte<2>(lo), magic_byte<3>(lo)), c.uo, c.no), c.mn), p.d);
    return make_uint4(pack_bf16x2_rne(a.x, b.x), pack_bf16x2_rne(a.y, b.y), pack_bf16x2_rne(d.x, e.x), pack_bf16x2_rne(d.y, e.y));
}

// One unit by the defining scalar form, elements from n on becoming 0: the tile's last, short unit, blocks whose step is
// subnormal, huge or no number, codes that are not on a word boundary.  qbs: of the tile's blocks, the first of which
// starts lrem0 elements before the tile.
__device__ __noinline__ void decode_unit_scalar(uint16_t* tile, const TileInfo& I, int u, int qbs) {
    for (int e = u * 16; e < u * 16 + 16; ++e) {
        uint16_t a = 0;
        if (e < I.n) {
            const int b = (I.lrem0 + e) / qbs;
            const QParams q = qparams(I.mn[b], I.mx[b]);
            const uint32_t code = (I.ef[e >> 1] >> ((e & 1) ? 0 : 4)) & 0xFu;
            a = f32_to_bf16_bits_rne(__fadd_rn(bf16_bits_to_f32(I.g[e]), qinv(code, q)));
        }
        tile[phys_pos(e)] = a;
    }
}

// ---------------------------------------------------------------------------------------------- encode
// Codes of one octet of bf16 values r (statistics = their exact block minimum and maximum, u in [2^-100, 2^100]): the defining
// form, two elements per instruction, the quotient as in encode_octet_div_f32 (codec_fast.cuh).
// floor: adding a power of two with rounding down leaves the integer in the mantissa; 2^23 for the odd elements puts it into
// bits 0-3, 2^19 for the even ones into bits 4-7, above four bits of fraction that the merge drops.
__device__ __forceinline__ uint32_t encode_octet_quotient(const uint4& v, const float2& nmn, const float2& r0, const float2& r1) {
    const float2 half2 = make_float2(0.5f, 0.5f), even2 = make_float2(524288.0f, 524288.0f), odd2 = make_float2(8388608.0f, 8388608.0f);
    auto floor_plus = [&](const float2& r, const float2& magic) {
        const float2 d = __fadd2_rn(r, nmn);                 // r - mn
        return __fadd2_rd(__fadd2_rn(__ffma2_rn(d, r0, __fmul2_rn(d, r1)), half2), magic);
    };
    auto merge = [](float e, float o) { return (__float_as_uint(e) & 0xF0u) | (__float_as_uint(o) & 0xFFFFFF0Fu); };
    const Pairs p = unpack_pairs(v);
    const float2 a = floor_plus(p.a, even2), b = floor_plus(p.b, odd2), c = floor_plus(p.c, even2), d = floor_plus(p.d, odd2);
    return __byte_perm(__byte_perm(merge(a.x, b.x), merge(a.y, b.y), 0x0040), __byte_perm(merge(c.x, d.x), merge(c.y, d.y), 0x0040), 0x5410);
}

// Codes of one block with the scalar form of the quantiser: the rare blocks that hold a NaN or whose step is zero (all
// values equal), subnormal or infinite.  Kept out of line so that the common path stays small.
__device__ __noinline__ void encode_block_exact(const uint4* tile4, int o0, int n_o, uint16_t mn_b, uint16_t mx_b, uint16_t* mn_out, uint8_t* dst, bool al4) {
    if ((mn_b & 0x7FFFu) > 0x7F80u) {                        // the statistics are those of the other values; the NaN's code is 0
        uint32_t lo2 = 0x7F807F80u;
        for (int c = 0; c < n_o; ++c) {
            const uint4 v = tile4[phys_oct(o0 + c)];
            lo2 = min_bf16x2(min_bf16x2(lo2, v.x), min_bf16x2(min_bf16x2(v.y, v.z), v.w));
        }
        mn_b = (uint16_t)min_bf16x2(lo2, lo2 >> 16 | lo2 << 16);
        *mn_out = mn_b;
    }
    const QParams q2 = qparams(mn_b, mx_b);
    for (int c = 0; c < n_o; ++c) {
        float r[8];
        unpack8(tile4[phys_oct(o0 + c)], r);
        store_code_word(dst, al4, c, n_o * 8, encode_octet_exact(r, q2, 8));
    }
}

// Statistics and codes of the whole quantisation blocks [b, b1) of 2^QS elements, a lane owning every 32nd.
template <int QS>
__device__ __forceinline__ void stats_encode(const uint4* tile4, int b, int b1, const TileInfo& I) {
    constexpr int CPQ = 1 << (QS - 3);                       // octets per block
    constexpr bool HOLD = CPQ <= 4;    // the block's values stay in registers between statistics and codes
                                                             // (those of 64 elements do not fit next to the rest)
    const uintptr_t ef_at = reinterpret_cast<uintptr_t>(I.ef);
    const int al = (int)min(ef_at & (~ef_at + 1), (uintptr_t)32);   // blocks are 4 CPQ bytes long: alignment beyond that is not used
    uint16_t* const mn_out = I.mn;
    uint16_t* const mx_out = I.mx;
    uint8_t* const ef = I.ef;
#pragma unroll 1
    for (; b < b1; b += 32) {
        const int o0 = b * CPQ;
        const uint4* row = tile4 + (o0 & ~7);
        const int key = ((o0 >> 3) & 7) ^ (o0 & 7);
        auto at = [&](int c) -> const uint4& { return CPQ <= 8 ? row[c ^ key] : tile4[phys_oct(o0 + c)]; };
        uint4 v[HOLD ? CPQ : 1];
        uint32_t hi2 = 0xFF80FF80u, lo2 = 0x7F807F80u;      // running packed max (from -inf) and min (from +inf)
#pragma unroll
        for (int c = 0; c < CPQ; ++c) {
            const uint4 x = at(c);
            if (HOLD) v[HOLD ? c : 0] = x;
            hi2 = max_bf16x2(max_bf16x2(hi2, x.x), max_bf16x2(max_bf16x2(x.y, x.z), x.w));
            lo2 = min_nan_bf16x2(min_nan_bf16x2(lo2, x.x), min_nan_bf16x2(min_nan_bf16x2(x.y, x.z), x.w));
        }
        hi2 = max_bf16x2(hi2, hi2 >> 16 | hi2 << 16);
        lo2 = min_nan_bf16x2(lo2, lo2 >> 16 | lo2 << 16);
        const uint16_t mn_b = (uint16_t)(lo2 & 0xFFFFu), mx_b = (uint16_t)(hi2 & 0xFFFFu);
        mn_out[b] = mn_b; mx_out[b] = mx_b;
        bool special = mn_b == mx_b;                          // all-equal block (u == 0), subnormal or infinite step, or a NaN in it
        const QParams q2 = block_params(lo2 << 16, hi2 << 16, special);
        uint8_t* dst = ef + b * (4 * CPQ);
        if (special || q2.u == 0.0f) {
            encode_block_exact(tile4, o0, CPQ, mn_b, mx_b, mn_out + b, dst, al >= 4);
            continue;
        }
        const float r0 = rcp_rn_normal(q2.u), r1 = rcp_rest(q2.u, r0);
        const float2 nmn = make_float2(-q2.mn, -q2.mn), r02 = make_float2(r0, r0), r12 = make_float2(r1, r1);
        uint32_t w[CPQ];
#pragma unroll
        for (int c = 0; c < CPQ; ++c) w[c] = encode_octet_quotient(HOLD ? v[HOLD ? c : 0] : at(c), nmn, r02, r12);
        store_codes<CPQ>(dst, w, al);
    }
}

// The tile's last, short block (elements [2^QS b, n)) by one warp, an octet per lane; all 32 call.
template <int QS>
__device__ __noinline__ void stats_encode_short(const uint4* tile4, int b, int n, const TileInfo& I) {
    constexpr int CPQ = 1 << (QS - 3);
    const int c = lane_id() & (CPQ - 1), o = b * CPQ + c;
    const int cnt = max(0, min(8, n - o * 8));
    const uint4 v = cnt > 0 ? tile4[phys_oct(o)] : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t hi2 = 0xFF80FF80u, lo2 = 0x7F807F80u;
    for (int e = 0; e < cnt; ++e) {
        const uint32_t x = (w[e >> 1] >> (16 * (e & 1))) & 0xFFFFu;
        hi2 = max_bf16x2(hi2, x | (x << 16));
        lo2 = min_bf16x2(lo2, x | (x << 16));
    }
#pragma unroll
    for (int d = 1; d < CPQ; d <<= 1) {
        hi2 = max_bf16x2(hi2, __shfl_xor_sync(0xffffffffu, hi2, d));
        lo2 = min_bf16x2(lo2, __shfl_xor_sync(0xffffffffu, lo2, d));
    }
    if (lane_id() >= CPQ || cnt == 0) return;
    const uint16_t mn_b = (uint16_t)(lo2 & 0xFFFFu), mx_b = (uint16_t)(hi2 & 0xFFFFu);
    if (c == 0) { I.mn[b] = mn_b; I.mx[b] = mx_b; }
    float r[8];
    unpack8(v, r);
    store_code_word(I.ef, (reinterpret_cast<uintptr_t>(I.ef) & 3) == 0, o, n, encode_octet_exact(r, qparams(mn_b, mx_b), cnt));
}

// Loose quantisation blocks: the residual of the warp's elements [e0, e1) goes back to the gradient buffer, and the extremes of
// the blocks they lie in, merged per warp first, to the scratch arrays.  All 32 lanes call.
__device__ __forceinline__ void residual_and_extremes(const uint16_t* tile, int e0, int e1, const TileInfo& I, const LooseArgs& la, uint32_t (&ext)[2][S_QTAB]) {
    const uint4* tile4 = reinterpret_cast<const uint4*>(tile);
    const int lane = lane_id();
    const bool big = la.qbs >= SEL_MAX_TILE;
    const int fb = loose_block(I.lrem0 + e0, la.qbs, big);
    const int nb = e1 > e0 ? loose_block(I.lrem0 + e1 - 1, la.qbs, big) - fb + 1 : 0;
    for (int i = lane; i < S_QTAB; i += 32) { ext[0][i] = 0xFFFFFFFFu; ext[1][i] = 0u; }
    __syncwarp();
    const bool vec = aligned16(I.g);
    int cur = -1;
    uint32_t alo = 0x7F807F80u, ahi = 0xFF80FF80u;           // packed bf16 pairs: running minimum from +inf, maximum from -inf
    auto hand_over = [&]() {
        alo = min_bf16x2(alo, alo >> 16 | alo << 16); ahi = max_bf16x2(ahi, ahi >> 16 | ahi << 16);
        atomicMin(&ext[0][cur], ord_key(__uint_as_float(alo << 16)));
        atomicMax(&ext[1][cur], ord_key(__uint_as_float(ahi << 16)));
    };
    for (int o = (e0 >> 3) + lane; o < (e1 >> 3); o += 32) {
        const uint4 v = tile4[phys_oct(o)];
        if (vec) {
            reinterpret_cast<uint4*>(I.g)[o] = v;
        } else {
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) I.g[o * 8 + e] = (uint16_t)(w[e >> 1] >> (16 * (e & 1)));
        }
        const int qi = loose_block(I.lrem0 + o * 8, la.qbs, big) - fb;
        if (qi != cur) {
            if (cur >= 0) hand_over();
            cur = qi; alo = 0x7F807F80u; ahi = 0xFF80FF80u;
        }
        ahi = max_bf16x2(max_bf16x2(ahi, v.x), max_bf16x2(max_bf16x2(v.y, v.z), v.w));
        alo = min_bf16x2(min_bf16x2(alo, v.x), min_bf16x2(min_bf16x2(v.y, v.z), v.w));
    }
    {
        const int c_first = __shfl_sync(0xffffffffu, cur, 0);
        if (__all_sync(0xffffffffu, cur == c_first) && c_first >= 0) {       // the whole warp ended in one block
            alo = min_bf16x2(alo, alo >> 16 | alo << 16); ahi = max_bf16x2(ahi, ahi >> 16 | ahi << 16);
            const uint32_t klo = __reduce_min_sync(0xffffffffu, ord_key(__uint_as_float(alo << 16)));
            const uint32_t khi = __reduce_max_sync(0xffffffffu, ord_key(__uint_as_float(ahi << 16)));
            if (lane == 0) { atomicMin(&ext[0][cur], klo); atomicMax(&ext[1][cur], khi); }
        } else if (cur >= 0) {
            hand_over();
        }
    }
    if (lane == 0) {                                         // a tensor's last, short octet
        for (int e = max(e0, e1 & ~7); e < e1; ++e) {
            const uint16_t x = tile[phys_pos(e)];
            I.g[e] = x;
            const float f = bf16_bits_to_f32(x);
            if (f != f) continue;                            // (a NaN is in no statistics)
            const int qi = loose_block(I.lrem0 + e, la.qbs, big) - fb;
            atomicMin(&ext[0][qi], ord_key(f)); atomicMax(&ext[1][qi], ord_key(f));
        }
    }
    __syncwarp();
    for (int i = lane; i < nb; i += 32) {
        atomicMin(la.st_min + I.qb_at + fb + i, ext[0][i]);
        atomicMax(la.st_max + I.qb_at + fb + i, ext[1][i]);
    }
    __syncwarp();
}

// QS: log2 of quant_block_size (3..7), or 0 for loose quantisation blocks of la.qbs elements, which ignore the borders of
// the top-k blocks; the kernel then ends a tile with the residual written back to the gradient buffer and the extremes of
// every block it touches merged into la.st_min / la.st_max (requant_loose.cu finishes the job).
template <int QS>
__global__ void __launch_bounds__(S_NT, S_CTAS)
ef_topk_quant_bf16_warps_kernel(const mab_tensor* __restrict__ tensors, int n_tensors, int total_units, int stage_elems, int allowing, LooseArgs la) {
    constexpr bool LOOSE = QS == 0;
    constexpr bool TABLE = LOOSE || QS >= 6;                 // constants of the warp's blocks from a table, else per unit
    extern __shared__ __align__(128) unsigned char smem_raw[];       // [tile][SmemSel]
    __shared__ int s_first[WIN_MAX_TENSORS + 1];
    __shared__ __align__(8) uint64_t s_bar[S_WARPS];
    uint16_t* const tile = reinterpret_cast<uint16_t*>(smem_raw);
    uint4* const tile4 = reinterpret_cast<uint4*>(smem_raw);
    SmemSel& ss = *reinterpret_cast<SmemSel*>(smem_raw + ((stage_elems * 2 + 127) & ~127));
    const int t = threadIdx.x, lane = lane_id(), warp = warp_id();
    if constexpr (!LOOSE) allow_next_kernel(allowing);
    // a CTA's tiles are neighbours: they mostly belong to one tensor, whose bound carries over from tile to tile
    const TileRange range = tiles_of_cta(total_units, gridDim.x, blockIdx.x);
    const int unit0 = range.first, unit1 = range.end;
    const bool big = LOOSE && la.qbs >= SEL_MAX_TILE;
    uint16_t* const list = ss.w[warp].list;
    const unsigned lower = (1u << lane) - 1u;
    uint32_t* const cand = ss.w[warp].cand;

    auto fill_info = [&](TileInfo& I, int unit, int ti) {    // one thread
        while (unit >= s_first[ti + 1]) ++ti;
        const mab_tensor& T = tensors[ti];
        const int blk = unit - s_first[ti];
        const int64_t base = (int64_t)blk * T.d_block_size;
        const int64_t qb0 = LOOSE ? base / la.qbs : base >> QS;
        const int64_t row_off = (int64_t)T.ring_index * row_pitch_of(T) + (int64_t)blk * T.k_block_size_many;
        I.g = reinterpret_cast<uint16_t*>(const_cast<void*>(static_cast<const void*>(T.grad))) + base;
        I.ef = T.error + (base >> 1);
        I.mn = T.min_vals + qb0; I.mx = T.max_vals + qb0;
        I.i_out = T.I + row_off; I.v_out = T.V + row_off;
        I.qe = T.quant_err != nullptr ? reinterpret_cast<uint16_t*>(T.quant_err) + base : nullptr;
        I.n = (int)min((int64_t)T.d_block_size, T.d - base);
        I.k = blk < T.topk_full_blocks_count ? T.k_block_size_many : T.k_block_size_few;
        I.ti = ti;
        I.lrem0 = LOOSE ? (int)(base - qb0 * la.qbs) : 0;
        I.qb_at = LOOSE ? la.qb_first[ti] + qb0 : 0;
    };

    // a tile's codes and statistics into L2; one thread.  (Its gradient only where plain loads fetch it; the copy engine brings a warp's part at a
    // time: 215 M elements 259 us a launch, 262 with it; loose blocks with the requantisation 395 and 398; 58 M with k = 5 % 104 and 105.  Off alignment 43 M 82
    // with it and 95 without, 133 M 220 and 249, blocks of 32, 116 M 210 and 232.)
    auto ask_tile = [&](const TileInfo& N) {
        auto ask = [](const void* at, int64_t bytes) {
            const uintptr_t from = reinterpret_cast<uintptr_t>(at) & ~(uintptr_t)15;
            const uint32_t len = (uint32_t)((reinterpret_cast<uintptr_t>(at) + bytes - from + 15) & ~(uintptr_t)15);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"(len) : "memory");
        };
        if (!aligned16(N.g) || (reinterpret_cast<uintptr_t>(N.ef) & 7) != 0) ask(N.g, (int64_t)N.n * 2);   // (`staged` below)
        ask(N.ef, ((int64_t)N.n + 1) >> 1);
        const int64_t nb = LOOSE ? loose_blocks_touched(N.lrem0, N.n, la.qbs) : ((int64_t)N.n + (1 << QS) - 1) >> QS;
        ask(N.mn, nb * 2);
        ask(N.mx, nb * 2);
    };

    for (int i = t; i < n_tensors; i += S_NT) s_first[i] = tensors[i].first_unit_a;
    if (t == 0) { s_first[n_tensors] = total_units; ss.kmax[0] = 0; ss.kmax[1] = 0; }
    if (lane == 0) mbar_init(&s_bar[warp], 1);
    if (t < S_BINS) { ss.hist[0][t] = 0; ss.hist[1][t] = 0; }
    for (int i = t; i < 256; i += S_NT) ss.cold_hist[i] = 0;
    __syncthreads();
    if (t == 0) { fill_info(ss.info[0], unit0, find_tensor(s_first, n_tensors, unit0)); ask_tile(ss.info[0]); }
    __syncthreads();

    // a tile's first loads, in flight when its turn comes: the gradient of the warp's segment on the copy engine, the code words of
    // its first slots and its statistics in registers
    struct Slot { uint2 c; uint32_t st[QS == 3 ? 2 : 1]; };  // st: statistics of the unit's block(s), where there is no table
    Slot ring[S_RING];
#pragma unroll
    for (int i = 0; i < S_RING; ++i) { ring[i].c = make_uint2(0u, 0u); ring[i].st[0] = 0u; ring[i].st[QS == 3 ? 1 : 0] = 0u; }
    uint32_t st_table[S_TABS];                               // min | max << 16 of the table's entries lane, lane + 32, ...
#pragma unroll
    for (int i = 0; i < S_TABS; ++i) st_table[i] = 0u;
    Segment seg = {0, 0};
    const int lane_off = ((lane >> 2) << 3) + ((2 * (lane & 3)) ^ (lane >> 2));   // where a unit's first octet sits in its slot; the second: ^ 1
    bool staged = false;                                     // gradient or codes not aligned for wide loads
    uint32_t parity = 0u;                                    // of the warp's next wait for the copy engine
    int u0 = 0, units = 0;                                   // the lane's first unit; whole units from there to the segment's end
    const uint8_t* ep = nullptr;                             // the code words of the lane's unit in the slot that follows the ring's ...
    const uint16_t* sp_mn = nullptr;                         // ... and its statistics, where there is no table
    const uint16_t* sp_mx = nullptr;
    auto load_stats = [&](Slot& r, int i, bool on) {
        if constexpr (!TABLE) {
            constexpr int STEP = S_SLOT >> (TABLE ? 0 : QS);
            if (on) {
                r.st[0] = sp_mn[i * STEP] | ((uint32_t)sp_mx[i * STEP] << 16);
                if constexpr (QS == 3) r.st[1] = sp_mn[i * STEP + 1] | ((uint32_t)sp_mx[i * STEP + 1] << 16);
            }
        }
    };
    // (i: slots behind the one where the pointers stand)
    auto load_slot = [&](Slot& r, int i, bool on) {
        if (!staged) {
            ld_global_8(ep + i * S_SLOT / 2, on, r.c);
        } else if (on && (reinterpret_cast<uintptr_t>(ep) & 3) == 0) {
            const uint32_t* e = reinterpret_cast<const uint32_t*>(ep + i * S_SLOT / 2);
            r.c = make_uint2(e[0], e[1]);
        }
        load_stats(r, i, on);
    };
    int tab0 = 0, tab_n = 0;                         // the table's first block and its length (from lane on)
    auto segment_of = [&](const TileInfo& I) {
        seg = warp_segment(I.n, (blockIdx.x + blockIdx.x * S_CTAS / gridDim.x) % S_WARPS, warp);
        u0 = seg.s0 * 32 + lane;
        units = min(I.n >> 4, (seg.s0 + seg.ns) * 32) - u0;
        if constexpr (TABLE && !LOOSE) {
            tab0 = (seg.s0 << (9 - QS)) + lane;
            tab_n = min((I.n + (1 << QS) - 1) >> QS, (seg.s0 + seg.ns) << (9 - QS)) - tab0;
        }
    };
    auto first_loads = [&](const TileInfo& I) {              // (a gradient that has to pass through the tile waits for its turn)
        staged = !aligned16(I.g) || (reinterpret_cast<uintptr_t>(I.ef) & 7) != 0;
        ep = I.ef + u0 * 8;
        if constexpr (TABLE) {
            if constexpr (LOOSE) {
                const int e0 = seg.s0 * S_SLOT, e1 = min(I.n, (seg.s0 + seg.ns) * S_SLOT);
                tab0 = loose_block(I.lrem0 + e0, la.qbs, big) + lane;
                tab_n = e1 > e0 ? loose_block(I.lrem0 + e1 - 1, la.qbs, big) - tab0 + 1 : 0;
            }
            const uint16_t* mn = I.mn + tab0;
            const uint16_t* mx = I.mx + tab0;
#pragma unroll
            for (int i = 0; i < S_TABS; ++i) st_table[i] = tab_n > 32 * i ? mn[32 * i] | ((uint32_t)mx[32 * i] << 16) : 0u;
        } else {
            const int b = QS == 3 ? 2 * u0 : u0 >> (QS > 4 ? QS - 4 : 0);
            sp_mn = I.mn + b; sp_mx = I.mx + b;
        }
#pragma unroll
        for (int i = 0; i < S_RING; ++i) load_slot(ring[i], i, units > 32 * i);
        ep += S_RING * S_SLOT / 2;
        if constexpr (!TABLE) { sp_mn += S_RING * (S_SLOT >> (TABLE ? 0 : QS)); sp_mx += S_RING * (S_SLOT >> (TABLE ? 0 : QS)); }
    };
    // the gradient of the warp's whole units into their places in the tile, in order; the warp is done with that part of the tile
    auto bring = [&](const TileInfo& I) {
        const int bytes = (units + lane) * 32;
        if (lane == 0 && bytes > 0) {
            mbar_arrive_expect_tx(&s_bar[warp], (uint32_t)bytes);
            bulk_g2s(tile + seg.s0 * S_SLOT, I.g + seg.s0 * S_SLOT, (uint32_t)bytes, &s_bar[warp]);
        }
    };
    segment_of(ss.info[0]);
    first_loads(ss.info[0]);
    if (!staged) bring(ss.info[0]);

    int guess = 0;                                           // bound on bf16 magnitudes from the tile before; 0: none
    int below = 4;                                           // how many magnitudes below the k-th value the next bound lies
    int i3 = 0;                                              // the tile's place among the three infos

    for (int unit = unit0; unit < unit1; ++unit) {
        const int p = (unit - unit0) & 1;
        const TileInfo& I = ss.info[i3];
        const int i3_next = i3 == 2 ? 0 : i3 + 1;
        const int n = I.n;
        // ---- decode: a = bf16(g + Qinv(e)) into the tile, units that reach the bound into the list -------------------
        const int e1 = min(n, (seg.s0 + seg.ns) * S_SLOT);   // end of the warp's elements
        const int lb0 = tab0 - lane;                         // loose: the table's first block
        bool slow = (reinterpret_cast<uintptr_t>(I.ef) & 3) != 0;    // some of the warp's units need the scalar decode
        if constexpr (TABLE) {
#pragma unroll
            for (int i = 0; i < S_TABS; ++i) {
                const QParams q = block_params(st_table[i] << 16, st_table[i] & 0xFFFF0000u, slow);
                ss.w[warp].mu[lane + 32 * i] = make_float4(q.mn, q.mn, q.u, q.u);
            }
            __syncwarp();
        }
        int n_w = 0;
        const uint32_t bound2 = guess > 0 ? (uint32_t)guess * 0x10001u : 0x7F817F81u;   // (without a bound nothing is listed)
        bool lost = false;                                   // the copy engine never delivered
        if (staged) {
            stage_anywhere(tile, I.g, seg.s0 * 64 + lane, min((n >> 4) * 2, (seg.s0 + seg.ns) * 64), (n + 7) >> 3);
            __syncwarp();
        } else if (__shfl_sync(0xffffffffu, units, 0) > 0) {
            lost = !mbar_wait(&s_bar[warp], parity);
            parity ^= 1u;
            if (lost && lane == 0) atomicExch(&g_copy_timeout, 1);
        }
        {
            uint4* at = tile4 + seg.s0 * 64;                 // the slot's octets: as they come 2 * lane and 2 * lane + 1 ...
            const int step = (lane_off ^ 1) - lane_off;      // ... and permuted at lane_off and 16 bytes on or back
            const float4* mup = &ss.w[warp].mu[QS >= 6 ? lane >> (QS >= 4 ? QS - 4 : 0) : 0];
            int left = units, u = u0;
            uint4 ga = make_uint4(0u, 0u, 0u, 0u), gb = ga;  // the gradient of the unit to decode next
            if (left > 0) { ga = at[2 * lane]; gb = at[2 * lane + 1]; }
            auto one = [&](Slot& r, int i) {
                uint4 oa, ob;
                if constexpr (TABLE && !LOOSE) {
                    const UnitConsts c = unit_consts(mup[i * (S_SLOT >> (QS >= 6 ? QS : 6))]);
                    oa = decode_add(ga, r.c.x, c); ob = decode_add(gb, r.c.y, c);
                } else if constexpr (LOOSE) {
                    const int e = I.lrem0 + (u + 32 * i) * 16;
                    const float4 ma = ss.w[warp].mu[min(loose_block(e, la.qbs, big) - lb0, S_QTAB - 1)];
                    const float4 mb = ss.w[warp].mu[min(loose_block(e + 8, la.qbs, big) - lb0, S_QTAB - 1)];
                    oa = decode_add(ga, r.c.x, unit_consts(ma)); ob = decode_add(gb, r.c.y, unit_consts(mb));
                } else {
                    const QParams qa = block_params(r.st[0] << 16, r.st[0] & 0xFFFF0000u, slow);
                    const QParams qb = QS == 3 ? block_params(r.st[QS == 3 ? 1 : 0] << 16, r.st[QS == 3 ? 1 : 0] & 0xFFFF0000u, slow) : qa;
                    oa = decode_add(ga, r.c.x, unit_consts(make_float4(qa.mn, qa.mn, qa.u, qa.u)));
                    ob = decode_add(gb, r.c.y, unit_consts(make_float4(qb.mn, qb.mn, qb.u, qb.u)));
                }
                load_slot(r, i, left > 32 * (i + S_RING));
                if (left > 32 * (i + 1)) { ga = at[(i + 1) * 64 + 2 * lane]; gb = at[(i + 1) * 64 + 2 * lane + 1]; }
                __syncwarp();                                // every lane has its octets of this slot
                const bool on = left > 32 * i;
                if (on) { at[i * 64 + lane_off] = oa; at[i * 64 + lane_off + step] = ob; }
                const uint32_t m2 = maxabs_bf16x2(maxabs_bf16x2(maxabs_bf16x2(oa.x, oa.y), maxabs_bf16x2(oa.z, oa.w)),
                                                  maxabs_bf16x2(maxabs_bf16x2(ob.x, ob.y), maxabs_bf16x2(ob.z, ob.w)));
                const bool hit = on && reach_mask(m2, bound2) != 0u;
                const unsigned hits = __ballot_sync(0xffffffffu, hit);
                if (hit) list[n_w + __popc(hits & lower)] = (uint16_t)(u + 32 * i);
                n_w += __popc(hits);
            };
#pragma unroll 1
            for (int s = seg.ns; s > 0; s -= S_RING) {
#pragma unroll
                for (int i = 0; i < S_RING; ++i) if (s > i) one(ring[i], i);
                ep += S_RING * S_SLOT / 2; at += S_RING * 64; mup += S_RING * (S_SLOT >> (QS >= 6 ? QS : 6));
                if constexpr (!TABLE) { sp_mn += S_RING * (S_SLOT >> (TABLE ? 0 : QS)); sp_mx += S_RING * (S_SLOT >> (TABLE ? 0 : QS)); }
                left -= S_RING * 32; u += S_RING * 32;
            }
        }
        if (__any_sync(0xffffffffu, slow)) {                 // the warp's whole units once more, the defining way
#pragma unroll 1
            for (int u = seg.s0 * 32 + lane; u < min((seg.s0 + seg.ns) * 32, n >> 4); u += 32) decode_unit_scalar(tile, I, u, LOOSE ? la.qbs : 1 << QS);
            __syncwarp();
            n_w = guess > 0 ? relist(tile4, list, seg.s0, seg.ns, n & ~15, bound2) : 0;
        }
        if ((n & 15) != 0) {                                 // the tile's last, short unit: one lane of the warp that owns its slot
            const int u = n >> 4;
            if (u >= seg.s0 * 32 && u < (seg.s0 + seg.ns) * 32) {
                if (lane == 0) decode_unit_scalar(tile, I, u, LOOSE ? la.qbs : 1 << QS);
                __syncwarp();
                if (guess > 0 && unit_mask(tile4, u, bound2) != 0u) { if (lane == 0) list[n_w] = (uint16_t)u; ++n_w; }
            }
        }
        __syncwarp();
        // one lane of one warp looks up the tile after this one and asks it into L2
        if (lane == 0 && warp == unit % S_WARPS && unit + 1 < unit1) {
            TileInfo& N = ss.info[i3_next];
            fill_info(N, unit + 1, I.ti);
            ask_tile(N);
        }

        // ---- exact top-k --------------------------------------------------------------------------------------------
        const int k = I.k;
        int bound = guess, need = 0, kth = 0;                // the k-th magnitude; how many values equal to it are selected
        bool cold = false, ok = false, zero = false;
        int n_c = 0;                                         // the warp's values that reach the bound
#pragma unroll 1
        for (int attempt = 0; attempt < 8; ++attempt) {
            if (bound == 0) {                                // no bound from the tile before, or one that fewer than k values reach
                if (cold || k > ((n + 7) >> 3)) break;
                cold = true;
                const Bound found = bound_from_octets(tile4, ss, p, list, seg.s0, seg.ns, n, k);
                bound = found.bound; n_w = found.n_w;
                if (bound <= 0) { zero = bound == 0; break; }
            }
            n_c = 0;
            {
                const uint32_t b2 = (uint32_t)bound * 0x10001u;
#pragma unroll 1
                for (int q0 = 0; q0 < n_w; q0 += 32) {       // a listed unit per lane
                    int u = 0;
                    uint32_t m = 0u;
                    if (q0 + lane < n_w) { u = list[q0 + lane]; m = unit_mask(tile4, u, b2); }
                    int total;
                    int to = n_c + mask_prefix(m, total);
                    n_c += total;
                    const uint16_t* at = tile + phys_oct(2 * u) * 8;
                    const uint16_t* at_odd = tile + phys_oct(2 * u + 1) * 8;
                    // the warp meets for every value: left to themselves the lanes come apart and take their turns one by one (loose blocks,
                    // k = 5 %, 29 M elements: this kernel 90 us without, 75 with the vote; 134 M, blocks of 64, k = 1 %: 176 and 168)
#pragma unroll 1
                    for (; __any_sync(0xffffffffu, m != 0u); m &= m - 1, ++to) {
                        if (m == 0u) continue;
                        const int b = __ffs(m) - 1;
                        const uint32_t v = (b < 8 ? at : at_odd - 8)[b];
                        atomicAdd(&ss.hist[p][min((int)(v & 0x7FFFu) - bound, S_BINS - 1)], 1);
                        if (to < S_CAND) cand[to] = (v << 16) | (uint32_t)(u * 16 + b);
                    }
                }
            }
            if (__syncthreads_or(lost)) return;
            // the bin of the k-th value, every warp for itself: a suffix sum over the lanes' four bins each
            const int4 h = reinterpret_cast<const int4*>(ss.hist[p])[lane];
            const int sum = h.x + h.y + h.z + h.w;
            int suf = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const int v = __shfl_down_sync(0xffffffffu, suf, d); if (lane + d < 32) suf += v; }
            const unsigned reach = __ballot_sync(0xffffffffu, suf >= k);
            if (reach != 0u) {
                const int owner = 31 - __clz(reach);
                int above = suf - sum, b = 3;
                if (above + h.w < k) { above += h.w; b = 2; if (above + h.z < k) { above += h.z; b = 1; if (above + h.y < k) { above += h.y; b = 0; } } }
                const int bin = __shfl_sync(0xffffffffu, lane * 4 + b, owner);
                need = k - __shfl_sync(0xffffffffu, above, owner);
                kth = bound + bin;
                if (bin < S_BINS - 1) {
                    ok = true;
                    // three standard deviations of the difference of two tiles' counts
                    const int extra = __shfl_sync(0xffffffffu, suf, 0) - k, want = min(k / 5 + 16, k / 16 + 72);
                    if (extra < want) ++below; else if (extra > 2 * want && below > 1) --below;
                    guess = max(1, kth - below);
                    break;
                }
                bound = kth;                                 // the last bin holds all that is larger: at least k values
                n_w = relist(tile4, list, seg.s0, seg.ns, n, (uint32_t)bound * 0x10001u);
            } else {
                bound = 0;
            }
            __syncthreads();
            if (t < S_BINS) ss.hist[p][t] = 0;
            __syncthreads();
        }
        if (ok) {
            // every warp counts its values above the k-th magnitude and equal to it ...
            __syncwarp();
            uint32_t mine = 0u;
            if (n_c <= S_CAND) {
#pragma unroll 1
                for (int i = lane; i < n_c; i += 32) {
                    const int key = (int)(cand[i] >> 16) & 0x7FFF;
                    mine += key > kth ? 1u : key == kth ? 0x10000u : 0u;
                }
            } else {
#pragma unroll 1
                for (int i = lane; i < n_w; i += 32) {
                    const uint32_t gt = unit_mask(tile4, list[i], (uint32_t)(kth + 1) * 0x10001u), ge = unit_mask(tile4, list[i], (uint32_t)kth * 0x10001u);
                    mine += __popc(gt) | (__popc(ge ^ gt) << 16);
                }
            }
            mine = __reduce_add_sync(0xffffffffu, mine);
            if (lane == 0) ss.counts[p][warp] = mine;
            __syncthreads();
            // ... and finds their places behind those of the warps before
            const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? ss.counts[p][lane] : 0u);
            int ties = (int)(before >> 16), rank = (int)(before & 0xFFFFu) + min(need, ties);
            const bool all_ties = ties + (int)(mine >> 16) <= need;
            int16_t* const i_out = I.i_out;
            uint16_t* const v_out = I.v_out;
            if (n_c <= S_CAND) {
#pragma unroll 1
                for (int i = 0; i < n_c; i += 32) {
                    const uint32_t c = i + lane < n_c ? cand[i + lane] : 0u;
                    const int key = (int)(c >> 16) & 0x7FFF;
                    bool take = key >= kth;
                    if (!all_ties) {                         // the lowest positions among the equal ones
                        const unsigned eq = __ballot_sync(0xffffffffu, key == kth);
                        take = key > kth || (key == kth && ties + __popc(eq & lower) < need);
                        ties += __popc(eq);
                    }
                    const unsigned sel = __ballot_sync(0xffffffffu, take);
                    if (take) {
                        const int to = rank + __popc(sel & lower), pos = (int)(c & 0xFFFFu);
                        i_out[to] = (int16_t)pos;
                        v_out[to] = (uint16_t)(c >> 16);
                        tile[phys_pos(pos)] = 0;
                    }
                    rank += __popc(sel);
                }
            } else {
                select_from_units(tile, list, n_w, kth, need, ties, rank, i_out, v_out);
            }
            __syncwarp();
        } else {
            if (__syncthreads_or(lost)) return;              // (a tile can come here without having counted candidates)
            select_by_bisection(tile, ss, n, k, zero, I.i_out, I.v_out);
            guess = 0;
        }
        if (t < S_BINS) ss.hist[p][t] = 0;                   // (everyone has read it; it is filled again two tiles from here)
        if (cold) for (int i = t; i < 256; i += S_NT) ss.cold_hist[i] = 0;   // (this not before the next tile's first barrier)
        if (t == S_NT - 1) ss.kmax[p] = 0;

        // ---- the residual: alpha == -2 keeps it, statistics and codes ----------------------------------------------
        if (I.qe != nullptr) {
            uint16_t* qe = I.qe;
            const bool vec = aligned16(qe);
#pragma unroll 1
            for (int o = seg.s0 * 64 + lane; o * 8 < e1; o += 32) {
                if (vec && o * 8 + 8 <= n) reinterpret_cast<uint4*>(qe)[o] = tile4[phys_oct(o)];
                else for (int e = o * 8; e < min(o * 8 + 8, n); ++e) qe[e] = tile[phys_pos(e)];
            }
        }
        if constexpr (LOOSE) {
            residual_and_extremes(tile, min(seg.s0 * S_SLOT, e1), e1, I, la, ss.w[warp].ext);
        } else {
            const int b1 = min(n >> QS, (seg.s0 + seg.ns) << (9 - QS));
            stats_encode<QS>(tile4, (seg.s0 << (9 - QS)) + lane, b1, I);
            if ((n & ((1 << QS) - 1)) != 0 && (n >> QS) >= (seg.s0 << (9 - QS)) && (n >> QS) < ((seg.s0 + seg.ns) << (9 - QS)))
                stats_encode_short<QS>(tile4, n >> QS, n, I);
        }
        if (unit + 1 < unit1) {
            const TileInfo& N = ss.info[i3_next];
            const bool moved = N.n != n;                     // another length: the warps' parts of the tile change hands
            if (moved) segment_of(N);
            first_loads(N);
            if (moved) __syncthreads();
            fence_async_smem();                              // this lane's accesses to the tile, before the copy engine's
            __syncwarp();                                    // the warp's part of the tile is overwritten next
            if (!staged) bring(N);
        }
        i3 = i3_next;
    }
}

}  // namespace warps

int launch_ef_topk_quant_bf16_warps(const mab_tensor* dev_tensors, int n_tensors, int total_units, int qbs, int max_dbs, int allowing, cudaStream_t s,
                              const LooseArgs* loose) {
    using namespace warps;
    const int smem = ((max_dbs * 2 + 127) & ~127) + (int)sizeof(SmemSel);
    const int per_sm = std::min(S_CTAS, (device_max_optin_smem() + 1024) / (smem + 3 * 1024 + 128));
    if (per_sm < 2) return 1;                                // not even two CTAs per SM: the caller uses the other kernel
    const int grid = (int)std::min<int64_t>(total_units, (int64_t)device_sm_count() * per_sm);
    LooseArgs la = {0, nullptr, nullptr, nullptr};
    if (loose) la = *loose;
    auto run = [&](auto kern) -> int {
        MAB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kern<<<grid, S_NT, smem, s>>>(dev_tensors, n_tensors, total_units, max_dbs, allowing, la);
        return MAB_OK;
    };
    const int rc = loose ? run(ef_topk_quant_bf16_warps_kernel<0>)
                 : qbs == 8 ? run(ef_topk_quant_bf16_warps_kernel<3>) : qbs == 16 ? run(ef_topk_quant_bf16_warps_kernel<4>)
                 : qbs == 32 ? run(ef_topk_quant_bf16_warps_kernel<5>) : qbs == 64 ? run(ef_topk_quant_bf16_warps_kernel<6>)
                 : run(ef_topk_quant_bf16_warps_kernel<7>);
    if (rc) return rc;
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "ef_topk_quant_bf16_warps_kernel launch");
    return MAB_OK;
}

int copy_timeout_bf16_warps(int* out, bool clear) {
    cudaError_t e = cudaMemcpyFromSymbol(out, warps::g_copy_timeout, sizeof(int));
    if (e == cudaSuccess && clear) { const int z = 0; e = cudaMemcpyToSymbol(warps::g_copy_timeout, &z, sizeof(int)); }
    return e == cudaSuccess ? MAB_OK : cuda_fail(e, "mab_device_error");
}

}  // namespace mab
