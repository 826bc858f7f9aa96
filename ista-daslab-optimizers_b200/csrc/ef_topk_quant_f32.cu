// Kernel A for fp32 gradients, two tiles per SM: a tile is split between registers and shared memory.
//
// An fp32 tile (29 056 values) is 116 KB; two of them are all the shared memory an SM has, and one tile per SM
// (ef_topk_quant.cu) leaves the chip waiting at every barrier of the selection.  Here a CTA of 512 threads holds the
// tile's first 1024 octets in registers (two per thread, 32 KB) and the other 2608 in shared memory (83 KB), next to
// 26 KB of selection scratch, so that two CTAs share an SM and one tile's chain of dependent phases overlaps the
// other's arithmetic.  The shared-memory part is staged by the bulk copy engine and turned into a = g + Qinv(e) in
// place; the beginning of the tile after this one is asked into L2 meanwhile.
//
// Thread t owns octets 2 t and 2 t + 1 (registers) and 1024 + t, 1024 + t + 512, ... (shared memory).  An octet in shared
// memory is two 16-byte pieces 32 bytes apart from the next lane's: lanes 4-7 of every 8 take the second piece first
// (`h`), so that a quarter warp's 16-byte accesses cover all banks; the code word is rotated by 16 bits to match.
//
// Regular tiles (whole blocks of 64, seven whole octets per thread, codes on a 16-byte boundary, every block with a finite
// step; the gradient may start anywhere: all but a tensor's last tile) take a leaner route: the decode has no branches and
// writes a with the sixteen 16-byte pieces of every 256-byte row (= one quantisation block) permuted by the row number
// (piece c of row r sits at c ^ (r & 7)), so that after the selection a thread owns whole rows, consecutive lanes reading
// different banks, and computes a block's statistics, constants and 32 code bytes without shuffles.
//
// Bound by instruction issue and the phases' barriers, not by memory: 33.6 M elements take 122 us with one tile per SM, 111
// with two on the general route (other block sizes), 92 on the regular one; with k = 5 % 141, 133 and 113.
#include "common.cuh"
#include "select.cuh"
#include "codec_fast.cuh"
#include "async_copy.cuh"
#include "fused.cuh"

namespace mab {

constexpr int F_NT = 512;
constexpr int F_CTAS = 2;                    // resident CTAs per SM the shared memory and the registers are sized for
constexpr int F_REG = 2;                     // octets a thread keeps in registers
constexpr int F_SLOTS = SEL_MAX_TILE / 8 / F_NT;   // octets per thread: 8
constexpr int F_REG_ELEMS = F_REG * F_NT * 8;      // tile elements that never enter shared memory
constexpr int F_WPT = SEL_WORDS / F_NT;      // bitmap words per thread: 2
constexpr int F_FULL = 5;                    // shared-memory octets every thread of a regular tile owns (some own one more)
constexpr int F_CAND_CAP = 3072;
constexpr int F_WLIST = 192;                 // shared-memory octets with a candidate, per warp
constexpr int F_MAX_K = 1880;                // largest k whose candidates fit the list (see launch_ef_topk_quant_f32)
static_assert(F_WPT == 2, "a thread owns two consecutive bitmap words");

// Set when a wait on the copy engine gave up; read through mab_device_error() together with the other kernels' flags.
__device__ int g_copy_timeout_f32;

struct __align__(16) SmemF {
    union {
        struct {                             // candidates: |value| bits and ((0x7FFF - position) << 1 | sign);
            uint32_t key[F_CAND_CAP];        //   (key, meta) pairs are distinct and "larger is better" contains the tie rule
            uint16_t meta[F_CAND_CAP];
        };
        float2 qtab[F_CAND_CAP * 6 / 8];     // before the selection: (min, u) of the tile's quantisation blocks
        struct { uint32_t gt_bm[SEL_WORDS], tie_bm[SEL_WORDS]; };   // general selection: key > T, key == T
    };
    union {
        struct {
            uint32_t sel_bm[SEL_WORDS];      // selected positions
            uint16_t sel_before[SEL_WORDS];  // selected positions in lower words
        };
        uint16_t oct_list[(F_NT / 32) * F_WLIST];      // before the selection: octets that hold a candidate, per warp
    };
    unsigned long long member[32];
    int hist[256];
    int rot[64];
    int counters[40];
    int scan[36];
    int n_member, n_cand, kmax, over, slow, pad[3];
};
constexpr int F_QTAB = F_CAND_CAP * 6 / 8;   // quantisation blocks whose constants fit the table: 2304 (all of a tile's when they have 16 elements or more)
static_assert(sizeof(uint16_t) * (F_NT / 32) * F_WLIST <= (4 + 2) * SEL_WORDS, "the octet lists reuse the bitmap");

// The octet thread t owns in slot j.
__device__ __forceinline__ int f32_oct(int j) { return j < F_REG ? F_REG * (int)threadIdx.x + j : j * F_NT + (int)threadIdx.x; }

// Where element e of the shared-memory part sits on a permuted (regular) tile.
__device__ __forceinline__ int f32_phys(int e, bool swz) { return swz ? e ^ (((e >> 6) & 7) << 2) : e; }

// Octet o of the shared-memory part; h: which of its two 16-byte pieces comes first in v.
__device__ __forceinline__ void octet_from_smem(const float4* tile4, int o, int h, bool swz, float (&v)[8]) {
    const int at = (o * 2 + h) ^ (swz ? (o >> 3) & 7 : 0);
    const float4 a = tile4[at], b = tile4[at ^ 1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void octet_to_smem(float4* tile4, int o, int h, bool swz, const float (&v)[8]) {
    const int at = (o * 2 + h) ^ (swz ? (o >> 3) & 7 : 0);
    tile4[at] = make_float4(v[0], v[1], v[2], v[3]);
    tile4[at ^ 1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ uint32_t rotate_codes(uint32_t w, int h) { return __funnelshift_l(w, w, h << 4); }

// The scalar forms of the codec on an octet, out of line: degenerate blocks and a tensor's last, short octet.
__device__ __noinline__ void decode_octet_scalar(uint32_t w, float mn, float u, float* x) {
    const QParams q = {mn, u};
    for (int e = 0; e < 8; ++e) x[e] = qinv((w >> (8 * (e >> 1) + ((e & 1) ? 0 : 4))) & 0xFu, q);
}
__device__ __noinline__ uint32_t encode_octet_scalar(const float* r, float mn, float u, int cnt) {
    const QParams q = {mn, u};
    uint32_t w = 0;
    for (int e = 0; e < cnt; ++e) w |= qcode_exact(r[e], q) << (8 * (e >> 1) + ((e & 1) ? 0 : 4));
    return w;
}

// Never a NaN (0 for an octet that holds nothing else): the bound search compares bits, and a NaN's would reach every bound.
__device__ __forceinline__ float octet_max_abs(const float (&v)[8]) {
    const float m0 = max3(fabsf(v[0]), fabsf(v[1]), fabsf(v[2])), m1 = max3(fabsf(v[3]), fabsf(v[4]), fabsf(v[5]));
    return max3(m0, m1, max3(fabsf(v[6]), fabsf(v[7]), 0.0f));
}
__device__ __forceinline__ void add_octet(float (&v)[8], const float (&x)[8]) {
#pragma unroll
    for (int b = 0; b < 8; b += 2) {
        const float2 s = __fadd2_rn(make_float2(v[b], v[b + 1]), make_float2(x[b], x[b + 1]));
        v[b] = s.x; v[b + 1] = s.y;
    }
}
// v <- v + Qinv(codes) with the constants (min, u) of a block whose step is finite and not negative; returns the largest |v|.
__device__ __forceinline__ float accumulate_regular(float (&v)[8], uint32_t codes, float2 mu) {
    const QParams q = {mu.x, mu.y};
    float x[8];
    decode_octet_fast(codes, decode_consts(q), x);
    add_octet(v, x);
    return octet_max_abs(v);
}

// v <- v + Qinv(codes), elements from `cnt` on to 0; returns the largest |v|.
__device__ __forceinline__ float accumulate_octet(float (&v)[8], uint32_t codes, const QParams& q, int cnt) {
    const DecodeConsts dc = decode_consts(q);
    float x[8];
    if (dc.fast) {
        decode_octet_fast(codes, dc, x);
    } else {
        float y[8];
        decode_octet_scalar(codes, q.mn, q.u, y);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = y[e];
    }
    add_octet(v, x);
    if (cnt < 8) {
#pragma unroll
        for (int e = 0; e < 8; ++e) if (e >= cnt) v[e] = 0.0f;
    }
    return octet_max_abs(v);
}

// Whether the codes of a block need no clamp: its values lie within half an ulp of bf16 (2^-8 of the larger statistic's
// magnitude) of [mn, mx], which is less than half a step when that magnitude is at most 125 steps: the quotients then
// stay in (-0.5, 15.5).
__device__ __forceinline__ bool codes_in_range(uint16_t mn_b, uint16_t mx_b, const QParams& q) {
    return fmaxf(fabsf(bf16_bits_to_f32(mn_b)), fabsf(bf16_bits_to_f32(mx_b))) <= 125.0f * q.u;
}
__device__ __forceinline__ bool step_in_range(const QParams& q) { return q.u >= CODEC_U_MIN && q.u <= CODEC_U_MAX; }

// The 32 code bytes of row r of a regular tile (one quantisation block, pieces permuted by key = r & 7).
template <bool CLAMP>
__device__ __forceinline__ void encode_row(const float4* row, int key, const DivConsts& dc, uint4* dst) {
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        uint32_t w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float4 a = row[(half * 8 + 2 * c) ^ key], b = row[(half * 8 + 2 * c + 1) ^ key];
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            w[c] = encode_octet_div_f32<CLAMP>(v, dc);
        }
        dst[half] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Statistics and codes of the shared-memory part of a regular tile: thread t owns rows t, t + F_NT, ...
__device__ __forceinline__ void stats_encode_rows(const float4* tile4, int n_rows, uint16_t* mn_out, uint16_t* mx_out, uint8_t* ef_out) {
    for (int r = threadIdx.x; r < n_rows; r += F_NT) {
        const float4* row = tile4 + (r << 4);
        const int key = r & 7;
        float lo = INFINITY, hi = -INFINITY;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            const float4 v = row[c ^ key];
            lo = min3_nan(min3_nan(lo, v.x, v.y), v.z, v.w);
            hi = max3(max3(hi, v.x, v.y), v.z, v.w);
        }
        const uint16_t mn_b = f32_to_bf16_bits_rne(lo), mx_b = f32_to_bf16_bits_rne(hi);
        mn_out[r] = mn_b; mx_out[r] = mx_b;
        QParams q = qparams(mn_b, mx_b);
        uint4* dst = reinterpret_cast<uint4*>(ef_out) + (r << 1);
        if (!step_in_range(q)) {                             // all-equal block (u == 0), subnormal or infinite step, or a NaN in it
            if (lo != lo) {                                  // the statistics are those of the other values; the NaN's code is 0
                lo = INFINITY;
                for (int i = 0; i < 64; ++i) lo = fminf(lo, reinterpret_cast<const float*>(row)[i]);
                mn_out[r] = f32_to_bf16_bits_rne(lo);
                q = qparams(f32_to_bf16_bits_rne(lo), mx_b);
            }
            for (int o = 0; o < 8; ++o) {
                float y[8];
                for (int e = 0; e < 8; ++e) y[e] = reinterpret_cast<const float*>(row)[((o * 8 + e) ^ (key << 2))];
                reinterpret_cast<uint32_t*>(dst)[o] = encode_octet_scalar(y, q.mn, q.u, 8);
            }
        } else if (codes_in_range(mn_b, mx_b, q)) {
            encode_row<false>(row, key, div_consts(q), dst);
        } else {
            encode_row<true>(row, key, div_consts(q), dst);
        }
    }
}

// Number of the tile's keys >= thr (key bits), every thread of the CTA calling; `counter` is zero on entry.
__device__ __forceinline__ int f32_count_ge(const float (&a)[F_REG][8], const float4* tile4, int n_oct, bool swz, int thr, int* counter) {
    const float thr_f = __int_as_float(thr);
    int c = 0;
#pragma unroll
    for (int j = 0; j < F_REG; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) c += (fabsf(a[j][e]) >= thr_f) ? 1 : 0;
    for (int o = threadIdx.x + F_REG * F_NT; o < n_oct; o += F_NT) {
        float v[8];
        octet_from_smem(tile4, o - F_REG * F_NT, 0, swz, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) c += (fabsf(v[e]) >= thr_f) ? 1 : 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane_id() == 0 && c) atomicAdd(counter, c);
    __syncthreads();
    return *reinterpret_cast<volatile int*>(counter);
}

// Whether the tile holds a NaN, every thread of the CTA calling.
__device__ __forceinline__ bool f32_any_nan(const float (&a)[F_REG][8], const float4* tile4, int n_oct) {
    bool nan = false;
#pragma unroll
    for (int j = 0; j < F_REG; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) nan |= isnan(a[j][e]);
    for (int i = threadIdx.x; i < (n_oct - F_REG * F_NT) * 2; i += F_NT) {
        const float4 v = tile4[i];
        nan |= isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w);
    }
    return __syncthreads_or(nan);
}

// sel_bm from gt | (the need_ties lowest positions of tie) of the thread's own two words, and sel_before.  Starts and
// ends with a barrier.
__device__ __forceinline__ void f32_resolve(uint32_t (&sel)[F_WPT], uint32_t (&tw)[F_WPT], int need_ties, SmemF& ss) {
    __syncthreads();
    int total;
    if (need_ties > 0) {
        int before = block_exclusive_scan(__popc(tw[0]) + __popc(tw[1]), ss.scan, total);
#pragma unroll
        for (int i = 0; i < F_WPT; ++i) {
            const int keep = need_ties - before;
            before += __popc(tw[i]);
            if (keep <= 0) tw[i] = 0;
            else while (__popc(tw[i]) > keep) tw[i] &= ~(0x80000000u >> __clz(tw[i]));
            sel[i] |= tw[i];
        }
        __syncthreads();
    }
    const int before = block_exclusive_scan(__popc(sel[0]) + __popc(sel[1]), ss.scan, total);
    const int w0 = threadIdx.x * F_WPT;
    ss.sel_bm[w0] = sel[0]; ss.sel_bm[w0 + 1] = sel[1];
    ss.sel_before[w0] = (uint16_t)before; ss.sel_before[w0 + 1] = (uint16_t)(before + __popc(sel[0]));
    __syncthreads();
}

__global__ void __launch_bounds__(F_NT, F_CTAS)
ef_topk_quant_f32_kernel(const mab_tensor* __restrict__ tensors, int n_tensors, int total_units, int qshift, int tile_bytes, int allowing) {
    extern __shared__ __align__(128) unsigned char smem_raw[];       // [tile elements from F_REG_ELEMS on][SmemF]
    __shared__ int s_first[WIN_MAX_TENSORS + 1];
    __shared__ __align__(8) uint64_t s_bar;
    float* tile = reinterpret_cast<float*>(smem_raw);
    float4* tile4 = reinterpret_cast<float4*>(smem_raw);
    SmemF& ss = *reinterpret_cast<SmemF*>(smem_raw + tile_bytes);
    const int t = threadIdx.x, lane = lane_id(), warp = warp_id();
    allow_next_kernel(allowing);
    for (int i = t; i < n_tensors; i += F_NT) s_first[i] = tensors[i].first_unit_a;
    if (t == 0) { s_first[n_tensors] = total_units; mbar_init(&s_bar, 1); ss.slow = 0; }
    __syncthreads();
    const int oshift = qshift - 3;              // octets per quantisation block, as a shift
    const int lanes_per_qb = 1 << oshift;
    uint32_t parity = 0;
    int guess = 0;                              // lower bound found for the previous tile, as key bits

    for (int unit = blockIdx.x; unit < total_units; unit += gridDim.x) {
        const int ti = find_tensor(s_first, n_tensors, unit);
        const mab_tensor& T = tensors[ti];
        const int blk = unit - s_first[ti];
        const int64_t base = (int64_t)blk * T.d_block_size;
        const int n = (int)min((int64_t)T.d_block_size, T.d - base);
        const int k = (blk < T.topk_full_blocks_count) ? T.k_block_size_many : T.k_block_size_few;
        const float* g = reinterpret_cast<const float*>(T.grad) + base;
        uint8_t* ef = T.error + (base >> 1);
        uint16_t* mn_g = T.min_vals + (base >> qshift);
        uint16_t* mx_g = T.max_vals + (base >> qshift);
        const int n_oct = (n + 7) >> 3;
        const int n_qb = (n + (1 << qshift) - 1) >> qshift;
        const bool whole = (n & 7) == 0;                             // no short octet
        const bool g_al16 = aligned16(g);
        const bool ef_al4 = (reinterpret_cast<uintptr_t>(ef) & 3) == 0;
        const bool tables = n_qb <= F_QTAB;
        const int64_t row_off = (int64_t)T.ring_index * row_pitch_of(T) + (int64_t)blk * T.k_block_size_many;
        int16_t* i_out = T.I + row_off;
        uint16_t* v_out = T.V + row_off;

        // ---- bring the tile in; meanwhile codes -> registers, decode constants -> table ---------------------
        const int n_smem = n - F_REG_ELEMS;                          // elements in shared memory, if any
        const bool staged = n_smem > 0 && whole && g_al16;           // the bulk copy moves whole 16-byte pieces
        if (staged) {
            if (t == 0) {
                fence_async_smem();
                mbar_arrive_expect_tx(&s_bar, (uint32_t)n_smem * 4u);
                bulk_g2s(tile, g + F_REG_ELEMS, (uint32_t)n_smem * 4u, &s_bar);
            }
        } else {
            for (int i = t; i < n_oct * 8 - F_REG_ELEMS; i += F_NT) {
                if (i < n_smem) cp_async_4(tile + i, g + F_REG_ELEMS + i);
                else tile[i] = 0.0f;
            }
            cp_async_commit();
        }
        if (t == 0) { ss.kmax = 0; ss.n_member = 0; ss.n_cand = 0; ss.over = 0; }
        if (t < 64) ss.rot[t] = 0;
        if (t < 256) ss.hist[t] = 0;
        float a[F_REG][8];
#pragma unroll
        for (int j = 0; j < F_REG; ++j) {
            const int o = f32_oct(j), cnt = n - o * 8;
            if (g_al16 && cnt >= 8) {
                const float4 x = __ldg(reinterpret_cast<const float4*>(g) + o * 2), y = __ldg(reinterpret_cast<const float4*>(g) + o * 2 + 1);
                a[j][0] = x.x; a[j][1] = x.y; a[j][2] = x.z; a[j][3] = x.w; a[j][4] = y.x; a[j][5] = y.y; a[j][6] = y.z; a[j][7] = y.w;
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) a[j][e] = e < cnt ? g[o * 8 + e] : 0.0f;
            }
        }
        uint32_t cw[F_SLOTS];
        if (ef_al4 && whole) {
#pragma unroll
            for (int j = 0; j < F_SLOTS; ++j) { const int o = f32_oct(j); cw[j] = o < n_oct ? reinterpret_cast<const uint32_t*>(ef)[o] : 0u; }
        } else {
#pragma unroll
            for (int j = 0; j < F_SLOTS; ++j) {
                const int o = f32_oct(j);
                uint32_t w = 0;
                if (ef_al4 && o * 8 + 8 <= n) w = reinterpret_cast<const uint32_t*>(ef)[o];
                else for (int b = 0; b < 4; ++b) if (o * 8 + 2 * b < n) w |= (uint32_t)ef[o * 4 + b] << (8 * b);
                cw[j] = w;
            }
        }
        if (tables) {
            bool slow = false;
            for (int b = t; b < n_qb; b += F_NT) {
                const QParams q = qparams(mn_g[b], mx_g[b]);
                ss.qtab[b] = make_float2(q.mn, q.u);
                slow |= !decode_consts(q).fast;
            }
            if (slow) ss.slow = 1;
        }
        if (staged) {
            const bool ok = mbar_wait(&s_bar, parity);
            parity ^= 1u;
            if (__syncthreads_or(!ok)) {                             // the copy engine never delivered: flag it and stop
                if (t == 0) atomicExch(&g_copy_timeout_f32, 1);
                return;
            }
        } else {
            cp_async_wait_all();
            __syncthreads();
        }
        if (unit + (int)gridDim.x < total_units) {                   // the tile after this one: into L2 while this one is worked on
            const int nu = unit + gridDim.x;
            const int nti = find_tensor(s_first, n_tensors, nu);
            const mab_tensor& N = tensors[nti];
            const int64_t nbase = (int64_t)(nu - s_first[nti]) * N.d_block_size;
            const int64_t nn = min((int64_t)N.d_block_size, N.d - nbase);
            // Of the gradient the first three eighths: what the threads load into registers (28 %) and a little more.  The rest is the copy engine's,
            // whose latency hides; asked for as well, it drove lines out of L2 before their turn (124.4 M elements, us a launch: all of it 274,
            // 5/8 267, 1/2 267, 3/8 264, 5/16 265, nothing 272; 67 M with k = 5 % 199, 3/8 193).
            prefetch_l2<F_NT>(reinterpret_cast<uintptr_t>(reinterpret_cast<const float*>(N.grad) + nbase), nn * 3 / 2);
            if (warp < 3) {                                          // codes and statistics: a warp each
                const uintptr_t pb = warp == 0 ? reinterpret_cast<uintptr_t>(N.error + (nbase >> 1))
                                   : reinterpret_cast<uintptr_t>((warp == 1 ? N.min_vals : N.max_vals) + (nbase >> qshift));
                const int64_t bytes = warp == 0 ? (nn + 1) >> 1 : ((nn + (1 << qshift) - 1) >> qshift) * 2;
                const uintptr_t first = pb & ~(uintptr_t)127;
                const int lines = (int)((pb + bytes - first + 127) >> 7);
                for (int i = lane; i < lines; i += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(first + ((uintptr_t)i << 7)));
            }
        }

        // ---- a = g + Qinv(e) in place; per-octet maxima stay in registers ------------------------------------
        const int h = whole ? (lane >> 2) & 1 : 0;                   // (a short octet needs its elements in order)
        const int n_so = n_oct - F_REG * F_NT;                       // octets in shared memory
        // regular tile: see the head of the file; its pieces are permuted from here on
        const bool swz = qshift == 6 && (n & 63) == 0 && n_so >= F_FULL * F_NT && (reinterpret_cast<uintptr_t>(ef) & 15) == 0 &&
                         ss.slow == 0;
        float omax[F_SLOTS];
        if (swz) {
#pragma unroll
            for (int j = 0; j < F_REG; ++j) omax[j] = accumulate_regular(a[j], cw[j], ss.qtab[t >> 2]);
#pragma unroll
            for (int j = F_REG; j < F_SLOTS; ++j) {
                const int so = t + (j - F_REG) * F_NT;
                omax[j] = 0.0f;
                if (j < F_REG + F_FULL || (so & ~31) < n_so) {       // whole warps: the 8 lanes of a row read it before they write it
                    const bool on = j < F_REG + F_FULL || so < n_so;
                    const int at = on ? so : 0;
                    float v[8];
                    octet_from_smem(tile4, at, h, false, v);
                    const float m = accumulate_regular(v, rotate_codes(cw[j], h), ss.qtab[(at >> 3) + F_REG_ELEMS / 64]);
                    __syncwarp();
                    if (on) { octet_to_smem(tile4, so, h, true, v); omax[j] = m; }
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < F_SLOTS; ++j) {
                const int o = f32_oct(j);
                omax[j] = 0.0f;
                if (o < n_oct) {
                    QParams q;
                    if (tables) { const float2 c = ss.qtab[o >> oshift]; q.mn = c.x; q.u = c.y; }
                    else q = qparams(mn_g[o >> oshift], mx_g[o >> oshift]);
                    const int cnt = whole ? 8 : n - o * 8;
                    if (j < F_REG) {
                        omax[j] = accumulate_octet(a[j < F_REG ? j : 0], cw[j], q, cnt);
                    } else {
                        float v[8];
                        octet_from_smem(tile4, o - F_REG * F_NT, h, false, v);
                        omax[j] = accumulate_octet(v, rotate_codes(cw[j], h), q, cnt);
                        octet_to_smem(tile4, o - F_REG * F_NT, h, false, v);
                    }
                }
            }
        }

        // ---- exact top-k ---------------------------------------------------------------------------
        {
            float tm = 0.0f;
#pragma unroll
            for (int j = 0; j < F_SLOTS; ++j) tm = fmaxf(tm, omax[j]);
            const int wm = __reduce_max_sync(0xffffffffu, __float_as_int(tm));
            if (lane == 0 && wm) atomicMax(&ss.kmax, wm);
        }
        __syncthreads();
        const int kmax = ss.kmax;
        if (t == 0) ss.slow = 0;                                     // (for the next tile)
        bool fast = false;                                           // the selection is described by the candidate list
        int C = 0;
        if (kmax > 0 && kmax < 0x7f800000 && k <= n_oct) {
            // lower bound of the k-th key on octet maxima: at least k octets reach it, at most ~1.5 k (fewer where that
            // would bring more candidates than the list holds)
            const int accept = k + (k > 1024 ? 192 : (k >> 1) + 8);
            int lo = 0, hi = kmax + 1, step = 1 << 20;
            int gq = (guess > 0 && guess <= kmax) ? guess : max(1, kmax - (2 << 23));
            bool have_lo = false, have_hi = false, search = true;
            const bool cold = guess <= 0 || guess > kmax;    // no bound from a tile before: the histogram of the maxima gives one
            if (cold) {
                const int c = bound_from_histogram(omax, kmax, k, ss.hist, lo, hi);
                have_lo = c > 0; have_hi = true;
                search = hi - lo > 1 && !(c > 0 && c <= accept);
                gq = have_lo ? lo + ((hi - lo) >> 1) : max(hi - step, 1);
            }
            for (int it = 0; search && it < 64; ++it) {
                int mine = 0;
#pragma unroll
                for (int j = 0; j < F_SLOTS; ++j) mine += (__float_as_int(omax[j]) >= gq) ? 1 : 0;
                mine = __reduce_add_sync(0xffffffffu, mine);
                if (lane == 0 && mine) atomicAdd(&ss.rot[it], mine);
                __syncthreads();
                const int c = *reinterpret_cast<volatile int*>(&ss.rot[it]);
                if (c >= k) { lo = gq; have_lo = true; if (c <= accept) break; }
                else { hi = gq; have_hi = true; }
                if (hi - lo <= 1) break;
                if (have_lo && have_hi) gq = lo + ((hi - lo) >> 1);
                else if (have_lo) { gq = (int)min((int64_t)lo + step, (int64_t)hi - 1); step <<= 1; }
                else { gq = (int)max((int64_t)hi - step, (int64_t)1); step <<= 1; }
            }
            guess = lo;
            if (have_lo && lo > 0) {
                const float lo_f = __int_as_float(lo);
                // 1. candidates = values that reach the bound, in any order: a thread's register octets directly ...
                {
                    uint32_t mask = 0u;
#pragma unroll
                    for (int j = 0; j < F_REG; ++j)
#pragma unroll
                        for (int e = 0; e < 8; ++e) mask |= (fabsf(a[j][e]) >= lo_f) ? (1u << (8 * j + e)) : 0u;
                    int slot = warp_alloc(__popc(mask), &ss.n_cand);
                    if (mask) {
#pragma unroll
                        for (int j = 0; j < F_REG; ++j) {
                            if ((mask >> (8 * j)) & 0xFFu) {
#pragma unroll
                                for (int e = 0; e < 8; ++e) {
                                    if (mask & (1u << (8 * j + e))) {
                                        if (slot < F_CAND_CAP) {
                                            const uint32_t bits = __float_as_uint(a[j][e]), pos = (uint32_t)f32_oct(j) * 8 + e;
                                            ss.key[slot] = bits & 0x7FFFFFFFu;
                                            ss.meta[slot] = (uint16_t)(((0x7FFFu - pos) << 1) | (bits >> 31));
                                        }
                                        ++slot;
                                    }
                                }
                            }
                        }
                    }
                }
                // ... and the octets in shared memory through a list per warp, one of them per lane and round
                uint16_t* wlist = ss.oct_list + warp * F_WLIST;
                int n_w = 0;
#pragma unroll
                for (int j = F_REG; j < F_SLOTS; ++j) {
                    const bool q = omax[j] >= lo_f;
                    const unsigned bal = __ballot_sync(0xffffffffu, q);
                    const int at = n_w + __popc(bal & ((1u << lane) - 1u));
                    if (q && at < F_WLIST) wlist[at] = (uint16_t)f32_oct(j);
                    n_w += __popc(bal);
                }
                if (lane == 0 && n_w > F_WLIST) ss.over = 1;
                n_w = min(n_w, F_WLIST);
                __syncwarp();
                for (int e0 = 0; e0 < n_w; e0 += 32) {
                    uint32_t o = 0u, mask = 0u;
                    if (e0 + lane < n_w) {
                        o = wlist[e0 + lane];
                        float v[8];
                        octet_from_smem(tile4, (int)o - F_REG * F_NT, 0, swz, v);
#pragma unroll
                        for (int e = 0; e < 8; ++e) mask |= (fabsf(v[e]) >= lo_f) ? (1u << e) : 0u;
                    }
                    int slot = warp_alloc(__popc(mask), &ss.n_cand);
                    while (mask) {
                        const uint32_t pos = (o << 3) + (__ffs(mask) - 1);
                        mask &= mask - 1;
                        if (slot < F_CAND_CAP) {
                            const uint32_t bits = __float_as_uint(tile[f32_phys((int)pos - F_REG_ELEMS, swz)]);
                            ss.key[slot] = bits & 0x7FFFFFFFu;
                            ss.meta[slot] = (uint16_t)(((0x7FFFu - pos) << 1) | (bits >> 31));
                        }
                        ++slot;
                    }
                }
                __syncthreads();
                C = ss.n_cand;
                fast = C <= F_CAND_CAP && ss.over == 0;
                if (cold) {                                          // the levels below count in the same bins
                    if (t < 256) ss.hist[t] = 0;
                    __syncthreads();
                }
            }
            if (fast) {
                ss.sel_bm[t] = 0u; ss.sel_bm[t + F_NT] = 0u;         // (the octet lists are done with; published by the barriers below)
                // 2. the k-th largest candidate by 256-bin radix levels over the live range, every warp reading the
                //    histogram for itself; the last <= 32 members are ranked directly
                unsigned long long lo_c = (unsigned long long)(uint32_t)lo << 16, hi_c = ((unsigned long long)(uint32_t)kmax << 16) | 0xFFFFu;
                unsigned long long kth = 0;
                int k_rem = k;
                auto cand = [&](int i) { return ((unsigned long long)ss.key[i] << 16) | ss.meta[i]; };
                for (int level = 0; level < 7; ++level) {            // 47 bits, 8 a level at least after the first
                    const unsigned long long W1 = hi_c - lo_c;
                    const int sh = W1 < 256u ? 0 : (64 - __clzll(W1)) - 8;
                    if (level > 0) {
                        __syncthreads();
                        if (t < 256) ss.hist[t] = 0;
                        __syncthreads();
                    }
                    for (int i = t; i < C; i += F_NT) {
                        const unsigned long long c = cand(i);
                        if (c >= lo_c && c <= hi_c) atomicAdd(&ss.hist[(int)((c - lo_c) >> sh)], 1);
                    }
                    __syncthreads();
                    int hh[8], sum = 0;
                    {
                        const int4 ha = reinterpret_cast<const int4*>(ss.hist)[lane * 2], hb4 = reinterpret_cast<const int4*>(ss.hist)[lane * 2 + 1];
                        hh[0] = ha.x; hh[1] = ha.y; hh[2] = ha.z; hh[3] = ha.w; hh[4] = hb4.x; hh[5] = hb4.y; hh[6] = hb4.z; hh[7] = hb4.w;
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) sum += hh[j];
                    int suf = sum;                                   // inclusive suffix over lanes >= lane
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) { const int v = __shfl_down_sync(0xffffffffu, suf, d); if (lane + d < 32) suf += v; }
                    const unsigned okm = __ballot_sync(0xffffffffu, suf >= k_rem);
                    const int owner = 31 - __clz(okm);               // highest lane whose suffix reaches k_rem (C >= k: there is one)
                    int above = suf - sum, bsel = 7;
#pragma unroll
                    for (int j = 7; j >= 0; --j) if (bsel == j && above + hh[j] < k_rem) { above += hh[j]; bsel = j - 1; }
                    int hb = 0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) if (j == bsel) hb = hh[j];
                    const int b_star = __shfl_sync(0xffffffffu, lane * 8 + bsel, owner);
                    k_rem -= __shfl_sync(0xffffffffu, above, owner);
                    hb = __shfl_sync(0xffffffffu, hb, owner);
                    lo_c += (unsigned long long)b_star << sh;
                    hi_c = min(hi_c, lo_c + ((1ull << sh) - 1ull));
                    if (sh == 0) { kth = lo_c; break; }
                    if (hb <= 32) {
                        for (int i = t; i < C; i += F_NT) {
                            const unsigned long long c = cand(i);
                            if (c >= lo_c && c <= hi_c) ss.member[atomicAdd(&ss.n_member, 1)] = c;
                        }
                        __syncthreads();
                        const unsigned long long me = lane < hb ? ss.member[lane] : 0ull;
                        int greater = 0;
                        for (int j = 0; j < hb; ++j) greater += (ss.member[j] > me) ? 1 : 0;
                        const unsigned hit = __ballot_sync(0xffffffffu, lane < hb && greater == k_rem - 1);
                        kth = __shfl_sync(0xffffffffu, me, __ffs(hit) - 1);
                        break;
                    }
                }
                // 3. selected positions -> bitmap -> ranks -> I[row], V[row]; selected values in shared memory become 0
                for (int i = t; i < C; i += F_NT) {
                    if (cand(i) >= kth) { const uint32_t pos = 0x7FFFu - (ss.meta[i] >> 1); atomicOr(&ss.sel_bm[pos >> 5], 1u << (pos & 31)); }
                }
                __syncthreads();
                {
                    const uint2 w2 = reinterpret_cast<const uint2*>(ss.sel_bm)[t];
                    const int c0 = __popc(w2.x);
                    int total;
                    const int before = block_exclusive_scan(c0 + __popc(w2.y), ss.scan, total);
                    reinterpret_cast<uint32_t*>(ss.sel_before)[t] = (uint32_t)before | ((uint32_t)(before + c0) << 16);
                }
                __syncthreads();
                for (int i = t; i < C; i += F_NT) {
                    if (cand(i) >= kth) {
                        const uint32_t pos = 0x7FFFu - (ss.meta[i] >> 1), w = pos >> 5;
                        const int rank = ss.sel_before[w] + __popc(ss.sel_bm[w] & ((1u << (pos & 31)) - 1u));
                        i_out[rank] = (int16_t)pos;
                        v_out[rank] = f32_to_bf16_bits_rne(__uint_as_float(ss.key[i] | ((uint32_t)ss.meta[i] << 31)));
                        if (pos >= (uint32_t)F_REG_ELEMS) tile[f32_phys((int)pos - F_REG_ELEMS, swz)] = 0.0f;
                    }
                }
                __syncthreads();
            }
        }
        if (!fast) {
            // general selection (all-zero or infinite tiles, k above the octet count, clustered candidates): bisection on the
            // key bits over the tile, at a cost that does not depend on the data
            uint32_t sel[F_WPT], tw[F_WPT];
            int need = 0;
            const bool all_zero = kmax == 0 && !f32_any_nan(a, tile4, n_oct);     // (a NaN leaves no trace in the maxima)
            if (all_zero) {                                          // every key is zero: the k lowest positions win the ties
#pragma unroll
                for (int i = 0; i < F_WPT; ++i) {
                    const int p0 = (t * F_WPT + i) * 32;
                    sel[i] = (p0 + 32 <= k) ? 0xFFFFFFFFu : (p0 < k ? ((1u << (k - p0)) - 1u) : 0u);
                    tw[i] = 0u;
                }
            } else {
                __syncthreads();                                     // the candidate list becomes the two masks
                if (t < 40) ss.counters[t] = 0;
                __syncthreads();
                int Tk = 0;
                for (int bit = 30; bit >= 0; --bit) {
                    const int c = Tk | (1 << bit);
                    if (f32_count_ge(a, tile4, n_oct, swz, c, &ss.counters[bit]) >= k) Tk = c;
                }
                need = k - f32_count_ge(a, tile4, n_oct, swz, Tk + 1, &ss.counters[32]);
                const float Tf = __int_as_float(Tk);
#pragma unroll
                for (int j = 0; j < F_SLOTS; ++j) {
                    const int o = f32_oct(j);
                    uint32_t gt = 0u, tie = 0u;
                    if (o < n_oct) {
                        float v[8];
                        if (j < F_REG) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] = a[j < F_REG ? j : 0][e];
                        } else {
                            octet_from_smem(tile4, o - F_REG * F_NT, 0, swz, v);
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) {                // (padding ties with T == 0 only, at the highest positions: never selected)
                            gt |= (fabsf(v[e]) > Tf) ? (1u << e) : 0u;
                            tie |= (fabsf(v[e]) == Tf) ? (1u << e) : 0u;
                        }
                    }
                    reinterpret_cast<uint8_t*>(ss.gt_bm)[o] = (uint8_t)gt;
                    reinterpret_cast<uint8_t*>(ss.tie_bm)[o] = (uint8_t)tie;
                }
                __syncthreads();
#pragma unroll
                for (int i = 0; i < F_WPT; ++i) { sel[i] = ss.gt_bm[t * F_WPT + i]; tw[i] = ss.tie_bm[t * F_WPT + i]; }
            }
            f32_resolve(sel, tw, need, ss);
#pragma unroll
            for (int i = 0; i < F_WPT; ++i) {
                uint32_t s = sel[i];
                int p = ss.sel_before[t * F_WPT + i];
                while (s) {
                    const int b = __ffs(s) - 1;
                    s &= s - 1;
                    i_out[p++] = (int16_t)((t * F_WPT + i) * 32 + b);
                }
            }
        }

        // ---- a[I] = 0 where that is still to be done; statistics; e = Q(a) ----------------------------------
        const uint8_t* sel_bytes = reinterpret_cast<const uint8_t*>(ss.sel_bm);
        auto octet_stats = [&](const float (&v)[8], int cnt) {       // as the rounded pair (-min, max): bf16 rounding is monotone and
            float lo = INFINITY, hi = -INFINITY;                     // odd, so a block's statistics are the maximum of its pairs
            if (cnt >= 8) {
                octet_min_max(v, lo, hi);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) if (e < cnt) { lo = fminf(lo, v[e]); hi = fmaxf(hi, v[e]); }
            }
            return pack_bf16x2_rne(-lo, hi);
        };
        auto finish_octet = [&](int o, const float (&v)[8], int hh, uint32_t st) {
            const int cnt = n - o * 8;
            if (cnt <= 0) return;
            if (T.quant_err != nullptr) {                            // alpha == -2: the residual a also goes to the caller's buffer
                float* qe = reinterpret_cast<float*>(T.quant_err) + base + o * 8;
                if (cnt >= 8 && aligned16(qe)) {
                    reinterpret_cast<float4*>(qe)[hh] = make_float4(v[0], v[1], v[2], v[3]);
                    reinterpret_cast<float4*>(qe)[hh ^ 1] = make_float4(v[4], v[5], v[6], v[7]);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) if (e < cnt) qe[e ^ (hh << 2)] = v[e];
                }
            }
            const uint16_t mn_b = (uint16_t)((st & 0xFFFFu) ^ 0x8000u), mx_b = (uint16_t)(st >> 16);
            if ((o & (lanes_per_qb - 1)) == 0) { mn_g[o >> oshift] = mn_b; mx_g[o >> oshift] = mx_b; }
            const QParams q = qparams(mn_b, mx_b);
            uint32_t w;
            if (cnt >= 8 && step_in_range(q)) {
                w = encode_octet_div_f32<true>(v, div_consts(q));    // values can lie outside statistics rounded to bf16: clamped
            } else {
                float y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = v[e];
                w = encode_octet_scalar(y, q.mn, q.u, min(cnt, 8));
            }
            w = rotate_codes(w, hh);
            if (ef_al4 && cnt >= 8) reinterpret_cast<uint32_t*>(ef)[o] = w;
            else
                for (int b = 0; b < 4; ++b) if (2 * b < cnt) ef[o * 4 + b] = (uint8_t)(w >> (8 * b));
        };
        auto take_selected = [&](int o, float (&v)[8], bool emit) {
            const uint32_t sel = sel_bytes[o];
            if (!sel) return;
            int p = ss.sel_before[o >> 2] + __popc(ss.sel_bm[o >> 2] & ((1u << (8 * (o & 3))) - 1u));
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (sel & (1u << e)) {
                    if (emit) v_out[p++] = f32_to_bf16_bits_rne(v[e]);
                    v[e] = 0.0f;
                }
        };
        if (swz && fast) {
            // registers: the four lanes that hold a block's eight octets meet in two shuffles
            const uint32_t sel2 = reinterpret_cast<const uint16_t*>(sel_bytes)[t];
            float lo = INFINITY, hi = -INFINITY;
#pragma unroll
            for (int j = 0; j < F_REG; ++j) {
#pragma unroll
                for (int e = 0; e < 8; ++e) a[j][e] = (sel2 & (1u << (8 * j + e))) ? 0.0f : a[j][e];
                float l, u;
                octet_min_max(a[j], l, u);
                lo = fminf(lo, l); hi = fmaxf(hi, u);
            }
            if (T.quant_err != nullptr) {                            // alpha == -2: the residual a also goes to the caller's buffer
                float* qe = reinterpret_cast<float*>(T.quant_err) + base;
                const bool vec = aligned16(qe);
#pragma unroll
                for (int j = 0; j < F_REG; ++j)
#pragma unroll
                    for (int e = 0; e < 8; e += 4) {
                        float* to = qe + f32_oct(j) * 8 + e;
                        if (vec) *reinterpret_cast<float4*>(to) = make_float4(a[j][e], a[j][e + 1], a[j][e + 2], a[j][e + 3]);
                        else { to[0] = a[j][e]; to[1] = a[j][e + 1]; to[2] = a[j][e + 2]; to[3] = a[j][e + 3]; }
                    }
                for (int c = t; c < n_so * 2; c += F_NT) {
                    const float4 v = tile4[c ^ ((c >> 4) & 7)];
                    float* to = qe + F_REG_ELEMS + c * 4;
                    if (vec) *reinterpret_cast<float4*>(to) = v;
                    else { to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w; }
                }
            }
            uint32_t st = pack_bf16x2_rne(-lo, hi);
            st = max_bf16x2(st, __shfl_xor_sync(0xffffffffu, st, 1));
            st = max_bf16x2(st, __shfl_xor_sync(0xffffffffu, st, 2));
            const uint16_t mn_b = (uint16_t)((st & 0xFFFFu) ^ 0x8000u), mx_b = (uint16_t)(st >> 16);
            if ((t & 3) == 0) { mn_g[t >> 2] = mn_b; mx_g[t >> 2] = mx_b; }
            const QParams q = qparams(mn_b, mx_b);
            uint2 w;
            if (step_in_range(q)) {
                const DivConsts dc = div_consts(q);
                w.x = encode_octet_div_f32<true>(a[0], dc);
                w.y = encode_octet_div_f32<true>(a[1], dc);
            } else {
                float y[F_REG][8];
#pragma unroll
                for (int j = 0; j < F_REG; ++j)
#pragma unroll
                    for (int e = 0; e < 8; ++e) y[j][e] = a[j][e];
                w.x = encode_octet_scalar(y[0], q.mn, q.u, 8);
                w.y = encode_octet_scalar(y[1], q.mn, q.u, 8);
            }
            reinterpret_cast<uint2*>(ef)[t] = w;
            stats_encode_rows(tile4, n_so >> 3, mn_g + F_REG_ELEMS / 64, mx_g + F_REG_ELEMS / 64, ef + F_REG_ELEMS / 2);
        } else {
            {
                uint32_t st[F_REG];
#pragma unroll
                for (int j = 0; j < F_REG; ++j) {
                    const int o = f32_oct(j);
                    take_selected(o, a[j], !fast);
                    st[j] = octet_stats(a[j], n - o * 8);
                }
                if (oshift > 0) {                                    // both octets lie in one block
                    st[0] = max_bf16x2(st[0], st[1]);
                    for (int off = 1; off < (lanes_per_qb >> 1); off <<= 1) st[0] = max_bf16x2(st[0], __shfl_xor_sync(0xffffffffu, st[0], off));
                    st[1] = st[0];
                }
#pragma unroll
                for (int j = 0; j < F_REG; ++j) finish_octet(f32_oct(j), a[j], 0, st[j]);
            }
#pragma unroll 1
            for (int o = t + F_REG * F_NT; (o & ~31) < n_oct; o += F_NT) {   // whole warps: the lanes of a block meet in the shuffles
                float v[8];
                const int hh = fast ? h : 0;
                if (o < n_oct) {
                    octet_from_smem(tile4, o - F_REG * F_NT, hh, swz, v);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
                }
                if (!fast) take_selected(o, v, true);
                uint32_t st = octet_stats(v, n - o * 8);
                for (int off = 1; off < lanes_per_qb; off <<= 1) st = max_bf16x2(st, __shfl_xor_sync(0xffffffffu, st, off));
                finish_octet(o, v, hh, st);
            }
        }
        __syncthreads();                                             // tile and scratch are overwritten by the next load
    }
}

// Returns 1 (without launching) when two CTAs of its shared memory do not fit an SM (tiles above 29 900 elements or so), or
// when the selection's candidates would not fit their list: with c of 3632 octets at the bound (k <= c <= k + 192) a tile of
// independent values holds about -3632 ln(1 - c / 3632) candidates, 2648 at c = 1880 and 3069 at c = 1880 + 192 (means: a
// tile that comes out above the list's 3072 goes to the bisection).  The one-tile kernel, whose
// list is longer, is the faster one from there on (k = 2325: 1165 us a step of 67 M elements, most of it in kernel B).
int launch_ef_topk_quant_f32(const mab_tensor* dev_tensors, int n_tensors, int total_units, int qbs, int max_dbs, int max_k, int allowing, cudaStream_t s) {
    int qshift = 0;
    while ((1 << qshift) < qbs) ++qshift;
    const int tile_bytes = (std::max(0, ((max_dbs + 7) & ~7) - F_REG_ELEMS) * 4 + 127) & ~127;
    const int smem = tile_bytes + (int)sizeof(SmemF);
    const int fixed = (int)sizeof(int) * (WIN_MAX_TENSORS + 1) + 128 + 1024;     // static arrays and the per-CTA reservation
    if (max_k > F_MAX_K || F_CTAS * (smem + fixed) > device_max_optin_smem() + 1024) return 1;
    const int grid = (int)std::min<int64_t>(total_units, (int64_t)device_sm_count() * F_CTAS);
    MAB_CUDA_TRY(cudaFuncSetAttribute(ef_topk_quant_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    ef_topk_quant_f32_kernel<<<grid, F_NT, smem, s>>>(dev_tensors, n_tensors, total_units, qshift, tile_bytes, allowing);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "ef_topk_quant_f32_kernel launch");
    return MAB_OK;
}

int copy_timeout_f32_split(int* out, bool clear) {
    cudaError_t e = cudaMemcpyFromSymbol(out, g_copy_timeout_f32, sizeof(int));
    if (e == cudaSuccess && clear) { const int z = 0; e = cudaMemcpyToSymbol(g_copy_timeout_f32, &z, sizeof(int)); }
    return e == cudaSuccess ? MAB_OK : cuda_fail(e, "mab_device_error");
}

}  // namespace mab
