// Block top-k by itself (micro_adam.py:193-200): the positions of the k largest magnitudes of every block, ascending, ties to the lower
// position; NaN last.
//
// A block is not held anywhere: one pass over it leaves the maxima of its octets in registers (sixteen a thread), a bound of the k-th
// magnitude is searched on them, and only the octets that reach the bound, one in eight or so, are read again, from L2.  Their values that
// reach it are the candidates, among which the k-th is found by radix levels, and the selected ones have their places in the row by a
// bitmap and a prefix count.  So a CTA needs 27 KB and 40 registers a thread, and six of them share an SM: one block's chain of
// phases overlaps the others' reads.  Where an SM has one block at most, its
// CTA has 1024 threads (us, 256 and 1024: 69 blocks 13.6 and 9.5, 207 blocks 14.4 and 17.5).  Bound by HBM and, past one wave of CTAs, by the
// phases: 25.6 M fp32 elements 27 us, 3.9 TB/s; held in the registers of one CTA of 1024 threads per SM it took 57, 60 M with k = 5 % 155 (101 now).
#include "common.cuh"
#include "select.cuh"
#include "fused.cuh"

namespace mab {
namespace topk {

constexpr int K_NT = 256, K_CTAS = 6;        // threads of a CTA, and CTAs per SM the registers are sized for ...
constexpr int K_NT_FEW = 1024;               // ... and the threads where an SM has one block at most
constexpr int K_CAP = 3072;                  // candidates
constexpr int K_INF = 0x7F800000;            // keys (|value| bits) above it are NaN

struct __align__(16) Smem {
    union {
        struct {                             // candidates: |value| bits (for bf16 their upper half) and 0x7FFF - position; "larger is better"
                                             //   contains the tie rule
            uint32_t key[K_CAP];
            uint16_t pos[K_CAP];
        };
        struct { uint32_t gt_bm[SEL_WORDS], tie_bm[SEL_WORDS]; };   // general selection: key > T, key == T
    };
    union {
        struct {
            uint32_t sel_bm[SEL_WORDS];      // selected positions
            uint16_t sel_before[SEL_WORDS];  // selected positions in lower words
        };
        uint16_t list[SEL_MAX_TILE / 8];     // before the selection: octets that reach the bound, a part per warp
    };
    unsigned long long member[32];
    int hist[256];
    int rot[64];                             // octets at each threshold of the search; [63]: candidates above a tied bound
    int scan[36];
    int n_member, n_cand, kmax;
};

template <typename T> struct Octet;           // eight values as they are in memory
template <> struct Octet<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) { a = __ldg(reinterpret_cast<const float4*>(p)); b = __ldg(reinterpret_cast<const float4*>(p) + 1); }
    __device__ __forceinline__ void values(float (&v)[8]) const {
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
};
template <> struct Octet<uint16_t> {
    uint4 a;
    __device__ __forceinline__ void load(const uint16_t* p) { a = __ldg(reinterpret_cast<const uint4*>(p)); }
    __device__ __forceinline__ void values(float (&v)[8]) const {
        v[0] = __uint_as_float(a.x << 16); v[1] = __uint_as_float(a.x & 0xFFFF0000u);
        v[2] = __uint_as_float(a.y << 16); v[3] = __uint_as_float(a.y & 0xFFFF0000u);
        v[4] = __uint_as_float(a.z << 16); v[5] = __uint_as_float(a.z & 0xFFFF0000u);
        v[6] = __uint_as_float(a.w << 16); v[7] = __uint_as_float(a.w & 0xFFFF0000u);
    }
};

// Octet o of a block of n values, 0 past its end.
template <typename T>
__device__ __forceinline__ void load_octet(const T* x, int o, int n, bool vec, float (&v)[8]) {
    if (vec && o * 8 + 8 <= n) {
        Octet<T> r;
        r.load(x + o * 8);
        r.values(v);
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = o * 8 + e < n ? Elem<T>::load(x, o * 8 + e) : 0.0f;
    }
}

__device__ __forceinline__ int key_of(float v) { return __float_as_int(fabsf(v)); }

// A level of the radix search, every warp for itself: the bin of the k_rem-th largest entry (hist[b]: entries of bin b); k_rem then counts
// within that bin, whose size is returned in `size`.  -1: there are fewer entries.
__device__ __forceinline__ int kth_bin(const int* hist, int& k_rem, int& size) {
    const int lane = lane_id();
    int h[8], sum = 0;
    {
        const int4 a = reinterpret_cast<const int4*>(hist)[lane * 2], b = reinterpret_cast<const int4*>(hist)[lane * 2 + 1];
        h[0] = a.x; h[1] = a.y; h[2] = a.z; h[3] = a.w; h[4] = b.x; h[5] = b.y; h[6] = b.z; h[7] = b.w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += h[j];
    int suf = sum;                                           // inclusive suffix over lanes >= lane
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const int v = __shfl_down_sync(0xffffffffu, suf, d); if (lane + d < 32) suf += v; }
    const unsigned reach = __ballot_sync(0xffffffffu, suf >= k_rem);
    if (reach == 0u) return -1;
    const int owner = 31 - __clz(reach);
    int above = suf - sum, b = 7, mine = h[7];
#pragma unroll
    for (int j = 7; j > 0; --j) if (b == j && above + h[j] < k_rem) { above += h[j]; b = j - 1; mine = h[j - 1]; }
    const int bin = __shfl_sync(0xffffffffu, lane * 8 + b, owner);
    k_rem -= __shfl_sync(0xffffffffu, above, owner);
    size = __shfl_sync(0xffffffffu, mine, owner);
    return bin;
}

// The `keep` lowest of the set bits (none where it is not positive).
__device__ __forceinline__ uint32_t lowest_bits(uint32_t bits, int keep) {
    if (keep <= 0) return 0u;
    while (__popc(bits) > keep) bits &= ~(0x80000000u >> __clz(bits));
    return bits;
}

// The selection of any block (zeros, infinities, equal magnitudes, k beyond the octets, more candidates than the list holds): the k-th key by
// digits of eight bits between two bounds, `lo`, which at least k numbers reach (0: none known), and the largest, over the whole block, read anew every
// time; then masks of the larger and equal keys, and the row by a warp per 32 positions.  Zeros are not counted: where fewer than k
// numbers are larger the k-th is one.  A NaN is selected only where the block holds fewer than k numbers: a row has k different positions of
// its block always (left short, it would keep the end of the row it replaces, whose positions may be the same again).  Bound by the reads' latency
// and the shared-memory counters.  us, 149 blocks (4.3 M fp32 elements), and in parentheses with four digits of eight bits from the top, an octet at a
// time, a thread writing its 128 positions: zeros 13.6 (56), equal magnitudes 31 (73), infinities 35 (48), k = 20 % 36 (53), 50 % 36 (66), all 20 (82);
// 881 blocks, zeros 32 (119), k = 20 % 78 (122), all 63 (299).
// Every thread of the CTA calls.
template <typename T, int NT>
__device__ __noinline__ void select_general(const T* x, int n, int k, int lo, int kmax, bool vec, Smem& ss, int16_t* out) {
    constexpr int K_WPT = SEL_WORDS / NT;                    // bitmap words per thread
    constexpr int ZB = sizeof(T) == 2 ? 16 : 0;              // low key bits that are always zero
    constexpr int B = 2;                                     // octets a thread has in flight (with four the bf16 kernel spills)
    const int t = threadIdx.x, n_oct = (n + 7) >> 3;
    auto each_octet = [&](auto&& f) {
        int o = t;
        if (vec)
            for (; o + (B - 1) * NT < n >> 3; o += B * NT) {
                Octet<T> r[B];
#pragma unroll
                for (int i = 0; i < B; ++i) r[i].load(x + (o + i * NT) * 8);
#pragma unroll
                for (int i = 0; i < B; ++i) { float v[8]; r[i].values(v); f(o + i * NT, v); }
            }
        for (; o < n_oct; o += NT) { float v[8]; load_octet(x, o, n, vec, v); f(o, v); }
    };
    const int inf = K_INF >> ZB;
    int lo_k = lo >> ZB, hi_k = kmax >> ZB, rem = k;
    while (lo_k < hi_k) {
        const int span = hi_k - lo_k, sh = span < 256 ? 0 : (32 - __clz(span)) - 8;
        __syncthreads();
        if (t < 256) ss.hist[t] = 0;
        __syncthreads();
        each_octet([&](int, const float (&v)[8]) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int key = key_of(v[e]) >> ZB;
                if (key >= lo_k && key <= hi_k && key != 0) atomicAdd(&ss.hist[(key - lo_k) >> sh], 1);
            }
        });
        __syncthreads();
        int size = 0;
        const int bin = kth_bin(ss.hist, rem, size);
        if (bin < 0) { lo_k = 0; break; }                    // fewer than k numbers above zero
        lo_k += bin << sh;
        hi_k = min(hi_k, lo_k + (1 << sh) - 1);
        if (rem == size) { lo_k = max(lo_k - 1, 0); break; } // all of the bin: the keys above what lies below it
    }
    const int kth = lo_k;
    each_octet([&](int o, const float (&v)[8]) {
        uint32_t gt = 0u, tie = 0u;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int key = key_of(v[e]) >> ZB;
            gt |= key > kth && key <= inf ? 1u << e : 0u;
            tie |= key == kth ? 1u << e : 0u;
        }
        reinterpret_cast<uint8_t*>(ss.gt_bm)[o] = (uint8_t)gt;
        reinterpret_cast<uint8_t*>(ss.tie_bm)[o] = (uint8_t)(n - o * 8 >= 8 ? tie : tie & ((1u << (n - o * 8)) - 1u));   // (not what lies past the end)
    });
    for (int o = n_oct + t; o < SEL_MAX_TILE / 8; o += NT) { reinterpret_cast<uint8_t*>(ss.gt_bm)[o] = 0; reinterpret_cast<uint8_t*>(ss.tie_bm)[o] = 0; }
    __syncthreads();
    uint32_t sel[K_WPT], tw[K_WPT];
    int ties = 0, cnt = 0, total;
#pragma unroll
    for (int i = 0; i < K_WPT; ++i) { sel[i] = ss.gt_bm[t * K_WPT + i]; tw[i] = ss.tie_bm[t * K_WPT + i]; ties += __popc(tw[i]); cnt += __popc(sel[i]); }
    int before = block_exclusive_scan(ties, ss.scan, total);
    __syncthreads();
    const int larger = [&] { int all; block_exclusive_scan(cnt, ss.scan, all); return all; }();
    __syncthreads();
    const int missing = k - larger - total;                  // > 0: fewer than k numbers, and every one of them is in a mask
    cnt = 0;
#pragma unroll
    for (int i = 0; i < K_WPT; ++i) {
        const int keep = k - larger - before;                // the lowest positions among the equal ones
        before += __popc(tw[i]);
        sel[i] |= lowest_bits(tw[i], keep);
        cnt += __popc(sel[i]);
    }
    if (missing > 0) {                                       // uniform; the lowest positions that hold a NaN complete the row
        int nans = 0;
#pragma unroll
        for (int i = 0; i < K_WPT; ++i) {
            const int left = n - (t * K_WPT + i) * 32;
            tw[i] = left >= 32 ? ~sel[i] : left > 0 ? ~sel[i] & ((1u << left) - 1u) : 0u;
            nans += __popc(tw[i]);
        }
        before = block_exclusive_scan(nans, ss.scan, total);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < K_WPT; ++i) {
            const uint32_t add = lowest_bits(tw[i], missing - before);
            before += __popc(tw[i]);
            sel[i] |= add;
            cnt += __popc(add);
        }
    }
    int to = block_exclusive_scan(cnt, ss.scan, total);
#pragma unroll
    for (int i = 0; i < K_WPT; ++i) { ss.sel_bm[t * K_WPT + i] = sel[i]; ss.sel_before[t * K_WPT + i] = (uint16_t)to; to += __popc(sel[i]); }
    __syncthreads();
#pragma unroll 4
    for (int w = warp_id(); w < (n + 31) >> 5; w += NT / 32) {
        const uint32_t s = ss.sel_bm[w];
        if (s >> lane_id() & 1u) out[ss.sel_before[w] + __popc(s & ((1u << lane_id()) - 1u))] = (int16_t)(w * 32 + lane_id());
    }
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT, NT == K_NT ? K_CTAS : 1)
block_topk_kernel(int64_t d, int dbs, int nfull, int k_many, int k_few, const T* __restrict__ x_all, int16_t* __restrict__ out_all) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& ss = *reinterpret_cast<Smem*>(smem_raw);
    constexpr int K_SLOTS = SEL_MAX_TILE / 8 / NT;           // octets per thread
    constexpr int ZB = sizeof(T) == 2 ? 16 : 0;              // low key bits that are always zero
    constexpr int K_WPT = SEL_WORDS / NT;                    // bitmap words per thread
    const int t = threadIdx.x, lane = lane_id();
    uint16_t* const list = ss.list + warp_id() * (32 * K_SLOTS);
    const int nblocks = nfull + (k_few > 0 ? 1 : 0);
    const TileRange range = tiles_of_cta(nblocks, gridDim.x, blockIdx.x);
    int guess = 0;                                           // bound found for the block before, as key bits
    for (int blk = range.first; blk < range.end; ++blk) {
        const int64_t base = (int64_t)blk * dbs;
        const int n = (int)min((int64_t)dbs, d - base), k = blk < nfull ? k_many : k_few, n_oct = (n + 7) >> 3;
        const T* x = x_all + base;
        int16_t* out = out_all + (int64_t)blk * k_many;
        const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
        if (t == 0) { ss.kmax = 0; ss.n_member = 0; ss.n_cand = 0; }
        if (t < 64) ss.rot[t] = 0;
        if (t < 256) ss.hist[t] = 0;
        // ---- the octets' maxima: never a NaN (0 for an octet that holds nothing else) ----------------------------------
        float omax[K_SLOTS];
        float tm = 0.0f;
#pragma unroll
        for (int j = 0; j < K_SLOTS; ++j) {
            const int o = j * NT + t;
            omax[j] = 0.0f;
            if (o < n_oct) {
                float v[8];
                load_octet(x, o, n, vec, v);
                omax[j] = fmaxf(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))), fmaxf(fmaxf(fabsf(v[4]), fabsf(v[5])), fmaxf(fabsf(v[6]), fmaxf(fabsf(v[7]), 0.0f))));
            }
            tm = fmaxf(tm, omax[j]);
        }
        __syncthreads();
        {
            const int wm = __reduce_max_sync(0xffffffffu, __float_as_int(tm));
            if (lane == 0 && wm) atomicMax(&ss.kmax, wm);
        }
        __syncthreads();
        const int kmax = ss.kmax;
        bool fast = false;
        int C = 0, lo = 0;
        bool tied = false;                                    // more octets than wanted reach the bound, and no higher one is reached by k
        if (kmax > 0 && kmax < K_INF && k <= n_oct) {
            // ---- a bound that at least k octets reach and at most about 1.5 k, fewer where that would bring more candidates than the list holds
            const int accept = k + (k > 1024 ? 192 : (k >> 1) + 8);
            int hi = kmax + 1, step = 1 << 20;
            int gq = guess;
            bool have_lo = false, have_hi = false, search = true;
            const bool cold = guess <= 0 || guess > kmax;    // no bound from a block before: the histogram of the maxima gives one
            if (cold) {
                const int c = bound_from_histogram(omax, kmax, k, ss.hist, lo, hi);
                have_lo = c > 0; have_hi = true;
                search = hi - lo > 1 && !(c > 0 && c <= accept);
                gq = have_lo ? lo + ((hi - lo) >> 1) : max(hi - step, 1);
            }
            for (int it = 0; search && it < 63; ++it) {
                int mine = 0;
#pragma unroll
                for (int j = 0; j < K_SLOTS; ++j) mine += __float_as_int(omax[j]) >= gq ? 1 : 0;
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
            tied = hi - lo <= 1;
            if (lo > 0) {                   // (an octet that reaches the bound is a candidate at least)
                // ---- candidates: the octets that reach the bound through a list per warp, one of them per lane and round ----------
                const float lo_f = __int_as_float(lo);
                int n_w = 0;
#pragma unroll
                for (int j = 0; j < K_SLOTS; ++j) {
                    const bool hit = omax[j] >= lo_f;
                    const unsigned hits = __ballot_sync(0xffffffffu, hit);
                    if (hit) list[n_w + __popc(hits & ((1u << lane) - 1u))] = (uint16_t)(j * NT + t);
                    n_w += __popc(hits);
                }
                __syncwarp();
                for (int q0 = 0; q0 < n_w; q0 += 32) {
                    int o = 0;
                    uint32_t mask = 0u;
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
                    if (q0 + lane < n_w) {
                        o = list[q0 + lane];
                        load_octet(x, o, n, vec, v);
#pragma unroll
                        for (int e = 0; e < 8; ++e) mask |= fabsf(v[e]) >= lo_f ? 1u << e : 0u;
                    }
                    int slot = warp_alloc(__popc(mask), &ss.n_cand);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (mask & (1u << e)) {
                            if (slot < K_CAP) { ss.key[slot] = (uint32_t)key_of(v[e]) >> ZB; ss.pos[slot] = (uint16_t)(0x7FFF - (o * 8 + e)); }
                            ++slot;
                        }
                }
                __syncthreads();
                C = ss.n_cand;
                fast = C <= K_CAP;
                if (cold) {                                  // the levels below count in the same bins
                    if (t < 256) ss.hist[t] = 0;
                    __syncthreads();
                }
            }
        }
        if (fast) {
            // ---- the k-th largest candidate by radix levels over the live range; the last <= 32 members are ranked directly --------
#pragma unroll
            for (int i = 0; i < K_WPT; ++i) ss.sel_bm[t + i * NT] = 0u;   // (the lists are done with; published by the barriers below)
            unsigned long long lo_c = (unsigned long long)(uint32_t)(lo >> ZB) << 15, hi_c = ((unsigned long long)(uint32_t)(kmax >> ZB) << 15) | 0x7FFFu;
            unsigned long long kth = 0;
            int k_rem = k;
            if (tied) {                                      // often their k-th is one of many with the bound's magnitude: then the positions decide
                int above = 0;
                for (int i = t; i < C; i += NT) above += ss.key[i] > (uint32_t)(lo >> ZB) ? 1 : 0;
                above = __reduce_add_sync(0xffffffffu, above);
                if (lane == 0 && above) atomicAdd(&ss.rot[63], above);
                __syncthreads();
                if (ss.rot[63] < k) { k_rem = k - ss.rot[63]; hi_c = lo_c | 0x7FFFu; }
            }
            auto cand = [&](int i) { return ((unsigned long long)ss.key[i] << 15) | ss.pos[i]; };
            for (int level = 0; level < 7; ++level) {        // 46 bits, 8 a level at least after the first
                const unsigned long long W1 = hi_c - lo_c;
                const int sh = W1 < 256u ? 0 : (64 - __clzll(W1)) - 8;
                if (level > 0) {
                    __syncthreads();
                    if (t < 256) ss.hist[t] = 0;
                    __syncthreads();
                }
                for (int i = t; i < C; i += NT) {
                    const unsigned long long c = cand(i);
                    if (c >= lo_c && c <= hi_c) atomicAdd(&ss.hist[(int)((c - lo_c) >> sh)], 1);
                }
                __syncthreads();
                int size = 0;
                const int bin = kth_bin(ss.hist, k_rem, size);   // (C >= k: there is one)
                lo_c += (unsigned long long)bin << sh;
                hi_c = min(hi_c, lo_c + ((1ull << sh) - 1ull));
                if (sh == 0) { kth = lo_c; break; }
                if (size <= 32) {
                    for (int i = t; i < C; i += NT) {
                        const unsigned long long c = cand(i);
                        if (c >= lo_c && c <= hi_c) ss.member[atomicAdd(&ss.n_member, 1)] = c;
                    }
                    __syncthreads();
                    const unsigned long long me = lane < size ? ss.member[lane] : 0ull;
                    int greater = 0;
                    for (int j = 0; j < size; ++j) greater += ss.member[j] > me ? 1 : 0;
                    kth = __shfl_sync(0xffffffffu, me, __ffs(__ballot_sync(0xffffffffu, lane < size && greater == k_rem - 1)) - 1);
                    break;
                }
            }
            // ---- selected positions -> bitmap -> places in the row -------------------------------------------------------
            for (int i = t; i < C; i += NT)
                if (cand(i) >= kth) { const uint32_t pos = 0x7FFFu - ss.pos[i]; atomicOr(&ss.sel_bm[pos >> 5], 1u << (pos & 31)); }
            __syncthreads();
            {
                int cnt = 0, total;
#pragma unroll
                for (int i = 0; i < K_WPT; ++i) cnt += __popc(ss.sel_bm[t * K_WPT + i]);
                int before = block_exclusive_scan(cnt, ss.scan, total);
#pragma unroll
                for (int i = 0; i < K_WPT; ++i) { ss.sel_before[t * K_WPT + i] = (uint16_t)before; before += __popc(ss.sel_bm[t * K_WPT + i]); }
            }
            __syncthreads();
            for (int i = t; i < C; i += NT)
                if (cand(i) >= kth) {
                    const uint32_t pos = 0x7FFFu - ss.pos[i], w = pos >> 5;
                    out[ss.sel_before[w] + __popc(ss.sel_bm[w] & ((1u << (pos & 31)) - 1u))] = (int16_t)pos;
                }
        } else {
            select_general<T, NT>(x, n, k, lo, kmax, vec, ss, out);
        }
        __syncthreads();                                     // everything is used again
    }
}

}  // namespace topk

template <typename T>
static int launch(int64_t d, int dbs, int nfull, int k_many, int k_few, const T* x, int16_t* out, cudaStream_t s) {
    constexpr int smem = (int)sizeof(topk::Smem);
    const int64_t blocks = (int64_t)nfull + (k_few > 0 ? 1 : 0);
    const bool few = blocks <= device_sm_count();
    const int per_sm = few ? 1 : std::max(1, std::min(topk::K_CTAS, (device_max_optin_smem() + 1024) / (smem + 1024)));
    const int grid = (int)std::min<int64_t>(blocks, (int64_t)device_sm_count() * per_sm);
    auto run = [&](auto kern, int threads) -> int {
        MAB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kern<<<grid, threads, smem, s>>>(d, dbs, nfull, k_many, k_few, x, out);
        return MAB_OK;
    };
    const int rc = few ? run(topk::block_topk_kernel<T, topk::K_NT_FEW>, topk::K_NT_FEW) : run(topk::block_topk_kernel<T, topk::K_NT>, topk::K_NT);
    if (rc) return rc;
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? MAB_OK : cuda_fail(e, "block_topk_kernel launch");
}

int launch_block_topk(int64_t d, int dbs, int nfull, int k_many, int k_few, const void* x, int dtype, int16_t* out, cudaStream_t s) {
    return dtype == MAB_F32 ? launch(d, dbs, nfull, k_many, k_few, static_cast<const float*>(x), out, s)
                            : launch(d, dbs, nfull, k_many, k_few, static_cast<const uint16_t*>(x), out, s);
}

}  // namespace mab
