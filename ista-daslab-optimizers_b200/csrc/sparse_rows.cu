// The two consumers of the (I, V) ring buffer outside MicroAdam: Sparse M-FAC's scalar products of a
// dense vector with every sparse row and its linear combination of the rows
// (sparse_mfac/sparse_core_mfac_w_ef.py:188-221, native calls SP and LCG of ista_daslab_cuda_sparse_mfac).
// Row r of the buffer holds, for top-k block b, the in-block positions I[r, b * kbs + j] and the
// values V[r, b * kbs + j]; entry j of a row addresses element (j / kbs) * dbs + I[r, j].
//
// Both results are reproducible bit for bit: fixed assignment of entries to threads, fixed
// reduction trees, rows accumulated in row order.
#include <cooperative_groups.h>
#include "common.cuh"
#include "codec_fast.cuh"
#include "window.cuh"

namespace mab {

constexpr int SPR_SR = 14592;         // elements of a block one CTA accumulates at a time (57 * 256): a 29 056-element block is two ranges
constexpr int SPR_THREADS = 384;      // three CTAs of 58 KB of accumulators per SM, 56 registers a thread (512 threads of 40 spill: 98 us, now 78)
static_assert(MAB_MAX_WINDOW <= SPR_THREADS, "a thread brings one row's multiplier");
// Rows whose entries a thread fetches at once; (row, round) pairs of long rows (bf16 values, 25.6 M elements, 32 rows of 5 %: 6 189 us, 8 198; of
// 1 %: 6 66.6, 8 65.4, products behind the barriers).
template <typename TV, bool LONG> constexpr int SPR_AHEAD = LONG && sizeof(TV) == 2 ? 6 : 8;

constexpr int SP_THREADS = 512;
constexpr int SP_CLUSTER = 8;         // CTAs per row (the portable cluster size) ...
constexpr int SP_ONE_CTA = 2048;      // ... and the longest row one CTA takes (2003 entries: 3.3 us, 3.6 by a cluster; 3005: 3.9 and 3.7)

template <typename T> __device__ __forceinline__ float load_value(const void* p, int64_t i);
template <> __device__ __forceinline__ float load_value<float>(const void* p, int64_t i) { return reinterpret_cast<const float*>(p)[i]; }
template <> __device__ __forceinline__ float load_value<uint16_t>(const void* p, int64_t i) { return bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(p)[i]); }

// out[0 .. 16 bytes) += v, element by element in out's type.
template <typename TO> constexpr int SPR_VEC = 16 / (int)sizeof(TO);
__device__ __forceinline__ void add_vector(float* o, const float* v) {
    float4 a = *reinterpret_cast<float4*>(o);
    const float4 b = *reinterpret_cast<const float4*>(v);
    a.x = __fadd_rn(a.x, b.x); a.y = __fadd_rn(a.y, b.y); a.z = __fadd_rn(a.z, b.z); a.w = __fadd_rn(a.w, b.w);
    *reinterpret_cast<float4*>(o) = a;
}
__device__ __forceinline__ void add_vector(uint16_t* o, const float* v) {
    uint4 a = *reinterpret_cast<uint4*>(o);
    const float4 b = reinterpret_cast<const float4*>(v)[0], c = reinterpret_cast<const float4*>(v)[1];
    auto pair = [](uint32_t w, float x, float y) {
        return pack_bf16x2_rne(__fadd_rn(__uint_as_float(w << 16), x), __fadd_rn(__uint_as_float(w & 0xFFFF0000u), y));
    };
    a.x = pair(a.x, b.x, b.y); a.y = pair(a.y, b.z, b.w); a.z = pair(a.z, c.x, c.y); a.w = pair(a.w, c.z, c.w);
    *reinterpret_cast<uint4*>(o) = a;
}

// acc + the products of a row's entries [first, end) of one top-k block with that block of g, by one warp.
template <typename TG, typename TV>
__device__ __forceinline__ float dot_entries(float acc, const TG* gb, const int16_t* __restrict__ I, const void* __restrict__ V, int64_t row, int first, int end) {
    constexpr int U = 5;                                     // entries a lane has in flight (32 rows of 1 278 028: 4 124-147 us, 5 111, 6 115, 8 123)
    for (int j0 = first + lane_id(); j0 < end; j0 += 32 * U) {
        int pos[U];
        float val[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
            const int j = j0 + 32 * i;
            pos[i] = j < end ? (int)I[row + j] : 0;
            val[i] = j < end ? load_value<TV>(V, row + j) : 0.0f;
        }
        float x[U];
#pragma unroll
        for (int i = 0; i < U; ++i) x[i] = j0 + 32 * i < end ? Elem<TG>::load(gb, pos[i]) : 0.0f;
#pragma unroll
        for (int i = 0; i < U; ++i) acc = __fadd_rn(acc, __fmul_rn(val[i], x[i]));
    }
    return acc;
}

// The sum of `acc` over the CTAs of a cluster, to *out; lanes, warps and CTAs (through distributed shared memory) in a fixed order.
template <int CTAS>
__device__ __forceinline__ void dot_sum(float acc, float* s_part, float* s_cta, float* out) {
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int rank = CTAS > 1 ? (int)cluster.block_rank() : 0;
#pragma unroll
    for (int o = 16; o; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    if (lane_id() == 0) s_part[warp_id()] = acc;
    if constexpr (CTAS > 1) cluster.sync();                  // (every CTA of the cluster runs by now: its shared memory may be written)
    else __syncthreads();
    if (threadIdx.x == 0) {
        float total = 0.0f;
        for (int w = 0; w < SP_THREADS / 32; ++w) total = __fadd_rn(total, s_part[w]);
        if constexpr (CTAS > 1) *cluster.map_shared_rank(&s_cta[rank], 0) = total;
        else *out = total;
    }
    if constexpr (CTAS > 1) {
        cluster.sync();
        if (rank == 0 && threadIdx.x == 0) {
            float total = 0.0f;
            for (int c = 0; c < CTAS; ++c) total = __fadd_rn(total, s_cta[c]);
            *out = total;
        }
    }
}

// out[r] = sum_j V[r, j] * g[(j / kbs) * dbs + I[r, j]]: a cluster of 8 CTAs per row (one CTA per row left most of the chip
// idle: 258 -> 38 us for 32 rows of 255 958 entries).  A warp takes whole top-k blocks, so that an entry's
// address needs no division and neighbouring lanes gather from neighbouring places.
template <typename TG, typename TV>
__global__ void __cluster_dims__(SP_CLUSTER, 1, 1) __launch_bounds__(SP_THREADS)
sparse_rows_dot_kernel(int64_t k, int64_t dbs, int kbs, int nfull, int k_few, const TG* __restrict__ g, const int16_t* __restrict__ I,
                       const void* __restrict__ V, float* __restrict__ out) {
    __shared__ float s_part[SP_THREADS / 32];
    __shared__ float s_cta[SP_CLUSTER];
    const int64_t r = blockIdx.x / SP_CLUSTER;
    const int nblocks = nfull + (k_few > 0 ? 1 : 0);
    float acc = 0.0f;
    for (int blk = (int)(blockIdx.x % SP_CLUSTER) * (SP_THREADS / 32) + warp_id(); blk < nblocks; blk += SP_CLUSTER * (SP_THREADS / 32))
        acc = dot_entries<TG, TV>(acc, g + (int64_t)blk * dbs, I, V, r * k + (int64_t)blk * kbs, 0, blk < nfull ? kbs : k_few);
    dot_sum<SP_CLUSTER>(acc, s_part, s_cta, out + r);
}

// The same where a row has fewer blocks than the cluster has warps: `parts` parts of `seg` entries of each block, a warp per
// part (32 rows of 10 002 entries in seven blocks: 11.2 us with a warp per block, 4.1 so), and for the shortest rows one CTA
// instead of a cluster, whose two meetings take longer than the work (370 entries: 4.3 us, 3.5 with parts, 2.2 so).
template <typename TG, typename TV, int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(SP_THREADS)
sparse_rows_dot_parts_kernel(int64_t k, int64_t dbs, int kbs, int nfull, int k_few, int parts, int seg, const TG* __restrict__ g,
                             const int16_t* __restrict__ I, const void* __restrict__ V, float* __restrict__ out) {
    __shared__ float s_part[SP_THREADS / 32];
    __shared__ float s_cta[CTAS];
    const int64_t r = blockIdx.x / CTAS;
    const int tasks = (nfull + (k_few > 0 ? 1 : 0)) * parts;
    float acc = 0.0f;
    for (int task = (int)(blockIdx.x % CTAS) * (SP_THREADS / 32) + warp_id(); task < tasks; task += CTAS * (SP_THREADS / 32)) {
        const int blk = task / parts, first = (task - blk * parts) * seg;
        acc = dot_entries<TG, TV>(acc, g + (int64_t)blk * dbs, I, V, r * k + (int64_t)blk * kbs, first, min(first + seg, blk < nfull ? kbs : k_few));
    }
    dot_sum<CTAS>(acc, s_part, s_cta, out + r);
}

// A thread's entry of a row: its position (negative: none) and its value.
template <typename TV> struct Entry;
template <> struct Entry<uint16_t> {
    uint32_t e;
    __device__ __forceinline__ void get(const int16_t* i, const uint16_t* v, bool on) { e = on ? (uint32_t)(uint16_t)*i | ((uint32_t)*v << 16) : 0xFFFFu; }
    __device__ __forceinline__ int pos() const { return (int16_t)(e & 0xFFFFu); }
    __device__ __forceinline__ float val() const { return __uint_as_float(e & 0xFFFF0000u); }
};
template <> struct Entry<float> {
    int p;
    float v;
    __device__ __forceinline__ void get(const int16_t* i, const float* x, bool on) { p = on ? (int)*i : -1; v = on ? *x : 0.0f; }
    __device__ __forceinline__ int pos() const { return p; }
    __device__ __forceinline__ float val() const { return v; }
};

// out[e] += sum_r M[r] * V[r, j] over the entries (r, j) that address e: one CTA per sub-range of a top-k block
// with a dense fp32 accumulator in shared memory; rows are added in row order (positions are unique inside a
// row, so a row needs no atomics, but a barrier).  Bound by the chain of rows: a thread fetches its entries of SPR_AHEAD rows at once,
// and, while the values are bf16, the next ones before it adds these, so that a row costs a shared-memory update and a barrier (25.6 M elements, 32
// rows of 1 %: 232 us with one load latency per row and four walks over a block's entries, 75 with one per eight rows, 65 with the next eight
// ahead; fp32 values have no registers for a second eight: 12 to 60 bytes of spills, bf16 out 73 against 54).
// The products of eight rows are made before the first of their barriers, off that chain (64 us; 1.28 M elements, bf16, 64 rows of 0.5 %: 14.4
// behind the barriers, 11.6 so; 60 M the same 217 / 202).  LONG, blocks with more entries than the CTA has threads: behind them, as the
// registers do not hold the products too (25.6 M, 32 rows of 5 %: 188, 206 before them).  Where a row has fewer entries a warp without one takes part in
// the barriers only, and groups behind the last row are not walked: with both in every warp one row of 1 % took,
// bf16 out, 28.2 us, 21.3 so.
template <typename TO, typename TV, bool LONG>
__global__ void __launch_bounds__(SPR_THREADS, 3)
sparse_rows_combine_kernel(int64_t d, int rows, int64_t k, int dbs, int kbs, int nfull, int k_few, const float* __restrict__ M,
                           const int16_t* __restrict__ I, const void* __restrict__ V, TO* __restrict__ out, int total_units) {
    extern __shared__ __align__(16) float acc[];
    __shared__ float s_M[MAB_MAX_WINDOW];
    const int t = threadIdx.x;
    const int subs_per_block = (dbs + SPR_SR - 1) / SPR_SR;
    const float factor = t < rows ? M[t] : 0.0f;
    for (int unit = blockIdx.x; unit < total_units; unit += gridDim.x) {
        int blk = unit / subs_per_block, sub = unit - blk * subs_per_block;
        if (blk > nfull) { sub += (blk - nfull) * subs_per_block; blk = nfull; }
        const int64_t blk_base = (int64_t)blk * dbs;
        const int n_blk = (int)min((int64_t)dbs, d - blk_base);
        const int kcnt = (blk < nfull) ? kbs : k_few;
        const int s0 = sub * SPR_SR;
        const int len = min(SPR_SR, n_blk - s0);
        const int64_t row0 = (int64_t)blk * kbs;
        for (int i = t; i < len; i += SPR_THREADS) acc[i] = 0.0f;
        // (row, round) pairs in row order, A of them fetched at once, and with bf16 values those after them before the current ones are added
        constexpr int A = SPR_AHEAD<TV, LONG>;
        const int rounds = LONG ? (kcnt + SPR_THREADS - 1) / SPR_THREADS : 1, pairs = rows * rounds;
        int fr = 0, fc = 0;                                      // the pair to fetch next ...
        const int16_t* fI = I + row0 + t;                        // ... from here
        const TV* fV = static_cast<const TV*>(V) + row0 + t;
        int r = 0, c = 0;                                        // ... and to add next
        auto fetch = [&](Entry<TV> (&e)[A]) {
#pragma unroll
            for (int i = 0; i < A; ++i) {
                const int j = LONG ? fc * SPR_THREADS : 0;
                e[i].get(fI + j, fV + j, fr < rows && j + t < kcnt);
                if (!LONG || ++fc == rounds) { fc = 0; ++fr; fI += k; fV += k; }
            }
        };
        auto add = [&](const Entry<TV> (&e)[A]) {
            int pos[A];
            float val[A];
            if constexpr (!LONG) {
#pragma unroll
                for (int i = 0; i < A; ++i) {
                    pos[i] = e[i].pos() - s0;
                    val[i] = __fmul_rn(s_M[min(r + i, rows - 1)], e[i].val());
                }
            }
#pragma unroll
            for (int i = 0; i < A; ++i) {
                if (r < rows) {                                  // uniform
                    if (c == 0) __syncthreads();                 // the row before (or the clearing) is done
                    if constexpr (LONG) { pos[i] = e[i].pos() - s0; val[i] = __fmul_rn(s_M[r], e[i].val()); }
                    if (pos[i] >= 0 && pos[i] < len) acc[pos[i]] = __fadd_rn(acc[pos[i]], val[i]);
                    if (!LONG || ++c == rounds) { c = 0; ++r; }
                }
            }
        };
        const bool mine = LONG || (t & ~31) < kcnt;              // a warp without entries only keeps step at the barriers
        Entry<TV> a[A];
        if (mine) fetch(a);
        if (unit == (int)blockIdx.x) {
            if (t < rows) s_M[t] = factor;
            if constexpr (!LONG) __syncthreads();                // the first products are made before the first row's barrier
        }
        if (!mine) {
            for (int i = 0; i < rows; ++i) __syncthreads();
        } else if constexpr (sizeof(TV) == 2) {
            Entry<TV> b[A];
            for (int p = 0; p < pairs; p += 2 * A) {
                if (p + A < pairs) fetch(b);
                add(a);
                if (p + 2 * A < pairs) fetch(a);
                if (p + A < pairs) add(b);
            }
        } else {
            for (int p = 0; p < pairs; p += A) {
                add(a);
                if (p + A < pairs) fetch(a);
            }
        }
        __syncthreads();
        TO* o = out + blk_base + s0;
        const int whole = ((reinterpret_cast<uintptr_t>(o) & 15) == 0) ? len / SPR_VEC<TO> : 0;
#pragma unroll 4
        for (int i = t; i < whole; i += SPR_THREADS) add_vector(o + i * SPR_VEC<TO>, acc + i * SPR_VEC<TO>);
        for (int i = whole * SPR_VEC<TO> + t; i < len; i += SPR_THREADS)
            Elem<TO>::store(o, i, __fadd_rn(Elem<TO>::load(o, i), acc[i]));
        __syncthreads();
    }
}

}  // namespace mab

using namespace mab;

static int check_geometry(const char* what, int64_t d, int64_t rows, int64_t k, int64_t dbs, int64_t kbs, int* nfull, int* k_few) {
    MAB_REQUIRE(d >= 0 && k >= 0 && rows >= 0 && dbs > 0 && kbs > 0, MAB_ERR_BAD_ARG, "%s: bad sizes", what);
    MAB_REQUIRE(rows <= MAB_MAX_WINDOW, MAB_ERR_LIMIT, "%s: %lld rows, at most %d", what, (long long)rows, MAB_MAX_WINDOW);
    MAB_REQUIRE(dbs <= 32768, MAB_ERR_LIMIT, "%s: d_block_size %lld exceeds 32768", what, (long long)dbs);
    const int64_t nf = d / dbs;
    const int64_t few = k - nf * kbs;
    MAB_REQUIRE(nf < ((int64_t)1 << 28) && few >= 0 && few <= d - nf * dbs, MAB_ERR_BAD_ARG,
                "%s: k=%lld inconsistent with d=%lld, d_block_size=%lld, k_block_size=%lld", what, (long long)k, (long long)d,
                (long long)dbs, (long long)kbs);
    *nfull = (int)nf; *k_few = (int)few;
    return MAB_OK;
}

extern "C" int mab_sparse_rows_dot(int64_t d, int64_t rows, int64_t k, int64_t d_block_size, int64_t k_block_size,
                                   const void* g, int g_dtype, const int16_t* I, const void* V, int v_dtype, float* out,
                                   void* stream) {
    int nfull, k_few;
    if (int rc = check_geometry("sparse_rows_dot", d, rows, k, d_block_size, k_block_size, &nfull, &k_few)) return rc;
    if (rows == 0) return MAB_OK;
    MAB_REQUIRE(g && I && V && out, MAB_ERR_BAD_ARG, "sparse_rows_dot: null pointer");
    MAB_REQUIRE((g_dtype == MAB_F32 || g_dtype == MAB_BF16) && (v_dtype == MAB_F32 || v_dtype == MAB_BF16), MAB_ERR_UNSUPPORTED,
                "sparse_rows_dot: dtypes %d, %d", g_dtype, v_dtype);
    cudaStream_t s = (cudaStream_t)stream;
    const int ctas = k <= SP_ONE_CTA ? 1 : SP_CLUSTER, grid = (int)rows * ctas, kbs = (int)k_block_size;
    const int blocks = std::max(1, nfull + (k_few > 0 ? 1 : 0)), longest = std::max(nfull > 0 ? kbs : 0, k_few);
    const int parts = std::max(1, std::min(ctas * (SP_THREADS / 32) / blocks, (longest + 31) / 32));
    const int seg = ((longest + parts - 1) / parts + 31) & ~31;
#define MAB_LAUNCH_DOT(TG, TV) do { \
        if (ctas > 1 && parts == 1) { \
            sparse_rows_dot_kernel<TG, TV><<<grid, SP_THREADS, 0, s>>>(k, d_block_size, kbs, nfull, k_few, (const TG*)g, I, V, out); \
        } else { \
            auto kern = ctas == 1 ? sparse_rows_dot_parts_kernel<TG, TV, 1> : sparse_rows_dot_parts_kernel<TG, TV, SP_CLUSTER>; \
            kern<<<grid, SP_THREADS, 0, s>>>(k, d_block_size, kbs, nfull, k_few, parts, seg, (const TG*)g, I, V, out); \
        } } while (0)
    if (g_dtype == MAB_F32 && v_dtype == MAB_BF16) MAB_LAUNCH_DOT(float, uint16_t);
    else if (g_dtype == MAB_F32) MAB_LAUNCH_DOT(float, float);
    else if (v_dtype == MAB_BF16) MAB_LAUNCH_DOT(uint16_t, uint16_t);
    else MAB_LAUNCH_DOT(uint16_t, float);
#undef MAB_LAUNCH_DOT
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? MAB_OK : cuda_fail(e, "sparse_rows_dot_kernel launch");
}

extern "C" int mab_sparse_rows_combine(int64_t d, int64_t rows, int64_t k, int64_t d_block_size, int64_t k_block_size,
                                       const float* M, const int16_t* I, const void* V, int v_dtype, void* out, int out_dtype,
                                       void* stream) {
    int nfull, k_few;
    if (int rc = check_geometry("sparse_rows_combine", d, rows, k, d_block_size, k_block_size, &nfull, &k_few)) return rc;
    if (rows == 0 || d == 0) return MAB_OK;
    MAB_REQUIRE(M && I && V && out, MAB_ERR_BAD_ARG, "sparse_rows_combine: null pointer");
    MAB_REQUIRE((out_dtype == MAB_F32 || out_dtype == MAB_BF16) && (v_dtype == MAB_F32 || v_dtype == MAB_BF16), MAB_ERR_UNSUPPORTED,
                "sparse_rows_combine: dtypes %d, %d", out_dtype, v_dtype);
    if (device_sm_count() < 0) return MAB_ERR_CUDA;
    const int dbs = (int)d_block_size;
    const int subs = (dbs + SPR_SR - 1) / SPR_SR;
    const int64_t tail = d - (int64_t)nfull * dbs;
    const int64_t units = (int64_t)nfull * subs + (tail > 0 ? (tail + SPR_SR - 1) / SPR_SR : 0);
    if (units == 0) return MAB_OK;
    const int grid = (int)std::min<int64_t>(units, (int64_t)device_sm_count() * 3);
    const int smem = SPR_SR * (int)sizeof(float);
    cudaStream_t s = (cudaStream_t)stream;
#define MAB_LAUNCH_COMBINE(TO, TV) do { \
        auto kern = std::max<int64_t>(nfull > 0 ? k_block_size : 0, k_few) > SPR_THREADS ? sparse_rows_combine_kernel<TO, TV, true> \
                                                                                       : sparse_rows_combine_kernel<TO, TV, false>; \
        MAB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); \
        kern<<<grid, SPR_THREADS, smem, s>>>(d, (int)rows, k, dbs, (int)k_block_size, nfull, k_few, M, I, V, (TO*)out, (int)units); } while (0)
    if (out_dtype == MAB_F32 && v_dtype == MAB_BF16) MAB_LAUNCH_COMBINE(float, uint16_t);
    else if (out_dtype == MAB_F32) MAB_LAUNCH_COMBINE(float, float);
    else if (v_dtype == MAB_BF16) MAB_LAUNCH_COMBINE(uint16_t, uint16_t);
    else MAB_LAUNCH_COMBINE(uint16_t, float);
#undef MAB_LAUNCH_COMBINE
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? MAB_OK : cuda_fail(e, "sparse_rows_combine_kernel launch");
}
