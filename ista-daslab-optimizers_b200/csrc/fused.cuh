// Declarations shared by the two fused kernels and the host-side step driver.
#pragma once
#include "common.cuh"
#include "window.cuh"

namespace mab {

__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Elements between consecutive rows of a tensor's I and V.
__host__ __device__ __forceinline__ int64_t row_pitch_of(const mab_tensor& t) { return t.row_pitch > 0 ? (int64_t)t.row_pitch : t.k; }

// Index of the tensor whose unit range contains `unit`: largest i with first[i] <= unit.
// first[0..n] is ascending with first[n] = total units; tensors without units repeat a value.
__device__ __forceinline__ int find_tensor(const int* first, int n, int unit) {
    int lo = 0, hi = n;                      // invariant: first[lo] <= unit < first[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= unit) lo = mid; else hi = mid;
    }
    return lo;
}

// The consecutive tiles [first, end) of CTA b.  The CTAs with one more than the others come first: those that share an SM are
// numbered an SM count apart (the grid is filled one CTA per SM at a time), so no SM gets two tiles more than another one.
// (Spread evenly over the numbers, some SMs had two of the longer ranges: bf16 kernel A on 600 tiles of loose blocks 47 us, now 35; on
// 3300 tiles with blocks of 64 132 and 121.)
struct TileRange { int first, end; };
__host__ __device__ __forceinline__ TileRange tiles_of_cta(int total, int ctas, int b) {
    const int each = total / ctas, more = total % ctas, first = b * each + (b < more ? b : more);
    return {first, first + each + (b < more ? 1 : 0)};
}

// The update kernel of a step is launched behind kernel A without the gap between two kernels (programmatic stream
// serialization): its CTAs read the descriptor table, which neither kernel writes, and wait there for kernel A's end and its
// results.  A kernel A allows it as soon as all its CTAs have started, if it has no more CTAs than there are SMs and the update is of the form below, or
// no more than half as many; with more the ones that wait take places unevenly among those that work, and the update runs on fewer SMs than it
// could (us a step, allowed and not: fp32, 254 tiles 72.8 and 55.5; the wide form of the update behind 100 tiles, 20 rows of 5 %, bf16 73.3 and
// 63.6, fp32 65.5 and 55.4).  Kernel A of loose blocks does not allow it, the requantisation being next; nor do the requantisation and the fp32
// kernel with one tile per SM (not tried there).
// What does not depend on kernel A comes before that wait where every CTA of the update has one tile (template flag EARLY): the other rows of
// the window are staged and marked, the weight decay is applied, or the bf16 parameters are on their way into shared memory; the row
// that kernel A writes follows behind the wait.  Kernel A itself is an ordinary launch, so everything before it is complete.  us a step, everything
// behind the wait and so: 7 690 fp32 elements 20.5 / 18.5, 40 tiles fp32 24.6 / 22.6, with weight decay 28 / 22.6, bf16 22.6 / 20.9; not allowed
// and so: 80 tiles bf16 22.6 / 21.9, 100 fp32 with weight decay 28.7 / 26.7, 110 with 20 rows 28.7 / 27.1, 148 fp32 26.5 / 25.5, bf16 22.7 / 22.6.
__device__ __forceinline__ void allow_next_kernel(int most_ctas) { if ((int)gridDim.x <= most_ctas) asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_kernel_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
static inline cudaError_t launch_behind_kernel(void (*kern)(P...), int grid, int threads, int smem, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid); c.blockDim = dim3(threads); c.dynamicSmemBytes = smem; c.stream = s;
    c.attrs = &early; c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kern, P(args)...);
}

// window_adam.cu
int fill_window_args(WindowArgs& a, int64_t steps, int m, double beta1, double beta2, double eps, float alpha, int qbs);
int launch_window_step(const mab_tensor* dev_tensors, int n_tensors, int units_tile, int units_wide, int max_k, int max_dbs,
                       int param_dtype, const WindowArgs& a, bool behind_a, cudaStream_t s);
int allowing_ctas(int units_tile, int rows, int max_k, int max_dbs, int param_dtype, float alpha);   // most CTAs of a kernel A that allows such an update
int units_b_of(const mab_tensor& t);
int launch_wait_selftest(int probe_limit, cudaStream_t s);

// probe.cu: adds sum g^2 (which & PROBE_G) and sum Qinv(e)^2 (which & PROBE_E) of the tensors to
// out[MAB_PROBE_NORM_G] / out[MAB_PROBE_NORM_E]
enum { PROBE_G = 1, PROBE_E = 2 };
int launch_probe(const mab_tensor* dev_tensors, int n_tensors, int total_units, int qbs, double* out, cudaStream_t s,
                 int which = PROBE_G | PROBE_E);

// Quantisation blocks of any size (a multiple of 8 elements), which ignore the borders of the top-k blocks
// (micro_adam.py:217-231): kernel A then leaves the residual in the gradient buffer and merges each block's
// extremes into two scratch arrays; requant_loose.cu turns them into statistics and codes.
struct LooseArgs {
    int qbs;                       // quant_block_size
    uint32_t* st_min;              // order-preserving key of the minimum per quantisation block (initialised to 0xFFFFFFFF)
    uint32_t* st_max;              // ... of the maximum (initialised to 0)
    const int64_t* qb_first;       // first scratch entry of every tensor of the call
};

constexpr int LOOSE_MAX_QB = 32768 / 64 + 2;        // quantisation blocks (>= 64 elements) a tile of at most 32768 elements can touch

// Monotone map float -> uint32 (negative values below positive ones, -0 below +0) and back.
__device__ __forceinline__ uint32_t ord_key(float f) {
    const uint32_t b = __float_as_uint(f);
    return b ^ ((uint32_t)((int32_t)b >> 31) | 0x80000000u);
}
__device__ __forceinline__ float ord_value(uint32_t k) {
    return __uint_as_float(k ^ ((k & 0x80000000u) ? 0x80000000u : 0xFFFFFFFFu));
}

// Quantisation block (relative to the tile's first) of the octet that starts `r` elements after that block's start;
// `big`: the block is at least as long as the longest tile, so the answer is 0 or 1.
__host__ __device__ __forceinline__ int loose_block(int r, int qbs, bool big) {
    return big ? (r >= qbs ? 1 : 0) : (int)((unsigned)r / (unsigned)qbs);
}

// Quantisation blocks that a tile of n elements touches which starts lrem0 elements into one (lrem0 < qbs <= 2^30: the sum of
// both and another qbs would not fit 32 bits).
__host__ __device__ __forceinline__ int loose_blocks_touched(int lrem0, int n, int qbs) {
    return loose_block(lrem0 + n - 1, qbs, false) + 1;
}

// ef_topk_quant.cu; allowing: see allow_next_kernel
int launch_ef_topk_quant(const mab_tensor* dev_tensors, int n_tensors, int total_units, int grad_dtype,
                         int qbs, int max_dbs, int max_k, int allowing, cudaStream_t s, const LooseArgs* loose = nullptr);
int units_a_of(const mab_tensor& t);

// requant_loose.cu: statistics (bf16) and codes of the residual kernel A left in the gradient buffers
int launch_requant_loose(const mab_tensor* dev_tensors, int n_tensors, int total_units, int grad_dtype,
                         const LooseArgs& la, cudaStream_t s);

// ef_topk_quant_bf16.cu (blocks of 64) and ef_topk_quant_bf16_warps.cu (all others, and large launches): return 1 (without
// launching) when two CTAs of their shared memory do not fit an SM
int launch_ef_topk_quant_bf16(const mab_tensor* dev_tensors, int n_tensors, int total_units, int max_dbs, int allowing, cudaStream_t s);
int launch_ef_topk_quant_bf16_warps(const mab_tensor* dev_tensors, int n_tensors, int total_units, int qbs, int max_dbs, int allowing, cudaStream_t s,
                                    const LooseArgs* loose);

// ef_topk_quant_f32.cu: returns 1 (without launching) where the tile or its candidates do not fit
int launch_ef_topk_quant_f32(const mab_tensor* dev_tensors, int n_tensors, int total_units, int qbs, int max_dbs, int max_k, int allowing, cudaStream_t s);

// Each kernel file keeps its own "a bounded wait gave up" flag (no relocatable device code): these read
// it into *out and optionally clear it.
int copy_timeout_f32(int* out, bool clear);      // ef_topk_quant.cu
int copy_timeout_f32_split(int* out, bool clear);   // ef_topk_quant_f32.cu
int copy_timeout_bf16(int* out, bool clear);     // ef_topk_quant_bf16.cu
int copy_timeout_bf16_warps(int* out, bool clear);  // ef_topk_quant_bf16_warps.cu
int copy_timeout_window(int* out, bool clear);   // window_adam.cu

}  // namespace mab
