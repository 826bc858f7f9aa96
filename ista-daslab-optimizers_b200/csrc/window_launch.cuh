// How the update kernel's tile form is launched: threads, CTAs and shared memory by the window, the tiles and the GPU.  Host side only, so that
// the choice can be checked without a GPU.
#pragma once
#include "window.cuh"
#include "fused.cuh"

namespace mab {

constexpr int WT_WORDS = 1024;            // bitmap words of a tile (32768 positions)
constexpr int WT_MAX_ENTRIES = 16384;     // window entries of one block the compact arrays may hold

// Bytes one row's slice of I (or V) occupies in the raw staging area: the slice is copied from the
// 16-byte boundary below its first element, in whole 16-byte pieces.
__host__ __device__ constexpr int wt_row_stride(int max_k) { return ((max_k * 2 + 30) + 15) & ~15; }

__host__ __device__ constexpr int wt_smem_bytes(int rows, int max_k) {
    const int e = (rows * max_k + 3) & ~3;
    return 8 * e + rows * 2 * wt_row_stride(max_k) + 4 * WT_WORDS + 2 * WT_WORDS + 2 * e;
}

// Threads of a CTA of the tile kernel; `fit`: how many CTAs' arrays fit an SM (`fit_384`: with 384 threads, the alpha forms' dense arrays grow with them).  us of this kernel, fp32, 10 rows; the row loop has its
// prefetching form while a row's entries do not outnumber the threads, and every tile in flight costs L2.
//   k = 0.5 % (146 entries), 116 M elements: 256 threads 105, 384 108, 512 120.
//   k = 1 % (291): 256 / 384 / 512 threads, 100 tiles 12.4 / 9.5 / 8.6, 300 tiles 18.8 / 15.5 / 18.6, 1000 55 / 42 / 44, 1500 77 / 61 / 61, 3000 143 / 124 /
//   118, 4282 201 / 186 / 166; with weight decay 1000 82 / 70 / 73, 4282 292 / 322 / 268; 120 ragged tensors 33 / 30 / 35.
//   The operator that writes every position's update: 384 (60 M elements k = 1 % 75, 256 and 512 threads 79; 0.5 % 59, 256 73, 512 67); with late zeros
//   256 for many short rows (232 M elements, 0.5 %, 10 and 20 rows 202 and 270, 384 threads 219 and 298; 1 and 3 rows 161 and 173, 155 and 164).
//   The alpha forms have 80 registers a thread: 256 threads while three CTAs fit (33.5 M elements 121, 384 threads 127), 384 where two do (bf16, 20
//   rows, 58 M elements 265 with 256, 209; one CTA of 384 alone 415, two of 256 373), and 512 where one does or an SM has no more than one tile (100 tiles 29 and 18).
static inline int threads_of(int write, bool alpha, int fit, int fit_384, int tiles, int rows, int max_k, int sms) {
    if (alpha) return fit < 2 || tiles <= sms ? 512 : fit < 3 && fit_384 >= 2 ? 384 : 256;
    if (fit < 2) return 1024;
    if (tiles <= 2 * sms || fit < 3) return 512;
    if (write == 1) return 384;
    if (write == 2) return max_k <= 256 && fit >= 4 && rows >= 8 ? 256 : 384;
    if (max_k <= 256 && fit >= 4) return 256;
    return max_k <= 384 && tiles <= 10 * sms ? 384 : 512;
}

// When the operator that writes every position's update stores the zeros: 1 before the window phases, 2 behind them.  (0: a step.)  Where the output does
// not fit the 126 MB of L2, zeros stored before are written to memory and brought back for their updates.  us, before / behind, fp32, 10 rows of 1 %:
// 25.6 M elements 35.3 / 35.4, 34.9 M 47.6 / 46.2, 58 M 78 / 72, 116 M 168 / 140, 232 M 342 / 274 (288 with a look-up for every element); bf16, half
// as long, 58 M 56 / 57, 232 M 215 / 220.
static inline int write_mode(int64_t bytes, bool bf16) { return !bf16 && bytes > ((int64_t)1 << 27) ? 2 : 1; }

// The EARLY form (see wait_for_kernel_before): every CTA has one tile, and kernel A no more CTAs than there are SMs.  Not a matter of the tiles alone: a
// CTA that an SM has to itself gets two tiles as soon as there are more tiles than the device shows SMs, a part of a GPU for instance.
static inline bool early_form(int tiles, int grid, int sms) { return tiles <= grid && tiles <= sms; }

// The AHEAD form of the alpha forms on bf16 parameters; fp32 spills.  It pays where a CTA has tiles enough or a row more entries than 256 threads.  us a
// step, ahead and not (alpha == -2, 444 CTAs): k = 0.5 % 444 tiles 55.5 / 54.3, 740 108.4 / 106.4, 1000 141.5 / 143.9, 2000 219.9 / 221.7; k = 1 %
// 200 tiles 43.1 / 45.0, 445 85.9 / 87.4, 2000 238.5 / 246.4; 20 rows (296 CTAs) 445 90.4 / 90.2, 600 115.8 / 118.3; k = 5 % (148) 600 181.7 / 185.4.
// alpha = 0.5, k = 0.5 %: 1000 143.1 / 143.9, 1500 183.9 / 183.1, 2000 228.4 / 226.2.
// Two entries a thread: rows of up to 512, and four of them at least (alpha == -2, 300 tiles of 1 %, 1, 2 and 3 rows 43.1 / 42.7, 44.9 / 43.9 and 44.3 / 43.8,
// 5 rows 45.7 / 45.8; alpha = 0.5, 2000 tiles, 1 row 212.7 / 210.4, 5 rows 225.9 / 227.6).
static inline bool rows_ahead(bool bf16, int alpha, int threads, int grid, int tiles, int rows, int max_k) {
    if (!bf16 || alpha == 0) return false;
    if (threads != 256) return tiles > grid;
    return (max_k > 256 && max_k <= 512 && rows >= 4) || (alpha == 2 && tiles > 2 * grid);
}

// CTAs of `dynamic` bytes of shared memory an SM holds, next to the kernel's static arrays (the tensors' first units, the scan's scratch, the rows'
// offsets) and the 1024 bytes that every CTA costs.  One CTA too many is a second wave of them, and threads chosen for what does not fit (us a step,
// 58 M elements, 10 rows, reckoned too small by 1280 bytes and right: alpha = 0.5, bf16, 419 entries a row 356 and 271, 670 411 and 345; fp32, alpha 0,
// 757 entries 342 and 298).
constexpr int WT_STATIC_BYTES = (4 * (WIN_MAX_TENSORS + 1 + 36 + 2 * MAB_MAX_WINDOW) + 127) & ~127;
static inline int ctas_of_sm(int dynamic, int optin_smem) { return (optin_smem + 1024) / (dynamic + WT_STATIC_BYTES + 1024); }

struct TileLaunch {
    int  threads, grid, smem;             // smem 0: the window is too large for the compact arrays, the wide form takes it
    int  dense_at;                        // the alpha forms' dense arrays of the warps in shared memory (0: they do not fit)
    bool early, ahead;
};

static inline TileLaunch plan_tile_launch(int write, int alpha, bool bf16, int rows, int max_k, int tiles, bool behind_a, int sms, int optin_smem) {
    TileLaunch L = {0, 0, 0, 0, false, false};
    // while the compact arrays fit one CTA's shared memory (next to the kernel's static arrays)
    const int smem_tile = (int64_t)rows * max_k <= WT_MAX_ENTRIES ? wt_smem_bytes(rows, max_k) : 0;
    if (smem_tile == 0 || smem_tile + 4096 > optin_smem) return L;
    // the forms with the alpha term: a dense array of 256 floats per warp behind the window's arrays, if it fits
    const int fit = std::max(1, std::min(8, ctas_of_sm(smem_tile + (alpha ? 8 * 1024 : 0), optin_smem)));
    L.threads = threads_of(write, alpha != 0, fit, ctas_of_sm(smem_tile + 12 * 1024, optin_smem), tiles, rows, max_k, sms);
    if (alpha && ((smem_tile + 15) & ~15) + L.threads * 32 + 4096 > optin_smem) L.threads = 256;
    const int nt = L.threads, dense = alpha ? nt * 32 : 0;
    L.dense_at = alpha && ((smem_tile + 15) & ~15) + dense + 4096 <= optin_smem ? (smem_tile + 15) & ~15 : 0;
    L.smem = L.dense_at > 0 ? L.dense_at + dense : smem_tile;
    const int per_sm = std::max(1, std::min(alpha ? 768 / nt : nt == 384 ? 3 : 1024 / nt, ctas_of_sm(L.smem, optin_smem)));   // (as in __launch_bounds__)
    L.grid = (int)std::min<int64_t>(tiles, (int64_t)sms * per_sm);
    L.early = behind_a && nt == 512 && early_form(tiles, L.grid, sms);
    L.ahead = !L.early && rows_ahead(bf16, alpha, nt, L.grid, tiles, rows, max_k);
    return L;
}

// Shared memory of one CTA of the resident-tile kernel, or 0 when two such CTAs do not fit an SM.
static inline int resident_smem_bytes(int rows, int max_k, int max_dbs, int optin_smem, int* tile_bytes) {
    *tile_bytes = (max_dbs * 2 + 127) & ~127;
    if ((int64_t)rows * max_k > WT_MAX_ENTRIES) return 0;
    const int smem = *tile_bytes + wt_smem_bytes(rows, max_k);
    const int static_and_reserved = 6 * 1024;                 // the kernel's static arrays + the per-CTA reservation
    return 2 * (smem + static_and_reserved) <= optin_smem + 1024 ? smem : 0;
}

// Whether the update of a step on such tensors takes the EARLY form.
static inline bool update_is_early(int tiles, int rows, int max_k, int max_dbs, bool bf16, int alpha, int sms, int optin_smem) {
    int tile_bytes;
    if (bf16 && alpha == 0 && resident_smem_bytes(rows, max_k, max_dbs, optin_smem, &tile_bytes) > 0) return early_form(tiles, std::min(tiles, 2 * sms), sms);
    return plan_tile_launch(0, alpha, bf16, rows, max_k, tiles, true, sms, optin_smem).early;
}

}  // namespace mab
