// CSR rows summed a warp at a time: the common core of the SpMV, the
// Jacobi smoother and the AMG transfer operators.
//
// (warp_row_sum) One warp owns 32 consecutive rows.  Their entries are contiguous, so the
// lanes read them 32 at a time -- fully coalesced, CSR_ROWS_CHUNK / 32
// independent loads per lane in flight -- and stage the products in shared
// memory; each lane then adds its own row's products in entry order, the
// order of a sequential CSR product.  (Striding each row's ~15 entries over
// a few lanes instead leaves each lane a short chain of dependent index ->
// value loads and sectors shared between neighbouring rows.)
#pragma once

#include "internal.cuh"

namespace up3d {

constexpr int CSR_ROWS_CHUNK = 256;   // entries staged per pass of a warp
constexpr int CSR_ROWS_BLOCK = 256;   // threads per block of the lanes form
constexpr int CSR_WARP_BLOCK = 64;    // threads per block of the warp-rows form (2 warps)

// Loads of the matrix entries, each read once per product: past L1, which
// keeps the vector's values (625 k-row P1 matrix, FP64: 36 -> 31 us; 2.5 M
// rows 131 -> 99 us).
__device__ __forceinline__ double ld_stream(const double* p) {
    double v;
    asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int32_t ld_stream(const int32_t* p) {
    int32_t v;
    asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Sum over row r0 + lane of term(column, value), over the row's entries, for
// the calling warp's rows [r0, min(r0 + 32, n)); 0 for lanes past n.  `sh`
// holds CSR_ROWS_CHUNK values private to the warp.  Every lane must call.
// All entry loads of a chunk are issued before the first gather.
template <class T, class Term>
__device__ __forceinline__ T warp_row_sum(const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                                          const T* __restrict__ Ax, int64_t r0, int64_t n, T* sh, Term term) {
    const int lane = threadIdx.x & 31;
    const int64_t r = r0 + lane;
    const int64_t rend = r0 + 32 < n ? r0 + 32 : n;
    const int32_t s = Ap[r0], e = Ap[rend];
    int32_t ms = 0, me = 0;
    if (r < n) {
        ms = Ap[r];
        me = Ap[r + 1];
    }
    T acc = T(0);
    for (int32_t c0 = s; c0 < e; c0 += CSR_ROWS_CHUNK) {
        int32_t c[CSR_ROWS_CHUNK / 32];
        T v[CSR_ROWS_CHUNK / 32];
#pragma unroll
        for (int j = 0; j < CSR_ROWS_CHUNK / 32; ++j) {
            const int32_t k = c0 + j * 32 + lane;
            c[j] = k < e ? ld_stream(Ai + k) : -1;
            v[j] = k < e ? ld_stream(Ax + k) : T(0);
        }
#pragma unroll
        for (int j = 0; j < CSR_ROWS_CHUNK / 32; ++j) v[j] = c[j] >= 0 ? term(c[j], v[j]) : T(0);
#pragma unroll
        for (int j = 0; j < CSR_ROWS_CHUNK / 32; ++j) sh[j * 32 + lane] = v[j];
        __syncwarp();
        const int32_t a = ms > c0 ? ms : c0;
        const int32_t b = me < c0 + CSR_ROWS_CHUNK ? me : c0 + CSR_ROWS_CHUNK;
        for (int32_t k = a; k < b; ++k) acc += sh[k - c0];
        __syncwarp();
    }
    return acc;
}

// Sum over row r of term(column, value) by TPR lanes striding the row's
// entries, reduced by a fixed shuffle tree; every lane of the warp must call
// (rows past n contribute 0).  For short matrices (few rows: the warp-rows
// form would leave most SMs idle) and long rows (AMG coarse levels,
// restriction).
template <class T, int TPR, class Term>
__device__ __forceinline__ T lanes_row_sum(const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                                           const T* __restrict__ Ax, int64_t r, int64_t n, Term term) {
    const int sub = threadIdx.x % TPR;
    T acc = T(0);
    if (r < n)
        for (int32_t k = Ap[r] + sub; k < Ap[r + 1]; k += TPR)   // few lanes share sectors between steps: those stay in L1
            acc += TPR >= 16 ? term(ld_stream(Ai + k), ld_stream(Ax + k)) : term(Ai[k], Ax[k]);
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, TPR);
    return acc;
}

// The warp-rows form pays once a matrix has rows enough to give every SM
// a few warps of 32 rows and its rows are short (measured on B200: the
// 625 k-row P1 Jacobian 0.045 -> 0.034 ms; a 24 k-row AMG level with 26
// entries per row 2x slower than 16 lanes per row).
constexpr int64_t CSR_ROWS_MIN_ROWS = 148 * 16 * 32;
inline bool use_warp_rows(int64_t n, int64_t nnz) { return n >= CSR_ROWS_MIN_ROWS && nnz <= 24 * n; }

// Lanes per row from the mean row length (thresholds tuned on B200).
inline int lanes_per_row(int64_t nnz, int64_t n) {
    const double avg = n > 0 ? (double)nnz / (double)n : 0.0;
    return avg <= 16 ? 4 : avg <= 24 ? 8 : avg <= 96 ? 16 : 32;
}
inline unsigned lanes_grid(int64_t n, int tpr) { return grid_for(n, 256 / tpr, (int64_t)148 * 64); }

// Blocks of `block` threads for n rows at 32 rows per warp.
inline unsigned csr_rows_grid(int64_t n, int block) { return grid_for(n, block, (int64_t)148 * 1024); }

// ------------------------------------------------------------ sliced rows
// The same rows in slices of 32: entry k of row 32 q + lane at Sp[q] + 32 k +
// lane, padded to the slice's longest row with column -1.  A lane owns a
// row, so the entry loads are coalesced without staging, and neighbouring
// rows of a mesh numbering read neighbouring vector entries (the entry-order
// loads above touch ~14 sectors per request).  625 k-row P1 matrix: FP64
// 36 -> 22 us, FP32 17 -> 12 us with the matrix in L2 and 37 -> 23 us without;
// 2.5 M rows FP64 131 -> 70 us (7.1 TB/s).
constexpr int SELL_BLOCK = 64, SELL_BATCH = 16;   // threads per block; entries in flight per lane
// worth it where warp_row_sum is (rows enough for several slices per SM)
// and the padding stays below an eighth
inline bool use_sell(int64_t n, int64_t nnz, int64_t padded) {
    return n >= CSR_ROWS_MIN_ROWS && padded <= nnz + nnz / 8;
}
inline unsigned sell_grid(int64_t n) { return (unsigned)((n + SELL_BLOCK - 1) / SELL_BLOCK); }

// Sum of the slice's row `lane`, entries in row order.  `ready` is called
// once the first batch of entries has been asked for and before the vector
// is read.
template <class T, class Ready>
__device__ __forceinline__ T sell_row_sum(const int32_t* __restrict__ Sp, const int32_t* __restrict__ Si,
                                          const T* __restrict__ Sx, const T* x, int64_t q, int lane, Ready ready) {
    const int32_t s = Sp[q], w = (Sp[q + 1] - s) >> 5;
    const int32_t* si = Si + s + lane;
    const T* sx = Sx + s + lane;
    T acc = T(0);
    for (int32_t k0 = 0; k0 < w || k0 == 0; k0 += SELL_BATCH) {   // warp-uniform
        int32_t c[SELL_BATCH];
        T v[SELL_BATCH];
#pragma unroll
        for (int j = 0; j < SELL_BATCH; ++j) {
            c[j] = k0 + j < w ? ld_stream(si + (k0 + j) * 32) : -1;
            v[j] = k0 + j < w ? ld_stream(sx + (k0 + j) * 32) : T(0);
        }
        if (k0 == 0) ready();
#pragma unroll
        for (int j = 0; j < SELL_BATCH; ++j)
            if (c[j] >= 0) acc = fma(v[j], x[c[j]], acc);
    }
    return acc;
}

}  // namespace up3d
