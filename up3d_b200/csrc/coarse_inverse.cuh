// Dense inverse of the AMG's coarsest operator by one thread-block cluster.
#pragma once

#include <cooperative_groups.h>

#include "internal.cuh"

namespace up3d {

// In-place Gauss-Jordan with partial pivoting of the n x n matrix (CSR Cp,
// Ci, Cx), n <= GJ_MAX, by one cluster; inv receives the inverse, *singular
// 1 when a column has no non-zero pivot (inv is then not written).
//
// The matrix lives in the cluster's shared memory: CTA q holds columns
// [q nb, (q + 1) nb) of every row, nb a multiple of the panel width.  The
// CTA that holds the next GJ_PANEL columns eliminates them among themselves
// with one row per thread in registers (pivot of each: the first unused row
// of largest magnitude) and writes the factors to global memory (`fac`, two
// buffers of n x GJ_PANEL, then the pivot rows and reciprocals); after one
// cluster barrier every CTA applies the panel's steps to its own columns,
// in order, with the matrix entry in a register.  Rows stay where they are
// (the pivot order is undone when the inverse is written).
//
// What bounds it is the chain of n pivots, not arithmetic.  One column per
// barrier instead of a panel (the factors pushed through distributed shared
// memory) took 2.9 us per column at n 208 and 8.6 us at n 500, this form 1.2
// and 2.2 us; two launches per column, the form for larger n, 7.8 us.
constexpr int GJ_THREADS = 512, GJ_MAX = GJ_THREADS, GJ_PANEL = 8;
constexpr size_t gj_fac_size(int64_t n) { return 2 * (size_t)GJ_PANEL * (n + 2); }   // doubles of `fac`

struct GjSmem {
    int ld;                    // row stride of the CTA's columns (odd: column walks without bank conflicts)
    size_t f, r, meta, red, perm, step, used, total;
    __host__ __device__ GjSmem(int n, int nb) {
        ld = nb + 1;
        size_t o = (sizeof(double) * (size_t)n * ld + 15) & ~size_t(15);
        f = o;     o += sizeof(double) * GJ_PANEL * (size_t)n;           // the panel's factors, by row
        r = o;     o += sizeof(double) * GJ_PANEL * (size_t)(nb + 1);    // the panel's pivot rows, scaled
        meta = o;  o += sizeof(double) * 2 * GJ_PANEL;                   // pivot rows, reciprocals
        red = o;   o += (sizeof(double) + sizeof(int)) * (GJ_THREADS / 32);
        perm = o;  o += sizeof(int) * (size_t)n;
        step = o;  o += (size_t)n;                                       // panel step a row is the pivot of, or 255
        total = (o + 15) & ~size_t(15);
    }
};

// The lowest index of the largest v >= 0 of a warp (v < 0: no candidate);
// every lane gets (v, i), i = `none` when there is no candidate.
// Non-negative doubles order like their bits, so this is three warp
// reductions of 32-bit words instead of a tree of 64-bit shuffles.
__device__ __forceinline__ void gj_argmax(double& v, int& i, int none) {
    const bool cand = v >= 0.0;
    const unsigned hi = cand ? (unsigned)__double2hiint(v) : 0u;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = cand && hi == mh ? (unsigned)__double2loint(v) : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
    const unsigned mi = __reduce_min_sync(0xffffffffu, cand && hi == mh && lo == ml ? (unsigned)i : 0xffffffffu);
    i = mi == 0xffffffffu ? none : (int)mi;
    v = mi == 0xffffffffu ? -1.0 : __hiloint2double((int)mh, (int)ml);
}

__global__ void __launch_bounds__(GJ_THREADS)
    k_gj_cluster(int n, int nb, const int32_t* __restrict__ Cp, const int32_t* __restrict__ Ci,
                 const double* __restrict__ Cx, double* __restrict__ inv, double* fac, int* __restrict__ singular) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char gj_sm[];
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const GjSmem L(n, nb);
    const int ld = L.ld;
    double* A = reinterpret_cast<double*>(gj_sm);
    double* F = reinterpret_cast<double*>(gj_sm + L.f);
    double* R = reinterpret_cast<double*>(gj_sm + L.r);
    double* meta = reinterpret_cast<double*>(gj_sm + L.meta);
    double* rv = reinterpret_cast<double*>(gj_sm + L.red);
    int* ri = reinterpret_cast<int*>(rv + GJ_THREADS / 32);
    int* perm = reinterpret_cast<int*>(gj_sm + L.perm);
    uint8_t* step = gj_sm + L.step;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int col0 = rank * nb, ncol = max(0, min(nb, n - col0));
    // lanes of a warp: kl columns x (32 / kl) rows
    int kl = 1;
    while (kl < 32 && kl < ncol) kl <<= 1;
    const int kk = lane & (kl - 1), rows_per_pass = (GJ_THREADS / 32) * (32 / kl);
    const int row0 = w * (32 / kl) + lane / kl;
    bool used = tid >= n;      // this thread's row has been a pivot

    for (int i = tid; i < n * ld; i += GJ_THREADS) A[i] = 0.0;
    for (int i = tid; i < n; i += GJ_THREADS) step[i] = 255;
    __syncthreads();
    for (int r = w; r < n; r += GJ_THREADS / 32)
        for (int32_t k = Cp[r] + lane; k < Cp[r + 1]; k += 32) {
            const int c = Ci[k] - col0;
            if (c >= 0 && c < ncol) A[r * ld + c] = Cx[k];
        }
    __syncthreads();

    for (int c0 = 0; c0 < n; c0 += GJ_PANEL) {
        const int width = min(GJ_PANEL, n - c0);
        double* out = fac + ((c0 / GJ_PANEL) & 1) * (size_t)GJ_PANEL * (n + 2);
        if (c0 >= col0 && c0 < col0 + ncol) {
            // ---- the panel, one row per thread
            double a[GJ_PANEL], f[GJ_PANEL];
#pragma unroll
            for (int j = 0; j < GJ_PANEL; ++j) {
                a[j] = tid < n && j < width ? A[tid * ld + c0 - col0 + j] : 0.0;
                f[j] = 0.0;
            }
#pragma unroll
            for (int s = 0; s < GJ_PANEL; ++s) {
                if (s >= width) break;   // the same for every thread
                // every thread's row as if it were the pivot's, under the search
                const double d = a[s] != 0.0 ? __ddiv_rn(1.0, a[s]) : 0.0;
                double best = used ? -1.0 : fabs(a[s]);   // NaN is never a pivot
                int p = tid;
                gj_argmax(best, p, n);
                if (lane == 0) {
                    rv[w] = best;
                    ri[w] = p;
                }
                __syncthreads();
                best = lane < GJ_THREADS / 32 ? rv[lane] : -1.0;
                p = lane < GJ_THREADS / 32 ? ri[lane] : n;
                gj_argmax(best, p, n);
                if (tid == p) {
#pragma unroll
                    for (int j = 0; j < GJ_PANEL; ++j) {
                        a[j] = j == s ? d : a[j] * d;
                        R[j] = a[j];
                    }
                    used = true;
                    meta[s] = d;
                }
                if (tid == 0) meta[GJ_PANEL + s] = best > 0.0 ? (double)p : -1.0;
                __syncthreads();
                if (tid != p && tid < n) {
                    f[s] = a[s];
                    if (f[s] != 0.0)
#pragma unroll
                        for (int j = 0; j < GJ_PANEL; ++j) a[j] = fma(-f[s], R[j], j == s ? 0.0 : a[j]);
                }
            }
            if (tid < n) {
#pragma unroll
                for (int j = 0; j < GJ_PANEL; ++j) {
                    if (j < width) A[tid * ld + c0 - col0 + j] = a[j];
                    out[(size_t)GJ_PANEL * tid + j] = f[j];
                }
            }
            if (tid < 2 * GJ_PANEL) {
                const int s = tid & (GJ_PANEL - 1);
                out[(size_t)GJ_PANEL * n + tid] = s < width ? meta[tid] : -1.0;
            }
        }
        cluster.sync();   // the factors are in; every CTA has applied the panel before
        for (int i = tid; i < GJ_PANEL * n; i += GJ_THREADS) F[i] = __ldcg(out + i);
        if (tid < 2 * GJ_PANEL) meta[tid] = __ldcg(out + (size_t)GJ_PANEL * n + tid);
        __syncthreads();
        bool bad = false;
        for (int s = 0; s < width; ++s) {
            bad |= meta[GJ_PANEL + s] < 0.0;
            used |= meta[GJ_PANEL + s] == (double)tid;
        }
        if (bad) {        // the same on every CTA
            if (rank == 0 && tid == 0) *singular = 1;
            return;
        }
        if (tid < width) {
            const int p = (int)meta[GJ_PANEL + tid];
            perm[c0 + tid] = p;
            step[p] = (uint8_t)tid;
        }
        // ---- the pivot rows of the CTA's other columns, in step order
        for (int k = tid; k < ncol; k += GJ_THREADS) {
            if (col0 + k >= c0 && col0 + k < c0 + width) continue;
            double rk[GJ_PANEL];
#pragma unroll
            for (int s = 0; s < GJ_PANEL; ++s) {
                if (s >= width) break;
                const int p = (int)meta[GJ_PANEL + s];
                double x = A[p * ld + k];
#pragma unroll
                for (int q = 0; q < s; ++q) {
                    const double f = F[GJ_PANEL * p + q];
                    if (f != 0.0) x = fma(-f, rk[q], x);
                }
                rk[s] = x * meta[s];
                R[s * nb + k] = rk[s];
            }
        }
        __syncthreads();
        // ---- every row of those columns
        for (int k = kk; k < ncol; k += kl) {
            if (col0 + k >= c0 && col0 + k < c0 + width) continue;
            double rk[GJ_PANEL];
#pragma unroll
            for (int s = 0; s < GJ_PANEL; ++s) rk[s] = s < width ? R[s * nb + k] : 0.0;
#pragma unroll 2
            for (int i = row0; i < n; i += rows_per_pass) {
                const double2* f2 = reinterpret_cast<const double2*>(F + GJ_PANEL * i);
                const int mine = step[i];
                double x = A[i * ld + k];
#pragma unroll
                for (int h = 0; h < GJ_PANEL / 2; ++h) {
                    const double2 f = f2[h];
                    if (f.x != 0.0) x = fma(-f.x, rk[2 * h], x);
                    if (mine == 2 * h) x = rk[2 * h];
                    if (f.y != 0.0) x = fma(-f.y, rk[2 * h + 1], x);
                    if (mine == 2 * h + 1) x = rk[2 * h + 1];
                }
                A[i * ld + k] = x;
            }
        }
        __syncthreads();
        if (tid < width) step[perm[c0 + tid]] = 255;
    }
    __syncthreads();
    // row perm[c] holds variable c, column j the identity column perm[j]
    for (int x = tid; x < n * ncol; x += GJ_THREADS) {
        const int c = x / ncol, k = x - c * ncol;
        inv[(size_t)c * n + perm[col0 + k]] = A[perm[c] * ld + k];
    }
}

// The inverse by one cluster of `ctas` CTAs; false, with nothing launched,
// when n is too large or no such cluster can be resident.  `fac` holds
// gj_fac_size(n) doubles.  Sixteen CTAs (the opt-in size) were the fastest
// at every n above a panel or two: n 81 / 208 / 500 in 88 / 257 / 1077 us,
// with eight 91 / 292 us (500 does not fit), with one 132 us at n 81.
inline bool launch_gj_cluster(int64_t n, const int32_t* Cp, const int32_t* Ci, const double* Cx, double* inv,
                              double* fac, int* singular, cudaStream_t s, int ctas) {
    if (n < 1 || n > GJ_MAX) return false;
    const int nb = (int)((n + (int64_t)ctas * GJ_PANEL - 1) / ((int64_t)ctas * GJ_PANEL)) * GJ_PANEL;
    const size_t smem = GjSmem((int)n, nb).total;
    if (smem > 227 * 1024) return false;
    UP3D_CUDA(cudaFuncSetAttribute(k_gj_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    UP3D_CUDA(cudaFuncSetAttribute(k_gj_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(GJ_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fits = 0;
    UP3D_CUDA(cudaOccupancyMaxActiveClusters(&fits, k_gj_cluster, &cfg));
    if (fits < 1) return false;
    UP3D_CUDA(cudaLaunchKernelEx(&cfg, k_gj_cluster, (int)n, nb, Cp, Ci, Cx, inv, fac, singular));
    UP3D_CHECK_LAUNCH();
    return true;
}

inline bool launch_gj(int64_t n, const int32_t* Cp, const int32_t* Ci, const double* Cx, double* inv, double* fac,
                      int* singular, cudaStream_t s) {
    if (n <= 2 * GJ_PANEL) return launch_gj_cluster(n, Cp, Ci, Cx, inv, fac, singular, s, 1);
    return launch_gj_cluster(n, Cp, Ci, Cx, inv, fac, singular, s, 16) ||
           launch_gj_cluster(n, Cp, Ci, Cx, inv, fac, singular, s, 8);
}

}  // namespace up3d
