// Residual, Picard matrix and Newton Jacobian assembly of the up3d library.
//
// Two passes, no atomics:
//   1. an element sweep computes, per element, its residual contributions
//      R_i and its symmetric local matrix J_ij (Terms 1 + 2) -- all the
//      floating-point work, once per element, with coalesced loads;
//   2. a row gather: one warp per CSR row sums the contributions of the row
//      node's incident elements in a fixed order (the mesh-setup plan) and
//      writes the row once, coalesced.
// Every entry's summation order is fixed by the mesh, so results are
// bit-reproducible run to run, as the reference's colour-ordered scatter is
// (kernels/jacobian.py:1-33, kernels/residual.py:44-76).
//
// Term 3 (upstream coupling, off the element pattern) is built per call,
// row by row: each row's entries from its incident active elements in
// ascending element order, stably sorted by column in shared memory and
// summed per column -- the order of the reference's fill_term3_coo + COO ->
// CSR merge (kernels/jacobian.py:184-229, :344-358), without a global sort.

#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "elem.cuh"
#include "internal.cuh"
#include "tiles.cuh"

namespace up3d {

namespace {

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

constexpr int RG_WARPS = 8;   // warps per block of the row gather

// Minimum resident blocks per SM of the row gather (launch bounds).
#ifndef UP3D_ROW_MINB
#define UP3D_ROW_MINB 8
#endif
// ------------------------------------------------------------ element math

__device__ __forceinline__ void gB_of(const double g[3], const double* __restrict__ b, double gB[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) gB[j] = g[0] * b[3 * j] + g[1] * b[3 * j + 1] + g[2] * b[3 * j + 2];
}

// Local matrix of one element (kernels/jacobian.py:406-433):
//   J_ij = w1 (B_i . B_j)  [+ w2 gB_i gB_j when w2 != 0]
// Term 2 only when its weight is non-zero, so J reduces to the Picard
// matrix bitwise at s_e = 0.  Explicit fma pins the rounding, so every
// kernel that builds a local matrix produces identical bits.
__device__ __forceinline__ double bbij(const double* b, int i, int j) {
    return fma(b[3 * i + 2], b[3 * j + 2], fma(b[3 * i + 1], b[3 * j + 1], b[3 * i] * b[3 * j]));
}
__device__ __forceinline__ double jij(const double* b, const double gB[4], double w1, double w2, int i, int j) {
    double v = w1 * bbij(b, i, j);
    if (w2 != 0.0) v = fma(w2 * gB[i], gB[j], v);
    return v;
}

// Writes [R_0, J_00, ..., R_3, J_33, J_01, J_02, J_03, J_12, J_13, J_23].
__device__ __forceinline__ double2* loc_of(double* __restrict__ loc, int64_t e) {
    return reinterpret_cast<double2*>(loc + (size_t)LOC_STRIDE * e);
}
__device__ __forceinline__ void store_local(double2* __restrict__ p, const double* b, const double gB[4], double w1,
                                            double w2, bool with_r) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        p[i] = make_double2(with_r ? w1 * gB[i] : 0.0, jij(b, gB, w1, w2, i, i));
    p[4] = make_double2(jij(b, gB, w1, w2, 0, 1), jij(b, gB, w1, w2, 0, 2));
    p[5] = make_double2(jij(b, gB, w1, w2, 0, 3), jij(b, gB, w1, w2, 1, 2));
    p[6] = make_double2(jij(b, gB, w1, w2, 1, 3), jij(b, gB, w1, w2, 2, 3));
}

__device__ __forceinline__ void store_res(double* __restrict__ res, int64_t e, const double gB[4], double w1) {
    double2* p = reinterpret_cast<double2*>(res + 4 * e);
    p[0] = make_double2(w1 * gB[0], w1 * gB[1]);
    p[1] = make_double2(w1 * gB[2], w1 * gB[3]);
}

// Term-3 vectors of an active element: a_i = w3 gB_i (the reference's
// wi = w * gi), b_k = grad_u . B_u,k (kernels/jacobian.py:469-481).
__device__ __forceinline__ void store_t3(double* __restrict__ t3v, int64_t e, double w3, const double gB[4],
                                         const double f[4]) {
    double2* p = reinterpret_cast<double2*>(t3v + 8 * e);
    p[0] = make_double2(w3 * gB[0], w3 * gB[1]);
    p[1] = make_double2(w3 * gB[2], w3 * gB[3]);
    p[2] = make_double2(f[0], f[1]);
    p[3] = make_double2(f[2], f[3]);
}

__device__ __forceinline__ void load_B(const double* __restrict__ B, int64_t e, double b[12]) { ld_B(B + 12 * e, b); }

// ------------------------------------------------------------ row gather

// Sums over a row's incident entries k < deg in a fixed order that does
// not depend on the lanes per row: entry k goes to slot k mod 4, each slot
// sums its entries in ascending k, and the row sum is (s0 + s2) + (s1 + s3).
// LPR lanes per row (LPR >= 4; lane `sub` of the row's group loads entry
// k0 + sub of each chunk of LPR entries through load(k) -> (x, y)); the
// sums of x and y land in lane sub == 0.  Every lane of the warp must call
// it (warp-uniform trip count over the warp's longest row).
template <int LPR, class Load>
__device__ __forceinline__ void slot_sum(int deg, int sub, Load&& load, double& sx, double& sy) {
    static_assert(LPR >= 4 && LPR <= 32 && (LPR & (LPR - 1)) == 0, "LPR: power of two in [4, 32]");
    const int maxdeg = __reduce_max_sync(0xffffffffu, deg);
    double x = 0.0, y = 0.0;  // slot sub & 3 in lanes sub < 4
    for (int k0 = 0; k0 < maxdeg; k0 += LPR) {
        double2 v = make_double2(0.0, 0.0);
        if (k0 + sub < deg) v = load(k0 + sub);
#pragma unroll
        for (int j = 0; j < LPR / 4; ++j) {
            const double vx = j == 0 ? v.x : __shfl_down_sync(0xffffffffu, v.x, 4 * j, LPR);
            const double vy = j == 0 ? v.y : __shfl_down_sync(0xffffffffu, v.y, 4 * j, LPR);
            if (k0 + (sub & 3) + 4 * j < deg) {
                x += vx;
                y += vy;
            }
        }
    }
    x += __shfl_down_sync(0xffffffffu, x, 2, LPR);
    y += __shfl_down_sync(0xffffffffu, y, 2, LPR);
    x += __shfl_down_sync(0xffffffffu, x, 1, LPR);
    y += __shfl_down_sync(0xffffffffu, y, 1, LPR);
    sx = x;
    sy = y;
}

// Jacobian rows (and, when R != null, the residual) from the local
// matrices, LPR lanes per row (32 / LPR rows per warp in flight):
//   R_n  = sum_e R_e,i        J_nn = sum_e J_e,ii      (in the order of
//   slot_sum: the same bits for every LPR and for the residual-only gather)
//   J_nm = sum_e J_e,ij  for the upper slots m > n (lanes stride the slots;
//   each slot sums its plan's contributors in ascending element order) and
//   is written to (n, m) and, the element matrices being symmetric and row m
//   listing the same elements in the same order, to its transposed slot.
// P8: the upper slots read their contributors from the fixed-width records
// (plan8, one 32-byte record per slot found from up_off) instead of
// plan_off -> plan: one dependent load less, the same order and bits.
template <int WARPS, int LPR, bool P8>
__global__ void __launch_bounds__(WARPS * 32, UP3D_ROW_MINB)
    k_row_gather(int64_t N, const int32_t* __restrict__ ent_off, const uint32_t* __restrict__ ent,
                 const int32_t* __restrict__ indptr, const int32_t* __restrict__ plan_off,
                 const uint32_t* __restrict__ plan, const int32_t* __restrict__ diag,
                 const int32_t* __restrict__ zt, const int32_t* __restrict__ up_off,
                 const uint32_t* __restrict__ plan8, const double* __restrict__ loc, double* __restrict__ R,
                 double* __restrict__ J) {
    static_assert(LPR >= 1 && LPR <= 32 && (LPR & (LPR - 1)) == 0, "LPR: power of two <= 32");
    constexpr int RPW = 32 / LPR;
    const int lane = threadIdx.x & 31, sub = lane & (LPR - 1);
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    // warp-uniform trip count: every lane reaches the shuffles
    for (int64_t base = warp * RPW; base < N; base += n_warps * RPW) {
        const int64_t n = base + lane / LPR;
        const bool valid = n < N;
        int32_t eb = 0, deg = 0, rb = 0, L = 0, ds = -1, uo = 0;
        if (valid) {
            eb = ent_off[n];
            deg = ent_off[n + 1] - eb;
            rb = indptr[n];
            L = indptr[n + 1] - rb;
            ds = diag[n];
            if (P8) uo = up_off[n];
        }
        double r, d;
        slot_sum<LPR>(deg, sub, [&](int k) {
            const uint32_t x = ent[eb + k];
            return reinterpret_cast<const double2*>(loc + (size_t)LOC_STRIDE * (x >> 2))[x & 3];
        }, r, d);
        for (int s = ds + 1 + sub; s < L; s += LPR) {
            double v = 0.0;
            if constexpr (P8) {
                const uint4* rec = reinterpret_cast<const uint4*>(plan8 + (size_t)PLAN8 * (uo + (s - ds - 1)));
                const uint4 h0 = __ldg(rec), h1 = __ldg(rec + 1);
                const uint32_t c[PLAN8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                double a[PLAN8];
#pragma unroll
                for (int k = 0; k < PLAN8; ++k)
                    a[k] = c[k] != PLAN8_END ? loc[(size_t)LOC_STRIDE * (c[k] >> 3) + 8 + (c[k] & 7)] : 0.0;
#pragma unroll
                for (int k = 0; k < PLAN8; ++k)
                    if (c[k] != PLAN8_END) v += a[k];
                J[rb + s] = v;
                J[zt[rb + s]] = v;
                continue;
            }
            int32_t p = plan_off[rb + s];
            const int32_t p1 = plan_off[rb + s + 1];
            for (; p + 3 < p1; p += 4) {
                const uint32_t c0 = plan[p], c1 = plan[p + 1], c2 = plan[p + 2], c3 = plan[p + 3];
                const double a0 = loc[(size_t)LOC_STRIDE * (c0 >> 3) + 8 + (c0 & 7)];
                const double a1 = loc[(size_t)LOC_STRIDE * (c1 >> 3) + 8 + (c1 & 7)];
                const double a2 = loc[(size_t)LOC_STRIDE * (c2 >> 3) + 8 + (c2 & 7)];
                const double a3 = loc[(size_t)LOC_STRIDE * (c3 >> 3) + 8 + (c3 & 7)];
                v += a0;
                v += a1;
                v += a2;
                v += a3;
            }
            for (; p < p1; ++p) {
                const uint32_t c0 = plan[p];
                v += loc[(size_t)LOC_STRIDE * (c0 >> 3) + 8 + (c0 & 7)];
            }
            J[rb + s] = v;
            J[zt[rb + s]] = v;
        }
        if (valid && sub == 0) {
            if (deg > 0) J[rb + ds] = d;  // a node of no element has an empty row
            if (R) R[n] = r;
        }
    }
}

// Residual rows only: R_n = sum_e R_e,i from the compact residual array,
// 8 lanes per row, in the row gather's order (slot_sum).
__global__ void __launch_bounds__(256)
    k_row_residual(int64_t N, const int32_t* __restrict__ ent_off, const uint32_t* __restrict__ ent,
                   const double* __restrict__ res, double* __restrict__ R) {
    constexpr int LPR = 8, RPW = 32 / LPR;
    const int lane = threadIdx.x & 31, sub = lane & (LPR - 1);
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = warp * RPW; base < N; base += n_warps * RPW) {
        const int64_t n = base + lane / LPR;
        int32_t eb = 0, deg = 0;
        if (n < N) {
            eb = ent_off[n];
            deg = ent_off[n + 1] - eb;
        }
        double r, unused;
        slot_sum<LPR>(deg, sub, [&](int k) {
            const uint32_t x = ent[eb + k];
            return make_double2(res[4 * (size_t)(x >> 2) + (x & 3)], 0.0);
        }, r, unused);
        if (n < N && sub == 0) R[n] = r;
    }
}

// ------------------------------------------------------------ prep kernels
// Element sweeps of the single-purpose entry points.

// assemble_residual: velocities into the workspace (kernels/jacobian.py:623)
// and the residual contributions w1 gB_i with w1 = rho_tilde V.
__global__ void k_prep_residual(const int4* __restrict__ conn, const double* __restrict__ B,
                                const double* __restrict__ V, const double* __restrict__ phi,
                                const double* __restrict__ rt, int64_t E, double* __restrict__ grad,
                                double* __restrict__ q2, double* __restrict__ res) {
    GRID_STRIDE(e, E) {
        double g[3], b[12];
        int4 c;
        elem_grad_B(conn, B, phi, e, g, b, c);
        grad[3 * e] = g[0];
        grad[3 * e + 1] = g[1];
        grad[3 * e + 2] = g[2];
        q2[e] = dot3r(g[0], g[1], g[2], g[0], g[1], g[2]);
        double gB[4];
        gB_of(g, b, gB);
        store_res(res, e, gB, (rt ? rt[e] : 1.0) * V[e]);
    }
}

// assemble_matrix: J_ij = rho_tilde V (B_i . B_j).
__global__ void k_prep_matrix(const double* __restrict__ B, const double* __restrict__ V,
                              const double* __restrict__ rt, int64_t E, double* __restrict__ loc) {
    GRID_STRIDE(e, E) {
        double b[12];
        load_B(B, e, b);
        const double z[4] = {0.0, 0.0, 0.0, 0.0};
        store_local(loc_of(loc, e), b, z, (rt ? rt[e] : 1.0) * V[e], 0.0, false);
    }
}

// assemble_newton_jacobian (kernels/jacobian.py:323-338, :410-414): the
// limiter mask gates s_e by lim[e] and s_u by lim[upstream[e]]; Term-2 and
// Term-3 weights 2 inv_u2 s V; Term-3 vectors of active elements
// (s_u != 0), counted into *n_active.  grad(phi) of the element, and of an
// active element's upstream, is formed here (the reference's scratch
// velocities, :328-332).
__global__ void k_prep_jacobian(const int4* __restrict__ conn, const double* __restrict__ B,
                                const double* __restrict__ V, const double* __restrict__ phi,
                                const double* __restrict__ rt, const double* __restrict__ se,
                                const double* __restrict__ su, const int64_t* __restrict__ up,
                                const uint8_t* __restrict__ lim, double inv_u2, int64_t E, double* __restrict__ loc,
                                double* __restrict__ t3v, uint8_t* __restrict__ t3flag, int32_t* __restrict__ up32,
                                unsigned long long* __restrict__ n_active) {
    unsigned long long count = 0;
    GRID_STRIDE(e, E) {
        double b[12], g[3], gB[4];
        int4 c;
        elem_grad_B(conn, B, phi, e, g, b, c);
        gB_of(g, b, gB);
        int64_t u = safe_up(up[e], e, E);
        double s_e = se[e], s_u = su[e];
        if (lim) {
            s_e = s_e * (lim[e] ? 1.0 : 0.0);
            s_u = s_u * (lim[u] ? 1.0 : 0.0);
        }
        const double Ve = V[e];
        const double w2 = 2.0 * inv_u2 * s_e * Ve;
        const double w3 = 2.0 * inv_u2 * s_u * Ve;
        const bool active = s_u != 0.0;
        if (active) {
            double bu[12], gu[3], f[4];
            int4 cu;
            elem_grad_B(conn, B, phi, u, gu, bu, cu);
            gB_of(gu, bu, f);
            store_t3(t3v, e, w3, gB, f);
            ++count;
        }
        t3flag[e] = active ? 1 : 0;
        up32[e] = (int32_t)u;
        store_local(loc_of(loc, e), b, gB, rt[e] * Ve, w2, false);
    }
    count = warp_sum_u64(count);
    if ((threadIdx.x & 31) == 0 && count) atomicAdd(n_active, count);
}

// ------------------------------------------------------------ fused sweep

struct MonAcc {   // one thread's counts: below 2^31 with the elements
    double nu_max = 0.0;
    unsigned sup = 0, flo = 0, lim = 0, act = 0;
};

__device__ __forceinline__ void flush(MonAcc a, up3d_monitors* mon) {
    double nm = warp_max(a.nu_max);
    unsigned long long s = warp_sum_u64(a.sup), f = warp_sum_u64(a.flo), l = warp_sum_u64(a.lim),
                       t = warp_sum_u64(a.act);
    if ((threadIdx.x & 31) == 0) {
        if (nm > 0.0) atomic_max_nonneg(&mon->nu_max, nm);
        if (s) atomicAdd(reinterpret_cast<unsigned long long*>(&mon->n_supersonic), s);
        if (f) atomicAdd(reinterpret_cast<unsigned long long*>(&mon->n_floored), f);
        if (l) atomicAdd(reinterpret_cast<unsigned long long*>(&mon->n_limited), l);
        if (t) atomicAdd(reinterpret_cast<unsigned long long*>(&mon->n_term3_active), t);
    }
}

// A warp's 32 consecutive records leave through a slab of shared memory as
// one bulk store of contiguous bytes: a lane storing its own 112 bytes puts a
// line per lane through the load/store unit (3.6 M tets: 275 -> 265 us).
__device__ __forceinline__ void slab_free(int lane) {  // the last store has read the slab
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
}
__device__ __forceinline__ void slab_store(double* dst, const double2* src, unsigned bytes, int lane) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                     "r"((unsigned)__cvta_generic_to_shared(src)), "r"(bytes)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
}
__device__ __forceinline__ void slab_done(int lane) {  // written, before the block ends
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// eval_residual + assemble_coupled, per element (pyfp3d/solve/newton.py:
// 345-372, :435-452): gradient, limiter, density, upstream walk (or the
// frozen selection), the upstream element's state recomputed in place, the
// flux, its sensitivities, and the element's residual contributions and
// local matrix (JAC) or residual contributions only.  B_e and V_e are
// recomputed from the node coordinates (geom_B, the mesh set-up's
// arithmetic, so the same bits) instead of streamed: the coordinates are
// gathered for the walk anyway, and 104 bytes per element stay in HBM.
// BATCH: several cases in one mesh (disconnected components), element e
// taking the flow of its case, flows[case_of[e]] (an index outside
// [0, n_cases) reads case 0: the host validates the indices, and a table
// reused without validation can never be read out of bounds).
// AIR: gamma == 1.4 in every flow (no pow, and the registers it takes).
// NT threads per block, MB resident blocks per SM that the register
// allocation must allow.
// What bounds it: the latency of the walk's dependent loads at the few warps
// that its registers leave (3.6 M tets, 20 warps per SM: issue slots 30 %,
// FP64 pipe 32 %, load/store wavefronts 68 % busy), so registers and
// wavefronts are what pays: 304 us with int64 ids and pow, 287 with neither,
// 275 without the switch of subcritical pairs, 264 with the records stored in
// bulk; residual only 238 -> 211.  14.7 M tets: 1187 -> 1092 us.  Tried and
// slower: the walk as a kernel of its own (297), B_e kept in the slab instead
// of formed again (259 against 256, residual only 230 against 214), the next
// tile's records prefetched into L2 (256 at 3.6 M, but 1240 at 14.7 M).
template <bool FROZEN, bool JAC, bool BATCH, bool AIR, int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    k_fused_elem(const int4* __restrict__ conn, const int4* __restrict__ fn, const double* __restrict__ disp,
                 const double4* __restrict__ X, const double* __restrict__ phi, Flow F0, double u2,
                 const int64_t* __restrict__ up_fz,
                 const int8_t* __restrict__ br_fz, int64_t E, double* __restrict__ loc, double* __restrict__ res,
                 double* __restrict__ t3v, uint8_t* __restrict__ t3flag, int32_t* __restrict__ up_out,
                 double* __restrict__ rt_out, up3d_monitors* mon, const Flow* __restrict__ flows,
                 const int32_t* __restrict__ case_of, int n_cases, int8_t* __restrict__ br_out) {
    constexpr int LOC2 = LOC_STRIDE / 2;
    // the test for subcritical pairs, except in the frozen Jacobian of other
    // gases, whose elements rarely take it and whose upstream pow is better
    // early (gamma 1.3, 8.2 M tets, 768 threads persistent: 968 us without, 1107
    // with it; 640 threads 1004 and 1078)
    constexpr bool SKIP = AIR || !FROZEN || !JAC;
    __shared__ double2 slab[JAC ? NT * LOC2 : 1];  // the local records of each warp's 32 elements
    const int lane = threadIdx.x & 31;
    double2* const mine = slab + (JAC ? (threadIdx.x - lane) * LOC2 : 0);
    MonAcc acc;
    // tiles of NT elements, block-strided over the grid; element ids in 32
    // bits (E < 2^29), which with the counts costs 12 registers less
    const int n = (int)E;
    for (int e0 = blockIdx.x * NT + (threadIdx.x - lane); e0 < n; e0 += gridDim.x * NT) {
        if (JAC) slab_free(lane);
        const int e = e0 + lane;
        if (e < n) {
            int ci = 0;
            if (BATCH) {
                ci = case_of[e];
                ci = (unsigned)ci < (unsigned)n_cases ? ci : 0;
            }
            const Flow& F = BATCH ? flows[ci] : F0;
            // only grad phi_e stays live through the walk; the element's own
            // state and gB_j = grad . B_j are formed after it (B_e recomputed
            // from the coordinates, L1/L2 hits)
            const int4 ce = conn[e];
            double g[3], Ve;
            {
                double bb[12];
                geom_B(X, ce, bb, Ve);
                grad_from_B(ce, bb, phi, g);
            }
            // frozen (upstream, branch) per element; a negative branch keeps the
            // element live (several cases in one mesh, frozen one by one)
            const int brf = FROZEN ? (int)br_fz[e] : -1;
            const bool frz = FROZEN && brf >= 0;
            const int u = frz ? (int)safe_up(up_fz[e], e, E) : upstream_walk(fn, disp, X, ce, e, n, g);
            double q2n = __ddiv_rn(dot3r(g[0], g[1], g[2], g[0], g[1], g[2]), u2);
            double q2l = q2n < F.q2cap ? q2n : F.q2cap;
            bool lim_e = q2l == q2n;
            double rho_e, drho_e;
            rho_drho<AIR>(q2l, F, rho_e, drho_e);
            // upstream state, and its Term-3 factors grad_u . B_u,k
            double q2lu = q2l, rho_u = rho_e;
            bool lim_u = lim_e;
            if (u != e) {
                double gu[3];
                {
                    const int4 cu = conn[u];
                    double bu[12], vu;
                    geom_B(X, cu, bu, vu);
                    grad_from_B(cu, bu, phi, gu);
                }
                double q2nu = __ddiv_rn(dot3r(gu[0], gu[1], gu[2], gu[0], gu[1], gu[2]), u2);
                q2lu = q2nu < F.q2cap ? q2nu : F.q2cap;
                lim_u = q2lu == q2nu;
                if (!SKIP) rho_u = rho_of<AIR>(q2lu, F);
            }
            // both elements surely subcritical: the switch is 0, no upstream
            // density, Mach number or switch enters (four divisions and a root)
            const bool sub = SKIP && !frz && q2l <= F.q2sub && q2lu <= F.q2sub;
            if (SKIP && u != e && !sub) rho_u = rho_of<AIR>(q2lu, F);
            acc.lim += !lim_e;

            double nu, rt, s_e = 0.0, s_u = 0.0;
            if (frz) {
                const int br = brf;
                if (br_out) br_out[e] = (int8_t)br;
                if (br == 3) {
                    nu = 0.0;
                    rt = F.floor_;
                    acc.flo += 1;
                } else if (br == 0) {
                    nu = 0.0;
                    rt = rho_e;
                } else {
                    nu = switch_of(mach2_of(br == 1 ? q2l : q2lu, F), F);
                    rt = rho_e - nu * (rho_e - rho_u);
                }
                if (JAC) frozen_sensitivities<AIR>(br, q2l, rho_e, q2lu, rho_u, F, s_e, s_u);
            } else if (sub) {
                nu = 0.0;
                const bool floored = rho_e <= F.floor_;
                rt = rho_e > F.floor_ ? rho_e : F.floor_;
                acc.flo += (rt == F.floor_);
                if (br_out) br_out[e] = floored ? 3 : 0;
                if (JAC) s_e = floored ? 0.0 : drho_e;
            } else {
                const double nu_e = switch_of(mach2_of(q2l, F), F), nu_u = switch_of(mach2_of(q2lu, F), F);
                nu = fmax(nu_e, nu_u);
                rt = rho_e - nu * (rho_e - rho_u);
                // the branch this live evaluation took (classify_upwind_branches,
                // kernels/upwind.py:504-541)
                if (br_out)
                    br_out[e] = (int8_t)(u == e ? (rho_e <= F.floor_ ? 3 : 0)
                                                : (rt <= F.floor_ ? 3 : (nu == 0.0 ? 0 : (nu_e >= nu_u ? 1 : 2))));
                rt = rt > F.floor_ ? rt : F.floor_;
                acc.flo += (rt == F.floor_);
                if (JAC) live_sensitivities<AIR>(q2l, rho_e, q2lu, rho_u, u == e, F, s_e, s_u);
            }
            acc.nu_max = fmax(acc.nu_max, nu);
            acc.sup += (nu > 0.0);

            const double w1 = rt * Ve;
            // B_e again (recomputed), held in registers from here
            double b[12];
            {
                double vtmp;
                geom_B(X, ce, b, vtmp);
            }
            double gB[4];
            gB_of(g, b, gB);
            if (JAC) {
                s_e = s_e * (lim_e ? 1.0 : 0.0);
                s_u = s_u * (lim_u ? 1.0 : 0.0);
                const double w2 = 2.0 * F.inv_u2 * s_e * Ve;
                const double w3 = 2.0 * F.inv_u2 * s_u * Ve;
                const bool active = s_u != 0.0;
                if (active) {
                    // Term-3 factors grad_u . B_u,k, recomputed for the (few)
                    // active elements only
                    double f[4] = {gB[0], gB[1], gB[2], gB[3]};
                    if (u != e) {
                        double gu[3], bu[12];
                        int4 cu;
                        cu = conn[u];
                        double vu;
                        geom_B(X, cu, bu, vu);
                        grad_from_B(cu, bu, phi, gu);
                        gB_of(gu, bu, f);
                    }
                    store_t3(t3v, e, w3, gB, f);
                    acc.act += 1;
                }
                t3flag[e] = active ? 1 : 0;
                store_local(mine + LOC2 * lane, b, gB, w1, w2, true);
            } else {
                store_res(res, e, gB, w1);
            }
            up_out[e] = (int32_t)u;
            if (rt_out) rt_out[e] = rt;
        }
        if (JAC)
            slab_store(loc + (size_t)LOC_STRIDE * e0, mine, min(32, n - e0) * LOC_STRIDE * sizeof(double), lane);
    }
    if (JAC) slab_done(lane);
    flush(acc, mon);
}

// ------------------------------------------------------------ tiled sweep

// Arguments of the tiled evaluation (tiles.cuh): the plan's arrays, the
// inputs and the outputs.  Element arrays of the plan are in internal
// (tile) order; per-element outputs are written in user order.
struct TileArgs {
    const int4* conn;        // (E) global node ids, internal order
    const int4* fnbr;        // (E) internal ids
    const double4* cen;      // (E) internal order
    const double* disp;      // (E, 12) internal order
    const double4* X;        // (N) node positions
    const double* phi;       // (N)
    const int32_t* perm;     // internal -> user
    const int32_t* iperm;    // user -> internal
    const int32_t* eoff;
    const int32_t* noff;
    const int32_t* uoff;
    const int32_t* tnode;
    const double4* txyz;
    const ushort4* lconn;
    const int32_t* nent_off;
    const uint16_t* nent;
    const int2* ndst;
    const int32_t* uent_off;
    const uint16_t* uent;
    const int2* udst;
    double* part;
    double* R;
    double* J;
    double* t3v;
    uint8_t* t3flag;
    int32_t* up_out;
    double* rt_out;
    int8_t* br_out;
    up3d_monitors* mon;
    const int64_t* up_fz;
    const int8_t* br_fz;
    const Flow* flows;
    const int32_t* case_of;
    int n_cases;
    int max_nodes;
    int max_edges;
    int64_t E;
    int64_t n_tiles;
    Flow F0;
    double u2;
};

// Shared memory of one tile of NT elements (byte offsets, each region
// 16-byte aligned): the tile's node positions (x, y, z, 0; copied
// asynchronously from the plan's tile-ordered table) and potentials; per
// element its centroid, gradient, unlimited q^2 and density, 14 local
// values (LOC layout), face neighbours, local connectivity, limiter flag
// and user id -- structure of arrays; then the tile's slice of the plan
// (node-entry offsets, node destinations, node-entry codes, edge offsets,
// edge destinations, edge codes), copied asynchronously in whole 16-byte
// blocks while the elements are evaluated.
constexpr int TS_DOUBLES = 8 + LOC_STRIDE;  // cx cy cz gx gy gz q2 rho + loc
struct TileSmem {
    size_t xs, phi, sd, fn, lc, lim, perm, noff, ndst, nent, uoff, udst, uent, total;
    __host__ __device__ static constexpr size_t up16(size_t b) { return (b + 15) & ~size_t(15); }
    __host__ __device__ TileSmem(int max_nodes, int max_edges, int nt) {
        size_t o = 0;
        xs = o;   o += up16((size_t)max_nodes * sizeof(double4));
        phi = o;  o += up16((size_t)max_nodes * sizeof(double));
        sd = o;   o += up16((size_t)nt * TS_DOUBLES * sizeof(double));
        fn = o;   o += up16((size_t)nt * sizeof(int4));
        lc = o;   o += up16((size_t)nt * sizeof(ushort4));
        lim = o;  o += up16((size_t)nt);
        perm = o; o += up16((size_t)nt * sizeof(int32_t));
        // staged plan ranges: at most 15 bytes before the range plus 15 after
        noff = o; o += up16((size_t)(max_nodes + 1) * sizeof(int32_t)) + 32;
        ndst = o; o += up16((size_t)max_nodes * sizeof(int2)) + 32;
        nent = o; o += up16((size_t)4 * nt * sizeof(uint16_t)) + 32;
        uoff = o; o += up16((size_t)(max_edges + 1) * sizeof(int32_t)) + 32;
        udst = o; o += up16((size_t)max_edges * sizeof(int2)) + 32;
        uent = o; o += up16((size_t)6 * nt * sizeof(uint16_t)) + 32;
        total = o;
    }
};

// Asynchronous global -> shared copies (cp.async, 16-byte blocks).
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// Copies the bytes [src, src + bytes) into shared memory at dst in whole
// 16-byte blocks starting at the block that holds src (the plan's arrays
// are padded by 16 bytes, so the last block stays inside the allocation);
// returns the offset of src's first byte within dst.
__device__ __forceinline__ int stage16(unsigned char* dst, const void* src, size_t bytes, int tid, int nt) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(src);
    const unsigned char* base = reinterpret_cast<const unsigned char*>(a & ~uintptr_t(15));
    const int delta = (int)(a & 15);
    const int nblk = (int)((delta + bytes + 15) >> 4);
    for (int b = tid; b < nblk; b += nt) cp_async16(dst + 16 * b, base + 16 * b);
    return delta;
}

// Local values of one element into the tile's shared memory (the
// arithmetic of store_local: R_i, J_ii pairs, then the six J_ij).
__device__ __forceinline__ void store_local_s(double* __restrict__ sloc, int nt, int l, const double* b,
                                              const double gB[4], double w1, double w2) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        sloc[(2 * i) * nt + l] = w1 * gB[i];
        sloc[(2 * i + 1) * nt + l] = jij(b, gB, w1, w2, i, i);
    }
    sloc[8 * nt + l] = jij(b, gB, w1, w2, 0, 1);
    sloc[9 * nt + l] = jij(b, gB, w1, w2, 0, 2);
    sloc[10 * nt + l] = jij(b, gB, w1, w2, 0, 3);
    sloc[11 * nt + l] = jij(b, gB, w1, w2, 1, 2);
    sloc[12 * nt + l] = jij(b, gB, w1, w2, 1, 3);
    sloc[13 * nt + l] = jij(b, gB, w1, w2, 2, 3);
}

// The fused evaluation of k_fused_elem with the row gather folded in, one
// CTA per tile of at most NT elements (one thread per element), a
// persistent grid looping over the tiles:
//   P0  the tile's node positions and potentials, the elements' local
//       connectivity and face neighbours into shared memory;
//   P1  per element: B_e and V_e from the staged positions (the mesh
//       set-up's arithmetic), the gradient, q^2, the limiter, the density
//       and the centroid (k_geometry's arithmetic) into shared memory;
//   P2  the upstream walk (or the frozen selection): displacements
//       cen(nbr) - cen(cur) formed from shared memory while the walk stays
//       in the tile, from the internal-order centroid table outside it --
//       the same IEEE operations as the precomputed displacements, so the
//       same selections;
//   P3  the upstream element's state from shared memory (or recomputed
//       from global memory when the walk left the tile);
//   P4  flux, sensitivities, residual vector and local matrix into shared
//       memory, Term-3 vectors of active elements to global memory;
//   P5  every output of the tile summed over its contributors in the
//       plan's order (ascending local element), written to R / J when the
//       tile holds all its contributors, else to the partial buffer.
// Per-element outputs (upstream, rho~, branch, Term-3 vectors and flags)
// go to user order through perm.
template <bool FROZEN, bool JAC, bool BATCH, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_tile_eval(const __grid_constant__ TileArgs a) {
    extern __shared__ __align__(16) unsigned char tsm[];
    const TileSmem L(a.max_nodes, a.max_edges, NT);
    double4* xs = reinterpret_cast<double4*>(tsm + L.xs);
    double* sphi = reinterpret_cast<double*>(tsm + L.phi);
    double* sd = reinterpret_cast<double*>(tsm + L.sd);
    double* scx = sd;
    double* scy = sd + NT;
    double* scz = sd + 2 * NT;
    double* sgx = sd + 3 * NT;
    double* sgy = sd + 4 * NT;
    double* sgz = sd + 5 * NT;
    double* sq2 = sd + 6 * NT;
    double* srho = sd + 7 * NT;
    double* sloc = sd + 8 * NT;
    int4* sfn = reinterpret_cast<int4*>(tsm + L.fn);
    ushort4* slc = reinterpret_cast<ushort4*>(tsm + L.lc);
    uint8_t* slim = tsm + L.lim;
    int32_t* sperm = reinterpret_cast<int32_t*>(tsm + L.perm);
    const int tid = threadIdx.x;
    const int64_t E = a.E;
    MonAcc acc;
    for (int64_t t = blockIdx.x; t < a.n_tiles; t += gridDim.x) {
        const int32_t e0 = a.eoff[t], ne = a.eoff[t + 1] - e0;
        const int32_t n0 = a.noff[t], nn = a.noff[t + 1] - n0;
        const int32_t u0 = a.uoff[t], nu = a.uoff[t + 1] - u0;
        // ---- P0: positions (group 1), the plan slice (group 2), potentials
        stage16(tsm + L.xs, a.txyz + n0, (size_t)nn * sizeof(double4), tid, NT);
        cp_async_commit();
        const int d_noff = stage16(tsm + L.noff, a.nent_off + n0, (size_t)(nn + 1) * sizeof(int32_t), tid, NT);
        const int d_ndst = stage16(tsm + L.ndst, a.ndst + n0, (size_t)nn * sizeof(int2), tid, NT);
        const int d_nent = stage16(tsm + L.nent, a.nent + 4 * (int64_t)e0, (size_t)4 * ne * sizeof(uint16_t), tid, NT);
        int d_uoff = 0, d_udst = 0, d_uent = 0;
        if (JAC) {
            d_uoff = stage16(tsm + L.uoff, a.uent_off + u0, (size_t)(nu + 1) * sizeof(int32_t), tid, NT);
            d_udst = stage16(tsm + L.udst, a.udst + u0, (size_t)nu * sizeof(int2), tid, NT);
            d_uent = stage16(tsm + L.uent, a.uent + 6 * (int64_t)e0, (size_t)6 * ne * sizeof(uint16_t), tid, NT);
        }
        cp_async_commit();
        for (int r = tid; r < nn; r += NT) sphi[r] = a.phi[a.tnode[n0 + r]];
        const bool act = tid < ne;
        const int64_t xe = (int64_t)e0 + tid;
        int32_t user = 0;
        ushort4 lc = make_ushort4(0, 0, 0, 0);
        if (act) {
            lc = a.lconn[xe];
            slc[tid] = lc;
            sfn[tid] = a.fnbr[xe];
            user = a.perm[xe];
            sperm[tid] = user;
        }
        cp_async_wait<1>();  // this thread's position blocks are in
        __syncthreads();
        // ---- P1
        int ci = 0;
        if (BATCH && act) {
            ci = a.case_of[user];
            ci = (unsigned)ci < (unsigned)a.n_cases ? ci : 0;
        }
        const Flow& F = BATCH ? a.flows[ci] : a.F0;
        double g[3] = {0.0, 0.0, 0.0}, Ve = 0.0, q2l = 0.0, rho_e = 0.0, ccx = 0.0, ccy = 0.0, ccz = 0.0;
        bool lim_e = true;
        if (act) {
            const double4 p0 = xs[lc.x], p1 = xs[lc.y], p2 = xs[lc.z], p3 = xs[lc.w];
            {
                double bb[12];
                geom_B_pts(p0.x, p0.y, p0.z, p1.x, p1.y, p1.z, p2.x, p2.y, p2.z, p3.x, p3.y, p3.z, bb, Ve);
                const double f0 = sphi[lc.x], f1 = sphi[lc.y], f2 = sphi[lc.z], f3 = sphi[lc.w];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    g[d] = radd(radd(radd(rmul(f0, bb[d]), rmul(f1, bb[3 + d])), rmul(f2, bb[6 + d])),
                                rmul(f3, bb[9 + d]));
            }
            const double q2n = __ddiv_rn(dot3r(g[0], g[1], g[2], g[0], g[1], g[2]), a.u2);
            q2l = q2n < F.q2cap ? q2n : F.q2cap;
            lim_e = q2l == q2n;
            rho_e = rho_of(q2l, F);
            ccx = radd(radd(radd(p0.x, p1.x), p2.x), p3.x) * 0.25;
            ccy = radd(radd(radd(p0.y, p1.y), p2.y), p3.y) * 0.25;
            ccz = radd(radd(radd(p0.z, p1.z), p2.z), p3.z) * 0.25;
            scx[tid] = ccx;
            scy[tid] = ccy;
            scz[tid] = ccz;
            sgx[tid] = g[0];
            sgy[tid] = g[1];
            sgz[tid] = g[2];
            sq2[tid] = q2n;
            srho[tid] = rho_e;
            slim[tid] = lim_e ? 1 : 0;
        }
        __syncthreads();
        if (act) {
            // ---- P2: upstream element (internal id)
            const int brf = FROZEN ? (int)a.br_fz[user] : -1;
            const bool frz = FROZEN && brf >= 0;
            int64_t u = xe;
            if (frz) {
                u = a.iperm[safe_up(a.up_fz[user], user, E)];
            } else {
                const double gx = g[0], gy = g[1], gz = g[2];
                double pmin = 1e300, pmax = -1e300;
                {
                    const unsigned short li[4] = {lc.x, lc.y, lc.z, lc.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const double4 p = xs[li[k]];
                        const double pr = dot3r(p.x, p.y, p.z, gx, gy, gz);
                        if (pr < pmin) pmin = pr;
                        if (pr > pmax) pmax = pr;
                    }
                }
                const double target = rmul(0.8, rsub(pmax, pmin));
                double reach = 0.0;
                int64_t cur = xe;
                for (int hops = 0; hops < 4 && reach < target; ++hops) {
                    const uint32_t lcur = (uint32_t)(cur - e0);
                    int nb[4];
                    double d[4];
                    if (lcur < (uint32_t)ne) {
                        // inside the tile: cen(nbr) - cen(cur) from shared memory
                        // (a neighbour outside the tile from the centroid table)
                        const int4 f = sfn[lcur];
                        nb[0] = f.x; nb[1] = f.y; nb[2] = f.z; nb[3] = f.w;
                        const double cx = scx[lcur], cy = scy[lcur], cz = scz[lcur];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            d[k] = 0.0;
                            if (nb[k] >= 0 && nb[k] < E) {
                                const uint32_t ln = (uint32_t)(nb[k] - e0);
                                double nx, ny, nz;
                                if (ln < (uint32_t)ne) {
                                    nx = scx[ln];
                                    ny = scy[ln];
                                    nz = scz[ln];
                                } else {
                                    double w;
                                    ld4(reinterpret_cast<const double*>(a.cen + nb[k]), nx, ny, nz, w);
                                }
                                d[k] = dot3r(rsub(nx, cx), rsub(ny, cy), rsub(nz, cz), gx, gy, gz);
                            }
                        }
                    } else {
                        // outside: the precomputed displacement record (the
                        // same rounded differences), one load next to fnbr
                        const int4 f = a.fnbr[cur];
                        nb[0] = f.x; nb[1] = f.y; nb[2] = f.z; nb[3] = f.w;
                        double r[12];
                        ld_B(a.disp + 12 * cur, r);
#pragma unroll
                        for (int k = 0; k < 4; ++k) d[k] = dot3r(r[3 * k], r[3 * k + 1], r[3 * k + 2], gx, gy, gz);
                    }
                    int64_t best = -1;
                    double best_disp = 0.0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (nb[k] >= 0 && nb[k] < E && d[k] < best_disp) {
                            best_disp = d[k];
                            best = nb[k];
                        }
                    }
                    if (best < 0) break;
                    cur = best;
                    reach = radd(reach, -best_disp);
                }
                u = cur;
            }
            // ---- P3: the upstream element's state
            const uint32_t lu = (uint32_t)(u - e0);
            const bool u_in = lu < (uint32_t)ne;
            double q2lu = q2l, rho_u = rho_e;
            bool lim_u = lim_e;
            if (u != xe) {
                double q2nu;
                if (u_in) {
                    q2nu = sq2[lu];
                } else {
                    const int4 cu = a.conn[u];
                    double bu[12], vu, gu[3];
                    geom_B(a.X, cu, bu, vu);
                    grad_from_B(cu, bu, a.phi, gu);
                    q2nu = __ddiv_rn(dot3r(gu[0], gu[1], gu[2], gu[0], gu[1], gu[2]), a.u2);
                }
                q2lu = q2nu < F.q2cap ? q2nu : F.q2cap;
                lim_u = q2lu == q2nu;
                rho_u = (u_in && !BATCH) ? srho[lu] : rho_of(q2lu, F);
            }
            acc.lim += !lim_e;
            // ---- P4: flux, sensitivities, local values
            double nu, rt, s_e = 0.0, s_u = 0.0;
            if (frz) {
                const int br = brf;
                if (a.br_out) a.br_out[user] = (int8_t)br;
                if (br == 3) {
                    nu = 0.0;
                    rt = F.floor_;
                    acc.flo += 1;
                } else if (br == 0) {
                    nu = 0.0;
                    rt = rho_e;
                } else {
                    nu = switch_of(mach2_of(br == 1 ? q2l : q2lu, F), F);
                    rt = rho_e - nu * (rho_e - rho_u);
                }
                if (JAC) frozen_sensitivities(br, q2l, rho_e, q2lu, rho_u, F, s_e, s_u);
            } else {
                const double nu_e = switch_of(mach2_of(q2l, F), F), nu_u = switch_of(mach2_of(q2lu, F), F);
                nu = fmax(nu_e, nu_u);
                rt = rho_e - nu * (rho_e - rho_u);
                if (a.br_out)
                    a.br_out[user] = (int8_t)(u == xe ? (rho_e <= F.floor_ ? 3 : 0)
                                                      : (rt <= F.floor_ ? 3 : (nu == 0.0 ? 0 : (nu_e >= nu_u ? 1 : 2))));
                rt = rt > F.floor_ ? rt : F.floor_;
                acc.flo += (rt == F.floor_);
                if (JAC) live_sensitivities(q2l, rho_e, q2lu, rho_u, u == xe, F, s_e, s_u);
            }
            acc.nu_max = fmax(acc.nu_max, nu);
            acc.sup += (nu > 0.0);
            const double w1 = rt * Ve;
            double b[12];
            {
                const double4 p0 = xs[lc.x], p1 = xs[lc.y], p2 = xs[lc.z], p3 = xs[lc.w];
                double vtmp;
                geom_B_pts(p0.x, p0.y, p0.z, p1.x, p1.y, p1.z, p2.x, p2.y, p2.z, p3.x, p3.y, p3.z, b, vtmp);
            }
            double gB[4];
            gB_of(g, b, gB);
            if (JAC) {
                s_e = s_e * (lim_e ? 1.0 : 0.0);
                s_u = s_u * (lim_u ? 1.0 : 0.0);
                const double w2 = 2.0 * F.inv_u2 * s_e * Ve;
                const double w3 = 2.0 * F.inv_u2 * s_u * Ve;
                const bool active = s_u != 0.0;
                if (active) {
                    double f[4] = {gB[0], gB[1], gB[2], gB[3]};
                    if (u != xe) {
                        double gu[3], bu[12], vu;
                        if (u_in) {
                            const ushort4 lcu = slc[lu];
                            const double4 q0 = xs[lcu.x], q1 = xs[lcu.y], q2 = xs[lcu.z], q3 = xs[lcu.w];
                            geom_B_pts(q0.x, q0.y, q0.z, q1.x, q1.y, q1.z, q2.x, q2.y, q2.z, q3.x, q3.y, q3.z, bu, vu);
                            gu[0] = sgx[lu];
                            gu[1] = sgy[lu];
                            gu[2] = sgz[lu];
                        } else {
                            const int4 cu = a.conn[u];
                            geom_B(a.X, cu, bu, vu);
                            grad_from_B(cu, bu, a.phi, gu);
                        }
                        gB_of(gu, bu, f);
                    }
                    store_t3(a.t3v, user, w3, gB, f);
                    acc.act += 1;
                }
                a.t3flag[user] = active ? 1 : 0;
                store_local_s(sloc, NT, tid, b, gB, w1, w2);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) sloc[(2 * i) * NT + tid] = w1 * gB[i];
            }
            a.up_out[user] = u_in ? sperm[lu] : a.perm[u];
            if (a.rt_out) a.rt_out[user] = rt;
        }
        cp_async_wait<0>();  // this thread's plan blocks are in
        __syncthreads();
        // ---- P5: the tile's outputs, the plan slice from shared memory
        const int32_t* pnoff = reinterpret_cast<const int32_t*>(tsm + L.noff + d_noff);
        const int2* pndst = reinterpret_cast<const int2*>(tsm + L.ndst + d_ndst);
        const uint16_t* pnent = reinterpret_cast<const uint16_t*>(tsm + L.nent + d_nent);
        const int32_t kbase = 4 * e0;
        for (int r = tid; r < nn; r += NT) {
            const int32_t k1 = pnoff[r + 1] - kbase;
            double rs = 0.0, ds = 0.0;
            for (int32_t k = pnoff[r] - kbase; k < k1; ++k) {
                const uint32_t c = pnent[k];
                const int l = c >> 2, i = c & 3;
                rs += sloc[(2 * i) * NT + l];
                if (JAC) ds += sloc[(2 * i + 1) * NT + l];
            }
            const int2 d = pndst[r];
            if (d.x >= 0) {
                a.R[d.x] = rs;
                if (JAC) a.J[d.y] = ds;
            } else {
                const int64_t q = -1 - (int64_t)d.x;
                a.part[q] = rs;
                if (JAC) a.part[q + 1] = ds;
            }
        }
        if (JAC) {
            const int32_t* puoff = reinterpret_cast<const int32_t*>(tsm + L.uoff + d_uoff);
            const int2* pudst = reinterpret_cast<const int2*>(tsm + L.udst + d_udst);
            const uint16_t* puent = reinterpret_cast<const uint16_t*>(tsm + L.uent + d_uent);
            const int32_t cbase = 6 * e0;
            for (int p = tid; p < nu; p += NT) {
                const int32_t k1 = puoff[p + 1] - cbase;
                double v = 0.0;
                for (int32_t k = puoff[p] - cbase; k < k1; ++k) {
                    const uint32_t c = puent[k];
                    v += sloc[(8 + (c & 7)) * NT + (c >> 3)];
                }
                const int2 d = pudst[p];
                if (d.x >= 0) {
                    a.J[d.x] = v;
                    a.J[d.y] = v;
                } else {
                    a.part[-1 - (int64_t)d.x] = v;
                }
            }
        }
        __syncthreads();
    }
    flush(acc, a.mon);
}

// Outputs summed from the tiles' partials, in tile order: residual and
// diagonal of the nodes shared by several tiles (and R = 0 at nodes of no
// element), then the shared upper slots and their transposes.
template <bool JAC>
__global__ void __launch_bounds__(256)
    k_tile_combine(int64_t n_cnode, const int32_t* __restrict__ cn_off, const int32_t* __restrict__ cn_idx,
                   const int2* __restrict__ cn_dst, int64_t n_cedge, const int32_t* __restrict__ ce_off,
                   const int32_t* __restrict__ ce_idx, const int2* __restrict__ ce_dst,
                   const double* __restrict__ part, double* __restrict__ R, double* __restrict__ J) {
    const int64_t n = n_cnode + (JAC ? n_cedge : 0);
    GRID_STRIDE(k, n) {
        if (k < n_cnode) {
            double rs = 0.0, ds = 0.0;
            const int32_t j1 = cn_off[k + 1];
            for (int32_t j = cn_off[k]; j < j1; ++j) {
                const int32_t q = cn_idx[j];
                rs += part[q];
                if (JAC) ds += part[q + 1];
            }
            const int2 d = cn_dst[k];
            R[d.x] = rs;
            if (JAC && d.y >= 0) J[d.y] = ds;
        } else {
            const int64_t kk = k - n_cnode;
            double v = 0.0;
            const int32_t j1 = ce_off[kk + 1];
            for (int32_t j = ce_off[kk]; j < j1; ++j) v += part[ce_idx[j]];
            const int2 d = ce_dst[kk];
            J[d.x] = v;
            J[d.y] = v;
        }
    }
}

// ------------------------------------------------------------ Term 3

// fill_term3_coo (kernels/jacobian.py:184-229) + the merge's duplicate
// sums (:344-358), one warp per row n.  An active element e (t3flag) with
// n = nodes(e)_i adds (n, nodes(u(e))_k, a_i b_k) for k = 0..3, where
// t3v[e] = (a_0..a_3, b_0..b_3).  The row's entries, in (element, k) order
// -- the COO order restricted to the row -- are stably sorted by column;
// each column's run is summed left to right and either added to the P1
// slot (data) or, off the pattern, written to the row's extras scratch at
// 4 ent_off[n] (at most 4 deg(n) columns), with the count in x_cnt[n].
//
// RECORD also writes, for the symbolic cache, every entry's code
// (e << 4 | i << 2 | k) and destination at 4 ent_off[n] + position: the P1
// slot, or -1 - (the extra's rank in its row); unused positions of the
// row's region get INT32_MAX.
//
// row_on: rows with an incident active element (k_t3_mark).  A warp looks at
// 32 of its rows' flags at a time and walks the entries of the flagged ones
// only: with a supersonic pocket nine rows in ten have none (3.6 M tets: 137 us
// when every row's entries were read).
__global__ void k_t3_mark(int64_t E, const uint8_t* __restrict__ flag, const int4* __restrict__ conn,
                          uint8_t* __restrict__ row_on) {
    GRID_STRIDE(e, E) {
        if (!flag[e]) continue;
        const int4 c = conn[e];
        row_on[c.x] = row_on[c.y] = row_on[c.z] = row_on[c.w] = 1;
    }
}

template <int WARPS, bool RECORD>
__global__ void __launch_bounds__(WARPS * 32)
    k_t3_rows(int64_t N, int cap, const int32_t* __restrict__ ent_off, const uint32_t* __restrict__ ent,
              const uint8_t* __restrict__ row_on, const uint8_t* __restrict__ flag, const int32_t* __restrict__ up,
              const int4* __restrict__ conn, const double* __restrict__ t3v, const int32_t* __restrict__ indptr,
              const int32_t* __restrict__ indices, double* __restrict__ data, int32_t* __restrict__ xs_col,
              double* __restrict__ xs_val, int32_t* __restrict__ x_cnt, uint32_t* __restrict__ rec_code,
              int32_t* __restrict__ rec_key) {
    extern __shared__ __align__(16) unsigned char t3_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t* col0 = reinterpret_cast<int32_t*>(t3_smem) + (size_t)w * cap;
    int32_t* col1 = reinterpret_cast<int32_t*>(t3_smem) + (size_t)(WARPS + w) * cap;
    double* val0 = reinterpret_cast<double*>(t3_smem + (size_t)2 * WARPS * cap * sizeof(int32_t)) + (size_t)w * cap;
    double* val1 = reinterpret_cast<double*>(t3_smem + (size_t)2 * WARPS * cap * sizeof(int32_t)) +
                   (size_t)(WARPS + w) * cap;
    // RECORD: each entry's distinct-column index and each distinct
    // column's destination
    unsigned char* rec_base = t3_smem + (size_t)2 * WARPS * cap * (sizeof(int32_t) + sizeof(double));
    int16_t* eidx = reinterpret_cast<int16_t*>(rec_base) + (size_t)w * cap;
    int32_t* dd = reinterpret_cast<int32_t*>(rec_base + (size_t)WARPS * cap * sizeof(int16_t)) + (size_t)w * cap;
    const unsigned lt = (1u << lane) - 1u;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t first = warp; first < N; first += 32 * n_warps) {   // warp-uniform
        const int64_t mine = first + lane * n_warps;
        const bool on = mine < N && row_on[mine];
        if (!RECORD && mine < N && !on) x_cnt[mine] = 0;
        unsigned todo = __ballot_sync(0xffffffffu, RECORD ? mine < N : on);
        for (; todo; todo &= todo - 1) {
            const int64_t n = first + (__ffs(todo) - 1) * n_warps;
            const int32_t eb = ent_off[n], deg = ent_off[n + 1] - eb;
            // 1. the row's entries in (element, k) order
            int P = 0;
            for (int base = 0; base < deg; base += 32) {
                const int j = base + lane;
                uint32_t x = 0;
                bool act = false;
                if (j < deg) {
                    x = ent[eb + j];
                    act = flag[x >> 2] != 0;
                }
                const unsigned m = __ballot_sync(0xffffffffu, act);
                if (act) {
                    const int64_t e = x >> 2;
                    const int i = x & 3;
                    const int4 cu = conn[up[e]];
                    const double* t = t3v + 8 * e;
                    const double ai = t[i];
                    const int pos = P + 4 * __popc(m & lt);
                    if (RECORD) {
                        uint32_t* rc = rec_code + 4 * (int64_t)eb + pos;
#pragma unroll
                        for (int k = 0; k < 4; ++k) rc[k] = ((uint32_t)e << 4) | (uint32_t)(i << 2) | (uint32_t)k;
                    }
                    col0[pos] = cu.x;
                    col0[pos + 1] = cu.y;
                    col0[pos + 2] = cu.z;
                    col0[pos + 3] = cu.w;
                    val0[pos] = ai * t[4];
                    val0[pos + 1] = ai * t[5];
                    val0[pos + 2] = ai * t[6];
                    val0[pos + 3] = ai * t[7];
                }
                P += 4 * __popc(m);
            }
            if (P == 0) {
                if (lane == 0) x_cnt[n] = 0;
                if (RECORD)
                    for (int p = lane; p < 4 * deg; p += 32) rec_key[4 * (int64_t)eb + p] = INT32_MAX;
                continue;
            }
            __syncwarp();
            // 2. the distinct columns in order of first appearance, each with the
            //    sequential sum of its entries in (element, k) order: chunks of 32
            //    entries, equal columns grouped by match_any, the group's lowest
            //    lane adding the group's values in lane (= entry) order to the
            //    column's running sum -- the reference's duplicate summation order
            int D = 0;
            for (int base = 0; base < P; base += 32) {
                const int p = base + lane;
                const bool valid = p < P;
                const int32_t c = valid ? col0[p] : -1 - lane;  // idle lanes: distinct dummies
                const unsigned grp = __match_any_sync(0xffffffffu, c);
                const bool leader = valid && (__ffs(grp) - 1) == lane;
                int idx = -1;
                if (leader)
                    for (int d = 0; d < D; ++d)
                        if (col1[d] == c) {
                            idx = d;
                            break;
                        }
                const unsigned newm = __ballot_sync(0xffffffffu, leader && idx < 0);
                if (leader) {
                    double acc_c = 0.0;
                    if (idx < 0) idx = D + __popc(newm & lt);
                    else acc_c = val1[idx];
                    unsigned gm = grp;
                    while (gm) {
                        const int j = __ffs(gm) - 1;
                        gm &= gm - 1;
                        acc_c += val0[base + j];
                        if (RECORD) eidx[base + j] = (int16_t)idx;
                    }
                    col1[idx] = c;
                    val1[idx] = acc_c;
                }
                D += __popc(newm);
                __syncwarp();
            }
            // 3. per distinct column: into the P1 slot, else an extra; extras are
            //    written in column order (rank among the row's extra columns)
            const int32_t rb = indptr[n], L = indptr[n + 1] - rb;
            for (int d = lane; d < D; d += 32) {
                const int32_t c = col1[d];
                int32_t lo = 0, hi = L;
                while (lo < hi) {
                    const int32_t mid = (lo + hi) >> 1;
                    if (indices[rb + mid] < c) lo = mid + 1;
                    else hi = mid;
                }
                const bool in_pattern = lo < L && indices[rb + lo] == c;
                if (in_pattern) data[rb + lo] += val1[d];
                if (RECORD && in_pattern) dd[d] = rb + lo;
                col0[d] = in_pattern ? INT32_MAX : c;  // extra columns, for the ranks
            }
            __syncwarp();
            int X = 0;
            for (int base = 0; base < D; base += 32) {
                const int d = base + lane;
                const bool extra = d < D && col0[d] != INT32_MAX;
                if (extra) {
                    const int32_t c = col0[d];
                    int r = 0;
                    for (int q = 0; q < D; ++q) r += col0[q] < c;
                    const int64_t o = 4 * (int64_t)eb + r;
                    xs_col[o] = c;
                    xs_val[o] = val1[d];
                    if (RECORD) dd[d] = -1 - r;
                }
                X += __popc(__ballot_sync(0xffffffffu, extra));
            }
            if (lane == 0) x_cnt[n] = X;
            __syncwarp();
            if (RECORD) {
                for (int p = lane; p < 4 * deg; p += 32) rec_key[4 * (int64_t)eb + p] = p < P ? dd[eidx[p]] : INT32_MAX;
                __syncwarp();
            }
        }
    }
}

// Extras of every row, compacted in (row, column) order: a warp looks at the
// counts of 32 of its rows at a time and copies the non-empty ones, coalesced.
__global__ void k_t3_compact(int64_t N, const int32_t* __restrict__ ent_off, const int32_t* __restrict__ x_ptr,
                             const int32_t* __restrict__ xs_col, const double* __restrict__ xs_val,
                             int32_t* __restrict__ x_row, int32_t* __restrict__ x_col, double* __restrict__ x_val) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t first = warp; first < N; first += 32 * n_warps) {   // warp-uniform
        const int64_t mine = first + lane * n_warps;
        int32_t o = 0, cnt = 0, eo = 0;
        if (mine < N) {
            o = x_ptr[mine];
            cnt = x_ptr[mine + 1] - o;
            if (cnt) eo = ent_off[mine];
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, cnt > 0); todo; todo &= todo - 1) {
            const int src_lane = __ffs(todo) - 1;
            const int64_t n = first + src_lane * n_warps;
            const int32_t on = __shfl_sync(0xffffffffu, o, src_lane), cn = __shfl_sync(0xffffffffu, cnt, src_lane);
            const int64_t src = 4 * (int64_t)__shfl_sync(0xffffffffu, eo, src_lane);
            for (int32_t j = lane; j < cn; j += 32) {
                x_row[on + j] = (int32_t)n;
                x_col[on + j] = xs_col[src + j];
                x_val[on + j] = xs_val[src + j];
            }
        }
    }
}

// Symbolic cache of Term 3: extras' destinations made global (Z + the
// extra's compacted position), then -- per destination, contributors in the
// order the row kernel sums them -- the values-only rebuild.
__global__ void k_t3_rec_fix(int64_t N, const int32_t* __restrict__ ent_off, const int32_t* __restrict__ x_ptr,
                             int64_t Z, int32_t* __restrict__ rec_key) {
    GRID_STRIDE(n, N) {
        const int64_t b = 4 * (int64_t)ent_off[n], e = 4 * (int64_t)ent_off[n + 1];
        for (int64_t p = b; p < e; ++p) {
            const int32_t k = rec_key[p];
            if (k < 0) rec_key[p] = (int32_t)(Z + x_ptr[n] + (-1 - k));
        }
    }
}

__global__ void k_t3_values(int64_t n_seg, const int32_t* __restrict__ seg, const int32_t* __restrict__ key,
                            const uint32_t* __restrict__ code, const double* __restrict__ t3v, int64_t Z,
                            double* __restrict__ data, double* __restrict__ x_val) {
    GRID_STRIDE(d, n_seg) {
        double v = 0.0;
        const int32_t j1 = seg[d + 1];
        for (int32_t j = seg[d]; j < j1; ++j) {
            const uint32_t c = code[j];
            const double* t = t3v + 8 * (int64_t)(c >> 4);
            // the row kernel rounds each product, then adds: no contraction
            v = __dadd_rn(v, __dmul_rn(t[(c >> 2) & 3], t[4 + (c & 3)]));
        }
        const int32_t k = key[d];
        if (k < Z) data[k] += v;
        else x_val[k - Z] = v;
    }
}

// Elements whose Term-3 activity or (active) upstream differ from the
// recorded signature.
__global__ void k_t3_sig_diff(int64_t E, const uint8_t* __restrict__ flag, const int32_t* __restrict__ up,
                              const uint8_t* __restrict__ cflag, const int32_t* __restrict__ cup,
                              unsigned long long* out) {
    unsigned long long c = 0;
    GRID_STRIDE(e, E) c += (flag[e] != cflag[e]) || (flag[e] && up[e] != cup[e]);
    c = warp_sum_u64(c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

__global__ void k_count_nonzero(const double* __restrict__ v, int64_t n, unsigned long long* out) {
    unsigned long long c = 0;
    GRID_STRIDE(i, n) c += (v[i] != 0.0);
    c = warp_sum_u64(c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// Merged row lengths / fill of (P1 data + extras), optionally dropping
// exact zeros (scipy's CSR addition does, kernels/jacobian.py:355-357).
// Eight lanes per row, eight entries at a time: an entry's place is the kept
// entries of its own list before it (a ballot) plus the kept entries of the
// other list in lower columns (eight shuffles per chunk; dropped entries
// stand as column INT32_MAX).  Entries past `capacity` are not written.  One thread per row, merging serially, took
// 187 us for the fill on the 625 k-row Jacobian.
template <bool FILL>
__global__ void __launch_bounds__(256)
    k_merge_rows(int64_t N, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                 const double* __restrict__ data, const int32_t* __restrict__ xptr, const int32_t* __restrict__ xcol,
                 const double* __restrict__ xval, bool drop_zeros, int32_t* __restrict__ out_ptr,
                 int32_t* __restrict__ out_idx, double* __restrict__ out_val, int64_t capacity) {
    constexpr int G = 8, RPW = 32 / G;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), shift = lane & ~(G - 1);
    const unsigned below = (1u << sub) - 1u;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = warp * RPW; base < N; base += n_warps * RPW) {   // warp-uniform
        const int64_t n = base + lane / G;
        int32_t a = 0, la = 0, b = 0, lb = 0;
        if (n < N) {
            a = indptr[n];
            la = indptr[n + 1] - a;
            if (xptr) {
                b = xptr[n];
                lb = xptr[n + 1] - b;
            }
        }
        const int la_max = __reduce_max_sync(0xffffffffu, la), lb_max = __reduce_max_sync(0xffffffffu, lb);
        // entry k0 + sub of a list: its column, INT32_MAX when past the end or dropped
        auto entry = [&](const int32_t* col, const double* val, int32_t o, int32_t len, int k, double& v) {
            if (k >= len) return INT32_MAX;
            v = val[o + k];
            if (drop_zeros && v == 0.0) return INT32_MAX;
            return FILL ? col[o + k] : 0;
        };
        // the kept entries of the other list in columns below c
        auto lower = [&](const int32_t* col, const double* val, int32_t o, int32_t len, int most, int32_t c) {
            int cnt = 0;
            for (int k0 = 0; k0 < most; k0 += G) {
                double v;
                const int32_t x = entry(col, val, o, len, k0 + sub, v);
#pragma unroll
                for (int j = 0; j < G; ++j) cnt += __shfl_sync(0xffffffffu, x, j, G) < c;
            }
            return cnt;
        };
        int kept = 0;
        const int32_t out = FILL && n < N ? out_ptr[n] : 0;
        auto list = [&](const int32_t* col, const double* val, int32_t o, int32_t len, int most, const int32_t* col2,
                        const double* val2, int32_t o2, int32_t len2, int most2) {
            int before = 0;
            for (int k0 = 0; k0 < most; k0 += G) {
                double v = 0.0;
                const int32_t c = entry(col, val, o, len, k0 + sub, v);
                const bool keep = c != INT32_MAX;
                const unsigned m = (__ballot_sync(0xffffffffu, keep) >> shift) & ((1u << G) - 1u);
                if (FILL) {
                    int place = before + __popc(m & below);
                    if (most2 > 0) place += lower(col2, val2, o2, len2, most2, c);
                    if (keep && out + place < capacity) {
                        out_idx[out + place] = c;
                        out_val[out + place] = v;
                    }
                }
                before += __popc(m);
            }
            kept += before;
        };
        list(indices, data, a, la, la_max, xcol, xval, b, lb, lb_max);
        list(xcol, xval, b, lb, lb_max, indices, data, a, la, la_max);
        if (!FILL && n < N && sub == 0) out_ptr[n] = kept;
    }
}

__global__ void k_set_i64(int64_t* __restrict__ dst, int64_t v) { *dst = v; }

template <class T>
void scan(up3d_mesh* m, const T* in, T* out, int64_t n, cudaStream_t s) {
    size_t bytes = 0;
    UP3D_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, n, s));
    m->cub_tmp.alloc(bytes);
    UP3D_CUDA(cub::DeviceScan::ExclusiveSum(m->cub_tmp.get(), bytes, in, out, n, s));
}

}  // namespace

// ------------------------------------------------------------ launchers

// Jacobian (+ residual) rows from m->loc, m->tune.row_lanes lanes per row,
// from the fixed-width contributor records when the mesh has them and the
// tuning asks for them (row_plan8).
template <int LPR, bool P8>
static void launch_row_gather_lpr(const up3d_mesh* m, double* R, double* J, cudaStream_t s) {
    constexpr int rows_per_block = RG_WARPS * 32 / LPR;
    const unsigned grid = grid_for(m->N, rows_per_block, (int64_t)m->n_sms * 64);
    k_row_gather<RG_WARPS, LPR, P8><<<grid, RG_WARPS * 32, 0, s>>>(
        m->N, m->ent_off.get(), m->ent.get(), m->indptr.get(), m->plan_off.get(), m->plan.get(), m->diag.get(),
        m->zt.get(), m->up_off.get(), m->plan8.get(), m->loc.get(), R, J);
    UP3D_CHECK_LAUNCH();
}
template <bool P8>
static void launch_row_gather_p(const up3d_mesh* m, double* R, double* J, cudaStream_t s) {
    switch (m->tune.row_lanes) {
        case 4: launch_row_gather_lpr<4, P8>(m, R, J, s); break;
        case 16: launch_row_gather_lpr<16, P8>(m, R, J, s); break;
        case 32: launch_row_gather_lpr<32, P8>(m, R, J, s); break;
        default: launch_row_gather_lpr<8, P8>(m, R, J, s); break;
    }
}
void launch_row_gather(const up3d_mesh* m, double* R, double* J, cudaStream_t s) {
    if (m->has_plan8 && m->tune.row_plan8) launch_row_gather_p<true>(m, R, J, s);
    else launch_row_gather_p<false>(m, R, J, s);
}

// Residual rows from m->res.
void launch_row_residual(const up3d_mesh* m, double* R, cudaStream_t s) {
    k_row_residual<<<grid_for(8 * m->N, 256, (int64_t)m->n_sms * 64), 256, 0, s>>>(m->N, m->ent_off.get(),
                                                                             m->ent.get(), m->res.get(), R);
    UP3D_CHECK_LAUNCH();
}

// Builds Term 3 from the active flags and vectors: folds the in-pattern
// part into `data`, keeps the extras (sorted by row, col) in the mesh
// workspace, and returns (n_active, n_extra).  Synchronises the stream.
// `known_active` is the active count, known to the caller (0 skips
// everything).
constexpr int T3_WARPS = 4;
static void build_term3(up3d_mesh* m, double* data, cudaStream_t s, int64_t& n_active, int64_t& n_extra,
                        int64_t known_active, const int32_t* upstream = nullptr) {
    if (!upstream) upstream = m->up32.get();
    const int64_t E = m->E, N = m->N, Z = m->nnz;
    n_extra = 0;
    m->last_extra = 0;
    m->jac_serial += 1;
    m->i64_ws.alloc(8);
    n_active = known_active;
    m->last_active = n_active;
    if (n_active == 0) return;
    // the symbolic cache: is the pattern the recorded one?
    const bool cacheable = E < (1ll << 28) && Z + 16 * E < INT32_MAX;
    bool same = false;
    if (cacheable && m->t3c_state >= 1 && m->t3c_active == n_active) {
        unsigned long long* c = reinterpret_cast<unsigned long long*>(m->i64_ws.get() + 3);
        UP3D_CUDA(cudaMemsetAsync(c, 0, sizeof(unsigned long long), s));
        k_t3_sig_diff<<<grid_for(E, 256), 256, 0, s>>>(E, m->t3_flag.get(), upstream, m->t3c_flag.get(),
                                                      m->t3c_up.get(), c);
        UP3D_CHECK_LAUNCH();
        same = read_back(c, s) == 0;
    }
    if (same && m->t3c_state == 2) {
        // values only: the P1 slots and extras of the recorded pattern
        if (m->t3c_nseg > 0) {
            k_t3_values<<<grid_for(m->t3c_nseg, 256, (int64_t)m->n_sms * 16), 256, 0, s>>>(
                m->t3c_nseg, m->t3c_seg.get(), m->t3c_key.get(), m->t3c_code.get(), m->t3v.get(), Z, data,
                m->x_val_c.get());
            UP3D_CHECK_LAUNCH();
        }
        n_extra = m->t3c_extra;
        m->last_extra = n_extra;
        m->t3c_hits += 1;
        return;
    }
    // a pattern seen twice in a row is recorded for the calls that follow
    const bool record = cacheable && same;
    const int cap = 4 * std::max<int32_t>(m->max_deg, 1);
    const size_t smem = (size_t)T3_WARPS * cap * 2 * (sizeof(int32_t) + sizeof(double)) +
                        (size_t)T3_WARPS * cap * (sizeof(int16_t) + sizeof(int32_t));
    UP3D_REQUIRE(smem <= 227 * 1024, UP3D_ERR_VALUE, "Term 3: node degree too large for the row kernel");
    auto kern = record ? k_t3_rows<T3_WARPS, true> : k_t3_rows<T3_WARPS, false>;
    if (smem > 48 * 1024) UP3D_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    m->x_col.alloc(16 * E);
    m->x_val.alloc(16 * E);
    m->extra_cnt.alloc(N + 1);
    m->x_ptr.alloc(N + 1);
    if (record) {
        m->t3c_code_tmp.alloc(16 * E);
        m->t3c_key_tmp.alloc(16 * E);
    }
    m->t3_row_on.alloc(N);
    UP3D_CUDA(cudaMemsetAsync(m->t3_row_on.get(), 0, N, s));
    k_t3_mark<<<grid_for(E, 256), 256, 0, s>>>(E, m->t3_flag.get(), m->conn.get(), m->t3_row_on.get());
    UP3D_CHECK_LAUNCH();
    UP3D_CUDA(cudaMemsetAsync(m->extra_cnt.get() + N, 0, sizeof(int32_t), s));
    kern<<<grid_for(32 * N, T3_WARPS * 32, (int64_t)148 * 32), T3_WARPS * 32, smem, s>>>(
        N, cap, m->ent_off.get(), m->ent.get(), m->t3_row_on.get(), m->t3_flag.get(), upstream, m->conn.get(),
        m->t3v.get(),
        m->indptr.get(), m->indices.get(), data, m->x_col.get(), m->x_val.get(), m->extra_cnt.get(),
        record ? m->t3c_code_tmp.get() : nullptr, record ? m->t3c_key_tmp.get() : nullptr);
    UP3D_CHECK_LAUNCH();
    scan(m, m->extra_cnt.get(), m->x_ptr.get(), N + 1, s);
    n_extra = read_back(m->x_ptr.get() + N, s);
    m->last_extra = n_extra;
    if (n_extra > 0) {
        m->x_row_c.alloc(n_extra);
        m->x_col_c.alloc(n_extra);
        m->x_val_c.alloc(n_extra);
        k_t3_compact<<<grid_for(32 * N, 256, (int64_t)m->n_sms * 32), 256, 0, s>>>(N, m->ent_off.get(), m->x_ptr.get(), m->x_col.get(),
                                                      m->x_val.get(), m->x_row_c.get(), m->x_col_c.get(),
                                                      m->x_val_c.get());
        UP3D_CHECK_LAUNCH();
    }
    if (!cacheable) return;
    if (record) {
        // destinations made global, a stable sort by destination (row-major
        // entry order kept within each), then the runs
        k_t3_rec_fix<<<grid_for(N, 256), 256, 0, s>>>(N, m->ent_off.get(), m->x_ptr.get(), Z, m->t3c_key_tmp.get());
        UP3D_CHECK_LAUNCH();
        const int64_t n_items = 16 * E;
        m->t3c_code.alloc(n_items);
        m->t3c_key.alloc(n_items);
        size_t bytes = 0;
        UP3D_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, m->t3c_key_tmp.get(), m->t3c_key.get(),
                                                  m->t3c_code_tmp.get(), m->t3c_code.get(), n_items, 0, 31, s));
        m->cub_tmp.alloc(bytes);
        UP3D_CUDA(cub::DeviceRadixSort::SortPairs(m->cub_tmp.get(), bytes, m->t3c_key_tmp.get(), m->t3c_key.get(),
                                                  m->t3c_code_tmp.get(), m->t3c_code.get(), n_items, 0, 31, s));
        // the valid entries (16 per active element) sort before the INT32_MAX fill
        const int64_t n_valid = 16 * n_active;
        m->t3c_cnt.alloc(n_valid + 1);
        m->t3c_seg.alloc(n_valid + 1);
        m->t3c_nruns.alloc(1);
        // unique keys over the sorted prefix, written over the front of the
        // tmp key array
        bytes = 0;
        UP3D_CUDA(cub::DeviceRunLengthEncode::Encode(nullptr, bytes, m->t3c_key.get(), m->t3c_key_tmp.get(),
                                                     m->t3c_cnt.get(), m->t3c_nruns.get(), n_valid, s));
        m->cub_tmp.alloc(bytes);
        UP3D_CUDA(cub::DeviceRunLengthEncode::Encode(m->cub_tmp.get(), bytes, m->t3c_key.get(), m->t3c_key_tmp.get(),
                                                     m->t3c_cnt.get(), m->t3c_nruns.get(), n_valid, s));
        const int64_t nruns = read_back(m->t3c_nruns.get(), s);
        UP3D_CUDA(cudaMemsetAsync(m->t3c_cnt.get() + nruns, 0, sizeof(int32_t), s));
        scan(m, m->t3c_cnt.get(), m->t3c_seg.get(), nruns + 1, s);
        // keep the run keys (destinations) where the values kernel reads them
        UP3D_CUDA(cudaMemcpyAsync(m->t3c_key.get(), m->t3c_key_tmp.get(), sizeof(int32_t) * nruns,
                                  cudaMemcpyDeviceToDevice, s));
        UP3D_CUDA(cudaStreamSynchronize(s));
        m->t3c_nseg = nruns;
        m->t3c_state = 2;
    } else {
        m->t3c_flag.alloc(E);
        m->t3c_up.alloc(E);
        UP3D_CUDA(cudaMemcpyAsync(m->t3c_flag.get(), m->t3_flag.get(), E, cudaMemcpyDeviceToDevice, s));
        UP3D_CUDA(cudaMemcpyAsync(m->t3c_up.get(), upstream, sizeof(int32_t) * E, cudaMemcpyDeviceToDevice, s));
        m->t3c_state = 1;
    }
    m->t3c_active = n_active;
    m->t3c_extra = n_extra;
}

// The merged CSR of the last Jacobian; at most `capacity` entries of indices
// and merged are written.
static void export_merged(up3d_mesh* m, const double* data, int32_t* indptr, int32_t* indices, double* merged,
                          int64_t capacity, cudaStream_t s) {
    UP3D_REQUIRE(m && data && indptr && indices && merged, UP3D_ERR_ARGUMENT,
                 "up3d_jacobian_export: null argument");
    const bool has_x = m->last_extra > 0;
    const int32_t* xptr = has_x ? m->x_ptr.get() : nullptr;
    m->extra_cnt.alloc(m->N + 1);
    int32_t* cnt = m->extra_cnt.get();
    UP3D_CUDA(cudaMemsetAsync(cnt + m->N, 0, sizeof(int32_t), s));
    const unsigned grid = grid_for(m->N, 32, (int64_t)m->n_sms * 64);
    k_merge_rows<false><<<grid, 256, 0, s>>>(m->N, m->indptr.get(), m->indices.get(), data, xptr,
                                                           m->x_col_c.get(), m->x_val_c.get(),
                                                           m->last_drop_zeros, cnt, nullptr, nullptr, 0);
    UP3D_CHECK_LAUNCH();
    scan(m, cnt, indptr, m->N + 1, s);
    k_merge_rows<true><<<grid, 256, 0, s>>>(m->N, m->indptr.get(), m->indices.get(), data, xptr,
                                                          m->x_col_c.get(), m->x_val_c.get(),
                                                          m->last_drop_zeros, indptr, indices, merged, capacity);
    UP3D_CHECK_LAUNCH();
}

static int64_t merged_nnz(up3d_mesh* m, const double* data, cudaStream_t s) {
    if (m->last_active == 0) return m->nnz;
    m->i64_ws.alloc(8);
    unsigned long long* c = reinterpret_cast<unsigned long long*>(m->i64_ws.get() + 2);
    UP3D_CUDA(cudaMemsetAsync(c, 0, sizeof(unsigned long long), s));
    k_count_nonzero<<<grid_for(m->nnz, 256), 256, 0, s>>>(data, m->nnz, c);
    UP3D_CHECK_LAUNCH();
    if (m->last_extra > 0) {
        k_count_nonzero<<<grid_for(m->last_extra, 256), 256, 0, s>>>(m->x_val_c.get(), m->last_extra, c);
        UP3D_CHECK_LAUNCH();
    }
    return (int64_t)read_back(c, s);
}

}  // namespace up3d

using namespace up3d;

extern "C" {

int up3d_residual(up3d_mesh* m, const double* phi, const double* rt, double* R, double* grad_out, double* q2_out,
                  up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && phi && R, UP3D_ERR_ARGUMENT, "up3d_residual: null argument");
        cudaStream_t s = S(stream);
        if (!grad_out) {
            m->grad_ws.alloc(3 * m->E);
            grad_out = m->grad_ws.get();
        }
        if (!q2_out) {
            m->q2_ws.alloc(m->E);
            q2_out = m->q2_ws.get();
        }
        k_prep_residual<<<grid_for(m->E, 256), 256, 0, s>>>(m->conn.get(), m->B.get(), m->V.get(), phi, rt, m->E,
                                                           grad_out, q2_out, m->res.get());
        UP3D_CHECK_LAUNCH();
        launch_row_residual(m, R, s);
    });
}

int up3d_picard_matrix(up3d_mesh* m, const double* rt, double* data, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && data, UP3D_ERR_ARGUMENT, "up3d_picard_matrix: null argument");
        cudaStream_t s = S(stream);
        k_prep_matrix<<<grid_for(m->E, 256), 256, 0, s>>>(m->B.get(), m->V.get(), rt, m->E, m->loc.get());
        UP3D_CHECK_LAUNCH();
        launch_row_gather(m, nullptr, data, s);
    });
}

int up3d_picard_matrix_data(up3d_mesh* m, const double* rt, double* data, up3d_stream stream) {
    return up3d_picard_matrix(m, rt, data, stream);
}

int up3d_jacobian(up3d_mesh* m, const double* phi, const double* rt, const double* se, const double* su,
                  const int64_t* upstream, double u_inf, const uint8_t* lim, double* data, int64_t* n_active,
                  int64_t* n_extra, int64_t* newton_nnz, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && phi && rt && se && su && upstream && data, UP3D_ERR_ARGUMENT,
                     "up3d_jacobian: null argument");
        cudaStream_t s = S(stream);
        const double inv_u2 = 1.0 / (u_inf * u_inf);
        m->i64_ws.alloc(8);
        unsigned long long* count = reinterpret_cast<unsigned long long*>(m->i64_ws.get());
        UP3D_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned long long), s));
        k_prep_jacobian<<<grid_for(m->E, 256), 256, 0, s>>>(m->conn.get(), m->B.get(), m->V.get(), phi, rt, se, su,
                                                           upstream, lim, inv_u2, m->E, m->loc.get(), m->t3v.get(),
                                                           m->t3_flag.get(), m->up32.get(), count);
        UP3D_CHECK_LAUNCH();
        launch_row_gather(m, nullptr, data, s);
        int64_t na = 0, nx = 0;
        build_term3(m, data, s, na, nx, read_back(reinterpret_cast<const int64_t*>(count), s));
        m->last_drop_zeros = na > 0;
        if (n_active) *n_active = na;
        if (n_extra) *n_extra = nx;
        if (newton_nnz) *newton_nnz = merged_nnz(m, data, s);
    });
}

int up3d_jacobian_data(up3d_mesh* m, const double* phi, const double* rt, const double* se, const double* su,
                       const int64_t* upstream, double u_inf, const uint8_t* lim, double* data, int64_t* n_active,
                       int64_t* n_extra, int64_t* newton_nnz, up3d_stream stream) {
    return up3d_jacobian(m, phi, rt, se, su, upstream, u_inf, lim, data, n_active, n_extra, newton_nnz, stream);
}

int up3d_jacobian_export(up3d_mesh* m, const double* data, int32_t* indptr, int32_t* indices, double* merged,
                         up3d_stream stream) {
    return guarded([&] { export_merged(m, data, indptr, indices, merged, INT64_MAX, S(stream)); });
}

int up3d_jacobian_merge(up3d_mesh* m, const double* data, int32_t* indptr, int32_t* indices, double* merged,
                        int64_t capacity, int64_t serial, int64_t* newton_nnz, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && newton_nnz, UP3D_ERR_ARGUMENT, "up3d_jacobian_merge: null argument");
        UP3D_REQUIRE(serial < 0 || serial == m->jac_serial, UP3D_ERR_RUNTIME,
                     "up3d_jacobian_merge: another Jacobian was formed on the mesh since; evaluate again");
        export_merged(m, data, indptr, indices, merged, capacity, S(stream));
        *newton_nnz = read_back(indptr + m->N, S(stream));
        UP3D_REQUIRE(*newton_nnz <= capacity, UP3D_ERR_VALUE,
                     "up3d_jacobian_merge: the merged matrix has more entries than the arrays hold");
    });
}

int up3d_jacobian_serial(const up3d_mesh* m, const int64_t** serial) {
    return guarded([&] {
        UP3D_REQUIRE(m && serial, UP3D_ERR_ARGUMENT, "up3d_jacobian_serial: null argument");
        *serial = &m->jac_serial;
    });
}

int up3d_jacobian_nnz(up3d_mesh* m, const double* data, int64_t* newton_nnz, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && data && newton_nnz, UP3D_ERR_ARGUMENT, "up3d_jacobian_nnz: null argument");
        *newton_nnz = merged_nnz(m, data, S(stream));
    });
}

}  // extern "C"

namespace up3d {
namespace {

__global__ void k_check_cases(const int32_t* __restrict__ case_of, int64_t E, int n_cases, int* __restrict__ bad) {
    GRID_STRIDE(e, E) if (case_of[e] < 0 || case_of[e] >= n_cases) *bad = 1;
}

}  // namespace

// One launch of the fused element sweep in the mesh's tuned shape: one
// thread per element (grid capped at 64 blocks per SM) or one resident
// wave (SMs x the kernel's occupancy) looping over block-sized tiles; the
// Jacobian sweep compiled for 512 (256 x 2), 640 (128 x 5) or 768 (128 x 6)
// resident threads per SM.
template <bool FR, bool JA, bool BA, bool AIR, int NT, int MB, class... A>
static void launch_sweep_mb(const up3d_mesh* m, cudaStream_t s, A... args) {
    auto kern = k_fused_elem<FR, JA, BA, AIR, NT, MB>;
    unsigned grid;
    if (m->tune.elem_persistent) {
        static int occ = 0;  // same for every device of the process (one architecture)
        if (occ == 0) {
            int nb = 0;
            UP3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, NT, 0));
            occ = nb > 0 ? nb : 1;
        }
        grid = grid_for(m->E, NT, (int64_t)m->n_sms * occ);
    } else {
        grid = grid_for(m->E, NT, (int64_t)m->n_sms * 64 * (256 / NT));
    }
    kern<<<grid, NT, 0, s>>>(args...);
    UP3D_CHECK_LAUNCH();
}

constexpr int64_t SWEEP_LARGE = 2'000'000;
template <bool FR, bool JA, bool BA, bool AIR, class... A>
static void launch_sweep_air(const up3d_mesh* m, cudaStream_t s, A... args) {
    // residual only: on a large mesh of air 28 warps per SM are fastest (72
    // registers, no spill); on one of a few waves of blocks 24 warps, and then
    // the form for any gas (the whole call, walk / frozen: 3.6 M tets 269 / 187
    // against 272 / 193 us, 0.97 M 86.1 / 57.6 and 84.7 / 57.9, 0.45 M 45.2 /
    // 29.6 against 43.2 / 28.6)
    if constexpr (!JA) {
        if constexpr (AIR)
            if (m->E >= SWEEP_LARGE) return launch_sweep_mb<FR, JA, BA, AIR, 128, 7>(m, s, args...);
        launch_sweep_mb<FR, JA, BA, false, 256, 3>(m, s, args...);
    } else {
        switch (m->tune.elem_threads_per_sm) {
            case 640: launch_sweep_mb<FR, JA, BA, AIR, 128, 5>(m, s, args...); break;
            case 768: launch_sweep_mb<FR, JA, BA, AIR, 128, 6>(m, s, args...); break;
            default: launch_sweep_mb<FR, JA, BA, AIR, 256, 2>(m, s, args...); break;
        }
    }
}

template <bool FR, bool JA, bool BA, class... A>
static void launch_sweep(const up3d_mesh* m, bool air, cudaStream_t s, A... args) {
    if (air) launch_sweep_air<FR, JA, BA, true>(m, s, args...);
    else launch_sweep_air<FR, JA, BA, false>(m, s, args...);
}

// One launch of the tiled evaluation over every tile (a persistent grid of
// SMs x occupancy CTAs).
template <bool FR, bool JA, bool BA, int NT, int MB>
static void launch_tiles_nt(const up3d_mesh* m, const TileArgs& ta, cudaStream_t s) {
    auto kern = k_tile_eval<FR, JA, BA, NT, MB>;
    const TilePlan& P = *m->tiles;
    const size_t smem = TileSmem(P.max_nodes, P.max_edges, NT).total;
    UP3D_REQUIRE(smem <= 227 * 1024, UP3D_ERR_VALUE, "tiled assembly: a tile's shared memory exceeds 227 KB");
    if (smem > 48 * 1024)  // per device: set on every launch that needs it
        UP3D_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int occ = 0;
    UP3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, NT, smem));
    UP3D_REQUIRE(occ > 0, UP3D_ERR_RUNTIME, "tiled assembly: the tile kernel cannot be resident");
    const int64_t grid = std::min<int64_t>(P.n_tiles, (int64_t)m->n_sms * occ);
    kern<<<(unsigned)std::max<int64_t>(grid, 1), NT, smem, s>>>(ta);
    UP3D_CHECK_LAUNCH();
}

template <bool FR, bool JA, bool BA>
static void launch_tiles(const up3d_mesh* m, const TileArgs& ta, cudaStream_t s) {
    if (m->tiles->T == 128) launch_tiles_nt<FR, JA, BA, 128, 4>(m, ta, s);
    else launch_tiles_nt<FR, JA, BA, 256, 2>(m, ta, s);
}

// The tiled evaluation: the tile kernel, then the combine pass.
static void tiled_evaluate(up3d_mesh* m, const double* phi, const Flow& F, double u2, const Flow* flows_d,
                           const int32_t* case_of, int n_cases, const int64_t* up_fz, const int8_t* br_fz,
                           double* R, double* data, double* rt_out, int32_t* up_dst, up3d_monitors* mo,
                           int8_t* br_out, cudaStream_t s) {
    ensure_tiles(m, m->tune.tile_elems, m->tune.tile_stretch, s);
    const TilePlan& P = *m->tiles;
    TileArgs ta;
    ta.conn = P.conn.get();
    ta.fnbr = P.fnbr.get();
    ta.cen = P.cen.get();
    ta.disp = P.disp.get();
    ta.X = m->nodes4.get();
    ta.phi = phi;
    ta.perm = P.perm.get();
    ta.iperm = P.iperm.get();
    ta.eoff = P.eoff.get();
    ta.noff = P.noff.get();
    ta.uoff = P.uoff.get();
    ta.tnode = P.tnode.get();
    ta.txyz = P.txyz.get();
    ta.lconn = P.lconn.get();
    ta.nent_off = P.nent_off.get();
    ta.nent = P.nent.get();
    ta.ndst = P.ndst.get();
    ta.uent_off = P.uent_off.get();
    ta.uent = P.uent.get();
    ta.udst = P.udst.get();
    ta.part = P.part.get();
    ta.R = R;
    ta.J = data;
    ta.t3v = m->t3v.get();
    ta.t3flag = m->t3_flag.get();
    ta.up_out = up_dst;
    ta.rt_out = rt_out;
    ta.br_out = br_out;
    ta.mon = mo;
    ta.up_fz = up_fz;
    ta.br_fz = br_fz;
    ta.flows = flows_d;
    ta.case_of = case_of;
    ta.n_cases = n_cases;
    ta.max_nodes = P.max_nodes;
    ta.max_edges = P.max_edges;
    ta.E = m->E;
    ta.n_tiles = P.n_tiles;
    ta.F0 = F;
    ta.u2 = u2;
    const bool jac = data != nullptr;
    prof_begin(PROF_ELEM, s);
    if (flows_d) {
        if (up_fz) {
            if (jac) launch_tiles<true, true, true>(m, ta, s);
            else launch_tiles<true, false, true>(m, ta, s);
        } else {
            if (jac) launch_tiles<false, true, true>(m, ta, s);
            else launch_tiles<false, false, true>(m, ta, s);
        }
    } else {
        if (up_fz) {
            if (jac) launch_tiles<true, true, false>(m, ta, s);
            else launch_tiles<true, false, false>(m, ta, s);
        } else {
            if (jac) launch_tiles<false, true, false>(m, ta, s);
            else launch_tiles<false, false, false>(m, ta, s);
        }
    }
    prof_end(PROF_ELEM, s, 1);
    prof_begin(PROF_ROW, s);
    const int64_t n_out = P.n_cnode + (jac ? P.n_cedge : 0);
    if (n_out > 0) {
        const unsigned grid = grid_for(n_out, 256, (int64_t)m->n_sms * 16);
        if (jac)
            k_tile_combine<true><<<grid, 256, 0, s>>>(P.n_cnode, P.cn_off.get(), P.cn_idx.get(), P.cn_dst.get(),
                                                      P.n_cedge, P.ce_off.get(), P.ce_idx.get(), P.ce_dst.get(),
                                                      P.part.get(), R, data);
        else
            k_tile_combine<false><<<grid, 256, 0, s>>>(P.n_cnode, P.cn_off.get(), P.cn_idx.get(), P.cn_dst.get(),
                                                       P.n_cedge, P.ce_off.get(), P.ce_idx.get(), P.ce_dst.get(),
                                                       P.part.get(), R, data);
        UP3D_CHECK_LAUNCH();
    }
    prof_end(PROF_ROW, s, 1);
}

// The fused evaluation: element sweep, row gather, Term 3.  flows_d /
// case_of select per-element flows (several cases in one mesh) when set.
static void fused_evaluate(up3d_mesh* m, const double* phi, const Flow& F, double u2, const Flow* flows_d,
                           const int32_t* case_of, const int64_t* up_fz, const int8_t* br_fz, double* R,
                           double* data, double* rt_out, int32_t* up_out, up3d_monitors* mon, cudaStream_t s,
                           int8_t* br_out = nullptr, int n_cases = 0) {
    up3d_monitors* mo = mon ? mon : m->mon_ws.get();
    UP3D_CUDA(cudaMemsetAsync(mo, 0, sizeof(up3d_monitors), s));
    const bool jac = data != nullptr;
    // a captured launch reads whatever flow table is there when it is
    // replayed: only a direct one may count on the table's gamma
    bool air = F.air;
    if (flows_d) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (m->batch_air) UP3D_CUDA(cudaStreamIsCapturing(s, &capture));
        air = m->batch_air && capture == cudaStreamCaptureStatusNone;
    }
    // the walk's result goes straight to the caller's buffer when there is
    // one (Term 3 reads it from there), else to the mesh workspace
    int32_t* up_dst = up_out ? up_out : m->up32.get();
    if (m->tune.assembly == 1) {
        tiled_evaluate(m, phi, F, u2, flows_d, case_of, n_cases, up_fz, br_fz, R, data, rt_out, up_dst, mo, br_out,
                       s);
    } else {
#define FUSED_ARGS                                                                                                \
    m->conn.get(), m->fnbr.get(), m->disp.get(), m->nodes4.get(), phi, F, u2, up_fz, br_fz,                       \
        m->E, m->loc.get(), m->res.get(), m->t3v.get(), m->t3_flag.get(), up_dst, rt_out, mo, flows_d, case_of, \
        n_cases, br_out
    prof_begin(PROF_ELEM, s);
    if (flows_d) {
        if (up_fz) {
            if (jac) launch_sweep<true, true, true>(m, air, s, FUSED_ARGS);
            else launch_sweep<true, false, true>(m, air, s, FUSED_ARGS);
        } else {
            if (jac) launch_sweep<false, true, true>(m, air, s, FUSED_ARGS);
            else launch_sweep<false, false, true>(m, air, s, FUSED_ARGS);
        }
    } else {
        if (up_fz) {
            if (jac) launch_sweep<true, true, false>(m, air, s, FUSED_ARGS);
            else launch_sweep<true, false, false>(m, air, s, FUSED_ARGS);
        } else {
            if (jac) launch_sweep<false, true, false>(m, air, s, FUSED_ARGS);
            else launch_sweep<false, false, false>(m, air, s, FUSED_ARGS);
        }
    }
#undef FUSED_ARGS
    prof_end(PROF_ELEM, s, 1);
    prof_begin(PROF_ROW, s);
    if (jac) launch_row_gather(m, R, data, s);
    else launch_row_residual(m, R, s);
    prof_end(PROF_ROW, s, 1);
    }
    if (jac) {
        // the element sweep counted the active elements: Term 3 is
        // built only when there are any (flags already written)
        const int64_t known = read_back(&mo->n_term3_active, s);
        int64_t na = 0, nx = 0;
        prof_begin(PROF_TERM3, s);
        build_term3(m, data, s, na, nx, known, up_dst);
        prof_end(PROF_TERM3, s, 0);
        m->last_drop_zeros = na > 0;
        if (nx) {
            k_set_i64<<<1, 1, 0, s>>>(&mo->n_term3_extra, nx);
            UP3D_CHECK_LAUNCH();
        }
    }
}

}  // namespace up3d

extern "C" {

int up3d_residual_jacobian(up3d_mesh* m, const double* phi, const up3d_flow* flow, const int64_t* up_fz,
                           const int8_t* br_fz, double* R, double* data, double* rt_out, int32_t* up_out,
                           up3d_monitors* mon, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && phi && flow && R, UP3D_ERR_ARGUMENT, "up3d_residual_jacobian: null argument");
        UP3D_REQUIRE((up_fz == nullptr) == (br_fz == nullptr), UP3D_ERR_ARGUMENT,
                     "up3d_residual_jacobian: frozen upstream and branch go together");
        const Flow F = make_flow(*flow);
        fused_evaluate(m, phi, F, flow->u_inf * flow->u_inf, nullptr, nullptr, up_fz, br_fz, R, data, rt_out,
                       up_out, mon, S(stream));
    });
}

int up3d_mesh_set_tuning(up3d_mesh* m, const up3d_tuning* t) {
    return guarded([&] {
        UP3D_REQUIRE(m && t, UP3D_ERR_ARGUMENT, "up3d_mesh_set_tuning: null argument");
        UP3D_REQUIRE(t->elem_persistent == 0 || t->elem_persistent == 1, UP3D_ERR_VALUE,
                     "up3d_mesh_set_tuning: elem_persistent must be 0 or 1");
        UP3D_REQUIRE(t->row_lanes == 4 || t->row_lanes == 8 || t->row_lanes == 16 || t->row_lanes == 32,
                     UP3D_ERR_VALUE, "up3d_mesh_set_tuning: row_lanes must be 4, 8, 16 or 32");
        UP3D_REQUIRE(t->elem_threads_per_sm == 512 || t->elem_threads_per_sm == 640 ||
                         t->elem_threads_per_sm == 768,
                     UP3D_ERR_VALUE, "up3d_mesh_set_tuning: elem_threads_per_sm must be 512, 640 or 768");

        UP3D_REQUIRE(t->row_plan8 == 0 || t->row_plan8 == 1, UP3D_ERR_VALUE,
                     "up3d_mesh_set_tuning: row_plan8 must be 0 or 1");
        UP3D_REQUIRE(t->assembly == 0 || t->assembly == 1, UP3D_ERR_VALUE,
                     "up3d_mesh_set_tuning: assembly must be 0 (two-pass) or 1 (tiled)");
        UP3D_REQUIRE(t->tile_elems == 128 || t->tile_elems == 256, UP3D_ERR_VALUE,
                     "up3d_mesh_set_tuning: tile_elems must be 128 or 256");
        UP3D_REQUIRE(t->tile_stretch == 1 || t->tile_stretch == 2 || t->tile_stretch == 4, UP3D_ERR_VALUE,
                     "up3d_mesh_set_tuning: tile_stretch must be 1, 2 or 4");
        m->tune = *t;
    });
}

int up3d_mesh_term3_cache_hits(const up3d_mesh* m, int64_t* hits) {
    return guarded([&] {
        UP3D_REQUIRE(m && hits, UP3D_ERR_ARGUMENT, "up3d_mesh_term3_cache_hits: null argument");
        *hits = m->t3c_hits;
    });
}

int up3d_mesh_get_tuning(const up3d_mesh* m, up3d_tuning* t) {
    return guarded([&] {
        UP3D_REQUIRE(m && t, UP3D_ERR_ARGUMENT, "up3d_mesh_get_tuning: null argument");
        *t = m->tune;
    });
}

int up3d_autotune(up3d_mesh* m, const double* phi, const up3d_flow* flow, int reps, up3d_tuning* out,
                  up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && phi && flow, UP3D_ERR_ARGUMENT, "up3d_autotune: null argument");
        UP3D_REQUIRE(reps >= 1 && reps <= 1000, UP3D_ERR_VALUE, "up3d_autotune: reps must be in [1, 1000]");
        cudaStream_t s = S(stream);
        const Flow F = make_flow(*flow);
        const double u2 = flow->u_inf * flow->u_inf;
        DBuf<double> R, J;
        R.alloc(m->N);
        J.alloc(m->nnz);
        struct Events {
            cudaEvent_t a = nullptr, b = nullptr;
            ~Events() {
                if (a) cudaEventDestroy(a);
                if (b) cudaEventDestroy(b);
            }
        } ev;
        UP3D_CUDA(cudaEventCreate(&ev.a));
        UP3D_CUDA(cudaEventCreate(&ev.b));
        // median device time (us) of `reps` launches after one warm-up
        auto time_it = [&](auto&& launch) {
            launch();
            std::vector<float> t(reps);
            for (int r = 0; r < reps; ++r) {
                UP3D_CUDA(cudaEventRecord(ev.a, s));
                launch();
                UP3D_CUDA(cudaEventRecord(ev.b, s));
                UP3D_CUDA(cudaEventSynchronize(ev.b));
                UP3D_CUDA(cudaEventElapsedTime(&t[r], ev.a, ev.b));
            }
            std::sort(t.begin(), t.end());
            return 1e3 * (double)t[reps / 2];
        };
        const up3d_tuning saved = m->tune;
        try {
            const int64_t* no_up = nullptr;
            const int8_t* no_br = nullptr;
            double* no_rt = nullptr;
            const Flow* no_flows = nullptr;
            const int32_t* no_case = nullptr;
            int8_t* no_brout = nullptr;
            up3d_monitors* mo = m->mon_ws.get();
            // the element sweep: Newton Jacobian, live upwind selection
            // (persistent, resident threads per SM)
            static const int shapes[][2] = {{0, 512}, {1, 512}, {1, 640}, {0, 768}, {1, 768}};
            double best_e = 0.0;
            int best_k = -1;
            for (int k = 0; k < (int)(sizeof(shapes) / sizeof(shapes[0])); ++k) {
                m->tune.elem_persistent = shapes[k][0];
                m->tune.elem_threads_per_sm = shapes[k][1];
                const double t = time_it([&] {
                    launch_sweep<false, true, false>(m, F.air, s, m->conn.get(), m->fnbr.get(),
                                                     m->disp.get(), m->nodes4.get(), phi, F, u2, no_up, no_br, m->E,
                                                     m->loc.get(), m->res.get(), m->t3v.get(), m->t3_flag.get(),
                                                     m->up32.get(), no_rt, mo, no_flows, no_case, 0, no_brout);
                });
                if (best_k < 0 || t < best_e) {
                    best_e = t;
                    best_k = k;
                }
            }
            m->tune.elem_persistent = shapes[best_k][0];
            m->tune.elem_threads_per_sm = shapes[best_k][1];
            // the row gather, on the local matrices the sweep left
            static const int lanes[] = {4, 8, 16, 32};
            double best_r = 0.0;
            int best_l = -1, best_p = 0;
            for (int p8 = 0; p8 <= (m->has_plan8 ? 1 : 0); ++p8)
                for (int l : lanes) {
                    m->tune.row_lanes = l;
                    m->tune.row_plan8 = p8;
                    const double t = time_it([&] { launch_row_gather(m, R.get(), J.get(), s); });
                    if (best_l < 0 || t < best_r) {
                        best_r = t;
                        best_l = l;
                        best_p = p8;
                    }
                }
            m->tune.row_lanes = best_l;
            m->tune.row_plan8 = best_p;
            m->tune.elem_us = best_e;
            m->tune.row_us = best_r;
            // the tiled form, one plan per tile size: the whole evaluation
            // (tile kernel + combine) against the two passes
            static const int tile_shapes[][2] = {{256, 1}, {256, 4}, {128, 4}};
            double best_t = 0.0;
            int best_ts = -1;
            for (int k = 0; k < (int)(sizeof(tile_shapes) / sizeof(tile_shapes[0])); ++k) {
                m->tune.tile_elems = tile_shapes[k][0];
                m->tune.tile_stretch = tile_shapes[k][1];
                const double t = time_it([&] {
                    tiled_evaluate(m, phi, F, u2, no_flows, no_case, 0, no_up, no_br, R.get(), J.get(), no_rt,
                                   m->up32.get(), mo, no_brout, s);
                });
                if (best_ts < 0 || t < best_t) {
                    best_t = t;
                    best_ts = k;
                }
            }
            m->tune.tile_elems = tile_shapes[best_ts][0];
            m->tune.tile_stretch = tile_shapes[best_ts][1];
            if (best_t < best_e + best_r) {
                m->tune.assembly = 1;
                m->tune.elem_us = best_t;
                m->tune.row_us = 0.0;
                ensure_tiles(m, m->tune.tile_elems, m->tune.tile_stretch, s);
            } else {
                m->tune.assembly = 0;
            }
        } catch (...) {
            m->tune = saved;
            throw;
        }
        if (out) *out = m->tune;
    });
}

int up3d_residual_jacobian_batched(up3d_mesh* m, const double* phi, int n_cases, const up3d_flow* flows,
                                   const int32_t* case_of, const int64_t* up_fz, const int8_t* br_fz, double* R,
                                   double* data, double* rt_out, int32_t* up_out, int8_t* branch_out,
                                   up3d_monitors* mon, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(m && phi && case_of && R && n_cases > 0, UP3D_ERR_ARGUMENT,
                     "up3d_residual_jacobian_batched: null argument");
        UP3D_REQUIRE((up_fz == nullptr) == (br_fz == nullptr), UP3D_ERR_ARGUMENT,
                     "up3d_residual_jacobian_batched: frozen upstream and branch go together");
        cudaStream_t s = S(stream);
        if (flows) {
            std::vector<Flow> host(n_cases);
            bool air = true;
            for (int c = 0; c < n_cases; ++c) {
                UP3D_REQUIRE(flows[c].u_inf == flows[0].u_inf, UP3D_ERR_VALUE,
                             "up3d_residual_jacobian_batched: the cases must share u_inf");
                host[c] = make_flow(flows[c]);
                air &= host[c].air;
            }
            m->flows_ws.alloc(n_cases);
            m->i64_ws.alloc(8);
            int* bad = reinterpret_cast<int*>(m->i64_ws.get() + 7);
            UP3D_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), s));
            k_check_cases<<<grid_for(m->E, 256), 256, 0, s>>>(case_of, m->E, n_cases, bad);
            UP3D_CHECK_LAUNCH();
            UP3D_CUDA(cudaMemcpyAsync(m->flows_ws.get(), host.data(), sizeof(Flow) * n_cases,
                                      cudaMemcpyHostToDevice, s));
            const int hbad = read_back(bad, s);   // also: `host` may go out of scope
            m->batch_cases = 0;
            UP3D_REQUIRE(!hbad, UP3D_ERR_VALUE, "up3d_residual_jacobian_batched: case index out of range");
            m->batch_cases = n_cases;
            m->batch_air = air;
            m->batch_flow0 = flows[0];
        } else {
            UP3D_REQUIRE(m->batch_cases == n_cases, UP3D_ERR_VALUE,
                         "up3d_residual_jacobian_batched: no flow table of this many cases on the mesh "
                         "(pass the flows once)");
        }
        const up3d_flow& f0 = m->batch_flow0;
        fused_evaluate(m, phi, make_flow(f0), f0.u_inf * f0.u_inf, m->flows_ws.get(), case_of, up_fz, br_fz, R,
                       data, rt_out, up_out, mon, s, branch_out, n_cases);
    });
}

}  // extern "C"
