// Smoothed-aggregation AMG preconditioner of the up3d library (the
// reference's build_amg_preconditioner, solve/linear.py:61-81, which wraps
// pyamg.smoothed_aggregation_solver with its defaults).
//
// Setup, symbolic (host, once per sparsity pattern): all off-diagonal
// connections strong (theta = 0), the three-pass standard aggregation, and
// the patterns of the tentative prolongator T (constant near-null-space
// vector), the smoothed prolongator P = (I - omega D^-1 A) T, A P and the
// Galerkin operator R A P with R = P^T, down to at most `max_coarse`
// unknowns.  With every connection strong the aggregates and all patterns
// depend on the fine pattern alone.
//
// Setup, numeric (device, on every setup and refresh): D^-1, rho(D^-1 A) by
// power iteration, omega = (4/3) / rho, the values of P, A P and R A P in a
// fixed per-row order, and the dense FP64 inverse of the coarsest operator
// (Gauss-Jordan with partial pivoting, coarse_inverse.cuh).  A refresh with a new matrix of the
// same pattern therefore reproduces a fresh setup bit for bit.
//
// Cycle (device): V-cycle with damped-Jacobi pre/post smoothing
// (omega_s = (4/3) / rho(D^-1 A) per level), in FP64 or FP32 (mixed
// precision: level operators, smoothing, restriction and prolongation in
// FP32, the coarsest solve in FP64).  No atomics: bit-reproducible.
// Constrained (Dirichlet) rows of the finest operator are identity rows and
// belong to no aggregate.

#include <omp.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <numeric>
#include <vector>

#include "coarse_inverse.cuh"
#include "csr_rows.cuh"
#include "internal.cuh"
#include "krylov.cuh"

namespace up3d {

namespace {

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

struct HostCSR {
    int64_t n = 0, m = 0;  // rows, cols
    std::vector<int32_t> p, i;
    std::vector<double> x;
};

// Host <-> device copies of the setup through one process-wide page-locked
// staging buffer (grown once, kept): pageable copies of the level patterns
// were a large part of the setup time.
struct Stage {
    std::mutex mu;
    unsigned char* p = nullptr;
    size_t n = 0;
};
Stage& stage() {
    static Stage st;
    return st;
}
constexpr size_t STAGE_CHUNK = size_t(32) << 20;
unsigned char* stage_buffer(Stage& st) {
    if (!st.p) {
        UP3D_CUDA(cudaMallocHost(&st.p, STAGE_CHUNK));
        st.n = STAGE_CHUNK;
    }
    return st.p;
}
// host memcpy spread over the OpenMP threads (1 MiB pieces): a single
// thread copies pageable memory at a fraction of the link's rate
void par_memcpy(unsigned char* dst, const unsigned char* src, size_t bytes) {
    constexpr size_t PIECE = size_t(1) << 20;
    const int64_t pieces = (int64_t)((bytes + PIECE - 1) / PIECE);
#pragma omp parallel for schedule(static) if (pieces > 1)
    for (int64_t k = 0; k < pieces; ++k) {
        const size_t o = (size_t)k * PIECE;
        std::memcpy(dst + o, src + o, std::min(PIECE, bytes - o));
    }
}
void h2d(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    Stage& st = stage();
    std::lock_guard<std::mutex> g(st.mu);
    unsigned char* buf = stage_buffer(st);
    for (size_t o = 0; o < bytes; o += STAGE_CHUNK) {
        const size_t b = std::min(STAGE_CHUNK, bytes - o);
        par_memcpy(buf, static_cast<const unsigned char*>(src) + o, b);
        UP3D_CUDA(cudaMemcpyAsync(static_cast<unsigned char*>(dst) + o, buf, b, cudaMemcpyHostToDevice, s));
        UP3D_CUDA(cudaStreamSynchronize(s));
    }
}
void d2h(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    Stage& st = stage();
    std::lock_guard<std::mutex> g(st.mu);
    unsigned char* buf = stage_buffer(st);
    for (size_t o = 0; o < bytes; o += STAGE_CHUNK) {
        const size_t b = std::min(STAGE_CHUNK, bytes - o);
        UP3D_CUDA(cudaMemcpyAsync(buf, static_cast<const unsigned char*>(src) + o, b, cudaMemcpyDeviceToHost, s));
        UP3D_CUDA(cudaStreamSynchronize(s));
        par_memcpy(static_cast<unsigned char*>(dst) + o, buf, b);
    }
}

// ------------------------------------------------------------ host symbolic setup

// Standard aggregation (three passes, node order).  agg[i] = -1 for nodes
// without strong connections (isolated / constrained).
int64_t standard_aggregation(const HostCSR& A, const std::vector<uint8_t>& skip, std::vector<int32_t>& agg) {
    const int64_t n = A.n;
    agg.assign(n, -1);
    int64_t na = 0;
    auto strong = [&](int64_t r, int32_t c) { return c != r && !skip[c]; };
    // pass 1: node whose strong neighbours are all free seeds an aggregate
    for (int64_t r = 0; r < n; ++r) {
        if (skip[r] || agg[r] >= 0) continue;
        bool free_nbhd = true, has_nbr = false;
        for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
            int32_t c = A.i[k];
            if (!strong(r, c)) continue;
            has_nbr = true;
            if (agg[c] >= 0) {
                free_nbhd = false;
                break;
            }
        }
        if (!has_nbr || !free_nbhd) continue;
        agg[r] = (int32_t)na;
        for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
            int32_t c = A.i[k];
            if (strong(r, c)) agg[c] = (int32_t)na;
        }
        ++na;
    }
    // pass 2: join an aggregated strong neighbour (first in row order)
    std::vector<int32_t> agg1 = agg;
    for (int64_t r = 0; r < n; ++r) {
        if (skip[r] || agg[r] >= 0) continue;
        for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
            int32_t c = A.i[k];
            if (strong(r, c) && agg1[c] >= 0) {
                agg[r] = agg1[c];
                break;
            }
        }
    }
    // pass 3: leftovers seed aggregates with their free strong neighbours
    for (int64_t r = 0; r < n; ++r) {
        if (skip[r] || agg[r] >= 0) continue;
        bool has_nbr = false;
        for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k)
            if (strong(r, A.i[k])) has_nbr = true;
        if (!has_nbr) continue;
        agg[r] = (int32_t)na;
        for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
            int32_t c = A.i[k];
            if (strong(r, c) && agg[c] < 0) agg[c] = (int32_t)na;
        }
        ++na;
    }
    return na;
}

int32_t find_col(const HostCSR& P, int64_t r, int32_t c) {
    auto b = P.i.begin() + P.p[r], e = P.i.begin() + P.p[r + 1];
    auto it = std::lower_bound(b, e, c);
    return (it != e && *it == c) ? (int32_t)(it - P.i.begin()) : -1;
}

// Pattern of P = (I - omega D^-1 A) T: row r holds agg[r] and agg[c] of its
// aggregated neighbours.  amap[k] = slot of A entry k's contribution (-1 when
// its column is unaggregated), self[r] = slot of agg[r] (-1 when none).
// Two passes (count, fill) with a per-thread marker array: no per-row
// allocation.
HostCSR prolongator_pattern(const HostCSR& A, const std::vector<int32_t>& agg, int64_t na,
                            std::vector<int32_t>& amap, std::vector<int32_t>& self) {
    const int64_t n = A.n;
    HostCSR P;
    P.n = n;
    P.m = na;
    P.p.assign(n + 1, 0);
#pragma omp parallel
    {
        std::vector<int32_t> mark(na, -1);
#pragma omp for schedule(static)
        for (int64_t r = 0; r < n; ++r) {
            int32_t cnt = 0;
            if (agg[r] >= 0) {
                mark[agg[r]] = (int32_t)r;
                ++cnt;
            }
            for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
                const int32_t a = agg[A.i[k]];
                if (a >= 0 && mark[a] != (int32_t)r) {
                    mark[a] = (int32_t)r;
                    ++cnt;
                }
            }
            P.p[r + 1] = cnt;
        }
    }
    for (int64_t r = 0; r < n; ++r) P.p[r + 1] += P.p[r];
    P.i.resize(P.p[n]);
    amap.assign(A.i.size(), -1);
    self.assign(n, -1);
#pragma omp parallel
    {
        std::vector<int32_t> mark(na, -1);
#pragma omp for schedule(static)
        for (int64_t r = 0; r < n; ++r) {
            int32_t o = P.p[r];
            if (agg[r] >= 0) {
                mark[agg[r]] = (int32_t)r;
                P.i[o++] = agg[r];
            }
            for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
                const int32_t a = agg[A.i[k]];
                if (a >= 0 && mark[a] != (int32_t)r) {
                    mark[a] = (int32_t)r;
                    P.i[o++] = a;
                }
            }
            std::sort(P.i.begin() + P.p[r], P.i.begin() + P.p[r + 1]);
            if (agg[r] >= 0) self[r] = find_col(P, r, agg[r]);
            for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k)
                if (agg[A.i[k]] >= 0) amap[k] = find_col(P, r, agg[A.i[k]]);
        }
    }
    return P;
}

// R = P^T pattern; R entry t takes the value of P entry tperm[t].  Each
// R row lists its P rows in ascending order: the P rows are cut into one
// contiguous range per thread, each thread counts its range's entries per
// column, and the column-major prefix over (column, thread) gives every
// thread its own slots, filled in row order.
HostCSR transpose_pattern(const HostCSR& P, std::vector<int32_t>& tperm) {
    HostCSR R;
    R.n = P.m;
    R.m = P.n;
    R.p.assign(R.n + 1, 0);
    R.i.resize(P.i.size());
    tperm.resize(P.i.size());
    const int T = std::max(1, std::min(omp_get_max_threads(), 64));
    const int64_t nc = R.n;
    std::vector<int64_t> cnt((size_t)T * (nc + 1), 0);  // (thread, column) counts, then offsets
    auto lo = [&](int t) { return P.n * t / T; };
#pragma omp parallel for schedule(static, 1) num_threads(T)
    for (int t = 0; t < T; ++t) {
        int64_t* c_t = cnt.data() + (size_t)t * (nc + 1);
        for (int64_t r = lo(t); r < lo(t + 1); ++r)
            for (int32_t k = P.p[r]; k < P.p[r + 1]; ++k) c_t[P.i[k]]++;
    }
    int64_t run = 0;
    for (int64_t c = 0; c < nc; ++c) {
        R.p[c] = (int32_t)run;
        for (int t = 0; t < T; ++t) {
            int64_t& v = cnt[(size_t)t * (nc + 1) + c];
            const int64_t n_tc = v;
            v = run;
            run += n_tc;
        }
    }
    R.p[nc] = (int32_t)run;
#pragma omp parallel for schedule(static, 1) num_threads(T)
    for (int t = 0; t < T; ++t) {
        int64_t* c_t = cnt.data() + (size_t)t * (nc + 1);
        for (int64_t r = lo(t); r < lo(t + 1); ++r)
            for (int32_t k = P.p[r]; k < P.p[r + 1]; ++k) {
                const int32_t c = P.i[k];
                const int64_t o = c_t[c]++;
                R.i[o] = (int32_t)r;
                tperm[o] = k;
            }
    }
    return R;
}

// Pattern of C = A B (sorted columns, OpenMP over rows; count and fill
// passes with a per-thread marker array, no per-row allocation).
HostCSR spgemm_pattern(const HostCSR& A, const HostCSR& B) {
    HostCSR C;
    C.n = A.n;
    C.m = B.m;
    C.p.assign(A.n + 1, 0);
#pragma omp parallel
    {
        std::vector<int32_t> mark(B.m, -1);
#pragma omp for schedule(dynamic, 1024)
        for (int64_t r = 0; r < A.n; ++r) {
            int32_t cnt = 0;
            for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
                const int32_t a = A.i[k];
                for (int32_t q = B.p[a]; q < B.p[a + 1]; ++q) {
                    const int32_t c = B.i[q];
                    if (mark[c] != (int32_t)r) {
                        mark[c] = (int32_t)r;
                        ++cnt;
                    }
                }
            }
            C.p[r + 1] = cnt;
        }
    }
    for (int64_t r = 0; r < A.n; ++r) C.p[r + 1] += C.p[r];
    C.i.resize(C.p[A.n]);
#pragma omp parallel
    {
        std::vector<int32_t> mark(B.m, -1);
#pragma omp for schedule(dynamic, 1024)
        for (int64_t r = 0; r < A.n; ++r) {
            int32_t o = C.p[r];
            for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k) {
                const int32_t a = A.i[k];
                for (int32_t q = B.p[a]; q < B.p[a + 1]; ++q) {
                    const int32_t c = B.i[q];
                    if (mark[c] != (int32_t)r) {
                        mark[c] = (int32_t)r;
                        C.i[o++] = c;
                    }
                }
            }
            std::sort(C.i.begin() + C.p[r], C.i.begin() + C.p[r + 1]);
        }
    }
    return C;
}

// Dense inverse by Gauss-Jordan with partial pivoting: the host fallback
// for a singular coarsest operator, inverted after diagonal regularisation.
bool dense_inverse(std::vector<double>& a, int64_t n, std::vector<double>& inv) {
    inv.assign(n * n, 0.0);
    for (int64_t r = 0; r < n; ++r) inv[r * n + r] = 1.0;
    for (int64_t c = 0; c < n; ++c) {
        int64_t piv = c;
        for (int64_t r = c + 1; r < n; ++r)
            if (std::fabs(a[r * n + c]) > std::fabs(a[piv * n + c])) piv = r;
        if (a[piv * n + c] == 0.0) return false;
        if (piv != c)
            for (int64_t k = 0; k < n; ++k) {
                std::swap(a[c * n + k], a[piv * n + k]);
                std::swap(inv[c * n + k], inv[piv * n + k]);
            }
        const double d = 1.0 / a[c * n + c];
        for (int64_t k = 0; k < n; ++k) {
            a[c * n + k] *= d;
            inv[c * n + k] *= d;
        }
#pragma omp parallel for schedule(static)
        for (int64_t r = 0; r < n; ++r) {
            if (r == c) continue;
            const double f = a[r * n + c];
            if (f == 0.0) continue;
            for (int64_t k = 0; k < n; ++k) {
                a[r * n + k] -= f * a[c * n + k];
                inv[r * n + k] -= f * inv[c * n + k];
            }
        }
    }
    return true;
}

// Power-iteration start vector (deterministic xorshift sequence; 0 on
// skipped rows).
std::vector<double> power_start(int64_t n, const std::vector<uint8_t>& skip) {
    std::vector<double> x(n);
    uint64_t h = 0x9E3779B97F4A7C15ull;
    for (int64_t r = 0; r < n; ++r) {
        h ^= h << 13;
        h ^= h >> 7;
        h ^= h << 17;
        x[r] = skip[r] ? 0.0 : 0.5 + (double)(h % 1000003) / 1000003.0;
    }
    return x;
}

// ------------------------------------------------------------ device numeric setup

__device__ __forceinline__ int32_t dev_lower_bound(const int32_t* __restrict__ a, int32_t len, int32_t v) {
    int32_t lo = 0, hi = len;
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Pattern of the finest operator from the caller's: entries of row r in
// cnt[r + 1] (cnt[0] = 0), then, with its row offsets p, the columns and the
// caller's entry of each.  Eight lanes per row (a lane's ballot among its
// row's eight orders the entries).  Bound by the pattern's bytes.
__global__ void __launch_bounds__(256)
    k_embed_count(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                  const uint8_t* __restrict__ dir, int32_t* __restrict__ cnt) {
    const int sub = threadIdx.x & 7;
    const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 3);
    for (int64_t base = (int64_t)blockIdx.x * (blockDim.x >> 3); base < n; base += step) {   // block-uniform
        const int64_t r = base + (threadIdx.x >> 3);
        int32_t c = 0;
        if (r < n && !(dir && dir[r]))
            for (int32_t k = Ap[r] + sub; k < Ap[r + 1]; k += 8) c += !(dir && dir[Ai[k]]);
        for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (r < n && sub == 0) cnt[r + 1] = dir && dir[r] ? 1 : c;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[0] = 0;
}
__global__ void __launch_bounds__(256)
    k_embed_fill(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                 const uint8_t* __restrict__ dir, const int32_t* __restrict__ p, int32_t* __restrict__ out,
                 int32_t* __restrict__ src) {
    const int sub = threadIdx.x & 7, group = threadIdx.x & 24;
    const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 3);
    for (int64_t base = (int64_t)blockIdx.x * (blockDim.x >> 3); base < n; base += step) {   // block-uniform
        const int64_t r = base + (threadIdx.x >> 3);
        int32_t k0 = 0, k1 = 0, o = 0;
        if (r < n) {
            o = p[r];
            if (dir && dir[r]) {
                if (sub == 0) {
                    out[o] = (int32_t)r;
                    src[o] = -1;
                }
            } else {
                k0 = Ap[r];
                k1 = Ap[r + 1];
            }
        }
        const int32_t most = __reduce_max_sync(0xffffffffu, k1 - k0);
        for (int32_t j = 0; j < most; j += 8) {
            const int32_t k = k0 + j + sub;
            const int32_t c = k < k1 ? Ai[k] : 0;
            const bool keep = k < k1 && !(dir && dir[c]);
            const unsigned m = __ballot_sync(0xffffffffu, keep) >> group & 0xffu;
            if (keep) {
                const int32_t at = o + __popc(m & ((1u << sub) - 1u));
                out[at] = c;
                src[at] = k;
            }
            o += __popc(m);
        }
    }
}

// finest operator from the caller's matrix: src[k] = caller entry, or -1
// for the identity entry of a constrained row
__global__ void k_embed(int64_t nnz, const int32_t* __restrict__ src, const double* __restrict__ data,
                        double* __restrict__ out) {
    GRID_STRIDE(k, nnz) out[k] = src[k] >= 0 ? data[src[k]] : 1.0;
}

// State of the power iteration for rho(D^-1 A): the iterate y (unscaled),
// z = s y with s = sqrt|D^-1|, and st = (power of two that brings y to unit
// size, Rayleigh quotient).
__global__ void k_dinv(int64_t n, const int32_t* __restrict__ diag, const double* __restrict__ Ax,
                       double* __restrict__ dinv, double* __restrict__ s, const double* __restrict__ x0,
                       double* __restrict__ y, double* __restrict__ z, double* __restrict__ st,
                       int* __restrict__ done) {
    GRID_STRIDE(r, n) {
        const double d = diag[r] >= 0 ? Ax[diag[r]] : 0.0;
        const double di = d != 0.0 ? __ddiv_rn(1.0, d) : 1.0;
        const double sr = sqrt(fabs(di));
        dinv[r] = di;
        s[r] = sr;
        y[r] = x0[r];
        z[r] = sr * x0[r];
        if (r == 0) {
            st[0] = 1.0;
            st[1] = 0.0;
            *done = 0;
        }
    }
}

// P = (I - omega D^-1 A) T, contributions in the order (T entry, then A's
// entries in row order).  Eight lanes per row, lane `sub` owning the P
// entry at position sub (and sub + 8, ... in further passes): each lane
// forms the term of one A entry, the row's lanes then see the terms one
// after the other.  (One thread per row, adding to P in global memory, took
// 61 us on average over the three levels of the 625 k-row matrix.)
__global__ void __launch_bounds__(128)
    k_prolong(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
              const double* __restrict__ Ax, const int32_t* __restrict__ amap, const int32_t* __restrict__ self,
              const double* __restrict__ t, const double* __restrict__ dinv, const double* __restrict__ omega,
              const int32_t* __restrict__ Pp, double* __restrict__ Px) {
    const int sub = threadIdx.x & 7;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const double om = *omega;
    for (int64_t base = warp * 4; base < n; base += n_warps * 4) {   // warp-uniform
        const int64_t r = base + ((threadIdx.x & 31) >> 3);
        int32_t pb = 0, pl = 0, s = 0, e = 0, own = -1;
        double f = 0.0, tr = 0.0;
        if (r < n) {
            pb = Pp[r];
            pl = Pp[r + 1] - pb;
            s = Ap[r];
            e = Ap[r + 1];
            own = self[r];
            f = __dmul_rn(om, dinv[r]);
            tr = t[r];
        }
        const int len = __reduce_max_sync(0xffffffffu, e - s), most = __reduce_max_sync(0xffffffffu, pl);
        for (int p0 = 0; p0 < most; p0 += 8) {
            const int32_t slot = pb + p0 + sub;
            double acc = slot == own ? tr : 0.0;
            for (int k0 = 0; k0 < len; k0 += 8) {
                int32_t q = -1;
                double v = 0.0;
                if (s + k0 + sub < e) {
                    const int32_t k = s + k0 + sub;
                    q = amap[k];
                    if (q >= 0) v = __dmul_rn(__dmul_rn(-f, Ax[k]), t[Ai[k]]);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int32_t qj = __shfl_sync(0xffffffffu, q, j, 8);
                    const double vj = __shfl_sync(0xffffffffu, v, j, 8);
                    if (qj == slot) acc = __dadd_rn(acc, vj);
                }
            }
            if (p0 + sub < pl) Px[slot] = acc;
        }
    }
}

__global__ void k_gather_vals(int64_t m, const int32_t* __restrict__ perm, const double* __restrict__ src,
                              double* __restrict__ dst) {
    GRID_STRIDE(k, m) dst[k] = src[perm[k]];
}

// C = A B on C's precomputed pattern, products added to each C entry in
// (A entry, B entry) order, each rounded (the same bits for every kernel
// below).  One thread per row left a coarse row's hundreds of products (a
// Galerkin row of the 625 k-row Picard matrix: 89 R entries x 8.5 A P
// entries) as one chain of dependent loads and global read-modify-writes:
// 1.26 ms per product on average, 7.5 of the 11.4 ms of a refresh; with the
// kernels below the six products take 0.9 ms (Picard step 25.5 -> 18.9 ms).

// Short C rows (at most 16 entries: A P of a P1 level, 15 x 3.6 products
// into 8.5 entries): eight lanes per row, each lane owning the columns at
// positions sub and sub + 8 of the row and adding the products that land
// there; the row's A entries are loaded eight at a time, one per lane, and
// the B rows read as broadcasts.  No search, no shared memory.
constexpr int SPGEMM_OWNED = 16;
__global__ void __launch_bounds__(128)
    k_spgemm_owned(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                   const double* __restrict__ Ax, const int32_t* __restrict__ Bp, const int32_t* __restrict__ Bi,
                   const double* __restrict__ Bx, const int32_t* __restrict__ Cp, const int32_t* __restrict__ Ci,
                   double* __restrict__ Cx) {
    const int sub = threadIdx.x & 7;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = warp * 4; base < n; base += n_warps * 4) {   // warp-uniform
        const int64_t r = base + ((threadIdx.x & 31) >> 3);
        int32_t cb = 0, cl = 0, s = 0, e = 0;
        if (r < n) {
            cb = Cp[r];
            cl = Cp[r + 1] - cb;
            s = Ap[r];
            e = Ap[r + 1];
        }
        const int32_t c0 = sub < cl ? Ci[cb + sub] : -1, c1 = sub + 8 < cl ? Ci[cb + sub + 8] : -1;
        double acc0 = 0.0, acc1 = 0.0;
        const int len = __reduce_max_sync(0xffffffffu, e - s);
        for (int k0 = 0; k0 < len; k0 += 8) {
            double a = 0.0;
            int32_t b0 = 0, b1 = 0;
            if (s + k0 + sub < e) {
                const int32_t j = Ai[s + k0 + sub];
                a = Ax[s + k0 + sub];
                b0 = Bp[j];
                b1 = Bp[j + 1];
            }
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const double at = __shfl_sync(0xffffffffu, a, t, 8);
                const int32_t q1 = __shfl_sync(0xffffffffu, b1, t, 8);
                for (int32_t q = __shfl_sync(0xffffffffu, b0, t, 8); q < q1; ++q) {
                    const int32_t c = Bi[q];
                    const double v = __dmul_rn(at, Bx[q]);
                    if (c == c0) acc0 = __dadd_rn(acc0, v);
                    if (c == c1) acc1 = __dadd_rn(acc1, v);
                }
            }
        }
        if (sub < cl) Cx[cb + sub] = acc0;
        if (sub + 8 < cl) Cx[cb + sub + 8] = acc1;
    }
}

// One C row by one warp: G lanes per A entry walk its B row (32 / G entries
// side by side, SPGEMM_UNROLL rounds of them loaded and located in the C
// row ahead of the adds), the groups then add in entry order, one after the
// other.  `cols` / `acc`: the C row's columns and its zeroed sums, in
// shared memory or (rows longer than the staging) in place.
constexpr int SPGEMM_UNROLL = 2;
template <int G>
__device__ __forceinline__ void spgemm_row(int32_t s, int32_t e, const int32_t* __restrict__ Ai,
                                           const double* __restrict__ Ax, const int32_t* __restrict__ Bp,
                                           const int32_t* __restrict__ Bi, const double* __restrict__ Bx,
                                           const int32_t* cols, int32_t cl, double* acc) {
    constexpr int NG = 32 / G;
    const int lane = threadIdx.x & 31, grp = lane / G, sub = lane % G;
    for (int32_t k0 = s; k0 < e; k0 += 32) {
        double a = 0.0;
        int32_t b0 = 0, b1 = 0;
        if (k0 + lane < e) {
            const int32_t j = Ai[k0 + lane];
            a = Ax[k0 + lane];
            b0 = Bp[j];
            b1 = Bp[j + 1];
        }
        const int cnt = e - k0 < 32 ? e - k0 : 32;
        for (int t0 = 0; t0 < cnt; t0 += NG * SPGEMM_UNROLL) {
            double av[SPGEMM_UNROLL], v[SPGEMM_UNROLL];
            int32_t q0[SPGEMM_UNROLL], q1[SPGEMM_UNROLL], pos[SPGEMM_UNROLL];
#pragma unroll
            for (int u = 0; u < SPGEMM_UNROLL; ++u) {
                const int src = t0 + u * NG + grp;   // past cnt: an empty entry or another lane's, masked below
                av[u] = __shfl_sync(0xffffffffu, a, src & 31);
                q0[u] = __shfl_sync(0xffffffffu, b0, src & 31);
                q1[u] = __shfl_sync(0xffffffffu, b1, src & 31);
                if (src >= cnt) q1[u] = q0[u];
                pos[u] = -1;
                if (q0[u] + sub < q1[u]) {
                    v[u] = __dmul_rn(av[u], Bx[q0[u] + sub]);
                    pos[u] = dev_lower_bound(cols, cl, Bi[q0[u] + sub]);
                }
            }
#pragma unroll
            for (int u = 0; u < SPGEMM_UNROLL; ++u)
                for (int g = 0; g < NG; ++g) {
                    if (grp == g) {
                        if (pos[u] >= 0) acc[pos[u]] = __dadd_rn(acc[pos[u]], v[u]);
                        for (int32_t q = q0[u] + sub + G; q < q1[u]; q += G) {   // B rows longer than G
                            const int32_t p = dev_lower_bound(cols, cl, Bi[q]);
                            acc[p] = __dadd_rn(acc[p], __dmul_rn(av[u], Bx[q]));
                        }
                    }
                    __syncwarp();
                }
        }
    }
}

// One warp per C row, the row's columns and sums staged in shared memory
// (`cap` entries per warp; longer rows work in place).
constexpr int SPGEMM_WARPS = 4, SPGEMM_CAP = 1024;
template <int G>
__global__ void __launch_bounds__(SPGEMM_WARPS * 32)
    k_spgemm_warp(int64_t n, int cap, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                  const double* __restrict__ Ax, const int32_t* __restrict__ Bp, const int32_t* __restrict__ Bi,
                  const double* __restrict__ Bx, const int32_t* __restrict__ Cp, const int32_t* __restrict__ Ci,
                  double* __restrict__ Cx) {
    extern __shared__ __align__(16) unsigned char spgemm_sm[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double* sacc = reinterpret_cast<double*>(spgemm_sm) + (size_t)w * cap;
    int32_t* scol = reinterpret_cast<int32_t*>(spgemm_sm + sizeof(double) * SPGEMM_WARPS * cap) + (size_t)w * cap;
    const int64_t n_warps = (int64_t)gridDim.x * SPGEMM_WARPS;
    for (int64_t r = (int64_t)blockIdx.x * SPGEMM_WARPS + w; r < n; r += n_warps) {
        const int32_t cb = Cp[r], cl = Cp[r + 1] - cb;
        if (cl <= cap) {
            for (int32_t q = lane; q < cl; q += 32) {
                scol[q] = Ci[cb + q];
                sacc[q] = 0.0;
            }
            __syncwarp();
            spgemm_row<G>(Ap[r], Ap[r + 1], Ai, Ax, Bp, Bi, Bx, scol, cl, sacc);
            for (int32_t q = lane; q < cl; q += 32) Cx[cb + q] = sacc[q];
            __syncwarp();
        } else {
            for (int32_t q = lane; q < cl; q += 32) Cx[cb + q] = 0.0;
            __syncwarp();
            spgemm_row<G>(Ap[r], Ap[r + 1], Ai, Ax, Bp, Bi, Bx, Ci + cb, cl, Cx + cb);
        }
    }
}

__global__ void k_densify(int64_t n, const int32_t* __restrict__ Cp, const int32_t* __restrict__ Ci,
                          const double* __restrict__ Cx, double* __restrict__ a, double* __restrict__ inv) {
    GRID_STRIDE(r, n) {
        for (int64_t c = 0; c < n; ++c) {
            a[r * n + c] = 0.0;
            inv[r * n + c] = (c == r) ? 1.0 : 0.0;
        }
        for (int32_t k = Cp[r]; k < Cp[r + 1]; ++k) a[r * n + Ci[k]] = Cx[k];
    }
}

// Gauss-Jordan column step c (one block): pivot = first row of largest
// |a[r][c]|, r >= c; swap; scale row c; fcol[r] = a[r][c] for r != c.
__global__ void __launch_bounds__(1024)
    k_gj_pivot(double* __restrict__ a, double* __restrict__ inv, int64_t n, int64_t c, double* __restrict__ fcol,
               int* __restrict__ singular) {
    __shared__ double sv[32];
    __shared__ int64_t si[32];
    __shared__ double sd;
    __shared__ int64_t spiv;
    if (*singular) return;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    double best = -1.0;
    int64_t bi = n;
    for (int64_t r = c + tid; r < n; r += blockDim.x) {
        const double v = fabs(a[r * n + c]);
        if (v > best) {
            best = v;
            bi = r;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int64_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) {
            best = ov;
            bi = oi;
        }
    }
    if (lane == 0) {
        sv[w] = best;
        si[w] = bi;
    }
    __syncthreads();
    if (tid == 0) {
        double b = -1.0;
        int64_t p = n;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k)
            if (sv[k] > b || (sv[k] == b && si[k] < p)) {
                b = sv[k];
                p = si[k];
            }
        spiv = p;
    }
    __syncthreads();
    const int64_t piv = spiv;
    if (piv >= n || a[piv * n + c] == 0.0) {
        if (tid == 0) *singular = 1;
        return;
    }
    if (piv != c)
        for (int64_t k = tid; k < n; k += blockDim.x) {
            double t0 = a[c * n + k];
            a[c * n + k] = a[piv * n + k];
            a[piv * n + k] = t0;
            t0 = inv[c * n + k];
            inv[c * n + k] = inv[piv * n + k];
            inv[piv * n + k] = t0;
        }
    __syncthreads();
    if (tid == 0) sd = __ddiv_rn(1.0, a[c * n + c]);
    __syncthreads();
    const double d = sd;
    for (int64_t k = tid; k < n; k += blockDim.x) {
        a[c * n + k] = __dmul_rn(a[c * n + k], d);
        inv[c * n + k] = __dmul_rn(inv[c * n + k], d);
    }
    __syncthreads();
    for (int64_t r = tid; r < n; r += blockDim.x) fcol[r] = r == c ? 0.0 : a[r * n + c];
}

// Gauss-Jordan elimination of column c from every other row.
__global__ void k_gj_elim(double* __restrict__ a, double* __restrict__ inv, int64_t n, int64_t c,
                          const double* __restrict__ fcol, const int* __restrict__ singular) {
    if (*singular) return;
    GRID_STRIDE(idx, n * 2 * n) {
        const int64_t r = idx / (2 * n), k = idx % (2 * n);
        const double f = fcol[r];
        if (r == c || f == 0.0) continue;
        if (k < n) a[r * n + k] = __dsub_rn(a[r * n + k], __dmul_rn(f, a[c * n + k]));
        else inv[r * n + k - n] = __dsub_rn(inv[r * n + k - n], __dmul_rn(f, inv[c * n + k - n]));
    }
}

// ------------------------------------------------------------ device kernels

// The kernels of the cycle take part in overlapped launches (pdl_wait) and
// read the smoothing weight from the device, so that a captured cycle stays
// valid when the values are refreshed.  Vectors are plain pointers, not
// __restrict__ (read-only loads): the kernel before may still be writing them
// when a kernel starts.

// x = w D^-1 b from b = b_in (kept in b_out unless null)
template <class T, class TI>
__global__ void __launch_bounds__(256)
    k_jacobi_first(const T* __restrict__ dinv, const TI* b_in, T* b_out, T* x, const double* __restrict__ omega,
                   int64_t n) {
    pdl_trigger();
    pdl_wait();
    const T w = (T)*omega;
    GRID_STRIDE(i, n) {
        const T b = (T)b_in[i];
        if (b_out) b_out[i] = b;
        x[i] = w * dinv[i] * b;
    }
}

// Row loop shared by the CSR kernels below: TPR = 0 is one warp per 32
// rows (csr_rows.cuh warp_row_sum), else TPR lanes per row; the row's sum of
// A_rc x_c goes to epi(r, acc), called once per row, by one lane.  BLOCK
// threads per block.
template <int TPR>
constexpr int rows_block = TPR == 0 ? CSR_WARP_BLOCK : CSR_ROWS_BLOCK;
template <class T, int TPR, int BLOCK, class Epi>
__device__ __forceinline__ void csr_rows_loop(int64_t n, const int32_t* __restrict__ Ap,
                                              const int32_t* __restrict__ Ai, const T* __restrict__ Ax,
                                              const T* x, Epi epi) {
    const int64_t warp = (blockIdx.x * (int64_t)BLOCK + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * BLOCK) >> 5;
    auto term = [&](int32_t c, T v) { return v * x[c]; };
    if constexpr (TPR == 0) {
        __shared__ T sh[BLOCK / 32][CSR_ROWS_CHUNK];
        const int lane = threadIdx.x & 31;
        for (int64_t r0 = warp * 32; r0 < n; r0 += n_warps * 32) {   // warp-uniform
            const T acc = warp_row_sum<T>(Ap, Ai, Ax, r0, n, sh[threadIdx.x >> 5], term);
            if (r0 + lane < n) epi(r0 + lane, acc);
        }
    } else {
        constexpr int RPW = 32 / TPR;
        const int sub = threadIdx.x % TPR, group = (threadIdx.x & 31) / TPR;
        for (int64_t base = warp * RPW; base < n; base += n_warps * RPW) {   // warp-uniform
            const int64_t r = base + group;
            const T acc = lanes_row_sum<T, TPR>(Ap, Ai, Ax, r, n, term);
            if (sub == 0 && r < n) epi(r, acc);
        }
    }
}

// One power-iteration step y' = S A S x, x = st[0] y: writes y' and z' = s y',
// and the last block to finish turns the blocks' sums of x.y', y'.y', x.x
// (added in block order) into the Rayleigh quotient st[1] and the next
// scale; *done stops the steps that follow once y' = 0.  With `omega`, the
// last step's: omega = (4/3) / rho, rho = 1.05 lambda (a small safety margin
// on the Rayleigh quotient), 2 when lambda <= 0.  The scale is a power of two
// so that normalising costs neither rounding nor a pass.  One launch per
// step; the product, two dots, scalar update and normalisation as five
// launches took 20 x 45 us on the 625 k-row matrix.
constexpr int PW_BLOCKS = 148 * 8;
template <int TPR>
__global__ void __launch_bounds__(256)
    k_pw_step(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
              const double* __restrict__ Ax, const double* __restrict__ s, const uint8_t* __restrict__ skip,
              const double* __restrict__ y, const double* __restrict__ z, double* __restrict__ y1,
              double* __restrict__ z1, double* __restrict__ st, int* __restrict__ done,
              double* __restrict__ partial, unsigned int* __restrict__ counter, double* __restrict__ omega) {
    __shared__ double sums[3][8];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto finish = [&](double lam) {
        if (omega) *omega = (4.0 / 3.0) / (lam > 0.0 ? 1.05 * lam : 2.0);
    };
    if (*done) {
        if (blockIdx.x == 0 && threadIdx.x == 0) finish(st[1]);
        return;
    }
    const double sc = st[0];
    double acc[3] = {0.0, 0.0, 0.0};
    csr_rows_loop<double, TPR, 256>(n, Ap, Ai, Ax, z, [&](int64_t r, double a) {
        const double v = skip && skip[r] ? 0.0 : s[r] * (sc * a), x = sc * y[r];
        y1[r] = v;
        z1[r] = s[r] * v;
        acc[0] += x * v;
        acc[1] += v * v;
        acc[2] += x * x;
    });
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const double v = warp_sum(acc[j]);
        if (lane == 0) sums[j][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
        for (int q = 0; q < 8; ++q) v += sums[threadIdx.x][q];
        partial[threadIdx.x * PW_BLOCKS + blockIdx.x] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (w < 3) {
        double v = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) v += __ldcg(partial + w * PW_BLOCKS + b);
        v = warp_sum(v);
        if (lane == 0) sums[w][0] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double xy = sums[0][0], yy = sums[1][0], xx = sums[2][0];
        const double lam = xx > 0.0 ? xy / xx : 0.0;
        st[1] = lam;
        if (yy == 0.0) *done = 1;
        else st[0] = isfinite(yy) ? ldexp(1.0, -ilogb(sqrt(yy))) : 1.0;
        finish(lam);
        *counter = 0u;
    }
}

// out = x + w D^-1 (b - A x)   (or, with RESID, out = b - A x).  The finest
// operator is the embedded one (identity rows, no constrained columns): no
// mask.  TO: type of out (the caller's vector behind the last sweep).
template <class T, bool RESID, int TPR, class TO>
__global__ void __launch_bounds__(rows_block<TPR>)
    k_jacobi_sweep(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                   const T* __restrict__ Ax, const T* __restrict__ dinv, const T* b, const T* x, TO* out,
                   const double* __restrict__ omega) {
    pdl_trigger();
    pdl_wait();
    const T w = (T)*omega;
    csr_rows_loop<T, TPR, rows_block<TPR>>(n, Ap, Ai, Ax, x, [&](int64_t r, T acc) {
        const T res = b[r] - acc;
        out[r] = (TO)(RESID ? res : x[r] + w * dinv[r] * res);
    });
}

// The same sweep on the sliced rows, one row per lane; the first entries are
// on their way while the kernel before drains.
template <class T, bool RESID, class TO>
__global__ void __launch_bounds__(SELL_BLOCK)
    k_jacobi_sell(int64_t n, const int32_t* __restrict__ Sp, const int32_t* __restrict__ Si,
                  const T* __restrict__ Sx, const T* __restrict__ dinv, const T* b, const T* x, TO* out,
                  const double* __restrict__ omega) {
    pdl_trigger();
    const int64_t r = blockIdx.x * (int64_t)SELL_BLOCK + threadIdx.x;
    const int lane = threadIdx.x & 31;
    if (r - lane >= n) return;   // warp-uniform
    const T acc = sell_row_sum<T>(Sp, Si, Sx, x, r >> 5, lane, pdl_wait);
    if (r >= n) return;
    const T res = b[r] - acc;
    out[r] = (TO)(RESID ? res : x[r] + (T)*omega * dinv[r] * res);
}

// Column indices of the sliced rows from the CSR ones (-1 on the padding),
// and the values at the cycle's precision.
__global__ void k_sell_index(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai,
                             const int32_t* __restrict__ Sp, int32_t* __restrict__ Si) {
    GRID_STRIDE(r, (n + 31) / 32 * 32) {   // the last slice's unused lanes are padding too
        const int64_t q = r >> 5;
        const int32_t s = Sp[q] + (int32_t)(r & 31), w = (Sp[q + 1] - Sp[q]) >> 5;
        const int32_t p = r < n ? Ap[r] : 0, len = r < n ? Ap[r + 1] - p : 0;
        for (int32_t k = 0; k < w; ++k) Si[s + 32 * k] = k < len ? Ai[p + k] : -1;
    }
}
template <class T>
__global__ void k_sell_values(int64_t n, const int32_t* __restrict__ Ap, const double* __restrict__ Ax,
                              const int32_t* __restrict__ Sp, T* __restrict__ Sx) {
    GRID_STRIDE(r, (n + 31) / 32 * 32) {   // the last slice's unused lanes are padding too
        const int64_t q = r >> 5;
        const int32_t s = Sp[q] + (int32_t)(r & 31), w = (Sp[q + 1] - Sp[q]) >> 5;
        const int32_t p = r < n ? Ap[r] : 0, len = r < n ? Ap[r + 1] - p : 0;
        for (int32_t k = 0; k < w; ++k) Sx[s + 32 * k] = k < len ? (T)Ax[p + k] : T(0);
    }
}

// y (+)= A x, rectangular (restriction / prolongation)
template <class T, bool ADD, int TPR>
__global__ void __launch_bounds__(rows_block<TPR>)
    k_spmv_rect(int64_t n, const int32_t* __restrict__ Ap, const int32_t* __restrict__ Ai, const T* __restrict__ Ax,
                const T* x, T* y) {
    pdl_trigger();
    pdl_wait();
    csr_rows_loop<T, TPR, rows_block<TPR>>(n, Ap, Ai, Ax, x,
                                           [&](int64_t r, T acc) { y[r] = ADD ? y[r] + acc : acc; });
}

template <class T, bool RESID, class TO>
void launch_sweep(bool overlap, int64_t n, int64_t nnz, const int32_t* Ap, const int32_t* Ai, const T* Ax,
                  const T* dinv, const T* b, const T* x, TO* out, const double* omega, cudaStream_t s) {
    const int tpr = use_warp_rows(n, nnz) ? 0 : lanes_per_row(nnz, n);
    auto kern = tpr == 0 ? k_jacobi_sweep<T, RESID, 0, TO> : tpr == 4 ? k_jacobi_sweep<T, RESID, 4, TO>
                : tpr == 8 ? k_jacobi_sweep<T, RESID, 8, TO> : tpr == 16 ? k_jacobi_sweep<T, RESID, 16, TO>
                : k_jacobi_sweep<T, RESID, 32, TO>;
    launch_kernel(overlap, kern, tpr == 0 ? csr_rows_grid(n, CSR_WARP_BLOCK) : lanes_grid(n, tpr),
                  tpr == 0 ? CSR_WARP_BLOCK : CSR_ROWS_BLOCK, s, n, Ap, Ai, Ax, dinv, b, x, out, omega);
}

void launch_pw_step(int64_t n, int64_t nnz, const int32_t* Ap, const int32_t* Ai, const double* Ax, const double* sq,
                    const uint8_t* skip, const double* y, const double* z, double* y1, double* z1, double* st,
                    int* done, double* partial, unsigned int* counter, double* omega, cudaStream_t s) {
    const int tpr = use_warp_rows(n, nnz) ? 0 : lanes_per_row(nnz, n);
    const unsigned grid = tpr == 0 ? std::min(csr_rows_grid(n, 256), (unsigned)PW_BLOCKS) : std::min(lanes_grid(n, tpr), (unsigned)PW_BLOCKS);
    auto kern = tpr == 0 ? k_pw_step<0> : tpr == 4 ? k_pw_step<4> : tpr == 8 ? k_pw_step<8>
                : tpr == 16 ? k_pw_step<16> : k_pw_step<32>;
    kern<<<grid, 256, 0, s>>>(n, Ap, Ai, Ax, sq, skip, y, z, y1, z1, st, done, partial, counter, omega);
    UP3D_CHECK_LAUNCH();
}

template <class T, bool ADD>
void launch_rect(bool overlap, int64_t n, int64_t nnz, const int32_t* Ap, const int32_t* Ai, const T* Ax, const T* x,
                 T* y, cudaStream_t s) {
    const int tpr = use_warp_rows(n, nnz) ? 0 : lanes_per_row(nnz, n);
    auto kern = tpr == 0 ? k_spmv_rect<T, ADD, 0> : tpr == 4 ? k_spmv_rect<T, ADD, 4>
                : tpr == 8 ? k_spmv_rect<T, ADD, 8> : tpr == 16 ? k_spmv_rect<T, ADD, 16> : k_spmv_rect<T, ADD, 32>;
    launch_kernel(overlap, kern, tpr == 0 ? csr_rows_grid(n, CSR_WARP_BLOCK) : lanes_grid(n, tpr),
                  tpr == 0 ? CSR_WARP_BLOCK : CSR_ROWS_BLOCK, s, n, Ap, Ai, Ax, x, y);
}

// x = Cinv b (dense, one warp per row), FP64, inputs/outputs of type T
template <class T>
__global__ void __launch_bounds__(256)
    k_dense_solve(const double* __restrict__ Cinv, int64_t n, const T* b, T* x) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = warp; r < n; r += n_warps) {
        double acc = 0.0;
        for (int64_t c = lane; c < n; c += 32) acc += Cinv[r * n + c] * (double)b[c];
        acc = warp_sum(acc);
        if (lane == 0) x[r] = (T)acc;
    }
}

__global__ void k_d2f(const double* __restrict__ a, float* __restrict__ b, int64_t n) {
    GRID_STRIDE(i, n) b[i] = (float)a[i];
}
__global__ void k_f2d(const float* __restrict__ a, double* __restrict__ b, int64_t n) {
    GRID_STRIDE(i, n) b[i] = (double)a[i];
}

template <class T>
struct DevCSR {
    int64_t n = 0, m = 0, nnz = 0;
    DBuf<int32_t> p, i;
    DBuf<T> x;
    void upload_pattern(const HostCSR& h, cudaStream_t s) {
        n = h.n;
        m = h.m;
        nnz = (int64_t)h.i.size();
        p.alloc(n + 1);
        i.alloc(std::max<int64_t>(nnz, 1));
        x.alloc(std::max<int64_t>(nnz, 1));
        h2d(p.get(), h.p.data(), sizeof(int32_t) * (n + 1), s);
        if (nnz) h2d(i.get(), h.i.data(), sizeof(int32_t) * nnz, s);
    }
    template <class U>
    void copy_pattern(const DevCSR<U>& o, cudaStream_t s) {
        n = o.n;
        m = o.m;
        nnz = o.nnz;
        p.alloc(n + 1);
        i.alloc(std::max<int64_t>(nnz, 1));
        x.alloc(std::max<int64_t>(nnz, 1));
        UP3D_CUDA(cudaMemcpyAsync(p.get(), o.p.get(), sizeof(int32_t) * (n + 1), cudaMemcpyDeviceToDevice, s));
        if (nnz)
            UP3D_CUDA(cudaMemcpyAsync(i.get(), o.i.get(), sizeof(int32_t) * nnz, cudaMemcpyDeviceToDevice, s));
    }
};

// Values of C = A B (all patterns set up); c_max = longest C row.
void launch_spgemm(const DevCSR<double>& A, const DevCSR<double>& B, const DevCSR<double>& C, int c_max,
                   cudaStream_t s) {
    if (c_max <= SPGEMM_OWNED) {
        k_spgemm_owned<<<grid_for(C.n, 16, (int64_t)148 * 64), 128, 0, s>>>(C.n, A.p.get(), A.i.get(), A.x.get(), B.p.get(), B.i.get(),
                                                          B.x.get(), C.p.get(), C.i.get(), C.x.get());
    } else {
        const int cap = std::min(c_max, SPGEMM_CAP);
        const size_t smem = (sizeof(double) + sizeof(int32_t)) * SPGEMM_WARPS * (size_t)cap;
        const unsigned grid = grid_for(C.n, SPGEMM_WARPS, (int64_t)148 * 64);
        // lanes per A entry: the mean B row length, rounded up
        auto kern = B.nnz <= 8 * B.n ? k_spgemm_warp<8> : B.nnz <= 16 * B.n ? k_spgemm_warp<16> : k_spgemm_warp<32>;
        kern<<<grid, SPGEMM_WARPS * 32, smem, s>>>(C.n, cap, A.p.get(), A.i.get(), A.x.get(), B.p.get(), B.i.get(),
                                                   B.x.get(), C.p.get(), C.i.get(), C.x.get());
    }
    UP3D_CHECK_LAUNCH();
}

template <class T>
void upload(DBuf<T>& d, const std::vector<T>& h, cudaStream_t s) {
    d.alloc(std::max<size_t>(h.size(), 1));
    if (!h.empty()) h2d(d.get(), h.data(), sizeof(T) * h.size(), s);
}

// values of type T from FP64 (copy or narrowing)
template <class T>
void convert(const double* src, T* dst, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    if constexpr (std::is_same<T, double>::value) {
        UP3D_CUDA(cudaMemcpyAsync(dst, src, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    } else {
        k_d2f<<<grid_for(n, 256), 256, 0, s>>>(src, dst, n);
        UP3D_CHECK_LAUNCH();
    }
}

template <class T>
struct Ref {  // non-owning device pointer with the DBuf accessor
    T* v = nullptr;
    T* get() const { return v; }
};
template <class T>
struct CsrRef {
    int64_t n = 0, m = 0, nnz = 0;
    Ref<const int32_t> p, i;
    Ref<T> x;
};

// One level of the cycle: views of the symbolic level's patterns and, for
// the FP64 cycle, of its FP64 values; the FP32 cycle owns FP32 copies.
template <class T>
struct Level {
    CsrRef<T> A, P, R;
    Ref<T> dinv;
    const int32_t* sell_p = nullptr;        // A in slices of 32 rows, when it is kept that way
    const int32_t* sell_i = nullptr;
    DBuf<T> sell_x;
    DBuf<T> own_A, own_P, own_R, own_dinv;  // FP32 values (unused for FP64)
    DBuf<T> x, b, r;
    const double* omega = nullptr;          // smoothing weight (device)
};

// Symbolic structure and FP64 values of one level.
struct SymLevel {
    DevCSR<double> A;            // level operator
    DBuf<int32_t> diag;          // (n) slot of the diagonal, -1 when absent
    DBuf<uint8_t> skip;          // (n) constrained rows (finest level only)
    DBuf<double> x0, dinv, sq;   // power-iteration start, D^-1, sqrt|D^-1|
    // to the next level (absent on the coarsest)
    DBuf<int32_t> amap, self;    // A entry / row -> P slot
    DBuf<double> t;              // tentative prolongator value of each row
    DevCSR<double> P, R, AP;     // prolongator, restriction (P^T), A P
    DBuf<int32_t> tperm;         // R entry -> P entry
    int a_max = 0, ap_max = 0;   // longest rows of A and A P
    bool has_skip = false;
    DBuf<int32_t> sell_p, sell_i;   // A's slices (sell_n = 0: not kept)
    int64_t sell_n = 0;
};

}  // namespace

struct Amg {
    bool fp32 = false;  // an FP32 cycle exists (Lf)
    bool fp64 = true;   // an FP64 cycle exists (Ld)
    int pre = 2, post = 2;
    int64_t n_coarse = 0;
    // the caller's finest pattern (refresh checks) and its embedding
    int64_t n_in = 0, nnz_in = 0;
    bool has_dir = false;
    DBuf<int32_t> in_p, in_i, emb_src;
    DBuf<uint8_t> in_dir;
    std::vector<SymLevel*> sym;
    // numeric scratch
    DBuf<double> pw_yz, pw_scal, omega_dev, gj_fac, dense_a, fcol;
    DBuf<int> flags;
    DBuf<double> cinv;
    std::vector<Level<double>*> Ld;
    std::vector<Level<float>*> Lf;
    up3d_amg_info info{};
    // the V-cycle of each precision between its first smoothing (which reads
    // the caller's vector) and its last (which writes the caller's) as a
    // CUDA graph on the levels' own buffers: captured once on a private
    // stream, replayed for every vector and every refresh of the values
    struct Body {
        cudaGraphExec_t exec = nullptr;
        long long launches = 0;
        void* x = nullptr;   // the level-0 iterate after the body
    };
    Body body64, body32;
    cudaStream_t capture_stream = nullptr;
    int device = 0;
    ~Amg() {
        for (Body* b : {&body64, &body32})
            if (b->exec) cudaGraphExecDestroy(b->exec);
        if (capture_stream) cudaStreamDestroy(capture_stream);
        for (auto* l : Ld) delete l;
        for (auto* l : Lf) delete l;
        for (auto* l : sym) delete l;
    }
};

namespace {

// One sweep (or residual) of a level's operator: the sliced rows where the
// level has them, else the CSR rows.
template <class T, bool RESID, class TO>
void smooth(bool overlap, const Level<T>& lv, const T* x, TO* out, cudaStream_t s) {
    const int64_t n = lv.A.n;
    if (lv.sell_p)
        launch_kernel(overlap, k_jacobi_sell<T, RESID, TO>, sell_grid(n), SELL_BLOCK, s, n, lv.sell_p, lv.sell_i,
                      lv.sell_x.get(), lv.dinv.get(), lv.b.get(), x, out, lv.omega);
    else
        launch_sweep<T, RESID, TO>(overlap, n, lv.A.nnz, lv.A.p.get(), lv.A.i.get(), lv.A.x.get(), lv.dinv.get(),
                               lv.b.get(), x, out, lv.omega, s);
}

// The V-cycle on level l from its b to its x; on the finest level (top)
// without the first and the last smoothing.  Its kernels overlap: the first
// that a caller launches must be ordered behind everything before it.
template <class T>
void vcycle(Amg& a, std::vector<Level<T>*>& L, size_t l, bool top, cudaStream_t s) {
    Level<T>& lv = *L[l];
    const int64_t n = lv.A.n;
    if (l + 1 == L.size()) {
        // coarsest: dense FP64 solve
        launch_kernel(true, k_dense_solve<T>, grid_for(32 * n, 256), 256, s, a.cinv.get(), n, lv.b.get(), lv.x.get());
        return;
    }
    // pre-smoothing from x = 0
    if (!top)
        launch_kernel(true, k_jacobi_first<T, T>, grid_for(n, 256), 256, s, lv.dinv.get(), lv.b.get(), nullptr,
                      lv.x.get(), lv.omega, n);
    for (int k = 1; k < a.pre; ++k) {
        smooth<T, false>(true, lv, lv.x.get(), lv.r.get(), s);
        std::swap(lv.x.p, lv.r.p);
    }
    // residual, restriction
    smooth<T, true>(true, lv, lv.x.get(), lv.r.get(), s);
    Level<T>& cv = *L[l + 1];
    launch_rect<T, false>(true, lv.R.n, lv.R.nnz, lv.R.p.get(), lv.R.i.get(), lv.R.x.get(), lv.r.get(), cv.b.get(), s);
    vcycle<T>(a, L, l + 1, false, s);
    // prolongation
    launch_rect<T, true>(true, lv.P.n, lv.P.nnz, lv.P.p.get(), lv.P.i.get(), lv.P.x.get(), cv.x.get(), lv.x.get(), s);
    for (int k = top ? 1 : 0; k < a.post; ++k) {
        smooth<T, false>(true, lv, lv.x.get(), lv.r.get(), s);
        std::swap(lv.x.p, lv.r.p);
    }
}

// Diagonal slot of each row of a pattern.
std::vector<int32_t> diag_slots(const HostCSR& A) {
    std::vector<int32_t> d(A.n, -1);
#pragma omp parallel for schedule(static)
    for (int64_t r = 0; r < A.n; ++r)
        for (int32_t k = A.p[r]; k < A.p[r + 1]; ++k)
            if (A.i[k] == r) d[r] = k;
    return d;
}

int longest_row(const HostCSR& A) {
    int32_t m = 0;
#pragma omp parallel for schedule(static) reduction(max : m)
    for (int64_t r = 0; r < A.n; ++r) m = std::max(m, A.p[r + 1] - A.p[r]);
    return m;
}

// Slices of a level operator (symbolic), when the sliced rows pay.
void make_slices(SymLevel& F, const HostCSR& A, cudaStream_t s) {
    const int64_t nq = (A.n + 31) / 32;
    std::vector<int32_t> sp(nq + 1, 0);
    int64_t run = 0;
    for (int64_t q = 0; q < nq; ++q) {
        int32_t w = 0;
        for (int64_t r = 32 * q; r < std::min(A.n, 32 * q + 32); ++r) w = std::max(w, A.p[r + 1] - A.p[r]);
        run += 32 * (int64_t)w;
        if (run > INT32_MAX) return;
        sp[q + 1] = (int32_t)run;
    }
    if (!use_sell(A.n, (int64_t)A.i.size(), run)) return;
    upload(F.sell_p, sp, s);
    F.sell_i.alloc(run);
    F.sell_n = run;
    k_sell_index<<<grid_for(A.n, 256), 256, 0, s>>>(A.n, F.A.p.get(), F.A.i.get(), F.sell_p.get(), F.sell_i.get());
    UP3D_CHECK_LAUNCH();
    UP3D_CUDA(cudaStreamSynchronize(s));
}

// Device numeric phase: every level's D^-1, omega, P, R, A P and coarser
// operator, then the coarsest inverse; fills the cycle's levels.
void numeric(Amg& a, cudaStream_t s) {
    const size_t L = a.sym.size();
    double* st = a.pw_scal.get();
    double* partial = a.pw_scal.get() + 2;
    unsigned int* counter = reinterpret_cast<unsigned int*>(a.flags.get() + 2);
    UP3D_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned int), s));
    int* done = a.flags.get();
    int* singular = a.flags.get() + 1;
    for (size_t l = 0; l + 1 < L; ++l) {
        SymLevel& F = *a.sym[l];
        SymLevel& C = *a.sym[l + 1];
        const int64_t n = F.A.n;
        double* y = a.pw_yz.get();
        double* z = y + n;
        double* y1 = z + n;
        double* z1 = y1 + n;
        k_dinv<<<grid_for(n, 256), 256, 0, s>>>(n, F.diag.get(), F.A.x.get(), F.dinv.get(), F.sq.get(),
                                                F.x0.get(), y, z, st, done);
        UP3D_CHECK_LAUNCH();
        constexpr int PW_STEPS = 20;
        for (int it = 0; it < PW_STEPS; ++it) {
            launch_pw_step(n, F.A.nnz, F.A.p.get(), F.A.i.get(), F.A.x.get(), F.sq.get(),
                           F.has_skip ? F.skip.get() : nullptr, y, z, y1, z1, st, done, partial, counter,
                           it + 1 == PW_STEPS ? a.omega_dev.get() + l : nullptr, s);
            std::swap(y, y1);
            std::swap(z, z1);
        }
        k_prolong<<<grid_for(n, 16, (int64_t)148 * 64), 128, 0, s>>>(n, F.A.p.get(), F.A.i.get(), F.A.x.get(),
                                                                     F.amap.get(), F.self.get(), F.t.get(),
                                                                     F.dinv.get(), a.omega_dev.get() + l,
                                                                     F.P.p.get(), F.P.x.get());
        UP3D_CHECK_LAUNCH();
        k_gather_vals<<<grid_for(F.R.nnz, 256), 256, 0, s>>>(F.R.nnz, F.tperm.get(), F.P.x.get(), F.R.x.get());
        UP3D_CHECK_LAUNCH();
        launch_spgemm(F.A, F.P, F.AP, F.ap_max, s);
        launch_spgemm(F.R, F.AP, C.A, C.a_max, s);
    }
    // coarsest dense inverse
    const SymLevel& Cl = *a.sym.back();
    const int64_t nc = Cl.A.n;
    UP3D_CUDA(cudaMemsetAsync(singular, 0, sizeof(int), s));
    if (!launch_gj(nc, Cl.A.p.get(), Cl.A.i.get(), Cl.A.x.get(), a.cinv.get(), a.gj_fac.get(), singular, s)) {
        // larger than a cluster holds: [A | I] in global memory, two
        // launches per column
        a.dense_a.alloc(nc * nc);
        a.fcol.alloc(nc);
        k_densify<<<grid_for(nc, 128), 128, 0, s>>>(nc, Cl.A.p.get(), Cl.A.i.get(), Cl.A.x.get(), a.dense_a.get(),
                                                    a.cinv.get());
        UP3D_CHECK_LAUNCH();
        for (int64_t c = 0; c < nc; ++c) {
            k_gj_pivot<<<1, 1024, 0, s>>>(a.dense_a.get(), a.cinv.get(), nc, c, a.fcol.get(), singular);
            UP3D_CHECK_LAUNCH();
            k_gj_elim<<<grid_for(2 * nc * nc, 256), 256, 0, s>>>(a.dense_a.get(), a.cinv.get(), nc, c, a.fcol.get(),
                                                                 singular);
            UP3D_CHECK_LAUNCH();
        }
    }
    int sing = 0;
    UP3D_CUDA(cudaMemcpyAsync(&sing, singular, sizeof(int), cudaMemcpyDeviceToHost, s));
    UP3D_CUDA(cudaStreamSynchronize(s));
    if (sing) {
        // singular coarse operator (e.g. pure-Neumann): regularise the
        // diagonal and invert on the host
        HostCSR h;
        h.n = h.m = nc;
        h.p.resize(nc + 1);
        h.i.resize(Cl.A.nnz);
        h.x.resize(Cl.A.nnz);
        UP3D_CUDA(cudaMemcpyAsync(h.p.data(), Cl.A.p.get(), sizeof(int32_t) * (nc + 1), cudaMemcpyDeviceToHost, s));
        UP3D_CUDA(cudaMemcpyAsync(h.i.data(), Cl.A.i.get(), sizeof(int32_t) * Cl.A.nnz, cudaMemcpyDeviceToHost, s));
        UP3D_CUDA(cudaMemcpyAsync(h.x.data(), Cl.A.x.get(), sizeof(double) * Cl.A.nnz, cudaMemcpyDeviceToHost, s));
        UP3D_CUDA(cudaStreamSynchronize(s));
        std::vector<double> dense(nc * nc, 0.0), inv;
        double dmax = 0.0;
        for (int64_t r = 0; r < nc; ++r)
            for (int32_t k = h.p[r]; k < h.p[r + 1]; ++k) {
                dense[r * nc + h.i[k]] = h.x[k];
                if (h.i[k] == r) dmax = std::max(dmax, std::fabs(h.x[k]));
            }
        for (int64_t r = 0; r < nc; ++r) dense[r * nc + r] += 1e-12 * (dmax > 0 ? dmax : 1.0);
        UP3D_REQUIRE(dense_inverse(dense, nc, inv), UP3D_ERR_RUNTIME, "AMG coarsest operator is singular");
        UP3D_CUDA(cudaMemcpyAsync(a.cinv.get(), inv.data(), sizeof(double) * nc * nc, cudaMemcpyHostToDevice, s));
        UP3D_CUDA(cudaStreamSynchronize(s));
    }
}

// Narrows the FP64 level values into the FP32 cycle (the FP64 cycle views
// them in place) and fills the slices.
template <class T>
void fill_levels(Amg& a, std::vector<Level<T>*>& Lv, cudaStream_t s) {
    for (size_t l = 0; l < a.sym.size(); ++l) {
        SymLevel& F = *a.sym[l];
        Level<T>& lv = *Lv[l];
        if (lv.sell_p) {
            k_sell_values<T><<<grid_for(F.A.n, 256), 256, 0, s>>>(F.A.n, F.A.p.get(), F.A.x.get(), lv.sell_p,
                                                                  lv.sell_x.get());
            UP3D_CHECK_LAUNCH();
        } else if constexpr (!std::is_same<T, double>::value) {
            convert<T>(F.A.x.get(), lv.A.x.get(), F.A.nnz, s);
        }
        if (l + 1 < a.sym.size()) {
            if constexpr (!std::is_same<T, double>::value) {
                convert<T>(F.P.x.get(), lv.P.x.get(), F.P.nnz, s);
                convert<T>(F.R.x.get(), lv.R.x.get(), F.R.nnz, s);
                convert<T>(F.dinv.get(), lv.dinv.get(), F.A.n, s);
            }
        }
    }
}

template <class T>
void view(CsrRef<T>& r, const DevCSR<double>& F, DBuf<T>& own) {
    r.n = F.n;
    r.m = F.m;
    r.nnz = F.nnz;
    r.p.v = F.p.get();
    r.i.v = F.i.get();
    if constexpr (std::is_same<T, double>::value) {
        r.x.v = F.x.get();
    } else {
        own.alloc(std::max<int64_t>(F.nnz, 1));
        r.x.v = own.get();
    }
}

template <class T>
void make_levels(Amg& a, std::vector<Level<T>*>& Lv, cudaStream_t s) {
    for (size_t l = 0; l < a.sym.size(); ++l) {
        SymLevel& F = *a.sym[l];
        auto* lv = new Level<T>();
        Lv.push_back(lv);
        const int64_t n = F.A.n;
        if (F.sell_n && l + 1 < a.sym.size()) {
            lv->A.n = lv->A.m = n;
            lv->A.nnz = F.A.nnz;
            lv->sell_p = F.sell_p.get();
            lv->sell_i = F.sell_i.get();
            lv->sell_x.alloc(F.sell_n);
        } else {
            view(lv->A, F.A, lv->own_A);
        }
        lv->x.alloc(n);
        lv->b.alloc(n);
        lv->r.alloc(n);
        if (l + 1 < a.sym.size()) {
            lv->omega = a.omega_dev.get() + l;
            view(lv->P, F.P, lv->own_P);
            view(lv->R, F.R, lv->own_R);
            if constexpr (std::is_same<T, double>::value) {
                lv->dinv.v = F.dinv.get();
            } else {
                lv->own_dinv.alloc(n);
                lv->dinv.v = lv->own_dinv.get();
            }
        }
    }
}

__global__ void k_diff_i32(int64_t n, const int32_t* __restrict__ a, const int32_t* __restrict__ b,
                           int* __restrict__ flag) {
    GRID_STRIDE(i, n) if (a[i] != b[i]) *flag = 1;
}
__global__ void k_diff_u8(int64_t n, const uint8_t* __restrict__ a, const uint8_t* __restrict__ b,
                          int* __restrict__ flag) {
    GRID_STRIDE(i, n) if ((a[i] != 0) != (b[i] != 0)) *flag = 1;
}

}  // namespace

template <class A, class B>
static void convert_copy(const A* src, B* dst, int64_t n, cudaStream_t s) {
    if constexpr (std::is_same<A, B>::value) {
        UP3D_CUDA(cudaMemcpyAsync(dst, src, sizeof(A) * n, cudaMemcpyDeviceToDevice, s));
    } else {
        if constexpr (std::is_same<A, double>::value) k_d2f<<<grid_for(n, 256), 256, 0, s>>>(src, dst, n);
        else k_f2d<<<grid_for(n, 256), 256, 0, s>>>(src, dst, n);
        UP3D_CHECK_LAUNCH();
    }
}

// Captures the body of the cycle at precision T.
template <class T>
static void capture_body(Amg& a, std::vector<Level<T>*>& L, Amg::Body& body) {
    if (!a.capture_stream) UP3D_CUDA(cudaStreamCreateWithFlags(&a.capture_stream, cudaStreamNonBlocking));
    // the levels' buffers swap between sweeps: put back afterwards
    std::vector<std::pair<T*, T*>> saved;
    for (auto* l : L) saved.emplace_back(l->x.p, l->r.p);
    auto restore = [&] {
        for (size_t i = 0; i < L.size(); ++i) {
            L[i]->x.p = saved[i].first;
            L[i]->r.p = saved[i].second;
        }
    };
    std::unique_lock<std::mutex> capturing(capture_mutex());   // no buffer is made or freed meanwhile
    const long long l0 = g_launches.load();
    cudaGraph_t graph = nullptr;
    UP3D_CUDA(cudaStreamBeginCapture(a.capture_stream, cudaStreamCaptureModeThreadLocal));
    try {
        vcycle<T>(a, L, 0, true, a.capture_stream);
    } catch (...) {
        cudaStreamEndCapture(a.capture_stream, &graph);
        if (graph) cudaGraphDestroy(graph);
        restore();
        throw;
    }
    body.x = L[0]->x.p;
    restore();
    UP3D_CUDA(cudaStreamEndCapture(a.capture_stream, &graph));
    capturing.unlock();
    body.launches = g_launches.load() - l0;
    g_launches.fetch_sub(body.launches);  // counted at each replay instead
    cudaGraphExec_t exec = nullptr;
    const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    UP3D_CUDA(e);
    body.exec = exec;
}

// One V-cycle z = M r at precision T on stream s.
template <class T, class TIO>
static void apply_cycle(Amg& a, std::vector<Level<T>*>& L, Amg::Body& body, const TIO* r, TIO* z, cudaStream_t s) {
    Level<T>& f = *L[0];
    const int64_t n = f.A.n;
    if (L.size() == 1) {   // the dense solve alone
        convert_copy(r, f.b.get(), n, s);
        launch_kernel(false, k_dense_solve<T>, grid_for(32 * n, 256), 256, s, a.cinv.get(), n, f.b.get(), f.x.get());
        convert_copy(f.x.get(), z, n, s);
        return;
    }
    if (!body.exec) capture_body<T>(a, L, body);
    launch_kernel(false, k_jacobi_first<T, TIO>, grid_for(n, 256), 256, s, f.dinv.get(), r, f.b.get(), f.x.get(),
                  f.omega, n);
    UP3D_CUDA(cudaGraphLaunch(body.exec, s));
    count_launch((int)body.launches);
    const T* x = static_cast<const T*>(body.x);
    if (a.post == 0) {
        convert_copy(x, z, n, s);
        return;
    }
    smooth<T, false>(false, f, x, z, s);   // in the caller's precision: a conversion behind it is 2 us of a small cycle
}

void amg_apply(void* p, const double* r, double* z, cudaStream_t s) {
    Amg& a = *static_cast<Amg*>(p);
    if (a.fp64) apply_cycle<double>(a, a.Ld, a.body64, r, z, s);
    else apply_cycle<float>(a, a.Lf, a.body32, r, z, s);
}

void amg_apply_f32(void* p, const float* r, float* z, cudaStream_t s) {
    Amg& a = *static_cast<Amg*>(p);
    if (a.fp32) apply_cycle<float>(a, a.Lf, a.body32, r, z, s);
    else apply_cycle<double>(a, a.Ld, a.body64, r, z, s);
}

void amg_destroy(void* p) { delete static_cast<Amg*>(p); }

// Builds the hierarchy for `A` (device CSR); the finest operator's
// constrained rows (A->dirichlet) are identity rows.
void* amg_setup(const up3d_csr& A, const up3d_amg_options& opt, cudaStream_t s) {
    auto* a = new Amg();
    try {
        // 0: FP64 cycle, 1: FP32 cycle, 2: both (each vector type gets its own)
        UP3D_REQUIRE(opt.fp32 >= 0 && opt.fp32 <= 2, UP3D_ERR_VALUE, "AMG setup: fp32 must be 0, 1 or 2");
        a->fp32 = opt.fp32 != 0;
        a->fp64 = opt.fp32 != 1;
        a->pre = std::max(1, opt.presmooth);
        a->post = std::max(0, opt.postsmooth);
        const int64_t n = A.n;
        UP3D_REQUIRE(n > 0, UP3D_ERR_VALUE, "AMG setup: empty matrix");
        const int64_t nnz = read_back(A.indptr + n, s);
        std::vector<uint8_t> skip(n, 0);
        if (A.dirichlet)
            UP3D_CUDA(cudaMemcpyAsync(skip.data(), A.dirichlet, n, cudaMemcpyDeviceToHost, s));
        UP3D_CUDA(cudaStreamSynchronize(s));
        for (auto& v : skip) v = v != 0;
        // the caller's pattern, kept for refresh checks
        a->n_in = n;
        a->nnz_in = nnz;
        a->has_dir = A.dirichlet != nullptr;
        a->in_p.alloc(n + 1);
        a->in_i.alloc(std::max<int64_t>(nnz, 1));
        UP3D_CUDA(cudaMemcpyAsync(a->in_p.get(), A.indptr, sizeof(int32_t) * (n + 1), cudaMemcpyDeviceToDevice, s));
        if (nnz)
            UP3D_CUDA(cudaMemcpyAsync(a->in_i.get(), A.indices, sizeof(int32_t) * nnz, cudaMemcpyDeviceToDevice, s));
        if (a->has_dir) upload(a->in_dir, skip, s);
        // finest operator as the embedded free-DOF system: identity rows,
        // constrained columns dropped; src = caller entry (-1: identity).
        // Formed on the device, the host reads the pattern it works on
        // (9.4 M entries: formed on the host, with the caller's pattern read
        // and two arrays sent, 20-40 ms of a set-up; so 5-14)
        auto* F0 = new SymLevel();
        a->sym.push_back(F0);
        const uint8_t* dir = a->has_dir ? a->in_dir.get() : nullptr;
        HostCSR e;
        e.n = e.m = n;
        e.p.resize(n + 1);
        F0->A.p.alloc(n + 1);
        k_embed_count<<<grid_for(n, 32, (int64_t)148 * 64), 256, 0, s>>>(n, a->in_p.get(), a->in_i.get(), dir,
                                                                       F0->A.p.get());
        UP3D_CHECK_LAUNCH();
        d2h(e.p.data(), F0->A.p.get(), sizeof(int32_t) * (n + 1), s);
        for (int64_t r = 0; r < n; ++r) e.p[r + 1] += e.p[r];
        F0->A.n = F0->A.m = n;
        F0->A.nnz = e.p[n];
        F0->A.i.alloc(std::max<int64_t>(e.p[n], 1));
        F0->A.x.alloc(std::max<int64_t>(e.p[n], 1));
        a->emb_src.alloc(std::max<int64_t>(e.p[n], 1));
        h2d(F0->A.p.get(), e.p.data(), sizeof(int32_t) * (n + 1), s);
        k_embed_fill<<<grid_for(n, 32, (int64_t)148 * 64), 256, 0, s>>>(n, a->in_p.get(), a->in_i.get(), dir,
                                                                      F0->A.p.get(), F0->A.i.get(), a->emb_src.get());
        UP3D_CHECK_LAUNCH();
        e.i.resize(e.p[n]);
        if (e.p[n]) d2h(e.i.data(), F0->A.i.get(), sizeof(int32_t) * e.p[n], s);
        // symbolic levels
        std::vector<HostCSR> As;
        As.push_back(std::move(e));
        std::vector<uint8_t> cur_skip = skip;
        const int64_t max_coarse = std::max<int64_t>(opt.max_coarse, 1);
        int64_t nmax = n;
        while (true) {
            const HostCSR& Al = As.back();
            if (As.size() > 1) {
                a->sym.push_back(new SymLevel());
                a->sym.back()->A.upload_pattern(Al, s);
            }
            SymLevel* F = a->sym.back();
            F->a_max = longest_row(Al);
            make_slices(*F, Al, s);
            upload(F->diag, diag_slots(Al), s);
            F->has_skip = a->sym.size() == 1 && a->has_dir;
            if (F->has_skip) upload(F->skip, cur_skip, s);
            F->dinv.alloc(Al.n);
            F->sq.alloc(Al.n);
            if (Al.n <= max_coarse || (int)As.size() >= std::max(2, opt.max_levels)) break;
            std::vector<int32_t> agg;
            const int64_t na = standard_aggregation(Al, cur_skip, agg);
            if (na == 0 || na >= Al.n) break;
            upload(F->x0, power_start(Al.n, cur_skip), s);
            std::vector<int32_t> amap, self, tperm;
            HostCSR P = prolongator_pattern(Al, agg, na, amap, self);
            std::vector<int32_t> size(na, 0);
            for (int64_t r = 0; r < Al.n; ++r)
                if (agg[r] >= 0) size[agg[r]]++;
            std::vector<double> t(Al.n, 0.0);
            for (int64_t r = 0; r < Al.n; ++r)
                if (agg[r] >= 0) t[r] = 1.0 / std::sqrt((double)size[agg[r]]);
            HostCSR R = transpose_pattern(P, tperm);
            HostCSR AP = spgemm_pattern(Al, P);
            HostCSR Ac = spgemm_pattern(R, AP);
            upload(F->amap, amap, s);
            upload(F->self, self, s);
            upload(F->t, t, s);
            upload(F->tperm, tperm, s);
            F->P.upload_pattern(P, s);
            F->R.upload_pattern(R, s);
            F->AP.upload_pattern(AP, s);
            F->ap_max = longest_row(AP);
            UP3D_CUDA(cudaStreamSynchronize(s));  // host vectors above go out of scope
            As.push_back(std::move(Ac));
            cur_skip.assign(As.back().n, 0);
        }
        // a level that stopped early without a start vector is the coarsest
        const int64_t nc = As.back().n;
        UP3D_REQUIRE(nc <= 8192, UP3D_ERR_RUNTIME, "AMG coarsest level too large for the dense solve");
        a->n_coarse = nc;
        a->pw_yz.alloc(4 * nmax);
        a->pw_scal.alloc(2 + 3 * PW_BLOCKS);
        a->omega_dev.alloc(std::max<size_t>(a->sym.size(), 1));
        a->flags.alloc(3);
        a->cinv.alloc(nc * nc);
        a->gj_fac.alloc(gj_fac_size(nc));
        k_embed<<<grid_for(a->sym[0]->A.nnz, 256), 256, 0, s>>>(a->sym[0]->A.nnz, a->emb_src.get(), A.data,
                                                                a->sym[0]->A.x.get());
        UP3D_CHECK_LAUNCH();
        numeric(*a, s);
        if (a->fp32) {
            make_levels<float>(*a, a->Lf, s);
            fill_levels<float>(*a, a->Lf, s);
        }
        if (a->fp64) {
            make_levels<double>(*a, a->Ld, s);
            fill_levels<double>(*a, a->Ld, s);
        }
        UP3D_CUDA(cudaStreamSynchronize(s));
        a->info.n_levels = (int32_t)As.size();
        int64_t tot = 0;
        for (auto& M : As) tot += (int64_t)M.i.size();
        a->info.operator_complexity = (double)tot / (double)std::max<size_t>(As[0].i.size(), 1);
        a->info.n_coarse = nc;
        for (size_t l = 0; l < As.size() && l < 16; ++l) a->info.level_rows[l] = As[l].n;
    } catch (...) {
        delete a;
        throw;
    }
    return a;
}

// New values for the hierarchy: `A` must have the pattern and Dirichlet
// mask of the matrix the hierarchy was set up from.
void amg_refresh(void* p, const up3d_csr& A, cudaStream_t s) {
    Amg& a = *static_cast<Amg*>(p);
    UP3D_REQUIRE(A.n == a.n_in, UP3D_ERR_VALUE, "AMG refresh: matrix size differs from the setup matrix");
    UP3D_REQUIRE((A.dirichlet != nullptr) == a.has_dir, UP3D_ERR_VALUE,
                 "AMG refresh: Dirichlet mask presence differs from the setup matrix");
    int* flag = a.flags.get();
    UP3D_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), s));
    k_diff_i32<<<grid_for(a.n_in + 1, 256), 256, 0, s>>>(a.n_in + 1, A.indptr, a.in_p.get(), flag);
    UP3D_CHECK_LAUNCH();
    int diff = 0;
    UP3D_CUDA(cudaMemcpyAsync(&diff, flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    UP3D_CUDA(cudaStreamSynchronize(s));
    UP3D_REQUIRE(!diff, UP3D_ERR_VALUE, "AMG refresh: sparsity pattern differs from the setup matrix");
    k_diff_i32<<<grid_for(a.nnz_in, 256), 256, 0, s>>>(a.nnz_in, A.indices, a.in_i.get(), flag);
    UP3D_CHECK_LAUNCH();
    if (a.has_dir) {
        k_diff_u8<<<grid_for(a.n_in, 256), 256, 0, s>>>(a.n_in, A.dirichlet, a.in_dir.get(), flag);
        UP3D_CHECK_LAUNCH();
    }
    UP3D_CUDA(cudaMemcpyAsync(&diff, flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    UP3D_CUDA(cudaStreamSynchronize(s));
    UP3D_REQUIRE(!diff, UP3D_ERR_VALUE, "AMG refresh: sparsity pattern or Dirichlet mask differs from the setup matrix");
    k_embed<<<grid_for(a.sym[0]->A.nnz, 256), 256, 0, s>>>(a.sym[0]->A.nnz, a.emb_src.get(), A.data,
                                                           a.sym[0]->A.x.get());
    UP3D_CHECK_LAUNCH();
    numeric(a, s);
    if (a.fp32) fill_levels<float>(a, a.Lf, s);
    if (a.fp64) fill_levels<double>(a, a.Ld, s);
}

const up3d_amg_info* amg_info(void* p) { return &static_cast<Amg*>(p)->info; }

}  // namespace up3d

using namespace up3d;

extern "C" {

int up3d_amg_setup(const up3d_csr* A, const up3d_amg_options* opt, up3d_precond** out, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(A && out && A->indptr && A->indices && A->data, UP3D_ERR_ARGUMENT,
                     "up3d_amg_setup: null argument");
        up3d_amg_options o{10, 500, 2, 2, 0};
        if (opt) o = *opt;
        auto* M = new up3d_precond();
        M->kind = 2;
        M->n = A->n;
        try {
            M->amg = amg_setup(*A, o, S(stream));
        } catch (...) {
            delete M;
            throw;
        }
        *out = M;
    });
}

int up3d_amg_refresh(up3d_precond* M, const up3d_csr* A, up3d_stream stream) {
    return guarded([&] {
        UP3D_REQUIRE(M && A && M->kind == 2 && M->amg && A->indptr && A->indices && A->data, UP3D_ERR_ARGUMENT,
                     "up3d_amg_refresh: null argument or not an AMG handle");
        amg_refresh(M->amg, *A, S(stream));
    });
}

int up3d_amg_get_info(const up3d_precond* M, up3d_amg_info* info) {
    return guarded([&] {
        UP3D_REQUIRE(M && info && M->kind == 2 && M->amg, UP3D_ERR_ARGUMENT, "up3d_amg_get_info: not an AMG handle");
        *info = *amg_info(M->amg);
    });
}

}  // extern "C"
