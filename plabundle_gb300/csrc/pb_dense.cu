// pb_dense.cu -- dense Cholesky preconditioner and FP64 conjugate gradients for the reduced system.
//
// The reduced camera system of the online Schur path is small (6 x cameras + refined intrinsics)
// but badly conditioned: the focal-length / altitude mode of a nadir block gives a normalised
// condition number near 1e7, where block-Jacobi PCG needs thousands of iterations.  Here the
// Jacobi-scaled matrix Sn = D^-1/2 S D^-1/2 is factored densely (Sn + shift I = L L^T, blocked
// right-looking Cholesky on tiles of 64 in FP32, of 32 in FP64), L is inverted (X = L^-1), and
// M^-1 = D^-1/2 X^T X D^-1/2
// preconditions conjugate gradients whose matrix-vector products use the FP64 reduced matrix.
// On the mixed path the factor and inverse are FP32 with a small shift that keeps the FP32
// factorisation positive definite; the FP64 CG recovers the FP64 solution (it plays the role of
// iterative refinement).  On the FP64 path the factor is FP64 and CG converges in one or two
// iterations.  The factorisation with its inverse and the whole CG solve are each one persistent kernel
// whose phases are separated by barriers, with no host round trips: of one thread-block cluster for small
// systems, of a cooperative grid beyond.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <mutex>

#include "pb_device.cuh"
#include "pb_kernels.h"

namespace pb {

namespace cgk = cooperative_groups;

namespace {
constexpr int TS = 64;        // tile size
constexpr int TP = TS + 1;    // padded shared-memory row

__device__ __forceinline__ int tri_row(int idx) {
    // i such that i (i + 1) / 2 <= idx < (i + 1) (i + 2) / 2
    int i = static_cast<int>((sqrtf(8.0f * static_cast<float>(idx) + 1.0f) - 1.0f) * 0.5f);
    while ((i + 1) * (i + 2) / 2 <= idx) ++i;
    while (i * (i + 1) / 2 > idx) --i;
    return i;
}
}  // namespace

// d_i = 1 / sqrt(S_ii) of the FP64 reduced matrix (pose diagonal blocks, intrinsic block).
__global__ void k_dense_scale(PcgSystem<double> sys, double* __restrict__ dscale, int* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n6 = 6 * sys.ncb, n = n6 + sys.nb;
    if (i >= n) return;
    double d;
    if (i < n6) {
        const int b = i / 6, a = i - b * 6;
        d = sys.vals[static_cast<size_t>(sys.diag_pos[b]) * 36 + a * 7];
    } else {
        const int c = i - n6;
        d = sys.Cm[c * sys.nb + c];
    }
    if (!(d > 0.0) || !isfinite(d)) {
        atomicOr(status, 1);
        d = 1.0;
    }
    dscale[i] = 1.0 / sqrt(d);
}

// Scatter of the scaled reduced matrix into a dense row-major np x np array (both triangles).
template <typename T>
__global__ void k_dense_fill(PcgSystem<double> sys, const double* __restrict__ dscale, T* __restrict__ A, int np) {
    const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int n6 = 6 * sys.ncb, nb = sys.nb;
    const long long nblk = static_cast<long long>(sys.row_ptr[sys.ncb]) * 36;
    const long long nbor = static_cast<long long>(n6) * nb;
    if (idx < nblk) {
        const int e = static_cast<int>(idx / 36), r = static_cast<int>(idx - static_cast<long long>(e) * 36);
        int lo = 0, hi = sys.ncb;  // block row of CSR entry e
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (sys.row_ptr[mid] <= e) lo = mid;
            else hi = mid;
        }
        const int row = 6 * lo + r / 6, col = 6 * sys.col_idx[e] + r % 6;
        A[static_cast<size_t>(row) * np + col] = static_cast<T>(sys.vals[idx] * dscale[row] * dscale[col]);
    } else if (idx < nblk + nbor) {
        const long long k = idx - nblk;
        const int row = static_cast<int>(k / nb), c = static_cast<int>(k - static_cast<long long>(row) * nb);
        const T v = static_cast<T>(sys.border[k] * dscale[row] * dscale[n6 + c]);
        A[static_cast<size_t>(row) * np + n6 + c] = v;
        A[static_cast<size_t>(n6 + c) * np + row] = v;
    } else if (idx < nblk + nbor + static_cast<long long>(nb) * nb) {
        const int k = static_cast<int>(idx - nblk - nbor), a = k / nb, b = k - a * nb;
        A[static_cast<size_t>(n6 + a) * np + n6 + b] = static_cast<T>(sys.Cm[k] * dscale[n6 + a] * dscale[n6 + b]);
    }
}

// Diagonal shift of the scaled matrix (1 + shift) and identity on the padding.
template <typename T>
__global__ void k_dense_diag(T* __restrict__ A, int n, int np, double shift) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    T* d = A + static_cast<size_t>(i) * np + i;
    *d = i < n ? static_cast<T>(static_cast<double>(*d) + shift) : T(1);
}

// C (64x64) += A (64x64) * B (64x64): sA holds A row-major [r][k], sB holds B k-major [k][c];
// 256 threads, thread (ty, tx) owns rows ty + 16 m and columns tx + 16 m'.
__device__ __forceinline__ void tile_mma(const float* __restrict__ sA, const float* __restrict__ sB, float acc[4][4]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 8
    for (int kk = 0; kk < TS; ++kk) {
        float a[4], b[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            a[m] = sA[(ty + 16 * m) * TP + kk];
            b[m] = sB[kk * TP + tx + 16 * m];
        }
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[m][q] += a[m] * b[q];
    }
}

// Loads a global 64x64 tile (row stride np, 16-byte aligned rows) into shared memory, row-major
// or transposed, with 16-byte loads.
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    using type = float4;
    static constexpr int n = 4;
    __device__ static __forceinline__ float get(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
    __device__ static __forceinline__ float dot(const float4& a, const float4& b) {
        return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
    }
};
template <>
struct Vec16<double> {
    using type = double2;
    static constexpr int n = 2;
    __device__ static __forceinline__ double get(const double2& v, int i) { return i == 0 ? v.x : v.y; }
    __device__ static __forceinline__ double dot(const double2& a, const double2& b) { return a.x * b.x + a.y * b.y; }
};

template <bool TRANSPOSE>
__device__ __forceinline__ void tile_load(const float* __restrict__ g, int np, float* __restrict__ s) {
    using V = Vec16<float>;
    constexpr int per_row = TS / V::n;
    for (int e = threadIdx.x; e < TS * per_row; e += blockDim.x) {
        const int r = e / per_row, c0 = (e % per_row) * V::n;
        const typename V::type v = *reinterpret_cast<const typename V::type*>(g + static_cast<size_t>(r) * np + c0);
#pragma unroll
        for (int q = 0; q < V::n; ++q) {
            if (TRANSPOSE) s[(c0 + q) * TP + r] = V::get(v, q);
            else s[r * TP + c0 + q] = V::get(v, q);
        }
    }
}

// Lower-triangle elements of a 64x64 tile owned by this thread (up to 9 of 2080).
__device__ __forceinline__ int owned_elements(int* ii, int* ll) {
    int cnt = 0;
#pragma unroll
    for (int s = 0; s < 9; ++s) {
        const int e = threadIdx.x + 256 * s;
        if (e < TS * (TS + 1) / 2) {
            const int i = tri_row(e);
            ii[s] = i;
            ll[s] = e - i * (i + 1) / 2;
            ++cnt;
        } else {
            ii[s] = -1;
            ll[s] = -1;
        }
    }
    return cnt;
}

// Block 0 of step k: L_kk (written to A_kk, zeros above the diagonal) and D_k = L_kk^-1.
//
// The factorisation is the unscaled right-looking elimination (after step j, column j holds
// d_j * L_:j): every lower element (i, l) receives a_il = fma(-(a_ij a_lj), 1 / d_j, a_il) for
// j < l in increasing j (one rounding of the product, one of the update, in every phase).  It runs in
// eight panels of eight columns: three warps take the rows of a panel, a lane per row with its eight
// columns in registers (lanes 0-7 of each hold the panel's own rows, so that the pivot entries come by
// shuffle and no warp waits for another), then every thread applies the panel's eight steps, in order,
// to its elements of the trailing block.  Each element sees the same updates in the same order as a
// column-by-column elimination.  (Against panels of sixteen columns, their own block on one warp and the
// rows below it after a barrier: 354 unknowns 239 -> 220 us a factorisation, 114 unknowns 109 -> 94.)  The
// inverse R = L^-1 (R = I, R_ic -= L_ij R_jc / L_jj for i > j >= c, then R_ic / L_ii) is independent per
// column: four lanes own a column (rows split mod 4, held in registers) and pass row j between them by
// shuffle, with no block barrier.
__device__ void diag_factor_inverse(float* __restrict__ A, float* __restrict__ Dinv, int np, int k, float* sA,
                                    float* sB, int* __restrict__ status) {
    float* Akk = A + static_cast<size_t>(k) * TS * np + static_cast<size_t>(k) * TS;
    tile_load<false>(Akk, np, sA);
    int ii[9], ll[9];
    owned_elements(ii, ll);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ float s_inv[TS];  // 1 / d_j of the elimination, then 1 / L_jj of the inverse
    constexpr int PW = 8;    // panel width
    __syncthreads();
    for (int c0 = 0; c0 < TS; c0 += PW) {
        // (a) the panel: row c0 + lane for lanes 0-7, then 24 of the rows below per warp
        const int below = TS - c0 - PW;
        float a[PW];
        const int i = lane < PW ? c0 + lane : c0 + PW + 24 * warp + lane - PW;
        const bool mine = i < TS;
        if (warp < max(1, (below + 23) / 24)) {
#pragma unroll
            for (int l = 0; l < PW; ++l) a[l] = mine ? sA[i * TP + c0 + l] : 0.f;
            // (no branch in the chain of pivots: the marks and reciprocals are written after it)
            bool bad = false;
            float my_inv = 0.f;
#pragma unroll
            for (int j = 0; j < PW; ++j) {
                const float d = __shfl_sync(0xffffffffu, a[j], j);
                const bool pos = d > 0.f;
                const float inv = __frcp_rn(pos ? d : 1.f) * (pos ? 1.f : 0.f);
                bad |= !pos;
                if (lane == j) my_inv = inv;
                const float aij = a[j];
#pragma unroll
                for (int l = j + 1; l < PW; ++l) {
                    const float alj = __shfl_sync(0xffffffffu, aij, l);
                    a[l] = fma(-(aij * alj), inv, a[l]);
                }
            }
            if (warp == 0) {
                if (lane < PW) s_inv[c0 + lane] = my_inv;
                if (lane == 0 && bad) atomicOr(status, 2);
            }
            if (mine && lane >= PW)
#pragma unroll
                for (int l = 0; l < PW; ++l) sA[i * TP + c0 + l] = a[l];
        }
        __syncthreads();
        // the panel's own rows, from warp 0, once every warp has read them (the trailing block does not;
        // entries above the diagonal are not read again)
        if (warp == 0 && lane < PW)
#pragma unroll
            for (int l = 0; l < PW; ++l) sA[i * TP + c0 + l] = a[l];
        // (b) the trailing block: elements (r, l), c0 + 8 <= l <= r < 64, the panel's steps in order; a lane
        // per column (and the column 32 to the right), a warp every eighth row
        {
            float inv[PW], t0[PW], t1[PW];
            const int l0 = c0 + PW + lane, l1 = l0 + 32;
#pragma unroll
            for (int j = 0; j < PW; ++j) {
                inv[j] = s_inv[c0 + j];
                t0[j] = l0 < TS ? sA[l0 * TP + c0 + j] : 0.f;
                t1[j] = l1 < TS ? sA[l1 * TP + c0 + j] : 0.f;
            }
            for (int r = c0 + PW + warp; r < TS; r += 8) {
                float rj[PW];
#pragma unroll
                for (int j = 0; j < PW; ++j) rj[j] = sA[r * TP + c0 + j];
                if (l0 <= r) {
                    float x = sA[r * TP + l0];
#pragma unroll
                    for (int j = 0; j < PW; ++j) x = fma(-(rj[j] * t0[j]), inv[j], x);
                    sA[r * TP + l0] = x;
                }
                if (l1 <= r) {
                    float x = sA[r * TP + l1];
#pragma unroll
                    for (int j = 0; j < PW; ++j) x = fma(-(rj[j] * t1[j]), inv[j], x);
                    sA[r * TP + l1] = x;
                }
            }
        }
        __syncthreads();
    }
    float v[9];
#pragma unroll
    for (int s = 0; s < 9; ++s) {
        if (ii[s] < 0) continue;
        const float d = sA[ll[s] * TP + ll[s]];
        const float sd = d > 0.f ? sqrt(d) : 1.f;
        v[s] = ii[s] == ll[s] ? sd : sA[ii[s] * TP + ll[s]] / sd;
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 9; ++s) {
        if (ii[s] < 0) continue;
        sA[ii[s] * TP + ll[s]] = v[s];
        if (ii[s] != ll[s]) sA[ll[s] * TP + ii[s]] = 0.f;
    }
    __syncthreads();
    // 1 / L_jj once per row for the inverse
    if (threadIdx.x < TS) s_inv[threadIdx.x] = 1.f / sA[threadIdx.x * TP + threadIdx.x];
    __syncthreads();
    {
        // column c = 8 warp + lane / 4; this lane holds rows i = part + 4 q
        const int c = 8 * warp + (lane >> 2), part = lane & 3;
        float r[TS / 4];
#pragma unroll
        for (int q = 0; q < TS / 4; ++q) r[q] = part + 4 * q == c ? 1.f : 0.f;
#pragma unroll
        for (int j = 0; j < TS; ++j) {
            // row j of the column, final from the steps before j, from the lane that holds it
            const float rj = __shfl_sync(0xffffffffu, r[j >> 2], (lane & ~3) | (j & 3));
            if (8 * warp <= j) {  // some column of this warp has c <= j
                const float inv = s_inv[j];
#pragma unroll
                for (int q = 0; q < TS / 4; ++q) {
                    if (4 * q + 3 <= j) continue;  // every row of this slot is <= j
                    const int i = part + 4 * q;
                    if (i > j && c <= j) r[q] = fma(-(sA[i * TP + j] * rj), inv, r[q]);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < TS / 4; ++q) sB[(part + 4 * q) * TP + c] = r[q];
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 9; ++s)
        if (ii[s] >= 0) v[s] = sB[ii[s] * TP + ll[s]] / sA[ii[s] * TP + ii[s]];
    __syncthreads();
    float* D = Dinv + static_cast<size_t>(k) * TS * TS;
    for (int e = threadIdx.x; e < TS * TS; e += blockDim.x) {
        const int r = e / TS, c = e % TS;
        Akk[static_cast<size_t>(r) * np + c] = sA[r * TP + c];
        D[e] = 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 9; ++s)
        if (ii[s] >= 0) D[ii[s] * TS + ll[s]] = v[s];
}

// C = (accumulate ? C : 0) + alpha * sA sB over one 64x64 tile (row stride ldc).
__device__ __forceinline__ void tile_product_store(float* __restrict__ C, int ldc, const float* sA, const float* sB,
                                                   float alpha, bool accumulate) {
    float acc[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[m][q] = 0.f;
    tile_mma(sA, sB, acc);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float* c = C + static_cast<size_t>(ty + 16 * m) * ldc + tx + 16 * q;
            *c = accumulate ? *c + alpha * acc[m][q] : alpha * acc[m][q];
        }
}

// Barrier between the phases of a cooperative kernel: of the whole grid, or, for grids of at most sixteen
// blocks, which one cluster holds, of the cluster (114 unknowns: FP32 factor 94 -> 90 us, FP64 factor 145 ->
// 139).  Either barrier orders the blocks' writes to global memory.
constexpr int kClusterMax = 16;
template <bool CLUSTER>
__device__ __forceinline__ void phase_barrier() {
    if constexpr (CLUSTER) cgk::this_cluster().sync();
    else cgk::this_grid().sync();
}

template <bool CLUSTER>
__global__ void __launch_bounds__(256) k_potrf_coop(float* __restrict__ A, float* __restrict__ X,
                                                   float* __restrict__ Dinv, int np, int nt, int* __restrict__ status,
                                                   int* __restrict__ host_status) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* sA = reinterpret_cast<float*>(smem_raw);
    float* sB = sA + TS * TP;
    auto tile = [np](float* M, int i, int j) { return M + static_cast<size_t>(i) * TS * np + static_cast<size_t>(j) * TS; };
    // X = I
    for (int r = blockIdx.x; r < np; r += gridDim.x)
        for (int c = threadIdx.x; c < np; c += blockDim.x) X[static_cast<size_t>(r) * np + c] = r == c ? 1.f : 0.f;
    phase_barrier<CLUSTER>();
    if (blockIdx.x == 0) diag_factor_inverse(A, Dinv, np, 0, sA, sB, status);
    phase_barrier<CLUSTER>();
    for (int k = 0; k < nt; ++k) {
        const int m = nt - 1 - k;
        const float* Dk = Dinv + static_cast<size_t>(k) * TS * TS;
        for (int it = blockIdx.x; it < m + k + 1; it += gridDim.x) {
            if (it < m) {
                // L_ik = A_ik D_k^T
                float* Aik = tile(A, k + 1 + it, k);
                tile_load<false>(Aik, np, sA);
                tile_load<true>(Dk, TS, sB);
                __syncthreads();
                tile_product_store(Aik, np, sA, sB, 1.f, false);
            } else {
                // X_kj = D_k R_kj
                float* Xkj = tile(X, k, it - m);
                tile_load<false>(Dk, TS, sA);
                tile_load<false>(Xkj, np, sB);
                __syncthreads();
                tile_product_store(Xkj, np, sA, sB, 1.f, false);
            }
            __syncthreads();
        }
        phase_barrier<CLUSTER>();
        // Trailing update and R update.  Item 0 is the next diagonal tile (k+1, k+1): block 0
        // updates it and factors it at once (lookahead), while the other blocks share the rest.
        const int ntrail = m * (m + 1) / 2;
        const int nitems = ntrail + m * (k + 1);
        const int first_it = blockIdx.x == 0 ? 0 : (gridDim.x > 1 ? blockIdx.x : 1);
        const int stride = gridDim.x > 1 ? static_cast<int>(gridDim.x) - 1 : 1;
        for (int it = first_it; it < nitems; it = (it == 0 && gridDim.x > 1) ? nitems : it + stride) {
            if (it < ntrail) {
                // A_ij -= L_ik L_jk^T
                const int t = tri_row(it);
                const int i = k + 1 + t, j = k + 1 + (it - t * (t + 1) / 2);
                tile_load<false>(tile(A, i, k), np, sA);
                tile_load<true>(tile(A, j, k), np, sB);
                __syncthreads();
                tile_product_store(tile(A, i, j), np, sA, sB, -1.f, true);
            } else {
                // R_ij -= L_ik X_kj
                const int q = it - ntrail;
                const int i = k + 1 + q / (k + 1), j = q % (k + 1);
                tile_load<false>(tile(A, i, k), np, sA);
                tile_load<false>(tile(X, k, j), np, sB);
                __syncthreads();
                tile_product_store(tile(X, i, j), np, sA, sB, -1.f, true);
            }
            __syncthreads();
            if (it == 0 && m > 0) {
                // tile (k+1, k+1) is final: factor it for the next step
                __threadfence_block();
                diag_factor_inverse(A, Dinv, np, k + 1, sA, sB, status);
            }
        }
        phase_barrier<CLUSTER>();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *host_status = __ldcg(status);
    // X^T into the upper triangle of A (tile (j, i) = X_ij^T, j <= i).  The preconditioner is
    // applied as X^T (X u): forming X^T X explicitly in the factor's precision would square the
    // condition number of its rounding error.
    for (int it = blockIdx.x; it < nt * (nt + 1) / 2; it += gridDim.x) {
        const int i = tri_row(it), j = it - i * (i + 1) / 2;
        tile_load<true>(tile(X, i, j), np, sA);
        __syncthreads();
        float* dst = tile(A, j, i);
        for (int e = threadIdx.x; e < TS * TS; e += blockDim.x) {
            const int r = e / TS, c = e % TS;
            dst[static_cast<size_t>(r) * np + c] = sA[r * TP + c];
        }
        __syncthreads();
    }
}

// ---- FP64 factorisation: 32 x 32 tiles
// A warp-wide FP64 FMA takes 64 cycles of a sub-partition, so a 64 x 64 x 64 tile product keeps an SM
// busy for 63 us and a system of a few hundred unknowns spends its time on a few SMs, one step after
// another.  Tiles of 32 cut a product to 8 us (4 where one factor is triangular, with the rows or
// columns of a warp chosen so that every warp sums 66 products) and spread the same work over four
// times as many SMs; the diagonal tile's chain (below) is a quarter of the 64 x 64 one.  A whole FP64
// step, of which this is the largest part: 114 unknowns 811 -> 451 us, 600 unknowns 3.56 -> 1.71 ms, 1216
// unknowns 9.8 -> 4.5 ms, 3010 unknowns 29.5 -> 20.6 ms (the FP64 pipes of all SMs are the bound there).
// The FP32 factor keeps its tiles of 64: its products are cheap and fewer steps cost fewer barriers.
namespace {
constexpr int TD = 32, TDP = TD + 1;
constexpr int kPotrf64Threads = 256;
constexpr size_t kPotrf64Smem = (4 * static_cast<size_t>(TD) * TDP + TD * 9 + 3 * TD) * sizeof(double);
}  // namespace

constexpr int kPanel = 4;

// (out of line: not on the way of the ordinary pivots)
__device__ __noinline__ double other_quotient(double a, double d) { return d > 0.0 ? a / d : 0.0; }
__device__ __noinline__ double other_sqrt(double d) { return d > 0.0 ? sqrt(d) : 1.0; }

// Inverse of the 8 x 8 diagonal block b of the tile's factor from its unscaled columns, by one warp
// (lane c < 8 a column): with L_ik = a_ik rs_k and z_k = rs_k x_k, x_i = -rs_i sum_k a_ik z_k.
__device__ __forceinline__ void inverse8(const double* sC, double* sX, const double* s_d, double* s_sd, double* s_rs,
                                         int b) {
    const int lane = threadIdx.x & 31, c = lane & 7, o = 8 * b;
    const double d = s_d[o + c];
    double sd, rs;
    if (plain_pivot(d)) {
        plain_roots(d, sd, rs);
    } else {
        sd = other_sqrt(d);
        rs = other_quotient(1.0, sd);
    }
    if (lane < 8) {
        s_sd[o + c] = sd;
        s_rs[o + c] = rs;
    }
    const double r2 = rs * rs;
    double below[28], ri[8], ri2[8];  // the block below its diagonal by columns; all lanes' rs and r2
#pragma unroll
    for (int i = 0, q = 0; i < 8; ++i) {
        ri[i] = __shfl_sync(0xffffffffu, rs, i);
        ri2[i] = __shfl_sync(0xffffffffu, r2, i);
#pragma unroll
        for (int l = i + 1; l < 8; ++l, ++q) below[q] = sC[(o + l) * TDP + o + i];
    }
    double t[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // sum_k a_ik z_k, grown column by column
#pragma unroll
    for (int i = 0, q = 0; i < 8; ++i) {
        const double z = i == c ? ri2[i] : -ri2[i] * t[i];  // (t is zero above the diagonal)
#pragma unroll
        for (int l = i + 1; l < 8; ++l, ++q) t[l] = fma(below[q], z, t[l]);
    }
    if (lane < 8)
#pragma unroll
        for (int i = 0; i < 8; ++i) sX[(o + i) * TDP + o + c] = i == c ? ri[i] : -ri[i] * t[i];
}

// The diagonal tile in sC (lower triangle), less L L^T of the tile left of it when sL holds L^T: L_kk into A
// (zeros above the diagonal) and D_k = L_kk^-1 into Dinv.  A dependent FP64 instruction takes 70 cycles, and
// a column is four of them, the next column's update and shuffles, about 470 cycles, so that
// warp 0 does nothing but the columns: panels of four, a lane per row with the columns in registers, where
// it also applies the panel before.  Meanwhile the other warps apply the panel before to the columns behind
// the current one, subtract L L^T from the columns that come up two panels later (these sums are the
// largest part of the tile's work, and an SM takes 16 cycles for any FP64 instruction of a warp), and warp
// 1 inverts the finished 8 x 8 blocks.  (A panel, its update of the rest and so on, after L L^T as a whole:
// 66 000 cycles a tile, this 50 000; an FP64 step's solve,
// with the panels' products shared by four blocks: 114 unknowns 208 -> 187 us, 380 unknowns 522 -> 450, 610
// unknowns 925 -> 700, 1 210 unknowns 1 980 -> 1 700.)  The square roots come once at the end, and the inverse grows
// from the 8 x 8 blocks by doubling: X21 = -X22 (L21 X11).
__device__ void diag_factor_inverse64(double* __restrict__ Akk, int np, double* __restrict__ D, const double* sL, double* sC,
                                      double* sX, double* sP, double* sT, double* s_d, int* __restrict__ status) {
    double* s_sd = s_d + TD;
    double* s_rs = s_sd + TD;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (sL && warp < kPanel && lane >= warp) {  // columns 0 .. 3: a warp per column
        double v = sC[lane * TDP + warp];
#pragma unroll 8
        for (int l = 0; l < TD; ++l) v = fma(-sL[l * TDP + lane], sL[l * TDP + warp], v);
        sC[lane * TDP + warp] = v;
    }
    for (int e = tid; e < TD * TDP; e += kPotrf64Threads) sX[e] = 0.0;
    __syncthreads();
    double tp[kPanel], ap[kPanel];  // warp 0: the panel before, multipliers and columns of the lane's row
    bool bad = false;
    for (int c0 = 0; c0 < TD; c0 += kPanel) {
        const int toff = (c0 / kPanel) % 2 * kPanel;
        if (warp == 0) {
            double a[kPanel], t[kPanel];
#pragma unroll
            for (int l = 0; l < kPanel; ++l) a[l] = sC[lane * TDP + c0 + l];
            if (c0 > 0) {
#pragma unroll
                for (int j = 0; j < kPanel; ++j)
#pragma unroll
                    for (int l = 0; l < kPanel; ++l) a[l] = fma(-tp[j], __shfl_sync(0xffffffffu, ap[j], c0 + l), a[l]);
            }
            double before[kPanel];
            bool plain = true;
#pragma unroll
            for (int j = 0; j < kPanel; ++j) before[j] = a[j];
#pragma unroll
            for (int j = 0; j < kPanel; ++j) {
                const double d = __shfl_sync(0xffffffffu, a[j], c0 + j);
                plain = plain && plain_pivot(d);
                t[j] = plain_quotient(a[j], d);
#pragma unroll
                for (int l = j + 1; l < kPanel; ++l) a[l] = fma(-t[j], __shfl_sync(0xffffffffu, a[j], c0 + l), a[l]);
                if (lane == c0 + j) s_d[c0 + j] = d;
            }
            if (!plain) {  // a pivot that is not positive, or out of the quotient's range: the panel again
#pragma unroll
                for (int j = 0; j < kPanel; ++j) a[j] = before[j];
#pragma unroll
                for (int j = 0; j < kPanel; ++j) {
                    const double d = __shfl_sync(0xffffffffu, a[j], c0 + j);
                    t[j] = other_quotient(a[j], d);
#pragma unroll
                    for (int l = j + 1; l < kPanel; ++l) a[l] = fma(-t[j], __shfl_sync(0xffffffffu, a[j], c0 + l), a[l]);
                    if (lane == c0 + j) s_d[c0 + j] = d;
                    bad = bad || !(d > 0.0);
                }
            }
            if (lane >= c0)
#pragma unroll
                for (int l = 0; l < kPanel; ++l) {
                    sC[lane * TDP + c0 + l] = a[l];
                    sT[lane * 9 + toff + l] = t[l];
                }
#pragma unroll
            for (int l = 0; l < kPanel; ++l) {
                ap[l] = a[l];
                tp[l] = t[l];
            }
        } else if (warp == 1 && c0 > 0 && c0 % 8 == 0) {
            inverse8(sC, sX, s_d, s_sd, s_rs, c0 / 8 - 1);
        } else if (warp > 1 || c0 == 0) {
            // columns c1 .. behind the panel: the panel before, and L L^T for the columns of the next but one
            // panel (with the first panel, for those of the next one too)
            const int c1 = c0 + kPanel, m = TD - c1;
            const int l0 = c0 == 0 ? c1 : c1 + kPanel, l1 = c1 + 2 * kPanel;
            const int first = c0 == 0 ? 32 : 64;
            for (int e = tid - first; e < m * (m + 1) / 2; e += kPotrf64Threads - first) {
                // by columns, so that a warp's elements share their kind: column c1 + q holds m - q of them
                int q = 0, r = e;
                while (r >= m - q) r -= m - q++;
                const int l = c1 + q, i = l + r;
                if (c0 == 0 && (!sL || l >= l1)) break;
                double v = sC[i * TDP + l];
                if (c0 > 0)
#pragma unroll
                    for (int j = 0; j < kPanel; ++j)
                        v = fma(-sT[i * 9 + kPanel - toff + j], sC[l * TDP + c0 - kPanel + j], v);
                if (sL && l >= l0 && l < l1)
#pragma unroll 8
                    for (int k = 0; k < TD; ++k) v = fma(-sL[k * TDP + i], sL[k * TDP + l], v);
                sC[i * TDP + l] = v;
            }
        }
        __syncthreads();
    }
    if (bad && lane == 0) atomicOr(status, 2);
    if (warp == 1) inverse8(sC, sX, s_d, s_sd, s_rs, 3);
    __syncthreads();
    // L: columns times 1 / sqrt(pivot); the 8 x 8 blocks of the inverse are final already
    for (int e = tid; e < TD * TD; e += kPotrf64Threads) {
        const int i = e / TD, j = e % TD;
        const double v = i > j ? sC[i * TDP + j] * s_rs[j] : (i == j ? s_sd[j] : 0.0);
        sC[i * TDP + j] = v;
        Akk[static_cast<size_t>(i) * np + j] = v;
    }
    __syncthreads();
#pragma unroll
    for (int h = 8; h <= 16; h *= 2) {
        // pairs of h x h blocks: rows r0 + h .. r0 + 2h - 1, columns r0 .. r0 + h - 1.  Products with a
        // triangular factor stop at its edge: a warp takes 32 / h columns (of L21 X11) or rows (of X22 P),
        // long ones on the warps that share a sub-partition with short ones.
        const int per = h * h, pairs = TD / (2 * h), wide = 32 / h, groups = h / wide;
        const int pr = tid / per, e = tid % per, g = e >> 5, at = lane % h, r0 = pr * 2 * h;
        const int line = (groups > 4 && g >= 4 ? groups + 3 - g : g) * wide + lane / h;
        if (pr < pairs) {
            const int first = line / wide * wide;  // the same for the warp
            double t = 0.0;
#pragma unroll 8
            for (int k = first; k < h; ++k) t = fma(sC[(r0 + h + at) * TDP + r0 + k], sX[(r0 + k) * TDP + r0 + line], t);
            sP[(r0 + at) * TDP + line] = t;
        }
        __syncthreads();
        if (pr < pairs) {
            const int last = line / wide * wide + wide - 1;
            double t = 0.0;
#pragma unroll 8
            for (int k = 0; k <= last; ++k) t = fma(sX[(r0 + h + line) * TDP + r0 + h + k], sP[(r0 + k) * TDP + at], t);
            sX[(r0 + h + line) * TDP + r0 + at] = -t;
        }
        __syncthreads();
    }
    for (int e = tid; e < TD * TD; e += kPotrf64Threads) D[e] = sX[(e / TD) * TDP + e % TD];
    (void)lane;
}

// Global 32 x 32 tile (row stride ld, 16-byte aligned rows) into shared memory, row-major.
__device__ __forceinline__ void tile32_load(const double* __restrict__ g, int ld, double* __restrict__ s) {
#pragma unroll
    for (int e = threadIdx.x; e < TD * TD / 2; e += kPotrf64Threads) {
        const int r = e >> 4, c = 2 * (e & 15);
        const double2 v = *reinterpret_cast<const double2*>(g + static_cast<size_t>(r) * ld + c);
        s[r * TDP + c] = v.x;
        s[r * TDP + c + 1] = v.y;
    }
}
// Rows (or columns) of a warp in a product with a triangular factor: four whose lengths add up to 66.
__device__ __forceinline__ int balanced32(int warp, int m) {
    return m == 0 ? warp : m == 1 ? 15 - warp : m == 2 ? 16 + warp : 31 - warp;
}

// A (lower triangle, np x np with identity padding) -> X = L^-1 in X and X^T in the upper triangle of A;
// nt tiles of 32.  The steps of k_potrf_coop: panel and inverse row, barrier, trailing and inverse
// update with the next diagonal tile factored by the block that updates it, barrier.
template <bool CLUSTER>
__global__ void __launch_bounds__(kPotrf64Threads) k_potrf64_coop(double* __restrict__ A, double* __restrict__ X,
                                                                  double* __restrict__ Dinv, int np, int nt,
                                                                  int* __restrict__ status,
                                                                  int* __restrict__ host_status) {
    extern __shared__ __align__(16) double smem64[];
    double* sA = smem64;
    double* sB = sA + TD * TDP;
    double* sC = sB + TD * TDP;
    double* sX = sC + TD * TDP;
    double* sT = sX + TD * TDP;
    double* s_d = sT + TD * 9;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto tile = [np](double* M, int i, int j) { return M + static_cast<size_t>(i) * TD * np + static_cast<size_t>(j) * TD; };
    // R_ij (j < i) gathers in tile (j, i) of X, above the diagonal, and X_ij goes below it; L_ik goes to tile
    // (k, i) of A.  No product is written over its operand, so that several blocks can share one.
    for (int r = blockIdx.x; r < nt * TD; r += gridDim.x)
        for (int c = (r / TD + 1) * TD + tid; c < nt * TD; c += kPotrf64Threads) X[static_cast<size_t>(r) * np + c] = 0.0;
    if (blockIdx.x == 0) {
        tile32_load(A, np, sC);
        __syncthreads();
        diag_factor_inverse64(A, np, Dinv, nullptr, sC, sA, sB, sT, s_d, status);
    }
    phase_barrier<CLUSTER>();
    for (int k = 0; k < nt; ++k) {
        const int m = nt - 1 - k;
        const double* Dk = Dinv + static_cast<size_t>(k) * TD * TD;
        // L_ik = A_ik D_k^T (a lane per row) and X_kj = D_k R_kj (a lane per column).  A warp takes four
        // columns (rows) whose lengths add up to 66; while four times the tiles fit the grid, four blocks
        // share a tile, a warp taking one of the four and a sub-partition's two warps at most 37 products.
        const int tiles = m + k + 1, parts = 4 * tiles <= static_cast<int>(gridDim.x) ? 4 : 1;
        for (int it = blockIdx.x; it < tiles * parts; it += gridDim.x) {
            const int tl = it / parts, pt = it - tl * parts;
            const int q0 = parts == 1 ? 0 : (warp < 4 ? (pt + warp) & 3 : 3 - ((pt + warp) & 3));
            const int q1 = parts == 1 ? 4 : q0 + 1;
            tile32_load(Dk, TD, sB);
            if (tl < m) {
                tile32_load(tile(A, k + 1 + tl, k), np, sA);
                __syncthreads();
                double* L = tile(A, k, k + 1 + tl);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (q < q0 || q >= q1) continue;
                    const int c = balanced32(warp, q);
                    double t = 0.0;
#pragma unroll 8
                    for (int l = 0; l <= c; ++l) t = fma(sA[lane * TDP + l], sB[c * TDP + l], t);
                    L[static_cast<size_t>(c) * np + lane] = t;  // (transposed: rows of the tile are columns of L)
                }
            } else {
                const int j = tl - m;
                if (j < k) tile32_load(tile(X, j, k), np, sA);
                __syncthreads();
                double* Xkj = tile(X, k, j);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (q < q0 || q >= q1) continue;
                    const int r = balanced32(warp, q);
                    double t = 0.0;
                    if (j == k) t = sB[r * TDP + lane];
                    else
#pragma unroll 8
                        for (int l = 0; l <= r; ++l) t = fma(sB[r * TDP + l], sA[l * TDP + lane], t);
                    Xkj[static_cast<size_t>(r) * np + lane] = t;
                }
            }
            __syncthreads();
        }
        phase_barrier<CLUSTER>();
        // trailing update and R update; item 0 is the next diagonal tile, updated and factored by
        // block 0 while the other blocks share the rest
        const int ntrail = m * (m + 1) / 2;
        const int nitems = ntrail + m * (k + 1);
        const int first_it = blockIdx.x == 0 ? 0 : (gridDim.x > 1 ? blockIdx.x : 1);
        const int stride = gridDim.x > 1 ? static_cast<int>(gridDim.x) - 1 : 1;
        for (int it = first_it; it < nitems; it = (it == 0 && gridDim.x > 1) ? nitems : it + stride) {
            if (it == 0) {
                const double* Lk = tile(A, k, k + 1);
                double* Akk = tile(A, k + 1, k + 1);
                tile32_load(Lk, np, sA);
                tile32_load(Akk, np, sC);
                __syncthreads();
                diag_factor_inverse64(Akk, np, Dinv + static_cast<size_t>(k + 1) * TD * TD, sA, sC, sX, sB, sT, s_d, status);
                __syncthreads();
                continue;
            }
            double* dst;
            const bool trail = it < ntrail;
            if (trail) {
                // A_ij -= L_ik L_jk^T
                const int t = tri_row(it);
                const int i = k + 1 + t, j = k + 1 + (it - t * (t + 1) / 2);
                tile32_load(tile(A, k, i), np, sA);
                tile32_load(tile(A, k, j), np, sB);
                dst = tile(A, i, j);
            } else {
                // R_ij -= L_ik X_kj
                const int q = it - ntrail;
                const int i = k + 1 + q / (k + 1), j = q % (k + 1);
                tile32_load(tile(A, k, i), np, sA);
                tile32_load(tile(X, k, j), np, sB);
                dst = tile(X, j, i);
            }
            double acc[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] = dst[static_cast<size_t>(warp + 8 * q) * np + lane];
            __syncthreads();
#pragma unroll 8
            for (int l = 0; l < TD; ++l) {
                const double bv = sB[l * TDP + lane];
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[q] = fma(-sA[l * TDP + warp + 8 * q], bv, acc[q]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[static_cast<size_t>(warp + 8 * q) * np + lane] = acc[q];
            __syncthreads();
        }
        phase_barrier<CLUSTER>();
    }
    if (blockIdx.x == 0 && tid == 0) *host_status = __ldcg(status);
    for (int it = blockIdx.x; it < nt * (nt + 1) / 2; it += gridDim.x) {
        const int i = tri_row(it), j = it - i * (i + 1) / 2;
        tile32_load(tile(X, i, j), np, sA);
        __syncthreads();
        double* dst = tile(A, j, i);
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[static_cast<size_t>(warp + 8 * q) * np + lane] = sA[lane * TDP + warp + 8 * q];
        __syncthreads();
    }
}

// ---- conjugate gradients on the FP64 reduced matrix, preconditioner D X^T X D (X = L^-1).
// One cooperative persistent kernel runs the whole solve; per iteration four phases separated
// by grid barriers: (1) the direction update fused with the block-CSR SpMV, (2) the x / r
// updates, (3) w = X D r and (4) z = D X^T w (a warp per row).  Grid-wide sums: p.q after (1),
// r.r after (2), r.z after (4).  (Reading r.r together with r.z after (4), one sum fewer, measured
// slower at 500 cameras: 82.7 against 79.0 ms of CG per solve.)
// FP64 arithmetic issues at 1/64 of the FP32 rate on this part: an SM sub-partition retires one
// warp-wide FP64 instruction about every 64 cycles.  The phases are therefore shaped by their
// FP64 instructions per sub-partition rather than by bytes: the SpMV runs as short work items (32
// pose blocks, or 256 entries of a border row, per warp) whose partial sums the owners of the
// rows add in a fixed order, and the dot-product reductions do their FP64 adds on four warps.
// Dot products go through per-block partials that every block sums in the same fixed order, so
// all blocks take the same convergence / breakdown decision and no result depends on timing.
namespace {
constexpr int kCgThreads = 256;
constexpr int kCgWarps = kCgThreads / 32;
constexpr int kCgPart = 4;  // partial slots per block
}  // namespace

// Block sum of v (all threads), written by thread 0 to *dst: warps 0-3 (one per sub-partition)
// each add 64 of the values, thread 0 the four sums.  Every caller passes a grid barrier before
// s_vals / s_q are written again.
__device__ __forceinline__ void block_partial(double v, double* s_vals, double* s_q, double* dst) {
    s_vals[threadIdx.x] = v;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 4) {
        double t = s_vals[64 * warp + lane] + s_vals[64 * warp + 32 + lane];
        t = warp_sum(t);
        if (lane == 0) s_q[warp] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) *dst = (s_q[0] + s_q[1]) + (s_q[2] + s_q[3]);
}

// Sums over blocks of partial slots `slot` and `slot + 1` (TWO) or `slot` alone, identical in
// every block: warps 0-3 each add a quarter of the blocks' partials (lane l: every 32nd), thread 0
// the four sums, broadcast through s_tot (a grid barrier separates two uses of one slot).
template <bool TWO>
__device__ __forceinline__ void grid_totals(const double* part, int slot, double* s_q, double* s_tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = static_cast<int>(gridDim.x);
    if (warp < 4) {
        const int k0 = G * warp / 4, k1 = G * (warp + 1) / 4;
        double t0 = 0.0, t1 = 0.0;
#pragma unroll 4
        for (int k = k0 + lane; k < k1; k += 32) {
            t0 += part[k * kCgPart + slot];
            if (TWO) t1 += part[k * kCgPart + slot + 1];
        }
        t0 = warp_sum(t0);
        if (TWO) t1 = warp_sum(t1);
        if (lane == 0) {
            s_q[4 + warp] = t0;
            if (TWO) s_q[8 + warp] = t1;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_tot[slot] = (s_q[4] + s_q[5]) + (s_q[6] + s_q[7]);
        if (TWO) s_tot[slot + 1] = (s_q[8] + s_q[9]) + (s_q[10] + s_q[11]);
    }
    __syncthreads();
}

// Warp sums of eight per-lane values with nine FP64 adds: a transposing butterfly in which, at
// each of the first three levels, a lane keeps half of its values and adds its partner's share of
// them.  The total of value x ends in lanes 4x .. 4x + 3 (all four hold the same bits).
__device__ __forceinline__ double warp_sum8(double (&a)[8]) {
    const int lane = threadIdx.x & 31;
    {
        const bool up = lane & 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double send = up ? a[j] : a[4 + j];
            const double keep = up ? a[4 + j] : a[j];
            a[j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
    }
    {
        const bool up = lane & 8;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double send = up ? a[j] : a[2 + j];
            const double keep = up ? a[2 + j] : a[j];
            a[j] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
    }
    double t;
    {
        const bool up = lane & 4;
        const double send = up ? a[0] : a[1];
        const double keep = up ? a[1] : a[0];
        t = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    return t;
}

// out_i = so_i * sum_j M_ij in_j over j <= i (LOWER) or j >= i, with in and the product in the
// factor's type T (FP32 on the mixed path: the preconditioner needs no more); one warp per row,
// rows interleaved over all warps of the grid, 16-byte loads from an aligned start (the extra
// elements lie in the diagonal tile, where the triangular factor is zero, and the padding of
// `in` beyond n is zero).  Writes out_t (T) or out_d (double, scaled by so) and returns this
// thread's share of dot_with . out_d.
template <typename T, bool LOWER>
__device__ __forceinline__ double tri_rows(const T* __restrict__ M, int np, int n, const T* __restrict__ in,
                                           T* __restrict__ out_t, double* __restrict__ out_d,
                                           const double* __restrict__ so, const double* __restrict__ dot_with) {
    using V = Vec16<T>;
    using VV = typename V::type;
    const int lane = threadIdx.x & 31;
    // warp-major row order: consecutive rows go to different blocks (SMs)
    const int gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = gridDim.x * kCgWarps;
    const VV* in_v = reinterpret_cast<const VV*>(in);
    double contrib = 0.0;
    for (int i = gw; i < n; i += nw) {
        const VV* row = reinterpret_cast<const VV*>(M + static_cast<size_t>(i) * np);
        const int q0 = LOWER ? 0 : i / V::n, q1 = LOWER ? (i + V::n) / V::n : (n + V::n - 1) / V::n;
        T acc = T(0);
#pragma unroll 8
        for (int q = q0 + lane; q < q1; q += 32) acc += V::dot(row[q], in_v[q]);
        acc = warp_sum(acc);
        if (lane == 0) {
            if (out_t) out_t[i] = acc;
            if (out_d) {
                const double v = static_cast<double>(acc) * so[i];
                out_d[i] = v;
                if (dot_with) contrib += dot_with[i] * v;
            }
        }
    }
    return contrib;
}

// Direction update fused with the SpMV: p = z + beta p_old, written to p_new by the first work
// item of each row, and the partial products of S p, with the entries of p formed on the fly by
// the same expression (so bitwise equal to p_new).  On the first iteration (beta == 0) p = z
// exactly, whatever p_old holds.  Work items, one warp each, in the warp-major order that spreads
// consecutive items over the blocks: segment s < pose_seg of pose block row r (its blocks
// 32 s .. 32 s + 31, a lane per block; the border columns with segment 0), then segment
// s < border_seg of border row c (a contiguous 256-entry share of its pose and intrinsic
// columns).  Item sums go to qpart: pose item (r, s) at 6 (r pose_seg + s), border item (c, s)
// at 6 ncb pose_seg + c border_seg + s; q is their sum over s, formed in order where q is read.
// Returns this thread's share of p.q = sum over items of p_i (item sum)_i.
__device__ __forceinline__ double spmv_update(const PcgSystem<double>& sys, const double* __restrict__ z,
                                              double beta, const double* __restrict__ p_old,
                                              double* __restrict__ p_new, double* __restrict__ qpart, int pose_seg,
                                              int border_seg) {
    const int lane = threadIdx.x & 31;
    // warp-major item order: consecutive items go to different blocks (SMs)
    const int gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = gridDim.x * kCgWarps;
    const int nb = sys.nb, n6 = 6 * sys.ncb, nrow = n6 + nb;
    const int npose = sys.ncb * pose_seg;
    const bool first = beta == 0.0;
    auto pv = [&](int i) { return first ? z[i] : fma(beta, p_old[i], z[i]); };
    double pq = 0.0;
    for (int t = gw; t < npose + nb * border_seg; t += nw) {
        if (t < npose) {
            const int r = t / pose_seg, sg = t - r * pose_seg;
            const int e0 = sys.row_ptr[r] + 32 * sg, e1 = sys.row_ptr[r + 1];
            double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            const int e = e0 + lane;
            if (e < e1) {
                const int j = sys.col_idx[e];
                const double* A = sys.vals + static_cast<size_t>(e) * 36;
                double pj[6];
#pragma unroll
                for (int c = 0; c < 6; ++c) pj[c] = pv(6 * j + c);
#pragma unroll
                for (int a = 0; a < 6; ++a)
#pragma unroll
                    for (int c = 0; c < 6; ++c) acc[a] = fma(A[a * 6 + c], pj[c], acc[a]);
            }
            if (sg == 0) {
                const double* Bi = sys.border + static_cast<size_t>(r) * 6 * nb;
                for (int c = lane; c < nb; c += 32) {
                    const double pc = pv(n6 + c);
#pragma unroll
                    for (int a = 0; a < 6; ++a) acc[a] = fma(Bi[a * nb + c], pc, acc[a]);
                }
            }
            const double v = warp_sum8(acc);
            const int x = lane >> 2;
            if ((lane & 3) == 0 && x < 6) {
                const int i = 6 * r + x;
                const double pi = pv(i);
                qpart[6 * t + x] = v;
                if (sg == 0) p_new[i] = pi;
                pq += pi * v;
            }
        } else {
            const int u = t - npose, c = u / border_seg, sg = u - c * border_seg;
            const int k0 = min(nrow, 256 * sg), k1 = min(nrow, 256 * (sg + 1));
            const double* Bc = sys.border_t + static_cast<size_t>(c) * n6;
            const double* Cc = sys.Cm + static_cast<size_t>(c) * nb;
            double v = 0.0;
#pragma unroll 4
            for (int k = k0 + lane; k < k1; k += 32) v = fma(k < n6 ? Bc[k] : Cc[k - n6], pv(k), v);
            v = warp_sum(v);
            if (lane == 0) {
                const int i = n6 + c;
                const double pi = pv(i);
                qpart[6 * npose + u] = v;
                if (sg == 0) p_new[i] = pi;
                pq += pi * v;
            }
        }
    }
    return pq;
}

// out: [0] iterations, [1] relative residual, [2] converged, [3] status (1: breakdown)
template <typename T>
__global__ void __launch_bounds__(kCgThreads, 2) k_dense_cg(PcgSystem<double> sys, const T* __restrict__ X,
                                                         const T* __restrict__ XT, int np,
                                                         const double* __restrict__ dscale,
                                                         const double* __restrict__ b, double* __restrict__ x,
                                                         double* __restrict__ r, double* __restrict__ z,
                                                         double* __restrict__ p, double* __restrict__ p2,
                                                         double* __restrict__ qpart, int pose_seg, int border_seg,
                                                         T* __restrict__ u, T* __restrict__ w,
                                                         double* __restrict__ part, double* __restrict__ out,
                                                         double rel_tol, double abs_tol, int max_it) {
    __shared__ double s_vals[kCgThreads];
    __shared__ double s_q[12];
    __shared__ double s_tot[kCgPart];
    const int n = 6 * sys.ncb + sys.nb;
    const int gt = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    double* mypart = part + static_cast<size_t>(blockIdx.x) * kCgPart;
    // r = b, x = 0, u = D r; z = D M u
    double bb = 0.0;
    for (int i = gt; i < n; i += nt) {
        x[i] = 0.0;
        r[i] = b[i];
        u[i] = static_cast<T>(dscale[i] * b[i]);
        bb += b[i] * b[i];
    }
    block_partial(bb, s_vals, s_q, mypart + 0);
    phase_barrier<false>();
    tri_rows<T, true>(X, np, n, u, w, nullptr, nullptr, nullptr);
    phase_barrier<false>();
    block_partial(tri_rows<T, false>(XT, np, n, w, nullptr, z, dscale, b), s_vals, s_q, mypart + 1);
    phase_barrier<false>();
    grid_totals<true>(part, 0, s_q, s_tot);
    const double bnorm = sqrt(s_tot[0]);
    double rz = s_tot[1];
    const double tol = fmax(rel_tol * bnorm, abs_tol);
    double rn = bnorm, beta = 0.0;
    int it = 0, status = 0;
    bool converged = rn <= tol;
    double* p_old = p2;
    double* p_cur = p;
    while (!converged && it < max_it) {
        // p = z + beta p and the partial products of S p (the direction buffers alternate)
        {
            double* t = p_old;
            p_old = p_cur;
            p_cur = t;
        }
        block_partial(spmv_update(sys, z, beta, p_old, p_cur, qpart, pose_seg, border_seg), s_vals, s_q, mypart + 2);
        phase_barrier<false>();
        grid_totals<false>(part, 2, s_q, s_tot);
        const double pq = s_tot[2];
        if (!(pq > 0.0) || !isfinite(pq) || !isfinite(rz)) {
            status = 1;
            break;
        }
        const double alpha = rz / pq;
        double rr = 0.0;
        const int n6 = 6 * sys.ncb;
        for (int i = gt; i < n; i += nt) {
            x[i] = fma(alpha, p_cur[i], x[i]);
            // (S p)_i: the row's item sums in order
            double qi;
            if (i < n6) {
                const double* qs = qpart + 6 * (i / 6) * pose_seg + i % 6;
                qi = qs[0];
                for (int sg = 1; sg < pose_seg; ++sg) qi += qs[6 * sg];
            } else {
                const double* qs = qpart + 6 * sys.ncb * pose_seg + (i - n6) * border_seg;
                qi = qs[0];
                for (int sg = 1; sg < border_seg; ++sg) qi += qs[sg];
            }
            const double rv = fma(-alpha, qi, r[i]);
            r[i] = rv;
            u[i] = static_cast<T>(dscale[i] * rv);
            rr += rv * rv;
        }
        block_partial(rr, s_vals, s_q, mypart + 0);
        phase_barrier<false>();
        ++it;
        grid_totals<false>(part, 0, s_q, s_tot);
        rn = sqrt(s_tot[0]);
        if (!isfinite(rn)) {
            status = 1;
            break;
        }
        if (rn <= tol) {
            converged = true;
            break;
        }
        tri_rows<T, true>(X, np, n, u, w, nullptr, nullptr, nullptr);
        phase_barrier<false>();
        block_partial(tri_rows<T, false>(XT, np, n, w, nullptr, z, dscale, r), s_vals, s_q, mypart + 1);
        phase_barrier<false>();
        grid_totals<false>(part, 1, s_q, s_tot);
        const double rz_new = s_tot[1];
        beta = rz_new / rz;
        rz = rz_new;
    }
    if (gt == 0) {
        out[0] = it;
        out[1] = bnorm > 0.0 ? rn / bnorm : 0.0;
        out[2] = converged ? 1.0 : 0.0;
        out[3] = status;
    }
}

// The same iteration for systems of at most kCgClusterDim unknowns, on one cluster whose blocks all keep the
// whole vectors in shared memory: a row's value goes from its warp to every block's copy, and what is not a
// matrix product (the scalars, x, r, p and u) is done by every block for itself, the same bits in each, so
// that an iteration takes three cluster barriers instead of four grid barriers and no vector or partial sum
// goes through L2 between them (a solve of two iterations, call included: 114 unknowns 67 -> 52 us, 234
// unknowns 69 -> 59, 380 unknowns 70 -> 67; 504 unknowns 74 on the grid against 88 here, sixteen blocks
// being too few for the FP64 products, and without pose blocks 312 unknowns 642 against 637, 364 unknowns
// 713 against 717 for a whole call).  An SpMV item is seg_blocks blocks of a block row, eight
// blocks by three pairs of rows at a time over 24 lanes (twelve FP64 products a turn), or 256 entries of a
// border row.  The matrices are read through L1, where a small system's shares stay.
constexpr int kCgClusterDim = 384, kCgClusterDimBorder = 320;
constexpr size_t kCgClusterSmem = 48 * 1024;
struct CgClusterShape {
    int seg_blocks, pose_seg, border_seg, items;  // items: sums of the SpMV items, 6 ncb pose_seg + nb border_seg
};
template <typename T>
__host__ __device__ constexpr size_t cg_cluster_smem(int n, int np, int items) {
    // u and w (padded, 16-byte rows), then r, z, p, scale, x, the item sums and the reduction's words
    return 2 * static_cast<size_t>(np) * sizeof(T) + (5 * static_cast<size_t>(n) + items + 8) * sizeof(double);
}

// Sum over the first four warps (one per sub-partition), the same in every thread.
__device__ __forceinline__ double four_warp_total(double v, double* s_red) {
    const int warp = threadIdx.x >> 5;
    __syncthreads();
    if (warp < 4) {
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) s_red[warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_red[4] = (s_red[0] + s_red[1]) + (s_red[2] + s_red[3]);
    __syncthreads();
    return s_red[4];
}

template <typename T>
__global__ void __launch_bounds__(kCgThreads) k_dense_cg_cluster(PcgSystem<double> sys, const T* __restrict__ X,
                                                                 const T* __restrict__ XT, int np,
                                                                 const double* __restrict__ dscale,
                                                                 const double* __restrict__ b, double* __restrict__ x,
                                                                 CgClusterShape shape, double* __restrict__ out,
                                                                 double rel_tol, double abs_tol, int max_it) {
    extern __shared__ __align__(16) unsigned char s_cg[];
    using V = Vec16<T>;
    using VV = typename V::type;
    const cgk::cluster_group cluster = cgk::this_cluster();
    const int n6 = 6 * sys.ncb, nb = sys.nb, n = n6 + nb;
    const int tid = threadIdx.x, lane = tid & 31, C = gridDim.x;
    const int gw = (tid >> 5) * C + blockIdx.x, nw = C * kCgWarps;  // consecutive rows go to different SMs
    T* u = reinterpret_cast<T*>(s_cg);
    T* w = u + np;
    double* r = reinterpret_cast<double*>(w + np);
    double* z = r + n;
    double* p = z + n;
    double* ds = p + n;
    double* xs = ds + n;
    double* q = xs + n;
    double* s_red = q + shape.items;
    double bb = 0.0;
    for (int i = tid; i < np; i += kCgThreads) {
        const double bi = i < n ? b[i] : 0.0, di = i < n ? dscale[i] : 0.0;
        u[i] = static_cast<T>(di * bi);
        w[i] = T(0);
        if (i < n) {
            r[i] = bi;
            ds[i] = di;
            p[i] = 0.0;
            xs[i] = 0.0;
        }
    }
    cluster.sync();
    if (tid < 128)
        for (int i = tid; i < n; i += 128) bb = fma(r[i], r[i], bb);
    const double bnorm = sqrt(four_warp_total(bb, s_red));
    const double tol = fmax(rel_tol * bnorm, abs_tol);
    double rn = bnorm, rz = 0.0;
    int it = 0, status = 0;
    bool converged = rn <= tol;
    T* w_to = lane < C ? cluster.map_shared_rank(w, lane) : nullptr;
    double* z_to = lane < C ? cluster.map_shared_rank(z, lane) : nullptr;
    double* q_to = lane < C ? cluster.map_shared_rank(q, lane) : nullptr;
    while (!converged && it < max_it) {
        // w = X u, z = D X^T w
        for (int i = gw; i < n; i += nw) {
            const VV* row = reinterpret_cast<const VV*>(X + static_cast<size_t>(i) * np);
            const int q1 = (i + V::n) / V::n;
            T acc = T(0);
#pragma unroll 4
            for (int k = lane; k < q1; k += 32) acc += V::dot(row[k], reinterpret_cast<const VV*>(u)[k]);
            acc = warp_sum(acc);
            if (w_to) w_to[i] = acc;
        }
        cluster.sync();
        for (int i = gw; i < n; i += nw) {
            const VV* row = reinterpret_cast<const VV*>(XT + static_cast<size_t>(i) * np);
            const int q1 = (n + V::n - 1) / V::n;
            T acc = T(0);
#pragma unroll 4
            for (int k = i / V::n + lane; k < q1; k += 32) acc += V::dot(row[k], reinterpret_cast<const VV*>(w)[k]);
            acc = warp_sum(acc);
            if (z_to) z_to[i] = static_cast<double>(acc) * ds[i];
        }
        cluster.sync();
        double part = 0.0;
        if (tid < 128)
            for (int i = tid; i < n; i += 128) part = fma(r[i], z[i], part);
        const double rz_new = four_warp_total(part, s_red);
        const double beta = it == 0 ? 0.0 : rz_new / rz;
        rz = rz_new;
        if (tid < 128)
            for (int i = tid; i < n; i += 128) p[i] = it == 0 ? z[i] : fma(beta, p[i], z[i]);
        __syncthreads();
        // item sums of S p
        const int npose = sys.ncb * shape.pose_seg, nitems = npose + nb * shape.border_seg;
        for (int t = gw; t < nitems; t += nw) {
            if (t < npose) {
                const int br = t / shape.pose_seg, sg = t - br * shape.pose_seg;
                const int e0 = sys.row_ptr[br] + shape.seg_blocks * sg, e1 = min(sys.row_ptr[br + 1], e0 + shape.seg_blocks);
                const int blk = lane >> 2, rows = lane & 3;
                double a0 = 0.0, a1 = 0.0;
                if (rows < 3) {
                    for (int e = e0 + blk; e < e1; e += 8) {
                        const double* pj = p + 6 * sys.col_idx[e];
                        const double2* A = reinterpret_cast<const double2*>(sys.vals + static_cast<size_t>(e) * 36 + 12 * rows);
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const double2 m0 = A[c], m1 = A[3 + c];
                            a0 = fma(m0.x, pj[2 * c], a0);
                            a1 = fma(m1.x, pj[2 * c], a1);
                            a0 = fma(m0.y, pj[2 * c + 1], a0);
                            a1 = fma(m1.y, pj[2 * c + 1], a1);
                        }
                    }
                    if (sg == 0) {
                        const double* Bi = sys.border + static_cast<size_t>(6 * br + 2 * rows) * nb;
                        for (int c = blk; c < nb; c += 8) {
                            a0 = fma(Bi[c], p[n6 + c], a0);
                            a1 = fma(Bi[nb + c], p[n6 + c], a1);
                        }
                    }
                }
                const bool up = lane & 16;
                double v = (up ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up ? a0 : a1, 16);
                v += __shfl_xor_sync(0xffffffffu, v, 8);
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                // the four lanes that hold a row's sum hand it to every fourth block
                if (rows < 3)
                    for (int k = blk & 3; k < C; k += 4) cluster.map_shared_rank(q, k)[6 * t + 2 * rows + (up ? 1 : 0)] = v;
            } else {
                const int k = t - npose, c = k / shape.border_seg, sg = k - c * shape.border_seg;
                const double* Bc = sys.border_t + static_cast<size_t>(c) * n6;
                const double* Cc = sys.Cm + static_cast<size_t>(c) * nb;
                const int k1 = min(n, 256 * (sg + 1));
                double v = 0.0;
#pragma unroll 4
                for (int j = 256 * sg + lane; j < k1; j += 32) v = fma(j < n6 ? Bc[j] : Cc[j - n6], p[j], v);
                v = warp_sum(v);
                if (q_to) q_to[6 * npose + k] = v;
            }
        }
        cluster.sync();
        // q from its items, p.q, and the updates
        part = 0.0;
        if (tid < 128)
            for (int i = tid; i < n; i += 128) {
                const double* qs = i < n6 ? q + 6 * (i / 6) * shape.pose_seg + i % 6 : q + 6 * npose + (i - n6) * shape.border_seg;
                const int step = i < n6 ? 6 : 1, m = i < n6 ? shape.pose_seg : shape.border_seg;
                double qi = qs[0];
                for (int sg = 1; sg < m; ++sg) qi += qs[step * sg];
                z[i] = qi;  // (z is free until the next product)
                part = fma(p[i], qi, part);
            }
        const double pq = four_warp_total(part, s_red);
        if (!(pq > 0.0) || !isfinite(pq) || !isfinite(rz)) {
            status = 1;
            break;
        }
        const double alpha = rz / pq;
        part = 0.0;
        if (tid < 128)
            for (int i = tid; i < n; i += 128) {
                xs[i] = fma(alpha, p[i], xs[i]);
                const double rv = fma(-alpha, z[i], r[i]);
                r[i] = rv;
                u[i] = static_cast<T>(ds[i] * rv);
                part = fma(rv, rv, part);
            }
        rn = sqrt(four_warp_total(part, s_red));
        ++it;
        if (!isfinite(rn)) {
            status = 1;
            break;
        }
        converged = rn <= tol;
    }
    if (blockIdx.x == 0) {
        __syncthreads();
        for (int i = tid; i < n; i += kCgThreads) x[i] = xs[i];
        if (tid == 0) {
            out[0] = it;
            out[1] = bnorm > 0.0 ? rn / bnorm : 0.0;
            out[2] = converged ? 1.0 : 0.0;
            out[3] = status;
        }
    }
}

// ---------------------------------------------------------------- host orchestration
template <typename T>
static void set_smem(const void* fn, size_t bytes) {
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

template <typename T>
size_t dense_bytes(int n) {
    const int np = ((n + TS - 1) / TS) * TS;
    return 2 * static_cast<size_t>(np) * np * sizeof(T) + static_cast<size_t>(np / TS) * TS * TS * sizeof(T);
}

// Launch of `grid` blocks as one cluster (more than eight need the non-portable size).
static void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at, int grid, int threads, size_t smem,
                           cudaStream_t st) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    at = cudaLaunchAttribute{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = static_cast<unsigned>(grid);
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
}

// Largest cluster (0, 8 or kClusterMax blocks) of the kernel that the device can hold.
static int largest_cluster(const void* kernel, int threads, size_t smem) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int size : {kClusterMax, 8}) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        cluster_config(cfg, at, size, threads, smem, nullptr);
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0) return size;
        cudaGetLastError();  // (a size that does not fit is not an error of the caller)
    }
    return 0;
}

// Launches a kernel of barrier-separated phases: as one cluster up to `cluster` blocks, else as a
// cooperative grid.
static cudaError_t launch_phased(const void* grid_kernel, const void* cluster_kernel, int cluster, int grid, int threads,
                                 void** args, size_t smem, cudaStream_t st) {
    if (grid > cluster) return cudaLaunchCooperativeKernel(grid_kernel, dim3(grid), dim3(threads), args, smem, st);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(cfg, at, grid, threads, smem, st);
    return cudaLaunchKernelExC(&cfg, cluster_kernel, args);
}

template <typename T>
int dense_factor(const PcgSystem<double>& sys, DenseWork<T>& W, double shift, int* h_status, cudaStream_t st,
                 int* launches) {
    const int n = W.n, np = W.np, nt = W.nt;
    // no unknowns: refused before any launch
    if (n <= 0) return -1;
    const size_t two_tiles = 2 * static_cast<size_t>(TS) * TP * sizeof(float);
    constexpr bool f64 = sizeof(T) == 8;
    const void *kernel, *cluster_kernel;
    if constexpr (f64) {
        kernel = reinterpret_cast<const void*>(&k_potrf64_coop<false>);
        cluster_kernel = reinterpret_cast<const void*>(&k_potrf64_coop<true>);
    } else {
        kernel = reinterpret_cast<const void*>(&k_potrf_coop<false>);
        cluster_kernel = reinterpret_cast<const void*>(&k_potrf_coop<true>);
    }
    const int threads = f64 ? kPotrf64Threads : 256;
    const size_t smem = f64 ? kPotrf64Smem : two_tiles;
    // (before the launches: the query clears its own errors, and must not clear one of theirs)
    if (W.fact_grid == 0) {
        set_smem<T>(kernel, smem);
        set_smem<T>(cluster_kernel, smem);
        W.fact_cluster = largest_cluster(cluster_kernel, threads, smem);
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
        W.fact_grid = std::max(1, std::min(per_sm, 2) * sms);
    }
    int L = 0;
    cudaMemsetAsync(W.status, 0, sizeof(int), st);
    cudaMemsetAsync(W.A, 0, static_cast<size_t>(np) * np * sizeof(T), st);
    k_dense_scale<<<(n + 255) / 256, 256, 0, st>>>(sys, W.dscale, W.status);
    const long long nfill = static_cast<long long>(sys.row_ptr ? W.nnzb : 0) * 36 + 6LL * sys.ncb * sys.nb +
                            static_cast<long long>(sys.nb) * sys.nb;
    if (nfill > 0) k_dense_fill<T><<<static_cast<unsigned>((nfill + 255) / 256), 256, 0, st>>>(sys, W.dscale, W.A, np);
    k_dense_diag<T><<<(np + 255) / 256, 256, 0, st>>>(W.A, n, np, shift);
    L += 3;
    {
        T* A = W.A;
        T* X = W.X;
        T* Dv = W.Dinv;
        int npv = np, ntv = f64 ? (n + TD - 1) / TD : nt;
        int* stv = W.status;
        void* args[] = {&A, &X, &Dv, &npv, &ntv, &stv, &h_status};
        // one block per lower tile, or four per tile of a panel, at most: small systems take a small grid
        const int fgrid = std::max(1, std::min(W.fact_grid, std::max(ntv * (ntv + 1) / 2, f64 ? 4 * ntv : 0)));
        if (launch_phased(kernel, cluster_kernel, W.fact_cluster, fgrid, threads, args, smem, st) != cudaSuccess) return -1;
        ++L;
    }
    if (launches) *launches += L;
    if (cudaGetLastError() != cudaSuccess) return -1;
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    const int status = *h_status;
    // opt-in trace (PB_GPU_TRACE=1): one line per factorisation
    static const bool trace = std::getenv("PB_GPU_TRACE") != nullptr;
    if (trace)
        std::fprintf(stderr, "PB_GPU_FACTOR precision=%d n=%d shift=%.3e status=%d\n", sizeof(T) == 4 ? 1 : 0, n, shift,
                     status);
    return status;
}

template <typename T>
int dense_pcg_launch(const PcgSystem<double>& sys, DenseWork<T>& W, const double* b, double rel_tol, double abs_tol,
                     int max_it, double* h_scal, cudaStream_t st, int* launches) {
    if (W.coop_grid == 0) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_dense_cg<T>, kCgThreads, 0);
        W.cg_cluster = largest_cluster(reinterpret_cast<const void*>(&k_dense_cg_cluster<T>), kCgThreads, kCgClusterSmem);
        W.coop_grid = std::max(1, std::min(per_sm, 2) * sms);
    }
    // one warp per row of the triangular products: small systems (local windows) take a small
    // grid and leave the rest of the device to concurrent work
    const int rows = (W.n + kCgWarps - 1) / kCgWarps;
    // items of eight blocks each until every warp of the cluster has one, then longer ones
    CgClusterShape shape{};
    {
        const int warps = kClusterMax * kCgWarps;
        shape.seg_blocks = 8 * std::max(1, (sys.ncb * ((W.longest + 7) / 8) + warps - 1) / warps);
        shape.pose_seg = sys.ncb > 0 ? std::max(1, (W.longest + shape.seg_blocks - 1) / shape.seg_blocks) : 0;
        shape.border_seg = W.border_seg;
        shape.items = 6 * sys.ncb * shape.pose_seg + sys.nb * shape.border_seg;
    }
    const size_t smem = cg_cluster_smem<T>(W.n, W.np, shape.items);
    if (W.cg_cluster == kClusterMax && W.n <= (sys.ncb > 0 ? kCgClusterDim : kCgClusterDimBorder) && smem <= kCgClusterSmem) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        W.cg_blocks = std::max(1, std::min(kClusterMax, rows));
        W.cg_max_it = max_it;
        cluster_config(cfg, at, W.cg_blocks, kCgThreads, smem, st);
        if (cudaLaunchKernelEx(&cfg, &k_dense_cg_cluster<T>, sys, static_cast<const T*>(W.X), static_cast<const T*>(W.A),
                               W.np, static_cast<const double*>(W.dscale), b, W.x, shape, h_scal, rel_tol, abs_tol,
                               max_it) != cudaSuccess)
            return -1;
        if (launches) *launches += 1;
        return 0;
    }
    const int grid = std::max(1, std::min(W.coop_grid, rows));
    W.cg_blocks = grid;
    W.cg_max_it = max_it;
    PcgSystem<double> s = sys;
    const T* X = W.X;
    const T* XT = W.A;
    int np = W.np;
    const double* dscale = W.dscale;
    double rt = rel_tol, at = abs_tol;
    int mi = max_it;
    int ps = W.pose_seg, bs = W.border_seg;
    void* args[] = {&s, &X, &XT, &np, &dscale, &b, &W.x, &W.r, &W.z, &W.p, &W.w, &W.qpart, &ps, &bs, &W.ut, &W.wt,
                    &W.part, &h_scal, &rt, &at, &mi};
    if (cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&k_dense_cg<T>), dim3(grid), dim3(kCgThreads), args, 0,
                                    st) != cudaSuccess)
        return -1;
    if (launches) *launches += 1;
    return 0;
}

template <typename T>
int dense_pcg_result(const DenseWork<T>& W, const double* h_scal, int* iterations, double* relres, bool* converged) {
    *iterations = static_cast<int>(h_scal[0]);
    *relres = h_scal[1];
    *converged = h_scal[2] != 0.0;
    // opt-in trace (PB_GPU_TRACE=1): one line per CG launch
    static const bool trace = std::getenv("PB_GPU_TRACE") != nullptr;
    if (trace)
        std::fprintf(stderr, "PB_GPU_CG precision=%d iterations=%d relres=%.3e converged=%d max_it=%d grid=%d\n",
                     sizeof(T) == 4 ? 1 : 0, *iterations, *relres, *converged ? 1 : 0, W.cg_max_it, W.cg_blocks);
    return h_scal[3] != 0.0 ? 1 : 0;
}

template <typename T>
int dense_pcg(const PcgSystem<double>& sys, DenseWork<T>& W, const double* b, double rel_tol, double abs_tol,
              int max_it, int* iterations, double* relres, bool* converged, double* h_scal, cudaStream_t st,
              int* launches) {
    if (dense_pcg_launch<T>(sys, W, b, rel_tol, abs_tol, max_it, h_scal, st, launches) != 0) return -1;
    if (cudaStreamSynchronize(st) != cudaSuccess) return -1;
    return dense_pcg_result<T>(W, h_scal, iterations, relres, converged);
}

template int dense_factor<float>(const PcgSystem<double>&, DenseWork<float>&, double, int*, cudaStream_t, int*);
template int dense_factor<double>(const PcgSystem<double>&, DenseWork<double>&, double, int*, cudaStream_t, int*);
template int dense_pcg_launch<float>(const PcgSystem<double>&, DenseWork<float>&, const double*, double, double, int,
                                     double*, cudaStream_t, int*);
template int dense_pcg_launch<double>(const PcgSystem<double>&, DenseWork<double>&, const double*, double, double, int,
                                      double*, cudaStream_t, int*);
template int dense_pcg_result<float>(const DenseWork<float>&, const double*, int*, double*, bool*);
template int dense_pcg_result<double>(const DenseWork<double>&, const double*, int*, double*, bool*);
template int dense_pcg<float>(const PcgSystem<double>&, DenseWork<float>&, const double*, double, double, int, int*,
                              double*, bool*, double*, cudaStream_t, int*);
template int dense_pcg<double>(const PcgSystem<double>&, DenseWork<double>&, const double*, double, double, int, int*,
                               double*, bool*, double*, cudaStream_t, int*);

}  // namespace pb
