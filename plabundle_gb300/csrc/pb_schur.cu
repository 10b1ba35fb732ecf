// pb_schur.cu -- damped Schur solve of host block normal equations on the device: the general
// (non-online) path's linear solve, plamatrix::internal::solveDampedSchurComplement.
//
// The reference calls it from its general LM driver (src/internal/BundleAdjustPlaMatrix.cpp:
// 311-357) and from the line-scan solver (src/linescan_plamatrix.cpp:147-158) with a
// BlockNormalEquations<double> assembled on the host (pb_bne.cpp).  PlaMatrix is absent from the
// reference tree, so the damping form and the elimination are restated from the online path,
// which the reference builds by hand (BundleAdjustPlaMatrixReferenceSchur.cpp:350-490, :930):
//   - every eliminated 3x3 block V_e has its diagonal scaled by (1 + damping) and is inverted by
//     its adjugate (singular when |det| <= 1e-15, tryInverse3x3RowMajor);
//   - every primary diagonal entry is scaled by (1 + damping); an entry that is exactly zero (a
//     padding column of a 13-column block) becomes 1 (finalizePrimaryDiagonal(1 + damping, 1));
//   - S = H_pp - sum_e W_e V_e^-1 W_e^T and b = -g_p + sum_e W_e V_e^-1 g_e;
//   - S x = b is solved by CG on the FP64 S preconditioned by a dense Cholesky factor of the
//     Jacobi-scaled S (FP64, or FP32 when mixed precision is requested), to
//     |b - S x| <= max(relative_tolerance |b|, absolute_tolerance);
//   - the eliminated steps are y_e = V_e^-1 (-g_e - W_e^T x).
// Kernels: one thread per coupling for Y = W V^-1 (and one per eliminated block for its inverse); one
// CTA per segment of the host-built list of coupling pairs of an upper primary block of S, then one
// thread per entry of S adding the segments in order (no atomics: the result is deterministic); one CTA
// per primary block for b; the dense factor and CG of pb_dense.cu on S held as a dense block (ncb = 0,
// nb = n); four lanes per eliminated block for the back-substitution.  The pattern (coupling order, pair
// lists) is built once per structure and reused while the structure hash is unchanged.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <unordered_map>
#include <vector>

#include "pb_kernels.h"

namespace pb {

long long bne_structure_hash(const pb_bne* q);
const std::vector<double>& bne_diag(const pb_bne* q);
const std::vector<double>& bne_gp(const pb_bne* q);
const std::vector<double>& bne_hee(const pb_bne* q);
const std::vector<double>& bne_ge(const pb_bne* q);
void bne_dims(const pb_bne* q, int* P, int* E, int* pbs, int* ebs);
void bne_pairs(const pb_bne* q, const std::vector<int>** row, const std::vector<int>** col, const std::vector<double>** vals);
void bne_couplings(const pb_bne* q, const std::vector<int>** elim, const std::vector<int>** prim,
                   const std::vector<double>** vals);

namespace {

constexpr int kEb = 3;
constexpr int kGatherThreads = 192;  // of the 169 elements of a pair of 13-column blocks, 88 % of the lanes work
constexpr int kSegItems = 64;        // coupling pairs of one block that one CTA sums

// Damped inverse of an eliminated block (row-major); false when singular.
__device__ __forceinline__ bool damped_inverse(const double* __restrict__ h, double damping, double* inv) {
    double V[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) V[i] = h[i];
#pragma unroll
    for (int d = 0; d < 3; ++d) V[d * 4] *= 1.0 + damping;
    const double c00 = V[4] * V[8] - V[5] * V[7], c01 = V[5] * V[6] - V[3] * V[8], c02 = V[3] * V[7] - V[4] * V[6];
    const double det = V[0] * c00 + V[1] * c01 + V[2] * c02;
    if (!(fabs(det) > 1e-15) || !isfinite(det)) {
#pragma unroll
        for (int i = 0; i < 9; ++i) inv[i] = 0.0;
        return false;
    }
    const double id = 1.0 / det;
    inv[0] = c00 * id;
    inv[1] = (V[2] * V[7] - V[1] * V[8]) * id;
    inv[2] = (V[1] * V[5] - V[2] * V[4]) * id;
    inv[3] = c01 * id;
    inv[4] = (V[0] * V[8] - V[2] * V[6]) * id;
    inv[5] = (V[2] * V[3] - V[0] * V[5]) * id;
    inv[6] = c02 * id;
    inv[7] = (V[1] * V[6] - V[0] * V[7]) * id;
    inv[8] = (V[0] * V[4] - V[1] * V[3]) * id;
    return true;
}

// Threads 0 .. E - 1: the damped inverse of their eliminated block.  Threads E .. E + ncpl - 1: Y_c = W_c V^-1
// of their coupling, with the inverse formed again (about 50 FP64 operations next to the 117 of the
// product).  A thread per coupling instead of one per eliminated block: a block's couplings no longer
// wait for each other on the few warps that the blocks fill.
__global__ void __launch_bounds__(128) k_schur_eliminate(int E, int ncpl, int pb, double damping,
                                                         const double* __restrict__ hee, const int* __restrict__ cpl_elim,
                                                         const double* __restrict__ cpl, double* __restrict__ vinv,
                                                         double* __restrict__ Y, int* __restrict__ flags) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= E + ncpl) return;
    const int c = t - E, e = c < 0 ? t : cpl_elim[c];
    double inv[9];
    const bool ok = damped_inverse(hee + static_cast<size_t>(e) * 9, damping, inv);
    if (c < 0) {
        if (!ok) atomicOr(flags, 1);
#pragma unroll
        for (int i = 0; i < 9; ++i) vinv[static_cast<size_t>(e) * 9 + i] = inv[i];
        return;
    }
    const double* W = cpl + static_cast<size_t>(c) * pb * kEb;
    double* y = Y + static_cast<size_t>(c) * pb * kEb;
#pragma unroll 4
    for (int a = 0; a < pb; ++a) {
        const double w0 = W[a * kEb], w1 = W[a * kEb + 1], w2 = W[a * kEb + 2];
#pragma unroll
        for (int k = 0; k < kEb; ++k) y[a * kEb + k] = w0 * inv[k] + w1 * inv[3 + k] + w2 * inv[6 + k];
    }
}

// Partial sums of the Schur terms sum Y_c1 W_c2^T of one segment (at most kSegItems consecutive
// coupling pairs of one upper block), a thread per element of the block (of its upper triangle for a
// diagonal block) and the pairs dealt to as many thread groups as fit, whose sums are added in
// order.  FP64-bound: three FMAs per element and pair.
__global__ void __launch_bounds__(kGatherThreads) k_schur_gather(int pb, const int* __restrict__ seg_blk,
                                                                 const int* __restrict__ seg_begin,
                                                                 const int* __restrict__ blk_i,
                                                                 const int* __restrict__ blk_j,
                                                                 const int2* __restrict__ items,
                                                                 const double* __restrict__ Y,
                                                                 const double* __restrict__ cpl,
                                                                 double* __restrict__ part) {
    __shared__ double s_acc[kGatherThreads + 64];
    const int seg = blockIdx.x, blk = seg_blk[seg];
    const bool diag = blk_i[blk] == blk_j[blk];
    const int ne = diag ? pb * (pb + 1) / 2 : pb * pb;
    const int groups = max(1, kGatherThreads / ne);
    const int i0 = seg_begin[seg], i1 = seg_begin[seg + 1];
    for (int e0 = 0; e0 < ne; e0 += kGatherThreads) {  // (once, up to thirteen columns)
        const int g = threadIdx.x / ne, e = e0 + (groups > 1 ? threadIdx.x - g * ne : threadIdx.x);
        const bool mine = (groups == 1 || g < groups) && e < ne;
        double acc = 0.0;
        int a = 0, b = 0;
        if (mine) {
            if (diag) {  // e-th element of the upper triangle, column by column
                while ((b + 1) * (b + 2) / 2 <= e) ++b;
                a = e - b * (b + 1) / 2;
            } else {
                a = e / pb;
                b = e - a * pb;
            }
#pragma unroll 4
            for (int it = i0 + (groups > 1 ? g : 0); it < i1; it += groups) {
                const int2 cc = items[it];
                const double* y = Y + (static_cast<size_t>(cc.x) * pb + a) * kEb;
                const double* W = cpl + (static_cast<size_t>(cc.y) * pb + b) * kEb;
                acc = fma(y[2], W[2], fma(y[1], W[1], fma(y[0], W[0], acc)));
            }
        }
        if (groups > 1) {
            s_acc[threadIdx.x] = acc;
            __syncthreads();
            if (threadIdx.x < ne)
                for (int q = 1; q < groups; ++q) acc += s_acc[q * ne + threadIdx.x];
        }
        if (mine && (groups == 1 || g == 0)) {
            double* p = part + static_cast<size_t>(seg) * pb * pb;
            p[a * pb + b] = acc;
            if (diag) p[b * pb + a] = acc;
        }
    }
}

// Upper blocks of S (and their transposes): damped H_pp minus the block's segments, in order.
__global__ void __launch_bounds__(256) k_schur_sum(int nblocks, int pb, int n, double damping, const int* __restrict__ blk_i,
                                                   const int* __restrict__ blk_j, const int* __restrict__ blk_src,
                                                   const int* __restrict__ blk_seg, const double* __restrict__ diag,
                                                   const double* __restrict__ off, const double* __restrict__ part,
                                                   double* __restrict__ S) {
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int pp = pb * pb;
    if (t >= static_cast<long long>(nblocks) * pp) return;
    const int blk = static_cast<int>(t / pp), e = static_cast<int>(t - static_cast<long long>(blk) * pp);
    const int a = e / pb, b = e - a * pb;
    const int bi = blk_i[blk], bj = blk_j[blk], src = blk_src[blk];
    double v = 0.0;
    if (bi == bj) v = diag[static_cast<size_t>(bi) * pp + e];
    else if (src >= 0) v = off[static_cast<size_t>(src) * pp + e];
    // damping of the primary diagonal (a structurally empty entry becomes 1)
    if (bi == bj && a == b) v = v != 0.0 ? v * (1.0 + damping) : 1.0;
#pragma unroll 4
    for (int s = blk_seg[blk]; s < blk_seg[blk + 1]; ++s) v -= part[static_cast<size_t>(s) * pp + e];
    const size_t row = static_cast<size_t>(bi) * pb + a, col = static_cast<size_t>(bj) * pb + b;
    S[row * n + col] = v;
    if (bi != bj) S[col * n + row] = v;
}

// b = -g_p + sum_c Y_c g_e(c): one block per primary block, its couplings dealt to thread groups of pb
// rows, the groups' sums added in order.
__global__ void __launch_bounds__(256) k_schur_rhs(int pb, const double* __restrict__ gp, const int* __restrict__ p_begin,
                                                   const int* __restrict__ p_list, const int* __restrict__ cpl_elim,
                                                   const double* __restrict__ Y, const double* __restrict__ ge,
                                                   double* __restrict__ b) {
    __shared__ double s_acc[256];
    const int blk = blockIdx.x, groups = 256 / pb;
    const int g = threadIdx.x / pb, a = threadIdx.x - g * pb;
    double v = 0.0;
    if (g < groups)
#pragma unroll 4
        for (int k = p_begin[blk] + g; k < p_begin[blk + 1]; k += groups) {
            const int c = p_list[k];
            const double* y = Y + (static_cast<size_t>(c) * pb + a) * kEb;
            const double* q = ge + static_cast<size_t>(cpl_elim[c]) * kEb;
            v = fma(y[2], q[2], fma(y[1], q[1], fma(y[0], q[0], v)));
        }
    s_acc[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x < pb) {
        double t = -gp[static_cast<size_t>(blk) * pb + threadIdx.x];
        for (int q = 0; q < groups; ++q) t += s_acc[q * pb + threadIdx.x];
        b[static_cast<size_t>(blk) * pb + threadIdx.x] = t;
    }
}

// y_e = V_e^-1 (-g_e - sum_c W_c^T x_prim(c)): four lanes per eliminated block, lane k < 3 its k-th
// component (neighbouring lanes read neighbouring columns of W).
__global__ void __launch_bounds__(128) k_schur_backsub(int E, int pb, const int* __restrict__ e_begin,
                                                       const int* __restrict__ cpl_prim, const double* __restrict__ cpl,
                                                       const double* __restrict__ vinv, const double* __restrict__ ge,
                                                       const double* __restrict__ x, double* __restrict__ y) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, e = t >> 2, k = t & 3, kk = min(k, 2);
    const int base = threadIdx.x & 28;
    double r = 0.0;
    if (e < E) {
        r = -ge[static_cast<size_t>(e) * 3 + kk];
        for (int c = e_begin[e]; c < e_begin[e + 1]; ++c) {
            const double* W = cpl + static_cast<size_t>(c) * pb * kEb + kk;
            const double* xp = x + static_cast<size_t>(cpl_prim[c]) * pb;
#pragma unroll 8
            for (int a = 0; a < pb; ++a) r = fma(-W[a * kEb], xp[a], r);
        }
    }
    __syncwarp();
    const double r0 = __shfl_sync(0xffffffffu, r, base), r1 = __shfl_sync(0xffffffffu, r, base + 1),
                 r2 = __shfl_sync(0xffffffffu, r, base + 2);
    if (e < E && k < 3) {
        const double* iv = vinv + static_cast<size_t>(e) * 9 + k * 3;
        y[static_cast<size_t>(e) * 3 + k] = iv[0] * r0 + iv[1] * r1 + iv[2] * r2;
    }
}

// r = b - S x0 (dense FP64 rows, one warp per row) for a warm start; out[0] = |r|^2 partials per row
__global__ void k_schur_residual(int n, const double* __restrict__ S, const double* __restrict__ b,
                                 const double* __restrict__ x0, double* __restrict__ r) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= n) return;
    double v = 0.0;
    for (int k = lane; k < n; k += 32) v = fma(S[static_cast<size_t>(row) * n + k], x0[k], v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) r[row] = b[row] - v;
}

__global__ void k_axpy_into(int n, const double* __restrict__ x0, const double* __restrict__ d, double* __restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = x0[i] + d[i];
}

struct Arena {
    std::vector<void*> ptrs;
    template <typename T>
    T* alloc(size_t count) {
        void* p = nullptr;
        if (cudaMalloc(&p, std::max<size_t>(1, count) * sizeof(T)) != cudaSuccess) throw std::bad_alloc();
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
    void free_all() {
        for (void* p : ptrs) cudaFree(p);
        ptrs.clear();
    }
};

}  // namespace

struct SchurWork {
    long long hash = 0;
    bool ready = false;
    int P = 0, E = 0, pb = 0, n = 0, ncpl = 0, nblocks = 0, nitems = 0, noff = 0;
    std::vector<int> cpl_perm;   // sorted position -> container coupling index
    std::vector<int> off_block;  // block of each container pair (upper)
    Arena pattern, values, dense;
    // pattern
    int *e_begin = nullptr, *cpl_prim = nullptr, *cpl_elim = nullptr, *p_begin = nullptr, *p_list = nullptr;
    int *blk_i = nullptr, *blk_j = nullptr, *blk_src = nullptr, *blk_seg = nullptr, *seg_blk = nullptr,
        *seg_begin = nullptr, *zero = nullptr;
    int nseg = 0;
    double* part = nullptr;  // Schur terms of the segments
    int2* items = nullptr;
    // values and work
    double *diag = nullptr, *off = nullptr, *gp = nullptr, *hee = nullptr, *ge = nullptr, *cpl = nullptr;
    double *vinv = nullptr, *Y = nullptr, *S = nullptr, *b = nullptr, *x = nullptr, *x0 = nullptr, *r0 = nullptr,
           *y = nullptr;
    int* flags = nullptr;
    DenseWork<double> dw64;
    DenseWork<float> dw32;
    int dense_n[2] = {0, 0};
    double* h_scal = nullptr;  // pinned: CG scalars
    cudaEvent_t ev[8] = {};
    ~SchurWork() {
        pattern.free_all();
        values.free_all();
        dense.free_all();
        if (h_scal) cudaFreeHost(h_scal);
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
    }
};

SchurWork* schur_work_create() { return new SchurWork; }
void schur_work_destroy(SchurWork* w) { delete w; }

namespace {

template <typename T>
DenseWork<T>& dense_of(SchurWork* w);
template <>
DenseWork<double>& dense_of<double>(SchurWork* w) { return w->dw64; }
template <>
DenseWork<float>& dense_of<float>(SchurWork* w) { return w->dw32; }

template <typename T>
void ensure_dense(SchurWork* w, int device) {
    const int idx = sizeof(T) == 4 ? 1 : 0;
    DenseWork<T>& W = dense_of<T>(w);
    if (w->dense_n[idx] == w->n) return;
    // a new dimension: fresh buffers (the old ones stay until the work is destroyed)
    W = DenseWork<T>{};
    W.n = w->n;
    W.nt = std::max(1, (w->n + 63) / 64);
    W.np = W.nt * 64;
    W.nnzb = 0;
    W.A = w->dense.alloc<T>(static_cast<size_t>(W.np) * W.np);
    W.X = w->dense.alloc<T>(static_cast<size_t>(W.np) * W.np);
    W.Dinv = w->dense.alloc<T>(static_cast<size_t>(W.nt) * 64 * 64);
    W.dscale = w->dense.alloc<double>(W.n);
    W.status = w->dense.alloc<int>(1);
    W.x = w->dense.alloc<double>(W.n);
    W.r = w->dense.alloc<double>(W.n);
    W.z = w->dense.alloc<double>(W.n);
    W.p = w->dense.alloc<double>(W.n);
    W.q = w->dense.alloc<double>(W.n);
    // SpMV work items of the CG: every row is a border row here, 256 entries per item
    W.pose_seg = 0;
    W.border_seg = (W.n + 255) / 256;
    W.qpart = w->dense.alloc<double>(static_cast<size_t>(W.n) * W.border_seg);
    W.w = w->dense.alloc<double>(W.n);
    W.ut = w->dense.alloc<T>(W.np);
    W.wt = w->dense.alloc<T>(W.np);
    cudaMemset(W.ut, 0, static_cast<size_t>(W.np) * sizeof(T));
    cudaMemset(W.wt, 0, static_cast<size_t>(W.np) * sizeof(T));
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    W.part = w->dense.alloc<double>(static_cast<size_t>(std::max(1, sms)) * 32 * 4);
    w->dense_n[idx] = w->n;
}

void build_pattern(SchurWork* w, const pb_bne* q) {
    w->pattern.free_all();
    w->values.free_all();
    int P, E, pbs, ebs;
    bne_dims(q, &P, &E, &pbs, &ebs);
    const std::vector<int>*orow, *ocol, *celim, *cprim;
    const std::vector<double>*oval, *cval;
    bne_pairs(q, &orow, &ocol, &oval);
    bne_couplings(q, &celim, &cprim, &cval);
    w->P = P;
    w->E = E;
    w->pb = pbs;
    w->n = P * pbs;
    w->ncpl = static_cast<int>(celim->size());
    w->noff = static_cast<int>(orow->size());
    // couplings by (eliminated block, primary block)
    std::vector<int> perm(w->ncpl);
    for (int i = 0; i < w->ncpl; ++i) perm[i] = i;
    std::sort(perm.begin(), perm.end(), [&](int a, int b) {
        return (*celim)[a] != (*celim)[b] ? (*celim)[a] < (*celim)[b] : (*cprim)[a] < (*cprim)[b];
    });
    w->cpl_perm = perm;
    std::vector<int> e_begin(E + 1, 0), sprim(w->ncpl), selim(w->ncpl);
    for (int k = 0; k < w->ncpl; ++k) {
        selim[k] = (*celim)[perm[k]];
        sprim[k] = (*cprim)[perm[k]];
        ++e_begin[selim[k] + 1];
    }
    for (int e = 0; e < E; ++e) e_begin[e + 1] += e_begin[e];
    // couplings of each primary block (for the right-hand side), in sorted-coupling order
    std::vector<int> p_begin(P + 1, 0), p_list(w->ncpl);
    for (int k = 0; k < w->ncpl; ++k) ++p_begin[sprim[k] + 1];
    for (int i = 0; i < P; ++i) p_begin[i + 1] += p_begin[i];
    {
        std::vector<int> fill(p_begin.begin(), p_begin.end() - 1);
        for (int k = 0; k < w->ncpl; ++k) p_list[fill[sprim[k]]++] = k;
    }
    // upper blocks of S: every diagonal block, every stored pair, every pair of couplings of one
    // eliminated block; items (c1, c2) with prim(c1) <= prim(c2), in eliminated-block order
    std::unordered_map<long long, int> bidx;
    std::vector<int> bi, bj, bsrc;
    auto block_of = [&](int i, int j) {
        const long long key = static_cast<long long>(i) * P + j;
        auto it = bidx.find(key);
        if (it != bidx.end()) return it->second;
        const int k = static_cast<int>(bi.size());
        bidx.emplace(key, k);
        bi.push_back(i);
        bj.push_back(j);
        bsrc.push_back(-1);
        return k;
    };
    for (int i = 0; i < P; ++i) block_of(i, i);
    w->off_block.assign(w->noff, -1);
    for (int k = 0; k < w->noff; ++k) {
        const int blk = block_of((*orow)[k], (*ocol)[k]);
        bsrc[blk] = k;
        w->off_block[k] = blk;
    }
    std::vector<std::vector<int2>> blk_items;
    auto add_item = [&](int blk, int2 it) {
        if (blk >= static_cast<int>(blk_items.size())) blk_items.resize(blk + 1);
        blk_items[blk].push_back(it);
    };
    for (int e = 0; e < E; ++e)
        for (int c1 = e_begin[e]; c1 < e_begin[e + 1]; ++c1)
            for (int c2 = c1; c2 < e_begin[e + 1]; ++c2) add_item(block_of(sprim[c1], sprim[c2]), make_int2(c1, c2));
    w->nblocks = static_cast<int>(bi.size());
    blk_items.resize(w->nblocks);
    // segments of at most kSegItems consecutive items of one block
    std::vector<int> blk_seg(1, 0), seg_blk, seg_begin(1, 0);
    std::vector<int2> items;
    for (int k = 0; k < w->nblocks; ++k) {
        for (size_t i = 0; i < blk_items[k].size(); i += kSegItems) {
            const size_t i1 = std::min(blk_items[k].size(), i + kSegItems);
            items.insert(items.end(), blk_items[k].begin() + i, blk_items[k].begin() + i1);
            seg_blk.push_back(k);
            seg_begin.push_back(static_cast<int>(items.size()));
        }
        blk_seg.push_back(static_cast<int>(seg_blk.size()));
    }
    w->nseg = static_cast<int>(seg_blk.size());
    w->nitems = static_cast<int>(items.size());
    auto up = [&](auto& arena, const auto& v) {
        using T = typename std::decay_t<decltype(v)>::value_type;
        T* p = arena.template alloc<T>(v.size());
        if (!v.empty()) cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
        return p;
    };
    w->e_begin = up(w->pattern, e_begin);
    w->cpl_prim = up(w->pattern, sprim);
    w->cpl_elim = up(w->pattern, selim);
    w->p_begin = up(w->pattern, p_begin);
    w->p_list = up(w->pattern, p_list);
    w->blk_i = up(w->pattern, bi);
    w->blk_j = up(w->pattern, bj);
    w->blk_src = up(w->pattern, bsrc);
    w->blk_seg = up(w->pattern, blk_seg);
    w->seg_blk = up(w->pattern, seg_blk);
    w->seg_begin = up(w->pattern, seg_begin);
    w->items = up(w->pattern, items);
    w->zero = up(w->pattern, std::vector<int>{0});
    const size_t n = static_cast<size_t>(w->n);
    w->diag = w->values.alloc<double>(static_cast<size_t>(P) * pbs * pbs);
    w->off = w->values.alloc<double>(static_cast<size_t>(w->noff) * pbs * pbs);
    w->gp = w->values.alloc<double>(n);
    w->hee = w->values.alloc<double>(static_cast<size_t>(E) * 9);
    w->ge = w->values.alloc<double>(static_cast<size_t>(E) * 3);
    w->cpl = w->values.alloc<double>(static_cast<size_t>(w->ncpl) * pbs * kEb);
    w->vinv = w->values.alloc<double>(static_cast<size_t>(E) * 9);
    w->Y = w->values.alloc<double>(static_cast<size_t>(w->ncpl) * pbs * kEb);
    w->part = w->values.alloc<double>(static_cast<size_t>(w->nseg) * pbs * pbs);
    w->S = w->values.alloc<double>(n * n);
    w->b = w->values.alloc<double>(n);
    w->x = w->values.alloc<double>(n);
    w->x0 = w->values.alloc<double>(n);
    w->r0 = w->values.alloc<double>(n);
    w->y = w->values.alloc<double>(static_cast<size_t>(E) * 3);
    w->flags = w->values.alloc<int>(1);
    w->hash = bne_structure_hash(q);
    w->ready = true;
}

float event_ms(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    return ms;
}

template <typename T>
int dense_solve(SchurWork* w, int device, const pb_schur_options& op, double tol_abs, int max_it, cudaStream_t st,
                pb_schur_report* rep, int* iterations, double* relres, bool* converged) {
    ensure_dense<T>(w, device);
    DenseWork<T>& W = dense_of<T>(w);
    PcgSystem<double> sys{};
    sys.ncb = 0;
    sys.nb = w->n;
    sys.ng = 0;
    sys.ni = 0;
    sys.row_ptr = w->zero;
    sys.vals = nullptr;
    sys.Cm = w->S;
    int launches = 0;
    cudaEventRecord(w->ev[3], st);
    // FP32 factors of an ill-conditioned S need a small shift; the CG runs on the FP64 S
    double shift = sizeof(T) == 4 ? 1e-7 : 0.0;
    int fst = 0;
    for (int attempt = 0; attempt < 6; ++attempt) {
        fst = dense_factor<T>(sys, W, shift, reinterpret_cast<int*>(w->h_scal + 8), st, &launches);
        if (fst < 0) return -1;
        if (fst == 0 || (fst & 1)) break;
        shift = shift == 0.0 ? 1e-9 : shift * 10.0;
    }
    cudaEventRecord(w->ev[4], st);
    if (fst) return 1;
    const bool warm = op.use_initial_guess != 0;
    const double* rhs = warm ? w->r0 : w->b;
    int rc = dense_pcg<T>(sys, W, rhs, 0.0, tol_abs, max_it, iterations, relres, converged, w->h_scal, st, &launches);
    cudaEventRecord(w->ev[5], st);
    if (rc < 0) return -1;
    if (rc) return 1;
    if (warm) k_axpy_into<<<(w->n + 255) / 256, 256, 0, st>>>(w->n, w->x0, W.x, w->x);
    else cudaMemcpyAsync(w->x, W.x, static_cast<size_t>(w->n) * sizeof(double), cudaMemcpyDeviceToDevice, st);
    (void)rep;
    return 0;
}

}  // namespace

int schur_solve(SchurWork* w, int device, cudaStream_t st, const pb_bne* q, double damping, const pb_schur_options& op,
                double* primary_step, double* eliminated_step, pb_schur_report* rep, std::string* err) {
    const auto t0 = std::chrono::steady_clock::now();
    std::memset(rep, 0, sizeof(*rep));
    int P, E, pbs, ebs;
    bne_dims(q, &P, &E, &pbs, &ebs);
    const int n = P * pbs;
    const bool mixed = op.use_mixed_precision != 0;
    if (n > (mixed ? 32768 : 16384)) {
        *err = "block-Schur system too large for the dense device solve";
        return PB_ERR_UNSUPPORTED;
    }
    if (!w->ev[0])
        for (cudaEvent_t& e : w->ev) cudaEventCreate(&e);
    if (!w->h_scal) cudaMallocHost(reinterpret_cast<void**>(&w->h_scal), 16 * sizeof(double));
    const long long h = bne_structure_hash(q);
    const bool reuse = w->ready && h == w->hash;
    if (!reuse) build_pattern(w, q);
    rep->schur_pattern_reused = reuse ? 1 : 0;
    rep->symbolic_analysis_reused = reuse ? 1 : 0;
    rep->schur_assembly_on_device = 1;
    rep->mixed_precision_used = mixed ? 1 : 0;
    std::snprintf(rep->preconditioner_name, sizeof rep->preconditioner_name, "%s dense Cholesky (Jacobi-scaled)",
                  mixed ? "FP32" : "FP64");
    cudaDeviceProp prop{};
    if (cudaGetDeviceProperties(&prop, device) == cudaSuccess)
        std::snprintf(rep->device_name, sizeof rep->device_name, "%s", prop.name);
    // values: container order, couplings in sorted order
    const std::vector<int>*orow, *ocol, *celim, *cprim;
    const std::vector<double>*oval, *cval;
    bne_pairs(q, &orow, &ocol, &oval);
    bne_couplings(q, &celim, &cprim, &cval);
    std::vector<double> cs(static_cast<size_t>(w->ncpl) * pbs * kEb);
    for (int k = 0; k < w->ncpl; ++k)
        std::memcpy(cs.data() + static_cast<size_t>(k) * pbs * kEb, cval->data() + static_cast<size_t>(w->cpl_perm[k]) * pbs * kEb,
                    sizeof(double) * pbs * kEb);
    auto h2d = [&](double* dst, const std::vector<double>& src) {
        if (!src.empty()) cudaMemcpyAsync(dst, src.data(), src.size() * sizeof(double), cudaMemcpyHostToDevice, st);
    };
    h2d(w->diag, bne_diag(q));
    h2d(w->off, *oval);
    h2d(w->gp, bne_gp(q));
    h2d(w->hee, bne_hee(q));
    h2d(w->ge, bne_ge(q));
    h2d(w->cpl, cs);
    if (op.use_initial_guess && primary_step)
        cudaMemcpyAsync(w->x0, primary_step, static_cast<size_t>(n) * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(w->flags, 0, sizeof(int), st);
    cudaMemsetAsync(w->S, 0, static_cast<size_t>(n) * n * sizeof(double), st);
    cudaEventRecord(w->ev[0], st);
    if (E > 0)
        k_schur_eliminate<<<(E + w->ncpl + 127) / 128, 128, 0, st>>>(E, w->ncpl, pbs, damping, w->hee, w->cpl_elim, w->cpl,
                                                                    w->vinv, w->Y, w->flags);
    cudaEventRecord(w->ev[1], st);
    if (w->nseg > 0)
        k_schur_gather<<<w->nseg, kGatherThreads, 0, st>>>(pbs, w->seg_blk, w->seg_begin, w->blk_i, w->blk_j, w->items, w->Y,
                                                          w->cpl, w->part);
    const long long entries = static_cast<long long>(w->nblocks) * pbs * pbs;
    if (entries > 0)
        k_schur_sum<<<static_cast<unsigned>((entries + 255) / 256), 256, 0, st>>>(
            w->nblocks, pbs, n, damping, w->blk_i, w->blk_j, w->blk_src, w->blk_seg, w->diag, w->off, w->part, w->S);
    if (n > 0) k_schur_rhs<<<P, 256, 0, st>>>(pbs, w->gp, w->p_begin, w->p_list, w->cpl_elim, w->Y, w->ge, w->b);
    cudaEventRecord(w->ev[2], st);
    if (cudaGetLastError() != cudaSuccess) {
        *err = "block-Schur assembly launch failed";
        return PB_ERR_CUDA;
    }
    int flags = 0;
    cudaMemcpyAsync(w->h_scal, w->flags, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        *err = "block-Schur assembly failed";
        return PB_ERR_CUDA;
    }
    std::memcpy(&flags, w->h_scal, sizeof(int));
    rep->small_block_inverse_ms = event_ms(w->ev[0], w->ev[1]);
    rep->schur_accumulation_ms = event_ms(w->ev[1], w->ev[2]);
    rep->schur_assembly_ms = event_ms(w->ev[0], w->ev[2]);
    if (flags & 1) {
        rep->eliminated_singular = 1;
        *err = "eliminated block is not numerically SPD (positive definite)";
        return PB_ERR_SINGULAR_BLOCK;
    }
    if (n == 0) {
        rep->converged = 1;
        if (E > 0) {
            k_schur_backsub<<<(4 * E + 127) / 128, 128, 0, st>>>(E, pbs, w->e_begin, w->cpl_prim, w->cpl, w->vinv, w->ge, w->x, w->y);
            cudaMemcpyAsync(eliminated_step, w->y, static_cast<size_t>(E) * 3 * sizeof(double), cudaMemcpyDeviceToHost, st);
        }
        cudaStreamSynchronize(st);
        rep->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        return PB_OK;
    }
    // stopping rule |b - S x| <= max(rel |b|, abs) on the full right-hand side
    std::vector<double> hb(n);
    cudaMemcpyAsync(hb.data(), w->b, static_cast<size_t>(n) * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (op.use_initial_guess)
        k_schur_residual<<<(n + 7) / 8, 256, 0, st>>>(n, w->S, w->b, w->x0, w->r0);
    cudaStreamSynchronize(st);
    double bn = 0.0;
    for (double v : hb) bn += v * v;
    bn = std::sqrt(bn);
    const double rel = op.relative_tolerance > 0 ? op.relative_tolerance : 1e-12;
    const double abs_tol = op.absolute_tolerance > 0 ? op.absolute_tolerance : 1e-12;
    const double tol = std::max(rel * bn, abs_tol);
    const int max_it = op.max_iterations > 0 ? op.max_iterations : std::max(200, 30 * P);
    int iterations = 0;
    double relres = 0.0;
    bool converged = false;
    const int rc = mixed ? dense_solve<float>(w, device, op, tol, max_it, st, rep, &iterations, &relres, &converged)
                         : dense_solve<double>(w, device, op, tol, max_it, st, rep, &iterations, &relres, &converged);
    if (rc < 0) {
        *err = std::string("block-Schur dense solve failed: ") + cudaGetErrorString(cudaGetLastError());
        return PB_ERR_CUDA;
    }
    if (rc > 0) {
        *err = "dense Schur matrix is not numerically SPD (positive definite): CG breakdown";
        return PB_ERR_SINGULAR_BLOCK;
    }
    // residual check of the result on the damped FP64 S: |b - S x| / |b|
    k_schur_residual<<<(n + 7) / 8, 256, 0, st>>>(n, w->S, w->b, w->x, w->r0);
    cudaMemcpyAsync(hb.data(), w->r0, static_cast<size_t>(n) * sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaEventRecord(w->ev[6], st);
    if (E > 0)
        k_schur_backsub<<<(4 * E + 127) / 128, 128, 0, st>>>(E, pbs, w->e_begin, w->cpl_prim, w->cpl, w->vinv, w->ge, w->x, w->y);
    cudaEventRecord(w->ev[7], st);
    if (primary_step)
        cudaMemcpyAsync(primary_step, w->x, static_cast<size_t>(n) * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (eliminated_step && E > 0)
        cudaMemcpyAsync(eliminated_step, w->y, static_cast<size_t>(E) * 3 * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        *err = "block-Schur back-substitution failed";
        return PB_ERR_CUDA;
    }
    double rn = 0.0;
    for (double v : hb) rn += v * v;
    // converged: the CG met the tolerance on its recursive residual; the true residual of the
    // result is reported (near a fixed point it can sit at the FP64 floor, above the tolerance)
    rep->converged = converged ? 1 : 0;
    rep->iterations = iterations;
    rep->relative_residual = bn > 0 ? std::sqrt(rn) / bn : std::sqrt(rn);
    (void)relres;
    rep->cholesky_factorization_ms = event_ms(w->ev[3], w->ev[4]);
    rep->triangular_solve_ms = event_ms(w->ev[4], w->ev[5]);
    rep->linear_solve_ms = event_ms(w->ev[3], w->ev[5]);
    rep->back_substitution_ms = event_ms(w->ev[6], w->ev[7]);
    rep->total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    return PB_OK;
}

}  // namespace pb
