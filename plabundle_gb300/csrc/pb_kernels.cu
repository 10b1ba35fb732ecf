// pb_kernels.cu -- reduction of the assembly partials, back-substitution, objective and
// state-update kernels (the assembly kernel itself is in pb_assemble.cu).
//
// `k_reduce_*` sum the chunk partials of every reduced block in a fixed order, with the
// accumulator of the arithmetic path (two-sum compensated float-float on the FP32 path), so the
// reduced matrix is assembled without atomics and reproducibly.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <mutex>
#include <type_traits>

#include "pb_device.cuh"
#include "pb_kernels.h"

namespace pb {

// The three fixed-order sums below are independent of one another and each is latency-bound on
// a small grid (the chunk-record sum has one CTA per 32 record entries), so one launch runs them
// side by side over block ranges [chunk records + cost | cameras | pose pairs].  Each keeps the
// summation order of its own loop.  A list's merges are a serial chain of a few FP32 additions (one FP64
// addition) each, and the lists are long (hundreds of chunks touch a camera), so the records in flight per
// list decide, unless the lists are short.
template <typename T>
struct ReduceArgs {
    using part_t = typename Acc<T>::part_type;
    const part_t* part_pair;
    const part_t* part_cam;
    const part_t* part_chunk;
    const double* part_cost;
    const int* part_flags;
    double *vals, *rhs, *direct, *border, *border_t, *Cm, *result;
    unsigned chunk_blocks;  // first block of the lists
    unsigned list_blocks;   // ring: blocks of the lists; entries: blocks of the pose pairs
    bool spread;            // ring: neighbouring lists to neighbouring blocks, not warps
};

// A warp sums up to 36 neighbouring entries of one list's records (lane l entries l and 32 + l) in the
// order of the list.  The records stream through a ring of six stages of eight in shared memory by
// asynchronous copies, their list indices loaded a vector of 32 ahead.  (A thread per entry with four
// loads ahead leaves the longest lists waiting: this sum and k_finalize, 100 cameras and 120 000 points,
// mixed 206 -> 104 us, FP64 270 -> 179; 500 cameras and 200 000 points 204 -> 101 and 358 -> 231; 40 cameras
// and 9 001 points, FP64 36 -> 30.)
constexpr int kRedWarps = 8, kRedEntries = 36, kRedStages = 6, kRedSlots = 8;
// Beyond the resident blocks of the ring, pose-block lists of fewer records on average take a thread per entry
// (500 cameras, this sum and k_finalize, ring against thread per entry: 7.8 records a list, mixed 27 / 20 us,
// FP64 31 / 24; 16 records 32 / 30, 45 / 40; 24 records 38 / 43, 58 / 54; 750 rig cameras, 44 000 lists of 42
// records 162 / 233, 302 / 310).  So many lists that either way keeps the device busy do so up to longer ones,
// the ring taking two FP64 additions (lanes l and 32 + l) where a thread per entry takes 36 / 32 (1 800 rig
// cameras, lists of 40: 463 / 475, 897 / 700; 3 000, 248 000 lists of 45: 930 / 831, 1843 / 1328; 3 000 nadir
// cameras, 76 000 lists of 120: 700 / 1244, 1788 / 2012).
template <typename T>
static bool short_lists(const Shape& S) {
    const bool fp64 = sizeof(T) == 8, many = S.nupper >= (fp64 ? 1 << 16 : 1 << 17);
    return S.pair_partials < (many ? 64LL : fp64 ? 32LL : 20LL) * S.nupper;
}
constexpr int kRedPieces = kRedEntries / 2;  // 16-byte pieces of a full record tile
constexpr size_t kRedSmem = static_cast<size_t>(kRedWarps) * kRedStages * kRedSlots * kRedEntries * 8;

__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// records: the tile's first entry of record 0; stride: entries from one record to the next (even);
// entries: width of the tile (even, at most 36).
template <typename T>
__device__ __forceinline__ void reduce_list(Acc<T>* acc, const typename Acc<T>::part_type* __restrict__ records,
                                            size_t stride, int entries, const int* __restrict__ list, int c0, int c1,
                                            typename Acc<T>::part_type* ring) {
    const int lane = threadIdx.x & 31, pieces = entries / 2;
    const int n = c1 - c0, stages = (n + kRedSlots - 1) / kRedSlots;
    int now = lane < n ? list[c0 + lane] : 0, next = 32 + lane < n ? list[c0 + 32 + lane] : 0;
    auto issue = [&](int st) {
        if (st < stages) {
            if (st > 0 && (st & 3) == 0) {
                const int ahead = 8 * st + 32 + lane;
                now = next;
                next = ahead < n ? list[c0 + ahead] : 0;
            }
            typename Acc<T>::part_type* to = ring + static_cast<size_t>(st % kRedStages) * kRedSlots * kRedEntries;
#pragma unroll
            for (int k = 0; k < kRedSlots * kRedPieces / 32 + (kRedSlots * kRedPieces % 32 ? 1 : 0); ++k) {
                const int p = lane + 32 * k, sl = p / kRedPieces, q = p - sl * kRedPieces;
                const int rec = __shfl_sync(0xffffffffu, now, (8 * (st & 3) + min(sl, kRedSlots - 1)) & 31);
                if (sl < kRedSlots && q < pieces && kRedSlots * st + sl < n)
                    copy16_async(to + sl * kRedEntries + 2 * q, records + static_cast<size_t>(rec) * stride + 2 * q);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int st = 0; st < kRedStages - 1; ++st) issue(st);
    for (int st = 0; st < stages; ++st) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kRedStages - 2) : "memory");
        __syncwarp();
        const typename Acc<T>::part_type* v = ring + static_cast<size_t>(st % kRedStages) * kRedSlots * kRedEntries;
        const int m = min(kRedSlots, n - kRedSlots * st);
        if (m == kRedSlots && entries == kRedEntries) {
#pragma unroll
            for (int i = 0; i < kRedSlots; ++i) {
                acc[0].merge_part(v[i * kRedEntries + lane]);
                if (lane < kRedEntries - 32) acc[1].merge_part(v[i * kRedEntries + 32 + lane]);
            }
        } else {
            for (int i = 0; i < m; ++i) {
                if (lane < entries) acc[0].merge_part(v[i * kRedEntries + lane]);
                if (32 + lane < entries) acc[1].merge_part(v[i * kRedEntries + 32 + lane]);
            }
        }
        __syncwarp();
        issue(st + kRedStages - 1);
    }
}

// Entry e of camera block i's record: right-hand side, direct right-hand side, border.
template <typename T>
__device__ __forceinline__ void store_cam_sum(const Shape& S, const ReduceArgs<T>& R, int i, int e, double v) {
    if (e < 6) R.rhs[i * 6 + e] = v;
    else if (e < 12) R.direct[i * 6 + e - 6] = v;
    else {
        const int f = e - 12;  // (g * 6 + a) * ni + c
        const int g = f / (6 * S.ni), rem = f - g * 6 * S.ni, a = rem / S.ni, c = rem - a * S.ni;
        R.border[(static_cast<size_t>(i) * 6 + a) * S.nb + g * S.ni + c] = v;
        R.border_t[static_cast<size_t>(g * S.ni + c) * 6 * S.ncb + i * 6 + a] = v;
    }
}

// Sums of the chunk partials of every upper pose block, written to both CSR orientations, and of the
// per-camera partials (rhs, direct rhs and the intrinsic border rows, in tiles of 36 entries): one warp
// per block or tile.
template <typename T>
__device__ __forceinline__ void reduce_lists(const Shape& S, const DevPtrs& D, const ReduceArgs<T>& R, unsigned blk,
                                             unsigned char* smem) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto* ring = reinterpret_cast<typename Acc<T>::part_type*>(smem) +
                 static_cast<size_t>(wid) * kRedStages * kRedSlots * kRedEntries;
    const int camrec = 12 + S.ng * 6 * S.ni, tiles = (camrec + kRedEntries - 1) / kRedEntries;
    // The cameras' lists first, then the pose blocks' by decreasing length (the diagonal blocks' are as long as
    // the cameras').  While every block is resident (two on each of 152 SMs) neighbours go to different
    // blocks, so that the long lists share the FP64 pipes evenly (60 cameras, FP64 58 -> 47 us).  Beyond, they
    // share a block, which keeps its shared memory until its longest list is done: in the order of the
    // reduced pattern the diagonal blocks' lists held up the short ones that came with them (750 rig cameras,
    // 44 000 lists, 290 -> 162 us, FP64 430 -> 302; 250 cameras 83 -> 65, FP64 181 -> 123).
    const int unit = static_cast<int>(R.spread ? wid * R.list_blocks + blk : blk * kRedWarps + wid), cams = S.ncb * tiles;
    Acc<T> acc[2];
    if (unit >= cams) {
        if (unit >= cams + S.nupper) return;
        const int u = D.up_order[unit - cams];
        reduce_list<T>(acc, R.part_pair, 36, 36, D.up_contrib, D.up_contrib_begin[u], D.up_contrib_begin[u + 1], ring);
        const int t = D.up_csr_t[u];
        double* vals = R.vals + static_cast<size_t>(D.up_csr[u]) * 36;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int e = 32 * k + lane;
            if (e >= 36) continue;
            const double v = acc[k].value64();
            vals[e] = v;
            if (t >= 0) R.vals[static_cast<size_t>(t) * 36 + (e % 6) * 6 + e / 6] = v;
        }
    } else {
        const int i = unit / tiles, tile = unit - i * tiles, e0 = tile * kRedEntries;
        const int width = min(kRedEntries, camrec - e0);
        reduce_list<T>(acc, R.part_cam + e0, camrec, width, D.cam_contrib, D.cam_contrib_begin[i], D.cam_contrib_begin[i + 1],
                       ring);
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (32 * k + lane < width) store_cam_sum<T>(S, R, i, e0 + 32 * k + lane, acc[k].value64());
    }
}

// The same sums with a thread per entry, four records of its list ahead: for short lists, whose start costs
// more than their records, eight times as many threads in flight.  In the order of the reduced pattern,
// whose neighbours share chunks.
template <typename T>
__device__ __forceinline__ void reduce_entries(const Shape& S, const DevPtrs& D, const ReduceArgs<T>& R, unsigned blk) {
    const int width = 12 + S.ng * 6 * S.ni;
    Acc<T> acc;
    if (blk < R.list_blocks) {
        const long long idx = static_cast<long long>(blk) * blockDim.x + threadIdx.x;
        if (idx >= static_cast<long long>(S.nupper) * 36) return;
        const int u = static_cast<int>(idx / 36), e = static_cast<int>(idx - static_cast<long long>(u) * 36);
        const int c1 = D.up_contrib_begin[u + 1];
#pragma unroll 4
        for (int c = D.up_contrib_begin[u]; c < c1; ++c)
            acc.merge_part(R.part_pair[static_cast<size_t>(D.up_contrib[c]) * 36 + e]);
        const double v = acc.value64();
        R.vals[static_cast<size_t>(D.up_csr[u]) * 36 + e] = v;
        const int t = D.up_csr_t[u];
        if (t >= 0) R.vals[static_cast<size_t>(t) * 36 + (e % 6) * 6 + e / 6] = v;
    } else {
        const long long idx = static_cast<long long>(blk - R.list_blocks) * blockDim.x + threadIdx.x;
        if (idx >= static_cast<long long>(S.ncb) * width) return;
        const int i = static_cast<int>(idx / width), e = static_cast<int>(idx - static_cast<long long>(i) * width);
        const int c1 = D.cam_contrib_begin[i + 1];
#pragma unroll 4
        for (int c = D.cam_contrib_begin[i]; c < c1; ++c)
            acc.merge_part(R.part_cam[static_cast<size_t>(D.cam_contrib[c]) * width + e]);
        store_cam_sum<T>(S, R, i, e, acc.value64());
    }
}

// Chunk-level sums (intrinsic block, intrinsic rhs): one CTA per 32 record entries, its warps
// striding over the chunks, merged in warp order.  The block after the last tile sums the costs
// and flags.
template <typename T, int kAhead>
__device__ __forceinline__ void reduce_chunks(const Shape& S, const ReduceArgs<T>& R, unsigned blk) {
    const int nb = S.nb, chrec = nb * nb + 2 * nb;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int tiles = (chrec + 31) / 32;
    double* Cm = R.Cm;
    double* rhs_b = R.rhs + 6 * S.ncb;
    double* direct_b = R.direct + 6 * S.ncb;
    if (static_cast<int>(blk) < tiles) {
        __shared__ typename Acc<T>::part_type s_acc[8][32];
        const int e = blk * 32 + lane;
        Acc<T> acc;
        if (e < chrec) {
            // kAhead records in registers while the next ones are on their way
            const typename Acc<T>::part_type* src = R.part_chunk + e;
            typename Acc<T>::part_type v[kAhead];
            int c = wid;
            const int step = kAhead * nw;
            if (c + step - nw < S.nchunks)
#pragma unroll
                for (int i = 0; i < kAhead; ++i) v[i] = src[static_cast<size_t>(c + i * nw) * chrec];
            for (; c + step - nw < S.nchunks; c += step) {
                typename Acc<T>::part_type w[kAhead];
                if (c + 2 * step - nw < S.nchunks)
#pragma unroll
                    for (int i = 0; i < kAhead; ++i) w[i] = src[static_cast<size_t>(c + step + i * nw) * chrec];
#pragma unroll
                for (int i = 0; i < kAhead; ++i) acc.merge_part(v[i]);
#pragma unroll
                for (int i = 0; i < kAhead; ++i) v[i] = w[i];
            }
#pragma unroll 4
            for (; c < S.nchunks; c += nw) acc.merge_part(src[static_cast<size_t>(c) * chrec]);
        }
        s_acc[wid][lane] = acc.part();
        __syncthreads();
        if (wid == 0 && e < chrec) {
            Acc<T> tot;
            for (int w = 0; w < nw; ++w) tot.merge_part(s_acc[w][lane]);
            const double v = tot.value64();
            if (e < nb * nb) Cm[e] = v;
            else if (e < nb * nb + nb) rhs_b[e - nb * nb] = v;
            else direct_b[e - nb * nb - nb] = v;
        }
        return;
    }
    __shared__ double s_cost[256];
    __shared__ int s_flag[256];
    double c = 0.0;
    int f = 0;
    for (int i = threadIdx.x; i < S.nchunks; i += blockDim.x) {
        c += R.part_cost[i];
        f |= R.part_flags[i];
    }
    s_cost[threadIdx.x] = c;
    s_flag[threadIdx.x] = f;
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st) {
            s_cost[threadIdx.x] += s_cost[threadIdx.x + st];
            s_flag[threadIdx.x] |= s_flag[threadIdx.x + st];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        R.result[0] = s_cost[0];
        R.result[1] = static_cast<double>(s_flag[0]);
    }
}

// 256 threads per block (the chunk-record sum's warp count and cost buffers assume it); the block
// range decides the sum, uniformly per block: the chunk records first, they take longest.
template <typename T, bool RING>
__global__ void __launch_bounds__(256, RING ? 2 : 8) k_reduce_sums(Shape S, DevPtrs D, ReduceArgs<T> R) {
    extern __shared__ __align__(16) unsigned char reduce_smem[];
    const unsigned b = blockIdx.x;
    if (b < R.chunk_blocks) reduce_chunks<T, RING ? 16 : 4>(S, R, b);
    else if constexpr (RING) reduce_lists<T>(S, D, R, b - R.chunk_blocks, reduce_smem);
    else reduce_entries<T>(S, D, R, b - R.chunk_blocks);
}

// Intrinsic priors (assembleReferencePriors, ...ReferenceSchur.cpp:492-536) and
// finalizePrimaryDiagonal(1 + lambda, 1): positive diagonal entries scaled, empty ones set to 1.
__global__ void k_finalize(Shape S, DevPtrs D, double* __restrict__ vals, double* __restrict__ Cm,
                           double* __restrict__ rhs_b, double* __restrict__ direct_b, double* __restrict__ result,
                           double* __restrict__ host_result, double damping) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    // rig problems damp the diagonal of the rig pose blocks after the map (pb_rig.cu) instead
    if (tid < S.ncb * 6 && !S.rig) {
        const int i = tid / 6, a = tid - i * 6;
        double* d = vals + static_cast<size_t>(D.diag_pos[i]) * 36 + a * 7;
        const double v = *d;
        *d = v != 0.0 ? v * (1.0 + damping) : 1.0;
    }
    // priors of the intrinsic columns, a lane each (one thread after the other took 18 us for 16 columns);
    // their costs are added in column order
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        double total = 0.0;
        for (int c0 = 0; c0 < S.nb; c0 += 32) {
            const int col = c0 + threadIdx.x;
            double cost = 0.0;
            if (col < S.nb) {
                const int g = col / S.ni, p = S.int_cols[col - g * S.ni];
                const double* G = D.groups + static_cast<size_t>(g) * kGroupRec;
                const double w = G[2 * kP + p];
                const double r = w * (G[p] - G[kP + p]);
                cost = 0.5 * r * r;
                double* cd = Cm + col * S.nb + col;
                const double v = *cd + w * w;
                *cd = v != 0.0 ? v * (1.0 + damping) : 1.0;
                rhs_b[col] -= w * r;
                direct_b[col] -= w * r;
            }
            for (int i = 0; i < min(32, S.nb - c0); ++i) total += __shfl_sync(0xffffffffu, cost, i);
        }
        if (threadIdx.x == 0) {
            const double cost = S.nb > 0 ? result[0] + total : result[0];
            result[0] = cost;
            host_result[0] = cost;
            host_result[1] = result[1];
        }
    }
}

// Effective cameras of the current state (group intrinsics applied, makeCameraWithSharedIntrinsics,
// BundleAdjustPlaMatrixProjection.cpp:134-171) and the gauge tangent basis
// (referenceGaugeTargetTangentBasis, BundleAdjustPlaMatrixAssembly.cpp:69-99).
__device__ void group_camera(const double* __restrict__ state, const double* __restrict__ ref,
                             const double* __restrict__ G, double* __restrict__ out) {
    for (int i = 0; i < kCamStride; ++i) out[i] = state[i];
    if (!G) return;
    const double* en = G + 5 * kP;
    const double fx = en[0] != 0.0 ? G[0] : state[12];
    const double src_aspect = state[12] > 1e-12 ? state[13] / state[12] : 1.0;
    const double aspect = en[1] != 0.0 ? exp(G[1]) : src_aspect;
    out[12] = fx;
    out[13] = fx * aspect;
    out[14] = en[2] != 0.0 ? ref[14] + G[2] : state[14];
    out[15] = en[3] != 0.0 ? ref[15] + G[3] : state[15];
    for (int p = 4; p < 9; ++p)
        if (en[p] != 0.0) out[12 + p] = G[p];
}

__device__ void gauge_basis(const double* anchor_c, const double* scale_c, double* target_basis, double* world_basis) {
    const double o[3] = {anchor_c[0], -anchor_c[1], -anchor_c[2]};
    const double c[3] = {scale_c[0], -scale_c[1], -scale_c[2]};
    double u[3] = {c[0] - o[0], c[1] - o[1], c[2] - o[2]};
    const double len = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    const double il = len >= 1e-20 ? 1.0 / len : 0.0;
    for (int i = 0; i < 3; ++i) u[i] *= il;
    int axis = fabs(u[0]) > fabs(u[1]) ? 1 : 0;
    if (fabs(u[axis]) > fabs(u[2])) axis = 2;
    double ax[3] = {0, 0, 0};
    ax[axis] = 1.0;
    double s[3] = {ax[1] * u[2] - ax[2] * u[1], ax[2] * u[0] - ax[0] * u[2], ax[0] * u[1] - ax[1] * u[0]};
    const double sl = sqrt(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
    const double isl = sl >= 1e-20 ? 1.0 / sl : 0.0;
    for (int i = 0; i < 3; ++i) s[i] *= isl;
    const double f[3] = {u[1] * s[2] - u[2] * s[1], u[2] * s[0] - u[0] * s[2], u[0] * s[1] - u[1] * s[0]};
    for (int i = 0; i < 3; ++i) {
        target_basis[i] = f[i];
        target_basis[3 + i] = s[i];
    }
    world_basis[0] = f[0]; world_basis[1] = -f[1]; world_basis[2] = -f[2];
    world_basis[3] = s[0]; world_basis[4] = -s[1]; world_basis[5] = -s[2];
}

__global__ void k_effective(Shape S, DevPtrs D) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < S.ntp) {
        const double* X = D.points + static_cast<size_t>(c) * 3;
        const double sc = S.ref_param ? point_scale(X[0], X[1], X[2]) : 1.0;
        D.pscale[c] = sc;
        D.pscale_ff[c] = ff_pack(sc);
    }
    if (c < S.nc) {
        const double* G = S.ng > 0 ? D.groups + static_cast<size_t>(D.cam_group[c]) * kGroupRec : nullptr;
        double* ef = D.cams_eff + static_cast<size_t>(c) * kCamStride;
        group_camera(D.cams_state + static_cast<size_t>(c) * kCamStride, D.cams_ref + static_cast<size_t>(c) * kCamStride,
                     G, ef);
        camera_ff(ef, D.cams_ff + static_cast<size_t>(c) * kCamFF);
    }
    if (c == 0 && S.gauge_anchor >= 0 && S.gauge_scale >= 0 && S.gauge_baseline > 0.0)
        gauge_basis(D.cams_state + static_cast<size_t>(S.gauge_anchor) * kCamStride + 9,
                    D.cams_state + static_cast<size_t>(S.gauge_scale) * kCamStride + 9, D.gauge_basis + 6,
                    D.gauge_basis);
}

// Trial states for a batch of step lengths: pose retraction (applyReferenceCameraPoseStep,
// BundleAdjustPlaMatrixAssembly.cpp:130-179; gauge tangent step :101-128; the plain
// parameterisation's pose delta :1134-1136) and clamped intrinsic update (applyIntrinsicStep,
// BundleAdjustPlaMatrixModel.cpp:248-269).
// Three lanes per camera, one rotation increment's sine and cosine each (a FP64 instruction takes the
// pipe 64 cycles whatever the number of lanes: 20 cameras 10.1 -> 9.2 us), then the first of them.
constexpr int kTrialCameras = 10;  // per warp
__global__ void __launch_bounds__(32) k_trial_cameras(Shape S, DevPtrs D, const double* __restrict__ step_c, Alphas alphas, int n_alpha) {
    const int lane = threadIdx.x & 31, lead = lane / 3 * 3;
    const int idx = blockIdx.x * kTrialCameras + lane / 3;
    const bool live = lane < 3 * kTrialCameras && idx < n_alpha * S.nc;
    const int a = live ? idx / S.nc : 0, c = live ? idx - a * S.nc : 0;
    const double alpha = alphas.v[a];
    const int b = live ? D.cam_block[c] : -1;
    double sn = 0.0, cs = 1.0;
    if (b >= 0 && S.ref_param) sincos(alpha * step_c[6 * b + lane - lead], &sn, &cs);
    const double sx = __shfl_sync(0xffffffffu, sn, lead), cx = __shfl_sync(0xffffffffu, cs, lead);
    const double sy = __shfl_sync(0xffffffffu, sn, (lead + 1) & 31), cy = __shfl_sync(0xffffffffu, cs, (lead + 1) & 31);
    const double sz = __shfl_sync(0xffffffffu, sn, (lead + 2) & 31), cz = __shfl_sync(0xffffffffu, cs, (lead + 2) & 31);
    if (!live || lane != lead) return;
    // trial groups (each camera thread of the first ng cameras writes one group)
    double Gt[kGroupRec];
    const double* Gs = nullptr;
    if (S.ng > 0) {
        const int g = D.cam_group[c];
        const double* G = D.groups + static_cast<size_t>(g) * kGroupRec;
        for (int i = 0; i < kGroupRec; ++i) Gt[i] = G[i];
        for (int k = 0; k < S.ni; ++k) {
            const int p = S.int_cols[k];
            const double v = G[p] + alpha * step_c[6 * S.ncb + g * S.ni + k];
            Gt[p] = fmin(fmax(v, G[3 * kP + p]), G[4 * kP + p]);
        }
        Gs = Gt;
        if (c < S.ng) {
            const double* G2 = D.groups + static_cast<size_t>(c) * kGroupRec;
            double* out = D.groups_trial + (static_cast<size_t>(a) * S.ng + c) * kGroupRec;
            for (int i = 0; i < kGroupRec; ++i) out[i] = G2[i];
            for (int k = 0; k < S.ni; ++k) {
                const int p = S.int_cols[k];
                const double v = G2[p] + alpha * step_c[6 * S.ncb + c * S.ni + k];
                out[p] = fmin(fmax(v, G2[3 * kP + p]), G2[4 * kP + p]);
            }
        }
    }
    double pose[kCamStride];
    const double* st = D.cams_state + static_cast<size_t>(c) * kCamStride;
    for (int i = 0; i < kCamStride; ++i) pose[i] = st[i];
    if (b >= 0 && !S.ref_param) {
        // plain parameterisation: the camera's own pose delta (CameraState::applyDeltaPose,
        // BundleAdjustPlaMatrixAssembly.cpp:1134-1136), C2W' = Exp(alpha w) C2W by Rodrigues'
        // formula and C' = C + alpha dC for every refined camera, the gauge scale camera's
        // tangent coordinates included
        const double* d = step_c + 6 * b;
        const double w0 = alpha * d[0], w1 = alpha * d[1], w2 = alpha * d[2];
        const double th2 = w0 * w0 + w1 * w1 + w2 * w2;
        double A, B;
        if (th2 < 1e-16) {
            A = 1.0 - th2 / 6.0;
            B = 0.5 - th2 / 24.0;
        } else {
            const double th = sqrt(th2), sh = sin(0.5 * th);
            A = sin(th) / th;
            B = 2.0 * sh * sh / th2;  // (1 - cos th) / th^2 without the cancellation
        }
        const double K[9] = {0.0, -w2, w1, w2, 0.0, -w0, -w1, w0, 0.0};
        double E[9];
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) {
                const double kk = K[r * 3] * K[q] + K[r * 3 + 1] * K[3 + q] + K[r * 3 + 2] * K[6 + q];
                E[r * 3 + q] = (r == q ? 1.0 : 0.0) + A * K[r * 3 + q] + B * kk;
            }
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q)
                pose[r * 3 + q] = E[r * 3] * st[q] + E[r * 3 + 1] * st[3 + q] + E[r * 3 + 2] * st[6 + q];
        for (int i = 0; i < 3; ++i) pose[9 + i] = st[9 + i] + alpha * d[3 + i];
    } else if (b >= 0) {
        const double* d = step_c + 6 * b;
        // E = Rx Ry Rz
        const double E[9] = {cy * cz, -cy * sz, sy,
                             sx * sy * cz + cx * sz, -sx * sy * sz + cx * cz, -sx * cy,
                             -cx * sy * cz + sx * sz, cx * sy * sz + sx * cz, cx * cy};
        const double sg[3] = {1.0, -1.0, -1.0};
        double Tl[9];
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) Tl[r * 3 + q] = sg[r] * E[q * 3 + r] * sg[q];
        double Rn[9];
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q)
                Rn[r * 3 + q] = Tl[r * 3 + 0] * st[0 * 3 + q] + Tl[r * 3 + 1] * st[1 * 3 + q] + Tl[r * 3 + 2] * st[2 * 3 + q];
        for (int i = 0; i < 9; ++i) pose[i] = Rn[i];
        const bool tangent = c == S.gauge_scale && S.gauge_anchor >= 0 && S.gauge_baseline > 0.0;
        if (tangent) {
            const double* tb = D.gauge_basis + 6;
            const double* ac = D.cams_state + static_cast<size_t>(S.gauge_anchor) * kCamStride + 9;
            const double o[3] = {ac[0], -ac[1], -ac[2]};
            const double ce[3] = {st[9], -st[10], -st[11]};
            const double ta = alpha * d[3], tb2 = alpha * d[4];
            double dir[3];
            for (int i = 0; i < 3; ++i) dir[i] = ce[i] + tb[i] * ta + tb[3 + i] * tb2 - o[i];
            const double len = sqrt(dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2]);
            double nc[3];
            if (len < 1e-20) {
                for (int i = 0; i < 3; ++i) nc[i] = o[i];
            } else {
                const double il = 1.0 / len;
                for (int i = 0; i < 3; ++i) nc[i] = o[i] + dir[i] * il * S.gauge_baseline;
            }
            pose[9] = nc[0];
            pose[10] = -nc[1];
            pose[11] = -nc[2];
        } else {
            pose[9] = st[9] + alpha * d[3];
            pose[10] = st[10] + alpha * d[4];
            pose[11] = st[11] + alpha * d[5];
        }
    }
    group_camera(pose, D.cams_ref + static_cast<size_t>(c) * kCamStride, Gs,
                 D.cams_trial + (static_cast<size_t>(a) * S.nc + c) * kCamStride);
}

// True in every thread of the block that is the last of `blocks` to come here: the partial results that the
// others wrote before are visible to it.  The ticket is zero again afterwards.
__device__ __forceinline__ bool last_block(unsigned* ticket, unsigned blocks) {
    __shared__ unsigned s_ticket;
    if (threadIdx.x == 0) {
        __threadfence();
        s_ticket = atomicInc(ticket, blocks - 1);
    }
    __syncthreads();
    if (s_ticket != blocks - 1) return false;
    __threadfence();
    return true;
}

// Objective of the trial states: image costs (FP64) per step length (blockIdx.y), block partials.
// FP64-pipe-bound: see the objective in pb_device.cuh for the form of a term.  A thread takes every
// (grid.x x block)-th observation; part holds the sums of step length a at a * gridDim.x and, from
// kMaxAlpha * gridDim.x on, the blocks' invalid-projection marks in the same order.  The last block of a
// step length adds them up in a fixed order (256 interleaved sums, two per thread) with the intrinsic priors
// of the trial groups (assemblePrimaryPriors cost, BundleAdjustPlaMatrixAssemblySurvey.cpp:43-91); a kernel
// of its own for it took as long as a small problem's objective (20 cameras: 7.6 + 3.5 us and the gap between them, now 10.2).
constexpr int kCostThreads = 128;
__global__ void __launch_bounds__(kCostThreads) k_cost_batch(Shape S, DevPtrs D, const double* __restrict__ step_p,
                                                             Alphas alphas, int use_trial, double c2,
                                                             double ic2, int plain, double* __restrict__ part,
                                                             unsigned* __restrict__ tickets,
                                                             double* __restrict__ out) {
    __shared__ double s_c[kCostThreads / 16];
    __shared__ int s_bad[kCostThreads / 32];
    const int a = blockIdx.y;
    const double* cams = use_trial ? D.cams_trial + static_cast<size_t>(a) * S.nc * kCamStride : D.cams_eff;
    const double alpha = use_trial ? alphas.v[a] : 0.0;
    RobustSum acc;
    double targets = 0.0;  // control-point costs
    int bad = 0;
    const long long stride = static_cast<long long>(gridDim.x) * kCostThreads;
    for (long long o = static_cast<long long>(blockIdx.x) * kCostThreads + threadIdx.x; o < S.nop; o += stride) {
        const int cam = D.obs_cam[o], trk = D.obs_trk[o];
        const double* X = D.points + static_cast<size_t>(trk) * 3;
        double X0 = X[0], X1 = X[1], X2 = X[2];
        if (use_trial && D.trk_free[trk]) {
            const double* dp = step_p + static_cast<size_t>(trk) * 3;
            const double f = D.pscale[trk] * alpha;
            X0 = fma(f, dp[0], X0);
            X1 = fma(f, dp[1], X1);
            X2 = fma(f, dp[2], X2);
        }
        DCam k;
        load_cam_objective<true>(cams + static_cast<size_t>(cam) * kCamStride, k);
        double s;
        if (!weighted_square64(k, X0, X1, X2, D.obs_u[o], D.obs_v[o], D.obs_w[o], s) ||
            !acc.add(s, S.loss, S.loss_scale, c2, ic2, plain != 0)) {
            bad = 1;
            continue;
        }
        if (S.ncp > 0 && o == D.trk_obs_begin[trk]) {
            // the track's control points, once per track (its first observation's thread); a
            // term that is not finite is skipped (BundleAdjustPlaMatrixAssembly.cpp:674-690)
            for (int q = D.trk_cp_begin[trk]; q < D.trk_cp_begin[trk + 1]; ++q) {
                double r[3], cc, cw;
                if (cp_eval(D.cp_rec + static_cast<size_t>(q) * 12, X0, X1, X2, S.cp_huber, r, cc, cw)) targets += cc;
            }
        }
    }
    __syncwarp();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double v = acc.value(S.loss, c2, plain != 0);
    if (S.ncp > 0) v += targets;
    v = warp_sum(v);
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
        s_c[wid] = v;
        s_bad[wid] = bad;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const size_t at = static_cast<size_t>(a) * gridDim.x + blockIdx.x;
        part[at] = (s_c[0] + s_c[1]) + (s_c[2] + s_c[3]);
        part[static_cast<size_t>(kMaxAlpha) * gridDim.x + at] = s_bad[0] | s_bad[1] | s_bad[2] | s_bad[3];
    }
    if (!last_block(tickets + a, gridDim.x)) return;
    const int nblocks = gridDim.x, tid = threadIdx.x;
    const double* sums = part + static_cast<size_t>(a) * nblocks;
    const double* marks = part + static_cast<size_t>(kMaxAlpha + a) * nblocks;
    double half[2] = {0.0, 0.0};  // sums tid and tid + 128 of the 256
    bad = 0;
#pragma unroll 5
    for (int i = tid; i < nblocks; i += 2 * kCostThreads) {
        half[0] += __ldcg(sums + i);
        bad |= __double_as_longlong(__ldcg(marks + i)) != 0;
        if (i + kCostThreads < nblocks) {
            half[1] += __ldcg(sums + i + kCostThreads);
            bad |= __double_as_longlong(__ldcg(marks + i + kCostThreads)) != 0;
        }
    }
    if (tid < S.nb) {  // (at most 36 columns)
        const int g = tid / S.ni, p = S.int_cols[tid - g * S.ni];
        const double* G = (use_trial ? D.groups_trial + static_cast<size_t>(a) * S.ng * kGroupRec : D.groups) +
                          static_cast<size_t>(g) * kGroupRec;
        const double r = G[2 * kP + p] * (G[p] - G[kP + p]);
        half[0] = fma(0.5 * r, r, half[0]);
    }
    half[0] = warp_sum(half[0]);
    half[1] = warp_sum(half[1]);
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
        s_c[wid] = half[0];
        s_c[wid + kCostThreads / 32] = half[1];
        s_bad[wid] = bad;
    }
    __syncthreads();
    if (tid == 0) {
        double total = half[0];
        for (int w = 1; w < kCostThreads / 16; ++w) total += s_c[w];
        bad = s_bad[0] | s_bad[1] | s_bad[2] | s_bad[3];
        out[a] = bad ? __longlong_as_double(0x7ff0000000000000ll) : total;
    }
}
static_assert(kCostThreads == 128 && kMaxNB <= kCostThreads, "four warps' sums; a thread per intrinsic column");

// Back-substitution (recoverReferencePointSteps, ...ReferenceSchur.cpp:982-1082), one thread per
// track:  dp = R^-T (q - R^-1 u),  u = sum_o w J_p^T (J_o dc).
// Per observation o of an eliminated track: the term Y_o^T A_o dc (3 values) of its track's sum,
// one thread per observation, FP64 accumulation.  The FP64 pipe bounds it, 2 (6 + ni) + 6 products an
// observation; the mixed path's records widen on the integer pipe (500 cameras, 1.3 million observations:
// 168 -> 83 us; the records staged in shared memory by consecutive lanes took the same).
template <typename T>
__global__ void __launch_bounds__(256) k_backsub_terms(Shape S, DevPtrs D, const T* __restrict__ obs_rec,
                                                       const double* __restrict__ step_c, double* __restrict__ terms) {
    const long long o = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (o >= S.nop) return;
    const int nA = 6 + S.ni, stride = 2 * nA + 6;
    const int cam = D.obs_cam[o];
    const T* rec = obs_rec + static_cast<size_t>(o) * stride;
    double e0 = 0.0, e1 = 0.0;
    const int b = D.cam_block[cam];
    if (b >= 0)
        for (int a = 0; a < 6; ++a) {
            const double dcv = step_c[6 * b + a];
            e0 = fma(f64_of(rec[a]), dcv, e0);
            e1 = fma(f64_of(rec[nA + a]), dcv, e1);
        }
    const int g = S.ng > 0 ? D.cam_group[cam] : -1;
    if (g >= 0)
        for (int a = 0; a < S.ni; ++a) {
            const double dcv = step_c[6 * S.ncb + g * S.ni + a];
            e0 = fma(f64_of(rec[6 + a]), dcv, e0);
            e1 = fma(f64_of(rec[nA + 6 + a]), dcv, e1);
        }
    const T* Y = rec + 2 * nA;
    double* u = terms + static_cast<size_t>(o) * 3;
    u[0] = f64_of(Y[0]) * e0 + f64_of(Y[3]) * e1;
    u[1] = f64_of(Y[1]) * e0 + f64_of(Y[4]) * e1;
    u[2] = f64_of(Y[2]) * e0 + f64_of(Y[5]) * e1;
}

// track:  dp = R^-T (q - R^-1 u),  u = sum_o w J_p^T (J_o dc).
// The last block adds up the blocks' parts of the directional decrease and of the squared point steps and
// the camera-side terms (dc . direct rhs, squared camera step), in a fixed order (20 cameras, 2 000 points: 9.1 + 5.1 us as two kernels, now 11.5).
constexpr int kBacksubThreads = 128;
__global__ void __launch_bounds__(kBacksubThreads) k_back_substitute(Shape S, DevPtrs D,
                                                                     const double* __restrict__ trk_data,
                                                                     const double* __restrict__ terms,
                                                                     double* __restrict__ step_p,
                                                                     double* __restrict__ step_e, double* __restrict__ part,
                                                                     const double* __restrict__ step_c,
                                                                     const double* __restrict__ direct64,
                                                                     unsigned* __restrict__ ticket,
                                                                     double* __restrict__ out) {
    // Point steps dp = V^-1 (g_p - W^T dc) = R^-T (q - sum_o Y_o^T A_o dc) from the records the
    // assembly kept (A = [J_pose | J_intr] rows and Y = w Jp R^-T of every observation), with
    // FP64 accumulation (recoverReferencePointSteps, BundleAdjustPlaMatrixReferenceSchur.cpp:982-1082).
    // The per-observation terms come from k_backsub_terms and are summed here in observation order,
    // the order of a single-thread loop over the track.
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double dd = 0.0, ss = 0.0;
    if (t < S.ntp && D.trk_block[t] >= 0) {
        double u0 = 0.0, u1 = 0.0, u2 = 0.0;
        const int oe = D.trk_obs_begin[t + 1];
#pragma unroll 4
        for (int o = D.trk_obs_begin[t]; o < oe; ++o) {
            const double* u = terms + static_cast<size_t>(o) * 3;
            u0 += u[0];
            u1 += u[1];
            u2 += u[2];
        }
        const double* td = trk_data + static_cast<size_t>(t) * kTrackRec;
        const double i00 = td[0], i10 = td[1], i11 = td[2], i20 = td[3], i21 = td[4], i22 = td[5];
        const double v0 = td[6] - u0;
        const double v1 = td[7] - u1;
        const double v2 = td[8] - u2;
        const double p0 = i00 * v0 + i10 * v1 + i20 * v2;
        const double p1 = i11 * v1 + i21 * v2;
        const double p2 = i22 * v2;
        step_p[static_cast<size_t>(t) * 3 + 0] = p0;
        step_p[static_cast<size_t>(t) * 3 + 1] = p1;
        step_p[static_cast<size_t>(t) * 3 + 2] = p2;
        if (step_e) {  // the caller's order (a scatter on the host: 200 000 points 1 220 -> 262 us a call)
            double* e = step_e + static_cast<size_t>(D.trk_block[t]) * 3;
            e[0] = p0;
            e[1] = p1;
            e[2] = p2;
        }
        dd = td[9] * p0 + td[10] * p1 + td[11] * p2;
        ss = p0 * p0 + p1 * p1 + p2 * p2;
    } else if (t < S.ntp) {
        step_p[static_cast<size_t>(t) * 3 + 0] = 0.0;
        step_p[static_cast<size_t>(t) * 3 + 1] = 0.0;
        step_p[static_cast<size_t>(t) * 3 + 2] = 0.0;
    }
    constexpr int kWarps = kBacksubThreads / 32;
    __shared__ double s_sum[3][kWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    dd = warp_sum(dd);
    ss = warp_sum(ss);
    if (lane == 0) {
        s_sum[0][wid] = dd;
        s_sum[1][wid] = ss;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        reinterpret_cast<double2*>(part)[blockIdx.x] =
            make_double2((s_sum[0][0] + s_sum[0][1]) + (s_sum[0][2] + s_sum[0][3]),
                         (s_sum[1][0] + s_sum[1][1]) + (s_sum[1][2] + s_sum[1][3]));
    if (!last_block(ticket, gridDim.x)) return;
    double sum[3] = {0.0, 0.0, 0.0};
    const int nblocks = gridDim.x;
#pragma unroll 4
    for (int i = threadIdx.x; i < nblocks; i += kBacksubThreads) {
        const double2 v = __ldcg(reinterpret_cast<const double2*>(part) + i);
        sum[0] += v.x;
        sum[1] += v.y;
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < S.n; i += kBacksubThreads) {
        const double c = step_c[i];
        sum[0] = fma(c, direct64[i], sum[0]);
        sum[2] = fma(c, c, sum[2]);
    }
    for (int i = 0; i < 3; ++i) {
        const double v = warp_sum(sum[i]);
        if (lane == 0) s_sum[i][wid] = v;
    }
    __syncthreads();
    // directional decrease, sum of squared point steps, sum of squared camera and intrinsic steps
    if (threadIdx.x < 3) {
        const double* v = s_sum[threadIdx.x];
        out[threadIdx.x] = (v[0] + v[1]) + (v[2] + v[3]);
    }
}
static_assert(kBacksubThreads == 128, "k_back_substitute adds the sums of four warps");

// Accept trial `a`: poses and effective cameras from the trial, groups, points += s(X) alpha dp.  The first
// blocks take a camera per warp, a lane per value (a thread per camera went through 32 values and 21
// conversions one after the other: 20 cameras 14.2 -> 5.8 us), the others a point or group value per thread.
constexpr int kAcceptThreads = 64;
__global__ void __launch_bounds__(kAcceptThreads) k_accept(Shape S, DevPtrs D, const double* __restrict__ step_p,
                                                           double alpha, int a) {
    constexpr int kCams = kAcceptThreads / 32;
    const int cam_blocks = (S.nc + kCams - 1) / kCams;
    if (static_cast<int>(blockIdx.x) < cam_blocks) {
        const int c = blockIdx.x * kCams + (threadIdx.x >> 5), q = threadIdx.x & 31;
        if (c >= S.nc) return;
        const double* tr = D.cams_trial + (static_cast<size_t>(a) * S.nc + c) * kCamStride;
        const double v = tr[q];
        if (q < 12) D.cams_state[static_cast<size_t>(c) * kCamStride + q] = v;
        D.cams_eff[static_cast<size_t>(c) * kCamStride + q] = v;
        if (q < kCamFF) D.cams_ff[static_cast<size_t>(c) * kCamFF + q] = camera_ff_value(q, v);
        // the gauge tangent basis follows the accepted state (referenceGaugeTargetTangentBasis is
        // evaluated on the current cameras, BundleAdjustPlaMatrixAssembly.cpp:69-99, :110, :205);
        // read from the trial records, which this kernel does not write
        if (q == 0 && c == S.gauge_scale && S.gauge_anchor >= 0 && S.gauge_baseline > 0.0)
            gauge_basis(D.cams_trial + (static_cast<size_t>(a) * S.nc + S.gauge_anchor) * kCamStride + 9, tr + 9,
                        D.gauge_basis + 6, D.gauge_basis);
        return;
    }
    const int i = (blockIdx.x - cam_blocks) * kAcceptThreads + threadIdx.x;
    if (i < S.ng * kGroupRec) D.groups[i] = D.groups_trial[static_cast<size_t>(a) * S.ng * kGroupRec + i];
    if (i < S.ntp && D.trk_free[i]) {
        double* X = D.points + static_cast<size_t>(i) * 3;
        const double f = D.pscale[i] * alpha;
        X[0] += f * step_p[static_cast<size_t>(i) * 3 + 0];
        X[1] += f * step_p[static_cast<size_t>(i) * 3 + 1];
        X[2] += f * step_p[static_cast<size_t>(i) * 3 + 2];
        const double sc = S.ref_param ? point_scale(X[0], X[1], X[2]) : 1.0;
        D.pscale[i] = sc;
        D.pscale_ff[i] = ff_pack(sc);
    }
}
static_assert(kCamStride == 32, "a lane per value of a camera record");

// Strict per-track RMS (strictTrackRms, BundleAdjustQuality.cpp:302-364) over the raw observations.
// `proc_of_track` maps an original track to its processing index (-1: use the initial point).
__global__ void k_strict_rms(Shape S, DevPtrs D, const double* __restrict__ cams, const double* __restrict__ init_points,
                             const int* __restrict__ proc_of_track, int use_state, int nt, double* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    double X0, X1, X2;
    const int pidx = use_state ? proc_of_track[t] : -1;
    if (use_state && pidx < 0) { out[t] = __longlong_as_double(0x7ff0000000000000ll); return; }
    if (pidx >= 0) {
        X0 = D.points[3 * pidx]; X1 = D.points[3 * pidx + 1]; X2 = D.points[3 * pidx + 2];
    } else {
        X0 = init_points[3 * t]; X1 = init_points[3 * t + 1]; X2 = init_points[3 * t + 2];
    }
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    if (!isfinite(X0) || !isfinite(X1) || !isfinite(X2)) { out[t] = inf; return; }
    double sum = 0.0;
    int count = 0, first = -1;
    bool second = false;
    for (long long k = D.raw_offsets[t]; k < D.raw_offsets[t + 1]; ++k) {
        const double w = D.raw_w[k];
        if (!(w > 0.0)) continue;
        if (D.raw_bad[k]) { out[t] = inf; return; }
        const int cam = D.raw_cam[k];
        DCam c;
        load_cam(cams + static_cast<size_t>(cam) * kCamStride, c);
        Proj p;
        if (!project64(c, X0, X1, X2, p)) { out[t] = inf; return; }
        const double du = p.px - D.raw_u[k], dv = p.py - D.raw_v[k];
        sum += w * (du * du + dv * dv);
        count += 2;
        if (first < 0) first = cam;
        else if (cam != first) second = true;
    }
    out[t] = (count < 4 || !second) ? inf : sqrt(sum / count);
}

// Per-observation linearisation in the original observation order (parity export of kernel (a)).
template <typename T>
__global__ void k_linearize_export(Shape S, DevPtrs D, double* __restrict__ res, double* __restrict__ jp,
                                   double* __restrict__ jpose, double* __restrict__ ji, double* __restrict__ nw,
                                   double* __restrict__ cost, signed char* __restrict__ valid) {
    const long long o = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (o >= S.nop) return;
    const int cam = D.obs_cam[o], trk = D.obs_trk[o];
    const long long k = D.obs_orig[o];
    DCam c;
    load_cam(D.cams_eff + static_cast<size_t>(cam) * kCamStride, c);
    const double* X = D.points + static_cast<size_t>(trk) * 3;
    const bool tangent = cam == S.gauge_scale && S.gauge_anchor >= 0 && S.gauge_baseline > 0.0;
    Lin<T> L;
    const bool ok = linearize_obs<T>(c, X[0], X[1], X[2], D.pscale[trk], D.obs_u[o], D.obs_v[o], D.obs_w[o], S.loss,
                                     S.loss_scale, tangent, !S.ref_param, D.gauge_basis, S.ni, S.int_cols, true, L);
    valid[k] = ok ? 1 : 0;
    if (!ok) return;
    res[2 * k] = static_cast<double>(L.r0);
    res[2 * k + 1] = static_cast<double>(L.r1);
    for (int i = 0; i < 6; ++i) jp[6 * k + i] = static_cast<double>(L.Jp[i]);
    for (int i = 0; i < 2 * kP; ++i) jpose[2 * kP * k + i] = 0.0;
    if (D.cam_block[cam] >= 0)
        for (int r = 0; r < 2; ++r)
            for (int i = 0; i < 6; ++i) jpose[2 * kP * k + r * kP + i] = static_cast<double>(L.Jc[r * 6 + i]);
    for (int i = 0; i < 2 * kP; ++i) ji[2 * kP * k + i] = 0.0;
    for (int r = 0; r < 2; ++r)
        for (int i = 0; i < S.ni; ++i) ji[2 * kP * k + r * kP + S.int_cols[i]] = static_cast<double>(L.Ji[r * kMaxNI + i]);
    nw[k] = static_cast<double>(L.w);
    cost[k] = L.cost;
    if constexpr (std::is_same<T, float>::value) {
        // the mixed path's weight and gradient chain are float-float (the assembly's phase A);
        // its residual, Jacobians and weight replace the FP64 ones, the cost stays the FP64 one
        Proj pr;
        LinFF F;
        const bool okf = project64(c, X[0], X[1], X[2], pr) &&
                         linearize_obs_ff(pr, D.obs_u[o], D.obs_v[o], D.cams_ff + static_cast<size_t>(cam) * kCamFF,
                                          ffl(D.pscale_ff[trk]), ffl(D.obs_w_ff[o]), S.loss,
                                          ff{S.loss_scale_hi, S.loss_scale_lo}, tangent, !S.ref_param, D.gauge_basis,
                                          S.ni, S.int_cols, F);
        valid[k] = okf ? 1 : 0;
        if (!okf) return;
        res[2 * k] = static_cast<double>(F.r0.hi) + static_cast<double>(F.r0.lo);
        res[2 * k + 1] = static_cast<double>(F.r1.hi) + static_cast<double>(F.r1.lo);
        for (int i = 0; i < 6; ++i) jp[6 * k + i] = static_cast<double>(F.Jp[i]);
        if (D.cam_block[cam] >= 0)
            for (int r = 0; r < 2; ++r)
                for (int i = 0; i < 6; ++i) jpose[2 * kP * k + r * kP + i] = static_cast<double>(F.Jc[r * 6 + i]);
        for (int r = 0; r < 2; ++r)
            for (int i = 0; i < S.ni; ++i)
                ji[2 * kP * k + r * kP + S.int_cols[i]] = static_cast<double>(F.Ji[r * kMaxNI + i]);
        nw[k] = static_cast<double>(F.w.hi) + static_cast<double>(F.w.lo);
    }
}

// ---------------------------------------------------------------- launchers
template <typename T>
static AsmOutT<T> typed(const AsmOut& o) {
    using P = typename Acc<T>::part_type;
    return {static_cast<P*>(o.part_pair_v), static_cast<P*>(o.part_cam_v), static_cast<P*>(o.part_chunk_v),
            o.part_cost, o.part_flags, static_cast<double*>(o.trk_data_v), static_cast<T*>(o.obs_rec_v)};
}

template <typename T>
void launch_reduce_sums(const Shape& S, const DevPtrs& D, const AsmOut& O, const RedOut<double>& R, cudaStream_t st) {
    const AsmOutT<T> P = typed<T>(O);
    ReduceArgs<T> A;
    A.part_pair = P.part_pair;
    A.part_cam = P.part_cam;
    A.part_chunk = P.part_chunk;
    A.part_cost = O.part_cost;
    A.part_flags = O.part_flags;
    A.vals = R.vals;
    A.rhs = R.rhs;
    A.direct = R.direct;
    A.border = R.border;
    A.border_t = R.border_t;
    A.Cm = R.Cm;
    A.result = R.result;
    const int tiles = (12 + S.ng * 6 * S.ni + kRedEntries - 1) / kRedEntries;
    const int chrec = S.nb * S.nb + 2 * S.nb;
    A.chunk_blocks = static_cast<unsigned>((chrec + 31) / 32) + 1;
    const unsigned list_blocks = static_cast<unsigned>((S.nupper + S.ncb * tiles + kRedWarps - 1) / kRedWarps);
    static std::once_flag once[64];
    int dev = 0;
    cudaGetDevice(&dev);
    std::call_once(once[dev & 63], [] {
        cudaFuncSetAttribute(k_reduce_sums<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kRedSmem));
    });
    A.list_blocks = list_blocks;
    A.spread = list_blocks <= 2 * 152;
    if (A.spread || !short_lists<T>(S)) {
        k_reduce_sums<T, true><<<A.chunk_blocks + list_blocks, 256, kRedSmem, st>>>(S, D, A);
        return;
    }
    A.list_blocks = static_cast<unsigned>((36LL * S.nupper + 255) / 256);
    const unsigned cam_blocks = static_cast<unsigned>((static_cast<long long>(S.ncb) * (12 + S.ng * 6 * S.ni) + 255) / 256);
    k_reduce_sums<T, false><<<A.chunk_blocks + A.list_blocks + cam_blocks, 256, 0, st>>>(S, D, A);
}

template <typename T>
void launch_reduce(const Shape& S, const DevPtrs& D, const AsmOut& O, const RedOut<double>& R, double damping,
                   double* host_result, cudaStream_t st) {
    launch_reduce_sums<T>(S, D, O, R, st);
    const int nf = std::max(S.ncb * 6, 1);
    k_finalize<<<(nf + 255) / 256, 256, 0, st>>>(S, D, R.vals, R.Cm, R.rhs + 6 * S.ncb, R.direct + 6 * S.ncb, R.result,
                                                  host_result, damping);
}

// The fixed-order sums of FP64 chunk partials of launch_reduce, without the damping and prior
// finalisation (the backward pass finalises its exact Hessian itself).
void launch_reduce_sums64(const Shape& S, const DevPtrs& D, const AsmOut& O, const RedOut<double>& R, cudaStream_t st) {
    launch_reduce_sums<double>(S, D, O, R, st);
}

int backsub_blocks(int ntp) { return std::max(1, (ntp + kBacksubThreads - 1) / kBacksubThreads); }

template <typename T>
void launch_back_substitute(const Shape& S, const DevPtrs& D, const double* trk_data, const T* obs_rec, const double* step_c,
                            double* step_p, double* step_e, double* terms, double* part, const double* direct64,
                            unsigned* ticket, double* out, cudaStream_t st) {
    const int nblk = backsub_blocks(S.ntp);
    if (S.nop > 0)
        k_backsub_terms<T><<<static_cast<unsigned>((S.nop + 255) / 256), 256, 0, st>>>(S, D, obs_rec, step_c, terms);
    k_back_substitute<<<nblk, kBacksubThreads, 0, st>>>(S, D, trk_data, terms, step_p, step_e, part, step_c, direct64,
                                                        ticket, out);
}

template <typename T>
void launch_linearize_export(const Shape& S, const DevPtrs& D, double* res, double* jp, double* jpose, double* ji,
                             double* nw, double* cost, signed char* valid, cudaStream_t st) {
    if (S.nop == 0) return;
    k_linearize_export<T><<<static_cast<unsigned>((S.nop + 255) / 256), 256, 0, st>>>(S, D, res, jp, jpose, ji, nw, cost,
                                                                                       valid);
}

__global__ void k_gather_obs(long long nop, int ntp, DevPtrs D) {
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < nop) {
        const int k = D.obs_orig[i];
        D.obs_cam[i] = D.raw_cam[k];
        D.obs_u[i] = D.raw_u[k];
        D.obs_v[i] = D.raw_v[k];
        D.obs_w[i] = D.raw_w[k];
        D.obs_w_ff[i] = ff_pack(D.raw_w[k]);
    }
    if (i < ntp)
        for (int o = D.trk_obs_begin[i]; o < D.trk_obs_begin[i + 1]; ++o) D.obs_trk[o] = static_cast<int>(i);
}

void launch_gather_obs(long long nop, int ntp, const DevPtrs& D, cudaStream_t st) {
    const long long n = std::max<long long>(std::max<long long>(nop, ntp), 1);
    k_gather_obs<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(nop, ntp, D);
}

// The dense symmetric matrix of a reduced system: pose blocks by their CSR row, the border in both
// triangles, the intrinsic block; entries without a block are zero.  A CTA per row: its zeros and blocks
// are written by consecutive lanes, so that the caller's copy is one transfer instead of a scatter on the
// host (234 unknowns 75 -> 43 us a call).
__global__ void __launch_bounds__(128) k_dense_rows(PcgSystem<double> A, double* __restrict__ out) {
    const int r = blockIdx.x, n6 = 6 * A.ncb, n = n6 + A.nb, tid = threadIdx.x;
    double* o = out + static_cast<size_t>(r) * n;
    if (r >= n6) {
        const int a = r - n6;
        for (int c = tid; c < n; c += 128)
            o[c] = c < n6 ? A.border[static_cast<size_t>(c) * A.nb + a] : A.Cm[static_cast<size_t>(a) * A.nb + c - n6];
        return;
    }
    for (int c = tid; c < n; c += 128) o[c] = c < n6 ? 0.0 : A.border[static_cast<size_t>(r) * A.nb + c - n6];
    __syncthreads();
    const int i = r / 6, a = r - 6 * i;
    const int p0 = A.row_ptr[i], m = 6 * (A.row_ptr[i + 1] - p0);
    for (int e = tid; e < m; e += 128) {
        const int p = p0 + e / 6, b = e % 6;
        o[6 * A.col_idx[p] + b] = A.vals[static_cast<size_t>(p) * 36 + 6 * a + b];
    }
}

void launch_dense_rows(const PcgSystem<double>& sys, double* out, cudaStream_t st) {
    const int n = 6 * sys.ncb + sys.nb;
    if (n > 0) k_dense_rows<<<n, 128, 0, st>>>(sys, out);
}

// The points of every track in the caller's order: the state of the processed tracks, the initial points of
// the others.
__global__ void __launch_bounds__(128) k_points_out(int nt, const int* __restrict__ proc_of_track,
                                                    const double* __restrict__ points, const double* __restrict__ init,
                                                    double* __restrict__ out) {
    const long long i = static_cast<long long>(blockIdx.x) * 128 + threadIdx.x;
    if (i >= 3ll * nt) return;
    const int t = static_cast<int>(i / 3), p = proc_of_track[t];
    out[i] = p >= 0 ? points[3ll * p + (i - 3ll * t)] : init[i];
}

void launch_points_out(int nt, const int* proc_of_track, const double* points, const double* init, double* out,
                       cudaStream_t st) {
    if (nt > 0) k_points_out<<<static_cast<unsigned>((3ll * nt + 127) / 128), 128, 0, st>>>(nt, proc_of_track, points, init, out);
}

void launch_effective(const Shape& S, const DevPtrs& D, cudaStream_t st) {
    const int n = std::max(std::max(S.nc, S.ntp), 1);
    k_effective<<<(n + 63) / 64, 64, 0, st>>>(S, D);
}

// Blocks per step length of k_cost_batch: eight resident blocks on each of 152 SMs share the batch;
// beyond, a thread takes several observations (one log1p per thread of a Cauchy sum, and at most
// 1216 partials a step length for the final sum).
static int cost_blocks(long long nop, int n_alpha) {
    const long long need = (nop + kCostThreads - 1) / kCostThreads;
    return static_cast<int>(std::max<long long>(1, std::min<long long>(need, std::max(152, kCostMaxBlocks / n_alpha))));
}

void launch_cost(const Shape& S, const DevPtrs& D, const double* step_c, const double* step_p, const Alphas& alphas,
                 int n_alpha, int use_trial, double* part, unsigned* tickets, double* out, cudaStream_t st,
                 const RigDev* rig) {
    if (use_trial) {
        const int n = n_alpha * S.nc;
        k_trial_cameras<<<(n + kTrialCameras - 1) / kTrialCameras, 32, 0, st>>>(S, D, step_c, alphas, n_alpha);
        // rig cameras: poses composed from the trial captures and sensors
        if (rig) launch_rig_trial(*rig, S.nc, alphas, n_alpha, D.cams_trial, st);
    }
    const int nblk = cost_blocks(S.nop, n_alpha);
    const double c2 = S.loss_scale * S.loss_scale, ic2 = 1.0 / c2;
    const int plain = S.loss != 0 && std::isnormal(c2) && std::isnormal(ic2) ? 1 : 0;
    k_cost_batch<<<dim3(nblk, n_alpha), kCostThreads, 0, st>>>(S, D, step_p, alphas, use_trial, c2, ic2, plain, part,
                                                                tickets, out);
}

void launch_accept(const Shape& S, const DevPtrs& D, const double* step_p, double alpha, int a, cudaStream_t st) {
    const int cam_blocks = (S.nc + kAcceptThreads / 32 - 1) / (kAcceptThreads / 32);
    const int n = std::max(S.ntp, S.ng * kGroupRec);
    const int blocks = cam_blocks + (n + kAcceptThreads - 1) / kAcceptThreads;
    if (blocks > 0) k_accept<<<blocks, kAcceptThreads, 0, st>>>(S, D, step_p, alpha, a);
}

void launch_strict_rms(const Shape& S, const DevPtrs& D, const double* cams, const double* init_points,
                       const int* proc_of_track, int use_state, int nt, double* out, cudaStream_t st) {
    k_strict_rms<<<(nt + 63) / 64, 64, 0, st>>>(S, D, cams, init_points, proc_of_track, use_state, nt, out);
}

// ---------------------------------------------------------------- quality finalisation
// finalizeBundleAdjustResult (BundleAdjustQuality.cpp:403-502) on the device: the strict RMS
// after the solve of every active track, the filter threshold max(filterMaxReprojError,
// filterSigmaFactor * median of the finite RMS values), the valid mask and the mean RMS of the
// kept tracks.  The median is an exact order statistic (radix select over the bit patterns of
// the non-negative doubles, which order like their values), the mean of the two middle values
// for an even count, as the host's finite median.

constexpr int kQualityThreads = 1024;

__device__ __forceinline__ bool quality_candidate(const signed char* active, const double* rms, int t) {
    return active[t] && isfinite(rms[t]);
}

// The two middle order statistics of the candidate values, ranks h - 1 and h (h alone for an odd count), by
// a radix select over the bit patterns: 11 bits a pass.  Two passes over the tracks leave few values that
// share the leading 22 bits; those are listed in shared memory, and the other passes run on the list (on
// the tracks again when they do not fit).  A sweep for the largest smaller value gives rank h - 1.  (Eight
// passes of eight bits for each of the two ranks: 283 -> 98 us for 40 000 tracks.)
constexpr int kSelectBits = 11, kSelectBins = 1 << kSelectBits, kSelectList = 4096;
struct SelectSmem {
    unsigned int hist[kSelectBins];
    unsigned long long list[kSelectList];
    unsigned long long prefix, below;
    unsigned int warp_sum[kQualityThreads / 32];
    unsigned int rank, count, listed;
};

// Applies f(bits) to every candidate value: from the list when `listed`, else from the tracks.
template <typename F>
__device__ __forceinline__ void select_sweep(int nt, const signed char* __restrict__ active, const double* __restrict__ rms,
                                             const SelectSmem& q, bool listed, F f) {
    if (listed) {
        for (int i = threadIdx.x; i < static_cast<int>(q.listed); i += blockDim.x) f(q.list[i]);
        return;
    }
    constexpr int kAhead = 8;
    for (int t0 = threadIdx.x; t0 < nt; t0 += kAhead * blockDim.x) {
        double v[kAhead];
        signed char on[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int t = t0 + i * blockDim.x;
            on[i] = t < nt ? active[t] : 0;
            v[i] = t < nt ? rms[t] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if (on[i] && isfinite(v[i])) f(static_cast<unsigned long long>(__double_as_longlong(v[i])));
    }
}

// Value of rank h, and the largest candidate value below it, or that value itself when rank h - 1 is equal
// to it (`lower`).  All threads take part.
__device__ double quality_select(int nt, const signed char* active, const double* rms, unsigned int h, SelectSmem& q,
                                 double& lower) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long prefix = 0ull, mask = 0ull;
    bool listed = false;
    if (tid == 0) q.rank = h;
    for (int pass = 0; pass < 6; ++pass) {
        // 64 bits: five fields of 11 and one of 9
        const int shift = pass < 5 ? 64 - kSelectBits * (pass + 1) : 0;
        const int bins = pass < 5 ? kSelectBins : 1 << 9;
        for (int i = tid; i < bins; i += blockDim.x) q.hist[i] = 0u;
        __syncthreads();
        select_sweep(nt, active, rms, q, listed, [&](unsigned long long bits) {
            if ((bits & mask) == prefix) atomicAdd(&q.hist[(bits >> shift) & (bins - 1)], 1u);
        });
        __syncthreads();
        // prefix sums over the bins (two per thread), the bin that holds the rank
        const unsigned int c0 = 2 * tid < bins ? q.hist[2 * tid] : 0u, c1 = 2 * tid + 1 < bins ? q.hist[2 * tid + 1] : 0u;
        unsigned int inc = c0 + c1;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int up = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += up;
        }
        if (lane == 31) q.warp_sum[warp] = inc;
        __syncthreads();
        unsigned int before = inc - c0 - c1;
        for (int w = 0; w < warp; ++w) before += q.warp_sum[w];
        const unsigned int r = q.rank;
        __syncthreads();
        if (r >= before && r < before + c0 + c1) {  // (one thread)
            const bool second = r >= before + c0;
            q.rank = r - before - (second ? c0 : 0u);
            q.count = second ? c1 : c0;
            q.prefix = prefix | (static_cast<unsigned long long>(2 * tid + (second ? 1 : 0)) << shift);
        }
        __syncthreads();
        prefix = q.prefix;
        mask |= static_cast<unsigned long long>(bins - 1) << shift;
        if (!listed && q.count <= kSelectList) {
            if (tid == 0) q.listed = 0u;
            __syncthreads();
            select_sweep(nt, active, rms, q, false, [&](unsigned long long bits) {
                if ((bits & mask) == prefix) q.list[atomicAdd(&q.listed, 1u)] = bits;
            });
            listed = true;
        }
        __syncthreads();
    }
    lower = __longlong_as_double(static_cast<long long>(prefix));
    if (q.rank == 0u) {  // (uniform) the value is the first of its equals: rank h - 1 lies below it
        if (tid == 0) q.below = 0ull;
        __syncthreads();
        unsigned long long best = 0ull;
        select_sweep(nt, active, rms, q, false, [&](unsigned long long bits) {
            if (bits < prefix && bits > best) best = bits;
        });
        atomicMax(&q.below, best);
        __syncthreads();
        lower = __longlong_as_double(static_cast<long long>(q.below));
    }
    return __longlong_as_double(static_cast<long long>(prefix));
}

// one CTA: out[0] = threshold, out[1] = candidate count
__global__ void __launch_bounds__(kQualityThreads) k_quality_threshold(int nt, const signed char* __restrict__ active,
                                                                       const double* __restrict__ rms, int enable,
                                                                       double max_err, double sigma,
                                                                       double* __restrict__ out) {
    __shared__ SelectSmem sel;
    __shared__ int s_count[kQualityThreads / 32];
    int cnt = 0;
    for (int t = threadIdx.x; t < nt; t += blockDim.x) cnt += quality_candidate(active, rms, t) ? 1 : 0;
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) s_count[threadIdx.x >> 5] = cnt;
    __syncthreads();
    long long n = 0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) n += s_count[w];
    double thr = __longlong_as_double(0x7ff0000000000000ll);
    if (enable) {
        thr = isfinite(max_err) && max_err >= 0.0 ? max_err : 0.0;
        if (n > 0 && isfinite(sigma) && sigma > 0.0) {
            double lower;
            const double upper = quality_select(nt, active, rms, static_cast<unsigned int>(n / 2), sel, lower);
            const double med = (n & 1) == 0 ? 0.5 * (lower + upper) : upper;
            thr = fmax(thr, sigma * med);
        }
    }
    if (threadIdx.x == 0) {
        out[0] = thr;
        out[1] = static_cast<double>(n);
    }
}

// valid mask and per-block partials (kept, sum RMS before, sum RMS after)
__global__ void __launch_bounds__(256) k_quality_filter(int nt, const signed char* __restrict__ active,
                                                        const double* __restrict__ rms_before,
                                                        const double* __restrict__ rms_after,
                                                        const double* __restrict__ thr_in, signed char* __restrict__ valid,
                                                        double* __restrict__ part) {
    __shared__ double s[3][8];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double k = 0.0, b = 0.0, a = 0.0;
    if (t < nt) {
        const double thr = thr_in[0];
        const bool v = quality_candidate(active, rms_after, t) && !(rms_after[t] > thr);
        valid[t] = v ? 1 : 0;
        if (v) {
            k = 1.0;
            b = rms_before[t];
            a = rms_after[t];
        }
    }
    const double w[3] = {warp_sum(k), warp_sum(b), warp_sum(a)};
    if ((threadIdx.x & 31) == 0)
        for (int i = 0; i < 3; ++i) s[i][threadIdx.x >> 5] = w[i];
    __syncthreads();
    if (threadIdx.x < 3) {
        double acc = 0.0;
        for (int i = 0; i < 8; ++i) acc += s[threadIdx.x][i];
        part[static_cast<size_t>(blockIdx.x) * 3 + threadIdx.x] = acc;
    }
}

// fixed-order sums of the block partials into out[2..4]
__global__ void k_quality_sums(int nblocks, const double* __restrict__ part, double* __restrict__ out) {
    __shared__ double s[3][256];
    for (int i = 0; i < 3; ++i) {
        double acc = 0.0;
        for (int b = threadIdx.x; b < nblocks; b += blockDim.x) acc += part[static_cast<size_t>(b) * 3 + i];
        s[i][threadIdx.x] = acc;
    }
    __syncthreads();
    for (int st = blockDim.x / 2; st > 0; st >>= 1) {
        if (threadIdx.x < st)
            for (int i = 0; i < 3; ++i) s[i][threadIdx.x] += s[i][threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x < 3) out[2 + threadIdx.x] = s[threadIdx.x][0];
}

size_t quality_part_size(int nt) { return static_cast<size_t>(std::max(1, (nt + 255) / 256)) * 3; }

void launch_quality(int nt, const signed char* active, const double* rms_before, const double* rms_after, int enable,
                    double max_err, double sigma, signed char* valid, double* part, double* out, cudaStream_t st) {
    k_quality_threshold<<<1, kQualityThreads, 0, st>>>(nt, active, rms_after, enable, max_err, sigma, out);
    const int nblk = std::max(1, (nt + 255) / 256);
    k_quality_filter<<<nblk, 256, 0, st>>>(nt, active, rms_before, rms_after, out, valid, part);
    k_quality_sums<<<1, 256, 0, st>>>(nblk, part, out);
}


template void launch_reduce<float>(const Shape&, const DevPtrs&, const AsmOut&, const RedOut<double>&, double, double*,
                                   cudaStream_t);
template void launch_reduce<double>(const Shape&, const DevPtrs&, const AsmOut&, const RedOut<double>&, double, double*,
                                    cudaStream_t);
template void launch_back_substitute<float>(const Shape&, const DevPtrs&, const double*, const float*, const double*,
                                            double*, double*, double*, double*, const double*, unsigned*, double*, cudaStream_t);
template void launch_back_substitute<double>(const Shape&, const DevPtrs&, const double*, const double*, const double*,
                                             double*, double*, double*, double*, const double*, unsigned*, double*, cudaStream_t);
template void launch_linearize_export<float>(const Shape&, const DevPtrs&, double*, double*, double*, double*, double*,
                                             double*, signed char*, cudaStream_t);
template void launch_linearize_export<double>(const Shape&, const DevPtrs&, double*, double*, double*, double*,
                                              double*, double*, signed char*, cudaStream_t);

}  // namespace pb
