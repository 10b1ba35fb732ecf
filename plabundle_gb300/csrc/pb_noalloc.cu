// pb_noalloc.cu -- allocation-free robust objective of caller-owned device arrays.
//
// pb_gpu_objective_noalloc is the objective of the LM line search (k_cost_batch: FP64 projection,
// robust loss, per-block partial sums reduced in a fixed order) for callers that own their device
// buffers and may not allocate.  Its per-block partials live in one file-scope device array of
// fixed size instead of context memory, so a call launches one or two kernels, brings three
// numbers back and allocates nothing.
//
// Limits and rules (also stated in include/pb_gpu.h):
//   - at most PB_NOALLOC_MAX_OBS observations; larger inputs are rejected before any launch;
//   - every element of the scratch array that the final sum reads is written earlier in the same
//     call, so nothing has to start at zero;
//   - the array and the host totals are shared by all callers on a device: a lock per device is held
//     from the launch until the totals are read, so that threads take turns, whatever their streams;
//   - the array's device address is resolved with cudaGetSymbolAddress on the first call on each
//     device (that call may load the module), so that first call should come before any stream
//     capture; the address is kept for the life of the process (not valid across a
//     cudaDeviceReset);
//   - an error already pending on the calling thread is left for its owner: the call returns
//     PB_ERR_CUDA without launching, and every status it reads afterwards is its own.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "pb_device.cuh"

namespace pb {

constexpr int kNoAllocThreads = 128;
// Eight blocks on each of 152 SMs: 155 648 threads fill the FP64 pipes, and beyond that a thread takes
// several observations, so that a Cauchy sum needs one log1p per thread and the final sum covers at
// most 1216 partials.
constexpr int kNoAllocMaxBlocks = 152 * 8;
constexpr int kClusterBlocks = 8, kClusterThreads = 256;
// Up to one observation per thread of the cluster, one launch beats two (a call of 2 001 observations: 23.6
// against 25.8 us); a second observation waits for the first on the same eight SMs (2 500: 27.1 against 25.7,
// 4 096: 27.5 against 25.7, 8 192: 34.5 against 25.9).
constexpr long long kClusterMaxObs = 1LL * kClusterBlocks * kClusterThreads;
constexpr int kNoAllocMaxDevices = 64;

// [0, B): cost partials; [B, 2B): invalid projections; [2B, 3B): index errors; [3B, 3B + 3): totals
// (B = 1216 blocks, eight per SM)
static __device__ __align__(256) double g_noalloc_scratch[3 * kNoAllocMaxBlocks + 3];

namespace {

struct ObjectiveArgs {
    const double* cameras;
    const double* points;
    const int* obs_camera;
    const int* obs_point;
    const double* obs_u;
    const double* obs_v;
    const double* obs_w;
    long long n_obs;
    int n_cameras, n_points, loss, plain;
    double scale, c2, ic2;
};

struct ObjectiveSums {
    double cost;
    int bad, oob;  // invalid projections, indices out of range
};

// The calling warp's observations first, first + stride, ... (one per lane and turn), summed over the
// warp.
template <bool VEC>
__device__ __forceinline__ ObjectiveSums objective_warp(const ObjectiveArgs& A, long long first, long long stride) {
    RobustSum acc;
    ObjectiveSums r{0.0, 0, 0};
    for (long long o = first; o < A.n_obs; o += stride) {
        const int cam = A.obs_camera[o], pt = A.obs_point[o];
        if (cam < 0 || cam >= A.n_cameras || pt < 0 || pt >= A.n_points) {
            ++r.oob;  // the access is skipped; the host reports PB_ERR_BOUNDS
            continue;
        }
        DCam c;
        load_cam_objective<VEC>(A.cameras + static_cast<size_t>(cam) * kCamStride, c);
        const double* X = A.points + static_cast<size_t>(pt) * 3;
        double s;
        if (!weighted_square64(c, X[0], X[1], X[2], A.obs_u[o], A.obs_v[o], A.obs_w[o], s) ||
            !acc.add(s, A.loss, A.scale, A.c2, A.ic2, A.plain != 0))
            ++r.bad;
    }
    __syncwarp();
    r.cost = warp_sum(acc.value(A.loss, A.c2, A.plain != 0));
    r.bad = __reduce_add_sync(0xffffffffu, r.bad);
    r.oob = __reduce_add_sync(0xffffffffu, r.oob);
    return r;
}

// One partial triple per block; a thread takes every (grid x block)-th observation.  FP64-pipe-bound
// (see the objective in pb_device.cuh).
template <bool VEC>
__global__ void __launch_bounds__(kNoAllocThreads) k_objective_part(ObjectiveArgs A, double* __restrict__ scratch) {
    __shared__ ObjectiveSums s_sum[kNoAllocThreads / 32];
    const ObjectiveSums r = objective_warp<VEC>(A, static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x,
                                                static_cast<long long>(gridDim.x) * blockDim.x);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
        ObjectiveSums t = s_sum[0];
        for (int w = 1; w < kNoAllocThreads / 32; ++w) {
            t.cost += s_sum[w].cost;
            t.bad += s_sum[w].bad;
            t.oob += s_sum[w].oob;
        }
        scratch[blockIdx.x] = t.cost;
        scratch[kNoAllocMaxBlocks + blockIdx.x] = t.bad;
        scratch[2 * kNoAllocMaxBlocks + blockIdx.x] = t.oob;
    }
}

// Fixed-order sums of the block partials into totals[0 .. 2].
__global__ void __launch_bounds__(kNoAllocThreads) k_objective_final(int nblocks, const double* __restrict__ scratch,
                                                                     double* __restrict__ totals) {
    __shared__ double s_red[3][kNoAllocThreads];
    for (int k = 0; k < 3; ++k) {
        double t = 0.0;
        for (int b = threadIdx.x; b < nblocks; b += kNoAllocThreads) t += scratch[k * kNoAllocMaxBlocks + b];
        s_red[k][threadIdx.x] = t;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 3) {  // one warp per total
        double t = s_red[warp][lane];
        for (int i = lane + 32; i < kNoAllocThreads; i += 32) t += s_red[warp][i];
        t = warp_sum(t);
        if (lane == 0) totals[warp] = t;
    }
}

// Small inputs in one launch: a cluster of eight blocks, whose partials the first block reads from
// the others' shared memory.
template <bool VEC>
__global__ void __cluster_dims__(kClusterBlocks, 1, 1) __launch_bounds__(kClusterThreads)
    k_objective_cluster(ObjectiveArgs A, double* __restrict__ totals) {
    __shared__ ObjectiveSums s_sum[kClusterThreads / 32];
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const ObjectiveSums r = objective_warp<VEC>(A, static_cast<long long>(blockIdx.x) * kClusterThreads + threadIdx.x,
                                                static_cast<long long>(kClusterBlocks) * kClusterThreads);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = r;
    cluster.sync();
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        double cost = 0.0;
        int bad = 0, oob = 0;
        for (int i = threadIdx.x; i < kClusterBlocks * (kClusterThreads / 32); i += 32) {
            const ObjectiveSums* p = cluster.map_shared_rank(&s_sum[i % (kClusterThreads / 32)], i / (kClusterThreads / 32));
            cost += p->cost;
            bad += p->bad;
            oob += p->oob;
        }
        cost = warp_sum(cost);
        bad = __reduce_add_sync(0xffffffffu, bad);
        oob = __reduce_add_sync(0xffffffffu, oob);
        if (threadIdx.x == 0) {
            totals[0] = cost;
            totals[1] = bad;
            totals[2] = oob;
        }
    }
    cluster.sync();  // the other blocks' shared memory stays until it has been read
}

// The scratch array on the current device and where its kernels write the three totals, resolved once per
// device.  Where the device reaches pageable host memory through the host's page tables (Grace), the totals
// go straight to a file-scope host array; elsewhere they follow the scratch and are copied (a call of 2 001
// observations: 33.6 -> 23.9 us).
struct NoAllocDevice {
    std::mutex turn;  // of the call that uses what follows
    double* scratch = nullptr;
    double* totals = nullptr;
    double* host = nullptr;  // the totals in host memory; null: copy them
};
NoAllocDevice* noalloc_device() {
    static std::mutex mu;
    static NoAllocDevice known[kNoAllocMaxDevices];
    alignas(64) static double host_totals[kNoAllocMaxDevices][8];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    NoAllocDevice& d = known[dev];
    if (!d.scratch) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) return nullptr;
        int reach = 0, tables = 0;
        cudaDeviceGetAttribute(&reach, cudaDevAttrPageableMemoryAccess, dev);
        cudaDeviceGetAttribute(&tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev);
        d.scratch = static_cast<double*>(p);
        if (reach && tables) d.host = d.totals = host_totals[dev];
        else d.totals = d.scratch + 3 * static_cast<size_t>(kNoAllocMaxBlocks);
    }
    return &d;
}

}  // namespace

}  // namespace pb

extern "C" pb_status pb_gpu_objective_noalloc(const double* cameras, int32_t n_cameras, const double* points,
                                              int32_t n_points, const int32_t* obs_camera, const int32_t* obs_point,
                                              const double* obs_u, const double* obs_v, const double* obs_w,
                                              int64_t n_obs, int32_t robust_loss, double robust_loss_scale,
                                              void* stream, double* cost, int64_t* invalid_projections) {
    using namespace pb;
    if (!cost || n_obs < 0 || n_cameras < 0 || n_points < 0) return PB_ERR_INVALID_ARGUMENT;
    if (robust_loss < 0 || robust_loss > 2 || (robust_loss != 0 && !(robust_loss_scale > 0.0)))
        return PB_ERR_INVALID_ARGUMENT;
    if (n_obs > static_cast<int64_t>(PB_NOALLOC_MAX_OBS)) return PB_ERR_BOUNDS;
    if (n_obs > 0 && (!cameras || !points || !obs_camera || !obs_point || !obs_u || !obs_v || !obs_w))
        return PB_ERR_INVALID_ARGUMENT;
    if (n_obs == 0) {
        *cost = 0.0;
        if (invalid_projections) *invalid_projections = 0;
        return PB_OK;
    }
    // an error pending from earlier work on this thread is not this call's: leave it in place
    if (cudaPeekAtLastError() != cudaSuccess) return PB_ERR_CUDA;
    NoAllocDevice* const known = noalloc_device();
    if (!known) return PB_ERR_CUDA;
    NoAllocDevice& d = *known;
    const std::lock_guard<std::mutex> turn(d.turn);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nblocks = static_cast<int>(std::min<int64_t>((n_obs + kNoAllocThreads - 1) / kNoAllocThreads, kNoAllocMaxBlocks));
    const double c2 = robust_loss_scale * robust_loss_scale, ic2 = 1.0 / c2;
    const int plain = robust_loss != 0 && std::isnormal(c2) && std::isnormal(ic2) ? 1 : 0;
    const ObjectiveArgs args{cameras, points, obs_camera, obs_point, obs_u, obs_v, obs_w, static_cast<long long>(n_obs),
                             n_cameras, n_points, robust_loss, plain, robust_loss_scale, c2, ic2};
    const bool vec = (reinterpret_cast<uintptr_t>(cameras) & 15) == 0;
    if (n_obs <= kClusterMaxObs) {
        (vec ? k_objective_cluster<true> : k_objective_cluster<false>)<<<kClusterBlocks, kClusterThreads, 0, st>>>(args, d.totals);
        if (cudaGetLastError() != cudaSuccess) return PB_ERR_CUDA;
    } else {
        (vec ? k_objective_part<true> : k_objective_part<false>)<<<nblocks, kNoAllocThreads, 0, st>>>(args, d.scratch);
        if (cudaGetLastError() != cudaSuccess) return PB_ERR_CUDA;
        k_objective_final<<<1, kNoAllocThreads, 0, st>>>(nblocks, d.scratch, d.totals);
        if (cudaGetLastError() != cudaSuccess) return PB_ERR_CUDA;
    }
    double totals[3] = {0.0, 0.0, 0.0};
    if ((!d.host && cudaMemcpyAsync(totals, d.totals, sizeof totals, cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return PB_ERR_CUDA;
    if (d.host) std::copy(d.host, d.host + 3, totals);
    if (totals[2] != 0.0) return PB_ERR_BOUNDS;
    *cost = totals[0];
    if (invalid_projections) *invalid_projections = static_cast<int64_t>(totals[1]);
    return PB_OK;
}
