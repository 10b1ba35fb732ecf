// pb_assemble.cu -- kernels (a)+(b): per-observation linearisation and online point Schur
// elimination into the block-sparse reduced camera system.
//
// One CTA of 256 threads per chunk of consecutive tracks (host-built: at most max_obs <= 256
// observations and max_tracks tracks), one thread per observation in phases A-C:
//   A. linearise the observation: residual, robust weight and gradient in FP64 with the cost on
//      the FP64 path, in float-float without the cost on the mixed path (FP64 runs at a small
//      fraction of the FP32 rate on this part; the LM takes the mixed path's FP64 cost from the
//      line search); Jacobians A = [J_pose | J_intr] and Jp in T (FP32 on the mixed path);
//   B. per track, V = sum w Jp^T Jp and the point gradient in FP64 and the factor V = R R^T
//      (the 3x3 point block inverse of BundleAdjustPlaMatrixReferenceSchur.cpp:350-490);
//   C. per observation, in FP64: Y = w Jp R^-T (2x3), the reduced weight M = w I - Y Y^T and Y q
//      (q = R^-1 g_p); then G = J_pose^T Y.  The matrix derives from the rounded Jacobians only,
//      so it is the exact Schur complement of one consistently perturbed linearisation (the
//      FP32 rounding of a Jacobian perturbs the weakest mode of S by ~eps*sqrt(cond), rounding
//      S itself by eps*cond).  The gradient g = -J^T w r does not carry the Jacobians' rounding
//      (FP64 or float-float, see linearize_obs / linearize_obs_ff): the rounded Jacobians shape
//      the step, never the fixed point;
//   K. per track and calibration group, K = sum over the group's observations of J_intr^T Y;
//   D. every output element of the chunk is owned by one thread, which gathers its terms in a
//      fixed order into compensated accumulators and writes the chunk partial once (which
//      thread owns which row is a host-built schedule that balances the warps' loads):
//        pose block (a, b):  sum_o J^T M J (own terms)  -  sum_(o != o') G_o G_o'^T
//        border (c, g):      sum_(o in c, g) w J_pose^T J_intr  -  sum_(o in c) G_o K_(t(o), g)^T
//        intrinsic (g, g'):  sum_(o in g) w J_intr^T J_intr  -  sum_t K_(t,g) K_(t,g')^T
//        rhs:                sum_o g_o - J^T Y q  (and the direct gradient sum_o g_o)
//      (the own term J^T M J plus the observation's own G G^T is w J^T J).  No atomics; the
//      result is deterministic.
// On the FP32 path all products and sums of D run in float-float arithmetic (exact FMA product
// residuals, two-sum accumulation): ~44 significant bits on the FP32 pipe, enough for reduced
// matrices of condition ~1e9, where FP32 products alone leave the weakest modes indefinite.
#include <cuda_runtime.h>

#include <type_traits>

#include "pb_device.cuh"
#include "pb_kernels.h"

namespace pb {

namespace {

template <typename T>
__device__ __forceinline__ T* carve(char*& ptr, size_t count) {
    T* out = reinterpret_cast<T*>(ptr);
    ptr += (count * sizeof(T) + 15) & ~static_cast<size_t>(15);
    return out;
}

constexpr int kOk = 1, kElim = 2;
__device__ __forceinline__ int info_group(int info) { return ((info >> 2) & 7) - 1; }
// per-observation track record: first observation (8 bits) | chunk track slot (8) | length (16)
__device__ __forceinline__ int trk_slot(int v) { return (v >> 8) & 0xFF; }

// The six sums of an owned row in phase D.  The FP32 path keeps them as three packed pairs: a term of a
// coupling is 108 packed operations and 15 loads instead of 216 and 21, each half rounded as the scalar
// operations round it, in the same order (100 cameras, 780 000 observations, two groups of eight
// intrinsics: 1555 -> 1416 us a launch).
template <typename T>
struct RowAcc;
template <>
struct RowAcc<double> {
    Acc<double> a[6];
    // += J0 u0 + J1 u1 for the pose columns of two Jacobian rows
    __device__ __forceinline__ void jacobian(const double* J0, const double* J1, double u0, double u1) {
#pragma unroll
        for (int y = 0; y < 6; ++y) {
            acc_fma(a[y], J0[y], u0);
            acc_fma(a[y], J1[y], u1);
        }
    }
    // += G (g0, g1, g2)^T (LEFT: g is the left factor of the products)
    template <bool LEFT>
    __device__ __forceinline__ void coupling(const double* G, double g0, double g1, double g2) {
#pragma unroll
        for (int y = 0; y < 6; ++y) {
            acc_fma(a[y], g0, G[3 * y]);
            acc_fma(a[y], g1, G[3 * y + 1]);
            acc_fma(a[y], g2, G[3 * y + 2]);
        }
    }
    __device__ __forceinline__ void add(const double* g) {
#pragma unroll
        for (int y = 0; y < 6; ++y) a[y].add(g[y]);
    }
    __device__ __forceinline__ double part(int y) const { return a[y].part(); }
};
template <>
struct RowAcc<float> {
    Acc2 a[3];
    __device__ __forceinline__ void jacobian(const float* J0, const float* J1, ff u0, ff u1) {
        const f2 h0 = f2_both(u0.hi), nh0 = f2_both(-u0.hi), nl0 = f2_both(-u0.lo);
        const f2 h1 = f2_both(u1.hi), nh1 = f2_both(-u1.hi), nl1 = f2_both(-u1.lo);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            a[q].fma_f(f2_pack(J0[2 * q], J0[2 * q + 1]), h0, nh0, nl0);
            a[q].fma_f(f2_pack(J1[2 * q], J1[2 * q + 1]), h1, nh1, nl1);
        }
    }
    template <bool LEFT>
    __device__ __forceinline__ void coupling(const float4* G, ff g0, ff g1, ff g2) {
        const ulonglong2* G2 = reinterpret_cast<const ulonglong2*>(G);
        const ff g[3] = {g0, g1, g2};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const f2 h = f2_both(g[k].hi), nh = f2_both(-g[k].hi), nl = f2_both(-g[k].lo);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const ulonglong2 v = G2[k * 3 + q];
                a[q].template fma_ff<LEFT>(h, nh, nl, v.x, v.y);
            }
        }
    }
    __device__ __forceinline__ void add(const ff* g) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            a[q].add(f2_pack(g[2 * q].hi, g[2 * q + 1].hi));
            a[q].lo = f2_add(a[q].lo, f2_pack(g[2 * q].lo, g[2 * q + 1].lo));
        }
    }
    __device__ __forceinline__ float2 part(int y) const {
        const float2 h = f2_parts(a[y >> 1].hi), l = f2_parts(a[y >> 1].lo);
        return y & 1 ? make_float2(h.y, l.y) : make_float2(h.x, l.x);
    }
};

// Two neighbouring columns of a track's K: sums of a0 y0 + a1 y1 over its observations.
template <typename T>
struct ColumnPair;
template <>
struct ColumnPair<double> {
    double s0 = 0.0, s1 = 0.0;
    __device__ __forceinline__ void add(double a0, double b0, double y0, double a1, double b1, double y1) {
        s0 = s0 + (a0 * y0 + a1 * y1);
        s1 = s1 + (b0 * y0 + b1 * y1);
    }
    __device__ __forceinline__ double first() const { return s0; }
    __device__ __forceinline__ double second() const { return s1; }
};
template <>
struct ColumnPair<float> {
    ff2p s{0ull, 0ull};
    __device__ __forceinline__ void add(float a0, float b0, ff y0, float a1, float b1, ff y1) {
        s = s + (f2_pack(a0, b0) * y0 + f2_pack(a1, b1) * y1);
    }
    __device__ __forceinline__ ff first() const { return {f2_parts(s.hi).x, f2_parts(s.lo).x}; }
    __device__ __forceinline__ ff second() const { return {f2_parts(s.hi).y, f2_parts(s.lo).y}; }
};

// Four neighbouring entries of a row of the intrinsic block (or of its gradient).  Four at a time read
// the row's own factors, the weight and the group marks once, and the FP32 path sums them as two packed
// pairs: with a warp per entry the phase took 64 000 of a chunk's 190 000 cycles (same launch, this and
// ColumnPair: 1416 -> 1200 us).
template <typename T>
struct QuadAcc;
template <>
struct QuadAcc<double> {
    Acc<double> a[4];
    __device__ __forceinline__ void weighted(double w, double r, double b0, double b1, double b2, double b3) {
        acc_fma(a[0], w, r * b0);
        acc_fma(a[1], w, r * b1);
        acc_fma(a[2], w, r * b2);
        acc_fma(a[3], w, r * b3);
    }
    __device__ __forceinline__ void minus(double r, double b0, double b1, double b2, double b3) {
        acc_fma(a[0], -r, b0);
        acc_fma(a[1], -r, b1);
        acc_fma(a[2], -r, b2);
        acc_fma(a[3], -r, b3);
    }
    __device__ __forceinline__ void jacobian(double b0, double b1, double b2, double b3, double r) { minus(-r, b0, b1, b2, b3); }
    __device__ __forceinline__ void add(double b0, double b1, double b2, double b3) {
        a[0].add(b0);
        a[1].add(b1);
        a[2].add(b2);
        a[3].add(b3);
    }
    __device__ __forceinline__ void split(Acc<double>* q) const {
        for (int i = 0; i < 4; ++i) q[i] = a[i];
    }
};
template <>
struct QuadAcc<float> {
    Acc2 a[2];
    // += w (r b): the product r b exact, acc_fma of w and it
    __device__ __forceinline__ void weighted(ff w, float r, float b0, float b1, float b2, float b3) {
        const f2 wh = f2_both(w.hi), nwh = f2_both(-w.hi), nwl = f2_both(-w.lo), rr = f2_both(r), nr = f2_both(-r);
        const f2 b[2] = {f2_pack(b0, b1), f2_pack(b2, b3)};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const f2 h = f2_mul(rr, b[q]), nl = f2_fma(nr, b[q], h);  // r b = h - nl
            const f2 p = f2_mul(wh, h);
            const f2 ne = f2_fma(nwl, h, f2_fma(wh, nl, f2_fma(nwh, h, p)));
            a[q].add(p);
            a[q].lo = f2_sub(a[q].lo, ne);
        }
    }
    // += (-r) b
    __device__ __forceinline__ void minus(ff r, ff b0, ff b1, ff b2, ff b3) {
        const f2 h = f2_both(-r.hi), nh = f2_both(r.hi), nl = f2_both(r.lo);
        a[0].template fma_ff<true>(h, nh, nl, f2_pack(b0.hi, b1.hi), f2_pack(b0.lo, b1.lo));
        a[1].template fma_ff<true>(h, nh, nl, f2_pack(b2.hi, b3.hi), f2_pack(b2.lo, b3.lo));
    }
    __device__ __forceinline__ void jacobian(float b0, float b1, float b2, float b3, ff r) {
        const f2 h = f2_both(r.hi), nh = f2_both(-r.hi), nl = f2_both(-r.lo);
        a[0].fma_f(f2_pack(b0, b1), h, nh, nl);
        a[1].fma_f(f2_pack(b2, b3), h, nh, nl);
    }
    __device__ __forceinline__ void add(ff b0, ff b1, ff b2, ff b3) {
        a[0].add(f2_pack(b0.hi, b1.hi));
        a[0].lo = f2_add(a[0].lo, f2_pack(b0.lo, b1.lo));
        a[1].add(f2_pack(b2.hi, b3.hi));
        a[1].lo = f2_add(a[1].lo, f2_pack(b2.lo, b3.lo));
    }
    __device__ __forceinline__ void split(Acc<float>* q) const {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float2 h = f2_parts(a[i].hi), l = f2_parts(a[i].lo);
            q[2 * i].hi = h.x;
            q[2 * i].lo = l.x;
            q[2 * i + 1].hi = h.y;
            q[2 * i + 1].lo = l.y;
        }
    }
};

// A fixed shuffle tree (lane l takes lane l + 16's value, then l + 8's, ...) for four values at once: at
// the first two levels a lane gives half of its values away and keeps the other half, in either case
// merging the higher lane's value into the lower lane's.  The total of value x ends in lane 8x.
template <typename T>
__device__ __forceinline__ Acc<T> quad_merge(Acc<T>* q) {
    const int lane = threadIdx.x & 31;
    Acc<T> two[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) two[i] = exchange_merge(q[i], q[2 + i], 16, (lane & 16) != 0);
    Acc<T> one = exchange_merge(two[0], two[1], 8, (lane & 8) != 0);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) one.merge_part(shfl_down_part(one.part(), o));
    return one;
}

// 256 threads per chunk whatever its observation count (at most 256): threads beyond the chunk's
// observations idle in phases A-C and take their share of the gathers of phase D.
constexpr int kAssembleThreads = 256;
static_assert(kAssembleThreads == 32 * kAssembleWarps, "the owner-gather schedule is planned for 8 warps");

}  // namespace

template <typename T>
__global__ void __launch_bounds__(kAssembleThreads, 2) k_assemble(Shape S, DevPtrs D, AsmOutT<T> O, double damping) {
    using P = typename Acc<T>::part_type;
    using Val = ValueOf<T>;
    using VT = typename Val::type;
    extern __shared__ __align__(16) char smem[];
    const int chunk = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int MO = S.max_obs, MT = S.max_tracks;
    const int ng = S.ng, ni = S.ni, nb = S.nb, nA = 6 + ni;
    // per-observation records are padded to an odd number of 4- or 8-byte words, so that the
    // lanes of a warp reading the same field of consecutive observations hit distinct banks
    const int sA = chunk_stride(2 * nA), sG = chunk_stride(18), sY = chunk_stride(6), sM = chunk_stride(6),
              sD = chunk_stride(nA);
    char* ptr = smem;
    double* s_V = carve<double>(ptr, static_cast<size_t>(MO) * 9);  // point normal terms, then the track factor
    T* s_A = carve<T>(ptr, static_cast<size_t>(MO) * sA);
    VT* s_G = carve<VT>(ptr, static_cast<size_t>(MO) * sG);
    // FP32 path: G in packed pairs of rows, G4[k * 3 + q] = (hi, hi, lo, lo) of G[2q][k] and G[2q + 1][k],
    // nine 16-byte words per observation (the lanes of a quarter-warp hit distinct banks)
    float4* s_G4 = reinterpret_cast<float4*>(s_G);
    VT* s_Y = carve<VT>(ptr, static_cast<size_t>(MO) * sY);
    VT* s_M = carve<VT>(ptr, static_cast<size_t>(MO) * sM);
    VT* s_D = carve<VT>(ptr, static_cast<size_t>(MO) * sD);
    int* s_info = carve<int>(ptr, MO);
    int* s_trk = carve<int>(ptr, MO);
    const int sK = chunk_stride(nb * 3);  // per-track K record (odd: lanes over tracks hit distinct banks)
    VT* s_K = carve<VT>(ptr, static_cast<size_t>(MT) * sK);
    int* s_tfirst = carve<int>(ptr, MT + 1);
    int* s_tmask = carve<int>(ptr, MT);  // calibration groups present in each chunk track
    double* s_cpc = carve<double>(ptr, MT);  // control-point cost of each chunk track
    double* s_misc = carve<double>(ptr, 40);
    int* s_flags = reinterpret_cast<int*>(s_misc + 32);
    int* s_wcount = reinterpret_cast<int*>(s_misc + 34);
    int* s_next_entry = reinterpret_cast<int*>(s_misc + 38);  // next intrinsic entry to take

    const int obs0 = D.ch_obs_begin[chunk], nobs = D.ch_obs_begin[chunk + 1] - obs0;
    if (tid == 0) {
        s_flags[0] = 0;
        s_next_entry[0] = 0;
    }
    __syncthreads();

    // ---- A: linearise one observation per thread; FP64 point normal equations
    const bool active = tid < nobs;
    const int o = obs0 + tid;
    Lin<T> L;
    double grad[9 + kMaxNI];
    double cost = 0.0;
    double w64 = 0.0;  // normal weight (FP64 value of the float-float weight on the mixed path)
    T jpT[6];          // point Jacobian of the arithmetic type
    int first = 0, k = 0;
    bool elim = false, ok = false;
    constexpr bool kMixed = std::is_same<T, float>::value;
    if constexpr (kMixed) {
        if (active) {
            // mixed path: FP64 projection, float-float weight and gradient (no cost: the LM takes it
            // from the line search)
            const int cam = D.obs_cam[o];
            const int trk = D.obs_trk[o];
            const int tb0 = D.trk_obs_begin[trk];
            first = tb0 - obs0;
            k = D.trk_obs_begin[trk + 1] - tb0;
            elim = D.trk_block[trk] >= 0;
            const int grp = ng > 0 ? D.cam_group[cam] : -1;
            const bool tangent = cam == S.gauge_scale && S.gauge_anchor >= 0 && S.gauge_baseline > 0.0;
            DCam c;
            load_cam(D.cams_eff + static_cast<size_t>(cam) * kCamStride, c);
            const double* X = D.points + static_cast<size_t>(trk) * 3;
            Proj pr;
            LinFF F;
            ok = project64(c, X[0], X[1], X[2], pr) &&
                 linearize_obs_ff(pr, D.obs_u[o], D.obs_v[o], D.cams_ff + static_cast<size_t>(cam) * kCamFF,
                                  ffl(D.pscale_ff[trk]), ffl(D.obs_w_ff[o]), S.loss,
                                  ff{S.loss_scale_hi, S.loss_scale_lo}, tangent, !S.ref_param, D.gauge_basis, ni,
                                  S.int_cols, F);
            if (!ok) atomicOr(s_flags, 2);
            s_info[tid] = (ok ? kOk : 0) | (elim ? kElim : 0) | ((grp + 1) << 2);
            T* A = s_A + static_cast<size_t>(tid) * sA;
            for (int a = 0; a < 6; ++a) {
                A[a] = ok ? F.Jc[a] : T(0);
                A[nA + a] = ok ? F.Jc[6 + a] : T(0);
            }
            for (int a = 0; a < ni; ++a) {
                A[6 + a] = ok ? F.Ji[a] : T(0);
                A[nA + 6 + a] = ok ? F.Ji[kMaxNI + a] : T(0);
            }
            VT* Dg = s_D + static_cast<size_t>(tid) * sD;
            for (int a = 0; a < 6; ++a) Dg[a] = ok ? F.g[a] : Val::zero();
            for (int a = 0; a < ni; ++a) Dg[6 + a] = ok ? F.g[9 + a] : Val::zero();
            // the point block, its factor and the projector of phases B and C stay in FP64: the
            // reduced weight M = w I - Y Y^T cancels to a small fraction of w, and the weakest modes
            // of the reduced matrix need its FP64 rounding
            double* V = s_V + static_cast<size_t>(tid) * 9;
            w64 = static_cast<double>(F.w.hi) + static_cast<double>(F.w.lo);
            for (int i = 0; i < 6; ++i) jpT[i] = F.Jp[i];
            if (elim && ok) {
                // V_o = w Jp^T Jp from the rounded Jacobian and the point gradient
                const double w = w64;
                const double j0 = F.Jp[0], j1 = F.Jp[1], j2 = F.Jp[2], j3 = F.Jp[3], j4 = F.Jp[4], j5 = F.Jp[5];
                V[0] = w * (j0 * j0 + j3 * j3);
                V[1] = w * (j0 * j1 + j3 * j4);
                V[2] = w * (j0 * j2 + j3 * j5);
                V[3] = w * (j1 * j1 + j4 * j4);
                V[4] = w * (j1 * j2 + j4 * j5);
                V[5] = w * (j2 * j2 + j5 * j5);
                for (int i = 0; i < 3; ++i)
                    V[6 + i] = static_cast<double>(F.g[6 + i].hi) + static_cast<double>(F.g[6 + i].lo);
            } else {
                for (int i = 0; i < 9; ++i) V[i] = 0.0;
            }
        }
    } else {
        if (active) {
            const int cam = D.obs_cam[o];
            const int trk = D.obs_trk[o];
            const int tb0 = D.trk_obs_begin[trk];
            first = tb0 - obs0;
            k = D.trk_obs_begin[trk + 1] - tb0;
            elim = D.trk_block[trk] >= 0;
            const int grp = ng > 0 ? D.cam_group[cam] : -1;
            DCam c;
            load_cam(D.cams_eff + static_cast<size_t>(cam) * kCamStride, c);
            const double* X = D.points + static_cast<size_t>(trk) * 3;
            const bool tangent = cam == S.gauge_scale && S.gauge_anchor >= 0 && S.gauge_baseline > 0.0;
            ok = linearize_obs<T>(c, X[0], X[1], X[2], D.pscale[trk], D.obs_u[o], D.obs_v[o], D.obs_w[o], S.loss,
                                  S.loss_scale, tangent, !S.ref_param, D.gauge_basis, ni, S.int_cols, true, L, grad);
            if (!ok) {
                atomicOr(s_flags, 2);
            } else {
                cost = L.cost;
            }
            s_info[tid] = (ok ? kOk : 0) | (elim ? kElim : 0) | ((grp + 1) << 2);
            T* A = s_A + static_cast<size_t>(tid) * sA;
            for (int a = 0; a < 6; ++a) {
                A[a] = ok ? L.Jc[a] : T(0);
                A[nA + a] = ok ? L.Jc[6 + a] : T(0);
            }
            for (int a = 0; a < ni; ++a) {
                A[6 + a] = ok ? L.Ji[a] : T(0);
                A[nA + 6 + a] = ok ? L.Ji[kMaxNI + a] : T(0);
            }
            // the observation's gradient -J^T w r (FP64): pose and intrinsic columns
            VT* Dg = s_D + static_cast<size_t>(tid) * sD;
            for (int a = 0; a < 6; ++a) Dg[a] = ok ? Val::make(grad[a]) : Val::zero();
            for (int a = 0; a < ni; ++a) Dg[6 + a] = ok ? Val::make(grad[9 + a]) : Val::zero();
            double* V = s_V + static_cast<size_t>(tid) * 9;
            w64 = L.wd;
            for (int i = 0; i < 6; ++i) jpT[i] = L.Jp[i];
            if (elim && ok) {
                // V_o = w Jp^T Jp from the Jacobian and the point gradient, in FP64
                const double w = L.wd;
                const double j0 = L.Jp[0], j1 = L.Jp[1], j2 = L.Jp[2], j3 = L.Jp[3], j4 = L.Jp[4], j5 = L.Jp[5];
                V[0] = w * (j0 * j0 + j3 * j3);
                V[1] = w * (j0 * j1 + j3 * j4);
                V[2] = w * (j0 * j2 + j3 * j5);
                V[3] = w * (j1 * j1 + j4 * j4);
                V[4] = w * (j1 * j2 + j4 * j5);
                V[5] = w * (j2 * j2 + j5 * j5);
                V[6] = grad[6];
                V[7] = grad[7];
                V[8] = grad[8];
            } else {
                for (int i = 0; i < 9; ++i) V[i] = 0.0;
            }
        }
    }
    // chunk-local track slots: rank of each track's first observation among the chunk's
    // track starts (all lanes of every warp take part: blockDim is a multiple of 32)
    const bool start = active && tid == first;
    const unsigned ballot = __ballot_sync(0xffffffffu, start);
    if (lane == 0) s_wcount[wid] = __popc(ballot);
    // block cost (FP64, fixed order)
    const double cw = warp_sum(cost);
    if (lane == 0) s_misc[wid] = cw;
    __syncthreads();

    // ---- B: track slots; per track FP64 Cholesky V(1+lambda) = R R^T.  R^-1 and q = R^-1 g_p
    // replace the track's first record of s_V (only this thread reads them in this phase).
    int ntc = 0, slot = 0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) {
        if (w == wid) slot = ntc + __popc(ballot & ((1u << lane) - 1u));
        ntc += s_wcount[w];
    }
    if (ntc > MT) {
        // the host bounds the tracks of a chunk; a larger count would overrun s_K
        if (tid == 0) atomicOr(s_flags, 4);
        ntc = 0;
    }
    if (start) {
        s_trk[tid] = first | (slot << 8) | (k << 16);
        if (slot < MT) {
            s_tfirst[slot] = tid;
            int mask = 0;
            for (int j = first; j < first + k; ++j) {
                const int g = info_group(s_info[j]);
                if (g >= 0) mask |= 1 << g;
            }
            s_tmask[slot] = mask;
        }
    }
    if (tid == 0 && ntc <= MT) s_tfirst[ntc] = nobs;
    __syncthreads();
    // Per track, one thread: track slot t goes to lane t / 4 of warp t % 4 (warps 4-7 for slots
    // 128 and up), so that the FP64 work of the chunk's tracks runs on a few warps spread over
    // the four sub-partitions rather than on scattered lanes of every warp.
    const int tslot = (wid >> 2) * 128 + lane * 4 + (wid & 3);
    const bool tact = tslot < ntc;
    const int tfirst = tact ? s_tfirst[tslot] : 0;
    const int tobs = obs0 + tfirst;
    const bool telim = tact && (s_info[tfirst] & kElim);
    // control points of the track (linearizeTrack, BundleAdjustPlaMatrixReferenceSchur.cpp:331-346):
    // their cost always, their point terms when the point is eliminated
    double cpV[6] = {0, 0, 0, 0, 0, 0}, cpg[3] = {0, 0, 0};
    if (tact && S.ncp > 0) {
        const int trk = D.obs_trk[tobs];
        const double* X = D.points + static_cast<size_t>(trk) * 3;
        double cc_sum = 0.0;
        for (int q = D.trk_cp_begin[trk]; q < D.trk_cp_begin[trk + 1]; ++q) {
            const double* rec = D.cp_rec + static_cast<size_t>(q) * 12;
            double r[3], cc, cw;
            if (!cp_eval(rec, X[0], X[1], X[2], S.cp_huber, r, cc, cw)) continue;  // not finite: skipped
            cc_sum += cc;
            // accumulatePointOnlyConstraint (:241-260): V += w J^T J, g -= w J^T r, J = sqrt(weight) W
            int e = 0;
            for (int a = 0; a < 3; ++a) {
                for (int b = a; b < 3; ++b)
                    cpV[e++] += cw * (rec[a] * rec[b] + rec[3 + a] * rec[3 + b] + rec[6 + a] * rec[6 + b]);
                cpg[a] -= cw * (rec[a] * r[0] + rec[3 + a] * r[1] + rec[6 + a] * r[2]);
            }
        }
        s_cpc[tslot] = cc_sum;
    }
    // sums of the track's nine point terms over its observations, in observation order: a thread per
    // track and term (a thread per track kept 10 of 32 lanes busy through 58 FP64 additions); the sums
    // and their start, the control points' terms, take the place of G, which phase C writes
    double* s_sum = reinterpret_cast<double*>(s_G);
    if (S.ncp > 0) {
        if (tact) {
            for (int i = 0; i < 6; ++i) s_sum[tslot * 9 + i] = cpV[i];
            for (int i = 0; i < 3; ++i) s_sum[tslot * 9 + 6 + i] = cpg[i];
        }
        __syncthreads();
    }
    for (int e = tid; e < 9 * ntc; e += kAssembleThreads) {
        const int t = e / 9, i = e - 9 * t, j0 = s_tfirst[t], j1 = s_tfirst[t + 1];
        double v = S.ncp > 0 ? s_sum[e] : 0.0;
        for (int j = j0; j < j1; ++j) v += s_V[static_cast<size_t>(j) * 9 + i];
        s_sum[e] = v;
    }
    __syncthreads();
    if (telim) {
        double V[6], rhs[3];
        for (int i = 0; i < 6; ++i) V[i] = s_sum[tslot * 9 + i];
        for (int i = 0; i < 3; ++i) rhs[i] = s_sum[tslot * 9 + 6 + i];
        V[0] *= 1.0 + damping;
        V[3] *= 1.0 + damping;
        V[5] *= 1.0 + damping;
        // tryInverse3x3 singularity rule: |det| <= 1e-15
        const double det = V[0] * (V[3] * V[5] - V[4] * V[4]) - V[1] * (V[1] * V[5] - V[4] * V[2]) +
                           V[2] * (V[1] * V[4] - V[3] * V[2]);
        double Ri[6] = {0, 0, 0, 0, 0, 0}, q[3] = {0, 0, 0};
        bool singular = !(fabs(det) > 1e-15) || !isfinite(det);
        if (!singular) {
            // Cholesky through reciprocal square roots (no FP64 division on the critical path)
            const double i00 = rsqrt(V[0]);
            const double R10 = V[1] * i00, R20 = V[2] * i00;
            const double a11 = V[3] - R10 * R10;
            const double i11 = rsqrt(a11);
            const double R21 = (V[4] - R20 * R10) * i11;
            const double a22 = V[5] - R20 * R20 - R21 * R21;
            const double i22 = rsqrt(a22);
            if (!(V[0] > 0.0) || !(a11 > 0.0) || !(a22 > 0.0) || !isfinite(i22)) {
                singular = true;
            } else {
                const double i10 = -R10 * i00 * i11;
                const double i21 = -R21 * i11 * i22;
                const double i20 = -(R20 * i00 + R21 * i10) * i22;
                Ri[0] = i00; Ri[1] = i10; Ri[2] = i11; Ri[3] = i20; Ri[4] = i21; Ri[5] = i22;
                q[0] = i00 * rhs[0];
                q[1] = i10 * rhs[0] + i11 * rhs[1];
                q[2] = i20 * rhs[0] + i21 * rhs[1] + i22 * rhs[2];
            }
        }
        if (singular) atomicOr(s_flags, 1);
        double* st = s_V + static_cast<size_t>(tfirst) * 9;
        double* gt = O.trk_data + static_cast<size_t>(D.obs_trk[tobs]) * kTrackRec;
        for (int i = 0; i < 6; ++i) { st[i] = Ri[i]; gt[i] = Ri[i]; }
        for (int i = 0; i < 3; ++i) {
            st[6 + i] = q[i];
            gt[6 + i] = q[i];
            gt[9 + i] = rhs[i];
        }
    }
    __syncthreads();

    // ---- C: per observation, in FP64: Y = w Jp R^-T, M = w I - Y Y^T and Y q; then
    // G = J_pose^T Y (values: float-float on the FP32 path; zero for tracks not eliminated)
    if (active) {
        if (!start) s_trk[tid] = s_trk[first];
        VT* G = s_G + static_cast<size_t>(tid) * sG;
        float4* G4 = s_G4 + static_cast<size_t>(tid) * 9;
        VT* Ys = s_Y + static_cast<size_t>(tid) * sY;
        VT* Mo = s_M + static_cast<size_t>(tid) * sM;
        if (ok) {
            VT y[6];
            {
                // FP64 from the rounded Jacobian and the weight of phase A
                const double w = w64;
                double Y[2][3] = {{0, 0, 0}, {0, 0, 0}}, q[3] = {0, 0, 0};
                if (elim) {
                    const double* st = s_V + static_cast<size_t>(first) * 9;
                    const double i00 = st[0], i10 = st[1], i11 = st[2], i20 = st[3], i21 = st[4], i22 = st[5];
                    q[0] = st[6]; q[1] = st[7]; q[2] = st[8];
                    for (int pa = 0; pa < 2; ++pa) {
                        const double p0 = f64_of(jpT[pa * 3]), p1 = f64_of(jpT[pa * 3 + 1]), p2 = f64_of(jpT[pa * 3 + 2]);
                        Y[pa][0] = w * (i00 * p0);
                        Y[pa][1] = w * (i10 * p0 + i11 * p1);
                        Y[pa][2] = w * (i20 * p0 + i21 * p1 + i22 * p2);
                    }
                }
                Mo[0] = Val::make(w - (Y[0][0] * Y[0][0] + Y[0][1] * Y[0][1] + Y[0][2] * Y[0][2]));
                Mo[1] = Val::make(-(Y[0][0] * Y[1][0] + Y[0][1] * Y[1][1] + Y[0][2] * Y[1][2]));
                Mo[2] = Val::make(w - (Y[1][0] * Y[1][0] + Y[1][1] * Y[1][1] + Y[1][2] * Y[1][2]));
                Mo[3] = Val::make(Y[0][0] * q[0] + Y[0][1] * q[1] + Y[0][2] * q[2]);
                Mo[4] = Val::make(Y[1][0] * q[0] + Y[1][1] * q[1] + Y[1][2] * q[2]);
                Mo[5] = Val::make(w);
                for (int i = 0; i < 6; ++i) y[i] = Val::make(Y[i / 3][i % 3]);
            }
            for (int i = 0; i < 6; ++i) Ys[i] = y[i];
            const T* A = s_A + static_cast<size_t>(tid) * sA;
            if constexpr (kMixed) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
#pragma unroll
                    for (int k3 = 0; k3 < 3; ++k3) {
                        const ff e = A[2 * q] * y[k3] + A[nA + 2 * q] * y[3 + k3];
                        const ff f = A[2 * q + 1] * y[k3] + A[nA + 2 * q + 1] * y[3 + k3];
                        G4[k3 * 3 + q] = make_float4(e.hi, f.hi, e.lo, f.lo);
                    }
            } else {
                for (int a = 0; a < 6; ++a) {
                    const T ja0 = A[a], ja1 = A[nA + a];
                    G[a * 3 + 0] = ja0 * y[0] + ja1 * y[3];
                    G[a * 3 + 1] = ja0 * y[1] + ja1 * y[4];
                    G[a * 3 + 2] = ja0 * y[2] + ja1 * y[5];
                }
            }
        } else {
            for (int i = 0; i < 6; ++i) Mo[i] = Val::zero();
            for (int i = 0; i < 6; ++i) Ys[i] = Val::zero();
            if constexpr (kMixed) {
                for (int i = 0; i < 9; ++i) G4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
                for (int i = 0; i < 18; ++i) G[i] = Val::zero();
            }
        }
    }
    __syncthreads();
    // back-substitution records of the chunk's observations: A rows, then Y (rounded to T), a warp per
    // observation (a thread per observation wrote 32 lines per store)
    {
        const int rl = 2 * nA + 6;
        for (int ob = wid; ob < nobs; ob += kAssembleWarps) {
            T* rec = O.obs_rec + static_cast<size_t>(obs0 + ob) * rl;
            const T* A = s_A + static_cast<size_t>(ob) * sA;
            const VT* Y = s_Y + static_cast<size_t>(ob) * sY;
            for (int i = lane; i < rl; i += 32) {
                T v;
                if (i < 2 * nA) v = A[i];
                else if constexpr (kMixed) v = Y[i - 2 * nA].hi;  // RN of the FP64 value
                else v = Y[i - 2 * nA];
                rec[i] = v;
            }
        }
    }
    // ---- K: per track and group, K[(g, c), k] = sum_(o in track, group g) (J_intr^T Y)[c, k]; a thread per
    // track, group, pair of columns and k
    if (nb > 0) {
        const int npc = (ni + 1) / 2, per = ng * npc * 3;
        for (int it = tid; it < ntc * per; it += kAssembleThreads) {
            const int t = it / per, r = it - t * per;
            const int gc = r / 3, kk = r - gc * 3;
            const int g = gc / npc, c = 2 * (gc - g * npc), c1 = min(c + 1, ni - 1);
            ColumnPair<T> acc;
            for (int ob = s_tfirst[t]; ob < s_tfirst[t + 1]; ++ob) {
                if (info_group(s_info[ob]) != g) continue;
                const T* A = s_A + static_cast<size_t>(ob) * sA + 6;
                const VT* Y = s_Y + static_cast<size_t>(ob) * sY;
                acc.add(A[c], A[c1], Y[kk], A[nA + c], A[nA + c1], Y[3 + kk]);
            }
            VT* K = s_K + static_cast<size_t>(t) * sK + (g * ni + c) * 3 + kk;
            K[0] = acc.first();
            if (c + 1 < ni) K[3] = acc.second();
        }
        __syncthreads();
    }

    // ---- D: owner gathers over [pose block rows | camera rows | intrinsic entries]
    const int pair0 = D.ch_pair_begin[chunk], npairs = D.ch_pair_begin[chunk + 1] - pair0;
    const int cam0 = D.ch_cam_begin[chunk], ncams = D.ch_cam_begin[chunk + 1] - cam0;
    const int camrec = 12 + ng * 6 * ni;
    const int crow = 2 + ng * ni;  // rows of a camera record: rhs, direct rhs, border (g, c)
    const int chrec = nb * nb + 2 * nb;
    const int w_pair = npairs * 6, w_cam = ncams * crow;
    // host-built schedule (schedule_owner_tasks, pb_host.cpp): this warp's rounds of 32 tasks,
    // dealt to the warps by longest processing time
    const int task_end = D.warp_task_begin[chunk * kAssembleWarps + wid + 1];
    for (int pos = D.warp_task_begin[chunk * kAssembleWarps + wid] + lane; pos < task_end; pos += 32) {
        const int wk = D.task_list[pos];
        if (wk == kNoTask) continue;
        if (wk < w_pair) {
            // row x of the pose block of chunk pair slot s
            const int s = wk / 6, x = wk - s * 6;
            const int pk = D.ch_pairs[pair0 + s];
            const bool diag = (pk & 0xFFFF) == (pk >> 16);
            RowAcc<T> acc;
            const int i1 = D.slot_item_begin[pair0 + s + 1];
            for (int it = D.slot_item_begin[pair0 + s]; it < i1; ++it) {
                const unsigned item = D.slot_items[it];
                const int oa = item & 0xFF, ob = item >> 8;
                if (oa == ob) {
                    // own term: row x of J^T M J
                    const T* A = s_A + static_cast<size_t>(oa) * sA;
                    const VT* M = s_M + static_cast<size_t>(oa) * sM;
                    const T ax0 = A[x], ax1 = A[nA + x];
                    const VT u0 = ax0 * M[0] + ax1 * M[1];
                    const VT u1 = ax0 * M[1] + ax1 * M[2];
                    acc.jacobian(A, A + nA, u0, u1);
                } else if constexpr (kMixed) {
                    const float4* Ga = s_G4 + static_cast<size_t>(oa) * 9;
                    const float* Gx = reinterpret_cast<const float*>(Ga + (x >> 1)) + (x & 1);
                    acc.template coupling<true>(s_G4 + static_cast<size_t>(ob) * 9, ff{-Gx[0], -Gx[2]}, ff{-Gx[12], -Gx[14]},
                                                 ff{-Gx[24], -Gx[26]});
                } else {
                    const VT* Ga = s_G + static_cast<size_t>(oa) * sG + 3 * x;
                    acc.template coupling<true>(s_G + static_cast<size_t>(ob) * sG, -Ga[0], -Ga[1], -Ga[2]);
                }
            }
            P* out = O.part_pair + static_cast<size_t>(pair0 + s) * 36;
#pragma unroll
            for (int y = 0; y < 6; ++y) {
                if (!diag) {
                    out[x * 6 + y] = acc.part(y);
                } else if (y >= x) {
                    out[x * 6 + y] = acc.part(y);
                    out[y * 6 + x] = acc.part(y);
                }
            }
        } else if (wk < w_pair + w_cam) {
            const int r = wk - w_pair;
            const int l = r / crow, row = r - l * crow;
            const int b0 = D.lcam_obs_begin[cam0 + l], b1 = D.lcam_obs_begin[cam0 + l + 1];
            P* out = O.part_cam + static_cast<size_t>(cam0 + l) * camrec;
            RowAcc<T> acc;
            if (row < 2) {
                // gradient rows: the reduced gradient -J_pose^T (w r + Y q) and the direct
                // gradient -J_pose^T w r (the point term with the rounded Jacobian)
                for (int it = b0; it < b1; ++it) {
                    const int ob = D.lcam_obs[it];
                    acc.add(s_D + static_cast<size_t>(ob) * sD);
                    if (row == 0) {
                        const T* A = s_A + static_cast<size_t>(ob) * sA;
                        const VT* M = s_M + static_cast<size_t>(ob) * sM;
                        acc.jacobian(A, A + nA, -M[3], -M[4]);
                    }
                }
#pragma unroll
                for (int a = 0; a < 6; ++a) out[row * 6 + a] = acc.part(a);
            } else {
                // border column (g, c2) of the camera's pose rows
                const int gc = row - 2, g = gc / ni, c2 = gc - g * ni;
                for (int it = b0; it < b1; ++it) {
                    const int ob = D.lcam_obs[it];
                    const int info = s_info[ob];
                    const T* A = s_A + static_cast<size_t>(ob) * sA;
                    if (info_group(info) == g) {
                        const VT w = s_M[static_cast<size_t>(ob) * sM + 5];
                        acc.jacobian(A, A + nA, A[6 + c2] * w, A[nA + 6 + c2] * w);
                    }
                    const int ts = trk_slot(s_trk[ob]);
                    if ((info & kElim) && ts < ntc && ((s_tmask[ts] >> g) & 1)) {
                        const VT* Kt = s_K + static_cast<size_t>(ts) * sK + gc * 3;
                        if constexpr (kMixed)
                            acc.template coupling<false>(s_G4 + static_cast<size_t>(ob) * 9, -Kt[0], -Kt[1], -Kt[2]);
                        else
                            acc.template coupling<false>(s_G + static_cast<size_t>(ob) * sG, -Kt[0], -Kt[1], -Kt[2]);
                    }
                }
#pragma unroll
                for (int a = 0; a < 6; ++a) out[12 + (g * 6 + a) * ni + c2] = acc.part(a);
            }
        }
    }
    // Intrinsic block entries (i, j), i <= j, and intrinsic gradient entries: a warp takes up to four
    // entries of one row, its lanes striding over the chunk's observations and tracks, then a fixed
    // shuffle tree (the entries sum over every observation of the chunk, so a thread per entry would be
    // the chunk's critical path).  Warps that finish their rows above start here at once.
    if (nb > 0) {
        P* out = O.part_chunk + static_cast<size_t>(chunk) * chrec;
        // units of up to four columns: of a row within its own group (from the diagonal on), of a row
        // with a later group, of the reduced and of the direct gradient
        const int nq = (ni + 3) / 4;
        int own = 0;  // units of one group's own rows
        for (int c = 0; c < ni; ++c) own += (ni - c + 3) / 4;
        const int u_own = ng * own, u_cross = ng * (ng - 1) / 2 * ni * nq, u_all = u_own + u_cross + 2 * ng * nq;
        // a warp takes the next unit when it is free (an entry is summed the same way by any warp, so
        // the order of taking changes no result)
        for (;;) {
            int e = 0;
            if (lane == 0) e = atomicAdd(s_next_entry, 1);
            e = __shfl_sync(0xffffffffu, e, 0);
            if (e >= u_all) break;
            QuadAcc<T> acc;
            int at = 0, row = -1, col = 0, c0 = 0;  // first entry; row and column of the block (row < 0: gradient)
            if (e < u_own + u_cross) {
                int g1, c1, g2;
                if (e < u_own) {
                    g1 = g2 = e / own;
                    int r = e - g1 * own;
                    for (c1 = 0; r >= (ni - c1 + 3) / 4; ++c1) r -= (ni - c1 + 3) / 4;
                    c0 = c1 + 4 * r;
                } else {
                    int r = e - u_own;
                    const int pr = r / (ni * nq);
                    r -= pr * (ni * nq);
                    c1 = r / nq;
                    c0 = 4 * (r - c1 * nq);
                    g1 = 0;
                    int left = pr;
                    while (left >= ng - 1 - g1) left -= ng - 1 - g1++;
                    g2 = g1 + 1 + left;
                }
                row = g1 * ni + c1;
                col = g2 * ni + c0;
                at = row * nb + col;
                // columns beyond the group's last one repeat it and are not written
                const int k1 = min(c0 + 1, ni - 1), k2 = min(c0 + 2, ni - 1), k3 = min(c0 + 3, ni - 1);
                if (g1 == g2)
                    for (int ob = lane; ob < nobs; ob += 32) {
                        if (info_group(s_info[ob]) != g1) continue;
                        const T* A = s_A + static_cast<size_t>(ob) * sA + 6;
                        const VT w = s_M[static_cast<size_t>(ob) * sM + 5];
                        acc.weighted(w, A[c1], A[c0], A[k1], A[k2], A[k3]);
                        acc.weighted(w, A[nA + c1], A[nA + c0], A[nA + k1], A[nA + k2], A[nA + k3]);
                    }
                const int need = (1 << g1) | (1 << g2);
                for (int t = lane; t < ntc; t += 32) {
                    if ((s_tmask[t] & need) != need) continue;
                    const VT* K1 = s_K + static_cast<size_t>(t) * sK + row * 3;
                    const VT* K2 = s_K + static_cast<size_t>(t) * sK + g2 * ni * 3;
#pragma unroll
                    for (int kk = 0; kk < 3; ++kk)
                        acc.minus(K1[kk], K2[c0 * 3 + kk], K2[k1 * 3 + kk], K2[k2 * 3 + kk], K2[k3 * 3 + kk]);
                }
            } else {
                const int r = e - u_own - u_cross, half = r / (ng * nq);
                const int g = (r - half * ng * nq) / nq;
                c0 = 4 * (r - half * ng * nq - g * nq);
                at = nb * nb + half * nb + g * ni + c0;
                const int k1 = min(c0 + 1, ni - 1), k2 = min(c0 + 2, ni - 1), k3 = min(c0 + 3, ni - 1);
                for (int ob = lane; ob < nobs; ob += 32) {
                    if (info_group(s_info[ob]) != g) continue;
                    const VT* Dg = s_D + static_cast<size_t>(ob) * sD + 6;
                    acc.add(Dg[c0], Dg[k1], Dg[k2], Dg[k3]);
                    if (half == 0) {  // the reduced gradient
                        const T* A = s_A + static_cast<size_t>(ob) * sA + 6;
                        const VT* M = s_M + static_cast<size_t>(ob) * sM;
                        acc.jacobian(A[c0], A[k1], A[k2], A[k3], -M[3]);
                        acc.jacobian(A[nA + c0], A[nA + k1], A[nA + k2], A[nA + k3], -M[4]);
                    }
                }
            }
            __syncwarp();
            Acc<T> q[4];
            acc.split(q);
            const Acc<T> v = quad_merge(q);
            const int x = lane >> 3;  // the entry whose total this lane's group of eight holds
            if ((lane & 7) == 0 && c0 + x < ni) {
                out[at + x] = v.part();
                if (row >= 0 && row != col + x) out[(col + x) * nb + row] = v.part();
            }
        }
    }
    if (tid == 0) {
        double c = 0.0;
        for (int w = 0; w < static_cast<int>((blockDim.x + 31) >> 5); ++w) c += s_misc[w];
        if (S.ncp > 0)
            for (int t = 0; t < ntc; ++t) c += s_cpc[t];
        O.part_cost[chunk] = c;
        O.part_flags[chunk] = s_flags[0];
    }
}

template <typename T>
static AsmOutT<T> typed_out(const AsmOut& o) {
    using P = typename Acc<T>::part_type;
    return {static_cast<P*>(o.part_pair_v), static_cast<P*>(o.part_cam_v), static_cast<P*>(o.part_chunk_v),
            o.part_cost, o.part_flags, static_cast<double*>(o.trk_data_v), static_cast<T*>(o.obs_rec_v)};
}

template <typename T>
void launch_assemble(const Shape& S, const DevPtrs& D, const AsmOut& O, double damping, size_t smem, cudaStream_t st) {
    if (S.nchunks == 0) return;
    k_assemble<T><<<S.nchunks, kAssembleThreads, smem, st>>>(S, D, typed_out<T>(O), damping);
}

void pb_set_assemble_smem_f32(size_t bytes) {
    cudaFuncSetAttribute(k_assemble<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}
void pb_set_assemble_smem_f64(size_t bytes) {
    cudaFuncSetAttribute(k_assemble<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

template void launch_assemble<float>(const Shape&, const DevPtrs&, const AsmOut&, double, size_t, cudaStream_t);
template void launch_assemble<double>(const Shape&, const DevPtrs&, const AsmOut&, double, size_t, cudaStream_t);

}  // namespace pb
