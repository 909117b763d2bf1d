// query.cu -- batched collision queries and the Gaussian-surface kernel.
#include "query.cuh"

namespace frw {
namespace {

// A square in one 256-bit store (32-byte aligned), past the caches that the
// cells want.
__device__ __forceinline__ void store_square(double4 *p, const double s[4]) {
    asm volatile("st.global.cs.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(s[0]), "d"(s[1]), "d"(s[2]), "d"(s[3])
                 : "memory");
}

// One point per thread: drawBiggestSquareAtPoint + checkCollisons(point),
// batched (the reference issues them one walk hop at a time,
// Cuda/randomwalk.cu:102-103).  kTies: L.tree_points is set, so points with
// many exact ties can reach the whole-tree replay (compiled out otherwise).
// Random points: bound by the reads of their records, in L2 for 10^4 rects (a
// warp's 32 records are 64 separate 32-byte reads; 16-byte reads doubled the
// L1 lookups, 1e7 points 0.304 -> 0.228 ms) and in HBM for 10^6 (150 bytes read
// and 40 written per point, 0.545 -> 0.432 ms by now).  24 blocks of 64 per SM:
// a block ends with its slowest lane, so small ones refill the SM sooner (0.216
// -> 0.208 and 0.436 -> 0.432 ms against 12 of 128; 10 of 128: 0.229; 28 of 64
// spill: 0.267).  Records fetched ahead of their points -- through shared memory
// by asynchronous copies, or the coordinates alone in a persistent grid -- were
// slower (1.05 and 0.59 ms).
// With the tree's code (kTies) a point's chain of nodes is what its warp waits
// for: 24 blocks as well, at 40 registers (4e6 points on 10^4 rects 1.318 ->
// 1.215 ms, on 3e5 1.49 -> 1.33, partly overflowed cells 0.70 -> 0.59; 16 blocks
// 1.375, 1.54 and 0.69), but the spills lengthen the chain, so points that are
// all resident at once anyway take 16 at 64 registers (1000 points on 10^4
// rects 55 us a call against 65).
constexpr int kQueryThreads = 64;
constexpr int64_t kTreeWave = 148 * 16 * kQueryThreads;
template <bool kTies, int kBlocks>
__global__ void __launch_bounds__(kQueryThreads, kBlocks)
    k_query(DevLayout L, const double2 *__restrict__ pts, int64_t n, double4 *__restrict__ sq,
            int64_t *__restrict__ hit, uint32_t *status) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t st = 0;
    if (i < n) {
        const double2 p = __ldcs(pts + i);
        double s[4];
        int h;
        if (kTies) st = query_point(L, p.x, p.y, s, h);
        else query_record<false>(L, p.x, p.y, s, h, st);
        store_square(sq + i, s);
        __stcs((long long *)hit + i, h == kNoHit ? -1ll : (long long)h);
    }
    if (st) atomicOr(status, st);
}

__global__ void __launch_bounds__(128) k_box(DevLayout L, const double4 *__restrict__ boxes, int64_t n,
                                             bool has_ign, double4 ign, uint8_t *__restrict__ out,
                                             uint32_t *status) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t st = 0;
    if (i < n) {
        const double4 b = boxes[i];
        const double B[4] = {b.x, b.y, b.z, b.w};
        const double I[4] = {ign.x, ign.y, ign.z, ign.w};
        out[i] = box_collides(L, B, has_ign, I, st) ? 1 : 0;
    }
    if (st) atomicOr(status, st);
}

// RectHost::createGaussianSurface (CPU/rectHost.cpp:84-100).
__device__ void scale_rect(const double r[4], double fx, double fy, double o[4]) {
    const double mx = __dmul_rn(__dadd_rn(r[0], r[2]), 0.5);
    const double my = __dmul_rn(__dadd_rn(r[1], r[3]), 0.5);
    const double vx = __dmul_rn(__dsub_rn(r[0], mx), fx);
    const double vy = __dmul_rn(__dsub_rn(r[1], my), fy);
    o[0] = __dadd_rn(mx, vx);
    o[1] = __dadd_rn(my, vy);
    o[2] = __dsub_rn(mx, vx);
    o[3] = __dsub_rn(my, vy);
}

// Tree::getAdjustedGaussianFactor (CPU/quadTree.cpp:315-349): bisection of
// the per-axis scale factor against collisions that ignore the target.
__device__ double adjusted_factor(const DevLayout &L, const double r[4], double factor, bool axis_y,
                                  uint32_t &st) {
    bool dividing = true, first = true;
    double adj = factor, lb = 1.0, rb = factor, s[4];
    for (int i = 0; i < 10; i++) {  // GAUSSIAN_ACCURACY
        if (axis_y) scale_rect(r, 1.0, adj, s);
        else scale_rect(r, adj, 1.0, s);
        const bool isc = box_collides(L, s, true, r, st);
        if (first && !isc) break;
        if ((isc && !dividing) || (!isc && dividing)) dividing = !dividing;
        const double mid = __dmul_rn(__dadd_rn(lb, rb), 0.5);
        if (dividing) adj = rb = mid;
        else adj = lb = mid;
        first = false;
    }
    return adj;
}

// creatGaussianSurfFrom (scale mode) or the target grown by `param`.
__device__ void gauss_one(const DevLayout &L, const double4 t, int mode, double param, double o[4], uint32_t &st) {
    const double r[4] = {t.x, t.y, t.z, t.w};
    if (mode == FRW_GAUSS_SCALE) {
        if (param < 1.0) {  // creatGaussianSurfFrom returns the rect itself
            o[0] = r[0]; o[1] = r[1]; o[2] = r[2]; o[3] = r[3];
        } else {
            const double fx = adjusted_factor(L, r, param, false, st);
            const double fy = adjusted_factor(L, r, param, true, st);
            scale_rect(r, fx, fy, o);
        }
    } else {
        o[0] = __dsub_rn(r[0], param);
        o[1] = __dsub_rn(r[1], param);
        o[2] = __dadd_rn(r[2], param);
        o[3] = __dadd_rn(r[3], param);
    }
}

__global__ void k_gauss(DevLayout L, const double4 *__restrict__ targets, int n, int mode, double param,
                        double4 *__restrict__ out, uint32_t *status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double o[4];
    uint32_t st = 0;
    gauss_one(L, targets[i], mode, param, o, st);
    out[i] = make_double4(o[0], o[1], o[2], o[3]);
    if (st) atomicOr(status, st);
}

__global__ void k_gauss_of(DevLayout L, double4 target, int mode, double param, double4 *__restrict__ out,
                           uint32_t *status) {
    double o[4];
    uint32_t st = 0;
    gauss_one(L, target, mode, param, o, st);
    *out = make_double4(o[0], o[1], o[2], o[3]);
    if (st) atomicOr(status, st);
}

// One job per thread, each on its own layout (batched runs).
__global__ void k_gauss_jobs(const WalkJob *__restrict__ jobs, const double4 *__restrict__ targets, int n, int mode,
                             double param, double4 *__restrict__ out, uint32_t *status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double o[4];
    uint32_t st = 0;
    gauss_one(jobs[i].L, targets[i], mode, param, o, st);
    out[i] = make_double4(o[0], o[1], o[2], o[3]);
    if (st) atomicOr(status, st);
}

}  // namespace

frw_status launch_gauss_jobs(const WalkJob *d_jobs, const double *d_targets, int njobs, int mode, double param,
                             double *d_out, uint32_t *d_status, cudaStream_t stream) {
    if (njobs <= 0) return FRW_OK;
    k_gauss_jobs<<<(njobs + 63) / 64, 64, 0, stream>>>(d_jobs, (const double4 *)d_targets, njobs, mode, param,
                                                      (double4 *)d_out, d_status);
    FRW_CK(cudaGetLastError());
    return FRW_OK;
}

frw_status launch_query(const DevLayout &L, const double *d_pts, int64_t n, double *d_sq, int64_t *d_hit,
                        uint32_t *d_status, cudaStream_t stream) {
    if (n <= 0) return FRW_OK;
    const int T = kQueryThreads;
    const unsigned g = (unsigned)((n + T - 1) / T);
    const auto kernel = !L.tree_points ? k_query<false, 24> : n <= kTreeWave ? k_query<true, 16> : k_query<true, 24>;
    kernel<<<g, T, 0, stream>>>(L, (const double2 *)d_pts, n, (double4 *)d_sq, d_hit, d_status);
    FRW_CK(cudaGetLastError());
    return FRW_OK;
}

frw_status launch_box_collides(const DevLayout &L, const double *d_boxes, int64_t n, bool has_ignore,
                               const double ignore[4], uint8_t *d_out, uint32_t *d_status,
                               cudaStream_t stream) {
    if (n <= 0) return FRW_OK;
    const int T = 128;
    double4 ig = has_ignore ? make_double4(ignore[0], ignore[1], ignore[2], ignore[3])
                            : make_double4(0, 0, 0, 0);
    k_box<<<(unsigned)((n + T - 1) / T), T, 0, stream>>>(L, (const double4 *)d_boxes, n, has_ignore, ig,
                                                         d_out, d_status);
    FRW_CK(cudaGetLastError());
    return FRW_OK;
}

frw_status launch_gauss_of(const DevLayout &L, const double t[4], int mode, double param, double *d_out,
                           uint32_t *d_status, cudaStream_t stream) {
    k_gauss_of<<<1, 1, 0, stream>>>(L, make_double4(t[0], t[1], t[2], t[3]), mode, param, (double4 *)d_out, d_status);
    FRW_CK(cudaGetLastError());
    return FRW_OK;
}

frw_status launch_gauss(const DevLayout &L, const double *d_targets, int n, int mode, double param,
                        double *d_out, uint32_t *d_status, cudaStream_t stream) {
    if (n <= 0) return FRW_OK;
    k_gauss<<<(n + 63) / 64, 64, 0, stream>>>(L, (const double4 *)d_targets, n, mode, param,
                                              (double4 *)d_out, d_status);
    FRW_CK(cudaGetLastError());
    return FRW_OK;
}

}  // namespace frw
