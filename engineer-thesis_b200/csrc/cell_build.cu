// cell_build.cu -- cell lists: a uniform grid over the layer bounds whose
// cells list the rects a clearance query from inside the cell can need.
//
// For a point p of cell C with centre c and side s,
//     d*(p) <= d*(c) + |p - c|_inf <= d*(c) + s/2 =: U_C
// (d* is 1-Lipschitz in the L-inf norm, bounds distance included), and a
// rect R with gap(R, p) <= d*(p) + 2 delta has L-inf distance to C at most
// U_C + 2 delta.  So the rects touching C grown by
//     r_C = max(U_C, 0) + 2 delta + margin
// are every rect the query at p can find nearest, tied within 2 delta, or
// containing p (max with 0).  The margin (M * 2^-30, M the layout's
// coordinate scale) covers the rounding of the cell index of p and of the
// cell's coordinates, both of order M * 2^-50.  One pass over the cells finds
// the clearance at each cell centre, enumerates the rects of its grown box and
// writes its record (up to kCellSlots rects in place; a longer list goes to
// the shared list buffer at an offset from a global cursor, one atomic per
// block; lists past the buffer's first room are written by a second pass over
// their cells).  Large grids first build coarse cells (4 x 4 cells each) from the
// tree, in one pass of the same kind, and answer each cell's clearance and
// enumeration from its coarse cell's list.  Cells with more than max_per_cell rects are
// left to the tree.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <initializer_list>
#include <vector>

#include "query.cuh"

namespace frw {
namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
// rects that a thread of the coarse pass keeps
constexpr int kStage = 12;

// Visits the tree's rects touching the closed box B, in tree order, until
// visit() returns false.  Returns false when the traversal stack overflowed
// (the visit is then incomplete).
template <typename F>
__device__ __forceinline__ bool touching(const DevLayout &L, const double B[4], F &&visit) {
    int stk[kStackMax];
    int sp = 1;
    stk[0] = 0;
    const FloatBox fb = float_box(B);
    while (sp > 0) {
        const int nd = stk[--sp];
        const int4 rf = __ldg(L.nref + nd);
        const int ref[4] = {rf.x, rf.y, rf.z, rf.w};
        for (int c = 0; c < 4; c++) {
            if (ref[c] == kRefEmpty) continue;
            const float4 b = __ldg(L.nbox + 4 * nd + c);
            if (!fb.touches(b)) continue;
            if (ref[c] >= 0) {
                if (sp == kStackMax) return false;
                stk[sp++] = ref[c];
                continue;
            }
            const int f = leaf_first(ref[c]), m = leaf_count(ref[c]);
            for (int k = f; k < f + m; k++) {
                const float4 r = __ldg(L.rects + k);
                if (fb.touches(r) && !visit(k, r)) return true;
            }
        }
    }
    return true;
}

struct Grid {
    double gx0, gy0, side, margin;
    int nx, ny;
};

// The passes visit the cells in tiles of 8 x 4, one tile per warp, so
// that a warp's tree traversals start from neighbouring points and take
// similar paths: thread t gets cell (tile_x * 8 + t % 8, tile_y * 4 + t % 32
// / 8) of tile t / 32, or -1 past the grid's edge.
constexpr int kTileW = 8, kTileH = 4;
__device__ __forceinline__ int64_t tiled_cell(const Grid &G, int64_t t) {
    const int64_t tile = t >> 5;
    const int lane = (int)(t & 31);
    const int64_t tiles_x = (G.nx + kTileW - 1) / kTileW;
    const int64_t ix = (tile % tiles_x) * kTileW + (lane % kTileW), iy = (tile / tiles_x) * kTileH + lane / kTileW;
    return ix < G.nx && iy < G.ny ? iy * G.nx + ix : -1;
}
int64_t tiled_threads(int64_t nx, int64_t ny) {
    return ((nx + kTileW - 1) / kTileW) * ((ny + kTileH - 1) / kTileH) * 32;
}

// The box of cell c grown by r.
__device__ __forceinline__ void grown_box(const Grid &G, int64_t c, double r, double B[4]) {
    const int ix = (int)(c % G.nx), iy = (int)(c / G.nx);
    const double x0 = G.gx0 + ix * G.side, y0 = G.gy0 + iy * G.side;
    B[0] = x0 - r;
    B[1] = y0 - r;
    B[2] = (x0 + G.side) + r;
    B[3] = (y0 + G.side) + r;
}

// Coarse cells of a build: cell (first, count) into rects and ids, count -1
// when the cell overflowed.
struct CoarseLists {
    int2 *cells = nullptr;
    float4 *rects = nullptr;
    int32_t *ids = nullptr;
    int nx = 0, ny = 0;
};

// The radius r_C of a cell from the clearance best at its centre.
__device__ __forceinline__ double radius_of(const DevLayout &L, const Grid &G, double best) {
    return fmax(best, 0.0) + 0.5 * G.side + 2.0 * L.delta + G.margin;
}

// A point's distance to the bounds.
__device__ __forceinline__ double bounds_distance(const DevLayout &L, double x, double y) {
    return dmin(dmin(x - L.bx0, L.bx1 - x), dmin(y - L.by0, L.by1 - y));
}

// The centre of cell c.
__device__ __forceinline__ double2 centre_of(const Grid &G, int64_t c) {
    const int ix = (int)(c % G.nx), iy = (int)(c / G.nx);
    return make_double2(G.gx0 + ix * G.side + 0.5 * G.side, G.gy0 + iy * G.side + 0.5 * G.side);
}

// The place of this thread's `want` entries in a buffer with cursor *tot: a
// scan over the block, one atomic.  Every thread of the block calls it.
__device__ __forceinline__ unsigned long long block_offset(unsigned want, unsigned long long *tot,
                                                           unsigned *s_warp, unsigned long long *s_base, int warps) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned x = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned s = 0;
        for (int k = 0; k < warps; k++) s += s_warp[k];
        *s_base = s ? atomicAdd(tot, (unsigned long long)s) : 0ull;
    }
    __syncthreads();
    unsigned long long at = *s_base + (x - want);
    for (int k = 0; k < w; k++) at += s_warp[k];
    return at;
}

// Coarse cells, from the tree (L without cells): every rect touching the cell
// grown by its radius, one margin above the Lipschitz bound r_cell <= r_coarse;
// (0, -1) when there are more than cap or the enumeration was incomplete.  The
// lists go to the shared buffers at offsets from a global cursor (tot), a block
// scan and one atomic per block; past `room` entries they have their place and
// radius but are not written (k_fill_coarse does).  A thread keeps its first
// kStage rects in shared memory and enumerates longer lists again.
// Bound by the traversals' chains of loads, two per cell; a count pass, a scan
// and a fill pass with 48 bytes per cell between them took 0.69 ms for 10^6
// rects' 10^6 coarse cells, this one 0.55.
constexpr int kCoarseThreads = 128;
__global__ void __launch_bounds__(kCoarseThreads)
    k_coarse_lists(DevLayout L, Grid G, int cap, int2 *__restrict__ cells, float *__restrict__ crad,
                   float4 *__restrict__ crects, int32_t *__restrict__ cids, int64_t room, unsigned long long *tot,
                   int64_t nthreads) {
    __shared__ int32_t s_stage[kStage][kCoarseThreads];
    __shared__ unsigned s_warp[kCoarseThreads / 32];
    __shared__ unsigned long long s_base;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t c = t < nthreads ? tiled_cell(G, t) : -1;
    double B[4] = {0, 0, 0, 0};
    int n = 0;
    bool ok = false;
    if (c >= 0) {
        const double2 p = centre_of(G, c);
        Cands C;
        int hit;
        double best;
        clearance(L, p.x, p.y, C, hit, best, bounds_distance(L, p.x, p.y));
        const float radius = __double2float_ru(radius_of(L, G, best) + G.margin);
        crad[c] = radius;
        grown_box(G, c, (double)radius, B);
        const bool complete = touching(L, B, [&](int k, float4) {
            if (n < kStage) s_stage[n][threadIdx.x] = k;
            return ++n <= cap;
        });
        ok = complete && n <= cap;
    }
    const unsigned want = ok ? (unsigned)n : 0u;
    const unsigned long long at = block_offset(want, tot, s_warp, &s_base, kCoarseThreads / 32);
    if (c < 0) return;
    cells[c] = make_int2(ok ? (int)at : 0, ok ? n : -1);
    if (!want || at + want > (unsigned long long)room) return;
    if (n <= kStage) {
        for (int i = 0; i < n; i++) {
            const int k = s_stage[i][threadIdx.x];
            crects[at + i] = __ldg(L.rects + k);
            cids[at + i] = __ldg(L.ids + k);
        }
    } else {
        int m = 0;
        touching(L, B, [&](int k, float4 r) {
            crects[at + m] = r;
            cids[at + m] = __ldg(L.ids + k);
            return ++m < n;
        });
    }
}

// The lists that k_coarse_lists had no room for, one traversal each: k_coarse_lists
// run again, two or three traversals each, made dense layouts slower to build than
// its count and fill passes had been (3e5 overlapping rects, 16 a coarse cell,
// 1.95 -> 1.40 ms in all against 1.42).
__global__ void __launch_bounds__(kCoarseThreads)
    k_fill_coarse(DevLayout L, Grid G, const int2 *__restrict__ cells, const float *__restrict__ crad,
                  float4 *__restrict__ crects, int32_t *__restrict__ cids, int64_t room, int64_t nthreads) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t c = t < nthreads ? tiled_cell(G, t) : -1;
    if (c < 0) return;
    const int2 ce = cells[c];
    if (ce.y <= 0 || (int64_t)ce.x + ce.y <= room) return;
    double B[4];
    grown_box(G, c, (double)crad[c], B);
    int m = 0;
    touching(L, B, [&](int k, float4 r) {
        crects[ce.x + m] = r;
        cids[ce.x + m] = __ldg(L.ids + k);
        return ++m < ce.y;
    });
}

constexpr int kRecordThreads = 256;

// The records of the cells, radii included.  kCoarse: rects come from the
// coarse cell (of `factor` x `factor` cells) covering the cell -- its list
// holds every rect the clearance at the centre and the grown box can need --
// unless it overflowed; else from the tree.  tot[0]: list entries reserved,
// tot[1]: entries of all cells (records included), tot[2]: cells left to the
// tree.  Lists past `room` entries have their place and radius in the record but
// are not written (k_fill_lists does).
// Bound by its writes (84 bytes a cell: 16e6 cells at 10^6 rects take 0.2 ms
// at the copy rate) and the FP64 gaps of the coarse lists (about 6 rects,
// twice); it replaces a count pass, a scan and a fill pass with 84 bytes of
// counts, radii and staged positions per cell between them.

// Visits the rects touching B in a fixed order: those of the coarse cell ce, or
// the tree's.  visit(layer index, rect) says whether to go on; false when the
// enumeration was incomplete.
template <bool kCoarse, typename F>
__device__ __forceinline__ bool each_touching(const DevLayout &L, const CoarseLists &K, int2 ce, const double B[4],
                                              F &&visit) {
    if (!kCoarse || ce.y < 0) return touching(L, B, [&](int k, float4 r) { return visit(L.ids + k, r); });
    const FloatBox fb = float_box(B);
    for (int k = ce.x; k < ce.x + ce.y; k++) {
        const float4 r = __ldg(K.rects + k);
        if (fb.touches(r) && !visit(K.ids + k, r)) break;
    }
    return true;
}

// The coarse cell covering cell c.
__device__ __forceinline__ int2 coarse_of(const CoarseLists &K, const Grid &G, int factor, int64_t c) {
    const int ix = (int)(c % G.nx), iy = (int)(c / G.nx);
    return __ldg(K.cells + (int64_t)(iy / factor) * K.nx + ix / factor);
}

template <bool kCoarse>
__global__ void __launch_bounds__(kRecordThreads)
    k_cell_records(DevLayout L, CoarseLists K, Grid G, int factor, int cap, float4 *__restrict__ cells,
                   int4 *__restrict__ cellids, float *__restrict__ crad, float4 *__restrict__ crects,
                   int32_t *__restrict__ cids, int64_t room, unsigned long long *tot, int64_t nthreads) {
    __shared__ unsigned s_warp[kRecordThreads / 32];
    __shared__ unsigned long long s_base;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t c = t < nthreads ? tiled_cell(G, t) : -1;
    int2 ce = make_int2(0, -1);
    double B[4] = {0, 0, 0, 0};
    int n = 0;
    bool tree = false, near = false;
    float radius = 0.f;
    auto each = [&](auto &&visit) { return each_touching<kCoarse>(L, K, ce, B, visit); };
    if (c >= 0) {
        const double2 p = centre_of(G, c);
        // clearance at the centre: of the bounds, and of the rects (at least)
        const double bd = bounds_distance(L, p.x, p.y);
        double gap = 1e300;
        if (kCoarse) ce = coarse_of(K, G, factor, c);
        if (kCoarse && ce.y >= 0) {
            // the clearance in FP32 on a split centre (two roundings of the gap's
            // own size), raised past its error: a radius a hair larger is as good
            const float xh = (float)p.x, yh = (float)p.y;
            const float xl = (float)(p.x - (double)xh), yl = (float)(p.y - (double)yh);
            float g = 3.0e38f;
            for (int k = ce.x; k < ce.x + ce.y; k++) {
                const float4 r = __ldg(K.rects + k);
                g = fminf(g, fmaxf(fmaxf((r.x - xh) - xl, (xh - r.z) + xl), fmaxf((r.y - yh) - yl, (yh - r.w) + yl)));
            }
            gap = (double)g + fabs((double)g) * 0x1p-21 + L.delta;
        } else {
            Cands C;
            int hit;
            if (bd >= 0.0) clearance(L, p.x, p.y, C, hit, gap, 1e300);
        }
        // both clearances change by at most the distance moved: no point of a
        // cell that is not `near` has the bounds as near as its nearest rect or 3
        near = !(bd - 0.5 * G.side > dmax(gap + 0.5 * G.side, 3.0) + 2.0 * L.delta + G.margin);
        // (raised to FP32: the record keeps it)
        radius = __double2float_ru(radius_of(L, G, dmin(bd, gap)));
        grown_box(G, c, (double)radius, B);
        // a point of the cell lies within margin/2 of it whatever the rounding of
        // its cell index, so every rect within radius - margin of the point is listed
        crad[c] = __double2float_rd((double)radius - G.margin);
        float4 *rec = cells + kCellSlots * c;
        int32_t *rid = reinterpret_cast<int32_t *>(cellids + c);
        const bool complete = each([&](const int32_t *id, float4 q) {
            if (n < kCellSlots) {
                rec[n] = q;
                rid[n] = __ldg(id);
            }
            return ++n <= cap;
        });
        tree = !complete || n > cap;
        for (int k = n; k < kCellSlots; k++) {
            rec[k] = make_float4(kFarRect, kFarRect, kFarRect, kFarRect);
            rid[k] = -1;
        }
    }
    // totals, and the offsets of the longer lists
    const unsigned want = !tree && n >= kCellSlots + (near ? 0 : 1) ? (unsigned)n : 0u;
    const unsigned kept = __reduce_add_sync(0xFFFFFFFFu, tree ? 0u : (unsigned)n);
    const unsigned trees = __popc(__ballot_sync(0xFFFFFFFFu, tree));
    if ((threadIdx.x & 31) == 0) {
        if (kept) atomicAdd(tot + 1, (unsigned long long)kept);
        if (trees) atomicAdd(tot + 2, (unsigned long long)trees);
    }
    const unsigned long long at = block_offset(want, tot, s_warp, &s_base, kRecordThreads / 32);
    if (c < 0 || !(want || tree || near)) return;
    float4 *rec = cells + kCellSlots * c;
    rec[kCellSlots - 1] = make_float4(kListRect, __int_as_float(tree ? 0 : (int)at), __int_as_float(tree ? kTreeCell : n),
                                      radius);
    if (!want || at + want > (unsigned long long)room) return;
    int m = 0;
    each([&](const int32_t *id, float4 q) {
        crects[at + m] = q;
        cids[at + m] = __ldg(id);
        return ++m < n;
    });
}

// The lists that k_cell_records had no room for: cells whose list ends past
// `room` take their rects again, by the radius in their record, and write them
// at their place (the lists before it are copied).  Only these cells do any
// work: the whole pass run again made layouts of long lists slower to build than
// a count and a fill pass had been (3e5 clustered rects 3.28 -> 1.96 ms against
// 2.25, 3e5 rects at one cell each 0.72 -> 0.52 against 0.64).
template <bool kCoarse>
__global__ void __launch_bounds__(kRecordThreads)
    k_fill_lists(DevLayout L, CoarseLists K, Grid G, int factor, const float4 *__restrict__ cells,
                 float4 *__restrict__ crects, int32_t *__restrict__ cids, int64_t room, int64_t nthreads) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t c = t < nthreads ? tiled_cell(G, t) : -1;
    if (c < 0) return;
    const float4 last = cells[kCellSlots * c + kCellSlots - 1];
    const int at = __float_as_int(last.y), n = __float_as_int(last.z);
    if (!(last.x > kFarRect) || n < kCellSlots || (int64_t)at + n <= room) return;
    double B[4];
    grown_box(G, c, (double)last.w, B);
    int m = 0;
    each_touching<kCoarse>(L, K, kCoarse ? coarse_of(K, G, factor, c) : make_int2(0, -1), B,
                           [&](const int32_t *id, float4 q) {
                               crects[at + m] = q;
                               cids[at + m] = __ldg(id);
                               return ++m < n;
                           });
}

// Exclusive scan of int64 values: tile sums, a one-block scan of the tile
// sums, then each tile rescanned with its offset.
__device__ __forceinline__ int64_t block_excl_scan(int64_t v, int64_t *warp_tot, int64_t &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        int64_t t = lane < kScanThreads / 32 ? warp_tot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t;  // inclusive over warps
    }
    __syncthreads();
    total = warp_tot[kScanThreads / 32 - 1];
    const int64_t before = w ? warp_tot[w - 1] : 0;
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) k_tile_sums(const int64_t *__restrict__ in, int64_t n,
                                                          int64_t *__restrict__ sums) {
    __shared__ int64_t wt[32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int64_t s = 0;
    for (int k = 0; k < kScanItems; k++)
        if (base + k < n) s += in[base + k];
    int64_t total;
    block_excl_scan(s, wt, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sums(int64_t *sums, int64_t n, int64_t *grand) {
    __shared__ int64_t wt[32];
    int64_t carry = 0;
    for (int64_t b = 0; b < n; b += kScanThreads) {
        const int64_t i = b + threadIdx.x;
        const int64_t v = i < n ? sums[i] : 0;
        int64_t total;
        const int64_t e = block_excl_scan(v, wt, total);
        if (i < n) sums[i] = carry + e;
        carry += total;
    }
    if (threadIdx.x == 0) *grand = carry;
}

__global__ void __launch_bounds__(kScanThreads) k_tile_scan(const int64_t *__restrict__ in, int64_t n,
                                                          const int64_t *__restrict__ offs,
                                                          int64_t *__restrict__ out) {
    __shared__ int64_t wt[32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    int64_t v[kScanItems], s = 0;
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    int64_t total;
    int64_t run = offs[blockIdx.x] + block_excl_scan(s, wt, total);
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
}

}  // namespace

void free_cells(CellBuffers *c, cudaStream_t st) {
    for (void *p : {(void *)c->cells, (void *)c->cellids, (void *)c->crects, (void *)c->cids, (void *)c->crad})
        if (p) cudaFreeAsync(p, st);
    *c = CellBuffers();
}

void attach_cells(DevLayout &L, const CellBuffers &c) {
    L.cells = c.cells;
    L.cellids = c.cellids;
    L.crects = c.crects;
    L.cids = c.cids;
    L.crad = c.crad;
    L.gx0 = c.gx0;
    L.gy0 = c.gy0;
    L.ginv = c.ginv;
    L.gnx = c.nx;
    L.gny = c.ny;
    L.tree_points = c.cells == nullptr || c.overflow > 0;
}

namespace {

// Coarse cells, of kCoarse x kCoarse cells each, serve the build of grids of
// at least kTwoLevelMin cells: their lists (from the tree, up to kCoarseCap
// rects) answer the cells' clearance and enumeration, so the tree is
// traversed once per coarse cell instead of once per cell.
constexpr int kCoarse = 4;
constexpr int64_t kTwoLevelMin = 1 << 16;
constexpr int kCoarseCap = 64;

// Device buffers of a build, released in stream order at scope exit unless
// taken.
struct BuildBufs {
    std::vector<void *> p;
    cudaStream_t st;
    explicit BuildBufs(cudaStream_t s) : st(s) {}
    template <typename T>
    frw_status get(T **x, size_t bytes, const char *what) {
        const cudaError_t e = cudaMallocAsync((void **)x, std::max<size_t>(bytes, 16), st);
        if (e != cudaSuccess) return cuda_fail(e, what);
        p.push_back(*x);
        return FRW_OK;
    }
    void drop(void *q) {
        p.erase(std::find(p.begin(), p.end(), q));
        cudaFreeAsync(q, st);
    }
    void take(void *q) { p.erase(std::find(p.begin(), p.end(), q)); }
    ~BuildBufs() {
        for (void *q : p) cudaFreeAsync(q, st);
    }
};

// Coarse cells over the tree of L.
frw_status build_coarse(const DevLayout &L, const Grid &G, cudaStream_t st, BuildBufs &B, CoarseLists *K) {
    const int64_t ncells = (int64_t)G.nx * G.ny, nt = tiled_threads(G.nx, G.ny);
    frw_status rc;
    unsigned long long *tot, total = 0;
    float *crad;
    if ((rc = B.get(&K->cells, (size_t)ncells * sizeof(int2), "malloc coarse cells"))) return rc;
    if ((rc = B.get(&crad, (size_t)ncells * sizeof(float), "malloc coarse radii"))) return rc;
    if ((rc = B.get(&tot, 8, "malloc total"))) return rc;
    // room for 12 rects a cell (8 to 9 at the benchmark's densities); k_fill_coarse writes the lists past it
    const int64_t room = std::max<int64_t>(12 * ncells, 4096);
    float4 *rects;
    int32_t *ids;
    if ((rc = B.get(&rects, (size_t)room * 16, "malloc coarse rects"))) return rc;
    if ((rc = B.get(&ids, (size_t)room * 4, "malloc coarse ids"))) return rc;
    FRW_CK(cudaMemsetAsync(tot, 0, 8, st));
    const unsigned blocks = (unsigned)((nt + kCoarseThreads - 1) / kCoarseThreads);
    k_coarse_lists<<<blocks, kCoarseThreads, 0, st>>>(L, G, kCoarseCap, K->cells, crad, rects, ids, room, tot, nt);
    FRW_CK(cudaGetLastError());
    if ((rc = read_back(&total, tot, 8, st, "build_cells: coarse list total"))) return rc;
    if (total > INT32_MAX) {
        set_error("build_cells: more than 2^31 list entries; use fewer cells per rect");
        return FRW_E_ARG;
    }
    K->rects = rects;
    K->ids = ids;
    if ((int64_t)total > room) {
        if ((rc = B.get(&K->rects, (size_t)total * 16, "malloc coarse rects"))) return rc;
        if ((rc = B.get(&K->ids, (size_t)total * 4, "malloc coarse ids"))) return rc;
        FRW_CK(cudaMemcpyAsync(K->rects, rects, (size_t)room * 16, cudaMemcpyDeviceToDevice, st));
        FRW_CK(cudaMemcpyAsync(K->ids, ids, (size_t)room * 4, cudaMemcpyDeviceToDevice, st));
        B.drop(rects);
        B.drop(ids);
        k_fill_coarse<<<blocks, kCoarseThreads, 0, st>>>(L, G, K->cells, crad, K->rects, K->ids, room, nt);
        FRW_CK(cudaGetLastError());
    }
    K->nx = G.nx;
    K->ny = G.ny;
    return FRW_OK;
}

// The records of grid G over L (from coarse cells when K has any), the
// buffers in C.
frw_status build_records(const DevLayout &L, const CoarseLists &K, const Grid &G, int cap, cudaStream_t st,
                         BuildBufs &B, CellBuffers &C) {
    const int64_t ncells = (int64_t)G.nx * G.ny, nt = tiled_threads(G.nx, G.ny);
    C.ncells = ncells;
    C.nx = G.nx;
    C.ny = G.ny;
    C.gx0 = G.gx0;
    C.gy0 = G.gy0;
    C.side = G.side;
    C.ginv = 1.0 / G.side;
    frw_status rc;
    unsigned long long *tot;
    if ((rc = B.get(&C.cells, (size_t)ncells * kCellSlots * sizeof(float4), "malloc cells"))) return rc;
    if ((rc = B.get(&C.cellids, (size_t)ncells * sizeof(int4), "malloc cell ids"))) return rc;
    if ((rc = B.get(&C.crad, (size_t)ncells * sizeof(float), "malloc cell radii"))) return rc;
    if ((rc = B.get(&tot, 24, "malloc totals"))) return rc;
    // half an entry of list room per cell holds the lists of the benchmark's
    // densities (0.16 at 16 cells per rect); k_fill_lists writes those past it
    const int64_t room = std::max<int64_t>(ncells / 2, 4096);
    unsigned long long h[3] = {0, 0, 0};
    float4 *rects = nullptr;
    int32_t *ids = nullptr;
    if ((rc = B.get(&rects, (size_t)room * 16, "malloc cell rects"))) return rc;
    if ((rc = B.get(&ids, (size_t)room * 4, "malloc cell ids"))) return rc;
    FRW_CK(cudaMemsetAsync(tot, 0, 24, st));
    const unsigned blocks = (unsigned)((nt + kRecordThreads - 1) / kRecordThreads);
    const auto records = K.cells ? k_cell_records<true> : k_cell_records<false>;
    records<<<blocks, kRecordThreads, 0, st>>>(L, K, G, kCoarse, cap, C.cells, C.cellids, C.crad, rects, ids, room, tot,
                                               nt);
    FRW_CK(cudaGetLastError());
    if ((rc = read_back(h, tot, 24, st, "build_cells: list total"))) return rc;
    if (h[0] >= (unsigned long long)kMaxListEntries) {
        set_error("build_cells: more than 2^31 list entries; use fewer cells per rect");
        return FRW_E_ARG;
    }
    // the lists in buffers of their size
    const int64_t total = (int64_t)h[0], written = std::min(total, room);
    if ((rc = B.get(&C.crects, (size_t)total * 16, "malloc cell rects"))) return rc;
    if ((rc = B.get(&C.cids, (size_t)total * 4, "malloc cell ids"))) return rc;
    if (written) {
        FRW_CK(cudaMemcpyAsync(C.crects, rects, (size_t)written * 16, cudaMemcpyDeviceToDevice, st));
        FRW_CK(cudaMemcpyAsync(C.cids, ids, (size_t)written * 4, cudaMemcpyDeviceToDevice, st));
    }
    if (total > room) {
        const auto fill = K.cells ? k_fill_lists<true> : k_fill_lists<false>;
        fill<<<blocks, kRecordThreads, 0, st>>>(L, K, G, kCoarse, C.cells, C.crects, C.cids, room, nt);
        FRW_CK(cudaGetLastError());
    }
    C.entries = (int64_t)h[1];
    C.overflow = (int64_t)h[2];
    C.bytes = ncells * (int64_t)(kCellSlots * sizeof(float4) + sizeof(int4) + sizeof(float)) + total * 20;
    for (void *q : {(void *)C.cells, (void *)C.cellids, (void *)C.crad, (void *)C.crects, (void *)C.cids}) B.take(q);
    return FRW_OK;
}

}  // namespace

frw_status build_cells(const DevLayout &Lin, double cells_per_rect, int cap, cudaStream_t st, CellBuffers *out) {
    *out = CellBuffers();
    if (!(cells_per_rect > 0) || cap < 1 || cap > (1 << 16)) {
        set_error("build_cells: cells_per_rect must be > 0 and max_per_cell in [1, 65536]");
        return FRW_E_ARG;
    }
    DevLayout L = Lin;
    L.cells = nullptr;  // the build queries the tree (and coarse lists of its own)
    const double W = L.bx1 - L.bx0, H = L.by1 - L.by0;
    const double target = std::min((double)kMaxCells, std::max(1.0, cells_per_rect * (double)L.n));
    double side = std::sqrt(std::max(W * H, 1e-300) / target);
    if (!(side > 0) || !std::isfinite(side)) side = std::max(std::max(W, H), 1.0);
    side = std::max(side, std::max(W, H) / 65536.0);  // at most 2^16 cells per axis
    if (!(side > 0)) side = 1.0;
    int64_t nx = 0, ny = 0;
    for (;;) {
        nx = std::max<int64_t>(1, (int64_t)std::ceil(W / side));
        ny = std::max<int64_t>(1, (int64_t)std::ceil(H / side));
        if (nx * ny <= kMaxCells && nx <= 65536 && ny <= 65536) break;
        side *= 1.25;
    }
    const int64_t ncells = nx * ny;
    const double M = 4.0 * std::max(std::max(std::max(std::fabs(L.bx0), std::fabs(L.by0)),
                                             std::max(std::fabs(L.bx1), std::fabs(L.by1))),
                                    std::max(W, H)) +
                     16.0;
    const double margin = std::ldexp(M, -30);
    const Grid G{L.bx0, L.by0, side, margin, (int)nx, (int)ny};

    Events ev(2);
    if (!ev.ok(2)) return cuda_fail(cudaErrorUnknown, "build_cells: cudaEventCreate");
    FRW_CK(cudaEventRecord(ev[0], st));
    CellBuffers C;
    {
        BuildBufs B(st);
        CoarseLists K;
        frw_status rc = FRW_OK;
        if (ncells >= kTwoLevelMin) {
            const Grid Gk{L.bx0, L.by0, side * kCoarse, margin, (int)((nx + kCoarse - 1) / kCoarse),
                          (int)((ny + kCoarse - 1) / kCoarse)};
            rc = build_coarse(L, Gk, st, B, &K);
        }
        if (!rc) rc = build_records(L, K, G, cap, st, B, C);
        if (rc) return rc;
    }
    frw_status rc = FRW_OK;
    const cudaError_t e = cudaEventRecord(ev[1], st);
    if (e != cudaSuccess) rc = cuda_fail(e, "event");
    if (!rc) rc = wait_event(ev[1], "build_cells");
    if (rc) {
        free_cells(&C, st);
        return rc;
    }
    cudaEventElapsedTime(&C.build_ms, ev[0], ev[1]);
    *out = C;
    return FRW_OK;
}

int64_t scan_i64_tiles(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

void launch_scan_i64(const int64_t *in, int64_t n, int64_t *out, int64_t *sums, int64_t *grand, cudaStream_t st) {
    const int64_t tiles = scan_i64_tiles(n);
    k_tile_sums<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, sums);
    k_scan_sums<<<1, kScanThreads, 0, st>>>(sums, tiles, grand);
    k_tile_scan<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, sums, out);
}

}  // namespace frw
