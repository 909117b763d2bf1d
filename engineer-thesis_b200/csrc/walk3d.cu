// walk3d.cu -- 3-D floating random walk on box conductors: cell-grid build,
// clearance queries and the persistent walk kernel.
//
// The reference has no 3-D walk (its cube Green's function, green/green.cpp:
// 232-431, is never called); this is its 2-D walk (CPU/mainFunctions.cpp:
// 48-90) lifted to cubes, written for B200 the way the 2-D kernels are:
//   * the clearance query reads one cell record and a short list of box
//     copies (32 bytes each), sorted by distance from the cell centre so
//     the scan stops at the first entry that cannot be nearer -- no tree
//     descent and no stack;
//   * the cell lists are built on the device: boxes binned by overlap
//     (count -> scan -> fill), then a warp per brick of 32 cells gathers the
//     boxes that its cells can need into shared memory and every lane finds
//     its cell's nearest box and list among them;
//   * the walk kernel is persistent (SM count x resident blocks); a warp
//     claims walks in chunks from one global counter and refills its idle
//     lanes every four hops, so lanes stay busy while walks of very different
//     lengths finish;
//   * random numbers are Philox4x32-10 words keyed by (seed) with counter
//     (t / 4, walk, stream): the trajectory of a walk depends only on its
//     index, so the CPU oracle replays every walk bit for bit;
//   * the landing bin comes from a 2^14-entry guide in shared memory and the
//     32-bit CDF thresholds (shared memory, or L1) -- one or two compares;
//   * FP64 geometry with explicitly rounded operations (no contraction):
//     exactly the oracle's arithmetic.
#include <math.h>

#include <algorithm>
#include <vector>

#include "frw3d_internal.h"
#include "query.cuh"

namespace frw {
namespace {

// Two launch shapes of 32 warps per SM at 64 registers: four blocks of 256,
// or one of 1024 that also holds the CDF thresholds in shared memory (60 KB at
// n = 50, read at a random place in every hop: from L1 they competed with the
// cells' lists, 78 -> 92% hits without them; 1e7 walks on 10^4 boxes 4.10 ->
// 3.47 ms, four rows of 10^5 boxes 1.10 -> 0.99 ms).
constexpr int kW3Threads = 256;
constexpr int kW3MinBlocks = 4;
constexpr int kW3BigThreads = 1024;
constexpr size_t kW3ThrBytes = 96 << 10;  // thresholds that fit beside the guide (n <= 64)
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int64_t kMaxCells3 = int64_t(1) << 26;
constexpr int kMaxAxisCells3 = 1 << 14;

// ---- grid ------------------------------------------------------------------
struct Grid3 {
    double o[3];   // origin
    double side, inv, h, margin;
    int n[3];
    int cap;       // largest search radius in rings (the top level: no cap)
};

__device__ __forceinline__ int cell_axis(double v, double o, double inv, int n) {
    // truncation and floor differ below 0 only, NaN converts to 0 and large
    // values saturate: clamped to the grid all the same
    return min(max(__double2int_rz(__dmul_rn(__dsub_rn(v, o), inv)), 0), n - 1);
}

// L-infinity distance from p to the box (x0,y0,z0,x1,y1,z1): the largest
// per-axis gap, 0 inside.
__device__ __forceinline__ double box_dist(double px, double py, double pz, float4 lo, float4 hi) {
    double d = 0.0;
    d = fmax(d, __dsub_rn((double)lo.x, px));
    d = fmax(d, __dsub_rn(px, (double)hi.x));
    d = fmax(d, __dsub_rn((double)lo.y, py));
    d = fmax(d, __dsub_rn(py, (double)hi.y));
    d = fmax(d, __dsub_rn((double)lo.z, pz));
    d = fmax(d, __dsub_rn(pz, (double)hi.z));
    return d;
}

// The same for finite p, without fmax's NaN rules.
__device__ __forceinline__ double box_dist_finite(double px, double py, double pz, float4 lo, float4 hi) {
    const double x = dmax(__dsub_rn((double)lo.x, px), __dsub_rn(px, (double)hi.x));
    const double y = dmax(__dsub_rn((double)lo.y, py), __dsub_rn(py, (double)hi.y));
    const double z = dmax(__dsub_rn((double)lo.z, pz), __dsub_rn(pz, (double)hi.z));
    return dmax(dmax(x, y), dmax(z, 0.0));
}

__device__ __forceinline__ void load_box(const float *__restrict__ boxes, int64_t i, float4 &lo, float4 &hi) {
    const float *b = boxes + 6 * i;
    lo = make_float4(__ldg(b), __ldg(b + 1), __ldg(b + 2), __int_as_float((int)i));
    hi = make_float4(__ldg(b + 3), __ldg(b + 4), __ldg(b + 5), 0.0f);
}

__global__ void k3_bin_count(const float *__restrict__ boxes, int64_t n, Grid3 G,
                             unsigned long long *__restrict__ cnt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *b = boxes + 6 * i;
    int lo[3], hi[3];
    for (int c = 0; c < 3; c++) {
        lo[c] = cell_axis((double)b[c], G.o[c], G.inv, G.n[c]);
        hi[c] = cell_axis((double)b[3 + c], G.o[c], G.inv, G.n[c]);
    }
    for (int z = lo[2]; z <= hi[2]; z++)
        for (int y = lo[1]; y <= hi[1]; y++)
            for (int x = lo[0]; x <= hi[0]; x++)
                atomicAdd(cnt + ((int64_t)z * G.n[1] + y) * G.n[0] + x, 1ull);
}

__global__ void k3_bin_fill(const float *__restrict__ boxes, int64_t n, Grid3 G,
                            unsigned long long *__restrict__ cursor, int32_t *__restrict__ items) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *b = boxes + 6 * i;
    int lo[3], hi[3];
    for (int c = 0; c < 3; c++) {
        lo[c] = cell_axis((double)b[c], G.o[c], G.inv, G.n[c]);
        hi[c] = cell_axis((double)b[3 + c], G.o[c], G.inv, G.n[c]);
    }
    for (int z = lo[2]; z <= hi[2]; z++)
        for (int y = lo[1]; y <= hi[1]; y++)
            for (int x = lo[0]; x <= hi[0]; x++)
                items[atomicAdd(cursor + ((int64_t)z * G.n[1] + y) * G.n[0] + x, 1ull)] = (int32_t)i;
}

// Layout checks.  out->bad: min over bad boxes of (index << 2 | reason: 1
// coordinate, 2 empty or inverted), the first reason met axis by axis; extents
// as order-preserving keys, the shortest and longest edge as the bits of
// positive doubles.
__global__ void __launch_bounds__(256) k3_check_boxes(const float *__restrict__ boxes, int64_t n,
                                                      BoxCheck *__restrict__ out) {
    unsigned lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0u, 0u, 0u};
    unsigned long long bad = ~0ull, emin = ~0ull, emax = 0ull;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float *b = boxes + 6 * i;
        int why = 0;
        for (int c = 0; c < 3 && !why; c++) {
            const float x0 = __ldg(b + c), x1 = __ldg(b + 3 + c);
            if (!(isfinite(x0) && fabsf(x0) < 16777216.0f && isfinite(x1) && fabsf(x1) < 16777216.0f)) why = 1;
            else if (!(x0 < x1)) why = 2;
            if (why) break;
            lo[c] = min(lo[c], f_key(x0));
            hi[c] = max(hi[c], f_key(x1));
            const unsigned long long e = (unsigned long long)__double_as_longlong((double)x1 - (double)x0);
            emin = min(emin, e);
            emax = max(emax, e);
        }
        if (why) bad = min(bad, ((unsigned long long)i << 2) | (unsigned)why);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        for (int c = 0; c < 3; c++) {
            lo[c] = min(lo[c], __shfl_xor_sync(kFull, lo[c], o));
            hi[c] = max(hi[c], __shfl_xor_sync(kFull, hi[c], o));
        }
        bad = min(bad, __shfl_xor_sync(kFull, bad, o));
        emin = min(emin, __shfl_xor_sync(kFull, emin, o));
        emax = max(emax, __shfl_xor_sync(kFull, emax, o));
    }
    if ((threadIdx.x & 31) == 0) {
        for (int c = 0; c < 3; c++) {
            atomicMin(&out->lo[c], lo[c]);
            atomicMax(&out->hi[c], hi[c]);
        }
        atomicMin(&out->emin, emin);
        atomicMax(&out->emax, emax);
        if (bad != ~0ull) atomicMin(&out->bad, bad);
    }
}

// Boxes of one bin compared pairwise, a thread per bin entry against those of its
// bin with a higher index (interiors meet): *pair = the lowest overlapping pair
// (lower index << 32 | higher), whatever order the bins were filled in.  Two
// overlapping boxes share a bin.  A thread whose box is above the lower one of a
// pair found has nothing to add, so layouts full of overlaps end soon.
__global__ void __launch_bounds__(256) k3_overlaps(const float *__restrict__ boxes, const int64_t *__restrict__ bstart,
                                                   int64_t nbins, const int32_t *__restrict__ items,
                                                   unsigned long long *pair) {
    const int64_t total = bstart[nbins];
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < total; u += (int64_t)gridDim.x * blockDim.x) {
        int64_t a = 0, b = nbins;  // the bin of entry u: bstart[a] <= u < bstart[a + 1]
        while (b - a > 1) {
            const int64_t m = (a + b) >> 1;
            if (bstart[m] <= u) a = m;
            else b = m;
        }
        const int64_t s = bstart[a], e = bstart[a + 1];
        const int i = items[u];
        float4 lo, hi;
        load_box(boxes, i, lo, hi);
        int lowest = INT32_MAX;  // box of the bin that overlaps box i
        for (int64_t v = s; v < e; v++) {
            if (((v - s) & 31) == 0 && (unsigned long long)i > (*(volatile unsigned long long *)pair >> 32)) break;
            const int j = items[v];
            if (j <= i || j >= lowest) continue;
            float4 l2, h2;
            load_box(boxes, j, l2, h2);
            if (lo.x < h2.x && l2.x < hi.x && lo.y < h2.y && l2.y < hi.y && lo.z < h2.z && l2.z < hi.z) {
                lowest = j;
                atomicMin(pair, ((unsigned long long)(unsigned)i << 32) | (unsigned)j);
            }
        }
    }
}

// List entries (pairs of float4) ordered by (d_c in hi.w, box index in lo.w).
__device__ __forceinline__ bool entry_less(const float4 *e, int64_t a, int64_t b) {
    const float ka = e[2 * a + 1].w, kb = e[2 * b + 1].w;
    return ka < kb || (ka == kb && __float_as_int(e[2 * a].w) < __float_as_int(e[2 * b].w));
}
__device__ __forceinline__ void entry_swap(float4 *e, int64_t a, int64_t b) {
    const float4 lo = e[2 * a], hi = e[2 * a + 1];
    e[2 * a] = e[2 * b];
    e[2 * a + 1] = e[2 * b + 1];
    e[2 * b] = lo;
    e[2 * b + 1] = hi;
}
// The lists left unordered (of the cells in `todo`), a block each, in place: a
// bitonic network whose merges start mirrored, so every comparator orders
// upwards and those past the list's end are left out.  (A lane per list, by
// heapsort in global memory, was bound by its chain of loads and slower still in a
// kernel that leaves the L1 little room: grids of 4096 boxes in wide bounds 323 ->
// 57 ms, of 10^5 boxes at half a cell each 3.13 -> 1.73, 300 and 2.15 with the
// heapsort in a kernel without shared memory.)
constexpr int kSortThreads = 128;
__global__ void __launch_bounds__(kSortThreads)
    k3_sort_lists(const uint2 *__restrict__ cells, const int32_t *__restrict__ todo, float4 *lists) {
    const uint2 cr = cells[todo[blockIdx.x]];
    float4 *e = lists + 2 * (int64_t)cr.x;
    const int64_t m = cr.y;
    auto step = [&](int lg, bool mirrored) {  // comparators of sequences of 2^lg entries
        const int64_t size = 1ll << lg, half = size >> 1;
        for (int64_t t = threadIdx.x;; t += kSortThreads) {
            const int64_t at = (t >> (lg - 1)) << lg, o = t & (half - 1), p = at + (mirrored ? size - 1 - o : half + o);
            if (at >= m) break;
            if (p < m && entry_less(e, p, at + o)) entry_swap(e, at + o, p);
        }
        __syncthreads();
    };
    for (int lg = 1; (1ll << (lg - 1)) < m; lg++) {
        step(lg, true);
        for (int k = lg - 1; k > 0; k--) step(k, false);
    }
}

// Cell lists, a warp per brick of 4 x 4 x 2 cells, a lane per cell.  For a cell
// with centre c and nearest-box distance D the list holds every box within
// R = D + 2h + margin of c.  The warp gathers the boxes within a radius of the
// box spanned by its cells' centres (every lane a share of the bins, each box
// once: in the first bin, in index order, where its cell range meets the
// search range) into shared memory, then every lane takes its cell's distances
// over the same candidates.  A distance up to the radius is exact (a box that
// near was gathered), so the radius is right when it reaches the largest R; it
// starts at first_radius and grows to what the distances found ask for.
// A cell whose R reaches the 2 G.cap + 1 half sides of its search limit (it lies
// far from every box) defers: record kDefer3, its parent cell of the next level
// needed; cells outside `need` (when given) are unused.  More candidates than
// fit (coarse cells facing a dense cluster) pass through in chunks.  Lists go to the shared
// buffer at an offset from a global cursor, ordered by (distance from the
// centre, index) -- longer ones by k3_sort_lists, their cells in todo[0 .. tot[3])
// --; past `room` entries they are counted, not written (the caller
// runs the pass again with room for tot[0]).
// Why: a thread per cell walked its own bins -- 7 of 32 lanes active -- twice,
// counting and then filling, and ordered 32-byte entries in place in global
// memory: 10^5 boxes 5.3 -> 1.5 ms (bins and read-backs included; 1.3 by now).
constexpr int kBrickX = 4, kBrickY = 4, kBrickZ = 2;
constexpr int kBrickWarps = 2;     // per block
constexpr int kBrickKeys = 32;     // list entries a lane orders in shared memory
// Candidates a warp keeps.  The finest level's bricks have about 75, and its
// warps are as many as their shared memory allows: 128 there against 256, and 32
// keys against 40.  Coarser levels have few cells, far from every box, each with
// many candidates in reach: 256 (128: 1e5 boxes no faster than before; 512 and
// 768 as 256).  Grids of 1e5 boxes 1.46 -> 1.31 ms, of 3e5 (two passes) 8.9
// -> 7.3.
constexpr int kFineCand = 128, kCoarseCand = 256;

template <int kBrickCand>
struct BrickShared {
    float4 box[2 * kBrickCand];  // (x0, y0, z0, index), (x1, y1, z1, -)
    float key[kBrickKeys][32];   // per lane: rounded-down distances, in order
    uint16_t at[kBrickKeys][32]; // and their candidates
};

template <int kBrickCand>
__global__ void __launch_bounds__(kBrickWarps * 32)
    k3_cell_lists(const float *__restrict__ boxes, Grid3 G, const int64_t *__restrict__ bstart,
                  const int32_t *__restrict__ items, const uint8_t *__restrict__ need, uint8_t *__restrict__ need_up,
                  int upnx, int upny, uint2 *__restrict__ cells, float4 *__restrict__ lists, int64_t room,
                  int32_t *__restrict__ todo, unsigned long long *__restrict__ tot, double first_radius,
                  int64_t nbricks) {
    __shared__ BrickShared<kBrickCand> s_brick[kBrickWarps];
    const int lane = threadIdx.x & 31;
    const int64_t brick = (int64_t)blockIdx.x * kBrickWarps + (threadIdx.x >> 5);
    if (brick >= nbricks) return;
    BrickShared<kBrickCand> &S = s_brick[threadIdx.x >> 5];
    const int bnx = (G.n[0] + kBrickX - 1) / kBrickX, bny = (G.n[1] + kBrickY - 1) / kBrickY;
    const int c0[3] = {(int)(brick % bnx) * kBrickX, (int)(brick / bnx % bny) * kBrickY,
                       (int)(brick / ((int64_t)bnx * bny)) * kBrickZ};
    const int c1[3] = {min(c0[0] + kBrickX, G.n[0]) - 1, min(c0[1] + kBrickY, G.n[1]) - 1,
                       min(c0[2] + kBrickZ, G.n[2]) - 1};
    const int cx = c0[0] + lane % kBrickX, cy = c0[1] + lane / kBrickX % kBrickY, cz = c0[2] + lane / (kBrickX * kBrickY);
    const int64_t c = ((int64_t)cz * G.n[1] + cy) * G.n[0] + cx;
    bool mine = cx <= c1[0] && cy <= c1[1] && cz <= c1[2];
    if (mine && need && !need[c]) {
        cells[c] = make_uint2(0u, kDefer3);
        mine = false;
    }
    if (!__any_sync(kFull, mine)) return;
    auto centre = [&](int k, int i) { return __dadd_rn(G.o[k], __dmul_rn((double)i + 0.5, G.side)); };
    const double px = centre(0, cx), py = centre(1, cy), pz = centre(2, cz);
    double hlo[3], hhi[3];  // the box spanned by the brick's centres
    for (int k = 0; k < 3; k++) {
        hlo[k] = centre(k, c0[k]);
        hhi[k] = centre(k, c1[k]);
    }
    // R at which a cell defers (its search would need more than G.cap rings)
    const double rcap = G.cap < (1 << 20) ? __dmul_rn((double)(2 * G.cap + 1), G.h) : INFINITY;
    double radius = first_radius, R = 0.0;
    int nc = 0;             // candidates in shared memory
    bool resident = false;  // they are all of them
    // Calls use(n) with the boxes within `radius` of the centres' box in chunks
    // of n in S.box (one chunk, kept for the next call, when they fit).
    auto candidates = [&](auto &&use) {
        if (resident) {
            use(nc);
            return;
        }
        int s0[3], s1[3];
        for (int k = 0; k < 3; k++) {
            s0[k] = cell_axis(hlo[k] - radius - G.margin, G.o[k], G.inv, G.n[k]);
            s1[k] = cell_axis(hhi[k] + radius + G.margin, G.o[k], G.inv, G.n[k]);
        }
        const int w0 = s1[0] - s0[0] + 1, w1 = s1[1] - s0[1] + 1;
        const int64_t nbin = (int64_t)w0 * w1 * (s1[2] - s0[2] + 1);
        bool flushed = false;
        nc = 0;
        for (int64_t q0 = 0; q0 < nbin; q0 += 32) {
            const int64_t q = q0 + lane;
            int x = 0, y = 0, z = 0;
            int64_t k = 0, ke = 0;
            if (q < nbin) {
                x = s0[0] + (int)(q % w0);
                y = s0[1] + (int)(q / w0 % w1);
                z = s0[2] + (int)(q / ((int64_t)w0 * w1));
                const int64_t bin = ((int64_t)z * G.n[1] + y) * G.n[0] + x;
                k = bstart[bin];
                ke = bstart[bin + 1];
            }
            while (__any_sync(kFull, k < ke)) {
                bool keep = false;
                float4 lo, hi;
                if (k < ke) {
                    load_box(boxes, items[k++], lo, hi);
                    keep = (double)lo.x - hhi[0] <= radius && hlo[0] - (double)hi.x <= radius &&
                           (double)lo.y - hhi[1] <= radius && hlo[1] - (double)hi.y <= radius &&
                           (double)lo.z - hhi[2] <= radius && hlo[2] - (double)hi.z <= radius &&
                           max(cell_axis((double)lo.x, G.o[0], G.inv, G.n[0]), s0[0]) == x &&
                           max(cell_axis((double)lo.y, G.o[1], G.inv, G.n[1]), s0[1]) == y &&
                           max(cell_axis((double)lo.z, G.o[2], G.inv, G.n[2]), s0[2]) == z;
                }
                const unsigned m = __ballot_sync(kFull, keep);
                if (nc + __popc(m) > kBrickCand) {  // full: use these, then go on
                    __syncwarp();
                    use(nc);
                    __syncwarp();
                    flushed = true;
                    nc = 0;
                }
                if (keep) {
                    const int at = nc + __popc(m & ((1u << lane) - 1u));
                    S.box[2 * at] = lo;
                    S.box[2 * at + 1] = hi;
                }
                nc += __popc(m);
            }
        }
        __syncwarp();
        use(nc);
        __syncwarp();
        resident = !flushed;
    };
    auto dist = [&](int k) { return box_dist_finite(px, py, pz, S.box[2 * k], S.box[2 * k + 1]); };
    for (;;) {
        double D = INFINITY;
        candidates([&](int n) {
            for (int k = 0; k < n; k++) D = dmin(D, dist(k));
        });
        R = __dadd_rn(__dadd_rn(D, __dmul_rn(2.0, G.h)), G.margin);
        double want = mine ? dmin(R, rcap) : 0.0;
#pragma unroll
        for (int o = 16; o; o >>= 1) want = dmax(want, __shfl_xor_sync(kFull, want, o));
        if (want <= radius) break;
        radius = want < INFINITY ? want : 2.0 * radius;
        resident = false;
    }
    const bool defer = mine && R >= rcap;
    const bool lists_here = mine && !defer;
    if (!resident) {  // gathered again: no farther than the lists reach
        radius = lists_here ? R : 0.0;
#pragma unroll
        for (int o = 16; o; o >>= 1) radius = dmax(radius, __shfl_xor_sync(kFull, radius, o));
    }
    // the cell's list: its keys kept in order while it fits, when the candidates
    // are all here already (a gather that fits only now is not ordered)
    const bool keyed = resident;
    int m = 0;
    candidates([&](int n) {
        for (int k = 0; k < n; k++) {
            const double d = dist(k);
            if (!lists_here || d > R) continue;
            if (keyed && m < kBrickKeys) {
                const float key = __double2float_rd(d);
                const int id = __float_as_int(S.box[2 * k].w);
                int j = m;
                for (; j > 0; j--) {
                    const float kj = S.key[j - 1][lane];
                    if (kj < key || (kj == key && __float_as_int(S.box[2 * S.at[j - 1][lane]].w) < id)) break;
                    S.key[j][lane] = kj;
                    S.at[j][lane] = S.at[j - 1][lane];
                }
                S.key[j][lane] = key;
                S.at[j][lane] = (uint16_t)k;
            }
            m++;
        }
    });
    // the list's place: a warp scan and one atomic per brick
    int64_t end = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(kFull, end, o);
        if (lane >= o) end += y;
    }
    const int64_t total = __shfl_sync(kFull, end, 31);
    unsigned long long base = 0;
    if (lane == 0 && total) base = atomicAdd(tot, (unsigned long long)total);
    base = __shfl_sync(kFull, base, 0);
    const int longest = __reduce_max_sync(kFull, m);
    const unsigned deferred = __popc(__ballot_sync(kFull, defer));
    if (lane == 0) {
        if ((unsigned long long)longest > *(volatile unsigned long long *)(tot + 1))
            atomicMax(tot + 1, (unsigned long long)longest);
        if (deferred) atomicAdd(tot + 2, (unsigned long long)deferred);
    }
    const int64_t first = (int64_t)base + end - m;
    if (mine) cells[c] = defer ? make_uint2(0u, kDefer3) : make_uint2((uint32_t)first, (uint32_t)m);
    if (defer && need_up) need_up[((int64_t)(cz >> 1) * upny + (cy >> 1)) * upnx + (cx >> 1)] = 1;
    if ((int64_t)base + total > room) return;
    float4 *out = lists + 2 * first;
    const bool ordered = keyed && m <= kBrickKeys;
    if (ordered)
        for (int k = 0; k < m; k++) {
            const int at = S.at[k][lane];
            float4 hi = S.box[2 * at + 1];
            hi.w = S.key[k][lane];
            out[2 * k] = S.box[2 * at];
            out[2 * k + 1] = hi;
        }
    if (__all_sync(kFull, ordered)) return;
    // long lists: written as they come, ordered by k3_sort_lists
    const bool later = lists_here && !ordered && m > 1;
    const unsigned l = __ballot_sync(kFull, later);
    unsigned long long t0 = 0;
    if (lane == 0 && l) t0 = atomicAdd(tot + 3, (unsigned long long)__popc(l));
    t0 = __shfl_sync(kFull, t0, 0);
    if (later) todo[t0 + __popc(l & ((1u << lane) - 1u))] = (int32_t)c;
    int w = 0;
    candidates([&](int n) {
        for (int k = 0; k < n; k++) {
            const double d = dist(k);
            if (!lists_here || ordered || d > R) continue;
            float4 hi = S.box[2 * k + 1];
            hi.w = __double2float_rd(d);
            out[2 * w] = S.box[2 * k];
            out[2 * w + 1] = hi;
            w++;
        }
    });
}

// ---- query -----------------------------------------------------------------
// A point as floats and their remainders: a gap lo - p = (lo - ph) - pl carries
// two roundings of its own size and the remainder's (2^-22 of the gap + 2^-46 of
// the coordinates; lo - ph is exact when the two are close).
struct Split3 {
    float xh, yh, zh, xl, yl, zl;
    __device__ __forceinline__ float gap(const float4 &lo, const float4 &hi) const {
        const float gx = fmaxf((lo.x - xh) - xl, (xh - hi.x) + xl);
        const float gy = fmaxf((lo.y - yh) - yl, (yh - hi.y) + yl);
        const float gz = fmaxf((lo.z - zh) - zl, (zh - hi.z) + zl);
        return fmaxf(fmaxf(gx, gy), fmaxf(gz, 0.f));
    }
    // (a point far outside the bounds has gaps of its own size, so the relative
    // slack covers its remainder's rounding; one past FP32's range, or NaN, is
    // left to FP64)
    __device__ __forceinline__ bool usable() const { return fabsf(xh) + fabsf(yh) + fabsf(zh) < 1e37f; }
};
__device__ __forceinline__ Split3 split3(double px, double py, double pz) {
    Split3 s;
    s.xh = (float)px;
    s.yh = (float)py;
    s.zh = (float)pz;
    s.xl = (float)__dsub_rn(px, (double)s.xh);
    s.yl = (float)__dsub_rn(py, (double)s.yh);
    s.zl = (float)__dsub_rn(pz, (double)s.zh);
    return s;
}

// kLong: for layouts with long lists (kLongQuery, kLongWalk), see below.  kKeep:
// entries one at a time, the best one kept in registers instead of read again:
// fewer reads, more registers.
template <bool kLong, bool kKeep = false>
__device__ __forceinline__ void nearest3(const Dev3Layout &L, double px, double py, double pz, double &best,
                                         int &bid) {
    const int ix = cell_axis(px, L.g0x, L.ginv, L.nx);
    const int iy = cell_axis(py, L.g0y, L.ginv, L.ny);
    const int iz = cell_axis(pz, L.g0z, L.ginv, L.nz);
    uint2 cr = __ldg(L.cells + ((int64_t)iz * L.ny + iy) * L.nx + ix);
    const float4 *e = L.lists;
    double hq = L.hq;
    if (cr.y == kDefer3) {  // far from every box: the coarser levels
        for (int l = 0; l < L.nup && cr.y == kDefer3; l++) {
            const Level3 *V = L.up + l;
            const double gi = __ldg(&V->ginv);
            const int nx = __ldg(&V->nx), ny = __ldg(&V->ny), nz = __ldg(&V->nz);
            const int jx = cell_axis(px, L.g0x, gi, nx), jy = cell_axis(py, L.g0y, gi, ny),
                      jz = cell_axis(pz, L.g0z, gi, nz);
            const uint2 *cells = (const uint2 *)__ldg((const unsigned long long *)&V->cells);
            cr = __ldg(cells + ((int64_t)jz * ny + jy) * nx + jx);
            e = (const float4 *)__ldg((const unsigned long long *)&V->lists);
            hq = __ldg(&V->hq);
        }
        if (cr.y == kDefer3) {  // cannot happen by construction; reported, never looped on
            atomicOr(L.status, kSt3LevelChain);
            cr.y = 0;
        }
    }
    e += 2 * (size_t)cr.x;
    best = INFINITY;
    bid = 0x7FFFFFFF;
    // The nearest entry in FP32 on a split point.  An entry is skipped when its
    // distance from the cell centre (hi.w, rounded down) leaves it farther than
    // the best; later ones are too.  A winner ahead by more than the errors is
    // the FP64 winner, and only its distance is taken in FP64.  Where two are
    // closer (ties, touching boxes), a list is scanned again in FP64; with kLong,
    // where that costs as much as the first scan and clusters of aligned boxes
    // seen from afar tie often, the two are compared in FP64 on the spot, so that
    // the best is the FP64 winner of the entries so far (a block of 4096 aligned
    // boxes in wide bounds, 3e5 points: 14.6 -> 6.2 ms against 8.1 for one FP64
    // scan, 3e4 walks 140 -> 91 ms against 156).
    // Why FP32: an FP64 gap costs conversions and compares, six of each per entry
    // and about 60 instructions, on lists whose longest of a warp sets the
    // pace (3 entries scanned on average, 7.5 by the slowest lane, at 8 cells
    // per box): 1e7 walks on 10^4 boxes 4.29 -> 4.20 ms, 1e7 queries 0.312 ->
    // 0.302 ms, then 4.12 and 0.300 ms with two entries read at a time.
    const Split3 S = split3(px, py, pz);
    if (!kLong || S.usable()) {
        const float hqf = __double2float_ru(hq);
        float b1 = 3.0e38f, b2 = 3.0e38f, lim = 3.0e38f;  // b2: the second nearest; kLong: past it clearly farther
        uint32_t w = 0;
        bool exact = false;  // kLong: best and bid are the best entry's
        float4 klo, khi;     // kKeep: the best entry
        if (kKeep) klo = khi = make_float4(0.f, 0.f, 0.f, 0.f);
        auto take = [&](uint32_t k, const float4 &lo, const float4 &hi) {
            const float g = S.gap(lo, hi);
            if (kLong) {
                if (g > b2) return;
                if (g * 1.000001f + L.fslack < b1) {
                    exact = false;
                } else {
                    if (!exact) {
                        const float4 blo = kKeep ? klo : __ldg(e + 2 * w), bhi = kKeep ? khi : __ldg(e + 2 * w + 1);
                        best = box_dist_finite(px, py, pz, blo, bhi);
                        bid = __float_as_int(blo.w);
                        exact = true;
                    }
                    const double d = box_dist_finite(px, py, pz, lo, hi);
                    const int id = __float_as_int(lo.w);
                    if (d > best || (d == best && id > bid)) return;
                    best = d;
                    bid = id;
                }
                b2 = g * 1.000001f + L.fslack;
            } else {
                b2 = fminf(b2, fmaxf(g, b1));
                if (!(g < b1)) return;
            }
            b1 = g;
            w = k;
            if (kKeep) {
                klo = lo;
                khi = hi;
            }
            lim = (b1 + hqf) * 1.000002f + L.fslack;
        };
        for (uint32_t k = 0; k < cr.y; k += kKeep ? 1 : 2) {  // two entries in flight (the lists end in a spare one)
            float4 lo, hi, lo2, hi2;
            load_pair(e + 2 * k, lo, hi);
            if (!kKeep) load_pair(e + 2 * k + 2, lo2, hi2);
            if (hi.w > lim) break;
            take(k, lo, hi);
            if (kKeep) continue;
            if (k + 1 >= cr.y || hi2.w > lim) break;
            take(k + 1, lo2, hi2);
        }
        if (kLong && (exact || !cr.y)) return;
        if (kLong || (b2 > b1 * 1.000001f + L.fslack && S.usable())) {
            if (!kKeep) load_pair(e + 2 * w, klo, khi);
            best = box_dist_finite(px, py, pz, klo, khi);
            bid = __float_as_int(klo.w);
            return;
        }
    }
    for (uint32_t k = 0; k < cr.y; k++) {
        const float4 lo = __ldg(e + 2 * k), hi = __ldg(e + 2 * k + 1);
        // hi.w <= the entry's distance from the cell centre and the point is
        // within hq of that centre: this entry and every later one are
        // farther than the best so far
        if (__dsub_rn((double)hi.w, hq) > best) break;
        const double d = box_dist(px, py, pz, lo, hi);
        const int id = __float_as_int(lo.w);
        if (d < best || (d == best && id < bid)) {
            best = d;
            bid = id;
        }
    }
}

// Bound by the latency of three dependent reads (cell, list, the winner again) of
// random cells in L2.  Blocks of 64: a block ends with its slowest lane, so
// smaller ones refill the SM sooner, and 24 of them keep the 40 registers (1e7
// points: 0.299 -> 0.286 ms on 10^4 boxes, 0.468 -> 0.435 on 10^5 against blocks
// of 256; 32 registers for full occupancy 0.312 and 0.424).  Layouts with longer
// lists than those of uniform boxes (39 entries at most among 10^5) compare ties
// on the spot, at the 64 registers that takes (3e5 points on 64 aligned boxes in
// wide bounds, lists of 64: 0.283 -> 0.138 ms against 0.160 for one FP64 scan; 10^5
// boxes at half a cell each, lists of 108: 0.063 -> 0.056; uniform ones 2-10%
// slower with it).  Lists of twice the L2 and more are read from HBM, whose
// requests bound them: the best entry stays in registers, 20 blocks at 48 (1e7
// points: on 2e5 boxes, 445 MB, 0.82 -> 0.73 ms against 0.80 for one FP64 scan; on
// 3e5 1.14 -> 1.00 against 1.03; on 6e5 2.11 -> 1.85 against 1.78; on 10^5, 200 MB,
// 0.44 -> 0.50).
constexpr int kLongQuery = 48;
constexpr int64_t kFarLists = int64_t(256) << 20;
enum : int { kQueryShort = 0, kQueryLong = 1, kQueryFar = 2 };
constexpr int kQuery3Threads = 64;
template <int kKind>
__global__ void __launch_bounds__(kQuery3Threads, kKind == kQueryShort ? 24 : kKind == kQueryLong ? 16 : 20)
    k3_query(const Dev3Layout L, const double *__restrict__ pts, int64_t n, double *__restrict__ clear,
             int64_t *__restrict__ nearest) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d;
    int id;
    nearest3<kKind != kQueryShort, kKind == kQueryFar>(L, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], d, id);
    if (clear) clear[i] = d;
    if (nearest) nearest[i] = id;
}

// ---- walk ------------------------------------------------------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        if (r) {
            k.x += 0x9E3779B9u;
            k.y += 0xBB67AE85u;
        }
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    }
    return c;
}

__device__ __forceinline__ uint4 block3(const Walk3Params &P, uint64_t walk, uint32_t blk) {
    return philox4x32_10(make_uint4(blk, (uint32_t)walk, (uint32_t)(walk >> 32), P.stream),
                         make_uint2((uint32_t)P.seed, (uint32_t)(P.seed >> 32)));
}

__device__ __forceinline__ uint32_t word_of(const uint4 &b, uint32_t t) {
    const uint32_t k = t & 3;
    return k == 0 ? b.x : (k == 1 ? b.y : (k == 2 ? b.z : b.w));
}

struct Walker {
    double px, py, pz;
    double a0, sgn;
    uint4 rnd;
    uint64_t idx;  // walk index relative to P.first
    int hops, b1, axis;
    int job;       // batched runs: the walk's job
};

// Start point on the Gaussian box: faces z0, z1, y0, y1, x0, x1 by area from
// u0 (its remainder places the first coordinate), u1 the second.
template <bool kMulti>
__device__ __forceinline__ void start_walk(const Walk3Params &P, Walker &W, uint64_t j) {
    const double *G = P.G;
    double S = P.S;
    if (kMulti) {  // walk j of the batch is walk j % walks_per_job of job j / walks_per_job
        const uint64_t q = j / P.walks_per_job;
        W.job = (int)q;
        j -= q * P.walks_per_job;
        G = P.jobs[q].G;
        S = __ldg(&P.jobs[q].S);
    }
    W.idx = j;
    W.rnd = block3(P, P.first + j, 0);
    double u0 = (double)W.rnd.x * 0x1p-32;
    const double u1 = (double)W.rnd.y * 0x1p-32;
    if (P.start_strata)  // stratum (walk mod S) of the surface, by the first uniform
        u0 = __ddiv_rn(__dadd_rn((double)(uint32_t)((P.first + j) % P.start_strata), u0), (double)P.start_strata);
    const double w = __dsub_rn(G[3], G[0]), h = __dsub_rn(G[4], G[1]), d = __dsub_rn(G[5], G[2]);
    const double axy = __dmul_rn(w, h), axz = __dmul_rn(w, d), ayz = __dmul_rn(h, d);
    double s = __dmul_rn(u0, S);
    int f = 0;
    double a = axy;
    for (; f < 5; f++) {
        a = f < 2 ? axy : (f < 4 ? axz : ayz);
        if (s < a) break;
        s = __dsub_rn(s, a);
    }
    if (f == 5) a = ayz;
    double t = __ddiv_rn(s, a);
    if (t > 1.0) t = 1.0;
    const int hi = f & 1;
    if ((f >> 1) == 0) {
        W.px = __dadd_rn(G[0], __dmul_rn(t, w));
        W.py = __dadd_rn(G[1], __dmul_rn(u1, h));
        W.pz = hi ? G[5] : G[2];
        W.axis = 2;
    } else if ((f >> 1) == 1) {
        W.px = __dadd_rn(G[0], __dmul_rn(t, w));
        W.py = hi ? G[4] : G[1];
        W.pz = __dadd_rn(G[2], __dmul_rn(u1, d));
        W.axis = 1;
    } else {
        W.px = hi ? G[3] : G[0];
        W.py = __dadd_rn(G[1], __dmul_rn(t, h));
        W.pz = __dadd_rn(G[2], __dmul_rn(u1, d));
        W.axis = 0;
    }
    W.sgn = hi ? 1.0 : -1.0;
    W.hops = 0;
    W.b1 = -1;
    W.a0 = 0.0;
}

// Landing on the cube of half-side h at the centre of bin b (face k, row i,
// column j): offsets o_i = (2 i + 1 - n) / n half-sides from the face centre.
__device__ __forceinline__ void land(const Walk3Params &P, const double *s_offs, Walker &W, int b, double h) {
    // b / n^2 and r / n as multiply-highs by ceil(2^32 / d): exact for every
    // b < 6 n^2, n <= 100 (checked exhaustively); n = 1 has no division
    int k = b, r = 0, i = 0, j = 0;
    if (P.n > 1) {
        k = (int)__umulhi((unsigned)b, P.magic_nn);
        r = b - k * P.n * P.n;
        i = (int)__umulhi((unsigned)r, P.magic_n);
        j = r - i * P.n;
    }
    const double hi_ = __dmul_rn(h, s_offs[i]), hj = __dmul_rn(h, s_offs[j]);
    // faces k and k + 3 are each other's negatives; x + (-d) rounds exactly as
    // x - d, so the six faces are one addition per coordinate of selected
    // offsets: lanes land on all of them, and a branch each ran one by one
    // (10^7 walks on 10^4 boxes 3.46 -> 3.30 ms)
    const int sign = k >= 3 ? (int)0x80000000 : 0, m = k >= 3 ? k - 3 : k;
    const double dx = m == 0 ? hi_ : (m == 1 ? h : -hj);
    const double dy = m == 0 ? hj : (m == 1 ? hi_ : h);
    const double dz = m == 0 ? -h : (m == 1 ? hj : hi_);
    auto signed_by = [&](double d) { return __hiloint2double(__double2hiint(d) ^ sign, __double2loint(d)); };
    W.px = __dadd_rn(W.px, signed_by(dx));
    W.py = __dadd_rn(W.py, signed_by(dy));
    W.pz = __dadd_rn(W.pz, signed_by(dz));
}

// kMulti: a batch of targets of one layout (jobs); every lane keeps its
// sums for one job at a time and flushes them when it starts a walk of
// another job (jobs are contiguous walk ranges, so that is rare).
template <bool kMulti>
__device__ __forceinline__ void flush_job(const Walk3Params &P, int job, unsigned long long &tn, double &ts,
                                          double &ts2, unsigned long long &n_esc, unsigned long long &n_ab,
                                          unsigned long long &n_hops, unsigned long long &n_done) {
    if (!kMulti || job < 0) return;
    const int64_t t = __ldg(&P.jobs[job].target), row = (int64_t)job * P.nboxes + t;
    if (tn) {
        atomicAdd(P.hits + row, tn);
        atomicAdd(P.sum_w + row, ts);
        atomicAdd(P.sum_w2 + row, ts2);
    }
    unsigned long long *st = P.stats + 4 * (int64_t)job;
    if (n_esc) atomicAdd(st + 0, n_esc);
    if (n_ab) atomicAdd(st + 1, n_ab);
    if (n_done) {
        atomicAdd(st + 2, n_hops);
        atomicAdd(st + 3, n_done);
    }
    tn = n_esc = n_ab = n_hops = n_done = 0;
    ts = ts2 = 0.0;
}

template <bool kMulti, bool kBig, bool kLong>
__global__ void __launch_bounds__(kBig ? kW3BigThreads : kW3Threads, kBig ? 1 : kW3MinBlocks)
    k_walk3(const Walk3Params P) {
    __shared__ uint16_t s_guide[1 << kGuide3Bits];
    __shared__ double s_offs[FRW3_NSAMPLE_MAX];
    extern __shared__ uint32_t s_thr[];  // kBig: the nb thresholds
    if (kBig)
        for (int k = threadIdx.x; k < P.nb; k += blockDim.x) s_thr[k] = P.thr[k];
    for (int k = threadIdx.x; k < (1 << kGuide3Bits); k += blockDim.x) s_guide[k] = P.guide[k];
    for (int k = threadIdx.x; k < P.n; k += blockDim.x) s_offs[k] = P.offs[k];
    __syncthreads();

    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const bool trace = P.rec_end || P.rec_hops || P.rec_bin || P.rec_w;
    Walker W;
    bool active = false;
    unsigned long long tn = 0, n_esc = 0, n_ab = 0, n_hops = 0, n_done = 0;
    double ts = 0.0, ts2 = 0.0;
    uint64_t next = 0, cend = 0;
    bool exhausted = false;
    int acc_job = -1;  // batched runs: the job the lane's sums belong to

    for (;;) {
        // refill idle lanes from the warp's chunk, claiming chunks as needed
        unsigned idle = __ballot_sync(kFull, !active);
        // refill only once refill_min lanes are idle (or none is walking):
        // fewer divergent starts, at the price of lanes idling meanwhile
        if (__popc(idle) < (unsigned)P.refill_min && idle != kFull) idle = 0;
        while (idle && !exhausted) {
            if (next >= cend) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(P.counter, (unsigned long long)P.chunk);
                base = __shfl_sync(kFull, base, 0);
                if (base >= P.walks) {
                    exhausted = true;
                    break;
                }
                next = (uint64_t)base;
                cend = next + P.chunk < P.walks ? next + P.chunk : P.walks;
            }
            const uint64_t avail = cend - next;
            const unsigned rank = __popc(idle & lt);
            if (!active && rank < avail) {
                start_walk<kMulti>(P, W, next + rank);
                if (kMulti && W.job != acc_job) {
                    flush_job<kMulti>(P, acc_job, tn, ts, ts2, n_esc, n_ab, n_hops, n_done);
                    acc_job = W.job;
                }
                active = true;
            }
            next += (uint64_t)__popc(idle) < avail ? (uint64_t)__popc(idle) : avail;
            idle = __ballot_sync(kFull, !active);
        }
        if (__ballot_sync(kFull, active) == 0) break;
        if (!active) continue;

        // up to four hops per round of refills and walk ends (4.12 -> 4.10 ms per
        // 1e7 walks against two, eight: 3.78 against 3.47 by then): hop h takes
        // Philox word h + 1, every walk has done a multiple of four hops here, so
        // all of them draw the next block before their third
        int64_t end = -3;  // still walking
        for (int pass = 0; pass < 4; pass++) {
            double d = 0.0;
            if (!(W.px > P.L.b[0] && W.py > P.L.b[1] && W.pz > P.L.b[2] && W.px < P.L.b[3] && W.py < P.L.b[4] &&
                  W.pz < P.L.b[5])) {
                end = -1;
            } else {
                int id;
                nearest3<kLong>(P.L, W.px, W.py, W.pz, d, id);
                W.hops++;
                if (d <= P.shell) end = id;
                else if (W.hops >= P.hop_cap) end = -2;
            }
            if (end != -3) break;
            const uint32_t t = (uint32_t)W.hops + 1;
            if (pass == 2) W.rnd = block3(P, P.first + W.idx, t >> 2);
            const uint32_t x = word_of(W.rnd, t);
            int b = s_guide[x >> (32 - kGuide3Bits)];
            while (b + 1 < P.nb && (kBig ? s_thr[b + 1] : __ldg(P.thr + b + 1)) <= x) b++;
            land(P, s_offs, W, b, d);
            if (W.hops == 1) {
                W.b1 = b;
                W.a0 = __dmul_rn(2.0, d);
            }
        }
        if (end == -3) continue;
        // the walk ended
        double c = 0.0;
        const double S = kMulti ? __ldg(&P.jobs[W.job].S) : P.S;
        const int64_t target = kMulti ? __ldg(&P.jobs[W.job].target) : P.target;
        if (W.b1 >= 0) {
            const double wv = __ldg(P.w + 3 * W.b1 + W.axis);
            c = __ddiv_rn(__dmul_rn(__dmul_rn(P.perm, S), __dmul_rn(W.sgn, wv)), W.a0);
        }
        if (kMulti) {
            if (end == target) {
                tn++;
                ts = __dadd_rn(ts, c);
                ts2 = __dadd_rn(ts2, __dmul_rn(c, c));
            } else if (end >= 0) {
                const int64_t row = (int64_t)W.job * P.nboxes + end;
                atomicAdd(P.hits + row, 1ull);
                atomicAdd(P.sum_w + row, c);
                atomicAdd(P.sum_w2 + row, __dmul_rn(c, c));
            }
        } else if (trace) {
            if (P.rec_end) P.rec_end[W.idx] = end;
            if (P.rec_hops) P.rec_hops[W.idx] = W.hops;
            if (P.rec_bin) P.rec_bin[W.idx] = W.b1;
            if (P.rec_w) P.rec_w[W.idx] = c;
        } else if (end == P.target) {
            tn++;
            ts = __dadd_rn(ts, c);
            ts2 = __dadd_rn(ts2, __dmul_rn(c, c));
        } else if (end >= 0) {
            atomicAdd(P.hits + end, 1ull);
            atomicAdd(P.sum_w + end, c);
            atomicAdd(P.sum_w2 + end, __dmul_rn(c, c));
        }
        if (end == -1) n_esc++;
        else if (end == -2) n_ab++;
        n_hops += (unsigned long long)W.hops;
        n_done++;
        active = false;
    }

    if (kMulti) {  // every lane flushes its last job's sums
        flush_job<kMulti>(P, acc_job, tn, ts, ts2, n_esc, n_ab, n_hops, n_done);
        return;
    }
    // warp totals -> global rows
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        tn += __shfl_xor_sync(kFull, tn, o);
        ts += __shfl_xor_sync(kFull, ts, o);
        ts2 += __shfl_xor_sync(kFull, ts2, o);
        n_esc += __shfl_xor_sync(kFull, n_esc, o);
        n_ab += __shfl_xor_sync(kFull, n_ab, o);
        n_hops += __shfl_xor_sync(kFull, n_hops, o);
        n_done += __shfl_xor_sync(kFull, n_done, o);
    }
    if (lane == 0) {
        if (!trace && tn) {
            atomicAdd(P.hits + P.target, tn);
            atomicAdd(P.sum_w + P.target, ts);
            atomicAdd(P.sum_w2 + P.target, ts2);
        }
        if (P.stats) {
            atomicAdd(P.stats + 0, n_esc);
            atomicAdd(P.stats + 1, n_ab);
            atomicAdd(P.stats + 2, n_hops);
            atomicAdd(P.stats + 3, n_done);
        }
    }
}

}  // namespace

void free_grid3(Grid3Buffers *g, cudaStream_t st) {
    if (g->cells) cudaFreeAsync(g->cells, st);
    if (g->lists) cudaFreeAsync(g->lists, st);
    for (int l = 0; l < kMaxLevels3; l++) {
        if (g->up_cells[l]) cudaFreeAsync(g->up_cells[l], st);
        if (g->up_lists[l]) cudaFreeAsync(g->up_lists[l], st);
    }
    if (g->up) cudaFreeAsync(g->up, st);
    if (g->status) cudaFreeAsync(g->status, st);
    *g = Grid3Buffers();
}

void attach_grid3(Dev3Layout &L, const Grid3Buffers &g, const double bounds[6]) {
    L.cells = g.cells;
    L.lists = g.lists;
    L.g0x = g.g0[0];
    L.g0y = g.g0[1];
    L.g0z = g.g0[2];
    L.ginv = 1.0 / g.side;
    L.hq = 0.5 * g.side + 2.0 * g.margin;
    L.nx = g.nx;
    L.ny = g.ny;
    L.nz = g.nz;
    L.nup = g.nup;
    L.up = g.up;
    L.status = g.status;
    double M = 0.0;  // coordinates in use: the bounds (points outside them get the slack of points on them)
    for (int c = 0; c < 6; c++) {
        L.b[c] = bounds[c];
        M = std::max(M, std::fabs(bounds[c]));
    }
    L.fslack = (float)std::ldexp(M, -43);
    L.max_list = g.max_list;
    L.list_bytes = g.entries * 32;
}

namespace {

// One level: bins, then lists and cell records.  need == nullptr: every cell.
struct LevelOut {
    uint2 *cells = nullptr;
    float4 *lists = nullptr;
    int64_t entries = 0, deferred = 0;
    unsigned long long max_list = 0;
};

frw_status build_level(const float *d_boxes, int64_t n, const Grid3 &G, const uint8_t *need, uint8_t *need_up,
                       int upnx, int upny, cudaStream_t st, LevelOut *out) {
    const int64_t ncells = (int64_t)G.n[0] * G.n[1] * G.n[2];
    const int64_t nbricks = (int64_t)((G.n[0] + kBrickX - 1) / kBrickX) * ((G.n[1] + kBrickY - 1) / kBrickY) *
                            ((G.n[2] + kBrickZ - 1) / kBrickZ);
    int64_t *bcnt = nullptr, *bstart = nullptr, *sums = nullptr, *grand = nullptr;
    int32_t *items = nullptr, *todo = nullptr;
    unsigned long long *tot = nullptr;  // list entries, longest list, deferred cells, lists to sort
    const int64_t tiles = scan_i64_tiles(ncells + 1);
    frw_status rc = FRW_OK;
    auto ck = [&](cudaError_t e, const char *what) {
        if (e != cudaSuccess && rc == FRW_OK) rc = cuda_fail(e, what);
        return rc == FRW_OK;
    };
    do {
        const size_t cb = (size_t)(ncells + 1) * 8;
        if (!ck(cudaMallocAsync(&bcnt, cb, st), "malloc bin counts")) break;
        if (!ck(cudaMallocAsync(&bstart, cb, st), "malloc bin starts")) break;
        if (!ck(cudaMallocAsync(&sums, (size_t)tiles * 8, st), "malloc tile sums")) break;
        if (!ck(cudaMallocAsync(&grand, 8, st), "malloc totals")) break;
        if (!ck(cudaMallocAsync(&tot, 32, st), "malloc stats")) break;
        if (!ck(cudaMallocAsync(&todo, (size_t)ncells * 4, st), "malloc lists to sort")) break;
        if (!ck(cudaMallocAsync(&out->cells, (size_t)ncells * sizeof(uint2), st), "malloc cells")) break;
        if (!ck(cudaMemsetAsync(bcnt, 0, cb, st), "memset")) break;
        const unsigned nb = (unsigned)((n + 255) / 256);
        k3_bin_count<<<nb, 256, 0, st>>>(d_boxes, n, G, (unsigned long long *)bcnt);
        launch_scan_i64(bcnt, ncells + 1, bstart, sums, grand, st);
        if (!ck(cudaGetLastError(), "bin count")) break;
        int64_t nitems = 0;
        if ((rc = read_back(&nitems, grand, 8, st, "build_grid3: bin total"))) break;
        if (nitems > INT32_MAX) {
            set_error("build_grid3: more than 2^31 bin entries; use fewer cells per box");
            rc = FRW_E_ARG;
            break;
        }
        if (!ck(cudaMallocAsync(&items, (size_t)std::max<int64_t>(nitems, 1) * 4, st), "malloc bins")) break;
        // the fill uses bcnt as its cursor: start it at the bin starts
        if (!ck(cudaMemcpyAsync(bcnt, bstart, cb, cudaMemcpyDeviceToDevice, st), "cursor")) break;
        k3_bin_fill<<<nb, 256, 0, st>>>(d_boxes, n, G, (unsigned long long *)bcnt, items);
        // room for the lists of the default density (7 to 9.2 entries per cell, the
        // more the larger the layout: 3e5 boxes passed 9 and
        // took a second pass, 7.3 -> 4.4 ms);
        // longer ones take a second pass, and a buffer mostly unused a copy.  Where
        // there is no memory for that room, the first pass counts only and the
        // second has the lists' own; without memory for the copy the buffer stays.
        int64_t room = 10 * ncells + 4096;
        unsigned long long h[4] = {0, 0, 0, 0};
        // the bricks' first search: a little over two cells, or little more than the
        // cell's diagonal where the bins hold several boxes each (R is hardly more;
        // 8000 boxes in 512 cells 2.49 -> 1.44 ms)
        const double first_radius = (nitems > 4 * ncells ? 2.5 : 5.0) * G.h;
        for (int pass = 0; pass < 2; pass++) {
            // (a query may read one entry past a list)
            cudaError_t e = cudaMallocAsync(&out->lists, (size_t)(room + 1) * 32, st);
            if (e == cudaErrorMemoryAllocation && pass == 0) {
                cudaGetLastError();
                room = 0;
                e = cudaMallocAsync(&out->lists, 32, st);
            }
            if (!ck(e, "malloc lists")) break;
            if (!ck(cudaMemsetAsync(tot, 0, 32, st), "memset")) break;
            const auto kernel = need ? k3_cell_lists<kCoarseCand> : k3_cell_lists<kFineCand>;
            kernel<<<(unsigned)((nbricks + kBrickWarps - 1) / kBrickWarps), kBrickWarps * 32, 0, st>>>(
                d_boxes, G, bstart, items, need, need_up, upnx, upny, out->cells, out->lists, room, todo, tot,
                first_radius, nbricks);
            if (!ck(cudaGetLastError(), "cell lists")) break;
            if ((rc = read_back(h, tot, 32, st, "build_grid3: list total"))) break;
            if (h[0] > (unsigned long long)INT32_MAX) {
                set_error("build_grid3: more than 2^31 list entries; use fewer cells per box");
                rc = FRW_E_ARG;
                break;
            }
            if ((int64_t)h[0] <= room) break;
            cudaFreeAsync(out->lists, st);
            out->lists = nullptr;
            room = (int64_t)h[0];
        }
        if (rc) break;
        out->entries = (int64_t)h[0];
        out->max_list = h[1];
        out->deferred = (int64_t)h[2];
        if (h[3]) {
            k3_sort_lists<<<(unsigned)h[3], kSortThreads, 0, st>>>(out->cells, todo, out->lists);
            if (!ck(cudaGetLastError(), "list order")) break;
        }
        if (out->entries < room - room / 3) {
            float4 *exact = nullptr;
            if (cudaMallocAsync(&exact, (size_t)(out->entries + 1) * 32, st) == cudaSuccess) {
                const cudaError_t e =
                    cudaMemcpyAsync(exact, out->lists, (size_t)out->entries * 32, cudaMemcpyDeviceToDevice, st);
                cudaFreeAsync(out->lists, st);
                out->lists = exact;
                if (!ck(e, "lists")) break;
            } else {
                cudaGetLastError();
            }
        }
    } while (0);
    for (void *p : {(void *)bcnt, (void *)bstart, (void *)sums, (void *)grand, (void *)items, (void *)todo, (void *)tot})
        if (p) cudaFreeAsync(p, st);
    if (rc != FRW_OK) {
        if (out->cells) cudaFreeAsync(out->cells, st);
        if (out->lists) cudaFreeAsync(out->lists, st);
        *out = LevelOut();
    }
    return rc;
}

}  // namespace

frw_status check_boxes3(const float *d_boxes, int64_t n, int sms, cudaStream_t st, BoxCheck *d_out) {
    // indices, minima: all ones; maxima: zero
    FRW_CK(cudaMemsetAsync(d_out, 0xFF, sizeof(BoxCheck), st));
    FRW_CK(cudaMemsetAsync(&d_out->emax, 0, 8, st));
    FRW_CK(cudaMemsetAsync(d_out->hi, 0, sizeof(d_out->hi), st));
    const int64_t blocks = std::min<int64_t>((n + 255) / 256, (int64_t)std::max(sms, 1) * 8);
    k3_check_boxes<<<(unsigned)blocks, 256, 0, st>>>(d_boxes, n, d_out);
    FRW_CK(cudaGetLastError());
    return FRW_OK;
}

// Bins about one box across over the boxes' own extent (a box meets at most
// two per axis), however wide the bounds are.
frw_status check_disjoint3(const float *d_boxes, int64_t n, const double lo[3], const double hi[3], double emax,
                           cudaStream_t st, BoxCheck *d_out) {
    double vol = 1.0;
    for (int c = 0; c < 3; c++) vol *= std::max(hi[c] - lo[c], 1e-30);
    double cs = std::max(emax, std::cbrt(vol / (double)n));
    int64_t nc[3], total;
    for (;;) {
        total = 1;
        for (int c = 0; c < 3; c++) {
            nc[c] = std::max<int64_t>(1, (int64_t)std::floor((hi[c] - lo[c]) / cs) + 1);
            total *= nc[c];
        }
        if (total <= 8 * n + 64) break;
        cs *= 1.25;
    }
    Grid3 G{};
    for (int c = 0; c < 3; c++) {
        G.o[c] = lo[c];
        G.n[c] = (int)nc[c];
    }
    G.inv = 1.0 / cs;
    const size_t cb = (size_t)(total + 1) * 8;
    const int64_t tiles = scan_i64_tiles(total + 1), most = 27 * n;  // entries: two bins per axis, three by rounding
    char *p = nullptr;
    FRW_CK(cudaMallocAsync(&p, 2 * cb + (size_t)tiles * 8 + 8 + (size_t)most * 4, st));
    int64_t *cnt = (int64_t *)p, *start = cnt + total + 1, *sums = start + total + 1, *grand = sums + tiles;
    int32_t *items = (int32_t *)(grand + 1);
    cudaError_t e = cudaMemsetAsync(cnt, 0, cb, st);
    const unsigned nb = (unsigned)((n + 255) / 256);
    k3_bin_count<<<nb, 256, 0, st>>>(d_boxes, n, G, (unsigned long long *)cnt);
    launch_scan_i64(cnt, total + 1, start, sums, grand, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(cnt, start, cb, cudaMemcpyDeviceToDevice, st);
    k3_bin_fill<<<nb, 256, 0, st>>>(d_boxes, n, G, (unsigned long long *)cnt, items);
    k3_overlaps<<<(unsigned)((3 * n + 255) / 256), 256, 0, st>>>(d_boxes, start, total, items, &d_out->pair);
    if (e == cudaSuccess) e = cudaGetLastError();
    cudaFreeAsync(p, st);
    return e == cudaSuccess ? FRW_OK : cuda_fail(e, "3-D layout check");
}

frw_status build_grid3(const float *d_boxes, int64_t n, const double bounds[6], double cells_per_box,
                       cudaStream_t st, Grid3Buffers *out) {
    *out = Grid3Buffers();
    if (!(cells_per_box > 0) || n < 1 || n > INT32_MAX) {
        set_error("build_grid3: cells_per_box must be > 0 and 1 <= n < 2^31");
        return FRW_E_ARG;
    }
    double ext[3], vol = 1.0, M = 16.0;
    for (int c = 0; c < 3; c++) {
        ext[c] = bounds[3 + c] - bounds[c];
        vol *= ext[c];
        M = std::max(M, 4.0 * std::max(std::max(std::fabs(bounds[c]), std::fabs(bounds[3 + c])), ext[c]));
    }
    const double target = std::min((double)kMaxCells3, std::max(1.0, cells_per_box * (double)n));
    double side = std::cbrt(vol / target);
    if (!(side > 0) || !std::isfinite(side)) side = std::max(ext[0], std::max(ext[1], ext[2]));
    for (int c = 0; c < 3; c++) side = std::max(side, ext[c] / kMaxAxisCells3);
    int64_t nc[3];
    for (;;) {
        int64_t tot = 1;
        for (int c = 0; c < 3; c++) {
            nc[c] = std::max<int64_t>(1, (int64_t)std::ceil(ext[c] / side));
            tot *= nc[c];
        }
        if (tot <= kMaxCells3 && nc[0] <= kMaxAxisCells3 && nc[1] <= kMaxAxisCells3 && nc[2] <= kMaxAxisCells3)
            break;
        side *= 1.25;
    }
    Grid3 G;
    for (int c = 0; c < 3; c++) {
        G.o[c] = bounds[c];
        G.n[c] = (int)nc[c];
    }
    G.side = side;
    G.inv = 1.0 / side;
    G.h = 0.5 * side;
    G.margin = std::ldexp(M, -30);

    Events ev(2);
    if (!ev.ok(2)) return cuda_fail(cudaErrorUnknown, "event create");
    Grid3Buffers B;
    B.ncells = nc[0] * nc[1] * nc[2];
    B.nx = G.n[0];
    B.ny = G.n[1];
    B.nz = G.n[2];
    for (int c = 0; c < 3; c++) B.g0[c] = G.o[c];
    B.side = side;
    B.margin = G.margin;
    frw_status rc = FRW_OK;
    uint8_t *need = nullptr, *need_up = nullptr;
    std::vector<Level3> up;
    unsigned long long max_list = 0;
    auto ck = [&](cudaError_t e, const char *what) {
        if (e != cudaSuccess && rc == FRW_OK) rc = cuda_fail(e, what);
        return rc == FRW_OK;
    };
    do {
        if (!ck(cudaEventRecord(ev[0], st), "event")) break;
        if (!ck(cudaMallocAsync(&B.status, 4, st), "malloc status")) break;
        if (!ck(cudaMemsetAsync(B.status, 0, 4, st), "memset")) break;
        for (int l = 0; l < kMaxLevels3; l++) {
            const bool top = std::max(G.n[0], std::max(G.n[1], G.n[2])) <= 2 * kRingCap3 + 1 || l == kMaxLevels3 - 1;
            G.cap = top ? (1 << 28) : kRingCap3;
            const int upnx = (G.n[0] + 1) / 2, upny = (G.n[1] + 1) / 2, upnz = (G.n[2] + 1) / 2;
            const int64_t upcells = (int64_t)upnx * upny * upnz;
            if (!top) {
                if (!ck(cudaMallocAsync(&need_up, (size_t)upcells, st), "malloc needs")) break;
                if (!ck(cudaMemsetAsync(need_up, 0, (size_t)upcells, st), "memset")) break;
            }
            LevelOut lo;
            rc = build_level(d_boxes, n, G, need, top ? nullptr : need_up, upnx, upny, st, &lo);
            if (rc != FRW_OK) break;
            max_list = std::max(max_list, lo.max_list);
            if (l == 0) {
                B.cells = lo.cells;
                B.lists = lo.lists;
                B.entries = lo.entries;
                B.deferred = lo.deferred;
            } else {
                B.up_cells[l - 1] = lo.cells;
                B.up_lists[l - 1] = lo.lists;
                B.up_entries += lo.entries;
                Level3 V;
                V.cells = lo.cells;
                V.lists = lo.lists;
                V.ginv = G.inv;
                V.hq = G.h + 2.0 * G.margin;
                V.nx = G.n[0];
                V.ny = G.n[1];
                V.nz = G.n[2];
                V.pad = 0;
                up.push_back(V);
                B.nup = l;
            }
            if (need) cudaFreeAsync(need, st);
            need = need_up;
            need_up = nullptr;
            if (top || lo.deferred == 0) break;
            // the next level: cells twice as large, same origin
            G.n[0] = upnx;
            G.n[1] = upny;
            G.n[2] = upnz;
            G.side = std::ldexp(G.side, 1);
            G.inv = std::ldexp(G.inv, -1);
            G.h = std::ldexp(G.h, 1);
        }
        if (rc != FRW_OK) break;
        if (!up.empty()) {
            if (!ck(cudaMallocAsync(&B.up, up.size() * sizeof(Level3), st), "malloc levels")) break;
            if (!ck(cudaMemcpyAsync(B.up, up.data(), up.size() * sizeof(Level3), cudaMemcpyHostToDevice, st),
                    "levels"))
                break;
        }
        if (!ck(cudaEventRecord(ev[1], st), "event")) break;
        if ((rc = wait_event(ev[1], "build_grid3"))) break;
        B.max_list = (int32_t)max_list;
        cudaEventElapsedTime(&B.build_ms, ev[0], ev[1]);
    } while (0);
    if (need) cudaFreeAsync(need, st);
    if (need_up) cudaFreeAsync(need_up, st);
    if (rc != FRW_OK) {
        free_grid3(&B, st);
        return rc;
    }
    *out = B;
    return FRW_OK;
}

frw_status launch_query3(const Dev3Layout &L, const double *d_pts, int64_t n, double *d_clear, int64_t *d_nearest,
                         cudaStream_t st) {
    if (n <= 0) return FRW_OK;
    const auto kernel = L.list_bytes > kFarLists   ? k3_query<kQueryFar>
                        : L.max_list > kLongQuery ? k3_query<kQueryLong>
                                                  : k3_query<kQueryShort>;
    kernel<<<(unsigned)((n + kQuery3Threads - 1) / kQuery3Threads), kQuery3Threads, 0, st>>>(L, d_pts, n, d_clear, d_nearest);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FRW_OK : cuda_fail(e, "k3_query");
}

namespace {
// One block of 1024 per SM from one walk per lane on (300,000 walks: 0.306 ms
// against 0.331 in blocks of 256; 100,000: 0.246 and 0.247, and small runs
// spread over more SMs in small blocks), unless the caller asks for a number of
// blocks or the table is too long.  A warp claims 32 walks at a time in runs of
// a few walks per lane -- claims of 128 put four walks one after another on a
// lane: 30,000 walks 0.37 -> 0.22 ms -- and 128 in long ones.  Layouts with lists
// past kLongWalk take the kernels that compare ties on the spot: they spill twice
// as much (uniform boxes 8-10% slower, lists of 300 6-10%), which lists of 8065
// with ties pay back (1e5 walks on a block over a plane 3.63 -> 2.17 ms, 3.29
// for one FP64 scan).
constexpr int kLongWalk = 512;
template <bool kMulti, bool kLong>
frw_status launch_walk3_as(Walk3Params P, int sms, int bps, cudaStream_t st) {
    const size_t thr = (size_t)P.nb * sizeof(uint32_t);
    const uint64_t warps = (uint64_t)sms * (kW3BigThreads / 32);
    const bool big = bps == 0 && thr <= kW3ThrBytes && P.walks >= warps * 32;
    P.chunk = P.walks < warps * 128 ? 32 : 128;
    if (big) {
        // the largest table's size, whichever table this launch has: the attribute
        // is the kernel's, and another host thread's launch may have a longer one
        const cudaError_t e =
            cudaFuncSetAttribute(k_walk3<kMulti, true, kLong>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kW3ThrBytes);
        if (e != cudaSuccess) return cuda_fail(e, "k_walk3: shared memory");
        k_walk3<kMulti, true, kLong><<<sms, kW3BigThreads, thr, st>>>(P);
    } else {
        const uint64_t need = std::max<uint64_t>((P.walks + kW3Threads - 1) / kW3Threads, 1);
        const int full = sms * (bps > 0 ? std::min(bps, kW3MinBlocks) : kW3MinBlocks);
        k_walk3<kMulti, false, kLong><<<(unsigned)std::min<uint64_t>(need, full), kW3Threads, 0, st>>>(P);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FRW_OK : cuda_fail(e, "k_walk3");
}
}  // namespace

frw_status launch_walk3(const Walk3Params &P, int sms, int blocks_per_sm, cudaStream_t st) {
    return P.L.max_list > kLongWalk ? launch_walk3_as<false, true>(P, sms, blocks_per_sm, st)
                          : launch_walk3_as<false, false>(P, sms, blocks_per_sm, st);
}

frw_status launch_walk3_batch(const Walk3Params &P, int sms, int blocks_per_sm, cudaStream_t st) {
    return P.L.max_list > kLongWalk ? launch_walk3_as<true, true>(P, sms, blocks_per_sm, st)
                          : launch_walk3_as<true, false>(P, sms, blocks_per_sm, st);
}

}  // namespace frw
