// cv_feat.cuh -- the control variate's input features of a first-hop point
// (shared by the feature, exact-mean and training kernels).
#pragma once

#include "cv.cuh"
#include "query.cuh"

namespace frw {
namespace cv {

// ---------------------------------------------------------------- features
// d / a0 as d * (1 / a0) (one division per point), clamped to [-16, 16]
static __device__ __forceinline__ float feat(double d, double inv) {
    double v = __dmul_rn(d, inv);
    v = fmin(fmax(v, -16.0), 16.0);
    return (float)v;
}

// (dx, dy) from p to the nearest point of each edge of rect r: top, right,
// bottom, left (layout axes, y down).
static __device__ __forceinline__ void edge_feats(double px, double py, double x0, double y0, double x1, double y1,
                                           double a0, float *f) {
    const double cx = fmin(fmax(px, x0), x1), cy = fmin(fmax(py, y0), y1);
    const double dcx = __dsub_rn(cx, px), dcy = __dsub_rn(cy, py);
    const double inv = __ddiv_rn(1.0, a0);
    f[0] = feat(dcx, inv);
    f[1] = feat(__dsub_rn(y0, py), inv);
    f[2] = feat(__dsub_rn(x1, px), inv);
    f[3] = feat(dcy, inv);
    f[4] = f[0];
    f[5] = feat(__dsub_rn(y1, py), inv);
    f[6] = feat(__dsub_rn(x0, px), inv);
    f[7] = f[3];
}

// Nearest rect other than layer index `exclude` (smallest L-inf gap, then
// smallest layer index) from the tree; Morton position or -1.
static __device__ int nearest_other_tree(const DevLayout &L, double px, double py, int exclude) {
    const float pxf = (float)px, pyf = (float)py, slack = L.slack;
    double best = 1e300;
    int best_id = 0x7FFFFFFF, best_k = -1;
    float limf = 3.0e38f;
    int stk[kStackMax];
    int sp = 0, nd = 0;
    for (;;) {
        const float4 *bp = L.nbox + 4 * nd;
        const int4 rf = __ldg(L.nref + nd);
        const int ref[4] = {rf.x, rf.y, rf.z, rf.w};
        float lb[4];
#pragma unroll
        for (int c = 0; c < 4; c++) lb[c] = ref[c] == kRefEmpty ? 3.0e38f : lb_box_f(__ldg(bp + c), pxf, pyf);
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (ref[c] >= kRefEmpty || lb[c] > limf) continue;
            const int f0 = leaf_first(ref[c]), m = leaf_count(ref[c]);
            for (int k = f0; k < f0 + m; k++) {
                const float4 r = __ldg(L.rects + k);
                const float gf = fmaxf(fmaxf(r.x - pxf, pxf - r.z), fmaxf(r.y - pyf, pyf - r.w));
                if (gf > limf) continue;
                const int id = __ldg(L.ids + k);
                if (id == exclude) continue;
                const double g = fmax(fmax((double)r.x - px, px - (double)r.z), fmax((double)r.y - py, py - (double)r.w));
                if (g < best || (g == best && id < best_id)) {
                    best = g;
                    best_id = id;
                    best_k = k;
                    limf = (float)best + slack;
                }
            }
        }
        int next = -1;
        float nlb = 0.f;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (ref[c] < 0 || lb[c] > limf) continue;
            int push = ref[c];
            if (next < 0 || lb[c] < nlb) {
                push = next;
                next = ref[c];
                nlb = lb[c];
            }
            if (push >= 0 && sp < kStackMax) stk[sp++] = push;
        }
        if (next >= 0) {
            nd = next;
            continue;
        }
        if (sp == 0) break;
        nd = stk[--sp];
    }
    return best_k;
}

// The same from the list of the target's neighbours (cv.cuh) at the largest reach
// that has a whole one, where it settles the answer: it holds every other rect
// within reach of the target rect, so a nearest one within reach less p's own
// distance to the target (two deltas cover the rounding) is the nearest, ties
// included.
static __device__ __forceinline__ bool nearest_neighbour(const DevLayout &L, double4 target, const Neighbours *nb,
                                                         double px, double py, float4 &o) {
    int l = 0;
    while (l < kNeighbourLevels && __ldg(nb->n + l) > kNeighbours) l++;
    if (l == kNeighbourLevels) return false;
    const int n = __ldg(nb->n + l);
    if (n <= 0) return false;
    const double away = dmax(dmax(dmax(target.x - px, px - target.z), dmax(target.y - py, py - target.w)), 0.0);
    const double within = __ldg(nb->reach + l) - away - 2.0 * L.delta;
    if (!(within > 0.0)) return false;
    const float pxf = (float)px, pyf = (float)py;
    float limf = 3.0e38f;
    double best = 1e300;
    int best_id = 0x7FFFFFFF;
#pragma unroll 4
    for (int k = 0; k < n; k++) {
        const float4 q = __ldg(nb->rects[l] + k);
        if (fmaxf(fmaxf(q.x - pxf, pxf - q.z), fmaxf(q.y - pyf, pyf - q.w)) > limf) continue;
        const double g = rect_gap(q, px, py);
        const int id = __ldg(nb->ids[l] + k);
        if (g < best || (g == best && id < best_id)) {
            best = g;
            best_id = id;
            o = q;
            limf = (float)best + L.slack;
        }
    }
    return best <= within;
}

// The same from the target's neighbours (nb, nullable), else from p's cell list when it
// settles the answer: every rect within crad of p is listed, so a listed
// nearest other within crad is the nearest (ties included); otherwise the
// tree.  Writes the rect, false when none.
static __device__ __forceinline__ bool nearest_other(const DevLayout &L, double4 target, const Neighbours *nb, double px,
                                                     double py, int exclude, float4 &o) {
    if (nb && nearest_neighbour(L, target, nb, px, py, o)) return true;
    if (L.cells && px >= L.bx0 && py >= L.by0 && px <= L.bx1 && py <= L.by1) {
        const int64_t cell = cell_of(L, px, py);
        const float4 *r = L.cells + kCellSlots * cell;
        const int32_t *ids = reinterpret_cast<const int32_t *>(L.cellids + cell);
        const float4 last = __ldg(r + kCellSlots - 1);
        int n = kCellSlots;
        if (last.x > kFarRect) {  // a longer list, a short one near the bounds, or (n < 0) the tree
            n = __float_as_int(last.z);
            if (n >= kCellSlots) {
                r = L.crects + __float_as_int(last.y);
                ids = L.cids + __float_as_int(last.y);
            }
        }
        if (n >= 0) {
            double best = 1e300;
            int best_id = 0x7FFFFFFF;
            float4 bo = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int k = 0; k < n; k++) {
                const int id = __ldg(ids + k);
                if (id == exclude || id < 0) continue;
                const float4 q = __ldg(r + k);
                const double g =
                    fmax(fmax((double)q.x - px, px - (double)q.z), fmax((double)q.y - py, py - (double)q.w));
                if (g < best || (g == best && id < best_id)) {
                    best = g;
                    best_id = id;
                    bo = q;
                }
            }
            if (best <= (double)__ldg(L.crad + cell)) {
                o = bo;
                return true;
            }
        }
    }
    const int k = nearest_other_tree(L, px, py, exclude);
    if (k < 0) return false;
    o = __ldg(L.rects + k);
    return true;
}

}  // namespace cv
}  // namespace frw
