// query.cuh -- device-side collision queries on the flat Morton quadtree.
//
// The reference answers drawBiggestSquareAtPoint (CPU/quadTree.cpp:264-312,
// Cuda/d_quadTree.cu:86-134) with 17-26 full tree traversals per point: one
// checkCollisions(box) per step of an expand/bisect loop.  Here ONE traversal
// per point computes the L-infinity clearance
//     d* = min( distance to the layer bounds, min_R gap(R, p) ),
//     gap(R, p) = max(R.x0 - p.x, p.x - R.x1, R.y0 - p.y, p.y - R.y1),
// and the short list of rects whose gap lies within 2*delta of d*; the loop is
// then replayed on scalars with the reference's own FP64 operations.  Every
// box of the loop is p +- h up to the rounding of its four coordinates
// (each within eps of the others, eps << delta), so a rect outside the list
// can only touch such a box when the box's smallest extent already exceeds d*
// + delta, and then the nearest rect (in the list) touches it too.  Hence
//     collides(box) = outside(bounds) || any(listed rect touches box)
// exactly, and the returned square is bit-identical to the reference's.
// The point query (checkCollisons(point), CPU/quadTree.cpp:240-262) falls out
// of the same traversal: rects with gap <= 0 contain p (closed intervals).
#pragma once

#include <cuda_runtime.h>

#include "frw_internal.h"

namespace frw {

constexpr int kStackMax = 64;
constexpr int kCandMax = 8;
constexpr int kReplayCap = 256;
constexpr int kNoHit = 0x7FFFFFFF;
constexpr double kMinDist = (double).095f;  // drawBiggestSquareAtPoint MIN_DIST

// The rects the replay tests for boxes within delta of the clearance: a
// point answered by a cell list keeps its cell (first >= 0), whose whole list
// is a superset of the near ties; a point answered by the tree keeps the
// near-tie list idx[0 .. n) of tree rects (first == -1).  Testing more rects
// than the ties is as exact: every listed rect is a real rect of the layout.
// More ties than kCandMax (rects whose near sides line up tie exactly) set
// first = -2: the replay's boxes near the clearance are then tested against
// the whole tree.
struct Cands {
    int idx[kCandMax];  // tree: positions of the near-tied rects among the tree's rects
    float g[kCandMax];  // their gaps, rounded down (keeping extra entries is harmless)
    int n;
    int first;
};

// Minimum and maximum without fmin / fmax's NaN rules (the operands are
// differences of finite coordinates): a comparison and a select each.
__device__ __forceinline__ double dmin(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }

// gap(R, p): <= 0 exactly when p lies in the closed rect (each difference is
// <= 0 exactly when p is on that side).
__device__ __forceinline__ double rect_gap(const float4 r, double px, double py) {
    return dmax(dmax((double)r.x - px, px - (double)r.z), dmax((double)r.y - py, py - (double)r.w));
}

// L-infinity distance from a point (in FP32) to a box, 0 inside.
__device__ __forceinline__ float lb_box_f(const float4 b, float px, float py) {
    return fmaxf(fmaxf(fmaxf(b.x - px, px - b.z), fmaxf(b.y - py, py - b.w)), 0.f);
}

// One rect of a leaf: FP32 screen, then the exact FP64 gap;
// tightens `best`, keeps the near-tie list and the containing rect.
// A full list marks the point (C.first = -2) for the whole-tree replay.
__device__ __forceinline__ void scan_rect(const float4 r, int k, const int32_t *ids, double px, double py,
                                          float pxf, float pyf, double r2, float slack, float &limf,
                                          double &best, int &hit, Cands &C) {
    const float gf = fmaxf(fmaxf(r.x - pxf, pxf - r.z), fmaxf(r.y - pyf, pyf - r.w));
    if (gf > limf) return;
    const double x0 = r.x, y0 = r.y, x1 = r.z, y1 = r.w;
    const double g = fmax(fmax(x0 - px, px - x1), fmax(y0 - py, py - y1));
    if (g <= 0.0 && px >= x0 && py >= y0 && px <= x1 && py <= y1) {
        const int id = __ldg(ids + k);
        hit = id < hit ? id : hit;
    }
    if (g < best) {
        best = g;
        limf = (float)(fmax(best, 0.0) + r2) + slack;
        int j = 0;
        for (int q = 0; q < C.n; q++)
            if ((double)C.g[q] <= best + r2) {
                C.idx[j] = C.idx[q];
                C.g[j] = C.g[q];
                j++;
            }
        C.n = j;
    }
    if (g <= best + r2) {
        if (C.n < kCandMax) {
            C.idx[C.n] = k;
            C.g[C.n] = __double2float_rd(g);
            C.n++;
        } else {
            // more ties than the list holds (rects with aligned sides tie
            // exactly: a column of equal x0 seen from its left): the replay's
            // boxes near the clearance are then tested against the whole tree
            C.first = -2;
        }
    }
}

// The tree part of clearance (no cell lists, or an overflowed cell): one
// depth-first, nearest-child-first traversal from the bounds distance in
// `best`; FP32 screens (errors below slack), the exact FP64 gap only for
// rects that can matter.
__device__ __forceinline__ uint32_t tree_clearance(const float4 *nbox, const int4 *nref, const float4 *rects,
                                                   const int32_t *ids, double px, double py, double r2, float slack,
                                                   Cands &C, int &hit, double &best) {
    uint32_t st = 0;
    const float pxf = (float)px, pyf = (float)py;
    float limf = (float)(fmax(best, 0.0) + r2) + slack;  // screen: FP32 value > limf => exact > limit
    int stk_node[kStackMax];
    float stk_lb[kStackMax];
    int sp = 0;
    int nd = 0;  // node being visited; the nearest qualifying child is visited next directly
    for (;;) {
        const float4 *bp = nbox + 4 * nd;
        float4 b[4];
        b[0] = __ldg(bp);
        b[1] = __ldg(bp + 1);
        b[2] = __ldg(bp + 2);
        b[3] = __ldg(bp + 3);
        const int4 rf = __ldg(nref + nd);
        const int ref[4] = {rf.x, rf.y, rf.z, rf.w};
        float lb[4];
#pragma unroll
        for (int c = 0; c < 4; c++) lb[c] = ref[c] == kRefEmpty ? 3.0e38f : lb_box_f(b[c], pxf, pyf);
        // leaves of this node first: they tighten `best` before descending
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (ref[c] >= kRefEmpty || lb[c] > limf) continue;
            const int f = leaf_first(ref[c]), m = leaf_count(ref[c]);
            for (int k = f; k < f + m; k++)
                scan_rect(__ldg(rects + k), k, ids, px, py, pxf, pyf, r2, slack, limf, best, hit, C);
        }
        // internal children within reach: visit the nearest next, stack the rest
        int next = -1;
        float nlb = 0.f;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (ref[c] < 0 || lb[c] > limf) continue;
            int push = ref[c];
            float plb = lb[c];
            if (next < 0 || lb[c] < nlb) {
                push = next;
                plb = nlb;
                next = ref[c];
                nlb = lb[c];
            }
            if (push >= 0) {
                if (sp < kStackMax) {
                    stk_node[sp] = push;
                    stk_lb[sp] = plb;
                    sp++;
                } else {
                    st |= kStStackOverflow;
                }
            }
        }
        if (next >= 0) {
            nd = next;
            continue;
        }
        // nothing below: resume the most recent stacked subtree still in reach
        while (sp > 0 && stk_lb[sp - 1] > limf) --sp;
        if (sp == 0) break;
        nd = stk_node[--sp];
    }
    return st;
}

// The same, out of line (a call: smaller code where the tree is rare).
static __device__ __noinline__ uint32_t tree_clearance_call(const float4 *nbox, const int4 *nref,
                                                            const float4 *rects, const int32_t *ids, double px,
                                                            double py, double r2, float slack, Cands &C, int &hit,
                                                            double &best) {
    return tree_clearance(nbox, nref, rects, ids, px, py, r2, slack, C, hit, best);
}

// The cell of a point inside the bounds (the far edge's cells by clamping).
__device__ __forceinline__ uint2 cell_xy(const DevLayout &L, double px, double py) {
    return make_uint2(min((unsigned)(int)__dmul_rn(__dsub_rn(px, L.gx0), L.ginv), (unsigned)(L.gnx - 1)),
                      min((unsigned)(int)__dmul_rn(__dsub_rn(py, L.gy0), L.ginv), (unsigned)(L.gny - 1)));
}
__device__ __forceinline__ int64_t cell_of(const DevLayout &L, double px, double py) {
    const uint2 c = cell_xy(L, px, py);
    return (int64_t)c.y * L.gnx + c.x;
}

// Two neighbouring rects of a record in one 256-bit read (32-byte aligned).
__device__ __forceinline__ void load_pair(const float4 *p, float4 &a, float4 &b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// The clearance of p from its cell's record r0 .. r3 (best: the bounds
// distance so far, hit: kNoHit).  False when the tree answers the cell.
__device__ __forceinline__ bool record_clearance(const DevLayout &L, int64_t cell, const float4 r0, const float4 r1,
                                                 const float4 r2, const float4 r3, double px, double py, Cands &C,
                                                 int &hit, double &best) {
    const int n = r3.x > kFarRect ? __float_as_int(r3.z) : 0;  // a longer list, or the tree
    if (n < 0) return false;
    const double g0 = rect_gap(r0, px, py), g1 = rect_gap(r1, px, py), g2 = rect_gap(r2, px, py),
                 g3 = rect_gap(r3, px, py);
    best = dmin(best, dmin(dmin(g0, g1), dmin(g2, g3)));
    C.first = (int)cell;
    if (!(best > 0.0)) {  // p may lie in listed rects: the lowest layer index
        const int4 id = __ldg(L.cellids + cell);
        if (g0 <= 0.0) hit = min(hit, id.x);
        if (g1 <= 0.0) hit = min(hit, id.y);
        if (g2 <= 0.0) hit = min(hit, id.z);
        if (g3 <= 0.0) hit = min(hit, id.w);
    }
    for (int k = kCellSlots - 1; k < n; k++) {  // the rest of a longer list
        const int i = __float_as_int(r3.y) + k;
        const double g = rect_gap(__ldg(L.crects + i), px, py);
        if (g <= 0.0) hit = min(hit, __ldg(L.cids + i));
        best = dmin(best, g);
    }
    return true;
}

// The clearance of p and its near-tie list.  With cell lists the list of
// p's cell holds every rect that can come within 2*delta of the clearance of
// any point of the cell (the cell's radius is bounded by the clearance of
// its centre plus half a side, with a margin far above the rounding of the
// cell index), so scanning it gives the same d*, the same containing rect and
// a superset of the same ties as the whole tree.  A cell lists about two
// rects, so its record keeps them in place: one aligned 64-byte read instead
// of a record and then its list (1e7 random points on 10^6 rects: 254 -> 150
// bytes of DRAM reads each, 0.545 -> 0.468 ms), every slot taking the exact
// FP64 gap without a loop or a test.  Otherwise (no cell lists, or an overflowed cell): one
// depth-first, nearest-child-first traversal.  Node boxes and rect gaps are
// screened in FP32 (errors below L.slack); only rects that can matter --
// inside the current tie window or containing p -- get the exact FP64 gap.
// Returns status bits.
// bd: p's distance to the bounds (negative outside).
// kInside: the caller has checked that p lies inside the bounds.
// kOutOfLineTree: the tree traversal is a call (smaller code at the caller).
template <bool kInside = false, bool kOutOfLineTree = false>
__device__ __forceinline__ uint32_t clearance(const DevLayout &L, double px, double py, Cands &C,
                                              int &hit, double &best, double bd) {
    uint32_t st = 0;
    const double r2 = 2.0 * L.delta;
    best = bd;
    hit = kNoHit;
    C.n = 0;
    C.first = -1;
    // outside the closed bounds (NaN coordinates included) no rect can contain
    // p and p+-1 already leaves the bounds: nothing to look up
    if (!kInside && !(px >= L.bx0 && py >= L.by0 && px <= L.bx1 && py <= L.by1)) {
        best = -1.0;
        return 0;
    }
    if (L.cells) {
        const int64_t cell = cell_of(L, px, py);
        float4 r0, r1, r2, r3;
        load_pair(L.cells + kCellSlots * cell, r0, r1);
        load_pair(L.cells + kCellSlots * cell + 2, r2, r3);
        if (record_clearance(L, cell, r0, r1, r2, r3, px, py, C, hit, best)) return st;
    }
    if (kOutOfLineTree)
        return tree_clearance_call(L.nbox, L.nref, L.rects, L.ids, px, py, r2, L.slack, C, hit, best);
    return tree_clearance(L.nbox, L.nref, L.rects, L.ids, px, py, r2, L.slack, C, hit, best);
}

__device__ __forceinline__ bool tree_box(const float4 *nbox, const int4 *nref, const float4 *rects,
                                         const double B[4], bool has_ign, const double ign[4], uint32_t &st);

// Tree::checkCollisions(box) restricted to the near-tie list (exact for the
// boxes of the replay, see the file comment).  Only boxes within delta of the
// clearance get here (rarely), so the listed rects are read back on demand
// rather than held in registers through the whole replay.
__device__ __forceinline__ bool touches_box(const float4 r, const double o[4]) {
    return (double)r.z >= o[0] && o[2] >= (double)r.x && (double)r.w >= o[1] && o[3] >= (double)r.y;
}
// The same test of FP32 rects without a conversion each: a float is >= an FP64
// bound exactly when it is >= the bound rounded up to FP32, and <= one when it
// is <= the bound rounded down.
struct FloatBox {
    float x0, y0, x1, y1;
    __device__ __forceinline__ bool touches(const float4 r) const {
        return r.z >= x0 && r.x <= x1 && r.w >= y0 && r.y <= y1;
    }
};
__device__ __forceinline__ FloatBox float_box(const double B[4]) {
    return FloatBox{__double2float_ru(B[0]), __double2float_ru(B[1]), __double2float_rd(B[2]), __double2float_rd(B[3])};
}
__device__ __forceinline__ bool leaves_bounds(const DevLayout &L, const double o[4]) {
    return !(o[1] >= L.by0 && o[0] >= L.bx0 && o[3] <= L.by1 && o[2] <= L.bx1);
}
// What the boxes within delta of the clearance are tested against: the rects
// of a cell (its record, or its list when it has one; slots too far touch
// nothing) ...
struct RecordTies {
    int64_t cell;
    __device__ __forceinline__ bool collides(const DevLayout &L, const double o[4], uint32_t &) const {
        if (leaves_bounds(L, o)) return true;
        const float4 *r = L.cells + kCellSlots * cell;
        int n = kCellSlots - 1;
        const float4 last = __ldg(r + kCellSlots - 1);
        if (last.x > kFarRect) {
            if (__float_as_int(last.z) >= kCellSlots) {
                r = L.crects + __float_as_int(last.y);
                n = __float_as_int(last.z);
            }
        } else if (touches_box(last, o)) {
            return true;
        }
        for (int q = 0; q < n; q++)
            if (touches_box(__ldg(r + q), o)) return true;
        return false;
    }
};
// ... the near-tie list of a point answered by the tree (or its cell) ...
struct ListedTies {
    const Cands &C;
    __device__ __forceinline__ bool collides(const DevLayout &L, const double o[4], uint32_t &st) const {
        if (C.first >= 0) return RecordTies{C.first}.collides(L, o, st);
        if (leaves_bounds(L, o)) return true;
        for (int q = 0; q < C.n; q++)
            if (touches_box(__ldg(L.rects + C.idx[q]), o)) return true;
        return false;
    }
};
// ... or, when that list overflowed, the whole tree (checkCollisions(box)).
struct TreeTies {
    __device__ __forceinline__ bool collides(const DevLayout &L, const double o[4], uint32_t &st) const {
        return leaves_bounds(L, o) || tree_box(L.nbox, L.nref, L.rects, o, false, nullptr, st);
    }
};

// Decision of one box of the replay.  Its four extents (distances from p to
// its sides) lie within eps << delta of each other, so comparing one extent
// with the clearance d* settles every box farther than delta from d*: all
// extents above d* means the nearest obstacle (bounds side or listed rect) is
// touched; all below means nothing can be.  Only boxes within delta of d*
// take the exact predicate.  The extent is compared as a coordinate: the x1
// side against p.x + (d* +- delta), both rounded once per query -- a shift of
// the window by an ulp of p.x, far inside the 32x margin of delta over eps.
struct Window {
    double hi, lo;  // x1 beyond hi: collides; below lo: free
};

__device__ __forceinline__ Window replay_window(const DevLayout &L, double px, double dstar) {
    return Window{__dadd_rn(px, __dadd_rn(dstar, L.delta)), __dadd_rn(px, __dsub_rn(dstar, L.delta))};
}

template <class Ties>
__device__ __forceinline__ bool collides_box(const DevLayout &L, const Ties &T, const double o[4],
                                             const Window &W, uint32_t &st) {
    bool c = o[2] > W.hi;
    if (!c && !(o[2] < W.lo)) c = T.collides(L, o, st);  // rare: within delta of the clearance
    return c;
}

// dist / 2 for the replay's step sizes (normal, positive, above MIN_DIST/2):
// one less in the exponent field is exactly the correctly rounded half, so
// the integer pipe does it.  A positive double's bit pattern orders like its
// value, so the MIN_DIST test is an integer compare too.
__device__ __forceinline__ double half_of(double d) {
    return __longlong_as_double(__double_as_longlong(d) - 0x0010000000000000ll);
}
__device__ __forceinline__ bool above_min(double d) {
    return __double_as_longlong(d) > __double_as_longlong(kMinDist);
}
// d when shrinking (the box collides), -d when growing: the sign bit set by
// an integer operation on the high word.
__device__ __forceinline__ double signed_step(double d, bool shrink) {
    const int hi = __double2hiint(d) ^ (shrink ? 0 : (int)0x80000000);
    return __hiloint2double(hi, __double2loint(d));
}

// The replay's decisions in closed form.  The loop's boxes are p +- E for
// E = 1 + j * dist0 * 2^-K (K = L.halvings): E grows by dist0 until the box
// collides, then moves by dist0/2, dist0/4, ... towards the clearance d* -- a
// binary search on that lattice, so step k grows exactly when bit K - k + 1 of
// q = floor((d* - 1) * 2^K / dist0) is set (the first step shrinks), and the
// last box collides exactly when bit 0 is clear.  A box that differs from d*
// by more than delta collides exactly when its E exceeds d*, so these are the
// loop's own decisions whenever (d* - 1) * 2^K / dist0 is farther than
// L.qguard (2 delta, and the rounding of the product) from every integer;
// other queries take the loop.  Only the four coordinates' additions are left
// to do one after another, because each rounds.
// Why: the walk is bound by instruction issue, and the loop's comparison and
// branch per step cost more than its additions (386 -> 305 warp instructions
// per walk on 10^6 rects together with the single test of p +- 1 and p +- 2;
// 1e8 walks 30.3 -> 26.7 ms, 1e7 capacitance walks on 10^4 rects 2.46 -> 2.18
// ms).  With 16 halvings of a step near 5100 the guard is 1e-5 of a step, so
// the loop stays for about one generic query in 10^5 and for exact ties.
struct Lattice {
    int q;    // floor((d* - 1) * 2^K / dist0)
    bool ok;  // every decision is settled by q
};

__device__ __forceinline__ Lattice replay_lattice(const DevLayout &L, double dstar) {
    const double x = __dmul_rn(__dsub_rn(dstar, 1.0), L.qscale);
    const double m = __dadd_rd(x, 0x1p52);  // floor(x) in the low word (0 <= x < 2^31)
    const double fr = __dsub_rn(x, __dsub_rn(m, 0x1p52));
    return Lattice{__double2loint(m), fr > L.qguard && fr < __dsub_rn(1.0, L.qguard)};
}

// The box of the closed form from o = p +- 1.
__device__ __forceinline__ void replay_settled(const DevLayout &L, int q, double o[4]) {
    double dist = L.dist0;
    const int K = L.halvings;
    int n = q >> K;  // growth steps before the first colliding box
    do {
        o[0] = __dsub_rn(o[0], dist);
        o[1] = __dsub_rn(o[1], dist);
        o[2] = __dadd_rn(o[2], dist);
        o[3] = __dadd_rn(o[3], dist);
    } while (--n >= 0);
    // bit 31: the step to take grows (x + (-d) rounds exactly as x - d)
    unsigned grow = (unsigned)(q & ((1 << K) - 1)) >> 1 << (32 - K);
    const int lo = __double2loint(dist);
    int hi = __double2hiint(dist);
#pragma unroll 4
    for (int k = 0; k < K; k++) {
        hi -= 0x00100000;  // dist / 2
        const double sd = __hiloint2double(hi ^ (int)(grow & 0x80000000u), lo);
        grow <<= 1;
        o[0] = __dadd_rn(o[0], sd);
        o[1] = __dadd_rn(o[1], sd);
        o[2] = __dsub_rn(o[2], sd);
        o[3] = __dsub_rn(o[3], sd);
    }
    if (!(q & 1)) {  // the last box collides: one step back
        const double d = __hiloint2double(hi, lo);
        o[0] = __dadd_rn(o[0], d);
        o[1] = __dadd_rn(o[1], d);
        o[2] = __dsub_rn(o[2], d);
        o[3] = __dsub_rn(o[3], d);
    }
}

// The box p +- h.
__device__ __forceinline__ void box_at(double px, double py, double h, double o[4]) {
    o[0] = __dsub_rn(px, h);
    o[1] = __dsub_rn(py, h);
    o[2] = __dadd_rn(px, h);
    o[3] = __dadd_rn(py, h);
}

// drawBiggestSquareAtPoint replayed on scalars: same operations, same order,
// explicit round-to-nearest intrinsics (no contraction); the halvings as
// above.  The reference first returns p +- 1 or p +- 2 when that box collides;
// d* settles both unless it lies within delta of 1 or 2 (then the other of
// the two is settled: it differs from d* by about 1), so one box is tested.
// Points with d* = 1 or 2 exactly are common -- walks start one unit from
// their target, and points truncated to int lie whole units from rects -- and
// collide: with |p| >= 4 on both axes a difference x0 - p near h <= 2 is
// exact (both are multiples of p's last place, 2^-50 or more), so the nearest
// rect's gap <= h holds without rounding, p + h >= x0, and rounding p + h
// keeps that.  Its test against the listed rects ran in nearly every round of
// a warp (1e7 capacitance walks on 10^4 rects 2.22 -> 2.06 ms without it).  Not so where
// the bounds, which a box may touch, are as near (bd: their distance).
template <class Ties>
__device__ __forceinline__ uint32_t replay_square(const DevLayout &L, const Ties &T, double px,
                                                  double py, double dstar, double bd, double o[4]) {
    uint32_t st = 0;
    const bool one = dstar < 1.5;
    const double h = one ? 1.0 : 2.0;
    box_at(px, py, h, o);
    const double e = __dsub_rn(dstar, h);
    bool c = e < -L.delta || (e <= 0.0 && bd > 3.0 && fabs(px) >= 4.0 && fabs(py) >= 4.0);
    if (!c && e <= L.delta) c = T.collides(L, o, st);  // rare: within delta of the clearance
    if (c) return st;
    box_at(px, py, one ? 2.0 : 1.0, o);
    if (one) return st;  // p +- 1 is free and p +- 2 collides
    const Lattice Q = replay_lattice(L, dstar);
    if (Q.ok) {
        replay_settled(L, Q.q, o);
        return st;
    }
    const Window W = replay_window(L, px, dstar);
    double dist = L.dist0;
    // the loop's first box is p +- 1 again, already found free: its step (grow
    // by dist, no halving before the first collision) is taken directly
    o[0] = __dsub_rn(o[0], dist);
    o[1] = __dsub_rn(o[1], dist);
    o[2] = __dadd_rn(o[2], dist);
    o[3] = __dadd_rn(o[3], dist);
    int it = 1;
    // Growth (the reference's maxReached still false): grow by dist, without
    // halving, until a box collides.
    bool isc = collides_box(L, T, o, W, st);
    while (!isc) {
        o[0] = __dsub_rn(o[0], dist);
        o[1] = __dsub_rn(o[1], dist);
        o[2] = __dadd_rn(o[2], dist);
        o[3] = __dadd_rn(o[3], dist);
        if (++it > kReplayCap) return st | kStReplayCap;
        isc = collides_box(L, T, o, W, st);
    }
    // Bisection (maxReached): the loop runs while the box collides or dist is
    // above MIN_DIST; a colliding box shrinks by dist, halved first while above
    // MIN_DIST, a free one grows by half of dist.  While dist is above MIN_DIST
    // every step halves it whatever the collision, so those steps are the
    // first L.halvings of the loop, a count fixed by the layout (dist starts at
    // dist0 every query); each is one signed step -- x + (-d) rounds exactly as
    // x - d -- so a warp whose lanes disagree on the collision issues the four
    // updates once.  After them the loop shrinks by dist while the box
    // collides.
    if (it + L.halvings > kReplayCap) return st | kStReplayCap;  // the bound falls inside the halvings
#pragma unroll 4
    for (int k = 0; k < L.halvings; k++) {
        dist = half_of(dist);
        const double sd = signed_step(dist, isc);
        o[0] = __dadd_rn(o[0], sd);
        o[1] = __dadd_rn(o[1], sd);
        o[2] = __dsub_rn(o[2], sd);
        o[3] = __dsub_rn(o[3], sd);
        isc = collides_box(L, T, o, W, st);
    }
    while (isc) {
        o[0] = __dadd_rn(o[0], dist);
        o[1] = __dadd_rn(o[1], dist);
        o[2] = __dsub_rn(o[2], dist);
        o[3] = __dsub_rn(o[3], dist);
        if (++it > kReplayCap - L.halvings) {
            st |= kStReplayCap;
            break;
        }
        isc = collides_box(L, T, o, W, st);
    }
    return st;
}

// The replay against the whole tree, out of line: one call site per query,
// taken only by points with more near ties than the list holds.
struct ReplayOut {
    double sq[4];
    uint32_t st;
};
static __device__ __noinline__ ReplayOut replay_tree_call(const DevLayout L, double px, double py,
                                                          double dstar, double bd) {
    ReplayOut r;
    r.st = replay_square(L, TreeTies{}, px, py, dstar, bd, r.sq);
    return r;
}

// drawBiggestSquareAtPoint + checkCollisons(point) for one point; points with
// more near ties than the list holds take the whole-tree replay.
template <bool kInside = false, bool kOutOfLineTree = false>
__device__ __forceinline__ uint32_t query_point(const DevLayout &L, double px, double py, double sq[4],
                                                int &hit, double bd = -1.0) {
    Cands C;
    double best;
    if (!kInside) bd = fmin(fmin(px - L.bx0, L.bx1 - px), fmin(py - L.by0, L.by1 - py));
    uint32_t st = clearance<kInside, kOutOfLineTree>(L, px, py, C, hit, best, bd);
    if (C.first == -2) {
        const ReplayOut r = replay_tree_call(L, px, py, best, bd);
        sq[0] = r.sq[0]; sq[1] = r.sq[1]; sq[2] = r.sq[2]; sq[3] = r.sq[3];
        st |= r.st;
    } else {
        st |= replay_square(L, ListedTies{C}, px, py, best, bd, sq);
    }
    return st;
}

// The same where cell records answer every point (no tree_points), without the
// tree's code.  kWalk: p is a walk's point, which ends the walk (false) when it
// is not strictly inside the bounds; only cells near them -- whose last slot
// says so, see cell_build.cu -- look at the bounds at all.  Otherwise p is any
// point.  (With the tree's code and the bounds in every hop: 2e7 walks on 10^6
// rects 5.48 ms against 5.09, 1e7 capacitance walks on 10^4 1.98 against 1.89,
// 1e7 queries 0.452 against 0.439.)
template <bool kWalk>
__device__ __forceinline__ bool query_record(const DevLayout &L, double px, double py, double sq[4], int &hit,
                                             uint32_t &st) {
    hit = kNoHit;
    double best = 1e300, bd = 1e300;
    int64_t cell = 0;
    auto bounds = [&]() { return dmin(dmin(px - L.bx0, L.bx1 - px), dmin(py - L.by0, L.by1 - py)); };
    bool in = true;
    if (!kWalk) {
        in = px >= L.bx0 && py >= L.by0 && px <= L.bx1 && py <= L.by1;
        bd = best = in ? bounds() : -1.0;
    }
    if (in) {
        cell = cell_of(L, px, py);
        float4 r0, r1, r2, r3;
        load_pair(L.cells + kCellSlots * cell, r0, r1);
        load_pair(L.cells + kCellSlots * cell + 2, r2, r3);
        const double g0 = rect_gap(r0, px, py), g1 = rect_gap(r1, px, py), g2 = rect_gap(r2, px, py),
                     g3 = rect_gap(r3, px, py);
        const double g = dmin(dmin(g0, g1), dmin(g2, g3));
        best = kWalk ? g : dmin(best, g);
        if (!(g > 0.0)) {  // p may lie in listed rects: the lowest layer index
            const int4 id = __ldg(L.cellids + cell);
            if (g0 <= 0.0) hit = min(hit, id.x);
            if (g1 <= 0.0) hit = min(hit, id.y);
            if (g2 <= 0.0) hit = min(hit, id.z);
            if (g3 <= 0.0) hit = min(hit, id.w);
        }
        if (r3.x > kFarRect) {  // near the bounds, or a longer list
            if (kWalk) {
                bd = bounds();
                if (!(bd > 0.0)) return false;
                best = dmin(best, bd);
            }
            const int n = __float_as_int(r3.z);
            for (int k = kCellSlots - 1; k < n; k++) {
                const int i = __float_as_int(r3.y) + k;
                const double gk = rect_gap(__ldg(L.crects + i), px, py);
                if (gk <= 0.0) hit = min(hit, __ldg(L.cids + i));
                best = dmin(best, gk);
            }
        }
    }
    st |= replay_square(L, RecordTies{cell}, px, py, best, bd, sq);
    return true;
}

// Tree::checkCollisions(box, ignore) for an arbitrary box (complete DFS).
__device__ __forceinline__ bool tree_box(const float4 *nbox, const int4 *nref, const float4 *rects,
                                         const double B[4], bool has_ign, const double ign[4], uint32_t &st) {
    int stk[kStackMax];
    int sp = 1;
    stk[0] = 0;
    const FloatBox fb = float_box(B);
    while (sp > 0) {
        const int nd = stk[--sp];
        const int4 rf = __ldg(nref + nd);
        const int ref[4] = {rf.x, rf.y, rf.z, rf.w};
        for (int c = 0; c < 4; c++) {
            if (ref[c] == kRefEmpty) continue;
            const float4 b = __ldg(nbox + 4 * nd + c);
            if (!fb.touches(b)) continue;
            if (ref[c] >= 0) {
                if (sp < kStackMax) stk[sp++] = ref[c];
                else st |= kStStackOverflow;
                continue;
            }
            const int f = leaf_first(ref[c]), m = leaf_count(ref[c]);
            for (int k = f; k < f + m; k++) {
                const float4 r = __ldg(rects + k);
                if (!fb.touches(r)) continue;
                const double x0 = r.x, y0 = r.y, x1 = r.z, y1 = r.w;
                if (has_ign && x0 == ign[0] && y0 == ign[1] && x1 == ign[2] && y1 == ign[3]) continue;
                return true;
            }
        }
    }
    return false;
}
__device__ __forceinline__ bool box_collides(const DevLayout &L, const double B[4], bool has_ign,
                                             const double ign[4], uint32_t &st) {
    if (!(B[1] >= L.by0 && B[0] >= L.bx0 && B[3] <= L.by1 && B[2] <= L.bx1)) return true;
    return tree_box(L.nbox, L.nref, L.rects, B, has_ign, ign, st);
}

// x / 200 for an integer-valued x in [0, 2^31), correctly rounded without the
// division sequence: q0 = x * RN(1/200), then one fused correction with the
// exact residual x - q0 * 200 (Markstein's quotient refinement).  Checked
// against IEEE division for every integer in the range.
static_assert(FRW_NSAMPLE == 200, "div200 is for the 200-bin perimeter");
__device__ __forceinline__ double div200(double x) {
    constexpr double r = 1.0 / 200.0;
    const double q0 = __dmul_rn(x, r);
    const double res = __fma_rn(-q0, 200.0, x);
    return __fma_rn(res, r, q0);
}

// RectHost::getPointFromNindex (CPU/rectHost.cpp:107-161; GPU twin
// Cuda/d_Rect.cu:34-101): its comparisons and operand order kept because they
// decide ties; the perimeter is truncated to int unless `exact`.  The
// reference branches seven ways (four sides and the corners between them),
// and the lanes of a warp take them all, so the sides are computed without
// branches -- the last two are the same operations on other operands -- and
// the point selected (319 -> 290 warp instructions per walk on 10^6 rects
// together with the cells' records).
__device__ __forceinline__ void point_from_index(const double s[4], int index, bool exact, double &ox,
                                                 double &oy) {
    const double h = __dsub_rn(s[3], s[1]);
    const double w = __dsub_rn(s[2], s[0]);
    const double w2 = __dmul_rn(2.0, w);
    const double per2 = __dadd_rn(w2, __dmul_rn(2.0, h));
    const double v = exact ? __ddiv_rn(per2, (double)FRW_NSAMPLE) : div200((double)__double2int_rz(per2));
    const double fi = (double)index;
    const double iv = __dmul_rn(fi, v), jv = __dmul_rn(__dsub_rn(fi, 1.0), v);
    const double hv = __dmul_rn(v, 0.5);
    const double wh = __dadd_rn(w, h), w2h = __dadd_rn(w2, h);
    // where the index lies, in the reference's order of tests: top, its corner
    // with the right side, right, corner, bottom, corner, left
    const int at = iv < w ? 0
                 : jv < w && iv > w ? 1
                 : iv < wh ? 2
                 : jv < wh && iv > wh ? 3
                 : iv < w2h ? 4
                 : jv < w2h && iv > w2h ? 5 : 6;
    // top: truncated to int
    const double top = (double)__double2int_rz(__dadd_rn(__dadd_rn(jv, hv), s[0]));
    // right
    const bool m2 = jv > w;
    const double right = __dadd_rn(__dsub_rn(__dadd_rn(s[1], m2 ? jv : iv), w), m2 ? hv : __dmul_rn(__dsub_rn(iv, w), 0.5));
    // bottom (from the right end, after w and h) or left (from the bottom end, after 2w and h)
    const bool bottom = at == 4, m3 = jv > (bottom ? wh : w2h);
    const double t = __dsub_rn(__dsub_rn(m3 ? jv : iv, bottom ? w : w2), h);
    const double back = __dsub_rn(bottom ? s[2] : s[3], __dadd_rn(t, m3 ? hv : __dmul_rn(t, 0.5)));
    ox = at == 0 ? top : at < 4 ? s[2] : bottom ? back : s[0];
    oy = at < 2 ? s[1] : at == 2 ? right : at < 6 ? s[3] : back;
}

// Uniform point on the Gaussian perimeter, clockwise from the top-left
// corner; side code 0 top, 1 right, 2 bottom, 3 left (outward normals
// (0,-1), (1,0), (0,1), (-1,0) in the layout's y-down axes).
__device__ __forceinline__ int perimeter_point(const double G[4], double u, double &x, double &y) {
    const double w = __dsub_rn(G[2], G[0]), h = __dsub_rn(G[3], G[1]);
    const double s = __dmul_rn(u, __dadd_rn(__dmul_rn(2.0, w), __dmul_rn(2.0, h)));
    if (s < w) {
        x = __dadd_rn(G[0], s);
        y = G[1];
        return 0;
    }
    if (s < __dadd_rn(w, h)) {
        x = G[2];
        y = __dadd_rn(G[1], __dsub_rn(s, w));
        return 1;
    }
    if (s < __dadd_rn(__dmul_rn(2.0, w), h)) {
        x = __dsub_rn(G[2], __dsub_rn(__dsub_rn(s, w), h));
        y = G[3];
        return 2;
    }
    x = G[0];
    y = __dsub_rn(G[3], __dsub_rn(__dsub_rn(s, __dmul_rn(2.0, w)), h));
    return 3;
}

}  // namespace frw
