// zncc.cuh — the bilateral-weighted ZNCC of warped_patch_zncc
// (crates/chiaro-fusion/src/depth.rs:1772-1822) split into its
// hypothesis-independent and hypothesis-dependent parts, plus the per-view
// geometry of score_one_view / map_at_depth (depth.rs:1593-1627, 1738-1759).
//
// For one node the reference samples, per tap, the reference value r_i, the
// weight w_i = spatial_i * exp(-1.2 |r_i - centre|) and the global-warp
// position g_i of every target; only the target samples depend on the depth
// hypothesis. The reference-only sums (sum w, sum w r, sum w r r) are
// sequential sums over the taps in the reference's order, so computing them
// once per node gives the same bits as recomputing them per hypothesis. The
// three target sums keep their own sequential order in zncc_score().
#pragma once

#include <type_traits>

#include "common.cuh"

namespace chiaro {

struct RefPatch {
    float count, sum_r, sum_rr;
    float ref_energy;  // sum_rr - sum_r * sum_r / count  (depth.rs:1818)
    float centre;      // centre reference sample
    int ok;            // centre and every reference tap sampled
};

// Per (node, target view) geometry, label-independent.
struct ViewGeom {
    double ox, oy, oz, dx, dy, dz;  // reference ray through the corrected reference pixel
    float gcx, gcy;                 // global warp at the node centre
    int gc_ok;                      // global.map(centre) is Some
    int ray_ok;                     // corrected reference pixel is Some
    int taps_ok;                    // global.map is Some at every tap
    int pad;
};

struct TapBox {
    float xmin, xmax, ymin, ymax;  // of g/2 over the taps
};

__device__ __forceinline__ void tap_offset(int t, int radius, int &dx, int &dy) {
    int side = 2 * radius + 1;
    dy = t / side - radius;
    dx = t % side - radius;
}

// The same with the row split by SmallDiv(2 radius + 1) (one multiply per tap).
__device__ __forceinline__ void tap_offset(int t, int radius, const SmallDiv &side, int &dx, int &dy) {
    const int row = side.quotient(t);
    dy = row - radius;
    dx = t - row * (int)side.d - radius;
}

// A tap's position in a target is kept as g/2: in f32 (g is f32 and halving is exact, a
// subnormal g apart, which no sample coordinate can tell from 0), or, for the f64 form alone,
// in f64, which spares it a conversion per coordinate. The weights (w, w r) lie apart, once per
// node.
template <typename Half>
struct Tap {
    Half half;       // g/2
    float2 weights;  // (w, w r)
};
template <typename Half>
__device__ __forceinline__ Tap<Half> load_tap(const Half *taps, const float2 *wt, int t) {
    return {taps[t], wt[t]};
}
__device__ __forceinline__ void store_tap(double2 &d, float qx, float qy) {
    d = make_double2((double)qx * 0.5, (double)qy * 0.5);
}
__device__ __forceinline__ void store_tap(float2 &d, float qx, float qy) { d = make_float2(qx * 0.5f, qy * 0.5f); }
template <typename Half>
__device__ __forceinline__ float2 tap_half(const Half *taps, int t) {
    return make_float2((float)taps[t].x, (float)taps[t].y);
}
// the coordinates of an f32 tap on the grid: g/2 + offset, rounded once
__device__ __forceinline__ f32x2 tap_on_grid(const float2 *taps, int t, f32x2 offset) {
    return add2(pack2(taps[t].x, taps[t].y), offset);
}

// Taps read where the tap lattice has them, as g: row after row of a patch, `skip` points from
// the end of one to the start of the next. NoTap stands for them as a slot's tap storage.
struct NoTap {};
struct LatticeTaps {
    const float2 *__restrict__ at;  // the first tap
    int skip;
    SmallDiv by_side;
};
__device__ __forceinline__ float2 lattice_tap(const LatticeTaps &taps, int t) {
    return taps.at[t + taps.by_side.quotient(t) * taps.skip];
}
__device__ __forceinline__ float2 tap_half(const LatticeTaps &taps, int t) {
    const float2 g = lattice_tap(taps, t);
    return make_float2(g.x * 0.5f, g.y * 0.5f);
}
__device__ __forceinline__ Tap<float2> load_tap(const LatticeTaps &taps, const float2 *wt, int t) {
    return {tap_half(taps, t), wt[t]};
}
__device__ __forceinline__ f32x2 tap_on_grid(const LatticeTaps &taps, int t, f32x2 offset) {
    const float2 g = lattice_tap(taps, t);
    return fma2(pack2(g.x, g.y), pack2(0.5f, 0.5f), offset);  // halving is exact: the same sum
}
__device__ __forceinline__ void store_tap(NoTap &, float, float) {}

// The taps of a patch in pairs, for packed arithmetic over both: half = (g/2 x, g/2 x', g/2 y,
// g/2 y') per target, weight = (w, w', w r, w' r'). A patch has an odd number of taps: the last
// pair's second half is unused.
struct PairedTaps {
    const float4 *half, *weight;
};
__device__ __forceinline__ Tap<float2> load_tap(const PairedTaps &taps, const float2 *, int t) {
    const float *g = reinterpret_cast<const float *>(taps.half + (t >> 1)) + (t & 1);
    const float *w = reinterpret_cast<const float *>(taps.weight + (t >> 1)) + (t & 1);
    return {make_float2(g[0], g[2]), make_float2(w[0], w[2])};
}

__device__ __forceinline__ float warp_min_f(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "r"(0xffffffffu));
    return r;
}
__device__ __forceinline__ float warp_max_f(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "r"(0xffffffffu));
    return r;
}
// The box of every lane's box.
__device__ __forceinline__ TapBox warp_tap_box(const TapBox &b) {
    return {warp_min_f(b.xmin), warp_max_f(b.xmax), warp_min_f(b.ymin), warp_max_f(b.ymax)};
}

// Bounding box of g/2 over one target's taps, computed by an aligned group of
// eight lanes (min and max are exact, so the reduction order does not matter).
// Every lane of the warp calls it; the groups reduce with shuffles.
template <typename TapT>
__device__ inline TapBox group8_tap_box(const TapT &gh, int taps) {
    const float2 first = tap_half(gh, 0);
    TapBox b{first.x, first.x, first.y, first.y};
    for (int t = threadIdx.x & 7; t < taps; t += 8) {
        const float2 half = tap_half(gh, t);
        b.xmin = fminf(b.xmin, half.x);
        b.xmax = fmaxf(b.xmax, half.x);
        b.ymin = fminf(b.ymin, half.y);
        b.ymax = fmaxf(b.ymax, half.y);
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {
        b.xmin = fminf(b.xmin, __shfl_xor_sync(0xffffffffu, b.xmin, off));
        b.xmax = fmaxf(b.xmax, __shfl_xor_sync(0xffffffffu, b.xmax, off));
        b.ymin = fminf(b.ymin, __shfl_xor_sync(0xffffffffu, b.ymin, off));
        b.ymax = fmaxf(b.ymax, __shfl_xor_sync(0xffffffffu, b.ymax, off));
    }
    return b;
}

// A sequential f32 sum in tap order of a[t * stride] (the reference's three
// patch sums add w, w r and (w r) r tap by tap).
__device__ inline float sequential_sum(const float *a, int stride, int taps) {
    float sum = 0.0f;
#pragma unroll 9
    for (int t = 0; t < taps; ++t) sum += a[t * stride];
    return sum;
}

__device__ inline void store_reference_sum(RefPatch &patch, int which, float sum) {
    if (which == 0)
        patch.count = sum;
    else if (which == 1)
        patch.sum_r = sum;
    else
        patch.sum_rr = sum;
}

// Tap lattice. A node of a grid with an even step sits at even pixel coordinates and its
// taps lie 2 px apart, so every tap of every node is a point (px, py) of the even lattice.
// The reference sample and each target's global warp at a tap depend on (px, py) alone,
// so they are evaluated once per lattice point and call (tap_lattice_kernel) instead of
// once per node and tap; a node reads them back with plain loads. Plane 0 holds the
// reference sample (plane_sample's value, 1 if it is Some else 0; the value is 0 when
// None, as the staging's initial value), plane 1 + v target v's Warp::map (NaN for None).
// Point (i, j) is the pixel (2 (i - margin), 2 (j - margin)). planes == nullptr: none.
struct TapLattice {
    const float2 *planes;  // [(V + 1)][rows][columns]
    int columns, rows, margin;
    __device__ __forceinline__ size_t plane_size() const { return (size_t)columns * rows; }
    // the lattice point of the even pixel (cx, cy)
    __device__ __forceinline__ size_t index(double cx, double cy) const {
        return (size_t)((int)(cy * 0.5) + margin) * columns + ((int)(cx * 0.5) + margin);
    }
};

struct LatticeParams {
    const DevView *views;
    int reference, n_targets;
    int targets[MAX_VIEWS];
    int columns, rows, margin;
    float2 *out;
};

// A thread per lattice point: the reference sample and every target's global warp there,
// with the staging's own expressions (warp_stage_patch).
__global__ void __launch_bounds__(256) tap_lattice_kernel(LatticeParams p) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long size = (long)p.columns * p.rows;
    if (i >= size) return;
    const double px = (double)(2 * ((int)(i % p.columns) - p.margin));
    const double py = (double)(2 * ((int)(i / p.columns) - p.margin));
    float value = 0.0f;
    const bool ok =
        plane_sample(p.views[p.reference].luma, (float)((px - 0.5) * 0.5), (float)((py - 0.5) * 0.5), value);
    p.out[i] = make_float2(value, ok ? 1.0f : 0.0f);
    for (int v = 0; v < p.n_targets; ++v) {
        float qx = 0.0f, qy = 0.0f;
        const bool defined = warp_map(p.views[p.targets[v]].warp, (float)px, (float)py, qx, qy);
        p.out[(size_t)(v + 1) * size + i] = defined ? make_float2(qx, qy) : make_float2(NAN, NAN);
    }
}

// The taps in target v of the patch of the node at (cx, cy), which lies on the lattice.
__device__ __forceinline__ LatticeTaps lattice_taps(const TapLattice &lattice, double cx, double cy, int v, int radius) {
    const int side = 2 * radius + 1;
    return {lattice.planes + (size_t)(v + 1) * lattice.plane_size() + lattice.index(cx, cy) -
                (ptrdiff_t)radius * (lattice.columns + 1),
            lattice.columns - side, SmallDiv(side)};
}

// Warp-cooperative staging of one node at (cx, cy) and `radius`: the
// reference patch ((w, w r) and (w r) r per tap, the three sums, the energy and the
// centre sample) and, for each target, every tap (store_tap) and the box of their g/2. Returns
// on every lane the mask of targets with a tap where the global warp is None
// (bit v); `patch` is written by lanes 0-2 and valid after the trailing
// __syncwarp(). `pre`: the node's patch from patch_sums_kernel at this radius, or
// nullptr; lane 0 copies it instead of the three lanes summing the taps.
template <typename TapT>
__device__ inline unsigned warp_stage_patch(const DevView *views, int reference, const int *targets, int V,
                                            double cx, double cy, int radius, const float *spatial, float *rr,
                                            float2 *wt, TapT *gh, TapBox *box, RefPatch &patch,
                                            const TapLattice &lattice, const RefPatch *pre) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int taps = (2 * radius + 1) * (2 * radius + 1);
    const DevView &rv = views[reference];
    float centre = 0.0f;
    bool centre_ok;
    const size_t at0 = lattice.planes ? lattice.index(cx, cy) : 0;
    if (lattice.planes) {
        const float2 c = __ldg(lattice.planes + at0);
        centre = c.x;
        centre_ok = c.y != 0.0f;
    } else {
        centre_ok = plane_sample(rv.luma, (float)((cx - 0.5) * 0.5), (float)((cy - 0.5) * 0.5), centre);
    }
    bool sampled = true;
    unsigned undefined = 0u;
    for (int t = lane; t < taps; t += 32) {
        int dx, dy;
        tap_offset(t, radius, dx, dy);
        float value = 0.0f;
        const double px = cx + (double)dx * 2.0, py = cy + (double)dy * 2.0;
        const size_t at = at0 + (ptrdiff_t)dy * lattice.columns + dx;
        if (lattice.planes) {
            const float2 r = __ldg(lattice.planes + at);
            value = r.x;
            sampled &= r.y != 0.0f;
        } else {
            sampled &= plane_sample(rv.luma, (float)((px - 0.5) * 0.5), (float)((py - 0.5) * 0.5), value);
        }
        const float weight = spatial[t] * exp_f32(-1.2f * fabsf(value - centre));
        const float2 weights = make_float2(weight, weight * value);
        wt[t] = weights;
        if (!pre) rr[t] = weights.y * value;
        for (int v = 0; v < V; ++v) {
            float2 q = make_float2(0.0f, 0.0f);
            if (lattice.planes) {
                q = __ldg(lattice.planes + (size_t)(v + 1) * lattice.plane_size() + at);
                if (q.x != q.x) undefined |= 1u << v;
            } else if (!warp_map(views[targets[v]].warp, (float)px, (float)py, q.x, q.y)) {
                undefined |= 1u << v;
            }
            store_tap(gh[v * taps + t], q.x, q.y);
        }
    }
    undefined = __reduce_or_sync(full, undefined);
    sampled = __all_sync(full, sampled);
    __syncwarp();
    for (int vb = 0; vb < V; vb += 4) {  // eight lanes per target
        const int v = vb + (lane >> 3);
        const int vs = v < V ? v : V - 1;
        TapBox b;
        if constexpr (std::is_same<TapT, NoTap>::value)
            b = group8_tap_box(lattice_taps(lattice, cx, cy, vs, radius), taps);
        else
            b = group8_tap_box(static_cast<const TapT *>(gh + vs * taps), taps);
        if ((lane & 7) == 0 && v < V) box[v] = b;
    }
    if (pre) {
        if (lane == 0) patch = *pre;
    } else {
        if (lane < 3)
            store_reference_sum(patch, lane,
                                lane == 2 ? sequential_sum(rr, 1, taps)
                                          : sequential_sum(reinterpret_cast<const float *>(wt) + lane, 2, taps));
        __syncwarp();
        if (lane == 0) {
            patch.centre = centre;
            patch.ok = centre_ok && sampled;
            patch.ref_energy = patch.sum_rr - patch.sum_r * patch.sum_r / patch.count;
        }
    }
    __syncwarp();
    return undefined;
}

// The reference patch of every node of a step-spaced grid at `radius`, a thread per node:
// what warp_stage_patch computes for it (the taps' weights w = spatial * exp(-1.2 |r -
// centre|), the sums of w, w r and (w r) r in tap order, the energy, the centre sample and
// whether the centre and every tap were sampled), with the same expressions in the same
// order, so the same bits. The direct pass and the decisions read it instead of summing 81
// or more taps in three lanes of a warp.
// Grid row y of the launch works on grid y (the fine and the coarse one).
struct PatchGrid {
    int columns, rows, step, radius;
    const float *spatial;
    TapLattice lattice;  // of this grid, or planes == nullptr
    RefPatch *out;
    const int *nodes;  // the nodes whose patches are wanted, `listed` of them, or nullptr: all
    int listed;
};
struct PatchParams {
    const DevView *views;
    int reference;
    PatchGrid grids[2];
};

__global__ void __launch_bounds__(256) patch_sums_kernel(PatchParams params) {
    const PatchGrid &p = params.grids[blockIdx.y];
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (p.nodes ? (long)p.listed : (long)p.columns * p.rows)) return;
    if (p.nodes) i = __ldg(p.nodes + i);
    const double cx = (double)((int)(i % p.columns) * p.step), cy = (double)((int)(i / p.columns) * p.step);
    const DevView &rv = params.views[params.reference];
    const TapLattice &lattice = p.lattice;
    float centre = 0.0f;
    bool centre_ok;
    const size_t at0 = lattice.planes ? lattice.index(cx, cy) : 0;
    if (lattice.planes) {
        const float2 c = __ldg(lattice.planes + at0);
        centre = c.x;
        centre_ok = c.y != 0.0f;
    } else {
        centre_ok = plane_sample(rv.luma, (float)((cx - 0.5) * 0.5), (float)((cy - 0.5) * 0.5), centre);
    }
    bool sampled = true;
    float count = 0.0f, sum_r = 0.0f, sum_rr = 0.0f;
    // eight taps' loads and weights at a time, ahead of their sums: on a small grid the kernel is
    // one thread's latency (27 us at 660 nodes with every tap's loads after the last one's sums)
    constexpr int AHEAD = 8;
    const int side = 2 * p.radius + 1, taps = side * side;
    const SmallDiv by_side(side);
    for (int t0 = 0; t0 < taps; t0 += AHEAD) {
        float value[AHEAD], weight[AHEAD];
        if (lattice.planes) {
            float2 r[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                int dx, dy;
                tap_offset(min(t0 + i, taps - 1), p.radius, by_side, dx, dy);
                r[i] = __ldg(lattice.planes + at0 + (ptrdiff_t)dy * lattice.columns + dx);
            }
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                value[i] = r[i].x;
                sampled &= r[i].y != 0.0f;
            }
        } else {
            for (int i = 0; i < AHEAD; ++i) {
                int dx, dy;
                tap_offset(min(t0 + i, taps - 1), p.radius, by_side, dx, dy);
                const double px = cx + (double)dx * 2.0, py = cy + (double)dy * 2.0;
                value[i] = 0.0f;
                sampled &= plane_sample(rv.luma, (float)((px - 0.5) * 0.5), (float)((py - 0.5) * 0.5), value[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            weight[i] = __ldg(p.spatial + min(t0 + i, taps - 1)) * exp_f32(-1.2f * fabsf(value[i] - centre));
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (t0 + i < taps) {
                const float weighted = weight[i] * value[i];
                count += weight[i];
                sum_r += weighted;
                sum_rr += weighted * value[i];
            }
    }
    RefPatch r;
    r.count = count;
    r.sum_r = sum_r;
    r.sum_rr = sum_rr;
    r.ref_energy = sum_rr - sum_r * sum_r / count;
    r.centre = centre;
    r.ok = centre_ok && sampled;
    p.out[i] = r;
}

// Label-independent geometry of map_at_depth for one (node, target); one thread.
__device__ void view_geometry(const DevCamera &rc, const DevCamera &tc, const WarpRef &warp, double cx, double cy,
                              ViewGeom &g) {
    float gx = 0.0f, gy = 0.0f;
    g.gc_ok = warp_map(warp, (float)cx, (float)cy, gx, gy) ? 1 : 0;
    g.gcx = gx;
    g.gcy = gy;
    g.ray_ok = 0;
    g.taps_ok = 1;
    if (!g.gc_ok) return;
    D3 o1, d1;
    pixel_to_ray(tc, (double)gx, (double)gy, o1, d1);
    double crx, cry;
    if (!project(rc, along(o1, d1, INFINITY_DEPTH), crx, cry)) return;
    D3 o2, d2;
    pixel_to_ray(rc, crx, cry, o2, d2);
    g.ox = o2.x;
    g.oy = o2.y;
    g.oz = o2.z;
    g.dx = d2.x;
    g.dy = d2.y;
    g.dz = d2.z;
    g.ray_ok = 1;
}

// Compact per (node, target) geometry kept in HBM between kernels. pixel_to_ray
// returns the camera centre as the origin for both pose kinds (geometry.rs:152-164),
// so only the direction varies per node. gcx is NaN when global.map(centre) is
// None, dx is NaN when the corrected reference pixel is None.
struct GeomRec {
    double dx, dy, dz;
    float gcx, gcy;
};

__device__ __forceinline__ D3 camera_origin(const DevCamera &c) {
    return c.pose_kind == 0 ? D3{c.center[0], c.center[1], c.center[2]}
                            : D3{c.virtual_center[0], c.virtual_center[1], c.virtual_center[2]};
}

__device__ __forceinline__ void geom_from_rec(const GeomRec &rec, const D3 &origin, ViewGeom &g) {
    g.gcx = rec.gcx;
    g.gcy = rec.gcy;
    g.gc_ok = !(rec.gcx != rec.gcx);
    g.ray_ok = g.gc_ok && !(rec.dx != rec.dx);
    g.ox = origin.x;
    g.oy = origin.y;
    g.oz = origin.z;
    g.dx = rec.dx;
    g.dy = rec.dy;
    g.dz = rec.dz;
    g.taps_ok = 1;
}

// One thread per (node, target) of a step-spaced grid: the label-independent
// part of map_at_depth (depth.rs:1745-1756). Grid row y of the launch works on grid y (the
// coarse and the fine one).
struct GeometryGrid {
    int columns, rows, step;
    GeomRec *out;  // [node][target]
};
struct GeometryParams {
    const DevView *views;
    int reference, n_targets;
    int targets[MAX_VIEWS];
    GeometryGrid grids[2];
};

__global__ void __launch_bounds__(128) view_geometry_kernel(GeometryParams params) {
    const GeometryParams &p = params;
    const GeometryGrid &grid = p.grids[blockIdx.y];
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    long total = (long)grid.columns * grid.rows * p.n_targets;
    if (i >= total) return;
    int v = (int)(i % p.n_targets);
    int node = (int)(i / p.n_targets);
    double cx = (double)((node % grid.columns) * grid.step), cy = (double)((node / grid.columns) * grid.step);
    const DevView &tv = p.views[p.targets[v]];
    ViewGeom g;
    view_geometry(p.views[p.reference].cam, tv.cam, tv.warp, cx, cy, g);
    GeomRec rec;
    rec.gcx = g.gc_ok ? g.gcx : NAN;
    rec.gcy = g.gc_ok ? g.gcy : NAN;
    rec.dx = g.ray_ok ? g.dx : NAN;
    rec.dy = g.ray_ok ? g.dy : NAN;
    rec.dz = g.ray_ok ? g.dz : NAN;
    grid.out[i] = rec;
}

// map_at_depth's last step and score_one_view's displacement check: the
// image displacement of a finite depth relative to the global centre. Returns
// false for None (depth.rs:1604-1614).
__device__ __forceinline__ bool depth_delta(const DevCamera &tc, const ViewGeom &g, double depth, double &ddx,
                                            double &ddy) {
    if (!g.gc_ok || !g.ray_ok) return false;
    double qx, qy;
    if (!project(tc, along({g.ox, g.oy, g.oz}, {g.dx, g.dy, g.dz}, depth), qx, qy)) return false;
    if (!(isfinite(qx) && isfinite(qy))) return false;
    ddx = qx - (double)g.gcx;
    ddy = qy - (double)g.gcy;
    return !(fabs(ddx) > 128.0 || fabs(ddy) > 128.0);
}

// Hypothesis-dependent part of warped_patch_zncc: sample the target at every
// tap shifted by (ddx, ddy) and finish the correlation. False for None.
template <typename TapT>
__device__ __forceinline__ bool zncc_score(const PlaneRef &target, TapT gh, const float2 *wt,
                                           const RefPatch &patch, int taps, double ddx, double ddy, float &score) {
    float st = 0.0f, stt = 0.0f, srt = 0.0f;
    for (int t = 0; t < taps; ++t) {
        const auto tap = load_tap(gh, wt, t);
        double qx = (double)tap.half.x * 2.0 + ddx;
        double qy = (double)tap.half.y * 2.0 + ddy;
        float tv;
        if (!plane_sample(target, (float)((qx - 0.5) * 0.5), (float)((qy - 0.5) * 0.5), tv)) return false;
        const float2 weights = tap.weights;
        float wv = weights.x * tv;
        st += wv;
        stt += wv * tv;
        srt += weights.y * tv;
    }
    float covariance = srt - patch.sum_r * st / patch.count;
    float target_energy = stt - st * st / patch.count;
    float denominator = sqrtf(fmaxf(patch.ref_energy, 0.0f) * fmaxf(target_energy, 0.0f));
    if (!(denominator > 1.0e-6f)) return false;
    score = clampf_r(covariance / denominator, -1.0f, 1.0f);
    return true;
}

// ---- fast paths --------------------------------------------------------------------
// The reference computes each target sample coordinate as
//   x = (f32)(((f64)g + d - 0.5) * 0.5)
// with two f64 roundings. Multiplying by 0.5 is exact and commutes with
// rounding, so the same bits come from x = (f32)((g/2 + d/2) - 0.25), where g/2
// is stored per tap and d/2 is computed once per hypothesis. The
// coordinate is monotone in g, so the bounding box of the taps' g decides for
// every tap at once whether all samples fall strictly inside [0, w-1) x [0, h-1);
// inside, the reference's bounds checks and edge clamps cannot trigger and the
// bilinear fetch reads the four neighbours from a quad plane with one 16-byte
// load (zncc_inside). Where grid_offset (common.cuh) also finds an f32 offset for both
// coordinates, one f32 addition gives each (zncc_grid): most inside hypotheses of a plane
// larger than a thumbnail.

// Quad plane: the quad of (x, y) is (L[y][x], L[y][x1], L[y1][x], L[y1][x1]) with
// x1 = min(x + 1, w - 1) and y1 = min(y + 1, h - 1), pair-interleaved: the quads of rows
// 2k and 2k + 1 alternate, so (x, y) sits at (y >> 1) * stride + 2 x + (y & 1) with
// stride = 2 * roundup(w, 4), and each 128-byte line holds a 4 x 2 block of quads. The
// taps of neighbouring labels spread along the epipolar line in any direction; against
// row-major quads (8 x 1 per line) a 4 x 2 block keeps more of a quarter-warp's gathers
// in one line.
__host__ __device__ inline int quad_stride(int width) { return 2 * ((width + 3) / 4 * 4); }
inline size_t quad_count(int width, int height) { return (size_t)quad_stride(width) * ((height + 1) / 2); }

__device__ __forceinline__ size_t quad_index(int x, int y, int stride) {
    return (size_t)(y >> 1) * stride + 2 * x + (y & 1);
}

// Every target's planes for the correlations, in one launch: the quad plane, and where the cost
// volume runs in node tiles the plane or its transpose (region_transposed) with rows padded to a
// multiple of 4 floats, for load_region. A CTA of 32 x 8 threads makes a 32 x 32 tile of target
// blockIdx.y from one read of it and its right and lower neighbours. HBM-bound: 4 B read, 16 B
// written per pixel, and 4 B more for the tiles.
struct PlanesParams {
    const DevView *views;
    int quads;  // whether the quad planes are written
    int targets[MAX_VIEWS];
};

__global__ void __launch_bounds__(256) sample_planes_kernel(PlanesParams p) {
    __shared__ float tile[33][34];
    const DevView &v = p.views[p.targets[blockIdx.y]];
    const int width = v.luma.width, height = v.luma.height;
    const int tiles_x = (width + 31) / 32, ty = blockIdx.x / tiles_x;
    const int x0 = (blockIdx.x - ty * tiles_x) * 32, y0 = ty * 32, lane = threadIdx.x;
    if (y0 >= height) return;
    for (int i = threadIdx.y * 32 + lane; i < 33 * 33; i += 256) {
        const int r = i / 33, c = i - r * 33;
        tile[r][c] = __ldg(v.luma.data + (size_t)min(y0 + r, height - 1) * width + min(x0 + c, width - 1));
    }
    __syncthreads();
    float4 *quads = const_cast<float4 *>(v.quads);
    float *const region = const_cast<float *>(v.region_plane.data);
    const bool rows = region && !v.region_transposed, columns = region && v.region_transposed;
    for (int r = threadIdx.y; r < 32; r += 8) {
        int x = x0 + lane, y = y0 + r;
        if (x < width && y < height) {
            if (rows) region[(size_t)y * v.region_plane.pitch + x] = tile[r][lane];
            if (p.quads)
                quads[quad_index(x, y, v.quad_stride)] =
                    make_float4(tile[r][lane], tile[r][lane + 1], tile[r + 1][lane], tile[r + 1][lane + 1]);
        }
        x = x0 + r;
        y = y0 + lane;
        if (columns && x < width && y < height) region[(size_t)x * v.region_plane.pitch + y] = tile[lane][r];
    }
}

// The smallest and largest sample coordinates of a box displaced by (hdx, hdy) = (ddx/2, ddy/2).
struct TapRange {
    float x0, x1, y0, y1;
};
__device__ __forceinline__ TapRange tap_range(const TapBox &box, double hdx, double hdy) {
    return {(float)(((double)box.xmin + hdx) - 0.25), (float)(((double)box.xmax + hdx) - 0.25),
            (float)(((double)box.ymin + hdy) - 0.25), (float)(((double)box.ymax + hdy) - 0.25)};
}

// True when every tap samples strictly inside the plane.
__device__ __forceinline__ bool taps_inside(const TapRange &r, int width, int height) {
    // width, height < 2^22 (checked on the host), so inside also means < 2^22
    return r.x0 >= 0.0f && r.y0 >= 0.0f && r.x1 < (float)(width - 1) && r.y1 < (float)(height - 1);
}

// True when every tap samples strictly inside the plane and one f32 addition of `offset`
// per coordinate gives the reference's sample positions; `r` is then their range.
__device__ __forceinline__ bool taps_on_grid(const TapBox &box, double ddx, double ddy, int width, int height,
                                             float2 &offset, TapRange &r) {
    if (max(width, height) > GRID_OFFSET_MAX_SIDE || !grid_offset(ddx * 0.5, box.xmin, offset.x) ||
        !grid_offset(ddy * 0.5, box.ymin, offset.y))
        return false;
    r = {box.xmin + offset.x, box.xmax + offset.x, box.ymin + offset.y, box.ymax + offset.y};
    return taps_inside(r, width, height);
}
__device__ __forceinline__ bool taps_on_grid(const TapBox &box, double ddx, double ddy, int width, int height,
                                             float2 &offset) {
    TapRange r;
    return taps_on_grid(box, ddx, ddy, width, height, offset, r);
}

// The correlation from the three target sums (depth.rs:1815-1822).
__device__ __forceinline__ float zncc_finish(const RefPatch &patch, float st, float stt, float srt, bool &ok) {
    float covariance = srt - patch.sum_r * st / patch.count;
    float target_energy = stt - st * st / patch.count;
    float denominator = sqrtf(fmaxf(patch.ref_energy, 0.0f) * fmaxf(target_energy, 0.0f));
    ok = denominator > 1.0e-6f;
    return clampf_r(covariance / denominator, -1.0f, 1.0f);
}

// The bilinear sample of a quad and its three sums.
__device__ __forceinline__ void add_sample(const float4 &q, float2 frac, float2 rest, float2 weights, float &st,
                                           float &stt, float &srt) {
    float top = q.x * rest.x + q.y * frac.x;
    float bottom = q.z * rest.x + q.w * frac.x;
    float tv = top * rest.y + bottom * frac.y;
    float wv = weights.x * tv;
    st += wv;
    stt += wv * tv;
    srt += weights.y * tv;
}

// warped_patch_zncc's hypothesis-dependent part for taps known to be inside
// (see taps_inside).
template <int UNROLL, typename TapT>
__device__ __forceinline__ float zncc_inside(const float4 *__restrict__ quads, int stride, TapT gh,
                                             const float2 *wt, const RefPatch &patch, int taps,
                                             double hdx, double hdy, bool &ok) {
    float st = 0.0f, stt = 0.0f, srt = 0.0f;
#pragma unroll UNROLL
    for (int t = 0; t < taps; ++t) {
        const auto tap = load_tap(gh, wt, t);
        const float x = (float)(((double)tap.half.x + hdx) - 0.25);
        const float y = (float)(((double)tap.half.y + hdy) - 0.25);
        const float mx = __fadd_rd(x, 8388608.0f), my = __fadd_rd(y, 8388608.0f);  // 2^23 + floor
        const float tx = x - (mx - 8388608.0f), ty = y - (my - 8388608.0f);
        const float4 q = __ldg(quads + quad_index((int)(f2u(mx) - 0x4B000000u), (int)(f2u(my) - 0x4B000000u), stride));
        add_sample(q, make_float2(tx, ty), make_float2(1.0f - tx, 1.0f - ty), tap.weights, st, stt, srt);
    }
    return zncc_finish(patch, st, stt, srt, ok);
}

// The same for taps that taps_on_grid accepted, with its offset. The two coordinates go
// through packed f32 instructions (two IEEE operations in one): the addition; the floor, by
// adding 2^23 rounded down (0 <= x < 2^22, so the sum is 2^23 + floor(x) and its low bits
// hold the index); the fraction x - floor(x), exact; and 1 - fraction, rounded once.
template <int UNROLL, typename TapT>
__device__ __forceinline__ float zncc_grid(const float4 *__restrict__ quads, int stride, TapT gh,
                                           const float2 *wt, const RefPatch &patch, int taps, float2 offset,
                                           bool &ok) {
    const f32x2 e = pack2(offset.x, offset.y), magic = pack2(8388608.0f, 8388608.0f);
    const f32x2 minus_magic = pack2(-8388608.0f, -8388608.0f), one = pack2(1.0f, 1.0f);
    const f32x2 minus_one = pack2(-1.0f, -1.0f);
    float st = 0.0f, stt = 0.0f, srt = 0.0f;
#pragma unroll UNROLL
    for (int t = 0; t < taps; ++t) {
        const float2 weights = wt[t];
        const f32x2 x = tap_on_grid(gh, t, e);
        const f32x2 m = add2_down(x, magic);
        const f32x2 frac = fma2(add2(m, minus_magic), minus_one, x), rest = fma2(frac, minus_one, one);
        const float2 mf = unpack2(m);
        const int ix = (int)(f2u(mf.x) - 0x4B000000u), iy = (int)(f2u(mf.y) - 0x4B000000u);
        const float4 q = __ldg(quads + quad_index(ix, iy, stride));
        add_sample(q, unpack2(frac), unpack2(rest), weights, st, stt, srt);
    }
    return zncc_finish(patch, st, stt, srt, ok);
}

// ---- samples from a region in shared memory ------------------------------------------
// A warp's lanes score neighbouring hypotheses: at one tap their samples lie along the
// target's epipolar line, half a pixel to two pixels apart. Gathered from the quad plane
// those are 20 to 30 128-byte lines an instruction, about 13 passes through the L1's data
// stage. From a copy of the rectangle around the whole segment, one float per pixel, the
// four neighbours of a sample are four 4-byte shared loads. Lanes in different banks cost
// nothing there, so the copy is laid out with its rows along the coordinate axis nearer to
// the epipolar line (the target's plane or its transpose) and a row pitch of a multiple of
// 32 words: the bank is the position along that axis, in which neighbouring lanes differ.
constexpr int REGION_PITCH = 96;  // a reach of 64 samples (128 px displacement), a patch, a tile and alignment

struct Region {
    int column, row, columns, rows;  // of the stored plane (transposed or not); column a multiple of 4
};

// The rectangle of a range of sample floors (lowest x, lowest y, -highest x, -highest y) and
// each one's right and lower neighbour. False where it does not fit the buffer.
__device__ __forceinline__ bool region_of(const int *range, bool transposed, int rows, Region &r) {
    const int c0 = range[transposed ? 1 : 0], r0 = range[transposed ? 0 : 1];
    const int c1 = -range[transposed ? 3 : 2], r1 = -range[transposed ? 2 : 3];
    r.column = c0 & ~3;
    r.row = r0;
    r.columns = c1 + 2 - r.column;
    r.rows = r1 + 2 - r0;
    return r.columns <= REGION_PITCH && r.rows <= rows;
}

// Copies a region with 16-byte asynchronous copies (copy_async_wait, then a barrier). The
// plane's rows are padded to its pitch, a multiple of 4, so a copy that starts inside a row
// ends inside it.
__device__ __forceinline__ void load_region(const Region &r, const PaddedPlane &plane, float *region, int tid,
                                            int threads) {
    const int quarters = (r.columns + 3) >> 2;
    const int groups = threads / 24;  // of 24 threads: a whole row
    const int row0 = tid / 24, at = tid - row0 * 24;
    if (row0 >= groups || at >= quarters) return;
    const float *src = plane.data + (size_t)(r.row + row0) * plane.pitch + r.column + 4 * at;
    uint32_t dst = (uint32_t)__cvta_generic_to_shared(region + row0 * REGION_PITCH + 4 * at);
    for (int row = row0; row < r.rows; row += groups) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        src += (size_t)groups * plane.pitch;
        dst += groups * REGION_PITCH * sizeof(float);
    }
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The samples' coordinates of a pair of taps: one f32 addition each for a hypothesis on the grid
// (place: its offset), else in f64 (place: half its displacement; see taps_inside).
__device__ __forceinline__ void pair_position(const float4 &half, const float2 &place, f32x2 &x, f32x2 &y) {
    x = add2(pack2(half.x, half.y), pack2(place.x, place.x));
    y = add2(pack2(half.z, half.w), pack2(place.y, place.y));
}
__device__ __forceinline__ void pair_position(const float4 &half, const double2 &place, f32x2 &x, f32x2 &y) {
    x = pack2((float)(((double)half.x + place.x) - 0.25), (float)(((double)half.y + place.x) - 0.25));
    y = pack2((float)(((double)half.z + place.y) - 0.25), (float)(((double)half.w + place.y) - 0.25));
}

// zncc_grid or zncc_inside with the samples in a region, two taps at a time in packed arithmetic
// (the sums take them in tap order). opaque_one: see add2_products.
template <bool TRANSPOSED, typename Place>
__device__ __forceinline__ float zncc_region(const float *region, const Region &r, const PairedTaps &tap,
                                             const RefPatch &patch, int taps, const Place &place, float opaque_one,
                                             bool &ok) {
    constexpr unsigned SX = TRANSPOSED ? REGION_PITCH : 1, SY = TRANSPOSED ? 1 : REGION_PITCH;
    const f32x2 magic = pack2(8388608.0f, 8388608.0f), minus_magic = pack2(-8388608.0f, -8388608.0f);
    const f32x2 one = pack2(opaque_one, opaque_one), minus_one = pack2(-1.0f, -1.0f);
    // word of a sample: bits(2^23 + x) SX + bits(2^23 + y) SY + c
    const unsigned c = 0u - (0x4B000000u + (unsigned)(TRANSPOSED ? r.row : r.column)) * SX -
                       (0x4B000000u + (unsigned)(TRANSPOSED ? r.column : r.row)) * SY;
    float st = 0.0f, stt = 0.0f, srt = 0.0f;
#pragma unroll 1
    for (int t = 0; t < taps >> 1; ++t) {
        const float4 b = tap.weight[t];
        f32x2 x, y;
        pair_position(tap.half[t], place, x, y);
        const f32x2 mx = add2_down(x, magic), my = add2_down(y, magic);
        const f32x2 fx = fma2(add2(mx, minus_magic), minus_one, x), fy = fma2(add2(my, minus_magic), minus_one, y);
        const f32x2 ux = fma2(fx, minus_one, one), uy = fma2(fy, minus_one, one);
        const float2 mxf = unpack2(mx), myf = unpack2(my);
        const float *q0 = region + (f2u(mxf.x) * SX + f2u(myf.x) * SY + c);
        const float *q1 = region + (f2u(mxf.y) * SX + f2u(myf.y) * SY + c);
        const f32x2 top = add2_products(mul2(pack2(q0[0], q1[0]), ux), mul2(pack2(q0[SX], q1[SX]), fx), one);
        const f32x2 bottom =
            add2_products(mul2(pack2(q0[SY], q1[SY]), ux), mul2(pack2(q0[SX + SY], q1[SX + SY]), fx), one);
        const f32x2 tv = add2_products(mul2(top, uy), mul2(bottom, fy), one);
        const f32x2 wv = mul2(pack2(b.x, b.y), tv);
        const float2 s0 = unpack2(wv), s1 = unpack2(mul2(wv, tv)), s2 = unpack2(mul2(pack2(b.z, b.w), tv));
        st += s0.x;
        stt += s1.x;
        srt += s2.x;
        st += s0.y;
        stt += s1.y;
        srt += s2.y;
    }
    {
        const float4 b = tap.weight[taps >> 1];
        f32x2 last_x, last_y;
        pair_position(tap.half[taps >> 1], place, last_x, last_y);
        const float x = unpack2(last_x).x, y = unpack2(last_y).x;
        const float mx = __fadd_rd(x, 8388608.0f), my = __fadd_rd(y, 8388608.0f);
        const float tx = x - (mx - 8388608.0f), ty = y - (my - 8388608.0f);
        const float *q = region + (f2u(mx) * SX + f2u(my) * SY + c);
        add_sample(make_float4(q[0], q[SX], q[SY], q[SX + SY]), make_float2(tx, ty), make_float2(1.0f - tx, 1.0f - ty),
                   make_float2(b.x, b.z), st, stt, srt);
    }
    return zncc_finish(patch, st, stt, srt, ok);
}

// Either path in f64, bit-identical to warped_patch_zncc: the fast loop when the box is inside,
// exact per-tap checks otherwise. The plane is copied: read through the view in device memory, its
// base and sides were loaded again at every tap of the exact path (direct pass of 400x300 with four
// targets at radius 8, most of whose wide patches cross an edge: depth kernel 0.54 -> 0.49 ms, retry
// 0.49 -> 0.46 ms).
template <int UNROLL, typename TapT>
__device__ __forceinline__ bool zncc_any(const DevView &target, TapT gh, const TapBox &box,
                                              const float2 *wt, const RefPatch &patch, int taps, double ddx,
                                              double ddy, float &score) {
    const PlaneRef plane = target.luma;
    const double hdx = ddx * 0.5, hdy = ddy * 0.5;
    if (taps_inside(tap_range(box, hdx, hdy), plane.width, plane.height)) {
        bool ok;
        score = zncc_inside<UNROLL>(target.quads, target.quad_stride, gh, wt, patch, taps, hdx, hdy, ok);
        return ok;
    }
    return zncc_score(plane, gh, wt, patch, taps, ddx, ddy, score);
}

// aggregate (depth.rs:1761-1770) over up to MAX_VIEWS scores (NaN = None).
__device__ __forceinline__ bool aggregate_scores(float *s, int n, int minimum_support, int best_view_count,
                                                 float &out) {
    // compact the Some values
    int m = 0;
    for (int i = 0; i < n; ++i)
        if (!(s[i] != s[i])) s[m++] = s[i];
    if (m < minimum_support) return false;
    // stable insertion sort, descending by total order
    for (int i = 1; i < m; ++i) {
        float v = s[i];
        int j = i - 1;
        while (j >= 0 && total_key(s[j]) < total_key(v)) {
            s[j + 1] = s[j];
            --j;
        }
        s[j + 1] = v;
    }
    int k = best_view_count < m ? best_view_count : m;
    if (k < minimum_support) return false;
    float sum = -0.0f;
    for (int i = 0; i < k; ++i) sum += s[i];
    out = sum / (float)k;
    return true;
}

}  // namespace chiaro
