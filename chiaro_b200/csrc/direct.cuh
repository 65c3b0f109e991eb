// direct.cuh — measure_direct_depths (crates/chiaro-fusion/src/depth.rs:715-876)
// with nearest_coarse_depth (1062-1076), direct_depth_candidates (1078-1107),
// select_direct_depth (1109-1165) and best_depth_candidate (1167-1185).
//
// A warp per fine-grid node, as many nodes per CTA as keep the most warps
// resident. The thirteen seeded candidates are computed one per lane and
// deduplicated by a uniform scan; the baseline and candidate scores are
// independent (candidate, view) ZNCC items, listed fast-path first and spread
// over the warp; the selection replaces the reference's sort by warp
// reductions. Nodes that need the wide-radius retry go to a list that a second
// kernel processes with its larger patch.
#pragma once

#include "cost.cuh"
#include "select.cuh"

namespace chiaro {

constexpr int MAX_DIRECT_CANDIDATES = 32;
constexpr int WIDE_CANDIDATES = 7;  // of the wide retry: the best one and three on each side
constexpr int KEY_NONE = -2147483647 - 1;  // below every total_key of a non-NaN float

// select_direct_depth (depth.rs:1109-1165) and best_depth_candidate
// (depth.rs:1167-1185) over (depth, score) pairs, score NaN = None, computed by
// a whole warp: lane c < n holds candidate c's objective. The reference sorts
// the objectives stably in descending total order; its head is the first
// maximum, and its first entry more than one index away from the head has the
// largest objective among those entries, so two warp max-reductions replace
// the sort. best_depth_candidate keeps the last maximum (`best_last`, -1 for
// None). Every lane returns the same result.
__device__ inline bool warp_select_direct(const double *depths, const float *scores, int n, bool has_baseline,
                                          float baseline, bool seeded, double far_depth, double near_depth,
                                          float minimum_score, float minimum_margin, float minimum_improvement,
                                          double &out_depth, float &out_confidence, float &out_improvement,
                                          int &best_last) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double far_inverse = 1.0 / far_depth;
    double inverse_range = 1.0 / near_depth - far_inverse;
    bool valid = false;
    float objective = 0.0f;
    if (lane < n) {
        float s = scores[lane];
        valid = !(s != s);
        if (valid) {
            double near_fraction = clampd_r((1.0 / depths[lane] - far_inverse) / inverse_range, 0.0, 1.0);
            objective = s - NEAR_DEPTH_PRIOR * (float)near_fraction;
        }
    }
    best_last = -1;
    if (!__ballot_sync(full, valid)) return false;
    const int key = valid ? total_key(objective) : KEY_NONE;
    const int top = __reduce_max_sync(full, key);
    const unsigned at_top = __ballot_sync(full, valid && key == top);
    const int best = __ffs(at_top) - 1;
    best_last = 31 - __clz(at_top);
    const float best_objective = __shfl_sync(full, objective, best);
    const bool away = valid && (lane - best > 1 || lane - best < -1);
    const unsigned away_mask = __ballot_sync(full, away);
    float competing = best_objective;
    if (away_mask) {
        const int away_top = __reduce_max_sync(full, away ? key : KEY_NONE);
        const int c = __ffs(__ballot_sync(full, away && key == away_top)) - 1;
        competing = __shfl_sync(full, objective, c);
    }
    float score = scores[best];
    float margin = fmaxf(best_objective - competing, 0.0f);
    float improvement = has_baseline ? score - baseline : 0.0f;
    float score_floor = fmaxf(minimum_score - 0.03f, MINIMUM_REGULARIZED_SCORE);
    float required_margin = seeded ? minimum_margin * 0.6f : minimum_margin;
    bool improves_global = !has_baseline || improvement >= minimum_improvement * 0.5f;
    bool supported = score >= score_floor && improves_global &&
                     (margin >= required_margin || improvement >= minimum_improvement);
    if (!supported) return false;
    float score_confidence = clampf_r((score - score_floor) / fmaxf(1.0f - score_floor, 1.0e-3f), 0.0f, 1.0f);
    float margin_confidence = clampf_r(margin / fmaxf(required_margin, 1.0e-3f), 0.0f, 1.0f);
    out_depth = depths[best];
    out_confidence = clampf_r(0.30f + 0.45f * score_confidence + 0.25f * margin_confidence, 0.0f, 1.0f);
    out_improvement = improvement;
    return true;
}

// ---- warp-per-node direct pass ---------------------------------------------------
struct DirectParams {
    const DevView *views;
    int reference, n_targets;
    int targets[MAX_VIEWS];
    int columns, rows, step;                           // fine grid
    Field coarse;                                      // SGM seed field
    int coarse_columns, coarse_rows, coarse_step;
    double inverse_step, near_depth, far_depth;
    const double *unseeded;                            // 32 candidates, far to near
    const GeomRec *geometry;                           // [node][target] of the fine grid
    TapLattice lattice;                                // of the fine grid, or planes == nullptr
    const RefPatch *patches;                           // [node] reference patch at `radius`, or nullptr
    int radius, wide_radius;
    const float *spatial, *spatial_wide;
    float minimum_score, minimum_margin, minimum_improvement;
    int minimum_support, best_view_count;
    int nodes_per_cta;
    Field out;
    float *guidance;
    uint8_t *tested;
    int *wide_count;                                   // wide-retry list length; entries taken beyond the first ones
    int4 *wide_list;                                   // (node, first, last, seeded)
};

// Per-warp shared memory of the direct pass for V targets, T taps and up to `most` candidates;
// TapT is the tap storage (load_tap; NoTap: they are read from the lattice).
template <typename TapT>
struct DirectSlot {
    float2 *wt;            // [T] (w, w r)
    ViewGeom *geom;        // [V]
    TapT *gh;              // [V][T] taps
    TapBox *box;           // [V]
    double *cand;          // [32]
    float *rr;             // [T] (w r) r: until the patch is summed, where the following then lie
    float2 *items;         // [V][most + 1] a listed item on the grid: its f32 offset, until it is scored;
                           // then the score in x (NaN = None)
    float *agg;            // [most + 1]: [0] baseline, [1 + c] candidates
    unsigned short *list;  // [V][most + 1] scored items: fast path from the front, exact path from the back
};

template <typename TapT>
__host__ __device__ inline size_t tap_bytes(int V, int taps) {
    return std::is_empty<TapT>::value ? 0 : align16((size_t)V * taps * sizeof(TapT));
}

template <typename TapT>
__host__ __device__ inline size_t direct_slot_bytes(int V, int taps, int most) {
    const size_t items = align16((size_t)(most + 1) * V * sizeof(float2)) + align16((most + 1) * sizeof(float)) +
                         align16((size_t)(most + 1) * V * sizeof(unsigned short));
    const size_t sums = align16(taps * sizeof(float));
    return align16(taps * sizeof(float2)) + align16(V * sizeof(ViewGeom)) +
           tap_bytes<TapT>(V, taps) + align16(V * sizeof(TapBox)) +
           align16(MAX_DIRECT_CANDIDATES * sizeof(double)) + (items > sums ? items : sums);
}

// The bound on targets and radius that the direct pass accepts, for its patch and its wide one:
// a node's weights, positions, sums and items apart.
inline size_t direct_bound_bytes(int V, int taps) {
    return align16(taps * sizeof(float)) + align16(taps * sizeof(float2)) + align16(V * sizeof(ViewGeom)) +
           align16((size_t)V * taps * sizeof(float2)) + align16(V * sizeof(TapBox)) +
           align16(MAX_DIRECT_CANDIDATES * sizeof(double)) +
           align16((size_t)(MAX_DIRECT_CANDIDATES + 1) * V * sizeof(float2)) +
           align16((MAX_DIRECT_CANDIDATES + 1) * sizeof(float)) +
           align16((size_t)(MAX_DIRECT_CANDIDATES + 1) * V * sizeof(unsigned short));
}

template <typename TapT>
__device__ inline DirectSlot<TapT> carve_direct_slot(unsigned char *base, int V, int taps, int most) {
    DirectSlot<TapT> d;
    size_t o = 0;
    d.wt = reinterpret_cast<float2 *>(base);
    o += align16(taps * sizeof(float2));
    d.geom = reinterpret_cast<ViewGeom *>(base + o);
    o += align16(V * sizeof(ViewGeom));
    d.gh = reinterpret_cast<TapT *>(base + o);
    o += tap_bytes<TapT>(V, taps);
    d.box = reinterpret_cast<TapBox *>(base + o);
    o += align16(V * sizeof(TapBox));
    d.cand = reinterpret_cast<double *>(base + o);
    o += align16(MAX_DIRECT_CANDIDATES * sizeof(double));
    d.rr = reinterpret_cast<float *>(base + o);
    d.items = reinterpret_cast<float2 *>(base + o);
    o += align16((size_t)(most + 1) * V * sizeof(float2));
    d.agg = reinterpret_cast<float *>(base + o);
    o += align16((most + 1) * sizeof(float));
    d.list = reinterpret_cast<unsigned short *>(base + o);
    return d;
}

// nearest_coarse_depth (depth.rs:1062-1076) and direct_depth_candidates
// (depth.rs:1078-1107) by a whole warp; returns the candidate count (every
// lane) and sets `seeded`. Lane k < 13 computes offset k - 6's depth and its
// inverse; the deduplication against the last kept entry is a uniform scan of
// those inverses (1 / cand[n - 1] is the kept entry's inverse, computed the
// same way), then the kept depths are written in order.
__device__ inline int warp_direct_candidates(const DirectParams &p, double cx, double cy, double *cand,
                                             int &seeded) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int cc = sat_index_d(clampd_r(round(cx / (double)p.coarse_step), 0.0, (double)(p.coarse_columns - 1)),
                         p.coarse_columns - 1);
    int cr = sat_index_d(clampd_r(round(cy / (double)p.coarse_step), 0.0, (double)(p.coarse_rows - 1)),
                         p.coarse_rows - 1);
    int ci = cr * p.coarse_columns + cc;
    seeded = p.coarse.has[ci];
    if (!seeded) {
        cand[lane] = p.unseeded[lane];  // 32 candidates
        return 32;
    }
    double seed = p.coarse.depth[ci];
    double far_inverse = 1.0 / p.far_depth, near_inverse = 1.0 / p.near_depth;
    double depth = 0.0, inverse = 0.0;
    if (lane < 13) {
        double inv = clampd_r(1.0 / seed + (double)(lane - 6) * p.inverse_step * 0.5, far_inverse, near_inverse);
        depth = 1.0 / inv;
        inverse = 1.0 / depth;
    }
    unsigned kept = 1u;
    double last = __shfl_sync(full, inverse, 0);
    for (int k = 1; k < 13; ++k) {
        double current = __shfl_sync(full, inverse, k);
        if (fabs(last - current) > p.inverse_step * 0.1) {
            kept |= 1u << k;
            last = current;
        }
    }
    if (lane < 13 && ((kept >> lane) & 1u)) cand[__popc(kept & ((1u << lane) - 1u))] = depth;
    return __popc(kept);
}

// Warp-cooperative: reference patch and every target's tap positions for one
// node at `radius` (warp_stage_patch); geometry from the records.
template <typename TapT>
__device__ inline void warp_stage_node(const DirectParams &p, const DirectSlot<TapT> &d, RefPatch &patch, double cx,
                                       double cy, int radius, const float *spatial, const GeomRec *recs,
                                       const RefPatch *pre) {
    const int lane = threadIdx.x & 31;
    const int V = p.n_targets;
    const unsigned undefined = warp_stage_patch(p.views, p.reference, p.targets, V, cx, cy, radius, spatial, d.rr,
                                                d.wt, d.gh, d.box, patch, p.lattice, pre);
    if (lane < V) {
        geom_from_rec(recs[lane], camera_origin(p.views[p.reference].cam), d.geom[lane]);
        d.geom[lane].taps_ok = ((undefined >> lane) & 1u) ? 0 : 1;
    }
    __syncwarp();
}

// The items of a node: candidate c in [-1, n) (-1 is the baseline) in target v. By target,
// neighbouring lanes sample one target, near one another; by candidate, neighbouring lanes hold
// one candidate's targets.
template <bool BY_TARGET>
struct DirectItems {
    int count, V;  // candidates with the baseline, targets
    __device__ __forceinline__ int item(int v, int c) const { return BY_TARGET ? v * count + c + 1 : (c + 1) * V + v; }
    __device__ __forceinline__ int target(int item) const { return BY_TARGET ? item / count : item % V; }
    __device__ __forceinline__ int candidate(int item, int v) const {
        return (BY_TARGET ? item - v * count : item / V) - 1;
    }
};

// Warp-cooperative listing of the baseline and candidates cand[0..n) over all
// targets (DirectItems). It settles which items reach the correlation and which of them are fast (on
// the grid, their offset in d.items; without GRID, inside the plane), sets the others'
// scores to None and lists the scored ones: fast from the front of d.list, the rest from the
// back of its (n + 1) V entries. Every lane returns the two counts.
template <bool GRID, bool BY_TARGET, typename TapT>
__device__ inline void warp_direct_list(const DirectParams &p, const DirectSlot<TapT> &d, const RefPatch &patch,
                                        const double *cand, int n, int &n_fast, int &n_exact) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int V = p.n_targets;
    const int total = (n + 1) * V;
    const SmallDiv split(BY_TARGET ? n + 1 : V);
    const ViewGeom *geom = d.geom;
    n_fast = 0;
    n_exact = 0;
    for (int base = 0; base < total; base += 32) {
        const int item = base + lane;
        bool scored = false, fast = false;
        if (item < total) {
            const int quotient = split.quotient(item), rest = item - quotient * (int)split.d;
            const int v = BY_TARGET ? quotient : rest, c = (BY_TARGET ? rest : quotient) - 1;
            const ViewGeom &g = geom[v];
            double ddx = 0.0, ddy = 0.0;
            bool ok = g.gc_ok;
            if (ok && c >= 0) ok = depth_delta(p.views[p.targets[v]].cam, g, cand[c], ddx, ddy);
            scored = ok && patch.ok && g.taps_ok;
            if (scored) {
                const PlaneRef &plane = p.views[p.targets[v]].luma;
                if (GRID) {
                    float2 offset;
                    fast = taps_on_grid(d.box[v], ddx, ddy, plane.width, plane.height, offset);
                    if (fast) d.items[item] = offset;
                } else {
                    fast = taps_inside(tap_range(d.box[v], ddx * 0.5, ddy * 0.5), plane.width, plane.height);
                }
            } else {
                d.items[item].x = NAN;
            }
        }
        const unsigned fast_mask = __ballot_sync(full, scored && fast);
        const unsigned exact_mask = __ballot_sync(full, scored && !fast);
        if (scored && fast) d.list[n_fast + __popc(fast_mask & below)] = (unsigned short)item;
        if (scored && !fast) d.list[total - 1 - (n_exact + __popc(exact_mask & below))] = (unsigned short)item;
        n_fast += __popc(fast_mask);
        n_exact += __popc(exact_mask);
    }
}

// The taps of target v in a node's slot, the node at (cx, cy).
template <typename TapT>
__device__ __forceinline__ auto direct_taps(const DirectParams &p, const DirectSlot<TapT> &d, double cx, double cy, int v,
                                            int radius) {
    if constexpr (std::is_same<TapT, NoTap>::value)
        return lattice_taps(p.lattice, cx, cy, v, radius);
    else
        return static_cast<const TapT *>(d.gh + v * (2 * radius + 1) * (2 * radius + 1));
}

// The correlation of candidate c in target v, listed as `item` (warp_direct_list), into d.items,
// with its target's taps; one thread. `fast`: listed as on the grid.
template <bool GRID, int UNROLL, typename TapT, typename Taps>
__device__ __forceinline__ void direct_item_score(const DirectParams &p, const DirectSlot<TapT> &d,
                                                  const RefPatch &patch, const double *cand, int item, int v, int c,
                                                  const Taps &tap, bool fast, int taps) {
    const DevView &tv = p.views[p.targets[v]];
    float score;
    bool ok;
    if (GRID && fast) {
        score = zncc_grid<UNROLL>(tv.quads, tv.quad_stride, tap, d.wt, patch, taps, d.items[item], ok);
    } else {
        double ddx = 0.0, ddy = 0.0;
        if (c >= 0) depth_delta(tv.cam, d.geom[v], cand[c], ddx, ddy);
        ok = zncc_any<GRID ? UNROLL : 9>(tv, tap, d.box[v], d.wt, patch, taps, ddx, ddy, score);
    }
    d.items[item].x = ok ? score : NAN;
}

// aggregate (depth.rs:1761-1770) of the baseline and candidates over the targets into
// d.agg[0..n]; the warp of the node.
template <bool BY_TARGET, typename TapT>
__device__ inline void warp_direct_aggregate(const DirectParams &p, const DirectSlot<TapT> &d, int n) {
    const int V = p.n_targets;
    const DirectItems<BY_TARGET> items{n + 1, V};
    for (int c = threadIdx.x & 31; c <= n; c += 32) {
        float sc[MAX_VIEWS];
        for (int v = 0; v < V; ++v) sc[v] = d.items[items.item(v, c - 1)].x;
        float a;
        d.agg[c] = aggregate_scores(sc, V, p.minimum_support, p.best_view_count, a) ? a : NAN;
    }
    __syncwarp();
}

// Warp-cooperative scores of the baseline and candidates cand[0..n) over all
// targets, aggregated into d.agg[0..n] (NaN = None): the node's list, scored by
// its own warp.
template <bool GRID, int UNROLL, typename TapT>
__device__ inline void warp_direct_scores(const DirectParams &p, const DirectSlot<TapT> &d, const RefPatch &patch,
                                          const double *cand, int n, int radius, double cx, double cy) {
    const int lane = threadIdx.x & 31;
    const int taps = (2 * radius + 1) * (2 * radius + 1);
    const int total = (n + 1) * p.n_targets;
    int n_fast, n_exact;
    warp_direct_list<GRID, true>(p, d, patch, cand, n, n_fast, n_exact);
    __syncwarp();
    const DirectItems<true> items{n + 1, p.n_targets};
    const int listed = n_fast + n_exact;
    for (int j = lane; j < listed; j += 32) {
        const int item = j < n_fast ? d.list[j] : d.list[total - 1 - (j - n_fast)], v = items.target(item);
        direct_item_score<GRID, UNROLL>(p, d, patch, cand, item, v, items.candidate(item, v),
                                        direct_taps(p, d, cx, cy, v, radius), j < n_fast, taps);
    }
    __syncwarp();
    warp_direct_aggregate<true>(p, d, n);
}

// A warp per fine node; the CTA holds nodes_per_cta nodes. Each warp lists its
// node's items; the CTA then scores the pooled lists (every node's fast items,
// then every node's exact items), so the lanes of all warps stay busy up to the
// pool's last round instead of each node's; each warp then selects its node. It is bound by the
// L1's data stage and instruction issue (each some 70% of its cycles): with GRID items lie target by target, so that neighbouring
// lanes gather near one another (8.70 -> 8.51 ms at 4160x3120 with four targets). Without, on
// planes small enough to lie in the L1, there is nothing to gain by that, and a target whose
// patches cross an edge fills whole warps with the slower exact path: by candidate there (400x300,
// four targets: 0.60 -> 0.54 ms at radius 8, 0.174 -> 0.157 at radius 4).
// GRID: items on the grid (taps_on_grid) come first and take the f32 form, the others the f64
// one; without it, the items inside the plane come first and all take the f64 form. The f32
// form pays where most patches are on the grid, that is away from the plane's left and top
// edges by a few displacements: from DIRECT_GRID_SIDE pixels on. Measured (direct stage, f64
// -> GRID): 4160x3120 raster 15.8 -> 14.0 ms, 1040x780 0.414 -> 0.387 ms, 320x240 0.177 -> 0.214 ms.
// Above GRID_OFFSET_MAX_SIDE pixels no item is on the grid, and the f64 form with nine taps in
// flight is the better one: 16640x1200, four targets, 21.4 against 22.4 ms.
constexpr int DIRECT_GRID_SIDE = 400;

template <bool GRID>
__global__ void __launch_bounds__(256, 4) direct_depth_kernel(DirectParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RefPatch patches[8];
    __shared__ int pool[8][3];  // per node: fast count, exact count, list length
    const int slot = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nodes = blockDim.x >> 5;  // == p.nodes_per_cta
    const int node = blockIdx.x * p.nodes_per_cta + slot;
    const bool active = node < p.columns * p.rows;  // whole warps
    const int V = p.n_targets;
    const int taps = (2 * p.radius + 1) * (2 * p.radius + 1);
    const size_t slot_bytes = direct_slot_bytes<float2>(V, taps, MAX_DIRECT_CANDIDATES);
    DirectSlot<float2> d =
        carve_direct_slot<float2>(smem_raw + (size_t)slot * slot_bytes, V, taps, MAX_DIRECT_CANDIDATES);
    RefPatch &patch = patches[slot];
    const double cx = (double)((node % p.columns) * p.step), cy = (double)((node / p.columns) * p.step);
    int seeded = 0, n = 0, n_fast = 0, n_exact = 0;
    if (active) {
        n = warp_direct_candidates(p, cx, cy, d.cand, seeded);
        warp_stage_node(p, d, patch, cx, cy, p.radius, p.spatial, p.geometry + (size_t)node * V,
                        p.patches ? p.patches + node : nullptr);
        warp_direct_list<GRID, GRID>(p, d, patch, d.cand, n, n_fast, n_exact);
    }
    if (lane == 0) {
        pool[slot][0] = n_fast;
        pool[slot][1] = n_exact;
        pool[slot][2] = n + 1;
    }
    __syncthreads();
    int fast_total = 0, pooled = 0;
    for (int k = 0; k < nodes; ++k) {
        fast_total += pool[k][0];
        pooled += pool[k][0] + pool[k][1];
    }
    for (int j = threadIdx.x; j < pooled; j += blockDim.x) {
        // node k and the position of pooled entry j in its list
        int k = 0, at = j;
        if (j < fast_total) {
            while (at >= pool[k][0]) at -= pool[k++][0];
        } else {
            at -= fast_total;
            while (at >= pool[k][1]) at -= pool[k++][1];
            at = pool[k][2] * V - 1 - at;
        }
        const DirectSlot<float2> dk =
            carve_direct_slot<float2>(smem_raw + (size_t)k * slot_bytes, V, taps, MAX_DIRECT_CANDIDATES);
        const DirectItems<GRID> items{pool[k][2], V};
        const int item = dk.list[at], v = items.target(item);
        direct_item_score<GRID, 3>(p, dk, patches[k], dk.cand, item, v, items.candidate(item, v),
                                   direct_taps(p, dk, 0.0, 0.0, v, p.radius), j < fast_total, taps);
    }
    __syncthreads();
    if (!active) return;
    warp_direct_aggregate<GRID>(p, d, n);
    bool seen = false;
    for (int c = lane; c <= n; c += 32) seen |= d.agg[c] == d.agg[c];
    const bool tested = __any_sync(0xffffffffu, seen);
    double depth = 0.0;
    float confidence = 0.0f, improvement = 0.0f;
    int best;
    const bool has = warp_select_direct(d.cand, d.agg + 1, n, d.agg[0] == d.agg[0], d.agg[0], seeded, p.far_depth,
                                        p.near_depth, p.minimum_score, p.minimum_margin, p.minimum_improvement,
                                        depth, confidence, improvement, best);
    if (lane != 0) return;
    p.tested[node] = tested;
    p.guidance[node] = patch.centre;  // reference_guidance (depth.rs:1824-1832)
    p.out.has[node] = has;
    p.out.depth[node] = has ? depth : NAN;
    p.out.confidence[node] = has ? confidence : 0.0f;
    p.out.improvement[node] = has ? improvement : 0.0f;
    p.out.regularized[node] = 0;
    if (!has && best >= 0 && d.agg[1 + best] == d.agg[1 + best] && d.agg[1 + best] >= MINIMUM_REGULARIZED_SCORE) {
        int first = best >= 3 ? best - 3 : 0;
        int last = best + 3 < n - 1 ? best + 3 : n - 1;
        int k = atomicAdd(p.wide_count, 1);
        p.wide_list[k] = make_int4(node, first, last, seeded);
    }
}

// The wide-radius retry (depth.rs:803-846) for the listed nodes; a warp per entry, its 8 V
// correlations lane by lane, persistent over the list: warps take their further entries from a
// counter, since an entry's work depends on how many of its samples are inside their targets.
// It waits for samples: what counts is how many warps an SM holds and how much of its memory is
// left to the L1 cache. A copy of the taps (289 at the default radius, 8 bytes a target) is most
// of a warp's shared memory, so on a large grid, where it leaves an SM fewer than
// WIDE_LATTICE_WARPS, the taps are read from the tap lattice (LATTICE), as lines that neighbouring
// nodes share, in as many warps as the registers allow (24 of 80 registers; bounded to 64 they are 32
// and spill: 1.85 against 1.77 ms, 4160x3120 with four targets). Each of its entries takes longer, so a grid below WIDE_LATTICE_NODES keeps the copy, nine
// taps in flight a lane: its list is a round or two of warps, whose latency counts. Direct stage,
// copy / lattice, in ms: 400x300 (7,676 fine nodes), three targets at radius 4, 0.22 / 0.24, four at
// radius 8, 0.81 / 1.02; 1200x900 (67,951) with four at radius 4 0.91 / 0.95; 1600x1200 (120,701) with
// three 1.15 / 1.19; 2080x1560 (204,000), four targets with a narrow view, 3.01 / 2.92; 3200x2400
// (481,000) with four 8.63 / 8.13; 4160x3120 (812,000) with four 14.77 / 13.77; 16640x1200 (1.25
// million, without GRID) with four 21.3 / 19.8. With one or two targets at the default radius the copy
// fits beside as many warps as the registers allow: 1.75 / 1.84 (2080x1560, two targets).
constexpr size_t WIDE_LATTICE_NODES = 150000;
constexpr int WIDE_LATTICE_WARPS = 24;

template <bool GRID, bool LATTICE>
__global__ void __launch_bounds__(256) direct_wide_kernel(DirectParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RefPatch patches[8];
    const int slot = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    const int V = p.n_targets;
    const int taps = (2 * p.wide_radius + 1) * (2 * p.wide_radius + 1);
    using TapT = typename std::conditional<LATTICE, NoTap, float2>::type;
    DirectSlot<TapT> d = carve_direct_slot<TapT>(
        smem_raw + (size_t)slot * direct_slot_bytes<TapT>(V, taps, WIDE_CANDIDATES), V, taps, WIDE_CANDIDATES);
    RefPatch &patch = patches[slot];
    const int count = *p.wide_count;
    for (int e = blockIdx.x * warps + slot; e < count;) {
        int4 entry = p.wide_list[e];
        const int node = entry.x, first = entry.y, last = entry.z;
        const double cx = (double)((node % p.columns) * p.step), cy = (double)((node / p.columns) * p.step);
        int seeded;
        warp_direct_candidates(p, cx, cy, d.cand, seeded);
        warp_stage_node(p, d, patch, cx, cy, p.wide_radius, p.spatial_wide, p.geometry + (size_t)node * V, nullptr);
        const int n = last - first + 1;
        warp_direct_scores<GRID, LATTICE ? 4 : 9>(p, d, patch, d.cand + first, n, p.wide_radius, cx, cy);
        double depth = 0.0;
        float confidence = 0.0f, improvement = 0.0f;
        int best;
        const bool has = warp_select_direct(d.cand + first, d.agg + 1, n, d.agg[0] == d.agg[0], d.agg[0],
                                            entry.w != 0, p.far_depth, p.near_depth, p.minimum_score,
                                            p.minimum_margin, p.minimum_improvement, depth, confidence,
                                            improvement, best);
        if (has && lane == 0) {
            p.out.has[node] = 1;
            p.out.depth[node] = depth;
            p.out.confidence[node] = confidence;
            p.out.improvement[node] = improvement;
        }
        __syncwarp();
        if (lane == 0) e = gridDim.x * warps + atomicAdd(p.wide_count + 1, 1);
        e = __shfl_sync(0xffffffffu, e, 0);
    }
}

}  // namespace chiaro
