// decisions.cuh — the per-target cross-camera consistency check
// (crates/chiaro-fusion/src/depth.rs:420-547): refine_one_view (1634-1708),
// score_one_view_at_point (1710-1736), the Refined / Occluded / Global
// classification (458-485), enforce_warp_consensus (582-618),
// suppress_warp_boundaries (620-672) and the output warp (490-532).
//
// Decisions for every target run in one launch: a warp per fine node stages
// the reference patch once and spreads the (target, offset) and (target, shift)
// correlations over its lanes.
#pragma once

#include "cost.cuh"
#include "select.cuh"

namespace chiaro {

struct Decisions {  // NodeWarp (depth.rs:256-271) as arrays
    uint8_t *kind;
    float2 *global;
    float2 *point;
    float *confidence;
    uint8_t *measured;
};

struct DecisionParams {
    const DevView *views;
    int reference, n_targets;
    int targets[MAX_VIEWS];
    int columns, rows, step;
    Field field;
    const GeomRec *geometry;  // [node][target] of the fine grid
    TapLattice lattice;       // of the fine grid, or planes == nullptr
    const RefPatch *patches;  // [node] reference patch at `radius`, or nullptr
    double inverse_step, near_depth, far_depth;
    int radius;
    const float *spatial;
    float minimum_score;
    Decisions out[MAX_VIEWS];  // per target (index into targets)
};

constexpr int DECISION_WARPS = 4;   // most nodes (warps) per CTA

// Per-warp shared memory of the decisions for V targets and T taps.
struct DecisionSlot {
    float *rr;             // [T] reference patch (w r) r
    float2 *wt;            // [T] reference patch (w, w r)
    double2 *gh;           // [V][T] tap positions g/2
    TapBox *box;           // [V]
    float *sc;             // [V][16]: 0-4 offsets, 5 baseline, 6-13 shifts, 14 best offset
    float2 *pts;           // [V][16]
    double2 *disp;         // [8 V] displacement of each listed correlation
    unsigned short *list;  // [8 V] listed correlations
    int *flags;            // [V]: nonzero once the target's refinement failed
};

__host__ __device__ inline size_t decision_slot_bytes(int V, int taps) {
    return align16(taps * sizeof(float)) + align16(taps * sizeof(float2)) + align16((size_t)V * taps * sizeof(double2)) +
           align16(V * sizeof(TapBox)) + align16((size_t)V * 16 * sizeof(float)) +
           align16((size_t)V * 16 * sizeof(float2)) + align16((size_t)8 * V * sizeof(double2)) +
           align16((size_t)8 * V * sizeof(unsigned short)) + align16(V * sizeof(int));
}

__device__ inline DecisionSlot carve_decision_slot(unsigned char *base, int V, int taps) {
    DecisionSlot d;
    size_t o = 0;
    d.rr = reinterpret_cast<float *>(base);
    o += align16(taps * sizeof(float));
    d.wt = reinterpret_cast<float2 *>(base + o);
    o += align16(taps * sizeof(float2));
    d.gh = reinterpret_cast<double2 *>(base + o);
    o += align16((size_t)V * taps * sizeof(double2));
    d.box = reinterpret_cast<TapBox *>(base + o);
    o += align16(V * sizeof(TapBox));
    d.sc = reinterpret_cast<float *>(base + o);
    o += align16((size_t)V * 16 * sizeof(float));
    d.pts = reinterpret_cast<float2 *>(base + o);
    o += align16((size_t)V * 16 * sizeof(float2));
    d.disp = reinterpret_cast<double2 *>(base + o);
    o += align16((size_t)8 * V * sizeof(double2));
    d.list = reinterpret_cast<unsigned short *>(base + o);
    o += align16((size_t)8 * V * sizeof(unsigned short));
    d.flags = reinterpret_cast<int *>(base + o);
    return d;
}

__device__ __forceinline__ void write_decision(const Decisions &o, int node, uint8_t kind, float2 g, float2 pt,
                                               float confidence, uint8_t measured) {
    o.kind[node] = kind;
    o.global[node] = g;
    o.point[node] = pt;
    o.confidence[node] = confidence;
    o.measured[node] = measured;
}

// Append the items whose `listed` is set to d.list (in item order) with their
// displacement; returns the new length on every lane. Every lane calls it.
__device__ __forceinline__ int list_items(const DecisionSlot &d, int count, bool listed, int item, double ddx,
                                          double ddy) {
    const unsigned mask = __ballot_sync(0xffffffffu, listed);
    if (listed) {
        const int at = count + __popc(mask & ((1u << (threadIdx.x & 31)) - 1u));
        d.list[at] = (unsigned short)item;
        d.disp[at] = make_double2(ddx, ddy);
    }
    return count + __popc(mask);
}

// The correlation of d's listed entry `at` (target v). The f64 form alone (zncc_any): a node
// lists 24 or 32 items for one warp, so one item off the grid would cost the warp both loops.
template <int UNROLL>
__device__ __forceinline__ bool decision_score(const DecisionParams &p, const DecisionSlot &d, const RefPatch &patch,
                                               int at, int v, int taps, float &score) {
    const double2 dd = d.disp[at];
    return zncc_any<UNROLL>(p.views[p.targets[v]], d.gh + v * taps, d.box[v], d.wt, patch, taps, dd.x, dd.y, score);
}

// Scores the pooled lists of the CTA's nodes (node k's count[k] entries of its
// d.list / d.disp, node after node), so the lanes of all warps share the
// correlations of one phase. Phase 1 items are (target, offset k < 5 or baseline
// k = 5), phase 2 items (target, shift j < 8). A failed correlation of an offset
// or shift marks its target's refinement as failed.
template <int UNROLL>
__device__ inline void decision_pool_scores(const DecisionParams &p, unsigned char *smem_raw, size_t slot_bytes,
                                            const RefPatch *patches, const int *count, int nodes, int taps,
                                            bool shifts) {
    const int V = p.n_targets;
    int pooled = 0;
    for (int k = 0; k < nodes; ++k) pooled += count[k];
    for (int j = threadIdx.x; j < pooled; j += blockDim.x) {
        int k = 0, at = j;
        while (at >= count[k]) at -= count[k++];
        const DecisionSlot d = carve_decision_slot(smem_raw + (size_t)k * slot_bytes, V, taps);
        const int item = d.list[at];
        const int v = shifts ? item >> 3 : item / 6;
        float score;
        const bool ok = decision_score<UNROLL>(p, d, patches[k], at, v, taps, score);
        const int kk = shifts ? 6 + (item & 7) : item - v * 6;
        if (ok)
            d.sc[v * 16 + kk] = score;
        else if (shifts || kk < 5)
            atomicOr(&d.flags[v], 1);
    }
}

// A warp per fine node, every target (depth.rs:420-485 with refine_one_view,
// depth.rs:1634-1708). Each phase first settles which correlations run, lists
// them, and runs the list from one call site, so the lanes stay converged.
// POOLED (for one or two targets, whose phases list at most 12 and 16 items per
// node): the CTA scores the pooled lists of all its nodes instead, so few warps
// issue each phase's correlations; nodes without work stay for the CTA's
// barriers.
// The kernel waits for samples, so it wants warps: CTAs of four nodes with 64 registers give an SM
// 32 of them (24 of 75 registers in CTAs of eight, whose barriers, or slots kept until the CTA is
// done, also cost more). That leaves room for four taps in flight a lane instead of nine.
// Where the shared memory holds fewer than 32 warps' slots (DECISION_DEEP_SLOT), the 64 registers buy
// none: nine taps in flight and up to 80 registers then (24 warps), on patches that fill rounds of
// nine (DECISION_DEEP_TAPS). Decisions, four / nine taps, in ms: four targets at radius 4 1.64 / 1.56
// (1800x1350), 4.70 / 4.19 (3200x2400), 8.30 / 7.07 (4160x3120), at radius 8 9.70 / 7.86; two at radius
// 6 2.66 / 2.14; eight at radius 4 4.29 / 3.69; twelve 5.84 / 4.87 (4000x400). Below: three targets at
// radius 4 (5.9 KB a slot) 3.98 / 4.13 (3200x2400), six at radius 3 (49 taps) 1.60 / 1.79 (1600x1200).
// Measured, decisions of four taps: 4160x3120 with four targets 5.28 -> 4.72 ms, 3120x2340 with three 2.19 ->
// 1.93, 1567x1173 with three 0.517 -> 0.501; pooled, 2080x1560 with two 1.021 -> 0.865, 1040x780
// with one 0.378 -> 0.349. Without pooling, CTAs of two 4.67 / 1.98 / 0.517, of one 4.88 / 2.02 /
// 0.526; 48 registers 5.69 ms.
constexpr int DECISION_DEEP_TAPS = 81;
constexpr size_t DECISION_DEEP_SLOT = 7 * 1024;

template <bool POOLED, int UNROLL>
__global__ void __launch_bounds__(32 * DECISION_WARPS, UNROLL > 4 ? 6 : 8)
    target_decision_kernel(DecisionParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RefPatch patches[DECISION_WARPS];
    __shared__ int count[DECISION_WARPS];
    const unsigned full = 0xffffffffu;
    const int slot = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nodes = blockDim.x >> 5;
    const int node = blockIdx.x * nodes + slot;
    const bool in_grid = node < p.columns * p.rows;  // whole warp
    if (!POOLED && !in_grid) return;
    const int V = p.n_targets;
    const int taps = (2 * p.radius + 1) * (2 * p.radius + 1);
    const size_t slot_bytes = decision_slot_bytes(V, taps);
    DecisionSlot d = carve_decision_slot(smem_raw + (size_t)slot * slot_bytes, V, taps);
    RefPatch &patch = patches[slot];
    const DevView &rv = p.views[p.reference];
    const double cx = (double)((node % p.columns) * p.step), cy = (double)((node / p.columns) * p.step);
    const bool has = in_grid && p.field.has[node];
    // the global warp at the node: Undefined, or Global without a depth (depth.rs:433-440);
    // lane v holds target v's mapping
    unsigned defined = 0u;
    float2 gq = make_float2(0.0f, 0.0f);
    if (in_grid && lane < V) {
        float gx = 0.0f, gy = 0.0f;
        const bool ok = warp_map(p.views[p.targets[lane]].warp, (float)cx, (float)cy, gx, gy);
        gq = make_float2(gx, gy);
        if (ok) defined = 1u << lane;
        if (!ok || !has)
            write_decision(p.out[lane], node, ok ? CHIARO_NW_GLOBAL : CHIARO_NW_UNDEFINED, gq, gq, 0.0f, 0);
        d.flags[lane] = 0;
    }
    defined = __reduce_or_sync(full, defined);
    const bool active = has && defined;  // whole warp
    if (!POOLED && !active) return;
    unsigned undefined_taps = 0u;
    if (active)
        undefined_taps = warp_stage_patch(p.views, p.reference, p.targets, V, cx, cy, p.radius, p.spatial, d.rr,
                                          d.wt, d.gh, d.box, patch, p.lattice, p.patches ? p.patches + node : nullptr);
    const bool patch_ok = active && patch.ok;
    const D3 origin = camera_origin(rv.cam);
    const double shared_inverse = active ? 1.0 / p.field.depth[node] : 0.0;
    const double min_inverse = 1.0 / p.far_depth, max_inverse = 1.0 / p.near_depth;
    // phase 1: per target, five inverse-depth offsets (k < 5) and the baseline (k = 5)
    int listed = 0;
    for (int base = 0; active && base < 6 * V; base += 32) {
        const int item = base + lane;
        const int v = item / 6, k = item - v * 6;
        const int vs = v < V ? v : 0;
        const float2 gq_c = make_float2(__shfl_sync(full, gq.x, vs), __shfl_sync(full, gq.y, vs));
        bool zncc = false;
        double ddx = 0.0, ddy = 0.0;
        if (item < 6 * V && ((defined >> v) & 1u)) {
            const DevView &tv = p.views[p.targets[v]];
            const bool zncc_ok = patch_ok && !((undefined_taps >> v) & 1u);
            if (k < 5) {
                ViewGeom g;
                geom_from_rec(p.geometry[(size_t)node * V + v], origin, g);
                const double label_offset = -1.0 + 0.5 * k;
                double inv = clampd_r(shared_inverse + label_offset * p.inverse_step, min_inverse, max_inverse);
                bool ok = g.ray_ok;
                double qx = 0.0, qy = 0.0;
                if (ok) ok = project(tv.cam, along({g.ox, g.oy, g.oz}, {g.dx, g.dy, g.dz}, 1.0 / inv), qx, qy);
                if (ok) ok = isfinite(qx) && isfinite(qy);
                const float2 point = make_float2((float)qx, (float)qy);
                if (ok) {
                    ddx = (double)(point.x - gq_c.x);
                    ddy = (double)(point.y - gq_c.y);
                    ok = !(fabs(ddx) > 128.0 || fabs(ddy) > 128.0) && zncc_ok;
                }
                if (!ok) atomicOr(&d.flags[v], 1);
                d.sc[v * 16 + k] = 0.0f;
                d.pts[v * 16 + k] = point;
                zncc = ok;
            } else {
                d.sc[v * 16 + 5] = NAN;
                zncc = zncc_ok;
            }
        }
        listed = list_items(d, listed, zncc, item, ddx, ddy);
    }
    if constexpr (POOLED) {
        if (lane == 0) count[slot] = listed;
        __syncthreads();
        decision_pool_scores<UNROLL>(p, smem_raw, slot_bytes, patches, count, nodes, taps, false);
        __syncthreads();
    } else {
        __syncwarp();
        for (int j = lane; j < listed; j += 32) {
            const int item = d.list[j];
            const int v = item / 6, k = item - v * 6;
            float score;
            if (decision_score<UNROLL>(p, d, patch, j, v, taps, score))
                d.sc[v * 16 + k] = score;
            else if (k < 5)
                atomicOr(&d.flags[v], 1);
        }
        __syncwarp();
    }
    // best offset per target: in order, strict improvement
    const unsigned failed = __ballot_sync(full, active && lane < V && d.flags[lane < V ? lane : 0]);
    if (active && lane < V && ((defined >> lane) & 1u) && !((failed >> lane) & 1u)) {
        float *sc = d.sc + lane * 16;
        float2 *pts = d.pts + lane * 16;
        float best_objective = 0.0f;
        for (int k = 0; k < 5; ++k) {
            float objective = sc[k] - (float)fabs(-1.0 + 0.5 * k) * 0.002f;
            if (k == 0 || objective > best_objective) {
                best_objective = objective;
                sc[14] = sc[k];
                pts[14] = pts[k];
            }
        }
    }
    __syncwarp();
    // phase 2: per target, eight residual shifts (dy outer, dx inner, centre skipped)
    listed = 0;
    for (int base = 0; active && base < 8 * V; base += 32) {
        const int item = base + lane;
        const int v = item >> 3, j = item & 7;
        const int vs = v < V ? v : 0;
        const float2 gq_c = make_float2(__shfl_sync(full, gq.x, vs), __shfl_sync(full, gq.y, vs));
        bool zncc = false;
        double ddx = 0.0, ddy = 0.0;
        if (item < 8 * V && ((defined >> v) & 1u) && !((failed >> v) & 1u)) {
            const int k = j < 4 ? j : j + 1;
            const float dx = -1.5f + 1.5f * (float)(k % 3), dy = -1.5f + 1.5f * (float)(k / 3);
            const float2 depth_point = d.pts[v * 16 + 14];
            const float2 point = make_float2(depth_point.x + dx, depth_point.y + dy);
            ddx = (double)(point.x - gq_c.x);
            ddy = (double)(point.y - gq_c.y);
            zncc = !(fabs(ddx) > 128.0 || fabs(ddy) > 128.0) && patch_ok && !((undefined_taps >> v) & 1u);
            if (!zncc) atomicOr(&d.flags[v], 1);
            d.sc[v * 16 + 6 + j] = 0.0f;
            d.pts[v * 16 + 6 + j] = point;
        }
        listed = list_items(d, listed, zncc, item, ddx, ddy);
    }
    if constexpr (POOLED) {
        __syncwarp();
        if (lane == 0) count[slot] = listed;
        __syncthreads();
        decision_pool_scores<UNROLL>(p, smem_raw, slot_bytes, patches, count, nodes, taps, true);
        __syncthreads();
    } else {
        __syncwarp();
        for (int j = lane; j < listed; j += 32) {
            const int item = d.list[j];
            const int v = item >> 3;
            float score;
            if (decision_score<UNROLL>(p, d, patch, j, v, taps, score))
                d.sc[v * 16 + 6 + (item & 7)] = score;
            else
                atomicOr(&d.flags[v], 1);
        }
        __syncwarp();
    }
    // classification (depth.rs:458-485), lane v for target v
    if (!active || lane >= V || !((defined >> lane) & 1u)) return;
    const Decisions o = p.out[lane];
    const float *sc = d.sc + lane * 16;
    const float2 *pts = d.pts + lane * 16;
    const bool selected = !d.flags[lane];
    float sel_score = 0.0f;
    float2 sel_point = make_float2(0.0f, 0.0f);
    if (selected) {
        float b0 = sc[14], b1 = sc[14];
        float2 b2 = pts[14];
        for (int j = 0; j < 8; ++j) {
            int k = j < 4 ? j : j + 1;
            float dx = -1.5f + 1.5f * (float)(k % 3), dy = -1.5f + 1.5f * (float)(k / 3);
            float objective = sc[6 + j] - (dx * dx + dy * dy) * 0.002f;
            if (objective > b0) {
                b0 = objective;
                b1 = sc[6 + j];
                b2 = pts[6 + j];
            }
        }
        sel_score = b1;
        sel_point = b2;
    }
    const float baseline = sc[5];
    const bool base_ok = baseline == baseline;
    const bool regularized = p.field.regularized[node] != 0;
    const float node_confidence = p.field.confidence[node];
    const bool supported = selected && sel_score >= p.minimum_score && (!base_ok || sel_score + 0.01f >= baseline);
    const bool contradicted = selected && base_ok && sel_score + 0.12f < baseline;
    const uint8_t measured = regularized ? 0 : 1;
    if (contradicted)
        write_decision(o, node, CHIARO_NW_OCCLUDED, gq, gq, 0.0f, measured);
    else if (supported)
        write_decision(o, node, CHIARO_NW_REFINED, gq, sel_point,
                       regularized ? node_confidence * 0.6f : 0.5f + 0.5f * node_confidence, measured);
    else
        write_decision(o, node, CHIARO_NW_GLOBAL, gq, gq, 0.0f, 0);
}

// warp_decisions_agree (depth.rs:682-712)
__device__ inline bool decisions_agree(int kind, uint8_t ck, float2 cg, float2 cp, uint8_t nk, float2 ng, float2 np) {
    if (kind == 0 && ck == CHIARO_NW_REFINED && nk == CHIARO_NW_REFINED) {
        float cdx = cp.x - cg.x, cdy = cp.y - cg.y;
        float ndx = np.x - ng.x, ndy = np.y - ng.y;
        float dx = cdx - ndx, dy = cdy - ndy;
        return dx * dx + dy * dy <= 9.0f;
    }
    return kind == 1 && ck == CHIARO_NW_OCCLUDED && nk == CHIARO_NW_OCCLUDED;
}

// The passes after the decisions, every target (blockIdx.y) in one launch. A node that consensus
// or a boundary overrules keeps its mappings and only changes its kind (its point becomes its
// global mapping, which every reader takes for those kinds), so a pass writes one byte per node
// instead of a copy of all five arrays.
struct WarpPasses {
    Decisions decisions[MAX_VIEWS];
    uint8_t *agreed;  // [target][node] kinds after enforce_warp_consensus
    uint8_t *kinds;   // [target][node] kinds after suppress_warp_boundaries, or nullptr
    const float *guidance;
    float2 *points[MAX_VIEWS];  // output warps, or nullptr
    float *confidence[MAX_VIEWS];
    unsigned long long *counts[MAX_VIEWS];  // refined, occluded, boundary
    int columns, rows;
};

// enforce_warp_consensus (depth.rs:582-618)
__global__ void warp_consensus_kernel(WarpPasses p) {
    const int columns = p.columns, rows = p.rows;
    int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= columns * rows) return;
    const Decisions &src = p.decisions[blockIdx.y];
    uint8_t *const agreed = p.agreed + (size_t)blockIdx.y * columns * rows;
    uint8_t k = src.kind[index];
    agreed[index] = k;
    int kind, minimum;
    if (k == CHIARO_NW_REFINED) {
        kind = 0;
        minimum = src.measured[index] ? 2 : 4;
    } else if (k == CHIARO_NW_OCCLUDED) {
        kind = 1;
        minimum = src.measured[index] ? 3 : 5;
    } else {
        return;
    }
    int column = index % columns, row = index / columns;
    float2 cg = src.global[index], cp = src.point[index];
    int neighbours = 0;
    for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
            if (dx == 0 && dy == 0) continue;
            int x = column + dx, y = row + dy;
            if (x < 0 || y < 0 || x >= columns || y >= rows) continue;
            int ni = y * columns + x;
            neighbours += decisions_agree(kind, k, cg, cp, src.kind[ni], src.global[ni], src.point[ni]) ? 1 : 0;
        }
    if (neighbours < minimum) agreed[index] = CHIARO_NW_GLOBAL;
}

// warp_mapping (depth.rs:674-680) of a node of kind k
__device__ inline bool decision_mapping(const Decisions &d, uint8_t k, int i, float2 &g, float2 &pt) {
    if (k == CHIARO_NW_GLOBAL) {
        g = d.global[i];
        pt = g;
        return true;
    }
    if (k == CHIARO_NW_REFINED) {
        g = d.global[i];
        pt = d.point[i];
        return true;
    }
    return false;
}

// Does the 4-connected pair (a, b), a west/north of b, form a warp boundary?
__device__ inline bool boundary_pair(const Decisions &d, const uint8_t *kinds, const float *guidance, int a, int b) {
    float2 ga, pa, gb, pb;
    if (!decision_mapping(d, kinds[a], a, ga, pa) || !decision_mapping(d, kinds[b], b, gb, pb)) return false;
    float dax = pa.x - ga.x, day = pa.y - ga.y;
    float dbx = pb.x - gb.x, dby = pb.y - gb.y;
    float ex = dax - dbx, ey = day - dby;
    bool mapping_edge = ex * ex + ey * ey > WARP_BOUNDARY_DELTA_PX * WARP_BOUNDARY_DELTA_PX;
    bool image_edge = fabsf(guidance[a] - guidance[b]) > WARP_BOUNDARY_CONTRAST;
    return mapping_edge && image_edge;
}

// suppress_warp_boundaries (depth.rs:620-672), the output warp and decision counts
// (depth.rs:490-532).
__global__ void warp_output_kernel(WarpPasses p) {
    const int columns = p.columns, rows = p.rows, n = columns * rows, v = blockIdx.y;
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    int refined = 0, occluded = 0, boundary = 0;
    if (index < n) {
        const Decisions &d = p.decisions[v];
        const uint8_t *const kinds = p.agreed + (size_t)v * n;
        uint8_t k = kinds[index];
        if (k == CHIARO_NW_GLOBAL || k == CHIARO_NW_REFINED) {
            const int column = index % columns, row = index / columns;
            if ((column + 1 < columns && boundary_pair(d, kinds, p.guidance, index, index + 1)) ||
                (row + 1 < rows && boundary_pair(d, kinds, p.guidance, index, index + columns)) ||
                (column > 0 && boundary_pair(d, kinds, p.guidance, index - 1, index)) ||
                (row > 0 && boundary_pair(d, kinds, p.guidance, index - columns, index)))
                k = CHIARO_NW_BOUNDARY;
        }
        if (p.kinds) p.kinds[(size_t)v * n + index] = k;
        float2 pt;
        float c;
        switch (k) {
            case CHIARO_NW_UNDEFINED: pt = make_float2(NAN, NAN); c = 0.0f; break;
            case CHIARO_NW_GLOBAL: pt = d.global[index]; c = 1.0f; break;
            case CHIARO_NW_REFINED: pt = d.point[index]; c = d.confidence[index]; refined = 1; break;
            case CHIARO_NW_OCCLUDED: pt = d.global[index]; c = 0.0f; occluded = 1; break;
            default: pt = d.global[index]; c = 0.0f; boundary = 1; break;
        }
        if (p.points[v]) {
            p.points[v][index] = pt;
            p.confidence[v][index] = c;
        }
    }
    if (!p.counts[v]) return;
    unsigned full = 0xffffffffu;
    int rc = __popc(__ballot_sync(full, refined)), oc = __popc(__ballot_sync(full, occluded)),
        bc = __popc(__ballot_sync(full, boundary));
    if ((threadIdx.x & 31) == 0) {
        if (rc) atomicAdd(p.counts[v] + 0, (unsigned long long)rc);
        if (oc) atomicAdd(p.counts[v] + 1, (unsigned long long)oc);
        if (bc) atomicAdd(p.counts[v] + 2, (unsigned long long)bc);
    }
}

}  // namespace chiaro
