// cost.cuh — build_cost_volume (crates/chiaro-fusion/src/depth.rs:1187-1277).
//
// A CTA takes a tile of up to 4 x 2 coarse nodes. For each target in turn it stages the
// nodes' taps, settles for every (node, label) item whether the hypothesis projects within
// reach and whether its taps lie on the grid (taps_on_grid), and lists the items that are
// scored. The listed hypotheses of a tile spread along one epipolar segment, so all their
// samples fall into one rectangle of the target's plane, which the CTA copies into shared
// memory; every correlation then gathers its samples there (zncc_region). Last, a thread per
// (node, label) aggregates the views (depth.rs:1761-1770) and writes the label-minor
// score and cost rows (node-major [N][D], as the reference lays them out).
//
// Bounds: a CTA per node that gathered 16-byte quads through the L1 was bound by the L1's data
// stage (88% busy; about 11 passes a gather, the samples of a warp's labels lying in some 20
// lines) and took 9.35 ms for 4160x3120, four targets, 129 labels. From the region a tap's four
// shared loads take 7 to 8 passes (a warp's labels are 0.5 to 1.6 pixels apart, so some share a
// bank) and the kernel is bound by instruction issue (68%) with the L1's data stage, which serves the
// shared memory, at 78%: 7.75 ms, with the sample planes and patches 7.96. Two things decide that: the inner loops are not
// unrolled (four-fold unrolled they missed the instruction cache, 9.58 ms), and the per-view
// scores and the rare f64 displacements go to scratch in global memory, so that seven CTAs
// stay resident (29 KB each).
//
// cost_volume_node_kernel, the form for small grids and planes, also scores a subset of the labels
// for the learned band: each node scores `slots` labels, slot 0 being label 0 (the global warp) and the others
// either one label list shared by every node (the band proposal's sampled labels)
// or its tile's band [O, O + slots - 1); rows are then [N][slots]. In either form
// a node list restricts the CTAs to some nodes (the fallback windows), each writing the row
// of its list position. A label's score and cost do not depend on which other
// labels a node scores, so every subset holds the full volume's values bit for bit.
#pragma once

#include "zncc.cuh"

namespace chiaro {

struct CostParams {
    const DevView *views;       // all modules
    int reference;              // reference module
    int n_targets;              // scored modules (accepted, calibrated, not the reference)
    int targets[MAX_VIEWS];
    int columns, rows, step;    // coarse grid
    int labels;                 // D = planes + 1
    const double *label_depth;  // [D], label 0 unused (the global warp)
    double near_depth;          // of the nearest label
    const float *spatial;       // [(2r+1)^2] spatial weights
    const GeomRec *geometry;    // [node][target]
    const RefPatch *patches;    // [node] reference patch at `radius`
    int radius;
    float one;                  // 1 (add2_products)
    int tile_w, tile_h;         // nodes of a CTA
    int region_rows;            // rows of the CTA's region buffer
    unsigned char transposed[MAX_VIEWS];  // per target: its epipolar lines run nearer to the y axis
    unsigned char passes[MAX_VIEWS];      // per target: parts that its labels are scored in
    TapLattice lattice;         // of this grid, or planes == nullptr
    int minimum_support, best_view_count;
    int first_block;            // of the launch, in tiles
    float *view_scores;         // scratch [CTA][tile nodes][target][slot] of the launch
    double2 *places;            // scratch [CTA (x, then y)][places_per_block]
    int places_per_block;
    float *scores, *costs, *guidance;
    uint8_t *tested;
    // label subsets (slots == labels with no list and no bands: the full volume; node tiles always)
    int slots;                  // labels scored per node; rows of the outputs
    const int *label_list;      // [slots]: slot -> label, or nullptr
    const int *band_first;      // [tiles_y][tiles_x]: slot s > 0 -> label band_first[tile] + s - 1, or nullptr
    int band_tile, band_tiles_x;
    const int *node_list;       // entry b is scored into output row b, or nullptr
};

// The label of a slot of `node` (see CostParams).
__device__ __forceinline__ int cost_slot_label(const CostParams &p, int node, int slot) {
    if (p.label_list) return __ldg(p.label_list + slot);
    if (p.band_first) {
        if (slot == 0) return 0;
        const int row = node / p.columns, column = node - row * p.columns;
        return __ldg(p.band_first + (row / p.band_tile) * p.band_tiles_x + column / p.band_tile) + slot - 1;
    }
    return slot;
}

// Threads of a tile's CTA: T (a multiple of 32) is the kernel's template parameter; the
// stage's default is COST_THREADS, and the autotuner times the COST_SHAPES once per
// (targets, labels scored, radius) bucket. Every shape lists, scores and aggregates the
// same items, each score computed alone and the views aggregated in their order, so the
// results are the same bits whatever the shape.
constexpr int COST_THREADS = 128;
constexpr int COST_SHAPES[] = {64, 96, 128, 160, 192};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) / 16 * 16; }

// Shared memory that one node's correlations need when every target's taps and every item's
// displacement are held at once: the bound on targets, labels and radius that the cost volume
// accepts (the kernel below holds less).
__host__ __device__ inline size_t node_smem_bytes(int V, int taps, int labels) {
    const size_t items = (size_t)V * labels;
    return align16(V * sizeof(ViewGeom)) + align16(V * 4 * sizeof(double)) + align16(taps * sizeof(float)) +
           align16(taps * sizeof(float2)) + align16((size_t)V * taps * sizeof(double2)) +
           align16(items * sizeof(float)) + align16(items * sizeof(unsigned short)) + items * sizeof(double2);
}

// Dynamic shared memory of a tile CTA of K nodes.
struct TileSmem {
    float *region;         // [region_rows][REGION_PITCH] the target's samples, while its items are scored
    float4 *half;          // [K][pairs] taps of the current target (PairedTaps)
    float4 *weight;        // [K][pairs] their weights
    float2 *offset;        // [K][D] f32 offset of the item at each place of the list's front
    unsigned short *list;  // [K][D] scored items (k * D + slot): on-grid ones from the front, others from the back
    int *tap_at;           // [2 pairs] each tap's place in the lattice, or its pixel offset (dy << 16 | dx)
};

__host__ __device__ inline size_t tile_smem_bytes(int K, int taps, int slots, int region_rows) {
    const size_t items = (size_t)K * slots, pairs = (taps + 1) / 2;
    return (size_t)region_rows * REGION_PITCH * sizeof(float) + 2 * K * pairs * sizeof(float4) +
           align16(items * sizeof(float2)) + align16(items * sizeof(unsigned short)) + align16(2 * pairs * sizeof(int));
}

__device__ inline TileSmem carve_tile_smem(unsigned char *base, int K, int taps, int slots, int region_rows) {
    const size_t items = (size_t)K * slots, pairs = (taps + 1) / 2;
    TileSmem s;
    s.region = reinterpret_cast<float *>(base);
    size_t o = (size_t)region_rows * REGION_PITCH * sizeof(float);
    s.half = reinterpret_cast<float4 *>(base + o);
    o += K * pairs * sizeof(float4);
    s.weight = reinterpret_cast<float4 *>(base + o);
    o += K * pairs * sizeof(float4);
    s.offset = reinterpret_cast<float2 *>(base + o);
    o += align16(items * sizeof(float2));
    s.list = reinterpret_cast<unsigned short *>(base + o);
    o += align16(items * sizeof(unsigned short));
    s.tap_at = reinterpret_cast<int *>(base + o);
    return s;
}

constexpr int TILE_NODES = 8;  // most nodes of a CTA

// Node k of a tile CTA (-1: none) and its output row: consecutive entries of a node list, or a
// block of the grid.
__device__ __forceinline__ int tile_node(const CostParams &p, int n_rows, int k, int &row) {
    const int tile = p.first_block + blockIdx.x;
    if (p.node_list) {
        row = tile * p.tile_w * p.tile_h + k;
        return row < n_rows ? __ldg(p.node_list + row) : -1;
    }
    const int tiles_x = (p.columns + p.tile_w - 1) / p.tile_w, ty = tile / tiles_x;
    const int r = ty * p.tile_h + k / p.tile_w, c = (tile - ty * tiles_x) * p.tile_w + k % p.tile_w;
    row = r * p.columns + c;
    return r < p.rows && c < p.columns ? row : -1;
}

// Aggregates the views per label of a tile's nodes and prices the labels (depth.rs:1233-1246);
// every thread of the CTA. score: [K][V][D].
__device__ inline void aggregate_tile(const CostParams &p, const float *score, const int *node_of, const int *row_of,
                                      int *tested) {
    const int K = p.tile_w * p.tile_h, V = p.n_targets, D = p.slots;
    const SmallDiv by_slots(D);
    if (threadIdx.x < K) tested[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < K * D; i += blockDim.x) {
        const int k = by_slots.quotient(i), slot = i - k * D, node = node_of[k];
        if (node < 0) continue;
        const float *views = score + k * V * D + slot;
        float agg = 0.0f;
        bool some;
        if (V <= 4) {  // the views' scores in registers (V is the same for the whole launch)
            some = aggregate_small<4>(views, D, V, p.minimum_support, p.best_view_count, agg);
        } else if (V <= 8) {
            some = aggregate_small<8>(views, D, V, p.minimum_support, p.best_view_count, agg);
        } else {
            float sc[MAX_VIEWS];
            for (int v = 0; v < V; ++v) sc[v] = views[v * D];
            some = aggregate_scores(sc, V, p.minimum_support, p.best_view_count, agg);
        }
        const float total = some ? agg : NAN;
        float cost;
        if (isfinite(total)) {
            tested[k] = 1;
            float near_prior = slot == 0 ? 0.0f : NEAR_DEPTH_PRIOR * (float)(slot - 1) / (float)(p.labels - 2);
            cost = clampf_r(1.0f - total, 0.0f, 2.0f) + near_prior;
        } else {
            cost = MISSING_COST;
        }
        const size_t o = (size_t)row_of[k] * D + slot;
        p.scores[o] = total;
        p.costs[o] = cost;
    }
    __syncthreads();
    if (threadIdx.x < K && node_of[threadIdx.x] >= 0) {
        p.tested[row_of[threadIdx.x]] = (uint8_t)tested[threadIdx.x];
        // reference_guidance (depth.rs:1824-1832)
        p.guidance[row_of[threadIdx.x]] = p.patches[node_of[threadIdx.x]].centre;
    }
}

// The aggregation of a launch whose CTAs scored one target each.
__global__ void __launch_bounds__(128) cost_aggregate_kernel(CostParams p, int n_rows) {
    __shared__ int node_of[TILE_NODES], row_of[TILE_NODES], tested[TILE_NODES];
    const int K = p.tile_w * p.tile_h;
    if (threadIdx.x < K) node_of[threadIdx.x] = tile_node(p, n_rows, threadIdx.x, row_of[threadIdx.x]);
    aggregate_tile(p, p.view_scores + (size_t)blockIdx.x * K * p.n_targets * p.slots, node_of, row_of, tested);
}

// A CTA scores its tile for every target in turn and aggregates; where the grid is so small that
// the targets' turns are the launch's latency, it scores target blockIdx.y alone and
// cost_aggregate_kernel follows (gridDim.y > 1).
// Registers bounded to 64 per thread at every shape (1024 / T CTAs per SM).
template <int T>
__global__ void __launch_bounds__(T, 1024 / T) cost_volume_kernel(CostParams p, int n_rows) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RefPatch patch[TILE_NODES];
    __shared__ ViewGeom geom[TILE_NODES];
    __shared__ TapBox box[TILE_NODES];
    __shared__ DevCamera cam;               // of the current target
    __shared__ int node_of[TILE_NODES];     // -1: none
    __shared__ int row_of[TILE_NODES];      // output row
    __shared__ size_t lattice_at[TILE_NODES];
    __shared__ int tested[TILE_NODES];
    __shared__ int ends[2];                 // items listed on the grid, others
    __shared__ int range[4];                // the lowest and highest sample floors: x, y, -x, -y
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int warps = T / 32;
    const int K = p.tile_w * p.tile_h, V = p.n_targets, D = p.slots;
    const int side = 2 * p.radius + 1, taps = side * side, pairs = (taps + 1) / 2;
    const SmallDiv by_slots(D), by_pairs(pairs);
    const TileSmem s = carve_tile_smem(smem_raw, K, taps, D, p.region_rows);
    float *const score = p.view_scores + (size_t)blockIdx.x * K * V * D;  // [K][V][D], NaN = None
    // displacements of the list's back, as many as the scratch holds
    double2 *const places = p.places + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * p.places_per_block;
    const DevView &rv = p.views[p.reference];
    const TapLattice &lat = p.lattice;

    if (tid < K) {
        int row;
        const int node = tile_node(p, n_rows, tid, row);
        node_of[tid] = node;
        row_of[tid] = row;
        if (node >= 0) {
            patch[tid] = p.patches[node];
            if (lat.planes)
                lattice_at[tid] = lat.index((double)((node % p.columns) * p.step), (double)((node / p.columns) * p.step));
        }
    }
    for (int t = tid; t < 2 * pairs; t += T) {
        int dx = 0, dy = 0;
        tap_offset(t < taps ? t : taps - 1, p.radius, dx, dy);
        s.tap_at[t] = lat.planes ? dy * lat.columns + dx : (int)((unsigned)dy << 16) | (dx & 0xffff);
    }
    __syncthreads();

    // ---- the nodes' weights (the sums over them come with the patches)
    for (int i = tid; i < K * pairs; i += T) {
        const int k = by_pairs.quotient(i), t = 2 * (i - k * pairs), node = node_of[k];
        if (node < 0) continue;
        float w[2], wr[2];
        for (int h = 0; h < 2; ++h) {
            const int at = s.tap_at[t + h];
            float value = 0.0f;
            if (lat.planes) {
                value = __ldg(lat.planes + lattice_at[k] + at).x;
            } else {
                const double px = (double)((node % p.columns) * p.step) + (double)(short)(at & 0xffff) * 2.0;
                const double py = (double)((node / p.columns) * p.step) + (double)(at >> 16) * 2.0;
                plane_sample(rv.luma, (float)((px - 0.5) * 0.5), (float)((py - 0.5) * 0.5), value);
            }
            w[h] = __ldg(p.spatial + min(t + h, taps - 1)) * exp_f32(-1.2f * fabsf(value - patch[k].centre));
            wr[h] = w[h] * value;
        }
        s.weight[i] = make_float4(w[0], w[1], wr[0], wr[1]);
    }

    const int first_target = gridDim.y > 1 ? blockIdx.y : 0, end_target = gridDim.y > 1 ? first_target + 1 : V;
    for (int v = first_target; v < end_target; ++v) {
        const DevView &tv = p.views[p.targets[v]];
        __syncthreads();  // the weights, or the last target's correlations
        for (int i = tid; i < (int)(sizeof(DevCamera) / 8); i += T)
            reinterpret_cast<double *>(&cam)[i] = __ldg(reinterpret_cast<const double *>(&tv.cam) + i);
        // ---- a warp per node: its taps in this target, their box, its geometry
        for (int k = warp; k < K; k += warps) {
            const int node = node_of[k];
            if (node < 0) continue;
            TapBox b{INFINITY, -INFINITY, INFINITY, -INFINITY};
            bool undefined = false;
            for (int i = lane; i < pairs; i += 32) {
                float2 q[2];
                const int2 at = *reinterpret_cast<const int2 *>(s.tap_at + 2 * i);
                if (lat.planes) {
                    const float2 *plane = lat.planes + (size_t)(v + 1) * lat.plane_size() + lattice_at[k];
                    q[0] = __ldg(plane + at.x);
                    q[1] = __ldg(plane + at.y);
                    undefined |= q[0].x != q[0].x || q[1].x != q[1].x;
                } else {
                    for (int h = 0; h < 2; ++h) {
                        const int o = h ? at.y : at.x;
                        const double px = (double)((node % p.columns) * p.step) + (double)(short)(o & 0xffff) * 2.0;
                        const double py = (double)((node / p.columns) * p.step) + (double)(o >> 16) * 2.0;
                        undefined |= !warp_map(tv.warp, (float)px, (float)py, q[h].x, q[h].y);
                    }
                }
                const float4 half = make_float4(q[0].x * 0.5f, q[1].x * 0.5f, q[0].y * 0.5f, q[1].y * 0.5f);
                s.half[k * pairs + i] = half;
                b.xmin = fminf(b.xmin, fminf(half.x, half.y));
                b.xmax = fmaxf(b.xmax, fmaxf(half.x, half.y));
                b.ymin = fminf(b.ymin, fminf(half.z, half.w));
                b.ymax = fmaxf(b.ymax, fmaxf(half.z, half.w));
            }
            b = warp_tap_box(b);
            undefined = __any_sync(full, undefined);
            if (lane == 0) {
                box[k] = b;
                geom_from_rec(p.geometry[(size_t)node * V + v], camera_origin(rv.cam), geom[k]);
                geom[k].taps_ok = !undefined && patch[k].ok;
            }
        }
        const int passes = p.passes[v];
        for (int pass = 0; pass < passes; ++pass) {
            const int first = pass * D / passes, slots = (pass + 1) * D / passes - first;
            const SmallDiv by_part(slots);
            if (tid < 2) ends[tid] = 0;
            if (tid < 4) range[tid] = INT32_MAX;
            __syncthreads();
            // ---- which items are scored, and how; a warp reserves its items' places at either
            // end of the list with one shared atomic add each (the order of the list only decides
            // which thread scores which item, so it does not change a result)
            const unsigned below = (1u << lane) - 1u;
            const int total = K * slots;
            TapRange span{INFINITY, -INFINITY, INFINITY, -INFINITY};  // of this thread's items inside the plane
            for (int base = warp * 32; base < total; base += T) {
                const int i = base + lane;
                bool scored = false, fast = false;
                double ddx = 0.0, ddy = 0.0;
                int item = 0;
                float2 offset;
                if (i < total) {
                    const int k = by_part.quotient(i), slot = first + i - k * slots, node = node_of[k];
                    item = k * D + slot;
                    if (node >= 0) {
                        const ViewGeom &g = geom[k];
                        scored = g.gc_ok && g.taps_ok;
                        if (scored && slot > 0) scored = depth_delta(cam, g, p.label_depth[slot], ddx, ddy);
                        if (scored) {
                            TapRange r;
                            fast = taps_on_grid(box[k], ddx, ddy, tv.luma.width, tv.luma.height, offset, r);
                            if (!fast) r = tap_range(box[k], ddx * 0.5, ddy * 0.5);
                            if (fast || taps_inside(r, tv.luma.width, tv.luma.height)) {
                                span.x0 = fminf(span.x0, r.x0);
                                span.x1 = fmaxf(span.x1, r.x1);
                                span.y0 = fminf(span.y0, r.y0);
                                span.y1 = fmaxf(span.y1, r.y1);
                            }
                        } else {
                            score[(k * V + v) * D + slot] = NAN;
                        }
                    }
                }
                const unsigned fast_mask = __ballot_sync(full, fast);
                const unsigned other_mask = __ballot_sync(full, scored && !fast);
                int fast_at = 0, other_at = 0;
                if (lane == 0) {
                    if (fast_mask) fast_at = atomicAdd(&ends[0], __popc(fast_mask));
                    if (other_mask) other_at = atomicAdd(&ends[1], __popc(other_mask));
                }
                fast_at = __shfl_sync(full, fast_at, 0) + __popc(fast_mask & below);
                other_at = __shfl_sync(full, other_at, 0) + __popc(other_mask & below);
                if (fast) {
                    s.list[fast_at] = (unsigned short)item;
                    s.offset[fast_at] = offset;
                } else if (scored) {
                    s.list[K * D - 1 - other_at] = (unsigned short)item;
                    if (other_at < p.places_per_block) places[other_at] = make_double2(ddx, ddy);
                }
            }
            if (__any_sync(full, span.x0 < INFINITY)) {
                const TapBox b = warp_tap_box({span.x0, span.x1, span.y0, span.y1});
                if (lane == 0) {
                    atomicMin(&range[0], (int)b.xmin);
                    atomicMin(&range[1], (int)b.ymin);
                    atomicMin(&range[2], -(int)b.xmax);
                    atomicMin(&range[3], -(int)b.ymax);
                }
            }
            __syncthreads();
            const int n_fast = ends[0], listed = n_fast + ends[1];
            // ---- the rectangle that every listed sample falls into, into shared memory
            const bool transposed = p.transposed[v];
            Region region;
            const bool fits = range[0] != INT32_MAX && region_of(range, transposed, p.region_rows, region);
            if (fits) load_region(region, tv.region_plane, s.region, tid, T);
            copy_async_wait();
            __syncthreads();
            // ---- the correlations of the listed items
            for (int j = tid; j < listed; j += T) {
                const bool fast = j < n_fast;
                const int item = s.list[fast ? j : K * D - 1 - (j - n_fast)];
                const int k = by_slots.quotient(item), slot = item - k * D;
                const PairedTaps tap{s.half + k * pairs, s.weight + k * pairs};
                float result;
                bool ok;
                if (fast && fits) {
                    result = transposed
                                 ? zncc_region<true>(s.region, region, tap, patch[k], taps, s.offset[j], p.one, ok)
                                 : zncc_region<false>(s.region, region, tap, patch[k], taps, s.offset[j], p.one, ok);
                } else {
                    double2 at;
                    if (!fast && j - n_fast < p.places_per_block) {
                        at = places[j - n_fast];
                    } else {  // the region does not fit, or the scratch is full: the displacement again
                        at = make_double2(0.0, 0.0);
                        if (slot > 0) depth_delta(cam, geom[k], p.label_depth[slot], at.x, at.y);
                    }
                    const double2 place = make_double2(at.x * 0.5, at.y * 0.5);
                    if (fits && taps_inside(tap_range(box[k], place.x, place.y), tv.luma.width, tv.luma.height))
                        result = transposed ? zncc_region<true>(s.region, region, tap, patch[k], taps, place, p.one, ok)
                                            : zncc_region<false>(s.region, region, tap, patch[k], taps, place, p.one, ok);
                    else
                        ok = zncc_any<3>(tv, tap, box[k], nullptr, patch[k], taps, at.x, at.y, result);
                }
                score[(k * V + v) * D + slot] = ok ? result : NAN;
            }
            if (pass + 1 < passes) __syncthreads();  // the list and the region are written again
        }
    }
    if (gridDim.y > 1) return;
    __syncthreads();
    aggregate_tile(p, score, node_of, row_of, tested);
}

// Dynamic shared memory of a node CTA.
struct NodeSmem {
    ViewGeom *geom;        // [V]
    TapBox *box;           // [V]
    float *rr;             // [T] (w r) r
    float2 *wt;            // [T] (w, w r)
    double2 *gh;           // [V][T] g/2 of the tap positions
    float *score;          // [V][D] per-view scores, NaN = None
    unsigned short *list;  // [V][D] scored items: fast path from the front, exact path from the back
    double2 *disp;         // [V][D] displacement (ddx, ddy) of each item; ddx NaN: out of reach
};

__host__ __device__ inline size_t node_form_bytes(int V, int taps, int labels) {
    const size_t items = (size_t)V * labels;
    return align16(V * sizeof(ViewGeom)) + align16(V * sizeof(TapBox)) + align16(taps * sizeof(float)) +
           align16(taps * sizeof(float2)) + align16((size_t)V * taps * sizeof(double2)) +
           align16(items * sizeof(float)) + align16(items * sizeof(unsigned short)) + items * sizeof(double2);
}

__device__ inline NodeSmem carve_node_smem(unsigned char *base, int V, int taps, int labels) {
    const size_t items = (size_t)V * labels;
    NodeSmem s;
    size_t o = 0;
    s.geom = reinterpret_cast<ViewGeom *>(base + o);
    o += align16(V * sizeof(ViewGeom));
    s.box = reinterpret_cast<TapBox *>(base + o);
    o += align16(V * sizeof(TapBox));
    s.rr = reinterpret_cast<float *>(base + o);
    o += align16(taps * sizeof(float));
    s.wt = reinterpret_cast<float2 *>(base + o);
    o += align16(taps * sizeof(float2));
    s.gh = reinterpret_cast<double2 *>(base + o);
    o += align16((size_t)V * taps * sizeof(double2));
    s.score = reinterpret_cast<float *>(base + o);
    o += align16(items * sizeof(float));
    s.list = reinterpret_cast<unsigned short *>(base + o);
    o += align16(items * sizeof(unsigned short));
    s.disp = reinterpret_cast<double2 *>(base + o);
    return s;
}

// The form for small planes: a CTA per node, every target's items at once, samples gathered from
// the quad plane in f64. A plane of a few hundred pixels has most of its patches near an edge,
// where the f32 positions do not hold, and its grid is a wave or two of CTAs, whose latency
// counts: there a tile's turns cost more than its shared samples give (coarse search, node / tile:
// 342x249 with five targets 62 / 87 us, 363x288 with four 187 / 232 us, 569x342 with four 216 / 231;
// 778x528 with five 154 / 154, 966x661 with three 98 / 84, 1041x764 with three 752 / 662).
constexpr int COST_TILE_SIDE = 320;  // the largest target side (of the luminance plane) from which tiles pay

template <int T>
__global__ void __launch_bounds__(T, 1024 / T) cost_volume_node_kernel(CostParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RefPatch patch;
    __shared__ unsigned warp_undefined[T / 32];  // bit v: a tap of target v has no global warp
    __shared__ int list_ends[2];                 // fast items listed, exact items listed
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int warps = T / 32;
    const int out_row = blockIdx.x;
    const int node = p.node_list ? __ldg(p.node_list + out_row) : out_row;
    const int V = p.n_targets, D = p.slots, full_labels = p.labels;
    const int taps = (2 * p.radius + 1) * (2 * p.radius + 1);
    const int total = V * D;
    const int chunks = (total + T - 1) / T;
    const SmallDiv by_slots(D), by_taps(taps), side(2 * p.radius + 1);  // item / D, i / taps, tap rows
    NodeSmem s = carve_node_smem(smem_raw, V, taps, D);
    const double cx = (double)((node % p.columns) * p.step), cy = (double)((node / p.columns) * p.step);
    const DevView &rv = p.views[p.reference];
    const D3 origin = camera_origin(rv.cam);

    // ---- staging: geometry, reference patch, tap positions (from the tap lattice when
    // the grid has one)
    if (tid < V) geom_from_rec(p.geometry[(size_t)node * V + tid], origin, s.geom[tid]);
    if (tid < 2) list_ends[tid] = 0;  // read after the staging's barriers
    const TapLattice &lat = p.lattice;
    const size_t at0 = lat.planes ? lat.index(cx, cy) : 0;
    float centre = 0.0f;
    bool centre_ok;
    if (lat.planes) {
        const float2 c = __ldg(lat.planes + at0);
        centre = c.x;
        centre_ok = c.y != 0.0f;
    } else {
        centre_ok = plane_sample(rv.luma, (float)((cx - 0.5) * 0.5), (float)((cy - 0.5) * 0.5), centre);
    }
    bool sampled = true;
    for (int t = tid; t < taps; t += T) {
        int dx, dy;
        tap_offset(t, p.radius, side, dx, dy);
        float value = 0.0f;
        if (lat.planes) {
            const float2 r = __ldg(lat.planes + at0 + (ptrdiff_t)dy * lat.columns + dx);
            value = r.x;
            sampled &= r.y != 0.0f;
        } else {
            double px = cx + (double)dx * 2.0, py = cy + (double)dy * 2.0;
            sampled &= plane_sample(rv.luma, (float)((px - 0.5) * 0.5), (float)((py - 0.5) * 0.5), value);
        }
        float weight = p.spatial[t] * exp_f32(-1.2f * fabsf(value - centre));
        float weighted = weight * value;
        s.wt[t] = make_float2(weight, weighted);
        s.rr[t] = weighted * value;
    }
    unsigned undefined = 0u;
    for (int i = tid; i < V * taps; i += T) {
        const int v = by_taps.quotient(i), t = i - v * taps;
        int dx, dy;
        tap_offset(t, p.radius, side, dx, dy);
        float qx = 0.0f, qy = 0.0f;
        if (lat.planes) {
            const float2 q = __ldg(lat.planes + (size_t)(v + 1) * lat.plane_size() + at0 +
                                   (ptrdiff_t)dy * lat.columns + dx);
            qx = q.x;
            qy = q.y;
            if (qx != qx) undefined |= 1u << v;
        } else {
            double px = cx + (double)dx * 2.0, py = cy + (double)dy * 2.0;
            if (!warp_map(p.views[p.targets[v]].warp, (float)px, (float)py, qx, qy)) undefined |= 1u << v;
        }
        store_tap(s.gh[i], qx, qy);
    }
    undefined = __reduce_or_sync(full, undefined);
    if (lane == 0) warp_undefined[warp] = undefined;
    const bool all_sampled = __syncthreads_and(sampled);
    // displacement of every (target, slot) item, view-major: item = v * D + slot
    for (int item = tid; item < total; item += T) {
        const int v = by_slots.quotient(item), label = cost_slot_label(p, node, item - v * D);
        const ViewGeom &g = s.geom[v];
        double ddx = 0.0, ddy = 0.0;
        bool ok = g.gc_ok;
        if (ok && label > 0) ok = depth_delta(p.views[p.targets[v]].cam, g, p.label_depth[label], ddx, ddy);
        s.disp[item] = make_double2(ok ? ddx : NAN, ddy);
    }
    // tap boxes (eight lanes per target) and the three sequential reference
    // sums (lanes 0-2 of the warp after the box warps)
    for (int vb = warp * 4; vb < V; vb += 4 * warps) {
        const int v = vb + (lane >> 3);
        TapBox b = group8_tap_box(s.gh + (v < V ? v : V - 1) * taps, taps);
        if ((lane & 7) == 0 && v < V) s.box[v] = b;
    }
    if (warp == ((V + 3) / 4) % warps) {
        float sum = 0.0f;
        if (lane < 3)
            sum = lane == 2 ? sequential_sum(s.rr, 1, taps)
                            : sequential_sum(reinterpret_cast<const float *>(s.wt) + lane, 2, taps);
        const float count = __shfl_sync(full, sum, 0), sum_r = __shfl_sync(full, sum, 1);
        const float sum_rr = __shfl_sync(full, sum, 2);
        if (lane == 0) {
            patch.count = count;
            patch.sum_r = sum_r;
            patch.sum_rr = sum_rr;
            patch.ref_energy = sum_rr - sum_r * sum_r / count;
            patch.centre = centre;
            patch.ok = centre_ok && all_sampled;
        }
    }
    __syncthreads();

    // ---- which items are scored, and on which path; then list them: fast ones from the
    // front, exact ones from the back. A warp reserves its chunk's places at either end with
    // one shared atomic add each; the order of the list only decides which thread scores
    // which item (each score is computed alone into its own slot), so it does not change
    // a result.
    const bool patch_ok = patch.ok;
    unsigned taps_bad = 0u;
    for (int w = 0; w < warps; ++w) taps_bad |= warp_undefined[w];
    const unsigned below = (1u << lane) - 1u;
    for (int c = 0; c < chunks; ++c) {
        const int item = c * T + tid;
        bool scored = false, fast = false;
        if (item < total) {
            const int v = by_slots.quotient(item);
            const double2 dd = s.disp[item];
            scored = !(dd.x != dd.x) && patch_ok && !((taps_bad >> v) & 1u);
            if (scored) {
                const PlaneRef &plane = p.views[p.targets[v]].luma;
                fast = taps_inside(tap_range(s.box[v], dd.x * 0.5, dd.y * 0.5), plane.width, plane.height);
            } else {
                s.score[item] = NAN;
            }
        }
        const unsigned fast_mask = __ballot_sync(full, scored && fast);
        const unsigned exact_mask = __ballot_sync(full, scored && !fast);
        int fast_at = 0, exact_at = 0;
        if (lane == 0) {
            if (fast_mask) fast_at = atomicAdd(&list_ends[0], __popc(fast_mask));
            if (exact_mask) exact_at = atomicAdd(&list_ends[1], __popc(exact_mask));
        }
        fast_at = __shfl_sync(full, fast_at, 0);
        exact_at = __shfl_sync(full, exact_at, 0);
        if (scored && fast) s.list[fast_at + __popc(fast_mask & below)] = (unsigned short)item;
        if (scored && !fast) s.list[total - 1 - (exact_at + __popc(exact_mask & below))] = (unsigned short)item;
    }
    __syncthreads();
    const int n_fast = list_ends[0], n_exact = list_ends[1];

    // ---- the correlations of the listed items; an item's path is known from its place
    const int listed = n_fast + n_exact;
    for (int j = tid; j < listed; j += T) {
        const bool fast = j < n_fast;
        const int item = s.list[fast ? j : total - 1 - (j - n_fast)];
        const int v = by_slots.quotient(item);
        const DevView &tv = p.views[p.targets[v]];
        const double2 dd = s.disp[item];
        float score;
        bool ok;
        if (fast)
            score = zncc_inside<9>(tv.quads, tv.quad_stride, s.gh + v * taps, s.wt, patch, taps, dd.x * 0.5, dd.y * 0.5,
                                   ok);
        else {
            const PlaneRef plane = tv.luma;  // in registers over the taps (see zncc_any)
            ok = zncc_score(plane, s.gh + v * taps, s.wt, patch, taps, dd.x, dd.y, score);
        }
        s.score[item] = ok ? score : NAN;
    }
    __syncthreads();

    // ---- aggregate the views per label and price the label (depth.rs:1233-1246)
    int any_finite = 0;
    for (int slot = tid; slot < D; slot += T) {
        const int label = cost_slot_label(p, node, slot);
        float agg = 0.0f;
        bool some;
        if (V <= 4) {  // the views' scores in registers (V is the same for the whole launch)
            some = aggregate_small<4>(s.score + slot, D, V, p.minimum_support, p.best_view_count, agg);
        } else if (V <= 8) {
            some = aggregate_small<8>(s.score + slot, D, V, p.minimum_support, p.best_view_count, agg);
        } else {
            float sc[MAX_VIEWS];
            for (int v = 0; v < V; ++v) sc[v] = s.score[v * D + slot];
            some = aggregate_scores(sc, V, p.minimum_support, p.best_view_count, agg);
        }
        float score = some ? agg : NAN;
        float cost;
        if (isfinite(score)) {
            any_finite = 1;
            float near_prior =
                label == 0 ? 0.0f : NEAR_DEPTH_PRIOR * (float)(label - 1) / (float)(full_labels - 2);
            cost = clampf_r(1.0f - score, 0.0f, 2.0f) + near_prior;
        } else {
            cost = MISSING_COST;
        }
        size_t o = (size_t)out_row * D + slot;
        p.scores[o] = score;
        p.costs[o] = cost;
    }
    const bool tested = __syncthreads_or(any_finite);
    if (tid == 0) {
        p.tested[out_row] = tested;
        p.guidance[out_row] = patch.centre;  // reference_guidance (depth.rs:1824-1832)
    }
}

}  // namespace chiaro
