// stats.cuh — the depth map (crates/chiaro-fusion/src/depth.rs:534-547), the report's node
// counts and its two medians (depth.rs:394-418).
//
// A median is one order statistic, so it is selected, not sorted for: the keys' bits are
// walked from the top in digits of 13, each pass a histogram of the keys that agree with the
// digits found so far, whose bin at the wanted rank is the next digit (5 passes for the f64
// depths, 3 for the f32 improvements, which ride along). The block that finishes a pass last
// picks the digit; no block waits for another. The first pass also writes the depth map and
// counts the nodes. Two full radix sorts did the same in 16 launches, each a few microseconds
// of latency: 215 us of the 4160x3120 stage and 117 us of the 320x240 one.
#pragma once

#include "select.cuh"

namespace chiaro {

struct Results {  // read back once at the end of a stage
    int status;   // UNION_GAVE_UP when a component join ran out of retries
    unsigned long long tested, measured, regularized;
    unsigned long long target_counts[MAX_VIEWS][3];
    double median_depth;
    float median_improvement;
    int has_median_depth, has_median_improvement;
};

constexpr int SELECT_BITS = 13;
constexpr int SELECT_BINS = 1 << SELECT_BITS;
constexpr int SELECT_PASSES = 5;  // of the f64 keys

// Per key kind (0: depths, 1: improvements); zeroed before the first pass.
struct SelectState {
    unsigned bins[2][SELECT_BINS];
    unsigned done[2];             // blocks that finished the pass
    unsigned long long prefix[2]; // digits found so far
    unsigned long long rank[2];   // of the wanted key among those that share them
};

// The key's order as an unsigned integer's (f64::total_cmp and f32::total_cmp).
__device__ __forceinline__ unsigned long long depth_key(double v) {
    const unsigned long long u = d2u(v);
    return u >> 63 ? ~u : u | (1ull << 63);
}
__device__ __forceinline__ unsigned improvement_key(float v) {
    const unsigned u = f2u(v);
    return u >> 31 ? ~u : u | (1u << 31);
}

// Lowest bit of pass `pass`'s digit of a `width`-bit key, and its bits.
__device__ __forceinline__ int digit_shift(int width, int pass) { return max(width - SELECT_BITS * (pass + 1), 0); }
__device__ __forceinline__ int digit_bits(int width, int pass) { return min(SELECT_BITS, width - SELECT_BITS * pass); }

struct StatsParams {
    Field field;
    const uint8_t *tested;
    int n, pass;
    Results *results;
    SelectState *state;
    double *depth;  // the depth map
    float *confidence;
    uint8_t *provenance;
};

// Pass `pass` of key kind blockIdx.y over all nodes; the first also writes the map and counts.
template <bool FIRST>
__global__ void __launch_bounds__(256) field_stats_kernel(StatsParams p) {
    __shared__ __align__(16) unsigned bins[SELECT_BINS];
    __shared__ unsigned warp_sums[8];
    __shared__ bool last;
    const int tid = threadIdx.x, kind = blockIdx.y, width = kind == 0 ? 64 : 32;
    SelectState &st = *p.state;
    const int shift = digit_shift(width, p.pass), bits = digit_bits(width, p.pass);
    if (bits <= 0) return;  // the f32 keys are done
    const int quads = ((1 << bits) + 3) / 4;
    for (int i = tid; i < quads; i += 256) reinterpret_cast<uint4 *>(bins)[i] = make_uint4(0u, 0u, 0u, 0u);
    const unsigned long long prefix = FIRST ? 0 : st.prefix[kind];
    __syncthreads();
    for (int base = blockIdx.x * 256; base < p.n; base += gridDim.x * 256) {  // whole warps
        const int i = base + tid;
        const bool in = i < p.n;
        const bool has = in && p.field.has[i], measured = has && !p.field.regularized[i];
        if (FIRST && kind == 0) {
            const bool tested = in && p.tested[i];
            const unsigned ct = __popc(__ballot_sync(0xffffffffu, tested));
            const unsigned cm = __popc(__ballot_sync(0xffffffffu, measured));
            const unsigned cr = __popc(__ballot_sync(0xffffffffu, has && !measured));
            if ((tid & 31) == 0) {
                if (ct) atomicAdd(&p.results->tested, (unsigned long long)ct);
                if (cm) atomicAdd(&p.results->measured, (unsigned long long)cm);
                if (cr) atomicAdd(&p.results->regularized, (unsigned long long)cr);
            }
            if (in) {
                p.depth[i] = has ? p.field.depth[i] : NAN;
                p.confidence[i] = has ? p.field.confidence[i] : (tested ? 1.0f : 0.0f);
                p.provenance[i] = has ? (measured ? CHIARO_MEASURED : CHIARO_REGULARIZED)
                                      : (tested ? CHIARO_GLOBAL : CHIARO_UNSUPPORTED);
            }
        }
        const bool member = kind == 0 ? has : measured;
        unsigned long long key = 0;
        if (member) key = kind == 0 ? depth_key(p.field.depth[i]) : improvement_key(p.field.improvement[i]);
        const bool match = member && (FIRST || (key >> (shift + bits)) == prefix);
        const unsigned voters = __ballot_sync(0xffffffffu, match);
        if (match) {  // lanes of a bin add together: the first digits are few
            const unsigned bin = (unsigned)(key >> shift) & ((1u << bits) - 1u);
            const unsigned peers = __match_any_sync(voters, bin);
            if ((tid & 31) == __ffs(peers) - 1) atomicAdd(&bins[bin], (unsigned)__popc(peers));
        }
    }
    __syncthreads();
    for (int i = tid; i < 1 << bits; i += 256)
        if (bins[i]) atomicAdd(&st.bins[kind][i], bins[i]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(&st.done[kind], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    // ---- the last block of this kind: every block's counts are in; the digit at the rank.
    // With the first pass the counts of members are whole too, this kind's own bins'.
    // The counts come to shared memory first, many loads at a time: read one after another where
    // they are added up and searched, they made a pass wait 32 and up to 32 more trips to L2:
    // 18-27 us a pass against 9-14 (1040x780 stage: 1216 -> 1171 us).
    __threadfence();
    uint4 *const counts = reinterpret_cast<uint4 *>(st.bins[kind]);
#pragma unroll 8
    for (int i = tid; i < quads; i += 256) {
        reinterpret_cast<uint4 *>(bins)[i] = __ldcg(counts + i);
        counts[i] = make_uint4(0u, 0u, 0u, 0u);  // for the next pass
    }
    __syncthreads();
    const int per = max((1 << bits) / 256, 1);  // bins of a thread: a power of two
    unsigned mine = 0;
    if (tid * per < 1 << bits)
        for (int i = 0; i < per; ++i) mine += bins[tid * per + ((i + tid) & (per - 1))];  // lanes on different banks
    unsigned upto = mine;  // inclusive sums over the block
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned add = __shfl_up_sync(0xffffffffu, upto, off);
        if ((tid & 31) >= off) upto += add;
    }
    if ((tid & 31) == 31) warp_sums[tid >> 5] = upto;
    __syncthreads();
    unsigned total = 0;
    for (int w = 0; w < 8; ++w) {
        if (w < tid >> 5) upto += warp_sums[w];
        total += warp_sums[w];
    }
    const unsigned long long rank = FIRST ? total / 2 : st.rank[kind];
    const unsigned long long before = upto - mine;
    const bool found = rank >= before && rank < before + mine;
    __syncthreads();
    if (found) {
        unsigned long long at = before;
        int b = tid * per;
        for (;; ++b) {
            const unsigned count = bins[b];
            if (rank < at + count) break;
            at += count;
        }
        const unsigned long long key = (prefix << bits) | (unsigned)b;
        st.prefix[kind] = key;
        st.rank[kind] = rank - at;
        if (shift == 0 && kind == 0) {
            p.results->median_depth = u2d(key >> 63 ? key & ~(1ull << 63) : ~key);
            p.results->has_median_depth = 1;
        } else if (shift == 0) {
            const unsigned k = (unsigned)key;
            p.results->median_improvement = __uint_as_float(k >> 31 ? k & 0x7fffffffu : ~k);
            p.results->has_median_improvement = 1;
        }
    }
    if (tid == 0) st.done[kind] = 0;
}

}  // namespace chiaro
