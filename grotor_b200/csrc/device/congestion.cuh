// congestion.cuh -- rip-up classification and congestion view of the
// committed demand (the reference's graph::ripup and extract_congestionView*,
// congestion.cuh:8-136).  Device functions shared by the standalone kernels
// and by the tail of the persistent L-shape stage.
#pragma once
#include "common.cuh"

namespace grb {

// The overflow marks and their prefix are stored track by track without
// padding (L*X*Y entries, so the fixed scratch of the allocation-free entry
// point holds the same grids as ever).
__device__ __forceinline__ int mark_index(const Tables& T, int l, int x, int y) {
    return l * T.XY + (along_y(T, l) ? x * T.Y + y : y * T.X + x);
}

// mark_overflow_edges (congestion.cuh:8-20): 1 where the edge of mark k's
// cell carries demand >= capacity + threshold (cells without an edge: 0).
__device__ __forceinline__ void overflow_mark(const Tables& T, int threshold, int* of_sum, int k) {
    const int l = T.by_xy(k), rem = k - l * T.XY;
    const bool ay = along_y(T, l);
    const int len = ay ? T.Y : T.X, track = ay ? T.by_y(rem) : T.by_x(rem), pos = rem - track * len;
    const int c = layer_base(T, l) + track * (ay ? T.yp : T.xp) + pos;
    of_sum[k] = (pos + 1 < len && T.capacity[c] + threshold <= static_cast<float>(T.demand[c]) * 0.5f) ? 1 : 0;
}

// Exclusive integer prefix of the marks along track t, by one warp
// (compute_presum_general, prefix_scan.cuh:42-72 -- integer sums are
// order-free).
__device__ __forceinline__ void overflow_prefix_track(const Tables& T, int* v, int t, int lane) {
    const int pair = T.X + T.Y, p = t / pair, r = t - p * pair, even = T.DIR ? T.X : T.Y;
    const int l = 2 * p + (r >= even ? 1 : 0), track = r >= even ? r - even : r;
    const int len = along_y(T, l) ? T.Y : T.X;
    int* a = v + l * T.XY + track * len;
    int carry = 0;
    for (int k0 = 0; k0 < len; k0 += 32) {
        const int x = k0 + lane < len ? a[k0 + lane] : 0;
        int incl = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        if (k0 + lane < len) a[k0 + lane] = carry + incl - x;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// mark_overflow_nets (congestion.cuh:22-58): net `id` is flagged when its
// wires cross more than 10 overflowing edges.
__device__ __forceinline__ unsigned char overflow_route(const Tables& T, const int* r, bool has, const int* of_sum) {
    int count = 0;
    unsigned char flag = 0;
    if (has) {
        for (int i = 1; i < r[0]; i += 2) {
            int l, x0, y0, lb, x1, y1;
            cell_position(T, r[i], l, x0, y0);
            cell_position(T, r[i + 1], lb, x1, y1);
            if (x0 != x1) count += of_sum[mark_index(T, l, max(x0, x1), y0)] - of_sum[mark_index(T, l, min(x0, x1), y0)];
            if (y0 != y1) count += of_sum[mark_index(T, l, x0, max(y0, y1))] - of_sum[mark_index(T, l, x0, min(y0, y1))];
            if (count > 10) { flag = 1; break; }
        }
    }
    return flag;
}
__device__ __forceinline__ void overflow_net(const Tables& T, const Plan& P, const int* of_sum, unsigned char* is_of,
                                             int id) {
    is_of[id] = overflow_route(T, P.routes + P.route_off[id], P.route_off[id + 1] > P.route_off[id], of_sum);
}

// extract_congestionView (congestion.cuh:60-80) for the 2-D cells of 32 x 32
// tile `tile`: the worst demand - capacity over the layers (at least 0).  One
// CTA of a multiple of 32 threads; layers along y are read with lanes over y,
// the others with lanes over x and transposed through shared memory, so every
// read is a run of consecutive slots.
constexpr int kViewTile = 32;
__host__ __device__ __forceinline__ int view_tiles(const Tables& T) {
    return ((T.X + kViewTile - 1) / kViewTile) * ((T.Y + kViewTile - 1) / kViewTile);
}
__device__ __forceinline__ void congestion_tile(const Tables& T, unsigned char* cong, float* xsum, float* ysum, int tile,
                                                float (*across)[kViewTile + 1]) {
    const int nty = (T.Y + kViewTile - 1) / kViewTile;
    const int x0 = tile / nty * kViewTile, y0 = tile % nty * kViewTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int q = warp; q < kViewTile; q += nw) {
        const int x = x0 + lane, y = y0 + q;
        float worst = 0.f;
        if (x < T.X && y < T.Y)
            for (int l = T.DIR; l < T.L; l += 2) {  // the layers along x
                const int e = slot_index(T, l, x, y);
                worst = fmaxf(worst, static_cast<float>(T.demand[e]) * 0.5f - T.capacity[e]);
            }
        across[q][lane] = worst;
    }
    __syncthreads();
    for (int q = warp; q < kViewTile; q += nw) {
        const int x = x0 + q, y = y0 + lane;
        if (x < T.X && y < T.Y) {
            float worst = across[lane][q];
            for (int l = T.DIR ^ 1; l < T.L; l += 2) {  // the layers along y
                const int e = slot_index(T, l, x, y);
                worst = fmaxf(worst, static_cast<float>(T.demand[e]) * 0.5f - T.capacity[e]);
            }
            const int i = x * T.Y + y;
            cong[i] = worst > 0.f;
            xsum[i] = worst;
            ysum[i] = worst;
        }
    }
    __syncthreads();  // `across` is reused by the next tile
}

// Float prefix of one line (extract_congestionView_xsum / _ysum,
// congestion.cuh:81-112): the shifted line [0, v0, v1, ...] summed in the
// reference's log-step association (for each set bit of i, lowest first, the
// total of the aligned block below), one thread per line.
__device__ __forceinline__ void congestion_line_prefix(float* a, int len, int elem_stride) {
    float tot[32];
    float prev = 0.f;
    for (int i = 0; i < len; ++i) {
        const float cur = a[size_t(i) * elem_stride];
        float acc = i ? prev : 0.f;
        prev = cur;
        float fresh[32];
        fresh[0] = acc;
        int d = 0;
        while ((i >> d) & 1) { acc = acc + tot[d]; ++d; fresh[d] = acc; }
        for (int j = 0; j <= d; ++j) tot[j] = fresh[j];
        for (int e = d + 1; (i >> e) != 0; ++e)
            if ((i >> e) & 1) acc = acc + tot[e];
        a[size_t(i) * elem_stride] = acc;
    }
}

// What the tail of an L-shape stage computes from the final demand
// (pipeline.hpp:86-93 runs the congestion view and graph::ripup right after
// the stage): flags bit 0 = rip-up classification, bit 1 = congestion view.
enum : int { kTailRipup = 1, kTailView = 2 };
struct StageTail {
    int flags;
    int threshold;
    int n_nets;
    int* of_sum;            // [cells]
    unsigned char* is_of;   // [n_nets]
    unsigned char* cong;    // [X*Y]
    float* xsum;            // [X*Y]
    float* ysum;            // [X*Y]
};

// The stage tail inside a persistent kernel (grid-stride over all threads):
// marks and per-cell view | track prefixes and line prefixes | net flags,
// separated by grid barriers.  `across`: shared memory of congestion_tile.
// False when a barrier gave up.
__device__ __forceinline__ bool stage_tail_persistent(const Tables& T, const Plan& P, const StageTail& tail,
                                                      GridSync& S, float (*across)[kViewTile + 1]) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    if (tail.flags & kTailRipup)
        for (int c = tid; c < T.cells; c += nth) overflow_mark(T, tail.threshold, tail.of_sum, c);
    if (tail.flags & kTailView)
        for (int i = blockIdx.x; i < view_tiles(T); i += gridDim.x)
            congestion_tile(T, tail.cong, tail.xsum, tail.ysum, i, across);
    if (!grid_sync(S, T)) return false;
    if (tail.flags & kTailRipup)
        for (int t = tid >> 5; t < T.tracks; t += nth >> 5) overflow_prefix_track(T, tail.of_sum, t, threadIdx.x & 31);
    if (tail.flags & kTailView) {
        // per x along y (ysum), then per y along x (xsum), one thread per line
        for (int t = tid; t < T.X + T.Y; t += nth) {
            if (t < T.X) congestion_line_prefix(tail.ysum + size_t(t) * T.Y, T.Y, 1);
            else congestion_line_prefix(tail.xsum + (t - T.X), T.X, T.Y);
        }
    }
    if (!grid_sync(S, T)) return false;
    if (tail.flags & kTailRipup)
        for (int id = tid; id < tail.n_nets; id += nth) overflow_net(T, P, tail.of_sum, tail.is_of, id);
    return true;
}

}  // namespace grb
