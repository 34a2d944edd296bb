// commit.cuh -- demand commit and rip-up of routed nets.
//
// Semantics of the reference's batch commit (demand.cuh:236-319): wires first
// (each unit edge gets K, its timestamp becomes the batch stamp, both segment
// endpoints are stamped), then -- after every wire of the batch is in -- vias:
// each via layer whose cell was not stamped by a wire of this batch adds K to
// its single neighbouring edge at a track end, else K/2 to the two edges it
// lands between.  K = -1 removes a route.  Half-unit integer demand makes every
// update exact and order-free, so warps may commit in any order.
#pragma once
#include "common.cuh"

namespace grb {

__device__ __forceinline__ const int* net_routes(const Plan& P, int id) { return P.routes + P.route_off[id]; }
// Words of the net's route in use: its count word, 0 for a net without route
// storage, never beyond the storage.
__device__ __forceinline__ int net_words(const Plan& P, int id) {
    const long long off = P.route_off[id], cap = P.route_off[id + 1] - off;
    return cap > 0 ? static_cast<int>(min(static_cast<long long>(P.routes[off]), cap)) : 0;
}

// A wire segment as its run of edges on a track: first slot and edge count
// (n = 0: a single cell).  `skew`: the segment runs across its layer's
// direction or between two tracks (no router emits that; a caller's own routes
// may), so its cells are not consecutive.
struct WireRun {
    int first = 0, n = 0;
    bool wire = false, skew = false;
    double length = 0.0;
};
__device__ __forceinline__ WireRun run_between(const Tables& T, int l, int x0, int y0, int x1, int y1) {
    WireRun R;
    R.wire = true;
    const bool ay = x0 == x1;
    const int lo = ay ? min(y0, y1) : min(x0, x1), hi = ay ? max(y0, y1) : max(x0, x1);
    R.n = hi - lo;
    R.skew = along_y(T, l) ? x0 != x1 : y0 != y1;
    R.first = slot_index(T, l, ay ? x0 : lo, ay ? lo : y0);
    R.length = ay ? T.ydist[hi] - T.ydist[lo] : T.xdist[hi] - T.xdist[lo];
    return R;
}
__device__ __forceinline__ WireRun wire_run(const Tables& T, int a, int b) {
    int l, x0, y0, lb, x1, y1;
    cell_position(T, a, l, x0, y0);
    cell_position(T, b, lb, x1, y1);
    return l == lb ? run_between(T, l, x0, y0, x1, y1) : WireRun();
}

// Edge at slot c of a segment gets K; its cell is stamped.
__device__ __forceinline__ void commit_edge(const Tables& T, int c, int stamp, int K) {
    red_add(T.demand + c, 2 * K);
    T.ts[c] = stamp;
}

// A skew segment, edge by edge (one thread).
__device__ __forceinline__ void commit_skew(const Tables& T, int a, int b, int stamp, int K) {
    int l, x0, y0, lb, x1, y1;
    cell_position(T, a, l, x0, y0);
    cell_position(T, b, lb, x1, y1);
    const bool ay = x0 == x1;
    const int lo = ay ? min(y0, y1) : min(x0, x1), hi = ay ? max(y0, y1) : max(x0, x1);
    for (int p = lo; p < hi; ++p) {
        const int c = slot_index(T, l, ay ? x0 : p, ay ? p : y0);
        commit_edge(T, c, stamp, K);
        mark_edge_dirty(T, c);
    }
}

// Both end cells of a segment are stamped.
__device__ __forceinline__ void stamp_ends(const Tables& T, const WireRun& R, int a, int b, int stamp) {
    if (R.skew) {
        int l, x, y;
        cell_position(T, a, l, x, y);
        T.ts[slot_index(T, l, x, y)] = stamp;
        cell_position(T, b, l, x, y);
        T.ts[slot_index(T, l, x, y)] = stamp;
    } else {
        T.ts[R.first] = stamp;
        T.ts[R.first + R.n] = stamp;
    }
}

// The edges of one run per lane (n = 0: none) are committed by the warp: those
// of all short runs shared out over the lanes together, each long run by the
// whole warp.  A run's edges are consecutive slots, so its dirty bits are set
// a bitmap word at a time by the edge that opens the word
// (fenwick.cuh:51-78).
constexpr int kLongRun = 64;
__device__ __forceinline__ void commit_runs(const Tables& T, int run_first, int n, int stamp, int K, int lane) {
    unsigned longs = __ballot_sync(0xffffffffu, n >= kLongRun);
    while (longs) {
        const int q = __ffs(longs) - 1;
        longs &= longs - 1;
        const int first = __shfl_sync(0xffffffffu, run_first, q), last = first + __shfl_sync(0xffffffffu, n, q) - 1;
        for (int c = first + lane; c <= last; c += 32) commit_edge(T, c, stamp, K);
        for (int w = (first >> 5) + lane; w <= (last >> 5); w += 32) red_or(T.dirty + w, range_bits(w, first, last));
    }
    const int m = n < kLongRun ? n : 0;
    int incl = m;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int k0 = 0; k0 < total; k0 += 32) {
        const int k = k0 + lane;
        int q = 0;  // the run of edge k: the first with incl > k
#pragma unroll
        for (int step = 16; step; step >>= 1) {
            const int v = __shfl_sync(0xffffffffu, incl, q + step - 1);
            if (v <= k) q += step;
        }
        const int first = __shfl_sync(0xffffffffu, run_first, q), cnt = __shfl_sync(0xffffffffu, m, q);
        const int end = __shfl_sync(0xffffffffu, incl, q);
        if (k < total) {
            const int c = first + (k - (end - cnt));
            commit_edge(T, c, stamp, K);
            if (c == first || (c & 31) == 0) red_or(T.dirty + (c >> 5), range_bits(c >> 5, first, first + cnt - 1));
        }
    }
}

// Sum of `length` over the warp into the wirelength.
__device__ __forceinline__ void add_wirelength(const Tables& T, double length, int K, int lane) {
    for (int s = 16; s; s >>= 1) length += __shfl_down_sync(0xffffffffu, length, s);
    if (lane == 0 && length != 0.0) atomicAdd(T.wirelength, length * K);
}

// One warp commits the wire segments of net `id` (of `parts` warps sharing a
// net, warp `part` takes every parts-th group of 32 segments), one segment per
// lane.
__device__ __forceinline__ void commit_net_wires(const Tables& T, const Plan& P, int id, int stamp, int K,
                                                 int lane, int part = 0, int parts = 1) {
    const int* r = net_routes(P, id);
    const int segs = (net_words(P, id) - 1) / 2;
    double length = 0;
    for (int s0 = 32 * part; s0 < segs; s0 += 32 * parts) {
        WireRun R;
        if (s0 + lane < segs) {
            const int a = r[1 + 2 * (s0 + lane)], b = r[2 + 2 * (s0 + lane)];
            R = wire_run(T, a, b);
            if (R.wire) {
                stamp_ends(T, R, a, b, stamp);
                length += R.length;
                if (R.skew) commit_skew(T, a, b, stamp, K);
            }
        }
        commit_runs(T, R.first, R.skew ? 0 : R.n, stamp, K, lane);
    }
    add_wirelength(T, length, K, lane);
}

// Via demand on the edge at slot c.
__device__ __forceinline__ void add_via_demand(const Tables& T, int c, int half) {
    red_add(T.demand + c, half);
    mark_edge_dirty(T, c);
}

// Demand of the via stack at (x, y) between layers low and high: every layer
// whose cell no wire of this batch stamped adds K at a track end, else K/2 to
// the two edges it lands between.  All timestamps of the stack are loaded
// before the first update.
__device__ __forceinline__ void via_stack_demand(const Tables& T, int x, int y, int low, int high, int stamp, int K) {
    int ts[kMaxLayers];
#pragma unroll
    for (int u = 0; u < kMaxLayers; ++u) ts[u] = low + u < high ? T.ts[slot_index(T, low + u, x, y)] : stamp;
#pragma unroll
    for (int u = 0; u < kMaxLayers; ++u) {
        const int layer = low + u;
        if (layer >= high || ts[u] >= stamp) continue;
        const int c = slot_index(T, layer, x, y);
        const bool ay = along_y(T, layer);
        const int pos = ay ? y : x, len = ay ? T.Y : T.X;
        if (!pos) add_via_demand(T, c, 2 * K);
        else if (pos == len - 1) add_via_demand(T, c - 1, 2 * K);
        else {
            add_via_demand(T, c - 1, K);
            add_via_demand(T, c, K);
        }
    }
}

// Route segment (a, b): if it is a via, commit its stack and return the
// number of layers it crosses, else 0.
__device__ __forceinline__ int via_segment(const Tables& T, int a, int b, int stamp, int K) {
    int la, x, y;
    cell_position(T, a, la, x, y);
    const int lb = T.by_xy(b), low = min(la, lb), high = max(la, lb);
    if (low == high) return 0;
    via_stack_demand(T, x, y, low, high, stamp, K);
    return high - low;
}

// One warp commits the via segments of the nets ids[first], ids[first +
// step], ... below ids[cnt] (routes of plan P), lanes over each net's
// segments.  The warp loads the ids and route offsets of 32 of
// its nets at once, and each net's first 32 segments (those inside its route
// capacity) while the previous net's via stacks are committed, so a net costs
// about one memory round trip instead of four.
__device__ __forceinline__ void commit_vias_strided(const Tables& T, const Plan& P, const int* ids, int cnt,
                                                    int first, int step, int stamp, int K, int lane) {
    long long vias = 0;
    for (int g0 = first; g0 < cnt; g0 += 32 * step) {
        const int mine = g0 + lane * step;
        long long off = 0, cap = 0;
        if (mine < cnt) {
            const int id = ids[mine];
            off = P.route_off[id];
            cap = P.route_off[id + 1] - off;
        }
        const int nn = min(32, (cnt - 1 - g0) / step + 1);
        const int i0 = 1 + 2 * lane;
        // Net j's word count and lane's first segment (if inside capacity).
        int words = 0, a = 0, b = 0;
        {
            const int* r = P.routes + __shfl_sync(0xffffffffu, off, 0);
            const long long c = __shfl_sync(0xffffffffu, cap, 0);
            words = c > 0 ? static_cast<int>(min(static_cast<long long>(r[0]), c)) : 0;
            if (i0 + 1 < c) { a = r[i0]; b = r[i0 + 1]; }
        }
        for (int j = 0; j < nn; ++j) {
            const int* r = P.routes + __shfl_sync(0xffffffffu, off, j);
            const long long c = __shfl_sync(0xffffffffu, cap, j);
            const int cw = words, ca = a, cb = b;
            if (j + 1 < nn) {
                const int* rn = P.routes + __shfl_sync(0xffffffffu, off, j + 1);
                const long long nc = __shfl_sync(0xffffffffu, cap, j + 1);
                words = nc > 0 ? static_cast<int>(min(static_cast<long long>(rn[0]), nc)) : 0;
                if (i0 + 1 < nc) { a = rn[i0]; b = rn[i0 + 1]; }
            }
            if (i0 + 1 < cw) vias += via_segment(T, ca, cb, stamp, K);
            for (int i = i0 + 64; i + 1 < cw; i += 64) vias += via_segment(T, r[i], r[i + 1], stamp, K);
        }
    }
    for (int s = 16; s; s >>= 1) vias += __shfl_down_sync(0xffffffffu, vias, s);
    if (lane == 0 && vias) atomicAdd(T.vias, static_cast<unsigned long long>(vias * K));
}

// Thread-per-net forms (commit_wire_demand / commit_via_demand,
// demand.cuh:129-232), used where the reference commits one net per thread
// (the Z-shape stage).  Same demand, timestamps, dirty marks and statistics as
// the warp forms above.
__device__ __forceinline__ void commit_thread_wires(const Tables& T, const Plan& P, int id, int stamp, int K) {
    const int* r = net_routes(P, id);
    const int words = net_words(P, id);
    double length = 0;
    for (int i = 1; i + 1 < words; i += 2) {
        const int a = r[i], b = r[i + 1];
        const WireRun R = wire_run(T, a, b);
        if (!R.wire) continue;
        stamp_ends(T, R, a, b, stamp);
        length += R.length;
        if (R.skew) { commit_skew(T, a, b, stamp, K); continue; }
        const int last = R.first + R.n - 1;
        for (int c = R.first; c <= last; ++c) commit_edge(T, c, stamp, K);
        if (R.n)
            for (int w = R.first >> 5; w <= (last >> 5); ++w) red_or(T.dirty + w, range_bits(w, R.first, last));
    }
    if (length != 0.0) atomicAdd(T.wirelength, length * K);
}

__device__ __forceinline__ void commit_thread_vias(const Tables& T, const Plan& P, int id, int stamp, int K) {
    const int* r = net_routes(P, id);
    const int words = net_words(P, id);
    long long vias = 0;
    for (int i = 1; i + 1 < words; i += 2) vias += via_segment(T, r[i], r[i + 1], stamp, K);
    if (vias) atomicAdd(T.vias, static_cast<unsigned long long>(vias * K));
}

}  // namespace grb
