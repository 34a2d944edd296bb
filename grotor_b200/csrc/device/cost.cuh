// cost.cuh -- per-edge congestion cost and per-track prefix tables.
//
// Cost formulas follow the reference's cost model (full_update.cuh:9-83) in
// the same arithmetic: float demand/capacity differences, double scaling,
// CUDA's __expf on a float argument, a double difference weighted per layer,
// stored as float.  The prefix table is the reference's double per-track
// prefix (prefix_scan.cuh:74-114, fenwick.cuh:129-168): presum[i] sums the
// shifted track [0, w0, w1, ...] in the same association (for each set bit d of
// i, lowest first, add the pairwise total of the aligned 2^d block below), so
// every presum value is bit-identical to the reference's.
//
// B200 form: one warp owns a wire track and does everything the track needs in
// one visit (refresh_track): it recomputes the costs its dirty bits name, then
// rebuilds the prefix from the first change on.  No pass waits for another, so
// the whole refresh is one phase between two grid barriers; the reference runs
// two cost kernels and one CTA per single track with stride-Y accesses.
#pragma once
#include "common.cuh"

namespace grb {

// The exponential of the cost model: CUDA's __expf on a float argument, the
// reference's choice (full_update.cuh:12-13).  grb_cost_exp evaluates the same
// function for checkers.
__device__ __forceinline__ float cost_exp(float a) { return __expf(a); }

__device__ __forceinline__ double of_cost_scaled(double scale, float capacity, float demand) {
    if (capacity > 0.001) {
        const float diff = demand - capacity;
        return cost_exp(static_cast<float>(fmin(0.5 * diff, scale * 0.5 * diff)));
    }
    if (demand > 0) return cost_exp(static_cast<float>(fmin(1.5 * demand, scale * 1.5 * demand)));
    return 0;
}

// Cost terms of one cell: the overflow increments of adding a whole unit
// and half a unit of demand (incremental_of_cost with incre 1.0 and 0.5, in
// its arithmetic; the exponential of the current demand is shared).
__device__ __forceinline__ void cell_terms(const Tables& T, float cap, int dem_half, double sc, double& one,
                                           double& half) {
    const float dem = static_cast<float>(dem_half) * 0.5f;
    const float w1 = static_cast<float>(static_cast<double>(dem) + 1.0 + 0.0);
    const float wh = static_cast<float>(static_cast<double>(dem) + 0.5 + 0.0);
    const float w0 = static_cast<float>(static_cast<double>(dem) + 0.0);
    const double o0 = of_cost_scaled(T.of_scale, cap, w0);
    one = fmin(1e12, (of_cost_scaled(T.of_scale, cap, w1) - o0) * sc);
    half = fmin(1e12, (of_cost_scaled(T.of_scale, cap, wh) - o0) * sc);
}

// The terms the cost kernels use per cell: `wof`, the overflow increment of
// a whole unit rounded to float (what the wire cost and the end-of-track via
// cost start from) and `half`, the increment of half a unit (double, what an
// interior via cost sums).
__device__ __forceinline__ double2 terms_of(double one, double half) {
    return make_double2(static_cast<double>(static_cast<float>(one)), half);
}

// Computed from capacity and demand (out of line: the table below covers
// almost every cell, and the refresh's unrolled loops stay small).
__device__ __noinline__ double2 cell_terms_computed(const Tables& T, int c, int dem_half, double sc) {
    double one, half;
    cell_terms(T, T.capacity[c], dem_half, sc, one, half);
    return terms_of(one, half);
}

// The terms of cell c (capacity row cid, demand dem_half half-units) on a
// layer of weight sc.  The demands the cost model evaluates are h/2, h/2 + 1/2
// and h/2 + 1 (exactly (h+1)/2 and (h+2)/2 in float), so for a capacity with a
// table row and a demand in range the terms are precomputed per (layer,
// capacity, demand) by the same functions: the same bits.
__device__ __forceinline__ double2 cell_terms_at(const Tables& T, int l, int c, unsigned cid, int dem_half,
                                                 double sc) {
    if (cid != kNoCapRow && dem_half >= 0 && dem_half < T.of_dmax)
        return __ldg(T.of_table + (size_t(l) * T.of_rows + cid) * T.of_stride + dem_half);
    return cell_terms_computed(T, c, dem_half, sc);
}

// update_single_wcost_ispd24 (full_update.cuh:34-51) from the cell's terms;
// the length term is the fused multiply-add the compiler forms for
// `w += unit * len`.  elen: the edge length (ignored at the track's end).
__device__ __forceinline__ float wire_cost_of(const Tables& T, double wof, int pos, int len, int elen) {
    float w = static_cast<float>(wof);
    if (pos < len - 1) w = static_cast<float>(fma(T.unit_wire, static_cast<double>(elen), wof));
    // The GGR build keeps integer DP edges non-negative and below its sentinel
    // (full_update.cuh:47-50).
    if (T.int_wire) w = static_cast<float>(static_cast<long long>(fminf(fmaxf(w, 0.f), 1.e7f)));
    return w;
}

// update_single_vcost_ispd24 (full_update.cuh:58-83) from the terms of the
// cell and of the previous cell along its track; cross points are zero on a
// single GPU (preprocess.hpp:1757).
__device__ __forceinline__ float via_cost_of(const Tables& T, const double2& t, const double2& prev, int pos,
                                             int len) {
    float v;
    if (pos == 0) v = static_cast<float>(t.x);
    else if (pos == len - 1) v = static_cast<float>(prev.x);
    else v = static_cast<float>(t.y + prev.y);
    return static_cast<float>(static_cast<double>(v) + T.unit_via);
}

// Position of the n-th (0-based) set bit of m, which has more than n set
// bits: a binary search over halves, quarters, ... by population count, the
// same few instructions for every lane whatever n is.
__device__ __forceinline__ int nth_set_bit(unsigned m, int n) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w; w >>= 1) {
        const unsigned low = m & ((1u << w) - 1u);
        const int c = __popc(low);
        const bool up = n >= c;
        n = up ? n - c : n;
        pos = up ? pos + w : pos;
        m = up ? m >> w : low;
    }
    return pos;
}

// Costs of the track's dirty cells in the 32 bitmap words from w0 on
// (update_dirty_costs, update_dirty_wire_cost, incremental_update.cuh:44-96).
// Lane q holds word w0 + q: wb the edges whose demand changed, vb the cells
// whose via cost changed.  The window's cells are ranked with a warp prefix sum
// and taken kRounds * 32 at a time, kRounds cells per lane whose inputs are all
// loaded before any cost is computed or stored.  A cell's costs depend on its
// own terms and those of the previous cell of the track.
template <int kRounds>
__device__ __forceinline__ void refresh_window(const Tables& T, const Track& K, int w0, unsigned wb, unsigned vb,
                                               int lane) {
    const int n = __popc(vb);
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    if (!total) return;
    const double sc = T.short_costs[K.l];
    const int* elen = along_y(T, K.l) ? T.ylen : T.xlen;
    for (int r = 0; r < total; r += 32 * kRounds) {
        int pos[kRounds];  // -1: none
        bool wire[kRounds];
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
            const int k = r + q * 32 + lane;
            // Owner lane: first lane whose inclusive count exceeds k.
            int lo = 0;
#pragma unroll
            for (int step = 16; step; step >>= 1) {
                const int v = __shfl_sync(0xffffffffu, incl, lo + step - 1);
                if (v <= k) lo += step;
            }
            const int owner_incl = __shfl_sync(0xffffffffu, incl, lo);
            const unsigned ov = __shfl_sync(0xffffffffu, vb, lo), ow = __shfl_sync(0xffffffffu, wb, lo);
            pos[q] = -1;
            wire[q] = false;
            if (k < total) {
                const int bit = nth_set_bit(ov, k - (owner_incl - __popc(ov)));  // rank inside the owner's word
                pos[q] = (w0 + lo) * 32 + bit;
                wire[q] = (ow >> bit) & 1u;
            }
        }
        unsigned cid0[kRounds], cid1[kRounds];
        int dem0[kRounds], dem1[kRounds], len[kRounds];
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
            if (pos[q] < 0) continue;
            const int c = K.base + pos[q];
            cid0[q] = T.cap_id[c];
            dem0[q] = T.demand[c];
            cid1[q] = pos[q] > 0 ? T.cap_id[c - 1] : 0u;
            dem1[q] = pos[q] > 0 ? T.demand[c - 1] : 0;
            len[q] = pos[q] < K.len - 1 ? elen[pos[q]] : 0;
        }
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
            if (pos[q] < 0) continue;
            const int c = K.base + pos[q];
            const double2 t0 = cell_terms_at(T, K.l, c, cid0[q], dem0[q], sc);
            const double2 t1 = pos[q] > 0 ? cell_terms_at(T, K.l, c - 1, cid1[q], dem1[q], sc) : make_double2(0.0, 0.0);
            if (wire[q]) T.wcost[c] = wire_cost_of(T, t0.x, pos[q], K.len, len[q]);
            T.vcost[c] = via_cost_of(T, t0, t1, pos[q], K.len);
        }
    }
}

// Prefix of one block of kScanBlock positions, four per lane: a[j] is input
// s[4 * lane + j] of the shifted track on entry, and on return the sum the
// reference's association gives inside the block -- for each set bit d < 7 of
// the position, lowest first, add the total of the aligned 2^d inputs below
// (bits 0 and 1 inside the lane, the others by shuffle: after the steps below
// d, the last element of an aligned 2^d run holds that run's total).
__device__ __forceinline__ void block_prefix(double (&a)[4], int lane) {
    a[1] = a[1] + a[0];
    a[3] = a[3] + a[2];
    a[2] = a[2] + a[1];
    a[3] = a[3] + a[1];
#pragma unroll
    for (int d = 0; d < 5; ++d) {
        const double t = __shfl_sync(0xffffffffu, a[3], ((lane >> d) << d) - 1);
        if ((lane >> d) & 1) {
#pragma unroll
            for (int j = 0; j < 4; ++j) a[j] = a[j] + t;
        }
    }
}

// Totals of the aligned 2^e-block runs that end at the current block (the
// binary counter of the sequential association).
constexpr int kScanLevels = 6;  // tracks are at most 8192 = 2^6 blocks long
struct ScanStack {
    double t[kScanLevels];
    // Block b, of total x, is complete.
    __device__ __forceinline__ void push(int b, double x) {
        bool carry = true;
#pragma unroll
        for (int e = 0; e < kScanLevels; ++e) {
            if (!carry) continue;
            if ((b >> e) & 1) x = x + t[e];
            else { t[e] = x; carry = false; }
        }
    }
};

// refresh_cost (incremental_update.cuh:98-132) for one track, by one warp:
// costs of the dirty cells, then -- from the block of the first change on --
// the prefix of the wire costs in one sequential pass over the track's blocks,
// its carry a stack of block totals in registers.  Blocks before the first
// change keep their prefix; their totals come from the previous rebuild.
//
// Bound by HBM: 4 bytes read and 8 written per rebuilt position.  The form
// before this one (costs by bitmap windows over the whole grid, then two
// passes over 32-track groups with a tree of totals between them, in IDX
// order) read the wire costs twice and needed four grid barriers.
template <int kRounds>
__device__ __forceinline__ void refresh_track(const Tables& T, int t, int lane) {
    const Track K = track_of(T, t);
    unsigned* bits = T.dirty + (K.base >> 5);
    double* totals = T.block_total + size_t(t) * T.track_blocks;
    const int blocks = (K.len + kScanBlock - 1) / kScanBlock;
    bool started = false;
    unsigned last_word = 0;  // the previous window's last word
    ScanStack S;
    float edge = 0.f;        // wire cost before the next block
    for (int w0 = 0; w0 < K.words; w0 += 32) {
        const int w = w0 + lane;
        unsigned wb = w < K.words ? bits[w] : 0u;
        int b = w0 >> 2;
        const int bend = min(b + 8, blocks);
        if (__any_sync(0xffffffffu, wb != 0u) || (last_word >> 31)) {
            if (wb) bits[w] = 0u;
            unsigned below = __shfl_up_sync(0xffffffffu, wb, 1);
            if (lane == 0) below = last_word;
            last_word = __shfl_sync(0xffffffffu, wb, 31);
            unsigned vb = wb | (wb << 1) | (below >> 31);
            const int rem = K.len - w * 32;
            const unsigned in = rem >= 32 ? ~0u : rem > 0 ? (1u << rem) - 1u : 0u;
            wb &= in;
            vb &= in;
            const unsigned any = __ballot_sync(0xffffffffu, wb != 0u);
            refresh_window<kRounds>(T, K, w0, wb, vb, lane);
            __syncwarp();  // the costs just stored are read below by other lanes
            if (!started && any) {
                started = true;
                b = (w0 + __ffs(any) - 1) >> 2;
                // The totals below block b, one per lane and half.
                const double lo = lane < b ? totals[lane] : 0.0, hi = lane + 32 < b ? totals[lane + 32] : 0.0;
                for (int k = 0; k < b; ++k) S.push(k, __shfl_sync(0xffffffffu, k < 32 ? lo : hi, k & 31));
                edge = b ? T.wcost[K.base + b * kScanBlock - 1] : 0.f;
            }
        } else {
            last_word = 0;
        }
        if (!started) continue;
        const int pad = K.words * 32;
        // Four blocks at a time, their loads issued together (one in flight a
        // warp left HBM reads at a quarter of what they can be).
        for (; b < bend; b += 4) {
            float4 in[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int p = (b + u) * kScanBlock + 4 * lane;
                in[u] = b + u < bend && p < pad ? *reinterpret_cast<const float4*>(T.wcost + K.base + p)
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (b + u >= bend) continue;
                const float4 v = in[u];
                const int p = (b + u) * kScanBlock + 4 * lane;
                float before = __shfl_up_sync(0xffffffffu, v.w, 1);
                if (lane == 0) before = edge;
                edge = __shfl_sync(0xffffffffu, v.w, 31);
                double a[4] = {before, v.x, v.y, v.z};
                block_prefix(a, lane);
                const double total = __shfl_sync(0xffffffffu, a[3], 31);
                if (lane == 0) totals[b + u] = total;
#pragma unroll
                for (int e = 0; e < kScanLevels; ++e)
                    if (((b + u) >> e) & 1) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) a[j] = a[j] + S.t[e];
                    }
                S.push(b + u, total);
                if (p < pad) {
                    double2* out = reinterpret_cast<double2*>(T.presum + K.base + p);
                    out[0] = make_double2(a[0], a[1]);
                    out[1] = make_double2(a[2], a[3]);
                }
            }
        }
    }
}

// The refresh by a grid of CTAs that are all resident, CTA i owning tracks i,
// i + gridDim.x, ...: warp w takes the w-th of every warps, or (kListed) the
// CTA's warps list its dirty tracks first and take them from the list in turn.
// A batch's nets dirty a minority of the tracks and by chance some warps'
// shares are several times the mean.  Refresh a batch without and with the list,
// by tracks a warp (nine routing layers, 296 CTAs of 8 warps): 3.0 (800x800)
// 33.9 and 29.9 us, 3.8 (1000x1000) 41.3 and 36.3, 4.4 (1150x1150) 56.7 and 45.8,
// 4.9 (1300x1300) 65.1 and 54.4, 5.5 (1450x1450) 70.1 and 61.2, 6.1 (1600x1600)
// 123 and 99.  The line was drawn between two sizes, before those in between were
// measured: it is where the list certainly pays, not where it begins to.
constexpr int kListTracks = 128;  // tracks of a CTA listed at once
constexpr int kListedPerWarp = 5; // the list from this many tracks a warp on
template <int kRounds, bool kListed>
__device__ __forceinline__ void refresh_tracks(const Tables& T) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, G = gridDim.x;
    if (!kListed) {
        for (int t = warp * G + blockIdx.x; t < T.tracks; t += warps * G) refresh_track<kRounds>(T, t, lane);
        return;
    }
    __shared__ int list[kListTracks], listed, taken;
    const int mine = (T.tracks - int(blockIdx.x) + G - 1) / G;
    for (int c = 0; c < mine; c += kListTracks) {
        if (threadIdx.x == 0) listed = taken = 0;
        __syncthreads();
        const int end = min(mine, c + kListTracks);
#pragma unroll 4
        for (int j = c + warp; j < end; j += warps) {
            const int t = blockIdx.x + j * G;
            const Track K = track_of(T, t);
            unsigned any = 0u;
            for (int w = lane; w < K.words; w += 32) any |= T.dirty[(K.base >> 5) + w];
            if (__any_sync(0xffffffffu, any != 0u) && lane == 0) list[atomicAdd(&listed, 1)] = t;
        }
        __syncthreads();
        for (;;) {
            int k = 0;
            if (lane == 0) k = atomicAdd(&taken, 1);
            k = __shfl_sync(0xffffffffu, k, 0);
            if (k >= listed) break;
            refresh_track<kRounds>(T, list[k], lane);
        }
        __syncthreads();
    }
}

}  // namespace grb
