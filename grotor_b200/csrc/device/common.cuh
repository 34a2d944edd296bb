// common.cuh -- device-side state view and shared helpers for the routing path.
//
// Grid positions in the ABI (tree nodes, route words, table transfers) follow
// the reference router (router_state.hpp:267): IDX(l,x,y) = (l*X + x)*Y + y, and
// layer l carries wires along y when ((l & 1) ^ DIR) is 1, along x otherwise.
// Demand is int32 half-units: a wire edge adds 2, a split via landing adds 1 to
// each neighbour (demand.cuh:300-304 uses 1.0f and 0.5f), so demand * 0.5f
// reproduces the reference's float.
//
// The tables themselves are stored track by track: the cells of one wire
// track (fixed x on layers along y, fixed y on the others) are consecutive
// "slots", each track padded to a multiple of 32.  A wire segment, its demand
// updates, its dirty bits, the costs they invalidate and the prefix sums over
// them are then runs of consecutive addresses on every layer; in IDX order the
// layers along x put every cell of a segment into a sector of its own.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace grb {

constexpr double kInf = 1e22;   // router_state.hpp:271
constexpr int kMaxLayers = 10;  // lshape_warp.cuh:115 asserts L <= 10
constexpr int kScanBlock = 128; // positions per prefix block (four per lane)
constexpr int kNoCapRow = 255;  // cap_id of a cell whose capacity has no table row

enum : int {
    kOk = 0, kEInval = 1, kENoMem = 2, kECuda = 3, kETimedOut = 4, kELimit = 5,
};

// Division by a number fixed per context: n / d for 0 <= n < 2^31, d >= 2, as a
// multiplication by ceil(2^p / d), p = 31 + ceil(log2 d), and a shift (Granlund
// and Montgomery, "Division by invariant integers using multiplication").
struct FastDiv {
    unsigned mul;
    int shift;
    __device__ __forceinline__ int operator()(int n) const {
        return static_cast<int>(__umulhi(static_cast<unsigned>(n), mul) >> shift);
    }
};
inline FastDiv fast_div(int d) {
    int l = 0;
    while ((1ll << l) < d) ++l;
    return FastDiv{static_cast<unsigned>(((1ull << (31 + l)) + static_cast<unsigned>(d) - 1) / static_cast<unsigned>(d)), l - 1};
}

// Device tables of one routing context.  Copied by value into every kernel.
struct Tables {
    int L, X, Y, DIR, XY;
    int cells;             // L * X * Y
    FastDiv by_xy, by_x, by_y;  // division by X * Y, X and Y
    // Track layout (slot_index): padded track lengths, slots of an even layer
    // and of an (even, odd) layer pair, all slots, all tracks.
    int xp, yp;
    int even_slots, pair_slots, slots, tracks;
    double unit_wire, unit_via, of_scale;
    const double* short_costs;
    const int* xlen;
    const int* ylen;
    const double* xdist;   // [X] distance of grid line x from line 0 (sums of xlen)
    const double* ydist;   // [Y]
    const float* capacity;
    int* demand;           // half-units
    int* ts;               // commit timestamps
    float* wcost;
    float* vcost;
    double* presum;
    // One bit per slot: the demand of the edge changed, so its wire cost, its
    // own via cost and the via cost of the next cell along the track are to
    // be recomputed (fenwick.cuh:27-38), and the track's prefix from there on.
    unsigned* dirty;
    int words;             // bitmap words (slots / 32)
    int int_wire;          // 1: wire costs clamped to [0, 1e7] and truncated (GGR build)
    // Cost-term table: row (l, k) holds, for demands h < of_dmax half-units,
    // the terms of a cell of capacity value k on layer l (cost.cuh
    // cell_terms_at); one row per layer and distinct capacity value (cap_id[c]
    // = k of cell c, kNoCapRow where the design has too many values).
    const unsigned char* cap_id;
    const double2* of_table;
    int of_rows;           // capacity values (rows per layer)
    int of_stride;         // entries per row
    int of_dmax;           // demands below this come from the table
    double* block_total;   // [tracks][track_blocks] totals of kScanBlock prefix inputs
    int track_blocks;      // prefix blocks of the longest track
    double* wirelength;
    unsigned long long* vias;
    int* error;            // first error code
    int* error_info;       // detail (net index, ...)
};

// Topology of the current plan (device pointers).
struct Plan {
    const int* node_off;       // [n_nets+1], indexed by net id
    const int* nodes;          // l*X*Y + x*Y + y, l == L for Steiner nodes
    const int* parents;        // parent < child, -1 at the root
    const long long* route_off;// [n_nets+1] word offsets into routes
    int* routes;               // [count, a0, b0, ...] per net
    const int* ids;            // net ids in execution order
    const int* batch_off;      // [n_batches+1] into ids
    int n_batches;
    // The same plan with each batch's nets grouped by size bucket
    // (kDpBuckets): bucket_ids, and per batch kDpBuckets+1 offsets into it.
    const int* bucket_ids;
    const int* bucket_off;
};

// Size buckets of the routing DP: tree nodes <= 2, <= 8, <= 16, more.
constexpr int kDpBuckets = 4;
__host__ __device__ __forceinline__ int dp_bucket(int nodes) {
    return nodes <= 2 ? 0 : nodes <= 8 ? 1 : nodes <= 16 ? 2 : 3;
}
__host__ __device__ __forceinline__ int dp_bucket_nodes(int b) { return b == 0 ? 2 : b == 1 ? 8 : 16; }

// Launch shape chosen per size bucket (grb_autotune): warps per CTA of the
// per-batch DP launch, nets per pack in the persistent form (0: by batch).
struct DpTune {
    int per_cta[kDpBuckets];
    int per_pack[kDpBuckets];
};

__device__ __forceinline__ bool along_y(const Tables& T, int l) { return ((l & 1) ^ T.DIR) != 0; }
// Position in the ABI's IDX order (route words).
__device__ __forceinline__ int cell_index(const Tables& T, int l, int x, int y) { return (l * T.X + x) * T.Y + y; }
// First slot of layer l, and the slot of a cell.
__device__ __forceinline__ int layer_base(const Tables& T, int l) {
    return (l >> 1) * T.pair_slots + ((l & 1) ? T.even_slots : 0);
}
__device__ __forceinline__ int slot_index(const Tables& T, int l, int x, int y) {
    return layer_base(T, l) + (along_y(T, l) ? x * T.yp + y : y * T.xp + x);
}
// Layer and grid position of an IDX position.
__device__ __forceinline__ void cell_position(const Tables& T, int c, int& l, int& x, int& y) {
    l = T.by_xy(c);
    const int r = c - l * T.XY;
    x = T.by_y(r);
    y = r - x * T.Y;
}

// One wire track: layer, length, padded words and first slot.
struct Track {
    int l, len, words, base;
};
__device__ __forceinline__ Track track_of(const Tables& T, int t) {
    const int pair = T.X + T.Y, p = t / pair, r = t - p * pair;
    const int even = T.DIR ? T.X : T.Y;  // tracks of an even layer
    const bool odd = r >= even;
    Track K;
    K.l = 2 * p + (odd ? 1 : 0);
    const bool ay = along_y(T, K.l);
    const int pad = ay ? T.yp : T.xp;
    K.len = ay ? T.Y : T.X;
    K.words = pad >> 5;
    K.base = layer_base(T, K.l) + (odd ? r - even : r) * pad;
    return K;
}

__device__ __forceinline__ void set_error(const Tables& T, int code, int info) {
    if (atomicCAS(T.error, 0, code) == 0) *T.error_info = info;
}

// Fire-and-forget reductions: the result is never read, so the instruction
// carries no return value and the issuing thread does not wait for L2.
__device__ __forceinline__ void red_or(unsigned* p, unsigned v) {
    asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add(int* p, int v) {
    asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// The demand of the edge at slot c changed.
__device__ __forceinline__ void mark_edge_dirty(const Tables& T, int c) { red_or(T.dirty + (c >> 5), 1u << (c & 31)); }

// Bits [first, last] of bitmap word w (32-bit words, bit positions counted
// over the whole bitmap).
__device__ __forceinline__ unsigned range_bits(int w, int first, int last) {
    unsigned m = ~0u;
    if (w == (first >> 5)) m &= ~0u << (first & 31);
    if (w == (last >> 5)) m &= ~0u >> (31 - (last & 31));
    return m;
}

// Grid-wide barrier for cooperative launches: one monotone arrival counter
// (zeroed before the launch).  Barrier k of a launch completes when the
// counter reaches k * gridDim.x, so no reset or generation word is needed and
// a barrier costs one acquire-release atomic plus acquire polls.  Every wait
// is bounded by the global timer; on expiry the kernel records kETimedOut and
// callers return.  `epoch` counts this block's barriers (a kernel-local copy).
struct GridSync {
    unsigned* count;
    unsigned long long timeout_ns;
    unsigned long long* phase_ns;  // optional per-phase time accumulators
    unsigned epoch;
};

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Thread 0 waits until *p >= target: relaxed polls (an acquire load per poll
// would invalidate the SM's L1 under the warps still working), backing off
// after the first polls so long waits do not flood the word's L2 slice, then
// one fence so later reads see the writes that preceded the producers'
// releases.  Gives up, recording kETimedOut, after timeout_ns; also returns
// false as soon as any error is recorded when `any_error` is set (the
// producer may have stopped), else only on a timeout elsewhere.
__device__ __forceinline__ bool wait_at_least(const unsigned* p, unsigned target, unsigned long long timeout_ns,
                                              const Tables& T, bool any_error) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if (v < target) {
        const unsigned long long start = global_ns();
        unsigned spins = 0;
        while (v < target) {
            if ((++spins & 63) == 0) {
                if (global_ns() - start > timeout_ns) { set_error(T, kETimedOut, blockIdx.x); return false; }
                const int e = *reinterpret_cast<volatile int*>(T.error);
                if (any_error ? e != 0 : e == kETimedOut) return false;
            }
            if (spins > 16) __nanosleep(spins > 256 ? 128 : 32);
            asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        }
    }
    __threadfence();  // acquire: later reads see every producer's writes
    return true;
}

// Barrier of `members` blocks (every block of the grid, or a subset that
// shares the counter); barrier k completes at k * members arrivals.
__device__ __forceinline__ bool grid_sync_of(GridSync& s, const Tables& T, unsigned members) {
    __shared__ int ok;
    const unsigned target = (++s.epoch) * members;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned v;
        __threadfence();
        asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(v) : "l"(s.count) : "memory");
        ok = v + 1 >= target ? 1 : wait_at_least(s.count, target, s.timeout_ns, T, false);
        if (v + 1 >= target) __threadfence();
    }
    __syncthreads();
    return ok != 0;
}
__device__ __forceinline__ bool grid_sync(GridSync& s, const Tables& T) { return grid_sync_of(s, T, gridDim.x); }

struct PhaseClock {
    unsigned long long last = 0;
    int owner = 0;  // the block whose thread 0 records
    __device__ __forceinline__ void start(const GridSync& s) {
        if (s.phase_ns && blockIdx.x == owner && threadIdx.x == 0) last = global_ns();
    }
    __device__ __forceinline__ void mark(const GridSync& s, int k) {
        if (s.phase_ns && blockIdx.x == owner && threadIdx.x == 0) {
            const unsigned long long now = global_ns();
            s.phase_ns[k] += now - last;
            last = now;
        }
    }
};

}  // namespace grb
