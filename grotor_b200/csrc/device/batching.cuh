// batching.cuh -- exact greedy first-fit net batching on the GPU.
//
// Semantics of the reference's CPU batching (generate_batches_cpu.hpp:7-73):
// nets are taken in the given order; a net joins the first batch that holds
// fewer than `limit` nets and none of whose marked cells contains one of the
// net's query points; it then marks its RSMT h-segments (step sparsity*Y),
// v-segments (step sparsity) and, at every point, the cell itself, its x
// neighbours and the cell below in y (not above, reference :38).
//
// B200 algorithm (replaces the RT-core/OptiX and CPU paths, which produce the
// same lists):
//   * once per run, every net's marked cells and query points are written to
//     flat lists in order-position order (k_flat_*), tagged with the net's
//     position inside a chunk, so each per-chunk step below is one balanced,
//     coalesced pass over a contiguous range;
//   * cellmask holds one bit per batch ("colour") already marking each cell,
//     plane-major (colour word w of all cells contiguous);
//   * nets are processed in chunks of CH (1024, or 512 when the solver's
//     shared memory for the colour words would not fit) in order; per chunk:
//       1. raster: every mark on a query point of this chunk or (persistent
//          form) of the two chunks after it (per-cell chunk bits,
//          L2-resident, filter the rest) ORs its net's bit into the
//          chunk-local mask of the cell (five buffers by chunk index);
//       2. gather: every query point ORs, into its net's column of the chunk
//          tables, the cell's colours (forbidden batches of earlier chunks),
//          the chunk-local bits of earlier nets of the chunk (predecessors),
//          and -- in the persistent form -- the bits of the previous chunk's
//          nets and the colours of the nets two chunks back;
//       3. solve: one CTA solves first-fit inside the chunk by Jacobi
//          iteration over the predecessor DAG (converges to the unique
//          sequential solution), then applies batch capacities in order;
//       4. publish: every mark ORs its net's colour into cellmask; the
//          chunk-local mask is emptied at the chunk's query points.
//   Positions inside the batches come from a stable counting pass after the
//   run.  Plain form: one launch per step per chunk.  Persistent form: one
//   cooperative kernel in which CTA 0 solves chunk r while the other CTAs, in
//   one phase and one grid barrier, publish chunk r-1, gather chunk r+1 and
//   raster chunk r+2; the gather reads cellmask as of chunk r-2 at least (chunk
//   r-1's publish runs beside it), resolves chunk r-1's nets through that
//   chunk's local mask and its solved colours, and takes chunk r's colours
//   through the previous-chunk bits, which the solver resolves from the colours
//   it keeps in shared memory.  The solver and the other CTAs hand chunks over
//   through two monotone counters (bounded waits), so the solve never waits
//   for a publish.
#pragma once
#include "common.cuh"

namespace grb {

// Nets per chunk: CH = 512 or 1024 (== threads of the solve CTA), a template
// parameter of every per-chunk step; storage is sized for the larger.
constexpr int kChunkMax = 1024;
constexpr int kChunkMaxWords = kChunkMax / 32;

struct BatchState {
    int X, Y, n, limit, sparsity, W;   // W: colour words per cell
    const int* order;
    const int* point_off; const int* points;
    const int* hseg_off; const int* hsegs;
    const int* vseg_off; const int* vsegs;
    // Flat lists by order position (k_flat_*).
    long long* mark_off;        // [n+1]
    unsigned* mark_cell;        // cells marked by the nets (duplicates allowed)
    unsigned short* mark_jj;    // position of the marking net inside its chunk
    long long* pt_off;          // [n+1]
    unsigned* pt_cell;          // query points
    unsigned short* pt_jj;
    unsigned* cellmask;         // [W][X*Y]: word w of every cell contiguous, so the
                                // colour ORs of consecutive cells share sectors
    unsigned* localmask[5];     // [X*Y][CH/32], chunk k in buffer k % 5
    unsigned* localset[5];      // [X*Y] which words of the cell's record are nonzero
    unsigned* ptchunk;          // [X*Y] bit k % 32: the cell is a query point of chunk k
    unsigned* fmask;            // [2][W][CH] forbidden colours, by chunk parity
    unsigned* pred;             // [2][CH/32][CH] predecessors inside the chunk
    unsigned* prevp;            // [2][CH/32][CH] marking nets of the previous chunk
    unsigned* words;            // [2][2][CH] per net, which words of its pred and prevp columns are set
    unsigned* fullmask;         // [W]
    int* count;                 // [32*W]
    int* n_colors;              // [1]
    int* batch_of;              // [n] colour per order position
    int* rank;                  // [n] position inside its batch
    unsigned* solved;           // [1] chunks solved (persistent form)
    int* error;
    int* error_info;
};

__device__ __forceinline__ void batch_error(const BatchState& B, int code, int info) {
    if (atomicCAS(B.error, 0, code) == 0) *B.error_info = info;
}

// Cells of the segments [s0, s1) of `segs` with step `step`, visited by the 32
// lanes of a warp: lanes fetch 32 segment endpoints per memory round trip and
// broadcast them by shuffle.  f(cell, k, cnt) gets each cell with its index
// k < cnt inside the segment; done(cnt) runs on every lane after a segment.
template <class F, class D>
__device__ __forceinline__ void warp_segment_cells(const int* segs, int s0, int s1, int step, F f, D done) {
    const int lane = threadIdx.x & 31;
    for (int base = s0; base < s1; base += 32) {
        int a = 0, b = -1;
        if (base + lane < s1) { a = segs[2 * (base + lane)]; b = segs[2 * (base + lane) + 1]; }
        const int m = min(32, s1 - base);
        for (int q = 0; q < m; ++q) {
            const int aq = __shfl_sync(0xffffffffu, a, q), bq = __shfl_sync(0xffffffffu, b, q);
            if (bq < aq) continue;
            const int cnt = (bq - aq) / step + 1;
            for (int k = lane; k < cnt; k += 32) f(aq + k * step, k, cnt);
            done(cnt);
        }
    }
}

// The (up to) four cells a query point marks: left, below, itself, right.
__device__ __forceinline__ bool point_mark(const BatchState& B, int p, int which, int* cell) {
    const int x = p / B.Y, y = p - x * B.Y;
    int cx = x, cy = y;
    if (which == 0) cx = x - 1;
    else if (which == 1) cy = y - 1;
    else if (which == 3) cx = x + 1;
    *cell = cx * B.Y + cy;
    return cx >= 0 && cx < B.X && cy >= 0;
}

// Warp per order position: number of marks and query points of its net.
__device__ __forceinline__ void flat_count(const BatchState& B, int p) {
    const int lane = threadIdx.x & 31;
    const int id = B.order[p];
    long long marks = 0;
    warp_segment_cells(B.hsegs, B.hseg_off[id], B.hseg_off[id + 1], B.sparsity * B.Y, [](int, int, int) {},
                       [&](int cnt) { marks += cnt; });
    warp_segment_cells(B.vsegs, B.vseg_off[id], B.vseg_off[id + 1], B.sparsity, [](int, int, int) {},
                       [&](int cnt) { marks += cnt; });
    const int p0 = B.point_off[id], np = B.point_off[id + 1] - p0;
    int own = 0;
    for (int k = lane; k < 4 * np; k += 32) {
        int cell;
        own += point_mark(B, B.points[p0 + k / 4], k & 3, &cell) ? 1 : 0;
    }
    for (int o = 16; o; o >>= 1) own += __shfl_xor_sync(0xffffffffu, own, o);
    if (lane == 0) {
        B.mark_off[p] = marks + own;
        B.pt_off[p] = np;
    }
}

// Warp per order position: writes its net's marks and query points at the
// (scanned) offsets.
__device__ __forceinline__ void flat_fill(const BatchState& B, int p) {
    const int lane = threadIdx.x & 31;
    const int id = B.order[p];
    // Position inside a chunk of kChunkMax; reduced mod CH where read.
    const unsigned short jj = static_cast<unsigned short>(p % kChunkMax);
    long long o = B.mark_off[p];
    auto put = [&](int cell, int k, int) {
        B.mark_cell[o + k] = static_cast<unsigned>(cell);
        B.mark_jj[o + k] = jj;
    };
    auto advance = [&](int cnt) { o += cnt; };
    warp_segment_cells(B.hsegs, B.hseg_off[id], B.hseg_off[id + 1], B.sparsity * B.Y, put, advance);
    warp_segment_cells(B.vsegs, B.vseg_off[id], B.vseg_off[id + 1], B.sparsity, put, advance);
    const int p0 = B.point_off[id], np = B.point_off[id + 1] - p0;
    for (int base = 0; base < 4 * np; base += 32) {
        const int k = base + lane;
        int cell = 0;
        const bool ok = k < 4 * np && point_mark(B, B.points[p0 + k / 4], k & 3, &cell);
        const unsigned ball = __ballot_sync(0xffffffffu, ok);
        if (ok) {
            const long long at = o + __popc(ball & ((1u << lane) - 1u));
            B.mark_cell[at] = static_cast<unsigned>(cell);
            B.mark_jj[at] = jj;
        }
        o += __popc(ball);
    }
    const long long q = B.pt_off[p];
    for (int k = lane; k < np; k += 32) {
        B.pt_cell[q + k] = static_cast<unsigned>(B.points[p0 + k]);
        B.pt_jj[q + k] = jj;
    }
}

constexpr int kLocalMasks = 5;
__device__ __forceinline__ unsigned* chunk_mask(const BatchState& B, int chunk) { return B.localmask[chunk % kLocalMasks]; }
// A cell's record is a few bits in 128 bytes (a chunk marks a cell a handful of
// times); one word per cell says which of its words to read or to clear.
__device__ __forceinline__ unsigned* chunk_set(const BatchState& B, int chunk) { return B.localset[chunk % kLocalMasks]; }

// Query-point bits of the chunk at s: bit (chunk % 32) of every query point
// cell of the chunk is set (set) or cleared.
template <int CH>
__device__ __forceinline__ void batch_point_bits(const BatchState& B, int s, bool set, long long t, long long nt) {
    const int m = min(CH, B.n - s);
    const unsigned bit = 1u << ((s / CH) & 31);
    const long long a = B.pt_off[s], b = B.pt_off[s + m];
    for (long long k = a + t; k < b; k += nt) {
        unsigned* w = B.ptchunk + __ldg(B.pt_cell + k);
        if (set) red_or(w, bit);
        else asm volatile("red.relaxed.gpu.global.and.b32 [%0], %1;" ::"l"(w), "r"(~bit) : "memory");
    }
}

// Step 1: the chunk at order position s rasters its marks.  Only a cell that
// is a query point of this chunk or of the `ahead` chunks after it is ever
// read back, so the raster keeps the marks whose cell has one of those
// query-point bits; the bits live in a 4-byte-per-cell array that stays in L2,
// the chunk-local masks do not.  Threads t of nt.
template <int CH>
__device__ __forceinline__ void batch_raster(const BatchState& B, int s, int ahead, long long t, long long nt) {
    const int m = min(CH, B.n - s), chunk = s / CH;
    unsigned want = 0u;
    for (int a = 0; a <= ahead; ++a) want |= 1u << ((chunk + a) & 31);
    unsigned *lm = chunk_mask(B, chunk), *ls = chunk_set(B, chunk);
    const long long a = B.mark_off[s], b = B.mark_off[s + m];
    // Four marks per thread and pass, every load of a pass issued first.
    for (long long k0 = a + t; k0 < b; k0 += 4 * nt) {
        unsigned q[4], bits[4];
        int jj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long k = k0 + u * nt;
            q[u] = k < b ? __ldg(B.mark_cell + k) : 0u;
            jj[u] = k < b ? (__ldg(B.mark_jj + k) & (CH - 1)) : -1;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) bits[u] = jj[u] >= 0 ? __ldcg(B.ptchunk + q[u]) : 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (bits[u] & want) {
                red_or(lm + size_t(q[u]) * (CH / 32) + (jj[u] >> 5), 1u << (jj[u] & 31));
                red_or(ls + q[u], 1u << (jj[u] >> 5));
            }
    }
}

// The chunk-local mask of the chunk at s is nonzero only at query points of
// this chunk and the `ahead` chunks after it: zero those cells' words.
template <int CH>
__device__ __forceinline__ void batch_clear(const BatchState& B, int s, int ahead, long long t, long long nt) {
    unsigned *lm = chunk_mask(B, s / CH), *ls = chunk_set(B, s / CH);
    const long long a = B.pt_off[s];
    const long long b = B.pt_off[min(s + (ahead + 1) * CH, B.n)];
    for (long long k = a + t; k < b; k += nt) {
        const unsigned q = __ldg(B.pt_cell + k);
        unsigned set = __ldcg(ls + q);  // several points may share the cell: whoever sees a set bit clears its word
        if (!set) continue;
        for (; set; set &= set - 1) lm[size_t(q) * (CH / 32) + __ffs(set) - 1] = 0u;
        ls[q] = 0u;
    }
}

// Step 2: per query point, OR into the net's columns the cell's colours, the
// earlier nets' bits of this chunk and, with lookback >= 1, the bits of the
// previous chunk's nets (resolved by the solver, which knows their colours);
// with lookback 2 also the colours of the nets two chunks back that mark the
// cell (that chunk is solved, its colours published or being published).
// An item is four colour words or one chunk's record at a point; of a record
// only the words its set word names are read (with whole records, 26 items a
// point at 8 colour words instead of 5, the gather was the longest task of a
// round).  Consecutive lanes take the items of one point.
template <int CH>
__device__ __forceinline__ void batch_gather(const BatchState& B, int s, int lookback, long long t, long long nt) {
    const int chunk = s / CH, m = min(CH, B.n - s), W = B.W;
    unsigned* F = B.fmask + size_t(chunk & 1) * W * CH;
    unsigned* P = B.pred + size_t(chunk & 1) * (CH / 32) * CH;
    unsigned* Q = B.prevp + size_t(chunk & 1) * (CH / 32) * CH;
    unsigned* words = B.words + size_t(chunk & 1) * 2 * CH;
    const int gw = W / 4, per = gw + 1 + lookback, shift = 32 - __clz(per - 1);  // 2^shift lanes a point
    const long long a = B.pt_off[s], b = B.pt_off[s + m];
    const long long items = (b - a) << shift;
    const size_t XY = size_t(B.X) * B.Y;
    for (long long k = t; k < items; k += nt) {
        const int g = int(k) & ((1 << shift) - 1);
        if (g >= per) continue;
        const long long pi = a + (k >> shift);
        const unsigned q = __ldg(B.pt_cell + pi);
        const int jj = __ldg(B.pt_jj + pi) & (CH - 1);
        if (g < gw) {
            unsigned v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = __ldcg(B.cellmask + (4 * g + u) * XY + q);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (v[u]) red_or(F + size_t(4 * g + u) * CH + jj, v[u]);
            continue;
        }
        const int back = g - gw;  // the record of chunk - back
        unsigned set = __ldcg(chunk_set(B, chunk - back) + q);
        if (back == 0) set &= (2u << (jj >> 5)) - 1u;  // words of earlier nets
        if (!set) continue;
        const unsigned* rec = chunk_mask(B, chunk - back) + size_t(q) * (CH / 32);
        unsigned found = 0u;
        for (; set; set &= set - 1) {
            const int w = __ffs(set) - 1;
            unsigned bits = __ldcg(rec + w);
            if (back == 0 && w == (jj >> 5)) bits &= (1u << (jj & 31)) - 1u;  // earlier nets of the own word
            if (!bits) continue;
            if (back < 2) {
                found |= 1u << w;
                red_or((back ? Q : P) + size_t(w) * CH + jj, bits);
            } else {
                const int* col2 = B.batch_of + size_t(chunk - 2) * CH + w * 32;
                for (; bits; bits &= bits - 1) {
                    const int c = __ldcg(col2 + __ffs(bits) - 1);
                    red_or(F + size_t(c >> 5) * CH + jj, 1u << (c & 31));
                }
            }
        }
        if (found) red_or(words + (back ? CH : 0) + jj, found);
    }
}

// Step 4: the chunk at s publishes its colours.
template <int CH>
__device__ __forceinline__ void batch_publish(const BatchState& B, int s, long long t, long long nt) {
    const int m = min(CH, B.n - s);
    const long long a = B.mark_off[s], b = B.mark_off[s + m];
    // Four marks per thread and pass, every load of a pass issued first.
    for (long long k0 = a + t; k0 < b; k0 += 4 * nt) {
        unsigned q[4];
        int jj[4], c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long k = k0 + u * nt;
            q[u] = k < b ? __ldg(B.mark_cell + k) : 0u;
            jj[u] = k < b ? (__ldg(B.mark_jj + k) & (CH - 1)) : -1;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = jj[u] >= 0 ? __ldcg(B.batch_of + s + jj[u]) : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (jj[u] >= 0) red_or(B.cellmask + size_t(c[u] >> 5) * B.X * B.Y + q[u], 1u << (c[u] & 31));
    }
}

// Shared memory of the solving CTA (kept across chunks in the persistent form).
struct SolveSmem {
    unsigned* U;     // [W][CH] colours a net may not take (published, full, previous chunk)
    unsigned* P;     // [(CH / 32)][CH] predecessor bits
    int* col;        // [CH] colour of each net of the chunk
    int* colp;       // [CH] colours of the previous chunk
    int* cnt;        // [32W] nets per colour so far
    int* wh;         // [CH/32][32W] per-warp colour counts (zero between uses), or
                     // for W > kWarpCountWords a [32W] running count
    bool per_warp;   // wh holds per-warp counts
    unsigned* full;  // [W] colours whose batch is full
};

// Up to this many colour words the ranks use per-warp colour counts (three
// barriers); beyond it, warps add their counts in turn (one barrier per warp).
constexpr int kWarpCountWords = 32;

// Shared memory a solving CTA may use (the per-warp colour counts are dropped
// for the running count when they do not fit).
constexpr size_t kSolveSmemLimit = 220 * 1024;
template <int CH>
__host__ __device__ __forceinline__ size_t solve_smem_base(int W) {
    const size_t C = 32 * size_t(W);
    return size_t(CH) * W * 4 + size_t(CH) * (CH / 32) * 4 + 2 * size_t(CH) * 4 + C * 4 + size_t(W) * 4;
}
template <int CH>
__host__ __device__ __forceinline__ bool solve_per_warp(int W) {
    return W <= kWarpCountWords && solve_smem_base<CH>(W) + (CH / 32) * 32 * size_t(W) * 4 <= kSolveSmemLimit;
}
template <int CH>
__host__ __device__ __forceinline__ size_t solve_smem_bytes(int W) {
    const size_t C = 32 * size_t(W);
    const size_t wh = solve_per_warp<CH>(W) ? (CH / 32) * C : C;
    return size_t(CH) * W * 4 + size_t(CH) * (CH / 32) * 4 + 2 * size_t(CH) * 4 + C * 4 + wh * 4 +
           size_t(W) * 4;
}

template <int CH>
__device__ __forceinline__ SolveSmem solve_smem(unsigned* base, int W) {
    const int C = 32 * W;
    SolveSmem S;
    S.U = base;
    S.P = S.U + size_t(CH) * W;
    S.col = reinterpret_cast<int*>(S.P + size_t(CH) * (CH / 32));
    S.colp = S.col + CH;
    S.cnt = S.colp + CH;
    S.wh = S.cnt + C;
    S.per_warp = solve_per_warp<CH>(W);
    S.full = reinterpret_cast<unsigned*>(S.wh + (S.per_warp ? (CH / 32) * C : C));
    return S;
}

// The smallest colour c >= c0 net `tid` may take: not in U, not held by a
// predecessor (pmask: which predecessor words are nonzero).  C if none.
// Word by word from c0's: the word's forbidden bits are U's plus the colours
// of the predecessors that fall in it (one pass over the predecessors per
// word, whatever the number of colours the net has to skip).
template <int CH>
__device__ __forceinline__ int first_fit(const SolveSmem& S, int tid, int W, unsigned pmask, int c0) {
    for (int w = c0 >> 5; w < W; ++w) {
        unsigned used = S.U[w * CH + tid];
        if (w == (c0 >> 5)) used |= (1u << (c0 & 31)) - 1u;
        if (used == 0xffffffffu) continue;
        for (unsigned pm = pmask; pm; pm &= pm - 1) {
            const int pw = __ffs(pm) - 1;
            unsigned bits = S.P[pw * CH + tid];
            while (bits) {
                const int ci = S.col[pw * 32 + __ffs(bits) - 1];
                bits &= bits - 1;
                if ((ci >> 5) == w) used |= 1u << (ci & 31);  // ci = -1 (not yet coloured) is in no word
            }
        }
        if (used != 0xffffffffu) return w * 32 + __ffs(~used) - 1;
    }
    return 32 * W;
}

// The solve runs on threads 0..CH-1 of its CTA and synchronises them
// with named barrier 1 (the CTA may hold more threads, which do not take part).
template <int CH>
__device__ __forceinline__ void solve_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CH) : "memory"); }
template <int CH>
__device__ __forceinline__ bool solve_sync_or(bool v) {
    int r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.s32 %0, 1, 0, q;\n}"
        : "=r"(r) : "r"(int(v)), "n"(CH) : "memory");
    return r != 0;
}

// First-fit of the chunk's nets from `fixed` on, warp after warp (32 nets in
// order): a warp settles its nets by sweeps among themselves once every earlier
// warp is final, and after a barrier the later warps add its colours to those
// their nets may not take.  Each predecessor is looked at once, where a sweep
// over the whole chunk looks at all of them again: for chunks whose nets depend
// on one another in long chains (small grids).  For W == 8: a thread holds the
// colours its net may not take in registers, twice over, and the CTA's 1024
// threads have 64 registers each; designs that need more than 256 colours keep
// the sweeps.  Leaves the colours in S.col; false if a net finds none.
template <int CH>
__device__ __forceinline__ bool colours_in_order(const SolveSmem& S, int m, int fixed, unsigned pmask) {
    constexpr int W = 8;
    const int tid = threadIdx.x, warp = tid >> 5;
    unsigned no[W];
#pragma unroll
    for (int w = 0; w < W; ++w) no[w] = tid < m ? S.U[w * CH + tid] : 0u;
    const bool open = tid < m && tid >= fixed;
    bool fits = true;
    for (int k = 0; 32 * k < m; ++k) {
        const unsigned preds = tid < m && ((pmask >> k) & 1u) ? S.P[k * CH + tid] : 0u;
        if (warp == k) {
            int mine = tid < m ? (open ? -1 : S.col[tid]) : -1;
            if (tid < m) S.col[tid] = mine;
            while (true) {
                __syncwarp();
                int next = mine;
                if (open) {
                    unsigned used[W];
#pragma unroll
                    for (int w = 0; w < W; ++w) used[w] = no[w];
                    for (unsigned b = preds; b; b &= b - 1) {
                        const int c = S.col[32 * k + __ffs(b) - 1];  // -1 (not yet coloured) is in no word
#pragma unroll
                        for (int w = 0; w < W; ++w) used[w] |= (c >> 5) == w ? 1u << (c & 31) : 0u;
                    }
                    next = 32 * W;
#pragma unroll
                    for (int w = W - 1; w >= 0; --w)
                        if (used[w] != 0xffffffffu) next = 32 * w + __ffs(~used[w]) - 1;
                    fits = next < 32 * W;
                    next = min(next, 32 * W - 1);
                }
                const bool again = __any_sync(0xffffffffu, next != mine);
                if (tid < m) S.col[tid] = next;
                mine = next;
                if (!again) break;
            }
        }
        solve_sync<CH>();
        if (warp > k)
            for (unsigned b = preds; b; b &= b - 1) {
                const int c = S.col[32 * k + __ffs(b) - 1];
#pragma unroll
                for (int w = 0; w < W; ++w) no[w] |= (c >> 5) == w ? 1u << (c & 31) : 0u;
            }
    }
    return fits;
}
// Sweeps over the whole chunk before it is coloured in order: most chunks of
// large designs settle in two or three (0.5 us each at 3 predecessors a net);
// in order a chunk takes about 60 us whatever its chains (64x64x5: 86 against 106).
constexpr int kSweeps = 6;

// Step 3 (threads 0..CH-1 of a CTA): first-fit of the chunk at order
// position s.  S.cnt and S.full hold the state of the chunks before it;
// with `lookback`, S.colp holds the previous chunk's colours.  The chunk's
// tables are read once and cleared for reuse by chunk s + 2 * CH.
// Returns false on colour overflow (kELimit recorded).
template <int CH>
__device__ __forceinline__ bool batch_solve(const BatchState& B, int s, bool lookback, const SolveSmem& S) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = s / CH, m = min(CH, B.n - s);
    const int W = B.W, C = 32 * W;
    unsigned* Fg = B.fmask + size_t(chunk & 1) * W * CH;
    unsigned* Pg = B.pred + size_t(chunk & 1) * (CH / 32) * CH;
    unsigned* Qg = B.prevp + size_t(chunk & 1) * (CH / 32) * CH;
    __shared__ int first_bad, overflow;
    if (tid == 0) overflow = 0;
    unsigned* set = B.words + size_t(chunk & 1) * 2 * CH;
    unsigned pmask = 0, qmask = 0;
    int c0 = 0;  // first colour not in U
    if (tid < m) {
        pmask = __ldcg(set + tid);
        if (lookback) qmask = __ldcg(set + CH + tid);
        // Every load of a group is issued before its stores, so the round
        // trips overlap (the tables were just written by other SMs).
        for (int w0 = 0; w0 < W; w0 += 8) {
            unsigned v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = w0 + k < W ? __ldcg(Fg + size_t(w0 + k) * CH + tid) : 0u;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (w0 + k >= W) break;
                if (v[k]) Fg[size_t(w0 + k) * CH + tid] = 0u;
                S.U[(w0 + k) * CH + tid] = v[k] | S.full[w0 + k];
            }
        }
        // Only the words the gather has set are read (a net has a few earlier
        // neighbours, in a few words of the 32), four at a time.
        auto words = [&](unsigned left, unsigned* table, auto use) {
            while (left) {
                int w[4];
                unsigned v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    w[k] = left ? __ffs(left) - 1 : -1;
                    left &= left - 1;  // 0 stays 0
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = w[k] >= 0 ? __ldcg(table + w[k] * CH + tid) : 0u;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (w[k] >= 0) {
                        table[w[k] * CH + tid] = 0u;
                        use(w[k], v[k]);
                    }
            }
        };
        if (pmask) set[tid] = 0u;
        words(pmask, Pg, [&](int w, unsigned bits) { S.P[w * CH + tid] = bits; });
        if (lookback) {
            if (qmask) set[CH + tid] = 0u;
            words(qmask, Qg, [&](int w, unsigned bits) {
                while (bits) {
                    const int c = S.colp[w * 32 + __ffs(bits) - 1];
                    bits &= bits - 1;
                    S.U[(c >> 5) * CH + tid] |= 1u << (c & 31);
                }
            });
        }
        c0 = first_fit<CH>(S, tid, W, 0u, 0);
    }
    // The first sweep, in which no net has a colour yet, gives every net c0.
    S.col[tid] = tid < m ? c0 : -1;
    solve_sync<CH>();
    int fixed = 0;  // nets below `fixed` are final
    int rank = 0;
    __shared__ int tight;
    while (true) {
        // Jacobi sweeps until the colouring is a fixed point.  A net may find no
        // colour on the way, while its predecessors' are provisional: only the
        // settled colouring says whether the colours suffice.
        bool none = false;
        for (int sweep = 0;; ++sweep) {
            if (sweep == kSweeps && W == 8) {
                none = !colours_in_order<CH>(S, m, fixed, pmask);
                break;
            }
            int mine = tid < m ? S.col[tid] : -1;
            if (tid < m && tid >= fixed) {
                mine = pmask ? first_fit<CH>(S, tid, W, pmask, c0) : c0;
                none = mine >= C;
                mine = min(mine, C - 1);
            }
            solve_sync<CH>();
            const bool changed = tid < m && S.col[tid] != mine;
            if (tid < m) S.col[tid] = mine;
            if (!solve_sync_or<CH>(changed)) break;
        }
        if (none) overflow = 1;
        // While no batch reaches its limit, no position inside a batch is
        // needed here (the rank pass after the run assigns them): the chunk's
        // nets are added to the per-colour totals.  Else the positions, in
        // chunk order -- colour counts of the earlier warps plus the rank inside
        // the own warp -- find the first net that does not fit.
        if (tid == 0) { first_bad = m; tight = 0; }
        const int c = tid < m ? S.col[tid] : -1 - lane;  // distinct dummies for idle lanes
        if (tid < m) atomicAdd(S.cnt + c, 1);
        solve_sync<CH>();
        if (overflow) break;
        if (tid < m && S.cnt[c] > B.limit) tight = 1;
        solve_sync<CH>();
        const bool counted = !tight;
        if (!counted) {
            if (tid < m) atomicSub(S.cnt + c, 1);
            const unsigned peers = __match_any_sync(0xffffffffu, c);
            const bool leader = tid < m && lane == __ffs(peers) - 1;
            const int within = __popc(peers & ((1u << lane) - 1u));
            if (S.per_warp && leader) S.wh[warp * C + c] = __popc(peers);
            solve_sync<CH>();
            if (S.per_warp) {
                if (tid < m) {
                    int r = S.cnt[c] + within;
                    for (int w = 0; w < warp; ++w) r += S.wh[w * C + c];
                    rank = r;
                    if (r >= B.limit) atomicMin(&first_bad, tid);
                }
                solve_sync<CH>();
                if (leader) S.wh[warp * C + c] = 0;
            } else {
                for (int k = tid; k < C; k += CH) S.wh[k] = S.cnt[k];
                solve_sync<CH>();
                for (int w = 0; w < (m + 31) / 32; ++w) {
                    if (warp == w && tid < m) {
                        rank = S.wh[c] + within;
                        if (leader) S.wh[c] += __popc(peers);
                        if (rank >= B.limit) atomicMin(&first_bad, tid);
                    }
                    solve_sync<CH>();
                }
            }
        }
        const int bad = first_bad;
        if (bad >= m) {
            if (!counted && tid < m) atomicAdd(S.cnt + c, 1);
            break;
        }
        // Net `bad` finds its colour full; so does every later net.
        const int fc = S.col[bad];
        if (tid == 0) S.full[fc >> 5] |= 1u << (fc & 31);
        if (tid >= bad && tid < m) {
            S.U[(fc >> 5) * CH + tid] |= 1u << (fc & 31);
            c0 = first_fit<CH>(S, tid, W, 0u, c0);
        }
        fixed = bad;
        solve_sync<CH>();
    }
    if (overflow) {
        if (tid == 0) batch_error(B, kELimit, s);
        return false;
    }
    int top = 0;
    if (tid < m) {
        const int c = S.col[tid];
        B.batch_of[s + tid] = c;
        S.colp[tid] = c;
        top = c + 1;
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0 && top) atomicMax(B.n_colors, top);
    solve_sync<CH>();
    return true;
}

}  // namespace grb
