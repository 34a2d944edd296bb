// flt.cuh -- FLT stage: mid-edge layer-change tables, DAG solve and trace.
//
// Semantics of the reference's FLT execution (flt_cost.cuh:25-130,
// flt_block.cuh:6-355).  Each net carries a DAG whose nodes are 3-D grid
// points (layer 9 = no pin layer) and whose edges connect a child node to one
// of its parents' child slots; alternative nodes compete for a slot.  Solve
// runs from the deepest level up: a node combines, per layer, the cheapest
// candidate of every child slot plus its via stack, then offers every parent
// slot a packed (fp32 cost, node*100 + choice) key per target layer, kept by
// a 64-bit atomicMin.  Trace runs from the root down and emits the chosen
// wires (straight, or split at the best sampled mid-edge layer change) and
// each node's via stack.
//
// B200 form: the layer-change tables of all the batch's edges are one
// grid-wide pass, a warp per edge (the reference launches a thread per (edge,
// from-layer)).  Then a net is walked by one warp, or by a CTA where its levels
// are wide; its topology, candidate keys and choices sit in shared memory.  A
// warp solves three nodes of a level at once, a lane per (node, layer): lane
// `low` walks its range tops, a column minimum per top picks the range, and a
// lane per target layer offers the node to each parent slot (the reference and
// the earlier form here give a node to one thread, which walks the ranges of
// all layers in thread-local arrays).  A batch lasts as long as its largest
// net's levels one after the other, so it is a level's latency that counts:
// 2,400 nets in 35 batches at 320x320x10 took 18 ms of solve and trace by a
// thread per node, 4.6 ms in this form.
// Node numbering is net-local: candidates for a slot always belong to one
// net, so the batch-global numbering of the reference orders them the same.
// Segments are appended in level order, ascending node index within a level,
// each node's wires before its via stack (the reference appends with atomics,
// so only its segment multiset is defined).
#pragma once
#include "commit.cuh"
#include "common.cuh"

namespace grb {

constexpr int kFltLayers = 10;                                  // MAX_LAYER, flt_cost.cuh:14
constexpr unsigned long long kFltInit = 7208259049189261824ull; // init_cost_with_road, flt_cost.cuh:48
constexpr int kFltStraight = 82;                                // flt_block.cuh:109
constexpr int kFltMaxChildren = 6;                              // flt_block.cuh:31-32

struct Flt {
    // per net id
    const int* node_off;     // [n+1] global node index of the net's node 0
    const int* edge_off;     // [n+1] global edge index of the net's edge 0
    const int* lvl_off;      // [n+1] into level: the net's depth levels
    const long long* route2_off;  // [n+1] phase-two route words
    // per depth level: first position in `order` (net-local), plus one end
    // entry per net at lvl_off[id+1]-1 ... stored as level[lvl_off[id] + d]
    const int* level;        // [sum over nets of depths+1]
    // per node (global index)
    const int* coord;        // l*X*Y + x*Y + y
    const int* children;     // child slots
    const int* child_off;    // global exclusive prefix of children
    const int* pend;         // net-local cumulative parent-edge count
    const int* order;        // net-local node indices by (depth, index)
    // per edge (global index)
    const int* eparent;      // net-local parent node
    const int* eslot;        // source slot: child node (net-local) * 10 + slot index at the parent
    // workspace
    double* costs;                 // [nodes*10]
    unsigned long long* packed;    // [children*10]
    unsigned long long* best;      // [children*10]
    int* lo;                       // [nodes] chosen layer (1-based), -1 unused
    double* ce;                    // [edges*81] layer-change cost
    int* bc;                       // [edges*81] layer-change position
    int* routes2;
    // per plan position: first edge slot (exclusive prefix of the plan's
    // edges, [plan+1]); per edge slot: its plan position
    const int* eprefix;
    const int* emap;
    // per plan position, batch by batch: the batch's positions with its wide
    // nets (those a CTA takes, grb_set_flt_block_width) first; per batch: its
    // wide nets
    const int* border;
    const int* nwide;
};

__device__ __forceinline__ double flt_wire(const Tables& T, int l, int xmin, int xmax, int ymin, int ymax) {
    // prefix_scan.cuh:10-40 (wire_segment_cost)
    return T.presum[slot_index(T, l, xmax, ymax)] - T.presum[slot_index(T, l, xmin, ymin)];
}

// flt_cost.cuh:25-46.
__device__ __forceinline__ unsigned long long flt_pack(float cost, int id) {
    int i = __float_as_int(cost);
    i = i >= 0 ? i : i ^ 0x7FFFFFFF;
    return (static_cast<unsigned long long>(static_cast<unsigned>(i)) << 32) | static_cast<unsigned>(id);
}
__device__ __forceinline__ double flt_cost(unsigned long long p) {
    int i = static_cast<int>(p >> 32);
    i = i >= 0 ? i : i ^ 0x7FFFFFFF;
    return static_cast<double>(__int_as_float(i));
}

// precompute_cost_edge (flt_cost.cuh:50-130) for every (from-layer,
// to-layer) entry of global edge `e`, one warp.  Entries the solve never
// reads -- an edge with a bend or of Manhattan length <= 4 (only straight
// wires are offered there), a from-layer across the edge's direction, a
// to-layer of the other parity -- are INF with position -1.  Otherwise the
// entry is the cheapest layer change over the sampled positions (every
// dd-th position strictly inside the edge, dd = distance / min(distance,
// 20)): the via stack between the layers there plus the wire from each end
// to it on its layer, the via costs added from the lower layer up and the two
// wires summed before they are added, the first minimum in increasing
// position kept.  Lanes take the positions (32 at a time) and evaluate every
// entry there; the first minimum comes from a warp reduction of (cost,
// position) pairs.
__device__ __forceinline__ void flt_edge_warp(const Tables& T, const Flt& F, int nb, int e, int lane) {
    const int to = nb + F.eparent[e], from = nb + F.eslot[e] / 10;
    const int ct = F.coord[to], cf = F.coord[from];
    const int tox = ct / T.Y % T.X, toy = ct % T.Y, fromx = cf / T.Y % T.X, fromy = cf % T.Y;
    double* ce = F.ce + size_t(e) * 81;
    int* bc = F.bc + size_t(e) * 81;
    for (int k = lane; k < 81; k += 32) { ce[k] = kInf; bc[k] = -1; }
    const int distance = abs(tox - fromx) + abs(toy - fromy);
    const bool vertical = fromx == tox;
    if (distance <= 4 || (!vertical && fromy != toy)) return;
    __syncwarp();  // the fill above comes before the entries below
    const int dd = distance / min(distance, 20);
    const int start = vertical ? min(fromy, toy) : min(fromx, tox);
    const int end = vertical ? max(fromy, toy) : max(fromx, tox);
    const int ns = start + dd < end ? (end - 1 - (start + dd)) / dd + 1 : 0;  // sampled positions
    // Layers of the edge's direction (the only from- and to-layers with
    // finite entries): l0, l0 + 2, ...
    const int l0 = (vertical ? (T.DIR ^ 1) : T.DIR) & 1;
    constexpr int KV = (kFltLayers + 1) / 2;
    for (int fi = 0; fi < KV; ++fi) {
        const int fl = l0 + 2 * fi;
        if (fl >= 9 || fl >= T.L) break;
        double bv[KV];
        int bp[KV];
#pragma unroll
        for (int ti = 0; ti < KV; ++ti) { bv[ti] = kInf; bp[ti] = -1; }
        const double pF = T.presum[slot_index(T, fl, fromx, fromy)];
        for (int base = 0; base < ns; base += 32) {
            const int s = base + lane;
            if (s < ns) {
                const int sp = start + dd + s * dd;
                const int sx = vertical ? fromx : sp, sy = vertical ? sp : fromy;
                float vc[kFltLayers];
#pragma unroll
                for (int ll = 0; ll < kFltLayers - 1; ++ll) vc[ll] = ll < T.L ? T.vcost[slot_index(T, ll, sx, sy)] : 0.f;
                const double pf = T.presum[slot_index(T, fl, sx, sy)];
                const double wf = vertical ? (sy > fromy ? pf - pF : pF - pf) : (sx > fromx ? pf - pF : pF - pf);
#pragma unroll
                for (int ti = 0; ti < KV; ++ti) {
                    const int tl = l0 + 2 * ti;
                    if (tl >= 9 || tl >= T.L) continue;
                    const double pT = T.presum[slot_index(T, tl, tox, toy)];
                    const double pt = T.presum[slot_index(T, tl, vertical ? tox : sp, vertical ? sp : toy)];
                    const double wt = vertical ? (sy > toy ? pt - pT : pT - pt) : (sx > tox ? pt - pT : pT - pt);
                    const int lo = min(fl, tl), hi = max(fl, tl);
                    double via = 0;
#pragma unroll
                    for (int ll = 0; ll < kFltLayers - 1; ++ll)
                        if (ll >= lo && ll < hi) via += vc[ll];  // in increasing order, as the reference adds
                    double c = via;
                    c += (wf + wt);
                    if (c < bv[ti]) { bv[ti] = c; bp[ti] = sp; }
                }
            }
        }
#pragma unroll
        for (int ti = 0; ti < KV; ++ti) {
            const int tl = l0 + 2 * ti;
            if (tl >= 9 || tl >= T.L) continue;
            double v = bv[ti];
            int p = bp[ti];
            for (int o = 16; o; o >>= 1) {
                const double ov = __shfl_down_sync(0xffffffffu, v, o);
                const int op = __shfl_down_sync(0xffffffffu, p, o);
                if (op >= 0 && (p < 0 || ov < v || (ov == v && op < p))) { v = ov; p = op; }
            }
            if (lane == 0 && p >= 0) { ce[fl * 9 + tl] = v; bc[fl * 9 + tl] = p; }
        }
    }
}

// The layer-change tables of every edge of batch b, one warp per edge over
// warps w, w + nw, ...: the reference's precompute_cost_edge launch over the
// batch's edges (flt.cuh:152).  Edge slot s of the plan belongs to plan
// position emap[s]; eprefix[k] is the first slot of position k.
__device__ __forceinline__ void flt_edges_batch(const Tables& T, const Flt& F, const Plan& P, int b, long long w,
                                                long long nw, int lane) {
    const int lo = P.batch_off[b], hi = P.batch_off[b + 1];
    const long long s0 = F.eprefix[lo], items = static_cast<long long>(F.eprefix[hi]) - s0;
    for (long long q = w; q < items; q += nw) {
        const int s = static_cast<int>(s0 + q);
        const int k = F.emap[s];
        const int id = P.ids[k];
        flt_edge_warp(T, F, F.node_off[id], F.edge_off[id] + (s - F.eprefix[k]), lane);
    }
}

// One net as its warp or CTA walks it: topology, candidate keys, choices, in
// shared memory where they fit, else in HBM.
struct FltNet {
    int N, nb, eb;
    const int *coord, *children, *coff, *pend, *order;  // per node; coff: first child slot in packed / best
    const int *epar, *eslot;                            // per edge of the net
    unsigned long long *packed, *best;                  // [child slots][kFltLayers]
    int* lo;                                            // [N] chosen layer (1-based), -1 unused
};
constexpr int kFltArena = 10240;  // shared memory of a net's arrays, per warp
constexpr int kFltRow = kFltLayers - 1;  // layers 1..9: lanes of a slot
constexpr int kFltSlots = 3;             // nodes a warp solves at once
constexpr int kFltScratch = kFltSlots * kFltRow * kFltRow * 8 + 256;  // range costs and tops, per warp

// Sets up net `id` for threads t of nth (a warp, or a CTA), its arrays in
// `arena` when they fit `bytes`.  The caller synchronises before the next use.
__device__ __forceinline__ FltNet flt_open(const Flt& F, int id, char* arena, int bytes, int t, int nth) {
    FltNet W;
    W.nb = F.node_off[id];
    W.N = F.node_off[id + 1] - W.nb;
    W.eb = F.edge_off[id];
    const int E = F.edge_off[id + 1] - W.eb, N = W.N;
    W.coord = F.coord + W.nb;
    W.children = F.children + W.nb;
    W.coff = F.child_off + W.nb;
    W.pend = F.pend + W.nb;
    W.order = F.order + W.nb;
    W.epar = F.eparent + W.eb;
    W.eslot = F.eslot + W.eb;
    W.packed = F.packed;
    W.best = F.best;
    W.lo = F.lo + W.nb;
    if (N <= 0) return W;
    const int cb = W.coff[0], C = W.coff[N - 1] + W.children[N - 1] - cb;
    const long long need = 16ll * kFltLayers * C + 24ll * N + 8ll * E;
    if (need > bytes) {
        for (int k = t; k < C * kFltLayers; k += nth) W.packed[size_t(cb) * kFltLayers + k] = kFltInit;
        return W;
    }
    unsigned long long* packed = reinterpret_cast<unsigned long long*>(arena);
    int* p = reinterpret_cast<int*>(packed + 2 * size_t(C) * kFltLayers);
    int *coord = p, *children = p + N, *coff = p + 2 * N, *pend = p + 3 * N, *order = p + 4 * N, *lo = p + 5 * N,
        *epar = p + 6 * N, *eslot = epar + E;
    for (int k = t; k < C * kFltLayers; k += nth) packed[k] = kFltInit;
    for (int k = t; k < N; k += nth) {
        coord[k] = W.coord[k];
        children[k] = W.children[k];
        coff[k] = W.coff[k] - cb;
        pend[k] = W.pend[k];
        order[k] = W.order[k];
    }
    for (int k = t; k < E; k += nth) {
        epar[k] = W.epar[k];
        eslot[k] = W.eslot[k];
    }
    W.packed = packed;
    W.best = packed + size_t(C) * kFltLayers;
    W.coord = coord; W.children = children; W.coff = coff; W.pend = pend; W.order = order;
    W.epar = epar; W.eslot = eslot; W.lo = lo;
    return W;
}

// solve_flt_node (flt_block.cuh:6-142) for one node per slot (lane = slot * 9 +
// layer - 1; i < 0: none), by one warp.  `scratch`: kFltScratch bytes of the
// warp's shared memory.
//
// The sequential loops keep, per range top, the first strict minimum over the
// range bottoms in ascending order and, at one bottom, over the tops from it
// up: lane `low` forms its bottom's costs and their suffix minima (lowest top
// on ties), then lane `top` takes the first minimum over the bottoms.
__device__ __forceinline__ void flt_solve_group(const Tables& T, const Flt& F, const FltNet& W, int i, int lane,
                                                char* scratch) {
    constexpr unsigned kAll = 0xffffffffu;
    const int slot = min(lane / kFltRow, kFltSlots - 1), s0 = slot * kFltRow, li = lane - lane / kFltRow * kFltRow + 1;
    const bool on = lane < kFltSlots * kFltRow && i >= 0;
    const int ii = on ? i : 0;
    double* cs = reinterpret_cast<double*>(scratch) + s0 * kFltRow;
    unsigned char* hs = reinterpret_cast<unsigned char*>(scratch) + kFltSlots * kFltRow * kFltRow * 8 + s0 * kFltRow;
    int l0, x, y;
    cell_position(T, W.coord[ii], l0, x, y);
    const int flow = 1 + l0, fhigh = flow == kFltLayers ? 0 : flow, nc = on ? W.children[ii] : 0;
    const unsigned long long* keys = W.packed + size_t(W.coff[ii]) * kFltLayers;
    // Via cost below layer li (between routing layers li - 2 and li - 1).
    const float below = on && li >= 2 && li - 2 < T.L ? T.vcost[slot_index(T, li - 2, x, y)] : 0.f;
    {
        double mcc[kFltMaxChildren], via = 0;
#pragma unroll
        for (int c = 0; c < kFltMaxChildren; ++c) mcc[c] = kInf;
#pragma unroll 1
        for (int h = 1; h <= kFltRow; ++h) {
            const float v = __shfl_sync(kAll, below, s0 + h - 1);
            if (!on || h < li || li > flow) continue;
            if (h > li) via += v;
            double cost = via;
#pragma unroll
            for (int c = 0; c < kFltMaxChildren; ++c) {
                if (c >= nc) continue;
                const double cc = flt_cost(keys[c * kFltLayers + h]);
                if (cc < mcc[c]) mcc[c] = cc;
                cost += mcc[c];
            }
            cs[(li - 1) * kFltRow + h - 1] = h >= fhigh && cost < kInf && h < T.L + 1 ? cost : kInf;
        }
        double best = kInf;
        int top = 0;
#pragma unroll 1
        for (int h = on && li <= flow ? kFltRow : 0; h >= li; --h) {
            const double v = cs[(li - 1) * kFltRow + h - 1];
            if (v <= best) { best = v; top = h; }
            cs[(li - 1) * kFltRow + h - 1] = best;
            hs[(li - 1) * kFltRow + h - 1] = static_cast<unsigned char>(top);
        }
    }
    __syncwarp();
    double cst = kInf;
    int low = 0;
#pragma unroll 1
    for (int l = 1; l <= (on ? min(li, flow) : 0); ++l) {
        const double v = cs[(l - 1) * kFltRow + li - 1];
        if (v < cst) { cst = v; low = l; }
    }
    if (low) {
        // The cheapest candidate of every child slot inside the chosen range.
        const int top = hs[(low - 1) * kFltRow + li - 1];
        unsigned long long* chosen = W.best + size_t(W.coff[ii]) * kFltLayers;
#pragma unroll 1
        for (int c = 0; c < nc; ++c) {
            double m = kInf;
            unsigned long long bp = 0;
#pragma unroll 1
            for (int h = low; h <= top; ++h) {
                const unsigned long long pv = keys[c * kFltLayers + h];
                const double cc = flt_cost(pv);
                if (cc < m) { m = cc; bp = static_cast<unsigned long long>(static_cast<unsigned>(pv)) * kFltLayers + h; }
            }
            chosen[c * kFltLayers + li] = bp;
        }
    }
    const int pb = on && ii ? W.pend[ii - 1] : 0, pe = on ? W.pend[ii] : 0;
    if (on && pb == pe) {  // a root: its layer is chosen from its costs
        F.costs[size_t(W.nb + ii) * kFltLayers + li] = cst;
        if (li == 1) F.costs[size_t(W.nb + ii) * kFltLayers] = kInf;
    }
    // Offers to the parents' slots, lane = target layer; sources are the layers
    // of the edge's direction (all of the target's parity).
    for (int e = pb; __any_sync(kAll, e < pe); ++e) {
        const bool live = e < pe;
        const int par = live ? W.epar[e] : 0;
        int pl, px, py;
        cell_position(T, W.coord[par], pl, px, py);
        const bool ay = ((li & 1) ^ T.DIR) == 1;  // 1-based layer index
        const bool use = live && (ay ? y == py : x == px);
        const bool far = abs(x - px) + abs(y - py) > 4;
        double ce[(kFltRow + 1) / 2];
#pragma unroll
        for (int k = 0; k < (kFltRow + 1) / 2; ++k) {
            const int layer = ((li - 1) & 1) + 1 + 2 * k;
            ce[k] = use && far && layer != li && layer <= kFltRow
                        ? F.ce[size_t(W.eb + e) * 81 + (layer - 1) * 9 + li - 1] : kInf;
        }
        unsigned long long offer = kFltInit;
        if (use) {
            const double c2 = cst + flt_wire(T, li - 1, min(x, px), max(x, px), min(y, py), max(y, py));
            offer = min(offer, flt_pack(static_cast<float>(c2), ii * 100 + kFltStraight));
        }
#pragma unroll
        for (int k = 0; k < (kFltRow + 1) / 2; ++k) {
            const int layer = ((li - 1) & 1) + 1 + 2 * k;
            const double cb = __shfl_sync(kAll, cst, (s0 + min(layer, kFltRow) - 1) & 31);
            if (ce[k] < kInf)
                offer = min(offer, flt_pack(static_cast<float>(cb + ce[k]), ii * 100 + (layer - 1) * 9 + li - 1));
        }
        if (live && offer != kFltInit)
            atomicMin(W.packed + size_t(W.coff[par] + W.eslot[e] % 10) * kFltLayers + li, offer);
    }
    __syncwarp();
}

// trace_flt_node (flt_block.cuh:144-331) for net-local node `i`: sets lo[i]
// and writes up to 4 segments (8 words) into `w`; returns the word count.
__device__ __forceinline__ int flt_trace_node(const Tables& T, const Flt& F, const FltNet& W, int i, int* w) {
    int l, cx, cy;
    cell_position(T, W.coord[i], l, cx, cy);
    const int pb = i ? W.pend[i - 1] : 0, pe = W.pend[i];
    int n = 0;
    int me;
    if (pb == pe) {
        const double* costs = F.costs + size_t(W.nb + i) * kFltLayers;
        int ml = 0;
        double mc = costs[0];
        for (int layer = 1; layer < kFltLayers; ++layer) {
            const double v = costs[layer];
            if (v < mc) { mc = v; ml = layer; }
        }
        me = ml;
    } else {
        int par_layer = -1, par_idx = -1, par_edge = -1;
        me = -1;
        for (int e = pb; e < pe; ++e) {
            const int pn = W.epar[e];
            const int pl = W.lo[pn];
            if (pl <= 0) continue;
            par_idx = pn; par_edge = e; par_layer = pl;
            const unsigned long long path = W.best[size_t(W.coff[pn] + W.eslot[e] % 10) * kFltLayers + pl];
            const unsigned long long cidx = path / kFltLayers / 100, choice = (path / kFltLayers) % 100;
            if (cidx != static_cast<unsigned long long>(i)) { me = -1; continue; }
            me = choice == kFltStraight ? int(path % kFltLayers) : int(choice / 9 + 1);
            int pq, px, py;
            cell_position(T, W.coord[pn], pq, px, py);
            const bool vert = px == cx && cy != py, horz = py == cy && cx != px;
            if (vert || horz) {
                if (choice == kFltStraight) {
                    const int ll = me - 1;
                    if (vert) { w[n++] = cell_index(T, ll, px, min(py, cy)); w[n++] = cell_index(T, ll, px, max(py, cy)); }
                    else { w[n++] = cell_index(T, ll, min(px, cx), py); w[n++] = cell_index(T, ll, max(px, cx), py); }
                } else {
                    const int fl = int(choice / 9), tl = int(choice % 9);
                    const int cp = F.bc[size_t(W.eb + e) * 81 + fl * 9 + tl];
                    if (vert) {
                        w[n++] = cell_index(T, fl, cx, min(cy, cp)); w[n++] = cell_index(T, fl, cx, max(cy, cp));
                        w[n++] = cell_index(T, min(fl, tl), cx, cp); w[n++] = cell_index(T, max(fl, tl), cx, cp);
                        w[n++] = cell_index(T, tl, cx, min(py, cp)); w[n++] = cell_index(T, tl, cx, max(py, cp));
                    } else {
                        w[n++] = cell_index(T, fl, min(cx, cp), cy); w[n++] = cell_index(T, fl, max(cx, cp), cy);
                        w[n++] = cell_index(T, min(fl, tl), cp, cy); w[n++] = cell_index(T, max(fl, tl), cp, cy);
                        w[n++] = cell_index(T, tl, min(px, cp), cy); w[n++] = cell_index(T, tl, max(px, cp), cy);
                    }
                }
            }
            break;
        }
        if (par_layer == -1) { W.lo[i] = -1; return 0; }
        const unsigned long long path = W.best[size_t(W.coff[par_idx] + W.eslot[par_edge] % 10) * kFltLayers + par_layer];
        if (path / kFltLayers / 100 != static_cast<unsigned long long>(i)) { W.lo[i] = -1; return 0; }
    }
    W.lo[i] = me;
    int minl = l + 1, maxl = (l + 1) == kFltLayers ? 1 : minl;
    minl = min(minl, me);
    maxl = max(maxl, me);
    const int nc = W.children[i];
    for (int c = 0; c < nc; ++c) {
        const int lc = int(W.best[size_t(W.coff[i] + c) * kFltLayers + me] % kFltLayers);
        minl = min(lc, minl);
        maxl = max(lc, maxl);
    }
    if (minl < 1) return -1;  // no finite layer at the root
    if (minl < maxl) { w[n++] = cell_index(T, minl - 1, cx, cy); w[n++] = cell_index(T, maxl - 1, cx, cy); }
    return n;
}

// Route net `id` with one warp: solve, trace into the phase-two routes, then
// (if `commit`) its wire demand.  P2 is the phase-two view of the plan (routes
// = routes2).  All 32 lanes call with the same id; `smem`: the CTA's shared
// memory (the warps' arenas, then their scratch).
__device__ __forceinline__ void flt_net(const Tables& T, const Flt& F, const Plan& P2, int id, int stamp, int lane,
                                        bool commit, char* smem) {
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    char* scratch = smem + size_t(nw) * kFltArena + size_t(warp) * kFltScratch;
    const FltNet W = flt_open(F, id, smem + size_t(warp) * kFltArena, kFltArena, lane, 32);
    if (W.N <= 0) return;
    __syncwarp();
    const int* lev = F.level + F.lvl_off[id];
    const int nl = F.lvl_off[id + 1] - F.lvl_off[id] - 1;
    for (int d = nl - 1; d >= 0; --d) {
        const int end = lev[d + 1];
        for (int k = lev[d]; k < end; k += kFltSlots) {
            const int at = k + lane / kFltRow;
            flt_solve_group(T, F, W, at < end && lane < kFltSlots * kFltRow ? W.order[at] : -1, lane, scratch);
        }
    }
    int* r = F.routes2 + P2.route_off[id];
    const long long cap = P2.route_off[id + 1] - P2.route_off[id];
    long long count = 1;
    bool bad = false;
    for (int d = 0; d < nl; ++d) {
        for (int base = lev[d]; base < lev[d + 1]; base += 32) {
            int w[8];
            int n = 0;
            if (base + lane < lev[d + 1]) n = flt_trace_node(T, F, W, W.order[base + lane], w);
            if (__any_sync(0xffffffffu, n < 0)) { bad = true; n = max(n, 0); }
            int off = n;
            for (int s = 1; s < 32; s <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, off, s);
                if (lane >= s) off += v;
            }
            const int total = __shfl_sync(0xffffffffu, off, 31);
            off -= n;
            if (count + total <= cap)
                for (int k = 0; k < n; ++k) r[count + off + k] = w[k];
            else bad = true;
            count += total;
            __syncwarp();
        }
    }
    if (lane == 0) {
        if (bad) { set_error(T, kELimit, id); r[0] = 1; }
        else r[0] = int(count);
    }
    __syncwarp();
    if (commit && !bad) commit_net_wires(T, P2, id, stamp, 1, lane);
}

// Route net `id` with the whole CTA: flt_net for nets with wide DAG levels, a
// level's nodes dealt to the warps.  The words go out in the same order (level
// by level, ascending node index, each node's wires before its via stack): a
// block scan of the words per node replaces the warp scan.  All threads of the
// CTA call with the same id.
__device__ __forceinline__ void flt_net_block(const Tables& T, const Flt& F, const Plan& P2, int id, int stamp,
                                              bool commit, char* smem) {
    __shared__ int wsum[32];
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nth >> 5;
    char* scratch = smem + size_t(nw) * kFltArena + size_t(warp) * kFltScratch;
    const FltNet W = flt_open(F, id, smem, nw * kFltArena, tid, nth);
    if (W.N <= 0) return;
    __syncthreads();
    const int* lev = F.level + F.lvl_off[id];
    const int nl = F.lvl_off[id + 1] - F.lvl_off[id] - 1;
    for (int d = nl - 1; d >= 0; --d) {
        const int end = lev[d + 1];
        for (int k = lev[d] + kFltSlots * warp; k < end; k += kFltSlots * nw) {
            const int at = k + lane / kFltRow;
            flt_solve_group(T, F, W, at < end && lane < kFltSlots * kFltRow ? W.order[at] : -1, lane, scratch);
        }
        __syncthreads();
    }
    int* r = F.routes2 + P2.route_off[id];
    const long long cap = P2.route_off[id + 1] - P2.route_off[id];
    long long count = 1;
    bool bad = false;
    for (int d = 0; d < nl; ++d) {
        for (int base = lev[d]; base < lev[d + 1]; base += nth) {
            int w[8];
            int n = 0;
            if (base + tid < lev[d + 1]) n = flt_trace_node(T, F, W, W.order[base + tid], w);
            const bool neg = n < 0;
            n = max(n, 0);
            int off = n;  // inclusive scan inside the warp
            for (int s = 1; s < 32; s <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, off, s);
                if (lane >= s) off += v;
            }
            if (lane == 31) wsum[warp] = off;
            if (__syncthreads_or(neg)) bad = true;
            if (warp == 0) {  // inclusive scan of the warp totals
                int v = lane < nw ? wsum[lane] : 0;
                for (int s = 1; s < 32; s <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, v, s);
                    if (lane >= s) v += u;
                }
                if (lane < nw) wsum[lane] = v;
            }
            __syncthreads();
            const int total = wsum[nw - 1];
            off += (warp ? wsum[warp - 1] : 0) - n;
            if (count + total <= cap)
                for (int k = 0; k < n; ++k) r[count + off + k] = w[k];
            else bad = true;
            count += total;
            __syncthreads();  // wsum is reused by the next round
        }
    }
    if (tid == 0) {
        if (bad) { set_error(T, kELimit, id); r[0] = 1; }
        else r[0] = int(count);
    }
    __syncthreads();
    if (commit && !bad) commit_net_wires(T, P2, id, stamp, 1, lane, warp, nw);
    __syncthreads();  // the arrays are reused by the CTA's next net
}

}  // namespace grb
