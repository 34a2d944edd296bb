// zshape.cuh -- Z-shape stage: two-bend candidates on projection planes,
// layer-range DP per tree node and traceback; bounding-box batch refinement.
//
// Semantics of the reference's Z-shape pipeline (zshape.cuh:5-404,
// zshape_topology.hpp:7-57 and 249-290).  All costs are int32: a wire costs
// |presum[a] - presum[b]| clamped to 5e8, a via clamp(vcost, 1, 1e6), with 1e9
// as infinity; sums wrap as 32-bit integers exactly as the device code does.
// The reference keeps, on planes of LAYER = L+1 layers of N x N (N = max(X, Y)),
// per 2-D position and layer: the node DP, the best arrival of child slot j,
// the current edge's candidate rows and columns, the chosen layer per node and
// their back-pointers, which are plane indexes.  A position on GGR layer i sits
// at i*N*N + (x*N + y) when ((i & 1) ^ D) is 1, at i*N*N + (y*N + x) otherwise,
// D = DIR ^ 1; GGR layer i is routing layer i-1 (layer 0 carries no wires and
// costs an infinite via).  Only cells at tree nodes outlive an edge, so here
// they are small per-net arrays in shared memory (nodes at one position share
// their cells, as on the planes), and no plane exists.
//
// B200 form: one CTA per net.  A two-bend candidate of an edge runs from the
// child along one side of the box, changes layer, crosses the box, changes
// layer again and runs to the node: everything between the child and the node
// depends on one position of that side only.  So a warp takes as many
// positions as it holds columns (a lane per position and layer) and walks the
// five steps in registers (zedge_chunk): one round of table reads, layer
// changes as prefix minima by shuffle, no barrier and no memory in between; a
// minimum in shared memory joins the positions.  The positions of all edges
// into the nodes of one depth are dealt out to the CTA's warps; two barriers
// per depth.  A batch lasts as long as its largest net, a few dozen short
// dependent steps: phases over planes in HBM, six barriers an edge and a serial
// traceback from global memory, took 136 us of DP a batch of 127 nets
// (320x320x10, 60K nets); a lane per position with its column in registers, 87
// us (2,500 instructions of straight-line code, fetched anew by every warp);
// this form 68 us.
#pragma once
#include "commit.cuh"
#include "common.cuh"

namespace grb {

constexpr int kZInf = 1000000000;  // zshape.cuh:6

struct ZTrees {
    const int* node_off;  // [n+1] by net id
    const int* pos;       // per node: x*N + y
    const int* pin;       // per node: pin layer + 1, -1 for Steiner points
    const int* child;     // [3 per node] net-local preorder index, -1 = none
    int fit;              // nodes whose arrays fit the CTA's shared memory
    int* scratch;         // the arrays of the nets beyond `fit` nodes
    const int* wide_off;  // [n] nodes of the nets beyond `fit` before this one: a place
                          // each; null: a place of `most` nodes per CTA
    int most;             // nodes of the largest net
    int N, NN, LAYER, D;
    FastDiv by_n, by_nn;
};

__device__ __forceinline__ int zadd(int a, int b) {
    return static_cast<int>(static_cast<unsigned>(a) + static_cast<unsigned>(b));
}
__device__ __forceinline__ int zidx(const ZTrees& Z, int i, int x, int y) {
    return i * Z.NN + (((i & 1) ^ Z.D) ? x * Z.N + y : y * Z.N + x);
}
// ViaCosts (zshape.cuh:20-31) and boundedWireCost over WireCosts
// (zshape.cuh:8-19, 32-35) for plane layer i (1..L, routing layer i-1) at grid
// positions.
__device__ __forceinline__ int zvia_at(const Tables& T, int i, int x, int y) {
    return static_cast<int>(fminf(fmaxf(T.vcost[slot_index(T, i - 1, x, y)], 1.f), 1.e6f));
}
__device__ __forceinline__ int zwire_of(double a, double b) {
    return static_cast<int>(fmin(fabs(a - b), static_cast<double>(kZInf / 2)));
}

// Arrays of one net (ints), by node and plane layer; `rep` is the first node at
// a node's position, whose cells it uses.
struct ZNet {
    int cnt, LY;
    int *m0, *p0;    // [cnt][LY] node DP and its code
    unsigned long long* key;  // [3][cnt][LY] the edge in progress: (least arrival, position, source and turn layer)
    int *mj, *pj, *qj;  // [3][cnt][LY] arrival of child slot j, its source and turn cells
    int* via;        // [cnt][LY] via cost at the node
    int *pos, *pin, *child, *rep, *dep, *par, *lay;  // child [3 * cnt]; lay: chosen layer
};
__host__ __device__ constexpr int znet_ints(int LY) { return 18 * LY + 10; }  // per node (even: 8-byte keys)
__device__ __forceinline__ ZNet znet(int* a, int cnt, int LY) {
    ZNet W;
    W.cnt = cnt; W.LY = LY;
    W.key = reinterpret_cast<unsigned long long*>(a); a += 6 * cnt * LY;
    W.m0 = a; a += cnt * LY;
    W.p0 = a; a += cnt * LY;
    W.mj = a; a += 3 * cnt * LY;
    W.pj = a; a += 3 * cnt * LY;
    W.qj = a; a += 3 * cnt * LY;
    W.via = a; a += cnt * LY;
    W.pos = a; a += cnt;
    W.pin = a; a += cnt;
    W.child = a; a += 3 * cnt;
    W.rep = a; a += cnt;
    W.dep = a; a += cnt;
    W.par = a; a += cnt;
    W.lay = a;
    return W;
}

// viaSweep (zshape.cuh:42-61) over one position's column, a lane per layer (the
// `width` lanes from lane - r on hold layers 1..width, r = layer - 1): up, then
// down, each keeping strict improvements.  In either direction a layer takes
// the least m[j] + (vias between), the nearest j on ties, which is a prefix
// minimum of m[j] - V[j], V the running via sum.  Sums stay below 2^31 (values
// at most 1.5e9, vias 1e6 each).  src: the layer offset whose back-pointer the
// value carries; q: the layer offset the value came from in its last step.
__device__ __forceinline__ void zsweep(int& m, int& src, int& q, int V, int r, int width, int lane) {
    const int lo = lane - r;
    int val = m - V, at = r;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const int ov = __shfl_sync(0xffffffffu, val, max(lane - d, 0)), oa = __shfl_sync(0xffffffffu, at, max(lane - d, 0));
        if (r >= d && ov < val) { val = ov; at = oa; }
    }
    q = at == r ? r : r - 1;
    src = __shfl_sync(0xffffffffu, src, (lo + at) & 31);
    m = val + V;
    val = m + V;
    at = r;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const int ov = __shfl_sync(0xffffffffu, val, min(lane + d, 31)), oa = __shfl_sync(0xffffffffu, at, min(lane + d, 31));
        if (r + d < width && ov < val) { val = ov; at = oa; }
    }
    if (at != r) q = r + 1;
    src = __shfl_sync(0xffffffffu, src, (lo + at) & 31);
    m = val - V;
}
// Exclusive sum of v over the layers below (same lanes).
__device__ __forceinline__ int zbelow(int v, int r, int lane) {
    int incl = v;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const int o = __shfl_sync(0xffffffffu, incl, max(lane - d, 0));
        if (r >= d) incl += o;
    }
    return incl - v;
}

// Geometry of the edge from child c to node v.
struct ZEdge {
    int fromx, fromy, tox, toy;
    bool bent;
    // Positions of the child's row (x changes, the first nx) and column, without
    // its own.
    int nx, items;
};
__device__ __forceinline__ ZEdge zedge(const ZTrees& Z, const ZNet& W, int c, int v) {
    ZEdge E;
    const int pc = W.pos[c], pv = W.pos[v];
    E.fromx = Z.by_n(pc); E.fromy = pc - E.fromx * Z.N;
    E.tox = Z.by_n(pv); E.toy = pv - E.tox * Z.N;
    E.bent = E.fromx != E.tox && E.fromy != E.toy;
    E.nx = abs(E.fromx - E.tox);
    E.items = E.bent ? E.nx + abs(E.fromy - E.toy) : 1;
    return E;
}

// A straight edge into child slot j of node v (zshape.cuh:213-237), a lane per
// layer.
__device__ __forceinline__ void zedge_straight(const Tables& T, const ZTrees& Z, const ZNet& W, const ZEdge& E, int j,
                                               int c, int v, int lane) {
    const int i = lane;
    if (i < 1 || i >= W.LY) return;
    const int at = (j * W.cnt + W.rep[v]) * W.LY + i;
    const bool ay = ((i & 1) ^ Z.D) != 0;
    if (E.fromx == E.tox ? ay : !ay) {
        const int w = zwire_of(T.presum[slot_index(T, i - 1, E.fromx, E.fromy)], T.presum[slot_index(T, i - 1, E.tox, E.toy)]);
        const int x = zadd(W.m0[W.rep[c] * W.LY + i], w);
        if (W.mj[at] > x) { W.mj[at] = x; W.pj[at] = zidx(Z, i, E.fromx, E.fromy); }
    } else {
        W.mj[at] = kZInf;
    }
}

// Positions k0, k0 + 1, ... (`rounds` times the S a warp holds) of a bent edge
// into child slot j of node v (zshape.cuh:87-212); lane = position * width +
// (layer - 1).
__device__ __forceinline__ void zedge_chunk(const Tables& T, const ZTrees& Z, const ZNet& W, const ZEdge& E, int j, int c,
                                            int v, int k0, int rounds, int lane) {
    const int width = W.LY - 1, S = 32 / width, D = Z.D;
    const int s = lane / width, r = lane - s * width, i = r + 1;  // plane layer i, routing layer r
    const bool on = s < S, ay = ((i & 1) ^ D) != 0;
    const int base = on ? W.m0[W.rep[c] * W.LY + i] : 0;
    const int lb = layer_base(T, on ? r : 0);
    auto slot = [&](int x, int y) { return lb + (ay ? x * T.yp + y : y * T.xp + x); };
    const double pf = on ? T.presum[slot(E.fromx, E.fromy)] : 0.0, pt = on ? T.presum[slot(E.tox, E.toy)] : 0.0;
    int best = 0x7fffffff;
    unsigned code = ~0u;
    for (int n = 0; n < rounds; ++n) {
        const int k = k0 + n * S + s;
        if (k0 + n * S >= E.items) break;
        const bool in = on && k < E.items, isx = k < E.nx;
        const int f = isx ? E.fromx : E.fromy;
        int b = (isx ? min(E.fromx, E.tox) : min(E.fromy, E.toy)) + (isx ? k : k - E.nx);
        if (b >= f) ++b;
        if (!in) b = f;  // any position of the box
        // At the box corner the run already ends on the node's other line: no
        // crossing, and the way goes on across the line's direction.
        const bool corner = b == (isx ? E.tox : E.toy);
        const int a1 = slot(isx ? b : E.fromx, isx ? E.fromy : b), a2 = slot(isx ? b : E.tox, isx ? E.toy : b);
        const double p1 = on ? T.presum[a1] : 0.0, p2 = on ? T.presum[a2] : 0.0;
        const int v1 = on ? static_cast<int>(fminf(fmaxf(T.vcost[a1], 1.f), 1.e6f)) : 0;
        const int v2 = on ? static_cast<int>(fminf(fmaxf(T.vcost[corner ? a1 : a2], 1.f), 1.e6f)) : 0;
        const bool own = ay != isx;  // the layer runs along this line
        int m = own ? zadd(base, zwire_of(pf, p1)) : kZInf, src = r, q;
        zsweep(m, src, q, zbelow(v1, r, lane), r, width, lane);
        const int step = own ? zwire_of(p2, pt) : zwire_of(p1, p2);  // the last run; the crossing
        if (!corner) {
            const int x = zadd(m, step);
            m = !own && x < kZInf ? x : kZInf;
        }
        zsweep(m, src, q, zbelow(v2, r, lane), r, width, lane);
        if (in && own != corner) {  // ends across the line at the corner, along it elsewhere
            const int x = zadd(m, step);
            const unsigned xc = unsigned((corner ? (isx ? E.fromy : E.fromx) : b) << 8) | unsigned((src + 1) << 4) | unsigned(q + 1);
            if (x < best || (x == best && xc < code)) { best = x; code = xc; }
        }
    }
    // Per layer the first minimum over the positions (the reference scans them
    // in order keeping strict improvements).
    if (on && code != ~0u)
        atomicMin(W.key + (j * W.cnt + W.rep[v]) * W.LY + i,
                  (static_cast<unsigned long long>(static_cast<unsigned>(best) ^ 0x80000000u) << 32) | code);
}

// The finished edge into child slot j of node v: its least arrival per layer,
// if an improvement, into the slot's cells.
__device__ __forceinline__ void zedge_apply(const ZTrees& Z, const ZNet& W, const ZEdge& E, int j, int v, int lane) {
    const int i = lane;
    if (i < 1 || i >= W.LY) return;
    const int at = (j * W.cnt + W.rep[v]) * W.LY + i;
    const unsigned long long key = W.key[at];
    if (key == ~0ull) return;
    W.key[at] = ~0ull;
    const int best = static_cast<int>(static_cast<unsigned>(key >> 32) ^ 0x80000000u);
    if (best >= W.mj[at]) return;
    const int b = static_cast<int>((key >> 8) & 0xffffff), pl = static_cast<int>(key >> 4) & 15, q = static_cast<int>(key) & 15;
    const bool ay = ((i & 1) ^ Z.D) != 0;
    W.mj[at] = best;
    W.pj[at] = zidx(Z, pl, E.fromx, E.fromy);
    W.qj[at] = zidx(Z, q, ay ? E.tox : b, ay ? b : E.toy);
}

// Layer-range DP of one node (zshape.cuh:241-267) with a warp: lane `lower`
// walks its uppers (the child and via values of every layer come by shuffle)
// and writes each range's value and code to shared memory `cand`
// (2 * LAYER * LAYER ints); then lane i takes, over the allowed ranges
// containing layer i in the sequential (lower, upper) order, the first strict
// minimum -- exactly the value and code the sequential loop leaves at layer i.
__device__ __forceinline__ void znode_dp_warp(const ZNet& W, int v, int lane, int* cand) {
    const int LAYER = W.LY, at = W.rep[v] * LAYER + lane, pin = W.pin[v];
    const int ch[3] = {W.child[3 * v], W.child[3 * v + 1], W.child[3 * v + 2]};
    int pv[3];
    for (int j = 0; j < 3; ++j) pv[j] = (lane < LAYER && ch[j] != -1) ? W.mj[j * W.cnt * LAYER + at] : 0;
    const int vc = lane < LAYER ? (lane >= 1 ? W.via[v * LAYER + lane] : kZInf) : 0;
    const int lower = lane;
    int viaSum = 0, minCost = kZInf, bestpos[3] = {0, 0, 0};
    int costs[3] = {ch[0] == -1 ? 0 : kZInf, ch[1] == -1 ? 0 : kZInf, ch[2] == -1 ? 0 : kZInf};
    for (int upper = 0; upper < LAYER; ++upper) {
        int x[3];
        for (int j = 0; j < 3; ++j) x[j] = __shfl_sync(0xffffffffu, pv[j], upper);
        const int vu = __shfl_sync(0xffffffffu, vc, upper);
        if (lower >= LAYER || upper < lower) continue;
        for (int j = 0; j < 3; ++j)
            if (ch[j] != -1 && x[j] < costs[j]) { costs[j] = x[j]; bestpos[j] = upper; }
        if (1LL * costs[0] + costs[1] + costs[2] < minCost) minCost = costs[0] + costs[1] + costs[2];
        const bool allowed = pin == -1 || (lower <= pin && pin <= upper);
        cand[lower * LAYER + upper] = zadd(minCost, viaSum);
        cand[LAYER * LAYER + lower * LAYER + upper] =
            allowed ? (((lower * LAYER + upper) * LAYER + bestpos[2]) * LAYER + bestpos[1]) * LAYER + bestpos[0] : -1;
        viaSum = zadd(viaSum, vu);
    }
    __syncwarp();
    if (lane < LAYER) {
        const int i = lane;
        int best = W.m0[at], code = 0;
        bool changed = false;
        for (int lo = 0; lo <= i; ++lo)
            for (int up = i; up < LAYER; ++up) {
                const int c = cand[LAYER * LAYER + lo * LAYER + up];
                const int val = cand[lo * LAYER + up];
                if (c >= 0 && best > val) { best = val; code = c; changed = true; }
            }
        if (changed) { W.m0[at] = best; W.p0[at] = code; }
    }
    __syncwarp();
}

// convert_routes (zshape_topology.hpp:249-290) of one (start, length | -1)
// pair straight into route words; returns a reference status on failure.
__device__ __forceinline__ int zemit(const Tables& T, const ZTrees& Z, int start, int len, int* r, int& out,
                                     long long cap) {
    const int n = Z.N, plane = Z.by_nn(start), rem = start - plane * Z.NN;
    const int layer = plane - 1;
    const int a = Z.by_n(rem), b = rem - a * n;
    const bool ay = ((layer & 1) ^ T.DIR) != 0;
    const int x = ay ? a : b, y = ay ? b : a;
    if (layer < 0 || layer >= T.L || x >= T.X || y >= T.Y) return 3;
    const int pos0 = cell_index(T, layer, x, y);
    int pos1;
    if (len == -1) {
        if (layer + 1 >= T.L) return 3;
        pos1 = pos0 + T.XY;
    } else {
        const int end = start + len, er = end - Z.by_nn(end) * Z.NN, ea = Z.by_n(er), eb = er - ea * n;
        const int ex = ay ? ea : eb, ey = ay ? eb : ea;
        if (ex >= T.X || ey >= T.Y) return 3;
        pos1 = cell_index(T, layer, ex, ey);
    }
    if (out + 1 < cap) { r[out++] = pos0; r[out++] = pos1; return 0; }
    return 1;
}

// Plane index -> layer and position.
__device__ __forceinline__ void zcell(const ZTrees& Z, int c, int& layer, int& x, int& y) {
    layer = Z.by_nn(c);
    const int r = c - layer * Z.NN, a = Z.by_n(r), b = r - a * Z.N;
    const bool ay = ((layer & 1) ^ Z.D) != 0;
    x = ay ? a : b;
    y = ay ? b : a;
}

// Traceback (zshape.cuh:271-386) of one net on one thread, converted into the
// net's route record.  Returns 0 or the reference's status (1 storage, 2 no
// finite route, 3 segment outside the grid).
__device__ __forceinline__ int ztrace(const Tables& T, const ZTrees& Z, const ZNet& W, int* r, long long cap) {
    const int LAYER = W.LY, D = Z.D;
    int out = 1, status = 0;
    auto emit = [&](int a, int b) { const int s = zemit(T, Z, a, b, r, out, cap); if (s) status = s; };
    auto run = [&](int a, int b) { emit(min(a, b), max(a, b) - min(a, b)); };
    int minTotal = kZInf;
    for (int i = 0; i < LAYER; ++i)
        if (W.m0[W.rep[0] * LAYER + i] < minTotal) { minTotal = W.m0[W.rep[0] * LAYER + i]; W.lay[W.rep[0]] = i; }
    if (minTotal == kZInf || minTotal < 0) { r[0] = 1; return 2; }
    for (int t = 0; t < W.cnt; ++t) {
        const int rt = W.rep[t], pt = W.pos[t], x = Z.by_n(pt), y = pt - x * Z.N, layer = W.lay[rt];
        const int code = W.p0[rt * LAYER + layer];
        const int minl = code / LAYER / LAYER / LAYER / LAYER, maxl = code / LAYER / LAYER / LAYER % LAYER;
        for (int i = minl; i < maxl; ++i) emit(zidx(Z, i, x, y), -1);
        int bestpos = code;
        for (int j = 0; j < 3; ++j) {
            const int c = W.child[3 * t + j];
            if (c == -1) break;
            const int entrylayer = bestpos % LAYER, entry = zidx(Z, entrylayer, x, y);
            const int at = (j * W.cnt + rt) * LAYER + entrylayer;
            bestpos /= LAYER;
            const int last = W.pj[at];
            int lastlayer, lastx, lasty;
            zcell(Z, last, lastlayer, lastx, lasty);
            if (lastx != x && lasty != y) {
                const int mid = W.qj[at];
                int midlayer, midx, midy;
                zcell(Z, mid, midlayer, midx, midy);
                const int q1 = ((entrylayer & 1) ^ D) ? entry - y + midy : entry - x + midx;
                const int q3 = ((midlayer & 1) ^ D) ? mid - midy + lasty : mid - midx + lastx;
                const int q4 = ((lastlayer & 1) ^ D) ? last - lasty + midy : last - lastx + midx;
                if (entry != q1) run(entry, q1);
                if (q1 != mid)
                    for (int i = min(entrylayer, midlayer); i < max(entrylayer, midlayer); ++i) emit(zidx(Z, i, midx, midy), -1);
                if (mid != q3) run(mid, q3);
                if (q3 != q4) {
                    int tl, tx, ty;
                    zcell(Z, q3, tl, tx, ty);
                    for (int i = min(midlayer, lastlayer); i < max(midlayer, lastlayer); ++i) emit(zidx(Z, i, tx, ty), -1);
                }
                if (q4 != last) run(q4, last);
            } else {
                run(last, entry);
            }
            W.lay[W.rep[c]] = lastlayer;
        }
    }
    r[0] = out;
    return status;
}

// Global scratch of net `id` (beyond Z.fit nodes).
__device__ __forceinline__ int* zscratch(const ZTrees& Z, int id) {
    const long long at = Z.wide_off ? Z.wide_off[id] : static_cast<long long>(blockIdx.x) * Z.most;
    return Z.scratch + at * znet_ints(Z.LAYER);
}

// Route net `id` with the whole CTA; with `commit`, also its wire demand (warp
// 0).  `smem`: the warps' node-DP ranges (2 * LAYER * LAYER ints each), then
// the arrays of a net of Z.fit nodes.
__device__ __forceinline__ void zshape_net(const Tables& T, const ZTrees& Z, const Plan& P, int id, int stamp, bool commit,
                                           int* smem) {
    __shared__ int zstatus, zdeep;
    const int t = threadIdx.x, nth = blockDim.x, lane = t & 31, warp = t >> 5, nw = nth >> 5, LY = Z.LAYER;
    const int nb = Z.node_off[id], cnt = Z.node_off[id + 1] - nb;
    int* r = P.routes + P.route_off[id];
    const long long cap = P.route_off[id + 1] - P.route_off[id];
    if (cnt <= 0) {
        if (t == 0 && cap > 0) r[0] = 1;
        return;
    }
    if (cap <= 0) {
        if (t == 0) set_error(T, kELimit, id);
        return;
    }
    int* cand = smem + warp * 2 * LY * LY;
    const ZNet W = znet(cnt <= Z.fit ? smem + nw * 2 * LY * LY : zscratch(Z, id), cnt, LY);
    // reset_nodes (zshape.cuh:392-404), and everything of the net the DP reads.
    if (t == 0) zdeep = 0;
    for (int k = t; k < cnt * LY; k += nth) {
        const int v = k / LY, i = k - v * LY, pt = Z.pos[nb + v], x = Z.by_n(pt);
        W.m0[k] = kZInf;
        W.p0[k] = 0;
        W.via[k] = i ? zvia_at(T, i, x, pt - x * Z.N) : kZInf;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            W.mj[j * cnt * LY + k] = kZInf;
            W.pj[j * cnt * LY + k] = 0;
            W.qj[j * cnt * LY + k] = 0;
            W.key[j * cnt * LY + k] = ~0ull;
        }
    }
    for (int v = t; v < cnt; v += nth) {
        W.pos[v] = Z.pos[nb + v];
        W.pin[v] = Z.pin[nb + v];
        W.par[v] = -1;
        for (int j = 0; j < 3; ++j) W.child[3 * v + j] = Z.child[3 * (nb + v) + j];
    }
    __syncthreads();
    bool shared_cell = false;
    for (int v = t; v < cnt; v += nth) {
        for (int j = 0; j < 3; ++j)
            if (W.child[3 * v + j] != -1) W.par[W.child[3 * v + j]] = v;
        int u = 0;
        while (W.pos[u] != W.pos[v]) ++u;
        W.rep[v] = u;
        shared_cell |= u != v;
    }
    // Nodes that share cells are taken one at a time in the reference's order;
    // else all nodes of a depth at once, from the deepest.
    const bool serial = __syncthreads_or(shared_cell);
    for (int v = t; v < cnt; v += nth) {
        int d = 0;
        if (serial) d = v;
        else
            for (int u = W.par[v]; u >= 0; u = W.par[u]) ++d;
        W.dep[v] = d;
        atomicMax(&zdeep, d);
    }
    __syncthreads();
    const int S = 32 / (LY - 1);  // positions a warp takes at once
    for (int d = zdeep; d >= 0; --d) {
        // The depth's edges: how many positions, so that every warp gets a share.
        int positions = 0, turn = 0;
        for (int u = lane; u < cnt; u += 32)
            if (W.dep[u] == d)
                for (int j = 0; j < 3; ++j)
                    if (W.child[3 * u + j] != -1) positions += zedge(Z, W, W.child[3 * u + j], u).items;
        positions = __reduce_add_sync(0xffffffffu, positions);
        const int rounds = max(1, (positions + nw * S - 1) / (nw * S));
        for (int pass = positions ? 0 : 1; pass < 2; ++pass) {  // edges, then nodes
            for (int u0 = 0; u0 < cnt; u0 += 32) {
                unsigned at = __ballot_sync(0xffffffffu, u0 + lane < cnt && W.dep[min(u0 + lane, cnt - 1)] == d);
                for (; at; at &= at - 1) {
                    const int v = u0 + __ffs(at) - 1;
                    if (pass && turn++ % nw != warp) continue;
                    for (int j = 0; j < 3; ++j) {
                        const int c = W.child[3 * v + j];
                        if (c == -1) continue;
                        const ZEdge E = zedge(Z, W, c, v);
                        if (pass) {
                            if (E.bent) zedge_apply(Z, W, E, j, v, lane);
                        } else {
                            for (int k0 = 0; k0 < E.items; k0 += rounds * S) {
                                if (turn++ % nw != warp) continue;
                                if (E.bent) zedge_chunk(T, Z, W, E, j, c, v, k0, rounds, lane);
                                else zedge_straight(T, Z, W, E, j, c, v, lane);
                            }
                        }
                    }
                    if (pass) {
                        __syncwarp();
                        znode_dp_warp(W, v, lane, cand);
                    }
                }
            }
            __syncthreads();
        }
    }
    if (t == 0) {
        zstatus = ztrace(T, Z, W, r, cap);
        if (zstatus) set_error(T, zstatus == 1 ? kELimit : kEInval, id);
    }
    __syncthreads();
    const int status = zstatus;
    if (commit && !status && t < 32) commit_net_wires(T, P, id, stamp, 1, lane);
    __syncthreads();
}

// --- bounding-box batch refinement (zshape_topology.hpp:7-57) --------------
// Within one first-fit group, nets sorted by box area (descending, larger id
// first on ties) form greedy rounds of at most `max_batch` nets with pairwise
// disjoint boxes; this is first-fit colouring with box-intersection conflicts.
__device__ __forceinline__ bool boxes_meet(int4 a, int4 b) {
    // int4 = (minx, maxx, miny, maxy)
    return !(a.y < b.x || b.y < a.x || a.w < b.z || b.w < a.z);
}

}  // namespace grb
