// lshape.cuh -- L-shape pattern routing with layer assignment: a warp per pack of
// small nets (route_pack), or per net beyond a pack (lshape_net).
//
// Semantics are those of the reference's tree DP (lshape_thread.cuh:18-171,
// lshape_warp.cuh:8-247): per tree node a table dist[low][high] over layer
// ranges (via stack cost inside the range, INF where a pin's layer falls
// outside); children are merged into their parent in descending node order;
// an edge is a straight wire or an L with a via stack at the corner; strict '<'
// keeps the first minimum in the reference's loop order; the root takes the
// first minimal range; traceback and segment emission follow node order.
//
// B200 mapping: all cost gathers of a net (via stacks at nodes and corners,
// wire costs of both legs on every layer) are issued up front by the 32 lanes
// into a per-warp shared-memory arena, so a net pays one memory latency; the
// DP itself then runs from shared memory with lanes over layers.  The
// reference keeps 81 doubles per node in global scratch and gathers inside the
// DP loop.
#pragma once
#include "commit.cuh"
#include "common.cuh"

namespace grb {

__host__ __device__ __forceinline__ int tri_count(int L) { return L * (L + 1) / 2; }
__device__ __forceinline__ int tri(int L, int lo, int hi) { return lo * L - lo * (lo - 1) / 2 + (hi - lo); }

struct Arena {
    double* dist;          // [nmax][TT]
    double* w1;            // [nmax][L] first leg (or straight) wire cost
    double* w2;            // [nmax][L] second leg wire cost
    float* vA;             // [nmax][L] via cost at corner (x, py)
    float* vB;             // [nmax][L] via cost at corner (px, y)
    float* vN;             // [nmax][L] via cost at the node
    unsigned short* from;  // [nmax][TT] choice*L*L + curl*L + parl
    int* range;            // [nmax] chosen range lo*L+hi
    int* xy;               // [nmax] node coordinate x << 16 | y (grids are at most 8192 wide)
    int* lay;              // [nmax] node layer (L: Steiner point)
    int* dep;              // [nmax] node depth (root 0)
    // Per-lane scratch of a level pass: lane = slot * L + layer for up to
    // 32 / L nodes at once.
    double* cur;           // [32] best range through each layer (of the slot's node)
    double* diag;          // [32] best parent-layer cost
    int* cur_from;         // [32]
    int* pdiag;            // [32]
};

__host__ __device__ __forceinline__ size_t arena_bytes(int L, int nmax) {
    const size_t TT = tri_count(L);
    size_t b = 0;
    b += nmax * TT * 8 + 2 * size_t(nmax) * L * 8 + 3 * size_t(nmax) * L * 4;
    b = (b + 7) & ~size_t(7);
    b += 2 * 32 * 8;
    b += nmax * TT * 2;
    b = (b + 7) & ~size_t(7);
    b += nmax * 4 + 2 * 32 * 4 + 3 * size_t(nmax) * 4;
    return (b + 15) & ~size_t(15);
}

__device__ __forceinline__ Arena carve_arena(char* base, int L, int nmax) {
    const int TT = tri_count(L);
    Arena A;
    char* p = base;
    A.dist = reinterpret_cast<double*>(p); p += size_t(nmax) * TT * 8;
    A.w1 = reinterpret_cast<double*>(p); p += size_t(nmax) * L * 8;
    A.w2 = reinterpret_cast<double*>(p); p += size_t(nmax) * L * 8;
    A.vA = reinterpret_cast<float*>(p); p += size_t(nmax) * L * 4;
    A.vB = reinterpret_cast<float*>(p); p += size_t(nmax) * L * 4;
    A.vN = reinterpret_cast<float*>(p); p += size_t(nmax) * L * 4;
    p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 7) & ~uintptr_t(7));
    A.cur = reinterpret_cast<double*>(p); p += 32 * 8;
    A.diag = reinterpret_cast<double*>(p); p += 32 * 8;
    A.from = reinterpret_cast<unsigned short*>(p); p += size_t(nmax) * TT * 2;
    p = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 7) & ~uintptr_t(7));
    A.range = reinterpret_cast<int*>(p); p += nmax * 4;
    A.cur_from = reinterpret_cast<int*>(p); p += 32 * 4;
    A.pdiag = reinterpret_cast<int*>(p); p += 32 * 4;
    A.xy = reinterpret_cast<int*>(p); p += nmax * 4;
    A.lay = reinterpret_cast<int*>(p); p += nmax * 4;
    A.dep = reinterpret_cast<int*>(p);
    return A;
}

__device__ __forceinline__ double wire_cost(const Tables& T, int l, int xmin, int xmax, int ymin, int ymax) {
    // prefix_scan.cuh:10-40 (wire_segment_cost)
    return T.presum[slot_index(T, l, xmax, ymax)] - T.presum[slot_index(T, l, xmin, ymin)];
}

// Route one net.  All 32 lanes of the warp call this with the same id.
// Returns false (and records kELimit) if the net's route storage is too small.
// LC: the number of routing layers when known at compile time (the loops
// over layers then unroll into independent loads and predicated compares, in
// the same order), 0 for any layer count.
template <int LC>
__device__ __forceinline__ void lshape_net_l(const Tables& T, const Plan& P, int id, int stamp, const Arena& A,
                                             int lane, bool fuse_wires) {
    const int L = LC > 0 ? LC : T.L, TT = tri_count(L);
    constexpr int LL = LC > 0 ? LC : kMaxLayers;  // static bound of the layer loops
    const int off = P.node_off[id], N = P.node_off[id + 1] - off;
    const int* nd = P.nodes + off;
    const int* par = P.parents + off;

    // 0. Node coordinates, once per net (the divisions by the runtime grid
    // sizes are not repeated per layer and step).
    int dmax = 0;
    for (int q = lane; q < N; q += 32) {
        int l, x, y;
        cell_position(T, nd[q], l, x, y);
        A.xy[q] = (x << 16) | y;
        A.lay[q] = l;
        int d = 0;
        for (int v = q; v > 0; v = par[v]) ++d;  // parents precede children
        A.dep[q] = d;
        dmax = max(dmax, d);
    }
    for (int s = 16; s; s >>= 1) dmax = max(dmax, __shfl_xor_sync(0xffffffffu, dmax, s));
    __syncwarp();
    // 1. Gather every cost the DP reads.  Each lane takes two (node, layer)
    // items per pass and issues all their loads before any arena store.
    for (int q0 = lane; q0 < N * L; q0 += 64) {
        float vn[2], va[2], vb[2];
        double w1[2], w2[2];
        int kind[2];  // 0: none, 1: node only, 2: straight edge, 3: L-shaped edge
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + 32 * u;
            kind[u] = 0;
            vn[u] = va[u] = vb[u] = 0.f;
            w1[u] = w2[u] = 0.0;
            if (q >= N * L) continue;
            const int i = q / L, l = q - i * L;
            const int x = A.xy[i] >> 16, y = A.xy[i] & 0xffff;
            vn[u] = T.vcost[slot_index(T, l, x, y)];
            kind[u] = 1;
            if (i > 0) {
                const int pxy = A.xy[par[i]], px = pxy >> 16, py = pxy & 0xffff;
                const int minx = min(x, px), maxx = max(x, px), miny = min(y, py), maxy = max(y, py);
                const bool ay = along_y(T, l);
                if (x == px || y == py) {
                    const bool valid = ay ? (x == px) : (y == py);
                    w1[u] = valid ? wire_cost(T, l, minx, maxx, miny, maxy) : 0.0;
                    kind[u] = 2;
                } else {
                    w1[u] = ay ? wire_cost(T, l, x, x, miny, maxy) : wire_cost(T, l, minx, maxx, y, y);
                    w2[u] = ay ? wire_cost(T, l, px, px, miny, maxy) : wire_cost(T, l, minx, maxx, py, py);
                    va[u] = T.vcost[slot_index(T, l, x, py)];
                    vb[u] = T.vcost[slot_index(T, l, px, y)];
                    kind[u] = 3;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + 32 * u;
            if (kind[u] >= 1) A.vN[q] = vn[u];
            if (kind[u] >= 2) A.w1[q] = w1[u];
            if (kind[u] == 3) {
                A.w2[q] = w2[u];
                A.vA[q] = va[u];
                A.vB[q] = vb[u];
            }
        }
    }
    __syncwarp();
    // 2. Via stacks at every node (lshape_thread.cuh:40-50).
    for (int q = lane; q < N * L; q += 32) {
        const int i = q / L, lo = q - i * L;
        const int fixed = A.lay[i];
        double acc = 0;
#pragma unroll
        for (int hi = 0; hi < LL; ++hi) {
            if (hi < lo || hi >= L) continue;
            if (hi > lo) acc = acc + static_cast<double>(A.vN[i * L + hi - 1]);
            A.dist[i * TT + tri(L, lo, hi)] = (fixed < L && (lo > fixed || hi < fixed)) ? kInf : acc;
        }
    }
    __syncwarp();
    // 3. Children into parents (lshape_thread.cuh:51-115), one depth at a
    // time from the deepest: the nodes of a depth have complete tables, so
    // up to 32 / L of them are processed at once (lane = slot * L + layer);
    // then every node of the depth, in descending node order, adds its table
    // into its parent.  A parent receives its children (all one depth below
    // it) in descending order, exactly the sequential loop's additions.
    const int S = max(1, 32 / L);
    const int slot = lane / L, sl = lane - slot * L;
    for (int d = dmax; d >= 1; --d) {
        for (int base = 0; base < N; base += 32) {
            const int q = base + lane;
            unsigned at = __ballot_sync(0xffffffffu, q < N && A.dep[q] == d);
            while (at) {
                // The next S nodes of this depth in this window.
                int mine = -1;
                {
                    unsigned m = at;
                    for (int k = 0; k < S && m; ++k) {
                        const int b = __ffs(m) - 1;
                        m &= m - 1;
                        if (k == slot) mine = base + b;
                    }
                    at = m;
                }
                const bool act = slot < S && mine >= 0;
                const int i = mine;
                if (act) {
                    const double* di = A.dist + i * TT;
                    const int l = sl;
                    double best = kInf;
                    int bf = 0;
#pragma unroll
                    for (int lo = 0; lo < LL; ++lo)
#pragma unroll
                        for (int hi = lo; hi < LL; ++hi) {
                            if (lo > l || hi < l || hi >= L) continue;
                            const double v = di[tri(L, lo, hi)];
                            if (v < best) { best = v; bf = lo * L + hi; }
                        }
                    A.cur[lane] = best;
                    A.cur_from[lane] = bf;
                }
                __syncwarp();
                if (act) {
                    const int pl = sl, p = par[i], s0 = slot * L;
                    const int x = A.xy[i] >> 16, y = A.xy[i] & 0xffff;
                    const int px = A.xy[p] >> 16, py = A.xy[p] & 0xffff;
                    double best = kInf;
                    int pb = 0;
                    if (x == px || y == py) {
                        const bool valid = along_y(T, pl) ? (x == px) : (y == py);
                        if (valid) {
                            best = A.cur[s0 + pl] + A.w1[i * L + pl];
                            pb = A.cur_from[s0 + pl] * L * L + pl * L + pl;
                        }
                    } else {
#pragma unroll
                        for (int cl = 0; cl < LL; ++cl) {
                            if (((cl ^ pl) & 1) == 0 || cl >= L) continue;  // the other parity, ascending
                            const double cost = A.cur[s0 + cl] + A.w1[i * L + cl];
                            double cost2 = 0;
                            const float* v = along_y(T, cl) ? A.vA + i * L : A.vB + i * L;
                            const int a = min(cl, pl), b = max(cl, pl);
#pragma unroll
                            for (int l = 0; l < LL; ++l)
                                if (l > a && l < b) cost2 += static_cast<double>(v[l]);
                            cost2 += A.w2[i * L + pl];
                            if (cost + cost2 < best) {
                                best = cost + cost2;
                                pb = A.cur_from[s0 + cl] * L * L + cl * L + pl;
                            }
                        }
                    }
                    A.diag[lane] = best;
                    A.pdiag[lane] = pb;
                }
                __syncwarp();
                if (act) {
                    // The node's contribution to its parent replaces its own
                    // table (read above, not needed again).
                    const int lo = sl, s0 = slot * L;
                    double c = A.diag[s0 + lo];
                    int path = A.pdiag[s0 + lo];
#pragma unroll
                    for (int hi = 0; hi < LL; ++hi) {
                        if (hi < lo || hi >= L) continue;
                        if (hi > lo && !(c <= A.diag[s0 + hi])) { c = A.diag[s0 + hi]; path = A.pdiag[s0 + hi]; }
                        const int t = tri(L, lo, hi);
                        A.dist[i * TT + t] = c;
                        A.from[i * TT + t] = static_cast<unsigned short>(path);
                    }
                }
                __syncwarp();
            }
        }
        for (int i = N - 1; i >= 1; --i) {
            if (A.dep[i] != d) continue;
            const int p = par[i];
            for (int t = lane; t < TT; t += 32) A.dist[p * TT + t] += A.dist[i * TT + t];
            __syncwarp();
        }
    }
    // 4. Root range (lshape_thread.cuh:117-120): the first minimum in loop
    // order (lo, then hi), i.e. the smallest triangular index among equal
    // values -- a warp argmin; then the traceback one depth at a time.
    {
        double bv = __longlong_as_double(0x7ff0000000000000ll);  // +infinity: every finite entry is below it
        int bt = 1 << 30;
        for (int t = lane; t < TT; t += 32) {
            const double v = A.dist[t];
            if (v < bv) { bv = v; bt = t; }
        }
        for (int s = 16; s; s >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, bv, s);
            const int ot = __shfl_xor_sync(0xffffffffu, bt, s);
            if (ov < bv || (ov == bv && ot < bt)) { bv = ov; bt = ot; }
        }
        if (lane == 0) {
            if (bt >= TT) bt = 0;  // no entry below infinity: the sequential loop keeps index 0
            int lo = 0;
            while (lo + 1 < L && tri(L, lo + 1, lo + 1) <= bt) ++lo;
            A.range[0] = lo * L + (lo + bt - tri(L, lo, lo));
            if (!(bv < kInf)) set_error(T, kEInval, id);
        }
    }
    __syncwarp();
    for (int d = 1; d <= dmax; ++d) {
        for (int i = lane; i < N; i += 32) {
            if (i == 0 || A.dep[i] != d) continue;
            const int pr = A.range[par[i]];
            A.range[i] = A.from[i * TT + tri(L, pr / L, pr % L)] / (L * L);
        }
        __syncwarp();
    }
    // 5. Segment emission in node order (lshape_warp.cuh:215-240).
    int* out = P.routes + P.route_off[id];
    const long long cap = P.route_off[id + 1] - P.route_off[id];
    int next = 1;
    for (int b0 = 0; b0 < N; b0 += 32) {
        const int i = b0 + lane;
        int words = 0, x = 0, y = 0, px = 0, py = 0, cl = 0, pl = 0, minl = 0, maxl = 0;
        if (i < N) {
            x = A.xy[i] >> 16; y = A.xy[i] & 0xffff;
            minl = A.range[i] / L; maxl = A.range[i] % L;
            words = minl < maxl ? 2 : 0;
            if (i) {
                px = A.xy[par[i]] >> 16; py = A.xy[par[i]] & 0xffff;
                const int pr = A.range[par[i]];
                const int f = A.from[i * TT + tri(L, pr / L, pr % L)];
                cl = f / L % L; pl = f % L;
                words += (x == px || y == py) ? 2 : 6;
            }
        }
        int prefix = words;
        for (int s = 1; s < 32; s <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, prefix, s);
            if (lane >= s) prefix += o;
        }
        const int total = __shfl_sync(0xffffffffu, prefix, 31);
        if (next + total > cap) {
            if (lane == 0) set_error(T, kELimit, id);
            return;
        }
        if (i < N) {
            int* w = out + next + prefix - words;
            if (minl < maxl) { *w++ = cell_index(T, minl, x, y); *w++ = cell_index(T, maxl, x, y); }
            if (i) {
                if (x == px || y == py) {
                    *w++ = cell_index(T, cl, min(x, px), min(y, py));
                    *w++ = cell_index(T, cl, max(x, px), max(y, py));
                } else if (along_y(T, cl)) {
                    *w++ = cell_index(T, cl, x, y);   *w++ = cell_index(T, cl, x, py);
                    *w++ = cell_index(T, cl, x, py);  *w++ = cell_index(T, pl, x, py);
                    *w++ = cell_index(T, pl, x, py);  *w++ = cell_index(T, pl, px, py);
                } else {
                    *w++ = cell_index(T, cl, x, y);   *w++ = cell_index(T, cl, px, y);
                    *w++ = cell_index(T, cl, px, y);  *w++ = cell_index(T, pl, px, y);
                    *w++ = cell_index(T, pl, px, y);  *w++ = cell_index(T, pl, px, py);
                }
            }
        }
        next += total;
    }
    if (lane == 0) out[0] = next;
    __syncwarp();
    if (fuse_wires) commit_net_wires(T, P, id, stamp, 1, lane);
}

// Route one net of any size.  Ten-layer designs have nine routing layers: with
// the loops over them unrolled, 10K nets of 320x320x10, 4,690 of them beyond 32
// nodes, take 82.7 ms of stage in the persistent form and 76.3 per batch, against
// 93.8 and 89.7 with the layer count read at run time.
__device__ __forceinline__ void lshape_net(const Tables& T, const Plan& P, int id, int stamp, const Arena& A,
                                           int lane, bool fuse_wires) {
    if (T.L == 9) lshape_net_l<9>(T, P, id, stamp, A, lane, fuse_wires);
    else lshape_net_l<0>(T, P, id, stamp, A, lane, fuse_wires);
}

// ---- Packs: several nets, at most 32 tree nodes, by one warp ------------------
// The same DP with a lane per tree node for the tree's bookkeeping (coordinates,
// parents and depths live in registers and travel by shuffle), so a warp can
// take several small nets at once: their nodes form one forest, processed one
// depth at a time like a single tree.  Fixed costs of a net -- the dependent
// loads of its id, offsets, nodes and tables, the route store, the commit --
// are paid once per pack.
//
// What a depth costs decides the DP's time (a batch with fewer nets than warps
// lasts as long as its deepest net), so the step of a depth is short:
//   * best range through each layer: a suffix minimum along each row lo (lane
//     lo), then a minimum down each column (lane l), 18 comparisons in place of
//     the 45 ranges;
//   * via stacks at a corner: the difference of two prefix sums of the column
//     wherever those are exact (below), in place of a sum per candidate;
//   * depths by pointer jumping, a depth's nodes by one ballot.
// Same comparisons, tie-breaks, sums and emission order as lshape_net_l, so the
// same routes.  At 320x320x10, 120K nets, 63 batches: 5.8 ms of DP with a warp per
// net, the longest net 110 us; 2.7 ms with packs, the longest of them 65 us.
struct PackArena {
    double* dist;          // [nmax][TT] ranges; during a step the row minima; then what goes into the parent
    double* w1;            // [nmax][L] first leg (or straight) wire cost
    double* w2;            // [nmax][L] second leg wire cost
    double* stack;         // [nmax][2][L] column sums at the corners (x, py), (px, y): entry j = sum of layers 1..j-1
    unsigned short* from;  // [nmax][FS] column of a row minimum, then choice*L*L + curl*L + parl
    char* rough;           // [nmax][2] the column's sums are not exact
    double* diag;          // [32] best parent-layer cost (lane = slot * L + layer)
    int* pdiag;            // [32]
};
constexpr int kPackNodes = 32;
__host__ __device__ __forceinline__ int pack_from_stride(int L) { return (tri_count(L) + 1) & ~1; }
__host__ __device__ __forceinline__ size_t pack_arena_bytes(int L, int nmax) {
    const size_t per = size_t(tri_count(L)) * 8 + 4 * size_t(L) * 8 + size_t(pack_from_stride(L)) * 2 + 2;
    return (nmax * per + 32 * 12 + 15) & ~size_t(15);
}
// Nodes a warp's shared-memory arena holds: 16, or what 16 warps' arenas of an
// SM leave room for.
constexpr size_t kPackSmemLimit = 220 * 1024;
__host__ __device__ __forceinline__ int pack_nmax(int L) {
    int n = 16;
    while (n > 2 && pack_arena_bytes(L, n) * 16 > kPackSmemLimit) --n;
    return n;
}
__device__ __forceinline__ PackArena pack_arena(char* p, int L, int nmax) {
    PackArena A;
    A.dist = reinterpret_cast<double*>(p); p += size_t(nmax) * tri_count(L) * 8;
    A.w1 = reinterpret_cast<double*>(p); p += size_t(nmax) * L * 8;
    A.w2 = reinterpret_cast<double*>(p); p += size_t(nmax) * L * 8;
    A.stack = reinterpret_cast<double*>(p); p += size_t(nmax) * 2 * L * 8;
    A.diag = reinterpret_cast<double*>(p); p += 32 * 8;
    A.pdiag = reinterpret_cast<int*>(p); p += 32 * 4;
    A.from = reinterpret_cast<unsigned short*>(p); p += size_t(nmax) * pack_from_stride(L) * 2;
    A.rough = p;
    return A;
}

// The trees of a pack: lane q < nodes holds tree node q of the forest.
struct Pack {
    int nets, nodes;
    int id;          // lane's net (nets without nodes have no lane)
    int first, count;// lane's net: its root's lane, its nodes
    int x, y, lay;   // lay = L: Steiner point
    int par;         // parent's lane, -1 at a root (and beyond the nodes)
    long long out, cap;  // lane's net: route words
};
// `k` <= 16 nets -- ids[0..k), or first_id on where ids is null --, at most 32
// nodes together.
__device__ __forceinline__ Pack load_pack(const Tables& T, const Plan& P, const int* ids, int first_id, int k, int lane) {
    Pack K;
    K.nets = k;
    int id = 0, off = 0, n = 0;
    if (lane < k) {
        id = ids ? ids[lane] : first_id + lane;
        off = P.node_off[id];
        n = P.node_off[id + 1] - off;
    }
    int incl = n;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    K.nodes = __shfl_sync(0xffffffffu, incl, k - 1);
    int j = 0;  // the net of node `lane`: the first with incl > lane
#pragma unroll
    for (int step = 8; step; step >>= 1) {
        const int v = __shfl_sync(0xffffffffu, incl, j + step - 1);
        if (j + step - 1 < k && v <= lane) j += step;
    }
    j = min(j, k - 1);
    K.id = __shfl_sync(0xffffffffu, id, j);
    K.count = __shfl_sync(0xffffffffu, n, j);
    K.first = __shfl_sync(0xffffffffu, incl, j) - K.count;
    off = __shfl_sync(0xffffffffu, off, j);
    K.x = K.y = K.lay = 0;
    K.par = -1;
    K.out = K.cap = 0;
    if (lane < K.nodes) {
        const int v = P.nodes[off + lane - K.first], p = P.parents[off + lane - K.first];
        K.out = P.route_off[K.id];
        K.cap = P.route_off[K.id + 1] - K.out;
        cell_position(T, v, K.lay, K.x, K.y);
        if (p >= 0) K.par = K.first + p;
    }
    return K;
}

constexpr int kUnroll = 3;
template <int LC>
__device__ __forceinline__ void route_pack_l(const Tables& T, const Plan& P, const Pack& K, int stamp,
                                             const PackArena& A, int lane, bool commit) {
    const int L = LC > 0 ? LC : T.L, TT = tri_count(L), FS = pack_from_stride(L);
    constexpr int LL = LC > 0 ? LC : kMaxLayers;  // static bound of the layer loops
    constexpr unsigned kAll = 0xffffffffu;
    const int M = K.nodes;
    if (M == 0) return;
    // Depths by pointer jumping (trees of at most 32 nodes: five rounds).
    int dep = K.par >= 0 ? 1 : 0;
    for (int anc = K.par; __any_sync(kAll, anc >= 0);) {
        const int od = __shfl_sync(kAll, dep, anc & 31), oa = __shfl_sync(kAll, anc, anc & 31);
        if (anc >= 0) { dep += od; anc = oa; }
    }
    if (lane >= M) dep = -1;
    const int dmax = __reduce_max_sync(kAll, dep);
    const int xy = (K.x << 16) | K.y;
    const int pxy = __shfl_sync(kAll, xy, K.par & 31);
    // 1. Gather every cost the DP reads.  Each lane takes two (node, layer)
    // items per pass and issues all their loads before any arena store; the
    // corner columns wait in the node's (still unused) range table.
    for (int q0 = 0; q0 < M * L; q0 += 64) {
        float vn[2], va[2], vb[2];
        double w1[2], w2[2];
        int kind[2];  // 0: none, 1: node only, 2: straight edge, 3: L-shaped edge
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + 32 * u + lane, i = min(q / L, M - 1), l = q - q / L * L;
            const int c = __shfl_sync(kAll, xy, i), pc = __shfl_sync(kAll, pxy, i), pa = __shfl_sync(kAll, K.par, i);
            kind[u] = 0;
            vn[u] = va[u] = vb[u] = 0.f;
            w1[u] = w2[u] = 0.0;
            if (q >= M * L) continue;
            const int x = c >> 16, y = c & 0xffff;
            const bool ay = along_y(T, l);
            const int base = layer_base(T, l);
            vn[u] = T.vcost[base + (ay ? x * T.yp + y : y * T.xp + x)];
            kind[u] = 1;
            if (pa >= 0) {
                const int px = pc >> 16, py = pc & 0xffff;
                const int minx = min(x, px), maxx = max(x, px), miny = min(y, py), maxy = max(y, py);
                const bool straight = x == px || y == py;
                const int lo = ay ? miny : minx, hi = ay ? maxy : maxx;
                const int t1 = base + (ay ? x * T.yp : y * T.xp), t2 = base + (ay ? px * T.yp : py * T.xp);
                const bool valid = !straight || (ay ? x == px : y == py);
                if (valid) w1[u] = T.presum[t1 + hi] - T.presum[t1 + lo];
                kind[u] = 2;
                if (!straight) {
                    w2[u] = T.presum[t2 + hi] - T.presum[t2 + lo];
                    va[u] = T.vcost[base + (ay ? x * T.yp + py : py * T.xp + x)];
                    vb[u] = T.vcost[base + (ay ? px * T.yp + y : y * T.xp + px)];
                    kind[u] = 3;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int q = q0 + 32 * u + lane, i = q / L, l = q - i * L;
            if (kind[u] >= 1) reinterpret_cast<float*>(A.from + i * FS)[l] = vn[u];
            if (kind[u] >= 2) A.w1[q] = w1[u];
            if (kind[u] == 3) {
                A.w2[q] = w2[u];
                float* col = reinterpret_cast<float*>(A.dist + i * TT);
                col[l] = va[u];
                col[L + l] = vb[u];
            }
        }
    }
    __syncwarp();
    // 2a. Column sums at the corners.  The sum of layers a+1..b-1 is wanted as
    // the sequential loop adds it; it is the difference of two prefix sums
    // whenever no addition of the column rounds, which holds when the values'
    // exponents span at most 25 bits (24-bit mantissas, at most 8 terms: every
    // partial sum fits the 53 bits of a double).  Other columns are summed
    // where they are used.
    for (int q = lane; q < 2 * M; q += 32) {
        const int i = q >> 1;
        const float* col = reinterpret_cast<const float*>(A.dist + i * TT) + (q & 1) * L;
        double* out = A.stack + size_t(q) * L;
        double acc = 0;
        unsigned emin = 255, emax = 0;
        bool odd = false;
#pragma unroll kUnroll
        for (int l = 1; l < LL; ++l) {
            if (l >= L) continue;
            out[l] = acc;
            const float v = col[l];
            const unsigned b = __float_as_uint(v), e = b >> 23;
            if (l < L - 1 && b != 0u) {
                odd |= e == 0 || e >= 255;  // denormal, negative, infinite or NaN
                emin = min(emin, e);
                emax = max(emax, e);
                acc = acc + static_cast<double>(v);
            }
        }
        A.rough[q] = odd || emax > emin + 25;
    }
    __syncwarp();
    // 2b. Via stacks at every node (lshape_thread.cuh:40-50).
    for (int q0 = 0; q0 < M * L; q0 += 32) {
        const int q = q0 + lane, i = min(q / L, M - 1), lo = q - q / L * L;
        const int fixed = __shfl_sync(kAll, K.lay, i);
        if (q >= M * L) continue;
        const float* vn = reinterpret_cast<const float*>(A.from + i * FS);
        double acc = 0;
        double* row = A.dist + i * TT + tri(L, lo, lo) - lo;
#pragma unroll kUnroll
        for (int hi = 0; hi < LL; ++hi) {
            if (hi < lo || hi >= L) continue;
            if (hi > lo) acc = acc + static_cast<double>(vn[hi - 1]);
            row[hi] = (fixed < L && (lo > fixed || hi < fixed)) ? kInf : acc;
        }
    }
    __syncwarp();
    // 3. Children into parents (lshape_thread.cuh:51-115), one depth at a time
    // from the deepest, up to 32 / L nodes at once (lane = slot * L + layer);
    // then every node of the depth, in descending order, adds its table into
    // its parent: exactly the sequential loop's additions.
    const int S = max(1, 32 / L);
    const int slot = lane / L, sl = lane - slot * L, s0 = min(slot, S - 1) * L;
    for (int d = dmax; d >= 1; --d) {
        const unsigned level = __ballot_sync(kAll, dep == d);
        for (unsigned at = level; at;) {
            int i = -1;
            for (int k = 0; k < S; ++k) {
                if (k == slot && at) i = __ffs(at) - 1;
                at &= at - 1;  // 0 stays 0
            }
            const bool act = i >= 0;
            const int ii = max(i, 0);
            const int c = __shfl_sync(kAll, xy, ii), pc = __shfl_sync(kAll, pxy, ii);
            const int x = c >> 16, y = c & 0xffff, px = pc >> 16, py = pc & 0xffff;
            double* dist = A.dist + ii * TT;
            unsigned short* from = A.from + ii * FS;
            if (act) {
                // Row sl: its first minimum over columns hi >= h, for every h.
                const int row = tri(L, sl, sl) - sl;
                double best = __longlong_as_double(0x7ff0000000000000ll);
                int bh = 0;
#pragma unroll
                for (int hi = LL - 1; hi >= 0; --hi) {
                    if (hi < sl || hi >= L) continue;
                    const double v = dist[row + hi];
                    if (v <= best) { best = v; bh = hi; }
                    dist[row + hi] = best;
                    from[row + hi] = static_cast<unsigned short>(bh);
                }
            }
            __syncwarp();
            double cur = kInf;
            int bf = 0;
            if (act) {
                // Column sl: the first row with the least of them.
                int bl = -1;
#pragma unroll
                for (int lo = 0; lo < LL; ++lo) {
                    if (lo > sl || lo >= L) continue;
                    const double v = dist[tri(L, lo, sl)];
                    if (v < cur) { cur = v; bl = lo; }
                }
                if (bl >= 0) bf = bl * L + from[tri(L, bl, sl)];
            }
            // Arrival on parent layer sl (first leg on cl, corner, second leg on sl).
            const double reach = act ? cur + A.w1[ii * L + sl] : 0.0;
            const bool straight = x == px || y == py;
            double best = kInf;
            int bc = -1;
            if (act && straight && (along_y(T, sl) ? x == px : y == py)) { best = reach; bc = sl; }
            if (__any_sync(kAll, act && !straight)) {
                const double leg2 = act ? A.w2[ii * L + sl] : 0.0;
                // The corner column depends on the first leg's direction, the other one than sl's.
                const int side = along_y(T, sl) ? 1 : 0;
                const double* col = A.stack + (2 * size_t(ii) + side) * L;
                const bool rough = act && !straight && A.rough[2 * ii + side];
                const int cx = side ? px : x, cy = side ? y : py;
#pragma unroll kUnroll
                for (int cl = 0; cl < LL; ++cl) {
                    if (cl >= L) continue;
                    const double cost = __shfl_sync(kAll, reach, s0 + cl);
                    if (!act || straight || ((cl ^ sl) & 1) == 0) continue;
                    const int a = min(cl, sl), b = max(cl, sl);
                    double cost2 = col[b] - col[a + 1];
                    if (rough) {
                        cost2 = 0;
                        for (int l = a + 1; l < b; ++l)
                            cost2 += static_cast<double>(T.vcost[slot_index(T, l, cx, cy)]);
                    }
                    cost2 += leg2;
                    if (cost + cost2 < best) { best = cost + cost2; bc = cl; }
                }
            }
            const int cf = __shfl_sync(kAll, bf, s0 + max(bc, 0));
            if (act) {
                A.diag[lane] = best;
                A.pdiag[lane] = bc >= 0 ? cf * L * L + bc * L + sl : 0;
            }
            __syncwarp();
            if (act) {
                // The node's contribution to its parent replaces its own
                // table (read above, not needed again).
                const int row = tri(L, sl, sl) - sl;
                double cc = A.diag[s0 + sl];
                int path = A.pdiag[s0 + sl];
#pragma unroll kUnroll
                for (int hi = 0; hi < LL; ++hi) {
                    if (hi < sl || hi >= L) continue;
                    const double v = A.diag[s0 + hi];
                    if (hi > sl && !(cc <= v)) { cc = v; path = A.pdiag[s0 + hi]; }
                    dist[row + hi] = cc;
                    from[row + hi] = static_cast<unsigned short>(path);
                }
            }
            __syncwarp();
        }
        for (unsigned m = level; m;) {
            const int i = 31 - __clz(m);
            m ^= 1u << i;
            const int p = __shfl_sync(kAll, K.par, i);
            for (int t = lane; t < TT; t += 32) A.dist[p * TT + t] += A.dist[i * TT + t];
        }
        __syncwarp();
    }
    // 4. Root ranges (lshape_thread.cuh:117-120): the first minimum in loop
    // order (lo, then hi), lane = slot * L + lo; then the traceback one depth
    // at a time.
    int range = 0, f = 0;
    for (unsigned at = __ballot_sync(kAll, dep == 0); at;) {
        int i = -1;
        for (int k = 0; k < S; ++k) {
            if (k == slot && at) i = __ffs(at) - 1;
            at &= at - 1;
        }
        double bv = __longlong_as_double(0x7ff0000000000000ll);
        int br = 0;
        if (i >= 0) {
            const double* row = A.dist + i * TT + tri(L, sl, sl) - sl;
#pragma unroll kUnroll
            for (int hi = 0; hi < LL; ++hi) {
                if (hi < sl || hi >= L) continue;
                const double v = row[hi];
                if (v < bv) { bv = v; br = sl * L + hi; }
            }
        }
        double best = __longlong_as_double(0x7ff0000000000000ll);
        int rr = 0;  // no entry below infinity: the sequential loop keeps range (0, 0)
#pragma unroll kUnroll
        for (int lo = 0; lo < LL; ++lo) {
            if (lo >= L) continue;
            const double v = __shfl_sync(kAll, bv, s0 + lo);
            const int r = __shfl_sync(kAll, br, s0 + lo);
            if (v < best) { best = v; rr = r; }
        }
        // Each slot's result to its root's lane.
        for (int k = 0; k < S; ++k) {
            const int to = __shfl_sync(kAll, i, k * L), r = __shfl_sync(kAll, rr, k * L);
            const double v = __shfl_sync(kAll, best, k * L);
            if (lane == to) {
                range = r;
                if (!(v < kInf)) set_error(T, kEInval, K.id);
            }
        }
    }
    for (int d = 1; d <= dmax; ++d) {
        const int pr = __shfl_sync(kAll, range, K.par & 31);
        if (dep == d) {
            f = A.from[lane * FS + tri(L, pr / L, pr % L)];
            range = f / (L * L);
        }
    }
    // 5. Segments in node order (lshape_warp.cuh:215-240), a lane per node.
    const int minl = range / L, maxl = range % L, cl = f / L % L, pl = f % L;
    const int x = K.x, y = K.y, px = pxy >> 16, py = pxy & 0xffff;
    const bool edge = K.par >= 0, straight = x == px || y == py;
    int words = 0;
    if (lane < M) words = (minl < maxl ? 2 : 0) + (edge ? (straight ? 2 : 6) : 0);
    int incl = words;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(kAll, incl, d);
        if (lane >= d) incl += o;
    }
    const int start = __shfl_sync(kAll, incl - words, K.first & 31);  // words of the nets before this one
    const int total = __shfl_sync(kAll, incl, (K.first + K.count - 1) & 31) - start;
    const bool fits = 1 + total <= K.cap;
    const bool mine = lane < M && fits;
    // The corner of an L-shaped edge: the end of the first leg.
    const int cx = along_y(T, cl) ? x : px, cy = along_y(T, cl) ? py : y;
    if (lane < M && lane == K.first) {
        if (fits) P.routes[K.out] = 1 + total;
        else set_error(T, kELimit, K.id);
    }
    if (mine) {
        int* w = P.routes + K.out + 1 + (incl - words - start);
        if (minl < maxl) { *w++ = cell_index(T, minl, x, y); *w++ = cell_index(T, maxl, x, y); }
        if (edge && straight) {
            *w++ = cell_index(T, cl, min(x, px), min(y, py));
            *w++ = cell_index(T, cl, max(x, px), max(y, py));
        } else if (edge) {
            const int corner = cell_index(T, cl, cx, cy), second = cell_index(T, pl, cx, cy);
            *w++ = cell_index(T, cl, x, y); *w++ = corner;
            *w++ = corner;                  *w++ = second;
            *w++ = second;                  *w++ = cell_index(T, pl, px, py);
        }
    }
    if (!commit) return;
    // The wires just emitted, from registers: the first leg (or the straight
    // run) of every lane, then the second legs.
    double length = 0;
#pragma unroll
    for (int leg = 0; leg < 2; ++leg) {
        WireRun R;
        if (mine && edge && (leg == 0 || !straight)) {
            const int l = leg ? pl : cl, ax = leg ? cx : x, ay = leg ? cy : y;
            const int bx = leg || straight ? px : cx, by = leg || straight ? py : cy;
            R = run_between(T, l, ax, ay, bx, by);
            const int a = cell_index(T, l, ax, ay), b = cell_index(T, l, bx, by);
            stamp_ends(T, R, a, b, stamp);
            length += R.length;
            if (R.skew) commit_skew(T, a, b, stamp, 1);
        }
        commit_runs(T, R.first, R.skew ? 0 : R.n, stamp, 1, lane);
    }
    add_wirelength(T, length, 1, lane);
}

__device__ __forceinline__ void route_pack(const Tables& T, const Plan& P, const Pack& K, int stamp, const PackArena& A,
                                           int lane, bool commit) {
    if (T.L == 9) route_pack_l<9>(T, P, K, stamp, A, lane, commit);
    else route_pack_l<0>(T, P, K, stamp, A, lane, commit);
}

}  // namespace grb
