// softmin.cuh -- temperature-tau soft-min version of the L-shape routing DAG
// and its hand-written adjoint.
//
// The DAG is the L-shape DP of lshape_thread.cuh:18-171 (and of lshape.cuh
// here): per tree node a table of via-stack layer ranges [lo, hi]; per tree
// edge the child's best range through each layer (cur), the arrival cost on
// each parent layer (a straight wire, or an L through one corner with its via
// stack), and the arrival over each parent range.  Every `min` of that DP is
// replaced by
//     smin(v) = m - tau * log(sum_k exp(-(v_k - m) / tau)),   m = min_k v_k,
// whose gradient is softmax(-v / tau); as tau -> 0 it becomes the hard min and
// the gradient the indicator of the chosen candidate.  Values >= kSoftAbsent
// (the hard DP's 1e22 infinity) are candidates that do not exist.
//
// Total routed cost F = sum over nets of the soft root value, with cost
// tables computed from the inputs in the working precision (fp32 or fp64):
//   wcost[c] = incr(c, 1) + unit_wire[c] * edge_len(c)
//   vcost[c] = half-split incr of the two edges a via lands between + unit_via
//   incr(c, k) = min(1e12, (of(d + k) - of(d)) * w_l),
//   of(d) = exp(0.5 * (d - capacity[c]))                        (capacity > 1e-3)
// (full_update.cuh:9-83 without the float narrowing, so FD checks in fp64 are
// smooth).  Demand d is the context's current demand, held fixed.
//
// B200 form: the hard DP's packs (lshape.cuh) -- one warp takes several nets,
// at most SoftArena's nodes together, a lane per tree node for the bookkeeping
// and lane = slot * L + layer for the steps of a depth, with every table of the
// pack in shared memory.  A soft minimum over nested sets is accumulated as a
// running pair (m, s) = (minimum, sum of exp(-(v - m) / tau)): suffixes of a
// row, then a column of them, give cur[l] with 18 exponentials a lane in place
// of up to 25 per layer twice over, and the running minimum of diag gives the
// nine ranges of a row with nine.  The adjoint walks the same running pairs
// backwards with the exponentials the forward walk left.  The adjoint of a
// wire or via cost is summed over its candidates inside the warp, so a tree
// edge updates each cell of the tables once.  All tables are track by track
// like the routing tables; inputs and gradients are converted on the way.  Nets
// beyond kPackNodes are walked by one thread each (soft_net_forward, _backward).
//
// Thread per net with the tables in local arrays (the form before, 120K nets
// at 320x320x10, fp32, tau = 1): forward 3.1 ms, adjoint 46 ms; now 0.7 and 2.3 ms.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "lshape.cuh"

namespace grb {

constexpr double kSoftAbsent = 1e21;

template <class T> __device__ __forceinline__ T s_exp(T v);
template <> __device__ __forceinline__ float s_exp<float>(float v) { return expf(v); }
template <> __device__ __forceinline__ double s_exp<double>(double v) { return exp(v); }
template <class T> __device__ __forceinline__ T s_log(T v);
template <> __device__ __forceinline__ float s_log<float>(float v) { return logf(v); }
template <> __device__ __forceinline__ double s_log<double>(double v) { return log(v); }

template <class T>
struct Soft {
    const T* cap;        // [slots] capacity
    const T* uw;         // [slots] unit wire cost per edge
    T uv;                // unit via cost
    T tau, inv_tau;
    T* vc;               // [slots] via cost
    T* P;                // [slots] exclusive prefix of the wire costs along each track
    T* dP;               // [slots] adjoint of P
    T* dvc;              // [slots] adjoint of vc
    T* slot;             // scratch of nets beyond a pack: 2 * L * L values per node
    T* net_cost;         // [n_nets] soft root value of each net
};

template <class T>
__device__ __forceinline__ T soft_of(const Tables& Tb, T cap, T d) {
    const T scale = static_cast<T>(Tb.of_scale);
    if (cap > static_cast<T>(0.001)) {
        const T a = static_cast<T>(0.5) * (d - cap), b = scale * static_cast<T>(0.5) * (d - cap);
        return s_exp<T>(a < b ? a : b);
    }
    if (d > 0) {
        const T a = static_cast<T>(1.5) * d, b = scale * static_cast<T>(1.5) * d;
        return s_exp<T>(a < b ? a : b);
    }
    return 0;
}
// d of / d cap.
template <class T>
__device__ __forceinline__ T soft_of_dcap(const Tables& Tb, T cap, T d) {
    if (!(cap > static_cast<T>(0.001))) return 0;
    const T scale = static_cast<T>(Tb.of_scale);
    const T a = static_cast<T>(0.5) * (d - cap), b = scale * static_cast<T>(0.5) * (d - cap);
    return a < b ? static_cast<T>(-0.5) * s_exp<T>(a) : -scale * static_cast<T>(0.5) * s_exp<T>(b);
}
// Increments of a whole and of half a unit on the edge at slot c of layer l,
// and (deriv) their derivatives with respect to the capacity.
template <class T>
struct SoftTerms {
    T one, half;
};
template <class T>
__device__ __forceinline__ SoftTerms<T> soft_terms(const Tables& Tb, const Soft<T>& S, int c, int l) {
    const T d = static_cast<T>(Tb.demand[c]) * static_cast<T>(0.5), cap = S.cap[c], w = static_cast<T>(Tb.short_costs[l]);
    const T o0 = soft_of<T>(Tb, cap, d), top = static_cast<T>(1e12);
    const T one = (soft_of<T>(Tb, cap, d + 1) - o0) * w, half = (soft_of<T>(Tb, cap, d + static_cast<T>(0.5)) - o0) * w;
    return {one < top ? one : top, half < top ? half : top};
}
template <class T>
__device__ __forceinline__ SoftTerms<T> soft_terms_dcap(const Tables& Tb, const Soft<T>& S, int c, int l) {
    const T d = static_cast<T>(Tb.demand[c]) * static_cast<T>(0.5), cap = S.cap[c], w = static_cast<T>(Tb.short_costs[l]);
    const SoftTerms<T> v = soft_terms<T>(Tb, S, c, l);
    const T o0 = soft_of_dcap<T>(Tb, cap, d), top = static_cast<T>(1e12);
    return {v.one < top ? (soft_of_dcap<T>(Tb, cap, d + 1) - o0) * w : static_cast<T>(0),
            v.half < top ? (soft_of_dcap<T>(Tb, cap, d + static_cast<T>(0.5)) - o0) * w : static_cast<T>(0)};
}

// Exclusive prefix (kUp) or suffix sums of the warp's v behind `carry`, which
// moves on by the warp's total.  fp32: accumulated in double, rounded once (a
// wire's cost is the difference of two sums, divided by tau).  fp64: added one
// by one in position order, whose rounding errors stay common to the sums of
// neighbouring positions.
template <bool kUp>
__device__ __forceinline__ float soft_scan(float v, double& carry, int lane) {
    double incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double o = kUp ? __shfl_up_sync(0xffffffffu, incl, d) : __shfl_down_sync(0xffffffffu, incl, d);
        if (kUp ? lane >= d : lane + d < 32) incl += o;
    }
    const double next = kUp ? __shfl_up_sync(0xffffffffu, incl, 1) : __shfl_down_sync(0xffffffffu, incl, 1);
    const float out = static_cast<float>(lane == (kUp ? 0 : 31) ? carry : carry + next);
    carry += __shfl_sync(0xffffffffu, incl, kUp ? 31 : 0);
    return out;
}
template <bool kUp>
__device__ __forceinline__ double soft_scan(double v, double& carry, int lane) {
    double out = 0;
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
        const int j = kUp ? k : 31 - k;
        if (lane == j) out = carry;
        carry += __shfl_sync(0xffffffffu, v, j);
    }
    return out;
}

// Via costs and the exclusive wire-cost prefix of one track, by one warp: lanes
// over the positions, the prefix of each 32 by a shuffle scan.
template <class T>
__device__ __forceinline__ void soft_tables_track(const Tables& Tb, const Soft<T>& S, int t, int lane) {
    const Track K = track_of(Tb, t);
    const int* elen = along_y(Tb, K.l) ? Tb.ylen : Tb.xlen;
    double carry = 0;
    T last_one = 0, last_half = 0;
    for (int p0 = 0; p0 < K.len; p0 += 32) {
        const int p = p0 + lane, c = K.base + p;
        SoftTerms<T> v{0, 0};
        T w = 0;
        if (p < K.len) {
            v = soft_terms<T>(Tb, S, c, K.l);
            w = v.one + S.uw[c] * static_cast<T>(p < K.len - 1 ? elen[p] : 0);
        }
        T one = __shfl_up_sync(0xffffffffu, v.one, 1), half = __shfl_up_sync(0xffffffffu, v.half, 1);
        if (lane == 0) { one = last_one; half = last_half; }
        last_one = __shfl_sync(0xffffffffu, v.one, 31);
        last_half = __shfl_sync(0xffffffffu, v.half, 31);
        const T before = soft_scan<true>(w, carry, lane);
        if (p < K.len) {
            S.vc[c] = (p == 0 ? v.one : p == K.len - 1 ? one : v.half + half) + S.uv;
            S.P[c] = before;
        }
    }
}

// The adjoints of one track's wire costs (dwc[j] = sum over later positions of
// dP, since P[i] = sum over j < i of wc[j]) and via costs, through the cost
// model to the capacity and the unit wire cost of each edge (written over vc
// and P, which the adjoint no longer needs).  Returns the lane's part of the
// sum of dvc, in double.
template <class T>
__device__ __forceinline__ double soft_chain_track(const Tables& Tb, const Soft<T>& S, int t, int lane, T* dcap, T* duw) {
    const Track K = track_of(Tb, t);
    const int* elen = along_y(Tb, K.l) ? Tb.ylen : Tb.xlen;
    double carry = 0, sum = 0;
    for (int p0 = (K.len - 1) / 32 * 32; p0 >= 0; p0 -= 32) {
        const int p = p0 + lane, c = K.base + p;
        const bool in = p < K.len;
        const T g = in ? S.dP[c] : static_cast<T>(0);
        const T dw = soft_scan<false>(g, carry, lane);
        if (in) {
            const T dv = S.dvc[c], next = p + 1 < K.len ? S.dvc[c + 1] : static_cast<T>(0);
            const SoftTerms<T> e = soft_terms_dcap<T>(Tb, S, c, K.l);
            T gc = dw * e.one;
            if (p == 0) gc += dv * e.one;
            else if (p < K.len - 1) gc += dv * e.half;
            if (p + 1 == K.len - 1) gc += next * e.one;
            else if (p + 1 < K.len - 1) gc += next * e.half;
            dcap[c] = gc;
            duw[c] = dw * static_cast<T>(p < K.len - 1 ? elen[p] : 0);
            sum += static_cast<double>(dv);
        }
    }
    return sum;
}

// Soft minimum of v[0..n) (entries >= kSoftAbsent do not exist); writes the
// softmax weights into w when given.  Returns kSoftAbsent * 10 when empty.
template <class T>
__device__ __forceinline__ T smin(const T* v, int n, T tau, T* w) {
    T m = static_cast<T>(kSoftAbsent);
    for (int k = 0; k < n; ++k) m = v[k] < m ? v[k] : m;
    if (!(m < static_cast<T>(kSoftAbsent))) {
        if (w) for (int k = 0; k < n; ++k) w[k] = 0;
        return static_cast<T>(kSoftAbsent) * 10;
    }
    T s = 0;
    for (int k = 0; k < n; ++k)
        if (v[k] < static_cast<T>(kSoftAbsent)) s += s_exp<T>(-(v[k] - m) / tau);
    if (w)
        for (int k = 0; k < n; ++k) w[k] = v[k] < static_cast<T>(kSoftAbsent) ? s_exp<T>(-(v[k] - m) / tau) / s : 0;
    return m - tau * s_log<T>(s);
}

template <class T>
__device__ __forceinline__ T soft_wire(const Tables& Tb, const Soft<T>& S, int l, int xmin, int xmax, int ymin, int ymax) {
    return S.P[slot_index(Tb, l, xmax, ymax)] - S.P[slot_index(Tb, l, xmin, ymin)];
}
template <class T>
__device__ __forceinline__ void soft_wire_adj(const Tables& Tb, const Soft<T>& S, int l, int xmin, int xmax, int ymin,
                                              int ymax, T g) {
    if (g == 0 || (xmin == xmax && ymin == ymax)) return;
    atomicAdd(S.dP + slot_index(Tb, l, xmax, ymax), g);
    atomicAdd(S.dP + slot_index(Tb, l, xmin, ymin), -g);
}

// Candidate set of one tree edge: the arrival on parent layer pl from child
// layer cl.  Straight edges have the single candidate cl == pl (layers of the
// edge's direction); L edges every cl of the other parity (lshape_thread.cuh).
struct SoftEdge {
    int x, y, px, py, minx, maxx, miny, maxy;
    bool straight;
};

// Candidate cost excluding cur[cl]; NaN-free, absent when not a candidate.
template <class T>
__device__ __forceinline__ T soft_leg(const Tables& Tb, const Soft<T>& S, const SoftEdge& E, int cl, int pl) {
    const int L = Tb.L;
    (void)L;
    if (E.straight) {
        if (cl != pl) return static_cast<T>(kSoftAbsent) * 10;
        if (!along_y(Tb, cl) && E.y != E.py) return static_cast<T>(kSoftAbsent) * 10;
        if (along_y(Tb, cl) && E.x != E.px) return static_cast<T>(kSoftAbsent) * 10;
        return soft_wire<T>(Tb, S, cl, E.minx, E.maxx, E.miny, E.maxy);
    }
    if (((cl ^ pl) & 1) == 0) return static_cast<T>(kSoftAbsent) * 10;
    T cost = along_y(Tb, cl) ? soft_wire<T>(Tb, S, cl, E.x, E.x, E.miny, E.maxy)
                             : soft_wire<T>(Tb, S, cl, E.minx, E.maxx, E.y, E.y);
    T cost2 = 0;
    for (int l = min(cl, pl) + 1; l < max(cl, pl); ++l)
        cost2 += along_y(Tb, cl) ? S.vc[slot_index(Tb, l, E.x, E.py)] : S.vc[slot_index(Tb, l, E.px, E.y)];
    cost2 += along_y(Tb, pl) ? soft_wire<T>(Tb, S, pl, E.px, E.px, E.miny, E.maxy)
                             : soft_wire<T>(Tb, S, pl, E.minx, E.maxx, E.py, E.py);
    return cost + cost2;
}
template <class T>
__device__ __forceinline__ void soft_leg_adj(const Tables& Tb, const Soft<T>& S, const SoftEdge& E, int cl, int pl, T g) {
    if (g == 0) return;
    if (E.straight) {
        soft_wire_adj<T>(Tb, S, cl, E.minx, E.maxx, E.miny, E.maxy, g);
        return;
    }
    if (along_y(Tb, cl)) soft_wire_adj<T>(Tb, S, cl, E.x, E.x, E.miny, E.maxy, g);
    else soft_wire_adj<T>(Tb, S, cl, E.minx, E.maxx, E.y, E.y, g);
    for (int l = min(cl, pl) + 1; l < max(cl, pl); ++l)
        atomicAdd(S.dvc + (along_y(Tb, cl) ? slot_index(Tb, l, E.x, E.py) : slot_index(Tb, l, E.px, E.y)), g);
    if (along_y(Tb, pl)) soft_wire_adj<T>(Tb, S, pl, E.px, E.px, E.miny, E.maxy, g);
    else soft_wire_adj<T>(Tb, S, pl, E.minx, E.maxx, E.py, E.py, g);
}

__device__ __forceinline__ SoftEdge soft_edge(const Tables& Tb, int node, int par) {
    SoftEdge E;
    E.x = node / Tb.Y % Tb.X; E.y = node % Tb.Y;
    E.px = par / Tb.Y % Tb.X; E.py = par % Tb.Y;
    E.minx = min(E.x, E.px); E.maxx = max(E.x, E.px); E.miny = min(E.y, E.py); E.maxy = max(E.y, E.py);
    E.straight = E.x == E.px || E.y == E.py;
    return E;
}

// Forward DP of one net into dist[N][L][L] (its final range tables); returns
// the soft root value.
template <class T>
__device__ T soft_net_forward(const Tables& Tb, const Soft<T>& S, const Plan& P, int id, T* dist) {
    const int L = Tb.L, LL = L * L;
    const int nb = P.node_off[id], N = P.node_off[id + 1] - nb;
    const T absent = static_cast<T>(kSoftAbsent) * 10;
    for (int i = 0; i < N; ++i) {
        const int v = P.nodes[nb + i], lp = v / Tb.XY, x = v / Tb.Y % Tb.X, y = v % Tb.Y;
        T* d = dist + size_t(i) * LL;
        for (int lo = 0; lo < L; ++lo) {
            d[lo * L + lo] = 0;
            for (int hi = lo + 1; hi < L; ++hi) d[lo * L + hi] = d[lo * L + hi - 1] + S.vc[slot_index(Tb, hi - 1, x, y)];
            for (int hi = 0; hi < lo; ++hi) d[lo * L + hi] = absent;
            if (lp < L)
                for (int hi = lo; hi < L; ++hi)
                    if (lo > lp || hi < lp) d[lo * L + hi] = absent;
        }
    }
    T vals[kMaxLayers * kMaxLayers];
    for (int i = N - 1; i >= 1; --i) {
        const int p = P.parents[nb + i];
        const SoftEdge E = soft_edge(Tb, P.nodes[nb + i], P.nodes[nb + p]);
        const T* di = dist + size_t(i) * LL;
        T cur[kMaxLayers], diag[kMaxLayers];
        for (int l = 0; l < L; ++l) {
            int n = 0;
            for (int lo = 0; lo <= l; ++lo)
                for (int hi = l; hi < L; ++hi) vals[n++] = di[lo * L + hi];
            cur[l] = smin<T>(vals, n, S.tau, nullptr);
        }
        for (int pl = 0; pl < L; ++pl) {
            for (int cl = 0; cl < L; ++cl) vals[cl] = cur[cl] + soft_leg<T>(Tb, S, E, cl, pl);
            diag[pl] = smin<T>(vals, L, S.tau, nullptr);
        }
        T* dp = dist + size_t(p) * LL;
        for (int lo = 0; lo < L; ++lo)
            for (int hi = lo; hi < L; ++hi) dp[lo * L + hi] += smin<T>(diag + lo, hi - lo + 1, S.tau, nullptr);
    }
    int n = 0;
    for (int lo = 0; lo < L; ++lo)
        for (int hi = lo; hi < L; ++hi) vals[n++] = dist[lo * L + hi];
    return smin<T>(vals, n, S.tau, nullptr);
}

// Adjoint of one net: recomputes the forward ranges, then propagates g (the
// gradient of F with respect to the net's root value) to the tables.
template <class T>
__device__ void soft_net_backward(const Tables& Tb, const Soft<T>& S, const Plan& P, int id, T* dist, T* gd, T g) {
    const int L = Tb.L, LL = L * L;
    const int nb = P.node_off[id], N = P.node_off[id + 1] - nb;
    soft_net_forward<T>(Tb, S, P, id, dist);
    for (size_t k = 0; k < size_t(N) * LL; ++k) gd[k] = 0;
    T vals[kMaxLayers * kMaxLayers], w[kMaxLayers * kMaxLayers];
    {
        int n = 0;
        for (int lo = 0; lo < L; ++lo)
            for (int hi = lo; hi < L; ++hi) vals[n++] = dist[lo * L + hi];
        smin<T>(vals, n, S.tau, w);
        n = 0;
        for (int lo = 0; lo < L; ++lo)
            for (int hi = lo; hi < L; ++hi) gd[lo * L + hi] = g * w[n++];
    }
    // Edges in the reverse of the forward order: a node's range adjoint is
    // complete once its own parent edge has been processed.
    for (int i = 1; i < N; ++i) {
        const int p = P.parents[nb + i];
        const SoftEdge E = soft_edge(Tb, P.nodes[nb + i], P.nodes[nb + p]);
        const T* di = dist + size_t(i) * LL;
        const T* gp = gd + size_t(p) * LL;
        T* gi = gd + size_t(i) * LL;
        T cur[kMaxLayers], diag[kMaxLayers], gdiag[kMaxLayers], gcur[kMaxLayers];
        for (int l = 0; l < L; ++l) {
            int n = 0;
            for (int lo = 0; lo <= l; ++lo)
                for (int hi = l; hi < L; ++hi) vals[n++] = di[lo * L + hi];
            cur[l] = smin<T>(vals, n, S.tau, nullptr);
            gcur[l] = 0;
            gdiag[l] = 0;
        }
        for (int pl = 0; pl < L; ++pl) {
            for (int cl = 0; cl < L; ++cl) vals[cl] = cur[cl] + soft_leg<T>(Tb, S, E, cl, pl);
            diag[pl] = smin<T>(vals, L, S.tau, nullptr);
        }
        // parent range [lo, hi] += smin(diag[lo..hi])
        for (int lo = 0; lo < L; ++lo)
            for (int hi = lo; hi < L; ++hi) {
                const T gr = gp[lo * L + hi];
                if (gr == 0) continue;
                smin<T>(diag + lo, hi - lo + 1, S.tau, w);
                for (int k = 0; k <= hi - lo; ++k) gdiag[lo + k] += gr * w[k];
            }
        // arrival on pl from child layer cl
        for (int pl = 0; pl < L; ++pl) {
            if (gdiag[pl] == 0) continue;
            T legs[kMaxLayers];
            for (int cl = 0; cl < L; ++cl) {
                legs[cl] = soft_leg<T>(Tb, S, E, cl, pl);
                vals[cl] = cur[cl] + legs[cl];
            }
            smin<T>(vals, L, S.tau, w);
            for (int cl = 0; cl < L; ++cl) {
                if (w[cl] == 0) continue;
                gcur[cl] += gdiag[pl] * w[cl];
                soft_leg_adj<T>(Tb, S, E, cl, pl, gdiag[pl] * w[cl]);
            }
        }
        // cur[l] = smin over the child's ranges containing l
        for (int l = 0; l < L; ++l) {
            if (gcur[l] == 0) continue;
            int n = 0;
            for (int lo = 0; lo <= l; ++lo)
                for (int hi = l; hi < L; ++hi) vals[n++] = di[lo * L + hi];
            smin<T>(vals, n, S.tau, w);
            n = 0;
            for (int lo = 0; lo <= l; ++lo)
                for (int hi = l; hi < L; ++hi) gi[lo * L + hi] += gcur[l] * w[n++];
        }
    }
    // Via stacks of every node's ranges.
    for (int i = 0; i < N; ++i) {
        const int v = P.nodes[nb + i], x = v / Tb.Y % Tb.X, y = v % Tb.Y;
        const T* gi = gd + size_t(i) * LL;
        const T* di = dist + size_t(i) * LL;
        for (int l = 0; l + 1 < L; ++l) {
            T acc = 0;  // every finite range [lo, hi] with lo <= l < hi holds vc[l]
            for (int lo = 0; lo <= l; ++lo)
                for (int hi = l + 1; hi < L; ++hi)
                    if (di[lo * L + hi] < static_cast<T>(kSoftAbsent)) acc += gi[lo * L + hi];
            if (acc != 0) atomicAdd(S.dvc + slot_index(Tb, l, x, y), acc);
        }
    }
}

// ---- packs -------------------------------------------------------------------
// Shared memory of one warp.
template <class T>
struct SoftArena {
    T* D;   // [nmax][TT] range tables
    T* G;   // [nmax][TT] their adjoints (backward)
    T* w1;  // [nmax][L] first leg (or straight) wire cost
    T* w2;  // [nmax][L] second leg
    T* col; // [nmax][2][L] via costs at the corners (x, py) and (px, y)
    T* X;   // [2][32][L] exchange between the lanes of a slot
    T* Y;   // [3][32][L] running minima of the rows and columns (backward)
};
__host__ __device__ __forceinline__ size_t soft_arena_values(int L, int nmax, bool backward) {
    return size_t(nmax) * ((backward ? 2 : 1) * tri_count(L) + 4 * L) + size_t(32) * L * (backward ? 5 : 2);
}
template <class T>
__device__ __forceinline__ SoftArena<T> soft_arena(T* p, int L, int nmax, bool backward) {
    SoftArena<T> A;
    A.D = p; p += size_t(nmax) * tri_count(L);
    A.G = p; if (backward) p += size_t(nmax) * tri_count(L);
    A.w1 = p; p += size_t(nmax) * L;
    A.w2 = p; p += size_t(nmax) * L;
    A.col = p; p += size_t(nmax) * 2 * L;
    A.X = p; p += size_t(2) * 32 * L;
    A.Y = p;
    return A;
}

// A candidate that exists: NaN, infinities and kSoftAbsent or more do not (smin).
template <class T>
__device__ __forceinline__ bool soft_exists(T v) { return v < static_cast<T>(kSoftAbsent); }

// A running soft minimum: m the least value, s the sum of exp(-(v - m) / tau).
// A value that does not exist counts as kSoftNone, far above those that do: it
// weighs exactly 0 beside any of them, and nothing asks for the weights among
// values none of which exists.  add() returns what the adjoint needs: e =
// exp(-|difference| / tau) and whether the added value became the minimum.
constexpr double kSoftNone = 1e30;
template <class T>
struct SoftRun {
    T m, s;
    __device__ __forceinline__ T add(T m2, T s2, T inv_tau, bool& less) {
        m2 = soft_exists<T>(m2) ? m2 : static_cast<T>(kSoftNone);
        const T d = m2 - m;
        less = d < 0;
        const T e = s_exp<T>(-(less ? -d : d) * inv_tau);
        s = less ? s * e + s2 : s + s2 * e;
        m = less ? m2 : m;
        return e;
    }
    __device__ __forceinline__ T value(T tau) const { return m - tau * s_log<T>(s); }
};

// Forward DP of a pack (net_cost of its nets), and with kBackward the adjoint
// of g * (their sum) into dP and dvc.  The loops over layers stay rolled, their
// state in shared memory: unrolled, the adjoint was several times the
// instruction cache and waited for instructions 11 cycles of every 17 (5.1 ms
// at 320x320x10, 120K nets, fp32; rolled 2.3 ms).
template <class T, bool kBackward>
__device__ __forceinline__ void soft_pack(const Tables& Tb, const Soft<T>& S, const Pack& K, const SoftArena<T>& A, T g,
                                          int lane) {
    const int L = Tb.L, TT = tri_count(L);
    constexpr unsigned kAll = 0xffffffffu;
    const T absent = static_cast<T>(kSoftAbsent) * 10, tau = S.tau, inv = S.inv_tau;
    constexpr T kNone = static_cast<T>(kSoftNone);
    const int M = K.nodes;
    if (M == 0) return;
    int dep = K.par >= 0 ? 1 : 0;
    for (int anc = K.par; __any_sync(kAll, anc >= 0);) {
        const int od = __shfl_sync(kAll, dep, anc & 31), oa = __shfl_sync(kAll, anc, anc & 31);
        if (anc >= 0) { dep += od; anc = oa; }
    }
    if (lane >= M) dep = -1;
    const int dmax = __reduce_max_sync(kAll, dep);
    const int xy = (K.x << 16) | K.y;
    const int pxy = __shfl_sync(kAll, xy, K.par & 31);
    // Costs of every (node, layer); the nodes' own columns in X.
    for (int q0 = 0; q0 < M * L; q0 += 32) {
        const int q = q0 + lane, i = min(q / L, M - 1), l = q - q / L * L;
        const int c = __shfl_sync(kAll, xy, i), pc = __shfl_sync(kAll, pxy, i), pa = __shfl_sync(kAll, K.par, i);
        if (q >= M * L) continue;
        const int x = c >> 16, y = c & 0xffff, px = pc >> 16, py = pc & 0xffff;
        const bool ay = along_y(Tb, l);
        const int base = layer_base(Tb, l);
        A.X[q] = S.vc[base + (ay ? x * Tb.yp + y : y * Tb.xp + x)];
        if (pa < 0) continue;
        const bool straight = x == px || y == py;
        const int lo = ay ? min(y, py) : min(x, px), hi = ay ? max(y, py) : max(x, px);
        const int t1 = base + (ay ? x * Tb.yp : y * Tb.xp), t2 = base + (ay ? px * Tb.yp : py * Tb.xp);
        A.w1[q] = !straight || (ay ? x == px : y == py) ? S.P[t1 + hi] - S.P[t1 + lo] : absent;
        if (straight) continue;
        A.w2[q] = S.P[t2 + hi] - S.P[t2 + lo];
        A.col[(2 * i) * L + l] = S.vc[base + (ay ? x * Tb.yp + py : py * Tb.xp + x)];
        A.col[(2 * i + 1) * L + l] = S.vc[base + (ay ? px * Tb.yp + y : y * Tb.xp + px)];
    }
    __syncwarp();
    // Via stacks: row lo of every node's table.
    for (int q0 = 0; q0 < M * L; q0 += 32) {
        const int q = q0 + lane, i = min(q / L, M - 1), lo = q - q / L * L;
        const int lay = __shfl_sync(kAll, K.lay, i);
        if (q >= M * L) continue;
        T acc = 0;
        T* row = A.D + i * TT + tri(L, lo, lo) - lo;
#pragma unroll 1
        for (int hi = lo; hi < L; ++hi) {
            if (hi > lo) acc += A.X[i * L + hi - 1];
            row[hi] = (lay < L && (lo > lay || hi < lay)) ? absent : acc;
        }
    }
    __syncwarp();
    const int NS = max(1, 32 / L);
    const int slot = lane / L, sl = lane - slot * L, s0 = min(slot, NS - 1) * L, own = lane * L;
    // The slot's exchange, [L][L] twice; the lane's running minima.
    T *X = A.X + size_t(s0) * L, *X2 = X + size_t(32) * L;
    T *Re = A.Y + own, *Rs = Re + size_t(32) * L, *Ce = Rs + size_t(32) * L;
    const int row = tri(L, sl, sl) - sl;
    // Nodes of a depth in descending order, NS at a time: forward, children
    // into parents; or the adjoint, parents to children.
    auto edges = [&](unsigned level, auto backward) {
        constexpr bool kAdj = decltype(backward)::value;
        for (unsigned at = level; at;) {
            int i = -1;
            for (int k = 0; k < NS; ++k) {
                if (!at) break;
                const int top = 31 - __clz(at);
                if (k == slot) i = top;
                at ^= 1u << top;
            }
            const bool act = i >= 0;
            const int ii = max(i, 0);
            const int c = __shfl_sync(kAll, xy, ii), pc = __shfl_sync(kAll, pxy, ii), p = __shfl_sync(kAll, K.par, ii) & 31;
            const int x = c >> 16, y = c & 0xffff, px = pc >> 16, py = pc & 0xffff;
            const bool straight = x == px || y == py;
            const T* Di = A.D + ii * TT;
            // Row sl: running soft minimum of columns L-1 down to hi.
            SoftRun<T> R{kNone, 0};
            unsigned rless = 0;
#pragma unroll 1
            for (int hi = act ? L - 1 : -1; hi >= sl; --hi) {
                bool less;
                const T e = R.add(Di[row + hi], 1, inv, less);
                if (kAdj) { Re[hi] = e; Rs[hi] = R.s; rless |= unsigned(less) << hi; }
                X[sl * L + hi] = R.m;
                X2[sl * L + hi] = R.s;
            }
            __syncwarp();
            // Column sl: over the rows lo <= sl.
            SoftRun<T> C{kNone, 0};
            unsigned cless = 0;
#pragma unroll 1
            for (int lo = 0; lo <= (act ? sl : -1); ++lo) {
                bool less;
                const T e = C.add(X[lo * L + sl], X2[lo * L + sl], inv, less);
                if (kAdj) { Ce[lo] = e; cless |= unsigned(less) << lo; }
            }
            __syncwarp();  // X is reused
            const T reach = act ? C.value(tau) + A.w1[ii * L + sl] : absent;
            // Arrival on parent layer sl: the candidates cl of the other parity
            // (or cl = sl along a straight edge).
            constexpr int NC = (kMaxLayers + 1) / 2;
            const int odd = (sl & 1) ^ 1;
            const int side = along_y(Tb, sl) ? 1 : 0;  // the corner is the end of the first leg
            const T* col = A.col + (2 * ii + side) * L;
            const T leg2 = act && !straight ? A.w2[ii * L + sl] : static_cast<T>(0);
            T v[NC];
            T dm = absent, ds = 0;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const int cl = 2 * j + odd;
                const T r = __shfl_sync(kAll, reach, s0 + min(cl, L - 1));
                v[j] = absent;
                if (!act || straight || cl >= L) continue;
                T via = 0;
#pragma unroll 1
                for (int l = min(cl, sl) + 1; l < max(cl, sl); ++l) via += col[l];
                v[j] = r + (via + leg2);
                dm = v[j] < dm ? v[j] : dm;
            }
            T diag = absent;
            if (act && straight) {
                if (soft_exists<T>(reach)) diag = reach;
            } else if (act) {
#pragma unroll
                for (int j = 0; j < NC; ++j) {
                    v[j] = soft_exists<T>(v[j]) ? s_exp<T>(-(v[j] - dm) * inv) : static_cast<T>(0);  // from here on: weights
                    ds += v[j];
                }
                if (soft_exists<T>(dm)) diag = dm - tau * s_log<T>(ds);
            }
            // Row sl of the contribution: running soft minimum of diag[sl..hi].
            SoftRun<T> B{kNone, 0};
            unsigned bless = 0;
#pragma unroll 1
            for (int hi = 0; hi < L; ++hi) {
                const T dv = __shfl_sync(kAll, diag, s0 + hi);
                if (!act || hi < sl) continue;
                bool less;
                const T e = B.add(dv, 1, inv, less);
                if (kAdj) { X[sl * L + hi] = e; X2[sl * L + hi] = B.s; bless |= unsigned(less) << hi; }
                else X[sl * L + hi] = B.value(tau);
            }
            if (!kAdj) {
                T* Dp = A.D + p * TT;
                for (int k = 0; k < NS; ++k) {  // slots in turn: a parent's children in descending order
                    if (act && slot == k)
#pragma unroll 1
                        for (int hi = sl; hi < L; ++hi) Dp[row + hi] += X[sl * L + hi];
                    __syncwarp();
                }
                continue;
            }
            // Adjoint.  Back along a running minimum: U is what a value v gets for
            // each unit of exp(-(v - m) / tau), m the minimum of that step, so a
            // step adds its adjoint over its sum, and going below the value that
            // made the minimum scales U by that value's e.  Contribution (the
            // lane's own row of X, its result in place):
            const T* Gp = A.G + p * TT;
            T U = 0;
#pragma unroll 1
            for (int hi = act ? L - 1 : -1; hi >= sl; --hi) {
                const T e = X[sl * L + hi];
                const bool less = (bless >> hi) & 1u;
                U += Gp[row + hi] / X2[sl * L + hi];
                X[sl * L + hi] = less ? U : U * e;
                U = less ? U * e : U;
            }
            __syncwarp();
            T gd = 0;  // adjoint of diag[sl]
#pragma unroll 1
            for (int lo = 0; lo <= (act ? sl : -1); ++lo) gd += X[lo * L + sl];
            __syncwarp();
            // Arrival: X[pl][cl] = adjoint of candidate (cl, pl).
            T gcur = 0, gleg2 = 0;
            if (act && straight) gcur = gd;
            if (act && !straight) {
                const T scale = ds > 0 ? gd / ds : static_cast<T>(0);
#pragma unroll
                for (int j = 0; j < NC; ++j) {
                    const int cl = 2 * j + odd;
                    if (cl >= L) continue;
                    const T w = scale * v[j];
                    X[sl * L + cl] = w;
                    gleg2 += w;
                }
            }
            __syncwarp();
            if (act && !straight) {
#pragma unroll 1
                for (int cl = odd; cl < L; cl += 2) gcur += X[cl * L + sl];
                // Via cells of layer sl at the two corners: every candidate
                // whose layers enclose it; the corner by the first leg cl.
                T va = 0, vb = 0;
#pragma unroll 1
                for (int a = 0; a < sl; ++a)
#pragma unroll 1
                    for (int b = a + 1 + (((sl - a + 1) >> 1) << 1); b < L; b += 2) {  // the other parity, above sl
                        const T up = X[b * L + a], down = X[a * L + b];  // cl = a, pl = b; cl = b, pl = a
                        const bool ay = along_y(Tb, a);
                        va += ay ? up : down;
                        vb += ay ? down : up;
                    }
                if (va != 0) atomicAdd(S.dvc + slot_index(Tb, sl, x, py), va);
                if (vb != 0) atomicAdd(S.dvc + slot_index(Tb, sl, px, y), vb);
            }
            if (act && (!straight || (along_y(Tb, sl) ? x == px : y == py))) {
                // First leg on sl (at the child's end), second leg on sl (at the parent's).
                const bool ay = along_y(Tb, sl);
                const int base = layer_base(Tb, sl);
                const int lo = ay ? min(y, py) : min(x, px), hi = ay ? max(y, py) : max(x, px);
                const int t1 = base + (ay ? x * Tb.yp : y * Tb.xp), t2 = base + (ay ? px * Tb.yp : py * Tb.xp);
                if (gcur != 0 && lo != hi) { atomicAdd(S.dP + t1 + hi, gcur); atomicAdd(S.dP + t1 + lo, -gcur); }
                if (gleg2 != 0 && lo != hi) { atomicAdd(S.dP + t2 + hi, gleg2); atomicAdd(S.dP + t2 + lo, -gleg2); }
            }
            __syncwarp();
            // Column sl back to the rows' running minima (a row's sum at column
            // sl is in its lane's Rs), then row sl back to the ranges.
            U = act ? gcur / C.s : static_cast<T>(0);
#pragma unroll 1
            for (int lo = act ? sl : -1; lo >= 0; --lo) {
                const T e = Ce[lo], w = A.Y[size_t(32 + s0 + lo) * L + sl];
                const bool less = (cless >> lo) & 1u;
                X[lo * L + sl] = less ? U * w : U * e * w;
                U = less ? U * e : U;
            }
            __syncwarp();
            T* Gi = A.G + ii * TT;
            U = 0;
#pragma unroll 1
            for (int hi = sl; hi < (act ? L : 0); ++hi) {
                const T e = Re[hi];
                const bool less = (rless >> hi) & 1u;
                U += X[sl * L + hi] / Rs[hi];
                Gi[row + hi] = less ? U : U * e;
                U = less ? U * e : U;
            }
            __syncwarp();
        }
    };
    for (int d = dmax; d >= 1; --d) edges(__ballot_sync(kAll, dep == d), std::integral_constant<bool, false>{});
    // Root values, lane = slot * L + lo.
    for (unsigned at = __ballot_sync(kAll, dep == 0); at;) {
        int i = -1;
        for (int k = 0; k < NS; ++k) {
            if (!at) break;
            const int top = 31 - __clz(at);
            if (k == slot) i = top;
            at ^= 1u << top;
        }
        const bool act = i >= 0;
        const int ii = max(i, 0), id = __shfl_sync(kAll, K.id, ii);
        const T* Di = A.D + ii * TT;
        T m = absent;
#pragma unroll 1
        for (int hi = sl; hi < (act ? L : 0); ++hi) m = Di[row + hi] < m ? Di[row + hi] : m;
        T best = absent;
#pragma unroll 1
        for (int l = 0; l < L; ++l) {
            const T o = __shfl_sync(kAll, m, s0 + l);
            best = o < best ? o : best;
        }
        T part = 0;
#pragma unroll 1
        for (int hi = sl; hi < (act ? L : 0); ++hi) {
            const T w = soft_exists<T>(Di[row + hi]) ? s_exp<T>(-(Di[row + hi] - best) * inv) : static_cast<T>(0);
            X[sl * L + hi] = w;
            part += w;
        }
        T sum = 0;
#pragma unroll 1
        for (int l = 0; l < L; ++l) sum += __shfl_sync(kAll, part, s0 + l);
        const bool feasible = soft_exists<T>(best);
        if (act && sl == 0 && S.net_cost) S.net_cost[id] = feasible ? best - tau * s_log<T>(sum) : absent;
        if (kBackward)
#pragma unroll 1
            for (int hi = sl; hi < (act ? L : 0); ++hi)
                A.G[ii * TT + row + hi] = feasible ? g * (X[sl * L + hi] / sum) : static_cast<T>(0);
    }
    __syncwarp();
    if constexpr (kBackward) {
        for (int d = 1; d <= dmax; ++d) edges(__ballot_sync(kAll, dep == d), std::integral_constant<bool, true>{});
        // Via stacks of every node's ranges: range [lo, hi] holds vc[lo..hi-1].
        for (int q0 = 0; q0 < M * L; q0 += 32) {
            const int q = q0 + lane, i = min(q / L, M - 1), l = q - q / L * L;
            const int c = __shfl_sync(kAll, xy, i);
            if (q >= M * L || l + 1 >= L) continue;
            const T* Gi = A.G + i * TT;
            T acc = 0;
#pragma unroll 1
            for (int lo = 0; lo <= l; ++lo)
#pragma unroll 1
                for (int hi = l + 1; hi < L; ++hi) acc += Gi[tri(L, lo, hi)];
            if (acc != 0) atomicAdd(S.dvc + slot_index(Tb, l, c >> 16, c & 0xffff), acc);
        }
    }
}

}  // namespace grb
