// sweep.cuh -- device code shared by the local-move kernels: the per-sweep
// scalars, the DeltaQ argmax of one vertex, hash-table inserts and the
// afterburner term (src/local_mover.cpp:280-634).  Included by the kernels of
// local_move.cu (one kernel per degree class, every graph size) and by
// lm_steps.cuh (one-launch local moves of small graphs, a launch per step above).
#pragma once
#include "kernels.cuh"

namespace pggc {

// workspace slots of the local move (shared by both paths: the own-cluster
// weights that one leaves in LM_PVC may be reused by the other)
enum LMSlot : int {
    LM_PART, LM_DEST, LM_CAND, LM_MOVES, LM_NEWL, LM_AVAIL, LM_PRIO, LM_GAIN, LM_PV, LM_PVC, LM_TD, LM_FLAGS, LM_KEEP,
    LM_HAS, LM_SC, LM_GK, LM_GV, LM_MOVED_AT, LM_CSIZE, LM_OVF, LM_OVF_CNT, LM_STAMP, LM_AFF, LM_AFF_CNT,
    LM_SPLIT_BEST, LM_NEWID, LM_TD2, LM_PARTIAL, LM_BLK, LM_CNT
};

template <class V>
struct LMScalars {
    i64 num_cand, split, num_moves, num_new, num_avail, avail_k;
    unsigned long long new_hint;  // NEW_PART moves counted while compacting the move list
    i64 label_count, best_label_count;
    V uncut, best_uncut, last_pval, pval_sum;
    i64 sumsq_i;
    double sumsq_d;
    double obj, best_obj;
    int improved;
    int err;  // copy of the context's device error word (end of a local move)
    int pad[2];
    i64 relabel_count;  // labels after the final relabel
};

__device__ __forceinline__ void vatomic_add(i64* a, i64 x) {
    if (__isShared(a)) shared_add(a, x);
    else ::atomicAdd((unsigned long long*)a, (unsigned long long)x);
}
__device__ __forceinline__ void vatomic_add(double* a, double x) { ::atomicAdd(a, x); }

struct Best {
    float jc;
    i32 c;
};
__device__ __forceinline__ bool better(float jc, i32 c, const Best& b) { return jc > b.jc || (jc == b.jc && c < b.c); }
__device__ __forceinline__ Best none_best() { return Best{-INFINITY, 2147483647}; }
// Order-preserving map of a float onto u32 (no NaN here); with it the best
// (largest gain, then smallest cluster id) of a lane group is two hardware
// reductions instead of a shuffle butterfly.  Gains are never -0.0 (a
// candidate has f > 0 and f - x is +0.0 when equal), so float equality and
// key equality agree.
__device__ __forceinline__ u32 f2ord(float f) {
    const u32 b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord2f(u32 k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k); }
__device__ __forceinline__ void reduce_best(Best& b, unsigned mask) {
    const u32 k = f2ord(b.jc);
    const u32 mk = __reduce_max_sync(mask, k);
    const u32 mc = __reduce_min_sync(mask, k == mk ? (u32)b.c : 0xFFFFFFFFu);
    b = Best{ord2f(mk), (i32)mc};
}
__device__ __forceinline__ void warp_best(Best& b) { reduce_best(b, FULL); }


template <class W>
struct SelArgs {
    using V = typename Traits<W>::V;
    DGraph<W> g;
    const i32* part;
    i32* dest;
    float* gain;
    const V* pvals;
    const V* td;
    const i32* constraint;
    const i64* label_count;  // device
    const V* rsum;           // row weight sums (NULL: no bound check)
    const WeightUnits* units;  // FP32 weights (NULL: none)
    int keys32;              // cluster ids < 2^29: group match keys fit 32 bits
    int dense;               // block kernels: every label indexes the shared table directly
    float pm;
    float fr;
    int initial;
    int* err;
    unsigned long long* prof;  // algorithmic-byte counter (profiling only)
    u32 probe_cap;             // fault-injection cap on hash probes (0: none)
    float inv_load;            // hash-table slots per distinct key (1 / load factor): 2 or 1/0.7
};

// table slots for up to U distinct keys at the tuned load factor (a power of two)
template <class W>
__device__ __forceinline__ u32 sel_table_slots(const SelArgs<W>& a, i64 U) {
    return next_pow2_u32((u32)ceilf((float)U * a.inv_load));
}

// algorithmic bytes of one select evaluation: list entry + dest read, then
// rowptr pair, vtx_w, part, pval, D[part], dest/gain writes, and per edge the
// column, weight and neighbour label (initial mode: column, weight, D[v])
template <class W>
__device__ __forceinline__ unsigned long long sel_bytes(const SelArgs<W>& a, i64 deg, bool evaluated) {
    if (!evaluated) return 8;
    const unsigned long long wb = a.g.w ? sizeof(W) : 0;
    return 60ull + (unsigned long long)deg * (a.initial ? (12ull + wb) : (8ull + wb));
}

struct VCtx {
    i32 p;
    float multi, p_conn, thr;
};

template <class W>
__device__ __forceinline__ VCtx sel_prologue(const SelArgs<W>& a, i32 i) {
    using V = typename Traits<W>::V;
    VCtx v;
    V w = a.g.vtx_w[i];
    v.multi = to_f(w) * a.pm;
    v.p = a.part[i];
    v.p_conn = to_f(a.pvals[i]) - to_f(V(a.td[v.p] - w)) * v.multi;
    v.thr = v.p_conn < 0.0f ? 0.0f : (float)((double)v.p_conn * (1.0 - (double)a.fr));
    return v;
}

// Exact skip: no neighbour cluster can carry more weight than the vertex's
// weight outside its own cluster, ext = rowsum - pval; when even ext rounds
// (one FP32 step up, covering FP64 rounding in either sum) below the
// candidate threshold, no cluster passes the `f >= thr` test of sel_eval and
// the edges need not be read: the outcome is the no-candidate outcome.
template <class W>
__device__ __forceinline__ bool sel_no_candidate(const SelArgs<W>& a, i32 i, const VCtx& vc) {
    if (!a.rsum || a.initial) return false;
    const float fe = nextafterf(to_f(a.rsum[i] - a.pvals[i]), INFINITY);
    return !(fe >= vc.thr);
}

template <class W, bool CON>
__device__ __forceinline__ void sel_eval(const SelArgs<W>& a, const VCtx& vc, i32 c, typename Traits<W>::V jv,
                                         Best& b) {
    using V = typename Traits<W>::V;
    if (!(jv > V(0))) return;
    float f = to_f(jv);
    if (!(f >= vc.thr)) return;
    if (CON && a.constraint[c] != a.constraint[vc.p]) return;
    float jc = f - to_f(a.td[c]) * vc.multi;
    if (jc >= vc.thr && better(jc, c, b)) b = Best{jc, c};
}

template <class W>
__device__ __forceinline__ void sel_finish(const SelArgs<W>& a, i32 i, const VCtx& vc, const Best& b) {
    if (b.c != 2147483647) {
        a.dest[i] = b.c;
        a.gain[i] = b.jc - vc.p_conn;
    } else if (vc.p_conn < 0.0f) {
        a.dest[i] = NEW_PART;
        a.gain[i] = -vc.p_conn;
    } else {
        a.dest[i] = NO_MOVE;
        a.gain[i] = OBJ_MIN;
    }
}

// One vertex of degree <= K by one thread: the row sits in registers, equal
// neighbour clusters are merged by pairwise compares and summed from 0 in edge
// order -- the order of the lane-order group sum, so the gains are
// bit-identical -- and the best cluster is kept under the same total order
// (gain, then smaller id).  Returns the edges read, -1 for a skipped vertex.
template <class W, bool CON, int K>
__device__ __forceinline__ int sel_thread(const SelArgs<W>& a, i32 i) {
    using V = typename Traits<W>::V;
    if (a.dest[i] == NO_MOVE) return -1;
    const VCtx vc = sel_prologue(a, i);
    const i64 b = a.g.rowptr[i];
    i64 e = a.g.rowptr[i + 1];
    if (sel_no_candidate(a, i, vc)) e = b;
    const int d = (int)(e - b);
    Best best = none_best();
    i32 c[K];
#pragma unroll
    for (int t = 0; t < K; t++) c[t] = t < d ? a.g.col[b + t] : -1;
    if (a.initial) {
#pragma unroll
        for (int t = 0; t < K; t++)
            if (t < d) sel_eval<W, CON>(a, vc, c[t], V(a.g.wgt(b + t)), best);
    } else {
#pragma unroll
        for (int t = 0; t < K; t++) c[t] = c[t] >= 0 ? a.part[c[t]] : -1;
        // weights are read where they are summed (the row is in L1)
#pragma unroll
        for (int t = 0; t < K; t++) {
            bool first = c[t] >= 0 && c[t] != vc.p;
#pragma unroll
            for (int m = 0; m < t; m++) first = first && c[m] != c[t];
            if (first) {
                V sum = V(0);
#pragma unroll
                for (int m = t; m < K; m++)
                    if (c[m] == c[t]) sum = sum + V(a.g.wgt(b + m));
                sel_eval<W, CON>(a, vc, c[t], sum, best);
            }
        }
    }
    sel_finish(a, i, vc, best);
    return d;
}

// Sum of `val` over the lanes of `peers` (lane order), valid at the group leader.
template <class V>
__device__ __forceinline__ V group_sum(unsigned peers, V val, bool leader) {
    int size = __popc(peers);
    int maxsize = __reduce_max_sync(FULL, (unsigned)size);
    V s = V(0);
    unsigned rem = peers;
    const int l = lane_id();
    for (int r = 0; r < maxsize; r++) {
        int src = l;
        bool take = leader && rem;
        if (take) {
            src = __ffs(rem) - 1;
            rem &= rem - 1;
        }
        V x = __shfl_sync(FULL, val, src);
        if (take) s = s + x;
    }
    return s;
}

// Sum of the weights of the lanes in `peers` (equal neighbour clusters), valid
// at the leader: the lane-order shuffle sum, or the count for unit weights.
template <class W>
__device__ __forceinline__ typename Traits<W>::V peer_sum(const SelArgs<W>& a, unsigned peers, W wr, bool keep,
                                                          bool leader) {
    using V = typename Traits<W>::V;
    if (!a.g.w) return V(__popc(peers));
    return group_sum<V>(peers, keep ? V(wr) : V(0), leader);
}

// Linear-probing insert; gives up (latching DEV_ERR_PROBE) after the table size
// or `cap` probes, whichever is smaller (cap = 0: no extra limit).
template <class V>
__device__ __forceinline__ void table_add(i32* keys, V* vals, u32 mask, i32 c, V x, int* err, u32 cap) {
    u32 s = xorshift32((u32)c) & mask;
    volatile i32* vk = keys;
    const u32 limit = (cap != 0 && cap <= mask) ? cap : mask + 1;
    for (u32 probe = 0; probe < limit; probe++) {
        i32 k = vk[s];
        if (k == c) {
            vatomic_add(&vals[s], x);
            return;
        }
        if (k == -1) {
            i32 old = atomicCAS(&keys[s], -1, c);
            if (old == -1 || old == c) {
                vatomic_add(&vals[s], x);
                return;
            }
        }
        s = (s + 1) & mask;
    }
    atomicExch(err, (int)DEV_ERR_PROBE);
}

// units of vertex i's shared-memory table
template <class W>
__device__ __forceinline__ Units<W> sel_units(const SelArgs<W>& a, i32 i) {
    return Units<W>::make(a.units, a.rsum ? (double)a.rsum[i] : INFINITY);
}

// Aggregates one 32-edge chunk (edges j = base + lane, valid if < e) into the
// shared-memory table, skipping the vertex's own cluster.  In units every edge
// adds itself; FP64 sums are merged in the warp first.
template <class W>
__device__ __forceinline__ void chunk_to_table(const SelArgs<W>& a, const VCtx& vc, i64 j, i64 e, i32* keys,
                                               typename Traits<W>::V* vals, u32 mask, const Units<W>& un) {
    using V = typename Traits<W>::V;
    bool valid = j < e;
    i32 c = valid ? a.part[a.g.col[j]] : -1;
    W wr = valid ? a.g.wgt(j) : W(0);
    bool keep = valid && c != vc.p;
    if (un.on) {
        if (keep) table_add(keys, (i64*)vals, mask, c, un.of(wr), a.err, a.probe_cap);
        return;
    }
    i32 key = keep ? c : (i32)(0x80000000u | lane_id());
    unsigned peers = __match_any_sync(FULL, key);
    bool leader = keep && ((peers & lanemask_lt()) == 0);
    V s = peer_sum<W>(a, peers, wr, keep, leader);
    if (leader) table_add(keys, vals, mask, c, s, a.err, a.probe_cap);
}

// Insert that gives up after TRY_PROBES probes (the caller sends the vertex
// to the global-table pass); a run that long means the table is nearly full.
constexpr u32 TRY_PROBES = 64;
template <class V>
__device__ __forceinline__ bool table_try_add(i32* keys, V* vals, u32 mask, i32 c, V x) {
    u32 s = xorshift32((u32)c) & mask;
    volatile i32* vk = keys;
    for (u32 probe = 0; probe < TRY_PROBES && probe <= mask; probe++) {
        i32 k = vk[s];
        if (k == c) {
            vatomic_add(&vals[s], x);
            return true;
        }
        if (k == -1) {
            i32 old = atomicCAS(&keys[s], -1, c);
            if (old == -1 || old == c) {
                vatomic_add(&vals[s], x);
                return true;
            }
        }
        s = (s + 1) & mask;
    }
    return false;
}

// chunk_to_table with table_try_add: false if this lane's insert failed
template <class W>
__device__ __forceinline__ bool chunk_to_table_try(const SelArgs<W>& a, const VCtx& vc, i64 j, i64 e, i32* keys,
                                                   typename Traits<W>::V* vals, u32 mask, const Units<W>& un) {
    using V = typename Traits<W>::V;
    bool valid = j < e;
    i32 c = valid ? a.part[a.g.col[j]] : -1;
    W wr = valid ? a.g.wgt(j) : W(0);
    bool keep = valid && c != vc.p;
    if (un.on) return keep ? table_try_add(keys, (i64*)vals, mask, c, un.of(wr)) : true;
    i32 key = keep ? c : (i32)(0x80000000u | lane_id());
    unsigned peers = __match_any_sync(FULL, key);
    bool leader = keep && ((peers & lanemask_lt()) == 0);
    V s = peer_sum<W>(a, peers, wr, keep, leader);
    return leader ? table_try_add(keys, vals, mask, c, s) : true;
}

// degree class of a vertex (NCLS classes, see ClassLists)
__device__ __forceinline__ int deg_class(i64 d) {
    return d <= 8 ? 0 : d <= 16 ? 1 : d <= 32 ? 2 : d < LARGE_CUTOFF ? 3 : d <= 1024 ? 4 : d <= HUGE_DEG ? 5 : 6;
}

template <int G>
__device__ __forceinline__ void group_best(Best& b) {
    const unsigned mask = G == 32 ? FULL : (((1u << G) - 1u) << (lane_id() & ~(G - 1)));
    reduce_best(b, mask);
}

// ---- afterburner (src/local_mover.cpp:280-433) ------------------------------
template <class W>
struct ABArgs {
    using V = typename Traits<W>::V;
    DGraph<W> g;
    const i32* part;
    const i32* dest;
    const float* gain;
    float pm;
    const i32* cand;
    unsigned char* keep;
    const LMScalars<V>* sc;
    unsigned long long* prof;
};

// algorithmic bytes of one afterburner evaluation: candidate entry, its
// dest/part/vtx_w/gain, rowptr pair, keep flag; per edge column, weight, gain[v]
template <class W>
__device__ __forceinline__ unsigned long long ab_bytes(const ABArgs<W>& a, i64 deg) {
    const unsigned long long wb = a.g.w ? sizeof(W) : 0;
    return 41ull + (unsigned long long)deg * (8ull + wb);
}

// algorithmic bytes of one own-cluster weight: list entry, offsets, own label,
// result; per edge column, weight, label
template <class W>
__device__ __forceinline__ unsigned long long own_bytes(const DGraph<W>& g, i64 deg) {
    return 24ull + sizeof(typename Traits<W>::V) + (unsigned long long)deg * (8 + (g.w ? sizeof(W) : 0));
}

// Rows are summed G lanes at a time, several groups of edges in flight: the
// columns of all of them are loaded, then their first gathers, then what those
// ask for.  One edge after another, a row of 2,000 edges was a chain of 63 times
// five dependent loads on one warp (0.1 ms, the length of the whole step).
// A row type says how many groups it takes at a time: eight where an edge asks
// for one gather, UG where it asks for more (registers).
// (Groups of 8 and 16 lanes only see rows of up to two groups.)
constexpr int UG = 4;

// afterburner terms of vertex (p, best, igain, hash hi) for the edges j with on
template <class W>
struct AbRow {
    static constexpr int BATCH = UG;
    const ABArgs<W>& a;
    i32 p, best, hi;
    float multi, igain;
    __device__ __forceinline__ double term(i64 j) const {
        const i32 v = a.g.col[j];
        const float d = a.gain[v] - igain;
        if (d >= AFTERBURNER_EPS || (fabsf(d) < AFTERBURNER_EPS && (i32)xorshift32((u32)v) < hi)) {
            const float q = (float)a.g.wgt(j) - multi * to_f(a.g.vtx_w[v]);
            int coef = 0;
            i32 vp = a.dest[v];
            if (vp == p) coef--;
            if (vp == best && best != NEW_PART) coef++;
            vp = a.part[v];
            if (vp == p) coef++;
            if (vp == best) coef--;
            return (double)coef * (double)q;
        }
        return 0.0;
    }
    template <int U>
    __device__ __forceinline__ void terms(const i64 (&j)[U], const bool (&on)[U], double (&t)[U]) const {
        i32 v[U];
        float vg[U];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = on[u] ? a.g.col[j[u]] : -1;
#pragma unroll
        for (int u = 0; u < U; u++) vg[u] = on[u] ? a.gain[v[u]] : 0.f;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float d = vg[u] - igain;
            in[u] = on[u] && (d >= AFTERBURNER_EPS ||
                              (fabsf(d) < AFTERBURNER_EPS && (i32)xorshift32((u32)v[u]) < hi));
        }
        i32 vd[U], vp[U];
        W w[U];
        typename Traits<W>::V vw[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            vd[u] = in[u] ? a.dest[v[u]] : 0;
            vp[u] = in[u] ? a.part[v[u]] : 0;
            w[u] = in[u] ? a.g.wgt(j[u]) : W(0);
            vw[u] = in[u] ? a.g.vtx_w[v[u]] : typename Traits<W>::V(0);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float q = (float)w[u] - multi * to_f(vw[u]);
            int coef = 0;
            if (vd[u] == p) coef--;
            if (vd[u] == best && best != NEW_PART) coef++;
            if (vp[u] == p) coef++;
            if (vp[u] == best) coef--;
            t[u] = in[u] ? (double)coef * (double)q : 0.0;
        }
    }
};

// own-cluster weights: edges to label li
template <class W>
struct OwnRow {
    static constexpr int BATCH = 8;
    const DGraph<W>& g;
    const i32* lab;
    i32 li;
    __device__ __forceinline__ typename Traits<W>::V term(i64 j) const {
        using V = typename Traits<W>::V;
        return lab[g.col[j]] == li ? V(g.wgt(j)) : V(0);
    }
    // the weights stream in beside the columns: waiting for the label first
    // made this slower than one edge at a time
    template <int U>
    __device__ __forceinline__ void terms(const i64 (&j)[U], const bool (&on)[U], typename Traits<W>::V (&t)[U]) const {
        using V = typename Traits<W>::V;
        i32 c[U];
        W w[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            c[u] = on[u] ? g.col[j[u]] : -1;
            w[u] = on[u] ? g.wgt(j[u]) : W(0);
        }
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = on[u] ? lab[c[u]] : -1;
#pragma unroll
        for (int u = 0; u < U; u++) t[u] = on[u] && c[u] == li ? V(w[u]) : V(0);
    }
};

// Canonical per-vertex sum of a row's terms by a G-lane group: lane r adds terms
// r, r + G, ... from 0, then the xor butterfly (exact match of the 32-lane
// association for degree <= 2G; integer sums are order-free).
template <int G, class V, class Row>
__device__ __forceinline__ V group_row_sum(i64 b, i64 e, int r, const Row& row) {
    V acc = V(0);
    i64 j0 = b + r;
    auto groups = [&](auto uc, auto full) {
        constexpr int U = decltype(uc)::value;
        i64 j[U];
        bool on[U];
        V t[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            j[u] = j0 + u * G;
            on[u] = decltype(full)::value || j[u] < e;
        }
        row.terms(j, on, t);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (on[u]) acc += t[u];
        j0 += U * G;
    };
    // Whole batches without a test an edge, the rest two groups at a time.  With
    // tested batches of four to the end, rows of 33 to 64 edges issued twice
    // their instructions.  R-MAT of 1 M vertices, 31 M edges: own-cluster weights
    // of the rows above 128 edges 148 us so, 111 us now (four at a time 150);
    // inner connectivity of the rows above 32 447 and 164 us.
    if (G == 32)
        while (e - (j0 - r) >= Row::BATCH * G) groups(std::integral_constant<int, Row::BATCH>{}, std::true_type{});
    while (j0 - r < e) groups(std::integral_constant<int, 2>{}, std::false_type{});
#pragma unroll
    for (int d = G / 2; d >= 1; d >>= 1) acc = acc + __shfl_xor_sync(FULL, acc, d);
    return acc;
}

}  // namespace pggc
