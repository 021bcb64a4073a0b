// lm_steps.cuh -- the steps of a sweep (select, afterburner, new cluster ids,
// moves, own-cluster weights) as device functions over all blocks of a launch:
// the one-launch local move (lm_cluster.cuh) runs them in turn, lm_steps.cu
// launches them one by one.
//
// The steps do the same arithmetic in the same association as the kernels of
// local_move.cu (shared code in sweep.cuh), so the results are bit-identical:
// exact integer sums, FP64 edge sums by the 32-lane canonical association,
// array sums as groups of 32, new cluster ids in order1 order.
#pragma once
#include "kernels.cuh"
#include "filter.cuh"
#include "sweep.cuh"
#include "gang.cuh"
#include "lm_small.cuh"

namespace pggc {

// ---- select -----------------------------------------------------------------
// Vertices of degree <= G by G-lane groups, UV vertices of a group in flight.
template <class W, bool CON, int G, int UV>
__device__ __forceinline__ void sel_grp(const SelArgs<W>& a, const i32* cls, i64 lo, i64 hi, i64 first, i64 nw) {
    using V = typename Traits<W>::V;
    constexpr int NG = 32 / G;
    const int l = lane_id(), r = l & (G - 1), grp = l / G;
    for (i64 base = lo + first * NG * UV; base < hi; base += nw * NG * UV) {
        i32 iv[UV];
        bool act[UV];
#pragma unroll
        for (int u = 0; u < UV; u++) {
            const i64 x = base + u * NG + grp;
            iv[u] = x < hi ? cls[x] : -1;
        }
#pragma unroll
        for (int u = 0; u < UV; u++) act[u] = iv[u] >= 0 && a.dest[iv[u]] != NO_MOVE;
        VCtx vc[UV];
        i64 b[UV], e[UV];
#pragma unroll
        for (int u = 0; u < UV; u++) {
            b[u] = act[u] ? a.g.rowptr[iv[u]] : 0;
            e[u] = act[u] ? a.g.rowptr[iv[u] + 1] : 0;
        }
        // the row is loaded while the vertex's own terms are: few vertices are
        // ruled out by their row sum, and a step is one or two of these chains
        i32 c[UV];
        W wv[UV];
#pragma unroll
        for (int u = 0; u < UV; u++) {
            const i64 j = b[u] + r;
            const bool valid = j < e[u];
            c[u] = valid ? a.g.col[j] : -1;
            wv[u] = valid ? a.g.wgt(j) : W(0);
        }
        if (!a.initial) {
#pragma unroll
            for (int u = 0; u < UV; u++) c[u] = c[u] >= 0 ? a.part[c[u]] : -1;
        }
#pragma unroll
        for (int u = 0; u < UV; u++) {
            vc[u] = VCtx{};
            if (act[u]) {
                vc[u] = sel_prologue(a, iv[u]);
                if (sel_no_candidate(a, iv[u], vc[u])) c[u] = -1;
            }
        }
#pragma unroll
        for (int u = 0; u < UV; u++) {
            Best best = none_best();
            if (a.initial) {
                if (c[u] >= 0) sel_eval<W, CON>(a, vc[u], c[u], V(wv[u]), best);
            } else {
                const bool keep = c[u] >= 0 && c[u] != vc[u].p;
                unsigned peers;
                if (a.keys32) {
                    // bit 31 marks lanes without a candidate (unique per lane), bits 29-30 the group
                    const u32 key = keep ? (((u32)grp << 29) | (u32)c[u]) : (0x80000000u | (u32)l);
                    peers = __match_any_sync(FULL, key);
                } else {
                    const u64 key = keep ? (((u64)grp << 32) | (u64)(u32)c[u]) : (0xFFFFFFFF00000000ull | (u64)l);
                    peers = __match_any_sync(FULL, key);
                }
                const bool leader = keep && ((peers & lanemask_lt()) == 0);
                const V sum = peer_sum<W>(a, peers, wv[u], keep, leader);
                if (leader) sel_eval<W, CON>(a, vc[u], c[u], sum, best);
            }
            group_best<G>(best);
            if (r == 0 && act[u]) sel_finish(a, iv[u], vc[u], best);
        }
    }
}

// A warp per vertex, hash table of a warp's share of shared memory.
template <class W, bool CON>
__device__ __forceinline__ void sel_warp_hash(const SelArgs<W>& a, i32 i, const VCtx& vc, i64 b, i64 e,
                                              unsigned char* smem, Best& best) {
    using V = typename Traits<W>::V;
    const int l = lane_id();
    const u32 T = sel_table_slots(a, e - b);  // <= 256 for degrees below 128
    V* vals = (V*)smem;
    i32* keys = (i32*)(smem + sizeof(V) * T);
    for (u32 s = l; s < T; s += 32) {
        keys[s] = -1;
        vals[s] = V(0);
    }
    __syncwarp();
    const Units<W> un = sel_units(a, i);
    for (i64 j = b + l; j - l < e; j += 32) chunk_to_table(a, vc, j, e, keys, vals, T - 1, un);
    __syncwarp();
    for (u32 s = l; s < T; s += 32) {
        const i32 c = keys[s];
        if (c != -1) sel_eval<W, CON>(a, vc, c, un.sum(vals[s]), best);
    }
    __syncwarp();
}

// A vertex by a warp or the block, table indexed by cluster id, labels
// [c0, c1) at a time.  T: u32 when the row's weights sum below 2^32 (shared-
// memory atomics of 32 bits are native, wider ones are compare-and-swap
// loops), V otherwise.  False (best not to be used) when a u32 pass met a
// negative weight, for which the row sum bounds nothing.
template <class W, bool CON, bool BLOCK, class T>
__device__ __forceinline__ bool sel_dense(const SelArgs<W>& a, const VCtx& vc, i64 b, i64 e, i64 L, T* tab, i64 room,
                                          const Units<W>& un, Best& best) {
    using V = typename Traits<W>::V;
    constexpr int NT = BLOCK ? LS_THREADS : 32;
    const int t = BLOCK ? (int)threadIdx.x : lane_id(), l = lane_id();
    auto sync = [&]() {
        if (BLOCK) __syncthreads();
        else __syncwarp();
    };
    for (i64 c0 = 0; c0 < L; c0 += room) {
        const i64 c1 = min(L, c0 + room);
        for (i64 s = t; s < c1 - c0; s += NT) tab[s] = T(0);
        sync();
        if constexpr (std::is_same<T, u32>::value) {
            bool neg = false;
#pragma unroll 4
            for (i64 j = b + t; j < e; j += NT) {
                const i32 c = a.part[a.g.col[j]];
                const i32 wr = (i32)a.g.wgt(j);
                neg = neg || wr < 0;
                if (c != vc.p && c >= c0 && c < c1) atomicAdd(&tab[c - c0], (u32)wr);
            }
            if (BLOCK ? __syncthreads_or(neg) : __any_sync(FULL, neg)) return false;
        } else if (un.on) {
#pragma unroll 4
            for (i64 j = b + t; j < e; j += NT) {
                const i32 c = a.part[a.g.col[j]];
                const W wr = a.g.wgt(j);
                if (c != vc.p && c >= c0 && c < c1) shared_add((i64*)&tab[c - c0], un.of(wr));
            }
        } else {
            for (i64 j = b + t; j - l < e; j += NT) {
                const bool valid = j < e;
                const i32 c = valid ? a.part[a.g.col[j]] : -1;
                const W wr = valid ? a.g.wgt(j) : W(0);
                const bool keep = valid && c != vc.p && c >= c0 && c < c1;
                const i32 key = keep ? c : (i32)(0x80000000u | l);
                const unsigned peers = __match_any_sync(FULL, key);
                const bool leader = keep && ((peers & lanemask_lt()) == 0);
                const V sum = peer_sum<W>(a, peers, wr, keep, leader);
                if (leader) vatomic_add(&tab[c - c0], sum);
            }
        }
        sync();
        for (i64 s = t; s < c1 - c0; s += NT) {
            V x;
            if constexpr (std::is_same<T, u32>::value) x = (V)tab[s];
            else x = un.sum(tab[s]);
            if (x > V(0)) sel_eval<W, CON>(a, vc, (i32)(c0 + s), x, best);
        }
        sync();
    }
    return true;
}

// the vertex's best cluster from a dense table of `bytes` bytes
template <class W, bool CON, bool BLOCK>
__device__ __forceinline__ void sel_dense_row(const SelArgs<W>& a, i32 i, const VCtx& vc, i64 b, i64 e, i64 L,
                                              unsigned char* smem, i64 bytes, Best& best) {
    using V = typename Traits<W>::V;
    const Units<W> un = sel_units(a, i);
    if constexpr (std::is_same<V, i64>::value) {
        if (a.rsum[i] < (i64)0xFFFFFFFFll) {
            if (sel_dense<W, CON, BLOCK, u32>(a, vc, b, e, L, (u32*)smem, bytes / (i64)sizeof(u32), un, best)) return;
            best = none_best();
        }
    }
    sel_dense<W, CON, BLOCK, V>(a, vc, b, e, L, (V*)smem, bytes / (i64)sizeof(V), un, best);
}

// Vertices of degree below 128; `mine`: the warp's shared memory (3 KB).
// Returns the warps' worth of work it handed out.
template <class W, bool CON>
__device__ __forceinline__ i64 select_low(const SelArgs<W>& a, const i32* cls, const i64* off, unsigned char* mine) {
    const int l = lane_id();
    const i64 nw = gang_warps();
    const i64 o0 = off[0], o1 = off[1], o2 = off[2], o3 = off[3], o4 = off[4];
    using V = typename Traits<W>::V;
    i64 rot = 0;
    // A thread per vertex from about six (degree 17-32) to twelve (up to 8)
    // vertices a warp: a lane group issues 150 instructions a vertex of the
    // 17-32 class, a thread a third of that, but its chain is longer.  Select
    // step of a 65,536-vertex graph: 31.7 us with groups, 26.7 us so.  One-
    // launch local moves, us with groups / so: 6,000 vertices of 14 edges 472 /
    // 409 (FP32 521 / 473), 8,000 of 8 edges 401 / 314; with a launch per
    // step, 65,536 vertices of 14 edges 626 / 594.
    auto thr = [&](auto kc, i64 lo, i64 hi) {
        constexpr int K = decltype(kc)::value;
        const i64 first = gang_first(rot);
        rot += (hi - lo + 31) >> 5;
        for (i64 x = lo + first * 32 + l; x < hi; x += nw * 32) sel_thread<W, CON, K>(a, cls[x]);
    };
    if ((o1 - o0) > 12 * nw) {
        thr(std::integral_constant<int, 8>{}, o0, o1);
    } else {
        const i64 first = gang_first(rot);
        rot += (o1 - o0 + 7) >> 3;
        sel_grp<W, CON, 8, 2>(a, cls, o0, o1, first, nw);
    }
    if ((o2 - o1) > 8 * nw) {
        thr(std::integral_constant<int, 16>{}, o1, o2);
    } else {
        const i64 first = gang_first(rot);
        rot += (o2 - o1 + 3) >> 2;
        sel_grp<W, CON, 16, 2>(a, cls, o1, o2, first, nw);
    }
    if ((o3 - o2) > 6 * nw) {
        thr(std::integral_constant<int, 32>{}, o2, o3);
    } else {
        const i64 first = gang_first(rot);
        rot += (o3 - o2 + 1) >> 1;
        sel_grp<W, CON, 32, 2>(a, cls, o2, o3, first, nw);
    }
    const i64 first = gang_first(rot);
    rot += o4 - o3;
    for (i64 x = o3 + first; x < o4; x += nw) {
        const i32 i = cls[x];
        if (a.dest[i] == NO_MOVE) continue;
        const VCtx vc = sel_prologue(a, i);
        const i64 b = a.g.rowptr[i];
        i64 e = a.g.rowptr[i + 1];
        if (sel_no_candidate(a, i, vc)) e = b;
        Best best = none_best();
        if (a.initial) {
            for (i64 j = b + l; j < e; j += 32) sel_eval<W, CON>(a, vc, a.g.col[j], V(a.g.wgt(j)), best);
        } else if (e > b) {
            sel_warp_hash<W, CON>(a, i, vc, b, e, mine, best);
        }
        warp_best(best);
        if (l == 0) sel_finish(a, i, vc, best);
    }
    return rot;
}

template <class W, bool CON>
__device__ __forceinline__ void select_step(const SelArgs<W>& a, const i32* cls, const i64* off, i64 L,
                                            unsigned char* smem, Best* wb) {
    using V = typename Traits<W>::V;
    const int l = lane_id(), w = threadIdx.x >> 5;
    const i64 nw = gang_warps();
    const i64 o4 = off[4], o7 = off[7];
    unsigned char* mine = smem + w * LS_WARP_BYTES;
    const i64 rot = select_low<W, CON>(a, cls, off, mine);
    const bool by_warp = L * (i64)(std::is_same<V, i64>::value ? sizeof(u32) : sizeof(V)) <= LS_WARP_BYTES;
    // degrees from 128 up: a warp where the labels fit its share
    if (by_warp) {
        for (i64 x = o4 + gang_first(rot); x < o7; x += nw) {
            const i32 i = cls[x];
            if (a.dest[i] == NO_MOVE) continue;
            const VCtx vc = sel_prologue(a, i);
            const i64 b = a.g.rowptr[i];
            i64 e = a.g.rowptr[i + 1];
            if (sel_no_candidate(a, i, vc)) e = b;
            Best best = none_best();
            if (a.initial) {
                for (i64 j = b + l; j < e; j += 32) sel_eval<W, CON>(a, vc, a.g.col[j], V(a.g.wgt(j)), best);
            } else if (e > b) {
                sel_dense_row<W, CON, false>(a, i, vc, b, e, L, mine, LS_WARP_BYTES, best);
            }
            warp_best(best);
            if (l == 0) sel_finish(a, i, vc, best);
        }
        return;
    }
    // a block per vertex
    __syncthreads();
    for (i64 x = o4 + blockIdx.x; x < o7; x += gridDim.x) {
        const i32 i = cls[x];
        if (a.dest[i] == NO_MOVE) continue;
        const VCtx vc = sel_prologue(a, i);
        const i64 b = a.g.rowptr[i];
        i64 e = a.g.rowptr[i + 1];
        if (sel_no_candidate(a, i, vc)) e = b;
        Best best = none_best();
        if (a.initial) {
            for (i64 j = b + threadIdx.x; j < e; j += LS_THREADS)
                sel_eval<W, CON>(a, vc, a.g.col[j], V(a.g.wgt(j)), best);
        } else if (e > b) {
            sel_dense_row<W, CON, true>(a, i, vc, b, e, L, smem, LS_TABLE_BYTES, best);
        }
        warp_best(best);
        if (l == 0) wb[w] = best;
        __syncthreads();
        if (w == 0) {
            best = l < LS_WARPS ? wb[l] : none_best();
            warp_best(best);
            if (l == 0) sel_finish(a, i, vc, best);
        }
        __syncthreads();
    }
}

// own-cluster weights of every vertex (all) or of the flagged ones, whose
// flag and dest cache are reset
template <class W>
__device__ __forceinline__ void own_step(const SmallArgs<W>& a, bool all, typename Traits<W>::V* out) {
    using V = typename Traits<W>::V;
    const DGraph<W>& g = a.g;
    const i32* lab = a.part;
    vsum_step<V>(
        a.cls, a.off, 6,
        [&](i32 i, i64& b, i64& e) -> OwnRow<W> {
            OwnRow<W> row{g, lab, -1};  // -1: skipped
            if (i >= 0 && (all || a.flags[i])) {
                row.li = lab[i];
                b = g.rowptr[i];
                e = g.rowptr[i + 1];
            }
            return row;
        },
        [&](i32 i, const OwnRow<W>& row, V v) {
            if (row.li < 0) return;
            out[i] = v;
            a.dest[i] = NULL_PART;
            a.flags[i] = 0;
        });
}

// afterburner: keep[i] = the move stands; counts the moves and the NEW_PART ones
template <class W>
__device__ __forceinline__ void afterburner_step(const SmallArgs<W>& a, unsigned long long* cnt, int* sh) {
    ABArgs<W> ab;
    ab.g = a.g;
    ab.part = a.part;
    ab.dest = a.dest;
    ab.gain = a.gain;
    ab.pm = a.pm;
    if (threadIdx.x < 2) sh[threadIdx.x] = 0;
    __syncthreads();
    int nm = 0, nn = 0;
    // (a thread's terms wait for one another's branches: 22 against 20 us for
    // the 51,000 vertices of 17-32 edges of a 65,536-vertex graph)
    vsum_step<double>(
        a.cls, a.off, 16,
        [&](i32 i, i64& b, i64& e) -> AbRow<W> {
            AbRow<W> row{ab, 0, NO_MOVE, 0, 0.f, 0.f};
            if (i >= 0) row.best = a.dest[i];
            if (row.best != NO_MOVE) {
                row.p = a.part[i];
                row.multi = to_f(a.g.vtx_w[i]) * a.pm;
                row.igain = a.gain[i];
                row.hi = (i32)xorshift32((u32)i);
                b = a.g.rowptr[i];
                e = a.g.rowptr[i + 1];
            }
            return row;
        },
        [&](i32 i, const AbRow<W>& row, double ch) {
            const bool k = row.best != NO_MOVE && (row.igain + (float)ch) >= 0.0f;
            a.keep[i] = k ? 1 : 0;
            nm += k ? 1 : 0;
            nn += k && row.best == NEW_PART ? 1 : 0;
        });
    nm = __reduce_add_sync(FULL, nm);
    nn = __reduce_add_sync(FULL, nn);
    if (lane_id() == 0 && nm) {
        atomicAdd(&sh[0], nm);
        if (nn) atomicAdd(&sh[1], nn);
    }
    __syncthreads();
    if (threadIdx.x == 0 && sh[0]) {
        atomicAdd(&cnt[0], (unsigned long long)sh[0]);
        if (sh[1]) atomicAdd(&cnt[1], (unsigned long long)sh[1]);
    }
}

// set_new_cluster_ids (src/local_mover.cpp:217-274): the NEW_PART movers in
// order1 order take the unused labels in ascending order, then appended ones.
// Returns the new label count.
template <class W, bool CON>
__device__ __forceinline__ i64 new_ids_step(const SmallArgs<W>& a, i64 L, int* wcnt) {
    using V = typename Traits<W>::V;
    const i64 n = a.g.n;
    const i64 t0 = (i64)blockIdx.x * LS_THREADS + threadIdx.x, nt = (i64)gridDim.x * LS_THREADS;
    for (i64 x = t0; x < L; x += nt) a.has[x] = 0;
    gang_sync();
    for (i64 i = t0; i < n; i += nt) a.has[a.part[i]] = 1;
    auto is_new = [&](i64 x) {
        const i32 i = a.order1[x];
        return a.dest[i] == NEW_PART && a.keep[i];
    };
    gang_count(n, is_new, a.blk);
    gang_sync();
    auto unused = [&](i64 x) { return a.has[x] == 0; };
    gang_count(L, unused, a.blk + 32);
    gang_emit(n, is_new, [&](i64 x, i64 r) { a.newl[r] = a.order1[x]; }, a.blk, wcnt);
    gang_sync();
    gang_emit(L, unused, [&](i64 x, i64 r) { a.avail[r] = (i32)x; }, a.blk + 32, wcnt);
    gang_sync();
    const i64 nn = gang_total(a.blk), na = gang_total(a.blk + 32);
    for (i64 r = t0; r < nn; r += nt) {
        const i32 x = a.newl[r];
        const i64 lab = r < na ? (i64)a.avail[r] : L + (r - na);
        if (lab >= a.cap) {
            atomicExch(a.err, (int)DEV_ERR_LABEL);
            continue;
        }
        a.dest[x] = (i32)lab;
        if (CON) a.constraint[lab] = a.constraint[a.part[x]];
        if (r >= na) a.td[lab] = V(0);
    }
    gang_sync();
    return nn > na ? min(L + (nn - na), a.cap) : L;
}

// perform_moves (src/local_mover.cpp:1241-1279): volumes and labels of the
// movers; with `mark`, the movers and their neighbours are flagged
template <class W>
__device__ __forceinline__ void moves_step(const SmallArgs<W>& a, bool mark, i32 stamp) {
    const DGraph<W>& g = a.g;
    const int l = lane_id();
    const i64 nw = gang_warps(), n = g.n;
    auto is_mover = [&](i32 i) { return a.dest[i] != NO_MOVE && a.keep[i]; };
    for (i64 i = (i64)gang_warp() * 32 + l; i < n; i += nw * 32) {
        if (!is_mover((i32)i)) continue;
        const i32 b = a.dest[i], p = a.part[i];
        if (b < 0) {  // an unresolved NEW_PART: never applied
            atomicExch(a.err, (int)DEV_ERR_LABEL);
            continue;
        }
        const auto wv = g.vtx_w[i];
        vatomic_add(&a.td[p], -wv);
        vatomic_add(&a.td[b], wv);
        a.part[i] = b;
        if (a.csize) {
            atomicSub(&a.csize[p], 1);
            atomicAdd(&a.csize[b], 1);
            a.moved_at[i] = stamp;
        }
    }
    if (!mark) return;
    // rows of up to 32 edges by 8-lane groups, longer ones by a warp
    const i64 o0 = a.off[0], o3 = a.off[3], o7 = a.off[7];
    const int r = l & 7, grp = l >> 3;
    i64 rot = 0;
    for (i64 base = o0 + gang_first(rot) * 4; base < o3; base += nw * 4) {
        const i64 x = base + grp;
        if (x >= o3) continue;
        const i32 i = a.cls[x];
        if (!is_mover(i)) continue;
        const i64 b = g.rowptr[i], e = g.rowptr[i + 1];
        if (r == 0) a.flags[i] = 1;
#pragma unroll 4
        for (i64 j = b + r; j < e; j += 8) a.flags[g.col[j]] = 1;
    }
    rot += (o3 - o0 + 3) >> 2;
    for (i64 x = o3 + gang_first(rot); x < o7; x += nw) {
        const i32 i = a.cls[x];
        if (!is_mover(i)) continue;
        const i64 b = g.rowptr[i], e = g.rowptr[i + 1];
        if (l == 0) a.flags[i] = 1;
#pragma unroll 4
        for (i64 j = b + l; j < e; j += 32) a.flags[g.col[j]] = 1;
    }
}

// The learned filter before a sweep's select (see filter.cuh).
template <class W>
__device__ __forceinline__ void filter_step(FiltArgs<W> f, unsigned char* smem) {
    float* xs = (float*)(smem + (threadIdx.x >> 5) * LS_WARP_BYTES);
    filter_warps(f, xs, xs + 32 * FW_XS, (i64)gang_warp(), (i64)gang_warps());
    __syncwarp();
}

// ---- algorithmic bytes (profiling only) ----------------------------------------
// Counted before a step from the state that it will read, as the class kernels
// count while they run.
template <class F>
__device__ __forceinline__ void count_bytes(i64 k, F f, unsigned long long* prof) {
    unsigned long long pb = 0;
    for (i64 x = (i64)blockIdx.x * LS_THREADS + threadIdx.x; x < k; x += (i64)gridDim.x * LS_THREADS) pb += f(x);
    pb = (unsigned long long)warp_sum_i64((i64)pb);
    if (lane_id() == 0 && pb) atomicAdd(prof, pb);
}
template <class W>
__device__ __forceinline__ void count_select(const SelArgs<W>& s, const i32* list, i64 count, unsigned long long* prof) {
    count_bytes(count, [&](i64 x) {
        const i32 i = list[x];
        if (s.dest[i] == NO_MOVE) return sel_bytes(s, 0, false);
        return sel_bytes(s, sel_no_candidate(s, i, sel_prologue(s, i)) ? 0 : s.g.rowptr[i + 1] - s.g.rowptr[i], true);
    }, prof);
}
template <class W>
__device__ __forceinline__ void count_afterburner(const SmallArgs<W>& a, unsigned long long* prof) {
    ABArgs<W> ab{};
    ab.g = a.g;
    count_bytes(a.g.n, [&](i64 i) {
        return a.dest[i] == NO_MOVE ? 0ull : ab_bytes(ab, a.g.rowptr[i + 1] - a.g.rowptr[i]);
    }, prof);
}
template <class W>
__device__ __forceinline__ void count_own(const SmallArgs<W>& a, bool all, unsigned long long* prof) {
    count_bytes(a.g.n, [&](i64 i) {
        return all || a.flags[i] ? own_bytes(a.g, a.g.rowptr[i + 1] - a.g.rowptr[i]) : 0ull;
    }, prof);
}

}  // namespace pggc
