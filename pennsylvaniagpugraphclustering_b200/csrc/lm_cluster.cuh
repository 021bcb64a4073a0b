// lm_cluster.cuh -- a whole local move of a small graph in one launch.
//
// A local move is up to six sweeps of select, afterburner, moves, own-cluster
// weights and objective (src/local_mover.cpp:1361-1417).  On graphs of a few
// thousand vertices every one of those steps is shorter than the launch that
// starts it: launched one by one (about 30 kernels, two compactions and a host
// round trip a sweep) a sweep takes 140-170 us whatever the graph's size.
// Here one thread-block cluster runs the local move from the copy of the input
// partition to the relabelling of the result: the steps are separated by the
// cluster's hardware barrier (which also orders global memory among its
// blocks) and the sweep decisions are taken on the device, so the host queues
// one launch and reads one result.  A cluster and not a cooperative grid: its
// blocks are scheduled together by the hardware, the barrier needs no
// spinning, and the local moves of a batch's other streams run beside it on
// the other SMs.
#pragma once
#include "lm_steps.cuh"

namespace pggc {

template <class W, bool CON, bool FILT>
__global__ void __launch_bounds__(LS_THREADS, 1) k_local_move_small(SmallArgs<W> a) {
    using V = typename Traits<W>::V;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ V red[32];
    __shared__ Best wb[LS_WARPS];
    __shared__ int sh[LS_WARPS];
    __shared__ i64 s_off[NCLS + 1];
    if (threadIdx.x <= NCLS) s_off[threadIdx.x] = a.off[threadIdx.x];
    a.off = s_off;
    const i64 n = a.g.n;
    const i64 t0 = (i64)blockIdx.x * LS_THREADS + threadIdx.x, nt = (i64)gridDim.x * LS_THREADS;

    // current state <- best state (src/local_mover.cpp:1365-1368)
    for (i64 i = t0; i < n; i += nt) {
        a.part[i] = a.best_part[i];
        a.dest[i] = NULL_PART;
        a.flags[i] = 0;
        if (a.initial) {
            a.pvals[i] = V(0);
            a.pv_best[i] = V(0);
        } else if (a.reuse) {
            a.pvals[i] = a.pv_best[i];
        }
        if (FILT) {
            a.moved_at[i] = -1;
            a.gain[i] = 0.f;
        }
    }
    for (i64 c = t0; c < a.label_count; c += nt) {
        a.td[c] = a.td_best[c];
        if (FILT) a.csize[c] = 0;
    }
    if (FILT)
        for (i64 c = a.label_count + t0; c < a.cap; c += nt) a.csize[c] = 0;
    if (t0 < 2 * LS_MAX_SWEEPS) a.cnt[t0] = 0;
    gang_sync();
    if (FILT)
        for (i64 i = t0; i < n; i += nt) atomicAdd(&a.csize[a.part[i]], 1);
    V last_pval = V(0);
    bool have_pvals = a.initial == 0;
    if (have_pvals) {
        if (!a.reuse) {
            if (a.prof) count_own(a, true, a.prof);
            own_step(a, true, a.pvals);
            gang_sync();
            for (i64 i = t0; i < n; i += nt) a.pv_best[i] = a.pvals[i];
        }
        chunk_sums<V>(n, [&](i64 i) { return a.pvals[i]; }, a.partial, red, 0);
        gang_sync();
        last_pval = chunk_total<V>(n, a.partial, red);
    }
    // every block holds the same copy of the scalars
    i64 L = a.label_count, best_L = L;
    V uncut = a.uncut, best_uncut = uncut;
    double best_obj = a.obj;
    int sweeps = 0;
    i64 moves = 0;

    SelArgs<W> s;
    s.g = a.g;
    s.part = a.part;
    s.dest = a.dest;
    s.gain = a.gain;
    s.pvals = a.pvals;
    s.td = a.td;
    s.constraint = a.constraint;
    s.label_count = nullptr;
    s.rsum = a.rsum;
    s.units = a.units;
    s.keys32 = a.keys32;
    s.dense = 0;
    s.pm = a.pm;
    s.err = a.err;
    s.prof = nullptr;
    s.probe_cap = 0;
    s.inv_load = a.inv_load;

    for (int x = 0; x < 2; x++) {
        const int limit = x == 0 ? 4 : 2;
        s.fr = a.sa && !a.strict ? (x == 0 ? 0.75f : 0.25f) : 0.0f;
        for (int count = 0; count < limit; count++) {
            if (a.sweep_limit >= 0 && sweeps >= a.sweep_limit) break;
            const int k = sweeps++;  // counter slot of the sweep
            gang_sync();             // labels, volumes, flags of the last sweep
            if (FILT) {
                FiltArgs<W> f = a.filt;
                f.sweep_f = (float)k / 8.f;
                f.prev_stamp = a.filt.prev_stamp + k;
                filter_step(f, smem);
                gang_sync();
            }
            s.initial = have_pvals ? 0 : 1;
            if (a.prof) {
                count_select(s, a.cls, n, a.prof);
                gang_sync();  // the select step writes dest
            }
            select_step<W, CON>(s, a.cls, a.off, L, smem, wb);
            gang_sync();
            if (a.strict) {
                // The strict variant (src/local_mover.cpp:1422-1483) mostly runs
                // where the last local move ended, finds no candidate and stops:
                // that sweep runs here, anything more on the general path, from
                // the untouched best state.
                int any = 0;
                for (i64 i = t0; i < n; i += nt) any |= a.dest[i] != NO_MOVE;
                if (__syncthreads_or(any) && threadIdx.x == 0) atomicExch(&a.cnt[0], 1ull);
                gang_sync();
                if (a.cnt[0] != 0) {
                    if (t0 == 0) a.sc->num_cand = 1;
                    return;
                }
                x = 2;
                break;
            }
            if (a.prof) count_afterburner(a, a.prof);
            afterburner_step(a, a.cnt + 2 * k, sh);
            gang_sync();
            const i64 nm = (i64)a.cnt[2 * k];
            if (nm == 0) break;
            if ((k > 0 || !a.initial) && a.cnt[2 * k + 1] != 0) L = new_ids_step<W, CON>(a, L, sh);
            moves_step(a, have_pvals, FILT ? a.filt.prev_stamp + k + 1 : 0);
            gang_sync();
            if (a.prof) {
                count_own(a, !have_pvals, a.prof);
                gang_sync();  // the step clears the flags
            }
            own_step(a, !have_pvals, a.pvals);
            have_pvals = true;
            chunk_sums<V>(L, [&](i64 c) { const V t = a.td[c]; return t * t; }, a.partial + a.sq_at, red,
                          (int)((n + 1023) >> 10));
            gang_sync();
            chunk_sums<V>(n, [&](i64 i) { return a.pvals[i]; }, a.partial, red, 0);
            gang_sync();
            // objective (interface/cluster_data.hpp:76-87)
            const V pv = chunk_total<V>(n, a.partial, red);
            const V sq = chunk_total<V>(L, a.partial + a.sq_at, red);
            const V change = pv - last_pval;
            last_pval = pv;
            uncut = uncut + change;
            double m = (double)uncut;
            m = m - a.lambda * (double)sq;
            if (m > best_obj) {
                best_obj = m;
                best_uncut = uncut;
                best_L = L;
                for (i64 i = t0; i < n; i += nt) {
                    a.best_part[i] = a.part[i];
                    a.pv_best[i] = a.pvals[i];
                }
                for (i64 c = t0; c < L; c += nt) a.td_best[c] = a.td[c];
            }
            moves += nm;
        }
    }
    // relabel_contiguously (src/local_mover.cpp:100-129) of the best state
    for (i64 c = t0; c < best_L; c += nt) a.has[c] = 0;
    gang_sync();
    for (i64 i = t0; i < n; i += nt) {
        const i32 c = a.best_part[i];
        if (c >= 0 && c < best_L) a.has[c] = 1;
    }
    gang_sync();
    auto used = [&](i64 c) { return a.has[c] != 0; };
    gang_count(best_L, used, a.blk + 64);
    gang_sync();
    gang_emit(best_L, used, [&](i64 c, i64 r) {
        a.newid[c] = (i32)r;
        a.td2[r] = a.td_best[c];
    }, a.blk + 64, sh);
    const i64 used_count = gang_total(a.blk + 64);
    gang_sync();
    for (i64 i = t0; i < n; i += nt) {
        const i32 c = a.best_part[i];
        if (c >= 0 && c < best_L) a.best_part[i] = a.newid[c];
    }
    for (i64 r = t0; r < used_count; r += nt) a.td_best[r] = a.td2[r];
    if (t0 == 0) {
        a.sc->best_label_count = best_L;
        a.sc->relabel_count = used_count;
        a.sc->best_uncut = best_uncut;
        a.sc->best_obj = best_obj;
        a.sc->num_cand = 0;
        a.sc->num_moves = moves;
        a.sc->split = sweeps;
        a.sc->err = *(volatile int*)a.err;
    }
}

template <class W>
bool local_move_small(Context& ctx, const Graph<W>& g, const Ordering& ord, i32* best_part,
                      ClusterState<typename Traits<W>::V>& best, bool is_initial, bool constrained, i32* constraint,
                      bool enable_sa, bool strict, int sweep_limit, MoveStats* stats, bool reuse_pvals) {
    using V = typename Traits<W>::V;
    const i64 n = g.n;
    const bool long_rows = g.nnz >= 64 * n;
    const bool fits =
        long_rows ? g.nnz <= LS_MOVE_NNZ_LONG : g.nnz <= LS_MOVE_NNZ && g.nnz + 4 * n <= LS_MOVE_SIZE;
    const int want = fits ? small_cluster_blocks(n, g.nnz) : 0;
    auto& F = ctx.filt;
    const bool filt_on = F.mode != 0 && !strict;
    const bool gating = F.mode == 2 && !strict && !F.suspended && F.level >= F.min_level &&
                        !(F.max_pass >= 0 && F.pass >= F.max_pass);
    // logging runs, rows summed by 1024 threads and injected probe faults keep the general path
    if (want == 0 || F.mode == 1 || (gating && constrained) || ord.off_large2 < n || ctx.probe_cap != 0 ||
        best.label_count > LS_MAX_LABELS || (strict && sweep_limit == 0))
        return false;
    const auto kern = gating        ? k_local_move_small<W, false, true>
                      : constrained ? k_local_move_small<W, true, false>
                                    : k_local_move_small<W, false, false>;
    const int blocks = gang_blocks(ctx, kern, want);
    if (blocks == 0) return false;
    ProfScope ps(ctx, "local_move_small");
    const ClassLists cls = graph_class_lists<W>(ctx, g, ord);
    // labels that the sweeps can reach: each appends at most one per vertex
    const i64 cap = std::min<i64>(best.capacity, best.label_count + LS_MAX_SWEEPS * n);
    SmallArgs<W> a{};
    a.g = g.view();
    a.cls = cls.list;
    a.off = cls.off;
    a.order1 = ord.order1.p;
    a.rsum = row_sums<W>(ctx, g);
    a.units = g.units.p;
    a.part = ctx.ws_get<i32>(LM_PART, n);
    a.dest = ctx.ws_get<i32>(LM_DEST, n);
    a.gain = ctx.ws_get<float>(LM_GAIN, n);
    a.keep = ctx.ws_get<unsigned char>(LM_KEEP, n);
    a.flags = ctx.ws_get<unsigned char>(LM_FLAGS, n);
    a.has = ctx.ws_get<unsigned char>(LM_HAS, cap);
    a.pvals = ctx.ws_get<V>(LM_PV, n);
    a.pv_best = ctx.ws_get<V>(LM_PVC, n);
    a.td = ctx.ws_get<V>(LM_TD, cap);
    a.best_part = best_part;
    a.td_best = best.total_deg.p;
    a.constraint = constraint;
    a.newl = ctx.ws_get<i32>(LM_NEWL, n);
    a.avail = ctx.ws_get<i32>(LM_AVAIL, cap);
    a.newid = ctx.ws_get<i32>(LM_NEWID, cap);
    a.td2 = ctx.ws_get<V>(LM_TD2, cap);
    a.partial = ctx.ws_get<V>(LM_PARTIAL, 2048);
    a.sq_at = 1024;
    a.blk = ctx.ws_get<i64>(LM_BLK, 96);
    a.cnt = ctx.ws_get<unsigned long long>(LM_CNT, 2 * LS_MAX_SWEEPS);
    a.sc = ctx.ws_get<LMScalars<V>>(LM_SC, 1);
    a.prof = ctx.prof_counter("local_move_small");
    a.err = ctx.d_err;
    a.cap = cap;
    a.label_count = best.label_count;
    a.uncut = best.uncut;
    a.obj = best.obj;
    a.lambda = best.lambda;
    a.pm = (float)best.lambda;
    a.inv_load = ctx.tune.load >= 0.7f ? 1.0f / 0.7f : 2.0f;
    a.initial = is_initial ? 1 : 0;
    a.sa = enable_sa ? 1 : 0;
    a.strict = strict ? 1 : 0;
    a.sweep_limit = sweep_limit;
    a.keys32 = cap < ((i64)1 << 29) ? 1 : 0;
    a.reuse = reuse_pvals && !is_initial && ctx.pv_uid == g.uid && ctx.pv_n == n && ctx.pv_ptr == (const void*)a.pv_best;
    const u64 pv_uid = ctx.pv_uid;
    ctx.pv_uid = 0;
    if (gating) {
        a.moved_at = ctx.ws_get<i32>(LM_MOVED_AT, n);
        a.csize = ctx.ws_get<i32>(LM_CSIZE, cap);
        FiltArgs<W>& f = a.filt;
        f.g = a.g;
        f.part = a.part;
        f.pvals = a.pvals;
        f.gain = a.gain;
        f.moved_at = a.moved_at;
        f.csize = a.csize;
        f.td = a.td;
        f.dest = a.dest;
        f.inv_vol = best.vol_total > 0 ? (float)(1.0 / best.vol_total) : 0.f;
        f.inv_log_n = (float)(1.0 / std::log2(2.0 + (double)n));
        f.level_f = (float)F.level / 16.f;
        f.prev_stamp = F.stamp;  // sweep k runs as stamp F.stamp + k + 1
        f.mode = F.mode;
        f.net = F.net;
        f.threshold = F.threshold;
        f.stats = F.stats;
    }
    launch_gang(ctx, kern, a, blocks);
    const LMScalars<V>* h = (const LMScalars<V>*)ctx.readback(a.sc, sizeof(LMScalars<V>));
    if (h->num_cand != 0) {  // strict, with candidates: the retained weights still stand
        ctx.pv_uid = pv_uid;
        return false;
    }
    const int err = h->err;
    best.label_count = h->best_label_count;
    best.uncut = h->best_uncut;
    best.obj = h->best_obj;
    const i64 used = h->relabel_count, sweeps = h->split, moves = h->num_moves;
    if (filt_on) F.stamp += (i32)sweeps;
    ctx.raise_device_error(err);
    best.label_count = used;
    ctx.pv_uid = g.uid;
    ctx.pv_ptr = a.pv_best;
    ctx.pv_n = n;
    if (stats) {
        stats->sweeps += sweeps;
        stats->moves += moves;
    }
    return true;
}

}  // namespace pggc
