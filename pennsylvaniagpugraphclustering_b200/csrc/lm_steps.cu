// lm_steps.cu -- the steps of a sweep as launches of their own.
//
// For graphs above the one-launch size (lm_cluster.cuh): one launch covers all
// degree classes (they share the launch's threads), moves are counted where
// the afterburner decides them and found again by their flag instead of from
// compacted lists, and array sums take one pass: seven launches a sweep in
// place of about thirty.
#include "lm_steps.cuh"

namespace pggc {

constexpr int ST_WARP_BYTES = 3 * 1024;

template <class W>
__global__ void __launch_bounds__(LS_THREADS, 2) k_step_init(SmallArgs<W> a) {
    using V = typename Traits<W>::V;
    const i64 t0 = (i64)blockIdx.x * LS_THREADS + threadIdx.x, nt = (i64)gridDim.x * LS_THREADS, n = a.g.n;
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
    }
    for (i64 c = t0; c < a.label_count; c += nt) a.td[c] = a.td_best[c];
    if (t0 < 2) a.cnt[t0] = 0;
    if (t0 == 0) {
        LMScalars<V> h{};
        h.label_count = h.best_label_count = a.label_count;
        h.uncut = h.best_uncut = a.uncut;
        h.obj = h.best_obj = a.obj;
        *a.sc = h;
    }
}
template <class W, bool CON>
__global__ void __launch_bounds__(LS_THREADS, 2) k_step_select(SelArgs<W> s, const i32* cls, const i64* off) {
    extern __shared__ __align__(16) unsigned char smem[];
    select_low<W, CON>(s, cls, off, smem + (threadIdx.x >> 5) * ST_WARP_BYTES);
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS, 2) k_step_afterburner(SmallArgs<W> a) {
    __shared__ int sh[2];
    afterburner_step(a, a.cnt, sh);
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS, 2) k_step_moves(SmallArgs<W> a, bool mark, i32 stamp) {
    moves_step(a, mark, stamp);
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS, 2) k_step_own(SmallArgs<W> a, bool all) {
    using V = typename Traits<W>::V;
    __shared__ V red[32];
    own_step(a, all, a.pvals);
    const i64 L = a.sc->label_count;
    chunk_sums<V>(L, [&](i64 c) { const V t = a.td[c]; return t * t; }, a.partial + a.sq_at, red, 0);
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS, 2) k_step_sums(SmallArgs<W> a) {
    using V = typename Traits<W>::V;
    __shared__ V red[32];
    chunk_sums<V>(a.g.n, [&](i64 i) { return a.pvals[i]; }, a.partial, red, 0);
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS) k_step_objective(SmallArgs<W> a, bool sweep) {
    using V = typename Traits<W>::V;
    __shared__ V red[32];
    __shared__ V upper[32];
    LMScalars<V>* sc = a.sc;
    const i64 L = sc->label_count;
    const V pv = chunk_total_wide<V>(a.g.n, a.partial, red, upper);
    const V sq = sweep ? chunk_total_wide<V>(L, a.partial + a.sq_at, red, upper) : V(0);
    if (threadIdx.x != 0) return;
    const V change = pv - sc->last_pval;
    sc->last_pval = pv;
    a.cnt[0] = 0;  // of the next sweep
    a.cnt[1] = 0;
    if (!sweep) return;
    sc->uncut = sc->uncut + change;
    double m = (double)sc->uncut;
    m = m - a.lambda * (double)sq;
    sc->obj = m;
    sc->improved = m > sc->best_obj ? 1 : 0;
    if (sc->improved) {
        sc->best_obj = m;
        sc->best_uncut = sc->uncut;
        sc->best_label_count = L;
    }
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS, 2) k_step_keep_best(SmallArgs<W> a, bool sweep) {
    if (sweep && !a.sc->improved) return;
    const i64 t0 = (i64)blockIdx.x * LS_THREADS + threadIdx.x, nt = (i64)gridDim.x * LS_THREADS, n = a.g.n;
    for (i64 i = t0; i < n; i += nt) {
        if (sweep) a.best_part[i] = a.part[i];
        a.pv_best[i] = a.pvals[i];
    }
    if (!sweep) return;
    const i64 L = a.sc->label_count;
    for (i64 c = t0; c < L; c += nt) a.td_best[c] = a.td[c];
}

// blocks of a step with `warps` warps of work, two to an SM
inline int step_grid(Context& ctx, i64 warps) {
    return (int)std::max<i64>(1, std::min<i64>(ceil_div(warps, LS_WARPS), (i64)ctx.num_sms * 2));
}
template <class W>
void step_init(Context& ctx, const SmallArgs<W>& a) {
    k_step_init<W><<<step_grid(ctx, ceil_div(std::max<i64>(a.g.n, a.label_count), 32)), LS_THREADS, 0, ctx.stream>>>(a);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_select(Context& ctx, const SelArgs<W>& s, const i32* cls, const i64* off, i64 count, bool constrained) {
    auto kern = constrained ? k_step_select<W, true> : k_step_select<W, false>;
    const int smem = ST_WARP_BYTES * LS_WARPS;
    set_dynamic_smem_once(kern, smem, ctx.device);
    kern<<<step_grid(ctx, ceil_div(count, 4)), LS_THREADS, smem, ctx.stream>>>(s, cls, off);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_afterburner(Context& ctx, const SmallArgs<W>& a) {
    k_step_afterburner<W><<<step_grid(ctx, ceil_div(a.g.n, 4)), LS_THREADS, 0, ctx.stream>>>(a);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_moves(Context& ctx, const SmallArgs<W>& a, bool mark, i32 stamp) {
    k_step_moves<W><<<step_grid(ctx, ceil_div(a.g.n, 4)), LS_THREADS, 0, ctx.stream>>>(a, mark, stamp);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_own(Context& ctx, const SmallArgs<W>& a, bool all) {
    k_step_own<W><<<step_grid(ctx, ceil_div(a.g.n, 4)), LS_THREADS, 0, ctx.stream>>>(a, all);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_sums(Context& ctx, const SmallArgs<W>& a) {
    k_step_sums<W><<<(int)std::min<i64>(ceil_div(a.g.n, 1024), (i64)ctx.num_sms * 2), LS_THREADS, 0, ctx.stream>>>(a);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_objective(Context& ctx, const SmallArgs<W>& a, bool sweep, i64 label_bound) {
    k_step_objective<W><<<1, LS_THREADS, 0, ctx.stream>>>(a, sweep);
    PGGC_LAUNCH_CHECK();
    if (!sweep && a.reuse) return;  // the best state's weights are the start's
    k_step_keep_best<W><<<step_grid(ctx, ceil_div(std::max(a.g.n, label_bound), 32)), LS_THREADS, 0, ctx.stream>>>(
        a, sweep);
    PGGC_LAUNCH_CHECK();
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS) k_step_select_bytes(SelArgs<W> s, const i32* cls, i64 count,
                                                                  unsigned long long* prof) {
    count_select(s, cls, count, prof);
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS) k_step_afterburner_bytes(SmallArgs<W> a, unsigned long long* prof) {
    count_afterburner(a, prof);
}
template <class W>
__global__ void __launch_bounds__(LS_THREADS) k_step_own_bytes(SmallArgs<W> a, bool all, unsigned long long* prof) {
    count_own(a, all, prof);
}
template <class W>
void step_select_bytes(Context& ctx, const SelArgs<W>& s, const i32* cls, i64 count, unsigned long long* prof) {
    if (!prof) return;
    k_step_select_bytes<W><<<step_grid(ctx, ceil_div(count, 32)), LS_THREADS, 0, ctx.stream>>>(s, cls, count, prof);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_afterburner_bytes(Context& ctx, const SmallArgs<W>& a, unsigned long long* prof) {
    if (!prof) return;
    k_step_afterburner_bytes<W><<<step_grid(ctx, ceil_div(a.g.n, 32)), LS_THREADS, 0, ctx.stream>>>(a, prof);
    PGGC_LAUNCH_CHECK();
}
template <class W>
void step_own_bytes(Context& ctx, const SmallArgs<W>& a, bool all, unsigned long long* prof) {
    if (!prof) return;
    k_step_own_bytes<W><<<step_grid(ctx, ceil_div(a.g.n, 32)), LS_THREADS, 0, ctx.stream>>>(a, all, prof);
    PGGC_LAUNCH_CHECK();
}

#define PGGC_INST_STEP(W)                                                                                \
    template void step_init<W>(Context&, const SmallArgs<W>&);                                           \
    template void step_select<W>(Context&, const SelArgs<W>&, const i32*, const i64*, i64, bool);        \
    template void step_afterburner<W>(Context&, const SmallArgs<W>&);                                    \
    template void step_moves<W>(Context&, const SmallArgs<W>&, bool, i32);                               \
    template void step_own<W>(Context&, const SmallArgs<W>&, bool);                                      \
    template void step_sums<W>(Context&, const SmallArgs<W>&);                                           \
    template void step_select_bytes<W>(Context&, const SelArgs<W>&, const i32*, i64, unsigned long long*); \
    template void step_afterburner_bytes<W>(Context&, const SmallArgs<W>&, unsigned long long*);         \
    template void step_own_bytes<W>(Context&, const SmallArgs<W>&, bool, unsigned long long*);           \
    template void step_objective<W>(Context&, const SmallArgs<W>&, bool, i64);
PGGC_INST_STEP(i32)
PGGC_INST_STEP(float)

// Sixteen blocks (the largest cluster) are the fastest from 1,000 vertices up:
// six sweeps of an SBM of mean degree 14 take 456 / 293 / 239 / 205 us with 1 /
// 4 / 8 / 16 blocks at 1,000 vertices, 1,627 / 618 / 421 / 333 us at 4,000, and
// 2,096 / 682 / 429 / 320 us at 1,000 vertices of 83 FP32 edges; at 300
// vertices (4 K edges) 232 / 205 / 168 / 167.
int small_cluster_blocks(i64 n, i64 nnz) {
    if (n > LS_MAX_N || nnz > LS_MAX_NNZ) return 0;
    return nnz + 4 * n <= 4096 ? 8 : 16;
}

}  // namespace pggc
