// gang.cuh -- steps run by all blocks of one thread-block cluster.
//
// The kernels for small graphs (lm_cluster.cuh, contract_small.cu, ...) run a
// whole sequence of steps in one launch of a single cluster, "the gang": the
// steps loop over their items with the gang's threads or warps and are
// separated by gang_sync().
#pragma once
#include "sweep.cuh"

namespace pggc {

constexpr int LS_THREADS = 512;
constexpr int LS_WARPS = LS_THREADS / 32;
constexpr int LS_TABLE_BYTES = 160 * 1024;             // hash / dense tables of one block
constexpr int LS_WARP_BYTES = LS_TABLE_BYTES / LS_WARPS;  // a warp's share

// All blocks of the launch (one cluster): threads may read after it what any
// thread wrote before it.
__device__ __forceinline__ void gang_sync() {
    if (gridDim.x == 1) {
        __syncthreads();
    } else {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// Consecutive warps of work go to different SMs.
__device__ __forceinline__ int gang_warp() { return (threadIdx.x >> 5) * gridDim.x + blockIdx.x; }
__device__ __forceinline__ int gang_warps() { return LS_WARPS * gridDim.x; }

// First unit of work of this warp when earlier work in the step has used `rot`
// warps: steps over several classes spread their vertices over all warps.
__device__ __forceinline__ i64 gang_first(i64 rot) {
    const int nw = gang_warps();
    return (gang_warp() + nw - (int)(rot % nw)) % nw;
}

// sum over [base, base + 1024) of f(i), i < k, in the canonical association
// (groups of 32 by xor butterfly, then the 32 group totals); every thread
// returns it
template <class V, class F>
__device__ __forceinline__ V chunk_sum(i64 base, i64 k, F f, V* red) {
    const int l = lane_id();
    for (int gidx = threadIdx.x >> 5; gidx < 32; gidx += LS_WARPS) {
        const i64 i = base + gidx * 32 + l;
        V v = i < k ? f(i) : V(0);
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) v = v + __shfl_xor_sync(FULL, v, d);
        if (l == 0) red[gidx] = v;
    }
    __syncthreads();
    V t = red[l];
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) t = t + __shfl_xor_sync(FULL, t, d);
    __syncthreads();
    return t;
}

// chunk sums of f over [0, k) into out, chunk c by block c mod blocks
template <class V, class F>
__device__ __forceinline__ void chunk_sums(i64 k, F f, V* out, V* red, int first_block) {
    const i64 nch = (k + 1023) >> 10;
    for (i64 c = (blockIdx.x + gridDim.x - first_block % gridDim.x) % gridDim.x; c < nch; c += gridDim.x) {
        const V s = chunk_sum<V>(c << 10, k, f, red);
        if (threadIdx.x == 0) out[c] = s;
    }
}
// total of the chunk sums (k <= 2^20 elements)
template <class V>
__device__ __forceinline__ V chunk_total(i64 k, const V* part, V* red) {
    if (k <= 0) return V(0);
    const i64 nch = (k + 1023) >> 10;
    if (nch == 1) return part[0];
    return chunk_sum<V>(0, nch, [&](i64 i) { return part[i]; }, red);
}

// the same for up to 2^25 elements (upper: 32 values of shared memory)
template <class V>
__device__ __forceinline__ V chunk_total_wide(i64 k, const V* part, V* red, V* upper) {
    const i64 nch = (k + 1023) >> 10;
    if (nch <= 1024) return chunk_total<V>(k, part, red);
    const int nup = (int)((nch + 1023) >> 10);
    for (int c = 0; c < nup; c++) {
        const V s = chunk_sum<V>((i64)c << 10, nch, [&](i64 i) { return part[i]; }, red);
        if (threadIdx.x == 0) upper[c] = s;
        __syncthreads();
    }
    return chunk_sum<V>(0, nup, [&](i64 i) { return upper[i]; }, red);
}

// Ordered compaction of [0, k): block b owns a contiguous range.  count: this
// block's flags into blk[b]; emit (after a gang_sync): e(x, rank) for every
// flagged x with its rank among all flagged positions.
__device__ __forceinline__ void gang_range(i64 k, i64& lo, i64& hi) {
    const i64 per = (k + gridDim.x - 1) / gridDim.x;
    lo = min(k, per * blockIdx.x);
    hi = min(k, lo + per);
}
template <class F>
__device__ __forceinline__ void gang_count(i64 k, F f, i64* blk) {
    i64 lo, hi, c = 0;
    gang_range(k, lo, hi);
    for (i64 x0 = lo; x0 < hi; x0 += LS_THREADS) {
        const i64 x = x0 + threadIdx.x;
        c += __syncthreads_count(x < hi && f(x));
    }
    if (threadIdx.x == 0) blk[blockIdx.x] = c;
}
__device__ __forceinline__ i64 gang_total(const i64* blk) {
    i64 t = 0;
    for (unsigned b = 0; b < gridDim.x; b++) t += blk[b];
    return t;
}
template <class F, class E>
__device__ __forceinline__ void gang_emit(i64 k, F f, E e, const i64* blk, int* wcnt) {
    i64 lo, hi, at = 0;
    gang_range(k, lo, hi);
    for (unsigned b = 0; b < blockIdx.x; b++) at += blk[b];
    const int l = lane_id(), w = threadIdx.x >> 5;
    for (i64 x0 = lo; x0 < hi; x0 += LS_THREADS) {
        const i64 x = x0 + threadIdx.x;
        const bool on = x < hi && f(x);
        const unsigned m = __ballot_sync(FULL, on);
        if (l == 0) wcnt[w] = __popc(m);
        __syncthreads();
        int before = 0, all = 0;
        for (int q = 0; q < LS_WARPS; q++) {
            before += q < w ? wcnt[q] : 0;
            all += wcnt[q];
        }
        if (on) e(x, at + before + __popc(m & lanemask_lt()));
        at += all;
        __syncthreads();
    }
}

// ---- sums over a vertex's edges ------------------------------------------------
// For every class range the canonical association of the class kernels: a
// thread (degree <= 32, canon_tree) from `thr` vertices a warp on (a group
// issues three times a thread's instructions a vertex, a thread's chain is the
// longer one), 8- or 16-lane groups below that, a warp above.  start(i, b, e) -> the row's terms
// (b == e: none; i < 0: no vertex); done(i, row, sum) by one lane.
template <class V, int G, class Start, class Done>
__device__ __forceinline__ void vsum_grp(const i32* list, i64 lo, i64 hi, i64 first, i64 nw, Start start, Done done) {
    constexpr int NG = 32 / G;
    const int l = lane_id(), r = l & (G - 1), grp = l / G;
    for (i64 base = lo + first * NG; base < hi; base += nw * NG) {
        const i64 x = base + grp;
        const i32 i = x < hi ? list[x] : -1;
        i64 b = 0, e = 0;
        const auto row = start(i, b, e);
        const V v = group_row_sum<G, V>(b, e, r, row);
        if (r == 0 && i >= 0) done(i, row, v);
    }
}
template <class V, int H, class Start, class Done>
__device__ __forceinline__ void vsum_thr(const i32* list, i64 lo, i64 hi, i64 first, i64 nw, Start start, Done done) {
    for (i64 x = lo + first * 32 + lane_id(); x < hi; x += nw * 32) {
        const i32 i = list[x];
        i64 b = 0, e = 0;
        const auto row = start(i, b, e);
        const V v = thread_vsum<H, V>(b, e, [&](i64 j) -> V { return row.term(j); });
        done(i, row, v);
    }
}
template <class V, class Start, class Done>
__device__ __forceinline__ void vsum_step(const i32* cls, const i64* off, int thr, Start start, Done done) {
    const i64 nw = gang_warps();
    const i64 o0 = off[0], o2 = off[2], o3 = off[3], o7 = off[7];
    i64 rot = 0;
    // long rows first: they are what the step ends with
    vsum_grp<V, 32>(cls, o3, o7, gang_first(rot), nw, start, done);
    rot += o7 - o3;
    if (o3 - o2 > thr * nw) {
        vsum_thr<V, 16>(cls, o2, o3, gang_first(rot), nw, start, done);
        rot += (o3 - o2 + 31) >> 5;
    } else {
        vsum_grp<V, 16>(cls, o2, o3, gang_first(rot), nw, start, done);
        rot += (o3 - o2 + 1) >> 1;
    }
    if (o2 - o0 > 16 * nw) vsum_thr<V, 8>(cls, o0, o2, gang_first(rot), nw, start, done);
    else vsum_grp<V, 8>(cls, o0, o2, gang_first(rot), nw, start, done);
}

// Inclusive scan of f over [0, k), k <= 32,768, in det_scan's association
// (groups of 32 by Kogge-Stone, then the group totals the same way).  Step 1
// scans the groups; after a gang_sync, scan_offsets gives every block the
// scanned totals in shared memory (1,024 values) and x's prefix is
// scan_at(x): offset of its group plus its value in `out`.
template <class V, class F>
__device__ __forceinline__ void scan_groups(i64 k, F f, V* out, V* tot) {
    const int l = lane_id();
    for (i64 gi = gang_warp(); gi * 32 < k; gi += gang_warps()) {
        const i64 x = gi * 32 + l;
        V v = x < k ? f(x) : V(0);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const V t = __shfl_up_sync(FULL, v, d);
            if (l >= d) v = v + t;
        }
        if (x < k) out[x] = v;
        if (l == 31) tot[gi] = v;
    }
}
template <class V>
__device__ __forceinline__ void scan_offsets(i64 k, const V* tot, V* S /* 1024 */, V* S2 /* 32 */) {
    const int l = lane_id(), w = threadIdx.x >> 5;
    const i64 groups = (k + 31) >> 5;
    for (int gi = w; gi < 32; gi += LS_WARPS) {
        const i64 x = gi * 32 + l;
        V v = x < groups ? tot[x] : V(0);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const V t = __shfl_up_sync(FULL, v, d);
            if (l >= d) v = v + t;
        }
        S[x] = v;
        if (l == 31) S2[gi] = v;
    }
    __syncthreads();
    if (w == 0) {
        V v = S2[l];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const V t = __shfl_up_sync(FULL, v, d);
            if (l >= d) v = v + t;
        }
        S2[l] = v;
    }
    __syncthreads();
    for (int x = 32 + threadIdx.x; x < 1024; x += LS_THREADS) S[x] = S2[(x >> 5) - 1] + S[x];
    __syncthreads();
}
template <class V>
__device__ __forceinline__ V scan_at(i64 x, const V* out, const V* S) {
    const i64 gi = x >> 5;
    return gi >= 1 ? S[gi - 1] + out[x] : out[x];
}

}  // namespace pggc
