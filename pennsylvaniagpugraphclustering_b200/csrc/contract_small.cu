// contract_small.cu -- build_coarse_graph of a small graph in one launch.
//
// The general contraction (contract.cu) is about 25 launches and two host
// round trips, 120-140 us however small the graph.  For the graphs that
// lm_cluster.cuh moves, one cluster does all of it, and the products the next
// level starts with: the degree ordering, the class lists and the row sums
// (12 launches and two round trips of their own).
//
// Up to CS_MATRIX_NC coarse vertices the edges are added into a dense
// nc x nc matrix in L2 (values and presence bytes): every thread has edges
// whatever the clusters' sizes, and a row's scan is its sorted order.  Above
// that the members of each coarse vertex are listed and a warp merges a row
// in a shared-memory hash table and ranks its entries; rows of more than
// CS_WARP_BOUND member edges take a block with a table indexed by coarse id,
// 16,384 ids at a time, written in id order.  Sums are exact, rows sorted by
// column: the output equals the general path's.
#include "kernels.cuh"
#include "gang.cuh"
#include "lm_small.cuh"

namespace pggc {

constexpr i64 CS_MATRIX_NC = 1024;
constexpr int CS_WARP_BOUND = 256;  // member edges of a warp's row (512 table slots)
constexpr int CS_DENSE = 16384;     // coarse ids of one pass of a block's table
// Where the one launch is the faster way.  Its lists are made for graphs of even
// degree: a giant cluster of a skewed graph is one block's, a hub's row eight
// lanes'.  One launch / the general path, us:
//   matrix: R-MAT 2,048 vertices 153 / 183; DC-SBM 10,000 (195 K edges, rows up
//   to 1,557) 161 / 237; star of 14,000 655 / 245 (eight lanes), hence the limit
//   lists, degrees up to 64: mean degree 6, 47 K edges 121 / 182, 140 K 196 / 219;
//   mean degree 15, 85 K edges 147 / 187 (FP32 175 / 172), 227 K 234 / 198;
//   mean degree 30, 108 K edges 149 / 172 (FP32 210 / 176)
//   lists, skewed: R-MAT 4,096 355 / 219, 16,384 688 / 299; DC-SBM 10,000 557 / 235
// A level of a run starts on the coarse graph next and would make its ordering,
// class lists and row sums then (80 us, part of the one launch): any size that
// lm_small.cuh allows and degrees up to 1,024 (whole runs with 64 / 4,096 there:
// R-MAT 8,192 3,490 / 3,880 us, 16,384 3,360 / 3,640, planted partition of
// 16,000 1,265 / 1,240, DC-SBM 10,000 2,450 / 2,350; a batch of 46 planted
// partitions 1.5 % slower with 64).
constexpr i64 CS_MATRIX_DEG = 8192;
constexpr i64 CS_LIST_DEG = 64, CS_LIST_NNZ = 81920;
constexpr i64 CS_LIST_NNZ_SHORT = 147456;  // mean degree of up to 8
constexpr i64 CS_LIST_DEG_RUN = 1024;
constexpr i64 CS_WIDE_ROW = 128;    // fine rows that the matrix takes by a warp, not by eight lanes

__device__ __forceinline__ void csum_add(i64* a, i64 x) {
    if (__isShared(a)) shared_add(a, x);
    else ::atomicAdd((unsigned long long*)a, (unsigned long long)x);
}
__device__ __forceinline__ void csum_add(double* a, double x) { ::atomicAdd(a, x); }

template <class W>
struct CSmallArgs {
    using V = typename Traits<W>::V;
    DGraph<W> g;
    const i32* vcmap;
    i64 nc;
    i64* rowptr;  // outputs
    i32* col;
    W* w;
    V* rsum;
    WeightUnits* units;  // of the coarse weights (FP32)
    const WeightUnits* fine_units;
    i32* order1;
    i32* cls;
    i64* cls_off;
    i64* res;     // [8] nnz, off_large, off_large2, max degree, error word
    i32* cnt;     // [2 * nc] members, member edges; then scatter cursors
    i32* cstart;  // [nc + 1]
    i32* P;       // [nc + 1] first slot of a row's entries in okey / oval
    i32* members;
    i32* ucount;
    i32* biglist;
    V* oval;      // [nnz], or the matrix [nc * nc]
    i32* okey;
    u32* pres;    // presence bytes of the matrix
    i64* blk;     // [4 * 32]
    u32* ccnt;    // [2 * NCLS + 3] class counts, class cursors, max degree, big rows
    const int* err;
};

// rows with few member edges: hash table, compact, rank
template <class W>
__device__ __forceinline__ void row_warp(const CSmallArgs<W>& a, i32 c, unsigned char* smem, const Units<W>& un) {
    using V = typename Traits<W>::V;
    const int l = lane_id(), r = l & 7, grp = l >> 3;
    const i32 m0 = a.cstart[c], m1 = a.cstart[c + 1], q0 = a.P[c];
    const u32 bound = (u32)(a.P[c + 1] - q0);
    const u32 T = next_pow2_u32(2 * (bound > 1 ? bound : 1));
    V* vals = (V*)smem;
    i32* keys = (i32*)(smem + sizeof(V) * 2 * CS_WARP_BOUND);
    i32* comp = keys + 2 * CS_WARP_BOUND;  // compacted keys
    for (u32 s = l; s < T; s += 32) {
        keys[s] = -1;
        vals[s] = V(0);
    }
    __syncwarp();
    for (i32 m = m0 + grp; m < m1; m += 4) {
        const i32 u = a.members[m];
        const i64 b = a.g.rowptr[u], e = a.g.rowptr[u + 1];
        for (i64 j = b + r; j < e; j += 8) {
            const i32 cv = a.vcmap[a.g.col[j]];
            if (cv == c) continue;
            const W x = a.g.wgt(j);
            u32 s = xorshift32((u32)cv) & (T - 1);
            for (u32 p = 0; p < T; p++) {  // at most `bound` < T distinct keys
                const i32 old = atomicCAS(&keys[s], -1, cv);
                if (old == -1 || old == cv) {
                    if (un.on) shared_add((i64*)&vals[s], un.of(x));
                    else csum_add(&vals[s], V(x));
                    break;
                }
                s = (s + 1) & (T - 1);
            }
        }
    }
    __syncwarp();
    u32 u = 0;
    for (u32 s0 = 0; s0 < T; s0 += 32) {
        const u32 s = s0 + l;
        const bool occ = s < T && keys[s] != -1;
        const unsigned m = __ballot_sync(FULL, occ);
        if (occ) comp[u + __popc(m & lanemask_lt())] = keys[s];
        u += __popc(m);
    }
    __syncwarp();
    for (u32 s = l; s < T; s += 32) {
        const i32 k = keys[s];
        if (k == -1) continue;
        u32 rank = 0;
        for (u32 t = 0; t < u; t++) rank += comp[t] < k ? 1 : 0;
        a.okey[q0 + rank] = k;
        a.oval[q0 + rank] = un.sum(vals[s]);
    }
    if (l == 0) a.ucount[c] = (i32)u;
    __syncwarp();
}

// rows with many member edges: dense table, a range of coarse ids at a time
template <class W>
__device__ __forceinline__ void row_block(const CSmallArgs<W>& a, i32 c, unsigned char* smem, i64* red, const Units<W>& un) {
    using V = typename Traits<W>::V;
    const int l = lane_id(), r = l & 7;
    V* vals = (V*)smem;
    u32* bits = (u32*)(smem + sizeof(V) * CS_DENSE);
    const i32 m0 = a.cstart[c], m1 = a.cstart[c + 1];
    i64 at = a.P[c];
    const i64 first = at;
    for (i64 c0 = 0; c0 < a.nc; c0 += CS_DENSE) {
        const int span = (int)min((i64)CS_DENSE, a.nc - c0);
        for (int s = threadIdx.x; s < span; s += LS_THREADS) vals[s] = V(0);
        for (int s = threadIdx.x; s < CS_DENSE / 32; s += LS_THREADS) bits[s] = 0u;
        __syncthreads();
        for (i32 m = m0 + (int)(threadIdx.x >> 3); m < m1; m += LS_THREADS / 8) {
            const i32 u = a.members[m];
            const i64 b = a.g.rowptr[u], e = a.g.rowptr[u + 1];
            for (i64 j = b + r; j < e; j += 8) {
                const i32 cv = a.vcmap[a.g.col[j]];
                if (cv == c || cv < c0 || cv >= c0 + span) continue;
                if (un.on) shared_add((i64*)&vals[cv - c0], un.of(a.g.wgt(j)));
                else csum_add(&vals[cv - c0], V(a.g.wgt(j)));
                atomicOr(&bits[(cv - c0) >> 5], 1u << ((cv - c0) & 31));
            }
        }
        __syncthreads();
        static_assert(CS_DENSE == 32 * LS_THREADS, "a presence word per thread");
        u32 word = bits[threadIdx.x];
        i64 total;
        i64 pos = at + block_excl_scan_i64<LS_THREADS>(__popc(word), red, &total);
        while (word) {
            const int q = (int)threadIdx.x * 32 + __ffs(word) - 1;
            word &= word - 1;
            a.okey[pos] = (i32)(c0 + q);
            a.oval[pos] = un.sum(vals[q]);
            pos++;
        }
        at += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) a.ucount[c] = (i32)(at - first);
}

template <class W>
__global__ void __launch_bounds__(LS_THREADS, 1) k_contract_small(CSmallArgs<W> a) {
    using V = typename Traits<W>::V;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ i64 red[LS_WARPS + 1];
    __shared__ int hist[NCLS];
    __shared__ int wc[2][LS_WARPS];
    const DGraph<W>& g = a.g;
    const i64 n = g.n, nc = a.nc;
    const int l = lane_id(), w = threadIdx.x >> 5, r8 = l & 7, grp = l >> 3;
    const i64 t0 = (i64)blockIdx.x * LS_THREADS + threadIdx.x, nt = (i64)gridDim.x * LS_THREADS;
    const i64 nw = gang_warps();
    const bool matrix = nc <= CS_MATRIX_NC;
    unsigned char* pres = (unsigned char*)a.pres;

    if (t0 < 2 * NCLS + 3) a.ccnt[t0] = 0;
    if (std::is_same<W, float>::value && t0 == 0) *a.units = WeightUnits{0, 0, 0.0};
    UnitScan<W> us;
    i64 lo, hi;
    gang_range(nc, lo, hi);
    if (matrix) {
        for (i64 x = t0; x < nc * nc; x += nt) a.oval[x] = V(0);
        for (i64 x = t0; x < (nc * nc + 3) / 4; x += nt) a.pres[x] = 0u;
        gang_sync();
        for (i64 base = (i64)gang_warp() * 4; base < n; base += nw * 4) {
            const i64 i = base + grp;
            i64 b = 0, e = 0;
            i32 self = 0;
            if (i < n) {
                b = g.rowptr[i];
                e = g.rowptr[i + 1];
                self = a.vcmap[i];
            }
            auto edge = [&](i64 j, i32 c) {
                const i32 cv = a.vcmap[g.col[j]];
                const W x = g.wgt(j);
                if (cv != c) {
                    csum_add(&a.oval[(i64)c * nc + cv], V(x));
                    pres[(i64)c * nc + cv] = 1;
                }
            };
            const bool wide = e - b > CS_WIDE_ROW;
            if (!wide) {
#pragma unroll 4
                for (i64 j = b + r8; j < e; j += 8) edge(j, self);
            }
            for (unsigned m = __ballot_sync(FULL, wide && r8 == 0); m; m &= m - 1) {
                const int from = __ffs(m) - 1;
                const i64 wb = __shfl_sync(FULL, b, from), we = __shfl_sync(FULL, e, from);
                const i32 wc = __shfl_sync(FULL, self, from);
#pragma unroll 4
                for (i64 j = wb + l; j < we; j += 32) edge(j, wc);
            }
        }
        gang_sync();
        for (i64 c = gang_warp(); c < nc; c += nw) {
            int u = 0;
            for (i64 s = l; s < nc; s += 32) u += pres[c * nc + s];
            u = __reduce_add_sync(FULL, u);
            if (l == 0) a.ucount[c] = u;
        }
    } else {
        i32 *mem = a.cnt, *bnd = a.cnt + nc;
        for (i64 x = t0; x < 2 * nc; x += nt) a.cnt[x] = 0;
        gang_sync();
        for (i64 i = t0; i < n; i += nt) {
            const i32 c = a.vcmap[i];
            atomicAdd(&mem[c], 1);
            atomicAdd(&bnd[c], (i32)(g.rowptr[i + 1] - g.rowptr[i]));
        }
        gang_sync();
        // member and entry offsets
        i64 s0 = 0, s1 = 0;
        for (i64 x = lo + threadIdx.x; x < hi; x += LS_THREADS) {
            s0 += mem[x];
            s1 += bnd[x];
        }
        i64 tot0, tot1;
        block_excl_scan_i64<LS_THREADS>(s0, red, &tot0);
        block_excl_scan_i64<LS_THREADS>(s1, red, &tot1);
        if (threadIdx.x == 0) {
            a.blk[blockIdx.x] = tot0;
            a.blk[32 + blockIdx.x] = tot1;
        }
        gang_sync();
        i64 at0 = 0, at1 = 0;
        for (unsigned b = 0; b < blockIdx.x; b++) {
            at0 += a.blk[b];
            at1 += a.blk[32 + b];
        }
        for (i64 x0 = lo; x0 < hi; x0 += LS_THREADS) {
            const i64 x = x0 + threadIdx.x;
            const i32 v0 = x < hi ? mem[x] : 0, v1 = x < hi ? bnd[x] : 0;
            const i64 e0 = block_excl_scan_i64<LS_THREADS>(v0, red, &tot0);
            const i64 e1 = block_excl_scan_i64<LS_THREADS>(v1, red, &tot1);
            if (x < hi) {
                a.cstart[x] = (i32)(at0 + e0);
                a.P[x] = (i32)(at1 + e1);
                mem[x] = (i32)(at0 + e0);  // scatter cursor
                if (v1 > CS_WARP_BOUND) a.biglist[atomicAdd(&a.ccnt[2 * NCLS + 1], 1u)] = (i32)x;
            }
            at0 += tot0;
            at1 += tot1;
        }
        if (t0 == 0) {
            a.cstart[nc] = (i32)n;
            a.P[nc] = (i32)g.nnz;
        }
        gang_sync();
        for (i64 i = t0; i < n; i += nt) a.members[atomicAdd(&mem[a.vcmap[i]], 1)] = (i32)i;
        gang_sync();
        const u32 nbig = a.ccnt[2 * NCLS + 1];
        const Units<W> un = Units<W>::make(a.fine_units, a.fine_units ? a.fine_units->total : 0.0);
        for (u32 x = blockIdx.x; x < nbig; x += gridDim.x) row_block(a, a.biglist[x], smem, red, un);
        __syncthreads();
        for (i64 c = gang_warp(); c < nc; c += nw)
            if (a.P[c + 1] - a.P[c] <= CS_WARP_BOUND) row_warp(a, (i32)c, smem + w * LS_WARP_BYTES, un);
    }
    gang_sync();
    // degrees: row offsets, buckets of order1, classes
    if (threadIdx.x < NCLS) hist[threadIdx.x] = 0;
    __syncthreads();
    {
        i64 sum = 0, c0 = 0, c1 = 0;
        i32 mx = 0;
        for (i64 x0 = lo; x0 < hi; x0 += LS_THREADS) {
            const i64 x = x0 + threadIdx.x;
            const i32 d = x < hi ? a.ucount[x] : -1;
            const int k = d >= 0 ? deg_class(d) : -1;
            sum += d > 0 ? d : 0;
            mx = max(mx, d);
            c0 += __syncthreads_count(d >= 0 && d < LARGE_CUTOFF);
            c1 += __syncthreads_count(d >= LARGE_CUTOFF && d < MASSIVE_CUTOFF);
            for (int q = 0; q < NCLS; q++) {
                const unsigned m = __ballot_sync(FULL, k == q);
                if (l == 0 && m) atomicAdd(&hist[q], __popc(m));
            }
        }
        mx = __reduce_max_sync(FULL, mx);
        if (l == 0 && mx > 0) atomicMax(&a.ccnt[2 * NCLS], (u32)mx);
        i64 tot;
        block_excl_scan_i64<LS_THREADS>(sum, red, &tot);
        if (threadIdx.x == 0) {
            a.blk[blockIdx.x] = tot;
            a.blk[32 + blockIdx.x] = c0;
            a.blk[64 + blockIdx.x] = c1;
        }
        if (threadIdx.x < NCLS && hist[threadIdx.x]) atomicAdd(&a.ccnt[threadIdx.x], (u32)hist[threadIdx.x]);
    }
    gang_sync();
    {
        i64 at = 0, p0 = 0, p1 = 0, tot = 0, tot0 = 0, tot1 = 0;
        for (unsigned b = 0; b < gridDim.x; b++) {
            if (b == blockIdx.x) {
                at = tot;
                p0 = tot0;
                p1 = tot1;
            }
            tot += a.blk[b];
            tot0 += a.blk[32 + b];
            tot1 += a.blk[64 + b];
        }
        i64 p2 = tot0 + tot1 + (lo - p0 - p1);
        p1 += tot0;
        i64 off[NCLS + 1];
        off[0] = 0;
#pragma unroll
        for (int q = 0; q < NCLS; q++) off[q + 1] = off[q] + a.ccnt[q];
        if (t0 == 0) {
#pragma unroll
            for (int q = 0; q <= NCLS; q++) a.cls_off[q] = off[q];
            a.rowptr[nc] = tot;
            a.res[0] = tot;
            a.res[1] = tot0;
            a.res[2] = tot0 + tot1;
            a.res[3] = a.ccnt[2 * NCLS];
            a.res[4] = *(const volatile int*)a.err;
        }
        for (i64 x0 = lo; x0 < hi; x0 += LS_THREADS) {
            const i64 x = x0 + threadIdx.x;
            const i32 d = x < hi ? a.ucount[x] : -1;
            i64 tile;
            const i64 e = block_excl_scan_i64<LS_THREADS>(d > 0 ? d : 0, red, &tile);
            if (d >= 0) a.rowptr[x] = at + e;
            at += tile;
            const bool b0 = d >= 0 && d < LARGE_CUTOFF, b1 = d >= LARGE_CUTOFF && d < MASSIVE_CUTOFF;
            const unsigned m0 = __ballot_sync(FULL, b0), m1 = __ballot_sync(FULL, b1);
            const unsigned m2 = __ballot_sync(FULL, d >= MASSIVE_CUTOFF);
            if (l == 0) {
                wc[0][w] = __popc(m0);
                wc[1][w] = __popc(m1);
            }
            __syncthreads();
            int q0 = 0, q1 = 0, a0 = 0, a1 = 0;
            for (int q = 0; q < LS_WARPS; q++) {
                q0 += q < w ? wc[0][q] : 0;
                q1 += q < w ? wc[1][q] : 0;
                a0 += wc[0][q];
                a1 += wc[1][q];
            }
            // before this warp in the tile: 32 w vertices (all in range where it has any)
            if (b0) a.order1[p0 + q0 + __popc(m0 & lanemask_lt())] = (i32)x;
            else if (b1) a.order1[p1 + q1 + __popc(m1 & lanemask_lt())] = (i32)x;
            else if (d >= 0) a.order1[p2 + (32 * w - q0 - q1) + __popc(m2 & lanemask_lt())] = (i32)x;
            p0 += a0;
            p1 += a1;
            p2 += min((i64)LS_THREADS, hi - x0) - a0 - a1;
            const int k = d >= 0 ? deg_class(d) : -1;
#pragma unroll
            for (int q = 0; q < NCLS; q++) {
                const unsigned m = __ballot_sync(FULL, k == q);
                if (!m) continue;
                u32 base = 0;
                if (l == 0) base = atomicAdd(&a.ccnt[NCLS + q], (u32)__popc(m));
                base = __shfl_sync(FULL, base, 0);
                if (k == q) a.cls[off[q] + base + __popc(m & lanemask_lt())] = (i32)x;
            }
            __syncthreads();
        }
    }
    gang_sync();
    // rows to their places, and their sums
    for (i64 c = gang_warp(); c < nc; c += nw) {
        i64 at = a.rowptr[c];
        V sum = V(0);
        if (matrix) {
            const i64 row = c * nc;
            for (i64 s0 = 0; s0 < nc; s0 += 32) {
                const i64 s = s0 + l;
                const bool on = s < nc && pres[row + s];
                const unsigned m = __ballot_sync(FULL, on);
                if (on) {
                    const i64 q = at + __popc(m & lanemask_lt());
                    const W x = (W)a.oval[row + s];
                    a.col[q] = (i32)s;
                    a.w[q] = x;
                    us.see(x);
                    sum = sum + V(x);
                }
                at += __popc(m);
            }
        } else {
            const i64 q0 = a.P[c], u = a.ucount[c];
            for (i64 k = l; k < u; k += 32) {
                const W x = (W)a.oval[q0 + k];
                a.col[at + k] = a.okey[q0 + k];
                a.w[at + k] = x;
                us.see(x);
                sum = sum + V(x);
            }
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) sum = sum + __shfl_xor_sync(FULL, sum, d);
        if (l == 0) a.rsum[c] = sum;
    }
    us.flush(a.units);
}

template <class W>
std::unique_ptr<Graph<W>> build_coarse_small(Context& ctx, const Graph<W>& g, const i32* vcmap, i64 nc,
                                             bool next_level) {
    using V = typename Traits<W>::V;
    const i64 n = g.n, nnz = g.nnz;
    if (nc == 0 || n == 0 || ctx.probe_cap != 0) return nullptr;
    const bool matrix = nc <= CS_MATRIX_NC;
    {
        GraphCache& c = *g.cache;
        std::lock_guard<std::mutex> lk(c.mu);
        const i64 deg = c.ord_ok ? c.ord.max_deg : -1;  // -1: not known
        const bool fits = matrix       ? deg <= CS_MATRIX_DEG
                          : next_level ? deg >= 0 && deg <= CS_LIST_DEG_RUN
                                       : deg >= 0 && deg <= CS_LIST_DEG &&
                                             nnz <= (nnz <= 8 * n ? CS_LIST_NNZ_SHORT : CS_LIST_NNZ);
        if (!fits)
            return nullptr;
    }
    const int blocks = gang_blocks(ctx, k_contract_small<W>, small_cluster_blocks(n, nnz));
    if (blocks == 0) return nullptr;
    ProfScope ps(ctx, "contract_small");
    const i64 room = std::max<i64>(std::min<i64>(nnz, nc * (nc - 1)), 1);
    auto cg = std::make_unique<Graph<W>>();
    cg->n = nc;
    cg->uniform = false;
    cg->rowptr = DBuf<i64>(ctx, nc + 1);
    cg->col = DBuf<i32>(ctx, room);
    cg->w = DBuf<W>(ctx, room);
    cg->rsum = DBuf<V>(ctx, nc);
    GraphCache& gc = *cg->cache;
    gc.ord.order1 = DBuf<i32>(ctx, nc);
    gc.cls_list = DBuf<i32>(ctx, nc);
    gc.cls_off = DBuf<i64>(ctx, NCLS + 1);
    CSmallArgs<W> a{};
    a.g = g.view();
    a.vcmap = vcmap;
    a.nc = nc;
    a.rowptr = cg->rowptr.p;
    a.col = cg->col.p;
    a.w = cg->w.p;
    a.rsum = cg->rsum.p;
    if (std::is_same<W, float>::value) {
        cg->units = DBuf<WeightUnits>(ctx, 1);
        a.units = cg->units.p;
        row_sums<W>(ctx, g);
        a.fine_units = g.units.p;
    }
    a.order1 = gc.ord.order1.p;
    a.cls = gc.cls_list.p;
    a.cls_off = gc.cls_off.p;
    a.oval = ctx.ws_get<V>(CSS_OVAL, matrix ? nc * nc : nnz);
    a.ucount = ctx.ws_get<i32>(CSS_UCOUNT, nc);
    i64* fixed = ctx.ws_get<i64>(CSS_FIXED, 8 + 4 * 32 + NCLS + 2);
    a.res = fixed;
    a.blk = fixed + 8;
    a.ccnt = (u32*)(fixed + 8 + 4 * 32);
    if (matrix) {
        a.pres = ctx.ws_get<u32>(CSS_PRES, (nc * nc + 3) / 4);
    } else {
        a.okey = ctx.ws_get<i32>(CSS_OKEY, nnz);
        a.cnt = ctx.ws_get<i32>(CSS_CNT, 2 * nc);
        a.cstart = ctx.ws_get<i32>(CSS_CSTART, nc + 1);
        a.P = ctx.ws_get<i32>(CSS_P, nc + 1);
        a.members = ctx.ws_get<i32>(CSS_MEMBERS, n);
        a.biglist = ctx.ws_get<i32>(CSS_BIG, nc);
    }
    a.err = ctx.d_err;
    launch_gang(ctx, k_contract_small<W>, a, blocks);
    const i64* h = (const i64*)ctx.readback(a.res, 5 * sizeof(i64));
    ctx.raise_device_error((int)h[4]);
    cg->nnz = h[0];
    // algorithmic bytes, as the general path counts them
    ctx.prof_add_bytes("contract", (double)nnz * (12.0 + sizeof(W) + (g.uniform ? 0.0 : sizeof(W))) + (double)n * 12.0 +
                                       (double)cg->nnz * (4.0 + sizeof(W)) + (double)(nc + 1) * 8.0);
    Ordering& o = gc.ord;
    o.n = nc;
    o.off_large = h[1];
    o.off_large2 = h[2];
    o.max_deg = h[3];
    // the list of vertices above HUGE_DEG edges is left to the general
    // orderings, as is the second permutation, which no level needs
    gc.ord_ok = o.max_deg <= HUGE_DEG;
    gc.cls_ok = true;
    return cg;
}

template std::unique_ptr<Graph<i32>> build_coarse_small<i32>(Context&, const Graph<i32>&, const i32*, i64,
                                                                    bool);
template std::unique_ptr<Graph<float>> build_coarse_small<float>(Context&, const Graph<float>&, const i32*, i64, bool);

}  // namespace pggc
