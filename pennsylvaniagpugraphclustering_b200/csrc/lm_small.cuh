// lm_small.cuh -- local moves of small graphs in one launch (lm_cluster.cuh).
#pragma once
#include "filter.cuh"
#include "gang.cuh"
#include "kernels.cuh"

namespace pggc {

// Above these a launch per step over the whole GPU is the faster way: the work
// on the cluster's 16 SMs grows with the edges while the launches do not.
// Local moves have the lower limits (their steps cover the GPU in 7 launches a
// sweep, contraction and refinement take 25 to 30), on the edges and on the
// edges plus what a vertex costs beside them, about four.  Six sweeps here and
// with a launch per step, us (planted partitions / power-law degrees):
//   mean degree 4:    49 K edges 371, 421 / 496, 499; 127 K 667, 468 / 938, 520
//   mean degree 8:    68 K edges 377, 412 / 511, 516; 155 K 559, 455 / 941, 532
//   mean degree 15:   57 K edges 329, 441; 104 K 447, 444 / 598, 599; 227 K 704, 464
//   mean degree 30:   81 K edges 370, 459 / 497, 603; 144 K 531, 469 / 805, 691
// One run at a time that would be 115 K edges and vertices; in a batch a launch
// and no round trip a sweep is worth more (32 graphs of 6,000 to 12,000 vertices
// of 14 edges on 4 streams: 21.9 ms with that limit, 21.0 ms with these).
// Long rows go further, a warp or block has enough to do in each:
//   mean degree 55:  133 K edges 459, 451;  75: 158 K 362, 386 (FP32 weights 520,
//   512);  94: 170 K 311, 369 (446, 490);  136: 130 K 189, 307 (335, 472)
constexpr i64 LS_MAX_N = 32768;
constexpr i64 LS_MAX_NNZ = 262144;
constexpr i64 LS_MOVE_NNZ = 131072;
constexpr i64 LS_MOVE_SIZE = 163840;      // edges plus four a vertex
constexpr i64 LS_MOVE_NNZ_LONG = 196608;  // edges, at a mean degree of 64 or more
constexpr i64 LS_MAX_LABELS = 131072;

constexpr int LS_MAX_SWEEPS = 6;

template <class W>
struct SmallArgs {
    using V = typename Traits<W>::V;
    DGraph<W> g;
    const i32* cls;       // vertices grouped by degree class
    const i64* off;       // [NCLS + 1]
    const i32* order1;
    const V* rsum;
    const WeightUnits* units;
    i32 *part, *dest;
    float* gain;
    unsigned char *keep, *flags, *has;
    V *pvals, *pv_best, *td;
    i32* best_part;
    V* td_best;
    i32* constraint;
    i32 *newl, *avail, *newid;
    V* td2;
    V* partial;                // chunk sums: of the own-cluster weights, then
    i64 sq_at;                 // from here of the squared volumes
    i64* blk;                  // [3 * 32] per-block counts
    unsigned long long* cnt;   // [2 * LS_MAX_SWEEPS] moves, NEW_PART moves of each sweep
    LMScalars<V>* sc;          // results
    int* err;
    i64 cap;
    i64 label_count;
    V uncut;
    double obj, lambda;
    float pm, inv_load;
    int initial, sa, reuse, sweep_limit, keys32;
    int strict;           // one sweep of the strict variant (see below)
    unsigned long long* prof;  // algorithmic-byte counter (profiling only)
    FiltArgs<W> filt;          // FILT only; prev_stamp is that of the first sweep
    i32* moved_at;
    i32* csize;
};

// The same steps launched one by one over the whole GPU, for graphs above the
// one-launch size (lm_steps.cu).
template <class W>
void step_init(Context& ctx, const SmallArgs<W>& a);  // current state <- best state
template <class W>
void step_select(Context& ctx, const SelArgs<W>& s, const i32* cls, const i64* off, i64 count, bool constrained);
template <class W>
void step_afterburner(Context& ctx, const SmallArgs<W>& a);
template <class W>
void step_moves(Context& ctx, const SmallArgs<W>& a, bool mark, i32 stamp);
// own-cluster weights (all vertices, or the flagged ones) and the chunk sums of
// the squared volumes, then the chunk sums of the weights
template <class W>
void step_own(Context& ctx, const SmallArgs<W>& a, bool all);
template <class W>
void step_sums(Context& ctx, const SmallArgs<W>& a);
// the sums' totals; after a sweep the objective and the copy of an improved
// state (at most label_bound labels), before the first the starting total
template <class W>
void step_objective(Context& ctx, const SmallArgs<W>& a, bool sweep, i64 label_bound);

// The algorithmic bytes of a step that is about to run, added to *prof (NULL:
// nothing is done): a count of its own, so that the steps carry none.
template <class W>
void step_select_bytes(Context& ctx, const SelArgs<W>& s, const i32* cls, i64 count, unsigned long long* prof);
template <class W>
void step_afterburner_bytes(Context& ctx, const SmallArgs<W>& a, unsigned long long* prof);
template <class W>
void step_own_bytes(Context& ctx, const SmallArgs<W>& a, bool all, unsigned long long* prof);

// Blocks of the cluster that should run a step of this graph, 0 when it is not small.
int small_cluster_blocks(i64 n, i64 nnz);

// local_move or local_move_strict of a small graph; false, with nothing done,
// when the general path has to run it.
template <class W>
bool local_move_small(Context& ctx, const Graph<W>& g, const Ordering& ord, i32* best_part,
                      ClusterState<typename Traits<W>::V>& best, bool is_initial, bool constrained, i32* constraint,
                      bool enable_sa, bool strict, int sweep_limit, MoveStats* stats, bool reuse_pvals);

// build_coarse_graph of a small graph, with its degree ordering, class lists
// and row sums; null, with nothing done, when the general path has to run it.
template <class W>
std::unique_ptr<Graph<W>> build_coarse_small(Context& ctx, const Graph<W>& g, const i32* vcmap, i64 nc,
                                             bool next_level);

// workspace slots of the small contraction
enum ContractSmallSlot : int {
    CSS_OVAL = 110, CSS_UCOUNT, CSS_FIXED, CSS_PRES, CSS_OKEY, CSS_CNT, CSS_CSTART, CSS_P, CSS_MEMBERS, CSS_BIG
};

// The cluster launch of `kern` with `blocks` blocks.
struct GangLaunch {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    GangLaunch(int blocks, cudaStream_t stream) {
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(LS_THREADS);
        cfg.dynamicSmemBytes = LS_TABLE_BYTES;
        cfg.stream = stream;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = blocks;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    GangLaunch(const GangLaunch&) = delete;
};

// Blocks for a cluster of `want` (8 or 16): want, 8 where the device places no
// 16 (a partition with fewer free SMs in a GPC), 0 where it places neither:
// the general path has to run (local moves take up to half as long again with
// 8 blocks as with 16 and up to 2.4 times as long with 4, see
// small_cluster_blocks; the launches of the general path 1.3 to 2 times).  The
// device is asked once per kernel.
template <class A>
inline int gang_blocks(Context& ctx, void (*kern)(A), int want) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, int> largest;
    if (want == 0) return 0;
    int most;
    {
        std::lock_guard<std::mutex> lk(mu);
        const auto key = std::make_pair((const void*)kern, ctx.device);
        auto it = largest.find(key);
        if (it == largest.end()) {
            most = 0;
            if (ctx.max_smem_optin >= LS_TABLE_BYTES) {
                set_dynamic_smem_once(kern, LS_TABLE_BYTES, ctx.device);
                PGGC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
                for (int b = 16; b >= 8 && most == 0; b >>= 1) {
                    GangLaunch g(b, ctx.stream);
                    int clusters = 0;
                    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &g.cfg) != cudaSuccess) cudaGetLastError();
                    else if (clusters > 0) most = b;
                }
            }
            it = largest.emplace(key, most).first;
        }
        most = std::min(it->second, ctx.max_cluster);
    }
    return most >= want ? want : most >= 8 ? 8 : 0;
}

// Launches `kern` as one cluster of `blocks` blocks (from gang_blocks).
template <class A>
inline void launch_gang(Context& ctx, void (*kern)(A), const A& a, int blocks) {
    GangLaunch g(blocks, ctx.stream);
    PGGC_CUDA(cudaLaunchKernelEx(&g.cfg, kern, a));
    PGGC_LAUNCH_CHECK();
}

}  // namespace pggc
