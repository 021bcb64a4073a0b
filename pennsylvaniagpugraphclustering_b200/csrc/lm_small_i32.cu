// lm_small_i32.cu -- one-launch local moves of graphs with integer weights (a
// file per weight type: the kernel takes nvcc most of a minute).
#include "lm_cluster.cuh"

namespace pggc {

template bool local_move_small<i32>(Context&, const Graph<i32>&, const Ordering&, i32*, ClusterState<i64>&, bool, bool,
                                    i32*, bool, bool, int, MoveStats*, bool);

}  // namespace pggc
