// lm_small_f32.cu -- one-launch local moves of graphs with FP32 weights (a
// file per weight type: the kernel takes nvcc most of a minute).
#include "lm_cluster.cuh"

namespace pggc {

template bool local_move_small<float>(Context&, const Graph<float>&, const Ordering&, i32*, ClusterState<double>&, bool, bool,
                                    i32*, bool, bool, int, MoveStats*, bool);

}  // namespace pggc
