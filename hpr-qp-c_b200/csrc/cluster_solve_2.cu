// k_cluster_solve for clusters of 2 CTAs (one file per size: they compile side by side).
#include "cluster_solve.cuh"

namespace hpr {
template const void *cluster_kernel<2>(bool);
template cudaError_t cluster_launch<2>(bool, const cudaLaunchConfig_t &, const ClusterArgs &);
}  // namespace hpr
