// k_cluster_solve for clusters of 8 CTAs (one file per size: they compile side by side).
#include "cluster_solve.cuh"

namespace hpr {
template const void *cluster_kernel<8>(bool);
template cudaError_t cluster_launch<8>(bool, const cudaLaunchConfig_t &, const ClusterArgs &);
}  // namespace hpr
