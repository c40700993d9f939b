// k_cluster_solve for clusters of 1 CTA (one file per size: they compile side by side).
#include "cluster_solve.cuh"

namespace hpr {
template const void *cluster_kernel<1>(bool);
template cudaError_t cluster_launch<1>(bool, const cudaLaunchConfig_t &, const ClusterArgs &);
}  // namespace hpr
