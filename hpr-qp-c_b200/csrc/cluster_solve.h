// Host side of k_cluster_solve (cluster_solve.cuh): its shape and launch.
#pragma once

#include "batch_device.cuh"

#include <cuda_runtime.h>

namespace hpr {

// Threads of a CTA.  One CTA with a whole instance in its shared memory has
// rows for more warps (us an iteration of n = 220 / 450 with all SMs busy:
// 8.6 / 16.1 with 256 threads, 6.9 / 13.8 with 512, 12.2 / 17.7 in
// k_batch_solve; n = 100: 4.6, 5.3, 7.9).
__host__ __device__ constexpr int cluster_threads(int C, bool resident) { return C == 1 && resident ? 512 : 256; }
constexpr int kClMaxLen = 8190;  // columns as 16-bit byte offsets, the zero entry included
// doubles of shared memory per own row of an n- and an m-vector (odd: a warp's
// rows fall on different banks)
constexpr int kClNOwn = 11, kClMOwn = 5;

struct ClusterArgs {
    BatchArgs B;
    int vw;          // virtual warps: warps of the one-CTA shape of these instances
    int smem_bytes;  // dynamic shared memory of a CTA
};

// bytes of shared memory an instance's vectors take in a CTA of a cluster:
// the gathered vectors, the own slices and the row pointers
__host__ __device__ __forceinline__ size_t cluster_vec_bytes(int n, int m, int vw, int C)
{
    const size_t big = n > m ? n : m;
    const size_t nl = (size_t)(vw / C) * ((n + vw - 1) / vw), ml = (size_t)(vw / C) * ((m + vw - 1) / vw);
    const size_t d = ((n + 2) & ~1) + ((big + 2) & ~size_t(1)) + ((m + 2) & ~1) + kClNOwn * nl + kClMOwn * ml;
    return 8 * (d + 1) + 4 * ((2 * (nl + 1) + ml + 1 + 3) & ~size_t(3));
}

// dynamic shared memory of k_cluster_solve: one CTA per SM, all there is but
// 8 KB for its static shared memory
constexpr size_t kClSmemLimit = 227 * 1024 - 8 * 1024;

// whether an instance whose one-CTA shape has vw warps can be solved by a
// cluster of C CTAs: every CTA has rows (the exchanges of a step order the
// CTAs through their rows) and the vectors fit
inline bool cluster_fits(long long n, long long m, int vw, int C)
{
    if (vw % C != 0 || n < 1 || n > kClMaxLen || m > kClMaxLen) return false;
    if (C > 1 && (m < 1 || (long long)(C - 1) * (vw / C) * ((n + vw - 1) / vw) >= n)) return false;
    return cluster_vec_bytes((int)n, (int)m, vw, C) <= kClSmemLimit;
}

// the smallest cluster that can, of the sizes the device holds (a part of a
// GPU may have no room for large ones; cap[l]: clusters of 2^l CTAs at once);
// 0: none
inline int smallest_cluster(long long n, long long m, int vw, const int cap[5])
{
    for (int l = 0; l < 5; ++l)
        if (cap[l] > 0 && cluster_fits(n, m, vw, 1 << l)) return 1 << l;
    return 0;
}

// Kernel for clusters of C CTAs; resident: every instance's matrices fit the
// CTAs' shared memory (no code for streaming them).
template <int C>
const void *cluster_kernel(bool resident);
template <int C>
cudaError_t cluster_launch(bool resident, const cudaLaunchConfig_t &cfg, const ClusterArgs &P);

}  // namespace hpr
