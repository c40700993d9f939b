// cluster_solve.h's choice of a cluster size, without a GPU: reads
// "n m warps cap0 .. cap4" a line, writes the smallest cluster.
#include "cluster_solve.h"

#include <cstdio>

int main()
{
    long long n, m;
    int vw, cap[5];
    while (scanf("%lld %lld %d %d %d %d %d %d", &n, &m, &vw, cap, cap + 1, cap + 2, cap + 3, cap + 4) == 8)
        printf("%d\n", hpr::smallest_cluster(n, m, vw, cap));
    return 0;
}
