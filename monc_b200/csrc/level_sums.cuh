// Level sums split over a cluster of blocks: each block sums a contiguous share of the level's points
// in a fixed order, and block 0 adds the shares in rank order through distributed shared memory.
// Deterministic, and a level keeps several blocks busy where one block a level left most of the GPU idle.
#pragma once

#include <cooperative_groups.h>

namespace mgpu {

constexpr int PSPLIT = 8;  // blocks of a cluster, at most

// the cluster's total of sh[q][0] over its blocks, valid in block 0 (thread 0)
template <int NV, int W>
__device__ __forceinline__ void cluster_total(double (*sh)[W], double* tot) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (cluster.block_rank() == 0 && threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) tot[q] = 0.0;
    for (int r = 0; r < (int)cluster.num_blocks(); ++r) {
      double(*rs)[W] = cluster.map_shared_rank(sh, r);
#pragma unroll
      for (int q = 0; q < NV; ++q) tot[q] += rs[q][0];
    }
  }
  cluster.sync();  // no block leaves while block 0 reads its partial sums
}

}  // namespace mgpu
