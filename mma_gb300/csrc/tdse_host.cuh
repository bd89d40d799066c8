// tdse_host.cuh -- library-internal host calls: the propagation that spreads an instance over a cluster,
// and the ground state of one grid.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/mma_tdse.h"

namespace mma {

struct ClusterPlan {
    int nc;       // CTAs per instance
    int m;        // sites per thread of the launch's widest grid
    size_t smem;  // dynamic shared memory per CTA
    int active;   // clusters resident at once; 0: the shape does not fit
};

// The cluster size for a batch of n_inst instances on grids of at most max_m 256-site rows, or false
// where the one-CTA kernel is expected to finish the batch sooner.
bool choose_cluster(int max_m, int precision, int n_inst, int sms, ClusterPlan* plan);
int launch_cluster(const ClusterPlan& p, const mma_tdse_instance* insts, int n_inst, const mma_tdse_grid* grids,
                   const mma_tdse_buffers* bufs, int max_m, int precision, void* stream);

// The ground states of a few grids by a cluster each (tdse_ground.cu).  Whether a cluster serves these grids
// (else a CTA each does), and the launch, from the tables and V that build_grids_kernel mode 3 left: false,
// and nothing launched, where it fails.
bool ground_state_fits(int n_grids, int64_t max_m, int sms);
bool ground_state_cluster(const mma_tdse_grid* grids_dev, int n_grids, int64_t max_m, cudaStream_t st);
// x and the ground state of one grid, without its Crank-Nicolson tables (tdse_kernels.cu)
int ground_state_only(const mma_tdse_grid* grid_dev, int64_t m, cudaStream_t st);

}  // namespace mma
