// Full-lattice CG with one thread-block cluster per right-hand side (cg_cluster.cu).
#pragma once

#include "solver.cuh"

namespace dwfb {

// Solve d's right-hand sides on the cluster kernel if the lattice fits one and the
// kernel is estimated faster than the grid-wide ones for this batch; *taken tells.
// d.bar is zeroed; d.part is not used. `before` (if not null) is recorded directly
// before the launch.
cudaError_t launch_cg_cluster(SolveDesc& d, bool mixed, int device, int nsm, cudaStream_t stream,
                              cudaEvent_t before, bool* taken);

// Load the code of every FP64 domain-wall instance launch_cg_cluster may pick on the
// current device.
cudaError_t load_cg_cluster64();

}  // namespace dwfb
