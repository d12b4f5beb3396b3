// Single-right-hand-side persistent CG (single.cu).
#pragma once

#include "solver.cuh"

namespace dwfb {

constexpr int kSingleThreads = 512;  // largest block of cg_single_kernel

// Doubles of d.part that launch_single needs on a device with nsm SMs.
size_t single_part_doubles(int nsm);

// Solve the one right-hand side of `d` (d.nrhs = 1; d.part holds
// single_part_doubles(nsm) doubles, d.bar is zeroed) on `stream`; sets d.nch,
// d.ch and d.expected_blocks. `before` (if not null) is recorded directly before the
// launch.
cudaError_t launch_single(SolveDesc& d, bool mixed, int nsm, cudaStream_t stream, cudaEvent_t before);

// Load the code of launch_single's FP64 or mixed instances on the current device.
cudaError_t load_single(bool mixed);

}  // namespace dwfb
