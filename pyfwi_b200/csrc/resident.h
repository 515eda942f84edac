// Host interface of the resident time loops (resident.cu).
#pragma once

#include "resident_kernels.cuh"

namespace pyfwi {

enum ResLoop { RES_FORWARD, RES_ADJOINT, RES_EXACT };  // (the reverse-time loop has the forward one's tilings)

// The tiling of a time loop of up to `shots` shots on `sms` SMs: tiles per
// shot and shots per launch.  False when no tiling fits on chip.
__attribute__((visibility("hidden"))) bool resident_tiles(const Grid &g, int R, const Lines &lines, int shots, int sms,
                                                          ResLoop loop, ResTiles *out);

__attribute__((visibility("hidden"))) cudaError_t launch_fwd_resident(FwdResArgs &a, int R, cudaStream_t s);
__attribute__((visibility("hidden"))) cudaError_t launch_adj_resident(AdjResArgs &a, int R, cudaStream_t s);
__attribute__((visibility("hidden"))) cudaError_t launch_exact_resident(AdjResArgs &a, int R, cudaStream_t s);
__attribute__((visibility("hidden"))) cudaError_t launch_rev_resident(RevResArgs &a, int R, cudaStream_t s);

// The same for one half order (resident.cu, resident8.cu).
template <int R>
__attribute__((visibility("hidden"))) cudaError_t launch_fwd_resident_r(FwdResArgs &a, cudaStream_t s);
template <int R>
__attribute__((visibility("hidden"))) cudaError_t launch_adj_resident_r(AdjResArgs &a, cudaStream_t s);
template <int R>
__attribute__((visibility("hidden"))) cudaError_t launch_exact_resident_r(AdjResArgs &a, cudaStream_t s);
template <int R>
__attribute__((visibility("hidden"))) cudaError_t launch_rev_resident_r(RevResArgs &a, cudaStream_t s);

}  // namespace pyfwi
