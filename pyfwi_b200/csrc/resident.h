// Host interface of the resident time loops (resident.cu).
#pragma once

#include "resident_kernels.cuh"

namespace pyfwi {

enum ResLoop { RES_FORWARD, RES_ADJOINT, RES_EXACT };  // (the reverse-time loop has the forward one's tilings)

// The tiling of a time loop of up to `shots` shots on `sms` SMs: tiles per
// shot and shots per launch; us: the modelled time of a step of all of them.
// False when no tiling fits on chip.
__attribute__((visibility("hidden"))) bool resident_tiles(const Grid &g, int R, const Lines &lines, int shots, int sms,
                                                          ResLoop loop, ResTiles *out, double *us = nullptr);

// Whether the passes of a survey of `shots` shots are faster on chip than by step
// kernels of `rows` rows per tile: fwd, bwd.  The store holds difference sets
// (RES_OF_SETS), the states of every step (RES_OF_STATES) or checkpoints, from which
// chunks of `chunk` steps are reconstructed (RES_OF_CHECKPOINTS; 0: no room for chunks).
enum ResStore { RES_OF_SETS, RES_OF_STATES, RES_OF_CHECKPOINTS };
__attribute__((visibility("hidden"))) void resident_pays(const Grid &g, int R, const Lines &lines, int shots, int rows, ResStore store,
                                                         int chunk, bool energy, bool *fwd, bool *bwd);

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
