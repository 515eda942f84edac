// The resident time loops of the eighth-order stencils.
#include "resident_launch.cuh"

namespace pyfwi {

template cudaError_t launch_fwd_resident_r<4>(FwdResArgs &a, cudaStream_t s);
template cudaError_t launch_adj_resident_r<4>(AdjResArgs &a, cudaStream_t s);
template cudaError_t launch_exact_resident_r<4>(AdjResArgs &a, cudaStream_t s);
template cudaError_t launch_rev_resident_r<4>(RevResArgs &a, cudaStream_t s);

}  // namespace pyfwi
