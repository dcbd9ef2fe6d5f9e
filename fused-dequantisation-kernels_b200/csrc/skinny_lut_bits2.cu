#include "skinny_lut_kernel.cuh"

namespace fdk {
template int launch_skinny_bits<2>(LinearParams, const void*, int, int, unsigned, cudaStream_t);
}  // namespace fdk
