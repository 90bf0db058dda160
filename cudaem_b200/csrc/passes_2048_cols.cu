// Slice-pass kernels for transforms of 2048 points: columns, and the slice engine.
#include "passes.cuh"

namespace msb {

template void col_dispatch<2048>(int op, const PassArgs& a, int nwaves, int nx, cudaStream_t st);
template bool engine_dispatch<2048>(int rowop, const PassArgs& a, const EngineArgs& e, int nwaves, cudaStream_t st);

}  // namespace msb
