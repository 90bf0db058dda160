// Slice-pass kernels for transforms of 2048 points: rows.
#include "passes.cuh"

namespace msb {

template void row_dispatch<2048>(int op, const PassArgs& a, int nwaves, int ny, cudaStream_t st);

}  // namespace msb
