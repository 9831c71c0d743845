// Instantiations of the GEMM kernel on 16-bit sums (gemm16_kernel.cuh): the sequential order.
#include "gemm16_kernel.cuh"

namespace mpt {

int launch_mm16_seq(const MmParams& p, int64_t batch, cudaStream_t st) { return launch_any16<ALGO_SEQ, CONV_NONE, 2>(p, batch, st); }

}  // namespace mpt
