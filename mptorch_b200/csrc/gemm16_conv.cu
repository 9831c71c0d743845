// Instantiations of the GEMM kernel on 16-bit sums (gemm16_kernel.cuh): convolution and its weight gradient.
#include "gemm16_kernel.cuh"

namespace mpt {

int launch_conv16(int algo, const MmParams& p, cudaStream_t st) {
    return algo == ALGO_SEQ ? launch_any16<ALGO_SEQ, CONV_FWD, 2>(p, 1, st) : launch_any16<ALGO_TILE8, CONV_FWD, 2>(p, 1, st);
}

int launch_conv16_wgrad(int algo, const MmParams& p, cudaStream_t st) {
    return algo == ALGO_SEQ ? launch_any16<ALGO_SEQ, CONV_WGRAD, 2>(p, 1, st) : launch_any16<ALGO_TILE8, CONV_WGRAD, 2>(p, 1, st);
}

}  // namespace mpt
