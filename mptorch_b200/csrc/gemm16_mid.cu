// Instantiations of the GEMM kernel on 16-bit sums (gemm16_kernel.cuh) with 64 x 64 tiles and 4 x 4 outputs per thread, three
// CTAs per SM: the same rate per SM as 128 x 64 tiles in half the granularity, for products whose 128-row tiles would
// leave SMs idle in the last wave (pick_tile16 in gemm.cu).
#define MPT_MM_TM 4
#include "gemm16_kernel.cuh"

namespace mpt {

int launch_mm16_mid(int algo, const MmParams& p, int64_t batch, cudaStream_t st) {
    return algo == ALGO_SEQ ? launch_any16<ALGO_SEQ, CONV_NONE, 3>(p, batch, st)
         : algo == ALGO_TILE8 ? launch_any16<ALGO_TILE8, CONV_NONE, 3>(p, batch, st) : launch_any16<ALGO_KAHAN, CONV_NONE, 3>(p, batch, st);
}

}  // namespace mpt
