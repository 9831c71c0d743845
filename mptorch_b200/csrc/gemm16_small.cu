// Instantiations of the GEMM kernel on 16-bit sums (gemm16_kernel.cuh) with 16 x 64 tiles and 1 x 4 outputs per thread, for
// products with a small result (see gemm_small.cu, whose shapes these are).
#define MPT_MM_TM 1
#include "gemm16_kernel.cuh"

namespace mpt {

static_assert(BM == kSmallTileRows, "the host side sizes its grid checks with kSmallTileRows");

int launch_mm16_small(int algo, const MmParams& p, int64_t batch, cudaStream_t st) {
    return algo == ALGO_SEQ ? launch_any16<ALGO_SEQ, CONV_NONE, 4>(p, batch, st) : launch_any16<ALGO_TILE8, CONV_NONE, 4>(p, batch, st);
}

int launch_conv16_wgrad_small(int algo, const MmParams& p, cudaStream_t st) {
    return algo == ALGO_SEQ ? launch_any16<ALGO_SEQ, CONV_WGRAD, 4>(p, 1, st) : launch_any16<ALGO_TILE8, CONV_WGRAD, 4>(p, 1, st);
}

}  // namespace mpt
