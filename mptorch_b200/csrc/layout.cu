// Batched transpose of the last two dimensions: out[b][c][r] = in[b][r][c].
//
// The layers hand the GEMM transposed views (W^T in the forward pass, dY^T and X^T for the weight gradient, K^T in
// attention), and the GEMM wants dense row-major operands; this kernel makes the dense copy at close to the copy
// bandwidth, where a generic strided elementwise copy reads or writes one of the two sides 4 bytes at a time per
// 32-byte sector.  A CTA moves a 64 x 64 tile through shared memory: 16-byte coalesced reads along the input rows,
// 16-byte coalesced writes along the output rows, the row pitch of 65 words keeping the column reads free of bank
// conflicts.  HBM-bound: 8 bytes per element.
#include "async_copy.cuh"
#include "common.cuh"

namespace mpt {
namespace {

constexpr int kTile = 64;

__global__ void __launch_bounds__(256) transpose_kernel(const float* __restrict__ in, float* __restrict__ out, int rows, int cols) {
    __shared__ float tile[kTile][kTile + 1];
    const int64_t plane = (int64_t)rows * cols;
    const float* src = in + blockIdx.z * plane;
    float* dst = out + blockIdx.z * plane;
    const int r0 = blockIdx.y * kTile, c0 = blockIdx.x * kTile;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;          // 16 x 16 threads, 4 columns each, 4 row passes
    const bool vec_in = (cols & 3) == 0 && ((reinterpret_cast<uintptr_t>(in) & 15u) == 0);
    const bool vec_out = (rows & 3) == 0 && ((reinterpret_cast<uintptr_t>(out) & 15u) == 0);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int r = r0 + ty + 16 * p, c = c0 + 4 * tx;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (r < rows) {
            if (vec_in && c + 3 < cols) {
                const float4 q = *reinterpret_cast<const float4*>(src + (int64_t)r * cols + c);
                v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (c + j < cols) v[j] = src[(int64_t)r * cols + c + j];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) tile[ty + 16 * p][4 * tx + j] = v[j];
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int c = c0 + ty + 16 * p, r = r0 + 4 * tx;             // output row c, output columns r .. r + 3
        if (c >= cols) continue;
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = tile[4 * tx + j][ty + 16 * p];
        if (vec_out && r + 3 < rows) *reinterpret_cast<float4*>(dst + (int64_t)c * rows + r) = make_float4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (r + j < rows) dst[(int64_t)c * rows + r + j] = v[j];
        }
    }
}

}  // namespace
}  // namespace mpt

extern "C" int mpt_transpose_last2(const float* in, float* out, int64_t batch, int64_t rows, int64_t cols, void* stream) {
    using namespace mpt;
    if (batch == 0 || rows == 0 || cols == 0) return MPT_OK;
    MPT_REQUIRE(in && out && batch > 0 && rows > 0 && cols > 0, "transpose_last2: bad arguments");
    MPT_REQUIRE(in != out, "transpose_last2: in place is not supported");
    const int64_t gx = (cols + kTile - 1) / kTile, gy = (rows + kTile - 1) / kTile;
    MPT_REQUIRE(rows <= 0x7FFFFFFF && cols <= 0x7FFFFFFF && gy <= 65535 && batch <= 65535,
                "transpose_last2: more than 65535 row tiles or batch entries");
    transpose_kernel<<<dim3((unsigned)gx, (unsigned)gy, (unsigned)batch), 256, 0, static_cast<cudaStream_t>(stream)>>>(in, out, (int)rows, (int)cols);
    return check_launch("transpose_last2");
}

// ---- folding an unfolded gradient ------------------------------------------------------------------------------------
// The input gradient of a convolution from the gradient of its unfolded input, cols [n_img][OH * OW][channels * KH * KW] (what
// the GEMM of the backward pass writes): every pixel is the fp32 sum, from zero, of the entries that were copies of it,
// in ascending output position.  HBM-bound: the unfolded gradient is read once (KH * KW times the image), the image
// written once.  A CTA owns a tile of one image's pixels and a few channels; it brings the output positions that touch
// the tile into shared memory, each position's channels as one contiguous run, and then sums with lanes along the
// image row.  64 x 64 x 56 x 56, 3 x 3, 462 MB unfolded: 0.385 ms (1.3 TB/s; the sums' index arithmetic and shared-memory
// reads are what is left), against 2.25 ms for a transposing copy and a pixel-by-pixel gather from global memory.
namespace mpt {
namespace {

struct FoldGeom {
    int H, W, KH, KW, OH, OW, sh, sw, ph, pw, dh, dw;
    int channels, cc, th, tw, rows, cols, pitch;       // channels per CTA, pixel tile, output positions a tile can touch, floats between them
    int64_t out_image_stride;
};

// VEC: the runs start on 16-byte boundaries and are multiples of 16 bytes.  DILATED: some kernel taps are apart.
template <bool VEC, bool DILATED>
__global__ void __launch_bounds__(256) fold_kernel(const float* __restrict__ cols, float* __restrict__ out, const __grid_constant__ FoldGeom g) {
    extern __shared__ __align__(16) float pos[];
    const int tiles_w = (g.W + g.tw - 1) / g.tw;
    const int h0 = ((int)blockIdx.x / tiles_w) * g.th, w0 = ((int)blockIdx.x % tiles_w) * g.tw;
    const int c0 = blockIdx.y * g.cc, nc = min(g.cc, g.channels - c0);
    const int64_t img = blockIdx.z;
    const int kk = g.KH * g.KW, run = nc * kk;
    // output rows and columns that can touch the tile
    const int reach_h = (g.KH - 1) * g.dh, reach_w = (g.KW - 1) * g.dw;
    const int oh0 = max(0, (h0 + g.ph - reach_h + g.sh - 1) / g.sh), ow0 = max(0, (w0 + g.pw - reach_w + g.sw - 1) / g.sw);
    const int oh1 = min(g.OH - 1, (min(h0 + g.th, g.H) - 1 + g.ph) / g.sh), ow1 = min(g.OW - 1, (min(w0 + g.tw, g.W) - 1 + g.pw) / g.sw);
    const int nr = max(0, oh1 - oh0 + 1), ncol = max(0, ow1 - ow0 + 1);
    const int64_t stride = (int64_t)g.channels * kk;
    const float* src = cols + img * ((int64_t)g.OH * g.OW) * stride + (int64_t)c0 * kk;
    const unsigned pieces = VEC ? run / 4 : run, row = ncol * pieces;
    for (int r = 0; r < nr; ++r) {
        const float* s = src + ((int64_t)(oh0 + r) * g.OW + ow0) * stride;
        float* d = pos + r * g.cols * g.pitch;
        for (unsigned i = threadIdx.x; i < row; i += 256) {
            const unsigned c = i / pieces, e = i - c * pieces;
            if (VEC) cp_async16(d + c * g.pitch + 4 * e, s + c * stride + 4 * e, 16);
            else cp_async4(d + c * g.pitch + e, s + c * stride + e, 4);
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int cy = warp; cy < nc * g.th; cy += 8) {
        const int c = cy / g.th, h = h0 + cy - c * g.th;
        if (h >= g.H) continue;
        const int lo_h = max(oh0, (h + g.ph - reach_h + g.sh - 1) / g.sh), hi_h = min(oh1, (h + g.ph) / g.sh);
        float* dst = out + img * g.out_image_stride + ((int64_t)(c0 + c) * g.H + h) * g.W;
        for (int w = w0 + lane; w < min(w0 + g.tw, g.W); w += 32) {
            const int lo_w = max(ow0, (w + g.pw - reach_w + g.sw - 1) / g.sw), hi_w = min(ow1, (w + g.pw) / g.sw);
            float sum = 0.0f;
            for (int oh = lo_h; oh <= hi_h; ++oh) {
                const int a = h + g.ph - oh * g.sh;                 // kernel row times dilation
                if (a < 0 || a > reach_h || (DILATED && a % g.dh)) continue;
                const float* p = pos + ((oh - oh0) * g.cols - ow0) * g.pitch + c * kk + (DILATED ? a / g.dh : a) * g.KW;
                for (int ow = lo_w; ow <= hi_w; ++ow) {
                    const int b = w + g.pw - ow * g.sw;
                    if (b < 0 || b > reach_w || (DILATED && b % g.dw)) continue;
                    sum = __fadd_rn(sum, p[ow * g.pitch + (DILATED ? b / g.dw : b)]);
                }
            }
            dst[w] = sum;
        }
    }
}

}  // namespace
}  // namespace mpt

extern "C" int mpt_fold(const float* cols, float* out, int n_img, int channels, int H, int W, int KH, int KW, int stride_h, int stride_w,
                        int pad_h, int pad_w, int dil_h, int dil_w, int64_t out_image_stride, void* stream) {
    using namespace mpt;
    MPT_REQUIRE(n_img >= 0 && channels >= 0 && H >= 0 && W >= 0, "fold: negative extent");
    MPT_REQUIRE(KH >= 1 && KW >= 1 && stride_h >= 1 && stride_w >= 1 && dil_h >= 1 && dil_w >= 1 && pad_h >= 0 && pad_w >= 0,
                "fold: invalid kernel / stride / padding / dilation");
    if (n_img == 0 || channels == 0 || H == 0 || W == 0) return MPT_OK;
    FoldGeom g;
    g.H = H; g.W = W; g.KH = KH; g.KW = KW; g.sh = stride_h; g.sw = stride_w; g.ph = pad_h; g.pw = pad_w; g.dh = dil_h; g.dw = dil_w;
    const int64_t span_h = H + 2 * (int64_t)pad_h - (int64_t)dil_h * (KH - 1) - 1, span_w = W + 2 * (int64_t)pad_w - (int64_t)dil_w * (KW - 1) - 1;
    MPT_REQUIRE(span_h >= 0 && span_w >= 0, "fold: no output position");
    // what the kernel works out about positions, reaches and kernel rows is 32 bits wide
    const auto fits = [](int64_t e, int64_t k, int64_t s, int64_t p, int64_t d, int64_t span) {
        return e + p + s - 2 <= 0x7FFFFFFF && (k - 1) * d <= 0x7FFFFFFF && span / s < 0x7FFFFFFF;
    };
    MPT_REQUIRE(fits(H, KH, stride_h, pad_h, dil_h, span_h) && fits(W, KW, stride_w, pad_w, dil_w, span_w), "fold: padded image or stride too large");
    g.OH = (int)(span_h / stride_h) + 1; g.OW = (int)(span_w / stride_w) + 1;
    g.channels = channels; g.out_image_stride = out_image_stride;
    MPT_REQUIRE(cols && out && out_image_stride >= (int64_t)channels * H * W, "fold: bad arguments");
    MPT_REQUIRE(n_img <= 65535, "fold: more than 65535 images");
    // The largest tile and channel count whose output positions fit the shared memory of half an SM; the halo (the positions
    // outside the tile that touch it) is read again by the neighbours, so the tile shrinks last.
    constexpr int64_t kFloats = 24 * 1024;
    const auto positions = [](int tile, int k, int dil, int stride, int o) { const int64_t n = ((int64_t)tile - 1 + (int64_t)(k - 1) * dil) / stride + 1; return (int)(n < o ? n : o); };
    MPT_REQUIRE((int64_t)KH * KW < (1 << 24), "fold: kernel too large");
    const int kk = KH * KW;
    const auto choose = [&](bool vec) {
        const int spare = vec ? 7 : 1, whole = vec ? 4 : 1;      // pitch above the run, at most; granularity of the channel count
        for (g.th = H < 8 ? H : 8, g.tw = W < 64 ? W : 64;;) {
            g.rows = positions(g.th, KH, dil_h, stride_h, g.OH); g.cols = positions(g.tw, KW, dil_w, stride_w, g.OW);
            const int64_t at = (int64_t)g.rows * g.cols;
            int64_t cc = (kFloats - at * spare) > 0 ? (kFloats - at * spare) / (at * kk) : 0;
            cc = cc > 16 ? 16 : cc;
            cc = cc >= channels ? channels : cc / whole * whole;
            const bool last = g.th == 1 && g.tw == 1;
            if (cc >= (channels < 4 ? channels : 4) || (cc >= 1 && last)) { g.cc = (int)cc; return true; }
            if (last) return false;
            if (g.th > 1 && (g.th >= 4 || g.tw <= 16)) g.th = (g.th + 1) / 2;
            else if (g.tw > 1) g.tw = (g.tw + 1) / 2;
            else g.th = (g.th + 1) / 2;
        }
    };
    bool vec = ((int64_t)channels * kk) % 4 == 0 && (reinterpret_cast<uintptr_t>(cols) & 15u) == 0 && choose(true);
    MPT_REQUIRE(vec || choose(false), "fold: one pixel's output positions exceed shared memory");
    // lanes read neighbouring positions: an odd pitch has no bank conflicts; runs of 16 bytes need a multiple of 4, 4 modulo 8
    g.pitch = vec ? ((g.cc * kk + 3) & ~3) | 4 : (g.cc * kk) | 1;
    const int64_t tiles = (int64_t)((H + g.th - 1) / g.th) * ((W + g.tw - 1) / g.tw), gy = (channels + g.cc - 1) / g.cc;
    MPT_REQUIRE(tiles <= 0x7FFFFFFF && gy <= 65535, "fold: image or channel count too large");
    const size_t smem = sizeof(float) * (size_t)g.rows * g.cols * (size_t)g.pitch;
    const bool dilated = (dil_h > 1 && KH > 1) || (dil_w > 1 && KW > 1);
    auto kern = vec ? (dilated ? fold_kernel<true, true> : fold_kernel<true, false>) : (dilated ? fold_kernel<false, true> : fold_kernel<false, false>);
    // the limit belongs to the function on this device, not to the call: the same for every call, so that threads with different
    // shapes leave one another's launches alone
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kFloats * sizeof(float)));
    if (e != cudaSuccess) { set_error("fold: cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return MPT_ERR_CUDA; }
    kern<<<dim3((unsigned)tiles, (unsigned)gy, (unsigned)n_img), 256, smem, static_cast<cudaStream_t>(stream)>>>(cols, out, g);
    return check_launch("fold");
}
