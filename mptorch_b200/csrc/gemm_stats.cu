// Operand statistics of the range-checked GEMM: the largest and the smallest nonzero magnitude of A and of B, per batch entry.
// Bound: HBM for large operands, launches for small ones.
//
// Small operands, or many entries: one cluster of up to eight CTAs reads an entry's A and B, folds its CTAs' extremes through
// distributed shared memory and stores the record: one launch, nothing to initialise.  Otherwise one launch initialises
// the records and one reads both operands with as many CTAs as the GPU holds, folding with atomics.  The line lies where
// eight CTAs alone take longer than the second launch: 512 x 512 twice is 12 us in a cluster and 9 in two launches, cold;
// 96 entries of (1024 x 64, 64 x 1024) are 16 us in clusters and were 78 in three launches (initialise, A, B).
#include <cooperative_groups.h>

#include "gemm_kernel.cuh"

namespace mpt {
namespace {

constexpr int kThreads = 512;
constexpr int64_t kClusterFew = 1 << 17, kClusterMany = 1 << 20;       // elements of A and B of one entry, few or many entries
constexpr int64_t kPerCta = 8192;              // elements that are worth a CTA of a cluster

struct Extremes {
    uint32_t top = 0u, low = 0xFFFFFFFFu;      // largest |x| pattern; smallest nonzero |x| pattern - 1
    __device__ __forceinline__ void take(float v) {
        const uint32_t a = __float_as_uint(v) & 0x7FFFFFFFu;
        top = max(top, a);
        low = min(low, a - 1u);                // zero wraps to the largest value and so never wins
    }
    static __device__ __forceinline__ int64_t quads(const float* x, int64_t n) { return (reinterpret_cast<uintptr_t>(x) & 15u) == 0 ? n / 4 : 0; }
    // elements `first`, first + stride, ... of x in units of 16 bytes (from `skip` strides on), and the remainder one by one
    __device__ __forceinline__ void read(const float* __restrict__ x, int64_t n, int64_t first, int64_t stride, int skip = 0) {
        const int64_t n4 = quads(x, n);
        const float4* x4 = reinterpret_cast<const float4*>(x);
#pragma unroll 4
        for (int64_t i = first + skip * stride; i < n4; i += stride) {
            const float4 v = x4[i];
            take(v.x); take(v.y); take(v.z); take(v.w);
        }
        for (int64_t i = 4 * n4 + first; i < n; i += stride) take(x[i]);
    }
    __device__ __forceinline__ void fold_warp() {
        top = __reduce_max_sync(0xFFFFFFFFu, top);
        low = __reduce_min_sync(0xFFFFFFFFu, low);
    }
    __device__ __forceinline__ uint32_t low_pattern() const { return low == 0xFFFFFFFFu ? low : low + 1u; }
};

__global__ void __launch_bounds__(kThreads) stats_cluster_kernel(const float* __restrict__ a, int64_t na, const float* __restrict__ b,
                                                                 int64_t nb, MmStats* stats) {
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    const int ctas = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int64_t entry = blockIdx.x / ctas;
    __shared__ uint32_t part[4][kThreads / 32];
    __shared__ uint32_t mine[4];
    const int64_t first = (int64_t)rank * kThreads + threadIdx.x, stride = (int64_t)ctas * kThreads;
    Extremes ea, eb;
    const float* x = a + entry * na;
    const float* y = b + entry * nb;
    // the first vectors of both operands travel together; for the smallest products there are no others
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 v = first < Extremes::quads(x, na) ? reinterpret_cast<const float4*>(x)[first] : zero;
    const float4 w = first < Extremes::quads(y, nb) ? reinterpret_cast<const float4*>(y)[first] : zero;
    ea.take(v.x); ea.take(v.y); ea.take(v.z); ea.take(v.w);
    eb.take(w.x); eb.take(w.y); eb.take(w.z); eb.take(w.w);
    ea.read(x, na, first, stride, 1);
    eb.read(y, nb, first, stride, 1);
    ea.fold_warp();
    eb.fold_warp();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { part[0][warp] = ea.top; part[1][warp] = eb.top; part[2][warp] = ea.low; part[3][warp] = eb.low; }
    __syncthreads();
    if (warp < 4) {
        uint32_t v = lane < kThreads / 32 ? part[warp][lane] : (warp < 2 ? 0u : 0xFFFFFFFFu);
        v = warp < 2 ? __reduce_max_sync(0xFFFFFFFFu, v) : __reduce_min_sync(0xFFFFFFFFu, v);
        if (lane == 0) mine[warp] = v;
    }
    cluster.sync();
    if (rank == 0 && threadIdx.x < 4) {
        const int w = threadIdx.x;
        uint32_t v = mine[w];
        for (int r = 1; r < ctas; ++r) {
            const uint32_t o = *cluster.map_shared_rank(&mine[w], r);
            v = w < 2 ? max(v, o) : min(v, o);
        }
        MmStats* s = &stats[entry];
        uint32_t* field = w == 0 ? &s->max_a : w == 1 ? &s->max_b : w == 2 ? &s->minnz_a : &s->minnz_b;
        *field = (w < 2 || v == 0xFFFFFFFFu) ? v : v + 1u;
    }
    cluster.sync();         // no CTA leaves while its shared memory is read
}

__global__ void stats_init_kernel(MmStats* s, int64_t batch) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < batch) { s[i].max_a = 0u; s[i].max_b = 0u; s[i].minnz_a = 0xFFFFFFFFu; s[i].minnz_b = 0xFFFFFFFFu; }
}

// blockIdx.y walks the batch; the first ctas_a CTAs of an entry read A, the others B.
__global__ void __launch_bounds__(kThreads) stats_kernel(const float* __restrict__ a, int64_t na, const float* __restrict__ b, int64_t nb,
                                                         int ctas_a, MmStats* stats) {
    const bool is_a = (int)blockIdx.x < ctas_a;
    const int64_t entry = blockIdx.y, cta = is_a ? blockIdx.x : blockIdx.x - ctas_a, ctas = is_a ? ctas_a : gridDim.x - ctas_a;
    Extremes e;
    if (is_a) e.read(a + entry * na, na, cta * kThreads + threadIdx.x, ctas * kThreads);
    else e.read(b + entry * nb, nb, cta * kThreads + threadIdx.x, ctas * kThreads);
    e.fold_warp();
    if ((threadIdx.x & 31) == 0) {
        atomicMax(is_a ? &stats[entry].max_a : &stats[entry].max_b, e.top);
        atomicMin(is_a ? &stats[entry].minnz_a : &stats[entry].minnz_b, e.low_pattern());
    }
}

}  // namespace

int launch_mm_stats(const float* a, int64_t na, const float* b, int64_t nb, int64_t batch, MmStats* stats, cudaStream_t st) {
    if (na + nb <= (batch >= 16 ? kClusterMany : kClusterFew)) {
        unsigned ctas = 1;
        while (ctas < 8 && (int64_t)ctas * kPerCta < na + nb) ctas *= 2;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)batch * ctas);
        cfg.blockDim = dim3(kThreads);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, stats_cluster_kernel, a, na, b, nb, stats);
        if (e != cudaSuccess) { set_error("operand statistics: %s", cudaGetErrorString(e)); return MPT_ERR_CUDA; }
        return check_launch("operand statistics");
    }
    stats_init_kernel<<<(unsigned)((batch + 255) / 256), 256, 0, st>>>(stats, batch);
    // four CTAs per SM in all, shared out by size, at least one for either operand
    const int64_t cap = ((int64_t)sm_count() * 4 + batch - 1) / batch, want = (na + nb + kPerCta - 1) / kPerCta;
    const int64_t total = want < cap ? want : cap;
    int64_t ctas_a = total * na / (na + nb), ctas_b = total - ctas_a;
    if (ctas_a < 1) ctas_a = 1;
    if (ctas_b < 1) ctas_b = 1;
    stats_kernel<<<dim3((unsigned)(ctas_a + ctas_b), (unsigned)batch), kThreads, 0, st>>>(a, na, b, nb, (int)ctas_a, stats);
    return check_launch("operand statistics");
}

}  // namespace mpt
