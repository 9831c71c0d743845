// The GEMM on 16-bit sums (gemm16_kernel.cuh) for products with a small result and a long K: the weight gradient of a layer over
// a large batch, the same gradient of a convolution, and small products altogether.
//
// Every output is one chain of rounded sums over K, so such a product has only its outputs to run in parallel, and what
// bounds it is the time one step takes in the few warps there are.  128 threads compute 8 x 32 outputs, ONE pair each:
// the weight gradient of a 3 x 3 layer of 64 channels (64 x 576 outputs) becomes 144 CTAs for 148 SMs, one warp per
// scheduler.  In the CUDA order four groups of eight steps run at once (their inner sums start from zero), so that the
// conversions' latencies overlap.  K slabs of 64 through three cp.async stages.  Against 16 x 64 tiles of mm16_kernel
// (1 x 4 outputs per thread): 256 x 256 x 4096 170 -> 114 us, that gradient 10.0 -> 4.0 ms (4.9 while the computing warps staged), 64 x 64 x 1024 36 -> 30 us.
//
// The weight gradient of a convolution gathers B from the input (CONV_WGRAD): a lane owns two output positions of the slab,
// walks them forward slab by slab without divisions, and copies them for eight of the tile's columns (channel, kernel
// row, kernel column), so that a warp's 32 copies are neighbouring pixels.  Its address arithmetic is as long as the sums
// themselves, and with one warp per scheduler nothing covers it, so four more warps of the CTA do the staging.
#include "gemm16_kernel.cuh"

namespace mpt {
namespace {

constexpr int TBM = 8, TBN = 32, TBK = 64, TTHREADS = 128, TSTAGES = 3;
constexpr int kRun = 4;         // groups of eight steps in flight per thread (CUDA order)
constexpr int TA_LD = TBK + 4;
__host__ __device__ constexpr int stagers(int conv) { return conv == CONV_WGRAD ? TTHREADS : 0; }      // threads that only stage
__host__ __device__ constexpr int tb_ld(int conv) { return conv == CONV_WGRAD ? TBN + 2 : TBN + 4; }   // 4-byte column writes / 16-byte rows

// `n` steps of a pair on the exact casters: a = the thread's row of the A slab, b = its column pair of the B slab.
// SHORT: the short form first (entries without a plan in formats with subnormals).
template <bool FMA, bool SHORT, bool EIGHT>
__device__ __noinline__ float2 thin_exact_steps(float2 acc, const float* a, const float* b, int ldb, int n, const MmParams* pp) {
    const MmParams& p = *pp;
    // a sum of an 8-bit-exponent format that continues from a -0 keeps its sign, which the short form does not
    const bool minus_zero = __float_as_uint(acc.x) == 0x80000000u || __float_as_uint(acc.y) == 0x80000000u;
    if (SHORT && !(EIGHT && minus_zero)) {
        float v[1][2] = {{acc.x, acc.y}};
        if (short_steps<FMA, EIGHT, 1, 2>(v, a, 0, b, ldb, n, ShortRn::make(p.wadd), ShortRn::make(p.wmul))) return make_float2(v[0][0], v[0][1]);
    }
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const float av = a[k];
        const float2 bv = *reinterpret_cast<const float2*>(b + k * ldb);
        if (FMA) {
            acc.x = round_add(p, fma_rn(av, bv.x, acc.x)); acc.y = round_add(p, fma_rn(av, bv.y, acc.y));
        } else {
            acc.x = round_add(p, add_rn(acc.x, round_mul(p, mul_rn(av, bv.x)))); acc.y = round_add(p, add_rn(acc.y, round_mul(p, mul_rn(av, bv.y))));
        }
    }
    return acc;
}

template <int SUM, int PROD, bool START, bool NOSUB>
__device__ __forceinline__ bool thin_group16(uint32_t& acc, const float* a, const float* b, int ldb, const Settle16& ns) {
    uint32_t below = 0xFFFFFFFFu;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float4 av = *reinterpret_cast<const float4*>(a + 4 * h);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 bv = *reinterpret_cast<const float2*>(b + (4 * h + j) * ldb);
            acc = step16<SUM, PROD, NOSUB, false>(acc, j == 0 ? av.x : j == 1 ? av.y : j == 2 ? av.z : av.w, bv, START && h == 0 && j == 0, ns, below);
        }
    }
    return NOSUB && sum_can_settle16(SUM, PROD) && any_small16(below, ns.min_norm);
}

template <int SUM> __device__ __forceinline__ bool pair_below16(uint32_t v, uint32_t lim) {
    v &= 0x7FFF7FFFu;
    return max(v & 0xFFFFu, v >> 16) < lim;
}

// An output position of the convolution: image, row, column; advanced by TBK positions per slab.
struct Position {
    int img, oh, ow;
    __device__ __forceinline__ void start(int k, const ConvGeom& g) {
        const int L = g.OH * g.OW;
        img = k / L;
        const int l = k - img * L;
        oh = l / g.OW; ow = l - oh * g.OW;
    }
    __device__ __forceinline__ void advance(int d_oh, int d_ow, const ConvGeom& g) {
        ow += d_ow; oh += d_oh;
        if (ow >= g.OW) { ow -= g.OW; ++oh; }
        while (oh >= g.OH) { oh -= g.OH; ++img; }
    }
};
struct Column { int64_t off; int dih, diw; };       // input offset of (channel, kernel row, kernel column); rows past N: dih out of every image

template <int ALGO, int SUM, int PROD, bool NOSUB, int CONV>
__global__ void __launch_bounds__(TTHREADS + stagers(CONV), CONV == CONV_WGRAD ? 3 : 6) mm16_thin_kernel(const __grid_constant__ MmParams p) {
    constexpr bool FMA = PROD == PROD16_FUSED;
    constexpr bool kFlush = NOSUB && sum_can_settle16(SUM, PROD);
    constexpr int LDB = tb_ld(CONV);
    __shared__ __align__(16) float As[TSTAGES][TBM * TA_LD];
    __shared__ __align__(16) float Bs[TSTAGES][TBK * LDB];
    __shared__ Column cols[CONV == CONV_WGRAD ? TBN : 1];

    const bool computes = threadIdx.x < TTHREADS, stages = stagers(CONV) == 0 || !computes;
    const int tid = threadIdx.x & (TTHREADS - 1), ty = tid >> 4, tx = tid & 15;
    const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
    const int64_t batch = blockIdx.z;
    const float* A = p.a + batch * p.stride_a;
    const float* B = p.b + batch * p.stride_b;
    float* C = p.c + batch * p.stride_c;

    const FastPlan plan = make_plan<ALGO, FMA>(p, batch);
    if (CONV == CONV_NONE && p.defer_exact && !plan.ok) return;
    // see mm16_kernel for the padding each form walks
    const int ksteps = plan.ok && (ALGO == ALGO_SEQ || !kFlush) ? (p.K + 7) / 8 * 8
                     : (ALGO == ALGO_SEQ || (p.resume & MM_MORE)) ? p.K : p.K + 8 - p.K % 8;
    const int ntiles = (ksteps + TBK - 1) / TBK;
    const uint32_t lim = SUM == SUM16_BF16 ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rd(plan.acc_limit))
                                           : (uint32_t)__half_as_ushort(__float2half_rd(plan.acc_limit));
    const Settle16 ns = Settle16::make(p.fmul);

    const int L = CONV == CONV_WGRAD ? p.cv.OH * p.cv.OW : 1;
    Position pos[2];
    if (CONV == CONV_WGRAD) {
        if (computes && tid < TBN) {
            const int gj = n0 + tid, khkw = p.cv.KH * p.cv.KW;
            const int ch = gj / khkw, rem = gj - ch * khkw, kh = rem / p.cv.KW, kw = rem - kh * p.cv.KW;
            Column c;
            c.dih = gj < p.N ? kh * p.cv.dh - p.cv.ph : -(1 << 30);
            c.diw = kw * p.cv.dw - p.cv.pw;
            c.off = gj < p.N ? (int64_t)ch * p.cv.H * p.cv.W : 0;
            cols[tid] = c;
        }
        pos[0].start(tid & 31, p.cv);
        pos[1].start((tid & 31) + 32, p.cv);
        __syncthreads();
    }
    const int d_oh = CONV == CONV_WGRAD ? TBK / p.cv.OW : 0, d_ow = CONV == CONV_WGRAD ? TBK - d_oh * p.cv.OW : 0;

    auto stage = [&](int s, int k0) {
        float* as = As[s];
        float* bs = Bs[s];
        if (CONV == CONV_WGRAD) {
            // A[m][k] = dY[image(k)][m][position(k)], B[k][j] = x[image(k)][channel(j)][ih][iw]; slabs come in order
            const int lane = tid & 31, w = tid >> 5;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int gk = k0 + 32 * hh + lane;
                const bool kok = gk < p.K;
                const Position ps = pos[hh];
                const int64_t ybase = (int64_t)ps.img * p.cv.y_image_stride + (ps.oh * p.cv.OW + ps.ow);
#pragma unroll
                for (int u = 0; u < TBM / 4; ++u) {
                    const int row = w + 4 * u, gm = m0 + row;
                    const bool ok = kok && gm < p.M;
                    cp_async4(as + row * TA_LD + 32 * hh + lane, ok ? A + ybase + (int64_t)gm * L : A, ok ? 4 : 0);
                }
                const int ih0 = ps.oh * p.cv.sh, iw0 = ps.ow * p.cv.sw;
                const int64_t xbase = (int64_t)ps.img * p.cv.x_image_stride;
#pragma unroll
                for (int u = 0; u < TBN / 4; ++u) {
                    const int j = w * (TBN / 4) + u;
                    const Column c = cols[j];
                    const int ih = ih0 + c.dih, iw = iw0 + c.diw;
                    const bool ok = kok && (unsigned)ih < (unsigned)p.cv.H && (unsigned)iw < (unsigned)p.cv.W;
                    cp_async4(bs + (32 * hh + lane) * LDB + j, ok ? B + xbase + c.off + (ih * p.cv.W + iw) : B, ok ? 4 : 0);
                }
                pos[hh].advance(d_oh, d_ow, p.cv);
            }
        } else if (p.vec) {
            {
                const int row = tid >> 4, kc = (tid & 15) << 2;
                const int gm = m0 + row, gk = k0 + kc;
                const int bytes = gm < p.M ? bytes16(p.K - gk) : 0;
                cp_async16(as + row * TA_LD + kc, bytes ? A + (int64_t)gm * p.K + gk : A, bytes);
            }
#pragma unroll
            for (int u = 0; u < TBK * TBN / 4 / TTHREADS; ++u) {
                const int c = tid + u * TTHREADS, kr = c >> 3, nc = (c & 7) << 2;
                const int gk = k0 + kr, gn = n0 + nc;
                const int bytes = gk < p.K ? bytes16(p.N - gn) : 0;
                cp_async16(bs + kr * LDB + nc, bytes ? B + (int64_t)gk * p.N + gn : B, bytes);
            }
        } else {
#pragma unroll
            for (int u = 0; u < TBM * TBK / TTHREADS; ++u) {
                const int c = tid + u * TTHREADS, row = c >> 6, kk = c & 63;
                const bool ok = m0 + row < p.M && k0 + kk < p.K;
                cp_async4(as + row * TA_LD + kk, ok ? A + (int64_t)(m0 + row) * p.K + k0 + kk : A, ok ? 4 : 0);
            }
#pragma unroll 4
            for (int u = 0; u < TBK * TBN / TTHREADS; ++u) {
                const int c = tid + u * TTHREADS, kr = c >> 5, nn = c & 31;
                const bool ok = k0 + kr < p.K && n0 + nn < p.N;
                cp_async4(bs + kr * LDB + nn, ok ? B + (int64_t)(k0 + kr) * p.N + n0 + nn : B, ok ? 4 : 0);
            }
        }
    };

    uint32_t acc = 0u, aux = 0u;        // running (inner) sums; outer sums of the CUDA order
    const int gm = m0 + ty, gn = n0 + 2 * tx;
    float2 c_in = make_float2(0.0f, 0.0f);
    bool wide_start = false;            // C holds something that is not a rounded sum: start from its 32 bits (mm16_kernel)
    if (CONV == CONV_NONE && (p.resume & MM_FROM_C) && gm < p.M) {
        if (gn < p.N) c_in.x = C[(int64_t)gm * p.N + gn];
        if (gn + 1 < p.N) c_in.y = C[(int64_t)gm * p.N + gn + 1];
        const auto odd = [&](float v) { return __float_as_uint(v) == 0x80000000u || (v == v && __float_as_uint(exact_add_cold(&p, v)) != __float_as_uint(v)); };
        wide_start = odd(c_in.x) || odd(c_in.y);
        (ALGO == ALGO_TILE8 ? aux : acc) = pack16<SUM>(c_in);
    }

#pragma unroll
    for (int s = 0; s < TSTAGES - 1; ++s) {
        if (stages && s < ntiles) stage(s, s * TBK);
        cp_async_commit();
    }
    int slot = 0;
    for (int t = 0; t < ntiles; ++t) {
        cp_async_wait<TSTAGES - 2>();
        __syncthreads();
        {
            const int nt = t + TSTAGES - 1;
            if (stages && nt < ntiles) stage(slot == 0 ? TSTAGES - 1 : slot - 1, nt * TBK);
            cp_async_commit();
        }
        const int now = slot;
        slot = slot == TSTAGES - 1 ? 0 : slot + 1;
        if (!computes) continue;
        const float* arow = As[now] + ty * TA_LD;
        const float* bcol = Bs[now] + 2 * tx;
        const int nk_tile = min(ksteps - t * TBK, TBK);
        int k0 = 0;
        // Several groups at once: the inner sums of the CUDA order start from zero, so four groups are four independent chains
        // in straight-line code; their folds are taken on trust and all conditions looked at together (the sums before every
        // fold below the limit, nothing to settle).  A run that fails is done again group by group below.
        if (ALGO == ALGO_TILE8 && plan.ok && !(wide_start && t == 0)) {
#pragma unroll 1
            for (; k0 + 8 * kRun <= nk_tile; k0 += 8 * kRun) {
                uint32_t inner[kRun], out = aux, top = 0u, below = 0xFFFFFFFFu;
                bool small = false;
#pragma unroll
                for (int g = 0; g < kRun; ++g) small |= thin_group16<SUM, PROD, true, NOSUB>(inner[g], arow + k0 + 8 * g, bcol + (k0 + 8 * g) * LDB, LDB, ns);
#pragma unroll
                for (int g = 0; g < kRun; ++g) {
                    top = maxabs16<SUM>(top, out);
                    out = sum16<SUM>(out, inner[g]);
                    if (kFlush) note_small16(below, out);
                }
                if (!pair_below16<SUM>(top, lim) || small || (kFlush && any_small16(below, ns.min_norm))) break;
                aux = out;
            }
        }
#pragma unroll 1
        for (; k0 < nk_tile; k0 += 8) {
            const float* ak = arow + k0;
            const float* bk = bcol + k0 * LDB;
            const bool wide = wide_start && t == 0 && k0 == 0;
            if (ALGO == ALGO_TILE8) {
                bool redo = !plan.ok;
                if (plan.ok) redo = thin_group16<SUM, PROD, true, NOSUB>(acc, ak, bk, LDB, ns);
                if (redo) acc = pack16<SUM>(thin_exact_steps<FMA, CONV == CONV_NONE && !NOSUB, SUM == SUM16_BF16>(make_float2(0.0f, 0.0f), ak, bk, LDB, min(nk_tile - k0, 8), &p));
                bool folded = false;
                if (plan.ok && !wide && pair_below16<SUM>(aux, lim)) {
                    uint32_t below = 0xFFFFFFFFu;
                    const uint32_t out = sum16<SUM>(aux, acc);
                    if (kFlush) note_small16(below, out);
                    folded = !(kFlush && any_small16(below, ns.min_norm));
                    if (folded) aux = out;
                }
                if (!folded) {
                    float2 f = unpack16<SUM>(acc);
                    const float2 o = wide ? c_in : unpack16<SUM>(aux);
                    if (wide && !redo) f = make_float2(add_rn(f.x, 0.0f), add_rn(f.y, 0.0f));
                    aux = pack16<SUM>(make_float2(exact_add_cold(&p, add_rn(o.x, f.x)), exact_add_cold(&p, add_rn(o.y, f.y))));
                }
            } else {
                const int kleft = p.K - t * TBK - k0;
                bool redo = true;
                const uint32_t saved = acc;
                const bool minus_zero = (acc & 0xFFFFu) == 0x8000u || (acc >> 16) == 0x8000u;
                if (plan.ok && !wide && pair_below16<SUM>(acc, lim) && !(kFlush && kleft < 8 && minus_zero))
                    redo = thin_group16<SUM, PROD, false, NOSUB>(acc, ak, bk, LDB, ns);
                if (redo) acc = pack16<SUM>(thin_exact_steps<FMA, CONV == CONV_NONE && !NOSUB, SUM == SUM16_BF16>(wide ? c_in : unpack16<SUM>(saved), ak, bk, LDB, min(min(nk_tile - k0, 8), kleft), &p));
            }
        }
    }
    cp_async_wait<0>();

    float2 r = unpack16<SUM>(ALGO == ALGO_TILE8 ? aux : acc);
    if (ALGO == ALGO_SEQ && FMA && SUM != SUM16_BF16) r = make_float2(add_rn(r.x, 0.0f), add_rn(r.y, 0.0f));      // conversions round to -0 as well
    if (!computes || gm >= p.M) return;
    float* dst = C + (int64_t)gm * p.N + gn;
    if (gn < p.N) dst[0] = r.x;
    if (gn + 1 < p.N) dst[1] = r.y;
}

template <int ALGO, int SUM, int PROD, int CONV>
int launch_thin_one(const MmParams& p, int64_t batch, cudaStream_t st) {
    constexpr bool kNosub = PROD != PROD16_FUSED && settles16(SUM, PROD);
    const dim3 grid((unsigned)((p.N + (int64_t)TBN - 1) / TBN), (unsigned)((p.M + (int64_t)TBM - 1) / TBM), (unsigned)batch);
    if (grid.y > 65535u) { set_error("float_mm: M=%d has more than 65535 row tiles of %d", p.M, TBM); return MPT_ERR_INVALID_ARGUMENT; }
    if (kNosub && p.nosub) mm16_thin_kernel<ALGO, SUM, PROD, kNosub, CONV><<<grid, TTHREADS + stagers(CONV), 0, st>>>(p);
    else mm16_thin_kernel<ALGO, SUM, PROD, false, CONV><<<grid, TTHREADS + stagers(CONV), 0, st>>>(p);
    return check_launch("float_mm");
}
template <int ALGO, int CONV>
int launch_thin(const MmParams& p, int64_t batch, cudaStream_t st) {
    switch (p.kind16) {
#define MPT_CASE16(S, P) case kind16(S, P): return launch_thin_one<ALGO, S, P, CONV>(p, batch, st);
        MPT_KINDS16(MPT_CASE16)
#undef MPT_CASE16
    }
    return no_kind16(p);
}

}  // namespace

int launch_mm16_thin(int algo, const MmParams& p, int64_t batch, cudaStream_t st) {
    return algo == ALGO_SEQ ? launch_thin<ALGO_SEQ, CONV_NONE>(p, batch, st) : launch_thin<ALGO_TILE8, CONV_NONE>(p, batch, st);
}

int launch_conv16_wgrad_thin(int algo, const MmParams& p, cudaStream_t st) {
    return algo == ALGO_SEQ ? launch_thin<ALGO_SEQ, CONV_WGRAD>(p, 1, st) : launch_thin<ALGO_TILE8, CONV_WGRAD>(p, 1, st);
}

}  // namespace mpt
