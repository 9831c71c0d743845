// Column chains with 16-bit running sums: layernorm parameter gradients and mpt_qsum_rows where the accumulation format is
// e5m10 or e8m7 (colsum_kernel in reduce.cu is the general form), and column sums over many columns in any format.
//
// out[c] = the running sum acc = Q(acc + v[r]) over the rows in order.  The chain is serial by definition, so its time is the
// rows times the latency of one rounded addition.  The value after each step is a binary16 (bfloat16) value, and the
// conversion instruction is the rounding: acc stays in 16 bits, add.f32 with a 16-bit operand gives RN32(acc + v), cvt.rn
// rounds it, two dependent instructions where the FP32 form has five (add, exponent mask, clamp, two FMAs).  Measured on a
// B200: 12.5 clocks per row against 56 (8192 x 768 column sums 232 -> 58 us, 200704 x 64 5.6 -> 1.28 ms; without
// subnormals, where the FP32 form walked the exact caster, 42.6 -> 1.46 ms).
//
// cvt.rn covers every sum an e5m10 chain can meet but an overflow in a saturating format, and every normal one of an e8m7
// chain; below the smallest normal value the reference rounds e8m7 in its own way, and flushes in formats without
// subnormals.  A tile of rows is added on trust; if it ends in an infinity or NaN (which no later addition removes), or
// met a nonzero sum below the smallest normal value where that matters, the lane adds the tile again on the exact caster.
#include "async_copy.cuh"
#include "reduce.cuh"

namespace mpt {
namespace {

constexpr int kCols = 8;              // columns per CTA: one 32-byte sector per row, so that few columns still fill SMs
constexpr int kTile = 192;            // rows per tile
constexpr int kStages = 3;            // tiles in flight from global memory: one tile's chain is longer than a trip to HBM
// Warp w runs on scheduler w % 4.  Warp 3 walks the chains and has its scheduler to itself (warp 7 only keeps the barriers'
// count): beside producers' bursts of arithmetic a layernorm row took 21 clocks instead of 14.
constexpr int kThreads = 256, kChainWarp = 3;
constexpr int kAdders = 32 * 6;       // producer threads: warps 0, 1, 2, 4, 5, 6 load tiles and work out their addends
constexpr int kPer = kTile * kCols / kAdders;      // elements per producer thread and tile
constexpr int kRunRows = 32;         // rows whose addends are loaded ahead
constexpr uint32_t kMinNormal16 = (uint32_t)(127 - 14) << 23;

enum Round16 : int { R16_ANY = 0, R16_F16 = 1, R16_BF16 = 2 };

__device__ __forceinline__ uint32_t mag(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }

// The running sum.  BF16: its bits are the upper half of the float.
template <bool BF16> struct Chain16 {
    uint32_t h;       // binary16 pattern, or the float's bits
    __device__ __forceinline__ float value() const {
        if (BF16) return __uint_as_float(h);
        float f;
        asm("{.reg .b16 l, g; mov.b32 {l, g}, %1; cvt.f32.f16 %0, l;}" : "=f"(f) : "r"(h));
        return f;
    }
    __device__ __forceinline__ void set(float v) {
        if (BF16) h = __float_as_uint(v);
        else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(0.0f), "f"(v));
    }
    // one rounded addition; returns the sum before its rounding
    __device__ __forceinline__ float add(float v) {
        float x;
        if (BF16) {
            x = __fadd_rn(__uint_as_float(h), v);
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(x), "f"(0.0f));
        } else {
            asm("{.reg .b16 l, g; mov.b32 {l, g}, %1; add.rn.f32.f16 %0, l, %2;}" : "=f"(x) : "r"(h), "f"(v));
            asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(0.0f), "f"(x));
        }
        return x;
    }
    __device__ __forceinline__ bool finite() const { return BF16 ? (h & 0x7F800000u) != 0x7F800000u : (h & 0x7C00u) != 0x7C00u; }
};

// A value rounded for the producers: the conversion where it is the format's rounding (see above), the caster elsewhere.
template <int R>
__device__ __forceinline__ float round_value(float x, const Caster& q) {
    if (R == R16_F16) {
        uint32_t h;
        float y;
        asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(0.0f), "f"(x));
        asm("{.reg .b16 l, g; mov.b32 {l, g}, %1; cvt.f32.f16 %0, l;}" : "=f"(y) : "r"(h));
        return __fadd_rn(y, 0.0f);                // -0 becomes +0, as in the caster
    }
    if (R == R16_BF16 && mag(x) - 1u >= 0x007FFFFFu) {
        uint32_t h;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(x), "f"(0.0f));
        return __uint_as_float(h);
    }
    return q(x);
}

// MODE 0: layernorm parameter gradients, chain A = Qmul(Qmul(Qacc(x - mean) * rstd) * dy) -> out0 in lanes 0-7 of the chain warp
// and chain B = dy -> out1 in lanes 8-15.  MODE 1: column sums of `in`, lanes 0-7.  ROUND: how the producers round.
// WATCH: nonzero sums below the smallest normal value (pattern `watch`) need the exact caster.
template <int MODE, bool BF16, int ROUND, bool WATCH>
__global__ void __launch_bounds__(kThreads) chain16_kernel(const float* __restrict__ in, const float* __restrict__ gout,
                                                           const float* __restrict__ mean, const float* __restrict__ rstd,
                                                           float* __restrict__ out0, float* __restrict__ out1, RowGeom g, Caster facc,
                                                           Caster fmul, uint32_t watch) {
    constexpr int W = MODE == 0 ? 2 * kCols : kCols;       // addends per row
    // MODE 0: two tiles of addends, then per stage what every producer thread loaded (x, dy, mean, rstd for its rows).
    // MODE 1: the addends are the loaded values, kStages tiles of them.
    extern __shared__ __align__(16) float smem[];
    float* raw = smem + 2 * kTile * W;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t ntiles = (g.rows + kTile - 1) / kTile;
    const bool producer = (warp & 3) != kChainWarp, chain = warp == kChainWarp;
    const int adder = threadIdx.x - (warp > kChainWarp ? 32 : 0);
    const int pc = adder & (kCols - 1), pr = adder / kCols;      // producer: its column and first row of a tile
    const int64_t pcol = (int64_t)blockIdx.x * kCols + pc;
    const bool pcol_ok = pcol < g.channel;

    auto fetch = [&](int64_t t) {
        if (t < ntiles) {
            const int s = (int)(t % kStages);
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int lr = pr + u * (kTile / kPer);
                const int64_t row = t * kTile + lr;
                const bool rok = row < g.rows, ok = rok && pcol_ok;
                const int64_t idx = ok ? row_base(g, row) + pcol * g.inner : 0;
                if (MODE == 1) cp_async4(smem + (s * kTile + lr) * W + pc, in + idx, ok ? 4 : 0);
                else {
                    float* r = raw + (s * 4 * kPer + u) * kAdders + adder;
                    cp_async4(r, in + idx, ok ? 4 : 0);
                    cp_async4(r + kPer * kAdders, gout + idx, ok ? 4 : 0);
                    cp_async4(r + 2 * kPer * kAdders, mean + (rok ? row : 0), rok ? 4 : 0);
                    cp_async4(r + 3 * kPer * kAdders, rstd + (rok ? row : 0), rok ? 4 : 0);
                }
            }
        }
        cp_async_commit();
    };
    // a producer thread reads back only what it copied itself
    auto fill = [&](int64_t t) {
        if (MODE == 1 || t >= ntiles) return;
        const int s = (int)(t % kStages);
        float* vals = smem + (int)(t & 1) * kTile * W;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const float* r = raw + (s * 4 * kPer + u) * kAdders + adder;
            const float dy = r[kPer * kAdders];
            const float xhat = round_value<ROUND>(__fmul_rn(round_value<ROUND>(__fsub_rn(r[0], r[2 * kPer * kAdders]), facc), r[3 * kPer * kAdders]), fmul);
            float* v = vals + (pr + u * (kTile / kPer)) * W;
            v[pc] = round_value<ROUND>(__fmul_rn(xhat, dy), fmul);
            v[kCols + pc] = dy;
        }
    };

    Chain16<BF16> acc;
    acc.h = 0u;
    if (producer) {
#pragma unroll
        for (int s = 0; s < kStages - 1; ++s) fetch(s);
        cp_async_wait<kStages - 2>();
        fill(0);
    }
    __syncthreads();
    for (int64_t t = 0; t < ntiles; ++t) {
        if (producer) {
            fetch(t + kStages - 1);          // into the stage the barrier before has freed
            cp_async_wait<kStages - 2>();
            fill(t + 1);
        } else if (chain) {
            const int64_t left = g.rows - t * kTile;
            const int nrows = left < kTile ? (int)left : kTile;
            const float* v = smem + (MODE == 1 ? (int)(t % kStages) : (int)(t & 1)) * kTile * W + (lane & (W - 1));
            const Chain16<BF16> before = acc;
            bool small = false;
            const auto step = [&](float addend) {
                const float x = acc.add(addend);
                if (WATCH) small |= mag(x) - 1u < watch - 1u;
            };
            float next[kRunRows];
#pragma unroll
            for (int u = 0; u < kRunRows; ++u) next[u] = v[u * W];
            int r = 0;
#pragma unroll 1
            for (; r + kRunRows <= nrows; r += kRunRows) {
                float cur[kRunRows];
#pragma unroll
                for (int u = 0; u < kRunRows; ++u) cur[u] = next[u];
                const float* ahead = v + (r + kRunRows < kTile ? r + kRunRows : 0) * W;
#pragma unroll
                for (int u = 0; u < kRunRows; ++u) next[u] = ahead[u * W];
#pragma unroll
                for (int u = 0; u < kRunRows; ++u) step(cur[u]);
            }
#pragma unroll 1
            for (; r < nrows; ++r) step(v[r * W]);
            if (!acc.finite() || (WATCH && small)) {
                float a = before.value();
#pragma unroll 1
                for (r = 0; r < nrows; ++r) a = facc(__fadd_rn(a, v[r * W]));
                acc.set(a);
            }
        }
        __syncthreads();
    }
    if (chain && lane < W) {
        const int64_t col = (int64_t)blockIdx.x * kCols + (lane & (kCols - 1));
        float r = acc.value();
        if (!BF16 && !WATCH) r = __fadd_rn(r, 0.0f);          // the conversion keeps the sign of a zero, the caster does not
        if (col < g.channel) (lane < kCols ? out0 : out1)[col] = r;
    }
}

// Few rows, many columns (a batch of weight or position gradients): one thread per column, the columns' loads coalesced
// and eight rows in flight.  Any format.
__global__ void __launch_bounds__(256) wide_colsum_kernel(const float* __restrict__ in, float* __restrict__ out, RowGeom g, SeqAdder seq) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.channel) return;
    float acc = 0.0f;
    int64_t r = 0;
    for (; r + 8 <= g.rows; r += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = in[(r + u) * g.channel + c];
        acc = seq.add(acc, v);
    }
    for (; r < g.rows; ++r) {
        const float v[1] = {in[r * g.channel + c]};
        acc = seq.add(acc, v);
    }
    out[c] = acc;
}

bool is_float(const Caster& c, int man, int exp) { return c.any.kind == FMT_FLOAT && c.any.fp.man == man && c.any.fp.exp == exp; }

}  // namespace

// The accumulation format's chain has the 16-bit form.
bool chain16_ok(const Caster& acc) { return is_float(acc, 10, 5) || is_float(acc, 7, 8); }

int launch_chain16(int mode, const float* in, const float* gout, const float* mean, const float* rstd, float* out0, float* out1,
                   const RowGeom& g, const Caster& facc, const Caster& fmul, cudaStream_t st, const char* who) {
    const bool bf16 = is_float(facc, 7, 8);
    const uint32_t watch = bf16 ? 0x00800000u : facc.any.fp.sub ? 0u : kMinNormal16;
    // the producers' roundings by conversion: no saturation to undo, and for e5m10 no flushing
    const bool plain = !facc.any.fp.sat && !fmul.any.fp.sat;
    const bool r16 = plain && facc.any.fp.sub && fmul.any.fp.sub && is_float(facc, 10, 5) && is_float(fmul, 10, 5);
    const bool rb16 = plain && bf16 && is_float(fmul, 7, 8);
    const unsigned grid = (unsigned)((g.channel + kCols - 1) / kCols);
    const size_t smem = sizeof(float) * (mode == 0 ? 2 * kTile * 2 * kCols + kStages * 4 * kPer * kAdders : kStages * kTile * kCols);
    const auto run = [&](auto kern) -> int {
        const cudaError_t e = smem > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
        if (e != cudaSuccess) { set_error("%s: cudaFuncSetAttribute: %s", who, cudaGetErrorString(e)); return MPT_ERR_CUDA; }
        kern<<<grid, kThreads, smem, st>>>(in, gout, mean, rstd, out0, out1, g, facc, fmul, watch);
        return check_launch(who);
    };
    if (mode == 1) return bf16 ? run(chain16_kernel<1, true, R16_ANY, true>) : watch ? run(chain16_kernel<1, false, R16_ANY, true>)
                                                                                   : run(chain16_kernel<1, false, R16_ANY, false>);
    if (bf16) return rb16 ? run(chain16_kernel<0, true, R16_BF16, true>) : run(chain16_kernel<0, true, R16_ANY, true>);
    if (watch) return run(chain16_kernel<0, false, R16_ANY, true>);
    return r16 ? run(chain16_kernel<0, false, R16_F16, false>) : run(chain16_kernel<0, false, R16_ANY, false>);
}

// Column sums (mode 1): which kernel?  Measured in us, inputs not in L2, general chain against the 16-bit chain:
//   e5m10:                 8192 columns x 1024 rows 38, 30; 12,288 x 1024: 42, 41 (e8m7 46); 16,384 x 1024: 44, 51; x 128: 10, 13
//   without subnormals:    16,384 x 128 rows 34, 37 (e8m7 12); x 256: 64, 58; x 1024: 245, 99 (e8m7 57)
// and the general chain against a thread per column (inputs in L2 where they fit):
//   e5m10:                 32,768 x 128 rows 15, 10; x 1024: 76, 107; 65,536 x 1024: 123, 113; 786,432 x 8: 50, 10
//   without subnormals:    32,768 x 1024 rows 469, 275; fp32 sums: 197, 161
// The 16-bit chain's short steps pay while columns are too few to fill the SMs.  A thread per column wants enough columns to
// cover the trips to memory, or few rows; against the general chain's exact casters it wins at any number of rows.
bool chain16_wins(const RowGeom& g, const Caster& acc) {
    return g.channel <= 8192 || (!acc.any.fp.sub && g.rows >= (acc.any.fp.exp == 8 ? 32 : 256));
}
bool wide_colsum_ok(const RowGeom& g, const SeqAdder& seq) {
    return g.inner == 1 && (g.channel >= 65536 || (g.channel >= 32768 && (g.rows <= 128 || !seq.chain_ok)));
}
int launch_wide_colsum(const float* in, float* out, const RowGeom& g, const SeqAdder& seq, cudaStream_t st, const char* who) {
    wide_colsum_kernel<<<(unsigned)((g.channel + 255) / 256), 256, 0, st>>>(in, out, g, seq);
    return check_launch(who);
}

}  // namespace mpt
