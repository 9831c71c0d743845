// The per-MAC rounded GEMM for formats whose values fit a 16-bit register: C = A x B, every product and every partial
// sum rounded to its format, with the same operations in the same order as mm_kernel (gemm_kernel.cuh) and the same bits.
//
// mm_kernel rounds with two FP32 operations and one or two integer ones per value, and is bound by the 128 FP32 + INT32
// lane operations an SM retires per clock: 9 such slots per MAC.  When the add format is e5m10 or e8m7, its values are
// binary16 / bfloat16 values, and the hardware's own 16-bit addition IS the rounded addition; when it is e5m2 or e4m3,
// its values are binary16 values and the conversion instructions round to it.  So the running sums, which the caller
// has asked to be rounded to that format after every step anyway, live in registers of that width, two outputs to a
// register, and a MAC pair costs one FMUL2, one or two conversions and one HADD2:
//
//   product   p = RN32(a * b) as in mm_kernel (the operands stay 32 bits), then rounded straight from 32 bits to the
//             multiply format by cvt.rn (e5m2, e4m3, e5m10, e8m7): one rounding, the one mm_kernel does.
//   sum       mm_kernel computes Q(RN32(acc + p)).  RN32 before Q changes nothing: for operands of at most p bits,
//             rounding a sum to q >= 2p + 2 bits first is harmless (Figueroa, "When is double rounding innocuous?",
//             SIGNUM 1995), and 24 >= 2 * 11 + 2.  So Q(acc + p) is one HADD2 for e5m10 and e8m7.  For e5m2 and e4m3
//             (p <= 4 bits, 11 >= 2p + 2) it is HADD2 and a conversion; that needs products of no more bits than sums.
//   fused     acc is widened to 32 bits (exact), FFMA2 gives RN32(a * b + acc), one conversion rounds it.
//
// All of it holds while nothing leaves the formats' finite ranges, which make_plan and the per-group check of the running
// sums establish exactly as in mm_kernel; a group that fails, or a batch entry without a plan, is computed in 32 bits on
// the exact casters, and its sums are packed again (they are add-format values, infinities and NaN included).
// A zero that mm_kernel would make +0 can be -0 here inside a group; sums start at +0, where x + -0 = x, so no result
// changes.  Only sums that flush (formats without subnormals, sum_can_settle16) are ever -0 themselves; they keep every
// sign and walk the padding as the reference does.
//
// Measured in isolation on one B200 (the MAC loop alone, 1965 MHz): e4m3 products into e5m10 sums 13.8 TMAC/s against
// 4.2 for the FP32 form, e5m2 into e5m2 8.2, e5m2 into e8m7 8.4, e8m7 into e8m7 14.8, fused e8m7 13.2 and e5m10 11.5 (6.9),
// compensated 6.9.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "gemm_kernel.cuh"

namespace mpt {

// ---- 16-bit pair primitives ----------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b) { uint32_t r; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
__device__ __forceinline__ uint32_t b2_add(uint32_t a, uint32_t b) { uint32_t r; asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t b2_fma(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
__device__ __forceinline__ uint32_t f2_to_h2(float2 v) { uint32_t r; asm("cvt.rn.f16x2.f32 %0, %2, %1;" : "=r"(r) : "f"(v.x), "f"(v.y)); return r; }
__device__ __forceinline__ uint32_t f2_to_b2(float2 v) { uint32_t r; asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(r) : "f"(v.x), "f"(v.y)); return r; }
__device__ __forceinline__ float2 h2_to_f2(uint32_t v) {
    float2 r;
    asm("{.reg .b16 l, h; mov.b32 {l, h}, %2; cvt.f32.f16 %0, l; cvt.f32.f16 %1, h;}" : "=f"(r.x), "=f"(r.y) : "r"(v));
    return r;
}
__device__ __forceinline__ float2 b2_to_f2(uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u)); }
// fp32 pair -> e5m2 / e4m3 pair (nearest even, subnormals) -> the same values as binary16
__device__ __forceinline__ uint32_t f2_round_e5m2(float2 v) {
    uint32_t r;
    asm("{.reg .b16 t; cvt.rn.satfinite.e5m2x2.f32 t, %2, %1; cvt.rn.f16x2.e5m2x2 %0, t;}" : "=r"(r) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ uint32_t f2_round_e4m3(float2 v) {
    uint32_t r;
    asm("{.reg .b16 t; cvt.rn.satfinite.e4m3x2.f32 t, %2, %1; cvt.rn.f16x2.e4m3x2 %0, t;}" : "=r"(r) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ uint32_t h2_round_e5m2(uint32_t v) {
    uint32_t r;
    asm("{.reg .b16 t; cvt.rn.satfinite.e5m2x2.f16x2 t, %1; cvt.rn.f16x2.e5m2x2 %0, t;}" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t h2_round_e4m3(uint32_t v) {
    uint32_t r;
    asm("{.reg .b16 t; cvt.rn.satfinite.e4m3x2.f16x2 t, %1; cvt.rn.f16x2.e4m3x2 %0, t;}" : "=r"(r) : "r"(v));
    return r;
}
// per half: the larger magnitude (signs multiply; NaN loses against a number)
__device__ __forceinline__ uint32_t h2_maxabs(uint32_t a, uint32_t b) { uint32_t r; asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t b2_maxabs(uint32_t a, uint32_t b) { uint32_t r; asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t u2_min(uint32_t a, uint32_t b) { uint32_t r; asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t u2_add(uint32_t a, uint32_t b) { uint32_t r; asm("add.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ float fma_sat(float a, float b, float c) { float r; asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }

// ---- formats ---------------------------------------------------------------------------------------------------------
// SUM16_BF16 keeps bfloat16 pairs, the others binary16 pairs.
enum Sum16 : int { SUM16_F16 = 0, SUM16_BF16 = 1, SUM16_E5M2 = 2, SUM16_E4M3 = 3 };
enum Prod16 : int { PROD16_E5M2 = 0, PROD16_E4M3 = 1, PROD16_F16 = 2, PROD16_BF16 = 3, PROD16_FUSED = 4 };
__host__ __device__ constexpr int kind16(int sum, int prod) { return sum * 8 + prod; }

// The kind of a format pair, or -1 where mm_kernel stays: formats that are none of the four, products that do not fit
// the sums' register (e8m7 or e5m10 products in bfloat16 / binary16 respectively the other way round) or carry more bits
// than an 8-bit sum format, and fused sums without subnormals (their result lands below the smallest normal value all
// the time, not only when a product does).
inline int kind16_of(const FpFmt& add, const FpFmt& mul, bool fma) {
    const auto is = [](const FpFmt& f, int man, int exp) { return f.man == man && f.exp == exp; };
    const int sum = is(add, 10, 5) ? SUM16_F16 : is(add, 7, 8) ? SUM16_BF16 : is(add, 2, 5) ? SUM16_E5M2 : is(add, 3, 4) ? SUM16_E4M3 : -1;
    if (sum < 0) return -1;
    if (fma) return (add.sub || sum == SUM16_BF16) ? kind16(sum, PROD16_FUSED) : -1;
    const int prod = is(mul, 2, 5) ? PROD16_E5M2 : is(mul, 3, 4) ? PROD16_E4M3 : is(mul, 10, 5) ? PROD16_F16 : is(mul, 7, 8) ? PROD16_BF16 : -1;
    if (prod < 0 || !add.sub != !mul.sub) return -1;
    const bool ok = sum == SUM16_F16 ? prod != PROD16_BF16 : sum == SUM16_BF16 ? prod != PROD16_F16
                  : sum == SUM16_E5M2 ? prod == PROD16_E5M2 : prod == PROD16_E4M3;
    return ok ? kind16(sum, prod) : -1;
}
// e8m7 without subnormals: the plan proves that nothing nonzero comes near 2^-126, so there is nothing to settle.
__host__ __device__ constexpr bool settles16(int sum, int prod) { return !(sum == SUM16_BF16 && (prod == PROD16_BF16 || prod == PROD16_FUSED)); }
// Formats without subnormals: can a sum of products land below the add format's smallest normal value (2^-14, e4m3 2^-6,
// e8m7 2^-126)?  A sum is a multiple of the products' smallest quantum: 2^-16 for e5m2, 2^-9 for e4m3, 2^-24 for e5m10.
__host__ __device__ constexpr bool sum_can_settle16(int sum, int prod) { return sum != SUM16_BF16 && !(sum == SUM16_F16 && prod == PROD16_E4M3); }

template <int SUM> __device__ __forceinline__ uint32_t pack16(float2 v) { return SUM == SUM16_BF16 ? f2_to_b2(v) : f2_to_h2(v); }
template <int SUM> __device__ __forceinline__ float2 unpack16(uint32_t v) { return SUM == SUM16_BF16 ? b2_to_f2(v) : h2_to_f2(v); }
// a pair of binary16 sums (already rounded once, to 11 bits) to the add format
template <int SUM> __device__ __forceinline__ uint32_t settle_sum16(uint32_t v) {
    return SUM == SUM16_E5M2 ? h2_round_e5m2(v) : SUM == SUM16_E4M3 ? h2_round_e4m3(v) : v;
}
template <int SUM> __device__ __forceinline__ uint32_t sum16(uint32_t a, uint32_t b) {
    return SUM == SUM16_BF16 ? b2_add(a, b) : settle_sum16<SUM>(h2_add(a, b));
}
// a - b
template <int SUM> __device__ __forceinline__ uint32_t diff16(uint32_t a, uint32_t b) {
    return SUM == SUM16_BF16 ? b2_fma(b, 0xBF80BF80u, a) : settle_sum16<SUM>(h2_fma(b, 0xBC00BC00u, a));
}
// fp32 pair to the add format
template <int SUM> __device__ __forceinline__ uint32_t round16(float2 v) {
    return SUM == SUM16_BF16 ? f2_to_b2(v) : SUM == SUM16_E5M2 ? f2_round_e5m2(v) : SUM == SUM16_E4M3 ? f2_round_e4m3(v) : f2_to_h2(v);
}
template <int SUM> __device__ __forceinline__ uint32_t maxabs16(uint32_t a, uint32_t b) { return SUM == SUM16_BF16 ? b2_maxabs(a, b) : h2_maxabs(a, b); }

// fp32 product pair to the multiply format, as the sums' pair type
template <int SUM, int PROD> __device__ __forceinline__ uint32_t prod16(float2 v) {
    if (PROD == PROD16_BF16) return f2_to_b2(v);
    const uint32_t h = PROD == PROD16_E5M2 ? f2_round_e5m2(v) : PROD == PROD16_E4M3 ? f2_round_e4m3(v) : f2_to_h2(v);
    return SUM == SUM16_BF16 ? f2_to_b2(h2_to_f2(h)) : h;
}

// ---- formats without subnormals ------------------------------------------------------------------------------------
// The reference rounds at the value's own exponent and settles what lands below m = 2^min_exp (nosub_settle, cast.cuh):
// in units of m, |x| < T = 1/2 - 2^-(man+3) gives 0, T <= |x| < 1/2 gives m (it rounds up to 1/2 with a mantissa field above
// one half), 1/2 <= |x| <= 3/4 gives 0, and 3/4 < |x| < 1 gives m.  Two saturating FMAs per value decide that without a
// compare: `far` is 1 outside [1/2, 3/4] (a distance of one fp32 ulp times 2^(25 - min_exp) is at least 1) and `big` is 1
// from T on; their product multiplies max(|rounded|, m), inside the addition (an FMA) where the sums are binary16.
// Both thresholds are exact: the fp32 neighbours of 1/2, 3/4 and T give exact differences, and rounding is monotone.
// 4.45 TMAC/s for e4m3 into e5m10 in isolation, against 2.9 with compares and selects.
struct Settle16 {
    float scale, centre, t_less_1;        // 2^(25 - min_exp); 0.625 m; T * scale - 1
    uint32_t min_norm;                    // m as a binary16 pair
    __host__ __device__ static Settle16 make(const FpFmt& f) {
        Settle16 s;
        union { uint32_t u; float v; } c;
        c.u = (uint32_t)(127 + 25 - f.min_exp) << 23; s.scale = c.v;
        c.u = ((uint32_t)(127 + f.min_exp - 1) << 23) | 0x200000u; s.centre = c.v;      // 1.25 * 2^(min_exp - 1)
        s.t_less_1 = 16777216.0f - (float)(1 << (22 - f.man)) - 1.0f;                    // (1/2 - 2^-(man+3)) * 2^25 - 1
        const uint32_t h = (uint32_t)(f.min_exp + 15) << 10;
        s.min_norm = h | (h << 16);
        return s;
    }
};
__device__ __forceinline__ float2 settle_keep16(const Settle16& s, float2 v) {
    const float ax = fabsf(v.x), ay = fabsf(v.y);
    const float2 far_ = make_float2(fma_sat(fabsf(add_rn(ax, -s.centre)), s.scale, -4194304.0f), fma_sat(fabsf(add_rn(ay, -s.centre)), s.scale, -4194304.0f));
    const float2 big = make_float2(fma_sat(ax, s.scale, -s.t_less_1), fma_sat(ay, s.scale, -s.t_less_1));
    return __fmul2_rn(far_, big);
}

// Where sums can land below the add format's smallest normal value, that value is the multiply format's too.
// `below` collects, per half, the smallest (|sum| pattern - 1): a nonzero sum below the smallest normal value shows there.
__device__ __forceinline__ void note_small16(uint32_t& below, uint32_t v) { below = u2_min(below, u2_add(v & 0x7FFF7FFFu, 0xFFFFFFFFu)); }
__device__ __forceinline__ bool any_small16(uint32_t below, uint32_t min_norm) {
    const uint32_t lim = (min_norm & 0xFFFFu) - 1u;
    return (below & 0xFFFFu) < lim || (below >> 16) < lim;
}

// ---- steps -------------------------------------------------------------------------------------------------------------
// One accumulation step of a pair.  PAIRED: the 32-bit operations as packed fp32x2 instructions (which want the A element
// twice in a register pair), or as two scalar ones (for threads with few outputs per A element).
template <bool PAIRED> __device__ __forceinline__ float2 mul2(float a, float2 b) {
    return PAIRED ? __fmul2_rn(make_float2(a, a), b) : make_float2(mul_rn(a, b.x), mul_rn(a, b.y));
}
template <bool PAIRED> __device__ __forceinline__ float2 fma2(float a, float2 b, float2 c) {
    return PAIRED ? __ffma2_rn(make_float2(a, a), b, c) : make_float2(fma_rn(a, b.x, c.x), fma_rn(a, b.y, c.y));
}
// `first`: the sum starts from zero, so it is the product itself (an add-format value) and needs no addition.
template <int SUM, int PROD, bool NOSUB, bool PAIRED>
__device__ __forceinline__ uint32_t step16(uint32_t s, float a, float2 b, bool first, const Settle16& ns, uint32_t& below) {
    if (PROD == PROD16_FUSED) return first ? round16<SUM>(mul2<PAIRED>(a, b)) : round16<SUM>(fma2<PAIRED>(a, b, unpack16<SUM>(s)));
    const float2 q = mul2<PAIRED>(a, b);
    if (!NOSUB) {
        const uint32_t v = prod16<SUM, PROD>(q);
        return first ? v : sum16<SUM>(s, v);
    }
    const float2 keep = settle_keep16(ns, q);
    const uint32_t r = h2_maxabs(PROD == PROD16_E5M2 ? f2_round_e5m2(q) : PROD == PROD16_E4M3 ? f2_round_e4m3(q) : f2_to_h2(q), ns.min_norm);
    if (SUM == SUM16_BF16) {
        const uint32_t v = f2_to_b2(__fmul2_rn(h2_to_f2(r), keep));
        return first ? v : b2_add(s, v);
    }
    const uint32_t k2 = f2_to_h2(keep);
    s = first ? h2_fma(r, k2, 0u) : settle_sum16<SUM>(h2_fma(r, k2, s));       // + 0: a sum from zero is never -0
    if (sum_can_settle16(SUM, PROD) && !first) note_small16(below, s);
    return s;
}

// Eight steps from slab row kbase for the thread's TM x 4 outputs.  START: the sums start from zero.  Returns true when a
// sum without subnormals has met a value that needs settling: the caller discards the sums and redoes the group on the
// exact casters.
template <int SUM, int PROD, bool START, bool NOSUB>
__device__ __forceinline__ bool group16(uint32_t (&acc)[TM][2], const float* As, const float* Bs, int kbase, int ty, int tx, const Settle16& ns) {
    uint32_t below = 0xFFFFFFFFu;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float4 av[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(As + (ty + 16 * i) * AS_LD + kbase + 4 * h);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 bv = *reinterpret_cast<const float4*>(Bs + (kbase + 4 * h + j) * BN + tx * 4);
            const bool first = START && h == 0 && j == 0;
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float a = j == 0 ? av[i].x : j == 1 ? av[i].y : j == 2 ? av[i].z : av[i].w;
                acc[i][0] = step16<SUM, PROD, NOSUB, true>(acc[i][0], a, make_float2(bv.x, bv.y), first, ns, below);
                acc[i][1] = step16<SUM, PROD, NOSUB, true>(acc[i][1], a, make_float2(bv.z, bv.w), first, ns, below);
            }
        }
    }
    return NOSUB && sum_can_settle16(SUM, PROD) && any_small16(below, ns.min_norm);
}

// Eight compensated steps (kahan_fast2 in gemm_kernel.cuh, on pairs): acc = running sums, nc = negated compensation terms.
template <int SUM, int PROD>
__device__ __forceinline__ void kahan_group16(uint32_t (&acc)[TM][2], uint32_t (&nc)[TM][2], const float* As, const float* Bs, int kbase, int ty, int tx) {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        float4 av[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(As + (ty + 16 * i) * AS_LD + kbase + 4 * h);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 bv = *reinterpret_cast<const float4*>(Bs + (kbase + 4 * h + j) * BN + tx * 4);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float a = j == 0 ? av[i].x : j == 1 ? av[i].y : j == 2 ? av[i].z : av[i].w;
                const float2 a2 = make_float2(a, a);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float2 b2 = c == 0 ? make_float2(bv.x, bv.y) : make_float2(bv.z, bv.w);
                    const uint32_t s = acc[i][c];
                    const uint32_t y = PROD == PROD16_FUSED ? round16<SUM>(__ffma2_rn(a2, b2, unpack16<SUM>(nc[i][c])))
                                                            : sum16<SUM>(prod16<SUM, PROD>(__fmul2_rn(a2, b2)), nc[i][c]);
                    const uint32_t t = sum16<SUM>(s, y);
                    nc[i][c] = diff16<SUM>(y, diff16<SUM>(t, s));
                    acc[i][c] = t;
                }
            }
        }
    }
}

// A magnitude limit as a 16-bit pattern of the sums' type, rounded down; 0 (which no sum is below) where there is none.
template <int SUM>
__device__ __forceinline__ uint32_t limit16(float limit) {
    const float l = fmaxf(limit, 0.0f);
    return SUM == SUM16_BF16 ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rd(l)) : (uint32_t)__half_as_ushort(__float2half_rd(l));
}
// Largest |x| of the thread's pairs is below `lim` (a 16-bit pattern of the sums' type, itself not above the limit)?
template <int SUM>
__device__ __forceinline__ bool all_below16(const uint32_t (&v)[TM][2], uint32_t lim) {
    uint32_t m = v[0][0];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c) m = maxabs16<SUM>(m, v[i][c]);
    m &= 0x7FFF7FFFu;
    return max(m & 0xFFFFu, m >> 16) < lim;
}
template <int SUM>
__device__ __forceinline__ void unpack_all16(float (&f)[TM][TN], const uint32_t (&v)[TM][2]) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const float2 lo = unpack16<SUM>(v[i][0]), hi = unpack16<SUM>(v[i][1]);
        f[i][0] = lo.x; f[i][1] = lo.y; f[i][2] = hi.x; f[i][3] = hi.y;
    }
}
template <int SUM>
__device__ __forceinline__ void pack_all16(uint32_t (&v)[TM][2], const float (&f)[TM][TN]) {
#pragma unroll
    for (int i = 0; i < TM; ++i) { v[i][0] = pack16<SUM>(make_float2(f[i][0], f[i][1])); v[i][1] = pack16<SUM>(make_float2(f[i][2], f[i][3])); }
}

__device__ __forceinline__ bool any_minus_zero16(const uint32_t (&v)[TM][2]) {
    uint32_t hit = 0u;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c) hit |= ((v[i][c] & 0xFFFFu) == 0x8000u || (v[i][c] >> 16) == 0x8000u) ? 1u : 0u;
    return hit != 0u;
}
__device__ __forceinline__ void negate_all(float (&f)[TM][TN]) {      // zeros become +0
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) f[i][j] = add_rn(0.0f, -f[i][j]);
}

// ---- entries without a plan ----------------------------------------------------------------------------------------------
// Operands that rule the range check out (an infinity or NaN, products or sums that may pass a format's range, as N(0,1) data in
// e4m3 sums do) take 32-bit sums and the FP-pipe rounding.  Bound: the ALU pipe.  A rounding in its whole-domain form costs
// nine ALU operations, of which six only find overflow; so a group is rounded without them, the largest magnitude that went
// in is kept, and rows of a group with one that the short form does not cover are done again in the whole-domain form.  1024^3 with
// one infinity, e5m10: 1.00 ms against 5.9 with the whole-domain form in a call per step (2.0 on 16-row tiles); 768 x 1024 x 768
// e4m3 sums of N(0,1): 0.45 against 3.0 (1.2 on 16-row tiles).
struct ShortRn {
    FastRn r;
    uint32_t lim;             // smallest |x| pattern that is not covered
    __device__ __forceinline__ static ShortRn make(const FullRn& f) { return ShortRn{f.fast, min(f.ovf_from, f.exact_from)}; }
};
// What went into a rounding: the largest |x| pattern and, for 8-bit exponents, the smallest (|x| pattern - 1), where fp32
// denormals show, which those formats treat specially.  Zero is covered: a sum from +0 is never -0, and the sign of a
// product that is zero does not matter to it.  A fused sum can underflow to -0, so there zero counts as a denormal.
template <bool EIGHT, bool FMA> struct Seen {
    uint32_t top = 0u, low = 0xFFFFFFFFu;
    __device__ __forceinline__ float round(const ShortRn& q, float x) {
        const uint32_t a = __float_as_uint(x) & 0x7FFFFFFFu;
        top = max(top, a);
        if (EIGHT) low = min(low, FMA ? a : a - 1u);
        return q.r(x);
    }
    __device__ __forceinline__ bool covered(const ShortRn& q) const { return top < q.lim && (!EIGHT || low >= (FMA ? 0x00800000u : 0x007FFFFFu)); }
};
// `nk` steps of R rows (`row` floats apart in the A slab) by C columns of outputs.  False: the sums are not to be used.
template <bool FMA, bool EIGHT, int R, int C>
__device__ __forceinline__ bool short_steps(float (&acc)[R][C], const float* a, int row, const float* b, int ldb, int nk, const ShortRn& qa,
                                            const ShortRn& qm) {
    Seen<EIGHT, FMA> sa, sm;
#pragma unroll 1
    for (int k = 0; k < nk; ++k) {
        float bv[C];
#pragma unroll
        for (int j = 0; j < C; j += 2) { const float2 t = *reinterpret_cast<const float2*>(b + k * ldb + j); bv[j] = t.x; bv[j + 1] = t.y; }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float av = a[i * row + k];
#pragma unroll
            for (int j = 0; j < C; ++j)
                acc[i][j] = sa.round(qa, FMA ? fma_rn(av, bv[j], acc[i][j]) : add_rn(acc[i][j], sm.round(qm, mul_rn(av, bv[j]))));
        }
    }
    return sa.covered(qa) && (FMA || sm.covered(qm));
}

// The thread's outputs of one batch entry without a plan.  EIGHT: a format has 8 exponent bits.
template <int ALGO, bool FMA, bool EIGHT>
__device__ __forceinline__ void exact_tile16(const MmParams* pp, float* smem, int64_t batch, int m0, int n0) {
    const MmParams& p = *pp;
    float* As = smem;
    float* Bs = smem + STAGES * SMEM_A;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const float* A = p.a + batch * p.stride_a;
    const float* B = p.b + batch * p.stride_b;
    float* C = p.c + batch * p.stride_c;
    const int ksteps = (ALGO == ALGO_SEQ || (p.resume & MM_MORE)) ? p.K : p.K + 8 - p.K % 8;
    const int ntiles = (ksteps + BK - 1) / BK;
    const ShortRn qa = ShortRn::make(p.wadd), qm = ShortRn::make(p.wmul);
    constexpr int R = 2;                 // rows at once: eight independent chains

    float acc[TM][TN], outer[TM][TN];    // running (inner) sums; outer sums of the CUDA order
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = outer[i][j] = 0.0f;
    if (p.resume & MM_FROM_C) {
        if (ALGO == ALGO_TILE8) load_c(p, C, m0, n0, ty, tx, outer); else load_c(p, C, m0, n0, ty, tx, acc);
    }
    auto stage = [&](int s, int k0) {
        if (p.vec) load_tiles<true>(p, A, B, As + s * SMEM_A, Bs + s * SMEM_B, m0, n0, k0, tid);
        else load_tiles<false>(p, A, B, As + s * SMEM_A, Bs + s * SMEM_B, m0, n0, k0, tid);
    };
#pragma unroll 1
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < ntiles) stage(s, s * BK);
        cp_async_commit();
    }
    // running sums of 8-bit-exponent formats that are -0 (continued from one, or flushed to one where there are no subnormals) keep
    // the sign, which the short form does not
    const bool never = EIGHT && ((p.resume & MM_FROM_C) || !p.whole_ok);
    uint32_t missed = 0u;                // bit i: rows i of the thread were not covered last time; tried again every eighth group
#pragma unroll 1
    for (int t = 0; t < ntiles; ++t) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        const int nt = t + STAGES - 1;
        if (nt < ntiles) stage(nt % STAGES, nt * BK);
        cp_async_commit();
        const float* a = As + (t % STAGES) * SMEM_A + ty * AS_LD;
        const float* b = Bs + (t % STAGES) * SMEM_B + tx * 4;
        const int nk_tile = min(ksteps - t * BK, BK);
#pragma unroll 1
        for (int k0 = 0; k0 < nk_tile; k0 += 8) {
            const int nk = min(nk_tile - k0, 8);
            const bool again = t % 2 == 0 && k0 == 0;
#pragma unroll
            for (int i = 0; i < TM; i += R) {
                float v[R][TN];
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int j = 0; j < TN; ++j) v[r][j] = ALGO == ALGO_TILE8 ? 0.0f : acc[i + r][j];
                const float* ai = a + 16 * i * AS_LD + k0;
                bool done = !never && (again || !(missed >> i & 1u));
                if (done) done = short_steps<FMA, EIGHT, R, TN>(v, ai, 16 * AS_LD, b + k0 * BN, BN, nk, qa, qm);
                missed &= ~(1u << i);
                if (!done) {
                    missed |= 1u << i;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        float4 e = ALGO == ALGO_TILE8 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : make_float4(acc[i + r][0], acc[i + r][1], acc[i + r][2], acc[i + r][3]);
#pragma unroll 1
                        for (int k = 0; k < nk; ++k)
                            e = mac_exact4<FMA>(e, a[16 * (i + r) * AS_LD + k0 + k], *reinterpret_cast<const float4*>(b + (k0 + k) * BN), pp);
                        v[r][0] = e.x; v[r][1] = e.y; v[r][2] = e.z; v[r][3] = e.w;
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        if (ALGO != ALGO_TILE8) { acc[i + r][j] = v[r][j]; continue; }
                        const float x = add_rn(outer[i + r][j], v[r][j]);
                        Seen<EIGHT, true> seen;
                        const float y = seen.round(qa, x);
                        outer[i + r][j] = seen.covered(qa) ? y : exact_add_cold(pp, x);
                    }
            }
        }
    }
    cp_async_wait<0>();
    if (ALGO == ALGO_TILE8) store_tile<CONV_NONE>(p, C, m0, n0, ty, tx, p.vec != 0, outer);
    else store_tile<CONV_NONE>(p, C, m0, n0, ty, tx, p.vec != 0, acc);
}

// As a call, for the sequential order's 128-row tiles: inlined it has their planned loop spill.
template <int ALGO, bool FMA, bool EIGHT>
__device__ __noinline__ void exact_tile16_call(const MmParams* pp) {
    extern __shared__ __align__(16) float smem[];
    int tile_m, tile_n;
    banded_tile(tile_m, tile_n);
    exact_tile16<ALGO, FMA, EIGHT>(pp, smem, blockIdx.z, tile_m * BM, tile_n * BN);
}

// `nk` steps of a group in formats without subnormals, in 32 bits with the settling of mm_kernel: the group is within the range
// that the plan and the look at the sums establish, but a sum of it lands below the smallest normal value.  Sequential e5m2 sums
// of products that are all that small, 1024^3: 3.2 ms, with the exact casters instead 12.5 (mm_kernel alone: 2.8).
static __device__ __noinline__ float4 settle_steps4(float4 c, const float* a, const float* b, int nk, const MmParams* pp) {
    const FastRn radd = pp->radd, rmul = pp->rmul;
#pragma unroll 1
    for (int k = 0; k < nk; ++k) {
        const float av = a[k];
        const float4 v = *reinterpret_cast<const float4*>(b + k * BN);
        c.x = mac_fast<false, true>(c.x, av, v.x, radd, rmul); c.y = mac_fast<false, true>(c.y, av, v.y, radd, rmul);
        c.z = mac_fast<false, true>(c.z, av, v.z, radd, rmul); c.w = mac_fast<false, true>(c.w, av, v.w, radd, rmul);
    }
    return c;
}
__device__ __forceinline__ void settle_group16(float (&f)[TM][TN], const float* as, const float* bs, int kbase, int nk, int ty, int tx,
                                               const MmParams& p) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const float4 r = settle_steps4(make_float4(f[i][0], f[i][1], f[i][2], f[i][3]), as + (ty + 16 * i) * AS_LD + kbase,
                                       bs + kbase * BN + tx * 4, nk, &p);
        f[i][0] = r.x; f[i][1] = r.y; f[i][2] = r.z; f[i][3] = r.w;
    }
}

// ---- the kernel ------------------------------------------------------------------------------------------------------
// Tiling, staging and epilogue are mm_kernel's: 128 x 64 outputs per CTA (64 x 64 in gemm16_mid.cu), 256 threads, 8 x 4
// outputs per thread as 16 pairs, K slabs of 32 through three cp.async stages.
template <int ALGO, int SUM, int PROD, bool NOSUB, int CONV, int MINB, int TILE_ROWS = BM>
__global__ void __launch_bounds__(THREADS, MINB) mm16_kernel(const __grid_constant__ MmParams p) {
    static_assert(TILE_ROWS == BM, "one tile height per translation unit");
    constexpr bool FMA = PROD == PROD16_FUSED;
    extern __shared__ __align__(16) float smem[];
    float* As = smem;
    float* Bs = smem + STAGES * SMEM_A;
    ConvRow* crow = reinterpret_cast<ConvRow*>(smem + STAGES * (SMEM_A + SMEM_B));      // CONV_FWD: BM entries

    const int tid = threadIdx.x;
    const int ty = tid >> 4, tx = tid & 15;
    int tile_m, tile_n;
    banded_tile(tile_m, tile_n);
    const int m0 = tile_m * BM, n0 = tile_n * BN;
    const int64_t batch = blockIdx.z;
    const float* A = p.a + batch * p.stride_a;
    const float* B = p.b + batch * p.stride_b;
    float* C = p.c + batch * p.stride_c;

    const FastPlan plan = make_plan<ALGO, FMA>(p, batch);
    if (CONV == CONV_NONE && p.defer_exact && !plan.ok) return;
    // Where the second loop costs the planned one registers or time, entries without a plan redo group by group below: on the
    // sequential order's 64-row tiles (768^3 in e8m7: 82 us with it, 72 without) and for fused sums on 128-row tiles in the CUDA
    // order (96 x 1024 x 1024 x 64: 662 and 644).  Sums in e4m3, which hardly ever have a plan, always take it.
    constexpr bool kPlanned = CONV == CONV_NONE && ALGO != ALGO_KAHAN && !NOSUB &&
                              (SUM == SUM16_E4M3 || (ALGO == ALGO_TILE8 ? !(FMA && TM >= 8) : TM >= 8));
    if constexpr (kPlanned) {         // from here on there is a plan
        if (!plan.ok) {
            if constexpr (ALGO == ALGO_SEQ && TM >= 8) exact_tile16_call<ALGO, FMA, SUM == SUM16_BF16>(&p);
            else exact_tile16<ALGO, FMA, SUM == SUM16_BF16>(&p, smem, batch, m0, n0);
            return;
        }
    }
    const bool ok = kPlanned || plan.ok;
    // With a plan, the zero padding the CUDA order walks (and the last partial group of the sequential one, zero filled in
    // shared memory) adds zeros to add-format values, which changes none of them: whole groups, and only those with data.
    // Compensated sums do move under it (their compensation term is added), so they walk all of it.
    // Flushing sums can be -0, which + 0 turns into +0: the CUDA order's padding is walked too (it does that in the
    // reference), the sequential order's last partial group looks for -0 first.
    constexpr bool kFlush = NOSUB && sum_can_settle16(SUM, PROD);
    const int ksteps = ok && (ALGO == ALGO_SEQ || (ALGO == ALGO_TILE8 && !kFlush)) ? (p.K + 7) / 8 * 8
                     : (ALGO == ALGO_SEQ || (p.resume & MM_MORE)) ? p.K : p.K + 8 - p.K % 8;
    const int ntiles = (ksteps + BK - 1) / BK;
    const uint32_t lim = limit16<SUM>(plan.acc_limit), slab_lim = limit16<SUM>(plan.slab_limit);
    const Settle16 ns = Settle16::make(p.fmul);

    if (CONV == CONV_FWD) {
        fill_conv_rows(p, crow, m0, tid);
        __syncthreads();
    }

    uint32_t acc[TM][2];        // running sums (inner sums in the CUDA order)
    uint32_t aux[TM][2];        // outer sums (CUDA order), negated compensation terms (compensated sums)
#pragma unroll
    for (int i = 0; i < TM; ++i) { acc[i][0] = acc[i][1] = aux[i][0] = aux[i][1] = 0u; }
    // Continuing from C: its values are the rounded sums of the pieces before, unless the caller put something else there;
    // then the first group starts from the 32-bit values on the exact path, after which the sums are add-format values.
    bool wide_start = false;
    if (CONV == CONV_NONE && ALGO != ALGO_KAHAN && (p.resume & MM_FROM_C)) {
        float f[TM][TN];
        load_c(p, C, m0, n0, ty, tx, f);
        if (ALGO == ALGO_TILE8) pack_all16<SUM>(aux, f); else pack_all16<SUM>(acc, f);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const uint32_t u = __float_as_uint(f[i][j]);
                wide_start |= u == 0x80000000u || (f[i][j] == f[i][j] && __float_as_uint(exact_add_cold(&p, f[i][j])) != u);
            }
    }

    // a tile inside the matrix needs no bounds: one address and a constant step per thread
    const bool inside = CONV == CONV_NONE && p.vec && m0 + BM <= p.M && n0 + BN <= p.N;
    const float* a_src = A + (int64_t)(m0 + (tid >> 3)) * p.K + ((tid & 7) << 2);
    const float* b_src = B + (int64_t)(tid >> 4) * p.N + n0 + ((tid & 15) << 2);
    auto stage = [&](int s, int k0) {
        if (inside && BM >= 32 && k0 + BK <= p.K) {
            const float* a = a_src + k0;
            const float* b = b_src + (int64_t)k0 * p.N;
            float* as = As + s * SMEM_A + (tid >> 3) * AS_LD + ((tid & 7) << 2);
            float* bs = Bs + s * SMEM_B + (tid >> 4) * BN + ((tid & 15) << 2);
#pragma unroll
            for (int u = 0; u < BM / 32; ++u) cp_async16(as + 32 * u * AS_LD, a + (int64_t)(32 * u) * p.K, 16);
#pragma unroll
            for (int u = 0; u < BK / 16; ++u) cp_async16(bs + 16 * u * BN, b + (int64_t)(16 * u) * p.N, 16);
        } else if (CONV == CONV_NONE && p.vec) load_tiles<true, CONV_NONE>(p, A, B, As + s * SMEM_A, Bs + s * SMEM_B, m0, n0, k0, tid, crow);
        else load_tiles<false, CONV>(p, A, B, As + s * SMEM_A, Bs + s * SMEM_B, m0, n0, k0, tid, crow);
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < ntiles) stage(s, s * BK);
        cp_async_commit();
    }

    for (int t = 0; t < ntiles; ++t) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        {
            const int nt = t + STAGES - 1;
            if (nt < ntiles) stage(nt % STAGES, nt * BK);
            cp_async_commit();
        }
        const float* as = As + (t % STAGES) * SMEM_A;
        const float* bs = Bs + (t % STAGES) * SMEM_B;
        const int nk_tile = min(ksteps - t * BK, BK);
        // one look at the sums for the slab's four groups; where it does not suffice every group looks for itself
        const bool slab_ok = ALGO != ALGO_KAHAN && !(wide_start && t == 0) && all_below16<SUM>(ALGO == ALGO_TILE8 ? aux : acc, slab_lim);
#pragma unroll 1
        for (int g = 0; g * 8 < nk_tile; ++g) {
            const int nk = min(nk_tile - g * 8, 8);
            const bool wide = wide_start && t == 0 && g == 0;
            if (ALGO == ALGO_TILE8) {
                bool redo = !ok;
                if (ok) redo = group16<SUM, PROD, true, NOSUB>(acc, as, bs, g * 8, ty, tx, ns);
                if (redo) {
                    float f[TM][TN];
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) f[i][j] = 0.0f;
                    group_steps<FMA, false, false, true>(f, as, bs, g * 8, nk, ty, tx, p);
                    pack_all16<SUM>(acc, f);
                }
                // fold the group into the outer sum
                bool folded = false;
                if (ok && !wide && (slab_ok || all_below16<SUM>(aux, lim))) {
                    uint32_t below = 0xFFFFFFFFu, out[TM][2];
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            out[i][c] = sum16<SUM>(aux[i][c], acc[i][c]);
                            if (kFlush) note_small16(below, out[i][c]);
                        }
                    folded = !(kFlush && any_small16(below, ns.min_norm));
                    if (folded) {
#pragma unroll
                        for (int i = 0; i < TM; ++i) { aux[i][0] = out[i][0]; aux[i][1] = out[i][1]; }
                    }
                }
                if (!folded) {
                    float f[TM][TN], o[TM][TN];
                    unpack_all16<SUM>(f, acc);
                    if (wide) load_c(p, C, m0, n0, ty, tx, o); else unpack_all16<SUM>(o, aux);
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) o[i][j] = exact_add_cold(&p, add_rn(o[i][j], wide && !redo ? add_rn(f[i][j], 0.0f) : f[i][j]));
                    pack_all16<SUM>(aux, o);
                }
            } else if (ALGO == ALGO_SEQ) {
                bool redo = true;
                const int kleft = p.K - t * BK - g * 8;
                const bool in_range = ok && !wide && (slab_ok || all_below16<SUM>(acc, lim));
                if (in_range && !(kFlush && kleft < 8 && any_minus_zero16(acc))) {
                    uint32_t saved[TM][2];
                    if (kFlush) {
#pragma unroll
                        for (int i = 0; i < TM; ++i) { saved[i][0] = acc[i][0]; saved[i][1] = acc[i][1]; }
                    }
                    redo = group16<SUM, PROD, false, NOSUB>(acc, as, bs, g * 8, ty, tx, ns);
                    if (kFlush && redo) {
#pragma unroll
                        for (int i = 0; i < TM; ++i) { acc[i][0] = saved[i][0]; acc[i][1] = saved[i][1]; }
                    }
                }
                if (redo) {
                    float f[TM][TN];
                    if (wide) load_c(p, C, m0, n0, ty, tx, f); else unpack_all16<SUM>(f, acc);
                    if (kFlush && in_range) settle_group16(f, as, bs, g * 8, min(nk, kleft), ty, tx, p);
                    else group_steps<FMA, false, false, true>(f, as, bs, g * 8, min(nk, kleft), ty, tx, p);
                    pack_all16<SUM>(acc, f);
                }
            } else {        // compensated sums; the reference pads K to a multiple of 8, so every group has 8 steps
                if (ok && all_below16<SUM>(acc, lim) && all_below16<SUM>(aux, lim)) {
                    kahan_group16<SUM, PROD>(acc, aux, as, bs, g * 8, ty, tx);
                } else {
                    float f[TM][TN], o[TM][TN];
                    unpack_all16<SUM>(f, acc);
                    unpack_all16<SUM>(o, aux);
                    negate_all(o);
                    kahan_exact_group<FMA>(f, o, as, bs, g * 8, ty, tx, p);
                    negate_all(o);
                    pack_all16<SUM>(acc, f);
                    pack_all16<SUM>(aux, o);
                }
            }
        }
    }
    cp_async_wait<0>();

    float r[TM][TN];
    unpack_all16<SUM>(r, ALGO == ALGO_TILE8 ? aux : acc);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) r[i][j] = ALGO == ALGO_SEQ && FMA && SUM != SUM16_BF16 ? add_rn(r[i][j], 0.0f) : r[i][j];   // conversions round to -0 as well
    store_tile<CONV>(p, C, m0, n0, ty, tx, p.vec != 0, r);
}

// ---- launches ----------------------------------------------------------------------------------------------------------
template <int ALGO, int SUM, int PROD, int CONV, int MINB, int TILE_ROWS = BM>
int launch_one16(const MmParams& p, int64_t batch, cudaStream_t st) {
    const dim3 grid((unsigned)(((int64_t)p.N + BN - 1) / BN), (unsigned)(((int64_t)p.M + BM - 1) / BM), (unsigned)batch);
    if (grid.y > 65535u) { set_error("float_mm: M=%d has more than 65535 row tiles of %d", p.M, BM); return MPT_ERR_INVALID_ARGUMENT; }
    constexpr bool kNosub = ALGO != ALGO_KAHAN && PROD != PROD16_FUSED && settles16(SUM, PROD);
    auto kern = mm16_kernel<ALGO, SUM, PROD, false, CONV, MINB, TILE_ROWS>;
    if (kNosub && p.nosub) kern = mm16_kernel<ALGO, SUM, PROD, kNosub, CONV, MINB, TILE_ROWS>;
    const size_t smem = SMEM_BYTES + (CONV == CONV_FWD ? BM * sizeof(ConvRow) : 0);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { set_error("float_mm: cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return MPT_ERR_CUDA; }
    kern<<<grid, THREADS, smem, st>>>(p);
    return check_launch("float_mm");
}
// One case per format pair of kind16_of.
#define MPT_KINDS16(CASE)                                                                                                 \
    CASE(SUM16_F16, PROD16_E5M2) CASE(SUM16_F16, PROD16_E4M3) CASE(SUM16_F16, PROD16_F16) CASE(SUM16_F16, PROD16_FUSED)      \
    CASE(SUM16_BF16, PROD16_E5M2) CASE(SUM16_BF16, PROD16_E4M3) CASE(SUM16_BF16, PROD16_BF16) CASE(SUM16_BF16, PROD16_FUSED) \
    CASE(SUM16_E5M2, PROD16_E5M2) CASE(SUM16_E5M2, PROD16_FUSED) CASE(SUM16_E4M3, PROD16_E4M3) CASE(SUM16_E4M3, PROD16_FUSED)
inline int no_kind16(const MmParams& p) {
    set_error("float_mm: no 16-bit kernel for kind %d", p.kind16);
    return MPT_ERR_INVALID_ARGUMENT;
}
template <int ALGO, int CONV, int MINB, int TILE_ROWS = BM>
int launch_any16(const MmParams& p, int64_t batch, cudaStream_t st) {
    switch (p.kind16) {
#define MPT_CASE16(S, P) case kind16(S, P): return launch_one16<ALGO, S, P, CONV, MINB, TILE_ROWS>(p, batch, st);
        MPT_KINDS16(MPT_CASE16)
#undef MPT_CASE16
    }
    return no_kind16(p);
}

}  // namespace mpt
