// Quantised tiles (layout.cuh) as FP16 values in registers, w * 2^e with a power of two per row (row_pow.cuh) that the product takes back.
//
// Quick: one multiply-add per two values.  The integers q of a tile enter the arithmetic as they lie: a field of up to eight bits in the low
// bits of a 16-bit word IS the FP16 (subnormal) number q * 2^-24, so masking is all the conversion there is, and w = s*q - m is one fused
// multiply-add with the factors S = s * 2^(e + 24) and m * 2^e.  The power of two puts the largest S of the row below 2^15; the weights, at most 2^-2
// then, are multiples of 2^-24.  FP16 arithmetic runs at half the rate of FP32 on these SMs, so operations count: subtracting the bias of an
// integer-to-float pattern first took two per pair of values and 223 cycles of a scheduler per 128 columns of a Q4_K tile (measured alone, four
// warps); see gemm_quant_tc.cu for what it takes now.  S and m round once from exact products, the result rounds once: the same error as s and m in
// FP16 have (products of random rows with Q4_K 5.8e-4, Q6_K 3.5e-4, Q8_0 2.9e-4 relative), as long as the blocks of a row are alike.
//
// Wide: for row tiles whose blocks lie far apart (row_pow_word), and in prompts (PRECISE).  The power of two puts the largest weight of the row below 2^15, so that
// weights down to 2^-29 of it are FP16 numbers of full precision.  Q4_K and Q6_K: s and m in FP32, exact, w = s*q - m by an FP32 multiply-add, rounded
// to FP16: once, but for the 2^-24 of the multiply-add, whatever the minima.  Q8_0: q, exact, times d * 2^e.  Errors of products of random rows 2.9e-4 for all
// formats, a third less for Q4_K and Q6_K.  It costs half as many instructions again; prompts do not notice, steps of few rows do: with all tiles wide
// Llama-3-8B with 4 layers, 9 / 32 / 64 requests 448 / 542 / 713 -> 534 / 628 / 798 us a step, TinyLlama 1273 / 1431 / 1680 -> 1383 / 1531 / 1719, in Q8_0 1236 /
// 1392 / 1679 -> 1253 / 1417 / 1684.
//
// A half of a tile is 128 of its 256 columns.  Lane (g, t) of the warp gets, for each of the half's eight 16-column groups, four
// registers of two values: row g columns (4t, 4t+2), row g columns (4t+1, 4t+3), and the same of row g + 8.  That is the order in
// which a tile's bytes lie, so no value is moved; the other operand of the product keeps its columns in the same order (quant_col).
#pragma once
#include <cuda_fp16.h>

#include "bulk.cuh"
#include "layout.cuh"
#include "row_pow.cuh"
#include "tile_math.cuh"

namespace juno {

__device__ __forceinline__ uint32_t h2_sub(uint32_t v, uint32_t c) {
    __half2 r = __hsub2(*reinterpret_cast<__half2 *>(&v), *reinterpret_cast<__half2 *>(&c));
    return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t v, uint32_t c) {
    __half2 r = __hmul2(*reinterpret_cast<__half2 *>(&v), *reinterpret_cast<__half2 *>(&c));
    return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    __half2 r = __hfma2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b), *reinterpret_cast<__half2 *>(&c));
    return *reinterpret_cast<uint32_t *>(&r);
}
constexpr uint32_t kH64 = 0x54005400u;    // (64, 64): 0x5400 | n is the FP16 number 64 + n / 16 for n < 1024
constexpr uint32_t kH1024 = 0x64006400u;  // (1024, 1024): 0x6400 | n is the FP16 number 1024 + n for n < 1024
constexpr uint32_t kH1152 = 0x64806480u;  // (1152, 1152)
constexpr uint32_t kHm19 = 0x80208020u;   // (-2^-19, -2^-19): 32 in the units of a masked field
constexpr uint32_t kHm17 = 0x80808080u;   // (-2^-17, -2^-17)
constexpr float kTo24 = 16777216.f;       // 2^24

__device__ __forceinline__ float low_f32(uint32_t v) { return __low2float(*reinterpret_cast<__half2 *>(&v)); }
__device__ __forceinline__ float high_f32(uint32_t v) { return __high2float(*reinterpret_cast<__half2 *>(&v)); }
// Two values times s plus c in FP32, rounded to FP16.
__device__ __forceinline__ uint32_t fma_f16(uint32_t v, float s, float c) {
    __half2 r = __floats2half2_rn(fmaf(low_f32(v), s, c), fmaf(high_f32(v), s, c));
    return *reinterpret_cast<uint32_t *>(&r);
}

// What a lane keeps of a tile's header while it goes through the halves of the tile: rows g and g + 8.
struct TileFactors {
    uint32_t f[12];
};
// The words of rows g and g + 8 (row_pow.cuh): all that a lane keeps of their powers of two while it goes through a row tile.
struct RowPow {
    uint32_t w[2];
    __device__ __forceinline__ bool wide(int type, bool precise) const { return (w[0] & kRowWide) != 0 || (precise && type != 8); }
    // What the product has to be multiplied with.
    __device__ __forceinline__ float undo(int k, bool wide) const {
        return __uint_as_float((uint32_t)(127 + kRowPowBias + (wide ? 0 : 24) - (int)(wide ? w[k] >> 8 & 0xFFu : w[k] & 0xFFu)) << 23);
    }
    // The exponent, from the word anew for every tile: kept, what follows from it would cost registers.
    template <bool WIDE>
    __device__ __forceinline__ int exponent(int k) const {
        uint32_t v = w[k];
        asm volatile("" : "+r"(v));
        return (int)(WIDE ? v >> 8 & 0xFFu : v & 0xFFu) - kRowPowBias;
    }
    template <bool WIDE>
    __device__ __forceinline__ float f32(int k) const {
        return __uint_as_float((uint32_t)(127 + exponent<WIDE>(k)) << 23);
    }
    // As two FP16 factors: their product may exceed FP16.
    template <bool WIDE>
    __device__ __forceinline__ void f16(int k, uint32_t &a, uint32_t &b) const {
        const int e = exponent<WIDE>(k), first = min(e, 15);
        a = (uint32_t)(15 + first) * 0x04000400u;
        b = (uint32_t)(15 + e - first) * 0x04000400u;
    }
};
// Byte K of w in both halves, under the high byte of hi.
template <int K>
__device__ __forceinline__ uint32_t byte_h2(uint32_t w, uint32_t hi) {
    return __byte_perm(w, hi, 0x4040 + K * 0x101);
}

// ── Q4_K ────────────────────────────────────────────────────────────────────────────────────
__device__ __forceinline__ void q4_factors(TileFactors &F, const RowPow &P, uint32_t tile, int lane) {
    const uint32_t row = tile + 64 + (lane >> 2) * 16;
    const uint4 a = lds128(row), b = lds128(row + 128);  // (scale, scale, min, min) bytes of the sub-block pairs
    F.f[0] = a.x, F.f[1] = a.y, F.f[2] = a.z, F.f[3] = a.w, F.f[4] = b.x, F.f[5] = b.y, F.f[6] = b.z, F.f[7] = b.w;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        uint32_t pa, pb;
        P.f16<false>(k, pa, pb);
        const uint32_t d = h2_mul(h2_mul(lds32(tile + 32 * k + (lane >> 2) * 4), pa), pb);  // d | dmin
        F.f[8 + k] = __byte_perm(d, 0, 0x1010);
        F.f[10 + k] = __byte_perm(d, 0, 0x3232) ^ 0x80008000u;
    }
}
__device__ __forceinline__ void q4_half_f16(const TileFactors &F, uint32_t tile, int half, int lane, uint32_t (&o)[32]) {
    uint4 w[2];
#pragma unroll
    for (int q = 0; q < 2; q++) w[q] = lds128(tile + kQ4KQsOff + ((2 * half + q) * 32 + lane) * 16);  // words x, y belong to row g, words z, w to row g + 8
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const uint32_t w4[4] = {w[q].x, w[q].y, w[q].z, w[q].w};
#pragma unroll
        for (int row = 0; row < 2; row++) {
            const uint32_t h = F.f[4 * row + 2 * half + q], d = F.f[8 + row], dm = F.f[10 + row];
            // scale of the low-nibble sub-block, a sixteenth of that of the high-nibble one, whose fields stay in place as 16 q
            const uint32_t s0 = h2_mul(h2_sub(byte_h2<0>(h, 0x64646464u), kH1024), d), s1 = h2_mul(h2_sub(byte_h2<1>(h, 0x54545454u), kH64), d);
            const uint32_t m0 = h2_mul(byte_h2<2>(h, 0u), dm), m1 = h2_mul(byte_h2<3>(h, 0u), dm);
#pragma unroll
            for (int i = 0; i < 2; i++) {  // 16-column groups i (low nibbles) and 2 + i (high nibbles) of the quarter
                const uint32_t a = w4[2 * row + i], b = a >> 8;
                uint32_t *p = o + 16 * q + 4 * i + 2 * row;
                p[0] = h2_fma(a & 0x000F000Fu, s0, m0);
                p[1] = h2_fma(b & 0x000F000Fu, s0, m0);
                p[8] = h2_fma(a & 0x00F000F0u, s1, m1);
                p[9] = h2_fma(b & 0x00F000F0u, s1, m1);
            }
        }
    }
}
__device__ __forceinline__ void q4_wide_factors(TileFactors &F, const RowPow &P, uint32_t tile, int lane) {
    const uint32_t row = tile + 64 + (lane >> 2) * 16;
    const uint4 a = lds128(row), b = lds128(row + 128);
    F.f[0] = a.x, F.f[1] = a.y, F.f[2] = a.z, F.f[3] = a.w, F.f[4] = b.x, F.f[5] = b.y, F.f[6] = b.z, F.f[7] = b.w;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint32_t d = lds32(tile + 32 * k + (lane >> 2) * 4);  // d | dmin
        const float p = P.f32<true>(k);
        F.f[8 + k] = __float_as_uint(low_f32(d) * p * kTo24 * kTo24);  // for a scale byte and a field in units of 2^-24 each
        F.f[10 + k] = __float_as_uint(high_f32(d) * p * -kTo24);
    }
}
__device__ __forceinline__ void q4_half_wide(const TileFactors &F, uint32_t tile, int half, int lane, uint32_t (&o)[32]) {
    uint4 w[2];
#pragma unroll
    for (int q = 0; q < 2; q++) w[q] = lds128(tile + kQ4KQsOff + ((2 * half + q) * 32 + lane) * 16);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const uint32_t w4[4] = {w[q].x, w[q].y, w[q].z, w[q].w};
#pragma unroll
        for (int row = 0; row < 2; row++) {
            const uint32_t h = F.f[4 * row + 2 * half + q], sc = __byte_perm(h, 0u, 0x4140), mn = __byte_perm(h, 0u, 0x4342);
            const float d = __uint_as_float(F.f[8 + row]), dm = __uint_as_float(F.f[10 + row]);
            const float s0 = low_f32(sc) * d, s1 = high_f32(sc) * (d * 0.0625f), m0 = low_f32(mn) * dm, m1 = high_f32(mn) * dm;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t a = w4[2 * row + i], b = a >> 8;
                uint32_t *p = o + 16 * q + 4 * i + 2 * row;
                p[0] = fma_f16(a & 0x000F000Fu, s0, m0);
                p[1] = fma_f16(b & 0x000F000Fu, s0, m0);
                p[8] = fma_f16(a & 0x00F000F0u, s1, m1);
                p[9] = fma_f16(b & 0x00F000F0u, s1, m1);
            }
        }
    }
}

// ── Q6_K ────────────────────────────────────────────────────────────────────────────────────
__device__ __forceinline__ void q6_factors(TileFactors &F, const RowPow &P, uint32_t tile, int lane) {
    const uint32_t row = tile + 3072 + (lane >> 2) * 16;
    const uint4 a = lds128(row), b = lds128(row + 128);  // the 16 signed scales
    F.f[0] = a.x, F.f[1] = a.y, F.f[2] = a.z, F.f[3] = a.w, F.f[4] = b.x, F.f[5] = b.y, F.f[6] = b.z, F.f[7] = b.w;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        uint32_t pa, pb;
        P.f16<false>(k, pa, pb);
        F.f[8 + k] = h2_mul(h2_mul(lds16(tile + 3328 + 16 * k + (lane >> 2) * 2) * 0x10001u, pa), pb);
    }
}
// Four 6-bit values (q + 32) per word, for sub-blocks 4m + 0..3 of quarter m; their bytes hold columns 4t + 0, 2, 1, 3.
__device__ __forceinline__ void q6_words(const uint4 &ql, const uint4 &qh, int q, int row, uint32_t NIB, uint32_t HI, uint32_t (&V)[4]) {
    const uint32_t A = row ? ql.z : ql.x, B = row ? ql.w : ql.y, H = row ? (q ? qh.w : qh.z) : (q ? qh.y : qh.x);
    V[0] = and_or(A, NIB, H & HI);
    V[1] = and_or(A >> 4, NIB, (H >> 2) & HI);
    V[2] = and_or(B, NIB, (H << 2) & HI);
    V[3] = and_or(B >> 4, NIB, (H << 4) & HI);
}
__device__ __forceinline__ void q6_half_f16(const TileFactors &F, uint32_t tile, int half, int lane, uint32_t (&o)[32]) {
    uint32_t NIB = 0x0F0F0F0Fu, HI = 0x30303030u;
    asm volatile("" : "+r"(NIB), "+r"(HI));
    uint4 ql[2];
#pragma unroll
    for (int q = 0; q < 2; q++) ql[q] = lds128(tile + ((2 * half + q) * 32 + lane) * 16);
    const uint4 qh = lds128(tile + 2048 + (half * 32 + lane) * 16);  // row g: quarters 2 half, 2 half + 1; row g + 8: the same
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int row = 0; row < 2; row++) {
            uint32_t V[4];
            q6_words(ql[q], qh, q, row, NIB, HI, V);
            const uint32_t h = F.f[4 * row + 2 * half + q] ^ 0x80808080u, d = F.f[8 + row];  // scales + 128
            const uint32_t n[4] = {h2_sub(byte_h2<0>(h, 0x64646464u), kH1152), h2_sub(byte_h2<1>(h, 0x64646464u), kH1152),
                                   h2_sub(byte_h2<2>(h, 0x64646464u), kH1152), h2_sub(byte_h2<3>(h, 0x64646464u), kH1152)};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t s = h2_mul(n[k], d), c = h2_mul(s, kHm19);  // c: -32 of the scale
                uint32_t *p = o + 16 * q + 4 * k + 2 * row;
                p[0] = h2_fma(__byte_perm(V[k], 0u, 0x4140), s, c);
                p[1] = h2_fma(__byte_perm(V[k], 0u, 0x4342), s, c);
            }
        }
}
__device__ __forceinline__ void q6_wide_factors(TileFactors &F, const RowPow &P, uint32_t tile, int lane) {
    const uint32_t row = tile + 3072 + (lane >> 2) * 16;
    const uint4 a = lds128(row), b = lds128(row + 128);
    F.f[0] = a.x, F.f[1] = a.y, F.f[2] = a.z, F.f[3] = a.w, F.f[4] = b.x, F.f[5] = b.y, F.f[6] = b.z, F.f[7] = b.w;
#pragma unroll
    for (int k = 0; k < 2; k++) F.f[8 + k] = __float_as_uint(low_f32(lds16(tile + 3328 + 16 * k + (lane >> 2) * 2)) * P.f32<true>(k) * kTo24);
}
__device__ __forceinline__ void q6_half_wide(const TileFactors &F, uint32_t tile, int half, int lane, uint32_t (&o)[32]) {
    uint32_t NIB = 0x0F0F0F0Fu, HI = 0x30303030u;
    asm volatile("" : "+r"(NIB), "+r"(HI));
    uint4 ql[2];
#pragma unroll
    for (int q = 0; q < 2; q++) ql[q] = lds128(tile + ((2 * half + q) * 32 + lane) * 16);
    const uint4 qh = lds128(tile + 2048 + (half * 32 + lane) * 16);
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int row = 0; row < 2; row++) {
            uint32_t V[4];
            q6_words(ql[q], qh, q, row, NIB, HI, V);
            const uint32_t h = F.f[4 * row + 2 * half + q] ^ 0x80808080u, n01 = __byte_perm(h, 0u, 0x4140), n23 = __byte_perm(h, 0u, 0x4342);  // scales + 128
            const float d = __uint_as_float(F.f[8 + row]), d128 = -128.f * d, d24 = d * kTo24;
            const float s[4] = {fmaf(low_f32(n01), d24, d128), fmaf(high_f32(n01), d24, d128), fmaf(low_f32(n23), d24, d128), fmaf(high_f32(n23), d24, d128)};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float c = s[k] * (-32.f / kTo24);
                uint32_t *p = o + 16 * q + 4 * k + 2 * row;
                p[0] = fma_f16(__byte_perm(V[k], 0u, 0x4140), s[k], c);
                p[1] = fma_f16(__byte_perm(V[k], 0u, 0x4342), s[k], c);
            }
        }
}

// ── Q8_0 ────────────────────────────────────────────────────────────────────────────────────
template <bool WIDE>
__device__ __forceinline__ void q8_factors(TileFactors &F, const RowPow &P, uint32_t tile, int lane) {
    const uint4 r = lds128(tile + 4096 + (lane >> 2) * 16), q = lds128(tile + 4224 + (lane >> 2) * 16);
    const uint32_t d[8] = {r.x, r.y, r.z, r.w, q.x, q.y, q.z, q.w};  // two blocks' d each
#pragma unroll
    for (int row = 0; row < 2; row++) {
        uint32_t pa, pb;
        P.f16<WIDE>(row, pa, pb);
#pragma unroll
        for (int k = 4 * row; k < 4 * row + 4; k++) F.f[k] = h2_mul(h2_mul(d[k], pa), pb);
    }
}
template <bool WIDE>
__device__ __forceinline__ void q8_half_f16(const TileFactors &F, uint32_t tile, int half, int lane, uint32_t (&o)[32]) {
    uint4 w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = lds128(tile + ((4 * half + j) * 32 + lane) * 16);  // words x, y: row g (two 16-column groups), z, w: row g + 8
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t w4[4] = {w[j].x ^ 0x80808080u, w[j].y ^ 0x80808080u, w[j].z ^ 0x80808080u, w[j].w ^ 0x80808080u};  // int8 + 128
#pragma unroll
        for (int row = 0; row < 2; row++) {
            const uint32_t s = __byte_perm(F.f[4 * row + 2 * half + (j >> 1)], 0, j & 1 ? 0x3232 : 0x1010), c = h2_mul(s, kHm17);  // c: -128 of the scale
#pragma unroll
            for (int i = 0; i < 2; i++) {
                uint32_t *p = o + 8 * j + 4 * i + 2 * row;
                const uint32_t v = w4[2 * row + i];
                if constexpr (WIDE) {  // q as it is, exact, times the scale
                    p[0] = h2_mul(h2_sub(__byte_perm(v, 0x64646464u, 0x4240), kH1152), s);
                    p[1] = h2_mul(h2_sub(__byte_perm(v, 0x64646464u, 0x4341), kH1152), s);
                } else {
                    p[0] = h2_fma(__byte_perm(v, 0u, 0x4240), s, c);
                    p[1] = h2_fma(__byte_perm(v, 0u, 0x4341), s, c);
                }
            }
        }
    }
}

template <int TYPE, bool WIDE>
__device__ __forceinline__ void tile_factors_f16(TileFactors &F, const RowPow &P, uint32_t tile, int lane) {
    if constexpr (TYPE == 8)
        q8_factors<WIDE>(F, P, tile, lane);
    else if constexpr (TYPE == 12 && WIDE)
        q4_wide_factors(F, P, tile, lane);
    else if constexpr (TYPE == 12)
        q4_factors(F, P, tile, lane);
    else if constexpr (WIDE)
        q6_wide_factors(F, P, tile, lane);
    else
        q6_factors(F, P, tile, lane);
}
template <int TYPE, bool WIDE>
__device__ __forceinline__ void tile_half_f16(const TileFactors &F, uint32_t tile, int half, int lane, uint32_t (&o)[32]) {
    if constexpr (TYPE == 8)
        q8_half_f16<WIDE>(F, tile, half, lane, o);
    else if constexpr (TYPE == 12 && WIDE)
        q4_half_wide(F, tile, half, lane, o);
    else if constexpr (TYPE == 12)
        q4_half_f16(F, tile, half, lane, o);
    else if constexpr (WIDE)
        q6_half_wide(F, tile, half, lane, o);
    else
        q6_half_f16(F, tile, half, lane, o);
}

}  // namespace juno
