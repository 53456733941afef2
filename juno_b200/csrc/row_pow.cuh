// What the product of quantised tiles with FP16 rows (gemm_quant_tc.cu) knows of a row of weights beforehand, found when the matrix is laid out:
// the powers of two that bring the row into the FP16 range, and whether its row tile is unpacked in the quick or in the wide way
// (tile_f16.cuh).  Also compiled for the host: the rule is tested there.
#pragma once
#include <math.h>
#include <stdint.h>

#include "layout.cuh"

namespace juno {

// A word per row: exponent for quick tiles | exponent for wide tiles << 8, both with the bias, | kRowWide where one row of the row tile needs it.
constexpr int kRowPowBias = 64;
constexpr uint32_t kRowWide = 1u << 16;

// Scales of a row, as far as they were seen.  top: bound of what quick unpacking multiplies fields with; most: bound of the weights; low: the
// super-block (Q8_0: block) whose largest scale is smallest; low_sub: the smallest scale of a sub-block.  Zeros do not count as small.
struct RowScales {
    float top = 0.f, most = 0.f, low = 3.4e38f, low_sub = 3.4e38f;
};
JHD void row_scales_low(RowScales &r, float low) {
    if (low > 0.f) r.low = fminf(r.low, low);
}
JHD void row_scales_q4(RowScales &r, float d, float dmin, const uint8_t *sc, const uint8_t *mn) {
    int s = 0, m = 0, least = 255;
    for (int j = 0; j < 8; j++) {
        s = sc[j] > s ? sc[j] : s;
        m = mn[j] > m ? mn[j] : m;
        least = sc[j] && sc[j] < least ? sc[j] : least;
    }
    r.top = fmaxf(r.top, fmaxf(63.f * d, dmin));
    r.most = fmaxf(r.most, 15.f * d * (float)s + dmin * (float)m);
    row_scales_low(r, fmaxf(d * (float)s, dmin * (float)m * 0.125f));
    if (s > 0 && d > 0.f) r.low_sub = fminf(r.low_sub, d * (float)least);
}
JHD void row_scales_q6(RowScales &r, float d, const int8_t *sc) {
    int s = 0, least = 255;
    for (int j = 0; j < 16; j++) {
        const int a = sc[j] < 0 ? -sc[j] : sc[j];
        s = a > s ? a : s;
        least = a && a < least ? a : least;
    }
    r.top = fmaxf(r.top, 128.f * d);
    r.most = fmaxf(r.most, 32.f * d * (float)s);
    row_scales_low(r, d * (float)s);
    if (s > 0 && d > 0.f) r.low_sub = fminf(r.low_sub, d * (float)least);
}
JHD void row_scales_q8(RowScales &r, float d) {
    r.top = fmaxf(r.top, d);
    r.most = fmaxf(r.most, 128.f * d);
    row_scales_low(r, d);
}

// Quick unpacking leaves a weight as a multiple of 2^-24 with the largest scale of the row at 2^14 to 2^15: a block far below that one loses digits.  Where
// that would show beside the rounding of the other operand and of the scale, the row tile is wide.  Relative error of a product in which only the
// blocks below the largest count, against rounding every scale and weight at its own size (Q4_K, centred blocks): super-blocks 16 / 32 / 64 / 128
// times below 5.7e-4 and 5.7e-4, 5.9e-4 and 6.1e-4, 4.7e-4 and 5.2e-4, 5.3e-4 and 8.2e-4; Q6_K 64 / 128 / 512 times 3.4e-4 and 3.4e-4, 3.3e-4 and 3.4e-4,
// 2.4e-4 and 6.3e-4; Q8_0 512 / 4096 times 2.1e-4 and 2.2e-4, 2.0e-4 and 1.1e-3.  A sub-block alone, 64 (128)
// times and more below the largest scale: at the limit 1.9e-4 and 2.1e-4 (Q4_K, scale 1), 2.01e-4 and 2.04e-4 (Q6_K); half of that scale 3.3e-4, 2.2e-4.
JHD uint32_t row_pow_word(int type, const RowScales &r) {
    int e = 15, p = 0, w = 0;
    if (r.top > 0.f && r.top < 3.0e38f) {
        frexpf(r.top, &e);
        p = 15 - e < 30 ? 15 - e : 30;
    }
    if (r.most > 0.f && r.most < 3.0e38f) {  // the weights below 2^15, and never below what they are unless they exceed FP16
        frexpf(r.most, &e);
        w = 15 - e < 30 ? 15 - e : 30;
        if (w < 0 && r.most <= 65504.f) w = 0;
    }
    const float low = type == 12 ? 512.f : type == 14 ? 256.f : 64.f, low_sub = type == 12 ? 256.f : type == 14 ? 128.f : 0.f;
    const bool wide = ldexpf(r.low, p) < low || ldexpf(r.low_sub, p) < low_sub;
    return (uint32_t)(p + kRowPowBias) | (uint32_t)(w + kRowPowBias) << 8 | (wide ? kRowWide : 0u);
}

}  // namespace juno
