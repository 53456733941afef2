// What the product of quantised tiles with FP16 rows (gemm_quant_tc.cu) knows of a row of weights beforehand, found when the matrix is laid out:
// the powers of two that bring the row into the FP16 range, for quick and for wide unpacking (tile_f16.cuh).  Also
// compiled for the host.
#pragma once
#include <math.h>
#include <stdint.h>

#include "layout.cuh"

namespace juno {

// A word per row: exponent for quick tiles | exponent for wide tiles << 8, both with the bias.
constexpr int kRowPowBias = 64;

// Scales of a row, as far as they were seen.  top: bound of what quick unpacking multiplies fields with; most: bound of the weights.
struct RowScales {
    float top = 0.f, most = 0.f;
};
JHD void row_scales_q4(RowScales &r, float d, float dmin, const uint8_t *sc, const uint8_t *mn) {
    int s = 0, m = 0;
    for (int j = 0; j < 8; j++) {
        s = sc[j] > s ? sc[j] : s;
        m = mn[j] > m ? mn[j] : m;
    }
    r.top = fmaxf(r.top, fmaxf(63.f * d, dmin));
    r.most = fmaxf(r.most, 15.f * d * (float)s + dmin * (float)m);
}
JHD void row_scales_q6(RowScales &r, float d, const int8_t *sc) {
    int s = 0;
    for (int j = 0; j < 16; j++) {
        const int a = sc[j] < 0 ? -sc[j] : sc[j];
        s = a > s ? a : s;
    }
    r.top = fmaxf(r.top, 128.f * d);
    r.most = fmaxf(r.most, 32.f * d * (float)s);
}
JHD void row_scales_q8(RowScales &r, float d) {
    r.top = fmaxf(r.top, d);
    r.most = fmaxf(r.most, 128.f * d);
}

JHD uint32_t row_pow_word(const RowScales &r) {
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
    return (uint32_t)(p + kRowPowBias) | (uint32_t)(w + kRowPowBias) << 8;
}

}  // namespace juno
