// Epilogues of the tcgen05 products of many rows (gemm_rows_tc.cu, gemm_pair_tc.cu): TMEM lane = output row, column = output column.
#pragma once
#include "gemm_rows.cuh"
#include "tc5.cuh"
#include "tile_math.cuh"

namespace juno {

using bf16 = __nv_bfloat16;

// 32 columns of one output row.  nv = columns that exist (0..32).
template <int EPI>
__device__ __forceinline__ void store_row(const GemmArgs &g, int z, int m, int n, int nv, const uint32_t (&r)[32]) {
    const size_t o = (size_t)m * g.ldo + (size_t)z * g.o_step + n;
    if (EPI == GE_F32) {
        float *out = static_cast<float *>(g.out) + o;
        if (g.bias) {  // nv is a multiple of 16 then
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                if (j >= nv) break;
                const float4 b = *reinterpret_cast<const float4 *>(g.bias + n + j);
                *reinterpret_cast<float4 *>(out + j) =
                    make_float4(__uint_as_float(r[j]) + b.x, __uint_as_float(r[j + 1]) + b.y, __uint_as_float(r[j + 2]) + b.z, __uint_as_float(r[j + 3]) + b.w);
            }
        } else if (nv == 32 && (g.ldo & 3) == 0 && (g.o_step & 3) == 0) {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4 *>(out + j) = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
        } else {
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (j < nv) out[j] = __uint_as_float(r[j]);
        }
        return;
    }
    if (EPI == GE_F32_ROW) {  // N and ldo are multiples of 16
        const float s = g.row_scale[m];
        float *out = static_cast<float *>(g.out) + o;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            if (j >= nv) break;
            *reinterpret_cast<float4 *>(out + j) = make_float4(__uint_as_float(r[j]) * s, __uint_as_float(r[j + 1]) * s, __uint_as_float(r[j + 2]) * s,
                                                               __uint_as_float(r[j + 3]) * s);
        }
        return;
    }
    if (EPI == GE_SILU_ROW) {
        const float s = g.row_scale[m];
        float *out = static_cast<float *>(g.out) + (size_t)m * g.ldo + (n >> 1);
#pragma unroll
        for (int j = 0; j < 32; j += 16) {
            if (j >= nv) break;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = __fmul_rn(silu_ref(__uint_as_float(r[j + e]) * s), __uint_as_float(r[j + 8 + e]) * s);
            *reinterpret_cast<float4 *>(out + j / 2) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4 *>(out + j / 2 + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
        return;
    }
    if (EPI == GE_GEGLU) {
        bf16 *act = static_cast<bf16 *>(g.out) + (size_t)m * g.ldo + (n >> 1);
#pragma unroll
        for (int j = 0; j < 32; j += 16) {
            if (j >= nv) break;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = fast_geglu(__uint_as_float(r[j + e]), __uint_as_float(r[j + 8 + e]));
            store4(act + j / 2, make_float4(v[0], v[1], v[2], v[3]));
            store4(act + j / 2 + 4, make_float4(v[4], v[5], v[6], v[7]));
        }
        return;
    }
    float gate = 1.f;
    if (EPI == GE_GROUP_GATE) gate = fast_sigmoid(static_cast<const float *>(g.aux)[(size_t)m * g.ldaux + z]);
    bf16 *out = static_cast<bf16 *>(g.out) + o;
    const bf16 *aux = EPI == GE_MUL ? static_cast<const bf16 *>(g.aux) + (size_t)m * g.ldaux + n : nullptr;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
        if (j >= nv) break;  // nv is a multiple of 16 on these outputs
        float4 v = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
        if (EPI == GE_SIGMOID) {
            const float4 b = *reinterpret_cast<const float4 *>(g.bias + n + j);
            v = make_float4(fast_sigmoid(v.x + b.x), fast_sigmoid(v.y + b.y), fast_sigmoid(v.z + b.z), fast_sigmoid(v.w + b.w));
        } else if (EPI == GE_RELU2) {
            v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
            v = make_float4(v.x * v.x, v.y * v.y, v.z * v.z, v.w * v.w);
        } else if (EPI == GE_MUL) {
            const float4 b = load4(aux + j);
            v = make_float4(v.x * b.x, v.y * b.y, v.z * b.z, v.w * b.w);
        } else if (EPI == GE_GROUP_GATE) {
            v = make_float4(v.x * gate, v.y * gate, v.z * gate, v.w * gate);
        }
        store4(out + j, v);
    }
}

}  // namespace juno
