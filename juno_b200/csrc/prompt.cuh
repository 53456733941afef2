// Row-major FP16 operands for prompts of the quantised LLaMA layers: many positions of one sequence at a time.
#pragma once
#include "attn.cuh"
#include "common.cuh"

namespace juno {

// The FP16 operands keep their columns in this order inside every group of 32: the eight values that one lane of a warp
// holds of a quantised tile's row (layout.cuh) lie side by side, so that the weights are written 16 bytes at a time.  Both
// operands of a product use the same order, so the product does not notice.
#if defined(__CUDACC__)
__host__ __device__ __forceinline__
#else
inline
#endif
int prompt_col(int col) {
    return (col & ~31) | ((col >> 2) & 3) << 3 | ((col >> 4) & 1) << 2 | (col & 3);
}

struct DequantSeg {
    const uint8_t *w = nullptr;  // tiled weights (layout.cuh)
    int type = 0;                // 12 / 14 / 8
    int row_tiles = 0;
};
// The segments' rows one below the other, each value rounded once to FP16: out [sum of 16 * row_tiles][K].
int launch_dequant_rows(juno_ctx *c, const DequantSeg *seg, int nseg, int K, void *out, cudaStream_t st);

// One FP16 row per position: v = x (+ add), optionally normed (rmsNorm: normw * v / rms), times the power of two that brings
// the row's largest magnitude into [256, 512); scale[row] undoes it.  x_out (optional) takes x + add.
struct StageRowsArgs {
    const float *x = nullptr, *add = nullptr, *normw = nullptr;
    float *x_out = nullptr;
    float eps = 0.f;
    int n = 0, K = 0;
    void *out = nullptr;
    float *scale = nullptr;
    bool quant_order = false;  // columns as quant_col has them (gemm_quant.cuh), else as prompt_col
};
int launch_stage_rows(juno_ctx *c, const StageRowsArgs &a, cudaStream_t st);

// out[i] = x[row[i]] + add[row[i]] for `n` rows of K columns; rows == null: row0 + i.
int launch_gather_rows(juno_ctx *c, const float *x, const float *add, const int32_t *rows, int row0, int n, int K, float *out, cudaStream_t st);

// Attention of rows r < n at positions pos0 + r of one sequence over FP16 pages that already hold every one of them:
// qkv [n][ld] unrotated, query heads first; cs: rope_cos_sin of the rows.
struct PromptAttnArgs {
    const juno_kvpool *pool = nullptr;
    int layer = 0, n = 0, pos0 = 0, n_heads = 0;
    const float *qkv = nullptr;
    int ld = 0;
    const float2 *cs = nullptr;
    const int32_t *slot = nullptr;  // device, one word
    float *out = nullptr;           // [n][n_heads * hd]
    double algo_bytes = 0;
    int32_t *v_odd = nullptr;       // set to 1 by an append with values that are not finite in FP16
    bool guard = false;             // such values may lie in the pages: rows are shielded from those of later positions
};
// Rotates k, rounds k and v to FP16 and writes them to the pages of their positions.
int launch_prompt_append(juno_ctx *c, const PromptAttnArgs &a, cudaStream_t st);
int launch_prompt_attn(juno_ctx *c, const PromptAttnArgs &a, cudaStream_t st);

}  // namespace juno
