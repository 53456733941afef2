// Products of quantised matrices with FP16 rows on tcgen05 (gemm_quant_tc.cu): device-level interface.
#pragma once
#include "common.cuh"
#include "gemv.cuh"

namespace juno {

// out[r][row] = scale[r] * sum_c w(row, c) x[r][c] for r < n, in one pass over the quantised blocks for up to 224 rows of x, in two, four, ... of
// equal parts above (quant_passes).
struct GemmQuantArgs {
    GemvSeg seg[3];  // matrices that share the input; any mix of block formats
    int nseg = 1;
    int K = 0, n = 0;
    const void *x = nullptr;  // FP16 [n][K], columns in the order of quant_col
    const float *scale = nullptr;  // [n]
    int ld_out = 0, epi = EPI_STORE;
    bool precise = false;  // weights rounded once (tile_f16.cuh)
};
int launch_gemm_quant(juno_ctx *c, const GemmQuantArgs &a, cudaStream_t st);

// The FP16 rows keep the four columns of every group of four in the order in which a tile's bytes give them (tile_f16.cuh).
#if defined(__CUDACC__)
__host__ __device__ __forceinline__
#else
inline
#endif
int quant_col(int col) {
    return (col & ~3) | (col & 1) << 1 | (col >> 1 & 1);
}

}  // namespace juno
