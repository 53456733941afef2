// Resident quantised matrices and the device-level interface of the batched (9..64 sequences) dequant-GEMM:
// used by the MatVec entry points and by the forward pass.  The 1..8 sequence GEMV is declared in qgemv.cuh.
#pragma once
#include "common.cuh"

struct juno_qmat {
    uint32_t magic;
    juno_ctx *ctx;
    int type;          // GGML type id
    int tiled;         // 1: 16x256 tile layout (layout.cuh); 0: raw row-major blocks
    int64_t rows, cols;
    int64_t row_tiles; // ceil(rows/16) when tiled
    int64_t nb;        // cols/256 when tiled
    uint8_t *dev;
    size_t bytes;
    uint32_t *row_pow; // tiled: power of two of every row (tile_f16.cuh), behind the tiles in the same allocation
};

namespace juno {

enum GemvEpilogue {
    EPI_STORE = 0,       // out[b][row] = y
    EPI_SILU_PAIR = 1,   // tile rows 0-7 are gate rows, 8-15 the matching up rows: out[b][8*tile+row] = silu(gate)*up
};

struct GemvSeg {
    const uint8_t *w; // tiled weights
    float *out;       // [batch][ld_out]
    int rows;         // valid rows
    int row_tiles;
    int type = 0;     // block format, 12 / 14 / 8
    const uint32_t *row_pow = nullptr;
};

constexpr int kGemmMaxBatch = 64;  // most sequences of a decode step, or positions of a short portion, that go through the batched path
int gemm_min_batch();              // smallest batch routed to the batched path (JUNO_GEMM_MIN_BATCH, default 9)

// Raw-layout / FP32 fallback (one warp per output), used for shapes the tile layout does not cover.
int launch_gemv_raw(juno_ctx *ctx, const juno_qmat *m, const float *x, int batch, float *y, cudaStream_t stream);
int launch_dequant(juno_ctx *ctx, const juno_qmat *m, int64_t row_start, int64_t n_rows, float *out,
                   cudaStream_t stream);
// Allocates and fills a resident matrix from raw host blocks (row range [row0,row0+nrows), super-block
// column range [sb0, sb0+nsb) of the host tensor — the slicing used by tensor parallelism).
int qmat_create(juno_ctx *ctx, const void *blocks, int type, int64_t rows_total, int64_t cols_total, int64_t row0,
                int64_t nrows, int64_t sb0, int64_t nsb, juno_qmat **out);
int qmat_destroy(juno_qmat *m);

}  // namespace juno
