// How a product of quantised tiles with FP16 rows is spread over the GPU (gemm_quant_tc.cu): rows of x per pass, CTAs that share K, and the row
// tiles of a cluster.  Also compiled for the host alone: the rules are tested there.
#pragma once
#include <stdint.h>

#include <algorithm>

#include "layout.cuh"

namespace juno {

constexpr int kQtWarps = 8;      // row tiles that a CTA takes at a time
constexpr int kQtMaxSplit = 8, kQtMaxN = 224;

struct QuantSplit {
    int N = 0, col_blocks = 0;       // rows of x per pass over the weights, a multiple of 16; passes
    int splits = 0, clusters = 0;    // CTAs of a cluster, which share K; 0: nothing fits the device
};

// Rows of x per pass over the weights: one pass up to 224 rows, then two, four, ...  With more than 224 only two stages of x fit.  Prompts
// of 256 positions in one and in two passes: Llama-3-8B 6.80 and 6.45 ms, TinyLlama Q4_K_M 2.57 and 2.19 ms; of 200: 5.44 and 6.06, 2.23 and
// 2.27; three passes or five were slower than two or four everywhere.
inline QuantSplit quant_passes(int n) {
    QuantSplit q;
    q.col_blocks = 1;
    while ((n + q.col_blocks - 1) / q.col_blocks > kQtMaxN) q.col_blocks *= 2;
    q.N = ((n + q.col_blocks - 1) / q.col_blocks + 15) / 16 * 16;
    q.col_blocks = (n + q.N - 1) / q.N;
    return q;
}

// CTAs that share K: estimated in SM cycles, unpacking or multiplying 128 columns of a piece, whatever takes longer, with both CTAs of
// an SM at it, plus what a piece and an exchange cost beside that.  2048 x 5632 Q4_K, 9 rows with 1 / 2 / 3 / 6: 20.2 / 17.2 / 15.7 / 12.6 us;
// 28672 x 4096 does not gain from any.  rt: row tiles, nb: blocks of 256 columns; fit[s]: clusters of s CTAs, one CTA per SM, that the device holds at
// a time, 0 for a size that it does not take; pair: two CTAs per SM.
inline void quant_split(QuantSplit &q, int rt, int nb, bool pair, const int *fit) {
    double best = 1e30;
    for (int s = 1; s <= kQtMaxSplit && s <= nb; s++) {
        if (fit[s] <= 0) continue;
        int n = fit[s] * (pair ? 2 : 1), per = 1;  // clusters; pieces of a cluster
        if (s > 1) {                               // every cluster one piece
            n = n / q.col_blocks * q.col_blocks;
            if (n < q.col_blocks || (rt + n / q.col_blocks - 1) / (n / q.col_blocks) > kQtWarps) continue;
        }
        const int share = (int)(((long long)rt * q.col_blocks + n - 1) / n);
        if (s == 1) per = (share + kQtWarps - 1) / kQtWarps;
        const double half = std::max(35.0 * std::max((share + per - 1) / per, 4), 4.0 * q.N) * (pair ? 2 : 1);
        const double cost = per * ((double)((nb + s - 1) / s) * 2 * half + 1500) + (s > 1 ? 2000 + 2.0 * q.N * share : 0);
        if (cost < best) {
            best = cost;
            q.splits = s;
            q.clusters = std::min(n, rt * q.col_blocks);
        }
    }
}

// `total` things over `n` takers, divided beforehand: taker i begins at total * i / n, rounded down.  One more than the least is taken at even distances: with the larger
// shares first Llama-3-8B prompts of 333 / 500 positions took 9.55 / 14.2 ms, with them spread 8.55 / 12.95.
struct EvenShares {
    int least, more;     // total / n and what is left
    uint32_t per_n;      // 2^32 / n, rounded up: the quotients below are exact for n up to 2^10
    JHD int begin(int i) const { return i * least + (int)((uint64_t)(uint32_t)(i * more) * per_n >> 32); }
};
inline EvenShares even_shares(int total, int n) { return EvenShares{total / n, total % n, (uint32_t)(((1ull << 32) + n - 1) / n)}; }

// What a launch knows of its clusters' shares of the (column block, row tile) pairs.
struct QuantShares {
    int total_rt, col_blocks;
    EvenShares of;
};
inline QuantShares quant_shares(const QuantSplit &q, int rt) { return QuantShares{rt, q.col_blocks, even_shares(rt * q.col_blocks, q.clusters)}; }
// A cluster's share of the (column block, row tile) pairs, in pieces of up to eight row tiles of one column block.
struct QtWalk {
    int f, end;        // flat index of the piece's first row tile; end of the share
    int block, lo, r;  // column block, first row tile, row tiles of the piece
};
JHD void qt_piece(QtWalk &w, int total_rt) {
    const int stop = (w.block + 1) * total_rt, rem = (w.end < stop ? w.end : stop) - w.f, k = (rem + kQtWarps - 1) / kQtWarps;
    w.lo = w.f - w.block * total_rt;
    w.r = k > 1 ? (rem + k - 1) / k : rem > 0 ? rem : 0;
}
JHD QtWalk qt_begin(const QuantShares &s, int cluster) {
    QtWalk w;
    w.f = s.of.begin(cluster);
    w.end = s.of.begin(cluster + 1);
    w.block = s.col_blocks == 1 ? 0 : w.f / s.total_rt;
    qt_piece(w, s.total_rt);
    return w;
}
JHD void qt_next(QtWalk &w, int total_rt) {
    w.f += w.r;
    if (w.f == (w.block + 1) * total_rt) w.block++;
    qt_piece(w, total_rt);
}

}  // namespace juno
