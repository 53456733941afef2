// Batched dequant-GEMM for decode batches above eight sequences (and for short prompt passes): Y[b][r] = sum_c w(r,c) x[b][c]
// in ONE pass over the quantised weights.
//
// Where the GEMV kernel (qgemv.cu) spends three int8 limb columns per sequence to keep the products exact, this kernel
// treats the batch as a real dense contraction: a warp owns one 16-row tile of the weights, turns each 16x256 quantised tile into
// FP16 A fragments (w = (d*sc)*q - dmin*m, scale and min in FP16, the integer q exact), and multiplies it with mma.sync.m16n8k16
// (f16 in, f32 accumulate) against the activations, one FP16 column per sequence.  Activations are pre-scaled per row by a power of
// two so that they sit well inside the FP16 range; the factor is multiplied back in the epilogue.  Rounding weights and activations
// to FP16 costs about 3e-4 relative on the products (the tolerance of this path is 1e-3).
//
// Data flow.  Eight warps and a ninth that streams the activations, two CTAs per SM.  Every warp brings its own tiles in with bulk
// copies, two or three in flight, the first before the kernel waits for its predecessor; the activations pass through a ring of
// 128-column stages that the warps free one by one, so no barrier ties them together.  K is split over the CTAs of a cluster until
// the grid fills the GPU; the partial sums meet in distributed shared memory and are added in rank order.  Against one CTA per eight
// row tiles that walked all of K with a barrier per 256 columns (latency bound, 10-30 % of the GPU busy on these shapes), per decode
// step: TinyLlama Q4_K_M, 32 requests 3.35 -> 1.64 ms; Q8_0, 9 requests 2.57 -> 1.26; Llama-3-8B with 4 layers, 16 requests 1.08 -> 0.64.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>

#include "bulk.cuh"
#include "gemv.cuh"
#include "layout.cuh"
#include "ring.cuh"
#include "tile_math.cuh"

namespace juno {

constexpr int kGemmWarps = 8, kGemmThreads = (kGemmWarps + 1) * 32;
constexpr int kGemmSmem = 112 * 1024;  // two CTAs per SM
constexpr int kGemmMaxRing = 3, kGemmMaxStages = 6, kGemmMaxSplit = 8;
constexpr int kGemmOutLd = kGemmWarps * 16 + 4;  // floats of a sequence's partial sums: the pad spreads a fragment over the banks

struct GemmParams {
    const uint8_t *w[3];  // tiled weights
    float *out[3];        // [batch][ld_out]
    int rows[3], row_tiles[3], type[3], unit_begin[4];  // a unit = eight row tiles of one matrix
    int nb;               // K / 256
    int batch, NC;        // NC = batch rounded up to a multiple of 8
    int ld_out, epi;
    const uint8_t *ximg;  // FP16 staged activation [K/16][NC][4][4]
    const float *xscale;  // [batch]: factor to multiply the products with
    int splits, ring, stages, slot_bytes;
    unsigned *err;
};

__device__ __forceinline__ void mma16816_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
}
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
__device__ __forceinline__ uint32_t h2_dup(float v) {
    __half2 r = __float2half2_rn(v);
    return *reinterpret_cast<uint32_t *>(&r);
}
constexpr uint32_t kH1024 = 0x64006400u;  // (1024, 1024): 0x6400 | n is the FP16 number 1024 + n for n < 1024
constexpr uint32_t kH1056 = 0x64206420u;  // (1056, 1056)
constexpr uint32_t kH1152 = 0x64806480u;  // (1152, 1152)

__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
// One 16-column step: fragment A against every n-tile.  `x` = address of this lane's (b0, b1) of n-tile 0.
template <int NT>
__device__ __forceinline__ void step16(float (&acc)[NT][4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t x) {
#pragma unroll
    for (int nt = 0; nt < NT; nt++) mma16816_f16(acc[nt], a0, a1, a2, a3, lds64(x + nt * 256));
}

// The factors of one tile that a lane keeps while it goes through the quarters (64 columns) of the tile, and one quarter.
// `tile`: shared address of the tile; `x`: this lane's B fragments of the quarter's first 16 columns, `xs` bytes between 16-column groups.
struct TileFactors {
    uint32_t f[8];
};
// ── Q4_K ────────────────────────────────────────────────────────────────────────────────────
// (scale, -min) of one row for the lane's two sub-blocks 2c, 2c+1, each as an FP16 pair packed in one word.
__device__ __forceinline__ void q4_header_f16(uint32_t dm, uint32_t sm, uint32_t &p0, uint32_t &p1) {
    const float d = f16bits_to_f32(dm), dmin = f16bits_to_f32(dm >> 16);
    const float s0 = d * (float)(sm & 0xFFu), s1 = d * (float)((sm >> 8) & 0xFFu);
    const float m0 = dmin * (float)((sm >> 16) & 0xFFu), m1 = dmin * (float)(sm >> 24);
    __half2 a = __floats2half2_rn(s0, -m0), b = __floats2half2_rn(s1, -m1);
    p0 = *reinterpret_cast<uint32_t *>(&a);
    p1 = *reinterpret_cast<uint32_t *>(&b);
}
__device__ __forceinline__ void q4_factors(TileFactors &F, uint32_t tile, int lane) {
    const uint32_t dm = tile + (lane >> 2) * 4, sm = tile + 64 + lane * 4;
    q4_header_f16(lds32(dm), lds32(sm), F.f[0], F.f[1]);             // row r8
    q4_header_f16(lds32(dm + 32), lds32(sm + 128), F.f[2], F.f[3]);  // row r8 + 8
}
template <int NT>
__device__ __forceinline__ void q4_quarter(const TileFactors &F, uint32_t tile, int g, uint32_t x, uint32_t xs, int lane, float (&acc)[NT][4]) {
    uint32_t M4 = 0x000F000Fu, K = kH1024;
    asm volatile("" : "+r"(M4), "+r"(K));
    const uint4 w = lds128(tile + kQ4KQsOff + (g * 32 + lane) * 16);  // words x, y belong to row r8, words z, w to row r8+8
    const int src = (lane & ~3) | g;  // quad lane g owns sub-blocks 2g and 2g+1
    const uint32_t r0 = __shfl_sync(0xffffffffu, F.f[0], src), r1 = __shfl_sync(0xffffffffu, F.f[1], src);
    const uint32_t q0 = __shfl_sync(0xffffffffu, F.f[2], src), q1 = __shfl_sync(0xffffffffu, F.f[3], src);
    // (s, s) and (-m, -m) for rows r / q and for the low-nibble (2g) / high-nibble (2g+1) sub-block
    const uint32_t sr0 = __byte_perm(r0, 0, 0x1010), mr0 = __byte_perm(r0, 0, 0x3232);
    const uint32_t sr1 = __byte_perm(r1, 0, 0x1010), mr1 = __byte_perm(r1, 0, 0x3232);
    const uint32_t sq0 = __byte_perm(q0, 0, 0x1010), mq0 = __byte_perm(q0, 0, 0x3232);
    const uint32_t sq1 = __byte_perm(q1, 0, 0x1010), mq1 = __byte_perm(q1, 0, 0x3232);
    uint32_t la[4], lb[4], ha[4], hb[4];  // index: word x, y, z, w of the group
    q4_unpack(w.x, M4, K, la[0], lb[0], ha[0], hb[0]);
    q4_unpack(w.y, M4, K, la[1], lb[1], ha[1], hb[1]);
    q4_unpack(w.z, M4, K, la[2], lb[2], ha[2], hb[2]);
    q4_unpack(w.w, M4, K, la[3], lb[3], ha[3], hb[3]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t s_lo = (i < 2) ? sr0 : sq0, m_lo = (i < 2) ? mr0 : mq0;
        const uint32_t s_hi = (i < 2) ? sr1 : sq1, m_hi = (i < 2) ? mr1 : mq1;
        la[i] = h2_fma(h2_sub(la[i], K), s_lo, m_lo);
        lb[i] = h2_fma(h2_sub(lb[i], K), s_lo, m_lo);
        ha[i] = h2_fma(h2_sub(ha[i], K), s_hi, m_hi);
        hb[i] = h2_fma(h2_sub(hb[i], K), s_hi, m_hi);
    }
    step16<NT>(acc, la[0], la[2], lb[0], lb[2], x);
    step16<NT>(acc, la[1], la[3], lb[1], lb[3], x + xs);
    step16<NT>(acc, ha[0], ha[2], hb[0], hb[2], x + 2 * xs);
    step16<NT>(acc, ha[1], ha[3], hb[1], hb[3], x + 3 * xs);
}

// ── Q6_K ────────────────────────────────────────────────────────────────────────────────────
__device__ __forceinline__ void q6_factors(TileFactors &F, uint32_t tile, int lane) {
    const float d_r = f16bits_to_f32(lds16(tile + 3328 + (lane >> 2) * 2)), d_q = f16bits_to_f32(lds16(tile + 3344 + (lane >> 2) * 2));
    const uint32_t sc0 = lds32(tile + 3072 + lane * 4), sc1 = lds32(tile + 3200 + lane * 4);
#pragma unroll
    for (int k = 0; k < 4; k++) {  // FP16 pairs (s, s) of sub-blocks 4c..4c+3 for rows r8 and r8+8
        F.f[k] = h2_dup(d_r * i8_to_f32(sc0, k));
        F.f[4 + k] = h2_dup(d_q * i8_to_f32(sc1, k));
    }
}
template <int NT>
__device__ __forceinline__ void q6_quarter(const TileFactors &F, uint32_t tile, int m, uint32_t x, uint32_t xs, int lane, float (&acc)[NT][4]) {
    uint32_t NIB = 0x0F0F0F0Fu, HI = 0x30303030u;
    asm volatile("" : "+r"(NIB), "+r"(HI));
    const uint4 ql = lds128(tile + (m * 32 + lane) * 16);
    const uint32_t hp = tile + 2048 + ((m >> 1) * 32 + lane) * 16 + (m & 1) * 4;
    const uint32_t WA_r = ql.x, WB_r = ql.y, WA_q = ql.z, WB_q = ql.w, H_r = lds32(hp), H_q = lds32(hp + 8);
    uint32_t V_r[4], V_q[4];  // four 6-bit values per word, for sub-blocks 4m+0..3
    V_r[0] = and_or(WA_r, NIB, H_r & HI);
    V_r[1] = and_or(WA_r >> 4, NIB, (H_r >> 2) & HI);
    V_r[2] = and_or(WB_r, NIB, (H_r << 2) & HI);
    V_r[3] = and_or(WB_r >> 4, NIB, (H_r << 4) & HI);
    V_q[0] = and_or(WA_q, NIB, H_q & HI);
    V_q[1] = and_or(WA_q >> 4, NIB, (H_q >> 2) & HI);
    V_q[2] = and_or(WB_q, NIB, (H_q << 2) & HI);
    V_q[3] = and_or(WB_q >> 4, NIB, (H_q << 4) & HI);
    const int src = (lane & ~3) | m;  // quad lane m owns the scales of sub-blocks 4m..4m+3
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t sr = __shfl_sync(0xffffffffu, F.f[k], src), sq = __shfl_sync(0xffffffffu, F.f[4 + k], src);
        const uint32_t a0 = h2_mul(h2_sub(__byte_perm(V_r[k], 0x64646464u, 0x4140), kH1056), sr);
        const uint32_t a2 = h2_mul(h2_sub(__byte_perm(V_r[k], 0x64646464u, 0x4342), kH1056), sr);
        const uint32_t a1 = h2_mul(h2_sub(__byte_perm(V_q[k], 0x64646464u, 0x4140), kH1056), sq);
        const uint32_t a3 = h2_mul(h2_sub(__byte_perm(V_q[k], 0x64646464u, 0x4342), kH1056), sq);
        step16<NT>(acc, a0, a1, a2, a3, x + k * xs);
    }
}

// ── Q8_0 ────────────────────────────────────────────────────────────────────────────────────
__device__ __forceinline__ void q8_factors(TileFactors &F, uint32_t tile, int lane) {
    const uint4 r = lds128(tile + 4096 + (lane >> 2) * 16), q = lds128(tile + 4224 + (lane >> 2) * 16);
    F.f[0] = r.x, F.f[1] = r.y, F.f[2] = r.z, F.f[3] = r.w, F.f[4] = q.x, F.f[5] = q.y, F.f[6] = q.z, F.f[7] = q.w;
}
template <int NT>
__device__ __forceinline__ void q8_quarter(const TileFactors &F, uint32_t tile, int g, uint32_t x, uint32_t xs, int lane, float (&acc)[NT][4]) {
    uint32_t SGN = 0x80808080u;
    asm volatile("" : "+r"(SGN));
    const uint32_t fr = g & 2 ? (g & 1 ? F.f[3] : F.f[2]) : (g & 1 ? F.f[1] : F.f[0]), fq = g & 2 ? (g & 1 ? F.f[7] : F.f[6]) : (g & 1 ? F.f[5] : F.f[4]);
#pragma unroll
    for (int jj = 0; jj < 2; jj++) {
        const uint4 w = lds128(tile + ((2 * g + jj) * 32 + lane) * 16);
        const uint32_t d_r = __byte_perm(fr, 0, jj ? 0x3232 : 0x1010), d_q = __byte_perm(fq, 0, jj ? 0x3232 : 0x1010);  // (d, d) as stored FP16 bits
        const uint32_t w4[4] = {w.x ^ SGN, w.y ^ SGN, w.z ^ SGN, w.w ^ SGN};  // int8 + 128
        uint32_t a[4][2];  // [word][bytes (0,2) | bytes (1,3)]
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t d = i < 2 ? d_r : d_q;
            a[i][0] = h2_mul(h2_sub(__byte_perm(w4[i], 0x64646464u, 0x4240), kH1152), d);
            a[i][1] = h2_mul(h2_sub(__byte_perm(w4[i], 0x64646464u, 0x4341), kH1152), d);
        }
        // words x, y: row r8 (16-column groups 2j, 2j+1); words z, w: row r8+8
        step16<NT>(acc, a[0][0], a[2][0], a[0][1], a[2][1], x + (2 * jj) * xs);
        step16<NT>(acc, a[1][0], a[3][0], a[1][1], a[3][1], x + (2 * jj + 1) * xs);
    }
}

__device__ __forceinline__ float peer_lds(uint32_t addr, int rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

template <int NT>
__global__ void __launch_bounds__(kGemmThreads, 2) gemm_kernel(const __grid_constant__ GemmParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[kGemmWarps * kGemmMaxRing + 2 * kGemmMaxStages];  // tiles per warp and slot, stages full, stages free
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, NC = p.NC;
    const int rank = (int)(blockIdx.x % (unsigned)p.splits), unit = (int)(blockIdx.x / (unsigned)p.splits);
    const int seg = unit >= p.unit_begin[2] ? 2 : unit >= p.unit_begin[1] ? 1 : 0, u = unit - p.unit_begin[seg], type = p.type[seg];
    const int s0 = p.nb * rank / p.splits, s1 = p.nb * (rank + 1) / p.splits;  // this CTA's 256-column slabs
    const int active = min(kGemmWarps, p.row_tiles[seg] - u * kGemmWarps);     // warps with a row tile
    const uint32_t ring = smem_u32(smem) + (uint32_t)(warp * p.ring * p.slot_bytes), act = smem_u32(smem) + (uint32_t)(kGemmWarps * p.ring * p.slot_bytes);
    const uint32_t stage_bytes = (uint32_t)NC * 256u;  // 128 columns
    const uint32_t tile_bar = smem_u32(bars) + (uint32_t)(warp * kGemmMaxRing * 8), full = smem_u32(bars) + kGemmWarps * kGemmMaxRing * 8, freed = full + kGemmMaxStages * 8;
    const unsigned tbytes = (unsigned)tile_bytes(type);
    const uint8_t *src = p.w[seg] + ((size_t)(u * kGemmWarps + warp) * p.nb + s0) * tbytes;
    const uint64_t pol = l2_evict_first_policy();
    auto fetch = [&](int i) {  // tile s0 + i of this warp's row tile
        const int slot = i % p.ring;
        mbar_expect_tx(tile_bar + slot * 8, tbytes);
        bulk_g2s(ring + slot * p.slot_bytes, src + (size_t)i * tbytes, tbytes, tile_bar + slot * 8, pol);
    };
    if (warp < active && lane == 0) {
        for (int i = 0; i < p.ring; i++) mbar_init(tile_bar + i * 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async;" ::: "memory");
        for (int i = 0; i < p.ring && s0 + i < s1; i++) fetch(i);
    }
    if (tid == kGemmWarps * 32) {
        for (int i = 0; i < p.stages; i++) {
            mbar_init(full + i * 8, 1);
            mbar_init(freed + i * 8, (unsigned)active);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    bool failed = false;
    int issued = 0;  // copies of this warp's slots, or of the stages (lane 0)
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    if (warp == kGemmWarps) {
        if (lane == 0) {
            for (; issued < 2 * (s1 - s0); issued++) {
                const int st = issued % p.stages;
                if (issued >= p.stages) mbar_wait_bounded(freed + st * 8, ring_parity(issued - p.stages, p.stages), 0, p.err, failed);
                if (failed) break;
                mbar_expect_tx(full + st * 8, stage_bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(act + st * stage_bytes),
                             "l"(p.ximg + (size_t)(2 * s0 + issued) * stage_bytes), "r"(stage_bytes), "r"(full + st * 8)
                             : "memory");
            }
        }
        __syncwarp();
    } else if (warp < active) {
        const uint32_t xs = (uint32_t)NC * 32u;
        int slot = 0, st = 0;
        issued = min(p.ring, s1 - s0);
        unsigned tpar = 0, spar = 0;
        for (int i = 0; i < s1 - s0; i++) {
            mbar_wait_bounded(tile_bar + slot * 8, tpar, 0, p.err, failed);
            const uint32_t tile = ring + slot * p.slot_bytes;
            TileFactors F;
            if (type == 12)
                q4_factors(F, tile, lane);
            else if (type == 14)
                q6_factors(F, tile, lane);
            else
                q8_factors(F, tile, lane);
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                mbar_wait_bounded(full + st * 8, spar, 0, p.err, failed);
                const uint32_t x = act + st * stage_bytes + lane * 8;
#pragma unroll 1
                for (int g = 0; g < 2; g++) {
                    if (type == 12)
                        q4_quarter<NT>(F, tile, 2 * h + g, x + g * 4 * xs, xs, lane, acc);
                    else if (type == 14)
                        q6_quarter<NT>(F, tile, 2 * h + g, x + g * 4 * xs, xs, lane, acc);
                    else
                        q8_quarter<NT>(F, tile, 2 * h + g, x + g * 4 * xs, xs, lane, acc);
                }
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(freed + st * 8) : "memory");
                if (++st == p.stages) {
                    st = 0;
                    spar ^= 1u;
                }
            }
            __syncwarp();  // every lane has used the slot's bytes before they are overwritten
            if (lane == 0 && !failed && s0 + i + p.ring < s1) {
                fetch(i + p.ring);
                issued++;
            }
            if (++slot == p.ring) {
                slot = 0;
                tpar ^= 1u;
            }
        }
    }
    // the stages are done with: their memory takes the partial sums, [sequence][row of the unit]
    if (__syncthreads_or(failed)) {  // somebody gave up waiting: what is still on its way has to land first
        if (failed) *reinterpret_cast<volatile unsigned *>(p.err) = 1u | (unsigned)warp << 8 | blockIdx.x << 16;
        if (lane == 0 && (warp < active || warp == kGemmWarps)) {
            const int slots = warp == kGemmWarps ? p.stages : p.ring;
            const uint32_t bar = warp == kGemmWarps ? full : tile_bar;
            for (int j = ring_open(issued, 0, slots); j < issued; j++) mbar_wait_bounded(bar + j % slots * 8, ring_parity(j, slots), 0, p.err, failed);
        }
        __syncthreads();
    }
    if (warp < active) {
        const uint32_t at = act + (uint32_t)((2 * (lane & 3)) * kGemmOutLd + warp * 16 + (lane >> 2)) * 4;
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (uint32_t)((nt * 8 + (j & 1)) * kGemmOutLd + (j >> 1) * 8) * 4), "f"(acc[nt][j]) : "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    {
        const int rows_sh = p.epi == EPI_SILU_PAIR ? 6 : 7, total = p.batch << rows_sh;  // outputs of a unit per sequence: 64 or 128
        for (int idx = (total * rank / p.splits) + tid; idx < total * (rank + 1) / p.splits; idx += kGemmThreads) {
            const int b = idx >> rows_sh, r = idx & ((1 << rows_sh) - 1), orow = (u << rows_sh) + r;
            if (orow >= p.rows[seg]) continue;
            const float sc = p.xscale[b];
            if (p.epi == EPI_SILU_PAIR) {  // rows 0-7 of a tile are gate rows, rows 8-15 the matching up rows
                const uint32_t at = act + (uint32_t)(b * kGemmOutLd + (r >> 3) * 16 + (r & 7)) * 4;
                float gate = 0.f, up = 0.f;
                for (int k = 0; k < p.splits; k++) {
                    gate += peer_lds(at, k);
                    up += peer_lds(at + 32, k);
                }
                p.out[seg][(size_t)b * p.ld_out + orow] = __fmul_rn(silu_ref(gate * sc), up * sc);
            } else {
                const uint32_t at = act + (uint32_t)(b * kGemmOutLd + r) * 4;
                float v = 0.f;
                for (int k = 0; k < p.splits; k++) v += peer_lds(at, k);
                p.out[seg][(size_t)b * p.ld_out + orow] = v * sc;
            }
        }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while its shared memory may still be read
}

// ───────────────────────────── FP16 staging ───────────────────────────────────────────────
// One CTA per image column: columns below `batch` hold one sequence (optionally residual add + RMSNorm), scaled by
// a power of two so that its largest magnitude lands in [256, 512); the remaining columns are zero.
struct StageF16Params {
    int mode;
    const float *x;
    int ldx;
    const float *x_add, *normw;
    float *x_out;
    float eps;
    int K, batch, NC;
    uint8_t *img;
    float *xscale;
    uint8_t *img_tc;  // optional second copy, chunk-major [K/8][N][8] for the tcgen05 kernel (gemm_tc.cu)
    int N_tc;
};

__global__ void __launch_bounds__(256) stage_f16_kernel(const StageF16Params p) {
    pdl_wait();
    pdl_launch_dependents();
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned short *xb = reinterpret_cast<unsigned short *>(p.img);
    const int K = p.K, NC = p.NC;
    __shared__ float red[8], redm[8];
    unsigned short *xt = reinterpret_cast<unsigned short *>(p.img_tc);
    auto tc_dst = [&](int i4) {  // where columns i4..i4+3 go in the chunk-major image (see gemm_tc.cu)
        const int s16 = i4 >> 4, c = (i4 >> 2) & 3, slab = s16 >> 4, t = s16 & 15;
        const int chunk = slab * 32 + ((t >> 2) * 2 + ((t >> 1) & 1)) * 4 + c;
        return ((size_t)chunk * p.N_tc + b) * 8 + (size_t)(t & 1) * 4;
    };
    if (b >= p.batch) {
        for (int i4 = tid * 4; i4 < K; i4 += 256 * 4) {
            const int s16 = i4 >> 4, c = (i4 >> 2) & 3;
            if (b < NC) *reinterpret_cast<uint2 *>(xb + ((size_t)(s16 * NC + b) * 4 + c) * 4) = make_uint2(0u, 0u);
            if (xt && b < p.N_tc) *reinterpret_cast<uint2 *>(xt + tc_dst(i4)) = make_uint2(0u, 0u);
        }
        return;
    }
    const float *xrow = p.x + (size_t)b * p.ldx;
    const float *arow = p.x_add ? p.x_add + (size_t)b * p.ldx : nullptr;
    float scale = 1.f;
    if (p.mode == STAGE_RMSNORM) {
        float part = 0.f;
        for (int i = tid; i < K; i += 256) {
            float r = xrow[i];
            if (arow) r = __fadd_rn(r, arow[i]);
            part = fmaf(r, r, part);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) red[warp] = part;
        __syncthreads();
        float ss = 0.f;
#pragma unroll
        for (int w8 = 0; w8 < 8; w8++) ss += red[w8];
        scale = __fdiv_rn(1.f, (float)sqrt((double)__fadd_rn(__fdiv_rn(ss, (float)K), p.eps)));
    }
    // pass 1: the values (kept in FP32) and their largest magnitude
    float vmax = 0.f;
    for (int i = tid; i < K; i += 256) {
        float r = xrow[i];
        if (p.mode == STAGE_RMSNORM) {
            if (arow) r = __fadd_rn(r, arow[i]);
            if (p.x_out) p.x_out[(size_t)b * p.ldx + i] = r;
            r = __fmul_rn(__fmul_rn(p.normw[i], r), scale);
        }
        vmax = fmaxf(vmax, fabsf(r));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    if (lane == 0) redm[warp] = vmax;
    __syncthreads();
    vmax = redm[0];
#pragma unroll
    for (int w8 = 1; w8 < 8; w8++) vmax = fmaxf(vmax, redm[w8]);
    // power of two that brings vmax into [256, 512) (1 for an all-zero or non-finite row)
    float down = 1.f, up = 1.f;
    if (vmax > 0.f && vmax < 3.0e38f) {
        int e;
        frexpf(vmax, &e);  // vmax = f * 2^e, f in [0.5, 1)
        down = ldexpf(1.f, 9 - e);
        up = ldexpf(1.f, e - 9);
    }
    if (tid == 0) p.xscale[b] = up;
    // pass 2: write the column
    for (int i4 = tid * 4; i4 < K; i4 += 256 * 4) {
        float v[4];
        const float4 xv = *reinterpret_cast<const float4 *>(xrow + i4);
        v[0] = xv.x; v[1] = xv.y; v[2] = xv.z; v[3] = xv.w;
        if (p.mode == STAGE_RMSNORM) {
            if (arow) {
                const float4 av = *reinterpret_cast<const float4 *>(arow + i4);
                v[0] = __fadd_rn(v[0], av.x); v[1] = __fadd_rn(v[1], av.y);
                v[2] = __fadd_rn(v[2], av.z); v[3] = __fadd_rn(v[3], av.w);
            }
            const float4 wv = *reinterpret_cast<const float4 *>(p.normw + i4);
            v[0] = __fmul_rn(__fmul_rn(wv.x, v[0]), scale);
            v[1] = __fmul_rn(__fmul_rn(wv.y, v[1]), scale);
            v[2] = __fmul_rn(__fmul_rn(wv.z, v[2]), scale);
            v[3] = __fmul_rn(__fmul_rn(wv.w, v[3]), scale);
        }
        unsigned short h[4];
#pragma unroll
        for (int t = 0; t < 4; t++) h[t] = __half_as_ushort(__float2half_rn(v[t] * down));
        const int s16 = i4 >> 4, c = (i4 >> 2) & 3;
        uint2 w;  // feed order: columns (4c, 4c+2 | 4c+1, 4c+3)
        w.x = (uint32_t)h[0] | ((uint32_t)h[2] << 16);
        w.y = (uint32_t)h[1] | ((uint32_t)h[3] << 16);
        *reinterpret_cast<uint2 *>(xb + ((size_t)(s16 * NC + b) * 4 + c) * 4) = w;
        if (xt) *reinterpret_cast<uint2 *>(xt + tc_dst(i4)) = w;  // same (x0, x2, x1, x3) packing
    }
}

// ───────────────────────────── host ───────────────────────────────────────────────────────
int gemm_min_batch() {
    static const int v = [] {
        const char *e = getenv("JUNO_GEMM_MIN_BATCH");
        const int n = (e && *e) ? atoi(e) : 9;
        return std::max(2, n);
    }();
    return v;
}

int gemm_padded_batch(int batch) { return (batch + 7) / 8 * 8; }
size_t gemm_image_bytes(int K, int batch) { return (size_t)K * gemm_padded_batch(batch) * 2; }

int launch_stage_f16(juno_ctx *ctx, const StageArgs &a, float *xscale, cudaStream_t st, uint8_t *img_tc) {
    JUNO_REQUIRE(a.K > 0 && a.K % 256 == 0 && a.batch >= 1 && a.batch <= kGemmMaxBatch && a.x && a.img && xscale,
                 "stage (fp16): bad arguments (K=%d, batch=%d)", a.K, a.batch);
    JUNO_REQUIRE(a.ldx % 4 == 0, "stage: row stride %d must be a multiple of 4", a.ldx);
    StageF16Params p;
    p.mode = a.mode;
    p.x = a.x;
    p.ldx = a.ldx;
    p.x_add = a.x_add;
    p.normw = a.normw;
    p.x_out = a.x_out;
    p.eps = a.eps;
    p.K = a.K;
    p.batch = a.batch;
    p.NC = gemm_padded_batch(a.batch);
    p.img = a.img;
    p.xscale = xscale;
    p.img_tc = img_tc;
    p.N_tc = gemm_tc_padded_batch(a.batch);
    ProfScope prof(ctx, st, PROF_OTHER, 0);
    JUNO_CUDA_TRY(launch_pdl(stage_f16_kernel, dim3((unsigned)(img_tc ? std::max(p.NC, p.N_tc) : p.NC)), dim3(256), 0, st, p));
    ctx->kernel_launches++;
    return JUNO_OK;
}

template <int NT>
static int gemm_launch_inst(juno_ctx *ctx, const GemmParams &p, size_t smem, cudaStream_t st) {
    static std::mutex mu;
    static bool configured[16] = {false};
    {
        std::lock_guard<std::mutex> g(mu);
        const int dev = ctx->device & 15;
        if (!configured[dev]) {
            JUNO_CUDA_TRY(cudaFuncSetAttribute(gemm_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem));
            configured[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.unit_begin[3] * p.splits));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    JUNO_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_kernel<NT>, p));
    ctx->kernel_launches++;
    return JUNO_OK;
}

// Segments that share the staged activation share a launch; those that take the tcgen05 kernel get one of their own.
int launch_gemm(juno_ctx *ctx, const GemvArgs &a, cudaStream_t st) {
    JUNO_REQUIRE(a.batch >= 1 && a.batch <= kGemmMaxBatch, "gemm: batch %d outside [1, %d]", a.batch, kGemmMaxBatch);
    JUNO_REQUIRE(a.K > 0 && a.K % 256 == 0 && a.ximg && a.xscale && a.nseg >= 1 && a.nseg <= 3, "gemm: bad arguments (K=%d)", a.K);
    GemmParams p;
    memset(&p, 0, sizeof(p));
    int n = 0, units = 0, first_type = 0;
    double algo = 0;
    for (int s = 0; s < a.nseg; s++) {
        const int t = a.seg[s].type ? a.seg[s].type : a.type;
        JUNO_REQUIRE(t == 12 || t == 14 || t == 8, "gemm: type %d has no tiled kernel", t);
        JUNO_REQUIRE(a.seg[s].out, "gemm: segment %d has no output", s);
        if (a.ximg_tc && a.tc_err && gemm_tc_enabled() && gemm_tc_shape_ok(ctx, a.seg[s].row_tiles, a.batch)) {
            JUNO_TRY(launch_gemm_tc(ctx, a.seg[s].w, t, a.seg[s].rows, a.seg[s].row_tiles, a.K, a.batch, a.ximg_tc, a.xscale, a.seg[s].out,
                                    a.ld_out, a.epi, a.tc_err, st));
            continue;
        }
        p.w[n] = a.seg[s].w;
        p.out[n] = a.seg[s].out;
        p.rows[n] = a.seg[s].rows;
        p.row_tiles[n] = a.seg[s].row_tiles;
        p.type[n] = t;
        p.unit_begin[n] = units;
        units += (a.seg[s].row_tiles + kGemmWarps - 1) / kGemmWarps;
        p.slot_bytes = std::max(p.slot_bytes, tile_bytes(t));
        if (!first_type) first_type = t;
        const double bpw = t == 12 ? 144.0 / 256 : t == 14 ? 210.0 / 256 : 34.0 / 32;
        algo += (double)a.seg[s].rows * a.K * bpw * (a.epi == EPI_SILU_PAIR ? 2 : 1) + (double)a.batch * a.seg[s].rows * 4 + (n == 0 ? (double)a.batch * a.K * 4 : 0.0);
        n++;
    }
    if (n == 0) return JUNO_OK;
    for (int s = n; s < 4; s++) p.unit_begin[s] = units;
    p.nb = a.K / 256;
    p.batch = a.batch;
    p.NC = gemm_padded_batch(a.batch);
    p.ld_out = a.ld_out;
    p.epi = a.epi;
    p.ximg = a.ximg;
    p.xscale = a.xscale;
    p.err = ctx->gemv_scratch.qerr;
    p.splits = 1;
    while (p.splits < kGemmMaxSplit && units * p.splits * 2 <= 2 * ctx->sm_count && p.nb >= 4 * p.splits) p.splits *= 2;
    // tiles in flight first, then stages of the activations; the stages' memory also holds the partial sums
    const size_t sums = (size_t)p.NC * kGemmOutLd * 4, stage = (size_t)p.NC * 256;
    p.ring = 2;
    while (p.ring < kGemmMaxRing && (size_t)kGemmWarps * (p.ring + 1) * p.slot_bytes + std::max(sums, 4 * stage) <= (size_t)kGemmSmem) p.ring++;
    const size_t tiles = (size_t)kGemmWarps * p.ring * p.slot_bytes;
    p.stages = (int)std::min<size_t>(kGemmMaxStages, ((size_t)kGemmSmem - tiles) / stage);
    const size_t smem = tiles + std::max(sums, p.stages * stage);
    JUNO_REQUIRE(p.stages >= 2 && smem <= (size_t)kGemmSmem, "gemm: batch %d does not fit shared memory", a.batch);
    ProfScope prof(ctx, st, first_type == 12 ? PROF_GEMV_Q4K : first_type == 14 ? PROF_GEMV_Q6K : PROF_GEMV_Q80, algo);
    switch (p.NC / 8) {
    case 1: return gemm_launch_inst<1>(ctx, p, smem, st);
    case 2: return gemm_launch_inst<2>(ctx, p, smem, st);
    case 3: return gemm_launch_inst<3>(ctx, p, smem, st);
    case 4: return gemm_launch_inst<4>(ctx, p, smem, st);
    case 5: return gemm_launch_inst<5>(ctx, p, smem, st);
    case 6: return gemm_launch_inst<6>(ctx, p, smem, st);
    case 7: return gemm_launch_inst<7>(ctx, p, smem, st);
    default: return gemm_launch_inst<8>(ctx, p, smem, st);
    }
}

}  // namespace juno
