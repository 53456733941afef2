// 16-bit matrix products of many rows on pairs of SMs: 256 x 256 tiles on tcgen05.mma.cta_group::2.
//
// With one SM per 128 x 256 tile (gemm_rows_tc.cu) a stage of 64 columns brings 48 KB into an SM for 512 cycles of multiplication, more
// than the L2 delivers.  A pair shares one 256 x 256 tile: each CTA holds 128 rows of either operand (32 KB a stage), the tensor
// cores read the other half from the neighbour, and every CTA keeps the accumulators of its own 128 rows.  The first CTA of the pair
// issues the multiplications; both load their operands into the same stage, whose barrier lies in the first CTA, and both store.
// Measured on whole prompts, single SMs against pairs on whole tiles: Llama-3-8B Q4_K_M, 2048 positions 43.8 -> 40.4 ms,
// Desilorn medium, 1500 positions 4.05 -> 3.49 ms, TinyLlama, 1500 positions 6.48 -> 6.14 ms.
#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "gemm_rows.cuh"
#include "gemm_store.cuh"
#include "tc5.cuh"

namespace juno {

constexpr int kPairThreads = 192, kPairN = 256, kPairStages = 6;
constexpr uint32_t kPairHalf = kBM * kBK * 2, kPairStageBytes = 2 * kPairHalf;  // 128 rows of one operand; both

struct GemmPairParams {
    CUtensorMap ta, tw;
    GemmArgs g;
    int m_tiles, n_work, k_steps, splits;
    unsigned *err;
};

__device__ __forceinline__ uint32_t in_cta(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void pair_tma(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
// Arrives at the barrier of this offset in both CTAs of pair q of the cluster when the multiplications issued so far are done.
__device__ __forceinline__ void pair_commit(uint32_t bar, int q = 0) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)(3 << (2 * q))) : "memory");
}
__device__ __forceinline__ void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int EPI>
__global__ void __launch_bounds__(kPairThreads, 1) gemm_pair_kernel(const __grid_constant__ GemmPairParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kPairStages + 4];  // full[stages], empty[stages], acc_full[2], acc_empty[2]
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned fail_s;
    volatile unsigned *fail = &fail_s;
    const uint32_t stage0 = (s_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)(blockIdx.x & 1u), pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const uint32_t full0 = s_u32(bars), empty0 = full0 + 8 * kPairStages, accf0 = empty0 + 8 * kPairStages, acce0 = accf0 + 16;
    if (threadIdx.x == 0) {
        prefetch_map(&p.tw);
        prefetch_map(&p.ta);
        for (int s = 0; s < kPairStages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * s) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + 8 * s) : "memory");
        }
        for (int s = 0; s < 2; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(accf0 + 8 * s) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(acce0 + 8 * s) : "memory");  // four warps of either CTA
        }
        fail_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(&tmem_slot)), "r"(2 * kPairN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_sync();  // the neighbour's barriers and accumulators exist
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot);
    const GemmArgs &g = p.g;
    pdl_wait();
    pdl_launch_dependents();  // not before the wait: dequant_rows_kernel (prompt.cu) may be next and write what the product before this one read

    if (warp == 0) {
        const bool leader = elect_one();
        unsigned s = 0, par = 0;
        bool ok = true;
        for (int work = pair; work < p.n_work; work += pairs) {
            const int mt = work % p.m_tiles, nt = work / p.m_tiles;
            for (int k = 0; k < p.k_steps; k++) {
                ok = bar_wait(empty0 + 8 * s, par ^ 1u, fail) && ok;
                if (leader && ok) {
                    if (rank == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full0 + 8 * s), "r"(2 * kPairStageBytes) : "memory");
                    const uint32_t bar = in_cta(full0 + 8 * s, 0), a_s = stage0 + s * kPairStageBytes;
                    pair_tma(a_s, &p.ta, k * kBK, mt * 2 * kBM + rank * kBM, bar);
                    pair_tma(a_s + kPairHalf, &p.tw, k * kBK, nt * kPairN + rank * kBM, bar);
                }
                __syncwarp();
                if (++s == kPairStages) {
                    s = 0;
                    par ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // D FP32, A and B BF16 or both FP16, both K-major, M 256
            const uint32_t idesc = (1u << 4) | (g.half ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)(kPairN >> 3) << 17) | ((uint32_t)(2 * kBM >> 4) << 24);
            const bool leader = elect_one();
            unsigned s = 0, par = 0, tile = 0;
            bool ok = true;
            for (int work = pair; work < p.n_work; work += pairs, tile++) {
                const unsigned acc = tile & 1u;
                ok = bar_wait(acce0 + 8 * acc, ((tile >> 1) & 1u) ^ 1u, fail) && ok;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + acc * kPairN;
                for (int k = 0; k < p.k_steps; k++) {
                    ok = bar_wait(full0 + 8 * s, par, fail) && ok;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = sw128_desc(stage0 + s * kPairStageBytes), bd = sw128_desc(stage0 + s * kPairStageBytes + kPairHalf);
                    if (leader && ok) {
#pragma unroll
                        for (int j = 0; j < kBK / 16; j++) pair_mma(d, ad + 2 * j, bd + 2 * j, idesc, (k > 0 || j > 0) ? 1u : 0u);
                        pair_commit(empty0 + 8 * s);
                    }
                    __syncwarp();
                    if (++s == kPairStages) {
                        s = 0;
                        par ^= 1u;
                    }
                }
                if (leader && ok) pair_commit(accf0 + 8 * acc);
                __syncwarp();
            }
        }
    } else {
        const int quad = warp & 3;  // TMEM lanes a warp can read: 32 * (warp % 4) ..
        unsigned tile = 0;
        for (int work = pair; work < p.n_work; work += pairs, tile++) {
            const int mt = work % p.m_tiles, nt = work / p.m_tiles;
            const unsigned acc = tile & 1u;
            int ok = 0;
            if (lane == 0) ok = bar_wait(accf0 + 8 * acc, (tile >> 1) & 1u, fail) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int m = mt * 2 * kBM + rank * kBM + quad * 32 + lane;
#pragma unroll 1
            for (int c0 = 0; c0 < kPairN; c0 += 32) {
                const int n = nt * kPairN + c0, nv = min(32, g.N - n);
                if (nv <= 0) break;
                uint32_t r[32];
                tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + acc * kPairN + (uint32_t)c0, r);
                if (m < g.M) store_row<EPI>(g, 0, m, n, nv, r);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_cta(acce0 + 8 * acc, 0)) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*fail) {  // copies and MMAs that were issued before the failure: let them finish (bounded) before memory is given back
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {
        }
        if (threadIdx.x == 0) atomicCAS(p.err, 0u, kErrStackWait | (1u << 8) | (blockIdx.x << 16));
    }
    __syncwarp();
    pair_sync();  // the neighbour has read this CTA's operands and signalled its barriers for the last time
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kPairN) : "memory");
    }
}

// Fewer tiles than pairs: the pairs of a cluster share the K of one tile.  Each keeps a share of the tile's columns; the sums of the
// other columns go through shared memory, and every pair adds up its share over all pairs, in order, and stores it.
template <int EPI>
__global__ void __launch_bounds__(kPairThreads, 1) gemm_pair_split_kernel(const __grid_constant__ GemmPairParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kPairStages + 1];  // full[stages], empty[stages], accumulator ready
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned fail_s;
    volatile unsigned *fail = &fail_s;
    const uint32_t stage0 = (s_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, members = 2 * p.splits, in = (int)(blockIdx.x % (unsigned)members), q = in >> 1, rank = in & 1;
    const int work = (int)(blockIdx.x / (unsigned)members), mt = work % p.m_tiles, nt = work / p.m_tiles;
    const int k0 = p.k_steps * q / p.splits, steps = p.k_steps * (q + 1) / p.splits - k0;
    const uint32_t full0 = s_u32(bars), empty0 = full0 + 8 * kPairStages, ready = empty0 + 8 * kPairStages;
    if (threadIdx.x == 0) {
        prefetch_map(&p.tw);
        prefetch_map(&p.ta);
        for (int s = 0; s < kPairStages; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * s) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + 8 * s) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ready) : "memory");
        fail_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(&tmem_slot)), "r"(kPairN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pair_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot);
    const GemmArgs &g = p.g;
    pdl_wait();
    pdl_launch_dependents();  // not before the wait: dequant_rows_kernel (prompt.cu) may be next and write what the product before this one read
    int ok = 0;  // epilogue warps: the accumulator is complete
    const int quad = warp & 3;
    const uint32_t acc = tmem + ((uint32_t)(quad * 32) << 16), mine = stage0 + (uint32_t)(quad * 32 + lane) * 4;  // partial sums: [column][row]
    const int share = kPairN / p.splits;
    if (warp == 0) {
        const bool leader = elect_one();
        bool good = true;
        for (int k = 0, s = 0, par = 0; k < steps; k++) {
            good = bar_wait(empty0 + 8 * s, (unsigned)par ^ 1u, fail) && good;
            if (leader && good) {
                if (rank == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full0 + 8 * s), "r"(2 * kPairStageBytes) : "memory");
                const uint32_t bar = in_cta(full0 + 8 * s, 2 * q), a_s = stage0 + s * kPairStageBytes;
                pair_tma(a_s, &p.ta, (k0 + k) * kBK, mt * 2 * kBM + rank * kBM, bar);
                pair_tma(a_s + kPairHalf, &p.tw, (k0 + k) * kBK, nt * kPairN + rank * kBM, bar);
            }
            __syncwarp();
            if (++s == kPairStages) {
                s = 0;
                par ^= 1;
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = (1u << 4) | (g.half ? 0u : (1u << 7) | (1u << 10)) | ((uint32_t)(kPairN >> 3) << 17) | ((uint32_t)(2 * kBM >> 4) << 24);
            const bool leader = elect_one();
            bool good = true;
            for (int k = 0, s = 0, par = 0; k < steps; k++) {
                good = bar_wait(full0 + 8 * s, (unsigned)par, fail) && good;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t ad = sw128_desc(stage0 + s * kPairStageBytes), bd = sw128_desc(stage0 + s * kPairStageBytes + kPairHalf);
                if (leader && good) {
#pragma unroll
                    for (int j = 0; j < kBK / 16; j++) pair_mma(tmem, ad + 2 * j, bd + 2 * j, idesc, (k > 0 || j > 0) ? 1u : 0u);
                    pair_commit(empty0 + 8 * s, q);
                }
                __syncwarp();
                if (++s == kPairStages) {
                    s = 0;
                    par ^= 1;
                }
            }
            if (leader && good) pair_commit(ready, q);
            __syncwarp();
        }
    } else {
        if (lane == 0) ok = bar_wait(ready, 0u, fail) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c0 = 0; c0 < kPairN; c0 += 32) {
                if (c0 / share == q) continue;  // this pair's own columns stay where they are
                uint32_t r[32];
                tmem_ld32(acc + (uint32_t)c0, r);
#pragma unroll
                for (int j = 0; j < 32; j++) asm volatile("st.shared.u32 [%0], %1;" ::"r"(mine + (uint32_t)(c0 + j) * (kBM * 4)), "r"(r[j]) : "memory");
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*fail) {  // copies and MMAs that were issued before the failure: let them finish (bounded) before memory is given back
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {
        }
        if (threadIdx.x == 0) atomicCAS(p.err, 0u, kErrStackWait | (1u << 8) | (blockIdx.x << 16));
    }
    __syncwarp();
    pair_sync();
    if (warp >= 2 && ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int m = mt * 2 * kBM + rank * kBM + quad * 32 + lane;
#pragma unroll 1
        for (int c0 = q * share; c0 < (q + 1) * share; c0 += 32) {
            const int n = nt * kPairN + c0, nv = min(32, g.N - n);
            if (nv <= 0) break;
            uint32_t r[32];
            float sum[32];
            tmem_ld32(acc + (uint32_t)c0, r);
#pragma unroll
            for (int j = 0; j < 32; j++) sum[j] = 0.f;
            for (int o = 0; o < p.splits; o++) {
                if (o == q) {
#pragma unroll
                    for (int j = 0; j < 32; j++) sum[j] += __uint_as_float(r[j]);
                    continue;
                }
                const uint32_t at = in_cta(mine + (uint32_t)c0 * (kBM * 4), 2 * o + rank);
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    float v;
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at + (uint32_t)j * (kBM * 4)) : "memory");
                    sum[j] += v;
                }
            }
#pragma unroll
            for (int j = 0; j < 32; j++) r[j] = __float_as_uint(sum[j]);
            if (m < g.M) store_row<EPI>(g, 0, m, n, nv, r);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncwarp();
    pair_sync();  // nobody leaves while its shared memory may still be read
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPairN) : "memory");
    }
}

// ───────────────────────────── host ───────────────────────────────────────────────────────
template <int EPI, bool SPLIT>
static int gemm_pair_inst(juno_ctx *c, const GemmPairParams &p, cudaStream_t st) {
    const size_t smem = (size_t)kPairStages * kPairStageBytes + 1024;
    static std::mutex mu;
    static int fit[16] = {0};  // pairs that the device holds at a time
    const auto kernel = SPLIT ? gemm_pair_split_kernel<EPI> : gemm_pair_kernel<EPI>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    int n = 0;
    {
        std::lock_guard<std::mutex> lk(mu);
        int &f = fit[c->device & 15];
        if (f == 0) {
            JUNO_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            cfg.numAttrs = 1;
            JUNO_CUDA_TRY(cudaOccupancyMaxActiveClusters(&f, kernel, &cfg));
            JUNO_REQUIRE(f > 0, "no pair of CTAs fits");
        }
        n = f;
    }
    attr[0].val.clusterDim.x = (unsigned)(2 * p.splits);
    cfg.gridDim = dim3((unsigned)(SPLIT ? 2 * p.splits * p.n_work : 2 * std::min(n, p.n_work)));
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    JUNO_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p));
    c->kernel_launches++;
    return JUNO_OK;
}

template <bool SPLIT>
static int gemm_pair_epi(juno_ctx *c, const GemmPairParams &p, cudaStream_t st) {
    switch (p.g.epi) {
    case GE_F32: return gemm_pair_inst<GE_F32, SPLIT>(c, p, st);
    case GE_OP: return gemm_pair_inst<GE_OP, SPLIT>(c, p, st);
    case GE_SIGMOID: return gemm_pair_inst<GE_SIGMOID, SPLIT>(c, p, st);
    case GE_RELU2: return gemm_pair_inst<GE_RELU2, SPLIT>(c, p, st);
    case GE_MUL: return gemm_pair_inst<GE_MUL, SPLIT>(c, p, st);
    case GE_GEGLU: return gemm_pair_inst<GE_GEGLU, SPLIT>(c, p, st);
    case GE_F32_ROW: return gemm_pair_inst<GE_F32_ROW, SPLIT>(c, p, st);
    case GE_SILU_ROW: return gemm_pair_inst<GE_SILU_ROW, SPLIT>(c, p, st);
    default: break;
    }
    set_error("product on pairs: epilogue %d is not taken", p.g.epi);
    return JUNO_ERR_UNSUPPORTED;
}

// How many pairs share the K of a tile (1: persistent pairs on whole tiles); 0: tiles of 128 rows on single SMs do better.  Estimated in
// steps of 64 columns on a pair: rounds of tiles, the exchange of a split beside them; a single SM takes 1.33 steps for 256 columns of 128 rows
// (fitted to prompts of 200 to 1900 positions; 1.7 takes splits that cost TinyLlama's 333 positions 3.22 -> 3.39 ms).  Without and with
// splits: Vosotar small, 1000 positions 2.55 -> 2.32 ms, 250 positions 1.78 -> 1.54; Vosotar medium, 400 positions 1.65 -> 1.38; TinyLlama
// Q4_K_M, 700 positions 3.97 -> 3.58; Llama-3-8B with 4 layers, 200 positions 1.52 -> 1.32.
int gemm_pair_splits(const juno_ctx *c, const GemmArgs &a) {
    if (a.groups > 1 || a.epi == GE_GROUP_GATE) return 0;
    const double f_single = 1.33, c_split = 8;
    const int steps = (a.K + kBK - 1) / kBK;
    double best = 1e30;
    int pick = 0;
    for (int w = 256; w >= 32; w /= 2) {
        if (w > 32 && w / 2 >= a.N) continue;
        const long long tiles = (long long)((a.M + kBM - 1) / kBM) * ((a.N + w - 1) / w);
        best = std::min(best, (double)((tiles + c->sm_count - 1) / c->sm_count) * steps * (w + 40) / 296 * f_single);
    }
    const long long tiles = (long long)((a.M + 2 * kBM - 1) / (2 * kBM)) * ((a.N + kPairN - 1) / kPairN), pairs = c->sm_count / 2;
    for (int s = 1; s <= 4; s *= 2) {
        if (s > 1 && (tiles * s > 4 * pairs || steps < 4 * s)) break;
        const double cost = (double)((tiles * s + pairs - 1) / pairs) * ((double)steps / s + (s > 1 ? c_split : 0));
        if (cost < best) {
            best = cost;
            pick = s;
        }
    }
    return pick;
}

int launch_gemm_pair_tc(juno_ctx *c, const GemmArgs &a, int splits, unsigned *err, cudaStream_t st) {
    GemmPairParams p;
    memset((void *)&p, 0, sizeof(p));
    p.g = a;
    p.err = err;
    p.splits = splits;
    p.m_tiles = (a.M + 2 * kBM - 1) / (2 * kBM);
    p.n_work = p.m_tiles * ((a.N + kPairN - 1) / kPairN);
    p.k_steps = (a.K + kBK - 1) / kBK;
    JUNO_TRY(tensor_map_bf16(&p.ta, a.a, a.M, a.K, a.lda, kBM));
    JUNO_TRY(tensor_map_bf16(&p.tw, a.w, a.w_rows ? a.w_rows : a.N, a.K, a.ldw, kBM));
    return splits > 1 ? gemm_pair_epi<true>(c, p, st) : gemm_pair_epi<false>(c, p, st);
}

}  // namespace juno
