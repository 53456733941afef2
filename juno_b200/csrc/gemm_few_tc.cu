// 16-bit matrix products of few rows (decode batches, short portions of a prompt, logits) on the 5th-generation tensor cores.
//
// Bound by the weights' way from memory, so what counts is the bytes that all SMs together keep in flight.  The operands are
// therefore swapped against gemm_rows_tc.cu: 128 weight rows are the M of the MMA and the (up to kFewRows) activation rows its N,
// so a stage is almost all weights and nothing is copied or multiplied for rows that do not exist; and K is split over the CTAs
// of a cluster until the grid fills the GPU (two CTAs per SM), because the 16 to 112 row tiles of these matrices alone leave most
// SMs idle.  The partial sums meet in shared memory: CTA r of the cluster adds rows r, r + S, ... over all members in order
// (the result does not depend on timing) and applies the epilogue.  The first stages' weights are requested before the kernel waits
// for its predecessor.  Measured on whole decode steps against the row products' 128-row tiles (one CTA per tile, 0.6-1.4 TB/s):
// Vosotar medium, 9 / 24 / 64 requests 1.47 / 1.53 / 1.84 -> 0.80 / 0.99 / 1.40 ms; Desilorn small, 50 requests 1.62 -> 1.21 ms.
#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "gemm_rows.cuh"
#include "tc5.cuh"

namespace juno {

using bf16 = __nv_bfloat16;

constexpr int kFewThreads = 192, kFewMaxStages = 8, kFewMaxSplit = 8;
constexpr int kFewSmem = 110 * 1024;  // two CTAs per SM
constexpr int kFewMinSteps = 4;       // stages of 64 columns below which a further split costs more than it brings

struct FewParams {
    CUtensorMap ta, tw;
    GemmArgs g;
    int n_tiles, k_steps, stages, cols, splits;  // cols: M rounded up to the MMA's N
    unsigned *err;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float peer_ld(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// One output element: weight row n of group z, activation row m.
template <int EPI>
__device__ __forceinline__ void few_store(const GemmArgs &g, int z, int m, int n, float v) {
    if (EPI == GE_GEGLU) {  // the value of a gate is eight rows on
        const float value = __shfl_down_sync(0xffffffffu, v, 8);
        if (n < g.N && !(n & 8)) static_cast<bf16 *>(g.out)[(size_t)m * g.ldo + (n >> 4) * 8 + (n & 7)] = __float2bfloat16(fast_geglu(v, value));
        return;
    }
    if (n >= g.N) return;
    const size_t o = (size_t)m * g.ldo + (size_t)z * g.o_step + n;
    if (EPI == GE_F32) {
        static_cast<float *>(g.out)[o] = g.bias ? v + g.bias[n] : v;
        return;
    }
    if (EPI == GE_SIGMOID) v = fast_sigmoid(v + g.bias[n]);
    if (EPI == GE_RELU2) {
        v = fmaxf(v, 0.f);
        v *= v;
    }
    if (EPI == GE_MUL) v *= __bfloat162float(static_cast<const bf16 *>(g.aux)[(size_t)m * g.ldaux + n]);
    if (EPI == GE_GROUP_GATE) v *= fast_sigmoid(static_cast<const float *>(g.aux)[(size_t)m * g.ldaux + z]);
    static_cast<bf16 *>(g.out)[o] = __float2bfloat16(v);
}

template <int EPI>
__global__ void __launch_bounds__(kFewThreads, 2) gemm_few_kernel(const __grid_constant__ FewParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2 * kFewMaxStages + 1];  // full[stages], empty[stages], accumulator ready
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned fail_s;
    volatile unsigned *fail = &fail_s;
    const uint32_t stage0 = (s_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t w_bytes = kBM * kBK * 2, stage_bytes = w_bytes + (uint32_t)p.cols * kBK * 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, S = p.stages;
    const uint32_t full0 = s_u32(bars), empty0 = full0 + 8 * kFewMaxStages, ready = empty0 + 8 * kFewMaxStages;
    const GemmArgs &g = p.g;
    const int rank = (int)(blockIdx.x % (unsigned)p.splits), tile = (int)(blockIdx.x / (unsigned)p.splits), nt = tile % p.n_tiles, z = tile / p.n_tiles;
    const int k_lo = (int)((long long)p.k_steps * rank / p.splits), steps = (int)((long long)p.k_steps * (rank + 1) / p.splits) - k_lo;
    const int tmem_cols = p.cols <= 32 ? 32 : p.cols <= 64 ? 64 : 128;
    if (threadIdx.x == 0) {
        prefetch_map(&p.tw);
        prefetch_map(&p.ta);
        for (int s = 0; s < S; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * s) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + 8 * s) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ready) : "memory");
        fail_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(&tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot);

    auto weights = [&](int k) {
        const int s = k % S;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full0 + 8 * s), "r"(stage_bytes) : "memory");
        tma_2d(stage0 + s * stage_bytes, &p.tw, (k_lo + k) * kBK, z * g.w_step + nt * kBM, full0 + 8 * s);
    };
    auto rows = [&](int k) {
        const int s = k % S;
        tma_2d(stage0 + s * stage_bytes + w_bytes, &p.ta, z * g.a_step + (k_lo + k) * kBK, 0, full0 + 8 * s);
    };
    const int first = min(S, steps);
    if (threadIdx.x == 0)
        for (int k = 0; k < first; k++) weights(k);
    pdl_wait();  // everything below reads or writes what earlier kernels use
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            for (int k = 0; k < first; k++) rows(k);
            int k = first;
            for (; k < steps; k++) {
                if (!bar_wait(empty0 + 8 * (k % S), (unsigned)(k / S - 1) & 1u, fail)) break;
                weights(k);
                rows(k);
            }
            // the last copies of every stage: nothing may be in flight when the CTA leaves
            for (int b = 0; b < S && b < k; b++) {
                const int j = k - 1 - b;
                const long long t0 = clock64();
                while (!bar_test(full0 + 8 * (j % S), (unsigned)(j / S) & 1u) && clock64() - t0 < kWaitClocks) {
                }
            }
        }
    } else if (warp == 1) {
        // D FP32, A and B BF16, both K-major
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.cols >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
        const bool leader = elect_one();
        bool ok = true;
        for (int k = 0, s = 0, par = 0; k < steps; k++) {
            ok = bar_wait(full0 + 8 * s, (unsigned)par, fail) && ok;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t wd = sw128_desc(stage0 + s * stage_bytes), ad = sw128_desc(stage0 + s * stage_bytes + w_bytes);
            if (leader && ok) {
#pragma unroll
                for (int j = 0; j < kBK / 16; j++) mma_bf16(tmem, wd + 2 * j, ad + 2 * j, idesc, (k > 0 || j > 0) ? 1u : 0u);
                mma_commit(empty0 + 8 * s);
            }
            __syncwarp();
            if (++s == S) {
                s = 0;
                par ^= 1;
            }
        }
        if (leader && ok) mma_commit(ready);
        __syncwarp();
    } else {
        const int quad = warp & 3;  // TMEM lanes a warp can read: 32 * (warp % 4) ..
        int ok = 0;
        if (lane == 0) ok = bar_wait(ready, 0u, fail) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok) {
            // every stage has been multiplied: the ring holds the partial sums now, [activation row][weight row]
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t dst = stage0 + (uint32_t)(quad * 32 + lane) * 4;
            for (int c0 = 0; c0 < p.cols; c0 += 32) {  // columns beyond p.cols are allocated (tmem_cols) and not stored
                uint32_t r[32];
                tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, r);
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (c0 + j < p.cols) asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + (uint32_t)(c0 + j) * (kBM * 4)), "r"(r[j]) : "memory");
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (warp >= 2) {
        const int i = (warp - 2) * 32 + lane, n = nt * kBM + i;
        uint32_t part[kFewMaxSplit];
#pragma unroll
        for (int s = 0; s < kFewMaxSplit; s++) part[s] = peer_addr(stage0 + (uint32_t)i * 4, s < p.splits ? s : rank);
#pragma unroll 2
        for (int m = rank; m < g.M; m += p.splits) {
            float v[kFewMaxSplit];
#pragma unroll
            for (int s = 0; s < kFewMaxSplit; s++) v[s] = s < p.splits ? peer_ld(part[s] + (uint32_t)m * (kBM * 4)) : 0.f;
            float sum = v[0];
#pragma unroll
            for (int s = 1; s < kFewMaxSplit; s++) sum += v[s];
            few_store<EPI>(g, z, m, n, sum);
        }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();  // nobody leaves while its shared memory may still be read
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (*fail) {  // MMAs that were issued before the failure still write TMEM: let them finish (bounded) before it is freed
            const long long t0 = clock64();
            while (clock64() - t0 < 4000000ll) {
            }
            if (lane == 0) atomicCAS(p.err, 0u, kErrStackWait | (1u << 8) | (blockIdx.x << 16));
        }
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
    }
}

// ───────────────────────────── host ───────────────────────────────────────────────────────
template <int EPI>
static int gemm_few_inst(juno_ctx *c, const FewParams &p, int grid, cudaStream_t st) {
    const size_t smem = (size_t)p.stages * (kBM + p.cols) * kBK * 2 + 1024;
    static std::mutex mu;
    static bool configured[16] = {false};
    {
        std::lock_guard<std::mutex> lk(mu);
        if (!configured[c->device & 15]) {
            JUNO_CUDA_TRY(cudaFuncSetAttribute(gemm_few_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewSmem));
            configured[c->device & 15] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kFewThreads);
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
    JUNO_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_few_kernel<EPI>, p));
    c->kernel_launches++;
    return JUNO_OK;
}

int launch_gemm_few_tc(juno_ctx *c, const GemmArgs &a, unsigned *err, cudaStream_t st) {
    JUNO_REQUIRE(a.M >= 1 && a.M <= kFewRows && !a.half, "product of few rows: bad arguments (M %d)", a.M);
    FewParams p;
    memset((void *)&p, 0, sizeof(p));
    p.g = a;
    p.err = err;
    p.cols = (a.M + 15) / 16 * 16;
    p.n_tiles = (a.N + kBM - 1) / kBM;
    p.k_steps = (a.K + kBK - 1) / kBK;
    const int tiles = p.n_tiles * a.groups;
    p.splits = 1;
    while (p.splits < kFewMaxSplit && tiles * p.splits * 2 <= 2 * c->sm_count && p.k_steps >= 2 * p.splits * kFewMinSteps) p.splits *= 2;
    p.stages = std::min(kFewMaxStages, (kFewSmem - 1024) / ((kBM + p.cols) * kBK * 2));
    const int a_cols = a.groups > 1 ? a.a_step * (a.groups - 1) + a.K : a.K;
    const int w_rows = a.w_rows ? a.w_rows : a.groups > 1 ? a.w_step * (a.groups - 1) + a.N : a.N;
    JUNO_TRY(tensor_map_bf16(&p.ta, a.a, a.M, a_cols, a.lda, p.cols));
    JUNO_TRY(tensor_map_bf16(&p.tw, a.w, w_rows, a.K, a.ldw, kBM));
    const int grid = tiles * p.splits;
    switch (a.epi) {
    case GE_F32: return gemm_few_inst<GE_F32>(c, p, grid, st);
    case GE_OP: return gemm_few_inst<GE_OP>(c, p, grid, st);
    case GE_SIGMOID: return gemm_few_inst<GE_SIGMOID>(c, p, grid, st);
    case GE_RELU2: return gemm_few_inst<GE_RELU2>(c, p, grid, st);
    case GE_MUL: return gemm_few_inst<GE_MUL>(c, p, grid, st);
    case GE_GEGLU: return gemm_few_inst<GE_GEGLU>(c, p, grid, st);
    default: return gemm_few_inst<GE_GROUP_GATE>(c, p, grid, st);
    }
}

}  // namespace juno
