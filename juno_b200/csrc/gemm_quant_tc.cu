// Products of quantised matrices with FP16 rows (decode batches, prompts) on tcgen05: the weights become FP16 on their way from the ring
// of quantised tiles to the tensor memory, from which the MMAs read them as operand A.
//
// The work per tile of 16 x 256 weights is its unpacking (tile_f16.cuh), whatever the number of rows it is multiplied with, and no FP16
// copy of the weights goes through memory.  Unpacked values that went through shared memory would cost 64 cycles of its bandwidth to
// write and as many for the MMA to read them; the tensor memory takes them in 32, in the register layout that a tile's lanes have anyway
// (tcgen05.st 16x256b is an mma fragment), and the multiplication costs the unpacking warps nothing.  Bound by the unpacking up to about
// 128 rows, by the MMAs above: quick 186 cycles of a scheduler per 128 columns of a Q4_K tile (Q6_K 250, Q8_0 166) where the multiply-adds
// would take 112; the byte permutes and shifts run at a quarter of the rate.
//
// A CTA takes up to eight row tiles (128 weight rows, the M of the MMA) at a time and walks along its part of K.  Eight warps own a row
// tile each and unpack 128 columns at a time into a stage of tensor memory; a ninth streams the rows of x by TMA into the same stage, a
// tenth issues the MMAs, an eleventh copies the tiles, one ring per unpacking warp, the first before the kernel waits for its
// predecessor.  Fewer row tiles than the GPU has places: the CTAs of a cluster share K, and their sums meet in shared memory, added in
// rank order.
//
// Measured in chains of 20 launches with their staging against the kernels before (mma.sync with the batch as N, tcgen05 through shared memory),
// Q4_K with quick tiles, 9 / 32 / 64 rows: 28672 x 4096 45.8 / 56.5 / 60.8 -> 25.7 / 27.0 / 29.2 us; 4096 x 14336 25.4 / 36 to 47 / 45 to 60 -> 18.9 / 20.0 /
// 23.6; 4096 x 4096 10.5 / 20.3 / 18.8 -> 11.1 / 11.6 / 16.0; 2048 x 2048 8.0 / 9.8 / 12.3 -> 8.3 / 9.0 / 11.1.  The smallest with 9 to 16 rows stay up to
// 0.6 us behind: tensor memory, tensor copies and the give-back before the exchange.  Whole calls: TinyLlama, 9 / 64 requests 1334 / 2363 -> 1102 / 1530 us;
// Llama-3-8B with 4 layers, 48 requests 1.04 -> 0.58 ms; 200 positions of the 8B model 9.9 -> 5.4 ms.
#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "gemm_quant.cuh"
#include "quant_split.cuh"
#include "ring.cuh"
#include "tc5.cuh"
#include "tile_f16.cuh"

namespace juno {

constexpr int kQtThreads = (kQtWarps + 3) * 32, kQtMaxRing = 4, kQtMaxStages = 4;
constexpr int kQtLd = kQtWarps * 16 + 4;       // floats of a row's partial sums: the pad spreads a fragment over the banks
constexpr int kQtPairSmem = 112 * 1024;        // two CTAs per SM
constexpr int kQtOneSmem = 224 * 1024;

struct GemmQuantParams {
    CUtensorMap tx;
    const uint8_t *w[3];
    const uint32_t *pow[3];  // powers of two of the rows
    float *out[3];
    int rows[3], type[3], rt_begin[4];
    QuantShares shares;
    EvenShares blocks;       // 256-column blocks over the CTAs of a cluster
    int nb, n, N;  // N: rows of x per pass, a multiple of 16
    int ld_out, epi, splits;
    int ring, slot_bytes, stages, tmem_cols;
    const float *scale;
    unsigned *err;
};

__device__ __forceinline__ int qt_seg(const GemmQuantParams &p, int rt) { return rt >= p.rt_begin[2] ? 2 : rt >= p.rt_begin[1] ? 1 : 0; }

__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
// 16 lanes x 64 columns: registers 4j .. 4j+3 are the fragment (rows g, g + 8; columns 2t, 2t + 1) of columns 8j .. 8j+7.
__device__ __forceinline__ void tmem_st_16x64(uint32_t addr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31,%32};\n" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_ld_16x16(uint32_t addr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Four neighbouring sums over the cluster, in rank order, four ranks' loads on their way at a time (one after the other they cost half a
// microsecond each).
__device__ __forceinline__ float4 qt_peer_sum(uint32_t addr, int splits) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int k0 = 0; k0 < splits; k0 += 4) {
        float4 part[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t a;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(min(k0 + k, splits - 1)));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(part[k].x), "=f"(part[k].y), "=f"(part[k].z), "=f"(part[k].w) : "r"(a) : "memory");
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (k0 + k < splits) v = make_float4(v.x + part[k].x, v.y + part[k].y, v.z + part[k].z, v.w + part[k].w);
    }
    return v;
}
__device__ __forceinline__ void qt_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

// The next tile of an unpacking warp, in the hands of a lane of the copying warp.
struct QtTiles {
    QtWalk w;
    const uint8_t *src;
    unsigned bytes;
    int sb, owner, s0, nb, issued;
    __device__ __forceinline__ void seek(const GemmQuantParams &p) {  // first piece from here on in which the warp has a row tile
        while (w.r > 0 && owner >= w.r) qt_next(w, p.shares.total_rt);
        if (w.r <= 0) return;
        const int rt = w.lo + owner, s = qt_seg(p, rt);
        bytes = (unsigned)tile_bytes(p.type[s]);
        src = p.w[s] + ((size_t)(rt - p.rt_begin[s]) * p.nb + s0) * bytes;
        sb = 0;
    }
    __device__ __forceinline__ void init(const GemmQuantParams &p, int warp, const QtWalk &begin, int first, int count) {
        w = begin;
        owner = warp;
        s0 = first;
        nb = count;
        issued = 0;
        seek(p);
    }
    __device__ __forceinline__ void fetch(const GemmQuantParams &p, uint32_t bar, uint32_t dst) {
        mbar_expect_tx(bar, bytes);
        bulk_g2s(dst, src, bytes, bar, l2_evict_first_policy());
        issued++;
        src += bytes;
        if (++sb == nb) {
            qt_next(w, p.shares.total_rt);
            seek(p);
        }
    }
};
// Where a warp is in its ring of tiles and in the stages of unpacked weights.
struct QtUnpack {
    uint32_t ring, tile_bar, tile_free, full, free, dst;
    int slots, slot_bytes, stages;
    int slot, sa;
    unsigned tpar, apar;
};
// The tiles of one row tile, nb of them, unpacked into the stages in turn.  TYPE 0: a warp without a row tile, which only keeps step.
// One body per format: the store takes 32 registers in a row, and where the formats' paths met before it every one was moved.
template <int TYPE, bool WIDE>
__device__ __forceinline__ void qt_unpack(QtUnpack &u, const RowPow &P, int nb, volatile unsigned *fail) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int i = 0; i < nb; i++) {
        const uint32_t tile = u.ring + u.slot * u.slot_bytes;
        TileFactors F;
        if constexpr (TYPE != 0) {
            bar_wait(u.tile_bar + u.slot * 8, u.tpar, fail);
            __syncwarp();
            tile_factors_f16<TYPE, WIDE>(F, P, tile, lane);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t r[32];
            if constexpr (TYPE != 0) tile_half_f16<TYPE, WIDE>(F, tile, h, lane, r);
            bar_wait(u.free + u.sa * 8, u.apar ^ 1u, fail);
            __syncwarp();
            if constexpr (TYPE != 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tmem_st_16x64(u.dst + u.sa * 64, r);
                if (h == 1 && lane == 0) qt_arrive(u.tile_free + u.slot * 8);  // every lane has used the slot's bytes
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) qt_arrive(u.full + u.sa * 8);
            if (++u.sa == u.stages) {
                u.sa = 0;
                u.apar ^= 1u;
            }
        }
        if (TYPE != 0 && ++u.slot == u.slots) {
            u.slot = 0;
            u.tpar ^= 1u;
        }
    }
}

// Read again where they are used: kept, they would cost the unpacking warps registers.
__device__ __forceinline__ int cluster_rank() {
    int r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ int cluster_id() {
    int r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}

template <bool PRECISE>
__global__ void __launch_bounds__((kQtWarps + 4) * 32, 2) gemm_quant_kernel(const __grid_constant__ GemmQuantParams p) {
    extern __shared__ uint8_t smem_raw[];
    // a tile landed, a tile used, per warp and slot; stages: weights written and x landed, used; sums: complete, taken
    __shared__ __align__(8) uint64_t bars[2 * kQtWarps * kQtMaxRing + 2 * kQtMaxStages + 2];
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned fail_s;
    __shared__ int issued_s[kQtWarps + 1];  // copies into each ring, and into the stages of x
    // not in registers while tiles are unpacked: where the copying warp is, and the piece of every unpacking warp
    __shared__ QtTiles tiles_s[kQtWarps];
    __shared__ QtWalk walk_s[kQtWarps];
    volatile unsigned *fail = &fail_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s0 = p.blocks.begin(cluster_rank()), nb = p.blocks.begin(cluster_rank() + 1) - s0;  // this CTA's 256-column blocks
    const uint32_t x0 = (s_u32(smem_raw) + 1023u) & ~1023u, x_bytes = (uint32_t)p.N * 256u;  // 128 columns of x: two boxes of 64
    // whose tiles: an unpacking warp's own; lane w of the copying warp sees to those of warp w
    const int owner = warp < kQtWarps ? warp : lane & (kQtWarps - 1);
    const uint32_t ring = x0 + (uint32_t)p.stages * x_bytes + (uint32_t)(owner * p.ring * p.slot_bytes);
    const uint32_t tile_bar = s_u32(bars) + (uint32_t)(owner * kQtMaxRing) * 8u, tile_free = tile_bar + kQtWarps * kQtMaxRing * 8, full = s_u32(bars) + 2 * kQtWarps * kQtMaxRing * 8, free = full + kQtMaxStages * 8,
                   acc_full = free + kQtMaxStages * 8, acc_free = acc_full + 8;
    // Before the CTA meets, every warp finds its first piece, an unpacking warp also the powers of two of its rows there: divisions and a load from
    // memory that would follow one another behind the dependency wait otherwise.
    QtWalk w;
    RowPow P{{0u, 0u}};
    auto load_pow = [&]() {
        const int rt = w.lo + warp, seg = qt_seg(p, rt);
        const uint32_t *pow = p.pow[seg] + (rt - p.rt_begin[seg]) * 16 + (lane >> 2);
        P.w[0] = __ldg(pow);
        P.w[1] = __ldg(pow + 8);
    };
    if (warp == kQtWarps + 2) {
        if (lane == 0) fail_s = 0;
        if (lane < kQtWarps) {
            for (int i = 0; i < p.ring; i++) {
                mbar_init(tile_bar + i * 8, 1);
                mbar_init(tile_free + i * 8, 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async;" ::: "memory");
            QtTiles t;
            t.init(p, owner, qt_begin(p.shares, cluster_id()), s0, nb);
            for (int i = 0; i < p.ring && t.w.r > 0; i++) t.fetch(p, tile_bar + i * 8, ring + i * p.slot_bytes);
            tiles_s[owner] = t;
        }
        __syncwarp();
    } else if (warp == kQtWarps) {
        if (lane == 0) {
            prefetch_map(&p.tx);
            for (int i = 0; i < p.stages; i++) {
                mbar_init(full + i * 8, kQtWarps + 1);
                mbar_init(free + i * 8, 1);
            }
            mbar_init(acc_full, 1);
            mbar_init(acc_free, kQtWarps);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        w = qt_begin(p.shares, cluster_id());
        __syncwarp();
    } else if (warp == kQtWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(&tmem_slot)), "r"(p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        w = qt_begin(p.shares, cluster_id());
    } else {
        w = qt_begin(p.shares, cluster_id());
        if (warp < w.r) load_pow();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot), tmem_a = tmem + (uint32_t)p.N;
    if (warp < kQtWarps) {
        const uint32_t lanes = (uint32_t)((warp & 3) * 32 + (warp >> 2) * 16) << 16;  // tensor memory lanes of this warp's row tile
        const int g = lane >> 2, t = lane & 3;
        QtUnpack u{ring, tile_bar, tile_free, full, free, tmem_a + lanes, p.ring, p.slot_bytes, p.stages, 0, 0, 0u, 0u};
        unsigned accpar = 0;
        bool waited = false;
        while (w.r > 0) {
            const int type = warp < w.r ? p.type[qt_seg(p, w.lo + warp)] : 0;
            const bool wide = P.wide(type, PRECISE);
            if (lane == 0) walk_s[warp] = w;
            __syncwarp();
            if (type == 0)
                qt_unpack<0, false>(u, P, nb, fail);
            else if (type == 12 && (PRECISE || wide))
                qt_unpack<12, true>(u, P, nb, fail);
            else if (type == 12)
                qt_unpack<12, PRECISE>(u, P, nb, fail);
            else if (type == 14 && (PRECISE || wide))
                qt_unpack<14, true>(u, P, nb, fail);
            else if (type == 14)
                qt_unpack<14, PRECISE>(u, P, nb, fail);
            else if (wide)
                qt_unpack<8, true>(u, P, nb, fail);
            else
                qt_unpack<8, false>(u, P, nb, fail);
            if (!waited) {  // what earlier kernels wrote and read is done with
                pdl_wait();
                waited = true;
            }
            {
                const volatile QtWalk &v = walk_s[warp];
                w = QtWalk{v.f, v.end, v.block, v.lo, v.r};
            }
            asm volatile("prefetch.global.L1 [%0];" ::"l"(p.scale + min(w.block * p.N + lane * 8, p.n - 1)));
            bar_wait(acc_full, accpar, fail);
            accpar ^= 1u;
            __syncwarp();
            if (warp < w.r) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int col0 = w.block * p.N, cols = min(p.N, p.n - col0), rt = w.lo + warp, seg = qt_seg(p, rt);
                const bool wide = P.wide(p.type[seg], PRECISE);
                const float undo0 = P.undo(0, wide), undo1 = P.undo(1, wide);
#pragma unroll 1
                for (int c = 0; c < cols; c += 16) {
                    uint32_t r[8];
                    tmem_ld_16x16(tmem + lanes + (uint32_t)c, r);
#pragma unroll
                    for (int j = 0; j < 8; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) * (j & 2 ? undo1 : undo0));
                    if (p.splits > 1) {
                        const uint32_t at = x0 + (uint32_t)((c + 2 * t) * kQtLd + warp * 16 + g) * 4;
#pragma unroll
                        for (int j = 0; j < 8; j++)
                            asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + (uint32_t)(((j >> 2) * 8 + (j & 1)) * kQtLd + (j >> 1 & 1) * 8) * 4), "r"(r[j]) : "memory");
                        continue;
                    }
                    float *out = p.out[seg];
                    const int tile_row = (rt - p.rt_begin[seg]) * (p.epi == EPI_SILU_PAIR ? 8 : 16) + g;
#pragma unroll
                    for (int j = 0; j < 4; j++) {  // row of x: c + 8 * (j / 2) + 2t + j % 2
                        const int b = col0 + c + (j >> 1) * 8 + 2 * t + (j & 1);
                        if (b >= p.n) continue;
                        const float sc = p.scale[b], v0 = __uint_as_float(r[(j >> 1) * 4 + (j & 1)]) * sc, v1 = __uint_as_float(r[(j >> 1) * 4 + (j & 1) + 2]) * sc;
                        float *o = out + (size_t)b * p.ld_out + tile_row;
                        if (p.epi == EPI_SILU_PAIR) {  // rows 0-7 of a tile are gate rows, rows 8-15 the matching up rows
                            if (tile_row < p.rows[seg]) *o = __fmul_rn(silu_ref(v0), v1);
                        } else {
                            if (tile_row < p.rows[seg]) o[0] = v0;
                            if (tile_row + 8 < p.rows[seg]) o[8] = v1;
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) qt_arrive(acc_free);
            qt_next(w, p.shares.total_rt);
            if (warp < w.r) load_pow();
        }
    } else if (warp == kQtWarps) {
        pdl_wait();
        pdl_launch_dependents();
        if (lane == 0) {
            int s = 0, issued = 0;
            unsigned par = 0;
            bool ok = true;
            for (; ok && w.r > 0; qt_next(w, p.shares.total_rt))
                for (int k = 0; k < 2 * nb; k++) {
                    if (!(ok = bar_wait(free + s * 8, par ^ 1u, fail))) break;
                    mbar_expect_tx(full + s * 8, x_bytes);
                    const uint32_t dst = x0 + s * x_bytes;
                    tma_2d(dst, &p.tx, (2 * s0 + k) * 128, w.block * p.N, full + s * 8);
                    tma_2d(dst + x_bytes / 2, &p.tx, (2 * s0 + k) * 128 + 64, w.block * p.N, full + s * 8);
                    issued++;
                    if (++s == p.stages) {
                        s = 0;
                        par ^= 1u;
                    }
                }
            issued_s[kQtWarps] = issued;
        }
        __syncwarp();
    } else if (warp == kQtWarps + 1) {
        // D FP32, A and B FP16, M 128; A from the tensor memory, B K-major
        const uint32_t idesc = (1u << 4) | ((uint32_t)(p.N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const bool leader = elect_one();
        int s = 0;
        unsigned par = 0, accpar = 0;
        bool ok = true;
        for (; w.r > 0; qt_next(w, p.shares.total_rt)) {
            ok = bar_wait(acc_free, accpar ^ 1u, fail) && ok;
            accpar ^= 1u;
            for (int k = 0; k < 2 * nb; k++) {
                ok = bar_wait(full + s * 8, par, fail) && ok;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t xd = sw128_desc(x0 + s * x_bytes), xd2 = sw128_desc(x0 + s * x_bytes + x_bytes / 2);
                const uint32_t a = tmem_a + s * 64;
                if (leader && ok) {
#pragma unroll
                    for (int j = 0; j < 8; j++) mma_f16_ts(tmem, a + j * 8, (j < 4 ? xd : xd2) + 2 * (j & 3), idesc, (k > 0 || j > 0) ? 1u : 0u);
                    mma_commit(free + s * 8);
                }
                __syncwarp();
                if (++s == p.stages) {
                    s = 0;
                    par ^= 1u;
                }
            }
            if (leader && ok) mma_commit(acc_full);
            __syncwarp();
        }
        pdl_wait();
    } else {
        // a slot is filled again when its tile is used; nothing can be missing for longer than a wait may take
        int slot = 0;
        unsigned par = 0;
        QtTiles t = tiles_s[owner];
        bool more = lane < kQtWarps && t.w.r > 0;
        long long t0 = clock64();
        while (__any_sync(0xffffffffu, more)) {
            const bool go = more && bar_test(tile_free + slot * 8, par);
            if (go) {
                t.fetch(p, tile_bar + slot * 8, ring + slot * p.slot_bytes);
                if (++slot == p.ring) {
                    slot = 0;
                    par ^= 1u;
                }
                more = t.w.r > 0;
            }
            if (__any_sync(0xffffffffu, go))
                t0 = clock64();
            else if (*fail || clock64() - t0 > kWaitClocks) {
                *fail = 1u;
                more = false;
            }
        }
        if (lane < kQtWarps) issued_s[lane] = t.issued;
        pdl_wait();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*fail) {  // copies and MMAs that were issued before the failure: let them finish (bounded) before memory is given back
        if ((warp == kQtWarps && lane == 0) || (warp == kQtWarps + 2 && lane < kQtWarps)) {
            const int slots = warp == kQtWarps ? p.stages : p.ring;
            const uint32_t bar = warp == kQtWarps ? full : tile_bar;
            bool failed = true;
            const int issued = issued_s[warp == kQtWarps ? kQtWarps : lane];
            for (int j = ring_open(issued, 0, slots); j < issued; j++) mbar_wait_bounded(bar + j % slots * 8, ring_parity(j, slots), 0, p.err, failed);
        }
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {
        }
        if (tid == 0) *reinterpret_cast<volatile unsigned *>(p.err) = 1u | blockIdx.x << 16;
    }
    if (warp == kQtWarps + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
    }
    if (p.splits == 1) return;
    // a cluster that shares K has one piece; four outputs at a time, a contiguous range of them per CTA
    w = qt_begin(p.shares, cluster_id());
    const int sh = p.epi == EPI_SILU_PAIR ? 1 : 2, col0 = w.block * p.N, per = w.r << sh, total = per * min(p.N, p.n - col0), chunk = (total + p.splits - 1) / p.splits;
    const int first = cluster_rank() * chunk, last = min(total, first + chunk);
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int idx = first + tid; idx < last; idx += kQtThreads) {
        const int c = idx / per, q = idx - c * per, l = q >> sh, row = (q - (l << sh)) * 4, rt = w.lo + l, seg = qt_seg(p, rt);
        const int orow = ((rt - p.rt_begin[seg]) << (sh + 2)) + row, b = col0 + c;
        const uint32_t at = x0 + (uint32_t)(c * kQtLd + l * 16 + row) * 4;
        const float sc = p.scale[b];
        float4 v = qt_peer_sum(at, p.splits);
        v = make_float4(v.x * sc, v.y * sc, v.z * sc, v.w * sc);
        if (p.epi == EPI_SILU_PAIR) {  // rows 0-7 of a tile are gate rows, rows 8-15 the matching up rows
            const float4 u = qt_peer_sum(at + 32, p.splits);
            v = make_float4(__fmul_rn(silu_ref(v.x), u.x * sc), __fmul_rn(silu_ref(v.y), u.y * sc), __fmul_rn(silu_ref(v.z), u.z * sc), __fmul_rn(silu_ref(v.w), u.w * sc));
        }
        float *o = p.out[seg] + (size_t)b * p.ld_out + orow;
        if (orow + 3 < p.rows[seg] && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
            *reinterpret_cast<float4 *>(o) = v;
        } else {
            const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (orow + k < p.rows[seg]) o[k] = e[k];
        }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while its shared memory may still be read
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

// Clusters of every size that the device holds at a time, one CTA per SM (the driver counts no more for a kernel that allocates tensor memory; two
// do run on an SM when they have half of it each); 0 for a size that it does not take.
static int qt_clusters(juno_ctx *c, int (&fit)[kQtMaxSplit + 1]) {
    static std::mutex mu;
    static int known[16][kQtMaxSplit + 1] = {{0}};
    std::lock_guard<std::mutex> lk(mu);
    int *f = known[c->device & 15];
    if (f[1] == 0) {
        JUNO_CUDA_TRY(cudaFuncSetAttribute(gemm_quant_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kQtOneSmem));
        JUNO_CUDA_TRY(cudaFuncSetAttribute(gemm_quant_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kQtOneSmem));
        for (int s = kQtMaxSplit; s >= 1; s--) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)s);
            cfg.blockDim = dim3(kQtThreads);
            cfg.dynamicSmemBytes = kQtOneSmem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)s;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            f[s] = 0;
            if (cudaOccupancyMaxActiveClusters(&f[s], gemm_quant_kernel<true>, &cfg) != cudaSuccess) {
                cudaGetLastError();
                f[s] = 0;
            }
        }
    }
    std::copy(f, f + kQtMaxSplit + 1, fit);
    return JUNO_OK;
}

int launch_gemm_quant(juno_ctx *c, const GemmQuantArgs &a, cudaStream_t st) {
    JUNO_REQUIRE(a.n >= 1 && a.K > 0 && a.K % 256 == 0 && a.x && a.scale && a.nseg >= 1 && a.nseg <= 3, "quantised product: bad arguments (K=%d, n=%d)", a.K, a.n);
    GemmQuantParams p;
    memset((void *)&p, 0, sizeof(p));
    int rt = 0, first_type = 0;
    double algo = (double)a.n * a.K * 2;
    for (int s = 0; s < a.nseg; s++) {
        const GemvSeg &g = a.seg[s];
        JUNO_REQUIRE(g.w && g.row_pow && g.out && (g.type == 12 || g.type == 14 || g.type == 8), "quantised product: type %d has no tiles", g.type);
        p.w[s] = g.w;
        p.pow[s] = g.row_pow;
        p.out[s] = g.out;
        p.rows[s] = g.rows;
        p.type[s] = g.type;
        p.rt_begin[s] = rt;
        rt += g.row_tiles;
        p.slot_bytes = std::max(p.slot_bytes, tile_bytes(g.type));
        if (!first_type) first_type = g.type;
        const double bpw = g.type == 12 ? 144.0 / 256 : g.type == 14 ? 210.0 / 256 : 34.0 / 32;
        algo += (double)g.rows * a.K * bpw * (a.epi == EPI_SILU_PAIR ? 2 : 1) + (double)a.n * g.rows * 4;
    }
    for (int s = a.nseg; s < 4; s++) p.rt_begin[s] = s < 3 ? 0x7fffffff : rt;
    p.nb = a.K / 256;
    p.n = a.n;
    p.ld_out = a.ld_out;
    p.epi = a.epi;
    p.scale = a.scale;
    p.err = c->gemv_scratch.qerr;
    QuantSplit q = quant_passes(a.n);
    p.N = q.N;
    // half an SM per CTA (the next kernel's copies start while this one ends, and one CTA's exchange hides behind the other's products),
    // as long as the sums and two stages fit half of the tensor memory
    const bool pair = p.N <= 128 && (size_t)p.slot_bytes * 2 * kQtWarps + 2 * (size_t)p.N * 256 + 1024 <= kQtPairSmem;
    int fit[kQtMaxSplit + 1];
    JUNO_TRY(qt_clusters(c, fit));
    quant_split(q, rt, p.nb, pair, fit);
    JUNO_REQUIRE(q.splits > 0, "quantised product: no cluster fits device %d", c->device);
    p.splits = q.splits;
    p.shares = quant_shares(q, rt);
    p.blocks = even_shares(p.nb, q.splits);
    const size_t budget = pair ? kQtPairSmem : kQtOneSmem, x_bytes = (size_t)p.N * 256;
    // stages before tiles in flight: as many as the tensor memory holds beside the sums
    p.tmem_cols = pair ? 256 : 512;
    p.stages = std::min(kQtMaxStages, (p.tmem_cols - p.N) / 64);
    while (p.stages > 2 && (size_t)kQtWarps * 2 * p.slot_bytes + p.stages * x_bytes + 1024 > budget) p.stages--;
    p.ring = 2;
    while (p.ring < kQtMaxRing && (size_t)kQtWarps * (p.ring + 1) * p.slot_bytes + p.stages * x_bytes + 1024 <= budget) p.ring++;
    const size_t ring = (size_t)kQtWarps * p.ring * p.slot_bytes;
    size_t smem = 1024 + ring + p.stages * x_bytes;
    if (p.splits > 1) smem = std::max(smem, 1024 + (size_t)p.N * kQtLd * 4);
    JUNO_REQUIRE(p.stages >= 2 && smem <= budget, "quantised product: %d rows do not fit shared memory", p.N);
    JUNO_TRY(tensor_map_bf16(&p.tx, a.x, a.n, a.K, a.K, p.N));
    ProfScope prof(c, st, first_type == 12 ? PROF_GEMV_Q4K : first_type == 14 ? PROF_GEMV_Q6K : PROF_GEMV_Q80, algo), prof_tc(c, st, PROF_GEMM_TC, algo);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(q.clusters * q.splits));
    cfg.blockDim = dim3(kQtThreads);
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
    JUNO_CUDA_TRY(cudaLaunchKernelEx(&cfg, a.precise ? gemm_quant_kernel<true> : gemm_quant_kernel<false>, p));
    c->kernel_launches++;
    return JUNO_OK;
}

}  // namespace juno
