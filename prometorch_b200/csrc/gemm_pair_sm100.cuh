// The same product by pairs of SMs: two CTAs of a cluster compute a 256 x 256 tile with tcgen05.mma.cta_group::2, each holding its 128
// rows of A, half of B's 256 rows, and the accumulators of its own rows.  A k-block moves 32 KB into each SM where a CTA with a 128 x 256
// tile of its own moves 48 KB for the same products; the latter is bound by that traffic (it asks for about 96 bytes a clock and SM of L2).
// Measured: 8192 x 11264 x 2048 298 -> 249 us (1520 TFLOP/s), 8192 x 32000 x 2048 1064 -> 722 us, 4096 x 4096 x 12288 640 -> 398 us, cut 349 us.
// The tiles that do not fill a wave are cut along K (`splits` items each, fp32 partials to `work`, then pair_reduce_kernel), so that
// a shape with few tiles still uses every pair.  All loads are plain (no multicast): the CTAs fetch disjoint halves.
#pragma once
#include "gemm_sm100.cuh"

namespace ptb {
namespace gemm {

constexpr int PAIR_M = 256, PAIR_N = 256, PAIR_STAGES = 6;
constexpr int PAIR_HALF = 128 * BK * 2;                      // one CTA's part of A, and of B, per k-block
constexpr int PAIR_STAGE = 2 * PAIR_HALF;
constexpr int PAIR_SMEM = PAIR_STAGES * PAIR_STAGE + 256 + 1024;

struct PairParams {
    int M, N, K;
    void* C;
    long long ldc;
    const float* bias;
    int flags;                 // EPI_BIAS | EPI_ACCUM | EPI_OUT_F32 | EPI_GELU | EPI_RELU2
    int* status;
    int tiles_m, tiles_n;
    int whole;                 // tiles [0, whole) run over all of K; the rest are cut
    int splits, kb_per_split;  // of a cut tile
    float* work;               // [cut tile][split][8 pieces of 32 columns][8 groups of 4][256 rows][4]
    int pdl;
};

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// A load into this CTA's memory whose bytes are counted by a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)), "l"(map),
        "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives at the barrier at this place in both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}

// bias, activation, sum with what C holds, and the store of 32 neighbouring values of a row.
__device__ __forceinline__ void pair_store(const PairParams& P, int row, int col, float* v, bool wide) {
    if (row >= P.M || col >= P.N) return;
    if (P.flags & EPI_BIAS) {
#pragma unroll
        for (int j = 0; j < 32; ++j) if (col + j < P.N) v[j] += P.bias[col + j];
    }
    if (P.flags & EPI_GELU) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
    }
    if (P.flags & EPI_RELU2) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = relu2(v[j]);
    }
    const bool full = col + 32 <= P.N;
    if (P.flags & EPI_OUT_F32) {
        float* cp = reinterpret_cast<float*>(P.C) + (size_t)row * P.ldc + col;
        if (full) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                float4 o = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                if (P.flags & EPI_ACCUM) { const float4 p = *reinterpret_cast<float4*>(cp + j); o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w; }
                *reinterpret_cast<float4*>(cp + j) = o;
            }
        } else {
            for (int j = 0; j < 32 && col + j < P.N; ++j) cp[j] = (P.flags & EPI_ACCUM) ? cp[j] + v[j] : v[j];
        }
        return;
    }
    __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(P.C) + (size_t)row * P.ldc + col;
    if (!full) {
        for (int j = 0; j < 32 && col + j < P.N; ++j) cp[j] = __float2bfloat16_rn((P.flags & EPI_ACCUM) ? __bfloat162float(cp[j]) + v[j] : v[j]);
        return;
    }
    if (P.flags & EPI_ACCUM) {
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            const uint4 pv = *reinterpret_cast<uint4*>(cp + j);
            const __nv_bfloat162* ph = reinterpret_cast<const __nv_bfloat162*>(&pv);
#pragma unroll
            for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(ph[e]); v[j + 2 * e] += f.x; v[j + 2 * e + 1] += f.y; }
        }
    }
#pragma unroll
    for (int j = 0; j < 32; j += 16) {
        uint4 o[2];
        __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
        for (int e = 0; e < 8; ++e) oh[e] = __floats2bfloat162_rn(v[j + 2 * e], v[j + 2 * e + 1]);
        if (wide) {
            st_global_32(cp + j, o[0], o[1]);
        } else {
            *reinterpret_cast<uint4*>(cp + j) = o[0];
            *reinterpret_cast<uint4*>(cp + j + 8) = o[1];
        }
    }
}
__device__ __forceinline__ bool pair_wide(const PairParams& P) { return P.ldc % 16 == 0 && ((uintptr_t)P.C & 31) == 0; }

template <bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const __grid_constant__ PairParams P) {
    extern __shared__ uint8_t smem_raw[];
    // the offset of the tiles is the same in both CTAs: the dynamic part starts at the same place
    uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + PAIR_STAGES * PAIR_STAGE);   // of the first CTA: both CTAs' loads
    uint64_t* empty = full + PAIR_STAGES;
    uint64_t* acc_full = empty + PAIR_STAGES;      // [2]
    uint64_t* acc_empty = acc_full + 2;            // [2], of the first CTA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = (int)blockIdx.x >> 1, n_pairs = (int)gridDim.x >> 1;
    const int kblocks = (P.K + BK - 1) / BK, tiles = P.tiles_m * P.tiles_n, cut = tiles - P.whole;
    const int items = P.whole + cut * P.splits;
    struct Item { int m0, n0, kb_lo, kb_hi, slot; };
    auto item = [&](int w) {
        Item it;
        int tile = w, sp = 0;
        it.slot = -1;
        if (w >= P.whole) {
            const int x = w - P.whole;
            sp = x / cut;
            tile = P.whole + x % cut;
            it.slot = (x % cut) * P.splits + sp;
        }
        it.m0 = (tile % P.tiles_m) * PAIR_M;
        it.n0 = (tile / P.tiles_m) * PAIR_N;
        it.kb_lo = it.slot < 0 ? 0 : sp * P.kb_per_split;
        it.kb_hi = it.slot < 0 ? kblocks : min(kblocks, it.kb_lo + P.kb_per_split);
        return it;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < PAIR_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * EPI_WARPS); }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&mapA);
        prefetch_tmap(&mapB);
    }
    if (P.pdl) pdl_launch_dependents();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                            // both CTAs' barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (of both CTAs)
        if (lane == 0) {
            int n = 0;
            bool ok = true;
            if (P.pdl) pdl_wait();
            for (int w = pair; w < items && ok; w += n_pairs) {
                const Item it = item(w);
                const int m0 = it.m0 + (int)rank * 128, n0 = it.n0 + (int)rank * 128;
                for (int kb = it.kb_lo; kb < it.kb_hi && ok; ++kb, ++n) {
                    const int s = n % PAIR_STAGES;
                    if (n >= PAIR_STAGES) ok = mbar_wait(&empty[s], (uint32_t)(((n / PAIR_STAGES) - 1) & 1), P.status);
                    if (!ok) break;
                    uint8_t* sa = smem + s * PAIR_STAGE;
                    uint8_t* sb = sa + PAIR_HALF;
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * PAIR_STAGE);
                    const uint32_t bar = mapa_u32(smem_u32(&full[s]), 0);
                    if (A_MN) {
                        for (int c = 0; c < 2; ++c) tma_load_2d_pair(sa + c * 8192, &mapA, m0 + c * 64, kb * BK, bar);
                    } else {
                        tma_load_2d_pair(sa, &mapA, kb * BK, m0, bar);
                    }
                    if (B_MN) {
                        for (int c = 0; c < 2; ++c) tma_load_2d_pair(sb + c * 8192, &mapB, n0 + c * 64, kb * BK, bar);
                    } else {
                        tma_load_2d_pair(sb, &mapB, kb * BK, n0, bar);
                    }
                }
            }
            if (!ok) *abort_flag = 1;
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (of the first CTA)
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = instr_desc(PAIR_M, PAIR_N, A_MN ? 1 : 0, B_MN ? 1 : 0);
            int n = 0, tl = 0;
            bool ok = true;
            for (int w = pair; w < items && ok; w += n_pairs, ++tl) {
                const Item it = item(w);
                const int b = tl & 1;
                if (tl >= 2) ok = mbar_wait(&acc_empty[b], (uint32_t)(((tl >> 1) - 1) & 1), P.status);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(b * PAIR_N);
                for (int kb = it.kb_lo; kb < it.kb_hi && ok; ++kb, ++n) {
                    const int s = n % PAIR_STAGES;
                    ok = mbar_wait(&full[s], (uint32_t)((n / PAIR_STAGES) & 1), P.status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + s * PAIR_STAGE), sb = sa + PAIR_HALF;
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        const uint64_t da = A_MN ? smem_desc(sa + k * 2048, 8192, 1024) : smem_desc(sa + k * 32, 16, 1024);
                        const uint64_t db = B_MN ? smem_desc(sb + k * 2048, 8192, 1024) : smem_desc(sb + k * 32, 16, 1024);
                        umma_bf16_pair(d_tmem, da, db, idesc, (kb > it.kb_lo || k > 0) ? 1u : 0u);
                    }
                    umma_commit_pair(&empty[s]);
                }
                if (ok) umma_commit_pair(&acc_full[b]);
            }
            if (!ok) *abort_flag = 1;
        }
    } else {
        // ------------------------------------------------------------------ epilogue (warps 2..9), each CTA its own 128 rows
        const int q = warp & 3;
        const bool wide = pair_wide(P);
        int tl = 0;
        bool ok = true;
        for (int w = pair; w < items && ok; w += n_pairs, ++tl) {
            const Item it = item(w);
            const int b = tl & 1;
            ok = mbar_wait(&acc_full[b], (uint32_t)((tl >> 1) & 1), P.status);
            if (!ok) break;
            tc_fence_after();
            const int in_tile = (int)rank * 128 + q * 32 + lane;
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * PAIR_N);
            const int c_lo = warp < 6 ? 0 : PAIR_N / 2;
#pragma unroll 1
            for (int c = c_lo; c < c_lo + PAIR_N / 2; c += 32) {
                float v[32];
                tmem_ld32(taddr + c, reinterpret_cast<uint32_t*>(v));
                tmem_ld_wait();
                if (it.slot < 0) {
                    pair_store(P, it.m0 + in_tile, it.n0 + c, v, wide);
                } else {
                    float4* wk = reinterpret_cast<float4*>(P.work) + ((size_t)it.slot * 64 + c / 4) * 256 + in_tile;
#pragma unroll
                    for (int j = 0; j < 8; ++j) wk[(size_t)j * 256] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[b]), 0));
        }
        if (!ok) *abort_flag = 1;
    }
    // ---- teardown: no CTA leaves while the other may still arrive at its barriers or use its tensor memory
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

// The cut tiles: the sum of their partials, and what the epilogue does with it.  One CTA per tile and 32 columns, a thread per row.
__global__ void __launch_bounds__(256) pair_reduce_kernel(const __grid_constant__ PairParams P) {
    pdl_wait();
    pdl_launch_dependents();
    const int piece = blockIdx.x & 7, ct = (int)blockIdx.x >> 3, tile = P.whole + ct;
    const int row = (tile % P.tiles_m) * PAIR_M + (int)threadIdx.x, col = (tile / P.tiles_m) * PAIR_N + piece * 32;
    if (row >= P.M || col >= P.N) return;
    const float4* wk = reinterpret_cast<const float4*>(P.work) + ((size_t)ct * P.splits * 64 + piece * 8) * 256 + threadIdx.x;
    float v[32];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float4 a = wk[(size_t)j * 256];
        v[4 * j] = a.x; v[4 * j + 1] = a.y; v[4 * j + 2] = a.z; v[4 * j + 3] = a.w;
    }
    for (int s = 1; s < P.splits; ++s) {
        const float4* ws = wk + (size_t)s * 64 * 256;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 a = ws[(size_t)j * 256];
            v[4 * j] += a.x; v[4 * j + 1] += a.y; v[4 * j + 2] += a.z; v[4 * j + 3] += a.w;
        }
    }
    pair_store(P, row, col, v, pair_wide(P));
}

}  // namespace gemm
}  // namespace ptb
