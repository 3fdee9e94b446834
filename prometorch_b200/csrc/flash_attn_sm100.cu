// FlashAttention on the 5th-generation tensor cores: both products of every 128 x 128 block run as
// tcgen05.mma with accumulators in tensor memory, operands arrive by TMA.
//
// Forward of grids that fill the GPU (others: flash_attn_tile_sm100.cuh): one CTA per two tiles of 128 query rows that read the same keys: the same rows of two
// heads of a group where the group's size is even, else 256 consecutive rows of one head.  Ten warps:
//   warp 8   TMA producer: both Q tiles once, then K and V tiles of 128 keys through two-stage rings;
//   warp 9   owns tensor memory and issues the MMAs.  Tile t has 128 columns for its scores S_t and D for its output O_t; for every
//            block j it issues, tile by tile, O_t += P_t(j) V_j and then S_t(j+1) = Q_t K_j+1^T, so that one tile's products run
//            under the other tile's softmax;
//   warps 0-3, 4-7   softmax of tile 0 and tile 1.  A thread owns one query row (its tensor-memory lane): it reads the 128 scores
//            with tcgen05.ld and writes the bf16 probabilities over them (tcgen05.st): they are the A operand of the second product
//            from tensor memory, and no other thread takes part in a row's maximum or sum.
// The completion of S_t(j) implies that of O_t's product with block j-1, issued before it, so until P_t(j) is published the softmax
// warps own O_t too.  They scale it whenever a row's maximum has grown, once the block's scores have left their registers.  Scaling only after a growth
// by 2^8 saves 1.7 % of the time but costs precision: under the true maximum the large weights lie just below a power of two, where
// a bf16 step is smallest beside the value (error of the output against 64 bits, 2049 queries, causal: 2.07e-3 against 2.03e-3, with scores three
// times as large 2.11e-3 against 1.77e-3).
// Causal masking and the sequence end are applied to the blocks that need them only.  Every wait is
// bounded.  Measured (2 x 4001 queries, 32 heads over 8, size 128, causal): 479 us with one tile a CTA, weights through shared memory and
// outputs in registers, 332 us now (790 TFLOP/s); 4 x 2048, 32 heads over 4, size 64: 245 -> 161 us, bound by the exponentials.  The reference's kernel is aten/src/ATen/cuda/FlashAttention.cu:83-258 (one thread per row).
#include "gemm_sm100.cuh"

int ptb_make_tmap_bf16(CUtensorMap* map, const void* base, long long inner, long long outer, long long ld, int box_inner, int box_outer);
int ptb_make_tmap_bf16_3d(CUtensorMap* map, const void* base, long long n0, long long n1, long long n2, int b0, int b1, int b2);
int ptb_make_tmap_f32_3d(CUtensorMap* map, const void* base, long long n0, long long n1, long long n2, int b0, int b1);

namespace ptb {
namespace fa100 {

using namespace ptb::gemm;

constexpr int BQ = 128, BKV = 128;
constexpr int NTHREADS = 320;

struct Params {
    __nv_bfloat16* O;        // [B, Tq, H, D]
    float* lse;              // [B, H, Tq] natural-log sum of exponentials, or null
    const int* cu;           // [B + 1] first row of each sequence in packed q, k and v (then Tq and Tk are read from it), or null
    int B, Tq, Tk, H, Hk;
    int causal, q_offset;
    float scale_log2;        // softmax scale x log2(e)
    int pair_heads;          // the CTA's tiles are two heads (else two row blocks)
    int units;               // CTAs per row block: B times heads (pairs of heads)
    int* status;
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)), "l"(map),
                 "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}

template <int D>
struct Sm {
    static constexpr int Q_BYTES = BQ * D * 2;
    static constexpr int KV_BYTES = BKV * D * 2;
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_K = OFF_Q + 2 * Q_BYTES;
    static constexpr int OFF_V = OFF_K + 2 * KV_BYTES;
    static constexpr int OFF_BAR = OFF_V + 2 * KV_BYTES;
    static constexpr int TOTAL = OFF_BAR + 256 + 1024;
};

// D = A B with A (bf16, lane = row, two values of K a column) in tensor memory.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <int D>
__global__ void __launch_bounds__(NTHREADS, 1)
fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
           const __grid_constant__ Params P) {
    using S = Sm<D>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sq = smem + S::OFF_Q;
    uint8_t* sk = smem + S::OFF_K;
    uint8_t* sv = smem + S::OFF_V;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    uint64_t* q_full = bars;             // [1]
    uint64_t* k_full = bars + 1;         // [2]
    uint64_t* k_empty = bars + 3;        // [2]
    uint64_t* v_full = bars + 5;         // [2]
    uint64_t* v_empty = bars + 7;        // [2]
    uint64_t* s_full = bars + 9;         // [2] tile t's scores are in tensor memory
    uint64_t* p_ready = bars + 11;       // [2] tile t's weights are (4 arrivals, one per warp)
    uint64_t* o_full = bars + 13;        // [2] tile t's output is complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // late row blocks (the long ones under a causal mask) first, over all heads and sequences
    const int n_rb = (int)gridDim.x / P.units;
    const int rb = n_rb - 1 - (int)blockIdx.x / P.units, unit = (int)blockIdx.x % P.units;
    const int per_b = P.units / P.B, b = unit / per_b;
    const int rows_per = P.pair_heads ? BQ : 2 * BQ;
    const int h0 = (unit % per_b) * (P.pair_heads ? 2 : 1), hk = h0 / (P.H / P.Hk);
    int Tq = P.Tq, Tk = P.Tk, qrow = b * P.Tq, krow = b * P.Tk;
    if (P.cu) {
        qrow = krow = P.cu[b];
        Tq = Tk = P.cu[b + 1] - qrow;
    }
    const int q0 = rb * rows_per;
    if (q0 >= Tq) return;                 // a shorter sequence than the longest
    // blocks of keys that tile t can see
    auto tile_q0 = [&](int t) { return P.pair_heads ? q0 : q0 + t * BQ; };
    auto tile_blocks = [&](int t) {
        const int tq0 = tile_q0(t);
        if (tq0 >= Tq) return 0;
        const int end = P.causal ? min(Tk, min(tq0 + BQ, Tq) + P.q_offset) : Tk;
        return max(0, (end + BKV - 1) / BKV);
    };
    const int n0 = tile_blocks(0), n1 = tile_blocks(1), nblk = max(n0, n1);

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
            mbar_init(&s_full[s], 1); mbar_init(&p_ready[s], 4); mbar_init(&o_full[s], 1);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmQ);
        prefetch_tmap(&tmK);
        prefetch_tmap(&tmV);
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    constexpr uint32_t TM_O = 256;                                 // S_t (and P_t over it) at 128 t, O_t at 256 + D t

    if (warp == 8) {
        // ---------------------------------------------------------------------------- TMA producer
        if (lane == 0 && nblk > 0) {
            bool ok = true;
            mbar_expect_tx(q_full, 2 * S::Q_BYTES);
            for (int t = 0; t < 2; ++t)
                for (int kb = 0; kb < D / 64; ++kb)
                    tma_load_2d(sq + t * S::Q_BYTES + kb * (BQ * 128), &tmQ, (h0 + (P.pair_heads ? t : 0)) * D + kb * 64, qrow + tile_q0(t), q_full);
            for (int j = 0; j < nblk && ok; ++j) {
                const int s = j & 1;
                if (j >= 2) ok = mbar_wait(&k_empty[s], (uint32_t)(((j >> 1) - 1) & 1), P.status);
                if (!ok) break;
                mbar_expect_tx(&k_full[s], S::KV_BYTES);
                for (int kb = 0; kb < D / 64; ++kb)
                    tma_load_2d(sk + s * S::KV_BYTES + kb * (BKV * 128), &tmK, hk * D + kb * 64, krow + j * BKV, &k_full[s]);
                if (j >= 2) ok = mbar_wait(&v_empty[s], (uint32_t)(((j >> 1) - 1) & 1), P.status);
                if (!ok) break;
                mbar_expect_tx(&v_full[s], S::KV_BYTES);
                for (int hh = 0; hh < 2; ++hh)                       // two halves of 64 keys, each D/64 chunks of [64 keys x 64 dims]
                    for (int c = 0; c < D / 64; ++c)
                        tma_load_2d(sv + s * S::KV_BYTES + hh * (D / 64) * 8192 + c * 8192, &tmV, hk * D + c * 64, krow + j * BKV + hh * 64,
                                    &v_full[s]);
            }
            if (!ok) *abort_flag = 1;
        }
    } else if (warp == 9) {
        // ---------------------------------------------------------------------------- MMA issuer
        if (lane == 0 && nblk > 0) {
            constexpr uint32_t idesc_s = instr_desc(BQ, BKV, 0, 0);          // S = Q K^T: both K-major
            constexpr uint32_t idesc_o = instr_desc(BQ, D, 0, 1);            // O = P V: V MN-major
            auto issue_s = [&](int t, int j) {
                const int s = j & 1;
                const uint32_t a0 = smem_u32(sq + t * S::Q_BYTES), b0 = smem_u32(sk + s * S::KV_BYTES);
#pragma unroll
                for (int kb = 0; kb < D / 64; ++kb)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base + (uint32_t)(t * BKV), smem_desc(a0 + kb * (BQ * 128) + k * 32, 16, 1024),
                                  smem_desc(b0 + kb * (BKV * 128) + k * 32, 16, 1024), idesc_s, (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(&s_full[t]);
            };
            bool ok = mbar_wait(q_full, 0, P.status) && mbar_wait(&k_full[0], 0, P.status);
            if (ok) {
                tc_fence_after();
                if (n0 > 0) issue_s(0, 0);
                if (n1 > 0) issue_s(1, 0);
                umma_commit(&k_empty[0]);
            }
            for (int j = 0; j < nblk && ok; ++j) {
                const int s = j & 1;
                ok = mbar_wait(&v_full[s], (uint32_t)((j >> 1) & 1), P.status);
                bool have_k = j + 1 >= nblk;
                for (int t = 0; t < 2 && ok; ++t) {
                    const int nt = t ? n1 : n0;
                    if (j >= nt) continue;
                    ok = mbar_wait(&p_ready[t], (uint32_t)(j & 1), P.status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t b0 = smem_u32(sv + s * S::KV_BYTES);
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_bf16_ts(tmem_base + TM_O + (uint32_t)(t * D), tmem_base + (uint32_t)(t * BKV + (hh * 4 + k) * 8),
                                         smem_desc(b0 + hh * (D / 64) * 8192 + k * 2048, 8192, 1024), idesc_o, (j > 0 || hh > 0 || k > 0) ? 1u : 0u);
                    if (j + 1 < nt) {
                        if (!have_k) {
                            ok = mbar_wait(&k_full[s ^ 1], (uint32_t)(((j + 1) >> 1) & 1), P.status);
                            if (!ok) break;
                            tc_fence_after();
                            have_k = true;
                        }
                        issue_s(t, j + 1);
                    } else {
                        umma_commit(&o_full[t]);
                    }
                }
                umma_commit(&v_empty[s]);
                if (j + 1 < nblk) umma_commit(&k_empty[s ^ 1]);
            }
            if (!ok) *abort_flag = 1;
        }
    } else {
        // ---------------------------------------------------------------------------- softmax warps
        const int t = warp >> 2;                         // tile
        const int row = 32 * (warp & 3) + lane;          // query row inside the tile = tensor-memory lane
        const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16);
        const uint32_t tm_s = lane_addr + (uint32_t)(t * BKV), tm_o = lane_addr + TM_O + (uint32_t)(t * D);
        const int tq0 = tile_q0(t), nt = t ? n1 : n0;
        const int q_pos = tq0 + row + P.q_offset;        // position of this query among the keys
        float m_run = -INFINITY, l_run = 0.f;
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < nt; ++j) {
            if (ok && !*abort_flag) ok = mbar_wait(&s_full[t], (uint32_t)(j & 1), P.status);
            else ok = false;
            tc_fence_after();
            float sc[128];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(tm_s + (uint32_t)(c * 32), reinterpret_cast<uint32_t*>(sc) + c * 32);
            tmem_ld_wait();
            float f = P.scale_log2;
            if (f <= 0.f) {                               // not the usual case: the maximum is that of the scaled scores
#pragma unroll
                for (int i = 0; i < 128; ++i) sc[i] *= f;
                f = 1.f;
            }
            const int key0 = j * BKV;
            if ((key0 + BKV > Tk) || (P.causal && key0 + BKV - 1 > tq0 + P.q_offset)) {
                const int last = P.causal ? min(Tk - 1, q_pos) : Tk - 1;          // last key of this row
#pragma unroll
                for (int i = 0; i < 128; ++i)
                    if (key0 + i > last) sc[i] = -INFINITY;
            }
            float m8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) m8[i] = sc[i];
#pragma unroll
            for (int i = 8; i < 128; ++i) m8[i & 7] = fmaxf(m8[i & 7], sc[i]);
            const float m_blk = fmaxf(fmaxf(fmaxf(m8[0], m8[1]), fmaxf(m8[2], m8[3])), fmaxf(fmaxf(m8[4], m8[5]), fmaxf(m8[6], m8[7]))) * f;
            float alpha = 1.f;
            const bool grown = __any_sync(0xffffffffu, m_blk > m_run);
            if (grown) {
                const float m_new = fmaxf(m_run, m_blk);
                if (m_new != -INFINITY) alpha = exp2f(m_run - m_new);
                m_run = m_new;
                l_run *= alpha;
            }
            const float m_use = m_run == -INFINITY ? 0.f : m_run;
            float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t pk[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float p0 = exp2f(sc[c * 64 + 2 * i] * f - m_use), p1 = exp2f(sc[c * 64 + 2 * i + 1] * f - m_use);
                    l4[i & 3] += p0 + p1;
                    const __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);
                    pk[i] = *reinterpret_cast<const uint32_t*>(&h2);
                }
                tmem_st32(tm_s + (uint32_t)(c * 32), pk);
            }
            l_run += (l4[0] + l4[1]) + (l4[2] + l4[3]);
            if (grown && j > 0) {             // after the exponentials: the scores' registers are free
#pragma unroll
                for (int c = 0; c < D / 32; ++c) {
                    uint32_t r[32];
                    tmem_ld32(tm_o + (uint32_t)(c * 32), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
                    tmem_st32(tm_o + (uint32_t)(c * 32), r);
                }
            }
            if (key0 + BKV > Tk) {
                // rows of V past the end belong to the next sequence: their weights are zero, but zero times what is not finite is not
                if (ok) ok = mbar_wait(&v_full[j & 1], (uint32_t)((j >> 1) & 1), P.status);
                if (key0 + row >= Tk && ok) {
                    uint8_t* vr = sv + (j & 1) * S::KV_BYTES + (row >> 6) * (D / 64) * 8192 + (row & 63) * 128;
#pragma unroll
                    for (int i = 0; i < D / 8; ++i) *reinterpret_cast<uint4*>(vr + (i >> 3) * 8192 + (i & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_proxy_async();
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[t]);
        }
        if (nt > 0) {
            if (ok && !*abort_flag) ok = mbar_wait(&o_full[t], 0, P.status);
            else ok = false;
            tc_fence_after();
        }
        const int q_idx = tq0 + row, h = h0 + (P.pair_heads ? t : 0);
        const bool valid = q_idx < Tq && ok;
        const float inv = l_run > 0.f ? 1.0f / l_run : l_run == 0.f ? 0.f : l_run;        // a sum that is not a number stays one
        __nv_bfloat16* op = P.O + ((size_t)(qrow + q_idx) * P.H + h) * D;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
            uint32_t r[32];
            if (nt > 0) {
                tmem_ld32(tm_o + (uint32_t)(c * 32), r);
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = 0;
            }
            if (valid) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    uint4 o;
                    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                    for (int e = 0; e < 4; ++e) oh[e] = __floats2bfloat162_rn(__uint_as_float(r[i + 2 * e]) * inv, __uint_as_float(r[i + 2 * e + 1]) * inv);
                    *reinterpret_cast<uint4*>(op + c * 32 + i) = o;
                }
            }
        }
        if (valid && P.lse) P.lse[((size_t)b * P.H + h) * P.Tq + q_idx] = l_run > 0.f ? m_run * 0.6931471805599453f + logf(l_run) : -INFINITY;
        if (!ok) *abort_flag = 1;
    }
    // ---- teardown
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem_base, 512);
}

}  // namespace fa100
}  // namespace ptb

#include "flash_attn_tile_sm100.cuh"

namespace ptb {
namespace fa100 {

// Which kernel: in units of a one-tile CTA's time a two-tile CTA takes about 4/3 (1.27 to 1.5 measured where both fit the GPU at once), so what counts is the
// waves.  One tile where it takes 3/4 of its waves or less: all grids that fit at once (1 x 4001 queries, 2 heads, size 128, causal: 63.5 us with one tile, 84.0 with
// two; 4 x 17 over 2000 keys, 16 heads: 36.9 and 45.1), and up to 128 rows of heads without a partner, whose second tile would be empty (16 x 100, 12 heads,
// size 64: 17.2 and 20.4).  Just past it (192 against 96 CTAs) two tiles are 0 to 41 % faster, at 512 against 256 between 18 and 62 %.
static bool pairs_of_heads(int H, int Hk) { return (H / Hk) % 2 == 0; }         // equal lengths side by side; else neighbouring rows, one block apart at most
static long long tile_count(int B, int Tq, int H) { return (long long)((Tq + BQ - 1) / BQ) * B * H; }
static long long pair_count(int B, int Tq, int H, int Hk) { return pairs_of_heads(H, Hk) ? tile_count(B, Tq, H / 2) : (long long)((Tq + 2 * BQ - 1) / (2 * BQ)) * B * H; }
static bool one_tile(int B, int Tq, int H, int Hk, int n_sm) {
    const long long tiles = tile_count(B, Tq, H), ctas = pair_count(B, Tq, H, Hk);
    return tiles <= 0x7fffffffLL && 3 * ((tiles + n_sm - 1) / n_sm) <= 4 * ((ctas + n_sm - 1) / n_sm);
}

// Of the current device; asked for once (the query costs the host more than the rule).
static int sm_count() {
    static thread_local int of = -1, n = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev != of && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) of = dev;
    return n > 0 ? n : 148;
}

template <int D>
static int launch_tile(const void* q, const void* k, const void* v, Params p, cudaStream_t st) {
    CUtensorMap mq, mk, mv;
    if (ptb_make_tmap_bf16_3d(&mq, q, (long long)p.H * D, p.Tq, p.B, 64, BQ, 1)) return -1;
    if (ptb_make_tmap_bf16_3d(&mk, k, (long long)p.Hk * D, p.Tk, p.B, 64, BKV, 1)) return -1;
    if (ptb_make_tmap_bf16_3d(&mv, v, (long long)p.Hk * D, p.Tk, p.B, 64, 64, 1)) return -1;
    static bool attr = false;
    if (!attr) {
        PTB_CUDA_OK(cudaFuncSetAttribute(fwd_tile_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmTile<D>::TOTAL));
        attr = true;
    }
    p.units = p.B * p.H;
    fwd_tile_kernel<D><<<(unsigned)tile_count(p.B, p.Tq, p.H), NTHREADS, SmTile<D>::TOTAL, st>>>(mq, mk, mv, p);
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}

// q, k, v: rows of ldq, ldk, ldv elements (heads packed along a row; without cu rows lie next to one another).
template <int D>
static int launch(const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv, void* o, float* lse, const int* cu, long long rows_q,
                  long long rows_k, int B, int Tq, int Tk, int H, int Hk, int causal, float scale, int q_offset, int* status, cudaStream_t st) {
    if (B <= 0 || Tq <= 0 || H <= 0) return 0;
    Params p;
    p.O = (__nv_bfloat16*)o; p.lse = lse; p.cu = cu; p.B = B; p.Tq = Tq; p.Tk = Tk; p.H = H; p.Hk = Hk; p.causal = causal; p.q_offset = q_offset;
    p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
    p.pair_heads = pairs_of_heads(H, Hk);
    p.units = B * (p.pair_heads ? H / 2 : H);
    const long long ctas = pair_count(B, Tq, H, Hk);
    if (ctas > 0x7fffffffLL) { ptb_set_error("flash attention: %lld tiles", ctas); return -1; }
    if (!cu && one_tile(B, Tq, H, Hk, sm_count())) return launch_tile<D>(q, k, v, p, st);
    CUtensorMap mq, mk, mv;
    if (ptb_make_tmap_bf16(&mq, q, (long long)H * D, rows_q, ldq, 64, BQ)) return -1;
    if (ptb_make_tmap_bf16(&mk, k, (long long)Hk * D, rows_k, ldk, 64, BKV)) return -1;
    if (ptb_make_tmap_bf16(&mv, v, (long long)Hk * D, rows_k, ldv, 64, 64)) return -1;
    static bool attr = false;
    if (!attr) {
        PTB_CUDA_OK(cudaFuncSetAttribute(fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sm<D>::TOTAL));
        attr = true;
    }
    fwd_kernel<D><<<(unsigned)ctas, NTHREADS, Sm<D>::TOTAL, st>>>(mq, mk, mv, p);
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}


// ---------------------------------------------------------------------------------------------- backward
// One CTA per (128 keys, KV head, batch); it keeps K_j and V_j in shared memory and dK_j, dV_j in tensor memory, and
// walks the query blocks that see those keys (all query heads of the KV head's group).  The scores are held transposed, a
// tensor-memory lane per key, so that P^T is the A operand of dV from tensor memory.  Per query block i, in the order of issue:
//   dV_j += P^T dO_i     P^T = exp2(S^T c - lse_i) in bf16, written by the compute warps over S^T
//   dP^T = V_j dO_i^T    head size 128: its columns are those of dQ_i-1, which is read out under dV
//   S^T  = K_j Q_i+1^T   the next block's scores
//   dP^T = V_j dO_i+1^T  head size 64, where dQ has columns of its own: the next block's, too
//   dQ_i = dS K_j        dS^T = P^T (dP^T - delta_i) scale in bf16, in shared memory
//   dK_j += dS^T Q_i
// so the exponentials of block i+1 run under dQ and dK of block i, and dS under the next scores.  CTAs start with the key blocks that most
// queries see, over all heads: with one head's blocks after another the last head's longest one started near the end.
// Measured (2 x 4001 queries, 32 heads over 8, size 128, causal; 4 x 2048, 32 over 4, size 64): all five products of a block in one chain behind its
// exponentials 1.70 and 0.73 ms; in this order by heads 0.95 and 0.41 ms (size 64 with dP behind its own exponentials 0.43; size 128 with the next
// dP ahead, behind dQ's read-out: 1.06), long CTAs first 0.84 and 0.34 ms.  Bound by the compute warps' latency (issue slots 22 to 29 % used,
// tensor pipe 25 to 35 %).
// Every tile lives in shared memory in ONE layout, [64-column chunk][row][128 B, 128-byte swizzle], which the
// descriptors read as a K-major operand (rows = M or N) or as an MN-major operand (rows = K): Q_i is the B operand
// of S^T and of dK, dO_i that of dP^T and of dV, K_j the A operand of S^T and the B operand of dQ, and dS^T
// an A operand in both orientations.  dQ_i is added to the fp32 dQ by TMA reductions of 128 x 32 pieces from shared memory: whole
// lines, where one thread per row added 16 bytes at a time.
// Sixteen warps: 0-7 compute (a thread has one key and 64 of the block's queries), 8 TMA producer, 9 MMA issuer, 12-15 dQ.
struct BwdParams {
    const float* lse;        // [B, H, Tq] natural log
    const float* delta;      // [B, H, Tq]
    __nv_bfloat16* dk;       // [B, Tk, Hk, D]
    __nv_bfloat16* dv;
    int B, Tq, Tk, H, Hk;
    int causal, q_offset;
    float scale, scale_log2;
    int* status;
    int gsplit;              // CTAs per KV head: each takes group / gsplit query heads and writes its own dk / dv slice
};

constexpr int BWD_THREADS = 512;
// Registers a thread of the compute, dQ and other warps: the launch's 512 x 128 shared out anew (256 x 144 + 128 x 176 + 128 x 48 = 65536).
// Without it the compiler spills more at head size 128 (260 bytes a thread): forward and backward of 2 x 4001 queries 1.39 ms in place of 1.32.
constexpr int REGS_COMPUTE = 144, REGS_DQ = 176, REGS_OTHER = 48;
template <int R> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

template <int D>
struct SmB {
    static constexpr int TILE = 128 * D * 2;                 // K, V, Q, dO
    static constexpr int PT = 128 * 128 * 2;                 // dS
    static constexpr int STG = 128 * 32 * 4;                 // a piece of dQ
    static constexpr int NDO = D == 64 ? 2 : 1;              // dO stages: two where shared memory allows (a block's dO is free again well before the next is needed)
    static constexpr int OFF_K = 0;
    static constexpr int OFF_V = OFF_K + TILE;
    static constexpr int OFF_Q = OFF_V + TILE;
    static constexpr int OFF_DO = OFF_Q + 2 * TILE;
    static constexpr int OFF_DS = OFF_DO + NDO * TILE;
    static constexpr int OFF_STG = OFF_DS + PT;
    static constexpr int OFF_ROW = OFF_STG + 2 * STG;        // lse and delta of two query blocks
    static constexpr int OFF_BAR = OFF_ROW + 2 * 2 * 128 * 4;
    static constexpr int TOTAL = OFF_BAR + 192;
    static_assert(TOTAL <= 232448, "shared memory of one CTA");
};

__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, const void* src, int c0, int c1, int c2) {
    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(map), "r"(smem_u32(src)), "r"(c0), "r"(c1),
                 "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ void dq_sync() { asm volatile("bar.sync 2, 128;" ::: "memory"); }

template <int D>
__global__ void __launch_bounds__(BWD_THREADS, 1)
bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
           const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ BwdParams P) {
    using S = SmB<D>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sk = smem + S::OFF_K;
    uint8_t* sv = smem + S::OFF_V;
    uint8_t* sq = smem + S::OFF_Q;
    uint8_t* sdo = smem + S::OFF_DO;
    uint8_t* sds = smem + S::OFF_DS;
    uint8_t* stg = smem + S::OFF_STG;
    float* srow = reinterpret_cast<float*>(smem + S::OFF_ROW);       // [block & 1][lse, delta][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    constexpr int NDO = S::NDO;
    uint64_t* kv_full = bars;            // K_j, V_j loaded (once)
    uint64_t* q_full = bars + 1;         // [2] Q_i loaded
    uint64_t* q_empty = bars + 3;        // [2] the MMAs that read it have completed
    uint64_t* do_full = bars + 5;        // [2] dO_i loaded
    uint64_t* do_empty = bars + 7;       // [2]
    uint64_t* s_full = bars + 9;         // S^T is in TMEM
    uint64_t* dp_full = bars + 10;       // dP^T is in TMEM
    uint64_t* p_ready = bars + 11;       // P^T is in TMEM (8 arrivals)
    uint64_t* ds_ready = bars + 12;      // dS^T is in shared memory (8 arrivals)
    uint64_t* dq_full = bars + 13;       // dQ_i is in TMEM
    uint64_t* dq_read = bars + 14;       // dQ_i has been read back (4 arrivals)
    uint64_t* all_done = bars + 15;      // dK and dV are complete
    uint64_t* ds_empty = bars + 16;      // the MMAs that read dS^T have completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    if (smem_u32(smem) & 1023) {         // the swizzled tiles need it, and there is no room to align by hand
        if (threadIdx.x == 0 && P.status) atomicExch(P.status, PTB_ERR_BOUNDS);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // early key blocks (with a causal mask those that most queries see) first, over all heads and sequences: the last CTAs to start are short
    const int per_jb = P.Hk * P.gsplit * P.B, jb = (int)blockIdx.x / per_jb, unit = (int)blockIdx.x % per_jb;
    const int hk = unit % P.Hk, part = unit / P.Hk % P.gsplit, b = unit / (P.Hk * P.gsplit);
    const int group = (P.H / P.Hk) / P.gsplit;          // query heads this CTA walks
    const int head0 = hk * (P.H / P.Hk) + part * group;
    const int key0 = jb * 128;
    const int nq = (P.Tq + 127) / 128;
    // first query block that sees key0: rows q with q + q_offset >= key0
    const int i_start = P.causal ? max(0, (key0 - P.q_offset) / 128) : 0;
    const int per_head = max(0, nq - i_start);
    const int n_it = per_head * group;

    if (threadIdx.x == 0) {
        mbar_init(kv_full, 1);
        for (int st = 0; st < 2; ++st) { mbar_init(&q_full[st], 1); mbar_init(&q_empty[st], 1); mbar_init(&do_full[st], 1); mbar_init(&do_empty[st], 1); }
        mbar_init(s_full, 1); mbar_init(dp_full, 1); mbar_init(p_ready, 8); mbar_init(ds_ready, 8);
        mbar_init(dq_full, 1); mbar_init(dq_read, 4); mbar_init(all_done, 1); mbar_init(ds_empty, 1);
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV); prefetch_tmap(&tmDO); prefetch_tmap(&tmDQ);
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // P^T over S^T: the weights of queries 0-63 in columns 0-31, of 64-127 in 64-95 (each half over the scores that its own thread has read)
    constexpr uint32_t TM_S = 0, TM_DP = 128, TM_DV = 256, TM_DK = 256 + D, TM_DQ = D == 64 ? 384 : TM_DP;

    if (warp >= 8 && warp < 12) {
        regs_dec<REGS_OTHER>();
        if (warp == 8 && lane == 0 && n_it > 0) {
            // ------------------------------------------------------------------------ TMA producer
            bool ok = true;
            mbar_expect_tx(kv_full, 2 * S::TILE);
            for (int c = 0; c < D / 64; ++c) {
                tma_load_3d(sk + c * 16384, &tmK, hk * D + c * 64, key0, b, kv_full);
                tma_load_3d(sv + c * 16384, &tmV, hk * D + c * 64, key0, b, kv_full);
            }
            for (int it = 0; it < n_it && ok; ++it) {
                const int h = head0 + it / per_head, i = i_start + it % per_head;
                const int qs = it & 1, ds = it % NDO;
                if (it >= 2) ok = mbar_wait(&q_empty[qs], (uint32_t)(((it >> 1) - 1) & 1), P.status);
                if (!ok) break;
                mbar_expect_tx(&q_full[qs], S::TILE);
                for (int c = 0; c < D / 64; ++c) tma_load_3d(sq + qs * S::TILE + c * 16384, &tmQ, h * D + c * 64, i * 128, b, &q_full[qs]);
                if (it >= NDO) ok = mbar_wait(&do_empty[ds], (uint32_t)(((it / NDO) - 1) & 1), P.status);
                if (!ok) break;
                mbar_expect_tx(&do_full[ds], S::TILE);
                for (int c = 0; c < D / 64; ++c) tma_load_3d(sdo + ds * S::TILE + c * 16384, &tmDO, h * D + c * 64, i * 128, b, &do_full[ds]);
            }
            if (!ok) *abort_flag = 1;
        } else if (warp == 9 && lane == 0 && n_it > 0) {
            // ------------------------------------------------------------------------ MMA issuer
            constexpr uint32_t idesc_t = instr_desc(128, 128, 0, 0);       // S^T, dP^T: both operands K-major
            constexpr uint32_t idesc_k = instr_desc(128, D, 0, 1);         // dV, dK: A with the queries along K, B = dO / Q MN-major
            constexpr uint32_t idesc_q = instr_desc(128, D, 1, 1);         // dQ: A = dS^T read MN-major, B = K MN-major
            const uint32_t aK = smem_u32(sk), aV = smem_u32(sv), aDS = smem_u32(sds);
            auto issue_s = [&](int it) {
                const uint32_t aQ = smem_u32(sq + (it & 1) * S::TILE);
                if (!mbar_wait(&q_full[it & 1], (uint32_t)((it >> 1) & 1), P.status)) return false;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < D / 64; ++c)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base + TM_S, smem_desc(aK + c * 16384 + k * 32, 16, 1024), smem_desc(aQ + c * 16384 + k * 32, 16, 1024), idesc_t,
                                  (c > 0 || k > 0) ? 1u : 0u);
                umma_commit(s_full);
                return true;
            };
            auto issue_dp = [&](int it) {
                const int st = it % NDO;
                const uint32_t aDO = smem_u32(sdo + st * S::TILE);
                if (!mbar_wait(&do_full[st], (uint32_t)((it / NDO) & 1), P.status)) return false;
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < D / 64; ++c)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base + TM_DP, smem_desc(aV + c * 16384 + k * 32, 16, 1024), smem_desc(aDO + c * 16384 + k * 32, 16, 1024), idesc_t,
                                  (c > 0 || k > 0) ? 1u : 0u);
                umma_commit(dp_full);
                return true;
            };
            constexpr bool AHEAD = D == 64;               // dP^T of the next block before this block is done
            bool ok = mbar_wait(kv_full, 0, P.status) && issue_s(0) && (!AHEAD || issue_dp(0));
            for (int it = 0; it < n_it && ok; ++it) {
                const uint32_t aQ = smem_u32(sq + (it & 1) * S::TILE), aDO = smem_u32(sdo + (it % NDO) * S::TILE);
                const uint32_t ph = (uint32_t)(it & 1), acc = it > 0 ? 1u : 0u;
                ok = mbar_wait(p_ready, ph, P.status);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int kq = 0; kq < 8; ++kq)        // K dimension = the 128 queries, 16 per step: 2048 B further down each chunk of dO
                    umma_bf16_ts(tmem_base + TM_DV, tmem_base + TM_S + (uint32_t)((kq >> 2) * 64 + (kq & 3) * 8), smem_desc(aDO + kq * 2048, 16384, 1024), idesc_k,
                                 (kq > 0) ? 1u : acc);
                if (!AHEAD) {                         // dQ_i-1 leaves these columns while dV runs
                    if (it > 0) ok = mbar_wait(dq_read, ph ^ 1, P.status);
                    if (ok) ok = issue_dp(it);
                    if (!ok) break;
                }
                umma_commit(&do_empty[it % NDO]);
                if (it + 1 < n_it) ok = issue_s(it + 1);
                if (ok) ok = mbar_wait(ds_ready, ph, P.status);          // dS^T is written, and dP^T has been read
                if (!ok) break;
                tc_fence_after();
                if (AHEAD) {
                    if (it + 1 < n_it) ok = issue_dp(it + 1);
                    if (ok && it > 0) ok = mbar_wait(dq_read, ph ^ 1, P.status);
                    if (!ok) break;
                    tc_fence_after();
                }
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)        // K dimension = the 128 keys
                    umma_bf16(tmem_base + TM_DQ, smem_desc(aDS + kk * 2048, 16384, 1024), smem_desc(aK + kk * 2048, 16384, 1024), idesc_q, kk > 0 ? 1u : 0u);
                umma_commit(dq_full);
#pragma unroll
                for (int kq = 0; kq < 8; ++kq)
                    umma_bf16(tmem_base + TM_DK, smem_desc(aDS + (kq >> 2) * 16384 + (kq & 3) * 32, 16, 1024), smem_desc(aQ + kq * 2048, 16384, 1024), idesc_k,
                              (kq > 0) ? 1u : acc);
                umma_commit(&q_empty[it & 1]);
                umma_commit(ds_empty);
            }
            umma_commit(all_done);
            if (!ok) *abort_flag = 1;
        }
    } else if (warp >= 12) {
        // ---------------------------------------------------------------------------- dQ warps
        regs_inc<REGS_DQ>();
        const int row = 32 * (warp & 3) + lane;          // query row of the block = TMEM lane
        const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + TM_DQ;
        const bool elected = warp == 12 && lane == 0;
        bool ok = true;
        int piece = 0;
#pragma unroll 1
        for (int it = 0; it < n_it; ++it) {
            const int h = head0 + it / per_head, i = i_start + it % per_head;
            if (ok && !*abort_flag) ok = mbar_wait(dq_full, (uint32_t)(it & 1), P.status);
            else ok = false;
            tc_fence_after();
            float r[D];
#pragma unroll
            for (int c = 0; c < D / 32; ++c) tmem_ld32(lane_addr + (uint32_t)(c * 32), reinterpret_cast<uint32_t*>(r) + c * 32);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(dq_read);
#pragma unroll
            for (int c = 0; c < D / 32; ++c, ++piece) {
                uint8_t* buf = stg + (piece & 1) * S::STG;
                if (elected) bulk_wait_read<1>();        // the piece before last has left this buffer
                dq_sync();
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    *reinterpret_cast<float4*>(buf + row * 128 + ((u ^ (row & 7)) * 16)) =
                        make_float4(r[c * 32 + 4 * u], r[c * 32 + 4 * u + 1], r[c * 32 + 4 * u + 2], r[c * 32 + 4 * u + 3]);
                fence_proxy_async();
                dq_sync();
                if (elected) {
                    if (ok) tma_reduce_add_3d(&tmDQ, buf, h * D + c * 32, i * 128, b);
                    bulk_commit();
                }
            }
        }
        if (elected) bulk_wait<0>();
        if (!ok) *abort_flag = 1;
    } else {
        // ---------------------------------------------------------------------------- compute warps
        regs_inc<REGS_COMPUTE>();
        const int row = 32 * (warp & 3) + lane;          // key of the block = TMEM lane
        const int hf = warp >> 2;                        // which 64 queries
        const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16);
        const int key = key0 + row;
        bool ok = true;
        // thread x brings lse (x < 128) or delta of query x % 128 of a block, ready to use: lse in powers of two, delta times the scale
        auto row_value = [&](int it) {
            const int h = head0 + it / per_head, q = (i_start + it % per_head) * 128 + (threadIdx.x & 127);
            const bool is_lse = threadIdx.x < 128;
            if (q >= P.Tq) return is_lse ? INFINITY : 0.f;                  // P = 0 for rows past the end
            const size_t at = ((size_t)b * P.H + h) * P.Tq + q;
            return is_lse ? P.lse[at] * 1.4426950408889634f : P.delta[at] * P.scale;
        };
        if (n_it > 0) {
            srow[threadIdx.x] = row_value(0);
            compute_sync();
        }
#pragma unroll 1
        for (int it = 0; it < n_it; ++it) {
            const int q0 = (i_start + it % per_head) * 128;
            const float next_row = it + 1 < n_it ? row_value(it + 1) : 0.f;
            const float4* lse4 = reinterpret_cast<const float4*>(srow + (it & 1) * 256 + hf * 64);
            const float4* dlt4 = lse4 + 32;
            if (ok && !*abort_flag) ok = mbar_wait(s_full, (uint32_t)(it & 1), P.status);
            else ok = false;
            tc_fence_after();
            float p[64];
            tmem_ld32(lane_addr + TM_S + (uint32_t)(hf * 64), reinterpret_cast<uint32_t*>(p));
            tmem_ld32(lane_addr + TM_S + (uint32_t)(hf * 64 + 32), reinterpret_cast<uint32_t*>(p) + 32);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float4 l = lse4[e];
                p[4 * e] = exp2f(p[4 * e] * P.scale_log2 - l.x);
                p[4 * e + 1] = exp2f(p[4 * e + 1] * P.scale_log2 - l.y);
                p[4 * e + 2] = exp2f(p[4 * e + 2] * P.scale_log2 - l.z);
                p[4 * e + 3] = exp2f(p[4 * e + 3] * P.scale_log2 - l.w);
            }
            const int qf = q0 + hf * 64;
            const bool need_mask = (key0 + 128 > P.Tk) || (P.causal && key0 + 127 > qf + P.q_offset);
            const int first = key >= P.Tk ? 64 : P.causal ? key - P.q_offset - qf : 0;        // of this thread's queries, those from here on see the key
            if (need_mask) {
#pragma unroll
                for (int e = 0; e < 64; ++e)
                    if (e < first) p[e] = 0.f;
            }
            {
                uint32_t pk[32];
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const __nv_bfloat162 h2 = __floats2bfloat162_rn(p[2 * e], p[2 * e + 1]);
                    pk[e] = *reinterpret_cast<const uint32_t*>(&h2);
                }
                tmem_st32(lane_addr + TM_S + (uint32_t)(hf * 64), pk);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
            if (ok && !*abort_flag) ok = mbar_wait(dp_full, (uint32_t)(it & 1), P.status);
            else ok = false;
            tc_fence_after();
            if (it > 0 && ok) ok = mbar_wait(ds_empty, (uint32_t)((it - 1) & 1), P.status);
            uint8_t* drow = sds + hf * 16384 + row * 128;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float d[32];
                tmem_ld32(lane_addr + TM_DP + (uint32_t)(hf * 64 + c * 32), reinterpret_cast<uint32_t*>(d));
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float4 dl = dlt4[c * 8 + e];
                    d[4 * e] = p[c * 32 + 4 * e] * (d[4 * e] * P.scale - dl.x);
                    d[4 * e + 1] = p[c * 32 + 4 * e + 1] * (d[4 * e + 1] * P.scale - dl.y);
                    d[4 * e + 2] = p[c * 32 + 4 * e + 2] * (d[4 * e + 2] * P.scale - dl.z);
                    d[4 * e + 3] = p[c * 32 + 4 * e + 3] * (d[4 * e + 3] * P.scale - dl.w);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint4 o;
                    __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                    for (int x = 0; x < 4; ++x) oh[x] = __floats2bfloat162_rn(d[8 * u + 2 * x], d[8 * u + 2 * x + 1]);
                    *reinterpret_cast<uint4*>(drow + (((c * 4 + u) ^ (row & 7)) * 16)) = o;
                }
            }
            srow[((it + 1) & 1) * 256 + threadIdx.x] = next_row;
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ds_ready);
            compute_sync();                   // the next block's lse and delta are there
        }
        // ---- dK_j, dV_j
        if (n_it > 0) {
            if (ok && !*abort_flag) ok = mbar_wait(all_done, 0, P.status);
            else ok = false;
            tc_fence_after();
#pragma unroll 1
            for (int which = 0; which < 2; ++which) {
                __nv_bfloat16* outp = (which ? P.dk : P.dv) + (size_t)part * P.B * P.Tk * P.Hk * D + (((size_t)b * P.Tk + key) * P.Hk + hk) * D +
                                      hf * (D / 2);
#pragma unroll
                for (int c = 0; c < D / 64; ++c) {
                    uint32_t r[32];
                    tmem_ld32(lane_addr + (which ? TM_DK : TM_DV) + (uint32_t)(hf * (D / 2) + c * 32), r);
                    tmem_ld_wait();
                    if (key < P.Tk && ok) {
#pragma unroll
                        for (int e = 0; e < 32; e += 8) {
                            uint4 o;
                            __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                            for (int x = 0; x < 4; ++x) oh[x] = __floats2bfloat162_rn(__uint_as_float(r[e + 2 * x]), __uint_as_float(r[e + 2 * x + 1]));
                            *reinterpret_cast<uint4*>(outp + c * 32 + e) = o;
                        }
                    }
                }
            }
        } else if (key < P.Tk) {
            // no query block sees these keys: their gradients are zero
            const size_t base = (size_t)part * P.B * P.Tk * P.Hk * D + (((size_t)b * P.Tk + key) * P.Hk + hk) * D;
            for (int d = hf * (D / 2); d < (hf + 1) * (D / 2); ++d) {
                P.dk[base + d] = __float2bfloat16_rn(0.f);
                P.dv[base + d] = __float2bfloat16_rn(0.f);
            }
        }
        if (!ok) *abort_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem_base, 512);
}

template <int D>
static int launch_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse, const float* delta, float* dq, void* dk,
                      void* dv, int B, int Tq, int Tk, int H, int Hk, int causal, float scale, int q_offset, int gsplit, int* status,
                      cudaStream_t st) {
    CUtensorMap mq, mk, mv, mdo, mdq;
    if (ptb_make_tmap_f32_3d(&mdq, dq, (long long)H * D, Tq, B, 32, 128)) return -1;
    // Rows past an entry's end arrive as zeros.  As rows of one [B T] matrix they were the next entry's: their weights are zero, but zero times
    // what is not finite is not, and one entry's infinities reached the gradients of the entry before it.
    if (ptb_make_tmap_bf16_3d(&mq, q, (long long)H * D, Tq, B, 64, 128, 1)) return -1;
    if (ptb_make_tmap_bf16_3d(&mdo, dout, (long long)H * D, Tq, B, 64, 128, 1)) return -1;
    if (ptb_make_tmap_bf16_3d(&mk, k, (long long)Hk * D, Tk, B, 64, 128, 1)) return -1;
    if (ptb_make_tmap_bf16_3d(&mv, v, (long long)Hk * D, Tk, B, 64, 128, 1)) return -1;
    static bool attr = false;
    if (!attr) {
        PTB_CUDA_OK(cudaFuncSetAttribute(bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmB<D>::TOTAL));
        attr = true;
    }
    BwdParams p;
    p.lse = lse; p.delta = delta; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
    p.B = B; p.Tq = Tq; p.Tk = Tk; p.H = H; p.Hk = Hk; p.causal = causal; p.q_offset = q_offset;
    p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status; p.gsplit = gsplit;
    const long long ctas = (long long)((Tk + 127) / 128) * Hk * gsplit * B;
    if (ctas > 0x7fffffffLL) { ptb_set_error("flash attention: %lld tiles", ctas); return -1; }
    if (ctas == 0) return 0;
    bwd_kernel<D><<<(unsigned)ctas, BWD_THREADS, SmB<D>::TOTAL, st>>>(mq, mk, mv, mdo, mdq, p);
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}

}  // namespace fa100
}  // namespace ptb

// q [B, Tq, H, D], k/v [B, Tk, Hk, D] bf16 contiguous, D in {64, 128}; o like q; lse [B, H, Tq] fp32 (natural log).
// status: device int, set non-zero if a wait timed out.
PTB_API int ptb_flash_attn_fwd_sm100(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Tq, int Tk, int H, int Hk,
                                     int D, int causal, float scale, int q_offset, int* status, cudaStream_t st) {
    if (H % Hk) { ptb_set_error("flash attention: %d query heads over %d KV heads", H, Hk); return -1; }
    if ((uintptr_t)o & 15) { ptb_set_error("flash attention: the output needs a 16-byte aligned base"); return -1; }
    {
        int dev = 0;
        PTB_CUDA_OK(cudaGetDevice(&dev));
        PTB_CUDA_OK(cudaSetDevice(dev));     // the tensor-map encoder is a driver call: bind the primary context to this thread
    }
    auto run = [&](auto f) {
        return f(q, (long long)H * D, k, (long long)Hk * D, v, (long long)Hk * D, o, lse, nullptr, (long long)B * Tq, (long long)B * Tk, B, Tq, Tk, H, Hk, causal,
                 scale, q_offset, status, st);
    };
    if (D == 128) return run(ptb::fa100::launch<128>);
    if (D == 64) return run(ptb::fa100::launch<64>);
    ptb_set_error("flash attention (tcgen05): head size %d not supported (64, 128)", D);
    return -1;
}

// Whether the forward of these sizes runs one tile of 128 rows per CTA on a GPU of n_sm SMs (packed sequences never do).
PTB_API int ptb_flash_attn_one_tile(int B, int Tq, int H, int Hk, int n_sm) { return ptb::fa100::one_tile(B, Tq, H, Hk, n_sm); }

// Sequences of different lengths packed by rows: sequence i has rows cu[i] .. cu[i + 1] (cu: device int [n_seq + 1], rows in all, none longer
// than max_len) of q, k and v, whose rows are ldq, ldk and ldv elements apart with the heads packed along them; o [rows, H, D].  One launch.
PTB_API int ptb_flash_attn_varlen_fwd(const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv, void* o, const int* cu, int n_seq,
                                      int max_len, long long rows, int H, int Hk, int D, int causal, float scale, int* status, cudaStream_t st) {
    if (Hk <= 0 || H % Hk) { ptb_set_error("flash attention: %d query heads over %d KV heads", H, Hk); return -1; }
    if ((uintptr_t)o & 15) { ptb_set_error("flash attention: the output needs a 16-byte aligned base"); return -1; }
    if (!cu || rows <= 0 || n_seq <= 0) { ptb_set_error("flash attention: packed sequences need their offsets and at least one row"); return -1; }
    {
        int dev = 0;
        PTB_CUDA_OK(cudaGetDevice(&dev));
        PTB_CUDA_OK(cudaSetDevice(dev));
    }
    if (D == 128) return ptb::fa100::launch<128>(q, ldq, k, ldk, v, ldv, o, nullptr, cu, rows, rows, n_seq, max_len, max_len, H, Hk, causal, scale, 0, status, st);
    if (D == 64) return ptb::fa100::launch<64>(q, ldq, k, ldk, v, ldv, o, nullptr, cu, rows, rows, n_seq, max_len, max_len, H, Hk, causal, scale, 0, status, st);
    ptb_set_error("flash attention (tcgen05): head size %d not supported (64, 128)", D);
    return -1;
}

extern "C" int ptb_flash_attn_delta(const void* o, const void* dout, float* delta, int B, int Tq, int H, int D, float* dq_zero, cudaStream_t st);

// Backward on tcgen05.  dq: fp32 [B, Tq, H, D] (cleared here, together with the delta pass); delta: fp32 [B, H, Tq] scratch.
// dk, dv: bf16 [gsplit][B, Tk, Hk, D]: with grouped-query heads the query heads of one KV head can be split over
// `gsplit` CTAs (a divisor of H / Hk) so that small problems fill the GPU; the caller sums the slices.
PTB_API int ptb_flash_attn_bwd_sm100(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse,
                                     float* delta, float* dq, void* dk, void* dv, int B, int Tq, int Tk, int H, int Hk, int D, int causal,
                                     float scale, int q_offset, int gsplit, int* status, cudaStream_t st) {
    if (H % Hk || gsplit < 1 || (H / Hk) % gsplit) { ptb_set_error("flash attention: %d query heads over %d KV heads, split %d", H, Hk, gsplit); return -1; }
    {
        int dev = 0;
        PTB_CUDA_OK(cudaGetDevice(&dev));
        PTB_CUDA_OK(cudaSetDevice(dev));
    }
    if (ptb_flash_attn_delta(o, dout, delta, B, Tq, H, D, dq, st)) return -1;      // also clears dq
    if (D == 128) return ptb::fa100::launch_bwd<128>(q, k, v, dout, lse, delta, dq, dk, dv, B, Tq, Tk, H, Hk, causal, scale, q_offset, gsplit, status, st);
    if (D == 64) return ptb::fa100::launch_bwd<64>(q, k, v, dout, lse, delta, dq, dk, dv, B, Tq, Tk, H, Hk, causal, scale, q_offset, gsplit, status, st);
    ptb_set_error("flash attention (tcgen05): head size %d not supported (64, 128)", D);
    return -1;
}
