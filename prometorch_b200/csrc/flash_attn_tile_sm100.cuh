// Forward of grids that leave SMs idle: one tile of 128 query rows of one head per CTA, two threads a row.
//
// Ten warps as in the two-tile kernel: warp 8 loads Q once and K and V tiles of 128 keys through two-stage rings, warp 9 issues S(j) = Q K_j^T into one of
// two 128-column buffers, two blocks ahead, and O_j = P_j V_j into a third once P_j is in shared memory; warps 0-7 are the softmax.  A
// thread owns one query row (its tensor-memory lane) and half of a block's columns, exchanges the row maximum with its partner through
// shared memory, and keeps its half of the output row in registers; the read-back of O_j-1 runs under the scores of block j.  What bounds a lone CTA
// is the chain scores, exponentials, product of each block, and with half a row a thread that chain is shorter than the two-tile kernel's.  Rows
// past an entry's end arrive as zeros.
#pragma once

namespace ptb {
namespace fa100 {

template <int D>
struct SmTile {
    static constexpr int Q_BYTES = BQ * D * 2;
    static constexpr int KV_BYTES = BKV * D * 2;
    static constexpr int P_BYTES = BQ * BKV * 2;
    static constexpr int OFF_Q = 0;
    static constexpr int OFF_K = OFF_Q + Q_BYTES;
    static constexpr int OFF_V = OFF_K + 2 * KV_BYTES;
    static constexpr int OFF_P = OFF_V + 2 * KV_BYTES;
    static constexpr int OFF_RED = OFF_P + P_BYTES;          // 2 x 128 floats
    static constexpr int OFF_BAR = OFF_RED + 2 * BQ * 4;
    static constexpr int TOTAL = OFF_BAR + 256 + 1024;
};

__device__ __forceinline__ void softmax_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }          // of the one-tile kernel's eight softmax warps

template <int D>
__global__ void __launch_bounds__(NTHREADS, 1)
fwd_tile_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
           const __grid_constant__ Params P) {
    using S = SmTile<D>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sq = smem + S::OFF_Q;
    uint8_t* sk = smem + S::OFF_K;
    uint8_t* sv = smem + S::OFF_V;
    uint8_t* sp = smem + S::OFF_P;
    float* red = reinterpret_cast<float*>(smem + S::OFF_RED);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::OFF_BAR);
    uint64_t* q_full = bars;             // [1]
    uint64_t* k_full = bars + 1;         // [2]
    uint64_t* k_empty = bars + 3;        // [2]
    uint64_t* v_full = bars + 5;         // [2]
    uint64_t* v_empty = bars + 7;        // [2]
    uint64_t* s_full = bars + 9;         // [2]
    uint64_t* p_ready = bars + 11;       // [1], 8 arrivals (one per softmax warp)
    uint64_t* o_full = bars + 12;        // [1]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // late row blocks (the long ones under a causal mask) first, over all heads and sequences
    const int qb = (int)gridDim.x / P.units - 1 - (int)blockIdx.x / P.units, unit = (int)blockIdx.x % P.units;
    const int h = unit % P.H, b = unit / P.H;
    const int hk = h / (P.H / P.Hk);
    const int q0 = qb * BQ;
    // keys this block can see: [0, kv_end)
    const int kv_end = P.causal ? min(P.Tk, q0 + BQ + P.q_offset) : P.Tk;
    const int nblk = max(0, (kv_end + BKV - 1) / BKV);

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); mbar_init(&s_full[s], 1); }
        mbar_init(p_ready, 8);
        mbar_init(o_full, 1);
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
    const uint32_t TM_S = 0, TM_O = 256;                           // column offsets: S buffers at 0 and 128, O_j at 256

    if (warp == 8) {
        // ---------------------------------------------------------------------------- TMA producer
        if (lane == 0 && nblk > 0) {
            bool ok = true;
            mbar_expect_tx(q_full, S::Q_BYTES);
            for (int kb = 0; kb < D / 64; ++kb) tma_load_3d(sq + kb * (BQ * 128), &tmQ, h * D + kb * 64, q0, b, q_full);
            for (int j = 0; j < nblk && ok; ++j) {
                const int s = j & 1;
                if (j >= 2) ok = mbar_wait(&k_empty[s], (uint32_t)(((j >> 1) - 1) & 1), P.status);
                if (!ok) break;
                mbar_expect_tx(&k_full[s], S::KV_BYTES);
                for (int kb = 0; kb < D / 64; ++kb)
                    tma_load_3d(sk + s * S::KV_BYTES + kb * (BKV * 128), &tmK, hk * D + kb * 64, j * BKV, b, &k_full[s]);
                if (j >= 2) ok = mbar_wait(&v_empty[s], (uint32_t)(((j >> 1) - 1) & 1), P.status);
                if (!ok) break;
                mbar_expect_tx(&v_full[s], S::KV_BYTES);
                for (int hh = 0; hh < 2; ++hh)                       // two halves of 64 keys, each D/64 chunks of [64 keys x 64 dims]
                    for (int c = 0; c < D / 64; ++c)
                        tma_load_3d(sv + s * S::KV_BYTES + hh * (D / 64) * 8192 + c * 8192, &tmV, hk * D + c * 64, j * BKV + hh * 64, b, &v_full[s]);
            }
            if (!ok) *abort_flag = 1;
        }
    } else if (warp == 9) {
        // ---------------------------------------------------------------------------- MMA issuer
        if (lane == 0 && nblk > 0) {
            constexpr uint32_t idesc_s = instr_desc(BQ, BKV, 0, 0);          // S = Q K^T: both K-major
            constexpr uint32_t idesc_o = instr_desc(BQ, D, 0, 1);            // O = P V: P K-major, V MN-major
            bool ok = mbar_wait(q_full, 0, P.status);
            auto issue_s = [&](int j) {
                const int s = j & 1;
                if (!mbar_wait(&k_full[s], (uint32_t)((j >> 1) & 1), P.status)) return false;
                tc_fence_after();
                const uint32_t a0 = smem_u32(sq), b0 = smem_u32(sk + s * S::KV_BYTES);
#pragma unroll
                for (int kb = 0; kb < D / 64; ++kb)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base + TM_S + (uint32_t)(s * BKV), smem_desc(a0 + kb * (BQ * 128) + k * 32, 16, 1024),
                                  smem_desc(b0 + kb * (BKV * 128) + k * 32, 16, 1024), idesc_s, (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(&k_empty[s]);
                umma_commit(&s_full[s]);
                return true;
            };
            if (ok) ok = issue_s(0);
            if (ok && nblk > 1) ok = issue_s(1);
            for (int j = 0; j < nblk && ok; ++j) {
                const int s = j & 1;
                ok = mbar_wait(p_ready, (uint32_t)(j & 1), P.status);        // P_j is in shared memory, O_{j-1} has been read
                if (ok) ok = mbar_wait(&v_full[s], (uint32_t)((j >> 1) & 1), P.status);
                if (!ok) break;
                tc_fence_after();
                const uint32_t a0 = smem_u32(sp), b0 = smem_u32(sv + s * S::KV_BYTES);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base + TM_O, smem_desc(a0 + hh * (BQ * 128) + k * 32, 16, 1024),
                                  smem_desc(b0 + hh * (D / 64) * 8192 + k * 2048, 8192, 1024), idesc_o, (hh > 0 || k > 0) ? 1u : 0u);
                umma_commit(&v_empty[s]);
                umma_commit(o_full);
                if (j + 2 < nblk) ok = issue_s(j + 2);
            }
            if (!ok) *abort_flag = 1;
        }
    } else {
        // ---------------------------------------------------------------------------- softmax warps
        const int row = 32 * (warp & 3) + lane;          // query row inside the block = tensor-memory lane
        const int hf = warp >> 2;                        // which 64 columns of S, which D/2 columns of O
        const uint32_t lane_addr = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16);
        const int q_pos = q0 + row + P.q_offset;         // position of this query among the keys
        float o_acc[D / 2];
#pragma unroll
        for (int i = 0; i < D / 2; ++i) o_acc[i] = 0.f;
        float m_run = -INFINITY, l_part = 0.f, alpha_prev = 1.f;
        bool ok = true;
        auto add_o = [&](float alpha) {                  // o_acc = o_acc * alpha + (my half of the row of O_j)
#pragma unroll
            for (int c = 0; c < D / 64; ++c) {
                uint32_t r[32];
                tmem_ld32(lane_addr + TM_O + (uint32_t)(hf * (D / 2) + c * 32), r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) o_acc[c * 32 + i] = o_acc[c * 32 + i] * alpha + __uint_as_float(r[i]);
            }
        };
        for (int j = 0; j < nblk; ++j) {
            const int s = j & 1;
            if (ok && !*abort_flag) ok = mbar_wait(&s_full[s], (uint32_t)((j >> 1) & 1), P.status);
            else ok = false;
            tc_fence_after();
            float sc[64];
            {
                uint32_t r[32];
                tmem_ld32(lane_addr + TM_S + (uint32_t)(s * BKV + hf * 64), r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) sc[i] = __uint_as_float(r[i]) * P.scale_log2;
                tmem_ld32(lane_addr + TM_S + (uint32_t)(s * BKV + hf * 64 + 32), r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) sc[32 + i] = __uint_as_float(r[i]) * P.scale_log2;
            }
            const int key0 = j * BKV + hf * 64;
            const bool need_mask = (key0 + 64 > P.Tk) || (P.causal && key0 + 63 > q0 + P.q_offset);
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    const int key = key0 + i;
                    if (key >= P.Tk || (P.causal && key > q_pos)) sc[i] = -INFINITY;
                }
            }
            // eight independent partial maxima: a 64-long dependent chain would stall the two warps a scheduler has
            float m8[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) m8[i] = sc[i];
#pragma unroll
            for (int i = 8; i < 64; ++i) m8[i & 7] = fmaxf(m8[i & 7], sc[i]);
            const float mx = fmaxf(fmaxf(fmaxf(m8[0], m8[1]), fmaxf(m8[2], m8[3])), fmaxf(fmaxf(m8[4], m8[5]), fmaxf(m8[6], m8[7])));
            red[hf * BQ + row] = mx;
            softmax_sync();
            const float m_blk = fmaxf(red[row], red[BQ + row]);
            const float m_new = fmaxf(m_run, m_blk);
            const float m_use = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = exp2f(m_run - m_use);
            float l4[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t pk[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float p0 = exp2f(sc[2 * i] - m_use), p1 = exp2f(sc[2 * i + 1] - m_use);
                l4[i & 3] += p0 + p1;
                const __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);
                pk[i] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            l_part = l_part * alpha + ((l4[0] + l4[1]) + (l4[2] + l4[3]));
            m_run = m_new;
            // the deferred read-back of O_{j-1}; its MMA ran while the scores above were reduced
            if (j > 0) {
                if (ok) ok = mbar_wait(o_full, (uint32_t)((j - 1) & 1), P.status);
                tc_fence_after();
                add_o(alpha_prev);
            }
            alpha_prev = alpha;
            // P_j -> shared memory, K-major with the 128-byte swizzle: sub-tile hf, row `row`, 16-byte chunk c at c ^ (row & 7)
            {
                uint8_t* prow = sp + hf * (BQ * 128) + row * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    *reinterpret_cast<uint4*>(prow + ((c ^ (row & 7)) * 16)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
            }
            fence_proxy_async();
            tc_fence_before();
            softmax_sync();                   // also keeps `red` from being overwritten before both partners have read it
            if (lane == 0) mbar_arrive(p_ready);
        }
        if (nblk > 0) {
            if (ok) ok = mbar_wait(o_full, (uint32_t)((nblk - 1) & 1), P.status);
            tc_fence_after();
            add_o(alpha_prev);
        }
        red[hf * BQ + row] = l_part;
        softmax_sync();
        const float l = red[row] + red[BQ + row];
        const int q_idx = q0 + row;
        if (q_idx < P.Tq && ok) {
            const float inv = l > 0.f ? 1.0f / l : l == 0.f ? 0.f : l;        // a sum that is not a number stays one
            __nv_bfloat16* op = P.O + (((size_t)b * P.Tq + q_idx) * P.H + h) * D + hf * (D / 2);
#pragma unroll
            for (int i = 0; i < D / 2; i += 8) {
                uint4 o;
                __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int e = 0; e < 4; ++e) oh[e] = __floats2bfloat162_rn(o_acc[i + 2 * e] * inv, o_acc[i + 2 * e + 1] * inv);
                *reinterpret_cast<uint4*>(op + i) = o;
            }
            if (hf == 0) P.lse[((size_t)b * P.H + h) * P.Tq + q_idx] = l > 0.f ? m_run * 0.6931471805599453f + logf(l) : -INFINITY;
        }
        if (!ok) *abort_flag = 1;
    }
    // ---- teardown
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem_base, 512);
}

}  // namespace fa100
}  // namespace ptb
