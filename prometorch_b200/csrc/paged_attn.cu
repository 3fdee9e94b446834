// Paged KV cache for the continuous-batching engine: rotary + page write, and one-token attention over a page table.
//
// The reference's engine (torch/serve/llm.h:299-334, 806-818) keeps the cache in 64-token pages that a request
// picks from a shared pool, and walks them on the CPU one request after another.  Here the pool is one bf16
// tensor per layer, [page][kv_head][64][D]; a step of the engine serves every active request in one batch:
//   paged_rope_write_kernel  rotates q (in place) and k of the new tokens and stores k, v in the slot the page
//                            table gives for (request, position);
//   paged_attn_decode_kernel one CTA per (kv head, request, split): its warps walk the split's tokens with an
//                            online softmax for the whole GQA group, merge through shared memory and across the cluster of
//                            the splits, or leave a partial (max, sum, acc) for paged_attn_merge_kernel.
// A page id outside the pool is never dereferenced: the kernel records PTB_ERR_BOUNDS and skips the page.
#include "common.cuh"
#include <algorithm>

namespace ptb {

constexpr int PAGE = 64;
constexpr int PA_WARPS = 8;
constexpr int PA_CLUSTER = 16;           // splits that merge within a cluster (more than eight need the attribute below)
constexpr int PA_THREADS = PA_WARPS * 32;

struct PagedWriteParams {
    __nv_bfloat16* qkv;            // [n, (H + 2 Hk) D]: q heads, then k heads, then v heads
    const int* pos;                // [n] position of each token in its request
    const int* req;                // [n] row of the page table
    const int* page_table;         // [requests, pt_stride] page ids
    int pt_stride, n_pages;
    const float* cos;              // [max_pos, D/2]
    const float* sin;
    __nv_bfloat16* k_pages;        // [n_pages, Hk, PAGE, D]
    __nv_bfloat16* v_pages;
    __nv_bfloat16* k_out;          // optional [n, Hk, D]: the rotated keys, contiguous (prompt pass)
    int n, H, Hk, D, max_pos;
    int* status;
    // when `work` is set the projection arrives as split-K partials [splits][n][(H + 2 Hk) D] fp32 (qkv is unused) and
    // the rotated q goes to q_out [n, H D] bf16
    const float* work;
    int splits;
    long long split_stride;
    __nv_bfloat16* q_out;
};

// Element `e` of token `i`'s projection row: from the bf16 row, or the sum of the split-K partials.
__device__ __forceinline__ float proj_elem(const PagedWriteParams& P, const __nv_bfloat16* row, size_t i, int e, int width) {
    if (!P.work) return __bfloat162float(row[e]);
    const float* w = P.work + i * width + e;
    float a = w[0];
    for (int s = 1; s < P.splits; ++s) a += w[(size_t)s * P.split_stride];
    return a;
}

// One CTA per token.  Rotation pairs are (j, j + D/2) within a head (the Hugging Face Llama convention).
__global__ void __launch_bounds__(256) paged_rope_write_kernel(const __grid_constant__ PagedWriteParams P) {
    pdl_wait();
    pdl_launch_dependents();
    const int i = blockIdx.x;
    const int half = P.D / 2;
    const int pos = P.pos[i];
    const int width = (P.H + 2 * P.Hk) * P.D;
    __nv_bfloat16* row = P.qkv ? P.qkv + (size_t)i * width : nullptr;
    const int page_slot = pos / PAGE, in_page = pos % PAGE;
    const int page = P.page_table[(size_t)P.req[i] * P.pt_stride + min(page_slot, P.pt_stride - 1)];
    const bool ok = pos >= 0 && pos < P.max_pos && page_slot < P.pt_stride && page >= 0 && page < P.n_pages;
    if (!ok) {
        if (threadIdx.x == 0 && P.status) atomicExch(P.status, PTB_ERR_BOUNDS);
        return;
    }
    const float* cs = P.cos + (size_t)pos * half;
    const float* sn = P.sin + (size_t)pos * half;
    const int n_rot = (P.H + P.Hk) * half;
    for (int e = threadIdx.x; e < n_rot; e += blockDim.x) {
        const int h = e / half, j = e % half;
        const float a = proj_elem(P, row, i, h * P.D + j, width), b = proj_elem(P, row, i, h * P.D + j + half, width);
        const float c = cs[j], s = sn[j];
        const __nv_bfloat16 ra = __float2bfloat16_rn(a * c - b * s), rb = __float2bfloat16_rn(b * c + a * s);
        if (h < P.H) {
            __nv_bfloat16* hp = P.work ? P.q_out + ((size_t)i * P.H + h) * P.D : row + (size_t)h * P.D;
            hp[j] = ra; hp[j + half] = rb;
        } else {
            const int kh = h - P.H;
            __nv_bfloat16* dst = P.k_pages + (((size_t)page * P.Hk + kh) * PAGE + in_page) * P.D;
            dst[j] = ra; dst[j + half] = rb;
            if (P.k_out) {
                __nv_bfloat16* ko = P.k_out + ((size_t)i * P.Hk + kh) * P.D;
                ko[j] = ra; ko[j + half] = rb;
            }
        }
    }
    const int v0 = (P.H + P.Hk) * P.D;
    for (int e = threadIdx.x; e < P.Hk * P.D; e += blockDim.x) {
        const int kh = e / P.D, d = e % P.D;
        P.v_pages[(((size_t)page * P.Hk + kh) * PAGE + in_page) * P.D + d] =
            P.work ? __float2bfloat16_rn(proj_elem(P, row, i, v0 + e, width)) : row[v0 + e];
    }
}

// The same in 16-byte pieces, for bf16 rows or (PARTS) split-K partials: a thread rotates eight pairs (two 16-byte loads, D/16 threads a head) or moves eight
// values.  What bounds it is bytes: each value is read once and written once or twice.  One CTA per token either way; two bytes
// an access it cost the 8-request, 14192-token prompt pass of a 4096-wide model (8 layers, then 16 tokens each) 88.4 ms in place of 84.2.
template <bool PARTS>
__global__ void __launch_bounds__(256) paged_rope_write_vec_kernel(const __grid_constant__ PagedWriteParams P) {
    pdl_wait();
    pdl_launch_dependents();
    const int i = blockIdx.x;
    const int half = P.D / 2, per_half = half / 8, per_head = P.D / 8;
    const int pos = P.pos[i];
    const size_t width = (size_t)(P.H + 2 * P.Hk) * P.D;
    uint4* row = PARTS ? nullptr : reinterpret_cast<uint4*>(P.qkv + i * width);
    // eight neighbouring values of the projection, from 16-byte piece `at` on
    auto load8 = [&](int at, float* f) {
        if constexpr (PARTS) {
            const float4* w = reinterpret_cast<const float4*>(P.work + i * width) + 2 * at;
            float4 a = w[0], b = w[1];
#pragma unroll 4
            for (int s = 1; s < P.splits; ++s) {
                const float4* ws = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(w) + (size_t)s * P.split_stride);
                const float4 c = ws[0], d = ws[1];
                a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
                b.x += d.x; b.y += d.y; b.z += d.z; b.w += d.w;
            }
            f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
        } else {
            const uint4 raw = row[at];
            const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
            for (int x = 0; x < 4; ++x) { const float2 v = __bfloat1622float2(h2[x]); f[2 * x] = v.x; f[2 * x + 1] = v.y; }
        }
    };
    const int page_slot = pos / PAGE, in_page = pos % PAGE;
    const int page = P.page_table[(size_t)P.req[i] * P.pt_stride + max(0, min(page_slot, P.pt_stride - 1))];
    const bool ok = pos >= 0 && pos < P.max_pos && page_slot < P.pt_stride && page >= 0 && page < P.n_pages;
    if (!ok) {
        if (threadIdx.x == 0 && P.status) atomicExch(P.status, PTB_ERR_BOUNDS);
        return;
    }
    const float4* cs = reinterpret_cast<const float4*>(P.cos + (size_t)pos * half);
    const float4* sn = reinterpret_cast<const float4*>(P.sin + (size_t)pos * half);
    auto slot = [&](__nv_bfloat16* pages, int kh) { return reinterpret_cast<uint4*>(pages + (((size_t)page * P.Hk + kh) * PAGE + in_page) * P.D); };
    const int n_rot = (P.H + P.Hk) * per_half, n_all = n_rot + P.Hk * per_head;
#pragma unroll 4
    for (int e = threadIdx.x; e < n_all; e += 256) {
        if (e < n_rot) {
            const int h = e / per_half, j = e - h * per_half;
            float lo[8], hi[8];
            load8(h * per_head + j, lo);
            load8(h * per_head + per_half + j, hi);
            const float4 c0 = cs[2 * j], c1 = cs[2 * j + 1], s0 = sn[2 * j], s1 = sn[2 * j + 1];
            const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w}, s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
            uint4 ra, rb;
            __nv_bfloat162 *oa = reinterpret_cast<__nv_bfloat162*>(&ra), *ob = reinterpret_cast<__nv_bfloat162*>(&rb);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const float2 a = make_float2(lo[2 * x], lo[2 * x + 1]), b = make_float2(hi[2 * x], hi[2 * x + 1]);
                oa[x] = __floats2bfloat162_rn(a.x * c[2 * x] - b.x * s[2 * x], a.y * c[2 * x + 1] - b.y * s[2 * x + 1]);
                ob[x] = __floats2bfloat162_rn(b.x * c[2 * x] + a.x * s[2 * x], b.y * c[2 * x + 1] + a.y * s[2 * x + 1]);
            }
            uint4* q_row = PARTS ? reinterpret_cast<uint4*>(P.q_out + (size_t)i * P.H * P.D) : row;
            uint4* dst = h < P.H ? q_row + h * per_head : slot(P.k_pages, h - P.H);
            dst[j] = ra; dst[per_half + j] = rb;
            if (h >= P.H && P.k_out) {
                uint4* ko = reinterpret_cast<uint4*>(P.k_out + ((size_t)i * P.Hk + h - P.H) * P.D);
                ko[j] = ra; ko[per_half + j] = rb;
            }
        } else {
            const int c = e - n_rot, kh = c / per_head, d = c - kh * per_head;
            if constexpr (PARTS) {
                float f[8];
                load8((P.H + P.Hk) * per_head + c, f);
                uint4 o;
                __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int x = 0; x < 4; ++x) oh[x] = __floats2bfloat162_rn(f[2 * x], f[2 * x + 1]);
                slot(P.v_pages, kh)[d] = o;
            } else {
                slot(P.v_pages, kh)[d] = row[(P.H + P.Hk) * per_head + c];
            }
        }
    }
}

struct PagedAttnParams {
    const __nv_bfloat16* q;        // [B, q_stride] with head h at column h * D
    long long q_stride;
    __nv_bfloat16* out;            // [B, H * D]
    const int* lens;               // [B] tokens in the cache (the new one included)
    const int* page_table;
    int pt_stride, n_pages;
    const __nv_bfloat16* k_pages;
    const __nv_bfloat16* v_pages;
    float* work;                   // [B, H, nsplit, D + 2] partial (acc, max, sum) when nsplit > PA_CLUSTER
    int B, H, Hk, nsplit;
    float scale_log2;              // softmax scale times log2(e)
    int q_wide;                    // rows of q start on 16 bytes
    int cluster;                   // the splits of a (kv head, request) are a cluster
    int* status;
};

__device__ __forceinline__ void unpack8(const uint4& raw, float* f) {
    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 v = __bfloat1622float2(h2[i]); f[2 * i] = v.x; f[2 * i + 1] = v.y; }
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr, uint32_t rank) {
    float v;
    asm volatile("{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %1, %2;\n ld.shared::cluster.f32 %0, [a];\n}" : "=f"(v) : "r"(addr), "r"(rank) : "memory");
    return v;
}
__device__ __forceinline__ void pa_cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// D / 8 lanes a token, eight values a lane: a warp's load covers whole rows, K and V of its group of TG tokens are requested together, and its
// online softmax needs no other warp until the end.  Bound by the cache's bytes at long contexts and by latency at short ones, so
// tokens, not pages, are dealt to warps: one lane per token and one warp per page had nine warps work on a request of 540 tokens
// (per kv head of 128, groups of 4: 27 us, and 3 for the merge).  Up to sixteen splits are the CTAs of a cluster, which merge through
// distributed shared memory; more leave partials for paged_attn_merge_kernel.
// V16: the pool of values starts on 16 bytes (otherwise its values come in 4-byte pieces; as a branch in one kernel that cost 4 to 7 %).
template <int D, int G, bool V16>
__global__ void __launch_bounds__(PA_THREADS, G == 8 ? 1 : 2) paged_attn_decode_kernel(const __grid_constant__ PagedAttnParams P) {
    constexpr int LPT = D / 8, TPI = 32 / LPT, U = G == 8 ? 2 : 4, TG = TPI * U;
    static_assert(D == 128 || D == 64, "head size 128 or 64");
    static_assert(PAGE % TG == 0, "a group lies in one page");
    __shared__ __align__(16) float acc_s[PA_WARPS][G][D];
    __shared__ float ml_s[PA_WARPS][G][2];
    __shared__ float part[G * D], part_ml[2 * G];
    const int kvh = blockIdx.x, b = blockIdx.y, split = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / LPT, l = lane % LPT;
    pdl_wait();
    pdl_launch_dependents();
    uint4 qr[G];
    {
        const __nv_bfloat16* qp = P.q + (size_t)b * P.q_stride + (size_t)kvh * G * D + l * 8;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            if (P.q_wide) {
                qr[g] = *reinterpret_cast<const uint4*>(qp + g * D);
            } else {
                __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&qr[g]);
#pragma unroll
                for (int i = 0; i < 8; ++i) e[i] = qp[g * D + i];
            }
        }
    }
    const int len = min(P.lens[b], P.pt_stride * PAGE);
    // tokens of this split, in groups dealt to the warps round-robin
    const int per = ((len + P.nsplit - 1) / P.nsplit + TG - 1) / TG * TG;
    const int lo = split * per, hi = min(lo + per, len);
    float m[G], sum[G], acc[G][8];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m[g] = -INFINITY; sum[g] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[g][i] = 0.f;
    }
    for (int t0 = lo + warp * TG; t0 < hi; t0 += PA_WARPS * TG) {
        const int page = P.page_table[(size_t)b * P.pt_stride + t0 / PAGE];
        if (page < 0 || page >= P.n_pages) {
            if (lane == 0 && P.status) atomicExch(P.status, PTB_ERR_BOUNDS);
            continue;
        }
        const size_t at = (((size_t)page * P.Hk + kvh) * PAGE + t0 % PAGE + sub) * D + l * 8;
        uint4 kr[U], vr[U];
#pragma unroll
        for (int u = 0; u < U; ++u) kr[u] = *reinterpret_cast<const uint4*>(P.k_pages + at + (size_t)u * TPI * D);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t* v = reinterpret_cast<const uint32_t*>(P.v_pages + at + (size_t)u * TPI * D);
            if constexpr (V16) vr[u] = *reinterpret_cast<const uint4*>(v);
            else vr[u] = make_uint4(v[0], v[1], v[2], v[3]);
        }
        float s[U][G];
        {
            float kf[U][8];
#pragma unroll
            for (int u = 0; u < U; ++u) unpack8(kr[u], kf[u]);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float qf[8];
                unpack8(qr[g], qf);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    float d0 = qf[0] * kf[u][0], d1 = qf[1] * kf[u][1];
#pragma unroll
                    for (int i = 2; i < 8; i += 2) { d0 += qf[i] * kf[u][i]; d1 += qf[i + 1] * kf[u][i + 1]; }
                    s[u][g] = d0 + d1;
                }
            }
        }
#pragma unroll
        for (int o = LPT / 2; o > 0; o >>= 1)
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int g = 0; g < G; ++g) s[u][g] += __shfl_xor_sync(0xffffffffu, s[u][g], o);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = t0 + u * TPI + sub < len;
#pragma unroll
            for (int g = 0; g < G; ++g) s[u][g] = in ? s[u][g] * P.scale_log2 : -INFINITY;
            if (!in) vr[u] = make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float mx = s[0][g];
#pragma unroll
            for (int u = 1; u < U; ++u) mx = fmaxf(mx, s[u][g]);
#pragma unroll
            for (int o = LPT; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m[g], mx), m_use = m_new == -INFINITY ? 0.f : m_new;
            const float corr = exp2f(m[g] - m_use);
            float add = 0.f;
#pragma unroll
            for (int u = 0; u < U; ++u) { s[u][g] = exp2f(s[u][g] - m_use); add += s[u][g]; }
            sum[g] = sum[g] * corr + add;                       // of this lane's tokens
            m[g] = m_new;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[g][i] *= corr;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float vf[8];
            unpack8(vr[u], vf);
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[g][i] += s[u][g] * vf[i];
        }
    }
    // the lanes that hold the same values of different tokens, then the warps
#pragma unroll
    for (int g = 0; g < G; ++g) {
#pragma unroll
        for (int o = LPT; o < 32; o <<= 1) {
            sum[g] += __shfl_xor_sync(0xffffffffu, sum[g], o);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[g][i] += __shfl_xor_sync(0xffffffffu, acc[g][i], o);
        }
        if (sub == 0) {
            float4* dst = reinterpret_cast<float4*>(&acc_s[warp][g][l * 8]);
            dst[0] = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
            dst[1] = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
        }
        if (lane == 0) { ml_s[warp][g][0] = m[g]; ml_s[warp][g][1] = sum[g]; }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < G * D; e += PA_THREADS) {
        const int g = e / D, d = e % D;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < PA_WARPS; ++w) M = fmaxf(M, ml_s[w][g][0]);
        float L = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < PA_WARPS; ++w) {
            const float f = ml_s[w][g][0] == -INFINITY ? 0.f : exp2f(ml_s[w][g][0] - M);
            L += ml_s[w][g][1] * f;
            o += acc_s[w][g][d] * f;
        }
        if (P.nsplit == 1) {
            P.out[((size_t)b * P.H + kvh * G + g) * D + d] = __float2bfloat16_rn(L > 0.f ? o / L : 0.f);
        } else if (P.cluster) {
            part[e] = o;
            if (d == 0) { part_ml[g] = M; part_ml[G + g] = L; }
        } else {
            float* wk = P.work + (((size_t)b * P.H + kvh * G + g) * P.nsplit + split) * (D + 2);
            wk[d] = o;
            if (d == 0) { wk[D] = M; wk[D + 1] = L; }
        }
    }
    if (!P.cluster) return;
    // split r of the cluster finishes every nsplit-th output
    pa_cluster_sync();
    const uint32_t a_part = smem_u32(part), a_ml = smem_u32(part_ml);
    for (int e = threadIdx.x * P.nsplit + split; e < G * D; e += PA_THREADS * P.nsplit) {
        const int g = e / D;
        float M = -INFINITY, L = 0.f, o = 0.f;
        for (int r = 0; r < P.nsplit; ++r) M = fmaxf(M, ld_cluster_f32(a_ml + g * 4, r));
        for (int r = 0; r < P.nsplit; ++r) {
            const float mr = ld_cluster_f32(a_ml + g * 4, r);
            const float f = mr == -INFINITY ? 0.f : exp2f(mr - M);
            L += ld_cluster_f32(a_ml + (G + g) * 4, r) * f;
            o += ld_cluster_f32(a_part + e * 4, r) * f;
        }
        P.out[((size_t)b * P.H + kvh * G + g) * D + e % D] = __float2bfloat16_rn(L > 0.f ? o / L : 0.f);
    }
    pa_cluster_sync();                             // the others may still read this CTA's part
}

// Combine the splits of one (request, head): grid (H, B), D threads.
__global__ void paged_attn_merge_kernel(const float* __restrict__ work, __nv_bfloat16* __restrict__ out, int H, int D, int nsplit) {
    pdl_wait();
    pdl_launch_dependents();
    const int h = blockIdx.x, b = blockIdx.y, d = threadIdx.x;
    const float* wk = work + ((size_t)b * H + h) * nsplit * (D + 2);
    float M = -INFINITY;
    for (int s = 0; s < nsplit; ++s) M = fmaxf(M, wk[s * (D + 2) + D]);
    float L = 0.f, o = 0.f;
    for (int s = 0; s < nsplit; ++s) {
        const float ms = wk[s * (D + 2) + D];
        const float f = ms == -INFINITY ? 0.f : exp2f(ms - M);
        L += wk[s * (D + 2) + D + 1] * f;
        o += wk[s * (D + 2) + d] * f;
    }
    out[((size_t)b * H + h) * D + d] = __float2bfloat16_rn(L > 0.f ? o / L : 0.f);
}

template <int D, int G, bool V16>
static cudaError_t launch_decode_g(const PagedAttnParams& p, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(p.Hk, p.B, p.nsplit);
    cfg.blockDim = dim3(PA_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (ptb_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.cluster) {
        static bool wide = false;
        if (p.nsplit > 8 && !wide) {
            const cudaError_t e = cudaFuncSetAttribute(paged_attn_decode_kernel<D, G, V16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e != cudaSuccess) return e;
            wide = true;
        }
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1; attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = (unsigned)p.nsplit;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, paged_attn_decode_kernel<D, G, V16>, p);
}

template <int D>
static int launch_decode(const PagedAttnParams& p, int G, cudaStream_t st) {
    cudaError_t e;
    const bool v16 = !((uintptr_t)p.v_pages & 15);
    switch (G) {
        case 1: e = v16 ? launch_decode_g<D, 1, true>(p, st) : launch_decode_g<D, 1, false>(p, st); break;
        case 2: e = v16 ? launch_decode_g<D, 2, true>(p, st) : launch_decode_g<D, 2, false>(p, st); break;
        case 4: e = v16 ? launch_decode_g<D, 4, true>(p, st) : launch_decode_g<D, 4, false>(p, st); break;
        case 8: e = v16 ? launch_decode_g<D, 8, true>(p, st) : launch_decode_g<D, 8, false>(p, st); break;
        default: ptb_set_error("paged attention: group size %d not in {1, 2, 4, 8}", G); return -1;
    }
    PTB_CUDA_OK(e);
    return 0;
}

}  // namespace ptb

using namespace ptb;

// Rotate q and k of `n` new tokens, store k and v in their page slots.  qkv: [n, (H + 2 Hk) D] bf16 (q rotated in
// place); pos / req: [n]; page_table: [requests, pt_stride]; cos / sin: [max_pos, D/2] fp32; k_out optional.
static int rope_write(void* qkv, const float* work, int splits, void* q_out, int n, int H, int Hk, int D, const int* pos, const int* req,
                      const int* page_table, int pt_stride, int n_pages, const float* cos, const float* sin, int max_pos, void* k_pages,
                      void* v_pages, void* k_out, int* status, cudaStream_t st) {
    if (n <= 0) return 0;
    if (D % 2) { ptb_set_error("paged_rope_write: odd head size"); return -1; }
    PagedWriteParams p;
    p.work = work; p.splits = splits; p.split_stride = (long long)n * (H + 2 * Hk) * D; p.q_out = (__nv_bfloat16*)q_out;
    p.qkv = (__nv_bfloat16*)qkv; p.pos = pos; p.req = req; p.page_table = page_table; p.pt_stride = pt_stride; p.n_pages = n_pages;
    p.cos = cos; p.sin = sin; p.k_pages = (__nv_bfloat16*)k_pages; p.v_pages = (__nv_bfloat16*)v_pages; p.k_out = (__nv_bfloat16*)k_out;
    p.n = n; p.H = H; p.Hk = Hk; p.D = D; p.max_pos = max_pos; p.status = status;
    // 16-byte pieces: half a head is a multiple of eight values and every base is aligned (a head then is too)
    const bool vec = D % 16 == 0 && !(((uintptr_t)qkv | (uintptr_t)work | (uintptr_t)q_out | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)k_out | (uintptr_t)cos |
                                       (uintptr_t)sin) & 15);
    PTB_CUDA_OK(ptb_launch(!vec ? paged_rope_write_kernel : work ? paged_rope_write_vec_kernel<true> : paged_rope_write_vec_kernel<false>, dim3(n), dim3(256), 0, st,
                           ptb_pdl_enabled(), p));
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}

PTB_API int ptb_paged_rope_write(void* qkv, int n, int H, int Hk, int D, const int* pos, const int* req, const int* page_table,
                                 int pt_stride, int n_pages, const float* cos, const float* sin, int max_pos, void* k_pages,
                                 void* v_pages, void* k_out, int* status, cudaStream_t st) {
    return rope_write(qkv, nullptr, 0, nullptr, n, H, Hk, D, pos, req, page_table, pt_stride, n_pages, cos, sin, max_pos, k_pages, v_pages, k_out,
                      status, st);
}

// The same, reading the projection as split-K partials `work` [splits][n][(H + 2 Hk) D] fp32 (what ptb_gemm_bf16_splitk_partials
// leaves) and writing the rotated q to q_out [n, H D] bf16: the sum of the partials costs no launch of its own.
PTB_API int ptb_paged_rope_write_partials(const float* work, int splits, void* q_out, int n, int H, int Hk, int D, const int* pos,
                                          const int* req, const int* page_table, int pt_stride, int n_pages, const float* cos,
                                          const float* sin, int max_pos, void* k_pages, void* v_pages, int* status, cudaStream_t st) {
    if (!work || splits < 1 || !q_out) { ptb_set_error("paged_rope_write_partials: needs partials and an output for q"); return -1; }
    return rope_write(nullptr, work, splits, q_out, n, H, Hk, D, pos, req, page_table, pt_stride, n_pages, cos, sin, max_pos, k_pages, v_pages,
                      nullptr, status, st);
}

// Floats of workspace ptb_paged_attn_decode needs (up to sixteen splits merge on the chip).
PTB_API long long ptb_paged_attn_work_floats(int B, int H, int D, int nsplit) { return nsplit > PA_CLUSTER ? (long long)B * H * nsplit * (D + 2) : 0; }

// One new token per request attends to its pages.  q: [B, q_stride] bf16; out: [B, H D] bf16; lens: [B].
PTB_API int ptb_paged_attn_decode(const void* q, long long q_stride, void* out, int B, int H, int Hk, int D, const int* lens,
                                  const int* page_table, int pt_stride, int n_pages, const void* k_pages, const void* v_pages,
                                  float scale, float* work, int nsplit, int* status, cudaStream_t st) {
    if (B <= 0) return 0;
    if (Hk <= 0 || H % Hk) { ptb_set_error("paged attention: %d heads over %d kv heads", H, Hk); return -1; }
    if (((uintptr_t)k_pages & 15) || ((uintptr_t)v_pages & 3)) { ptb_set_error("paged attention: keys need a 16-byte aligned pool, values a 4-byte aligned one"); return -1; }
    if (nsplit < 1 || (nsplit > PA_CLUSTER && !work)) { ptb_set_error("paged attention: nsplit %d needs a workspace", nsplit); return -1; }
    PagedAttnParams p;
    p.q = (const __nv_bfloat16*)q; p.q_stride = q_stride; p.out = (__nv_bfloat16*)out; p.lens = lens; p.page_table = page_table;
    p.pt_stride = pt_stride; p.n_pages = n_pages; p.k_pages = (const __nv_bfloat16*)k_pages; p.v_pages = (const __nv_bfloat16*)v_pages;
    p.work = work; p.B = B; p.H = H; p.Hk = Hk; p.nsplit = nsplit; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
    p.cluster = nsplit > 1 && nsplit <= PA_CLUSTER;
    p.q_wide = !((uintptr_t)q & 15) && q_stride % 8 == 0;
    int rc;
    if (D == 128) rc = launch_decode<128>(p, H / Hk, st);
    else if (D == 64) rc = launch_decode<64>(p, H / Hk, st);
    else { ptb_set_error("paged attention: head size %d not in {64, 128}", D); return -1; }
    if (rc) return rc;
    if (nsplit > PA_CLUSTER)
        PTB_CUDA_OK(ptb_launch(paged_attn_merge_kernel, dim3(H, B), dim3(D), 0, st, ptb_pdl_enabled(), (const float*)work, (__nv_bfloat16*)out, H, D, nsplit));
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}
