// Dequantisation to bf16 for the batched prompt pass: whole matrices from the GEMV streaming layout
// ([segment][row][segment bytes], see decode_kernels.cuh) and rows of the embedding table chosen by token id.
// The prompt is then processed with the tcgen05 GEMM instead of one matrix-vector product per token
// (the reference dequantises per tile inside its prefill GEMM, aten/src/ATen/cuda/CUDAQuantGemv.cu:1115-1190).
#include "decode_kernels.cuh"

namespace ptb {

// value e (0..255) of a Q4_K super-block at `bp` (GGUF byte layout)
__device__ __forceinline__ float q4k_value(const uint8_t* bp, int e) {
    const float d = __half2float(*reinterpret_cast<const __half*>(bp));
    const float dmin = __half2float(*reinterpret_cast<const __half*>(bp + 2));
    const uint8_t* s = bp + 4;
    const int is = e >> 5;
    int scv, mv;
    if (is < 4) { scv = s[is] & 63; mv = s[is + 4] & 63; }
    else { scv = (s[is + 4] & 0xF) | ((s[is - 4] >> 6) << 4); mv = (s[is + 4] >> 4) | ((s[is] >> 6) << 4); }
    const uint8_t qb = bp[16 + (e >> 6) * 32 + (e & 31)];
    const int q = (is & 1) ? (qb >> 4) : (qb & 0xF);
    return d * scv * q - dmin * mv;
}
// value e of block b of a Q6_K structure-of-arrays segment/row of nb blocks: ql[nb*128] | qh[nb*64] | scales[nb*16] | d[nb]
__device__ __forceinline__ float q6k_value(const uint8_t* seg, int nb, int b, int e) {
    const int n = e >> 7, r = e & 127, quad = r >> 5, l = r & 31;
    const uint8_t qlb = seg[b * 128 + n * 64 + (quad & 1) * 32 + l];
    const uint8_t qhb = seg[nb * 128 + b * 64 + n * 32 + l];
    const int lo4 = (quad >> 1) ? (qlb >> 4) : (qlb & 0xF);
    const int hi2 = (qhb >> (2 * quad)) & 3;
    const int q = (lo4 | (hi2 << 4)) - 32;
    const int8_t scv = reinterpret_cast<const int8_t*>(seg + nb * 192 + b * 16)[e >> 4];
    const float d = __half2float(*reinterpret_cast<const __half*>(seg + nb * 208 + b * 2));
    return d * scv * q;
}

__device__ __forceinline__ uint4 pack8(const float* v) {
    uint4 o;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    return o;
}
// Q4_K and Q6_K in tiles of 16 rows.  A warp takes eight rows of one 256-value block: every lane reads eight packed bytes (Q4_K: one
// piece with both nibbles, two rows a step; Q6_K: two pieces of low bits and one of high bits, four rows a step) and stores 16-byte
// pieces of the bf16 rows, all loads of the eight rows before the first store.  Bound by the bytes written (2 a value against 0.56 or
// 0.82 read); one value a thread, with its scales unpacked again for each, took 35 us on average over the matrices of a 2560-wide layer
// (a prompt of 1999 tokens through 12 such layers: 15.1 ms, now 13.0).
// Matrices of one width that are read together (q, k, v; gate, up) are one launch into one stack of rows, each with its own type.
constexpr int DQ_WARPS = 8, DQ_PARTS = 4;
struct DequantGroup {
    const uint8_t* w[DQ_PARTS];
    int qtype[DQ_PARTS], rows[DQ_PARTS], row0[DQ_PARTS];
    long long first[DQ_PARTS + 1];      // first item of each part, the unused ones and the end last
    int nblk;
    __nv_bfloat16* out;
};
__global__ void __launch_bounds__(DQ_WARPS * 32) dequant_t16_vec_kernel(const __grid_constant__ DequantGroup G) {
    const int lane = threadIdx.x & 31;
    long long item = (long long)blockIdx.x * DQ_WARPS + (threadIdx.x >> 5);       // (part, tile, block, upper or lower eight rows)
    if (item >= G.first[DQ_PARTS]) return;
    int part_no = 0;
#pragma unroll
    for (int i = 1; i < DQ_PARTS; ++i) part_no += item >= G.first[i];
    item -= G.first[part_no];
    const uint8_t* __restrict__ w = G.w[part_no];
    const int N = G.rows[part_no], nblk = G.nblk;
    __nv_bfloat16* __restrict__ out = G.out + (size_t)G.row0[part_no] * nblk * 256;
    const int r8 = (int)(item & 1) * 8;
    const int b = (int)((item >> 1) % nblk), tile = (int)((item >> 1) / nblk);
    const int row0 = tile * 16 + r8;
    if (row0 >= N) return;
    __nv_bfloat16* o = out + (size_t)row0 * nblk * 256 + (size_t)b * 256;
    const size_t pitch = (size_t)nblk * 256;
    if (G.qtype[part_no] == QT_Q4K) {
        const uint8_t* blk = w + (((size_t)tile * nblk + b) * 16 + r8) * 144;
        const int rr = lane >> 4, g = (lane >> 2) & 3, part = lane & 3;                 // 64-value group, its eight bytes
        uint4 head[4];
        uint2 q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint8_t* bp = blk + (i * 2 + rr) * 144;
            head[i] = __ldg(reinterpret_cast<const uint4*>(bp));
            q[i] = __ldg(reinterpret_cast<const uint2*>(bp + 16 + g * 32 + part * 8));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 dm = __half22float2(*reinterpret_cast<const __half2*>(&head[i].x));
            // scales 2 g and 2 g + 1 (six bits each): bytes of the three words after d and dmin
            const uint32_t s0 = head[i].y >> (16 * (g & 1)), s1 = head[i].z >> (16 * (g & 1)), s2 = head[i].w >> (16 * (g & 1));
            const uint32_t sc = g < 2 ? s0 & 0x3f3fu : (s2 & 0x0f0fu) | ((s0 >> 2) & 0x3030u);
            const uint32_t mn = g < 2 ? s1 & 0x3f3fu : ((s2 >> 4) & 0x0f0fu) | ((s1 >> 2) & 0x3030u);
            const float d0 = dm.x * (float)(sc & 255u), d1 = dm.x * (float)((sc >> 8) & 255u), m0 = dm.y * (float)(mn & 255u), m1 = dm.y * (float)((mn >> 8) & 255u);
            float lo[8], hi[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const uint32_t by = ((x < 4 ? q[i].x : q[i].y) >> (8 * (x & 3))) & 255u;
                lo[x] = d0 * (float)(by & 15u) - m0;
                hi[x] = d1 * (float)(by >> 4) - m1;
            }
            if (row0 + i * 2 + rr < N) {
                uint4* dst = reinterpret_cast<uint4*>(o + (i * 2 + rr) * pitch + g * 64);
                dst[part] = pack8(lo);
                dst[4 + part] = pack8(hi);
            }
        }
    } else {
        const uint8_t* blk = w + ((size_t)tile * nblk + b) * 3360;
        const int sub = lane >> 3, n = (lane >> 2) & 1, part = lane & 3;                // half of the block, its eight columns of four quarters
        uint2 l0[2], l1[2], h[2];
        uint4 sc[2];
        float d[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int rr = r8 + i * 4 + sub, c0 = n * 4 + (part >> 1), byte = (part & 1) * 8;
            l0[i] = __ldg(reinterpret_cast<const uint2*>(blk + rr * 128 + ((c0 ^ (rr & 7)) << 4) + byte));
            l1[i] = __ldg(reinterpret_cast<const uint2*>(blk + rr * 128 + (((c0 + 2) ^ (rr & 7)) << 4) + byte));
            h[i] = __ldg(reinterpret_cast<const uint2*>(blk + 2048 + rr * 64 + (((n * 2 + (part >> 1)) ^ ((rr >> 1) & 3)) << 4) + byte));
            sc[i] = __ldg(reinterpret_cast<const uint4*>(blk + 3072 + rr * 16));
            d[i] = __half2float(*reinterpret_cast<const __half*>(blk + 3328 + rr * 2));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int rr = i * 4 + sub;
            const uint32_t s_lo = n ? sc[i].z : sc[i].x, s_hi = n ? sc[i].w : sc[i].y;   // eight scales of this half: quarter * 2 + (column >= 16)
            uint4* dst = reinterpret_cast<uint4*>(o + rr * pitch + n * 128);
#pragma unroll
            for (int quad = 0; quad < 4; ++quad) {
                const uint32_t sw = (quad < 2 ? s_lo : s_hi) >> (8 * ((quad & 1) * 2 + (part >> 1)));
                const float ds = d[i] * (float)(int)(int8_t)(sw & 255u);
                float v[8];
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const uint2 lw = (quad & 1) ? l1[i] : l0[i];
                    const uint32_t lb = ((x < 4 ? lw.x : lw.y) >> (8 * (x & 3))) & 255u, hb = ((x < 4 ? h[i].x : h[i].y) >> (8 * (x & 3))) & 255u;
                    const uint32_t qv = ((quad >> 1) ? lb >> 4 : lb & 15u) | (((hb >> (2 * quad)) & 3u) << 4);
                    v[x] = ds * (float)((int)qv - 32);
                }
                if (row0 + rr < N) dst[quad * 4 + part] = pack8(v);
            }
        }
    }
}

// grid (nblk, ceil(N / 4)), 256 threads: thread e of the block handles element e of 4 consecutive rows
__global__ void __launch_bounds__(256) dequant_segmajor_kernel(const uint8_t* __restrict__ w, int qtype, int N, int nblk, int KS,
                                                               int seg_base, int seg_rem, __nv_bfloat16* __restrict__ out) {
    const int b = blockIdx.x, e = threadIdx.x;
    // segment of block b: the first seg_rem segments hold seg_base + 1 blocks
    const int big = seg_rem * (seg_base + 1);
    int s, bi;
    if (b < big) { s = b / (seg_base + 1); bi = b - s * (seg_base + 1); }
    else { s = seg_rem + (b - big) / seg_base; bi = (b - big) - (s - seg_rem) * seg_base; }
    const int nb = seg_base + (s < seg_rem ? 1 : 0);
    const int sz0 = seg_bytes(qtype, seg_base), sz1 = seg_bytes(qtype, seg_base + 1);
    const int extra = min(s, seg_rem);
    const size_t seg_off = (size_t)N * ((size_t)s * sz0 + (size_t)extra * (sz1 - sz0));
    const int sb = s < seg_rem ? sz1 : sz0;
    for (int r = blockIdx.y * 4; r < min(N, (int)blockIdx.y * 4 + 4); ++r) {
        const uint8_t* rowseg = w + seg_off + (size_t)r * sb;
        const float v = qtype == QT_Q4K ? q4k_value(rowseg + bi * 144, e) : q6k_value(rowseg, nb, bi, e);
        out[(size_t)r * nblk * 256 + (size_t)b * 256 + e] = __float2bfloat16_rn(v);
    }
}

// The tiles-of-16-rows layout of the tensor-pipe GEMV (decode_gemv_mma.cuh).  grid (nblk, ceil(N / 4)), 256 threads.
__global__ void __launch_bounds__(256) dequant_t16_kernel(const uint8_t* __restrict__ w, int qtype, int N, int nblk,
                                                          __nv_bfloat16* __restrict__ out) {
    const int b = blockIdx.x, e = threadIdx.x;
    for (int r = blockIdx.y * 4; r < min(N, (int)blockIdx.y * 4 + 4); ++r) {
        const int tile = r >> 4, rr = r & 15;
        float v;
        if (qtype == QT_Q4K) {
            v = q4k_value(w + (((size_t)tile * nblk + b) * 16 + rr) * 144, e);
        } else if (qtype == QT_Q5K) {
            // Q4_K with a fifth bit per value: bit (sub-block) of byte (value in sub-block) of the 32 bytes at offset 16
            const uint8_t* bp = w + (((size_t)tile * nblk + b) * 16 + rr) * 176;
            const float d = __half2float(*reinterpret_cast<const __half*>(bp));
            const float dmin = __half2float(*reinterpret_cast<const __half*>(bp + 2));
            const uint8_t* s = bp + 4;
            const int is = e >> 5;
            int scv, mv;
            if (is < 4) { scv = s[is] & 63; mv = s[is + 4] & 63; }
            else { scv = (s[is + 4] & 0xF) | ((s[is - 4] >> 6) << 4); mv = (s[is + 4] >> 4) | ((s[is] >> 6) << 4); }
            const uint8_t qb = bp[48 + (e >> 6) * 32 + (e & 31)];
            const int q = ((is & 1) ? (qb >> 4) : (qb & 0xF)) | (((bp[16 + (e & 31)] >> is) & 1) << 4);
            v = d * scv * q - dmin * mv;
        } else if (qtype == QT_Q8_0) {
            const uint8_t* blk = w + ((size_t)tile * nblk + b) * 4352;
            const int u = e >> 5;
            const int8_t q = reinterpret_cast<const int8_t*>(blk + rr * 256)[((u ^ (rr & 7)) << 5) | (e & 31)];
            v = __half2float(*reinterpret_cast<const __half*>(blk + 4096 + rr * 16 + u * 2)) * (float)q;
        } else if (qtype == QT_F16) {
            // four 64-value blocks of 2048 bytes make up these 256 values
            const uint8_t* blk = w + ((size_t)tile * (nblk * 4) + (size_t)b * 4 + (e >> 6)) * 2048;
            const int i = e & 63, u = i >> 4;
            v = __half2float(reinterpret_cast<const __half*>(blk + rr * 128)[((u ^ (rr & 3)) << 4) | (i & 15)]);
        } else {
            const uint8_t* blk = w + ((size_t)tile * nblk + b) * 3360;
            const int n = e >> 7, r7 = e & 127, quad = r7 >> 5, l = r7 & 31;
            const int qi = n * 64 + (quad & 1) * 32 + l, hi = n * 32 + l;
            const uint8_t qlb = blk[rr * 128 + ((((qi >> 4) ^ (rr & 7)) << 4) | (qi & 15))];
            const uint8_t qhb = blk[2048 + rr * 64 + ((((hi >> 4) ^ ((rr >> 1) & 3)) << 4) | (hi & 15))];
            const int lo4 = (quad >> 1) ? (qlb >> 4) : (qlb & 0xF);
            const int q = (lo4 | (((qhb >> (2 * quad)) & 3) << 4)) - 32;
            const int8_t scv = reinterpret_cast<const int8_t*>(blk + 3072 + rr * 16)[e >> 4];
            const float d = __half2float(*reinterpret_cast<const __half*>(blk + 3328 + rr * 2));
            v = d * scv * q;
        }
        out[(size_t)r * nblk * 256 + (size_t)b * 256 + e] = __float2bfloat16_rn(v);
    }
}

// grid (nblk, T), 256 threads: row ids[t] of a row-major table (Q4_K bytes / Q6_K SoA rows / fp16 / fp32)
__global__ void __launch_bounds__(256) dequant_rows_kernel(const uint8_t* __restrict__ table, int qtype, int rowbytes, int nblk,
                                                           const int* __restrict__ ids, float scale, int vocab, int* status,
                                                           __nv_bfloat16* __restrict__ out) {
    const int b = blockIdx.x, t = blockIdx.y, e = threadIdx.x;
    int tok = ids[t];
    if (tok < 0 || tok >= vocab) {
        if (e == 0 && b == 0) atomicExch(status, PTB_ERR_BOUNDS);
        tok = 0;
    }
    const uint8_t* row = table + (size_t)tok * rowbytes;
    const int i = b * 256 + e;
    float v;
    if (qtype == QT_Q4K) v = q4k_value(row + b * 144, e);
    else if (qtype == QT_Q6K) v = q6k_value(row, nblk, b, e);
    else if (qtype == 2) v = __half2float(reinterpret_cast<const __half*>(row)[i]);
    else v = reinterpret_cast<const float*>(row)[i];
    out[(size_t)t * nblk * 256 + i] = __float2bfloat16_rn(v * scale);
}

// D / 4 lanes a head, four values a lane: two neighbours of each half.  Bound by bytes (each value read once, k and v written twice); as
// norms, rotations, conversions and copies of their own these were eight passes and eight launches a layer.
template <int D>
__global__ void __launch_bounds__(256) prompt_heads_kernel(__nv_bfloat16* __restrict__ qkv, long long heads, int H, int Hk, const float* __restrict__ q_norm,
                                                           const float* __restrict__ k_norm, float more, float eps, const float* __restrict__ cos,
                                                           const float* __restrict__ sin, int neox, int pos0, __half* __restrict__ kc, __half* __restrict__ vc, int S) {
    constexpr int LANES = D / 4;
    const long long at = ((long long)blockIdx.x * 256 + threadIdx.x) / LANES;
    const int l = threadIdx.x % LANES, per = H + 2 * Hk;
    const bool on = at < heads;
    const int t = on ? (int)(at / per) : 0, h = on ? (int)(at % per) : 0;
    __nv_bfloat162* row = reinterpret_cast<__nv_bfloat162*>(qkv + (on ? at : 0) * D);
    const __nv_bfloat162 ra = row[l], rb = row[D / 4 + l];
    float2 a = __bfloat1622float2(ra), b = __bfloat1622float2(rb);
    const float* w = h < H ? q_norm : h < H + Hk ? k_norm : nullptr;
    float ss = a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y;
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (!on) return;
    if (h < H + Hk) {
        if (w) {
            const float rs = rsqrtf(ss / (float)D + eps);
            const float2 wa = *reinterpret_cast<const float2*>(w + 2 * l), wb = *reinterpret_cast<const float2*>(w + D / 2 + 2 * l);
            a.x *= rs * (wa.x + more); a.y *= rs * (wa.y + more); b.x *= rs * (wb.x + more); b.y *= rs * (wb.y + more);
        }
        const float* cs = cos + (size_t)(pos0 + t) * (D / 2);
        const float* sn = sin + (size_t)(pos0 + t) * (D / 2);
        if (neox) {
            const float2 c = *reinterpret_cast<const float2*>(cs + 2 * l), s = *reinterpret_cast<const float2*>(sn + 2 * l);
            const float2 x = a;
            a.x = x.x * c.x - b.x * s.x; b.x = b.x * c.x + x.x * s.x;
            a.y = x.y * c.y - b.y * s.y; b.y = b.y * c.y + x.y * s.y;
        } else {
            const float c0 = cs[l], s0 = sn[l], c1 = cs[D / 4 + l], s1 = sn[D / 4 + l];
            a = make_float2(a.x * c0 - a.y * s0, a.y * c0 + a.x * s0);
            b = make_float2(b.x * c1 - b.y * s1, b.y * c1 + b.x * s1);
        }
        row[l] = __floats2bfloat162_rn(a.x, a.y);
        row[D / 4 + l] = __floats2bfloat162_rn(b.x, b.y);
    }
    if (h >= H) {
        const bool is_k = h < H + Hk;
        __half2* dst = reinterpret_cast<__half2*>((is_k ? kc : vc) + ((size_t)(is_k ? h - H : h - H - Hk) * S + pos0 + t) * D);
        dst[l] = __floats2half2_rn(a.x, a.y);
        dst[D / 4 + l] = __floats2half2_rn(b.x, b.y);
    }
}

}  // namespace ptb

using namespace ptb;

static int dequant_group(const void* const* w, const int* qtypes, const int* rows, int n, int nblk, void* out, cudaStream_t st) {
    DequantGroup g;
    memset(&g, 0, sizeof(g));
    g.nblk = nblk;
    g.out = (__nv_bfloat16*)out;
    long long items = 0;
    int row = 0;
    for (int i = 0; i < DQ_PARTS; ++i) {
        g.first[i] = items;
        if (i >= n) continue;
        g.w[i] = (const uint8_t*)w[i]; g.qtype[i] = qtypes[i]; g.rows[i] = rows[i]; g.row0[i] = row;
        items += (long long)((rows[i] + 15) / 16) * 2 * nblk;
        row += rows[i];
    }
    for (int i = n; i < DQ_PARTS; ++i) g.first[i] = items;
    g.first[DQ_PARTS] = items;
    dequant_t16_vec_kernel<<<(unsigned)((items + DQ_WARPS - 1) / DQ_WARPS), DQ_WARPS * 32, 0, st>>>(g);
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}

// w: a matrix of N rows x cols in a GEMV streaming layout -> out bf16 [N, cols] row-major.
// layout: 0 = [segment][row][segment bytes], 1 = tiles of 16 rows.
PTB_API int ptb_dequant_weight(const void* w, int qtype, int layout, int N, int cols, void* out, cudaStream_t st) {
    if (cols % 256 || N <= 0) { ptb_set_error("dequant: %d x %d not supported", N, cols); return -1; }
    const bool tile_only = qtype == QT_Q5K || qtype == QT_Q8_0 || qtype == QT_F16;
    if (!(qtype == QT_Q4K || qtype == QT_Q6K || (tile_only && layout == 1))) {
        ptb_set_error("dequant: quantisation type %d is not available in layout %d", qtype, layout);
        return -1;
    }
    const int nblk = cols / 256;
    if (layout == 1 && !tile_only && !(((uintptr_t)w | (uintptr_t)out) & 15)) return dequant_group(&w, &qtype, &N, 1, nblk, out, st);
    if (layout == 1) {
        dequant_t16_kernel<<<dim3(nblk, (N + 3) / 4), 256, 0, st>>>((const uint8_t*)w, qtype, N, nblk, (__nv_bfloat16*)out);
        PTB_CUDA_OK(cudaGetLastError());
        return 0;
    }
    const int KS = (nblk + GEMV_SEG_BLOCKS - 1) / GEMV_SEG_BLOCKS;
    dequant_segmajor_kernel<<<dim3(nblk, (N + 3) / 4), 256, 0, st>>>((const uint8_t*)w, qtype, N, nblk, KS, nblk / KS, nblk % KS,
                                                                    (__nv_bfloat16*)out);
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}

// `n` matrices of the same width, one below the other in `out` [sum of rows, cols]: one launch where they are Q4_K or Q6_K in tiles of 16 rows.
PTB_API int ptb_dequant_weights(const void* const* w, const int* qtypes, const int* rows, int n, int layout, int cols, void* out, cudaStream_t st) {
    if (n < 1 || n > DQ_PARTS || cols % 256) { ptb_set_error("dequant: %d matrices of %d columns not supported", n, cols); return -1; }
    bool one = layout == 1 && !((uintptr_t)out & 15);
    for (int i = 0; i < n; ++i) one = one && rows[i] > 0 && (qtypes[i] == QT_Q4K || qtypes[i] == QT_Q6K) && !((uintptr_t)w[i] & 15);
    if (one) return dequant_group(w, qtypes, rows, n, cols / 256, out, st);
    __nv_bfloat16* o = (__nv_bfloat16*)out;
    for (int i = 0; i < n; ++i) {
        if (ptb_dequant_weight(w[i], qtypes[i], layout, rows[i], cols, o, st)) return -1;
        o += (size_t)rows[i] * cols;
    }
    return 0;
}

// What stands between the packed projection of a prompt and its attention: norm of the q and k heads (weights fp32 [D] or null; add_one: they are
// stored less one), rotary positions from pos0 (pairs (j, j + D/2), or (2j, 2j + 1)), both in place and rounded once, and k and v into the
// fp16 cache [Hk, S, D].  qkv bf16 [T, (H + 2 Hk) D]; cos, sin fp32 [S, D/2]; D 64 or 128.
PTB_API int ptb_prompt_heads(void* qkv, int T, int H, int Hk, int D, const float* q_norm, const float* k_norm, int add_one, float eps, const float* cos,
                             const float* sin, int neox, int pos0, void* k_cache, void* v_cache, int S, cudaStream_t st) {
    if (T <= 0) return 0;
    if (pos0 < 0 || pos0 + T > S) { ptb_set_error("prompt heads: positions %d .. %d outside a cache of %d", pos0, pos0 + T, S); return -1; }
    if (((uintptr_t)qkv | (uintptr_t)q_norm | (uintptr_t)k_norm | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)cos | (uintptr_t)sin) & 7) { ptb_set_error("prompt heads: needs 8-byte aligned buffers"); return -1; }
    const long long heads = (long long)T * (H + 2 * Hk);
    auto go = [&](auto kern, int per_cta) {
        kern<<<(unsigned)((heads + per_cta - 1) / per_cta), 256, 0, st>>>((__nv_bfloat16*)qkv, heads, H, Hk, q_norm, k_norm, add_one ? 1.f : 0.f, eps, cos, sin, neox, pos0,
                                                                        (__half*)k_cache, (__half*)v_cache, S);
    };
    if (D == 128) go(prompt_heads_kernel<128>, 8);
    else if (D == 64) go(prompt_heads_kernel<64>, 16);
    else { ptb_set_error("prompt heads: head size %d not in {64, 128}", D); return -1; }
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}

// out[t] = scale * table[ids[t]] for T ids (device int32).  status: device word, set if an id is out of range.
PTB_API int ptb_dequant_rows(const void* table, int qtype, int rowbytes, int cols, const int* ids, int T, float scale, int vocab,
                             int* status, void* out, cudaStream_t st) {
    if (cols % 256 || T <= 0) { ptb_set_error("dequant rows: %d ids x %d columns not supported", T, cols); return -1; }
    dequant_rows_kernel<<<dim3(cols / 256, T), 256, 0, st>>>((const uint8_t*)table, qtype, rowbytes, cols / 256, ids, scale, vocab, status,
                                                             (__nv_bfloat16*)out);
    PTB_CUDA_OK(cudaGetLastError());
    return 0;
}
