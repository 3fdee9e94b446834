// The layers of a quantised model over a prompt, launched from one call.  Each layer is the same dozen launches whoever issues them: matrices with
// one input unpacked into one stack and multiplied once, one kernel between projection and attention, split-K sums that carry residual, norm and
// gate.  Issued from Python a layer of a 2560-wide model cost the host about 0.3 ms against 0.13 ms of GPU work for 128 tokens (12 layers and a
// decode step: 4.07 ms, now 2.88; logits of 57 positions: 3.36, now 2.48).
#include "ptb200.h"
#include "common.cuh"
#include <algorithm>

namespace {

struct Shape { int N, K; };
// the four products of a layer, in order
void shapes(const PtbPromptRun* r, Shape (&s)[4]) {
    const int Q = r->heads * r->D, KV = r->kv_heads * r->D;
    s[0] = {Q + 2 * KV, r->H};
    s[1] = {r->H, Q};
    s[2] = {2 * r->I, r->H};
    s[3] = {r->H, r->I};
}
int skinny(int M, Shape s, int n_sm) { return M <= 128 && s.N % 4 == 0 ? ptb_gemm_pick_splits(M, s.N, s.K, n_sm) : 0; }

// out[M, N] = x[M, K] w[N, K]^T
int product(const PtbPromptRun* r, const void* x, Shape s, void* out, cudaStream_t st) {
    const int splits = skinny(r->T, s, r->n_sm);
    if (splits > 0)
        return ptb_gemm_bf16_splitk(x, s.K, r->weights, s.K, out, s.N, r->T, s.N, s.K, nullptr, 0, splits, r->work, r->status, 0, st);
    const long long floats = ptb_gemm_work_floats(r->T, s.N, s.K, r->n_sm);
    return ptb_gemm_bf16_ws(x, s.K, 0, r->weights, s.K, 0, out, s.N, r->T, s.N, s.K, nullptr, 0, floats ? r->work : nullptr, floats, r->status, 0, st);
}

// x_out = x w^T + x_in; h = norm(x_out)
int into_stream(const PtbPromptRun* r, const void* x, Shape s, const void* x_in, void* x_out, const void* norm, cudaStream_t st) {
    const int splits = skinny(r->T, s, r->n_sm);
    if (splits > 0 && s.N <= 8192)
        return ptb_gemm_bf16_splitk_add_norm(x, s.K, r->weights, s.K, r->T, s.N, s.K, splits, r->work, x_in, x_out, norm, r->eps, r->h, r->status, 0, st);
    if (product(r, x, s, r->o, st)) return -1;
    return ptb_rmsnorm_fwd(r->o, norm, r->h, nullptr, r->T, s.N, r->eps, x_in, x_out, 1, st);
}

}  // namespace

// Floats of workspace that ptb_prompt_layers needs (T, H, heads, kv_heads, D, I and n_sm of the run are read).
PTB_API long long ptb_prompt_work_floats(const PtbPromptRun* r) {
    Shape s[4];
    shapes(r, s);
    long long most = 0;
    for (const Shape& x : s) {
        const int splits = skinny(r->T, x, r->n_sm);
        most = std::max(most, splits > 0 ? (long long)splits * r->T * x.N : ptb_gemm_work_floats(r->T, x.N, x.K, r->n_sm));
    }
    return most;
}

// Runs `n` layers: the caches filled for positions 0 .. T - 1, and, where the last layer has a next norm, the normed rows left in r->h.
PTB_API int ptb_prompt_layers(const PtbPromptLayer* layers, int n, const PtbPromptRun* r, cudaStream_t st) {
    if (r->T <= 0 || n <= 0) return 0;
    if (r->T > r->S || r->work_floats < ptb_prompt_work_floats(r)) { ptb_set_error("prompt layers: %d tokens for a cache of %d, %lld floats of workspace", r->T, r->S, r->work_floats); return -1; }
    Shape s[4];
    shapes(r, s);
    const int Q = r->heads * r->D, KV = r->kv_heads * r->D, pitch = Q + 2 * KV;
    uint16_t* qkv = (uint16_t*)r->qkv;
    const int qkv_rows[3] = {Q, KV, KV}, gu_rows[2] = {r->I, r->I};
    for (int i = 0; i < n; ++i) {
        const PtbPromptLayer& L = layers[i];
        if (ptb_dequant_weights(L.w, L.qtype, qkv_rows, 3, r->layout, r->H, r->weights, st)) return -1;
        if (product(r, r->h, s[0], r->qkv, st)) return -1;
        if (ptb_prompt_heads(r->qkv, r->T, r->heads, r->kv_heads, r->D, L.q_norm, L.k_norm, r->add_one, r->eps, r->cos, r->sin, r->neox, 0, L.k_cache, L.v_cache, r->S, st))
            return -1;
        if (!L.next_norm) break;          // nothing reads what follows
        if (ptb_flash_attn_varlen_fwd(qkv, pitch, qkv + Q, pitch, qkv + Q + KV, pitch, r->att, r->offsets, 1, r->T, r->T, r->heads, r->kv_heads, r->D, 1, r->scale,
                                      r->status, st))
            return -1;
        if (ptb_dequant_weights(L.w + 3, L.qtype + 3, &r->H, 1, r->layout, Q, r->weights, st)) return -1;
        if (into_stream(r, r->att, s[1], r->x[0], r->x[1], L.ffn_norm, st)) return -1;
        if (ptb_dequant_weights(L.w + 4, L.qtype + 4, gu_rows, 2, r->layout, r->H, r->weights, st)) return -1;
        const int splits = skinny(r->T, s[2], r->n_sm);
        if (splits > 0) {
            if (ptb_gemm_bf16_splitk_gated(r->h, r->H, r->weights, r->H, r->T, s[2].N, r->H, splits, r->work, r->gelu, r->act, r->status, 0, st)) return -1;
        } else {
            if (product(r, r->h, s[2], r->gate_up, st)) return -1;
            if (ptb_gated_act_fwd(r->gate_up, r->act, r->T, r->I, r->gelu, 1, st)) return -1;
        }
        if (ptb_dequant_weights(L.w + 6, L.qtype + 6, &r->H, 1, r->layout, r->I, r->weights, st)) return -1;
        if (into_stream(r, r->act, s[3], r->x[1], r->x[0], L.next_norm, st)) return -1;
    }
    return 0;
}
