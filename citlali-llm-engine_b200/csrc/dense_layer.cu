// A whole layer of a dense decoder over few rows (short prompts, sequences that go on by a few tokens) from one call: the six launches
//   qkv = rms(x) W_qkv^T | head norms, rotation, cache | attention | x += . W_o^T | act = silu(gate) up | x += act W_down^T
// of citlali_gemm_tc_normed, citlali_qk_norm_rope_cache and citlali_attention_prefill(_tc), with the two norms in the products.
// What bounds a step of few rows is the host: 15 us a launch from Python, where the call itself is 3 to 4, against 6 to 10 us of a kernel
// of 23 rows.  (14 layers of width 2,048, a prompt of 23: 1,360 -> 850 us a step; three sequences behind some 700 tokens that go on by 1
// or 2: 1,310 -> 1,000; 100 rows as before, 1,350: there, as in the second case by now, the kernels are as long.)
#include "api.h"
#include "common.cuh"

using namespace citlali;

static int attention_form(int nq, int nkv, int head_dim, int page_size, int max_new) {
    return citlali_attention_run_form((nq + 2 * nkv) * head_dim, nq * head_dim, head_dim, page_size, max_new);
}

extern "C" int citlali_dense_layer_supports(int nq, int nkv, int head_dim, int page_size, int max_new) {
    if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || (nq * head_dim) % 8 != 0) return 0;
    return attention_form(nq, nkv, head_dim, page_size, max_new) != 0 ? 1 : 0;
}

extern "C" int citlali_dense_layer(const CitlaliDenseLayer* l, float* x, void* qkv, void* heads, void* act, const void* in_rows,
                                   const float* in_sumsq, void* mid_rows, float* mid_sumsq, void* out_rows, float* out_sumsq,
                                   const int32_t* row_slot, const int32_t* row_pos, const int32_t* seq_start, const int32_t* seq_slot,
                                   const int32_t* seq_past, int rows, int sequences, int max_new, int32_t* error_flag, int sm_count,
                                   cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (rows > 128) {       // refused before the first launch: from there on a product may run the form that does no norm's work
        set_last_error("dense_layer: %d rows (128 at most)", rows);
        return kBadShape;
    }
    if (!citlali_dense_layer_supports(l->nq, l->nkv, l->head_dim, l->page_size, max_new) || l->hidden % 32 != 0 || l->inter % 16 != 0) {
        set_last_error("dense_layer: %d heads over %d of %d, pages of %d, width %d, inner width %d", l->nq, l->nkv, l->head_dim,
                       l->page_size, l->hidden, l->inter);
        return kBadShape;
    }
    const int width = (l->nq + 2 * l->nkv) * l->head_dim, out = l->nq * l->head_dim, groups = l->hidden / 32;
    int code = citlali_gemm_tc_normed(in_rows, l->qkv, qkv, kBF16, rows, width, l->hidden, 0, 0, error_flag, sm_count, nullptr, nullptr,
                                      in_sumsq, groups, l->hidden, l->mixer_eps, stream);
    if (code) return code;
    code = citlali_qk_norm_rope_cache(qkv, kBF16, l->q_gain, l->k_gain, l->gain_dtype, l->inv_freq, l->rotary_dim, row_slot, row_pos,
                                      l->page_table, l->page_table_stride, l->k_pool, l->v_pool, kBF16, l->page_size, rows, l->nq,
                                      l->nkv, l->head_dim, l->head_eps, 1, stream);
    if (code) return code;
    code = attention_form(l->nq, l->nkv, l->head_dim, l->page_size, max_new) == 2
               ? citlali_attention_prefill_tc(qkv, width, rows, l->k_pool, l->v_pool, l->pool_pages, l->page_table, l->page_table_stride,
                                              seq_start, seq_slot, seq_past, heads, out, sequences, max_new, l->nq, l->nkv,
                                              l->head_dim, l->page_size, l->window, l->scale, nullptr, stream)
               : citlali_attention_prefill(qkv, width, l->k_pool, l->v_pool, l->page_table, l->page_table_stride, seq_start, seq_slot,
                                           seq_past, heads, out, sequences, max_new, l->nq, l->nkv, l->head_dim, l->head_dim,
                                           l->page_size, l->window, 0, l->scale, 0.0f, nullptr, 0, nullptr, nullptr, 0, nullptr, stream);
    if (code) return code;
    code = citlali_gemm_tc_normed(heads, l->o, x, kF32, rows, l->hidden, out, 1, 0, error_flag, sm_count, mid_rows, mid_sumsq, nullptr, 0,
                                  0, 0.0f, stream);
    if (code) return code;
    code = citlali_gemm_tc_normed(mid_rows, l->gate_up, act, kBF16, rows, 2 * l->inter, l->hidden, 2, 0, error_flag, sm_count, nullptr,
                                  nullptr, mid_sumsq, groups, l->hidden, l->ff_eps, stream);
    if (code) return code;
    return citlali_gemm_tc_normed(act, l->down, x, kF32, rows, l->hidden, l->inter, 1, 0, error_flag, sm_count, out_rows, out_sumsq,
                                  nullptr, 0, 0, 0.0f, stream);
}
