// The launches of a whole layer for a short prompt, from one call of the host.
//
// A step that begins sequences is not captured (every prompt is another size), and with up to 128 tokens the device needs about
// 70 us for a layer of the Gemma 2 2B sizes while Python, the library's products and the argument conversion took 165 us for
// its eight to nine launches (one prompt of 37 tokens: 4.35 ms, of which the device was busy for 2.0).  Here they are one
// conversion and seven or eight launches (37 tokens: 2.42 ms).  The kernels are those of the other libraries, whose entry points
// the caller passes: up to 16 tokens the few-token product (rotation and cache in its epilogue), beyond the weight stream, its
// slices of K added by the kernels behind it.  Up to 32 tokens these are the launches that are made one by one otherwise; beyond,
// the products one by one are the library's and gemm_tc's (q/k/v of 64 tokens 9.2 us here with its sums, 7.0 there; down 12.6 and
// 14.6).  What a layer takes either way is at prompt_layer_ok in kernels/__init__.py.
#include "common.cuh"

extern "C" {

typedef int (*GemmStream)(const void* x, int ldx, const void* w, int ldw, void* y, int ldy, int M, int N, int K, int epilogue,
                          int out_f32, int act, float cap, float mul, int ksplit, long long part_stride, cudaStream_t stream);
typedef int (*RopeKvWriteParts)(const void* parts, int n_parts, long long part_stride, void* qkv, int ld_out, const void* positions,
                                const void* cos_sin, int n_q, int n_kv, int hd, void* k_pages, void* v_pages,
                                const void* cache_rows, int page_size, int tokens, cudaStream_t stream);
typedef int (*AttnPrefillTc)(const void* q, int q_stride, void* out, int out_stride, const void* cu_q, const void* k, const void* v,
                             int kv_stride, int total_tokens, int n_kv, int group, int hd, float scale, float cap, int window,
                             int batch, int max_q_len, int v_lbo, int v_sbo, int n_split, void* part_o, void* part_ml, int tight,
                             cudaStream_t stream);
typedef int (*ResidualRmsnorm)(void* h, const void* y, int y_dtype, int n_parts, long long part_stride, const void* w_post,
                               float eps_post, float off_post, const void* w_next, float eps_next, float off_next, int w_dtype,
                               void* out, int out_dtype, int n, int hidden, cudaStream_t stream);

typedef int (*SkinnyGemm)(const void* x, int ldx, const void* w, int ldw, void* y, int ldy, int M, int N, int K, int epilogue, int out_f32,
                          int act, float cap, int tiles, int ksplit, long long part_stride, cudaStream_t stream);
typedef int (*SkinnyQkvRope)(const void* x, int ldx, const void* w, int ldw, void* y, int ldy, int M, int K, const void* positions,
                             const void* cos_sin, int n_q, int n_kv, int hd, void* k_pages, void* v_pages, const void* cache_rows,
                             int page_size, int tiles, cudaStream_t stream);

struct PromptNorm {
    const void* weight;      // null: none
    float eps, offset;
};

struct PromptLayer {
    GemmStream gemm_stream;
    RopeKvWriteParts rope_kv_write_parts;
    AttnPrefillTc attn_prefill_tc;
    ResidualRmsnorm residual_rmsnorm;
    SkinnyGemm skinny_gemm;
    SkinnyQkvRope skinny_qkv_rope;
    void* h;                 // float [tokens][hidden], updated
    const void* x;           // bfloat16 [tokens][hidden]: the norm of h
    void* next;              // bfloat16 [tokens][hidden]: the next layer's x; null: there is none
    const void *w_qkv, *w_o, *w_gate_up, *w_down;
    void *sums, *qkv, *attn, *mid, *act;          // scratch
    const void *positions, *cos_sin, *cu_q, *cache_rows;
    void *k_pages, *v_pages;
    PromptNorm post_mixer, pre_ffn, post_ffn, after;
    int w_dtype_mid, w_dtype_end;
    int tokens, hidden, inter, n_q, n_kv, head_dim, page_size, batch, max_q_len, window;
    float scale, cap, limit;
    int activation;
    int qkv_slices, o_slices, down_slices;
    int few;                 // the few-token product, with so many tiles of 16 rows a block:
    int qkv_tiles, o_tiles, down_tiles, gate_up_stream;
};

}

// Every buffer is 16-byte aligned; weights and rows lie without gaps.
BROLM_API int brolm_prompt_layer(const PromptLayer* p, cudaStream_t stream) {
    const PromptLayer& a = *p;
    const int T = a.tokens, H = a.hidden, q = a.n_q * a.head_dim, kv = a.n_kv * a.head_dim, cols = q + 2 * kv;
    // y = x w^T in slices
    auto product = [&](const void* x, const void* w, int N, int K, int slices, int tiles) {
        const long long stride = slices > 1 ? (long long)T * N : 0;
        return a.few ? a.skinny_gemm(x, K, w, K, a.sums, N, T, N, K, 0, 1, 0, 0.0f, tiles, slices, stride, stream)
                     : a.gemm_stream(x, K, w, K, a.sums, N, T, N, K, 0, 1, 0, 0.0f, 1.0f, slices, stride, stream);
    };
    int st;
    if (a.few) {
        st = a.skinny_qkv_rope(a.x, H, a.w_qkv, H, a.qkv, cols, T, H, a.positions, a.cos_sin, a.n_q, a.n_kv, a.head_dim, a.k_pages,
                               a.v_pages, a.cache_rows, a.page_size, a.qkv_tiles, stream);
    } else {
        st = product(a.x, a.w_qkv, cols, H, a.qkv_slices, 0);
        if (st) return st;
        st = a.rope_kv_write_parts(a.sums, a.qkv_slices, (long long)T * cols, a.qkv, cols, a.positions, a.cos_sin, a.n_q, a.n_kv, a.head_dim,
                                   a.k_pages, a.v_pages, a.cache_rows, a.page_size, T, stream);
    }
    if (st) return st;
    const bf16* rows = (const bf16*)a.qkv;
    st = a.attn_prefill_tc(rows, cols, a.attn, q, a.cu_q, rows + q, rows + q + kv, cols, T, a.n_kv, a.n_q / a.n_kv, a.head_dim, a.scale,
                           a.cap, a.window, a.batch, a.max_q_len, 0, 0, 0, nullptr, nullptr, 0, stream);
    if (st) return st;
    st = product(a.attn, a.w_o, H, q, a.o_slices, a.o_tiles);
    if (st) return st;
    st = a.residual_rmsnorm(a.h, a.sums, BROLM_F32, a.o_slices, (long long)T * H, a.post_mixer.weight, a.post_mixer.eps, a.post_mixer.offset,
                            a.pre_ffn.weight, a.pre_ffn.eps, a.pre_ffn.offset, a.w_dtype_mid, a.mid, BROLM_BF16, T, H, stream);
    if (st) return st;
    st = a.few && !a.gate_up_stream
             ? a.skinny_gemm(a.mid, H, a.w_gate_up, H, a.act, a.inter, T, a.inter, H, 1, 0, a.activation, a.limit, 2, 1, 0, stream)
             : a.gemm_stream(a.mid, H, a.w_gate_up, H, a.act, a.inter, T, a.inter, H, 1, 0, a.activation, a.limit, 1.0f, 1, 0, stream);
    if (st) return st;
    st = product(a.act, a.w_down, H, a.inter, a.down_slices, a.down_tiles);
    if (st) return st;
    return a.residual_rmsnorm(a.h, a.sums, BROLM_F32, a.down_slices, (long long)T * H, a.post_ffn.weight, a.post_ffn.eps, a.post_ffn.offset,
                              a.next ? a.after.weight : nullptr, a.after.eps, a.after.offset, a.w_dtype_end, a.next,
                              a.next ? BROLM_BF16 : BROLM_F32, T, H, stream);
}

BROLM_API int brolm_prompt_layer_size() { return (int)sizeof(PromptLayer); }
