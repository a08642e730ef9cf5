// Internal declarations shared by the layer library sources (not part of the C ABI).
#pragma once
#include <cublas_v2.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "rfk_layers.h"

struct rfk_ctx {
    cublasHandle_t blas = nullptr;
    void* ws = nullptr;      // cuBLAS workspace, set explicitly so capture never allocates
    size_t ws_bytes = 0;
    void* attn_ws = nullptr;  // split workspace of the attention kernel (rfk_ctx_reserve_attention_workspace), else NULL
    size_t attn_ws_bytes = 0;
    // Every sum in the order that images have always been made with: no key split of grids of one round or more, and 128-wide
    // heads on attention with the mma.sync kernel's bits, GEMM -> softmax -> GEMM in the windows and a separate query norm. Set
    // for sessions with an image head (rfk_session_create_batched says why).
    bool reproducible = false;
    int device = 0;
};

namespace rfk_layers {
constexpr float kEpsFp16 = 0.0009765625f;   // 2^-10, the reference's kEpsFp16 (src/kernels/rmsnorm.h:9)
constexpr float kEpsFp32 = 1.1920929e-07f;  // 2^-23, the reference's kEpsFp32 (src/kernels/rmsnorm.h:10)

// rfk_decoder_layer_forward_cached with cache_flags (bit 0: keys arrive rotated and carrying the query norm weight; bit 1:
// the values are shared by the batch elements; see layers.cu); the session calls this form.
int decoder_layer_impl(rfk_ctx* ctx, const rfk_decoder_layer_weights* w, const rfk_half* x_in, rfk_half* x, rfk_half* x_out,
                       const rfk_half* pending_residual,
                       const rfk_half** pending_out, rfk_half* temp, rfk_half* proj_buf, rfk_half* qkv_buf, rfk_half* ffn_buf,
                       rfk_half* window_buf, float* cross_score_buf, float* self_score_buf, const rfk_half* K_cached,
                       const rfk_half* V_cached, int B, int Sq, int Sk, int n_keys, int dim, int num_heads, int ffn_hidden,
                       int patch_h, int patch_w, int window_size, int shift_size, const uint8_t* shift_mask,
                       const rfk_half* q_rope_cos, const rfk_half* q_rope_sin, const rfk_half* k_rope_cos,
                       const rfk_half* k_rope_sin, int cache_flags, rfk_stream_t stream);

// A decoder layer whose norms are folded into its products (gemm_folded): eight launches instead of eleven. The token rows are the 4 x 4 blocks of
// the grid in the window order of the layer's own shift; x is read there and, where next is not NULL, written in the order of shift
// next_shift; raster (may be NULL): the result in raster order. The mask's tokens are in row order.
struct FoldedWeights {
    rfk_half *q, *in, *w1, *w3;        // the products' weights with the norms' multiplied in,
    float *mul_q, *mul_in, *mul_w1, *mul_w3;   // divided by these (fold_weights)
};
struct FoldedBuffers {                 // work space of a frame of M rows
    rfk_half *attn, *q, *qkv, *act;    // [M, dim] twice, [3 M, dim] (q may lie in it), [M, ffn_hidden]
    float *x_ss, *qk_ss;               // M * dim / 32 floats, and twice that
    int x_tiles;                       // how many sums a row of x has, in and out
};
int decoder_layer_folded(rfk_ctx* ctx, const rfk_decoder_layer_weights* w, const FoldedWeights& f, FoldedBuffers& b, rfk_half* x, rfk_half* next,
                         rfk_half* raster, const rfk_half* K_rotated, const rfk_half* V_cached, bool v_shared, int B, int Sq, int Sk, int n_keys,
                         int dim, int num_heads, int ffn_hidden, int patch_h, int patch_w, int shift, int next_shift, const uint8_t* mask,
                         rfk_stream_t stream);
// whether it takes a layer of these sizes and weights
bool layer_folds(const rfk_decoder_layer_weights& w, int Sq, int dim, int num_heads, int ffn_hidden, int patch_h, int patch_w, int window_size,
                 int shift_size);
}  // namespace rfk_layers

// rfk_dpt_create, with every 3x3 convolution left to the library if library_only, for the tests that compare the two;
// *own_convolutions (may be NULL) = how many convolutions the tcgen05 kernel took.
extern "C" int rfk_dpt_create_from(rfk_ctx* ctx, const rfk_dpt_weights* w, int B, int dim, int patch_h, int patch_w, int patch_size,
                                   int library_only, int* own_convolutions, rfk_dpt** out);
// how many convolutions of a head the library takes: those of stride 2, all of a head over several views, and those whose order of
// sums the tcgen05 kernel does not have
extern "C" int rfk_dpt_num_library_convolutions(rfk_dpt* d);
