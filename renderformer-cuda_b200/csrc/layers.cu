// Attention / transformer layer boundaries: cuBLAS GEMMs joined by the rfk kernels.
//
// Reference call sequences (BANANASJIM/renderformer-cuda):
//   src/layers/linear.cu:7-25            linear
//   src/layers/transformer.cu:63-79      ffn_swiglu           (2 GEMMs + gate + GEMM)
//   src/layers/attention.cu:112-165      sdpa, cuBLAS path    (GEMM, softmax, GEMM)
//   src/layers/attention.cu:170-231      self_attention
//   src/layers/attention.cu:302-373      precompute_cross_kv, cross_attention_cached
//   src/layers/attention.cu:476-576      swin_self_attention
//   src/layers/transformer.cu:151-224    decoder_layer_forward_cached, encoder_layer_forward_mixed
//
// What is re-cut here (launches per decoder layer: ~36 in the reference, 11 here and 8 where the
// norms are folded into their products (decoder_layer_folded), plus the rotation of the cached
// keys, which the session runs on a parallel graph branch):
//   - residual add + RMSNorm (+ fp16 cast) is one kernel; the FFN residual of a layer is
//     deferred into the first norm of the next layer;
//   - QK-RMSNorm + [B,S,H,D]->[B,H,S,D] + RoPE (+ QKV de-interleave) is one kernel;
//   - the cached K is rotated out of place (no device-to-device copy first);
//   - attention is one fused kernel whenever head_dim is 64 or 128 (rfk_flash_attention: no
//     score matrix, output written [B,Sq,H*D] directly); other head sizes keep GEMM -> softmax
//     (fp16 probabilities over its own fp32 score rows) -> GEMM;
//   - swin attention with 64-token windows and head_dim 64 or 128 is one kernel per layer
//     (rfk_window_attention); cyclic shift + window partition are folded into the norm before
//     it, window reverse + un-shift + residual add into the norm after it
//     (rfk_rmsnorm_residual_f16_windows); other window / head sizes keep the gather ->
//     GEMM -> softmax -> GEMM -> scatter sequence;
//   - w1 and w3 run as one GEMM when stored back to back; the gate overwrites its own input.
#include "kernels_internal.h"
#include "layers_internal.h"

#include <algorithm>
#include <atomic>
#include <cmath>

using namespace rfk_layers;

#define TRY(expr)                       \
    do {                                \
        int rc_ = (expr);               \
        if (rc_ != RFK_OK) return rc_;  \
    } while (0)

static int blas_status(cublasStatus_t s) {
    if (s == CUBLAS_STATUS_SUCCESS) return RFK_OK;
    return 1000 + (int)s;  // distinct from cudaError_t values used by the kernels
}

// C[M,N] (ldc) = alpha * A[M,K] (lda) * B[N,K]^T (ldb), row-major fp16, fp32 accumulation: the tcgen05 kernel of
// librfk.so (rfk_gemm_f16) when it serves the shape, the library GEMM otherwise
static int gemm_nt(rfk_ctx* ctx, cudaStream_t st, int M, int N, int K, float alpha, const __half* A,
                   int lda, const __half* B, int ldb, __half* C, int ldc) {
    if (M == 0 || N == 0) return RFK_OK;
    if (alpha == 1.0f) {
        const int rc = rfk_gemm_f16((const rfk_half*)A, lda, (const rfk_half*)B, ldb, nullptr, nullptr, nullptr, 0,
                                    (rfk_half*)C, ldc, M, N, K, RFK_GEMM_EPI_NONE, (rfk_stream_t)st);
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    TRY(blas_status(cublasSetStream(ctx->blas, st)));
    const float beta = 0.0f;
    return blas_status(cublasGemmEx(ctx->blas, CUBLAS_OP_T, CUBLAS_OP_N, N, M, K, &alpha, B,
                                    CUDA_R_16F, ldb, A, CUDA_R_16F, lda, &beta, C, CUDA_R_16F, ldc,
                                    CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT));
}

extern "C" int rfk_ctx_create(rfk_ctx** out) {
    if (!out) return RFK_EINVAL;
    rfk_ctx* c = new rfk_ctx();
    cudaError_t e = cudaGetDevice(&c->device);
    if (e != cudaSuccess) { delete c; return (int)e; }
    cublasStatus_t s = cublasCreate(&c->blas);
    if (s != CUBLAS_STATUS_SUCCESS) { delete c; return blas_status(s); }
    c->ws_bytes = 64ull << 20;
    e = cudaMalloc(&c->ws, c->ws_bytes);
    if (e != cudaSuccess) { cublasDestroy(c->blas); delete c; return (int)e; }
    // an explicit workspace keeps cuBLAS from allocating while a graph is being captured
    s = cublasSetWorkspace(c->blas, c->ws, c->ws_bytes);
    if (s != CUBLAS_STATUS_SUCCESS) { cudaFree(c->ws); cublasDestroy(c->blas); delete c; return blas_status(s); }
    *out = c;
    return RFK_OK;
}

extern "C" int rfk_ctx_destroy(rfk_ctx* ctx) {
    if (!ctx) return RFK_OK;
    cublasDestroy(ctx->blas);
    cudaFree(ctx->ws);
    cudaFree(ctx->attn_ws);
    delete ctx;
    return RFK_OK;
}

extern "C" int rfk_ctx_reserve_attention_workspace(rfk_ctx* ctx) {
    if (!ctx) return RFK_EINVAL;
    if (ctx->attn_ws) return RFK_OK;
    const size_t bytes = rfk_flash_attention_workspace_bytes();
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e != cudaSuccess) return (int)e;
    e = cudaMemset(p, 0, 1024);  // the unit counters; the kernel returns them to zero after every launch
    if (e != cudaSuccess) { cudaFree(p); return (int)e; }
    ctx->attn_ws = p;
    ctx->attn_ws_bytes = bytes;
    return RFK_OK;
}

extern "C" int rfk_linear(rfk_ctx* ctx, const rfk_half* X, const rfk_half* W, const rfk_half* bias,
                          rfk_half* Y, int M, int N, int K, rfk_stream_t stream) {
    if (!ctx || !X || !W || !Y || M < 0 || N <= 0 || K <= 0) return RFK_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    if (bias && M > 0) {  // bias added in the GEMM's epilogue when the tcgen05 kernel serves the shape
        const int rc = rfk_gemm_f16(X, K, W, K, nullptr, bias, nullptr, 0, Y, N, M, N, K, RFK_GEMM_EPI_NONE, stream);
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    TRY(gemm_nt(ctx, st, M, N, K, 1.0f, (const __half*)X, K, (const __half*)W, K, (__half*)Y, N));
    if (bias) TRY(rfk_broadcast_add(Y, bias, (long long)M * N, N, stream));
    return RFK_OK;
}

// C = A B^T + R (R [M,N] fp16 with pitch ldr, may be C itself): the residual add rides in the epilogue of the
// tcgen05 GEMM; on the library route R is first copied into C (unless it is C) and the GEMM accumulates onto it
// (beta = 1), which rounds once as well.
static int gemm_nt_residual(rfk_ctx* ctx, cudaStream_t st, int M, int N, int K, const __half* A, int lda, const __half* B,
                            int ldb, __half* C, int ldc, const __half* R, int ldr) {
    if (M == 0 || N == 0) return RFK_OK;
    const int rc = rfk_gemm_f16((const rfk_half*)A, lda, (const rfk_half*)B, ldb, nullptr, nullptr, (const rfk_half*)R, ldr,
                                (rfk_half*)C, ldc, M, N, K, RFK_GEMM_EPI_RESIDUAL, (rfk_stream_t)st);
    if (rc != RFK_EUNSUPPORTED) return rc;
    if (R != C) {
        cudaError_t e = cudaMemcpy2DAsync(C, (size_t)ldc * 2, R, (size_t)ldr * 2, (size_t)N * 2, (size_t)M,
                                          cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return (int)e;
    }
    TRY(blas_status(cublasSetStream(ctx->blas, st)));
    const float one = 1.0f;
    return blas_status(cublasGemmEx(ctx->blas, CUBLAS_OP_T, CUBLAS_OP_N, N, M, K, &one, B, CUDA_R_16F, ldb, A, CUDA_R_16F,
                                    lda, &one, C, CUDA_R_16F, ldc, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT));
}

// out = (residual +) W2 (silu(W1 x) * (W3 x)). With the tcgen05 GEMM the gate and up projections and the
// activation are one kernel that writes [M, hidden] directly (no gate|up intermediate); otherwise one or two
// library GEMMs into a [M, 2*hidden] gate|up buffer and the gate kernel. The residual add (if asked; `residual`
// may be `out`) is part of the W2 product either way.
static int ffn_core(rfk_ctx* ctx, const rfk_ffn_weights* w, const rfk_half* x, rfk_half* out, const rfk_half* residual,
                    rfk_half* buf, int M, int dim, int hidden, rfk_stream_t stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (M == 0) return RFK_OK;
    const __half* act = (const __half*)buf;
    int act_ld = hidden;
    const int rc = rfk_gemm_f16(x, dim, w->w1, dim, w->w3, nullptr, nullptr, 0, buf, hidden, M, hidden, dim,
                                RFK_GEMM_EPI_SWIGLU, stream);
    if (rc == RFK_EUNSUPPORTED) {
        __half* gu = (__half*)buf;  // [M, 2*hidden]: gate | up per row
        if (w->w3 == w->w1 + (size_t)hidden * dim) {
            TRY(gemm_nt(ctx, st, M, 2 * hidden, dim, 1.0f, (const __half*)x, dim, (const __half*)w->w1, dim, gu, 2 * hidden));
        } else {
            TRY(gemm_nt(ctx, st, M, hidden, dim, 1.0f, (const __half*)x, dim, (const __half*)w->w1, dim, gu, 2 * hidden));
            TRY(gemm_nt(ctx, st, M, hidden, dim, 1.0f, (const __half*)x, dim, (const __half*)w->w3, dim, gu + hidden, 2 * hidden));
        }
        TRY(rfk_swiglu_inplace(buf, M, hidden, stream));  // activation over the gate half, pitch 2*hidden
        act_ld = 2 * hidden;
    } else if (rc != RFK_OK) {
        return rc;
    }
    if (residual)
        return gemm_nt_residual(ctx, st, M, dim, hidden, act, act_ld, (const __half*)w->w2, hidden, (__half*)out, dim,
                                (const __half*)residual, dim);
    return gemm_nt(ctx, st, M, dim, hidden, 1.0f, act, act_ld, (const __half*)w->w2, hidden, (__half*)out, dim);
}

extern "C" int rfk_ffn_swiglu(rfk_ctx* ctx, const rfk_ffn_weights* w, const rfk_half* x,
                              rfk_half* out, rfk_half* buf, int M, int dim, int hidden,
                              rfk_stream_t stream) {
    if (!ctx || !w || !w->w1 || !w->w2 || !w->w3 || !x || !out || !buf) return RFK_EINVAL;
    if (M < 0 || dim <= 0 || hidden <= 0) return RFK_EINVAL;
    return ffn_core(ctx, w, x, out, nullptr, buf, M, dim, hidden, stream);
}

extern "C" int rfk_sdpa(rfk_ctx* ctx, const rfk_half* Q, const rfk_half* K, const rfk_half* V,
                        rfk_half* O, float* workspace, const uint8_t* mask, int B, int H, int Sq,
                        int Sk, int n_keys, int D, int o_bshd, rfk_stream_t stream) {
    if (!ctx || !Q || !K || !V || !O || !workspace) return RFK_EINVAL;
    if (B < 0 || H <= 0 || Sq < 0 || Sk <= 0 || D <= 0 || n_keys <= 0 || n_keys > Sk) return RFK_EINVAL;
    if (mask) return RFK_EUNSUPPORTED;
    if (B == 0 || Sq == 0) return RFK_OK;
    const int ld = (Sk + 7) & ~7;  // score row pitch in floats; P row pitch is 2*ld halves
    if (ld > 8192) return RFK_EUNSUPPORTED;  // the in-place softmax holds a whole row in registers
    cudaStream_t st = (cudaStream_t)stream;
    TRY(blas_status(cublasSetStream(ctx->blas, st)));
    const int BH = B * H;
    const float scale = 1.0f / sqrtf((float)D), zero = 0.0f, one = 1.0f;
    // scores[bh] (Sq x Sk, pitch ld) = scale * Q[bh] K[bh]^T
    TRY(blas_status(cublasGemmStridedBatchedEx(
        ctx->blas, CUBLAS_OP_T, CUBLAS_OP_N, Sk, Sq, D, &scale, K, CUDA_R_16F, D, (long long)Sk * D,
        Q, CUDA_R_16F, D, (long long)Sq * D, &zero, workspace, CUDA_R_32F, ld, (long long)Sq * ld, BH,
        CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT)));
    TRY(rfk_softmax_probs_inplace(workspace, BH * Sq, n_keys, ld, 1.0f, stream));
    const __half* P = reinterpret_cast<const __half*>(workspace);
    // O[bh] (Sq x D) = P[bh] (Sq x Sk, pitch 2*ld) V[bh] (Sk x D); only the n_keys live columns
    // of P are multiplied (the rest are zero), rounded up to the GEMM's preferred multiple of 8
    const int kk = std::min(Sk, (n_keys + 7) & ~7);
    if (!o_bshd) {
        return blas_status(cublasGemmStridedBatchedEx(
            ctx->blas, CUBLAS_OP_N, CUBLAS_OP_N, D, Sq, kk, &one, V, CUDA_R_16F, D, (long long)Sk * D,
            P, CUDA_R_16F, 2 * ld, 2LL * Sq * ld, &zero, O, CUDA_R_16F, D, (long long)Sq * D, BH,
            CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT));
    }
    // [B,Sq,H*D]: head h of batch b starts at b*Sq*H*D + h*D with row pitch H*D
    for (int b = 0; b < B; ++b) {
        TRY(blas_status(cublasGemmStridedBatchedEx(
            ctx->blas, CUBLAS_OP_N, CUBLAS_OP_N, D, Sq, kk, &one,
            (const __half*)V + (size_t)b * H * Sk * D, CUDA_R_16F, D, (long long)Sk * D,
            P + (size_t)b * H * 2 * Sq * ld, CUDA_R_16F, 2 * ld, 2LL * Sq * ld, &zero,
            (__half*)O + (size_t)b * Sq * H * D, CUDA_R_16F, H * D, (long long)D, H,
            CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT)));
    }
    return RFK_OK;
}

// Attention core: the fused kernel (no score matrix) for the head sizes it implements, the
// materialised GEMM -> softmax -> GEMM sequence (score_buf) for any other.
static int attention_core(rfk_ctx* ctx, const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O,
                          float* score_buf, int B, int H, int Sq, int Sk, int n_keys, int D, int o_bshd,
                          rfk_stream_t stream) {
    int rc = RFK_EUNSUPPORTED;
    if (D == 128 && ctx->reproducible) {
        // The bits that these sessions have always had, those of the mma.sync kernel, from the tcgen05 kernel (a layer of a 320 x 320
        // image at 4575 triangles: 148 -> 62 us, the image 3889 -> 2781 us).
        rc = rfk::flash_attention_ex(Q, K, V, O, nullptr, 0, 0, 0.0f, ctx->attn_ws, ctx->attn_ws_bytes, rfk::AttnCut::kNone, 0, B, H,
                                     Sq, Sk, n_keys, D, o_bshd, 1.0f / sqrtf((float)D), stream);
        if (rc == RFK_EUNSUPPORTED)
            rc = rfk::flash_attention_mma(Q, K, V, O, B, H, Sq, Sk, n_keys, D, o_bshd, 1.0f / sqrtf((float)D), stream);
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    if (ctx->attn_ws)  // tcgen05 kernel with the balanced key split; declines what only the other kernels serve
        rc = rfk::flash_attention_ex(Q, K, V, O, nullptr, 0, 0, 0.0f, ctx->attn_ws, ctx->attn_ws_bytes,
                                     ctx->reproducible ? rfk::AttnCut::kBelowOneRound : rfk::AttnCut::kLastRound, 0, B, H, Sq, Sk, n_keys, D, o_bshd, 1.0f / sqrtf((float)D), stream);
    if (rc == RFK_EUNSUPPORTED)
        rc = rfk_flash_attention(Q, K, V, O, B, H, Sq, Sk, n_keys, D, o_bshd, 1.0f / sqrtf((float)D), stream);
    if (rc != RFK_EUNSUPPORTED) return rc;
    if (!score_buf) return RFK_EINVAL;  // the materialised path needs its score matrix
    return rfk_sdpa(ctx, Q, K, V, O, score_buf, nullptr, B, H, Sq, Sk, n_keys, D, o_bshd, stream);
}

// Q/K/V epilogue of a projection: fused kernel when the shape allows, else the unfused steps.
static int project_epilogue(const rfk_half* x, long long row_stride, int n_parts,
                            const float* const* gamma, rfk_half* const* out, const int* use_rope,
                            const rfk_half* cosv, const rfk_half* sinv, int B, int S, int H, int D,
                            int out_seq_stride, rfk_half* tmp, rfk_stream_t stream) {
    int rc = rfk_qkv_norm_rope_transpose(x, row_stride, n_parts, gamma, out, use_rope, cosv, sinv, B,
                                         S, H, D, kEpsFp16, out_seq_stride, stream);
    if (rc != RFK_EUNSUPPORTED) return rc;
    // unfused: needs a contiguous copy of each part in tmp [B*S, H*D]
    if (!tmp || (out_seq_stride && out_seq_stride != S)) return RFK_EUNSUPPORTED;
    const int dim = H * D;
    const long long M = (long long)B * S;
    for (int p = 0; p < n_parts; ++p) {
        cudaError_t e = cudaMemcpy2DAsync(tmp, (size_t)dim * 2, x + (size_t)p * dim, (size_t)row_stride * 2,
                                          (size_t)dim * 2, (size_t)M, cudaMemcpyDeviceToDevice,
                                          (cudaStream_t)stream);
        if (e != cudaSuccess) return (int)e;
        if (gamma[p]) TRY(rfk_rmsnorm(tmp, gamma[p], tmp, (int)M, dim, kEpsFp16, stream));
        TRY(rfk_transpose_bshd_to_bhsd(tmp, out[p], B, S, H, D, stream));
        if (use_rope[p]) TRY(rfk_apply_rope_one(out[p], cosv, sinv, B, H, S, D, stream));
    }
    return RFK_OK;
}

extern "C" int rfk_precompute_cross_kv(rfk_ctx* ctx, const rfk_cross_attn_weights* w,
                                       const rfk_half* ctx_normed, rfk_half* K_out, rfk_half* V_out,
                                       rfk_half* proj_buf, int B, int Sk, int Sk_pad, int kv_dim,
                                       int dim, int num_heads, rfk_stream_t stream) {
    if (!ctx || !w || !ctx_normed || !K_out || !V_out || !proj_buf) return RFK_EINVAL;
    if (B <= 0 || Sk <= 0 || Sk_pad < Sk || dim <= 0 || num_heads <= 0 || dim % num_heads) return RFK_EINVAL;
    const int Mk = B * Sk, hd = dim / num_heads;
    rfk_half* Kp = proj_buf;
    rfk_half* Vp = proj_buf + (size_t)Mk * dim;
    TRY(rfk_linear(ctx, ctx_normed, w->k_proj_w, w->k_proj_b, Kp, Mk, dim, kv_dim, stream));
    if (Sk_pad != Sk) {
        // only the rows behind the last key of each head; every other element is written below
        const size_t pitch = (size_t)Sk_pad * hd * 2, width = (size_t)(Sk_pad - Sk) * hd * 2, heads = (size_t)B * num_heads;
        cudaError_t e = cudaMemset2DAsync(K_out + (size_t)Sk * hd, pitch, 0, width, heads, (cudaStream_t)stream);
        if (e == cudaSuccess) e = cudaMemset2DAsync(V_out + (size_t)Sk * hd, pitch, 0, width, heads, (cudaStream_t)stream);
        if (e != cudaSuccess) return (int)e;
    }
    const float* g[1] = {w->k_norm_gamma};
    rfk_half* o[1] = {K_out};
    const int no_rope[1] = {0};
    // K and V cannot share a launch: they live in two separate [Mk, dim] projections. (K head-split by its projection and normalised in place, as
    // the encoder's q and k are, was no faster for large scenes and slower for most: us, transposing norm / in place, 16 heads of 64: 33 rows 5.5 / 5.8, 600 rows
    // 7.4 / 6.9, 1100 rows 8.2 / 9.5, 3300 rows 14.0 / 14.9, 5665 rows 19.0 / 19.0; the head-split store costs its product what the norm gains.)
    TRY(project_epilogue(Kp, dim, 1, g, o, no_rope, nullptr, nullptr, B, Sk, num_heads, hd, Sk_pad,
                         nullptr, stream));
    // V has no norm: its projection is stored head-split by the GEMM when the shape allows (one batch element, no bias); a
    // transposing pass less per layer (scene of 300 triangles 983 -> 965 us, of 1500 triangles 1650 -> 1628 us)
    int rc = RFK_EUNSUPPORTED;
    if (B == 1 && !w->v_proj_b && (hd == 64 || hd == 128))
        rc = rfk::gemm_heads(ctx_normed, kv_dim, w->v_proj_w, kv_dim, V_out, 0, nullptr, 0, Mk, dim, kv_dim, Sk, Sk_pad, num_heads, hd,
                             stream);
    if (rc != RFK_EUNSUPPORTED) return rc;
    TRY(rfk_linear(ctx, ctx_normed, w->v_proj_w, w->v_proj_b, Vp, Mk, dim, kv_dim, stream));
    g[0] = nullptr; o[0] = V_out;
    return project_epilogue(Vp, dim, 1, g, o, no_rope, nullptr, nullptr, B, Sk, num_heads, hd, Sk_pad,
                            nullptr, stream);
}

// `residual` (may be `out`, may be NULL): out = residual + attention output, the add being the epilogue of the
// output projection.
// norm_ss (may be NULL): scratch of B*Sq*(dim/256) floats for the row statistics of the deferred Q-RMSNorm;
// cache_flags bit 1: V_cached is [H, Sk, hd], shared by all B batch elements (views of one scene rendered together).
// cache_flags bit 0 (k_prescaled): K_cached is already rotated AND multiplied by the query's norm weight (the session does both for all
// layers at once).
static int cross_attention_impl(rfk_ctx* ctx, const rfk_cross_attn_weights* w,
                                          const rfk_half* q_in, rfk_half* out, const rfk_half* residual,
                                          rfk_half* proj_buf, float* norm_ss, int cache_flags,
                                          float* score_buf, const rfk_half* K_cached,
                                          const rfk_half* V_cached, int B, int Sq, int Sk, int n_keys,
                                          int q_dim, int dim, int num_heads,
                                          const rfk_half* q_rope_cos, const rfk_half* q_rope_sin,
                                          const rfk_half* k_rope_cos, const rfk_half* k_rope_sin,
                                          rfk_stream_t stream) {
    if (!ctx || !w || !q_in || !out || !proj_buf || !K_cached || !V_cached) return RFK_EINVAL;
    if (B <= 0 || Sq <= 0 || Sk <= 0 || dim <= 0 || num_heads <= 0 || dim % num_heads) return RFK_EINVAL;
    const int Mq = B * Sq, hd = dim / num_heads;
    rfk_half* Q = proj_buf;                          // [Mq, dim] projection, later the attention output
    rfk_half* Q_bhsd = proj_buf + (size_t)Mq * dim;  // [B,H,Sq,hd]
    rfk_half* K_rot = Q_bhsd + (size_t)Mq * dim;     // [B,H,Sk,hd]
    // Deferred Q-RMSNorm: the projection writes Q head-split and the rows' sums of squares, the attention kernel scales
    // each row's scores by 1 / rms, and the norm's weight rides on the keys (multiplied in by the rotation kernel, here
    // or by the caller). One kernel (norm + head split) and 18 MB of traffic less per layer. Needs: no query rotation
    // (the view decoder's query tables are the identity), keys that are rotated here or arrive prescaled, head size 64
    // or 128.
    const int k_prescaled = cache_flags & 1, v_shared = (cache_flags >> 1) & 1;
    const bool deferred = norm_ss && w->q_norm_gamma && !w->q_proj_b && !q_rope_cos &&
                          (hd == 64 || (hd == 128 && !ctx->reproducible)) && (k_prescaled || k_rope_cos) &&
                          (reinterpret_cast<uintptr_t>(w->q_norm_gamma) & 15u) == 0;
    if (k_prescaled && !deferred) return RFK_EUNSUPPORTED;  // prescaled keys only make sense with the deferred norm
    if (deferred) {
        int rc = RFK_EUNSUPPORTED;
        if (Sq % 32 == 0)
            rc = rfk::gemm_heads(q_in, q_dim, w->q_proj_w, q_dim, Q_bhsd, 0, norm_ss, 1, Mq, dim, q_dim, Sq, Sq, num_heads, hd, stream);
        if (rc == RFK_OK) {
            const rfk_half* K_use = K_cached;
            if (!k_prescaled) {
                rc = rfk_rope_one_oop_strided(K_cached, K_rot, k_rope_cos, k_rope_sin, B, (long long)num_heads * Sk * hd,
                                              (long long)num_heads * Sk * hd, (long long)Sk * hd, num_heads, Sk, hd, Sk, Sk,
                                              w->q_norm_gamma, 0, stream);
                K_use = K_rot;
            }
            // With 64-wide heads a view is rendered alone or in a frame of several and must have the same bits: a view alone
            // that fills the SMs (208 units at 448 x 448) is not cut along the keys, as it is not among the units of a frame; its units
            // are handed over, which keeps their bits (184 units of 33 tiles 60 -> 44 us). 128-wide heads have no such frames.
            if (rc == RFK_OK)
                rc = rfk::flash_attention_ex(Q_bhsd, K_use, V_cached, Q, norm_ss, dim / 256, dim, kEpsFp16, ctx->attn_ws,
                                             ctx->attn_ws_bytes, hd == 64 ? rfk::AttnCut::kBelowOneRound : rfk::AttnCut::kLastRound,
                                             v_shared, B, num_heads, Sq, Sk, n_keys, hd, 1, 1.0f / sqrtf((float)hd), stream);
        }
        if (rc != RFK_OK && rc != RFK_EUNSUPPORTED) return rc;
        if (rc == RFK_EUNSUPPORTED && (k_prescaled || (v_shared && B > 1))) return rc;  // only the fused route serves these
        if (rc == RFK_OK) goto out_projection;
    }
    if (v_shared && B > 1) return RFK_EUNSUPPORTED;  // the separate-norm route below reads V per batch element
    {
        TRY(rfk_linear(ctx, q_in, w->q_proj_w, w->q_proj_b, Q, Mq, dim, q_dim, stream));
        const float* g[1] = {w->q_norm_gamma};
        rfk_half* o[1] = {Q_bhsd};
        const int rope[1] = {q_rope_cos != nullptr};
        TRY(project_epilogue(Q, dim, 1, g, o, rope, q_rope_cos, q_rope_sin, B, Sq, num_heads, hd, 0, K_rot, stream));
        const rfk_half* K_use = K_cached;
        if (k_rope_cos) {
            TRY(rfk_rope_one_oop(K_cached, K_rot, k_rope_cos, k_rope_sin, B, num_heads, Sk, hd, Sk, Sk, 0, stream));
            K_use = K_rot;
        }
        TRY(attention_core(ctx, Q_bhsd, K_use, V_cached, Q /* [B,Sq,dim] */, score_buf, B, num_heads, Sq, Sk, n_keys,
                           hd, 1, stream));
    }
out_projection:
    if (residual && !w->out_proj_b)
        return gemm_nt_residual(ctx, (cudaStream_t)stream, Mq, q_dim, dim, (const __half*)Q, dim, (const __half*)w->out_proj_w,
                                dim, (__half*)out, q_dim, (const __half*)residual, q_dim);
    if (residual) return RFK_EUNSUPPORTED;  // callers with a bias keep the separate residual add
    return rfk_linear(ctx, Q, w->out_proj_w, w->out_proj_b, out, Mq, q_dim, dim, stream);
}

extern "C" int rfk_cross_attention_cached(rfk_ctx* ctx, const rfk_cross_attn_weights* w,
                                          const rfk_half* q_in, rfk_half* out, rfk_half* proj_buf,
                                          float* score_buf, const rfk_half* K_cached,
                                          const rfk_half* V_cached, int B, int Sq, int Sk, int n_keys,
                                          int q_dim, int dim, int num_heads,
                                          const rfk_half* q_rope_cos, const rfk_half* q_rope_sin,
                                          const rfk_half* k_rope_cos, const rfk_half* k_rope_sin,
                                          rfk_stream_t stream) {
    return cross_attention_impl(ctx, w, q_in, out, nullptr, proj_buf, nullptr, 0, score_buf, K_cached, V_cached, B, Sq, Sk,
                                n_keys, q_dim, dim, num_heads, q_rope_cos, q_rope_sin, k_rope_cos, k_rope_sin, stream);
}

// Window attention over tokens that are already in window order: window_buf [BnW * ws2, dim] in,
// qkv_buf [BnW * ws2, dim] out (still in window order); window_buf and scratch are overwritten.
// norm_ss (may be NULL): scratch of 2 * M * (dim / 256) floats for the row statistics of the deferred QK-RMSNorm.
static int swin_core(rfk_ctx* ctx, const rfk_mha_weights* w, rfk_half* window_buf, rfk_half* qkv_buf,
                     float* score_buf, rfk_half* scratch, int BnW, int nW, int ws2, int dim, int num_heads,
                     const uint8_t* win_mask, rfk_stream_t stream, float* norm_ss = nullptr) {
    cudaStream_t st = (cudaStream_t)stream;
    const int hd = dim / num_heads, M = BnW * ws2, BH = BnW * num_heads;
    rfk_half* Qt = scratch;
    rfk_half* Kt = scratch + (size_t)M * dim;
    rfk_half* Vt = scratch + (size_t)2 * M * dim;
    // Deferred QK-RMSNorm: the packed projection writes q, k, v head-split per window and the sums of squares of the q and
    // k rows; the window attention kernel normalises the two tiles while it stages them (same formula and rounding as
    // the separate kernel). One kernel and 50 MB of traffic less per layer.
    const bool fused = ws2 == 64 && (hd == 64 || (hd == 128 && !ctx->reproducible));  // the window attention kernel, in forms with sums of its own
    if (hd != 64 && !score_buf) return RFK_EINVAL;            // score space is only optional for 64-wide heads
    if (norm_ss && fused && w->q_norm_gamma && w->k_norm_gamma && !w->in_proj_b) {
        const int tiles = dim / 256;
        int rc = rfk::gemm_heads(window_buf, dim, w->in_proj_w, dim, Qt, (long long)M * dim, norm_ss, 3, M, 3 * dim, dim, ws2,
                                 ws2, num_heads, hd, stream);
        if (rc == RFK_OK)
            rc = rfk::window_attention(Qt, Kt, Vt, window_buf, win_mask, norm_ss, norm_ss + (size_t)M * tiles, tiles,
                                       w->q_norm_gamma, w->k_norm_gamma, dim, kEpsFp16, BnW, num_heads, ws2, hd, nW,
                                       1.0f / sqrtf((float)hd), stream);
        if (rc == RFK_OK) return rfk_linear(ctx, window_buf, w->out_proj_w, w->out_proj_b, qkv_buf, M, dim, dim, stream);
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    TRY(rfk_linear(ctx, window_buf, w->in_proj_w, w->in_proj_b, qkv_buf, M, 3 * dim, dim, stream));
    const float* g[3] = {w->q_norm_gamma, w->k_norm_gamma, nullptr};
    rfk_half* o[3] = {Qt, Kt, Vt};
    const int no_rope[3] = {0, 0, 0};
    TRY(project_epilogue(qkv_buf, 3LL * dim, 3, g, o, no_rope, nullptr, nullptr, BnW, ws2, num_heads, hd, 0,
                         window_buf, stream));
    const float scale = 1.0f / sqrtf((float)hd), zero = 0.0f, one = 1.0f;
    if (fused) {  // the whole window attention in one kernel, output already token-major
        const int rc = rfk::window_attention(Qt, Kt, Vt, window_buf, win_mask, nullptr, nullptr, 0, nullptr, nullptr, 0, 0.0f,
                                             BnW, num_heads, ws2, hd, nW, scale, stream);
        if (rc == RFK_OK) return rfk_linear(ctx, window_buf, w->out_proj_w, w->out_proj_b, qkv_buf, M, dim, dim, stream);
        if (rc != RFK_EUNSUPPORTED || hd == 64) return rc;   // the separate steps below serve 128-wide heads without it
    }
    if (ws2 == 64 && hd == 128 && ctx->reproducible) {
        // one kernel with the bits of the four steps below (the 320 x 320 image at 4575 triangles 2781 -> 2653 us)
        const int rc = rfk::window_attention_steps(Qt, Kt, Vt, window_buf, win_mask, BnW, num_heads, ws2, hd, nW, scale, stream);
        if (rc == RFK_OK) return rfk_linear(ctx, window_buf, w->out_proj_w, w->out_proj_b, qkv_buf, M, dim, dim, stream);
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    if (!score_buf) return RFK_EINVAL;
    TRY(blas_status(cublasSetStream(ctx->blas, st)));
    const long long sQ = (long long)ws2 * hd, sS = (long long)ws2 * ws2;
    TRY(blas_status(cublasGemmStridedBatchedEx(ctx->blas, CUBLAS_OP_T, CUBLAS_OP_N, ws2, ws2, hd, &scale, Kt,
                                               CUDA_R_16F, hd, sQ, Qt, CUDA_R_16F, hd, sQ, &zero, score_buf,
                                               CUDA_R_32F, ws2, sS, BH, CUBLAS_COMPUTE_32F,
                                               CUBLAS_GEMM_DEFAULT)));
    TRY(rfk_swin_softmax_probs_inplace(score_buf, win_mask, BnW, num_heads, ws2, nW, stream));
    // O (over Q) = P V ; P pitch is 2*ws2 halves inside the score rows
    TRY(blas_status(cublasGemmStridedBatchedEx(
        ctx->blas, CUBLAS_OP_N, CUBLAS_OP_N, hd, ws2, ws2, &one, Vt, CUDA_R_16F, hd, sQ,
        reinterpret_cast<const __half*>(score_buf), CUDA_R_16F, 2 * ws2, 2 * sS, &zero, Qt, CUDA_R_16F, hd,
        sQ, BH, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT)));
    TRY(rfk_transpose_bhsd_to_bsd(Qt, window_buf, BnW, num_heads, ws2, hd, stream));
    return rfk_linear(ctx, window_buf, w->out_proj_w, w->out_proj_b, qkv_buf, M, dim, dim, stream);
}

extern "C" int rfk_swin_self_attention(rfk_ctx* ctx, const rfk_mha_weights* w, const rfk_half* x,
                                       rfk_half* out, rfk_half* residual_x, rfk_half* window_buf,
                                       rfk_half* qkv_buf, float* score_buf, rfk_half* scratch, int B,
                                       int H, int W, int dim, int num_heads, int window_size,
                                       int shift_size, const uint8_t* shift_mask, rfk_stream_t stream) {
    if (!ctx || !w || !x || (!out && !residual_x) || !window_buf || !qkv_buf || !scratch)
        return RFK_EINVAL;
    if (B <= 0 || H <= 0 || W <= 0 || window_size <= 0 || H % window_size || W % window_size) return RFK_EINVAL;
    if (dim <= 0 || num_heads <= 0 || dim % num_heads) return RFK_EINVAL;
    const int ws = window_size, ws2 = ws * ws, nW = (H / ws) * (W / ws);
    TRY(rfk_window_gather(x, window_buf, B, H, W, dim, ws, shift_size, stream));
    TRY(swin_core(ctx, w, window_buf, qkv_buf, score_buf, scratch, B * nW, nW, ws2, dim, num_heads,
                  (shift_mask && shift_size > 0) ? shift_mask : nullptr, stream));
    if (residual_x) return rfk_window_scatter(qkv_buf, residual_x, B, H, W, dim, ws, shift_size, 1, stream);
    return rfk_window_scatter(qkv_buf, out, B, H, W, dim, ws, shift_size, 0, stream);
}

extern "C" int rfk_self_attention(rfk_ctx* ctx, const rfk_mha_weights* w, const rfk_half* x,
                                  rfk_half* out, rfk_half* qkv_buf, float* score_buf, int B, int S,
                                  int dim, int num_heads, const rfk_half* rope_cos,
                                  const rfk_half* rope_sin, rfk_stream_t stream) {
    if (!ctx || !w || !x || !out || !qkv_buf) return RFK_EINVAL;
    if (B <= 0 || S <= 0 || dim <= 0 || num_heads <= 0 || dim % num_heads) return RFK_EINVAL;
    const int M = B * S, hd = dim / num_heads;
    rfk_half* Qb = qkv_buf + (size_t)M * 3 * dim;
    rfk_half* Kb = Qb + (size_t)M * dim;
    rfk_half* Vb = Kb + (size_t)M * dim;
    const float* g[3] = {w->q_norm_gamma, w->k_norm_gamma, nullptr};
    rfk_half* o[3] = {Qb, Kb, Vb};
    // One batch element: the projection stores q, k and v head-split, and only q and k go through the norm and the rotation, in
    // place (v passed through that kernel only to be transposed: a third of its 70 MB at 5665 rows,
    // a scene of 5633 triangles 5900 -> 5820 us).
    int rc = RFK_EUNSUPPORTED;
    if (B == 1 && !w->in_proj_b && (hd == 64 || hd == 128) && dim <= 2048 &&
        ((reinterpret_cast<uintptr_t>(w->q_norm_gamma) | reinterpret_cast<uintptr_t>(w->k_norm_gamma) |
          reinterpret_cast<uintptr_t>(rope_cos) | reinterpret_cast<uintptr_t>(rope_sin)) & 15u) == 0)
        rc = rfk::gemm_heads(x, dim, w->in_proj_w, dim, Qb, (long long)M * dim, nullptr, 0, M, 3 * dim, dim, S, S, num_heads, hd, stream);
    if (rc == RFK_OK) {
        TRY(rfk::qk_norm_rope_heads(2, g, o, rope_cos, rope_sin, S, S, num_heads, hd, kEpsFp16, stream));
    } else if (rc == RFK_EUNSUPPORTED) {
        TRY(rfk_linear(ctx, x, w->in_proj_w, w->in_proj_b, qkv_buf, M, 3 * dim, dim, stream));
        const int rope[3] = {rope_cos != nullptr, rope_cos != nullptr, 0};
        TRY(project_epilogue(qkv_buf, 3LL * dim, 3, g, o, rope, rope_cos, rope_sin, B, S, num_heads, hd, 0, nullptr, stream));
    } else {
        return rc;
    }
    // attention output lands in the (dead) front of qkv_buf as [B,S,dim]
    TRY(attention_core(ctx, Qb, Kb, Vb, qkv_buf, score_buf, B, num_heads, S, S, S, hd, 1, stream));
    return rfk_linear(ctx, qkv_buf, w->out_proj_w, w->out_proj_b, out, M, dim, dim, stream);
}

// cache_flags: bit 1: V_cached is shared by the B batch elements; bit 0: K_cached is this view's rotated keys already multiplied by the cross-attention query norm's weight
// (what rfk_session prepares for all layers at once); 0 for keys as the public entry point receives them.
// x_in: what the layer reads, x or another buffer, which stays as it is; x_out: where its result goes, x or another buffer.
int rfk_layers::decoder_layer_impl(
    rfk_ctx* ctx, const rfk_decoder_layer_weights* w, const rfk_half* x_in, rfk_half* x, rfk_half* x_out, const rfk_half* pending_residual,
    const rfk_half** pending_out, rfk_half* temp, rfk_half* proj_buf, rfk_half* qkv_buf, rfk_half* ffn_buf,
    rfk_half* window_buf, float* cross_score_buf, float* self_score_buf, const rfk_half* K_cached,
    const rfk_half* V_cached, int B, int Sq, int Sk, int n_keys, int dim, int num_heads, int ffn_hidden,
    int patch_h, int patch_w, int window_size, int shift_size, const uint8_t* shift_mask,
    const rfk_half* q_rope_cos, const rfk_half* q_rope_sin, const rfk_half* k_rope_cos,
    const rfk_half* k_rope_sin, int cache_flags, rfk_stream_t stream) {
    if (!ctx || !w || !x_in || !x || !x_out || !temp || !proj_buf || !qkv_buf || !ffn_buf || !window_buf) return RFK_EINVAL;
    if (Sq != patch_h * patch_w) return RFK_EINVAL;
    const int Mq = B * Sq;
    // 2) residual + pre-norm -> swin attention -> residual + pre-norm of the FFN. When the fused norm can take an
    //    operand in window order, the cyclic shift / window partition and their inverse cost no launch: the first norm
    //    writes the windows, the second reads the attention output out of them; and the residual add of the
    //    cross-attention is the epilogue of its output projection (x += ...), so the first norm reads x only.
    auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const bool win_ok = window_size > 0 && patch_h % window_size == 0 && patch_w % window_size == 0 &&
                        num_heads > 0 && dim % num_heads == 0 && dim % 8 == 0 && dim <= 2048 && a16(x_in) && a16(x) && a16(x_out) && a16(window_buf) &&
                        a16(temp) && a16(qkv_buf) && a16(w->self_attn_norm_gamma) && a16(w->ffn_norm_gamma);
    if (x_in != x && (!win_ok || w->cross_attn.out_proj_b || pending_residual)) {   // the steps below that add onto x itself
        cudaError_t e = cudaMemcpyAsync(x, x_in, (size_t)Mq * dim * sizeof(rfk_half), cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
        if (e != cudaSuccess) return (int)e;
        x_in = x;
    }
    // 1) (deferred residual of the previous layer, if any +) pre-norm -> cached cross-attention
    if (pending_residual) TRY(rfk_rmsnorm_residual_f16(x, pending_residual, w->query_norm_gamma, temp, Mq, dim, kEpsFp16, stream));
    else TRY(rfk_rmsnorm(x_in, w->query_norm_gamma, temp, Mq, dim, kEpsFp16, stream));
    // Row statistics of the deferred QK-norms live in buffers that are idle while they are needed: window_buf during the
    // cross-attention, temp during the window attention (each holds Mq*dim halves; the statistics need Mq*dim/128 floats).
    float* cross_ss = dim % 256 == 0 ? reinterpret_cast<float*>(window_buf) : nullptr;
    float* swin_ss = dim % 256 == 0 ? reinterpret_cast<float*>(temp) : nullptr;
    if (win_ok) {
        if (!w->cross_attn.out_proj_b) {
            TRY(cross_attention_impl(ctx, &w->cross_attn, temp, x, x_in, proj_buf, cross_ss, cache_flags, cross_score_buf, K_cached,
                                     V_cached, B, Sq, Sk, n_keys, dim, dim, num_heads, q_rope_cos, q_rope_sin, k_rope_cos,
                                     k_rope_sin, stream));
            TRY(rfk_rmsnorm_residual_f16_windows(x, nullptr, w->self_attn_norm_gamma, window_buf, B, patch_h, patch_w, dim,
                                                 window_size, shift_size, 1, kEpsFp16, stream));
        } else {
            rfk_half* cross_out = qkv_buf;
            TRY(rfk_cross_attention_cached(ctx, &w->cross_attn, temp, cross_out, proj_buf, cross_score_buf, K_cached, V_cached,
                                           B, Sq, Sk, n_keys, dim, dim, num_heads, q_rope_cos, q_rope_sin, k_rope_cos,
                                           k_rope_sin, stream));
            TRY(rfk_rmsnorm_residual_f16_windows_in_l2(x, cross_out, w->self_attn_norm_gamma, window_buf, B, patch_h, patch_w, dim,
                                                       window_size, shift_size, 1, kEpsFp16, stream));
        }
        const int ws2 = window_size * window_size, nW = (patch_h / window_size) * (patch_w / window_size);
        TRY(swin_core(ctx, &w->self_attn, window_buf, qkv_buf, self_score_buf, proj_buf, B * nW, nW, ws2, dim, num_heads,
                      (shift_mask && shift_size > 0) ? shift_mask : nullptr, stream, swin_ss));
        TRY(rfk_rmsnorm_residual_f16_windows_in_l2(x, qkv_buf, w->ffn_norm_gamma, temp, B, patch_h, patch_w, dim, window_size,
                                                   shift_size, 2, kEpsFp16, stream));
    } else {
        rfk_half* cross_out = qkv_buf;
        TRY(rfk_cross_attention_cached(ctx, &w->cross_attn, temp, cross_out, proj_buf, cross_score_buf, K_cached, V_cached, B,
                                       Sq, Sk, n_keys, dim, dim, num_heads, q_rope_cos, q_rope_sin, k_rope_cos, k_rope_sin,
                                       stream));
        TRY(rfk_rmsnorm_residual_f16(x, cross_out, w->self_attn_norm_gamma, temp, Mq, dim, kEpsFp16, stream));
        TRY(rfk_swin_self_attention(ctx, &w->self_attn, temp, nullptr, x, window_buf, qkv_buf, self_score_buf,
                                    proj_buf, B, patch_h, patch_w, dim, num_heads, window_size, shift_size,
                                    shift_mask, stream));
        TRY(rfk_rmsnorm(x, w->ffn_norm_gamma, temp, Mq, dim, kEpsFp16, stream));
    }
    // 3) FFN with its residual add in the epilogue of the W2 product: x is complete when the layer returns and
    //    nothing is left pending for the next layer
    if (!w->ffn.w1 || !w->ffn.w2 || !w->ffn.w3 || ffn_hidden <= 0) return RFK_EINVAL;
    TRY(ffn_core(ctx, &w->ffn, temp, x_out, x, qkv_buf, Mq, dim, ffn_hidden, stream));
    if (pending_out) *pending_out = nullptr;
    return RFK_OK;
}

// 1024 columns: what embed_tokens, fold_weights and the grouped sums of the attention are written for, and the models have; gemm_folded itself takes any multiple
// of 256. Other widths keep their separate norms, and the bits of the public layer calls; what folding them would gain is not measured.
bool rfk_layers::layer_folds(const rfk_decoder_layer_weights& w, int Sq, int dim, int num_heads, int ffn_hidden, int patch_h, int patch_w,
                             int window_size, int shift_size) {
    const auto given = [](const void* p) { return p && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    return dim == 1024 && num_heads > 0 && (dim == num_heads * 64 || dim == num_heads * 128) && ffn_hidden > 0 && ffn_hidden % 256 == 0 &&
           window_size == 8 && (shift_size == 0 || shift_size == 4) && patch_h > 0 && patch_w > 0 && patch_h % 8 == 0 && patch_w % 8 == 0 &&
           Sq == patch_h * patch_w && given(w.query_norm_gamma) && given(w.self_attn_norm_gamma) && given(w.ffn_norm_gamma) &&
           given(w.cross_attn.q_proj_w) && given(w.cross_attn.out_proj_w) && given(w.cross_attn.q_norm_gamma) && !w.cross_attn.q_proj_b &&
           !w.cross_attn.out_proj_b && given(w.self_attn.in_proj_w) && given(w.self_attn.out_proj_w) && given(w.self_attn.q_norm_gamma) &&
           given(w.self_attn.k_norm_gamma) && !w.self_attn.in_proj_b && !w.self_attn.out_proj_b && given(w.ffn.w1) && given(w.ffn.w2) && given(w.ffn.w3);
}

int rfk_layers::decoder_layer_folded(rfk_ctx* ctx, const rfk_decoder_layer_weights* w, const FoldedWeights& f, FoldedBuffers& b, rfk_half* x,
                                     rfk_half* next, rfk_half* raster, const rfk_half* K_rotated, const rfk_half* V_cached, bool v_shared, int B,
                                     int Sq, int Sk, int n_keys, int dim, int num_heads, int ffn_hidden, int patch_h, int patch_w, int shift,
                                     int next_shift, const uint8_t* mask, rfk_stream_t stream) {
    const int M = B * Sq, hd = dim / num_heads;
    const auto group = [dim](int tiles) { return tiles == dim / 256 ? 1 : 8; };
    rfk::FoldedProduct p{};
    p.M = M;
    p.eps = kEpsFp16;
    const auto normed = [&](const rfk_half* W, rfk_half* C, int N) {              // a product behind a norm
        rfk::FoldedProduct g = p;
        g.A = x; g.W = W; g.C = C; g.N = N; g.K = dim; g.in_ss = b.x_ss; g.in_tiles = b.x_tiles; g.in_mul = 1.0f;
        return g;
    };
    const auto onto_x = [&](const rfk_half* A, const rfk_half* W, int K) {        // x += A W^T
        rfk::FoldedProduct g = p;
        g.A = A; g.W = W; g.R = x; g.C = x; g.N = dim; g.K = K; g.out_ss = b.x_ss;
        return g;
    };
    int tiles = 0;
    // cross-attention (its query norm stays deferred: attention applies 1 / rms, the rotated keys carry the weight; the cut along the keys: see cross_attention_impl)
    rfk::FoldedProduct g = normed(f.q, b.q, dim);
    g.num_heads = num_heads; g.head_dim = hd; g.seq = Sq; g.out_ss = b.qk_ss; g.ss_mask = 1;
    TRY(rfk::gemm_folded(g, &tiles, stream, {0, f.mul_q}));
    TRY(rfk::flash_attention_ex(b.q, K_rotated, V_cached, b.attn, b.qk_ss, tiles, dim, kEpsFp16, ctx->attn_ws, ctx->attn_ws_bytes,
                                hd == 64 ? rfk::AttnCut::kBelowOneRound : rfk::AttnCut::kLastRound, v_shared, B, num_heads, Sq, Sk, n_keys, hd, 1,
                                1.0f / sqrtf((float)hd), stream, group(tiles)));
    TRY(rfk::gemm_folded(onto_x(b.attn, w->cross_attn.out_proj_w, dim), &b.x_tiles, stream));
    // window attention
    g = normed(f.in, b.qkv, 3 * dim);
    g.num_heads = num_heads; g.head_dim = hd; g.seq = 64; g.part_stride = (long long)M * dim; g.out_ss = b.qk_ss; g.ss_mask = 3;
    TRY(rfk::gemm_folded(g, &tiles, stream, {0, f.mul_in}));
    const size_t part = (size_t)M * dim;
    TRY(rfk::window_attention(b.qkv, b.qkv + part, b.qkv + 2 * part, b.attn, mask, b.qk_ss, b.qk_ss + (size_t)M * tiles, tiles, w->self_attn.q_norm_gamma,
                              w->self_attn.k_norm_gamma, dim, kEpsFp16, M / 64, num_heads, 64, hd, Sq / 64, 1.0f / sqrtf((float)hd), stream,
                              group(tiles), true));
    TRY(rfk::gemm_folded(onto_x(b.attn, w->self_attn.out_proj_w, dim), &b.x_tiles, stream));
    // FFN; its result leaves in the next layer's order
    g = normed(f.w1, b.act, ffn_hidden);
    g.W_up = f.w3;
    TRY(rfk::gemm_folded(g, &tiles, stream, {0, f.mul_w1, f.mul_w3}));
    g = onto_x(b.act, w->ffn.w2, ffn_hidden);
    g.C = next; g.raster = raster; g.out_ss = next ? b.x_ss : nullptr;
    g.blocks_across = patch_w / 4; g.blocks_down = patch_h / 4; g.shift_from = shift / 4; g.shift_to = next_shift / 4;
    g.quarters = Sq <= 256 && ffn_hidden % 512 == 0;   // by the rows of a view, not of the frame: a view has the same bits alone and in any frame
    return rfk::gemm_folded(g, &b.x_tiles, stream);
}

extern "C" int rfk_decoder_layer_forward_cached(
    rfk_ctx* ctx, const rfk_decoder_layer_weights* w, rfk_half* x, const rfk_half* pending_residual,
    const rfk_half** pending_out, rfk_half* temp, rfk_half* proj_buf, rfk_half* qkv_buf, rfk_half* ffn_buf,
    rfk_half* window_buf, float* cross_score_buf, float* self_score_buf, const rfk_half* K_cached,
    const rfk_half* V_cached, int B, int Sq, int Sk, int n_keys, int dim, int num_heads, int ffn_hidden,
    int patch_h, int patch_w, int window_size, int shift_size, const uint8_t* shift_mask,
    const rfk_half* q_rope_cos, const rfk_half* q_rope_sin, const rfk_half* k_rope_cos,
    const rfk_half* k_rope_sin, rfk_stream_t stream) {
    return rfk_layers::decoder_layer_impl(ctx, w, x, x, x, pending_residual, pending_out, temp, proj_buf, qkv_buf, ffn_buf, window_buf,
                                          cross_score_buf, self_score_buf, K_cached, V_cached, B, Sq, Sk, n_keys, dim, num_heads,
                                          ffn_hidden, patch_h, patch_w, window_size, shift_size, shift_mask, q_rope_cos,
                                          q_rope_sin, k_rope_cos, k_rope_sin, 0, stream);
}

extern "C" int rfk_encoder_layer_forward_mixed(
    rfk_ctx* ctx, const rfk_encoder_layer_weights* w, float* x, const rfk_half* pending_residual,
    const rfk_half** pending_out, rfk_half* temp, rfk_half* qkv_buf, rfk_half* ffn_buf, float* score_buf,
    int B, int S, int dim, int num_heads, int ffn_hidden, const rfk_half* rope_cos, const rfk_half* rope_sin,
    rfk_stream_t stream) {
    if (!ctx || !w || !x || !temp || !qkv_buf || !ffn_buf) return RFK_EINVAL;
    const int M = B * S;
    // fp32 hidden (+= fp16 sub-layer output) -> fp32 norm -> fp16, one kernel instead of three
    TRY(rfk_rmsnorm_residual_mixed_cast16(x, pending_residual, w->query_norm_gamma, temp, M, dim, kEpsFp32, stream));
    TRY(rfk_self_attention(ctx, &w->attn, temp, ffn_buf, qkv_buf, score_buf, B, S, dim, num_heads, rope_cos,
                           rope_sin, stream));
    TRY(rfk_rmsnorm_residual_mixed_cast16(x, ffn_buf, w->ffn_norm_gamma, temp, M, dim, kEpsFp32, stream));
    TRY(rfk_ffn_swiglu(ctx, &w->ffn, temp, ffn_buf, qkv_buf, M, dim, ffn_hidden, stream));
    if (pending_out) { *pending_out = ffn_buf; return RFK_OK; }
    return rfk_residual_add_mixed(x, ffn_buf, (long long)M * dim, stream);
}

// ------------------------------------------------------------------------------------------
// rfk_sdpa without a caller-supplied score buffer.
//
// Some callers of this library are not in a position to allocate device memory: host
// callbacks enqueued on a stream (no CUDA allocation call is allowed there), code that runs
// while another thread's stream capture forbids cudaMalloc, and plug-in hosts that hand the
// library a fixed set of tensors and forbid it to grow the process's memory. For them the fp32 score matrix of
// the attention lives in the library itself: a file-scope __device__ array of fixed size that
// every GPU that loads this library holds until the process exits.
constexpr size_t kStaticScoreFloats = 8u << 20;  // 8 Mi floats = 32 MiB
static __device__ __align__(256) float g_static_scores[kStaticScoreFloats];
// In host code the array's name is only a handle for the symbol, not a device address: the
// address is looked up once per device, with that device current, and cached here.
constexpr int kMaxDevices = 64;
static std::atomic<float*> g_static_scores_addr[kMaxDevices];

extern "C" int rfk_sdpa_static(rfk_ctx* ctx, const rfk_half* Q, const rfk_half* K, const rfk_half* V,
                               rfk_half* O, int B, int H, int Sq, int Sk, int n_keys, int D, int o_bshd,
                               rfk_stream_t stream) {
    if (!ctx || !Q || !K || !V || !O) return RFK_EINVAL;
    if (B < 0 || H <= 0 || Sq < 0 || Sk <= 0 || D <= 0 || n_keys <= 0 || n_keys > Sk) return RFK_EINVAL;
    const size_t ld = ((size_t)Sk + 7) & ~(size_t)7;
    if (ld > 8192) return RFK_EUNSUPPORTED;  // same limit as rfk_sdpa: the softmax keeps a row in registers
    // B*H*Sq*roundup8(Sk) floats must fit in 32 MiB; each factor is bounded by division so that the
    // product cannot wrap around for huge arguments
    size_t room = kStaticScoreFloats / ld;
    for (const int f : {B, H, Sq}) {
        if (f == 0) return RFK_OK;  // nothing to compute
        if ((size_t)f > room) return RFK_ETOOBIG;
        room /= (size_t)f;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev != ctx->device) return RFK_EINVAL;  // the array that is looked up below belongs to the current device
    if (dev < 0 || dev >= kMaxDevices) return RFK_EUNSUPPORTED;
    float* scores = g_static_scores_addr[dev].load(std::memory_order_acquire);
    if (!scores) {  // first call on this device (two threads racing here both store the same address)
        e = cudaGetSymbolAddress((void**)&scores, g_static_scores);
        if (e != cudaSuccess) return (int)e;
        g_static_scores_addr[dev].store(scores, std::memory_order_release);
    }
    // Nothing in the array has to be cleared first: the score GEMM overwrites (beta = 0) every
    // element the softmax reads, and the softmax writes every element the second GEMM reads.
    return rfk_sdpa(ctx, Q, K, V, O, scores, nullptr, B, H, Sq, Sk, n_keys, D, o_bshd, stream);
}
