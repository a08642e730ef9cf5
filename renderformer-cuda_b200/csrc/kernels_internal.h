// Forms of the kernels that only the layer library uses (not part of the C ABI): more head sizes than the C entry points
// of the same name take.
#pragma once
#include "rfk.h"

namespace rfk {

// rfk_gemm_f16_heads for heads of 64 or 128: out is [part][group][head][out_seq][head_dim], of which the first seq_len rows of
// each head are written. out_seq other than seq_len, and a seq_len that is not a multiple of 32, need one group (M == seq_len).
int gemm_heads(const rfk_half* A, long long lda, const rfk_half* W, long long ldw, rfk_half* out, long long part_stride,
               float* row_ss, int ss_parts_mask, int M, int N, int K, int seq_len, int out_seq, int num_heads,
               int head_dim, rfk_stream_t stream);

// Products of a layer whose norms are folded into them ("Folded norms" in gemm_tc.cu): A [M, K] un-normalised with its rows' sums of squares, W
// [N, K] with the norm's weight multiplied in. One of: W_up (SwiGLU, C [M, N]), num_heads > 0 (head-split, C as gemm_heads'), R (C = R + A W^T).
// out_ss (may be NULL; residual and head-split): the sums of squares of the rows written, *ss_tiles a row (of a part). A residual product's
// rows may be the 4 x 4 blocks of a token grid in window order, of a grid shifted by shift_from blocks; they are then written in the order
// of a grid shifted by shift_to blocks (C, with out_ss) and in raster order (raster), each where it is not NULL; C is then not R. W is not written by the
// kernel right ahead in the stream, unless FoldedMore::pairs is asked for.
// RFK_EUNSUPPORTED: shapes or a device that these kernels do not serve, nothing launched.
struct FoldedProduct {
    const rfk_half *A, *W, *W_up, *R;
    rfk_half *C, *raster;
    int M, N, K;
    const float* in_ss; int in_tiles; float in_mul, eps;    // SwiGLU and head-split: a row's factor is in_mul / sqrt(mean square + eps)
    float* out_ss; int ss_mask;                             // head-split: parts that get sums
    long long part_stride; int seq, num_heads, head_dim;
    int out_seq;                                            // head-split: rows a head has room for (0: seq)
    int blocks_across, blocks_down, shift_from, shift_to;   // 0: rows stay where they are
    int quarters;                                           // residual: the sum over K is ((a + b) + c) + d of its quarters (K % 512 == 0), whatever M
};
struct FoldedMore {
    int pairs;      // CTA pairs with one sum each 256 columns, which read W behind the kernel before, or RFK_EUNSUPPORTED: small tiles write one each
                    // 32 columns, and ask for W while the kernel before may still be writing it
    const float *w_mul, *w_up_mul;   // SwiGLU and head-split: what each 64 rows of W and W_up are to be multiplied by (fold_weights); device memory, or NULL
};
int gemm_folded(const FoldedProduct& f, int* ss_tiles, rfk_stream_t stream, const FoldedMore& more = {});
// whether a product (SwiGLU aside) goes to the pairs of FoldedMore::pairs, by its size
bool folded_on_pairs(int M, int N);

// The tokens that enter a view's folded layers, 1024 wide (else RFK_EUNSUPPORTED): x = half(half(rmsnorm(e) * gamma) + token), with the bits of the
// separate steps, and its rows' sums of squares row_ss [rows][4]. e is a token grid in raster order, x in the block order of gemm_folded, of
// the unshifted grid.
int embed_tokens(const rfk_half* e, const float* gamma, const rfk_half* token, rfk_half* x, float* row_ss, int rows, int dim, float eps,
                 int blocks_across, int blocks_down, rfk_stream_t stream);

// The keys and values of several layers from one set of rows (1024 wide, else RFK_EUNSUPPORTED): y = half(x + r) with its rows' sums of squares
// row_ss [rows][4] (r may be NULL); and the keys' own norm, in place on [layers] slabs [head][out_seq][head_dim], layer_stride apart,
// with sums row_ss [2 * layers][rows][4] of which the keys' are read
int context_rows(const float* x, const rfk_half* r, rfk_half* y, float* row_ss, int rows, int dim, rfk_stream_t stream);
int keys_norm(rfk_half* keys, long long layer_stride, const float* const* gamma, const float* row_ss, int layers, int rows, int out_seq, int num_heads,
              int head_dim, float eps, rfk_stream_t stream);

// Weights for gemm_folded, 1024 wide (else RFK_EUNSUPPORTED): n matrices [rows[i]][1024], rows in whole 64s, one after the other in out as
// half(w * gamma[i][column] / mul), where mul is a power of two for each 64 rows of them all, written to device memory: their largest product
// comes to between 2^13 and 2^14
constexpr int kMaxFolded = 64;
int fold_weights(const rfk_half* const* w, const float* const* gamma, const int* rows, int n, int cols, rfk_half* out, float* mul, rfk_stream_t stream);

// rfk_qkv_norm_rope_transpose behind gemm_heads: parts [heads][out_seq][head_dim], of which the first seq_len rows of each head are
// normalised over the row (all heads) and, unless cos_vals is NULL, rotated in place, with that kernel's bits
int qk_norm_rope_heads(int n_parts, const float* const* gamma, rfk_half* const* parts, const rfk_half* cos_vals,
                       const rfk_half* sin_vals, int seq_len, int out_seq, int num_heads, int head_dim, float eps, rfk_stream_t stream);

// out = rmsnorm_f32(a) + rmsnorm_f32(b) + c, fp32, in one pass with the bits of the separate steps; a, b fp16 [rows, dim], c fp16 [dim];
// dim % 8 == 0, dim <= 1024, 16-byte aligned, else RFK_EUNSUPPORTED
int norm_pair_add(const rfk_half* a, const float* gamma_a, const rfk_half* b, const float* gamma_b, const rfk_half* c, float* out,
                  int rows, int dim, float eps, rfk_stream_t stream);

// rfk_window_attention (q_row_ss NULL) / rfk_window_attention_normed for heads of 64 or 128. ss_group: how many of a row's sums make up 256
// columns, 1 or 8 (gemm_folded). blocks (rows of 1024): a window's tokens are its 4 x 4 blocks one after the other, the mask stays in row
// order; only that form takes groups of 8
int window_attention(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O, const uint8_t* mask,
                     const float* q_row_ss, const float* k_row_ss, int ss_tiles, const float* gamma_q, const float* gamma_k,
                     int norm_dim, float eps, int BnW, int num_heads, int window_tokens, int head_dim, int nW, float scale,
                     rfk_stream_t stream, int ss_group = 1, bool blocks = false);

// The same for heads of 128 with the bits of the separate steps: library Q K^T with the scale as its alpha,
// rfk_swin_softmax_probs_inplace, library P V, rfk_transpose_bhsd_to_bsd
int window_attention_steps(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O, const uint8_t* mask, int BnW,
                           int num_heads, int window_tokens, int head_dim, int nW, float scale, rfk_stream_t stream);

// Which grids a workspace may cut along the keys (plan_work in attention_tc.cu): none, those of less than one round of the SMs,
// or the last, partial round of larger ones too. kNone also takes the row sums of 128-wide heads in the order of
// flash_attention_mma, whose bits the result then has.
enum class AttnCut { kNone, kBelowOneRound, kLastRound };

// rfk_flash_attention_ex for heads of 64 or 128
int flash_attention_ex(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O, const float* q_row_ss, int ss_tiles,
                       int norm_dim, float eps, void* workspace, size_t workspace_bytes, AttnCut cut, int v_shared, int B, int H,
                       int Sq, int Sk, int n_keys, int D, int o_bshd, float scale, rfk_stream_t stream, int ss_group = 1);

// the mma.sync kernel of rfk_flash_attention, whatever path is set
int flash_attention_mma(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O, int B, int H, int Sq, int Sk,
                        int n_keys, int D, int o_bshd, float scale, rfk_stream_t stream);

}  // namespace rfk

// The same with AttnCut::kLastRound, and with kNone, for the tests of the 128-wide kernel, which reach the library through its C
// symbols.
extern "C" int rfk_flash_attention_ex_wide(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O,
                                           const float* q_row_ss, int ss_tiles, int norm_dim, float eps, void* workspace,
                                           size_t workspace_bytes, int v_shared, int B, int H, int Sq, int Sk, int n_keys, int D,
                                           int o_bshd, float scale, rfk_stream_t stream);
extern "C" int rfk_flash_attention_ordered(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O, int B, int H, int Sq,
                                           int Sk, int n_keys, int D, int o_bshd, float scale, rfk_stream_t stream);
extern "C" int rfk_flash_attention_ordered_ws(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O, void* workspace,
                                              size_t workspace_bytes, int B, int H, int Sq, int Sk, int n_keys, int D, int o_bshd,
                                              float scale, rfk_stream_t stream);
// The clock of the attention's wait for a unit's first piece on a sequence of readings of the timer, in ns, the first at the wait's start: index of the
// reading that ends the wait, 0 if none does; for its test, host only
extern "C" int rfk_wait_clock(const unsigned long long* readings, int n);
// One step on the word of a handed-over unit (handover.cuh), for its test, host only: event 0 / 1 the first piece is done / gave up,
// 2 the second piece looks, 3 it is past its wait. Returns what that piece does next (handover::Act), *next the word.
extern "C" int rfk_handover_step(int word, int event, int* next);
// A piece of a unit cut into `pieces` arrives at its counter, for its test, host only: 1 if it merges the unit.
extern "C" int rfk_piece_arrives(int* counter, int failed, int pieces);
// Which units of a grid that is not cut the launcher hands over from one SM to another (plan_handover in attention_tc.cu): units
// [0, *whole_units) stay whole, then for each of *n_handed units {unit, key tiles of its first piece, slot} in launch order.
extern "C" int rfk_flash_attention_handover_plan(long long units, int n_tiles, int sms, int* whole_units, int* n_handed,
                                                 unsigned short* first, int max_handed);
// Columns of the pair kernel's tiles, 192 or 256, for a product of M x N on a device that runs `pairs` CTA pairs at once (narrow_tile
// in gemm_tc.cu), for its test; host only
extern "C" int rfk_gemm_pair_tile(int M, int N, int pairs);
// window_attention_steps, for its test
extern "C" int rfk_window_attention_steps(const rfk_half* Q, const rfk_half* K, const rfk_half* V, rfk_half* O, const uint8_t* mask,
                                          int BnW, int num_heads, int nW, float scale, rfk_stream_t stream);

// 3x3 convolution of the DPT head (conv_tc.cu): x [N,H,W,C_in], w [C_out,3,3,C_in], stride 1, padding 1;
// out [N,H,W,C_out] = act(half(conv) + bias) (+ residual), act SiLU if silu, every intermediate rounded to fp16; out_silu (may be
// NULL) = silu(out). bias and residual may be NULL; out and out_silu must not be x or one another. rows_outside: the order of the
// sums (see conv_tc.cu). C_in % 64 == 0, C_out % 128 == 0, else RFK_EUNSUPPORTED.
extern "C" int rfk_conv3x3_nhwc(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, rfk_half* out,
                                rfk_half* out_silu, int N, int H, int W, int C_in, int C_out, int silu, int rows_outside,
                                rfk_stream_t stream);
// The same for C_out % 32 == 0, with the tile named: output channels x pixels of a CTA 128 x 128 (1; C_out % 128 == 0), 64 x 128 (2), 64 x 64 (3), 32 x 128 with
// the weights resident (4; C_out == 32, C_in <= 128), or by the rule on sizes (0). All of them have the same bits.
extern "C" int rfk_conv3x3_nhwc_tiled(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, rfk_half* out,
                                      rfk_half* out_silu, int N, int H, int W, int C_in, int C_out, int silu, int rows_outside, int tile,
                                      rfk_stream_t stream);
// sum += half(half(half(conv) + bias) + residual) and sum_silu = silu(sum): a residual unit's second convolution, the sum into the path and the SiLU that
// opens the next unit (rfk_residual_add_silu_nhwc), with the bits of the separate steps. sum and sum_silu must not be x, residual or one another; not for
// the shapes whose weights stay resident (RFK_EUNSUPPORTED).
extern "C" int rfk_conv3x3_nhwc_add(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, rfk_half* sum,
                                    rfk_half* sum_silu, int N, int H, int W, int C_in, int C_out, int rows_outside, int tile, rfk_stream_t stream);
// whether it takes these operands on the current device
extern "C" int rfk_conv3x3_nhwc_serves(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual,
                                       const rfk_half* out, const rfk_half* out_silu, int C_in, int C_out);

// y += r in fp16, and silu(y) beside it: rfk_residual_add and rfk_silu in one pass; n % 8 == 0, 16-byte aligned
extern "C" int rfk_residual_add_silu_nhwc(rfk_half* y, const rfk_half* r, rfk_half* y_silu, long long n, rfk_stream_t stream);

extern "C" int rfk_embed_tokens(const rfk_half* e, const float* gamma, const rfk_half* token, rfk_half* x, float* row_ss, int rows, int dim, float eps,
                                int blocks_across, int blocks_down, rfk_stream_t stream);   // embed_tokens and fold_weights, for their tests
extern "C" int rfk_fold_weights(const rfk_half* const* w, const float* const* gamma, const int* rows, int n, int cols, rfk_half* out, float* mul,
                                rfk_stream_t stream);
extern "C" int rfk_gemm_folded(const rfk::FoldedProduct* f, int* ss_tiles, rfk_stream_t stream);   // gemm_folded and folded_on_pairs, for their tests
extern "C" int rfk_gemm_folded_more(const rfk::FoldedProduct* f, const rfk::FoldedMore* more, int* ss_tiles, rfk_stream_t stream);
extern "C" int rfk_folded_on_pairs(int M, int N);
// rfk_rmsnorm_residual_f16_windows for operands that the kernels before have just written (the layers' case): the same values, another
// split of the rows (one_warp_per_row in rmsnorm.cu)
extern "C" int rfk_rmsnorm_residual_f16_windows_in_l2(rfk_half* x, const rfk_half* r, const float* gamma, rfk_half* y, int B, int H, int W,
                                                      int dim, int window_size, int shift_size, int windowed_operand, float eps,
                                                      rfk_stream_t stream);

// qk_norm_rope_heads of q and k, or of q alone (k NULL), for its test
extern "C" int rfk_qk_norm_rope_heads(rfk_half* q, rfk_half* k, const float* gamma_q, const float* gamma_k, const rfk_half* cos_vals,
                                      const rfk_half* sin_vals, int seq_len, int out_seq, int num_heads, int head_dim, float eps,
                                      rfk_stream_t stream);
// norm_pair_add, for its test
extern "C" int rfk_norm_pair_add(const rfk_half* a, const float* gamma_a, const rfk_half* b, const float* gamma_b, const rfk_half* c,
                                 float* out, int rows, int dim, float eps, rfk_stream_t stream);
