// Channels-last companions of the DPT head's element-wise operators.
//
// The head (csrc/dpt.cu) keeps its activations as [N, H, W, C] fp16: the decoder's token maps already are
// ([S, dim] = [pH, pW, dim]), the tensor-core convolution kernels of the library want that layout (given NCHW
// tensors they convert every operand on the way in and out: 35 % of the head's time), and a 1x1 convolution is then
// a plain row-major GEMM that the tcgen05 projection kernel serves. Every operator here works on rows of C
// contiguous channels with C % 8 == 0, one thread per 8 channels (one 128-bit access per operand).
//
// Arithmetic and roundings are those of the reference's NCHW operators applied one after the other
// (BANANASJIM/renderformer-cuda, src/layers/dpt.cu: add_bias_nchw_kernel :88-96, silu_inplace :289-298,
// residual_add via src/layers/transformer.cu, bilinear_upsample :240-277): where two of them are fused here the
// intermediate is still rounded to fp16, so the values are bit-identical to the unfused sequence.
#include "common.cuh"
#include "dpt_math.cuh"
#include "kernels_internal.h"

namespace rfk {

// x[r, c] = act(half(x[r, c] + bias[c])) (+ residual[r, c]); bias / residual may be null; act: 0 none, 1 SiLU.
template <bool BIAS, bool SILU, bool RES>
__global__ void __launch_bounds__(256)
bias_act_residual_nhwc_kernel(__half* __restrict__ x, const __half* __restrict__ bias, const __half* __restrict__ res,
                              long long chunks, int c8 /* C / 8 */) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= chunks) return;
    float f[8];
    load8(x + i * 8, f);
    if (BIAS) {
        float b[8];
        load8(bias + (int)((unsigned)i % (unsigned)c8) * 8, b);  // chunks < 2^32 (checked by the launcher)
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = __half2float(__float2half(f[k] + b[k]));
    }
    if (SILU) {
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = silu_sfu(f[k]);
        if (RES) {
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] = __half2float(__float2half(f[k]));
        }
    }
    if (RES) {
        float r[8];
        load8(res + i * 8, r);
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] += r[k];
    }
    store8(x + i * 8, f);
}

__global__ void __launch_bounds__(256)
silu_nhwc_kernel(const __half* __restrict__ x, __half* __restrict__ y, long long chunks) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= chunks) return;
    float f[8];
    load8(x + i * 8, f);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = silu_sfu(f[k]);
    store8(y + i * 8, f);
}

// y += r, and silu of the sum beside it: the operand of the residual unit that follows the addition
__global__ void __launch_bounds__(256)
residual_add_silu_nhwc_kernel(__half* __restrict__ y, const __half* __restrict__ r, __half* __restrict__ s, long long chunks) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= chunks) return;
    float f[8], g[8];
    load8(y + i * 8, f);
    load8(r + i * 8, g);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = round_half(f[k] + g[k]);
    store8(y + i * 8, f);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = silu_sfu(f[k]);
    store8(s + i * 8, f);
}

// out[n, ho, wo, :] from in[n, :, :, :], align_corners = true; a thread owns 8 channels of one output column in ROWS
// consecutive rows, so every access is 16 bytes, the column's coordinates are computed once, and the two source pixels of a source
// row are loaded and converted once for all the output rows that lie on it (enlarging by two: five source rows for eight outputs,
// where a thread per output loads sixteen). Those loads, not the 134 MB it writes, bound the 256 -> 512 resample of 256 channels:
// 71 us with a thread per output, 51 with eight rows; upsample_rows says which maps take how many. Grid: x over
// (wo, channel chunk) of one output row, y = groups of rows, z = n: the row arithmetic is uniform over a CTA and the only
// division left is a 32-bit one (with one thread per flat 64-bit index the three divisions cost more than the loads).
template <int ROWS>
__global__ void __launch_bounds__(256)
bilinear_upsample_nhwc_kernel(const __half* __restrict__ in, __half* __restrict__ out, int H_in, int W_in, int H_out, int W_out,
                              int c8) {
    pdl_wait();
    pdl_trigger();
    const unsigned idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (unsigned)W_out * (unsigned)c8) return;
    const int w_out = (int)(idx / (unsigned)c8), cc = (int)(idx % (unsigned)c8);
    const long long n = blockIdx.z;
    const float h_scale = (H_out > 1) ? (float)(H_in - 1) / (H_out - 1) : 0.0f;
    const float w_scale = (W_out > 1) ? (float)(W_in - 1) / (W_out - 1) : 0.0f;
    const long long C = (long long)c8 * 8;
    if (ROWS == 1) {   // nothing to share
        const int h_out = blockIdx.y;
        const float h_in_f = __fmul_rn((float)h_out, h_scale), w_in_f = __fmul_rn((float)w_out, w_scale);
        const int h0 = (int)h_in_f, w0 = (int)w_in_f;
        const int h1 = min(h0 + 1, H_in - 1), w1 = min(w0 + 1, W_in - 1);
        const float hf = __fsub_rn(h_in_f, (float)h0), wf = __fsub_rn(w_in_f, (float)w0);
        const __half* base = in + n * H_in * W_in * C + cc * 8;
        float v00[8], v01[8], v10[8], v11[8], o[8];
        unpack8(ldg_half8(base + ((long long)h0 * W_in + w0) * C), v00);
        unpack8(ldg_half8(base + ((long long)h0 * W_in + w1) * C), v01);
        unpack8(ldg_half8(base + ((long long)h1 * W_in + w0) * C), v10);
        unpack8(ldg_half8(base + ((long long)h1 * W_in + w1) * C), v11);
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = bilerp_ref(v00[k], v01[k], v10[k], v11[k], hf, wf);
        store8(out + ((n * H_out + h_out) * W_out) * C + (long long)idx * 8, o);
        return;
    }
    const float w_in_f = __fmul_rn((float)w_out, w_scale);
    const int w0 = (int)w_in_f, w1 = min(w0 + 1, W_in - 1);
    const float wf = __fsub_rn(w_in_f, (float)w0);   // not contracted with the product: so are the operators this one equals
    const __half* left = in + (n * H_in * W_in + w0) * C + cc * 8;
    const __half* right = in + (n * H_in * W_in + w1) * C + cc * 8;
    float t0[8], t1[8], b0[8], b1[8];   // the two pixels of source rows h0 and h1
    int have0 = -1, have1 = -1;      // which rows they are
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int h_out = blockIdx.y * ROWS + r;
        if (h_out >= H_out) return;
        const float h_in_f = __fmul_rn((float)h_out, h_scale);
        const int h0 = (int)h_in_f, h1 = min(h0 + 1, H_in - 1);
        const float hf = __fsub_rn(h_in_f, (float)h0);
        if (h0 != have0) {           // uniform over the CTA
            if (h0 == have1) {
#pragma unroll
                for (int k = 0; k < 8; ++k) { t0[k] = b0[k]; t1[k] = b1[k]; }
            } else {
                unpack8(ldg_half8(left + (long long)h0 * W_in * C), t0);
                unpack8(ldg_half8(right + (long long)h0 * W_in * C), t1);
            }
            have0 = h0;
        }
        if (h1 != have1) {
            if (h1 == h0) {
#pragma unroll
                for (int k = 0; k < 8; ++k) { b0[k] = t0[k]; b1[k] = t1[k]; }
            } else {
                unpack8(ldg_half8(left + (long long)h1 * W_in * C), b0);
                unpack8(ldg_half8(right + (long long)h1 * W_in * C), b1);
            }
            have1 = h1;
        }
        float o[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = bilerp_ref(t0[k], t1[k], b0[k], b1[k], hf, wf);
        store8(out + ((n * H_out + h_out) * W_out) * C + (long long)idx * 8, o);
    }
}

// A transposed convolution whose stride equals its kernel size f, as GEMM + this scatter: in [N*H*W, f*f*C] holds, for
// every input pixel, the f x f output pixels it produces (column (i*f + j)*C + c); out [N, H*f, W*f, C] (+ bias[c]).
__global__ void __launch_bounds__(256)
depth_to_space_bias_nhwc_kernel(const __half* __restrict__ in, const __half* __restrict__ bias, __half* __restrict__ out,
                                long long chunks, int H, int W, int c8, int f) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // over the OUTPUT, 8 channels each
    if (i >= chunks) return;
    const int cc = (int)(i % c8);
    long long p = i / c8;
    const int wo = (int)(p % (W * f));
    p /= (W * f);
    const int ho = (int)(p % (H * f));
    const long long n = p / (H * f);
    const int h = ho / f, di = ho % f, w = wo / f, dj = wo % f;
    const long long src = (((n * H + h) * W + w) * (f * f) + (di * f + dj)) * c8 + cc;
    float v[8];
    load8(in + src * 8, v);
    if (bias) {
        float b[8];
        load8(bias + cc * 8, b);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] += b[k];
    }
    store8(out + i * 8, v);
}

// [N, HW, C] -> [N, C, HW] for small C (the head's last layer: C = 3): one thread per output element
__global__ void __launch_bounds__(256)
permute_nhwc_to_nchw_kernel(const __half* __restrict__ in, __half* __restrict__ out, long long total, long long HW, int C) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const long long hw = i % HW;
    const long long nc = i / HW;
    const int c = (int)(nc % C);
    const long long n = nc / C;
    out[i] = in[(n * HW + hw) * C + c];
}

// The head's last layer: a 1x1 convolution to a few channels (C_out <= 4: the image's colour channels) + bias, written
// planar. in [N*HW, C_in] channels-last, w [C_out, C_in], out [N, C_out, HW]; one thread per pixel: the pixel's C_in
// values are read once (16 bytes at a time) and every output plane is written with consecutive threads on consecutive
// pixels. fp32 accumulation over the channels in order, the product rounded to fp16 before the bias is added (as a
// convolution followed by the bias kernel does).
template <int COUT>
__global__ void __launch_bounds__(256)
pointwise_to_planar_kernel(const __half* __restrict__ in, const __half* __restrict__ w, const __half* __restrict__ bias,
                           __half* __restrict__ out, long long HW, long long total, int c_in) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ float sw[];  // [COUT][c_in]
    for (int i = threadIdx.x; i < COUT * c_in; i += blockDim.x) sw[i] = __half2float(w[i]);
    __syncthreads();
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= total) return;
    float acc[COUT];
#pragma unroll
    for (int o = 0; o < COUT; ++o) acc[o] = 0.0f;
    const __half* px = in + p * c_in;
    for (int c = 0; c < c_in; c += 8) {
        float v[8];
        load8(px + c, v);
#pragma unroll
        for (int o = 0; o < COUT; ++o)
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[o] = fmaf(v[k], sw[o * c_in + c + k], acc[o]);
    }
    const long long n = p / HW, hw = p % HW;
#pragma unroll
    for (int o = 0; o < COUT; ++o) {
        float r = __half2float(__float2half(acc[o]));
        if (bias) r += __half2float(bias[o]);
        out[(n * COUT + o) * HW + hw] = __float2half(r);
    }
}

// One-off weight layouts (at plan time): mode 0: [K, C, RS] -> [K, RS, C] (filter for channels-last convolutions);
// mode 1: transposed-convolution filter [Cin = K, Cout = C, RS = f*f] -> GEMM weight [(p * Cout + co)][ci].
__global__ void __launch_bounds__(256)
permute_filter_kernel(const __half* __restrict__ w, __half* __restrict__ out, int K, int C, int RS, int mode) {
    const long long total = (long long)K * C * RS;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int p = (int)(i % RS);
    const int c = (int)((i / RS) % C);
    const int k = (int)(i / ((long long)RS * C));
    const long long dst = mode == 0 ? ((long long)k * RS + p) * C + c : ((long long)p * C + c) * K + k;
    out[dst] = w[i];
}

template <bool BIAS, bool SILU, bool RES>
static int launch_bar(__half* x, const __half* bias, const __half* res, long long chunks, int c8, cudaStream_t st) {
    launch_pdl(bias_act_residual_nhwc_kernel<BIAS, SILU, RES>, dim3((unsigned)ceil_div(chunks, 256)), dim3(256), 0, st, x, bias, res, chunks, c8);
    return launch_status();
}

}  // namespace rfk

using namespace rfk;

extern "C" int rfk_bias_act_residual_nhwc(rfk_half* x, const rfk_half* bias, const rfk_half* residual, long long rows, int C,
                                          int silu, rfk_stream_t stream) {
    if (!x || rows < 0 || C <= 0) return RFK_EINVAL;
    if (rows == 0) return RFK_OK;
    if (C % 8 || !aligned16(x) || (bias && !aligned16(bias)) || (residual && !aligned16(residual))) return RFK_EUNSUPPORTED;
    const long long chunks = rows * (C / 8);
    if (chunks > 0xffffffffLL) return RFK_EUNSUPPORTED;
    __half* px = (__half*)x;
    const __half *pb = (const __half*)bias, *pr = (const __half*)residual;
    cudaStream_t st = as_stream(stream);
    const int c8 = C / 8;
    switch ((bias ? 4 : 0) | (silu ? 2 : 0) | (residual ? 1 : 0)) {
        case 0: return RFK_OK;
        case 1: return launch_bar<false, false, true>(px, pb, pr, chunks, c8, st);
        case 2: return launch_bar<false, true, false>(px, pb, pr, chunks, c8, st);
        case 3: return launch_bar<false, true, true>(px, pb, pr, chunks, c8, st);
        case 4: return launch_bar<true, false, false>(px, pb, pr, chunks, c8, st);
        case 5: return launch_bar<true, false, true>(px, pb, pr, chunks, c8, st);
        case 6: return launch_bar<true, true, false>(px, pb, pr, chunks, c8, st);
        default: return launch_bar<true, true, true>(px, pb, pr, chunks, c8, st);
    }
}

extern "C" int rfk_silu(const rfk_half* x, rfk_half* y, long long n, rfk_stream_t stream) {
    if (!x || !y || n < 0) return RFK_EINVAL;
    if (n == 0) return RFK_OK;
    if (n % 8 || !aligned16(x) || !aligned16(y)) return RFK_EUNSUPPORTED;
    launch_pdl(silu_nhwc_kernel, dim3((unsigned)ceil_div(n / 8, 256)), dim3(256), 0, as_stream(stream), (const __half*)x, (__half*)y, n / 8);
    return launch_status();
}

extern "C" int rfk_residual_add_silu_nhwc(rfk_half* y, const rfk_half* r, rfk_half* y_silu, long long n, rfk_stream_t stream) {
    if (!y || !r || !y_silu || n < 0) return RFK_EINVAL;
    if (n == 0) return RFK_OK;
    if (n % 8 || !aligned16(y) || !aligned16(r) || !aligned16(y_silu) || n / 8 > 0x7fffffffLL) return RFK_EUNSUPPORTED;
    launch_pdl(residual_add_silu_nhwc_kernel, dim3((unsigned)ceil_div(n / 8, 256)), dim3(256), 0, as_stream(stream), (__half*)y,
               (const __half*)r, (__half*)y_silu, n / 8);
    return launch_status();
}

// Output rows a thread: 1, 4 or 8, by the number of CTAs that one row a thread would be. Sharing source rows needs output rows closer
// together than source rows, and costs threads. Measured (us, one / four / eight rows; 256 channels): 32 -> 64 (512 CTAs) 2.46 / 2.86 / 3.99,
// 56 -> 112 (1568) 4.71 / 5.12 / 5.02, 64 -> 128 (2048) 5.63 / 5.12 / 5.01, 72 -> 144 (2592) 6.86 / 6.14 / 7.68, 88 -> 176 (3872) 9.52 / 7.88 / 7.88,
// 128 -> 256 (8192) 18.6 / 14.5 / 12.7, 256 -> 512 70.8 / 58.4 / 50.7; shrinking, 256 -> 230 15.5 / 13.9 / 14.2, 256 -> 200 11.9 / 11.3 / 12.1,
// 512 -> 256 25.3 / 31.8 / 31.2.
static int upsample_rows(long long ctas, int H_in, int H_out) {
    if (8LL * H_out < 7LL * H_in || ctas < 1800) return 1;
    return ctas < 3800 ? 4 : 8;
}

extern "C" int rfk_bilinear_upsample_nhwc(const rfk_half* in, rfk_half* out, int N, int H_in, int W_in, int H_out, int W_out,
                                          int C, rfk_stream_t stream) {
    if (!in || !out || N < 0 || C <= 0 || H_in <= 0 || W_in <= 0 || H_out <= 0 || W_out <= 0) return RFK_EINVAL;
    if (N == 0) return RFK_OK;
    if (C % 8 || !aligned16(in) || !aligned16(out)) return RFK_EUNSUPPORTED;
    const long long per_row = (long long)W_out * (C / 8);
    if (per_row > 0x7fffffffLL || H_out > 65535 || N > 65535) return RFK_EUNSUPPORTED;
    const int rows = upsample_rows(ceil_div(per_row, 256) * H_out * N, H_in, H_out);
    const dim3 grid((unsigned)ceil_div(per_row, 256), (unsigned)ceil_div(H_out, rows), (unsigned)N);
    launch_pdl(rows == 8 ? bilinear_upsample_nhwc_kernel<8> : rows == 4 ? bilinear_upsample_nhwc_kernel<4> : bilinear_upsample_nhwc_kernel<1>,
               grid, dim3(256), 0, as_stream(stream),
               (const __half*)in, (__half*)out, H_in, W_in, H_out, W_out, C / 8);
    return launch_status();
}

extern "C" int rfk_depth_to_space_bias_nhwc(const rfk_half* in, const rfk_half* bias, rfk_half* out, int N, int H, int W, int C,
                                            int f, rfk_stream_t stream) {
    if (!in || !out || N < 0 || H <= 0 || W <= 0 || C <= 0 || f <= 0) return RFK_EINVAL;
    if (N == 0) return RFK_OK;
    if (C % 8 || !aligned16(in) || !aligned16(out) || (bias && !aligned16(bias))) return RFK_EUNSUPPORTED;
    const long long chunks = (long long)N * H * f * W * f * (C / 8);
    if (chunks > 0x7fffffffLL * 256) return RFK_EUNSUPPORTED;
    launch_pdl(depth_to_space_bias_nhwc_kernel, dim3((unsigned)ceil_div(chunks, 256)), dim3(256), 0, as_stream(stream),
        (const __half*)in, (const __half*)bias, (__half*)out, chunks, H, W, C / 8, f);
    return launch_status();
}

extern "C" int rfk_permute_nhwc_to_nchw(const rfk_half* in, rfk_half* out, int N, long long HW, int C, rfk_stream_t stream) {
    if (!in || !out || N < 0 || HW < 0 || C <= 0) return RFK_EINVAL;
    const long long total = (long long)N * HW * C;
    if (total == 0) return RFK_OK;
    if (total > 0x7fffffffLL * 256) return RFK_EUNSUPPORTED;
    launch_pdl(permute_nhwc_to_nchw_kernel, dim3((unsigned)ceil_div(total, 256)), dim3(256), 0, as_stream(stream), (const __half*)in, (__half*)out,
                                                                                               total, HW, C);
    return launch_status();
}

extern "C" int rfk_permute_filter(const rfk_half* w, rfk_half* out, int K, int C, int RS, int mode, rfk_stream_t stream) {
    if (!w || !out || K <= 0 || C <= 0 || RS <= 0 || mode < 0 || mode > 1) return RFK_EINVAL;
    const long long total = (long long)K * C * RS;
    if (total > 0x7fffffffLL * 256) return RFK_EUNSUPPORTED;
    permute_filter_kernel<<<(unsigned)ceil_div(total, 256), 256, 0, as_stream(stream)>>>((const __half*)w, (__half*)out, K, C, RS,
                                                                                         mode);
    return launch_status();
}

extern "C" int rfk_pointwise_conv_to_planar(const rfk_half* in, const rfk_half* weight, const rfk_half* bias, rfk_half* out, int N,
                                            long long HW, int C_in, int C_out, rfk_stream_t stream) {
    if (!in || !weight || !out || N < 0 || HW < 0 || C_in <= 0 || C_out <= 0) return RFK_EINVAL;
    const long long total = (long long)N * HW;
    if (total == 0) return RFK_OK;
    if (C_out > 4 || C_in % 8 || C_in > 2048 || !aligned16(in)) return RFK_EUNSUPPORTED;
    if (total > 0x7fffffffLL * 256) return RFK_EUNSUPPORTED;
    const unsigned grid = (unsigned)ceil_div(total, 256);
    const size_t smem = (size_t)C_out * C_in * sizeof(float);
    cudaStream_t st = as_stream(stream);
    const __half *pi = (const __half*)in, *pw = (const __half*)weight, *pb = (const __half*)bias;
    __half* po = (__half*)out;
    switch (C_out) {
        case 1: launch_pdl(pointwise_to_planar_kernel<1>, dim3(grid), dim3(256), smem, st, pi, pw, pb, po, HW, total, C_in); break;
        case 2: launch_pdl(pointwise_to_planar_kernel<2>, dim3(grid), dim3(256), smem, st, pi, pw, pb, po, HW, total, C_in); break;
        case 3: launch_pdl(pointwise_to_planar_kernel<3>, dim3(grid), dim3(256), smem, st, pi, pw, pb, po, HW, total, C_in); break;
        default: launch_pdl(pointwise_to_planar_kernel<4>, dim3(grid), dim3(256), smem, st, pi, pw, pb, po, HW, total, C_in); break;
    }
    return launch_status();
}
