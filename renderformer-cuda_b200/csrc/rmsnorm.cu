// RMSNorm family: plain, and fused with the residual add that precedes it and the
// fp16 cast that follows it.
//
// Reference semantics (BANANASJIM/renderformer-cuda):
//   src/kernels/rmsnorm.cu:17-50,67-90   s = sum x^2 ; r = rsqrtf(s/dim + eps) ; y = (x*r)*gamma
//   src/layers/transformer.cu:9-19       y16 = half(float(y16) + float(r16))
//   src/layers/transformer.cu:21-30      y32 += r32
//   src/layers/transformer.cu:52-61      y32 += float(r16)
//   src/layers/transformer.cu:32-35      out16 = half(in32)
//
// Design: the op is a pure HBM stream (config 1: 3 fp32 row passes + 1 fp16 pass,
// < 1 flop/byte). A row lives in registers between the sum-of-squares and the scaling
// pass, so every byte crosses HBM exactly once. Each lane moves 8 consecutive elements per
// access (128-bit loads/stores for fp16, 2 x 128-bit for fp32).
// A row is spread over W warps of a 128-thread CTA (W = 4 for dim 1024, i.e. one row per
// CTA and one chunk per thread). A first version gave each warp a whole row (32 floats of h
// and of r per lane): ncu showed 30 % DRAM utilisation with every warp stalled on its own
// loads (long-scoreboard 35 cycles/issue), because the whole grid loaded in lock step and
// then stored in lock step, in 1.4 waves. Small CTAs of short-lived threads (32 registers,
// 16 CTAs per SM) retire and get replaced continuously, so loads of new rows overlap the
// stores of finished ones. The W partial sums meet through 16 bytes of shared memory.
#include "common.cuh"
#include "kernels_internal.h"
#include "tc_pair.cuh"

namespace rfk {

template <typename T> struct IsHalf { static constexpr bool value = false; };
template <> struct IsHalf<__half> { static constexpr bool value = true; };

constexpr int kRmsThreads = 128;

// Token (b, h, w) of a [B, H, W] grid -> its row in swin window order (windows of ws x ws over the
// grid shifted by -shift, as the reference's cyclic shift + window_partition produce).
struct WinRows {
    int H, W, ws, shift;
    __device__ __forceinline__ long long operator()(long long token) const {
        const int w = (int)(token % W);
        const long long t = token / W;
        const int h = (int)(t % H);
        const long long b = t / H;
        const int hs = (h + shift) % H, wsft = (w + shift) % W;  // position in the shifted grid
        const int nWw = W / ws, nW = (H / ws) * nWw;
        const int win = (hs / ws) * nWw + wsft / ws, local = (hs % ws) * ws + wsft % ws;
        return (b * nW + win) * (long long)(ws * ws) + local;
    }
};

// TH: hidden-state storage, TR: residual storage, TY: normalised output storage.
// MAP: 0 all operands in token order; 1 y is written in window order; 2 r is read in window order.
// W: warps per row (1, 2 or 4); NCH: 8-element chunks per lane (dim <= NCH * W * 256).
// SUMS: 1, or the number of warps (256-element chunks) whose partial sums a lone warp adds as W warps would, so that a row has
// the same bits either way.
template <typename TH, typename TR, typename TY, int NCH, int W, bool HAS_RES, bool WRITE_H, int MAP = 0, int SUMS = 1>
__global__ void __launch_bounds__(kRmsThreads)
rmsnorm_row_kernel(const TH* x, TH* xw, const TR* __restrict__ r,
                   const float* __restrict__ gamma, TY* y,  // x, xw, y may alias
                   int rows, int dim, float eps, WinRows wr = WinRows{}) {
    constexpr int kWarps = kRmsThreads / 32;
    constexpr int kRowsPerCta = kWarps / W;
    __shared__ float s_part[kWarps];
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wir = warp % W;  // warp index within its row
    long long row = (long long)blockIdx.x * kRowsPerCta + warp / W;
    const bool live = row < rows;
    if (!live) row = rows - 1;  // idle warps shadow the last row and never store
    const size_t base = (size_t)row * dim;
    const size_t rbase = MAP == 2 ? (size_t)wr(row) * dim : base;
    const size_t ybase = MAP == 1 ? (size_t)wr(row) * dim : base;

    float v[NCH][8];
#pragma unroll
    for (int k = 0; k < NCH; ++k) {
        const int off = (wir * 32 + lane + k * W * 32) * 8;
        if (off < dim) load8(x + base + off, v[k]);
    }
    if (HAS_RES) {
#pragma unroll
        for (int k = 0; k < NCH; ++k) {
            const int off = (wir * 32 + lane + k * W * 32) * 8;
            if (off < dim) {
                float rr[8];
                load8(r + rbase + off, rr);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float s = v[k][i] + rr[i];
                    // an fp16 hidden state is stored, then re-read by the norm
                    v[k][i] = IsHalf<TH>::value ? round_half(s) : s;
                }
                if (WRITE_H && live) store8(xw + base + off, v[k]);
            }
        }
    }
    float ss = 0.0f;
    if (SUMS > 1) {
        static_assert(SUMS == 1 || (W == 1 && SUMS == NCH), "one chunk per warp of the other form");
        float part[NCH];
#pragma unroll
        for (int k = 0; k < NCH; ++k) {
            part[k] = 0.0f;
            if ((lane + k * 32) * 8 < dim) {
#pragma unroll
                for (int i = 0; i < 8; ++i) part[k] = fmaf(v[k][i], v[k][i], part[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < NCH; ++k) part[k] = warp_sum(part[k]);
#pragma unroll
        for (int k = 0; k < NCH; ++k) ss += part[k];
    } else {
#pragma unroll
        for (int k = 0; k < NCH; ++k) {
            const int off = (wir * 32 + lane + k * W * 32) * 8;
            if (off < dim) {
#pragma unroll
                for (int i = 0; i < 8; ++i) ss = fmaf(v[k][i], v[k][i], ss);
            }
        }
        ss = warp_sum(ss);
    }
    if (W > 1) {
        if (lane == 0) s_part[warp] = ss;
        __syncthreads();
        ss = 0.0f;
#pragma unroll
        for (int i = 0; i < W; ++i) ss += s_part[(warp / W) * W + i];
    }
    const float rinv = rsqrtf(ss * (1.0f / (float)dim) + eps);
    if (!live) return;
#pragma unroll
    for (int k = 0; k < NCH; ++k) {
        const int off = (wir * 32 + lane + k * W * 32) * 8;
        if (off < dim) {
            float g[8], o[8];
            ldg_float8(gamma + off, g);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = (v[k][i] * rinv) * g[i];
            store8(y + ybase + off, o);
        }
    }
}

// out = norm(a) + norm(b) + c in fp32, a and b fp16, c one fp16 row for all: the two embeddings of a scene's triangles and the
// triangle token, with the bits of two casts to fp32, two fp32 norms and the sum (same chunks, same order of the partial sums as
// rmsnorm_row_kernel with W warps a row). One pass over 46 MB at 5633 x 1024 where the five took 185.
template <int W>
__global__ void __launch_bounds__(kRmsThreads)
norm_pair_add_kernel(const __half* __restrict__ a, const float* __restrict__ gamma_a, const __half* __restrict__ b,
                     const float* __restrict__ gamma_b, const __half* __restrict__ c, float* __restrict__ out, int rows, int dim, float eps) {
    constexpr int kWarps = kRmsThreads / 32;
    __shared__ float s_part[2][kWarps];
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long row = (long long)blockIdx.x * (kWarps / W) + warp / W;
    const bool live = row < rows;
    if (!live) row = rows - 1;  // idle warps shadow the last row and never store
    const int off = ((warp % W) * 32 + lane) * 8;
    const bool in = off < dim;
    float v[2][8], ss[2] = {0.0f, 0.0f};
    if (in) {
        load8(a + (size_t)row * dim + off, v[0]);
        load8(b + (size_t)row * dim + off, v[1]);
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int i = 0; i < 8; ++i) ss[t] = fmaf(v[t][i], v[t][i], ss[t]);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) ss[t] = warp_sum(ss[t]);
    if (W > 1) {
        if (lane == 0) { s_part[0][warp] = ss[0]; s_part[1][warp] = ss[1]; }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            ss[t] = 0.0f;
#pragma unroll
            for (int i = 0; i < W; ++i) ss[t] += s_part[t][(warp / W) * W + i];
        }
    }
    if (!live || !in) return;
    float ga[8], gb[8], cc[8], o[8];
    ldg_float8(gamma_a + off, ga);
    ldg_float8(gamma_b + off, gb);
    load8(c + off, cc);
    const float ra = rsqrtf(ss[0] * (1.0f / (float)dim) + eps), rb = rsqrtf(ss[1] * (1.0f / (float)dim) + eps);
#pragma unroll
    for (int i = 0; i < 8; ++i)   // each term rounded as it was when it was stored
        o[i] = __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(v[0][i], ra), ga[i]), __fmul_rn(__fmul_rn(v[1][i], rb), gb[i])), cc[i]);
    store8(out + (size_t)row * dim + off, o);
}

// The tokens that enter folded layers (gemm_folded), one CTA a row of 1024 (dim): norm, weight, token in one pass, with the bits of rmsnorm_row_kernel
// and a broadcast add, the row's squares added as gemm_folded's epilogues do, and the row's place in block order. Three launches in one.
__global__ void __launch_bounds__(kRmsThreads)
embed_tokens_kernel(const __half* __restrict__ e, const float* __restrict__ gamma, const __half* __restrict__ token, __half* __restrict__ x,
                    float* __restrict__ row_ss, int dim, float eps, int blocks_across, int blocks_down) {
    constexpr int W = kRmsThreads / 32;
    __shared__ float s_part[W];
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, off = threadIdx.x * 8;   // dim = 256 * W
    float v[8], a[8], t[8], ss = 0.0f;
    load8(e + (size_t)blockIdx.x * dim + off, v);
    ldg_float8(gamma + off, a);
    unpack8(ldg_half8(token + off), t);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
    ss = warp_sum(ss);
    if (lane == 0) s_part[warp] = ss;
    __syncthreads();
    ss = 0.0f;
#pragma unroll
    for (int i = 0; i < W; ++i) ss += s_part[i];
    const float rinv = rsqrtf(ss * (1.0f / (float)dim) + eps);
    float c = 0.0f;   // eight squares in column order
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = round_half(round_half((v[i] * rinv) * a[i]) + t[i]);
        c = fmaf(v[i], v[i], c);
    }
    const int across = blocks_across * 4, view_rows = across * blocks_down * 4, view = blockIdx.x / view_rows, r = blockIdx.x - view * view_rows;
    const int y = r / across, z = r - y * across, by = y >> 2, bx = z >> 2;
    const int row = view * view_rows + ((((by >> 1) * (blocks_across >> 1) + (bx >> 1)) << 2) + ((by & 1) << 1) + (bx & 1)) * 16 + (y & 3) * 4 + (z & 3);
    store8(x + (size_t)row * dim + off, v);
    c += __shfl_xor_sync(0xffffffffu, c, 1);   // four of those in pairs
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    float sum = __shfl_sync(0xffffffffu, c, 0);
#pragma unroll
    for (int k = 1; k < 8; ++k) sum += __shfl_sync(0xffffffffu, c, 4 * k);
    if (lane == 0) row_ss[(size_t)row * W + warp] = sum;
}

// Weights of the folded products (gemm_folded): out = half(w * gamma[column] / mul), one matrix after the other, each 64 rows with a power of two of theirs.
// The scale lies in device memory beside the weights, where a captured graph's products find the one that they were divided by last. It is that of
// the largest product and not of the norm's weights: a product that is 2^27 times smaller still has all its bits, where a small norm
// weight that holds down a large channel would otherwise leave products below 2^-14, which have fewer (512 x 1024 x 1024, W of 0.02 n, norm weights
// exp(a n), channels inversely as large, error against 64 bits, separate norm / the norm's weights brought below 1 / this: a = 1 2.9e-4 / 3.2e-4 / 2.9e-4,
// 1.5 2.9e-4 / 3.5e-3 / 2.9e-4, 2 2.9e-4 / 6.9e-2 / 2.9e-4). 2^14 leaves two bits below fp16's largest; the sums are fp32.
// Bound: HBM, each weight once in and once out; the rows stay in registers until their scale is known. A cluster of two CTAs with 32 rows each, two of them an
// SM, loads while another stores: twelve layers' weights (302 MB in, 302 out) 106 us, 5.7 TB/s; 64 rows a CTA 132, 256 threads a CTA 123.
struct FoldList {
    const __half* w[kMaxFolded];
    const float* gamma[kMaxFolded];
    int first[kMaxFolded], groups[kMaxFolded];   // of 64 rows
};
constexpr int kFoldThreads = 512, kFoldCols = 1024, kFoldRows = 32, kFoldChunks = kFoldRows * kFoldCols / 8 / kFoldThreads;
__global__ void __cluster_dims__(2) __launch_bounds__(kFoldThreads, 2)
fold_weights_kernel(const __grid_constant__ FoldList m, __half* __restrict__ out, float* __restrict__ mul) {
    __shared__ float s_max[kFoldThreads / 32], s_half[2];
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.y, tid = threadIdx.x, part = blockIdx.x & 1;
    if ((int)blockIdx.x >= 2 * m.groups[i]) return;   // both CTAs of a cluster
    pair_ptx::cluster_arrive();                       // met ahead of the store into the other CTA: by then it runs
    const size_t at = (size_t)blockIdx.x * kFoldRows * kFoldCols + tid * 8;
    const __half* w = m.w[i] + at;
    Half8 raw[kFoldChunks];
#pragma unroll
    for (int k = 0; k < kFoldChunks; ++k) raw[k] = ldcs_half8(w + (size_t)k * kFoldThreads * 8);
    float g[8], mx = 0.0f;      // a thread keeps its columns: the threads walk whole rows
    ldg_float8(m.gamma[i] + tid * 8 % kFoldCols, g);
#pragma unroll
    for (int k = 0; k < kFoldChunks; ++k) {
        float v[8];
        unpack8(raw[k], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(v[j] * g[j]));
    }
    mx = warp_max(mx);
    if ((tid & 31) == 0) s_max[tid >> 5] = mx;
    __syncthreads();
    pair_ptx::cluster_wait();
    if (tid < 2) {              // into both CTAs
        for (int k = 0; k < kFoldThreads / 32; ++k) mx = fmaxf(mx, s_max[k]);
        const uint32_t to = pair_ptx::map_to_cta(tc::smem_addr(&s_half[part]), tid);
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(mx) : "memory");
    }
    __syncwarp();
    pair_ptx::cluster_arrive();
    pair_ptx::cluster_wait();
    mx = fmaxf(s_half[0], s_half[1]);
    const int e = (int)(__float_as_uint(mx) >> 23) + 1;   // biased exponent of the next power of two; 255, 256: not finite
    const float scale = mx > 0.0f && e < 255 ? __uint_as_float((uint32_t)min(max(e - 14, 27), 227) << 23) : 1.0f, by = 1.0f / scale;
    if (tid == 0 && part == 0) mul[m.first[i] + (blockIdx.x >> 1)] = scale;
    __half* o = out + (size_t)m.first[i] * 64 * kFoldCols + at;
#pragma unroll
    for (int k = 0; k < kFoldChunks; ++k) {
        float v[8];
        uint32_t* q = reinterpret_cast<uint32_t*>(&raw[k]);
        asm volatile("" : "+r"(q[0]), "+r"(q[1]), "+r"(q[2]), "+r"(q[3]));   // unpacked anew: all of them in fp32 are more than the registers
        unpack8(raw[k], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (v[j] * g[j]) * by;
        store8(o + (size_t)k * kFoldThreads * 8, v);
    }
}

// y = half(x + r) and the sums of its squares, added as gemm_folded's epilogues do: a scene's context rows, one CTA a row of 1024 (5665 rows
// 8.4 us, where the residual add and the cast took 16)
__global__ void __launch_bounds__(kRmsThreads)
context_rows_kernel(const float* __restrict__ x, const __half* __restrict__ r, __half* __restrict__ y, float* __restrict__ row_ss, int dim) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t at = (size_t)blockIdx.x * dim + threadIdx.x * 8;
    float v[8], c = 0.0f;
    ldcs_float8(x + at, v);
    if (r) {
        float a[8];
        unpack8(ldcs_half8(r + at), a);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += a[i];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = round_half(v[i]);
        c = fmaf(v[i], v[i], c);
    }
    store8(y + at, v);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    float sum = __shfl_sync(0xffffffffu, c, 0);
#pragma unroll
    for (int k = 1; k < 8; ++k) sum += __shfl_sync(0xffffffffu, c, 4 * k);
    if (lane == 0) row_ss[(size_t)blockIdx.x * (kRmsThreads / 32) + warp] = sum;
}

constexpr int kMaxKvLayers = 32;

// Bound: HBM, each key once in and once out. A thread takes its chunk of a row in four heads, whose sum it reads once.
struct KeyGammas { const float* gamma[kMaxKvLayers]; };
__global__ void __launch_bounds__(128)
keys_norm_kernel(__half* keys, long long layer_stride, const __grid_constant__ KeyGammas m, const float* __restrict__ row_ss, int rows, int out_seq,
                 int num_heads, int head_dim, float inv_dim, float eps) {
    constexpr int UN = 4;
    pdl_wait();
    pdl_trigger();
    const int cpr = head_dim / 8, idx = blockIdx.x * 128 + threadIdx.x, s = idx / cpr, c = idx % cpr;
    const int groups = num_heads / UN, layer = blockIdx.y / groups, h0 = (blockIdx.y % groups) * UN;
    if (s >= rows) return;
    __half* at = keys + (size_t)layer * layer_stride + ((size_t)h0 * out_seq + s) * head_dim + c * 8;
    Half8 v[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) v[u] = ldcs_half8(at + (size_t)u * out_seq * head_dim);
    const float4 a = __ldg(reinterpret_cast<const float4*>(row_ss) + (size_t)(2 * layer) * rows + s);
    const float rinv = rsqrtf((((a.x + a.y) + a.z) + a.w) * inv_dim + eps);
#pragma unroll
    for (int u = 0; u < UN; ++u) {
        float f[8], g[8];
        unpack8(v[u], f);
        ldg_float8(m.gamma[layer] + (h0 + u) * head_dim + c * 8, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = (f[i] * rinv) * g[i];
        store8(at + (size_t)u * out_seq * head_dim, f);
    }
}

// Any dim / any alignment: one CTA per row, scalar accesses, the row is re-read.
template <typename TH, typename TR, typename TY, bool HAS_RES, bool WRITE_H>
__global__ void __launch_bounds__(256)
rmsnorm_generic_kernel(const TH* x, TH* xw, const TR* __restrict__ r,
                       const float* __restrict__ gamma, TY* y, int dim, float eps) {
    pdl_wait();
    pdl_trigger();
    __shared__ float red[8];
    const size_t base = (size_t)blockIdx.x * dim;
    auto value = [&](int i) -> float {
        float s = (float)x[base + i];
        if (HAS_RES) {
            s += (float)r[base + i];
            if (IsHalf<TH>::value) s = round_half(s);
        }
        return s;
    };
    float ss = 0.0f;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        float s = value(i);
        ss = fmaf(s, s, ss);
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) tot += red[w];
    const float rinv = rsqrtf(tot / (float)dim + eps);
    // every thread re-reads exactly the elements it will overwrite, so y == x is safe
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        float s = value(i);
        if (HAS_RES && WRITE_H) xw[base + i] = (TH)s;
        y[base + i] = (TY)((s * rinv) * gamma[i]);
    }
}

// Whether fp16 rows of 513 to 1024 elements go to one warp each (four chunks per lane) instead of four warps, with the same bits. With
// four, 4096 rows are 1.7 rounds of CTAs of which each waits once for memory; with one, a single round that has four times the
// loads in flight - but loads all it loads before it stores anything, which costs where a residual and x come from and go back to HBM.
// So with a residual only the layers' own call asks for it, whose operands the kernels before have just written. Measured (us, four
// warps / one, 1024 wide; operands in L2, then from HBM):
//   plain             2304 rows 2.71 / 2.66, 3.23 / 3.30; 3136 rows 3.68 / 4.04, 4.31 / 4.71; 4096 rows 4.61 / 3.99, 4.96 / 4.86; 16384 rows
//                     17.5 / 10.0, 17.5 / 12.4 (768 wide at 2304 rows 2.71 / 2.40, 2.87 / 3.40)
//   with residual     4096 rows 4.86 / 5.38, 6.76 / 8.24; 8192 rows 9.21 / 8.90, 11.7 / 14.5: never
//   to windows        1024 rows 2.7 / 2.9; 1600 rows 4.14 / 3.02, 4.59 / 3.72; 4096 rows 6.50 / 4.61, 7.06 / 5.53; 16384 rows 22.2 / 11.4, 22.6 / 14.4
//   windows, residual 1600 rows 4.71 / 3.89, 5.12 / 6.45; 4096 rows 7.42 / 5.84, 8.09 / 8.75; 8192 rows 13.3 / 9.5, 14.0 / 15.3; 16384 rows, 134 MB
//                     of traffic and more than L2, 25.5 / 26.7
static bool one_warp_per_row(int rows, int dim, bool windows, bool residual, bool in_l2) {
    if (dim <= 512 || dim > 1024) return false;
    if (residual && (!windows || !in_l2 || (long long)rows * dim * 8 > (96ll << 20))) return false;
    return rows >= (windows ? 1280 : 4096);
}

template <typename TH, typename TR, typename TY, bool HAS_RES, bool WRITE_H>
static int launch_variant(const TH* x, TH* xw, const TR* r, const float* gamma, TY* y,
                          int rows, int dim, float eps, cudaStream_t st) {
    const bool vec = (dim % 8 == 0) && dim <= 2048 && aligned16(x) && aligned16(y) &&
                     aligned16(gamma) && (!HAS_RES || aligned16(r)) &&
                     (!WRITE_H || aligned16(xw));
    if (vec) {
#define RFK_RMS_LAUNCH(N, WW)                                                                         \
    launch_pdl(rmsnorm_row_kernel<TH, TR, TY, N, WW, HAS_RES, WRITE_H, 0>,                             \
               dim3(ceil_div(rows, (kRmsThreads / 32) / WW)), dim3(kRmsThreads), 0, st, x, xw, r, gamma, y, \
               rows, dim, eps, WinRows{})
        if constexpr (IsHalf<TH>::value && IsHalf<TY>::value && !HAS_RES) {
            if (one_warp_per_row(rows, dim, false, false, false)) {
                launch_pdl(rmsnorm_row_kernel<TH, TR, TY, 4, 1, false, WRITE_H, 0, 4>, dim3(ceil_div(rows, kRmsThreads / 32)), dim3(kRmsThreads),
                           0, st, x, xw, r, gamma, y, rows, dim, eps, WinRows{});
                return launch_status();
            }
        }
        if (dim <= 256) RFK_RMS_LAUNCH(1, 1);
        else if (dim <= 512) RFK_RMS_LAUNCH(1, 2);
        else if (dim <= 1024) RFK_RMS_LAUNCH(1, 4);
        else RFK_RMS_LAUNCH(2, 4);
#undef RFK_RMS_LAUNCH
    } else {
        launch_pdl(rmsnorm_generic_kernel<TH, TR, TY, HAS_RES, WRITE_H>, dim3(rows), dim3(256), 0, st,
            x, xw, r, gamma, y, dim, eps);
    }
    return launch_status();
}

template <typename TH, typename TR, typename TY>
static int launch_rmsnorm(const TH* x, TH* xw, const TR* r, const float* gamma, TY* y,
                          int rows, int dim, float eps, cudaStream_t st) {
    if (!x || !gamma || !y || rows < 0 || dim <= 0) return RFK_EINVAL;
    if (rows == 0) return RFK_OK;
    if (r) return launch_variant<TH, TR, TY, true, true>(x, xw, r, gamma, y, rows, dim, eps, st);
    return launch_variant<TH, TR, TY, false, false>(x, xw, r, gamma, y, rows, dim, eps, st);
}

int norm_pair_add(const rfk_half* a, const float* gamma_a, const rfk_half* b, const float* gamma_b, const rfk_half* c, float* out,
                  int rows, int dim, float eps, rfk_stream_t stream) {
    if (!a || !gamma_a || !b || !gamma_b || !c || !out || rows < 0 || dim <= 0) return RFK_EINVAL;
    if (dim % 8 || dim > 1024 || !aligned16(a) || !aligned16(gamma_a) || !aligned16(b) || !aligned16(gamma_b) || !aligned16(c) || !aligned16(out))
        return RFK_EUNSUPPORTED;
    if (rows == 0) return RFK_OK;
    const int w = dim <= 256 ? 1 : dim <= 512 ? 2 : 4;
    launch_pdl(w == 1 ? norm_pair_add_kernel<1> : w == 2 ? norm_pair_add_kernel<2> : norm_pair_add_kernel<4>,
               dim3(ceil_div(rows, (kRmsThreads / 32) / w)), dim3(kRmsThreads), 0, as_stream(stream), (const __half*)a, gamma_a,
               (const __half*)b, gamma_b, (const __half*)c, out, rows, dim, eps);
    return launch_status();
}

int embed_tokens(const rfk_half* e, const float* gamma, const rfk_half* token, rfk_half* x, float* row_ss, int rows, int dim, float eps,
                 int blocks_across, int blocks_down, rfk_stream_t stream) {
    if (!e || !gamma || !token || !x || !row_ss || rows < 0 || blocks_across <= 0 || blocks_down <= 0) return RFK_EINVAL;
    if (dim != 256 * (kRmsThreads / 32) || !aligned16(e) || !aligned16(gamma) || !aligned16(token) || !aligned16(x) || blocks_across % 2 ||
        blocks_down % 2 || rows % (blocks_across * blocks_down * 16))
        return RFK_EUNSUPPORTED;
    if (rows == 0) return RFK_OK;
    launch_pdl(embed_tokens_kernel, dim3(rows), dim3(kRmsThreads), 0, as_stream(stream), (const __half*)e, gamma, (const __half*)token, (__half*)x,
               row_ss, dim, eps, blocks_across, blocks_down);
    return launch_status();
}

int context_rows(const float* x, const rfk_half* r, rfk_half* y, float* row_ss, int rows, int dim, rfk_stream_t stream) {
    if (!x || !y || !row_ss || rows < 0) return RFK_EINVAL;
    if (dim != 256 * (kRmsThreads / 32) || !aligned16(x) || !aligned16(r) || !aligned16(y)) return RFK_EUNSUPPORTED;
    if (rows == 0) return RFK_OK;
    launch_pdl(context_rows_kernel, dim3(rows), dim3(kRmsThreads), 0, as_stream(stream), x, (const __half*)r, (__half*)y, row_ss, dim);
    return launch_status();
}

int keys_norm(rfk_half* keys, long long layer_stride, const float* const* gamma, const float* row_ss, int layers, int rows, int out_seq, int num_heads,
              int head_dim, float eps, rfk_stream_t stream) {
    if (!keys || !gamma || !row_ss || layers <= 0 || rows < 0 || out_seq < rows || num_heads <= 0 || head_dim <= 0) return RFK_EINVAL;
    if (num_heads * head_dim != 1024 || num_heads % 4 || head_dim % 8 || layers > kMaxKvLayers || !aligned16(keys) || layer_stride % 8 ||
        !aligned16(row_ss))
        return RFK_EUNSUPPORTED;
    KeyGammas m{};
    for (int i = 0; i < layers; ++i) {
        if (!gamma[i]) return RFK_EINVAL;
        if (!aligned16(gamma[i])) return RFK_EUNSUPPORTED;
        m.gamma[i] = gamma[i];
    }
    if (rows == 0) return RFK_OK;
    launch_pdl(keys_norm_kernel, dim3(ceil_div((long long)rows * (head_dim / 8), 128), layers * (num_heads / 4)), dim3(128), 0, as_stream(stream),
               (__half*)keys, layer_stride, m, row_ss, rows, out_seq, num_heads, head_dim, 1.0f / (float)(num_heads * head_dim), eps);
    return launch_status();
}

int fold_weights(const rfk_half* const* w, const float* const* gamma, const int* rows, int n, int cols, rfk_half* out, float* mul, rfk_stream_t stream) {
    if (!w || !gamma || !rows || !out || !mul || n < 1 || cols <= 0) return RFK_EINVAL;
    if (cols != kFoldCols || n > kMaxFolded || !aligned16(out)) return RFK_EUNSUPPORTED;
    FoldList m{};
    int groups = 0, most = 0;
    for (int i = 0; i < n; ++i) {
        if (!w[i] || !gamma[i] || rows[i] <= 0) return RFK_EINVAL;
        if (!aligned16(w[i]) || !aligned16(gamma[i]) || rows[i] % 64) return RFK_EUNSUPPORTED;
        m.w[i] = (const __half*)w[i]; m.gamma[i] = gamma[i]; m.first[i] = groups; m.groups[i] = rows[i] / 64;
        groups += m.groups[i];
        most = std::max(most, m.groups[i]);
    }
    launch_pdl(fold_weights_kernel, dim3(2 * most, n), dim3(kFoldThreads), 0, as_stream(stream), m, (__half*)out, mul);
    return launch_status();
}

}  // namespace rfk

using namespace rfk;

extern "C" int rfk_embed_tokens(const rfk_half* e, const float* gamma, const rfk_half* token, rfk_half* x, float* row_ss, int rows, int dim, float eps,
                                int blocks_across, int blocks_down, rfk_stream_t stream) {
    return embed_tokens(e, gamma, token, x, row_ss, rows, dim, eps, blocks_across, blocks_down, stream);
}

extern "C" int rfk_fold_weights(const rfk_half* const* w, const float* const* gamma, const int* rows, int n, int cols, rfk_half* out, float* mul,
                                rfk_stream_t stream) {
    return fold_weights(w, gamma, rows, n, cols, out, mul, stream);
}

extern "C" int rfk_norm_pair_add(const rfk_half* a, const float* gamma_a, const rfk_half* b, const float* gamma_b, const rfk_half* c,
                                 float* out, int rows, int dim, float eps, rfk_stream_t stream) {
    return norm_pair_add(a, gamma_a, b, gamma_b, c, out, rows, dim, eps, stream);
}

extern "C" int rfk_rmsnorm(const rfk_half* x, const float* gamma, rfk_half* y, int rows, int dim,
                           float eps, rfk_stream_t stream) {
    return launch_rmsnorm<__half, __half, __half>((const __half*)x, nullptr, nullptr, gamma,
                                                  (__half*)y, rows, dim, eps, as_stream(stream));
}

extern "C" int rfk_rmsnorm_f32(const float* x, const float* gamma, float* y, int rows, int dim,
                               float eps, rfk_stream_t stream) {
    return launch_rmsnorm<float, float, float>(x, nullptr, nullptr, gamma, y, rows, dim, eps,
                                               as_stream(stream));
}

extern "C" int rfk_rmsnorm_residual_f32_cast16(float* h, const float* r, const float* gamma,
                                               rfk_half* y16, int rows, int dim, float eps,
                                               rfk_stream_t stream) {
    return launch_rmsnorm<float, float, __half>(h, h, r, gamma, (__half*)y16, rows, dim, eps,
                                                as_stream(stream));
}

extern "C" int rfk_rmsnorm_residual_mixed_cast16(float* h, const rfk_half* r, const float* gamma,
                                                 rfk_half* y16, int rows, int dim, float eps,
                                                 rfk_stream_t stream) {
    return launch_rmsnorm<float, __half, __half>(h, h, (const __half*)r, gamma, (__half*)y16, rows,
                                                 dim, eps, as_stream(stream));
}

static int rmsnorm_windows(rfk_half* x, const rfk_half* r, const float* gamma, rfk_half* y, int B, int H, int W, int dim, int window_size,
                           int shift_size, int windowed_operand, float eps, bool in_l2, rfk_stream_t stream) {
    if (!x || !gamma || !y || B < 0 || H <= 0 || W <= 0 || dim <= 0) return RFK_EINVAL;
    if (window_size <= 0 || H % window_size || W % window_size || shift_size < 0) return RFK_EINVAL;
    if (windowed_operand != 1 && windowed_operand != 2) return RFK_EINVAL;
    if (!r && windowed_operand != 1) return RFK_EINVAL;  // without a residual only the output can be in window order
    if ((const void*)x == (const void*)y || (r && (const void*)r == (const void*)y)) return RFK_EINVAL;
    if (dim % 8 != 0 || dim > 2048 || !aligned16(x) || !aligned16(y) || !aligned16(gamma) || (r && !aligned16(r)))
        return RFK_EUNSUPPORTED;
    const long long rows_ll = (long long)B * H * W;
    if (rows_ll > 0x7fffffffLL) return RFK_EUNSUPPORTED;
    const int rows = (int)rows_ll;
    if (rows == 0) return RFK_OK;
    const WinRows wr{H, W, window_size, shift_size};
    cudaStream_t st = as_stream(stream);
    __half* xh = (__half*)x;
#define RFK_RMS_WIN(N, WW, M, SUMS)                                                                             \
    if (r)                                                                                                      \
        launch_pdl(rmsnorm_row_kernel<__half, __half, __half, N, WW, true, true, M, SUMS>,                       \
                   dim3(ceil_div(rows, (kRmsThreads / 32) / WW)), dim3(kRmsThreads), 0, st, (const __half*)xh, xh, \
                   (const __half*)r, gamma, (__half*)y, rows, dim, eps, wr);                                     \
    else                                                                                                        \
        launch_pdl(rmsnorm_row_kernel<__half, __half, __half, N, WW, false, false, 1, SUMS>,                     \
                   dim3(ceil_div(rows, (kRmsThreads / 32) / WW)), dim3(kRmsThreads), 0, st, (const __half*)xh, xh, \
                   (const __half*)nullptr, gamma, (__half*)y, rows, dim, eps, wr)
#define RFK_RMS_WIN_DIM(M)                               \
    if (one_warp_per_row(rows, dim, true, r != nullptr, in_l2)) { RFK_RMS_WIN(4, 1, M, 4); } \
    else if (dim <= 256) { RFK_RMS_WIN(1, 1, M, 1); }    \
    else if (dim <= 512) { RFK_RMS_WIN(1, 2, M, 1); }    \
    else if (dim <= 1024) { RFK_RMS_WIN(1, 4, M, 1); }   \
    else { RFK_RMS_WIN(2, 4, M, 1); }
    if (windowed_operand == 1) { RFK_RMS_WIN_DIM(1); } else { RFK_RMS_WIN_DIM(2); }
#undef RFK_RMS_WIN_DIM
#undef RFK_RMS_WIN
    return launch_status();
}

extern "C" int rfk_rmsnorm_residual_f16_windows(rfk_half* x, const rfk_half* r, const float* gamma,
                                                rfk_half* y, int B, int H, int W, int dim,
                                                int window_size, int shift_size, int windowed_operand,
                                                float eps, rfk_stream_t stream) {
    return rmsnorm_windows(x, r, gamma, y, B, H, W, dim, window_size, shift_size, windowed_operand, eps, false, stream);
}

extern "C" int rfk_rmsnorm_residual_f16_windows_in_l2(rfk_half* x, const rfk_half* r, const float* gamma, rfk_half* y, int B, int H, int W,
                                                      int dim, int window_size, int shift_size, int windowed_operand, float eps,
                                                      rfk_stream_t stream) {
    return rmsnorm_windows(x, r, gamma, y, B, H, W, dim, window_size, shift_size, windowed_operand, eps, true, stream);
}

extern "C" int rfk_rmsnorm_residual_f16(rfk_half* x, const rfk_half* r, const float* gamma,
                                        rfk_half* y, int rows, int dim, float eps,
                                        rfk_stream_t stream) {
    if (r && (const void*)x == (const void*)y) return RFK_EINVAL;
    return launch_rmsnorm<__half, __half, __half>((const __half*)x, (__half*)x, (const __half*)r,
                                                  gamma, (__half*)y, rows, dim, eps,
                                                  as_stream(stream));
}
