// Triangle-vertex RoPE: table generation, rotate-half application (in place and out of
// place), and the fused projection epilogue (QK-RMSNorm + BSHD->BHSD transpose + RoPE).
//
// Reference semantics (BANANASJIM/renderformer-cuda, src/kernels/rope.cu):
//   :23-43  tables: l = d mod (hd/2); theta = l < 9*nf ? pos[l / nf] * freq[l mod nf] : 0;
//           cos_d = half(cosf(theta)), sin_d = half(sinf(theta))
//   :75-88  apply: out_d = x_d*c_d + (x_rot*sign)*s_d, rot = d +- hd/2, sign = -1 for d < hd/2
// and src/layers/attention.cu:73-85,184-210,341-361 for the sequence the fused epilogue
// replaces.
//
// Design: the reference assigns one thread per element; both partners of a rotation
// pair are read by two different threads and written in place without ordering. Here
// one thread owns the 8-wide chunk d..d+7 of the first half of a head and the matching
// chunk of the second half, so each element is read once (two 128-bit loads), written
// once, and the in-place update is race-free by construction. The cos/sin chunk is
// loaded once per thread and reused across the heads the thread walks.
#include <algorithm>
#include "common.cuh"
#include "kernels_internal.h"

namespace rfk {

// ---------------------------------------------------------------- tables

// thread -> (token, chunk of PER angles of the first half); writes both halves (they are equal). One scene's tables are short work
// of a long dependent chain each (cosf and sinf with their reductions), so what counts is how many run side by side: with eight
// angles a thread the tables of 5633 triangles took 3.6 us, with two 2.2 (301 triangles 3.4 and 1.9; 64-wide heads). Eight keep
// the wider stores where threads abound (eight / two angles, 64-wide heads): 55000 triangles, 0.88 million threads of two, 9.8 / 8.8 us;
// 70000, 1.12 million, 9.9 / 10.9; 140000 17.0 / 20.3; 45000 with 128-wide heads, 1.44 million, 11.9 / 13.5.
template <int PER>
__global__ void __launch_bounds__(256)
rope_table_vec_kernel(const __half* __restrict__ pos, const float* __restrict__ freqs,
                      __half* __restrict__ out_cos, __half* __restrict__ out_sin,
                      long long tokens, int num_freqs, int head_dim) {
    pdl_wait();
    pdl_trigger();
    const int cpt = head_dim / (2 * PER);  // chunks per token (first half)
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= tokens * cpt) return;
    const long long tok = idx / cpt;
    const int j = (int)(idx % cpt);
    const int freq_dim = 9 * num_freqs;
    float c[PER], s[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int l = j * PER + i;
        float val = 0.0f;
        if (l < freq_dim) {
            const float p = __half2float(pos[tok * 9 + l / num_freqs]);
            val = p * __ldg(freqs + l % num_freqs);
        }
        c[i] = cosf(val);
        s[i] = sinf(val);
    }
    const size_t o = (size_t)tok * head_dim + j * PER;
    store_twice(out_cos + o, c, head_dim / 2);
    store_twice(out_sin + o, s, head_dim / 2);
}

__global__ void __launch_bounds__(256)
rope_table_generic_kernel(const __half* __restrict__ pos, const float* __restrict__ freqs,
                          __half* __restrict__ out_cos, __half* __restrict__ out_sin,
                          long long tokens, int num_freqs, int head_dim) {
    pdl_wait();
    pdl_trigger();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= tokens * head_dim) return;
    const long long tok = idx / head_dim;
    const int d = (int)(idx % head_dim);
    const int l = d % (head_dim / 2);
    float val = 0.0f;
    if (l < 9 * num_freqs)
        val = __half2float(pos[tok * 9 + l / num_freqs]) * freqs[l % num_freqs];
    out_cos[idx] = __float2half(cosf(val));
    out_sin[idx] = __float2half(sinf(val));
}

// ---------------------------------------------------------------- apply

// rotate one (lo, hi) chunk pair; c/s are the table chunks at the lo and hi positions
__device__ __forceinline__ void rotate8(float (&lo)[8], float (&hi)[8], const float (&cl)[8],
                                        const float (&sl)[8], const float (&ch)[8],
                                        const float (&sh)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float x_lo = lo[i], x_hi = hi[i];
        const float rot_lo = x_hi * -1.0f;  // partner of a first-half element, sign -1
        const float rot_hi = x_lo * 1.0f;
        lo[i] = x_lo * cl[i] + rot_lo * sl[i];
        hi[i] = x_hi * ch[i] + rot_hi * sh[i];
    }
}

// Eight elements as they lie in memory.
template <typename T> struct Raw8;
template <> struct Raw8<__half> {
    Half8 h;
    __device__ __forceinline__ void load(const __half* p) { h = ld_half8(p); }
    __device__ __forceinline__ void unpack(float (&f)[8]) const { unpack8(h, f); }
};
template <> struct Raw8<float> {
    float v[8];
    __device__ __forceinline__ void load(const float* p) { ld_float8(p, v); }
    __device__ __forceinline__ void unpack(float (&f)[8]) const {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = v[i];
    }
};

// The row and chunk of a thread: thread idx of `cpt` chunks a row.
__device__ __forceinline__ bool row_and_chunk(int cpt, long long rows, long long& s, int& j) {
    if (rows * cpt <= 0x7fffffffLL) {
        const unsigned idx = blockIdx.x * blockDim.x + threadIdx.x;
        s = idx / (unsigned)cpt;
        j = (int)(idx % (unsigned)cpt);
    } else {
        const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        s = idx / cpt;
        j = (int)(idx % cpt);
    }
    return s < rows;
}

// T = __half or float data. NT tensors (1 or 2) share the tables. src/dst are [B,H,src_rows,D] / [B,H,dst_rows,D]; rows s >= seq_len
// (dst only) are copied. PLAIN: no such rows, no col_scale.
// Bound: HBM. A thread has one chunk pair of one head (blockIdx.y, z) of each tensor, and asks for everything it needs before it stores
// anything: source and destination may be the same, so the compiler keeps a load behind a store that comes before it, and a thread
// that went from one tensor to the other waited for memory twice. Q and K of 5633 triangles, 47 MB, us from HBM / from L2: 16 heads of 64 11.6 / 9.5
// that way, 8.5 / 7.6 now (5.5 TB/s); 8 heads of 128 12.1 / 8.9, now 8.9 / 6.3; eight scenes (380 MB) 78, now 58; 60 triangles 2.3, now 1.9. Several heads a
// thread, which read the tables less often, take 8.8 (two) and 10.8 (four), 256 threads a CTA 9.4.
template <typename T, int NT, bool PLAIN>
__global__ void __launch_bounds__(128)
rope_apply_kernel(const T* src0, T* dst0, const T* src1, T* dst1,
                  const __half* __restrict__ cos_vals, const __half* __restrict__ sin_vals,
                  int num_heads, long long heads_total, int seq_len, int rows_total, int head_dim,
                  long long src_rows, long long dst_rows, long long src_bstride, long long dst_bstride,
                  long long tab_bstride, const float* __restrict__ col_scale, long long scale_bstride) {
    pdl_wait();
    pdl_trigger();
    const int half_d = head_dim / 2;
    long long s;
    int j;
    int b = blockIdx.z, h = blockIdx.y;
    if (heads_total) {   // more heads or batches than a grid has blocks that way: both in y and z
        const long long bh = (long long)blockIdx.z * gridDim.y + blockIdx.y;
        if (bh >= heads_total) return;
        b = (int)(bh / num_heads);
        h = (int)(bh % num_heads);
    }
    if (!row_and_chunk(head_dim / 16, rows_total, s, j)) return;
    const size_t so = (size_t)b * src_bstride + ((size_t)h * src_rows + s) * head_dim + j * 8;
    const size_t dofs = (size_t)b * dst_bstride + ((size_t)h * dst_rows + s) * head_dim + j * 8;
    Raw8<T> lo8[NT], hi8[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const T* sp = (n == 0 ? src0 : src1) + so;
        lo8[n].load(sp);
        hi8[n].load(sp + half_d);
    }
    const bool rotate = PLAIN || s < seq_len;
    float cl[8], sl[8], ch[8], sh[8];
    if (rotate) {
        const size_t to = (size_t)b * tab_bstride + (size_t)s * head_dim + j * 8;
        const Half8 t0 = ldg_half8(cos_vals + to), t1 = ldg_half8(sin_vals + to), t2 = ldg_half8(cos_vals + to + half_d),
                    t3 = ldg_half8(sin_vals + to + half_d);
        unpack8(t0, cl); unpack8(t1, sl); unpack8(t2, ch); unpack8(t3, sh);
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        float lo[8], hi[8];
        lo8[n].unpack(lo);
        hi8[n].unpack(hi);
        if (rotate) rotate8(lo, hi, cl, sl, ch, sh);
        if (!PLAIN && col_scale) {  // per-(head, element) factor applied to the rotated value before the one rounding
            float g0[8], g1[8];
            const float* gs = col_scale + (size_t)b * scale_bstride + (size_t)h * head_dim + j * 8;
            ldg_float8(gs, g0);
            ldg_float8(gs + half_d, g1);
#pragma unroll
            for (int i = 0; i < 8; ++i) { lo[i] *= g0[i]; hi[i] *= g1[i]; }
        }
        T* dp = (n == 0 ? dst0 : dst1) + dofs;
        store8(dp, lo);
        store8(dp + half_d, hi);
    }
}

// The cached keys of several layers by one view's tables, out of place: batches of one tensor that share a table. A thread keeps its part of the
// tables in registers and walks pairs of heads over all batches, four loads in flight; the stores leave the L2 to others (STREAM)
// where the result is longer than half of it. Twelve layers, 16 heads of 64, us warm / cold, a thread per four heads of a layer (which read the tables
// again for each four) and now: 5672 rows (279 MB) 68.8 / 69.9, 52.5 / 57.7; 7232 rows 88.9 / 91.1, 66.1 / 74.0; 1536 rows 19.9 / 22.0, 14.9 / 18.8;
// 336 rows 6.6 / 7.0, 6.0 / 7.0. Some 2400 CTAs are enough: 600 to 9600 are within 5 %, 300 take 40 % longer.
template <bool STREAM>
__global__ void __launch_bounds__(128)
rope_shared_table_kernel(const __half* src, __half* dst, const __half* __restrict__ cos_vals, const __half* __restrict__ sin_vals,
                         int pairs, long long pairs_total, int rows, int head_dim, long long src_rows, long long dst_rows,
                         long long src_bstride, long long dst_bstride, const float* __restrict__ col_scale, long long scale_bstride) {
    constexpr int UN = 2;
    pdl_wait();
    pdl_trigger();
    const int half_d = head_dim / 2;
    long long s;
    int j;
    if (!row_and_chunk(head_dim / 16, rows, s, j)) return;
    const size_t at = (size_t)s * head_dim + j * 8;
    float cl[8], sl[8], ch[8], sh[8];
    unpack8(ldg_half8(cos_vals + at), cl);
    unpack8(ldg_half8(sin_vals + at), sl);
    unpack8(ldg_half8(cos_vals + at + half_d), ch);
    unpack8(ldg_half8(sin_vals + at + half_d), sh);
    for (long long g = blockIdx.y; g < pairs_total; g += gridDim.y) {
        const int b = (int)(g / pairs), h0 = (int)(g % pairs) * UN;
        const __half* sp = src + (size_t)b * src_bstride + (size_t)h0 * src_rows * head_dim + at;
        __half* dp = dst + (size_t)b * dst_bstride + (size_t)h0 * dst_rows * head_dim + at;
        Half8 lo8[UN], hi8[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            lo8[u] = ldcs_half8(sp + (size_t)u * src_rows * head_dim);
            hi8[u] = ldcs_half8(sp + (size_t)u * src_rows * head_dim + half_d);
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            float lo[8], hi[8];
            unpack8(lo8[u], lo);
            unpack8(hi8[u], hi);
            rotate8(lo, hi, cl, sl, ch, sh);
            if (col_scale) {
                const float* gs = col_scale + (size_t)b * scale_bstride + (size_t)(h0 + u) * head_dim + j * 8;
                float g0[8], g1[8];
                ldg_float8(gs, g0);
                ldg_float8(gs + half_d, g1);
#pragma unroll
                for (int i = 0; i < 8; ++i) { lo[i] *= g0[i]; hi[i] *= g1[i]; }
            }
            __half* d = dp + (size_t)u * dst_rows * head_dim;
            if (STREAM) {
                stcs_half8(d, pack8(lo));
                stcs_half8(d + half_d, pack8(hi));
            } else {
                store8(d, lo);
                store8(d + half_d, hi);
            }
        }
    }
}

// head_dim not a multiple of 16 (but even): one thread per rotation pair, scalar accesses.
template <typename T, int NT>
__global__ void __launch_bounds__(256)
rope_apply_generic_kernel(const T* src0, T* dst0, const T* src1, T* dst1,
                          const __half* __restrict__ cos_vals,
                          const __half* __restrict__ sin_vals, int batch, int num_heads,
                          int seq_len, int rows_total, int head_dim, long long src_rows,
                          long long dst_rows, long long src_bstride, long long dst_bstride,
                          long long tab_bstride) {
    pdl_wait();
    pdl_trigger();
    const int half_d = head_dim / 2;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long total = (long long)batch * num_heads * rows_total * half_d;
    if (idx >= total) return;
    const int d = (int)(idx % half_d);
    long long t = idx / half_d;
    const int s = (int)(t % rows_total);
    t /= rows_total;
    const int h = (int)(t % num_heads);
    const int b = (int)(t / num_heads);
    const size_t so = (size_t)b * src_bstride + ((size_t)h * src_rows + s) * head_dim + d;
    const size_t dofs = (size_t)b * dst_bstride + ((size_t)h * dst_rows + s) * head_dim + d;
#pragma unroll
    for (int tsel = 0; tsel < NT; ++tsel) {
        const T* sp = tsel == 0 ? src0 : src1;
        T* dp = tsel == 0 ? dst0 : dst1;
        float x_lo = (float)sp[so], x_hi = (float)sp[so + half_d];
        float o_lo = x_lo, o_hi = x_hi;
        if (s < seq_len) {
            const size_t to = (size_t)b * tab_bstride + (size_t)s * head_dim + d;
            const float c_lo = __half2float(cos_vals[to]), s_lo = __half2float(sin_vals[to]);
            const float c_hi = __half2float(cos_vals[to + half_d]);
            const float s_hi = __half2float(sin_vals[to + half_d]);
            o_lo = x_lo * c_lo + (x_hi * -1.0f) * s_lo;
            o_hi = x_hi * c_hi + (x_lo * 1.0f) * s_hi;
        }
        dp[dofs] = (T)o_lo;
        dp[dofs + half_d] = (T)o_hi;
    }
}

template <typename T, int NT>
static int launch_rope(const T* src0, T* dst0, const T* src1, T* dst1, const __half* cos_vals,
                       const __half* sin_vals, int batch, int num_heads, int seq_len,
                       int rows_total, int head_dim, long long src_rows, long long dst_rows,
                       cudaStream_t st, long long src_bstride = -1, long long dst_bstride = -1,
                       long long tab_bstride = -1, const float* col_scale = nullptr, long long scale_bstride = 0) {
    // batch strides in elements; by default the tensors and the tables are densely packed
    if (src_bstride < 0) src_bstride = (long long)num_heads * src_rows * head_dim;
    if (dst_bstride < 0) dst_bstride = (long long)num_heads * dst_rows * head_dim;
    if (tab_bstride < 0) tab_bstride = (long long)seq_len * head_dim;
    if (!src0 || !dst0 || (NT == 2 && (!src1 || !dst1)) || !cos_vals || !sin_vals)
        return RFK_EINVAL;
    if (batch < 0 || num_heads <= 0 || seq_len < 0 || head_dim <= 0 || (head_dim & 1))
        return RFK_EINVAL;
    if (rows_total < seq_len || src_rows < rows_total || dst_rows < rows_total) return RFK_EINVAL;
    if (batch == 0 || rows_total == 0) return RFK_OK;
    if constexpr (NT == 2) {
        if (dst0 == dst1) {   // one tensor given twice is rotated twice: the second time from what the first has left
            const int rc = launch_rope<T, 1>(src0, dst0, nullptr, nullptr, cos_vals, sin_vals, batch, num_heads, seq_len, rows_total, head_dim, src_rows, dst_rows, st,
                                             src_bstride, dst_bstride, tab_bstride, col_scale, scale_bstride);
            return rc != RFK_OK ? rc : launch_rope<T, 1>(src1, dst1, nullptr, nullptr, cos_vals, sin_vals, batch, num_heads, seq_len, rows_total, head_dim,
                                                         src_rows, dst_rows, st, src_bstride, dst_bstride, tab_bstride, col_scale, scale_bstride);
        }
    }
    const bool vec = head_dim % 16 == 0 && aligned16(src0) && aligned16(dst0) &&
                     (NT == 1 || (aligned16(src1) && aligned16(dst1))) && aligned16(cos_vals) &&
                     aligned16(sin_vals) && src_bstride % 8 == 0 && dst_bstride % 8 == 0 &&
                     tab_bstride % 8 == 0 && (!col_scale || (aligned16(col_scale) && scale_bstride % 4 == 0));
    if (col_scale && !vec) return RFK_EUNSUPPORTED;  // the scaled form exists in the vector kernel only
    if (vec) {
        const unsigned blocks = ceil_div((long long)rows_total * (head_dim / 16), 128);
        const long long heads_total = (long long)batch * num_heads;
        if constexpr (NT == 1 && sizeof(T) == 2) {
            if (src0 != dst0 && batch > 1 && tab_bstride == 0 && seq_len == rows_total && num_heads % 2 == 0) {
                const long long pairs_total = heads_total / 2;
                const unsigned split = (unsigned)std::min<long long>({pairs_total, 65535, (long long)ceil_div(2400, blocks)});
                const bool out_of_l2 = heads_total * rows_total * head_dim * 2 > (63ll << 20);
                launch_pdl(out_of_l2 ? rope_shared_table_kernel<true> : rope_shared_table_kernel<false>, dim3(blocks, split), dim3(128), 0, st,
                           src0, dst0, cos_vals, sin_vals, num_heads / 2, pairs_total, rows_total, head_dim, src_rows, dst_rows,
                           src_bstride, dst_bstride, col_scale, scale_bstride);
                return launch_status();
            }
        }
        const bool flat = num_heads > 65535 || batch > 65535;
        const unsigned gy = flat ? 65535u : num_heads, gz = flat ? ceil_div(heads_total, 65535) : batch;
        launch_pdl(seq_len == rows_total && !col_scale ? rope_apply_kernel<T, NT, true> : rope_apply_kernel<T, NT, false>, dim3(blocks, gy, gz), dim3(128), 0, st, src0, dst0, src1, dst1, cos_vals, sin_vals,
                   num_heads, flat ? heads_total : 0, seq_len, rows_total, head_dim, src_rows, dst_rows, src_bstride, dst_bstride,
                   tab_bstride, col_scale, scale_bstride);
    } else {
        const long long total = (long long)batch * num_heads * rows_total * (head_dim / 2);
        launch_pdl(rope_apply_generic_kernel<T, NT>, dim3(ceil_div(total, 256)), dim3(256), 0, st,
            src0, dst0, src1, dst1, cos_vals, sin_vals, batch, num_heads, seq_len, rows_total,
            head_dim, src_rows, dst_rows, src_bstride, dst_bstride, tab_bstride);
    }
    return launch_status();
}

// ------------------------------------------- fused projection epilogue

struct QkvParts {
    const float* gamma[3];
    __half* out[3];
    int use_rope[3];
};

// WPR warps per token row and part, 4 warps per CTA. A thread owns rotation-pair chunks
// p = t + 32 * WPR * k (t = its index within the row's threads) of the dim/16 pairs in the row:
// head h = p / (D/16), chunk j = p % (D/16). With WPR > 1 the sum of squares crosses the warps
// of a row through shared memory; rows past the end are clamped (and not stored) so that every
// thread reaches the barrier.
// HEADS: the projection has stored its parts head-split already (gemm_heads): each is normalised and rotated in place, x is not
// read. A thread reads and writes the same chunks.
template <int NPAIR, int WPR, bool HEADS = false>
__global__ void __launch_bounds__(128, NPAIR == 1 ? 8 : 1)
qkv_epilogue_kernel(const __half* __restrict__ x, long long row_stride,
                    const __grid_constant__ QkvParts parts,
                    const __half* __restrict__ cos_vals, const __half* __restrict__ sin_vals,
                    int batch, int seq_len, int num_heads, int head_dim, float eps,
                    long long out_seq_stride) {
    constexpr int RPC = 4 / WPR;  // rows per CTA
    pdl_wait();
    pdl_trigger();
    const int lane = (WPR == 1) ? (threadIdx.x & 31) : (threadIdx.x % (32 * WPR));  // index within the row's threads
    const long long rows = (long long)batch * seq_len;
    long long row = (long long)blockIdx.x * RPC + threadIdx.x / (32 * WPR);
    const bool live = row < rows;
    if (WPR == 1 && !live) return;
    if (!live) row = rows - 1;
    const int part = blockIdx.y;
    const int dim = num_heads * head_dim;
    const int npairs = dim / 16, cpt = head_dim / 16, half_d = head_dim / 2;
    const int b = (int)(row / seq_len), s = (int)(row % seq_len);
    const __half* xr = x + row * row_stride + (long long)part * dim;
    const float* gamma = parts.gamma[part];
    __half* out = parts.out[part];
    auto out_at = [&](int p) { return (((size_t)b * num_heads + p / cpt) * out_seq_stride + s) * head_dim + (p % cpt) * 8; };

    // every load of the row is issued before the first use: the row itself (streamed), the norm weights
    // and the rotation tables (both shared by all rows, L2-resident)
    const bool rope = parts.use_rope[part] != 0;
    Half8 xl[NPAIR], xh[NPAIR], cl8[NPAIR], sl8[NPAIR], ch8[NPAIR], sh8[NPAIR];
    float gl[NPAIR][8], gh[NPAIR][8];
#pragma unroll
    for (int k = 0; k < NPAIR; ++k) {
        const int p = lane + 32 * WPR * k;
        if (HEADS && !live) {   // a row past the end only reaches the barrier: its clamped row is being overwritten in place by its own warps
            xl[k] = xh[k] = Half8{};
        } else if (p < npairs) {
            const __half* src = HEADS ? out + out_at(p) : xr + (p / cpt) * head_dim + (p % cpt) * 8;
            xl[k] = HEADS ? ld_half8(src) : ldcs_half8(src);
            xh[k] = HEADS ? ld_half8(src + half_d) : ldcs_half8(src + half_d);
        }
    }
#pragma unroll
    for (int k = 0; k < NPAIR; ++k) {
        const int p = lane + 32 * WPR * k;
        if (p < npairs) {
            const int o = (p / cpt) * head_dim + (p % cpt) * 8;
            if (gamma) {
                ldg_float8(gamma + o, gl[k]);
                ldg_float8(gamma + o + half_d, gh[k]);
            }
            if (rope) {
                const size_t to = ((size_t)b * seq_len + s) * head_dim + (p % cpt) * 8;
                cl8[k] = ldg_half8(cos_vals + to);
                sl8[k] = ldg_half8(sin_vals + to);
                ch8[k] = ldg_half8(cos_vals + to + half_d);
                sh8[k] = ldg_half8(sin_vals + to + half_d);
            }
        }
    }
    float lo[NPAIR][8], hi[NPAIR][8];
    float ss = 0.0f;
#pragma unroll
    for (int k = 0; k < NPAIR; ++k) {
        const int p = lane + 32 * WPR * k;
        if (p < npairs) {
            unpack8(xl[k], lo[k]);
            unpack8(xh[k], hi[k]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                ss = fmaf(lo[k][i], lo[k][i], ss);
                ss = fmaf(hi[k][i], hi[k][i], ss);
            }
        }
    }
    if (gamma) {  // uniform over the CTA
        ss = warp_sum(ss);
        if (WPR > 1) {
            __shared__ float s_part[4];
            const int w = threadIdx.x >> 5;
            if ((threadIdx.x & 31) == 0) s_part[w] = ss;
            __syncthreads();
            const int w0 = (w / WPR) * WPR;
            ss = 0.0f;
#pragma unroll
            for (int i = 0; i < WPR; ++i) ss += s_part[w0 + i];
        }
        const float rinv = rsqrtf(ss / (float)dim + eps);
#pragma unroll
        for (int k = 0; k < NPAIR; ++k) {
            const int p = lane + 32 * WPR * k;
            if (p < npairs) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    // the unfused path stores the normalised value as fp16 before rotating it
                    lo[k][i] = round_half((lo[k][i] * rinv) * gl[k][i]);
                    hi[k][i] = round_half((hi[k][i] * rinv) * gh[k][i]);
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NPAIR; ++k) {
        const int p = lane + 32 * WPR * k;
        if (p < npairs) {
            if (rope) {
                float cl[8], sl[8], ch[8], sh[8];
                unpack8(cl8[k], cl);
                unpack8(sl8[k], sl);
                unpack8(ch8[k], ch);
                unpack8(sh8[k], sh);
                rotate8(lo[k], hi[k], cl, sl, ch, sh);
            }
            const size_t oo = out_at(p);
            if (live) {
                store8(out + oo, lo[k]);
                store8(out + oo + half_d, hi[k]);
            }
        }
    }
}

// The HEADS form for q and k that both have a norm, rows of 32 * WPR rotation-pair chunks: a thread keeps its chunk of
// every part over all of its rows, so that the norm weights are read once, the rotation tables once for both parts, and the next
// row's loads are in flight while a row is summed. Bound by L2 and that latency: as many CTAs as are resident at once (160
// registers: three an SM) are the best; us for 5665 rows of q and k, 16 heads of 64: one row a block and part 14.3, two CTAs an SM 13.9,
// three 10.1, four 12.3 (a second, partial round), eight 11.4; held to 128 registers four 12.6. Same arithmetic, same bits.
template <int WPR>
__global__ void __launch_bounds__(128)
qk_rows_kernel(const __grid_constant__ QkvParts parts, const __half* __restrict__ cos_vals, const __half* __restrict__ sin_vals,
               int seq_len, int out_seq, int num_heads, int head_dim, float eps) {
    constexpr int RPC = 4 / WPR, NP = 2;  // rows per CTA at a time; parts
    __shared__ float s_part[2][NP][4];
    pdl_wait();
    pdl_trigger();
    const int p = threadIdx.x % (32 * WPR), sub = threadIdx.x / (32 * WPR), w = threadIdx.x >> 5;
    const int dim = num_heads * head_dim, cpt = head_dim / 16, half_d = head_dim / 2;
    const int h = p / cpt, j = (p % cpt) * 8;
    __half* out[NP];
    float g[NP][2][8];
#pragma unroll
    for (int t = 0; t < NP; ++t) {
        out[t] = parts.out[t] + (size_t)h * out_seq * head_dim + j;
        ldg_float8(parts.gamma[t] + h * head_dim + j, g[t][0]);
        ldg_float8(parts.gamma[t] + h * head_dim + j + half_d, g[t][1]);
    }
    const bool rope = cos_vals != nullptr;
    struct Row { Half8 x[NP][2], c[2], s[2]; };
    auto load = [&](int row, Row& r) {   // a row past the end reads nothing: it may be another thread's, in place
        if (row >= seq_len) { r = Row{}; return; }
        const size_t o = (size_t)row * head_dim;
#pragma unroll
        for (int t = 0; t < NP; ++t) {
            r.x[t][0] = ld_half8(out[t] + o);
            r.x[t][1] = ld_half8(out[t] + o + half_d);
        }
        if (rope) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                r.c[e] = ldg_half8(cos_vals + o + j + e * half_d);
                r.s[e] = ldg_half8(sin_vals + o + j + e * half_d);
            }
        }
    };
    Row cur, nxt;
    int base = blockIdx.x * RPC, buf = 0;
    load(base + sub, cur);
    for (; base < seq_len; base += gridDim.x * RPC, buf ^= 1) {
        const int row = base + sub;
        load(row + gridDim.x * RPC, nxt);
        float lo[2][8], hi[2][8], ss[NP] = {};
#pragma unroll
        for (int t = 0; t < NP; ++t) {
            unpack8(cur.x[t][0], lo[t]);
            unpack8(cur.x[t][1], hi[t]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                ss[t] = fmaf(lo[t][i], lo[t][i], ss[t]);
                ss[t] = fmaf(hi[t][i], hi[t][i], ss[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < NP; ++t) ss[t] = warp_sum(ss[t]);
        if (WPR > 1) {
            if ((threadIdx.x & 31) == 0) {
#pragma unroll
                for (int t = 0; t < NP; ++t) s_part[buf][t][w] = ss[t];
            }
            __syncthreads();   // the buffers take turns: one barrier a row
            const int w0 = (w / WPR) * WPR;
#pragma unroll
            for (int t = 0; t < NP; ++t) {
                ss[t] = 0.0f;
#pragma unroll
                for (int i = 0; i < WPR; ++i) ss[t] += s_part[buf][t][w0 + i];
            }
        }
#pragma unroll
        for (int t = 0; t < NP; ++t) {
            const float rinv = rsqrtf(ss[t] / (float)dim + eps);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                // the unfused path stores the normalised value as fp16 before rotating it
                lo[t][i] = round_half((lo[t][i] * rinv) * g[t][0][i]);
                hi[t][i] = round_half((hi[t][i] * rinv) * g[t][1][i]);
            }
            if (rope) {
                float cl[8], sl[8], ch[8], sh[8];
                unpack8(cur.c[0], cl);
                unpack8(cur.s[0], sl);
                unpack8(cur.c[1], ch);
                unpack8(cur.s[1], sh);
                rotate8(lo[t], hi[t], cl, sl, ch, sh);
            }
            if (row < seq_len) {
                store8(out[t] + (size_t)row * head_dim, lo[t]);
                store8(out[t] + (size_t)row * head_dim + half_d, hi[t]);
            }
        }
        cur = nxt;
    }
}

}  // namespace rfk

using namespace rfk;

int rfk::qk_norm_rope_heads(int n_parts, const float* const* gamma, rfk_half* const* parts_io, const rfk_half* cos_vals,
                            const rfk_half* sin_vals, int seq_len, int out_seq, int num_heads, int head_dim, float eps, rfk_stream_t stream) {
    if (!gamma || !parts_io || n_parts < 1 || n_parts > 3 || seq_len < 0 || out_seq < seq_len || num_heads <= 0 || head_dim <= 0) return RFK_EINVAL;
    const long long dim = (long long)num_heads * head_dim;
    if (head_dim % 16 != 0 || dim > 2048) return RFK_EUNSUPPORTED;
    QkvParts parts{};
    for (int p = 0; p < n_parts; ++p) {
        if (!parts_io[p]) return RFK_EINVAL;
        if (!aligned16(parts_io[p]) || (gamma[p] && !aligned16(gamma[p]))) return RFK_EUNSUPPORTED;
        parts.gamma[p] = gamma[p];
        parts.out[p] = (__half*)parts_io[p];
        parts.use_rope[p] = cos_vals != nullptr;
    }
    if (cos_vals && (!sin_vals || !aligned16(cos_vals) || !aligned16(sin_vals))) return RFK_EINVAL;
    if (seq_len == 0) return RFK_OK;
    const int npairs = (int)(dim / 16);
    if (n_parts == 2 && gamma[0] && gamma[1] && (npairs == 32 || npairs == 64)) {   // wider rows are summed two chunks a thread
        const int wpr = npairs / 32;
        const unsigned grid = std::min(ceil_div(seq_len, 4 / wpr), 3u * kNumSMs);   // 160 registers a thread
        launch_pdl(wpr == 1 ? qk_rows_kernel<1> : qk_rows_kernel<2>, dim3(grid), dim3(128), 0, as_stream(stream), parts, (const __half*)cos_vals,
                   (const __half*)sin_vals, seq_len, out_seq, num_heads, head_dim, eps);
        return launch_status();
    }
#define RFK_QK_HEADS(N, W)                                                                                   \
    launch_pdl(qkv_epilogue_kernel<N, W, true>, dim3(ceil_div(seq_len, 4 / W), n_parts), dim3(128), 0, as_stream(stream), \
               (const __half*)nullptr, 0LL, parts, (const __half*)cos_vals, (const __half*)sin_vals, 1, seq_len, num_heads, \
               head_dim, eps, (long long)out_seq)
    if (npairs <= 32) RFK_QK_HEADS(1, 1);
    else if (npairs <= 64) RFK_QK_HEADS(1, 2);
    else RFK_QK_HEADS(2, 2);
#undef RFK_QK_HEADS
    return launch_status();
}

extern "C" int rfk_qk_norm_rope_heads(rfk_half* q, rfk_half* k, const float* gamma_q, const float* gamma_k, const rfk_half* cos_vals,
                                      const rfk_half* sin_vals, int seq_len, int out_seq, int num_heads, int head_dim, float eps,
                                      rfk_stream_t stream) {
    const float* g[2] = {gamma_q, gamma_k};
    rfk_half* x[2] = {q, k};
    return qk_norm_rope_heads(k ? 2 : 1, g, x, cos_vals, sin_vals, seq_len, out_seq, num_heads, head_dim, eps, stream);
}

extern "C" int rfk_triangle_rope_freqs(const rfk_half* pos, const float* learned_freqs,
                                       rfk_half* out_cos, rfk_half* out_sin, int batch,
                                       int seq_len, int num_freqs, int head_dim,
                                       rfk_stream_t stream) {
    if (!pos || !learned_freqs || !out_cos || !out_sin) return RFK_EINVAL;
    if (batch < 0 || seq_len < 0 || num_freqs <= 0 || head_dim <= 0 || (head_dim & 1))
        return RFK_EINVAL;
    const long long tokens = (long long)batch * seq_len;
    if (tokens == 0) return RFK_OK;
    cudaStream_t st = as_stream(stream);
    if (head_dim % 16 == 0 && aligned16(out_cos) && aligned16(out_sin)) {
        const bool many = tokens * (head_dim / 4) > (1 << 20);
        const long long n = tokens * (head_dim / (many ? 16 : 4));
        launch_pdl(many ? rope_table_vec_kernel<8> : rope_table_vec_kernel<2>, dim3(ceil_div(n, 256)), dim3(256), 0, st,
            (const __half*)pos, learned_freqs, (__half*)out_cos, (__half*)out_sin, tokens,
            num_freqs, head_dim);
    } else {
        const long long n = tokens * head_dim;
        launch_pdl(rope_table_generic_kernel, dim3(ceil_div(n, 256)), dim3(256), 0, st,
            (const __half*)pos, learned_freqs, (__half*)out_cos, (__half*)out_sin, tokens,
            num_freqs, head_dim);
    }
    return launch_status();
}

extern "C" int rfk_apply_rope(rfk_half* q, rfk_half* k, const rfk_half* c, const rfk_half* s,
                              int batch, int num_heads, int seq_len, int head_dim,
                              rfk_stream_t stream) {
    return launch_rope<__half, 2>((const __half*)q, (__half*)q, (const __half*)k, (__half*)k,
                                  (const __half*)c, (const __half*)s, batch, num_heads, seq_len,
                                  seq_len, head_dim, seq_len, seq_len, as_stream(stream));
}

extern "C" int rfk_apply_rope_one(rfk_half* x, const rfk_half* c, const rfk_half* s, int batch,
                                  int num_heads, int seq_len, int head_dim, rfk_stream_t stream) {
    return launch_rope<__half, 1>((const __half*)x, (__half*)x, nullptr, nullptr, (const __half*)c,
                                  (const __half*)s, batch, num_heads, seq_len, seq_len, head_dim,
                                  seq_len, seq_len, as_stream(stream));
}

extern "C" int rfk_apply_rope_f32(float* q, float* k, const rfk_half* c, const rfk_half* s,
                                  int batch, int num_heads, int seq_len, int head_dim,
                                  rfk_stream_t stream) {
    return launch_rope<float, 2>(q, q, k, k, (const __half*)c, (const __half*)s, batch, num_heads,
                                 seq_len, seq_len, head_dim, seq_len, seq_len, as_stream(stream));
}

extern "C" int rfk_apply_rope_one_f32(float* x, const rfk_half* c, const rfk_half* s, int batch,
                                      int num_heads, int seq_len, int head_dim,
                                      rfk_stream_t stream) {
    return launch_rope<float, 1>(x, x, nullptr, nullptr, (const __half*)c, (const __half*)s, batch,
                                 num_heads, seq_len, seq_len, head_dim, seq_len, seq_len,
                                 as_stream(stream));
}

extern "C" int rfk_rope_one_oop(const rfk_half* src, rfk_half* dst, const rfk_half* c,
                                const rfk_half* s, int batch, int num_heads, int seq_len,
                                int head_dim, int src_seq_stride, int dst_seq_stride,
                                int copy_tail, rfk_stream_t stream) {
    if (src_seq_stride < seq_len || dst_seq_stride < seq_len) return RFK_EINVAL;
    int rows_total = seq_len;
    if (copy_tail) {
        rows_total = dst_seq_stride;
        if (src_seq_stride < rows_total) return RFK_EINVAL;
    }
    return launch_rope<__half, 1>((const __half*)src, (__half*)dst, nullptr, nullptr,
                                  (const __half*)c, (const __half*)s, batch, num_heads, seq_len,
                                  rows_total, head_dim, src_seq_stride, dst_seq_stride,
                                  as_stream(stream));
}

extern "C" int rfk_rope_one_oop_strided(const rfk_half* src, rfk_half* dst, const rfk_half* c,
                                        const rfk_half* s, int batch, long long src_batch_stride,
                                        long long dst_batch_stride, long long table_batch_stride,
                                        int num_heads, int seq_len, int head_dim, int src_seq_stride,
                                        int dst_seq_stride, const float* col_scale,
                                        long long col_scale_batch_stride, rfk_stream_t stream) {
    if (src_seq_stride < seq_len || dst_seq_stride < seq_len) return RFK_EINVAL;
    if (src_batch_stride < 0 || dst_batch_stride < 0 || table_batch_stride < 0 || col_scale_batch_stride < 0) return RFK_EINVAL;
    return launch_rope<__half, 1>((const __half*)src, (__half*)dst, nullptr, nullptr,
                                  (const __half*)c, (const __half*)s, batch, num_heads, seq_len,
                                  seq_len, head_dim, src_seq_stride, dst_seq_stride,
                                  as_stream(stream), src_batch_stride, dst_batch_stride,
                                  table_batch_stride, (const float*)col_scale, col_scale_batch_stride);
}

extern "C" int rfk_qkv_norm_rope_transpose(const rfk_half* x, long long row_stride, int n_parts,
                                           const float* const* gamma, rfk_half* const* out,
                                           const int* use_rope, const rfk_half* cos_vals,
                                           const rfk_half* sin_vals, int batch, int seq_len,
                                           int num_heads, int head_dim, float eps,
                                           int out_seq_stride, rfk_stream_t stream) {
    if (!x || !gamma || !out || !use_rope || n_parts < 1 || n_parts > 3) return RFK_EINVAL;
    if (out_seq_stride == 0) out_seq_stride = seq_len;
    if (out_seq_stride < seq_len) return RFK_EINVAL;
    if (batch < 0 || seq_len < 0 || num_heads <= 0 || head_dim <= 0) return RFK_EINVAL;
    const long long dim = (long long)num_heads * head_dim;
    if (row_stride < dim * n_parts) return RFK_EINVAL;
    if (head_dim % 16 != 0 || dim > 2048 || row_stride % 8 != 0 || !aligned16(x))
        return RFK_EUNSUPPORTED;
    QkvParts parts{};
    for (int p = 0; p < n_parts; ++p) {
        if (!out[p] || !aligned16(out[p])) return RFK_EINVAL;
        if (gamma[p] && !aligned16(gamma[p])) return RFK_EUNSUPPORTED;
        if (use_rope[p] && (!cos_vals || !sin_vals || !aligned16(cos_vals) || !aligned16(sin_vals)))
            return RFK_EINVAL;
        parts.gamma[p] = gamma[p];
        parts.out[p] = (__half*)out[p];
        parts.use_rope[p] = use_rope[p];
    }
    const long long rows = (long long)batch * seq_len;
    if (rows == 0) return RFK_OK;
    cudaStream_t st = as_stream(stream);
    const int npairs = (int)(dim / 16);
    // two warps per row from 64 chunk pairs on (dim 1024: one pair per thread, 64 registers, 8 CTAs per SM)
#define RFK_QKV(N, W)                                                                            \
    launch_pdl(qkv_epilogue_kernel<N, W>, dim3(ceil_div(rows, 4 / W), n_parts), dim3(128), 0, st, \
               (const __half*)x, row_stride, parts, (const __half*)cos_vals, (const __half*)sin_vals, \
               batch, seq_len, num_heads, head_dim, eps, (long long)out_seq_stride)
    if (npairs <= 32) RFK_QKV(1, 1);
    else if (npairs <= 64) RFK_QKV(1, 2);
    else RFK_QKV(2, 2);
#undef RFK_QKV
    return launch_status();
}
