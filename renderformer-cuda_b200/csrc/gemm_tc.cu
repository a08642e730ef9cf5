// Dense projection C = epilogue(A W^T) on the 5th-generation tensor cores (tcgen05 + tensor memory
// + TMA), fp16 operands, fp32 accumulation, with the element-wise step that follows the projection
// in the layer fused into the epilogue:
//   RFK_GEMM_EPI_NONE      C = A W^T (+ bias)                                   rf::linear
//   RFK_GEMM_EPI_RESIDUAL  C = A W^T (+ bias) + R                               rf::linear + rf::residual_add
//   RFK_GEMM_EPI_SWIGLU    C = silu(A Wg^T) * (A Wu^T)                          the two projections and the
//                                                                               gate of rf::ffn_swiglu
// Reference boundary: rf::linear, src/layers/linear.cu:7-25 (one cublasGemmEx + a bias kernel), and
// rf::ffn_swiglu, src/layers/transformer.cu:63-79 (two GEMMs into [M, hidden] buffers, fused_silu_mul,
// a third GEMM) of BANANASJIM/renderformer-cuda.
//
// One persistent CTA per SM walks output tiles of 128 rows x 256 accumulator columns (row-tile index
// fastest, so that the CTAs running together share weight tiles in L2). K is consumed in blocks of
// 64 halves (one 128-byte swizzle row) through a ring of kStages shared-memory stages:
//   warp 0   producer: one thread issues three TMA tile loads per stage (A 128 x 64; two weight boxes
//            of 128 x 64 - rows n0..n0+127 and n0+128..n0+255 of W, or, with the SwiGLU epilogue,
//            the gate rows and the up rows of the same 128 hidden units) that complete on the
//            stage's mbarrier; rows and columns past the end of a tensor arrive as zeros.
//   warp 1   one thread issues tcgen05.mma M128 N256 K16 x 4 per stage into one of two accumulators
//            in tensor memory (2 x 256 columns), then commits the stage's "empty" barrier; after
//            the last K block it commits the accumulator's "full" barrier.
//   warps 2-5 epilogue: a thread owns one output row (= its tensor-memory lane), reads the row in
//            chunks of 32 columns with tcgen05.ld, applies bias / residual / gate in fp32, rounds
//            once to fp16 and writes 64 contiguous bytes per chunk. While they drain accumulator a,
//            the tensor core already fills accumulator a ^ 1 with the CTA's next tile.
// Every mbarrier wait is bounded; on a time-out the CTA raises an error word, waits (bounded) for its
// own copies and products in flight, frees its tensor memory and returns.
#include <cuda.h>  // CUtensorMap and its enums; the encoder itself is looked up at run time
#include <cstdlib>
#include "common.cuh"
#include "kernels_internal.h"
#include "tc_pair.cuh"

namespace rfk {

__device__ int g_gemm_tc_error = 0;  // first time-out / failure code seen by any CTA since load

namespace tcgemm {

constexpr int BM = 128, BNACC = 256, BK = 64;
constexpr int kStages = 4;
constexpr int kThreads = 192;                  // warp 0 producer, warp 1 MMA issuer, warps 2-5 epilogue
constexpr int kABytes = BM * BK * 2;           // 16 KB
constexpr int kWBoxBytes = 128 * BK * 2;       // 16 KB, two per stage
constexpr int kStageBytes = kABytes + 2 * kWBoxBytes;
constexpr int kTmemCols = 512;                 // two accumulators of 256 fp32 columns

struct __align__(8) Ctrl {
    uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base;
    int abort;
};
constexpr int kSmemBytes = kStages * kStageBytes + 256;
static_assert(sizeof(Ctrl) <= 256, "control block");
static_assert(kSmemBytes + 1024 <= 227 * 1024, "one CTA per SM");

enum : int { kErrTimeout = 1, kErrSmemAlign = 2 };

// Build with -DRFK_GEMM_TIMELINE to make CTA 0 of the pair kernel record %globaltimer stamps (ns) of its phases
// in a device array that rfk_gemm_timeline() reads back; compiled out otherwise.
#ifdef RFK_GEMM_TIMELINE
__device__ unsigned long long g_timeline[16];
#define RFK_STAMP(i) do { if (blockIdx.x == 0) g_timeline[i] = tc::global_timer_ns(); } while (0)
#else
#define RFK_STAMP(i) do { } while (0)
#endif

// Fourth epilogue of the pair kernel (own entry point, rfk_gemm_f16_heads): the output is stored head-split,
// [part][group][head][seq][64], through a rank-5 tile store, and every row's sum of squares over each 256-column
// tile (of the fp16-rounded values) is written to row_ss[part][row][tile] for the parts selected by ss_mask: the
// statistic of the QK-RMSNorm that follows the projection, so that the consumer can normalise while it loads.
constexpr int kEpiHeads = 3;

// Folded norms. A projection behind an RMSNorm, C = epilogue((x / rms(x) * gamma) W^T), is rms(x)^-1 * (x (W gamma)^T) a row: with the norm's
// weight multiplied into W once, the product can take x as it is, and the norm costs a factor a row in the epilogue, from the row's sum
// of squares, which whoever wrote x has summed beside it. Three launches of a decoder layer's eleven go, and with them 2 to 3 us each of a small
// view and 5 to 8 of a large one (us a view, separate norms / folded: 128 x 128 pixels 772 / 650, 512 x 512 3902 / 3787, with 128-wide heads
// 3456 / 3370, frames of four 14460 / 13930); the sums and the reordering cost a product 0.3 to 1.5. Writing x * gamma beside x instead of
// folding gamma into W cost 36 products of a view 2.4 us each (512 x 512 3863, 128 x 128 680). EPI with this bit: SwiGLU and head-split products whose rows get such a
// factor; residual products that write the sums of squares of their rows, and may put the rows elsewhere (Grid).
// The sums lie [row][tiles]: one each 256 columns, or one each 32 where tiles of fewer columns wrote them. Both add the
// same way - eight squares in column order, four of those in pairs (square_sum), eight of these in order, the 256s in order - so that whoever reads
// them gets the same bits.
constexpr int kFold = 8;

// Rows that are the 4 x 4 blocks of a token grid, block by block (16 rows), windows of 2 x 2 blocks one after the other, of a grid that has been
// shifted by `from` blocks: where they go in a grid shifted by `to` blocks, and where in raster order.
struct Grid {
    int bw, bh;       // blocks across and down; 0: rows stay where they are
    int from, to;
    __device__ __forceinline__ void block(int k, int& view, int& by, int& bx) const {   // k-th block, in the unshifted grid
        const int per = bw * bh;
        view = k / per;
        const int i = k - view * per, win = i >> 2, ww = bw >> 1;
        by = (win / ww) * 2 + ((i >> 1) & 1) - from;
        bx = (win % ww) * 2 + (i & 1) - from;
        if (by < 0) by += bh;
        if (bx < 0) bx += bw;
    }
    __device__ __forceinline__ int next(int view, int by, int bx) const {   // that block's index in the grid shifted by `to`
        by += to;
        bx += to;
        if (by >= bh) by -= bh;
        if (bx >= bw) bx -= bw;
        return view * bw * bh + (((by >> 1) * (bw >> 1) + (bx >> 1)) << 2) + ((by & 1) << 1) + (bx & 1);
    }
};

struct Params {
    __half* C; long long ldc;
    const __half* R; long long ldr;     // residual (EPI_RESIDUAL), may alias C
    const __half* bias;                 // [N] or null
    int M, N, K;                        // N = output columns
    int tiles_m, tiles_n;
    float* row_ss;                      // kEpiHeads: [parts][M][tiles per part] partial sums of squares, or null
    long long part_stride;              // kEpiHeads on small tiles, which store without a tensor map: halves between parts
    int seq, out_seq, units, head_units, ss_mask;  // kEpiHeads: rows per group, 64-column units per part and per head, parts that get row_ss
    const float* in_ss; int in_tiles, in_group;    // kFold: A's rows' sums of squares, how many a row, and how many of them make up 256 columns
    float in_inv_dim, in_eps, in_mul;              // the row's factor: in_mul * rsqrt(sum * in_inv_dim + in_eps)
    const float *col_mul, *up_mul;                 // if not null, another factor for each 64 columns (and of the up columns)
    int ss_tiles;                                  // kFold: sums a row that row_ss gets, of a part
    __half* raster;                                // kFold, residual: the rows in raster order too, or alone if C is null; pitch ldc
    Grid grid;
};

// the further factor of the columns that begin at col, a multiple of 64 or inside one (kFold)
__device__ const float g_one = 1.0f;
__device__ __forceinline__ float column_factor(const Params& p, const float* mul, int col) {
    float f;   // volatile: asked for where it is written, ahead of the loads that row_factor waits for, and not behind the products
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(f) : "l"(mul ? mul + (min(col, p.N - 1) >> 6) : &g_one));
    return f;
}
// a row's factor (kFold)
__device__ __forceinline__ float row_factor(const Params& p, int row) {
    const float* s = p.in_ss + (size_t)row * p.in_tiles;
    float sum = 0.0f;
    if (p.in_group == 1) {
        for (int t = 0; t < p.in_tiles; ++t) sum += __ldg(s + t);
    } else {
        for (int t = 0; t < p.in_tiles; t += 8) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(s + t)), b = __ldg(reinterpret_cast<const float4*>(s + t + 4));
            sum += ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
        }
    }
    return p.in_mul * rsqrtf(fmaf(sum, p.in_inv_dim, p.in_eps));
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_half2(uint32_t w) {
    return __half22float2(*reinterpret_cast<__half2*>(&w));
}

// The sum of the squares of 32 fp16 values, packed in order; four chains, for their latency
__device__ __forceinline__ float square_sum(const uint32_t (&o)[16]) {
    float c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c[k] = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 v = unpack_half2(o[4 * k + i]);
            c[k] = fmaf(v.x, v.x, c[k]);
            c[k] = fmaf(v.y, v.y, c[k]);
        }
    }
    return (c[0] + c[1]) + (c[2] + c[3]);
}

__device__ __forceinline__ void tma_prefetch_2d(const void* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
// A product's weights on their way from device memory into L2 while the kernel before it still runs, asked for by one lane of a CTA ahead of the
// wait: `ask` walks the K blocks of the CTA's first tile that fall to it among the tiles that read the same weights. A hint only, and L2 is where
// writes meet: what the product reads is copied after the wait, so weights that the kernel before writes are read as it left them. A model's weights are 0.3 GB
// a view or scene, more than L2 keeps. us without / with: encodings of 300 triangles 698 / 685, of 2500 2103 / 2073, of 5633 5337 / 5286; an image of
// 128 x 128 1119 / 1100, of 320 x 320 2468 / 2437; a view of 512 x 512 no difference.
template <typename Ask> __device__ __forceinline__ void prefetch_weights(bool leader, Ask ask) {
    if (leader) ask();
    __syncwarp();
}
// Tiled copy global -> shared of one box of a rank-2 tensor map (x innermost, in elements; x * 2 bytes
// is always a multiple of 128 here); the bytes are counted on `bar`.
__device__ __forceinline__ void tma_load_2d(uint32_t dst_smem, const void* tmap, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst_smem), "l"(tmap), "r"(x), "r"(y), "r"(tc::smem_addr(bar)) : "memory");
}

// Epilogue of one thread for one tile: the thread's accumulator row (tensor-memory address t_acc, BN_OUT output
// columns, for SwiGLU the up columns 128 further on) -> bias / residual / gate in fp32 -> fp16 -> global row `row`.
template <int EPI>
__device__ __forceinline__ void epilogue_tile(const Params& p, uint32_t t_acc, int row, int n0) {
    constexpr int BN_OUT = (EPI == RFK_GEMM_EPI_SWIGLU) ? 128 : 256;
    uint32_t v[32];
    const bool row_ok = row < p.M;
    __half* crow = p.C + (size_t)(row_ok ? row : 0) * p.ldc + n0;
    if (EPI == RFK_GEMM_EPI_SWIGLU) {
        uint32_t u[32];
#pragma unroll 1
        for (int c = 0; c < BN_OUT / 32; ++c) {
            tc::tmem_ld32(t_acc + c * 32, v);          // gate columns
            tc::tmem_ld32(t_acc + 128 + c * 32, u);    // up columns of the same hidden units
            tc::tc_wait_ld(v);
            tc::tc_wait_ld(u);
            uint32_t o[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                const float g0 = __uint_as_float(v[i]), g1 = __uint_as_float(v[i + 1]);
                // silu(g) * u = g * u / (1 + 2^(-g log2 e))
                const float s0 = g0 * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * g0));
                const float s1 = g1 * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * g1));
                o[i >> 1] = pack_half2(s0 * __uint_as_float(u[i]), s1 * __uint_as_float(u[i + 1]));
            }
            if (row_ok) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int col = n0 + c * 32 + q * 8;
                    if (col < p.N)
                        *reinterpret_cast<uint4*>(crow + c * 32 + q * 8) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                }
            }
        }
    } else {
        const __half* rrow = (EPI == RFK_GEMM_EPI_RESIDUAL) ? p.R + (size_t)(row_ok ? row : 0) * p.ldr + n0 : nullptr;
        // The residual row is read two chunks ahead of its use (each thread reads 64 bytes of its own row per chunk:
        // the latency of these scattered loads, not their volume, is what an un-pipelined epilogue pays 8 times).
        constexpr int kAhead = 2;
        uint4 res[kAhead + 1][4];
        auto load_res = [&](int c) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int col = n0 + c * 32 + q * 8;
                res[c % (kAhead + 1)][q] = (row_ok && c < BN_OUT / 32 && col < p.N)
                                               ? *reinterpret_cast<const uint4*>(rrow + c * 32 + q * 8) : make_uint4(0, 0, 0, 0);
            }
        };
        if (EPI == RFK_GEMM_EPI_RESIDUAL) {
#pragma unroll
            for (int c = 0; c < kAhead; ++c) load_res(c);
        }
#pragma unroll
        for (int c = 0; c < BN_OUT / 32; ++c) {
            if (n0 + c * 32 >= p.N) break;             // uniform over the CTA: the tile's tail lies beyond N
            tc::tmem_ld32(t_acc + c * 32, v);
            if (EPI == RFK_GEMM_EPI_RESIDUAL) load_res(c + kAhead);
            tc::tc_wait_ld(v);
            if (p.bias) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const int col = n0 + c * 32 + i;
                    if (col < p.N) {
                        const float2 b = unpack_half2(__ldg(reinterpret_cast<const uint32_t*>(p.bias + col)));
                        // the unfused path rounds the product to fp16 before the bias is added (linear.cu:15-25)
                        v[i] = __float_as_uint(round_half(__uint_as_float(v[i])) + b.x);
                        v[i + 1] = __float_as_uint(round_half(__uint_as_float(v[i + 1])) + b.y);
                    }
                }
            }
            uint32_t o[16];
            if (EPI == RFK_GEMM_EPI_RESIDUAL) {
                const uint32_t* rw = reinterpret_cast<const uint32_t*>(res[c % (kAhead + 1)]);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 rr = unpack_half2(rw[i]);
                    o[i] = pack_half2(__uint_as_float(v[2 * i]) + rr.x, __uint_as_float(v[2 * i + 1]) + rr.y);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = pack_half2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
            }
            if (row_ok) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int col = n0 + c * 32 + q * 8;
                    if (col < p.N)
                        *reinterpret_cast<uint4*>(crow + c * 32 + q * 8) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                }
            }
        }
    }
}

// out columns per tile: 256 (plain / residual) or 128 (SwiGLU: 128 gate + 128 up accumulator columns)
template <int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w0,
               const __grid_constant__ CUtensorMap map_w1, const Params p) {
    constexpr int BN_OUT = (EPI == RFK_GEMM_EPI_SWIGLU) ? 128 : 256;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = tc::smem_addr(smem_raw);
    if (base & 1023u) {  // uniform over the CTA, nothing allocated yet
        if (threadIdx.x == 0) atomicCAS(&g_gemm_tc_error, 0, kErrSmemAlign);
        return;
    }
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + kStages * kStageBytes);
    volatile int* abort_flag = &ctrl->abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int num_kb = (p.K + BK - 1) / BK;
    const int num_tiles = p.tiles_m * p.tiles_n;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { tc::mbar_init(&ctrl->full[s], 1); tc::mbar_init(&ctrl->empty[s], 1); }
        for (int a = 0; a < 2; ++a) { tc::mbar_init(&ctrl->acc_full[a], 1); tc::mbar_init(&ctrl->acc_empty[a], 4); }
        tc::mbar_init(&ctrl->drain, 1);
        ctrl->abort = 0;
        tc::fence_barrier_init();
    }
    if (warp == 0) {  // one warp allocates the CTA's tensor memory and later frees it
        tc::tmem_alloc(&ctrl->tmem_base, kTmemCols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem_cta = ctrl->tmem_base;
    pdl_wait();      // set-up above is on-chip only; the operands are another kernel's output
    pdl_trigger();

    if (warp == 0) {
        // ------------------------------------------------------------ producer (one thread)
        if (lane == 0) {
            tc::prefetch_tensormap(&map_a); tc::prefetch_tensormap(&map_w0); tc::prefetch_tensormap(&map_w1);
            int it = 0;       // K blocks issued so far by this CTA, over all of its tiles
            bool ok = true;
            for (int t = blockIdx.x; ok && t < num_tiles; t += gridDim.x) {
                const int m0 = (t % p.tiles_m) * BM, n0 = (t / p.tiles_m) * BN_OUT;
                // second weight box: the next 128 rows of W, or the up-projection rows of the same hidden units
                const int n1 = (EPI == RFK_GEMM_EPI_SWIGLU) ? n0 : n0 + 128;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % kStages;
                    // stage s was last read by the products of K block it - kStages
                    if (it >= kStages && !tc::mbar_wait(&ctrl->empty[s], ((it / kStages) + 1) & 1, abort_flag)) { ok = false; break; }
                    const uint32_t sA = base + s * kStageBytes;
                    tc::mbar_arrive_expect_tx(&ctrl->full[s], kStageBytes);
                    tma_load_2d(sA, &map_a, kb * BK, m0, &ctrl->full[s]);
                    tma_load_2d(sA + kABytes, &map_w0, kb * BK, n0, &ctrl->full[s]);
                    tma_load_2d(sA + kABytes + kWBoxBytes, &map_w1, kb * BK, n1, &ctrl->full[s]);
                }
            }
            if (*abort_flag) {
                // The CTA is giving up: every copy this thread started lands in this CTA's shared memory and counts on a
                // full[] barrier; wait (bounded) for the last copy of each stage before the CTA exits.
                for (int s = 0; s < kStages && s < it; ++s) {
                    const int last = ((it - 1 - s) / kStages) * kStages + s;
                    tc::mbar_wait_drain(&ctrl->full[s], (last / kStages) & 1);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ issuer of the products (one thread)
        if (lane == 0) {
            constexpr uint32_t idesc = tc::umma_idesc_f16(BM, BNACC, 0);  // A and B both K-major
            int it = 0, tl = 0;  // K blocks and tiles consumed so far
            bool ok = true;
            for (int t = blockIdx.x; ok && t < num_tiles; t += gridDim.x, ++tl) {
                const int acc = tl & 1;
                // the epilogue must have drained this accumulator's previous tile (tile tl - 2)
                if (tl >= 2) ok = tc::mbar_wait(&ctrl->acc_empty[acc], ((tl >> 1) + 1) & 1, abort_flag);
                if (!ok) break;
                tc::tc_fence_after();
                const uint32_t d_tmem = tmem_cta + acc * BNACC;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % kStages;
                    ok = tc::mbar_wait(&ctrl->full[s], (it / kStages) & 1, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint32_t a_lo = tc::umma_desc_lo(base + s * kStageBytes);
                    const uint32_t b_lo = tc::umma_desc_lo(base + s * kStageBytes + kABytes);
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks)  // 16 halves = 32 bytes along a swizzled row
                        tc::umma_f16_lo(d_tmem, a_lo + ks * 2, b_lo + ks * 2, idesc, (kb > 0) || (ks > 0));
                    tc::umma_commit(&ctrl->empty[s]);     // the stage is free once these products have read it
                }
                if (ok) tc::umma_commit(&ctrl->acc_full[acc]);
            }
            if (*abort_flag) {  // giving up: let this thread's products finish before tensor memory is freed
                tc::umma_commit(&ctrl->drain);
                tc::mbar_wait_drain(&ctrl->drain, 0);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue, warps 2-5
        const int lane_grp = warp & 3;                        // a warp reaches tensor-memory lanes [32 * (warp % 4), +32)
        const int r = lane_grp * 32 + lane;                   // row within the tile
        const uint32_t lane_off = (uint32_t)(lane_grp * 32) << 16;
        bool ok = true;
        int tl = 0;
        for (int t = blockIdx.x; t < num_tiles; t += gridDim.x, ++tl) {
            const int acc = tl & 1;
            const int m0 = (t % p.tiles_m) * BM, n0 = (t / p.tiles_m) * BN_OUT;
            ok = tc::mbar_wait_warp(&ctrl->acc_full[acc], (tl >> 1) & 1, abort_flag);
            if (!ok) break;
            tc::tc_fence_after();
            epilogue_tile<EPI>(p, tmem_cta + lane_off + acc * BNACC, m0 + r, n0);
            // every tcgen05.ld of this warp has completed (wait::ld above): hand the accumulator back
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&ctrl->acc_empty[acc]);
        }
    }

    // ---- teardown: every path (normal or aborted) arrives here with no divergence inside a warp
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem_cta, kTmemCols);
    }
    if (tid == 0 && ctrl->abort) atomicCAS(&g_gemm_tc_error, 0, kErrTimeout);
}

namespace pair { using namespace pair_ptx; }

// ------------------------------------------------------------------------------------------------
// The same product on small tiles, one per CTA, for calls that do not fill the machine: a view of 256 tokens gives the pair
// kernel below four tiles for its 74 pairs, and a 4096-wide K then runs 64 K blocks of 0.3 us one after the other. Here a
// tile is 64 or 128 rows by 32 to 128 accumulator columns, so that there are many and each takes few operand bytes per K
// block (one SM takes them at about 110 GB/s). But for the sums in quarters below every output is summed over the K blocks in the same order
// as by the other kernels and has the same bits, so that a call may move between them with its size (the views of a frame
// must equal the views one by one).
//   Sums in quarters (SUM_): of a 64-row view's product with K = 4096 a CTA takes 64 K blocks of 64 x 32 columns one after the other, 7 us of loads
//   on 32 SMs, and with 256 rows the 128 tiles take 98 MB out of L2. The sum is therefore defined as ((a + b) + c) + d of its quarters of K for views of
//   at most 256 rows, whatever frame they are in. For few rows a cluster of four CTAs takes a quarter each, of wider tiles; the fp32 rows go to the CTA
//   of their quarter of the tile through the cluster's shared memory, and a warp of it finishes 32 columns. For more rows one CTA keeps the four
//   sums in accumulators of their own, and for more than a round of those the pair kernel makes them (kSumThreads). us, one sum / quarters, K = 4096, N = 1024: 64 rows 8.7 / 5.6, 128 8.7 / 6.3, 192 8.9 / 7.8, 256 9.1 / 7.9, and on single
//   CTAs 320 9.8 / 10.0, 512 10.0 / 10.2, 1024 13.8 / 13.8; a view of 64 x 64 pixels 539 / 505, of 128 x 128 648 / 637, frames of four of these 847 / 843. With
//   K = 1024 the exchange (0.8 to 1.5 us) costs more than it gains (64 rows 3.63 / 3.87): these keep one sum.
//   A stage is two K blocks: one wait, one announcement and one commit for eight products. The issuing lane and the producer's are
//   elected ones (elect.sync). With one block per stage and lane 0's loops a K block took 0.30 us on every tile size, the cost
//   of issuing and not of the operands; two blocks and elected lanes in loops of whole warps took the 64 x 32 tile to 0.12 us, loops of
//   the elected lanes alone, the others waiting at the warp's barrier, to 0.10 (us, whole warps / lanes alone, weights in L2: 256 x 1024 x
//   4096 9.63 / 8.23, 256 x 1024 x 1024 3.90 / 3.62, 576 x 1024 x 4096 11.1 / 9.3; 128 x 64 tiles 1024 x 1024 x 4096 12.45 / 12.18; the
//   tensor pipe alone would take 0.05 us a block). 128 x 128 tiles keep whole warps: 2304 x 1024 x 4096 16.9 / 17.6, 1600 x 1024 x 4096
//   16.4 / 17.4. The 128 x 64 tile's producer is lane 0 with the plain and residual epilogues (elected / lane 0, issuer elected in both: 2779 x 384 x
//   4096 13.2 / 12.6, 1115 x 1024 x 4096 12.2 / 11.5, x 1024 4.87 / 4.88) and an elected lane with the others (SwiGLU 1024 x 512 x 1024 5.09 /
//   5.70, head-split 1024 x 1024 x 4096 12.0 / 12.3). Half the ring costs 7 % (the copies in flight cover their latency); one copy per operand and stage instead of two changed
//   nothing. Weights copied ahead of the kernel's wait for its predecessor gain where norms are folded (below); with separate norms they changed nothing or
//   cost (320 x 320 views +4 %), and only the prefetch into L2 is left there.
//   BM 64: the accumulator's row r is tensor-memory lane 32 * (r / 16) + r % 16, half the lanes of each warp's quarter.
//   SwiGLU: the first BN / 2 accumulator columns are gate columns, the others the up columns of the same hidden units.
// The epilogue's threads store their own rows: a tile row is 32 to 256 bytes, one to eight whole sectors.
namespace small {

constexpr int kSub = 2;                  // K blocks per stage
template <int BM_, int BN_, bool SPLIT = false> struct Cfg {
    static constexpr int kBlockBytes = (BM_ + BN_) * BK * 2;      // operands of one K block
    static constexpr int kStageBytes = kSub * kBlockBytes;
    static constexpr int kStages = (SPLIT ? 180 : 192) * 1024 / kStageBytes;   // 8 to 3: a lone CTA waits for memory, so as deep as fits
    static constexpr int kSmemBytes = kStages * kStageBytes + 256;
    static_assert(kStages >= 2 && kStages <= 8 && kSmemBytes + 1024 <= 227 * 1024, "control block, shared memory of an SM");
};

struct __align__(8) Ctrl {
    uint64_t full[8], empty[8], acc_full, drain;
    uint32_t tmem_base;
    int abort;
};
static_assert(sizeof(Ctrl) <= 256, "control block");

// The pieces of a split sum on their way to the CTA that adds them: [the other pieces, its own][four columns][row of its quarter of the tile][4 floats], so
// that a warp's stores into another CTA are 512 (256) bytes on end
template <int BM_, int BN_> constexpr int kHandedPiece = (BM_ / 4) * BN_ * 4;
template <int BM_, int BN_> constexpr int kHandedBytes = 4 * kHandedPiece<BM_, BN_>;

// SUM 1: one sum over K. 4: ((a + b) + c) + d over the quarters of K, each a sum of its own; kSplit: by a cluster of four CTAs with a quarter each.
enum : int { kSplit = 8 };
template <int EPI_, int BM_, int BN_, int SUM_ = 1>
__global__ void __launch_bounds__(kThreads)
gemm_tc_small_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w0,
                     const __grid_constant__ CUtensorMap map_w1, const Params p) {
    constexpr int EPI = EPI_ & 7;
    constexpr bool FOLD = (EPI_ & kFold) != 0;
    constexpr bool kGate = EPI == RFK_GEMM_EPI_SWIGLU;
    constexpr bool SPLIT = (SUM_ & kSplit) != 0;
    constexpr int kSums = SUM_ == 4 ? 4 : 1;            // accumulators of this CTA
    static_assert(SUM_ == 1 || (SUM_ == 4 && kSums * BN_ <= 512) || SUM_ == (4 | kSplit), "a whole sum, or one of four quarters");
    static_assert(SUM_ == 1 || (FOLD && EPI == RFK_GEMM_EPI_RESIDUAL), "the form that is summed in quarters");
    constexpr bool kWhole = BM_ == 128 && BN_ == 128;   // producer and issuer run their loops as whole warps
    constexpr bool kLane0 = BM_ == 128 && BN_ == 64 && (EPI == RFK_GEMM_EPI_NONE || EPI == RFK_GEMM_EPI_RESIDUAL);   // the producer is lane 0
    constexpr int BN_OUT = kGate ? BN_ / 2 : BN_;
    using C = Cfg<BM_, BN_, SPLIT>;
    constexpr int kStages = C::kStages, kStage = C::kStageBytes, kBlock = C::kBlockBytes;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = tc::smem_addr(smem_raw);
    if (base & 1023u) {  // uniform over the CTA, nothing allocated yet
        if (threadIdx.x == 0) atomicCAS(&g_gemm_tc_error, 0, kErrSmemAlign);
        return;
    }
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + kStages * kStage);
    volatile int* abort_flag = &ctrl->abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int all_st = (p.K + kSub * BK - 1) / (kSub * BK);   // stages of K; a second block beyond K arrives as zeros
    const int piece = SPLIT ? blockIdx.x & 3 : 0, num_st = SPLIT ? all_st / 4 : all_st, st0 = piece * num_st;   // this CTA's
    const unsigned tile = SPLIT ? blockIdx.x >> 2 : blockIdx.x;
    // rows fastest, so that the tiles running together share weights; the heads form runs columns fastest, because the tiles
    // of 256 columns are one cluster
    const int m0 = (EPI == kEpiHeads && !FOLD ? tile / p.tiles_n : tile % p.tiles_m) * BM_;
    const int n0 = (EPI == kEpiHeads && !FOLD ? tile % p.tiles_n : tile / p.tiles_m) * BN_OUT;
    const bool want_ss = EPI == kEpiHeads && p.row_ss && ((p.ss_mask >> (n0 / (p.units * 64))) & 1);   // uniform over a cluster
    bool acc_ok = false;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { tc::mbar_init(&ctrl->full[s], 1); tc::mbar_init(&ctrl->empty[s], 1); }
        tc::mbar_init(&ctrl->acc_full, 1);
        tc::mbar_init(&ctrl->drain, 1);
        ctrl->abort = 0;
        tc::fence_barrier_init();
    }
    if (warp == 2) {   // beside the barriers
        tc::tmem_alloc(&ctrl->tmem_base, kSums * BN_);
        tc::tmem_relinquish();
    }
    if (warp == 1 && lane == 0) {   // descriptors are kernel arguments: fetched ahead of the wait for the kernel before
        tc::prefetch_tensormap(&map_a); tc::prefetch_tensormap(&map_w0);
        if (kGate) tc::prefetch_tensormap(&map_w1);
    }
    if (SPLIT) {                 // met again ahead of the first store into another CTA: by then all four run
        __syncwarp();
        pair::cluster_arrive();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem_cta = ctrl->tmem_base;
    // A folded layer's weights are no output of the kernel before (gemm_folded's callers see to it, or ask for pairs): a ring of them is asked for ahead of the wait for it (a view of 64 x 64 pixels 579 ->
    // 542 us, 128 x 128 658 -> 645, 320 x 320 1469 -> 1449; half a ring 556, 647, 1459).
    const int early = FOLD ? min(kStages, num_st) : 0;
    if (FOLD && warp == 0 && (kLane0 ? lane == 0 : tc::elect_one())) {
        for (int t = 0; t < early; ++t) {
            tc::mbar_arrive_expect_tx(&ctrl->full[t], kStage);
#pragma unroll
            for (int h = 0; h < kSub; ++h) {
                const uint32_t sW = base + t * kStage + h * kBlock + BM_ * BK * 2;
                const int x = ((st0 + t) * kSub + h) * BK;
                tma_load_2d(sW, &map_w0, x, n0, &ctrl->full[t]);
                if (kGate) tma_load_2d(sW + BN_OUT * BK * 2, &map_w1, x, n0, &ctrl->full[t]);
            }
        }
    }
    // Folded ones have asked for their ring above: the rest, for wide tiles only (views of 128 x 128 pixels 649.0 -> 645.6 us, 192 x 192 1145.5 ->
    // 1141.3, 256 x 256 1172.9 -> 1168.7; for every tile 64 x 64 pixels 535 -> 548).
    if (!FOLD || kWhole)
        prefetch_weights(warp == 0 && (kLane0 ? lane == 0 : tc::elect_one()), [&] {
            for (int t = early + m0 / BM_; t < num_st; t += p.tiles_m) {
#pragma unroll
                for (int h = 0; h < kSub; ++h) {
                    tma_prefetch_2d(&map_w0, (t * kSub + h) * BK, n0);
                    if (kGate) tma_prefetch_2d(&map_w1, (t * kSub + h) * BK, n0);
                }
            }
        });
    pdl_wait();      // set-up above is on-chip only; the operands are another kernel's output
    pdl_trigger();

    if (warp == 0) {
        // ------------------------------------------------------------ producer (one lane of the warp)
        const bool leader = kLane0 ? lane == 0 : tc::elect_one();
        if (kWhole || leader) {
            int it = 0, s = 0, par = 1;   // stage of `it`, and the parity of its barrier's previous phase
            for (; it < num_st; ++it) {
                if (it >= kStages && !(kWhole ? tc::mbar_wait_warp(&ctrl->empty[s], par, abort_flag) : tc::mbar_wait(&ctrl->empty[s], par, abort_flag)))
                    break;
                if (leader) {
                    if (it >= early) tc::mbar_arrive_expect_tx(&ctrl->full[s], kStage);
#pragma unroll
                    for (int h = 0; h < kSub; ++h) {
                        const uint32_t sA = base + s * kStage + h * kBlock, sW = sA + BM_ * BK * 2;
                        const int x = ((st0 + it) * kSub + h) * BK;
                        tma_load_2d(sA, &map_a, x, m0, &ctrl->full[s]);
                        if (it < early) continue;
                        tma_load_2d(sW, &map_w0, x, n0, &ctrl->full[s]);
                        if (kGate) tma_load_2d(sW + BN_OUT * BK * 2, &map_w1, x, n0, &ctrl->full[s]);
                    }
                }
                if (++s == kStages) { s = 0; par ^= 1; }
            }
            if (leader && *abort_flag) {   // giving up: wait (bounded) for the last copy of each stage before the CTA exits
                for (int t = 0; t < kStages && t < it; ++t) {
                    const int last = ((it - 1 - t) / kStages) * kStages + t;
                    tc::mbar_wait_drain(&ctrl->full[t], (last / kStages) & 1);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ issuer of the products (the warp's elected lane)
        constexpr uint32_t idesc = tc::umma_idesc_f16(BM_, BN_, 0);  // A and B both K-major
        const bool leader = tc::elect_one();
        bool ok = true;
        const int quarter = num_st / 4;
        int sum = 0;
        for (int it = 0; (kWhole || leader) && it < num_st; ++it) {
            if (kSums > 1 && it == (sum + 1) * quarter) ++sum;
            const int s = it % kStages;
            ok = kWhole ? tc::mbar_wait_warp(&ctrl->full[s], (it / kStages) & 1, abort_flag)
                        : tc::mbar_wait(&ctrl->full[s], (it / kStages) & 1, abort_flag);
            if (!ok) break;
            tc::tc_fence_after();
            if (leader) {
#pragma unroll
                for (int h = 0; h < kSub; ++h) {
                    const uint32_t a_lo = tc::umma_desc_lo(base + s * kStage + h * kBlock);
                    const uint32_t b_lo = tc::umma_desc_lo(base + s * kStage + h * kBlock + BM_ * BK * 2);
#pragma unroll
                    for (int ks = 0; ks < BK / 16; ++ks)  // 16 halves = 32 bytes along a swizzled row
                        tc::umma_f16_lo(kSums > 1 ? tmem_cta + sum * BN_ : tmem_cta, a_lo + ks * 2, b_lo + ks * 2, idesc,
                                        (kSums > 1 ? it > sum * quarter : it > 0) || (h > 0) || (ks > 0));
                }
                tc::umma_commit(&ctrl->empty[s]);
            }
        }
        if (leader) {
            if (ok) tc::umma_commit(&ctrl->acc_full);
            if (*abort_flag) {  // giving up: let this lane's products finish before tensor memory is freed
                tc::umma_commit(&ctrl->drain);
                tc::mbar_wait_drain(&ctrl->drain, 0);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue, warps 2-5
        const int lane_grp = warp & 3;                        // a warp reaches tensor-memory lanes [32 * (warp % 4), +32)
        // SPLIT: the CTA finishes the rows of one quarter of the tile, a warp 32 columns of them
        const int row_grp = SPLIT ? piece : lane_grp, first_c = SPLIT ? (lane_grp - piece) & 3 : 0;
        const int row = m0 + (BM_ == 64 ? row_grp * 16 + lane : row_grp * 32 + lane);
        const bool row_ok = row < p.M && (BM_ == 128 || lane < 16);
        const uint32_t t_acc = tmem_cta + ((uint32_t)(lane_grp * 32) << 16);
        __half* crow = p.C + (size_t)(row_ok ? row : 0) * p.ldc + n0;
        __half* rrow2 = nullptr;                              // kFold, residual: the row's place in raster order
        int ss_row = row;
        if (FOLD && EPI == RFK_GEMM_EPI_RESIDUAL && p.grid.bw && row_ok) {
            int view, by, bx;
            p.grid.block(row >> 4, view, by, bx);
            ss_row = p.grid.next(view, by, bx) * 16 + (row & 15);
            crow = p.C ? p.C + (size_t)ss_row * p.ldc + n0 : nullptr;
            if (p.raster) {
                const size_t at = ((size_t)view * p.grid.bh + by) * 4 + ((row >> 2) & 3);
                rrow2 = p.raster + (at * (p.grid.bw * 4) + bx * 4 + (row & 3)) * p.ldc + n0;
            }
        }
        constexpr bool kScaled = FOLD && EPI != RFK_GEMM_EPI_RESIDUAL;
        float factors[BN_OUT > 64 ? 2 : 1];                   // of the row, in each 64 columns
        float up_factor = 1.0f;
        if (kScaled) {
#pragma unroll
            for (int i = 0; i < (BN_OUT > 64 ? 2 : 1); ++i) factors[i] = column_factor(p, p.col_mul, n0 + 64 * i);
            if (kGate) up_factor = column_factor(p, p.up_mul, n0);
            const float row_mul = row_ok ? row_factor(p, row) : 1.0f;
#pragma unroll
            for (int i = 0; i < (BN_OUT > 64 ? 2 : 1); ++i) factors[i] *= row_mul;
            up_factor *= row_mul;
        }
        constexpr int kChunk = BN_OUT < 32 ? BN_OUT : 32;     // output columns per step
        uint4 res[EPI == RFK_GEMM_EPI_RESIDUAL ? BN_OUT / 8 : 1];
        if (EPI == RFK_GEMM_EPI_RESIDUAL) {                   // the row's residual arrives while the products run
            const __half* rrow = p.R + (size_t)(row_ok ? row : 0) * p.ldr + n0;
#pragma unroll
            for (int q = 0; q < BN_OUT / 8; ++q)
                res[q] = (row_ok && n0 + q * 8 < p.N && (!SPLIT || q / 4 == first_c)) ? *reinterpret_cast<const uint4*>(rrow + q * 8) : make_uint4(0, 0, 0, 0);
        }
        // Lane l of the first 16 holds columns 2l and 2l + 1 of each 32 of the bias (see the pair kernel's epilogue)
        constexpr bool kBiased = !FOLD && (EPI == RFK_GEMM_EPI_NONE || EPI == RFK_GEMM_EPI_RESIDUAL);
        uint32_t bias[kBiased ? BN_OUT / 32 : 1] = {};
        if (kBiased && p.bias) {
#pragma unroll
            for (int c = 0; c < BN_OUT / 32; ++c) {
                const int col = n0 + c * 32 + 2 * (lane & 15);
                if (col < p.N) bias[kBiased ? c : 0] = __ldg(reinterpret_cast<const uint32_t*>(p.bias + col));
            }
        }
        acc_ok = tc::mbar_wait_warp(&ctrl->acc_full, 0, abort_flag);
        constexpr int kRows = BM_ / 4, kPiece = kHandedPiece<BM_, BN_>;
        const int handed = C::kSmemBytes + (lane & (kRows - 1)) * 16;   // the row's first four columns, of the first piece
        if (SPLIT) {                                          // a warp's rows to the CTA of their quarter
            pair::cluster_wait();
            if (acc_ok) {
                tc::tc_fence_after();
                const int slot = lane_grp == piece ? 3 : piece < lane_grp ? piece : piece - 1;
                const uint32_t to = pair::map_to_cta(base + handed + slot * kPiece, lane_grp);
#pragma unroll
                for (int c = 0; c < BN_ / 32; ++c) {
                    uint32_t v[32];
                    tc::tmem_ld32(t_acc + c * 32, v);
                    tc::tc_wait_ld(v);
                    if (BM_ == 128 || lane < 16) {
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};"
                                         ::"r"(to + (c * 8 + q) * kRows * 16), "r"(v[4 * q]), "r"(v[4 * q + 1]), "r"(v[4 * q + 2]), "r"(v[4 * q + 3]) : "memory");
                    }
                }
            }
            __syncwarp();
            pair::cluster_arrive();
            pair::cluster_wait();
        }
        if ((EPI != kEpiHeads || FOLD) && acc_ok) {
            tc::tc_fence_after();
#pragma unroll
            for (int c = 0; c < BN_OUT / kChunk; ++c) {
                if (n0 + c * kChunk >= p.N) break;            // uniform over the CTA: the tile's tail lies beyond N
                if (SPLIT && c != first_c) continue;
                const float factor = factors[c * kChunk / 64];
                uint32_t v[32], o[kChunk / 2];
                if (!SPLIT) tc::tmem_ld32(t_acc + c * 32, v);
                if (SPLIT) {                                  // ((a + b) + c) + d, whichever of them is this CTA's
                    const float4* at = reinterpret_cast<const float4*>(smem_raw + handed) + c * 8 * kRows;
                    constexpr int kPiece4 = kPiece / 16;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 own = at[3 * kPiece4 + q * kRows], s0 = at[q * kRows], s1 = at[kPiece4 + q * kRows], s2 = at[2 * kPiece4 + q * kRows];
                        const auto sum = [&](float o, float a0, float a1, float a2) {
                            const float x1 = piece <= 1 ? o : a1, x2 = piece <= 1 ? a1 : piece == 2 ? o : a2, x3 = piece <= 2 ? a2 : o;
                            return __float_as_uint(((a0 + x1) + x2) + x3);   // (pieces 0 and 1 either way round)
                        };
                        v[4 * q] = sum(own.x, s0.x, s1.x, s2.x);
                        v[4 * q + 1] = sum(own.y, s0.y, s1.y, s2.y);
                        v[4 * q + 2] = sum(own.z, s0.z, s1.z, s2.z);
                        v[4 * q + 3] = sum(own.w, s0.w, s1.w, s2.w);
                    }
                } else if (kSums > 1) {
#pragma unroll
                    for (int a = 1; a < kSums; ++a) {
                        uint32_t u[32];
                        tc::tmem_ld32(t_acc + a * BN_ + c * 32, u);
                        if (a == 1) tc::tc_wait_ld(v);
                        tc::tc_wait_ld(u);
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(u[i]));
                    }
                }
                if (kGate) {
                    uint32_t u[32];
                    if (kChunk == 32) {
                        tc::tmem_ld32(t_acc + BN_OUT + c * 32, u);
                        tc::tc_wait_ld(v);
                        tc::tc_wait_ld(u);
                    } else {                                  // 16 gate and 16 up columns in one load
                        tc::tc_wait_ld(v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) u[i] = v[16 + i];
                    }
                    if (FOLD) {
#pragma unroll
                        for (int i = 0; i < kChunk; ++i) {
                            v[i] = __float_as_uint(__uint_as_float(v[i]) * factor);
                            u[i] = __float_as_uint(__uint_as_float(u[i]) * up_factor);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < kChunk; i += 2) {
                        const float g0 = __uint_as_float(v[i]), g1 = __uint_as_float(v[i + 1]);
                        // silu(g) * u = g * u / (1 + 2^(-g log2 e))
                        const float s0 = g0 * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * g0));
                        const float s1 = g1 * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * g1));
                        o[i >> 1] = pack_half2(s0 * __uint_as_float(u[i]), s1 * __uint_as_float(u[i + 1]));
                    }
                } else {
                    if (SUM_ == 1) tc::tc_wait_ld(v);
                    if (kBiased && p.bias) {
#pragma unroll
                        for (int i = 0; i < kChunk; i += 2) {
                            const float2 b = unpack_half2(__shfl_sync(0xffffffffu, bias[kBiased ? c : 0], i / 2));
                            // the unfused path rounds the product to fp16 before the bias is added (linear.cu:15-25)
                            v[i] = __float_as_uint(round_half(__uint_as_float(v[i])) + b.x);
                            v[i + 1] = __float_as_uint(round_half(__uint_as_float(v[i + 1])) + b.y);
                        }
                    }
                    if (EPI == RFK_GEMM_EPI_RESIDUAL) {
#pragma unroll
                        for (int i = 0; i < kChunk / 2; ++i) {
                            const uint4 w = res[EPI == RFK_GEMM_EPI_RESIDUAL ? c * 4 + i / 4 : 0];
                            const float2 rr = unpack_half2(i % 4 == 0 ? w.x : i % 4 == 1 ? w.y : i % 4 == 2 ? w.z : w.w);
                            o[i] = pack_half2(__uint_as_float(v[2 * i]) + rr.x, __uint_as_float(v[2 * i + 1]) + rr.y);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < kChunk / 2; ++i)
                            o[i] = FOLD ? pack_half2(__uint_as_float(v[2 * i]) * factor, __uint_as_float(v[2 * i + 1]) * factor)
                                        : pack_half2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                    }
                    if (FOLD && p.row_ss && row_ok) {         // the sum of the chunk's squares, as they are stored
                        const int part = EPI == kEpiHeads ? n0 / (p.units * 64) : 0, col = n0 + c * 32 - part * p.units * 64;
                        if constexpr (kChunk == 32) {
                            if (EPI != kEpiHeads || ((p.ss_mask >> part) & 1))
                                p.row_ss[((size_t)part * p.M + ss_row) * p.ss_tiles + (col >> 5)] = square_sum(o);
                        }
                    }
                }
                if (FOLD && EPI == kEpiHeads) {               // [part][group][head][seq][hd]
                    if (row_ok) {
                        const int hd = p.head_units * 64, heads = p.units / p.head_units, g = (n0 + c * 32) / 64, u = g % p.units;
                        __half* dst = p.C + (size_t)(g / p.units) * p.part_stride + ((size_t)(row / p.seq) * heads * p.out_seq + row % p.seq) * hd +
                                      (size_t)(u / p.head_units) * p.out_seq * hd + (u % p.head_units) * 64 + ((n0 / 32 + c) & 1) * 32;
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            *reinterpret_cast<uint4*>(dst + q * 8) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                    }
                } else if (row_ok) {
#pragma unroll
                    for (int q = 0; q < kChunk / 8; ++q) {
                        const int col = n0 + c * kChunk + q * 8;
                        const uint4 w = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                        if (col < p.N && (!FOLD || crow)) *reinterpret_cast<uint4*>(crow + c * kChunk + q * 8) = w;
                        if (FOLD && col < p.N && rrow2) *reinterpret_cast<uint4*>(rrow2 + c * kChunk + q * 8) = w;
                    }
                }
            }
        }
        __syncwarp();
    }

    if (SPLIT && warp < 2) {     // the other warps' share in the cluster's barriers
        pair::cluster_wait();
        pair::cluster_arrive();
        pair::cluster_wait();
    }
    if (EPI == kEpiHeads && !FOLD) {
        // ------------------------------------------------------------ epilogue of the head-split form
        // [part][group][head][seq][hd] by plain stores. The row statistic has the bits of the pair kernel's: one thread adds
        // a row's 256 squares in column order. So the cluster's tiles are gathered in its first CTA's ring, which is idle
        // once every CTA has its accumulator (first barrier), and summed there (second barrier).
        constexpr int kPitch = 512 + 16;                      // bytes per gathered row; the odd 16 bytes spread the banks
        static_assert(BM_ * kPitch <= kStages * kStage, "the gathered rows lie in the ring");
        const int lane_grp = warp & 3;
        const int local = BM_ == 64 ? lane_grp * 16 + lane : lane_grp * 32 + lane, row = m0 + local;
        const bool mine = warp >= 2 && (BM_ == 128 || lane < 16), row_ok = mine && row < p.M;
        // The gathering stores come ahead of the output's: the second barrier's arrival waits for the stores before it, and the output's
        // are on their way while the cluster meets (256 x 1024 x 1024 6.10 -> 5.68 us, 1600 x 1024 x 1024 9.89 -> 8.91).
        if (want_ss) pair::cluster_arrive();
        uint32_t o[BN_ / 2];
        if (warp >= 2 && acc_ok) {
            tc::tc_fence_after();
            const uint32_t t_acc = tmem_cta + ((uint32_t)(lane_grp * 32) << 16);
#pragma unroll
            for (int c = 0; c < BN_ / 32; ++c) {
                uint32_t v[32];
                tc::tmem_ld32(t_acc + c * 32, v);
                tc::tc_wait_ld(v);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[c * 16 + i] = pack_half2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
            }
        }
        if (want_ss) {
            __syncwarp();
            pair::cluster_wait();
            if (mine && acc_ok) {
                const uint32_t gather = pair::map_to_cta(base, 0) + local * kPitch + (n0 % 256) * 2;
#pragma unroll
                for (int q = 0; q < BN_ / 8; ++q)
                    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};"
                                 ::"r"(gather + q * 16), "r"(o[4 * q]), "r"(o[4 * q + 1]), "r"(o[4 * q + 2]), "r"(o[4 * q + 3]) : "memory");
            }
            __syncwarp();
            pair::cluster_arrive();
        }
        if (row_ok && acc_ok) {
            const int hd = p.head_units * 64, heads = p.units / p.head_units;
            const size_t rows_off = ((size_t)(row / p.seq) * heads * p.out_seq + row % p.seq) * hd;
#pragma unroll
            for (int c = 0; c < BN_ / 32; ++c) {
                const int g = (n0 + c * 32) / 64, u = g % p.units;   // 64-column unit over all parts, and within its part
                __half* dst = p.C + (size_t)(g / p.units) * p.part_stride + rows_off + (size_t)(u / p.head_units) * p.out_seq * hd +
                              (u % p.head_units) * 64 + (c & 1) * 32;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    *reinterpret_cast<uint4*>(dst + q * 8) = make_uint4(o[c * 16 + 4 * q], o[c * 16 + 4 * q + 1], o[c * 16 + 4 * q + 2], o[c * 16 + 4 * q + 3]);
            }
        }
        if (want_ss) {
            __syncwarp();
            pair::cluster_wait();
            if (pair::cluster_rank() == 0 && row_ok) {
                const uint4* src = reinterpret_cast<const uint4*>(smem_raw + local * kPitch);
                float ss = 0.0f;
#pragma unroll
                for (int q = 0; q < 32; ++q) {
                    const uint4 w = src[q];
                    const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 r2 = unpack_half2(x[i]);
                        ss = fmaf(r2.x, r2.x, ss);
                        ss = fmaf(r2.y, r2.y, ss);
                    }
                }
                const int dim = p.units * 64, part = n0 / dim;
                p.row_ss[((size_t)part * p.M + row) * (dim / 256) + (n0 % dim) / 256] = ss;
            }
            __syncwarp();
        }
    }

    // ---- teardown: every path (normal or aborted) arrives here with no divergence inside a warp
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem_cta, kSums * BN_);
    }
    if (tid == 0 && ctrl->abort) atomicCAS(&g_gemm_tc_error, 0, kErrTimeout);
}

}  // namespace small

// ------------------------------------------------------------------------------------------------
// The same product on CTA pairs: a cluster of two CTAs (two SMs of one TPC) owns a tile of 256 rows x 256 [or 192, narrow_tile]
// accumulator columns and one thread of the pair's first CTA issues tcgen05.mma.cta_group::2 (M = 256):
// each CTA stages only ITS 128 rows of A and ITS half of the weight tile (128 of the 256 [96 of the 192] accumulator
// columns' rows; with the SwiGLU epilogue CTA 0 holds the gate rows and CTA 1 the up rows), so a K block
// costs each SM 32 KB [28] of L2 -> shared-memory traffic instead of 48 KB for the same number of products.
// That traffic, not the tensor pipe, bounds the single-CTA kernel above (the same ~510 ns per K block on
// every shape = 14 TB/s over 148 SMs). Both accumulator halves live in the two CTAs' tensor memories at the
// same address; each CTA's epilogue warps drain their own 128 rows.
//   barriers: full[s] in CTA 0 collects both CTAs' copies (one arrive.expect_tx of 64 KB [56] by CTA 0); empty[s] and
//   acc_full[a] exist in both CTAs and are signalled together by one multicast tcgen05.commit;
//   acc_empty[a] in CTA 0 counts the 8 epilogue warps of the pair.
// The copies are ordinary per-CTA TMA loads (no cluster multicast), with the .cta_group::2 form that lets
// CTA 1's copies count on CTA 0's barrier.
namespace pair {

// The epilogue goes through shared memory both ways: an epilogue warp owns staging buffers of 32 rows x 64 halves
// (4 KB, the 128-byte-swizzled layout of a TMA box) for its 32 rows of the tile; it writes the finished fp16 values
// of 64 output columns there and one lane issues a TMA tile store, so the global writes are whole 128-byte lines
// issued by the copy engine instead of 16-byte pieces of 32 different rows per store instruction (measured:
// 2.8 us per tile for the register-to-global epilogue, most of it the scattered stores). With the residual
// epilogue the same buffers first receive the residual tile by TMA loads issued before the accumulator is ready
// (one buffer per 64-column unit, so the loads of a whole tile are in flight during its main loop); the sum
// overwrites the residual in place and is stored from there. Plain / SwiGLU / head-split: two buffers per warp in turn, one
// store after the other, over unit and tile ends alike: a unit may be written once at most one store is still reading, which is then
// the one before it, of the other buffer. (Counted from each tile's start instead, a tile of an odd number of units - 192 columns, or
// a tail of N - ends in the buffer that the next one begins with, whose last store may still be reading it.)
constexpr int kUnitCols = 64;
constexpr int kUnitBytes = 32 * kUnitCols * 2;       // 4 KB
// BN: accumulator columns of a tile, 256 or 192 (narrow_tile); 128 with SwiGLU (narrow_gate)
template <int EPI_, int BN> struct Cfg {
    static constexpr int EPI = EPI_ & 7;
    static constexpr int kStageBytes = kABytes + (BN == 128 ? 64 * BK * 2 : kWBoxBytes);   // 32 KB per CTA, of which a tile of 192 columns leaves 4 free, or 24
    static constexpr int kUnits = (EPI == RFK_GEMM_EPI_SWIGLU) ? BN / 128 : BN / 64;       // 64-column units per tile
    static constexpr int kBufsPerWarp = (EPI == RFK_GEMM_EPI_RESIDUAL) ? 4 : 2;
    static constexpr int kStagingBytes = 4 * kBufsPerWarp * kUnitBytes;                      // 4 epilogue warps
    static constexpr int kStages = BN == 128 ? 8 : (EPI == RFK_GEMM_EPI_RESIDUAL) ? 5 : 6;
    static constexpr int kSmemBytes = kStages * kStageBytes + kStagingBytes + 512;
    static_assert(kSmemBytes + 1024 <= 227 * 1024, "one CTA per SM");
};
constexpr int kMaxStages = 8;

struct __align__(8) Ctrl {
    uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], drain;
    uint64_t started;          // one phase only: the products of the CTA's first K block are complete
    uint64_t res_full[4][4];   // residual epilogue: [epilogue warp][unit], completes when that unit's residual box has landed
    uint32_t tmem_base;
    int abort;
};
static_assert(sizeof(Ctrl) <= 512, "control block");

// ---- shared <-> global tile copies used by the epilogue
__device__ __forceinline__ void tma_store_2d(const void* tmap, uint32_t src_smem, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(tmap), "r"(src_smem), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const void* tmap, uint32_t src_smem, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(tmap), "r"(src_smem), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_store_5d(const void* tmap, uint32_t src_smem, int c0, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
                 ::"l"(tmap), "r"(src_smem), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4) : "memory");
}
// Residual epilogue, before the tile's accumulator is waited for: bring the warp's residual rows of the whole tile
// into its four staging buffers. Lane 0 only. The buffers were last read by the TMA stores of the previous tile.
template <int EPI, int UNITS>
__device__ __forceinline__ void epilogue_prefetch_residual(const CUtensorMap* map_r, uint32_t stage_base, uint64_t* res_full,
                                                           int row0, int n0) {
    if (EPI != RFK_GEMM_EPI_RESIDUAL) return;
    bulk_wait_read<0>();
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {   // units beyond N are loaded too (all zeros): every barrier sees one phase per tile
        tc::mbar_arrive_expect_tx(&res_full[u], kUnitBytes);
        tma_load_2d(stage_base + u * kUnitBytes, map_r, n0 + u * kUnitCols, row0, &res_full[u]);
    }
}

// FOLD, residual: where a warp's 32 rows go
struct RowPlaces {
    int ss_row;        // the lane's sums of squares
    int block[2][3];   // view and place of the warp's two blocks, if rows move
    __device__ __forceinline__ RowPlaces(const Params& p, int row0, int lane) : ss_row(row0 + lane), block{} {
        if (!p.grid.bw) return;
#pragma unroll
        for (int h = 0; h < 2; ++h) p.grid.block((row0 >> 4) + h, block[h][0], block[h][1], block[h][2]);
        const int h = lane >> 4;
        ss_row = p.grid.next(h ? block[1][0] : block[0][0], h ? block[1][1] : block[0][1], h ? block[1][2] : block[0][2]) * 16 + (lane & 15);
    }
    // one lane: a unit's stores from its buffer
    __device__ __forceinline__ void store(const Params& p, const CUtensorMap* map_c, const CUtensorMap* map_raster, uint32_t buf, int col, int row0) const {
        if (!p.grid.bw) {
            tma_store_2d(map_c, buf, col, row0);   // rows >= M, columns >= N are clipped
        } else if (row0 < p.M) {                   // two blocks of 16 rows; M is a whole number of them, 32 at a time
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t src = buf + h * (kUnitBytes / 2);
                if (p.C) tma_store_2d(map_c, src, col, p.grid.next(block[h][0], block[h][1], block[h][2]) * 16);
                if (p.raster) tma_store_3d(map_raster, src, col, block[h][2] * 4, (block[h][0] * p.grid.bh + block[h][1]) * 4);
            }
        }
    }
};

// One epilogue warp, one tile: accumulator rows [lane] -> (bias / residual / gate) -> fp16 -> staging buffer -> TMA store.
// t_acc: tensor-memory address of the thread's accumulator row; row0: global row of the warp's lane 0. turn: the staging buffer of the
// next store, kept from tile to tile (not with the residual epilogue). factors (FOLD): of the row, in each unit.
// (Kept by the lanes, a unit each, and shuffled in the loop they cost a head-split tile 0.5 us: 1024 x 3072 x 1024 11.3, so 10.7, without any 10.6.)
template <int EPI_, int BN> struct UnitFactors {
    static constexpr int kUnits = Cfg<EPI_, BN>::kUnits;
    float own[kUnits], up[(EPI_ & 7) == RFK_GEMM_EPI_SWIGLU ? kUnits : 1];
    template <int N> static __device__ __forceinline__ float pick(const float (&f)[N], int u) {
        float v = f[0];
#pragma unroll
        for (int i = 1; i < N; ++i) v = u == i ? f[i] : v;
        return v;
    }
};
template <int EPI_, int BN>
__device__ __forceinline__ bool epilogue_tile_staged(const Params& p, const CUtensorMap* map_c, const CUtensorMap* map_raster, uint32_t t_acc,
                                                     const UnitFactors<EPI_, BN>& factors, unsigned char* stage_ptr, uint64_t* res_full, uint32_t res_parity,
                                                     int row0, int n0, int lane, int& turn, volatile int* abort_flag) {
    constexpr int EPI = EPI_ & 7;
    constexpr bool FOLD = (EPI_ & kFold) != 0;
    constexpr int kUnits = Cfg<EPI, BN>::kUnits;
    const uint32_t stage_base = tc::smem_addr(stage_ptr);
    uint32_t v[32];
    float ss = 0.0f;   // kEpiHeads: this row's sum of squares over the tile
    constexpr bool kPlaced = FOLD && EPI == RFK_GEMM_EPI_RESIDUAL;
    const RowPlaces places = kPlaced ? RowPlaces(p, row0, lane) : RowPlaces(Params{}, row0, lane);
    const int ss_row = places.ss_row;
    // Lane l holds columns 2l and 2l + 1 of a unit's bias, fetched a unit ahead. Each thread reading all 64 of them, one load's latency after the other, was
    // 2.5 us a tile: 262144 x 256 x 256 90.7 -> 57.5 us (54.7 without a bias), 65536 x 256 x 256 25.4 -> 15.8, 4096 x 1024 x 1024 13.4 -> 11.0, x 192 9.1 -> 6.7.
    constexpr bool kBiased = !FOLD && (EPI == RFK_GEMM_EPI_NONE || EPI == RFK_GEMM_EPI_RESIDUAL);
    const auto bias_of = [&](int u) {
        const int col = n0 + u * kUnitCols + 2 * lane;
        return kBiased && p.bias && u < kUnits && col < p.N ? __ldg(reinterpret_cast<const uint32_t*>(p.bias + col)) : 0u;
    };
    uint32_t bias_next = bias_of(0);
#pragma unroll 1
    for (int u = 0; u < kUnits; ++u) {
        const uint32_t bias_unit = bias_next;
        bias_next = bias_of(u + 1);
        const float factor = FOLD && EPI != RFK_GEMM_EPI_RESIDUAL ? factors.pick(factors.own, u) : 1.0f;
        const float up_factor = FOLD && EPI == RFK_GEMM_EPI_SWIGLU ? factors.pick(factors.up, u) : 1.0f;
        const int b = (EPI == RFK_GEMM_EPI_RESIDUAL) ? u : turn;
        unsigned char* buf = stage_ptr + b * kUnitBytes;
        if (EPI == RFK_GEMM_EPI_RESIDUAL) {                 // this unit's residual box has landed (also for units beyond N)
            if (!tc::mbar_wait_warp(&res_full[u], res_parity, abort_flag)) return false;
        }

        if (n0 + u * kUnitCols >= p.N) continue;            // uniform: the tile's tail lies beyond N
        if (EPI != RFK_GEMM_EPI_RESIDUAL) {                 // the store before the last one must have read this buffer
            if (lane == 0) bulk_wait_read<1>();
            __syncwarp();
        }
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {                    // two half units of 32 output columns
            const int c32 = u * 2 + hc;                     // 32-column chunk index within the tile's output
            uint32_t o[16];
            if (EPI == RFK_GEMM_EPI_SWIGLU) {
                uint32_t up[32];
                tc::tmem_ld32(t_acc + c32 * 32, v);          // gate columns
                tc::tmem_ld32(t_acc + BN / 2 + c32 * 32, up);   // up columns of the same hidden units
                tc::tc_wait_ld(v);
                tc::tc_wait_ld(up);
                if (FOLD) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        v[i] = __float_as_uint(__uint_as_float(v[i]) * factor);
                        up[i] = __float_as_uint(__uint_as_float(up[i]) * up_factor);
                    }
                }
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float g0 = __uint_as_float(v[i]), g1 = __uint_as_float(v[i + 1]);
                    // silu(g) * u = g * u / (1 + 2^(-g log2 e))
                    const float s0 = g0 * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * g0));
                    const float s1 = g1 * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * g1));
                    o[i >> 1] = pack_half2(s0 * __uint_as_float(up[i]), s1 * __uint_as_float(up[i + 1]));
                }
            } else {
                tc::tmem_ld32(t_acc + c32 * 32, v);
                uint4 res[4];
                if (EPI == RFK_GEMM_EPI_RESIDUAL) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) res[q] = *reinterpret_cast<const uint4*>(buf + staged(lane, hc * 4 + q));
                }
                tc::tc_wait_ld(v);
                if (kBiased && p.bias) {
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float2 bb = unpack_half2(__shfl_sync(0xffffffffu, bias_unit, hc * 16 + i / 2));
                        // the unfused path rounds the product to fp16 before the bias is added (linear.cu:15-25)
                        v[i] = __float_as_uint(round_half(__uint_as_float(v[i])) + bb.x);
                        v[i + 1] = __float_as_uint(round_half(__uint_as_float(v[i + 1])) + bb.y);
                    }
                }
                if (EPI == RFK_GEMM_EPI_RESIDUAL) {
                    const uint32_t* rw = reinterpret_cast<const uint32_t*>(res);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float2 rr = unpack_half2(rw[i]);
                        o[i] = pack_half2(__uint_as_float(v[2 * i]) + rr.x, __uint_as_float(v[2 * i + 1]) + rr.y);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        o[i] = FOLD ? pack_half2(__uint_as_float(v[2 * i]) * factor, __uint_as_float(v[2 * i + 1]) * factor)
                                    : pack_half2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                    if (EPI == kEpiHeads && !FOLD) {   // the norm that follows sees the stored fp16 values
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 r2 = unpack_half2(o[i]);
                            ss = fmaf(r2.x, r2.x, ss);
                            ss = fmaf(r2.y, r2.y, ss);
                        }
                    }
                }
            }
            if (FOLD && EPI != RFK_GEMM_EPI_SWIGLU) {
                const float part_ss = square_sum(o);
                if (BN == 256) {
                    ss = c32 == 0 ? part_ss : ss + part_ss;
                } else if (p.row_ss && row0 + lane < p.M) {
                    const int part = EPI == kEpiHeads ? n0 / (p.units * 64) : 0;
                    if (EPI != kEpiHeads || ((p.ss_mask >> part) & 1))
                        p.row_ss[((size_t)part * p.M + ss_row) * p.ss_tiles + (n0 >> 5) + c32 - part * p.units * 2] = part_ss;
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(buf + staged(lane, hc * 4 + q)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        }
        tc::fence_proxy_async();                            // the copy engine reads what the threads just wrote
        __syncwarp();
        if (lane == 0) {
            if (EPI == kEpiHeads) {
                const int g = (n0 + u * kUnitCols) / kUnitCols;   // 64-column unit over all parts
                tma_store_5d(map_c, stage_base + b * kUnitBytes, (g % p.head_units) * kUnitCols, row0 % p.seq,
                             (g % p.units) / p.head_units, row0 / p.seq, g / p.units);
            } else if (kPlaced) {
                places.store(p, map_c, map_raster, stage_base + b * kUnitBytes, n0 + u * kUnitCols, row0);
            } else {
                tma_store_2d(map_c, stage_base + b * kUnitBytes, n0 + u * kUnitCols, row0);   // rows >= M, columns >= N are clipped
            }
            bulk_commit();
        }
        turn ^= 1;
    }
    if (FOLD && EPI == RFK_GEMM_EPI_RESIDUAL && BN == 256 && p.row_ss && row0 + lane < p.M) p.row_ss[(size_t)ss_row * p.ss_tiles + n0 / 256] = ss;
    if (EPI == kEpiHeads && p.row_ss && (!FOLD || BN == 256)) {
        const int dim = p.units * kUnitCols, part = n0 / dim, row = row0 + lane;
        if (((p.ss_mask >> part) & 1) && row < p.M)
            p.row_ss[((size_t)part * p.M + row) * (dim / 256) + (n0 % dim) / 256] = ss;
    }
    return true;
}

// Sums in quarters of K (small tiles have the definition) for frames of many small views: each quarter is an accumulation of its own in the two accumulators in
// turn, and eight epilogue warps add them up in registers, 128 columns of a row a thread, under the next quarter's products. (Four accumulators of 128
// columns would read 24 KB a K block for half the products; small tiles, which read as much as this for half, were what such frames had.) us, small
// tiles in rounds / this / one sum on pairs, K = 4096, N = 1024: 2560 rows 34.8 / 31.0 / 24.0 (192 columns a tile), 4096 37.8 / 32.2 / 29.8, 8192 80.9 / 62.3 / 57.6,
// 16384 196 / 130 / 122; 2304, the most that small tiles take in one round, 19.7 there.
constexpr int kSumThreads = 64 + 8 * 32;   // ten warps, three on a scheduler: 168 registers a thread, of which the sums take 128
// 16 columns of the warp's rows, and the wait for them (tc::tmem_ld32 and tc::tc_wait_ld for fewer registers)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
template <int SUM> constexpr int kPairThreads = SUM == 4 ? kSumThreads : kThreads;
// One of those warps, one tile: the sums of its 32 rows x 128 columns -> residual -> fp16 -> staging buffers -> TMA stores, and squares
__device__ __forceinline__ bool epilogue_sums(const Params& p, const CUtensorMap* map_c, const CUtensorMap* map_raster, const float (&sum)[128],
                                              unsigned char* stage_ptr, uint64_t* res_full, uint32_t res_parity, int row0, int n0, int lane,
                                              volatile int* abort_flag) {
    const uint32_t stage_base = tc::smem_addr(stage_ptr);
    const RowPlaces places(p, row0, lane);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        unsigned char* buf = stage_ptr + u * kUnitBytes;
        if (!tc::mbar_wait_warp(&res_full[u], res_parity, abort_flag)) return false;
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {
            uint32_t o[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 res = *reinterpret_cast<const uint4*>(buf + staged(lane, hc * 4 + q));
                const uint32_t rw[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 rr = unpack_half2(rw[i]);
                    const int c = u * 64 + hc * 32 + q * 8 + 2 * i;
                    o[4 * q + i] = pack_half2(sum[c] + rr.x, sum[c + 1] + rr.y);
                }
            }
            if (p.row_ss && row0 + lane < p.M) p.row_ss[(size_t)places.ss_row * p.ss_tiles + (n0 >> 5) + u * 2 + hc] = square_sum(o);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(buf + staged(lane, hc * 4 + q)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        }
        tc::fence_proxy_async();                            // the copy engine reads what the threads just wrote
        __syncwarp();
        if (lane == 0) {
            places.store(p, map_c, map_raster, stage_base + u * kUnitBytes, n0 + u * kUnitCols, row0);
            bulk_commit();
        }
    }
    return true;
}

// SUM: one sum over K, or four of its quarters
template <int EPI_, int BN, int SUM = 1>
__global__ void __launch_bounds__(kPairThreads<SUM>, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w0,
                    const __grid_constant__ CUtensorMap map_w1, const __grid_constant__ CUtensorMap map_c,
                    const __grid_constant__ CUtensorMap map_r, const Params p) {
    constexpr int EPI = EPI_ & 7;
    constexpr bool FOLD = (EPI_ & kFold) != 0;
    static_assert(BN == 256 || (BN == 192 && EPI != RFK_GEMM_EPI_SWIGLU) || (BN == 128 && EPI == RFK_GEMM_EPI_SWIGLU), "whole 64-column units");
    static_assert(SUM == 1 || (SUM == 4 && BN == 256 && FOLD && EPI == RFK_GEMM_EPI_RESIDUAL), "the form that is summed in quarters");
    constexpr int BN_OUT = (EPI == RFK_GEMM_EPI_SWIGLU) ? BN / 2 : BN;
    constexpr int kStageBytes = Cfg<EPI, BN>::kStageBytes;
    constexpr int kTxBytes = kABytes + BN / 2 * BK * 2;   // of a stage, per CTA
    constexpr int kStages = Cfg<EPI, BN>::kStages;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = tc::smem_addr(smem_raw);
    const uint32_t rank = cluster_rank();            // 0: issues the products for the pair; 1: its peer
    unsigned char* staging = smem_raw + kStages * kStageBytes;   // 1024-byte aligned: the stages are 32 KB each
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(staging + Cfg<EPI, BN>::kStagingBytes);
    volatile int* abort_flag = &ctrl->abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) RFK_STAMP(0);   // kernel entry
    const int num_kb = (p.K + BK - 1) / BK;
    const int num_tiles = p.tiles_m * p.tiles_n;      // pair tiles: tiles_m counts 256-row blocks
    const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
    const bool aligned = (base & 1023u) == 0;         // the same in both CTAs (same kernel, same shared-memory layout)
    auto wait = [&](uint64_t* bar, uint32_t parity) { return tc::mbar_wait(bar, parity, abort_flag); };

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { tc::mbar_init(&ctrl->full[s], 1); tc::mbar_init(&ctrl->empty[s], 1); }
        for (int a = 0; a < 2; ++a) { tc::mbar_init(&ctrl->acc_full[a], 1); tc::mbar_init(&ctrl->acc_empty[a], (kPairThreads<SUM> - 64) / 16); }   // a warp of both CTAs each
        tc::mbar_init(&ctrl->drain, 1);
        tc::mbar_init(&ctrl->started, 1);
        for (int w = 0; w < 4; ++w)
            for (int u = 0; u < 4; ++u) tc::mbar_init(&ctrl->res_full[w][u], 1);
        ctrl->abort = 0;
        tc::fence_barrier_init();
    }
    __syncwarp();
    cluster_arrive();            // this CTA's barriers are initialised; the rest of the set-up runs under the cluster barrier's latency
    if (warp == 1 && lane == 0) {   // descriptors are kernel arguments: fetched ahead of the wait for the kernel before
        tc::prefetch_tensormap(&map_a); tc::prefetch_tensormap(rank == 0 || (FOLD && EPI == RFK_GEMM_EPI_RESIDUAL) ? &map_w0 : &map_w1); tc::prefetch_tensormap(&map_c);
        if (EPI == RFK_GEMM_EPI_RESIDUAL) tc::prefetch_tensormap(&map_r);
    }
    if (warp == 2 && aligned) {  // beside the barriers; the same in both CTAs of the pair
        tmem_alloc_pair(&ctrl->tmem_base, kTmemCols);
        tmem_relinquish_pair();
    }
    tc::tc_fence_before();
    __syncthreads();
    cluster_wait();              // both CTAs' barriers are initialised before either signals the other
    tc::tc_fence_after();
    if (!aligned) {
        if (tid == 0) atomicCAS(&g_gemm_tc_error, 0, kErrSmemAlign);
        return;
    }
    const uint32_t tmem_cta = ctrl->tmem_base;
    prefetch_weights(warp == 0 && tc::elect_one(), [&] {
        const void* map_w = rank == 0 || (FOLD && EPI == RFK_GEMM_EPI_RESIDUAL) ? (const void*)&map_w0 : (const void*)&map_w1;
        const int n0 = (first_tile / p.tiles_m) * BN_OUT, nw = (EPI == RFK_GEMM_EPI_SWIGLU || rank == 0) ? n0 : n0 + BN / 2;
        for (int kb = first_tile % p.tiles_m; kb < num_kb; kb += p.tiles_m) tma_prefetch_2d(map_w, kb * BK, nw);
    });
    pdl_wait();      // set-up above is on-chip only; the operands are another kernel's output
    pdl_trigger();
    if (tid == 0) RFK_STAMP(1);   // prologue done (barriers, tensor memory, cluster barrier)

    bool left = false, ok = true;   // left: this warp has made its half of the teardown's cluster barrier
    if (warp == 0) {
        // ------------------------------------------------------------ producer (an elected lane per CTA)
        if (tc::elect_one()) {
            // (FOLD, residual: map_w1 is the raster output's map)
            const void* map_w = rank == 0 || (FOLD && EPI == RFK_GEMM_EPI_RESIDUAL) ? (const void*)&map_w0 : (const void*)&map_w1;
            int it = 0;
            bool ok = true;
            for (int t = first_tile; ok && t < num_tiles; t += tile_step) {
                const int m0 = (t % p.tiles_m) * (2 * BM) + (int)rank * BM, n0 = (t / p.tiles_m) * BN_OUT;
                // this CTA's half of the weight tile: rows n0.. (CTA 0) / n0 + BN / 2.. (CTA 1) of W, or the gate / up rows
                const int nw = (EPI == RFK_GEMM_EPI_SWIGLU || rank == 0) ? n0 : n0 + BN / 2;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % kStages;
                    if (it >= kStages && !wait(&ctrl->empty[s], ((it / kStages) + 1) & 1)) { ok = false; break; }
                    const uint32_t sA = base + s * kStageBytes;
                    const uint32_t full0 = map_to_cta(tc::smem_addr(&ctrl->full[s]), 0);
                    // CTA 0 announces the bytes of both CTAs' copies on its own barrier (one local arrival); CTA 1 only
                    // copies. CTA 1's bytes may land before CTA 0's announcement: the phase still cannot complete before
                    // that arrival, and the transaction count balances once it is made.
                    if (rank == 0) tc::mbar_arrive_expect_tx(&ctrl->full[s], 2 * kTxBytes);
                    tma_load_2d_pair(sA, &map_a, kb * BK, m0, full0);
                    tma_load_2d_pair(sA + kABytes, map_w, kb * BK, nw, full0);
                }
            }
            if (*abort_flag) drain_pause();   // this CTA's copies count on CTA 0's barriers: give them time to land
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ issuer of the pair's products (an elected lane of CTA 0)
        // Under elect.sync a K block takes 543 clocks, inside `if (lane == 0)` 598 (the tensor pipe's own time: 512). A loop of the whole warp that issues under the same predicate needs 548, but the epilogue that
        // followed it took twice as long (4137 clocks for 2086), for a reason that its code does not show.
        // us, lane 0 / elected lane: 4096 x 1024 x 4096 + residual 27.9 / 26.4, w1|w3 + SwiGLU 48.1 / 46.1, 3072 x 1024 20.5 / 20.2.
        if (rank == 0 && tc::elect_one()) {
            constexpr uint32_t idesc = tc::umma_idesc_f16(2 * BM, BN, 0);
            const int sum_kb = SUM == 1 ? num_kb : num_kb / SUM;
            int it = 0, tl = 0;   // tl: accumulations, SUM a tile
            bool ok = true;
            for (int t = first_tile; ok && t < num_tiles; t += tile_step) {
                for (int q = 0; q < SUM; ++q, ++tl) {
                    const int acc = tl & 1;
                    if (tl >= 2) ok = wait_remote(&ctrl->acc_empty[acc], ((tl >> 1) + 1) & 1, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint32_t d_tmem = tmem_cta + acc * BNACC;
                    for (int kb = 0; kb < sum_kb; ++kb, ++it) {
                        const int s = it % kStages;
                        ok = wait(&ctrl->full[s], (it / kStages) & 1);
                        if (!ok) break;
                        if (it == 0) RFK_STAMP(2);   // first K block has landed
                        tc::tc_fence_after();
                        const uint32_t a_lo = tc::umma_desc_lo(base + s * kStageBytes);
                        const uint32_t b_lo = tc::umma_desc_lo(base + s * kStageBytes + kABytes);
#pragma unroll
                        for (int ks = 0; ks < BK / 16; ++ks)
                            umma_pair_f16_lo(d_tmem, a_lo + ks * 2, b_lo + ks * 2, idesc, (kb > 0) || (ks > 0));
                        umma_pair_commit(&ctrl->empty[s]);
                        if (EPI == RFK_GEMM_EPI_RESIDUAL && it == 0) umma_pair_commit(&ctrl->started);
                    }
                    if (!ok) break;
                    umma_pair_commit(&ctrl->acc_full[acc]);
                    if (tl == 0) RFK_STAMP(3);       // all products of the first tile issued
                }
            }
            if (*abort_flag) {
                umma_pair_commit(&ctrl->drain);
                tc::mbar_wait_drain(&ctrl->drain, 0);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue, warps 2-5 of both CTAs (2-9: 6-9 take a tile's second half of columns)
        const int lane_grp = warp & 3;                        // a warp reaches tensor-memory lanes [32 * (warp % 4), +32)
        const uint32_t lane_off = (uint32_t)(lane_grp * 32) << 16;
        const int unit0 = SUM == 4 ? (warp - 2) / 4 * 2 : 0;  // first unit
        unsigned char* my_stage = staging + (lane_grp * Cfg<EPI, BN>::kBufsPerWarp + unit0) * kUnitBytes;
        uint64_t* my_res = ctrl->res_full[lane_grp] + unit0;
        int tl = 0, turn = 0;
        for (int t = first_tile; t < num_tiles; t += tile_step, ++tl) {
            const bool last = t + tile_step >= num_tiles;
            const int acc = tl & 1;
            const int m0 = (t % p.tiles_m) * (2 * BM) + (int)rank * BM, n0 = (t / p.tiles_m) * BN_OUT;
            const int row0 = m0 + lane_grp * 32;
            if (lane == 0) {
                // The residual boxes of the CTA's first tile are asked for only once the first K block has been consumed
                // (a multicast commit): issued at kernel start they delay the first operand tiles by ~0.5 us. The barrier has one
                // phase, so a warp that comes late cannot miss it; empty[0] goes on to other phases.
                if (EPI == RFK_GEMM_EPI_RESIDUAL && tl == 0) tc::mbar_wait(&ctrl->started, 0, abort_flag);
                epilogue_prefetch_residual<EPI, SUM == 4 ? 2 : Cfg<EPI, BN>::kUnits>(&map_r, tc::smem_addr(my_stage), my_res, row0, n0 + unit0 * kUnitCols);
            }
            if constexpr (SUM == 4) {
                float sum[128];
#pragma unroll 1
                for (int q = 0; q < 4; ++q) {
                    const int n = 4 * tl + q, a = n & 1;
                    ok = tc::mbar_wait_warp(&ctrl->acc_full[a], (n >> 1) & 1, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after();
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        uint32_t v[16];
                        tmem_ld16(tmem_cta + lane_off + a * BNACC + unit0 * kUnitCols + c * 16, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) sum[c * 16 + i] = q == 0 ? __uint_as_float(v[i]) : sum[c * 16 + i] + __uint_as_float(v[i]);
                    }
                    tc::tc_fence_before();
                    __syncwarp();
                    if (last && q == 3) {   // nobody waits for the last one, see below
                        cluster_arrive();
                        left = true;
                    } else if (lane == 0) {
                        remote_arrive(map_to_cta(tc::smem_addr(&ctrl->acc_empty[a]), 0));
                    }
                }
                if (!ok) break;
                ok = epilogue_sums(p, &map_c, &map_w1, sum, my_stage, my_res, tl & 1, row0, n0 + unit0 * kUnitCols, lane, abort_flag);
                if (!ok) break;
                continue;
            }
            UnitFactors<EPI_, BN> factors;
            if (FOLD && EPI != RFK_GEMM_EPI_RESIDUAL) {
#pragma unroll
                for (int u = 0; u < Cfg<EPI_, BN>::kUnits; ++u) {
                    factors.own[u] = column_factor(p, p.col_mul, n0 + u * kUnitCols);
                    if (EPI == RFK_GEMM_EPI_SWIGLU) factors.up[u] = column_factor(p, p.up_mul, n0 + u * kUnitCols);
                }
                const float row_mul = row_factor(p, min(row0 + lane, p.M - 1));
#pragma unroll
                for (int u = 0; u < Cfg<EPI_, BN>::kUnits; ++u) {
                    factors.own[u] *= row_mul;
                    if (EPI == RFK_GEMM_EPI_SWIGLU) factors.up[u] *= row_mul;
                }
            }
            ok = tc::mbar_wait_warp(&ctrl->acc_full[acc], (tl >> 1) & 1, abort_flag);
            if (!ok) break;
            tc::tc_fence_after();
            if (tl == 0 && warp == 2 && lane == 0) RFK_STAMP(4);   // first tile's accumulator complete
            ok = epilogue_tile_staged<EPI_, BN>(p, &map_c, &map_w1, tmem_cta + lane_off + acc * BNACC, factors, my_stage, my_res, tl & 1,
                                                  row0, n0, lane, turn, abort_flag);
            if (!ok) break;
            if (tl == 0 && warp == 2 && lane == 0) RFK_STAMP(5);   // its epilogue done (stores issued)
            // every tcgen05.ld of this warp has completed: hand the accumulator back
            tc::tc_fence_before();
            __syncwarp();
            // Nobody waits for the last accumulator: the teardown's cluster barrier instead, under the stores' last reads (4096 x 1024 x 1024
            // 9.9 -> 9.65 us).
            if (last) {
                cluster_arrive();
                left = true;
            } else if (lane == 0) {
                remote_arrive(map_to_cta(tc::smem_addr(&ctrl->acc_empty[acc]), 0));
            }
        }
        // this lane's stores must have left shared memory (and, on an aborted run, its residual loads landed) before
        // the CTA gives the memory up
        if (lane == 0) {
            if (*abort_flag) drain_pause();
            bulk_wait_read<0>();   // the stores themselves complete with the grid; shared memory only has to outlive their reads
        }
        __syncwarp();
    }

    // ---- teardown: neither CTA leaves while the other may still signal its barriers or read its shared memory
    tc::tc_fence_before();
    if (!left) cluster_arrive();
    __syncthreads();
    cluster_wait();
    if (warp == 0) {
        tc::tc_fence_after();
        tmem_dealloc_pair(tmem_cta, kTmemCols);
    }
    if (tid == 0 && ctrl->abort) atomicCAS(&g_gemm_tc_error, 0, kErrTimeout);
    if (tid == 0) RFK_STAMP(6);   // CTA exit
}

}  // namespace pair
}  // namespace tcgemm

// 0 automatic (tcgen05 kernels when the shape allows: small tiles or CTA pairs by the rule of small_tile), 1 never (callers use
// their library GEMM), 2 CTA pairs whatever the size, 3 the single-CTA tcgen05 kernel. The environment variable RFK_GEMM_PATH
// sets the initial value, for side-by-side runs of an unchanged program.
static int initial_gemm_path() {
    const char* e = getenv("RFK_GEMM_PATH");
    return (e && e[0] >= '0' && e[0] <= '3' && e[1] == 0) ? e[0] - '0' : 0;
}
std::atomic<int> g_gemm_path{initial_gemm_path()};

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled, taken from the driver the runtime already has loaded (no link against libcuda)
EncodeTiledFn tensor_map_encoder() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// fp16 matrix [rows][cols] with a row pitch of ld elements; boxes of 128 rows x 64 columns in the
// 128-byte-swizzled layout; elements outside the matrix read as zeros
bool make_map_2d(CUtensorMap* m, const void* base, long long rows, long long cols, long long ld, int box_rows = 128) {
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int EPI>
int launch_gemm_single(const CUtensorMap& ma, const CUtensorMap& mw0, const CUtensorMap& mw1, tcgemm::Params p, int dev,
                       cudaStream_t st) {
    static std::atomic<bool> configured[64];
    static std::atomic<int> sm_count[64];
    if (!configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(tcgemm::gemm_tc_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             tcgemm::kSmemBytes);
        if (e != cudaSuccess) return (int)e;
        int n = 0;
        e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        sm_count[dev].store(n, std::memory_order_relaxed);
        configured[dev].store(true, std::memory_order_release);
    }
    const int tiles = p.tiles_m * p.tiles_n;
    const int grid = std::min(tiles, std::max(1, sm_count[dev].load(std::memory_order_relaxed)));
    launch_pdl(tcgemm::gemm_tc_kernel<EPI>, dim3(grid), dim3(tcgemm::kThreads), tcgemm::kSmemBytes, st, ma, mw0, mw1, p);
    return launch_status();
}

int sm_count(int dev) {
    static std::atomic<int> count[64];
    int n = count[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) { cudaGetLastError(); return 0; }
        count[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

std::atomic<int> g_pair_clusters[64];  // CTA pairs the device can run at once, per device (0 not asked yet, -1 none)

template <int EPI, int BN, int SUM = 1> cudaLaunchConfig_t pair_config(cudaLaunchAttribute (&attr)[2], cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see launch_pdl in common.cuh
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(tcgemm::pair::kPairThreads<SUM>); cfg.dynamicSmemBytes = tcgemm::pair::Cfg<EPI, BN>::kSmemBytes; cfg.stream = st;
    cfg.attrs = attr; cfg.numAttrs = g_pdl_enabled ? 2 : 1;
    return cfg;
}

// *pairs: how many CTA pairs of this form the device runs at once (asked once per device and form; every form takes a whole SM a CTA);
// RFK_EUNSUPPORTED where it cannot co-schedule pairs.
template <int EPI, int BN, int SUM = 1>
int resident_pairs(int dev, int* pairs) {
    static std::atomic<bool> configured[64];
    int nc = g_pair_clusters[dev].load(std::memory_order_acquire);
    if (nc == 0 || !configured[dev].load(std::memory_order_acquire)) {
        constexpr auto kernel = tcgemm::pair::gemm_tc_pair_kernel<EPI, BN, SUM>;
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = pair_config<EPI, BN, SUM>(attr, nullptr);
        cfg.numAttrs = 1;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
        if (e != cudaSuccess) return (int)e;
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        const int half = std::max(1, sms / 2);
        cfg.gridDim = dim3(2 * half);
        int n = 0;
        e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
        if (e != cudaSuccess) { cudaGetLastError(); n = 0; }
        nc = n > 0 ? std::min(n, half) : -1;
        g_pair_clusters[dev].store(nc, std::memory_order_release);
        configured[dev].store(true, std::memory_order_release);
    }
    *pairs = nc;
    return nc > 0 ? RFK_OK : RFK_EUNSUPPORTED;
}

// CTA-pair kernel: clusters of two; returns RFK_EUNSUPPORTED (nothing launched) when the device cannot co-schedule pairs
template <int EPI_, int BN, int SUM = 1>
int launch_pair_tiles(const CUtensorMap& ma, const CUtensorMap& mw0, const CUtensorMap& mw1, tcgemm::Params p, int dev,
                      cudaStream_t st, const CUtensorMap* heads_map) {
    constexpr int EPI = EPI_ & 7;
    constexpr auto kernel = tcgemm::pair::gemm_tc_pair_kernel<EPI_, BN, SUM>;
    // tile maps of the output (stores) and of the residual (loads): boxes of 32 rows x 64 columns, one per epilogue warp
    CUtensorMap mc, mr;
    if (heads_map) mc = *heads_map;
    if ((!heads_map && !make_map_2d(&mc, p.C ? p.C : p.raster, p.M, p.N, p.ldc, p.grid.bw ? 16 : 32)) ||
        !make_map_2d(&mr, EPI == RFK_GEMM_EPI_RESIDUAL ? (const void*)p.R : (const void*)p.C, p.M, p.N,
                     EPI == RFK_GEMM_EPI_RESIDUAL ? p.ldr : p.ldc, 32))
        return RFK_EUNSUPPORTED;
    int pairs = 0;
    const int rc = resident_pairs<EPI_, BN, SUM>(dev, &pairs);
    if (rc != RFK_OK) return rc;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = pair_config<EPI_, BN, SUM>(attr, st);
    p.tiles_m = (p.M + 2 * tcgemm::BM - 1) / (2 * tcgemm::BM);
    constexpr int BN_OUT = EPI == RFK_GEMM_EPI_SWIGLU ? BN / 2 : BN;
    p.tiles_n = (p.N + BN_OUT - 1) / BN_OUT;
    const int tiles = p.tiles_m * p.tiles_n;
    cfg.gridDim = dim3(2 * std::min(tiles, pairs));
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ma, mw0, mw1, mc, mr, p);
    if (e != cudaSuccess) { cudaGetLastError(); return (int)e; }
    return launch_status();
}

// Tiles of 192 accumulator columns instead of 256 where they need no more rounds of the pairs that the device places (resident_pairs): a
// K block of them takes three quarters of the products and seven eighths of the copies, and the bits are the same. us, 256 / 192: 2500 x 1024 x 4096 (0.54 and 0.81 rounds) 25.3 / 20.1,
// 4864 x 1024 x 4096 (1.03, 1.54) 42.8 / 34.7, 5665 x 1024 x 4096 (1.24, 1.86) 43.5 / 38.6, x 1024 14.6 / 12.8, 3136 x 3072 x 1024 (2.11, 2.81)
// 19.9 / 17.3. One round more loses even where three quarters of the rounds are fewer: 6400 x 3072 x 1024 (5, 6 rounds) 30.9 / 31.4,
// 3400 x 3072 x 1024 (3, 4) 20.0 / 20.6, 4096 x 1024 x 4096 (1, 2) 25.6 / 33.7, because a round that is not full runs its K blocks faster
// (0.30 us on few pairs, 0.36 to 0.45 on all).
bool narrow_tile(int M, int N, int pairs) {
    const long long rows = ceil_div(M, 2 * tcgemm::BM);
    const long long wide = ceil_div(rows * ceil_div(N, 256), pairs), narrow = ceil_div(rows * ceil_div(N, 192), pairs);
    return narrow == wide;
}

// W (and W_up) as in launch_gemm, for the boxes of the tile width; the head-split form with row statistics needs 256 columns, one sum
template <int EPI_>
int launch_gemm_pair(const CUtensorMap& ma, const void* W, const void* W_up, long long ldw, tcgemm::Params p, int dev, cudaStream_t st,
                     const CUtensorMap* heads_map = nullptr, const CUtensorMap* raster_map = nullptr, int* ss_tiles = nullptr) {
    constexpr int EPI = EPI_ & 7;
    constexpr bool FOLD = (EPI_ & tcgemm::kFold) != 0;
    constexpr bool kGate = EPI == RFK_GEMM_EPI_SWIGLU;
    CUtensorMap mw0, mw1;
    if constexpr (!kGate) {
        if (FOLD || !(EPI == tcgemm::kEpiHeads && p.row_ss)) {
            int pairs = 0;
            const int rc = resident_pairs<EPI_, 192>(dev, &pairs);
            if (rc != RFK_OK) return rc;
            // (a head-split tile with sums lies inside one part)
            if (narrow_tile(p.M, p.N, pairs) && !(FOLD && EPI == tcgemm::kEpiHeads && p.row_ss && p.units * 64 != p.N)) {
                if (FOLD) *ss_tiles = p.ss_tiles = p.N / 32;
                return make_map_2d(&mw0, W, p.N, p.K, ldw, 96)
                           ? launch_pair_tiles<EPI_, 192>(ma, mw0, raster_map ? *raster_map : mw0, p, dev, st, heads_map) : RFK_EUNSUPPORTED;
            }
        }
    }
    if (!make_map_2d(&mw0, W, p.N, p.K, ldw) || (kGate && !make_map_2d(&mw1, W_up, p.N, p.K, ldw))) return RFK_EUNSUPPORTED;
    return launch_pair_tiles<EPI_, 256>(ma, mw0, kGate ? mw1 : raster_map ? *raster_map : mw0, p, dev, st, heads_map);
}

// rank-5 map of a head-split output: [part][group][head][seq][hd] halves, boxes of 32 rows x 64 columns
bool make_map_heads(CUtensorMap* m, const void* base, int seq, int out_seq, int heads, int hd, long long groups, int parts,
                    long long part_stride) {
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t row = (cuuint64_t)hd * 2;
    const cuuint64_t dims[5] = {(cuuint64_t)hd, (cuuint64_t)seq, (cuuint64_t)heads, (cuuint64_t)groups, (cuuint64_t)parts};
    const cuuint64_t strides[4] = {row, (cuuint64_t)out_seq * row, (cuuint64_t)heads * out_seq * row, (cuuint64_t)part_stride * 2};
    const cuuint32_t box[5] = {64, 32, 1, 1, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- small tiles: their launch, and the rules that choose them
// CTAs of the head-split form on this tile that the device runs at once, in whole clusters of 256 columns (a cluster needs its
// SMs within one GPC): the occupancy query's answer, asked once per device. 0: it cannot place such a cluster at all. At most
// seven eighths of the SMs: the query gives 132 of 148 for clusters of four and all 148 for clusters of two, but a grid that
// takes every SM is no faster than CTA pairs (2304 x 1024 x 1024, 144 tiles of 128 x 128: 11.7 us, pairs 11.3).
template <int BM_, int BN_>
int heads_resident(int dev) {
    static std::atomic<int> asked[64];   // the answer + 1
    int n = asked[dev].load(std::memory_order_acquire);
    if (n == 0) {
        constexpr auto kernel = tcgemm::small::gemm_tc_small_kernel<tcgemm::kEpiHeads, BM_, BN_>;
        constexpr int smem = tcgemm::small::Cfg<BM_, BN_>::kSmemBytes, size = 256 / BN_;
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = size; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(size * std::max(1, sm_count(dev))); cfg.blockDim = dim3(tcgemm::kThreads); cfg.dynamicSmemBytes = smem;
        cfg.attrs = attr; cfg.numAttrs = 1;
        int clusters = 0;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
        if (e != cudaSuccess) { cudaGetLastError(); clusters = 0; }
        n = std::min(std::max(clusters, 0) * size, sm_count(dev) - sm_count(dev) / 8) + 1;
        asked[dev].store(n, std::memory_order_release);
    }
    return n - 1;
}

template <int EPI_, int BM_, int BN_, int SUM_ = 1>
int launch_gemm_small(const void* A, long long lda, const void* W, const void* W_up, long long ldw, tcgemm::Params p, int dev,
                      cudaStream_t st) {
    constexpr int EPI = EPI_ & 7;
    constexpr bool FOLD = (EPI_ & tcgemm::kFold) != 0;
    constexpr bool kGate = EPI == RFK_GEMM_EPI_SWIGLU;
    constexpr int BN_OUT = kGate ? BN_ / 2 : BN_;
    constexpr bool SPLIT = (SUM_ & tcgemm::small::kSplit) != 0;
    constexpr int smem = tcgemm::small::Cfg<BM_, BN_, SPLIT>::kSmemBytes + (SPLIT ? tcgemm::small::kHandedBytes<BM_, BN_> : 0);
    static_assert(smem + 1024 <= 227 * 1024, "shared memory of an SM");
    CUtensorMap ma, mw0, mw1;
    if (!make_map_2d(&ma, A, p.M, p.K, lda, BM_) || !make_map_2d(&mw0, W, p.N, p.K, ldw, BN_OUT)) return RFK_EUNSUPPORTED;
    if (!kGate) mw1 = mw0;
    else if (!make_map_2d(&mw1, W_up, p.N, p.K, ldw, BN_OUT)) return RFK_EUNSUPPORTED;
    static std::atomic<bool> configured[64];
    if (!configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(tcgemm::small::gemm_tc_small_kernel<EPI_, BM_, BN_, SUM_>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        configured[dev].store(true, std::memory_order_release);
    }
    p.tiles_m = (p.M + BM_ - 1) / BM_;
    p.tiles_n = (p.N + BN_OUT - 1) / BN_OUT;
    const dim3 grid((unsigned)(p.tiles_m * p.tiles_n) * (SPLIT ? 4 : 1));
    if ((EPI != tcgemm::kEpiHeads || FOLD) && !SPLIT) {   // the sums of a folded form need no cluster
        launch_pdl(tcgemm::small::gemm_tc_small_kernel<EPI_, BM_, BN_, SUM_>, grid, dim3(tcgemm::kThreads), smem, st, ma, mw0, mw1, p);
        return launch_status();
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SPLIT ? 4 : 256 / BN_; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see launch_pdl in common.cuh
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid; cfg.blockDim = dim3(tcgemm::kThreads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = attr; cfg.numAttrs = g_pdl_enabled ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, tcgemm::small::gemm_tc_small_kernel<EPI_, BM_, BN_, SUM_>, ma, mw0, mw1, p);
    if (e != cudaSuccess) { cudaGetLastError(); return (int)e; }
    return launch_status();
}

// The smallest tile whose tiles all run at once, one per SM; 0: none of them, the pair kernel. Smaller tiles take fewer
// operand bytes per K block and CTA, and a second round costs as much as the first. Measured on both sides of the line
// (us, small tile / pair kernel, weights from HBM): 256 x 1024 x 4096 10.9 / 24.5 (64 x 32), 1024 x 1024 x 1024 5.5 / 10.5
// (128 x 64), 2304 x 1024 x 4096 18.8 / 24.6 (128 x 128, 144 tiles); 3136 x 1024 x 4096 35.3 / 26.3 (200 tiles),
// 576 x 8192 x 1024 21.0 / 15.4 (320 tiles).
int small_tile(int M, int acc_cols, int sms) {
    constexpr int kTiles[4][2] = {{64, 32}, {64, 64}, {128, 64}, {128, 128}};   // rows, accumulator columns
    for (int i = 0; i < 4; ++i)
        if ((long long)ceil_div(M, kTiles[i][0]) * ceil_div(acc_cols, kTiles[i][1]) <= sms) return i + 1;
    return 0;
}

// The same rule for the head-split form, over its tiles of at least 64 columns: resident[i] CTAs of tile i run at once
// (heads_resident; 0: that tile cannot run). 1 to 3: the tile, 0: the pair kernel.
int heads_tile(int M, int N, const int* resident) {
    constexpr int kTiles[3][2] = {{64, 64}, {128, 64}, {128, 128}};
    for (int i = 0; i < 3; ++i)
        if ((long long)ceil_div(M, kTiles[i][0]) * ceil_div(N, kTiles[i][1]) <= resident[i]) return i + 1;
    return 0;
}

// Gate products whose small tiles would be 128 x 128: pairs with 64 hidden units each (128 accumulator columns), if they all run at once. A pair's CTA takes 24 KB
// a K block where a small tile takes 32, and 256 x 4096 hidden x 1024 is bound by what comes out of L2. us, small tiles / these, weights from HBM: 256 rows
// 8.10 / 7.59, 192 rows 7.98 / 7.57; a view of 128 x 128 pixels 634 / 630, an image of it 1087 / 1077, sixteen views of 64 x 64 in frames of four 2048 / 2014,
// an encoding of 200 triangles 604 / 595. RFK_EUNSUPPORTED: not that one.
template <int EPI_>
int launch_narrow_gate(const void* A, long long lda, const void* W, const void* W_up, long long ldw, const tcgemm::Params& p, int dev, cudaStream_t st) {
    int pairs = 0;
    if (small_tile(p.M, 2 * p.N, sm_count(dev)) != 4) return RFK_EUNSUPPORTED;
    const int rc = resident_pairs<EPI_, 128>(dev, &pairs);
    if (rc != RFK_OK || (long long)ceil_div(p.M, 256) * ceil_div(p.N, 64) > pairs) return RFK_EUNSUPPORTED;
    CUtensorMap ma, mw0, mw1;
    if (!make_map_2d(&ma, A, p.M, p.K, lda) || !make_map_2d(&mw0, W, p.N, p.K, ldw, 64) || !make_map_2d(&mw1, W_up, p.N, p.K, ldw, 64)) return RFK_EUNSUPPORTED;
    return launch_pair_tiles<EPI_, 128>(ma, mw0, mw1, p, dev, st, nullptr);
}

// path 0: small tiles or CTA pairs; path 2: CTA pairs; the single-CTA kernel if pairs are unavailable; path 3: that kernel
template <int EPI>
int launch_gemm(const void* A, long long lda, const void* W, const void* W_up, long long ldw, const tcgemm::Params& p, int dev,
                cudaStream_t st) {
    constexpr bool kGate = EPI == RFK_GEMM_EPI_SWIGLU;
    const int path = g_gemm_path.load(std::memory_order_relaxed);
    if (path == 0) {
        int rc = RFK_EUNSUPPORTED;
        if constexpr (kGate) rc = launch_narrow_gate<EPI>(A, lda, W, W_up, ldw, p, dev, st);
        if (rc != RFK_EUNSUPPORTED) return rc;
        switch (small_tile(p.M, kGate ? 2 * p.N : p.N, sm_count(dev))) {
            case 1: rc = launch_gemm_small<EPI, 64, 32>(A, lda, W, W_up, ldw, p, dev, st); break;
            case 2: rc = launch_gemm_small<EPI, 64, 64>(A, lda, W, W_up, ldw, p, dev, st); break;
            case 3: rc = launch_gemm_small<EPI, 128, 64>(A, lda, W, W_up, ldw, p, dev, st); break;
            case 4: rc = launch_gemm_small<EPI, 128, 128>(A, lda, W, W_up, ldw, p, dev, st); break;
        }
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    CUtensorMap ma, mw0, mw1;
    if (!make_map_2d(&ma, A, p.M, p.K, lda)) return RFK_EUNSUPPORTED;
    if (path != 3) {
        const int rc = launch_gemm_pair<EPI>(ma, W, W_up, ldw, p, dev, st);
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    if (!make_map_2d(&mw0, W, p.N, p.K, ldw) || !make_map_2d(&mw1, kGate ? W_up : W, p.N, p.K, ldw)) return RFK_EUNSUPPORTED;
    return launch_gemm_single<EPI>(ma, mw0, mw1, p, dev, st);
}

}  // namespace
}  // namespace rfk

using namespace rfk;

extern "C" int rfk_gemm_f16(const rfk_half* A, long long lda, const rfk_half* W, long long ldw, const rfk_half* W_up,
                            const rfk_half* bias, const rfk_half* R, long long ldr, rfk_half* C, long long ldc, int M,
                            int N, int K, int epilogue, rfk_stream_t stream) {
    if (!A || !W || !C || M < 0 || N <= 0 || K <= 0) return RFK_EINVAL;
    if (epilogue < RFK_GEMM_EPI_NONE || epilogue > RFK_GEMM_EPI_SWIGLU) return RFK_EINVAL;
    if (epilogue == RFK_GEMM_EPI_SWIGLU && (!W_up || bias)) return RFK_EINVAL;
    if (epilogue == RFK_GEMM_EPI_RESIDUAL && !R) return RFK_EINVAL;
    if (lda < K || ldw < K || ldc < N || (epilogue == RFK_GEMM_EPI_RESIDUAL && ldr < N)) return RFK_EINVAL;
    if (M == 0) return RFK_OK;
    if (g_gemm_path.load(std::memory_order_relaxed) == 1) return RFK_EUNSUPPORTED;
    // TMA needs 16-byte aligned bases and pitches; the epilogue moves 8 halves per access
    if ((lda | ldw | ldc | (epilogue == RFK_GEMM_EPI_RESIDUAL ? ldr : 0)) % 8 != 0 || N % 8 != 0 || K % 8 != 0)
        return RFK_EUNSUPPORTED;
    if (!aligned16(A) || !aligned16(W) || !aligned16(C) || (W_up && !aligned16(W_up)) || (R && !aligned16(R)) ||
        (bias && (reinterpret_cast<uintptr_t>(bias) & 3u)))
        return RFK_EUNSUPPORTED;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return RFK_EUNSUPPORTED;
    const bool swiglu = epilogue == RFK_GEMM_EPI_SWIGLU;
    tcgemm::Params p{};
    p.C = (__half*)C; p.ldc = ldc; p.R = (const __half*)R; p.ldr = ldr; p.bias = (const __half*)bias;
    p.M = M; p.N = N; p.K = K;
    p.tiles_m = (M + tcgemm::BM - 1) / tcgemm::BM;
    p.tiles_n = (N + (swiglu ? 128 : 256) - 1) / (swiglu ? 128 : 256);
    cudaStream_t st = as_stream(stream);
    switch (epilogue) {
        case RFK_GEMM_EPI_NONE: return launch_gemm<RFK_GEMM_EPI_NONE>(A, lda, W, W_up, ldw, p, dev, st);
        case RFK_GEMM_EPI_RESIDUAL: return launch_gemm<RFK_GEMM_EPI_RESIDUAL>(A, lda, W, W_up, ldw, p, dev, st);
        default: return launch_gemm<RFK_GEMM_EPI_SWIGLU>(A, lda, W, W_up, ldw, p, dev, st);
    }
}

int rfk::gemm_heads(const rfk_half* A, long long lda, const rfk_half* W, long long ldw, rfk_half* out, long long part_stride,
                    float* row_ss, int ss_parts_mask, int M, int N, int K, int seq_len, int out_seq, int num_heads,
                    int head_dim, rfk_stream_t stream) {
    if (!A || !W || !out || M < 0 || N <= 0 || K <= 0 || seq_len <= 0 || num_heads <= 0 || lda < K || ldw < K) return RFK_EINVAL;
    if (head_dim != 64 && head_dim != 128) return RFK_EUNSUPPORTED;
    const int dim = num_heads * head_dim;
    if (N % dim != 0 || (ss_parts_mask && !row_ss)) return RFK_EINVAL;
    const int parts = N / dim;
    if (parts > 1 && part_stride < (long long)M * dim) return RFK_EINVAL;
    if (M == 0) return RFK_OK;
    const int path = g_gemm_path.load(std::memory_order_relaxed);
    if (path == 1 || path == 3) return RFK_EUNSUPPORTED;   // the single-CTA kernel has no head-split epilogue
    // a 256-column tile must lie inside one part, a 32-row store box inside one group
    if (dim % 256 != 0 || M % seq_len != 0) return RFK_EUNSUPPORTED;
    if (out_seq < seq_len || (M != seq_len && (seq_len % 32 != 0 || out_seq != seq_len))) return RFK_EUNSUPPORTED;
    if ((lda | ldw | part_stride) % 8 != 0 || K % 8 != 0 || !aligned16(A) || !aligned16(W) || !aligned16(out) ||
        (row_ss && !aligned16(row_ss)))
        return RFK_EUNSUPPORTED;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return RFK_EUNSUPPORTED;
    tcgemm::Params p{};
    p.C = (__half*)out; p.ldc = N; p.M = M; p.N = N; p.K = K;
    p.row_ss = row_ss; p.seq = seq_len; p.units = dim / 64; p.head_units = head_dim / 64; p.ss_mask = ss_parts_mask;
    p.part_stride = part_stride; p.out_seq = out_seq;
    if (path == 0) {
        const int resident[3] = {heads_resident<64, 64>(dev), heads_resident<128, 64>(dev), heads_resident<128, 128>(dev)};
        const cudaStream_t st = as_stream(stream);
        int rc = RFK_EUNSUPPORTED;
        switch (heads_tile(M, N, resident)) {
            case 1: rc = launch_gemm_small<tcgemm::kEpiHeads, 64, 64>(A, lda, W, nullptr, ldw, p, dev, st); break;
            case 2: rc = launch_gemm_small<tcgemm::kEpiHeads, 128, 64>(A, lda, W, nullptr, ldw, p, dev, st); break;
            case 3: rc = launch_gemm_small<tcgemm::kEpiHeads, 128, 128>(A, lda, W, nullptr, ldw, p, dev, st); break;
        }
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    CUtensorMap ma, mh;
    if (!make_map_2d(&ma, A, M, K, lda) ||
        !make_map_heads(&mh, out, seq_len, out_seq, num_heads, head_dim, M / seq_len, parts, parts > 1 ? part_stride : (long long)M * dim))
        return RFK_EUNSUPPORTED;
    p.tiles_m = (M + tcgemm::BM - 1) / tcgemm::BM;
    p.tiles_n = N / 256;
    return launch_gemm_pair<tcgemm::kEpiHeads>(ma, W, nullptr, ldw, p, dev, as_stream(stream), &mh);
}

extern "C" int rfk_gemm_f16_heads(const rfk_half* A, long long lda, const rfk_half* W, long long ldw, rfk_half* out,
                                  long long part_stride, float* row_ss, int ss_parts_mask, int M, int N, int K, int seq_len,
                                  int num_heads, rfk_stream_t stream) {
    const int out_seq = seq_len % 32 == 0 ? seq_len : 0;   // 0: refused, as the header says
    return gemm_heads(A, lda, W, ldw, out, part_stride, row_ss, ss_parts_mask, M, N, K, seq_len, out_seq, num_heads, 64,
                      stream);
}

// 3-D map of a token grid in raster order, [height of all views][width][N] halves: boxes of 4 x 4 tokens x 64 columns
static bool make_map_raster(CUtensorMap* m, const void* base, int n, int width, long long height) {
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)width, (cuuint64_t)height};
    const cuuint64_t strides[2] = {(cuuint64_t)n * 2, (cuuint64_t)width * n * 2};
    const cuuint32_t box[3] = {64, 4, 4}, estr[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// small tiles, by the size of a product (SwiGLU aside)
static bool folded_small(int M, int N, int dev) {
    return g_gemm_path.load(std::memory_order_relaxed) == 0 && small_tile(M, N, sm_count(dev)) != 0;
}

// clusters of the split kernel that the device runs at once (asked once per device)
template <int BM_, int BN_> static int resident_quarters(int dev) {
    constexpr int SUM = 4 | tcgemm::small::kSplit;
    const auto kernel = tcgemm::small::gemm_tc_small_kernel<RFK_GEMM_EPI_RESIDUAL | tcgemm::kFold, BM_, BN_, SUM>;
    static std::atomic<int> asked[64];   // the answer + 1
    int n = asked[dev].load(std::memory_order_acquire);
    if (n == 0) {
        constexpr int smem = tcgemm::small::Cfg<BM_, BN_, true>::kSmemBytes + tcgemm::small::kHandedBytes<BM_, BN_>;
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 4; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(4 * 64); cfg.blockDim = dim3(tcgemm::kThreads); cfg.dynamicSmemBytes = smem;
        cfg.attrs = attr; cfg.numAttrs = 1;
        int clusters = 0;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
        if (e != cudaSuccess) { cudaGetLastError(); clusters = 0; }
        n = std::max(clusters, 0) + 1;
        asked[dev].store(n, std::memory_order_release);
    }
    return n - 1;
}

// A residual product summed in quarters (FoldedProduct::quarters): one cluster a tile where they all run at once, else a CTA a tile with the
// same sums where those do, else CTA pairs
static int launch_quarters(const FoldedProduct& f, const tcgemm::Params& p, int dev, cudaStream_t st) {
    constexpr int E = RFK_GEMM_EPI_RESIDUAL | tcgemm::kFold, kSplit = 4 | tcgemm::small::kSplit;
    if (!folded_small(p.M, p.N, dev)) {
        CUtensorMap ma, mw, mraster;
        if (!make_map_2d(&ma, f.A, p.M, p.K, p.K) || !make_map_2d(&mw, f.W, p.N, p.K, p.K) ||
            (p.raster && !make_map_raster(&mraster, p.raster, p.N, p.grid.bw * 4, p.M / (p.grid.bw * 4))))
            return RFK_EUNSUPPORTED;
        const int rc = launch_pair_tiles<E, 256, 4>(ma, mw, p.raster ? mraster : mw, p, dev, st, nullptr);
        if (rc != RFK_EUNSUPPORTED || g_gemm_path.load(std::memory_order_relaxed) == 2) return rc;
        return launch_gemm_small<E, 128, 128, 4>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
    }
    const auto tiles = [&](int bm, int bn) { return (long long)ceil_div(p.M, bm) * ceil_div(p.N, bn); };
    int rc = RFK_EUNSUPPORTED;
    if (tiles(64, 32) <= resident_quarters<64, 32>(dev)) rc = launch_gemm_small<E, 64, 32, kSplit>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
    else if (tiles(64, 64) <= resident_quarters<64, 64>(dev)) rc = launch_gemm_small<E, 64, 64, kSplit>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
    else if (tiles(128, 64) <= resident_quarters<128, 64>(dev)) rc = launch_gemm_small<E, 128, 64, kSplit>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
    if (rc == RFK_OK) return rc;
    switch (small_tile(p.M, p.N, sm_count(dev))) {
        case 1: return launch_gemm_small<E, 64, 32, 4>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
        case 2: return launch_gemm_small<E, 64, 64, 4>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
        case 3: return launch_gemm_small<E, 128, 64, 4>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
        default: return launch_gemm_small<E, 128, 128, 4>(f.A, p.K, f.W, nullptr, p.K, p, dev, st);
    }
}

bool rfk::folded_on_pairs(int M, int N) {
    int dev = 0;
    if (M <= 0 || N <= 0 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { cudaGetLastError(); return false; }
    return !folded_small(M, N, dev);
}

template <int EPI>
static int launch_folded(const FoldedProduct& f, tcgemm::Params p, int dev, cudaStream_t st, int* ss_tiles) {
    constexpr int E = EPI | tcgemm::kFold;
    constexpr bool kGate = EPI == RFK_GEMM_EPI_SWIGLU;
    const int sums = (EPI == tcgemm::kEpiHeads ? p.units * 64 : p.N) / 32;
    p.ss_tiles = sums;
    *ss_tiles = sums;
    if constexpr (EPI == RFK_GEMM_EPI_RESIDUAL)
        if (f.quarters) return launch_quarters(f, p, dev, st);
    if (g_gemm_path.load(std::memory_order_relaxed) == 0) {
        int rc = RFK_EUNSUPPORTED;
        if constexpr (kGate) rc = launch_narrow_gate<E>(f.A, p.K, f.W, f.W_up, p.K, p, dev, st);
        if (rc != RFK_EUNSUPPORTED) return rc;
        switch (small_tile(p.M, kGate ? 2 * p.N : p.N, sm_count(dev))) {
            case 1: rc = launch_gemm_small<E, 64, 32>(f.A, p.K, f.W, f.W_up, p.K, p, dev, st); break;
            case 2: rc = launch_gemm_small<E, 64, 64>(f.A, p.K, f.W, f.W_up, p.K, p, dev, st); break;
            case 3: rc = launch_gemm_small<E, 128, 64>(f.A, p.K, f.W, f.W_up, p.K, p, dev, st); break;
            case 4: rc = launch_gemm_small<E, 128, 128>(f.A, p.K, f.W, f.W_up, p.K, p, dev, st); break;
        }
        if (rc != RFK_EUNSUPPORTED) return rc;
    }
    p.ss_tiles = sums / 8;
    *ss_tiles = sums / 8;
    CUtensorMap ma, mh, mraster;
    if (!make_map_2d(&ma, f.A, p.M, p.K, p.K)) return RFK_EUNSUPPORTED;
    if (EPI == tcgemm::kEpiHeads &&
        !make_map_heads(&mh, f.C, p.seq, p.out_seq, p.units / p.head_units, p.head_units * 64, p.M / p.seq, p.N / (p.units * 64), p.part_stride))
        return RFK_EUNSUPPORTED;
    if (p.raster && !make_map_raster(&mraster, p.raster, p.N, p.grid.bw * 4, p.M / (p.grid.bw * 4))) return RFK_EUNSUPPORTED;
    return launch_gemm_pair<E>(ma, f.W, f.W_up, p.K, p, dev, st, EPI == tcgemm::kEpiHeads ? &mh : nullptr, p.raster ? &mraster : nullptr, ss_tiles);
}

int rfk::gemm_folded(const FoldedProduct& f, int* ss_tiles, rfk_stream_t stream, const FoldedMore& more) {
    const bool residual = f.R != nullptr, heads = f.num_heads > 0, gate = f.W_up != nullptr;
    if (!f.A || !f.W || (!f.C && !f.raster) || f.M <= 0 || f.N <= 0 || f.K <= 0 || residual + heads + gate != 1 || !ss_tiles) return RFK_EINVAL;
    if (!residual && (!f.in_ss || f.in_tiles <= 0)) return RFK_EINVAL;
    const int path = g_gemm_path.load(std::memory_order_relaxed), dim = heads ? f.num_heads * f.head_dim : f.N;
    if (path == 1 || path == 3) return RFK_EUNSUPPORTED;
    if ((f.M % 64 && !(heads && f.seq == f.M)) || f.K % 256 || f.N % dim || dim % 256) return RFK_EUNSUPPORTED;
    if (!aligned16(f.A) || !aligned16(f.W) || !aligned16(f.W_up) || !aligned16(f.R) || !aligned16(f.C) || !aligned16(f.raster) ||
        !aligned16(f.in_ss) || !aligned16(f.out_ss))
        return RFK_EUNSUPPORTED;
    if (!residual && f.in_tiles != f.K / 256 && f.in_tiles != f.K / 32) return RFK_EINVAL;
    if (heads && ((f.head_dim != 64 && f.head_dim != 128) || f.seq <= 0 || (f.seq % 32 && f.seq != f.M) || f.M % f.seq || (f.out_seq && (f.seq != f.M || f.out_seq < f.seq)) ||
                  (f.N > dim && f.part_stride < (long long)f.M * dim) || f.part_stride % 8))
        return RFK_EUNSUPPORTED;
    if (f.blocks_across && (!residual || f.blocks_across % 2 || f.blocks_down % 2 || f.blocks_down <= 0 || f.M % (f.blocks_across * f.blocks_down * 16)))
        return RFK_EUNSUPPORTED;
    if (!f.blocks_across && (f.raster || !f.C)) return RFK_EINVAL;
    if (f.quarters && (!residual || f.K % 512)) return RFK_EUNSUPPORTED;
    if ((more.w_mul || more.w_up_mul) && (residual || gate != (more.w_up_mul != nullptr) || !more.w_mul)) return RFK_EINVAL;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return RFK_EUNSUPPORTED;
    // (pairs of 192 columns write sums of 32 too: head-split products of several parts have none, see launch_gemm_pair)
    if (more.pairs && (!heads || f.N == dim || !f.out_ss || folded_small(f.M, f.N, dev))) return RFK_EUNSUPPORTED;
    tcgemm::Params p{};
    p.C = (__half*)f.C; p.ldc = f.N; p.R = (const __half*)f.R; p.ldr = f.N;
    p.M = f.M; p.N = f.N; p.K = f.K;
    p.tiles_m = (f.M + tcgemm::BM - 1) / tcgemm::BM;
    p.tiles_n = (f.N + (gate ? 128 : 256) - 1) / (gate ? 128 : 256);
    p.in_ss = f.in_ss; p.in_tiles = f.in_tiles; p.in_group = f.in_tiles == f.K / 256 ? 1 : 8;
    p.in_inv_dim = 1.0f / (float)f.K; p.in_eps = f.eps; p.in_mul = f.in_mul;
    p.row_ss = f.out_ss;
    p.raster = (__half*)f.raster;
    p.grid = tcgemm::Grid{f.blocks_across, f.blocks_down, f.shift_from, f.shift_to};
    if (heads) {
        p.seq = f.seq; p.out_seq = f.out_seq ? f.out_seq : f.seq; p.units = dim / 64; p.head_units = f.head_dim / 64; p.ss_mask = f.ss_mask;
        p.part_stride = f.N > dim ? f.part_stride : (long long)f.M * dim;
    }
    p.col_mul = more.w_mul;
    p.up_mul = more.w_up_mul;
    const cudaStream_t st = as_stream(stream);
    return gate ? launch_folded<RFK_GEMM_EPI_SWIGLU>(f, p, dev, st, ss_tiles)
                : heads ? launch_folded<tcgemm::kEpiHeads>(f, p, dev, st, ss_tiles) : launch_folded<RFK_GEMM_EPI_RESIDUAL>(f, p, dev, st, ss_tiles);
}

extern "C" int rfk_gemm_folded(const rfk::FoldedProduct* f, int* ss_tiles, rfk_stream_t stream) { return f ? rfk::gemm_folded(*f, ss_tiles, stream) : RFK_EINVAL; }
extern "C" int rfk_gemm_folded_more(const rfk::FoldedProduct* f, const rfk::FoldedMore* more, int* ss_tiles, rfk_stream_t stream) {
    return f && more ? rfk::gemm_folded(*f, ss_tiles, stream, *more) : RFK_EINVAL;
}
extern "C" int rfk_folded_on_pairs(int M, int N) { return rfk::folded_on_pairs(M, N); }

extern "C" int rfk_gemm_heads_tile(int M, int N, const int* resident) {
    return M > 0 && N > 0 && resident ? heads_tile(M, N, resident) : RFK_EINVAL;
}

extern "C" int rfk_gemm_pair_tile(int M, int N, int pairs) {
    return M > 0 && N > 0 && pairs > 0 ? (narrow_tile(M, N, pairs) ? 192 : 256) : RFK_EINVAL;
}

extern "C" int rfk_gemm_pair_clusters(void) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    return g_pair_clusters[dev].load(std::memory_order_relaxed);
}

#ifdef RFK_GEMM_TIMELINE
extern "C" int rfk_gemm_timeline(unsigned long long* host_out8) {
    return (int)cudaMemcpyFromSymbol(host_out8, tcgemm::g_timeline, 16 * sizeof(unsigned long long));
}
#endif

extern "C" int rfk_gemm_set_path(int path) {
    if (path < 0 || path > 3) return RFK_EINVAL;
    g_gemm_path.store(path, std::memory_order_relaxed);
    return RFK_OK;
}

extern "C" int rfk_gemm_error(int* code, int clear) {
    if (!code) return RFK_EINVAL;
    cudaError_t e = cudaMemcpyFromSymbol(code, g_gemm_tc_error, sizeof(int));
    if (e != cudaSuccess) return (int)e;
    if (clear) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_gemm_tc_error, &zero, sizeof(int));
        if (e != cudaSuccess) return (int)e;
    }
    return RFK_OK;
}
