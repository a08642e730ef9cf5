// 3x3 convolution, stride 1, padding 1, channels-last fp16, as an implicit GEMM on CTA pairs (tcgen05 + tensor memory + TMA), with the
// element-wise steps that follow it in the DPT head as its epilogue:
//   out = act(half(conv(x, w)) + bias) (+ residual), every intermediate rounded to fp16 as by the separate operators;
//   and, if asked, silu(out) beside it, the operand of the residual unit that follows.
// Reference boundary: rf::conv2d and the residual units of rf::dpt_forward, src/layers/dpt.cu:100-178, :397-409 of
// BANANASJIM/renderformer-cuda.
//
// A pair of CTAs owns two boxes of pixels (one per CTA, 16 x 8 or 8 x 8) x BN output channels. The GEMM's rows are pixels and its K index is
// (tap, input channel): a K block is 64 channels of one tap. The three taps of a row of taps read the same pixels but for a shift by one
// column, so a box comes with a column on either side, once for the three of them, by one TMA copy of a rank-4 map that has a column's pixels one
// after the other ([c][y][x][n]): 8 pixels of a column are one 8-row group of the tensor core's swizzled layout, and a tap's operand
// starts one group further. Pixels beyond the image arrive as zeros, which is the padding. So no patch matrix exists, and a K block
// brings 6 KB of pixels into an SM instead of the 16 that a box per tap takes.
// Otherwise the kernel is the projection kernel's (gemm_tc.cu: pair tiles, ring of operand stages filled by per-CTA copies that
// count on CTA 0's barrier, two accumulators so that a tile's epilogue runs under the next tile's products, staged TMA stores).
//
// Order of the sums. The library kernels that this replaces add the K blocks in one of two orders, and images rest on the bits:
//   taps inside  for each 64 input channels: the nine taps        (its implicit-GEMM kernels)
//   rows outside for each row of taps: for each 64 channels: the three taps of that row   (its weight-stationary kernels)
// The caller names the order (dpt.cu finds out, size by size, which the library takes); both cost the same here.
// Bound, by the tile (a K block of a pair, clocks): 128 channels x 2 x 128 pixels 260 with few pairs at work, which is the tensor pipe's own 256, and
// 350 with all of them, where 14 KB a K block and SM are 11 TB/s out of L2; 64 x 2 x 128 177, 64 x 2 x 64 125: the tensor core's reads of the pixels
// from shared memory, for fewer products each. To that a launch adds 3 to 4 us, of which the last tile's epilogue is 1.4 us for each 64
// channels x 128 pixels. us, with bias and SiLU, a box per tap and tiles of 256 channels / now: 256 -> 256 at 256 x 256 57.0 / 51.5 (1.5 PFLOP/s), at 128 x 128
// 20.9 / 18, 64 x 64 19.6 / 8.6, 32 x 32 19.0 / 6.2; 256 -> 128 at 512 x 512 144 / 107; 1024 -> 256 at 32 x 32 49 / 14.2. Tiles of 256 channels with the boxes shared
// were slower up to 352 x 352 (98 for 100 there; 224 x 224 42.6 for 41.0, 128 x 128 21.3 for 18), 5 percent faster at 512 x 512, beyond the maps of
// images that a session makes, and need a ring of their own for the weights: not kept.
// Weights of at most 128 -> 32 channels stay in shared memory (BN = 32): 320 x 320 23.0 / 16.0, 512 x 512 58 / 38 against a stream of them in tiles of 64.
#include <algorithm>
#include <cuda.h>  // CUtensorMap and its enums; the encoder itself is looked up at run time
#include "common.cuh"
#include "dpt_math.cuh"
#include "kernels_internal.h"
#include "tc_pair.cuh"

namespace rfk {

__device__ int g_conv_tc_error = 0;  // first time-out / failure code seen by any CTA since load

namespace tcconv {
using namespace pair_ptx;

constexpr int BK = 64, kBoxY = 8;
constexpr int kThreads = 192;                    // warp 0 producer, warp 1 issuer of the products, warps 2-5 epilogue
constexpr int kResidentBlocks = 2;               // blocks of 64 input channels whose weights fit beside the boxes (32 output channels)
constexpr int kColBytes = kBoxY * BK * 2;        // a column of 8 pixels: one 8-row group of the tensor core's layout
static_assert(kColBytes == 1024, "a tap's operand starts on the swizzle's period");

// BN output channels x a box of BX x 8 pixels per CTA
template <int BN, int BX> struct Cfg {
    static constexpr int kRows = BX * kBoxY;
    static_assert(kRows == 128 || (kRows == 64 && BN == 64), "the tensor core's tiles of a pair that are used here");
    static constexpr int kHaloBytes = (BX + 2) * kColBytes;  // the box with a column of pixels on either side
    // The ring's stages hold a halo box and the weights of its three taps, so that one barrier serves three K blocks. kResident: boxes
    // alone, the weights come once, ahead of the first tile.
    static constexpr bool kResident = BN == 32;
    static constexpr int kWBytes = BN / 2 * BK * 2;          // this CTA's half of a tap's weights
    static constexpr int kStages = BN == 128 ? 4 : BN == 32 ? 9 : kRows == 64 ? 4 : 3;
    static constexpr int kWTiles = kResident ? 9 * kResidentBlocks : 3 * kStages;
    static constexpr int kStageTx = 2 * (kHaloBytes + (kResident ? 0 : 3 * kWBytes));   // what a stage's barrier counts, of both CTAs
    // An accumulator: a row's channels in the lane of that row, or, with 64 rows, the second half of them in the lane 64 further
    static constexpr int kAccCols = kRows == 64 ? BN / 2 : BN;
    static constexpr int kUnitCh = kAccCols < 64 ? kAccCols : 64;   // the epilogue's units: 32 pixels x kUnitCh channels, a staging buffer each
    static constexpr int kUnitBytes = 32 * kUnitCh * 2;
    static constexpr int kUnits = kAccCols / kUnitCh;
    static constexpr int kStagingBytes = 4 * kUnits * kUnitBytes;
    static constexpr int kSmemBytes = kStages * kHaloBytes + kWTiles * kWBytes + kStagingBytes + 512;
    static constexpr int kCtas = BN == 64 ? 2 : 1;           // of an SM
    static_assert(kCtas * (kSmemBytes + 1024) <= 227 * 1024 && kCtas * 2 * kAccCols <= 512, "shared and tensor memory of an SM");
    // 16-byte chunk j of pixel r in a staging buffer, in the copy engine's swizzled layout (128-byte rows, or 64-byte ones)
    static __device__ __forceinline__ uint32_t chunk(int r, int j) {
        return kUnitCh == 64 ? staged(r, j) : (uint32_t)(r * 64 + ((j ^ ((r >> 1) & 3)) << 4));
    }
};

struct __align__(8) Ctrl {
    uint64_t full[9], empty[9];
    uint64_t weights;          // kResident: all of them have landed; one phase
    uint64_t acc_full[2], acc_empty[2], drain;
    uint64_t started;          // one phase only: the products of the CTA's first K block are complete
    uint64_t res_full[4][4];   // [epilogue warp][unit]: that unit's residual box has landed
    uint32_t tmem_base;
    int abort;
};
static_assert(sizeof(Ctrl) <= 512, "control block");

enum : int { kErrTimeout = 1, kErrSmemAlign = 2 };

struct Params {
    const __half* bias;
    int tiles, tiles_x, tiles_img;    // boxes in all images, per row of an image, per image
    int tiles_m, tiles_n;             // pairs of boxes, blocks of BN output channels
    int cb, c_out;                    // blocks of 64 input channels; output channels
    int rows_outside, silu, has_res, dual;
    const __half* sum;                // ADD: [N][H][W][c_out] to which the output is added (it may be the output)
    int H, W;
};

// boxes of pixels: the maps have the columns' pixels (y) ahead of the rows' (x), see make_map_pixels
__device__ __forceinline__ void tma_load_4d_pair(uint32_t dst, const void* map, int c, int x, int y, int n, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c), "r"(y), "r"(x), "r"(n), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* map, int c, int n, int tap, uint32_t cluster_bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c), "r"(n), "r"(tap), "r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tma_prefetch_3d(const void* map, int c, int n, int tap) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(map), "r"(c), "r"(n), "r"(tap) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* map, int c, int x, int y, int n, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c), "r"(y), "r"(x), "r"(n), "r"(tc::smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tma_store_4d(const void* map, uint32_t src, int c, int x, int y, int n) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(c), "r"(y), "r"(x), "r"(n) : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_half2(uint32_t w) { return __half22float2(*reinterpret_cast<__half2*>(&w)); }

struct Box { int x, y, n; };   // first pixel of a CTA's box, and its image
template <int BX> __device__ __forceinline__ Box box_of(const Params& p, int tile) {
    const int n = tile / p.tiles_img, r = tile - n * p.tiles_img, ty = r / p.tiles_x;
    return {(r - ty * p.tiles_x) * BX, ty * kBoxY, n};
}

// from one box's block of input channels and row of taps to the next one's
__device__ __forceinline__ void step(const Params& p, int& c, int& ty) {
    if (p.rows_outside) { if (++c == p.cb) { c = 0; ++ty; } }
    else if (++ty == 3) { ty = 0; ++c; }
}

// ADD: the output is what the epilogue has made so far plus p.sum, whose values a thread reads itself, half a unit ahead (the staging buffers hold the
// residual). That takes a pass over four maps (19 us at 256 x 256 x 256) out of a fusion block: an image of 512 x 512 4930 -> 4877 us,
// of 128 x 128 1086 -> 1082, of 320 x 320 no difference. Forms without it keep their registers.
template <int BN, int BX, bool ADD>
__global__ void __launch_bounds__(kThreads, (Cfg<BN, BX>::kCtas))
conv3x3_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ CUtensorMap map_o, const __grid_constant__ CUtensorMap map_r,
                    const __grid_constant__ CUtensorMap map_s, const Params p) {
    using C = Cfg<BN, BX>;
    constexpr int kStages = C::kStages, kUnits = C::kUnits, kUnitBytes = C::kUnitBytes, kUnitCh = C::kUnitCh, kTmemCols = 2 * C::kAccCols < 32 ? 32 : 2 * C::kAccCols;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = tc::smem_addr(smem_raw);
    const uint32_t rank = cluster_rank();            // 0: issues the products for the pair; 1: its peer
    const uint32_t base_w = base + kStages * C::kHaloBytes;
    unsigned char* staging = smem_raw + kStages * C::kHaloBytes + C::kWTiles * C::kWBytes;
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(staging + C::kStagingBytes);
    volatile int* abort_flag = &ctrl->abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int num_boxes = 3 * p.cb;                  // halo boxes a tile: one for each row of taps and block of 64 input channels
    const int num_tiles = p.tiles_m * p.tiles_n;
    const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
    const bool aligned = (base & 1023u) == 0;        // the same in both CTAs (same kernel, same shared-memory layout)

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { tc::mbar_init(&ctrl->full[s], 1); tc::mbar_init(&ctrl->empty[s], 1); }
        tc::mbar_init(&ctrl->weights, 1);
        for (int a = 0; a < 2; ++a) { tc::mbar_init(&ctrl->acc_full[a], 1); tc::mbar_init(&ctrl->acc_empty[a], 8); }
        tc::mbar_init(&ctrl->drain, 1);
        tc::mbar_init(&ctrl->started, 1);
        for (int w = 0; w < 4; ++w)
            for (int u = 0; u < 4; ++u) tc::mbar_init(&ctrl->res_full[w][u], 1);
        ctrl->abort = 0;
        tc::fence_barrier_init();
    }
    if (warp == 1 && lane == 0) {   // descriptors are kernel arguments: fetched ahead of the wait for the kernel before
        tc::prefetch_tensormap(&map_x); tc::prefetch_tensormap(&map_w); tc::prefetch_tensormap(&map_o);
        if (p.has_res) tc::prefetch_tensormap(&map_r);
    }
    if (warp == 2 && aligned) {  // beside the barriers; the same in both CTAs of the pair
        tmem_alloc_pair(&ctrl->tmem_base, kTmemCols);
        tmem_relinquish_pair();
    }
    tc::tc_fence_before();
    __syncthreads();
    cluster_sync();              // both CTAs' barriers are initialised before either signals the other
    tc::tc_fence_after();
    if (!aligned) {
        if (tid == 0) atomicCAS(&g_conv_tc_error, 0, kErrSmemAlign);
        return;
    }
    const uint32_t tmem_cta = ctrl->tmem_base;
    // The weights on their way into L2 while the kernel before still runs: of a tile's boxes each pair that reads the same weights asks
    // for its share. A hint only: what is copied below is read after the wait. Images of 64 x 64 pixels 911 -> 896 us, 128 x 128 1137 -> 1119, 192 x 192 1443 -> 1420.
    if (warp == 0 && tc::elect_one()) {
        const int nw = (first_tile / p.tiles_m) * BN + (int)rank * (BN / 2), sharing = min(p.tiles_m, tile_step);
        for (int i = first_tile % p.tiles_m; i < num_boxes; i += sharing) tma_prefetch_3d(&map_w, i / 3 * BK, nw, i % 3 * 3);
    }
    __syncwarp();
    pdl_wait();      // set-up above is on-chip only; the operands are another kernel's output
    pdl_trigger();

    if (warp == 0) {
        // ------------------------------------------------------------ producer (the warp's elected lane, one per CTA)
        const bool leader = tc::elect_one();
        int s = 0, par = 1, filled = 0;   // stage, parity of its previous phase, stages filled once
        bool ok = true;
        if (C::kResident && leader && first_tile < num_tiles) {
            const uint32_t full0 = map_to_cta(tc::smem_addr(&ctrl->weights), 0);
            if (rank == 0) tc::mbar_arrive_expect_tx(&ctrl->weights, 2 * 9 * p.cb * C::kWBytes);
            for (int i = 0; i < 3 * p.cb; ++i) tma_load_3d_pair(base_w + i * 3 * C::kWBytes, &map_w, i / 3 * BK, rank * (BN / 2), i % 3 * 3, full0);
        }
        for (int t = first_tile; ok && t < num_tiles; t += tile_step) {
            const Box b = box_of<BX>(p, 2 * (t % p.tiles_m) + (int)rank);   // a box beyond the last one reads as zeros
            const int nw = (t / p.tiles_m) * BN + (int)rank * (BN / 2);      // channels beyond the last one too
            int c = 0, ty = 0;            // channel block and row of taps of the box
            for (int i = 0; i < num_boxes; ++i) {
                if (filled == kStages) ok = tc::mbar_wait_warp(&ctrl->empty[s], par, abort_flag);
                else ++filled;
                if (!ok) break;
                if (leader) {
                    const uint32_t full0 = map_to_cta(tc::smem_addr(&ctrl->full[s]), 0);
                    // CTA 0 announces the bytes of both CTAs' copies on its own barrier; CTA 1's may land before that: the phase
                    // cannot complete without the announcement's arrival
                    if (rank == 0) tc::mbar_arrive_expect_tx(&ctrl->full[s], C::kStageTx);
                    tma_load_4d_pair(base + s * C::kHaloBytes, &map_x, c * BK, b.x - 1, b.y + ty - 1, b.n, full0);
                    if (!C::kResident) tma_load_3d_pair(base_w + s * 3 * C::kWBytes, &map_w, c * BK, nw, ty * 3, full0);
                }
                step(p, c, ty);
                if (++s == kStages) { s = 0; par ^= 1; }
            }
        }
        if (leader && *abort_flag) drain_pause();   // this CTA's copies count on CTA 0's barriers: give them time to land
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ issuer of the pair's products (elected lane of CTA 0)
        if (rank == 0) {
            constexpr uint32_t idesc = tc::umma_idesc_f16(2 * C::kRows, BN, 0);
            const bool leader = tc::elect_one();
            int s = 0, par = 0, tl = 0;
            bool ok = true;
            for (int t = first_tile; ok && t < num_tiles; t += tile_step, ++tl) {
                const int acc = tl & 1;
                if (tl >= 2) ok = wait_remote_warp(&ctrl->acc_empty[acc], ((tl >> 1) + 1) & 1, abort_flag);
                if (!ok) break;
                tc::tc_fence_after();
                const uint32_t d_tmem = tmem_cta + acc * C::kAccCols;
                if (C::kResident && tl == 0) ok = tc::mbar_wait_warp(&ctrl->weights, 0, abort_flag);
                if (!ok) break;
                int c = 0, ty = 0;            // of the box: where its weights lie, if they are resident
                for (int i = 0; i < num_boxes; ++i) {
                    ok = tc::mbar_wait_warp(&ctrl->full[s], par, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after();
                    if (leader) {
                        const uint32_t w0 = base_w + (C::kResident ? c * 3 + ty : s) * (3 * C::kWBytes);
#pragma unroll
                        for (int tx = 0; tx < 3; ++tx) {
                            const uint32_t a_lo = tc::umma_desc_lo(base + s * C::kHaloBytes + tx * kColBytes);
                            const uint32_t b_lo = tc::umma_desc_lo(w0 + tx * C::kWBytes);
#pragma unroll
                            for (int ks = 0; ks < BK / 16; ++ks)
                                umma_pair_f16_lo(d_tmem, a_lo + ks * 2, b_lo + ks * 2, idesc, (i > 0) || (tx > 0) || (ks > 0));
                        }
                        umma_pair_commit(&ctrl->empty[s]);
                        if (tl == 0 && i == 0) umma_pair_commit(&ctrl->started);
                    }
                    step(p, c, ty);
                    if (++s == kStages) { s = 0; par ^= 1; }
                }
                if (ok && leader) umma_pair_commit(&ctrl->acc_full[acc]);
            }
            if (leader && *abort_flag) {
                umma_pair_commit(&ctrl->drain);
                tc::mbar_wait_drain(&ctrl->drain, 0);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue, warps 2-5 of both CTAs
        const int lane_grp = warp & 3;                        // a warp reaches tensor-memory lanes [32 * (warp % 4), +32)
        const uint32_t lane_off = (uint32_t)(lane_grp * 32) << 16;
        unsigned char* my_stage = staging + lane_grp * kUnits * kUnitBytes;
        const uint32_t stage_base = tc::smem_addr(my_stage);
        uint64_t* my_res = ctrl->res_full[lane_grp];
        bool ok = true;
        int tl = 0;
        for (int t = first_tile; ok && t < num_tiles; t += tile_step, ++tl) {
            const int acc = tl & 1;
            const Box b = box_of<BX>(p, 2 * (t % p.tiles_m) + (int)rank);
            // this warp's 32 pixels, four columns of the box, and its first channel
            const int x0 = b.x + 4 * (lane_grp & (BX / 4 - 1)), n0 = (t / p.tiles_m) * BN + (C::kRows == 64 ? (lane_grp >> 1) * C::kAccCols : 0);
            const bool live = 2 * (t % p.tiles_m) + (int)rank < p.tiles;
            // ADD: the thread's pixel of p.sum, 32 channels of which are fetched ahead of the half unit that adds them
            const int px = x0 + (lane >> 3), py = b.y + (lane & 7);
            const bool inside = ADD && live && px < p.W && py < p.H;
            const __half* sum_row = ADD ? p.sum + ((size_t)(inside ? b.n : 0) * p.H * p.W + (inside ? (size_t)py * p.W + px : 0)) * p.c_out + n0 : nullptr;
            uint4 add[ADD ? 4 : 1];
            const auto fetch = [&](int half) {
                if constexpr (ADD) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int ch = half * 32 + q * 8;
                        add[q] = inside && ch < kUnits * kUnitCh && n0 + ch < p.c_out ? *reinterpret_cast<const uint4*>(sum_row + ch) : make_uint4(0, 0, 0, 0);
                    }
                }
            };
            fetch(0);
            if (lane == 0) {
                bulk_wait_read<0>();   // the previous tile's stores have read the buffers
                if (p.has_res) {
                    // of the first tile only once its first K block has been consumed, so that the operands are not held up;
                    // the barrier has one phase, which a late warp cannot miss
                    if (tl == 0) tc::mbar_wait(&ctrl->started, 0, abort_flag);
#pragma unroll
                    for (int u = 0; u < kUnits; ++u) {
                        tc::mbar_arrive_expect_tx(&my_res[u], kUnitBytes);
                        tma_load_4d(stage_base + u * kUnitBytes, &map_r, n0 + u * kUnitCh, x0, b.y, b.n, &my_res[u]);
                    }
                }
            }
            __syncwarp();
            // Lane l holds channels 2l and 2l + 1 of a unit's bias, fetched a unit ahead (each thread reading the 64 of them itself
            // was 8 us of load latencies a tile)
            const uint32_t* bias_lane = reinterpret_cast<const uint32_t*>(p.bias + n0) + lane;
            const bool biased = p.bias != nullptr;
            uint32_t bias_next = biased && n0 + 2 * lane < p.c_out ? __ldg(bias_lane) : 0;
            ok = tc::mbar_wait_warp(&ctrl->acc_full[acc], (tl >> 1) & 1, abort_flag);
            if (!ok) break;
            tc::tc_fence_after();
            const uint32_t t_acc = tmem_cta + lane_off + acc * C::kAccCols;
#pragma unroll 1
            for (int u = 0; u < kUnits; ++u) {
                const uint32_t bias_u = bias_next;
                if (biased && u + 1 < kUnits) bias_next = n0 + (u + 1) * kUnitCh + 2 * lane < p.c_out ? __ldg(bias_lane + (u + 1) * (kUnitCh / 2)) : 0;
                unsigned char* buf = my_stage + u * kUnitBytes;
                if (p.has_res) ok = tc::mbar_wait_warp(&my_res[u], tl & 1, abort_flag);
                if (!ok) break;
                uint32_t second[kUnitCh / 2];      // silu(out), if asked
#pragma unroll
                for (int hc = 0; hc < kUnitCh / 32; ++hc) {
                    uint32_t v[32], o[16];
                    tc::tmem_ld32(t_acc + u * kUnitCh + hc * 32, v);
                    uint4 res[4];
                    if (p.has_res) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) res[q] = *reinterpret_cast<const uint4*>(buf + C::chunk(lane, hc * 4 + q));
                    }
                    tc::tc_wait_ld(v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = pack_half2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                    if (biased) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 y = unpack_half2(o[i]), bb = unpack_half2(__shfl_sync(0xffffffffu, bias_u, hc * 16 + i));
                            o[i] = pack_half2(y.x + bb.x, y.y + bb.y);
                        }
                    }
                    if (p.silu) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 y = unpack_half2(o[i]);
                            o[i] = pack_half2(silu_sfu(y.x), silu_sfu(y.y));
                        }
                    }
                    if (p.has_res) {
                        const uint32_t* rw = reinterpret_cast<const uint32_t*>(res);
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 y = unpack_half2(o[i]), rr = unpack_half2(rw[i]);
                            o[i] = pack_half2(y.x + rr.x, y.y + rr.y);
                        }
                    }
                    if constexpr (ADD) {
                        const uint32_t* aw = reinterpret_cast<const uint32_t*>(add);
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 y = unpack_half2(o[i]), aa = unpack_half2(aw[i]);
                            o[i] = pack_half2(aa.x + y.x, aa.y + y.y);
                        }
                        fetch(u * (kUnitCh / 32) + hc + 1);
                    }
                    if (p.dual) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 z = unpack_half2(o[i]);
                            second[hc * 16 + i] = pack_half2(silu_sfu(z.x), silu_sfu(z.y));
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        *reinterpret_cast<uint4*>(buf + C::chunk(lane, hc * 4 + q)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
                }
                tc::fence_proxy_async();                      // the copy engine reads what the threads just wrote
                __syncwarp();
                if (lane == 0 && live) {
                    tma_store_4d(&map_o, stage_base + u * kUnitBytes, n0 + u * kUnitCh, x0, b.y, b.n);   // pixels beyond the image are clipped
                    bulk_commit();
                }
                if (p.dual) {                                 // the same buffer again, once that store has read it
                    if (lane == 0) bulk_wait_read<0>();
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < kUnitCh / 8; ++q)
                        *reinterpret_cast<uint4*>(buf + C::chunk(lane, q)) =
                            make_uint4(second[4 * q], second[4 * q + 1], second[4 * q + 2], second[4 * q + 3]);
                    tc::fence_proxy_async();
                    __syncwarp();
                    if (lane == 0 && live) {
                        tma_store_4d(&map_s, stage_base + u * kUnitBytes, n0 + u * kUnitCh, x0, b.y, b.n);
                        bulk_commit();
                    }
                }
            }
            if (!ok) break;
            // every tcgen05.ld of this warp has completed: hand the accumulator back
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) remote_arrive(map_to_cta(tc::smem_addr(&ctrl->acc_empty[acc]), 0));
        }
        if (lane == 0) {
            if (*abort_flag) drain_pause();
            bulk_wait_read<0>();   // the stores complete with the grid; shared memory only has to outlive their reads
        }
        __syncwarp();
    }

    // ---- teardown: neither CTA leaves while the other may still signal its barriers or read its shared memory
    tc::tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == 0) {
        tc::tc_fence_after();
        tmem_dealloc_pair(tmem_cta, kTmemCols);
    }
    if (tid == 0 && ctrl->abort) atomicCAS(&g_conv_tc_error, 0, kErrTimeout);
}

}  // namespace tcconv

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

// fp16 tensor of 3 or 4 dimensions, innermost first, strides in bytes from the second on; boxes swizzled by 128 bytes (of 32 channels: by 64),
// elements outside read as zeros
bool make_map(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
    static_assert(tcconv::BK == 64, "rows of 128 bytes, or of 64 for units of 32 channels");
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, rank, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, box[0] == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// [N][H][W][C] as (c, y, x, n): boxes of `channels` channels x kBoxY x columns pixels of one image, a column's pixels one after the other
bool make_map_pixels(CUtensorMap* m, const void* base, int N, int H, int W, int C, int columns, int channels) {
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)H, (cuuint64_t)W, (cuuint64_t)N};
    const cuuint64_t strides[3] = {(cuuint64_t)2 * W * C, (cuuint64_t)2 * C, (cuuint64_t)2 * H * W * C};
    const cuuint32_t box[4] = {(cuuint32_t)channels, (cuuint32_t)tcconv::kBoxY, (cuuint32_t)columns, 1};
    return make_map(m, base, 4, dims, strides, box);
}

template <int BN, int BX> cudaLaunchConfig_t pair_config(cudaLaunchAttribute (&attr)[2], cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see launch_pdl in common.cuh
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(tcconv::kThreads); cfg.dynamicSmemBytes = tcconv::Cfg<BN, BX>::kSmemBytes; cfg.stream = st;
    cfg.attrs = attr; cfg.numAttrs = g_pdl_enabled ? 2 : 1;
    return cfg;
}

// CTA pairs of the kernel that the device runs at once (asked once per device; 0: it cannot place them)
template <int BN, int BX, bool ADD = false> int resident_pairs(int dev) {
    static std::atomic<int> asked[64];   // the answer + 1
    int n = asked[dev].load(std::memory_order_acquire);
    if (n == 0) {
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = pair_config<BN, BX>(attr, nullptr);
        int sms = 0, pairs = 0;
        cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(tcconv::conv3x3_pair_kernel<BN, BX, ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, tcconv::Cfg<BN, BX>::kSmemBytes);
        cfg.gridDim = dim3(2 * std::max(1, sms / 2));
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&pairs, tcconv::conv3x3_pair_kernel<BN, BX, ADD>, &cfg);
        if (e != cudaSuccess) { cudaGetLastError(); pairs = 0; }
        n = std::max(pairs, 0) + 1;
        asked[dev].store(n, std::memory_order_release);
    }
    return n - 1;
}

template <int BN, int BX, bool ADD = false>
int launch_conv(const CUtensorMap& mx, const CUtensorMap& mo, const CUtensorMap& mr, const CUtensorMap& ms, const __half* w,
                tcconv::Params p, int dev, cudaStream_t st) {
    CUtensorMap mw;   // [C_out][9][C_in] as (c_in, c_out, tap)
    const cuuint64_t C_in = (cuuint64_t)p.cb * 64;
    const cuuint64_t dims[3] = {C_in, (cuuint64_t)p.c_out, 9}, strides[2] = {18 * C_in, 2 * C_in};
    const cuuint32_t box[3] = {64, BN / 2, 3};
    if (!make_map(&mw, w, 3, dims, strides, box)) return RFK_EUNSUPPORTED;
    const int pairs = resident_pairs<BN, BX, ADD>(dev);
    if (pairs <= 0) return RFK_EUNSUPPORTED;
    p.tiles_n = ceil_div(p.c_out, BN);
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = pair_config<BN, BX>(attr, st);
    cfg.gridDim = dim3(2 * std::min(p.tiles_m * p.tiles_n, pairs));
    cudaError_t e = cudaLaunchKernelEx(&cfg, tcconv::conv3x3_pair_kernel<BN, BX, ADD>, mx, mw, mo, mr, ms, p);
    if (e != cudaSuccess) { cudaGetLastError(); return (int)e; }
    return launch_status();
}

// shapes and alignments that the kernel takes
bool conv_serves(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, const rfk_half* out,
                 const rfk_half* out_silu, int C_in, int C_out) {
    return C_in % 64 == 0 && C_out % 32 == 0 && aligned16(x) && aligned16(w) && aligned16(out) && (!residual || aligned16(residual)) &&
           (!out_silu || aligned16(out_silu)) && (!bias || (reinterpret_cast<uintptr_t>(bias) & 3u) == 0);
}

// Tiles (rfk_conv3x3_nhwc_tiled's `tile`): output channels x pixels of a pair's CTA
enum : int { kByRule = 0, k128x128 = 1, k64x128 = 2, k64x64 = 3, k32x128 = 4 };

// all weights beside the ring of boxes (at 64 x 64 pixels the launch is all there is: 5.3 for 4.9 in tiles of 64 x 64; 128 x 128 6.1 / 6.9 / 8.0)
bool resident_weights(int C_in, int C_out) { return C_out == 32 && C_in <= 64 * tcconv::kResidentBlocks; }

// pairs of boxes of BX x kBoxY pixels
long long box_pairs(int N, int H, int W, int BX) { return ((long long)ceil_div(W, BX) * ceil_div(H, tcconv::kBoxY) * N + 1) / 2; }

// The tile whose busiest pair is done first: it takes its tiles one after the other, a K block of each in the clocks named at the top, and
// the last one's epilogue shows. us, tiles of 128 x 128 / 64 x 128 / 64 x 64: 256 -> 256 channels at 48^2 11.7 / 8.3 / 6.5, 56^2 11.8 / 8.5 / 9.5, 64^2 12.0 / 8.7 / 9.7,
// 80^2 12.7 / 12.5 / 13.0, 96^2 13.3 / 13.2 / 16.2, 112^2 17.1 / 17.1 / 22.1, 128^2 17.9 / 21.6 / 25.6, 160^2 23.4 / 30.0 / 37.4; 512 -> 256 at 48^2 16.7 / 12.1 / 9.8, 64^2 17.2 / 12.6 /
// 15.0, 80^2 18.2 / 19.7 / 20.6; 1024 -> 256 at 48^2 26.6 / 18.9 / 15.3, 64^2 28.5 / 20.1 / 25.9.
int choose_tile(int N, int H, int W, int C_in, int C_out, int pairs) {
    if (resident_weights(C_in, C_out)) return k32x128;
    struct { int tile, bx, bn, clocks; } const kinds[] = {{k128x128, 16, 128, 260}, {k64x128, 16, 64, 177}, {k64x64, 8, 64, 125}};
    int best = 0;
    long long least = 0;
    for (const auto& k : kinds) {
        if (k.bn > 64 && C_out % k.bn) continue;
        const long long rounds = ceil_div(box_pairs(N, H, W, k.bx) * ceil_div(C_out, k.bn), pairs);
        const long long clocks = rounds * (9 * C_in / 64) * k.clocks + 20 * k.bn * k.bx / 8;
        if (!best || clocks < least) { best = k.tile; least = clocks; }
    }
    return best;
}

}  // namespace
}  // namespace rfk

using namespace rfk;

extern "C" int rfk_conv3x3_nhwc_serves(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual,
                                       const rfk_half* out, const rfk_half* out_silu, int C_in, int C_out) {
    int dev = 0;
    if (!conv_serves(x, w, bias, residual, out, out_silu, C_in, C_out) || !tensor_map_encoder()) return 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    return resident_pairs<128, 16>(dev) > 0 && resident_pairs<64, 16>(dev) > 0 && resident_pairs<64, 8>(dev) > 0 && resident_pairs<32, 16>(dev) > 0;
}

static int conv3x3(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, const rfk_half* sum, rfk_half* out,
                   rfk_half* out_silu, int N, int H, int W, int C_in, int C_out, int silu, int rows_outside, int tile, rfk_stream_t stream) {
    if (!x || !w || !out || N < 0 || H <= 0 || W <= 0 || C_in <= 0 || C_out <= 0) return RFK_EINVAL;
    if (x == out || x == out_silu || out == out_silu) return RFK_EINVAL;   // a pixel is read by its neighbours' tiles
    if (tile < kByRule || tile > k32x128 || (tile == k128x128 && C_out % 128) || (tile == k32x128 && !resident_weights(C_in, C_out))) return RFK_EINVAL;
    if (N == 0) return RFK_OK;
    if (!conv_serves(x, w, bias, residual, out, out_silu, C_in, C_out) || (sum && (!aligned16(sum) || resident_weights(C_in, C_out)))) return RFK_EUNSUPPORTED;
    if (box_pairs(N, H, W, 8) * ceil_div(C_out, 64) > 0x1fffffffLL || 9LL * C_in > 0x7fffffffLL) return RFK_EUNSUPPORTED;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return RFK_EUNSUPPORTED;
    if (tile == kByRule) {
        const int pairs = resident_pairs<128, 16>(dev);   // one on every two SMs
        if (pairs <= 0) return RFK_EUNSUPPORTED;
        tile = choose_tile(N, H, W, C_in, C_out, pairs);
    }
    const int bx = tile == k64x64 ? 8 : 16, unit = tile == k64x64 || tile == k32x128 ? 32 : 64;
    CUtensorMap mx, mo, mr, ms;
    if (!make_map_pixels(&mx, x, N, H, W, C_in, bx + 2, 64) || !make_map_pixels(&mo, out, N, H, W, C_out, 4, unit) ||
        !make_map_pixels(&mr, residual ? residual : out, N, H, W, C_out, 4, unit) ||
        !make_map_pixels(&ms, out_silu ? out_silu : out, N, H, W, C_out, 4, unit))
        return RFK_EUNSUPPORTED;
    tcconv::Params p{};
    p.bias = (const __half*)bias;
    p.tiles_x = (int)ceil_div(W, bx); p.tiles_img = p.tiles_x * (int)ceil_div(H, tcconv::kBoxY); p.tiles = p.tiles_img * N;
    p.tiles_m = (p.tiles + 1) / 2;
    p.cb = C_in / 64; p.c_out = C_out;
    p.rows_outside = rows_outside != 0; p.silu = silu != 0; p.has_res = residual != nullptr; p.dual = out_silu != nullptr;
    p.sum = (const __half*)sum; p.H = H; p.W = W;
    if (sum)
        return (tile == k128x128 ? launch_conv<128, 16, true> : tile == k64x128 ? launch_conv<64, 16, true> : launch_conv<64, 8, true>)(
            mx, mo, mr, ms, (const __half*)w, p, dev, as_stream(stream));
    const auto launch = tile == k128x128 ? launch_conv<128, 16, false> : tile == k64x128 ? launch_conv<64, 16, false> : tile == k64x64 ? launch_conv<64, 8, false>
                                            : launch_conv<32, 16, false>;
    return launch(mx, mo, mr, ms, (const __half*)w, p, dev, as_stream(stream));
}

extern "C" int rfk_conv3x3_nhwc_tiled(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, rfk_half* out,
                                      rfk_half* out_silu, int N, int H, int W, int C_in, int C_out, int silu, int rows_outside, int tile,
                                      rfk_stream_t stream) {
    return conv3x3(x, w, bias, residual, nullptr, out, out_silu, N, H, W, C_in, C_out, silu, rows_outside, tile, stream);
}

extern "C" int rfk_conv3x3_nhwc_add(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, rfk_half* sum,
                                    rfk_half* sum_silu, int N, int H, int W, int C_in, int C_out, int rows_outside, int tile, rfk_stream_t stream) {
    if (!sum || !sum_silu || residual == sum || residual == sum_silu) return RFK_EINVAL;
    return conv3x3(x, w, bias, residual, sum, sum, sum_silu, N, H, W, C_in, C_out, 0, rows_outside, tile, stream);
}

extern "C" int rfk_conv3x3_nhwc(const rfk_half* x, const rfk_half* w, const rfk_half* bias, const rfk_half* residual, rfk_half* out,
                                rfk_half* out_silu, int N, int H, int W, int C_in, int C_out, int silu, int rows_outside,
                                rfk_stream_t stream) {
    if (C_out > 0 && C_out % 128) return x && w && out ? RFK_EUNSUPPORTED : RFK_EINVAL;
    return rfk_conv3x3_nhwc_tiled(x, w, bias, residual, out, out_silu, N, H, W, C_in, C_out, silu, rows_outside, kByRule, stream);
}

extern "C" int rfk_conv_error(int* code, int clear) {
    if (!code) return RFK_EINVAL;
    cudaError_t e = cudaMemcpyFromSymbol(code, g_conv_tc_error, sizeof(int));
    if (e != cudaSuccess) return (int)e;
    if (clear) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_conv_tc_error, &zero, sizeof(int));
        if (e != cudaSuccess) return (int)e;
    }
    return RFK_OK;
}
