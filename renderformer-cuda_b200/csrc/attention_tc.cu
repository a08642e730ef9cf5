// Fused attention on the 5th-generation tensor cores (tcgen05 + tensor memory + TMA), head_dim 64 and 128 (sizes below: 64,
// with 128 in brackets where it differs).
//
// Same function as flash_attention_kernel (attention.cu): O = softmax(scale * Q K^T) V over
// the first n_keys keys, fp16 operands, fp32 accumulation, probabilities rounded to fp16.
// Reference boundary: rf::sdpa, src/layers/attention.cu:89-166 of BANANASJIM/renderformer-cuda.
//
// One CTA = 256 queries of one head as two blocks of 128 that share the K/V tiles in shared
// memory (every key tile is fetched once per CTA, i.e. half as often as with one block per CTA),
// keys in tiles of 64, 16 warps (13 with a role):
//   warp 8       producer: one thread issues TMA tile loads (both Q blocks once, then K and V tiles
//                through a ring of kStages shared-memory stages); the copies land in the tensor
//                core's 128-byte-swizzled layout and complete on mbarriers, no thread touches the bytes.
//   warps 11-12  one warp per block [warp 11 for both], whose elected lane issues S = Q K^T (tcgen05.mma M128 N64 K16
//                x 4 [8]) into one of the block's three [two] score buffers in tensor memory, as
//                soon as the P V product that read that buffer's previous contents is complete:
//                the softmax warps find their next two [one] tiles ready.
//   warps 0-7    softmax (block = warp / 4): a thread owns one query row = its tensor-memory lane,
//                so row maximum and row sum are thread-local (no shuffles). The 64 scores come to
//                registers with tcgen05.ld; the common tile exponentiates them against the running
//                reference right away and checks afterwards that this was admissible (the exact path,
//                with the tile's maximum first, runs for the first tile, a padded last tile, a
//                failed check and every tile of 128-wide heads); P = exp2(...) is rounded to fp16
//                and stored back with tcgen05.st over the first 32 columns of the same score
//                buffer, from where
//   warps 9-10   one warp per block, whose elected lane issues O += P V with P as the A operand
//                from tensor memory and V (MN-major) from shared memory: P never passes through
//                shared memory. The output accumulator O (128 x 64 [128] fp32 per block) is rescaled in place only when a
//                row's running maximum has grown by more than 2^8 (the factor cancels in O / l): by the softmax warps.
//   [warps 12-15 with 128-wide heads, where O is rescaled whenever a maximum has grown at all: they take each row's factor from
//                its softmax thread as soon as that has the tile's maximum, wait for the previous P V, rescale, and arrive
//                beside the softmax warps on the barrier that P V waits for. One block per CTA: warps 4-7.]
// A stage of the ring is free again when both blocks' P V products of its tile are complete
// (kv_empty counts two arrivals). The products have separate issuing warps because one warp's
// instruction stream (8 products, 3 commits and 2-3 waits per tile, all dependent) takes about as
// long as the softmax of a tile; the order between them is kept by mbarriers, not by issue order.
// Tensor memory: all 512 columns (per block S0, S1, S2, O: 64 each [S0, S1: 64, O: 128]); shared
// memory 32 [64] KB (Q) + 6 x 16 KB [4 x 32 KB]; one CTA per SM. Every mbarrier wait is bounded; on a time-out the CTA raises an
// error word, frees its tensor memory and returns.
//
// Key split for grids that do not fill the machine. A unit = 256 queries of one head over all keys = one CTA. With few
// units (a 256 x 256 view has 64 of them for 148 SMs) most SMs idle, so when the caller supplies a workspace and the
// estimate below says it pays, the key range of the units is cut into one equal share per SM; a share is one or two
// pieces (it may cross a unit boundary), a piece is one CTA over a range of key tiles. A piece writes its un-normalised
// O, running maximum and sum to the workspace and increments its unit's counter; the CTA that finds the counter
// complete (no CTA ever waits for another) merges the unit's pieces, writes the output and zeroes the counter for the
// next launch. A piece costs about 10 us beyond its tiles (pipeline fill, publishing, merging), so the last, partial
// round of a larger grid is cut the same way only when few units are left for it (plan_work).
//
// Hand-over. Any other grid of more than one round (256 units of a 512 x 512 view: 1.73 rounds of 148 SMs) would leave SMs idle in
// its last round. With a workspace every SM gets the same number of key tiles instead: some units are begun by one CTA, which leaves
// O, running maximum and row sum as they stand in the workspace, and finished by another, which takes them up and goes on with the
// next tile (plan_handover). That is the same sequence of operations on every row, so the bits are those of whole units, for every
// caller. First pieces are the grid's first blocks, second pieces its last, and a first piece waits for nobody. Blocks are handed out in
// order, and by the plan a unit's first piece has been done for half a round when its second begins; but nothing promises that order, and
// nothing depends on it: a second piece that finds no state within 50 ms, or a first piece that failed, takes all of the unit, and a first piece
// that comes after that leaves it to it (handover.cuh). Measured (us, whole / handed over; estimates agree within 2 %): 16 x 4096 x 5665 x 64 138 / 128, 16 x 5665 x 5665 207 / 182,
// 448 units of 89 tiles 275 / 220, 149 of 16 32 / 26; 128-wide heads 184 of 89 tiles 181 / 143, 256 of 89 185 / 183. Of 137 grids of 149 to 600
// units and 16 to 113 tiles none lost. It needs a gain of 5 % by the plan's estimate; 256 units of 24 tiles stay whole.
//
// One block per CTA. Two blocks share a CTA so that they share the K/V tiles; their softmax warps then share the SM's
// schedulers and special-function unit (a tile of one block alone takes 1020 clocks, of two together 1410, 64-wide heads).
// Where all blocks of 128 queries find an SM of their own, each gets one (BLOCKS = 1): 16 x 576 x 4607, 48 units of 256 queries,
// 62 -> 47 us; 16 x 1100 x 5665 72 -> 53 us; 8 x 1600 x 4607 x 128 84 -> 62 us. Past that line the blocks without an SM would be
// a second round, and two rounds of one block take longer than one round of two (2 x 1020 against 1410).
// A row's arithmetic does not depend on its block's company: both forms have the same bits.
#include <algorithm>
#include <cuda.h>  // CUtensorMap and its enums; the encoder itself is looked up at run time
#define RFK_TC_WAIT_INLINE  // this kernel re-partitions its registers (setmaxnreg)
#include "attention_tc.cuh"
#include "common.cuh"
#include "handover.cuh"
#include "kernels_internal.h"

namespace rfk {

__device__ int g_attn_tc_error = 0;  // first time-out / failure code seen by any CTA since load

namespace tcattn {

constexpr int BM = 128, BN = 64;
constexpr int kBlocks = 2;                     // 128-query blocks per CTA, sharing the K/V ring (at most; see "One block per CTA")
constexpr int kThreads = 512;                  // warps 0-7 softmax (block = warp / 4), 8 producer, 9-10 PV, 11-12 QK issuers, 13-15 none (128-wide heads: see Cfg)
// Registers (64-wide heads): the CTA starts with 128 per thread. The two warpgroups that only issue copies and products (warps 8-15)
// hand theirs back down to kRegsIssue and the softmax warpgroups (warps 0-7) grow to kRegsSoftmax, which lets the
// compiler keep both halves of a score tile and their exponentials in flight without reusing registers early
// (measured: 3 % off the kernel's time). 256 * 40 + 256 * 216 = 65536, the register file.
constexpr int kRegsIssue = 40, kRegsSoftmax = 216;
constexpr int kTmemCols = 512;                 // 256 per block: the score buffers (64 columns each), then O
// Per head size. A row of the operand tiles is HD / 64 swizzle rows of 128 bytes: the tiles are kept as HD / 64
// sub-tiles of 64 columns, each fetched by its own TMA box.
template <int HD, int BLOCKS> struct Cfg {
    static constexpr int kSub = HD / 64;
    static constexpr int kQSub = BM * 128, kQBytes = kSub * kQSub;     // 16 KB per 64 columns
    static constexpr int kKSub = BN * 128, kKBytes = kSub * kKSub;     // 8 KB per 64 columns; a stage is K then V
    static constexpr int kStageBytes = 2 * kKBytes;
    static constexpr int kStages = HD == 64 || BLOCKS == 1 ? 6 : 4;
    // O takes HD of a block's 256 tensor-memory columns, score buffers the rest: three at 64, two at 128; a block that has the
    // CTA to itself always has three
    static constexpr int kSBufs = BLOCKS == 1 ? 3 : (256 - HD) / 64;
    // 128-wide heads follow the exact maximum, which moves in every second tile of a warp's 32 rows: the 128 columns of O are rescaled
    // by a warpgroup of its own beside the exponentials.
    // (unit-variance scores: 8 x 4096 x 5665 101.6 -> 92 us, 8 x 1600 x 4607 with one block per CTA 62.2 -> 52.5; where the maxima
    // hardly move 84.7 -> 80 and 49.4 -> 49.4.) Its latency counts: 16 columns of O at a time 103 us, 32 95.5, 32 fetched under the
    // multiplication of the 32 before 92, which takes 104 registers. 256 * 160 + 128 * 120 + 128 * 72 = 65536; of the splits that keep
    // the softmax from spilling this one was the fastest on scenes and views (1 to 2 % ahead of 168 / 120 / 56). With
    // one block per CTA 128 * 216 + 128 * 104 + 256 * 40 are within the launch's 65536 (softmax with 160: 55 us).
    static constexpr bool kCorr = HD == 128;
    static constexpr int kRegSoftmax = !kCorr || BLOCKS == 1 ? kRegsSoftmax : 160, kRegCorr = BLOCKS == 1 ? 104 : 120,
                         kRegIssue = !kCorr || BLOCKS == 1 ? kRegsIssue : 72;
    static constexpr int kCorrWarp = !kCorr ? 99 : BLOCKS == 2 ? 12 : 4;   // its first warp
    static constexpr int kFactorBytes = kCorr ? BLOCKS * kSBufs * BM * 4 : 0;   // behind the control block
    static constexpr int kQkWarp = 11;                                     // kCorr: one warp issues Q K^T of both blocks
    // The shared-memory window is declared 1024-byte aligned (swizzled tiles need it) and the kernel checks it.
    static constexpr int kSmemBytes = BLOCKS * kQBytes + kStages * kStageBytes + 512 + kFactorBytes;
    static_assert(kSmemBytes + 1024 <= 227 * 1024, "one CTA per SM");
};
constexpr int kMaxStages = 6, kMaxSBufs = 3;

struct __align__(8) Ctrl {
    uint64_t q_full, kv_full[kMaxStages], kv_empty[kMaxStages], s_full[kBlocks][kMaxSBufs], p_full[kBlocks][kMaxSBufs],
        pv_done[kBlocks][kMaxSBufs], move_full[kBlocks][kMaxSBufs];
    uint64_t drain[2 * kBlocks];  // abort path only, one per issuing lane: completes once that lane's products have finished
    uint32_t tmem_base;
    int abort;
    int merge;  // set by thread 0 of a split unit's last piece: this CTA merges the unit; of a second piece: it takes up the first one's state
};

static_assert(sizeof(Ctrl) <= 512, "control block");

enum : int { kErrTimeout = 1, kErrSmemAlign = 2 };

// A CTA's share of a unit whose keys are split: key tiles [t0, t0 + nt) of unit `unit`; the unit's pieces own the
// workspace slots [first, first + count), this one `slot`.
struct Piece { uint16_t unit, t0, nt, first, count, slot; };
constexpr int kMaxPieces = 320;
struct WorkList {
    int whole_units;  // CTAs [heads, heads + whole_units) take the unit of their index, less heads, over all keys
    int n_pieces;     // the CTAs behind them take pieces[index - whole_units]
    int q_blocks;     // units per head: ceil(Sq / 256)
    int heads;        // units handed over (else 0): CTAs [0, heads) take their first pieces, pieces[0, heads); n_pieces = 2 * heads
    Piece pieces[kMaxPieces];
};
// Workspace: 256 counters (one per split unit, zero between launches, also after one whose waits timed out), then per slot 256 x {m, l}, then per slot the
// un-normalised output as [16 or 32 groups of 4 columns][256 rows] float4 (a warp's 32 rows of one group are contiguous).
constexpr int kUnitRows = kBlocks * BM;
constexpr size_t kWsCounterBytes = 1024;
constexpr size_t kWsMlBytes = (size_t)kMaxPieces * kUnitRows * 2 * sizeof(float);
constexpr size_t kWsOBytes = (size_t)kMaxPieces * kUnitRows * 128 * sizeof(float);  // for the larger head size
constexpr size_t kWsBytes = kWsCounterBytes + kWsMlBytes + kWsOBytes;
// A unit that is handed over (see "Hand-over") takes its counter, by slot, and two of the output areas: O in 2 * slot, the row sums
// and the reference in the first two groups of 2 * slot + 1.
constexpr int kMaxHanded = kMaxPieces / 2;
static_assert(kMaxHanded * sizeof(int) <= kWsCounterBytes, "a counter each");

template <int N> __device__ __forceinline__ void regs_release() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ void softmax_warps_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }  // warps 0-7 only

// The clock of the wait for a first piece, given a reading of the timer at its start and then now and then. As in mbar_wait_slow the
// limit counts from two readings, as signed differences, and here it has to be exceeded by two in a row, so that no one reading of
// the 64-bit timer that is off ends a wait.
constexpr uint64_t kHandedLimitNs = 50ull * 1000 * 1000;
struct WaitClock {
    uint64_t t0, first = 0;
    bool over = false;
    __host__ __device__ explicit WaitClock(uint64_t start) : t0(start) {}
    __host__ __device__ bool ended(uint64_t now) {
        if (first == 0) first = now;
        const bool late = (int64_t)(now - t0) > (int64_t)kHandedLimitNs && (int64_t)(now - first) > (int64_t)kHandedLimitNs, twice = late && over;
        over = late;
        return twice;
    }
};
// One step of a party on the word (handover.cuh), `seen`: what it probably is. The other party changes it once at most, and so often is
// the exchange tried again.
template <typename StepOf> __device__ __forceinline__ int handover_step(int* word, int seen, StepOf step_of) {
    for (int tries = 0; tries < 8; ++tries) {
        const handover::Step step = step_of(seen);
        const int old = atomicCAS(word, seen, step.next);
        if (old == seen) return step.act;
        seen = old;
    }
    return handover::kWhole;
}
// One thread of the second piece waits for the first one. True: its state is there, and is visible to the CTA behind its next barrier.
// False: the first piece failed, or did not come within the limit; the second one takes all of the unit.
__device__ __forceinline__ bool wait_handed(int* word) {
    int found;   // nearly always: the first piece has long been done, one exchange is all
    asm volatile("atom.acquire.gpu.global.cas.b32 %0, [%1], %2, %3;"
                 : "=r"(found) : "l"(__cvta_generic_to_global(word)), "n"((int)handover::kReady), "n"(handover::settle(handover::kReady).next) : "memory");
    if (found == handover::kReady) return true;
    WaitClock clock(tc::global_timer_ns());
    for (uint32_t it = 0; it < tc::kSpinLimit; ++it) {
        int seen;
        asm volatile("ld.acquire.gpu.b32 %0, [%1];" : "=r"(seen) : "l"(word) : "memory");
        if (handover::look(seen).act != handover::kWait) break;
        if ((it & 63u) == 63u && clock.ended(tc::global_timer_ns())) break;
        __nanosleep(32);
    }
    const int act = handover_step(word, handover::kReady, [](int w) { return handover::settle(w); });
    __threadfence();
    return act == handover::kGo;
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// 2^x for two values on the FMA pipes (no special-function unit): x = n + f with n = round(x),
// 2^f from a polynomial on [-0.5, 0.5] and n added into the exponent field. Degree 3 (the default;
// relative error 7.5e-5, a sixth of the fp16 rounding of the result) or, with -DRFK_ATTN_POLY_DEG=4,
// degree 4 (2.6e-6). Inputs below -125 give a value near 2^-125; the result is only good for inputs
// below 128 (the caller checks the largest it passes).
#ifndef RFK_ATTN_POLY_DEG
#define RFK_ATTN_POLY_DEG 3
#endif
__device__ __forceinline__ float2 exp2_poly(float2 x) {
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: x + kMagic holds round(x) in its low mantissa bits
    x.x = fmaxf(x.x, -125.0f);
    x.y = fmaxf(x.y, -125.0f);
    const float2 t = __fadd2_rn(x, make_float2(kMagic, kMagic));
    const float2 n = __fadd2_rn(t, make_float2(-kMagic, -kMagic));
    const float2 f = __ffma2_rn(n, make_float2(-1.0f, -1.0f), x);
#if RFK_ATTN_POLY_DEG == 3
    float2 p = __ffma2_rn(f, make_float2(0.05517136f, 0.05517136f), make_float2(0.2426111f, 0.2426111f));
    p = __ffma2_rn(p, f, make_float2(0.69326103f, 0.69326103f));
    p = __ffma2_rn(p, f, make_float2(0.99992806f, 0.99992806f));
#else
    float2 p = __ffma2_rn(f, make_float2(0.009570092f, 0.009570092f), make_float2(0.05591786f, 0.05591786f));
    p = __ffma2_rn(p, f, make_float2(0.24024744f, 0.24024744f));
    p = __ffma2_rn(p, f, make_float2(0.6931218f, 0.6931218f));
    p = __ffma2_rn(p, f, make_float2(0.9999993f, 0.9999993f));
#endif
    return make_float2(__uint_as_float(__float_as_uint(p.x) + (__float_as_uint(t.x) << 23)),
                       __uint_as_float(__float_as_uint(p.y) + (__float_as_uint(t.y) << 23)));
}

// 32 raw scores -> 32 probabilities exp2(s * c - mc), packed two fp16 per word into pk[0..16); their
// fp32 sums are added to acc0 / acc1 (two lanes each). ORDERED: the four lanes are the partial sums of the four threads that
// share a row in flash_attention_kernel (columns 8n + 2t and 8n + 2t + 1, in that order), so that the row sum has its bits.
// Packed fp32x2 multiply-adds and adds halve the instruction count around the exponentials. With 64-wide heads the
// special-function unit (16 exponentials per clock and SM) is the scarcest resource of this kernel, so of every four
// pairs those selected by the mask take the polynomial path instead. With 128-wide heads there are half as many
// exponentials per product and every one comes from the special-function unit, as in flash_attention_kernel (the
// polynomial was worth 5 % of the kernel's time while the reference trailed, for 0.4 % of the result's distance from 64 bits).
#ifndef RFK_ATTN_POLY_MASK
#define RFK_ATTN_POLY_MASK 0x1
#endif
#ifndef RFK_ATTN_POLY_PERIOD
#define RFK_ATTN_POLY_PERIOD 4
#endif
template <int HD> constexpr int kPolyMask = HD == 64 ? RFK_ATTN_POLY_MASK : 0;
template <int HD> __device__ __forceinline__ constexpr bool poly_pair(int pair) { return (kPolyMask<HD> >> (pair % RFK_ATTN_POLY_PERIOD)) & 1; }

template <int HD, bool ORDERED>
__device__ __forceinline__ void exp_half(uint32_t (&v)[32], uint32_t* pk /* may alias v */, float c, float mc, float2& acc0,
                                         float2& acc1, float& poly_max) {
    const float2 c2 = make_float2(c, c), nm2 = make_float2(-mc, -mc);
    // three passes over the registers, each a run of independent instructions: exponents, exponentials
    // (back to back, so that one warp alone can keep the special-function unit busy), then sums and packing
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        const float2 x = __ffma2_rn(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), c2, nm2);
        v[i] = __float_as_uint(x.x);
        v[i + 1] = __float_as_uint(x.y);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        if (poly_pair<HD>(i >> 1)) continue;  // this pair takes the polynomial path below
        v[i] = __float_as_uint(fast_exp2(__uint_as_float(v[i])));
    }
    if (kPolyMask<HD>) {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            if (poly_pair<HD>(i >> 1)) {
                // the polynomial path is only good for exponents below 128: the caller checks the largest it was given
                poly_max = fmax3(poly_max, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
                const float2 p = exp2_poly(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])));
                v[i] = __float_as_uint(p.x);
                v[i + 1] = __float_as_uint(p.y);
            }
        }
    }
    if (ORDERED) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            float e[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) e[j] = __uint_as_float(v[i + j]);
#pragma unroll
            for (int j = 0; j < 4; ++j) pk[(i >> 1) + j] = pack_half2(e[2 * j], e[2 * j + 1]);
            acc0 = __fadd2_rn(acc0, __fadd2_rn(make_float2(e[0], e[2]), make_float2(e[1], e[3])));
            acc1 = __fadd2_rn(acc1, __fadd2_rn(make_float2(e[4], e[6]), make_float2(e[5], e[7])));
        }
        return;
    }
    // four independent chains of packed adds (with two, the adds of a half waited on each other: -3 % with four), the
    // packing written ahead of the adds (the compiler keeps this order; -1 %)
    float2 a2 = make_float2(0.0f, 0.0f), a3 = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
        const float2 p0 = make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1]));
        const float2 p1 = make_float2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
        const float2 p2 = make_float2(__uint_as_float(v[i + 4]), __uint_as_float(v[i + 5]));
        const float2 p3 = make_float2(__uint_as_float(v[i + 6]), __uint_as_float(v[i + 7]));
        pk[i >> 1] = pack_half2(p0.x, p0.y);
        pk[(i >> 1) + 1] = pack_half2(p1.x, p1.y);
        pk[(i >> 1) + 2] = pack_half2(p2.x, p2.y);
        pk[(i >> 1) + 3] = pack_half2(p3.x, p3.y);
        acc0 = __fadd2_rn(acc0, p0);
        acc1 = __fadd2_rn(acc1, p1);
        a2 = __fadd2_rn(a2, p2);
        a3 = __fadd2_rn(a3, p3);
    }
    acc0 = __fadd2_rn(acc0, a2);
    acc1 = __fadd2_rn(acc1, a3);
}

// 32 fp32 values (as raw words) * inv -> fp16 -> 64 bytes at dst
__device__ __forceinline__ void store_row_half(__half* dst, const uint32_t (&v)[32], float inv) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        uint4 o;
        o.x = pack_half2(__uint_as_float(v[8 * c + 0]) * inv, __uint_as_float(v[8 * c + 1]) * inv);
        o.y = pack_half2(__uint_as_float(v[8 * c + 2]) * inv, __uint_as_float(v[8 * c + 3]) * inv);
        o.z = pack_half2(__uint_as_float(v[8 * c + 4]) * inv, __uint_as_float(v[8 * c + 5]) * inv);
        o.w = pack_half2(__uint_as_float(v[8 * c + 6]) * inv, __uint_as_float(v[8 * c + 7]) * inv);
        *reinterpret_cast<uint4*>(dst + c * 8) = o;
    }
}

// ORDERED (128-wide heads): the row sums in the order of flash_attention_kernel. The products of both kernels sum in the same
// order (mma.sync and tcgen05.mma add 16 products at a time, with the same bits, which the tests compare), the running maximum is
// exact in both, so that whole units then have the bits of that kernel at a third of its time: 8 x 1600 x 4607 148 -> 62 us (one
// block per CTA), 8 x 4096 x 5665 363 -> 105 us. It costs 2 %: the packed sums follow the register pairs of the exponents otherwise.
// EIGHTS: a row's sums of squares come in groups of eight (ss_group). A form of its own: as a branch of the others it cost them 1 to 3 %.
template <int HD, int BLOCKS, bool ORDERED, bool HAND, bool EIGHTS>
__global__ void __launch_bounds__(kThreads, 1)
attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, __half* __restrict__ O, int H, int Sq, int n_keys,
                    int o_bshd, float scale_log2e_all, const float* __restrict__ row_ss, int ss_tiles, float inv_norm_dim,
                    float norm_eps, unsigned char* __restrict__ ws, int v_heads, const __grid_constant__ WorkList work) {
    using C = Cfg<HD, BLOCKS>;
    constexpr int kRows = BLOCKS * BM;  // queries of a unit
    constexpr int kStages = C::kStages, kSBufs = C::kSBufs, kQBytes = C::kQBytes, kKBytes = C::kKBytes, kStageBytes = C::kStageBytes;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = tc::smem_addr(smem_raw);
    if (base & 1023u) {  // uniform over the CTA, nothing allocated yet
        if (threadIdx.x == 0) atomicCAS(&g_attn_tc_error, 0, kErrSmemAlign);
        return;
    }
    const uint32_t sQ = base, sKV = base + BLOCKS * kQBytes;
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + BLOCKS * kQBytes + kStages * kStageBytes);
    volatile int* abort_flag = &ctrl->abort;
    // kCorr: [block][score buffer][row], what a row's O is multiplied by ahead of the tile in that buffer
    float* const factors = reinterpret_cast<float*>(smem_raw + BLOCKS * kQBytes + kStages * kStageBytes + 512);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // this CTA's work: a whole unit, or a piece of one (n_tiles key tiles from tile t0)
    int unit = blockIdx.x, t0 = 0, n_tiles = (n_keys + BN - 1) / BN, split_count = 1, split_first = 0, split_slot = 0;
    const bool gives = HAND && (int)blockIdx.x < work.heads;   // the first piece of a unit, whose state another CTA takes over
    const bool second = HAND && (int)blockIdx.x >= work.heads + work.whole_units;
    bool takes = false;                                         // a second piece that has the first one's state
    if (HAND) {
        unit = blockIdx.x - work.heads;
        if (gives || second) {
            const Piece& pc = work.pieces[gives ? blockIdx.x : blockIdx.x - work.whole_units];
            unit = pc.unit; t0 = pc.t0; n_tiles = pc.nt; split_slot = pc.slot;
        }
    } else if ((int)blockIdx.x >= work.whole_units) {
        const Piece& pc = work.pieces[blockIdx.x - work.whole_units];
        unit = pc.unit; t0 = pc.t0; n_tiles = pc.nt; split_count = pc.count; split_first = pc.first; split_slot = pc.slot;
    }
    const int q0 = (unit % work.q_blocks) * kRows;
    const int bh = unit / work.q_blocks;

    if (tid == 0) {
        tc::mbar_init(&ctrl->q_full, 1);
        for (int s = 0; s < kStages; ++s) { tc::mbar_init(&ctrl->kv_full[s], 1); tc::mbar_init(&ctrl->kv_empty[s], BLOCKS); }
        for (int k = 0; k < BLOCKS; ++k)
            for (int b = 0; b < kSBufs; ++b) {
                tc::mbar_init(&ctrl->s_full[k][b], 1); tc::mbar_init(&ctrl->p_full[k][b], C::kCorr ? 8 : 4); tc::mbar_init(&ctrl->pv_done[k][b], 1);
                tc::mbar_init(&ctrl->move_full[k][b], 4);
            }
        for (int k = 0; k < 2 * BLOCKS; ++k) tc::mbar_init(&ctrl->drain[k], 1);
        ctrl->abort = 0;
        ctrl->merge = 0;
        tc::fence_barrier_init();
    }
    if (warp == 8 && lane == 0) {  // descriptors are kernel arguments: fetched ahead of the wait for the kernel before
        tc::prefetch_tensormap(&map_q); tc::prefetch_tensormap(&map_k); tc::prefetch_tensormap(&map_v);
    }
    if (warp == 9) {  // beside the barriers
        tc::tmem_alloc(&ctrl->tmem_base, kTmemCols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem_cta = ctrl->tmem_base;
    // everything above touched only this CTA's shared and tensor memory; the operands below are another kernel's output
    pdl_wait();
    pdl_trigger();
    if (second) {   // ahead of the roles, which then take either the rest of the unit or all of it
        if (tid == 0) ctrl->merge = wait_handed(reinterpret_cast<int*>(ws) + split_slot);
        __syncthreads();
        takes = __any_sync(0xffffffffu, ctrl->merge != 0);   // the same in every lane: by a vote, so that what follows from it takes no registers a thread
        if (!takes) { t0 = 0; n_tiles = (n_keys + BN - 1) / BN; }
    }

    // The register hand-over: every warp of a warpgroup executes the same setmaxnreg instruction (warpgroups 2 and 3 the
    // release, 0 and 1 the take), as the first statement of a branch that does not meet the other again before the
    // teardown - placed ahead of the branch, the compiler bound every role by the smaller budget.
    if (C::kCorr && warp >= C::kCorrWarp && warp < C::kCorrWarp + 4) {
        regs_release<C::kRegCorr>();
        // ------------------------------------------------------------ rescale of O (128-wide heads), a warp for its 32 lanes of every block
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const int r = (warp & 3) * 32 + lane;
        bool ok = true;
        int buf = 0, buf_par = 0;
        for (int j = 0; ok && j < n_tiles; ++j) {
            const int pbuf = buf == 0 ? kSBufs - 1 : buf - 1, pbuf_par = buf == 0 ? buf_par ^ 1 : buf_par;  // of tile j - 1
            for (int blk = 0; ok && blk < BLOCKS; ++blk) {
                ok = tc::mbar_wait_warp(&ctrl->move_full[blk][buf], buf_par, abort_flag);
                if (!ok) break;
                const float alpha = factors[(blk * kSBufs + buf) * BM + r];
                if (__any_sync(0xffffffffu, alpha != 1.0f)) {
                    // O belongs to the tensor core until the previous tile's P V is done (a tile's move_full comes behind its s_full, so
                    // the parity is unambiguous); ahead of its first tile a taken-over O is the softmax warps'.
                    if (j > 0) ok = tc::mbar_wait_warp(&ctrl->pv_done[blk][pbuf], pbuf_par, abort_flag);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint32_t tO = tmem_cta + blk * 256 + kSBufs * 64 + lane_off;
                    uint32_t v[2][32];
                    tc::tmem_ld32(tO, v[0]);
#pragma unroll
                    for (int hc = 0; hc < HD / 32; ++hc) {
                        tc::tc_wait_ld(v[hc & 1]);
                        if (hc + 1 < HD / 32) tc::tmem_ld32(tO + (hc + 1) * 32, v[(hc + 1) & 1]);
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[hc & 1][i] = __float_as_uint(__uint_as_float(v[hc & 1][i]) * alpha);
                        tc::tmem_st32(tO + hc * 32, v[hc & 1]);
                    }
                    tc::tc_wait_st();
                    tc::tc_fence_before();
                }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&ctrl->p_full[blk][buf]);
            }
            if (++buf == kSBufs) { buf = 0; buf_par ^= 1; }
        }
    } else if (warp >= 4 * BLOCKS) {
    regs_release<C::kRegIssue>();
    if (warp == 8) {
        // ------------------------------------------------------------ producer (one thread)
        if (lane == 0) {
            tc::mbar_arrive_expect_tx(&ctrl->q_full, BLOCKS * kQBytes);
            for (int k = 0; k < BLOCKS; ++k)
                for (int x = 0; x < C::kSub; ++x)
                    tc::tma_load_3d(sQ + k * kQBytes + x * C::kQSub, &map_q, x * 64, q0 + k * BM, bh, &ctrl->q_full);
            int issued = 0;
            for (int j = 0; j < n_tiles; ++j) {
                const int s = j % kStages;
                // stage s was last read by the products of tile j - kStages (phase j / kStages - 1 of kv_empty[s])
                if (j >= kStages && !tc::mbar_wait(&ctrl->kv_empty[s], ((j / kStages) + 1) & 1, abort_flag)) break;
                tc::mbar_arrive_expect_tx(&ctrl->kv_full[s], kStageBytes);
#pragma unroll
                for (int x = 0; x < C::kSub; ++x)
                    tc::tma_load_3d(sKV + s * kStageBytes + x * C::kKSub, &map_k, x * 64, (t0 + j) * BN, bh, &ctrl->kv_full[s]);
#pragma unroll
                for (int x = 0; x < C::kSub; ++x)
                    tc::tma_load_3d(sKV + s * kStageBytes + kKBytes + x * C::kKSub, &map_v, x * 64, (t0 + j) * BN, bh % v_heads,
                                    &ctrl->kv_full[s]);
                issued = j + 1;
            }
            if (*abort_flag) {
                // The CTA is giving up. Every copy this thread started lands in this CTA's shared memory and counts
                // on a kv_full / q_full barrier: wait (bounded) for the last copy of each stage before the CTA exits.
                tc::mbar_wait_drain(&ctrl->q_full, 0);
                for (int s = 0; s < kStages && s < issued; ++s) {
                    const int last = ((issued - 1 - s) / kStages) * kStages + s;  // last tile loaded into stage s
                    tc::mbar_wait_drain(&ctrl->kv_full[s], (last / kStages) & 1);
                }
            }
        }
        __syncwarp();
    } else if (warp == 9 || (BLOCKS == 2 && warp == 10)) {
        const int blk = warp - 9;
        const uint32_t tmem = tmem_cta + blk * 256, tmem_O = tmem + kSBufs * 64;
        // ------------------------------------------------------------ issuer of O += P V (the warp's elected lane)
        // The whole warp runs the loop and one lane issues (elect_one): with a single thread's loop the issue of a tile's
        // products, not the tensor pipe, paced the 128-wide heads (8 x 4096 x 5665: 96 -> 84 us with the trailing reference they
        // had then; 64-wide heads 142 -> 139 us). The elected lane in a loop of its own is 1 to 4 % slower here.
        // tile j: score buffer j % kSBufs (its use number j / kSBufs gives the barrier phase), ring stage j % kStages
        const bool leader = tc::elect_one();
        constexpr uint32_t idesc_pv = tc::umma_idesc_f16(BM, HD, 1);  // B = V tile, MN-major
        // MN-major operand: the leading byte offset is the distance between its 64-column sub-tiles
        const uint32_t v_lo = ((sKV + kKBytes) >> 4 & 0x3fffu) | ((HD == 64 ? 1u : (uint32_t)(C::kKSub >> 4)) << 16);
        bool ok = true;
        int buf = 0, buf_par = 0, st = 0;
        for (int j = 0; ok && j < n_tiles; ++j) {
            ok = tc::mbar_wait_warp(&ctrl->p_full[blk][buf], buf_par, abort_flag);
            if (!ok) break;
            tc::tc_fence_after();
            if (leader) {
                const uint32_t p_tmem = tmem + buf * 64, vt_lo = v_lo + st * (kStageBytes >> 4);
#pragma unroll
                for (int ks = 0; ks < BN / 16; ++ks)  // P: 16 keys = 8 columns; V: 16 keys = 16 rows of 128 bytes
                    tc::umma_f16_ts_lo(tmem_O, p_tmem + ks * 8, vt_lo + ks * (2048 >> 4), idesc_pv, (j > 0) || (ks > 0) || (HAND && takes));
                tc::umma_commit(&ctrl->kv_empty[st]);  // K of this stage was consumed before its scores could be read
                tc::umma_commit(&ctrl->pv_done[blk][buf]);
            }
            if (++buf == kSBufs) { buf = 0; buf_par ^= 1; }
            if (++st == kStages) st = 0;
        }
        if (leader && *abort_flag) {  // giving up: let this lane's products finish before tensor memory is freed
            tc::umma_commit(&ctrl->drain[blk]);
            tc::mbar_wait_drain(&ctrl->drain[blk], 0);
        }
        __syncwarp();
    } else if (warp == C::kQkWarp || (BLOCKS == 2 && !C::kCorr && warp == 12)) {
        constexpr int kBlks = C::kCorr ? BLOCKS : 1;    // blocks of this warp
        const int blk0 = warp - C::kQkWarp;
        // ------------------------------------------------------------ issuer of S = Q K^T (the warp's elected lane)
        const bool leader = tc::elect_one();
        constexpr uint32_t idesc_qk = tc::umma_idesc_f16(BM, BN, 0);  // B = K tile, K-major
        const uint32_t q_lo0 = tc::umma_desc_lo(sQ + blk0 * kQBytes), k_lo = tc::umma_desc_lo(sKV);
        bool ok = tc::mbar_wait_warp(&ctrl->q_full, 0, abort_flag);
        int buf = 0, buf_par = 0, st = 0, st_par = 0;
        for (int j = 0; ok && j < n_tiles; ++j) {
            ok = tc::mbar_wait_warp(&ctrl->kv_full[st], st_par, abort_flag);
#pragma unroll
            for (int b = 0; b < kBlks; ++b) {
                const int blk = blk0 + b;
                // the buffer still holds P of tile j - kSBufs until that tile's P V is complete
                if (ok && j >= kSBufs) ok = tc::mbar_wait_warp(&ctrl->pv_done[blk][buf], buf_par ^ 1, abort_flag);
                if (!ok) break;
                tc::tc_fence_after();
                if (leader) {
                    const uint32_t kt_lo = k_lo + st * (kStageBytes >> 4), q_lo = q_lo0 + b * (kQBytes >> 4);
#pragma unroll
                    for (int ks = 0; ks < HD / 16; ++ks)  // 16 head-dim elements = 32 bytes along a row of a sub-tile
                        tc::umma_f16_lo(tmem_cta + blk * 256 + buf * 64, q_lo + (ks / 4) * (C::kQSub >> 4) + (ks % 4) * 2,
                                        kt_lo + (ks / 4) * (C::kKSub >> 4) + (ks % 4) * 2, idesc_qk, ks > 0);
                    tc::umma_commit(&ctrl->s_full[blk][buf]);
                }
            }
            if (++buf == kSBufs) { buf = 0; buf_par ^= 1; }
            if (++st == kStages) { st = 0; st_par ^= 1; }
        }
        if (leader && *abort_flag) {
            tc::umma_commit(&ctrl->drain[BLOCKS + blk0]);
            tc::mbar_wait_drain(&ctrl->drain[BLOCKS + blk0], 0);
        }
        __syncwarp();
    }  // the other warps have no role beyond handing their registers back together with their warpgroup
    } else {
        regs_take<C::kRegSoftmax>();
        // ------------------------------------------------------------ softmax, warps 0-7 (query block = warp / 4)
        constexpr unsigned kFull = 0xffffffffu;
        constexpr float kSumLimit = 256.0f;  // 2^8, the threshold below
        constexpr uint32_t kNegInf = 0xff800000u;
        // The reference ahead of a row's first finite score: far below every such score (at most 65504^2 * HD), so that the
        // first one moves it, and finite, so that scores of -inf give P = 0 and not the exponential of a difference of
        // infinities.
        constexpr float kNoMax = -1.0e30f;
        // In exponent units: P stays below 2^8, well inside fp16. With 128-wide heads the reference is the row's exact running
        // maximum, as in flash_attention_kernel: a row's largest probabilities are then exactly 1 or round on the finer half
        // of their binade. Against 64 bits the deferred reference was 3 % further off than that kernel on unit-variance
        // scores and 19 to 21 % on scores of two and three times that; with the exact one the two agree to 1e-4 (8 x 4096 x
        // 5665: 81 us deferred, 102 us exact, 92 with O rescaled by its own warpgroup, 361 us flash_attention_kernel).
        constexpr bool kExactMax = HD == 128;
        constexpr float kRescaleThreshold = kExactMax ? 0.0f : 8.0f;
        const int blk = warp >> 2;
        const int r = (warp & 3) * 32 + lane;                       // query row within the block = its tensor-memory lane
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;  // a warp reaches lanes [32 * (warp % 4), +32)
        const uint32_t tmem = tmem_cta + blk * 256, tmem_O = tmem + kSBufs * 64;
        const uint32_t tO = tmem_O + lane_off;
        // Queries that arrive un-normalised (rfk_gemm_f16_heads) bring the partial sums of squares of their rows: the
        // RMSNorm's 1 / rms is a per-row factor of the scores, i.e. of this thread's exponent scale (the norm's weight
        // is folded into the keys by the caller). The row statistic spans all heads of the token.
        float scale_log2e = scale_log2e_all;
        if (row_ss) {
            const int q = min(q0 + blk * BM + r, Sq - 1);
            const float* sp = row_ss + ((size_t)(bh / H) * Sq + q) * ss_tiles;
            float ss = 0.0f;
            if constexpr (!EIGHTS) {
                for (int t = 0; t < ss_tiles; ++t) ss += __ldg(sp + t);
            } else {
                for (int t = 0; t < ss_tiles; t += 8) {
                    const float4 a = __ldg(reinterpret_cast<const float4*>(sp + t)), b = __ldg(reinterpret_cast<const float4*>(sp + t + 4));
                    ss += ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
                }
            }
            scale_log2e *= rsqrtf(ss * inv_norm_dim + norm_eps);
        }
        float m_run = kNoMax, l_run = 0.0f;
        float2 l01 = make_float2(0.0f, 0.0f), l23 = l01;  // ORDERED: the row sum in its four parts (exp_half)
        uint32_t va[32], vb[32];
        bool ok = true;
        int buf = 0, buf_par = 0;  // score buffer of tile j and the phase parity of its barriers
        // HAND: this row's place in the handed-over state, [16 or 32 groups of 4 columns][256 rows] float4 as above
        auto handed_row = [&](int slot) {
            return reinterpret_cast<uint4*>(ws + kWsCounterBytes + kWsMlBytes) + (size_t)slot * (2 * HD / 4) * kUnitRows + blk * BM + r;
        };
        if (HAND && takes) {  // O, the row sum and the reference where the first piece left them
            const uint4* const handed = handed_row(split_slot);
#pragma unroll
            for (int hc = 0; hc < HD / 32; ++hc) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 w = __ldcg(handed + (hc * 8 + c) * kUnitRows);
                    va[4 * c] = w.x; va[4 * c + 1] = w.y; va[4 * c + 2] = w.z; va[4 * c + 3] = w.w;
                }
                tc::tmem_st32(tO + hc * 32, va);
            }
            tc::tc_wait_st();
            if (C::kCorr) tc::tc_fence_before();   // the rescaling warps' from here on, by way of move_full
            const uint4 l = __ldcg(handed + (HD / 4) * kUnitRows), m = __ldcg(handed + (HD / 4 + 1) * kUnitRows);
            l_run = __uint_as_float(l.x);
            l01 = make_float2(__uint_as_float(l.x), __uint_as_float(l.y));
            l23 = make_float2(__uint_as_float(l.z), __uint_as_float(l.w));
            m_run = __uint_as_float(m.x);
        }
        // From 1 on for a taken-over unit: tile 0 is where a unit begins. (The tile before its first counts as multiplied: a wait for the
        // previous phase of a new barrier returns at once.)
        const int j0 = HAND && takes ? 1 : 0, j_end = n_tiles + j0, j_key = t0 - j0;
        for (int j = j0; ok && j < j_end; ++j) {
            const uint32_t tS = tmem + lane_off + buf * 64;
            ok = tc::mbar_wait_warp(&ctrl->s_full[blk][buf], buf_par, abort_flag);
            if (!ok) break;
            tc::tc_fence_after();
            const int n_valid = min(BN, n_keys - (j_key + j) * BN);  // real keys among this tile's 64 columns
            tc::tmem_ld32(tS, va);
            tc::tc_wait_ld(va);
            tc::tmem_ld32(tS + 32, vb);  // in flight during the first half's arithmetic
            if (n_valid != BN) {  // last tile: keys at or beyond n_keys score -inf, i.e. contribute nothing
                tc::tc_wait_ld(vb);
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    if (i >= n_valid) va[i] = kNegInf;
                    if (32 + i >= n_valid) vb[i] = kNegInf;
                }
            }
            // The running maximum only follows a tile's maximum when it would move by more than the threshold; until
            // then the probabilities of the row are scaled by up to 2^threshold, which cancels in O / l. So the common
            // tile leaves the reference where it is, and its exponentials start from the reference already known,
            // without this tile's maximum ahead of them: if afterwards no row's probabilities sum to more than
            // 2^threshold, none of them exceeded it and the tile is done. Otherwise (and for the first and the last
            // tile) the scores are read again, the maximum is taken and the same code runs once more.
            float2 acc0, acc1;
            float m_new = m_run, alpha = 1.0f;
            bool any_move = false, need_max = kExactMax || j == 0 || n_valid != BN;
#pragma unroll 1
            for (;;) {
                acc0 = make_float2(0.0f, 0.0f);
                acc1 = make_float2(0.0f, 0.0f);
                if (need_max) {
                    tc::tc_wait_ld(vb);
                    float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        m0 = fmax3(m0, __uint_as_float(va[i]), __uint_as_float(va[i + 1]));
                        m1 = fmax3(m1, __uint_as_float(va[i + 2]), __uint_as_float(va[i + 3]));
                        m2 = fmax3(m2, __uint_as_float(vb[i]), __uint_as_float(vb[i + 1]));
                        m3 = fmax3(m3, __uint_as_float(vb[i + 2]), __uint_as_float(vb[i + 3]));
                    }
                    const float m_tile = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
                    // first tile: always, with a finite score
                    const bool move = kExactMax ? m_tile > m_run : (m_tile - m_run) * scale_log2e > kRescaleThreshold;
                    m_new = move ? m_tile : m_run;
                    any_move = __any_sync(kFull, move);
                    if (any_move && move) alpha = fast_exp2((m_run - m_new) * scale_log2e);  // first tile: 0
                    if (C::kCorr) {  // the first tile's product overwrites O, unless it was taken over
                        factors[(blk * kSBufs + buf) * BM + r] = j > 0 ? alpha : 1.0f;
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&ctrl->move_full[blk][buf]);
                    }
                }
                // P = exp2(scale * log2e * (S - max)), two fp16 per 32-bit column: keys 2i, 2i+1 in column i;
                // the 32 packed words end up in va, which is what the store below takes
                const float mc = m_new * scale_log2e;
                float poly_max = -INFINITY;
                exp_half<HD, ORDERED>(va, va, scale_log2e, mc, acc0, acc1, poly_max);
                tc::tc_wait_ld(vb);
                exp_half<HD, ORDERED>(vb, va + 16, scale_log2e, mc, acc0, acc1, poly_max);
                if (need_max) break;
                const float sum = (acc0.x + acc0.y) + (acc1.x + acc1.y);
                if (!__any_sync(kFull, !(sum <= kSumLimit) || poly_max > kRescaleThreshold)) break;
                need_max = true;
                tc::tmem_ld32(tS, va);
                tc::tc_wait_ld(va);
                tc::tmem_ld32(tS + 32, vb);
            }
            if (!C::kCorr && j > 0 && any_move) {  // rescale this warp's 32 rows of O (vb is free here)
                // O belongs to the tensor core until the previous tile's P V is done. Having seen s_full of tile j,
                // P V of tile j - 1 - kSBufs (the previous phase of this barrier) is known complete: the parity is unambiguous.
                const int pbuf = buf == 0 ? kSBufs - 1 : buf - 1, pbuf_par = buf == 0 ? buf_par ^ 1 : buf_par;  // of tile j - 1
                ok = tc::mbar_wait_warp(&ctrl->pv_done[blk][pbuf], pbuf_par, abort_flag);
                if (!ok) break;
                tc::tc_fence_after();
#pragma unroll
                for (int hc = 0; hc < HD / 32; ++hc) {
                    tc::tmem_ld32(tO + hc * 32, vb);
                    tc::tc_wait_ld(vb);
#pragma unroll
                    for (int i = 0; i < 32; ++i) vb[i] = __float_as_uint(__uint_as_float(vb[i]) * alpha);
                    tc::tmem_st32(tO + hc * 32, vb);
                }
            }
            if (ORDERED) {
                const float2 a2 = make_float2(alpha, alpha);
                l01 = __ffma2_rn(l01, a2, acc0);
                l23 = __ffma2_rn(l23, a2, acc1);
            } else {
                l_run = (any_move ? l_run * alpha : l_run) + ((acc0.x + acc0.y) + (acc1.x + acc1.y));
            }
            m_run = m_new;
            tc::tmem_st32(tS, va);    // P over the first 32 columns of this thread's own lane of S
            tc::tc_wait_st();
            tc::tc_fence_before();    // the writes of P and O come before the arrival
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&ctrl->p_full[blk][buf]);
            if (++buf == kSBufs) { buf = 0; buf_par ^= 1; }
        }
        if (ORDERED && !gives) l_run = (l01.x + l01.y) + (l23.x + l23.y);
        // ---- epilogue: O / l -> fp16 -> global, one 128-byte row per thread
        if (ok) {  // buf / buf_par have moved on to tile n_tiles: step back to the last tile
            const int lbuf = buf == 0 ? kSBufs - 1 : buf - 1, lbuf_par = buf == 0 ? buf_par ^ 1 : buf_par;
            ok = tc::mbar_wait_warp(&ctrl->pv_done[blk][lbuf], lbuf_par, abort_flag);
        }
        const int q = q0 + blk * BM + r;
        __half* dst = o_bshd ? O + (((size_t)(bh / H) * Sq + q) * H + bh % H) * HD : O + ((size_t)bh * Sq + q) * HD;
        if (gives) {
            // ---- first piece of a unit that is handed over: O, row sum and reference as they stand
            if (ok) {
                uint4* const handed = handed_row(work.pieces[blockIdx.x].slot);
                tc::tc_fence_after();
#pragma unroll
                for (int hc = 0; hc < HD / 32; ++hc) {
                    tc::tmem_ld32(tO + hc * 32, va);
                    tc::tc_wait_ld(va);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        __stcg(handed + (hc * 8 + c) * kUnitRows, make_uint4(va[4 * c], va[4 * c + 1], va[4 * c + 2], va[4 * c + 3]));
                }
                __stcg(handed + (HD / 4) * kUnitRows,
                       ORDERED ? make_uint4(__float_as_uint(l01.x), __float_as_uint(l01.y), __float_as_uint(l23.x), __float_as_uint(l23.y))
                               : make_uint4(__float_as_uint(l_run), 0, 0, 0));
                __stcg(handed + (HD / 4 + 1) * kUnitRows, make_uint4(__float_as_uint(m_run), 0, 0, 0));
                __threadfence();
            }
        } else if (BLOCKS == 1 || HAND || split_count == 1) {
            if (ok) {
                tc::tc_fence_after();
                const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
#pragma unroll
                for (int hc = 0; hc < HD / 32; ++hc) {
                    tc::tmem_ld32(tO + hc * 32, va);
                    tc::tc_wait_ld(va);
                    if (q < Sq) store_row_half(dst + hc * 32, va, inv);
                }
            }
        } else {
            // ---- a piece of a split unit: publish (m, l, O), count, and merge if this CTA completes the unit
            float* ws_ml = reinterpret_cast<float*>(ws + kWsCounterBytes);
            float* ws_o = reinterpret_cast<float*>(ws + kWsCounterBytes + kWsMlBytes);
            const int row = blk * BM + r;
            if (ok) {
                tc::tc_fence_after();
                uint4* po = reinterpret_cast<uint4*>(ws_o) + (size_t)split_slot * (HD / 4) * kUnitRows + row;
#pragma unroll
                for (int hc = 0; hc < HD / 32; ++hc) {
                    tc::tmem_ld32(tO + hc * 32, va);
                    tc::tc_wait_ld(va);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        __stcg(po + (hc * 8 + c) * kUnitRows, make_uint4(va[4 * c], va[4 * c + 1], va[4 * c + 2], va[4 * c + 3]));
                }
                // the exponent reference in exponent units (the row's own scale applied), so that pieces compare directly
                __stcg(reinterpret_cast<float2*>(ws_ml + ((size_t)split_slot * kUnitRows + row) * 2), make_float2(m_run * scale_log2e, l_run));
                __threadfence();
            }
            softmax_warps_sync();  // every softmax warp comes here, whatever its ok: the barrier cannot be left short
            if (tid == 0) {
                int* counter = reinterpret_cast<int*>(ws) + (unit - work.whole_units);
                const bool failed = *abort_flag != 0;
                const handover::Arrival a = handover::arrive(atomicAdd(counter, handover::piece(failed)), failed, split_count);
                if (a.last) {
                    *counter = 0;  // every piece of the unit has arrived, or given up: ready for the next launch
                    __threadfence();
                }
                ctrl->merge = a.merge;
            }
            softmax_warps_sync();
            if (ctrl->merge && ok) {
                float m_all = -INFINITY;
                for (int p = 0; p < split_count; ++p)
                    m_all = fmaxf(m_all, __ldcg(ws_ml + ((size_t)(split_first + p) * kUnitRows + row) * 2));
                float l_all = 0.0f;
                for (int p = 0; p < split_count; ++p) {  // in slot order, whichever CTA merges: the sum is reproducible
                    const float2 ml = __ldcg(reinterpret_cast<const float2*>(ws_ml + ((size_t)(split_first + p) * kUnitRows + row) * 2));
                    l_all += fast_exp2(ml.x - m_all) * ml.y;
                }
                const float inv = l_all > 0.0f ? 1.0f / l_all : 0.0f;
#pragma unroll 1
                for (int x = 0; x < C::kSub; ++x) {  // 64 merged outputs of this row at a time, in va and vb
                    float* acc = reinterpret_cast<float*>(va);
                    float* acc2 = reinterpret_cast<float*>(vb);
#pragma unroll
                    for (int i = 0; i < 32; ++i) { acc[i] = 0.0f; acc2[i] = 0.0f; }
                    for (int p = 0; p < split_count; ++p) {
                        const float w = fast_exp2(__ldcg(ws_ml + ((size_t)(split_first + p) * kUnitRows + row) * 2) - m_all);
                        const float4* src = reinterpret_cast<const float4*>(ws_o) +
                                            ((size_t)(split_first + p) * (HD / 4) + x * 16) * kUnitRows + row;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            const float4 a = __ldcg(src + c * kUnitRows), b = __ldcg(src + (8 + c) * kUnitRows);
                            acc[4 * c] += w * a.x; acc[4 * c + 1] += w * a.y; acc[4 * c + 2] += w * a.z; acc[4 * c + 3] += w * a.w;
                            acc2[4 * c] += w * b.x; acc2[4 * c + 1] += w * b.y; acc2[4 * c + 2] += w * b.z; acc2[4 * c + 3] += w * b.w;
                        }
                    }
                    if (q < Sq) {
                        store_row_half(dst + x * 64, va, inv);
                        store_row_half(dst + x * 64 + 32, vb, inv);
                    }
                }
            }
        }
    }

    // ---- teardown: every path (normal or aborted) arrives here with no divergence inside a warp
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem_cta, kTmemCols);
    }
    if (gives && tid == 32) {   // every softmax warp has written its rows of the state, or given up
        const bool left = *abort_flag == 0;
        __threadfence();
        handover_step(reinterpret_cast<int*>(ws) + split_slot, handover::kIdle, [left](int w) { return handover::give(w, left); });
    }
    if (tid == 0 && ctrl->abort) atomicCAS(&g_attn_tc_error, 0, kErrTimeout);
}

}  // namespace tcattn

std::atomic<int> g_attn_path{0};  // 0 automatic, 1 mma.sync kernel, 2 tcgen05 kernel
std::atomic<int> g_attn_split{1};  // 0: never split keys, even with a workspace (to time both side by side)

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

// fp16 tensor [n_heads][rows][hd], contiguous; boxes of box_rows x 64 in the 128-byte-swizzled layout,
// rows past the end of a head read as zeros
bool make_map(CUtensorMap* m, const void* base, long long n_heads, long long rows, int hd, int box_rows) {
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)rows, (cuuint64_t)n_heads};
    const cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)rows * hd * 2};  // bytes, dimensions 1 and 2
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Fills `w` for `units` units of `n_tiles` key tiles each on a device with `sms` SMs (see "Key split" above): full rounds
// of units run whole, and the units of the last, partial round are cut when the estimate says it pays. split = false: every
// unit whole; cut_last_round = false: every unit of a grid of one round or more whole. A cut changes the order of the sums, so
// whether a unit is cut, and where, must not depend on what else is in the launch where the caller promises equal bits.
void plan_work(tcattn::WorkList& w, long long units, int n_tiles, int sms, bool split, bool cut_last_round) {
    using tcattn::Piece;
    constexpr int kPieceCostTiles = 12;  // what a piece costs beyond its tiles (fill, publishing, merging), in tile times
    w.whole_units = (int)units;
    w.n_pieces = w.heads = 0;
    if (!split || sms <= 0 || units <= 0 || n_tiles > 65535 || units > 65535) return;
    const int rounds = (int)(units / sms), rest = (int)(units % sms);
    if (rest == 0 || rest > 256 || (rounds > 0 && !cut_last_round)) return;  // 256 unit counters
    const long long tiles = (long long)rest * n_tiles;
    constexpr int kMaxPiecesPerUnit = 8;  // the CTA that merges a unit reads its pieces one after the other
    const int shares = (int)std::min<long long>(std::min(sms, tcattn::kMaxPieces / 2), (long long)rest * kMaxPiecesPerUnit);
    // whole: one more round of n_tiles; split: a share's tiles plus the piece overhead. Cut only for a clear gain: a fifth of
    // the launch. (Measured where the estimate gives 7 %, 256 units of 89 tiles on 148 SMs: nothing gained. 184 units of 89
    // tiles, estimate 31 %: 200 -> 153 us at head size 128; 208 units, estimate 23 %: 139 -> 114 us and 160 units of 40 tiles,
    // 29 %: 68 -> 52 us at head size 64.) A line of a tenth gains too (368 units of 89 tiles, estimate 12 %: 209 -> 189 us at head
    // size 64), but it moves the sums, and so the K/V cache and every view, of scenes that this line leaves whole: the line is
    // part of what rfk_flash_attention_ex and the sessions promise, and stays.
    if (((long long)rounds * n_tiles + (tiles + shares - 1) / shares + kPieceCostTiles) * 5 > (long long)(rounds + 1) * n_tiles * 4) return;
    const int whole = rounds * sms;
    Piece* pc = w.pieces;
    int n = 0;
    for (int s = 0; s < shares; ++s) {
        long long b = tiles * s / shares;
        const long long e = tiles * (s + 1) / shares;
        while (b < e) {  // at most twice: a share is shorter than a unit
            const long long u = b / n_tiles, pe = std::min(e, (u + 1) * n_tiles);
            pc[n].unit = (uint16_t)(whole + u);
            pc[n].t0 = (uint16_t)(b - u * n_tiles);
            pc[n].nt = (uint16_t)(pe - b);
            pc[n].slot = (uint16_t)n;
            ++n;
            b = pe;
        }
    }
    for (int i = 0; i < n;) {  // pieces of a unit are consecutive here: give each its unit's slot range
        int j = i;
        while (j < n && pc[j].unit == pc[i].unit) ++j;
        for (int k = i; k < j; ++k) { pc[k].first = (uint16_t)i; pc[k].count = (uint16_t)(j - i); }
        i = j;
    }
    // longest first: in-order dispatch then hands the short pieces to the SMs that finish their long ones first
    std::stable_sort(pc, pc + n, [](const Piece& a, const Piece& b) { return a.nt > b.nt; });
    w.whole_units = whole;
    w.n_pieces = n;
}

// Hand-over (see above) for a grid that plan_work leaves whole: fills the SMs one after the other to the same budget of tile times,
// each with the first piece of the unit that the SM before it left cut, whole units, and the last keys of one more unit. The
// hardware hands the blocks out in order: the first pieces, the whole units, then the second pieces, longest first, which
// comes to the same.
void plan_handover(tcattn::WorkList& w, long long units, int n_tiles, int sms) {
    using tcattn::Piece;
    // Beyond its tiles every CTA costs some (set-up, first scores, last product, output), a hand-over some more on both sides.
    constexpr int kCtaCost = 5, kGiveCost = 2, kTakeCost = 2, kMinPiece = 4;
    if (sms <= 0 || sms > tcattn::kMaxHanded || units <= sms || units > 65535 || n_tiles > 65535 || n_tiles < 4 * kMinPiece) return;
    const int whole = n_tiles + kCtaCost;
    const long long uncut = (units + sms - 1) / sms * whole;
    uint16_t tail[tcattn::kMaxHanded];
    for (long long budget = (units * whole + (sms - 1) * (kCtaCost + kGiveCost + kTakeCost)) / sms; budget * 100 <= uncut * 95; ++budget) {
        long long left = units;   // units not yet begun
        int n = 0, open = 0;      // cut units; tiles of the first piece of the last of them, not yet placed
        for (int s = 0; s < sms && (left > 0 || open > 0); ++s) {
            long long room = budget;
            if (open > 0) room -= open + kCtaCost + kGiveCost;
            open = 0;
            const long long k = std::min(left, std::max(0LL, room / whole));
            left -= k;
            room -= k * whole + kCtaCost + kTakeCost;
            if (left > 0 && room >= kMinPiece) {
                tail[n] = (uint16_t)std::min<long long>(room, n_tiles - kMinPiece);
                open = n_tiles - tail[n++];
                --left;
            }
        }
        if (left > 0 || open > 0) continue;   // the budget does not hold them
        if (n == 0) return;
        w.whole_units = (int)units - n;
        w.heads = n;
        w.n_pieces = 2 * n;
        for (int i = 0; i < n; ++i) {
            const uint16_t unit = (uint16_t)(w.whole_units + i), t0 = (uint16_t)(n_tiles - tail[i]);
            w.pieces[i] = Piece{unit, 0, t0, (uint16_t)i, 1, (uint16_t)i};
            w.pieces[n + i] = Piece{unit, t0, tail[i], (uint16_t)i, 1, (uint16_t)i};
        }
        const auto longer = [](const Piece& a, const Piece& b) { return a.nt > b.nt; };
        std::stable_sort(w.pieces, w.pieces + n, longer);
        std::stable_sort(w.pieces + n, w.pieces + 2 * n, longer);
        return;
    }
}

// Whether a grid without cut units runs with one block of 128 queries per CTA (see "One block per CTA" above): when each block
// finds an SM of its own.
bool one_block_per_cta(int n_pieces, long long blocks, int sms) { return n_pieces == 0 && blocks <= sms; }

}  // namespace

size_t attention_tc_workspace_bytes() { return tcattn::kWsBytes; }

// The launcher's plan for a grid, without launching anything (host only: no device is touched).
int attention_tc_plan(long long units, int n_tiles, int sms, int* whole_units, int* n_pieces, unsigned short* pieces, int max_pieces) {
    if (units < 0 || n_tiles <= 0 || sms <= 0 || !whole_units || !n_pieces || max_pieces < 0 || (max_pieces && !pieces)) return RFK_EINVAL;
    tcattn::WorkList w;
    plan_work(w, units, n_tiles, sms, true, true);
    *whole_units = w.whole_units;
    *n_pieces = w.n_pieces;
    for (int i = 0; i < w.n_pieces && i < max_pieces; ++i) {
        const tcattn::Piece& pc = w.pieces[i];
        const unsigned short rec[6] = {pc.unit, pc.t0, pc.nt, pc.first, pc.count, pc.slot};
        for (int k = 0; k < 6; ++k) pieces[i * 6 + k] = rec[k];
    }
    return RFK_OK;
}

// plan_handover's, the same way: *n_handed units, each three values {unit, tiles of its first piece, slot}, in launch order.
int attention_tc_handover_plan(long long units, int n_tiles, int sms, int* whole_units, int* n_handed, unsigned short* first, int max_handed) {
    if (units < 0 || n_tiles <= 0 || sms <= 0 || !whole_units || !n_handed || max_handed < 0 || (max_handed && !first)) return RFK_EINVAL;
    tcattn::WorkList w;
    plan_work(w, units, n_tiles, sms, false, false);
    plan_handover(w, units, n_tiles, sms);
    *whole_units = w.whole_units;
    *n_handed = w.heads;
    for (int i = 0; i < w.heads && i < max_handed; ++i) {
        first[3 * i] = w.pieces[i].unit; first[3 * i + 1] = w.pieces[i].nt; first[3 * i + 2] = w.pieces[i].slot;
    }
    return RFK_OK;
}

int attention_tc_wait_clock(const unsigned long long* readings, int n) {
    if (n <= 0 || !readings) return RFK_EINVAL;
    tcattn::WaitClock clock(readings[0]);
    for (int i = 1; i < n; ++i)
        if (clock.ended(readings[i])) return i;
    return 0;
}

int attention_tc_arrive(int* counter, int failed, int pieces) {
    if (!counter || pieces <= 0) return RFK_EINVAL;
    const handover::Arrival a = handover::arrive(*counter, failed != 0, pieces);
    *counter = a.last ? 0 : *counter + handover::piece(failed != 0);
    return a.merge;
}

int attention_tc_handover_step(int word, int event, int* next) {
    if (!next || word < 0 || word > handover::kTaken) return RFK_EINVAL;
    const handover::Step s = event == 0 ? handover::give(word, true) : event == 1 ? handover::give(word, false)
                             : event == 2 ? handover::look(word) : handover::settle(word);
    *next = s.next;
    return s.act;
}

namespace {
template <int HD, int BLOCKS, bool ORDERED, bool HAND, bool EIGHTS>
int launch_units(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, __half* O, int H, int Sq, int n_keys, int o_bshd,
                 float scale, cudaStream_t st, const float* row_ss, int ss_tiles, int norm_dim, float norm_eps, void* ws, int v_heads,
                 const tcattn::WorkList& work, int dev) {
    constexpr auto kernel = tcattn::attention_tc_kernel<HD, BLOCKS, ORDERED, HAND, EIGHTS>;
    constexpr int smem = tcattn::Cfg<HD, BLOCKS>::kSmemBytes;
    // per-device "kernel attributes set" marks; setting them twice from racing threads is harmless
    static std::atomic<bool> configured[64];
    if (!configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return (int)e;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return (int)e;
        configured[dev].store(true, std::memory_order_release);
    }
    launch_pdl(kernel, dim3((unsigned)(work.whole_units + work.n_pieces)), dim3(tcattn::kThreads), smem, st, mq, mk, mv, O, H, Sq, n_keys,
               o_bshd, scale * 1.4426950408889634f, row_ss, ss_tiles, norm_dim > 0 ? 1.0f / (float)norm_dim : 0.0f, norm_eps,
               static_cast<unsigned char*>(ws), v_heads, work);
    return launch_status();
}

template <int HD, bool ORDERED, bool EIGHTS>
int launch_hd(const __half* Q, const __half* K, const __half* V, __half* O, int B, int H, int Sq, int Sk,
              int n_keys, int o_bshd, float scale, cudaStream_t st, const float* row_ss, int ss_tiles,
              int norm_dim, float norm_eps, void* ws, size_t ws_bytes, AttnCut cut, int v_shared) {
    static std::atomic<int> sm_count[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return RFK_EUNSUPPORTED;
    int sms = sm_count[dev].load(std::memory_order_relaxed);
    if (sms == 0) {
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return (int)e;
        sm_count[dev].store(sms, std::memory_order_relaxed);
    }
    CUtensorMap mq, mk, mv;
    if (!make_map(&mq, Q, (long long)B * H, Sq, HD, tcattn::BM) || !make_map(&mk, K, (long long)B * H, Sk, HD, tcattn::BN) ||
        !make_map(&mv, V, v_shared ? (long long)H : (long long)B * H, Sk, HD, tcattn::BN))
        return RFK_EUNSUPPORTED;
    tcattn::WorkList work;
    work.q_blocks = ceil_div(Sq, tcattn::kUnitRows);
    const long long units = (long long)B * H * work.q_blocks;
    if (units > 0x7fffffffLL) return RFK_EUNSUPPORTED;
    const bool shared = ws && ws_bytes >= tcattn::kWsBytes && aligned16(ws) && g_attn_split.load(std::memory_order_relaxed);
    plan_work(work, units, ceil_div(n_keys, tcattn::BN), sms, shared && cut != AttnCut::kNone, cut == AttnCut::kLastRound);
    if (shared && work.n_pieces == 0) plan_handover(work, units, ceil_div(n_keys, tcattn::BN), sms);
    const int v_heads = v_shared ? H : B * H;
    if (one_block_per_cta(work.n_pieces, (long long)B * H * ceil_div(Sq, tcattn::BM), sms)) {
        work.q_blocks = ceil_div(Sq, tcattn::BM);
        work.whole_units = B * H * work.q_blocks;
        return launch_units<HD, 1, ORDERED, false, EIGHTS>(mq, mk, mv, O, H, Sq, n_keys, o_bshd, scale, st, row_ss, ss_tiles, norm_dim, norm_eps, ws, v_heads, work, dev);
    }
    const auto launch = work.heads ? launch_units<HD, 2, ORDERED, true, EIGHTS> : launch_units<HD, 2, ORDERED, false, EIGHTS>;
    return launch(mq, mk, mv, O, H, Sq, n_keys, o_bshd, scale, st, row_ss, ss_tiles, norm_dim, norm_eps, ws, v_heads, work, dev);
}
}  // namespace

// Launches the tcgen05 kernel; the caller has validated pointers, alignment and sizes (D 64 or 128). v_shared: V is
// [H, Sk, D], one set of values for every batch element (views of one scene). ws (may be NULL):
// attention_tc_workspace_bytes() bytes whose first 1024 are zero, for the key split.
int launch_attention_tc(const __half* Q, const __half* K, const __half* V, __half* O, int B, int H, int Sq, int Sk,
                        int n_keys, int D, int o_bshd, float scale, cudaStream_t st, const float* row_ss, int ss_tiles,
                        int norm_dim, float norm_eps, void* ws, size_t ws_bytes, AttnCut cut, int v_shared, int ss_group) {
    if (ss_group == 8 && (ss_tiles % 8 || !aligned16(row_ss) || (D != 64 && cut == AttnCut::kNone))) return RFK_EUNSUPPORTED;
    const auto launch = ss_group == 8 ? (D == 64 ? launch_hd<64, false, true> : launch_hd<128, false, true>)
                        : D == 64     ? launch_hd<64, false, false>
                        : cut == AttnCut::kNone ? launch_hd<128, true, false> : launch_hd<128, false, false>;
    return launch(Q, K, V, O, B, H, Sq, Sk, n_keys, o_bshd, scale, st, row_ss, ss_tiles, norm_dim, norm_eps, ws, ws_bytes, cut, v_shared);
}

}  // namespace rfk

using namespace rfk;

extern "C" int rfk_flash_attention_set_path(int path) {
    if (path < 0 || path > 2) return RFK_EINVAL;
    g_attn_path.store(path, std::memory_order_relaxed);
    return RFK_OK;
}

extern "C" int rfk_flash_attention_error(int* code, int clear) {
    if (!code) return RFK_EINVAL;
    cudaError_t e = cudaMemcpyFromSymbol(code, g_attn_tc_error, sizeof(int));
    if (e != cudaSuccess) return (int)e;
    if (clear) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_attn_tc_error, &zero, sizeof(int));
        if (e != cudaSuccess) return (int)e;
    }
    return RFK_OK;
}
