// Dense fp32 convolution on the tensor cores, without giving up a bit of fp32: an implicit GEMM of operands that are split into three
// bf16 parts each.
//
//   D[m, n] = sum_k A[m, k] * B[k, n]     m = output pixel (all images back to back), n = output channel,
//                                          k = (tap, input channel), taps of 32-channel chunks
//
// Both are multiplied by 2^16 first, so that bf16 holds the ends of the least fp32 value, too; then A = a0 + a1 + a2 and B = b0 + b1 + b2 exactly (8 bits
// of mantissa each, rounded to nearest, so 24 and the signs).  a1 is 2^-8 of A at most and a2 2^-17, so of the nine products all are multiplied but a2 b2, 2^-34 of
// a product.  (Without a1 b2 and a2 b1, up to 2^-24 of it, a sum of one product is 7.7e-8 off instead of 5.9e-8, its one rounding: 256 -> 256 channels on 16 maps
// of 28 x 28 98.0 us, with them 103.8.)
// The sums are multiplied by 2^-32 at the end.
// Products of bf16 values are exact in fp32.  The tensor core's own additions do not round to nearest, so its sums are kept
// short: an accumulator holds 64 values of k, and the products a0 b0 have one of their own, apart from the seven small ones (whose
// roundings are 2^-8 of theirs).  After every 64 k both are read from tensor memory and added to the sums in registers, which are
// ordinary fp32.
//
// Block = 26 warps on a tile of 128 pixels x BN channels, in steps of 64 k:
//   warp 24      copies, three or four steps ahead: two im2col boxes of 128 pixels x 32 channels and two of 32 x BN weights, fp32
//   warps 8-15   split them: a thread has one box of a pixel, and leaves its three rows of bf16 in TENSOR memory, from where the tensor core
//                takes operand A (shared memory then moves operand B only: eight multiplications per 16 k read 8 x 2 KB there, not 8 x 6 KB)
//   warps 16-23  split the weights, into shared memory
//   warp 25      multiplies: 4 x 8 instructions of 128 x BN x 16 a step
//   warps 0-7    add up, half of the columns each, and finish the tile: bias, residual, activation
// Tensor memory: two steps of operand A (192 columns) and two pairs of accumulators (4 BN).  A layer with few tiles splits its k range over
// the blocks of a cluster, whose sums meet through distributed shared memory, in rank order: results do not depend on timing.
//
// Bound by the tensor pipe and the instructions of all warps together (59 % and 1120 issue slots a scheduler and step, 64 %, in a large layer) and, where a
// launch has few steps, by the latency of a step's chain: 0.84 us at 64 columns, 0.74 at 32.  Measured against the kernel on the fp32 units, us a launch in a
// row of equal ones: 64 -> 64 3x3 on 2 maps of 56 x 56 23.3 -> 10.6, 128 -> 128 on 2 of 28 x 28 22.1 -> 11.0, 512 -> 512 on 2 of 7 x 7 29.5 -> 14.6,
// 256 -> 256 on 16 of 28 x 28 408 -> 103 (143 TFLOP/s of fp32 multiply-adds); ResNet-18 x 2 images 429 -> 213.  Error against 64 bits, relative, fp32 units / here:
// 1.62e-7 / 8.3e-8, 1.14e-7 / 8.1e-8, 1.86e-7 / 9.8e-8, 3.03e-7 / 1.24e-7 (the layers above), 64 -> 64 1x1 7.1e-8 / 5.9e-8.
//
// Infinities, NaN and operands of 2^112 and more make 0 x inf of the parts, and sums of 2^96 and more overflow: a block that finds one of its sums not finite
// makes them all again in a second pass, as plain fp32 multiply-adds of the same copies (32 TFLOP/s; one thread a poisoned output, as it was, took
// 10.9 ms for 256 -> 256 on 16 of 28 x 28 where every pixel is NaN, 0.49 ms for 64 -> 64 on 2 of 56 x 56; this 0.57 ms and 34 us, the fp32 units 0.41 and 23).
// What is small is exact (64 -> 64 3x3, relative error against 64 bits here / on the fp32 units: inputs of 2^-122 and weights of 2^30 8.5e-8 / 1.1e-7, 2^-140 and
// 2^100 7.0e-8 / 1.1e-7, results of 2^-134 3.3e-6 / 3.7e-5; without the scaling 1.4e-4, 1.0 and 5.8e-5).
//
// This is the fp32 member of the kernel family the reference's TVM adapters launch
// (jobs/tvm_<model>/tvm_<model>.cpp:24-47; generated fp32 kernels there).
#include <cuda.h>
#include <llis/job/finished_block_notifier.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "conv_f32.h"
#include "launch_slot.cuh"
#include "ops.h"
#include "pb_common.h"
#include "umma.cuh"

using llis::job::FinishedBlockNotifier;

namespace pb {

__device__ uint32_t g_f32_err_flag;      // raised when a bounded wait runs out

namespace {

constexpr int kTileRows = 128, kChunk = 32;             // pixels of a tile, channels of a copy box
constexpr int kMaxRing = 4;
constexpr uint32_t kBox = kTileRows * kChunk * 4;       // 16 KB
constexpr int kWarpA = 8, kWarpB = 16, kWarpCopy = 24, kWarpMma = 25;
constexpr int kThreadsF = 26 * 32;                      // 832
constexpr uint32_t kTmemCols = 512;
constexpr uint64_t kUp = 0x4780000047800000ull, kDown = 0x2f8000002f800000ull;      // pairs of 2^16 and 2^-32

struct SplitArgs {
    OpArgs op;
    int M, PQ, Kp;       // rows of the GEMM, pixels per image, channels of a row of packed weights
    int cpt, chunks;     // chunks of 32 channels per tap, and of the whole reduction
    int splits;          // cluster size
    int a_tiled;         // pointwise: operand A is a plain matrix
};

// Shared memory: the ring of raw operands (two boxes of pixels, two of weights a step), the split weights of two steps, and where the sums
// of a tile meet.  Tensor memory columns: accumulators [buffer][large, small][BN], then operand A [step][part][32].
template <int BN>
struct Layout {
    static constexpr uint32_t ring = BN == 64 ? 3 : 4;
    static constexpr uint32_t raw_w = 2 * kBox, w_box = kChunk * BN * 4, stage = raw_w + 2 * w_box;
    static constexpr uint32_t part = BN * 128, parts = ring * stage, parts_step = 3 * part;
    static constexpr uint32_t meet = parts + 2 * parts_step, bytes = meet + kTileRows * BN * 4;
    static constexpr uint32_t acc = 0, a = 4 * BN;
};

__device__ __forceinline__ void mma_ta(uint32_t d, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tcgen05_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t x, uint64_t y) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t x, uint64_t y, uint64_t z) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
__device__ __forceinline__ void tcgen05_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// lo and hi less the bf16 values of the pair, exactly.  (The mixed multiply-add reads a half of a register: two instructions where widening the
// halves and subtracting takes three.)
__device__ __forceinline__ void less_bf16(uint32_t pair, float& lo, float& hi) {
    asm("{\n\t.reg .b16 l, h, m;\n\tmov.b32 {l, h}, %2;\n\tmov.b16 m, 0xbf80;\n\t"
        "fma.rn.f32.bf16 %0, l, m, %0;\n\tfma.rn.f32.bf16 %1, h, m, %1;\n\t}"
        : "+f"(lo), "+f"(hi)
        : "r"(pair));
}
// Two values, times 2^16, to three pairs of bf16 that add up to them (the first in the low halves).
__device__ __forceinline__ void split2(uint32_t x0, uint32_t x1, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    float lo, hi;
    unpack_f32x2(mul_f32x2(pack_f32x2(x0, x1), kUp), lo, hi);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p0) : "f"(hi), "f"(lo));
    less_bf16(p0, lo, hi);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p1) : "f"(hi), "f"(lo));
    less_bf16(p1, lo, hi);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p2) : "f"(hi), "f"(lo));
}

// Where a summing thread's row of sums goes.  Rank z finishes rows [z, z + 1) x 128 / splits of the tile: every rank sends it its sums (st.async: the sums
// go from registers into the owner's shared memory and count on its barrier), laid out as [rank][row][channel], 16-byte chunks in an order that
// keeps both the writers (a row each) and the readers (a chunk each) free of bank conflicts.
template <int BN>
struct Meeting {
    uint32_t at, to, bar, mix;
    bool mine;
    __device__ __forceinline__ Meeting(const SplitArgs& f, uint32_t smem, int row, int rank, uint64_t* s_sums) {
        const int ranks_log2 = 31 - __clz(f.splits), share = kTileRows >> ranks_log2, owner = row >> (7 - ranks_log2), rl = row & (share - 1);
        at = to = smem + Layout<BN>::meet + (uint32_t)((rank * share + rl) * (BN * 4));
        mix = (uint32_t)rl & 7u;
        bar = 0;
        mine = owner == rank;
        if (f.splits > 1) {
            to = cluster_addr(at, (uint32_t)owner);
            bar = cluster_addr(smem_u32(s_sums), (uint32_t)owner);
        }
    }
    __device__ __forceinline__ void put(int col, const float4& v) const {      // columns col .. col + 3
        const uint32_t off = (((uint32_t)col >> 2) ^ mix) << 4;
        if (mine) st_shared_v4(at + off, __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
        else st_async_v4(to + off, __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w), bar);
    }
};

// Is `p` true anywhere in the summing warps?
__device__ __forceinline__ bool sums_any(bool p) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(p ? 1u : 0u) : "memory");
    return r != 0;
}
// The summing warps have decided whether there is a second pass (they go on at once); the others wait for that.
__device__ __forceinline__ void block_arrive() { asm volatile("barrier.cta.arrive 2, 832;" ::: "memory"); }
__device__ __forceinline__ void block_await() { asm volatile("barrier.cta.sync 2, 832;" ::: "memory"); }
// Everybody: the second pass is complete.
__device__ __forceinline__ void block_meet() { asm volatile("barrier.cta.sync 3, 832;" ::: "memory"); }

// ---- a block's share of the reduction once more, as plain fp32 multiply-adds ----------------------------------------
// The raw operands come again, through the ring's first two stages; its third takes the sums.  (Called with what is constant only: arguments that live
// through the loops of the first pass for this cost it 5 %.)
template <int BN>
struct Share {          // the tile and the steps of this block
    int m0, n0, kb0, n_kb;
    uint32_t smem;
    __device__ __forceinline__ Share(const SplitArgs& f, const uint8_t* smem_raw)
        : m0((int)blockIdx.x * kTileRows), n0((int)blockIdx.y * BN), smem((smem_u32(smem_raw) + 1023u) & ~1023u) {
        const int steps = (f.chunks + 1) / 2, ranks_log2 = 31 - __clz(f.splits), rank = (int)blockIdx.z;
        kb0 = (steps * rank) >> ranks_log2;
        n_kb = ((steps * (rank + 1)) >> ranks_log2) - kb0;
    }
};
// How often stage st was used by the first pass:
template <int BN>
__device__ __forceinline__ uint32_t ring_uses(uint32_t st, int n_kb) { return ((uint32_t)n_kb + Layout<BN>::ring - 1u - st) / Layout<BN>::ring; }

template <int BN, bool kRows>
__device__ __noinline__ void copy_again(const CUtensorMap* tmap_x, const CUtensorMap* tmap_w, const SplitArgs& f, uint8_t* smem_raw, uint64_t* s_full, uint64_t* s_empty,
                                        volatile uint32_t* s_abort) {
    using L = Layout<BN>;
    const OpArgs& a = f.op;
    const Share<BN> b(f, smem_raw);
    const int m0 = b.m0, n0 = b.n0, kb0 = b.kb0, n_kb = b.n_kb;
    const uint32_t smem = b.smem;
    const int img = m0 / f.PQ, pix = m0 - img * f.PQ, p = pix / a.Q, w_org = (pix - p * a.Q) * a.stride_w - a.pad_w, h_org = p * a.stride_h - a.pad_h;
    for (int kb = 0; kb < n_kb; ++kb) {
        const uint32_t st = (uint32_t)kb & 1u, bar = smem_u32(&s_full[st]), to = smem + st * L::stage;
        if (kb >= 2 && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[st]), (ring_uses<BN>(st, n_kb) + (uint32_t)(kb >> 1) - 1u) & 1u, s_abort, &g_f32_err_flag, 0x2au))) break;
        const int chunk = 2 * (kb0 + kb), have = min(2, f.chunks - chunk);
        if (elect_one()) {
            mbar_arrive_expect_tx(bar, (uint32_t)have * ((kRows ? 0u : kBox) + L::w_box));
            for (int h = 0; h < have; ++h) {
                const int tap = (chunk + h) / f.cpt, c = (chunk + h - tap * f.cpt) * kChunk, r = tap / a.S;
                tma_load_3d(to + L::raw_w + (uint32_t)h * L::w_box, tmap_w, n0, c, tap, bar);
                if (kRows) continue;
                if (f.a_tiled) tma_load_2d(to + (uint32_t)h * kBox, tmap_x, c, m0, bar);
                else tma_load_im2col_4d(to + (uint32_t)h * kBox, tmap_x, c, w_org, h_org, img, (uint16_t)((tap - r * a.S) * a.dil_w), (uint16_t)(r * a.dil_h), bar);
            }
        }
        __syncwarp();
    }
}

// Warps 8-23: two groups of 256 threads, a box of a step each; a thread has rows t / 8 + 32 i and columns 4 (t % 8) + 32 j, + 0 .. 3.  The sums of a box go
// to shared memory, [group][i][j][t][4]: no chain is longer than 32.
template <int BN, bool kRows>
__device__ __noinline__ void sum_again(const SplitArgs& f, uint8_t* smem_raw, uint64_t* s_full, uint64_t* s_empty, volatile uint32_t* s_abort) {
    using L = Layout<BN>;
    constexpr int kWide = BN / 32;                 // column quads of a thread
    const OpArgs& a = f.op;
    const Share<BN> b(f, smem_raw);
    const int m0 = b.m0, kb0 = b.kb0, n_kb = b.n_kb;
    const uint32_t smem = b.smem;
    const int t = (int)threadIdx.x & 255, h = ((int)threadIdx.x >> 8) - 1;
    const uint32_t row = (uint32_t)t >> 3, swz = row & 7u, box = smem + (uint32_t)h * kBox, w_at = smem + L::raw_w + (uint32_t)h * L::w_box + ((uint32_t)t & 7u) * 16u;
    const uint32_t sums = smem + 2 * L::stage + ((uint32_t)(h * 4 * kWide) * 256u + (uint32_t)t) * 16u;
    // kRows: this thread brings four pixels of a row's window
    const int m = m0 + (t & 127), img = m / f.PQ, pix = m - img * f.PQ, p = pix / a.Q, ih0 = p * a.stride_h - a.pad_h, px0 = (t >> 7) * 4;
    const int iw0 = (pix - p * a.Q) * a.stride_w - a.pad_w + px0;
#pragma unroll 1
    for (int kb = 0; kb < n_kb; ++kb) {
        const uint32_t st = (uint32_t)kb & 1u;
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[st]), (ring_uses<BN>(st, n_kb) + (uint32_t)(kb >> 1)) & 1u, s_abort, &g_f32_err_flag, 0x2bu)) && !kRows) break;      // (kRows: the group meets below)
        const bool have = 2 * (kb0 + kb) + h < f.chunks;
        if constexpr (kRows) {
            const int ih = ih0 + (2 * (kb0 + kb) + h) * a.dil_h;
            const uint4* const from = static_cast<const uint4*>(a.x) + ((ptrdiff_t)img * a.H + ih) * a.W + iw0;
            for (int c = 0; c < 4; ++c) {
                uint4 v = make_uint4(0, 0, 0, 0);
                if (have && m < f.M && px0 + c < a.S && ih >= 0 && ih < a.H && iw0 + c >= 0 && iw0 + c < a.W) v = from[c];
                st_shared_v4(box + st * L::stage + (uint32_t)(t & 127) * 128u + ((uint32_t)((px0 + c) ^ (t & 7)) << 4), v.x, a.C > 1 ? v.y : 0u, a.C > 2 ? v.z : 0u, a.C > 3 ? v.w : 0u);
            }
            asm volatile("bar.sync %0, 256;" ::"r"(4 + h) : "memory");
        }
        float acc[4][4 * kWide];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4 * kWide; ++j) acc[i][j] = 0.f;
        if (have) {
#pragma unroll 1
            for (uint32_t c = 0; c < 8; ++c) {
                float x[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 v = ld_shared_v4(box + st * L::stage + (row + 32u * (uint32_t)i) * 128u + ((c ^ swz) << 4));
                    x[i][0] = __uint_as_float(v.x); x[i][1] = __uint_as_float(v.y); x[i][2] = __uint_as_float(v.z); x[i][3] = __uint_as_float(v.w);
                }
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) {
#pragma unroll
                    for (int j = 0; j < kWide; ++j) {
                        const uint4 w = ld_shared_v4(w_at + st * L::stage + (c * 4u + q) * (uint32_t)(BN * 4) + (uint32_t)j * 128u);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            acc[i][4 * j] = fmaf(x[i][q], __uint_as_float(w.x), acc[i][4 * j]);
                            acc[i][4 * j + 1] = fmaf(x[i][q], __uint_as_float(w.y), acc[i][4 * j + 1]);
                            acc[i][4 * j + 2] = fmaf(x[i][q], __uint_as_float(w.z), acc[i][4 * j + 2]);
                            acc[i][4 * j + 3] = fmaf(x[i][q], __uint_as_float(w.w), acc[i][4 * j + 3]);
                        }
                    }
                }
            }
        }
        __syncwarp();
        if (elect_one()) mbar_arrive(smem_u32(&s_empty[st]));
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < kWide; ++j) {
                const uint32_t to = sums + (uint32_t)(i * kWide + j) * 4096u;
                float4 v = make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
                if (kb > 0) {
                    const uint4 o = ld_shared_v4(to);
                    v = make_float4(__uint_as_float(o.x) + v.x, __uint_as_float(o.y) + v.y, __uint_as_float(o.z) + v.z, __uint_as_float(o.w) + v.w);
                }
                st_shared_v4(to, __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
            }
    }
}

// Summing warps: the second pass's sums to where they meet.  (A call of its own: with the sums read back into the registers of the first pass every
// launch pays 5 % for the copies.)
template <int BN>
__device__ __noinline__ void send_again(const SplitArgs& f, uint8_t* smem_raw, uint64_t* s_sums) {
    using L = Layout<BN>;
    constexpr int kCols = BN / 2;
    constexpr uint32_t kGroup = (uint32_t)kTileRows * BN * 4;
    block_meet();
    const int row = (int)threadIdx.x & 127, col0 = ((int)threadIdx.x >> 7) * kCols;
    const Share<BN> b(f, smem_raw);
    const Meeting<BN> to(f, b.smem, row, (int)blockIdx.z, s_sums);
    const uint32_t from = b.smem + 2 * L::stage + (uint32_t)(row >> 5) * (uint32_t)(BN / 32) * 4096u + (uint32_t)(row & 31) * 128u;
    for (int c = col0; c < col0 + kCols; c += 4) {
        const uint32_t at = from + (uint32_t)(c >> 5) * 4096u + (uint32_t)(c & 31) * 4u;
        const uint4 v = ld_shared_v4(at), w = ld_shared_v4(at + kGroup);
        to.put(c, make_float4(__uint_as_float(v.x) + __uint_as_float(w.x), __uint_as_float(v.y) + __uint_as_float(w.y), __uint_as_float(v.z) + __uint_as_float(w.z),
                              __uint_as_float(v.w) + __uint_as_float(w.w)));
    }
}

// Four outputs of row m, from channel k on: bias, residual, activation, whatever the alignment.
__device__ __forceinline__ void finish4(const OpArgs& a, int m, int k, float4 v, const float4& b, const float4& s, bool vec, bool vec_r) {
    v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
    if (a.residual) {
        const float* res = static_cast<const float*>(a.residual) + (size_t)m * a.res_Cs + k;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vec_r && k + 4 <= a.K) q = *reinterpret_cast<const float4*>(res);
        else {
            q.x = res[0];
            if (k + 1 < a.K) q.y = res[1];
            if (k + 2 < a.K) q.z = res[2];
            if (k + 3 < a.K) q.w = res[3];
        }
        v = make_float4(v.x + q.x, v.y + q.y, v.z + q.z, v.w + q.w);
    }
    if (a.act == 3) {           // PReLU
        v = make_float4(v.x > 0.f ? v.x : v.x * s.x, v.y > 0.f ? v.y : v.y * s.y, v.z > 0.f ? v.z : v.z * s.z, v.w > 0.f ? v.w : v.w * s.w);
    } else if (a.act == 1 || a.act == 2) {
        v = make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
        if (a.act == 2) v = make_float4(fminf(v.x, 6.f), fminf(v.y, 6.f), fminf(v.z, 6.f), fminf(v.w, 6.f));
    }
    float* y = static_cast<float*>(a.y) + (size_t)m * a.Ks + a.out_c_off + k;
    if (vec && k + 4 <= a.K) {
        *reinterpret_cast<float4*>(y) = v;
    } else {
        y[0] = v.x;
        if (k + 1 < a.K) y[1] = v.y;
        if (k + 2 < a.K) y[2] = v.z;
        if (k + 3 < a.K) y[3] = v.w;
    }
}

// kRows: a stem, whose pixels have four channels (up to four of them real).  There a chunk is a row of the filter - up to eight pixels side by
// side, 32 values - and the splitting warps read the pixels themselves: a tap of its own would fill an eighth of a chunk.  (7 x 7, stride 2, 64
// channels on 2 maps of 224 x 224: 32.3 us on the fp32 units, 17.9 here.)
template <int BN, bool kRows>
__global__ void __launch_bounds__(kThreadsF, 1)
conv_f32_split_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ SplitArgs f, uint32_t job_id, FinishedBlockNotifier* nf) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxRing], s_empty[kMaxRing];      // raw operands
    __shared__ __align__(8) uint64_t s_ready[2], s_done[2], s_free[2];   // operands split; multiplied; accumulators read
    __shared__ __align__(8) uint64_t s_sums[1];                          // the other ranks' sums have arrived
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile uint32_t s_abort, s_again;
    __shared__ __align__(16) float s_bias[BN], s_slope[BN];
    using L = Layout<BN>;

    resolve_slot(job_id, nf);
    if (nf) nf->start(job_id);
    const OpArgs& a = f.op;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = (int)uniform((uint32_t)tid >> 5);
    const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int m0 = (int)blockIdx.x * kTileRows, n0 = (int)blockIdx.y * BN, rank = (int)blockIdx.z;
    const int steps = (f.chunks + 1) / 2;                          // of 64 k
    const int ranks_log2 = 31 - __clz(f.splits);                   // (a power of two)
    const int kb0 = (steps * rank) >> ranks_log2, n_kb = ((steps * (rank + 1)) >> ranks_log2) - kb0;
    constexpr uint32_t ring = L::ring;
    uint32_t* const err = &g_f32_err_flag;

    if (warp == kWarpCopy) {            // the maps are on their way while the barriers are set up, a lane per barrier
        if (elect_one()) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            if (!kRows) asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
        }
        if (lane < (int)ring) {
            mbar_init(smem_u32(&s_full[lane]), 1);
            mbar_init(smem_u32(&s_empty[lane]), 16);
        } else if (lane >= 8 && lane < 10) {
            mbar_init(smem_u32(&s_ready[lane - 8]), 16);
            mbar_init(smem_u32(&s_done[lane - 8]), 1);
            mbar_init(smem_u32(&s_free[lane - 8]), 8);
        } else if (lane == 16) {
            mbar_init(smem_u32(s_sums), 1);
            if (f.splits > 1) mbar_arrive_expect_tx(smem_u32(s_sums), (uint32_t)((f.splits - 1) * (kTileRows >> ranks_log2) * BN * 4));
            s_abort = 0;
            s_again = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
        __syncwarp();
    }
    if (warp == kWarpMma) {
        tcgen05_alloc(smem_u32(&s_tmem_base), kTmemCols);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    if (f.splits > 1) cluster_arrive_relaxed();        // (the barriers' fence has released them; a release here takes 1100 clocks)
    const uint32_t tmem = uniform(s_tmem_base);

    if (warp >= kWarpA) griddep_launch();       // the next launch's blocks may have the SMs that this one leaves idle
    if (warp < kWarpA) {
        // ===== sums =====
        griddep_wait();
        griddep_launch();
        if (f.splits > 1) cluster_wait();              // every block of the cluster is running and has set its barriers up
        constexpr int kCols = BN / 2;                  // of this thread, of one row
        const int row = tid & 127, col0 = (tid >> 7) * kCols;
        if (tid < BN) {
            const int k = n0 + tid;
            s_bias[tid] = a.bias && k < a.K ? __ldg(a.bias + k) : 0.f;
            s_slope[tid] = a.act == 3 && k < a.K ? __ldg(a.bias + a.K + k) : 0.f;      // the slopes follow the biases
        }
        uint64_t acc[kCols / 2];
#pragma unroll
        for (int j = 0; j < kCols / 2; ++j) acc[j] = 0;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16) + L::acc + (uint32_t)col0;
        bool ok = true;
        for (int kb = 0; kb < n_kb; ++kb) {
            const int t = kb & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_done[t]), (uint32_t)(kb >> 1) & 1u, &s_abort, err, 0x21u));
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t d = lanes + (uint32_t)(t * 2 * BN);
#pragma unroll
            for (int c = 0; c < kCols; c += 16) {
                uint32_t big[16], small[16];
                tcgen05_ld16(d + (uint32_t)c, big);
                tcgen05_ld16(d + (uint32_t)(BN + c), small);
                tcgen05_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; j += 2)
                    acc[(c + j) / 2] = add_f32x2(acc[(c + j) / 2], add_f32x2(pack_f32x2(big[j], big[j + 1]), pack_f32x2(small[j], small[j + 1])));
            }
            tcgen05_fence_before();
            __syncwarp();
            if (elect_one()) mbar_arrive(smem_u32(&s_free[t]));
            __syncwarp();
        }
        // Sums that are not finite - operands of 2^112 and more, infinities and NaN among them, or products that overflow - are made again in plain fp32, those
        // of the block's whole share of the reduction.
        uint64_t finite[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < kCols / 2; ++j) {
            acc[j] = mul_f32x2(acc[j], kDown);
            finite[j & 3] = fma_f32x2(acc[j], 0ull, finite[j & 3]);
        }
        float f0, f1;
        unpack_f32x2(add_f32x2(add_f32x2(finite[0], finite[1]), add_f32x2(finite[2], finite[3])), f0, f1);
        const bool again = sums_any(!(f0 == f1) && !s_abort);      // (zeros or NaN)
        if (again && tid == 0) s_again = 1;
        __syncwarp();
        block_arrive();
        const uint32_t meet = smem + L::meet;
        const int share = kTileRows >> ranks_log2;
        if (__builtin_expect(again, 0)) {
            send_again<BN>(f, smem_raw, s_sums);
        } else {
            const Meeting<BN> to(f, smem, row, rank, s_sums);
#pragma unroll
            for (int c = 0; c < kCols; c += 4) {
                float4 v;
                unpack_f32x2(acc[c / 2], v.x, v.y);
                unpack_f32x2(acc[c / 2 + 1], v.z, v.w);
                to.put(col0 + c, v);
            }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (f.splits > 1) {       // (also when this block gives up: it stays until the others have written to it)
            bool here = false;
            for (uint32_t i = 0; i < kWaitLimit && !here; ++i) here = mbar_try_wait(smem_u32(s_sums), 0u);
            if (!here) atomicExch(err, 0x28u);
            ok = __all_sync(0xffffffffu, here) && ok;
        }
        ok = ok && !s_abort;           // (the second pass may have given up)
        if (ok) {
            const bool vec = ((a.Ks | a.out_c_off) & 3) == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
            const bool vec_r = (a.res_Cs & 3) == 0 && (reinterpret_cast<uintptr_t>(a.residual) & 15) == 0;
            // this rank's share of the tile's rows; a thread has four columns of every kStepR-th
            constexpr int kStepR = 256 / (BN / 4);
            const int r1 = min(share, f.M - m0 - rank * share), c = tid % (BN / 4) * 4, k = n0 + c, m_share = m0 + rank * share;
            int r = tid / (BN / 4);                             // in the share
            auto sum4 = [&](int row) {
                const uint32_t at = meet + (uint32_t)row * (BN * 4) + ((((uint32_t)c >> 2) ^ ((uint32_t)row & 7u)) << 4);
                uint4 q = ld_shared_v4(at);
                float4 v = make_float4(__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z), __uint_as_float(q.w));
#pragma unroll 1
                for (int z = 1; z < f.splits; ++z) {             // in rank order
                    q = ld_shared_v4(at + (uint32_t)(z * share) * (BN * 4));
                    v = make_float4(v.x + __uint_as_float(q.x), v.y + __uint_as_float(q.y), v.z + __uint_as_float(q.z), v.w + __uint_as_float(q.w));
                }
                return v;
            };
            const float4 bias = *reinterpret_cast<const float4*>(s_bias + c), slope = *reinterpret_cast<const float4*>(s_slope + c);
            auto any_row = [&](int row) { finish4(a, m_share + row, k, sum4(row), bias, slope, vec, vec_r); };      // whatever the alignment and the activation
            // Branches cost a lone warp more than the arithmetic: rows four at a time, their loads together, nothing left to decide.
            auto rows4 = [&](auto with_residual, auto with_clamp) {
                constexpr bool residual = decltype(with_residual)::value, clamp = decltype(with_clamp)::value;
                const float top = a.act == 2 ? 6.f : INFINITY;
                const float* res = static_cast<const float*>(a.residual) + (size_t)(m_share + r) * a.res_Cs + k;
                float* y = static_cast<float*>(a.y) + (size_t)(m_share + r) * a.Ks + a.out_c_off + k;
#pragma unroll 1
                for (; r < r1; r += 4 * kStepR) {
                    float4 v[4], q[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (residual && r + u * kStepR < r1) q[u] = *reinterpret_cast<const float4*>(res + (size_t)(u * kStepR) * a.res_Cs);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (r + u * kStepR < r1) v[u] = sum4(r + u * kStepR);
                        v[u] = make_float4(v[u].x + bias.x, v[u].y + bias.y, v[u].z + bias.z, v[u].w + bias.w);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float4 x = v[u];
                        if (residual) x = make_float4(x.x + q[u].x, x.y + q[u].y, x.z + q[u].z, x.w + q[u].w);
                        if (clamp) x = make_float4(fminf(fmaxf(x.x, 0.f), top), fminf(fmaxf(x.y, 0.f), top), fminf(fmaxf(x.z, 0.f), top), fminf(fmaxf(x.w, 0.f), top));
                        if (r + u * kStepR < r1) *reinterpret_cast<float4*>(y + (size_t)(u * kStepR) * a.Ks) = x;
                    }
                    res += (size_t)(4 * kStepR) * a.res_Cs;
                    y += (size_t)(4 * kStepR) * a.Ks;
                }
            };
            const bool has_res = a.residual != nullptr;
            if (k >= a.K) {
            } else if (!vec || (has_res && !vec_r) || k + 4 > a.K || a.act == 3) {
#pragma unroll 1
                for (; r < r1; r += kStepR) any_row(r);
            } else if (a.act == 1 || a.act == 2) {
                if (has_res) rows4(std::true_type{}, std::true_type{});
                else rows4(std::false_type{}, std::true_type{});
            } else {
                if (has_res) rows4(std::true_type{}, std::false_type{});
                else rows4(std::false_type{}, std::false_type{});
            }
        }
    } else if (warp < kWarpB) {
        // ===== pixels to three parts, in tensor memory =====
        const uint32_t row = (uint32_t)tid & 127u, swz = row & 7u;
        const int h = (warp >> 2) & 1;                             // this thread's box
        const uint32_t at0 = tmem + ((uint32_t)((warp & 3) * 32) << 16) + L::a + (uint32_t)(h * 16);
        uint32_t st = 0, parity = 0;
        // kRows: where this thread's filter window begins
        int ih0 = 0, iw0 = 0;
        const float4* image = nullptr;
        if constexpr (kRows) {
            const int m = m0 + (int)row, img = m / f.PQ, rem = m - img * f.PQ, p = rem / a.Q, q = rem - p * a.Q;
            ih0 = m < f.M ? p * a.stride_h - a.pad_h : -(1 << 28);      // fails every bounds check
            iw0 = q * a.stride_w - a.pad_w;
            image = static_cast<const float4*>(a.x) + (size_t)(m < f.M ? img : 0) * a.H * a.W;
            griddep_wait();                        // the pixels are the previous launch's
        }
        for (int kb = 0; kb < n_kb; ++kb) {
            const int t = kb & 1;
            const bool have = 2 * (kb0 + kb) + h < f.chunks;       // an odd number of chunks ends with half a step
            uint4 v[kRows ? 8 : 4];
            const uint32_t from = smem + st * L::stage + (uint32_t)h * kBox + row * 128u;
            if constexpr (kRows) {
                const int ih = ih0 + (2 * (kb0 + kb) + h) * a.dil_h;
                const bool row_ok = have && ih >= 0 && ih < a.H;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const int iw = iw0 + c;
                    v[c] = make_uint4(0, 0, 0, 0);
                    if (row_ok && c < a.S && iw >= 0 && iw < a.W) v[c] = *reinterpret_cast<const uint4*>(image + (size_t)ih * a.W + iw);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    if (a.C < 4) v[c].w = 0;
                    if (a.C < 3) v[c].z = 0;
                    if (a.C < 2) v[c].y = 0;
                }
            } else {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[st]), parity, &s_abort, err, 0x22u))) break;
            }
            bool ok = true;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if constexpr (!kRows) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) v[c] = ld_shared_v4(from + (((uint32_t)(q * 4 + c) ^ swz) << 4));      // (without a second box: not used)
                }
                uint32_t p[3][8];
                if (have) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint4& x = v[kRows ? q * 4 + c : c];
                        split2(x.x, x.y, p[0][2 * c], p[1][2 * c], p[2][2 * c]);
                        split2(x.z, x.w, p[0][2 * c + 1], p[1][2 * c + 1], p[2][2 * c + 1]);
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 8; ++c) p[0][c] = p[1][c] = p[2][c] = 0u;
                }
                if (q == 0 && kb >= 2) {
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_done[t]), (uint32_t)((kb >> 1) - 1) & 1u, &s_abort, err, 0x23u));
                    if (!ok) break;
                    tcgen05_fence_after();
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) tcgen05_st8(at0 + (uint32_t)(t * 96 + i * 32 + q * 8), p[i]);
            }
            if (!ok) break;
            tcgen05_wait_st();
            tcgen05_fence_before();
            __syncwarp();
            if (elect_one()) {
                mbar_arrive(smem_u32(&s_ready[t]));
                mbar_arrive(smem_u32(&s_empty[st]));
            }
            __syncwarp();
            if (++st == ring) { st = 0; parity ^= 1u; }
        }
        block_await();
        if (s_again) {
            sum_again<BN, kRows>(f, smem_raw, s_full, s_empty, &s_abort);
            block_meet();
        }
    } else if (warp < kWarpCopy) {
        // ===== weights to three parts, in shared memory: eight k of one channel at a time, lanes along the channels =====
        const int bw = warp - kWarpB, n = lane + (BN == 64 ? 32 * (bw & 1) : 0), kg0 = BN == 64 ? bw >> 1 : bw;
        constexpr int kTasks = BN == 64 ? 2 : 1;
        uint32_t st = 0, parity = 0;
        for (int kb = 0; kb < n_kb; ++kb) {
            const int t = kb & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[st]), parity, &s_abort, err, 0x29u))) break;
            uint32_t p[kTasks][3][4];
            uint32_t v[kTasks][8];
#pragma unroll
            for (int j = 0; j < kTasks; ++j) {
                const uint32_t from = smem + st * L::stage + L::raw_w + (uint32_t)((kg0 + 4 * j) * 8 * BN + n) * 4u;
#pragma unroll
                for (int i = 0; i < 8; ++i) asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v[j][i]) : "r"(from + (uint32_t)(i * BN) * 4u) : "memory");
            }
#pragma unroll
            for (int j = 0; j < kTasks; ++j) {
                if (2 * (kb0 + kb) + ((kg0 + 4 * j) >> 2) < f.chunks) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) split2(v[j][2 * i], v[j][2 * i + 1], p[j][0][i], p[j][1][i], p[j][2][i]);
                } else {      // (no second box)
#pragma unroll
                    for (int i = 0; i < 4; ++i) p[j][0][i] = p[j][1][i] = p[j][2][i] = 0u;
                }
            }
            if (kb >= 2 && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_done[t]), (uint32_t)((kb >> 1) - 1) & 1u, &s_abort, err, 0x24u))) break;
            const uint32_t to = smem + L::parts + (uint32_t)t * L::parts_step + (uint32_t)n * 128u;
#pragma unroll
            for (int j = 0; j < kTasks; ++j)
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    st_shared_v4(to + (uint32_t)q * L::part + ((uint32_t)((kg0 + 4 * j) ^ (n & 7)) << 4), p[j][q][0], p[j][q][1], p[j][q][2], p[j][q][3]);
            fence_proxy_async();
            __syncwarp();
            if (elect_one()) {
                mbar_arrive(smem_u32(&s_ready[t]));
                mbar_arrive(smem_u32(&s_empty[st]));
            }
            __syncwarp();
            if (++st == ring) { st = 0; parity ^= 1u; }
        }
        block_await();
        if (s_again) {
            sum_again<BN, kRows>(f, smem_raw, s_full, s_empty, &s_abort);
            block_meet();
        }
    } else if (warp == kWarpCopy) {
        // ===== copies =====
        // The weights are constants: those of the first steps are on their way before the previous launch has to be waited for.  (A stage's barrier
        // is armed with the bytes of both operands.)
        int chunk = 2 * kb0, c = chunk, r = 0, s = 0, tap = 0;
        if (kb0 > 0) {
            tap = chunk / f.cpt;
            c = chunk - tap * f.cpt;
            r = tap / a.S;
            s = tap - r * a.S;
        }
        int w_tap = tap, w_c = c;
        auto copy_weights = [&](uint32_t st, int chunk_w) {
            const int have = min(2, f.chunks - chunk_w);
            const uint32_t bar = smem_u32(&s_full[st]), to = smem + st * L::stage + L::raw_w;
            if (elect_one()) mbar_arrive_expect_tx(bar, (uint32_t)have * ((kRows ? 0u : kBox) + L::w_box));
            for (int h = 0; h < have; ++h) {
                if (elect_one()) tma_load_3d(to + (uint32_t)h * L::w_box, &tmap_w, n0, w_c * kChunk, w_tap, bar);
                __syncwarp();
                if (++w_c == f.cpt) { w_c = 0; ++w_tap; }
            }
        };
        const int ahead = min((int)ring, n_kb);
        for (int kb = 0; kb < ahead; ++kb) copy_weights((uint32_t)kb, chunk + 2 * kb);
        int img = 0, w_org = 0, h_org = 0;
        if (!f.a_tiled) {
            img = m0 / f.PQ;
            const int rem = m0 - img * f.PQ, p = rem / a.Q, q = rem - p * a.Q;
            w_org = q * a.stride_w - a.pad_w;
            h_org = p * a.stride_h - a.pad_h;
        }
        griddep_wait();                            // the pixels are the previous launch's
        uint32_t st = 0, parity = 1u;
        for (int kb = 0; kb < n_kb; ++kb) {
            if (kb >= (int)ring) {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[st]), parity, &s_abort, err, 0x25u))) break;
                copy_weights(st, chunk);
            }
            const int have = kRows ? 0 : min(2, f.chunks - chunk);
            const uint32_t bar = smem_u32(&s_full[st]);
            for (int h = 0; h < have; ++h) {
                if (elect_one()) {
                    const uint32_t to = smem + st * L::stage + (uint32_t)h * kBox;
                    if (f.a_tiled) tma_load_2d(to, &tmap_x, c * kChunk, m0, bar);
                    else tma_load_im2col_4d(to, &tmap_x, c * kChunk, w_org, h_org, img, (uint16_t)(s * a.dil_w), (uint16_t)(r * a.dil_h), bar);
                }
                __syncwarp();
                if (++c == f.cpt) {
                    c = 0;
                    if (++s == a.S) { s = 0; ++r; }
                }
            }
            chunk += 2;
            if (++st == ring) { st = 0; parity ^= 1u; }
        }
        block_await();
        if (s_again) {
            copy_again<BN, kRows>(&tmap_x, &tmap_w, f, smem_raw, s_full, s_empty, &s_abort);
            block_meet();
        }
    } else {
        // ===== multiplications =====
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
        const uint64_t b0 = umma_desc_sw128(uniform(smem) + L::parts);
        bool ok = true;
        for (int kb = 0; kb < n_kb && ok; ++kb) {
            const int t = kb & 1;
            if (kb >= 2) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_free[t]), (uint32_t)((kb >> 1) - 1) & 1u, &s_abort, err, 0x27u));
            ok = ok && __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_ready[t]), (uint32_t)(kb >> 1) & 1u, &s_abort, err, 0x26u));
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t big = tmem + L::acc + (uint32_t)(t * 2 * BN), small = big + BN, at = tmem + L::a + (uint32_t)(t * 96);
            const uint64_t bt = b0 + (uint64_t)((uint32_t)t * (L::parts_step >> 4));
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t a0 = at + (uint32_t)(k * 8), a1 = a0 + 32u, a2 = a0 + 64u;
                    const uint64_t w0 = bt + (uint64_t)(k * 2), w1 = w0 + (L::part >> 4), w2 = w1 + (L::part >> 4);
                    mma_ta(small, a1, w2, idesc, k > 0 ? 1u : 0u);
                    mma_ta(small, a2, w1, idesc, 1u);
                    mma_ta(small, a0, w2, idesc, 1u);
                    mma_ta(small, a2, w0, idesc, 1u);
                    mma_ta(small, a1, w1, idesc, 1u);
                    mma_ta(small, a0, w1, idesc, 1u);
                    mma_ta(small, a1, w0, idesc, 1u);
                    mma_ta(big, a0, w0, idesc, k > 0 ? 1u : 0u);
                }
                tcgen05_commit(smem_u32(&s_done[t]));
            }
            __syncwarp();
        }
        block_await();
        if (s_again) block_meet();
    }
    tcgen05_fence_before();
    __syncthreads();
    if (s_abort) {          // copies and multiplications in flight finish before their memory goes
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t i = 0; i < (1u << 20); ++i)
            if (globaltimer_ns() - t0 > 50000ull) break;
        __syncthreads();
    }
    if (warp == kWarpMma) {
        tcgen05_fence_after();
        tcgen05_dealloc(tmem, kTmemCols);
    }
    if (nf) nf->end(job_id);
}

int batch_of(const pb_op_params* p) { return p->batch > 1 ? p->batch : 1; }
int dil(int d) { return d > 1 ? d : 1; }
bool pointwise(const pb_op_params* p) { return p->R == 1 && p->S == 1 && p->stride_h == 1 && p->stride_w == 1 && p->pad_h == 0 && p->pad_w == 0; }

// A filter row of such a layer is one chunk.
bool stem(const pb_op_params* p) { return p->Cs == 4 && p->S <= 8 && dil(p->dil_w) == 1 && p->R * p->S > 1 && p->K >= 16; }

struct SplitGeometry {
    int BN, m_tiles, n_tiles, splits, cpt, chunks;
    bool rows;                  // chunks are rows of the filter
    uint32_t smem;
    const void* fn;
};

SplitGeometry split_geometry(const pb_op_params* p) {
    SplitGeometry g;
    g.rows = stem(p);
    g.cpt = g.rows ? 1 : ceil_div(p->C, kChunk);
    g.chunks = g.rows ? p->R : p->R * p->S * g.cpt;
    g.m_tiles = ceil_div(batch_of(p) * p->P * p->Q, kTileRows);
    const int steps = ceil_div(g.chunks, 2);
    // Least modelled time: waves of one block an SM, each a block's fixed time (operand latency, the meeting of the ranks' sums, stores) and
    // its steps.  Measured in chains of equal launches (with six products a step; eight take 0.74 and 0.84 us), tile width / ranks -> us: 256 -> 256 channels 3x3 on 2 maps of 14 x 14 64/1 31.4, 64/2 18.2,
    // 64/4 11.9, 64/8 17.5 (two waves), 32/1 27.6, 32/2 15.9, 32/4 11.1; 512 -> 512 on 2 of 7 x 7 58.6, 31.8, 18.6, 12.5, 52.2, 28.0, 16.1, 20.6; 512 -> 512
    // 1x1 on one of 14 x 14 9.9, 7.4, 6.2, -, 8.5, 6.2, 5.9.
    static const struct { int splits, blocks; double fixed[2]; } kRanks[] = {{1, 148, {3.2, 4.0}}, {2, 148, {3.7, 4.6}}, {4, 132, {4.2, 5.1}}, {8, 120, {4.6, 5.6}}};
    double best = 1e30;
    for (int wide = 0; wide < (p->K > 32 ? 2 : 1); ++wide)
        for (const auto& c : kRanks) {
            if (c.splits > 1 && (steps < 2 * c.splits || conv_split_gain_us() > 1e6)) break;
            const int BN = wide ? 64 : 32, blocks = g.m_tiles * ceil_div(p->K, BN) * c.splits;
            const double us = ceil_div(blocks, c.blocks) * (c.fixed[wide] + ceil_div(steps, c.splits) * (wide ? 0.755 : 0.683));
            if (us < best) { best = us; g.BN = BN; g.splits = c.splits; }
        }
    g.n_tiles = ceil_div(p->K, g.BN);
    g.smem = (g.BN == 64 ? Layout<64>::bytes : Layout<32>::bytes) + 1024u;
    g.fn = g.BN == 64 ? (g.rows ? (const void*)conv_f32_split_kernel<64, true> : (const void*)conv_f32_split_kernel<64, false>)
                      : (g.rows ? (const void*)conv_f32_split_kernel<32, true> : (const void*)conv_f32_split_kernel<32, false>);
    return g;
}

// Modelled microseconds of a launch of up to 32 output channels here (fitted as conv_f32_units_us is, 2.3 % off in the mean).
double narrow_us(const pb_op_params* p) {
    const SplitGeometry g = split_geometry(p);
    const int waves = ceil_div(g.m_tiles * g.n_tiles * g.splits, g.splits == 8 ? 120 : g.splits == 4 ? 132 : 148);
    return 0.3 + waves * (4.1 + 0.736 * ceil_div(ceil_div(g.chunks, 2), g.splits) + (g.splits == 1 ? 0.0 : g.splits == 2 ? 0.65 : g.splits == 4 ? 1.0 : 1.2));
}

}  // namespace

uint32_t* conv_f32_error_flag_ptr() {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_f32_err_flag) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return static_cast<uint32_t*>(p);
}

// The layers that run here: what the copies can express - the output size that follows from
// padding, filter and stride (im2col boxes walk exactly those pixels), offsets within the descriptor's fields - and what gains.
// - A box is 32 channels of one tap, so a layer of fewer than 24 would multiply zeros: 56 x 56, 3x3, 8 images, 8 / 16 / 24 / 32 channels -> 64 the
//   fp32 units 18.7 / 24.5 / 30.7 / 36.1 us, here 19.1 / 19.1 / 19.2 / 19.1; one image 8.2 / 8.9 / 10.1 / 11.2 and 8.2 / 8.0 / 8.2 / 8.1.
// - 1x1 layers of up to 32 output channels are short and store little: 256 -> 24 at 14 x 14 5.6 and 7.3, 128 -> 24 at 28 x 28 x 8 6.2 and 6.4 (36
//   columns: 7.2 and 7.2, 9.1 and 6.7).
// - Larger filters of up to 32 output channels: whichever of two fitted times is less (narrow_us, conv_f32_units_us): 64 -> 16 3x3 on one of 28 x 28 5.6 and
//   7.5, 1x7 on one of 7 x 7 5.3 and 7.9, 64 -> 8 3x3 on 8 of 56 x 56 28 and 23.  Over 381 such layers of 32 channels and more the units take 9.36 ms, this kernel
//   6.16, the faster of the two 5.996, the modelled one 5.997.  (With 24 to 31 channels and in stems, below, this kernel takes them all.)
// - Stems: 7 x 7, stride 2, 64 channels on 1 / 2 / 8 images of 224 x 224 22.4 / 32.3 / 110 and 9.7 / 17.9 / 51 us; 3 x 3, stride 2, 32 channels on 2
//   and 8 10.6 / 31.2 and 10.1 / 28.1, 16 channels on 8 of 320 x 320 51.3 and 51.4, 8 channels 5 x 5 on one of 28 x 28 5.8 and 6.4.
// PB_F32_SPLIT=0 (read at every use; for tests and comparisons) keeps every layer on the fp32 units.
bool conv_f32_split_layer(const pb_op_params* p) {
    const char* e = getenv("PB_F32_SPLIT");
    if (e && e[0] == '0') return false;
    const int reach_h = (p->R - 1) * dil(p->dil_h), reach_w = (p->S - 1) * dil(p->dil_w);
    return (p->C >= 24 || stem(p)) && (p->K > 32 || (p->R * p->S > 1 && (p->C < kChunk || narrow_us(p) < conv_f32_units_us(p)))) && p->pad_h >= 0 && p->pad_w >= 0 && p->pad_h <= 100 &&
           p->pad_w <= 100 && reach_h <= 100 && reach_w <= 100 && p->stride_h >= 1 && p->stride_w >= 1 && p->stride_h <= 8 && p->stride_w <= 8 &&
           p->P == (p->H + 2 * p->pad_h - reach_h - 1) / p->stride_h + 1 && p->Q == (p->W + 2 * p->pad_w - reach_w - 1) / p->stride_w + 1;
}

int conv_f32_split_info(const pb_op_params* p, pb_launch_info* out) {
    const SplitGeometry g = split_geometry(p);
    out->num_blocks = (uint32_t)(g.m_tiles * g.n_tiles * g.splits);
    out->threads_per_block = kThreadsF;
    cudaFuncAttributes at;
    out->regs_per_thread = 72;
    if (cudaFuncGetAttributes(&at, g.fn) == cudaSuccess) out->regs_per_thread = (uint32_t)at.numRegs;
    else cudaGetLastError();
    out->smem_per_block = g.smem;
    out->tmem_cols_per_block = kTmemCols;
    return PB_OK;
}

int conv_f32_split_launch(const pb_op_params* p, const OpArgs& op, cudaStream_t st, uint32_t job_id, void* notifier, bool pdl) {
    const SplitGeometry g = split_geometry(p);
    SplitArgs f;
    f.op = op;
    f.PQ = p->P * p->Q;
    f.M = batch_of(p) * f.PQ;
    f.Kp = round_up(p->K, 4);
    f.cpt = g.cpt;
    f.chunks = g.chunks;
    f.splits = g.splits;
    f.a_tiled = pointwise(p) ? 1 : 0;
    CUtensorMap map, wmap;
    memset(&map, 0, sizeof(map));
    int rc = g.rows ? PB_OK
                    : encode_pixels_f32(p->x, p->C, p->Cs, p->W, p->H, batch_of(p), p->pad_w, p->pad_h, (p->S - 1) * dil(p->dil_w), (p->R - 1) * dil(p->dil_h),
                                        p->stride_w, p->stride_h, f.a_tiled != 0, kChunk, kTileRows, &map);
    if (rc == PB_OK) rc = g.rows ? encode_weights_f32(p->w, f.Kp, p->S * p->Cs, p->R, g.BN, kChunk, &wmap) : encode_weights_f32(p->w, f.Kp, p->Cs, p->R * p->S, g.BN, kChunk, &wmap);
    if (rc != PB_OK) return rc;
    PB_CUDA(cudaFuncSetAttribute(g.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)g.m_tiles, (unsigned)g.n_tiles, (unsigned)g.splits);
    cfg.blockDim = dim3(kThreadsF);
    cfg.dynamicSmemBytes = g.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (g.splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = (unsigned)g.splits;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    PB_CUDA(cudaLaunchKernelEx(&cfg, (void (*)(const CUtensorMap, const CUtensorMap, const SplitArgs, uint32_t, FinishedBlockNotifier*))g.fn, map, wmap, f, job_id,
                               static_cast<FinishedBlockNotifier*>(notifier)));
    return PB_OK;
}

}  // namespace pb
