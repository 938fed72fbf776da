// Dense convolution as an implicit GEMM on the 5th-generation tensor cores (sm_100a).
//
//   D[m, n] = sum_k A[m, k] * B[n, k]     m = output pixel (p*Q + q), n = output channel,
//                                          k = (r*S + s)*Cs + c   (filter tap, input channel)
//
// A is never materialised.  One thread per CTA issues, per 64-deep k-block, an im2col-mode TMA
// (cp.async.bulk.tensor.4d...im2col: 128 consecutive output pixels x 64 channels of one filter tap,
// padding and the ragged last tile zero-filled by the hardware; a plain tiled TMA when the layer is
// pointwise) that lands A in the 128-byte-swizzled K-major shared-memory layout tcgen05.mma reads,
// and a tiled TMA for B (packed weights [Kout_pad][Kdim_pad], no multicast).  One elected thread
// issues tcgen05.mma (M=128, N=BN, K=16, bf16 x bf16 -> fp32) with the accumulator in tensor
// memory; tcgen05.commit releases pipeline stages and signals the epilogue, which reads TMEM with
// tcgen05.ld, adds bias and residual, applies the activation and stores bf16 into the channel
// slice of the output tensor.
//
// CTA = 6 warps: warps 0-3 run the epilogue (thread t owns accumulator lane t), before it warp 3 loads
// operand B; warp 4 loads operand A, warp 5 allocates TMEM and issues the MMAs.  Sized for three CTAs per SM.
// Two entry points share the body (conv_tile_tma): conv_umma_tma_kernel runs one convolution,
// conv_umma_multi_kernel runs several independent ones as one grid from a descriptor table in
// device memory; conv_umma_pre_kernel also normalises its input tiles.  conv_umma_pair_kernel puts two blocks (cta_group::2)
// on a tile of 256 rows where a lone launch is large.  conv_umma_gather_kernel (PB_CONV_GATHER=1) is the earlier design, kept for
// comparison: 128 producer threads gather A with 16-byte cp.async copies (a lone Inception-v3 request
// takes 1656 us with it, 266 without).
//
// Every wait is bounded: when a wait runs out the CTA raises a device-global error flag,
// sets a shared abort flag that releases all other waits of the CTA, skips the epilogue,
// lets in-flight copies land, frees its TMEM and still reports block end.
//
// This is the tensor-core member of the kernel family the reference's TVM adapters launch
// (jobs/tvm_<model>/tvm_<model>.cpp:24-47; generated SIMT fp32 kernels there).
#include <cuda.h>
#include <cuda_bf16.h>
#include <llis/job/finished_block_notifier.h>

#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "conv_f32.h"
#include "launch_slot.cuh"
#include "ops.h"
#include "pb_common.h"
#include "umma.cuh"

using llis::job::FinishedBlockNotifier;

namespace pb {

namespace {

constexpr int kBM = 128;            // tile rows (output pixels) = TMEM lanes
constexpr int kBK = 64;             // bf16 elements per k-block = one 128-byte swizzle row
// Pipeline depth is a template parameter: kStages shared-memory stages.  Each producer thread keeps
// kLag = kStages/2 cp.async groups in flight (it arrives on a stage's barrier kLag iterations after
// issuing its copies).  The other half of the stages is slack for the hand-off round trip
// (producer arrive -> MMA issue -> tcgen05.commit -> producer may refill), which the probe measured
// at well over a microsecond: with only two stages of slack that round trip paced the whole loop.
#ifndef PB_LAG_OF
#define PB_LAG_OF(stages) ((stages) / 2)
#endif
constexpr int kMaxStages = 8;
constexpr int kMaxBN = 256;          // output channels per CTA tile at most (tcgen05.mma N <= 256)
constexpr uint32_t kSmemBudget = 200u * 1024u;   // one CTA per SM (gather kernel)
// The TMA kernel is sized for THREE CTAs per SM (73 KB of pipeline + ~2 KB static and reserved each
// out of 228 KB; <= 112 registers; <= 128 of 512 TMEM columns).  One CTA cannot pull more than about
// 60 bytes per clock through its SM and spends a third of its life in fixed latencies (set-up, first
// operand arrival, epilogue), so with many requests in flight residency, not pipeline depth, sets the
// GPU's convolution throughput: the co-resident CTAs keep the SM's load path busy between them.
#ifndef PB_CONV_SMEM_KB
#define PB_CONV_SMEM_KB 73
#endif
constexpr uint32_t kSmemBudgetTma = PB_CONV_SMEM_KB * 1024u;
constexpr uint32_t kSmemBudgetDeep = 110u * 1024u;      // small launches on a GPU they have to themselves: two CTAs per SM
constexpr uint32_t kSmemLimit = kSmemBudget + 2048u;    // dynamic shared memory the kernels are allowed
constexpr uint32_t kPreBytes = 512u;                    // scales and biases of a k-block of a normalising convolution
// What a split launch asks of pb_op_params.scratch.  The partial tiles meet in the shared memory of a thread-block
// cluster, so the memory itself is not touched: supplying it is how a caller allows the split (NULL = no split).
constexpr uint64_t kSplitScratchBytes = 256;
constexpr int kATileBytes = kBM * kBK * 2;   // 16 KiB
constexpr int kThreads = 160;

struct ConvArgs {
    const __nv_bfloat16* x;
    const __nv_bfloat16* residual;
    const float* bias;
    __nv_bfloat16* y;
    uint32_t* err_flag;
    int H, W, Cs;
    int P, Q, M;          // M = batch * P*Q: the images of a batch are consecutive rows of the GEMM
    int PQ;               // output pixels per image
    int dh, dw;           // filter dilation
    int K, Ks, out_c_off, res_Cs;
    int R, S, sh, sw, ph, pw;
    int act;
    int a_tiled;          // 1: pointwise convolution, operand A is the plain [M][Cs] matrix (tiled TMA, no im2col)
    int nkb;              // k-blocks of 64 = taps * chunks per tap
    int taps;             // R*S
    int Cp;               // channels per tap rounded up to 64: k = tap*Cp + c
    int BN;               // output channels per CTA (multiple of 16, <= 256)
    uint32_t idesc;       // tcgen05 instruction descriptor
    uint32_t tmem_cols;   // power of two >= max(32, BN)
    uint32_t b_stage_bytes;
    int out_box;          // channels of one TMA store box: 64 or 32 (divides BN); 0 = the epilogue stores directly
    int splits;           // thread blocks (one cluster) that share a tile's reduction: rank z takes k-blocks [nkb*z/splits, nkb*(z+1)/splits)
    uint32_t meet;        // where the other ranks' sums arrive in shared memory (0: in the pipeline buffers, once their multiplications are done)
    // A pointwise layer may take act(x * pre_scale + pre_bias), per input channel, instead of x (pre_scale NULL: x itself).
    const float* pre_scale;
    const float* pre_bias;
    int pre_act;
    uint32_t pre_offset;  // where their part of shared memory begins
    float inv_PQ, inv_Q, inv_cpt, inv_S;      // reciprocals of the divisors of a block's set-up
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Optional phase stamps for development builds (-DPB_CONV_TIMING): %globaltimer at ten points of
// the first 64 CTAs (8: sent to the other ranks, 9: their parts are here), written to a device array the probe program reads back.
#ifdef PB_CONV_TIMING
constexpr int kConvStamps = 10;
__device__ unsigned long long g_conv_t[64 * kConvStamps];
#define PB_T(i)                                                                                         \
    do {                                                                                                \
        static_assert((i) < kConvStamps, "a slot of its own for every stamp");                         \
        const unsigned b_ = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);             \
        if (b_ < 64) g_conv_t[b_ * kConvStamps + (i)] = globaltimer_ns();                                         \
    } while (0)
// per-k-block SM-clock stamps of the first 8 CTAs: [cta][kb][0 = loads issued, 1 = operands landed, 2 = MMAs issued]
__device__ unsigned long long g_conv_kb[8 * 64 * 3];
#define PB_TK(kb, i)                                                                                    \
    do {                                                                                                \
        const unsigned b_ = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);             \
        if (b_ < 8 && (kb) < 64) g_conv_kb[(b_ * 64 + (kb)) * 3 + (i)] = (unsigned long long)clock64();              \
    } while (0)
#else
#define PB_T(i) do {} while (0)
#define PB_TK(kb, i) do {} while (0)
#endif

// Optional per-phase cycle sums over every CTA of the TMA kernels (-DPB_CONV_STATS, development builds):
// [0] CTAs, [1] k-blocks, then clock64 differences: [2] set-up, [3] wait for the previous kernel, [4] first
// operands, [5] main loop (first operands landed -> last MMA issued), [6] accumulator drain, [7] epilogue,
// [8] tear-down, [9] whole CTA.
#ifdef PB_CONV_STATS
__device__ unsigned long long g_conv_stats[16];      // [10..15]: CTAs that found 0..5+ other conv CTAs resident on their SM
__device__ unsigned int g_conv_resident[256];        // conv CTAs resident per SM right now
__device__ long long g_persist_kb[64 * 6];          // CTA 0, its first tile: per k-block clock64 stamps (see PB_PK)
#define PB_PK(kb, i) do { if (blockIdx.x == 0 && first_tile && (kb) < 64) g_persist_kb[(kb) * 6 + (i)] = clock64(); } while (0)
__device__ unsigned int g_persist_resident;          // persistent CTAs resident GPU-wide right now
__device__ unsigned long long g_persist_hist[16];     // [b]: CTAs that found 32*b .. 32*b+31 others resident when they started; [15]: sum of lifetimes (clk)
__device__ long long g_persist_tile[16 * 6];        // CTA 0: per tile clock64 stamps (see PB_PT)
#define PB_PT(ti, i) do { if (blockIdx.x == 0 && (ti) < 16) g_persist_tile[(ti) * 6 + (i)] = clock64(); } while (0)
__device__ unsigned long long g_conv_ns;             // sum of the CTAs' lifetimes by %globaltimer (ns): cycles / ns = the SM clock
#define PB_S(i) do { s_clk[(i)] = clock64(); } while (0)
#else
#define PB_S(i) do {} while (0)
#define PB_PK(kb, i) do {} while (0)
#define PB_PT(ti, i) do {} while (0)
#endif

// ---- the kernel -----------------------------------------------------------------------
// Packed fp32 pairs (sm_100 has two-wide fp32 adds) and the bf16 pair conversion with the activation
// folded in: cvt's .relu clamps negatives to zero, ReLU6 is one more packed min against 6.0.
// Rounding is monotonic and 0 and 6 are bf16 values, so activation-after-rounding equals
// rounding-after-activation.
// n / d for n >= 0, with d's reciprocal: a few instructions where the integer division is a chain of twenty to forty (a block's set-up had five
// of them in a row).  The estimate is off by one at most while the quotient is below 2^22; the loops make it right whatever it is.
__device__ __forceinline__ int quotient(int n, int d, float inv, int& rem) {
    int q = (int)((float)n * inv);
    rem = n - q * d;
    while (rem < 0) { --q; rem += d; }
    while (rem >= d) { ++q; rem -= d; }
    return q;
}
// Cluster sizes are powers of two.
__device__ __forceinline__ int log2_of(int splits) { return 31 - __clz(splits); }

// What the epilogues of grouped and normalising launches need of a convolution's arguments, in registers before they wait for the
// accumulator.  (A grouped launch has its arguments in shared memory, and a compiler that sees a memory barrier reads them again behind
// each.)  Lone launches read their arguments where they are, in the constant bank, so that the compiler knows every branch on
// them to be taken alike, and have the activation's branch outside of the column loops (kAct).  Measured, a launch in a row of equal ones, us,
// registers and a branch per 8 columns / this: 64 -> 256 channels 1x1 on 8 maps of 56 x 56 7.04 / 6.39, 256 -> 1024 at 14 x 14
// with a residual 5.92 / 5.58, 184 -> 120 at 112 x 112, stride 2, with a residual 5.25 / 5.11; ResNet-50 x 8 images 373 / 359.  (For grouped and
// normalising launches this is the slower way: Inception-v3 alone 298.7 / 300.2, DenseNet-121 x 3 images 641 / 650.)
struct EpiArgs {
    const __nv_bfloat16* residual;
    const float* bias;
    __nv_bfloat16* y;
    uint32_t* err_flag;
    int M, K, Ks, out_c_off, res_Cs, act, BN, out_box, splits, nkb;
    uint32_t meet;
};
__device__ __forceinline__ EpiArgs epi_args(const ConvArgs& a) {
    return {a.residual, a.bias, a.y, a.err_flag, a.M, a.K, a.Ks, a.out_c_off, a.res_Cs, a.act, a.BN, a.out_box, a.splits, a.nkb, a.meet};
}

// The activation is chosen at run time, by branches all threads take alike: as a template parameter of the epilogues it made four
// copies of each (and of each cluster size), 124 KB of code per kernel, and a launch whose copy had not run on its SM lately
// spent 0.5 to 1.6 us of its epilogue fetching it.  The loops below are kept rolled for the same reason.  Two copies, ReLU and ReLU6 /
// the others, are as fast as four where the arguments are constants (the lone launches): see EpiArgs.
// kAct: 0 = the activation is chosen here, 1 = it is ReLU or ReLU6, 2 = it is neither.
// Eight accumulator columns of this thread's row, from channel k on: + bias (+ residual), activation, bf16.  The four epilogue
// warps run one per scheduler with nothing to hide instruction latency behind, so this is kept to one packed add and one
// convert per two columns.
template <int kAct, class Args>
__device__ __forceinline__ uint4 finish8(const Args& a, const uint32_t* v, const uint4& res, bool has_res, int k, const float* bias) {
    uint64_t f[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 b = *reinterpret_cast<const uint4*>(bias + 4 * h);
        f[2 * h] = add_f32x2(pack_f32x2(v[4 * h], v[4 * h + 1]), pack_f32x2(b.x, b.y));
        f[2 * h + 1] = add_f32x2(pack_f32x2(v[4 * h + 2], v[4 * h + 3]), pack_f32x2(b.z, b.w));
    }
    if (has_res) {
        const uint32_t ru[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) f[j] = add_f32x2(f[j], pack_f32x2(ru[j] << 16, ru[j] & 0xffff0000u));
    }
    uint32_t o[4];
    if (kAct == 1 || (kAct == 0 && (a.act == 1 || a.act == 2))) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float lo, hi;
            unpack_f32x2(f[j], lo, hi);
            asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(o[j]) : "f"(hi), "f"(lo));
        }
        if (a.act == 2) {
#pragma unroll
            for (int j = 0; j < 4; ++j) asm("min.bf16x2 %0, %1, %2;" : "=r"(o[j]) : "r"(o[j]), "r"(0x40C040C0u));
        }
    } else {
        if (a.act == 3) {           // PReLU: v > 0 ? v : slope * v, per channel; the slopes follow the biases
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float lo, hi;
                unpack_f32x2(f[j], lo, hi);
                float2 sl = make_float2(0.f, 0.f);
                if (k + 2 * j < a.K) sl = __ldg(reinterpret_cast<const float2*>(a.bias + a.K + k) + j);
                lo = lo > 0.f ? lo : lo * sl.x;
                hi = hi > 0.f ? hi : hi * sl.y;
                f[j] = pack_f32x2(__float_as_uint(lo), __float_as_uint(hi));
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float lo, hi;
            unpack_f32x2(f[j], lo, hi);
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[j]) : "f"(hi), "f"(lo));
        }
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
template <int kAct, class Args>
__device__ __forceinline__ void epilogue_chunk(const Args& a, const uint32_t (&v)[16], const uint4 (&rv)[2], int cb, int n0, bool row_valid,
                                               __nv_bfloat16* yrow, bool has_res, const float* s_bias) {
    if (!row_valid) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int k = n0 + cb + h * 8;
        if (k + 8 <= a.K) *reinterpret_cast<uint4*>(yrow + k) = finish8<kAct>(a, v + h * 8, rv[h], has_res, k, s_bias + cb + h * 8);
    }
}

// The residual of the 16 columns from cb on (zeros where there is none).
template <class Args>
__device__ __forceinline__ void load_residual(const Args& a, int k0, bool row_valid, const __nv_bfloat16* rrow, uint4 (&rv)[2]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        rv[h] = make_uint4(0, 0, 0, 0);
        if (row_valid && rrow && k0 + h * 8 + 8 <= a.K) rv[h] = *reinterpret_cast<const uint4*>(rrow + k0 + h * 8);
    }
}

// Columns in steps of 16, two steps in flight: the next step leaves tensor memory (and its residual is on its way)
// while this one is converted and stored.
template <int kAct, class Args>
__device__ __forceinline__ void epilogue_columns(const Args& a, uint32_t lane_addr, int n0, bool row_valid, __nv_bfloat16* yrow,
                                                 const __nv_bfloat16* rrow, const float* s_bias) {
    uint32_t v0[16], v1[16];
    uint4 r0[2], r1[2];
    const bool has_res = rrow != nullptr;
    tcgen05_ld16(lane_addr, v0);             // warp-collective: all lanes take part
    load_residual(a, n0, row_valid, rrow, r0);
#pragma unroll 1
    for (int cb = 0; cb < a.BN; cb += 32) {
        tcgen05_wait_ld();
        const bool second = cb + 16 < a.BN;
        if (second) {
            tcgen05_ld16(lane_addr + (uint32_t)(cb + 16), v1);
            load_residual(a, n0 + cb + 16, row_valid, rrow, r1);
        }
        epilogue_chunk<kAct>(a, v0, r0, cb, n0, row_valid, yrow, has_res, s_bias);
        if (!second) break;
        tcgen05_wait_ld();
        if (cb + 32 < a.BN) {
            tcgen05_ld16(lane_addr + (uint32_t)(cb + 32), v0);
            load_residual(a, n0 + cb + 32, row_valid, rrow, r0);
        }
        epilogue_chunk<kAct>(a, v1, r1, cb + 16, n0, row_valid, yrow, has_res, s_bias);
    }
}

// The same with the tile leaving, and the residual arriving, through TMA.  A warp's 16-byte accesses to its 32 rows touch 32
// lines each: 128 columns are 16 x 32 line accesses per warp, 2048 clocks of the SM's one load / store path per tile
// (1.9 us measured, and co-resident tiles queue behind each other; with a residual twice that: half of a ResNet-50 tile's life).
// So the tile is laid out in shared memory, boxes of 128 rows x U columns in the swizzle of their row length (no bank
// conflicts): the residual lands there before the accumulator is complete (s_res), each thread replaces its row's part by the
// result, and one lane of a warp stores the warp's 32 rows of a finished box with one instruction.  `buf`: 128 x BN x 2 bytes
// of the pipeline memory, free by now.  publish: this launch reports to the host, so the stores have to be in memory when the
// warp leaves; otherwise they only have to have been read (the next kernel waits for this one's memory operations).
template <int kAct, class Args>
__device__ __forceinline__ void epilogue_columns_tma(const Args& a, uint32_t lane_addr, int n0, bool has_res, const float* s_bias, uint32_t buf,
                                                     const CUtensorMap* tmap_y, int m0, bool publish) {
    const uint32_t r = threadIdx.x;                 // tile row
    const int U = a.out_box, m_warp = m0 + (int)(r & ~31u);
    const uint32_t swz = U == 64 ? r & 7u : (r >> 1) & 3u;
    const uint32_t row = buf + r * (uint32_t)(U * 2), warp_row = buf + (r & ~31u) * (uint32_t)(U * 2);
    uint32_t v0[16], v1[16];
    auto put = [&](const uint32_t (&v)[16], int cb) {
        const int in_box = cb & (U - 1);
        const uint32_t box = (uint32_t)(cb - in_box) * 256u;      // 128 rows x 2 bytes per column before this box
        // both halves' loads before either's store: a store is a barrier to the compiler
        const uint32_t at0 = row + box + (((uint32_t)(in_box >> 3) ^ swz) << 4), at1 = row + box + ((((uint32_t)(in_box >> 3) + 1u) ^ swz) << 4);
        uint4 res0 = make_uint4(0, 0, 0, 0), res1 = res0;
        if (has_res) { res0 = ld_shared_v4(at0); res1 = ld_shared_v4(at1); }
        const uint4 o0 = finish8<kAct>(a, v, res0, has_res, n0 + cb, s_bias + cb);
        const uint4 o1 = finish8<kAct>(a, v + 8, res1, has_res, n0 + cb + 8, s_bias + cb + 8);
        st_shared_v4(at0, o0.x, o0.y, o0.z, o0.w);
        st_shared_v4(at1, o1.x, o1.y, o1.z, o1.w);
        if (in_box + 16 == U) {
            fence_proxy_async();
            __syncwarp();
            const int x = n0 + cb - in_box;
            if (x < a.K && m_warp < a.M && elect_one()) tma_store_2d(tmap_y, x, m_warp, warp_row + box);
            __syncwarp();
        }
    };
    tcgen05_ld16(lane_addr, v0);             // warp-collective: all lanes take part
#pragma unroll 1
    for (int cb = 0; cb < a.BN; cb += 32) {
        tcgen05_wait_ld();
        tcgen05_ld16(lane_addr + (uint32_t)(cb + 16), v1);
        put(v0, cb);
        tcgen05_wait_ld();
        if (cb + 32 < a.BN) tcgen05_ld16(lane_addr + (uint32_t)(cb + 32), v0);
        put(v1, cb + 16);
    }
    if (elect_one()) {
        if (publish) tma_store_wait();
        else tma_store_wait_read();
    }
    __syncwarp();
}

// Epilogue, run by warps 0-3 (thread t owns accumulator lane t = tile row t): wait for the
// accumulator, then bias + residual + activation and bf16 stores into the output channel slice.
// tmap_y (the one-tile kernels): through TMA stores staged at `buf`.
// kByAct: a copy of the column loops for either kind of activation.
template <bool kByAct, class Args>
__device__ __forceinline__ void epilogue(const Args& a, uint32_t tmem_base, bool ok, int m0, int n0, const float* s_bias,
                                         uint64_t* s_accum_p, volatile uint32_t* s_abort_p, uint32_t accum_parity = 0u,
                                         const CUtensorMap* tmap_y = nullptr, uint32_t buf = 0, uint64_t* s_res = nullptr, bool publish = true) {
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int m = m0 + tid;
    const bool row_valid = m < a.M;
    if (ok) ok = mbar_wait(smem_u32(s_accum_p), accum_parity, s_abort_p, a.err_flag, 3u);
    ok = __all_sync(0xffffffffu, ok);   // tcgen05.ld below is warp-collective
    if (tid == 0) PB_T(5);
    tcgen05_fence_after();
    const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
    if (!ok) return;
    if (tmap_y) {
        const bool has_res = a.residual != nullptr;
        if (has_res && !__all_sync(0xffffffffu, mbar_wait(smem_u32(s_res), 0u, s_abort_p, a.err_flag, 6u))) return;
        if constexpr (!kByAct) epilogue_columns_tma<0>(a, lane_addr, n0, has_res, s_bias, buf, tmap_y, m0, publish);
        else if (a.act == 1 || a.act == 2) epilogue_columns_tma<1>(a, lane_addr, n0, has_res, s_bias, buf, tmap_y, m0, publish);
        else epilogue_columns_tma<2>(a, lane_addr, n0, has_res, s_bias, buf, tmap_y, m0, publish);
        return;
    }
    const __nv_bfloat16* rrow = a.residual ? a.residual + (size_t)m * a.res_Cs : nullptr;
    __nv_bfloat16* yrow = a.y + (size_t)m * a.Ks + a.out_c_off;
    if constexpr (!kByAct) epilogue_columns<0>(a, lane_addr, n0, row_valid, yrow, rrow, s_bias);
    else if (a.act == 1 || a.act == 2) epilogue_columns<1>(a, lane_addr, n0, row_valid, yrow, rrow, s_bias);
    else epilogue_columns<2>(a, lane_addr, n0, row_valid, yrow, rrow, s_bias);
}

// ---- split reduction: the thread blocks of a cluster share one output tile -----------------------------------
// Rank z of the cluster multiplies its share of the k-blocks; then rank d finishes columns [d*w, (d+1)*w) of the
// tile, w = BN / splits.  Every rank sends each owner its part straight from tensor memory (st.async: registers into the owner's
// shared memory, counted by the owner's barrier), 16 bytes per lane and consecutive lanes (= rows) side by side; the owner adds them
// in rank order to its own part, from its tensor memory, so the fp32 result does not depend on timing (in rank order all told, with its own among
// them, Inception-v3 alone takes 264 us instead of 262, ResNet-18 x 3 images 116.6 instead of 114.8).  Where the pipeline leaves
// room the parts have a place of their own and a rank sends as soon as its accumulator is complete; else they land in
// the owner's pipeline buffers, and every rank first tells the others that its multiplications are done with them.
// Nobody waits for having been read: a block ends when the others' parts, and before them their messages, have arrived.
// Bound by the way between SMs: with development probes 800 clocks and 20 bytes a clock per SM, however it is used; owners that pulled parked
// tiles with loads saw 8 to 10 (48 KB at four ranks 5080 clocks, 28 KB at eight 5070; st.async 3110 and 2410), and two cluster barriers
// besides.  (A global workspace under an atomic counter, before: +4 to +8 us per launch.)
// (Relaxed: it says that memory has been read, and a release takes 1500 clocks.)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tcgen05_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
// Ranks that have k-blocks: all of them unless a grouped launch splits a short reduction.
template <class Args>
__device__ __forceinline__ uint32_t active_ranks(const Args& a) {
    const int S = a.splits;
    if (a.nkb >= S) return (1u << S) - 1u;
    uint32_t active = 0;
#pragma unroll 1
    for (int z = 0; z < S; ++z) active |= ((a.nkb * (z + 1)) >> log2_of(S) > (a.nkb * z) >> log2_of(S) ? 1u : 0u) << z;
    return active;
}
// What arrives at a rank, in bytes.
template <class Args>
__device__ __forceinline__ uint32_t meet_bytes(const Args& a, int rank) {
    return (uint32_t)__popc(active_ranks(a) & ~(1u << rank)) * (uint32_t)(a.BN >> log2_of(a.splits)) * 512u;
}

// The columns of this rank: its own part, then the others' in rank order.  `at` is this thread's row of those, [rank but this][4 columns][row].
template <class Args>
__device__ __forceinline__ void cluster_finish(const Args& a, uint32_t own_addr, int k0, bool row_valid, __nv_bfloat16* yrow, const __nv_bfloat16* rrow,
                                               const float* bias, uint32_t others, uint32_t at, int w, bool mine, uint32_t (&own)[8], uint4 res) {
    const uint32_t step = (uint32_t)(w >> 2) * 2048u;      // between two ranks' parts
    const int n = a.splits - 1;
    const bool all = others == (1u << n) - 1u;
#pragma unroll 1
    for (int c = 0; c < w; c += 8) {
        const int k = k0 + c;
        uint64_t sum[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j] = pack_f32x2(own[2 * j], own[2 * j + 1]);
        uint4 next = make_uint4(0, 0, 0, 0);      // the residual and this rank's part of the next turn
        if (c + 8 < w) {
            tcgen05_ld8(own_addr + (uint32_t)c + 8u, own);
            if (rrow && row_valid && k + 8 < a.K) next = *reinterpret_cast<const uint4*>(rrow + k + 8);
        }
        auto add = [&](const uint4& p, const uint4& q) {
            sum[0] = add_f32x2(sum[0], pack_f32x2(p.x, p.y));
            sum[1] = add_f32x2(sum[1], pack_f32x2(p.z, p.w));
            sum[2] = add_f32x2(sum[2], pack_f32x2(q.x, q.y));
            sum[3] = add_f32x2(sum[3], pack_f32x2(q.z, q.w));
        };
        const uint32_t from = at + (uint32_t)(c >> 2) * 2048u;
        if (all && n == 3) {
            uint4 p[3], q[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                p[i] = ld_shared_v4(from + (uint32_t)i * step);
                q[i] = ld_shared_v4(from + (uint32_t)i * step + 2048u);
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) add(p[i], q[i]);
        } else {
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
                if (!((others >> i) & 1u)) continue;
                const uint4 p = ld_shared_v4(from + (uint32_t)i * step), q = ld_shared_v4(from + (uint32_t)i * step + 2048u);
                add(p, q);
            }
        }
        if (row_valid && k < a.K) {
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) asm("mov.b64 {%0, %1}, %2;" : "=r"(v[2 * j]), "=r"(v[2 * j + 1]) : "l"(sum[j]));
            *reinterpret_cast<uint4*>(yrow + k) = finish8<0>(a, v, res, rrow != nullptr, k, bias + c);
        }
        res = next;
        tcgen05_wait_ld();
        if (!mine) {
#pragma unroll
            for (int j = 0; j < 8; ++j) own[j] = 0;
        }
    }
}

// Run by warps 0-3 of every rank.  s_go: the other ranks' pipelines are free (splits - 1 arrivals); s_parts: their parts are here.
template <class Args>
__device__ __forceinline__ void epilogue_cluster(const Args& a, uint32_t tmem_base, int m0, int n0, int rank, uint32_t smem_base, const float* s_bias,
                                                 uint64_t* s_accum_p, uint64_t* s_go, uint64_t* s_parts, volatile uint32_t* s_abort_p) {
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int m = m0 + tid, S = a.splits, w = a.BN >> log2_of(S), k0 = n0 + rank * w;
    const bool row_valid = m < a.M;
    const uint32_t active = active_ranks(a);
    const bool mine = (active >> rank) & 1u;
    // What can be had before the accumulator is waited for: the residual's first part, the other ranks' arrival.
    const __nv_bfloat16* rrow = a.residual ? a.residual + (size_t)m * a.res_Cs : nullptr;
    uint4 res = make_uint4(0, 0, 0, 0);
    if (rrow && row_valid && k0 < a.K) res = *reinterpret_cast<const uint4*>(rrow + k0);
    cluster_wait();                 // every rank is running and has set its barriers up
    const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
    const uint32_t at = smem_base + a.meet + (uint32_t)tid * 16u, parts = smem_u32(s_parts);
    // Columns in steps of 8 from the next rank's on, so that not everybody sends to the same one at once.
    int d = rank + 1 < S ? rank + 1 : 0, c = d * w, left = w;
    uint32_t to = 0, bar = 0;
    auto address = [&]() {
        to = cluster_addr(at + (uint32_t)((rank - (rank > d ? 1 : 0)) * (w >> 2)) * 2048u, (uint32_t)d);
        bar = cluster_addr(parts, (uint32_t)d);
    };
    address();
    bool ok = mbar_wait(smem_u32(s_accum_p), 0u, s_abort_p, a.err_flag, 3u);
    ok = __all_sync(0xffffffffu, ok);
    if (tid == 0) PB_T(5);
    tcgen05_fence_after();
    bool go = true;
    if (a.meet == 0) {
        if (tid > 0 && tid < S) mbar_arrive_cluster(cluster_addr(smem_u32(s_go), (uint32_t)((rank + tid) & (S - 1))));
        __syncwarp();
    }
    uint32_t v0[8], v1[8];
    tcgen05_ld8(lane_addr + (uint32_t)c, v0);
    if (a.meet == 0) go = __all_sync(0xffffffffu, mbar_wait(smem_u32(s_go), 0u, s_abort_p, a.err_flag, 9u));
    if (mine && go) {
        auto send = [&](const uint32_t (&v)[8]) {
            st_async_v4(to, v[0], v[1], v[2], v[3], bar);
            st_async_v4(to + 2048u, v[4], v[5], v[6], v[7], bar);
            to += 4096u;
            if ((left -= 8) == 0) {
                left = w;
                d = d + 1 < S ? d + 1 : 0;
                address();
            }
        };
#pragma unroll 1
        for (int g = (a.BN - w) >> 3; g > 0; g -= 2) {
            c = c + 8 < a.BN ? c + 8 : 0;
            tcgen05_wait_ld();
            if (g > 1) tcgen05_ld8(lane_addr + (uint32_t)c, v1);
            send(v0);
            if (g == 1) break;
            c = c + 8 < a.BN ? c + 8 : 0;
            tcgen05_wait_ld();
            if (g > 2) tcgen05_ld8(lane_addr + (uint32_t)c, v0);
            send(v1);
        }
    }
    if (tid == 0) PB_T(8);
    // This rank's own first columns (zeros if it had no k-blocks), under the wait for the others' parts.
    tcgen05_wait_ld();
    const uint32_t own_addr = lane_addr + (uint32_t)(rank * w);
    tcgen05_ld8(own_addr, v0);
    // (Also when this block gives up: it stays until the others have written to it.)
    bool here = false;
    for (uint32_t i = 0; i < kWaitLimit && !here; ++i) here = mbar_try_wait(parts, 0u);
    if (!here) { *s_abort_p = 1; atomicExch(a.err_flag, 10u); }
    ok = __all_sync(0xffffffffu, here) && ok;
    tcgen05_wait_ld();
    if (!mine) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v0[j] = 0;
    }
    if (tid == 0) PB_T(9);
    if (ok) {
        __nv_bfloat16* yrow = a.y + (size_t)m * a.Ks + a.out_c_off;
        const uint32_t others = (active & ((1u << rank) - 1u)) | ((active >> (rank + 1)) << rank);
        const float* bias = s_bias + rank * w;
        cluster_finish(a, own_addr, k0, row_valid, yrow, rrow, bias, others, at, w, mine, v0, res);
    }
}

template <int kStages>
__global__ void __launch_bounds__(kThreads, 1)
conv_umma_gather_kernel(const __grid_constant__ CUtensorMap tmap_w, const ConvArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kStages];
    __shared__ __align__(8) uint64_t s_empty[kStages];
    __shared__ __align__(8) uint64_t s_accum;
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile uint32_t s_abort;
    __shared__ __align__(16) float s_bias[128];
    constexpr int kLag = PB_LAG_OF(kStages);

    resolve_slot(job_id, nf);
    if (nf) nf->start(job_id);
    if (threadIdx.x == 0) PB_T(0);

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_bytes = (uint32_t)kATileBytes + a.b_stage_bytes;

    const int m0 = blockIdx.x * kBM;
    const int n0 = blockIdx.y * a.BN;
    const int kb_begin = 0, nkb = a.nkb;         // this kernel never splits the reduction

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&s_full[s]), 4);      // one arrival per producer warp
            mbar_init(smem_u32(&s_empty[s]), 1);
        }
        mbar_init(smem_u32(&s_accum), 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 128) {
        const int k = n0 + tid;
        s_bias[tid] = (a.bias && tid < a.BN && k < a.K) ? __ldg(a.bias + k) : 0.f;
    }
    if (warp == 4) {
        tcgen05_alloc(smem_u32(&s_tmem_base), a.tmem_cols);
        tcgen05_relinquish();
    }

    // A-gather geometry.  Eight consecutive lanes cover the eight 16-byte chunks of one 128-byte tile
    // row, so one warp-wide cp.async touches 4 rows = 4 full 128-byte lines of the activation tensor
    // (when a row's chunks share a filter tap) instead of 32 partial ones.  Thread t copies chunk
    // t%8 of rows t/8 + 16*i, i = 0..7.
    const int chunk = tid & 7;
    const int rbase = (tid >> 3) & 15;
    int ih0[8], iw0[8];
    if (warp < 4) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int m = m0 + rbase + 16 * i;
            if (m < a.M) {
                const int p = m / a.Q, q = m - p * a.Q;
                ih0[i] = p * a.sh - a.ph;
                iw0[i] = q * a.sw - a.pw;
            } else {
                ih0[i] = -(1 << 28);      // fails every bounds check: the row is zero-filled
                iw0[i] = 0;
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    if (threadIdx.x == 0) PB_T(1);

    if (warp < 4) {
        // ===== A producer =====
        // position of this thread's chunk in k: filter tap (r, s) and first channel c
        const int kk0 = kb_begin * kBK + chunk * 8;
        int tap = kk0 / a.Cp;
        int c = kk0 - tap * a.Cp;
        int r = tap / a.S, s = tap - r * a.S;
        const uint32_t dst_off = (uint32_t)rbase * 128u + (((uint32_t)chunk ^ (uint32_t)(rbase & 7)) << 4);
        bool ok = true;
        for (int kb = 0; kb < nkb; ++kb) {
            const int st = kb % kStages;
            const uint32_t use = (uint32_t)(kb / kStages);
            if (ok) ok = mbar_wait(smem_u32(&s_empty[st]), (use & 1u) ^ 1u, &s_abort, a.err_flag, 1u);
            const uint32_t a_tile = smem_base + (uint32_t)st * stage_bytes;
            if (ok) {
                if (tid == 0) {
                    mbar_expect_tx(smem_u32(&s_full[st]), a.b_stage_bytes);
                    tma_load_2d(a_tile + kATileBytes, &tmap_w, (kb_begin + kb) * kBK, n0, smem_u32(&s_full[st]));
                }
                const bool tap_ok = tap < a.taps && c < a.Cs;
                const __nv_bfloat16* xc = a.x + c;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int ih = ih0[i] + r * a.dh, iw = iw0[i] + s * a.dw;
                    const bool inb = tap_ok && ih >= 0 && ih < a.H && iw >= 0 && iw < a.W;
                    const __nv_bfloat16* src = inb ? xc + ((size_t)ih * a.W + iw) * a.Cs : a.x;
                    cp_async_16(a_tile + dst_off + (uint32_t)i * 2048u, src, inb ? 16u : 0u);
                }
                c += kBK;
                while (c >= a.Cp) {
                    c -= a.Cp; ++tap; ++s;
                    if (s == a.S) { s = 0; ++r; }
                }
            }
            cp_async_commit();
            if (kb == 0 && tid == 0) PB_T(2);
            // One arrival per warp: 128 threads arriving on the same shared-memory word serialise
            // (measured: ~0.2 us per k-block); every lane first makes its own copies visible to the
            // async proxy, the warp converges, one lane arrives.
            if (kb >= kLag) {
                cp_async_wait<kLag>();
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_full[(kb - kLag) % kStages]));
            }
        }
        // drain: the last kLag k-blocks
        cp_async_wait<0>();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0)
            for (int kb = (nkb > kLag ? nkb - kLag : 0); kb < nkb; ++kb) mbar_arrive(smem_u32(&s_full[kb % kStages]));

        // ===== epilogue: accumulator lane `tid` = tile row `tid` =====
        epilogue<true>(a, tmem_base, ok, m0, n0, s_bias, &s_accum, &s_abort);
        if (tid == 0) PB_T(6);
    } else {
        // ===== MMA issuer: one thread =====
        if (lane == 0) {
            bool ok = true;
            for (int kb = 0; kb < nkb && ok; ++kb) {
                const int st = kb % kStages;
                const uint32_t use = (uint32_t)(kb / kStages);
                ok = mbar_wait(smem_u32(&s_full[st]), use & 1u, &s_abort, a.err_flag, 2u);
                if (!ok) break;
                if (kb == 0) PB_T(3);
                tcgen05_fence_after();
                const uint32_t a_tile = smem_base + (uint32_t)st * stage_bytes;
                const uint32_t b_tile = a_tile + kATileBytes;
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) {
                    tcgen05_mma_bf16(tmem_base, umma_desc_sw128(a_tile + k * 32), umma_desc_sw128(b_tile + k * 32), a.idesc,
                                     (kb > 0 || k > 0) ? 1u : 0u);
                }
                tcgen05_commit(smem_u32(&s_empty[st]));   // frees the stage once these MMAs have read it
            }
            if (ok) tcgen05_commit(smem_u32(&s_accum));   // accumulator complete
            PB_T(4);
        }
        __syncwarp();
    }

    tcgen05_fence_before();
    __syncthreads();
    if (s_abort) {
        // Let copies that may still be in flight land before shared memory is released.
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t i = 0; i < (1u << 20); ++i) {
            if (globaltimer_ns() - t0 > 50000ull) break;
        }
        __syncthreads();
    }
    if (warp == 4) {
        tcgen05_fence_after();
        tcgen05_dealloc(tmem_base, a.tmem_cols);
    }
    if (threadIdx.x == 0) PB_T(7);
    if (nf) nf->end(job_id);
}

constexpr int kThreadsTma = 192;
constexpr int kWarpB = 3;          // issues operand B's copies

// ---- a batch-norm in front of a pointwise convolution -----------------------------------------------------------
// DenseNet normalises the concatenated features before each 1x1 convolution, each time with other constants, so no earlier
// epilogue can do it.  As a launch of its own that is 2.5 us and a hand-over of 0.75 us for a few hundred KB.  Here the tile of
// raw features is normalised where it landed: the epilogue's warps, idle until the accumulator is complete, rewrite each stage of
// operand A in shared memory and then let the MMA warp have it (operand A's warp loads operand B too).  Two warps take a stage, so
// that one pair's wait and fence lie beside the other's arithmetic; a thread has one vector of 8 channels of sixteen rows, eight in
// flight.  Bound by these warps' instructions: about 0.35 us a k-block, where a layer without it takes 0.2 (all four warps on one
// stage: 0.37; three warps: 0.48; constants read from global memory per k-block: 1.0, slower than the launch it replaces).
// The arithmetic is affine_kernel's - fp32 multiply-add, ReLU, one rounding to bf16 - and so are the bits (the maximum with
// zero may follow the rounding: rounding is monotonic and keeps zeros; NaN gives zero either way).
// The normalised tiles also go to the affine's own tensor, where whoever launches or reads single stages afterwards looks for them:
// operand A's warp stores a stage through TMA before it loads the next tile there, and the blocks of a row tile, which normalise the same
// k-blocks, take turns at that.  (DenseNet-121 of three images: 622 us without these stores, 637 with them, 670 when the normalising
// threads store.)
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t x, uint64_t y, uint64_t z) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
// consts: [k-block][64 scales, 64 biases] of this rank's k-blocks, in shared memory.
__device__ __forceinline__ void normalise_constants(const ConvArgs& a, float* consts, int kb_begin, int nkb) {
    for (int i = threadIdx.x; i < nkb * 32; i += 128) {
        const int c = (i & 15) * 4, from = (kb_begin + (i >> 5)) * kBK + c;
        const float* src = (i & 16 ? a.pre_bias : a.pre_scale) + from;
        *reinterpret_cast<float4*>(consts + i * 4) = from < a.Cs ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
}
__device__ __forceinline__ void normalise_stages(const ConvArgs& a, uint32_t smem_base, uint32_t stage_bytes, int stages, int nkb, const float* consts,
                                                 uint64_t* s_full, uint64_t* s_ready, volatile uint32_t* s_abort) {
    const uint32_t vec = threadIdx.x & 7u, row = threadIdx.x >> 3 & 7u;      // rows row + 8 i: the swizzle is the same for all
    const uint32_t pair = uniform(threadIdx.x >> 6);
    const uint32_t at = smem_base + row * 128u + ((vec ^ (row & 7u)) << 4);
    uint32_t st = pair, parity = 0;              // (a pipeline has two stages at least)
    const bool relu = a.pre_act == 1;
#pragma unroll 1
    for (int kb = (int)pair; kb < nkb; kb += 2) {
        uint64_t sc[4], bi[4];
        const ulonglong2* k = reinterpret_cast<const ulonglong2*>(consts + kb * 128 + vec * 8);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const ulonglong2 s = k[h], b = k[h + 16];
            sc[2 * h] = s.x; sc[2 * h + 1] = s.y;
            bi[2 * h] = b.x; bi[2 * h + 1] = b.y;
        }
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[st]), parity, s_abort, a.err_flag, 7u))) return;
#pragma unroll 1
        for (uint32_t half = 0; half < 2; ++half) {
            const uint32_t tile = at + st * stage_bytes + half * 8192u;
            uint4 v[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) v[i] = ld_shared_v4(tile + i * 1024u);
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float lo, hi;
                    unpack_f32x2(fma_f32x2(pack_f32x2(u[j] << 16, u[j] & 0xffff0000u), sc[j], bi[j]), lo, hi);
                    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[j]) : "f"(hi), "f"(lo));
                }
                if (relu) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) asm("max.bf16x2 %0, %1, %2;" : "=r"(o[j]) : "r"(o[j]), "r"(0u));
                }
                st_shared_v4(tile + i * 1024u, o[0], o[1], o[2], o[3]);
            }
        }
        fence_proxy_async();
        __syncwarp();
        if (elect_one()) mbar_arrive(smem_u32(&s_ready[st]));
        __syncwarp();
        if ((st += 2u) >= (uint32_t)stages) { st -= (uint32_t)stages; parity ^= 1u; }
    }
}

// ---- the kernel, operand A by im2col TMA ---------------------------------------------------------
// CTA = 6 warps, each with a short loop of its own: warps 0-3 the epilogue, before it warp 3 operand B (one tiled TMA of
// weights per k-block), warp 4 operand A (one im2col TMA of 128 output pixels x 64 channels of one filter tap), warp 5
// tensor memory and the MMAs.  No thread computes an address in the main loop.  (A seventh warp for operand B would
// leave 80 registers a thread at three CTAs per SM instead of 96.)

// One CTA's share of one convolution: output tile (bx, by), rank bz of the cluster that shares the tile's
// reduction, `stages` pipeline buffers.  Shared by the single-convolution kernel and the grouped one.
// kPre: the tile's input is normalised first (see above; a kernel of its own: the others' code and registers stay as they are).
// kLone: the launch has this convolution only and does not normalise.
template <bool kPre, bool kLone>
__device__ __forceinline__ void conv_tile_tma(const CUtensorMap* tmap_w, const CUtensorMap* tmap_x, const CUtensorMap* tmap_y, const CUtensorMap* tmap_r,
                                              const CUtensorMap* tmap_n, const ConvArgs& a, const int stages,
                                              const int bx, const int by, const int bz, uint8_t* smem_raw,
                                              uint64_t* s_full, uint64_t* s_empty, uint64_t* s_accum, uint32_t* s_tmem_base,
                                              volatile uint32_t* s_abort, float* s_bias, uint64_t* s_res, uint64_t* s_ready, uint64_t* s_go, uint64_t* s_parts, bool publish) {
    const int tid = threadIdx.x;
    const int warp = (int)uniform((uint32_t)tid >> 5);
    const int lane = tid & 31;
#ifdef PB_CONV_STATS
    __shared__ long long s_clk[8];
    __shared__ unsigned s_smid;
    __shared__ unsigned long long s_ns0;
    if (tid == 0) {
        PB_S(0);
        s_ns0 = globaltimer_ns();
        unsigned smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        s_smid = smid & 255u;
        const unsigned others = atomicAdd(&g_conv_resident[s_smid], 1u);
        atomicAdd(&g_conv_stats[10 + (others < 5 ? others : 5)], 1ull);
    }
#endif
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_bytes = (uint32_t)kATileBytes + a.b_stage_bytes;

    const int m0 = bx * kBM;
    const int n0 = by * a.BN;
    const int ranks_log2 = log2_of(a.splits);
    const int kb_begin = (a.nkb * bz) >> ranks_log2;
    const int nkb = ((a.nkb * (bz + 1)) >> ranks_log2) - kb_begin;       // 0 for some ranks of a cluster larger than the k-block count

    // Operand B's warp sets the barriers up and starts at once on the first turn of the pipeline: the weights are
    // constant, so they need neither the other warps nor the previous kernel.  It also arms each stage's barrier with the
    // byte count of both operands.  (Operand A's bytes may land before that: the transaction count goes negative for a
    // moment, and the phase cannot complete before the arrival.)
    const uint32_t tx_bytes = (uint32_t)kATileBytes + a.b_stage_bytes;
    if (warp == kWarpB) {
        // The weights' map is on its way while the barriers are set up (behind them a launch of a few k-blocks waits for it: 32 -> 16 channels 1x1 on
        // 8 x 8 3.00 us, this 2.75).
        if (elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(tmap_w) : "memory");
        // a lane per barrier: one thread took 20 initialisations in a row
        if (lane < stages) {
            mbar_init(smem_u32(&s_full[lane]), 1);      // this warp's arrive.expect_tx, for the bytes of both operands
            mbar_init(smem_u32(&s_empty[lane]), 1);     // tcgen05.commit
            if (kPre) mbar_init(smem_u32(&s_ready[lane]), 2);     // normalised: one arrival of each of two warps
        } else if (lane == kMaxStages) {
            mbar_init(smem_u32(s_accum), kPre ? 2 : 1);                // normalised: its memory is free, too
            mbar_init(smem_u32(s_res), 1);
            *s_abort = 0;
        } else if (lane == kMaxStages + 1 && a.splits > 1) {
            mbar_init(smem_u32(s_go), (uint32_t)(a.splits - 1));
            mbar_init(smem_u32(s_parts), 1);
            mbar_arrive_expect_tx(smem_u32(s_parts), meet_bytes(a, bz));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        // The first k-block's weights only: its other copies leave in the main loop (six of them here held every warp at the
        // barrier below for 0.3 us a tile).
        if (nkb > 0) {
            if (elect_one()) {
                mbar_arrive_expect_tx(smem_u32(&s_full[0]), tx_bytes);
                tma_load_2d(smem_base + kATileBytes, tmap_w, kb_begin * kBK, n0, smem_u32(&s_full[0]));
            }
            __syncwarp();
        }
    }
    // Where the tile's pixels start is worked out before the wait for the previous kernel.
    int img = 0, w0 = 0, h0 = 0, tap_r = 0, tap_s = 0, chunk = 0;
    const int cpt = a.Cp / kBK;               // k-blocks per filter tap
    if (warp == 4) {
        if (elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(tmap_x) : "memory");
        if (!a.a_tiled) {
            int rem, q0;
            img = quotient(m0, a.PQ, a.inv_PQ, rem);      // the tile may run on into the next image
            const int p0 = quotient(rem, a.Q, a.inv_Q, q0);
            w0 = q0 * a.sw - a.pw;                // filter-window origin of the tile's first pixel
            h0 = p0 * a.sh - a.ph;
        }
        if (kb_begin > 0) tap_r = quotient(quotient(kb_begin, cpt, a.inv_cpt, chunk), a.S, a.inv_S, tap_s);
    }
    if (warp == 5) {
        tcgen05_alloc(smem_u32(s_tmem_base), a.tmem_cols);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    if (a.splits > 1) cluster_arrive_relaxed();      // (the barriers' fence has released them) the epilogue waits for the other ranks before it sends them anything
    const uint32_t tmem_base = uniform(*s_tmem_base);
    if (tid == 0) { PB_T(1); PB_S(1); }

    if (warp < 4) {
        if (warp == kWarpB && !kPre) {
            // ===== operand B =====
            uint32_t* const err_flag = a.err_flag;
            uint32_t st = stages > 1 ? 1u : 0u, parity = stages > 1 ? 1u : 0u;
            for (int kb = 1; kb < nkb; ++kb) {
                if (kb >= stages && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[st]), parity, s_abort, err_flag, 1u))) break;
                if (elect_one()) {
                    mbar_arrive_expect_tx(smem_u32(&s_full[st]), tx_bytes);
                    tma_load_2d(smem_base + st * stage_bytes + kATileBytes, tmap_w, (kb_begin + kb) * kBK, n0, smem_u32(&s_full[st]));
                }
                __syncwarp();
                if (++st == (uint32_t)stages) { st = 0; parity ^= 1u; }
            }
        } else if (warp != kWarpB) {
            // the epilogue's biases
            for (int j = tid; j < a.BN; j += 32 * kWarpB) {
                const int k = n0 + j;
                s_bias[j] = (a.bias && k < a.K) ? __ldg(a.bias + k) : 0.f;
            }
        }
        if (kPre) {
            float* const consts = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)) + a.pre_offset);
            normalise_constants(a, consts, kb_begin, nkb);
            griddep_wait();
            griddep_launch();
            normalise_stages(a, smem_base, stage_bytes, stages, nkb, consts, s_full, s_ready, s_abort);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        // The residual and the output may only be touched once the previous kernel has completed; the next kernel's
        // blocks may be scheduled as SM resources free up.
        griddep_wait();
        if (tid == 0) PB_S(2);
        griddep_launch();
        if (a.splits > 1) epilogue_cluster(epi_args(a), tmem_base, m0, n0, bz, smem_base, s_bias, s_accum, s_go, s_parts, s_abort);
        else if constexpr (kLone) epilogue<true>(a, tmem_base, true, m0, n0, s_bias, s_accum, s_abort, 0u, a.out_box ? tmap_y : nullptr, smem_base, s_res, publish);
        else epilogue<false>(epi_args(a), tmem_base, true, m0, n0, s_bias, s_accum, s_abort, 0u, a.out_box ? tmap_y : nullptr, smem_base, s_res, publish);
        if (tid == 0) { PB_T(6); PB_S(6); }
    } else if (warp == 4) {
        // ===== operand A =====
        uint32_t* const err_flag = a.err_flag;
        for (int kb = 1; kPre && kb < min(stages, nkb); ++kb) {      // operand B's warp normalises
            if (elect_one()) {
                mbar_arrive_expect_tx(smem_u32(&s_full[kb]), tx_bytes);
                tma_load_2d(smem_base + kb * stage_bytes + kATileBytes, tmap_w, (kb_begin + kb) * kBK, n0, smem_u32(&s_full[kb]));
            }
            __syncwarp();
        }
        griddep_wait();                           // the activations are the previous kernel's
        const int S = a.S, dw = a.dw, dh = a.dh, a_tiled = a.a_tiled;
        // The normalised k-block kb, in stage st, to its tensor (by one lane: it waits for its own stores).
        auto store_normalised = [&](int kb, uint32_t st, uint32_t parity) {
            if ((unsigned)(kb_begin + kb) % gridDim.y != (unsigned)by) return true;
            if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_ready[st]), parity, s_abort, err_flag, 8u))) return false;
            if (lane == 0) tma_store_2d(tmap_n, (kb_begin + kb) * kBK, m0, smem_base + st * stage_bytes);
            __syncwarp();
            return true;
        };
        uint32_t st = 0, parity = 1u;             // a fresh barrier passes a wait on the "previous" phase
        for (int kb = 0; kb < nkb; ++kb) {
            if (kPre && kb >= stages && !store_normalised(kb - stages, st, parity)) break;
            if (kb >= stages && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[st]), parity, s_abort, err_flag, 1u))) break;
            if (kPre && kb >= stages) {
                if (lane == 0) tma_store_wait_read();
                __syncwarp();
            }
            if (elect_one()) {
                const uint32_t a_tile = smem_base + st * stage_bytes, bar = smem_u32(&s_full[st]);
                if (kPre && kb >= stages) {
                    mbar_arrive_expect_tx(bar, tx_bytes);
                    tma_load_2d(a_tile + kATileBytes, tmap_w, (kb_begin + kb) * kBK, n0, bar);
                }
                if (a_tiled) tma_load_2d(a_tile, tmap_x, chunk * kBK, m0, bar);
                else tma_load_im2col_4d(a_tile, tmap_x, chunk * kBK, w0, h0, img, (uint16_t)(tap_s * dw), (uint16_t)(tap_r * dh), bar);
                if (kb == 0) PB_T(2);
                PB_TK(kb, 0);
            }
            __syncwarp();
            if (++chunk == cpt) {
                chunk = 0;
                if (++tap_s == S) { tap_s = 0; ++tap_r; }
            }
            if (++st == (uint32_t)stages) { st = 0; parity ^= 1u; }
        }
        if (kPre) {
            // The epilogue may start once the stages whose memory it uses (for the others' parts or the finished tile) have been stored; the
            // others leave beside it.
            const uint32_t bytes = a.splits > 1 ? (a.meet ? 0u : (uint32_t)(a.BN - (a.BN >> ranks_log2)) * 512u) : a.out_box ? (uint32_t)a.BN * 256u : 0u;
            const int used = (int)((bytes + stage_bytes - 1) / stage_bytes), last_st = nkb > 0 ? (nkb - 1) % stages : 0;
            const int until = used > 0 ? nkb - 1 - max(0, last_st - (used - 1)) : -1;        // the last k-block in one of them
            auto let_epilogue = [&]() {
                if (lane == 0) {
                    tma_store_wait_read();
                    mbar_arrive(smem_u32(s_accum));
                }
                __syncwarp();
            };
            if (until < 0) let_epilogue();
            for (int kb = max(0, nkb - stages); kb < nkb; ++kb) {
                if (!store_normalised(kb, (uint32_t)(kb % stages), (uint32_t)(kb / stages) & 1u)) break;
                if (kb == until) let_epilogue();
            }
        }
        // The residual goes where the tile will be laid out, as soon as the multiplications have read the pipeline buffers there.
        if (a.residual && a.out_box) {
            const uint32_t bytes = (uint32_t)a.BN * 256u;
            bool ok = true;
            for (uint32_t q = 0; q * stage_bytes < bytes && ok; ++q) {
                const int uses = nkb > (int)q ? (nkb - (int)q + stages - 1) / stages : 0;
                if (uses > 0) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[q]), (uint32_t)(uses - 1) & 1u, s_abort, err_flag, 1u));
            }
            if (ok && elect_one()) {
                mbar_arrive_expect_tx(smem_u32(s_res), bytes);
                for (int c = 0; c < a.BN; c += a.out_box) tma_load_2d(smem_base + (uint32_t)c * 256u, tmap_r, n0 + c, m0, smem_u32(s_res));
            }
            __syncwarp();
        }
        griddep_launch();
        if (kPre && lane == 0) tma_store_wait_read();
    } else {
        // ===== MMA issuer =====
        // A wait on a complete barrier costs about 130 clocks and the tensor pipe holds few instructions, so it drains meanwhile:
        // four multiplications of 32 columns take 160 clocks, a k-block 325.  Probing the next barrier before the multiplications
        // are issued only puts the probe's latency in front of them (360).  The descriptors are stage 0's plus a stride.
        uint32_t st = 0, parity = 0u;
        bool ok = true;
        uint32_t* const err_flag = a.err_flag;
        const uint32_t idesc = uniform(a.idesc), n_kb = uniform((uint32_t)nkb), n_st = uniform((uint32_t)stages);
        const uint64_t desc_a0 = umma_desc_sw128(uniform(smem_base)), desc_b0 = umma_desc_sw128(uniform(smem_base) + kATileBytes);
        const uint32_t desc_step = uniform(stage_bytes) >> 4;      // address field counts 16-byte units; no carry out of its 14 bits
        uint64_t* const s_operands = kPre ? s_ready : s_full;
        for (uint32_t kb = 0; kb < n_kb; ++kb) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_operands[st]), parity, s_abort, err_flag, 2u));
            if (!ok) break;
            if (lane == 0) { if (kb == 0) { PB_T(3); PB_S(3); } PB_TK(kb, 1); }
            tcgen05_fence_after();
            uint32_t st_n = st + 1, parity_n = parity;
            if (st_n == n_st) { st_n = 0; parity_n ^= 1u; }
            const uint64_t da = desc_a0 + st * desc_step, db = desc_b0 + st * desc_step;
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k)
                    tcgen05_mma_bf16(tmem_base, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);   // +32 bytes per K=16 slice
                tcgen05_commit(smem_u32(&s_empty[st]));
            }
            __syncwarp();
            if (lane == 0) PB_TK(kb, 2);
            st = st_n;
            parity = parity_n;
        }
        if (lane == 0) PB_S(4);
        if (ok && elect_one()) tcgen05_commit(smem_u32(s_accum));
        __syncwarp();
        if (lane == 0) PB_T(4);
#ifdef PB_CONV_STATS
        if (ok) mbar_wait(smem_u32(s_accum), 0u, s_abort, a.err_flag, 3u);
        if (lane == 0) PB_S(5);
#endif
        __syncwarp();
        griddep_launch();
    }

    tcgen05_fence_before();
    __syncthreads();
    if (*s_abort) {
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t i = 0; i < (1u << 20); ++i) {
            if (globaltimer_ns() - t0 > 50000ull) break;
        }
        __syncthreads();
    }
    if (warp == 5) {
        tcgen05_fence_after();
        tcgen05_dealloc(tmem_base, a.tmem_cols);
    }
    if (threadIdx.x == 0) PB_T(7);
#ifdef PB_CONV_STATS
    __syncthreads();
    if (threadIdx.x == 0) {
        const long long c7 = clock64();
        atomicAdd(&g_conv_stats[0], 1ull);
        atomicAdd(&g_conv_stats[1], (unsigned long long)nkb);
        for (int i = 0; i < 6; ++i) atomicAdd(&g_conv_stats[2 + i], (unsigned long long)(s_clk[i + 1] - s_clk[i]));
        atomicAdd(&g_conv_stats[8], (unsigned long long)(c7 - s_clk[6]));
        atomicAdd(&g_conv_stats[9], (unsigned long long)(c7 - s_clk[0]));
        atomicSub(&g_conv_resident[s_smid], 1u);
        atomicAdd(&g_conv_ns, globaltimer_ns() - s_ns0);
    }
#endif
}

__global__ void __launch_bounds__(kThreadsTma, 3)
conv_umma_tma_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                     const __grid_constant__ CUtensorMap tmap_y, const __grid_constant__ CUtensorMap tmap_r, const ConvArgs a, int stages, uint32_t job_id, FinishedBlockNotifier* nf) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxStages];
    __shared__ __align__(8) uint64_t s_empty[kMaxStages];
    __shared__ __align__(8) uint64_t s_res;
    __shared__ __align__(8) uint64_t s_accum;
    __shared__ __align__(8) uint64_t s_go;
    __shared__ __align__(8) uint64_t s_parts;
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile uint32_t s_abort;
    __shared__ __align__(16) float s_bias[kMaxBN];

    resolve_slot(job_id, nf);
    if (nf) nf->start(job_id);
    if (threadIdx.x == 0) PB_T(0);
    conv_tile_tma<false, true>(&tmap_w, &tmap_x, &tmap_y, &tmap_r, nullptr, a, stages, (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, smem_raw, s_full, s_empty, &s_accum,
                         &s_tmem_base, &s_abort, s_bias, &s_res, nullptr, &s_go, &s_parts, nf != nullptr);
    if (nf) nf->end(job_id);
}

// The same with the input normalised; tmap_n: the normalised input's own tensor.
__global__ void __launch_bounds__(kThreadsTma, 3)
conv_umma_pre_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y,
                     const __grid_constant__ CUtensorMap tmap_r, const __grid_constant__ CUtensorMap tmap_n, const ConvArgs a, int stages, uint32_t job_id,
                     FinishedBlockNotifier* nf) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxStages];
    __shared__ __align__(8) uint64_t s_empty[kMaxStages];
    __shared__ __align__(8) uint64_t s_ready[kMaxStages];
    __shared__ __align__(8) uint64_t s_res;
    __shared__ __align__(8) uint64_t s_accum;
    __shared__ __align__(8) uint64_t s_go;
    __shared__ __align__(8) uint64_t s_parts;
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile uint32_t s_abort;
    __shared__ __align__(16) float s_bias[kMaxBN];

    resolve_slot(job_id, nf);
    if (nf) nf->start(job_id);
    if (threadIdx.x == 0) PB_T(0);
    conv_tile_tma<true, false>(&tmap_w, &tmap_x, &tmap_y, &tmap_r, &tmap_n, a, stages, (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, smem_raw, s_full, s_empty, &s_accum,
                        &s_tmem_base, &s_abort, s_bias, &s_res, s_ready, &s_go, &s_parts, nf != nullptr);
    if (nf) nf->end(job_id);
}

// ---- a pair of blocks on one tile of 256 rows ---------------------------------------------------------------------
// A lone block of 128 rows loads 16 KB of activations and BN x 128 bytes of weights for each k-block, and its tensor core reads both
// from shared memory again: 40 KB each way at 192 columns against 384 clocks of multiplications, where an SM loads 60 bytes a
// clock and its shared memory moves 128.  Here two SMs share a tile of 256 x BN (tcgen05 with cta_group::2): each holds 128 rows of
// operand A and HALF of operand B's columns, so the weights cross each SM's load path and shared memory once for 256 rows.
// Each block loads its own halves; the copies of both count on the barriers of the first (its "full" barriers), whose MMA warp
// issues for the pair and commits to the barriers of both ("empty", "accumulator complete").  Each block has its own rows of
// the accumulator in its tensor memory and finishes them as a lone block does.  Two pairs share a pair of SMs, so one's epilogue
// and barrier latencies lie under the other's multiplications.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_im2col_4d_pair(uint32_t dst, const CUtensorMap* map, int c, int w, int h, int n, uint16_t w_off, uint16_t h_off,
                                                        uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
        ::"r"(dst), "l"(map), "r"(leader_bar), "r"(c), "r"(w), "r"(h), "r"(n), "h"(w_off), "h"(h_off)
        : "memory");
}
__device__ __forceinline__ void tcgen05_mma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier at this offset in both blocks once the pair's multiplications so far are complete.
__device__ __forceinline__ void tcgen05_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}

__global__ void __launch_bounds__(kThreadsTma, 2)
conv_umma_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y,
                      const __grid_constant__ CUtensorMap tmap_r, const ConvArgs a, int stages, uint32_t job_id, FinishedBlockNotifier* nf) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxStages];
    __shared__ __align__(8) uint64_t s_empty[kMaxStages];
    __shared__ __align__(8) uint64_t s_res;
    __shared__ __align__(8) uint64_t s_accum;
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile uint32_t s_abort;
    __shared__ __align__(16) float s_bias[kMaxBN];

    resolve_slot(job_id, nf);
    if (nf) nf->start(job_id);
    const int tid = threadIdx.x;
    const int warp = (int)uniform((uint32_t)tid >> 5);
    const int rank = (int)(blockIdx.x & 1u);                       // in the pair (clusters are two blocks along x)
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t stage_bytes = (uint32_t)kATileBytes + a.b_stage_bytes;      // b_stage_bytes: this block's half
    const int m0 = (int)blockIdx.x * kBM, n0 = (int)blockIdx.y * a.BN, half = a.BN / 2;
    const int nkb = a.nkb;

    if (warp == kWarpB) {
        if (elect_one()) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            for (int s = 0; s < stages; ++s) {
                mbar_init(smem_u32(&s_full[s]), 1);
                mbar_init(smem_u32(&s_empty[s]), 1);
            }
            mbar_init(smem_u32(&s_accum), 1);
            mbar_init(smem_u32(&s_res), 1);
            s_abort = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
    }
    const int cpt = a.Cp / kBK;
    int rem, q0;
    const int img = quotient(m0, a.PQ, a.inv_PQ, rem), p0 = quotient(rem, a.Q, a.inv_Q, q0);
    const int w0 = q0 * a.sw - a.pw, h0 = p0 * a.sh - a.ph;
    if (warp == 4 && elect_one()) asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(a.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();                     // both blocks' barriers and tensor memory are set up
    tcgen05_fence_after();
    const uint32_t tmem_base = uniform(s_tmem_base);

    if (warp < 4) {
        if (warp == kWarpB) {
            // ===== operand B: this block's half of the columns =====
            uint32_t* const err_flag = a.err_flag;
            uint32_t st = 0, parity = 1u;
            for (int kb = 0; kb < nkb; ++kb) {
                if (kb >= stages && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[st]), parity, &s_abort, err_flag, 1u))) break;
                if (elect_one()) {
                    const uint32_t bar = smem_u32(&s_full[st]);
                    if (rank == 0) mbar_arrive_expect_tx(bar, 2u * stage_bytes);       // both blocks' copies
                    tma_load_2d_pair(smem_base + st * stage_bytes + kATileBytes, &tmap_w, kb * kBK, n0 + rank * half, cluster_addr(bar, 0u));
                }
                __syncwarp();
                if (++st == (uint32_t)stages) { st = 0; parity ^= 1u; }
            }
        } else {
            for (int j = tid; j < a.BN; j += 32 * kWarpB) {
                const int k = n0 + j;
                s_bias[j] = (a.bias && k < a.K) ? __ldg(a.bias + k) : 0.f;
            }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        griddep_wait();
        griddep_launch();
        epilogue<true>(a, tmem_base, true, m0, n0, s_bias, &s_accum, &s_abort, 0u, a.out_box ? &tmap_y : nullptr, smem_base, &s_res, nf != nullptr);
    } else if (warp == 4) {
        // ===== operand A: this block's 128 rows =====
        griddep_wait();
        uint32_t* const err_flag = a.err_flag;
        uint32_t st = 0, parity = 1u;
        int tap_r = 0, tap_s = 0, chunk = 0;
        for (int kb = 0; kb < nkb; ++kb) {
            if (kb >= stages && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[st]), parity, &s_abort, err_flag, 1u))) break;
            if (elect_one()) {
                const uint32_t a_tile = smem_base + st * stage_bytes, bar = cluster_addr(smem_u32(&s_full[st]), 0u);
                if (a.a_tiled) tma_load_2d_pair(a_tile, &tmap_x, chunk * kBK, m0, bar);
                else tma_load_im2col_4d_pair(a_tile, &tmap_x, chunk * kBK, w0, h0, img, (uint16_t)(tap_s * a.dw), (uint16_t)(tap_r * a.dh), bar);
            }
            __syncwarp();
            if (++chunk == cpt) {
                chunk = 0;
                if (++tap_s == a.S) { tap_s = 0; ++tap_r; }
            }
            if (++st == (uint32_t)stages) { st = 0; parity ^= 1u; }
        }
        if (a.residual && a.out_box) {      // as in conv_tile_tma
            const uint32_t bytes = (uint32_t)a.BN * 256u;
            bool ok = true;
            for (uint32_t q = 0; q * stage_bytes < bytes && ok; ++q) {
                const int uses = q < (uint32_t)stages && nkb > (int)q ? (nkb - (int)q + stages - 1) / stages : 0;
                if (uses > 0) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[q]), (uint32_t)(uses - 1) & 1u, &s_abort, err_flag, 1u));
            }
            if (ok && elect_one()) {
                mbar_arrive_expect_tx(smem_u32(&s_res), bytes);
                for (int c = 0; c < a.BN; c += a.out_box) tma_load_2d(smem_base + (uint32_t)c * 256u, &tmap_r, n0 + c, m0, smem_u32(&s_res));
            }
            __syncwarp();
        }
        griddep_launch();
    } else if (rank == 0) {
        // ===== the pair's multiplications =====
        uint32_t st = 0, parity = 0u;
        bool ok = true;
        uint32_t* const err_flag = a.err_flag;
        const uint32_t idesc = uniform(a.idesc), n_kb = uniform((uint32_t)nkb), n_st = uniform((uint32_t)stages);
        const uint64_t desc_a0 = umma_desc_sw128(uniform(smem_base)), desc_b0 = umma_desc_sw128(uniform(smem_base) + kATileBytes);
        const uint32_t desc_step = uniform(stage_bytes) >> 4;
        // The last channels of a tap may fill less than a k-block: what is past them are zeros, which need no multiplying (288 -> 384 channels
        // 3x3 on 64 maps of 35 x 35 150.9 -> 144.5 us; in conv_tile_tma, whose launches the tensor pipe does not bound, the choice costs more than it
        // saves: ResNet-50 x 8 images 347 -> 352).
        const uint32_t n_cpt = uniform((uint32_t)cpt), last_slices = uniform((uint32_t)(a.Cs - (cpt - 1) * kBK + 15) >> 4);
        uint32_t chunk_k = 0;
        for (uint32_t kb = 0; kb < n_kb; ++kb) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[st]), parity, &s_abort, err_flag, 2u));
            if (!ok) break;
            tcgen05_fence_after();
            const uint64_t da = desc_a0 + st * desc_step, db = desc_b0 + st * desc_step;
            uint32_t slices = kBK / 16;
            if (++chunk_k == n_cpt) { chunk_k = 0; slices = last_slices; }
            if (elect_one()) {
#pragma unroll
                for (uint32_t k = 0; k < kBK / 16; ++k)
                    if (k < slices) tcgen05_mma_bf16_pair(tmem_base, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                tcgen05_commit_pair(smem_u32(&s_empty[st]));
            }
            __syncwarp();
            if (++st == n_st) { st = 0; parity ^= 1u; }
        }
        if (ok && elect_one()) tcgen05_commit_pair(smem_u32(&s_accum));
        __syncwarp();
        griddep_launch();
    } else {
        griddep_launch();
    }

    tcgen05_fence_before();
    __syncthreads();
    if (s_abort) {
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t i = 0; i < (1u << 20); ++i) {
            if (globaltimer_ns() - t0 > 50000ull) break;
        }
    }
    cluster_arrive();
    cluster_wait();                     // neither block's memory goes before both have finished
    if (warp == 5) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(a.tmem_cols) : "memory");
    }
    if (nf) nf->end(job_id);
}

// Grouped launch: several independent convolutions (the parallel branches of an Inception block at the
// same depth, a ResNet block's shortcut beside its first convolution) in ONE grid.  Kernel-level
// concurrency on a GPU is capped by its hardware queues, and a batch-1 convolution rarely has more
// than a dozen tiles, so running the branches side by side in one launch is what fills the SMs.
// Block b belongs to the sub-problem i with first_block[i] <= b < first_block[i + 1]; the table with
// each sub-problem's tensor maps and arguments lives in device memory, written once per instance.
// A 3x3 pooling layer of the same dependence depth can ride along as one more entry (stages == kSubPool): its blocks
// run pool_sub_block() instead of a convolution tile.  Why it was tried: under serving load every launch of a request's
// chain waits about 45 us for SM resources behind the other requests' CTAs, whatever its own size, so the 13 pooling
// launches of an Inception-v3 request cost 20 % of the throughput although they are 6 % of a lone request's time.
// What came of it: see PB_FUSE_POOLS where the launches are planned (off by default).
struct PoolSubArgs {
    const __nv_bfloat16* x;
    __nv_bfloat16* y;
    int C, H, W, Cs, P, Q, Ks, out_c_off;
    int sh, sw, ph, pw;
    int is_max, count_pad, batch, reserved;
};
struct alignas(128) SubConv {
    CUtensorMap tmap_w;
    CUtensorMap tmap_x;
    CUtensorMap tmap_y;
    CUtensorMap tmap_r;
    union {
        ConvArgs a;
        PoolSubArgs pool;
    };
    uint32_t first_block, gx, gy, stages;
    float inv_gx;
};
static_assert(sizeof(PoolSubArgs) <= sizeof(ConvArgs), "a pooling entry fits where a convolution's arguments are");
constexpr int kMaxSubConvs = 8;
struct SubStarts { uint32_t first[kMaxSubConvs]; };      // first block of each entry; past the last entry, of none
constexpr uint32_t kSubPool = 0xffffffffu;
constexpr int kPoolVecsPerThread = 2;                 // output vectors (8 channels) per thread of a pooling block

// One block's share of a 3x3 pooling layer: thread t takes output vectors base + t and base + 192 + t.  All nine
// loads of a window are issued before the first use (addresses clamped into the tensor, taps outside dropped
// afterwards).  Arithmetic and its order are those of pool_kernel / window3_strip_kernel (the columns of a row, then the rows, fp32
// sums from +0, IEEE division; fmaxf from -inf), so the bits are theirs.
__device__ __forceinline__ void pool_sub_block(const PoolSubArgs& a, uint32_t local_block) {
    const int cv = a.Cs >> 3;
    const long long total = (long long)a.batch * a.P * a.Q * cv;
    const long long base = (long long)local_block * (kThreadsTma * kPoolVecsPerThread) + threadIdx.x;
#pragma unroll 1
    for (int u = 0; u < kPoolVecsPerThread; ++u) {
        const long long idx = base + (long long)u * kThreadsTma;
        if (idx >= total) break;
        const int c0 = (int)(idx % cv) * 8;
        long long pix = idx / cv;
        const int q = (int)(pix % a.Q);
        pix /= a.Q;
        const int p = (int)(pix % a.P), img = (int)(pix / a.P);
        const __nv_bfloat16* x = a.x + (size_t)img * a.H * a.W * a.Cs + c0;
        uint4 raw[3][3];
        uint32_t ok = 0;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int ih = p * a.sh + r - a.ph;
            const bool row_ok = ih >= 0 && ih < a.H;
            const __nv_bfloat16* xrow = x + (size_t)min(max(ih, 0), a.H - 1) * a.W * a.Cs;
#pragma unroll
            for (int s2 = 0; s2 < 3; ++s2) {
                const int iw = q * a.sw + s2 - a.pw;
                if (row_ok && iw >= 0 && iw < a.W) ok |= 1u << (r * 3 + s2);
                raw[r][s2] = *reinterpret_cast<const uint4*>(xrow + (size_t)min(max(iw, 0), a.W - 1) * a.Cs);
            }
        }
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = a.is_max ? -INFINITY : 0.f;
        int cnt = 0;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            float row[8];                     // sums: the columns of a row first, as in the pooling kernels
#pragma unroll
            for (int j = 0; j < 8; ++j) row[j] = 0.f;
#pragma unroll
            for (int s2 = 0; s2 < 3; ++s2) {
                if (!((ok >> (r * 3 + s2)) & 1u)) continue;
                const uint32_t w[4] = {raw[r][s2].x, raw[r][s2].y, raw[r][s2].z, raw[r][s2].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xffff0000u);
                    if (a.is_max) {
                        acc[2 * j] = fmaxf(acc[2 * j], lo);
                        acc[2 * j + 1] = fmaxf(acc[2 * j + 1], hi);
                    } else {
                        row[2 * j] += lo;
                        row[2 * j + 1] += hi;
                    }
                }
                ++cnt;
            }
            if (!a.is_max) {
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] += row[j];
            }
        }
        const float div = a.count_pad ? 9.f : (float)(cnt > 0 ? cnt : 1);
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v0 = a.is_max ? acc[2 * j] : acc[2 * j] / div, v1 = a.is_max ? acc[2 * j + 1] : acc[2 * j + 1] / div;
            if (c0 + 2 * j >= a.C) v0 = 0.f;
            if (c0 + 2 * j + 1 >= a.C) v1 = 0.f;
            const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
            o[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        __nv_bfloat16* y = a.y + (((size_t)img * a.P + p) * a.Q + q) * a.Ks + a.out_c_off + c0;
        *reinterpret_cast<uint4*>(y) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

__global__ void __launch_bounds__(kThreadsTma, 3)
conv_umma_multi_kernel(const SubConv* __restrict__ table, const SubStarts starts, uint32_t job_id, FinishedBlockNotifier* nf) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxStages];
    __shared__ __align__(8) uint64_t s_empty[kMaxStages];
    __shared__ __align__(8) uint64_t s_res;
    __shared__ __align__(8) uint64_t s_accum;
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile uint32_t s_abort;
    __shared__ __align__(16) float s_bias[kMaxBN];
    __shared__ __align__(8) uint64_t s_go;
    __shared__ __align__(8) uint64_t s_parts;
    __shared__ __align__(16) ConvArgs s_args;

    resolve_slot(job_id, nf);
    if (nf) nf->start(job_id);
    if (threadIdx.x == 0) PB_T(0);

    // Which sub-problem: its first block is in the constant bank (looked up in the table it took a chain of up to seven loads from L2).
    int sub = 0;
    uint32_t first = 0;
#pragma unroll
    for (int i = 1; i < kMaxSubConvs; ++i)
        if (blockIdx.x >= starts.first[i]) { sub = i; first = starts.first[i]; }
    const SubConv* sc = table + sub;
    const uint32_t gx = __ldg(&sc->gx), stages = __ldg(&sc->stages);
    const float inv_gx = __ldg(&sc->inv_gx);
    // the table is constant for the life of the instance: it may be read before griddepcontrol.wait
    static_assert(sizeof(ConvArgs) % 4 == 0, "ConvArgs is copied word by word");
    if (threadIdx.x < sizeof(ConvArgs) / 4)
        reinterpret_cast<uint32_t*>(&s_args)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&sc->a)[threadIdx.x];
    __syncthreads();
    const uint32_t local = blockIdx.x - first;
    if (stages == kSubPool) {        // a pooling layer riding along: no tensor memory, no pipeline
        griddep_wait();
        griddep_launch();
        pool_sub_block(*reinterpret_cast<const PoolSubArgs*>(&s_args), local);
        if (nf) nf->end(job_id);
        return;
    }
    // the ranks of a cluster are consecutive blocks (every sub-problem of a launch has the same split)
    const uint32_t S = (uint32_t)s_args.splits, tile = local >> log2_of((int)S), bz = local & (S - 1u);
    int bx;
    const int by = quotient((int)tile, (int)gx, inv_gx, bx);
    conv_tile_tma<false, false>(&sc->tmap_w, &sc->tmap_x, &sc->tmap_y, &sc->tmap_r, nullptr, s_args, (int)stages, bx, by, (int)bz, smem_raw, s_full, s_empty, &s_accum,
                  &s_tmem_base, &s_abort, s_bias, &s_res, nullptr, &s_go, &s_parts, nf != nullptr);
    if (nf) nf->end(job_id);
}


// ---- persistent form: a CTA walks several tiles ------------------------------------------------------------
// What a one-tile CTA costs besides its main loop was measured under serving load (cycle stamps summed over all
// CTAs): 1.0 us of set-up, 1.4 us until the first operands land, 0.2 us of accumulator drain, 1.4 us of epilogue,
// 0.35 us of tear-down and about 1 us before the SM slot holds the next CTA, against 4.7 us of main loop; and the
// GPU's throughput on these layers is what its CTA slots turn over.  Here a CTA is given several tiles of the
// launch (tile t = blockIdx.x, + gridDim.x, ...) and pays set-up and tear-down once; the producers run on
// into the next tile's k-blocks while the current tile finishes, so operand latency is paid once per CTA; and
// there are TWO accumulators in tensor memory, so the epilogue of tile i (warps 0-3) runs under the MMAs of tile
// i + 1 (warp 4).  9 warps: 0-3 epilogue, 4 TMEM allocation + MMA issue, 5-8 producers (a thread that issues
// tensor copies back to back sustains only one copy per ~500 clocks - ~170 for the wait on the stage's barrier,
// ~250 for the copy instruction itself - so the 2 x stages (stage, operand) pairs are dealt to four threads; a
// pair is always refilled by the same thread).  Sized for two CTAs per SM: <= 108 KB of pipeline, 288 threads
// of <= 112 registers, 2 x 128 tensor-memory columns.
// Every tile comes from the launch's table of sub-problems (one entry for a lone convolution, several for the
// independent convolutions of a grouped launch): tile index -> entry by first_block, then (m tile, n tile)
// inside it.  It never splits a reduction.
constexpr int kPersistProducers = 4;
constexpr int kThreadsPersist = 32 * (5 + kPersistProducers);
#ifndef PB_CONV_PERSIST_SMEM_KB
#define PB_CONV_PERSIST_SMEM_KB 108
#endif
constexpr uint32_t kSmemBudgetPersist = PB_CONV_PERSIST_SMEM_KB * 1024u;

// A sub-problem's arguments as the CTA keeps them in shared memory (the tensor maps stay in global memory,
// where the TMA unit reads them): decoding a tile and reading its arguments from the global table cost every
// role a chain of dependent loads at each tile boundary, about 5 us per tile.
struct SubArgs {
    ConvArgs a;
    uint32_t first_block, gx, gy, pad;
};
struct TileRef {
    const SubArgs* sa;
    const SubConv* sc;
    int bx, by;
};
__device__ __forceinline__ TileRef tile_ref(const SubConv* __restrict__ table, const SubArgs* s_sub, int n_sub, uint32_t t) {
    int sub = 0;
    while (sub + 1 < n_sub && t >= s_sub[sub + 1].first_block) ++sub;
    TileRef r;
    r.sa = s_sub + sub;
    r.sc = table + sub;
    const uint32_t local = t - r.sa->first_block;
    const uint32_t gx = r.sa->gx;
    r.by = (int)(local / gx);
    r.bx = (int)(local - (uint32_t)r.by * gx);
    return r;
}

__global__ void __launch_bounds__(kThreadsPersist, 2)
conv_umma_persist_kernel(const SubConv* __restrict__ table, int n_sub, uint32_t total_tiles, int stages, uint32_t stage_bytes,
                         uint32_t acc_cols, uint32_t job_id, FinishedBlockNotifier* nf) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t s_full[kMaxStages];
    __shared__ __align__(8) uint64_t s_empty[kMaxStages];
    __shared__ __align__(8) uint64_t s_tfull[2];       // accumulator complete (tcgen05.commit)
    __shared__ __align__(8) uint64_t s_tempty[2];      // accumulator read out (one arrival per epilogue warp)
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile uint32_t s_abort;
    __shared__ __align__(16) float s_bias[2][kMaxBN];
    __shared__ __align__(16) SubArgs s_sub[kMaxSubConvs];

    resolve_slot(job_id, nf);
    if (nf) nf->start(job_id);

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
#ifdef PB_CONV_STATS
    __shared__ long long s_cta_t0;
    if (tid == 0) {
        const unsigned others = atomicAdd(&g_persist_resident, 1u);
        atomicAdd(&g_persist_hist[others / 32u < 14u ? others / 32u : 14u], 1ull);
        s_cta_t0 = clock64();
    }
#endif

    // the table is constant for the life of the instance: it may be read before griddepcontrol.wait
    {
        static_assert(sizeof(ConvArgs) % 4 == 0 && sizeof(SubArgs) % 4 == 0, "copied word by word");
        constexpr int kWords = (int)(sizeof(ConvArgs) / 4);
        for (int j = tid; j < n_sub * (kWords + 3); j += kThreadsPersist) {
            const int sub = j / (kWords + 3), w = j - sub * (kWords + 3);
            if (w < kWords) reinterpret_cast<uint32_t*>(&s_sub[sub].a)[w] = reinterpret_cast<const uint32_t*>(&table[sub].a)[w];
            else (&s_sub[sub].first_block)[w - kWords] = (&table[sub].first_block)[w - kWords];
        }
    }

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(smem_u32(&s_full[s]), 1);
            mbar_init(smem_u32(&s_empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&s_tfull[b]), 1);
            mbar_init(smem_u32(&s_tempty[b]), 4);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        tcgen05_alloc(smem_u32(&s_tmem_base), 2u * acc_cols);
        tcgen05_relinquish();
    }
    // the first tile's descriptors: their fetch into the descriptor cache overlaps the rest of the set-up
    if (warp >= 5 && warp <= 6 && lane == 0) {
        int sub = 0;
        while (sub + 1 < n_sub && blockIdx.x >= table[sub + 1].first_block) ++sub;
        asm volatile("prefetch.tensormap [%0];" ::"l"(warp == 5 ? &table[sub].tmap_x : &table[sub].tmap_w) : "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    // Nothing above touched activations, the output or the split-K workspace: it may overlap the previous
    // kernel's tail.  From here on this kernel reads what the previous one wrote.
    griddep_wait();

    if (warp < 4) {
        // ===== epilogue warps: thread t owns accumulator lane t = tile row t =====
        uint32_t i = 0;
        for (uint32_t t = blockIdx.x; t < total_tiles; t += gridDim.x, ++i) {
            const uint32_t acc = i & 1u, use = i >> 1;
            const TileRef tr = tile_ref(table, s_sub, n_sub, t);
            const ConvArgs& a = tr.sa->a;
            // the tile's biases, staged by these four warps for themselves
            asm volatile("bar.sync 1, 128;" ::: "memory");      // the tile that used this buffer before is done with it
            const int n0 = tr.by * a.BN;
            for (int j = tid; j < a.BN; j += 128) {
                const int k = n0 + j;
                s_bias[acc][j] = (a.bias && k < a.K) ? __ldg(a.bias + k) : 0.f;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (tid == 0) PB_PT(i, 2);
            epilogue<false>(epi_args(a), tmem_base + acc * acc_cols, true, tr.bx * kBM, n0, s_bias[acc], &s_tfull[acc], &s_abort, use & 1u);
            if (tid == 0) PB_PT(i, 3);
            // this accumulator may be overwritten: every tcgen05.ld of the warp has completed (wait::ld)
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_tempty[acc]));
        }
    } else if (warp == 4) {
        // ===== MMA issuer: one thread =====
        // The thread's own instruction chain per k-block decides the pace of the CTA (measured: four MMA issues +
        // commit 360 clocks, most of it the tensor cores taking the instructions; then 415 clocks until the next
        // k-block's barrier had been looked at: a division for the stage index, a load of the error-flag pointer, and
        // an mbarrier wait that costs ~170 clocks even when the phase is long complete).  So: stage and parity are
        // carried, not divided; and the NEXT k-block's barrier is probed (test_wait, never blocks) before this
        // k-block's MMAs are issued, so the probe's latency runs under them.
        if (lane == 0) {
            uint32_t i = 0;                         // tiles of this CTA so far
            uint32_t st = 0, parity = 0;            // pipeline stage and phase of the next k-block
            bool ok = true;
            uint32_t* const err_flag = s_sub[0].a.err_flag;
            // descriptors of stage 0; stage q is stage_bytes further on (the address field counts 16-byte units and
            // cannot carry out of its 14 bits: shared memory ends below 256 KB)
            const uint64_t desc_a0 = umma_desc_sw128(smem_base), desc_b0 = umma_desc_sw128(smem_base + kATileBytes);
            const uint64_t desc_step = (uint64_t)(stage_bytes >> 4);
            bool have_next = false;                 // the barrier of (st, parity) is already known to be complete
            for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++i) {
                const uint32_t acc = i & 1u, use = i >> 1;
                const TileRef tr = tile_ref(table, s_sub, n_sub, t);
                const ConvArgs& a = tr.sa->a;
                const int nkb = a.nkb;
                const uint32_t idesc = a.idesc;
#ifdef PB_CONV_STATS
                const bool first_tile = i == 0;
#endif
                ok = mbar_wait(smem_u32(&s_tempty[acc]), (use & 1u) ^ 1u, &s_abort, err_flag, 4u);
                if (!ok) break;
                PB_PT(i, 0);
                tcgen05_fence_after();
                const uint32_t d_tmem = tmem_base + acc * acc_cols;
                for (int kb = 0; kb < nkb; ++kb) {
                    if (!have_next) {
                        ok = mbar_wait(smem_u32(&s_full[st]), parity, &s_abort, err_flag, 2u);
                        if (!ok) break;
                    }
                    PB_PK(kb, 4);
                    tcgen05_fence_after();
                    // stage of the k-block after this one (of this tile or of the CTA's next tile: the pipeline runs on)
                    uint32_t st_n = st + 1, parity_n = parity;
                    if (st_n == (uint32_t)stages) { st_n = 0; parity_n ^= 1u; }
                    have_next = mbar_test_wait(smem_u32(&s_full[st_n]), parity_n);
                    const uint64_t da = desc_a0 + (uint64_t)st * desc_step, db = desc_b0 + (uint64_t)st * desc_step;
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k)
                        tcgen05_mma_bf16(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb > 0 || k > 0) ? 1u : 0u);   // +32 bytes per K=16 slice
                    tcgen05_commit(smem_u32(&s_empty[st]));
                    PB_PK(kb, 5);
                    st = st_n;
                    parity = parity_n;
                }
                if (ok) tcgen05_commit(smem_u32(&s_tfull[acc]));
                PB_PT(i, 1);
            }
        }
        __syncwarp();
    } else {
        // ===== producers: lane 0 of warps 5-8 =====
        if (lane == 0) {
            const uint32_t prod = (uint32_t)(warp - 5);
            // which (stage, operand) pairs are this thread's: bit st of mask_a / mask_b (no division in the loop)
            uint32_t mask_a = 0, mask_b = 0;
            for (int q = 0; q < stages; ++q) {
                if ((uint32_t)(q * 2) % kPersistProducers == prod) mask_a |= 1u << q;
                if ((uint32_t)(q * 2 + 1) % kPersistProducers == prod) mask_b |= 1u << q;
            }
            uint32_t st = 0, parity = 1u;           // a fresh barrier passes a wait on the "previous" phase
            bool ok = true;
            uint32_t* const err_flag = s_sub[0].a.err_flag;
            for (uint32_t t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
#ifdef PB_CONV_STATS
                const bool first_tile = t == blockIdx.x;
#endif
                const TileRef tr = tile_ref(table, s_sub, n_sub, t);
                const ConvArgs& a = tr.sa->a;
                const CUtensorMap* tmap_w = &tr.sc->tmap_w;
                const CUtensorMap* tmap_x = &tr.sc->tmap_x;
                const int nkb = a.nkb;
                const int m0 = tr.bx * kBM, n0 = tr.by * a.BN;
                const int PQ = a.PQ, Q = a.Q;
                const int img = m0 / PQ, rem = m0 - img * PQ;
                const int p0 = rem / Q, q0 = rem - p0 * Q;
                const int w0 = q0 * a.sw - a.pw, h0 = p0 * a.sh - a.ph;
                const int cpt = a.Cp / kBK, S = a.S, dw = a.dw, dh = a.dh, a_tiled = a.a_tiled;
                const uint32_t tx_bytes = (uint32_t)kATileBytes + a.b_stage_bytes;
                // filter tap (r, s2) and channel chunk of the k-block, carried along
                int chunk = 0, r = 0, s2 = 0;
                if (prod == 0) PB_PT((t - blockIdx.x) / gridDim.x, 4);
                for (int kb = 0; kb < nkb; ++kb) {
                    const bool mine_a = (mask_a >> st) & 1u, mine_b = (mask_b >> st) & 1u;
                    if (mine_a || mine_b) {
                        if (mine_a) PB_PK(kb, 0);
                        if (mine_b) PB_PK(kb, 2);
                        ok = mbar_wait(smem_u32(&s_empty[st]), parity, &s_abort, err_flag, 1u);
                        if (!ok) break;
                        const uint32_t a_tile = smem_base + st * stage_bytes;
                        const uint32_t bar = smem_u32(&s_full[st]);
                        if (mine_a) {
                            mbar_arrive_expect_tx(bar, tx_bytes);
                            if (a_tiled) tma_load_2d(a_tile, tmap_x, chunk * kBK, m0, bar);
                            else tma_load_im2col_4d(a_tile, tmap_x, chunk * kBK, w0, h0, img, (uint16_t)(s2 * dw), (uint16_t)(r * dh), bar);
                            PB_PK(kb, 1);
                        }
                        if (mine_b) { tma_load_2d(a_tile + kATileBytes, tmap_w, kb * kBK, n0, bar); PB_PK(kb, 3); }
                    }
                    if (++chunk == cpt) {
                        chunk = 0;
                        if (++s2 == S) { s2 = 0; ++r; }
                    }
                    if (++st == (uint32_t)stages) { st = 0; parity ^= 1u; }
                }
            }
        }
        __syncwarp();
    }

    // the next kernel's blocks may take SM slots from here on: this CTA is about to leave
    griddep_launch();
    tcgen05_fence_before();
    __syncthreads();
    if (s_abort) {
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t i = 0; i < (1u << 20); ++i) {
            if (globaltimer_ns() - t0 > 50000ull) break;
        }
        __syncthreads();
    }
    if (warp == 4) {
        tcgen05_fence_after();
        tcgen05_dealloc(tmem_base, 2u * acc_cols);
    }
#ifdef PB_CONV_STATS
    if (tid == 0) {
        atomicSub(&g_persist_resident, 1u);
        atomicAdd(&g_persist_hist[15], (unsigned long long)(clock64() - s_cta_t0));
    }
#endif
    if (nf) nf->end(job_id);
}

// ---- host side ----------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
        else
            cudaGetLastError();
    });
    return fn;
}

typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const int*, const int*, cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeIm2colFn encode_im2col_fn() {
    static EncodeIm2colFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeIm2colFn)p;
        else
            cudaGetLastError();
    });
    return fn;
}

// Operand A by im2col TMA unless PB_CONV_GATHER=1 asks for the cp.async gather kernel.
bool use_tma_a() {
    static const bool v = [] {
        const char* e = getenv("PB_CONV_GATHER");
        return !(e && e[0] == '1');
    }();
    return v;
}

// Widest output-channel tile: 256 (PB_CONV_MAX_BN=128 caps it; the gather kernel takes 128).
int bn_limit() {
    static const int fixed = [] {
        const char* e = getenv("PB_CONV_MAX_BN");
        return e && atoi(e) < 256 ? 128 : 256;
    }();
    return use_tma_a() ? fixed : 128;
}

// PB_CONV_PERSIST=1: model launches run the persistent kernel (a CTA walks several tiles).  Off by default.
// Measured on B200 with 3 tiles per CTA: a lone Inception-v3 request 342 -> 1119 us (266 with the one-tile kernel today), the mix MNIST : Inception-v3 = 9 : 1 in a closed
// loop of 192 clients 317 -> 166 thousand requests a second.  It has not followed the one-tile kernel: no split reductions, no
// stores through TMA, multiplications and copies issued under `lane == 0` (390 clocks a k-block), and the tiles it walks are cut
// for one tile per CTA.  (Against the one-tile kernel of its time it had a lone request at 604 us instead of 723.)
bool persist_enabled() {
    const char* e = getenv("PB_CONV_PERSIST");      // read at every use: a model keeps what it was loaded with
    return e && e[0] == '1' && use_tma_a();
}
// Tiles a persistent CTA is given (PB_CONV_TILES_PER_CTA): more tiles per CTA spread the per-CTA costs thinner
// and leave SM slots to the other requests in flight; fewer tiles per CTA finish a lone launch sooner.
int tiles_per_cta() {
    const char* e = getenv("PB_CONV_TILES_PER_CTA");      // read at every use: a model instance keeps what it was built with
    const int n = e ? atoi(e) : 3;
    return n < 1 ? 1 : (n > 64 ? 64 : n);
}

// How reluctant a launch is to split its reduction, in the unit of pb_set_conv_split_gain_us (see choose_tiling, which asks
// for a 60th of it; above 1e6 nothing splits).  PB_CONV_SPLIT_GAIN_US or the function override the default of 6.
std::atomic<double> g_split_gain_us{-1.0};      // < 0: not set yet, take PB_CONV_SPLIT_GAIN_US or the default
}  // namespace

double conv_split_gain_us() {
    double v = g_split_gain_us.load(std::memory_order_relaxed);
    if (v < 0) {
        const char* e = getenv("PB_CONV_SPLIT_GAIN_US");
        v = e ? atof(e) : 6.0;
        if (v < 0) v = 0;
        g_split_gain_us.store(v, std::memory_order_relaxed);
    }
    return v;
}

namespace {

int batch_of(const pb_op_params* p) { return p->batch > 1 ? p->batch : 1; }
int dil_h(const pb_op_params* p) { return p->dil_h > 1 ? p->dil_h : 1; }
int dil_w(const pb_op_params* p) { return p->dil_w > 1 ? p->dil_w : 1; }

struct Geometry {
    int cpt, Cp;                // 64-channel k-blocks per filter tap; Cp = cpt * 64
    int Kdim_pad, nkb;          // k = tap * Cp + c
    int Kp16, n_tiles, BN;
    int m_tiles;
    int stages;                 // pipeline buffers
    int splits;                 // blocks (one cluster) per tile
    bool pair;                  // two blocks on a tile of 256 rows
    int out_box;                // ConvArgs::out_box
    uint32_t tmem_cols, b_stage_bytes, smem_bytes, idesc;
    uint32_t meet;              // ConvArgs::meet
};

// Rows of the packed weight matrix: the layout does not depend on how a launch tiles it (a box that reaches past
// the last row reads zeros).
int packed_rows(const pb_op_params* p) {
    const int Kp16 = round_up(p->K, 16), n = ceil_div(Kp16, 128);
    return n * round_up(ceil_div(Kp16, n), 16);
}

// What the tiling of a launch of m_tiles x 128 rows depends on.
struct ConvShape {
    int m_tiles, Kp16, nkb;
    bool residual, shared;      // shared: other requests use the GPU too
};

// Pipeline depth: as many stages as the k-loop can use and the shared-memory budget holds.  On a GPU it has to itself a
// launch of up to two blocks per SM gets a deeper pipeline (a refill takes about 1.1 us; 36 k-blocks of 64 columns: 13.6 us
// at 73 KB, 12.3 at 110, 11.7 at 150, where the next launch's blocks no longer fit beside it: Inception-v3 402 us
// instead of 346).
// Where the other ranks' parts of a split tile arrive: beside the pipeline where that leaves it three stages (or as many as there are
// k-blocks) - and, over more than 20 k-blocks on a GPU of its own, as many as it would have without: a stage less costs each of them 15 ns, the message that says the
// buffers are free 0.17 us (256 -> 72 channels 5x5, stride 2, on 16 maps of 56 x 56, two ranks of 50 k-blocks: 20.5 us with three stages, 19.3 with four;
// 18 k-blocks on two ranks 10.3 and 11.1) - else in its buffers.
struct Pipeline { int stages; uint32_t meet, bytes; };        // meet: offset of that place, 0 = in the buffers
Pipeline pipeline(int ctas, int BN, int k_blocks, int splits, bool shared) {
    const int budget = (int)(!shared && ctas <= 296 ? kSmemBudgetDeep : kSmemBudgetTma) - 1024, stage = (int)kATileBytes + BN * 128;
    const int parts = splits > 1 ? (BN - BN / splits) * 512 : 0, most = std::min(kMaxStages, k_blocks);
    const int beside = (budget - parts) / stage;
    if (parts && beside >= std::max(2, std::min(3, k_blocks)) && (shared || k_blocks <= 20 || beside >= std::min(most, budget / stage))) {
        const int stages = std::max(2, std::min(most, beside));
        return {stages, (uint32_t)(stages * stage), (uint32_t)(stages * stage + parts)};
    }
    const int stages = std::max(2, std::min(most, budget / stage));
    return {stages, 0u, (uint32_t)std::max(stages * stage, parts)};
}

// Modelled microseconds of a lone launch inside a stage graph, fitted to 3372 measured (layer shape, tile width, split, way
// out) combinations on B200 - chains of equal layers of 7x7 to 149x149 maps, 32 to 2048 channels, 1x1 and 3x3, 1 to 8 images,
// with and without a residual, either pipeline budget:
//   a launch costs 3.7 us outside its k-loop and epilogue (operand latency, accumulator drain, hand-over to the next launch);
//   a k-block costs the issue of its copies (0.2 us), its share of a refill's latency, or its bytes at 137 KB/us per SM,
//   shared by the blocks of the SM (between the mean and the fullest one);
//   the epilogue costs 11 ns per column of a block with direct stores (24 with a residual), 8 through TMA;
//   a cluster costs 21 ns per column that a rank sends, 4 / 4 / 6 ns of placement per block at 2 / 4 / 8 ranks, and a message to and fro
//   where the parts land in the pipeline's buffers (fitted to 912 combinations of 66 shapes, launches with st.async; the tiles it
//   picks for the shapes take 391.5 us in all, the best measured 386.8).
// On a GPU that other requests share, the costs that a cluster had with barriers and pulled parts stay: with these, clusters win where
// lone blocks serve the mixes better (192 requests of MNIST : Inception-v3 = 9 : 1 1144 and 1195 us, 64 of MobileNet and ResNet-50 1633 and 1679).
// Its mean error there is 3 %, and what it picks is within 1.5 % of the best measured tiles summed over the layers of a network.
// A layer repeated 40 times in one graph, all launches alike, takes 1.8 us less than modelled (0.3 us spread over 19 layers of 7x7 to
// 56x56 maps, 1 and 8 images); the tiles picked for those 19 take 91.6 us in all, the best of 6 to 33 measured for each 90.4.
// (Before, the model knew neither the stores' path nor the residual, and a width of 80 or 176 columns, which TMA cannot
// store, cost a 14 x 14 layer of 256 -> 1024 channels 8.8 us instead of 6.4 alone and 3.1 instead of 1.7 under load.)
int tiling_ctas(const ConvShape& c, const ConvTiling& t) { return c.m_tiles * ceil_div(c.Kp16, t.BN) * t.splits; }
double tiling_us(int ctas, const ConvShape& c, const ConvTiling& t) {
    const int k_blocks = ceil_div(c.nkb, t.splits);
    const Pipeline pipe = pipeline(ctas, t.BN, k_blocks, t.splits, c.shared);
    const int stages = pipe.stages;
    const double mean = std::max(1.0, ctas / 148.0), per_sm = mean + 0.639 * (ceil_div(ctas, 148) - mean);
    const double crowd = 1.0 + 1.39 * (per_sm - 1.0);
    double kb = std::max(0.197 + 0.0003 * t.BN, per_sm * (16.384 + 0.128 * t.BN) / 137.0);
    if (k_blocks > stages) kb = std::max(kb, (0.452 + 0.0015 * t.BN) / stages);
    double us = 3.68 + k_blocks * kb;
    if (t.tma) us += 0.164 + 0.0081 * t.BN * crowd + (c.residual ? 0.327 + 0.0006 * t.BN * crowd : 0.0);
    else us += (c.residual ? 0.0242 : 0.0114) * t.BN / t.splits * crowd;
    if (t.splits > 1) {
        if (c.shared) us += 0.401 + 0.017 * t.BN + ctas * (t.splits == 2 ? 0.0023 : t.splits == 4 ? 0.0055 : 0.0133);
        else us += 0.021 * (t.BN - t.BN / t.splits) + ctas * (t.splits == 2 ? 0.0044 : t.splits == 4 ? 0.0042 : 0.0062) + (pipe.meet ? 0.0 : 0.17);
    }
    return us;
}
// Relative length of a block's stay on its SM.
double tiling_stay(const ConvShape& c, const ConvTiling& t) {
    const double column = (t.tma ? 0.012 : 0.0192) * (c.residual ? 1.5 : 1.0);
    return 1.5 + 0.12 * ceil_div(c.nkb, t.splits) + column * t.BN + (t.splits > 1 ? 1.0 : 0.0);
}

// Tile width (output channels), split and way out of a launch: the combination with the least modelled time, plus a charge
// for the block slots it takes (444 = 148 SMs x 3): on a GPU that other requests share, what counts is not when a launch
// ends but what it occupies.  Measured, charge -> 192 requests of MNIST : Inception-v3 = 9 : 1 at once, us / 32 of ResNet-18 /
// 64 of MobileNet and ResNet-50 / the first mix in a closed loop of 192 clients, thousand requests a second: 6 -> 1309 / 848 /
// 1679 / 300, 9 -> 1270 / 849 / 1688 / 305, 13 -> 1276 / 845 / 1742 / 317, 16 -> 1243 / 821 / 1730 / 318, 20 -> - / - / - / 312.
// A chain that has the GPU to itself, ResNet-50 x 8 images / Inception-v3 x 8 / ResNet-18 x 8: 0 -> 397 / 405 / 163 us,
// 0.5 -> 399 / 402 / 164, 1 -> 401 / 404 / 164.
ConvTiling best_tiling(const ConvShape& c, int bn_max, int want_splits, double gain_us) {
    const double charge = c.shared ? 16.0 : 0.5;
    ConvTiling best{0, 1, false, c.shared};
    double best_us = 1e30;
    for (int S = 1; S <= 8; S *= 2) {
        if (want_splits > 0 ? S != want_splits : (S > 1 && c.nkb < 2 * S)) continue;
        const int widest = S > 1 ? std::min(bn_max, 128) : bn_max;
        for (int n = ceil_div(c.Kp16, widest); n <= ceil_div(c.Kp16, 32); ++n) {
            for (int tma = 0; tma < (S > 1 ? 1 : 2); ++tma) {          // TMA stores boxes of 32 or 64 columns of a whole tile
                const ConvTiling t{round_up(ceil_div(c.Kp16, n), tma ? 32 : std::max(16, 8 * S)), S, tma != 0, c.shared};
                if (t.BN > widest) continue;
                const int ctas = tiling_ctas(c, t);
                double us = tiling_us(ctas, c, t) + (S > 1 ? gain_us / 60.0 : 0.0);
                us += charge * ctas * tiling_stay(c, t) / 444.0;
                if (us < best_us - 1e-9) { best_us = us; best = t; }
            }
        }
    }
    return best;
}

// The search takes 1 to 6 us, as long as a launch: the tilings of the last shapes that operator calls asked for are kept.  The
// table is the library's and not a thread's (thread-local storage is allocated when a thread first touches it, which
// pb_conv2d_umma_noalloc may not do); a thread that finds it in use searches for itself.
ConvTiling choose_tiling(const ConvShape& c, int bn_max, int want_splits, double gain_us) {
    struct Kept { ConvShape c; int bn_max, want_splits; double gain_us; ConvTiling t; };
    static Kept kept[256];                       // BN 0: empty
    static std::atomic_flag busy = ATOMIC_FLAG_INIT;
    unsigned slot = (unsigned)c.m_tiles * 8191u + (unsigned)c.Kp16 * 131u + (unsigned)c.nkb * 8u + (unsigned)want_splits + (c.residual ? 4u : 0u);
    slot ^= slot >> 8;
    Kept& k = kept[slot % 256u];
    if (!busy.test_and_set(std::memory_order_acquire)) {
        const Kept found = k;
        busy.clear(std::memory_order_release);
        if (found.t.BN != 0 && found.c.m_tiles == c.m_tiles && found.c.Kp16 == c.Kp16 && found.c.nkb == c.nkb && found.c.residual == c.residual &&
            found.c.shared == c.shared && found.bn_max == bn_max && found.want_splits == want_splits && found.gain_us == gain_us)
            return found.t;
    }
    const ConvTiling t = best_tiling(c, bn_max, want_splits, gain_us);
    if (!busy.test_and_set(std::memory_order_acquire)) {
        k = {c, bn_max, want_splits, gain_us, t};
        busy.clear(std::memory_order_release);
    }
    return t;
}

ConvShape conv_shape(const pb_op_params* p, bool shared) {
    return {ceil_div(batch_of(p) * p->P * p->Q, kBM), round_up(p->K, 16), p->R * p->S * ceil_div(p->Cs, kBK), p->residual != nullptr, shared};
}
// Would lone blocks have less to do on the fullest SM than pairs, with n tiles of BN columns?
// - In fewer waves (148 pairs, two on a pair of SMs, against 296 blocks): with an odd m_tiles the last pair holds one real row tile.
//   Measured, lone blocks / pairs, 768 columns at 16 / 36 / 72 k-blocks: 297 pairs 0.83 / 0.84 / 0.88, 741 0.99 / 0.97 / 0.94, 1185 1.04 / 0.97 / 1.00;
//   half a wave more is none (519 pairs 1.06 / 1.02 / 1.06).
// - In as many rounds of one block an SM, with tiles of three quarters of the columns.  One round: 384 columns on 48 row tiles (128 wide
//   against 192) 0.86 to 0.91 at 16 to 72 k-blocks, 640 on 31 (160 / 224) 0.83 to 0.89, 576 on 31 (144 / 192) 0.92 to 0.95, 512 on 48
//   (176 / 256) 0.97 at 16, 1.07 at 36, 1.13 at 72, 768 on 31 (192 / 256) 0.97 / 1.05 / 1.11.  Three rounds, 99 row tiles, at 16 / 36 / 72 k-blocks:
//   640 columns 0.89 / 0.96 / 1.01, 768 columns 0.90 / 0.92 to 0.97 / 1.00, 576 columns (144 wide, which TMA does not store) 1.00 / 1.10 / 1.13.
//   Four fifths of the columns are no match: 1024 on 25 row tiles (208 / 256) 1.04 / 1.12 / 1.20.
bool lone_is_lighter(const ConvShape& c, int n, int BN, int pairs) {
    const int waves = ceil_div(pairs, 148), rounds = ceil_div(pairs, 74);
    if (waves <= 6 && ceil_div(c.m_tiles * n, 296) < waves) return true;
    for (int k = n + 1; ceil_div(c.m_tiles * k, 148) <= rounds; ++k) {
        const int w = round_up(ceil_div(c.Kp16, k), 16);
        if (4 * w > 3 * BN) continue;
        if (c.nkb < 36 || (rounds == 1 ? BN < 256 : c.nkb < 64 && w % 32 == 0)) return true;
    }
    return false;
}
// When a launch runs on pairs of blocks: wide tiles (the weights are what is shared), a k-loop long enough to carry the pair's
// set-up, and 48 to 74 pairs, one for each pair of SMs, or 140 and more, where two share a pair of SMs and are replaced as they finish -
// where lone blocks do not come out lighter.  Measured, lone blocks / pairs, us: 288 -> 384 3x3 35 x 35 x 64 images (614 pairs, 192
// columns) 143.8 / 132.8, 1024 -> 1024 3x3 14 x 14 x 16 (52) 61.3 / 49.4, 512 -> 512 3x3 28 x 28 x 8 (50) 32.9 / 29.3, 256 -> 256 3x3
// 28 x 28 x 16 with a residual (49) 22.7 / 19.1; 256 and 512 columns on maps of 16 x 32 by pairs, lone / pairs, at 18 / 36 / 72 k-blocks: 48 to
// 72 pairs 1.09 to 1.11 / 1.18 to 1.20 / 1.13 to 1.27, 140 to 148 0.99 to 1.01 / 1.00 / 1.01, 152 to 176 1.05 / 1.06 to 1.11 / 1.11 to 1.22, 184
// to 208 1.10 / 1.00 / 1.00, 220 to 296 1.00 / 1.00 to 1.02 / 1.00 to 1.02, 304 and more 1.00 to 1.06 / 1.01 to 1.12 / 1.01 to 1.05.  Outside: 76 to
// 96 pairs 0.98 / 0.99 / 0.88, 32 pairs 0.76, 4 k-blocks (196 pairs) 0.97.
// Not on a GPU that other requests share, where three lone blocks an SM do better.
// PB_CONV_PAIR (read at every use; for tests and comparisons): 0 = no pairs, 1 = pairs wherever their kernel can run.
ConvTiling pair_tiling(const ConvShape& c) {
    ConvTiling none{0, 1, false, c.shared};
    const char* e = getenv("PB_CONV_PAIR");
    const int force = e && (e[0] == '0' || e[0] == '1') ? e[0] - '0' : -1;
    if (force == 0 || !use_tma_a() || persist_enabled() || bn_limit() < 256) return none;
    const int n = ceil_div(c.Kp16, 256), BN = round_up(ceil_div(c.Kp16, n), 32);
    const int pairs = ceil_div(c.m_tiles, 2) * n;
    if (force < 0 && (c.shared || BN < 192 || c.nkb < 16 || pairs < 48 || (pairs > 74 && pairs < 140) || lone_is_lighter(c, n, BN, pairs))) return none;
    return {BN, 1, true, c.shared, true};
}
bool splits_off() { return !use_tma_a() || conv_split_gain_us() > 1e6; }
// want_splits: the cluster size (0: the fastest).
ConvTiling tiling_for(const pb_op_params* p, bool shared, int want_splits, bool may_pair = false) {
    if (may_pair) {
        const ConvTiling t = pair_tiling(conv_shape(p, shared));
        if (t.BN) return t;
    }
    return choose_tiling(conv_shape(p, shared), bn_limit(), splits_off() ? 1 : want_splits, conv_split_gain_us());
}
// The split is the caller's to allow: by the scratch memory that pb_launch_info.scratch_bytes asks for.
bool split_allowed(const pb_op_params* p) { return p->scratch != nullptr && p->scratch_bytes >= kSplitScratchBytes; }
ConvTiling tiling_or(const ConvTiling* given, const pb_op_params* p, bool pre) {
    return given ? *given : tiling_for(p, false, split_allowed(p) ? 0 : 1, !pre);      // the pair kernel does not normalise
}

Geometry geometry(const pb_op_params* p, const ConvTiling& t) {
    Geometry g;
    g.cpt = ceil_div(p->Cs, kBK);
    g.Cp = g.cpt * kBK;
    g.nkb = p->R * p->S * g.cpt;
    g.Kdim_pad = g.nkb * kBK;
    g.Kp16 = round_up(p->K, 16);
    g.m_tiles = ceil_div(batch_of(p) * p->P * p->Q, kBM);
    g.pair = t.pair;
    if (g.pair) g.m_tiles = round_up(g.m_tiles, 2);
    g.BN = t.BN;
    g.splits = t.splits;
    g.n_tiles = ceil_div(g.Kp16, g.BN);
    g.tmem_cols = 32;
    while ((int)g.tmem_cols < g.BN) g.tmem_cols <<= 1;
    g.b_stage_bytes = (uint32_t)(g.pair ? g.BN / 2 : g.BN) * 128u;
    const uint32_t stage_bytes = (uint32_t)kATileBytes + g.b_stage_bytes;
    uint32_t pipe_bytes = 0;
    g.meet = 0;
    if (use_tma_a()) {
        if (g.pair) {
            g.stages = std::min(kMaxStages, (int)((kSmemBudgetDeep - 1024u) / stage_bytes));
        } else {
            const Pipeline pipe = pipeline(g.m_tiles * g.n_tiles * g.splits, g.BN, ceil_div(g.nkb, g.splits), g.splits, t.shared);
            g.stages = pipe.stages;
            g.meet = pipe.meet;
            pipe_bytes = pipe.bytes;
        }
    } else {
        static const int kDepths[] = {8, 6, 4};                     // the gather kernel exists for 4, 6, 8
        g.stages = 4;
        for (int d : kDepths)
            if ((uint32_t)d * stage_bytes + 1024u <= kSmemBudget && d <= g.nkb + 1) { g.stages = d; break; }
    }
    g.out_box = !t.tma ? 0 : g.BN % 64 == 0 ? 64 : 32;
    g.smem_bytes = (pipe_bytes ? pipe_bytes : (uint32_t)g.stages * stage_bytes) + 1024u;
    // c_format f32 (1 << 4), a/b format bf16 (1 << 7, 1 << 10), K-major both, N >> 3 at bit 17, M >> 4 at bit 24
    g.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(g.BN >> 3) << 17) | ((uint32_t)((g.pair ? 2 * kBM : kBM) >> 4) << 24);
    return g;
}

// Dynamic shared memory of a launch; pre: it normalises its input.
uint32_t dynamic_smem(const Geometry& g, bool pre) { return g.smem_bytes + (pre ? (uint32_t)ceil_div(g.nkb, g.splits) * kPreBytes : 0u); }

const void* kernel_for(int stages, bool tma, bool pair, bool pre) {
    if (pair) return (const void*)conv_umma_pair_kernel;
    if (pre) return (const void*)conv_umma_pre_kernel;
    if (tma) return (const void*)conv_umma_tma_kernel;
    switch (stages) {
        case 4: return (const void*)conv_umma_gather_kernel<4>;
        case 6: return (const void*)conv_umma_gather_kernel<6>;
        default: return (const void*)conv_umma_gather_kernel<8>;
    }
}

// Raises the dynamic shared-memory limit of every kernel of this file on the current device.
cudaError_t raise_smem_limits() {
    const void* kernels[] = {(const void*)conv_umma_pair_kernel, (const void*)conv_umma_tma_kernel, (const void*)conv_umma_pre_kernel, (const void*)conv_umma_multi_kernel, (const void*)conv_umma_persist_kernel,
                             (const void*)conv_umma_gather_kernel<4>, (const void*)conv_umma_gather_kernel<6>,
                             (const void*)conv_umma_gather_kernel<8>};
    for (const void* k : kernels) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
        if (e != cudaSuccess) return e;
        // An SM's split between shared memory and L1 is fixed while blocks are resident.  Left to the default, the
        // first block to land on an idle SM sizes the split for itself alone and the SM then holds one or two blocks
        // instead of three until it has drained (measured under load: 14 % of the blocks started alone on their SM,
        // 40 % with one other, 45 % with two).  Ask for the largest shared-memory split whenever these kernels run.
        e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

struct ConvUmmaPlan {
    const void* w_dev;       // packed weights [rows][Kdim_pad]
    int rows, Kdim_pad;
    int device;
};

#ifdef PB_CONV_STATS
extern "C" __attribute__((visibility("default"))) int pb_debug_persist_hist(unsigned long long* out16, int reset) {
    if (cudaMemcpyFromSymbol(out16, g_persist_hist, sizeof(unsigned long long) * 16) != cudaSuccess) return -1;
    if (reset) { unsigned long long z[16] = {0}; cudaMemcpyToSymbol(g_persist_hist, z, sizeof(z)); }
    return 0;
}
extern "C" __attribute__((visibility("default"))) int pb_debug_persist_tile(long long* out96) {
    return cudaMemcpyFromSymbol(out96, g_persist_tile, sizeof(long long) * 16 * 6) == cudaSuccess ? 0 : -1;
}
extern "C" __attribute__((visibility("default"))) int pb_debug_persist_kb(long long* out384) {
    return cudaMemcpyFromSymbol(out384, g_persist_kb, sizeof(long long) * 64 * 6) == cudaSuccess ? 0 : -1;
}
extern "C" __attribute__((visibility("default"))) int pb_debug_conv_stats(unsigned long long* out16, int reset) {
    if (cudaMemcpyFromSymbol(out16, g_conv_stats, sizeof(unsigned long long) * 16) != cudaSuccess) return -1;
    unsigned long long ns = 0;
    if (cudaMemcpyFromSymbol(&ns, g_conv_ns, sizeof(ns)) != cudaSuccess) return -1;
    out16[15] = ns;          // replaces the 5+ bucket of the residency histogram
    if (reset) { const unsigned long long z1 = 0; cudaMemcpyToSymbol(g_conv_ns, &z1, sizeof(z1)); }
    if (reset) {
        unsigned long long z[16] = {0};
        if (cudaMemcpyToSymbol(g_conv_stats, z, sizeof(z)) != cudaSuccess) return -1;
    }
    return 0;
}
#endif

void conv_umma_set_split_gain_us(double us) { g_split_gain_us.store(us, std::memory_order_relaxed); }

bool conv_umma_supported(const pb_op_params* p) {
    const int groups = p->groups > 0 ? p->groups : 1;
    return p->dtype == 1 && groups == 1 && p->Cs % 8 == 0 && p->Ks % 8 == 0 && p->out_c_off % 8 == 0 && p->K % 8 == 0 &&
           (p->residual == nullptr || p->res_Cs % 8 == 0) && p->R >= 1 && p->S >= 1 && p->P * p->Q >= 1 &&
           !(p->flags & 2);
}

ConvTiling conv_umma_tiling(const pb_op_params* p, bool shared, bool may_split, bool may_pair) { return tiling_for(p, shared, may_split ? 0 : 1, may_pair); }

double conv_umma_us(const pb_op_params* p, const ConvTiling& t) {
    const ConvShape c = conv_shape(p, t.shared);
    return tiling_us(tiling_ctas(c, t), c, t);
}

int conv_umma_info(const pb_op_params* p, pb_launch_info* out, const ConvTiling* tiling, bool pre) {
    PB_REQUIRE(conv_umma_supported(p), "conv_umma: unsupported convolution");
    const Geometry g = geometry(p, tiling_or(tiling, p, pre));
    memset(out, 0, sizeof(*out));
    // what a split launch asks for, if it may split
    out->scratch_bytes = (tiling ? g.splits : tiling_for(p, false, 0, !pre).splits) > 1 ? kSplitScratchBytes : 0;
    out->kind = PB_STAGE_CONV_UMMA;
    out->num_blocks = (uint32_t)(g.m_tiles * g.n_tiles * g.splits);
    out->threads_per_block = use_tma_a() ? kThreadsTma : kThreads;
    cudaFuncAttributes at;
    uint32_t regs = 64, sstatic = 128;
    if (cudaFuncGetAttributes(&at, kernel_for(g.stages, use_tma_a(), g.pair, pre)) == cudaSuccess) {
        regs = (uint32_t)at.numRegs;
        sstatic = (uint32_t)at.sharedSizeBytes;
    } else {
        cudaGetLastError();
    }
    out->regs_per_thread = regs;
    out->smem_per_block = dynamic_smem(g, pre) + sstatic;
    out->tmem_cols_per_block = g.tmem_cols;
    const uint64_t nb = (uint64_t)batch_of(p);
    const uint64_t out_elems = nb * p->K * p->P * p->Q;
    out->flops = 2ull * out_elems * p->C * p->R * p->S;
    out->bytes = 2ull * (nb * p->C * p->H * p->W + (uint64_t)p->K * p->C * p->R * p->S + out_elems +
                         (p->residual ? out_elems : 0)) + 4ull * p->K;
    return PB_OK;
}

int64_t conv_umma_pack_weights(const pb_op_params* p, const float* w, void* dst) {
    if (!conv_umma_supported(p)) { set_error("conv_umma: unsupported convolution"); return PB_ERR_INVALID; }
    const int Cp = round_up(p->Cs, kBK), Kdim_pad = p->R * p->S * Cp;
    const size_t n = (size_t)packed_rows(p) * Kdim_pad;
    if (dst) {
        memset(dst, 0, n * 2);
        for (int k = 0; k < p->K; ++k)
            for (int c = 0; c < p->C; ++c)
                for (int r = 0; r < p->R; ++r)
                    for (int s = 0; s < p->S; ++s)
                        store_elem(dst, (size_t)k * Kdim_pad + (size_t)(r * p->S + s) * Cp + c,
                                   w[(((size_t)k * p->C + c) * p->R + r) * p->S + s], 1);
    }
    return (int64_t)(n * 2);
}

// Weight map of a launch with tiles of BN output channels.
// (BN: rows of a box, half a tile's columns for a pair of blocks)
static int make_tmap(const ConvUmmaPlan* plan, int BN, CUtensorMap* out) {
    const void* w_dev = plan->w_dev;
    EncodeTiledFn enc = encode_fn();
    PB_REQUIRE(enc != nullptr, "cuTensorMapEncodeTiled is not available from this driver");
    PB_REQUIRE(((uintptr_t)w_dev & 15) == 0, "conv_umma: packed weights must be 16-byte aligned");
    const cuuint64_t dims[2] = {(cuuint64_t)plan->Kdim_pad, (cuuint64_t)plan->rows};
    const cuuint64_t strides[1] = {(cuuint64_t)plan->Kdim_pad * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)BN};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(w_dev), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return PB_ERR_CUDA;
    }
    return PB_OK;
}

// im2col tensor map over the channels-last activation tensor [N=1][H][W][Cs] (dims listed innermost
// first).  The bounding box of filter-window origins is [-pad, dim + pad - (filter-1)); traversal
// strides are the convolution strides; each load brings 128 pixels x 64 channels.
// A 1x1, stride-1, unpadded convolution reads its input as the matrix [pixels][channels]: a tiled
// load moves the same 128 x 64 tile with far fewer requests than the im2col mode's per-pixel walk.
static bool pointwise(const pb_op_params* p) {
    return p->R == 1 && p->S == 1 && p->stride_h == 1 && p->stride_w == 1 && p->pad_h == 0 && p->pad_w == 0;      // any batch: images are contiguous
}

static int make_xmap(const pb_op_params* p, const ConvPre* pre, CUtensorMap* out) {
    if (pointwise(p)) {
        EncodeTiledFn enc2 = encode_fn();
        PB_REQUIRE(enc2 != nullptr, "cuTensorMapEncodeTiled is not available from this driver");
        const void* const x = pre ? pre->x : p->x;
        PB_REQUIRE(((uintptr_t)x & 15) == 0, "conv_umma: activations must be 16-byte aligned");
        const cuuint64_t dims2[2] = {(cuuint64_t)p->Cs, (cuuint64_t)batch_of(p) * p->H * p->W};
        const cuuint64_t strides2[1] = {(cuuint64_t)(pre ? pre->x_Cs : p->Cs) * 2};
        const cuuint32_t box2[2] = {(cuuint32_t)kBK, (cuuint32_t)kBM};
        const cuuint32_t estr2[2] = {1, 1};
        const CUresult r2 = enc2(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims2, strides2, box2, estr2,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r2 != CUDA_SUCCESS) {
            set_error("cuTensorMapEncodeTiled (activations) failed with CUresult %d (C %d, %d pixels)", (int)r2, p->Cs, p->H * p->W);
            return PB_ERR_CUDA;
        }
        return PB_OK;
    }
    EncodeIm2colFn enc = encode_im2col_fn();
    PB_REQUIRE(enc != nullptr, "cuTensorMapEncodeIm2col is not available from this driver");
    PB_REQUIRE(((uintptr_t)p->x & 15) == 0, "conv_umma: activations must be 16-byte aligned");
    const cuuint64_t dims[4] = {(cuuint64_t)p->Cs, (cuuint64_t)p->W, (cuuint64_t)p->H, (cuuint64_t)batch_of(p)};
    const cuuint64_t strides[3] = {(cuuint64_t)p->Cs * 2, (cuuint64_t)p->W * p->Cs * 2, (cuuint64_t)p->H * p->W * p->Cs * 2};
    const int lower[2] = {-p->pad_w, -p->pad_h};
    const int upper[2] = {p->pad_w - (p->S - 1) * dil_w(p), p->pad_h - (p->R - 1) * dil_h(p)};
    const cuuint32_t estr[4] = {1, (cuuint32_t)p->stride_w, (cuuint32_t)p->stride_h, 1};
    const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p->x), dims, strides, lower, upper,
                           (cuuint32_t)kBK, (cuuint32_t)kBM, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeIm2col failed with CUresult %d (C %d W %d H %d pad %d,%d filter %dx%d stride %d,%d)", (int)r, p->Cs,
                  p->W, p->H, p->pad_h, p->pad_w, p->R, p->S, p->stride_h, p->stride_w);
        return PB_ERR_CUDA;
    }
    return PB_OK;
}


// Map of [pixels of all images][channels] in boxes of U channels and so many rows.
static int make_rows_map(const pb_op_params* p, const __nv_bfloat16* base, int channels, int stride, int U, uint32_t rows, CUtensorMap* out) {
    EncodeTiledFn enc = encode_fn();
    PB_REQUIRE(enc != nullptr, "cuTensorMapEncodeTiled is not available from this driver");
    PB_REQUIRE(((uintptr_t)base & 15) == 0, "conv_umma: output and residual must be 16-byte aligned");
    const cuuint64_t dims[2] = {(cuuint64_t)channels, (cuuint64_t)batch_of(p) * p->P * p->Q};
    const cuuint64_t strides[1] = {(cuuint64_t)stride * 2};
    const cuuint32_t box[2] = {(cuuint32_t)U, rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUtensorMapSwizzle sw = U == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (output) failed with CUresult %d (%d channels, stride %d)", (int)r, channels, stride);
        return PB_ERR_CUDA;
    }
    return PB_OK;
}

// Map of the output slice (boxes of 32 rows) or of the residual (boxes of 128 rows).
static int make_ymap(const pb_op_params* p, int U, bool residual, CUtensorMap* out) {
    if (!U || (residual && !p->residual)) { memset(out, 0, sizeof(*out)); return PB_OK; }
    if (residual) return make_rows_map(p, static_cast<const __nv_bfloat16*>(p->residual), p->K, p->res_Cs, U, 128u, out);
    return make_rows_map(p, static_cast<const __nv_bfloat16*>(p->y) + p->out_c_off, p->K, p->Ks, U, 32u, out);
}

// The affine's channels are the layer's input channels, in whole vectors (x_Cs apart from pixel to pixel), and their constants fit
// beside the deepest pipeline even if the reduction is not split: 184 k-blocks, 11776 channels.
bool conv_umma_pre_supported(const pb_op_params* p, const ConvPre& pre) {
    return use_tma_a() && pointwise(p) && p->C == p->Cs && (uint32_t)ceil_div(p->Cs, kBK) * kPreBytes <= kSmemLimit - kSmemBudgetDeep && p->C % 8 == 0 && pre.x_Cs % 8 == 0 && pre.y_Cs % 8 == 0 && (pre.act == 0 || pre.act == 1) &&
           (((uintptr_t)pre.scale | (uintptr_t)pre.bias) & 15) == 0;
}

struct alignas(64) ConvUmmaXMap {
    CUtensorMap map;
    CUtensorMap normalised;      // of a launch with an input affine: the affine's tensor, in tiles of operand A
};

// Descriptors of a launch's input.
static int make_input_maps(const pb_op_params* p, const ConvPre* pre, ConvUmmaXMap* m) {
    const int rc = make_xmap(p, pre, &m->map);
    if (rc != PB_OK || !pre) return rc;
    return make_rows_map(p, static_cast<const __nv_bfloat16*>(pre->y), p->C, pre->y_Cs, kBK, (uint32_t)kBM, &m->normalised);
}

int encode_tiled_bf16(const void* base, int rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box, bool nan_fill, CUtensorMap* out) {
    EncodeTiledFn enc = encode_fn();
    PB_REQUIRE(enc != nullptr, "cuTensorMapEncodeTiled is not available from this driver");
    PB_REQUIRE(rank >= 1 && rank <= 5 && ((uintptr_t)base & 15) == 0, "tensor map: the tensor must be 16-byte aligned");
    cuuint64_t d[5], st[5];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; ++i) {
        d[i] = dims[i];
        bx[i] = box[i];
        es[i] = 1;
        if (i + 1 < rank) st[i] = strides[i];
    }
    const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), d, st, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           nan_fill ? CU_TENSOR_MAP_FLOAT_OOB_FILL_NAN_REQUEST_ZERO_FMA : CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with CUresult %d (rank %d, box %u x %u)", (int)r, rank, box[0], box[1]);
        return PB_ERR_CUDA;
    }
    return PB_OK;
}

int encode_pixels_f32(const void* base, int channels, int stride, int W, int H, int batch, int pad_w, int pad_h, int reach_w, int reach_h, int stride_w,
                      int stride_h, bool tiled, int box_channels, int box_pixels, CUtensorMap* out) {
    CUresult r;
    if (tiled) {
        EncodeTiledFn enc = encode_fn();
        PB_REQUIRE(enc != nullptr, "cuTensorMapEncodeTiled is not available from this driver");
        const cuuint64_t dims[2] = {(cuuint64_t)channels, (cuuint64_t)batch * H * W};
        const cuuint64_t strides[1] = {(cuuint64_t)stride * 4};
        const cuuint32_t box[2] = {(cuuint32_t)box_channels, (cuuint32_t)box_pixels}, estr[2] = {1, 1};
        r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        EncodeIm2colFn enc = encode_im2col_fn();
        PB_REQUIRE(enc != nullptr, "cuTensorMapEncodeIm2col is not available from this driver");
        const cuuint64_t dims[4] = {(cuuint64_t)channels, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)batch};
        const cuuint64_t strides[3] = {(cuuint64_t)stride * 4, (cuuint64_t)W * stride * 4, (cuuint64_t)H * W * stride * 4};
        const int lower[2] = {-pad_w, -pad_h}, upper[2] = {pad_w - reach_w, pad_h - reach_h};
        const cuuint32_t estr[4] = {1, (cuuint32_t)stride_w, (cuuint32_t)stride_h, 1};
        r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(base), dims, strides, lower, upper, (cuuint32_t)box_channels,
                (cuuint32_t)box_pixels, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncode (fp32 pixels) failed with CUresult %d (%d channels, %d apart, %d x %d)", (int)r, channels, stride, H, W);
        return PB_ERR_CUDA;
    }
    return PB_OK;
}

int encode_weights_f32(const void* base, int columns, int rows, int taps, int box_columns, int box_rows, CUtensorMap* out) {
    EncodeTiledFn enc = encode_fn();
    PB_REQUIRE(enc != nullptr, "cuTensorMapEncodeTiled is not available from this driver");
    const cuuint64_t dims[3] = {(cuuint64_t)columns, (cuuint64_t)rows, (cuuint64_t)taps};
    const cuuint64_t strides[2] = {(cuuint64_t)columns * 4, (cuuint64_t)rows * columns * 4};
    const cuuint32_t box[3] = {(cuuint32_t)box_columns, (cuuint32_t)box_rows, 1}, estr[3] = {1, 1, 1};
    const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled (fp32 weights) failed with CUresult %d (%d x %d, %d taps)", (int)r, rows, columns, taps);
        return PB_ERR_CUDA;
    }
    return PB_OK;
}

int conv_umma_xmap_create(const pb_op_params* p, ConvUmmaXMap** out, const ConvPre* pre) {
    if (!use_tma_a()) { *out = nullptr; return PB_OK; }
    ConvUmmaXMap* m = new ConvUmmaXMap();
    const int rc = make_input_maps(p, pre, m);
    if (rc != PB_OK) { delete m; return rc; }
    *out = m;
    return PB_OK;
}

void conv_umma_xmap_destroy(ConvUmmaXMap* m) { delete m; }

int conv_umma_plan_create(const pb_op_params* p, const void* w_dev, ConvUmmaPlan** out) {
    PB_REQUIRE(conv_umma_supported(p), "conv_umma: unsupported convolution");
    PB_REQUIRE(((uintptr_t)w_dev & 15) == 0, "conv_umma: packed weights must be 16-byte aligned");
    ConvUmmaPlan* plan = new ConvUmmaPlan();
    plan->w_dev = w_dev;
    plan->rows = packed_rows(p);
    plan->Kdim_pad = p->R * p->S * ceil_div(p->Cs, kBK) * kBK;
    cudaGetDevice(&plan->device);
    // The shared-memory limit is a per-device function attribute: raise it once on every device used.
    static std::once_flag once[16];
    static cudaError_t attr_errs[16] = {};
    if (plan->device < 0 || plan->device >= 16) {
        const int bad = plan->device;
        delete plan;
        set_error("conv_umma: device index %d outside 0..15 (the per-device kernel attributes are kept for 16 devices)", bad);
        return PB_ERR_INVALID;
    }
    const int dev = plan->device;
    std::call_once(once[dev], [dev] { attr_errs[dev] = raise_smem_limits(); });
    const cudaError_t attr_err = attr_errs[dev];
    if (attr_err != cudaSuccess) { delete plan; return cuda_fail(attr_err, "cudaFuncSetAttribute(conv_umma)", __FILE__, __LINE__); }
    *out = plan;
    return PB_OK;
}

void conv_umma_plan_destroy(ConvUmmaPlan* plan) { delete plan; }

// Kernel arguments of one convolution.
static int fill_args(const ConvUmmaPlan* plan, const Geometry& g, const pb_op_params* p, uint32_t* err_flag, ConvArgs* out) {
    ConvArgs& a = *out;
    memset(&a, 0, sizeof(a));
    a.x = static_cast<const __nv_bfloat16*>(p->x);
    a.residual = static_cast<const __nv_bfloat16*>(p->residual);
    a.bias = p->bias;
    a.y = static_cast<__nv_bfloat16*>(p->y);
    a.err_flag = err_flag ? err_flag : device_error_flag_ptr(plan->device);
    PB_REQUIRE(a.err_flag != nullptr, "conv_umma: no device error flag");
    a.H = p->H; a.W = p->W; a.Cs = p->Cs; a.P = p->P; a.Q = p->Q; a.PQ = p->P * p->Q; a.M = batch_of(p) * a.PQ;
    a.dh = dil_h(p); a.dw = dil_w(p);
    a.K = p->K; a.Ks = p->Ks; a.out_c_off = p->out_c_off; a.res_Cs = p->res_Cs;
    a.R = p->R; a.S = p->S; a.sh = p->stride_h; a.sw = p->stride_w; a.ph = p->pad_h; a.pw = p->pad_w;
    a.act = p->act; a.a_tiled = pointwise(p) ? 1 : 0; a.nkb = g.nkb; a.taps = p->R * p->S; a.Cp = g.Cp; a.BN = g.BN; a.idesc = g.idesc; a.tmem_cols = g.tmem_cols;
    a.b_stage_bytes = g.b_stage_bytes;
    a.splits = g.splits;
    a.meet = g.meet;
    a.inv_PQ = 1.f / (float)a.PQ; a.inv_Q = 1.f / (float)a.Q; a.inv_cpt = 1.f / (float)g.cpt; a.inv_S = 1.f / (float)a.S;
    a.out_box = g.out_box;
    return PB_OK;
}

template <typename... Args>
static cudaError_t launch_pdl(void (*kern)(Args...), dim3 grid, dim3 cluster, uint32_t smem, cudaStream_t st, bool pdl, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreadsTma);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster.x * cluster.y * cluster.z > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster.x;
        attr[n].val.clusterDim.y = cluster.y;
        attr[n++].val.clusterDim.z = cluster.z;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

int conv_umma_launch_planned(const ConvUmmaPlan* plan, const ConvUmmaXMap* xmap, const pb_op_params* p, cudaStream_t st,
                             uint32_t job_id, void* notifier, uint32_t* err_flag, bool pdl, const ConvTiling* tiling, const ConvPre* pre) {
    const Geometry g = geometry(p, tiling_or(tiling, p, pre != nullptr));
    if (!use_tma_a()) PB_REQUIRE(batch_of(p) == 1, "conv_umma: the cp.async gather kernel (PB_CONV_GATHER=1) runs one image per launch");
    ConvArgs a;
    const int frc = fill_args(plan, g, p, err_flag, &a);
    if (frc != PB_OK) return frc;
    if (pre) {
        PB_REQUIRE(use_tma_a() && !g.pair && conv_umma_pre_supported(p, *pre), "conv_umma: this layer cannot take an input affine");
        a.pre_scale = pre->scale; a.pre_bias = pre->bias; a.pre_act = pre->act; a.pre_offset = g.smem_bytes - 1024u;
    }
    const uint32_t smem = dynamic_smem(g, pre != nullptr);
    const dim3 grid((unsigned)g.m_tiles, (unsigned)g.n_tiles, (unsigned)g.splits);
    FinishedBlockNotifier* nf = static_cast<FinishedBlockNotifier*>(notifier);
    if (use_tma_a()) {
        ConvUmmaXMap local;
        if (!xmap) {
            const int rc = make_input_maps(p, pre, &local);
            if (rc != PB_OK) return rc;
            xmap = &local;
        }
        CUtensorMap wmap, ymap, rmap;
        int mrc = make_tmap(plan, g.pair ? g.BN / 2 : g.BN, &wmap);
        if (mrc == PB_OK) mrc = make_ymap(p, g.out_box, false, &ymap);
        if (mrc == PB_OK) mrc = make_ymap(p, g.out_box, true, &rmap);
        if (mrc != PB_OK) return mrc;
        const dim3 cluster = g.pair ? dim3(2, 1, 1) : dim3(1, 1, (unsigned)g.splits);
        const cudaError_t e =
            pre ? launch_pdl(conv_umma_pre_kernel, grid, cluster, smem, st, pdl, wmap, xmap->map, ymap, rmap, xmap->normalised, a, g.stages, job_id, nf)
                : launch_pdl(g.pair ? conv_umma_pair_kernel : conv_umma_tma_kernel, grid, cluster, smem, st, pdl, wmap, xmap->map, ymap, rmap, a, g.stages, job_id, nf);
        if (e != cudaSuccess)
            return cuda_fail(e, pre ? "launch of conv_umma_pre_kernel" : g.pair ? "launch of conv_umma_pair_kernel" : "launch of conv_umma_tma_kernel", __FILE__, __LINE__);
        return PB_OK;
    } else {
        CUtensorMap wmap;
        const int wrc = make_tmap(plan, g.BN, &wmap);
        if (wrc != PB_OK) return wrc;
        switch (g.stages) {
            case 4: conv_umma_gather_kernel<4><<<grid, kThreads, g.smem_bytes, st>>>(wmap, a, job_id, nf); break;
            case 6: conv_umma_gather_kernel<6><<<grid, kThreads, g.smem_bytes, st>>>(wmap, a, job_id, nf); break;
            default: conv_umma_gather_kernel<8><<<grid, kThreads, g.smem_bytes, st>>>(wmap, a, job_id, nf); break;
        }
    }
    return launch_check("conv_umma");
}

// ---- grouped launch ----------------------------------------------------------------------------
struct ConvUmmaMulti {
    SubConv* table_dev = nullptr;
    int n = 0;
    unsigned total_blocks = 0;      // tiles of all sub-problems (= CTAs of the one-tile-per-CTA kernel)
    uint32_t smem = 0;
    uint32_t tmem_cols = 0;
    SubStarts starts;
    unsigned splits = 1;            // cluster size of the launch
    bool has_pool = false;          // pooling layers ride along (one-tile kernel only)
    // persistent kernel
    bool persist = false;
    unsigned grid = 0;
    int stages = 0;
    uint32_t stage_bytes = 0, persist_smem = 0;
};

bool conv_umma_multi_available() { return use_tma_a(); }

// The cluster size of a grouped launch is one for all its convolutions: the one whose slowest member is modelled fastest.
void conv_umma_group_tilings(const pb_op_params* const* params, int n, bool shared, bool may_split, ConvTiling* out) {
    const int most = may_split && !splits_off() ? 8 : 1;
    int longest = 0;
    for (int i = 0; i < n; ++i) longest = std::max(longest, conv_shape(params[i], shared).nkb);
    double best_us = 1e30;
    std::vector<ConvTiling> t((size_t)n);
    for (int S = 1; S <= most && (S == 1 || longest >= 2 * S); S *= 2) {
        int ctas = 0;
        for (int i = 0; i < n; ++i) {
            t[(size_t)i] = tiling_for(params[i], shared, S);
            ctas += tiling_ctas(conv_shape(params[i], shared), t[(size_t)i]);
        }
        double us = S > 1 ? conv_split_gain_us() / 60.0 : 0.0, slowest = 0;
        for (int i = 0; i < n; ++i) slowest = std::max(slowest, tiling_us(ctas, conv_shape(params[i], shared), t[(size_t)i]));
        us += slowest;
        if (us < best_us) { best_us = us; std::copy(t.begin(), t.end(), out); }
    }
}

bool conv_umma_persist_enabled() { return persist_enabled(); }
uint32_t conv_umma_persist_grid(uint32_t total_tiles) {
    const uint32_t g = ceil_div<uint32_t>(total_tiles, (uint32_t)tiles_per_cta());
    return g < 1 ? 1 : g;
}

// A 3x3 max / average pooling layer (bf16, vector-aligned slice) can ride along in a grouped launch.
bool conv_umma_pool_fusable(int kind, const pb_op_params* p) {
    return (kind == PB_STAGE_MAXPOOL || kind == PB_STAGE_AVGPOOL) && p->dtype == 1 && p->R == 3 && p->S == 3 && p->Cs % 8 == 0 &&
           p->Ks % 8 == 0 && p->out_c_off % 8 == 0 && !(p->flags & 2) && p->H >= 1 && p->W >= 1 && p->bias == nullptr && p->act == 0;
}
uint32_t conv_umma_pool_blocks(const pb_op_params* p) {
    const uint64_t vecs = (uint64_t)batch_of(p) * p->P * p->Q * (p->Cs / 8);
    return (uint32_t)ceil_div<uint64_t>(vecs, (uint64_t)kThreadsTma * kPoolVecsPerThread);
}

int conv_umma_multi_create(const ConvUmmaPlan* const* plans, const ConvUmmaXMap* const* xmaps, const pb_op_params* const* params, const int* kinds,
                           const ConvTiling* tilings, int n, ConvUmmaMulti** out) {
    PB_REQUIRE(out && plans && xmaps && params && n >= 1 && n <= kMaxSubConvs, "conv_umma_multi_create: 1..%d entries", kMaxSubConvs);
    PB_REQUIRE(use_tma_a(), "conv_umma_multi_create: needs the TMA operand path");
    std::vector<SubConv> table((size_t)n);
    memset(table.data(), 0, sizeof(SubConv) * (size_t)n);
    ConvUmmaMulti* m = new ConvUmmaMulti();
    m->n = n;
    auto is_pool = [&](int i) { return kinds && kinds[i] != PB_STAGE_CONV_UMMA; };
    // the convolutions first: with clusters their blocks have to start on a cluster boundary
    int at = 0;
    for (int i = 0; i < n; ++i) {
        if (is_pool(i)) continue;
        PB_REQUIRE(plans[i] && xmaps[i] && params[i], "conv_umma_multi_create: NULL entry %d", i);
        const bool split = split_allowed(params[i]) && !persist_enabled();
        const Geometry g = geometry(params[i], tilings ? tilings[i] : tiling_for(params[i], false, split ? 0 : 1));
        SubConv& sc = table[(size_t)at++];
        int rc = make_tmap(plans[i], g.BN, &sc.tmap_w);
        if (rc == PB_OK) rc = make_ymap(params[i], g.out_box, false, &sc.tmap_y);
        if (rc == PB_OK) rc = make_ymap(params[i], g.out_box, true, &sc.tmap_r);
        if (rc != PB_OK) { delete m; return rc; }
        sc.tmap_x = xmaps[i]->map;
        rc = fill_args(plans[i], g, params[i], nullptr, &sc.a);
        if (rc != PB_OK) { delete m; return rc; }
        if (at > 1 && (unsigned)g.splits != m->splits) { delete m; set_error("conv_umma_multi_create: the entries of a launch must share one split"); return PB_ERR_INVALID; }
        m->splits = (unsigned)g.splits;
        sc.first_block = m->total_blocks;
        sc.gx = (uint32_t)g.m_tiles;
        sc.inv_gx = 1.f / (float)g.m_tiles;
        sc.gy = (uint32_t)g.n_tiles;
        sc.stages = (uint32_t)g.stages;
        m->total_blocks += (unsigned)(g.m_tiles * g.n_tiles * g.splits);
        m->smem = std::max(m->smem, g.smem_bytes);
        m->tmem_cols = std::max(m->tmem_cols, g.tmem_cols);
        m->stage_bytes = std::max(m->stage_bytes, (uint32_t)kATileBytes + g.b_stage_bytes);
    }
    for (int i = 0; i < n; ++i) {
        if (!is_pool(i)) continue;
        const pb_op_params* p = params[i];
        if (!p || !conv_umma_pool_fusable(kinds[i], p)) { delete m; set_error("conv_umma_multi_create: entry %d cannot ride along", i); return PB_ERR_INVALID; }
        SubConv& sc = table[(size_t)at++];
        PoolSubArgs& a = sc.pool;
        a.x = static_cast<const __nv_bfloat16*>(p->x);
        a.y = static_cast<__nv_bfloat16*>(p->y);
        a.C = p->C; a.H = p->H; a.W = p->W; a.Cs = p->Cs; a.P = p->P; a.Q = p->Q; a.Ks = p->Ks; a.out_c_off = p->out_c_off;
        a.sh = p->stride_h; a.sw = p->stride_w; a.ph = p->pad_h; a.pw = p->pad_w;
        a.is_max = kinds[i] == PB_STAGE_MAXPOOL; a.count_pad = p->flags & 1; a.batch = batch_of(p);
        sc.first_block = m->total_blocks;
        sc.gx = sc.gy = 1;
        sc.inv_gx = 1.f;
        sc.stages = kSubPool;
        m->total_blocks += conv_umma_pool_blocks(p);
        m->has_pool = true;
    }
    m->total_blocks = round_up(m->total_blocks, m->splits);      // blocks past the last pooling vector find nothing to do
    if (m->stage_bytes == 0) { delete m; set_error("conv_umma_multi_create: no convolution among the entries"); return PB_ERR_INVALID; }
    // persistent kernel: one pipeline for every sub-problem (stages of the widest), two accumulators
    m->stages = (int)std::min<uint32_t>(kMaxStages, (kSmemBudgetPersist - 1024u) / m->stage_bytes);
    m->persist_smem = (uint32_t)m->stages * m->stage_bytes + 1024u;
    m->grid = conv_umma_persist_grid(m->total_blocks);
    m->persist = persist_enabled() && m->splits == 1 && m->stages >= 2 && 2u * m->tmem_cols <= 512u && !m->has_pool;
    for (int i = 0; i < kMaxSubConvs; ++i) m->starts.first[i] = i < n ? table[(size_t)i].first_block : 0xffffffffu;
    cudaError_t e = cudaMalloc((void**)&m->table_dev, sizeof(SubConv) * (size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(m->table_dev, table.data(), sizeof(SubConv) * (size_t)n, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { conv_umma_multi_destroy(m); return cuda_fail(e, "conv_umma_multi_create", __FILE__, __LINE__); }
    *out = m;
    return PB_OK;
}

void conv_umma_multi_destroy(ConvUmmaMulti* m) {
    if (!m) return;
    if (m->table_dev) cudaFree(m->table_dev);
    delete m;
}

void conv_umma_persist_footprint(uint32_t total_tiles, uint32_t max_tmem_cols, pb_launch_info* out) {
    memset(out, 0, sizeof(*out));
    out->num_blocks = conv_umma_persist_grid(total_tiles);
    out->threads_per_block = kThreadsPersist;
    out->smem_per_block = kSmemBudgetPersist;
    cudaFuncAttributes at;
    out->regs_per_thread = 128;
    if (cudaFuncGetAttributes(&at, (const void*)conv_umma_persist_kernel) == cudaSuccess) out->regs_per_thread = (uint32_t)at.numRegs;
    else cudaGetLastError();
    out->tmem_cols_per_block = 2u * max_tmem_cols;
    out->kind = PB_STAGE_CONV_UMMA;
}

void conv_umma_multi_info(const ConvUmmaMulti* m, pb_launch_info* out) {
    memset(out, 0, sizeof(*out));
    out->num_blocks = m->persist ? m->grid : m->total_blocks;
    out->threads_per_block = m->persist ? kThreadsPersist : kThreadsTma;
    out->smem_per_block = m->persist ? m->persist_smem : m->smem;
    cudaFuncAttributes at;
    out->regs_per_thread = 112;
    if (cudaFuncGetAttributes(&at, m->persist ? (const void*)conv_umma_persist_kernel : (const void*)conv_umma_multi_kernel) == cudaSuccess)
        out->regs_per_thread = (uint32_t)at.numRegs;
    else cudaGetLastError();
    out->tmem_cols_per_block = m->persist ? 2u * m->tmem_cols : m->tmem_cols;
    out->kind = PB_STAGE_CONV_UMMA;
}

int conv_umma_multi_launch(const ConvUmmaMulti* m, cudaStream_t st, uint32_t job_id, void* notifier, bool pdl) {
    if (m->persist) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(m->grid);
        cfg.blockDim = dim3(kThreadsPersist);
        cfg.dynamicSmemBytes = m->persist_smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = pdl ? 1 : 0;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, conv_umma_persist_kernel, (const SubConv*)m->table_dev, m->n, (uint32_t)m->total_blocks, m->stages,
                                                 m->stage_bytes, m->tmem_cols, job_id, static_cast<FinishedBlockNotifier*>(notifier));
        if (e != cudaSuccess) return cuda_fail(e, "launch of conv_umma_persist_kernel", __FILE__, __LINE__);
        return PB_OK;
    }
    const cudaError_t e = launch_pdl(conv_umma_multi_kernel, dim3(m->total_blocks), dim3(m->splits), m->smem, st, pdl,
                                     (const SubConv*)m->table_dev, m->starts, job_id, static_cast<FinishedBlockNotifier*>(notifier));
    if (e != cudaSuccess) return cuda_fail(e, "launch of conv_umma_multi_kernel", __FILE__, __LINE__);
    return PB_OK;
}

int conv_umma_launch(const pb_op_params* p, cudaStream_t st, uint32_t job_id, void* notifier) {
    ConvUmmaPlan* plan = nullptr;
    int rc = conv_umma_plan_create(p, p->w, &plan);
    if (rc != PB_OK) return rc;
    // PB_CONV_PERSIST_OPS=1 (read at every call; for tests): a lone operator launch also runs the persistent kernel
    // the model launches use, through a one-entry table that lives for this call only (allocates and synchronises).
    const char* po = getenv("PB_CONV_PERSIST_OPS");
    if (po && po[0] == '1' && persist_enabled()) {
        ConvUmmaXMap* xm = nullptr;
        ConvUmmaMulti* mu = nullptr;
        rc = conv_umma_xmap_create(p, &xm);
        if (rc == PB_OK) {
            const ConvUmmaPlan* plans[1] = {plan};
            const ConvUmmaXMap* xms[1] = {xm};
            const pb_op_params* pp[1] = {p};
            rc = conv_umma_multi_create(plans, xms, pp, nullptr, nullptr, 1, &mu);
        }
        if (rc == PB_OK && !mu->persist) { set_error("conv_umma: this shape does not fit the persistent kernel"); rc = PB_ERR_INVALID; }
        if (rc == PB_OK) rc = conv_umma_multi_launch(mu, st, job_id, notifier, false);
        if (rc == PB_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = cuda_fail(cudaGetLastError(), "persistent convolution", __FILE__, __LINE__);
        conv_umma_multi_destroy(mu);
        conv_umma_xmap_destroy(xm);
        conv_umma_plan_destroy(plan);
        return rc;
    }
    rc = conv_umma_launch_planned(plan, nullptr, p, st, job_id, notifier, nullptr);
    conv_umma_plan_destroy(plan);   // the tensor maps were copied into the launch parameters
    return rc;
}

// Times `iters` launches of one convolution between CUDA events (after 3 warm-up launches), an L2 flush (a write
// of flush_bytes) before each when asked: mode 0 = the kernel pb_op_launch takes, 1 = the persistent kernel.
int conv_umma_time(const pb_op_params* p, int mode, int iters, size_t flush_bytes, double* us_out) {
    PB_REQUIRE(p && us_out && iters > 0, "pb_conv_umma_time: bad arguments");
    ConvUmmaPlan* plan = nullptr;
    ConvUmmaXMap* xm = nullptr;
    ConvUmmaMulti* mu = nullptr;
    void* flush = nullptr;
    cudaStream_t st = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int rc = conv_umma_plan_create(p, p->w, &plan);
    if (rc == PB_OK) rc = conv_umma_xmap_create(p, &xm);
    if (rc == PB_OK && mode == 1) {
        const ConvUmmaPlan* plans[1] = {plan};
        const ConvUmmaXMap* xms[1] = {xm};
        const pb_op_params* pp[1] = {p};
        rc = conv_umma_multi_create(plans, xms, pp, nullptr, nullptr, 1, &mu);
        if (rc == PB_OK && !mu->persist) { set_error("pb_conv_umma_time: the persistent kernel is off or does not fit this shape"); rc = PB_ERR_INVALID; }
    }
    cudaError_t e = cudaSuccess;
    if (rc == PB_OK) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (rc == PB_OK && e == cudaSuccess && flush_bytes) e = cudaMalloc(&flush, flush_bytes);
    if (rc == PB_OK && e == cudaSuccess) e = cudaEventCreate(&e0);
    if (rc == PB_OK && e == cudaSuccess) e = cudaEventCreate(&e1);
    double total_ms = 0;
    auto launch = [&]() { return mode == 1 ? conv_umma_multi_launch(mu, st, 0, nullptr, false) : conv_umma_launch_planned(plan, xm, p, st, 0, nullptr, nullptr, false); };
    for (int i = 0; rc == PB_OK && e == cudaSuccess && i < 3; ++i) rc = launch();
    for (int i = 0; rc == PB_OK && e == cudaSuccess && i < iters; ++i) {
        if (flush) cudaMemsetAsync(flush, i & 0xff, flush_bytes, st);
        cudaEventRecord(e0, st);
        rc = launch();
        cudaEventRecord(e1, st);
        e = cudaEventSynchronize(e1);
        float ms = 0;
        if (e == cudaSuccess) { cudaEventElapsedTime(&ms, e0, e1); total_ms += ms; }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (flush) cudaFree(flush);
    if (st) cudaStreamDestroy(st);
    conv_umma_multi_destroy(mu);
    conv_umma_xmap_destroy(xm);
    conv_umma_plan_destroy(plan);
    if (rc != PB_OK) return rc;
    if (e != cudaSuccess) return cuda_fail(e, "pb_conv_umma_time", __FILE__, __LINE__);
    *us_out = total_ms * 1000.0 / iters;
    return PB_OK;
}

// ---- launch without any allocation -----------------------------------------------------------------
static __device__ uint32_t g_noalloc_err_flag;

namespace {
struct NoAllocDevice {
    bool ready = false;
    uint32_t* err_flag = nullptr;
};
NoAllocDevice g_noalloc_dev[16];
std::mutex g_noalloc_mu;
}  // namespace

uint32_t* noalloc_error_flag_ptr(int device) {
    if (device < 0 || device >= 16) return nullptr;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    return g_noalloc_dev[device].ready ? g_noalloc_dev[device].err_flag : nullptr;
}

int conv_umma_launch_noalloc(const pb_op_params* p, cudaStream_t st, uint32_t job_id, void* notifier) {
    PB_REQUIRE(p != nullptr && conv_umma_supported(p), "pb_conv2d_umma_noalloc: unsupported convolution");
    int device = -1;
    PB_CUDA(cudaGetDevice(&device));
    PB_REQUIRE(device >= 0 && device < 16, "pb_conv2d_umma_noalloc: device %d out of range", device);
    NoAllocDevice& nd = g_noalloc_dev[device];
    {
        // First call on this device: resolve the device address of the file-scope flag.  In host
        // code its name is only a stand-in, not a device address; the kernel must be given what
        // cudaGetSymbolAddress returns, with this device current.
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!nd.ready) {
            void* fp = nullptr;
            PB_CUDA(cudaGetSymbolAddress(&fp, g_noalloc_err_flag));
            PB_CUDA(raise_smem_limits());
            nd.err_flag = static_cast<uint32_t*>(fp);
            nd.ready = true;
        }
    }
    ConvUmmaPlan plan{p->w, packed_rows(p), p->R * p->S * ceil_div(p->Cs, kBK) * kBK, device};      // on the stack: no host allocation either
    pb_op_params q = *p;
    q.scratch = (void*)nd.err_flag;         // never touched: allows the split, whose partial tiles meet in shared memory
    q.scratch_bytes = kSplitScratchBytes;
    return conv_umma_launch_planned(&plan, nullptr, &q, st, job_id, notifier, nd.err_flag);
}

}  // namespace pb
