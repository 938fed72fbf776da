// Dense convolution in full precision: an implicit GEMM on the fp32 units.
//
//   D[m, n] = sum_k A[m, k] * B[k, n]     m = output pixel (all images back to back), n = output channel,
//                                          k = (r*S + s)*Cs + c   (filter tap, input channel)
//
// The layers that conv_f32_umma.cu leaves: five to 23 input channels, short layers of few outputs, unaligned tensors, output sizes of the caller's own.
// The ceiling is the fused multiply-add rate: 148 SMs x 128 x 2 x 1.9 GHz = 72 TFLOP/s.  The direct kernel this replaces for dense layers (conv_simt_kernel: one output per thread, every operand
// through L1 for each multiplication) ran at 1.9 TFLOP/s.
//
// Block = 256 threads on a tile of 64 pixels x BN channels.  A stage is 32 values of k, three stages deep, brought by
// cp.async: 64 x 32 activations (zero-filled outside the image), turned to [k][pixel] on the way by 4-byte copies, and
// 32 x BN weights.  The groups of threads that cover the tile once (64 at BN = 64) split every stage's k between them, so
// a tile this small still feeds eight warps, and their partial tiles are added in group order at the end.  A layer with
// few tiles additionally splits its k range over the blocks of a cluster (up to 8), whose sums meet through distributed
// shared memory, in rank order: results do not depend on timing.
//
// This is the fp32 member of the kernel family the reference's TVM adapters launch
// (jobs/tvm_<model>/tvm_<model>.cpp:24-47; generated fp32 kernels there).
#include <llis/job/finished_block_notifier.h>

#include <algorithm>
#include <cstring>

#include "conv_f32.h"
#include "launch_slot.cuh"
#include "ops.h"
#include "pb_common.h"

using llis::job::FinishedBlockNotifier;

namespace pb {

namespace {

constexpr int kTM = 64, kTK = 32, kDepth = 3;
constexpr int kBlock = 256;

struct F32Args {
    OpArgs op;
    int M, PQ;           // rows of the GEMM (all images), pixels per image
    int Kp;              // channels of a row of packed weights (K rounded up to 4)
    int n_stages;        // k stages of the whole reduction
    int splits;          // cluster size
    uint32_t declared;   // blocks this launch was declared as, where they are not the grid's (else 0)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int Bytes>
__device__ __forceinline__ void cp_async(uint32_t dst, const float* src, bool ok) {
    if (Bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16u : 0u) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4u : 0u) : "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t rank) {
    float4 v;
    asm volatile(
        "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "r"(addr), "r"(rank)
        : "memory");
    return v;
}
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Bias, residual, activation and store of four channels of one output pixel.
__device__ __forceinline__ void finish4(const OpArgs& a, int m, int k, const float4& s, bool vec) {
    const float v[4] = {s.x, s.y, s.z, s.w};
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int kk = k + j;
        if (kk >= a.K) break;
        float x = v[j] + (a.bias ? __ldg(a.bias + kk) : 0.f);
        if (a.residual) x += static_cast<const float*>(a.residual)[(size_t)m * a.res_Cs + kk];
        if (a.act == 3) x = x > 0.f ? x : x * __ldg(a.bias + a.K + kk);      // PReLU: slopes follow the biases
        else if (a.act == 1) x = fmaxf(x, 0.f);
        else if (a.act == 2) x = fminf(fmaxf(x, 0.f), 6.f);
        o[j] = x;
    }
    float* y = static_cast<float*>(a.y) + (size_t)m * a.Ks + a.out_c_off + k;
    if (vec && k + 4 <= a.K) {
        *reinterpret_cast<float4*>(y) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (k + j < a.K) y[j] = o[j];
    }
}

// Aligned: the weights start on a 16-byte boundary.  Padded: channels from C to the stride Cs are not the layer's; they count as
// zeros whatever lies there.  (Tested in every instance it costs a ResNet-18 2 %: 428 -> 438 us for two images.)
//
// A thread owns 8 pixels x TJ channels and takes, per k, its 8 activations and TJ weights as 16-byte loads and multiplies
// the outer product.  Operand order matters: with the pixels of one k side by side in registers the compiler can place the
// accumulators so that the three operands of a multiply-add come from different register banks.  (With the k of one pixel
// side by side - the layout a 16-byte copy of the activations gives - every other multiply-add conflicts: 37 TFLOP/s on a
// layer that fills the GPU; the packed two-wide multiply-add has no conflicts, but issues at half the rate or less: 38.)
template <int BN, bool Aligned, bool Padded>
__global__ void __launch_bounds__(kBlock, 2) conv_f32_kernel(const F32Args f, uint32_t job_id, FinishedBlockNotifier* nf) {
    griddep_wait();
    resolve_slot(job_id, nf);
    if (nf) {
        if (f.declared) nf->start_as(job_id, f.declared);
        else nf->start(job_id);
    }
    constexpr int TJ = BN == 64 ? 8 : 4;           // channels per thread
    constexpr int kGroupThreads = 8 * BN / TJ, kGroups = kBlock / kGroupThreads, kGroupK = kTK / kGroups;
    constexpr int kStageFloats = kTK * kTM + kTK * BN;
    constexpr int kLdR = BN + 4;                   // row of a partial tile
    extern __shared__ __align__(16) float smem[];
    const OpArgs& a = f.op;
    const int tid = threadIdx.x;
    const int m0 = blockIdx.x * kTM, n0 = blockIdx.y * BN, rank = blockIdx.z;
    const int s0 = f.n_stages * rank / f.splits, s1 = f.n_stages * (rank + 1) / f.splits;

    // ---- what this thread copies: chunk `tid % 8` (4 channels) of pixels tid/8 and tid/8 + 32 ----
    const int taps = a.R * a.S, c4n = a.Cs / 4;
    int ih0[2], iw0[2], row0[2];                   // filter-window origin, first input row of the image
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int m = m0 + (tid >> 3) + 32 * i;
        const bool in = m < f.M;
        const int img = in ? m / f.PQ : 0, pix = in ? m - img * f.PQ : 0;
        const int p = pix / a.Q, q = pix - p * a.Q;
        ih0[i] = in ? p * a.stride_h - a.pad_h : -(1 << 28);      // fails every bounds check: the row is zero-filled
        iw0[i] = q * a.stride_w - a.pad_w;
        row0[i] = img * a.H;
    }
    int ta = (s0 * 8 + (tid & 7)) / c4n, ca = (s0 * 8 + (tid & 7)) - ta * c4n;      // filter tap and channel group of the chunk
    int ra = ta / a.S, sa = ta - ra * a.S;
    size_t src[2];
    bool ok[2];                                    // the pixels' chunks (in units of 16 bytes) and whether they exist, for this tap
    auto locate = [&]() {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int ih = ih0[i] + ra * a.dil_h, iw = iw0[i] + sa * a.dil_w;
            ok[i] = ta < taps && (unsigned)ih < (unsigned)a.H && (unsigned)iw < (unsigned)a.W;
            src[i] = ok[i] ? ((size_t)(row0[i] + ih) * a.W + iw) * c4n + ca : 0;
        }
    };
    locate();
    // ---- and of the packed weights [tap][Cs][Kp]: row kb (of 32), then every kRowStep-th, four channels each ----
    constexpr int kCols = BN / 4, kRowStep = kBlock / kCols, kCopies = (kTK + kRowStep - 1) / kRowStep;
    const int kb = tid / kCols, nb = (tid % kCols) * 4;
    int rows_left = n0 + nb < f.Kp ? taps * a.Cs - (s0 * kTK + kb) : 0;       // rows from this one to the last
    uint32_t wsrc = (uint32_t)(s0 * kTK + kb) * (uint32_t)f.Kp + (uint32_t)(n0 + nb);

    // Pixel m of k row kk is word kk * 64 + (m ^ (kk / 4 % 8 * 4)): a warp's 4-byte copies (8 chunks x 4 pixels) and the
    // threads' 16-byte reads of 4 pixels are both free of bank conflicts.
    const uint32_t chunk = (uint32_t)tid & 7u;
    const uint32_t da0 = smem_u32(smem) + (chunk * 4u * kTM + (((uint32_t)tid >> 3) ^ (chunk * 4u))) * 4u;
    const uint32_t db0 = smem_u32(smem) + (uint32_t)(kTK * kTM + kb * BN + nb) * 4u;
    auto fill = [&](int buf) {
        const uint32_t da = da0 + (uint32_t)(buf * kStageFloats) * 4u, db = db0 + (uint32_t)(buf * kStageFloats) * 4u;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float* g = static_cast<const float*>(a.x) + src[i] * 4;
#pragma unroll
            for (int j = 0; j < 4; ++j)      // +32 pixels: the XOR stays below bit 5
                cp_async<4>(da + (uint32_t)(j * kTM) * 4u + (uint32_t)(i * 32) * 4u, g + j, ok[i] && (!Padded || ca * 4 + j < a.C));
        }
#pragma unroll
        for (int i = 0; i < kCopies; ++i)
            if (kTK % kRowStep == 0 || kb + i * kRowStep < kTK) {
                const bool in = i * kRowStep < rows_left;
                const float* g = static_cast<const float*>(a.w) + (in ? wsrc + (uint32_t)(i * kRowStep) * (uint32_t)f.Kp : 0u);
                if (Aligned) {
                    cp_async<16>(db + (uint32_t)(i * kRowStep * BN) * 4u, g, in);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) cp_async<4>(db + (uint32_t)(i * kRowStep * BN + j) * 4u, g + j, in);
                }
            }
        rows_left -= kTK;
        wsrc += (uint32_t)kTK * (uint32_t)f.Kp;
        // the next stage's chunk: eight further on, in the same tap or a later one
        ca += 8;
        if (ca < c4n) {
#pragma unroll
            for (int i = 0; i < 2; ++i) src[i] += ok[i] ? 8u : 0u;
        } else {
            do {
                ca -= c4n;
                ++ta;
                if (++sa == a.S) { sa = 0; ++ra; }
            } while (ca >= c4n);
            locate();
        }
    };

    float acc[8][TJ];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TJ; ++j) acc[i][j] = 0.f;
    // pixels tm*4 .. +3 and 32 further on; channels tn*4 .. +3 and (TJ == 8) BN/2 further on
    const int grp = tid / kGroupThreads, tm = tid & 7, tn = (tid % kGroupThreads) >> 3;

#pragma unroll
    for (int d = 0; d < kDepth - 1; ++d) {
        if (s0 + d < s1) fill(d);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int buf = 0, fill_buf = kDepth - 1;
    for (int s = s0; s < s1; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 2) : "memory");
        __syncthreads();                 // the stage has landed for everyone; everyone is done with the buffer refilled next
        if (s + kDepth - 1 < s1) fill(fill_buf);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* As = smem + buf * kStageFloats + grp * kGroupK * kTM;
        const float* Bs = smem + buf * kStageFloats + kTK * kTM + grp * kGroupK * BN + tn * 4;
        float av[2][8], bv[2][TJ];
        auto load = [&](int q) {
            const float* ar = As + q * kTM + ((tm ^ ((grp * kGroupK + q) >> 2 & 7)) << 2);
            *reinterpret_cast<float4*>(av[q & 1]) = *reinterpret_cast<const float4*>(ar);
            *reinterpret_cast<float4*>(av[q & 1] + 4) = *reinterpret_cast<const float4*>(ar + 32);
            *reinterpret_cast<float4*>(bv[q & 1]) = *reinterpret_cast<const float4*>(Bs + q * BN);
            if constexpr (TJ == 8) *reinterpret_cast<float4*>(bv[q & 1] + 4) = *reinterpret_cast<const float4*>(Bs + q * BN + BN / 2);
        };
        load(0);
#pragma unroll
        for (int q = 0; q < kGroupK; ++q) {
            if (q + 1 < kGroupK) load(q + 1);          // under this k's multiplications
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TJ; ++j) acc[i][j] = fmaf(av[q & 1][i], bv[q & 1][j], acc[i][j]);
        }
        if (++buf == kDepth) buf = 0;
        if (++fill_buf == kDepth) fill_buf = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // ---- the groups' partial tiles meet in shared memory ----
    float* red = smem;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float* row = red + (grp * kTM + tm * 4 + (i & 3) + (i >> 2) * 32) * kLdR + tn * 4;
        *reinterpret_cast<float4*>(row) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        if constexpr (TJ == 8) *reinterpret_cast<float4*>(row + BN / 2) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
    }
    __syncthreads();
    constexpr int kVecs = kTM * BN / 4;
    const bool vec = ((a.Ks | a.out_c_off) & 3) == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
    for (int v = tid; v < kVecs; v += kBlock) {
        const int row = v / (BN / 4), col = (v - row * (BN / 4)) * 4;
        float4 s = *reinterpret_cast<const float4*>(red + row * kLdR + col);
#pragma unroll
        for (int g = 1; g < kGroups; ++g) s = add4(s, *reinterpret_cast<const float4*>(red + (g * kTM + row) * kLdR + col));
        if (f.splits == 1) {
            if (m0 + row < f.M && n0 + col < a.K) finish4(a, m0 + row, n0 + col, s, vec);
        } else {
            *reinterpret_cast<float4*>(red + row * kLdR + col) = s;
        }
    }
    if (f.splits > 1) {
        // ---- and the ranks' sums through distributed shared memory: each rank finishes a share of the tile ----
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        const int v1 = kVecs * (rank + 1) / f.splits;
        for (int v = kVecs * rank / f.splits + tid; v < v1; v += kBlock) {
            const int row = v / (BN / 4), col = (v - row * (BN / 4)) * 4;
            const uint32_t at = smem_u32(red + row * kLdR + col);
            float4 part[8];          // every rank's sum on its way before the first is used
#pragma unroll
            for (int z = 0; z < 8; ++z)
                if (z < f.splits) part[z] = ld_cluster(at, (uint32_t)z);
            float4 s = part[0];
#pragma unroll
            for (int z = 1; z < 8; ++z)
                if (z < f.splits) s = add4(s, part[z]);
            if (m0 + row < f.M && n0 + col < a.K) finish4(a, m0 + row, n0 + col, s, vec);
        }
        asm volatile("barrier.cluster.arrive.relaxed;\n\tbarrier.cluster.wait.acquire;" ::: "memory");      // every rank has been read
    }
    griddep_launch();
    if (nf) {
        if (f.declared) nf->end_as(job_id, f.declared);
        else nf->end(job_id);
    }
}

struct F32Geometry {
    int BN, m_tiles, n_tiles, splits, n_stages;
    double load;                // stages that the fullest SM works on at a time
    uint32_t smem;
    const void* fn;
};

int batch_of(const pb_op_params* p) { return p->batch > 1 ? p->batch : 1; }

F32Geometry conv_f32_geometry(const pb_op_params* p) {
    F32Geometry g;
    g.BN = p->K > 32 ? 64 : (p->K > 16 ? 32 : 16);
    g.m_tiles = ceil_div(batch_of(p) * p->P * p->Q, kTM);
    g.n_tiles = ceil_div(p->K, g.BN);
    g.n_stages = ceil_div(p->R * p->S * p->Cs, kTK);
    // Split: least modelled time of a lone launch.  A stage of a 64-column tile takes an SM 1.0 us whether one block runs or
    // two side by side (measured), so what counts is how many stages the fullest SM gets: one block as long as the launch
    // fits one per SM, else two, then in waves.  Clusters reach fewer SMs than lone blocks (measured with idle kernels).
    // A launch costs 5 us besides, a split 1.5 to 2.7 us (two cluster barriers and the exchange).
    static const int kOnePerSm[9] = {0, 148, 148, 135, 132, 130, 132, 0, 120}, kTwoPerSm[9] = {0, 296, 296, 279, 284, 280, 270, 0, 264};
    const int tiles = g.m_tiles * g.n_tiles;
    g.splits = 1;
    double best = 1e30;
    for (int S = 1; S <= 8; ++S) {
        if (S > 1 && (g.n_stages < 2 * S || conv_split_gain_us() > 1e6)) break;
        if (S == 7) continue;      // two clusters of 7 on a GPC's SMs leave the rest idle: 47 us where 5 takes 37
        const int blocks = tiles * S;
        const double load = blocks <= kOnePerSm[S] ? 1.0 : (S == 1 ? std::max(2.0, blocks / 148.0) : 2.0 * ceil_div(blocks, kTwoPerSm[S]));
        const double us = load * ceil_div(g.n_stages, S) * g.BN / 64.0 + (S > 1 ? 1.5 + 0.15 * S : 0.0);
        if (us < best) { best = us; g.splits = S; g.load = load; }
    }
    const int groups = g.BN == 16 ? 8 : 4;
    const size_t pipe = (size_t)kDepth * (kTK * kTM + kTK * g.BN) * 4, red = (size_t)groups * kTM * (g.BN + 4) * 4;
    g.smem = (uint32_t)std::max(pipe, red);
    const bool wide = ((uintptr_t)p->w & 15) == 0, padded = p->C != p->Cs;
#define PB_F32(BN_) (padded ? (wide ? (const void*)conv_f32_kernel<BN_, true, true> : (const void*)conv_f32_kernel<BN_, false, true>) \
                            : (wide ? (const void*)conv_f32_kernel<BN_, true, false> : (const void*)conv_f32_kernel<BN_, false, false>))
    g.fn = g.BN == 64 ? PB_F32(64) : (g.BN == 32 ? PB_F32(32) : PB_F32(16));
#undef PB_F32
    return g;
}

bool aligned(const pb_op_params* p) { return (((uintptr_t)p->x | (uintptr_t)p->w) & 15) == 0; }

}  // namespace

// Dense fp32 layers; the rest (groups, a handful of outputs) keeps conv_simt_kernel, whose thread per output is the better
// shape for reductions of a few values.
bool conv_f32_supported(const pb_op_params* p) {
    return p->dtype == 0 && p->groups <= 1 && p->Cs % 4 == 0 && p->K >= 8 && p->R * p->S * p->Cs >= 16 && (uint64_t)p->R * p->S * (p->Cs + 32) * (p->K + 64) <= 0xffffffffull;
}

// Fitted to 476 measured 3x3, 5x5 and 1x7 layers (24 to 512 channels, maps of 7 x 7 to 112 x 112, 1 to 8 images; 4 % off in the mean).
double conv_f32_units_us(const pb_op_params* p) {
    const F32Geometry g = conv_f32_geometry(p);
    return (g.BN == 16 ? 2.5 : 2.6) + g.load * (1.2 + (g.BN == 16 ? 0.456 : 0.65) * ceil_div(g.n_stages, g.splits)) + (g.splits > 1 ? 0.3 + 0.07 * g.splits : 0.0);
}

// [tap][Cs][K rounded up to 4], zero past C and K.
int64_t conv_f32_pack_weights(const pb_op_params* p, const float* w, void* dst) {
    const int taps = p->R * p->S, Kp = round_up(p->K, 4);
    const size_t n = (size_t)taps * p->Cs * Kp;
    if (dst) {
        float* d = static_cast<float*>(dst);
        memset(d, 0, n * 4);
        for (int k = 0; k < p->K; ++k)
            for (int c = 0; c < p->C; ++c)
                for (int t = 0; t < taps; ++t) d[((size_t)t * p->Cs + c) * Kp + k] = w[((size_t)k * p->C + c) * taps + t];
    }
    return (int64_t)(n * 4);
}

int conv_f32_info(const pb_op_params* p, pb_launch_info* out) {
    const F32Geometry g = conv_f32_geometry(p);
    memset(out, 0, sizeof(*out));
    out->kind = PB_STAGE_CONV_SIMT;
    out->num_blocks = (uint32_t)(g.m_tiles * g.n_tiles * g.splits);
    out->threads_per_block = kBlock;
    cudaFuncAttributes at;
    out->regs_per_thread = 128;
    if (cudaFuncGetAttributes(&at, g.fn) == cudaSuccess) out->regs_per_thread = (uint32_t)at.numRegs;
    else cudaGetLastError();
    out->smem_per_block = g.smem;
    if (conv_f32_split_layer(p)) {
        // The blocks do not depend on where the tensors are: the launch may be declared before that is known.
        pb_launch_info split = *out;
        conv_f32_split_info(p, &split);
        if (aligned(p)) *out = split;
        else out->num_blocks = split.num_blocks;
    }
    const uint64_t nb = (uint64_t)batch_of(p), y = nb * p->K * p->P * p->Q;
    out->flops = 2ull * y * p->C * p->R * p->S;
    out->bytes = 4ull * (nb * p->C * p->H * p->W + (uint64_t)p->K * p->C * p->R * p->S + y + (p->residual ? y : 0)) + 4ull * p->K;
    return PB_OK;
}

int conv_f32_launch(const pb_op_params* p, const OpArgs& op, cudaStream_t st, uint32_t job_id, void* notifier, bool pdl) {
    const bool split = conv_f32_split_layer(p);
    if (split && aligned(p)) return conv_f32_split_launch(p, op, st, job_id, notifier, pdl);
    const F32Geometry g = conv_f32_geometry(p);
    F32Args f;
    f.op = op;
    f.PQ = p->P * p->Q;
    f.M = batch_of(p) * f.PQ;
    f.Kp = round_up(p->K, 4);
    f.n_stages = g.n_stages;
    f.splits = g.splits;
    f.declared = 0;
    if (split) {
        pb_launch_info li;
        conv_f32_split_info(p, &li);
        f.declared = li.num_blocks;
    }
    PB_CUDA(cudaFuncSetAttribute(g.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)g.m_tiles, (unsigned)g.n_tiles, (unsigned)g.splits);
    cfg.blockDim = dim3(kBlock);
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
    PB_CUDA(cudaLaunchKernelEx(&cfg, (void (*)(const F32Args, uint32_t, FinishedBlockNotifier*))g.fn, f, job_id, static_cast<FinishedBlockNotifier*>(notifier)));
    return PB_OK;
}

}  // namespace pb
