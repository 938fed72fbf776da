// Inference operators other than the tensor-core convolution: channels-last
// ([H][W][Cs]) kernels for layout conversion, direct (SIMT) convolution, depthwise
// convolution, pooling, dense, add and softmax.  These are the memory-bound members
// of the kernel family the reference's TVM adapters launch
// (jobs/tvm_<model>/tvm_<model>.cpp:24-47); every kernel reports block start/end on
// the job's notifier exactly once per block.
//
// Access pattern: the channel dimension is innermost and padded to a 16-byte vector
// (4 fp32 / 8 bf16), so one thread moves one 128-bit vector and a warp reads a
// contiguous 512-byte span whenever Cs >= 32 vectors.
#include <cuda.h>
#include <cuda_bf16.h>
#include <llis/job/finished_block_notifier.h>

#include <cstdlib>
#include <cstring>

#include "launch_slot.cuh"
#include "ops.h"
#include "pb_common.h"

using llis::job::FinishedBlockNotifier;

namespace pb {

// ---- 128-bit vectors of activations ---------------------------------------
template <typename T> struct Vec;
template <> struct Vec<float> {
    static constexpr int N = 4;
    float v[4];
    __device__ __forceinline__ static Vec load(const float* p) {
        Vec r; const float4 t = *reinterpret_cast<const float4*>(p);
        r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w; return r;
    }
    __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};
template <> struct Vec<__nv_bfloat16> {
    static constexpr int N = 8;
    float v[8];
    __device__ __forceinline__ static Vec load(const __nv_bfloat16* p) {
        Vec r; const uint4 t = *reinterpret_cast<const uint4*>(p);
        const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            r.v[2 * i] = __uint_as_float(u[i] << 16);
            r.v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
        return r;
    }
    __device__ __forceinline__ void store(__nv_bfloat16* p) const {
        uint32_t u[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            u[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(u[0], u[1], u[2], u[3]);
    }
};

template <typename T> __device__ __forceinline__ float to_f(T x);
template <> __device__ __forceinline__ float to_f<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ float act_fn(float v, int act) {
    if (act == 1) return fmaxf(v, 0.f);
    if (act == 2) return fminf(fmaxf(v, 0.f), 6.f);
    return v;
}

// Every kernel here may be launched as a programmatic dependent of the previous kernel of its stage
// graph: it waits for that kernel on the device before touching memory (a no-op otherwise).  PB_NOTIFY_START_EARLY then lets
// the next kernel's blocks in, which set themselves up (tensor memory, barriers, first weights) while this one runs: 2.0 us
// from this kernel's end to the next one's first instruction after its wait without that trigger, 0.75 us with it (window3_tile_kernel
// has none: not measured there).
// Only where this kernel is short, so that the blocks that wait hold their SM slots for a microsecond or two (the input kernels
// take 8 to 25 us: triggered at their start, 32 ResNet-18 requests took 833 instead of 808 us), and only in bf16: the
// full-precision convolution's blocks, when they come in beside other blocks, are dealt two to an SM while others idle
// (ResNet-18 of two images: 430 -> 447 us).
#define PB_NOTIFY_START()                                        \
    pb::griddep_wait();                                           \
    const pb::LaunchSlot* slot_ = pb::resolve_slot(job_id, nf);  \
    (void)slot_;                                                  \
    if (nf) nf->start(job_id)
#define PB_NOTIFY_START_EARLY(T)                                  \
    PB_NOTIFY_START();                                            \
    if constexpr (sizeof(T) == 2) pb::griddep_launch()
#define PB_NOTIFY_END() if (nf) nf->end(job_id)

// Batched launches (a gang of requests of one model): blockIdx.y is the image.  Image i of an
// activation tensor follows image i - 1 without padding, so the tensor-core convolution sees the
// images as one [batch * pixels][channels] matrix.
template <typename T> __device__ __forceinline__ const T* x_img(const OpArgs& a) {
    return static_cast<const T*>(a.x) + (size_t)blockIdx.y * a.H * a.W * a.Cs;
}
template <typename T> __device__ __forceinline__ T* y_img(const OpArgs& a) {
    return static_cast<T*>(a.y) + (size_t)blockIdx.y * a.P * a.Q * a.Ks;
}
// fp32 model output of this image (a.flags & 2): the request's own buffer when a.y is NULL
__device__ __forceinline__ float* out_f32_img(const OpArgs& a, const pb::LaunchSlot* slot, int n_out) {
    return (!a.y && slot) ? slot->io_out[blockIdx.y] : static_cast<float*>(a.y) + (size_t)blockIdx.y * n_out;
}

// ---- NCHW fp32 -> channels-last T ------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) input_transform_kernel(const float* x, T* __restrict__ y, int C, int HW,
                                                              int Cs, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    x = (!x && slot_) ? slot_->io_in[blockIdx.y] : x + (size_t)blockIdx.y * C * HW;   // the request's input buffer, known only at dispatch
    y += (size_t)blockIdx.y * HW * Cs;
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix < HW) {
        for (int c0 = 0; c0 < Cs; c0 += Vec<T>::N) {
            Vec<T> o;
#pragma unroll
            for (int j = 0; j < Vec<T>::N; ++j) o.v[j] = (c0 + j < C) ? x[(size_t)(c0 + j) * HW + pix] : 0.f;
            o.store(y + (size_t)pix * Cs + c0);
        }
    }
    PB_NOTIFY_END();
}

// ---- NCHW fp32 -> patch matrix [P*Q][Ks] ------------------------------------------------
// The first convolution of an image model has 3 input channels: as an implicit GEMM every filter tap
// would be padded to a 64-channel k-block (1/21 useful).  This kernel writes the im2col rows themselves,
// y[(p, q)][k] with k = (r*S + s)*C + c (zero for k >= R*S*C and outside the image), so that the
// convolution becomes a pointwise one over R*S*C "channels": 1 k-block instead of 9 for a 3x3 stem,
// 3 instead of 49 for a 7x7 one.  One thread per (output pixel, 8 consecutive k).
template <typename T>
__global__ void __launch_bounds__(256) input_patch_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    const float* __restrict__ x = (!a.x && slot_) ? slot_->io_in[blockIdx.y]      // the request's input buffer, known only at dispatch
                                                  : static_cast<const float*>(a.x) + (size_t)blockIdx.y * a.C * a.H * a.W;
    constexpr int N = Vec<T>::N;
    const int kv = a.Ks / N;
    const int total = a.P * a.Q * kv;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) {
        const int k0 = (idx % kv) * N;
        const int pix = idx / kv;
        const int q = pix % a.Q, p = pix / a.Q;
        const int taps_c = a.R * a.S * a.C;
        Vec<T> o;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int k = k0 + j;
            float v = 0.f;
            if (k < taps_c) {
                const int tap = k / a.C, c = k - tap * a.C;
                const int r = tap / a.S, s = tap - r * a.S;
                const int ih = p * a.stride_h + r - a.pad_h, iw = q * a.stride_w + s - a.pad_w;
                if (ih >= 0 && ih < a.H && iw >= 0 && iw < a.W) v = __ldg(x + ((size_t)c * a.H + ih) * a.W + iw);
            }
            o.v[j] = v;
        }
        o.store(y_img<T>(a) + (size_t)pix * a.Ks + k0);
    }
    PB_NOTIFY_END();
}

// The same patch matrix, a tile of output pixels per block.  input_patch_kernel reads every input value through eight
// scattered 4-byte loads per output vector (each value about 2.25 times, with the index arithmetic of its filter tap
// every time) and holds a block slot for 256 output vectors; under serving load that costs more than its share of a
// lone request (6.7 % of the Inception-v3 throughput, measured by leaving it out).  Here a block first copies the
// window of its kPatchTileP x kPatchTileQ output pixels into shared memory, as T (zero outside the image): a warp takes rows
// of the window and has twelve coalesced loads in flight.  Then it writes its output vectors from there.  A thread keeps
// ONE vector position k0 for all its pixels, so the eight offsets of its values in the window are registers; consecutive
// threads write consecutive vectors.  Bound by those 2-byte reads of shared memory (a value is read R*S / stride^2 times).
// (Offsets looked up in a table in shared memory for every value, and fp32 values there: the table's reads alone were 8-way
// bank conflicts; 8 images of 224 x 224, 7 x 7 stride 2: 25 us.)  Same values, same rounding: identical bits.
constexpr int kPatchTileP = 8, kPatchTileQ = 32;
__host__ __device__ __forceinline__ int patch_tile_rows(int R, int sh) { return (kPatchTileP - 1) * sh + R; }
__host__ __device__ __forceinline__ int patch_tile_cols(int S, int sw) { return (kPatchTileQ - 1) * sw + S; }

__device__ __forceinline__ void patch_store(float* y, const float (&v)[4]) { *reinterpret_cast<float4*>(y) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void patch_store(__nv_bfloat16* y, const __nv_bfloat16 (&v)[8]) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = (uint32_t)__bfloat16_as_ushort(v[2 * i]) | (uint32_t)__bfloat16_as_ushort(v[2 * i + 1]) << 16;
    *reinterpret_cast<uint4*>(y) = make_uint4(u[0], u[1], u[2], u[3]);
}

template <typename T>
__global__ void __launch_bounds__(256) input_patch_tile_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    extern __shared__ __align__(16) unsigned char s_patch[];
    const float* __restrict__ x = (!a.x && slot_) ? slot_->io_in[blockIdx.y]      // the request's input buffer, known only at dispatch
                                                  : static_cast<const float*>(a.x) + (size_t)blockIdx.y * a.C * a.H * a.W;
    constexpr int N = Vec<T>::N;
    const int rows = patch_tile_rows(a.R, a.stride_h), cols = patch_tile_cols(a.S, a.stride_w);
    T* s_win = reinterpret_cast<T*>(s_patch);                     // [C][rows][cols]
    const int tiles_q = (a.Q + kPatchTileQ - 1) / kPatchTileQ;
    const int p0 = (blockIdx.x / tiles_q) * kPatchTileP, q0 = (blockIdx.x % tiles_q) * kPatchTileQ;
    const int ih0 = p0 * a.stride_h - a.pad_h, iw0 = q0 * a.stride_w - a.pad_w;

    const int lane = threadIdx.x & 31, n_rows = a.C * rows;
    for (int row0 = threadIdx.x >> 5; row0 < n_rows; row0 += 32) {
        for (int col0 = lane; col0 < cols; col0 += 96) {
            float v[4][3];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int row = row0 + 8 * u, c = row / rows, ih = ih0 + row - c * rows;
                const bool row_ok = row < n_rows && (unsigned)ih < (unsigned)a.H;
                const float* __restrict__ g = x + ((ptrdiff_t)c * a.H + ih) * a.W + iw0;
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    const int col = col0 + 32 * t;
                    v[u][t] = row_ok && col < cols && (unsigned)(iw0 + col) < (unsigned)a.W ? __ldg(g + col) : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int t = 0; t < 3; ++t)
                    if (row0 + 8 * u < n_rows && col0 + 32 * t < cols) s_win[(row0 + 8 * u) * cols + col0 + 32 * t] = from_f<T>(v[u][t]);
        }
    }
    // this thread's vector of k, where its values lie in a pixel's window, and its first pixel
    const int kv = a.Ks / N, groups = 256 / kv;
    const int grp = threadIdx.x / kv, k0 = (threadIdx.x - grp * kv) * N;
    int off[N];
    uint32_t real = 0;                       // values of the filter window; the others are zeros
    {
        int c = k0 % a.C, s2 = k0 / a.C % a.S, r = k0 / (a.C * a.S);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            real |= (r < a.R ? 1u : 0u) << j;
            off[j] = r < a.R ? (c * rows + r) * cols + s2 : 0;
            if (++c == a.C) {
                c = 0;
                if (++s2 == a.S) { s2 = 0; ++r; }
            }
        }
    }
    __syncthreads();
    if constexpr (sizeof(T) == 2) pb::griddep_launch();      // the window has arrived: what is left is short
    if (grp < groups) {
        T* __restrict__ y = y_img<T>(a) + k0;
#pragma unroll 2
        for (int px = grp; px < kPatchTileP * kPatchTileQ; px += groups) {
            const int pr = px / kPatchTileQ, pc = px % kPatchTileQ;
            const int p = p0 + pr, q = q0 + pc;
            if (p >= a.P || q >= a.Q) continue;
            const T* __restrict__ w = s_win + pr * a.stride_h * cols + pc * a.stride_w;
            T o[N];
#pragma unroll
            for (int j = 0; j < N; ++j) o[j] = (real >> j) & 1u ? w[off[j]] : from_f<T>(0.f);
            patch_store(y + ((size_t)p * a.Q + q) * a.Ks, o);
        }
    }
    PB_NOTIFY_END();
}
// Dynamic shared memory of the tiled patch kernel, or 0 when the layer keeps input_patch_kernel (a window that does
// not fit, more than 256 values of k).
static size_t patch_tile_smem(const pb_op_params* p) {
    if (p->Ks > 256 || p->R * p->S <= 1) return 0;
    const size_t n = (size_t)p->C * patch_tile_rows(p->R, p->stride_h) * patch_tile_cols(p->S, p->stride_w) * (p->dtype == 0 ? 4 : 2);
    return n <= 40 * 1024 ? n : 0;
}
static uint32_t patch_tile_blocks(const pb_op_params* p) {
    return (uint32_t)(((p->P + kPatchTileP - 1) / kPatchTileP) * ((p->Q + kPatchTileQ - 1) / kPatchTileQ));
}

// ---- direct convolution ------------------------------------------------------
// One thread per (output pixel, output channel).  Weights [R][S][C/groups][K]: a warp
// reads consecutive k (coalesced) and shares the input value (broadcast).
template <typename T>
__global__ void __launch_bounds__(256) conv_simt_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    const T* __restrict__ x = x_img<T>(a);
    const T* __restrict__ w = static_cast<const T*>(a.w);
    const int total = a.P * a.Q * a.K;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) {
        const int k = idx % a.K;
        const int pix = idx / a.K;
        const int q = pix % a.Q, p = pix / a.Q;
        const int cg = a.C / a.groups;
        const int g = k / (a.K / a.groups);
        float acc = 0.f;
        for (int r = 0; r < a.R; ++r) {
            const int ih = p * a.stride_h + r * a.dil_h - a.pad_h;
            if (ih < 0 || ih >= a.H) continue;
            for (int s = 0; s < a.S; ++s) {
                const int iw = q * a.stride_w + s * a.dil_w - a.pad_w;
                if (iw < 0 || iw >= a.W) continue;
                const T* xp = x + ((size_t)ih * a.W + iw) * a.Cs + g * cg;
                const T* wp = w + ((size_t)(r * a.S + s) * cg) * a.K + k;
                for (int c = 0; c < cg; ++c) acc = fmaf(to_f<T>(xp[c]), to_f<T>(wp[(size_t)c * a.K]), acc);
            }
        }
        if (a.bias) acc += a.bias[k];
        if (a.residual) acc += to_f<T>(static_cast<const T*>(a.residual)[((size_t)blockIdx.y * a.P * a.Q + pix) * a.res_Cs + k]);
        if (a.act == 3) acc = acc > 0.f ? acc : acc * a.bias[a.K + k];      // PReLU: slopes follow the biases
        else acc = act_fn(acc, a.act);
        y_img<T>(a)[(size_t)pix * a.Ks + a.out_c_off + k] = from_f<T>(acc);
    }
    PB_NOTIFY_END();
}

// ---- depthwise convolution -----------------------------------------------------
// One thread per (output pixel, channel vector); weights [R][S][Cs].
template <typename T>
__global__ void __launch_bounds__(256, 6) dwconv_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    const int cv = a.Cs / N;
    const int total = a.P * a.Q * cv;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) {
        const int c0 = (idx % cv) * N;
        const int pix = idx / cv;
        const int q = pix % a.Q, p = pix / a.Q;
        const T* __restrict__ x = x_img<T>(a);
        const T* __restrict__ w = static_cast<const T*>(a.w);
        float acc[N];
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] = 0.f;
        for (int r = 0; r < a.R; ++r) {
            const int ih = p * a.stride_h + r - a.pad_h;
            if (ih < 0 || ih >= a.H) continue;
            for (int s = 0; s < a.S; ++s) {
                const int iw = q * a.stride_w + s - a.pad_w;
                if (iw < 0 || iw >= a.W) continue;
                const Vec<T> xv = Vec<T>::load(x + ((size_t)ih * a.W + iw) * a.Cs + c0);
                const Vec<T> wv = Vec<T>::load(w + (size_t)(r * a.S + s) * a.Cs + c0);
#pragma unroll
                for (int j = 0; j < N; ++j) acc[j] = fmaf(xv.v[j], wv.v[j], acc[j]);
            }
        }
        Vec<T> o;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float v = acc[j] + ((a.bias && c0 + j < a.K) ? a.bias[c0 + j] : 0.f);
            o.v[j] = (c0 + j < a.K) ? act_fn(v, a.act) : 0.f;
        }
        o.store(y_img<T>(a) + (size_t)pix * a.Ks + a.out_c_off + c0);
    }
    PB_NOTIFY_END();
}

// ---- pooling -------------------------------------------------------------------
template <typename T, bool kMax>
__global__ void __launch_bounds__(256, 6) pool_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    const int cv = a.Cs / N;
    const int total = a.P * a.Q * cv;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < total) {
        const int c0 = (idx % cv) * N;
        const int pix = idx / cv;
        const int q = pix % a.Q, p = pix / a.Q;
        const T* __restrict__ x = x_img<T>(a);
        float acc[N];
#pragma unroll
        for (int j = 0; j < N; ++j) acc[j] = kMax ? -INFINITY : 0.f;
        int cnt = 0;
        for (int r = 0; r < a.R; ++r) {
            const int ih = p * a.stride_h + r - a.pad_h;
            if (ih < 0 || ih >= a.H) continue;
            float row[N];                     // average pooling: the columns of a row first
#pragma unroll
            for (int j = 0; j < N; ++j) row[j] = 0.f;
            for (int s = 0; s < a.S; ++s) {
                const int iw = q * a.stride_w + s - a.pad_w;
                if (iw < 0 || iw >= a.W) continue;
                const Vec<T> xv = Vec<T>::load(x + ((size_t)ih * a.W + iw) * a.Cs + c0);
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    if (kMax) acc[j] = fmaxf(acc[j], xv.v[j]);
                    else row[j] += xv.v[j];
                }
                ++cnt;
            }
            if (!kMax) {
#pragma unroll
                for (int j = 0; j < N; ++j) acc[j] += row[j];
            }
        }
        Vec<T> o;
        const float div = (a.flags & 1) ? (float)(a.R * a.S) : (float)(cnt > 0 ? cnt : 1);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float v = kMax ? acc[j] : acc[j] / div;
            if (a.bias && c0 + j < a.C) v += a.bias[c0 + j];      // the tail of a convolution that ran before the pooling
            o.v[j] = (c0 + j < a.C) ? act_fn(v, a.act) : 0.f;
        }
        o.store(y_img<T>(a) + (size_t)pix * a.Ks + a.out_c_off + c0);
    }
    PB_NOTIFY_END();
}

// ---- 3x3 windows over large tensors: a strip of output pixels per thread ------------------
// dwconv_kernel and pool_kernel issue one guarded 128-bit load per filter tap and output vector: on a
// tensor that fills the GPU each thread has about one load in flight at a time and every input vector is
// fetched up to nine times through L1, so they run at the latency of the load path, not at HBM speed
// (depthwise 3x3 stride 1 at 128 x 1024 x 1024 bf16: 19 % of the measured copy bandwidth).  Here a thread
// owns one channel vector of kStrip consecutive output pixels of one output row.  Per input row it issues
// ALL loads of the strip's window back to back, unconditionally (addresses clamped into the tensor, the
// taps that fall outside are dropped afterwards), so 6-9 loads per thread are in flight; each loaded
// vector feeds every output it belongs to, and a row of weights is loaded once per thread.
// The order of the additions per output is the one of dwconv_kernel / pool_kernel (depthwise: rows, then columns; average:
// the columns of each row, then the rows), so results are bit-identical to theirs.  Used when the strips alone fill the GPU (strip_threads()).
// With kStrip = 1 (every other 3x3 layer of stride 1 or 2, i.e. the batch-1 layers of the served models)
// the thread owns one output vector as in dwconv_kernel / pool_kernel, but its nine loads are
// unconditional and in flight together instead of one guarded load after the other.
constexpr int kStripWide1 = 4, kStripWide2 = 2;   // stride 1: 18 loads per thread; stride 2: 15
enum { kWinDw = 0, kWinMax = 1, kWinAvg = 2 };

template <typename T> struct RawVec;
template <> struct RawVec<float> { typedef float4 type; };
template <> struct RawVec<__nv_bfloat16> { typedef uint4 type; };
__device__ __forceinline__ Vec<float> vec_of(const float4& t) {
    Vec<float> r; r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w; return r;
}
__device__ __forceinline__ Vec<__nv_bfloat16> vec_of(const uint4& t) {
    Vec<__nv_bfloat16> r;
    const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        r.v[2 * i] = __uint_as_float(u[i] << 16);
        r.v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
    }
    return r;
}

// Pairs of fp32 values.  PB_F32X2=1 keeps a pair in one 64-bit register and uses the packed fp32
// instructions of sm_100 (fma.rn.f32x2 / add.rn.f32x2: each half is the IEEE operation of the scalar
// instruction); otherwise the pair is two scalars and the compiler schedules scalar instructions.
#ifndef PB_F32X2
#define PB_F32X2 0
#endif
#if PB_F32X2
typedef uint64_t f2_t;
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
    f2_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
    f2_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
    f2_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_max(f2_t a, f2_t b) {
    float a0, a1, b0, b1;
    f2_unpack(a, a0, a1);
    f2_unpack(b, b0, b1);
    return f2_pack(fmaxf(a0, b0), fmaxf(a1, b1));
}
#else
struct f2_t { float lo, hi; };
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) { f2_t r; r.lo = lo; r.hi = hi; return r; }
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) { lo = v.lo; hi = v.hi; }
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) { return f2_pack(fmaf(a.lo, b.lo, c.lo), fmaf(a.hi, b.hi, c.hi)); }
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) { return f2_pack(a.lo + b.lo, a.hi + b.hi); }
__device__ __forceinline__ f2_t f2_max(f2_t a, f2_t b) { return f2_pack(fmaxf(a.lo, b.lo), fmaxf(a.hi, b.hi)); }
#endif
// A 128-bit vector of activations as fp32 pairs: 2 pairs from float4, 4 pairs from 8 bf16.
__device__ __forceinline__ void unpack_pairs(const float4& t, f2_t (&r)[2]) {
    r[0] = f2_pack(t.x, t.y);
    r[1] = f2_pack(t.z, t.w);
}
__device__ __forceinline__ void unpack_pairs(const uint4& t, f2_t (&r)[4]) {
    const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = f2_pack(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xffff0000u));
}

// Dynamic shared memory of a depthwise launch: filter [3][3][Cs] + fp32 biases [Cs], or 0 when that
// exceeds what a kernel gets without opting in (the kernel then reads the filter from global memory).
__host__ __device__ __forceinline__ int window3_smem_bytes(int Cs, int elem_bytes) {
    const int n = 9 * Cs * elem_bytes + 4 * Cs;
    return n <= 40 * 1024 ? n : 0;
}

template <typename T, int kMode, int kStride, int kStrip>
__global__ void __launch_bounds__(256, 2) window3_strip_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    constexpr int NP = N / 2;
    constexpr int kCols = (kStrip - 1) * kStride + 3;
    typedef typename RawVec<T>::type Raw;
    const int cv = a.Cs / N;
    const int strips = (a.Q + kStrip - 1) / kStrip;
    const int total = a.P * strips * cv;
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    // Depthwise: the block's copy of the filter ([3][3][Cs]) and of the biases, in shared memory.  Read
    // through L1 they compete with the streamed activations for cache lines, and a miss sits on every
    // thread's critical path three times; the host passes window3_smem_bytes() of dynamic shared memory
    // (0 = the filter does not fit: read it from global memory).  Wide strips only: on a batch-1 layer the
    // staging round trip would come before the first activation load of a block that lives a few microseconds.
    extern __shared__ __align__(16) unsigned char s_w3[];
    const bool staged = kMode == kWinDw && kStrip > 1 && window3_smem_bytes(a.Cs, (int)sizeof(T)) > 0;
    if (staged) {
        Raw* sw = reinterpret_cast<Raw*>(s_w3);
        const Raw* gw = static_cast<const Raw*>(a.w);
        for (int i = threadIdx.x; i < 9 * cv; i += blockDim.x) sw[i] = __ldg(gw + i);
        float* sb = reinterpret_cast<float*>(s_w3 + (size_t)9 * a.Cs * sizeof(T));
        for (int i = threadIdx.x; i < a.Cs; i += blockDim.x) sb[i] = (a.bias && i < a.K) ? a.bias[i] : 0.f;
        __syncthreads();
    }
    if (idx < total) {
        const int c0 = (idx % cv) * N;
        const int rest = idx / cv;
        const int q0 = (rest % strips) * kStrip, p = rest / strips;
        const T* __restrict__ x = x_img<T>(a) + c0;
        const T* __restrict__ w = (staged ? reinterpret_cast<const T*>(s_w3) : static_cast<const T*>(a.w)) + c0;
        f2_t acc[kStrip][NP];
        const f2_t init = (kMode == kWinMax) ? f2_pack(-INFINITY, -INFINITY) : f2_pack(0.f, 0.f);
#pragma unroll
        for (int t = 0; t < kStrip; ++t)
#pragma unroll
            for (int j = 0; j < NP; ++j) acc[t][j] = init;
        const int iw0 = q0 * kStride - a.pad_w;
        uint32_t col_ok = 0;                    // bit col: input column iw0 + col lies inside the tensor
        int off[kCols];                         // element offset of that column within a row (clamped)
#pragma unroll
        for (int col = 0; col < kCols; ++col) {
            const int iw = iw0 + col;
            if (iw >= 0 && iw < a.W) col_ok |= 1u << col;
            off[col] = min(max(iw, 0), a.W - 1) * a.Cs;
        }
        // every load of the 3 x kCols window first, so that all of them are in flight together
        Raw raw[3][kCols];
        uint32_t ok[3];
        int rows = 0;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int ih = p * kStride + r - a.pad_h;
            const bool row_ok = ih >= 0 && ih < a.H;
            rows += row_ok ? 1 : 0;
            ok[r] = row_ok ? col_ok : 0u;
            const T* xrow = x + (size_t)min(max(ih, 0), a.H - 1) * a.W * a.Cs;
#pragma unroll
            for (int col = 0; col < kCols; ++col) raw[r][col] = *reinterpret_cast<const Raw*>(xrow + off[col]);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            f2_t wv[3][NP];
            if (kMode == kWinDw) {
#pragma unroll
                for (int s = 0; s < 3; ++s) unpack_pairs(*reinterpret_cast<const Raw*>(w + (r * 3 + s) * a.Cs), wv[s]);
            }
            f2_t row_sum[kStrip][NP];         // average pooling: the columns of a row first
#pragma unroll
            for (int t = 0; t < kStrip; ++t)
#pragma unroll
                for (int j = 0; j < NP; ++j) row_sum[t][j] = f2_pack(0.f, 0.f);
#pragma unroll
            for (int col = 0; col < kCols; ++col) {
                if (!((ok[r] >> col) & 1u)) continue;
                f2_t xv[NP];
                unpack_pairs(raw[r][col], xv);
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    // input column col is tap s of output t when col == t * kStride + s
                    if (col - s < 0 || (col - s) % kStride != 0 || (col - s) / kStride >= kStrip) continue;
                    const int t = (col - s) / kStride;
#pragma unroll
                    for (int j = 0; j < NP; ++j) {
                        if (kMode == kWinDw) acc[t][j] = f2_fma(xv[j], wv[s][j], acc[t][j]);
                        else if (kMode == kWinMax) acc[t][j] = f2_max(acc[t][j], xv[j]);
                        else row_sum[t][j] = f2_add(row_sum[t][j], xv[j]);
                    }
                }
            }
            if (kMode == kWinAvg) {
#pragma unroll
                for (int t = 0; t < kStrip; ++t)
#pragma unroll
                    for (int j = 0; j < NP; ++j) acc[t][j] = f2_add(acc[t][j], row_sum[t][j]);
            }
        }
        T* yrow = y_img<T>(a) + ((size_t)p * a.Q + q0) * a.Ks + a.out_c_off + c0;
        float bias[N];
        if (kMode == kWinDw) {
#pragma unroll
            for (int j = 0; j < N; ++j)
                bias[j] = staged ? reinterpret_cast<const float*>(s_w3 + (size_t)9 * a.Cs * sizeof(T))[c0 + j]
                                 : ((a.bias && c0 + j < a.K) ? a.bias[c0 + j] : 0.f);
        }
#pragma unroll
        for (int t = 0; t < kStrip; ++t) {
            const int q = q0 + t;
            if (q >= a.Q) break;
            float v[N];
#pragma unroll
            for (int j = 0; j < NP; ++j) f2_unpack(acc[t][j], v[2 * j], v[2 * j + 1]);
            Vec<T> o;
            if (kMode == kWinDw) {
                // the activation is the same for every element: branch once, not per element
                if (a.act == 2) {
#pragma unroll
                    for (int j = 0; j < N; ++j) o.v[j] = (c0 + j < a.K) ? fminf(fmaxf(v[j] + bias[j], 0.f), 6.f) : 0.f;
                } else if (a.act == 1) {
#pragma unroll
                    for (int j = 0; j < N; ++j) o.v[j] = (c0 + j < a.K) ? fmaxf(v[j] + bias[j], 0.f) : 0.f;
                } else {
#pragma unroll
                    for (int j = 0; j < N; ++j) o.v[j] = (c0 + j < a.K) ? v[j] + bias[j] : 0.f;
                }
            } else if (kMode == kWinMax) {
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const float pv = (a.bias && c0 + j < a.C) ? v[j] + a.bias[c0 + j] : v[j];
                    o.v[j] = (c0 + j < a.C) ? act_fn(pv, a.act) : 0.f;
                }
            } else {
                float div = 9.f;
                if (!(a.flags & 1)) {
                    const int lo = max(q * kStride - a.pad_w, 0), hi = min(q * kStride - a.pad_w + 3, a.W);
                    const int cnt = rows * max(hi - lo, 0);
                    div = (float)(cnt > 0 ? cnt : 1);
                }
                // v / div, correctly rounded, in three instructions per element instead of the division
                // sequence (which was more than half of this kernel's instructions): with inv the correctly
                // rounded reciprocal, q = v * inv is within an ulp, the fused residual v - div * q is exact
                // and q + r * inv rounds to the quotient (Markstein); non-finite q passes through.  (-0.0
                // would come out as +0.0, but a sum that starts from +0.0 is never -0.0.)
                const float inv = 1.f / div;
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const float qv = v[j] * inv;
                    const float rv = fmaf(-div, qv, v[j]);
                    float out = fabsf(qv) <= 3.0e38f ? fmaf(rv, inv, qv) : qv;
                    if (a.bias && c0 + j < a.C) out += a.bias[c0 + j];
                    o.v[j] = (c0 + j < a.C) ? act_fn(out, a.act) : 0.f;
                }
            }
            o.store(yrow + (size_t)t * a.Ks);
        }
    }
    PB_NOTIFY_END();
}

// ---- 3x3 windows over tensors that fill the GPU, staged through shared memory ------------------------------------
// window3_strip_kernel loads every input row three times (once per output row it belongs to) and converts it to fp32 each
// time: about 300 instructions per output vector of 8 bf16 channels, which is what bounds it.  Here a block owns a tile of
// output rows x columns of ONE slab of 64 channels.  One TMA copy brings the tile's input window into shared memory
// (zero-filled outside the tensor; NaN for max, which the other operand of a maximum beats), then every half-warp walks down
// a strip of output columns, its 16 lanes holding four channels each: a row is read with one 8-byte load per input column, converted once, and feeds the
// (up to) three output rows it belongs to, whose accumulators stay in registers, as do the filter and the biases of the
// four channels.  Sums and products are packed pairs of fp32 (two IEEE operations per instruction).
//
// What bounds it is instruction issue, so the instructions per output are what the layout is chosen for: four channels a
// lane instead of two halve the loads, stores and address arithmetic, the packed arithmetic halves the rest, and a copy by
// 16-byte cp.async cost as much as a fifth of the walk in addresses and bounds checks.
// The activation and how an average counts its padding are template parameters: with all variants in one body the kernel
// ran out of the instruction cache.  Four or five warps (one per two units) and up to 74 KB of window: three blocks per SM
// fill and walk in turn.
//
// Max pooling compares the bf16 pairs themselves (a maximum needs no wider type); ReLU / ReLU6 clamp the rounded bf16 pair
// (rounding is monotonic and 0 and 6 are bf16 values).  Taps outside the tensor contribute the neutral element; an
// output's first tap opens its accumulator, so only the sign of a sum of zeros could show it.  The additions per output happen in the order of dwconv_kernel / pool_kernel (depthwise: filter
// rows, then columns; average: the columns of each row, then the rows, so that a row's three columns are added once for the three
// output rows they belong to: 4 additions instead of 9 a channel, 256 maps of 35 x 35 x 192 54.4 -> 49.2 us), so the results are theirs bit for bit (finite filter values
// assumed).  bf16 only.
constexpr int kTileStrip1 = 4, kTileStrip2 = 2;      // output columns per strip at stride 1 / 2
constexpr int kTileRows1 = 13, kTileRows2 = 6;       // output rows per tile (single images; batches: see win_tile())
constexpr int kTileSlab = 64;                        // channels per block
constexpr int kTileMaxThreads = 160;

// Tile geometry of a launch: strips x bands of output rows are the units the half-warps take.
struct WinTile {
    int col_tiles, strips, in_cols;      // column tiles per image, strips per tile, window columns
    int rows, bands, band_rows;          // output rows per tile, split into bands
    int in_rows, alloc_rows;             // window rows that are copied / that a walk may read
    int threads, smem;
};

__device__ __forceinline__ uint64_t p2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t p2_add(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t p2_mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t p2_of(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 p2_split(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t p2_bf16(uint32_t u) { return p2_of(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ uint32_t bits_of(__nv_bfloat162 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __nv_bfloat162 bf2_of(uint32_t u) { return *reinterpret_cast<const __nv_bfloat162*>(&u); }

// What a lane keeps per (output, channel pair): fp32 pairs for sums, the bf16 pair itself for a maximum.
template <int kMode> struct WinAcc { typedef uint64_t type; };
template <> struct WinAcc<kWinMax> { typedef uint32_t type; };
template <int kMode> __device__ __forceinline__ typename WinAcc<kMode>::type win_value(uint32_t raw) { return p2_bf16(raw); }
template <> __device__ __forceinline__ uint32_t win_value<kWinMax>(uint32_t raw) { return raw; }
__device__ __forceinline__ uint64_t win_open(uint64_t x, uint64_t w, bool dw) { return dw ? p2_mul(x, w) : x; }
__device__ __forceinline__ uint32_t win_open(uint32_t x, uint64_t, bool) { return x; }
__device__ __forceinline__ uint64_t win_step(uint64_t acc, uint64_t x, uint64_t w, bool dw) { return dw ? p2_fma(x, w, acc) : p2_add(acc, x); }
__device__ __forceinline__ uint32_t win_step(uint32_t acc, uint32_t x, uint64_t, bool) { return bits_of(__hmax2(bf2_of(acc), bf2_of(x))); }

// One finished output (two channels) -> bf16 pair.  kAct: 0 none, 1 ReLU, 2 ReLU6.  div / inv: the average pool's divisor
// and its reciprocal.  tail: a pooling layer with biases (a convolution that ran before the pooling).
template <int kMode, int kAct>
__device__ __forceinline__ uint32_t win_finish(uint64_t v, uint64_t bias, float div, float inv, bool tail) {
    if (kMode == kWinDw) {
        v = p2_add(v, bias);
    } else {
        // v / div, correctly rounded, without the division sequence: with inv the correctly rounded reciprocal, q = v * inv is
        // within an ulp, the fused residual v - div * q is exact and q + r * inv rounds to the quotient (Markstein).  An
        // infinite q makes the residual NaN; clamped to a finite value it leaves q as it is.
        const uint64_t inv2 = p2_of(inv, inv), q = p2_mul(v, inv2);
        const float2 r = p2_split(p2_fma(p2_of(-div, -div), q, v));
        v = p2_fma(p2_of(fmaxf(r.x, -3.402823466e38f), fmaxf(r.y, -3.402823466e38f)), inv2, q);
        if (tail) v = p2_add(v, bias);
    }
    const float2 f = p2_split(v);
    uint32_t h;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(f.y), "f"(f.x));
    if (kAct >= 1) h = bits_of(__hmax2(bf2_of(h), bf2_of(0u)));                   // zero for NaN, which cvt.rn.relu would keep
    if (kAct == 2) h = bits_of(__hmin2(bf2_of(h), bf2_of(0x40c040c0u)));          // (6, 6)
    return h;
}
template <int kMode, int kAct>
__device__ __forceinline__ uint32_t win_finish(uint32_t acc, uint64_t bias, float, float, bool tail) {
    acc = bits_of(__hmax2(bf2_of(acc), bf2_of(0xff80ff80u)));      // a window with nothing but NaN and padding: -infinity
    if (tail) {
        const float2 f = p2_split(p2_add(p2_bf16(acc), bias));
        acc = bits_of(__floats2bfloat162_rn(f.x, f.y));
    }
    __nv_bfloat162 h = bf2_of(acc);
    if (kAct >= 1) h = __hmax2(h, bf2_of(0u));
    if (kAct == 2) h = __hmin2(h, bf2_of(0x40c040c0u));
    return bits_of(h);
}

// Raised when the window's copy does not land.  In the module, not allocated: a program's first launch may be inside a stream
// capture, where nothing may be.
static __device__ uint32_t g_window_err_flag;

// What a lane knows of its four channels (from c0 on), and the steps of a walk down the window's rows.
// kWide: output and filter start on an 8-byte boundary, so a lane's four channels are one access; otherwise two of 4 bytes.
template <int kMode, int kStride, int kAct, bool kCountPad, bool kWide>
struct WinLane {
    typedef __nv_bfloat16 T;
    typedef typename WinAcc<kMode>::type Acc;
    static constexpr bool kDw = kMode == kWinDw;
    static constexpr int kStrip = kStride == 1 ? kTileStrip1 : kTileStrip2, kCols = (kStrip - 1) * kStride + 3;
    // A window row as the walk wants it: its columns (depthwise), or for pooling each output's three columns already reduced, once
    // for the three output rows the window row belongs to.
    static constexpr int kRow = kDw ? kCols : kStrip;
    uint64_t w[3][3][2], bias[2];
    uint32_t keep0, keep1;
    bool tail;

    __device__ __forceinline__ void channels(const OpArgs& a, int c0) {
        const int c_lim = kDw ? a.K : a.C;
        if (kDw) {
            const T* wp = static_cast<const T*>(a.w) + (c0 < a.Cs ? c0 : 0);
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int s2 = 0; s2 < 3; ++s2) {
                    const T* tap = wp + (r * 3 + s2) * a.Cs;
                    const uint2 u = kWide ? __ldg(reinterpret_cast<const uint2*>(tap))
                                          : make_uint2(__ldg(reinterpret_cast<const uint32_t*>(tap)), __ldg(reinterpret_cast<const uint32_t*>(tap) + 1));
                    w[r][s2][0] = p2_bf16(u.x);
                    w[r][s2][1] = p2_bf16(u.y);
                }
        }
        bias[0] = bias[1] = 0;
        tail = !kDw && a.bias != nullptr;
        if (a.bias) {
            float f[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) f[j] = c0 + j < c_lim ? a.bias[c0 + j] : 0.f;
            bias[0] = p2_of(f[0], f[1]);
            bias[1] = p2_of(f[2], f[3]);
        }
        // channels past the last one are stored as zeros
        keep0 = c0 + 1 < c_lim ? 0xffffffffu : (c0 < c_lim ? 0x0000ffffu : 0u);
        keep1 = c0 + 3 < c_lim ? 0xffffffffu : (c0 + 2 < c_lim ? 0x0000ffffu : 0u);
    }
    __device__ __forceinline__ void row_into(Acc (&acc)[kStrip][2], const Acc (&xv)[kRow][2], int r) const {
#pragma unroll
        for (int t = 0; t < kStrip; ++t) {
            if constexpr (!kDw) {
#pragma unroll
                for (int j = 0; j < 2; ++j) acc[t][j] = r == 0 ? xv[t][j] : win_step(acc[t][j], xv[t][j], 0, false);
            } else {
#pragma unroll
                for (int s2 = 0; s2 < 3; ++s2) {
                    if (r == 0 && s2 == 0) {
                        acc[t][0] = win_open(xv[t * kStride][0], w[0][0][0], true);
                        acc[t][1] = win_open(xv[t * kStride][1], w[0][0][1], true);
                        continue;
                    }
                    acc[t][0] = win_step(acc[t][0], xv[t * kStride + s2][0], w[r][s2][0], true);
                    acc[t][1] = win_step(acc[t][1], xv[t * kStride + s2][1], w[r][s2][1], true);
                }
            }
        }
    }
    __device__ __forceinline__ void load_row(const uint2* row, Acc (&xv)[kRow][2]) const {
        Acc col_v[kCols][2];
#pragma unroll
        for (int col = 0; col < kCols; ++col) {
            const uint2 v = row[col * (kTileSlab / 4)];
            col_v[col][0] = win_value<kMode>(v.x);
            col_v[col][1] = win_value<kMode>(v.y);
        }
#pragma unroll
        for (int t = 0; t < kRow; ++t)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if constexpr (kDw) xv[t][j] = col_v[t][j];
                else xv[t][j] = win_step(win_step(col_v[t * kStride][j], col_v[t * kStride + 1][j], 0, false), col_v[t * kStride + 2][j], 0, false);
            }
    }
    // The strip's outputs of row p (nt of them, from column q0 on), finished and stored at y.
    __device__ __forceinline__ void store_row(const OpArgs& a, const Acc (&acc)[kStrip][2], T* __restrict__ y, int p, int q0, int nt, bool all) const {
        const float inv9 = 1.f / 9.f;
        float div = 9.f, inv = inv9;
        int rows_in = 3;
        if (kMode == kWinAvg && !kCountPad) rows_in = min(p * kStride - a.pad_h + 3, a.H) - max(p * kStride - a.pad_h, 0);
#pragma unroll
        for (int t = 0; t < kStrip; ++t) {
            if (!all && t >= nt) break;
            if (kMode == kWinAvg && !kCountPad) {
                const int cols_in = max(min((q0 + t) * kStride - a.pad_w + 3, a.W) - max((q0 + t) * kStride - a.pad_w, 0), 0);
                const int cnt = rows_in * cols_in;
                if (cnt != 9) { div = (float)(cnt > 0 ? cnt : 1); inv = 1.f / div; }
                else { div = 9.f; inv = inv9; }
            }
            uint32_t o0 = win_finish<kMode, kAct>(acc[t][0], bias[0], div, inv, tail);
            uint32_t o1 = win_finish<kMode, kAct>(acc[t][1], bias[1], div, inv, tail);
            if (!all) { o0 &= keep0; o1 &= keep1; }
            if (kWide) {
                *reinterpret_cast<uint2*>(y + (uint32_t)(t * a.Ks)) = make_uint2(o0, o1);
            } else {
                uint32_t* const out = reinterpret_cast<uint32_t*>(y + (uint32_t)(t * a.Ks));
                out[0] = o0;
                out[1] = o1;
            }
        }
    }
    __device__ __forceinline__ bool whole(int nt) const { return nt == kStrip && (keep0 & keep1) == 0xffffffffu; }      // every output of the strip and all four channels exist
};

template <int kMode, int kStride, int kAct, bool kCountPad, bool kWide>
__global__ void __launch_bounds__(kTileMaxThreads, kMode == kWinAvg ? 4 : 3) window3_tile_kernel(OpArgs a, WinTile g, const __grid_constant__ CUtensorMap tmap, uint32_t job_id,
                                                                        FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    typedef WinLane<kMode, kStride, kAct, kCountPad, kWide> Lane;
    typedef typename Lane::T T;
    typedef typename Lane::Acc Acc;
    constexpr int kStrip = Lane::kStrip, kRow = Lane::kRow;
    extern __shared__ __align__(128) unsigned char s_tile[];
    __shared__ __align__(8) uint64_t s_full;

    const int slabs = (a.Cs + kTileSlab - 1) / kTileSlab;
    int b = blockIdx.x;
    const int slab = b % slabs; b /= slabs;
    const int q_tile = (b % g.col_tiles) * g.strips * kStrip;
    const int p_tile = (b / g.col_tiles) * g.rows;
    const int p_end = min(p_tile + g.rows, a.P);
    const int ih0 = p_tile * kStride - a.pad_h, iw0 = q_tile * kStride - a.pad_w;
    const int ch0 = slab * kTileSlab;

    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&s_full);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(g.in_rows * g.in_cols * kTileSlab * 2) : "memory");
        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(s_tile)), "l"(&tmap), "r"(ch0), "r"(iw0), "r"(ih0), "r"((int)blockIdx.y), "r"(bar)
                     : "memory");
    }

    const int half = threadIdx.x >> 4, c0 = ch0 + (threadIdx.x & 15) * 4;      // half-warp, first of the lane's four channels
    const bool ch_in = c0 < a.Cs;
    Lane lane;
    lane.channels(a, c0);
    const int pitch = g.in_cols * (kTileSlab / 4);                             // 8-byte words per window row
    __syncthreads();                                                           // the barrier exists
    bool landed = false;
    for (int i = 0; i < (1 << 22) && !landed; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar) : "memory");
        landed = ok != 0;
    }
    if (!landed) {          // the copy is given 50 us more to land before shared memory is released
        if (threadIdx.x == 0) atomicExch(&g_window_err_flag, 5u);
        unsigned long long t0, t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        for (int i = 0; i < (1 << 20); ++i) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t - t0 > 50000ull) break;
        }
    }

    // ---- walk ----
    const int units = landed ? g.strips * g.bands : 0;
    for (int u0 = 0; u0 + (half & ~1) < units; u0 += blockDim.x / 16) {      // both halves of a warp take the same turns
        const int unit = min(u0 + half, units - 1);
        const int band = unit / g.strips, strip = unit - band * g.strips;
        const int q0 = q_tile + strip * kStrip;
        const int p0 = p_tile + band * g.band_rows, p1 = min(p0 + g.band_rows, p_end);
        const int nt = u0 + half < units && ch_in ? min(kStrip, a.Q - q0) : 0;      // outputs this lane stores
        const bool full = lane.whole(nt);
        const uint2* row = reinterpret_cast<const uint2*>(s_tile) + (band * g.band_rows * kStride) * pitch + strip * kStrip * kStride * (kTileSlab / 4) + (threadIdx.x & 15);
        T* __restrict__ y = y_img<T>(a) + ((size_t)p0 * a.Q + q0) * a.Ks + a.out_c_off + c0;

        auto row_into = [&](Acc (&acc)[kStrip][2], const Acc (&xv)[kRow][2], int r) { lane.row_into(acc, xv, r); };
        auto load_row = [&](Acc (&xv)[kRow][2]) {
            lane.load_row(row, xv);
            row += pitch;
        };
        auto store_row = [&](const Acc (&acc)[kStrip][2], int p, bool all) {
            lane.store_row(a, acc, y, p, q0, nt, all);
            y += (size_t)a.Q * a.Ks;
        };
        // output rows are closed in order: p is the one after the last closed, rows before p0 and from p1 on are not stored
        auto close_row = [&](const Acc (&acc)[kStrip][2], int p) {
            if (p >= p0 && p < p1) {
                if (full) store_row(acc, p, true);
                else store_row(acc, p, false);
            }
        };

        if (kStride == 1) {
            // window row r opens output row p0 + r (filter row 0), continues p0 + r - 1, closes p0 + r - 2; three window rows per
            // turn (the last turn may run past the band, into rows that are not stored)
            Acc accA[kStrip][2], accB[kStrip][2], accC[kStrip][2];
#pragma unroll
            for (int t = 0; t < kStrip; ++t)
#pragma unroll
                for (int j = 0; j < 2; ++j) accB[t][j] = accC[t][j] = 0;          // (rows before p0: never stored)
#pragma unroll 1
            for (int p = p0; p < p1 + 2; p += 3) {
                Acc xv[kRow][2];
                load_row(xv); row_into(accB, xv, 2); row_into(accC, xv, 1); row_into(accA, xv, 0); close_row(accB, p - 2);
                load_row(xv); row_into(accC, xv, 2); row_into(accA, xv, 1); row_into(accB, xv, 0); close_row(accC, p - 1);
                load_row(xv); row_into(accA, xv, 2); row_into(accB, xv, 1); row_into(accC, xv, 0); close_row(accA, p);
            }
        } else {
            // window row 2i closes output row p0 + i - 1 (filter row 2) and opens p0 + i (row 0); row 2i + 1 is filter row 1 of p0 + i
            Acc acc[kStrip][2];
#pragma unroll
            for (int t = 0; t < kStrip; ++t) acc[t][0] = acc[t][1] = 0;
#pragma unroll 1
            for (int p = p0; p < p1; ++p) {
                Acc xv[kRow][2];
                load_row(xv); row_into(acc, xv, 2); close_row(acc, p - 1); row_into(acc, xv, 0);
                load_row(xv); row_into(acc, xv, 1);
            }
            Acc xv[kRow][2];
            load_row(xv);
            row_into(acc, xv, 2);
            close_row(acc, p1 - 1);
        }
    }
    PB_NOTIFY_END();
}

// The depthwise walk (stride 1) over tensors of many rows, with the window in a ring: a fixed number of blocks share all rows of all
// (image, column tile) units of their slab between them, each a contiguous range, and walk down it while one warp copies the next three window
// rows.  A tile of window3_tile_kernel reads two rows more than the thirteen it writes; here that is once per unit or range, and the blocks
// neither fill and walk in turn nor end in waves.  Bound by DRAM with reads and writes mixed: 128 x 1024 x 1024 104 -> 98.4 us (84 % of the copy
// rate); rings of three, four and five stages take 2, 9 and 13 % more - more rows under way are more places open at once; with the slabs of
// a pixel in different ranges 18 %.  Average pooling gains nothing here (256 maps of 35 x 35 x 192: tiles 49.2, rings 49.4 to 55 us).
constexpr int kRingStages = 2;
struct WinRing {
    int col_tiles, strips, in_cols, slabs;
    int rows;                       // output rows of a slab, all images and column tiles
    int blocks, threads;            // no blocks: the launch keeps its tiles
    int stage_bytes, smem;
};
// A block's next piece of work: rows [p0, p1) of one unit.
struct WinPiece {
    int img, col, p0, p1;
    __device__ __forceinline__ void at(const WinRing& g, int P, int row, int end) {
        const int unit = row / P;
        p0 = row - unit * P;
        p1 = min(P, p0 + end - row);
        img = unit / g.col_tiles;
        col = unit - img * g.col_tiles;
    }
};
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity, volatile uint32_t* s_abort) {
    for (int i = 0; i < (1 << 22); ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((i & 63) == 63 && *s_abort) return false;
    }
    *s_abort = 1;
    atomicExch(&g_window_err_flag, 6u);
    return false;
}

// (128 registers: at most four walking warps.)
template <int kAct, bool kWide>
__global__ void __launch_bounds__(160, 3) window3_ring_kernel(OpArgs a, const WinRing g, const __grid_constant__ CUtensorMap tmap, uint32_t job_id,
                                                                                FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    typedef WinLane<kWinDw, 1, kAct, true, kWide> Lane;
    typedef typename Lane::T T;
    typedef typename Lane::Acc Acc;
    constexpr int kStrip = Lane::kStrip, kRow = Lane::kRow;
    extern __shared__ __align__(128) unsigned char s_ring[];
    __shared__ __align__(8) uint64_t s_full[kRingStages], s_empty[kRingStages];
    __shared__ volatile uint32_t s_abort;

    const int warp = threadIdx.x >> 5, walkers = (blockDim.x >> 5) - 1;
    const uint32_t full = (uint32_t)__cvta_generic_to_shared(s_full), empty = (uint32_t)__cvta_generic_to_shared(s_empty);
    if (threadIdx.x == 0) {
        for (int i = 0; i < kRingStages; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + 8u * i));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + 8u * i), "r"(walkers));
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    // neighbouring blocks take the slabs of the same rows: together they read whole pixels
    const int range = (int)blockIdx.x / g.slabs, slab = (int)blockIdx.x - range * g.slabs, ranges = (int)gridDim.x / g.slabs;
    const int begin = (int)((long long)g.rows * range / ranges), end = (int)((long long)g.rows * (range + 1) / ranges);
    WinPiece piece;
    int st = 0;
    uint32_t parity = 0;

    if (warp == walkers) {
        // ===== copies: three window rows a stage =====
        if ((threadIdx.x & 31) == 0) {
            int turn = 0;
            bool ok = true;
            for (int row = begin; row < end && ok; row += piece.p1 - piece.p0) {
                piece.at(g, a.P, row, end);
                const int ch0 = slab * kTileSlab, iw0 = piece.col * g.strips * kStrip - a.pad_w;
                for (int p = piece.p0; p < piece.p1 + 2 && ok; p += 3) {
                    if (turn >= kRingStages) ok = ring_wait(empty + 8u * st, parity ^ 1u, &s_abort);
                    if (!ok) break;
                    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(full + 8u * st), "r"(g.stage_bytes) : "memory");
                    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
                                     (uint32_t)__cvta_generic_to_shared(s_ring) + (uint32_t)(st * g.stage_bytes)), "l"(&tmap), "r"(ch0), "r"(iw0), "r"(p - a.pad_h), "r"(piece.img),
                                 "r"(full + 8u * st)
                                 : "memory");
                    ++turn;
                    if (++st == kRingStages) { st = 0; parity ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else {
        // ===== walks =====
        const int half = threadIdx.x >> 4, strip = min(half, g.strips - 1);        // (a last half-warp without a strip repeats one and stores nothing)
        const int pitch = g.in_cols * (kTileSlab / 4);                             // 8-byte words per window row
        const uint2* const ring0 = reinterpret_cast<const uint2*>(s_ring) + strip * kStrip * (kTileSlab / 4) + (threadIdx.x & 15);
        const int c0 = slab * kTileSlab + (threadIdx.x & 15) * 4;
        Lane lane;
        lane.channels(a, c0);
        bool ok = true;
        for (int at = begin; at < end && ok; at += piece.p1 - piece.p0) {
            piece.at(g, a.P, at, end);
            const int q0 = (piece.col * g.strips + strip) * kStrip, p0 = piece.p0, p1 = piece.p1;
            const int nt = half < g.strips && c0 < a.Cs ? min(kStrip, a.Q - q0) : 0;      // outputs this lane stores
            const bool whole = lane.whole(nt);
            T* __restrict__ y = static_cast<T*>(a.y) + (((size_t)piece.img * a.P + p0) * a.Q + q0) * a.Ks + a.out_c_off + c0;
            auto close_row = [&](const Acc (&acc)[kStrip][2], int p) {
                if (p >= p0 && p < p1) {
                    if (whole) lane.store_row(a, acc, y, p, q0, nt, true);
                    else lane.store_row(a, acc, y, p, q0, nt, false);
                    y += (size_t)a.Q * a.Ks;
                }
            };
            // window row r opens output row p0 + r (filter row 0), continues p0 + r - 1, closes p0 + r - 2; three window rows per turn
            Acc accA[kStrip][2], accB[kStrip][2], accC[kStrip][2];
#pragma unroll
            for (int t = 0; t < kStrip; ++t)
#pragma unroll
                for (int j = 0; j < 2; ++j) accB[t][j] = accC[t][j] = 0;          // (rows before p0: never stored)
#pragma unroll 1
            for (int p = p0; p < p1 + 2; p += 3) {
                ok = __all_sync(0xffffffffu, ring_wait(full + 8u * st, parity, &s_abort));
                if (!ok) break;
                const uint2* row = ring0 + (size_t)st * (g.stage_bytes / 8);
                Acc xv[kRow][2];
                lane.load_row(row, xv); lane.row_into(accB, xv, 2); lane.row_into(accC, xv, 1); lane.row_into(accA, xv, 0); close_row(accB, p - 2);
                lane.load_row(row + pitch, xv); lane.row_into(accC, xv, 2); lane.row_into(accA, xv, 1); lane.row_into(accB, xv, 0); close_row(accC, p - 1);
                lane.load_row(row + 2 * pitch, xv); lane.row_into(accA, xv, 2); lane.row_into(accB, xv, 1); lane.row_into(accC, xv, 0);
                __syncwarp();
                if ((threadIdx.x & 31) == 0) asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.shared::cta.b64 s, [%0];\n\t}" ::"r"(empty + 8u * st) : "memory");
                close_row(accA, p);
                if (++st == kRingStages) { st = 0; parity ^= 1u; }
            }
        }
    }
    __syncthreads();
    if (s_abort) {          // copies are given 50 us more to land before shared memory is released
        unsigned long long t0, t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        for (int i = 0; i < (1 << 20); ++i) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t - t0 > 50000ull) break;
        }
        __syncthreads();
    }
    PB_NOTIFY_END();
}

// ---- global average pool: [HW][Cs] -> [Cs] ---------------------------------------
// Block = 32 channel vectors x 8 pixel groups; shared-memory reduction over the groups.
template <typename T>
__global__ void __launch_bounds__(256) gap_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    __shared__ float red[8][32][N + 1];
    const int cv = a.Cs / N;
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int v = blockIdx.x * 32 + lane;
    const int HW = a.H * a.W;
    float acc[N];
#pragma unroll
    for (int j = 0; j < N; ++j) acc[j] = 0.f;
    if (v < cv) {
        const T* __restrict__ x = x_img<T>(a);
        for (int pix = grp; pix < HW; pix += 8) {
            const Vec<T> xv = Vec<T>::load(x + (size_t)pix * a.Cs + v * N);
#pragma unroll
            for (int j = 0; j < N; ++j) acc[j] += xv.v[j];
        }
    }
#pragma unroll
    for (int j = 0; j < N; ++j) red[grp][lane][j] = acc[j];
    __syncthreads();
    if (grp == 0 && v < cv) {
        const float inv = 1.f / (float)HW;
        float o[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float s = 0.f;
#pragma unroll
            for (int gI = 0; gI < 8; ++gI) s += red[gI][lane][j];
            o[j] = s * inv;
        }
        if (a.flags & 2) {
            float* y = out_f32_img(a, slot_, a.C);
#pragma unroll
            for (int j = 0; j < N; ++j) if (v * N + j < a.C) y[v * N + j] = o[j];
        } else {
            Vec<T> ov;
#pragma unroll
            for (int j = 0; j < N; ++j) ov.v[j] = (v * N + j < a.C) ? o[j] : 0.f;
            ov.store(y_img<T>(a) + v * N);
        }
    }
    PB_NOTIFY_END();
}

// ---- dense: y[k] = act(w[k,:] . x + b[k]); one warp per output row -----------------
// x has n_in = a.C elements (already in the device's flattened channels-last order, padded
// entries zero); w is [K][C] with C a multiple of the vector width.
//
// A row of weights is streamed once, from HBM, and that is what bounds it.  U raw 128-bit loads per lane are issued before
// the first is used (cache-streaming, so they do not evict the input vector from L1); the sum keeps the order of the plain
// loop.  U = 8 with four blocks per SM: fewer rows in flight than eight blocks with U = 4, each in longer runs of DRAM.
// 16384 -> 8192 in bf16 (268 MB) / 4096 -> 4096 / 25088 -> 512, us: U = 4, eight blocks 49.5 / 10.2 / 28.5; U = 8, eight blocks
// 46.3; U = 8, four blocks 41.5 (6.5 TB/s) / 9.0 / 18.5; U = 12 42.9 / 9.8 / 18.4; U = 16 (spills) 41.2 / 9.9 / 16.4; U = 16,
// three blocks 45.4 / 10.5 / 14.6.  What is left of a row takes U = 4 (a classifier of 1024 inputs is one such step), then one.
template <int U, typename T>
__device__ __forceinline__ void dense_run(const T* __restrict__ x, const T* __restrict__ w, int C, int& i, float& acc) {
    constexpr int N = Vec<T>::N, kStep = 32 * N;
    typedef typename RawVec<T>::type Raw;
    for (; i + (U - 1) * kStep < C; i += U * kStep) {
        Raw wr[U];
#pragma unroll
        for (int u = 0; u < U; ++u) wr[u] = __ldcs(reinterpret_cast<const Raw*>(w + i + u * kStep));
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const Vec<T> xv = Vec<T>::load(x + i + u * kStep);
            const Vec<T> wv = vec_of(wr[u]);
#pragma unroll
            for (int j = 0; j < N; ++j) acc = fmaf(xv.v[j], wv.v[j], acc);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256, 4) dense_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp < a.K) {
        const T* __restrict__ x = x_img<T>(a);
        const T* __restrict__ w = static_cast<const T*>(a.w) + (size_t)warp * a.C;
        float acc = 0.f;
        int i = lane * N;
        dense_run<8>(x, w, a.C, i, acc);
        dense_run<4>(x, w, a.C, i, acc);
        dense_run<1>(x, w, a.C, i, acc);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            const float v = act_fn(acc + (a.bias ? a.bias[warp] : 0.f), a.act);
            if (a.flags & 2) out_f32_img(a, slot_, a.K)[warp] = v;
            else y_img<T>(a)[warp] = from_f<T>(v);
        }
    }
    PB_NOTIFY_END();
}

// ---- elementwise add (+activation) over [HW][Cs] ----------------------------------
template <typename T>
__global__ void __launch_bounds__(256) add_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    const size_t nv = (size_t)a.H * a.W * a.Cs / N;      // the host folds the images into H
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nv) {
        const Vec<T> u = Vec<T>::load(static_cast<const T*>(a.x) + i * N);
        const Vec<T> v = Vec<T>::load(static_cast<const T*>(a.residual) + i * N);
        Vec<T> o;
#pragma unroll
        for (int j = 0; j < N; ++j) o.v[j] = act_fn(u.v[j] + v.v[j], a.act);
        o.store(static_cast<T*>(a.y) + i * N);
    }
    PB_NOTIFY_END();
}

// ---- 2 x 2 pooling, stride 2, no border --------------------------------------------------------------------------
// A block owns 512 consecutive channel vectors of one output row, a thread two of them: eight 128-bit loads in flight, one
// division per vector, bf16 maxima taken two at a time as bf16 (a maximum rounds nothing).  pool_kernel, a vector and
// four loads in turn per thread, is bound by its 64-bit addresses and conversions: maxima of 16 x 256 x 256 x 128 in bf16 84.4 us, 50.8
// here (all of the copy bandwidth).
__device__ __forceinline__ float4 pool2_max(const float4 (&v)[4]) {
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        o[j] = -INFINITY;
#pragma unroll
        for (int i = 0; i < 4; ++i) o[j] = fmaxf(o[j], (&v[i].x)[j]);
    }
    return make_float4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ uint4 pool2_max(const uint4 (&v)[4]) {
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        o[j] = 0xff80ff80u;                  // -inf: a window of NaNs gives it, as fmaxf would
#pragma unroll
        for (int i = 0; i < 4; ++i) asm("max.bf16x2 %0, %0, %1;" : "+r"(o[j]) : "r"((&v[i].x)[j]));
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
constexpr int kPool2Vecs = 512;
__host__ __device__ __forceinline__ int pool2_chunks(int Q, int cv) { return (Q * cv + kPool2Vecs - 1) / kPool2Vecs; }

template <typename T, bool kMax>
__global__ void __launch_bounds__(256) pool2_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    typedef typename RawVec<T>::type Raw;
    const int cv = a.Cs / N, row = a.Q * cv, chunks = pool2_chunks(a.Q, cv);
    const int p = (int)blockIdx.x / chunks, i0 = ((int)blockIdx.x - p * chunks) * kPool2Vecs + (int)threadIdx.x;
    const T* __restrict__ x = x_img<T>(a) + (size_t)(2 * p) * a.W * a.Cs;
    const size_t below = (size_t)a.W * a.Cs;
    Raw raw[2][4];
    int q[2], c0[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = i0 + 256 * u < row ? i0 + 256 * u : 0;
        q[u] = i / cv;
        c0[u] = (i - q[u] * cv) * N;
        const T* at = x + (size_t)(2 * q[u]) * a.Cs + c0[u];
        raw[u][0] = *reinterpret_cast<const Raw*>(at);
        raw[u][1] = *reinterpret_cast<const Raw*>(at + a.Cs);
        raw[u][2] = *reinterpret_cast<const Raw*>(at + below);
        raw[u][3] = *reinterpret_cast<const Raw*>(at + below + a.Cs);
    }
    T* __restrict__ y = y_img<T>(a) + (size_t)p * a.Q * a.Ks + a.out_c_off;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        if (i0 + 256 * u >= row) break;
        T* at = y + (size_t)q[u] * a.Ks + c0[u];
        Vec<T> o;
        if constexpr (kMax) {
            const Raw m = pool2_max(raw[u]);
            if (!a.bias && a.act == 0 && c0[u] + N <= a.C) {
                *reinterpret_cast<Raw*>(at) = m;
                continue;
            }
            o = vec_of(m);
        } else {
#pragma unroll
            for (int j = 0; j < N; ++j) o.v[j] = 0.f;
#pragma unroll
            for (int r = 0; r < 2; ++r) {        // the columns of a row first, as in pool_kernel
                const Vec<T> v0 = vec_of(raw[u][2 * r]), v1 = vec_of(raw[u][2 * r + 1]);
#pragma unroll
                for (int j = 0; j < N; ++j) o.v[j] += v0.v[j] + v1.v[j];
            }
#pragma unroll
            for (int j = 0; j < N; ++j) o.v[j] *= 0.25f;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float v = o.v[j] + (a.bias && c0[u] + j < a.C ? a.bias[c0[u] + j] : 0.f);
            o.v[j] = c0[u] + j < a.C ? act_fn(v, a.act) : 0.f;
        }
        o.store(at);
    }
    PB_NOTIFY_END();
}

// ---- per-channel affine (+activation) over [HW][C] of a tensor with channel stride Cs ----------
// y[pix][c] = act(x[pix][c] * scale[c] + bias[c]) for the first a.C channels: the folded batch-norm +
// ReLU that DenseNet applies to the concatenated features BEFORE each convolution.
constexpr int kAffinePer = 4;      // vectors per thread
// Threads of a launch over `pixels` pixels of `cv` vectors: a quarter of the pixels, rounded up.
__host__ __device__ __forceinline__ size_t affine_threads(size_t pixels, int cv) { return (pixels + kAffinePer - 1) / kAffinePer * cv; }

template <typename T>
__global__ void __launch_bounds__(256) affine_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START_EARLY(T);
    constexpr int N = Vec<T>::N;
    typedef typename RawVec<T>::type Raw;
    const int cv = (a.C + N - 1) / N;
    // A thread takes the same kAffinePer channels' vector of kAffinePer pixels, a quarter of the tensor apart: all loads are issued
    // (as raw 128-bit words) before any is used - with one load in flight per thread the kernel ran at 54 % of the copy
    // bandwidth on a tensor larger than L2, which needs about 50 KB in flight per SM - and scale and bias are loaded once.
    // (Loaded for every vector they were two thirds of the bytes through L1, whose data pipe was 76 % busy: 16 x 256 x 256 x 128 in
    // bf16 108.4 us, 86.3 now: 95 % of the copy bandwidth.)
    const size_t pixels = (size_t)a.H * a.W, part = affine_threads(pixels, cv), step = part / cv;
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 < part) {
        // 32-bit division whenever the index fits (always, short of a 256 GB tensor)
        const size_t pix0 = part <= 0xffffffffull ? (size_t)((uint32_t)i0 / (uint32_t)cv) : i0 / cv;
        const int c0 = (int)(i0 - pix0 * cv) * N;
        const T* __restrict__ x = static_cast<const T*>(a.x) + c0;
        Raw raw[kAffinePer];
#pragma unroll
        for (int h = 0; h < kAffinePer; ++h) {
            const size_t pix = pix0 + h * step;
            raw[h] = *reinterpret_cast<const Raw*>(x + (pix < pixels ? pix : pix0) * a.Cs);
        }
        const float* __restrict__ sc = static_cast<const float*>(a.w) + c0;
        const float* __restrict__ bi = a.bias + c0;
        float scv[N], biv[N];
        if (c0 + N <= a.C && ((reinterpret_cast<uintptr_t>(sc) | reinterpret_cast<uintptr_t>(bi)) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < N; j += 4) {
                *reinterpret_cast<float4*>(scv + j) = __ldg(reinterpret_cast<const float4*>(sc + j));
                *reinterpret_cast<float4*>(biv + j) = __ldg(reinterpret_cast<const float4*>(bi + j));
            }
        } else {
#pragma unroll
            for (int j = 0; j < N; ++j) {
                scv[j] = c0 + j < a.C ? __ldg(sc + j) : 0.f;
                biv[j] = c0 + j < a.C ? __ldg(bi + j) : 0.f;
            }
        }
#pragma unroll
        for (int h = 0; h < kAffinePer; ++h) {
            const size_t pix = pix0 + h * step;
            if (pix >= pixels) break;
            const Vec<T> u = vec_of(raw[h]);
            Vec<T> o;
#pragma unroll
            for (int j = 0; j < N; ++j) o.v[j] = c0 + j < a.C ? act_fn(u.v[j] * scv[j] + biv[j], a.act) : 0.f;
            o.store(static_cast<T*>(a.y) + pix * a.Ks + a.out_c_off + c0);
        }
    }
    PB_NOTIFY_END();
}

// ---- softmax over a.C values, one block --------------------------------------------
template <typename T, bool kInF32>
__global__ void __launch_bounds__(256) softmax_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    __shared__ float red[8];
    __shared__ float bc;
    const int n = a.C;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // flags bit2: a bare fp32 vector per image; otherwise image i is tensor i of [H][W][Cs]
    const float* xf = static_cast<const float*>(a.x) + (size_t)blockIdx.y * ((a.flags & 4) ? (size_t)n : (size_t)a.H * a.W * a.Cs);
    const T* xt = x_img<T>(a);
    auto ld = [&](int i) { return kInF32 ? xf[i] : to_f<T>(xt[i]); };
    float m = -INFINITY;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, ld(i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[wid] = m;
    __syncthreads();
    if (threadIdx.x == 0) { float t = red[0]; for (int i = 1; i < 8; ++i) t = fmaxf(t, red[i]); bc = t; }
    __syncthreads();
    m = bc;
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += __expf(ld(i) - m);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncthreads();
    if (lane == 0) red[wid] = s;
    __syncthreads();
    if (threadIdx.x == 0) { float t = 0.f; for (int i = 0; i < 8; ++i) t += red[i]; bc = t; }
    __syncthreads();
    const float inv = 1.f / bc;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float v = __expf(ld(i) - m) * inv;
        if (a.flags & 2) out_f32_img(a, slot_, n)[i] = v;
        else y_img<T>(a)[i] = from_f<T>(v);
    }
    PB_NOTIFY_END();
}

// ---- detection head over one feature map ----------------------------------------------
// One thread per prior (cell, anchor) of the map.  x is [H][W][Cs] with C = 6A channels: 2A class logits
// (anchor, class), then 4A box regressions (anchor, coordinate).  a.w = fp32 priors [H*W*A][4] = (cx, cy, w, h),
// a.bias = {centre variance, size variance}, a.K = priors of the whole model, a.out_c_off = this map's first
// prior.  The fp32 model output is [K*2 scores | K*4 corner-form boxes].
template <typename T>
__global__ void __launch_bounds__(256) detect_kernel(OpArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    PB_NOTIFY_START();
    const int A = a.C / 6;
    const int n = a.H * a.W * A;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const int cell = i / A, an = i - cell * A;
        const T* __restrict__ x = x_img<T>(a) + (size_t)cell * a.Cs;
        const float c0 = to_f<T>(x[an * 2]), c1 = to_f<T>(x[an * 2 + 1]);
        const float m = fmaxf(c0, c1);
        const float e0 = expf(c0 - m), e1 = expf(c1 - m);
        const float inv = 1.f / (e0 + e1);
        float* out = out_f32_img(a, slot_, a.K * 6);
        float* sc = out + (size_t)(a.out_c_off + i) * 2;       // scalar stores: a request's buffer need not be 16-byte aligned
        sc[0] = e0 * inv; sc[1] = e1 * inv;
        const float4 pr = __ldg(reinterpret_cast<const float4*>(a.w) + i);
        const float cv = __ldg(a.bias), sv = __ldg(a.bias + 1);
        const T* l = x + 2 * A + an * 4;
        const float cx = to_f<T>(l[0]) * cv * pr.z + pr.x, cy = to_f<T>(l[1]) * cv * pr.w + pr.y;
        const float bw = expf(to_f<T>(l[2]) * sv) * pr.z, bh = expf(to_f<T>(l[3]) * sv) * pr.w;
        float* bo = out + (size_t)a.K * 2 + (size_t)(a.out_c_off + i) * 4;
        bo[0] = cx - bw * 0.5f; bo[1] = cy - bh * 0.5f; bo[2] = cx + bw * 0.5f; bo[3] = cy + bh * 0.5f;
    }
    PB_NOTIFY_END();
}

// ---- whole MNIST-CNN in one launch ---------------------------------------------------
// conv5x5(1->8)+ReLU, maxpool2, conv5x5(8->16)+ReLU, maxpool3, dense 256->10 for 28x28 images, fp32, activations in shared
// memory.  The network is 1.2 MFLOP (the outer two rows and columns of the second convolution are never pooled) and 24 KB of
// weights, so one kernel (one start and one end record) replaces six.
// A lone request is the serial chain of its blocks, so what counts is multiply-adds per word read from shared memory and how many SMs
// share them.  A lone image has a cluster of four blocks, and rank r row r of the pooled 4x4 result: its rows of the second convolution need
// seven rows of the pooled first one (five at the borders), which it works out itself - twice the multiply-adds of a quarter of that
// layer, but nothing is exchanged before the ten partial sums of the classifier, which meet in rank 0's shared memory.  In the second
// convolution a warp has one input channel and a thread its 25 weights of two output channels, in registers since before the
// request's pointers have been read (they and the image come from the host's memory); warp 0 reports the start while the others
// fetch the image.  (All of it in one block of 256 threads: about 9 us of arithmetic, a lone request 19.2 us; this: 16.1.)
// Weights: w1 [5][5][1][8], w2 [5][5][8][16], wd [10][4*4*16] (h, w, c order), biases fp32.
struct MnistArgs {
    const float* x;     // [28][28]
    const float* w1; const float* b1;
    const float* w2; const float* b2;
    const float* wd; const float* bd;
    float* y;           // [10]
};

constexpr int kMnistRanks = 4;
__global__ void __launch_bounds__(256, 1) mnist_fused_kernel(MnistArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    constexpr int kInRows = 18, kInPitch = 34, kP1Rows = 7, kP1Pitch = 20, kP1Plane = kP1Rows * kP1Pitch, kPartPitch = 16;
    __shared__ __align__(16) float s_in[kInRows * kInPitch];  // image rows 6 r - 6 on, with a 2-pixel zero border
    __shared__ __align__(16) float s_w1[25 * 8];
    __shared__ __align__(16) float s_p1[8 * kP1Plane];        // pool1 rows 3 r - 2 on, 8 planes with a 2-pixel zero border
    __shared__ __align__(16) float s_part[8 * 36 * kPartPitch];      // [input channel][pooled pixel][position][16]
    __shared__ float s_max[3 * 64];
    __shared__ float s_p2[64];
    __shared__ float s_sum[kMnistRanks][12];                  // rank 0: the ranks' shares of the classifier's sums
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, rank = (int)blockIdx.x;
    const int kp = t & 7, px = (t >> 3) & 3;                  // second convolution: channel pair, pooled pixel
    // every block of the cluster is running before its shared memory is written to
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    // the weights do not depend on the request
    float2 w2r[25];
#pragma unroll
    for (int j = 0; j < 25; ++j) w2r[j] = __ldg(reinterpret_cast<const float2*>(a.w2 + j * 128 + wid * 16 + kp * 2));
    float wdr[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j) wdr[h][j] = wid + 8 * h < 10 ? __ldg(a.wd + (wid + 8 * h) * 256 + rank * 64 + lane + 32 * j) : 0.f;
    const float b2r = __ldg(a.b2 + (t & 15)), bdr = t < 10 ? __ldg(a.bd + t) : 0.f;
    if (t < 200) s_w1[t] = __ldg(a.w1 + t);
    for (int i = t; i < kInRows * kInPitch; i += 256) s_in[i] = 0.f;
    for (int i = t; i < 8 * kP1Plane; i += 256) s_p1[i] = 0.f;
    pb::griddep_wait();
    const pb::LaunchSlot* slot = pb::resolve_slot(job_id, nf);
    const float* const x = (!a.x && slot) ? slot->io_in[0] : a.x;
    float* const y = (!a.y && slot) ? slot->io_out[0] : a.y;
    __syncthreads();                                          // the zeros are down
    if (wid == 0) {
        // the cluster is declared, and reports, as one block of 1024 threads
        if (nf && rank == 0 && t == 0) nf->channel_.write(llis::job::InstrumentInfo::kStart, 0, 1, job_id, false);
    } else {
        const int top = 6 * rank - 6, lo = max(top, 0), n = min(top + kInRows, 28) - lo;
        if ((reinterpret_cast<uintptr_t>(x) & 7) == 0) {
            for (int i = t - 32; i < n * 14; i += 224) {
                const float2 v = reinterpret_cast<const float2*>(x)[lo * 14 + i];
                float* d = s_in + (lo - top + i / 14) * kInPitch + (i % 14) * 2 + 2;
                d[0] = v.x;
                d[1] = v.y;
            }
        } else {
            for (int i = t - 32; i < n * 28; i += 224) s_in[(lo - top + i / 28) * kInPitch + i % 28 + 2] = x[lo * 28 + i];
        }
    }
    __syncthreads();
    // conv1 + ReLU + 2x2 max pool: thread = (pooled pixel, four channels)
    {
        const int half = t >= 98 ? 1 : 0, pix = t - 98 * half, row = pix / 14, col = pix - row * 14;
        if (t < 196 && 3 * rank - 2 + row >= 0) {             // (the last rank's rows end with the map)
            float p[6][6];
#pragma unroll
            for (int r = 0; r < 6; ++r)
#pragma unroll
                for (int c = 0; c < 6; c += 2) {
                    const float2 v = *reinterpret_cast<const float2*>(s_in + (2 * row + r) * kInPitch + 2 * col + c);
                    p[r][c] = v.x;
                    p[r][c + 1] = v.y;
                }
            float acc[4][4];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[0][k] = acc[1][k] = acc[2][k] = acc[3][k] = __ldg(a.b1 + half * 4 + k);
#pragma unroll
            for (int r = 0; r < 5; ++r)
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    const float4 w = *reinterpret_cast<const float4*>(s_w1 + (r * 5 + c) * 8 + half * 4);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float v = p[r + (q >> 1)][c + (q & 1)];
                        acc[q][0] = fmaf(v, w.x, acc[q][0]);
                        acc[q][1] = fmaf(v, w.y, acc[q][1]);
                        acc[q][2] = fmaf(v, w.z, acc[q][2]);
                        acc[q][3] = fmaf(v, w.w, acc[q][3]);
                    }
                }
            float* d = s_p1 + half * 4 * kP1Plane + row * kP1Pitch + col + 2;
#pragma unroll
            for (int k = 0; k < 4; ++k)      // ReLU and pooling in one: the largest of the four and zero
                d[k * kP1Plane] = fmaxf(fmaxf(fmaxf(acc[0][k], acc[1][k]), fmaxf(acc[2][k], acc[3][k])), 0.f);
        }
    }
    __syncthreads();
    // conv2: thread = (input channel, pooled pixel, pair of output channels), the nine positions of the pooling window
    {
        const float* ip = s_p1 + wid * kP1Plane + px * 3;
        float acc[9][2];
#pragma unroll
        for (int o = 0; o < 9; ++o) acc[o][0] = acc[o][1] = 0.f;
#pragma unroll
        for (int r = 0; r < 7; ++r) {
            float v[7];
#pragma unroll
            for (int j = 0; j < 7; ++j) v[j] = ip[r * kP1Pitch + j];
#pragma unroll
            for (int oy = 0; oy < 3; ++oy) {
                if (r - oy < 0 || r - oy > 4) continue;
#pragma unroll
                for (int ox = 0; ox < 3; ++ox)
#pragma unroll
                    for (int j = 0; j < 5; ++j) {
                        acc[oy * 3 + ox][0] = fmaf(v[ox + j], w2r[(r - oy) * 5 + j].x, acc[oy * 3 + ox][0]);
                        acc[oy * 3 + ox][1] = fmaf(v[ox + j], w2r[(r - oy) * 5 + j].y, acc[oy * 3 + ox][1]);
                    }
            }
        }
        float* d = s_part + (wid * 36 + px * 9) * kPartPitch + kp * 2;
#pragma unroll
        for (int o = 0; o < 9; ++o) *reinterpret_cast<float2*>(d + o * kPartPitch) = make_float2(acc[o][0], acc[o][1]);
    }
    __syncthreads();
    // the channels' sums in channel order, + bias, ReLU, 3x3 max pool: thread = (row of the window, pooled pixel, channel), then its rows
    if (t < 192) {
        const int oy = t >> 6, f = t & 63;
        const float* s = s_part + ((f >> 4) * 9 + oy * 3) * kPartPitch + (f & 15);
        float best = 0.f;
#pragma unroll
        for (int ox = 0; ox < 3; ++ox) {
            float sum[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                sum[h] = s[(h * 144 + ox) * kPartPitch];
#pragma unroll
                for (int c = 1; c < 4; ++c) sum[h] += s[(h * 144 + c * 36 + ox) * kPartPitch];
            }
            best = fmaxf(best, sum[0] + sum[1] + b2r);
        }
        s_max[t] = best;
    }
    __syncthreads();
    if (t < 64) s_p2[t] = fmaxf(fmaxf(s_max[t], s_max[t + 64]), s_max[t + 128]);
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    // dense 256 -> 10, this rank's 64 values: warps 0..7 take rows w, w+8
    const uint32_t sum0 = (uint32_t)__cvta_generic_to_shared(&s_sum[0][0]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int o = wid + 8 * h;
        if (o < 10) {
            float acc = s_p2[lane] * wdr[h][0];
            acc = fmaf(s_p2[lane + 32], wdr[h][1], acc);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
            if (lane == 0)
                asm volatile("{\n\t.reg .b32 at;\n\tmapa.shared::cluster.u32 at, %0, 0;\n\tst.shared::cluster.f32 [at], %1;\n\t}" ::"r"(sum0 + (uint32_t)(rank * 12 + o) * 4u), "f"(acc)
                             : "memory");
        }
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    if (rank != 0) return;                                    // nobody reads or writes this block's memory any more
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    if (wid == 0) {
        if (t < 10) y[t] = ((s_sum[0][t] + s_sum[1][t]) + (s_sum[2][t] + s_sum[3][t])) + bdr;
        __syncwarp();
        if (nf && t == 0) {
            __threadfence();
            nf->channel_.write(llis::job::InstrumentInfo::kEnd, 0, 1, job_id, true);
        }
    }
}

// The images of a gang, one block each, the same sums in the same order.  On a GPU full of other requests' blocks four free places on one
// GPC are longer in coming than one (192 requests of MNIST : Inception-v3 = 9 : 1 with clusters for gangs, too, 1197 us; with these blocks
// 1175), and the images of a gang are side by side anyway.
__global__ void __launch_bounds__(256, 2) mnist_gang_kernel(MnistArgs a, uint32_t job_id, FinishedBlockNotifier* nf) {
    constexpr int kInPitch = 34, kP1Pitch = 20, kP1Plane = 18 * kP1Pitch;
    __shared__ __align__(16) float s_in[32 * kInPitch];       // 28x28 image with a 2-pixel zero border
    __shared__ __align__(16) float s_w1[25 * 8];
    __shared__ __align__(16) float s_p1[8 * kP1Plane];        // pool1 output, 8 planes of 14x14 with a 2-pixel zero border
    __shared__ __align__(16) float s_w2[8 * 25 * 16];         // [channel][tap][16]
    __shared__ __align__(16) float s_part[128 * 19];          // half of the second convolution's sums
    __shared__ float s_p2[256];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    // the weights do not depend on the previous kernel or the request
    float w2r[13], wdr[2][8];
#pragma unroll
    for (int i = 0; i < 13; ++i) w2r[i] = t + 256 * i < 3200 ? __ldg(a.w2 + t + 256 * i) : 0.f;
    const float w1r = t < 200 ? __ldg(a.w1 + t) : 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 8; ++j) wdr[h][j] = wid + 8 * h < 10 ? __ldg(a.wd + (wid + 8 * h) * 256 + lane + 32 * j) : 0.f;
    for (int i = t; i < 32 * kInPitch; i += 256) s_in[i] = 0.f;
    for (int i = t; i < 8 * kP1Plane; i += 256) s_p1[i] = 0.f;
    pb::griddep_wait();
    const pb::LaunchSlot* slot = pb::resolve_slot(job_id, nf);
    // one block per image of the gang
    const float* x = (!a.x && slot) ? slot->io_in[blockIdx.x] : a.x + (size_t)blockIdx.x * 784;
    float* y = (!a.y && slot) ? slot->io_out[blockIdx.x] : a.y + (size_t)blockIdx.x * 10;
    __syncthreads();                                          // the zeros are down
    if (wid == 0) {
        if (nf) nf->start(job_id);
    } else if ((reinterpret_cast<uintptr_t>(x) & 7) == 0) {
        for (int i = t - 32; i < 392; i += 224) {
            const float2 v = reinterpret_cast<const float2*>(x)[i];
            float* d = s_in + (i / 14 + 2) * kInPitch + (i % 14) * 2 + 2;
            d[0] = v.x;
            d[1] = v.y;
        }
    } else {
        for (int i = t - 32; i < 784; i += 224) s_in[(i / 28 + 2) * kInPitch + i % 28 + 2] = x[i];
    }
#pragma unroll
    for (int i = 0; i < 13; ++i) {
        const int e = t + 256 * i;
        if (e < 3200) s_w2[((e >> 4 & 7) * 25 + (e >> 7)) * 16 + (e & 15)] = w2r[i];
    }
    if (t < 200) s_w1[t] = w1r;
    __syncthreads();
    // conv1 + ReLU + 2x2 max pool: one thread per pooled pixel, four channels at a time
    if (t < 196) {
        const int py = t / 14, px = t - py * 14;
        float p[6][6];
#pragma unroll
        for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int c = 0; c < 6; c += 2) {
                const float2 v = *reinterpret_cast<const float2*>(s_in + (2 * py + r) * kInPitch + 2 * px + c);
                p[r][c] = v.x;
                p[r][c + 1] = v.y;
            }
        float* d = s_p1 + (py + 2) * kP1Pitch + px + 2;
#pragma unroll 1
        for (int kb = 0; kb < 8; kb += 4) {
            float acc[4][4];
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[0][k] = acc[1][k] = acc[2][k] = acc[3][k] = __ldg(a.b1 + kb + k);
#pragma unroll
            for (int r = 0; r < 5; ++r)
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    const float4 w = *reinterpret_cast<const float4*>(s_w1 + (r * 5 + c) * 8 + kb);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float v = p[r + (q >> 1)][c + (q & 1)];
                        acc[q][0] = fmaf(v, w.x, acc[q][0]);
                        acc[q][1] = fmaf(v, w.y, acc[q][1]);
                        acc[q][2] = fmaf(v, w.z, acc[q][2]);
                        acc[q][3] = fmaf(v, w.w, acc[q][3]);
                    }
                }
#pragma unroll
            for (int k = 0; k < 4; ++k)      // ReLU and pooling in one: the largest of the four and zero
                d[(kb + k) * kP1Plane] = fmaxf(fmaxf(fmaxf(acc[0][k], acc[1][k]), fmaxf(acc[2][k], acc[3][k])), 0.f);
        }
    }
    __syncthreads();
    // conv2 + ReLU + 3x3 max pool (floor: 14 -> 4): thread = (pooled pixel, pair of channels, half of the input channels)
    {
        const int kp = t & 7, pix = (t >> 3) & 15, ch = (t >> 7) * 4;
        const float* ip0 = s_p1 + ch * kP1Plane + (pix >> 2) * 3 * kP1Pitch + (pix & 3) * 3;
        const float* wp0 = s_w2 + ch * 25 * 16 + kp * 2;
        float sum[9][2];                          // the channels' sums, each complete, are added in order, as the cluster does
#pragma unroll
        for (int o = 0; o < 9; ++o) sum[o][0] = sum[o][1] = 0.f;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            float acc[9][2];
#pragma unroll
            for (int o = 0; o < 9; ++o) acc[o][0] = acc[o][1] = 0.f;
            float2 w[25];
#pragma unroll
            for (int j = 0; j < 25; ++j) w[j] = *reinterpret_cast<const float2*>(wp0 + c * 25 * 16 + j * 16);
#pragma unroll
            for (int r = 0; r < 7; ++r) {
                float v[7];
#pragma unroll
                for (int j = 0; j < 7; ++j) v[j] = ip0[c * kP1Plane + r * kP1Pitch + j];
#pragma unroll
                for (int oy = 0; oy < 3; ++oy) {
                    if (r - oy < 0 || r - oy > 4) continue;
#pragma unroll
                    for (int ox = 0; ox < 3; ++ox)
#pragma unroll
                        for (int j = 0; j < 5; ++j) {
                            acc[oy * 3 + ox][0] = fmaf(v[ox + j], w[(r - oy) * 5 + j].x, acc[oy * 3 + ox][0]);
                            acc[oy * 3 + ox][1] = fmaf(v[ox + j], w[(r - oy) * 5 + j].y, acc[oy * 3 + ox][1]);
                        }
                }
            }
#pragma unroll
            for (int o = 0; o < 9; ++o) {
                sum[o][0] += acc[o][0];
                sum[o][1] += acc[o][1];
            }
        }
        if (t >= 128) {
#pragma unroll
            for (int o = 0; o < 9; ++o) {
                s_part[(t - 128) * 19 + o * 2] = sum[o][0];
                s_part[(t - 128) * 19 + o * 2 + 1] = sum[o][1];
            }
        }
        __syncthreads();
        if (t < 128) {
            float best0 = 0.f, best1 = 0.f;      // ReLU: at least zero
            const float b0 = __ldg(a.b2 + kp * 2), b1 = __ldg(a.b2 + kp * 2 + 1);
#pragma unroll
            for (int o = 0; o < 9; ++o) {
                best0 = fmaxf(best0, sum[o][0] + s_part[t * 19 + o * 2] + b0);
                best1 = fmaxf(best1, sum[o][1] + s_part[t * 19 + o * 2 + 1] + b1);
            }
            s_p2[pix * 16 + kp * 2] = best0;
            s_p2[pix * 16 + kp * 2 + 1] = best1;
        }
    }
    __syncthreads();
    // dense 256 -> 10: warps 0..7 take rows w, w+8
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int o = wid + 8 * h;
        if (o < 10) {
            float acc[kMnistRanks];              // a rank's 64 values at a time
#pragma unroll
            for (int r = 0; r < kMnistRanks; ++r) acc[r] = fmaf(s_p2[lane + 64 * r + 32], wdr[h][2 * r + 1], s_p2[lane + 64 * r] * wdr[h][2 * r]);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int r = 0; r < kMnistRanks; ++r) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], off);
            if (lane == 0) y[o] = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + __ldg(a.bd + o);
        }
    }
    PB_NOTIFY_END();
}

// ---------------------------------------------------------------------------------
// Host: geometry, resources, weight layouts, dispatch
// ---------------------------------------------------------------------------------
static OpArgs to_args(const pb_op_params* p) {
    OpArgs a;
    a.C = p->C; a.H = p->H; a.W = p->W; a.Cs = p->Cs; a.K = p->K; a.P = p->P; a.Q = p->Q; a.Ks = p->Ks;
    a.out_c_off = p->out_c_off; a.R = p->R; a.S = p->S; a.stride_h = p->stride_h; a.stride_w = p->stride_w;
    a.pad_h = p->pad_h; a.pad_w = p->pad_w; a.groups = p->groups > 0 ? p->groups : 1; a.act = p->act; a.flags = p->flags;
    a.res_Cs = p->res_Cs; a.dil_h = p->dil_h > 1 ? p->dil_h : 1; a.dil_w = p->dil_w > 1 ? p->dil_w : 1; a.x = p->x; a.w = p->w; a.bias = p->bias; a.residual = p->residual; a.y = p->y;
    return a;
}

static int vec_n(int dtype) { return dtype == 0 ? 4 : 8; }
static int batch_of(const pb_op_params* p) { return p->batch > 1 ? p->batch : 1; }
static size_t elem_size(int dtype) { return dtype == 0 ? 4 : 2; }

template <typename F>
static uint32_t regs_of(F fn) {
    cudaFuncAttributes at;
    if (cudaFuncGetAttributes(&at, (const void*)fn) != cudaSuccess) { cudaGetLastError(); return 32; }
    return (uint32_t)at.numRegs;
}
template <typename F>
static uint32_t static_smem_of(F fn) {
    cudaFuncAttributes at;
    if (cudaFuncGetAttributes(&at, (const void*)fn) != cudaSuccess) { cudaGetLastError(); return 0; }
    return (uint32_t)at.sharedSizeBytes;
}

// Does a pooling layer run pool2_kernel?  Rows of less than 192 vectors leave most of a block idle: they keep pool_kernel.
static bool pool2(const pb_op_params* p) {
    const int N = p->dtype == 0 ? 4 : 8;
    return p->R == 2 && p->S == 2 && p->stride_h == 2 && p->stride_w == 2 && p->pad_h == 0 && p->pad_w == 0 && 2 * p->P <= p->H && 2 * p->Q <= p->W &&
           p->Cs % N == 0 && (int64_t)p->Q * (p->Cs / N) >= 192 && (int64_t)p->Q * p->Cs < (1 << 30);
}
// Threads of work -> blocks of 256.
static uint32_t blocks_for(size_t work) { return (uint32_t)((work + 255) / 256 > 0 ? (work + 255) / 256 : 1); }

// Output pixels per thread of window3_strip_kernel for a depthwise convolution or pooling layer: 0 when the
// window is not 3x3 with stride 1 or 2 (the layer keeps dwconv_kernel / pool_kernel); the wide strip when the
// strips (4 pixels at stride 1, 2 at stride 2) alone give each SM 2048 threads; else 1 (all batch-1 layers of the
// served models: there the launch is latency-bound and more, smaller threads finish sooner).
static int strip_of(const pb_op_params* p) {
    if (p->R != 3 || p->S != 3 || p->stride_h != p->stride_w || (p->stride_h != 1 && p->stride_h != 2)) return 0;
    static thread_local int sms = 0;      // of the device current at the first call of this thread (replicas: one GPU per thread)
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
            cudaGetLastError();
            sms = 148;
        }
    }
    const int wide = p->stride_h == 1 ? kStripWide1 : kStripWide2;
    const size_t n = (size_t)batch_of(p) * p->P * ((p->Q + wide - 1) / wide) * (p->Cs / vec_n(p->dtype));
    // Below that size the one-pixel variant still pays: its nine loads are in flight together.  (Tried for the sake of
    // a busy GPU: the plain kernels, 40 registers instead of 100-126, so that their blocks fit beside resident
    // tensor-core CTAs.  Serving throughput FELL, 26.9k -> 24.8k Inception-v3 req/s with 96 in flight: under load these
    // launches cost what they take in time, not in registers.)
    return n >= (size_t)sms * 2048 ? wide : 1;
}
static size_t strip_threads(const pb_op_params* p, int strip) {
    return (size_t)p->P * ((p->Q + strip - 1) / strip) * (p->Cs / vec_n(p->dtype));
}

// Tile of window3_tile_kernel.  A single image is cut into tiles of 8 strips x 13 (stride 2: 6) rows, 65 KB of window.  The
// images of a batch are mostly small maps, where that tile hangs over the edges (35 columns: a tile of 32 and one of 3, 101 us
// for 256 images of 35 x 35 x 192 instead of 51), so their tiles are fitted to the map: as few column tiles as hold at most 40 columns
// each, as many rows as keep the window (the rows a walk runs past the tile included) within 74 KB, so that three blocks fit an SM,
// and bands of rows where a map has fewer strips than half-warps.
// A pooling lane holds no filter, so four of its blocks fit an SM's registers (maxima without asking: asked for, 26 of 71 x 71 x 192 take 17.4 us instead of
// 17.2), and a batch's windows are cut for four (average, 256 maps of 35 x 35 x 192 49.2 -> 48.3 us, the smaller windows alone 53.1; 256 of
// 17 x 17 x 256 25.0 -> 20.7; maximum 20.7 -> 17.5, stride 2 on 64 of 35 x 35 x 288 14.3 -> 12.6) - not where whole
// waves of them read a quarter more (97 of 56 x 30 x 192 at stride 2, two waves of the larger or three 8.3 and 9.0; 78 of them, two and two, 7.4 and 7.0).  Depthwise blocks, whose registers allow three, lose with them (256 of 35 x 35 x 192 55.7 -> 59.8).
constexpr int kTileWindowBytes = 74 * 1024, kTileWindowBytesPool = 54 * 1024;
static WinTile win_tile_within(const pb_op_params* p, int limit) {
    const int st = p->stride_h, strip = st == 1 ? kTileStrip1 : kTileStrip2;
    WinTile g;
    if (batch_of(p) == 1) {
        g.strips = 8;
        g.col_tiles = ceil_div(p->Q, g.strips * strip);
        g.rows = st == 1 ? kTileRows1 : kTileRows2;
    } else {
        const int n = ceil_div(p->Q, st == 1 ? 40 : 20);
        g.strips = ceil_div(ceil_div(p->Q, n), strip);
        g.col_tiles = ceil_div(p->Q, g.strips * strip);
    }
    g.in_cols = (g.strips * strip - 1) * st + 3;
    if (batch_of(p) > 1) {
        int fit = (limit / (g.in_cols * kTileSlab * 2) - 3) / st + 1;      // rows of output whose window fits
        if (fit < 1) fit = 1;
        g.rows = p->P < fit ? p->P : fit;
        if (st == 1 && fit < p->P && fit > 3) g.rows = (fit - 1) / 3 * 3 + 1;     // a walk takes three window rows per turn: no turn half used
    }
    for (;;) {
        g.bands = g.strips >= 8 ? 1 : (8 / g.strips < g.rows ? 8 / g.strips : g.rows);
        g.band_rows = ceil_div(g.rows, g.bands);
        g.bands = ceil_div(g.rows, g.band_rows);
        const int walked = st == 1 ? ceil_div(g.band_rows + 2, 3) * 3 : 2 * g.band_rows + 1;      // window rows a unit reads
        g.alloc_rows = (g.bands - 1) * g.band_rows * st + walked;
        g.in_rows = (g.rows - 1) * st + 3;
        g.alloc_rows = g.alloc_rows > g.in_rows ? g.alloc_rows : g.in_rows;
        g.smem = g.alloc_rows * g.in_cols * kTileSlab * 2;
        if (g.smem <= limit || g.rows == 1) break;
        g.rows = ceil_div(p->P, ceil_div(p->P, g.rows) + 1) < g.rows ? ceil_div(p->P, ceil_div(p->P, g.rows) + 1) : g.rows - 1;      // one more row tile
    }
    g.threads = 32 * ceil_div(g.strips * g.bands < 10 ? g.strips * g.bands : 10, 2);
    return g;
}
static size_t win_blocks(const pb_op_params* p, const WinTile& g) { return (size_t)ceil_div(p->Cs, kTileSlab) * g.col_tiles * ceil_div(p->P, g.rows); }
static WinTile win_tile(int kind, const pb_op_params* p) {
    const WinTile g = win_tile_within(p, kTileWindowBytes);
    const bool fills = win_blocks(p, g) * batch_of(p) >= 3 * 148;      // else more blocks are only more halo: 8 of 147 x 147 x 64 4.4 -> 4.8
    if (kind == PB_STAGE_DWCONV || batch_of(p) == 1 || !fills) return g;
    const WinTile small = win_tile_within(p, kTileWindowBytesPool);
    // whole waves of blocks, each as long as its windows
    auto waves = [&](const WinTile& t, int per_sm) { return (double)ceil_div((int)std::min<size_t>(win_blocks(p, t) * batch_of(p), 1u << 30), 148 * per_sm) * per_sm * t.alloc_rows * t.in_cols; };
    return waves(small, 4) > 1.25 * waves(g, 3) ? g : small;
}

// Blocks of window3_tile_kernel for one image, or 0 when the layer keeps the strip kernels: bf16, a 3x3 window of stride 1
// or 2, and at least 100 blocks in the launch (all images).  Measured on Inception-v3 served in gangs of 8: thresholds of
// 30, 100 and 300 blocks give the same +2 % requests/s over 592 (its two stem max pools then run here); below 100 a lone
// request's pooling layers are a few dozen blocks and keep the strip kernels, which finish sooner on an idle GPU.
// PB_WINDOW_TILE=0 switches it off (=1: see win_ring); PB_WINDOW_TILE_MIN_BLOCKS sets another threshold (tests use 1).  Read at every call:
// this runs when a launch is built (graph capture, direct operator calls), never on the replay path.
static uint32_t tile_blocks(int kind, const pb_op_params* p) {
    if (p->dtype != 1 || (p->Cs & 7) || (p->Ks & 3) || (p->out_c_off & 3) || p->act > 2 || strip_of(p) == 0) return 0;
    const char* e = getenv("PB_WINDOW_TILE");
    if (e && e[0] == '0') return 0;
    size_t least = 100;
    if (const char* m = getenv("PB_WINDOW_TILE_MIN_BLOCKS")) least = (size_t)strtoull(m, nullptr, 10);
    const WinTile g = win_tile(kind, p);
    const size_t n = win_blocks(p, g);
    return n * (size_t)batch_of(p) >= least ? (uint32_t)n : 0;
}
uint32_t* window_error_flag_ptr() {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_window_err_flag) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return static_cast<uint32_t*>(p);
}

// Window map of a launch: boxes of one slab x in_cols x in_rows of the images.
static int win_map(int kind, const pb_op_params* p, const WinTile& g, CUtensorMap* out) {
    const uint64_t dims[4] = {(uint64_t)p->Cs, (uint64_t)p->W, (uint64_t)p->H, (uint64_t)batch_of(p)};
    const uint64_t strides[3] = {(uint64_t)p->Cs * 2, (uint64_t)p->W * p->Cs * 2, (uint64_t)p->H * p->W * p->Cs * 2};
    const uint32_t box[4] = {(uint32_t)kTileSlab, (uint32_t)g.in_cols, (uint32_t)g.in_rows, 1};
    return encode_tiled_bf16(p->x, 4, dims, strides, box, kind == PB_STAGE_MAXPOOL, out);
}
template <int kMode, bool kCountPad, bool kWide>
static const void* tile_fn(int stride, int act) {
#define PB_TILE(S) (act == 2 ? (const void*)window3_tile_kernel<kMode, S, 2, kCountPad, kWide> \
                             : act == 1 ? (const void*)window3_tile_kernel<kMode, S, 1, kCountPad, kWide> : (const void*)window3_tile_kernel<kMode, S, 0, kCountPad, kWide>)
    return stride == 1 ? PB_TILE(1) : PB_TILE(2);
#undef PB_TILE
}
template <bool kWide>
static const void* tile_fn(int kind, const pb_op_params* p) {
    if (kind == PB_STAGE_DWCONV) return tile_fn<kWinDw, true, kWide>(p->stride_h, p->act);
    if (kind == PB_STAGE_MAXPOOL) return tile_fn<kWinMax, true, kWide>(p->stride_h, p->act);
    return (p->flags & 1) ? tile_fn<kWinAvg, true, kWide>(p->stride_h, p->act) : tile_fn<kWinAvg, false, kWide>(p->stride_h, p->act);
}
// The tile needs pairs of channels on 4-byte boundaries only.  (As a run-time test in one kernel the narrow accesses cost 2 % of an
// average pooling: 256 maps of 35 x 35 x 192 53.8 -> 54.9 us.)
static const void* tile_fn(int kind, const pb_op_params* p) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p->y) | (kind == PB_STAGE_DWCONV ? reinterpret_cast<uintptr_t>(p->w) : 0);
    return (at & 7) == 0 ? tile_fn<true>(kind, p) : tile_fn<false>(kind, p);
}

// Ring of a launch's window: depthwise windows of stride 1 whose column tiles have seven or eight strips (four walking warps; with five
// strips, 256 maps of 64 x 40 x 16, 37 us become 47) and whose rows give every block 24 and more (a block's range starts with two rows of
// no output; fewer blocks than the GPU holds lose more than the ring gains), and where its walks are a tenth shorter than the tiles': one walk down a map of
// P rows takes P + 2, in threes, a tile's two more than its own; a map that one tile holds gains nothing and pays for ranges that end inside of it
// (tiles / ring: 100 MB of 14 x 28 x 64 maps 45.1 / 46.9 us, 10 x 32 36.7 / 40.7, 5 x 112 56.6 / 63.8, 20 x 112 42.1 / 45.9; 19 x 28 49.7 / 42.5, 28 x 28 43.7 / 41.7).
// PB_WINDOW_TILE=1: wherever it can run (for tests).  Tiles / ring: 64 maps of 112 x 112 x 128 86.0 / 82.0 us, 32 of
// 224 x 224 x 64 83.6 / 71.9, 4 of 300 x 500 x 96 63.4 / 55.5, 64 of 57 x 57 x 200 50.6 / 45.7, 2 of 200 x 200 x 640 45.3 / 44.8.
static WinRing win_ring(int kind, const pb_op_params* p) {
    WinRing g = {};
    if (kind != PB_STAGE_DWCONV || p->stride_h != 1 || p->stride_w != 1 || tile_blocks(kind, p) == 0) return g;
    g.strips = ceil_div(ceil_div(p->Q, ceil_div(p->Q, 32)), kTileStrip1);
    g.col_tiles = ceil_div(p->Q, g.strips * kTileStrip1);
    g.slabs = ceil_div(p->Cs, kTileSlab);
    g.in_cols = g.strips * kTileStrip1 + 2;
    g.stage_bytes = 3 * g.in_cols * kTileSlab * 2;
    g.smem = kRingStages * g.stage_bytes;
    g.threads = 32 * (ceil_div(g.strips, 2) + 1);
    const int ranges = 3 * 148 / g.slabs;
    const long long rows = (long long)batch_of(p) * g.col_tiles * p->P;      // of a slab
    if (g.strips < 7 || ranges < 1 || rows < 24ll * ranges || rows > 0x3fffffff) return g;
    const char* e = getenv("PB_WINDOW_TILE");
    if (!e || e[0] != '1') {
        const WinTile t = win_tile(kind, p);
        const long long tile_walks = (long long)ceil_div(p->P, t.rows) * t.col_tiles * t.strips * t.bands * ceil_div(t.band_rows + 2, 3);
        const long long ring_walks = (long long)g.col_tiles * g.strips * ceil_div(p->P + 2, 3);
        if (t.rows >= p->P || 10 * tile_walks < 11 * ring_walks) return g;
    }
    g.rows = (int)rows;
    g.blocks = ranges * g.slabs;
    return g;
}
static int ring_map(const pb_op_params* p, const WinRing& g, CUtensorMap* out) {
    const uint64_t dims[4] = {(uint64_t)p->Cs, (uint64_t)p->W, (uint64_t)p->H, (uint64_t)batch_of(p)};
    const uint64_t strides[3] = {(uint64_t)p->Cs * 2, (uint64_t)p->W * p->Cs * 2, (uint64_t)p->H * p->W * p->Cs * 2};
    const uint32_t box[4] = {(uint32_t)kTileSlab, (uint32_t)g.in_cols, 3, 1};
    return encode_tiled_bf16(p->x, 4, dims, strides, box, false, out);
}
static const void* ring_fn(const pb_op_params* p) {
#define PB_RING(W) (p->act == 2 ? (const void*)window3_ring_kernel<2, W> : p->act == 1 ? (const void*)window3_ring_kernel<1, W> : (const void*)window3_ring_kernel<0, W>)
    return ((reinterpret_cast<uintptr_t>(p->y) | reinterpret_cast<uintptr_t>(p->w)) & 7) == 0 ? PB_RING(true) : PB_RING(false);
#undef PB_RING
}

template <int kMode>
static const void* window3_fn(bool f32, int stride, int strip) {
#define PB_W3(T) (stride == 1 ? (strip == 1 ? (const void*)window3_strip_kernel<T, kMode, 1, 1> : (const void*)window3_strip_kernel<T, kMode, 1, kStripWide1>) \
                              : (strip == 1 ? (const void*)window3_strip_kernel<T, kMode, 2, 1> : (const void*)window3_strip_kernel<T, kMode, 2, kStripWide2>))
    return f32 ? PB_W3(float) : PB_W3(__nv_bfloat16);
#undef PB_W3
}
static const void* window3_fn(int kind, bool f32, int stride, int strip) {
    return kind == PB_STAGE_DWCONV ? window3_fn<kWinDw>(f32, stride, strip)
         : kind == PB_STAGE_MAXPOOL ? window3_fn<kWinMax>(f32, stride, strip) : window3_fn<kWinAvg>(f32, stride, strip);
}

// Geometry of ONE image of the launch (blocks, algorithmic work); strip_of() alone looks at the batch.
static int info_one_image(int kind, const pb_op_params* p, pb_launch_info* out) {
    memset(out, 0, sizeof(*out));
    out->kind = (uint32_t)kind;
    out->threads_per_block = 256;
    const int N = vec_n(p->dtype);
    const size_t es = elem_size(p->dtype);
    const bool f32 = p->dtype == 0;
    const size_t in_elems = (size_t)p->C * p->H * p->W;
    const size_t out_elems = (size_t)p->K * p->P * p->Q;
    switch (kind) {
        case PB_STAGE_INPUT:
            if (p->R * p->S > 1) {      // patch-matrix form (see input_patch_kernel)
                out->num_blocks = blocks_for((size_t)p->P * p->Q * (p->Ks / N));
                out->regs_per_thread = f32 ? regs_of(input_patch_kernel<float>) : regs_of(input_patch_kernel<__nv_bfloat16>);
                if (const size_t sm = patch_tile_smem(p)) {
                    out->num_blocks = patch_tile_blocks(p);
                    out->regs_per_thread = f32 ? regs_of(input_patch_tile_kernel<float>) : regs_of(input_patch_tile_kernel<__nv_bfloat16>);
                    out->smem_per_block = (uint32_t)sm;
                }
                out->bytes = in_elems * 4 + (size_t)p->P * p->Q * p->Ks * es;
                break;
            }
            out->num_blocks = blocks_for((size_t)p->H * p->W);
            out->regs_per_thread = f32 ? regs_of(input_transform_kernel<float>) : regs_of(input_transform_kernel<__nv_bfloat16>);
            // the output is counted as laid out, Ks channels per pixel: the zero padding up to the vector width is part
            // of the format the convolutions read
            out->bytes = in_elems * 4 + (size_t)p->H * p->W * p->Ks * es;
            break;
        case PB_STAGE_CONV_SIMT:
            out->num_blocks = blocks_for((size_t)p->P * p->Q * p->K);
            out->regs_per_thread = f32 ? regs_of(conv_simt_kernel<float>) : regs_of(conv_simt_kernel<__nv_bfloat16>);
            out->flops = 2ull * out_elems * (p->C / (p->groups > 0 ? p->groups : 1)) * p->R * p->S;
            out->bytes = es * (in_elems + (size_t)p->K * (p->C / (p->groups > 0 ? p->groups : 1)) * p->R * p->S + out_elems +
                               (p->residual ? out_elems : 0)) + 4ull * p->K;
            break;
        case PB_STAGE_DWCONV:
            out->num_blocks = blocks_for((size_t)p->P * p->Q * (p->Cs / N));
            out->regs_per_thread = f32 ? regs_of(dwconv_kernel<float>) : regs_of(dwconv_kernel<__nv_bfloat16>);
            if (const int strip = strip_of(p)) {
                out->num_blocks = blocks_for(strip_threads(p, strip));
                out->regs_per_thread = regs_of(window3_fn(kind, f32, p->stride_h, strip));
                out->smem_per_block = strip > 1 ? (uint32_t)window3_smem_bytes(p->Cs, f32 ? 4 : 2) : 0;
            }
            if (const uint32_t nblk = tile_blocks(kind, p)) {
                out->num_blocks = nblk;
                out->regs_per_thread = regs_of(tile_fn(kind, p));
                out->smem_per_block = (uint32_t)win_tile(kind, p).smem;
                out->threads_per_block = (uint32_t)win_tile(kind, p).threads;
            }
            out->flops = 2ull * out_elems * p->R * p->S;
            out->bytes = es * (in_elems + (size_t)p->K * p->R * p->S + out_elems) + 4ull * p->K;
            break;
        case PB_STAGE_MAXPOOL:
        case PB_STAGE_AVGPOOL:
            out->num_blocks = blocks_for((size_t)p->P * p->Q * (p->Cs / N));
            if (kind == PB_STAGE_MAXPOOL)
                out->regs_per_thread = f32 ? regs_of(pool_kernel<float, true>) : regs_of(pool_kernel<__nv_bfloat16, true>);
            else
                out->regs_per_thread = f32 ? regs_of(pool_kernel<float, false>) : regs_of(pool_kernel<__nv_bfloat16, false>);
            if (pool2(p)) {
                out->num_blocks = (uint32_t)(p->P * pool2_chunks(p->Q, p->Cs / N));
                if (kind == PB_STAGE_MAXPOOL) out->regs_per_thread = f32 ? regs_of(pool2_kernel<float, true>) : regs_of(pool2_kernel<__nv_bfloat16, true>);
                else out->regs_per_thread = f32 ? regs_of(pool2_kernel<float, false>) : regs_of(pool2_kernel<__nv_bfloat16, false>);
            }
            if (const int strip = strip_of(p)) {
                out->num_blocks = blocks_for(strip_threads(p, strip));
                out->regs_per_thread = regs_of(window3_fn(kind, f32, p->stride_h, strip));
            }
            if (const uint32_t nblk = tile_blocks(kind, p)) {
                out->num_blocks = nblk;
                out->regs_per_thread = regs_of(tile_fn(kind, p));
                out->smem_per_block = (uint32_t)win_tile(kind, p).smem;
                out->threads_per_block = (uint32_t)win_tile(kind, p).threads;
            }
            out->bytes = es * (in_elems + out_elems) + (p->bias ? 4ull * p->K : 0);
            break;
        case PB_STAGE_GAP:
            out->num_blocks = (uint32_t)pb::ceil_div(p->Cs / N, 32);
            out->regs_per_thread = f32 ? regs_of(gap_kernel<float>) : regs_of(gap_kernel<__nv_bfloat16>);
            out->smem_per_block = f32 ? static_smem_of(gap_kernel<float>) : static_smem_of(gap_kernel<__nv_bfloat16>);
            out->bytes = es * in_elems + ((p->flags & 2) ? 4 : es) * (size_t)p->C;
            break;
        case PB_STAGE_DENSE:
            out->num_blocks = (uint32_t)pb::ceil_div(p->K, 8);
            out->regs_per_thread = f32 ? regs_of(dense_kernel<float>) : regs_of(dense_kernel<__nv_bfloat16>);
            out->flops = 2ull * p->C * p->K;
            out->bytes = es * ((size_t)p->C + (size_t)p->C * p->K) + 4ull * p->K + ((p->flags & 2) ? 4 : es) * (size_t)p->K;
            break;
        case PB_STAGE_ADD:
            out->num_blocks = blocks_for((size_t)p->H * p->W * p->Cs / N);
            out->regs_per_thread = f32 ? regs_of(add_kernel<float>) : regs_of(add_kernel<__nv_bfloat16>);
            out->bytes = es * 3 * in_elems;
            break;
        case PB_STAGE_AFFINE:
            out->num_blocks = blocks_for(affine_threads((size_t)p->H * p->W, pb::ceil_div(p->C, N)));
            out->regs_per_thread = f32 ? regs_of(affine_kernel<float>) : regs_of(affine_kernel<__nv_bfloat16>);
            out->flops = 2ull * p->C * p->H * p->W;
            out->bytes = es * 2ull * p->C * p->H * p->W + 8ull * p->C;
            break;
        case PB_STAGE_SOFTMAX:
            out->num_blocks = 1;
            out->regs_per_thread = regs_of(softmax_kernel<float, true>);
            out->smem_per_block = static_smem_of(softmax_kernel<float, true>);
            out->bytes = 8ull * p->C;
            break;
        case PB_STAGE_DETECT:
            out->num_blocks = blocks_for((size_t)p->H * p->W * (p->C / 6));
            out->regs_per_thread = f32 ? regs_of(detect_kernel<float>) : regs_of(detect_kernel<__nv_bfloat16>);
            out->flops = 20ull * p->H * p->W * (p->C / 6);
            out->bytes = es * (uint64_t)p->H * p->W * p->C + (16ull + 24ull) * p->H * p->W * (p->C / 6);
            break;
        default:
            set_error("pb_op_info: unknown stage kind %d", kind);
            return PB_ERR_INVALID;
    }
    return PB_OK;
}

// Elementwise kernels see a batch as one taller tensor (images are contiguous).
static bool folds_batch(int kind) { return kind == PB_STAGE_ADD || kind == PB_STAGE_AFFINE; }

int simple_op_info(int kind, const pb_op_params* p, pb_launch_info* out) {
    if (kind == PB_STAGE_CONV_SIMT && conv_f32_supported(p)) return conv_f32_info(p, out);
    const int nb = batch_of(p);
    const int rc = info_one_image(kind, p, out);
    if (rc != PB_OK) return rc;
    const WinRing ring = win_ring(kind, p);
    if (ring.blocks) {          // the blocks share all images
        out->num_blocks = (uint32_t)ring.blocks;
        out->regs_per_thread = regs_of(ring_fn(p));
        out->smem_per_block = (uint32_t)ring.smem;
        out->threads_per_block = (uint32_t)ring.threads;
    }
    if (nb == 1) return rc;
    if (folds_batch(kind)) {
        pb_op_params q = *p;
        q.H *= nb;
        return info_one_image(kind, &q, out);
    }
    out->num_blocks *= (uint32_t)nb;
    if (ring.blocks) out->num_blocks = (uint32_t)ring.blocks;
    out->flops *= (uint64_t)nb;
    // the weights are read once per launch whatever the batch
    const uint64_t es = p->dtype == 0 ? 4 : 2;
    const uint64_t wbytes = kind == PB_STAGE_DENSE ? es * (uint64_t)p->C * p->K
                          : kind == PB_STAGE_DWCONV ? es * (uint64_t)p->K * p->R * p->S : 0;
    out->bytes = wbytes + (out->bytes - wbytes) * (uint64_t)nb;
    return PB_OK;
}

static thread_local size_t t_launch_smem = 0;      // dynamic shared memory of the next launch_k (reset by it)

template <typename... KArgs, typename... Args>
static void launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, bool pdl, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.dynamicSmemBytes = t_launch_smem;
    t_launch_smem = 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

int simple_op_launch(int kind, const pb_op_params* p, cudaStream_t st, uint32_t job_id, void* notifier, bool pdl) {
    if (kind == PB_STAGE_CONV_SIMT && conv_f32_supported(p)) return conv_f32_launch(p, to_args(p), st, job_id, notifier, pdl);
    FinishedBlockNotifier* nf = static_cast<FinishedBlockNotifier*>(notifier);
    pb_launch_info li;
    pb_op_params folded;
    int nb = batch_of(p);
    if (nb > 1 && folds_batch(kind)) {
        folded = *p;
        folded.H *= nb;
        folded.batch = 1;
        p = &folded;
        nb = 1;
    }
    int rc = info_one_image(kind, p, &li);
    if (rc != PB_OK) return rc;
    const OpArgs a = to_args(p);
    const bool f32 = p->dtype == 0;
    const int N = vec_n(p->dtype);
    if (kind == PB_STAGE_INPUT) PB_REQUIRE(p->Ks % N == 0, "output channel stride %d is not a multiple of the %d-element vector", p->Ks, N);
    else PB_REQUIRE(p->Cs % N == 0, "channel stride %d is not a multiple of the %d-element vector", p->Cs, N);
    const dim3 grid(li.num_blocks, (unsigned)nb), block(256);      // blockIdx.y = image
#ifdef PB_DEBUG_SKIP
    // development builds only: PB_DEBUG_SKIP_MEMBOUND=1 leaves out the pooling / layout kernels that never notify
    // (wrong results; shows what they cost the tensor-core kernels under load)
    if (job_id != kSlotNotify && nf == nullptr || job_id == kSlotQuiet) {
        const char* e = getenv("PB_DEBUG_SKIP_MEMBOUND");
        const int mask = e ? atoi(e) : 0;      // 1 layout, 2 max pooling, 4 average pooling
        if ((kind == PB_STAGE_INPUT && (mask & 1)) || (kind == PB_STAGE_MAXPOOL && (mask & 2)) || (kind == PB_STAGE_AVGPOOL && (mask & 4))) return PB_OK;
    }
#endif
#define PB_DISPATCH(kern_f32, kern_bf16, ...)                                           \
    do {                                                                                \
        if (f32) launch_k(kern_f32, grid, block, st, pdl, __VA_ARGS__);                 \
        else launch_k(kern_bf16, grid, block, st, pdl, __VA_ARGS__);                    \
    } while (0)
    switch (kind) {
        case PB_STAGE_INPUT:
            if (p->R * p->S > 1) {
                PB_REQUIRE(p->Ks >= p->R * p->S * p->C, "input patches: row stride %d is shorter than R*S*C = %d", p->Ks, p->R * p->S * p->C);
                if (const size_t sm = patch_tile_smem(p)) {
                    t_launch_smem = sm;
                    if (f32) launch_k(input_patch_tile_kernel<float>, grid, block, st, pdl, a, job_id, nf);
                    else launch_k(input_patch_tile_kernel<__nv_bfloat16>, grid, block, st, pdl, a, job_id, nf);
                    break;
                }
                PB_DISPATCH(input_patch_kernel<float>, input_patch_kernel<__nv_bfloat16>, a, job_id, nf);
                break;
            }
            if (f32) launch_k(input_transform_kernel<float>, grid, block, st, pdl, (const float*)p->x, (float*)p->y, p->C, p->H * p->W, p->Ks, job_id, nf);
            else launch_k(input_transform_kernel<__nv_bfloat16>, grid, block, st, pdl, (const float*)p->x, (__nv_bfloat16*)p->y, p->C, p->H * p->W, p->Ks, job_id, nf);
            break;
        case PB_STAGE_CONV_SIMT:
            PB_REQUIRE(a.C % a.groups == 0 && a.K % a.groups == 0, "conv: groups must divide channels");
            PB_DISPATCH(conv_simt_kernel<float>, conv_simt_kernel<__nv_bfloat16>, a, job_id, nf);
            break;
        case PB_STAGE_DWCONV:
            PB_REQUIRE(a.groups == a.C && a.K == a.C, "dwconv: needs groups == C == K");
            PB_REQUIRE((a.Ks % N) == 0 && (a.out_c_off % N) == 0, "dwconv: output slice must be vector aligned");
            if (const WinRing r = win_ring(kind, p); r.blocks) {
                const void* fn = ring_fn(p);
                PB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, r.smem));
                t_launch_smem = (size_t)r.smem;
                CUtensorMap tmap;
                const int mrc = ring_map(p, r, &tmap);
                if (mrc != PB_OK) return mrc;
                launch_k((void (*)(OpArgs, const WinRing, const CUtensorMap, uint32_t, FinishedBlockNotifier*))fn, dim3((unsigned)r.blocks), dim3((unsigned)r.threads), st, pdl, a, r, tmap, job_id, nf);
                break;
            }
            if (tile_blocks(kind, p)) {
                const WinTile g = win_tile(kind, p);
                const void* fn = tile_fn(kind, p);
                PB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, g.smem));
                t_launch_smem = (size_t)g.smem;
                CUtensorMap tmap;
                const int mrc = win_map(kind, p, g, &tmap);
                if (mrc != PB_OK) return mrc;
                launch_k((void (*)(OpArgs, WinTile, const CUtensorMap, uint32_t, FinishedBlockNotifier*))fn, grid, dim3((unsigned)g.threads), st, pdl, a, g, tmap, job_id, nf);
                break;
            }
            if (const int strip = strip_of(p)) {
                t_launch_smem = strip > 1 ? (size_t)window3_smem_bytes(p->Cs, f32 ? 4 : 2) : 0;
                launch_k((void (*)(OpArgs, uint32_t, FinishedBlockNotifier*))window3_fn(kind, f32, p->stride_h, strip), grid, block, st, pdl, a, job_id, nf);
                break;
            }
            PB_DISPATCH(dwconv_kernel<float>, dwconv_kernel<__nv_bfloat16>, a, job_id, nf);
            break;
        case PB_STAGE_MAXPOOL:
            PB_REQUIRE((a.Ks % N) == 0 && (a.out_c_off % N) == 0, "pool: output slice must be vector aligned");
            if (tile_blocks(kind, p)) {
                const WinTile g = win_tile(kind, p);
                const void* fn = tile_fn(kind, p);
                PB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, g.smem));
                t_launch_smem = (size_t)g.smem;
                CUtensorMap tmap;
                const int mrc = win_map(kind, p, g, &tmap);
                if (mrc != PB_OK) return mrc;
                launch_k((void (*)(OpArgs, WinTile, const CUtensorMap, uint32_t, FinishedBlockNotifier*))fn, grid, dim3((unsigned)g.threads), st, pdl, a, g, tmap, job_id, nf);
                break;
            }
            if (const int strip = strip_of(p)) {
                launch_k((void (*)(OpArgs, uint32_t, FinishedBlockNotifier*))window3_fn(kind, f32, p->stride_h, strip), grid, block, st, pdl, a, job_id, nf);
                break;
            }
            if (pool2(p)) {
                PB_DISPATCH((pool2_kernel<float, true>), (pool2_kernel<__nv_bfloat16, true>), a, job_id, nf);
                break;
            }
            PB_DISPATCH((pool_kernel<float, true>), (pool_kernel<__nv_bfloat16, true>), a, job_id, nf);
            break;
        case PB_STAGE_AVGPOOL:
            PB_REQUIRE((a.Ks % N) == 0 && (a.out_c_off % N) == 0, "pool: output slice must be vector aligned");
            if (tile_blocks(kind, p)) {
                const WinTile g = win_tile(kind, p);
                const void* fn = tile_fn(kind, p);
                PB_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, g.smem));
                t_launch_smem = (size_t)g.smem;
                CUtensorMap tmap;
                const int mrc = win_map(kind, p, g, &tmap);
                if (mrc != PB_OK) return mrc;
                launch_k((void (*)(OpArgs, WinTile, const CUtensorMap, uint32_t, FinishedBlockNotifier*))fn, grid, dim3((unsigned)g.threads), st, pdl, a, g, tmap, job_id, nf);
                break;
            }
            if (const int strip = strip_of(p)) {
                launch_k((void (*)(OpArgs, uint32_t, FinishedBlockNotifier*))window3_fn(kind, f32, p->stride_h, strip), grid, block, st, pdl, a, job_id, nf);
                break;
            }
            if (pool2(p)) {
                PB_DISPATCH((pool2_kernel<float, false>), (pool2_kernel<__nv_bfloat16, false>), a, job_id, nf);
                break;
            }
            PB_DISPATCH((pool_kernel<float, false>), (pool_kernel<__nv_bfloat16, false>), a, job_id, nf);
            break;
        case PB_STAGE_GAP:
            PB_DISPATCH(gap_kernel<float>, gap_kernel<__nv_bfloat16>, a, job_id, nf);
            break;
        case PB_STAGE_DENSE:
            PB_REQUIRE(a.C % N == 0, "dense: input length %d is not a multiple of %d", a.C, N);
            PB_DISPATCH(dense_kernel<float>, dense_kernel<__nv_bfloat16>, a, job_id, nf);
            break;
        case PB_STAGE_ADD:
            PB_REQUIRE(a.residual != nullptr, "add: second operand missing");
            PB_DISPATCH(add_kernel<float>, add_kernel<__nv_bfloat16>, a, job_id, nf);
            break;
        case PB_STAGE_AFFINE:
            PB_REQUIRE(a.w != nullptr && a.bias != nullptr, "affine: scale and bias are required");
            PB_REQUIRE((a.Ks % N) == 0 && (a.out_c_off % N) == 0, "affine: output slice must be vector aligned");
            PB_DISPATCH(affine_kernel<float>, affine_kernel<__nv_bfloat16>, a, job_id, nf);
            break;
        case PB_STAGE_SOFTMAX:
            // flags bit2: the input is fp32 regardless of dtype
            if (f32 || (p->flags & 4)) launch_k(softmax_kernel<float, true>, grid, block, st, pdl, a, job_id, nf);
            else launch_k(softmax_kernel<__nv_bfloat16, false>, grid, block, st, pdl, a, job_id, nf);
            break;
        case PB_STAGE_DETECT:
            PB_REQUIRE(a.w != nullptr && a.bias != nullptr && a.C % 6 == 0 && a.C > 0, "detect: priors, variances and 6 channels per anchor are required");
            PB_REQUIRE((p->flags & 2) != 0, "detect: writes the fp32 model output only");
            PB_REQUIRE((size_t)a.out_c_off + (size_t)a.H * a.W * (a.C / 6) <= (size_t)a.K, "detect: priors of this map exceed the model's count");
            PB_DISPATCH(detect_kernel<float>, detect_kernel<__nv_bfloat16>, a, job_id, nf);
            break;
        default:
            set_error("pb_op_launch: unknown stage kind %d", kind);
            return PB_ERR_INVALID;
    }
#undef PB_DISPATCH
    return launch_check("operator kernel");
}

// Weight layouts (host side).  Source: OIHW fp32.
//  conv_simt: [R][S][C/groups][K]      dwconv: [R][S][Cs]      dense: see graph loader
static uint16_t f32_to_bf16_bits(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)((u >> 16) | 0x40);
    u += 0x7fffu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}

void store_elem(void* dst, size_t i, float v, int dtype) {
    if (dtype == 0) static_cast<float*>(dst)[i] = v;
    else static_cast<uint16_t*>(dst)[i] = f32_to_bf16_bits(v);
}

int64_t simple_pack_weights(int kind, const pb_op_params* p, const float* w, void* dst) {
    if (kind == PB_STAGE_CONV_SIMT && conv_f32_supported(p)) return conv_f32_pack_weights(p, w, dst);
    const size_t es = elem_size(p->dtype);
    const int groups = p->groups > 0 ? p->groups : 1;
    if (kind == PB_STAGE_CONV_SIMT) {
        const int cg = p->C / groups;
        const size_t n = (size_t)p->R * p->S * cg * p->K;
        if (dst) {
            for (int k = 0; k < p->K; ++k)
                for (int c = 0; c < cg; ++c)
                    for (int r = 0; r < p->R; ++r)
                        for (int s = 0; s < p->S; ++s)
                            store_elem(dst, ((size_t)(r * p->S + s) * cg + c) * p->K + k,
                                       w[(((size_t)k * cg + c) * p->R + r) * p->S + s], p->dtype);
        }
        return (int64_t)(n * es);
    }
    if (kind == PB_STAGE_DWCONV) {
        const size_t n = (size_t)p->R * p->S * p->Cs;
        if (dst) {
            memset(dst, 0, n * es);
            for (int c = 0; c < p->C; ++c)
                for (int r = 0; r < p->R; ++r)
                    for (int s = 0; s < p->S; ++s)
                        store_elem(dst, (size_t)(r * p->S + s) * p->Cs + c, w[((size_t)c * p->R + r) * p->S + s], p->dtype);
        }
        return (int64_t)(n * es);
    }
    set_error("pb_op_pack_weights: stage kind %d has no packed weights here", kind);
    return PB_ERR_INVALID;
}

int mnist_fused_info(int batch, pb_launch_info* out) {
    const bool gang = batch > 1;
    const uint32_t nb = gang ? (uint32_t)batch : 1u;
    memset(out, 0, sizeof(*out));
    out->kind = PB_STAGE_MNIST_FUSED;
    out->num_blocks = nb;
    out->threads_per_block = gang ? 256 : 256 * kMnistRanks;      // a lone image's cluster counts as one block
    out->regs_per_thread = gang ? regs_of(mnist_gang_kernel) : regs_of(mnist_fused_kernel);
    out->smem_per_block = gang ? static_smem_of(mnist_gang_kernel) : kMnistRanks * static_smem_of(mnist_fused_kernel);
    out->flops = nb * 2ull * (156800 + 627200 + 2560);      // the layers as the model states them
    out->bytes = nb * 4ull * (784 + 200 + 8 + 3200 + 16 + 2560 + 10 + 10);
    return PB_OK;
}

int mnist_fused_launch(const float* x, const float* w1, const float* b1, const float* w2, const float* b2,
                       const float* wd, const float* bd, float* y, int batch, cudaStream_t st, uint32_t job_id, void* notifier) {
    MnistArgs a{x, w1, b1, w2, b2, wd, bd, y};
    FinishedBlockNotifier* const nf = static_cast<FinishedBlockNotifier*>(notifier);
    if (batch > 1) {
        mnist_gang_kernel<<<batch, 256, 0, st>>>(a, job_id, nf);
        return launch_check("mnist_gang");
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kMnistRanks);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kMnistRanks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PB_CUDA(cudaLaunchKernelEx(&cfg, mnist_fused_kernel, a, job_id, nf));
    return PB_OK;
}

}  // namespace pb
