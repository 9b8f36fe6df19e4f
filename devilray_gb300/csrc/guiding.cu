// guiding.cu -- the path-guiding network on tensor cores: inference, one
// training step (forward, loss gradient, backward, weight gradients) and Adam.
//
// Network: 80 inputs (12-frequency encoding of the normalised position, a
// direction, zero padding) -> 4 hidden layers of 64 (ReLU) -> 48 outputs (40
// used: the 8-lobe vMF mixture of guide_math.cuh). Weights and layer inputs
// are BF16, every product accumulates in FP32; master weights and Adam moments
// are FP32. Inference and training run on the 5th-generation tensor cores
// (k_guide_infer_tc, k_guide_train_fused); the kernels with warp-level mma.sync
// m16n8k16 are their alternatives and work as follows.
//
// A warp carries 16 rows through all layers in registers: the FP32
// accumulator fragment of one layer is, pair by pair, the BF16 A fragment of
// the next (m16n8 C layout = m16k16 A layout of two adjacent column tiles).
// Backward products use the transposed weights, staged in shared memory; the
// deltas enter the tensor cores as a BF16 high part plus a BF16 remainder so
// the propagated gradient keeps about 16 bits. Weight gradients are
// delta^T x activations over the batch (K = rows), split over row chunks and
// summed with atomics.

#include "dr_internal.h"
#include "mbarrier.cuh"
#include "guide_math.cuh"
#include "guide_internal.h"
#include "launch.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <random>
#include <vector>

namespace dr {
namespace {

constexpr int kIn = 80, kHid = 64, kOut = 48, kLayers = 5;

__host__ __device__ constexpr int fan_in(int l) { return l == 0 ? kIn : kHid; }
__host__ __device__ constexpr int fan_out(int l) { return l == kLayers - 1 ? kOut : kHid; }

__host__ __device__ constexpr int w_off(int l)
{
    int o = 0;
    for (int i = 0; i < l; ++i) o += fan_out(i) * fan_in(i) + fan_out(i);
    return o;
}
__host__ __device__ constexpr int b_off(int l) { return w_off(l) + fan_out(l) * fan_in(l); }
constexpr int kNumParams = w_off(kLayers);
// BF16 weights (no biases) in the same order, for the kernels
__host__ __device__ constexpr int wb_off(int l)
{
    int o = 0;
    for (int i = 0; i < l; ++i) o += fan_out(i) * fan_in(i);
    return o;
}
constexpr int kNumWeights = wb_off(kLayers);

// shared-memory strides (bf16 elements), padded so the 8 rows of a fragment
// load fall in distinct banks
constexpr int kStrideIn = kIn + 8;    // 88
constexpr int kStrideHid = kHid + 8;  // 72
constexpr int kStrideOutT = kOut + 8; // 56: transposed last layer [64][48]

struct GuideParams {
    float center[3];
    float half;
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Encoded input pair (columns c, c + 1; c even) of a row.
__device__ __forceinline__ void encode_pair(const float p[3], const float d[3], int c, float &v0, float &v1)
{
    if (c < 72) {
        const int a = c / 24, k = (c % 24) >> 1;
        const float x = p[a] * (float)(1 << k);  // exact: a power of two
        sincospif(x, &v0, &v1);
    } else if (c == 72) {
        v0 = d[0];
        v1 = d[1];
    } else if (c == 74) {
        v0 = d[2];
        v1 = 0.0f;
    } else {
        v0 = v1 = 0.0f;
    }
}

// Shared-memory image of the weights: forward W_l [out][in] and, for the
// backward pass, W_l^T [in][out] of layers 1..4.
struct SmemWeights {
    __nv_bfloat16 w0[kHid * kStrideIn];
    __nv_bfloat16 w[3][kHid * kStrideHid];     // layers 1..3
    __nv_bfloat16 w4[kOut * kStrideHid];
    float bias[4 * kHid + kOut];
};
struct SmemWeightsT {
    __nv_bfloat16 t[3][kHid * kStrideHid];     // W_l^T, l = 1..3: [in 64][out 64]
    __nv_bfloat16 t4[kHid * kStrideOutT];      // W_4^T: [in 64][out 48]
};

__device__ void load_weights(SmemWeights &s, const __nv_bfloat16 *wb, const float *params)
{
    for (int i = threadIdx.x; i < kHid * kIn; i += blockDim.x) s.w0[(i / kIn) * kStrideIn + i % kIn] = wb[i];
    for (int l = 1; l <= 3; ++l)
        for (int i = threadIdx.x; i < kHid * kHid; i += blockDim.x)
            s.w[l - 1][(i / kHid) * kStrideHid + i % kHid] = wb[wb_off(l) + i];
    for (int i = threadIdx.x; i < kOut * kHid; i += blockDim.x) s.w4[(i / kHid) * kStrideHid + i % kHid] = wb[wb_off(4) + i];
    for (int l = 0; l < kLayers; ++l)
        for (int i = threadIdx.x; i < fan_out(l); i += blockDim.x) s.bias[l * kHid + i] = params[b_off(l) + i];
}

__device__ void load_weights_t(SmemWeightsT &s, const __nv_bfloat16 *wb)
{
    for (int l = 1; l <= 3; ++l)
        for (int i = threadIdx.x; i < kHid * kHid; i += blockDim.x) {
            const int o = i / kHid, in = i % kHid;
            s.t[l - 1][in * kStrideHid + o] = wb[wb_off(l) + i];
        }
    for (int i = threadIdx.x; i < kOut * kHid; i += blockDim.x) {
        const int o = i / kHid, in = i % kHid;
        s.t4[in * kStrideOutT + o] = wb[wb_off(4) + i];
    }
}

__device__ __forceinline__ uint32_t ld_pair(const __nv_bfloat16 *p) { return *reinterpret_cast<const uint32_t *>(p); }

// acc[nt] += A (16 x 16 ks-slices) x B where B[k][n] = W[n][k], W row-major with
// `stride`; NT column tiles of 8, KS k-steps of 16.
template <int NT, int KS>
__device__ __forceinline__ void layer_mma(float (&acc)[NT][4], const uint32_t (&a)[KS][4], const __nv_bfloat16 *W,
                                          int stride)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const __nv_bfloat16 *row = W + (8 * nt + g) * stride + 16 * ks + 2 * tig;
            mma_bf16(acc[nt], a[ks], ld_pair(row), ld_pair(row + 8));
        }
}

template <int NT>
__device__ __forceinline__ void init_bias(float (&acc)[NT][4], const float *bias)
{
    const int tig = threadIdx.x & 3;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const float b0 = bias[8 * nt + 2 * tig], b1 = bias[8 * nt + 2 * tig + 1];
        acc[nt][0] = b0, acc[nt][1] = b1, acc[nt][2] = b0, acc[nt][3] = b1;
    }
}

// ReLU of a 64-wide accumulator, as the A fragments of the next layer.
__device__ __forceinline__ void relu_to_a(const float (&acc)[8][4], uint32_t (&a)[4][4])
{
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        const float *l = acc[2 * ks], *h = acc[2 * ks + 1];
        a[ks][0] = pack_bf16(fmaxf(l[0], 0.0f), fmaxf(l[1], 0.0f));
        a[ks][1] = pack_bf16(fmaxf(l[2], 0.0f), fmaxf(l[3], 0.0f));
        a[ks][2] = pack_bf16(fmaxf(h[0], 0.0f), fmaxf(h[1], 0.0f));
        a[ks][3] = pack_bf16(fmaxf(h[2], 0.0f), fmaxf(h[3], 0.0f));
    }
}

// Input fragments of 16 rows (5 k-steps of 16 encoded columns).
__device__ __forceinline__ void input_frags(const float p_g[3], const float d_g[3], const float p_h[3],
                                            const float d_h[3], uint32_t (&a)[5][4])
{
    const int tig = threadIdx.x & 3;
#pragma unroll
    for (int ks = 0; ks < 5; ++ks) {
        float v0, v1;
        const int c0 = 16 * ks + 2 * tig, c1 = c0 + 8;
        encode_pair(p_g, d_g, c0, v0, v1);
        a[ks][0] = pack_bf16(v0, v1);
        encode_pair(p_h, d_h, c0, v0, v1);
        a[ks][1] = pack_bf16(v0, v1);
        encode_pair(p_g, d_g, c1, v0, v1);
        a[ks][2] = pack_bf16(v0, v1);
        encode_pair(p_h, d_h, c1, v0, v1);
        a[ks][3] = pack_bf16(v0, v1);
    }
}

__device__ __forceinline__ void load_row(const float *pos, const float *dir, const uint32_t *list, uint32_t n, uint32_t r,
                                         const GuideParams &gp, float p[3], float d[3], uint32_t &slot)
{
    slot = r < n ? (list ? list[r] : r) : 0xffffffffu;
    if (r >= n) {
        p[0] = p[1] = p[2] = d[0] = d[1] = d[2] = 0.0f;
        return;
    }
    for (int a = 0; a < 3; ++a) {
        const float x = (pos[3 * (size_t)slot + a] - gp.center[a]) / gp.half;
        p[a] = fminf(1.0f, fmaxf(-1.0f, x));
        d[a] = dir[3 * (size_t)slot + a];
    }
}

// Forward pass of 16 rows per warp; y[slot][40] for rows r < n (slot = list[r]
// or r). Grid-stride over 16-row tiles.
__global__ void __launch_bounds__(128) k_guide_infer(const __nv_bfloat16 *wb, const float *params, GuideParams gp,
                                                     const float *pos, const float *dir, const uint32_t *list,
                                                     const uint32_t *count, uint32_t n_fixed, float *y)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SmemWeights &s = *reinterpret_cast<SmemWeights *>(smem);
    load_weights(s, wb, params);
    __syncthreads();
    const uint32_t n = count ? *count : n_fixed;
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); 16ull * tile < n; tile += warps) {
        const uint32_t r0 = 16 * tile;
        float pg[3], dg[3], ph[3], dh[3];
        uint32_t sg, sh;
        load_row(pos, dir, list, n, r0 + g, gp, pg, dg, sg);
        load_row(pos, dir, list, n, r0 + g + 8, gp, ph, dh, sh);
        uint32_t a0[5][4];
        input_frags(pg, dg, ph, dh, a0);
        float acc[8][4];
        uint32_t a[4][4];
        init_bias(acc, s.bias);
        layer_mma<8, 5>(acc, a0, s.w0, kStrideIn);
        relu_to_a(acc, a);
#pragma unroll
        for (int l = 1; l <= 3; ++l) {
            init_bias(acc, s.bias + l * kHid);
            layer_mma<8, 4>(acc, a, s.w[l - 1], kStrideHid);
            relu_to_a(acc, a);
        }
        float out[6][4];
        init_bias(out, s.bias + 4 * kHid);
        layer_mma<6, 4>(out, a, s.w4, kStrideHid);
#pragma unroll
        for (int nt = 0; nt < 5; ++nt) {
            const int c = 8 * nt + 2 * tig;
            if (sg != 0xffffffffu)
                *reinterpret_cast<float2 *>(y + (size_t)sg * kGuideOut + c) = make_float2(out[nt][0], out[nt][1]);
            if (sh != 0xffffffffu)
                *reinterpret_cast<float2 *>(y + (size_t)sh * kGuideOut + c) = make_float2(out[nt][2], out[nt][3]);
        }
    }
}


// ---- inference on the 5th-generation tensor cores (tcgen05) -------------------
//
// One CTA per SM holds the weights in shared memory once, in the canonical
// K-major layout without swizzle, and kInferGroups groups of 128 threads, each
// with an input tile, 64 tensor-memory columns and an mbarrier of its own. A
// group carries tiles of 128 rows (the M of one tcgen05.mma) through the
// network: one lane of its first warp, elected while the warp is converged,
// issues the K/16 MMAs of a layer into the 128 x N FP32 accumulator and commits
// them to the mbarrier (chosen by its thread index instead, it moved every
// operand to the uniform registers by itself: 106 against 95 us), and each warp
// reads its 32 rows back with tcgen05.ld for the bias / ReLU / BF16 epilogue, which writes
// the next layer's input. Groups do not wait for one another: while one is in
// its chain of MMA, commit, tensor-memory read and barrier, the others encode
// inputs and run epilogues. Same arithmetic as k_guide_infer (BF16 products,
// FP32 sums). Bound by the shared / tensor memory data path (0.6 of it by loads
// and stores, the operands of the MMAs beside them) and by that chain's latency;
// 0.58 of the issue slots, 0.3 of HBM for 2^20 rows in 95 us (98 since the ReLU takes
// a NaN to 0, an instruction more per pair). The sines and cosines
// of the inputs are some 19 us of it; outputs of whole tiles leave as one bulk copy
// (117 against 108 us when every tile's rows went through loads and stores).

constexpr int kTcRows = 128;

// Byte offset of element (r, c) of an R x K BF16 matrix in the canonical
// K-major layout: core matrices of 8 rows x 8 columns (8 rows of 16 bytes);
// column chunk j (columns 8j..8j+7) of all R rows is contiguous.
__device__ __forceinline__ uint32_t canon_off(int r, int c, int R) { return (uint32_t)((c >> 3) * R * 16 + r * 16 + (c & 7) * 2); }

// Shared-memory matrix descriptor: start address, leading byte offset (between
// core matrices adjacent along K) and stride byte offset (between core
// matrices adjacent along M or N), all >> 4; version 1 (bits 46-47); no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded wait on an mbarrier phase; false after the iteration limit.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase, uint32_t polls = kMbarWaitPolls)
{
    return mbar_wait_bounded(mbar, phase, polls);
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t arrivals)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(mbar), "r"(arrivals) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

// Arrives on `mbar` once every product that this thread has issued is complete.
__device__ __forceinline__ void commit_products(uint32_t mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar) : "memory");
}

// True in one lane of a converged warp, always the same one.
__device__ __forceinline__ bool elect_one()
{
    uint32_t one;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v)
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float tmem_ld1(uint32_t taddr)
{
    uint32_t r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(r) : "r"(taddr));
    return __uint_as_float(r);
}

// Shared memory of k_guide_infer_tc (byte offsets).
constexpr uint32_t kTcW0 = 0;                        // 64 x 80
constexpr uint32_t kTcW1 = kTcW0 + 64 * 80 * 2;      // 3 x 64 x 64
constexpr uint32_t kTcW4 = kTcW1 + 3 * 64 * 64 * 2;  // 48 x 64
constexpr uint32_t kTcA = kTcW4 + 48 * 64 * 2;       // per group: 128 x 80 input / 128 x 64 hidden / 128 x 40 output
constexpr uint32_t kTcABytes = kTcRows * kIn * 2;
static_assert(kTcABytes == kTcRows * kGuideOut * 4, "the output rows fit the input tile");
// Groups per CTA, at that time: 6 run at 80 registers (2^20 rows: 95 us; 200,000
// rows 23.8), 5 at 96 (101; 27.0), 7 and 8 spill at 72 and 64 (94; 24.7 and 25.7). Three CTAs
// of one group each, with their own copies of the weights, took 178 us.
constexpr int kInferGroups = 6;
constexpr uint32_t kTcBias = kTcA + kInferGroups * kTcABytes;
constexpr uint32_t kTcBar = kTcBias + (4 * kHid + kOut) * 4;  // MMA mbarrier of each group, copy mbarrier, TMEM address, drain mbarrier
constexpr uint32_t kTcSmem = kTcBar + 8 * (kInferGroups + 3);

// The weights as the tcgen05 kernels hold them in shared memory, kept in
// global memory beside the BF16 copy so a CTA fetches them with one bulk
// asynchronous copy: W_l at kTcW0..kTcW4 as N = out, K = in, canonical K-major
// (the backward product reads the same bytes MN-major).
constexpr uint32_t kImgBytes = kNumWeights * 2;

__device__ __forceinline__ void store_weight(__nv_bfloat16 *wb, unsigned char *img, int l, int idx, float p)
{
    const __nv_bfloat16 b = __float2bfloat16_rn(p);
    wb[wb_off(l) + idx] = b;
    const int o = idx / fan_in(l), in = idx % fan_in(l);
    const uint32_t fwd = l == 0 ? kTcW0 : l == 4 ? kTcW4 : kTcW1 + (uint32_t)(l - 1) * kHid * kHid * 2;
    *reinterpret_cast<__nv_bfloat16 *>(img + fwd + canon_off(o, in, fan_out(l))) = b;
}

// One bulk asynchronous copy of `bytes` of the weight image into shared
// memory, completing on the mbarrier `cbar` (issued by one thread).
__device__ __forceinline__ void fetch_weight_image(uint32_t dst, const unsigned char *img, uint32_t bytes, uint32_t cbar)
{
    mbar_init(cbar, 1);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(cbar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(img), "r"(bytes), "r"(cbar)
                 : "memory");
}

// BF16 pair (lo, hi) of max(x, 0), as the layers' inputs are rounded; 0 for a NaN.
__device__ __forceinline__ uint32_t relu_bf16(float lo, float hi)
{
    const __nv_bfloat162 v = __hmax2(__floats2bfloat162_rn(lo, hi), __floats2bfloat162_rn(0.0f, 0.0f));
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;\n" ::"r"(group + 1) : "memory"); }

template <bool DECODED>
__global__ void __launch_bounds__(128 * kInferGroups, 1)
k_guide_infer_tc(const unsigned char *img, const float *params, GuideParams gp, const float *pos, const float *dir,
                 const uint32_t *list, const uint32_t *count, uint32_t n_fixed, float *y, uint32_t polls, uint32_t *error)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ int s_failed;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, group = warp >> 2, row = tid & 127;
    allow_next();
    wait_previous();
    const uint32_t n = count ? *count : n_fixed;
    if ((uint64_t)blockIdx.x * kTcRows >= n) return;  // the whole block
    // weights in the canonical layout (B operands: N = outputs, K = inputs):
    // the weight image, one bulk copy
    const uint32_t cbar = smem_u32(smem + kTcBar + 8 * kInferGroups);
    const uint32_t tslot = cbar + 8, dbar = cbar + 16, mbar = smem_u32(smem + kTcBar) + 8 * group;
    if (tid == 0) {
        s_failed = 0;
        mbar_init(dbar, kInferGroups);
        fetch_weight_image(smem_u32(smem + kTcW0), img, kImgBytes, cbar);
    }
    if (row == 0) mbar_init(mbar, 1);
    float *bias = reinterpret_cast<float *>(smem + kTcBias);
    for (int i = tid; i < 4 * kHid + kOut; i += blockDim.x) bias[i] = params[b_off(i / kHid) + i % kHid];
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(tslot) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t taddr = *reinterpret_cast<volatile uint32_t *>(smem + kTcBar + 8 * kInferGroups + 8);
    const uint32_t acc = taddr + 64u * group, lane_addr = acc + ((uint32_t)((warp & 3) * 32) << 16);
    unsigned char *A = smem + kTcA + group * kTcABytes;
    const uint32_t a_base = smem_u32(A);
    uint32_t phase = 0;
    // Every wait is bounded. A thread whose wait gives up (or that sees the
    // block's flag) goes on through its group's barriers without working, so the
    // block ends together.
    auto wait = [&](uint32_t bar, uint32_t ph, uint32_t limit) {
        if (*reinterpret_cast<volatile int *>(&s_failed)) return false;
        if (mbar_wait(bar, ph, limit)) return true;
        *reinterpret_cast<volatile int *>(&s_failed) = 1;
        atomicOr(error, ERR_TIMEOUT);
        return false;
    };
    bool ok = wait(cbar, 0, kMbarWaitPolls);  // the weights have landed
    // tiles go to the blocks first, then to the groups of each block
    for (uint32_t tile = blockIdx.x + gridDim.x * group; (uint64_t)tile * kTcRows < n; tile += gridDim.x * kInferGroups) {
        const uint32_t r = tile * kTcRows + row;
        float p[3], d[3];
        uint32_t slot;
        load_row(pos, dir, list, n, r, gp, p, d, slot);
        // the next tile's rows, while this one is carried through
        const uint32_t ahead = r + 128u * gridDim.x * kInferGroups;
        if (ahead < n) {
            const uint32_t s2 = list ? list[ahead] : ahead;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(pos + 3 * (size_t)s2));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(dir + 3 * (size_t)s2));
        }
        // input row: 10 chunks of 8 encoded columns
#pragma unroll
        for (int j = 0; j < kIn / 8; ++j) {
            uint32_t q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float v0, v1;
                encode_pair(p, d, 8 * j + 2 * k, v0, v1);
                q[k] = pack_bf16(v0, v1);
            }
            *reinterpret_cast<uint4 *>(A + canon_off(row, 8 * j, kTcRows)) = make_uint4(q[0], q[1], q[2], q[3]);
        }
        const bool run = !DECODED && !list && (tile + 1) * kTcRows <= n;  // the tile's outputs are one run of memory
        uint32_t w_base = smem_u32(smem + kTcW0);
#pragma unroll 1
        for (int l = 0; l < kLayers; ++l) {
            const int K = fan_in(l), N = fan_out(l);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            group_sync(group);
            if ((warp & 3) == 0) {
                if (__all_sync(0xffffffffu, ok) && elect_one()) {
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t idesc = idesc_bf16(kTcRows, N);
                    uint64_t ad = smem_desc(a_base, kTcRows * 16, 128), bd = smem_desc(w_base, (uint32_t)N * 16, 128);
#pragma unroll
                    for (int s2 = 0; s2 < kIn / 16; ++s2) {
                        if (16 * s2 >= K) break;
                        asm volatile(
                            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc),
                            "l"(ad), "l"(bd), "r"(idesc), "r"(s2));
                        ad += 2 * kTcRows * 16 / 16;  // the next 16 columns of both operands
                        bd += 2 * N * 16 / 16;
                    }
                    commit_products(mbar);
                }
                __syncwarp();
            }
            ok = wait(mbar, phase, polls) && ok;
            phase ^= 1u;
            w_base += (uint32_t)(K * N * 2);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const float4 *b = reinterpret_cast<const float4 *>(bias + l * kHid);
            if (l < kLayers - 1) {
#pragma unroll
                for (int h = 0; h < 64; h += 16) {  // 16 columns at once: 32 are no faster
                    float v[16];
                    tmem_ld16(lane_addr + h, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        uint32_t q[4];
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int i = 8 * j + 4 * k;
                            const float4 c = b[(h + i) / 4];
                            const float2 x = __fadd2_rn(make_float2(v[i], v[i + 1]), make_float2(c.x, c.y));
                            const float2 z = __fadd2_rn(make_float2(v[i + 2], v[i + 3]), make_float2(c.z, c.w));
                            q[2 * k] = relu_bf16(x.x, x.y);
                            q[2 * k + 1] = relu_bf16(z.x, z.y);
                        }
                        *reinterpret_cast<uint4 *>(A + canon_off(row, h + 8 * j, kTcRows)) = make_uint4(q[0], q[1], q[2], q[3]);
                    }
                }
            } else {
                // the output rows, through shared memory (the tile's inputs are
                // spent): each warp stages its 32 rows and writes them out as
                // runs of 160 bytes, ten lanes per row
                // rows 4..7 of every 8 are turned by one float4, so that eight
                // lanes' stores fall in distinct banks
                constexpr int kQ = kGuideOut / 4;
                float4 *stage = reinterpret_cast<float4 *>(A + (warp & 3) * 32 * kGuideOut * 4);
                const int turn = (lane >> 2) & 1;
                auto put = [&](int j, float4 q) { stage[lane * kQ + (j < kQ - 1 ? turn + j : turn ? 0 : kQ - 1)] = q; };
                if (DECODED) {
                    float o[48], out[kGuideOut];
#pragma unroll
                    for (int c = 0; c < 48; c += 16) tmem_ld16(lane_addr + c, o + c);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                    float v[kGuideOut];
#pragma unroll
                    for (int i = 0; i < kQ; ++i) {
                        const float4 c = b[i];
                        v[4 * i] = o[4 * i] + c.x, v[4 * i + 1] = o[4 * i + 1] + c.y;
                        v[4 * i + 2] = o[4 * i + 2] + c.z, v[4 * i + 3] = o[4 * i + 3] + c.w;
                    }
                    guide_store_decoded(out, guide_mix_values(v));
#pragma unroll
                    for (int j = 0; j < kQ; ++j) put(j, reinterpret_cast<const float4 *>(out)[j]);
                } else {
                    float o[kGuideOut];
                    {
                        float v[48];
#pragma unroll
                        for (int c = 0; c < 48; c += 16) tmem_ld16(lane_addr + c, v + c);
                        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                        for (int i = 0; i < kQ; ++i) {
                            const float4 c = b[i];
                            o[4 * i] = v[4 * i] + c.x, o[4 * i + 1] = v[4 * i + 1] + c.y;
                            o[4 * i + 2] = v[4 * i + 2] + c.z, o[4 * i + 3] = v[4 * i + 3] + c.w;
                        }
                    }
                    const float4 *q = reinterpret_cast<const float4 *>(o);
                    if (run) {
                        // rows in place; lanes 4..7 of every 8 are one float4 ahead,
                        // so that eight lanes' stores fall in distinct banks
#pragma unroll
                        for (int j = 0; j < kQ; ++j) {
                            const float4 v0 = q[j], v1 = q[(j + 1) % kQ];
                            stage[lane * kQ + (turn ? (j + 1) % kQ : j)] =
                                make_float4(turn ? v1.x : v0.x, turn ? v1.y : v0.y, turn ? v1.z : v0.z, turn ? v1.w : v0.w);
                        }
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        group_sync(group);
                        if (row == 0 && ok) {
                            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(
                                             y + (size_t)tile * kTcRows * kGuideOut),
                                         "r"(a_base), "r"(kTcABytes)
                                         : "memory");
                            asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                            asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                        }
                        break;  // the last layer
                    }
#pragma unroll
                    for (int j = 0; j < kQ; ++j) put(j, q[j]);
                }
                __syncwarp();
                const int part = lane / kQ, col = lane - part * kQ;
#pragma unroll
                for (int j = 0; j < 11; ++j) {
                    const int at = 3 * j + part;
                    const uint32_t to = __shfl_sync(0xffffffffu, slot, at & 31);
                    if (part < 3 && at < 32 && to != 0xffffffffu && ok) {
                        const int c = col + ((at >> 2) & 1);
                        reinterpret_cast<float4 *>(y + (size_t)to * kGuideOut)[col] = stage[at * kQ + (c < kQ ? c : 0)];
                    }
                }
            }
        }
        group_sync(group);  // the staged rows are read before the next tile's inputs replace them
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    // After a wait gave up, products or the weight copy may still be in flight:
    // wait (bounded) before their memory is freed. The lane that issued a group's
    // products commits them all to a barrier of its own: the parity of the
    // group's last commit depends on where the wait gave up.
    if (*reinterpret_cast<volatile int *>(&s_failed)) {
        if ((warp & 3) == 0 && elect_one()) commit_products(dbar);
        if (warp == 0) {
            mbar_wait(dbar, 0);
            mbar_wait(cbar, 0);
        }
        __syncthreads();
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(taddr) : "memory");
}

// ---- training -----------------------------------------------------------------

struct TrainBuffers {
    // per layer l (0..4): delta of the layer output, transposed [out][rows] (FP32),
    // and the layer input, transposed [in][rows] (BF16)
    float *deltaT[kLayers];
    __nv_bfloat16 *actT[kLayers];
    uint32_t rows;  // row stride of the transposed arrays (batch capacity)
};

// Writes a 16 x (8 NT) FP32 accumulator transposed: dst[col][row0 + row].
template <int NT>
__device__ __forceinline__ void store_t(float *dst, uint32_t stride, uint32_t row0, const float (&acc)[NT][4], uint32_t n,
                                        int ncols)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int c = 8 * nt + 2 * tig;
        if (c >= ncols) continue;
        if (row0 + g < n) {
            dst[(size_t)c * stride + row0 + g] = acc[nt][0];
            dst[(size_t)(c + 1) * stride + row0 + g] = acc[nt][1];
        }
        if (row0 + g + 8 < n) {
            dst[(size_t)c * stride + row0 + g + 8] = acc[nt][2];
            dst[(size_t)(c + 1) * stride + row0 + g + 8] = acc[nt][3];
        }
    }
}

// Writes BF16 A fragments (KS k-steps) transposed: dst[col][row0 + row].
template <int KS>
__device__ __forceinline__ void store_a_t(__nv_bfloat16 *dst, uint32_t stride, uint32_t row0, const uint32_t (&a)[KS][4],
                                          uint32_t n)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int row = g + ((q & 1) ? 8 : 0);
            const int c = 16 * ks + 2 * tig + ((q & 2) ? 8 : 0);
            if (row0 + row >= n) continue;
            const uint32_t v = a[ks][q];
            __nv_bfloat16 lo, hi;
            const uint16_t lb = (uint16_t)(v & 0xffffu), hb = (uint16_t)(v >> 16);
            memcpy(&lo, &lb, 2);
            memcpy(&hi, &hb, 2);
            dst[(size_t)c * stride + row0 + row] = lo;
            dst[(size_t)(c + 1) * stride + row0 + row] = hi;
        }
}

// Splits FP32 accumulators of 64 (or 48) columns into BF16 high and low A
// fragments (KS k-steps), after masking by the ReLU of `act` (the layer's
// output fragments) when MASK.
template <int KS, bool MASK>
__device__ __forceinline__ void delta_frags(float (&acc)[2 * KS][4], const uint32_t (&act)[4][4], uint32_t (&hi)[KS][4],
                                            uint32_t (&lo)[KS][4])
{
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            // q: 0 (rows g, tile 2ks) 1 (rows g+8, tile 2ks) 2 (rows g, tile 2ks+1) 3 (rows g+8, tile 2ks+1)
            float *c = acc[2 * ks + (q >> 1)] + ((q & 1) ? 2 : 0);
            if (MASK) {
                const uint32_t m = act[ks][q];
                if ((m & 0x7fffu) == 0) c[0] = 0.0f;
                if ((m & 0x7fff0000u) == 0) c[1] = 0.0f;
            }
            const __nv_bfloat162 h = __floats2bfloat162_rn(c[0], c[1]);
            const float2 hf = __bfloat1622float2(h);
            hi[ks][q] = *reinterpret_cast<const uint32_t *>(&h);
            lo[ks][q] = pack_bf16(c[0] - hf.x, c[1] - hf.y);
        }
    }
}

// One block = 4 warps = 64 rows. Forward with stored activations, loss
// gradient, backward deltas; writes deltaT / actT of every layer and adds the
// batch loss. weight_sum: sum of the batch's sample weights (device scalar).
__global__ void __launch_bounds__(128) k_guide_train_fb(const __nv_bfloat16 *wb, const float *params, GuideParams gp,
                                                        const float *pos, const float *dir, const float *sdir,
                                                        const float *weight, uint32_t n, const float *weight_sum,
                                                        TrainBuffers tb, float *loss)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SmemWeights &s = *reinterpret_cast<SmemWeights *>(smem);
    SmemWeightsT &t = *reinterpret_cast<SmemWeightsT *>(smem + sizeof(SmemWeights));
    float *ybuf = reinterpret_cast<float *>(smem + sizeof(SmemWeights) + sizeof(SmemWeightsT));  // [4 warps][16][48]
    load_weights(s, wb, params);
    load_weights_t(t, wb);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    float *yw = ybuf + warp * 16 * kOut;
    const uint32_t r0 = 64 * blockIdx.x + 16 * warp;
    if (r0 >= n) return;  // no block-wide barrier follows
    float pg[3], dg[3], ph[3], dh[3];
    uint32_t sg, sh;
    load_row(pos, dir, nullptr, n, r0 + g, gp, pg, dg, sg);
    load_row(pos, dir, nullptr, n, r0 + g + 8, gp, ph, dh, sh);
    uint32_t a0[5][4], h[4][4][4];  // inputs; outputs of layers 0..3 (post-ReLU)
    input_frags(pg, dg, ph, dh, a0);
    float acc[8][4];
    init_bias(acc, s.bias);
    layer_mma<8, 5>(acc, a0, s.w0, kStrideIn);
    relu_to_a(acc, h[0]);
#pragma unroll
    for (int l = 1; l <= 3; ++l) {
        init_bias(acc, s.bias + l * kHid);
        layer_mma<8, 4>(acc, h[l - 1], s.w[l - 1], kStrideHid);
        relu_to_a(acc, h[l]);
    }
    float out[6][4];
    init_bias(out, s.bias + 4 * kHid);
    layer_mma<6, 4>(out, h[3], s.w4, kStrideHid);
    // layer inputs, transposed
    store_a_t<5>(tb.actT[0], tb.rows, r0, a0, n);
#pragma unroll
    for (int l = 1; l < kLayers; ++l) store_a_t<4>(tb.actT[l], tb.rows, r0, h[l - 1], n);
    // loss gradient, one row per lane
#pragma unroll
    for (int nt = 0; nt < 6; ++nt) {
        const int c = 8 * nt + 2 * tig;
        yw[g * kOut + c] = out[nt][0];
        yw[g * kOut + c + 1] = out[nt][1];
        yw[(g + 8) * kOut + c] = out[nt][2];
        yw[(g + 8) * kOut + c + 1] = out[nt][3];
    }
    __syncwarp();
    float dyrow[kGuideOut];
    if (lane < 16) {
        const uint32_t r = r0 + lane;
        float lq = 0.0f;
        if (r < n) {
            const float wm = *weight_sum / (float)n;
            const float c = wm > 0.0f ? weight[r] / wm : 0.0f;
            lq = guide_loss_grad(yw + lane * kOut, sdir[3 * (size_t)r], sdir[3 * (size_t)r + 1], sdir[3 * (size_t)r + 2],
                                 c / (float)n, dyrow);
            atomicAdd(loss, -c * lq / (float)n);
        } else {
            for (int i = 0; i < kGuideOut; ++i) dyrow[i] = 0.0f;
        }
    }
    __syncwarp();
    if (lane < 16) {
        for (int i = 0; i < kGuideOut; ++i) yw[lane * kOut + i] = dyrow[i];
        for (int i = kGuideOut; i < kOut; ++i) yw[lane * kOut + i] = 0.0f;
    }
    __syncwarp();
    float dy[6][4];
#pragma unroll
    for (int nt = 0; nt < 6; ++nt) {
        const int c = 8 * nt + 2 * tig;
        dy[nt][0] = yw[g * kOut + c];
        dy[nt][1] = yw[g * kOut + c + 1];
        dy[nt][2] = yw[(g + 8) * kOut + c];
        dy[nt][3] = yw[(g + 8) * kOut + c + 1];
    }
    store_t<6>(tb.deltaT[4], tb.rows, r0, dy, n, kOut);
    // delta of h4 = (dy W4) * relu'(h4): A = dy (K = 48), B[k][n] = W4[k][n] = W4T[n][k]
    uint32_t dhi3[3][4], dlo3[3][4];
    {
        uint32_t dummy[4][4] = {};
        delta_frags<3, false>(dy, dummy, dhi3, dlo3);
    }
    float dacc[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) dacc[nt][0] = dacc[nt][1] = dacc[nt][2] = dacc[nt][3] = 0.0f;
    layer_mma<8, 3>(dacc, dhi3, t.t4, kStrideOutT);
    layer_mma<8, 3>(dacc, dlo3, t.t4, kStrideOutT);
    uint32_t dhi[4][4], dlo[4][4];
#pragma unroll
    for (int l = 3; l >= 1; --l) {
        delta_frags<4, true>(dacc, h[l], dhi, dlo);  // masks dacc in place by relu'(h_l)
        store_t<8>(tb.deltaT[l], tb.rows, r0, dacc, n, kHid);
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) dacc[nt][0] = dacc[nt][1] = dacc[nt][2] = dacc[nt][3] = 0.0f;
        layer_mma<8, 4>(dacc, dhi, t.t[l - 1], kStrideHid);
        layer_mma<8, 4>(dacc, dlo, t.t[l - 1], kStrideHid);
    }
    delta_frags<4, true>(dacc, h[0], dhi, dlo);
    store_t<8>(tb.deltaT[0], tb.rows, r0, dacc, n, kHid);
}

// ---- training on the 5th-generation tensor cores (tcgen05) ----------------------
//
// One CTA of 512 workers per SM carries 128-row tiles through the forward pass,
// the loss gradient, the backward deltas and the weight gradients, with the
// same arithmetic as k_guide_train_fb + k_guide_wgrad (BF16 operands, FP32
// sums; deltas enter the tensor cores as a BF16 high part plus a BF16
// remainder). Four threads share a row: warp w reads the tensor-memory lanes of
// rows 32 (w & 3) .., and w >> 2 picks a quarter of the columns (or two of the
// eight lobes), so the serial work between two matrix products is a quarter of
// a row's. Forward layer l: D[128 x out] = x_l W_l^T as in k_guide_infer_tc.
// Backward layer l: D[128 x in] = delta_hi W_l + delta_lo W_l, the forward
// weights read through an MN-major descriptor. Every layer input x_l stays in
// shared memory for the whole tile, and a delta tile holds [delta_hi |
// delta_lo] as one 128 x 128 matrix. Both serve twice, through two descriptors of
// the same bytes: K-major (the forward product over inputs, the backward
// product over outputs) and MN-major (the weight-gradient product over rows):
// dW_l[128 x (in + 16)] += [delta_hi | delta_lo]^T x_l, whose rows 0-63 and
// 64-127 are the high and low parts of dW_l. The 16 extra columns of x_l hold
// 1.0, so column `in` of the product is the bias gradient. Two delta tiles
// alternate between layers, so the weight gradient of a layer runs while the
// next delta is formed. The per-layer sums stay in tensor memory across the
// CTA's tiles; each CTA writes its sums to a row of `parts`, and k_guide_adam
// adds the rows in order, so a step has the same bits every time.
//
// Bound by the serial chain of a tile, 16,500 cycles: five forward steps of 950
// cycles (operands ready, four products, epilogue), the loss gradient 4,700
// (issue slots), four backward steps of 1,450 (eight products behind the eight
// of the last weight gradient), the last weight gradient. Shared memory holds
// one tile, so nothing else can run meanwhile but the encoding of the next
// tile's rows, which is spread over the waits. The products are issued by a
// warp of their own, which alone waits for all workers. An Adam step of 65,536
// rows takes 51 us (58 us with the products issued by a worker and the encoding
// between the tiles, 64 us without the programmatic launches of its three
// kernels); with one thread per row, 128 threads per CTA and atomic adds of the
// sums it took 153 us (20 us of it the atomics).

// Shared memory of k_guide_train_fused (byte offsets).
constexpr int kTfThreads = 512;  // workers; one more warp issues the products
constexpr uint32_t kTfX0 = 0;                                  // x_0: 128 x (80 + 16)
constexpr uint32_t kTfX1 = kTfX0 + 12 * 2048;                  // x_1..x_4: 128 x (64 + 16) each
constexpr uint32_t kTfD = kTfX1 + 4 * 10 * 2048;               // two tiles [delta_hi | delta_lo]: 128 x 128
constexpr uint32_t kTfW = kTfD + 2 * 16 * 2048;                // forward weights, as kTcW0..kTcW4
constexpr uint32_t kTfBias = kTfW + kImgBytes;
constexpr uint32_t kTfLse = kTfBias + (4 * kHid + kOut) * 4;   // [part][row] log densities of two lobes
constexpr uint32_t kTfBar = kTfLse + 4 * kTcRows * 8;          // MMA mbarrier, TMEM address, copy mbarrier, drain mbarrier
constexpr uint32_t kTfSmem = kTfBar + 32;
// tensor-memory columns: [0, 64) the forward / backward product, then dW_l
__host__ __device__ constexpr uint32_t tf_dcol(int l) { return l == 0 ? 64u : 160u + 80u * (uint32_t)(l - 1); }
// 16-column chunks of the dW_l (weights and the bias column), in order of their columns
constexpr int kTfChunks = 6 + 4 * 5;
static_assert(tf_dcol(1) == 64 + 16 * 6 && tf_dcol(4) + 80 == 64 + 16 * kTfChunks, "chunk f begins at column 64 + 16 f");
static_assert(2 * kTfChunks * 64 * 64 <= (int)kTfBias, "the staged sums fit the tiles and the weights");
// floats of one CTA's row of partial sums: the gradients, the loss
constexpr int kPartStride = (kNumParams + 1 + 31) & ~31;
constexpr int kWeightParts = 64;  // blocks of k_guide_weight_sum

__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u));
}

// Splits a pair into its BF16 high part and the BF16 rounding of the rest.
__device__ __forceinline__ void split_bf16(float c0, float c1, uint32_t &hi, uint32_t &lo)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(c0, c1);
    const float2 hf = __bfloat1622float2(h);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = pack_bf16(c0 - hf.x, c1 - hf.y);
}

// Named barriers of k_guide_train_fused (0 is __syncthreads).
constexpr int kTfRowBar = 1;    // + row group: the four threads of each of 32 rows
constexpr int kTfReadyBar = 5;  // + step & 1: the operands of the step's products are in shared memory
constexpr int kTfWorkBar = 7;   // all workers
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads)
{
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

__global__ void __launch_bounds__(kTfThreads + 32, 1)
k_guide_train_fused(const unsigned char *img, const float *params, GuideParams gp, const float *pos, const float *dir,
                    const float *sdir, const float *weight, uint32_t n, const float *weight_parts, uint32_t nweight,
                    float *parts, uint32_t polls, uint32_t *error)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ float s_loss[4];
    __shared__ int s_failed;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int row = 32 * (warp & 3) + lane, part = warp >> 2;
    const bool worker = warp < kTfThreads / 32;  // the last warp issues the products
    const uint32_t cbar = smem_u32(smem + kTfBar + 16), dbar = cbar + 8;
    float *bias = reinterpret_cast<float *>(smem + kTfBias);
    const uint32_t xoff[kLayers] = {kTfX0, kTfX1, kTfX1 + 20480, kTfX1 + 40960, kTfX1 + 61440};
    // the columns of ones (in .. in + 15) of every x_l
    if (part < 2) {
        const uint32_t one2 = 0x3f803f80u;
#pragma unroll
        for (int l = 0; l < kLayers; ++l)
            *reinterpret_cast<uint4 *>(smem + xoff[l] + canon_off(row, fan_in(l) + 8 * part, kTcRows)) =
                make_uint4(one2, one2, one2, one2);
    }
    const uint32_t mbar = smem_u32(smem + kTfBar);
    const uint32_t tslot = smem_u32(smem + kTfBar + 8);
    if (tid == 0) {
        mbar_init(mbar, 1);
        mbar_init(dbar, 1);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(tslot) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    wait_previous();  // the parameters and the weight sums
    if (tid == 0) s_failed = 0;
    if (tid == 0) fetch_weight_image(smem_u32(smem + kTfW), img, kImgBytes, cbar);
    for (int i = tid; i < 4 * kHid + kOut; i += kTfThreads + 32) bias[i] = params[b_off(i / kHid) + i % kHid];
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t taddr = *reinterpret_cast<volatile uint32_t *>(smem + kTfBar + 8);
    const uint32_t d_base = smem_u32(smem + kTfD), w_img = smem_u32(smem + kTfW), x_base = smem_u32(smem);
    const uint32_t woff[kLayers] = {kTcW0, kTcW1, kTcW1 + 8192, kTcW1 + 16384, kTcW4};
    uint32_t step = 0;  // steps begun: products that the workers wait for

    if (!worker) {
        // The products of every step, by one lane of a warp of their own: in a
        // worker's warp their issue (up to 1,000 cycles a step, as the tensor
        // pipe takes them) would keep that warp's rows waiting.
        const bool leader = elect_one();
        if (!mbar_wait(cbar, 0)) {  // the weights have landed
            *reinterpret_cast<volatile int *>(&s_failed) = 1;
            atomicOr(error, ERR_TIMEOUT);
        }
        auto ready = [&] {
            bar_sync(kTfReadyBar + (int)(step++ & 1u), kTfThreads + 32);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        };
        // dW_l += [delta_hi | delta_lo]^T x_l over the tile's 128 rows (8 MMAs of
        // 16 rows; MN-major operands: 8-row groups 128 B apart, 8-column groups
        // 2048 B apart)
        auto wgrad = [&](int l, bool acc) {
            const uint32_t idesc = idesc_bf16(kTcRows, fan_in(l) + 16) | (1u << 15) | (1u << 16);
            uint64_t a = smem_desc(d_base + (uint32_t)(l & 1) * 32768, 128, 2048), b = smem_desc(x_base + xoff[l], 128, 2048);
#pragma unroll
            for (int s2 = 0; s2 < kTcRows / 16; ++s2, a += 16, b += 16) tc_mma(taddr + tf_dcol(l), a, b, idesc, acc || s2 > 0);
        };
        bool first = true;
        for (uint32_t tile = blockIdx.x; (uint64_t)tile * kTcRows < n; tile += gridDim.x) {
#pragma unroll
            for (int l = 0; l < kLayers; ++l) {  // forward
                ready();
                if (leader) {
                    const uint32_t N = fan_out(l), idesc = idesc_bf16(kTcRows, N);
                    uint64_t a = smem_desc(x_base + xoff[l], kTcRows * 16, 128), b = smem_desc(w_img + woff[l], N * 16, 128);
#pragma unroll
                    for (uint32_t s2 = 0; s2 < fan_in(l) / 16; ++s2, a += kTcRows * 2, b += N * 2) tc_mma(taddr, a, b, idesc, s2 > 0);
                    commit_products(mbar);
                }
                __syncwarp();
            }
            // backward: delta_{l-1} = (delta_l W_l) masked by the ReLU of layer
            // l - 1; dW_l runs behind it
#pragma unroll
            for (int l = kLayers - 1; l >= 1; --l) {
                ready();
                if (leader) {
                    const uint32_t O = fan_out(l), idesc = idesc_bf16(kTcRows, kHid) | (1u << 16);
                    const uint64_t b0 = smem_desc(w_img + woff[l], 128, O * 16);
#pragma unroll
                    for (int half = 0; half < 2; ++half) {  // high parts, then remainders
                        uint64_t a = smem_desc(d_base + (uint32_t)(l & 1) * 32768 + half * 8 * 2048, kTcRows * 16, 128), b = b0;
#pragma unroll
                        for (uint32_t s2 = 0; s2 < O / 16; ++s2, a += kTcRows * 2, b += 16) tc_mma(taddr, a, b, idesc, half + s2 > 0);
                    }
                    commit_products(mbar);
                    wgrad(l, !first);
                }
                __syncwarp();
            }
            ready();
            if (leader) {
                wgrad(0, !first);
                commit_products(mbar);
            }
            __syncwarp();
            first = false;
        }
        allow_next();
    } else {
        const uint32_t lane_addr = taddr + ((uint32_t)(32 * (warp & 3)) << 16);
        float wsum = (uint32_t)lane < nweight ? weight_parts[lane] : 0.0f;
        const float wsum2 = (uint32_t)lane + 32 < nweight ? weight_parts[lane + 32] : 0.0f;
        float loss_sum = 0.0f;  // of the part 0 threads' rows
        bool failed = false;  // warp-uniform
        // this thread's shared-memory stores (and tensor-memory loads) are done
        auto ready = [&] {
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            const int bar = kTfReadyBar + (int)(step++ & 1u);
            if (failed) bar_sync(bar, kTfThreads + 32);
            else bar_arrive(bar, kTfThreads + 32);
        };
        // Waits for the step's commit (which covers every product issued before it).
        // Every wait is bounded; once one gives up the block runs on without waiting
        // (but in step, at the barriers), so that it ends together, and its sums are
        // dropped. A warp that gives up may come to the next step's barrier before
        // the others have come to this one's, so two barriers take turns: on one
        // alone it would arrive twice in a phase and leave a later phase short of an
        // arrival.
        auto finish = [&] {
            bool bad = *reinterpret_cast<volatile int *>(&s_failed) != 0;
            if (!bad && !mbar_wait(mbar, (step - 1u) & 1u, polls)) {
                *reinterpret_cast<volatile int *>(&s_failed) = 1;
                atomicOr(error, ERR_TIMEOUT);
                bad = true;
            }
            failed = __any_sync(0xffffffffu, bad);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        };
        // Pair k of the encoded columns of chunk part + 4 j (8 columns) of a row.
        // A tile's rows are loaded a tile ahead and encoded while the products of
        // the tile before run (3,700 cycles a tile otherwise).
        float p[3] = {}, d[3] = {};
        uint32_t in[3][4] = {};
        auto encode = [&](int j, int k) {
            const int c = 8 * (part + 4 * j) + 2 * k, axis = c / 24;
            float v0 = 0.0f, v1 = 0.0f;
            if (c < 72) {
                const float x = axis == 0 ? p[0] : axis == 1 ? p[1] : p[2];
                sincospif(x * __int_as_float((127 + ((c % 24) >> 1)) << 23), &v0, &v1);
            } else if (c == 72) {
                v0 = d[0], v1 = d[1];
            } else if (c == 74) {
                v0 = d[2];
            }
            in[j][k] = pack_bf16(v0, v1);
        };
        uint32_t tile = blockIdx.x, slot;
        if ((uint64_t)tile * kTcRows < n) {
            load_row(pos, dir, nullptr, n, tile * kTcRows + row, gp, p, d, slot);
#pragma unroll
            for (int i = 0; i < 12; ++i) encode(i / 4, i % 4);
        }
        // mean sample weight: the same sum in every thread of every block
        wsum += wsum2;
        for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
        const float wmean = wsum / (float)n;
        for (; (uint64_t)tile * kTcRows < n; tile += gridDim.x) {
            const uint32_t r = tile * kTcRows + row;
            const bool live = r < n;
#pragma unroll
            for (int j = 0; j < 3; ++j)
                if (part + 4 * j < kIn / 8)
                    *reinterpret_cast<uint4 *>(smem + kTfX0 + canon_off(row, 8 * (part + 4 * j), kTcRows)) =
                        make_uint4(in[j][0], in[j][1], in[j][2], in[j][3]);
            const uint64_t ahead = ((uint64_t)tile + gridDim.x) * kTcRows + row;
#pragma unroll
            for (int l = 0; l < kLayers - 1; ++l) {
                ready();
                if (l == 0) load_row(pos, dir, nullptr, n, (uint32_t)min((uint64_t)n, ahead), gp, p, d, slot);
                else encode(0, l - 1);
                finish();
                float v[16];
                tmem_ld16(lane_addr + 16 * part, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                const float4 *b = reinterpret_cast<const float4 *>(bias + l * kHid + 16 * part);
                uint32_t q[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 c = b[i];
                    const float2 x = __fadd2_rn(make_float2(v[4 * i], v[4 * i + 1]), make_float2(c.x, c.y));
                    const float2 z = __fadd2_rn(make_float2(v[4 * i + 2], v[4 * i + 3]), make_float2(c.z, c.w));
                    q[2 * i] = relu_bf16(x.x, x.y);
                    q[2 * i + 1] = relu_bf16(z.x, z.y);
                }
                *reinterpret_cast<uint4 *>(smem + xoff[l + 1] + canon_off(row, 16 * part, kTcRows)) = make_uint4(q[0], q[1], q[2], q[3]);
                *reinterpret_cast<uint4 *>(smem + xoff[l + 1] + canon_off(row, 16 * part + 8, kTcRows)) =
                    make_uint4(q[4], q[5], q[6], q[7]);
            }
            ready();
            const float c = live && wmean > 0.0f ? weight[r] / wmean : 0.0f;
            float wx = 0.0f, wy = 0.0f, wz = 1.0f;
            if (live) wx = sdir[3 * (size_t)r], wy = sdir[3 * (size_t)r + 1], wz = sdir[3 * (size_t)r + 2];
            finish();
            {
                // loss and its gradient: lobes 2 part and 2 part + 1 of the row
                float v[16], y[10], z[kGuideLobes];
                tmem_ld16(lane_addr + 10 * part, v);
#pragma unroll
                for (int j = 0; j < kGuideLobes; ++j) z[j] = tmem_ld1(lane_addr + 5 * j);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int i = 0; i < 10; ++i) y[i] = v[i] + bias[4 * kHid + 10 * part + i];
                // mixture weights: every thread of a row takes the sum over all lobes
                float mx = z[0] = z[0] + bias[4 * kHid];
#pragma unroll
                for (int j = 1; j < kGuideLobes; ++j) mx = fmaxf(mx, z[j] = z[j] + bias[4 * kHid + 5 * j]);
                float s = 0.0f;
#pragma unroll
                for (int j = 0; j < kGuideLobes; ++j) s += guide_exp(z[j] - mx);
                const float inv = 1.0f / s, pi[2] = {guide_exp(y[0] - mx) * inv, guide_exp(y[5] - mx) * inv};
                GuideLobeTerm t[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) t[j] = guide_lobe_term(y + 5 * j, pi[j], wx, wy, wz);
                float2 *lse = reinterpret_cast<float2 *>(smem + kTfLse);
                lse[part * kTcRows + row] = make_float2(t[0].t, t[1].t);
                bar_sync(kTfRowBar + (warp & 3), 128);
                float2 e[4];
                mx = -3.0e38f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    e[k] = lse[k * kTcRows + row];
                    mx = fmaxf(mx, fmaxf(e[k].x, e[k].y));
                }
                s = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s += guide_exp(e[k].x - mx);
                    s += guide_exp(e[k].y - mx);
                }
                const float logq = mx + logf(s), scale = c / (float)n;
                if (part == 0 && live) loss_sum += -c * logq / (float)n;
                float dy[10];
#pragma unroll
                for (int j = 0; j < 2; ++j) guide_lobe_grad(y + 5 * j, t[j], pi[j], logq, wx, wy, wz, scale, dy + 5 * j);
#pragma unroll
                for (int i = 0; i < 5; ++i) {
                    uint32_t hi, lo;
                    split_bf16(live ? dy[2 * i] : 0.0f, live ? dy[2 * i + 1] : 0.0f, hi, lo);
                    *reinterpret_cast<uint32_t *>(smem + kTfD + canon_off(row, 10 * part + 2 * i, kTcRows)) = hi;
                    *reinterpret_cast<uint32_t *>(smem + kTfD + canon_off(row, 64 + 10 * part + 2 * i, kTcRows)) = lo;
                }
                if (part < 3) {  // unused outputs
                    *reinterpret_cast<uint4 *>(smem + kTfD + canon_off(row, kGuideOut + 8 * part, kTcRows)) = make_uint4(0, 0, 0, 0);
                    *reinterpret_cast<uint4 *>(smem + kTfD + canon_off(row, 64 + kGuideOut + 8 * part, kTcRows)) =
                        make_uint4(0, 0, 0, 0);
                }
            }
#pragma unroll
            for (int l = kLayers - 1; l >= 1; --l) {
                ready();
                if (l == kLayers - 1) encode(0, 3);
                else encode(1, kLayers - 2 - l);
                finish();
                float v[16];
                tmem_ld16(lane_addr + 16 * part, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                // the ReLU of layer l - 1 passes where its output x_l is not zero
                unsigned char *D = smem + kTfD + ((l - 1) & 1) * 32768;
                const __nv_bfloat162 zero2 = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint4 x = *reinterpret_cast<const uint4 *>(smem + xoff[l] + canon_off(row, 16 * part + 8 * j, kTcRows));
                    const uint32_t q[4] = {x.x, x.y, x.z, x.w};
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int i = 8 * j + 2 * k;
                        const uint32_t pass = __hneu2_mask(*reinterpret_cast<const __nv_bfloat162 *>(&q[k]), zero2);
                        split_bf16(v[i], v[i + 1], hi[k], lo[k]);
                        hi[k] &= pass, lo[k] &= pass;
                    }
                    *reinterpret_cast<uint4 *>(D + canon_off(row, 16 * part + 8 * j, kTcRows)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4 *>(D + canon_off(row, 64 + 16 * part + 8 * j, kTcRows)) =
                        make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
            }
            ready();
            encode(1, 3);
#pragma unroll
            for (int k = 0; k < 4; ++k) encode(2, k);
            finish();  // the last weight gradient reads x_0 and a delta tile
        }
        allow_next();
        bar_sync(kTfWorkBar, kTfThreads);
        float *out = parts + (size_t)blockIdx.x * kPartStride;
        if (!*reinterpret_cast<volatile int *>(&s_failed)) {
            // The CTA's sums: rows m < 64 of dW_l carry the high part of output m, rows
            // 64 + m the low part. Both go to shared memory as [half][chunk][output][16]
            // (chunk f: tensor-memory columns 64 + 16 f ..; layers 1 to 4 have 5 each)
            // and leave, added, as whole rows. The 16-byte pieces are turned so that
            // neither side has bank conflicts.
            const int half = row >> 6, o = row & 63;
            auto piece = [&](int h, int f, int m, int q) {
                return reinterpret_cast<float4 *>(smem + ((h * kTfChunks + f) * 64 + (m ^ (f & 1))) * 64 + 16 * (q ^ ((m >> 1) & 3)));
            };
#pragma unroll 1
            for (int f0 = part; f0 < kTfChunks; f0 += 8) {  // two at a time
                float v[2][16];
                tmem_ld16(lane_addr + 64 + 16 * f0, v[0]);
                if (f0 + 4 < kTfChunks) tmem_ld16(lane_addr + 64 + 16 * (f0 + 4), v[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (f0 + 4 * k < kTfChunks)
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            *piece(half, f0 + 4 * k, o, i) = make_float4(v[k][4 * i], v[k][4 * i + 1], v[k][4 * i + 2], v[k][4 * i + 3]);
            }
            bar_sync(kTfWorkBar, kTfThreads);
            auto sum = [&](int f, int m, int q) {
                const float4 hi = *piece(0, f, m, q), lo = *piece(1, f, m, q);
                return make_float4(hi.x + lo.x, hi.y + lo.y, hi.z + lo.z, hi.w + lo.w);
            };
#pragma unroll
            for (int l = 0; l < kLayers; ++l) {
                const int rowv = fan_in(l) / 4, f = ((int)tf_dcol(l) - 64) / 16;
                for (int i = tid; i < fan_out(l) * rowv; i += kTfThreads) {
                    const int m = i / rowv, q = i % rowv;
                    reinterpret_cast<float4 *>(out + w_off(l))[i] = sum(f + q / 4, m, q % 4);
                }
                if (tid < fan_out(l)) out[b_off(l) + tid] = sum(f + fan_in(l) / 16, tid, 0).x;
            }
            for (int k = 16; k > 0; k >>= 1) loss_sum += __shfl_down_sync(0xffffffffu, loss_sum, k);
            if (part == 0 && lane == 0) s_loss[warp] = loss_sum;
            bar_sync(kTfWorkBar, kTfThreads);
            if (tid == 0) out[kNumParams] = (s_loss[0] + s_loss[1]) + (s_loss[2] + s_loss[3]);
        } else {  // the sums of this CTA count as nothing
            for (int i = tid; i < kPartStride; i += kTfThreads) out[i] = 0.0f;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    // After a wait gave up, products or the weight copy may still be in flight,
    // several commits deep: the issuing lane commits them all to a barrier of its
    // own, and its warp waits (bounded) before their memory is freed.
    if (*reinterpret_cast<volatile int *>(&s_failed)) {
        if (!worker) {
            if (elect_one()) commit_products(dbar);
            mbar_wait(dbar, 0);
            mbar_wait(cbar, 0);
        }
        __syncthreads();
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(taddr) : "memory");
}

// Weight gradients of all layers in one launch (layer l = block z):
// dW[o][i] += sum over rows of deltaT[o][r] actT[i][r] (tensor cores, K = rows;
// delta as BF16 high + low parts), bias gradient db[o] += sum deltaT[o][r].
// Each warp computes one 16 x 8 tile (16 outputs, 8 inputs) over a chunk of
// kWgradRows rows and adds it with atomics; block x = (output tile, group of
// 4 input tiles), block y = row chunk. Measured per training step of 16,384
// rows: five launches of 256-row chunks 0.15 ms.
constexpr uint32_t kWgradRows = 512;

__host__ __device__ constexpr int wgrad_blocks_x(int l)
{
    return (l == kLayers - 1 ? kOut : kHid) / 16 * (((l == 0 ? kIn : kHid) / 8 + 3) / 4);
}

__global__ void __launch_bounds__(128) k_guide_wgrad(TrainBuffers tb, uint32_t n, float *grad)
{
    const int l = (int)blockIdx.z;
    if ((int)blockIdx.x >= wgrad_blocks_x(l)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int fan_in_l = l == 0 ? kIn : kHid;
    const int in_tiles = fan_in_l / 8, groups = (in_tiles + 3) / 4;
    const int o0 = 16 * (blockIdx.x / groups);
    const int it = 4 * (blockIdx.x % groups) + warp;
    const uint32_t k0 = kWgradRows * blockIdx.y, k1 = min(n, k0 + kWgradRows);
    const float *dT = tb.deltaT[l];
    const __nv_bfloat16 *aT = tb.actT[l];
    const uint32_t stride = tb.rows;
    if (it < in_tiles) {
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const __nv_bfloat16 *col = aT + (size_t)(8 * it + g) * stride;
        for (uint32_t k = k0; k < k1; k += 16) {
            // A[m = o][k = row]: a0 (o0+g, k+2tig..+1), a1 (o0+g+8, ...), a2 (o0+g, k+8+2tig..), a3 (o0+g+8, k+8+..)
            uint32_t ahi[4], alo[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int o = o0 + g + ((q & 1) ? 8 : 0);
                const uint32_t kk = k + 2 * tig + ((q & 2) ? 8 : 0);
                const float v0 = kk < k1 ? dT[(size_t)o * stride + kk] : 0.0f;
                const float v1 = kk + 1 < k1 ? dT[(size_t)o * stride + kk + 1] : 0.0f;
                const __nv_bfloat162 hb = __floats2bfloat162_rn(v0, v1);
                const float2 hf = __bfloat1622float2(hb);
                ahi[q] = *reinterpret_cast<const uint32_t *>(&hb);
                alo[q] = pack_bf16(v0 - hf.x, v1 - hf.y);
            }
            // B[k = row][n = input]: b0 (rows k+2tig..+1, input 8it+g), b1 (rows k+8+2tig..)
            const uint32_t kk = k + 2 * tig;
            uint32_t b0 = 0, b1 = 0;
            if (kk + 1 < k1) b0 = ld_pair(col + kk);
            else if (kk < k1) b0 = (uint32_t) * reinterpret_cast<const uint16_t *>(col + kk);
            if (kk + 9 < k1) b1 = ld_pair(col + kk + 8);
            else if (kk + 8 < k1) b1 = (uint32_t) * reinterpret_cast<const uint16_t *>(col + kk + 8);
            mma_bf16(acc, ahi, b0, b1);
            mma_bf16(acc, alo, b0, b1);
        }
        float *G = grad + w_off(l);
        const int i = 8 * it + 2 * tig;
        atomicAdd(&G[(o0 + g) * fan_in_l + i], acc[0]);
        atomicAdd(&G[(o0 + g) * fan_in_l + i + 1], acc[1]);
        atomicAdd(&G[(o0 + g + 8) * fan_in_l + i], acc[2]);
        atomicAdd(&G[(o0 + g + 8) * fan_in_l + i + 1], acc[3]);
    }
    // bias gradient: in the first input-tile group, warp 0's lanes 0..15 sum the
    // chunk's rows of outputs o0 + lane
    if (blockIdx.x % groups == 0 && warp == 0 && lane < 16) {
        float sum = 0.0f;
        const float *row = dT + (size_t)(o0 + lane) * stride;
        for (uint32_t k = k0; k < k1; ++k) sum += row[k];
        atomicAdd(grad + b_off(l) + o0 + lane, sum);
    }
}

// Sums of the sample weights, one per block (gridDim.x <= kWeightParts).
__global__ void __launch_bounds__(256) k_guide_weight_sum(const float *w, uint32_t n, float *sums)
{
    __shared__ float s[8];
    float v = 0.0f;
    wait_previous();  // the sums' last reader, and whatever wrote the weights
    allow_next();
    const uint32_t stride = gridDim.x * blockDim.x;
    uint64_t i = blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * stride < n; i += 4 * stride) {  // four loads in flight, added in order
        const float a = w[i], b = w[i + stride], c = w[i + 2 * stride], d = w[i + 3 * stride];
        v += a, v += b, v += c, v += d;
    }
    for (; i < n; i += stride) v += w[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 8) {
        v = s[threadIdx.x];
        for (int o = 4; o > 0; o >>= 1) v += __shfl_down_sync(0xffu, v, o);
        if (threadIdx.x == 0) sums[blockIdx.x] = v;
    }
}

// The blocks' weight sums as one (mma.sync path).
__global__ void k_guide_add_sums(const float *sums, uint32_t count, float *sum)
{
    const int lane = threadIdx.x;
    float v = (uint32_t)lane < count ? sums[lane] : 0.0f;
    if ((uint32_t)lane + 32 < count) v += sums[lane + 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) *sum = v;
}

// Adds the nparts rows of partial sums (in a fixed order: kAdamSplits
// interleaved sums, then those) into grad and the loss and, with `adam`, takes
// the Adam step. 64 entries per block, four per thread and load, so that a
// block's loads are all in flight at once.
constexpr int kAdamSplits = 32;
struct AdamArgs {
    float *params, *m, *v;
    __nv_bfloat16 *wb;
    unsigned char *img;
    int t;
    float lr, b1, b2, eps;
};
__global__ void __launch_bounds__(16 * kAdamSplits) k_guide_adam(const float *parts, int nparts, float *grad, float *loss, bool adam, AdamArgs a)
{
    __shared__ float4 s[kAdamSplits][16];
    const int quad = threadIdx.x & 15, split = threadIdx.x >> 4;
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    wait_previous();
    allow_next();
    if (blockIdx.x * 64 + 4 * quad < kPartStride) {
        const float4 *p = reinterpret_cast<const float4 *>(parts) + blockIdx.x * 16 + quad;
#pragma unroll 8
        for (int q = split; q < nparts; q += kAdamSplits) {
            const float4 x = p[(size_t)q * (kPartStride / 4)];
            sum.x += x.x, sum.y += x.y, sum.z += x.z, sum.w += x.w;
        }
    }
    s[split][quad] = sum;
    __syncthreads();
    const int i = blockIdx.x * 64 + (int)threadIdx.x;
    if (threadIdx.x >= 64 || i > kNumParams) return;
    float g = 0.0f;
#pragma unroll
    for (int q = 0; q < kAdamSplits; ++q) g += reinterpret_cast<const float *>(s[q])[threadIdx.x];
    if (i == kNumParams) {
        if (loss) *loss = g;
        return;
    }
    if (grad) grad[i] = g;
    if (!adam) return;
    const float mi = a.b1 * a.m[i] + (1.0f - a.b1) * g;
    const float vi = a.b2 * a.v[i] + (1.0f - a.b2) * g * g;
    a.m[i] = mi;
    a.v[i] = vi;
    const float c1 = 1.0f - powf(a.b1, (float)a.t), c2 = 1.0f - powf(a.b2, (float)a.t);
    const float p = a.params[i] - a.lr * (mi / c1) / (sqrtf(vi / c2) + a.eps);
    a.params[i] = p;
    // BF16 weight copy and weight image (biases stay FP32)
    for (int l = 0; l < kLayers; ++l)
        if (i >= w_off(l) && i < b_off(l)) store_weight(a.wb, a.img, l, i - w_off(l), p);
}

// The BF16 copies of the parameters; clears the Adam moments unless m is NULL.
__global__ void k_guide_export(const float *params, __nv_bfloat16 *wb, unsigned char *img, float *m, float *v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kNumParams) return;
    if (m) m[i] = v[i] = 0.0f;
    for (int l = 0; l < kLayers; ++l)
        if (i >= w_off(l) && i < b_off(l)) store_weight(wb, img, l, i - w_off(l), params[i]);
}

// The network input of each row (80 columns), as the forward pass forms it
// before rounding to BF16.
__global__ void k_guide_encode(GuideParams gp, const float *pos, const float *dir, uint32_t n, float *out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * 40u) return;
    const uint32_t r = i / 40, c = 2 * (i % 40);
    float p[3], d[3];
    uint32_t slot;
    load_row(pos, dir, nullptr, n, r, gp, p, d, slot);
    float v0, v1;
    encode_pair(p, d, (int)c, v0, v1);
    out[(size_t)r * kIn + c] = v0;
    out[(size_t)r * kIn + c + 1] = v1;
}

__global__ void k_guide_sample(const float *y, const float *u, uint32_t n, float *dir, float *pdf)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GuideLobes L = guide_decode(y + (size_t)i * kGuideOut);
    float wx, wy, wz;
    guide_sample(L, u[3 * (size_t)i], u[3 * (size_t)i + 1], u[3 * (size_t)i + 2], wx, wy, wz);
    dir[3 * (size_t)i] = wx, dir[3 * (size_t)i + 1] = wy, dir[3 * (size_t)i + 2] = wz;
    pdf[i] = guide_pdf(L, wx, wy, wz);
}

__global__ void k_guide_pdf(const float *y, const float *dir, uint32_t n, uint32_t y_stride, float *pdf)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const GuideLobes L = guide_decode(y + (size_t)(y_stride ? i : 0) * kGuideOut);
    pdf[i] = guide_pdf(L, dir[3 * (size_t)i], dir[3 * (size_t)i + 1], dir[3 * (size_t)i + 2]);
}

constexpr size_t kScalarBytes = (4 + kWeightParts) * sizeof(float);
constexpr size_t kInferSmem = sizeof(SmemWeights);
constexpr size_t kTrainSmem = sizeof(SmemWeights) + sizeof(SmemWeightsT) + 4 * 16 * kOut * sizeof(float);

}  // namespace
}  // namespace dr

struct dr_guide {
    dr_context *ctx = nullptr;
    dr_guide_config cfg{};
    unsigned char *mem = nullptr;  // one allocation; the pointers below point into it
    float *params = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr;
    __nv_bfloat16 *wb = nullptr;
    unsigned char *img = nullptr;  // weight image of the tcgen05 kernels (kImgBytes)
    float *scalars = nullptr;  // [0] sum of the batch's sample weights (mma.sync path), [1] loss, [4..] weight sums per block
    float *parts = nullptr;    // partial gradients and loss, one row per CTA of the training kernel
    int part_rows = 0;
    void *parts_mem = nullptr; // the rows of a batch of several tiles (ensure_parts)
    dr::TrainBuffers tb{};
    void *tb_mem = nullptr;
    uint32_t capacity = 0;
    int step = 0;
};

using namespace dr;

namespace {

GuideParams guide_params(const dr_guide *g)
{
    GuideParams p{};
    for (int a = 0; a < 3; ++a) p.center[a] = g->cfg.center[a];
    p.half = g->cfg.half_extent > 0.0f ? g->cfg.half_extent : 1.0f;
    return p;
}

void free_guide(dr_guide *g)
{
    if (!g) return;
    cudaFree(g->mem);
    cudaFree(g->parts_mem);
    cudaFree(g->tb_mem);
    delete g;
}

dr_status ensure_train_capacity(dr_guide *g, uint32_t n)
{
    if (n <= g->capacity) return DR_OK;
    DR_CUDA(cudaDeviceSynchronize());
    cudaFree(g->tb_mem);
    g->tb_mem = nullptr;
    g->capacity = 0;
    const uint32_t rows = (n + 63) & ~63u;
    size_t bytes = 0;
    for (int l = 0; l < kLayers; ++l) bytes += (size_t)fan_out(l) * rows * 4 + (size_t)fan_in(l) * rows * 2 + 512;
    DR_CUDA(dev_malloc(&g->tb_mem, bytes));
    char *p = static_cast<char *>(g->tb_mem);
    for (int l = 0; l < kLayers; ++l) {
        g->tb.deltaT[l] = reinterpret_cast<float *>(p);
        p += ((size_t)fan_out(l) * rows * 4 + 255) & ~size_t(255);
        g->tb.actT[l] = reinterpret_cast<__nv_bfloat16 *>(p);
        p += ((size_t)fan_in(l) * rows * 2 + 255) & ~size_t(255);
    }
    g->tb.rows = rows;
    g->capacity = rows;
    return DR_OK;
}

// Rows for the partial sums of `blocks` CTAs: the network comes with one (a
// network that only infers needs none, and mapping 12.6 MB takes 0.1 ms), the
// first batch of several tiles allocates one per SM. That call may be under
// stream capture, where an allocation, which is no stream operation, needs the
// relaxed mode.
dr_status ensure_parts(dr_guide *g, int blocks)
{
    if (blocks <= g->part_rows) return DR_OK;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    DR_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    const cudaError_t e = dev_malloc(&g->parts_mem, (size_t)g->ctx->num_sms * kPartStride * sizeof(float));
    DR_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    DR_CUDA(e);
    g->parts = static_cast<float *>(g->parts_mem);
    g->part_rows = g->ctx->num_sms;
    return DR_OK;
}

// Loss and gradients of one batch, as *nparts rows of partial sums at *parts.
dr_status run_gradients(dr_guide *g, const float *pos, const float *dir, const float *sdir, const float *weight,
                        uint32_t n, cudaStream_t st, const float **parts, int *nparts)
{
    const GuideParams gp = guide_params(g);
    const unsigned sum_blocks = std::min<unsigned>((n + 255) / 256, kWeightParts);
    float *sums = g->scalars + 4;
    // the tcgen05 kernel: one CTA per SM (its shared memory and 512 tensor-memory
    // columns); the per-layer delta and activation buffers serve the mma.sync path
    // only (the tcgen05 kernel keeps them on chip), whose sums meet in one row
    const bool tc = g->cfg.infer_kernel == DR_GUIDE_INFER_TCGEN05;
    const unsigned blocks = std::min<unsigned>((n + kTcRows - 1) / kTcRows, (unsigned)g->ctx->num_sms);
    const dr_status r = tc ? ensure_parts(g, (int)blocks) : ensure_train_capacity(g, n);
    if (r != DR_OK) return r;
    DR_CUDA(launch_after(k_guide_weight_sum, sum_blocks, 256, 0, st, weight, n, sums));
    if (tc) {
        DR_CUDA(launch_after(k_guide_train_fused, blocks, kTfThreads + 32, kTfSmem, st, g->img, g->params, gp, pos, dir, sdir, weight, n,
                             sums, sum_blocks, g->parts, g->ctx->product_polls, g->ctx->d_error));
        *parts = g->parts;
        *nparts = (int)blocks;
    } else {
        DR_CUDA(cudaMemsetAsync(g->parts, 0, kPartStride * sizeof(float), st));
        k_guide_add_sums<<<1, 32, 0, st>>>(sums, sum_blocks, g->scalars);
        k_guide_train_fb<<<(n + 63) / 64, 128, kTrainSmem, st>>>(g->wb, g->params, gp, pos, dir, sdir, weight, n,
                                                                 g->scalars, g->tb, g->parts + kNumParams);
        int bx = 0;
        for (int l = 0; l < kLayers; ++l) bx = std::max(bx, wgrad_blocks_x(l));
        const dim3 grid((unsigned)bx, (n + kWgradRows - 1) / kWgradRows, (unsigned)kLayers);
        k_guide_wgrad<<<grid, 128, 0, st>>>(g->tb, n, g->parts);
        *parts = g->parts;
        *nparts = 1;
    }
    DR_CUDA(cudaGetLastError());
    return DR_OK;
}

constexpr unsigned kAdamBlocks = (kNumParams + 1 + 63) / 64;

}  // namespace

namespace dr {

// Rewrites rows list[0 .. *count) of y (or rows 0 .. n_fixed) in the decoded
// layout, after the mma.sync inference (whose rows are spread over 4 lanes).
__global__ void __launch_bounds__(128) k_guide_decode_rows(const uint32_t *list, const uint32_t *count, uint32_t n_fixed,
                                                           float *y)
{
    const uint32_t n = count ? *count : n_fixed;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float *row = y + (size_t)(list ? list[i] : i) * kGuideOut;
        guide_store_decoded(row, guide_mix(row));
    }
}

cudaError_t launch_guide_infer(const dr_guide *g, const float *pos, const float *dir, const uint32_t *list,
                               const uint32_t *count, uint32_t max_rows, float *y, cudaStream_t st, bool decoded)
{
    if (max_rows == 0) return cudaSuccess;
    if (g->cfg.infer_kernel == DR_GUIDE_INFER_TCGEN05) {
        const unsigned tiles = (max_rows + kTcRows - 1) / kTcRows;
        const unsigned blocks = std::min<unsigned>(tiles, (unsigned)g->ctx->num_sms);
        const auto kernel = decoded ? k_guide_infer_tc<true> : k_guide_infer_tc<false>;
        // early also beside the waves of other streams, where the renderer's own
        // kernels are not: guided renders of 2 to 32 waves on 2 and 3 streams take
        // the same time either way, and 2 to 3 % less with early training kernels
        const cudaError_t e = launch_after(kernel, blocks, 128 * kInferGroups, kTcSmem, st, g->img, g->params, guide_params(g),
                                           pos, dir, list, count, max_rows, y, g->ctx->product_polls, g->ctx->d_error);
        if (e != cudaSuccess) return e;
    } else {
        const unsigned tiles = (max_rows + 15) / 16;
        const unsigned blocks = std::min<unsigned>((tiles + 3) / 4, (unsigned)g->ctx->num_sms * 4);
        k_guide_infer<<<blocks, 128, kInferSmem, st>>>(g->wb, g->params, guide_params(g), pos, dir, list, count,
                                                       max_rows, y);
        if (decoded)
            k_guide_decode_rows<<<std::min<unsigned>((max_rows + 127) / 128, (unsigned)g->ctx->num_sms * 8), 128, 0,
                                  st>>>(list, count, max_rows, y);
    }
    return cudaGetLastError();
}

uint32_t guide_steps(const dr_guide *g) { return (uint32_t)g->step; }

dr_status guide_train_step(dr_guide *g, const float *pos, const float *dir, const float *sdir, const float *weight,
                           uint32_t n, cudaStream_t st)
{
    return dr_guide_train_step(g, pos, dir, sdir, weight, n, st);
}

}  // namespace dr

extern "C" {

uint32_t dr_guide_num_params(void) { return (uint32_t)kNumParams; }

dr_status dr_guide_create(dr_context *ctx, const dr_guide_config *cfg, dr_guide **out)
{
    DR_CHECK_ARG(ctx && out, "dr_guide_create: NULL argument");
    *out = nullptr;
    DR_CUDA(cudaSetDevice(ctx->device));
    static bool attr = false;
    if (!attr) {
        DR_CUDA(cudaFuncSetAttribute(k_guide_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInferSmem));
        DR_CUDA(cudaFuncSetAttribute(k_guide_train_fb, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem));
        DR_CUDA(cudaFuncSetAttribute(k_guide_infer_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
        DR_CUDA(cudaFuncSetAttribute(k_guide_infer_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
        DR_CUDA(cudaFuncSetAttribute(k_guide_train_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTfSmem));
        attr = true;
    }
    auto *g = new (std::nothrow) dr_guide;
    if (!g) return fail(DR_ERR_OUT_OF_MEMORY, "dr_guide_create: host allocation failed");
    g->ctx = ctx;
    if (cfg) g->cfg = *cfg;
    if (g->cfg.learning_rate <= 0.0f) g->cfg.learning_rate = 1e-3f;
    if (g->cfg.beta1 <= 0.0f) g->cfg.beta1 = 0.9f;
    if (g->cfg.beta2 <= 0.0f) g->cfg.beta2 = 0.999f;
    if (g->cfg.epsilon <= 0.0f) g->cfg.epsilon = 1e-8f;
    if (g->cfg.half_extent <= 0.0f) g->cfg.half_extent = 1.0f;
    if (g->cfg.infer_kernel > DR_GUIDE_INFER_MMA_SYNC) {
        free_guide(g);
        return fail(DR_ERR_INVALID_ARGUMENT, "dr_guide_create: unknown inference kernel");
    }
    // one allocation, its parts on 256-byte boundaries
    size_t bytes = 0;
    auto place = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) & ~size_t(255);
        return at;
    };
    const size_t at_params = place(kNumParams * 4), at_m = place(kNumParams * 4), at_v = place(kNumParams * 4),
                 at_grad = place(kNumParams * 4), at_wb = place(kNumWeights * 2), at_img = place(kImgBytes),
                 at_scalars = place(kScalarBytes), at_parts = place(kPartStride * 4);
    cudaError_t e = dev_malloc(&g->mem, bytes);
    if (e == cudaSuccess) e = cudaMemset(g->mem + at_scalars, 0, kScalarBytes);
    if (e != cudaSuccess) {
        free_guide(g);
        return cuda_fail(e, "dr_guide_create");
    }
    g->params = reinterpret_cast<float *>(g->mem + at_params);
    g->m = reinterpret_cast<float *>(g->mem + at_m);
    g->v = reinterpret_cast<float *>(g->mem + at_v);
    g->grad = reinterpret_cast<float *>(g->mem + at_grad);
    g->wb = reinterpret_cast<__nv_bfloat16 *>(g->mem + at_wb);
    g->img = g->mem + at_img;
    g->scalars = reinterpret_cast<float *>(g->mem + at_scalars);
    g->parts = reinterpret_cast<float *>(g->mem + at_parts);
    g->part_rows = 1;
    // He-uniform initialisation (ReLU), last layer scaled by 0.1, zero biases
    std::mt19937_64 rng(g->cfg.seed);
    std::vector<float> p(kNumParams, 0.0f);
    for (int l = 0; l < kLayers; ++l) {
        const float bound = std::sqrt(6.0f / (float)fan_in(l)) * (l == kLayers - 1 ? 0.1f : 1.0f);
        std::uniform_real_distribution<float> U(-bound, bound);
        for (int i = 0; i < fan_out(l) * fan_in(l); ++i) p[w_off(l) + i] = U(rng);
    }
    const dr_status r = dr_guide_set_params(g, p.data(), kNumParams);
    if (r != DR_OK) {
        free_guide(g);
        return r;
    }
    *out = g;
    return DR_OK;
}

dr_status dr_guide_destroy(dr_guide *g)
{
    if (!g) return DR_OK;
    cudaSetDevice(g->ctx->device);
    cudaDeviceSynchronize();
    free_guide(g);
    return DR_OK;
}

dr_status dr_guide_set_params(dr_guide *g, const float *host, uint32_t n)
{
    DR_CHECK_ARG(g && host && n == (uint32_t)kNumParams, "dr_guide_set_params: bad argument");
    DR_CUDA(cudaSetDevice(g->ctx->device));
    DR_CUDA(cudaMemcpy(g->params, host, kNumParams * 4, cudaMemcpyHostToDevice));
    g->step = 0;
    k_guide_export<<<(kNumParams + 255) / 256, 256>>>(g->params, g->wb, g->img, g->m, g->v);
    DR_CUDA(cudaGetLastError());
    DR_CUDA(cudaDeviceSynchronize());
    return DR_OK;
}

// State blob: a header (magic, version, parameter count, Adam step), the
// configuration, then params, m and v (FP32, kNumParams each).
namespace {
constexpr uint32_t kStateMagic = 0x53475244u;  // "DRGS"
constexpr uint32_t kStateVersion = 1;
struct StateHeader {
    uint32_t magic, version, num_params, step;
    dr_guide_config cfg;
};
constexpr uint64_t kStateBytes = sizeof(StateHeader) + 3ull * kNumParams * sizeof(float);
}  // namespace

uint64_t dr_guide_state_bytes(void) { return kStateBytes; }

dr_status dr_guide_get_state(dr_guide *g, void *host, uint64_t bytes)
{
    DR_CHECK_ARG(g && host, "dr_guide_get_state: NULL argument");
    if (bytes != kStateBytes)
        return fail(DR_ERR_INVALID_ARGUMENT, "dr_guide_get_state: the state takes %llu bytes, got %llu",
                    (unsigned long long)kStateBytes, (unsigned long long)bytes);
    DR_CUDA(cudaSetDevice(g->ctx->device));
    DR_CUDA(cudaDeviceSynchronize());
    StateHeader h{kStateMagic, kStateVersion, (uint32_t)kNumParams, (uint32_t)g->step, g->cfg};
    auto *out = static_cast<unsigned char *>(host);
    memcpy(out, &h, sizeof h);
    float *f = reinterpret_cast<float *>(out + sizeof h);
    DR_CUDA(cudaMemcpy(f, g->params, kNumParams * 4, cudaMemcpyDeviceToHost));
    DR_CUDA(cudaMemcpy(f + kNumParams, g->m, kNumParams * 4, cudaMemcpyDeviceToHost));
    DR_CUDA(cudaMemcpy(f + 2 * kNumParams, g->v, kNumParams * 4, cudaMemcpyDeviceToHost));
    return DR_OK;
}

dr_status dr_guide_set_state(dr_guide *g, const void *host, uint64_t bytes)
{
    DR_CHECK_ARG(g && host, "dr_guide_set_state: NULL argument");
    if (bytes != kStateBytes)
        return fail(DR_ERR_INVALID_ARGUMENT, "dr_guide_set_state: the state takes %llu bytes, got %llu",
                    (unsigned long long)kStateBytes, (unsigned long long)bytes);
    StateHeader h;
    memcpy(&h, host, sizeof h);
    DR_CHECK_ARG(h.magic == kStateMagic && h.version == kStateVersion && h.num_params == (uint32_t)kNumParams,
                 "dr_guide_set_state: not a guiding-network state of this version");
    const float *f = reinterpret_cast<const float *>(static_cast<const unsigned char *>(host) + sizeof h);
    DR_CUDA(cudaSetDevice(g->ctx->device));
    DR_CUDA(cudaDeviceSynchronize());
    DR_CUDA(cudaMemcpy(g->params, f, kNumParams * 4, cudaMemcpyHostToDevice));
    DR_CUDA(cudaMemcpy(g->m, f + kNumParams, kNumParams * 4, cudaMemcpyHostToDevice));
    DR_CUDA(cudaMemcpy(g->v, f + 2 * kNumParams, kNumParams * 4, cudaMemcpyHostToDevice));
    g->cfg = h.cfg;
    g->step = (int)h.step;
    k_guide_export<<<(kNumParams + 255) / 256, 256>>>(g->params, g->wb, g->img, nullptr, nullptr);
    DR_CUDA(cudaGetLastError());
    DR_CUDA(cudaDeviceSynchronize());
    return DR_OK;
}

dr_status dr_guide_get_params(dr_guide *g, float *host, uint32_t n)
{
    DR_CHECK_ARG(g && host && n == (uint32_t)kNumParams, "dr_guide_get_params: bad argument");
    DR_CUDA(cudaSetDevice(g->ctx->device));
    DR_CUDA(cudaDeviceSynchronize());
    DR_CUDA(cudaMemcpy(host, g->params, kNumParams * 4, cudaMemcpyDeviceToHost));
    return DR_OK;
}

dr_status dr_guide_infer(dr_guide *g, const float *pos_dev, const float *dir_dev, uint32_t n, float *y_dev, void *stream)
{
    DR_CHECK_ARG(g && (n == 0 || (pos_dev && dir_dev && y_dev)), "dr_guide_infer: NULL argument");
    if (n == 0) return DR_OK;
    DR_CUDA(cudaSetDevice(g->ctx->device));
    DR_CUDA(launch_guide_infer(g, pos_dev, dir_dev, nullptr, nullptr, n, y_dev, static_cast<cudaStream_t>(stream)));
    return DR_OK;
}

dr_status dr_guide_gradients(dr_guide *g, const float *pos_dev, const float *dir_dev, const float *sdir_dev,
                             const float *weight_dev, uint32_t n, float *loss_host, float *grad_host)
{
    DR_CHECK_ARG(g && n > 0 && pos_dev && dir_dev && sdir_dev && weight_dev, "dr_guide_gradients: bad argument");
    DR_CUDA(cudaSetDevice(g->ctx->device));
    const float *parts = nullptr;
    int nparts = 0;
    dr_status r = run_gradients(g, pos_dev, dir_dev, sdir_dev, weight_dev, n, nullptr, &parts, &nparts);
    if (r != DR_OK) return r;
    k_guide_adam<<<kAdamBlocks, 16 * kAdamSplits>>>(parts, nparts, g->grad, g->scalars + 1, false, AdamArgs{});
    DR_CUDA(cudaGetLastError());
    DR_CUDA(cudaDeviceSynchronize());
    if (loss_host) DR_CUDA(cudaMemcpy(loss_host, g->scalars + 1, 4, cudaMemcpyDeviceToHost));
    if (grad_host) DR_CUDA(cudaMemcpy(grad_host, g->grad, kNumParams * 4, cudaMemcpyDeviceToHost));
    return DR_OK;
}

dr_status dr_guide_train_step(dr_guide *g, const float *pos_dev, const float *dir_dev, const float *sdir_dev,
                              const float *weight_dev, uint32_t n, void *stream)
{
    DR_CHECK_ARG(g && pos_dev && dir_dev && sdir_dev && weight_dev, "dr_guide_train_step: NULL argument");
    if (n == 0) return DR_OK;
    DR_CUDA(cudaSetDevice(g->ctx->device));
    auto st = static_cast<cudaStream_t>(stream);
    const float *parts = nullptr;
    int nparts = 0;
    dr_status r = run_gradients(g, pos_dev, dir_dev, sdir_dev, weight_dev, n, st, &parts, &nparts);
    if (r != DR_OK) return r;
    ++g->step;
    const float lr = g->cfg.warmup_steps && (uint32_t)g->step < g->cfg.warmup_steps
                         ? g->cfg.learning_rate * (float)g->step / (float)g->cfg.warmup_steps
                         : g->cfg.learning_rate;
    DR_CUDA(launch_after(k_guide_adam, kAdamBlocks, 16 * kAdamSplits, 0, st, parts, nparts, (float *)nullptr, g->scalars + 1, true,
                         AdamArgs{g->params, g->m, g->v, g->wb, g->img, g->step, lr, g->cfg.beta1, g->cfg.beta2,
                                  g->cfg.epsilon}));
    DR_CUDA(cudaGetLastError());
    return DR_OK;
}

dr_status dr_guide_encode(dr_guide *g, const float *pos_dev, const float *dir_dev, uint32_t n, float *out_dev)
{
    DR_CHECK_ARG(g && (n == 0 || (pos_dev && dir_dev && out_dev)), "dr_guide_encode: NULL argument");
    if (n == 0) return DR_OK;
    DR_CUDA(cudaSetDevice(g->ctx->device));
    k_guide_encode<<<(n * 40 + 255) / 256, 256>>>(guide_params(g), pos_dev, dir_dev, n, out_dev);
    DR_CUDA(cudaGetLastError());
    return DR_OK;
}

dr_status dr_guide_mixture_sample(const float *y_dev, const float *u_dev, uint32_t n, float *dir_dev, float *pdf_dev,
                                  void *stream)
{
    DR_CHECK_ARG(n == 0 || (y_dev && u_dev && dir_dev && pdf_dev), "dr_guide_mixture_sample: NULL argument");
    if (n == 0) return DR_OK;
    k_guide_sample<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(y_dev, u_dev, n, dir_dev, pdf_dev);
    DR_CUDA(cudaGetLastError());
    return DR_OK;
}

dr_status dr_guide_mixture_pdf(const float *y_dev, uint32_t y_per_row, const float *dir_dev, uint32_t n, float *pdf_dev,
                               void *stream)
{
    DR_CHECK_ARG(n == 0 || (y_dev && dir_dev && pdf_dev), "dr_guide_mixture_pdf: NULL argument");
    if (n == 0) return DR_OK;
    k_guide_pdf<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(y_dev, dir_dev, n, y_per_row, pdf_dev);
    DR_CUDA(cudaGetLastError());
    return DR_OK;
}

dr_status dr_guide_last_loss(dr_guide *g, float *loss_host)
{
    DR_CHECK_ARG(g && loss_host, "dr_guide_last_loss: NULL argument");
    DR_CUDA(cudaSetDevice(g->ctx->device));
    DR_CUDA(cudaMemcpy(loss_host, g->scalars + 1, 4, cudaMemcpyDeviceToHost));
    return DR_OK;
}

}  // extern "C"
