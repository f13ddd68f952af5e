// kpax_learn.cu — training and inference entry points of the learned proposal network.
//
// Training runs in FP32 on the SIMT cores with hand-written kernels: one for a block of rows through the
// forward pass, the mixture-density loss and the backward pass, one for the weight gradients of all
// layers, and one for their fixed-order sums and Adam.
// Every reduction has a fixed order, so a training step is deterministic.  Inference for the
// planner runs on the tensor cores (kpax_mlp_tc.cuh) from a BF16 image packed here.
// The reference planner has no learned component; the network replaces nothing in it and only
// reshapes the distribution of the uniform control/duration draws.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <vector>

#include "kpax.h"
#include "kpax_internal.h"
#include "kpax_mlp.h"
#include "kpax_mlp_tc.cuh"

using namespace kpax;
using namespace kpax::mlp;

namespace {

// ---------------------------------------------------------------------------------------------
// FP32 training kernels.  A gradient is three launches:
//   k_mlp_rows  a CTA takes R rows through the three layers, the loss and back to the first layer's
//               pre-activation gradient, its activations in shared memory and the weights streamed
//               through two 36 KB buffers; it leaves what the weight gradients need in global memory
//   k_mlp_dw    dW = dZ^T A of all layers, 64 x 64 tiles, the rows split over up to kSplits partial sums
//   k_mlp_grad  partial sums added in split order (and Adam)
// Products accumulate in pairs of FP32 values (fma.rn.f32x2), each output in a fixed order.
// B200, loss and gradient of 4096 rows: 1770-1840 us with one 64 x 64-tile SGEMM per product (8-16 CTAs
// summing all rows for a weight gradient, 645-695 us each) and one thread per column for the bias
// gradients (230 us each); now 120 us: rows 75, weight gradients 34 (46 with 4 x 8 outputs per thread),
// sums 5.5.  Both products are bound by shared memory's return bandwidth, 21-26 of 72.6 TFLOP/s.
// Error of the gradient against 64 bits, by seed: 2.3-2.9e-6 before, 2.1-2.7e-6 now.

constexpr int kRowThreads = 256;
constexpr int kChunkK = 32, kWStride = kChunkK + 4;  // weights chunk: [columns][32], rows 36 floats apart (conflict-free)
constexpr int kActStride = kH + 4, kXStride = kInPad + 4, kOStride = kOutPad + 4;
constexpr int kWBuf = kH * kWStride;
// Transposed copies for the backward products: W3^T [kH][kOutPad], then W2^T [kH][kH].
constexpr size_t kOffW3T = 0, kOffW2T = kOffW3T + kH * kOutPad, kNumT = kOffW2T + kH * kH;
constexpr int kSplits = 16;

template <int R>
constexpr size_t kRowSmem = sizeof(float) * (R * (kXStride + 2 * kActStride + kOStride) + 2 * kWBuf);

struct RowArgs {
    const float* x;        // rows of kInPad features
    const float* y;        // rows of kDim targets
    const uint32_t* idx;   // row indices (null: 0, 1, ...)
    uint32_t n;
    const float* w;
    const float* wt;
    const float* mask;
    float inv_n;
    float *xb, *a1, *a2, *dz1, *dz2, *d_o, *ls;  // for the weight gradients
    float* out;            // forward only: n x kOutPad
};

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid = true)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Weight chunks in the order the layers read them: W1 (2 chunks of 32 inputs), W2 (8), W3 (8), and back
// W3^T (3), W2^T (8).
constexpr int kChunksForward = 18, kChunksTrain = 29;
__device__ __forceinline__ void load_chunk(const RowArgs& p, int id, float* buf)
{
    const float* src;
    int K, cols = kH;
    if(id < 2) src = p.w + kOffW1 + id * kChunkK, K = kInPad;
    else if(id < 10) src = p.w + kOffW2 + (id - 2) * kChunkK, K = kH;
    else if(id < 18) src = p.w + kOffW3 + (id - 10) * kChunkK, K = kH, cols = kOutPad;
    else if(id < 21) src = p.wt + kOffW3T + (id - 18) * kChunkK, K = kOutPad;
    else src = p.wt + kOffW2T + (id - 21) * kChunkK, K = kH;
    for(int i = threadIdx.x; i < cols * (kChunkK / 4); i += kRowThreads) {
        const int c = i >> 3, q = i & 7;
        cp_async16(buf + c * kWStride + 4 * q, src + (size_t)c * K + 4 * q);
    }
    cp_commit();
}

// acc[i][j] += sum over `chunks` chunks of A[row i][k] W[col + 32 j][k], even and odd k in the halves of
// acc.  a: the thread's first row (stride lda); chunk id + 1 is loaded while chunk id is used.  Shared
// memory returns 128 bytes per clock whether or not the lanes' addresses agree, so a 16-byte vector of
// k costs 4 (RT + CT) clocks per warp against RT CT for its FMAs on the SM.  256 x 256 layer of 32 rows,
// whole kernel: 8 x 4 outputs per thread and eight warps 75 us; 8 x 2 and sixteen warps 85 us; 8 x 8 and
// four warps (the balanced tile, but one warp per scheduler) 91 us.
template <int RT, int CT>
__device__ __forceinline__ void mac_chunks(const RowArgs& p, const float* a, int lda, int col, int first, int chunks, int total,
                                           float* wbuf, F2 (&acc)[RT][CT])
{
    for(int c = 0; c < chunks; ++c) {
        const int id = first + c;
        cp_wait();
        __syncthreads();  // chunk id is there, and the other buffer is no longer read
        if(id + 1 < total) load_chunk(p, id + 1, wbuf + ((id + 1) & 1) * kWBuf);
        const float* w = wbuf + (id & 1) * kWBuf + col * kWStride;
        const float* ac = a + c * kChunkK;
#pragma unroll 2  // 150 instructions: a chunk unrolled as a whole stalls on instruction fetches (80 us)
        for(int q = 0; q < kChunkK / 4; ++q) {
            ulonglong2 wv[CT];
#pragma unroll
            for(int j = 0; j < CT; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(w + 32 * j * kWStride + 4 * q);
#pragma unroll
            for(int i = 0; i < RT; ++i) {
                const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(ac + i * lda + 4 * q);
#pragma unroll
                for(int j = 0; j < CT; ++j) acc[i][j] = fma2(av.y, wv[j].y, fma2(av.x, wv[j].x, acc[i][j]));
            }
        }
    }
}

__device__ __forceinline__ float halves(F2 v)
{
    const float2 f = unpack(v);
    return f.x + f.y;
}

// Mixture-density negative log-likelihood of the logit targets y (masked dimensions only) and its
// gradient with respect to the outputs, scaled by inv_n, in place: eight lanes per sample, one component
// each (o: the sample's kOutPad outputs; lane k its component's 11).  Returns the loss.
__device__ __forceinline__ float mdn(float* o, const float* y, const float* mask, float inv_n, int k)
{
    constexpr float kHalfLog2Pi = 0.918938533204672742f;
    auto max8 = [](float v) {
#pragma unroll
        for(int d = 4; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
        return v;
    };
    auto sum8 = [](float v) {
#pragma unroll
        for(int d = 4; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        return v;
    };
    float* c = o + k * kCompStride;
    const float logit = c[0], amax = max8(logit);
    const float alse = amax + logf(sum8(expf(logit - amax)));
    float th[kDim], e[kDim], is[kDim], m[kDim], lp = logit - alse;
#pragma unroll
    for(int d = 0; d < kDim; ++d) {
        m[d] = mask[d];
        th[d] = tanhf(c[1 + kDim + d] * (1.0f / kSigHalf));
        const float s = kSigMid + kSigHalf * th[d];
        is[d] = expf(-s);
        e[d] = (y[d] - c[1 + d]) * is[d];
        lp += m[d] * (-0.5f * e[d] * e[d] - s - kHalfLog2Pi);
    }
    const float lmax = max8(lp), lse = lmax + logf(sum8(expf(lp - lmax)));
    const float r = expf(lp - lse), pi = expf(logit - alse);
    c[0] = (pi - r) * inv_n;
#pragma unroll
    for(int d = 0; d < kDim; ++d) {
        c[1 + d] = -r * m[d] * e[d] * is[d] * inv_n;
        c[1 + kDim + d] = -r * m[d] * (e[d] * e[d] - 1.0f) * (1.0f - th[d] * th[d]) * inv_n;
    }
    o[kOut + k] = 0.0f;  // padding outputs
    return -lse;
}

// R rows (32, or 16 where 32 would leave SMs without a CTA).  Warp w holds rows (w & 3) * R / 4 ... of the
// 256-column products and columns (w >> 2) * 128 + lane + 32 j: weights are read a 16-byte vector of k per
// column, activations as broadcasts.
template <int R, bool kTrain>
__global__ void __launch_bounds__(kRowThreads, 1) k_mlp_rows(const RowArgs p)
{
    static_assert(kOutPad - kOut == kComp, "one padding output per lane of a sample");
    constexpr int RT = R / 4, RO = R / 8, kTotal = kTrain ? kChunksTrain : kChunksForward;
    extern __shared__ __align__(16) float smem_f[];
    float* sX = smem_f;
    float* sA1 = sX + R * kXStride;
    float* sA2 = sA1 + R * kActStride;
    float* sO = sA2 + R * kActStride;
    float* wbuf = sO + R * kOStride;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t row0 = blockIdx.x * R;
    const int rows = (int)min((uint32_t)R, p.n - row0);
    load_chunk(p, 0, wbuf);
    for(int i = tid; i < R * kInPad; i += kRowThreads) {
        const int r = i / kInPad, c = i % kInPad;
        float v = 0.0f;
        if(r < rows) {
            v = p.x[(size_t)(p.idx ? p.idx[row0 + r] : row0 + r) * kInPad + c];
            if constexpr(kTrain) p.xb[(size_t)(row0 + r) * kInPad + c] = v;
        }
        sX[r * kXStride + c] = v;
    }
    const int r0 = (warp & 3) * RT, col = (warp >> 2) * 128 + lane;
    float g1[RT][4], g2[RT][4];  // SiLU' of both hidden layers (training)
    auto hidden = [&](F2 (&acc)[RT][4], const float* bias, float* s_act, float* d_act, float (&g)[RT][4]) {
#pragma unroll
        for(int j = 0; j < 4; ++j) {
            const float b = __ldg(bias + col + 32 * j);
#pragma unroll
            for(int i = 0; i < RT; ++i) {
                const float z = halves(acc[i][j]) + b, sg = sigmoid_f(z), a = z * sg;
                s_act[(r0 + i) * kActStride + col + 32 * j] = a;
                if constexpr(kTrain) {
                    g[i][j] = sg * (1.0f + z * (1.0f - sg));
                    if(r0 + i < rows) d_act[(size_t)(row0 + r0 + i) * kH + col + 32 * j] = a;
                }
                acc[i][j] = 0ull;
            }
        }
    };
    F2 acc[RT][4] = {};
    mac_chunks(p, sX + r0 * kXStride, kXStride, col, 0, 2, kTotal, wbuf, acc);
    hidden(acc, p.w + kOffB1, sA1, p.a1, g1);
    mac_chunks(p, sA1 + r0 * kActStride, kActStride, col, 2, 8, kTotal, wbuf, acc);
    hidden(acc, p.w + kOffB2, sA2, p.a2, g2);
    {
        F2 ao[RO][3] = {};
        mac_chunks(p, sA2 + warp * RO * kActStride, kActStride, lane, 10, 8, kTotal, wbuf, ao);
#pragma unroll
        for(int j = 0; j < 3; ++j) {
            const float b = __ldg(p.w + kOffB3 + lane + 32 * j);
#pragma unroll
            for(int i = 0; i < RO; ++i) {
                const float v = halves(ao[i][j]) + b;
                const int r = warp * RO + i;
                if constexpr(kTrain) sO[r * kOStride + lane + 32 * j] = v;
                else if(r < rows) p.out[(size_t)(row0 + r) * kOutPad + lane + 32 * j] = v;
            }
        }
    }
    if constexpr(kTrain) {
        __syncthreads();
        if(tid < 8 * R) {
            const int r = tid >> 3, k = tid & 7;
            const size_t src = r < rows ? (p.idx ? p.idx[row0 + r] : row0 + r) : 0;
            float y[kDim];
#pragma unroll
            for(int d = 0; d < kDim; ++d) y[d] = r < rows ? p.y[src * kDim + d] : 0.0f;
            const float loss = mdn(sO + r * kOStride, y, p.mask, r < rows ? p.inv_n : 0.0f, k);
            if(k == 0 && r < rows) p.ls[row0 + r] = loss;
        }
        __syncthreads();
        for(int i = tid; i < rows * kOutPad; i += kRowThreads)
            p.d_o[(size_t)row0 * kOutPad + i] = sO[(i / kOutPad) * kOStride + i % kOutPad];
        mac_chunks(p, sO + r0 * kOStride, kOStride, col, 18, 3, kTotal, wbuf, acc);
        // dZ2 takes A2's place (every warp is past the products that read A2)
#pragma unroll
        for(int j = 0; j < 4; ++j)
#pragma unroll
            for(int i = 0; i < RT; ++i) {
                const float d = halves(acc[i][j]) * g2[i][j];
                sA2[(r0 + i) * kActStride + col + 32 * j] = d;
                if(r0 + i < rows) p.dz2[(size_t)(row0 + r0 + i) * kH + col + 32 * j] = d;
                acc[i][j] = 0ull;
            }
        mac_chunks(p, sA2 + r0 * kActStride, kActStride, col, 21, 8, kTotal, wbuf, acc);
#pragma unroll
        for(int j = 0; j < 4; ++j)
#pragma unroll
            for(int i = 0; i < RT; ++i)
                if(r0 + i < rows) p.dz1[(size_t)(row0 + r0 + i) * kH + col + 32 * j] = halves(acc[i][j]) * g1[i][j];
    }
}

// Tile blockIdx.x (layer 3: 2 x 4 tiles, layer 2: 4 x 4, layer 1: 4 x 1) of the weight gradients
// over the rows of split blockIdx.y: part[split][parameter].  Thread (tm, tj) holds the 8 x 8 outputs of
// rows 4 tm .., 32 + 4 tm .. and columns 4 tj .., 32 + 4 tj .. (conflict-free 16-byte loads).
constexpr int kDwThreads = 64, kDwRows = 32, kDwTiles = 8 + 16 + 4;
__global__ void __launch_bounds__(kDwThreads) k_mlp_dw(const float* __restrict__ d_o, const float* __restrict__ dz2,
                                                       const float* __restrict__ dz1, const float* __restrict__ a2,
                                                       const float* __restrict__ a1, const float* __restrict__ xb, uint32_t n,
                                                       uint32_t rows_per_split, float* __restrict__ part)
{
    __shared__ __align__(16) float sP[2][kDwRows * 64], sQ[2][kDwRows * 64];
    const int tid = threadIdx.x, tm = tid >> 3, tj = tid & 7;
    const int tile = blockIdx.x;
    const float *P, *Q;
    int ldp, ldq, mt, jt, M;
    size_t off_w, off_b;
    if(tile < 8) P = d_o, Q = a2, ldp = M = kOutPad, ldq = kH, mt = tile >> 2, jt = tile & 3, off_w = kOffW3, off_b = kOffB3;
    else if(tile < 24) P = dz2, Q = a1, ldp = M = kH, ldq = kH, mt = (tile - 8) >> 2, jt = tile & 3, off_w = kOffW2, off_b = kOffB2;
    else P = dz1, Q = xb, ldp = M = kH, ldq = kInPad, mt = tile - 24, jt = 0, off_w = kOffW1, off_b = kOffB1;
    const uint32_t lo = min(n, blockIdx.y * rows_per_split), hi = min(n, lo + rows_per_split);
    auto load = [&](uint32_t r, int b) {  // rows r .. r + 31 (zero past the split's end and past column M)
        for(int i = tid; i < kDwRows * 16; i += kDwThreads) {
            const uint32_t row = r + (i >> 4);
            const int q = 4 * (i & 15);
            const bool in = row < hi, inp = in && 64 * mt + q < M;
            cp_async16(&sP[b][(i >> 4) * 64 + q], P + (inp ? (size_t)row * ldp + 64 * mt + q : 0), inp);
            cp_async16(&sQ[b][(i >> 4) * 64 + q], Q + (in ? (size_t)row * ldq + 64 * jt + q : 0), in);
        }
        cp_commit();
    };
    F2 acc[8][4] = {};
    float bsum[8] = {};
    const bool bias = jt == 0 && tj == 0;
    if(lo < hi) load(lo, 0);
    int b = 0;
    for(uint32_t r = lo; r < hi; r += kDwRows, b ^= 1) {
        cp_wait();
        __syncthreads();
        if(r + kDwRows < hi) load(r + kDwRows, b ^ 1);
#pragma unroll 2
        for(int k = 0; k < kDwRows; ++k) {
            const float4 p0 = *reinterpret_cast<const float4*>(&sP[b][k * 64 + 4 * tm]);
            const float4 p1 = *reinterpret_cast<const float4*>(&sP[b][k * 64 + 32 + 4 * tm]);
            const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(&sQ[b][k * 64 + 4 * tj]);
            const ulonglong2 q1 = *reinterpret_cast<const ulonglong2*>(&sQ[b][k * 64 + 32 + 4 * tj]);
            const float pa[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
            for(int i = 0; i < 8; ++i) {
                const F2 d = f2(pa[i]);
                acc[i][0] = fma2(d, q0.x, acc[i][0]), acc[i][1] = fma2(d, q0.y, acc[i][1]);
                acc[i][2] = fma2(d, q1.x, acc[i][2]), acc[i][3] = fma2(d, q1.y, acc[i][3]);
            }
            if(bias) {
#pragma unroll
                for(int i = 0; i < 8; ++i) bsum[i] += pa[i];
            }
        }
    }
    float* out = part + (size_t)blockIdx.y * kNumParams;
#pragma unroll
    for(int i = 0; i < 8; ++i) {
        const int m = 64 * mt + 32 * (i >> 2) + 4 * tm + (i & 3);
        if(m >= M) continue;
        float* w = out + off_w + (size_t)m * ldq + 64 * jt + 4 * tj;
        *reinterpret_cast<ulonglong2*>(w) = make_ulonglong2(acc[i][0], acc[i][1]);
        *reinterpret_cast<ulonglong2*>(w + 32) = make_ulonglong2(acc[i][2], acc[i][3]);
        if(bias) out[off_b + m] = bsum[i];
    }
}

struct AdamArgs {
    float *w, *wt, *m, *v;
    float b1, b2, c1, c2, eps;  // bias corrections folded into c1 = lr / (1 - b1^t) and c2 = 1 / (1 - b2^t)
};

// Index of parameter i in the transposed copies, or kNumT.
__device__ __forceinline__ size_t transposed(size_t i)
{
    if(i >= kOffW2 && i < kOffB2) return kOffW2T + ((i - kOffW2) % kH) * kH + (i - kOffW2) / kH;
    if(i >= kOffW3 && i < kOffB3) return kOffW3T + ((i - kOffW3) % kH) * kOutPad + (i - kOffW3) / kH;
    return kNumT;
}

// g = the splits' partial sums in split order; with kAdam also the optimiser's step.  The last block
// adds the rows' losses (strided partial sums, then a fixed halving tree).
template <bool kAdam>
__global__ void __launch_bounds__(256) k_mlp_grad(const float* __restrict__ part, int splits, float* __restrict__ g,
                                                  const float* __restrict__ ls, uint32_t n, float* __restrict__ loss,
                                                  const AdamArgs o)
{
    if(blockIdx.x == gridDim.x - 1) {
        __shared__ float s[256];
        float acc = 0.0f;
        for(uint32_t i = threadIdx.x; i < n; i += 256) acc += ls[i];
        s[threadIdx.x] = acc;
        __syncthreads();
        for(int h = 128; h > 0; h >>= 1) {
            if((int)threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
            __syncthreads();
        }
        if(threadIdx.x == 0) *loss = s[0];
        return;
    }
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= kNumParams) return;
    float gi = 0.0f;
#pragma unroll 8
    for(int s = 0; s < splits; ++s) gi += part[(size_t)s * kNumParams + i];
    g[i] = gi;
    if constexpr(kAdam) {
        const float mi = o.b1 * o.m[i] + (1.0f - o.b1) * gi, vi = o.b2 * o.v[i] + (1.0f - o.b2) * gi * gi;
        o.m[i] = mi, o.v[i] = vi;
        const float w = o.w[i] - o.c1 * mi / (sqrtf(vi * o.c2) + o.eps);
        o.w[i] = w;
        const size_t t = transposed(i);
        if(t < kNumT) o.wt[t] = w;
    }
}

__global__ void k_transpose(const float* __restrict__ w, float* __restrict__ wt)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= kNumParams) return;
    const size_t t = transposed(i);
    if(t < kNumT) wt[t] = w[i];
}

// FP32 master -> BF16 image in the MMA's shared-memory layout, plus the FP32 biases.
__global__ void k_pack(const float* __restrict__ w, uint8_t* __restrict__ img)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n1 = kH * kInPad, n2 = kH * kH, n3 = kOutPad * kH, nb = kH + kH + kOutPad;
    if(i < n1) {
        const uint32_t r = i / kInPad, k = i % kInPad;
        *reinterpret_cast<__nv_bfloat16*>(img + kImgW1 + swz(r, k)) = __float2bfloat16_rn(w[kOffW1 + i]);
    } else if(i < n1 + n2) {
        const uint32_t j = i - n1, r = j / kH, k = j % kH;
        *reinterpret_cast<__nv_bfloat16*>(img + kImgW2 + (k >> 6) * kH * kSlabRowBytes + swz(r, k & 63)) =
          __float2bfloat16_rn(w[kOffW2 + j]);
    } else if(i < n1 + n2 + n3) {
        const uint32_t j = i - n1 - n2, r = j / kH, k = j % kH;
        *reinterpret_cast<__nv_bfloat16*>(img + kImgW3 + (k >> 6) * kOutPad * kSlabRowBytes + swz(r, k & 63)) =
          __float2bfloat16_rn(w[kOffW3 + j]);
    } else if(i < n1 + n2 + n3 + nb) {
        const uint32_t j = i - n1 - n2 - n3;
        const float b = j < (uint32_t)kH ? w[kOffB1 + j] : j < 2u * kH ? w[kOffB2 + j - kH] : w[kOffB3 + j - 2 * kH];
        reinterpret_cast<float*>(img + kImgBias)[j] = b;
    }
}

__global__ void k_features(const KParams p, const uint32_t* __restrict__ occ, const float* __restrict__ states, uint32_t stride,
                           const float* __restrict__ goals, uint32_t n, float* __restrict__ X)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    float s[12], g[3], x[kInPad];
#pragma unroll
    for(int d = 0; d < 12; ++d) s[d] = states[(size_t)i * stride + d];
#pragma unroll
    for(int d = 0; d < 3; ++d) g[d] = goals[(size_t)i * 3 + d];
    features(p, occ, s, g, x);
#pragma unroll
    for(int c = 0; c < kInPad; ++c) X[(size_t)i * kInPad + c] = x[c];
}

// Rows given as arrays of states and goals (tests and offline use of the tensor-core pass).
struct ArraySrc {
    static constexpr bool kDebug = true;
    KParams p;
    const uint32_t* occ;
    const float* states;
    const float* goals;
    uint32_t stride, n;
    float* mix;
    float* out;
    uint16_t* h1;
    uint16_t* h2;
    uint32_t row0;  // first row of the current tile
    __device__ uint32_t tiles() const { return (n + tc::kRows - 1) / tc::kRows; }
    __device__ void seek(uint32_t tile) { row0 = tile * tc::kRows; }
    __device__ uint32_t rows() const { return min((uint32_t)tc::kRows, n - row0); }
    __device__ float* records() const { return mix + (size_t)row0 * kMixFloats; }
    __device__ void row_features(uint32_t r, float x[kInPad]) const
    {
        const uint32_t row = row0 + r;
        float s[12], g[3];
        for(int d = 0; d < 12; ++d) s[d] = states[(size_t)row * stride + d];
        for(int d = 0; d < 3; ++d) g[d] = goals[(size_t)row * 3 + d];
        features(p, occ, s, g, x);
    }
    __device__ void dump_h(int layer, uint32_t r, uint32_t col0, const uint4 bits[2]) const
    {
        uint16_t* dst = layer == 1 ? h1 : h2;
        if(!dst) return;
        uint4* d = reinterpret_cast<uint4*>(dst + (size_t)(row0 + r) * kH + col0);
        d[0] = bits[0], d[1] = bits[1];
    }
    __device__ void dump_out(uint32_t r, uint32_t col, float v) const
    {
        if(out) out[(size_t)(row0 + r) * kOutPad + col] = v;
    }
};

__global__ void __launch_bounds__(tc::kThreads, 1) k_forward_tc(const ArraySrc src, const uint8_t* __restrict__ img, uint32_t* err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    ArraySrc s = src;  // per-thread cursor
    tc::forward(s, img, smem, err);
}

// One warp per R1 workspace cell: the cell is blocked when at least half of the 4x4x4 lattice
// of points at offsets (i + 1/2) / 4 lies inside an obstacle (closed boxes).  `words` must be
// zeroed by the caller.
__global__ void k_occupancy(const KParams p, const Grid g, uint32_t* __restrict__ words)
{
    const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int ncell = p.W1 * p.W1 * p.W1;
    if(warp >= ncell) return;
    const int c[3] = {warp % p.W1, (warp / p.W1) % p.W1, warp / (p.W1 * p.W1)};
    uint32_t inside = 0;
#pragma unroll
    for(int h = 0; h < 2; ++h) {
        const int j = lane + 32 * h, i3[3] = {j & 3, (j >> 2) & 3, j >> 4};
        float q[3];
#pragma unroll
        for(int d = 0; d < 3; ++d)
            q[d] = __fadd_rn(p.wmin, __fmul_rn(__fadd_rn((float)c[d], 0.125f * (float)(2 * i3[d] + 1)), p.w1size));
        const int gc = grid_coord(g, q[0]) + g.dim * (grid_coord(g, q[1]) + g.dim * grid_coord(g, q[2]));
        bool in = false;
        for(uint32_t k = __ldg(g.off + gc), e = __ldg(g.off + gc + 1); k < e && !in; ++k) {
            const uint32_t o = __ldg(g.ent + k);
            const float4 a = __ldg(g.obs + 2 * o), m = __ldg(g.obs + 2 * o + 1);
            in = a.x <= q[0] && q[0] <= m.x && a.y <= q[1] && q[1] <= m.y && a.z <= q[2] && q[2] <= m.z;
        }
        inside += __popc(__ballot_sync(0xffffffffu, in));
    }
    if(lane == 0 && inside >= 32) atomicOr(words + (warp >> 5), 1u << (warp & 31));
}

inline uint32_t blocks(size_t n, int bs) { return (uint32_t)((n + bs - 1) / bs); }

}  // namespace

struct kpax_mlp {
    uint32_t max_batch = 0;
    float* w = nullptr;     // FP32 master parameters
    float* g = nullptr;     // gradients
    float* m = nullptr;     // Adam moments
    float* v = nullptr;
    uint8_t* img = nullptr; // BF16 image
    uint32_t* err = nullptr;
    float* mask = nullptr;  // 5 loss-dimension weights
    float* loss = nullptr;  // scalar
    float* h_loss = nullptr;  // pinned scalar
    float* wt = nullptr;    // transposed copies of W3 and W2
    // a batch's gathered rows, activations, gradients and losses, and the splits' partial gradients
    float *xb = nullptr, *a1 = nullptr, *a2 = nullptr, *dz1 = nullptr, *dz2 = nullptr, *d_o = nullptr, *ls = nullptr, *part = nullptr;
    int sms = 148;
    uint64_t step = 0;
    bool packed = false;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;  // around the last tensor-core pass
    float last_ms = 0.0f;
};

namespace kpax {

// Splits of the weight gradients' rows: enough 64 x 64 tiles for three CTAs per SM, at least two chunks
// of rows each (partial sums cost a write and a read of every parameter).
static int grad_splits(uint32_t rows) { return (int)std::min<uint32_t>(kSplits, std::max<uint32_t>(1, rows / (2 * kDwRows))); }

template <bool kTrain>
static kpax_status launch_rows(const kpax_mlp* n, const RowArgs& a, cudaStream_t st)
{
    // 16 rows per CTA while that gives no SM a second one: less work per CTA, the same weights to stream
    const bool small = a.n <= 16u * (uint32_t)n->sms;
    const void* fn = small ? (const void*)k_mlp_rows<16, kTrain> : (const void*)k_mlp_rows<32, kTrain>;
    const size_t smem = small ? kRowSmem<16> : kRowSmem<32>;
    KPAX_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if(small) k_mlp_rows<16, kTrain><<<blocks(a.n, 16), kRowThreads, smem, st>>>(a);
    else k_mlp_rows<32, kTrain><<<blocks(a.n, 32), kRowThreads, smem, st>>>(a);
    count_launch();
    KPAX_CHECK_LAUNCH();
    return KPAX_OK;
}

// Loss sum (into n->loss) and gradient (into g) of the rows idx (null: all) of (x, y); with adam the
// optimiser's step as well.
static kpax_status mlp_gradient(kpax_mlp* n, const float* x, const float* y, const uint32_t* idx, uint32_t rows, float* g,
                                const AdamArgs* adam, cudaStream_t st)
{
    RowArgs a{x, y, idx, rows, n->w, n->wt, n->mask, 1.0f / (float)rows, n->xb, n->a1, n->a2, n->dz1, n->dz2, n->d_o, n->ls, nullptr};
    kpax_status s = launch_rows<true>(n, a, st);
    if(s != KPAX_OK) return s;
    const int splits = grad_splits(rows);
    const uint32_t per = (rows + (uint32_t)splits - 1) / (uint32_t)splits;
    k_mlp_dw<<<dim3(kDwTiles, splits), kDwThreads, 0, st>>>(n->d_o, n->dz2, n->dz1, n->a2, n->a1, n->xb, rows, per, n->part);
    const uint32_t grid = blocks(kNumParams, 256) + 1;
    if(adam) k_mlp_grad<true><<<grid, 256, 0, st>>>(n->part, splits, g, n->ls, rows, n->loss, *adam);
    else k_mlp_grad<false><<<grid, 256, 0, st>>>(n->part, splits, g, n->ls, rows, n->loss, AdamArgs{});
    count_launch(2);
    KPAX_CHECK_LAUNCH();
    return KPAX_OK;
}

kpax_status launch_occupancy(const KParams& p, const Grid& g, uint32_t* d_words, cudaStream_t st)
{
    const uint32_t cells = (uint32_t)(p.W1 * p.W1 * p.W1);
    KPAX_CUDA(cudaMemsetAsync(d_words, 0, sizeof(uint32_t) * ((cells + 31) / 32), st));
    k_occupancy<<<blocks((size_t)cells * 32, 256), 256, 0, st>>>(p, g, d_words);
    count_launch();
    KPAX_CHECK_LAUNCH();
    return KPAX_OK;
}

const uint8_t* mlp_image(const kpax_mlp* n) { return n && n->packed ? n->img : nullptr; }

}  // namespace kpax

static kpax_status env_occupancy(kpax_env* e, cudaStream_t st)
{
    if(e->d_occ) return KPAX_OK;
    const uint32_t words = (uint32_t)((e->params.W1 * e->params.W1 * e->params.W1 + 31) / 32);
    KPAX_CUDA(cudaMalloc(&e->d_occ, sizeof(uint32_t) * words));
    return launch_occupancy(e->params, e->env.view(), e->d_occ, st);
}

static kpax_status check_learned_env(const kpax_env* e, const char* fn)
{
    if(!e) return set_error("%s: null env", fn), KPAX_EINVAL;
    if(e->params.model != KPAX_MODEL_QUADROTOR) return set_error("%s: the proposal network is defined for the quadrotor", fn), KPAX_EINVAL;
    return KPAX_OK;
}

extern "C" {

kpax_status kpax_mlp_create(uint32_t max_batch, kpax_mlp** out)
{
    if(!out || max_batch == 0 || max_batch > (1u << 22)) return set_error("kpax_mlp_create: bad arguments"), KPAX_EINVAL;
    *out = nullptr;
    kpax_mlp* n = new(std::nothrow) kpax_mlp();
    if(!n) return set_error("kpax_mlp_create: host allocation failed"), KPAX_ENOMEM;
    n->max_batch = max_batch;
    const size_t P = kNumParams, B = max_batch;
    auto fail = [&](kpax_status st) {
        cudaGetLastError();  // reported here, not by the next launch check
        kpax_mlp_destroy(n);
        return st;
    };
#define KPAX_MLP_ALLOC(ptr, bytes)                                                          \
    do {                                                                                    \
        cudaError_t e_ = cudaMalloc(&(ptr), (bytes));                                       \
        if(e_ != cudaSuccess) {                                                             \
            set_error("kpax_mlp_create: %s", cudaGetErrorString(e_));                       \
            return fail(e_ == cudaErrorMemoryAllocation ? KPAX_ENOMEM : KPAX_ECUDA);        \
        }                                                                                   \
    } while(0)
    KPAX_MLP_ALLOC(n->w, P * 4);
    KPAX_MLP_ALLOC(n->g, P * 4);
    KPAX_MLP_ALLOC(n->m, P * 4);
    KPAX_MLP_ALLOC(n->v, P * 4);
    KPAX_MLP_ALLOC(n->img, kImgBytes);
    KPAX_MLP_ALLOC(n->err, 4);
    KPAX_MLP_ALLOC(n->mask, kDim * 4);
    KPAX_MLP_ALLOC(n->loss, 4);
    KPAX_MLP_ALLOC(n->wt, kNumT * 4);
    KPAX_MLP_ALLOC(n->xb, B * kInPad * 4);
    KPAX_MLP_ALLOC(n->a1, B * kH * 4);
    KPAX_MLP_ALLOC(n->a2, B * kH * 4);
    KPAX_MLP_ALLOC(n->dz1, B * kH * 4);
    KPAX_MLP_ALLOC(n->dz2, B * kH * 4);
    KPAX_MLP_ALLOC(n->d_o, B * kOutPad * 4);
    KPAX_MLP_ALLOC(n->ls, B * 4);
    KPAX_MLP_ALLOC(n->part, P * 4 * (size_t)grad_splits(max_batch));
#undef KPAX_MLP_ALLOC
    if(cudaMallocHost(&n->h_loss, 4) != cudaSuccess) return set_error("kpax_mlp_create: pinned alloc"), fail(KPAX_ENOMEM);
    if(cudaEventCreate(&n->ev0) != cudaSuccess || cudaEventCreate(&n->ev1) != cudaSuccess)
        return set_error("kpax_mlp_create: event creation failed"), fail(KPAX_ECUDA);
    int dev = 0;
    if(cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return set_error("kpax_mlp_create: no device"), fail(KPAX_ECUDA);
    if(cudaMemset(n->w, 0, P * 4) != cudaSuccess || cudaMemset(n->wt, 0, kNumT * 4) != cudaSuccess || cudaMemset(n->m, 0, P * 4) != cudaSuccess ||
       cudaMemset(n->v, 0, P * 4) != cudaSuccess || cudaMemset(n->err, 0, 4) != cudaSuccess ||
       cudaMemset(n->img, 0, kImgBytes) != cudaSuccess)
        return set_error("kpax_mlp_create: memset failed"), fail(KPAX_ECUDA);
    const float ones[kDim] = {1, 1, 1, 1, 1};
    if(cudaMemcpy(n->mask, ones, sizeof(ones), cudaMemcpyHostToDevice) != cudaSuccess)
        return set_error("kpax_mlp_create: copy failed"), fail(KPAX_ECUDA);
    *out = n;
    return KPAX_OK;
}

kpax_status kpax_mlp_destroy(kpax_mlp* n)
{
    if(!n) return KPAX_OK;
    void* dev[] = {n->w, n->g, n->m, n->v, n->img, n->err, n->mask, n->loss, n->wt, n->xb, n->a1, n->a2, n->dz1, n->dz2, n->d_o, n->ls, n->part};
    for(void* p : dev)
        if(p) cudaFree(p);
    if(n->h_loss) cudaFreeHost(n->h_loss);
    if(n->ev0) cudaEventDestroy(n->ev0);
    if(n->ev1) cudaEventDestroy(n->ev1);
    delete n;
    return KPAX_OK;
}

uint32_t kpax_mlp_num_params(void) { return (uint32_t)kNumParams; }

float kpax_mlp_last_propose_ms(const kpax_mlp* n) { return n ? n->last_ms : 0.0f; }

kpax_status kpax_mlp_set_params(kpax_mlp* n, const float* h_params, void* stream)
{
    if(!n || !h_params) return set_error("kpax_mlp_set_params: null argument"), KPAX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    KPAX_CUDA(cudaMemcpyAsync(n->w, h_params, kNumParams * 4, cudaMemcpyHostToDevice, st));
    KPAX_CUDA(cudaMemsetAsync(n->m, 0, kNumParams * 4, st));
    KPAX_CUDA(cudaMemsetAsync(n->v, 0, kNumParams * 4, st));
    k_transpose<<<blocks(kNumParams, 256), 256, 0, st>>>(n->w, n->wt);
    count_launch();
    KPAX_CHECK_LAUNCH();
    KPAX_CUDA(cudaStreamSynchronize(st));
    n->step = 0;
    return kpax_mlp_pack(n, stream);
}

kpax_status kpax_mlp_get_params(kpax_mlp* n, float* h_params, void* stream)
{
    if(!n || !h_params) return set_error("kpax_mlp_get_params: null argument"), KPAX_EINVAL;
    KPAX_CUDA(cudaMemcpyAsync(h_params, n->w, kNumParams * 4, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    KPAX_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return KPAX_OK;
}

kpax_status kpax_mlp_set_loss_mask(kpax_mlp* n, const float* h_mask5, void* stream)
{
    if(!n || !h_mask5) return set_error("kpax_mlp_set_loss_mask: null argument"), KPAX_EINVAL;
    KPAX_CUDA(cudaMemcpyAsync(n->mask, h_mask5, kDim * 4, cudaMemcpyHostToDevice, (cudaStream_t)stream));
    KPAX_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return KPAX_OK;
}

kpax_status kpax_mlp_pack(kpax_mlp* n, void* stream)
{
    if(!n) return set_error("kpax_mlp_pack: null network"), KPAX_EINVAL;
    const uint32_t total = kH * kInPad + kH * kH + kOutPad * kH + kH + kH + kOutPad;
    k_pack<<<blocks(total, 256), 256, 0, (cudaStream_t)stream>>>(n->w, n->img);
    count_launch();
    KPAX_CHECK_LAUNCH();
    n->packed = true;
    return KPAX_OK;
}

kpax_status kpax_mlp_forward(kpax_mlp* n, const float* d_x, uint32_t rows, float* d_out, void* stream)
{
    if(!n || !d_x || !d_out || rows > n->max_batch) return set_error("kpax_mlp_forward: bad arguments"), KPAX_EINVAL;
    if(!rows) return KPAX_OK;
    // a CTA writes its rows' outputs while others still read their inputs: buffers that overlap go through the
    // net's own (kH floats a row)
    static_assert(kOutPad <= kH, "outputs fit an activation buffer");
    const uintptr_t x = (uintptr_t)d_x, o = (uintptr_t)d_out;
    const size_t bytes = sizeof(float) * (size_t)rows * kOutPad;
    const bool overlap = x < o + bytes && o < x + sizeof(float) * (size_t)rows * kInPad;
    RowArgs a{};
    a.x = d_x, a.n = rows, a.w = n->w, a.wt = n->wt, a.out = overlap ? n->a1 : d_out;
    kpax_status s = launch_rows<false>(n, a, (cudaStream_t)stream);
    if(s != KPAX_OK || !overlap) return s;
    KPAX_CUDA(cudaMemcpyAsync(d_out, n->a1, bytes, cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
    return KPAX_OK;
}

kpax_status kpax_mlp_loss_grad(kpax_mlp* n, const float* d_x, const float* d_y, uint32_t rows, float* h_loss, float* d_grad,
                               void* stream)
{
    if(!n || !d_x || !d_y || !rows || rows > n->max_batch) return set_error("kpax_mlp_loss_grad: bad arguments"), KPAX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    kpax_status s = mlp_gradient(n, d_x, d_y, nullptr, rows, d_grad ? d_grad : n->g, nullptr, st);
    if(s != KPAX_OK) return s;
    if(h_loss) {
        KPAX_CUDA(cudaMemcpyAsync(n->h_loss, n->loss, 4, cudaMemcpyDeviceToHost, st));
        KPAX_CUDA(cudaStreamSynchronize(st));
        *h_loss = *n->h_loss / (float)rows;
    }
    return KPAX_OK;
}

kpax_status kpax_mlp_train_step(kpax_mlp* n, const float* d_x, const float* d_y, const uint32_t* d_idx, uint32_t batch, float lr,
                                float* h_loss, void* stream)
{
    if(!n || !d_x || !d_y || !d_idx || !batch || batch > n->max_batch || !(lr > 0.0f))
        return set_error("kpax_mlp_train_step: bad arguments"), KPAX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    const double b1 = 0.9, b2 = 0.999, t = (double)(n->step + 1);
    const AdamArgs o{n->w, n->wt, n->m, n->v, (float)b1, (float)b2, (float)(lr / (1.0 - pow(b1, t))), (float)(1.0 / (1.0 - pow(b2, t))), 1e-8f};
    kpax_status s = mlp_gradient(n, d_x, d_y, d_idx, batch, n->g, &o, st);
    if(s != KPAX_OK) return s;
    n->step += 1;
    n->packed = false;
    if(h_loss) {
        KPAX_CUDA(cudaMemcpyAsync(n->h_loss, n->loss, 4, cudaMemcpyDeviceToHost, st));
        KPAX_CUDA(cudaStreamSynchronize(st));
        *h_loss = *n->h_loss / (float)batch;
    }
    return KPAX_OK;
}

kpax_status kpax_mlp_adam_state(kpax_mlp* n, float* h_m, float* h_v, uint64_t* step, void* stream)
{
    if(!n) return set_error("kpax_mlp_adam_state: null network"), KPAX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    if(h_m) KPAX_CUDA(cudaMemcpyAsync(h_m, n->m, kNumParams * 4, cudaMemcpyDeviceToHost, st));
    if(h_v) KPAX_CUDA(cudaMemcpyAsync(h_v, n->v, kNumParams * 4, cudaMemcpyDeviceToHost, st));
    KPAX_CUDA(cudaStreamSynchronize(st));
    if(step) *step = n->step;
    return KPAX_OK;
}

kpax_status kpax_env_occupancy(kpax_env* e, uint32_t* d_words, void* stream)
{
    kpax_status s = check_learned_env(e, "kpax_env_occupancy");
    if(s != KPAX_OK) return s;
    if(!d_words) return set_error("kpax_env_occupancy: null output"), KPAX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    s = env_occupancy(e, st);
    if(s != KPAX_OK) return s;
    const uint32_t words = (uint32_t)((e->params.W1 * e->params.W1 * e->params.W1 + 31) / 32);
    KPAX_CUDA(cudaMemcpyAsync(d_words, e->d_occ, sizeof(uint32_t) * words, cudaMemcpyDeviceToDevice, st));
    return KPAX_OK;
}

kpax_status kpax_mlp_features(kpax_env* e, const float* d_states, uint32_t stride, const float* d_goals, uint32_t n,
                              float* d_x, void* stream)
{
    kpax_status s = check_learned_env(e, "kpax_mlp_features");
    if(s != KPAX_OK) return s;
    if(!n) return KPAX_OK;
    if(!d_states || !d_goals || !d_x || stride < 12) return set_error("kpax_mlp_features: bad arguments"), KPAX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    s = env_occupancy(e, st);
    if(s != KPAX_OK) return s;
    k_features<<<blocks(n, 128), 128, 0, st>>>(e->params, e->d_occ, d_states, stride, d_goals, n, d_x);
    count_launch();
    KPAX_CHECK_LAUNCH();
    return KPAX_OK;
}

kpax_status kpax_mlp_propose(kpax_mlp* net, kpax_env* e, const float* d_states, uint32_t stride, const float* d_goals, uint32_t n,
                             float* d_mix, float* d_out, uint16_t* d_h1, uint16_t* d_h2, void* stream)
{
    kpax_status s = check_learned_env(e, "kpax_mlp_propose");
    if(s != KPAX_OK) return s;
    if(!net || !net->packed) return set_error("kpax_mlp_propose: network not packed"), KPAX_EINVAL;
    if(!n) return KPAX_OK;
    if(!d_states || !d_goals || !d_mix || stride < 12) return set_error("kpax_mlp_propose: bad arguments"), KPAX_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    s = env_occupancy(e, st);
    if(s != KPAX_OK) return s;
    KPAX_CUDA(cudaFuncSetAttribute(k_forward_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::kSmemBytes));
    int dev = 0, sms = 0;
    KPAX_CUDA(cudaGetDevice(&dev));
    KPAX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint32_t tiles = (n + tc::kRows - 1) / tc::kRows;
    ArraySrc src{e->params, e->d_occ, d_states, d_goals, stride, n, d_mix, d_out, d_h1, d_h2};
    KPAX_CUDA(cudaMemsetAsync(net->err, 0, 4, st));
    KPAX_CUDA(cudaEventRecord(net->ev0, st));
    k_forward_tc<<<std::min<uint32_t>(tiles, (uint32_t)sms), tc::kThreads, tc::kSmemBytes, st>>>(src, net->img, net->err);
    count_launch();
    KPAX_CHECK_LAUNCH();
    KPAX_CUDA(cudaEventRecord(net->ev1, st));
    uint32_t h_err = 0;
    KPAX_CUDA(cudaMemcpyAsync(&h_err, net->err, 4, cudaMemcpyDeviceToHost, st));
    KPAX_CUDA(cudaStreamSynchronize(st));
    KPAX_CUDA(cudaEventElapsedTime(&net->last_ms, net->ev0, net->ev1));
    if(h_err) return set_error("kpax_mlp_propose: a tensor-core pipeline wait expired (code %u)", h_err), KPAX_ETIMEOUT;
    return KPAX_OK;
}

}  // extern "C"
