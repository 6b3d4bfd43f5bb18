// Learned sizer: a 16 -> 64 -> 64 -> 64 -> 2 MLP (ReLU hidden layers,
// linear output) with BF16 weights and FP32 accumulation, trained on the GPU
// by the kernels below (fused forward + backward over tiles of samples, Adam
// update of FP32 master weights that re-quantises the BF16 copy). It
// predicts (log2 group cardinality / 24, filter selectivity) from 16
// features of a query, replacing the exact count pass that sizes hash
// tables; see gpudb_batch.h.
//
// Parameter layout (9,538 floats): W1[64][16] b1[64] W2[64][64] b2[64]
// W3[64][64] b3[64] W4[2][64] b4[2] — weights out-major.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <memory>
#include <random>
#include <string>
#include <utility>
#include <vector>

#include "../../../include/gpudb_batch.h"

namespace gpudb {
void setThreadError(const std::string& message);
}

namespace {

constexpr int kIn = 16, kH = 64, kOut = 2;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kH * kIn, kOffW2 = kOffB1 + kH, kOffB2 = kOffW2 + kH * kH,
              kOffW3 = kOffB2 + kH, kOffB3 = kOffW3 + kH * kH, kOffW4 = kOffB3 + kH, kOffB4 = kOffW4 + kOut * kH,
              kParams = kOffB4 + kOut;
static_assert(kParams == 9538, "parameter count");
constexpr int kThreads = 256;  // threads per CTA
// Samples up to which a prediction reads and answers in pinned memory, over
// the link, instead of by two copies of pageable memory. B200, whole call:
// 23 us instead of 35 for 16 samples, 32 / 37 for 1,024, 43 / 68 for 4,096,
// 62 / 89 for 8,192.
constexpr int kFew = 8192;

// A CTA works on tiles of TS samples. Weights (as FP32) and activations lie
// in shared memory feature-major with 4 floats of padding per row, so that
// the lanes of a warp, whether they differ in sample or in feature row, read
// 16-byte words of different banks. A thread owns 4 x SV outputs of each
// layer (SV = TS / 16 neighbouring samples) and, in the weight gradients, 4 x 4
// of a layer's matrix, which it keeps in registers over all tiles of its
// CTA: one atomic per parameter and CTA instead of one per 32 samples. The
// CTAs' sums meet in FP64: as many FP32 adds in a row as there are CTAs made
// the gradients of 700 samples in tiles of 16 a third less accurate than those
// in tiles of 32 (1.0e-7 of their norm against 7.5e-8).
// Bound by shared-memory reads beside the FP32 adds (77 us of FMA at 100K
// samples). B200, kernel alone, a 32-sample tile per CTA (weights read as
// BF16 with all lanes in one bank, 30M atomics) -> this: training pass over
// 100,003 samples 873 -> 175 us, 9,472 90 -> 31, 512 55 -> 20; prediction
// 479 -> 78, 51 -> 17, 30 -> 15 us.
constexpr int kPad = 4;

template <int TS>
struct Smem {
    static constexpr int LD = TS + kPad;     // activations: row = feature
    static constexpr int LW = kH + kPad, LW1 = kIn + kPad;
    float w1[kH * LW1], w2[kH * LW], w3[kH * LW], w4[kOut * LW];
    float b1[kH], b2[kH], b3[kH], b4[kOut + 2];
    float x[kIn * LD];
    float h1[kH * LD], h2[kH * LD], h3[kH * LD];  // then the gradients at these layers
    float y[kOut * LD];                           // outputs, then their gradients
};

template <int V>
__device__ __forceinline__ void vload(const float* p, float (&v)[V]) {
    if constexpr (V == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
    } else if constexpr (V == 2) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x, v[1] = t.y;
    } else {
        v[0] = *p;
    }
}
template <int V>
__device__ __forceinline__ void vstore(float* p, const float (&v)[V]) {
    if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else *p = v[0];
}

template <int TS>
__device__ void loadWeights(Smem<TS>& sm, const __nv_bfloat16* __restrict__ wbf) {
    using S = Smem<TS>;
    for (int i = threadIdx.x; i < kH * kIn; i += kThreads)
        sm.w1[i / kIn * S::LW1 + i % kIn] = __bfloat162float(wbf[kOffW1 + i]);
    for (int i = threadIdx.x; i < kH * kH; i += kThreads) {
        sm.w2[i / kH * S::LW + i % kH] = __bfloat162float(wbf[kOffW2 + i]);
        sm.w3[i / kH * S::LW + i % kH] = __bfloat162float(wbf[kOffW3 + i]);
    }
    for (int i = threadIdx.x; i < kOut * kH; i += kThreads)
        sm.w4[i / kH * S::LW + i % kH] = __bfloat162float(wbf[kOffW4 + i]);
    if (threadIdx.x < kH) {
        sm.b1[threadIdx.x] = __bfloat162float(wbf[kOffB1 + threadIdx.x]);
        sm.b2[threadIdx.x] = __bfloat162float(wbf[kOffB2 + threadIdx.x]);
        sm.b3[threadIdx.x] = __bfloat162float(wbf[kOffB3 + threadIdx.x]);
    }
    if (threadIdx.x < kOut) sm.b4[threadIdx.x] = __bfloat162float(wbf[kOffB4 + threadIdx.x]);
}

// Samples s0 .. s0 + ns of X, feature-major; the rest of the tile is zero.
template <int TS>
__device__ void loadSamples(Smem<TS>& sm, const float* __restrict__ X, long long s0, int ns) {
    for (int i = threadIdx.x; i < TS * (kIn / 4); i += kThreads) {
        const int s = i / (kIn / 4), k = i % (kIn / 4) * 4;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (s < ns) v = *reinterpret_cast<const float4*>(X + (s0 + s) * kIn + k);
        sm.x[k * Smem<TS>::LD + s] = v.x;
        sm.x[(k + 1) * Smem<TS>::LD + s] = v.y;
        sm.x[(k + 2) * Smem<TS>::LD + s] = v.z;
        sm.x[(k + 3) * Smem<TS>::LD + s] = v.w;
    }
}

// out[j][s] = relu(b[j] + sum_k W[j][k] * in[k][s]), 64 outputs.
template <int TS, int NI, int LDW>
__device__ __forceinline__ void dense(const float* W, const float* b, const float* in, float* out) {
    constexpr int SV = TS / 16, LD = TS + kPad;
    const int sg = threadIdx.x & 15, jg = threadIdx.x >> 4;
    float acc[4][SV];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int v = 0; v < SV; ++v) acc[i][v] = b[jg + 16 * i];
#pragma unroll 4
    for (int k = 0; k < NI; k += 4) {
        float w[4][4], a[4][SV];
#pragma unroll
        for (int i = 0; i < 4; ++i) vload<4>(W + (jg + 16 * i) * LDW + k, w[i]);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) vload<SV>(in + (k + kk) * LD + sg * SV, a[kk]);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int v = 0; v < SV; ++v) acc[i][v] = fmaf(w[i][kk], a[kk][v], acc[i][v]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int v = 0; v < SV; ++v) acc[i][v] = fmaxf(acc[i][v], 0.0f);
        vstore<SV>(out + (jg + 16 * i) * LD + sg * SV, acc[i]);
    }
}

// Layers 1..4 of the tile in sm.x; ends with a barrier.
template <int TS>
__device__ __forceinline__ void forwardTile(Smem<TS>& sm) {
    using S = Smem<TS>;
    dense<TS, kIn, S::LW1>(sm.w1, sm.b1, sm.x, sm.h1);
    __syncthreads();
    dense<TS, kH, S::LW>(sm.w2, sm.b2, sm.h1, sm.h2);
    __syncthreads();
    dense<TS, kH, S::LW>(sm.w3, sm.b3, sm.h2, sm.h3);
    __syncthreads();
    if (threadIdx.x < kOut * TS) {
        const int j = threadIdx.x / TS, s = threadIdx.x % TS;
        float acc = sm.b4[j];
#pragma unroll 8
        for (int k = 0; k < kH; ++k) acc = fmaf(sm.w4[j * S::LW + k], sm.h3[k * S::LD + s], acc);
        sm.y[j * S::LD + s] = acc;
    }
    __syncthreads();
}

// acc[i][v] = dIn[4 kg + i][sample] = sum_j dOut[j][sample] * W[j][4 kg + i],
// zero where the layer's own activation was not positive.
template <int TS, int NO>
__device__ __forceinline__ void backIn(const float* W, const float* dOut, const float* act, float (&acc)[4][TS / 16]) {
    constexpr int SV = TS / 16, LD = TS + kPad, LDW = kH + kPad;
    const int sg = threadIdx.x & 15, kg = threadIdx.x >> 4;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int v = 0; v < SV; ++v) acc[i][v] = 0.0f;
#pragma unroll 4
    for (int j = 0; j < NO; ++j) {
        float w[4], d[SV];
        vload<4>(W + j * LDW + 4 * kg, w);
        vload<SV>(dOut + j * LD + sg * SV, d);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int v = 0; v < SV; ++v) acc[i][v] = fmaf(d[v], w[i], acc[i][v]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a[SV];
        vload<SV>(act + (4 * kg + i) * LD + sg * SV, a);
#pragma unroll
        for (int v = 0; v < SV; ++v) acc[i][v] = a[v] > 0.0f ? acc[i][v] : 0.0f;
    }
}
template <int TS>
__device__ __forceinline__ void storeIn(float* act, const float (&acc)[4][TS / 16]) {
    const int sg = threadIdx.x & 15, kg = threadIdx.x >> 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) vstore<TS / 16>(act + (4 * kg + i) * (TS + kPad) + sg * (TS / 16), acc[i]);
}

// g[i][c] += sum_s dOut[jg + 16 i][s] * in[kg + 16 c][s]; threads below 64
// also add their row of dOut to gb.
template <int TS, int C>
__device__ __forceinline__ void backW(const float* dOut, const float* in, float (&g)[4][C], float& gb) {
    constexpr int LD = TS + kPad;
    const int kg = threadIdx.x & 15, jg = threadIdx.x >> 4;
#pragma unroll 2
    for (int s = 0; s < TS; s += 4) {
        float d[4][4], a[C][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) vload<4>(dOut + (jg + 16 * i) * LD + s, d[i]);
#pragma unroll
        for (int c = 0; c < C; ++c) vload<4>(in + (kg + 16 * c) * LD + s, a[c]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int c = 0; c < C; ++c) g[i][c] = fmaf(d[i][q], a[c][q], g[i][c]);
    }
    if (threadIdx.x < kH) {
        float t = 0.0f;
#pragma unroll 4
        for (int s = 0; s < TS; s += 4) {
            float d[4];
            vload<4>(dOut + threadIdx.x * LD + s, d);
            t += (d[0] + d[1]) + (d[2] + d[3]);
        }
        gb += t;
    }
}

// Forward + backward over tiles of TS samples, a CTA's tiles gridDim.x
// apart; gradients of the mean squared error over `total` samples x 2
// outputs accumulate into `grad`.
template <int TS>
__global__ void __launch_bounds__(kThreads, 2) mlpTrainStep(const __nv_bfloat16* __restrict__ wbf,
                                                            const float* __restrict__ X, const float* __restrict__ Y,
                                                            int n, int total, double* __restrict__ grad,
                                                            double* __restrict__ loss) {
    using S = Smem<TS>;
    extern __shared__ __align__(16) unsigned char smraw[];
    S& sm = *reinterpret_cast<S*>(smraw);
    const int tid = threadIdx.x;
    loadWeights(sm, wbf);
    float g1[4][1] = {}, g2[4][4] = {}, g3[4][4] = {}, g4 = 0.0f, gb1 = 0.0f, gb2 = 0.0f, gb3 = 0.0f, gb4 = 0.0f;
    float l = 0.0f;
    const float scale = 2.0f / (float)(total * kOut);
    for (int t = blockIdx.x; t * TS < n; t += gridDim.x) {
        const int s0 = t * TS, ns = min(TS, n - s0);
        loadSamples(sm, X, s0, ns);
        __syncthreads();
        forwardTile(sm);
        if (tid < kOut * TS) {
            const int s = tid / kOut, j = tid % kOut;
            float diff = 0.0f;
            if (s < ns) diff = sm.y[j * S::LD + s] - Y[(long long)s0 * kOut + tid];
            l += diff * diff;
            sm.y[j * S::LD + s] = diff * scale;  // each thread its own element
        }
        __syncthreads();
        if (tid < kOut * kH) {  // W4 and b4
            const int j = tid / kH, k = tid % kH;
#pragma unroll 4
            for (int s = 0; s < TS; s += 4) {
                float d[4], a[4];
                vload<4>(sm.y + j * S::LD + s, d);
                vload<4>(sm.h3 + k * S::LD + s, a);
#pragma unroll
                for (int q = 0; q < 4; ++q) g4 = fmaf(d[q], a[q], g4);
            }
        } else if (tid < kOut * kH + kOut) {
            for (int s = 0; s < TS; ++s) gb4 += sm.y[(tid - kOut * kH) * S::LD + s];
        }
        float d[4][TS / 16];
        backIn<TS, kOut>(sm.w4, sm.y, sm.h3, d);
        __syncthreads();
        storeIn<TS>(sm.h3, d);  // the gradient at layer 3 replaces its activations
        __syncthreads();
        backW<TS, 4>(sm.h3, sm.h2, g3, gb3);
        backIn<TS, kH>(sm.w3, sm.h3, sm.h2, d);
        __syncthreads();
        storeIn<TS>(sm.h2, d);
        __syncthreads();
        backW<TS, 4>(sm.h2, sm.h1, g2, gb2);
        backIn<TS, kH>(sm.w2, sm.h2, sm.h1, d);
        __syncthreads();
        storeIn<TS>(sm.h1, d);
        __syncthreads();
        backW<TS, 1>(sm.h1, sm.x, g1, gb1);
        __syncthreads();
    }
    const int kg = tid & 15, jg = tid >> 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int j = jg + 16 * i;
        atomicAdd(grad + kOffW1 + j * kIn + kg, (double)g1[i][0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            atomicAdd(grad + kOffW2 + j * kH + kg + 16 * c, (double)g2[i][c]);
            atomicAdd(grad + kOffW3 + j * kH + kg + 16 * c, (double)g3[i][c]);
        }
    }
    if (tid < kH) {
        atomicAdd(grad + kOffB1 + tid, (double)gb1);
        atomicAdd(grad + kOffB2 + tid, (double)gb2);
        atomicAdd(grad + kOffB3 + tid, (double)gb3);
    }
    if (tid < kOut * kH) atomicAdd(grad + kOffW4 + tid, (double)g4);
    else if (tid < kOut * kH + kOut) atomicAdd(grad + kOffB4 + tid - kOut * kH, (double)gb4);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((tid & 31) == 0 && l != 0.0f) atomicAdd(loss, (double)(l / (float)(total * kOut)));
}

template <int TS>
__global__ void __launch_bounds__(kThreads) mlpPredict(const __nv_bfloat16* __restrict__ wbf,
                                                       const float* __restrict__ X, int n, float* __restrict__ Yout) {
    using S = Smem<TS>;
    extern __shared__ __align__(16) unsigned char smraw[];
    S& sm = *reinterpret_cast<S*>(smraw);
    const int s0 = blockIdx.x * TS, ns = min(TS, n - s0);
    loadWeights(sm, wbf);
    loadSamples(sm, X, s0, ns);
    __syncthreads();
    forwardTile(sm);
    if (threadIdx.x < kOut * ns) {
        const int s = threadIdx.x / kOut, j = threadIdx.x % kOut;
        Yout[(long long)s0 * kOut + threadIdx.x] = sm.y[j * S::LD + s];
    }
}

// Adam on the FP32 master weights; refreshes the BF16 copy; clears grads.
__global__ void adamStep(float* __restrict__ w, __nv_bfloat16* __restrict__ wbf, float* __restrict__ m,
                         float* __restrict__ v, double* __restrict__ grad, float lr, float b1, float b2, float eps,
                         float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    const float g = (float)grad[i];
    const float mi = b1 * m[i] + (1.0f - b1) * g;
    const float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    wbf[i] = __float2bfloat16_rn(wi);
    grad[i] = 0.0;
}

// The gradients and the loss as FP32; clears the sums.
__global__ void roundGrads(double* __restrict__ grad, float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > kParams) return;
    out[i] = (float)grad[i];
    grad[i] = 0.0;
}

__global__ void quantize(const float* __restrict__ w, __nv_bfloat16* __restrict__ wbf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kParams) wbf[i] = __float2bfloat16_rn(w[i]);
}

#define SZ_CHECK(call, code)                                                                        \
    do {                                                                                            \
        const cudaError_t _e = (call);                                                              \
        if (_e != cudaSuccess) {                                                                    \
            gpudb::setThreadError(std::string("sizer: ") + #call + ": " + cudaGetErrorString(_e)); \
            return code;                                                                            \
        }                                                                                           \
    } while (0)

}  // namespace

struct gpudb_sizer {
    int device = 0, numSMs = 148;
    cudaStream_t stream = nullptr;
    float *w = nullptr, *m = nullptr, *v = nullptr;
    double *grad = nullptr, *loss = nullptr;  // loss = grad + kParams
    float* rounded = nullptr;                 // pinned: gradients and loss of gpudb_sizer_grads
    float* few = nullptr;                     // pinned: X and Y of a prediction of at most kFew samples
    __nv_bfloat16* wbf = nullptr;
    float *X = nullptr, *Y = nullptr;
    int cap = 0;  // samples X/Y can hold
    long long step = 0;
};

namespace {

int ensureCapacity(gpudb_sizer* s, int n) {
    if (n <= s->cap) return GPUDB_OK;
    if (s->X) cudaFree(s->X);
    if (s->Y) cudaFree(s->Y);
    s->X = s->Y = nullptr;
    SZ_CHECK(cudaMalloc(&s->X, sizeof(float) * (size_t)n * kIn), GPUDB_E_ALLOC);
    SZ_CHECK(cudaMalloc(&s->Y, sizeof(float) * (size_t)n * kOut), GPUDB_E_ALLOC);
    s->cap = n;
    return GPUDB_OK;
}

// Tiles of 64 samples where that gives every SM one, else smaller ones: a
// training batch of 512 is work for 32 CTAs instead of 8. At most two CTAs
// per SM: further tiles add to the same registers.
template <int TS>
int launchTrainTiles(gpudb_sizer* s, const float* X, const float* Y, int n, int total) {
    const int blocks = std::min((n + TS - 1) / TS, 2 * s->numSMs);
    mlpTrainStep<TS><<<blocks, kThreads, sizeof(Smem<TS>), s->stream>>>(s->wbf, X, Y, n, total, s->grad, s->loss);
    SZ_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
    return GPUDB_OK;
}

int launchTrain(gpudb_sizer* s, const float* X, const float* Y, int n, int total) {
    if (n >= 64 * s->numSMs) return launchTrainTiles<64>(s, X, Y, n, total);
    if (n >= 32 * s->numSMs) return launchTrainTiles<32>(s, X, Y, n, total);
    return launchTrainTiles<16>(s, X, Y, n, total);
}

}  // namespace

extern "C" {

int gpudb_sizer_create(int device, uint64_t seed, gpudb_sizer** out) {
    if (!out) return GPUDB_E_INVALID;
    *out = nullptr;
    auto s = std::make_unique<gpudb_sizer>();
    s->device = device;
    SZ_CHECK(cudaSetDevice(device), GPUDB_E_NOGPU);
    SZ_CHECK(cudaDeviceGetAttribute(&s->numSMs, cudaDevAttrMultiProcessorCount, device), GPUDB_E_NOGPU);
    for (const auto& [k, bytes] : {std::pair<const void*, size_t>{(const void*)mlpTrainStep<64>, sizeof(Smem<64>)},
                                   {(const void*)mlpTrainStep<32>, sizeof(Smem<32>)},
                                   {(const void*)mlpTrainStep<16>, sizeof(Smem<16>)},
                                   {(const void*)mlpPredict<16>, sizeof(Smem<16>)},
                                   {(const void*)mlpPredict<64>, sizeof(Smem<64>)}})
        SZ_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), GPUDB_E_LAUNCH);
    SZ_CHECK(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking), GPUDB_E_CUDA);
    SZ_CHECK(cudaMalloc(&s->w, sizeof(float) * kParams), GPUDB_E_ALLOC);
    SZ_CHECK(cudaMalloc(&s->m, sizeof(float) * kParams), GPUDB_E_ALLOC);
    SZ_CHECK(cudaMalloc(&s->v, sizeof(float) * kParams), GPUDB_E_ALLOC);
    SZ_CHECK(cudaMalloc(&s->grad, sizeof(double) * (kParams + 1)), GPUDB_E_ALLOC);
    s->loss = s->grad + kParams;
    SZ_CHECK(cudaHostAlloc((void**)&s->rounded, sizeof(float) * (kParams + 1), cudaHostAllocDefault), GPUDB_E_ALLOC);
    SZ_CHECK(cudaHostAlloc((void**)&s->few, sizeof(float) * (kIn + kOut) * kFew, cudaHostAllocDefault), GPUDB_E_ALLOC);
    SZ_CHECK(cudaMalloc(&s->wbf, sizeof(__nv_bfloat16) * kParams), GPUDB_E_ALLOC);
    // He-uniform initialisation on the host (seeded), biases zero
    std::vector<float> w(kParams, 0.0f);
    std::mt19937_64 rng(seed);
    auto init = [&](int off, int fanIn, int count) {
        const float lim = std::sqrt(6.0f / (float)fanIn);
        std::uniform_real_distribution<float> u(-lim, lim);
        for (int i = 0; i < count; i++) w[off + i] = u(rng);
    };
    init(kOffW1, kIn, kH * kIn);
    init(kOffW2, kH, kH * kH);
    init(kOffW3, kH, kH * kH);
    init(kOffW4, kH, kOut * kH);
    SZ_CHECK(cudaMemcpy(s->w, w.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice), GPUDB_E_CUDA);
    SZ_CHECK(cudaMemset(s->m, 0, sizeof(float) * kParams), GPUDB_E_CUDA);
    SZ_CHECK(cudaMemset(s->v, 0, sizeof(float) * kParams), GPUDB_E_CUDA);
    SZ_CHECK(cudaMemset(s->grad, 0, sizeof(double) * (kParams + 1)), GPUDB_E_CUDA);
    quantize<<<(kParams + 255) / 256, 256, 0, s->stream>>>(s->w, s->wbf);
    SZ_CHECK(cudaStreamSynchronize(s->stream), GPUDB_E_CUDA);
    *out = s.release();
    return GPUDB_OK;
}

void gpudb_sizer_free(gpudb_sizer* s) {
    if (!s) return;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    for (void* p : {(void*)s->w, (void*)s->m, (void*)s->v, (void*)s->grad, (void*)s->wbf, (void*)s->X,
                    (void*)s->Y})
        if (p) cudaFree(p);
    for (float* p : {s->rounded, s->few})
        if (p) cudaFreeHost(p);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

int gpudb_sizer_param_count(void) { return kParams; }

int gpudb_sizer_get_params(gpudb_sizer* s, float* out) {
    if (!s || !out) return GPUDB_E_INVALID;
    cudaSetDevice(s->device);
    SZ_CHECK(cudaMemcpyAsync(out, s->w, sizeof(float) * kParams, cudaMemcpyDeviceToHost, s->stream), GPUDB_E_CUDA);
    SZ_CHECK(cudaStreamSynchronize(s->stream), GPUDB_E_CUDA);
    return GPUDB_OK;
}

int gpudb_sizer_set_params(gpudb_sizer* s, const float* in) {
    if (!s || !in) return GPUDB_E_INVALID;
    cudaSetDevice(s->device);
    SZ_CHECK(cudaMemcpyAsync(s->w, in, sizeof(float) * kParams, cudaMemcpyHostToDevice, s->stream), GPUDB_E_CUDA);
    quantize<<<(kParams + 255) / 256, 256, 0, s->stream>>>(s->w, s->wbf);
    SZ_CHECK(cudaStreamSynchronize(s->stream), GPUDB_E_CUDA);
    return GPUDB_OK;
}

int gpudb_sizer_grads(gpudb_sizer* s, const float* X, const float* Y, int n, float* grads_out, float* loss_out) {
    if (!s || !X || !Y || n <= 0 || !grads_out) return GPUDB_E_INVALID;
    cudaSetDevice(s->device);
    if (int st = ensureCapacity(s, n)) return st;
    SZ_CHECK(cudaMemcpyAsync(s->X, X, sizeof(float) * (size_t)n * kIn, cudaMemcpyHostToDevice, s->stream), GPUDB_E_CUDA);
    SZ_CHECK(cudaMemcpyAsync(s->Y, Y, sizeof(float) * (size_t)n * kOut, cudaMemcpyHostToDevice, s->stream),
             GPUDB_E_CUDA);
    SZ_CHECK(cudaMemsetAsync(s->grad, 0, sizeof(double) * (kParams + 1), s->stream), GPUDB_E_CUDA);
    if (int st = launchTrain(s, s->X, s->Y, n, n)) return st;
    roundGrads<<<kParams / 256 + 1, 256, 0, s->stream>>>(s->grad, s->rounded);
    SZ_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
    SZ_CHECK(cudaStreamSynchronize(s->stream), GPUDB_E_CUDA);
    std::copy(s->rounded, s->rounded + kParams, grads_out);
    if (loss_out) *loss_out = s->rounded[kParams];
    return GPUDB_OK;
}

int gpudb_sizer_train(gpudb_sizer* s, const float* X, const float* Y, int n, int epochs, int batch, float lr,
                      uint64_t seed, float* final_loss) {
    if (!s || !X || !Y || n <= 0 || epochs <= 0 || batch <= 0) return GPUDB_E_INVALID;
    cudaSetDevice(s->device);
    if (int st = ensureCapacity(s, n)) return st;
    // shuffle once per epoch on the host, upload the permuted set
    std::vector<int> idx(n);
    for (int i = 0; i < n; i++) idx[i] = i;
    std::mt19937_64 rng(seed);
    std::vector<float> px((size_t)n * kIn), py((size_t)n * kOut);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const long long totalSteps = (long long)epochs * ((n + batch - 1) / batch);
    long long runStep = 0;
    float last = 0.0f;
    for (int ep = 0; ep < epochs; ep++) {
        std::shuffle(idx.begin(), idx.end(), rng);
        for (int i = 0; i < n; i++) {
            std::copy(X + (size_t)idx[i] * kIn, X + (size_t)idx[i] * kIn + kIn, px.begin() + (size_t)i * kIn);
            std::copy(Y + (size_t)idx[i] * kOut, Y + (size_t)idx[i] * kOut + kOut, py.begin() + (size_t)i * kOut);
        }
        SZ_CHECK(cudaMemcpyAsync(s->X, px.data(), sizeof(float) * px.size(), cudaMemcpyHostToDevice, s->stream),
                 GPUDB_E_CUDA);
        SZ_CHECK(cudaMemcpyAsync(s->Y, py.data(), sizeof(float) * py.size(), cudaMemcpyHostToDevice, s->stream),
                 GPUDB_E_CUDA);
        SZ_CHECK(cudaMemsetAsync(s->loss, 0, sizeof(double), s->stream), GPUDB_E_CUDA);
        int nb = 0;
        for (int off = 0; off < n; off += batch, nb++) {
            const int cur = std::min(batch, n - off);
            if (int st = launchTrain(s, s->X + (size_t)off * kIn, s->Y + (size_t)off * kOut, cur, cur)) return st;
            s->step++;
            const float c1 = 1.0f - std::pow(b1, (float)s->step), c2 = 1.0f - std::pow(b2, (float)s->step);
            // cosine decay of the learning rate over this call's steps
            const float lrNow =
                totalSteps > 1 ? lr * 0.5f * (1.0f + std::cos(3.14159265358979f * (float)runStep / (float)totalSteps))
                               : lr;
            runStep++;
            adamStep<<<(kParams + 255) / 256, 256, 0, s->stream>>>(s->w, s->wbf, s->m, s->v, s->grad, lrNow, b1, b2,
                                                                    eps, c1, c2);
        }
        SZ_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
        double l = 0;
        SZ_CHECK(cudaMemcpyAsync(&l, s->loss, sizeof(double), cudaMemcpyDeviceToHost, s->stream), GPUDB_E_CUDA);
        SZ_CHECK(cudaStreamSynchronize(s->stream), GPUDB_E_CUDA);
        last = nb ? (float)(l / nb) : 0.0f;  // mean of the batches' losses
    }
    if (final_loss) *final_loss = last;
    return GPUDB_OK;
}

int gpudb_sizer_predict(gpudb_sizer* s, const float* X, int n, float* Y_out) {
    if (!s || !X || n < 0 || (n && !Y_out)) return GPUDB_E_INVALID;
    if (n == 0) return GPUDB_OK;
    cudaSetDevice(s->device);
    if (n <= kFew) {
        float *x = s->few, *y = s->few + kIn * kFew;
        std::copy(X, X + (size_t)n * kIn, x);
        mlpPredict<16><<<(n + 15) / 16, kThreads, sizeof(Smem<16>), s->stream>>>(s->wbf, x, n, y);
        SZ_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
        SZ_CHECK(cudaStreamSynchronize(s->stream), GPUDB_E_CUDA);
        std::copy(y, y + (size_t)n * kOut, Y_out);
        return GPUDB_OK;
    }
    if (int st = ensureCapacity(s, n)) return st;
    SZ_CHECK(cudaMemcpyAsync(s->X, X, sizeof(float) * (size_t)n * kIn, cudaMemcpyHostToDevice, s->stream), GPUDB_E_CUDA);
    if (n >= 64 * s->numSMs)
        mlpPredict<64><<<(n + 63) / 64, kThreads, sizeof(Smem<64>), s->stream>>>(s->wbf, s->X, n, s->Y);
    else
        mlpPredict<16><<<(n + 15) / 16, kThreads, sizeof(Smem<16>), s->stream>>>(s->wbf, s->X, n, s->Y);
    SZ_CHECK(cudaGetLastError(), GPUDB_E_LAUNCH);
    SZ_CHECK(cudaMemcpyAsync(Y_out, s->Y, sizeof(float) * (size_t)n * kOut, cudaMemcpyDeviceToHost, s->stream),
             GPUDB_E_CUDA);
    SZ_CHECK(cudaStreamSynchronize(s->stream), GPUDB_E_CUDA);
    return GPUDB_OK;
}

}  // extern "C"
