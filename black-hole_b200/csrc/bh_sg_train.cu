// ---------------------------------------------------------------------------
// bh_sg_train.cu -- training of the lensing surrogate on the GPU: the
// RK4-traced ray set, the forward and backward passes (tensor-core kernels of
// bh_sg_layer.cu, the head's GEMM of bh_gemm.cu, the loss below) and Adam.
//
// Batch of n rays, layer l = 0..3 hidden, 4 = head:
//   X0 = features(inputs)                          BF16 n x 256
//   Z_l = X_l W_l^T + b_l,  X_{l+1} = gelu(Z_l)     FP32 / BF16
//   Y = X4 Wh^T + bh                               FP32 n x 16
//   dY = d loss / dY (batch mean)                  BF16 n x 64 (cols >= 16 zero)
//   dW_l = dZ_l^T X_l,  db_l = sum_rows dZ_l,  dX_l = dZ_l W_l
//   dZ_l = dX_{l+1} * gelu'(Z_l)
// dX_l reads W_l^T, kept next to W_l after every update.  16,384 rows: 13 launches,
// 162 us a step (36 launches, 710 us, with the activations, transposes and one weight
// gradient a layer as launches of their own).
// No counterpart in the reference (it has no learned component).
// ---------------------------------------------------------------------------
#include <cmath>
#include <cuda_bf16.h>
#include "bh_integrate.cuh"
#include "bh_launch.h"
#include "bh_sg_net.cuh"
#include "bh_sg_train.h"
#include "bh_surrogate.h"

using namespace bhsg;

namespace {

// ---- element-wise kernels -------------------------------------------------------

__global__ void feat_kernel(const float* __restrict__ in, uint4* __restrict__ X, int n)
{
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)n * 32) return;
    const long long row = t >> 5;
    float x[kIn];
#pragma unroll
    for (int k = 0; k < kIn; ++k) x[k] = __ldg(in + row * 8 + k);
    X[t] = sg_feature_chunk(x, (int)(t & 31));
}

struct LossWeights
{
    float esc, diskR, diskG, conf, escTol;
};

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Per-ray loss terms and dY (scaled by 1/n); loss[0..4] += CE, escape, disk r,
// disk g, confidence (sums); dbh += column sums of dY.
__global__ void loss_kernel(const float* __restrict__ Y, const float* __restrict__ in, const float* __restrict__ tgt,
                            __nv_bfloat16* __restrict__ dY, float* __restrict__ dbh, float* __restrict__ loss, int n,
                            LossWeights w)
{
    const int row = blockIdx.x * blockDim.x + threadIdx.x;
    float g[kOut], l[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    const float4* Y4 = reinterpret_cast<const float4*>(Y);
#pragma unroll
    for (int k = 0; k < kOut; ++k) g[k] = 0.f;
    if (row < n)
    {
        float y[kOut];
#pragma unroll
        for (int k = 0; k < kOut / 4; ++k)
        {
            const float4 v = Y4[(size_t)row * (kOut / 4) + k];
            y[4 * k] = v.x; y[4 * k + 1] = v.y; y[4 * k + 2] = v.z; y[4 * k + 3] = v.w;
        }
        const float *t = tgt + (size_t)row * 8, *x = in + (size_t)row * 8;   // the caller's, of any alignment
        const int cls = (int)t[0];
        const float m = fmaxf(y[0], fmaxf(y[1], y[2]));
        const float e0 = expf(y[0] - m), e1 = expf(y[1] - m), e2 = expf(y[2] - m), se = e0 + e1 + e2;
        const float p[3] = {e0 / se, e1 / se, e2 / se};
        l[0] = -logf(fmaxf(p[cls], 1e-30f));
        for (int k = 0; k < 3; ++k) g[k] = p[k] - (k == cls ? 1.f : 0.f);
        float errE = 0.f;
        if (cls == kClsEscaped)
        {
            float r[3];
            for (int k = 0; k < 3; ++k) r[k] = x[k] + y[kOEsc + k] - t[1 + k];
            errE = sqrtf(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
            l[1] = w.esc * errE * errE;
            for (int k = 0; k < 3; ++k) g[kOEsc + k] = 2.f * w.esc * r[k];
        }
        if (t[6] > 0.5f)
        {
            const float dr = y[kODiskR] - t[4], dg = y[kODiskG] - t[5];
            l[2] = w.diskR * dr * dr;
            l[3] = w.diskG * dg * dg;
            g[kODiskR] = 2.f * w.diskR * dr;
            g[kODiskG] = 2.f * w.diskG * dg;
        }
        const int pred = (p[0] >= p[1] && p[0] >= p[2]) ? 0 : (p[1] >= p[2] ? 1 : 2);
        const float good = (pred == cls && (cls != kClsEscaped || errE < w.escTol)) ? 1.f : 0.f;
        const float s = 1.f / (1.f + expf(-y[kOConf]));
        l[4] = -w.conf * (good * logf(fmaxf(s, 1e-30f)) + (1.f - good) * logf(fmaxf(1.f - s, 1e-30f)));
        g[kOConf] = w.conf * (s - good);
        const float inv = 1.f / (float)n;
        uint4* d = reinterpret_cast<uint4*>(dY + (size_t)row * kOutPad);
        __nv_bfloat162 h[kOut / 2];
#pragma unroll
        for (int k = 0; k < kOut; k += 2)
        {
            g[k] *= inv;
            g[k + 1] *= inv;
            h[k / 2] = __floats2bfloat162_rn(g[k], g[k + 1]);
        }
        const uint32_t* b = reinterpret_cast<const uint32_t*>(h);
        d[0] = make_uint4(b[0], b[1], b[2], b[3]);
        d[1] = make_uint4(b[4], b[5], b[6], b[7]);
#pragma unroll
        for (int k = 2; k < kOutPad / 8; ++k) d[k] = make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < kOut; ++k)
    {
        const float s = warp_sum(g[k]);
        if ((threadIdx.x & 31) == 0 && s != 0.f) atomicAdd(dbh + k, s);
    }
#pragma unroll
    for (int k = 0; k < 5; ++k)
    {
        const float s = warp_sum(l[k]);
        if ((threadIdx.x & 31) == 0 && s != 0.f) atomicAdd(loss + k, s);
    }
}

// BF16 weights W_l (out x in) and their transposes (head transpose padded to 64 columns)
// from the parameters; ADAM: after this Adam step on them (one pass over both).
struct AdamStep
{
    const float* g;
    float *m, *v;
    float lr, b1, b2, eps, c1, c2;
};

template <bool ADAM>
__global__ void pack_kernel(float* __restrict__ params, __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ Wt,
                            float* __restrict__ biasPacked, AdamStep A)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= SgLayout::count()) return;
    float p = params[i];
    if constexpr (ADAM)
    {
        const float gi = A.g[i];
        const float mi = A.b1 * A.m[i] + (1.f - A.b1) * gi, vi = A.b2 * A.v[i] + (1.f - A.b2) * gi * gi;
        A.m[i] = mi;
        A.v[i] = vi;
        p -= A.lr * (mi * A.c1) / (sqrtf(vi * A.c2) + A.eps);
        params[i] = p;
    }
    const int l = min(i / SgLayout::kHid, kHidden), j = i - SgLayout::w(l);
    const int out = l < kHidden ? kWidth : kOut;
    if (j < out * kWidth)
    {
        const int r = j / kWidth, c = j % kWidth;
        const __nv_bfloat16 h = __float2bfloat16_rn(p);
        W[(size_t)l * kWidth * kWidth + j] = h;
        // the head's transpose is padded to 64 columns, which stay zero
        Wt[(size_t)l * kWidth * kWidth + c * (l < kHidden ? kWidth : kOutPad) + r] = h;
    }
    else biasPacked[l * kWidth + j - out * kWidth] = p;
}

// batch rows gathered from the ray set at hashed indices, with their features: 32 threads a row
__global__ void gather_kernel(const float4* __restrict__ dsIn, const float4* __restrict__ dsTgt, long long N,
                              unsigned seed, float4* __restrict__ in, float4* __restrict__ tgt, uint4* __restrict__ X,
                              int n)
{
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int k = (int)(t >> 5), j = (int)(t & 31);
    if (k >= n) return;
    unsigned h = (unsigned)k * 0x9E3779B1u ^ seed;
    h ^= h >> 16; h *= 0x7feb352du; h ^= h >> 15; h *= 0x846ca68bu; h ^= h >> 16;
    unsigned h2 = h * 0x2C1B3C6Du + 0x297A2D39u;
    h2 ^= h2 >> 15;
    const long long idx = (long long)((((unsigned long long)h << 32) | h2) % (unsigned long long)N);
    const float4 a = __ldg(dsIn + 2 * idx), b = __ldg(dsIn + 2 * idx + 1);
    const float x[kIn] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z};
    X[t] = sg_feature_chunk(x, j);
    if (j == 0) in[2 * k] = a;
    else if (j == 1) in[2 * k + 1] = b;
    else if (j == 2) tgt[2 * k] = __ldg(dsTgt + 2 * idx);
    else if (j == 3) tgt[2 * k + 1] = __ldg(dsTgt + 2 * idx + 1);
}

inline unsigned blocksFor(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
cudaError_t sg_features(const float* in, void* X0, int n, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    feat_kernel<<<blocksFor((long long)n * 32, 256), 256, 0, s>>>(in, reinterpret_cast<uint4*>(X0), n);
    return cudaGetLastError();
}

cudaError_t sg_pack_weights(SgState& S, cudaStream_t s)
{
    const int count = SgLayout::count();
    pack_kernel<false><<<blocksFor(count, 256), 256, 0, s>>>(S.params, S.W, S.Wt, S.biasPacked, AdamStep{});
    return cudaGetLastError();
}

cudaError_t sg_reserve(SgState& S, int n)
{
    if (n <= S.cap) return cudaSuccess;
    sg_free_batch(S);
    const size_t nw = (size_t)n * kWidth;
    cudaError_t e = cudaSuccess;
    auto take = [&](void** p, size_t bytes) { if (e == cudaSuccess) e = bh_device_alloc(reinterpret_cast<void**>(p), bytes); };
    for (int l = 0; l <= kHidden; ++l) take((void**)&S.X[l], nw * 2);
    for (int l = 0; l < kHidden; ++l) take((void**)&S.Z[l], (size_t)((n + 127) / 128) * 128 * kWidth * 4);
    take((void**)&S.Y, (size_t)n * kOut * 4);
    take((void**)&S.dY, (size_t)n * kOutPad * 2);
    for (int l = 0; l < kHidden; ++l) take((void**)&S.dZ[l], nw * 2);
    if (e != cudaSuccess) { sg_free_batch(S); return e; }
    S.cap = n;
    return cudaSuccess;
}

void sg_free_batch(SgState& S)
{
    void* ps[] = {S.X[0], S.X[1], S.X[2], S.X[3], S.X[4], S.Z[0], S.Z[1], S.Z[2], S.Z[3], S.Y, S.dY, S.dZ[0],
                  S.dZ[1], S.dZ[2], S.dZ[3]};
    for (void* p : ps)
        if (p) cudaFree(p);
    for (int l = 0; l <= kHidden; ++l) S.X[l] = nullptr;
    for (int l = 0; l < kHidden; ++l) { S.Z[l] = nullptr; S.dZ[l] = nullptr; }
    S.Y = nullptr; S.dY = nullptr;
    S.cap = 0;
}

// forward pass in the training form: Y = net(in)
cudaError_t sg_forward_train(SgState& S, const float* in, int n, bool haveFeatures, cudaStream_t s)
{
    cudaError_t e = sg_reserve(S, n);
    if (e == cudaSuccess && !haveFeatures) e = sg_features(in, S.X[0], n, s);
    for (int l = 0; l < kHidden && e == cudaSuccess; ++l) e = sg_layer_forward(S, l, n, s);
    if (e == cudaSuccess)
        e = bh_gemm_bf16(S.X[kHidden], kWidth, S.W + (size_t)kHidden * kWidth * kWidth, kWidth, S.Y, kOut, n, kOut,
                         kWidth, 1, false, S.params + SgLayout::b(kHidden), S.err, s);
    return e;
}

// forward + loss + backward; gradients (batch mean) in S.grads, loss sums in `loss`
cudaError_t sg_gradients(SgState& S, const float* in, const float* tgt, int n, float* loss, bool haveFeatures,
                         cudaStream_t s)
{
    if (n <= 0 || n % 128) return cudaErrorInvalidValue;
    cudaError_t e = sg_forward_train(S, in, n, haveFeatures, s);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(S.grads, 0, SgLayout::count() * sizeof(float), s)) != cudaSuccess) return e;
    LossWeights w{S.wEsc, S.wDiskR, S.wDiskG, S.wConf, S.escTol};
    loss_kernel<<<blocksFor(n, 128), 128, 0, s>>>(S.Y, in, tgt, reinterpret_cast<__nv_bfloat16*>(S.dY),
                                                  S.grads + SgLayout::b(kHidden), loss, n, w);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    for (int l = kHidden - 1; l >= 0 && e == cudaSuccess; --l) e = sg_layer_backward(S, l, n, s);
    return e == cudaSuccess ? sg_weight_grads(S, n, s) : e;
}

cudaError_t sg_adam(SgState& S, float lr, cudaStream_t s)
{
    ++S.step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f / (1.f - std::pow(b1, (float)S.step)), c2 = 1.f / (1.f - std::pow(b2, (float)S.step));
    pack_kernel<true><<<blocksFor(SgLayout::count(), 256), 256, 0, s>>>(
        S.params, S.W, S.Wt, S.biasPacked, AdamStep{S.grads, S.adamM, S.adamV, lr, b1, b2, 1e-8f, c1, c2});
    return cudaGetLastError();
}

cudaError_t sg_gather(SgState& S, unsigned seed, float* in, float* tgt, int n, cudaStream_t s)
{
    if (S.dsN <= 0) return cudaErrorInvalidValue;
    const cudaError_t e = sg_reserve(S, n);
    if (e != cudaSuccess) return e;
    gather_kernel<<<blocksFor((long long)n * 32, 256), 256, 0, s>>>(
        reinterpret_cast<const float4*>(S.dsIn), reinterpret_cast<const float4*>(S.dsTgt), S.dsN, seed,
        reinterpret_cast<float4*>(in), reinterpret_cast<float4*>(tgt), reinterpret_cast<uint4*>(S.X[0]), n);
    return cudaGetLastError();
}
