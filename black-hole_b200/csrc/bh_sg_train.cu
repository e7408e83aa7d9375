// ---------------------------------------------------------------------------
// bh_sg_train.cu -- training of the lensing surrogate on the GPU: the
// RK4-traced ray set's features, the passes' order and scratch, and Adam.
//
// Batch of n rays, layer l = 0..3 hidden, 4 = head:
//   X0 = features(inputs)                          BF16 n x 256
//   Z_l = X_l W_l^T + b_l,  X_{l+1} = gelu(Z_l)     FP32 / BF16
//   Y = X4 Wh^T + bh                               FP32 n x 16
//   dY = d loss / dY (batch mean)                  BF16 n x 64 (cols >= 16 zero)
//   dW_l = dZ_l^T X_l,  db_l = sum_rows dZ_l,  dX_l = dZ_l W_l
//   dZ_l = dX_{l+1} * gelu'(Z_l)
// dX_l reads W_l^T, kept next to W_l after every update.  A step is three launches: the
// passes of 128 rays a CTA and the parts of all gradients (bh_sg_chain.cu), and Adam, which adds
// the parts, with the packing of the BF16 weights; each starts while the one before it ends
// (set-up, and the features of the next batch).  16,384 rays: 103 us (97 us with sums in an order that changed from
// run to run; 710 us as 36 launches).
// No counterpart in the reference (it has no learned component).
// ---------------------------------------------------------------------------
#include <cmath>
#include <cuda_bf16.h>
#include "bh_integrate.cuh"
#include "bh_launch.h"
#include "bh_sg_net.cuh"
#include "bh_sg_train.h"
#include "bh_surrogate.h"
#include "bh_tc.cuh"

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

// What a parameter's thread does: pack it (BF16 weights W_l (out x in), their transposes, the head's
// padded to 64 columns, and the biases), after an Adam step with the sum of its parts, or only that sum.
enum { PACK, ADAM, SUM };
struct StepArgs
{
    const float* parts;           // nParts x kSgPart
    int nParts;
    float *g, *m, *v, *loss;
    float lr, b1, b2, eps, c1, c2;
};

// Groups of four parameters (`at`, at + step, ...) in the parts' order (weight_grad_kernel): tiles of 128
// weight rows as [column / 4][row] (the head's as [output / 4][input]), then the layer's biases.
struct SgQuad
{
    int l, at, step;
    bool weight;
};

__device__ __forceinline__ SgQuad sg_quad(int q)
{
    const int l = min(q / (SgLayout::kHid / 4), kHidden), j = q - l * (SgLayout::kHid / 4);
    const int out = l < kHidden ? kWidth : kOut, tile = l < kHidden ? 128 * kWidth / 4 : 128 * kOut / 4;
    if (j >= out * kWidth / 4) return SgQuad{l, 4 * q, 1, false};
    const int row = j / tile * 128 + j % 128, c = j % tile / 128 * 4;
    return l < kHidden ? SgQuad{l, SgLayout::w(l) + row * kWidth + c, 1, true}
                       : SgQuad{l, SgLayout::w(l) + c * kWidth + row, kWidth, true};
}

// A CTA takes 32 groups: warp w adds the parts w, w + 4, ..., then takes the groups' parameters w.
// Bound: latency, and the parts, read from L2 (15 MB): 15 us from DRAM (22 us with
// a part per share, 34 us with a thread a group).
template <int WHAT>
__global__ void __launch_bounds__(128)
pack_kernel(float* __restrict__ params, __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ Wt,
            float* __restrict__ biasPacked, StepArgs A)
{
    __shared__ double sums[WHAT == PACK ? 1 : 4][4][32];
    if constexpr (WHAT == ADAM)
    {
        bhtc::launch_dependents();
        bhtc::wait_for_previous();
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, q = blockIdx.x * 32 + lane;
    const bool any = q < (WHAT == PACK ? SgLayout::count() : kSgPart) / 4, isLoss = q >= SgLayout::count() / 4;
    const SgQuad Q = sg_quad(isLoss ? 0 : q);
    const int i = Q.at + w * Q.step;
    float g = 0.f, p = 0.f, m = 0.f, v = 0.f;
    if (WHAT != SUM && any && !isLoss) p = params[i];
    if (WHAT == ADAM && any && !isLoss) { m = A.m[i]; v = A.v[i]; }
    if constexpr (WHAT != PACK)
    {   // in FP64: rounded once
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        if (any)
        {
            const float4* from = reinterpret_cast<const float4*>(A.parts) + q;
#pragma unroll 4
            for (int k = w; k < A.nParts; k += 4)
            {
                const float4 t = from[(size_t)k * (kSgPart / 4)];
                s[0] += t.x; s[1] += t.y; s[2] += t.z; s[3] += t.w;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) sums[w][k][lane] = s[k];
        __syncthreads();
        g = (float)((sums[0][w][lane] + sums[1][w][lane]) + (sums[2][w][lane] + sums[3][w][lane]));
    }
    if (!any) return;
    if (isLoss)
    {
        A.loss[4 * q - SgLayout::count() + w] = g;
        return;
    }
    if constexpr (WHAT == SUM) A.g[i] = g;
    else
    {
        if constexpr (WHAT == ADAM)
        {
            const float mi = A.b1 * m + (1.f - A.b1) * g, vi = A.b2 * v + (1.f - A.b2) * g * g;
            A.m[i] = mi;
            A.v[i] = vi;
            p -= A.lr * (mi * A.c1) / (sqrtf(vi * A.c2) + A.eps);
            params[i] = p;
        }
        const int j = i - SgLayout::w(Q.l);
        if (Q.weight)
        {
            const __nv_bfloat16 h = __float2bfloat16_rn(p);
            W[(size_t)Q.l * kWidth * kWidth + j] = h;
            // the head's transpose is padded to 64 columns, which stay zero
            Wt[(size_t)Q.l * kWidth * kWidth + j % kWidth * (Q.l < kHidden ? kWidth : kOutPad) + j / kWidth] = h;
        }
        else biasPacked[Q.l * kWidth + j - (Q.l < kHidden ? kWidth : kOut) * kWidth] = p;
    }
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
    pack_kernel<PACK><<<blocksFor(SgLayout::count() / 4, 32), 128, 0, s>>>(S.params, S.W, S.Wt, S.biasPacked, StepArgs{});
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
    // dY, the slices and the parts in one allocation (each costs the first step some 0.3 ms)
    const size_t dyBytes = (size_t)n * kOutPad * 2, sliceBytes = (size_t)(n / 128) * kSgSlice * 4;
    take((void**)&S.dY, dyBytes + sliceBytes + (size_t)sg_parts(n / 128) * kSgPart * 4);
    for (int l = 0; l < kHidden; ++l) take((void**)&S.dZ[l], nw * 2);
    if (e != cudaSuccess) { sg_free_batch(S); return e; }
    S.slices = reinterpret_cast<float*>(static_cast<uint8_t*>(S.dY) + dyBytes);
    S.parts = reinterpret_cast<float*>(static_cast<uint8_t*>(S.dY) + dyBytes + sliceBytes);
    S.cap = n;
    return cudaSuccess;
}

void sg_free_batch(SgState& S)
{
    void* ps[] = {S.X[0], S.X[1], S.X[2], S.X[3], S.X[4], S.Z[0], S.Z[1], S.Z[2], S.Z[3], S.dY, S.dZ[0],
                  S.dZ[1], S.dZ[2], S.dZ[3]};
    for (void* p : ps)
        if (p) cudaFree(p);
    for (int l = 0; l <= kHidden; ++l) S.X[l] = nullptr;
    for (int l = 0; l < kHidden; ++l) { S.Z[l] = nullptr; S.dZ[l] = nullptr; }
    S.dY = nullptr; S.slices = nullptr; S.parts = nullptr;
    S.cap = 0;
}

cudaError_t sg_backward(SgState& S, const float* in, const float* tgt, long long N, unsigned seed, int n, bool early,
                        cudaStream_t s)
{
    if (n <= 0 || n % 128) return cudaErrorInvalidValue;
    cudaError_t e = sg_reserve(S, n);
    if (e == cudaSuccess) e = sg_chain_train(S, in, tgt, N, seed, n, early, s);
    return e == cudaSuccess ? sg_weight_grads(S, n, s) : e;
}

cudaError_t sg_gradients(SgState& S, int n, float* loss, cudaStream_t s)
{
    StepArgs A{};
    A.parts = S.parts; A.nParts = sg_parts(n / 128);
    A.g = S.grads; A.loss = loss;
    return sg_launch(pack_kernel<SUM>, dim3(blocksFor(kSgPart / 4, 32)), 128, 0, false, s, S.params, S.W, S.Wt,
                     S.biasPacked, A);
}

cudaError_t sg_adam(SgState& S, int n, float lr, float* loss, cudaStream_t s)
{
    ++S.step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f / (1.f - std::pow(b1, (float)S.step)), c2 = 1.f / (1.f - std::pow(b2, (float)S.step));
    return sg_launch(pack_kernel<ADAM>, dim3(blocksFor(kSgPart / 4, 32)), 128, 0, true, s, S.params, S.W, S.Wt,
                     S.biasPacked,
                     StepArgs{S.parts, sg_parts(n / 128), nullptr, S.adamM, S.adamV, loss, lr, b1, b2, 1e-8f, c1, c2});
}
