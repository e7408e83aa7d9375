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
// passes of 128 rays a CTA and all weight gradients (bh_sg_chain.cu), and Adam with
// the packing of the BF16 weights; each starts while the one before it ends (set-up, and the
// features of the next batch).  16,384 rays: 97 us (105 us as ordinary launches with a zero
// fill of the gradients between, 710 us as 36 launches).
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

// BF16 weights W_l (out x in) and their transposes (head transpose padded to 64 columns)
// from the parameters; ADAM: after this Adam step on them (one pass over both).
struct AdamStep
{
    float *g, *m, *v;
    float lr, b1, b2, eps, c1, c2;
};

template <bool ADAM>
__global__ void pack_kernel(float* __restrict__ params, __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ Wt,
                            float* __restrict__ biasPacked, AdamStep A)
{
    if constexpr (ADAM)
    {
        bhtc::launch_dependents();
        bhtc::wait_for_previous();
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= SgLayout::count()) return;
    float p = params[i];
    if constexpr (ADAM)
    {
        const float gi = A.g[i];
        A.g[i] = 0.f;
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
    take((void**)&S.dY, (size_t)n * kOutPad * 2);
    for (int l = 0; l < kHidden; ++l) take((void**)&S.dZ[l], nw * 2);
    if (e != cudaSuccess) { sg_free_batch(S); return e; }
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
    S.dY = nullptr;
    S.cap = 0;
}

// forward + loss + backward of n rays (rows of `in` and `tgt`: the first n, or with N > 0 at
// indices below N hashed with `seed`); gradients (batch mean) in S.grads, loss sums in `loss`
cudaError_t sg_gradients(SgState& S, const float* in, const float* tgt, long long N, unsigned seed, int n, float* loss,
                         bool early, cudaStream_t s)
{
    if (n <= 0 || n % 128) return cudaErrorInvalidValue;
    cudaError_t e = sg_reserve(S, n);
    if (e == cudaSuccess) e = sg_chain_train(S, in, tgt, N, seed, n, loss, early, s);
    return e == cudaSuccess ? sg_weight_grads(S, n, s) : e;
}

cudaError_t sg_adam(SgState& S, float lr, cudaStream_t s)
{
    ++S.step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f / (1.f - std::pow(b1, (float)S.step)), c2 = 1.f / (1.f - std::pow(b2, (float)S.step));
    return sg_launch(pack_kernel<true>, dim3(blocksFor(SgLayout::count(), 256)), 256, 0, true, s, S.params, S.W, S.Wt,
                     S.biasPacked, AdamStep{S.grads, S.adamM, S.adamV, lr, b1, b2, 1e-8f, c1, c2});
}
