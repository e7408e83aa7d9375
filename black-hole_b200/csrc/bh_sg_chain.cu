// ---------------------------------------------------------------------------
// bh_sg_chain.cu -- the surrogate's training passes on the tensor cores (tcgen05 + TMA):
//
//   chain_kernel        features, four layers, head (and loss, and the way back):
//                       Z_l = X_l W_l^T + b_l,  X_{l+1} = gelu(Z_l),  Y = X_4 Wh^T + bh,
//                       dY,  dZ_l = (dZ_{l+1} W_{l+1}) * gelu'(Z_l),  db_l
//   weight_grad_kernel  dW_l = dZ_l^T X_l of every layer and the head
//
// All sums over the batch are added in a fixed order (bh_sg_train.h), so a step repeats bit for bit.
//
// chain_kernel: a ray's passes need no other ray, so one CTA takes 128 rays all the way.
// Its 128 x 256 BF16 operand stays in shared memory and each layer's result takes its place
// (and leaves by TMA for the weight gradients); the next layer's 128 KB of weights are
// fetched as soon as the products before are done, under the epilogue.  Sixteen warps read
// the accumulator back (one row a thread, a quarter of the columns a warp).  Z is kept as
// [column / 4][row], which a warp writes and reads in 512-byte runs; the thread that wrote it
// reads it and forms gelu' from it under the products.  Bound: the chain of nine products
// (2048 cycles a layer, 3700 with its stores) and epilogues (5400 to 6600 forward, with 128 KB
// of Z a layer and SM to write) on 128 of the 148 SMs.  16,384 rays: 78 us; with a launch a
// layer, gather, head and loss 9.4 + 4 x 11.3 + 8 + 10 + 4 x 15.4 us; with a GEMM, an activation
// and their transposes as launches 3.7 + 4.3 + 4 x 51 + 8 + 19 + 4 x 52 us.
//
// weight_grad_kernel: the contraction runs over the rows of the batch, so both
// operands are read as they lie, with the contraction index as the outer one
// (MN-major descriptors), instead of through transposed copies.  One launch for
// all five products: a CTA takes one 128-row tile of one product over one part of the
// batch, an accumulator per share of it.  An accumulator's error grows with its rows (against FP64 over the
// same BF16 operands 5.0e-7 to 5.6e-7 with shares of 512, 1.1e-6 to 1.3e-6 with 14 of 1,170).  16,384 rows:
// 21.3 us (24.4 us with the shares added to the part in L2; 20.7 us with those 14, added by reductions in an
// order that changed from run to run; 26.6 + 4 x 31 us a product at a time, and ten transposes of 12.4).
// ---------------------------------------------------------------------------
#include <cuda.h>
#include <cuda_bf16.h>
#include "bh_sg_net.cuh"
#include "bh_sg_train.h"
#include "bh_surrogate.h"
#include "bh_tc.cuh"

using namespace bhtc;
using namespace bhsg;

namespace {

constexpr uint32_t kABlock = 128u * 128u;        // 128 rows x 64 BF16
constexpr uint32_t kBBlock = 256u * 128u;        // 256 rows x 64 BF16
constexpr uint32_t kChainSmem = 4u * (kABlock + kBBlock) + 1024u;
constexpr int kChainThreads = 512;
constexpr int kChainCols = kWidth / (kChainThreads / 128);   // accumulator columns a warp reads back
constexpr int kForwardSteps = kHidden + 1, kTrainSteps = 2 * kHidden + 1;

__device__ __forceinline__ uint32_t bits(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }

// Column sums over the warp's 32 rows of v[0..31] (one row a lane): lane j gets column j's.
__device__ __forceinline__ float column_sum(float* v)
{
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
    {
        const bool up = (lane & (unsigned)o) != 0u;
#pragma unroll
        for (int i = 0; i < o; ++i)
        {
            const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0];
}

struct ChainMaps
{
    CUtensorMap W, Wh, Wt, Wht;                  // weights: layers, head; transposed
    CUtensorMap X[kLayers], dY, dZ[kHidden];     // results
};

struct ChainArgs
{
    const float *in, *tgt;        // 8 floats a ray
    long long N;                  // > 0: ray k is row hash(k, seed) of N; 0: row k
    unsigned seed;
    const float* params;
    float4* Z[kHidden];           // 128-row tiles of [column / 4][row]
    float *slices, *Y;
    float wEsc, wDiskR, wDiskG, wConf, escTol;
    int n;
    unsigned* err;
};

// row of the ray set that ray k of the batch takes
__device__ __forceinline__ long long chain_row(const ChainArgs& A, int k)
{
    if (A.N <= 0) return k;
    unsigned h = (unsigned)k * 0x9E3779B1u ^ A.seed;
    h ^= h >> 16; h *= 0x7feb352du; h ^= h >> 15; h *= 0x846ca68bu; h ^= h >> 16;
    unsigned h2 = h * 0x2C1B3C6Du + 0x297A2D39u;
    h2 ^= h2 >> 15;
    return (long long)((((unsigned long long)h << 32) | h2) % (unsigned long long)A.N);
}

// chunk j (8 BF16) of operand row r: 64-column blocks as a copy would lay them out
__device__ __forceinline__ void st_operand(uint8_t* tile, uint32_t r, uint32_t j, uint4 v)
{
    *reinterpret_cast<uint4*>(tile + (j >> 3) * kABlock + (r >> 3) * 1024u + (r & 7u) * 128u + (((j & 7u) ^ (r & 7u)) << 4)) = v;
}

template <int J0>
__device__ __forceinline__ void st_features(uint8_t* tile, uint32_t r, const float* x)
{
#pragma unroll
    for (int j = J0; j < J0 + 8; ++j) st_operand(tile, r, (uint32_t)j, sg_feature_chunk(x, j));
}

// Loss terms of one ray from its outputs y; its dY (times 1/n) to row r of the operand.
// Returns a warp sum a lane: 0..15 the columns of dY, then CE, escape, disk r, disk g, confidence.
__device__ __forceinline__ float chain_loss(const ChainArgs& A, const float* y, const float* x, const float* t,
                                            uint8_t* tile, uint32_t r)
{
    float g[kOut], l[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < kOut; ++k) g[k] = 0.f;
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
        l[1] = A.wEsc * errE * errE;
        for (int k = 0; k < 3; ++k) g[kOEsc + k] = 2.f * A.wEsc * r[k];
    }
    if (t[6] > 0.5f)
    {
        const float dr = y[kODiskR] - t[4], dg = y[kODiskG] - t[5];
        l[2] = A.wDiskR * dr * dr;
        l[3] = A.wDiskG * dg * dg;
        g[kODiskR] = 2.f * A.wDiskR * dr;
        g[kODiskG] = 2.f * A.wDiskG * dg;
    }
    const int pred = (p[0] >= p[1] && p[0] >= p[2]) ? 0 : (p[1] >= p[2] ? 1 : 2);
    const float good = (pred == cls && (cls != kClsEscaped || errE < A.escTol)) ? 1.f : 0.f;
    const float s = 1.f / (1.f + expf(-y[kOConf]));
    l[4] = -A.wConf * (good * logf(fmaxf(s, 1e-30f)) + (1.f - good) * logf(fmaxf(1.f - s, 1e-30f)));
    g[kOConf] = A.wConf * (s - good);
    const float inv = 1.f / (float)A.n;
    uint32_t h[kOut / 2];
#pragma unroll
    for (int k = 0; k < kOut; k += 2)
    {
        g[k] *= inv;
        g[k + 1] *= inv;
        h[k / 2] = bits(__floats2bfloat162_rn(g[k], g[k + 1]));
    }
    st_operand(tile, r, 0, make_uint4(h[0], h[1], h[2], h[3]));
    st_operand(tile, r, 1, make_uint4(h[4], h[5], h[6], h[7]));
#pragma unroll
    for (uint32_t k = 2; k < kOutPad / 8; ++k) st_operand(tile, r, k, make_uint4(0u, 0u, 0u, 0u));
    // lane j < 16: column j of dY; then the loss terms
    float v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = k < kOut ? g[k] : k < kOut + 5 ? l[k - kOut] : 0.f;
    return column_sum(v);
}

// 64-column blocks of step s's contraction, and the phase of block kb's barrier in it
// (blocks 1 .. 3 have none in the head's one-block gradient)
__device__ __forceinline__ int chain_blocks(int s) { return s == kHidden + 1 ? 1 : 4; }
__device__ __forceinline__ uint32_t chain_phase(int s, int kb)
{
    return (uint32_t)(kb > 0 && s > kHidden + 1 ? s - 1 : s) & 1u;
}

// step s's weights are in shared memory
__device__ __forceinline__ bool chain_landed(int s, uint64_t* full, unsigned* err)
{
    bool all = true;
    for (int kb = 0; kb < chain_blocks(s) && all; ++kb) all = mbar_wait(&full[kb], chain_phase(s, kb), err);
    return all;
}

__device__ __forceinline__ void chain_load(const ChainMaps& M, int s, uint8_t* w, uint64_t* full)
{
    const CUtensorMap* m = s < kHidden ? &M.W : s == kHidden ? &M.Wh : s == kHidden + 1 ? &M.Wht : &M.Wt;
    // step 4 + k reads the transposed weights of layer 5 - k
    const int row = s < kHidden ? s * kWidth : s > kHidden + 1 ? (2 * kHidden + 1 - s) * kWidth : 0;
    for (int kb = 0; kb < chain_blocks(s); ++kb)
    {
        mbar_expect_tx(&full[kb], s == kHidden ? kOut * 128u : kBBlock);
        tma_load_2d(w + kb * kBBlock, m, &full[kb], kb * 64, row);
    }
}

template <bool TRAIN>
__global__ void __launch_bounds__(kChainThreads, 1)
chain_kernel(const __grid_constant__ ChainMaps M, const __grid_constant__ ChainArgs A)
{
    extern __shared__ uint8_t smemRaw[];
    __shared__ uint64_t full[4], done;
    __shared__ uint32_t tmemSlot;
    // sSum: sums over a warp's 32 rows of dZ_l, dY and the loss terms, a row of them per 32 rays
    __shared__ float sBias[kHidden * kWidth + kOut], sSum[TRAIN ? 4 : 1][TRAIN ? kSgSlice : 1];
    uint8_t* tile = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    uint8_t* weights = tile + 4u * kABlock;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * 128;
    constexpr int kSteps = TRAIN ? kTrainSteps : kForwardSteps;

    if (threadIdx.x == 0)
    {
        for (int k = 0; k < 4; ++k) mbar_init(&full[k], 1);
        mbar_init(&done, 1);
        fence_barrier_init();
    }
    __syncwarp();
    if (TRAIN) launch_dependents();
    if (warp == 0) tmem_alloc(&tmemSlot, 512);

    // warp w: rows 32 (w % 4) .., columns kChainCols (w / 4) ..
    const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * kChainCols;
    const bool valid = m0 + r < A.n;
    const long long row = valid ? chain_row(A, m0 + r) : 0;
    {
        float x[kIn];
#pragma unroll
        for (int k = 0; k < kIn; ++k) x[k] = valid ? __ldg(A.in + row * 8 + k) : 0.f;
        switch (warp >> 2)
        {
            case 0: st_features<0>(tile, (uint32_t)r, x); break;
            case 1: st_features<8>(tile, (uint32_t)r, x); break;
            case 2: st_features<16>(tile, (uint32_t)r, x); break;
            default: st_features<24>(tile, (uint32_t)r, x); break;
        }
    }
    // so far nothing of the step before: its weights, gradients and buffers from here on
    if (TRAIN) wait_for_previous();
    if (threadIdx.x == 0) chain_load(M, 0, weights, full);
    for (int i = threadIdx.x; i < kHidden * kWidth + kOut; i += kChainThreads)
    {
        const int l = min(i / kWidth, kHidden);
        sBias[i] = A.params[SgLayout::b(l) + i - l * kWidth];
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmemSlot;
    const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const size_t zAt = (size_t)blockIdx.x * (128 * kWidth / 4) + (c0 / 4) * 128 + r;

    bool ok = true, fine = true;
    int loaded = 0;                              // the last step whose weights are on their way
#pragma unroll 1
    for (int s = 0; s < kSteps && ok; ++s)
    {   // the operand of step s is in `tile`; its weights are on their way
        const int blocks = chain_blocks(s);
        if (threadIdx.x == 32)
        {
            if (TRAIN)
            {   // the operand as the weight gradients read it
                const CUtensorMap* m = s <= kHidden ? &M.X[s] : s == kHidden + 1 ? &M.dY : &M.dZ[2 * kHidden + 1 - s];
                for (int kb = 0; kb < blocks; ++kb) tma_store_2d(m, tile + kb * kABlock, kb * 64, m0);
                tma_store_commit();
            }
            const uint32_t idesc = s == kHidden ? idesc_bf16_f32(kOut) : idesc_bf16_f32(kWidth);
            for (int kb = 0; kb < blocks; ++kb)
            {
                if (!(fine = mbar_wait(&full[kb], chain_phase(s, kb), A.err))) break;
                tc_fence_after();
                const uint32_t sa = smem_u32(tile + kb * kABlock), sb = smem_u32(weights + kb * kBBlock);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    mma_bf16(tmem + (s == kHidden ? kWidth : 0), sdesc_sw128(sa + j * 32), sdesc_sw128(sb + j * 32),
                             idesc, kb > 0 || j > 0);
            }
            if (TRAIN) tma_store_wait_read();    // the epilogue writes over the operand
            mma_commit(&done);
        }
        __syncwarp();
        float4 zin[TRAIN ? kChainCols / 4 : 1];
        const int back = 2 * kHidden - s;        // s > kHidden: the layer whose dZ this step makes
        if (TRAIN && s > kHidden)
        {
#pragma unroll
            for (int i = 0; i < kChainCols / 4; ++i) zin[i] = A.Z[back][zAt + i * 128];
            // gelu' under the products (tanhf: two thirds of this step's instructions)
#pragma unroll
            for (int i = 0; i < kChainCols / 4; ++i)
            {
                zin[i].x = gelu_grad(__bfloat162float(__float2bfloat16_rn(zin[i].x)));
                zin[i].y = gelu_grad(__bfloat162float(__float2bfloat16_rn(zin[i].y)));
                zin[i].z = gelu_grad(__bfloat162float(__float2bfloat16_rn(zin[i].z)));
                zin[i].w = gelu_grad(__bfloat162float(__float2bfloat16_rn(zin[i].w)));
            }
        }
        float x[3], t[7];                        // the loss's row (of any alignment: maybe the caller's)
        if (TRAIN && s == kHidden && warp < 4)
        {
#pragma unroll
            for (int k = 0; k < 3; ++k) x[k] = __ldg(A.in + row * 8 + k);
#pragma unroll
            for (int k = 0; k < 7; ++k) t[k] = __ldg(A.tgt + row * 8 + k);
        }
        ok = __all_sync(0xffffffffu, mbar_wait(&done, (uint32_t)s & 1u, A.err) && fine);
        tc_fence_after();
        if (ok && threadIdx.x == 0 && s + 1 < kSteps)
        {   // the products are done with the weights
            fine = chain_landed(s, full, A.err);
            if (fine) chain_load(M, loaded = s + 1, weights, full);
        }
        __syncwarp();
        if (ok && s == kHidden)
        {   // head: one thread a ray
            if (warp < 4)
            {
                float y[kOut];
                tmem_ld16(tl + kWidth, y);
#pragma unroll
                for (int k = 0; k < kOut; ++k) y[k] += sBias[kHidden * kWidth + k];
                if constexpr (TRAIN)
                {
                    const float sum = chain_loss(A, y, x, t, tile, (uint32_t)r);
                    if (lane < kSgSlice - kHidden * kWidth) sSum[warp][kHidden * kWidth + lane] = sum;
                }
                else if (valid)
                {
#pragma unroll
                    for (int k = 0; k < kOut; ++k) A.Y[(size_t)(m0 + r) * kOut + k] = y[k];
                }
            }
        }
        else if (ok)
        {
#pragma unroll
            for (int k = 0; k < kChainCols; k += 32)
            {
                const int c = c0 + k;
                float v[32];
                tmem_ld32(tl + (uint32_t)c, v);
                uint32_t o[16];
                if (s < kHidden)
                {
                    const float* bl = sBias + s * kWidth + c;
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                    {
                        v[2 * i] += bl[2 * i];
                        v[2 * i + 1] += bl[2 * i + 1];
                        // = gelu2 of bf16(z)
                        o[i] = bits(gelu2_half(__floats2bfloat162_rn(0.5f * v[2 * i], 0.5f * v[2 * i + 1])));
                    }
                    if constexpr (TRAIN)
                    {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            A.Z[s][zAt + (k / 4 + i) * 128] =
                                make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    }
                }
                else if constexpr (TRAIN)
                {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                    {
                        const float2 g = reinterpret_cast<const float2*>(zin)[k / 2 + i];
                        v[2 * i] *= g.x;
                        v[2 * i + 1] *= g.y;
                        o[i] = bits(__floats2bfloat162_rn(v[2 * i], v[2 * i + 1]));
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    st_operand(tile, (uint32_t)r, (uint32_t)(c / 8 + i),
                               make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]));
                if constexpr (TRAIN)
                    if (s > kHidden) sSum[warp & 3][back * kWidth + c + lane] = column_sum(v);
            }
        }
        fence_async_smem();
        tc_fence_before();
        ok = __syncthreads_and(ok && fine);
        tc_fence_after();
    }
    if (TRAIN && threadIdx.x == 32)
    {   // dZ_0, and every store before it, done
        if (ok)
            for (int kb = 0; kb < 4; ++kb) tma_store_2d(&M.dZ[0], tile + kb * kABlock, kb * 64, m0);
        tma_store_commit();
        tma_store_wait();
    }
    // after a timed-out wait: the CTA leaves only once its copies have landed
    if (!ok && threadIdx.x == 0) chain_landed(loaded, full, A.err);
    if constexpr (TRAIN)
        if (ok)
            for (int i = threadIdx.x; i < kSgSlice; i += kChainThreads)
                A.slices[(size_t)blockIdx.x * kSgSlice + i] = (sSum[0][i] + sSum[1][i]) + (sSum[2][i] + sSum[3][i]);
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 512);
}

// ---- weight gradients ----------------------------------------------------------
constexpr int kGradStages = 4, kGradThreads = 576;        // sixteen epilogue warps, TMA, MMA
constexpr uint32_t kBox = 64u * 128u;                     // 64 batch rows x 64 columns
constexpr uint32_t kGradStage = 6u * kBox;                // 2 boxes of one operand, up to 4 of the other
constexpr uint32_t kGradSmem = kGradStages * kGradStage + 1024u;

// MN-major operand (the contraction index outermost), 128-byte swizzle: 8 batch rows
// x 64 columns make an atom of 1024 B, atoms of further batch rows follow (SBO), the
// next 64 columns are a box away (LBO).
__device__ __forceinline__ uint64_t sdesc_mn_sw128(uint32_t saddr)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(kBox >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
           ((uint64_t)1u << 46) | ((uint64_t)2u << 61);
}

struct GradMaps
{
    CUtensorMap rows[kLayers];   // the operand whose columns are the tile's rows: dZ_l; X of the head
    CUtensorMap cols[kLayers];   // the other one: X_l; dY
};

// 128-ray tiles of the batch that share k takes start at ...
__device__ __forceinline__ int share_tile(int tiles, int shares, int k) { return (int)((long long)tiles * k / shares); }

// Tile t = 2 l + h: rows 128 h .. of product l.  The head's is X^T dY (its gradient's transpose).
// blockIdx.y: the part.  Its shares' products go to the two accumulators in turn, so one share is
// read back and added in registers while the next is multiplied.  The first warps also add the slices
// of the biases.
__global__ void __launch_bounds__(kGradThreads, 1)
weight_grad_kernel(const __grid_constant__ GradMaps maps, const float* slices, float* parts, int tiles,
                   unsigned* __restrict__ err)
{
    extern __shared__ uint8_t smemRaw[];
    __shared__ uint64_t full[kGradStages], empty[kGradStages], done[2], taken[2];
    __shared__ uint32_t tmemSlot;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = blockIdx.x >> 1, m0 = (blockIdx.x & 1) * 128;
    const bool head = l == kHidden;
    const int boxes = head ? 1 : 4;                       // 64-column boxes of the second operand
    const int shares = sg_shares(tiles);
    const int k0 = shares * (int)blockIdx.y / (int)gridDim.y, k1 = shares * ((int)blockIdx.y + 1) / (int)gridDim.y;
    float* part = parts + (size_t)blockIdx.y * kSgPart;
    const CUtensorMap* tA = &maps.rows[l];
    const CUtensorMap* tB = &maps.cols[l];

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kGradStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&done[b], 1); mbar_init(&taken[b], 16); }
        fence_barrier_init();
        tma_prefetch_desc(tA);
        tma_prefetch_desc(tB);
    }
    __syncwarp();
    launch_dependents();
    if (warp == 0) tmem_alloc(&tmemSlot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    wait_for_previous();
    const uint32_t tmem = tmemSlot;

    if (threadIdx.x == 512)
    {
        const int first = 2 * share_tile(tiles, shares, k0), blocks = 2 * share_tile(tiles, shares, k1) - first;
        int issued = 0;
        for (int kb = 0; kb < blocks; ++kb, ++issued)
        {
            const int s = kb % kGradStages;
            if (kb >= kGradStages && !mbar_wait(&empty[s], ((kb / kGradStages) - 1) & 1, err)) break;
            uint8_t* st = smem + s * kGradStage;
            const int y = (first + kb) * 64;
            mbar_expect_tx(&full[s], (2u + (uint32_t)boxes) * kBox);
            tma_load_2d(st, tA, &full[s], m0, y);
            tma_load_2d(st + kBox, tA, &full[s], m0 + 64, y);
            for (int b = 0; b < boxes; ++b) tma_load_2d(st + (2 + b) * kBox, tB, &full[s], b * 64, y);
        }
        // the CTA leaves only once its copies have landed, also after a timed-out wait
        for (int kb = issued > kGradStages ? issued - kGradStages : 0; kb < issued; ++kb)
            if (!mbar_wait(&full[kb % kGradStages], (kb / kGradStages) & 1, err)) break;
    }
    else if (threadIdx.x == 544)
    {
        const uint32_t idesc = idesc_bf16_f32(head ? 64 : 256) | (1u << 15) | (1u << 16);   // A and B MN-major
        bool ok = true;
        int kb = 0;
        for (int k = k0; k < k1 && ok; ++k)
        {
            const int turn = k - k0, buf = turn & 1;
            if (turn >= 2 && !mbar_wait(&taken[buf], (uint32_t)((turn >> 1) - 1) & 1u, err)) break;
            tc_fence_after();
            const int end = kb + 2 * (share_tile(tiles, shares, k + 1) - share_tile(tiles, shares, k));
            for (bool more = false; kb < end; ++kb, more = true)
            {
                const int s = kb % kGradStages;
                if (!(ok = mbar_wait(&full[s], (kb / kGradStages) & 1, err))) break;
                tc_fence_after();
                const uint32_t sa = smem_u32(smem + s * kGradStage), sb = sa + 2u * kBox;
#pragma unroll
                for (int j = 0; j < 4; ++j)      // 16 batch rows each: two atoms on
                    mma_bf16(tmem + (uint32_t)buf * 256u, sdesc_mn_sw128(sa + j * 2048), sdesc_mn_sw128(sb + j * 2048),
                             idesc, more || j > 0);
                mma_commit(&empty[s]);
            }
            mma_commit(&done[buf]);
        }
    }
    else if (warp < 16)
    {
        // this tile's biases, one a thread (the head's first tile: its 16 and the loss's 8)
        if (threadIdx.x < (head ? (m0 == 0 ? kOut + 8 : 0) : 128))
        {
            const float* from = slices + (head ? kHidden * kWidth : l * kWidth + m0) + threadIdx.x;
            float sum = 0.f;
            for (int k = k0; k < k1; ++k)
            {
                double share = 0.0;
                const int end = share_tile(tiles, shares, k + 1);
                for (int t = share_tile(tiles, shares, k); t < end; ++t) share += (double)from[(size_t)t * kSgSlice];
                sum = k == k0 ? (float)share : sum + (float)share;
            }
            part[SgLayout::b(l) + m0 + threadIdx.x] = sum;
        }
        __syncwarp();
        // a row and 64 columns a thread (the head: 16, of the first four warps)
        const int c0 = (warp >> 2) * 64, cols = !head ? 64 : c0 == 0 ? kOut : 0, row = (warp & 3) * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
        float acc[64] = {};
        bool ok = true;
        for (int k = k0; k < k1 && ok; ++k)
        {
            const int turn = k - k0, buf = turn & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(&done[buf], (uint32_t)(turn >> 1) & 1u, err));
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < 64; c += 16)
                if (c < cols && ok)
                {
                    float v[16];
                    tmem_ld16(tl + (uint32_t)(buf * 256 + c), v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[c + i] += v[i];
                }
            tc_fence_before();
            if (lane == 0) mbar_arrive(&taken[buf]);
        }
        // four columns of a row are a float4, the rows of a tile follow one another (sg_quad)
        float4* g = reinterpret_cast<float4*>(part + SgLayout::w(l)) + (m0 / 4) * (head ? kOut : kWidth) + c0 * 32 + row;
#pragma unroll
        for (int c = 0; c < 64; c += 4)
            if (c < cols && ok) g[c * 32] = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 512);
}

template <bool TRAIN>
cudaError_t launch_chain(const SgState& S, ChainArgs& A, bool early, cudaStream_t s)
{
    ChainMaps M{};
    const __nv_bfloat16* head = S.W + (size_t)kHidden * kWidth * kWidth;
    const __nv_bfloat16* headT = S.Wt + (size_t)kHidden * kWidth * kWidth;
    cudaError_t e = bh_tensor_map_bf16(&M.W, S.W, kHidden * kWidth, kWidth, kWidth, kWidth);
    if (e == cudaSuccess) e = bh_tensor_map_bf16(&M.Wh, head, kOut, kWidth, kWidth, kOut);
    if (TRAIN)
    {
        if (e == cudaSuccess) e = bh_tensor_map_bf16(&M.Wt, S.Wt, kHidden * kWidth, kWidth, kWidth, kWidth);
        if (e == cudaSuccess) e = bh_tensor_map_bf16(&M.Wht, headT, kWidth, kOutPad, kOutPad, kWidth);
        for (int l = 0; l < kLayers && e == cudaSuccess; ++l) e = bh_tensor_map_bf16(&M.X[l], S.X[l], A.n, kWidth, kWidth, 128);
        for (int l = 0; l < kHidden && e == cudaSuccess; ++l) e = bh_tensor_map_bf16(&M.dZ[l], S.dZ[l], A.n, kWidth, kWidth, 128);
        if (e == cudaSuccess) e = bh_tensor_map_bf16(&M.dY, S.dY, A.n, kOutPad, kOutPad, 128);
    }
    A.params = S.params;
    A.err = S.err;
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(chain_kernel<TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChainSmem);
    if (e != cudaSuccess) return e;
    return sg_launch(chain_kernel<TRAIN>, dim3((A.n + 127) / 128), kChainThreads, kChainSmem, early, s, M, A);
}

}  // namespace

cudaError_t sg_chain_forward(const SgState& S, const float* in, float* Y, int n, cudaStream_t s)
{
    ChainArgs A{};
    A.in = in;
    A.Y = Y;
    A.n = n;
    return launch_chain<false>(S, A, false, s);
}

cudaError_t sg_chain_train(const SgState& S, const float* in, const float* tgt, long long N, unsigned seed, int n,
                           bool early, cudaStream_t s)
{
    ChainArgs A{};
    A.in = in;
    A.tgt = tgt;
    A.N = N;
    A.seed = seed;
    for (int l = 0; l < kHidden; ++l) A.Z[l] = reinterpret_cast<float4*>(S.Z[l]);
    A.slices = S.slices;
    A.wEsc = S.wEsc; A.wDiskR = S.wDiskR; A.wDiskG = S.wDiskG; A.wConf = S.wConf; A.escTol = S.escTol;
    A.n = n;
    return launch_chain<true>(S, A, early, s);
}

cudaError_t sg_weight_grads(const SgState& S, int n, cudaStream_t s)
{
    GradMaps maps;
    cudaError_t e = cudaSuccess;
    for (int l = 0; l < kLayers && e == cudaSuccess; ++l)
    {
        const bool head = l == kHidden;
        e = bh_tensor_map_bf16(&maps.rows[l], head ? S.X[kHidden] : S.dZ[l], n, kWidth, kWidth, 64);
        if (e == cudaSuccess)
            e = head ? bh_tensor_map_bf16(&maps.cols[l], S.dY, n, kOutPad, kOutPad, 64)
                     : bh_tensor_map_bf16(&maps.cols[l], S.X[l], n, kWidth, kWidth, 64);
    }
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGradSmem);
    if (e != cudaSuccess) return e;
    return sg_launch(weight_grad_kernel, dim3(2 * kLayers, sg_parts(n / 128)), kGradThreads, kGradSmem, true, s, maps,
                     static_cast<const float*>(S.slices), S.parts, n / 128, S.err);
}
