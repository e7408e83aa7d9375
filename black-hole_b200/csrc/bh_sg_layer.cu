// ---------------------------------------------------------------------------
// bh_sg_layer.cu -- the surrogate's training GEMMs with what follows them in
// their epilogues (tcgen05 + TMA):
//
//   forward    Z = X W^T + b,  X' = gelu(Z)                  (layer_kernel<false>)
//   backward   dZ = (dZ' W') * gelu'(Z),  db += column sums   (layer_kernel<true>)
//   weights    dW_l += dZ_l^T X_l of every layer and the head (weight_grad_kernel)
//
// layer_kernel: one CTA per 128 rows, all 256 columns.  The whole contraction
// (256, or 64 for the head's gradient) fits in shared memory, so every copy is
// issued at once and each 64-wide block is multiplied as it lands.  Sixteen warps
// read the accumulator back (one row a thread, a quarter of the columns a warp).
// Z is kept as [column / 4][row], which a warp writes and reads in 512-byte runs
// (15 and 22 us a forward and backward layer with row-major Z and eight warps); the
// BF16 result leaves by TMA from over the first operand.  Bound: one tile's chain of
// copy, products and epilogue on 128 of the 148 SMs, and the launch.  At 16,384 rows:
// forward layer 11.3 us (42.6 for a GEMM with 4-byte stores + 8.3 for the activation
// as launches of their own), backward 15.4 us (27.3 + 24.4).
//
// weight_grad_kernel: the contraction runs over the rows of the batch, so both
// operands are read as they lie, with the contraction index as the outer one
// (MN-major descriptors), instead of through transposed copies (10 x 12.4 us
// before).  One launch for all five products: a CTA takes one 128-row tile of one
// product over a share of the batch and adds it to the gradient with 16-byte
// reductions: 20.7 us (26.6 + 4 x 31 us, on top of the transposes).
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
constexpr uint32_t kLayerSmem = 4u * (kABlock + kBBlock) + 1024u;
constexpr int kLayerThreads = 512;
constexpr int kLayerCols = kWidth / (kLayerThreads / 128);   // accumulator columns a warp reads back

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

template <bool BACK>
__global__ void __launch_bounds__(kLayerThreads, 1)
layer_kernel(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tB,
             const __grid_constant__ CUtensorMap tOut, float4* __restrict__ Z, const float* __restrict__ bias,
             float* __restrict__ db, int n, int kBlocks, unsigned* __restrict__ err)
{
    extern __shared__ uint8_t smemRaw[];
    __shared__ uint64_t full[4], done;
    __shared__ uint32_t tmemSlot;
    __shared__ float sCol[kWidth];               // forward: biases; backward: column sums
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * 128;

    if (threadIdx.x < kWidth) sCol[threadIdx.x] = BACK ? 0.f : bias[threadIdx.x];
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < 4; ++s) mbar_init(&full[s], 1);
        mbar_init(&done, 1);
        fence_barrier_init();
        tma_prefetch_desc(&tA);
        tma_prefetch_desc(&tB);
        tma_prefetch_desc(&tOut);
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(&tmemSlot, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmemSlot;

    if (threadIdx.x == 0)
    {
        for (int kb = 0; kb < kBlocks; ++kb)
        {
            uint8_t* a = smem + kb * (kABlock + kBBlock);
            mbar_expect_tx(&full[kb], kABlock + kBBlock);
            tma_load_2d(a, &tA, &full[kb], kb * 64, m0);
            tma_load_2d(a + kABlock, &tB, &full[kb], kb * 64, 0);
        }
        // the CTA leaves only once its copies have landed
        for (int kb = 0; kb < kBlocks; ++kb)
            if (!mbar_wait(&full[kb], 0, err)) break;
    }
    else if (threadIdx.x == 32)
    {
        constexpr uint32_t idesc = idesc_bf16_f32(256);
        for (int kb = 0; kb < kBlocks; ++kb)
        {
            if (!mbar_wait(&full[kb], 0, err)) break;
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + kb * (kABlock + kBBlock)), sb = sa + kABlock;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                mma_bf16(tmem, sdesc_sw128(sa + j * 32), sdesc_sw128(sb + j * 32), idesc, kb > 0 || j > 0);
        }
        mma_commit(&done);
    }
    __syncwarp();
    // warp w: rows 32 (w % 4) .., columns kLayerCols (w / 4) ..
    const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * kLayerCols;
    float4* z = Z + (size_t)blockIdx.x * (128 * kWidth / 4) + r;          // [column / 4][row]
    float4 zin[BACK ? kLayerCols / 4 : 1];
    if constexpr (BACK)
    {   // under the copies and products
#pragma unroll
        for (int i = 0; i < kLayerCols / 4; ++i) zin[i] = __ldg(z + (c0 / 4 + i) * 128);
    }
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&done, 0, err));
    tc_fence_after();
    if (ok)
    {   // all operands are used up
        const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const bool valid = m0 + r < n;
#pragma unroll
        for (int k = 0; k < kLayerCols; k += 32)
        {
            const int c = c0 + k;
            float v[32];
            tmem_ld32(tl + (uint32_t)c, v);
            uint32_t o[16];
#pragma unroll
            for (int i = 0; i < 16; ++i)
            {
                float a = v[2 * i], b = v[2 * i + 1];
                if constexpr (BACK)
                {
                    const float2 zz = reinterpret_cast<const float2*>(zin)[k / 2 + i];
                    a = valid ? a * gelu_grad(__bfloat162float(__float2bfloat16_rn(zz.x))) : 0.f;
                    b = valid ? b * gelu_grad(__bfloat162float(__float2bfloat16_rn(zz.y))) : 0.f;
                    o[i] = bits(__floats2bfloat162_rn(a, b));
                }
                else
                {
                    a += sCol[c + 2 * i];
                    b += sCol[c + 2 * i + 1];
                    o[i] = bits(gelu2_half(__floats2bfloat162_rn(0.5f * a, 0.5f * b)));   // = gelu2 of bf16(z)
                }
                v[2 * i] = a;
                v[2 * i + 1] = b;
            }
            // over the first operand: 64-column blocks as the copies laid them out
            uint8_t* block = smem + (c >> 6) * (kABlock + kBBlock);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<uint4*>(block + sw128_offset((uint32_t)r, (uint32_t)((c & 63) + 8 * i), 128u)) =
                    make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            if constexpr (BACK)
            {
                const float s = column_sum(v);
                atomicAdd(&sCol[c + lane], s);
            }
            else
            {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    z[(c / 4 + i) * 128] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        }
        fence_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    if (ok && threadIdx.x == 0)
    {
        for (int kb = 0; kb < kWidth / 64; ++kb) tma_store_2d(&tOut, smem + kb * (kABlock + kBBlock), kb * 64, m0);
        tma_store_wait();
    }
    if (BACK && ok && threadIdx.x < kWidth) atomicAdd(db + threadIdx.x, sCol[threadIdx.x]);
    __syncwarp();
    if (warp == 0) tmem_free(tmem, 256);
}

// ---- weight gradients ----------------------------------------------------------
constexpr int kGradStages = 4;
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

__device__ __forceinline__ void red4(float* p, float a, float b, float c, float d)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

struct GradMaps
{
    CUtensorMap rows[kLayers];   // the operand whose columns are the tile's rows: dZ_l; X of the head
    CUtensorMap cols[kLayers];   // the other one: X_l; dY
};

// Tile t = 2 l + h: rows 128 h .. of product l.  The head's is X^T dY (its gradient's transpose).
__global__ void __launch_bounds__(128, 1)
weight_grad_kernel(const __grid_constant__ GradMaps maps, float* __restrict__ grads, int kBlocks,
                   unsigned* __restrict__ err)
{
    extern __shared__ uint8_t smemRaw[];
    __shared__ uint64_t full[kGradStages], empty[kGradStages], done;
    __shared__ uint32_t tmemSlot;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = blockIdx.x >> 1, m0 = (blockIdx.x & 1) * 128;
    const bool head = l == kHidden;
    const int boxes = head ? 1 : 4;                       // 64-column boxes of the second operand
    const int kb0 = (int)((long long)kBlocks * blockIdx.y / gridDim.y);
    const int kb1 = (int)((long long)kBlocks * (blockIdx.y + 1) / gridDim.y);
    const CUtensorMap* tA = &maps.rows[l];
    const CUtensorMap* tB = &maps.cols[l];

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kGradStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&done, 1);
        fence_barrier_init();
        tma_prefetch_desc(tA);
        tma_prefetch_desc(tB);
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(&tmemSlot, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmemSlot;
    const int blocks = kb1 - kb0;

    if (threadIdx.x == 0)
    {
        int issued = 0;
        for (int kb = 0; kb < blocks; ++kb, ++issued)
        {
            const int s = kb % kGradStages;
            if (kb >= kGradStages && !mbar_wait(&empty[s], ((kb / kGradStages) - 1) & 1, err)) break;
            uint8_t* st = smem + s * kGradStage;
            const int y = (kb0 + kb) * 64;
            mbar_expect_tx(&full[s], (2u + (uint32_t)boxes) * kBox);
            tma_load_2d(st, tA, &full[s], m0, y);
            tma_load_2d(st + kBox, tA, &full[s], m0 + 64, y);
            for (int b = 0; b < boxes; ++b) tma_load_2d(st + (2 + b) * kBox, tB, &full[s], b * 64, y);
        }
        // the CTA leaves only once its copies have landed, also after a timed-out wait
        for (int kb = issued > kGradStages ? issued - kGradStages : 0; kb < issued; ++kb)
            if (!mbar_wait(&full[kb % kGradStages], (kb / kGradStages) & 1, err)) break;
    }
    else if (threadIdx.x == 32)
    {
        const uint32_t idesc = idesc_bf16_f32(head ? 64 : 256) | (1u << 15) | (1u << 16);   // A and B MN-major
        for (int kb = 0; kb < blocks; ++kb)
        {
            const int s = kb % kGradStages;
            if (!mbar_wait(&full[s], (kb / kGradStages) & 1, err)) break;
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + s * kGradStage), sb = sa + 2u * kBox;
#pragma unroll
            for (int j = 0; j < 4; ++j)      // 16 batch rows each: two atoms on
                mma_bf16(tmem, sdesc_mn_sw128(sa + j * 2048), sdesc_mn_sw128(sb + j * 2048), idesc, kb > 0 || j > 0);
            mma_commit(&empty[s]);
        }
        mma_commit(&done);
    }
    __syncwarp();
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&done, 0, err));
    tc_fence_after();
    if (ok && blocks > 0)
    {
        const int row = m0 + warp * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)(warp * 32) << 16);
        if (!head)
        {
            float* g = grads + SgLayout::w(l) + (size_t)row * kWidth;
#pragma unroll 1
            for (int c = 0; c < kWidth; c += 32)
            {
                __syncwarp();
                float v[32];
                tmem_ld32(tl + (uint32_t)c, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) red4(g + c + 4 * i, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        }
        else
        {   // row = input unit, column = output unit
            float v[16];
            tmem_ld16(tl, v);
#pragma unroll
            for (int o = 0; o < kOut; ++o) atomicAdd(grads + SgLayout::w(kHidden) + o * kWidth + row, v[o]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 256);
}

template <bool BACK>
cudaError_t launch_layer(const void* A, int K, const void* B, float* Z, void* out, const float* bias, float* db, int n,
                         unsigned* err, cudaStream_t s)
{
    CUtensorMap ta, tb, to;
    cudaError_t e = bh_tensor_map_bf16(&ta, A, n, K, K, 128);
    if (e == cudaSuccess) e = bh_tensor_map_bf16(&to, out, n, kWidth, kWidth, 128);
    if (e == cudaSuccess) e = bh_tensor_map_bf16(&tb, B, kWidth, K, K, kWidth);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(layer_kernel<BACK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLayerSmem);
    if (e != cudaSuccess) return e;
    layer_kernel<BACK><<<(n + 127) / 128, kLayerThreads, kLayerSmem, s>>>(
        ta, tb, to, reinterpret_cast<float4*>(Z), bias, db, n, K / 64, err);
    return cudaGetLastError();
}

}  // namespace

cudaError_t sg_layer_forward(const SgState& S, int l, int n, cudaStream_t s)
{
    return launch_layer<false>(S.X[l], kWidth, S.W + (size_t)l * kWidth * kWidth, S.Z[l], S.X[l + 1],
                               S.params + SgLayout::b(l), nullptr, n, S.err, s);
}

cudaError_t sg_layer_backward(const SgState& S, int l, int n, cudaStream_t s)
{
    const bool head = l == kHidden - 1;
    return launch_layer<true>(head ? S.dY : S.dZ[l + 1], head ? kOutPad : kWidth,
                              S.Wt + (size_t)(l + 1) * kWidth * kWidth, S.Z[l], S.dZ[l], nullptr,
                              S.grads + SgLayout::b(l), n, S.err, s);
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
    // ten tiles, the batch cut so that all CTAs of the 148 SMs run at once
    const int kBlocks = n / 64, splits = kBlocks < 14 ? kBlocks : 14;
    weight_grad_kernel<<<dim3(2 * kLayers, splits), 128, kGradSmem, s>>>(maps, S.grads, kBlocks, S.err);
    return cudaGetLastError();
}
