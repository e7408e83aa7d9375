// ---------------------------------------------------------------------------
// bh_sg_train.h -- state of the lensing surrogate and its training passes
// (bh_sg_train.cu), used by the C-ABI in bh_sg_api.cpp.
// ---------------------------------------------------------------------------
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include "bh_trace_params.h"

// Flat FP32 parameter vector: for each hidden layer l = 0..3 the 256 x 256
// weight (row = output unit) then its 256 biases; then the 16 x 256 head
// weight and its 16 biases.
struct SgLayout
{
    static constexpr int kHid = 256 * 256 + 256;
    static constexpr __host__ __device__ int w(int l) { return l * kHid; }
    static constexpr __host__ __device__ int b(int l) { return l < 4 ? l * kHid + 256 * 256 : 4 * kHid + 16 * 256; }
    static constexpr __host__ __device__ int count() { return 4 * kHid + 16 * 256 + 16; }
};

// What a training step sums over the batch, it sums in a fixed order, so two runs are the same bits:
// a slice per 128 rays (all biases' gradients and the loss terms); shares of at most four of them (one
// accumulator of the weight gradients; longer ones only above 64 shares, 32,768 rays); at most 14 parts of
// some consecutive shares, added in FP32 (ten tiles of products x 14: one CTA an SM); then the parts, in FP64.
// All by the batch alone, not by the GPU.
constexpr int kSgBias = 4 * 256 + 16;                       // biases of all layers
constexpr int kSgSlice = kSgBias + 8;                       // ... and 8 loss terms
constexpr int kSgPart = SgLayout::count() + 8;              // all gradients and 8 loss terms
inline __host__ __device__ int sg_shares(int tiles) { return tiles < 4 * 64 ? (tiles + 3) / 4 : 64; }
inline __host__ __device__ int sg_parts(int tiles) { return sg_shares(tiles) < 14 ? sg_shares(tiles) : 14; }

// A launch; `early`: a programmatic one, whose CTAs may start before the kernel launched before it
// on the stream has ended (a step's three launches wait for one another inside the kernels)
template <class... P, class... A>
inline cudaError_t sg_launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, bool early, cudaStream_t s,
                             A&&... args)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

struct SgState
{
    int device = 0;
    float* params = nullptr;          // FP32 master copy (SgLayout)
    float* grads = nullptr;
    float* adamM = nullptr;
    float* adamV = nullptr;
    __nv_bfloat16* W = nullptr;       // BF16 W_l (out x in), hidden layers then the 16 x 256 head
    __nv_bfloat16* Wt = nullptr;      // BF16 W_l^T (in x out), hidden layers then the 256 x 64 padded head
    float* biasPacked = nullptr;      // all biases, contiguous (4 x 256 + 16), for the fused kernel
    float* loss = nullptr;            // 8 floats: loss sums of bhSurrogateGradients' batch
    unsigned* err = nullptr;          // tensor-core kernels' error word
    int step = 0;                     // Adam steps taken
    float wEsc = 100.f, wDiskR = 1.f, wDiskG = 1.f, wConf = 0.1f, escTol = 1e-3f;

    // per-batch scratch (capacity `cap` rays)
    int cap = 0;
    void* X[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};   // BF16 n x 256 activations
    float* Z[4] = {nullptr, nullptr, nullptr, nullptr};           // FP32 pre-activations, 128-row tiles of [column / 4][row][4]
    void* dY = nullptr;               // BF16 n x 64
    void* dZ[4] = {nullptr, nullptr, nullptr, nullptr};           // BF16 n x 256
    float* slices = nullptr;          // n / 128 x kSgSlice
    float* parts = nullptr;           // sg_parts(n / 128) x kSgPart, in groups of four parameters (sg_quad, bh_sg_train.cu)

    // the RK4-traced ray set: inputs (n x 8) and targets (n x 8)
    float* dsIn = nullptr;
    float* dsTgt = nullptr;
    long long dsN = 0;
};

cudaError_t sg_features(const float* in, void* X0, int n, cudaStream_t s);
cudaError_t sg_pack_weights(SgState& S, cudaStream_t s);
// grows the per-batch scratch to n rays
cudaError_t sg_reserve(SgState& S, int n);
void sg_free_batch(SgState& S);
// Forward, loss and backward of n rays; the gradients' parts are left in S.parts.  N > 0: the
// batch is rows of in / tgt at hashed indices below N.  `early`: the launch before it on the
// stream is sg_adam's.
cudaError_t sg_backward(SgState& S, const float* in, const float* tgt, long long N, unsigned seed, int n, bool early,
                        cudaStream_t s);
// Right after sg_backward of n rays: its loss sums to `loss` (8 floats), and the sums of the
// gradients to S.grads, or an Adam step with them.
cudaError_t sg_gradients(SgState& S, int n, float* loss, cudaStream_t s);
cudaError_t sg_adam(SgState& S, int n, float lr, float* loss, cudaStream_t s);
// the kernels of bh_sg_chain.cu: Y (n x 16) = net(in) in the training form; its activations, dZ_l
// and slices; the parts of all gradients
cudaError_t sg_chain_forward(const SgState& S, const float* in, float* Y, int n, cudaStream_t s);
cudaError_t sg_chain_train(const SgState& S, const float* in, const float* tgt, long long N, unsigned seed, int n,
                           bool early, cudaStream_t s);
cudaError_t sg_weight_grads(const SgState& S, int n, cudaStream_t s);
