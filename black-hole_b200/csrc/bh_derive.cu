// ---------------------------------------------------------------------------
// bh_derive.cu -- bhValidateAndDerive on the GPU for many black holes at once
// (one CTA per request), so batched views can be derived without a host round
// trip.
//
// Restates the reference's host derivation (src/metric.cuh:257-329, numeric
// ISCO metric.cuh:224-248) exactly as bh_params.cpp does: every operation is
// an IEEE single operation with contraction blocked (__fadd_rn, __fmul_rn,
// __fdiv_rn, __fsqrt_rn), in the same order, so the results are bit-identical
// to the host build.  acos and cos of the Kerr photon orbit are evaluated in
// double and rounded to float (correctly rounded; the host libm's float acos
// differs from that by one ulp on some inputs, a few ulps of rPhoton).
//
// The ISCO scan visits r = rStart, rStart + dr, ... as a running float sum whose
// rounding fixes the visited radii, and keeps the first of the lowest energies.
// Neither the sum nor the whole scan has to be walked:
//   * inside one binade every radius is a multiple of the binade's ulp, and after
//     the first sum there (which may round a tie by the parity it comes with) the
//     rounded increment is the same until the binade ends, so the visited
//     radii are a handful of exact arithmetic sequences (Segment);
//   * of a hole with a horizon the energy of the circular orbits falls from the
//     photon orbit to the ISCO and rises from there on, so every kStride-th radius
//     is evaluated first, and then all radii between those within kWindow of the
//     lowest.  Near the minimum the energies of neighbouring visits differ by less
//     than their rounding, so the window is evaluated exactly as the scan does it.
//     A naked singularity, a hole without a valid coarse radius, and masses outside
//     kMassLow .. kMassHigh get the whole scan: far outside, products of an energy
//     leave FP32's normal range, and below 1e-6 the scan starts inside the horizon.
// Bound: instruction issue (the IEEE divisions and roots of ~2,600 energies a hole)
// with one thread's set-up before it.  13,824 holes: 4.39 ms with the running sum
// (a chain of 12,000 dependent sums a hole) and the whole scan, 0.19 ms so.
// ---------------------------------------------------------------------------
#include <cmath>
#include <cuda_runtime.h>
#include "bh_launch.h"

namespace {

constexpr int kThreads = 128;
constexpr int kStride = 16;           // coarse pass of the scan
constexpr float kWindow = 1e-3f;      // relative: coarse radii this close to the lowest energy mark the window
constexpr float kMassLow = 1e-5f, kMassHigh = 1e5f;
constexpr int kMaxSegments = 64;
constexpr float kExtremal = 0.995f;
constexpr float kNakedCap = 2.25f;
constexpr float kSingCut = 0.05f;

__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ float fq(float a) { return __fsqrt_rn(a); }

__device__ bool spinning(int m) { return m == BH_KERR || m == BH_KERR_NEWMAN; }
__device__ bool charged(int m) { return m == BH_REISSNER_NORDSTROM || m == BH_KERR_NEWMAN; }

__device__ float outerHorizon(float M, float a, float Q)
{
    const float d = fs(fs(fm(M, M), fm(a, a)), fm(Q, Q));
    return fa(M, fq(d < 0.f ? 0.f : d));
}

__device__ float innerHorizon(float M, float a, float Q)
{
    const float d = fs(fs(fm(M, M), fm(a, a)), fm(Q, Q));
    return fs(M, fq(d < 0.f ? 0.f : d));
}

__device__ float photonSphere(float M, float Q)
{
    const float d = fs(fm(fm(9.f, M), M), fm(fm(8.f, Q), Q));
    return fm(0.5f, fa(fm(3.f, M), fq(d < 0.f ? 0.f : d)));
}

__device__ float photonOrbitKerr(float M, float aStar)
{
    const float x = aStar > 1.f ? 1.f : (aStar < -1.f ? -1.f : aStar);
    const float ac = (float)acos((double)(-x));
    const float c = (float)cos((double)fm(2.f / 3.f, ac));
    return fm(fm(2.f, M), fa(1.f, c));
}

__device__ float photonOrbitKN(float M, float aStar, float q)
{
    const float rK = photonOrbitKerr(M, aStar);
    const float rS = photonSphere(M, fm(q, M));
    if (fabsf(aStar) < 1e-5f) return rS;
    float w = fm(q, q);
    w = w < 0.f ? 0.f : (w > 1.f ? 1.f : w);
    return fa(fm(fs(1.f, fm(0.35f, w)), rK), fm(fm(0.35f, w), rS));
}

__device__ float ergoRadius(float M, float Q)
{
    const float d = fs(fm(M, M), fm(Q, Q));
    return fa(M, fq(d < 0.f ? 0.f : d));
}

// specific energy of the circular orbit at r (metric.cuh:145-199 via bh_params.cpp)
__device__ bool orbitEnergy(float r, float M, float a, float Q, float& E)
{
    const float w2 = fs(fm(M, r), fm(Q, Q));
    if (w2 <= 0.f) return false;
    const float sw = fq(w2);
    const float Om = fd(sw, fa(fm(r, r), fm(a, sw)));
    if (Om <= 0.f) return false;
    const float r2 = fm(r, r);
    const float m2r = fs(fm(fm(2.f, M), r), fm(Q, Q));
    const float gtt = -fs(1.f, fd(m2r, r2));
    const float gtp = fd(fm(-a, m2r), r2);
    const float gpp = fa(fa(r2, fm(a, a)), fd(fm(fm(m2r, a), a), r2));
    const float den = -fa(fa(gtt, fm(fm(2.f, Om), gtp)), fm(fm(Om, Om), gpp));
    if (den <= 1e-6f) return false;
    E = fd(-fa(gtt, fm(Om, gtp)), fq(den));
    return true;
}

// The visits first .. first + n - 1 of the scan: r = start + i step, exactly.
struct Segment
{
    float start, step;
    int first, n;
};

// The visiting sequence of `for (r = rStart; r <= rEnd; r += dr)` as exact
// arithmetic sequences, as far as r is finite; returns the number of segments, the visits in *total.
__device__ int scan_segments(float rStart, float rEnd, float dr, Segment* seg, int* total)
{
    int m = 0, k = 0;
    float r = rStart;
    while (r <= rEnd && r <= 3.402823466e38f && m < kMaxSegments)
    {
        // ulp of r's binade and its upper end, in ulps 2^24 (normal numbers)
        const int e = max((__float_as_int(r) >> 23) & 255, 1);
        const double perUlp = __hiloint2double((1023 + 150 - e) << 20, 0);
        const float r1 = fa(r, dr), step = fs(fa(r1, dr), r1);
        constexpr int top = 1 << 24;
        const bool same = max((__float_as_int(r1) >> 23) & 255, 1) == e;
        // the visit at r itself; then the constant increments from r1 on, if r1 is in the binade
        seg[m++] = Segment{r, 0.f, k, 1};
        ++k;
        r = r1;
        if (!same || !(r1 <= rEnd) || m >= kMaxSegments) continue;    // (r1 infinite: another exponent)
        const int i1 = (int)((double)r1 * perUlp), inc = (int)fmin((double)step * perUlp, (double)top);
        if (inc < 1) break;
        const int lim = (int)fmin((double)rEnd * perUlp, (double)(top - 1));   // last multiple a visit may take
        const int n = (lim - i1) / inc + 1;
        seg[m++] = Segment{r1, step, k, n};
        k += n;
        r = fa(__fmaf_rn((float)(n - 1), step, r1), dr);
    }
    *total = k;
    return m;
}

__device__ __forceinline__ float visit(const Segment* seg, int& at, int k)
{
    while (k >= seg[at].first + seg[at].n) ++at;
    return __fmaf_rn((float)(k - seg[at].first), seg[at].step, seg[at].start);
}

// Lowest energy of the CTA and the earliest visit that has it (thread 0's values).
__device__ void cta_lowest(float& E, int& k, float* sE, int* sK)
{
#pragma unroll
    for (int o = 16; o; o >>= 1)
    {
        const float e2 = __shfl_down_sync(0xffffffffu, E, o);
        const int k2 = __shfl_down_sync(0xffffffffu, k, o);
        if (e2 < E || (e2 == E && k2 < k)) { E = e2; k = k2; }
    }
    if ((threadIdx.x & 31) == 0) { sE[threadIdx.x >> 5] = E; sK[threadIdx.x >> 5] = k; }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < kThreads / 32; ++w)
            if (sE[w] < E || (sE[w] == E && sK[w] < k)) { E = sE[w]; k = sK[w]; }
}

__global__ void __launch_bounds__(kThreads)
derive_kernel(BHDeriveRequest* __restrict__ req, BHDerived* __restrict__ out, int n)
{
    __shared__ Segment seg[kMaxSegments];
    __shared__ float sE[kThreads / 32], sLow;
    __shared__ int sK[kThreads / 32], sTotal, sLo, sHi;
    __shared__ bool sWindow;
    __shared__ BHDerived sD;
    __shared__ float sM, sRp, sA, sQ;
    const int i = blockIdx.x;
    if (i >= n) return;

    if (threadIdx.x == 0 || threadIdx.x == 32)
    {   // both validate; one sets up the scan, the other derives the closed-form radii
        const BHDeriveRequest R = req[i];
        float M = R.M, aStar = R.aStar, q = R.q;
        BHDerived d{0.f, 0.f, 1.f, 0.f, 1.5f, 1.f, 3.f, 0, 0};
        if (!(M > 0.f) || !isfinite(M)) { M = 0.5f; d.clamped = 1; }
        if (!isfinite(aStar)) { aStar = 0.f; d.clamped = 1; }
        if (!isfinite(q)) { q = 0.f; d.clamped = 1; }
        const float knob = R.allowNaked ? 1.5f : kExtremal;   // sqrt(2.25) = 1.5 exactly
        if (aStar < -knob) { aStar = -knob; d.clamped = 1; }
        if (aStar > knob) { aStar = knob; d.clamped = 1; }
        if (q < 0.f) { q = 0.f; d.clamped = 1; }
        if (q > knob) { q = knob; d.clamped = 1; }
        float aEff = spinning(R.model) ? aStar : 0.f;
        float qEff = charged(R.model) ? q : 0.f;
        const float bound = R.allowNaked ? kNakedCap : kExtremal;
        const float s2 = fa(fm(aEff, aEff), fm(qEff, qEff));
        if (s2 > bound)
        {
            const float k = fq(fd(bound, s2));
            aEff = fm(aEff, k);
            qEff = fm(qEff, k);
            if (spinning(R.model)) aStar = aEff;
            if (charged(R.model)) q = qEff;
            d.clamped = 1;
        }
        d.a = fm(aEff, M);
        d.Q = fm(qEff, M);
        const float disc = fs(fs(fm(M, M), fm(d.a, d.a)), fm(d.Q, d.Q));   // NaN for a spinning M above 1.8e19
        d.naked = disc < 0.f ? 1 : 0;
        d.rPlus = d.naked ? 0.f : outerHorizon(M, d.a, d.Q);
        if (threadIdx.x == 0)
        {   // iscoRadius
            const float rp = disc >= 0.f ? d.rPlus : fm(kSingCut, M);
            sRp = rp;
            sM = M;
            sWindow = disc >= 0.f && M >= kMassLow && M <= kMassHigh;
            sLo = 0x7fffffff;
            sHi = -1;
            scan_segments(rp > 1e-6f ? fm(rp, 1.02f) : fm(0.5f, M), fm(12.f, M), fm(0.001f, M), seg, &sTotal);
        }
        else
        {
            d.rMinus = d.naked ? 0.f : innerHorizon(M, d.a, d.Q);
            d.rErgo = d.naked ? 0.f : ergoRadius(M, d.Q);
            if (spinning(R.model))
            {
                d.rPhoton = (R.model == BH_KERR_NEWMAN) ? photonOrbitKN(M, aEff, qEff) : photonOrbitKerr(M, aEff);
                if (d.rPlus > 0.f) { if (d.rPhoton < fm(d.rPlus, 1.02f)) d.rPhoton = fm(d.rPlus, 1.02f); }
                else if (d.rPhoton < fm(fm(kSingCut, M), 2.f)) d.rPhoton = fm(3.f, M);
            }
            else
            {
                d.rPhoton = photonSphere(M, d.Q);
                if (d.naked && !(d.rPhoton > 0.f)) d.rPhoton = fm(3.f, M);
            }
            sD = d;
            sA = aStar;
            sQ = q;
        }
    }
    __syncthreads();
    const float M = sM, a = sD.a, Q = sD.Q;
    const int total = sTotal;
    float bestE = 1e30f;
    int bestK = 0x7fffffff;
    int lo = 0, hi = total;               // visits to evaluate
    if (sWindow)
    {
        int at = 0;
        for (int k = (int)threadIdx.x * kStride; k < total; k += kThreads * kStride)
        {
            float E;
            if (orbitEnergy(visit(seg, at, k), M, a, Q, E) && E < bestE) { bestE = E; bestK = k; }
        }
        cta_lowest(bestE, bestK, sE, sK);
        if (threadIdx.x == 0) sLow = bestE;
        __syncthreads();
        const float low = sLow;
        if (low < 1e30f)
        {
            const float top = low + kWindow * fabsf(low);
            at = 0;
            for (int k = (int)threadIdx.x * kStride; k < total; k += kThreads * kStride)
            {
                float E;
                if (orbitEnergy(visit(seg, at, k), M, a, Q, E) && E <= top)
                {
                    atomicMin(&sLo, k);
                    atomicMax(&sHi, k);
                }
            }
            __syncthreads();
            lo = max(sLo - kStride + 1, 0);
            hi = min(sHi + kStride, total);
        }
        bestE = 1e30f;
        bestK = 0x7fffffff;
        __syncthreads();
    }
    {
        int at = 0;
        for (int k = lo + (int)threadIdx.x; k < hi; k += kThreads)
        {
            float E;
            if (orbitEnergy(visit(seg, at, k), M, a, Q, E) && E < bestE) { bestE = E; bestK = k; }
        }
    }
    cta_lowest(bestE, bestK, sE, sK);
    if (threadIdx.x == 0)
    {
        const float rp = sRp;
        float best;
        if (bestK != 0x7fffffff)
        {
            int at = 0;
            best = visit(seg, at, bestK);
        }
        else
        {
            best = (fm(6.f, M) > fm(rp, 1.5f)) ? fm(6.f, M) : fm(rp, 1.5f);
        }
        const float floorR = rp > 1e-6f ? fm(rp, 1.15f) : fm(0.5f, M);
        BHDerived d = sD;
        d.rIsco = best > floorR ? best : floorR;
        out[i] = d;
        req[i].M = sM; req[i].aStar = sA; req[i].q = sQ;
    }
}

}  // namespace

extern "C" cudaError_t bhDeriveBatch(BHDeriveRequest* requests, BHDerived* out, int n, cudaStream_t stream)
{
    if (n < 0 || (n > 0 && (!requests || !out))) return cudaErrorInvalidValue;
    if (n == 0) return cudaSuccess;
    derive_kernel<<<n, kThreads, 0, stream>>>(requests, out, n);
    return cudaGetLastError();
}
