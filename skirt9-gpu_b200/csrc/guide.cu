// Learned path guiding: network state, training on the GPU (own FP32 forward / backward kernels and
// Adam), the BF16 tensor-core inference of a batch, and the pilot records.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "ctx.hpp"
#include "guide_internal.hpp"
#include "guide_mma.cuh"

namespace skg {

namespace {

// ---------------------------------------------------------------------------------------------
// FP32 forward pass of one sample: raw outputs and the activations of the hidden layers
// ---------------------------------------------------------------------------------------------
SKG_D void mlpForward(const float* P, const float* in, float* h /*4 x 64*/, float* out)
{
    const float* cur = in;
    int nin = GUIDE_IN;
    for (int l = 0; l < GUIDE_LAYERS; ++l)
    {
        const float* W = P + guideParamOffset(l);
        const float* b = W + guideDimOut(l) * nin;
        float* dst = l + 1 < GUIDE_LAYERS ? h + 64 * l : out;
        for (int o = 0; o < guideDimOut(l); ++o)
        {
            float acc = b[o];
            for (int i = 0; i < nin; ++i) acc = fmaf(W[o * nin + i], cur[i], acc);
            dst[o] = l + 1 < GUIDE_LAYERS ? fmaxf(acc, 0.f) : acc;
        }
        cur = dst;
        nin = guideDimOut(l);
    }
}

// ---------------------------------------------------------------------------------------------
// Loss and gradient of a batch, in FP32 on the CUDA cores (the training keeps 32 bits throughout).
//
// One block per SM takes its share of the batch in tiles of S samples and keeps everything of a tile
// on chip: the network (67 KB) and the activations of all layers in shared memory, the sums of the
// weight gradients in registers (a thread holds a 4 x 4 patch of every layer's matrix) until its last
// tile. Forward pass, back-propagation and weight gradients are all products of a 64-wide and an
// S-wide side, computed as 4 x S/16 patches per thread from float4 reads; rows are padded to 68 floats
// so that the reads of a warp fall on different banks. The blocks' sums go to `partial` and
// gradSumKernel adds them, in block order: the result does not depend on timing.
//
// 12 wavefronts of shared memory per 64 multiply-adds of a warp, so the multiply-adds bound a tile: 1.5
// GFLOP for 16 384 samples. One thread per sample with its activations in local memory, and one thread
// per parameter that went over the whole batch, took 1.9 ms for them, copies and all 2.05 ms. Now the kernel
// and the sum of its blocks take 94 us, measured as a step of training (B200): 29 us for each of a block's
// two tiles, at 40 % of the multiply-add rate, and some 35 us for the launches, the network's way into
// shared memory and the blocks' sums out of it. guideLossGrad takes 0.21 ms with the copies of its host arrays.
// ---------------------------------------------------------------------------------------------
constexpr int GB_THREADS = 256;
constexpr int GB_LD = 68, GB_LD0 = 12;  // row lengths in floats: 64-wide rows, and the 8 inputs
// row-padded weights of layer l in shared memory, then the biases
SKG_HD constexpr int gbW(int l) { return l == 0 ? 0 : 64 * GB_LD0 + (l - 1) * 64 * GB_LD; }
constexpr int GB_B = 64 * GB_LD0 + 3 * 64 * GB_LD + GUIDE_OUT * GB_LD;
constexpr int GB_X = GB_B + 4 * 64 + GUIDE_OUT;  // activations: inputs, 4 hidden layers, 2 delta buffers
constexpr int gbFloats(int S) { return GB_X + S * GB_LD0 + 6 * S * GB_LD + 4 * S; }
constexpr int GB_PARTIAL = GUIDE_NPARAMS + 1;  // per block: the gradient and the loss

SKG_D float dot4(float4 a, float4 b, float acc)
{
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
SKG_D float4 axpy4(float a, float4 x, float4 y)
{
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}
SKG_D float4 row4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Y[s][o] = act(b[o] + sum_i W[o][i] X[s][i]) for the S samples of a tile
template<int S, int K, int LD, int N, bool Relu>
SKG_D void tileForward(const float* W, const float* b, const float* X, float* Y)
{
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    constexpr int SJ = S / 16, OJ = (N + 15) / 16;
    float acc[SJ][OJ];
#pragma unroll
    for (int j = 0; j < OJ; ++j)
#pragma unroll
        for (int i = 0; i < SJ; ++i) acc[i][j] = tx + 16 * j < N ? b[tx + 16 * j] : 0.f;
#pragma unroll 4
    for (int k = 0; k < K; k += 4)
    {
        float4 w[OJ], x[SJ];
#pragma unroll
        for (int j = 0; j < OJ; ++j) w[j] = row4(W + min(tx + 16 * j, N - 1) * LD + k);
#pragma unroll
        for (int i = 0; i < SJ; ++i) x[i] = row4(X + (ty + 16 * i) * LD + k);
#pragma unroll
        for (int i = 0; i < SJ; ++i)
#pragma unroll
            for (int j = 0; j < OJ; ++j) acc[i][j] = dot4(w[j], x[i], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < SJ; ++i)
#pragma unroll
        for (int j = 0; j < OJ; ++j)
            if (tx + 16 * j < N) Y[(ty + 16 * i) * GB_LD + tx + 16 * j] = Relu ? fmaxf(acc[i][j], 0.f) : acc[i][j];
}

// P[s][i] = (sum_o W[o][i] D[s][o]) where the activation H[s][i] is positive, else 0
template<int S, int N>
SKG_D void tileBackward(const float* W, const float* D, const float* H, float* P)
{
    const int i0 = 4 * (threadIdx.x & 15), ty = threadIdx.x >> 4;
    constexpr int SJ = S / 16;
    float4 acc[SJ];
#pragma unroll
    for (int i = 0; i < SJ; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int o = 0; o < N; o += 4)
    {
        const float4 w0 = row4(W + o * GB_LD + i0), w1 = row4(W + (o + 1) * GB_LD + i0), w2 = row4(W + (o + 2) * GB_LD + i0),
                     w3 = row4(W + (o + 3) * GB_LD + i0);
#pragma unroll
        for (int i = 0; i < SJ; ++i)
        {
            const float4 d = row4(D + (ty + 16 * i) * GB_LD + o);
            acc[i] = axpy4(d.w, w3, axpy4(d.z, w2, axpy4(d.y, w1, axpy4(d.x, w0, acc[i]))));
        }
    }
#pragma unroll
    for (int i = 0; i < SJ; ++i)
    {
        const float4 h = row4(H + (ty + 16 * i) * GB_LD + i0);
        *reinterpret_cast<float4*>(P + (ty + 16 * i) * GB_LD + i0) =
            make_float4(h.x > 0.f ? acc[i].x : 0.f, h.y > 0.f ? acc[i].y : 0.f, h.z > 0.f ? acc[i].z : 0.f,
                        h.w > 0.f ? acc[i].w : 0.f);
    }
}

// G[r] += sum_s D[s][4 ty + r] H[s][4 tx ...] over the tile (rows of the weight gradient)
template<int S>
SKG_D void tileWeights(const float* D, const float* H, float4* G)
{
    const int i0 = 4 * (threadIdx.x & 15), o0 = 4 * (threadIdx.x >> 4);
#pragma unroll 4
    for (int s = 0; s < S; ++s)
    {
        const float4 d = row4(D + s * GB_LD + o0), h = row4(H + s * GB_LD + i0);
        G[0] = axpy4(d.x, h, G[0]);
        G[1] = axpy4(d.y, h, G[1]);
        G[2] = axpy4(d.z, h, G[2]);
        G[3] = axpy4(d.w, h, G[3]);
    }
}

// the part of a bias gradient of N outputs that a quarter of the block's threads sums: thread t the
// output t % 64 over every fourth sample from t / 64 on
template<int S>
SKG_D float tileBias(const float* D, int N)
{
    const int o = threadIdx.x & 63;
    float acc = 0.f;
    if (o < N)
        for (int s = threadIdx.x >> 6; s < S; s += 4) acc += D[s * GB_LD + o];
    return acc;
}

// Log density of the mixture of a sample's outputs `o` at the direction k, and the deltas of the
// outputs for the loss -w log q: GS neighbouring lanes share a sample, each with 8 / GS lobes. Returns
// the sample's loss in the first of them, 0 in the others.
template<int S>
SKG_D float tileHead(const float* o, const float* k, float w, bool valid, float* dout)
{
    constexpr int GS = GB_THREADS / S, J = GUIDE_LOBES / GS;
    const int q = threadIdx.x % GS;
    auto over = [](float v, bool mx) {
#pragma unroll
        for (int m = 1; m < GS; m <<= 1)
        {
            const float u = __shfl_xor_sync(0xffffffffu, v, m);
            v = mx ? fmaxf(v, u) : v + u;
        }
        return v;
    };
    float amax = -INFINITY;
#pragma unroll
    for (int j = 0; j < J; ++j) amax = fmaxf(amax, o[5 * (q * J + j)]);
    amax = over(amax, true);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j) sum += expf(o[5 * (q * J + j)] - amax);
    const float lse = amax + logf(over(sum, false));
    float logw[J], l[J], cs[J], kap[J], mu[J][3], len[J];
    float lmax = -INFINITY;
#pragma unroll
    for (int j = 0; j < J; ++j)
    {
        const float* r = o + 5 * (q * J + j);
        logw[j] = r[0] - lse;
        len[j] = sqrtf(r[1] * r[1] + r[2] * r[2] + r[3] * r[3]);
        const bool ok = len[j] > 1e-12f;
        mu[j][0] = ok ? r[1] / len[j] : 0.f;
        mu[j][1] = ok ? r[2] / len[j] : 0.f;
        mu[j][2] = ok ? r[3] / len[j] : 1.f;
        kap[j] = fminf(softplusf(r[4]) + GUIDE_KAPPA_MIN, GUIDE_KAPPA_MAX);
        cs[j] = mu[j][0] * k[0] + mu[j][1] * k[1] + mu[j][2] * k[2];
        l[j] = logw[j] + logVmf(kap[j], cs[j]);
        lmax = fmaxf(lmax, l[j]);
    }
    lmax = over(lmax, true);
    sum = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j) sum += expf(l[j] - lmax);
    const float logq = lmax + logf(over(sum, false));
#pragma unroll
    for (int j = 0; j < J; ++j)
    {
        const float r = expf(l[j] - logq);  // responsibility
        float g[5];
        g[0] = r - expf(logw[j]);
        // direction: mu = a / |a|, d log f / d a = kappa (k - (mu.k) mu) / |a|
        const float c = len[j] > 1e-12f ? r * kap[j] / len[j] : 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) g[1 + a] = c != 0.f ? c * (k[a] - cs[j] * mu[j][a]) : 0.f;
        // concentration: kappa = softplus(s) + kmin, clamped at kmax
        const float e = expf(-2.f * kap[j]);
        const float dlogf = 1.f / kap[j] - 2.f * e / (1.f - e) + (cs[j] - 1.f);
        const float sraw = o[5 * (q * J + j) + 4];
        const float dk = (softplusf(sraw) + GUIDE_KAPPA_MIN < GUIDE_KAPPA_MAX) ? 1.f / (1.f + expf(-sraw)) : 0.f;
        g[4] = r * dlogf * dk;
#pragma unroll
        for (int a = 0; a < 5; ++a) dout[5 * (q * J + j) + a] = valid ? -w * g[a] : 0.f;
    }
    return valid && q == 0 ? -w * logq : 0.f;
}

// position bin of a record (inputs 0..2 are the position scaled to [-1, 1])
SKG_D int positionBin(const GuideRecord& q, int nb)
{
    int idx = 0;
    for (int a = 0; a < 3; ++a)
    {
        int i = static_cast<int>((q.f[a] + 1.f) * 0.5f * static_cast<float>(nb));
        idx = idx * nb + min(nb - 1, max(0, i));
    }
    return idx;
}

// per position bin: sum of I (binSum) and number of records (binCount)
__global__ void binRecordsKernel(const GuideRecord* rec, unsigned long long n, int nb, float* binSum, unsigned* binCount)
{
    unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    int b = positionBin(rec[i], nb);
    atomicAdd(binSum + b, rec[i].I);
    atomicAdd(binCount + b, 1u);
}

__global__ void binMeanKernel(int nbins, const float* binSum, const unsigned* binCount, float* binMean)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < nbins) binMean[b] = binCount[b] ? binSum[b] / static_cast<float>(binCount[b]) : 0.f;
}

// the samples of a batch: explicit ones (gradient checks), or random pilot records of weight
// I / (mean I * B), or I / (mean I of the bin * B)
struct BatchSource
{
    const float *in, *k, *w;  // explicit samples: 8, 3 and 1 floats each
    const GuideRecord* rec;
    unsigned long long nrec;
    float invMeanI;
    int nb;
    const float* binMean;
    unsigned long long seed;
    unsigned step;

    SKG_D void load(int b, int n, float* x, float* dir, float& weight) const
    {
        if (in)
        {
            for (int i = 0; i < GUIDE_IN; ++i) x[i] = in[static_cast<size_t>(b) * GUIDE_IN + i];
            for (int i = 0; i < 3; ++i) dir[i] = k[3 * static_cast<size_t>(b) + i];
            weight = w[b];
            return;
        }
        U4 r = philox4x32_10(U4{step, static_cast<uint32_t>(b), 0x6d6c70u, 0u}, static_cast<uint32_t>(seed),
                             static_cast<uint32_t>(seed >> 32));
        const GuideRecord& q = rec[((static_cast<unsigned long long>(r.x) << 32) | r.y) % nrec];
        float wq = q.I * invMeanI;
        if (nb > 0)
        {
            float m = binMean[positionBin(q, nb)];
            wq = m > 0.f ? q.I / m : 0.f;
        }
        for (int i = 0; i < GUIDE_IN; ++i) x[i] = q.f[i];
        for (int i = 0; i < 3; ++i) dir[i] = q.k[i];
        weight = wq / static_cast<float>(n);
    }
};

template<int S>
__global__ void __launch_bounds__(GB_THREADS, 1) batchKernel(const float* __restrict__ P, int n, BatchSource src,
                                                             float* __restrict__ partial)
{
    extern __shared__ __align__(16) float sm[];
    float* X = sm + GB_X;
    float* H = X + S * GB_LD0;          // 4 hidden layers
    float* D0 = H + 4 * S * GB_LD;      // delta buffers (the raw outputs start in the first)
    float* D1 = D0 + S * GB_LD;
    float* K = D1 + S * GB_LD;          // direction and weight of each sample
    constexpr int GS = GB_THREADS / S;
    // the network into its padded rows
    for (int l = 0; l < GUIDE_LAYERS; ++l)
    {
        const int nin = guideDimIn(l), nout = guideDimOut(l), ld = l == 0 ? GB_LD0 : GB_LD;
        const float* W = P + guideParamOffset(l);
        for (int i = threadIdx.x; i < nout * nin; i += GB_THREADS) sm[gbW(l) + (i / nin) * ld + i % nin] = W[i];
        for (int i = threadIdx.x; i < nout; i += GB_THREADS) sm[GB_B + 64 * l + i] = W[nout * nin + i];
    }
    float4 G[4][4];  // layers 1 - 4
    float g0[2] = {0.f, 0.f};  // layer 0: outputs o, o + 32 of input i = t % 8
    float gb[GUIDE_LAYERS];
    for (int l = 0; l < 4; ++l)
        for (int r = 0; r < 4; ++r) G[l][r] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int l = 0; l < GUIDE_LAYERS; ++l) gb[l] = 0.f;
    float loss = 0.f;

    // an even share of the batch per block
    const int lo = static_cast<int>(static_cast<long long>(n) * blockIdx.x / gridDim.x);
    const int hi = static_cast<int>(static_cast<long long>(n) * (blockIdx.x + 1) / gridDim.x);
    for (int b0 = lo; b0 < hi; b0 += S)
    {
        __syncthreads();
        if (threadIdx.x < S)
        {
            float x[GUIDE_IN] = {}, dir[3] = {0.f, 0.f, 1.f}, w = 0.f;
            if (b0 + static_cast<int>(threadIdx.x) < hi) src.load(b0 + threadIdx.x, n, x, dir, w);
            for (int i = 0; i < GUIDE_IN; ++i) X[threadIdx.x * GB_LD0 + i] = x[i];
            for (int i = 0; i < 3; ++i) K[4 * threadIdx.x + i] = dir[i];
            K[4 * threadIdx.x + 3] = w;
        }
        __syncthreads();
        tileForward<S, GUIDE_IN, GB_LD0, 64, true>(sm + gbW(0), sm + GB_B, X, H);
        __syncthreads();
        for (int l = 1; l < 4; ++l)
        {
            tileForward<S, 64, GB_LD, 64, true>(sm + gbW(l), sm + GB_B + 64 * l, H + (l - 1) * S * GB_LD, H + l * S * GB_LD);
            __syncthreads();
        }
        tileForward<S, 64, GB_LD, GUIDE_OUT, false>(sm + gbW(4), sm + GB_B + 256, H + 3 * S * GB_LD, D0);
        __syncthreads();
        {
            const int s = threadIdx.x / GS;
            loss += tileHead<S>(D0 + s * GB_LD, K + 4 * s, K[4 * s + 3], b0 + s < hi, D1 + s * GB_LD);
        }
        __syncthreads();
        // back through the layers: delta_l = (W_{l+1}^T delta_{l+1}) * relu'(h_l)
        if (threadIdx.x >> 4 < GUIDE_OUT / 4) tileWeights<S>(D1, H + 3 * S * GB_LD, G[3]);
        gb[4] += tileBias<S>(D1, GUIDE_OUT);
        tileBackward<S, GUIDE_OUT>(sm + gbW(4), D1, H + 3 * S * GB_LD, D0);
        __syncthreads();
        float *d = D0, *dn = D1;
#pragma unroll
        for (int l = 3; l >= 1; --l)
        {
            tileWeights<S>(d, H + (l - 1) * S * GB_LD, G[l - 1]);
            gb[l] += tileBias<S>(d, 64);
            tileBackward<S, 64>(sm + gbW(l), d, H + (l - 1) * S * GB_LD, dn);
            __syncthreads();
            float* t = d;
            d = dn;
            dn = t;
        }
        gb[0] += tileBias<S>(d, 64);
        const int o = threadIdx.x >> 3, i = threadIdx.x & 7;
        for (int s = 0; s < S; ++s)
        {
            const float x = X[s * GB_LD0 + i];
            g0[0] = fmaf(d[s * GB_LD + o], x, g0[0]);
            g0[1] = fmaf(d[s * GB_LD + o + 32], x, g0[1]);
        }
    }
    // this block's sums, in the layout of the parameters
    float* out = partial + static_cast<size_t>(blockIdx.x) * GB_PARTIAL;
    const int i0 = 4 * (threadIdx.x & 15), o0 = 4 * (threadIdx.x >> 4);
    for (int r = 0; r < 2; ++r) out[((threadIdx.x >> 3) + 32 * r) * GUIDE_IN + (threadIdx.x & 7)] = g0[r];
#pragma unroll
    for (int l = 1; l < GUIDE_LAYERS; ++l)
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (o0 + r < guideDimOut(l))
            {
                float* at = out + guideParamOffset(l) + (o0 + r) * 64 + i0;
                at[0] = G[l - 1][r].x;
                at[1] = G[l - 1][r].y;
                at[2] = G[l - 1][r].z;
                at[3] = G[l - 1][r].w;
            }
    __syncthreads();
#pragma unroll
    for (int l = 0; l < GUIDE_LAYERS; ++l) X[l * GB_THREADS + threadIdx.x] = gb[l];
    X[GUIDE_LAYERS * GB_THREADS + threadIdx.x] = loss;
    __syncthreads();
    for (int t = threadIdx.x; t < 64 * GUIDE_LAYERS; t += GB_THREADS)
    {
        const int l = t / 64, oo = t % 64;
        const float* q = X + l * GB_THREADS + oo;
        if (oo < guideDimOut(l))
            out[guideParamOffset(l) + guideDimOut(l) * guideDimIn(l) + oo] = (q[0] + q[64]) + (q[128] + q[192]);
    }
    if (threadIdx.x < 32)
    {
        float v = 0.f;
        for (int t = threadIdx.x; t < GB_THREADS; t += 32) v += X[GUIDE_LAYERS * GB_THREADS + t];
        for (int m = 16; m > 0; m >>= 1) v += __shfl_down_sync(0xffffffffu, v, m);
        if (threadIdx.x == 0) out[GUIDE_NPARAMS] = v;
    }
}

// grad[p] = the blocks' sums added in block order (p = GUIDE_NPARAMS: the loss), and with `lr` > 0 the
// Adam step of parameter p
__global__ void __launch_bounds__(128) gradSumKernel(const float* __restrict__ partial, int blocks, float* grad, float* P,
                                                     float* m, float* v, float lr, float b1, float b2, float eps, float c1,
                                                     float c2, float clip)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= GB_PARTIAL) return;
    float acc = 0.f;
#pragma unroll 8
    for (int b = 0; b < blocks; ++b) acc += partial[static_cast<size_t>(b) * GB_PARTIAL + p];
    grad[p] = acc;
    if (!(lr > 0.f) || p >= GUIDE_NPARAMS) return;
    float gp = fminf(clip, fmaxf(-clip, acc));
    if (!isfinite(gp)) gp = 0.f;
    float mp = b1 * m[p] + (1.f - b1) * gp;
    float vp = b2 * v[p] + (1.f - b2) * gp * gp;
    m[p] = mp;
    v[p] = vp;
    P[p] -= lr * (mp / c1) / (sqrtf(vp / c2) + eps);
}

template<typename T>
cudaError_t allocN(T** p, size_t n)
{
    return cudaMalloc(reinterpret_cast<void**>(p), std::max<size_t>(n, 1) * sizeof(T));
}

// Tiles of 64 samples, which read shared memory half as often per multiply-add, or of 32 for a batch of
// at most 32 per SM: a block then has one tile of either size, and the small one is done sooner. A step of
// training with tiles of 32 / 64: 500 samples 43 / 53 us, 4736 (32 per SM) 53 / 59, 4737 72 / 59, 9472 73 / 65, 16 384
// 111 / 94.
cudaError_t launchBatch(GuideState* g, int n, const BatchSource& src, int numSMs, int* blocks)
{
    const bool small = n <= 32 * numSMs;
    const int S = small ? 32 : 64;
    const size_t bytes = gbFloats(S) * sizeof(float);
    const void* f = small ? reinterpret_cast<const void*>(batchKernel<32>) : reinterpret_cast<const void*>(batchKernel<64>);
    cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
    *blocks = std::max(1, std::min(numSMs, (n + S - 1) / S));
    if (g->partialBlocks < *blocks)
    {
        cudaFree(g->partial);
        g->partial = nullptr;
        g->partialBlocks = 0;
        e = allocN(&g->partial, static_cast<size_t>(*blocks) * GB_PARTIAL);
        if (e != cudaSuccess) return e;
        g->partialBlocks = *blocks;
    }
    if (small)
        batchKernel<32><<<*blocks, GB_THREADS, bytes>>>(g->params, n, src, g->partial);
    else
        batchKernel<64><<<*blocks, GB_THREADS, bytes>>>(g->params, n, src, g->partial);
    return cudaGetLastError();
}

// tensor-core forward pass of n explicit samples (tests): 128 samples per CTA
__global__ void __launch_bounds__(GM_TILE) inferKernel(const unsigned char* blob, int n, const float* in, float* out,
                                                       int* err)
{
    extern __shared__ __align__(128) unsigned char smem[];
    GuideTile t;
    guideTileBegin(t, smem, blob);
    for (int tile = blockIdx.x; tile * GM_TILE < n; tile += gridDim.x)
    {
        int i = tile * GM_TILE + threadIdx.x;
        float f[GUIDE_IN], o[GUIDE_OUT];
        for (int k = 0; k < GUIDE_IN; ++k) f[k] = i < n ? in[static_cast<size_t>(i) * GUIDE_IN + k] : 0.f;
        if (!guideTileForward(t, f, o))
        {
            if (threadIdx.x == 0) atomicOr(err, 1);
            break;  // uniform across the CTA
        }
        if (i < n)
            for (int k = 0; k < GUIDE_OUT; ++k) out[static_cast<size_t>(i) * GUIDE_OUT + k] = o[k];
    }
    guideTileEnd(t);
}

// FP32 (CUDA-core) forward pass of n explicit samples (reference for the tensor-core pass)
__global__ void inferFp32Kernel(const float* P, int n, const float* in, float* out)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    float h[256];
    mlpForward(P, in + static_cast<size_t>(b) * GUIDE_IN, h, out + static_cast<size_t>(b) * GUIDE_OUT);
}

// sum of the records' downstream luminosities (set at the end of each recorded history)
__global__ void sumRecordsKernel(const GuideRecord* rec, unsigned long long n, double* sumI)
{
    unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x;
    double v = i < n ? static_cast<double>(rec[i].I) : 0.;
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(sumI, v);
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// state
// ---------------------------------------------------------------------------------------------
GuideState::~GuideState()
{
    void* ps[] = {params, blob, adamM, adamV, grad, records, recCount, batchIn, partial, importance, errFlag, binMean};
    for (void* p : ps)
        if (p) cudaFree(p);
}

cudaError_t guideEnsure(skgpu_ctx* ctx)
{
    if (ctx->guide) return cudaSuccess;
    GuideState* g = new GuideState();
    cudaError_t e = allocN(&g->params, GUIDE_NPARAMS);
    if (e == cudaSuccess) e = allocN(&g->blob, GM_BLOB_BYTES);
    if (e == cudaSuccess) e = allocN(&g->adamM, GUIDE_NPARAMS);
    if (e == cudaSuccess) e = allocN(&g->adamV, GUIDE_NPARAMS);
    if (e == cudaSuccess) e = allocN(&g->grad, GB_PARTIAL);
    if (e == cudaSuccess) e = allocN(&g->recCount, 1);
    if (e == cudaSuccess) e = allocN(&g->errFlag, 1);
    if (e == cudaSuccess) e = cudaMemset(g->recCount, 0, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(g->errFlag, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(inferKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GM_SMEM_BYTES);
    if (e != cudaSuccess)
    {
        delete g;
        return e;
    }
    ctx->guide = g;
    return cudaSuccess;
}

void guideDestroy(skgpu_ctx* ctx)
{
    delete ctx->guide;
    ctx->guide = nullptr;
}

cudaError_t guideSetParams(skgpu_ctx* ctx, const float* host)
{
    GuideState* g = ctx->guide;
    cudaError_t e = cudaMemcpy(g->params, host, GUIDE_NPARAMS * sizeof(float), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return e;
    e = cudaMemset(g->adamM, 0, GUIDE_NPARAMS * sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(g->adamV, 0, GUIDE_NPARAMS * sizeof(float));
    g->adamStep = 0;
    g->hasParams = true;
    return e == cudaSuccess ? guideRepack(ctx) : e;
}

cudaError_t guideGetParams(skgpu_ctx* ctx, float* host)
{
    return cudaMemcpy(host, ctx->guide->params, GUIDE_NPARAMS * sizeof(float), cudaMemcpyDeviceToHost);
}

// BF16 blob of the inference kernel from the FP32 master parameters
cudaError_t guideRepack(skgpu_ctx* ctx)
{
    GuideState* g = ctx->guide;
    std::vector<float> p(GUIDE_NPARAMS);
    cudaError_t e = cudaMemcpy(p.data(), g->params, p.size() * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    std::vector<unsigned char> blob(GM_BLOB_BYTES);
    guidePackBlob(p.data(), blob.data());
    return cudaMemcpy(g->blob, blob.data(), blob.size(), cudaMemcpyHostToDevice);
}

// device space for the explicit samples of a batch, kept for the next call (12 floats a sample)
static cudaError_t ensureBatch(GuideState* g, int n)
{
    if (g->batchRows >= n) return cudaSuccess;
    cudaFree(g->batchIn);
    g->batchIn = nullptr;
    g->batchRows = 0;
    cudaError_t e = allocN(&g->batchIn, static_cast<size_t>(n) * (GUIDE_IN + 4));
    if (e == cudaSuccess) g->batchRows = n;
    return e;
}

cudaError_t guideLossGrad(skgpu_ctx* ctx, int n, const float* in, const float* k, const float* w, float* loss,
                          float* grad)
{
    GuideState* g = ctx->guide;
    cudaError_t e = ensureBatch(g, n);
    if (e != cudaSuccess) return e;
    const size_t rows = static_cast<size_t>(n);
    float *dIn = g->batchIn, *dK = dIn + rows * GUIDE_IN, *dW = dK + 3 * rows;
    e = cudaMemcpy(dIn, in, rows * GUIDE_IN * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dK, k, 3 * rows * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dW, w, rows * sizeof(float), cudaMemcpyHostToDevice);
    BatchSource src{};
    src.in = dIn;
    src.k = dK;
    src.w = dW;
    int blocks = 0;
    if (e == cudaSuccess) e = launchBatch(g, n, src, ctx->numSMs, &blocks);
    if (e == cudaSuccess)
    {
        gradSumKernel<<<(GB_PARTIAL + 127) / 128, 128>>>(g->partial, blocks, g->grad, nullptr, nullptr, nullptr, 0.f, 0.f,
                                                         0.f, 0.f, 1.f, 1.f, 0.f);
        e = cudaGetLastError();
    }
    float out[GB_PARTIAL];
    if (e == cudaSuccess) e = cudaMemcpy(out, g->grad, sizeof out, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    std::copy(out, out + GUIDE_NPARAMS, grad);
    *loss = out[GUIDE_NPARAMS];
    return cudaSuccess;
}

cudaError_t guideInfer(skgpu_ctx* ctx, int n, const float* in, float* out, int tensorCores, int* deviceErr)
{
    GuideState* g = ctx->guide;
    float *dIn = nullptr, *dOut = nullptr;
    cudaError_t e = allocN(&dIn, static_cast<size_t>(n) * GUIDE_IN);
    if (e == cudaSuccess) e = allocN(&dOut, static_cast<size_t>(n) * GUIDE_OUT);
    if (e == cudaSuccess) e = cudaMemcpy(dIn, in, static_cast<size_t>(n) * GUIDE_IN * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(g->errFlag, 0, sizeof(int));
    if (e == cudaSuccess)
    {
        if (tensorCores)
        {
            int tiles = (n + GM_TILE - 1) / GM_TILE;
            int grid = std::max(1, std::min(tiles, 4 * ctx->numSMs));
            inferKernel<<<grid, GM_TILE, GM_SMEM_BYTES>>>(g->blob, n, dIn, dOut, g->errFlag);
        }
        else
        {
            inferFp32Kernel<<<(n + 127) / 128, 128>>>(g->params, n, dIn, dOut);
        }
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(out, dOut, static_cast<size_t>(n) * GUIDE_OUT * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(deviceErr, g->errFlag, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(dIn);
    cudaFree(dOut);
    return e;
}

cudaError_t guideEnsureRecords(skgpu_ctx* ctx, unsigned long long capacity)
{
    GuideState* g = ctx->guide;
    if (g->recCapacity != capacity)
    {
        cudaFree(g->records);
        g->records = nullptr;
        g->recCapacity = 0;
        cudaError_t e = allocN(&g->records, capacity);
        if (e != cudaSuccess) return e;
        g->recCapacity = capacity;
    }
    return cudaMemset(g->recCount, 0, sizeof(unsigned long long));
}

cudaError_t guideRecordCount(skgpu_ctx* ctx, unsigned long long* n)
{
    cudaError_t e = cudaMemcpy(n, ctx->guide->recCount, sizeof *n, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) *n = std::min(*n, ctx->guide->recCapacity);
    return e;
}

cudaError_t guideFetchRecords(skgpu_ctx* ctx, unsigned long long n, float* out /* n x 13: f[8], k[3], I, L */)
{
    std::vector<GuideRecord> r(n);
    cudaError_t e = cudaMemcpy(r.data(), ctx->guide->records, n * sizeof(GuideRecord), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    for (unsigned long long i = 0; i < n; ++i)
    {
        float* o = out + 13 * i;
        for (int k = 0; k < GUIDE_IN; ++k) o[k] = r[i].f[k];
        for (int k = 0; k < 3; ++k) o[8 + k] = r[i].k[k];
        o[11] = r[i].I;
        o[12] = r[i].L;
    }
    return cudaSuccess;
}

cudaError_t guideTrain(skgpu_ctx* ctx, int steps, int batch, float lr, unsigned long long seed, float* lossOut)
{
    GuideState* g = ctx->guide;
    unsigned long long nrec = 0;
    cudaError_t e = guideRecordCount(ctx, &nrec);
    if (e != cudaSuccess) return e;
    if (nrec == 0) return cudaErrorInvalidValue;
    // mean downstream luminosity of the records (weights are I / mean I)
    double* dSum = nullptr;
    e = allocN(&dSum, 1);
    if (e == cudaSuccess) e = cudaMemset(dSum, 0, sizeof(double));
    if (e == cudaSuccess)
    {
        sumRecordsKernel<<<static_cast<unsigned>((nrec + 255) / 256), 256>>>(g->records, nrec, dSum);
        e = cudaGetLastError();
    }
    double sumI = 0.;
    if (e == cudaSuccess) e = cudaMemcpy(&sumI, dSum, sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(dSum);
    if (e != cudaSuccess) return e;
    if (!(sumI > 0.)) return cudaErrorInvalidValue;  // the pilot detected nothing downstream
    float invMeanI = static_cast<float>(static_cast<double>(nrec) / sumI);
    int nb = g->positionBins;
    if (nb > 0)
    {
        int nbins = nb * nb * nb;
        float* binSum = nullptr;
        unsigned* binCount = nullptr;
        cudaFree(g->binMean);
        g->binMean = nullptr;
        e = allocN(&g->binMean, nbins);
        if (e == cudaSuccess) e = allocN(&binSum, nbins);
        if (e == cudaSuccess) e = allocN(&binCount, nbins);
        if (e == cudaSuccess) e = cudaMemset(binSum, 0, nbins * sizeof(float));
        if (e == cudaSuccess) e = cudaMemset(binCount, 0, nbins * sizeof(unsigned));
        if (e == cudaSuccess)
        {
            binRecordsKernel<<<static_cast<unsigned>((nrec + 255) / 256), 256>>>(g->records, nrec, nb, binSum, binCount);
            binMeanKernel<<<(nbins + 255) / 256, 256>>>(nbins, binSum, binCount, g->binMean);
            e = cudaGetLastError();
        }
        cudaFree(binSum);
        cudaFree(binCount);
        if (e != cudaSuccess) return e;
    }
    BatchSource src{};
    src.rec = g->records;
    src.nrec = nrec;
    src.invMeanI = invMeanI;
    src.nb = nb;
    src.binMean = g->binMean;
    src.seed = seed;
    const float b1 = 0.9f, b2 = 0.999f;
    float lastLoss = 0.f;
    for (int it = 0; it < steps && e == cudaSuccess; ++it)
    {
        src.step = static_cast<unsigned>(g->adamStep);
        int blocks = 0;
        e = launchBatch(g, batch, src, ctx->numSMs, &blocks);
        g->adamStep++;
        float c1 = 1.f - std::pow(b1, static_cast<float>(g->adamStep));
        float c2 = 1.f - std::pow(b2, static_cast<float>(g->adamStep));
        if (e == cudaSuccess)
        {
            gradSumKernel<<<(GB_PARTIAL + 127) / 128, 128>>>(g->partial, blocks, g->grad, g->params, g->adamM, g->adamV, lr,
                                                             b1, b2, 1e-8f, c1, c2, 10.f);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess && steps > 0)
        e = cudaMemcpy(&lastLoss, g->grad + GUIDE_NPARAMS, sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = guideRepack(ctx);
    if (lossOut) *lossOut = lastLoss;
    return e;
}

}  // namespace skg
