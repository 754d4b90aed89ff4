// mlp_train.cu - forward, backward and Adam kernels of the learned start
// value (the network of mlp.cuh), and the C entry points that train it.
//
// Loss: mean squared error of y = log(p*/p_L) over a batch.  A CTA takes 64
// samples at a time, four threads a sample (eight units of each layer each),
// and then reduces the per-sample weight gradients from shared memory (each
// weight gradient is a sum over the samples of an outer-product term, four
// W2 entries a thread); the sums of its samples go to the global gradient by
// one atomic each.  The last CTA of a training batch takes the Adam step, so a
// batch is one launch.  The network is too small (1313 weights) for
// tensor-core tiles to pay; everything is FP32 SIMT.  A batch of 16384 is
// bound by the latency of a CTA's phases: with one thread a sample, 256 samples
// a CTA and the Adam step as a second launch it took 34 us on 64 SMs, as here
// 12 us on all SMs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../../include/asteriy_gb300.h"
#include "mlp.cuh"

namespace ast {
int cuda_fail(cudaError_t e, const char* what);
}

using namespace ast;

namespace {

constexpr int kB = 64;           // samples of a CTA at a time
constexpr int kG = 4;            // threads per sample
constexpr int kT = kB * kG;
constexpr int kBatchUnit = 256;  // ast_mlp_train's batches are multiples of this
constexpr int kH = kMlpH, kI = kMlpIn;
constexpr int kU = kH / kG;      // units of a thread in each layer
constexpr int kPad = kH + 2;     // row pitch of the per-sample activations (pairs aligned)
static_assert(kH * kH == 4 * kT, "four W2 entries a thread");

struct GradSmem {
    alignas(16) float W[kMlpParams + 3];
    float X[kB][kI + 1];
    alignas(8) float H1[kB][kPad];
    alignas(8) float H2[kB][kPad];
    alignas(8) float DZ1[kB][kPad];
    alignas(8) float DZ2[kB][kPad];
    float Y[kG][kB];
    float DY[kB];
    int last;
};

// the Adam step that ends a training batch (shift/scale are fixed): the
// moments and the CTAs' ticket (null: no step)
// The CTAs' atomics on one address follow one another at some 10 ns each, so
// in training they are spread over kSums copies of the gradient, which the
// step adds up: a batch of 16384 20 -> 12 us with it
// and with every load of the step in flight at once.
constexpr int kSums = 4, kSumPitch = (kMlpParams + 3) / 4 * 4;
struct Adam {
    float *m1, *m2;
    unsigned* ticket;
    float lr, b1, b2, eps, c1, c2;
};

// samples: n records of AST_RECORD_FLOATS (x[6], target, ...); idx: optional
// permutation (sample i of this pass is samples[idx[i]]).  grad (1325 floats,
// the shift/scale slots stay zero; with Adam kSums of them) and loss_sum are
// accumulated; with Adam, W_g is updated and grad zeroed.  W_g and grad lie on
// 16 bytes and W_g has kSumPitch floats.
__global__ void __launch_bounds__(kT) mlp_grad_kernel(float* __restrict__ W_g, const float* __restrict__ samples,
                                                      const int* __restrict__ idx, long long first, long long count,
                                                      float inv_count, float* grad, float* loss_sum, Adam adam)
{
    __shared__ GradSmem s;
    const int t = threadIdx.x, q = t % kB, j0 = t / kB * kU;   // a warp's threads: one group of units
    // the mapped inputs of sample base + q; its target
    auto features = [&](long long base) {
        const bool valid = base + q < count;
        const float* rec = samples;
        if (valid) rec += (idx ? (long long)idx[first + base + q] : first + base + q) * AST_RECORD_FLOATS;
        for (int i = t / kB; i < kI; i += kG)
            s.X[q][i] = valid ? (mlp_map(i, rec[i]) - __ldcg(&W_g[kOffShift + i])) * __ldcg(&W_g[kOffScale + i]) : 0.0f;
        return valid ? rec[6] : 0.0f;
    };
    // In training a launch may begin while the batch before it still runs:
    // up to the wait it reads only what no launch writes (the samples and
    // their order, shift and scale) and writes only shared memory.  The
    // weights are read past L1, where the early reads may have left old ones.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long base0 = (long long)blockIdx.x * kB;
    float target = features(base0);
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int r = 0; r < kSumPitch / 4; r += kT)
        if (r + t < kSumPitch / 4)
            reinterpret_cast<float4*>(s.W)[r + t] = __ldcg(reinterpret_cast<const float4*>(W_g) + r + t);
    // this thread's gradient entries: W2[k0..k0+1][l0..l0+1], then the others in turn
    const int k0 = t / (kH / 2) * 2, l0 = t % (kH / 2) * 2;
    constexpr int kRest = kH * kI + 3 * kH + 1, kR = (kRest + kT - 1) / kT;
    float g2[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gr[kR];
#pragma unroll
    for (int r = 0; r < kR; r++) gr[r] = 0.0f;
    float loss = 0.0f;
    for (long long base = base0; base < count; base += (long long)gridDim.x * kB) {
        if (base != base0) {
            __syncthreads();   // the last block's activations are read
            target = features(base);
        }
        __syncthreads();
        const bool valid = base + q < count;
        // forward
        float z1[kU], z2[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) {
            float z = s.W[kOffB1 + j0 + u];
#pragma unroll
            for (int i = 0; i < kI; i++) z = fmaf(s.W[kOffW1 + (j0 + u) * kI + i], s.X[q][i], z);
            z1[u] = z;
            s.H1[q][j0 + u] = silu(z);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kU; u++) z2[u] = s.W[kOffB2 + j0 + u];
#pragma unroll
        for (int j = 0; j < kH; j += 4) {
            const float2 ha = *reinterpret_cast<const float2*>(&s.H1[q][j]);
            const float2 hb = *reinterpret_cast<const float2*>(&s.H1[q][j + 2]);
#pragma unroll
            for (int u = 0; u < kU; u++) {
                const float4 w = *reinterpret_cast<const float4*>(&s.W[kOffW2 + (j0 + u) * kH + j]);
                z2[u] = fmaf(w.w, hb.y, fmaf(w.z, hb.x, fmaf(w.y, ha.y, fmaf(w.x, ha.x, z2[u]))));
            }
        }
        float y = 0.0f;
#pragma unroll
        for (int u = 0; u < kU; u++) {
            const float h2 = silu(z2[u]);
            s.H2[q][j0 + u] = h2;
            y = fmaf(s.W[kOffW3 + j0 + u], h2, y);
        }
        s.Y[t / kB][q] = y;
        __syncthreads();
        // backward through the output and the second layer
        y = s.W[kOffB3] + ((s.Y[0][q] + s.Y[1][q]) + (s.Y[2][q] + s.Y[3][q]));
        const float err = valid ? y - target : 0.0f;
        const float dy = 2.0f * err * inv_count;
        if (t < kB) {
            s.DY[q] = dy;
            loss = fmaf(err, err, loss);
        }
#pragma unroll
        for (int u = 0; u < kU; u++) s.DZ2[q][j0 + u] = dy * s.W[kOffW3 + j0 + u] * silu_grad(z2[u]);
        __syncthreads();
        float dh1[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) dh1[u] = 0.0f;
#pragma unroll 8
        for (int k = 0; k < kH; k++) {
            const float dz2 = s.DZ2[q][k];
#pragma unroll
            for (int u = 0; u < kU; u += 4) {
                const float4 w = *reinterpret_cast<const float4*>(&s.W[kOffW2 + k * kH + j0 + u]);
                dh1[u] = fmaf(w.x, dz2, dh1[u]);
                dh1[u + 1] = fmaf(w.y, dz2, dh1[u + 1]);
                dh1[u + 2] = fmaf(w.z, dz2, dh1[u + 2]);
                dh1[u + 3] = fmaf(w.w, dz2, dh1[u + 3]);
            }
        }
#pragma unroll
        for (int u = 0; u < kU; u++) s.DZ1[q][j0 + u] = dh1[u] * silu_grad(z1[u]);
        __syncthreads();
        // the outer-product sums over the CTA's samples
#pragma unroll 8
        for (int n = 0; n < kB; n++) {             // W2[k][l]: sum_n dz2[n][k] h1[n][l]
            const float2 d = *reinterpret_cast<const float2*>(&s.DZ2[n][k0]);
            const float2 h = *reinterpret_cast<const float2*>(&s.H1[n][l0]);
            g2[0] = fmaf(d.x, h.x, g2[0]);
            g2[1] = fmaf(d.x, h.y, g2[1]);
            g2[2] = fmaf(d.y, h.x, g2[2]);
            g2[3] = fmaf(d.y, h.y, g2[3]);
        }
#pragma unroll
        for (int r = 0; r < kR; r++) {
            int o = t + r * kT;
            float acc = 0.0f;
            if (o < kH * kI) {                     // W1[j][i]: sum_n dz1[n][j] x[n][i]
                const int j = o / kI, i = o - j * kI;
#pragma unroll 8
                for (int n = 0; n < kB; n++) acc = fmaf(s.DZ1[n][j], s.X[n][i], acc);
            } else if ((o -= kH * kI) < kH) {      // b1[j]
#pragma unroll 8
                for (int n = 0; n < kB; n++) acc += s.DZ1[n][o];
            } else if ((o -= kH) < kH) {           // b2[k]
#pragma unroll 8
                for (int n = 0; n < kB; n++) acc += s.DZ2[n][o];
            } else if ((o -= kH) < kH) {           // w3[k]: sum_n dy[n] h2[n][k]
#pragma unroll 8
                for (int n = 0; n < kB; n++) acc = fmaf(s.DY[n], s.H2[n][o], acc);
            } else if (o == kH) {                  // b3
                for (int n = 0; n < kB; n++) acc += s.DY[n];
            }
            gr[r] += acc;
        }
    }
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if ((t & 31) == 0 && loss != 0.0f) atomicAdd(loss_sum, loss);
    if (adam.ticket) grad += blockIdx.x % kSums * kSumPitch;
    atomicAdd(reinterpret_cast<float2*>(&grad[kOffW2 + k0 * kH + l0]), make_float2(g2[0], g2[1]));
    atomicAdd(reinterpret_cast<float2*>(&grad[kOffW2 + (k0 + 1) * kH + l0]), make_float2(g2[2], g2[3]));
#pragma unroll
    for (int r = 0; r < kR; r++) {
        // W1 and b1 lie before W2, then b2, w3 and b3 after it
        const int o = t + r * kT, lo = kH * kI + kH;
        if (o < kRest) atomicAdd(&grad[o < lo ? kOffW1 + o : kOffB2 + o - lo], gr[r]);
    }
    if (!adam.ticket) return;
    // the CTA that gives last takes the step
    __threadfence();
    __syncthreads();
    if (t == 0) s.last = atomicAdd(adam.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s.last) return;
    __threadfence();
    if (t == 0) *adam.ticket = 0u;
    grad -= blockIdx.x % kSums * kSumPitch;
    constexpr int kP = (kMlpParams - kOffW1 + kT - 1) / kT;
    float g[kP], a[kP], v[kP];
#pragma unroll
    for (int r = 0; r < kP; r++) {     // every load in flight before the first is used
        const int i = kOffW1 + t + r * kT;
        if (i >= kMlpParams) continue;
        g[r] = 0.0f;
#pragma unroll
        for (int c = 0; c < kSums; c++) g[r] += __ldcg(&grad[c * kSumPitch + i]);
        a[r] = __ldcg(&adam.m1[i]);
        v[r] = __ldcg(&adam.m2[i]);
    }
#pragma unroll
    for (int r = 0; r < kP; r++) {
        const int i = kOffW1 + t + r * kT;
        if (i >= kMlpParams) continue;
#pragma unroll
        for (int c = 0; c < kSums; c++) grad[c * kSumPitch + i] = 0.0f;
        a[r] = adam.b1 * a[r] + (1.0f - adam.b1) * g[r];
        v[r] = adam.b2 * v[r] + (1.0f - adam.b2) * g[r] * g[r];
        adam.m1[i] = a[r];
        adam.m2[i] = v[r];
        W_g[i] = s.W[i] - adam.lr * (a[r] * adam.c1) / (sqrtf(v[r] * adam.c2) + adam.eps);
    }
}
static_assert(kOffW1 + kH * kI == kOffB1 && kOffB1 + kH == kOffW2 && kOffB2 + kH == kOffW3 && kOffW3 + kH == kOffB3 && kOffW2 % 2 == 0,
              "the parameter block's order");

// CTAs of a pass over count samples: at most two per SM of a GB300
int grad_blocks(long long count) { return (int)std::min<long long>((count + kB - 1) / kB, 304); }

__global__ void mlp_forward_kernel(const float* __restrict__ W_g, const float* __restrict__ x, long long n,
                                   int stride, float* __restrict__ y)
{
    __shared__ float W[kMlpParams];
    for (int i = threadIdx.x; i < kMlpParams; i += blockDim.x) W[i] = W_g[i];
    __syncthreads();
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float xin[kI];
#pragma unroll
    for (int i = 0; i < kI; i++) xin[i] = x[k * stride + i];
    y[k] = mlp_forward(W, xin);
}

thread_local std::string g_err;

struct DevBuf {
    void* p = nullptr;
    ~DevBuf() { cudaFree(p); }
    cudaError_t alloc(size_t bytes) { return cudaMalloc(&p, bytes); }
    template <typename T> T* as() { return (T*)p; }
};

#define TRY(call)                                                   \
    do {                                                            \
        cudaError_t e_ = (call);                                    \
        if (e_ != cudaSuccess) return ast::cuda_fail(e_, #call);    \
    } while (0)

}  // namespace

extern "C" {

// Initial parameters: input shift/scale = mean and 1/std of the samples'
// mapped features (log of the positive ratios, asinh of the velocity jump),
// weights ~ U(-sqrt(6/(fan_in+fan_out)), +...) from mt19937_64(seed),
// biases 0, output bias = mean target.  Host function.
int ast_mlp_init(const float* samples, int64_t n, uint64_t seed, float* params)
{
    if (!samples || !params || n < 2) return AST_ERR_INVALID;
    std::memset(params, 0, sizeof(float) * AST_MLP_NPARAM);
    double mean[kI] = {0}, sq[kI] = {0}, ty = 0.0;
    for (int64_t k = 0; k < n; k++) {
        const float* r = samples + k * AST_RECORD_FLOATS;
        for (int i = 0; i < kI; i++) {
            double v = r[i];
            if (i == 0 || i == 1 || i == 3) v = std::log(v);
            else if (i == 2) v = std::asinh(v);
            mean[i] += v;
            sq[i] += v * v;
        }
        ty += r[6];
    }
    for (int i = 0; i < kI; i++) {
        const double m = mean[i] / n;
        const double var = std::max(sq[i] / n - m * m, 0.0);
        params[kOffShift + i] = (float)m;
        params[kOffScale + i] = (float)(var > 1e-12 ? 1.0 / std::sqrt(var) : 1.0);
    }
    std::mt19937_64 gen(seed);
    auto uni = [&](double lim) { return (float)(((gen() >> 11) * 0x1.0p-53 * 2.0 - 1.0) * lim); };
    const double l1 = std::sqrt(6.0 / (kI + kH)), l2 = std::sqrt(6.0 / (kH + kH)), l3 = std::sqrt(6.0 / (kH + 1));
    for (int i = 0; i < kH * kI; i++) params[kOffW1 + i] = uni(l1);
    for (int i = 0; i < kH * kH; i++) params[kOffW2 + i] = uni(l2);
    for (int i = 0; i < kH; i++) params[kOffW3 + i] = uni(l3);
    params[kOffB3] = (float)(ty / n);
    return AST_OK;
}

// Mean-squared-error loss and its gradient over n host samples (device
// kernels).  grad: AST_MLP_NPARAM floats (shift/scale slots 0).
int ast_mlp_grad(const float* params, const float* samples, int64_t n, float* grad, float* loss)
{
    if (!params || !samples || !grad || n < 1) return AST_ERR_INVALID;
    DevBuf dW, dS, dG, dL;
    TRY(dW.alloc(sizeof(float) * kSumPitch));
    TRY(dS.alloc(sizeof(float) * AST_RECORD_FLOATS * n));
    TRY(dG.alloc(sizeof(float) * kMlpParams));
    TRY(dL.alloc(sizeof(float)));
    TRY(cudaMemcpy(dW.p, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
    TRY(cudaMemcpy(dS.p, samples, sizeof(float) * AST_RECORD_FLOATS * n, cudaMemcpyHostToDevice));
    TRY(cudaMemset(dG.p, 0, sizeof(float) * kMlpParams));
    TRY(cudaMemset(dL.p, 0, sizeof(float)));
    mlp_grad_kernel<<<grad_blocks(n), kT>>>(dW.as<float>(), dS.as<float>(), nullptr, 0, n, 1.0f / (float)n,
                                            dG.as<float>(), dL.as<float>(), Adam{});
    TRY(cudaGetLastError());
    TRY(cudaMemcpy(grad, dG.p, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost));
    float l = 0.0f;
    TRY(cudaMemcpy(&l, dL.p, sizeof(float), cudaMemcpyDeviceToHost));
    if (loss) *loss = l / (float)n;
    return AST_OK;
}

int ast_mlp_forward(const float* params, const float* x, int64_t n, int stride, float* y)
{
    if (!params || !x || !y || n < 1 || stride < kI) return AST_ERR_INVALID;
    DevBuf dW, dX, dY;
    TRY(dW.alloc(sizeof(float) * kMlpParams));
    TRY(dX.alloc(sizeof(float) * stride * n));
    TRY(dY.alloc(sizeof(float) * n));
    TRY(cudaMemcpy(dW.p, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
    TRY(cudaMemcpy(dX.p, x, sizeof(float) * stride * n, cudaMemcpyHostToDevice));
    mlp_forward_kernel<<<(int)((n + 255) / 256), 256>>>(dW.as<float>(), dX.as<float>(), n, stride, dY.as<float>());
    TRY(cudaGetLastError());
    TRY(cudaMemcpy(y, dY.p, sizeof(float) * n, cudaMemcpyDeviceToHost));
    return AST_OK;
}

// Adam on the GPU: `epochs` passes over the n host samples in batches of
// `batch` (a multiple of 256), the sample order drawn once from
// mt19937_64(seed) and the batch order redrawn every epoch.  params holds the
// initial parameters (ast_mlp_init) and receives the trained ones;
// loss_per_epoch (optional, `epochs` floats) the mean batch loss.
int ast_mlp_train(const float* samples, int64_t n, int epochs, int batch, float lr, uint64_t seed, float* params,
                  float* loss_per_epoch)
{
    if (!samples || !params || n < batch || epochs < 1 || batch < kBatchUnit || batch % kBatchUnit)
        return AST_ERR_INVALID;
    const int64_t nb = n / batch;
    std::vector<int> perm(n);
    for (int64_t i = 0; i < n; i++) perm[i] = (int)i;
    std::mt19937_64 gen(seed);
    std::shuffle(perm.begin(), perm.end(), gen);
    // one allocation (seven took some 200 us more): the samples and their
    // order, the parameters, then what starts at zero (gradient, moments,
    // losses, ticket)
    auto pad = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t bS = pad(sizeof(float) * AST_RECORD_FLOATS * n), bI = pad(sizeof(int) * n);
    const size_t bW = pad(sizeof(float) * kSumPitch), bL = pad(sizeof(float) * epochs);
    DevBuf buf;
    TRY(buf.alloc(bS + bI + (3 + kSums) * bW + bL + pad(sizeof(unsigned))));
    char* at = buf.as<char>();
    float* dS = (float*)at;
    int* dI = (int*)(at += bS);
    float* dW = (float*)(at += bI);
    float* dG = (float*)(at += bW);
    float* dM1 = (float*)(at += kSums * bW);
    float* dM2 = (float*)(at += bW);
    float* dL = (float*)(at += bW);
    unsigned* ticket = (unsigned*)(at += bL);
    TRY(cudaMemcpy(dW, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
    TRY(cudaMemcpy(dS, samples, sizeof(float) * AST_RECORD_FLOATS * n, cudaMemcpyHostToDevice));
    TRY(cudaMemcpy(dI, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
    TRY(cudaMemset(dG, 0, (2 + kSums) * bW + bL + sizeof(unsigned)));
    std::vector<int64_t> order(nb);
    const float b1 = 0.9f, b2 = 0.999f;
    long long t = 0;
    for (int e = 0; e < epochs; e++) {
        for (int64_t i = 0; i < nb; i++) order[i] = i;
        std::shuffle(order.begin(), order.end(), gen);
        for (int64_t bi = 0; bi < nb; bi++) {
            t++;
            const float c1 = 1.0f / (1.0f - std::pow(b1, (float)t));
            const float c2 = 1.0f / (1.0f - std::pow(b2, (float)t));
            cudaLaunchConfig_t lc{};
            lc.gridDim = grad_blocks(batch);
            lc.blockDim = kT;
            cudaLaunchAttribute early{};
            early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            early.val.programmaticStreamSerializationAllowed = 1;
            lc.attrs = &early;
            lc.numAttrs = t > 1;   // the first one waits for the copies above
            TRY(cudaLaunchKernelEx(&lc, mlp_grad_kernel, dW, (const float*)dS, (const int*)dI,
                                   (long long)(order[bi] * batch), (long long)batch, 1.0f / (float)batch, dG, dL + e,
                                   Adam{dM1, dM2, ticket, lr, b1, b2, 1e-8f, c1, c2}));
        }
    }
    TRY(cudaMemcpy(params, dW, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost));
    if (loss_per_epoch) {
        TRY(cudaMemcpy(loss_per_epoch, dL, sizeof(float) * epochs, cudaMemcpyDeviceToHost));
        for (int e = 0; e < epochs; e++) loss_per_epoch[e] /= (float)(nb * batch);
    }
    return AST_OK;
}

}  // extern "C"

// ------------------------------------------------------------------ tensor-core inference on given inputs
namespace {

// the step kernel's inference path (tc::forward16, 16 faces per warp tile)
// applied to n given feature rows; one warp per tile
__global__ void mlp_forward_tc_kernel(const float* __restrict__ W_g, const float* __restrict__ x, long long n,
                                      int stride, float* __restrict__ y)
{
    __shared__ float V[kVLen];
    __shared__ unsigned B1[tc::kL1], B2[tc::kL2];
    __shared__ float X[4][16][8];
    __shared__ float Y[4][16];
    for (int i = threadIdx.x; i < kVLen; i += blockDim.x) V[i] = mlp_vec(W_g, i);
    tc::pack_weights(W_g, B1, B2);
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long t0 = ((long long)blockIdx.x * 4 + w) * 16;
    if (lane < 16) {
        const long long k = t0 + lane;
        for (int i = 0; i < kMlpIn; i++) {
            const float v = (k < n) ? mlp_map(i, x[k * stride + i]) : 0.0f;
            X[w][lane][i] = fminf(fmaxf((v - V[kVShift + i]) * V[kVScale + i], -30.0f), 30.0f);
        }
        X[w][lane][6] = 0.0f;
        X[w][lane][7] = 0.0f;
    }
    __syncwarp();
    tc::forward16(V, B1, B2, X[w], Y[w]);
    __syncwarp();
    if (lane < 16 && t0 + lane < n) y[t0 + lane] = Y[w][lane];
}

}  // namespace

namespace {
// the packed network after the parameter block of a device copy
__global__ void __launch_bounds__(256) mlp_pack_kernel(float* W) { pack_network(W); }
}  // namespace

namespace ast {
int launch_mlp_pack(float* W, cudaStream_t st)
{
    mlp_pack_kernel<<<1, 256, 0, st>>>(W);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? AST_OK : cuda_fail(e, "network packing kernel launch");
}
}  // namespace ast

extern "C" int ast_mlp_forward_tc(const float* params, const float* x, int64_t n, int stride, float* y)
{
    if (!params || !x || !y || n < 1 || stride < kI) return AST_ERR_INVALID;
    DevBuf dW, dX, dY;
    TRY(dW.alloc(sizeof(float) * kMlpParams));
    TRY(dX.alloc(sizeof(float) * stride * n));
    TRY(dY.alloc(sizeof(float) * n));
    TRY(cudaMemcpy(dW.p, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
    TRY(cudaMemcpy(dX.p, x, sizeof(float) * stride * n, cudaMemcpyHostToDevice));
    mlp_forward_tc_kernel<<<(int)((n + 63) / 64), 128>>>(dW.as<float>(), dX.as<float>(), n, stride, dY.as<float>());
    TRY(cudaGetLastError());
    TRY(cudaMemcpy(y, dY.p, sizeof(float) * n, cudaMemcpyDeviceToHost));
    return AST_OK;
}
