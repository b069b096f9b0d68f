// Threshold MLP (32 -> 64 -> 64 -> 1, ReLU, FP32): forward, backward and Adam
// kernels, exported through the C ABI (include/bm25_b200.h).
//
// The network predicts, from per-query features, the log of the query's K-th
// best score; the pruned Search uses exp(prediction - margin) as its starting
// bound (a wrong guess costs a re-run on the plain path, never a wrong result).
// No counterpart in the reference: this is the learned part of the engine.
//
// Training is deterministic: each CTA of the backward kernel writes its partial
// gradient to its own slice of the scratch array and a second kernel sums the
// slices in a fixed order.
#include "bm25_b200.h"
#include "mlp.cuh"

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>

namespace bm25mlp {

// Programmatic launch: until the kernel before it in the stream has completed / the next kernel may
// start.  Both do nothing in a plain launch.
__device__ __forceinline__ void WaitPrerequisites() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void AllowDependents() { asm volatile("griddepcontrol.launch_dependents;" :::); }

constexpr int kRows = 64;   // samples per forward CTA
constexpr int kBRows = 32;  // samples per backward CTA
constexpr int kBThreads = 256;
constexpr int kBWarps = kBThreads / 32;
constexpr int kTs = kBRows + 4;  // row strides in shared memory: a multiple of 16 bytes, and 8 lanes reading
constexpr int kW2s = kH + 4;     // 16 bytes each from consecutive rows touch all 32 banks once
static_assert(kH == 64 && kIn == 32 && kBRows == 32 && kBWarps * 4 == kBRows && kBWarps * 8 == kH,
              "the backward kernel's thread tiles");

__global__ void __launch_bounds__(kRows) ForwardKernel(const float *params, const float *x, long long batch, float *y)
{
    __shared__ float p[kParams];
    for (int i = threadIdx.x; i < kParams; i += kRows)
        p[i] = params[i];
    __syncthreads();
    const long long r = (long long)blockIdx.x * kRows + threadIdx.x;
    if (r >= batch)
        return;
    float xi[kIn], h1[kH], h2[kH];
    for (int j = 0; j < kIn; ++j)
        xi[j] = x[r * kIn + j];
    y[r] = Forward(p, xi, h1, h2);
}

// acc[u][c] += sum over the row of w[unit lane + 32u][j] * in[j][4 * warp + c], j ascending.
template <int kLen, int kStride>
__device__ __forceinline__ void LayerTile(const float *w, const float *in, int lane, int warp, float (&acc)[2][4])
{
#pragma unroll 4
    for (int j = 0; j < kLen; j += 4) {
        const float4 w0 = *reinterpret_cast<const float4 *>(w + lane * kStride + j);
        const float4 w1 = *reinterpret_cast<const float4 *>(w + (lane + 32) * kStride + j);
        const float wa[2][4] = {{w0.x, w0.y, w0.z, w0.w}, {w1.x, w1.y, w1.z, w1.w}};
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const float4 v = *reinterpret_cast<const float4 *>(in + (j + d) * kTs + 4 * warp);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                acc[u][0] = fmaf(wa[u][d], v.x, acc[u][0]);
                acc[u][1] = fmaf(wa[u][d], v.y, acc[u][1]);
                acc[u][2] = fmaf(wa[u][d], v.z, acc[u][2]);
                acc[u][3] = fmaf(wa[u][d], v.w, acc[u][3]);
            }
        }
    }
}

// out[i][j] = sum over the CTA's samples, in row order, of d[i][s] * in[j][s]; warp w takes rows
// 8w .. 8w + 7, lane l columns l, l + 32, ... (consecutive lanes write consecutive floats).
template <int kCols> __device__ __forceinline__ void WeightGradient(const float *d, const float *in, int lane, int warp, float *out)
{
    constexpr int kN = kCols / 32;
    float g[8][kN] = {};
#pragma unroll 2
    for (int s = 0; s < kBRows; s += 4) {
        float4 v[kN];
#pragma unroll
        for (int n = 0; n < kN; ++n)
            v[n] = *reinterpret_cast<const float4 *>(in + (lane + 32 * n) * kTs + s);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float4 e = *reinterpret_cast<const float4 *>(d + (8 * warp + r) * kTs + s);
#pragma unroll
            for (int n = 0; n < kN; ++n) {
                g[r][n] = fmaf(e.x, v[n].x, g[r][n]);
                g[r][n] = fmaf(e.y, v[n].y, g[r][n]);
                g[r][n] = fmaf(e.z, v[n].z, g[r][n]);
                g[r][n] = fmaf(e.w, v[n].w, g[r][n]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int n = 0; n < kN; ++n)
            out[(8 * warp + r) * kCols + lane + 32 * n] = g[r][n];
}

// Loss per sample: w * (y - t)^2 with w = over_weight when y > t (an over-estimate
// of the K-th score sends the query to the plain path), else 1.  Mean over the batch.
// Each CTA writes its partial gradient (kParams floats) and its loss sum.  Sample r is
// row index[r] of x and t (index nullptr: row r).
//
// Bound: shared-memory loads and the FMA chains' latency, not HBM (a 4096-sample batch is 0.5 MB).
// A thread owns units lane and lane + 32 of samples 4 * warp .. + 3 through all three layers, so a
// 128-bit load of weights feeds 16 FMAs and one of activations 8; activations are kept [unit][sample],
// which the layers read as broadcasts and the gradients along the samples.  Every sum is the chain
// it would be with a thread per sample: index order, one accumulator.  Areas are reused as they die
// (W1 -> h2 -> d2, W2 -> d1) to stay within the 48 KB that need no opt-in.  With a thread per sample,
// its layers in local memory and one warp per CTA, 60 training steps of 4096 samples took 11.3 ms;
// with this kernel and the batched sums below 4.3 ms, most of it the host's (same bits).
// In a training loop this kernel starts while the update before it still writes p: p makes no promise
// of being constant, and is read after the wait, from L2 (x, t and index are constant).
__global__ void __launch_bounds__(kBThreads) BackwardKernel(const float *p, const float *__restrict__ x,
                                                            const float *__restrict__ t,
                                                            const long long *__restrict__ index, long long batch,
                                                            float over_weight, float *partial, float *partial_loss)
{
    __shared__ __align__(16) float sa[kH * kTs];   // W1 [unit][j], then h2, then d2 [unit][sample]
    __shared__ __align__(16) float sw[kH * kW2s];  // W2 [unit][j], then d1 [unit][sample]
    __shared__ __align__(16) float sx[kIn * kTs];  // x [j][sample]
    __shared__ __align__(16) float sh1[kH * kTs];  // h1 [unit][sample]
    __shared__ __align__(16) float sdy[kBRows];
    __shared__ float sw3[kH], sloss[kBRows];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long r0 = (long long)blockIdx.x * kBRows;
    float *out = partial + (long long)blockIdx.x * kParams;
    AllowDependents();
#pragma unroll
    for (int i = 0; i < kBRows / kBWarps; ++i) {  // a warp reads one sample's row
        const int s = warp * (kBRows / kBWarps) + i;
        const long long r = r0 + s;
        sx[lane * kTs + s] = r < batch ? x[(index ? index[r] : r) * kIn + lane] : 0.0f;
    }
    WaitPrerequisites();
#pragma unroll
    for (int i = 0; i < kH * kIn / kBThreads; ++i) {
        const int q = tid + i * kBThreads;
        sa[q / kIn * kTs + q % kIn] = __ldcg(p + kOffW1 + q);
    }
#pragma unroll
    for (int i = 0; i < kH * kH / kBThreads; ++i) {
        const int q = tid + i * kBThreads;
        sw[q / kH * kW2s + q % kH] = __ldcg(p + kOffW2 + q);
    }
    if (tid < kH)
        sw3[tid] = __ldcg(p + kOffW3 + tid);
    float h1[2][4], h2[2][4];
    bool live[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
        live[c] = r0 + 4 * warp + c < batch;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            h1[u][c] = __ldcg(p + kOffB1 + lane + 32 * u);
            h2[u][c] = __ldcg(p + kOffB2 + lane + 32 * u);
        }
    __syncthreads();
    LayerTile<kIn, kTs>(sa, sx, lane, warp, h1);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            h1[u][c] = live[c] ? fmaxf(h1[u][c], 0.0f) : 0.0f;
        *reinterpret_cast<float4 *>(sh1 + (lane + 32 * u) * kTs + 4 * warp) =
            make_float4(h1[u][0], h1[u][1], h1[u][2], h1[u][3]);
    }
    __syncthreads();
    LayerTile<kH, kW2s>(sw, sh1, lane, warp, h2);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            h2[u][c] = live[c] ? fmaxf(h2[u][c], 0.0f) : 0.0f;
        *reinterpret_cast<float4 *>(sa + (lane + 32 * u) * kTs + 4 * warp) =
            make_float4(h2[u][0], h2[u][1], h2[u][2], h2[u][3]);
    }
    __syncthreads();
    if (warp == 0) {  // the output of sample `lane`
        const long long r = r0 + lane;
        float dy = 0.0f, loss = 0.0f;
        if (r < batch) {
            float y = __ldcg(p + kOffB3);
#pragma unroll 16
            for (int j = 0; j < kH; ++j)
                y = fmaf(sw3[j], sa[j * kTs + lane], y);
            const float e = y - t[index ? index[r] : r];
            const float w = e > 0.0f ? over_weight : 1.0f;
            loss = w * e * e;
            dy = 2.0f * w * e / (float)batch;
        }
        sdy[lane] = dy;
        sloss[lane] = loss;
    }
    __syncthreads();
    if (tid < kH) {  // w3's gradient, while h2 is there
        float g = 0.0f;
#pragma unroll 8
        for (int s = 0; s < kBRows; ++s)
            g = fmaf(sdy[s], sa[tid * kTs + s], g);
        out[kOffW3 + tid] = g;
    } else if (tid == kH) {
        float g = 0.0f, l = 0.0f;
        for (int s = 0; s < kBRows; ++s) {
            g += sdy[s];
            l += sloss[s];
        }
        out[kOffB3] = g;
        partial_loss[blockIdx.x] = l;
    }
    __syncthreads();
    // dh2 = dy * w3 (ReLU gate), dh1 = W2^T dh2 (ReLU gate)
    const float4 dy4 = *reinterpret_cast<const float4 *>(sdy + 4 * warp);
    const float dy[4] = {dy4.x, dy4.y, dy4.z, dy4.w};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const float w3 = sw3[lane + 32 * u];
        float d[4];
#pragma unroll
        for (int c = 0; c < 4; ++c)
            d[c] = h2[u][c] > 0.0f ? dy[c] * w3 : 0.0f;
        *reinterpret_cast<float4 *>(sa + (lane + 32 * u) * kTs + 4 * warp) = make_float4(d[0], d[1], d[2], d[3]);
    }
    __syncthreads();
    float d1[2][4] = {};
#pragma unroll 8
    for (int i = 0; i < kH; ++i) {
        const float4 v = *reinterpret_cast<const float4 *>(sa + i * kTs + 4 * warp);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float w = sw[i * kW2s + lane + 32 * u];
            d1[u][0] = fmaf(w, v.x, d1[u][0]);
            d1[u][1] = fmaf(w, v.y, d1[u][1]);
            d1[u][2] = fmaf(w, v.z, d1[u][2]);
            d1[u][3] = fmaf(w, v.w, d1[u][3]);
        }
    }
    WeightGradient<kH>(sa, sh1, lane, warp, out + kOffW2);
    __syncthreads();  // W2 has been read by every warp
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            d1[u][c] = h1[u][c] > 0.0f ? d1[u][c] : 0.0f;
        *reinterpret_cast<float4 *>(sw + (lane + 32 * u) * kTs + 4 * warp) =
            make_float4(d1[u][0], d1[u][1], d1[u][2], d1[u][3]);
    }
    __syncthreads();
    WeightGradient<kIn>(sw, sx, lane, warp, out + kOffW1);
    if (tid < 2 * kH) {  // the biases' gradients
        const float *d = (tid < kH ? sw : sa) + tid % kH * kTs;
        float g = 0.0f;
#pragma unroll 8
        for (int s = 0; s < kBRows; ++s)
            g += d[s];
        out[(tid < kH ? kOffB1 : kOffB2) + tid % kH] = g;
    }
}

constexpr int kReduceThreads = 64;  // 100 CTAs: each thread's chain of loads is what takes the time

// Sum of partial[c][q] in CTA order (32 loads in flight, one accumulator).
__device__ __forceinline__ float SumPartials(const float *partial, int q, int ctas)
{
    float g = 0.0f;
    int c = 0;
    for (; c + 32 <= ctas; c += 32) {
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i)
            v[i] = partial[(long long)(c + i) * kParams + q];
#pragma unroll
        for (int i = 0; i < 32; ++i)
            g += v[i];
    }
    for (; c < ctas; ++c)
        g += partial[(long long)c * kParams + q];
    return g;
}

// The batch's mean loss: one warp loads, the sum is in CTA order.
__device__ __forceinline__ void BatchLoss(const float *partial_loss, int ctas, long long batch, int lane,
                                          float *loss)
{
    float l = 0.0f;
    for (int c = 0; c < ctas; c += 32) {
        const float v = c + lane < ctas ? partial_loss[c + lane] : 0.0f;
        for (int i = 0; i < min(32, ctas - c); ++i)
            l += __shfl_sync(0xffffffffu, v, i);
    }
    if (lane == 0)
        *loss = l / (float)batch;
}

// Adam (beta1 0.9, beta2 0.999, eps 1e-8) with bias correction for step `step` (1-based).
__device__ __forceinline__ void AdamUpdate(float *params, float *m, float *v, float g, float lr, int step, int q)
{
    const float mq = 0.9f * m[q] + 0.1f * g, vq = 0.999f * v[q] + 0.001f * g * g;
    m[q] = mq;
    v[q] = vq;
    const float mh = mq / (1.0f - powf(0.9f, (float)step)), vh = vq / (1.0f - powf(0.999f, (float)step));
    params[q] -= lr * mh / (sqrtf(vh) + 1e-8f);
}

// grad[q] = sum over CTAs of partial[c][q] in CTA order; loss = sum of partial losses / batch.
// The loss is the last CTA's, which has no parameters.
__global__ void __launch_bounds__(kReduceThreads) ReduceKernel(const float *partial, const float *partial_loss, int ctas,
                                                               long long batch, float *grad, float *loss)
{
    if (blockIdx.x == gridDim.x - 1) {
        if (threadIdx.x < 32 && loss)
            BatchLoss(partial_loss, ctas, batch, threadIdx.x, loss);
        return;
    }
    const int q = blockIdx.x * kReduceThreads + threadIdx.x;
    if (q < kParams)
        grad[q] = SumPartials(partial, q, ctas);
}

__global__ void AdamKernel(float *params, float *m, float *v, const float *grad, float lr, int step)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < kParams)
        AdamUpdate(params, m, v, grad[q], lr, step, q);
}

// One training step's end: ReduceKernel's sums and loss and AdamKernel's update in one pass (the
// gradient never reaches memory).  Every thread waits, so that the step's completion follows its
// backward kernel's, whose partial sums the next step overwrites.
__global__ void __launch_bounds__(kReduceThreads) ReduceAdamKernel(const float *partial, const float *partial_loss, int ctas,
                                                                   long long batch, float *params, float *m, float *v,
                                                                   float lr, int step, float *loss)
{
    AllowDependents();
    WaitPrerequisites();
    if (blockIdx.x == gridDim.x - 1) {
        if (threadIdx.x < 32 && loss)
            BatchLoss(partial_loss, ctas, batch, threadIdx.x, loss);
        return;
    }
    const int q = blockIdx.x * kReduceThreads + threadIdx.x;
    if (q < kParams)
        AdamUpdate(params, m, v, SumPartials(partial, q, ctas), lr, step, q);
}

} // namespace bm25mlp

namespace {
constexpr int kReduceCtas = (bm25mlp::kParams + bm25mlp::kReduceThreads - 1) / bm25mlp::kReduceThreads;
thread_local std::string g_mlp_error;
int Fail(int status, const std::string &m)
{
    g_mlp_error = m;
    return status;
}
int CudaStatus(cudaError_t e, const char *what)
{
    if (e == cudaSuccess)
        return BM25_OK;
    return Fail(BM25_ERR_INNER_ERROR, std::string(what) + ": " + cudaGetErrorString(e));
}
} // namespace

extern "C" int64_t bm25_mlp_param_count(void) { return bm25mlp::kParams; }

extern "C" int64_t bm25_mlp_scratch_floats(int64_t batch)
{
    const int64_t ctas = (batch + bm25mlp::kBRows - 1) / bm25mlp::kBRows;
    return ctas * (bm25mlp::kParams + 1);
}

extern "C" int bm25_mlp_forward(const float *params, const float *features, int64_t batch, float *out, void *stream)
{
    if (!params || !features || !out || batch < 1)
        return Fail(BM25_ERR_INVALID_PARAM, "Null buffer or empty batch");
    const int64_t ctas = (batch + bm25mlp::kRows - 1) / bm25mlp::kRows;
    bm25mlp::ForwardKernel<<<(unsigned)ctas, bm25mlp::kRows, 0, static_cast<cudaStream_t>(stream)>>>(
        params, features, batch, out);
    return CudaStatus(cudaGetLastError(), "MLP forward launch");
}

extern "C" int bm25_mlp_gradient(const float *params, const float *features, const float *targets, int64_t batch,
                                 float over_weight, float *scratch, float *grad, float *loss, void *stream)
{
    if (!params || !features || !targets || !scratch || !grad || batch < 1)
        return Fail(BM25_ERR_INVALID_PARAM, "Null buffer or empty batch");
    const int64_t ctas = (batch + bm25mlp::kBRows - 1) / bm25mlp::kBRows;
    if (ctas > (1 << 20))
        return Fail(BM25_ERR_INVALID_PARAM, "Batch too large");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float *partial = scratch, *partial_loss = scratch + ctas * bm25mlp::kParams;
    bm25mlp::BackwardKernel<<<(unsigned)ctas, bm25mlp::kBThreads, 0, s>>>(params, features, targets, nullptr, batch,
                                                                         over_weight, partial, partial_loss);
    int st = CudaStatus(cudaGetLastError(), "MLP backward launch");
    if (st != BM25_OK)
        return st;
    bm25mlp::ReduceKernel<<<kReduceCtas + 1, bm25mlp::kReduceThreads, 0, s>>>(partial, partial_loss, (int)ctas, batch,
                                                                              grad, loss);
    return CudaStatus(cudaGetLastError(), "MLP reduce launch");
}

// Two launches per step, each set up while the one before it runs.  With a copy, two gathers and
// three launches per step the host took most of the 4.3 ms of 60 steps of 4096 samples; 1.9 ms now.
extern "C" int bm25_mlp_train_steps(float *params, float *m, float *v, const float *features, const float *targets,
                                    const int64_t *rows, int64_t batch, int32_t steps, int32_t first_step,
                                    float over_weight, float lr, float *scratch, float *loss, void *stream)
{
    if (!params || !m || !v || !features || !targets || !rows || !scratch || batch < 1 || steps < 0 || first_step < 1)
        return Fail(BM25_ERR_INVALID_PARAM, "Null buffer, empty batch or step < 1");
    const int64_t ctas = (batch + bm25mlp::kBRows - 1) / bm25mlp::kBRows;
    if (ctas > (1 << 20))
        return Fail(BM25_ERR_INVALID_PARAM, "Batch too large");
    float *partial = scratch, *partial_loss = scratch + ctas * bm25mlp::kParams;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = static_cast<cudaStream_t>(stream);
    cfg.attrs = attr;
    for (int32_t i = 0; i < steps; ++i) {
        cfg.gridDim = dim3((unsigned)ctas);
        cfg.blockDim = dim3(bm25mlp::kBThreads);
        cfg.numAttrs = i > 0 ? 1 : 0;  // the first step waits for the row numbers' copy
        int st = CudaStatus(cudaLaunchKernelEx(&cfg, bm25mlp::BackwardKernel, (const float *)params, features, targets,
                                               (const long long *)rows + i * batch, (long long)batch, over_weight,
                                               partial, partial_loss),
                            "MLP backward launch");
        if (st != BM25_OK)
            return st;
        cfg.gridDim = dim3(kReduceCtas + 1);
        cfg.blockDim = dim3(bm25mlp::kReduceThreads);
        cfg.numAttrs = 1;
        st = CudaStatus(cudaLaunchKernelEx(&cfg, bm25mlp::ReduceAdamKernel, (const float *)partial,
                                           (const float *)partial_loss, (int)ctas, (long long)batch, params, m, v, lr,
                                           (int)(first_step + i), loss ? loss + i : nullptr),
                        "MLP update launch");
        if (st != BM25_OK)
            return st;
    }
    return BM25_OK;
}

extern "C" int bm25_mlp_adam(float *params, float *m, float *v, const float *grad, float lr, int32_t step,
                             void *stream)
{
    if (!params || !m || !v || !grad || step < 1)
        return Fail(BM25_ERR_INVALID_PARAM, "Null buffer or step < 1");
    bm25mlp::AdamKernel<<<(bm25mlp::kParams + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(params, m, v,
                                                                                                   grad, lr, step);
    return CudaStatus(cudaGetLastError(), "MLP Adam launch");
}

extern "C" int bm25_mlp_last_error(char *buffer, size_t length)
{
    if (buffer && length) {
        const size_t n = g_mlp_error.size() < length - 1 ? g_mlp_error.size() : length - 1;
        g_mlp_error.copy(buffer, n);
        buffer[n] = '\0';
    }
    return BM25_OK;
}
