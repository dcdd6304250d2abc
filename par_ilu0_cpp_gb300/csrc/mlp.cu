// Learned diagonal shift: the feature pre-pass fused with MLP inference (run right
// before the factorisation kernel), and the hand-written training kernels (forward,
// backward, Adam) used to fit the MLP on the GPU.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <stdexcept>
#include <vector>

#include "common.cuh"
#include "device_util.hpp"
#include "gmres_kernels.cuh"
#include "mlp.cuh"
#include "mlp_impl.hpp"

namespace gb300 {

constexpr int kPrepassThreads = 256;

// Sum of |a_ii| over rows (deterministic: per-block partials, last block adds them).
__global__ void __launch_bounds__(kPrepassThreads)
    shift_mean_diag_kernel(int n, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
                           const int* __restrict__ diag, double* partial, unsigned* counter, double* mean_out) {
    __shared__ double sred[kPrepassThreads / kWarp];
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int pd = diag ? diag[i] : -1;
        if (pd >= 0) {
            s += fabs(v[pd]);
        } else {
            for (int p = rp[i]; p < rp[i + 1]; ++p)
                if (ci[p] == i) s += fabs(v[p]);
        }
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < kPrepassThreads / kWarp; ++k) t += sred[k];
        partial[blockIdx.x] = t;
    }
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
        if (last) *counter = 0u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int b = 0; b < static_cast<int>(gridDim.x); ++b) t += __ldcg(partial + b);
        *mean_out = n > 0 ? t / n : 1.0;
    }
}

// Per row: features -> MLP -> shift = sign(a_ii) * y * sum_j!=i |a_ij| (0 when y is
// below min_shift).  Optionally also writes the features and y.
__global__ void __launch_bounds__(kPrepassThreads)
    shift_prepass_kernel(int n, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ v,
                         const int* __restrict__ diag, const int* __restrict__ depth, int nlev,
                         const double* __restrict__ mean_d, const float* __restrict__ params, float min_shift,
                         double* __restrict__ shift_out, float* __restrict__ X_out, float* __restrict__ y_out) {
    __shared__ float P[kMlpParams];
    for (int k = threadIdx.x; k < kMlpParams; k += blockDim.x) P[k] = params ? params[k] : 0.f;
    __syncthreads();
    const double md = *mean_d;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double d, offsum, off2;
        row_stats(i, rp, ci, v, diag, d, offsum, off2);
        float x[kMlpIn];
        make_features(d, offsum, off2, md, depth ? depth[i] : 0, nlev, x);
        if (X_out) {
#pragma unroll
            for (int m = 0; m < kMlpIn; ++m) X_out[static_cast<size_t>(i) * kMlpIn + m] = x[m];
        }
        if (params) {
            MlpAct a;
            const float y = mlp_forward(P, x, a);
            if (y_out) y_out[i] = y;
            if (shift_out) {
                const int pd = diag ? diag[i] : -1;
                const double aii = pd >= 0 ? v[pd] : 1.0;
                const double sgn = aii < 0.0 ? -1.0 : 1.0;
                shift_out[i] = y >= min_shift ? sgn * static_cast<double>(y) * offsum : 0.0;
            }
        }
    }
}

__global__ void __launch_bounds__(kPrepassThreads)
    mlp_forward_kernel(int n, const float* __restrict__ X, const float* __restrict__ params, float* __restrict__ y) {
    __shared__ float P[kMlpParams];
    for (int k = threadIdx.x; k < kMlpParams; k += blockDim.x) P[k] = params[k];
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float x[kMlpIn];
#pragma unroll
        for (int m = 0; m < kMlpIn; ++m) x[m] = X[static_cast<size_t>(i) * kMlpIn + m];
        MlpAct a;
        y[i] = mlp_forward(P, x, a);
    }
}

// One training step over `batch` samples (indices idx, or 0..batch-1): mean squared
// error between y = softplus(z) and the target t, gradient by backpropagation (chain
// rule through softplus, two tanh layers).  mlp_train_kernel leaves per-block sums of the
// gradient and the loss, mlp_reduce_kernel adds them in block order (FP64) and (apply != 0)
// takes one Adam step.
//
// Split: one sample per lane for the forward and backward pass; a warp's 32 samples then go
// through shared memory and each lane sums its own 13 of the 370 gradient entries over them
// in registers (the outer products dh2 x h1 and dh1 x x as small matrix products).  Adding
// every entry of every sample atomically in shared memory, the 32 lanes on one address at a
// time, took 370 serialised updates per sample: a step on 65,536 samples (index upload and
// readback of loss and parameters included) 1,037 us, now 60 us.  The order of all sums is
// fixed.
constexpr int kTrainWarps = kPrepassThreads / kWarp;
constexpr int kTrainPitch = kMlpH + 4;  // staged values of a sample: 16-byte accesses of 8 lanes meet no bank twice
constexpr int kGradEntries = kMlpParams + 1;  // and the loss

struct TrainStage {  // of one warp
    float a[kWarp][kTrainPitch];
    float b[kWarp][kTrainPitch];
    float x[kWarp][kMlpIn];
};
static_assert(sizeof(TrainStage) >= kGradEntries * sizeof(float), "a warp's sums fit its stage");

__device__ __forceinline__ void stage_row(float* row, const float (&v)[kMlpH]) {
#pragma unroll
    for (int k = 0; k < kMlpH; k += 4) *reinterpret_cast<float4*>(row + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
}

__global__ void __launch_bounds__(kPrepassThreads)
    mlp_train_kernel(const float* __restrict__ X, const float* __restrict__ T, const int* __restrict__ idx, int batch,
                     const float* __restrict__ params, float* __restrict__ partial) {
    __shared__ float P[kMlpParams];
    __shared__ __align__(16) TrainStage stage[kTrainWarps];
    for (int k = threadIdx.x; k < kMlpParams; k += blockDim.x) P[k] = params[k];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    TrainStage& st = stage[w];
    const int k2 = lane >> 1;        // the lane's row of W2 (8 entries), W1 (2 entries) ...
    const int j2 = (lane & 1) * 8;   // ... from these columns
    const int m1 = (lane & 1) * 2;
    float g2[8] = {}, g1[2] = {}, gb1 = 0.f, g3 = 0.f;  // g3: W3 (lanes 0-15), b2 (lanes 16-31)
    float gb3 = 0.f, loss = 0.f;     // this lane's samples
    const float inv_b = 1.f / static_cast<float>(batch);
    const int warps = static_cast<int>(gridDim.x) * kTrainWarps;
    for (int s0 = (static_cast<int>(blockIdx.x) * kTrainWarps + w) * kWarp; s0 < batch; s0 += warps * kWarp) {
        const int s = s0 + lane;
        float dz = 0.f;
        float x[kMlpIn] = {};
        MlpAct a;
        float dh2[kMlpH];
        if (s < batch) {
            const int i = idx ? idx[s] : s;
            const float4 xv = *reinterpret_cast<const float4*>(X + static_cast<size_t>(i) * kMlpIn);
            x[0] = xv.x;
            x[1] = xv.y;
            x[2] = xv.z;
            x[3] = xv.w;
            const float y = mlp_forward(P, x, a);
            const float diff = y - T[i];
            loss = fmaf(diff, diff, loss);
            dz = 2.f * diff * inv_b * sigmoid(a.z);
            gb3 += dz;
#pragma unroll
            for (int k = 0; k < kMlpH; ++k) dh2[k] = dz * P[kMlpW3 + k] * (1.f - a.h2[k] * a.h2[k]);
        } else {  // no sample: nothing is added
#pragma unroll
            for (int k = 0; k < kMlpH; ++k) a.h1[k] = a.h2[k] = dh2[k] = 0.f;
        }
        stage_row(st.a[lane], a.h1);
        stage_row(st.b[lane], dh2);
        *reinterpret_cast<float4*>(st.x[lane]) = make_float4(x[0], x[1], x[2], x[3]);
        __syncwarp();
#pragma unroll 4
        for (int q = 0; q < kWarp; ++q) {
            const float d = st.b[q][k2];
            const float4 u = *reinterpret_cast<const float4*>(&st.a[q][j2]);
            const float4 v = *reinterpret_cast<const float4*>(&st.a[q][j2 + 4]);
            g2[0] = fmaf(d, u.x, g2[0]);
            g2[1] = fmaf(d, u.y, g2[1]);
            g2[2] = fmaf(d, u.z, g2[2]);
            g2[3] = fmaf(d, u.w, g2[3]);
            g2[4] = fmaf(d, v.x, g2[4]);
            g2[5] = fmaf(d, v.y, g2[5]);
            g2[6] = fmaf(d, v.z, g2[6]);
            g2[7] = fmaf(d, v.w, g2[7]);
            if (lane >= kMlpH) g3 += st.b[q][lane - kMlpH];
        }
        __syncwarp();
        // the first layer's deltas and the output layer's products
        float dh1[kMlpH];
#pragma unroll
        for (int j = 0; j < kMlpH; ++j) {
            float t = 0.f;
#pragma unroll
            for (int k = 0; k < kMlpH; ++k) t = fmaf(dh2[k], P[kMlpW2 + k * kMlpH + j], t);
            dh1[j] = t * (1.f - a.h1[j] * a.h1[j]);
        }
#pragma unroll
        for (int k = 0; k < kMlpH; ++k) dh2[k] = dz * a.h2[k];
        stage_row(st.a[lane], dh1);
        stage_row(st.b[lane], dh2);
        __syncwarp();
#pragma unroll 4
        for (int q = 0; q < kWarp; ++q) {
            const float d = st.a[q][k2];
            const float2 u = *reinterpret_cast<const float2*>(&st.x[q][m1]);
            g1[0] = fmaf(d, u.x, g1[0]);
            g1[1] = fmaf(d, u.y, g1[1]);
            gb1 += d;
            if (lane < kMlpH) g3 += st.b[q][lane];
        }
        __syncwarp();
    }
    // the warp's sums, then the block's (the stages are free)
    loss *= inv_b;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
        loss += __shfl_xor_sync(0xffffffffu, loss, o);
    }
    float* const G = &st.a[0][0];
#pragma unroll
    for (int j = 0; j < 8; ++j) G[kMlpW2 + k2 * kMlpH + j2 + j] = g2[j];
    G[kMlpW1 + k2 * kMlpIn + m1] = g1[0];
    G[kMlpW1 + k2 * kMlpIn + m1 + 1] = g1[1];
    if ((lane & 1) == 0) G[kMlpB1 + k2] = gb1;
    G[lane < kMlpH ? kMlpW3 + lane : kMlpB2 + lane - kMlpH] = g3;
    if (lane == 0) {
        G[kMlpB3] = gb3;
        G[kMlpParams] = loss;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kGradEntries; k += blockDim.x) {
        float t = 0.f;
#pragma unroll
        for (int v = 0; v < kTrainWarps; ++v) t += (&stage[v].a[0][0])[k];
        partial[static_cast<size_t>(blockIdx.x) * kGradEntries + k] = t;
    }
}

// Sums entry k of the nblk blocks' partials in FP64, a warp per entry (GB300 adds FP64 at
// 16 cycles per warp and SM: one block adding all 370 x 304 partials would take 27 us), and
// takes the Adam step of parameter k.  grad_out: the mean gradient, loss_out: the mean loss.
__global__ void __launch_bounds__(kPrepassThreads)
    mlp_reduce_kernel(const float* __restrict__ partial, int nblk, float* __restrict__ params,
                      float* __restrict__ grad_out, double* __restrict__ loss_out, float* __restrict__ adam_m,
                      float* __restrict__ adam_v, int step, float lr, int apply) {
    const int lane = threadIdx.x & 31;
    const int k = static_cast<int>(blockIdx.x) * kTrainWarps + static_cast<int>(threadIdx.x >> 5);
    if (k >= kGradEntries) return;
    double g = 0.0;
    for (int b = lane; b < nblk; b += kWarp) g += static_cast<double>(partial[static_cast<size_t>(b) * kGradEntries + k]);
    g = warp_sum(g);
    if (lane != 0) return;
    if (k == kMlpParams) {
        *loss_out = g;
        return;
    }
    const float gf = static_cast<float>(g);
    grad_out[k] = gf;
    if (apply) {
        constexpr float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
        const float m = b1 * adam_m[k] + (1.f - b1) * gf;
        const float v = b2 * adam_v[k] + (1.f - b2) * gf * gf;
        adam_m[k] = m;
        adam_v[k] = v;
        const float mh = m / (1.f - powf(b1, static_cast<float>(step)));
        const float vh = v / (1.f - powf(b2, static_cast<float>(step)));
        params[k] = params[k] - lr * mh / (sqrtf(vh) + eps);
    }
}

// ---------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------
void ShiftPrepass::ensure(int sms) {
    if (grid == 0) {
        grid = 4 * sms;
        partial.reserve(static_cast<size_t>(grid));
        counter.reserve(1);
        mean.reserve(1);
        GB_CUDA_CHECK(cudaMemset(counter.get(), 0, sizeof(unsigned)));
    }
}

void ShiftPrepass::run(cudaStream_t s, int sms, int n, const int* rp, const int* ci, const double* v, const int* diag,
                       const int* depth, int nlev, const float* params, float min_shift, double* shift_out,
                       float* X_out, float* y_out) {
    ensure(sms);
    if (n <= 0) return;
    shift_mean_diag_kernel<<<grid, kPrepassThreads, 0, s>>>(n, rp, ci, v, diag, partial.get(), counter.get(), mean.get());
    shift_prepass_kernel<<<grid, kPrepassThreads, 0, s>>>(n, rp, ci, v, diag, depth, nlev, mean.get(), params,
                                                          min_shift, shift_out, X_out, y_out);
    GB_CUDA_CHECK(cudaGetLastError());
}

ShiftTrainer::ShiftTrainer(unsigned seed) {
    dev = current_device();
    GB_CUDA_CHECK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    grid = 2 * dev.sms;
    params.reserve(kMlpParams);
    adam_m.reserve(kMlpParams);
    adam_v.reserve(kMlpParams);
    grad.reserve(kMlpParams);
    partial.reserve(static_cast<size_t>(grid) * kGradEntries);
    loss.reserve(1);
    // Glorot-uniform initialisation; the output bias starts at softplus^{-1}(0.01) so the
    // untrained network predicts a small shift.
    std::mt19937 rng(seed);
    std::vector<float> p(kMlpParams, 0.f);
    auto glorot = [&](int off, int fan_in, int fan_out) {
        std::uniform_real_distribution<float> u(-1.f, 1.f);
        const float a = std::sqrt(6.f / static_cast<float>(fan_in + fan_out));
        for (int k = 0; k < fan_in * fan_out; ++k) p[off + k] = a * u(rng);
    };
    glorot(kMlpW1, kMlpIn, kMlpH);
    glorot(kMlpW2, kMlpH, kMlpH);
    glorot(kMlpW3, kMlpH, 1);
    p[kMlpB3] = std::log(std::expm1(0.01f));
    set_params(p.data());
}

ShiftTrainer::~ShiftTrainer() {
    if (stream) cudaStreamDestroy(stream);
}

void ShiftTrainer::set_params(const float* host) {
    GB_CUDA_CHECK(cudaMemcpyAsync(params.get(), host, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, stream));
    GB_CUDA_CHECK(cudaMemsetAsync(adam_m.get(), 0, sizeof(float) * kMlpParams, stream));
    GB_CUDA_CHECK(cudaMemsetAsync(adam_v.get(), 0, sizeof(float) * kMlpParams, stream));
    GB_CUDA_CHECK(cudaStreamSynchronize(stream));
    step = 0;
}

void ShiftTrainer::get_params(float* host) {
    GB_CUDA_CHECK(cudaMemcpyAsync(host, params.get(), sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, stream));
    GB_CUDA_CHECK(cudaStreamSynchronize(stream));
}

void ShiftTrainer::set_data(const float* X_host, const float* T_host, int n_samples) {
    n = n_samples;
    X.upload(X_host, static_cast<size_t>(n) * kMlpIn, stream);
    T.upload(T_host, static_cast<size_t>(n), stream);
    GB_CUDA_CHECK(cudaStreamSynchronize(stream));
}

double ShiftTrainer::run(const int* idx_host, int batch, float lr, bool apply, float* grad_host) {
    if (n <= 0) throw std::runtime_error("trainer has no data");
    const int* d_idx = nullptr;
    if (idx_host) {
        idx.upload(idx_host, static_cast<size_t>(batch), stream);
        d_idx = idx.get();
    } else {
        batch = n;
    }
    if (apply) ++step;
    // (no more blocks than hold samples: their partials are all added up)
    const int blocks = std::max(1, std::min(grid, ceil_div(batch, kPrepassThreads)));
    mlp_train_kernel<<<blocks, kPrepassThreads, 0, stream>>>(X.get(), T.get(), d_idx, batch, params.get(), partial.get());
    mlp_reduce_kernel<<<ceil_div(kGradEntries, kTrainWarps), kPrepassThreads, 0, stream>>>(
        partial.get(), blocks, params.get(), grad.get(), loss.get(), adam_m.get(), adam_v.get(), std::max(step, 1), lr,
        apply ? 1 : 0);
    GB_CUDA_CHECK(cudaGetLastError());
    double h_loss = 0.0;
    GB_CUDA_CHECK(cudaMemcpyAsync(&h_loss, loss.get(), sizeof(double), cudaMemcpyDeviceToHost, stream));
    if (grad_host)
        GB_CUDA_CHECK(cudaMemcpyAsync(grad_host, grad.get(), sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, stream));
    GB_CUDA_CHECK(cudaStreamSynchronize(stream));
    return h_loss;
}

void ShiftTrainer::predict(float* y_host) {
    if (n <= 0) return;
    y.reserve(static_cast<size_t>(n));
    mlp_forward_kernel<<<grid, kPrepassThreads, 0, stream>>>(n, X.get(), params.get(), y.get());
    GB_CUDA_CHECK(cudaGetLastError());
    GB_CUDA_CHECK(cudaMemcpyAsync(y_host, y.get(), sizeof(float) * static_cast<size_t>(n), cudaMemcpyDeviceToHost, stream));
    GB_CUDA_CHECK(cudaStreamSynchronize(stream));
}

void shift_features_host(int n, const int* rp, const int* ci, const double* v, const int* depth, int nlev, float* X,
                         const float* params_host, float* y_host) {
    DeviceInfo dev = current_device();
    cudaStream_t s = nullptr;
    GB_CUDA_CHECK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    DeviceBuffer<int> d_rp, d_ci, d_depth;
    DeviceBuffer<double> d_v;
    DeviceBuffer<float> d_X, d_p, d_y;
    const long long nnz = rp[n];
    d_rp.upload(rp, static_cast<size_t>(n) + 1, s);
    d_ci.upload(ci, static_cast<size_t>(nnz), s);
    d_v.upload(v, static_cast<size_t>(nnz), s);
    if (depth) d_depth.upload(depth, static_cast<size_t>(n), s);
    d_X.reserve(static_cast<size_t>(std::max(n, 1)) * kMlpIn);
    if (params_host) {
        d_p.upload(params_host, kMlpParams, s);
        d_y.reserve(static_cast<size_t>(std::max(n, 1)));
    }
    ShiftPrepass pre;
    pre.run(s, dev.sms, n, d_rp.get(), d_ci.get(), d_v.get(), nullptr, depth ? d_depth.get() : nullptr, nlev,
            params_host ? d_p.get() : nullptr, 0.f, nullptr, d_X.get(), params_host ? d_y.get() : nullptr);
    if (n > 0) {
        GB_CUDA_CHECK(cudaMemcpyAsync(X, d_X.get(), sizeof(float) * static_cast<size_t>(n) * kMlpIn,
                                      cudaMemcpyDeviceToHost, s));
        if (params_host && y_host)
            GB_CUDA_CHECK(cudaMemcpyAsync(y_host, d_y.get(), sizeof(float) * static_cast<size_t>(n),
                                          cudaMemcpyDeviceToHost, s));
    }
    GB_CUDA_CHECK(cudaStreamSynchronize(s));
    cudaStreamDestroy(s);
}

}  // namespace gb300
