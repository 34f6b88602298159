// The learned cost model's network: a 3-layer FP32 perceptron
//   h1 = relu(x W1 + b1), h2 = relu(h1 W2 + b2), y = h2 w3 + b3
// with hand-written forward, backward (mean squared error) and Adam kernels.
// It replaces the reference tuner's XGBoost regressor
// (tuning/tuning/role/modeling.py:16-162): it maps (schedule, configuration,
// graph statistics) features to log run time and ranks candidate
// configurations; it is trained on the GPU from timings the engine itself
// records.
//
// Sizes are tiny (input <= 64 features, hidden = 64), so the kernels are
// plain CUDA-core FP32 and a training step is bound by latency, not by its
// 10 MFLOP: it is two launches, one warp per sample row for the forward pass
// and the row's deltas (weights staged in shared memory, W2's rows padded so
// that both passes read it without bank conflicts), then one thread per
// parameter for its gradient over the rows in order (deterministic, no
// atomics; the rows are staged in shared memory first, since 256 dependent
// global reads were most of a step) and its Adam update.  Mini-batches name
// their rows by index, so an epoch copies its shuffled order to the device
// and nothing else.  Every sum is formed in the order of the plain loops, so
// results do not depend on the launch shape.  Training 4,001 rows of 38
// features for 10 epochs at batch 256 on a B200: 9.4 ms with four launches a
// step, host-gathered batches and the global reads, now 2.3 ms (14 us a step:
// about 6 per launch); predicting 64 rows 44 -> 30 us.  Tensor cores would not pay at this size.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <algorithm>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../../include/gat.h"
#include "devmem.hpp"

namespace {

constexpr int kHidden = 64;
constexpr int kMaxIn = 64;
constexpr int kRowsPerCta = 8;  // one warp per row, 256 threads

thread_local std::string g_mlp_err;

struct Shape {
    int in;
    // parameter offsets in the flat vector
    int w1, b1, w2, b2, w3, b3, total;
    explicit Shape(int in_) : in(in_) {
        w1 = 0;
        b1 = w1 + in * kHidden;
        w2 = b1 + kHidden;
        b2 = w2 + kHidden * kHidden;
        w3 = b2 + kHidden;
        b3 = w3 + kHidden;
        total = b3 + 1;
    }
};

// A training step's two launches follow one another within a microsecond:
// each may start while the other ends and waits here for its results.  The
// next launch is let in only after the wait, so that at most two overlap, and
// what one launch writes and the next reads (parameters, activations, deltas)
// is read past L1 (__ldcg): the read-only path may hold lines from before the
// writer ran.
__device__ __forceinline__ void after_previous_launch() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

constexpr int kW2Pitch = kHidden + 1;  // padded rows: lanes on k or on u, no conflicts

// Forward pass for rows [0, n): y[r].  Row r is X's row order[r] (r itself
// without an order).  BACK also stores the hidden activations and the loss
// gradients at the output and at both hidden layers' pre-activations, for
// L = mean_r (y_r - t_r)^2:
//   dy_r = 2 (y_r - t_r) / n,  d2 = dy w3 . [h2 > 0],  d1 = (d2 W2^T) . [h1 > 0]
template <bool BACK>
__global__ void __launch_bounds__(256)
    mlp_rows_kernel(const float *params, int in, const float *__restrict__ X,
                    const int *__restrict__ order, const float *__restrict__ T, int n,
                    float *__restrict__ y, float *__restrict__ h1, float *__restrict__ h2,
                    float *__restrict__ dyo, float *__restrict__ d2o, float *__restrict__ d1o) {
    extern __shared__ float sm[];
    const int nw1 = in * kHidden;
    float *W1 = sm, *B1 = W1 + nw1, *W2 = B1 + kHidden, *B2 = W2 + kHidden * kW2Pitch,
          *W3 = B2 + kHidden;
    float *act = W3 + kHidden + 1;  // per warp: x, a1, a2, d2
    after_previous_launch();
    // every section before b3 is a whole number of 16-byte groups
    const float4 *p4 = reinterpret_cast<const float4 *>(params);
    const int q1 = (nw1 + kHidden) / 4, q2 = kHidden * kHidden / 4;
#pragma unroll 4
    for (int i = threadIdx.x; i < q2; i += 256) {
        const float4 v = __ldcg(p4 + q1 + i);
        float *to = W2 + (4 * i / kHidden) * kW2Pitch + 4 * i % kHidden;
        to[0] = v.x, to[1] = v.y, to[2] = v.z, to[3] = v.w;
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < q1; i += 256) reinterpret_cast<float4 *>(sm)[i] = __ldcg(p4 + i);
    for (int i = threadIdx.x; i < 2 * kHidden + 1; i += 256)
        B2[i] = __ldcg(params + nw1 + kHidden + kHidden * kHidden + i);
    __syncthreads();
    const float b3 = W3[kHidden];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *x = act + warp * 4 * kHidden, *a1 = x + kHidden, *a2 = a1 + kHidden, *d2 = a2 + kHidden;
    const float scale = 2.f / (float)n;
    for (int r = blockIdx.x * kRowsPerCta + warp; r < n; r += gridDim.x * kRowsPerCta) {
        const int64_t row = order ? order[r] : r;
        for (int f = lane; f < in; f += 32) x[f] = X[row * in + f];
        __syncwarp();
        // a lane forms units lane and lane + 32, each sum in order
        float s0 = B1[lane], s1 = B1[lane + 32];
#pragma unroll 8
        for (int f = 0; f < in; f++) {
            s0 += x[f] * W1[f * kHidden + lane];
            s1 += x[f] * W1[f * kHidden + lane + 32];
        }
        a1[lane] = s0 > 0.f ? s0 : 0.f;
        a1[lane + 32] = s1 > 0.f ? s1 : 0.f;
        __syncwarp();
        s0 = B2[lane], s1 = B2[lane + 32];
#pragma unroll 16
        for (int k = 0; k < kHidden; k++) {
            s0 += a1[k] * W2[k * kW2Pitch + lane];
            s1 += a1[k] * W2[k * kW2Pitch + lane + 32];
        }
        a2[lane] = s0 > 0.f ? s0 : 0.f;
        a2[lane + 32] = s1 > 0.f ? s1 : 0.f;
        __syncwarp();
        float part = a2[lane] * W3[lane] + a2[lane + 32] * W3[lane + 32];
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        const float yr = part + b3;
        if (lane == 0) y[r] = yr;
        if constexpr (BACK) {
            const float dy = scale * (yr - T[row]);
            for (int u = lane; u < kHidden; u += 32) {
                const int64_t at = (int64_t)r * kHidden + u;
                const float v = a2[u] > 0.f ? dy * W3[u] : 0.f;
                d2[u] = v;
                d2o[at] = v;
                h1[at] = a1[u];
                h2[at] = a2[u];
            }
            __syncwarp();
            s0 = s1 = 0.f;
#pragma unroll 16
            for (int u = 0; u < kHidden; u++) {
                s0 += d2[u] * W2[lane * kW2Pitch + u];
                s1 += d2[u] * W2[(lane + 32) * kW2Pitch + u];
            }
            d1o[(int64_t)r * kHidden + lane] = a1[lane] > 0.f ? s0 : 0.f;
            d1o[(int64_t)r * kHidden + lane + 32] = a1[lane + 32] > 0.f ? s1 : 0.f;
            if (lane == 0) dyo[r] = dy;
        }
        __syncwarp();
    }
}

// Adam (Kingma & Ba 2015) with bias correction; step is 1-based.
struct AdamState {
    float *p, *m, *v;
    float lr, b1, b2, eps;
    int step;
};

__device__ __forceinline__ void adam_update(const AdamState &a, int i, float gi) {
    const float mi = a.b1 * a.m[i] + (1.f - a.b1) * gi;
    const float vi = a.b2 * a.v[i] + (1.f - a.b2) * gi * gi;
    a.m[i] = mi;
    a.v[i] = vi;
    const float mh = mi / (1.f - powf(a.b1, (float)a.step));
    const float vh = vi / (1.f - powf(a.b2, (float)a.step));
    a.p[i] -= a.lr * mh / (sqrtf(vh) + a.eps);
}

// Gradient of every parameter over rows [0, n), each summed by one thread in
// row order: dW1 = X^T d1, db1 = sum d1, dW2 = h1^T d2, db2 = sum d2,
// dw3 = h2^T dy, db3 = sum dy.  A CTA takes kGradRows rows of W1 or of W2, or
// one of the three vectors; kChunk sample rows at a time are staged in shared
// memory.  ADAM applies the update, otherwise the gradient is written.
constexpr int kGradRows = 4;
constexpr int kChunk = 256;
constexpr int kGradThreads = kGradRows * kHidden;

template <bool ADAM>
__global__ void __launch_bounds__(kGradThreads)
    mlp_param_kernel(int in, const float *__restrict__ X, const int *__restrict__ order,
                     const float *h1, const float *h2, const float *dy, const float *d2,
                     const float *d1, int n, float *__restrict__ grad, const AdamState adam) {
    extern __shared__ float sm[];
    float *B = sm;                     // d1, d2 or h2 of the chunk's rows
    float *A = B + kChunk * kHidden;   // their factors
    after_previous_launch();
    const int u = threadIdx.x % kHidden, g = threadIdx.x / kHidden;
    const int ctas1 = (in + kGradRows - 1) / kGradRows, ctas2 = kHidden / kGradRows;
    const int nw1 = in * kHidden, b1 = nw1, w2 = b1 + kHidden, b2 = w2 + kHidden * kHidden,
              w3 = b2 + kHidden, b3 = w3 + kHidden;
    int cta = blockIdx.x;
    int kind, row = 0;  // 0 W1, 1 W2, 2 b1, 3 b2, 4 w3 and b3
    if (cta < ctas1) {
        kind = 0;
        row = cta * kGradRows;
    } else if (cta < ctas1 + ctas2) {
        kind = 1;
        row = (cta - ctas1) * kGradRows;
    } else {
        kind = 2 + (cta - ctas1 - ctas2);
    }
    const float *src = kind == 0 || kind == 2 ? d1 : kind == 4 ? h2 : d2;
    int out = -1;  // this thread's parameter
    if (kind == 0) {
        if (row + g < in) out = (row + g) * kHidden + u;
    } else if (kind == 1) {
        out = w2 + (row + g) * kHidden + u;
    } else if (g == 0) {
        out = (kind == 2 ? b1 : kind == 3 ? b2 : w3) + u;
    } else if (kind == 4 && threadIdx.x == kHidden) {
        out = b3;
    }
    float s = 0.f;
    for (int r0 = 0; r0 < n; r0 += kChunk) {
        const int rows = min(kChunk, n - r0);
        __syncthreads();
        const float4 *from = reinterpret_cast<const float4 *>(src + (int64_t)r0 * kHidden);
        float4 *to = reinterpret_cast<float4 *>(B);
#pragma unroll 16
        for (int i = threadIdx.x; i < rows * kHidden / 4; i += kGradThreads) to[i] = __ldcg(from + i);
        for (int i = threadIdx.x; i < rows * kGradRows; i += kGradThreads) {
            const int r = r0 + i / kGradRows, c = row + i % kGradRows;
            float v = 0.f;
            if (kind == 0) {
                if (c < in) v = X[(int64_t)(order ? order[r] : r) * in + c];
            } else if (kind == 1) {
                v = __ldcg(h1 + (int64_t)r * kHidden + c);
            } else if (kind == 4 && i % kGradRows == 0) {
                v = __ldcg(dy + r);
            }
            A[i] = v;
        }
        __syncthreads();
        if (kind < 2) {
#pragma unroll 16
            for (int r = 0; r < rows; r++) s += A[r * kGradRows + g] * B[r * kHidden + u];
        } else if (kind < 4) {
            if (g == 0)
#pragma unroll 8
                for (int r = 0; r < rows; r++) s += B[r * kHidden + u];
        } else if (g == 0) {
#pragma unroll 8
            for (int r = 0; r < rows; r++) s += B[r * kHidden + u] * A[r * kGradRows];
        } else if (out == b3) {
            for (int r = 0; r < rows; r++) s += A[r * kGradRows];
        }
    }
    if (out < 0) return;
    if constexpr (ADAM)
        adam_update(adam, out, s);
    else
        grad[out] = s;
}

__global__ void sq_err_kernel(const float *y, const float *t, int n, float *out) {
    float s = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float d = y[i] - t[i];
        s += d * d;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

int grid_for(int n) {
    int g = (n + kRowsPerCta - 1) / kRowsPerCta;
    return g < 1 ? 1 : (g > 1184 ? 1184 : g);
}

size_t rows_smem(int in) {
    return sizeof(float) * (in * kHidden + kHidden + kHidden * kW2Pitch + 2 * kHidden + 1 +
                            kRowsPerCta * 4 * kHidden);
}

constexpr size_t kParamSmem = sizeof(float) * kChunk * (kHidden + kGradRows);
int param_ctas(int in) { return (in + kGradRows - 1) / kGradRows + kHidden / kGradRows + 3; }

// Device room for n rows, one allocation from the library's pool: inputs and
// what a training step keeps between its two launches.
struct Work {
    char *p = nullptr;
    float *X = nullptr, *T = nullptr, *y = nullptr, *loss = nullptr, *grad = nullptr;
    float *h1 = nullptr, *h2 = nullptr, *dy = nullptr, *d2 = nullptr, *d1 = nullptr;
    int *order = nullptr;
    ~Work() { gat::dev_free(p, nullptr); }
    // hidden: rows of hidden values (a batch), 0 for prediction alone
    cudaError_t alloc(int n, int in, int hidden, int params) {
        size_t at = 0;
        auto take = [&](size_t floats) {
            const size_t here = at;
            at += (floats * 4 + 255) / 256 * 256;
            return here;
        };
        const size_t h = size_t(hidden) * kHidden;
        const size_t oX = take(size_t(n) * in), oy = take(n), oT = take(hidden ? n : 0),
                     ol = take(1), og = take(params), o1 = take(h), o2 = take(h),
                     od = take(hidden), o3 = take(h), o4 = take(h), oo = take(hidden ? n : 0);
        const cudaError_t e = gat::dev_alloc((void **)&p, at, nullptr);
        if (e != cudaSuccess) return e;
        auto f = [&](size_t o) { return reinterpret_cast<float *>(p + o); };
        X = f(oX), y = f(oy), T = f(oT), loss = f(ol), grad = f(og);
        h1 = f(o1), h2 = f(o2), dy = f(od), d2 = f(o3), d1 = f(o4);
        order = reinterpret_cast<int *>(p + oo);
        return e;
    }
};

}  // namespace

struct gat_mlp {
    gat::PoolUser pool;
    Shape shape{1};
    float *params = nullptr, *m = nullptr, *v = nullptr;
    int step = 0;
    ~gat_mlp() {
        cudaFree(params);
        cudaFree(m);
        cudaFree(v);
    }
};

namespace {
int mlp_fail(int code, const std::string &msg) {
    g_mlp_err = msg;
    return code;
}
int cerr(cudaError_t e, const char *what) {
    return mlp_fail(GAT_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

template <class F>
cudaError_t allow_smem(F *kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

cudaError_t set_attrs(int in) {
    cudaError_t e;
    if ((e = allow_smem(mlp_rows_kernel<false>, rows_smem(in))) != cudaSuccess ||
        (e = allow_smem(mlp_rows_kernel<true>, rows_smem(in))) != cudaSuccess ||
        (e = allow_smem(mlp_param_kernel<false>, kParamSmem)) != cudaSuccess)
        return e;
    return allow_smem(mlp_param_kernel<true>, kParamSmem);
}

// Launches on the default stream; the kernel may be scheduled before the one
// ahead of it has ended (after_previous_launch).
template <class... Params, class... Args>
void launch(void (*kernel)(Params...), int grid, int block, size_t smem, Args... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, Params(args)...);
}

void forward(const gat_mlp *net, const Work &w, int n) {
    const int in = net->shape.in;
    launch(mlp_rows_kernel<false>, grid_for(n), 256, rows_smem(in), net->params, in, w.X, nullptr,
           nullptr, n, w.y, nullptr, nullptr, nullptr, nullptr, nullptr);
}

}  // namespace

extern "C" {

const char *gat_mlp_last_error(void) { return g_mlp_err.c_str(); }

int gat_mlp_create(int in_features, uint64_t seed, gat_mlp **out) {
    if (!out || in_features < 1 || in_features > kMaxIn)
        return mlp_fail(GAT_ERR_ARGUMENT, "in_features must be in [1, 64]");
    auto *net = new gat_mlp;
    net->shape = Shape(in_features);
    const int P = net->shape.total;
    cudaError_t e;
    if ((e = cudaMalloc(&net->params, sizeof(float) * P)) != cudaSuccess ||
        (e = cudaMalloc(&net->m, sizeof(float) * P)) != cudaSuccess ||
        (e = cudaMalloc(&net->v, sizeof(float) * P)) != cudaSuccess) {
        delete net;
        return cerr(e, "mlp allocation");
    }
    // He-uniform initial weights, zero biases (host generated, seeded).
    std::vector<float> h(P, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int fan_in, int count) {
        const float lim = std::sqrt(6.f / (float)fan_in);
        std::uniform_real_distribution<float> d(-lim, lim);
        for (int i = 0; i < count; i++) h[off + i] = d(rng);
    };
    const Shape &s = net->shape;
    fill(s.w1, s.in, s.in * kHidden);
    fill(s.w2, kHidden, kHidden * kHidden);
    fill(s.w3, kHidden, kHidden);
    if ((e = cudaMemcpy(net->params, h.data(), sizeof(float) * P, cudaMemcpyHostToDevice)) !=
            cudaSuccess ||
        (e = cudaMemset(net->m, 0, sizeof(float) * P)) != cudaSuccess ||
        (e = cudaMemset(net->v, 0, sizeof(float) * P)) != cudaSuccess ||
        (e = set_attrs(s.in)) != cudaSuccess) {
        delete net;
        return cerr(e, "mlp init");
    }
    *out = net;
    return GAT_OK;
}

void gat_mlp_free(gat_mlp *net) { delete net; }

int gat_mlp_num_params(const gat_mlp *net) { return net ? net->shape.total : 0; }

int gat_mlp_get_params(const gat_mlp *net, float *out, int n) {
    if (!net || !out || n < net->shape.total) return mlp_fail(GAT_ERR_ARGUMENT, "bad buffer");
    cudaError_t e = cudaMemcpy(out, net->params, sizeof(float) * net->shape.total,
                               cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? GAT_OK : cerr(e, "get params");
}

int gat_mlp_set_params(gat_mlp *net, const float *in, int n) {
    if (!net || !in || n < net->shape.total) return mlp_fail(GAT_ERR_ARGUMENT, "bad buffer");
    cudaError_t e = cudaMemcpy(net->params, in, sizeof(float) * net->shape.total,
                               cudaMemcpyHostToDevice);
    net->step = 0;
    if (e == cudaSuccess) e = cudaMemset(net->m, 0, sizeof(float) * net->shape.total);
    if (e == cudaSuccess) e = cudaMemset(net->v, 0, sizeof(float) * net->shape.total);
    return e == cudaSuccess ? GAT_OK : cerr(e, "set params");
}

int gat_mlp_predict(const gat_mlp *net, const float *X, int n, float *y) {
    if (!net || !X || !y || n < 0) return mlp_fail(GAT_ERR_ARGUMENT, "bad arguments");
    if (n == 0) return GAT_OK;
    const int in = net->shape.in;
    Work w;
    cudaError_t e;
    if ((e = w.alloc(n, in, 0, 0)) != cudaSuccess) return cerr(e, "predict buffers");
    cudaMemcpyAsync(w.X, X, sizeof(float) * n * in, cudaMemcpyHostToDevice, nullptr);
    forward(net, w, n);
    if ((e = cudaGetLastError()) != cudaSuccess) return cerr(e, "forward");
    e = cudaMemcpy(y, w.y, sizeof(float) * n, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? GAT_OK : cerr(e, "predict");
}

// Mean squared error and its gradient over all n rows (no update), for
// checking the kernels against a CPU reference.
int gat_mlp_gradient(const gat_mlp *net, const float *X, const float *T, int n,
                     float *grad_out, float *loss) {
    if (!net || !X || !T || !grad_out || n <= 0) return mlp_fail(GAT_ERR_ARGUMENT, "bad arguments");
    const int in = net->shape.in, P = net->shape.total;
    Work w;
    cudaError_t e;
    if ((e = w.alloc(n, in, n, P)) != cudaSuccess) return cerr(e, "gradient buffers");
    cudaMemcpyAsync(w.X, X, sizeof(float) * n * in, cudaMemcpyHostToDevice, nullptr);
    cudaMemcpyAsync(w.T, T, sizeof(float) * n, cudaMemcpyHostToDevice, nullptr);
    cudaMemsetAsync(w.loss, 0, sizeof(float), nullptr);
    launch(mlp_rows_kernel<true>, grid_for(n), 256, rows_smem(in), net->params, in, w.X, nullptr,
           w.T, n, w.y, w.h1, w.h2, w.dy, w.d2, w.d1);
    launch(mlp_param_kernel<false>, param_ctas(in), kGradThreads, kParamSmem, in, w.X, nullptr,
           w.h1, w.h2, w.dy, w.d2, w.d1, n, w.grad, AdamState{});
    sq_err_kernel<<<32, 256>>>(w.y, w.T, n, w.loss);
    if ((e = cudaGetLastError()) != cudaSuccess) return cerr(e, "gradient kernels");
    float s = 0.f;
    if ((e = cudaMemcpy(grad_out, w.grad, sizeof(float) * P, cudaMemcpyDeviceToHost)) !=
            cudaSuccess ||
        (e = cudaMemcpy(&s, w.loss, sizeof(float), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cerr(e, "gradient copy");
    if (loss) *loss = s / (float)n;
    return GAT_OK;
}

// Mini-batch Adam training on (X, T); rows are visited in a seeded random
// order each epoch.  *final_loss (may be null) is the full-data MSE after
// training.
int gat_mlp_train(gat_mlp *net, const float *X, const float *T, int n, int epochs,
                  int batch, float lr, uint64_t seed, float *final_loss) {
    if (!net || !X || !T || n <= 0 || epochs < 0 || batch <= 0)
        return mlp_fail(GAT_ERR_ARGUMENT, "bad arguments");
    const int in = net->shape.in;
    Work w;
    cudaError_t e;
    if ((e = w.alloc(n, in, std::min(batch, n), 0)) != cudaSuccess) return cerr(e, "train buffers");
    cudaMemcpyAsync(w.X, X, sizeof(float) * n * in, cudaMemcpyHostToDevice, nullptr);
    cudaMemcpyAsync(w.T, T, sizeof(float) * n, cudaMemcpyHostToDevice, nullptr);
    std::vector<int> order(n);
    for (int i = 0; i < n; i++) order[i] = i;
    std::mt19937_64 rng(seed);
    for (int ep = 0; ep < epochs; ep++) {
        std::shuffle(order.begin(), order.end(), rng);
        // (pageable memory: the copy has read `order` when the call returns)
        cudaMemcpyAsync(w.order, order.data(), sizeof(int) * n, cudaMemcpyHostToDevice, nullptr);
        for (int b0 = 0; b0 < n; b0 += batch) {
            const int nb = std::min(batch, n - b0);
            const int *rows = w.order + b0;
            launch(mlp_rows_kernel<true>, grid_for(nb), 256, rows_smem(in), net->params, in, w.X,
                   rows, w.T, nb, w.y, w.h1, w.h2, w.dy, w.d2, w.d1);
            net->step++;
            launch(mlp_param_kernel<true>, param_ctas(in), kGradThreads, kParamSmem, in, w.X, rows,
                   w.h1, w.h2, w.dy, w.d2, w.d1, nb, nullptr,
                   AdamState{net->params, net->m, net->v, lr, 0.9f, 0.999f, 1e-8f, net->step});
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return cerr(e, "training kernels");
    }
    if (final_loss) {
        cudaMemsetAsync(w.loss, 0, sizeof(float), nullptr);
        forward(net, w, n);
        sq_err_kernel<<<32, 256>>>(w.y, w.T, n, w.loss);
        float s = 0.f;
        if ((e = cudaMemcpy(&s, w.loss, sizeof(float), cudaMemcpyDeviceToHost)) != cudaSuccess)
            return cerr(e, "final loss");
        *final_loss = s / (float)n;
    }
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return cerr(e, "train");
    return GAT_OK;
}

}  // extern "C"
