// Learned schedule cost model: a small FP32 multilayer perceptron
// (inputs -> hidden -> hidden -> 1, ReLU) that predicts the log run time of a
// unit under a schedule from plan and schedule features.  Training and
// inference run on the GPU with the two kernels below (forward and backward
// pass of a tile of samples; gradient sum and Adam update); the training data
// are the autotuner's own timings.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "symgb.h"
#include "unit.hpp"

namespace {

// Samples of one tile.  One block evaluates a tile's forward and backward pass
// with the weights and every activation in shared memory: nothing but X, y and
// the parameter gradients touches global memory.  16 samples give the cost
// model's few thousand samples about one block per SM (157 blocks at 2500);
// with 32 half the SMs would idle, with 8 the partial gradients double.
constexpr int kTile = 16;
constexpr int kQuad = 4;                    // samples per thread (one 16-byte load)
constexpr int kRow = kTile + 4;             // activation row [unit][sample]: 80 bytes keep 16-byte loads conflict-free
constexpr int kThreads = 256;
constexpr std::size_t kLayerBytes = 48 * 1024;  // most weights of one layer

struct Layout {  // offsets of the flattened parameters
    int in, h;
    __host__ __device__ int W1() const { return 0; }
    __host__ __device__ int b1() const { return in * h; }
    __host__ __device__ int W2() const { return b1() + h; }
    __host__ __device__ int b2() const { return W2() + h * h; }
    __host__ __device__ int W3() const { return b2() + h; }
    __host__ __device__ int b3() const { return W3() + h; }
    __host__ __device__ int count() const { return b3() + 1; }
    // Shared memory: W1, W2 (rows h + 1 long: read along rows by the forward
    // and along columns by the backward pass, both without bank conflicts),
    // W3, b1, b2, then the activation rows X, H1, H2, D2, D1 and d3.
    __host__ __device__ int rowsAt() const { return (in * h + h * (h + 1) + 3 * h + 3) / 4 * 4; }
    std::size_t sharedBytes() const { return sizeof(float) * (rowsAt() + (std::size_t)(in + 4 * h + 1) * kRow); }
};

// out[o][s] = act(b[o] + sum_i in[i][s] W[i * ld + o]), i ascending, for the
// tile's samples; a thread takes one unit o of four samples.
__device__ __forceinline__ void forwardLayer(const float* __restrict__ src, const float* __restrict__ W, int ld,
                                             const float* __restrict__ b, float* __restrict__ dst, int in, int out) {
    for (int q = threadIdx.x; q < out * (kTile / kQuad); q += kThreads) {
        const int o = q % out, s = q / out * kQuad;
        const float b0 = b[o];
        float4 a = make_float4(b0, b0, b0, b0);
#pragma unroll 8
        for (int i = 0; i < in; ++i) {
            const float w = W[i * ld + o];
            const float4 x = *reinterpret_cast<const float4*>(src + i * kRow + s);
            a.x = fmaf(x.x, w, a.x);
            a.y = fmaf(x.y, w, a.y);
            a.z = fmaf(x.z, w, a.z);
            a.w = fmaf(x.w, w, a.w);
        }
        *reinterpret_cast<float4*>(dst + o * kRow + s) =
            make_float4(fmaxf(a.x, 0.f), fmaxf(a.y, 0.f), fmaxf(a.z, 0.f), fmaxf(a.w, 0.f));
    }
}

// dW[i * out + o] (+)= sum_s act[i][s] dZ[o][s] over the tile's samples, and
// db[o] (+)= sum_s dZ[o][s]; a thread takes one column o of four rows i.
__device__ __forceinline__ void gradLayer(const float* __restrict__ act, const float* __restrict__ dZ,
                                          float* __restrict__ dW, float* __restrict__ db, int in, int out, bool add) {
    const int groups = (in + 3) / 4;
    for (int q = threadIdx.x; q < out * groups; q += kThreads) {
        const int o = q % out, i0 = q / out * 4;
        float4 d[kTile / kQuad];
#pragma unroll
        for (int s = 0; s < kTile / kQuad; ++s) d[s] = *reinterpret_cast<const float4*>(dZ + o * kRow + s * kQuad);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + j;
            if (i >= in) break;
            float acc = 0.f;
#pragma unroll
            for (int s = 0; s < kTile / kQuad; ++s) {
                const float4 a = *reinterpret_cast<const float4*>(act + i * kRow + s * kQuad);
                acc = fmaf(d[s].x, a.x, acc);
                acc = fmaf(d[s].y, a.y, acc);
                acc = fmaf(d[s].z, a.z, acc);
                acc = fmaf(d[s].w, a.w, acc);
            }
            float* w = dW + i * out + o;
            *w = add ? *w + acc : acc;
        }
        if (i0 == 0) {
            float acc = 0.f;
#pragma unroll
            for (int s = 0; s < kTile / kQuad; ++s) acc += ((d[s].x + d[s].y) + (d[s].z + d[s].w));
            db[o] = add ? db[o] + acc : acc;
        }
    }
}

// Forward pass of every tile (tiles blockIdx.x, blockIdx.x + gridDim.x, ...):
// out and, with y, the squared errors sq; with `parts`, also the backward pass
// of the mean squared error, the block's summed parameter gradients going to
// parts[blockIdx.x * count + ...].
// One launch in place of eleven (three layers forward, the loss, seven
// backward) that each re-read the activations from global memory, the weight
// gradients with one block per column over all samples.  An epoch on a GB300,
// 64 hidden units: 2500 samples of 50 features 688 us before, 23 us now (16
// this kernel, 6 the gradient sum); 5000 of 62 1230 us, 39 us.  What remains
// is the latency of one tile's chain of layers: 512 threads of two samples
// each take 25 us and 31 us.
__global__ void __launch_bounds__(kThreads) tilePass(const float* __restrict__ X, const float* __restrict__ y,
                                                     const float* __restrict__ P, int n, Layout L,
                                                     float* __restrict__ out, float* __restrict__ sq,
                                                     float* __restrict__ parts) {
    extern __shared__ __align__(16) float sm[];
    const int in = L.in, h = L.h;
    float* sW1 = sm;
    float* sW2 = sW1 + in * h;
    float* sW3 = sW2 + h * (h + 1);
    float* sb1 = sW3 + h;
    float* sb2 = sb1 + h;
    float* sX = sm + L.rowsAt();
    float* sH1 = sX + in * kRow;
    float* sH2 = sH1 + h * kRow;
    float* sD2 = sH2 + h * kRow;
    float* sD1 = sD2 + h * kRow;
    float* sd3 = sD1 + h * kRow;
    for (int q = threadIdx.x; q < in * h; q += kThreads) sW1[q] = P[L.W1() + q];
    for (int q = threadIdx.x; q < h * h; q += kThreads) sW2[q / h * (h + 1) + q % h] = P[L.W2() + q];
    for (int q = threadIdx.x; q < h; q += kThreads) {
        sW3[q] = P[L.W3() + q];
        sb1[q] = P[L.b1() + q];
        sb2[q] = P[L.b2() + q];
    }
    float* G = parts ? parts + (std::size_t)blockIdx.x * L.count() : nullptr;
    bool add = false;
    const int tiles = (n + kTile - 1) / kTile;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, add = true) {
        const int row0 = t * kTile, rows = min(kTile, n - row0);
        for (int q = threadIdx.x; q < kTile * in; q += kThreads) {  // past the end zeros, their error taken as zero
            const int r = q / in, i = q % in;
            sX[i * kRow + r] = r < rows ? X[(std::size_t)(row0 + r) * in + i] : 0.f;
        }
        __syncthreads();
        forwardLayer(sX, sW1, h, sb1, sH1, in, h);
        __syncthreads();
        forwardLayer(sH1, sW2, h + 1, sb2, sH2, h, h);
        __syncthreads();
        if (threadIdx.x < kTile) {
            const int r = threadIdx.x;
            float acc = P[L.b3()], d = 0.f;
#pragma unroll 8
            for (int i = 0; i < h; ++i) acc = fmaf(sH2[i * kRow + r], sW3[i], acc);
            if (r < rows) {
                out[row0 + r] = acc;
                if (y) {
                    const float e = acc - y[row0 + r];
                    sq[row0 + r] = e * e;
                    d = 2.f * e / n;
                }
            }
            sd3[r] = d;
        }
        __syncthreads();
        if (parts) {
            for (int q = threadIdx.x; q < h * kTile; q += kThreads) {
                const int o = q / kTile, r = q % kTile;
                sD2[o * kRow + r] = sH2[o * kRow + r] <= 0.f ? 0.f : sd3[r] * sW3[o];
            }
            __syncthreads();
            // D1[i][s] = sum_o D2[o][s] W2[i][o], o ascending, where H1 > 0
            for (int q = threadIdx.x; q < h * (kTile / kQuad); q += kThreads) {
                const int i = q % h, s = q / h * kQuad;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
                for (int o = 0; o < h; ++o) {
                    const float w = sW2[i * (h + 1) + o];
                    const float4 d = *reinterpret_cast<const float4*>(sD2 + o * kRow + s);
                    a.x = fmaf(d.x, w, a.x);
                    a.y = fmaf(d.y, w, a.y);
                    a.z = fmaf(d.z, w, a.z);
                    a.w = fmaf(d.w, w, a.w);
                }
                const float4 f = *reinterpret_cast<const float4*>(sH1 + i * kRow + s);
                *reinterpret_cast<float4*>(sD1 + i * kRow + s) =
                    make_float4(f.x <= 0.f ? 0.f : a.x, f.y <= 0.f ? 0.f : a.y, f.z <= 0.f ? 0.f : a.z,
                                f.w <= 0.f ? 0.f : a.w);
            }
            gradLayer(sH2, sd3, G + L.W3(), G + L.b3(), h, 1, add);
            gradLayer(sH1, sD2, G + L.W2(), G + L.b2(), h, h, add);
            __syncthreads();
            gradLayer(sX, sD1, G + L.W1(), G + L.b1(), in, h, add);
        }
        __syncthreads();  // the next tile overwrites the rows
    }
}

// s + e += v, e the rounding error of the running sum (Knuth's TwoSum); NaN
// once the sum is not finite.
__device__ __forceinline__ void addCompensated(float& s, float& e, float v) {
    const float t = __fadd_rn(s, v), z = __fsub_rn(t, s);
    e = __fadd_rn(e, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(v, z)));
    s = t;
}

struct Adam {
    float lr, b1, b2, c1, c2, eps;
};

// Sum of the blocks' gradients, compensated (the sum over a few hundred
// partial sums adds no error to speak of to theirs), 32 parameters per
// block and 8 threads each; then Adam's update, or with p == nullptr the
// gradient itself into g.
__global__ void __launch_bounds__(kThreads) reduceUpdate(const float* __restrict__ parts, int blocks, int count,
                                                         float* __restrict__ g, float* __restrict__ p,
                                                         float* __restrict__ m, float* __restrict__ v, Adam A) {
    __shared__ float ss[kThreads], se[kThreads];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, slices = kThreads / 32;
    const int q = blockIdx.x * 32 + lane;
    float s = 0.f, e = 0.f;
    if (q < count)
#pragma unroll 8
        for (int b = slice; b < blocks; b += slices) addCompensated(s, e, parts[(std::size_t)b * count + q]);
    ss[threadIdx.x] = s;
    se[threadIdx.x] = e;
    __syncthreads();
    if (slice || q >= count) return;
    for (int t = 1; t < slices; ++t) {
        addCompensated(s, e, ss[t * 32 + lane]);
        e += se[t * 32 + lane];
    }
    const float gi = isfinite(s) ? s + e : s;
    if (!p) {
        g[q] = gi;
        return;
    }
    m[q] = A.b1 * m[q] + (1.f - A.b1) * gi;
    v[q] = A.b2 * v[q] + (1.f - A.b2) * gi * gi;
    p[q] -= A.lr * (m[q] / A.c1) / (sqrtf(v[q] / A.c2) + A.eps);
}

}  // namespace

struct symgb_mlp {
    int in = 0, hidden = 0;
    // parameter layout: W1 (in x h), b1 (h), W2 (h x h), b2 (h), W3 (h x 1), b3 (1)
    std::size_t oW1, ob1, oW2, ob2, oW3, ob3, count;
    float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
    float *X = nullptr, *y = nullptr, *out = nullptr, *sq = nullptr, *parts = nullptr;
    int partBlocks = 0;  // blocks `parts` holds
    int smCount = 1;
    Layout layout() const { return Layout{in, hidden}; }
    int cap = 0, step = 0;
    ~symgb_mlp() {
        for (float* p : {params, grads, m, v, X, y, out, sq, parts})
            if (p) cudaFree(p);
    }
};

namespace {

int mlpFail(int code, const std::string& msg) { return symgb::engine::setLastError(code, msg); }

#define MLP_CUDA(call)                                                                                      \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) return mlpFail(SYMGB_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// Blocks of a pass over n samples: one tile each, at most two per SM.
int passBlocks(const symgb_mlp* net, int n) { return std::min((n + kTile - 1) / kTile, 2 * net->smCount); }

int ensureBatch(symgb_mlp* net, int n) {
    if (n <= net->cap) return SYMGB_OK;
    for (float** p : {&net->X, &net->y, &net->out, &net->sq})
        if (*p) {
            cudaFree(*p);
            *p = nullptr;
        }
    net->cap = 0;
    MLP_CUDA(cudaMalloc(&net->X, sizeof(float) * n * net->in));
    MLP_CUDA(cudaMalloc(&net->y, sizeof(float) * n));
    MLP_CUDA(cudaMalloc(&net->out, sizeof(float) * n));
    MLP_CUDA(cudaMalloc(&net->sq, sizeof(float) * n));
    net->cap = n;
    return SYMGB_OK;
}

int ensureParts(symgb_mlp* net, int n) {
    const int blocks = passBlocks(net, n);
    if (blocks <= net->partBlocks) return SYMGB_OK;
    if (net->parts) cudaFree(net->parts);
    net->parts = nullptr;
    net->partBlocks = 0;
    MLP_CUDA(cudaMalloc(&net->parts, sizeof(float) * blocks * net->count));
    net->partBlocks = blocks;
    return SYMGB_OK;
}

// Forward pass, with `y` the squared errors, with `backward` the blocks' gradients.
int pass(symgb_mlp* net, int n, const float* y, bool backward) {
    const Layout L = net->layout();
    const std::size_t h = (std::size_t)net->hidden;
    if (sizeof(float) * std::max(net->in * h, h * h) > kLayerBytes)
        return mlpFail(SYMGB_ERR_CUDA, "MLP layer exceeds 48 KB of weights");
    const std::size_t smem = L.sharedBytes();
    tilePass<<<passBlocks(net, n), kThreads, smem>>>(net->X, y, net->params, n, L, net->out, net->sq,
                                                     backward ? net->parts : nullptr);
    return SYMGB_OK;
}

// Sums the blocks' gradients; with `A` updates the parameters, else into net->grads.
void reduce(symgb_mlp* net, int n, const Adam* A) {
    reduceUpdate<<<(unsigned)((net->count + 31) / 32), kThreads>>>(net->parts, passBlocks(net, n), (int)net->count,
                                                                   net->grads, A ? net->params : nullptr, net->m,
                                                                   net->v, A ? *A : Adam{});
}

int upload(symgb_mlp* net, const float* X, const float* y, int n) {
    if (int e = ensureBatch(net, n)) return e;
    MLP_CUDA(cudaMemcpy(net->X, X, sizeof(float) * n * net->in, cudaMemcpyHostToDevice));
    if (y) MLP_CUDA(cudaMemcpy(net->y, y, sizeof(float) * n, cudaMemcpyHostToDevice));
    return SYMGB_OK;
}

int meanLoss(symgb_mlp* net, int n, float* loss) {
    std::vector<float> sq(n);
    MLP_CUDA(cudaMemcpy(sq.data(), net->sq, sizeof(float) * n, cudaMemcpyDeviceToHost));
    double s = 0;
    for (float e : sq) s += e;
    *loss = (float)(s / n);
    return SYMGB_OK;
}

}  // namespace

extern "C" {

int symgb_mlp_create(int inputs, int hidden, unsigned long long seed, symgb_mlp_t* out) {
    if (!out || inputs <= 0 || hidden <= 0 || hidden > 256 || inputs > 256) return mlpFail(SYMGB_ERR_ARGUMENT, "bad MLP shape");
    std::unique_ptr<symgb_mlp> net(new symgb_mlp());
    net->in = inputs;
    net->hidden = hidden;
    std::size_t o = 0;
    net->oW1 = o; o += (std::size_t)inputs * hidden;
    net->ob1 = o; o += hidden;
    net->oW2 = o; o += (std::size_t)hidden * hidden;
    net->ob2 = o; o += hidden;
    net->oW3 = o; o += hidden;
    net->ob3 = o; o += 1;
    net->count = o;
    // He-style initialisation from a seeded generator (host), biases zero.
    std::vector<float> p(o, 0.f);
    std::uint64_t s = seed * 0x9e3779b97f4a7c15ULL + 1;
    auto uni = [&]() {
        s ^= s << 13; s ^= s >> 7; s ^= s << 17;
        return (float)((s >> 11) * (1.0 / 9007199254740992.0)) * 2.f - 1.f;
    };
    const float a1 = std::sqrt(6.f / inputs), a2 = std::sqrt(6.f / hidden);
    for (std::size_t q = 0; q < (std::size_t)inputs * hidden; ++q) p[net->oW1 + q] = a1 * uni();
    for (std::size_t q = 0; q < (std::size_t)hidden * hidden; ++q) p[net->oW2 + q] = a2 * uni();
    for (int q = 0; q < hidden; ++q) p[net->oW3 + q] = a2 * uni();
    for (float** b : {&net->params, &net->grads, &net->m, &net->v}) MLP_CUDA(cudaMalloc(b, sizeof(float) * o));
    MLP_CUDA(cudaMemcpy(net->params, p.data(), sizeof(float) * o, cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemset(net->m, 0, sizeof(float) * o));
    MLP_CUDA(cudaMemset(net->v, 0, sizeof(float) * o));
    int device = 0;
    MLP_CUDA(cudaGetDevice(&device));
    MLP_CUDA(cudaDeviceGetAttribute(&net->smCount, cudaDevAttrMultiProcessorCount, device));
    // The shared memory a pass may have is the kernel's, not the network's: the
    // most there is, as another thread's network could lower a size of this
    // one's own between here and its launch.
    int most = 0;
    MLP_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    MLP_CUDA(cudaFuncSetAttribute(tilePass, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    *out = net.release();
    return SYMGB_OK;
}

int symgb_mlp_num_params(symgb_mlp_t net) { return net ? (int)net->count : 0; }

int symgb_mlp_get_params(symgb_mlp_t net, float* p) {
    if (!net || !p) return mlpFail(SYMGB_ERR_ARGUMENT, "null argument");
    MLP_CUDA(cudaMemcpy(p, net->params, sizeof(float) * net->count, cudaMemcpyDeviceToHost));
    return SYMGB_OK;
}

int symgb_mlp_set_params(symgb_mlp_t net, const float* p) {
    if (!net || !p) return mlpFail(SYMGB_ERR_ARGUMENT, "null argument");
    MLP_CUDA(cudaMemcpy(net->params, p, sizeof(float) * net->count, cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemset(net->m, 0, sizeof(float) * net->count));
    MLP_CUDA(cudaMemset(net->v, 0, sizeof(float) * net->count));
    net->step = 0;
    return SYMGB_OK;
}

int symgb_mlp_forward(symgb_mlp_t net, const float* X, int n, float* y) {
    if (!net || !X || !y || n <= 0) return mlpFail(SYMGB_ERR_ARGUMENT, "bad forward arguments");
    if (int e = upload(net, X, nullptr, n)) return e;
    if (int e = pass(net, n, nullptr, false)) return e;
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaMemcpy(y, net->out, sizeof(float) * n, cudaMemcpyDeviceToHost));
    return SYMGB_OK;
}

int symgb_mlp_gradient(symgb_mlp_t net, const float* X, const float* y, int n, float* grad, float* loss) {
    if (!net || !X || !y || !grad || n <= 0) return mlpFail(SYMGB_ERR_ARGUMENT, "bad gradient arguments");
    if (int e = upload(net, X, y, n)) return e;
    if (int e = ensureParts(net, n)) return e;
    if (int e = pass(net, n, net->y, true)) return e;
    reduce(net, n, nullptr);
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaMemcpy(grad, net->grads, sizeof(float) * net->count, cudaMemcpyDeviceToHost));
    if (loss) return meanLoss(net, n, loss);
    return SYMGB_OK;
}

int symgb_mlp_train(symgb_mlp_t net, const float* X, const float* y, int n, int epochs, float lr, float* loss) {
    if (!net || !X || !y || n <= 0 || epochs < 0) return mlpFail(SYMGB_ERR_ARGUMENT, "bad training arguments");
    if (int e = upload(net, X, y, n)) return e;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    if (epochs)
        if (int e = ensureParts(net, n)) return e;
    for (int ep = 0; ep < epochs; ++ep) {
        if (int e = pass(net, n, net->y, true)) return e;
        ++net->step;
        const float c1 = 1.f - std::pow(b1, (float)net->step), c2 = 1.f - std::pow(b2, (float)net->step);
        const Adam A{lr, b1, b2, c1, c2, eps};
        reduce(net, n, &A);
    }
    MLP_CUDA(cudaGetLastError());
    if (int e = pass(net, n, net->y, false)) return e;
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaDeviceSynchronize());
    if (loss) return meanLoss(net, n, loss);
    return SYMGB_OK;
}

void symgb_mlp_destroy(symgb_mlp_t net) { delete net; }

}  // extern "C"
