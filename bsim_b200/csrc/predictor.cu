// The firing predictor's MLP (9 -> 64 -> 64 -> 1, ReLU): deterministic
// initialisation, batched forward pass, mean-squared-error backward pass and
// Adam training, all as hand-written CUDA kernels. Inference inside the
// simulation step lives in step.cu (one warp per population).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "engine.h"
#include "netgen.h"

namespace bsim {
int record_error(int code, const std::string &msg);
}
using namespace bsim;

namespace {

constexpr int IN = BSIM_MLP_IN, H = BSIM_MLP_HIDDEN, NP = BSIM_MLP_PARAMS;
constexpr int OFF_W1 = 0, OFF_B1 = H * IN, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H, OFF_W3 = OFF_B2 + H,
              OFF_B3 = OFF_W3 + H;
static_assert(OFF_B3 + 1 == NP, "parameter layout");

int fail(int code, const std::string &m, cudaError_t st = cudaSuccess)
{
    return record_error(code, st == cudaSuccess ? m : m + ": " + cudaGetErrorString(st));
}

// One block evaluates tiles of GT samples, its 256 threads as 16 x 16 over the (sample, unit) outputs
// of a layer, 4 x 4 outputs per thread in registers, operands in shared memory (rows of LD floats:
// 16-byte loads of 8 neighbouring rows fall on distinct banks). The products are fp32 FMAs; the
// arithmetic bounds it: 28,000 FMAs per sample, forward and backward. Each sum runs over its terms in
// ascending order from the bias (or zero), and a tile's gradients are added to the result with one
// reduction per parameter.
//
// MLP_FORWARD writes y, MLP_LOSS adds the mean squared error, MLP_GRAD the gradients as well. With
// `adam` set (training), samples are taken through idx and the last block to finish applies the
// update and clears the gradients, so a training step is one launch.
//
// Measured against one thread per sample and 64 samples per block, with gathering, clearing and
// the update as launches of their own: one epoch over 65,001 host samples in batches of 8,192, medians
// of 80 calls 2.9 to 3.3 ms -> 1.5 to 1.7 ms (5th to 95th percentile 2.8 to 3.8 and 1.5 to 1.9 without
// stragglers; the rest is mostly allocation, the shuffle and the samples' way to the GPU).
enum { MLP_FORWARD, MLP_LOSS, MLP_GRAD };
constexpr int GT = 64, LD = H + 4, MLP_THREADS = 256;
constexpr int64_t MLP_MAX_BLOCKS = 4096;  // blocks of a large pass take several tiles
constexpr int SM_W1 = 0, SM_B1 = SM_W1 + H * IN, SM_W2 = SM_B1 + H, SM_B2 = SM_W2 + H * LD, SM_W3 = SM_B2 + H,
              SM_H1 = SM_W3 + H, SM_H2 = SM_H1 + GT * LD, SM_X = SM_H2 + GT * LD, SM_DY = SM_X + GT * IN,
              SM_DZ2 = SM_DY + GT, SM_DZ1 = SM_DZ2 + GT * LD, SM_END = SM_DZ1 + GT * LD;
static_assert(SM_W2 % 4 == 0 && SM_H1 % 4 == 0 && SM_DZ2 % 4 == 0, "16-byte rows");

struct AdamArgs {
    float *m, *v;
    const uint32_t *idx;    // the batch's samples
    unsigned int *ticket;   // blocks done
    float lr, b1t, b2t;     // learning rate, 0.9^t, 0.999^t
};

__device__ __forceinline__ void adam_update(float *p, float g, float *m, float *v, const AdamArgs &o)
{
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * *m + (1.0f - b1) * g, vi = b2 * *v + (1.0f - b2) * g * g;
    *m = mi;
    *v = vi;
    const float mh = mi / (1.0f - o.b1t), vh = vi / (1.0f - o.b2t);
    *p -= o.lr * mh / (sqrtf(vh) + eps);
}

template <int MODE>
__global__ void __launch_bounds__(MLP_THREADS) mlp_kernel(float *params, const float *x, const float *y_target, int64_t n,
                                                          float *y_out, float *grad, double *loss_acc, const AdamArgs adam)
{
    extern __shared__ __align__(16) float sm[];
    __shared__ bool s_last;
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    for (int i = t; i < H * IN; i += MLP_THREADS) sm[SM_W1 + i] = params[OFF_W1 + i];
    for (int i = t; i < H * H; i += MLP_THREADS) sm[SM_W2 + (i / H) * LD + i % H] = params[OFF_W2 + i];
    if (t < H) {
        sm[SM_B1 + t] = params[OFF_B1 + t];
        sm[SM_B2 + t] = params[OFF_B2 + t];
        sm[SM_W3 + t] = params[OFF_W3 + t];
    }
    const float b3 = params[OFF_B3];
    double sq = 0.0;
    for (int64_t tile = blockIdx.x; tile * GT < n; tile += gridDim.x) {
        const int64_t i0 = tile * GT;
        __syncthreads();  // the previous tile's values have been read
        for (int i = t; i < GT * IN; i += MLP_THREADS) {  // samples past the end are zeros
            const int64_t r = i0 + i / IN;
            sm[SM_X + i] = r < n ? x[(adam.idx ? (int64_t)adam.idx[r] : r) * IN + i % IN] : 0.0f;
        }
        __syncthreads();
        float acc[4][4];
        // first layer
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = sm[SM_B1 + tx + 16 * b];
        for (int k = 0; k < IN; k++) {
            float xs[4], w[4];
#pragma unroll
            for (int a = 0; a < 4; a++) xs[a] = sm[SM_X + (ty + 16 * a) * IN + k];
#pragma unroll
            for (int b = 0; b < 4; b++) w[b] = sm[SM_W1 + (tx + 16 * b) * IN + k];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) acc[a][b] = fmaf(w[b], xs[a], acc[a][b]);
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) sm[SM_H1 + (ty + 16 * a) * LD + tx + 16 * b] = fmaxf(acc[a][b], 0.0f);
        __syncthreads();
        // second layer
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = sm[SM_B2 + tx + 16 * b];
        for (int k = 0; k < H; k += 4) {
            float4 h[4], w[4];
#pragma unroll
            for (int a = 0; a < 4; a++) h[a] = *reinterpret_cast<const float4 *>(sm + SM_H1 + (ty + 16 * a) * LD + k);
#pragma unroll
            for (int b = 0; b < 4; b++) w[b] = *reinterpret_cast<const float4 *>(sm + SM_W2 + (tx + 16 * b) * LD + k);
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    acc[a][b] = fmaf(w[b].x, h[a].x, acc[a][b]);
                    acc[a][b] = fmaf(w[b].y, h[a].y, acc[a][b]);
                    acc[a][b] = fmaf(w[b].z, h[a].z, acc[a][b]);
                    acc[a][b] = fmaf(w[b].w, h[a].w, acc[a][b]);
                }
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) sm[SM_H2 + (ty + 16 * a) * LD + tx + 16 * b] = fmaxf(acc[a][b], 0.0f);
        __syncthreads();
        // output and error, one thread per sample
        if (t < GT) {
            float y = b3;
            for (int u = 0; u < H; u++) y = fmaf(sm[SM_W3 + u], sm[SM_H2 + t * LD + u], y);
            if (i0 + t < n) {
                if (MODE == MLP_FORWARD) {
                    y_out[i0 + t] = y;
                } else {
                    const float e = y - y_target[adam.idx ? (int64_t)adam.idx[i0 + t] : i0 + t];
                    sq += (double)e * (double)e;
                    sm[SM_DY + t] = 2.0f * e / (float)n;
                }
            } else {
                sm[SM_DY + t] = 0.0f;  // contributes nothing
            }
        }
        if (MODE != MLP_GRAD) continue;
        __syncthreads();
        for (int i = t; i < GT * H; i += MLP_THREADS) {
            const int s = i / H, u = i % H;
            sm[SM_DZ2 + s * LD + u] = sm[SM_H2 + s * LD + u] > 0.0f ? sm[SM_DY + s] * sm[SM_W3 + u] : 0.0f;
        }
        __syncthreads();
        // error at the first layer
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = 0.0f;
        for (int u = 0; u < H; u += 4) {
            float4 d[4];
#pragma unroll
            for (int a = 0; a < 4; a++) d[a] = *reinterpret_cast<const float4 *>(sm + SM_DZ2 + (ty + 16 * a) * LD + u);
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const float *w = sm + SM_W2 + u * LD + tx + 16 * b;
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    acc[a][b] = fmaf(d[a].x, w[0], acc[a][b]);
                    acc[a][b] = fmaf(d[a].y, w[LD], acc[a][b]);
                    acc[a][b] = fmaf(d[a].z, w[2 * LD], acc[a][b]);
                    acc[a][b] = fmaf(d[a].w, w[3 * LD], acc[a][b]);
                }
            }
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int at = (ty + 16 * a) * LD + tx + 16 * b;
                sm[SM_DZ1 + at] = sm[SM_H1 + at] > 0.0f ? acc[a][b] : 0.0f;
            }
        __syncthreads();
        // gradients of the tile: W2 in 4 x 4 pieces, the rest one parameter per thread
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = 0.0f;
        for (int s = 0; s < GT; s++) {
            const float4 d = *reinterpret_cast<const float4 *>(sm + SM_DZ2 + s * LD + 4 * ty);
            const float4 h = *reinterpret_cast<const float4 *>(sm + SM_H1 + s * LD + 4 * tx);
            const float dd[4] = {d.x, d.y, d.z, d.w}, hh[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) acc[a][b] = fmaf(dd[a], hh[b], acc[a][b]);
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++)
                if (acc[a][b] != 0.0f) atomicAdd(&grad[OFF_W2 + (4 * ty + a) * H + 4 * tx + b], acc[a][b]);
        for (int j = t; j < H * IN + 3 * H + 1; j += MLP_THREADS) {
            float g = 0.0f;
            int at;
            if (j < H * IN) {  // W1[u][k]
                const int u = j / IN, k = j % IN;
                for (int b = 0; b < GT; b++) g = fmaf(sm[SM_DZ1 + b * LD + u], sm[SM_X + b * IN + k], g);
                at = OFF_W1 + j;
            } else if (j < H * IN + H) {  // b1[u]
                at = OFF_B1 + j - H * IN;
                for (int b = 0; b < GT; b++) g += sm[SM_DZ1 + b * LD + (j - H * IN)];
            } else if (j < H * IN + 2 * H) {  // b2[u]
                at = OFF_B2 + j - H * IN - H;
                for (int b = 0; b < GT; b++) g += sm[SM_DZ2 + b * LD + (j - H * IN - H)];
            } else if (j < H * IN + 3 * H) {  // W3[u]
                at = OFF_W3 + j - H * IN - 2 * H;
                for (int b = 0; b < GT; b++) g = fmaf(sm[SM_DY + b], sm[SM_H2 + b * LD + (j - H * IN - 2 * H)], g);
            } else {  // b3
                at = OFF_B3;
                for (int b = 0; b < GT; b++) g += sm[SM_DY + b];
            }
            if (g != 0.0f) atomicAdd(&grad[at], g);
        }
    }
    if (MODE != MLP_FORWARD && loss_acc && t < GT) {
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if ((t & 31) == 0 && sq != 0.0) atomicAdd(loss_acc, sq / (double)n);
    }
    if (MODE == MLP_GRAD && adam.ticket) {
        __threadfence();
        __syncthreads();
        if (t == 0) s_last = atomicAdd(adam.ticket, 1u) == gridDim.x - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        for (int i = t; i < NP; i += MLP_THREADS) {
            adam_update(&params[i], __ldcg(&grad[i]), &adam.m[i], &adam.v[i], adam);
            grad[i] = 0.0f;
        }
        if (t == 0) *adam.ticket = 0u;
    }
}

// One pass over n samples: a block per tile (two blocks share an SM).
template <int MODE>
cudaError_t launch_mlp(float *p, const float *x, const float *y, int64_t n, float *y_out, float *g, double *l,
                       const AdamArgs &adam = AdamArgs{})
{
    const size_t bytes = sizeof(float) * (MODE == MLP_GRAD ? SM_END : SM_DZ2);
    cudaError_t st = cudaFuncSetAttribute(mlp_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (st != cudaSuccess) return st;
    const int64_t tiles = (n + GT - 1) / GT;
    mlp_kernel<MODE><<<(unsigned)std::min<int64_t>(tiles, MLP_MAX_BLOCKS), MLP_THREADS, bytes>>>(p, x, y, n, y_out, g, l, adam);
    return cudaGetLastError();
}

// The shuffle's partner of each position (Fisher-Yates, i from n-1 down): j[i] = hash % (i + 1).
__global__ void shuffle_kernel(uint64_t seed, uint64_t epoch, int64_t n, uint32_t *j)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        j[i] = (uint32_t)(hash3(seed, epoch, (uint64_t)i) % (uint64_t)(i + 1));
}

struct DevBuf {
    std::vector<void *> p;
    ~DevBuf()
    {
        for (void *q : p) cudaFree(q);
    }
    template <typename T>
    cudaError_t get(T **out, size_t count)
    {
        cudaError_t st = cudaMalloc((void **)out, sizeof(T) * (count ? count : 1));
        if (st == cudaSuccess) p.push_back(*out);
        return st;
    }
};

}  // namespace

extern "C" int bsim_mlp_init(float *params, uint64_t seed)
{
    if (!params) return fail(BSIM_ERR_ARG, "bsim_mlp_init: null params");
    memset(params, 0, sizeof(float) * NP);
    auto fill = [&](int off, int fan_in, int fan_out, int count, uint64_t salt) {
        const float a = sqrtf(6.0f / (float)(fan_in + fan_out));
        for (int i = 0; i < count; i++) {
            const float u = unit24((uint32_t)(hash3(seed, salt, (uint64_t)i) >> 40));
            params[off + i] = (2.0f * u - 1.0f) * a;
        }
    };
    fill(OFF_W1, IN, H, H * IN, 1);
    fill(OFF_W2, H, H, H * H, 2);
    fill(OFF_W3, H, 1, H, 3);
    return BSIM_OK;
}

extern "C" int bsim_mlp_forward(const float *params, const float *x, int64_t n, float *y)
{
    if (!params || n < 0 || (n > 0 && (!x || !y))) return fail(BSIM_ERR_ARG, "bsim_mlp_forward: invalid arguments");
    if (n == 0) return BSIM_OK;
    DevBuf b;
    float *dp, *dx, *dy;
    cudaError_t st;
    if ((st = b.get(&dp, NP)) || (st = b.get(&dx, n * IN)) || (st = b.get(&dy, n)))
        return fail(BSIM_ERR_NOMEM, "bsim_mlp_forward: allocation", st);
    cudaMemcpy(dp, params, sizeof(float) * NP, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x, sizeof(float) * n * IN, cudaMemcpyHostToDevice);
    if ((st = launch_mlp<MLP_FORWARD>(dp, dx, nullptr, n, dy, nullptr, nullptr)) != cudaSuccess)
        return fail(BSIM_ERR_CUDA, "bsim_mlp_forward", st);
    st = cudaMemcpy(y, dy, sizeof(float) * n, cudaMemcpyDeviceToHost);
    if (st != cudaSuccess) return fail(BSIM_ERR_CUDA, "bsim_mlp_forward", st);
    return BSIM_OK;
}

extern "C" int bsim_mlp_grad(const float *params, const float *x, const float *y_target, int64_t n, float *grad,
                             float *loss)
{
    if (!params || n <= 0 || !x || !y_target || !grad) return fail(BSIM_ERR_ARG, "bsim_mlp_grad: invalid arguments");
    DevBuf b;
    float *dp, *dx, *dt, *dg;
    double *dl;
    cudaError_t st;
    if ((st = b.get(&dp, NP)) || (st = b.get(&dx, n * IN)) || (st = b.get(&dt, n)) || (st = b.get(&dg, NP)) ||
        (st = b.get(&dl, 1)))
        return fail(BSIM_ERR_NOMEM, "bsim_mlp_grad: allocation", st);
    cudaMemcpy(dp, params, sizeof(float) * NP, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x, sizeof(float) * n * IN, cudaMemcpyHostToDevice);
    cudaMemcpy(dt, y_target, sizeof(float) * n, cudaMemcpyHostToDevice);
    cudaMemset(dg, 0, sizeof(float) * NP);
    cudaMemset(dl, 0, sizeof(double));
    if ((st = launch_mlp<MLP_GRAD>(dp, dx, dt, n, nullptr, dg, dl)) != cudaSuccess)
        return fail(BSIM_ERR_CUDA, "bsim_mlp_grad", st);
    double l = 0;
    st = cudaMemcpy(grad, dg, sizeof(float) * NP, cudaMemcpyDeviceToHost);
    if (st == cudaSuccess) st = cudaMemcpy(&l, dl, sizeof(double), cudaMemcpyDeviceToHost);
    if (st != cudaSuccess) return fail(BSIM_ERR_CUDA, "bsim_mlp_grad", st);
    if (loss) *loss = (float)l;
    return BSIM_OK;
}

extern "C" int bsim_mlp_train(float *params, const float *x, const float *y_target, int64_t n, int32_t epochs,
                              int32_t batch, float lr, uint64_t seed, float *final_loss)
{
    if (!params || n <= 0 || !x || !y_target || epochs < 0 || batch <= 0 || !(lr > 0))
        return fail(BSIM_ERR_ARG, "bsim_mlp_train: invalid arguments");
    if (n > (int64_t)UINT32_MAX) return fail(BSIM_ERR_LIMIT, "bsim_mlp_train: more than 2^32 samples");
    DevBuf b;
    const int64_t bs = std::min<int64_t>(batch, n);
    // one allocation: parameters, gradients, moments, loss and ticket, samples, the order of an epoch
    float *dp;
    cudaError_t st;
    const size_t head = 4 * (size_t)((NP + 3) / 4 * 4) + 4;
    if ((st = b.get(&dp, head + (size_t)n * (IN + 2) + 4))) return fail(BSIM_ERR_NOMEM, "bsim_mlp_train: allocation", st);
    const size_t np4 = (NP + 3) / 4 * 4;
    float *dg = dp + np4, *dm = dp + 2 * np4, *dv = dp + 3 * np4;
    double *dl = reinterpret_cast<double *>(dp + 4 * np4);
    unsigned int *ticket = reinterpret_cast<unsigned int *>(dp + 4 * np4 + 2);
    float *dx = dp + head, *dt = dx + (size_t)n * IN;
    uint32_t *didx = reinterpret_cast<uint32_t *>(dt + n);
    cudaMemset(dg, 0, sizeof(float) * (head - np4));
    cudaMemcpy(dp, params, sizeof(float) * NP, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x, sizeof(float) * n * IN, cudaMemcpyHostToDevice);
    cudaMemcpy(dt, y_target, sizeof(float) * n, cudaMemcpyHostToDevice);
    std::vector<uint32_t> idx(n), to(n);
    for (int64_t i = 0; i < n; i++) idx[i] = (uint32_t)i;
    AdamArgs adam{dm, dv, didx, ticket, lr, 1.0f, 1.0f};
    for (int ep = 0; ep < epochs; ep++) {
        // deterministic shuffle (Fisher-Yates on the seeded hash): the partners are drawn on the GPU,
        // into the place of the order they replace once the last epoch's batches have read it
        shuffle_kernel<<<256, 256>>>(seed, (uint64_t)ep, n, didx);
        cudaMemcpy(to.data(), didx, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost);
        for (int64_t i = n - 1; i > 0; i--) std::swap(idx[i], idx[to[i]]);
        cudaMemcpy(didx, idx.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice);
        for (int64_t b0 = 0; b0 + bs <= n; b0 += bs) {
            adam.idx = didx + b0;
            adam.b1t *= 0.9f;
            adam.b2t *= 0.999f;
            if ((st = launch_mlp<MLP_GRAD>(dp, dx, dt, bs, nullptr, dg, nullptr, adam)) != cudaSuccess)
                return fail(BSIM_ERR_CUDA, "bsim_mlp_train", st);
        }
    }
    // loss over the whole set
    if ((st = launch_mlp<MLP_LOSS>(dp, dx, dt, n, nullptr, nullptr, dl)) != cudaSuccess)
        return fail(BSIM_ERR_CUDA, "bsim_mlp_train", st);
    double l = 0;
    st = cudaMemcpy(params, dp, sizeof(float) * NP, cudaMemcpyDeviceToHost);
    if (st == cudaSuccess) st = cudaMemcpy(&l, dl, sizeof(double), cudaMemcpyDeviceToHost);
    if (st != cudaSuccess) return fail(BSIM_ERR_CUDA, "bsim_mlp_train", st);
    if (final_loss) *final_loss = (float)l;
    return BSIM_OK;
}
