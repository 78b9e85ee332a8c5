// Training and evaluation of the warm-start MLP (the C ABI jbgpu_mlp_* of include/jbgpu.h):
// mini-batch Adam on mean squared error of normalised targets, with the forward and backward
// products on the tensor cores (mlp.cuh) and FP32 gradients accumulated with atomics.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "../../include/jbgpu.h"
#include "mlp.cuh"

namespace jbg {
int set_last_error(int code, const char* msg);   // world.cu
}
using namespace jbg;

struct jbgpu_mlp {
    int device = 0, sms = 1;
    cudaStream_t s = nullptr;
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr, *norm = nullptr;
    float* loss = nullptr;                // behind the gradient: both are cleared and read together
    float* hostGrad = nullptr;            // pinned: gradient and loss
    __nv_bfloat16 *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
    float *X = nullptr, *T = nullptr;     // training set on the device
    int n = 0, cap = 0;
    int* idx = nullptr;                   // epoch permutation
    long long adamStep = 0;
    float* io = nullptr;                  // staging for forward / gradients (capacity ioCap samples)
    int ioCap = 0;
};

namespace jbg {

MlpDev mlp_view(const jbgpu_mlp* h) {
    MlpDev d;
    d.w1 = h->w1;
    d.w2 = h->w2;
    d.w3 = h->w3;
    d.p = h->p;
    d.norm = h->norm;
    return d;
}

// FP32 parameters -> padded BF16 weight copies.
__global__ void k_mlp_pack(const float* p, __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < MLP_H * MLP_INP) {
        int r = i / MLP_INP, c = i % MLP_INP;
        w1[i] = __float2bfloat16_rn(c < MLP_IN ? p[MLP_OFF_W1 + r * MLP_IN + c] : 0.0f);
    }
    if (i < MLP_H * MLP_H) w2[i] = __float2bfloat16_rn(p[MLP_OFF_W2 + i]);
    if (i < MLP_OUTP * MLP_H) {
        int r = i / MLP_H, c = i % MLP_H;
        w3[i] = __float2bfloat16_rn(r < MLP_OUT ? p[MLP_OFF_W3 + r * MLP_H + c] : 0.0f);
    }
}

// Normalised sample rows [first, first + 64) of X (through idx when given) into S.x.
JBD int mlp_load_inputs(MlpSmem& S, const MlpDev& M, const float* X, const int* idx, int first, int count) {
    int valid = min(MLP_TILE, count - first);
    for (int e = threadIdx.x; e < MLP_TILE * MLP_INP; e += blockDim.x) {
        int i = e / MLP_INP, k = e % MLP_INP;
        float v = 0.0f;
        if (i < valid && k < MLP_IN) {
            int row = idx ? idx[first + i] : first + i;
            v = mlp_norm_in(M.norm, k, X[(size_t)row * MLP_IN + k]);
        }
        S.x[i][k] = __float2bfloat16_rn(v);
    }
    return valid;
}

// c * gelu' as bf16 into dz (rows m0.., columns n0.. of the warp) and its column sums into b.
template <int NT>
JBD void mlp_dz(const float (&c)[NT][4], const float (&grad)[NT][4], __nv_bfloat16 (*dz)[MLP_LDH], float (&b)[NT][2], int m0,
                int n0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const __nv_bfloat16 x = __float2bfloat16_rn(c[q][2 * h] * grad[q][2 * h]);
            const __nv_bfloat16 y = __float2bfloat16_rn(c[q][2 * h + 1] * grad[q][2 * h + 1]);
            *(uint32_t*)&dz[m0 + g + 8 * h][n0 + 8 * q + 2 * t] = pack_bf16(x, y);
            b[q][0] += __bfloat162float(x);
            b[q][1] += __bfloat162float(y);
        }
}

// sum += A^T B over the tile's samples.  The tensor cores' sum starts from zero for each tile and is added
// rounded to nearest: kept as their accumulator over a block's tiles, every step cuts the sum towards zero,
// 3e-6 of the gradient at a million samples and 1.5e-5 at four million.
template <int NT>
JBD void mlp_add_tile(float (&sum)[NT][4], const __nv_bfloat16* a, int lda, const __nv_bfloat16* b, int ldb) {
    float c[NT][4] = {};
    warp_gemm<NT, MLP_TILE, true, true>(c, a, lda, b, ldb);
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
        for (int e = 0; e < 4; e++) sum[q][e] += c[q][e];
}

JBD void red_add2(float* p, float a, float b) {   // p 8-byte aligned
    asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b) : "memory");
}

// 64-sample tiles of a mini-batch: forward, loss, backward; the block's gradients stay in registers over
// its tiles and are added into grad at the end.  coef = 2 / (batch samples x outputs): the derivative of
// the batch-mean squared error.
// What bounds it: the length of one tile's chain, five products deep with a block barrier between.
// Operands gathered element by element from rows on the same banks, gelu' worked out again and a
// quarter as many warps took 55 us for 256 tiles; 21 us so.
__global__ void __launch_bounds__(MLP_TRAIN_THREADS) k_mlp_train(MlpDev M, const float* X, const float* T, const int* idx,
                                                                  int first, int count, float coef, float* grad,
                                                                  float* loss) {
    constexpr int WARPS = MLP_TRAIN_THREADS / 32, NT = MlpTiles<WARPS>::NT;
    extern __shared__ __align__(16) unsigned char mlpSmem[];
    MlpSmem& S = *reinterpret_cast<MlpSmem*>(mlpSmem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * 8 * NT;
    const int tiles = (count + MLP_TILE - 1) / MLP_TILE;
    mlp_load_weights(S, M);
    float lossSum = 0.0f;
    float b3 = 0.0f;                        // lane o of warp 0: db3[o]
    float b1[NT][2] = {}, b2[NT][2] = {};   // the lane's columns n0 + 8 q + 2 t + e, its rows alone
    float w3[2][4] = {}, w2[NT][4] = {}, w1[2][4] = {};
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int tileFirst = first + tile * MLP_TILE;
        const int valid = mlp_load_inputs(S, M, X, idx, tileFirst, first + count);
        __syncthreads();
        MlpTiles<WARPS> G;
        mlp_forward<WARPS>(S, M, G);
        // loss and dY (FP32 kept in S.y, BF16 copy padded to 16 columns in S.dy)
        for (int e = threadIdx.x; e < MLP_TILE * MLP_OUTP; e += blockDim.x) {
            int i = e / MLP_OUTP, o = e % MLP_OUTP;
            float d = 0.0f;
            if (i < valid && o < MLP_OUT) {
                int row = idx ? idx[tileFirst + i] : tileFirst + i;
                float tn = (T[(size_t)row * MLP_OUT + o] - M.norm[2 * MLP_IN + o]) / M.norm[2 * MLP_IN + MLP_OUT + o];
                float r = S.y[i][o] - tn;
                lossSum += r * r;
                d = coef * r;
            }
            S.dy[i][o] = __float2bfloat16_rn(d);
            if (o < MLP_OUT) S.y[i][o] = d;
        }
        __syncthreads();
        // dZ2 = (dY W3) * gelu'(Z2)
        {
            float c[NT][4] = {};
            warp_gemm<NT, MLP_OUTP, false, true>(c, &S.dy[m0][0], MLP_LDO, &S.w3[0][n0], MLP_LDH);
            mlp_dz(c, G.g2, S.dz2, b2, m0, n0);
        }
        // dW3 = dY^T H2 (16 padded rows), the columns over the warps by twos of tiles
        if (warp < 4) mlp_add_tile<2>(w3, &S.dy[0][0], MLP_LDO, &S.h2[0][16 * warp], MLP_LDH);
        else if (warp == 4 && lane < MLP_OUT)
            for (int i = 0; i < MLP_TILE; i++) b3 += S.y[i][lane];
        __syncthreads();
        // dZ1 = (dZ2 W2) * gelu'(Z1); dW2 = dZ2^T H1
        {
            float c[NT][4] = {};
            warp_gemm<NT, MLP_H, false, true>(c, &S.dz2[m0][0], MLP_LDH, &S.w2[0][n0], MLP_LDH);
            mlp_dz(c, G.g1, S.dz1, b1, m0, n0);
        }
        mlp_add_tile<NT>(w2, &S.dz2[0][m0], MLP_LDH, &S.h1[0][n0], MLP_LDH);
        __syncthreads();
        // dW1 = dZ1^T X: 16 columns a warp
        mlp_add_tile<2>(w1, &S.dz1[0][m0], MLP_LDH, &S.x[0][16 * (warp >> 2)], MLP_LDX);
        __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) lossSum += __shfl_xor_sync(0xffffffffu, lossSum, o);
    if (lane == 0 && lossSum != 0.0f) atomicAdd(loss, lossSum * coef * 0.5f);
    if (warp == 4 && lane < MLP_OUT) atomicAdd(&grad[MLP_OFF_B3 + lane], b3);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int i = g + 8 * h;
#pragma unroll
        for (int q = 0; q < NT; q++)
            red_add2(&grad[MLP_OFF_W2 + (m0 + i) * MLP_H + n0 + 8 * q + 2 * t], w2[q][2 * h], w2[q][2 * h + 1]);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int n = 16 * (warp >> 2) + 8 * q + 2 * t;
            if (n < MLP_IN) red_add2(&grad[MLP_OFF_W1 + (m0 + i) * MLP_IN + n], w1[q][2 * h], w1[q][2 * h + 1]);
            if (warp < 4 && i < MLP_OUT)
                red_add2(&grad[MLP_OFF_W3 + i * MLP_H + 16 * warp + 8 * q + 2 * t], w3[q][2 * h], w3[q][2 * h + 1]);
        }
    }
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
        for (int e = 0; e < 2; e++)
            for (int o = 4; o < 32; o <<= 1) {   // over the rows g
                b1[q][e] += __shfl_xor_sync(0xffffffffu, b1[q][e], o);
                b2[q][e] += __shfl_xor_sync(0xffffffffu, b2[q][e], o);
            }
    if (g == 0)
#pragma unroll
        for (int q = 0; q < NT; q++) {
            red_add2(&grad[MLP_OFF_B1 + n0 + 8 * q + 2 * t], b1[q][0], b1[q][1]);
            red_add2(&grad[MLP_OFF_B2 + n0 + 8 * q + 2 * t], b2[q][0], b2[q][1]);
        }
}

// Raw features -> raw outputs (y = y' * outScale + outMean) for `count` rows.
__global__ void __launch_bounds__(MLP_THREADS) k_mlp_forward(MlpDev M, const float* X, int count, float* Y) {
    extern __shared__ __align__(16) unsigned char mlpSmem[];
    MlpSmem& S = *reinterpret_cast<MlpSmem*>(mlpSmem);
    mlp_load_weights(S, M);
    for (int first = blockIdx.x * MLP_TILE; first < count; first += gridDim.x * MLP_TILE) {
        const int valid = mlp_load_inputs(S, M, X, nullptr, first, count);
        __syncthreads();
        MlpTiles<MLP_THREADS / 32> G;
        mlp_forward<MLP_THREADS / 32>(S, M, G);
        for (int e = threadIdx.x; e < valid * MLP_OUT; e += blockDim.x) {
            int i = e / MLP_OUT, o = e % MLP_OUT;
            Y[(size_t)(first + i) * MLP_OUT + o] = S.y[i][o] * M.norm[2 * MLP_IN + MLP_OUT + o] + M.norm[2 * MLP_IN + o];
        }
        __syncthreads();
    }
}

// Adam (bias-corrected step sizes a1 = lr / (1 - b1^t), a2 = 1 / (1 - b2^t)); clears the gradient.
__global__ void k_mlp_adam(float* p, float* g, float* m, float* v, float lr1, float bc2, float b1, float b2, float eps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= MLP_NPARAM) return;
    float gi = g[i];
    float mi = b1 * m[i] + (1.0f - b1) * gi;
    float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr1 * mi / (sqrtf(vi * bc2) + eps);
    g[i] = 0.0f;
}

size_t mlp_smem_bytes() { return sizeof(MlpSmem); }

}  // namespace jbg

namespace {

#define MCK(x)                                                                 \
    do {                                                                       \
        cudaError_t e_ = (x);                                                  \
        if (e_ != cudaSuccess) return set_last_error(JBGPU_ERR_CUDA, cudaGetErrorString(e_)); \
    } while (0)

int mlp_repack(jbgpu_mlp* h) {
    k_mlp_pack<<<(MLP_H * MLP_H + 255) / 256, 256, 0, h->s>>>(h->p, h->w1, h->w2, h->w3);
    note_launch();
    MCK(cudaGetLastError());
    return JBGPU_OK;
}

int ensure_io(jbgpu_mlp* h, int n) {
    if (n <= h->ioCap) return JBGPU_OK;
    if (h->io) cudaFree(h->io);
    h->io = nullptr;
    MCK(cudaMalloc(&h->io, sizeof(float) * (size_t)n * (MLP_IN + MLP_OUT)));
    h->ioCap = n;
    return JBGPU_OK;
}

void launch_train_batch(jbgpu_mlp* h, const float* X, const float* T, const int* idx, int first, int count) {
    int tiles = (count + MLP_TILE - 1) / MLP_TILE;
    float coef = 2.0f / (float)(count * MLP_OUT);
    k_mlp_train<<<std::min(tiles, 2 * h->sms), MLP_TRAIN_THREADS, mlp_smem_bytes(), h->s>>>(mlp_view(h), X, T, idx, first, count, coef, h->g, h->loss);
    note_launch();
}

}  // namespace

extern "C" {

int jbgpu_mlp_create(int32_t device, uint64_t seed, jbgpu_mlp** out) {
    if (!out) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "null out");
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return set_last_error(JBGPU_ERR_NO_DEVICE, "no CUDA device");
    if (device < 0 || device >= ndev) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "bad device ordinal");
    MCK(cudaSetDevice(device));
    jbgpu_mlp* h = new jbgpu_mlp();
    h->device = device;
    auto fail = [&](cudaError_t e) {
        jbgpu_mlp_destroy(h);
        return set_last_error(JBGPU_ERR_CUDA, cudaGetErrorString(e));
    };
    cudaError_t e;
    if ((e = cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) return fail(e);
    if ((e = cudaStreamCreateWithFlags(&h->s, cudaStreamNonBlocking)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->p, sizeof(float) * MLP_NPARAM)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->g, sizeof(float) * (MLP_NPARAM + 1))) != cudaSuccess) return fail(e);
    h->loss = h->g + MLP_NPARAM;
    if ((e = cudaMallocHost(&h->hostGrad, sizeof(float) * (MLP_NPARAM + 1))) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->m, sizeof(float) * MLP_NPARAM)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->v, sizeof(float) * MLP_NPARAM)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->norm, sizeof(float) * MLP_NORM)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->w1, sizeof(__nv_bfloat16) * MLP_H * MLP_INP)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->w2, sizeof(__nv_bfloat16) * MLP_H * MLP_H)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&h->w3, sizeof(__nv_bfloat16) * MLP_OUTP * MLP_H)) != cudaSuccess) return fail(e);
    if ((e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_smem_bytes())) != cudaSuccess)
        return fail(e);
    if ((e = cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp_smem_bytes())) != cudaSuccess)
        return fail(e);
    // Xavier-uniform weights from a seeded generator, zero biases, identity normalisation
    std::vector<float> p(MLP_NPARAM, 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int fanOut, int fanIn) {
        float a = std::sqrt(6.0f / (float)(fanIn + fanOut));
        std::uniform_real_distribution<float> U(-a, a);
        for (int i = 0; i < fanOut * fanIn; i++) p[off + i] = U(rng);
    };
    fill(MLP_OFF_W1, MLP_H, MLP_IN);
    fill(MLP_OFF_W2, MLP_H, MLP_H);
    fill(MLP_OFF_W3, MLP_OUT, MLP_H);
    std::vector<float> nrm(MLP_NORM, 0.0f);
    for (int k = 0; k < MLP_IN; k++) nrm[MLP_IN + k] = 1.0f;
    for (int o = 0; o < MLP_OUT; o++) nrm[2 * MLP_IN + MLP_OUT + o] = 1.0f;
    nrm[MLP_NORM_UNIT] = 1.0f;
    if ((e = cudaMemcpy(h->p, p.data(), sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e);
    if ((e = cudaMemcpy(h->norm, nrm.data(), sizeof(float) * MLP_NORM, cudaMemcpyHostToDevice)) != cudaSuccess) return fail(e);
    if ((e = cudaMemset(h->g, 0, sizeof(float) * MLP_NPARAM)) != cudaSuccess) return fail(e);
    if ((e = cudaMemset(h->m, 0, sizeof(float) * MLP_NPARAM)) != cudaSuccess) return fail(e);
    if ((e = cudaMemset(h->v, 0, sizeof(float) * MLP_NPARAM)) != cudaSuccess) return fail(e);
    if (mlp_repack(h) != JBGPU_OK || (e = cudaStreamSynchronize(h->s)) != cudaSuccess) return fail(cudaGetLastError());
    *out = h;
    return JBGPU_OK;
}

int jbgpu_mlp_destroy(jbgpu_mlp* h) {
    if (!h) return JBGPU_OK;
    cudaSetDevice(h->device);
    if (h->s) cudaStreamSynchronize(h->s);
    for (void* q : {(void*)h->p, (void*)h->g, (void*)h->m, (void*)h->v, (void*)h->norm, (void*)h->w1,
                    (void*)h->w2, (void*)h->w3, (void*)h->X, (void*)h->T, (void*)h->idx, (void*)h->io})
        if (q) cudaFree(q);
    if (h->hostGrad) cudaFreeHost(h->hostGrad);
    if (h->s) cudaStreamDestroy(h->s);
    delete h;
    return JBGPU_OK;
}

int jbgpu_mlp_get_params(jbgpu_mlp* h, float* params, float* normalization) {
    if (!h) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "null mlp");
    MCK(cudaSetDevice(h->device));
    MCK(cudaStreamSynchronize(h->s));
    if (params) MCK(cudaMemcpy(params, h->p, sizeof(float) * MLP_NPARAM, cudaMemcpyDeviceToHost));
    if (normalization) MCK(cudaMemcpy(normalization, h->norm, sizeof(float) * MLP_NORM, cudaMemcpyDeviceToHost));
    return JBGPU_OK;
}

int jbgpu_mlp_set_params(jbgpu_mlp* h, const float* params, const float* normalization) {
    if (!h) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "null mlp");
    MCK(cudaSetDevice(h->device));
    MCK(cudaStreamSynchronize(h->s));
    if (normalization) {
        for (int o = 0; o < MLP_OUT; o++)
            if (!(normalization[2 * MLP_IN + MLP_OUT + o] != 0.0f))
                return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "output scale must be non-zero");
        MCK(cudaMemcpy(h->norm, normalization, sizeof(float) * MLP_NORM, cudaMemcpyHostToDevice));
    }
    if (params) {
        MCK(cudaMemcpy(h->p, params, sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice));
        MCK(cudaMemset(h->m, 0, sizeof(float) * MLP_NPARAM));
        MCK(cudaMemset(h->v, 0, sizeof(float) * MLP_NPARAM));
        h->adamStep = 0;
        int rc = mlp_repack(h);
        if (rc) return rc;
    }
    MCK(cudaStreamSynchronize(h->s));
    return JBGPU_OK;
}

int jbgpu_mlp_forward(jbgpu_mlp* h, const float* x, int32_t n, float* y) {
    if (!h || (n > 0 && (!x || !y)) || n < 0) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "bad argument");
    if (n == 0) return JBGPU_OK;
    MCK(cudaSetDevice(h->device));
    int rc = ensure_io(h, n);
    if (rc) return rc;
    float* dx = h->io;
    float* dy = h->io + (size_t)n * MLP_IN;
    MCK(cudaMemcpyAsync(dx, x, sizeof(float) * (size_t)n * MLP_IN, cudaMemcpyHostToDevice, h->s));
    int blocks = std::min((n + MLP_TILE - 1) / MLP_TILE, 1024);
    k_mlp_forward<<<blocks, MLP_THREADS, mlp_smem_bytes(), h->s>>>(mlp_view(h), dx, n, dy);
    note_launch();
    MCK(cudaGetLastError());
    MCK(cudaMemcpyAsync(y, dy, sizeof(float) * (size_t)n * MLP_OUT, cudaMemcpyDeviceToHost, h->s));
    MCK(cudaStreamSynchronize(h->s));
    return JBGPU_OK;
}

int jbgpu_mlp_gradients(jbgpu_mlp* h, const float* x, const float* t, int32_t n, float* grad, float* loss) {
    if (!h || n <= 0 || !x || !t || !grad) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "bad argument");
    MCK(cudaSetDevice(h->device));
    int rc = ensure_io(h, n);
    if (rc) return rc;
    float* dx = h->io;
    float* dt = h->io + (size_t)n * MLP_IN;
    MCK(cudaMemcpyAsync(dx, x, sizeof(float) * (size_t)n * MLP_IN, cudaMemcpyHostToDevice, h->s));
    MCK(cudaMemcpyAsync(dt, t, sizeof(float) * (size_t)n * MLP_OUT, cudaMemcpyHostToDevice, h->s));
    MCK(cudaMemsetAsync(h->g, 0, sizeof(float) * (MLP_NPARAM + 1), h->s));
    launch_train_batch(h, dx, dt, nullptr, 0, n);
    MCK(cudaGetLastError());
    MCK(cudaMemcpyAsync(h->hostGrad, h->g, sizeof(float) * (MLP_NPARAM + 1), cudaMemcpyDeviceToHost, h->s));
    MCK(cudaMemsetAsync(h->g, 0, sizeof(float) * MLP_NPARAM, h->s));
    MCK(cudaStreamSynchronize(h->s));
    std::memcpy(grad, h->hostGrad, sizeof(float) * MLP_NPARAM);
    if (loss) *loss = h->hostGrad[MLP_NPARAM];
    return JBGPU_OK;
}

int jbgpu_mlp_load_samples(jbgpu_mlp* h, const float* x, const float* t, int32_t n) {
    if (!h || n <= 0 || !x || !t) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "bad argument");
    MCK(cudaSetDevice(h->device));
    MCK(cudaStreamSynchronize(h->s));
    if (n > h->cap) {
        for (void* q : {(void*)h->X, (void*)h->T, (void*)h->idx}) if (q) cudaFree(q);
        h->X = h->T = nullptr;
        h->idx = nullptr;
        h->cap = 0;
        MCK(cudaMalloc(&h->X, sizeof(float) * (size_t)n * MLP_IN));
        MCK(cudaMalloc(&h->T, sizeof(float) * (size_t)n * MLP_OUT));
        MCK(cudaMalloc(&h->idx, sizeof(int) * (size_t)n));
        h->cap = n;
    }
    MCK(cudaMemcpy(h->X, x, sizeof(float) * (size_t)n * MLP_IN, cudaMemcpyHostToDevice));
    MCK(cudaMemcpy(h->T, t, sizeof(float) * (size_t)n * MLP_OUT, cudaMemcpyHostToDevice));
    h->n = n;
    return JBGPU_OK;
}

int jbgpu_mlp_train(jbgpu_mlp* h, int32_t epochs, int32_t batch, float lr, uint64_t seed, float* loss_per_epoch) {
    if (!h || epochs <= 0 || batch < MLP_TILE || !(lr > 0.0f)) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "bad argument");
    if (h->n <= 0) return set_last_error(JBGPU_ERR_INVALID_ARGUMENT, "no samples loaded");
    MCK(cudaSetDevice(h->device));
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    std::vector<int> perm(h->n);
    std::mt19937_64 rng(seed);
    for (int ep = 0; ep < epochs; ep++) {
        for (int i = 0; i < h->n; i++) perm[i] = i;
        std::shuffle(perm.begin(), perm.end(), rng);
        MCK(cudaMemcpyAsync(h->idx, perm.data(), sizeof(int) * (size_t)h->n, cudaMemcpyHostToDevice, h->s));
        MCK(cudaMemsetAsync(h->loss, 0, sizeof(float), h->s));
        int batches = 0;
        for (int first = 0; first < h->n; first += batch) {
            int count = std::min(batch, h->n - first);
            launch_train_batch(h, h->X, h->T, h->idx, first, count);
            ++h->adamStep;
            double t = (double)h->adamStep;
            float lr1 = (float)(lr / (1.0 - std::pow((double)b1, t)));
            float bc2 = (float)(1.0 / (1.0 - std::pow((double)b2, t)));
            k_mlp_adam<<<(MLP_NPARAM + 255) / 256, 256, 0, h->s>>>(h->p, h->g, h->m, h->v, lr1, bc2, b1, b2, eps);
            note_launch();
            int rc = mlp_repack(h);
            if (rc) return rc;
            ++batches;
        }
        MCK(cudaGetLastError());
        float l = 0.0f;
        MCK(cudaMemcpyAsync(&l, h->loss, sizeof(float), cudaMemcpyDeviceToHost, h->s));
        MCK(cudaStreamSynchronize(h->s));
        if (loss_per_epoch) loss_per_epoch[ep] = l / (float)batches;
    }
    return JBGPU_OK;
}

}  // extern "C"
