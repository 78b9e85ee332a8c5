// Per-contact MLP of the learned warm start: 24 -> 64 -> 64 -> 3, GELU (tanh form), BF16
// weights and activations into the tensor cores (mma.sync m16n8k16, FP32 accumulate), FP32
// elementwise work.  A block handles 64 samples with 4 warps, a training block with 8; the operands
// of every matrix product are in shared memory and read by ldmatrix, from rows padded so that its
// eight rows fall on all banks.
#pragma once
#include <cuda_bf16.h>
#include "../../include/jbgpu.h"
#include "jbgpu_internal.cuh"

namespace jbg {

constexpr int MLP_IN = 24, MLP_INP = 32;     // inputs, padded to two k-steps
constexpr int MLP_H = 64;
constexpr int MLP_OUT = 3, MLP_OUTP = 16;   // outputs, padded for the transposed products
constexpr int MLP_TILE = 64;                // samples per block
constexpr int MLP_THREADS = 128;
constexpr int MLP_TRAIN_THREADS = 256;
constexpr int MLP_LDX = MLP_INP + 8, MLP_LDH = MLP_H + 8, MLP_LDO = MLP_OUTP + 8;   // padded rows
// parameter packing (FP32 master copy): W1[64][24] b1[64] W2[64][64] b2[64] W3[3][64] b3[3]
constexpr int MLP_OFF_W1 = 0, MLP_OFF_B1 = MLP_OFF_W1 + MLP_H * MLP_IN, MLP_OFF_W2 = MLP_OFF_B1 + MLP_H,
              MLP_OFF_B2 = MLP_OFF_W2 + MLP_H * MLP_H, MLP_OFF_W3 = MLP_OFF_B2 + MLP_H,
              MLP_OFF_B3 = MLP_OFF_W3 + MLP_OUT * MLP_H, MLP_NPARAM = MLP_OFF_B3 + MLP_OUT;
// normalisation block: x' = asinh((x - inMean) * inScale);  y = y' * outScale + outMean; then
// the impulse unit (impulse that stops one step of gravity for unit inverse mass) used by the
// warm-start transform
constexpr int MLP_NORM = 2 * MLP_IN + 2 * MLP_OUT + 1;
constexpr int MLP_NORM_UNIT = 2 * MLP_IN + 2 * MLP_OUT;

JBD float mlp_norm_in(const float* norm, int k, float x) { return asinhf((x - norm[k]) * norm[MLP_IN + k]); }

// The warm-start outputs are relative impulse corrections r, carried by the network as
// asinh(r / MLP_REL) so that the many small corrections and the few large ones both matter.
constexpr float MLP_REL = 0.01f;

struct MlpDev {
    const __nv_bfloat16* w1;   // [64][32] (k >= 24 zero)
    const __nv_bfloat16* w2;   // [64][64]
    const __nv_bfloat16* w3;   // [16][64] (rows >= 3 zero)
    const float* p;            // FP32 parameters (biases read from here)
    const float* norm;         // MLP_NORM floats
};

MlpDev mlp_view(const jbgpu_mlp* h);   // mlp.cu

// Shared-memory working set of one 64-sample block (dy and below: training alone).
struct MlpSmem {
    __nv_bfloat16 x[MLP_TILE][MLP_LDX];
    __nv_bfloat16 h1[MLP_TILE][MLP_LDH];
    __nv_bfloat16 h2[MLP_TILE][MLP_LDH];
    float y[MLP_TILE][4];
    __nv_bfloat16 w1[MLP_H][MLP_LDX];
    __nv_bfloat16 w2[MLP_H][MLP_LDH];
    __nv_bfloat16 w3[MLP_OUTP][MLP_LDH];
    __nv_bfloat16 dy[MLP_TILE][MLP_LDO];
    __nv_bfloat16 dz2[MLP_TILE][MLP_LDH];
    __nv_bfloat16 dz1[MLP_TILE][MLP_LDH];
};

JBD uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

JBD void mma_bf16_16816(float c[4], const uint32_t a[4], const uint32_t b[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Operand fragments of m16n8k16 by ldmatrix (p: the 16 x 16 tile's corner, ld: row length), the
// stored matrix having the product's rows (A) or columns (B) as its rows, or (_t) its k as its rows.
// B: two tiles of 8 columns, r[0], r[1] the first's.
JBD void ldm4(uint32_t r[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
JBD void ldm4_t(uint32_t r[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
JBD void frag_a(uint32_t r[4], const __nv_bfloat16* p, int ld) {
    const int l = threadIdx.x & 31;
    ldm4(r, p + (l & 15) * ld + (l >> 4) * 8);
}
JBD void frag_a_t(uint32_t r[4], const __nv_bfloat16* p, int ld) {
    const int l = threadIdx.x & 31;
    ldm4_t(r, p + ((l >> 4) * 8 + (l & 7)) * ld + ((l >> 3) & 1) * 8);
}
JBD void frag_b(uint32_t r[4], const __nv_bfloat16* p, int ld) {
    const int l = threadIdx.x & 31;
    ldm4(r, p + ((l >> 4) * 8 + (l & 7)) * ld + ((l >> 3) & 1) * 8);
}
JBD void frag_b_t(uint32_t r[4], const __nv_bfloat16* p, int ld) {
    const int l = threadIdx.x & 31;
    ldm4_t(r, p + (((l >> 3) & 1) * 8 + (l & 7)) * ld + (l >> 4) * 8);
}

// One warp: c += A B for 16 rows and NT tiles of 8 columns (NT even), K a multiple of 16.  Lane
// (g = lane / 4, t = lane % 4) holds rows g, g + 8 and columns 2t, 2t + 1 of each tile.  AT / BT: the
// operand is stored with k as its rows; a, b: its corner, rows and columns of k = 0.
template <int NT, int K, bool AT, bool BT>
JBD void warp_gemm(float (*c)[4], const __nv_bfloat16* a, int lda, const __nv_bfloat16* b, int ldb) {
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t fa[4];
        if (AT) frag_a_t(fa, a + k0 * lda, lda);
        else frag_a(fa, a + k0, lda);
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
            uint32_t fb[4];
            if (BT) frag_b_t(fb, b + k0 * ldb + 8 * n, ldb);
            else frag_b(fb, b + 8 * n * ldb + k0, ldb);
            mma_bf16_16816(c[n], fa, fb);
            mma_bf16_16816(c[n + 1], fa, fb + 2);
        }
    }
}

// GELU, tanh form: 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))), and its derivative.
JBD float gelu(float x, float& grad) {
    const float k = 0.7978845608028654f;
    const float u = k * (x + 0.044715f * x * x * x);
    const float th = tanhf(u);
    grad = 0.5f * (1.0f + th) + 0.5f * x * (1.0f - th * th) * k * (1.0f + 3.0f * 0.044715f * x * x);
    return 0.5f * x * (1.0f + th);
}

// Weights into shared memory (all threads of the block).
template <int ROWS, int COLS, int LD>
JBD void mlp_copy_rows(__nv_bfloat16 (*to)[LD], const __nv_bfloat16* from) {   // 16 bytes at a time
    for (int i = threadIdx.x; i < ROWS * COLS / 8; i += blockDim.x)
        *(uint4*)&to[i / (COLS / 8)][8 * (i % (COLS / 8))] = ((const uint4*)from)[i];
}
JBD void mlp_load_weights(MlpSmem& S, const MlpDev& M) {
    mlp_copy_rows<MLP_H, MLP_INP>(S.w1, M.w1);
    mlp_copy_rows<MLP_H, MLP_H>(S.w2, M.w2);
    mlp_copy_rows<MLP_OUTP, MLP_H>(S.w3, M.w3);
}

// Forward pass over S.x (normalised inputs, bf16): S.h1, S.h2, S.y (normalised outputs) and, per
// lane, gelu' of its elements of both layers.  Warp w owns rows 16 (w % 4).. and, of WARPS / 4 column
// groups, group w / 4.  Called after a block barrier, ends with one.
template <int WARPS>
struct MlpTiles {
    static constexpr int GROUPS = WARPS / 4, NT = 8 / GROUPS;
    float g1[NT][4], g2[NT][4];
};
template <int WARPS>
JBD void mlp_layer(float (*grad)[4], const __nv_bfloat16* in, int ldi, const __nv_bfloat16* wt, int ldw, const float* bias,
                   __nv_bfloat16 (*out)[MLP_LDH], bool first) {
    constexpr int NT = MlpTiles<WARPS>::NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * 8 * NT;
    float c[NT][4] = {};
    if (first) warp_gemm<NT, MLP_INP, false, false>(c, in + m0 * ldi, ldi, wt + n0 * ldw, ldw);
    else warp_gemm<NT, MLP_H, false, false>(c, in + m0 * ldi, ldi, wt + n0 * ldw, ldw);
#pragma unroll
    for (int q = 0; q < NT; q++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int n = n0 + 8 * q + 2 * t;
            const float z0 = c[q][2 * h] + bias[n], z1 = c[q][2 * h + 1] + bias[n + 1];
            const float y0 = gelu(z0, grad[q][2 * h]), y1 = gelu(z1, grad[q][2 * h + 1]);
            *(uint32_t*)&out[m0 + g + 8 * h][n] = pack_bf16(__float2bfloat16_rn(y0), __float2bfloat16_rn(y1));
        }
}
template <int WARPS>
JBD void mlp_forward(MlpSmem& S, const MlpDev& M, MlpTiles<WARPS>& T) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    mlp_layer<WARPS>(T.g1, &S.x[0][0], MLP_LDX, &S.w1[0][0], MLP_LDX, M.p + MLP_OFF_B1, S.h1, true);
    __syncthreads();
    mlp_layer<WARPS>(T.g2, &S.h1[0][0], MLP_LDH, &S.w2[0][0], MLP_LDH, M.p + MLP_OFF_B2, S.h2, false);
    __syncthreads();
    if (warp < 4) {
        const int m0 = warp * 16;
        float c[2][4] = {};
        warp_gemm<2, MLP_H, false, false>(c, &S.h2[m0][0], MLP_LDH, &S.w3[0][0], MLP_LDH);
        for (int q = 0; q < 4; q++) {
            int i = m0 + g + (q >> 1) * 8, n = 2 * t + (q & 1);
            if (n < MLP_OUT) S.y[i][n] = c[0][q] + M.p[MLP_OFF_B3 + n];
        }
    }
    __syncthreads();
}

}  // namespace jbg
