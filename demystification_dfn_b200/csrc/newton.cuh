// newton.cuh — training kernels of the MLP initial guess (FP32, hand-written
// forward and backward passes); the solve itself is in newton_core.cuh.
#pragma once
#include "newton_core.cuh"

// ---------------------------------------------------------------------------
// Training kernels (FP32). One CTA of 256 threads takes MLP_SB samples and
// writes its partial gradient of the summed squared error (scaled by
// 1/n_total) and its partial loss; a second kernel adds the partials in a
// fixed order and applies Adam.
//
// The products of a CTA (three 32 x 64 x 64 contractions) come from shared
// memory, so registers hold a tile per thread: 2 samples x 4 units of a layer
// or 4 x 4 entries of W2's gradient, fed by 16-byte reads; W2 is also kept
// transposed for the backward product, and rows are padded to 68 floats so
// that these reads meet no bank twice. Every sum keeps its order (inputs,
// units or samples ascending). A minibatch of 4096: 37 -> 14 us (one
// output per thread and two 4-byte reads per product before, W2's columns
// from one bank).
#define MLP_SB 32
#define MLP_LD (MLP_H + 4)   // padded row of a hidden layer

struct __align__(16) MlpSmem {
    float W[MLP_NPAR + 3];            // flat weights (W2 rows are 16-byte aligned)
    float W2t[MLP_H][MLP_LD];
    float H1[MLP_SB][MLP_LD], H2[MLP_SB][MLP_LD];
    float D1[MLP_SB][MLP_LD], D2[MLP_SB][MLP_LD];
    float X[MLP_SB][MLP_IN + 1];
    float dout[MLP_SB];
    float lsum[MLP_SB];
};
static_assert(MLP_W2 % 4 == 0 && MLP_W3 % 4 == 0, "16-byte reads of W2 and W3");

__device__ __forceinline__ float mlp_at(const float4 &v, int c)
{
    return c == 0 ? v.x : (c == 1 ? v.y : (c == 2 ? v.z : v.w));
}

__global__ void __launch_bounds__(256) mlp_grad_kernel(const float *__restrict__ X, const float *__restrict__ T,
                                                       int64_t n, int64_t n_total, const float *W,
                                                       float *__restrict__ gpart, float *__restrict__ lpart)
{
    extern __shared__ __align__(16) unsigned char mlp_smem_raw[];
    MlpSmem &S = *reinterpret_cast<MlpSmem *>(mlp_smem_raw);
    const int tid = threadIdx.x;
    const int64_t s0 = (int64_t)blockIdx.x * MLP_SB;
    const int u = 4 * (tid & 15), sp = 2 * (tid >> 4);   // this thread's 4 units and 2 samples
    for (int q = tid; q < MLP_SB * MLP_IN; q += blockDim.x) {
        const int s = q / MLP_IN, i = q % MLP_IN;
        S.X[s][i] = (s0 + s < n) ? X[(s0 + s) * MLP_IN + i] : 0.0f;
    }
    const float target = (tid < MLP_SB && s0 + tid < n) ? T[s0 + tid] : 0.0f;
    pdl_wait();   // the previous minibatch's update of W
    pdl_trigger();
    for (int p = tid; p < MLP_NPAR; p += blockDim.x) {
        const float w = W[p];
        S.W[p] = w;
        const int q = p - MLP_W2;
        if (q >= 0 && q < MLP_H * MLP_H) S.W2t[q % MLP_H][q / MLP_H] = w;
    }
    __syncthreads();
    float z1[2][4], z2[2][4];   // pre-activations of the tile
    // layer 1
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            float z = S.W[MLP_B1 + u + c];
#pragma unroll
            for (int i = 0; i < MLP_IN; i++) z = fmaf(S.X[sp + a][i], S.W[MLP_W1 + i * MLP_H + u + c], z);
            z1[a][c] = z;
            S.H1[sp + a][u + c] = silu_f(z);
        }
    __syncthreads();
    // layer 2
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) z2[a][c] = S.W[MLP_B2 + u + c];
#pragma unroll 4
    for (int i = 0; i < MLP_H; i += 4) {
        const float4 h0 = *reinterpret_cast<const float4 *>(&S.H1[sp][i]);
        const float4 h1 = *reinterpret_cast<const float4 *>(&S.H1[sp + 1][i]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4 w = *reinterpret_cast<const float4 *>(&S.W[MLP_W2 + (i + k) * MLP_H + u]);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                z2[0][c] = fmaf(mlp_at(h0, k), mlp_at(w, c), z2[0][c]);
                z2[1][c] = fmaf(mlp_at(h1, k), mlp_at(w, c), z2[1][c]);
            }
        }
    }
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) S.H2[sp + a][u + c] = silu_f(z2[a][c]);
    __syncthreads();
    // output, loss and its derivative (mean over n_total samples)
    if (tid < MLP_SB) {
        const int s = tid;
        float o = S.W[MLP_B3];
#pragma unroll 4
        for (int j = 0; j < MLP_H; j += 4) {
            const float4 h = *reinterpret_cast<const float4 *>(&S.H2[s][j]);
            const float4 w = *reinterpret_cast<const float4 *>(&S.W[MLP_W3 + j]);
#pragma unroll
            for (int c = 0; c < 4; c++) o = fmaf(mlp_at(h, c), mlp_at(w, c), o);
        }
        const bool valid = s0 + s < n;
        const float d = valid ? o - target : 0.0f;
        S.lsum[s] = d * d;
        S.dout[s] = 2.0f * d / (float)n_total;
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) S.D2[sp + a][u + c] = S.dout[sp + a] * S.W[MLP_W3 + u + c] * dsilu_f(z2[a][c]);
    __syncthreads();
    {
        float g[2][4] = {};
#pragma unroll 4
        for (int j = 0; j < MLP_H; j += 4) {
            const float4 d0 = *reinterpret_cast<const float4 *>(&S.D2[sp][j]);
            const float4 d1 = *reinterpret_cast<const float4 *>(&S.D2[sp + 1][j]);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 w = *reinterpret_cast<const float4 *>(&S.W2t[j + k][u]);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    g[0][c] = fmaf(mlp_at(d0, k), mlp_at(w, c), g[0][c]);
                    g[1][c] = fmaf(mlp_at(d1, k), mlp_at(w, c), g[1][c]);
                }
            }
        }
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int c = 0; c < 4; c++) S.D1[sp + a][u + c] = g[a][c] * dsilu_f(z1[a][c]);
    }
    __syncthreads();
    float *gp = gpart + (int64_t)blockIdx.x * MLP_NPAR;
    {
        // W2[i0 .. i0 + 3][j0 .. j0 + 3]
        const int i0 = 4 * (tid >> 4), j0 = u;
        float g[4][4] = {};
#pragma unroll 4
        for (int s = 0; s < MLP_SB; s++) {
            const float4 h = *reinterpret_cast<const float4 *>(&S.H1[s][i0]);
            const float4 d = *reinterpret_cast<const float4 *>(&S.D2[s][j0]);
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int c = 0; c < 4; c++) g[a][c] = fmaf(mlp_at(h, a), mlp_at(d, c), g[a][c]);
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int c = 0; c < 4; c++) gp[MLP_W2 + (i0 + a) * MLP_H + j0 + c] = g[a][c];
    }
    for (int q = tid; q < MLP_NPAR - MLP_H * MLP_H; q += blockDim.x) {
        const int p = q < MLP_W2 ? q : q + MLP_H * MLP_H;   // the other parameters
        float g = 0.0f;
        if (p < MLP_B1) {                        // W1[i][j]
            const int i = p / MLP_H, j = p % MLP_H;
            for (int s = 0; s < MLP_SB; s++) g = fmaf(S.X[s][i], S.D1[s][j], g);
        } else if (p < MLP_W2) {                 // b1[j]
            const int j = p - MLP_B1;
            for (int s = 0; s < MLP_SB; s++) g += S.D1[s][j];
        } else if (p < MLP_W3) {                 // b2[j]
            const int j = p - MLP_B2;
            for (int s = 0; s < MLP_SB; s++) g += S.D2[s][j];
        } else if (p < MLP_B3) {                 // W3[j]
            const int j = p - MLP_W3;
            for (int s = 0; s < MLP_SB; s++) g = fmaf(S.H2[s][j], S.dout[s], g);
        } else {                                 // b3
            for (int s = 0; s < MLP_SB; s++) g += S.dout[s];
        }
        gp[p] = g;
    }
    if (tid == 0) {
        float l = 0.0f;
        for (int s = 0; s < MLP_SB; s++) l += S.lsum[s];
        lpart[blockIdx.x] = l;
    }
}

// The FP16 tensor-core image of the FP32 weights (one block).
__global__ void mlp_image_kernel(const float *__restrict__ W, MlpTC *img) { mlp_tc_stage(*img, W); }

// Inference of n rows by the friction kernel's tensor-core path; every lane
// of every warp takes part (rows past n are zero inputs, not stored).
__global__ void __launch_bounds__(256) mlp_infer_kernel(const float *__restrict__ X, int64_t n,
                                                        const float *__restrict__ W, float *__restrict__ Y)
{
    extern __shared__ __align__(16) unsigned char infer_smem[];
    MlpTC &S = *reinterpret_cast<MlpTC *>(infer_smem);
    mlp_tc_stage(S, W);
    __syncthreads();
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    float x[MLP_IN];
#pragma unroll
    for (int i = 0; i < MLP_IN; i++) x[i] = (r < n) ? X[r * MLP_IN + i] : 0.0f;
    const float y = mlp_warp_tc(S, x);
    if (r < n) Y[r] = y;
}

// n partials `stride` apart, added in order; sixteen loads in flight.
__device__ __forceinline__ float mlp_sum_partials(const float *p, int n, int64_t stride)
{
    float s = 0.0f;
    int b = 0;
    for (; b + 16 <= n; b += 16) {
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = p[(b + q) * stride];
#pragma unroll
        for (int q = 0; q < 16; q++) s += v[q];
    }
    for (; b < n; b++) s += p[b * stride];
    return s;
}

// Sum of the block partials (fixed order); with lr > 0 also one Adam step.
// The thread after the parameters adds up the losses.
__global__ void __launch_bounds__(128) mlp_reduce_adam_kernel(const float *gpart, const float *lpart, int nblk, float *W,
                                                              float *m, float *v, float *gout, float *loss, int step,
                                                              float lr)
{
    pdl_wait();
    pdl_trigger();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > MLP_NPAR) return;
    if (p == MLP_NPAR) {
        *loss = mlp_sum_partials(lpart, nblk, 1);
        return;
    }
    const float g = mlp_sum_partials(gpart + p, nblk, MLP_NPAR);
    if (gout) gout[p] = g;
    if (lr > 0.0f) {
        const float b1 = 0.9f, b2 = 0.999f, epsa = 1e-8f;
        const float mm = b1 * m[p] + (1.0f - b1) * g;
        const float vv = b2 * v[p] + (1.0f - b2) * g * g;
        m[p] = mm;
        v[p] = vv;
        const float mh = mm / (1.0f - powf(b1, (float)step)), vh = vv / (1.0f - powf(b2, (float)step));
        W[p] -= lr * mh / (sqrtf(vh) + epsa);
    }
}
