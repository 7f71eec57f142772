// Learned subgrid closure (no reference counterpart; Smagorinsky, m_les.f90:1142-1215,
// is the fallback and the baseline).
//
// Per point, from the filtered velocity gradient A_ij = d ubar_i / dx_j:
//   S = (A + A^T)/2, R = (A - A^T)/2, |S| = sqrt(2 S:S), s = S/|S|, r = R/|S|
//   inputs  x = [tr(s^2), tr(r^2), tr(s^3), tr(s r^2), tr(s^2 r^2), Delta / (2 pi / 32)]
//   basis   T1 = s, T2 = s r - r s, T3 = s^2 - tr(s^2) I/3, T4 = r^2 - tr(r^2) I/3,
//           T5 = r s^2 - s^2 r
//   stress  tau = Delta^2 |S|^2 sum_n g_n(x) T_n   (deviatoric)
// g = MLP(x): 6 -> 64 -> 64 -> 64 -> 5 with GELU; the weights are stored as bf16
// and every product is accumulated in fp32.  Smagorinsky is g = (-2 Cs^2, 0, 0, 0, 0).
//
// Inference on the CUDA cores runs one thread per point: the weights sit in
// shared memory (fp32 values of the bf16 weights), the running layer's 64
// accumulators in registers, and the previous layer's activations in a
// per-thread column of shared memory, so that no register array is indexed by a
// loop variable.  Training (k_mlp_grad) takes 64 points per CTA as block products.
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

constexpr int MLP_IN = 6, MLP_H = 64, MLP_OUT = 5, MLP_NB = 5, MLP_TC = 6;
// flat parameter layout (floats): W_l is [out][in] row-major, then b_l
constexpr int MLP_W1 = 0, MLP_B1 = MLP_W1 + MLP_H * MLP_IN, MLP_W2 = MLP_B1 + MLP_H, MLP_B2 = MLP_W2 + MLP_H * MLP_H,
              MLP_W3 = MLP_B2 + MLP_H, MLP_B3 = MLP_W3 + MLP_H * MLP_H, MLP_W4 = MLP_B3 + MLP_H,
              MLP_B4 = MLP_W4 + MLP_OUT * MLP_H, MLP_NPARAM = MLP_B4 + MLP_OUT;
constexpr int MLP_NT = 128;                                               // threads per block
constexpr int MLP_WPAD = (MLP_NPARAM + 3) / 4 * 4;                        // weights in shared memory
constexpr size_t MLP_SMEM = sizeof(float) * (MLP_WPAD + MLP_H * MLP_NT);  // + activation columns
static_assert(MLP_W2 % 4 == 0 && MLP_W3 % 4 == 0, "float4 rows");

// GELU in its tanh form (Hendrycks and Gimpel, "Gaussian Error Linear Units",
// 2016): gelu(z) = z/2 (1 + tanh(a (z + b z^3))), a = sqrt(2/pi), b = 0.044715;
// the activation of the network, in training and inference
constexpr float GELU_A = 0.79788456080286535588f, GELU_B = 0.044715f;
H3D_D float gelu(float z)
{
    const float u = GELU_A * (z + GELU_B * (z * z * z));
    return 0.5f * z * (1.0f + tanhf(u));
}
// the same with the hardware tanh approximation (tanh.approx.f32, one special
// function unit instruction), for the tensor-core inference kernel, whose
// activations are rounded to bf16 afterwards anyway
H3D_D float gelu_fast(float z)
{
    const float u = GELU_A * z * fmaf(GELU_B, z * z, 1.0f);
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(u));
    const float h = 0.5f * z;
    return fmaf(h, t, h);
}

struct Feat {
    float x[MLP_IN];
    float T[MLP_NB][MLP_TC];  // symmetric 3x3 as (11, 12, 13, 22, 23, 33)
    float sbar[MLP_TC];       // unnormalised strain rate
    float pref;               // Delta^2 |S|^2
};
// Frobenius weights of the (11, 12, 13, 22, 23, 33) storage
H3D_HD float frob_w(int c) { return (c == 1 || c == 2 || c == 4) ? 2.0f : 1.0f; }

H3D_D void mat_mul3(const float a[3][3], const float b[3][3], float c[3][3])
{
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) c[i][j] = a[i][0] * b[0][j] + a[i][1] * b[1][j] + a[i][2] * b[2][j];
}

H3D_D void features(const float A[3][3], float delta, Feat &f)
{
    float S[3][3], R[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            S[i][j] = 0.5f * (A[i][j] + A[j][i]);
            R[i][j] = 0.5f * (A[i][j] - A[j][i]);
        }
    const int ii[6] = {0, 0, 0, 1, 1, 2}, jj[6] = {0, 1, 2, 1, 2, 2};
    float ss = 0.f;
#pragma unroll
    for (int q = 0; q < 6; q++) {
        f.sbar[q] = S[ii[q]][jj[q]];
        ss += frob_w(q) * f.sbar[q] * f.sbar[q];
    }
    const float smag = sqrtf(2.0f * ss) + 1e-30f;
    const float inv = 1.0f / smag;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) { S[i][j] *= inv; R[i][j] *= inv; }
    float s2[3][3], r2[3][3], s3[3][3], sr[3][3], rs[3][3], sr2[3][3], s2r2[3][3], rs2[3][3], s2r[3][3];
    mat_mul3(S, S, s2);
    mat_mul3(R, R, r2);
    mat_mul3(s2, S, s3);
    mat_mul3(S, R, sr);
    mat_mul3(R, S, rs);
    mat_mul3(S, r2, sr2);
    mat_mul3(s2, r2, s2r2);
    mat_mul3(R, s2, rs2);
    mat_mul3(s2, R, s2r);
    const float ts2 = s2[0][0] + s2[1][1] + s2[2][2], tr2 = r2[0][0] + r2[1][1] + r2[2][2];
    f.x[0] = ts2;
    f.x[1] = tr2;
    f.x[2] = s3[0][0] + s3[1][1] + s3[2][2];
    f.x[3] = sr2[0][0] + sr2[1][1] + sr2[2][2];
    f.x[4] = s2r2[0][0] + s2r2[1][1] + s2r2[2][2];
    f.x[5] = delta * (32.0f / 6.283185307179586f);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const int i = ii[q], j = jj[q];
        const float d = (i == j) ? 1.0f : 0.0f;
        f.T[0][q] = S[i][j];
        f.T[1][q] = sr[i][j] - rs[i][j];
        f.T[2][q] = s2[i][j] - d * ts2 * (1.0f / 3.0f);
        f.T[3][q] = r2[i][j] - d * tr2 * (1.0f / 3.0f);
        f.T[4][q] = rs2[i][j] - s2r[i][j];
    }
    f.pref = delta * delta * smag * smag;
}

// weights into shared memory as fp32, each W_l as [in][out]
H3D_D int param_slot(int q)
{
    int off = -1, nin = 0, nout = 0;
    if (q < MLP_B1) { off = MLP_W1; nin = MLP_IN; nout = MLP_H; }
    else if (q >= MLP_W2 && q < MLP_B2) { off = MLP_W2; nin = MLP_H; nout = MLP_H; }
    else if (q >= MLP_W3 && q < MLP_B3) { off = MLP_W3; nin = MLP_H; nout = MLP_H; }
    else if (q >= MLP_W4 && q < MLP_B4) { off = MLP_W4; nin = MLP_H; nout = MLP_OUT; }
    if (off < 0) return q;
    const int j = (q - off) / nin, i = (q - off) % nin;
    return off + i * nout + j;
}
// wb must be 16-byte aligned (eight bf16 per load)
H3D_D void load_params(const __nv_bfloat16 *__restrict__ wb, float *sw)
{
    constexpr int NV = MLP_NPARAM / 8;
    for (int k = threadIdx.x; k < NV; k += blockDim.x) {
        const uint4 v = reinterpret_cast<const uint4 *>(wb)[k];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            sw[param_slot(8 * k + 2 * e)] = __uint_as_float(u[e] << 16);
            sw[param_slot(8 * k + 2 * e + 1)] = __uint_as_float(u[e] & 0xffff0000u);
        }
    }
    for (int q = 8 * NV + threadIdx.x; q < MLP_NPARAM; q += blockDim.x) sw[param_slot(q)] = __bfloat162float(wb[q]);
    __syncthreads();
}

// acc[j] = b[j] + sum_i Wt[i][j] act[i], act a column of stride MLP_NT
template <int NIN, int NOUT>
H3D_D void dense_col(const float *__restrict__ Wt, const float *__restrict__ b, const float *act, float acc[NOUT])
{
#pragma unroll
    for (int j = 0; j < NOUT; j++) acc[j] = b ? b[j] : 0.0f;
#pragma unroll 2
    for (int i = 0; i < NIN; i++) {
        const float ai = act[i * MLP_NT];
        if constexpr (NOUT % 4 == 0) {
            const float4 *w4 = reinterpret_cast<const float4 *>(Wt + i * NOUT);
#pragma unroll
            for (int q = 0; q < NOUT / 4; q++) {
                const float4 w = w4[q];
                acc[4 * q] = fmaf(w.x, ai, acc[4 * q]);
                acc[4 * q + 1] = fmaf(w.y, ai, acc[4 * q + 1]);
                acc[4 * q + 2] = fmaf(w.z, ai, acc[4 * q + 2]);
                acc[4 * q + 3] = fmaf(w.w, ai, acc[4 * q + 3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < NOUT; j++) acc[j] = fmaf(Wt[i * NOUT + j], ai, acc[j]);
        }
    }
}

// forward pass of one point; sw holds the transposed weights, act is this
// thread's activation column
H3D_D void mlp_forward(const float *__restrict__ sw, float *act, const float x[MLP_IN], float g[MLP_OUT])
{
    float acc[MLP_H];
#pragma unroll
    for (int j = 0; j < MLP_H; j++) {
        float s = sw[MLP_B1 + j];
#pragma unroll
        for (int i = 0; i < MLP_IN; i++) s = fmaf(sw[MLP_W1 + i * MLP_H + j], x[i], s);
        acc[j] = s;
    }
#pragma unroll
    for (int l = 0; l < 2; l++) {
#pragma unroll
        for (int j = 0; j < MLP_H; j++) act[j * MLP_NT] = gelu(acc[j]);
        dense_col<MLP_H, MLP_H>(sw + (l == 0 ? MLP_W2 : MLP_W3), sw + (l == 0 ? MLP_B2 : MLP_B3), act, acc);
    }
#pragma unroll
    for (int j = 0; j < MLP_H; j++) act[j * MLP_NT] = gelu(acc[j]);
    dense_col<MLP_H, MLP_OUT>(sw + MLP_W4, sw + MLP_B4, act, g);
}

H3D_D void basis_sum(const Feat &f, const float g[MLP_OUT], float tau[MLP_TC])
{
#pragma unroll
    for (int c = 0; c < MLP_TC; c++) {
        float t = 0.f;
#pragma unroll
        for (int n = 0; n < MLP_NB; n++) t = fmaf(g[n], f.T[n][c], t);
        tau[c] = f.pref * t;
    }
}
// subgrid dissipation -tau : S
H3D_D float sgs_diss(const float tau[MLP_TC], const float sbar[MLP_TC])
{
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < MLP_TC; c++) s = fmaf(frob_w(c) * tau[c], sbar[c], s);
    return -s;
}

struct MlpBatch {
    int64_t np;          // points in this minibatch
    const int32_t *idx;  // indices into the dataset
    const float *A;      // dataset gradients [9][P]
    const float *tau;    // dataset deviatoric stresses [6][P]
    int64_t P;
    float delta;         // filter width
    float inv_norm;      // 1 / mean |tau|_F^2 over the dataset
    float inv_norm_p;    // 1 / mean (tau:S)^2 over the dataset
    float lam;           // weight of the dissipation term
    float *part;         // [chunk][MLP_NPARAM + 1]: a chunk's gradient, then its loss
};

// Loss and gradient of a chunk of WG_C points per CTA, forward and backward in
// one kernel:
//   L = inv_norm/np sum_p |tau_pred - tau|_F^2 + lam inv_norm_p/np sum_p (Pi_pred - Pi)^2
// with Pi = -tau : S the subgrid dissipation.  Every 64 x 64 x 64 product
// (two layers forward, two backward, two weight gradients) is a block product
// of 256 threads with a 4 x 4 tile each: eight 16-byte shared-memory loads feed
// 64 multiply-adds.  A thread owns the same (neuron, point) tile in every layer,
// so the slopes gelu'(z) wait in its registers; activations stay in shared
// memory and the deltas take their place, so that nothing but the chunk's
// gradient leaves the SM.  94 KB and 128 registers: two CTAs per SM, the 256
// chunks of a 16384-point minibatch in one wave.  A thread per point, with
// pre-activations and deltas through HBM in three kernels, had one warp per
// scheduler to hide the multiply-add latency: 67 + 113 + 64 us of device time
// for 16384 points, against 40 here (0.88 GFLOP; the FP32 rate's floor is 12).
constexpr int WG_C = 64, WG_P = WG_C + 4;  // points per chunk, row pitch (conflict-free 16-byte rows)
constexpr int GS_W2 = 0, GS_W3 = GS_W2 + MLP_H * WG_P, GS_A = GS_W3 + MLP_H * WG_P, GS_X = GS_A + 3 * MLP_H * WG_P,
              GS_D4 = GS_X + MLP_IN * WG_P, GS_W1 = GS_D4 + MLP_OUT * WG_P, GS_T = GS_W1 + MLP_W2, GS_B2 = GS_T + 400,
              GS_END = GS_B2 + MLP_H;  // GS_W1: W1 b1;  GS_T: b3 W4 b4
constexpr size_t GS_SMEM = sizeof(float) * GS_END;
static_assert(MLP_NPARAM - MLP_B3 <= 400 && MLP_W2 % 8 == 0 && MLP_B2 % 8 == 0 && MLP_W3 % 8 == 0 && MLP_B3 % 8 == 0, "layout");

// shared-memory slot of parameter q (eight consecutive ones from a multiple of 8
// share a row)
H3D_D int grad_slot(int q)
{
    if (q < MLP_W2) return GS_W1 + q;
    if (q < MLP_B2) return GS_W2 + ((q - MLP_W2) >> 6) * WG_P + ((q - MLP_W2) & 63);
    if (q < MLP_W3) return GS_B2 + q - MLP_B2;
    if (q < MLP_B3) return GS_W3 + ((q - MLP_W3) >> 6) * WG_P + ((q - MLP_W3) & 63);
    return GS_T + q - MLP_B3;
}
// acc[r][e] += sum_k X[xr + 16 r][k] Y[yr + 16 e][k]
H3D_D void tile_rows(const float *__restrict__ X, const float *__restrict__ Y, int xr, int yr, float (&acc)[4][4])
{
#pragma unroll 4
    for (int k = 0; k < WG_C; k += 4) {
        float4 x[4], y[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            x[r] = *reinterpret_cast<const float4 *>(X + (xr + 16 * r) * WG_P + k);
            y[r] = *reinterpret_cast<const float4 *>(Y + (yr + 16 * r) * WG_P + k);
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                acc[r][e] = fmaf(x[r].x, y[e].x, acc[r][e]);
                acc[r][e] = fmaf(x[r].y, y[e].y, acc[r][e]);
                acc[r][e] = fmaf(x[r].z, y[e].z, acc[r][e]);
                acc[r][e] = fmaf(x[r].w, y[e].w, acc[r][e]);
            }
    }
}
H3D_D float row_sum(const float *__restrict__ r)
{
    float s = 0.f;
#pragma unroll 4
    for (int q = 0; q < WG_C; q += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(r + q);
        s += v.x; s += v.y; s += v.z; s += v.w;
    }
    return s;
}
H3D_D float row_dot(const float *__restrict__ u, const float *__restrict__ v)
{
    float s = 0.f;
#pragma unroll 4
    for (int q = 0; q < WG_C; q += 4) {
        const float4 a = *reinterpret_cast<const float4 *>(u + q), c = *reinterpret_cast<const float4 *>(v + q);
        s = fmaf(a.x, c.x, s); s = fmaf(a.y, c.y, s); s = fmaf(a.z, c.z, s); s = fmaf(a.w, c.w, s);
    }
    return s;
}

static __global__ void __launch_bounds__(256, 2) k_mlp_grad(const MlpBatch b, const __nv_bfloat16 *__restrict__ wb)
{
    extern __shared__ __align__(16) float sm[];
    __shared__ float red[2];
    const int tid = threadIdx.x, tj = tid & 15, tp = tid >> 4;
    constexpr int NV = MLP_NPARAM / 8;
    for (int k = tid; k < NV; k += 256) {
        const uint4 v = reinterpret_cast<const uint4 *>(wb)[k];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        float *d = sm + grad_slot(8 * k);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            d[2 * e] = __uint_as_float(u[e] << 16);
            d[2 * e + 1] = __uint_as_float(u[e] & 0xffff0000u);
        }
    }
    for (int q = 8 * NV + tid; q < MLP_NPARAM; q += 256) sm[grad_slot(q)] = __bfloat162float(wb[q]);
    const int64_t p = blockIdx.x * (int64_t)WG_C + tid;  // the point of threads 0..63
    const bool live = tid < WG_C && p < b.np;
    const int64_t at = live ? b.idx[p] : 0;
    auto point = [&](Feat &f) {
        float Am[3][3];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) Am[i][j] = b.A[(3 * i + j) * b.P + at];
        features(Am, b.delta, f);
    };
    if (tid < WG_C) {
        Feat f;
        if (live) point(f);
#pragma unroll
        for (int i = 0; i < MLP_IN; i++) sm[GS_X + i * WG_P + tid] = live ? f.x[i] : 0.f;
    }
    __syncthreads();
    float *const A1 = sm + GS_A, *const A2 = A1 + MLP_H * WG_P, *const A3 = A2 + MLP_H * WG_P;
    const float *const W4 = sm + GS_T + MLP_H, *const b4 = W4 + MLP_OUT * MLP_H;
    float sl[3][4][4];  // gelu'(z) of neurons tj + 16 r, points 4 tp + e
    auto activate = [&](const float (&z)[4][4], float (&d)[4][4], float *A) {
#pragma unroll
        for (int r = 0; r < 4; r++) {
            float4 v;
            float *o = &v.x;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                // gelu and its derivative with one tanh
                const float zz = z[r][e], u = GELU_A * (zz + GELU_B * (zz * zz * zz)), t = tanhf(u);
                o[e] = 0.5f * zz * (1.0f + t);
                d[r][e] = 0.5f * (1.0f + t) + 0.5f * zz * (1.0f - t * t) * GELU_A * (1.0f + 3.0f * GELU_B * (zz * zz));
            }
            *reinterpret_cast<float4 *>(A + (tj + 16 * r) * WG_P + 4 * tp) = v;
        }
    };
    {
        float z[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 4; e++) z[r][e] = sm[GS_W1 + MLP_B1 + tj + 16 * r];
#pragma unroll
        for (int i = 0; i < MLP_IN; i++) {
            const float4 x = *reinterpret_cast<const float4 *>(sm + GS_X + i * WG_P + 4 * tp);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float w = sm[GS_W1 + (tj + 16 * r) * MLP_IN + i];
                z[r][0] = fmaf(w, x.x, z[r][0]);
                z[r][1] = fmaf(w, x.y, z[r][1]);
                z[r][2] = fmaf(w, x.z, z[r][2]);
                z[r][3] = fmaf(w, x.w, z[r][3]);
            }
        }
        activate(z, sl[0], A1);
    }
    __syncthreads();
#pragma unroll
    for (int l = 1; l < 3; l++) {
        const float *W = sm + (l == 1 ? GS_W2 : GS_W3), *bias = l == 1 ? sm + GS_B2 : sm + GS_T, *A = l == 1 ? A1 : A2;
        float z[4][4];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int e = 0; e < 4; e++) z[r][e] = bias[tj + 16 * r];
#pragma unroll 4
        for (int k = 0; k < MLP_H; k += 4) {
            float4 w[4], x[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                w[r] = *reinterpret_cast<const float4 *>(W + (tj + 16 * r) * WG_P + k);
                x[r] = *reinterpret_cast<const float4 *>(A + (k + r) * WG_P + 4 * tp);
            }
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const float wv = kk == 0 ? w[r].x : kk == 1 ? w[r].y : kk == 2 ? w[r].z : w[r].w;
                    z[r][0] = fmaf(wv, x[kk].x, z[r][0]);
                    z[r][1] = fmaf(wv, x[kk].y, z[r][1]);
                    z[r][2] = fmaf(wv, x[kk].z, z[r][2]);
                    z[r][3] = fmaf(wv, x[kk].w, z[r][3]);
                }
        }
        activate(z, sl[l], l == 1 ? A2 : A3);
        __syncthreads();
    }
    // output layer: g[o][point] into the d4 rows, then the loss and dL/dg in place
    for (int o = tid >> 6; o < MLP_OUT; o += 4) {
        const int q = tid & 63;
        float g = b4[o];
#pragma unroll 8
        for (int k = 0; k < MLP_H; k++) g = fmaf(W4[o * MLP_H + k], A3[k * WG_P + q], g);
        sm[GS_D4 + o * WG_P + q] = g;
    }
    __syncthreads();
    if (tid < WG_C) {
        float lsum = 0.f, d4[MLP_OUT] = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (live) {
            Feat f;
            point(f);
            float g[MLP_OUT], tpr[MLP_TC], tt[MLP_TC], e[MLP_TC];
#pragma unroll
            for (int o = 0; o < MLP_OUT; o++) g[o] = sm[GS_D4 + o * WG_P + tid];
            basis_sum(f, g, tpr);
#pragma unroll
            for (int c = 0; c < MLP_TC; c++) {
                tt[c] = b.tau[c * b.P + at];
                e[c] = tpr[c] - tt[c];
            }
            float lt = 0.f;
#pragma unroll
            for (int c = 0; c < MLP_TC; c++) lt = fmaf(frob_w(c) * e[c], e[c], lt);
            const float ep = sgs_diss(tpr, f.sbar) - sgs_diss(tt, f.sbar);
            const float inp = 1.0f / (float)b.np;
            lsum = (b.inv_norm * lt + b.lam * b.inv_norm_p * ep * ep) * inp;
            const float st = 2.0f * b.inv_norm * inp * f.pref, sp = -2.0f * b.lam * b.inv_norm_p * inp * ep * f.pref;
#pragma unroll
            for (int n = 0; n < MLP_NB; n++) {
                float a1 = 0.f, a2 = 0.f;
#pragma unroll
                for (int c = 0; c < MLP_TC; c++) {
                    a1 = fmaf(frob_w(c) * e[c], f.T[n][c], a1);
                    a2 = fmaf(frob_w(c) * f.sbar[c], f.T[n][c], a2);
                }
                d4[n] = st * a1 + sp * a2;
            }
        }
#pragma unroll
        for (int o = 0; o < MLP_OUT; o++) sm[GS_D4 + o * WG_P + tid] = d4[o];
        for (int off = 16; off > 0; off >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
        if ((tid & 31) == 0) red[tid >> 5] = lsum;
    }
    __syncthreads();
    float *const out = b.part + (int64_t)blockIdx.x * (MLP_NPARAM + 1);
    if (tid == 0) out[MLP_NPARAM] = red[0] + red[1];
    for (int q = tid; q < MLP_OUT * (MLP_H + 1); q += 256) {
        const int o = q / (MLP_H + 1), i = q - o * (MLP_H + 1);
        const float *d = sm + GS_D4 + o * WG_P;
        if (i < MLP_H) out[MLP_W4 + o * MLP_H + i] = row_dot(d, A3 + i * WG_P);
        else out[MLP_B4 + o] = row_sum(d);
    }
    // d_l[j][point] of this thread's tile: backward through layer l + 1, times the slope
    float d[4][4];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int e = 0; e < 4; e++) d[r][e] = 0.f;
#pragma unroll
    for (int o = 0; o < MLP_OUT; o++) {
        const float4 x = *reinterpret_cast<const float4 *>(sm + GS_D4 + o * WG_P + 4 * tp);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float w = W4[o * MLP_H + tj + 16 * r];
            d[r][0] = fmaf(w, x.x, d[r][0]);
            d[r][1] = fmaf(w, x.y, d[r][1]);
            d[r][2] = fmaf(w, x.z, d[r][2]);
            d[r][3] = fmaf(w, x.w, d[r][3]);
        }
    }
#pragma unroll
    for (int l = 2; l >= 0; l--) {
        __syncthreads();  // A3 (the activations, then the previous layer's deltas) is read
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float4 v = make_float4(d[r][0] * sl[l][r][0], d[r][1] * sl[l][r][1], d[r][2] * sl[l][r][2],
                                         d[r][3] * sl[l][r][3]);
            *reinterpret_cast<float4 *>(A3 + (tj + 16 * r) * WG_P + 4 * tp) = v;
        }
        __syncthreads();
        if (tid < MLP_H) out[(l == 0 ? MLP_B1 : l == 1 ? MLP_B2 : MLP_B3) + tid] = row_sum(A3 + tid * WG_P);
        if (l == 0) {
            for (int q = tid; q < MLP_H * MLP_IN; q += 256)
                out[MLP_W1 + q] = row_dot(A3 + (q / MLP_IN) * WG_P, sm + GS_X + (q % MLP_IN) * WG_P);
        } else {
            // weight gradient rows j = tp + 16 r, columns i = tj + 16 e (16 adjacent
            // columns per half warp: whole sectors)
            float g[4][4];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int e = 0; e < 4; e++) g[r][e] = 0.f;
            tile_rows(A3, l == 2 ? A2 : A1, tp, tj, g);
            const int wo = l == 2 ? MLP_W3 : MLP_W2;
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int e = 0; e < 4; e++) out[wo + (tp + 16 * r) * MLP_H + tj + 16 * e] = g[r][e];
            // next deltas: sum_k W[k][j] d[k][point]
            const float *W = sm + (l == 2 ? GS_W3 : GS_W2);
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int e = 0; e < 4; e++) d[r][e] = 0.f;
#pragma unroll 8
            for (int k = 0; k < MLP_H; k++) {
                const float4 x = *reinterpret_cast<const float4 *>(A3 + k * WG_P + 4 * tp);
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const float w = W[k * WG_P + tj + 16 * r];
                    d[r][0] = fmaf(w, x.x, d[r][0]);
                    d[r][1] = fmaf(w, x.y, d[r][1]);
                    d[r][2] = fmaf(w, x.z, d[r][2]);
                    d[r][3] = fmaf(w, x.w, d[r][3]);
                }
            }
        }
    }
}

// gradient and loss: the chunks' values, eight groups of consecutive chunks per
// parameter, each summed in order, then the groups in order
static __global__ void __launch_bounds__(256) k_mlp_grad_sum(int nchunk, const float *__restrict__ part, float *__restrict__ grad,
                                                             float *__restrict__ loss)
{
    __shared__ float sh[8][32];
    const int q = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
    const int per = (nchunk + 7) / 8, c0 = w * per, c1 = min(nchunk, c0 + per);
    float s = 0.f;
    if (q <= MLP_NPARAM) {
#pragma unroll 8
        for (int c = c0; c < c1; c++) s += part[(int64_t)c * (MLP_NPARAM + 1) + q];
    }
    sh[w][threadIdx.x & 31] = s;
    __syncthreads();
    if (w != 0 || q > MLP_NPARAM) return;
    for (int k = 1; k < 8; k++) s += sh[k][threadIdx.x & 31];
    if (q < MLP_NPARAM) grad[q] = s;
    else *loss = s;
}

H3D_HD uint64_t splitmix64(uint64_t z)
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// minibatch indices drawn uniformly from [0, P) by a counter-based hash
static __global__ void k_sample_idx(int64_t np, int64_t P, uint64_t key, int32_t *__restrict__ idx)
{
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p < np) idx[p] = (int32_t)(splitmix64(key ^ ((uint64_t)p * 0xd1b54a32d192ed03ull)) % (uint64_t)P);
}

// Adam on the fp32 master parameters; the bf16 copy used by the kernels follows
static __global__ void k_adam(int n, float lr, float b1, float b2, float eps, float c1, float c2,
                              const float *__restrict__ g, float *__restrict__ w, float *__restrict__ m,
                              float *__restrict__ v, __nv_bfloat16 *__restrict__ wb)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        wb[i] = __float2bfloat16_rn(wi);
    }
}

static __global__ void k_to_bf16(int n, const float *__restrict__ w, __nv_bfloat16 *__restrict__ wb)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) wb[i] = __float2bfloat16_rn(w[i]);
}

// inference on gradient fields of precision TS: point t of np reads A_ij at
// G[(3i+j) fs + off(t)] and writes tau_c to G[c fs + off(t)] (each point is
// read completely before it is written, by the same thread), where off(t)
// maps the x-fastest point index onto rows of n points at pitch rp.  With
// clip, points whose predicted dissipation -tau:S is negative get tau = 0.
template <typename TS>
__global__ void __launch_bounds__(MLP_NT) k_mlp_apply(int64_t np, int64_t n, int64_t rp, int64_t fs, float delta,
                                                      int clip, const __nv_bfloat16 *__restrict__ wb, TS *G)
{
    extern __shared__ __align__(16) float sm[];
    load_params(wb, sm);
    float *act = sm + MLP_WPAD + threadIdx.x;
    const int64_t t = blockIdx.x * (int64_t)MLP_NT + threadIdx.x;
    if (t < np) {
        const int64_t row = t / n, o = row * rp + (t - row * n);
        float Am[3][3];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) Am[i][j] = (float)G[(3 * i + j) * fs + o];
        Feat f;
        features(Am, delta, f);
        float g[MLP_OUT], tau[MLP_TC];
        mlp_forward(sm, act, f.x, g);
        basis_sum(f, g, tau);
        const bool zero = clip && sgs_diss(tau, f.sbar) < 0.f;
#pragma unroll
        for (int c = 0; c < MLP_TC; c++) G[c * fs + o] = zero ? (TS)0 : (TS)tau[c];
    }
}
