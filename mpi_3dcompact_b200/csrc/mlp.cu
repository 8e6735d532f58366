// Learned SGS closure: a 9 -> 64 -> 64 -> 64 -> 2 MLP (GELU) mapping local
// invariants of the resolved velocity-gradient tensor and the grid scale to
// the Smagorinsky-form coefficient C (nu_t = C Delta^2 |S|) and the turbulent
// Prandtl number. No counterpart in the reference: it stands in for
// VremanSGS / DSMSGS (src/VremanSGS.hpp, src/DSMSGS.hpp) behind the same
// solver path, with DSM kept as the fallback.
//
// Training (FP32, CUDA cores): mlp_tile runs forward, backward and the weight
// gradients of 128 samples at a time in shared memory and registers, each CTA's
// gradients summed over its tiles; mlp_update sums the CTAs' gradients and
// applies Adam with bias correction.
// Inference (BF16 tensor cores, FP32 accumulate in tensor memory) runs on
// tcgen05 MMAs over tiles of 128 points (mlp_tc.cuh, kernels in sgs_mlp.cu);
// mlp_pack writes its weight image after every change of the parameters.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <string>
#include <vector>

#include "mlp_common.cuh"

namespace mc3d {

// parameter offsets (floats) of the FP32 master copy
constexpr int MLP_W1 = 0;                          // [64][9]
constexpr int MLP_B1 = MLP_W1 + 64 * MLP_IN;       // [64]
constexpr int MLP_W2 = MLP_B1 + 64;                // [64][64]
constexpr int MLP_B2 = MLP_W2 + 64 * 64;
constexpr int MLP_W3 = MLP_B2 + 64;
constexpr int MLP_B3 = MLP_W3 + 64 * 64;
constexpr int MLP_W4 = MLP_B3 + 64;                // [2][64]
constexpr int MLP_B4 = MLP_W4 + MLP_OUT * 64;
constexpr int MLP_NP = MLP_B4 + MLP_OUT;           // 9090
static_assert(MLP_NP == MLP_NPARAM, "parameter count");

namespace {

// ---------------------------------------------------------------------------
// training: forward, backward and weight gradients of a tile of samples in one
// kernel, the gradients summed in registers over a persistent CTA's tiles
// ---------------------------------------------------------------------------
constexpr int TB = 128;        // samples per tile
constexpr int TT = 512;        // threads
constexpr int PA = TB + 4;     // pitch of the activation arrays [feature][sample]
constexpr int PW = 64 + 4;     // pitch of the 64 x 64 weights
// shared memory (floats): weights, then a0, h1, g1, h2, g2, d3
constexpr int TS_W2 = 0, TS_W3 = TS_W2 + 64 * PW, TS_W1 = TS_W3 + 64 * PW, TS_B1 = TS_W1 + 64 * MLP_IN;
constexpr int TS_B2 = TS_B1 + 64, TS_B3 = TS_B2 + 64, TS_W4 = TS_B3 + 64, TS_B4 = TS_W4 + MLP_OUT * 64;
constexpr int TS_A0 = TS_B4 + 4, TS_H1 = TS_A0 + MLP_IN * PA, TS_G1 = TS_H1 + 64 * PA, TS_H2 = TS_G1 + 64 * PA;
constexpr int TS_G2 = TS_H2 + 64 * PA, TS_D3 = TS_G2 + 64 * PA, TS_END = TS_D3 + 64 * PA;
static_assert(TS_A0 % 4 == 0 && TS_H1 % 4 == 0, "16-byte rows");
static_assert(TS_END * 4 <= 227 * 1024, "shared memory of the training kernel");

__device__ __forceinline__ float4 ld4s(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// acc[j][s] += sum_k W[tx + 16 j][k] in[k][s0 + s]
__device__ __forceinline__ void tile_forward(const float *Wm, const float *in, int tx, int s0, float (&acc)[4][4]) {
#pragma unroll 4
    for (int k0 = 0; k0 < 64; k0 += 4) {
        float4 w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = ld4s(Wm + (tx + 16 * j) * PW + k0);
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            const float4 a = ld4s(in + (k0 + kk) * PA + s0);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float wv = kk == 0 ? w[j].x : kk == 1 ? w[j].y : kk == 2 ? w[j].z : w[j].w;
                acc[j][0] += wv * a.x;
                acc[j][1] += wv * a.y;
                acc[j][2] += wv * a.z;
                acc[j][3] += wv * a.w;
            }
        }
    }
}

// g[k][s] = (sum_o W[o][k] d[o][s]) g[k][s] for k = 4 tx .. 4 tx + 3, the thread's four samples
__device__ __forceinline__ void tile_backward(const float *Wm, const float *d, float *gbuf, int tx, int s0) {
    float acc[4][4] = {};
#pragma unroll 8
    for (int o = 0; o < 64; o++) {
        const float4 w = ld4s(Wm + o * PW + 4 * tx), a = ld4s(d + o * PA + s0);
        const float wj[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            acc[j][0] += wj[j] * a.x;
            acc[j][1] += wj[j] * a.y;
            acc[j][2] += wj[j] * a.z;
            acc[j][3] += wj[j] * a.w;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        float4 *q = reinterpret_cast<float4 *>(gbuf + (4 * tx + j) * PA + s0);
        const float4 g = *q;
        *q = make_float4(acc[j][0] * g.x, acc[j][1] * g.y, acc[j][2] * g.z, acc[j][3] * g.w);
    }
}

// G[j][i] += sum over the half tile's samples of d[tx + 16 j][b] h[ty + 16 i][b]
__device__ __forceinline__ void tile_wgrad(const float *d, const float *h, int tx, int ty, int half, float (&G)[4][4]) {
#pragma unroll 2
    for (int b = half * (TB / 2); b < (half + 1) * (TB / 2); b += 4) {
        float4 dv[4], hv[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            dv[j] = ld4s(d + (tx + 16 * j) * PA + b);
            hv[j] = ld4s(h + (ty + 16 * j) * PA + b);
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                G[j][i] += dv[j].x * hv[i].x;
                G[j][i] += dv[j].y * hv[i].y;
                G[j][i] += dv[j].z * hv[i].z;
                G[j][i] += dv[j].w * hv[i].w;
            }
    }
}

// TRAIN: per-CTA gradient sums into part[blockIdx.x][MLP_NP] (MSE loss =
// (1/n) sum_b sum_o (out - y)^2) and loss sums into lpart[blockIdx.x];
// otherwise the network's outputs.
// FP32 throughout: 26 k multiply-adds a sample, 47 us for 65536 samples at the
// FP32 pipes' full rate. A thread holds 4 x 4 outputs of every product, so an
// inner step is 64 FMAs on 8 16-byte shared loads; activations are laid out
// [feature][sample] so that forward, backward and the sums over samples all
// load 16 bytes, nearly without bank conflicts, and nothing of a tile goes to memory.
// Bound by issue (57% of the slots) and the shared loads (61% of that pipe; FMA
// pipe 39%), at one CTA an SM: 149 us of the 201 us a training step of 65536
// samples takes on a B200.
template <bool TRAIN>
__global__ void __launch_bounds__(TT, 1) mlp_tile_kernel(const float *__restrict__ P, const float *__restrict__ x,
                                                         const float *__restrict__ y, int n, MlpNorm nrm,
                                                         float *__restrict__ out, float *__restrict__ part,
                                                         double *__restrict__ lpart) {
    extern __shared__ __align__(16) float sm[];
    const int t = threadIdx.x;
    for (int k = t; k < 64 * 64; k += TT) {
        sm[TS_W2 + (k >> 6) * PW + (k & 63)] = P[MLP_W2 + k];
        sm[TS_W3 + (k >> 6) * PW + (k & 63)] = P[MLP_W3 + k];
    }
    for (int k = t; k < 64 * MLP_IN; k += TT) sm[TS_W1 + k] = P[MLP_W1 + k];
    if (t < 64) {
        sm[TS_B1 + t] = P[MLP_B1 + t];
        sm[TS_B2 + t] = P[MLP_B2 + t];
        sm[TS_B3 + t] = P[MLP_B3 + t];
    }
    if (t < MLP_OUT * 64) sm[TS_W4 + t] = P[MLP_W4 + t];
    if (t < MLP_OUT) sm[TS_B4 + t] = P[MLP_B4 + t];

    const int tx = t & 15, s0 = 4 * (t >> 4);                  // products: outputs tx + 16 j (or 4 tx + j), samples s0 + s
    const int half = t >> 8, wy = (t >> 4) & 15;               // weight gradients
    const int bo = t & 63, bq = t >> 6;                        // layer 1 and biases: output bo, samples 16 bq ..
    float G2[4][4] = {}, G3[4][4] = {}, G4[MLP_OUT][4] = {}, g4b[MLP_OUT] = {};
    float G1[MLP_IN] = {}, gb[3] = {};
    double loss = 0.0;
    const long long ntile = ((long long)n + TB - 1) / TB;
    for (long long tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const long long b0 = tile * TB;
        __syncthreads();   // the last tile's readers, and the weights
        for (int k = t; k < TB * MLP_IN; k += TT) {
            const int c = k % MLP_IN, b = k / MLP_IN;
            sm[TS_A0 + c * PA + b] = b0 + b < n ? (x[b0 * MLP_IN + k] - nrm.mean[c]) * nrm.inv_std[c] : 0.0f;
        }
        __syncthreads();
        float acc[4][4];
        // layer 1
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int s = 0; s < 4; s++) acc[j][s] = sm[TS_B1 + tx + 16 * j];
#pragma unroll
        for (int k = 0; k < MLP_IN; k++) {
            const float4 a = ld4s(sm + TS_A0 + k * PA + s0);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float w = sm[TS_W1 + (tx + 16 * j) * MLP_IN + k];
                acc[j][0] += w * a.x;
                acc[j][1] += w * a.y;
                acc[j][2] += w * a.z;
                acc[j][3] += w * a.w;
            }
        }
        auto activate = [&](int hoff, int goff) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float h[4], g[4];
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    if (TRAIN) gelu_both(acc[j][s], h[s], g[s]);
                    else h[s] = gelu(acc[j][s]);
                }
                const int at = (tx + 16 * j) * PA + s0;
                *reinterpret_cast<float4 *>(sm + hoff + at) = make_float4(h[0], h[1], h[2], h[3]);
                if (TRAIN) *reinterpret_cast<float4 *>(sm + goff + at) = make_float4(g[0], g[1], g[2], g[3]);
            }
        };
        activate(TS_H1, TS_G1);
        __syncthreads();
        // layer 2
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int s = 0; s < 4; s++) acc[j][s] = sm[TS_B2 + tx + 16 * j];
        tile_forward(sm + TS_W2, sm + TS_H1, tx, s0, acc);
        activate(TS_H2, TS_G2);
        __syncthreads();
        // layer 3, kept in registers: its outputs feed layer 4 only
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int s = 0; s < 4; s++) acc[j][s] = sm[TS_B3 + tx + 16 * j];
        tile_forward(sm + TS_W3, sm + TS_H2, tx, s0, acc);
        float o4[MLP_OUT][4] = {};
        float g3[4][4];
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int s = 0; s < 4; s++) {
                float h;
                if (TRAIN) gelu_both(acc[j][s], h, g3[j][s]);
                else h = gelu(acc[j][s]);
                acc[j][s] = h;
#pragma unroll
                for (int o = 0; o < MLP_OUT; o++) o4[o][s] += sm[TS_W4 + o * 64 + tx + 16 * j] * h;
            }
        // layer 4: the 16 threads of a sample group hold four outputs each
#pragma unroll
        for (int o = 0; o < MLP_OUT; o++)
#pragma unroll
            for (int s = 0; s < 4; s++) {
#pragma unroll
                for (int m = 8; m > 0; m >>= 1) o4[o][s] += __shfl_xor_sync(0xffffffffu, o4[o][s], m);
                o4[o][s] += sm[TS_B4 + o];
            }
        if constexpr (!TRAIN) {
            if (tx == 0) {
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (b0 + s0 + s < n) {
#pragma unroll
                        for (int o = 0; o < MLP_OUT; o++) out[(b0 + s0 + s) * MLP_OUT + o] = o4[o][s];
                    }
            }
        } else {
            // o4 becomes the output deltas; samples past the batch have none
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const bool valid = b0 + s0 + s < n;
#pragma unroll
                for (int o = 0; o < MLP_OUT; o++) {
                    const float e = valid ? o4[o][s] - y[(b0 + s0 + s) * MLP_OUT + o] : 0.0f;
                    if (tx == 0) loss += (double)e * e;
                    o4[o][s] = 2.0f * e / (float)n;
                    g4b[o] += o4[o][s];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float d[4];
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    float v = 0.0f;
#pragma unroll
                    for (int o = 0; o < MLP_OUT; o++) {
                        G4[o][j] += o4[o][s] * acc[j][s];
                        v += sm[TS_W4 + o * 64 + tx + 16 * j] * o4[o][s];
                    }
                    d[s] = v * g3[j][s];
                }
                *reinterpret_cast<float4 *>(sm + TS_D3 + (tx + 16 * j) * PA + s0) = make_float4(d[0], d[1], d[2], d[3]);
            }
            __syncthreads();
            tile_wgrad(sm + TS_D3, sm + TS_H2, tx, wy, half, G3);
            tile_backward(sm + TS_W3, sm + TS_D3, sm + TS_G2, tx, s0);   // g2 becomes delta 2
            __syncthreads();
            tile_wgrad(sm + TS_G2, sm + TS_H1, tx, wy, half, G2);
            tile_backward(sm + TS_W2, sm + TS_G2, sm + TS_G1, tx, s0);   // g1 becomes delta 1
            __syncthreads();
#pragma unroll
            for (int b = 0; b < TB / 8; b += 4) {
                const int at = 16 * bq + b;
                const float4 d = ld4s(sm + TS_G1 + bo * PA + at);
#pragma unroll
                for (int k = 0; k < MLP_IN; k++) {
                    const float4 a = ld4s(sm + TS_A0 + k * PA + at);
                    G1[k] += d.x * a.x;
                    G1[k] += d.y * a.y;
                    G1[k] += d.z * a.z;
                    G1[k] += d.w * a.w;
                }
                const float4 d2 = ld4s(sm + TS_G2 + bo * PA + at), d3 = ld4s(sm + TS_D3 + bo * PA + at);
                gb[0] += (d.x + d.y) + (d.z + d.w);
                gb[1] += (d2.x + d2.y) + (d2.z + d2.w);
                gb[2] += (d3.x + d3.y) + (d3.z + d3.w);
            }
        }
    }
    if constexpr (TRAIN) {
        // the CTA's sums: shared-memory scratch over the activation arrays
        float *r2 = sm + TS_H1, *r3 = r2 + 64 * 64, *r4 = r3 + 64 * 64, *r1 = r4 + 32 * MLP_OUT * 64;
        float *rb = r1 + 8 * 64 * (MLP_IN + 3);
        double *rl = reinterpret_cast<double *>(rb + 32 * MLP_OUT);
        __syncthreads();
        if (half == 1) {
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    r2[(tx + 16 * j) * 64 + wy + 16 * i] = G2[j][i];
                    r3[(tx + 16 * j) * 64 + wy + 16 * i] = G3[j][i];
                }
        }
        const int ty = t >> 4;
#pragma unroll
        for (int o = 0; o < MLP_OUT; o++)
#pragma unroll
            for (int j = 0; j < 4; j++) r4[(ty * MLP_OUT + o) * 64 + tx + 16 * j] = G4[o][j];
#pragma unroll
        for (int k = 0; k < MLP_IN; k++) r1[(bq * (MLP_IN + 3) + k) * 64 + bo] = G1[k];
#pragma unroll
        for (int k = 0; k < 3; k++) r1[(bq * (MLP_IN + 3) + MLP_IN + k) * 64 + bo] = gb[k];
        if (tx == 0) {
#pragma unroll
            for (int o = 0; o < MLP_OUT; o++) rb[ty * MLP_OUT + o] = g4b[o];
            rl[ty] = loss;
        }
        __syncthreads();
        float *G = part + (size_t)blockIdx.x * MLP_NP;
        if (half == 0) {
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int at = (tx + 16 * j) * 64 + wy + 16 * i;
                    r2[at] += G2[j][i];
                    r3[at] += G3[j][i];
                }
        }
        __syncthreads();
        for (int k = t; k < 64 * 64; k += TT) {
            G[MLP_W2 + k] = r2[k];
            G[MLP_W3 + k] = r3[k];
        }
        for (int k = t; k < (MLP_IN + 3) * 64; k += TT) {
            float s = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; q++) s += r1[q * (MLP_IN + 3) * 64 + k];
            const int c = k >> 6, o = k & 63;
            G[c < MLP_IN ? MLP_W1 + o * MLP_IN + c : (c == MLP_IN ? MLP_B1 : c == MLP_IN + 1 ? MLP_B2 : MLP_B3) + o] = s;
        }
        if (t < MLP_OUT * 64) {
            float s = 0.0f;
            for (int q = 0; q < 32; q++) s += r4[q * MLP_OUT * 64 + t];
            G[MLP_W4 + t] = s;
        }
        if (t < MLP_OUT) {
            float s = 0.0f;
            for (int q = 0; q < 32; q++) s += rb[q * MLP_OUT + t];
            G[MLP_B4 + t] = s;
        }
        if (t == 0) {
            double s = 0.0;
            for (int q = 0; q < 32; q++) s += rl[q];
            lpart[blockIdx.x] = s;
        }
    }
}

// Sums the CTAs' gradients, 32 parameters by 8 groups of CTAs a block, in a
// fixed order. ADAM: one Adam step with the sum; otherwise the sum into G. The
// first block also sums the loss.
template <bool ADAM>
__global__ void __launch_bounds__(256) mlp_update_kernel(const float *__restrict__ part,
                                                         const double *__restrict__ lpart, int nparts, int n,
                                                         float *P, float *G, float *M, float *V, float lr, float b1t,
                                                         float b2t, double *loss) {
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = blockIdx.x * 32 + lane;
    float s = 0.0f;
    if (k < MLP_NP)
        for (int c = w; c < nparts; c += 8) s += part[(size_t)c * MLP_NP + k];
    red[w][lane] = s;
    if (blockIdx.x == 0 && w == 1) {
        double l = 0.0;
        for (int c = lane; c < nparts; c += 32) l += lpart[c];
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) *loss = l / (double)n;
    }
    __syncthreads();
    if (w != 0 || k >= MLP_NP) return;
    float g = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) g += red[q][lane];
    if constexpr (!ADAM) {
        G[k] = g;
    } else {
        const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
        const float m = b1 * M[k] + (1.0f - b1) * g;
        const float v = b2 * V[k] + (1.0f - b2) * g * g;
        M[k] = m;
        V[k] = v;
        const float mh = m / (1.0f - b1t), vh = v / (1.0f - b2t);
        P[k] -= lr * mh / (sqrtf(vh) + eps);
    }
}

// The weight image of the tensor-core inference (layout in mlp_common.cuh),
// written over a zeroed buffer: one thread per element of the eight blocks.
// A bias b is carried as the BF16 pair (b_hi, b_lo), b_hi = bf16(b) and
// b_lo = bf16(b - b_hi), against two constant-one input columns.
__device__ __forceinline__ void bias_pair(float b, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
    hi = __float2bfloat16_rn(b);
    lo = __float2bfloat16_rn(b - __bfloat162float(hi));
}

__global__ void mlp_pack_kernel(const float *__restrict__ P, unsigned char *__restrict__ img) {
    // element counts of W1 [64][16], W2, W3 [64][64], W4 [16][64], B2, B3 [64][16], B4 [16][16], Ac [128][16]
    constexpr int n1 = 64 * 16, n2 = 64 * 64, n4 = 16 * 64, nb = 64 * 16, nb4 = 16 * 16, nac = 128 * 16;
    constexpr int total = n1 + 2 * n2 + n4 + 2 * nb + nb4 + nac;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        int k = e, off;
        __nv_bfloat16 v = __float2bfloat16_rn(0.0f);
        if (k < n1) {   // W1 and the layer-1 bias
            const int o = k / 16, c = k % 16;
            __nv_bfloat16 hi, lo;
            bias_pair(P[MLP_B1 + o], hi, lo);
            if (c < MLP_IN) v = __float2bfloat16_rn(P[MLP_W1 + o * MLP_IN + c]);
            else if (c == MLP_IN) v = hi;
            else if (c == MLP_IN + 1) v = lo;
            off = MLPT_W1 + tc_off16(o, c);
        } else if ((k -= n1) < 2 * n2) {   // W2, W3, halved: their inputs are twice GELU (gelu2_bf16x2)
            const int w = k < n2 ? MLP_W2 : MLP_W3, kk = k % n2, o = kk / 64, c = kk % 64;
            v = __float2bfloat16_rn(0.5f * P[w + o * 64 + c]);
            off = (k < n2 ? MLPT_W2 : MLPT_W3) + tc_off64(o, c);
        } else if ((k -= 2 * n2) < n4) {   // W4, halved likewise; rows past the outputs zero
            const int o = k / 64, c = k % 64;
            if (o < MLP_OUT) v = __float2bfloat16_rn(0.5f * P[MLP_W4 + o * 64 + c]);
            off = MLPT_W4 + tc_off64(o, c);
        } else if ((k -= n4) < 2 * nb + nb4) {   // bias blocks of layers 2, 3, 4
            const int blk = k < nb ? 0 : k < 2 * nb ? 1 : 2, kk = k - blk * nb, o = kk / 16, c = kk % 16;
            const int nout = blk == 2 ? MLP_OUT : 64;
            if (o < nout && c < 2) {
                __nv_bfloat16 hi, lo;
                bias_pair(P[(blk == 0 ? MLP_B2 : blk == 1 ? MLP_B3 : MLP_B4) + o], hi, lo);
                v = c == 0 ? hi : lo;
            }
            off = (blk == 0 ? MLPT_B2 : blk == 1 ? MLPT_B3 : MLPT_B4) + tc_off16(o, c);
        } else {   // the constant-one columns of the bias MMAs
            k -= 2 * nb + nb4;
            const int r = k / 16, c = k % 16;
            if (c < 2) v = __float2bfloat16_rn(1.0f);
            off = MLPT_AC + tc_off16(r, c);
        }
        *reinterpret_cast<__nv_bfloat16 *>(img + off) = v;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
int mlp_pack(const MlpDev &m, cudaStream_t st) {
    MC3D_CUDA_TRY(cudaMemsetAsync(m.Tw, 0, MLPT_BYTES, st));
    mlp_pack_kernel<<<16, 256, 0, st>>>(m.P, m.Tw);
    MC3D_CUDA_TRY(cudaGetLastError());
    return MC3D_OK;
}

namespace {
// the tile kernel's launch: one persistent CTA an SM (nparts: the CTAs launched)
template <bool TRAIN>
int launch_tiles(const MlpDev &m, const float *x, const float *y, int n, float *out, float *part, double *lpart,
                 int *nparts, cudaStream_t st) {
    static KernelLaunchState ls;
    const size_t smem = TS_END * sizeof(float);
    int ctas = 0;
    if (int rc = open_kernel(mlp_tile_kernel<TRAIN>, ls, smem, TT, &ctas)) return rc;
    if (ctas > MLP_MAXPARTS) ctas = MLP_MAXPARTS;
    const int tiles = (int)(((long long)n + TB - 1) / TB);
    *nparts = tiles < ctas ? tiles : ctas;
    mlp_tile_kernel<TRAIN><<<*nparts, TT, smem, st>>>(m.P, x, y, n, m.norm, out, part, lpart);
    MC3D_CUDA_TRY(cudaGetLastError());
    return MC3D_OK;
}
}  // namespace

int mlp_forward_fp32(const MlpDev &m, const float *x, int n, float *out, cudaStream_t st) {
    int nparts;
    return launch_tiles<false>(m, x, nullptr, n, out, nullptr, nullptr, &nparts, st);
}

int mlp_gradient(MlpDev &m, const float *x, const float *y, int n, float *part, double *lpart, double *loss,
                 cudaStream_t st) {
    int nparts;
    if (int rc = launch_tiles<true>(m, x, y, n, nullptr, part, lpart, &nparts, st)) return rc;
    mlp_update_kernel<false><<<(MLP_NP + 31) / 32, 256, 0, st>>>(part, lpart, nparts, n, m.P, m.G, m.M, m.V, 0.0f, 0.0f,
                                                                 0.0f, loss);
    MC3D_CUDA_TRY(cudaGetLastError());
    return MC3D_OK;
}

int mlp_train_step(MlpDev &m, const float *x, const float *y, int n, float lr, float *part, double *lpart,
                   double *loss, cudaStream_t st) {
    int nparts;
    if (int rc = launch_tiles<true>(m, x, y, n, nullptr, part, lpart, &nparts, st)) return rc;
    m.t += 1;
    const float b1t = (float)std::pow(0.9, (double)m.t), b2t = (float)std::pow(0.999, (double)m.t);
    mlp_update_kernel<true><<<(MLP_NP + 31) / 32, 256, 0, st>>>(part, lpart, nparts, n, m.P, m.G, m.M, m.V, lr, b1t,
                                                                b2t, loss);
    MC3D_CUDA_TRY(cudaGetLastError());
    return mlp_pack(m, st);
}

}  // namespace mc3d
