// k_mlp.cu — the learned kernel-class selector: matrix features and a small
// MLP (12 -> 64 -> 64 -> 6, ReLU, FP32) with its forward, backward and Adam
// kernels.
//
// No counterpart in the reference: its only "autotuner" is the (ngpu, q)
// sweep of test/dspmv_test.cu:314-332.  The MLP predicts, per kernel class,
// log2(t_class / t_best) of a plain launch from 12 features of the matrix;
// the selector takes the class with the smallest prediction.
//
// Determinism: the features come from integer accumulators (exact, so the
// order of the atomics does not matter), and every sum over samples in the
// backward pass runs in a fixed order, so training is bit-reproducible.
#include <math.h>
#include <stdint.h>

#include "../sbb_internal.h"
#include "common.cuh"

namespace sbb {

namespace {

// ---- features ---------------------------------------------------------------
// Integer accumulators over rows (index: meaning):
//   0: sum L^2   1: max L   2: empty rows   3: rows with L <= 4
//   4: rows with L > 32   5: nnz in rows with L > 128   6: sum of column spans
//   7: non-empty rows
constexpr int kAcc = 8;

__global__ void __launch_bounds__(256)
feature_acc_kernel(const int *__restrict__ rp, const int *__restrict__ col, int m,
                   unsigned long long *__restrict__ acc)
{
    unsigned long long a[kAcc] = {};
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < m;
         r += (long long)gridDim.x * blockDim.x) {
        const int lo = __ldg(rp + r), hi = __ldg(rp + r + 1);
        const unsigned long long L = hi > lo ? (unsigned long long)(hi - lo) : 0ull;
        a[0] += L * L;
        a[1] = L > a[1] ? L : a[1];
        a[2] += L == 0;
        a[3] += L <= 4;
        a[4] += L > 32;
        a[5] += L > 128 ? L : 0ull;
        if (L) {
            const int c0 = __ldg(col + lo), c1 = __ldg(col + hi - 1);
            a[6] += (unsigned long long)(c1 >= c0 ? c1 - c0 + 1 : c0 - c1 + 1);
            a[7] += 1;
        }
    }
#pragma unroll
    for (int k = 0; k < kAcc; ++k) {
        unsigned long long v = a[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
            v = k == 1 ? (u > v ? u : v) : v + u;
        }
        if ((threadIdx.x & 31) == 0) {
            if (k == 1)
                atomicMax(acc + 1, v);
            else if (v)
                atomicAdd(acc + k, v);
        }
    }
}

// The 12 features (all O(1) in magnitude before normalisation):
//   0 log2(1+m)  1 log2(1+n)  2 log2(1+nnz)  3 log2(1+mean L)
//   4 coefficient of variation of L  5 log2(1+max L)  6 log2(1+max L/mean L)
//   7 empty-row fraction  8 fraction of rows with L <= 4  9 fraction with L > 32
//   10 fraction of nnz in rows with L > 128  11 mean column span / n
__global__ void feature_final_kernel(const unsigned long long *__restrict__ acc, int m, int n,
                                     long long nnz, float *__restrict__ f)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double M = m > 0 ? m : 1, N = n > 0 ? n : 1, Z = (double)nnz;
    const double mean = Z / M;
    const double var = fmax((double)acc[0] / M - mean * mean, 0.0);
    const double mx = (double)acc[1];
    const double ne = acc[7] > 0 ? (double)acc[7] : 1.0;
    f[0] = (float)log2(1.0 + m);
    f[1] = (float)log2(1.0 + n);
    f[2] = (float)log2(1.0 + Z);
    f[3] = (float)log2(1.0 + mean);
    f[4] = (float)(mean > 0 ? sqrt(var) / mean : 0.0);
    f[5] = (float)log2(1.0 + mx);
    f[6] = (float)log2(1.0 + (mean > 0 ? mx / mean : 0.0));
    f[7] = (float)((double)acc[2] / M);
    f[8] = (float)((double)acc[3] / M);
    f[9] = (float)((double)acc[4] / M);
    f[10] = (float)(Z > 0 ? (double)acc[5] / Z : 0.0);
    f[11] = (float)((double)acc[6] / ne / N);
}

// ---- MLP --------------------------------------------------------------------
// Parameter blob (floats): mu[12], sd[12] (feature normalisation, fixed),
// W1[64][12], b1[64], W2[64][64], b2[64], W3[6][64], b3[6].
constexpr int F = kMlpFeatures, H = kMlpHidden, C = kMlpClasses;
constexpr int oMU = 0, oSD = F, oW1 = 2 * F, oB1 = oW1 + H * F, oW2 = oB1 + H, oB2 = oW2 + H * H,
              oW3 = oB2 + H, oB3 = oW3 + C * H, kParams = oB3 + C;
static_assert(kParams == kMlpParams, "parameter blob layout");

__device__ __forceinline__ float relu(float v) { return v > 0.f ? v : 0.f; }

// A block of 256 threads works on kTile samples at a time, with the
// parameters and the samples' layers in shared memory.  16 samples a block, twice
// the blocks, is as fast on 500 samples and slower on 4,000 (22.6 and 16.8 us a
// step), where the sums over twice the parts cost more.  Rows of 64 are 68
// floats apart: 16-byte reads of eight consecutive rows then fall into
// different banks.
constexpr int MT = 256, kTile = 32, kRow = 68;
constexpr int kPer = kTile / 16;  // samples of a thread in the 64 x 64 layers
struct TileMem {
    float mu[F], sd[F], W1[H * F], W2[H * kRow], W3[C * kRow];
    float b1[H], b2[H], b3[C + 2];
    float x[kTile * F];
    float h1[kTile * kRow];  // layer 1, later its error terms
    float h2[kTile * kRow];  // layer 2, later its error terms
    float y[kTile * 8], dy[kTile * 8];
};
static_assert(sizeof(TileMem) <= 48 * 1024, "static shared memory");

// Every load of a thread is issued before its first store.
__device__ __forceinline__ void load_params(TileMem &T, const float *__restrict__ P)
{
    const int t = threadIdx.x;
    float w2[H * H / MT], w1[H * F / MT], w3[2];
#pragma unroll
    for (int q = 0; q < H * H / MT; ++q) w2[q] = __ldcg(P + oW2 + t + q * MT);
#pragma unroll
    for (int q = 0; q < H * F / MT; ++q) w1[q] = __ldcg(P + oW1 + t + q * MT);
    w3[0] = __ldcg(P + oW3 + t);
    w3[1] = t < C * H - MT ? __ldcg(P + oW3 + MT + t) : 0.f;
    // the normalisation and the biases, one a thread
    const int rest = t < oW1                ? t
                     : t < oW1 + H         ? oB1 + t - oW1
                     : t < oW1 + 2 * H     ? oB2 + t - oW1 - H
                     : t < oW1 + 2 * H + C ? oB3 + t - oW1 - 2 * H
                                           : -1;
    const float r = rest >= 0 ? __ldcg(P + rest) : 0.f;
#pragma unroll
    for (int q = 0; q < H * H / MT; ++q) T.W2[(t / H + q * (MT / H)) * kRow + t % H] = w2[q];
#pragma unroll
    for (int q = 0; q < H * F / MT; ++q) T.W1[t + q * MT] = w1[q];
    T.W3[t / H * kRow + t % H] = w3[0];
    if (t < C * H - MT) T.W3[(t + MT) / H * kRow + t % H] = w3[1];
    if (rest >= oB3) T.b3[rest - oB3] = r;
    else if (rest >= oB2) T.b2[rest - oB2] = r;
    else if (rest >= oB1) T.b1[rest - oB1] = r;
    else if (rest >= oSD) T.sd[rest - oSD] = r;
    else if (rest >= oMU) T.mu[rest - oMU] = r;
}
static_assert(H * H % MT == 0 && H * F % MT == 0 && C * H >= MT && C * H <= 2 * MT &&
                  oW1 + 2 * H + C <= MT, "load_params");

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Forward pass of samples n0 .. n0 + ns - 1 (rows past ns stay zero): each sum
// starts from the bias and runs over the inputs in order.
__device__ __forceinline__ void tile_forward(TileMem &T, const float *__restrict__ X, int n0, int ns)
{
    const int t = threadIdx.x;
    for (int i = t; i < kTile * F; i += MT) {
        const int k = i % F;
        const float sd = T.sd[k];
        T.x[i] = i < ns * F ? __fdiv_rn(__fsub_rn(X[(size_t)n0 * F + i], T.mu[k]), sd > 0.f ? sd : 1.f)
                            : 0.f;
    }
    __syncthreads();
    {  // layer 1: neuron j of 8 samples
        const int j = t % H;
        float w[F];
#pragma unroll
        for (int q = 0; q < F; q += 4) {
            const float4 v = ld4(T.W1 + j * F + q);
            w[q] = v.x, w[q + 1] = v.y, w[q + 2] = v.z, w[q + 3] = v.w;
        }
        const float b = T.b1[j];
#pragma unroll
        for (int i = 0; i < kTile * H / MT; ++i) {
            const int n = t / H + i * (MT / H);
            float z = b;
#pragma unroll
            for (int k = 0; k < F; ++k) z = __fmaf_rn(w[k], T.x[n * F + k], z);
            T.h1[n * kRow + j] = n < ns ? relu(z) : 0.f;
        }
    }
    __syncthreads();
    {  // layer 2: neurons j, j+16, j+32, j+48 of sample n (and n+16)
        const int j = t % 16, n = t / 16;
        float z[kPer][4];
#pragma unroll
        for (int i = 0; i < kPer; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) z[i][q] = T.b2[j + 16 * q];
#pragma unroll 4
        for (int k = 0; k < H; k += 4) {
            float4 a[kPer];
#pragma unroll
            for (int i = 0; i < kPer; ++i) a[i] = ld4(T.h1 + (n + 16 * i) * kRow + k);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 w = ld4(T.W2 + (j + 16 * q) * kRow + k);
#pragma unroll
                for (int i = 0; i < kPer; ++i) {
                    z[i][q] = __fmaf_rn(w.x, a[i].x, z[i][q]);
                    z[i][q] = __fmaf_rn(w.y, a[i].y, z[i][q]);
                    z[i][q] = __fmaf_rn(w.z, a[i].z, z[i][q]);
                    z[i][q] = __fmaf_rn(w.w, a[i].w, z[i][q]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kPer; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                T.h2[(n + 16 * i) * kRow + j + 16 * q] = n + 16 * i < ns ? relu(z[i][q]) : 0.f;
    }
    __syncthreads();
    if (t < kTile * C) {  // layer 3: one output of one sample
        const int n = t / C, c = t % C;
        float z = T.b3[c];
#pragma unroll 4
        for (int k = 0; k < H; k += 4) {
            const float4 a = ld4(T.h2 + n * kRow + k), w = ld4(T.W3 + c * kRow + k);
            z = __fmaf_rn(w.x, a.x, z);
            z = __fmaf_rn(w.y, a.y, z);
            z = __fmaf_rn(w.z, a.z, z);
            z = __fmaf_rn(w.w, a.w, z);
        }
        T.y[n * 8 + c] = z;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(MT)
mlp_forward_kernel(const float *__restrict__ P, const float *__restrict__ X, int N,
                   float *__restrict__ Y)
{
    __shared__ __align__(16) TileMem T;
    load_params(T, P);
    __syncthreads();
    const int n0 = blockIdx.x * kTile, ns = min(kTile, N - n0);
    tile_forward(T, X, n0, ns);
    for (int i = threadIdx.x; i < ns * C; i += MT)
        Y[(size_t)n0 * C + i] = T.y[i / C * 8 + i % C];
}

// Forward pass, error terms and gradient of the loss
//   L = sum_n w_n sum_c (Y[n,c] - T[n,c])^2 / (C * sum_n w_n)
// of the block's samples, summed over them in order: parts[block][kParams + 1]
// (the loss last).  The step was a kernel per stage, with the activations in
// global memory and one thread per parameter running over all samples: 4,000
// samples took 716 us, 0.6 ms of it in 22 blocks of 4,000-step chains.  Here
// 125 blocks hold 32 samples each, every stage is a register-tiled product
// over shared memory, and the sums over blocks are left to
// mlp_update_kernel: two launches and 17 us a step (12 us for 500 samples), bound by the latency of
// its seven dependent stages (1.0 MFLOP a block).
constexpr int kPartRow = (kParams + 1 + 31) / 32 * 32;
__global__ void __launch_bounds__(MT)
mlp_step_kernel(const float *__restrict__ P, const float *__restrict__ X, int N,
                const float *__restrict__ Tg, const float *__restrict__ W, float inv_norm,
                float *__restrict__ parts)
{
    __shared__ __align__(16) TileMem T;
    const int t = threadIdx.x;
    allow_dependent_launch();
    grid_dependency_wait();  // the parameters come from the kernel before
    load_params(T, P);
    // this thread's gradient entries: a 4 x 4 block of W2 (rows 4*tj.., columns
    // 4*tk..), 4 entries of W1 or none, 4 of W3 or none, a bias or none
    const int tj = t / 16, tk = t % 16;
    float g2[4][4] = {}, g1[4] = {}, g3[4] = {}, gb = 0.f, loss = 0.f;
    for (int n0 = blockIdx.x * kTile; n0 < N; n0 += gridDim.x * kTile) {
        const int ns = min(kTile, N - n0);
        __syncthreads();  // parameters loaded; the tile before is done with
        tile_forward(T, X, n0, ns);
        if (t < kTile) {  // errors of the outputs, one sample a thread
            const float w = t < ns ? (W ? W[n0 + t] : 1.f) : 0.f;
            const float scale = __fmul_rn(2.f * inv_norm, w);
            float e = 0.f;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const float d = t < ns ? __fsub_rn(T.y[t * 8 + c], Tg[(size_t)(n0 + t) * C + c]) : 0.f;
                e = __fmaf_rn(d, d, e);
                T.dy[t * 8 + c] = t < ns ? __fmul_rn(scale, d) : 0.f;
            }
            if (t < ns) loss = __fmaf_rn(w, e, loss);
        }
        __syncthreads();
        if (t < C * H / 4) {  // W3: output c, layer-2 neurons 4k ..
            const int c = t / 16, k = t % 16 * 4;
#pragma unroll 8
            for (int n = 0; n < kTile; ++n) {
                const float4 a = ld4(T.h2 + n * kRow + k);
                const float d = T.dy[n * 8 + c];
                g3[0] = __fmaf_rn(d, a.x, g3[0]);
                g3[1] = __fmaf_rn(d, a.y, g3[1]);
                g3[2] = __fmaf_rn(d, a.z, g3[2]);
                g3[3] = __fmaf_rn(d, a.w, g3[3]);
            }
        }
        __syncthreads();
        {  // errors of layer 2 in place of its values: neuron k of 8 samples
            const int k = t % H;
#pragma unroll
            for (int i = 0; i < kTile * H / MT; ++i) {
                const int n = t / H + i * (MT / H);
                float g = 0.f;
#pragma unroll
                for (int c = 0; c < C; ++c) g = __fmaf_rn(T.W3[c * kRow + k], T.dy[n * 8 + c], g);
                float &h = T.h2[n * kRow + k];
                h = h > 0.f ? g : 0.f;
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int n = 0; n < kTile; ++n) {  // W2
            const float4 d = ld4(T.h2 + n * kRow + 4 * tj), a = ld4(T.h1 + n * kRow + 4 * tk);
            const float dd[4] = {d.x, d.y, d.z, d.w}, aa[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int r = 0; r < 4; ++r) g2[q][r] = __fmaf_rn(dd[q], aa[r], g2[q][r]);
        }
        // errors of layer 1: neurons 4*tk .. of sample tj (and tj + 16)
        float d1[kPer][4] = {};
#pragma unroll 4
        for (int j = 0; j < H; j += 4) {
            float e[kPer][4];
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const float4 v = ld4(T.h2 + (tj + 16 * i) * kRow + j);
                e[i][0] = v.x, e[i][1] = v.y, e[i][2] = v.z, e[i][3] = v.w;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 w = ld4(T.W2 + (j + q) * kRow + 4 * tk);
                const float ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int i = 0; i < kPer; ++i)
#pragma unroll
                    for (int r = 0; r < 4; ++r) d1[i][r] = __fmaf_rn(ww[r], e[i][q], d1[i][r]);
            }
        }
        __syncthreads();  // every thread is done with layer 1's values
#pragma unroll
        for (int i = 0; i < kPer; ++i)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float &h = T.h1[(tj + 16 * i) * kRow + 4 * tk + r];
                h = h > 0.f ? d1[i][r] : 0.f;
            }
        __syncthreads();
        if (t < H * F / 4) {  // W1: neuron j, inputs 4f ..
            const int j = t / 3, f = t % 3 * 4;
#pragma unroll 8
            for (int n = 0; n < kTile; ++n) {
                const float4 a = ld4(T.x + n * F + f);
                const float d = T.h1[n * kRow + j];
                g1[0] = __fmaf_rn(d, a.x, g1[0]);
                g1[1] = __fmaf_rn(d, a.y, g1[1]);
                g1[2] = __fmaf_rn(d, a.z, g1[2]);
                g1[3] = __fmaf_rn(d, a.w, g1[3]);
            }
        }
        // biases: b1 by threads 0-63, b2 by 64-127, b3 by 128-133
        if (t < 2 * H) {
            const float *d = (t < H ? T.h1 : T.h2) + t % H;
#pragma unroll 8
            for (int n = 0; n < kTile; ++n) gb = __fadd_rn(gb, d[n * kRow]);
        } else if (t < 2 * H + C) {
#pragma unroll 8
            for (int n = 0; n < kTile; ++n) gb = __fadd_rn(gb, T.dy[n * 8 + t - 2 * H]);
        }
    }
    float *out = parts + (size_t)blockIdx.x * kPartRow;
    if (t < oW1) out[t] = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        *reinterpret_cast<float4 *>(out + oW2 + (4 * tj + q) * H + 4 * tk) =
            make_float4(g2[q][0], g2[q][1], g2[q][2], g2[q][3]);
        if (t < H * F / 4) out[oW1 + t / 3 * F + t % 3 * 4 + q] = g1[q];
        if (t < C * H / 4) out[oW3 + t / 16 * H + t % 16 * 4 + q] = g3[q];
    }
    if (t < H) out[oB1 + t] = gb;
    else if (t < 2 * H) out[oB2 + t - H] = gb;
    else if (t < 2 * H + C) out[oB3 + t - 2 * H] = gb;
    if (t < 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) loss = __fadd_rn(loss, __shfl_xor_sync(0xffffffffu, loss, o));
        if (t == 0) out[kParams] = loss;
    }
}
static_assert(oW2 % 4 == 0 && kPartRow % 4 == 0, "float4 stores of the W2 gradient");

// Sums the blocks' parts in a fixed order (warp w of eight: parts w, w + 8, ...;
// then the warps in order), one parameter a lane, and takes the Adam step
// (bias-corrected; the normalisation entries stay fixed), or with G stores the
// gradient.  The entry after the parameters is the loss.
struct AdamArgs {
    float lr, b1, b2, eps, c1, c2, wd;
};
__global__ void __launch_bounds__(MT)
mlp_update_kernel(const float *__restrict__ parts, int nparts, float *__restrict__ P,
                  float *__restrict__ Mo, float *__restrict__ Vo, AdamArgs A, float inv_norm,
                  float *__restrict__ loss, float *__restrict__ G)
{
    __shared__ float s[MT / 32][32];
    allow_dependent_launch();
    grid_dependency_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
    float g = 0.f;
    if (p <= kParams) {
#pragma unroll 16
        for (int b = w; b < nparts; b += MT / 32)
            g = __fadd_rn(g, __ldcg(parts + (size_t)b * kPartRow + p));
    }
    s[w][lane] = g;
    __syncthreads();
    if (w != 0 || p > kParams) return;
#pragma unroll
    for (int q = 1; q < MT / 32; ++q) g = __fadd_rn(g, s[q][lane]);
    if (p == kParams) {
        if (loss) *loss = __fmul_rn(g, inv_norm);
        return;
    }
    if (G) {
        G[p] = g;
        return;
    }
    if (p < oW1) return;
    const float q = P[p];
    g = __fmaf_rn(A.wd, q, g);
    const float m = __fmaf_rn(A.b1, Mo[p], __fmul_rn(1.f - A.b1, g));
    const float v = __fmaf_rn(A.b2, Vo[p], __fmul_rn(__fmul_rn(1.f - A.b2, g), g));
    Mo[p] = m;
    Vo[p] = v;
    const float mh = __fdiv_rn(m, A.c1), vh = __fdiv_rn(v, A.c2);
    P[p] = __fsub_rn(q, __fdiv_rn(__fmul_rn(A.lr, mh), __fadd_rn(__fsqrt_rn(vh), A.eps)));
}

// The class with the smallest predicted score (first on ties), per sample.
__global__ void mlp_argmin_kernel(const float *__restrict__ Y, int N, int *__restrict__ cls)
{
    const int nidx = blockIdx.x * blockDim.x + threadIdx.x;
    if (nidx >= N) return;
    int best = 0;
    for (int c = 1; c < C; ++c)
        if (Y[nidx * C + c] < Y[nidx * C + best]) best = c;
    cls[nidx] = best;
}

int blocks(long long work, int tpb) { return (int)((work + tpb - 1) / tpb); }

}  // namespace

void launch_features(const int *rp, const int *col, int m, int n, long long nnz,
                     unsigned long long *acc, float *feat, cudaStream_t s)
{
    cudaMemsetAsync(acc, 0, sizeof(unsigned long long) * kAcc, s);
    if (m > 0) {
        int g = blocks(m, 256);
        if (g > 148 * 8) g = 148 * 8;
        feature_acc_kernel<<<g, 256, 0, s>>>(rp, col, m, acc);
    }
    feature_final_kernel<<<1, 32, 0, s>>>(acc, m, n, nnz, feat);
}

void launch_mlp_forward(const float *P, const float *X, int N, float *Y, cudaStream_t s)
{
    if (N > 0) mlp_forward_kernel<<<blocks(N, kTile), MT, 0, s>>>(P, X, N, Y);
}

// At most this many blocks (one an SM) share the samples; the bound is fixed,
// so the order of the sums depends on N alone.
constexpr int kMaxParts = 148;
static int parts_of(int N) { return blocks(N, kTile) < kMaxParts ? blocks(N, kTile) : kMaxParts; }

size_t mlp_parts_floats(int N) { return (size_t)parts_of(N) * kPartRow; }

// Each of the two kernels is a programmatic dependent launch: its blocks are
// placed while the one before drains and wait in grid_dependency_wait().
template <typename... K, typename... Args>
static void launch_dependent(void (*kern)(K...), int grid, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(MT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, K(args)...);
}

void launch_mlp_grad(const float *P, const float *X, int N, const float *T, const float *W,
                     float inv_norm, float *parts, float *G, float *loss, cudaStream_t s)
{
    if (N <= 0) return;
    launch_dependent(mlp_step_kernel, parts_of(N), s, P, X, N, T, W, inv_norm, parts);
    launch_dependent(mlp_update_kernel, kPartRow / 32, s, parts, parts_of(N), nullptr, nullptr,
                     nullptr, AdamArgs{}, inv_norm, loss, G);
}

void launch_mlp_step(float *P, const float *X, int N, const float *T, const float *W,
                     float inv_norm, float *parts, float *M, float *V, int step, float lr, float wd,
                     float *loss, cudaStream_t s)
{
    if (N <= 0) return;
    const float b1 = 0.9f, b2 = 0.999f;
    const AdamArgs A{lr, b1, b2, 1e-8f, 1.f - powf(b1, (float)step), 1.f - powf(b2, (float)step), wd};
    launch_dependent(mlp_step_kernel, parts_of(N), s, P, X, N, T, W, inv_norm, parts);
    launch_dependent(mlp_update_kernel, kPartRow / 32, s, parts, parts_of(N), P, M, V, A, inv_norm,
                     loss, nullptr);
}

void launch_mlp_argmin(const float *Y, int N, int *cls, cudaStream_t s)
{
    if (N > 0) mlp_argmin_kernel<<<blocks(N, 128), 128, 0, s>>>(Y, N, cls);
}

}  // namespace sbb
