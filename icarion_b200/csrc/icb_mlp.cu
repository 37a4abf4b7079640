// icb_mlp.cu — training and evaluation of the learned deflection network
// (2 -> 64 -> 64 -> 1, tanh; parameter layout in icb_mlp.cuh).
//
// Training: Adam on the mean squared error, mini-batches drawn from a
// per-epoch permutation.  An Adam step is two launches: k_mlp_samples runs
// the forward and backward pass of every sample and leaves its activations
// and deltas, k_mlp_update forms every parameter's gradient from them and
// applies the step.  Gradients are summed as fixed chains (the 128 samples
// of a group in order, then the groups in order), so training is
// deterministic.  With bf16_forward the forward pass rounds weights and the
// first hidden layer to BF16 exactly as the collision path does
// (quantisation-aware; gradients pass straight through the rounding).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <random>
#include <string>
#include <vector>

#include "../../include/icarion_b200.h"
#include "icb_internal.h"
#include "icb_mlp.cuh"

namespace icb {

namespace {

constexpr int kGroup = 128;            // samples per gradient chain
constexpr int kSB = 16;                // samples per block of k_mlp_samples
constexpr int kSThreads = 256;         // (sample, 16 unit lanes)
constexpr int kWs = kMlpH + 4;         // shared-memory row stride (float4 aligned)
constexpr uint64_t kChunk = 128 * kGroup;   // samples per pair of launches (bounds the workspace)
constexpr int kUGroups = 8;            // groups whose chains run at once in k_mlp_update
constexpr int kUThreads = 128;         // W2 tile: (group, 4-row half, column); others: (group, unit)
constexpr int kUUnits = 16;            // units per block of the other parameters
constexpr int kUTiles2 = (kMlpH / 8) * (kMlpH / 8);              // 8 x 8 tiles of W2
constexpr int kUSlices = kMlpH / kUUnits;
constexpr int kUBlocks = kUTiles2 + 3 * kUSlices + 1;            // + W1 and b1, b2, W3; b3 and the loss

// What k_mlp_samples leaves for k_mlp_update: per sample a row of kRowLen
// floats, H1, H2, D2 = dL/d(pre-activation 2) and D1 (64 each), then four
// arrays of one value per sample: dout, the two inputs and the output error.
// The padding samples of the last group are zero.
constexpr int kRowH1 = 0, kRowH2 = kMlpH, kRowD2 = 2 * kMlpH, kRowD1 = 3 * kMlpH, kRowLen = 4 * kMlpH;
constexpr int kColDout = 0, kColX0 = 1, kColX1 = 2, kColErr = 3, kCols = 4;

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 :: "r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Loads of what the previous kernel of a programmatic launch chain wrote.
// That kernel may still run when this one starts, so the data is not
// read-only for this kernel's life: no const __restrict__ pointer (which
// allows the non-coherent path, and a load above the wait), but volatile
// ordinary loads, which stay behind cudaGridDependencySynchronize and see
// all that the kernels before it wrote.
__device__ __forceinline__ float ld_after(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_after2(const float* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_after4(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// Forward of one sample in FP32 arithmetic (optionally with BF16-rounded
// weights and first-layer activations); h1, h2 receive the activations.
template <bool BF16>
__device__ float mlp_forward_one(const float* w, float x0, float x1, float* h1, float* h2) {
    for (int c = 0; c < kMlpH; ++c) {
        float w0 = w[kMlpOffW1 + 2 * c], w1 = w[kMlpOffW1 + 2 * c + 1];
        if (BF16) { w0 = bf16r(w0); w1 = bf16r(w1); }
        float a = tanhf(fmaf(w0, x0, fmaf(w1, x1, w[kMlpOffB1 + c])));
        if (BF16) a = bf16r(a);
        h1[c] = a;
    }
    float y = w[kMlpOffB3];
    for (int n = 0; n < kMlpH; ++n) {
        float acc = 0.f;
        const float* row = w + kMlpOffW2 + n * kMlpH;
        for (int k = 0; k < kMlpH; ++k) acc = fmaf(BF16 ? bf16r(row[k]) : row[k], h1[k], acc);
        const float a = tanhf(acc + w[kMlpOffB2 + n]);
        h2[n] = a;
        y = fmaf(BF16 ? bf16r(w[kMlpOffW3 + n]) : w[kMlpOffW3 + n], a, y);
    }
    return y;
}

// Forward and backward pass of kSB samples per block: thread (sample s, lane
// q) holds units q, q + 16, q + 32, q + 48 of that sample in the forward
// layers and inputs 4q .. 4q + 3 in the backward product, so every
// shared-memory read is a conflict-free or broadcast float4.  Every sum is one
// FMA chain in unit order, the order of a serial evaluation (mlp_forward_one).
// Latency bound: a batch of 1,024 samples is 64 blocks of 8 warps, each a few
// dependent chains of 64 FMAs; 16 samples a block spread it over 64 SMs (one
// thread per sample in 8 blocks took 104 us).
template <bool BF16>
__global__ void __launch_bounds__(kSThreads) k_mlp_samples(const float* params,
                                                           const float* __restrict__ x, const float* __restrict__ y,
                                                           const uint32_t* __restrict__ perm, uint64_t first,
                                                           uint32_t count, float inv_batch, uint32_t ld,
                                                           float* __restrict__ rows, float* __restrict__ cols) {
    extern __shared__ __align__(16) float sm[];
    float* W2 = sm;                                    // [64][kWs] as stored
    float* W2r = BF16 ? W2 + kMlpH * kWs : W2;         // ... rounded for the forward pass
    float* H1 = W2r + kMlpH * kWs;                     // [kSB][kWs]
    float* H2 = H1 + kSB * kWs;
    float* D2 = H2 + kSB * kWs;
    float* w3 = D2 + kSB * kWs;                        // [64]
    float* dout = w3 + kMlpH;                          // [kSB]
    float* xs = dout + kSB;                            // [2][kSB]
    float* er = xs + 2 * kSB;                          // [kSB]
    const int tid = static_cast<int>(threadIdx.x);
    const int s = tid >> 4, q = tid & 15;
    const uint32_t local = blockIdx.x * kSB + static_cast<uint32_t>(s);
    const bool valid = local < count;
    float x0 = 0.f, x1 = 0.f, yt = 0.f;
    if (valid) {
        const uint32_t sidx = perm ? perm[first + local] : static_cast<uint32_t>(first + local);
        x0 = x[2 * static_cast<size_t>(sidx)];
        x1 = x[2 * static_cast<size_t>(sidx) + 1];
        yt = y[sidx];
    }
    // the previous step's update (the sample's loads above do not need it);
    // then the weights, all loads in flight together
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    float4 wv[kMlpH * kMlpH / 4 / kSThreads];
#pragma unroll
    for (int j = 0; j < kMlpH * kMlpH / 4 / kSThreads; ++j)
        wv[j] = ld_after4(params + kMlpOffW2 + 4 * (tid + j * kSThreads));
    float b1v[4], b2v[4];
    float2 w1v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = q + 16 * j;
        b1v[j] = ld_after(params + kMlpOffB1 + c);
        b2v[j] = ld_after(params + kMlpOffB2 + c);
        w1v[j] = ld_after2(params + kMlpOffW1 + 2 * c);
    }
    const float b3v = ld_after(params + kMlpOffB3);
    if (tid < kMlpH) w3[tid] = ld_after(params + kMlpOffW3 + tid);
#pragma unroll
    for (int j = 0; j < kMlpH * kMlpH / 4 / kSThreads; ++j) {
        const int e = 4 * (tid + j * kSThreads);
        const int o = (e >> 6) * kWs + (e & 63);
        *reinterpret_cast<float4*>(W2 + o) = wv[j];
        if (BF16)
            *reinterpret_cast<float4*>(W2r + o) = make_float4(bf16r(wv[j].x), bf16r(wv[j].y), bf16r(wv[j].z),
                                                              bf16r(wv[j].w));
    }
    if (q == 0) { xs[s] = x0; xs[kSB + s] = x1; }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = q + 16 * j;
        float w0 = w1v[j].x, w1 = w1v[j].y;
        if (BF16) { w0 = bf16r(w0); w1 = bf16r(w1); }
        float a = tanhf(fmaf(w0, x0, fmaf(w1, x1, b1v[j])));
        if (BF16) a = bf16r(a);
        H1[s * kWs + c] = valid ? a : 0.f;
    }
    __syncthreads();
    {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int k = 0; k < kMlpH; k += 4) {
            const float4 h = *reinterpret_cast<const float4*>(H1 + s * kWs + k);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(W2r + (q + 16 * j) * kWs + k);
                acc[j] = fmaf(w.x, h.x, acc[j]);
                acc[j] = fmaf(w.y, h.y, acc[j]);
                acc[j] = fmaf(w.z, h.z, acc[j]);
                acc[j] = fmaf(w.w, h.w, acc[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = q + 16 * j;
            const float a = tanhf(acc[j] + b2v[j]);
            H2[s * kWs + n] = valid ? a : 0.f;
        }
    }
    __syncthreads();
    if (q == 0) {
        float out = b3v;
#pragma unroll 4
        for (int n = 0; n < kMlpH; n += 4) {
            const float4 h = *reinterpret_cast<const float4*>(H2 + s * kWs + n);
            const float4 w = *reinterpret_cast<const float4*>(w3 + n);
            out = fmaf(BF16 ? bf16r(w.x) : w.x, h.x, out);
            out = fmaf(BF16 ? bf16r(w.y) : w.y, h.y, out);
            out = fmaf(BF16 ? bf16r(w.z) : w.z, h.z, out);
            out = fmaf(BF16 ? bf16r(w.w) : w.w, h.w, out);
        }
        const float e = valid ? out - yt : 0.f;
        er[s] = e;
        dout[s] = valid ? 2.f * e * inv_batch : 0.f;
    }
    __syncthreads();
    // D2[n] = dout W3[n] (1 - h2^2)
    {
        const float d = dout[s];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = q + 16 * j;
            const float a = H2[s * kWs + n];
            D2[s * kWs + n] = d * w3[n] * (1.f - a * a);
        }
    }
    __syncthreads();
    // D1[k] = (1 - h1^2) sum_n D2[n] W2[n][k]
    float4 d1v;
    {
        float d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int n = 0; n < kMlpH; n += 4) {
            const float4 dn = *reinterpret_cast<const float4*>(D2 + s * kWs + n);
            const float dv[4] = {dn.x, dn.y, dn.z, dn.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(W2 + (n + j) * kWs + 4 * q);
                d1[0] = fmaf(dv[j], w.x, d1[0]);
                d1[1] = fmaf(dv[j], w.y, d1[1]);
                d1[2] = fmaf(dv[j], w.z, d1[2]);
                d1[3] = fmaf(dv[j], w.w, d1[3]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float a = H1[s * kWs + 4 * q + j];
            d1[j] *= (1.f - a * a);
        }
        d1v = make_float4(d1[0], d1[1], d1[2], d1[3]);
    }
    const size_t c0 = static_cast<size_t>(blockIdx.x) * kSB;
    {
        float* r = rows + (c0 + static_cast<size_t>(s)) * kRowLen + 4 * q;
        const int o = s * kWs + 4 * q;
        *reinterpret_cast<float4*>(r + kRowH1) = *reinterpret_cast<const float4*>(H1 + o);
        *reinterpret_cast<float4*>(r + kRowH2) = *reinterpret_cast<const float4*>(H2 + o);
        *reinterpret_cast<float4*>(r + kRowD2) = *reinterpret_cast<const float4*>(D2 + o);
        *reinterpret_cast<float4*>(r + kRowD1) = d1v;
    }
    if (tid < kSB) {
        cols[static_cast<size_t>(kColDout) * ld + c0 + tid] = dout[tid];
        cols[static_cast<size_t>(kColX0) * ld + c0 + tid] = xs[tid];
        cols[static_cast<size_t>(kColX1) * ld + c0 + tid] = xs[kSB + tid];
        cols[static_cast<size_t>(kColErr) * ld + c0 + tid] = er[tid];
    }
}

struct AdamState {
    float lr, b1, b2, eps, c1, c2;   // c1 = 1/(1-b1^t), c2 = 1/(1-b2^t)
};

// Every parameter's gradient is one chain over the samples per group of
// kGroup samples (an FMA per sample, an add for a bias), then the groups'
// sums in order.  kUGroups groups run at once.  A block owns an 8 x 8 tile of
// W2 (8 columns of D2, 8 of H1), 16 units
// of W1 and b1, of b2 or of W3 (16 columns), or b3 and the sum of squared
// errors; the columns are staged in shared memory by asynchronous copies.  Chunks of a batch larger than
// kChunk carry their sums in gsum_buf and lsum_buf; on the last chunk the
// Adam step is applied (ADAM) or the gradient written.  Latency bound: a
// batch of 1,024 samples is one round of 128-step chains, spread so that no
// SM reads more than 72 KB of the samples' 1 MB (9.2 us with cold caches;
// reading the samples in place, strided, took 16 us, and unit-major rows 14.5).
template <bool ADAM>
__global__ void __launch_bounds__(kUThreads) k_mlp_update(const float* rows, const float* cols,
                                                          uint32_t ld, int ngroups,
                                                          int first_chunk, int last_chunk,
                                                          float* __restrict__ gsum_buf,
                                                          double* __restrict__ lsum_buf,
                                                          float* __restrict__ params, float* __restrict__ m,
                                                          float* __restrict__ v, AdamState a,
                                                          float* __restrict__ grad, double* __restrict__ loss_acc) {
    extern __shared__ __align__(16) float tile[];       // [kUGroups * kGroup][16]
    float* xcol = tile + kUGroups * kGroup * 16;        // [2][kUGroups * kGroup]
    __shared__ float part[3][kUGroups][64];
    __shared__ double lpart[kUGroups];
    const int tid = static_cast<int>(threadIdx.x), blk = static_cast<int>(blockIdx.x);
    // the parameters this thread sums and steps: up to one (three in the W1
    // and b1 blocks), p[c] < 0: none
    int p[3] = {-1, -1, -1};
    const bool w2 = blk < kUTiles2;
    const int n0 = (blk >> 3) * 8, k0 = (blk & 7) * 8;
    const int kind = w2 ? 0 : 1 + (blk - kUTiles2) / kUSlices;       // 1: W1, b1; 2: b2; 3: W3; 4: b3, loss
    const int u0 = w2 ? 0 : ((blk - kUTiles2) % kUSlices) * kUUnits;
    if (w2) {
        if (tid < 64) p[0] = kMlpOffW2 + (n0 + (tid >> 3)) * kMlpH + k0 + (tid & 7);
    } else if (kind == 1) {
        if (tid < kUUnits) {
            p[0] = kMlpOffW1 + 2 * (u0 + tid);
            p[1] = p[0] + 1;
            p[2] = kMlpOffB1 + u0 + tid;
        }
    } else if (kind == 2) {
        if (tid < kUUnits) p[0] = kMlpOffB2 + u0 + tid;
    } else if (kind == 3) {
        if (tid < kUUnits) p[0] = kMlpOffW3 + u0 + tid;
    } else if (tid == 0) {
        p[0] = kMlpOffB3;
    }
    // the samples kernel of this batch (and through it the previous step)
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    float gsum[3] = {0.f, 0.f, 0.f}, pm[3], pv[3], pp[3];
    double lsum = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (p[c] < 0) continue;
        if (!first_chunk) gsum[c] = gsum_buf[p[c]];
        if (ADAM && last_chunk) { pm[c] = m[p[c]]; pv[c] = v[p[c]]; pp[c] = params[p[c]]; }
    }
    if (kind == 4 && tid == 0 && !first_chunk) lsum = *lsum_buf;
    const int gi = tid / kUUnits, u = tid % kUUnits;
    // the 16 floats of a sample this block reads, as 4 float4: W2 tiles 8 of
    // D2 and 8 of H1, the others 16 units of D1, D2 or H2
    const int c4 = tid & 3;
    const int col = w2 ? (c4 < 2 ? kRowD2 + n0 + 4 * c4 : kRowH1 + k0 + 4 * (c4 - 2))
                       : (kind == 1 ? kRowD1 : kind == 2 ? kRowD2 : kRowH2) + u0 + 4 * c4;
    for (int g0 = 0; g0 < ngroups; g0 += kUGroups) {
        const int ng = min(kUGroups, ngroups - g0);
        if (kind < 4) {
            const float* src = rows + static_cast<size_t>(g0) * kGroup * kRowLen + col;
#pragma unroll 8
            for (int s = tid >> 2; s < ng * kGroup; s += kUThreads / 4)
                cp_async16(tile + s * 16 + 4 * c4, src + static_cast<size_t>(s) * kRowLen);
            if (kind != 2) {
                // the samples' inputs, or their dout
                const float* x0 = cols + static_cast<size_t>(kind == 1 ? kColX0 : kColDout) * ld +
                                  static_cast<size_t>(g0) * kGroup;
                const float* x1 = cols + static_cast<size_t>(kColX1) * ld + static_cast<size_t>(g0) * kGroup;
                for (int s = 4 * tid; s < ng * kGroup; s += 4 * kUThreads) {
                    cp_async16(xcol + s, x0 + s);
                    if (kind == 1) cp_async16(xcol + kUGroups * kGroup + s, x1 + s);
                }
            }
            cp_async_wait_all();
            __syncthreads();
        }
        if (w2) {
            const int h = (tid >> 3) & 1, k = tid & 7;
            if (gi < ng) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                const float* t = tile + gi * kGroup * 16;
#pragma unroll 16
                for (int s = 0; s < kGroup; ++s) {
                    const float4 d = *reinterpret_cast<const float4*>(t + s * 16 + 4 * h);
                    const float b = t[s * 16 + 8 + k];
                    acc[0] = fmaf(d.x, b, acc[0]);
                    acc[1] = fmaf(d.y, b, acc[1]);
                    acc[2] = fmaf(d.z, b, acc[2]);
                    acc[3] = fmaf(d.w, b, acc[3]);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) part[0][gi][(4 * h + j) * 8 + k] = acc[j];
            }
        } else if (kind < 4) {
            if (gi < ng) {
                const float* t = tile + gi * kGroup * 16 + u;
                const float* x0 = xcol + gi * kGroup;
                const float* x1 = x0 + kUGroups * kGroup;
                float a0 = 0.f, a1 = 0.f, ab = 0.f;
                if (kind == 1) {
#pragma unroll 16
                    for (int s = 0; s < kGroup; ++s) {
                        const float d = t[s * 16];
                        a0 = fmaf(d, x0[s], a0);
                        a1 = fmaf(d, x1[s], a1);
                        ab += d;
                    }
                } else if (kind == 2) {
#pragma unroll 16
                    for (int s = 0; s < kGroup; ++s) ab += t[s * 16];
                } else {
#pragma unroll 16
                    for (int s = 0; s < kGroup; ++s) a0 = fmaf(x0[s], t[s * 16], a0);
                }
                part[0][gi][u] = kind == 2 ? ab : a0;
                part[1][gi][u] = a1;
                part[2][gi][u] = ab;
            }
        } else if (tid < 2 * kUGroups) {
            const int b = tid >> 1;
            if (b < ng) {
                const float* e1 = cols + static_cast<size_t>((tid & 1) ? kColErr : kColDout) * ld +
                                  static_cast<size_t>(g0 + b) * kGroup;
                float acc = 0.f;
                double lacc = 0.0;
#pragma unroll 32
                for (int s = 0; s < kGroup / 4; ++s) {
                    const float4 e = ld_after4(e1 + 4 * s);
                    if (tid & 1) {
                        lacc += static_cast<double>(e.x) * e.x;
                        lacc += static_cast<double>(e.y) * e.y;
                        lacc += static_cast<double>(e.z) * e.z;
                        lacc += static_cast<double>(e.w) * e.w;
                    } else {
                        acc += e.x; acc += e.y; acc += e.z; acc += e.w;
                    }
                }
                if (tid & 1) lpart[b] = lacc;
                else part[0][b][0] = acc;
            }
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (p[c] >= 0)
                for (int b = 0; b < ng; ++b) gsum[c] += part[c][b][tid];
        if (kind == 4 && tid == 0)
            for (int b = 0; b < ng; ++b) lsum += lpart[b];
        __syncthreads();
    }
    if (kind == 4 && tid == 0) {
        if (last_chunk) *loss_acc += lsum;
        else *lsum_buf = lsum;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (p[c] < 0) continue;
        if (!last_chunk) {
            gsum_buf[p[c]] = gsum[c];
        } else if (ADAM) {
            // written as the fused operations they are rounded as
            const float mm = fmaf(1.f - a.b1, gsum[c], a.b1 * pm[c]);
            const float vv = fmaf((1.f - a.b2) * gsum[c], gsum[c], a.b2 * pv[c]);
            m[p[c]] = mm;
            v[p[c]] = vv;
            pp[c] -= a.lr * (mm * a.c1) / (sqrtf(vv * a.c2) + a.eps);
            params[p[c]] = pp[c];
        } else {
            grad[p[c]] = gsum[c];
        }
    }
}

__global__ void k_mlp_forward_fp32(const float* __restrict__ params, uint64_t n, const float* __restrict__ x,
                                   float* __restrict__ y) {
    __shared__ float w[kMlpParams];
    for (int k = threadIdx.x; k < kMlpParams; k += blockDim.x) w[k] = params[k];
    __syncthreads();
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float h1[kMlpH], h2[kMlpH];
    y[i] = mlp_forward_one<false>(w, x[2 * i], x[2 * i + 1], h1, h2);
}

// The collision path's evaluation: each warp takes 32 consecutive samples.
__global__ void k_mlp_forward_mma(const uint32_t* __restrict__ frag, const float* __restrict__ f, uint64_t n,
                                  const float* __restrict__ x, float* __restrict__ y) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool want = i < n;
    const float x0 = want ? x[2 * i] : 0.f, x1 = want ? x[2 * i + 1] : 0.f;
    const float out = mlp_warp_eval(frag, f, x0, x1, want);
    if (want) y[i] = out;
}

float bf16_round_host(float x) {
    uint32_t u;
    std::memcpy(&u, &x, 4);
    if ((u & 0x7f800000u) == 0x7f800000u) return x;       // inf / nan unchanged
    const uint32_t lsb = (u >> 16) & 1u;
    u += 0x7fffu + lsb;                                    // round to nearest even
    u &= 0xffff0000u;
    float r;
    std::memcpy(&r, &u, 4);
    return r;
}

uint32_t bf16_bits_host(float x) {
    const float r = bf16_round_host(x);
    uint32_t u;
    std::memcpy(&u, &r, 4);
    return u >> 16;
}

template <class T>
struct DevVec {
    T* p = nullptr;
    ~DevVec() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t n) { return cudaMalloc(reinterpret_cast<void**>(&p), std::max<size_t>(n, 1) * sizeof(T)); }
};

}  // namespace

// Pool for the memory of one-shot calls.  cudaMalloc and cudaFree of a call's
// workspace cost 0.6 ms on the host, more than half of a short training run;
// the pool hands the same memory to the next call in a few microseconds.  It
// keeps at most kCallPoolKeep bytes per device between calls (the driver
// releases the rest when a stream is synchronised after a free: each call
// does so last), belongs to no handle, and is safe with several threads and
// streams: allocations are stream ordered and the driver orders their reuse.
// Null when the device has no pools or the creation fails (the caller then
// allocates plainly).  A device reset takes the pool with its context: it is
// used only in the context it was made in, known by the context's id.
constexpr uint64_t kCallPoolKeep = 32ull << 20;
static cudaMemPool_t call_pool(int device) {
    static std::mutex m;
    static cudaMemPool_t pools[64] = {};
    static unsigned long long ctxs[64] = {};
    if (device < 0 || device >= 64) return nullptr;
    const unsigned long long ctx = current_context_id();
    if (ctx == 0) return nullptr;
    std::lock_guard<std::mutex> lock(m);
    if (pools[device] && ctxs[device] == ctx) return pools[device];
    pools[device] = nullptr;
    uint64_t keep = kCallPoolKeep;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();
        if (pool) cudaMemPoolDestroy(pool);
        return nullptr;
    }
    pools[device] = pool;
    ctxs[device] = ctx;
    return pool;
}

// Collision-path parameter blocks: B fragments of W2 (BF16 pairs) and the
// float block (W1, W3 rounded to BF16; biases FP32).
void mlp_pack(const float* params, std::vector<uint32_t>& frag, std::vector<float>& fblock) {
    frag.assign(kMlpFragWords, 0u);
    // W2 as A fragments of m-tile mt (units 16mt..16mt+15) and k-step ks
    auto pair = [&](int n, int k) {
        const float* row = params + kMlpOffW2 + n * kMlpH;
        return bf16_bits_host(row[k]) | (bf16_bits_host(row[k + 1]) << 16);
    };
    for (int mt = 0; mt < 4; ++mt)
        for (int ks = 0; ks < 4; ++ks)
            for (int lane = 0; lane < 32; ++lane) {
                const int g = lane >> 2, t = lane & 3;
                const int n0 = 16 * mt + g, n1 = n0 + 8;
                const int k0 = 16 * ks + 2 * t, k1 = k0 + 8;
                const size_t base = (static_cast<size_t>(mt * 4 + ks) * 32 + lane) * 4;
                frag[base] = pair(n0, k0);
                frag[base + 1] = pair(n1, k0);
                frag[base + 2] = pair(n0, k1);
                frag[base + 3] = pair(n1, k1);
            }
    // layer 1 as A fragments: rows h of [W1[h][0] twice, W1[h][1] twice,
    // b1[h] hi, b1[h] lo, 0 ...], words for rows 16mt+g and 16mt+g+8
    auto l1 = [&](int h, int t) {
        if (t < 2) {
            const uint32_t b = bf16_bits_host(params[kMlpOffW1 + 2 * h + t]);
            return b | (b << 16);
        }
        if (t == 2) {
            const float b1 = params[kMlpOffB1 + h];
            const float hi = bf16_round_host(b1);
            return bf16_bits_host(hi) | (bf16_bits_host(b1 - hi) << 16);
        }
        return 0u;
    };
    for (int mt = 0; mt < 4; ++mt)
        for (int lane = 0; lane < 32; ++lane) {
            const int g = lane >> 2, t = lane & 3;
            const size_t base = static_cast<size_t>(kMlpFragW1Off) + (static_cast<size_t>(mt) * 32 + lane) * 2;
            frag[base] = l1(16 * mt + g, t);
            frag[base + 1] = l1(16 * mt + g + 8, t);
        }
    fblock.assign(kMlpFSize, 0.f);
    for (int k = 0; k < 128; ++k) fblock[kMlpFW1 + k] = bf16_round_host(params[kMlpOffW1 + k]);
    for (int k = 0; k < kMlpH; ++k) {
        fblock[kMlpFB1 + k] = params[kMlpOffB1 + k];
        fblock[kMlpFB2 + k] = params[kMlpOffB2 + k];
        fblock[kMlpFW3 + k] = bf16_round_host(params[kMlpOffW3 + k]);
    }
    fblock[kMlpFB3] = params[kMlpOffB3];
}

}  // namespace icb

using namespace icb;

template <class K>
static cudaError_t smem_attr(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

#define MLP_CUDA(expr)                                                                   \
    do {                                                                                 \
        cudaError_t e_ = (expr);                                                         \
        if (e_ != cudaSuccess) {                                                         \
            return set_error(e_ == cudaErrorMemoryAllocation ? ICB_ERR_OUT_OF_MEMORY : ICB_ERR_CUDA, \
                             (std::string(#expr) + ": " + cudaGetErrorString(e_)).c_str());        \
        }                                                                                \
    } while (0)

extern "C" {

int icb_mlp_init(uint64_t seed, float* params) {
    if (!params) return set_error(ICB_ERR_INVALID_ARGUMENT, "null params");
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    std::fill(params, params + kMlpParams, 0.f);
    const double a1 = std::sqrt(6.0 / (2 + kMlpH)), a2 = std::sqrt(6.0 / (kMlpH + kMlpH)), a3 = std::sqrt(6.0 / (kMlpH + 1));
    for (int k = 0; k < 128; ++k) params[kMlpOffW1 + k] = static_cast<float>(a1 * u(rng));
    for (int k = 0; k < kMlpH * kMlpH; ++k) params[kMlpOffW2 + k] = static_cast<float>(a2 * u(rng));
    for (int k = 0; k < kMlpH; ++k) params[kMlpOffW3 + k] = static_cast<float>(a3 * u(rng));
    return ICB_OK;
}

// Memory of one training or gradient call from the library's pool of the
// device (call_pool), stream ordered; plain device memory where there is none.
struct CallMem {
    unsigned char* p = nullptr;
    cudaStream_t s = nullptr;
    bool pooled = false;
    ~CallMem() {
        if (!p) return;
        if (!pooled) {
            cudaFree(p);
            return;
        }
        // the pool gives back what it holds above its bound at a
        // synchronisation after the free; the call's work is done by now
        cudaFreeAsync(p, s);
        cudaStreamSynchronize(s);
    }
    cudaError_t alloc(size_t bytes, int device, cudaStream_t stream) {
        s = stream;
        if (cudaMemPool_t pool = call_pool(device)) {
            if (cudaMallocFromPoolAsync(reinterpret_cast<void**>(&p), bytes, pool, s) == cudaSuccess) {
                pooled = true;
                return cudaSuccess;
            }
            cudaGetLastError();
            p = nullptr;
        }
        return cudaMalloc(reinterpret_cast<void**>(&p), bytes);
    }
};

// Device workspace of one training or gradient call, one allocation: the
// samples, the parameter state, the permutation and the rows of one chunk.
struct MlpWork {
    CallMem mem;
    float *x = nullptr, *y = nullptr, *params = nullptr, *m = nullptr, *v = nullptr, *gsum = nullptr, *rows = nullptr,
          *cols = nullptr;
    uint32_t* perm = nullptr;
    double *lsum = nullptr, *loss = nullptr;
    uint32_t ld = 0;
    cudaError_t alloc(uint64_t n, uint64_t batch, bool with_perm, int device, cudaStream_t stream) {
        const uint64_t chunk = std::min<uint64_t>(batch, kChunk);
        ld = static_cast<uint32_t>((chunk + kGroup - 1) / kGroup * kGroup);
        size_t at = 0;
        auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~size_t(255); return o; };
        const size_t ox = take(2 * n * sizeof(float)), oy = take(n * sizeof(float));
        const size_t op = take(kMlpParams * sizeof(float)), om = take(kMlpParams * sizeof(float));
        const size_t ov = take(kMlpParams * sizeof(float)), og = take(kMlpParams * sizeof(float));
        const size_t orow = take(static_cast<size_t>(kRowLen) * ld * sizeof(float));
        const size_t ocol = take(static_cast<size_t>(kCols) * ld * sizeof(float));
        const size_t operm = take(with_perm ? n * sizeof(uint32_t) : 0);
        const size_t ol = take(2 * sizeof(double));
        const cudaError_t e = mem.alloc(at, device, stream);
        if (e != cudaSuccess) return e;
        x = reinterpret_cast<float*>(mem.p + ox);
        y = reinterpret_cast<float*>(mem.p + oy);
        params = reinterpret_cast<float*>(mem.p + op);
        m = reinterpret_cast<float*>(mem.p + om);
        v = reinterpret_cast<float*>(mem.p + ov);
        gsum = reinterpret_cast<float*>(mem.p + og);
        rows = reinterpret_cast<float*>(mem.p + orow);
        cols = reinterpret_cast<float*>(mem.p + ocol);
        perm = with_perm ? reinterpret_cast<uint32_t*>(mem.p + operm) : nullptr;
        lsum = reinterpret_cast<double*>(mem.p + ol);
        loss = lsum + 1;
        return cudaSuccess;
    }
};

static size_t samples_smem(bool bf16) {
    return (static_cast<size_t>(bf16 ? 2 : 1) * kMlpH * kWs + 3 * kSB * kWs + kMlpH + 4 * kSB) * sizeof(float);
}

constexpr size_t kUpdateSmem = static_cast<size_t>(kUGroups) * kGroup * (16 + 2) * sizeof(float);

static cudaError_t batch_attrs(bool bf16, bool adam) {
    const cudaError_t e = bf16 ? smem_attr(k_mlp_samples<true>, samples_smem(true))
                               : smem_attr(k_mlp_samples<false>, samples_smem(false));
    if (e != cudaSuccess) return e;
    return adam ? smem_attr(k_mlp_update<true>, kUpdateSmem) : smem_attr(k_mlp_update<false>, kUpdateSmem);
}

// Gradient of the mean squared error over `count` samples from `first` on
// (through w.perm when set), followed by the Adam step or the store to grad.
static int launch_batch(bool bf16, bool adam, const MlpWork& w, uint64_t first, uint64_t count, const AdamState& a,
                        float* grad, cudaStream_t s) {
    const float inv_batch = 1.f / static_cast<float>(count);
    const size_t smem = samples_smem(bf16);
    for (uint64_t c = 0; c < count; c += kChunk) {
        const uint32_t nc = static_cast<uint32_t>(std::min<uint64_t>(kChunk, count - c));
        const int ngroups = static_cast<int>((nc + kGroup - 1) / kGroup);
        const unsigned blocks = static_cast<unsigned>(ngroups * (kGroup / kSB));
        // programmatic launches: each kernel's start overlaps the end of the
        // one before it, whose results it waits for itself
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(blocks);
        lc.blockDim = dim3(kSThreads);
        lc.dynamicSmemBytes = smem;
        lc.stream = s;
        lc.attrs = &at;
        lc.numAttrs = 1;
        const uint32_t* perm = w.perm;
        const float *px = w.x, *py = w.y, *pw = w.params;
        MLP_CUDA(cudaLaunchKernelEx(&lc, bf16 ? k_mlp_samples<true> : k_mlp_samples<false>, pw, px, py, perm,
                                    first + c, nc, inv_batch, w.ld, w.rows, w.cols));
        lc.gridDim = dim3(kUBlocks);
        lc.blockDim = dim3(kUThreads);
        lc.dynamicSmemBytes = kUpdateSmem;
        const float *rows = w.rows, *cols = w.cols;
        MLP_CUDA(cudaLaunchKernelEx(&lc, adam ? k_mlp_update<true> : k_mlp_update<false>, rows, cols, w.ld, ngroups,
                                    static_cast<int>(c == 0), static_cast<int>(c + nc == count), w.gsum, w.lsum,
                                    w.params, w.m, w.v, a, grad, w.loss));
    }
    return ICB_OK;
}

int icb_mlp_train(int device, const icb_mlp_train_config* cfg, uint64_t n, const float* x, const float* y,
                  float* params, double* loss_per_epoch) {
    if (!cfg || !x || !y || !params) return set_error(ICB_ERR_INVALID_ARGUMENT, "null argument");
    if (cfg->epochs < 1 || cfg->batch < 1 || cfg->batch > (1 << 20) || n < static_cast<uint64_t>(cfg->batch) ||
        n >= (1ull << 32))
        return set_error(ICB_ERR_INVALID_ARGUMENT, "need epochs >= 1, 1 <= batch <= min(n, 2^20), n < 2^32");
    if (!(cfg->lr > 0.0) || !(cfg->lr_min >= 0.0)) return set_error(ICB_ERR_INVALID_ARGUMENT, "bad learning rate");
    MLP_CUDA(cudaSetDevice(device));
    cudaStream_t s = nullptr;
    MLP_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamGuard { cudaStream_t s; ~StreamGuard() { cudaStreamDestroy(s); } } guard{s};
    const uint32_t B = static_cast<uint32_t>(cfg->batch);
    const bool bf16 = cfg->bf16_forward != 0;
    MlpWork w;
    MLP_CUDA(w.alloc(n, B, true, device, s));
    MLP_CUDA(batch_attrs(bf16, true));
    MLP_CUDA(cudaMemcpyAsync(w.x, x, 2 * n * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_CUDA(cudaMemcpyAsync(w.y, y, n * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_CUDA(cudaMemcpyAsync(w.params, params, kMlpParams * sizeof(float), cudaMemcpyHostToDevice, s));
    MLP_CUDA(cudaMemsetAsync(w.m, 0, kMlpParams * sizeof(float), s));
    MLP_CUDA(cudaMemsetAsync(w.v, 0, kMlpParams * sizeof(float), s));
    std::vector<uint32_t> perm(n);
    std::iota(perm.begin(), perm.end(), 0u);
    std::mt19937_64 rng(cfg->seed ^ 0x9e3779b97f4a7c15ull);
    const uint64_t steps_per_epoch = n / B;
    const uint64_t total = steps_per_epoch * static_cast<uint64_t>(cfg->epochs);
    const double b1 = 0.9, b2 = 0.999;
    double b1t = 1.0, b2t = 1.0;
    uint64_t step = 0;
    // Fisher-Yates with the generator's raw 64-bit output
    auto shuffle = [&] {
        for (uint64_t i = n - 1; i > 0; --i) {
            const uint64_t j = rng() % (i + 1);
            std::swap(perm[i], perm[j]);
        }
    };
    shuffle();
    for (int ep = 0; ep < cfg->epochs; ++ep) {
        MLP_CUDA(cudaMemcpyAsync(w.perm, perm.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
        MLP_CUDA(cudaMemsetAsync(w.loss, 0, sizeof(double), s));
        for (uint64_t k = 0; k < steps_per_epoch; ++k, ++step) {
            b1t *= b1;
            b2t *= b2;
            const double frac = static_cast<double>(step) / static_cast<double>(total);
            const double lr = cfg->lr_min + 0.5 * (cfg->lr - cfg->lr_min) * (1.0 + std::cos(M_PI * frac));
            AdamState a{static_cast<float>(lr), static_cast<float>(b1), static_cast<float>(b2), 1e-8f,
                        static_cast<float>(1.0 / (1.0 - b1t)), static_cast<float>(1.0 / (1.0 - b2t))};
            if (int r = launch_batch(bf16, true, w, k * B, B, a, nullptr, s)) return r;
        }
        // the next epoch's permutation while the device trains this one (the
        // copy above returned with the host array read)
        if (ep + 1 < cfg->epochs) shuffle();
        double l = 0.0;
        MLP_CUDA(cudaMemcpyAsync(&l, w.loss, sizeof(double), cudaMemcpyDeviceToHost, s));
        MLP_CUDA(cudaStreamSynchronize(s));
        if (loss_per_epoch) loss_per_epoch[ep] = l / static_cast<double>(steps_per_epoch * B);
    }
    MLP_CUDA(cudaMemcpyAsync(params, w.params, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost, s));
    MLP_CUDA(cudaStreamSynchronize(s));
    return ICB_OK;
}

int icb_mlp_forward(int device, const float* params, uint64_t n, const float* x, float* y, int mode) {
    if (!params || (n > 0 && (!x || !y))) return set_error(ICB_ERR_INVALID_ARGUMENT, "null argument");
    if (mode != 0 && mode != 1) return set_error(ICB_ERR_INVALID_ARGUMENT, "mode must be 0 (FP32) or 1 (BF16 MMA)");
    if (n == 0) return ICB_OK;
    MLP_CUDA(cudaSetDevice(device));
    DevVec<float> dx, dy, dp, df;
    DevVec<uint32_t> dfrag;
    MLP_CUDA(dx.alloc(2 * n));
    MLP_CUDA(dy.alloc(n));
    MLP_CUDA(cudaMemcpy(dx.p, x, 2 * n * sizeof(float), cudaMemcpyHostToDevice));
    const unsigned blocks = static_cast<unsigned>((n + 127) / 128);
    if (mode == 0) {
        MLP_CUDA(dp.alloc(kMlpParams));
        MLP_CUDA(cudaMemcpy(dp.p, params, kMlpParams * sizeof(float), cudaMemcpyHostToDevice));
        k_mlp_forward_fp32<<<blocks, 128>>>(dp.p, n, dx.p, dy.p);
    } else {
        std::vector<uint32_t> frag;
        std::vector<float> fb;
        mlp_pack(params, frag, fb);
        MLP_CUDA(dfrag.alloc(frag.size()));
        MLP_CUDA(df.alloc(fb.size()));
        MLP_CUDA(cudaMemcpy(dfrag.p, frag.data(), frag.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
        MLP_CUDA(cudaMemcpy(df.p, fb.data(), fb.size() * sizeof(float), cudaMemcpyHostToDevice));
        k_mlp_forward_mma<<<blocks, 128>>>(dfrag.p, df.p, n, dx.p, dy.p);
    }
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaMemcpy(y, dy.p, n * sizeof(float), cudaMemcpyDeviceToHost));
    return ICB_OK;
}

int icb_mlp_gradients(int device, const float* params, uint64_t n, const float* x, const float* y, float* grad,
                      double* loss) {
    if (!params || !x || !y || !grad) return set_error(ICB_ERR_INVALID_ARGUMENT, "null argument");
    if (n == 0 || n > (1u << 20)) return set_error(ICB_ERR_INVALID_ARGUMENT, "need 1 <= n <= 2^20");
    MLP_CUDA(cudaSetDevice(device));
    MlpWork w;
    MLP_CUDA(w.alloc(n, n, false, device, nullptr));
    float* const dg = w.m;           // no Adam state in this call
    MLP_CUDA(batch_attrs(false, false));
    MLP_CUDA(cudaMemcpy(w.x, x, 2 * n * sizeof(float), cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemcpy(w.y, y, n * sizeof(float), cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemcpy(w.params, params, kMlpParams * sizeof(float), cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemset(w.loss, 0, sizeof(double)));
    if (int r = launch_batch(false, false, w, 0, n, AdamState{}, dg, nullptr)) return r;
    MLP_CUDA(cudaMemcpy(grad, dg, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost));
    double l = 0.0;
    MLP_CUDA(cudaMemcpy(&l, w.loss, sizeof(double), cudaMemcpyDeviceToHost));
    if (loss) *loss = l / static_cast<double>(n);
    return ICB_OK;
}

}  // extern "C"
