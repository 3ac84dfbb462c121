// Learned search budget: a 256 -> 256 -> 256 -> 2 MLP (GELU) with BF16 weights,
// trained and run on the device with the kernels below.
//
//   GEMMs: Y = X W^T + b (forward), dX = dY W, dW = dY^T X (backward); both
//   operands are rounded to BF16 (round to nearest) as they are staged, products
//   are accumulated in FP32.  The two 256 x 256 forward layers run on the tensor
//   cores (tcgen05, mlp_tc.cu, GELU in the epilogue); the 2-output layer and the
//   backward GEMMs on the CUDA cores (shared-memory tiles).  Master
//   weights and Adam state are FP32.  Loss: binary cross-entropy with logits on
//   both outputs.
//
// The two outputs are the logits of "the query's answer is complete with budget
// level 0" and "... with level 1" (the levels are set by hrnn_set_budget); the
// search takes the cheapest level whose probability reaches the confidence
// cutoff and falls back to the caller's (m, ef) otherwise.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

#include "index.hpp"
#include "mlp.hpp"
#include "mlp_ranges.hpp"

namespace hrnn {

namespace {

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

constexpr int kTile = 64;  // GEMM tiles (kTileK deep); 256 threads, 4 x 4 outputs each

// Z[M x 2] = A[M x 256] W^T + b (W [2 x 256]): a thread sums one row's both outputs over
// k in order.  Rows are staged 32 columns at a time so the loads stay coalesced.
__global__ void __launch_bounds__(64) k_out_layer(const float* __restrict__ A, const float* __restrict__ W,
                                                  const float* __restrict__ bias, float* __restrict__ Z, int M) {
    __shared__ float As[64][33];
    __shared__ float Ws[kMlpOut][kMlpH];
    const int t = threadIdx.x, m0 = blockIdx.x * 64;
    for (int i = t; i < kMlpOut * kMlpH; i += 64) Ws[i / kMlpH][i % kMlpH] = bf16r(W[i]);
    float z0 = 0.f, z1 = 0.f;
    for (int k0 = 0; k0 < kMlpH; k0 += 32) {
        __syncthreads();
#pragma unroll 8
        for (int r = t >> 3; r < 64; r += 8) {
            const int c = (t & 7) * 4;
            const float4 v = m0 + r < M ? __ldg(reinterpret_cast<const float4*>(A + (size_t)(m0 + r) * kMlpH + k0 + c))
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
            As[r][c] = bf16r(v.x);
            As[r][c + 1] = bf16r(v.y);
            As[r][c + 2] = bf16r(v.z);
            As[r][c + 3] = bf16r(v.w);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const float a = As[t][k];
            z0 = fmaf(a, Ws[0][k0 + k], z0);
            z1 = fmaf(a, Ws[1][k0 + k], z1);
        }
    }
    if (m0 + t < M) {
        Z[2 * (m0 + t)] = z0 + bias[0];
        Z[2 * (m0 + t) + 1] = z1 + bias[1];
    }
}

__device__ __forceinline__ float gelu_d(float x) {
    return 0.5f * (1.f + erff(x * 0.70710678f)) + x * 0.39894228f * expf(-0.5f * x * x);
}

// xn = (x - mean) * inv, per input feature (plain IEEE FP32 subtract and multiply).
__global__ void k_normalize(const float* __restrict__ x, const float* __restrict__ nrm, float* __restrict__ xn,
                            size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const int f = (int)(i % kMlpIn);
        xn[i] = __fmul_rn(__fsub_rn(x[i], nrm[f]), nrm[kMlpIn + f]);
    }
}

// dZ3 = (sigmoid(z) - y) / B for both outputs (loss accumulated in *loss), and through
// the output layer and GELU: G2 = (dZ3 W3) gelu'(Z2).  One block per 16 rows.
__global__ void __launch_bounds__(256) k_bce_back(const float* __restrict__ z3, const uint8_t* __restrict__ y,
                                                  const float* __restrict__ W3, const float* __restrict__ z2,
                                                  float* __restrict__ g3, float* __restrict__ g2, int B,
                                                  float* __restrict__ loss) {
    __shared__ float gs[32];
    const int t = threadIdx.x, m0 = blockIdx.x * 16;
    if (t < 32) {
        const int i = 2 * m0 + t;
        float l = 0.f, g = 0.f;
        if (i < 2 * B) {
            const float u = y[i] ? 1.f : 0.f, x = z3[i];
            const float s = 1.f / (1.f + expf(-x));
            g = (s - u) / (float)B;
            g3[i] = g;
            l = (fmaxf(x, 0.f) - x * u + log1pf(expf(-fabsf(x)))) / (float)B;
        }
        gs[t] = bf16r(g);
        for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xFFFFFFFFu, l, o);
        if (t == 0) atomicAdd(loss, l);
    }
    __syncthreads();
    const float w0 = bf16r(W3[t]), w1 = bf16r(W3[kMlpH + t]);
#pragma unroll 4
    for (int r = 0; r < 16; ++r)
        if (m0 + r < B) {
            const size_t i = (size_t)(m0 + r) * kMlpH + t;
            g2[i] = fmaf(gs[2 * r + 1], w1, fmaf(gs[2 * r], w0, 0.f)) * gelu_d(z2[i]);
        }
}

// G1[M x 256] = (G2[M x 256] W2[256 x 256]) gelu'(Z1); every output sums over k in order.
__global__ void __launch_bounds__(256) k_back_layer(const float* __restrict__ G2, const float* __restrict__ W2,
                                                    const float* __restrict__ z1, float* __restrict__ G1, int M) {
    __shared__ float As[kTileK][kTile + 4], Bs[kTileK][kTile];
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4, m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < kMlpH; k0 += kTileK) {
        const int ar = t >> 2, ac = (t & 3) * 4, br = t >> 4, bc = (t & 15) * 4;
        const float4 a = m0 + ar < M ? __ldg(reinterpret_cast<const float4*>(G2 + (size_t)(m0 + ar) * kMlpH + k0 + ac))
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 b = __ldg(reinterpret_cast<const float4*>(W2 + (size_t)(k0 + br) * kMlpH + n0 + bc));
        __syncthreads();
        As[ac][ar] = bf16r(a.x);
        As[ac + 1][ar] = bf16r(a.y);
        As[ac + 2][ar] = bf16r(a.z);
        As[ac + 3][ar] = bf16r(a.w);
        *reinterpret_cast<float4*>(&Bs[br][bc]) = make_float4(bf16r(b.x), bf16r(b.y), bf16r(b.z), bf16r(b.w));
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTileK; ++k) {
            const float4 u = *reinterpret_cast<const float4*>(&As[k][4 * ty]);
            const float4 w = *reinterpret_cast<const float4*>(&Bs[k][4 * tx]);
            const float uu[4] = {u.x, u.y, u.z, u.w}, ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(uu[i], ww[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (m0 + 4 * ty + i < M)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const size_t o = (size_t)(m0 + 4 * ty + i) * kMlpH + n0 + 4 * tx + j;
                G1[o] = acc[i][j] * gelu_d(z1[o]);
            }
}

// Weight gradients dW = G^T X (both [B x 256]) and bias gradients db = sum_b G, as
// partial sums over ranges of `per` rows (one per blockIdx.z; even layer first, then
// the other), 64 x 64 outputs per block; k_sum_parts adds the ranges.  One block per
// 32 x 32 outputs going through all rows left most of the device idle: 1,080 us at
// B = 4096 (and 590 us for the column sums, one block), now 40 us for both and 13 for
// the summing pass.
struct WGrad {
    const float *g, *x;
};
constexpr size_t kPartW = (size_t)kMlpH * kMlpIn, kPart = kPartW + kMlpH;  // floats of one range

__global__ void __launch_bounds__(256) k_weight_grad(WGrad l0, WGrad l1, int B, int per, int ranges,
                                                     float* __restrict__ part) {
    __shared__ float As[kTileK][kTile], Bs[kTileK][kTile];
    __shared__ float cs[16][kTile];
    const int layer = blockIdx.z / ranges, z = blockIdx.z % ranges;
    const float* __restrict__ g = layer ? l1.g : l0.g;
    const float* __restrict__ x = layer ? l1.x : l0.x;
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4, m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    const int b0 = z * per, b1 = min(B, b0 + per);
    float acc[4][4] = {};
    float col[4] = {};
    const int c = (t & 15) * 4, r = t >> 4;
    for (int k0 = b0; k0 < b1; k0 += kTileK) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (k0 + r < b1) {
            a = __ldg(reinterpret_cast<const float4*>(g + (size_t)(k0 + r) * kMlpH + m0 + c));
            b = __ldg(reinterpret_cast<const float4*>(x + (size_t)(k0 + r) * kMlpH + n0 + c));
        }
        col[0] += a.x;
        col[1] += a.y;
        col[2] += a.z;
        col[3] += a.w;
        __syncthreads();
        *reinterpret_cast<float4*>(&As[r][c]) = make_float4(bf16r(a.x), bf16r(a.y), bf16r(a.z), bf16r(a.w));
        *reinterpret_cast<float4*>(&Bs[r][c]) = make_float4(bf16r(b.x), bf16r(b.y), bf16r(b.z), bf16r(b.w));
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTileK; ++k) {
            const float4 u = *reinterpret_cast<const float4*>(&As[k][4 * ty]);
            const float4 w = *reinterpret_cast<const float4*>(&Bs[k][4 * tx]);
            const float uu[4] = {u.x, u.y, u.z, u.w}, ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(uu[i], ww[j], acc[i][j]);
        }
    }
    float* p = part + (size_t)blockIdx.z * kPart;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(p + (size_t)(m0 + 4 * ty + i) * kMlpIn + n0 + 4 * tx) =
            make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    if (blockIdx.x == 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) cs[r][c + j] = col[j];
        __syncthreads();
        if (t < kTile) {
            float sum = 0.f;
            for (int q = 0; q < 16; ++q) sum += cs[q][t];
            p[kPartW + m0 + t] = sum;
        }
    }
}

// The output layer's dW3 = G3^T A2 and db3, over ranges of their own.
constexpr size_t kPart3 = (size_t)kMlpOut * kMlpH + kMlpOut;
__global__ void __launch_bounds__(256) k_weight_grad3(const float* __restrict__ g3, const float* __restrict__ a2, int B,
                                                      int per, float* __restrict__ part) {
    const int t = threadIdx.x, b0 = blockIdx.x * per, b1 = min(B, b0 + per);
    float w0 = 0.f, w1 = 0.f, s = 0.f;
#pragma unroll 8
    for (int b = b0; b < b1; ++b) {
        const float a = bf16r(a2[(size_t)b * kMlpH + t]);
        w0 = fmaf(bf16r(__ldg(g3 + 2 * b)), a, w0);
        w1 = fmaf(bf16r(__ldg(g3 + 2 * b + 1)), a, w1);
        if (t < kMlpOut) s += g3[2 * b + t];
    }
    float* p = part + (size_t)blockIdx.x * kPart3;
    p[t] = w0;
    p[kMlpH + t] = w1;
    if (t < kMlpOut) p[kMlpOut * kMlpH + t] = s;
}

// The sums over the ranges into the gradients (layer 0 and 1: weights and biases; 2).
__global__ void __launch_bounds__(256) k_sum_parts(const float* __restrict__ part, const float* __restrict__ part3,
                                                   int ranges, int ranges3, float* __restrict__ w0, float* __restrict__ b0,
                                                   float* __restrict__ w1, float* __restrict__ b1,
                                                   float* __restrict__ w2, float* __restrict__ b2) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 2 * kPart) {
        const int l = i >= kPart;
        const size_t j = i - l * kPart;
        const float* p = part + (size_t)l * ranges * kPart + j;
        float s = 0.f;
#pragma unroll 8
        for (int z = 0; z < ranges; ++z) s += p[(size_t)z * kPart];
        (j < kPartW ? (l ? w1 : w0) + j : (l ? b1 : b0) + (j - kPartW))[0] = s;
    } else if (i < 2 * kPart + kPart3) {
        const size_t j = i - 2 * kPart;
        float s = 0.f;
#pragma unroll 8
        for (int z = 0; z < ranges3; ++z) s += part3[(size_t)z * kPart3 + j];
        (j < (size_t)kMlpOut * kMlpH ? w2 + j : b2 + (j - (size_t)kMlpOut * kMlpH))[0] = s;
    }
}

__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m1,
                       float* __restrict__ m2, size_t n, float lr, float b1, float b2, float eps, float bc1, float bc2,
                       float wd) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i] + wd * w[i];
    m1[i] = b1 * m1[i] + (1.f - b1) * gi;
    m2[i] = b2 * m2[i] + (1.f - b2) * gi * gi;
    w[i] -= lr * (m1[i] / bc1) / (sqrtf(m2[i] / bc2) + eps);
}

__global__ void k_gather_rows(const float* __restrict__ X, const uint8_t* __restrict__ Y, const uint32_t* __restrict__ idx,
                              int B, int D, float* __restrict__ xb, uint8_t* __restrict__ yb) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < B * D) xb[t] = X[(size_t)idx[t / D] * D + (t % D)];
    if (t < B * 2) yb[t] = Y[(size_t)idx[t / 2] * 2 + (t % 2)];
}

unsigned blocks(size_t n) { return (unsigned)((n + 255) / 256); }

}  // namespace

Mlp::Mlp() {
    const size_t sz[6] = {(size_t)kMlpH * kMlpIn, kMlpH, (size_t)kMlpH * kMlpH, kMlpH, (size_t)kMlpOut * kMlpH, kMlpOut};
    for (int i = 0; i < 6; ++i) n[i] = sz[i];
}

void Mlp::init(uint64_t seed, cudaStream_t s) {
    gr.alloc(grad_floats() * 4);
    std::mt19937_64 g(seed);
    const int fan_in[6] = {kMlpIn, kMlpIn, kMlpH, kMlpH, kMlpH, kMlpH};
    for (int i = 0; i < 6; ++i) {
        std::vector<float> h(n[i], 0.f);
        if (i % 2 == 0) {  // weights: U(-1/sqrt(fan_in), 1/sqrt(fan_in)); biases 0
            std::uniform_real_distribution<float> U(-1.f / std::sqrt((float)fan_in[i]), 1.f / std::sqrt((float)fan_in[i]));
            for (auto& x : h) x = U(g);
        }
        p[i].alloc(n[i] * 4);
        m1[i].alloc(n[i] * 4);
        m2[i].alloc(n[i] * 4);
        CUDA_CHECK(cudaMemcpyAsync(p[i].p, h.data(), n[i] * 4, cudaMemcpyHostToDevice, s));
        CUDA_CHECK(cudaMemsetAsync(m1[i].p, 0, n[i] * 4, s));
        CUDA_CHECK(cudaMemsetAsync(m2[i].p, 0, n[i] * 4, s));
    }
    std::vector<float> nr(2 * kMlpIn, 0.f);
    for (int f = 0; f < kMlpIn; ++f) nr[kMlpIn + f] = 1.f;
    norm.alloc(nr.size() * 4);
    CUDA_CHECK(cudaMemcpyAsync(norm.p, nr.data(), nr.size() * 4, cudaMemcpyHostToDevice, s));
    tc_err.alloc(16);
    CUDA_CHECK(cudaMemsetAsync(tc_err.p, 0, 16, s));
    step = 0;
    ready = true;
    CUDA_CHECK(cudaStreamSynchronize(s));
}

void Mlp::ensure_work(int B) {
    if (cap >= B) return;
    cap = 0;  // until the parts stand: an allocation that fails has freed the former one
    const size_t b = (size_t)B;
    const MostRanges r(B);
    Part* const parts[] = {&xn, &z1, &a1, &z2, &a2, &g1, &g2, &z3, &g3, &part, &part3};
    const size_t floats[] = {b * kMlpIn, b * kMlpH, b * kMlpH, b * kMlpH, b * kMlpH, b * kMlpH, b * kMlpH,
                             b * kMlpOut, b * kMlpOut, 2 * r.n * kPart, r.n3 * kPart3};
    size_t at = 0;
    for (size_t x : floats) at += (x + 63) & ~(size_t)63;
    work.ensure(at * 4);
    at = 0;
    for (int i = 0; i < 11; ++i) {
        parts[i]->p = work.as<float>() + at;
        at += (floats[i] + 63) & ~(size_t)63;
    }
    cap = B;
}

void Mlp::forward(const float* X, int B, cudaStream_t s) {
    ensure_work(B);
    forward_into(X, B, xn.as<float>(), z1.as<float>(), a1.as<float>(), z2.as<float>(), a2.as<float>(), z3.as<float>(),
                 s);
}

void Mlp::forward_into(const float* X, int B, float* xn_, float* z1_, float* a1_, float* z2_, float* a2_, float* z3_,
                       cudaStream_t s) const {
    k_normalize<<<blocks((size_t)B * kMlpIn), 256, 0, s>>>(X, norm.as<float>(), xn_, (size_t)B * kMlpIn);
    CUDA_LAUNCH_CHECK();
    // the two 256 x 256 layers on the tensor cores (GELU in the epilogue), the
    // 2-output layer on the CUDA cores
    mlp_layer_tc(xn_, B, w(0), b(0), nullptr, z1_, a1_, true, tc_err.as<int>(), s);
    mlp_layer_tc(a1_, B, w(1), b(1), nullptr, z2_, a2_, true, tc_err.as<int>(), s);
    k_out_layer<<<(unsigned)((B + 63) / 64), 64, 0, s>>>(a2_, w(2), b(2), z3_, B);
    CUDA_LAUNCH_CHECK();
}

// Gradients of the mean BCE over the batch into gr[] (forward must have run on X;
// layer 1 reads the normalised copy it left in xn).
void Mlp::backward(const float* X, const uint8_t* Y, int B, float* loss, cudaStream_t s) {
    (void)X;
    k_bce_back<<<(unsigned)((B + 15) / 16), 256, 0, s>>>(z3.as<float>(), Y, w(2), z2.as<float>(), g3.as<float>(),
                                                         g2.as<float>(), B, loss);
    CUDA_LAUNCH_CHECK();
    k_back_layer<<<dim3(kMlpH / kTile, (B + kTile - 1) / kTile), 256, 0, s>>>(g2.as<float>(), w(1), z1.as<float>(),
                                                                              g1.as<float>(), B);
    CUDA_LAUNCH_CHECK();
    const Ranges r(B);
    k_weight_grad<<<dim3(kMlpIn / kTile, kMlpH / kTile, 2 * (unsigned)r.n), 256, 0, s>>>(
        WGrad{g1.as<float>(), xn.as<float>()}, WGrad{g2.as<float>(), a1.as<float>()}, B, r.per, (int)r.n,
        part.as<float>());
    CUDA_LAUNCH_CHECK();
    k_weight_grad3<<<(unsigned)r.n3, 256, 0, s>>>(g3.as<float>(), a2.as<float>(), B, r.per3, part3.as<float>());
    CUDA_LAUNCH_CHECK();
    k_sum_parts<<<blocks(2 * kPart + kPart3), 256, 0, s>>>(part.as<float>(), part3.as<float>(), (int)r.n, (int)r.n3, grad(0),
                                                          grad(1), grad(2), grad(3),
                                                          grad(4), grad(5));
    CUDA_LAUNCH_CHECK();
}

void Mlp::check_tc() {
    int e = 0;
    CUDA_CHECK(cudaMemcpy(&e, tc_err.p, 4, cudaMemcpyDeviceToHost));
    if (e) fail(HRNN_ERR_TIMEOUT, "budget MLP: a tensor-core wait ran out");
}

void Mlp::adam(float lr, float wd, cudaStream_t s) {
    ++step;
    const float b1 = 0.9f, b2 = 0.999f;
    const float bc1 = 1.f - std::pow(b1, (float)step), bc2 = 1.f - std::pow(b2, (float)step);
    for (int i = 0; i < 6; ++i) {
        k_adam<<<blocks(n[i]), 256, 0, s>>>(p[i].as<float>(), grad(i), m1[i].as<float>(), m2[i].as<float>(),
                                            n[i], lr, b1, b2, 1e-8f, bc1, bc2, (i % 2 == 0) ? wd : 0.f);
        CUDA_LAUNCH_CHECK();
    }
}

float Mlp::train(const float* d_X, const uint8_t* d_Y, size_t N, int epochs, int batch, float lr, uint64_t seed,
                 cudaStream_t s) {
    if (!ready) fail(HRNN_ERR_STATE, "budget: model not initialised");
    DevMem idx, xb, yb, loss;
    idx.alloc(N * 4);
    xb.alloc((size_t)batch * kMlpIn * 4);
    yb.alloc((size_t)batch * 2);
    loss.alloc(4);
    std::vector<uint32_t> perm(N);
    for (size_t i = 0; i < N; ++i) perm[i] = (uint32_t)i;
    std::mt19937_64 g(seed ^ 0x9E3779B97F4A7C15ull);
    float last = 0.f;
    for (int ep = 0; ep < epochs; ++ep) {
        std::shuffle(perm.begin(), perm.end(), g);
        CUDA_CHECK(cudaMemcpyAsync(idx.p, perm.data(), N * 4, cudaMemcpyHostToDevice, s));
        CUDA_CHECK(cudaMemsetAsync(loss.p, 0, 4, s));
        int nb = 0;
        for (size_t b0 = 0; b0 + (size_t)batch <= N; b0 += batch, ++nb) {
            k_gather_rows<<<blocks((size_t)batch * kMlpIn), 256, 0, s>>>(d_X, d_Y, idx.as<uint32_t>() + b0, batch,
                                                                        kMlpIn, xb.as<float>(), yb.as<uint8_t>());
            CUDA_LAUNCH_CHECK();
            forward(xb.as<float>(), batch, s);
            backward(xb.as<float>(), yb.as<uint8_t>(), batch, loss.as<float>(), s);
            adam(lr, 1e-4f, s);
        }
        float l = 0.f;
        CUDA_CHECK(cudaMemcpyAsync(&l, loss.p, 4, cudaMemcpyDeviceToHost, s));
        CUDA_CHECK(cudaStreamSynchronize(s));
        check_tc();
        last = nb ? l / nb : 0.f;
    }
    return last;
}

}  // namespace hrnn
