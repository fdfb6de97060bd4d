// Learned warm start: a small MLP (BF16 weights and activations, FP32
// accumulation, FP32 master weights) mapping size-distribution descriptors to
// a predicted phi_J and a growth schedule. Hand-written training and inference
// kernels: tensor-core tile products (mma.sync BF16 -> FP32) with GELU, mean
// squared error and their gradients in the epilogues, and Adam.
//
// Parameters of an L-layer MLP with widths w[0..L] are packed in one FP32
// array: layer l holds W_l [w[l+1] x w[l]] row-major, then b_l [w[l+1]]. The
// hidden layers use GELU (0.5 x (1 + erf(x / sqrt 2))), the output is linear.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/rcpg.h"

namespace {

// Tensor-core tile products: C[m, n] = sum_k A[m, k] B[k, n] by mma.sync
// m16n8k16 (BF16 operands, FP32 accumulators, k ascending). These layers are
// 256 wide, so a product of a training batch is a few hundred tiles at most and
// a launch is bound by latency, not by the tensor cores: a block takes a 32x32
// tile of C (64 blocks where 64x64 tiles gave 16) and stages up to 256 of k at
// once, every load of the chunk in flight before the first mma, instead of 16
// with two barriers each; activation, loss, gradient and bias sums are the
// tiles' epilogues, and the two products of a layer's backward pass and its
// bias sums share a launch. A training step of batch 256 is 9 launches (it was
// 26). A step of batch 256 on one B200, whole call: 226 -> 89 us. The sums keep
// their order, so the results are those of the larger tiles bit for bit.
constexpr int kTM = 32, kTN = 32;      // tile of C
constexpr int kKC = 256;               // k staged at once
constexpr int kRow = kKC + 8;          // staged row: fragment loads of a warp fall in distinct banks
constexpr int kMmaThreads = 128;

__device__ __forceinline__ std::uint32_t lds_pair(const __nv_bfloat16* p) {
    return *reinterpret_cast<const std::uint32_t*>(p);
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// An operand as rows over k: element (r, k) at p[r * rs + k * ks]. FP32 inputs
// are rounded to BF16 as they are staged.
template <typename T>
struct Operand {
    const T* p;
    long long rs, ks;
};

__device__ __forceinline__ __nv_bfloat16 as_bf16(__nv_bfloat16 v) { return v; }
__device__ __forceinline__ __nv_bfloat16 as_bf16(float v) { return __float2bfloat16(v); }

// Stages rows r0 .. r0 + 31 (of `rows`), k0 .. k0 + kc - 1 (of K; kc a multiple
// of 16) into s[32][kRow], zeros outside. 16-byte loads where the operand is
// BF16, contiguous along k or along the rows, and aligned; else one by one.
template <typename T>
__device__ __forceinline__ void stage(__nv_bfloat16 (*s)[kRow], const Operand<T>& o, int r0, int rows, int k0, int K,
                                      int kc) {
    const __nv_bfloat16 zero = __float2bfloat16(0.0f);
    if constexpr (sizeof(T) == 2) {
        const bool base16 = (reinterpret_cast<std::uintptr_t>(o.p) & 15u) == 0;
        if (base16 && o.ks == 1 && (o.rs & 7) == 0 && (K & 7) == 0) {
            const int per = kc / 8;
            for (int e = threadIdx.x; e < 32 * per; e += kMmaThreads) {
                const int r = e / per, k = (e - r * per) * 8;
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (r0 + r < rows && k0 + k < K)
                    v = *reinterpret_cast<const uint4*>(o.p + (r0 + r) * o.rs + k0 + k);
                *reinterpret_cast<uint4*>(&s[r][k]) = v;
            }
            return;
        }
        if (base16 && o.rs == 1 && (o.ks & 7) == 0 && (rows & 7) == 0) {
            for (int e = threadIdx.x; e < 4 * kc; e += kMmaThreads) {
                const int k = e >> 2, r = (e & 3) * 8;
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (r0 + r < rows && k0 + k < K)
                    v = *reinterpret_cast<const uint4*>(o.p + (k0 + k) * o.ks + r0 + r);
                const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
                for (int q = 0; q < 8; ++q) s[r + q][k] = w[q];
            }
            return;
        }
    }
    const bool along_k = o.ks == 1;
    for (int e = threadIdx.x; e < 32 * kc; e += kMmaThreads) {
        const int r = along_k ? e / kc : (e & 31), k = along_k ? e - r * kc : (e >> 5);
        s[r][k] = (r0 + r < rows && k0 + k < K) ? as_bf16(o.p[(r0 + r) * o.rs + (k0 + k) * o.ks]) : zero;
    }
}

struct Tile {
    __nv_bfloat16 a[kTM][kRow], b[kTN][kRow];
};

// The 32x32 tile at (m0, n0) of A (M x K) times B (K x N, given by columns);
// out(m, n, c) for every element inside the matrix. Each of the four warps
// holds 16x16 of it.
template <typename TA, typename TB, typename Out>
__device__ __forceinline__ void tile_product(Tile& t, const Operand<TA>& A, const Operand<TB>& B, int M, int N, int K,
                                             int m0, int n0, Out&& out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
    float acc[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[j][r] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += kKC) {
        const int kc = min(kKC, (K - k0 + 15) & ~15);
        if (k0) __syncthreads();
        stage(t.a, A, m0, M, k0, K, kc);
        stage(t.b, B, n0, N, k0, K, kc);
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < kc; k += 16) {
            std::uint32_t af[4], bf[2][2];
            af[0] = lds_pair(&t.a[wm + g][k + 2 * q]);
            af[1] = lds_pair(&t.a[wm + g + 8][k + 2 * q]);
            af[2] = lds_pair(&t.a[wm + g][k + 2 * q + 8]);
            af[3] = lds_pair(&t.a[wm + g + 8][k + 2 * q + 8]);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                bf[j][0] = lds_pair(&t.b[wn + j * 8 + g][k + 2 * q]);
                bf[j][1] = lds_pair(&t.b[wn + j * 8 + g][k + 2 * q + 8]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
                asm volatile(
                    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
                    "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                    : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                    : "r"(af[0]), "r"(af[1]), "r"(af[2]), "r"(af[3]), "r"(bf[j][0]), "r"(bf[j][1]));
        }
    }
    // c0, c1 at (g, 2q..2q+1), c2, c3 at (g+8, 2q..2q+1) of each 16x8 tile
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int m = m0 + wm + g + (r >= 2 ? 8 : 0);
            const int n = n0 + wn + j * 8 + 2 * q + (r & 1);
            if (m < M && n < N) out(m, n, acc[j][r]);
        }
}

// One layer forward: z = a W^T + bias; a hidden layer stores gelu(z) in BF16
// (and z where the backward pass will need it), the output layer z, and with
// `target` the loss terms and dL/dz = 2 w (z - t) / (batch * outputs) in BF16;
// with `y64` the destandardised prediction.
template <typename TA>
__global__ void __launch_bounds__(kMmaThreads)
    k_forward(int M, int N, int K, const TA* __restrict__ a, const __nv_bfloat16* __restrict__ W,
              const float* __restrict__ bias, float* __restrict__ z, __nv_bfloat16* __restrict__ act,
              const float* __restrict__ target, const float* __restrict__ weight, __nv_bfloat16* __restrict__ dz,
              float* __restrict__ lterm, const double* __restrict__ scale, double* __restrict__ y64) {
    __shared__ __align__(16) Tile t;
    tile_product(t, Operand<TA>{a, K, 1}, Operand<__nv_bfloat16>{W, K, 1}, M, N, K, blockIdx.x * kTM, blockIdx.y * kTN,
                 [&](int m, int n, float c) {
                     const long long e = static_cast<long long>(m) * N + n;
                     const float v = c + bias[n];
                     if (z) z[e] = v;
                     if (y64)  // scale: y_mean[N], y_std[N]
                         y64[e] = __dadd_rn(__dmul_rn(static_cast<double>(v), scale[N + n]), scale[n]);
                     if (act) act[e] = __float2bfloat16(gelu(v));
                     if (target) {
                         const float w = weight ? weight[n] : 1.0f;
                         const float d = v - target[e];
                         lterm[e] = w * d * d;
                         dz[e] = __float2bfloat16(2.0f * w * d / static_cast<float>(M * N));
                     }
                 });
}

// One layer backward from dz (B x O): blocks 0 .. nx-1 the tiles of dz_prev =
// (dz W) gelu'(z_prev) (B x I, BF16; none for the first layer), then the tiles
// of dW = dz^T a (O x I), then the bias sums db[o] = sum_b dz[b, o] (FP32, b
// ascending; 128 outputs per block).
template <typename TA>
__global__ void __launch_bounds__(kMmaThreads)
    k_backward(int B, int O, int I, const __nv_bfloat16* __restrict__ dz, const TA* __restrict__ a,
               const __nv_bfloat16* __restrict__ W, const float* __restrict__ z_prev,
               __nv_bfloat16* __restrict__ dz_prev, float* __restrict__ dW, float* __restrict__ db, int nx, int nw) {
    __shared__ __align__(16) Tile t;
    int b = blockIdx.x;
    const int ti = (I + kTN - 1) / kTN;
    if (b < nx) {
        tile_product(t, Operand<__nv_bfloat16>{dz, O, 1}, Operand<__nv_bfloat16>{W, 1, I}, B, I, O, (b / ti) * kTM,
                     (b % ti) * kTN, [&](int m, int n, float c) {
                         const long long e = static_cast<long long>(m) * I + n;
                         dz_prev[e] = __float2bfloat16(c * gelu_grad(z_prev[e]));
                     });
        return;
    }
    b -= nx;
    if (b < nw) {
        tile_product(t, Operand<__nv_bfloat16>{dz, 1, O}, Operand<TA>{a, 1, I}, O, I, B, (b / ti) * kTM, (b % ti) * kTN,
                     [&](int m, int n, float c) { dW[static_cast<long long>(m) * I + n] = c; });
        return;
    }
    b -= nw;
    const int o = b * kMmaThreads + threadIdx.x;
    if (o >= O) return;
    float s = 0.0f;
    int r = 0;
    for (; r + 16 <= B; r += 16) {  // sixteen loads in flight, added in order
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = __bfloat162float(dz[static_cast<long long>(r + q) * O + o]);
#pragma unroll
        for (int q = 0; q < 16; ++q) s += v[q];
    }
    for (; r < B; ++r) s += __bfloat162float(dz[static_cast<long long>(r) * O + o]);
    db[o] = s;
}

// Descriptors held in the training range, standardised (FP64), rounded to FP32
// and then to the BF16 that the first layer multiplies. norm: lo, hi, mean, std.
// This and the output's scaling were three quarters of a prediction's time on
// the host: 4,096 rows 562 -> 209 us on one B200, of which the two copies and
// the call are most.
__global__ void __launch_bounds__(256) k_standardise(int n, int I, const double* __restrict__ X,
                                                     const double* __restrict__ norm, __nv_bfloat16* __restrict__ a) {
    const int e = blockIdx.x * 256 + threadIdx.x;
    if (e >= n) return;
    const int i = e % I;
    double x = X[e];
    if (x < norm[i]) x = norm[i];  // a NaN stays one
    if (x > norm[I + i]) x = norm[I + i];
    a[e] = __float2bfloat16(static_cast<float>(__ddiv_rn(__dsub_rn(x, norm[2 * I + i]), norm[3 * I + i])));
}

__global__ void k_to_bf16(int n, const float* __restrict__ x, __nv_bfloat16* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16(x[i]);
}

// Adam on the FP32 master weights, then the BF16 copy
__global__ void k_adam(int n, float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, float lr, float b1, float b2, float c1, float c2,
                       __nv_bfloat16* __restrict__ wb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
    w[i] = wi;
    wb[i] = __float2bfloat16(wi);
}

unsigned blocks(long long n) { return static_cast<unsigned>((n + 255) / 256); }

std::size_t param_count(const int32_t* w, int L) {
    std::size_t n = 0;
    for (int l = 0; l < L; ++l) n += static_cast<std::size_t>(w[l + 1]) * w[l] + w[l + 1];
    return n;
}

// Scratch of one forward/backward pass, carved from the caller's workspace.
struct Work {
    std::vector<__nv_bfloat16*> act;  // act[l] = output of layer l - 1 (BF16), l >= 1
    std::vector<float*> z;            // pre-activations of layer l (FP32)
    __nv_bfloat16* dz;                // BF16 gradient w.r.t. a pre-activation
    __nv_bfloat16* dzp;               // the previous layer's
    float* lterm;
};

bool carve(void* ws, std::size_t ws_bytes, const int32_t* w, int L, int B, Work& wk) {
    auto* p = static_cast<unsigned char*>(ws);
    std::size_t used = 0;
    auto take = [&](std::size_t bytes) -> void* {
        used = (used + 255) & ~std::size_t{255};
        void* r = p + used;
        used += bytes;
        return r;
    };
    int wmax = 0;
    for (int l = 0; l <= L; ++l) wmax = w[l] > wmax ? w[l] : wmax;
    wk.act.resize(L + 1);
    wk.z.resize(L);
    for (int l = 0; l <= L; ++l) wk.act[l] = static_cast<__nv_bfloat16*>(take(static_cast<std::size_t>(B) * w[l] * 2));
    for (int l = 0; l < L; ++l) wk.z[l] = static_cast<float*>(take(static_cast<std::size_t>(B) * w[l + 1] * 4));
    take(static_cast<std::size_t>(B) * wmax * 4);  // unused; rcpg_mlp_workspace_bytes keeps the size it has always returned
    wk.dz = static_cast<__nv_bfloat16*>(take(static_cast<std::size_t>(B) * wmax * 2));
    wk.dzp = static_cast<__nv_bfloat16*>(take(static_cast<std::size_t>(B) * wmax * 2));
    wk.lterm = static_cast<float*>(take(static_cast<std::size_t>(B) * w[L] * 4));
    return used <= ws_bytes;
}

// The layers' launches, from X or (X null) from the BF16 input in wk.act[0]. y:
// where the output layer's z goes; with T the loss
// terms go to lterm and the gradient to wk.dz, and the hidden z are kept.
void forward(cudaStream_t st, const int32_t* w, int L, int B, const __nv_bfloat16* wb, const float* w32,
             const float* X, Work& wk, float* y, const float* T, const float* weight, float* lterm,
             const double* scale = nullptr, double* y64 = nullptr) {
    std::size_t off = 0;
    for (int l = 0; l < L; ++l) {
        const int I = w[l], O = w[l + 1];
        const bool last = l + 1 == L;
        const dim3 grid((B + kTM - 1) / kTM, (O + kTN - 1) / kTN);  // rows along x: y ends at 65,535 tiles
        const float* bias = w32 + off + static_cast<std::size_t>(O) * I;
        float* z = last ? y : (T ? wk.z[l] : nullptr);
        __nv_bfloat16* act = last ? nullptr : wk.act[l + 1];
        const float* tgt = last ? T : nullptr;
        double* out64 = last ? y64 : nullptr;
        if (l == 0 && X)
            k_forward<float><<<grid, kMmaThreads, 0, st>>>(B, O, I, X, wb + off, bias, z, act, tgt, weight, wk.dz, lterm,
                                                           scale, out64);
        else
            k_forward<__nv_bfloat16><<<grid, kMmaThreads, 0, st>>>(B, O, I, wk.act[l], wb + off, bias, z, act, tgt, weight,
                                                                   wk.dz, lterm, scale, out64);
        off += static_cast<std::size_t>(O) * I + O;
    }
}

int32_t fail(char* err, std::size_t errlen, int32_t code, const char* msg) {
    if (err && errlen) std::snprintf(err, errlen, "%s", msg);
    return code;
}

bool widths_ok(const int32_t* w, int L) {
    if (!w || L <= 0) return false;
    for (int l = 0; l <= L; ++l)
        if (w[l] <= 0 || w[l] > (1 << 20)) return false;
    return true;
}

}  // namespace

extern "C" {

uint64_t rcpg_mlp_param_count(const int32_t* widths, int32_t layers) {
    return widths_ok(widths, layers) ? param_count(widths, layers) : 0;
}

uint64_t rcpg_mlp_workspace_bytes(const int32_t* widths, int32_t layers, int32_t batch) {
    if (!widths_ok(widths, layers) || batch <= 0) return 0;
    int wmax = 0;
    std::size_t b = 0;
    for (int l = 0; l <= layers; ++l) {
        wmax = widths[l] > wmax ? widths[l] : wmax;
        b += static_cast<std::size_t>(batch) * widths[l] * 2 + 256;
    }
    for (int l = 0; l < layers; ++l) b += static_cast<std::size_t>(batch) * widths[l + 1] * 4 + 256;
    b += static_cast<std::size_t>(batch) * wmax * 8 + 3 * 256 + static_cast<std::size_t>(batch) * widths[layers] * 4 + 256;
    return b;
}

int32_t rcpg_mlp_forward(const int32_t* widths, int32_t layers, int32_t batch, const void* w_bf16,
                         const float* w_fp32, const float* X, float* Y, void* workspace,
                         uint64_t workspace_bytes, void* stream, char* err, size_t errlen) {
    if (!widths_ok(widths, layers) || batch <= 0 || !w_bf16 || !w_fp32 || !X || !Y || !workspace)
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: bad arguments to rcpg_mlp_forward");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Work wk;
    if (!carve(workspace, workspace_bytes, widths, layers, batch, wk))
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: MLP workspace too small");
    forward(st, widths, layers, batch, static_cast<const __nv_bfloat16*>(w_bf16), w_fp32, X, wk, Y, nullptr, nullptr,
            nullptr);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(err, errlen, RCPG_ECUDA, cudaGetErrorString(e));
    return RCPG_OK;
}

int32_t rcpg_mlp_predict(const int32_t* widths, int32_t layers, int32_t batch, const void* w_bf16,
                         const float* w_fp32, const double* X, const double* norm, double* Y, void* workspace,
                         uint64_t workspace_bytes, void* stream, char* err, size_t errlen) {
    if (!widths_ok(widths, layers) || batch <= 0 || !w_bf16 || !w_fp32 || !X || !norm || !Y || !workspace)
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: bad arguments to rcpg_mlp_predict");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Work wk;
    if (!carve(workspace, workspace_bytes, widths, layers, batch, wk))
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: MLP workspace too small");
    const int I = widths[0], n = batch * I;
    k_standardise<<<blocks(n), 256, 0, st>>>(n, I, X, norm, wk.act[0]);
    forward(st, widths, layers, batch, static_cast<const __nv_bfloat16*>(w_bf16), w_fp32, nullptr, wk, nullptr, nullptr,
            nullptr, nullptr, norm + 4 * static_cast<std::size_t>(I), Y);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(err, errlen, RCPG_ECUDA, cudaGetErrorString(e));
    return RCPG_OK;
}

int32_t rcpg_mlp_train_step(const int32_t* widths, int32_t layers, int32_t batch, float* w_fp32,
                            void* w_bf16, float* adam_m, float* adam_v, float* grad, const float* X,
                            const float* T, const float* out_weight, float lr, int32_t step,
                            float* loss_terms, void* workspace, uint64_t workspace_bytes, void* stream,
                            char* err, size_t errlen) {
    if (!widths_ok(widths, layers) || batch <= 0 || !w_fp32 || !w_bf16 || !grad || !X || !T || !workspace)
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: bad arguments to rcpg_mlp_train_step");
    if (adam_m && adam_v && lr > 0.0f && step < 1)
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: the Adam step counter starts at 1");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    Work wk;
    if (!carve(workspace, workspace_bytes, widths, layers, batch, wk))
        return fail(err, errlen, RCPG_EINVAL, "rcpgenerator_b200: MLP workspace too small");
    auto* wb = static_cast<__nv_bfloat16*>(w_bf16);
    forward(st, widths, layers, batch, wb, w_fp32, X, wk, wk.z[layers - 1], T, out_weight,
            loss_terms ? loss_terms : wk.lterm);
    // offsets of the layers in the packed parameters
    std::vector<std::size_t> off(layers + 1, 0);
    for (int l = 0; l < layers; ++l) off[l + 1] = off[l] + static_cast<std::size_t>(widths[l + 1]) * widths[l] + widths[l + 1];
    for (int l = layers - 1; l >= 0; --l) {
        const int I = widths[l], Ol = widths[l + 1];
        float* gW = grad + off[l];
        float* gb = gW + static_cast<std::size_t>(Ol) * I;
        const int ti = (I + kTN - 1) / kTN, tb = (batch + kTM - 1) / kTM, to = (Ol + kTM - 1) / kTM;
        const int nx = l > 0 ? tb * ti : 0, nw = to * ti, nb = (Ol + kMmaThreads - 1) / kMmaThreads;
        const unsigned grid = static_cast<unsigned>(nx + nw + nb);
        if (l > 0) {
            k_backward<__nv_bfloat16><<<grid, kMmaThreads, 0, st>>>(batch, Ol, I, wk.dz, wk.act[l], wb + off[l],
                                                                    wk.z[l - 1], wk.dzp, gW, gb, nx, nw);
            std::swap(wk.dz, wk.dzp);
        } else {
            k_backward<float><<<grid, kMmaThreads, 0, st>>>(batch, Ol, I, wk.dz, X, wb + off[l], nullptr, nullptr, gW, gb,
                                                            nx, nw);
        }
    }
    if (adam_m && adam_v && lr > 0.0f) {
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.0f - std::pow(b1, static_cast<float>(step)), c2 = 1.0f - std::pow(b2, static_cast<float>(step));
        const int n = static_cast<int>(off[layers]);
        k_adam<<<blocks(n), 256, 0, st>>>(n, w_fp32, adam_m, adam_v, grad, lr, b1, b2, c1, c2, wb);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(err, errlen, RCPG_ECUDA, cudaGetErrorString(e));
    return RCPG_OK;
}

int32_t rcpg_mlp_to_bf16(uint64_t n, const float* x, void* y, void* stream) {
    if (!x || !y) return RCPG_EINVAL;
    k_to_bf16<<<blocks(static_cast<long long>(n)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<int>(n), x, static_cast<__nv_bfloat16*>(y));
    return cudaGetLastError() == cudaSuccess ? RCPG_OK : RCPG_ECUDA;
}

}  // extern "C"
