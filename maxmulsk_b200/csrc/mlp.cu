// Learned cost model: a 2-hidden-layer MLP (64 GELU units each, FP32) that
// predicts the log-time of every candidate plan of a shape. Hand-written
// CUDA for training (forward, backward, Adam) and batched inference, plus a
// host forward pass with the same arithmetic order for the per-call picker.
//
// Counterpart in the reference: the hand-written shape rules and table it
// replaces (SMEKernels1x4V4C::choose, sme/v4/sme-1x4-v4c-dispatch.cpp:17-22;
// the v5.1 fixed plan, sme/v5/sme-1x4-fusedpack-v51.cpp:744-747; the tuning
// table, sme/support/gemm_tuning.cpp:34-37).
//
// Parameters are one flat FP32 array:
//   W1[F][H] b1[H] W2[H][H] b2[H] W3[H][O] b3[O]     (F = 7, H = 64, O = 48)
// Features of a shape (M, K, N, class):
//   ln(M), ln(N), ln(K) / ln(16384); (M, N, K mod 16) / 16; class (0 FP32, 1 split)
// Every kernel is deterministic: reductions run in a fixed order, no atomics.
#include <cooperative_groups.h>
#include <dlfcn.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "internal.hpp"
#include "launch.cuh"
#include "mlp.hpp"
#include "runtime.hpp"
#include "split_math.cuh"

namespace cg = cooperative_groups;

namespace mmsk {

namespace {

constexpr int F = MAXMULSK_MLP_FEATURES, H = MAXMULSK_MLP_HIDDEN, O = MAXMULSK_MLP_OUTPUTS;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + F * H, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H,
              OFF_W3 = OFF_B2 + H, OFF_B3 = OFF_W3 + H * O, NPARAM = OFF_B3 + O;
static_assert(NPARAM == MAXMULSK_MLP_PARAMS, "parameter count");

// GELU, exact form 0.5 x (1 + erf(x / sqrt 2)), and its derivative.
__host__ __device__ inline float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__host__ __device__ inline float gelu_grad(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// Forward pass, all three layers: Z[b][o] = bias[o] + sum_i X[b][i] W[i][o], i
// upward, and H = gelu(Z) after the first two. A block takes kFwdRows rows; the
// weights (30 KB) and the rows' activations stay in shared memory between the
// layers. Thread t computes output o = t % 64 of rows t / 64 + 4 j: a row of W
// is read by consecutive lanes, four inputs of a row by broadcast. Bound by
// latency (61 MFLOP at 4000 rows): one launch instead of three.
constexpr int kFwdRows = 16;
__global__ void __launch_bounds__(256)
mlp_forward_kernel(const float* __restrict__ params, const float* __restrict__ X, int B, float* __restrict__ Z1,
                   float* __restrict__ H1, float* __restrict__ Z2, float* __restrict__ H2, float* __restrict__ Y) {
    __shared__ float w[NPARAM];
    __shared__ __align__(16) float in[2][kFwdRows][H];           // X or H2, and H1
    const int tid = threadIdx.x, o = tid & 63, rq = tid >> 6;
    const int b0 = blockIdx.x * kFwdRows;
    grid_wait();
#pragma unroll
    for (int j = 0; j < (NPARAM + 255) / 256; j++)
        if (tid + j * 256 < NPARAM) w[tid + j * 256] = params[tid + j * 256];
    for (int i = tid; i < kFwdRows * 8; i += 256) {
        const int r = i >> 3, c = i & 7;
        in[0][r][c] = (c < F && b0 + r < B) ? X[(size_t)(b0 + r) * F + c] : 0.f;   // an eighth, zero input
    }
    __syncthreads();
    auto layer = [&](const float (*x)[H], int n, const float* W, const float* bias, int out, float (&z)[4]) {
#pragma unroll
        for (int j = 0; j < 4; j++) z[j] = bias[o];
        for (int i = 0; i < n; i += 4) {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = *reinterpret_cast<const float4*>(&x[rq + 4 * j][i]);
            const float w0 = W[i * out + o], w1 = W[(i + 1) * out + o], w2 = W[(i + 2) * out + o];
#pragma unroll
            for (int j = 0; j < 4; j++) z[j] = fmaf(v[j].z, w2, fmaf(v[j].y, w1, fmaf(v[j].x, w0, z[j])));
            if (i + 3 < n) {
                const float w3 = W[(i + 3) * out + o];
#pragma unroll
                for (int j = 0; j < 4; j++) z[j] = fmaf(v[j].w, w3, z[j]);
            }
        }
    };
    auto hidden = [&](const float (&z)[4], float (*dst)[H], float* Z, float* A) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = rq + 4 * j;
            const float h = gelu(z[j]);
            dst[r][o] = h;
            if (b0 + r < B) {
                const size_t k = (size_t)(b0 + r) * H + o;
                if (Z) Z[k] = z[j];
                A[k] = h;
            }
        }
        __syncthreads();
    };
    float z[4];
    layer(in[0], F, w + OFF_W1, w + OFF_B1, H, z);
    hidden(z, in[1], Z1, H1);
    layer(in[1], H, w + OFF_W2, w + OFF_B2, H, z);
    hidden(z, in[0], Z2, H2);
    if (o >= O) return;
    layer(in[0], H, w + OFF_W3, w + OFF_B3, O, z);
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (b0 + rq + 4 * j < B) Y[(size_t)(b0 + rq + 4 * j) * O + o] = z[j];
}

// Backward pass. dY = 2 (Y - T) / count over the entries with mask != 0 (else
// 0), rowloss[b] the row's squared errors; through each layer
//   dX[b][i] = sum_o dZ[b][o] W[i][o], times gelu'(Zprev[b][i]);
//   dW[i][o] = sum_b X[b][i] dZ[b][o],  db[o] = sum_b dZ[b][o].
// A block takes eight rows at a time through shared memory (W2 and W3 padded so
// that lanes walking i hit distinct banks) and keeps its sums of all weight
// gradients in registers: thread t owns 12 of dW3, 16 of dW2, 2 of dW1. Eight
// blocks form a cluster; at the end each adds an eighth of the weights over the
// cluster's shared memories, in block order, into parts[cluster][NPARAM], and
// mlp_grad_sum adds the clusters in order (with one cluster, parts is grads).
// Bound by latency, so the rows are spread thin. At 4000 rows 22.8-24.2 us (ncu, cold
// caches) on 256 blocks; 89 blocks of 45 rows without clusters 44 us, one thread
// per weight walking all rows, in six launches, 840 us. A whole training step
// 893 -> 39 us, 30 with its launches overlapped (launch.cuh).
constexpr int kBwdRows = 8, kBwdCluster = 8;
__global__ void __launch_bounds__(256)
mlp_backward_kernel(const float* __restrict__ params, const float* __restrict__ X, const float* __restrict__ Z1,
                    const float* __restrict__ H1, const float* __restrict__ Z2, const float* __restrict__ H2,
                    const float* __restrict__ Y, const float* __restrict__ T, const float* __restrict__ mask, int B,
                    float inv_count, float* __restrict__ parts, float* __restrict__ rowloss) {
    constexpr int R = kBwdRows;
    static_assert(R == 8, "one row a warp, two rows a thread");
    constexpr int P3 = O + 4, P2 = H + 4;                  // row strides: quads of eight rows on distinct banks
    __shared__ __align__(16) float buf[NPARAM];            // W3 and W2, then this block's gradient sums
    static_assert(H * P3 + H * P2 <= NPARAM, "padded weights fit the gradients' buffer");
    float (*w3)[P3] = reinterpret_cast<float (*)[P3]>(buf);
    float (*w2)[P2] = reinterpret_cast<float (*)[P2]>(buf + H * P3);
    __shared__ __align__(16) float dy[R][O], h2[R][H], dz2[R][H], h1[R][H], dz1[R][H];
    __shared__ float xs[R][F];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    grid_wait();
#pragma unroll
    for (int i = tid; i < H * O; i += 256) w3[i / O][i % O] = params[OFF_W3 + i];
#pragma unroll
    for (int i = tid; i < H * H; i += 256) w2[i / H][i % H] = params[OFF_W2 + i];
    const int wi = tid >> 2, o3 = (tid & 3) * 12, o2 = (tid & 3) * 16;   // dW3[wi][o3 ..], dW2[wi][o2 ..]
    const int hi = tid & 63, hr = tid >> 6;                              // dZ[hr + 4 j][hi]
    const int i1 = tid / 32, o1 = (tid & 31) * 2;                        // dW1[i1][o1 ..], i1 < F
    float g3[12], g2[16], g1[2], gb = 0.f;                               // gb: db3, db2 or db1 by thread range
#pragma unroll
    for (int j = 0; j < 12; j++) g3[j] = 0.f;
#pragma unroll
    for (int j = 0; j < 16; j++) g2[j] = 0.f;
    g1[0] = g1[1] = 0.f;

    // The next eight rows are read while the current ones are worked on; rows
    // past B count as zeros.
    float ny[2], nt[2], nm[2], nh2[2], nh1[2], nz2[2], nz1[2], nx;
    auto fetch = [&](int r0) {
        const int b = r0 + warp;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int o = lane + 32 * j;
            const bool ok = b < B && o < O;
            const size_t k = (size_t)b * O + o;
            ny[j] = ok ? Y[k] : 0.f;
            nt[j] = ok ? T[k] : 0.f;
            nm[j] = ok ? mask[k] : 0.f;
            const int bh = r0 + hr + 4 * j;
            const size_t kh = (size_t)bh * H + hi;
            const bool okh = bh < B;
            nh2[j] = okh ? H2[kh] : 0.f;
            nh1[j] = okh ? H1[kh] : 0.f;
            nz2[j] = okh ? Z2[kh] : 0.f;
            nz1[j] = okh ? Z1[kh] : 0.f;
        }
        nx = (tid < R * F && r0 + tid / F < B) ? X[(size_t)r0 * F + tid] : 0.f;
    };
    const int stride = (int)gridDim.x * R;
    fetch((int)blockIdx.x * R);
    for (int r0 = (int)blockIdx.x * R; r0 < B; r0 += stride) {
        float l = 0.f, z2[2], z1[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float d = nm[j] != 0.f ? ny[j] - nt[j] : 0.f;
            if (lane + 32 * j < O) dy[warp][lane + 32 * j] = 2.f * d * inv_count;
            l = fmaf(d, d, l);
            h2[hr + 4 * j][hi] = nh2[j];
            h1[hr + 4 * j][hi] = nh1[j];
            z2[j] = nz2[j];
            z1[j] = nz1[j];
        }
        if (tid < R * F) xs[tid / F][tid % F] = nx;
        if (r0 < B - stride) fetch(r0 + stride);
#pragma unroll
        for (int m = 16; m; m >>= 1) l += __shfl_xor_sync(0xffffffffu, l, m);
        if (lane == 0 && r0 + warp < B) rowloss[r0 + warp] = l;
        __syncthreads();
        {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
            for (int o = 0; o < O; o += 4) {
                const float4 wv = *reinterpret_cast<const float4*>(&w3[hi][o]);
                const float4 a = *reinterpret_cast<const float4*>(&dy[hr][o]);
                const float4 c = *reinterpret_cast<const float4*>(&dy[hr + 4][o]);
                s0 = fmaf(a.w, wv.w, fmaf(a.z, wv.z, fmaf(a.y, wv.y, fmaf(a.x, wv.x, s0))));
                s1 = fmaf(c.w, wv.w, fmaf(c.z, wv.z, fmaf(c.y, wv.y, fmaf(c.x, wv.x, s1))));
            }
            dz2[hr][hi] = s0 * gelu_grad(z2[0]);
            dz2[hr + 4][hi] = s1 * gelu_grad(z2[1]);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float x = h2[r][wi];
#pragma unroll
                for (int j = 0; j < 12; j += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(&dy[r][o3 + j]);
                    g3[j] = fmaf(x, v.x, g3[j]);
                    g3[j + 1] = fmaf(x, v.y, g3[j + 1]);
                    g3[j + 2] = fmaf(x, v.z, g3[j + 2]);
                    g3[j + 3] = fmaf(x, v.w, g3[j + 3]);
                }
            }
        }
        __syncthreads();
        {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
            for (int o = 0; o < H; o += 4) {
                const float4 wv = *reinterpret_cast<const float4*>(&w2[hi][o]);
                const float4 a = *reinterpret_cast<const float4*>(&dz2[hr][o]);
                const float4 c = *reinterpret_cast<const float4*>(&dz2[hr + 4][o]);
                s0 = fmaf(a.w, wv.w, fmaf(a.z, wv.z, fmaf(a.y, wv.y, fmaf(a.x, wv.x, s0))));
                s1 = fmaf(c.w, wv.w, fmaf(c.z, wv.z, fmaf(c.y, wv.y, fmaf(c.x, wv.x, s1))));
            }
            dz1[hr][hi] = s0 * gelu_grad(z1[0]);
            dz1[hr + 4][hi] = s1 * gelu_grad(z1[1]);
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float x = h1[r][wi];
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(&dz2[r][o2 + j]);
                    g2[j] = fmaf(x, v.x, g2[j]);
                    g2[j + 1] = fmaf(x, v.y, g2[j + 1]);
                    g2[j + 2] = fmaf(x, v.z, g2[j + 2]);
                    g2[j + 3] = fmaf(x, v.w, g2[j + 3]);
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (i1 < F) {
                const float x = xs[r][i1];
                g1[0] = fmaf(x, dz1[r][o1], g1[0]);
                g1[1] = fmaf(x, dz1[r][o1 + 1], g1[1]);
            }
            if (tid < O) gb += dy[r][tid];
            else if (tid >= 64 && tid < 64 + H) gb += dz2[r][tid - 64];
            else if (tid >= 128 && tid < 128 + H) gb += dz1[r][tid - 128];
        }
        __syncthreads();                     // the next rows overwrite these
    }
    __syncthreads();                         // W2 and W3 are done with (and, in a block without rows, stored)
#pragma unroll
    for (int j = 0; j < 12; j++) buf[OFF_W3 + wi * O + o3 + j] = g3[j];
#pragma unroll
    for (int j = 0; j < 16; j++) buf[OFF_W2 + wi * H + o2 + j] = g2[j];
    if (i1 < F) {
        buf[OFF_W1 + i1 * H + o1] = g1[0];
        buf[OFF_W1 + i1 * H + o1 + 1] = g1[1];
    }
    if (tid < O) buf[OFF_B3 + tid] = gb;
    else if (tid >= 64 && tid < 64 + H) buf[OFF_B2 + tid - 64] = gb;
    else if (tid >= 128 && tid < 128 + H) buf[OFF_B1 + tid - 128] = gb;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    float* out = parts + (size_t)(blockIdx.x / kBwdCluster) * NPARAM;
    const int share = (NPARAM + kBwdCluster - 1) / kBwdCluster, first = (int)cluster.block_rank() * share;
    for (int i = first + tid; i < min(NPARAM, first + share); i += 256) {
        float v[kBwdCluster];
#pragma unroll
        for (int c = 0; c < kBwdCluster; c++) v[c] = cluster.map_shared_rank(buf, c)[i];
        float g = v[0];
#pragma unroll
        for (int c = 1; c < kBwdCluster; c++) g += v[c];
        out[i] = g;
    }
    cluster.sync();                          // no block leaves while another reads its sums
}

// grads[i] = parts[0][i] + parts[1][i] + ..., in block order.
__global__ void __launch_bounds__(128)
mlp_grad_sum(const float* __restrict__ parts, int n, float* __restrict__ grads) {
    grid_wait();
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i < NPARAM) grads[i] = ordered_sum<31>(parts + i, (size_t)NPARAM, n);
}

// Adam (bias-corrected), elementwise.
__global__ void adam_step(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                          float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    grid_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// best[b] = argmin over o with mask != 0 of Y[b][o] (lowest index on ties; -1 if none).
__global__ void masked_argmin(const float* __restrict__ Y, const float* __restrict__ mask, int B, int* __restrict__ best) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    int bi = -1;
    float bv = 0.f;
    for (int o = 0; o < O; o++) {
        if (mask[b * O + o] == 0.f) continue;
        const float y = Y[b * O + o];
        if (bi < 0 || y < bv) { bi = o; bv = y; }
    }
    best[b] = bi;
}

inline unsigned blocks(int n) { return (unsigned)((n + 255) / 256); }

// ----------------------------------------------------------------- host model
struct Model {
    bool loaded = false;
    std::vector<float> w;                     // NPARAM, or 2 NPARAM: the FP32 class's, then the split class's
};
std::mutex g_model_mu;
Model g_model;
bool g_env_tried = false;
std::atomic<uint64_t> g_model_gen{1};         // counts the models there have been

// z[o] = bias[o] + sum_i x[i] W[i][o], i upward, one fused multiply-add a step
// (the order and rounding of mlp_forward_kernel): a row of W at a time, so that the
// outputs' chains fill vector registers instead of a library call per term.
#define MMSK_ROWS_FMA(NAME, ATTR)                                                                 \
    ATTR void NAME(const float* x, const float* w, const float* bias, int in, int out, float* z) { \
        for (int o = 0; o < out; o++) z[o] = bias[o];                                             \
        for (int i = 0; i < in; i++)                                                              \
            for (int o = 0; o < out; o++) z[o] = __builtin_fmaf(x[i], w[i * out + o], z[o]);      \
    }
MMSK_ROWS_FMA(rows_fma_plain, )
#if defined(__x86_64__)
MMSK_ROWS_FMA(rows_fma_avx2, __attribute__((target("avx2,fma"))))
#endif
#undef MMSK_ROWS_FMA

void host_linear(const float* x, const float* w, const float* bias, int in, int out, float* z) {
#if defined(__x86_64__)
    static const bool wide = __builtin_cpu_supports("avx2") && __builtin_cpu_supports("fma");
    if (wide) return rows_fma_avx2(x, w, bias, in, out, z);
#endif
    rows_fma_plain(x, w, bias, in, out, z);
}

void host_forward(const float* w, const float* x, float* y) {
    float h1[H], h2[H];
    host_linear(x, w + OFF_W1, w + OFF_B1, F, H, h1);
    for (float& v : h1) v = gelu(v);
    host_linear(h1, w + OFF_W2, w + OFF_B2, H, H, h2);
    for (float& v : h2) v = gelu(v);
    host_linear(h2, w + OFF_W3, w + OFF_B3, H, O, y);
}

// <directory of this library>/../data/picker_model.bin
std::string default_model_path() {
    Dl_info info;
    if (!dladdr(reinterpret_cast<void*>(&mlp_features), &info) || !info.dli_fname) return std::string();
    std::string so(info.dli_fname);
    const size_t slash = so.rfind('/');
    const std::string dir = (slash == std::string::npos) ? std::string(".") : so.substr(0, slash);
    return dir + "/../data/picker_model.bin";
}

bool load_file(const char* path, std::vector<float>& w) {
    FILE* f = std::fopen(path, "rb");
    if (!f) return false;
    char magic[8];
    int32_t dims[4];
    bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "MMSKMLP1", 8) == 0 &&
              std::fread(dims, sizeof(int32_t), 4, f) == 4 && dims[0] == F && dims[1] == H && dims[2] == O &&
              dims[3] == NPARAM;
    if (ok) {
        w.resize(NPARAM);
        ok = std::fread(w.data(), sizeof(float), NPARAM, f) == (size_t)NPARAM;
        // Weights of the split class's own, if they follow whole.
        std::vector<float> split(NPARAM);
        if (ok && std::fread(split.data(), sizeof(float), NPARAM, f) == (size_t)NPARAM)
            w.insert(w.end(), split.begin(), split.end());
    }
    std::fclose(f);
    return ok;
}

}  // namespace

void mlp_features(size_t M, size_t K, size_t N, int cls, float* x) {
    const double s = 1.0 / std::log(16384.0);
    x[0] = (float)(std::log((double)(M ? M : 1)) * s);
    x[1] = (float)(std::log((double)(N ? N : 1)) * s);
    x[2] = (float)(std::log((double)(K ? K : 1)) * s);
    x[3] = (float)(M % 16) / 16.0f;
    x[4] = (float)(N % 16) / 16.0f;
    x[5] = (float)(K % 16) / 16.0f;
    x[6] = (float)cls;
}

int mlp_load(const char* path) {
    std::vector<float> w;
    if (!load_file(path, w)) return -1;
    std::lock_guard<std::mutex> lk(g_model_mu);
    g_env_tried = true;
    g_model.w = std::move(w);
    g_model.loaded = true;
    g_model_gen++;
    return 0;
}

void mlp_unload() {
    std::lock_guard<std::mutex> lk(g_model_mu);
    g_env_tried = true;
    g_model.loaded = false;
    g_model.w.clear();
    g_model_gen++;
}

namespace {

// mlp_predict_host, and what the first weights say (`y0`) where the file holds a
// second set for the split class; `two` tells whether it does.
bool predict_host(size_t M, size_t K, size_t N, int cls, float* y, float* y0, bool* two) {
    std::lock_guard<std::mutex> lk(g_model_mu);
    if (!g_env_tried) {
        // MAXMULSK_MODEL names the weights; unset, the model shipped beside
        // the library (data/picker_model.bin) is used if present; "" or
        // "none" runs without a model (the rule picks).
        g_env_tried = true;
        const char* env = std::getenv("MAXMULSK_MODEL");
        const std::string path = env ? std::string(env) : default_model_path();
        std::vector<float> w;
        if (!path.empty() && path != "none" && load_file(path.c_str(), w)) {
            g_model.w = std::move(w);
            g_model.loaded = true;
        }
    }
    if (!g_model.loaded) return false;
    float x[F];
    mlp_features(M, K, N, cls, x);
    *two = cls == 1 && g_model.w.size() > (size_t)NPARAM;
    host_forward(g_model.w.data() + (*two ? NPARAM : 0), x, y);
    if (*two && y0) host_forward(g_model.w.data(), x, y0);
    return true;
}

// The model's pick for a shape (mlp_predict_plan without its memory).
//
// Weights of the split class's own rank plans by time; how a product is summed is
// not theirs to trade. The plan taken has the precision of the first weights' pick
// (it matters under SPLIT_AUTO) and cuts K into no fewer slices, so that no chain
// of adds is longer. Of 5,400 timed shapes SPLIT_AUTO would otherwise move 12 % to
// 3xTF32's fewer bits, and 9 % would get longer chains, with up to 15 % more error
// against FP64 (243 shapes); with the floor the worst of those has 3.3 % more (37 x
// 664 x 17, twice the slices), the geometric mean is 0.3 % less. On the 800 shapes
// held out the SPLIT_AUTO picks cost 7.1 % over the best plan with the first weights,
// 3.3 % with the second alone, 4.1 % above the floor (geometric mean).
bool predict_plan(size_t M, size_t K, size_t N, int precision, maxmulsk_plan* out, float* margin) {
    const int cls = (precision == MAXMULSK_PREC_FP32) ? 0 : 1;
    float y[O], y0[O];
    bool two = false;
    if (!predict_host(M, K, N, cls, y, y0, &two)) return false;
    maxmulsk_plan cands[O];
    const int n = candidate_plans(cls, cands, O);
    const size_t max_workspace = (64u << 20) + 4 * sizeof(float) * (M * K + K * N + M * N);
    bool runs[O];
    int first = -1;                                                // the first weights' pick
    for (int i = 0; i < n; i++) {
        runs[i] = false;
        if (precision != MAXMULSK_PREC_FP32 && precision != MAXMULSK_PREC_SPLIT_AUTO &&
            cands[i].precision != precision)
            continue;                                              // an explicit split mode
        if (classify_plan(M, K, N, &cands[i]) != MAXMULSK_OK) continue;
        // Plans with outsized split-K scratch were never timed (the autotuner
        // masks them), so the model's estimate for them means nothing.
        if (workspace_bytes(M, K, N, cands[i]) > max_workspace) continue;
        runs[i] = true;
        if (two && (first < 0 || y0[i] < y0[first])) first = i;
    }
    auto slices = [&](const maxmulsk_plan& p) {
        return tc_slice_count((int64_t)M, (int64_t)K, (int64_t)N, p.precision, p.tile_m, p.tile_n, p.split_k);
    };
    const int floor_slices = first >= 0 ? slices(cands[first]) : 0;
    int best = -1, second = -1;
    for (int i = 0; i < n; i++) {
        if (!runs[i]) continue;
        if (first >= 0 && (cands[i].precision != cands[first].precision || slices(cands[i]) < floor_slices)) continue;
        if (best < 0 || y[i] < y[best]) { second = best; best = i; }
        else if (second < 0 || y[i] < y[second]) second = i;
    }
    if (best < 0) return false;
    *out = cands[best];
    // Predicted log-time gap to the runner-up (infinite with one candidate).
    *margin = second < 0 ? INFINITY : y[second] - y[best];
    return true;
}

// The last picks of this thread, by shape: a program calls few shapes many
// times, and a pick (forward pass, 24 or 48 candidates checked and sized) costs
// 29-34 us on the host with scalar multiply-adds, several times a small
// product on the GPU; 4.3-5.7 us with host_linear, 1 us or less found here. A
// 256^3 matmul from Python 34 -> 16 us a call (13 with what came after). Per thread, so no
// lock; a direct-mapped table of fixed size; an entry holds for one model and
// one device, whose work slots decide the workspaces.
struct PickEntry {
    uint64_t gen = 0;
    size_t M = 0, K = 0, N = 0;
    int precision = 0, device = 0;
    bool ok = false;
    float margin = 0.f;
    maxmulsk_plan plan{};
};
constexpr size_t kPickEntries = 128;
thread_local PickEntry t_picks[kPickEntries];

}  // namespace

bool mlp_predict_host(size_t M, size_t K, size_t N, int cls, float* y) {
    bool two = false;
    return predict_host(M, K, N, cls, y, nullptr, &two);
}

bool mlp_predict_plan(size_t M, size_t K, size_t N, int precision, maxmulsk_plan* out, float* margin) {
    if (precision == MAXMULSK_PREC_BF16X9) return false;          // not among the candidates
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t h = (M * 0x9E3779B97F4A7C15ull) ^ (K * 0xC2B2AE3D27D4EB4Full) ^ (N * 0x165667B19E3779F9ull) ^ (uint64_t)precision;
    PickEntry& e = t_picks[(h >> 32) % kPickEntries];
    const uint64_t gen = g_model_gen.load(std::memory_order_acquire);
    if (!(e.gen == gen && e.M == M && e.K == K && e.N == N && e.precision == precision && e.device == dev)) {
        PickEntry f;
        f.gen = gen; f.M = M; f.K = K; f.N = N; f.precision = precision; f.device = dev;
        f.ok = predict_plan(M, K, N, precision, &f.plan, &f.margin);
        e = f;
    }
    if (!e.ok) return false;
    *out = e.plan;
    if (margin) *margin = e.margin;
    return true;
}

}  // namespace mmsk

using namespace mmsk;

extern "C" {

maxmulsk_status maxmulsk_mlp_forward_dev(const float* params, const float* X, int32_t B, float* Z1, float* H1,
                                         float* Z2, float* H2, float* Y, void* stream) {
    if (!params || !X || !H1 || !H2 || !Y || B < 0) return MAXMULSK_ERR_INVALID;
    if (B == 0) return MAXMULSK_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned grid = (unsigned)(((int64_t)B + kFwdRows - 1) / kFwdRows);
    return cuda_status(launch_overlapped(mlp_forward_kernel, dim3(grid), 256, 0, s, 1, params, X, (int)B, Z1, H1, Z2, H2, Y),
                       "mlp forward");
}

maxmulsk_status maxmulsk_mlp_backward_dev(const float* params, const float* X, const float* Z1, const float* H1,
                                          const float* Z2, const float* H2, const float* Y, const float* T,
                                          const float* mask, int32_t B, float count, float* grads, float* work,
                                          float* rowloss, void* stream) {
    if (!params || !X || !Z1 || !H1 || !Z2 || !H2 || !Y || !T || !mask || !grads || !work || !rowloss || B <= 0 ||
        !(count > 0))
        return MAXMULSK_ERR_INVALID;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // Clusters for one wave of two blocks an SM with equal turns of eight rows a
    // block (32 clusters, two turns at 4000 rows: 22.8 us; 63 clusters in two waves
    // 28.0), as far as their gradient sums fit in `work` (B (O + 2 H) floats, NPARAM
    // each). One cluster writes grads itself.
    const int64_t fit = (int64_t)B * (O + 2 * H) / NPARAM;
    const int64_t turns = ((int64_t)B + kBwdRows - 1) / kBwdRows, wave = std::max(1, 2 * device_sm_count());
    const int64_t each = (turns + wave - 1) / wave;
    const int64_t want = (turns + each * kBwdCluster - 1) / (each * kBwdCluster);
    const int nc = (int)std::max<int64_t>(1, std::min(want, fit));
    cudaError_t e = launch_overlapped(mlp_backward_kernel, dim3((unsigned)(nc * kBwdCluster)), 256, 0, s, kBwdCluster, params,
                                      X, Z1, H1, Z2, H2, Y, T, mask, (int)B, 1.0f / count, nc > 1 ? work : grads, rowloss);
    if (e == cudaSuccess && nc > 1)
        e = launch_overlapped(mlp_grad_sum, dim3((NPARAM + 127) / 128), 128, 0, s, 1, (const float*)work, nc, grads);
    return cuda_status(e, "mlp backward");
}

maxmulsk_status maxmulsk_mlp_adam_dev(float* params, const float* grads, float* m, float* v, float lr, float beta1,
                                      float beta2, float eps, int32_t step, void* stream) {
    if (!params || !grads || !m || !v || step < 1) return MAXMULSK_ERR_INVALID;
    const float c1 = 1.0f - std::pow(beta1, (float)step), c2 = 1.0f - std::pow(beta2, (float)step);
    return cuda_status(launch_overlapped(adam_step, dim3(blocks(NPARAM)), 256, 0, static_cast<cudaStream_t>(stream), 1, params,
                                         grads, m, v, (int)NPARAM, lr, beta1, beta2, eps, c1, c2), "mlp adam");
}

maxmulsk_status maxmulsk_mlp_predict_dev(const float* params, const float* X, const float* mask, int32_t B,
                                         float* work, float* Y, int32_t* best, void* stream) {
    if (!params || !X || !Y || !work || B < 0) return MAXMULSK_ERR_INVALID;
    if (B == 0) return MAXMULSK_OK;
    float* H1 = work;
    float* H2 = work + (size_t)B * H;
    maxmulsk_status st = maxmulsk_mlp_forward_dev(params, X, B, nullptr, H1, nullptr, H2, Y, stream);
    if (st != MAXMULSK_OK) return st;
    if (best && mask) {
        masked_argmin<<<blocks(B), 256, 0, static_cast<cudaStream_t>(stream)>>>(Y, mask, B, best);
        return cuda_status(cudaGetLastError(), "mlp argmin");
    }
    return MAXMULSK_OK;
}

maxmulsk_status maxmulsk_mlp_features(size_t M, size_t K, size_t N, int32_t cls, float* out) {
    if (!out) return MAXMULSK_ERR_INVALID;
    mlp_features(M, K, N, cls, out);
    return MAXMULSK_OK;
}

maxmulsk_status maxmulsk_mlp_predict_host(size_t M, size_t K, size_t N, int32_t cls, float* out) {
    if (!out) return MAXMULSK_ERR_INVALID;
    return mlp_predict_host(M, K, N, cls, out) ? MAXMULSK_OK : MAXMULSK_ERR_UNSUPPORTED;
}

maxmulsk_status maxmulsk_model_load(const char* path) {
    if (!path) { mlp_unload(); return MAXMULSK_OK; }
    return mlp_load(path) == 0 ? MAXMULSK_OK : MAXMULSK_ERR_INVALID;
}

}  // extern "C"
