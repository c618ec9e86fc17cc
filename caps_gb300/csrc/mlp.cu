// mlp.cu -- a small MLP trained on the GPU that predicts log|logdetD(xi, m)|.
//
// Network: 5 inputs -> 64 -> 64 -> 64 -> 1, SiLU activations, FP32.  Inputs are
// the normalised features (log R/L, 2 xi L/c, m/sqrt(R/L), omega_p, gamma) built by the
// caller.  Hand-written kernels:
//   k_mlp_fwdbwd  one CTA of 256 threads walks a slice of the batch 16 samples at a
//                 time: forward pass, MSE loss, backward pass; a thread owns one
//                 neuron for four samples in the passes and 16 weights of each square
//                 layer in the gradient (in registers, so no atomics), written out per CTA;
//   k_mlp_reduce  fixed-order sum of the CTA partials (deterministic gradients);
//   k_mlp_adam    Adam update, one thread per parameter;
//   k_mlp_fwd     inference.
// Parameter layout (floats): W1[64][5] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] W4[64] b4[1].
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <random>
#include <vector>

#include "../../include/libcaps.h"
#include "internal.h"

namespace capsgpu {

constexpr int HN = 64, NIN = 5;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + HN * NIN, OFF_W2 = OFF_B1 + HN, OFF_B2 = OFF_W2 + HN * HN,
              OFF_W3 = OFF_B2 + HN, OFF_B3 = OFF_W3 + HN * HN, OFF_W4 = OFF_B3 + HN, OFF_B4 = OFF_W4 + HN,
              NPARAM = OFF_B4 + 1;

__device__ __forceinline__ float sig(float x) { return 1.0f / (1.0f + expf(-x)); }

// shared memory in floats: parameters (rows of the square layers padded to 65), then per layer the
// activations of 16 samples, [neuron][sample]
constexpr int SB = 16, MLP_NT = 256;
constexpr int SW1 = 0, SW2 = SW1 + HN * NIN, SW3 = SW2 + HN * (HN + 1), SB1 = SW3 + HN * (HN + 1), SB2 = SB1 + HN, SB3 = SB2 + HN,
              SW4 = SB3 + HN, SH1 = SW4 + HN + 4, SH2 = SH1 + HN * SB, SH3 = SH2 + HN * SB, SD3 = SH3 + HN * SB, SD2 = SD3 + HN * SB,
              SX = SD2 + HN * SB, SRED = SX + NIN * SB, SMEMF = SRED + 8 * 4 + 2 * SB;
static_assert(SH1 % 4 == 0 && SX % 4 == 0, "vector loads of four samples");

// forward (and optionally backward) of the samples [blockIdx.x*per, ...); y == nullptr: inference only.
// Bound by latency (2600 samples: 163 CTAs of one batch): one sample after the other with a thread per neuron took
// 150 us, 16 at once take 24 (loss, gradient and prediction of 2600 samples, copies included: 0.378 -> 0.095 ms).
__global__ void __launch_bounds__(MLP_NT) k_mlp_fwdbwd(const float *__restrict__ P, const float *__restrict__ X, const float *__restrict__ Y,
                                                       int n, int per, float *out, float *gpart, float *lpart)
{
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, j = tid & 63, q = tid >> 6, lane = tid & 31, warp = tid >> 5; // neuron, group of four samples
    for (int i = tid; i < NPARAM; i += MLP_NT) {
        const float w = P[i];
        if (i < OFF_B1) sm[SW1 + i] = w;
        else if (i < OFF_W2) sm[SB1 + i - OFF_B1] = w;
        else if (i < OFF_B2) sm[SW2 + (i - OFF_W2) / HN * (HN + 1) + (i - OFF_W2) % HN] = w;
        else if (i < OFF_W3) sm[SB2 + i - OFF_B2] = w;
        else if (i < OFF_B3) sm[SW3 + (i - OFF_W3) / HN * (HN + 1) + (i - OFF_W3) % HN] = w;
        else if (i < OFF_W4) sm[SB3 + i - OFF_B3] = w;
        else sm[SW4 + i - OFF_W4] = w; // W4, b4
    }
    const int s0 = blockIdx.x * per, s1 = min(n, s0 + per);
    float loss = 0.0f;
    // this thread's gradients: W2[j][16 q ..], W3[j][16 q ..]; q = 0: W1[j], b1..b3[j], W4[j]; thread 0: b4
    float g2[16], g3[16], g1[NIN], gb1 = 0, gb2 = 0, gb3 = 0, gw4 = 0, gb4 = 0;
#pragma unroll
    for (int k = 0; k < 16; k++) g2[k] = g3[k] = 0.0f;
#pragma unroll
    for (int c = 0; c < NIN; c++) g1[c] = 0.0f;
    auto vec = [&](int layer, int k, int s) { return *reinterpret_cast<const float4 *>(sm + layer + k * SB + s); };
    for (int base = s0; base < s1; base += SB) {
        __syncthreads(); // the parameters are in; the last batch's activations have been read
        if (tid < SB * NIN) {
            const int s = tid / NIN, c = tid % NIN;
            sm[SX + c * SB + s] = X[(size_t)min(base + s, s1 - 1) * NIN + c]; // past the end: the last sample again, with d = 0
        }
        __syncthreads();
        float sg1[4], z1[4], sg2[4], z2[4], sg3[4], z3[4], h[4];
        // one layer: z = W h + b for four samples, h' = z sig(z)
        auto act = [&](int layer, const float (&z)[4], float (&sg)[4]) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                sg[i] = sig(z[i]);
                h[i] = z[i] * sg[i];
            }
            *reinterpret_cast<float4 *>(sm + layer + j * SB + 4 * q) = make_float4(h[0], h[1], h[2], h[3]);
        };
        auto dot = [&](const float *w, int step, int layer, float z0, float (&z)[4]) {
            z[0] = z[1] = z[2] = z[3] = z0;
#pragma unroll 16
            for (int k = 0; k < HN; k++) {
                const float a = w[k * step];
                const float4 v = vec(layer, k, 4 * q);
                z[0] = fmaf(a, v.x, z[0]);
                z[1] = fmaf(a, v.y, z[1]);
                z[2] = fmaf(a, v.z, z[2]);
                z[3] = fmaf(a, v.w, z[3]);
            }
        };
        z1[0] = z1[1] = z1[2] = z1[3] = sm[SB1 + j];
#pragma unroll
        for (int c = 0; c < NIN; c++) {
            const float a = sm[SW1 + j * NIN + c];
            const float4 v = vec(SX, c, 4 * q);
            z1[0] = fmaf(a, v.x, z1[0]);
            z1[1] = fmaf(a, v.y, z1[1]);
            z1[2] = fmaf(a, v.z, z1[2]);
            z1[3] = fmaf(a, v.w, z1[3]);
        }
        act(SH1, z1, sg1);
        __syncthreads();
        dot(sm + SW2 + j * (HN + 1), 1, SH1, sm[SB2 + j], z2);
        act(SH2, z2, sg2);
        __syncthreads();
        dot(sm + SW3 + j * (HN + 1), 1, SH2, sm[SB3 + j], z3);
        act(SH3, z3, sg3);
        // output: b4 + sum_j W4[j] h3[j], over the two warps of a group of samples
        const float w4 = sm[SW4 + j];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float t = w4 * h[i];
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) sm[SRED + warp * 4 + i] = t;
        }
        __syncthreads();
        if (tid < SB) {
            const int s = base + tid;
            const float yhat = sm[SRED + (tid >> 2) * 8 + (tid & 3)] + sm[SRED + (tid >> 2) * 8 + 4 + (tid & 3)] + sm[SW4 + HN];
            if (!Y) {
                if (s < s1) out[s] = yhat;
            } else {
                const float e = s < s1 ? yhat - Y[s] : 0.0f;
                sm[SRED + 32 + tid] = 2.0f * e / n; // d loss / d yhat, loss = mean (yhat - y)^2
                sm[SRED + 32 + SB + tid] = e * e;
            }
        }
        if (!Y) continue;
        __syncthreads();
        float d4[4], dz[4];
#pragma unroll
        for (int i = 0; i < 4; i++) d4[i] = sm[SRED + 32 + 4 * q + i];
        if (tid == 0)
            for (int s = 0; s < SB; s++) {
                loss += sm[SRED + 32 + SB + s];
                gb4 += sm[SRED + 32 + s];
            }
#pragma unroll
        for (int i = 0; i < 4; i++) dz[i] = d4[i] * w4 * sg3[i] * (1.0f + z3[i] * (1.0f - sg3[i]));
        *reinterpret_cast<float4 *>(sm + SD3 + j * SB + 4 * q) = make_float4(dz[0], dz[1], dz[2], dz[3]);
        __syncthreads();
        // gradient of a square layer: G[j][16 q + k] += sum_s d[j][s] h[16 q + k][s]
        auto outer = [&](int dl, int hl, float (&g)[16]) {
            float d[SB];
#pragma unroll
            for (int s = 0; s < SB; s += 4) {
                const float4 v = vec(dl, j, s);
                d[s] = v.x; d[s + 1] = v.y; d[s + 2] = v.z; d[s + 3] = v.w;
            }
#pragma unroll
            for (int k = 0; k < 16; k++)
#pragma unroll
                for (int s = 0; s < SB; s += 4) {
                    const float4 v = vec(hl, 16 * q + k, s);
                    g[k] = fmaf(d[s], v.x, g[k]);
                    g[k] = fmaf(d[s + 1], v.y, g[k]);
                    g[k] = fmaf(d[s + 2], v.z, g[k]);
                    g[k] = fmaf(d[s + 3], v.w, g[k]);
                }
            float t = 0.0f;
#pragma unroll
            for (int s = 0; s < SB; s++) t += d[s];
            return t;
        };
        const float t3 = outer(SD3, SH2, g3);
        float a[4];
        dot(sm + SW3 + j, HN + 1, SD3, 0.0f, a); // a2 = W3^T d3
#pragma unroll
        for (int i = 0; i < 4; i++) dz[i] = a[i] * sg2[i] * (1.0f + z2[i] * (1.0f - sg2[i]));
        *reinterpret_cast<float4 *>(sm + SD2 + j * SB + 4 * q) = make_float4(dz[0], dz[1], dz[2], dz[3]);
        if (q == 0) {
            gb3 += t3;
#pragma unroll
            for (int s = 0; s < SB; s++) gw4 = fmaf(sm[SRED + 32 + s], sm[SH3 + j * SB + s], gw4);
        }
        __syncthreads();
        const float t2 = outer(SD2, SH1, g2);
        dot(sm + SW2 + j, HN + 1, SD2, 0.0f, a); // a1 = W2^T d2
#pragma unroll
        for (int i = 0; i < 4; i++) dz[i] = a[i] * sg1[i] * (1.0f + z1[i] * (1.0f - sg1[i]));
        __syncthreads(); // d3 has been read: d1 takes its place
        *reinterpret_cast<float4 *>(sm + SD3 + j * SB + 4 * q) = make_float4(dz[0], dz[1], dz[2], dz[3]);
        __syncthreads();
        if (q == 0) {
            gb2 += t2;
#pragma unroll
            for (int s = 0; s < SB; s++) {
                const float d = sm[SD3 + j * SB + s];
                gb1 += d;
#pragma unroll
                for (int c = 0; c < NIN; c++) g1[c] = fmaf(d, sm[SX + c * SB + s], g1[c]);
            }
        }
    }
    if (!Y) return;
    float *g = gpart + (size_t)blockIdx.x * NPARAM;
#pragma unroll
    for (int k = 0; k < 16; k++) {
        g[OFF_W2 + j * HN + 16 * q + k] = g2[k];
        g[OFF_W3 + j * HN + 16 * q + k] = g3[k];
    }
    if (q == 0) {
#pragma unroll
        for (int c = 0; c < NIN; c++) g[OFF_W1 + j * NIN + c] = g1[c];
        g[OFF_B1 + j] = gb1;
        g[OFF_B2 + j] = gb2;
        g[OFF_B3 + j] = gb3;
        g[OFF_W4 + j] = gw4;
    }
    if (tid == 0) {
        g[OFF_B4] = gb4;
        lpart[blockIdx.x] = loss;
    }
}

// grid ceil(NPARAM / 32): 32 parameters by 8 slices of the CTAs each, slices added in order; the loss by
// one more block
__global__ void __launch_bounds__(256) k_mlp_reduce(const float *gpart, const float *lpart, int nblk, float *grad, float *loss, int n)
{
    __shared__ float part[8][33];
    const int c = threadIdx.x & 31, sl = threadIdx.x >> 5, i = blockIdx.x * 32 + c;
    const bool is_loss = blockIdx.x == gridDim.x - 1;
    const int per = (nblk + 7) / 8, b1 = min(nblk, (sl + 1) * per);
    float s = 0.0f;
    if (is_loss) {
        if (c == 0)
            for (int b = sl * per; b < b1; b++) s += lpart[b];
    } else if (i < NPARAM)
        for (int b = sl * per; b < b1; b++) s += gpart[(size_t)b * NPARAM + i];
    part[sl][c] = s;
    __syncthreads();
    if (sl) return;
    for (int k = 1; k < 8; k++) s += part[k][c];
    if (is_loss) {
        if (c == 0) *loss = s / n;
    } else if (i < NPARAM)
        grad[i] = s;
}
constexpr int MLP_RED_GRID = (NPARAM + 31) / 32 + 1;

__global__ void k_mlp_adam(float *P, const float *grad, float *m1, float *m2, int t, float lr)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NPARAM) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float gi = grad[i];
    m1[i] = b1 * m1[i] + (1 - b1) * gi;
    m2[i] = b2 * m2[i] + (1 - b2) * gi * gi;
    const float mh = m1[i] / (1 - powf(b1, (float)t)), vh = m2[i] / (1 - powf(b2, (float)t));
    P[i] -= lr * mh / (sqrtf(vh) + eps);
}

} // namespace capsgpu

using namespace capsgpu;

struct caps_mlp {
    float *P = nullptr, *G = nullptr, *M1 = nullptr, *M2 = nullptr, *loss = nullptr;
    float *X = nullptr, *Y = nullptr, *out = nullptr, *gpart = nullptr, *lpart = nullptr; // Y behind X
    size_t cap = 0, blk_cap = 0;
    int t = 0;
};

static void mlp_reserve(caps_mlp_t *m, size_t n)
{
    if (n > m->cap) {
        if (m->X) { CK(cudaFree(m->X)); CK(cudaFree(m->out)); }
        m->cap = std::max(n, (size_t)2048);
        CK(cudaMalloc(&m->X, m->cap * (NIN + 1) * sizeof(float)));
        CK(cudaMalloc(&m->out, m->cap * sizeof(float)));
    }
}

// Pinned memory that samples, gradients and predictions pass through, one block for all networks: taken by the first
// network that is made, given back with the last.  Six pageable copies, each with a synchronisation, were half of the
// time of a loss, gradient and prediction of 2600 samples (121 us; 95 so); a block per network, taken at its
// first call, cost that call up to 110 us (a new network's first loss, gradient and prediction 322 us, 211 so; the other
// 110 are its device memory).  A call holds
// the lock while its data are in the block; what does not fit goes by pageable copies.
static constexpr size_t MLP_STAGE = 16384 * (NIN + 1); // floats
static_assert(NPARAM + 1 <= MLP_STAGE, "gradient and loss fit");
static struct {
    std::mutex mu;
    float *p = nullptr;
    int users = 0;
} g_stage;

static void stage_enter()
{
    std::lock_guard<std::mutex> lk(g_stage.mu);
    if (g_stage.users++ == 0) CK(cudaMallocHost(&g_stage.p, MLP_STAGE * sizeof(float)));
}
static void stage_leave()
{
    std::lock_guard<std::mutex> lk(g_stage.mu);
    if (--g_stage.users == 0) {
        CK(cudaFreeHost(g_stage.p));
        g_stage.p = nullptr;
    }
}

// n samples and (y != nullptr) their values to the device, by one copy; the caller holds the lock and synchronises before
// it lets go
static void mlp_upload(caps_mlp_t *m, const float *X, const float *y, int n)
{
    mlp_reserve(m, n);
    const size_t nx = (size_t)n * NIN, ny = y ? n : 0;
    m->Y = m->X + nx;
    if (nx + ny > MLP_STAGE) {
        CK(cudaMemcpy(m->X, X, nx * sizeof(float), cudaMemcpyHostToDevice));
        if (y) CK(cudaMemcpy(m->Y, y, ny * sizeof(float), cudaMemcpyHostToDevice));
        return;
    }
    std::copy(X, X + nx, g_stage.p);
    if (y) std::copy(y, y + ny, g_stage.p + nx);
    CK(cudaMemcpyAsync(m->X, g_stage.p, (nx + ny) * sizeof(float), cudaMemcpyHostToDevice, 0));
}

static int mlp_blocks(int n, int *per)
{
    // whole batches of SB samples per CTA, at most two CTAs per SM
    const int nb = (n + SB - 1) / SB, nblk = std::max(1, std::min(304, nb));
    *per = (nb + nblk - 1) / nblk * SB;
    return (n + *per - 1) / *per;
}

static void mlp_reserve_blocks(caps_mlp_t *m, size_t nblk)
{
    if (nblk > m->blk_cap) {
        if (m->gpart) { CK(cudaFree(m->gpart)); CK(cudaFree(m->lpart)); }
        m->blk_cap = std::max(nblk, (size_t)304);
        CK(cudaMalloc(&m->gpart, m->blk_cap * NPARAM * sizeof(float)));
        CK(cudaMalloc(&m->lpart, m->blk_cap * sizeof(float)));
    }
}

static constexpr size_t MLP_SMEM = SMEMF * sizeof(float);

extern "C" int caps_mlp_nparams(void) { return NPARAM; }

extern "C" caps_mlp_t *caps_mlp_create(unsigned seed)
{
    caps_mlp_t *m = new caps_mlp_t();
    stage_enter();
    std::vector<float> p(NPARAM, 0.0f);
    std::mt19937 rng(seed);
    auto init = [&](int off, int fan_in, int count) {
        std::normal_distribution<float> d(0.0f, std::sqrt(2.0f / fan_in));
        for (int i = 0; i < count; i++) p[off + i] = d(rng);
    };
    init(OFF_W1, NIN, HN * NIN);
    init(OFF_W2, HN, HN * HN);
    init(OFF_W3, HN, HN * HN);
    init(OFF_W4, HN, HN);
    CK(cudaMalloc(&m->P, NPARAM * sizeof(float)));
    CK(cudaMalloc(&m->G, (NPARAM + 1) * sizeof(float))); // the loss behind it
    m->loss = m->G + NPARAM;
    CK(cudaMalloc(&m->M1, NPARAM * sizeof(float)));
    CK(cudaMalloc(&m->M2, NPARAM * sizeof(float)));
    CK(cudaMemcpy(m->P, p.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice));
    CK(cudaMemset(m->M1, 0, NPARAM * sizeof(float)));
    CK(cudaMemset(m->M2, 0, NPARAM * sizeof(float)));
    static bool attr = false;
    if (!attr) {
        CK(cudaFuncSetAttribute(k_mlp_fwdbwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MLP_SMEM));
        attr = true;
    }
    return m;
}

extern "C" void caps_mlp_free(caps_mlp_t *m)
{
    if (!m) return;
    for (float *p : {m->P, m->G, m->M1, m->M2, m->X, m->out, m->gpart, m->lpart})
        if (p) CK(cudaFree(p));
    stage_leave();
    delete m;
}

extern "C" void caps_mlp_get_params(caps_mlp_t *m, float *out) { CK(cudaMemcpy(out, m->P, NPARAM * sizeof(float), cudaMemcpyDeviceToHost)); }
extern "C" void caps_mlp_set_params(caps_mlp_t *m, const float *in) { CK(cudaMemcpy(m->P, in, NPARAM * sizeof(float), cudaMemcpyHostToDevice)); }

extern "C" double caps_mlp_loss_grad(caps_mlp_t *m, const float *X, const float *y, int n, float *grad)
{
    std::lock_guard<std::mutex> lk(g_stage.mu);
    mlp_upload(m, X, y, n);
    int per;
    const int nblk = mlp_blocks(n, &per);
    mlp_reserve_blocks(m, nblk);
    k_mlp_fwdbwd<<<nblk, MLP_NT, MLP_SMEM>>>(m->P, m->X, m->Y, n, per, nullptr, m->gpart, m->lpart);
    k_mlp_reduce<<<MLP_RED_GRID, 256>>>(m->gpart, m->lpart, nblk, m->G, m->loss, n);
    COUNT_LAUNCH(2);
    CK(cudaGetLastError());
    // gradient and loss lie one after the other
    CK(cudaMemcpyAsync(g_stage.p, m->G, (NPARAM + 1) * sizeof(float), cudaMemcpyDeviceToHost, 0));
    CK(cudaStreamSynchronize(0));
    if (grad) std::copy(g_stage.p, g_stage.p + NPARAM, grad);
    return g_stage.p[NPARAM];
}

extern "C" double caps_mlp_train(caps_mlp_t *m, const float *X, const float *y, int n, int epochs, float lr)
{
    {
        std::lock_guard<std::mutex> lk(g_stage.mu);
        mlp_upload(m, X, y, n);
        CK(cudaStreamSynchronize(0)); // other networks may use the block during the epochs
    }
    int per;
    const int nblk = mlp_blocks(n, &per);
    mlp_reserve_blocks(m, nblk);
    for (int e = 0; e < epochs; e++) {
        // full-batch Adam; cosine-decayed step size
        const float lr_e = lr * 0.5f * (1.0f + cosf(3.14159265f * e / epochs)) + 1e-5f;
        k_mlp_fwdbwd<<<nblk, MLP_NT, MLP_SMEM>>>(m->P, m->X, m->Y, n, per, nullptr, m->gpart, m->lpart);
        k_mlp_reduce<<<MLP_RED_GRID, 256>>>(m->gpart, m->lpart, nblk, m->G, m->loss, n);
        k_mlp_adam<<<(NPARAM + 255) / 256, 256>>>(m->P, m->G, m->M1, m->M2, ++m->t, lr_e);
        COUNT_LAUNCH(3);
    }
    CK(cudaGetLastError());
    float loss;
    CK(cudaMemcpy(&loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
    return epochs > 0 ? loss : 0.0;
}

extern "C" void caps_mlp_predict(caps_mlp_t *m, const float *X, int n, float *y)
{
    if (n <= 0) return;
    std::lock_guard<std::mutex> lk(g_stage.mu);
    mlp_upload(m, X, nullptr, n);
    int per;
    const int nblk = mlp_blocks(n, &per);
    k_mlp_fwdbwd<<<nblk, MLP_NT, MLP_SMEM>>>(m->P, m->X, nullptr, n, per, m->out, nullptr, nullptr);
    COUNT_LAUNCH(1);
    CK(cudaGetLastError());
    if ((size_t)n > MLP_STAGE) {
        CK(cudaMemcpy(y, m->out, n * sizeof(float), cudaMemcpyDeviceToHost));
        return;
    }
    CK(cudaMemcpyAsync(g_stage.p, m->out, n * sizeof(float), cudaMemcpyDeviceToHost, 0));
    CK(cudaStreamSynchronize(0));
    std::copy(g_stage.p, g_stage.p + n, y);
}

// features of one (geometry, material, xi_, m): the normalisation the network is trained with.
// The frequency enters as 2 xi L / c = 2 xi_ / (1 + R/L), the exponent of the round trip's
// decay e^{-2 xi L / c}, and m as m / sqrt(R/L), the scale on which the m sum of a
// plane-sphere geometry ends; log(R/L) carries what is left.  With these, geometries of
// different R/L put their values on nearly the same surface, so a network trained on small
// R/L serves larger ones.
extern "C" void caps_mlp_features(double RbyL, double xi_, int m, double omegap_eV, double gamma_eV, float *x)
{
    x[0] = (float)(log(RbyL) / 5.0);
    x[1] = (float)(2.0 * xi_ / (1.0 + RbyL) / 8.0);
    x[2] = (float)(m / sqrt(RbyL) / 10.0);
    x[3] = (float)(omegap_eV / 10.0);
    x[4] = (float)(gamma_eV / 0.05);
}
