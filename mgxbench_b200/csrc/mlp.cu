// mlp.cu -- the autotuner's learned cost model: a 3-layer FP32 MLP (6 -> 64 -> 64 -> 2, tanh),
// trained and run on the GPU by these kernels.
//
// Inputs (standardised by the caller): log2 M, log2 N, log2 K, input exponent range, tile shape
// id, split count.  Outputs: predicted (standardised) log runtime and log10 normwise error.
// Loss: sum_o w_o (out_o - y_o)^2 / batch.  Optimiser: Adam.
//
// Parameter vector layout (floats):
//   W1[64][6] | b1[64] | W2[64][64] | b2[64] | W3[2][64] | b3[2]     (4738 values)
#include <cmath>

#include "mgx_common.cuh"

namespace mgx {
namespace mlp {

constexpr int NI = 6, NH = 64, NO = 2;
constexpr int OW1 = 0, OB1 = OW1 + NH * NI, OW2 = OB1 + NH, OB2 = OW2 + NH * NH, OW3 = OB2 + NH,
              OB3 = OW3 + NO * NH, NPARAM = OB3 + NO;
constexpr int SPB = 16;        // samples of a block
constexpr int THREADS = 256;
constexpr int SG = 4;          // samples of a thread: thread (unit j = t % 64, samples 4 (t / 64) ...)
static_assert(THREADS == NH * (SPB / SG), "one thread per unit and sample group");

// The work is a few MFLOP, so the kernels are bound by the latency of their phases: each thread
// computes one hidden unit for four samples from registers.  Weights are staged with rows of 68
// floats (W1: 7) and activations transposed, [unit][sample] with rows of 20 floats, so that every
// shared-memory access, 16 bytes wide where it can be, is free of bank conflicts.  (With the
// parameter vector's own rows of 64, the lanes of a warp read one bank 32 deep; with one thread per
// sample, the activations lived in local memory.)  Gradients, update and prediction at a batch of
// 256: 47 + 4 + 24 us of kernels before; now 10.6 us in all, replayed from a CUDA graph.
constexpr int W1_LD = 7, W2_LD = 68, S_LD = 20;

struct Net {
    float w1[NH * W1_LD], b1[NH], w3[NO * NH], b3[NO];
    __align__(16) float w2[NH * W2_LD];
    float b2[NH];
    float x[SPB][NI];
    __align__(16) float h1[NH][S_LD];
    __align__(16) float h2[NH][S_LD];
};

// All of a thread's loads are issued before its first store: one trip to memory, not one per step.
__device__ __forceinline__ void load_params(Net &n, const float *__restrict__ P)
{
    const int t = threadIdx.x;
    float w2[NH * NH / THREADS], w1[2], r[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NH * NH / THREADS; ++i) w2[i] = P[OW2 + i * THREADS + t];
    w1[0] = P[OW1 + t];
    w1[1] = t < NH * NI - THREADS ? P[OW1 + THREADS + t] : 0.f;
    // the rest, b1 | b2 and W3 | b3, each a run of the vector
    if (t < 2 * NH) r[0] = t < NH ? P[OB1 + t] : P[OB2 + t - NH];
    if (t < NO * NH + NO) r[1] = P[OW3 + t];
#pragma unroll
    for (int i = 0; i < NH * NH / THREADS; ++i) n.w2[(i * (THREADS / NH) + t / NH) * W2_LD + t % NH] = w2[i];
    n.w1[t / NI * W1_LD + t % NI] = w1[0];
    if (t < NH * NI - THREADS) n.w1[(THREADS + t) / NI * W1_LD + (THREADS + t) % NI] = w1[1];
    if (t < 2 * NH) (t < NH ? n.b1[t] : n.b2[t - NH]) = r[0];
    if (t < NO * NH + NO) (t < NO * NH ? n.w3[t] : n.b3[t - NO * NH]) = r[1];
}

// Samples [s0, s0 + ns) into shared memory, the rest of the SPB as zeros.
__device__ __forceinline__ void load_samples(Net &n, const float *__restrict__ X, int s0, int ns)
{
    for (int i = threadIdx.x; i < SPB * NI; i += THREADS) {
        const int s = i / NI;
        n.x[s][i % NI] = (s < ns) ? X[(size_t)s0 * NI + i] : 0.f;
    }
}

__device__ __forceinline__ float4 f4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Both hidden layers of the SPB samples (the caller synchronises before and after).
__device__ __forceinline__ void hidden_layers(Net &n)
{
    const int j = threadIdx.x % NH, s = threadIdx.x / NH * SG;
    float a[SG];
#pragma unroll
    for (int u = 0; u < SG; ++u) {
        a[u] = n.b1[j];
#pragma unroll
        for (int q = 0; q < NI; ++q) a[u] = fmaf(n.w1[j * W1_LD + q], n.x[s + u][q], a[u]);
        a[u] = tanhf(a[u]);
    }
    *reinterpret_cast<float4 *>(&n.h1[j][s]) = make_float4(a[0], a[1], a[2], a[3]);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < SG; ++u) a[u] = n.b2[j];
#pragma unroll 4
    for (int k = 0; k < NH; k += 4) {
        const float4 w = f4(&n.w2[j * W2_LD + k]);
        const float wk[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const float4 h = f4(&n.h1[k + v][s]);
            a[0] = fmaf(wk[v], h.x, a[0]);
            a[1] = fmaf(wk[v], h.y, a[1]);
            a[2] = fmaf(wk[v], h.z, a[2]);
            a[3] = fmaf(wk[v], h.w, a[3]);
        }
    }
    *reinterpret_cast<float4 *>(&n.h2[j][s]) = make_float4(tanhf(a[0]), tanhf(a[1]), tanhf(a[2]), tanhf(a[3]));
}

// Output o of sample s.
__device__ __forceinline__ float output_of(const Net &n, int s, int o)
{
    float a = n.b3[o];
#pragma unroll 16
    for (int k = 0; k < NH; ++k) a = fmaf(n.w3[o * NH + k], n.h2[k][s], a);
    return a;
}

// Inference: SPB samples at a time, parameters staged once per block.
__global__ void __launch_bounds__(THREADS) forward_kernel(const float *__restrict__ X, int batch,
                                                          const float *__restrict__ params, float *__restrict__ out)
{
    __shared__ Net n;
    pdl_wait();
    load_params(n, params);
    for (int s0 = blockIdx.x * SPB; s0 < batch; s0 += gridDim.x * SPB) {
        const int ns = min(SPB, batch - s0);
        load_samples(n, X, s0, ns);
        __syncthreads();
        hidden_layers(n);
        __syncthreads();
        if (threadIdx.x < SPB * NO) {
            const int s = threadIdx.x % SPB, o = threadIdx.x / SPB;
            const float v = output_of(n, s, o);
            if (s < ns) out[(size_t)(s0 + s) * NO + o] = v;
        }
        __syncthreads();  // the next samples overwrite h2
    }
}

// The same for large batches: one thread per sample, the parameters broadcast from shared memory.  A sample
// group's two barriers and unit tiles cost more here than the tiles save: 131072 samples 61.2 us by
// groups, 56.7 so; 1,000,000 446 and 362.  Smaller batches do not fill the SMs: 98304 46.2 and 49.3, 4096 4.5
// and 22.6.  Both add in the same order, so the rule changes no bit.
constexpr int SAMPLE_THREADS_BATCH = 131072;

__device__ __forceinline__ void forward_sample(const float *P, const float *x, float *h1, float *h2, float *out)
{
    for (int j = 0; j < NH; ++j) {
        float a = P[OB1 + j];
        for (int i = 0; i < NI; ++i) a = fmaf(P[OW1 + j * NI + i], x[i], a);
        h1[j] = tanhf(a);
    }
    for (int j = 0; j < NH; ++j) {
        float a = P[OB2 + j];
        for (int k = 0; k < NH; ++k) a = fmaf(P[OW2 + j * NH + k], h1[k], a);
        h2[j] = tanhf(a);
    }
    for (int o = 0; o < NO; ++o) {
        float a = P[OB3 + o];
        for (int k = 0; k < NH; ++k) a = fmaf(P[OW3 + o * NH + k], h2[k], a);
        out[o] = a;
    }
}

__global__ void __launch_bounds__(THREADS) forward_samples_kernel(const float *__restrict__ X, int batch,
                                                                  const float *__restrict__ params,
                                                                  float *__restrict__ out)
{
    __shared__ float P[NPARAM];
    pdl_wait();
    for (int i = threadIdx.x; i < NPARAM; i += blockDim.x) P[i] = params[i];
    __syncthreads();
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= batch) return;
    float x[NI], h1[NH], h2[NH], o[NO];
    for (int i = 0; i < NI; ++i) x[i] = X[s * NI + i];
    forward_sample(P, x, h1, h2, o);
    for (int k = 0; k < NO; ++k) out[s * NO + k] = o[k];
}

// grads = 0, *loss = 0, in one launch.  It lets the gradient kernel start only once every kernel before
// it has finished, so that kernel may read its inputs before its own wait.
__global__ void __launch_bounds__(THREADS) zero_kernel(float *__restrict__ grads, float *__restrict__ loss)
{
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * THREADS + threadIdx.x;
    if (i < NPARAM) grads[i] = 0.f;
    if (i == NPARAM) *loss = 0.f;
}

// Gradients of the loss over `batch` samples; each block handles SPB samples and adds its share
// into grads and loss (zeroed by zero_kernel, whose run the passes up to the wait overlap).
__global__ void __launch_bounds__(THREADS) grad_kernel(const float *__restrict__ X, const float *__restrict__ Y,
                                                       const float *__restrict__ wout, int batch,
                                                       const float *__restrict__ params, float *__restrict__ grads,
                                                       float *__restrict__ loss)
{
    __shared__ Net n;
    __shared__ __align__(16) float d2[NH][S_LD];
    __shared__ __align__(16) float d1[NH][S_LD];
    __shared__ float dout[SPB][NO];
    const int t = threadIdx.x;
    const int s0 = blockIdx.x * SPB;
    const int ns = min(SPB, batch - s0);
    load_params(n, params);
    load_samples(n, X, s0, ns);
    __syncthreads();
    hidden_layers(n);
    __syncthreads();
    // output, loss and its gradient (the first warp)
    float lpart = 0.f;
    if (t < SPB * NO) {
        const int s = t / NO, o = t % NO;
        float g = 0.f;
        if (s < ns) {
            const float diff = output_of(n, s, o) - Y[(size_t)(s0 + s) * NO + o];
            lpart = wout[o] * diff * diff / batch;
            g = 2.f * wout[o] * diff / batch;
        }
        dout[s][o] = g;
        for (int k = 16; k > 0; k >>= 1) lpart += __shfl_xor_sync(0xffffffffu, lpart, k);
    }
    __syncthreads();
    // dH2 = (dout W3) * (1 - h2^2)
    const int j = t % NH, s = t / NH * SG;
    {
        const float4 h = f4(&n.h2[j][s]);
        const float hs[SG] = {h.x, h.y, h.z, h.w};
        float d[SG];
#pragma unroll
        for (int u = 0; u < SG; ++u) {
            float a = 0.f;
#pragma unroll
            for (int o = 0; o < NO; ++o) a = fmaf(dout[s + u][o], n.w3[o * NH + j], a);
            d[u] = a * (1.f - hs[u] * hs[u]);
        }
        *reinterpret_cast<float4 *>(&d2[j][s]) = make_float4(d[0], d[1], d[2], d[3]);
    }
    __syncthreads();
    // dH1 = (dH2 W2) * (1 - h1^2): thread (k, samples), k = its own unit
    {
        float a[SG] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
        for (int i = 0; i < NH; ++i) {
            const float w = n.w2[i * W2_LD + j];
            const float4 d = f4(&d2[i][s]);
            a[0] = fmaf(d.x, w, a[0]);
            a[1] = fmaf(d.y, w, a[1]);
            a[2] = fmaf(d.z, w, a[2]);
            a[3] = fmaf(d.w, w, a[3]);
        }
        const float4 h = f4(&n.h1[j][s]);
        *reinterpret_cast<float4 *>(&d1[j][s]) = make_float4(a[0] * (1.f - h.x * h.x), a[1] * (1.f - h.y * h.y),
                                                             a[2] * (1.f - h.z * h.z), a[3] * (1.f - h.w * h.w));
    }
    // dW2: thread (four rows j, columns k = kx + 16 i), summed over the samples in order
    float g2[4][4];
    const int kx = t % 16, jy = t / 16 * 4;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) g2[a][b] = 0.f;
#pragma unroll
    for (int q = 0; q < SPB; q += 4) {
        float4 dj[4], hk[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) dj[a] = f4(&d2[jy + a][q]);
#pragma unroll
        for (int b = 0; b < 4; ++b) hk[b] = f4(&n.h1[kx + 16 * b][q]);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                g2[a][b] = fmaf(dj[a].x, hk[b].x, g2[a][b]);
                g2[a][b] = fmaf(dj[a].y, hk[b].y, g2[a][b]);
                g2[a][b] = fmaf(dj[a].z, hk[b].z, g2[a][b]);
                g2[a][b] = fmaf(dj[a].w, hk[b].w, g2[a][b]);
            }
    }
    __syncthreads();
    pdl_wait();  // grads and loss are zero from here on
    if (t == 0) atomicAdd(loss, lpart);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) atomicAdd(&grads[OW2 + (jy + a) * NH + kx + 16 * b], g2[a][b]);
    // dW3, dW1 and the biases, one output per thread and step
    for (int i = t; i < NO * NH + NH * NI + 2 * NH + NO; i += THREADS) {
        float g = 0.f;
        int at = i;
        if (i < NO * NH) {
            for (int q = 0; q < SPB; ++q) g = fmaf(dout[q][i / NH], n.h2[i % NH][q], g);
            at = OW3 + i;
        } else if ((at -= NO * NH) < NH * NI) {
            for (int q = 0; q < SPB; ++q) g = fmaf(d1[at / NI][q], n.x[q][at % NI], g);
            at += OW1;
        } else if ((at -= NH * NI) < 2 * NH) {
            const float *d = at < NH ? d1[at] : d2[at - NH];
            for (int q = 0; q < SPB; ++q) g += d[q];
            at = at < NH ? OB1 + at : OB2 + at - NH;
        } else {
            at -= 2 * NH;
            for (int q = 0; q < SPB; ++q) g += dout[q][at];
            at += OB3;
        }
        atomicAdd(&grads[at], g);
    }
}

__global__ void adam_kernel(float *__restrict__ params, const float *__restrict__ grads, float *__restrict__ m,
                            float *__restrict__ v, int step, float lr, float beta1, float beta2, float eps)
{
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NPARAM) return;
    const float g = grads[i];
    const float mi = beta1 * m[i] + (1.f - beta1) * g;
    const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float mhat = mi / (1.f - powf(beta1, (float)step));
    const float vhat = vi / (1.f - powf(beta2, (float)step));
    params[i] -= lr * mhat / (sqrtf(vhat) + eps);
}

// Glorot-uniform weights from a counter-based hash, zero biases.
__global__ void init_kernel(float *__restrict__ params, unsigned long long seed)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NPARAM) return;
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const float u = 2.f * ((float)(z >> 40) * (1.f / 16777216.f)) - 1.f;
    float limit = 0.f;
    if (i < OB1) limit = sqrtf(6.f / (NI + NH));
    else if (i >= OW2 && i < OB2) limit = sqrtf(6.f / (NH + NH));
    else if (i >= OW3 && i < OB3) limit = sqrtf(6.f / (NH + NO));
    params[i] = u * limit;
}

}  // namespace mlp
}  // namespace mgx

using namespace mgx;

template <typename... Params, typename... Args>
static cudaError_t launch_dependent(void (*kernel)(Params...), int grid, cudaStream_t stream, const Args &...args)
{
    return mgx_launch_dependent(kernel, dim3((unsigned)grid), dim3(mlp::THREADS), 0, stream, args...);
}

extern "C" {

MGX_API int mgx_mlp_param_count(void) { return mlp::NPARAM; }

MGX_API int mgx_mlp_init(float *params, uint64_t seed, void *stream)
{
    if (!params) return MGX_E_INVALID;
    mlp::init_kernel<<<(mlp::NPARAM + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, seed);
    MGX_HOST_CHECK(cudaGetLastError());
    return MGX_SUCCESS;
}

MGX_API int mgx_mlp_forward(const float *X, int batch, const float *params, float *out, void *stream)
{
    if (batch < 0 || (batch > 0 && (!X || !params || !out))) return MGX_E_INVALID;
    if (batch == 0) return MGX_SUCCESS;
    if (batch >= mlp::SAMPLE_THREADS_BATCH) {
        MGX_HOST_CHECK(launch_dependent(mlp::forward_samples_kernel, (batch - 1) / mlp::THREADS + 1, (cudaStream_t)stream,
                                        X, batch, params, out));
        return MGX_SUCCESS;
    }
    // up to four blocks per SM, then blocks take further samples with the parameters they hold
    const int groups = (batch + mlp::SPB - 1) / mlp::SPB, most = 4 * mgx_sm_count();
    MGX_HOST_CHECK(launch_dependent(mlp::forward_kernel, groups < most ? groups : most, (cudaStream_t)stream, X, batch,
                                    params, out));
    return MGX_SUCCESS;
}

MGX_API int mgx_mlp_gradients(const float *X, const float *Y, const float *out_weights, int batch,
                              const float *params, float *grads, float *loss, void *stream)
{
    if (batch <= 0 || !X || !Y || !out_weights || !params || !grads || !loss) return MGX_E_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    MGX_HOST_CHECK(launch_dependent(mlp::zero_kernel, (mlp::NPARAM + mlp::THREADS) / mlp::THREADS, s, grads, loss));
    MGX_HOST_CHECK(launch_dependent(mlp::grad_kernel, (batch + mlp::SPB - 1) / mlp::SPB, s, X, Y, out_weights, batch,
                                    params, grads, loss));
    return MGX_SUCCESS;
}

MGX_API int mgx_mlp_adam_step(float *params, const float *grads, float *m, float *v, int step, float lr,
                              void *stream)
{
    if (!params || !grads || !m || !v || step < 1 || !(lr > 0.f)) return MGX_E_INVALID;
    MGX_HOST_CHECK(launch_dependent(mlp::adam_kernel, (mlp::NPARAM + mlp::THREADS - 1) / mlp::THREADS,
                                    (cudaStream_t)stream, params, grads, m, v, step, lr, 0.9f, 0.999f, 1e-8f));
    return MGX_SUCCESS;
}

}  // extern "C"
