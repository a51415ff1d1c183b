// Learned result-size estimator: a 16 -> 64 -> 64 -> 2 ReLU MLP on per-cell
// features predicts log2(1 + distance calcs) and log2(1 + hits) of a cell.
// Forward, backward and Adam are plain FP32 CUDA-core kernels (the network is
// tiny).  The sampling estimator it replaces (GPU.cu:854-1065, which counts
// the hits of every 100th point) runs as the join's own count pass over
// tasks for the sampled points (sj_tasks.cu builds them, sj_api.cpp runs it).
#include <mutex>

#include "sj_internal.h"

namespace {

// ------------------------------------------------------------------ MLP ----
// parameter offsets
constexpr int OW1 = 0;
constexpr int OB1 = OW1 + SJ_NFEAT * SJ_HID;
constexpr int OW2 = OB1 + SJ_HID;
constexpr int OB2 = OW2 + SJ_HID * SJ_HID;
constexpr int OW3 = OB2 + SJ_HID;
constexpr int OB3 = OW3 + SJ_HID * SJ_NOUT;
constexpr int NP = OB3 + SJ_NOUT;
static_assert(NP == SJ_MLP_NPARAM, "parameter layout");

__device__ __forceinline__ void mlp_forward(const float *__restrict__ w, const float *x, float *z1, float *z2,
                                            float *y)
{
    for (int j = 0; j < SJ_HID; j++) {
        float s = w[OB1 + j];
#pragma unroll
        for (int i = 0; i < SJ_NFEAT; i++) s = fmaf(x[i], w[OW1 + i * SJ_HID + j], s);
        z1[j] = s;
    }
    for (int j = 0; j < SJ_HID; j++) {
        float s = w[OB2 + j];
        for (int i = 0; i < SJ_HID; i++) s = fmaf(fmaxf(z1[i], 0.f), w[OW2 + i * SJ_HID + j], s);
        z2[j] = s;
    }
#pragma unroll
    for (int o = 0; o < SJ_NOUT; o++) {
        float s = w[OB3 + o];
        for (int i = 0; i < SJ_HID; i++) s = fmaf(fmaxf(z2[i], 0.f), w[OW3 + i * SJ_NOUT + o], s);
        y[o] = s;
    }
}

__global__ void __launch_bounds__(128) k_mlp_infer(const float *__restrict__ feat, uint32_t m,
                                                   const float *__restrict__ wg, float *__restrict__ out)
{
    __shared__ float w[NP];
    for (int i = threadIdx.x; i < NP; i += blockDim.x) w[i] = wg[i];
    __syncthreads();
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= m) return;
    float x[SJ_NFEAT], z1[SJ_HID], z2[SJ_HID], y[SJ_NOUT];
    for (int i = 0; i < SJ_NFEAT; i++) x[i] = feat[(uint64_t)s * SJ_NFEAT + i];
    mlp_forward(w, x, z1, z2, y);
    for (int o = 0; o < SJ_NOUT; o++) out[(uint64_t)s * SJ_NOUT + o] = y[o];
}

// Loss and gradient in two launches.  k_mlp_grad: a CTA takes tiles of GT
// samples and runs the three layers forward and backward on them as small
// matrix products out of shared memory (weights and activations stay there;
// nothing per sample goes to global memory), keeping its sums of the weight
// gradients in registers over all of its tiles; it then writes one partial
// gradient (and loss).  k_mlp_grad_sum adds the partials in a fixed order, so
// the result does not depend on scheduling.  Loss = 1/(2m) * sum (y - t)^2.
//
// Bound: latency -- 8192 samples are 0.24 GFLOP (3 us of the FP32 pipe) and
// 0.6 MB of input.  Per-sample threads with their activations in local memory
// and one thread per parameter summing all m samples in turn took 44 + 1063 us
// at m = 8192 on a B200; this form takes 24.6 us for the call (both launches).
constexpr int GT = 32;           // samples per tile
constexpr int GTH = 256;         // threads: 16 x 16
constexpr int GLD = SJ_HID + 4;  // row stride in shared memory: 16-byte accesses of 8 consecutive rows hit all banks
constexpr int GXLD = SJ_NFEAT + 4;
constexpr int GSTRIDE = NP + 1;  // a partial: the gradient, then the loss
constexpr int GMAX_CTAS = 296;   // two CTAs on each of 148 SMs; more tiles are taken in turn
static_assert(SJ_HID == 64 && SJ_NFEAT == 16 && SJ_NOUT == 2, "thread mapping of k_mlp_grad");

struct __align__(16) GradSmem {
    float w1[SJ_NFEAT][GLD], w2[SJ_HID][GLD], w3[SJ_HID * SJ_NOUT], b1[SJ_HID], b2[SJ_HID];
    float x[GT][GXLD];
    float a1[GT][GLD];           // relu(z1), later the gradient at z1
    float a2[GT][GLD];           // relu(z2), later the gradient at z2
    float g3[GT][SJ_NOUT];
    float b3[SJ_NOUT];
    float loss[GT];
};

// s[r][c] += the products of one 4-vector of a row with a 4 x 4 block
__device__ __forceinline__ float dot4(float4 a, float4 b, float s)
{
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

__device__ __forceinline__ void axpy4(float a, float4 b, float (&s)[4])
{
    s[0] = fmaf(a, b.x, s[0]);
    s[1] = fmaf(a, b.y, s[1]);
    s[2] = fmaf(a, b.z, s[2]);
    s[3] = fmaf(a, b.w, s[3]);
}

__global__ void __launch_bounds__(GTH, 2) k_mlp_grad(const float *__restrict__ X, const float *__restrict__ Yt,
                                                     uint32_t m, const float *__restrict__ wg,
                                                     float *__restrict__ part)
{
    __shared__ GradSmem sm;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    for (int i = tid; i < SJ_NFEAT * SJ_HID; i += GTH) sm.w1[i / SJ_HID][i % SJ_HID] = wg[OW1 + i];
    for (int i = tid; i < SJ_HID * SJ_HID; i += GTH) sm.w2[i / SJ_HID][i % SJ_HID] = wg[OW2 + i];
    if (tid < SJ_HID * SJ_NOUT) sm.w3[tid] = wg[OW3 + tid];
    if (tid < SJ_HID) {
        sm.b1[tid] = wg[OB1 + tid];
        sm.b2[tid] = wg[OB2 + tid];
    }
    if (tid < SJ_NOUT) sm.b3[tid] = wg[OB3 + tid];
    const float inv = 1.0f / (float)m;
    float dw1[4] = {0.f, 0.f, 0.f, 0.f};                  // row ty, columns 4 tx ..
    float dw2[4][4] = {};                                 // rows 4 ty .., columns 4 tx ..
    float dw3 = 0.f, db = 0.f, db3 = 0.f, lsum = 0.f;     // by thread, see below
    const uint32_t nTiles = (m + GT - 1) / GT;
    for (uint32_t tile = blockIdx.x; tile < nTiles; tile += gridDim.x) {
        const uint32_t s0 = tile * GT;
        const uint32_t ns = min((uint32_t)GT, m - s0);
        __syncthreads();   // the weights are there; the previous tile is done with the arrays
        for (int i = tid; i < GT * SJ_NFEAT; i += GTH) {
            const uint32_t r = i / SJ_NFEAT;
            sm.x[r][i % SJ_NFEAT] = r < ns ? X[(uint64_t)s0 * SJ_NFEAT + i] : 0.f;
        }
        __syncthreads();
        // layers 1 and 2: thread (ty, tx) has samples 2 ty, 2 ty + 1 and units 4 tx ..
        {
            float z[2][4];
#pragma unroll
            for (int c = 0; c < 4; c++) z[0][c] = z[1][c] = sm.b1[4 * tx + c];
#pragma unroll
            for (int i = 0; i < SJ_NFEAT; i++) {
                const float4 w = ld4(&sm.w1[i][4 * tx]);
                axpy4(sm.x[2 * ty][i], w, z[0]);
                axpy4(sm.x[2 * ty + 1][i], w, z[1]);
            }
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) sm.a1[2 * ty + r][4 * tx + c] = fmaxf(z[r][c], 0.f);
        }
        __syncthreads();
        {
            float z[2][4];
#pragma unroll
            for (int c = 0; c < 4; c++) z[0][c] = z[1][c] = sm.b2[4 * tx + c];
#pragma unroll 4
            for (int i = 0; i < SJ_HID; i++) {
                const float4 w = ld4(&sm.w2[i][4 * tx]);
                axpy4(sm.a1[2 * ty][i], w, z[0]);
                axpy4(sm.a1[2 * ty + 1][i], w, z[1]);
            }
#pragma unroll
            for (int r = 0; r < 2; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) sm.a2[2 * ty + r][4 * tx + c] = fmaxf(z[r][c], 0.f);
        }
        __syncthreads();
        // output layer: threads 0..63 = (sample, output)
        if (tid < GT * SJ_NOUT) {
            const int r = tid / SJ_NOUT, o = tid % SJ_NOUT;
            float y = sm.b3[o];
            for (int i = 0; i < SJ_HID; i++) y = fmaf(sm.a2[r][i], sm.w3[i * SJ_NOUT + o], y);
            const float e = (uint32_t)r < ns ? y - Yt[(uint64_t)(s0 + r) * SJ_NOUT + o] : 0.f;
            lsum += 0.5f * e * e;
            sm.g3[r][o] = e * inv;
        }
        __syncthreads();
        // dW3 (threads 0..127: unit, output) and db3 (threads 128, 129)
        if (tid < SJ_HID * SJ_NOUT) {
            const int i = tid / SJ_NOUT, o = tid % SJ_NOUT;
#pragma unroll 8
            for (int r = 0; r < GT; r++) dw3 = fmaf(sm.a2[r][i], sm.g3[r][o], dw3);
        } else if (tid < SJ_HID * SJ_NOUT + SJ_NOUT) {
            for (int r = 0; r < GT; r++) db3 += sm.g3[r][tid - SJ_HID * SJ_NOUT];
        }
        __syncthreads();
        // gradient at z2, in place
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int s = 2 * ty + r;
            const float e0 = sm.g3[s][0], e1 = sm.g3[s][1];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int i = 4 * tx + c;
                const float g = fmaf(e1, sm.w3[i * SJ_NOUT + 1], e0 * sm.w3[i * SJ_NOUT]);
                sm.a2[s][i] = sm.a2[s][i] > 0.f ? g : 0.f;
            }
        }
        __syncthreads();
        // dW2; then the gradient at z1: thread (ty, tx) has samples 2 ty, 2 ty + 1 and units tx + 16 c
#pragma unroll 4
        for (int r = 0; r < GT; r++) {
            const float4 h = ld4(&sm.a1[r][4 * ty]);
            const float4 g = ld4(&sm.a2[r][4 * tx]);
            axpy4(h.x, g, dw2[0]);
            axpy4(h.y, g, dw2[1]);
            axpy4(h.z, g, dw2[2]);
            axpy4(h.w, g, dw2[3]);
        }
        float g1[2][4] = {};
#pragma unroll 4
        for (int j = 0; j < SJ_HID; j += 4) {
            const float4 p = ld4(&sm.a2[2 * ty][j]), q = ld4(&sm.a2[2 * ty + 1][j]);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float4 w = ld4(&sm.w2[tx + 16 * c][j]);
                g1[0][c] = dot4(p, w, g1[0][c]);
                g1[1][c] = dot4(q, w, g1[1][c]);
            }
        }
        __syncthreads();   // every thread has read the activations of layer 1
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                float &a = sm.a1[2 * ty + r][tx + 16 * c];
                a = a > 0.f ? g1[r][c] : 0.f;
            }
        __syncthreads();
        // dW1, db1 (threads 0..63) and db2 (threads 64..127)
#pragma unroll 8
        for (int r = 0; r < GT; r++) axpy4(sm.x[r][ty], ld4(&sm.a1[r][4 * tx]), dw1);
        if (tid < SJ_HID) {
            for (int r = 0; r < GT; r++) db += sm.a1[r][tid];
        } else if (tid < 2 * SJ_HID) {
            for (int r = 0; r < GT; r++) db += sm.a2[r][tid - SJ_HID];
        }
    }
    float *const out = part + (uint64_t)blockIdx.x * GSTRIDE;
#pragma unroll
    for (int c = 0; c < 4; c++) out[OW1 + ty * SJ_HID + 4 * tx + c] = dw1[c];
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) out[OW2 + (4 * ty + r) * SJ_HID + 4 * tx + c] = dw2[r][c];
    if (tid < SJ_HID * SJ_NOUT) out[OW3 + tid] = dw3;
    else if (tid < SJ_HID * SJ_NOUT + SJ_NOUT) out[OB3 + tid - SJ_HID * SJ_NOUT] = db3;
    if (tid < SJ_HID) out[OB1 + tid] = db;
    else if (tid < 2 * SJ_HID) out[OB2 + tid - SJ_HID] = db;
    // the loss: threads 0..63 hold (sample, output) parts
    if (tid < 2 * 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if ((tid & 31) == 0) sm.loss[tid >> 5] = lsum;
    }
    __syncthreads();
    if (tid == 0) out[NP] = (sm.loss[0] + sm.loss[1]) * inv;
}

// grad[p] = sum of the nPart partials of parameter p; entry NP is the loss.
// A CTA has 32 parameters; its 8 warps take the partials in turn (coalesced
// over the parameters) and meet in shared memory.
__global__ void __launch_bounds__(256) k_mlp_grad_sum(const float *__restrict__ part, uint32_t nPart,
                                                      float *__restrict__ grad, float *__restrict__ loss)
{
    __shared__ float red[8][32];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t p = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (p < GSTRIDE) {
#pragma unroll 4
        for (uint32_t k = w; k < nPart; k += 8) s += part[(uint64_t)k * GSTRIDE + p];
    }
    red[w][lane] = s;
    __syncthreads();
    if (w == 0 && p < GSTRIDE) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < 8; k++) t += red[k][lane];
        if (p < NP) grad[p] = t;
        else *loss = t;
    }
}

uint32_t grad_ctas(uint32_t m)
{
    const uint32_t tiles = m / GT + (m % GT ? 1u : 0u);
    return tiles < (uint32_t)GMAX_CTAS ? tiles : (uint32_t)GMAX_CTAS;
}

// part: grad_ctas(m) * GSTRIDE floats of scratch
cudaError_t launch_grad(const float *x, const float *y, uint32_t m, const float *w, float *grad, float *loss,
                        float *part, cudaStream_t s)
{
    const uint32_t n = grad_ctas(m);
    k_mlp_grad<<<n, GTH, 0, s>>>(x, y, m, w, part);
    sj_note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_mlp_grad_sum<<<(GSTRIDE + 31) / 32, 256, 0, s>>>(part, n, grad, loss);
    sj_note_launch();
    return cudaGetLastError();
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ mm,
                       float *__restrict__ vv, int step, float lr)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= NP) return;
    const float b1 = 0.9f, b2 = 0.999f, e = 1e-8f;
    float m = b1 * mm[p] + (1.f - b1) * g[p];
    float v = b2 * vv[p] + (1.f - b2) * g[p] * g[p];
    mm[p] = m;
    vv[p] = v;
    float mh = m / (1.f - powf(b1, (float)step));
    float vh = v / (1.f - powf(b2, (float)step));
    w[p] -= lr * mh / (sqrtf(vh) + e);
}

}  // namespace



cudaError_t sj_launch_mlp_infer(const float *feat, uint32_t nCells, const float *weights, float *out, cudaStream_t s)
{
    if (nCells == 0) return cudaSuccess;
    k_mlp_infer<<<(nCells + 127) / 128, 128, 0, s>>>(feat, nCells, weights, out); sj_note_launch();
    return cudaGetLastError();
}

static cudaError_t mlp_grad_impl(const float *x, const float *y, uint32_t m, const float *w, float *grad,
                                 float *lossOut, cudaStream_t s)
{
    float *part = nullptr;
    cudaError_t e = cudaMallocAsync((void **)&part, (size_t)grad_ctas(m) * GSTRIDE * sizeof(float), s);
    if (e != cudaSuccess) return e;
    e = launch_grad(x, y, m, w, grad, lossOut, part, s);
    cudaFreeAsync(part, s);
    return e;
}

cudaError_t sj_launch_mlp_grad(const float *x, const float *y, uint32_t m, const float *weights, float *grad,
                               float *lossOut, cudaStream_t s)
{
    return mlp_grad_impl(x, y, m, weights, grad, lossOut, s);
}

cudaError_t sj_launch_mlp_train_step(const float *x, const float *y, uint32_t m, float *weights, float *grad,
                                     float *adamM, float *adamV, int step, float lr, float *lossOut, cudaStream_t s)
{
    cudaError_t e = mlp_grad_impl(x, y, m, weights, grad, lossOut, s);
    if (e != cudaSuccess) return e;
    k_adam<<<(NP + 255) / 256, 256, 0, s>>>(weights, grad, adamM, adamV, step, lr); sj_note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------- allocation-free gradient --
// Fixed scratch for sj_mlp_loss_grad_noalloc: the partial gradients of at most
// SJ_MLP_NOALLOC_MAX_SAMPLES samples.  Every device that loads this library
// holds it (about 5.5 MB) until the process exits.
constexpr int kNoallocCtas = SJ_MLP_NOALLOC_MAX_SAMPLES / GT;
static_assert(kNoallocCtas <= GMAX_CTAS && SJ_MLP_NOALLOC_MAX_SAMPLES % GT == 0, "one partial per tile");
static __device__ __align__(256) float g_mlpNoallocScratch[kNoallocCtas * GSTRIDE];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noallocMutex;
float *g_noallocScratchPtr[kMaxDevices] = {nullptr};
}  // namespace

extern "C" sj_status sj_mlp_loss_grad_noalloc(const float *x, const float *y, uint32_t m, const float *w, float *loss,
                                              float *grad, void *stream)
{
    if (!x || !y || !w || !loss || !grad || m == 0) {
        sj_set_error_message("sj_mlp_loss_grad_noalloc: null pointer or zero samples");
        return SJ_ERR_BAD_INPUT;
    }
    if (m > SJ_MLP_NOALLOC_MAX_SAMPLES) {
        sj_set_error_message("sj_mlp_loss_grad_noalloc: more samples than the fixed scratch holds "
                             "(limit SJ_MLP_NOALLOC_MAX_SAMPLES = 8192); split the batch");
        return SJ_ERR_BAD_INPUT;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        sj_set_error_message("sj_mlp_loss_grad_noalloc: no usable current device");
        return SJ_ERR_CUDA;
    }
    float *scratch;
    {
        // first call on a device: resolve the device address of the scratch
        // array (a host-side name of a __device__ array is not a device pointer)
        std::lock_guard<std::mutex> lock(g_noallocMutex);
        if (!g_noallocScratchPtr[dev]) {
            void *ptr = nullptr;
            e = cudaGetSymbolAddress(&ptr, g_mlpNoallocScratch);
            if (e != cudaSuccess || !ptr) {
                sj_set_error_message("sj_mlp_loss_grad_noalloc: cudaGetSymbolAddress failed");
                return SJ_ERR_CUDA;
            }
            g_noallocScratchPtr[dev] = (float *)ptr;
        }
        scratch = g_noallocScratchPtr[dev];
    }
    // an error left pending by earlier work on this thread is reported, not consumed,
    // so the error checks after the launches below see this call's launches only
    e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        sj_set_error_message("sj_mlp_loss_grad_noalloc: a CUDA error from earlier work is pending");
        return SJ_ERR_CUDA;
    }
    // every partial and every output is overwritten by each call
    e = launch_grad(x, y, m, w, grad, loss, scratch, (cudaStream_t)stream);
    if (e != cudaSuccess) {
        sj_set_error_message(cudaGetErrorString(e));
        return SJ_ERR_CUDA;
    }
    return SJ_OK;
}
