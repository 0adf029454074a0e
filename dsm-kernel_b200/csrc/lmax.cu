// Learned angular-order cutoff: a 4-layer MLP (width 128, GELU) from
// (omega, source radius, receiver radius, 8 model summaries) to log(lmax),
// with bf16 weights and FP32 accumulation; forward, backward and Adam are
// the kernels below.  The engine uses the prediction to size the first
// order range of each frequency; the plain DSM amplitude test still decides
// the cutoff on the device and extends any range that falls short, so the
// truncation is the plain method's (src/SGTpsv/SGTpsv-MPI.f90:606-609).
//
// Parameter block (float, DSM_LMAX_NPARAM entries):
//   x_mean[NF] x_std[NF] y_mean y_std | W1[H][NF] b1[H] | W2[H][H] b2[H] |
//   W3[H][H] b3[H] | W4[H] b4
// Inputs are standardised with (x_mean, x_std); the network output is the
// standardised log(lmax).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <utility>
#include <vector>

#include "common.cuh"
#include "lmax.cuh"

namespace dsm {
namespace lmax {

namespace {

constexpr int H = DSM_LMAX_WIDTH, NF = DSM_LMAX_NFEAT;
constexpr int S = 32;   // samples per block of the prediction
constexpr int ST = 2;   // samples per block of a training step

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float dgelu(float z) {
    const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

// bf16 working copy of the weights (biases and normalisation stay FP32);
// for training also the transposes of W1, W2, W3 at the same offsets of Pt,
// so that the forward pass reads them neuron-contiguous
__device__ __forceinline__ int transposed(int k) {  // index of entry k in Pt, -1 outside W1..W3
    auto in = [&](int off, int nin) { return k >= off && k < off + H * nin ? off + (k - off) % nin * H + (k - off) / nin : -1; };
    int t = in(OFF_W1, NF);
    if (t < 0) t = in(OFF_W2, H);
    return t < 0 ? in(OFF_W3, H) : t;
}
__global__ void k_to_bf16(const float* __restrict__ P, __nv_bfloat16* __restrict__ Pb,
                          __nv_bfloat16* __restrict__ Pt, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Pb[i] = __float2bfloat16_rn(P[i]);
    if (Pt && transposed(i) >= 0) Pt[transposed(i)] = Pb[i];
}
__device__ __forceinline__ float wt(const __nv_bfloat16* Pb, int i) { return __bfloat162float(Pb[i]); }

// Prediction of S samples per block, thread j = neuron j: log(lmax) in out[n].
__global__ void __launch_bounds__(H) k_fwd(const float* __restrict__ P, const __nv_bfloat16* __restrict__ Pb,
                                           const float* __restrict__ X, int n, float* __restrict__ out) {
    __shared__ float a[S][H + 1];
    __shared__ float xin[S][NF];
    const int j = threadIdx.x, s0 = blockIdx.x * S;
    for (int t = j; t < S * NF; t += H) {
        const int s = t / NF, i = t % NF;
        xin[s][i] = s0 + s < n ? (X[(size_t)(s0 + s) * NF + i] - P[OFF_XM + i]) / P[OFF_XS + i] : 0.0f;
    }
    __syncthreads();
    float acc[S];
    // layer 1
#pragma unroll
    for (int s = 0; s < S; ++s) acc[s] = P[OFF_B1 + j];
    for (int i = 0; i < NF; ++i) {
        const float w = wt(Pb, OFF_W1 + j * NF + i);
#pragma unroll
        for (int s = 0; s < S; ++s) acc[s] += w * xin[s][i];
    }
    for (int layer = 0; layer < 3; ++layer) {
        if (layer > 0) {
            const int ow = layer == 1 ? OFF_W2 : OFF_W3, ob = layer == 1 ? OFF_B2 : OFF_B3;
#pragma unroll
            for (int s = 0; s < S; ++s) acc[s] = P[ob + j];
            for (int i = 0; i < H; ++i) {
                const float w = wt(Pb, ow + j * H + i);
#pragma unroll
                for (int s = 0; s < S; ++s) acc[s] += w * a[s][i];
            }
            __syncthreads();  // everyone has read a[] of the previous layer
        }
#pragma unroll
        for (int s = 0; s < S; ++s) a[s][j] = gelu(acc[s]);
        __syncthreads();
    }
    if (j < S && s0 + j < n) {
        float v = P[OFF_B4];
        for (int i = 0; i < H; ++i) v += wt(Pb, OFF_W4 + i) * a[j][i];
        out[s0 + j] = v * P[OFF_YS] + P[OFF_YM];
    }
}

// ---- one training step: two kernels.  A step is 53 MFLOP on 140 KB of
// weights, so it is bound by latency: launches, and the chain of each sum
// (the sums run in a fixed order, one fused multiply-add after the other).
// A kernel per layer and pass, with the activations recomputed from their
// pre-activations for every weight, took 360 us a step of 256 samples; two
// kernels with staged weights and stored activations, the start of each
// overlapping the end of the one before, take 28 us (a call of 192 steps,
// 5.3 to 5.8 ms; the host's launches show, 49 us on a busy host).
//
// What the kernel before writes is not const __restrict__: that promises data
// nobody writes while the kernel runs, and the compiler might read it before
// the wait.

// Per-sample part, ST samples per block, thread j = neuron j: forward pass,
// difference to the target, and the derivatives dZ of the three hidden
// layers.  Stores what the weight gradients sum over samples: standardised
// inputs Xn, activations A[layer][n][H], dZ[layer][n][H], differences dif
// and dY = 2 dif / n (loss = mean dif^2 on standardised targets).
// The bf16 weights of the four 128 x 128 products (W2, W3 and their
// transposes) are staged in shared memory while the first layer runs.
static_assert(OFF_W2 % 8 == 0 && OFF_W3 % 8 == 0, "16-byte copies of the weights");
constexpr size_t STEP_SMEM = (size_t)4 * H * H * sizeof(__nv_bfloat16);
__global__ void __launch_bounds__(H) k_step_samples(const float* P, const __nv_bfloat16* Pb, const __nv_bfloat16* Pt,
                                                    const float* __restrict__ norm, const float* __restrict__ X,
                                                    const float* __restrict__ T, const int* __restrict__ idx, int n,
                                                    float* __restrict__ Xn, float* __restrict__ A,
                                                    float* __restrict__ dZ, float* __restrict__ dif,
                                                    float* __restrict__ dY, int* __restrict__ step) {
    extern __shared__ __align__(16) unsigned char step_smem[];
    __nv_bfloat16* sw = reinterpret_cast<__nv_bfloat16*>(step_smem);  // W2^T, W3^T, W3, W2
    __shared__ float2 a2[2][H];  // of the two samples, two layers in turn
    __shared__ float xin[ST][NF], dy[ST], w4s[H];
    static_assert(ST == 2, "one float2 per neuron");
    const int j = threadIdx.x, s0 = blockIdx.x * ST;
    // before the previous step's update is done: this step's inputs (norm: the
    // parameters' standardisation block, which no step writes)
    for (int t = j; t < ST * NF; t += H) {
        const int s = t / NF, i = t % NF;
        float v = 0.0f;
        if (s0 + s < n) {
            const int row = idx ? idx[s0 + s] : s0 + s;
            v = (X[(size_t)row * NF + i] - norm[OFF_XM + i]) / norm[OFF_XS + i];
        }
        xin[s][i] = v;
    }
    float target = 0.0f;
    if (j < ST && s0 + j < n) target = (T[idx ? idx[s0 + j] : s0 + j] - norm[OFF_YM]) / norm[OFF_YS];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (blockIdx.x == 0 && j == 0) *step += 1;
    {
        const __nv_bfloat16* src[4] = {Pt + OFF_W2, Pt + OFF_W3, Pb + OFF_W3, Pb + OFF_W2};
#pragma unroll
        for (int m = 0; m < 4; ++m)
            for (int c = j; c < H * H / 8; c += H)  // (W2, W3 lie on 16-byte boundaries of the block)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 static_cast<uint32_t>(__cvta_generic_to_shared(sw + m * H * H + 8 * c))),
                             "l"(src[m] + 8 * c)
                             : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    w4s[j] = wt(Pb, OFF_W4 + j);
    __syncthreads();
    for (int t = j; t < ST * NF; t += H)
        if (s0 + t / NF < n) Xn[(size_t)s0 * NF + t] = xin[t / NF][t % NF];
    float acc[ST], z[3][ST];
#pragma unroll
    for (int s = 0; s < ST; ++s) acc[s] = P[OFF_B1 + j];
#pragma unroll
    for (int i = 0; i < NF; ++i) {
        const float w = wt(Pt, OFF_W1 + i * H + j);
#pragma unroll
        for (int s = 0; s < ST; ++s) acc[s] += w * xin[s][i];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int layer = 0; layer < 3; ++layer) {
        if (layer > 0) {
            const __nv_bfloat16* W = sw + (layer - 1) * H * H;
            const float bias = P[(layer == 1 ? OFF_B2 : OFF_B3) + j];
#pragma unroll
            for (int s = 0; s < ST; ++s) acc[s] = bias;
#pragma unroll 16
            for (int i = 0; i < H; ++i) {
                const float w = __bfloat162float(W[i * H + j]);
                const float2 x = a2[(layer - 1) & 1][i];
                acc[0] += w * x.x;
                acc[1] += w * x.y;
            }
        }
        float g[ST];
#pragma unroll
        for (int s = 0; s < ST; ++s) {
            z[layer][s] = acc[s];
            g[s] = gelu(acc[s]);
            if (s0 + s < n) A[((size_t)layer * n + s0 + s) * H + j] = g[s];
        }
        a2[layer & 1][j] = make_float2(g[0], g[1]);
        __syncthreads();
    }
    if (j < ST) {
        float v = P[OFF_B4];
        const float* x = reinterpret_cast<const float*>(a2[0]) + j;
#pragma unroll 32
        for (int i = 0; i < H; ++i) v += w4s[i] * x[i * ST];
        float q = 0.0f;
        if (s0 + j < n) {
            const float e = v - target;
            q = 2.0f * e / (float)n;
            dif[s0 + j] = e;
            dY[s0 + j] = q;
        }
        dy[j] = q;
    }
    __syncthreads();
    // dZ of the last hidden layer: dY W4 gelu'(Z); of the one below from it:
    // sum_j dZ[j] W[j][i] gelu'(Z)
#pragma unroll
    for (int layer = 2; layer >= 0; --layer) {
        float dz[ST];
        if (layer == 2) {
#pragma unroll
            for (int s = 0; s < ST; ++s) dz[s] = dy[s] * w4s[j] * dgelu(z[2][s]);
        } else {
            const __nv_bfloat16* W = sw + (layer == 1 ? 2 : 3) * H * H;
#pragma unroll
            for (int s = 0; s < ST; ++s) acc[s] = 0.0f;
#pragma unroll 16
            for (int i = 0; i < H; ++i) {
                const float w = __bfloat162float(W[i * H + j]);
                const float2 x = a2[(layer + 1) & 1][i];
                acc[0] += x.x * w;
                acc[1] += x.y * w;
            }
#pragma unroll
            for (int s = 0; s < ST; ++s) dz[s] = acc[s] * dgelu(z[layer][s]);
        }
#pragma unroll
        for (int s = 0; s < ST; ++s)
            if (s0 + s < n) dZ[((size_t)layer * n + s0 + s) * H + j] = dz[s];
        a2[layer & 1][j] = make_float2(dz[0], dz[1]);
        __syncthreads();
    }
}

// Adam on one weight or bias (the normalisation block is not trained).  The
// parameter and its moments are loaded before the gradient sums run.
struct AdamVal {
    float p, a, b;
};
__device__ __forceinline__ AdamVal adam_load(int i, const float* P, const float* m1, const float* m2) {
    return {P[i], m1[i], m2[i]};
}
struct AdamStep {
    float lr, wd, c1, c2;  // c = 1 - beta^t
    __device__ AdamStep(float lr_, float wd_, int t)
        : lr(lr_), wd(wd_), c1(1.0f - powf(0.9f, (float)t)), c2(1.0f - powf(0.999f, (float)t)) {}
};
__device__ __forceinline__ void adam(int i, float g, AdamVal v, const AdamStep& st, float* P, float* m1, float* m2,
                                     __nv_bfloat16* Pb, __nv_bfloat16* Pt) {
    const float b1 = 0.9f, b2 = 0.999f;
    // (the fused operations spelled out: training amplifies a rounding, and
    // which product is fused is otherwise up to the compiler)
    const float a = __fmaf_rn(1.0f - b1, g, __fmul_rn(b1, v.a));
    const float b = __fmaf_rn(__fmul_rn(1.0f - b2, g), g, __fmul_rn(b2, v.b));
    m1[i] = a;
    m2[i] = b;
    const float ah = a / st.c1, bh = b / st.c2;
    // decoupled weight decay (AdamW) keeps the network from leaning on
    // inputs that hardly vary between the training models
    const float p = v.p - st.lr * (ah / (sqrtf(bh) + 1e-8f) + st.wd * v.p);
    P[i] = p;
    Pb[i] = __float2bfloat16_rn(p);
    const int k = transposed(i);
    if (k >= 0) Pt[k] = Pb[i];
}

// use(s, load(s)) for s = 0 .. n - 1 in order; the loads of 32 samples are in
// flight while the 32 before them are used
template <class Load, class Use>
__device__ __forceinline__ void sample_loop(int n, Load load, Use use) {
    constexpr int U = 32;
    using V = decltype(load(0));
    V x[U], y[U];
    const int full = n / U * U;
    if (full) {
#pragma unroll
        for (int u = 0; u < U; ++u) x[u] = load(u);
        for (int s = 0; s < full; s += U) {
            const int nx = s + U < full ? s + U : s;  // (the last round loads its own again)
#pragma unroll
            for (int u = 0; u < U; ++u) y[u] = load(nx + u);
#pragma unroll
            for (int u = 0; u < U; ++u) use(s + u, x[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) x[u] = y[u];
        }
    }
    for (int s = full; s < n; ++s) use(s, load(s));
}

// Gradients summed over the batch in sample order, and their Adam update
// (UPDATE; otherwise they go to G).  Blocks 0 .. 127: JT output neurons of
// W2 or W3, thread i = input; then one block per input of W1 and one each
// for b1, b2, b3 (thread = output neuron); W4, b4 and the batch's loss.
// The parameters and moments are loaded before the sums: they are final
// once k_step_samples of this step has started its own work.
constexpr int JT = 2;
constexpr int NWB = 2 * H / JT, WBLOCKS = NWB + NF + 4;
template <bool UPDATE>
__global__ void __launch_bounds__(H) k_step_weights(const float* Xn, const float* A, const float* dZ, const float* dif,
                                                    const float* dY, int n, float* __restrict__ G,
                                                    float* __restrict__ P, float* __restrict__ m1,
                                                    float* __restrict__ m2, const int* step, float lr,
                                                    float wd, __nv_bfloat16* __restrict__ Pb,
                                                    __nv_bfloat16* __restrict__ Pt, float* __restrict__ loss) {
    const int i = threadIdx.x, blk = blockIdx.x;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    auto before = [&](int k) { return UPDATE ? adam_load(k, P, m1, m2) : AdamVal{}; };
    auto out = [&](int k, float g, AdamVal v) {
        if (UPDATE) adam(k, g, v, AdamStep(lr, wd, *step), P, m1, m2, Pb, Pt);
        else G[k] = g;
    };
    auto ready = [] { asm volatile("griddepcontrol.wait;" ::: "memory"); };
    if (blk < NWB) {
        const int layer = 1 + blk / (H / JT), j0 = blk % (H / JT) * JT;
        const float* Al = A + (size_t)(layer - 1) * n * H + i;
        const float* D = dZ + (size_t)layer * n * H + j0;
        const int k = (layer == 1 ? OFF_W2 : OFF_W3) + j0 * H + i;
        const AdamVal v0 = before(k), v1 = before(k + H);
        ready();
        float g0 = 0.0f, g1 = 0.0f;
        struct In {
            float x;
            float2 d;
        };
        sample_loop(
            n, [&](int s) { return In{Al[(size_t)s * H], *reinterpret_cast<const float2*>(D + (size_t)s * H)}; },
            [&](int, const In& v) {
                g0 += v.d.x * v.x;
                g1 += v.d.y * v.x;
            });
        out(k, g0, v0);
        out(k + H, g1, v1);
    } else if (blk < NWB + NF) {
        const int q = blk - NWB, k = OFF_W1 + i * NF + q;
        const AdamVal v = before(k);
        ready();
        float g = 0.0f;
        sample_loop(n, [&](int s) { return make_float2(dZ[(size_t)s * H + i], Xn[(size_t)s * NF + q]); },
                    [&](int, float2 v) { g += v.x * v.y; });
        out(k, g, v);
    } else if (blk < NWB + NF + 3) {
        const int layer = blk - NWB - NF, k = (layer == 0 ? OFF_B1 : (layer == 1 ? OFF_B2 : OFF_B3)) + i;
        const AdamVal v = before(k);
        ready();
        float gb = 0.0f;
        sample_loop(n, [&](int s) { return dZ[((size_t)layer * n + s) * H + i]; }, [&](int, float d) { gb += d; });
        out(k, gb, v);
    } else {
        __shared__ float red[256];
        const AdamVal v4 = before(OFF_W4 + i), vb = before(OFF_B4);
        ready();
        float g = 0.0f, gb = 0.0f;
        sample_loop(n, [&](int s) { return make_float2(A[((size_t)2 * n + s) * H + i], dY[s]); },
                    [&](int, float2 v) {
                        g += v.y * v.x;
                        gb += v.y;
                    });
        out(OFF_W4 + i, g, v4);
        if (i == 0) out(OFF_B4, gb, vb);
        for (int v = i; v < 256; v += H) {
            float l = 0.0f;
            for (int s = v; s < n; s += 256) l += dif[s] * dif[s];
            red[v] = l;
        }
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (i < o) red[i] += red[i + o];
            __syncthreads();
        }
        if (i == 0) *loss += red[0] / (float)n;
    }
}

// Device buffers of a training or gradient call, in one allocation: a
// batch of nb samples out of n.
struct Net {
    DBuf<float> mem;
    float *P, *G, *m1, *m2, *X, *T, *Xn, *A, *dZ, *dif, *dY, *loss;
    __nv_bfloat16 *Pb, *Pt;
    int *idx, *step;
    Net(int n, int nb, int nloss) {
        size_t off = 0;
        std::vector<std::pair<float**, size_t>> at;
        auto take = [&](float** p, size_t floats) {
            at.push_back({p, off});
            off += (floats + 63) / 64 * 64;  // 256-byte boundaries
        };
        float *pb, *pt, *ix, *sp;
        constexpr size_t NP = DSM_LMAX_NPARAM;
        // G .. step start as zero
        take(&G, NP);
        take(&m1, NP);
        take(&m2, NP);
        take(&loss, nloss);
        take(&sp, 1);
        const size_t nzero = off;
        take(&P, NP);
        take(&pb, (NP + 1) / 2);
        take(&pt, (NP + 1) / 2);
        take(&X, (size_t)n * NF);
        take(&T, n);
        take(&ix, n);
        take(&Xn, (size_t)nb * NF);
        take(&A, (size_t)3 * nb * H);
        take(&dZ, (size_t)3 * nb * H);
        take(&dif, nb);
        take(&dY, nb);
        mem.reserve(off);
        for (auto& a : at) *a.first = mem.p + a.second;
        Pb = reinterpret_cast<__nv_bfloat16*>(pb);
        Pt = reinterpret_cast<__nv_bfloat16*>(pt);
        idx = reinterpret_cast<int*>(ix);
        step = reinterpret_cast<int*>(sp);
        zero = nzero;
    }
    size_t zero;
    void upload(const float* hP, const float* hX, const float* hT, int n, cudaStream_t st) {
        DSM_CUDA(cudaMemsetAsync(mem.p, 0, zero * sizeof(float), st));
        DSM_CUDA(cudaMemcpyAsync(P, hP, sizeof(float) * DSM_LMAX_NPARAM, cudaMemcpyHostToDevice, st));
        k_to_bf16<<<(DSM_LMAX_NPARAM + 255) / 256, 256, 0, st>>>(P, Pb, Pt, DSM_LMAX_NPARAM);
        DSM_CUDA(cudaMemcpyAsync(X, hX, sizeof(float) * (size_t)n * NF, cudaMemcpyHostToDevice, st));
        DSM_CUDA(cudaMemcpyAsync(T, hT, sizeof(float) * n, cudaMemcpyHostToDevice, st));
        DSM_CUDA(cudaFuncSetAttribute(k_step_samples, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STEP_SMEM));
    }
    // forward and backward of one batch (idx into X/T, or the first n rows)
    // and, with update, the Adam step
    void run(const int* d_idx, int n, bool update, float lr, float wd, float* l, cudaStream_t st) {
        // each kernel may start while the one before it still runs and waits
        // inside for its end (griddepcontrol)
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.blockDim = dim3(H);
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3((n + ST - 1) / ST);
        cfg.dynamicSmemBytes = STEP_SMEM;
        DSM_CUDA(cudaLaunchKernelEx(&cfg, k_step_samples, (const float*)P, (const __nv_bfloat16*)Pb,
                                    (const __nv_bfloat16*)Pt, (const float*)P, (const float*)X, (const float*)T, d_idx,
                                    n, Xn, A, dZ, dif, dY, step));
        cfg.gridDim = dim3(WBLOCKS);
        cfg.dynamicSmemBytes = 0;
        DSM_CUDA(cudaLaunchKernelEx(&cfg, update ? k_step_weights<true> : k_step_weights<false>, (const float*)Xn,
                                    (const float*)A, (const float*)dZ, (const float*)dif, (const float*)dY, n, G, P,
                                    m1, m2, (const int*)step, lr, wd, Pb, Pt, l));
    }
};
// a stream for one call, destroyed with it also when the call throws
struct CallStream {
    cudaStream_t st = nullptr;
    CallStream() { DSM_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)); }
    ~CallStream() {
        if (st) {
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
    }
};

}  // namespace

void init_params(const float* X, const float* T, int n, unsigned seed, float* P) {
    std::memset(P, 0, sizeof(float) * DSM_LMAX_NPARAM);
    for (int i = 0; i < NF; ++i) {
        double m = 0.0, v = 0.0;
        for (int s = 0; s < n; ++s) m += X[(size_t)s * NF + i];
        m /= std::max(n, 1);
        for (int s = 0; s < n; ++s) v += (X[(size_t)s * NF + i] - m) * (X[(size_t)s * NF + i] - m);
        v = std::sqrt(v / std::max(n, 1));
        P[OFF_XM + i] = (float)m;
        P[OFF_XS + i] = (float)(v > 1e-6 ? v : 1.0);
    }
    double m = 0.0, v = 0.0;
    for (int s = 0; s < n; ++s) m += T[s];
    m /= std::max(n, 1);
    for (int s = 0; s < n; ++s) v += (T[s] - m) * (T[s] - m);
    v = std::sqrt(v / std::max(n, 1));
    P[OFF_YM] = (float)m;
    P[OFF_YS] = (float)(v > 1e-6 ? v : 1.0);
    std::mt19937 rng(seed);
    auto fill = [&](int off, int rows, int cols) {
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (float)cols));
        for (int k = 0; k < rows * cols; ++k) P[off + k] = nd(rng);
    };
    fill(OFF_W1, H, NF);
    fill(OFF_W2, H, H);
    fill(OFF_W3, H, H);
    fill(OFF_W4, 1, H);
}

void train(const float* X, const float* T, int n, int epochs, int batch, float lr, float wd, unsigned seed,
           float* P, float* losses, int device) {
    if (n <= 0 || batch <= 0 || epochs <= 0) throw Error(DSM_ERR_INVALID, "empty training set");
    DSM_CUDA(cudaSetDevice(device));
    batch = std::min(batch, n);
    Net net(n, batch, epochs);
    CallStream cs;
    cudaStream_t st = cs.st;
    net.upload(P, X, T, n, st);
    std::vector<int> perm(n);
    for (int i = 0; i < n; ++i) perm[i] = i;
    std::mt19937 rng(seed ^ 0x9e3779b9u);
    const int nb = n / batch;  // full batches per epoch
    for (int e = 0; e < epochs; ++e) {
        std::shuffle(perm.begin(), perm.end(), rng);
        // (a copy from pageable memory: perm may change once it returns)
        DSM_CUDA(cudaMemcpyAsync(net.idx, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
        for (int b = 0; b < nb; ++b) net.run(net.idx + (size_t)b * batch, batch, true, lr, wd, net.loss + e, st);
    }
    std::vector<float> hl(epochs);
    DSM_CUDA(cudaMemcpyAsync(hl.data(), net.loss, sizeof(float) * epochs, cudaMemcpyDeviceToHost, st));
    DSM_CUDA(cudaMemcpyAsync(P, net.P, sizeof(float) * DSM_LMAX_NPARAM, cudaMemcpyDeviceToHost, st));
    DSM_CUDA(cudaStreamSynchronize(st));
    // epoch loss = mean of the batch losses
    if (losses)
        for (int e = 0; e < epochs; ++e) losses[e] = hl[e] / (float)std::max(nb, 1);
}

void grad(const float* P, const float* X, const float* T, int n, float* G, float* loss, int device) {
    DSM_CUDA(cudaSetDevice(device));
    Net net(n, n, 1);
    CallStream cs;
    cudaStream_t st = cs.st;
    net.upload(P, X, T, n, st);
    net.run(nullptr, n, false, 0.0f, 0.0f, net.loss, st);
    DSM_CUDA(cudaMemcpyAsync(G, net.G, sizeof(float) * DSM_LMAX_NPARAM, cudaMemcpyDeviceToHost, st));
    DSM_CUDA(cudaMemcpyAsync(loss, net.loss, sizeof(float), cudaMemcpyDeviceToHost, st));
    DSM_CUDA(cudaStreamSynchronize(st));
}

void Predictor::load(const float* P, cudaStream_t st) {
    params.upload(P, DSM_LMAX_NPARAM, st);
    pb.reserve(DSM_LMAX_NPARAM);
    k_to_bf16<<<(DSM_LMAX_NPARAM + 255) / 256, 256, 0, st>>>(params.p, pb.p, nullptr, DSM_LMAX_NPARAM);
    DSM_CUDA(cudaGetLastError());
    ready = true;
}

void Predictor::predict(const float* hX, int n, float* hout, cudaStream_t st) {
    if (!ready) throw Error(DSM_ERR_INVALID, "no lmax model loaded");
    X.upload(hX, (size_t)n * NF, st);
    out.reserve(n);
    k_fwd<<<(n + S - 1) / S, H, 0, st>>>(params.p, pb.p, X.p, n, out.p);
    DSM_CUDA(cudaGetLastError());
    DSM_CUDA(cudaMemcpyAsync(hout, out.p, sizeof(float) * n, cudaMemcpyDeviceToHost, st));
    DSM_CUDA(cudaStreamSynchronize(st));
}

}  // namespace lmax
}  // namespace dsm
