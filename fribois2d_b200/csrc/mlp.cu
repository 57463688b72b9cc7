// A small multilayer perceptron trained and evaluated with hand-written
// kernels: the learned initial guess of the strong fluid-structure coupling
// iteration (no counterpart in the reference, whose coupling is explicit).
//
//   x (n_in) -> tanh(W1 x + b1) (64) -> tanh(W2 h1 + b2) (64) -> W3 h2 + b3 (n_out)
//
// FP32 throughout.  Parameters are one flat array [W1 b1 W2 b2 W3 b3] with
// W[out][in] row-major.  Loss: mean over the samples of the summed squared
// output errors.  Gradients are accumulated per block in a fixed order and
// summed over blocks in a fixed order, so training is deterministic.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <new>
#include <random>
#include <vector>

#include "../../include/fribois2d.h"

namespace {

constexpr int kH = 64;      // hidden width
constexpr int kMaxIn = 64;  // input width limit
constexpr int kMaxOut = 8;  // output width limit
constexpr int kS = 16;      // samples per block

struct Shape {
    int nin, nout;
    int oW1, ob1, oW2, ob2, oW3, ob3, n;
    explicit Shape(int ni = 0, int no = 0) : nin(ni), nout(no) {
        oW1 = 0;
        ob1 = oW1 + kH * nin;
        oW2 = ob1 + kH;
        ob2 = oW2 + kH * kH;
        oW3 = ob2 + kH;
        ob3 = oW3 + nout * kH;
        n = ob3 + nout;
    }
};

// forward pass of kS samples per block (64 threads: one per hidden unit);
// H1, H2 keep the activations for the backward pass (may be null)
__global__ void __launch_bounds__(kH) k_mlp_fwd(Shape sh, const float *__restrict__ P, const float *__restrict__ X,
                                                 int B, float *__restrict__ H1, float *__restrict__ H2,
                                                 float *__restrict__ Y) {
    __shared__ float xs[kS][kMaxIn];
    __shared__ float h1[kS][kH], h2[kS][kH];
    const int t = threadIdx.x, s0 = blockIdx.x * kS;
    const int ns = min(kS, B - s0);
    for (int i = t; i < kS * sh.nin; i += kH) {
        const int s = i / sh.nin, k = i - s * sh.nin;
        xs[s][k] = (s < ns) ? X[static_cast<size_t>(s0 + s) * sh.nin + k] : 0.0f;
    }
    __syncthreads();
    const float *w1 = P + sh.oW1 + t * sh.nin;
    for (int s = 0; s < kS; ++s) {
        float a = P[sh.ob1 + t];
        for (int k = 0; k < sh.nin; ++k) a = fmaf(w1[k], xs[s][k], a);
        h1[s][t] = tanhf(a);
    }
    __syncthreads();
    const float *w2 = P + sh.oW2 + t * kH;
    for (int s = 0; s < kS; ++s) {
        float a = P[sh.ob2 + t];
        for (int k = 0; k < kH; ++k) a = fmaf(w2[k], h1[s][k], a);
        h2[s][t] = tanhf(a);
    }
    __syncthreads();
    for (int i = t; i < ns * kH; i += kH) {
        const int s = i / kH, k = i - s * kH;
        if (H1) H1[static_cast<size_t>(s0 + s) * kH + k] = h1[s][k];
        if (H2) H2[static_cast<size_t>(s0 + s) * kH + k] = h2[s][k];
    }
    for (int i = t; i < ns * sh.nout; i += kH) {
        const int s = i / sh.nout, o = i - s * sh.nout;
        const float *w3 = P + sh.oW3 + o * kH;
        float a = P[sh.ob3 + o];
        for (int k = 0; k < kH; ++k) a = fmaf(w3[k], h2[s][k], a);
        Y[static_cast<size_t>(s0 + s) * sh.nout + o] = a;
    }
}

// backward pass: per-block parameter gradients (G[block][param]) and loss
// partials for the samples of the block; dL/dy = 2 (y - target) / B
__global__ void __launch_bounds__(kH) k_mlp_bwd(Shape sh, const float *__restrict__ P, const float *__restrict__ X,
                                                 const float *__restrict__ H1, const float *__restrict__ H2,
                                                 const float *__restrict__ Y, const float *__restrict__ T, int B,
                                                 float *__restrict__ G, float *__restrict__ L) {
    __shared__ float xs[kS][kMaxIn];
    __shared__ float h1[kS][kH], h2[kS][kH], d1[kS][kH], d2[kS][kH];
    __shared__ float dy[kS][kMaxOut];
    __shared__ float lsum[kH];
    const int t = threadIdx.x, s0 = blockIdx.x * kS;
    const int ns = min(kS, B - s0);
    float *g = G + static_cast<size_t>(blockIdx.x) * sh.n;
    for (int i = t; i < kS * sh.nin; i += kH) {
        const int s = i / sh.nin, k = i - s * sh.nin;
        xs[s][k] = (s < ns) ? X[static_cast<size_t>(s0 + s) * sh.nin + k] : 0.0f;
    }
    for (int i = t; i < kS * kH; i += kH) {
        const int s = i / kH, k = i - s * kH;
        h1[s][k] = (s < ns) ? H1[static_cast<size_t>(s0 + s) * kH + k] : 0.0f;
        h2[s][k] = (s < ns) ? H2[static_cast<size_t>(s0 + s) * kH + k] : 0.0f;
    }
    float l = 0.0f;
    for (int i = t; i < kS * sh.nout; i += kH) {
        const int s = i / sh.nout, o = i - s * sh.nout;
        float e = 0.0f;
        if (s < ns) e = Y[static_cast<size_t>(s0 + s) * sh.nout + o] - T[static_cast<size_t>(s0 + s) * sh.nout + o];
        dy[s][o] = 2.0f * e / static_cast<float>(B);
        l = fmaf(e, e, l);
    }
    lsum[t] = l;
    __syncthreads();
    // layer 3: dW3[o][k] = sum_s dy[s][o] h2[s][k]; db3[o] = sum_s dy[s][o]
    for (int i = t; i < sh.nout * kH; i += kH) {
        const int o = i / kH, k = i - o * kH;
        float a = 0.0f;
        for (int s = 0; s < kS; ++s) a = fmaf(dy[s][o], h2[s][k], a);
        g[sh.oW3 + i] = a;
    }
    if (t < sh.nout) {
        float a = 0.0f;
        for (int s = 0; s < kS; ++s) a += dy[s][t];
        g[sh.ob3 + t] = a;
    }
    // d2 = (W3^T dy) * (1 - h2^2)
    for (int s = 0; s < kS; ++s) {
        float a = 0.0f;
        for (int o = 0; o < sh.nout; ++o) a = fmaf(P[sh.oW3 + o * kH + t], dy[s][o], a);
        d2[s][t] = a * (1.0f - h2[s][t] * h2[s][t]);
    }
    __syncthreads();
    // layer 2: dW2[t][k] = sum_s d2[s][t] h1[s][k]
    for (int k = 0; k < kH; ++k) {
        float a = 0.0f;
        for (int s = 0; s < kS; ++s) a = fmaf(d2[s][t], h1[s][k], a);
        g[sh.oW2 + t * kH + k] = a;
    }
    {
        float a = 0.0f;
        for (int s = 0; s < kS; ++s) a += d2[s][t];
        g[sh.ob2 + t] = a;
    }
    // d1 = (W2^T d2) * (1 - h1^2)
    for (int s = 0; s < kS; ++s) {
        float a = 0.0f;
        for (int j = 0; j < kH; ++j) a = fmaf(P[sh.oW2 + j * kH + t], d2[s][j], a);
        d1[s][t] = a * (1.0f - h1[s][t] * h1[s][t]);
    }
    __syncthreads();
    for (int k = 0; k < sh.nin; ++k) {
        float a = 0.0f;
        for (int s = 0; s < kS; ++s) a = fmaf(d1[s][t], xs[s][k], a);
        g[sh.oW1 + t * sh.nin + k] = a;
    }
    {
        float a = 0.0f;
        for (int s = 0; s < kS; ++s) a += d1[s][t];
        g[sh.ob1 + t] = a;
    }
    if (t == 0) {
        float a = 0.0f;
        for (int i = 0; i < kH; ++i) a += lsum[i];
        L[blockIdx.x] = a;
    }
}

// sums the per-block partials in block order (deterministic)
__global__ void k_mlp_reduce(int n, int nb, const float *__restrict__ G, float *__restrict__ out,
                             const float *__restrict__ L, float *__restrict__ loss, int B) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        float a = 0.0f;
        for (int b = 0; b < nb; ++b) a += G[static_cast<size_t>(b) * n + i];
        out[i] = a;
    }
    if (i == 0) {
        float a = 0.0f;
        for (int b = 0; b < nb; ++b) a += L[b];
        *loss = a / static_cast<float>(B);
    }
}

// Adam (Kingma and Ba 2015) with bias correction: one parameter
__device__ __forceinline__ void adam_update(float g, float &p, float &m, float &v, float lr, float b1, float b2,
                                            float eps, float c1, float c2) {
    m = b1 * m + (1.0f - b1) * g;
    v = b2 * v + (1.0f - b2) * g * g;
    p -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

__global__ void k_adam(int n, float *__restrict__ P, const float *__restrict__ G, float *__restrict__ M,
                       float *__restrict__ V, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float p = P[i], m = M[i], v = V[i];
    adam_update(G[i], p, m, v, lr, b1, b2, eps, c1, c2);
    M[i] = m;
    V[i] = v;
    P[i] = p;
}

// ---- an epoch in one launch -------------------------------------------------
// All minibatches of an epoch by one thread-block cluster.  CTA r takes the
// minibatch's groups r, r + C, ... of kS samples: forward and backward passes
// from the CTA's own copy of the parameters in shared memory, each group's
// gradient sums into its own slot there.  After a cluster barrier every CTA
// sums its share of the parameters over the groups in group order (reads of
// the other CTAs' shared memory), applies Adam, and stores the new values to
// every CTA's copy; a second barrier starts the next minibatch.  Every sum
// runs in the order of k_mlp_fwd, k_mlp_bwd and k_mlp_reduce.  The next
// group's order entries, then its samples, are loaded into registers while the
// current group is worked on; Adam's moments stay in the owner's shared memory.
//
// What bounds it: latency (a minibatch of 128 is 4.6 MFLOP on 8 SMs).  As four
// launches, two copies of the host-gathered batch and a read of the loss, a
// minibatch of 128 took 71 us; in the cluster 13.5 us with scalar shared-memory
// accesses and 9 us with 16-byte ones (9.1 -> 1.4 ms for two epochs of 8192
// samples, the copies of the samples and the shuffles included).
struct TrainArgs {
    Shape sh;
    float *P, *M, *V;
    const float *X, *T;      // all samples
    const int *idx;          // the epoch's order
    const float *c;          // Adam's bias corrections c1, c2 per minibatch
    float *loss;             // mean loss per minibatch
    int B, nbt, slots;       // batch, minibatches, group slots per CTA
    float lr, b1, b2, eps;
};

constexpr int kTrainThreads = 256;
constexpr int kTrainCtas = 8;                 // portable cluster size
constexpr int kQ = kTrainThreads / kH;        // samples per pass over the hidden units
constexpr int kSq = kS / kQ;                  // samples per thread
constexpr int kHp = kH + 4;                   // activation rows: 16-byte aligned, conflict-free down a column
constexpr size_t kTrainSmemMax = 227 * 1024;

// Parameters, gradients and moments move in 16-byte chunks: flat arrays
// padded to whole chunks.  The shared-memory copy is flat but for W2, whose row
// u holds its 16 chunks rotated by u: chunk reads of a column of rows (the
// forward pass) and reads along a row (the backward pass) are both free of bank
// conflicts.
__host__ __device__ inline int train_chunks(const Shape &sh) { return (sh.n + 3) / 4; }
__device__ __forceinline__ int w2_chunk(int u, int c) { return u * (kH / 4) + ((c + u) & (kH / 4 - 1)); }
__device__ __forceinline__ int chunk_place(const Shape &sh, int f) {
    const int c = f - sh.oW2 / 4;
    return (c >= 0 && c < kH * kH / 4) ? sh.oW2 / 4 + w2_chunk(c / (kH / 4), c % (kH / 4)) : f;
}

// activations and deltas of one group of samples
struct alignas(16) TrainAct {
    float xs[kS][kMaxIn];
    float h1[kS][kHp], h2[kS][kHp], d1[kS][kHp], d2[kS][kHp];
    float dy[kS][kMaxOut];
    float lsum[kH];
};

inline int train_slots(int B, int ctas) { return ((B + kS - 1) / kS + ctas - 1) / ctas; }
inline size_t train_smem(const Shape &sh, int slots, int ctas) {
    const int nc = train_chunks(sh), share = (nc + ctas - 1) / ctas;
    return sizeof(TrainAct) + 16 * static_cast<size_t>(nc + 2 * share + slots * (nc + 1));
}

// v += w . x of one chunk, in element order
__device__ __forceinline__ float fma4(float4 w, float4 x, float v) {
    v = fmaf(w.x, x.x, v);
    v = fmaf(w.y, x.y, v);
    v = fmaf(w.z, x.z, v);
    return fmaf(w.w, x.w, v);
}
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

__global__ void __launch_bounds__(kTrainThreads) k_mlp_epoch(const __grid_constant__ TrainArgs a) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ float4 smf[];
    const Shape &sh = a.sh;
    const int C = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
    const int t = threadIdx.x, u = t % kH, q = t / kH;
    const int ni = sh.nin, no = sh.nout, B = a.B, ng = (B + kS - 1) / kS;
    // this CTA's share of the parameters: chunks p0 + t, p0 + t + blockDim ...
    const int nc = train_chunks(sh), share = (nc + C - 1) / C, p0 = min(rank * share, nc), p1 = min(p0 + share, nc);
    TrainAct &act = *reinterpret_cast<TrainAct *>(smf);
    float4 *W4 = smf + sizeof(TrainAct) / 16;            // parameters
    float4 *M4 = W4 + nc, *V4 = M4 + share;              // Adam's moments of the CTA's share
    float4 *G4 = V4 + share;                             // slots x (gradient chunks, loss partial)
    float *W = reinterpret_cast<float *>(W4);
    const float *W1 = W + sh.oW1, *b1 = W + sh.ob1, *b2 = W + sh.ob2, *W3 = W + sh.oW3, *b3 = W + sh.ob3;
    const float4 *W2 = W4 + sh.oW2 / 4;
    auto flat4 = [&](const float *p, int f) {   // chunk f of a flat array of sh.n floats
        float4 x;
        x.x = p[4 * f];
        x.y = (4 * f + 1 < sh.n) ? p[4 * f + 1] : 0.0f;
        x.z = (4 * f + 2 < sh.n) ? p[4 * f + 2] : 0.0f;
        x.w = (4 * f + 3 < sh.n) ? p[4 * f + 3] : 0.0f;
        return x;
    };
    for (int f = t; f < nc; f += kTrainThreads) W4[chunk_place(sh, f)] = flat4(a.P, f);
    for (int f = p0 + t; f < p1; f += kTrainThreads) {
        M4[f - p0] = flat4(a.M, f);
        V4[f - p0] = flat4(a.V, f);
    }
    for (int i = t; i < kS * kMaxIn; i += kTrainThreads) act.xs[i / kMaxIn][i % kMaxIn] = 0.0f;
    // a group's inputs and targets in registers: element i = t + r blockDim of
    // its kS x ni inputs, element t of its kS x no targets
    constexpr int kXr = kS * kMaxIn / kTrainThreads;
    static_assert(kS * kMaxOut <= kTrainThreads, "one target per thread");
    int xi[kXr], ti = 0;
    float xv[kXr], tv = 0.0f;
    auto load_order = [&](int mb, int g) {   // sample numbers (-1: past the batch)
        const int s0 = g * kS;
        const int *id = a.idx + static_cast<size_t>(mb) * B + s0;
#pragma unroll
        for (int r = 0; r < kXr; ++r) {
            const int i = t + r * kTrainThreads, s = i / ni;
            xi[r] = (i < kS * ni && s0 + s < B) ? id[s] : -1;
        }
        ti = (t < kS * no && s0 + t / no < B) ? id[t / no] : -1;
    };
    auto load_samples = [&]() {
#pragma unroll
        for (int r = 0; r < kXr; ++r)
            xv[r] = (xi[r] >= 0) ? a.X[static_cast<size_t>(xi[r]) * ni + (t + r * kTrainThreads) % ni] : 0.0f;
        tv = (ti >= 0) ? a.T[static_cast<size_t>(ti) * no + t % no] : 0.0f;
    };
    if (rank < ng) {
        load_order(0, rank);
        load_samples();
    }
    __syncthreads();
    for (int mb = 0; mb < a.nbt; ++mb) {
        for (int gi = 0, g = rank; g < ng; ++gi, g += C) {
            const int s0 = g * kS, ns = min(kS, B - s0);
            float *G = reinterpret_cast<float *>(G4 + static_cast<size_t>(gi) * (nc + 1));
#pragma unroll
            for (int r = 0; r < kXr; ++r) {
                const int i = t + r * kTrainThreads;
                if (i < kS * ni) act.xs[i / ni][i % ni] = xv[r];
            }
            const float target = tv;
            const bool same = g + C < ng, more = same || mb + 1 < a.nbt;   // the group after this one
            if (more) load_order(same ? mb : mb + 1, same ? g + C : rank);
            __syncthreads();
            // forward: unit u of samples q, q + kQ, ...
            {
                float v[kSq];
#pragma unroll
                for (int r = 0; r < kSq; ++r) v[r] = b1[u];
                const float *w1 = W1 + u * ni;
                int k = 0;
                for (; k + 4 <= ni; k += 4) {
                    const float4 w = make_float4(w1[k], w1[k + 1], w1[k + 2], w1[k + 3]);
#pragma unroll
                    for (int r = 0; r < kSq; ++r) v[r] = fma4(w, ld4(&act.xs[q + kQ * r][k]), v[r]);
                }
                for (; k < ni; ++k) {
                    const float w = w1[k];
#pragma unroll
                    for (int r = 0; r < kSq; ++r) v[r] = fmaf(w, act.xs[q + kQ * r][k], v[r]);
                }
#pragma unroll
                for (int r = 0; r < kSq; ++r) act.h1[q + kQ * r][u] = tanhf(v[r]);
            }
            __syncthreads();
            {
                float v[kSq];
#pragma unroll
                for (int r = 0; r < kSq; ++r) v[r] = b2[u];
#pragma unroll 4
                for (int c = 0; c < kH / 4; ++c) {
                    const float4 w = W2[w2_chunk(u, c)];
#pragma unroll
                    for (int r = 0; r < kSq; ++r) v[r] = fma4(w, ld4(&act.h1[q + kQ * r][4 * c]), v[r]);
                }
#pragma unroll
                for (int r = 0; r < kSq; ++r) act.h2[q + kQ * r][u] = tanhf(v[r]);
            }
            __syncthreads();
            // outputs and their errors (kept in d1, free until the backward
            // pass writes it)
            if (more) load_samples();
            if (t < kS * no) {
                const int s = t / no, o = t - s * no;
                float e = 0.0f;
                if (s < ns) {
                    const float *w3 = W3 + o * kH;
                    float v = b3[o];
#pragma unroll
                    for (int c = 0; c < kH / 4; ++c) v = fma4(ld4(w3 + 4 * c), ld4(&act.h2[s][4 * c]), v);
                    e = v - target;
                }
                act.dy[s][o] = 2.0f * e / static_cast<float>(B);
                act.d1[s][o] = e;
            }
            __syncthreads();
            if (t < kH) {
                float l = 0.0f;
                for (int i = t; i < kS * no; i += kH) {
                    const float e = act.d1[i / no][i % no];
                    l = fmaf(e, e, l);
                }
                act.lsum[t] = l;
            }
            // layer 3 gradients; d2 = (W3^T dy) * (1 - h2^2)
            for (int i = t; i < no * kH; i += kTrainThreads) {
                const int o = i / kH, k = i - o * kH;
                float v = 0.0f;
#pragma unroll
                for (int s = 0; s < kS; ++s) v = fmaf(act.dy[s][o], act.h2[s][k], v);
                G[sh.oW3 + i] = v;
            }
            if (t < no) {
                float v = 0.0f;
#pragma unroll
                for (int s = 0; s < kS; ++s) v += act.dy[s][t];
                G[sh.ob3 + t] = v;
            }
#pragma unroll
            for (int r = 0; r < kSq; ++r) {
                const int s = q + kQ * r;
                float v = 0.0f;
                for (int o = 0; o < no; ++o) v = fmaf(W3[o * kH + u], act.dy[s][o], v);
                act.d2[s][u] = v * (1.0f - act.h2[s][u] * act.h2[s][u]);
            }
            __syncthreads();
            // dW2: a 4 x 4 block per thread (units j0 .., inputs k0 ..)
            {
                const int j0 = 4 * (t / 16), k0 = 4 * (t % 16);
                float v[4][4] = {};
#pragma unroll 4
                for (int s = 0; s < kS; ++s) {
                    const float4 x = ld4(&act.d2[s][j0]), y = ld4(&act.h1[s][k0]);
                    const float xx[4] = {x.x, x.y, x.z, x.w}, yy[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int c = 0; c < 4; ++c) v[j][c] = fmaf(xx[j], yy[c], v[j][c]);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    reinterpret_cast<float4 *>(G + sh.oW2)[(j0 + j) * (kH / 4) + t % 16] =
                        make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
            }
            if (t < kH) {
                float v = 0.0f;
#pragma unroll
                for (int s = 0; s < kS; ++s) v += act.d2[s][t];
                G[sh.ob2 + t] = v;
            }
            // d1 = (W2^T d2) * (1 - h1^2)
            {
                float v[kSq] = {};
#pragma unroll 2
                for (int j = 0; j < kH; j += 4) {
                    float4 w;
                    w.x = W[sh.oW2 + 4 * w2_chunk(j, u / 4) + u % 4];
                    w.y = W[sh.oW2 + 4 * w2_chunk(j + 1, u / 4) + u % 4];
                    w.z = W[sh.oW2 + 4 * w2_chunk(j + 2, u / 4) + u % 4];
                    w.w = W[sh.oW2 + 4 * w2_chunk(j + 3, u / 4) + u % 4];
#pragma unroll
                    for (int r = 0; r < kSq; ++r) v[r] = fma4(w, ld4(&act.d2[q + kQ * r][j]), v[r]);
                }
#pragma unroll
                for (int r = 0; r < kSq; ++r) {
                    const int s = q + kQ * r;
                    act.d1[s][u] = v[r] * (1.0f - act.h1[s][u] * act.h1[s][u]);
                }
            }
            __syncthreads();
            // dW1: unit u, input chunks q, q + kQ, ... (inputs past ni are zero)
            for (int k = 4 * q; k < ni; k += 4 * kQ) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int s = 0; s < kS; ++s) {
                    const float d = act.d1[s][u];
                    const float4 x = ld4(&act.xs[s][k]);
                    v.x = fmaf(d, x.x, v.x);
                    v.y = fmaf(d, x.y, v.y);
                    v.z = fmaf(d, x.z, v.z);
                    v.w = fmaf(d, x.w, v.w);
                }
                float *g1 = G + sh.oW1 + u * ni + k;
                g1[0] = v.x;
                if (k + 1 < ni) g1[1] = v.y;
                if (k + 2 < ni) g1[2] = v.z;
                if (k + 3 < ni) g1[3] = v.w;
            }
            if (t < kH) {
                float v = 0.0f;
#pragma unroll
                for (int s = 0; s < kS; ++s) v += act.d1[s][t];
                G[sh.ob1 + t] = v;
            } else if (t == kTrainThreads - 1) {
                float v = 0.0f;
#pragma unroll
                for (int i = 0; i < kH; ++i) v += act.lsum[i];
                G[4 * nc] = v;   // the loss partial, after the gradient chunks
            }
            __syncthreads();   // the next group overwrites the activations
        }
        cl.sync();   // every group's gradients are in place
        const float c1 = a.c[2 * mb], c2 = a.c[2 * mb + 1];
        for (int f = p0 + t; f < p1; f += kTrainThreads) {
            float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
            for (int b = 0; b < ng; ++b) {
                const float4 x = *cl.map_shared_rank(G4 + static_cast<size_t>(b / C) * (nc + 1) + f, b % C);
                g.x += x.x;
                g.y += x.y;
                g.z += x.z;
                g.w += x.w;
            }
            const int at = chunk_place(sh, f);
            float4 p = W4[at], m = M4[f - p0], v = V4[f - p0];
            // (the padding of the last chunk: gradient slots that nothing writes)
            adam_update(g.x, p.x, m.x, v.x, a.lr, a.b1, a.b2, a.eps, c1, c2);
            adam_update(g.y, p.y, m.y, v.y, a.lr, a.b1, a.b2, a.eps, c1, c2);
            adam_update(g.z, p.z, m.z, v.z, a.lr, a.b1, a.b2, a.eps, c1, c2);
            adam_update(g.w, p.w, m.w, v.w, a.lr, a.b1, a.b2, a.eps, c1, c2);
            M4[f - p0] = m;
            V4[f - p0] = v;
            for (int c = 0; c < C; ++c) *cl.map_shared_rank(W4 + at, c) = p;
        }
        if (rank == 0 && t == kTrainThreads - 1) {
            float l = 0.0f;
            for (int b = 0; b < ng; ++b)
                l += *cl.map_shared_rank(reinterpret_cast<float *>(G4 + static_cast<size_t>(b / C) * (nc + 1) + nc),
                                         b % C);
            a.loss[mb] = l / static_cast<float>(B);
        }
        cl.sync();   // the new parameters are in every copy, the slots free
    }
    for (int f = p0 + t; f < p1; f += kTrainThreads) {
        const float4 p4 = W4[chunk_place(sh, f)], m4 = M4[f - p0], v4 = V4[f - p0];
        const float p[4] = {p4.x, p4.y, p4.z, p4.w}, m[4] = {m4.x, m4.y, m4.z, m4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (4 * f + i >= sh.n) break;
            a.P[4 * f + i] = p[i];
            a.M[4 * f + i] = m[i];
            a.V[4 * f + i] = v[i];
        }
    }
}

}  // namespace

struct fb_mlp {
    int device = 0;
    Shape sh;
    float *P = nullptr, *M = nullptr, *V = nullptr, *G = nullptr;
    int step = 0;
    // scratch sized for cap samples
    int cap = 0;
    float *X = nullptr, *T = nullptr, *Y = nullptr, *H1 = nullptr, *H2 = nullptr, *Gb = nullptr, *Lb = nullptr,
          *loss = nullptr;
    // fb_mlp_train: all samples, the epoch's order, bias corrections and losses
    int tcap_n = 0, tcap_b = 0;
    float *TX = nullptr, *TT = nullptr, *TC = nullptr, *TL = nullptr;
    int *TI = nullptr;
};

namespace {

#define MK(call)                                     \
    do {                                             \
        if ((call) != cudaSuccess) return FB_ERR_CUDA; \
    } while (0)

int ensure(fb_mlp *m, int B) {
    if (B <= m->cap) return FB_OK;
    cudaFree(m->X);
    cudaFree(m->T);
    cudaFree(m->Y);
    cudaFree(m->H1);
    cudaFree(m->H2);
    cudaFree(m->Gb);
    cudaFree(m->Lb);
    const int nb = (B + kS - 1) / kS;
    MK(cudaMalloc(&m->X, sizeof(float) * B * m->sh.nin));
    MK(cudaMalloc(&m->T, sizeof(float) * B * m->sh.nout));
    MK(cudaMalloc(&m->Y, sizeof(float) * B * m->sh.nout));
    MK(cudaMalloc(&m->H1, sizeof(float) * B * kH));
    MK(cudaMalloc(&m->H2, sizeof(float) * B * kH));
    MK(cudaMalloc(&m->Gb, sizeof(float) * static_cast<size_t>(nb) * m->sh.n));
    MK(cudaMalloc(&m->Lb, sizeof(float) * nb));
    m->cap = B;
    return FB_OK;
}

// buffers of the one-launch epochs: n samples, nbt minibatches per epoch
// (FB_ERR_CUDA: the device has no room; nothing is kept then)
int ensure_train(fb_mlp *m, int n, int nbt) {
    if (n <= m->tcap_n && nbt <= m->tcap_b) return FB_OK;
    const size_t cn = static_cast<size_t>(std::max(n, m->tcap_n)), cb = static_cast<size_t>(std::max(nbt, m->tcap_b));
    auto release = [m] {
        for (float **p : {&m->TX, &m->TT, &m->TC, &m->TL}) {
            cudaFree(*p);
            *p = nullptr;
        }
        cudaFree(m->TI);
        m->TI = nullptr;
        m->tcap_n = m->tcap_b = 0;
    };
    release();
    if (cudaMalloc(&m->TX, sizeof(float) * cn * m->sh.nin) != cudaSuccess ||
        cudaMalloc(&m->TT, sizeof(float) * cn * m->sh.nout) != cudaSuccess ||
        cudaMalloc(&m->TI, sizeof(int) * cn) != cudaSuccess ||
        cudaMalloc(&m->TC, sizeof(float) * 2 * cb) != cudaSuccess ||
        cudaMalloc(&m->TL, sizeof(float) * cb) != cudaSuccess) {
        cudaGetLastError();
        release();
        return FB_ERR_CUDA;
    }
    m->tcap_n = static_cast<int>(cn);
    m->tcap_b = static_cast<int>(cb);
    return FB_OK;
}

// forward + backward + block reduction on the B samples already in m->X, m->T
void grad_on_device(fb_mlp *m, int B) {
    const int nb = (B + kS - 1) / kS;
    k_mlp_fwd<<<nb, kH>>>(m->sh, m->P, m->X, B, m->H1, m->H2, m->Y);
    k_mlp_bwd<<<nb, kH>>>(m->sh, m->P, m->X, m->H1, m->H2, m->Y, m->T, B, m->Gb, m->Lb);
    k_mlp_reduce<<<(m->sh.n + 255) / 256, 256>>>(m->sh.n, nb, m->Gb, m->G, m->Lb, m->loss, B);
}

// fb_mlp_train with one launch per epoch (k_mlp_epoch) on ensure_train's buffers; the host shuffles the
// next epoch's order while the device works on the current one
int train_epochs(fb_mlp *m, const float *x, const float *t, int n, int epochs, int batch, float lr, uint64_t seed,
                 float *loss_out, int ctas, size_t smem) {
    const int nbt = n / batch, used = nbt * batch;
    MK(cudaFuncSetAttribute(k_mlp_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTrainSmemMax)));
    MK(cudaMemcpy(m->TX, x, sizeof(float) * static_cast<size_t>(n) * m->sh.nin, cudaMemcpyHostToDevice));
    MK(cudaMemcpy(m->TT, t, sizeof(float) * static_cast<size_t>(n) * m->sh.nout, cudaMemcpyHostToDevice));
    TrainArgs a{m->sh, m->P, m->M, m->V, m->TX, m->TT, m->TI, m->TC, m->TL, batch, nbt,
                train_slots(batch, ctas), lr, 0.9f, 0.999f, 1e-8f};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(kTrainThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = static_cast<unsigned>(ctas);
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    std::vector<int> idx(static_cast<size_t>(n));
    for (int i = 0; i < n; ++i) idx[static_cast<size_t>(i)] = i;
    std::mt19937_64 rng(seed);
    std::vector<float> c(2 * static_cast<size_t>(nbt));
    for (int e = 0; e < epochs; ++e) {
        std::shuffle(idx.begin(), idx.end(), rng);
        for (int b = 0; b < nbt; ++b) {
            ++m->step;
            c[2 * static_cast<size_t>(b)] = 1.0f - std::pow(a.b1, static_cast<float>(m->step));
            c[2 * static_cast<size_t>(b) + 1] = 1.0f - std::pow(a.b2, static_cast<float>(m->step));
        }
        // (both copies wait for the previous epoch's launch)
        MK(cudaMemcpy(m->TI, idx.data(), sizeof(int) * static_cast<size_t>(used), cudaMemcpyHostToDevice));
        MK(cudaMemcpy(m->TC, c.data(), sizeof(float) * c.size(), cudaMemcpyHostToDevice));
        MK(cudaLaunchKernelEx(&cfg, k_mlp_epoch, a));
    }
    std::vector<float> l(static_cast<size_t>(nbt));
    MK(cudaMemcpy(l.data(), m->TL, sizeof(float) * l.size(), cudaMemcpyDeviceToHost));
    if (loss_out) {
        double esum = 0.0;
        for (float v : l) esum += v;
        *loss_out = static_cast<float>(esum / nbt);
    }
    return FB_OK;
}

}  // namespace

extern "C" {

int fb_mlp_destroy(fb_mlp *m) {
    if (!m) return FB_OK;
    cudaSetDevice(m->device);
    for (float *p : {m->P, m->M, m->V, m->G, m->X, m->T, m->Y, m->H1, m->H2, m->Gb, m->Lb, m->loss, m->TX, m->TT,
                     m->TC, m->TL})
        cudaFree(p);
    cudaFree(m->TI);
    delete m;
    return FB_OK;
}

int fb_mlp_create(int device, int n_in, int n_out, uint64_t seed, fb_mlp **out) {
    if (!out || n_in < 1 || n_in > kMaxIn || n_out < 1 || n_out > kMaxOut) return FB_ERR_STATE;
    *out = nullptr;
    fb_mlp *m = new (std::nothrow) fb_mlp;
    if (!m) return FB_ERR_CUDA;
    m->device = device;
    m->sh = Shape(n_in, n_out);
    if (cudaSetDevice(device) != cudaSuccess) {
        delete m;
        return FB_ERR_CUDA;
    }
    const size_t bytes = sizeof(float) * m->sh.n;
    if (cudaMalloc(&m->P, bytes) != cudaSuccess || cudaMalloc(&m->M, bytes) != cudaSuccess ||
        cudaMalloc(&m->V, bytes) != cudaSuccess || cudaMalloc(&m->G, bytes) != cudaSuccess ||
        cudaMalloc(&m->loss, sizeof(float)) != cudaSuccess) {
        fb_mlp_destroy(m);
        return FB_ERR_CUDA;
    }
    // Glorot-uniform weights, zero biases, from a seeded generator
    std::vector<float> p(static_cast<size_t>(m->sh.n), 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int fan_out, int fan_in) {
        const float a = std::sqrt(6.0f / static_cast<float>(fan_in + fan_out));
        std::uniform_real_distribution<float> u(-a, a);
        for (int i = 0; i < fan_out * fan_in; ++i) p[static_cast<size_t>(off + i)] = u(rng);
    };
    fill(m->sh.oW1, kH, n_in);
    fill(m->sh.oW2, kH, kH);
    fill(m->sh.oW3, n_out, kH);
    if (cudaMemcpy(m->P, p.data(), bytes, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(m->M, 0, bytes) != cudaSuccess || cudaMemset(m->V, 0, bytes) != cudaSuccess) {
        fb_mlp_destroy(m);
        return FB_ERR_CUDA;
    }
    *out = m;
    return FB_OK;
}

int fb_mlp_params(fb_mlp *m, int *n) {
    if (!m || !n) return FB_ERR_STATE;
    *n = m->sh.n;
    return FB_OK;
}

int fb_mlp_get(fb_mlp *m, float *params) {
    if (!m || !params) return FB_ERR_STATE;
    MK(cudaSetDevice(m->device));
    MK(cudaMemcpy(params, m->P, sizeof(float) * m->sh.n, cudaMemcpyDeviceToHost));
    return FB_OK;
}

int fb_mlp_set(fb_mlp *m, const float *params) {
    if (!m || !params) return FB_ERR_STATE;
    MK(cudaSetDevice(m->device));
    MK(cudaMemcpy(m->P, params, sizeof(float) * m->sh.n, cudaMemcpyHostToDevice));
    MK(cudaMemset(m->M, 0, sizeof(float) * m->sh.n));
    MK(cudaMemset(m->V, 0, sizeof(float) * m->sh.n));
    m->step = 0;
    return FB_OK;
}

// outputs for n samples (host arrays: x n x n_in, y n x n_out)
int fb_mlp_predict(fb_mlp *m, const float *x, int n, float *y) {
    if (!m || !x || !y || n < 1) return FB_ERR_STATE;
    MK(cudaSetDevice(m->device));
    int st = ensure(m, n);
    if (st) return st;
    MK(cudaMemcpy(m->X, x, sizeof(float) * n * m->sh.nin, cudaMemcpyHostToDevice));
    k_mlp_fwd<<<(n + kS - 1) / kS, kH>>>(m->sh, m->P, m->X, n, nullptr, nullptr, m->Y);
    MK(cudaGetLastError());
    MK(cudaMemcpy(y, m->Y, sizeof(float) * n * m->sh.nout, cudaMemcpyDeviceToHost));
    return FB_OK;
}

// full-batch loss and gradient (host arrays), for checking the kernels
int fb_mlp_grad(fb_mlp *m, const float *x, const float *t, int n, float *grad, float *loss) {
    if (!m || !x || !t || n < 1 || !grad || !loss) return FB_ERR_STATE;
    MK(cudaSetDevice(m->device));
    int st = ensure(m, n);
    if (st) return st;
    MK(cudaMemcpy(m->X, x, sizeof(float) * n * m->sh.nin, cudaMemcpyHostToDevice));
    MK(cudaMemcpy(m->T, t, sizeof(float) * n * m->sh.nout, cudaMemcpyHostToDevice));
    grad_on_device(m, n);
    MK(cudaGetLastError());
    MK(cudaMemcpy(grad, m->G, sizeof(float) * m->sh.n, cudaMemcpyDeviceToHost));
    MK(cudaMemcpy(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
    return FB_OK;
}

// Adam on minibatches of `batch` samples for `epochs` passes over the n
// samples (host arrays, shuffled each epoch by a seeded generator);
// loss_out (may be null) receives the mean minibatch loss of the last epoch.
int fb_mlp_train(fb_mlp *m, const float *x, const float *t, int n, int epochs, int batch, float lr, uint64_t seed,
                 float *loss_out) {
    if (!m || !x || !t || n < 1 || epochs < 1 || batch < 1) return FB_ERR_STATE;
    MK(cudaSetDevice(m->device));
    batch = std::min(batch, n);
    const int groups = (batch + kS - 1) / kS, ctas = std::min(kTrainCtas, groups);
    const size_t smem = train_smem(m->sh, train_slots(batch, ctas), ctas);
    if (smem <= kTrainSmemMax && ensure_train(m, n, n / batch) == FB_OK)
        return train_epochs(m, x, t, n, epochs, batch, lr, seed, loss_out, ctas, smem);
    // batches whose gradient slots do not fit the cluster's shared memory, or more
    // samples than the device has room for: one minibatch at a time
    int st = ensure(m, batch);
    if (st) return st;
    const int ni = m->sh.nin, no = m->sh.nout;
    std::vector<int> idx(static_cast<size_t>(n));
    for (int i = 0; i < n; ++i) idx[static_cast<size_t>(i)] = i;
    std::mt19937_64 rng(seed);
    std::vector<float> bx(static_cast<size_t>(batch) * ni), bt(static_cast<size_t>(batch) * no);
    double last = 0.0;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int e = 0; e < epochs; ++e) {
        std::shuffle(idx.begin(), idx.end(), rng);
        double esum = 0.0;
        int nbt = 0;
        for (int s0 = 0; s0 + batch <= n; s0 += batch) {
            for (int r = 0; r < batch; ++r) {
                const int i = idx[static_cast<size_t>(s0 + r)];
                std::memcpy(&bx[static_cast<size_t>(r) * ni], x + static_cast<size_t>(i) * ni, sizeof(float) * ni);
                std::memcpy(&bt[static_cast<size_t>(r) * no], t + static_cast<size_t>(i) * no, sizeof(float) * no);
            }
            MK(cudaMemcpy(m->X, bx.data(), sizeof(float) * bx.size(), cudaMemcpyHostToDevice));
            MK(cudaMemcpy(m->T, bt.data(), sizeof(float) * bt.size(), cudaMemcpyHostToDevice));
            grad_on_device(m, batch);
            ++m->step;
            const float c1 = 1.0f - std::pow(b1, static_cast<float>(m->step));
            const float c2 = 1.0f - std::pow(b2, static_cast<float>(m->step));
            k_adam<<<(m->sh.n + 255) / 256, 256>>>(m->sh.n, m->P, m->G, m->M, m->V, lr, b1, b2, eps, c1, c2);
            float l = 0.0f;
            MK(cudaMemcpy(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
            esum += l;
            ++nbt;
        }
        last = nbt ? esum / nbt : 0.0;
    }
    MK(cudaGetLastError());
    if (loss_out) *loss_out = static_cast<float>(last);
    return FB_OK;
}

}  // extern "C"

namespace fb {
// the parameters as the coupling's device-side inference reads them
const float *mlp_params_device(const fb_mlp *m, int *n_in, int *n_out) {
    if (!m) return nullptr;
    if (n_in) *n_in = m->sh.nin;
    if (n_out) *n_out = m->sh.nout;
    return m->P;
}
}  // namespace fb
