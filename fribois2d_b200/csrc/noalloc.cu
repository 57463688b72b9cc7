// fb_cfl_noalloc: the CFL number and mean streamwise velocity of cfl.F90 for
// a caller that cannot allocate device memory.
//
// Who needs this: hosts whose device memory belongs to another runtime --
// a Fortran code whose arrays live in CUDA Fortran or OpenACC data regions,
// or an application that carves all GPU memory out of its own arena under a
// hard budget -- and that therefore must not let a library call cudaMalloc
// (which can fail, fragment the arena, or exceed the budget).  They hand us
// device pointers to their own velocity and grid arrays and get two numbers
// back; nothing is allocated here.
//
// How: the per-block partial results live in one file-scope __device__ array
// of fixed size, shared by every call on a device.  Its device address is
// looked up once per device with cudaGetSymbolAddress (host code must not use
// the symbol itself as a pointer).  The last block of a call to arrive at its
// completion counter combines the partials and clears the counter.  Calls
// take the kCounters counters in turn, and each also clears the one half a
// turn away: two calls whose kernels overlap on the GPU (different streams, no
// ordering between them) race on the partials, and a counter that such a race
// left wrong is right again before its next use.  A captured call cannot take
// turns: it has a counter of its own, which its graph clears ahead of the kernel
// in every replay.
//
// What bounds it: latency.  With one block per row, a single thread that
// combined all rows in order and a memset node for the counter a call took
// 64.4 us at 1024 x 768 cells; with the rows over two blocks per SM, a thread's
// loads issued together and a parallel combination 9.6 us, which is the host's
// time to issue the call.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdio>

#include "../../include/fribois2d.h"

namespace {

constexpr int kThreads = 256;
constexpr unsigned kMaxBlocks = 2 * 148;   // two per SM
constexpr unsigned kCounters = 64;

// [0, 2*kMaxBlocks): per-block (max, sum) pairs; then the completion counters,
// the captured calls' one last
__device__ __align__(256) double g_cfl_scratch[2 * kMaxBlocks + kCounters / 2 + 1];

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// (max, sum) over the block; valid in thread 0
__device__ __forceinline__ void block_max_sum(double &mx, double &sm, double *shm, double *shs) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    mx = warp_max(mx);
    sm = warp_sum(sm);
    if (lane == 0) {
        shm[w] = mx;
        shs[w] = sm;
    }
    __syncthreads();
    if (w == 0) {
        mx = warp_max(lane < kThreads / 32 ? shm[lane] : 0.0);
        sm = warp_sum(lane < kThreads / 32 ? shs[lane] : 0.0);
    }
}

// rows k = 1..n3m over the blocks, two at a time, four columns per thread and
// pass (their loads all issued before the first use); the last block combines
// the blocks' partials; q fields are (j, k) at q[k*pitch + j-1]
__global__ void __launch_bounds__(kThreads, 2)
    k_cfl_rows(double *scratch, unsigned slot, unsigned other, const double *__restrict__ q2, const double *__restrict__ q3, int pitch,
               int n2m, int n3m, const double *__restrict__ rc, const double *__restrict__ zz,
               const double *__restrict__ udx2m, const double *__restrict__ udx3m, double dt, double rext2,
               double alx3, double *out) {
    __shared__ double shm[kThreads / 32], shs[kThreads / 32];
    __shared__ bool last;
    constexpr int kR = 2, kU = 4;
    const int t = threadIdx.x, nb = gridDim.x;
    double mx = 1.0e-8, sm = 0.0;
    for (int k0 = blockIdx.x + 1; k0 <= n3m; k0 += kR * nb) {
        for (int j0 = t + 1; j0 <= n2m; j0 += kU * kThreads) {
            double a2[kR][kU], b2[kR][kU], a3[kR][kU], b3[kR][kU], u2[kU], dy[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int j = min(j0 + u * kThreads, n2m);
                u2[u] = udx2m[j - 1];
                dy[u] = rc[j] - rc[j - 1];
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    const size_t i = static_cast<size_t>(min(k0 + r * nb, n3m)) * pitch + j;
                    a2[r][u] = q2[i - 1];
                    b2[r][u] = q2[i];
                    a3[r][u] = q3[i - 1];
                    b3[r][u] = q3[i + pitch - 1];
                }
            }
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                const int k = k0 + r * nb;
                if (k > n3m) break;
                const double udx3 = udx3m[k - 1], dz = zz[k] - zz[k - 1];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    if (j0 + u * kThreads > n2m) break;
                    const double q = fabs((a2[r][u] + b2[r][u]) * 0.5 * u2[u]) + fabs((a3[r][u] + b3[r][u]) * 0.5 * udx3);
                    mx = fmax(mx, (q == q) ? q : INFINITY);   // a NaN velocity reads as +inf
                    sm = sm + a3[r][u] * dz * dy[u];
                }
            }
        }
    }
    block_max_sum(mx, sm, shm, shs);
    unsigned *counter = reinterpret_cast<unsigned *>(scratch + 2 * kMaxBlocks);
    if (t == 0) {
        scratch[2 * blockIdx.x] = mx;
        scratch[2 * blockIdx.x + 1] = sm;
        __threadfence();
        last = (atomicAdd(counter + slot, 1u) == static_cast<unsigned>(nb - 1));
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    mx = 1.0e-8;
    sm = 0.0;
    for (int b = t; b < nb; b += kThreads) {
        mx = fmax(mx, __ldcg(scratch + 2 * b));
        sm = sm + __ldcg(scratch + 2 * b + 1);
    }
    block_max_sum(mx, sm, shm, shs);
    if (t == 0) {
        out[0] = mx * dt;
        out[1] = sm / (rext2 * alx3);
        counter[slot] = 0u;
        counter[other] = 0u;
    }
}

double *scratch_for_device(int dev) {
    // device addresses of g_cfl_scratch, looked up on first use per device;
    // two host threads may both look it up the first time, and both store
    // the same address
    static std::atomic<double *> addr[64];
    if (dev < 0 || dev >= 64) return nullptr;
    double *a = addr[dev].load(std::memory_order_acquire);
    if (!a) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_cfl_scratch) != cudaSuccess) return nullptr;
        a = static_cast<double *>(p);
        addr[dev].store(a, std::memory_order_release);
    }
    return a;
}

}  // namespace

extern "C" int fb_cfl_noalloc(const double *q2, const double *q3, int pitch, int n2, int n3, const double *rc,
                              const double *zz, const double *udx2m, const double *udx3m, double dt,
                              double rext2, double alx3, double *out, void *stream) {
    if (!q2 || !q3 || !rc || !zz || !udx2m || !udx3m || !out || n2 < 2 || n3 < 2 || pitch < n2)
        return FB_ERR_STATE;
    const int n2m = n2 - 1, n3m = n3 - 1;
    if (n3m > FB_NOALLOC_MAX_ROWS) {
        std::fprintf(stderr,
                     "fribois2d: fb_cfl_noalloc: %d z cells exceed the limit of %d\n",
                     n3m, FB_NOALLOC_MAX_ROWS);
        return FB_ERR_UNSUPPORTED;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return FB_ERR_CUDA;
    double *scratch = scratch_for_device(dev);
    if (!scratch) return FB_ERR_CUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    static std::atomic<unsigned> calls{0};
    unsigned slot, other;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) return FB_ERR_CUDA;
    if (cap == cudaStreamCaptureStatusNone) {
        slot = calls.fetch_add(1, std::memory_order_relaxed) % kCounters;
        other = (slot + kCounters / 2) % kCounters;
    } else {
        slot = other = kCounters;
        unsigned *counter = reinterpret_cast<unsigned *>(scratch + 2 * kMaxBlocks) + slot;
        if (cudaMemsetAsync(counter, 0, sizeof(unsigned), st) != cudaSuccess) return FB_ERR_CUDA;
    }
    // the launch's own status (cudaGetLastError would also return, and clear,
    // an earlier error of the caller's); the runtime may still report an
    // earlier asynchronous error here
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(n3m) < kMaxBlocks ? static_cast<unsigned>(n3m) : kMaxBlocks);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_cfl_rows, scratch, slot, other, q2, q3, pitch, n2m, n3m, rc, zz,
                                             udx2m, udx3m, dt, rext2, alx3, out);
    return e == cudaSuccess ? FB_OK : FB_ERR_CUDA;
}
