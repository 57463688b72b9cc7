// Batched tridiagonal line solves (solve_fluid.F90 solq2j/solq2k/solq3j/
// solq3k and the per-mode y solves of phcalc_outflow.F90:34-56).
//
// Every system is factorised once on the host (DGTTRF without row
// interchanges, which these diagonally dominant systems never need); a
// line solve is then the two first-order recurrences of the LU
// substitution,
//     forward   y(i) = a(i) y(i-1) + b(i),        a(0)   = 0
//     backward  x(i) = e(i) x(i+1) + g(i) y(i),   e(n-1) = 0
// A line is cut into contiguous chunks held in registers by consecutive
// threads.  Each thread composes the affine map of its chunk, a scan over
// the chunks (warp shuffles, plus shared memory across warps for long
// lines) gives every chunk its incoming value, and the chunk is applied.
// Depth is O(n/chunks + log chunks); every element is loaded and stored
// once, with all of a thread's loads independent and in flight together.
//
// Lines along y are contiguous in memory: one warp per line, staged through
// shared memory so that global accesses are coalesced.  Lines along z are
// strided: four neighbouring lines share each 32-byte sector, so a block
// interleaves four lines over its lanes and splits k among its warps.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "device.cuh"
#include "pdl.h"
#include "tri.h"

namespace fb {

#define Fv(a, j, k) (a)[fidx(d, (j), (k))]

namespace {

constexpr unsigned kFull = 0xffffffffu;

struct CoefShared {      // y or z systems: 1-D factors shared by all lines
    const double *a, *e, *g;
    template <int M>
    __device__ __forceinline__ void loadA(double (&c)[M], int i0, int cnt) const {
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) c[t] = __ldg(a + i0 + t);
    }
    template <int M>
    __device__ __forceinline__ void loadE(double (&c)[M], int i0, int cnt) const {
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) c[t] = __ldg(e + i0 + t);
    }
    template <int M>
    __device__ __forceinline__ void loadG(double (&c)[M], int i0, int cnt) const {
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) c[t] = __ldg(g + i0 + t);
    }
};

struct CoefModeS {       // Poisson mode: reciprocal pivots of the mode and the 1-based y
                         // off-diagonals, staged in shared memory
    const double *g, *amphj, *apphj;
    int n;
    template <int M>
    __device__ __forceinline__ void loadA(double (&c)[M], int i0, int cnt) const {
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) {
                const int i = i0 + t;
                c[t] = (i == 0) ? 0.0 : -(amphj[i + 1] * g[i - 1]);
            }
    }
    template <int M>
    __device__ __forceinline__ void loadE(double (&c)[M], int i0, int cnt) const {
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) {
                const int i = i0 + t;
                c[t] = (i == n - 1) ? 0.0 : -(apphj[i + 1] * g[i]);
            }
    }
    template <int M>
    __device__ __forceinline__ void loadG(double (&c)[M], int i0, int cnt) const {
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) c[t] = g[i0 + t];
    }
};

// The chains below only read registers: the coefficients of a chunk are
// loaded into c[] before each recurrence starts.
template <int M>
__device__ __forceinline__ void fwd_compose(const double (&v)[M], const double (&c)[M], int cnt, double &A,
                                            double &C) {
    A = 1.0;
    C = 0.0;
#pragma unroll
    for (int t = 0; t < M; ++t)
        if (t < cnt) {
            C = fma(c[t], C, v[t]);
            A *= c[t];
        }
}

template <int M>
__device__ __forceinline__ void fwd_apply(double (&v)[M], const double (&c)[M], int cnt, double y) {
#pragma unroll
    for (int t = 0; t < M; ++t)
        if (t < cnt) {
            y = fma(c[t], y, v[t]);
            v[t] = y;
        }
}

template <int M>
__device__ __forceinline__ void bwd_compose(const double (&v)[M], const double (&c)[M], int cnt, double &A,
                                            double &C) {
    A = 1.0;
    C = 0.0;
#pragma unroll
    for (int t = M - 1; t >= 0; --t)
        if (t < cnt) {
            C = fma(c[t], C, v[t]);
            A *= c[t];
        }
}

template <int M>
__device__ __forceinline__ void bwd_apply(double (&v)[M], const double (&c)[M], int cnt, double x) {
#pragma unroll
    for (int t = M - 1; t >= 0; --t)
        if (t < cnt) {
            x = fma(c[t], x, v[t]);
            v[t] = x;
        }
}

template <int M>
__device__ __forceinline__ void scale(double (&v)[M], const double (&c)[M], int cnt) {
#pragma unroll
    for (int t = 0; t < M; ++t)
        if (t < cnt) v[t] = c[t] * v[t];
}

// one warp = one line of n unknowns, one contiguous chunk per lane
template <int M, class Co>
__device__ __forceinline__ void warp_line(double (&v)[M], int i0, int cnt, const Co &co) {
    const int lane = threadIdx.x & 31;
    double c[M], A, C;
    co.loadA(c, i0, cnt);
    fwd_compose(v, c, cnt, A, C);
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
        const double Ao = __shfl_up_sync(kFull, A, dd), Co_ = __shfl_up_sync(kFull, C, dd);
        if (lane >= dd) {
            C = fma(A, Co_, C);
            A *= Ao;
        }
    }
    double y = __shfl_up_sync(kFull, C, 1);
    if (lane == 0) y = 0.0;
    fwd_apply(v, c, cnt, y);
    co.loadG(c, i0, cnt);
    scale(v, c, cnt);  // g(i) y(i)
    co.loadE(c, i0, cnt);
    bwd_compose(v, c, cnt, A, C);
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
        const double Ao = __shfl_down_sync(kFull, A, dd), Co_ = __shfl_down_sync(kFull, C, dd);
        if (lane + dd < 32) {
            C = fma(A, Co_, C);
            A *= Ao;
        }
    }
    double x = __shfl_down_sync(kFull, C, 1);
    if (lane == 31) x = 0.0;
    bwd_apply(v, c, cnt, x);
}

// the barrier of one line's G warps (bar > 0: a named one), or the block's
template <int G>
__device__ __forceinline__ void line_sync(int bar) {
    if (bar) asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(32 * G) : "memory");
    else __syncthreads();
}

// G consecutive warps share one line (lane chunks in warp-major order);
// warps exchange their chunk composites through sh (2 * G doubles per line).
template <int M, int G, class Co>
__device__ __forceinline__ void group_line(double (&v)[M], int i0, int cnt, const Co &co, double *sh, int bar = 0) {
    const int lane = threadIdx.x & 31, gw = (threadIdx.x >> 5) % G;
    double c[M], A, C;
    co.loadA(c, i0, cnt);
    fwd_compose(v, c, cnt, A, C);
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
        const double Ao = __shfl_up_sync(kFull, A, dd), Co_ = __shfl_up_sync(kFull, C, dd);
        if (lane >= dd) {
            C = fma(A, Co_, C);
            A *= Ao;
        }
    }
    if (lane == 31) {
        sh[2 * gw] = A;
        sh[2 * gw + 1] = C;
    }
    double Cex = __shfl_up_sync(kFull, C, 1), Aex = __shfl_up_sync(kFull, A, 1);
    if (lane == 0) {
        Aex = 1.0;
        Cex = 0.0;
    }
    line_sync<G>(bar);
    double PC = 0.0;
    for (int q = 0; q < gw; ++q) PC = fma(sh[2 * q], PC, sh[2 * q + 1]);
    fwd_apply(v, c, cnt, fma(Aex, PC, Cex));
    co.loadG(c, i0, cnt);
    scale(v, c, cnt);
    co.loadE(c, i0, cnt);
    line_sync<G>(bar);
    bwd_compose(v, c, cnt, A, C);
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
        const double Ao = __shfl_down_sync(kFull, A, dd), Co_ = __shfl_down_sync(kFull, C, dd);
        if (lane + dd < 32) {
            C = fma(A, Co_, C);
            A *= Ao;
        }
    }
    if (lane == 0) {
        sh[2 * gw] = A;
        sh[2 * gw + 1] = C;
    }
    Cex = __shfl_down_sync(kFull, C, 1);
    Aex = __shfl_down_sync(kFull, A, 1);
    if (lane == 31) {
        Aex = 1.0;
        Cex = 0.0;
    }
    line_sync<G>(bar);
    double SC = 0.0;
    for (int q = G - 1; q > gw; --q) SC = fma(sh[2 * q], SC, sh[2 * q + 1]);
    bwd_apply(v, c, cnt, fma(Aex, SC, Cex));
}

// kZLines lines interleaved over the lanes (line = lane % 4), chunks over
// lane/4 and the block's warps; shA/shC hold one composite per (warp, line)
template <int M, class Co>
__device__ __forceinline__ void block_lines(double (&v)[M], int i0, int cnt, const Co &co, double *shA,
                                            double *shC) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int l = lane & (kZLines - 1), sub = lane / kZLines;
    constexpr int kSub = 32 / kZLines;
    double c[M], A, C, Ao, Co_;
    // ---- forward
    co.loadA(c, i0, cnt);
    fwd_compose(v, c, cnt, A, C);
#pragma unroll
    for (int dd = kZLines; dd < 32; dd <<= 1) {
        Ao = __shfl_up_sync(kFull, A, dd);
        Co_ = __shfl_up_sync(kFull, C, dd);
        if (lane >= dd) {
            C = fma(A, Co_, C);
            A *= Ao;
        }
    }
    if (sub == kSub - 1) {
        shA[w * kZLines + l] = A;
        shC[w * kZLines + l] = C;
    }
    double Aex = __shfl_up_sync(kFull, A, kZLines), Cex = __shfl_up_sync(kFull, C, kZLines);
    if (sub == 0) {
        Aex = 1.0;
        Cex = 0.0;
    }
    __syncthreads();
    double PC = 0.0;
    for (int q = 0; q < w; ++q) PC = fma(shA[q * kZLines + l], PC, shC[q * kZLines + l]);
    fwd_apply(v, c, cnt, fma(Aex, PC, Cex));
    co.loadG(c, i0, cnt);
    scale(v, c, cnt);
    co.loadE(c, i0, cnt);
    __syncthreads();
    // ---- backward
    bwd_compose(v, c, cnt, A, C);
#pragma unroll
    for (int dd = kZLines; dd < 32; dd <<= 1) {
        Ao = __shfl_down_sync(kFull, A, dd);
        Co_ = __shfl_down_sync(kFull, C, dd);
        if (lane + dd < 32) {
            C = fma(A, Co_, C);
            A *= Ao;
        }
    }
    if (sub == 0) {
        shA[w * kZLines + l] = A;
        shC[w * kZLines + l] = C;
    }
    Aex = __shfl_down_sync(kFull, A, kZLines);
    Cex = __shfl_down_sync(kFull, C, kZLines);
    if (sub == kSub - 1) {
        Aex = 1.0;
        Cex = 0.0;
    }
    __syncthreads();
    double SC = 0.0;
    for (int q = W - 1; q > w; --q) SC = fma(shA[q * kZLines + l], SC, shC[q * kZLines + l]);
    bwd_apply(v, c, cnt, fma(Aex, SC, Cex));
}

}  // namespace

// ---------------------------------------------------------------- y lines

// Rows of a k-major field staged through shared memory: load row (scaled),
// solve with a warp per line, write back.  kind: 0 = solq2j, 1 = solq3j,
// 2 = Poisson mode (rows of hmn).
// kKind 0: the v and w systems of helsolve in one launch (solq2j on rows
// k = 1..n3m of rhs2, then solq3j on rows k = 2..n3m of rhs3; they are
// independent).  kKind 2: Poisson modes (rows of hmn).
// W: warps per line (the Poisson modes use 4: fewer values and registers per
// thread, more lines resident per SM)
template <int M, int kKind, int W = kYWarps>
__device__ __forceinline__ void ylines_body(const Dev &d, const ScanSys &s2, const double *by2, const ScanSys &s3, const double *by3) {
    extern __shared__ double sm[];
    __shared__ double shx[kYLines][2 * W];
    const int wl = (threadIdx.x >> 5) / W;       // line slot in the block
    const int tl = threadIdx.x % (32 * W);       // thread within the line group
    int line = blockIdx.x * kYLines + wl;
    int sys = 0, n, r;
    if (kKind == 2) {
        n = d.n2m;
        r = line;
        if (r >= d.n3m) r = -1;
    } else if (line < d.n3m) {
        sys = 0;
        n = d.n2;
        r = line + 1;
    } else {
        sys = 1;
        n = d.n2m;
        r = line - d.n3m + 2;
        if (r > d.n3m) r = -1;
    }
    const bool live = (r >= 0);
    if (!live) n = d.n2m;  // idle line slot: still takes part in the block barriers
    double *row = nullptr;
    if (live) row = (kKind == 2) ? d.hmn + static_cast<size_t>(r) * d.ldh : (sys == 0 ? d.rhs2 : d.rhs3) + fidx(d, 1, r);
    const double *by = (sys == 0) ? by2 : by3;
    double *buf = sm + wl * (d.n2 + 1);
    constexpr int kT = 32 * W;
    // Poisson modes: the mode's reciprocal pivots and the y off-diagonals
    // are staged with the line, so the recurrences read shared memory only
    double *pgs = sm + kYLines * (d.n2 + 1) + wl * (d.n2m + 1);
    double *ams = sm + kYLines * (d.n2 + 1) + kYLines * (d.n2m + 1), *aps = ams + (d.n2m + 2);
    if (kKind == 2) {
        for (int i = threadIdx.x; i <= d.n2m; i += blockDim.x) {
            ams[i] = __ldg(d.amphj + i);
            aps[i] = __ldg(d.apphj + i);
        }
    }
    // coalesced staging: thread-strided loads, all independent
    if (live) {
        const double *pgr = d.pg + static_cast<size_t>(r) * d.ldh;
#pragma unroll
        for (int it = 0; it < M; ++it) {
            const int i = tl + kT * it;
            if (i < n) {
                double v = __ldcg(row + i);
                if (kKind != 2) {
                    if (sys == 0) v = (i >= 1 && i <= n - 2) ? v * __ldg(by + i + 1) : 0.0;
                    else v = v * __ldg(by + i + 1);
                } else {
                    pgs[i] = __ldg(pgr + i);
                }
                buf[i] = v;
            }
        }
    }
    __syncthreads();
    const int m = ((n + kT - 1) / kT) | 1;  // odd chunk: conflict-free 64-bit shared loads
    const int i0 = min(tl * m, n), cnt = live ? min(m, n - i0) : 0;
    double v[M];
#pragma unroll
    for (int t = 0; t < M; ++t)
        if (t < cnt) v[t] = buf[i0 + t];
    if (kKind == 2) {
        group_line<M, W>(v, i0, cnt, CoefModeS{pgs, ams, aps, n}, shx[wl]);
    } else {
        const ScanSys &s = (sys == 0) ? s2 : s3;
        group_line<M, W>(v, i0, cnt, CoefShared{s.a, s.e, s.g}, shx[wl]);
    }
#pragma unroll
    for (int t = 0; t < M; ++t)
        if (t < cnt) buf[i0 + t] = v[t];
    __syncthreads();
    if (live) {
#pragma unroll
        for (int it = 0; it < M; ++it) {
            const int i = tl + kT * it;
            if (i < n) row[i] = buf[i];
        }
    }
}

template <int M, int kKind, int W = kYWarps>
__global__ void __launch_bounds__(kYLines * W * 32) k_ylines(Dev d, ScanSys s2, const double *by2, ScanSys s3, const double *by3) {
    FB_GRID_WAIT();
    ylines_body<M, kKind, W>(d, s2, by2, s3, by3);
}

// ---------------------------------------------------------------- Poisson modes

// The per-mode y solves of phcalc (phcalc_outflow.F90:34-56): W warps per
// mode.  The block copies the y off-diagonals once and each mode's warps its
// right-hand side (a row of hmn) and reciprocal pivots to the mode's own
// shared-memory rows, all with cp.async in flight together (one wait instead
// of a round trip per element group), then solves with lane chunks of an odd
// length m (conflict-free 8-byte shared accesses): the forward recurrence
// y(i) = a(i) y(i-1) + b(i), a(i) = -amphj(i+1) g(i-1), scaled by g(i), and the
// backward one with e(i) = -apphj(i+1) g(i), each composed per chunk, scanned
// over the chunks and applied.  A chunk and its coefficients are held in
// registers (M >= m of them, every loop unrolled), so a step of a chain is one
// dependent FMA: with the chunk in shared memory a step also waits for its loads
// behind the store of the step before, ~100 cycles, and the solve took 8.7 of
// the 14.5 us between the launches before and after it at 1024 x 768 (8.4 us
// now).  A longer chunk does not fit the registers: up to 1088 unknowns two warps
// share a mode (1500 x 1000: 19.5 -> 16.6 us), above that the chunk stays in
// shared memory (M = 0; 1536 unknowns: 26.2 us, 30.4 with two and 31.7 with three
// warps, whose registers spill, 39.5 with the chunk in two register parts).  The
// split-precision form (one_warp) never takes two: a scan over more lanes rounds
// differently, and its TF32 roundings turn a last bit into 1e-8 of the pressure.
// nw modes per block, as many as the shared memory holds.

constexpr int kYmModes = 8;   // modes per block at most

// one warp's mode with its chunks in shared memory (solved in place)
__device__ __forceinline__ void ymodes_loop(int n, const double *am, const double *ap, double *line,
                                            const double *piv) {
    const int lane = threadIdx.x & 31;
    const int m = ((n + 31) / 32) | 1;
    const int i0 = min(lane * m, n), cnt = min(m, n - i0);
    // forward: composite of the chunk, y_out = A y_in + C
    double A = 1.0, C = 0.0;
    for (int t = 0; t < cnt; ++t) {
        const int i = i0 + t;
        const double a = (i == 0) ? 0.0 : -(am[i + 1] * piv[i - 1]);
        C = fma(a, C, line[i]);
        A *= a;
    }
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
        const double Ao = __shfl_up_sync(kFull, A, dd), Co = __shfl_up_sync(kFull, C, dd);
        if (lane >= dd) {
            C = fma(A, Co, C);
            A *= Ao;
        }
    }
    double y = __shfl_up_sync(kFull, C, 1);
    if (lane == 0) y = 0.0;
    for (int t = 0; t < cnt; ++t) {
        const int i = i0 + t;
        const double a = (i == 0) ? 0.0 : -(am[i + 1] * piv[i - 1]);
        y = fma(a, y, line[i]);
        line[i] = piv[i] * y;   // g(i) y(i)
    }
    // backward: x(i) = e(i) x(i+1) + g(i) y(i)
    A = 1.0;
    C = 0.0;
    for (int t = cnt - 1; t >= 0; --t) {
        const int i = i0 + t;
        const double e = (i == n - 1) ? 0.0 : -(ap[i + 1] * piv[i]);
        C = fma(e, C, line[i]);
        A *= e;
    }
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
        const double Ao = __shfl_down_sync(kFull, A, dd), Co = __shfl_down_sync(kFull, C, dd);
        if (lane + dd < 32) {
            C = fma(A, Co, C);
            A *= Ao;
        }
    }
    double x = __shfl_down_sync(kFull, C, 1);
    if (lane == 31) x = 0.0;
    for (int t = cnt - 1; t >= 0; --t) {
        const int i = i0 + t;
        const double e = (i == n - 1) ? 0.0 : -(ap[i + 1] * piv[i]);
        x = fma(e, x, line[i]);
        line[i] = x;
    }
}

// rmax (may be null): the maxima of |hmn| over each row j (over the modes:
// the rows of the INT8 transform's data operand) are accumulated into rmax[j]
// from the block's modes, for the digit cut that follows
// kWait: the body waits for the kernel before it (the transform, which writes
// hmn) once the constant operands are under way.
template <int M, int W, bool kWait>
__device__ __forceinline__ void ymodes_body(const Dev &d, int nw, double *rmax = nullptr) {
    extern __shared__ double sm[];
    __shared__ double shx[kYmModes][2 * W];
    const int n = d.n2m, w = threadIdx.x / (32 * W), tl = threadIdx.x % (32 * W);
    double *am = sm, *ap = sm + (n + 2);                       // 1-based off-diagonals
    double *lines = sm + 2 * (n + 2);
    double *line = lines + static_cast<size_t>(w) * 2 * (n + 1);
    double *piv = line + (n + 1);
    // every copy of the block in flight at once (cp.async), one wait
    for (int i = threadIdx.x; i <= n + 1; i += blockDim.x) {
        cp8(am + i, d.amphj + i);
        cp8(ap + i, d.apphj + i);
    }
    const int r = blockIdx.x * nw + w;
    const bool live = r < d.n3m;
    if (live) {
        const double *pgr = d.pg + static_cast<size_t>(r) * d.ldh;
        for (int i = tl; i < n; i += 32 * W) cp8(piv + i, pgr + i);
    }
    if (kWait) FB_GRID_WAIT();
    if (live) {
        const double *row = d.hmn + static_cast<size_t>(r) * d.ldh;
        for (int i = tl; i < n; i += 32 * W) cp8(line + i, row + i);
    }
    cp_wait();
    __syncthreads();   // the off-diagonals (and every line) are staged
    if (live) {
        if constexpr (M == 0) {
            ymodes_loop(n, am, ap, line, piv);
        } else {
            const int m = ((n + 32 * W - 1) / (32 * W)) | 1;
            const int i0 = min(tl * m, n), cnt = min(m, n - i0);
            double v[M];
#pragma unroll
            for (int t = 0; t < M; ++t)
                if (t < cnt) v[t] = line[i0 + t];
            const CoefModeS co{piv, am, ap, n};
            if constexpr (W == 1) warp_line<M>(v, i0, cnt, co);
            else group_line<M, W>(v, i0, cnt, co, shx[w], w + 1);
#pragma unroll
            for (int t = 0; t < M; ++t)
                if (t < cnt) line[i0 + t] = v[t];
        }
    }
    __syncthreads();   // every live mode's solved line is in shared memory
    const int nlive = max(0, min(nw, d.n3m - static_cast<int>(blockIdx.x) * nw));
    double *row0 = d.hmn + static_cast<size_t>(blockIdx.x) * nw * d.ldh;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        double mx = 0.0;
#pragma unroll 4
        for (int q = 0; q < nlive; ++q) {
            const double x = lines[static_cast<size_t>(q) * 2 * (n + 1) + j];
            row0[static_cast<size_t>(q) * d.ldh + j] = x;
            mx = fmax(mx, fabs(x));
        }
        if (rmax && mx > 0.0) atomic_max_nonneg(rmax + j, mx);
    }
}

template <int M, int W>
__global__ void __launch_bounds__(32 * W * kYmModes, 1) k_ymodes(Dev d, int nw, double *rmax) {
    ymodes_body<M, W, true>(d, nw, rmax);
}

template <int M, int W>
__global__ void __launch_bounds__(32 * W * kYmModes, 1) kg_ymodes(const GroupCase *__restrict__ g, int nw) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    ymodes_body<M, W, false>(d, nw, g[blockIdx.z].rmax_hmn);
}

// ---------------------------------------------------------------- z lines

// solq2k (+ helsolve wall columns) on blocks [0, nb2) and solq3k on the
// rest, one launch (the two are independent).  Lines j0..j0+3.
template <int M, int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads) k_zlines(Dev d, SubDev sd, int nb2) {
    FB_GRID_WAIT();
    __shared__ double shA[16 * kZLines], shC[16 * kZLines];
    const int kKind = (static_cast<int>(blockIdx.x) < nb2) ? 0 : 1;
    const int blk = (kKind == 0) ? blockIdx.x : blockIdx.x - nb2;
    const ScanSys &s = (kKind == 0) ? sd.sz2 : sd.sz3;
    const double *bz = (kKind == 0) ? sd.bz2 : sd.bz3;
    const double ugkks = sd.ugkks, ugkkn = sd.ugkkn;
    const int n = (kKind == 0) ? d.n3m : d.n3;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int l = lane & (kZLines - 1);
    const int c = w * (32 / kZLines) + lane / kZLines;  // chunk index within the line
    const int nc = W * (32 / kZLines);
    const int m = (n + nc - 1) / nc;
    const int i0 = min(c * m, n), cnt = min(m, n - i0);
    const int j0 = blk * kZLines + 1, j = j0 + l;
    const bool live = (j <= d.n2m) && (kKind == 1 || j >= 2);
    const int jj = live ? j : 2;  // a valid column for the (discarded) loads of idle lanes
    const double *src = (kKind == 0) ? d.rhs2 : d.rhs3;
    double v[M];
    // gather this thread's chunk (row k = i + 1 of column j): loads first
#pragma unroll
    for (int t = 0; t < M; ++t)
        if (t < cnt) v[t] = __ldcg(src + fidx(d, jj, i0 + t + 1));
    double *qf = (kKind == 0) ? d.q2 : d.q3;
    double bs = 0.0, bn = 0.0;
    if (kKind == 0) {
        bs = d.dqb2s[jj] * ugkks;
        bn = d.dqb2n[jj] * ugkkn;
    } else {
        bs = d.dqb3s[jj];
        bn = d.dqb3n[jj];
    }
#pragma unroll
    for (int t = 0; t < M; ++t)
        if (t < cnt) {
            const int k = i0 + t + 1;
            double x = 0.0;
            if (live) {
                if (kKind == 0) {
                    x = v[t] * __ldg(bz + k);
                    if (k == 1) x = x + bs;
                    if (k == n) x = x + bn;
                } else {
                    if (k == 1) x = bs;
                    else if (k == n) x = bn;
                    else x = v[t] * __ldg(bz + k);
                }
            }
            v[t] = x;
        }
    block_lines(v, i0, cnt, CoefShared{s.a, s.e, s.g}, shA, shC);
    if (live) {
        double q[M];
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) q[t] = __ldcg(qf + fidx(d, j, i0 + t + 1));
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) {
                const int k = i0 + t + 1;
                const double add = (kKind == 1 && k == n) ? bn : v[t];
                qf[fidx(d, j, k)] = q[t] + add;
            }
    }
    if (kKind == 0 && j0 == 1) {
        for (int k = threadIdx.x; k <= d.n3; k += blockDim.x) {
            Fv(d.q2, 1, k) = 0.0;
            Fv(d.q2, d.n2, k) = 0.0;
        }
    }
}

// ---------------------------------------------------------------- windowed ADI

// helsolve (helsolve.F90:4-56 with solq2j/solq2k/solq3j/solq3k) as one
// launch over 2-D tiles, both velocity components.  The four Helmholtz
// operators are strongly diagonally dominant (off-diagonals ~ beta*al/h^2
// against a unit diagonal), so the influence of a value on the LU
// recurrences dies out geometrically: the products of K+1 consecutive
// multipliers a(i) (forward) and e(i) (backward) fall below 2^-56 for a
// window K that the host measures from the factors of each substep
// (overlapped, truncated partitions: the truncated-SPIKE idea of Polizzi and
// Sameh for diagonally dominant banded systems).  A thread computes a segment
// of kWSeg unknowns exactly as the sequential recurrences would, except that it
// starts the forward one K positions before the segment, from zero, and the
// backward one K positions behind it; the forward values stay in registers
// between the two, and segments need no communication.  A tile runs two phases
// through shared memory: the y solves of its rows plus a halo of K rows on
// either side in k, then the z solves of its columns, added to q2/q3.
// rhs2/rhs3 are read once and q2/q3 read and written once; the tile of q and
// the recurrence coefficients are staged in shared memory with the right-hand
// side, all of it in flight at once.
//
// What bounds it: shared-memory reads and the latency of the chains.  As four
// phases (forward and backward recurrences apart, their values exchanged
// through shared memory) a tile of 32 x 64 made 53 thousand 8-byte accesses and
// three blocks of 72 KB fitted an SM; the fused segments make 28 thousand
// (coefficients in pairs) and 51 KB.  Repeated behind itself (fb_time_stage):
// 20.6 -> 16.6 us at 1024 x 768, 88.4 -> 72.9 at 2048 x 1536 (K = 15), 8.7 -> 6.2 at
// 384 x 256 and 7.8 -> 5.6 at 48 x 32 (the last two with 32 instead of 64 rows too).
constexpr int kWTj = 32;        // tile columns (j): one lane each in the z phase
constexpr int kWSeg = 16;       // unknowns per thread segment
constexpr int kWThreads = 192;  // six warps: the y segments of a 32 x 64 tile with K <= 16
constexpr int kWXp = kWTj + 1;  // row stride of the z right-hand side tile (odd: conflict-free column stores)

namespace {

// One segment: x(i) for the kWSeg positions from s on, i = s + t, from
//   y(i) = a(i) y(i-1) + F(i)   (positions from s - K on, and from line index 0)
//   x(i) = e(i) x(i+1) + g(i) y(i)   (positions below s + kWSeg + K)
// A(u), F(u), EG(u) are indexed relative to s; lo: line index 0 relative to s;
// positions at or past nmax are outside the line (x stays 0).
// kB > 0: the forward recurrence starts anew, K positions early and from zero, at
// the positions that are multiples of kB from the tile's edge (b0: the last of
// them at or before s, relative to s) instead of once before s.  The values
// differ by less than 2^-56 of their influence.  The split-precision Poisson
// form takes it, with the blocks of 24 (y) and 16 (z) positions that its results
// have always been computed with: its TF32 roundings turn a last bit of the
// right-hand side into 1e-8 of the pressure.
template <int KM, int kB, class FA, class FE>
__device__ __forceinline__ void win_segment(const FA &AF, const FE &EG, int K, int lo, int nmax, int b0,
                                            double (&x)[kWSeg]) {
    double y[kWSeg + KM], v = 0.0;
    if constexpr (kB == 0) {
#pragma unroll
        for (int u = -KM; u < 0; ++u)
            if (u >= -K && u >= lo) v = AF(u, v);
    } else {
        for (int u = max(b0 - K, lo); u < 0; ++u) v = AF(u, v);
    }
#pragma unroll
    for (int t = 0; t < kWSeg + KM; ++t) {
        y[t] = 0.0;
        if (t < kWSeg + K && t < nmax) {
            if (kB > 0 && t > 0 && (t - b0) % (kB > 0 ? kB : 1) == 0) {
                v = 0.0;
                for (int u = max(t - K, lo); u < t; ++u) v = AF(u, v);
            }
            v = AF(t, v);
            y[t] = v;
        }
    }
    v = 0.0;
#pragma unroll
    for (int t = kWSeg + KM - 1; t >= 0; --t) {
        if (t < kWSeg + K && t < nmax) {
            const double2 c = EG(t);
            v = fma(c.x, v, c.y * y[t]);
        }
        if (t < kWSeg) x[t] = (t < nmax) ? v : 0.0;
    }
}

template <int kWTk>
struct WinShape {            // shared-memory layout of one tile of kWTk rows (in doubles)
    int rows, cols, pitch;   // right-hand side tile (row stride pitch, odd)
    int ncz;                 // staged z coefficients
    int a_size, q_size, c_size;   // regions A (rhs, then z rhs), Q (the tile of q), C (coefficients)
    __host__ __device__ WinShape(int Ky, int Kz) {
        rows = kWTk + 2 * Kz;
        cols = kWTj + 2 * Ky;
        pitch = cols | 1;
        ncz = kWTk + 2 * Kz;
        const int a1 = rows * pitch, a2 = rows * kWXp;
        a_size = ((a1 > a2 ? a1 : a2) + 1) & ~1;   // (the pairs behind it 16-byte aligned)
        q_size = kWTk * kWTj;
        c_size = 4 * cols + 2 * ncz + ncz;   // pairs (a, s) and (e, g) of y, (e, g) of z, a of z
    }
};

}  // namespace

// blockIdx.y = 0: v (solq2j + solq2k + walls), 1: w (solq3j + solq3k);
// blockIdx.x = tile (tj fastest).
// kWait: the body waits for the kernel before it, which writes rhs2/rhs3 (the
// spreading, or nl_rhs): the coefficients and the tile of q are under way then.
// kBlk: the forward recurrences in blocks (win_segment's kB).
template <int KM, int kWTk, bool kBlk, bool kWait>
__device__ __forceinline__ void helsolve_win_body(const Dev &d, const SubDev &sd, int ntj, int Ky, int Kz) {
    extern __shared__ __align__(16) double sm[];
    const WinShape<kWTk> sh(Ky, Kz);
    double *A = sm, *Q = sm + sh.a_size, *C = Q + sh.q_size;
    const int fld = blockIdx.y;
    const int tj = blockIdx.x % ntj, tk = blockIdx.x / ntj;
    const int j0 = 1 + tj * kWTj, k0 = 1 + tk * kWTk;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int kWarps = kWThreads / 32;
    const ScanSys sy = fld ? sd.sy3 : sd.sy2, sz = fld ? sd.sz3 : sd.sz2;
    const double *by = fld ? sd.by3 : sd.by2, *bz = fld ? sd.bz3 : sd.bz2;
    const double *rhs = fld ? d.rhs3 : d.rhs2;
    double *q = fld ? d.q3 : d.q2;
    const int ny = fld ? d.n2m : d.n2;   // y unknowns (j = 1..ny, line index j-1)
    const int nz = fld ? d.n3 : d.n3m;   // z unknowns (k = 1..nz, line index k-1)
    const int jlo = fld ? 1 : 2;          // columns with a right-hand side
    const int klo = fld ? 2 : 1;          // rows whose y lines are solved
    const int rows = sh.rows, cols = sh.cols;
    double *cas = C, *ceg = C + 2 * cols;                              // (a, normaliser), (e, g) of y by tile column
    double *zeg = C + 4 * cols, *za = zeg + 2 * sh.ncz;                // (e, g), a of z by tile row

    // 1. coefficients, the y row normalisers, the right-hand side tile
    //    (A[r * pitch + c] holds (j0 - Ky + c, k0 - Kz + r)) and the tile of q:
    //    all copies issued at once (cp.async); the forward y recurrence scales
    //    the right-hand side as it reads it
    for (int c = threadIdx.x; c < cols; c += kWThreads) {
        const int i = j0 - 1 - Ky + c, jc = i + 1;   // line index, column
        if (i >= 0 && i < ny) {
            cp8(cas + 2 * c, sy.a + i);
            cp8(ceg + 2 * c, sy.e + i);
            cp8(ceg + 2 * c + 1, sy.g + i);
        } else {
            cas[2 * c] = ceg[2 * c] = ceg[2 * c + 1] = 0.0;
        }
        if (jc >= jlo && jc <= d.n2m) cp8(cas + 2 * c + 1, by + jc);
        else cas[2 * c + 1] = 0.0;
    }
    for (int c = threadIdx.x; c < sh.ncz; c += kWThreads) {
        const int i = k0 - 1 - Kz + c;
        if (i >= 0 && i < nz) {
            cp8(za + c, sz.a + i);
            cp8(zeg + 2 * c, sz.e + i);
            cp8(zeg + 2 * c + 1, sz.g + i);
        } else {
            za[c] = zeg[2 * c] = zeg[2 * c + 1] = 0.0;
        }
    }
    const int j = j0 + lane;
    const bool jlive = (j >= jlo && j <= d.n2m);
    if (jlive)
        for (int r = w; r < kWTk && k0 + r <= d.n3m; r += kWarps) cp8(Q + r * kWTj + lane, q + fidx(d, j, k0 + r));
    if (kWait) FB_GRID_WAIT();
    {
        constexpr int kCC = 3;   // column chunks of 32 (cols <= 80)
        int jc[kCC];
        bool okc[kCC];
#pragma unroll
        for (int cc = 0; cc < kCC; ++cc) {
            const int c = lane + 32 * cc;
            jc[cc] = j0 - Ky + c;
            okc[cc] = (c < cols) && (jc[cc] >= jlo && jc[cc] <= d.n2m);
        }
        for (int r = w; r < rows; r += kWarps) {
            const int k = k0 - Kz + r;
            const bool kok = (k >= klo && k <= d.n3m);
#pragma unroll
            for (int cc = 0; cc < kCC; ++cc) {
                if (lane + 32 * cc >= cols) continue;
                double *dst = A + r * sh.pitch + lane + 32 * cc;
                if (kok && okc[cc]) cp8(dst, rhs + fidx(d, jc[cc], k));
                else *dst = 0.0;
            }
        }
    }
    cp_wait();
    __syncthreads();

    // 2. y solves: lanes = rows, one segment per warp task; the results go to A
    //    as the z right-hand side once every thread has read its inputs:
    //    A[r * kWXp + c] = f at (j0 + c, k0 - Kz + r), scaled by the z row normalisers
    constexpr int kSegs = kWTj / kWSeg;
    constexpr int kTasks = (kWTk + 2 * KM + 31) / 32 * kSegs;
    constexpr int kRounds = (kTasks + kWarps - 1) / kWarps;
    double xs[kRounds][kWSeg];
    const int ntask = (rows + 31) / 32 * kSegs;
#pragma unroll
    for (int it = 0; it < kRounds; ++it) {
        const int task = w + it * kWarps;
        if (task >= ntask) break;
        const int sg = task % kSegs, rr = min(task / kSegs * 32 + lane, rows - 1);
        const int c0 = Ky + sg * kWSeg;   // tile column of the segment's start
        const double *arow = A + rr * sh.pitch + c0;
        const double2 *as = reinterpret_cast<const double2 *>(cas) + c0;
        const double2 *eg = reinterpret_cast<const double2 *>(ceg) + c0;
        const int s0 = j0 - 1 + sg * kWSeg;   // line index of the segment's start
        win_segment<KM, kBlk ? 24 : 0>(
            [&](int u, double v) {
                const double2 c = as[u];
                return fma(c.x, v, arow[u] * c.y);
            },
            [&](int u) { return eg[u]; }, Ky, -s0, ny - s0, -sg * kWSeg, xs[it]);
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kRounds; ++it) {
        const int task = w + it * kWarps;
        if (task >= ntask) break;
        const int sg = task % kSegs, r = task / kSegs * 32 + lane, k = k0 - Kz + r;
        if (r >= rows) continue;
        const bool live = k >= klo && k <= d.n3m;
        const double bzk = (k >= 1 && k <= nz) ? __ldg(bz + k) : 0.0;
        double *arow = A + r * kWXp + sg * kWSeg;
#pragma unroll
        for (int t = 0; t < kWSeg; ++t) arow[t] = live ? xs[it][t] * bzk : 0.0;
    }
    // the inflow/outflow terms of rows k = 1 and nz (solve_fluid.F90:208-209,
    // 266-275), where the tile or its halo holds them; one lane per column
    const int rs = 1 - (k0 - Kz), rn = nz - (k0 - Kz);   // their tile rows
    const bool ends = (rs >= 0 && rs < rows) || (rn >= 0 && rn < rows);
    if (ends) {
        const int jj = min(max(j, 1), d.n2m);
        double fs = 0.0, fn = 0.0;
        if (w == 0) {
            fs = fld ? d.dqb3s[jj] : d.dqb2s[jj];
            fn = fld ? d.dqb3n[jj] : d.dqb2n[jj];
        }
        __syncthreads();
        if (w == 0) {
            if (rs >= 0 && rs < rows) {
                double &f = A[rs * kWXp + lane];
                f = fld ? fs : f + fs * sd.ugkks;
            }
            if (rn >= 0 && rn < rows) {
                double &f = A[rn * kWXp + lane];
                f = fld ? fn : f + fn * sd.ugkkn;
            }
        }
    }
    __syncthreads();

    // 3. z solves: lanes = columns, warps = segments of rows; q += result
    for (int sg = w; sg < kWTk / kWSeg; sg += kWarps) {
        const int s0 = k0 - 1 + sg * kWSeg;   // line index of the segment's start
        if (s0 >= d.n3m) continue;
        const int c0 = Kz + sg * kWSeg;       // its tile row
        const double *acol = A + c0 * kWXp + lane;
        const double *a = za + c0;
        const double2 *eg = reinterpret_cast<const double2 *>(zeg) + c0;
        double x[kWSeg];
        win_segment<KM, kBlk ? 16 : 0>([&](int u, double v) { return fma(a[u], v, acol[u * kWXp]); },
                                       [&](int u) { return eg[u]; }, Kz, -s0, nz - s0, 0, x);
        if (jlive) {
            const double *qc = Q + sg * kWSeg * kWTj + lane;
#pragma unroll
            for (int t = 0; t < kWSeg; ++t)
                if (s0 + 1 + t <= d.n3m) q[fidx(d, j, s0 + 1 + t)] = qc[t * kWTj] + x[t];
        }
    }
    if (w != kWarps - 1) return;   // the last warp, without a segment, does the edges
    const bool top = k0 + kWTk > d.n3m;
    if (fld == 1 && jlive && top) Fv(q, j, d.n3) = Fv(q, j, d.n3) + d.dqb3n[j];
    if (fld == 0) {   // helsolve.F90:35-36: wall values of v, each tile its rows
        const int ka = (tk == 0) ? 0 : k0, kb = top ? d.n3 : k0 + kWTk - 1;
        if (tj == 0)
            for (int k = ka + lane; k <= kb; k += 32) Fv(d.q2, 1, k) = 0.0;
        if (tj == ntj - 1)
            for (int k = ka + lane; k <= kb; k += 32) Fv(d.q2, d.n2, k) = 0.0;
    }
}

// resident blocks per SM that the registers of the window's segments allow (10 rows:
// the four blocks of 8 with 80 registers; a 20-case batch takes 93.1 ms per 50
// steps so, 94.4 with its 9 and 10 row windows in the form of 12)
constexpr int win_blocks(int KM) { return KM <= 10 ? 4 : KM <= 16 ? 3 : 2; }

template <int KM, int kWTk, bool kBlk>
__global__ void __launch_bounds__(kWThreads, win_blocks(KM)) k_helsolve_win(Dev d, SubDev sd, int ntj, int Ky, int Kz) {
    helsolve_win_body<KM, kWTk, kBlk, true>(d, sd, ntj, Ky, Kz);
}

// grouped forms (blockIdx.z = case; substep n 0-based): each case keeps its
// own windows, the group's shared memory fits the largest
template <int KM, int kWTk, bool kBlk>
__global__ void __launch_bounds__(kWThreads, win_blocks(KM)) kg_helsolve_win(const GroupCase *__restrict__ g, int n, int ntj) {
    __shared__ Dev d;
    __shared__ SubDev s;
    if (!stage_case(g, &d, &s, n)) return;
    helsolve_win_body<KM, kWTk, kBlk, false>(d, s, ntj, s.win_y, s.win_z);
}


// ---------------------------------------------------------------- dispatch

namespace {

// line buffers; for the Poisson modes also the pivot rows and the two y
// off-diagonal arrays
size_t ylines_smem(const Dev &d, int kind) {
    size_t n = static_cast<size_t>(kYLines) * (d.n2 + 1);
    if (kind == 2) n += static_cast<size_t>(kYLines) * (d.n2m + 1) + 2 * static_cast<size_t>(d.n2m + 2);
    return n * sizeof(double);
}

template <int kKind>
void ylaunch(const Dev &d, const SubDev *sd, cudaStream_t st) {
    constexpr int W = (kKind == 2) ? kYPoissonWarps : kYWarps;
    const int lines = (kKind == 2) ? d.n3m : d.n3m + (d.n3m - 1);
    const int blocks = (lines + kYLines - 1) / kYLines;
    const int m = ((d.n2 + 32 * W - 1) / (32 * W)) | 1;
    const size_t smem = ylines_smem(d, kKind);
    const ScanSys z{nullptr, nullptr, nullptr};
    const ScanSys s2 = sd ? sd->sy2 : z, s3 = sd ? sd->sy3 : z;
    const double *b2 = sd ? sd->by2 : nullptr, *b3 = sd ? sd->by3 : nullptr;
    const int threads = kYLines * W * 32;
    if (m <= 9) pdl(k_ylines<9, kKind, W>, dim3(blocks), dim3(threads), smem, st, d, s2, b2, s3, b3);
    else if (m <= 17) pdl(k_ylines<17, kKind, W>, dim3(blocks), dim3(threads), smem, st, d, s2, b2, s3, b3);
    else pdl(k_ylines<33, kKind, W>, dim3(blocks), dim3(threads), smem, st, d, s2, b2, s3, b3);
}

void zlaunch(const Dev &d, const SubDev &sd, cudaStream_t st) {
    const int nb2 = (d.n2m + kZLines - 1) / kZLines;
    const int blocks = 2 * nb2;
    const int n = d.n3;  // the longer of the two systems sets the chunking
    constexpr int kChunksPerWarp = 32 / kZLines;
    int warps = (n + kChunksPerWarp * 16 - 1) / (kChunksPerWarp * 16);
    if (warps <= 16) {
        pdl(k_zlines<16, 512>, dim3(blocks), dim3(warps * 32), 0, st, d, sd, nb2);
        return;
    }
    warps = (n + kChunksPerWarp * 32 - 1) / (kChunksPerWarp * 32);
    if (warps <= 10) {
        pdl(k_zlines<32, 320>, dim3(blocks), dim3(warps * 32), 0, st, d, sd, nb2);
        return;
    }
    warps = (n + kChunksPerWarp * 64 - 1) / (kChunksPerWarp * 64);
    pdl(k_zlines<64, 256>, dim3(blocks), dim3(warps * 32), 0, st, d, sd, nb2);
}

template <class K>
cudaError_t allow_smem(K kern) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}

}  // namespace

// shared memory of the mode solves: the 227 KB opt-in less the static arrays
// (the grouped kernel's Dev)
constexpr int kYmSmem = 225 * 1024;

cudaError_t scan_configure() {
    cudaError_t e;
#define AL(K)                                  \
    if ((e = allow_smem(K)) != cudaSuccess) return e;
    AL((k_ylines<9, 0>)) AL((k_ylines<17, 0>)) AL((k_ylines<33, 0>))
#define WN(KM)                                                                                  \
    AL((k_helsolve_win<KM, 32, false>)) AL((k_helsolve_win<KM, 64, false>))                     \
    AL((k_helsolve_win<KM, 32, true>)) AL((k_helsolve_win<KM, 64, true>))                       \
    AL((kg_helsolve_win<KM, 32, false>)) AL((kg_helsolve_win<KM, 64, false>))                   \
    AL((kg_helsolve_win<KM, 32, true>)) AL((kg_helsolve_win<KM, 64, true>))
    WN(8) WN(10) WN(12) WN(16) WN(kWinMax)
#undef WN
#define YM(M, W)                                                                                                \
    if ((e = cudaFuncSetAttribute(k_ymodes<M, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, kYmSmem)) !=      \
            cudaSuccess ||                                                                                      \
        (e = cudaFuncSetAttribute(kg_ymodes<M, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, kYmSmem)) !=     \
            cudaSuccess)                                                                                        \
        return e;
    YM(9, 1) YM(17, 1) YM(25, 1) YM(0, 1) YM(17, 2)
#undef YM
#undef AL
    return cudaSuccess;
}

namespace {
// calls go with the smallest instantiated warm-up length that covers the window
template <class F>
void win_form(int km, F go) {
    using std::integral_constant;
    if (km <= 8) go(integral_constant<int, 8>{});
    else if (km <= 10) go(integral_constant<int, 10>{});
    else if (km <= 12) go(integral_constant<int, 12>{});
    else if (km <= 16) go(integral_constant<int, 16>{});
    else go(integral_constant<int, kWinMax>{});
}

template <int TK>
void win_launch(const Dev &d, const SubDev &s, cudaStream_t st, bool blocks) {
    const int ntj = (d.n2m + kWTj - 1) / kWTj, ntk = (d.n3m + TK - 1) / TK;
    const WinShape<TK> sh(s.win_y, s.win_z);
    const size_t smem = static_cast<size_t>(sh.a_size + sh.q_size + sh.c_size) * sizeof(double);
    win_form(std::max(s.win_y, s.win_z), [&](auto KM) {
        pdl(blocks ? k_helsolve_win<KM, TK, true> : k_helsolve_win<KM, TK, false>, dim3(ntj * ntk, 2), dim3(kWThreads),
            smem, st, d, s, ntj, s.win_y, s.win_z);
    });
}
}  // namespace

void launch_win_helsolve(const Dev &d, const SubDev &s, cudaStream_t st, bool blocks) {
    if (s.win_tk == 32) win_launch<32>(d, s, st, blocks);
    else win_launch<64>(d, s, st, blocks);
}

void launch_scan_helsolve(const Dev &d, const SubDev &s, cudaStream_t st) {
    ylaunch<0>(d, &s, st);
    zlaunch(d, s, st);
}

namespace {
// modes per block and shared bytes of k_ymodes: as many as fit
int ymodes_shape(const Dev &d, size_t *smem) {
    const size_t shared = 2 * static_cast<size_t>(d.n2m + 2) * sizeof(double);
    const size_t per = 2 * static_cast<size_t>(d.n2m + 1) * sizeof(double);
    const int nw = std::max(1, static_cast<int>(std::min<size_t>(kYmModes, (kYmSmem - shared) / per)));
    *smem = shared + per * static_cast<size_t>(nw);
    return nw;
}

// calls go(M, W) as integral constants: lane chunks of M values (0: in shared
// memory), W warps per mode
template <class F>
void ymodes_form(const Dev &d, bool one_warp, F go) {
    using std::integral_constant;
    const int m = ((d.n2m + 31) / 32) | 1;   // one warp's lane chunk
    if (m <= 9) go(integral_constant<int, 9>{}, integral_constant<int, 1>{});
    else if (m <= 17) go(integral_constant<int, 17>{}, integral_constant<int, 1>{});
    else if (m <= 25) go(integral_constant<int, 25>{}, integral_constant<int, 1>{});
    else if (d.n2m <= 64 * 17 && !one_warp) go(integral_constant<int, 17>{}, integral_constant<int, 2>{});
    else go(integral_constant<int, 0>{}, integral_constant<int, 1>{});
}
}  // namespace

void launch_scan_poisson(const Dev &d, cudaStream_t st, double *rmax, bool one_warp) {
    ymodes_form(d, one_warp, [&](auto M, auto W) {
        size_t smem = 0;
        const int nw = ymodes_shape(d, &smem);
        pdl(k_ymodes<M, W>, dim3((d.n3m + nw - 1) / nw), dim3(32 * W * nw), smem, st, d, nw, rmax);
    });
}

namespace {
template <int TK>
void gwin_launch(const Group &g, int n, cudaStream_t st, bool blocks) {
    const Dev &d = g.rep;
    const int ntj = (d.n2m + kWTj - 1) / kWTj, ntk = (d.n3m + TK - 1) / TK;
    const int ky = g.win_ky[n], kz = g.win_kz[n];
    const WinShape<TK> sh(ky, kz);   // sizes grow with the windows: fits every case
    const size_t smem = static_cast<size_t>(sh.a_size + sh.q_size + sh.c_size) * sizeof(double);
    win_form(std::max(ky, kz), [&](auto KM) {
        pdl(blocks ? kg_helsolve_win<KM, TK, true> : kg_helsolve_win<KM, TK, false>, dim3(ntj * ntk, 2, g.n),
            dim3(kWThreads), smem, st, g.cases, n, ntj);
    });
}
}  // namespace

void glaunch_win_helsolve(const Group &g, int n, cudaStream_t st, bool blocks) {
    if (g.win_tk == 32) gwin_launch<32>(g, n, st, blocks);
    else gwin_launch<64>(g, n, st, blocks);
}

void glaunch_scan_poisson(const Group &g, cudaStream_t st, bool one_warp) {
    const Dev &d = g.rep;
    ymodes_form(d, one_warp, [&](auto M, auto W) {
        size_t smem = 0;
        const int nw = ymodes_shape(d, &smem);
        pdl(kg_ymodes<M, W>, dim3((d.n3m + nw - 1) / nw, 1, g.n), dim3(32 * W * nw), smem, st, g.cases, nw);
    });
}

}  // namespace fb
