// CUDA kernels of the FRiBoIS2D fluid time step (sm_100a, FP64).
//
// This translation unit is compiled with -fmad=false: every expression keeps
// the reference's left-to-right evaluation without fused multiply-adds, so
// the stencil stages reproduce the CPU restatement bit for bit.  Each kernel
// cites the reference routine it implements.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include <cudaTypedefs.h>

#include "device.cuh"
#include "kernels.h"
#include "pdl.h"
#include "tma.cuh"
#include "../../include/fribois2d.h"

namespace fb {

#define Fv(a, j, k) (a)[fidx(d, (j), (k))]

// ------------------------------------------------------------ helpers

__device__ __forceinline__ void raise_status(const Dev &d, int code) {
    atomicCAS(d.status, 0, code);
}

// indic.F90:276-303 as arithmetic (no dependent index loads)
__device__ __forceinline__ int jmv_(int jc) { return jc == 1 ? 1 : jc - 1; }
__device__ __forceinline__ int jpv_(const Dev &d, int jc) { return jc >= d.n2m ? jc : jc + 1; }
__device__ __forceinline__ int kmv_(int kc) { return kc == 1 ? 1 : kc - 1; }
__device__ __forceinline__ int kpv_(const Dev &d, int kc) { return kc == d.n3m ? kc : kc + 1; }

template <bool kMax>
__device__ __forceinline__ double warp_reduce(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, v, o);
        v = kMax ? fmax(v, x) : v + x;
    }
    return v;
}

// block reduction with shuffles; sh holds 32 doubles; result in every thread
template <bool kMax>
__device__ double block_reduce_fast(double v, double *sh) {
    const int t = threadIdx.x + threadIdx.y * blockDim.x;
    const int nw = (blockDim.x * blockDim.y + 31) >> 5;
    v = warp_reduce<kMax>(v);
    if ((t & 31) == 0) sh[t >> 5] = v;
    __syncthreads();
    double r = (t < nw) ? sh[t] : (kMax ? -INFINITY : 0.0);
    if (t < 32) r = warp_reduce<kMax>(r);
    if (t == 0) sh[0] = r;
    __syncthreads();
    r = sh[0];
    __syncthreads();
    return r;
}

// block_reduce_fast<false> of N values at once (the same shuffle tree for
// each, so the same sums), three barriers in all; sh holds 32 N doubles
template <int N>
__device__ void block_sum_n(double (&v)[N], double *sh) {
    const int t = threadIdx.x + threadIdx.y * blockDim.x;
    const int nw = (blockDim.x * blockDim.y + 31) >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = warp_reduce<false>(v[i]);
    if ((t & 31) == 0)
#pragma unroll
        for (int i = 0; i < N; ++i) sh[32 * i + (t >> 5)] = v[i];
    __syncthreads();
    if (t < 32) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            double r = (t < nw) ? sh[32 * i + t] : 0.0;
            r = warp_reduce<false>(r);
            v[i] = r;
        }
    }
    if (t == 0)   // (lane 0 read slot 32 i itself before; the other lanes read other slots)
#pragma unroll
        for (int i = 0; i < N; ++i) sh[32 * i] = v[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = sh[32 * i];
    __syncthreads();
}

// ------------------------------------------------------------ cfl

// cfl.F90 (fluid_tsch.F90:211-258) and the fixed-dt check fluid_tsch.F90:49-55.
// Both reductions (max for the CFL number, sum for the mean w) share one
// last-block pass so that a single block finalises them.
__device__ __forceinline__ void cfl_body(const Dev &d) {
    __shared__ double sh[32];
    __shared__ bool last;
    const int t = threadIdx.x, nt = blockDim.x;
    const int b = blockIdx.x, nb = gridDim.x;
    double qcf = 1.0e-8, q3a = 0.0;
    // rows k over the blocks, columns j over the threads (no index division);
    // kR rows (k, k + nb, ...) by kU columns of a thread per pass, their loads
    // all issued before the first use; a row's terms are summed before the
    // next row's (for rows of up to kU x blockDim columns, the per-thread
    // order of the sum is that of one value at a time)
    constexpr int kU = 4, kR = 2;
    for (int k0 = b + 1; k0 <= d.n3m; k0 += kR * nb) {
        double udx3[kR], dz[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const int k = min(k0 + r * nb, d.n3m);
            udx3[r] = d.udx3m[k];
            dz[r] = d.zz[k + 1] - d.zz[k];
        }
        for (int j0 = t + 1; j0 <= d.n2m; j0 += kU * nt) {
            double a2[kR][kU], b2[kR][kU], a3[kR][kU], b3[kR][kU], u2[kU], rj[kU], rjp[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int j = min(j0 + u * nt, d.n2m), jp = j + 1;
                u2[u] = d.udx2m[j];
                rj[u] = d.rc[j];
                rjp[u] = d.rc[jp];
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    const int k = min(k0 + r * nb, d.n3m);
                    a2[r][u] = Fv(d.q2, j, k);
                    b2[r][u] = Fv(d.q2, jp, k);
                    a3[r][u] = Fv(d.q3, j, k);
                    b3[r][u] = Fv(d.q3, j, k + 1);
                }
            }
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                if (k0 + r * nb > d.n3m) break;
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    if (j0 + u * nt > d.n2m) break;
                    const double q = (fabs((a2[r][u] + b2[r][u]) * 0.5 * u2[u]) +
                                      fabs((a3[r][u] + b3[r][u]) * 0.5 * udx3[r]));
                    // fmax drops a NaN: a non-finite velocity turns into +inf, which
                    // every later fmax keeps, so the CFL test below catches it
                    qcf = fmax(qcf, (q == q) ? q : INFINITY);
                    q3a = q3a + a3[r][u] * dz[r] * (rjp[u] - rj[u]);
                }
            }
        }
    }
    const double pm = block_reduce_fast<true>(qcf, sh);
    const double ps = block_reduce_fast<false>(q3a, sh);
    double *rm = d.red, *rs = d.red + kRedSlot;
    if (t == 0) {
        rm[b] = pm;
        rs[b] = ps;
        __threadfence();
        last = (atomicAdd(d.count, 1u) == static_cast<unsigned>(nb - 1));
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double am = 1.0e-8, as = 0.0;
    for (int i = t; i < nb; i += nt) {
        am = fmax(am, __ldcg(rm + i));
        as = as + __ldcg(rs + i);
    }
    am = block_reduce_fast<true>(am, sh);
    as = block_reduce_fast<false>(as, sh);
    if (t == 0) {
        d.count[0] = 0u;
        const double cflm = am * d.dt;
        d.scal[S_CFLM] = cflm;
        d.scal[S_CFLRAW] = am;
        d.scal[S_Q3AVG] = as / (d.rext2 * d.alx3);
        // fixed dt: the stability check of fluid_tsch.F90:49-55; variable dt
        // is set from am on the host (fluid_tsch.F90:34-48)
        if (!d.vardt && !(cflm <= d.cfllim)) raise_status(d, FB_ERR_CFL);
    }
}

__global__ void __launch_bounds__(256) k_cfl(Dev d) {
    FB_GRID_WAIT();
    cfl_body(d);
}

// the scalars and the status word as they are ahead of a step, kept beside them (a
// variable-dt step may be taken back behind its marker set-up).  A launch of its own:
// a copy to the host in its place cost 12 us per step of 180.
__global__ void k_note(double *scal) {
    FB_GRID_WAIT();
    unsigned long long *s = reinterpret_cast<unsigned long long *>(scal);
    if (threadIdx.x <= kScalStatus) s[kScalNoted + threadIdx.x] = s[threadIdx.x];
}

// ------------------------------------------------------------ boundaries

// iobcs.F90:5-77 (boucdq): radiative outflow increments + mass-flux correction;
// one block.  In the fused step it is a block of nl_rhs's launch: nl_rhs reads
// the boundary values qb*, not their increments, which only helsolve needs.
__device__ __forceinline__ void boucdq_body(const Dev &d, double ga, double ro) {
    __shared__ double sh[32];
    const int n3 = d.n3, n3m = d.n3m;
    const int t = threadIdx.x + blockDim.x * threadIdx.y, nt = blockDim.x * blockDim.y;
    double qout = 0.0;
    for (int j = t + 1; j <= d.n2; j += nt) {
        d.dqb2s[j] = 0.0;
        d.dqb3s[j] = 0.0;
    }
    for (int j = t + 1; j <= d.n2m; j += nt) {
        double dq2x2 = (d.qb2n[j] - Fv(d.q2, j, n3m)) * 2.0 * d.udx3c[n3];
        double dqb2n = -d.dt * (ga * dq2x2 + ro * d.dq2x2o[j]) * d.cou;
        double dq3x2 = (d.qb3n[j] - Fv(d.q3, j, n3m)) * d.udx3c[n3];
        double dqb3n = -d.dt * (ga * dq3x2 + ro * d.dq3x2o[j]) * d.cou;
        d.dqb2n[j] = dqb2n;
        d.dqb3n[j] = dqb3n;
        d.dq2x2o[j] = dq2x2;
        d.dq3x2o[j] = dq3x2;
        qout = qout + dqb3n * (d.g2rm[j] / d.dx2);
    }
    double q = block_reduce_fast<false>(qout, sh);
    const double cor = (0.0 - q) / d.area_out;
    __syncthreads();
    for (int j = t + 1; j <= d.n2m; j += nt) d.dqb3n[j] = d.dqb3n[j] + cor;
}

// pr_submean (updvp.F90:336) of a step's three pressure means, in order, for
// the entries of pr that updvp never rewrites and no stencil of the step reads
// (j = n2, k = 0, k = n3); one block.  (The probes of the loads read row k = 0
// ahead of it and subtract the three means themselves.)
__device__ __forceinline__ void edge_means_body(const Dev &d) {
    const int t = threadIdx.x + blockDim.x * threadIdx.y, nt = blockDim.x * blockDim.y;
    const double m1 = d.scal[S_PRAVG1], m2 = d.scal[S_PRAVG2], m3 = d.scal[S_PRAVG];
    const int n = (d.n3 + 1) + 2 * d.n2m;   // column j = n2, then rows k = 0 and n3
    constexpr int kU = 4;
    for (int i0 = t; i0 < n; i0 += kU * nt) {
        double *p[kU], v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {   // every load before the first store
            const int i = min(i0 + u * nt, n - 1), e = i - (d.n3 + 1);
            p[u] = d.pr + (e < 0 ? fidx(d, d.n2, i) : e < d.n2m ? fidx(d, e + 1, 0) : fidx(d, e - d.n2m + 1, d.n3));
            v[u] = *p[u];
        }
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if (i0 + u * nt < n) *p[u] = ((v[u] - m1) - m2) - m3;
    }
}

__global__ void __launch_bounds__(1024) k_boucdq(Dev d, double ga, double ro) {
    FB_GRID_WAIT();
    boucdq_body(d, ga, ro);
}

// ------------------------------------------------------------ explicit terms

// HDNL.F90:5-171 (hdnl2, hdnl3) fused with INVTR.F90:4-280 (invtr2, invtr3).
// The convective terms stay in registers; ru2/ru3 receive them as the
// reference's invtr does (ru2 = dph, ru3 = qcap).  q2f/q3f are not stored:
// the forcing stage forms q + rhs at the few support nodes it reads.
// Tiles of kNlJ x kNlK cells: a block holds q2, q3 and pr of a tile plus a
// one-cell halo, and the tile's j and k coefficients, in shared memory, so
// each cell's stencil reads shared memory instead of issuing ~24 global
// loads.  Blocks are persistent over tiles with two buffers: the copies of
// the next tile (cp.async) and its ru2/ru3 (registers) are in flight while
// the current tile is computed.  Thread (tx, ty) of the 32 x 8 block computes
// the cells j = j0 + tx, k = k0 + 4 ty + i, i = 0..3 of a tile (consecutive
// rows share their stencil loads).
constexpr int kNlJ = 32, kNlK = 32, kNlS = kNlJ + 3;  // odd row stride
constexpr int kNlBlocksPerSM = 2;
struct NlTile {
    double q2[kNlK + 2][kNlS], q3[kNlK + 2][kNlS], pr[kNlK + 2][kNlS];  // rows k0-1.., cols j0-1..
    double udx3m[kNlK], ap3sk[kNlK], ac3sk[kNlK], am3sk[kNlK];           // k coefficients, rows k0..
    double udx3c[kNlK], ap3ck[kNlK], ac3ck[kNlK], am3ck[kNlK];
    double udx2c[kNlJ], am2j[kNlJ], ac2j[kNlJ], ap2j[kNlJ];              // j coefficients, columns j0..
    double udx2m[kNlJ], am3j[kNlJ], ac3j[kNlJ], ap3j[kNlJ];
};
constexpr size_t kNlSmem = 2 * sizeof(NlTile);

// The TMA-staged tile: one box per field of kNlTH rows (k0 - 1 .. k0 + 32) by
// kNlTW columns.  A box must start on a 16-byte boundary, so it starts one
// column left of the halo: column c holds j = j0 - 2 + c, and the stencil
// reads columns 1 .. 34.  Each field array starts on a 128-byte boundary.
constexpr int kNlTW = kNlJ + 4, kNlTH = kNlK + 2;
struct alignas(128) NlTileT {
    alignas(128) double q2[kNlTH][kNlTW];
    alignas(128) double q3[kNlTH][kNlTW];
    alignas(128) double pr[kNlTH][kNlTW];
    double udx3m[kNlK], ap3sk[kNlK], ac3sk[kNlK], am3sk[kNlK];
    double udx3c[kNlK], ap3ck[kNlK], ac3ck[kNlK], am3ck[kNlK];
    double udx2c[kNlJ], am2j[kNlJ], ac2j[kNlJ], ap2j[kNlJ];
    double udx2m[kNlJ], am3j[kNlJ], ac3j[kNlJ], ap3j[kNlJ];
};
constexpr uint32_t kNlBoxBytes = kNlTH * kNlTW * 8;
static_assert(kNlBoxBytes % 16 == 0 && (kNlTW * 8) % 16 == 0, "TMA box rows in 16-byte units");
// two tiles, their two mbarriers, and the slack to align the tiles to 128 bytes
constexpr size_t kNlSmemT = 2 * sizeof(NlTileT) + 128 + 128;

// ru2v, ru3v: ru2/ru3 at the cell, read before any cell of the thread is
// stored (0 when ro = 0)
// kC0: the tile column of j = j0 (1 for the cp.async tile, 2 for the TMA tile)
template <int kC0, class Tile>
__device__ __forceinline__ void nl_cell(const Dev &d, const Tile &t, int j0, int k0, int jc, int kc, double al,
                                        double ga, double ro, double ru2v, double ru3v) {
#define S2(j, k) t.q2[(k) - k0 + 1][(j) - j0 + kC0]
#define S3(j, k) t.q3[(k) - k0 + 1][(j) - j0 + kC0]
#define SP(j, k) t.pr[(k) - k0 + 1][(j) - j0 + kC0]
    const int n2m = d.n2m, n3m = d.n3m;
    const double dt = d.dt, alre = al / d.ren;

    // ---- v momentum at (jc, kc), jc = 2..n2m
    if (jc >= 2) {
        const int jm = jc - 1, jp = jc + 1;
        double h22 = ((S2(jp, kc) + S2(jc, kc)) * (S2(jp, kc) + S2(jc, kc)) -
                      (S2(jm, kc) + S2(jc, kc)) * (S2(jm, kc) + S2(jc, kc))) *
                     t.udx2c[jc - j0] * 0.25;
        double dph = -h22;
        const int jmv = jc - 1;  // jmv(jc) for jc >= 2
        if (kc >= 2 && kc <= n3m - 1) {
            const int kmm = kc - 1, kpp = kc + 1, kp = kc + 1;  // kmv, kpv in the interior
            double h23 = ((S3(jc, kp) + S3(jmv, kp)) * (S2(jc, kpp) + S2(jc, kc)) -
                          (S3(jc, kc) + S3(jmv, kc)) * (S2(jc, kc) + S2(jc, kmm))) *
                         t.udx3m[kc - k0] * 0.25;
            dph = dph - h23;
        } else if (kc == n3m) {
            const int kmm = kc - 1;
            double h23 = (d.qb2n[jc] * (d.qb3n[jc] + d.qb3n[jmv]) -
                          (S3(jc, kc) + S3(jmv, kc)) * (S2(jc, kc) + S2(jc, kmm)) * 0.5) *
                         t.udx3m[kc - k0] * 0.5;
            dph = dph - h23;
        }
        if (kc == 1) {
            const int kp = kc + 1;
            double h23 = ((S3(jc, kp) + S3(jmv, kp)) * (S2(jc, kc) + S2(jc, kp)) * 0.5 -
                          d.qb2s[jc] * (d.qb3s[jc] + d.qb3s[jmv])) *
                         t.udx3m[kc - k0] * 0.5;
            dph = dph - h23;
        }
        const double ammj = t.am2j[jc - j0], accj = t.ac2j[jc - j0], appj = t.ap2j[jc - j0];
        const double d22q2 = S2(jp, kc) * appj + S2(jc, kc) * accj + S2(jm, kc) * ammj;
        double d33q2, dpx22;
        if (kc >= 2 && kc <= n3m - 1) {
            const int km = kc - 1, kp = kc + 1;
            d33q2 = S2(jc, kp) * t.ap3sk[kc - k0] + S2(jc, kc) * t.ac3sk[kc - k0] + S2(jc, km) * t.am3sk[kc - k0];
            const double udx2 = al * t.udx2c[jc - j0];
            dpx22 = (SP(jc, kc) - SP(jm, kc)) * udx2;
        } else if (kc == 1) {
            const int kp = kc + 1;
            const double codea = d.dx3q / (d.g3rc[kp] * d.g3rm[kc]);
            const double codeb = d.dx3q / (d.g3rc[kc] * d.g3rm[kc]);
            d33q2 = ((S2(jc, kp) - S2(jc, kc)) * codea - (S2(jc, kc) - d.qb2s[jc]) * codeb * 2.0);
            dpx22 = (SP(jc, kc) - SP(jm, kc)) * t.udx2c[jc - j0] * al;
        } else {
            const int km = kc - 1, kp = kc + 1;
            const double codea = d.dx3q / (d.g3rc[kp] * d.g3rm[kc]);
            const double codeb = d.dx3q / (d.g3rc[kc] * d.g3rm[kc]);
            d33q2 = ((d.qb2n[jc] - S2(jc, kc)) * codea * 2.0 - (S2(jc, kc) - S2(jc, km)) * codeb);
            dpx22 = (SP(jc, kc) - SP(jm, kc)) * t.udx2c[jc - j0] * al;
        }
        const double dcq2 = d22q2 + d33q2;
        const size_t i = fidx(d, jc, kc);
        // the first RK3 substep has ro = 0: ru2 is not read (one field pass less)
        const double ru = ru2v;
        // global stores (st.global): the compiler then knows they do not
        // alias the shared-memory tile and reuses the tile loads across the
        // thread's consecutive cells
        __stcg(d.rhs2 + i, (ga * dph + ro * ru + alre * dcq2 - dpx22) * dt);
        __stcg(d.ru2 + i, dph);
    }

    // ---- w momentum at (jc, kc), kc = 2..n3m
    if (kc >= 2) {
        double qcap = 0.0;  // hdnl3 never writes kc = n3m (HDNL.F90:143)
        if (kc <= n3m - 1) {
            const int kmm = kc - 1, km = kc - 1, kp = kc + 1;
            const int jmm = jmv_(jc), jpp = jpv_(d, jc), jp = jc + 1;
            double h32 = (((S2(jp, kc) + S2(jp, km)) * (S3(jpp, kc) + S3(jc, kc))) -
                          ((S2(jc, kc) + S2(jc, km)) * (S3(jc, kc) + S3(jmm, kc)))) *
                         t.udx2m[jc - j0] * 0.25;
            double h33 = ((S3(jc, kp) + S3(jc, kc)) * (S3(jc, kp) + S3(jc, kc)) -
                          (S3(jc, kc) + S3(jc, kmm)) * (S3(jc, kc) + S3(jc, kmm))) *
                         t.udx3c[kc - k0] * 0.25;
            qcap = -(h32 + h33);
        }
        const int km = kc - 1, kp = kc + 1;
        const double udx3 = al * t.udx3c[kc - k0];
        const double ammj = t.am3j[jc - j0], accj = t.ac3j[jc - j0], appj = t.ap3j[jc - j0];
        double dq32;
        if (jc == 1) {
            dq32 = S3(jc + 1, kc) * appj + S3(jc, kc) * accj + d.q3lw * ammj;
        } else if (jc == n2m) {
            dq32 = d.q3uw * appj + S3(jc, kc) * accj + S3(jc - 1, kc) * ammj;
        } else {
            dq32 = S3(jpv_(d, jc), kc) * appj + S3(jc, kc) * accj + S3(jmv_(jc), kc) * ammj;
        }
        const double dq33 = S3(jc, kp) * t.ap3ck[kc - k0] + S3(jc, kc) * t.ac3ck[kc - k0] + S3(jc, km) * t.am3ck[kc - k0];
        const double dcq3 = dq32 + dq33;
        const double dpx33 = (SP(jc, kc) - SP(jc, km)) * udx3;
        const size_t i = fidx(d, jc, kc);
        const double ru = ru3v;
        __stcg(d.rhs3 + i, (ga * qcap + ro * ru + alre * dcq3 - dpx33) * dt);
        __stcg(d.ru3 + i, qcap);
    }
}
#undef S2
#undef S3
#undef SP

// cfl.F90 (fluid_tsch.F90:211-258) for one cell of a staged tile: the CFL sum
// into mx and w times the cell's area (dz x dy) into sm, as cfl_body forms them
template <int kC0, class Tile>
__device__ __forceinline__ void cfl_cell(const Tile &t, int cj, int ck, double dz, double dy, double &mx, double &sm) {
    const double a2 = t.q2[ck + 1][cj + kC0], b2 = t.q2[ck + 1][cj + 1 + kC0];
    const double a3 = t.q3[ck + 1][cj + kC0], b3 = t.q3[ck + 2][cj + kC0];
    const double q = fabs((a2 + b2) * 0.5 * t.udx2m[cj]) + fabs((a3 + b3) * 0.5 * t.udx3m[ck]);
    mx = fmax(mx, (q == q) ? q : INFINITY);   // a NaN velocity reads as +inf
    sm = sm + a3 * dz * dy;
}

// the block partials of nl_rhs's CFL number and mean w, combined by the last
// of the nb tile blocks into S_CFLNEXT and S_Q3NEXT (divg of the substep makes
// them the step's).  The partials lie in updvp's reduction slot, past its own.
__device__ __forceinline__ void cfl_finish(const Dev &d, double mx, double sm, int nb) {
    __shared__ double sh[32];
    __shared__ bool last;
    const int t = threadIdx.x + blockDim.x * threadIdx.y, nt = blockDim.x * blockDim.y;
    double *rm = d.red + 2 * static_cast<size_t>(kRedSlot) + kRedSlot / 2, *rs = rm + kRedSlot / 4;
    mx = block_reduce_fast<true>(mx, sh);
    sm = block_reduce_fast<false>(sm, sh);
    if (t == 0) {
        rm[blockIdx.x] = mx;
        rs[blockIdx.x] = sm;
        __threadfence();
        last = (atomicAdd(d.count, 1u) == static_cast<unsigned>(nb - 1));
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    mx = 1.0e-8;
    sm = 0.0;
    for (int i = t; i < nb; i += nt) {
        mx = fmax(mx, __ldcg(rm + i));
        sm = sm + __ldcg(rs + i);
    }
    mx = block_reduce_fast<true>(mx, sh);
    sm = block_reduce_fast<false>(sm, sh);
    if (t == 0) {
        d.count[0] = 0u;
        d.scal[S_CFLNEXT] = mx;
        d.scal[S_Q3NEXT] = sm / (d.rext2 * d.alx3);
    }
}

// the tile's coefficient vectors (cp.async), and the commit of the thread's
// cp.async group
template <class Tile>
__device__ __forceinline__ void nl_prefetch_coef(const Dev &d, Tile &t, int j0, int k0, int tid) {
    if (tid < kNlK) {
        const int k = min(k0 + tid, d.n3m);
        cp8(&t.udx3m[tid], d.udx3m + k);
        cp8(&t.ap3sk[tid], d.ap3sk + k);
        cp8(&t.ac3sk[tid], d.ac3sk + k);
        cp8(&t.am3sk[tid], d.am3sk + k);
        cp8(&t.udx3c[tid], d.udx3c + k);
        cp8(&t.ap3ck[tid], d.ap3ck + k);
        cp8(&t.ac3ck[tid], d.ac3ck + k);
        cp8(&t.am3ck[tid], d.am3ck + k);
    } else if (tid < kNlK + kNlJ) {
        const int c = tid - kNlK, j = min(j0 + c, d.n2m);
        cp8(&t.udx2c[c], d.udx2c + j);
        cp8(&t.am2j[c], d.am2j + j);
        cp8(&t.ac2j[c], d.ac2j + j);
        cp8(&t.ap2j[c], d.ap2j + j);
        cp8(&t.udx2m[c], d.udx2m + j);
        cp8(&t.am3j[c], d.am3j + j);
        cp8(&t.ac3j[c], d.ac3j + j);
        cp8(&t.ap3j[c], d.ap3j + j);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// issues the copies of one tile into t (one cp.async group per thread)
__device__ __forceinline__ void nl_prefetch(const Dev &d, NlTile &t, int tile, int ntj, int tid) {
    const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
    // tile + halo: j = j0-1 .. j0+kNlJ, k = k0-1 .. k0+kNlK (entries outside
    // the stored arrays, j < 1, j > n2, k > n3, are never read by a cell)
    constexpr int kW = kNlJ + 2, kH = kNlK + 2;
    for (int e = tid; e < kW * kH; e += 256) {
        const int r = e / kW, c = e % kW;
        const int j = j0 - 1 + c, k = k0 - 1 + r;
        if (j >= 1 && j <= d.n2 && k >= 0 && k <= d.n3) {
            const size_t i = fidx(d, j, k);
            cp8(&t.q2[r][c], d.q2 + i);
            cp8(&t.q3[r][c], d.q3 + i);
            cp8(&t.pr[r][c], d.pr + i);
        } else {
            t.q2[r][c] = 0.0;
            t.q3[r][c] = 0.0;
            t.pr[r][c] = 0.0;
        }
    }
    nl_prefetch_coef(d, t, j0, k0, tid);
}

// ru2/ru3 at this thread's cells of a tile (0 when ro = 0)
__device__ __forceinline__ void nl_ru(const Dev &d, int tile, int ntj, double ro, double (&r2)[kNlK / 8],
                                      double (&r3)[kNlK / 8]) {
    const int jc = 1 + (tile % ntj) * kNlJ + threadIdx.x, k0 = 1 + (tile / ntj) * kNlK;
#pragma unroll
    for (int i = 0; i < kNlK / 8; ++i) {
        const int kc = k0 + (kNlK / 8) * threadIdx.y + i;
        const bool ok = jc <= d.n2m && kc <= d.n3m && ro != 0.0;
        const size_t x = fidx(d, min(jc, d.n2m), min(kc, d.n3m));
        r2[i] = ok ? d.ru2[x] : 0.0;
        r3[i] = ok ? d.ru3[x] : 0.0;
    }
}

// tiles blockIdx.x, blockIdx.x + gridDim.x, ...; buf: two NlTile in shared memory
// pend: the previous substep's pressure mean (scal[S_PRAVG]) is still to be
// subtracted from pr (the fused step defers pr_submean of RK3 substeps 1 and
// 2): the staged tile gets pr - pravg, the value pr_submean would have stored.
// nb: the launch's tile blocks.  kCfl: also the field's CFL number and mean w.
template <bool kCfl>
__device__ __forceinline__ void nl_rhs_body(const Dev &d, double al, double ga, double ro, NlTile *buf, bool pend,
                                            int nb) {
    const double pravg = pend ? d.scal[S_PRAVG] : 0.0;
    double cmx = 1.0e-8, csm = 0.0;
    const int ntj = (d.n2m + kNlJ - 1) / kNlJ, ntk = (d.n3m + kNlK - 1) / kNlK, ntiles = ntj * ntk;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    int tile = blockIdx.x;
    if (tile >= ntiles) return;
    nl_prefetch(d, buf[0], tile, ntj, tid);
    double r2n[kNlK / 8], r3n[kNlK / 8];
    nl_ru(d, tile, ntj, ro, r2n, r3n);
    for (int it = 0; tile < ntiles; ++it, tile += nb) {
        const NlTile &t = buf[it & 1];
        double r2[kNlK / 8], r3[kNlK / 8];
#pragma unroll
        for (int i = 0; i < kNlK / 8; ++i) {
            r2[i] = r2n[i];
            r3[i] = r3n[i];
        }
        const int nxt = tile + nb;
        if (nxt < ntiles) {
            nl_prefetch(d, buf[(it + 1) & 1], nxt, ntj, tid);
            nl_ru(d, nxt, ntj, ro, r2n, r3n);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (pend) {
            NlTile &tw = buf[it & 1];
            for (int e = tid; e < (kNlK + 2) * (kNlJ + 2); e += 256) {
                double &x = tw.pr[e / (kNlJ + 2)][e % (kNlJ + 2)];
                x = x - pravg;
            }
            __syncthreads();
        }
        const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
        const int jc = j0 + threadIdx.x;
        if (jc <= d.n2m) {
            const double dy = kCfl ? d.rc[jc + 1] - d.rc[jc] : 0.0;
#pragma unroll
            for (int i = 0; i < kNlK / 8; ++i) {
                const int kc = k0 + (kNlK / 8) * threadIdx.y + i;
                if (kc > d.n3m) break;
                nl_cell<1>(d, t, j0, k0, jc, kc, al, ga, ro, r2[i], r3[i]);
                if (kCfl) cfl_cell<1>(t, jc - j0, kc - k0, d.zz[kc + 1] - d.zz[kc], dy, cmx, csm);
            }
        }
        __syncthreads();   // this buffer is refilled two tiles on
    }
    if (kCfl) cfl_finish(d, cmx, csm, nb);
}

// the three field boxes of a tile, issued by one thread on the buffer's
// mbarrier.  The proxy fence orders the threads' earlier reads (and the pend
// pass's writes) of this buffer before the copies overwrite it.  Boxes that
// reach past the fields (j < 1, j > n2, k > n3) are zero-filled there; no cell
// reads those entries.
__device__ __forceinline__ void nl_issue_tma(const NlMaps &m, NlTileT &t, uint32_t bar, int tile, int ntj) {
    const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
    const int x = j0 - 3, y = k0 - 1;   // x: element j - 1 of the column j = j0 - 2 (even: 16-byte aligned)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(bar, 3u * kNlBoxBytes);
    tma_load_2d(smem_u32(&t.q2[0][0]), &m.q2, bar, x, y);
    tma_load_2d(smem_u32(&t.q3[0][0]), &m.q3, bar, x, y);
    tma_load_2d(smem_u32(&t.pr[0][0]), &m.pr, bar, x, y);
}

// nl_rhs_body with the field tiles staged by TMA: tile it waits on phase
// it / 2 of its buffer's mbarrier; the coefficient vectors stay cp.async.  A
// wait that gives up (one second) records FB_ERR_TIMEOUT and ends the block's
// tiles.
template <bool kCfl>
__device__ __forceinline__ void nl_rhs_tma_body(const Dev &d, const NlMaps &m, double al, double ga, double ro,
                                                NlTileT *buf, uint64_t *bars, bool pend, int nb) {
    double cmx = 1.0e-8, csm = 0.0;
    const int ntj = (d.n2m + kNlJ - 1) / kNlJ, ntk = (d.n3m + kNlK - 1) / kNlK, ntiles = ntj * ntk;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    int tile = blockIdx.x;
    const uint32_t bar0 = smem_u32(bars), bar1 = smem_u32(bars + 1);
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar1, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {
        const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
        nl_prefetch_coef(d, buf[0], j0, k0, tid);
    }
    double r2n[kNlK / 8], r3n[kNlK / 8];
    nl_ru(d, tile, ntj, ro, r2n, r3n);
    FB_GRID_WAIT();   // (updvp before it writes q2, q3, pr and the mean)
    const double pravg = pend ? d.scal[S_PRAVG] : 0.0;
    if (tid == 0) nl_issue_tma(m, buf[0], bar0, tile, ntj);
    __syncthreads();   // the barriers are initialised before any thread waits on them
    for (int it = 0; tile < ntiles; ++it, tile += nb) {
        NlTileT &t = buf[it & 1];
        double r2[kNlK / 8], r3[kNlK / 8];
#pragma unroll
        for (int i = 0; i < kNlK / 8; ++i) {
            r2[i] = r2n[i];
            r3[i] = r3n[i];
        }
        const int nxt = tile + nb;
        if (nxt < ntiles) {
            if (tid == 0) nl_issue_tma(m, buf[(it + 1) & 1], (it & 1) ? bar0 : bar1, nxt, ntj);
            nl_prefetch_coef(d, buf[(it + 1) & 1], 1 + (nxt % ntj) * kNlJ, 1 + (nxt / ntj) * kNlK, tid);
            nl_ru(d, nxt, ntj, ro, r2n, r3n);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        const bool landed = mbar_wait((it & 1) ? bar1 : bar0, static_cast<uint32_t>(it >> 1) & 1u);
        if (__syncthreads_or(!landed)) {
            if (tid == 0) atomicCAS(d.status, 0, FB_ERR_TIMEOUT);
            break;
        }
        if (pend) {
            for (int e = tid; e < kNlTH * kNlTW; e += 256) {
                double &x = t.pr[e / kNlTW][e % kNlTW];
                x = x - pravg;
            }
            __syncthreads();
        }
        const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
        const int jc = j0 + threadIdx.x;
        if (jc <= d.n2m) {
            const double dy = kCfl ? d.rc[jc + 1] - d.rc[jc] : 0.0;
#pragma unroll
            for (int i = 0; i < kNlK / 8; ++i) {
                const int kc = k0 + (kNlK / 8) * threadIdx.y + i;
                if (kc > d.n3m) break;
                nl_cell<2>(d, t, j0, k0, jc, kc, al, ga, ro, r2[i], r3[i]);
                if (kCfl) cfl_cell<2>(t, jc - j0, kc - k0, d.zz[kc + 1] - d.zz[kc], dy, cmx, csm);
            }
        }
        __syncthreads();   // this buffer is refilled two tiles on
    }
    if (kCfl) cfl_finish(d, cmx, csm, nb);
}

// the blocks of nl_rhs's launch beyond the tiles' (kernels.h: extra)
__host__ __device__ inline int nl_more(int extra) {
    return ((extra & kNlBoucdq) ? 1 : 0) + ((extra & kNlMeans) ? 1 : 0);
}

template <bool kCfl>
__global__ void __launch_bounds__(256, kNlBlocksPerSM)
    k_nl_rhs_tma(const __grid_constant__ Dev d, const __grid_constant__ NlMaps m, double al, double ga, double ro,
                 int pend, int extra) {
    extern __shared__ __align__(16) unsigned char nl_smem[];
    const uint32_t raw = smem_u32(nl_smem);
    unsigned char *base = nl_smem + ((128u - (raw & 127u)) & 127u);   // the tiles on 128-byte boundaries
    NlTileT *buf = reinterpret_cast<NlTileT *>(base);
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + 2 * sizeof(NlTileT));
    const int nb = gridDim.x - nl_more(extra);   // (at most one block per tile)
    if (static_cast<int>(blockIdx.x) >= nb) {
        FB_GRID_WAIT();
        if ((extra & kNlBoucdq) && static_cast<int>(blockIdx.x) == nb) boucdq_body(d, ga, ro);
        else edge_means_body(d);
        return;
    }
    nl_rhs_tma_body<kCfl>(d, m, al, ga, ro, buf, bars, pend != 0, nb);
}

// ------------------------------------------------------------ MLS forcing

__device__ int nearest_sorted(const double *a, int lo, int hi, double x, int guess) {
    // first index of min |a(i) - x| over a(lo..hi), a strictly increasing.
    // The bracket a(l) <= x < a(l+1) is unique: it is searched from the
    // marker's index of the previous step (a few steps) and by bisection
    // when that guess is off; both give the same l.
    if (x <= a[lo]) return lo;
    if (x >= a[hi]) return hi;
    int l = -1;
    if (guess >= lo && guess < hi) {
        int g = guess;
        for (int s = 0; s < 16 && g > lo && a[g] > x; ++s) --g;
        for (int s = 0; s < 16 && g < hi - 1 && a[g + 1] <= x; ++s) ++g;
        if (a[g] <= x && x < a[g + 1]) l = g;
    }
    if (l < 0) {
        int h = hi;
        l = lo;
        while (h - l > 1) {
            int m = (l + h) >> 1;
            if (a[m] <= x) l = m;
            else h = m;
        }
    }
    const int h = l + 1;
    double dl = fabs(a[l] - x), dh = fabs(a[h] - x);
    return (dh < dl) ? h : l;
}

// entry of a spreading-table key (Fibonacci hashing: the top hlog bits of
// key x 2^64 / golden ratio)
__device__ __forceinline__ unsigned bucket_hash(unsigned long long key, int hlog) {
    return static_cast<unsigned>((key * 0x9E3779B97F4A7C15ull) >> (64 - hlog));
}

// empties the spreading-table entry that (marker, direction) tt filled.  Every
// used entry is some marker's own, so all of them together empty the table.
__device__ __forceinline__ void clear_entry(const Dev &d, int tt) {
    const int e = d.hslot[tt];
    if (!e) return;
    d.hkey[e - 1] = 0ull;
    d.hcnt[e - 1] = 0;
    d.hslot[tt] = 0;
}

// lgrdistribution.F90:189-267: nearest nodes per marker and direction
__device__ __forceinline__ void lgrdist_body(const Dev &d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.nlm) return;
    for (int dir = 0; dir < 2; ++dir) clear_entry(d, 2 * i + dir);   // empty before the set-up fills it
    const double y = d.lmcc[2 * i], z = d.lmcc[2 * i + 1];
    if (y > d.rext2 || y < 0.0 || z > d.alx3 || z < 0.0 || !(y == y) || !(z == z)) {
        raise_status(d, FB_ERR_MARKER_OUT);
        for (int c = 0; c < 4; ++c) d.lmind[4 * i + c] = -1;
        return;
    }
    int ind;
    const int g0 = d.lmind[4 * i + 0], g1 = d.lmind[4 * i + 1], g2 = d.lmind[4 * i + 2], g3 = d.lmind[4 * i + 3];
    d.lmind[4 * i + 0] = nearest_sorted(d.rc, 1, d.n2, y, g0);
    if (z < d.zm[1] && z > 0.0) ind = 1;
    else if (z > d.zm[d.n3m] && z < d.alx3) ind = d.n3m;
    else ind = nearest_sorted(d.zm, 1, d.n3, z, g1);
    d.lmind[4 * i + 1] = ind;
    if (y < d.rm[1] && y > 0.0) ind = 1;
    else if (y > d.rm[d.n2m] && y < d.rext2) ind = d.n2m;
    else ind = nearest_sorted(d.rm, 1, d.n2, y, g2);
    d.lmind[4 * i + 2] = ind;
    d.lmind[4 * i + 3] = nearest_sorted(d.zz, 1, d.n3, z, g3);
}

__global__ void k_lgrdist(Dev d) {
    FB_GRID_WAIT();
    lgrdist_body(d);
}

// utils_math.f90:637-725 (GEsolve), n = 3, scaled partial pivoting: the
// elimination of the matrix, whose multipliers and row exchanges are kept so
// that further right-hand sides take the same operations without repeating it
// (the same results).  Every loop is unrolled and the row exchange written per
// candidate row, so that the matrix stays in registers.
struct GeLu {
    double a[3][3];   // upper triangle
    double c[2][3];   // multipliers c[k][i], i > k
    int l[2];         // row exchanged with row k
    bool ok;
};

__device__ __forceinline__ void ge_factor(const double ai[3][3], GeLu &f) {
    f.ok = true;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) f.a[i][j] = ai[i][j];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        double s[3];
#pragma unroll
        for (int i = k; i < 3; ++i) {
            s[i] = 0.0;
#pragma unroll
            for (int j = k; j < 3; ++j) s[i] = fmax(s[i], fabs(f.a[i][j]));
        }
        double pivot = fabs(f.a[k][k] / s[k]);
        int l = k;
#pragma unroll
        for (int j = k + 1; j < 3; ++j) {
            const double q = fabs(f.a[j][k] / s[j]);
            if (q > pivot) {
                pivot = q;
                l = j;
            }
        }
        if (pivot == 0.0) f.ok = false;
        f.l[k] = l;
#pragma unroll
        for (int r = k + 1; r < 3; ++r) {
            if (l != r) continue;
#pragma unroll
            for (int j = k; j < 3; ++j) {
                const double t = f.a[k][j];
                f.a[k][j] = f.a[r][j];
                f.a[r][j] = t;
            }
        }
#pragma unroll
        for (int i = k + 1; i < 3; ++i) {
            const double c = f.a[i][k] / f.a[k][k];
            f.c[k][i] = c;
#pragma unroll
            for (int j = k + 1; j < 3; ++j) f.a[i][j] = f.a[i][j] - c * f.a[k][j];
        }
    }
}

__device__ __forceinline__ void ge_apply(const GeLu &f, const double bi[3], double x[3]) {
    double b[3] = {bi[0], bi[1], bi[2]};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
#pragma unroll
        for (int r = k + 1; r < 3; ++r) {
            if (f.l[k] != r) continue;
            const double t = b[k];
            b[k] = b[r];
            b[r] = t;
        }
#pragma unroll
        for (int i = k + 1; i < 3; ++i) b[i] = b[i] - f.c[k][i] * b[k];
    }
    x[2] = b[2] / f.a[2][2];
#pragma unroll
    for (int i = 1; i >= 0; --i) {
        double c = 0.0;
#pragma unroll
        for (int j = i + 1; j < 3; ++j) c = c + f.a[i][j] * x[j];
        x[i] = (b[i] - c) / f.a[i][i];
    }
}

// MLSint.F90:406-486 (one axis of the weight function) and its derivative
// MLSint.F90:492-593
__device__ void wkernel(int wfun, double difc, double sdds, double &wc, double &dw) {
    double drdc = (fabs(difc) <= 1.0e-20) ? 0.0 : (difc / fabs(difc)) / sdds;
    double rc = fabs(difc) / sdds;
    double rc2 = rc * rc, rc3 = rc * rc * rc, rc4 = rc * rc * rc * rc;
    wc = 0.0;
    dw = 0.0;
    if (wfun == 1) {
        if (rc > 1.0) {
        } else if (rc <= 0.5) {
            wc = (2.0 / 3.0) - 4.0 * rc2 + 4.0 * rc3;
            dw = (-8.0 * rc + 12.0 * rc2) * drdc;
        } else {
            wc = (4.0 / 3.0) - 4.0 * rc + 4.0 * rc2 - (4.0 / 3.0) * rc3;
            dw = (-4.0 + 8.0 * rc - 4.0 * rc2) * drdc;
        }
    } else if (wfun == 2) {
        if (rc <= 1.0) {
            double e = exp(-((rc / 0.3) * (rc / 0.3)));
            wc = e;
            dw = (-1.0 / (0.3 * 0.3) * 2.0 * rc * e) * drdc;
        }
    } else if (wfun == 3) {
        if (rc <= 1.0) {
            wc = 1.0 - 6.0 * rc2 + 8.0 * rc3 - 3.0 * rc4;
            dw = -12.0 * rc + 24.0 * rc2 - 12.0 * rc3;
        }
    } else if (wfun == 4) {
        if (rc > 1.0) {
        } else if (rc < 0.5) {
            wc = 1.0 / 3.0 * (1.0 + sqrt(-3.0 * rc2 + 1.0));
            dw = -rc * pow(-3.0 * rc2 - 1.0, -0.5);
        } else {
            wc = 1.0 / 6.0 * (5.0 - 3.0 * rc - sqrt(-3.0 * ((1.0 - rc) * (1.0 - rc)) + 1.0));
            dw = -(1.0 - rc) / (2.0 * sqrt(1.0 - 3.0 * ((1.0 - rc) * (1.0 - rc)))) - 0.5;
        }
    }
}

// Groups of kNodeLanes lanes work on one (marker, direction) each, support
// node m on lane m < kSD; a sum over the support is formed in node order
// (group_sums; the sequential loop's sum).  Every lane of a warp reaches every
// exchange: a group that stops (outside the channel, an error) carries on with
// its loads and stores switched off.
constexpr int kNodeLanes = 16;

// N sums over the group's nodes through shared memory (buf: 10 N doubles of the
// group's own): lane i forms sums i, i + kNodeLanes, ... from the nine terms the nodes
// left there, in node order, and every lane reads them back.  One shuffle and
// addition after another per sum (18 of them for a probe) was most of the
// instructions of these latency-bound kernels.
template <int N>
__device__ __forceinline__ void group_sums(double (&x)[N], int m, double *buf) {
    __syncwarp();   // (the buffer's earlier values are read)
    if (m < kSD)
#pragma unroll
        for (int i = 0; i < N; ++i) buf[i * kSD + m] = x[i];
    __syncwarp();
#pragma unroll
    for (int i0 = 0; i0 < N; i0 += kNodeLanes) {
        const int i = i0 + m;
        if (i < N) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < kSD; ++q) s = s + buf[i * kSD + q];
            buf[N * kSD + i] = s;
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = buf[N * kSD + i];
}

// the group's lane index of the least v, the first of equal values (as a
// sequential search with a strict comparison finds it); lanes past the
// searched range hold +inf
__device__ __forceinline__ int group_argmin(double v, int m) {
    int i = m;
#pragma unroll
    for (int o = kNodeLanes / 2; o; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        if (ov < v || (ov == v && oi < i)) {
            v = ov;
            i = oi;
        }
    }
    return i;
}

// true when no lane of the group (base .. base + kNodeLanes - 1) has flag set
__device__ __forceinline__ bool group_none(bool flag, int base) {
    return (__ballot_sync(0xffffffffu, flag) & (((1u << kNodeLanes) - 1u) << base)) == 0u;
}

// the support arrays of MLS_SD_ind (MLSint.F90:4-104) for direction idir
__device__ __forceinline__ void sd_axes(const Dev &d, int idir, const double *&y, int &dimy, const double *&z,
                                        int &dimz) {
    if (idir == 1) {
        y = d.rc; dimy = d.n2; z = d.zm; dimz = d.n3m;
    } else if (idir == 2) {
        y = d.rm; dimy = d.n2m; z = d.zz; dimz = d.n3;
    } else {
        y = d.rm; dimy = d.n2m; z = d.zm; dimz = d.n3m;
    }
}

// Marker set-up at substep 1: MLS_SD_ind + MLS_SF + momentum coefficient cl
// (forcing_MLS.F90:57-94, MLSint.F90:115-166, compute_AB :284-338), and the
// spreading keys.  One (marker, direction) per group of kNodeLanes lanes.
// kFind: the group also finds its nearest y and z lines
// (lgrdistribution.F90:189-267), one per lane, in place of a launch of its own
// whose threads made the four searches of a marker one after another; the
// spreading table has to be empty then: k_mls_interp empties it behind the
// chains, k_table_clear where a step ends before it.
constexpr int kSetupThreads = 128;
template <bool kFind>
__device__ __forceinline__ void mls_setup_body(const Dev &d) {
    if (!d.nlm) return;
    const int T = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = T / kNodeLanes, m = T % kNodeLanes;
    const int base = (threadIdx.x & 31) & ~(kNodeLanes - 1);
    __shared__ double bufs[kSetupThreads / kNodeLanes][10 * 6];
    double *buf = bufs[threadIdx.x / kNodeLanes];
    const bool have = t < 2 * d.nlm;
    const int tt = have ? t : 0;
    const int n = tt >> 1, idir = (tt & 1) + 1;
    const bool node = m < kSD;
    double *phi = d.phi + static_cast<size_t>(tt) * kSD;
    int *eu = d.eulins + static_cast<size_t>(tt) * 2 * kSD;
    if (have && node) phi[m] = 0.0;
    if (have && m == 0) d.cl[tt] = 0.0;
    const bool stopped = __shfl_sync(0xffffffffu, static_cast<int>(*d.status != 0), base) != 0;
    const double pos[2] = {d.lmcc[2 * n], d.lmcc[2 * n + 1]};
    const bool ok = have && !stopped && (d.zz[1] < pos[1] && pos[1] < d.zz[d.n3]);
    int *lmi = d.lmind + 4 * n + 2 * (idir - 1);   // nearest y line, nearest z line
    int i0, k0;
    if constexpr (kFind) {
        int ind = -1;
        if (have && m < 2) {
            const double x = pos[m], far = (m == 0) ? d.rext2 : d.alx3;
            const bool out = pos[0] > d.rext2 || pos[0] < 0.0 || pos[1] > d.alx3 || pos[1] < 0.0 ||
                             !(pos[0] == pos[0]) || !(pos[1] == pos[1]);
            if (out) {
                if (m == 0) raise_status(d, FB_ERR_MARKER_OUT);
            } else {
                // cell-centred lines (zm of v, rm of w) keep a marker beyond
                // their first or last one
                const bool centred = (m == 1) == (idir == 1);
                const double *a = (m == 0) ? (centred ? d.rm : d.rc) : (centred ? d.zm : d.zz);
                const int hi = (m == 0) ? d.n2 : d.n3, mid = hi - 1;
                if (centred && x < a[1] && x > 0.0) ind = 1;
                else if (centred && x > a[mid] && x < far) ind = mid;
                else ind = nearest_sorted(a, 1, hi, x, lmi[m]);
            }
            lmi[m] = ind;
        }
        i0 = __shfl_sync(0xffffffffu, ind, base);
        k0 = __shfl_sync(0xffffffffu, ind, base + 1);
    } else {
        i0 = lmi[0];
        k0 = lmi[1];
    }
    // MLS_SD_ind: node m = 3 (j - 1) + (k - 1) of the 3 x 3 support, moved
    // inside the field
    const double *y, *z;
    int dimy, dimz;
    sd_axes(d, idir, y, dimy, z, dimz);
    const int sj = (i0 == 1) ? 1 : (i0 == d.n2m ? -1 : 0);
    const int sk = (k0 == 1) ? 1 : (k0 == d.n3m ? -1 : 0);
    const int mm = node ? m : 0;
    const int ej = i0 + (mm / 3 + 1 + sj) - 2, ek = k0 + (mm % 3 + 1 + sk) - 2;
    const bool bad = ok && node && (ej < 1 || ej + 1 > dimy || ek < 1 || ek + 1 > dimz);
    const bool good = group_none(bad, base) && ok && i0 >= 1 && k0 >= 1;
    if (ok && !good && m == 0) raise_status(d, FB_ERR_MARKER_OUT);
    double sc0 = 0.0, sc1 = 0.0, sd0 = 0.0, sd1 = 0.0, w = 0.0;
    if (good && node) {
        sc0 = y[ej];
        sd0 = y[ej + 1] - y[ej];
        sc1 = z[ek];
        sd1 = z[ek + 1] - z[ek];
        double wc0, wc1, dw;
        wkernel(d.wfun, pos[0] - sc0, d.radiusSD * sd0, wc0, dw);
        wkernel(d.wfun, pos[1] - sc1, d.radiusSD * sd1, wc1, dw);
        w = wc0 * wc1;
    }
    const double pk[3] = {1.0, sc0, sc1};
    double mom[6];   // pk[a] pk[b] = pk[b] pk[a]: the same terms, the same sums
    int q = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a; b < 3; ++b) mom[q++] = w * (pk[a] * pk[b]);
    group_sums<6>(mom, m, buf);
    const double A[3][3] = {{mom[0], mom[1], mom[2]}, {mom[1], mom[3], mom[4]}, {mom[2], mom[4], mom[5]}};
    const double gps[3] = {1.0, pos[0], pos[1]};
    double ptA[3];
    GeLu lu;
    ge_factor(A, lu);
    ge_apply(lu, gps, ptA);
    const double B0 = 1.0 * w, B1 = sc0 * w, B2 = sc1 * w;
    double ph = 0.0;
    ph = ph + ptA[0] * B0;
    ph = ph + ptA[1] * B1;
    ph = ph + ptA[2] * B2;
    const double vol = sd0 * sd1;
    double sums[3] = {ph, ph * vol, 1.0 / 2.0 * ph * (sd0 + sd1)};
    group_sums<3>(sums, m, buf);
    const double sumphi = sums[0], dvel = sums[1], lgr_h = sums[2];
    if (good && m == 0 && !(fabs(1.0 - fabs(sumphi)) <= 1.0e-10)) raise_status(d, FB_ERR_MLS);
    if (!good) return;   // (after the group's last exchange)
    if (node) {
        phi[m] = ph;
        eu[m] = ej;
        eu[kSD + m] = ek;
    }
    if (m != 0) return;
    d.cl[tt] = d.lmA[n] * lgr_h / dvel;
    // register the support box (start cell = node m = 0, this lane's) for the spreading
    const unsigned long long cell = static_cast<unsigned long long>(idir - 1) * d.NK * d.P + fidx(d, ej, ek);
    const unsigned mask = (1u << d.hlog) - 1u;
    for (int lev = 0; lev < kBucketLevels; ++lev) {
        const unsigned long long key = cell * kBucketLevels + lev + 1;
        unsigned h = bucket_hash(key, d.hlog);
        for (unsigned probes = 0;; ++probes) {   // find or claim the key's entry
            const unsigned long long prev = atomicCAS(d.hkey + h, 0ull, key);
            if (prev == 0ull || prev == key) break;
            if (probes == mask) {   // full: cannot happen at the table's sizing
                raise_status(d, FB_ERR_UNSUPPORTED);
                return;
            }
            h = (h + 1) & mask;
        }
        const int slot = atomicAdd(d.hcnt + h, 1);
        if (slot < kBucket) {
            d.hval[static_cast<size_t>(h) * kBucket + slot] = n;
            d.hslot[tt] = static_cast<int>(h) + 1;
            return;
        }
    }
    raise_status(d, FB_ERR_UNSUPPORTED);   // more than kBucket x kBucketLevels boxes start in one cell
}

template <bool kFind>
__global__ void k_mls_setup(Dev d) {
    FB_GRID_WAIT();
    mls_setup_body<kFind>(d);
}

// interp_spread (forcing_MLS.F90:135-182), interpolation half: the
// provisional velocity q* = q + rhs (INVTR.F90:147,275) at the support,
// direct forcing F = (V - u*)/dt and the per-node contributions cl*phi*F.
// One (marker, direction) per 16 lanes, node m on lane m < kSD: the nine
// support loads are independent, and each lane forms the sum of the nine
// products in node order from the group's shuffles (the sequential sum).
// clear (substep 1): the spreading table, read for the last time by
// k_spread_chains, is emptied for the next step.  cfl (substep 1 at fixed dt): a
// CFL number beyond the limit, which nl_rhs has just formed, ends the step's
// forcing here in every substep (divg makes it the step's number).
constexpr int kInterpLanes = 16;
// kWait: the body waits for the kernel before it (nl_rhs, which writes
// rhs2/rhs3, or the spreading chains) with everything else loaded.
template <bool kWait>
__device__ __forceinline__ void mls_interp_body(const Dev &d, bool clear, bool cfl) {
    const int T = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = T / kInterpLanes, m = T % kInterpLanes, lane = threadIdx.x & 31;
    const bool have = t < 2 * d.nlm;
    const int tt = have ? t : 0;
    const int n = tt >> 1, idir = (tt & 1) + 1;
    const double pos2 = d.lmcc[2 * n + 1], vel = d.lmvel[2 * n + idir - 1], cl = d.cl[tt];
    const bool inside = (d.zz[1] < pos2 && pos2 < d.zz[d.n3]);
    const bool node = have && inside && m < kSD;
    double phim = 0.0, qv = 0.0;
    const double *rp = nullptr;
    if (node) {
        const int *eu = d.eulins + static_cast<size_t>(tt) * 2 * kSD;
        const double *q = (idir == 1) ? d.q2 : d.q3;
        phim = d.phi[static_cast<size_t>(tt) * kSD + m];
        const int j = eu[m], k = eu[kSD + m];
        // q2f/q3f are written only where invtr2/invtr3 write them; elsewhere
        // the reference reads storage that was never set (zero here)
        const bool written = (idir == 1) ? (j >= 2 && j <= d.n2m && k >= 1 && k <= d.n3m)
                                         : (j >= 1 && j <= d.n2m && k >= 2 && k <= d.n3m);
        if (written) {
            const size_t i = fidx(d, j, k);
            qv = __ldcg(q + i);
            rp = ((idir == 1) ? d.rhs2 : d.rhs3) + i;
        }
    }
    if (kWait) FB_GRID_WAIT();
    const bool over = cfl && !(d.scal[S_CFLNEXT] * d.dt <= d.cfllim);
    if (over && T == 0) raise_status(d, FB_ERR_CFL);
    const bool stopped = over || *d.status != 0;
    if (clear && have && m == kInterpLanes - 1) clear_entry(d, tt);   // (a lane without a node)
    const double prod = rp ? phim * (qv + *rp) : phim * 0.0;
    double u = 0.0;
#pragma unroll
    for (int mm = 0; mm < kSD; ++mm) u = u + __shfl_sync(0xffffffffu, prod, (lane & ~(kInterpLanes - 1)) + mm);
    if (!have || stopped || m >= kSD) return;
    double *c = d.contrib + static_cast<size_t>(tt) * kSD;
    if (!inside) {
        c[m] = 0.0;
        return;
    }
    const double f = (vel - u) / d.dt;
    c[m] = cl * phim * f;
}

__global__ void k_mls_interp(Dev d, int clear, int cfl) { mls_interp_body<true>(d, clear != 0, cfl != 0); }

// the spreading table emptied on its own: a step that ends between its marker
// set-up and its interpolation (a refused dt)
__global__ void k_table_clear(Dev d) {
    FB_GRID_WAIT();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 2 * d.nlm) clear_entry(d, t);
}

// interp_spread, spreading half, without atomics on the field.  Once per
// step (the supports are fixed for the three substeps) every cell's touchers
// are found in the buckets of the 3 x 3 possible box start cells and chained
// in increasing marker index (the reference's loop order,
// forcing_MLS.F90:51-104); the head of each chain is the lowest-index
// toucher.  Every substep the heads then add their chain's sum fe*dt to rhs
// (helsolve.F90:22,47).
// one slot's chain by one thread: dense marker clusters (more touchers than a
// group's list holds, or cells with more than one table entry)
__device__ __noinline__ void spread_chain_serial(const Dev &d, int g) {
    const int t = g / kSD, m = g % kSD, n = t >> 1, dir = t & 1;
    const int *eu = d.eulins + static_cast<size_t>(t) * 2 * kSD;
    const int j = eu[m], k = eu[kSD + m];
    const size_t plane = static_cast<size_t>(dir) * d.NK * d.P;
    // the cell's touchers are the markers registered at the 3 x 3 possible
    // box start cells (table lookups); a lower-index toucher means this slot
    // is not the head
    constexpr int kMaxTouch = 9 * kBucket;   // touchers of one cell kept at most
    int ln[kMaxTouch], ls[kMaxTouch];         // touchers after n, ascending marker index
    int L = 0;
    bool over = false;
    const unsigned mask = (1u << d.hlog) - 1u;
    for (int q = 0; q < 9; ++q) {
        const int sj = j - q / 3, sk = k - q % 3;
        if (sj < 1 || sk < 0) continue;
        const unsigned long long cell = plane + fidx(d, sj, sk);
        for (int lev = 0; lev < kBucketLevels; ++lev) {
            const unsigned long long key = cell * kBucketLevels + lev + 1;
            unsigned h = bucket_hash(key, d.hlog);
            unsigned long long kh = d.hkey[h];
            for (unsigned probes = 0; kh != key && kh != 0ull && probes < mask; ++probes) {
                h = (h + 1) & mask;
                kh = d.hkey[h];
            }
            if (kh != key) break;   // no (further) boxes start in this cell
            const int cnt = d.hcnt[h];
            for (int e = 0; e < min(cnt, kBucket); ++e) {
                const int nn = d.hval[static_cast<size_t>(h) * kBucket + e];
                if (nn < n) return;
                if (nn == n) continue;
                if (L >= kMaxTouch) {   // denser than the marker spacing the spreading is built for
                    over = true;
                    continue;
                }
                // insertion in increasing marker index (a marker has one box start cell)
                int p = L++;
                while (p > 0 && ln[p - 1] > nn) {
                    ln[p] = ln[p - 1];
                    ls[p] = ls[p - 1];
                    --p;
                }
                ln[p] = nn;
                ls[p] = (2 * nn + dir) * kSD + q;   // node (dj, dk) = (q / 3, q % 3) of marker nn
            }
            if (cnt <= kBucket) break;   // the cell's last entry
        }
    }
    if (over) {
        raise_status(d, FB_ERR_UNSUPPORTED);
        return;
    }
    // this slot heads the cell's chain: link the touchers in marker order;
    // the head also keeps the first kHeadList of them in line
    d.chead[g] = 1;
    int prev_slot = g;
    for (int p = 0; p < L; ++p) {
        d.chain[prev_slot] = ls[p];
        prev_slot = ls[p];
    }
    d.chain[prev_slot] = -1;
    d.hlen[g] = L;
    int *hl = d.hlist + static_cast<size_t>(g) * kHeadList;
    for (int p = 0; p < kHeadList; ++p) hl[p] = (p < L) ? ls[p] : g;
}

// A slot's cell by a group of kNodeLanes lanes: lane q < 9 looks up the box
// start cell q (the nine dependent chains of table reads side by side, where
// one thread's went one after another), the touchers found go to the group's
// list in shared memory, and each is placed by its rank among them.  Under ncu
// 23.9 -> 9.5 us with 1200 markers, 17.6 -> 6.5 us with 302.
constexpr int kChainThreads = 256;
constexpr int kChainList = 64;   // touchers per group's list (9 boxes of up to 7 markers)
__device__ __forceinline__ void spread_chains_body(const Dev &d) {
    __shared__ int lists[kChainThreads / kNodeLanes][3][kChainList];   // marker, slot, slots in order
    constexpr unsigned kAll = 0xffffffffu;
    const int T = blockIdx.x * blockDim.x + threadIdx.x;
    const int g0 = T / kNodeLanes, m = T % kNodeLanes;
    const int base = (threadIdx.x & 31) & ~(kNodeLanes - 1);
    const bool have = g0 < 2 * d.nlm * kSD;
    const int g = have ? g0 : 0;
    if (have && m == 0) d.chead[g] = 0;
    const int t = g / kSD, n = t >> 1, dir = t & 1;
    const double pos2 = d.lmcc[2 * n + 1];
    const int *eu = d.eulins + static_cast<size_t>(t) * 2 * kSD;
    const int j = eu[g % kSD], k = eu[kSD + g % kSD];
    // cells helsolve reads: v at j = 2..n2m, k = 1..n3m; w at j = 1..n2m, k = 2..n3m
    const bool used = (dir == 0) ? (j >= 2 && j <= d.n2m && k >= 1 && k <= d.n3m)
                                 : (j >= 1 && j <= d.n2m && k >= 2 && k <= d.n3m);
    const bool stopped = __shfl_sync(kAll, static_cast<int>(*d.status != 0), base) != 0;
    const bool act = have && !stopped && used && (d.zz[1] < pos2 && pos2 < d.zz[d.n3]);
    // the cell's touchers are the markers registered at the 3 x 3 possible
    // box start cells
    int cnt = 0;
    unsigned h = 0;
    const int sj = j - m / 3, sk = k - m % 3;
    if (act && m < kSD && sj >= 1 && sk >= 0) {
        const unsigned mask = (1u << d.hlog) - 1u;
        const unsigned long long key =
            (static_cast<unsigned long long>(dir) * d.NK * d.P + fidx(d, sj, sk)) * kBucketLevels + 1;
        h = bucket_hash(key, d.hlog);
        unsigned long long kh = d.hkey[h];
        cnt = d.hcnt[h];
        for (unsigned probes = 0; kh != key && kh != 0ull && probes < mask; ++probes) {
            h = (h + 1) & mask;
            kh = d.hkey[h];
            cnt = d.hcnt[h];
        }
        if (kh != key) cnt = 0;   // no boxes start in this cell
    }
    int off = cnt;   // inclusive sums over the group's lanes
#pragma unroll
    for (int o = 1; o < kNodeLanes; o <<= 1) {
        const int x = __shfl_up_sync(kAll, off, o, kNodeLanes);
        if (m >= o) off += x;
    }
    const int total = __shfl_sync(kAll, off, base + kNodeLanes - 1);
    const bool serial = !group_none(cnt > kBucket, base) || total > kChainList;
    int(&list)[3][kChainList] = lists[threadIdx.x / kNodeLanes];
    bool lower = false;   // a lower-index toucher: this slot is not the head
    if (!serial)
        for (int e = 0; e < cnt; ++e) {
            const int nn = d.hval[static_cast<size_t>(h) * kBucket + e];
            lower = lower || nn < n;
            list[0][off - cnt + e] = nn;
            list[1][off - cnt + e] = (2 * nn + dir) * kSD + m;   // node (dj, dk) = (m / 3, m % 3) of marker nn
        }
    const bool head = group_none(lower, base) && act;
    __syncwarp();
    if (head && !serial) {
        for (int i = m; i < total; i += kNodeLanes) {
            const int nn = list[0][i];
            if (nn == n) continue;
            int r = -1;   // rank among the touchers after n (n itself is lower)
            for (int p = 0; p < total; ++p) r += (list[0][p] < nn) ? 1 : 0;
            list[2][r] = list[1][i];
        }
    }
    __syncwarp();
    if (!head) return;
    if (serial) {
        if (m == 0) spread_chain_serial(d, g);
        return;
    }
    // this slot heads the cell's chain: link the touchers in marker order;
    // the head also keeps the first kHeadList of them in line
    const int L = total - 1;
    for (int p = m; p <= L; p += kNodeLanes) d.chain[p ? list[2][p - 1] : g] = (p < L) ? list[2][p] : -1;
    if (m < kHeadList) d.hlist[static_cast<size_t>(g) * kHeadList + m] = (m < L) ? list[2][m] : g;
    if (m == 0) {
        d.hlen[g] = L;
        d.chead[g] = 1;
    }
}

// (a grid constant: the call of the serial form takes its address, and a copy
// of it on every thread's stack cost more than the kernel)
__global__ void k_spread_chains(const __grid_constant__ Dev d) {
    FB_GRID_WAIT();
    spread_chains_body(d);
}

// kWait: the body waits for the kernel before it (k_mls_interp, which writes
// contrib) with the slot's chain and its cell's right-hand side loaded.
template <bool kWait>
__device__ __forceinline__ void mls_spread_body(const Dev &d) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const bool head = g < 2 * d.nlm * kSD && d.chead[g] != 0;   // the head of a cell's chain
    int L = 0;
    int4 h0{}, h1{};
    double *r = nullptr, rv = 0.0;
    if (head) {
        const int t = g / kSD, dir = t & 1, m = g % kSD;
        const int *eu = d.eulins + static_cast<size_t>(t) * 2 * kSD;
        // the head's in-line list gives the first kHeadList members at once
        // (independent loads); a longer chain continues along chain[]; the sum
        // runs in chain order
        L = d.hlen[g];
        const int4 *hl = reinterpret_cast<const int4 *>(d.hlist + static_cast<size_t>(g) * kHeadList);
        h0 = hl[0];
        h1 = hl[1];
        r = ((dir == 0) ? d.rhs2 : d.rhs3) + fidx(d, eu[m], eu[kSD + m]);
        rv = __ldcg(r);
    }
    if (kWait) FB_GRID_WAIT();
    if (!head || *d.status) return;
    const int idx[kHeadList] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    double cv[kHeadList];
#pragma unroll
    for (int p = 0; p < kHeadList; ++p) cv[p] = d.contrib[idx[p]];   // the head's own slot past the end
    double fe = 0.0;
    fe = fe + d.contrib[g];
#pragma unroll
    for (int p = 0; p < kHeadList; ++p)
        if (p < L) fe = fe + cv[p];
    if (L > kHeadList)
        for (int s = d.chain[idx[kHeadList - 1]]; s >= 0; s = d.chain[s]) fe = fe + d.contrib[s];
    *r = rv + fe * d.dt;
}

__global__ void k_mls_spread(Dev d) { mls_spread_body<true>(d); }

// ------------------------------------------------------------ tridiagonal

// DGTTS2 (LAPACK) for one line with precomputed DGTTRF factors; b strided.
// The pivots are stored as reciprocals, so the back substitution multiplies.
__device__ __forceinline__ void gtts2(const TriDev &f, size_t off, double *b, size_t s) {
    const int n = f.n;
    const double *dl = f.dl + off, *dinv = f.dinv + off, *du = f.du + off, *du2 = f.du2 + off;
    if (!f.pivoted) {
        double prev = b[0];
        for (int i = 0; i < n - 1; ++i) {
            double cur = b[(i + 1) * s] - dl[i] * prev;
            b[(i + 1) * s] = cur;
            prev = cur;
        }
        double x1 = b[(n - 1) * s] * dinv[n - 1];
        b[(n - 1) * s] = x1;
        for (int i = n - 2; i >= 0; --i) {
            double x0 = (b[i * s] - du[i] * x1) * dinv[i];
            b[i * s] = x0;
            x1 = x0;
        }
    } else {
        const int *ipiv = f.ipiv + off;
        for (int i = 0; i < n - 1; ++i) {
            if (ipiv[i] == i + 1) {
                b[(i + 1) * s] = b[(i + 1) * s] - dl[i] * b[i * s];
            } else {
                double temp = b[i * s] - dl[i] * b[(i + 1) * s];
                b[i * s] = b[(i + 1) * s];
                b[(i + 1) * s] = temp;
            }
        }
        b[(n - 1) * s] = b[(n - 1) * s] * dinv[n - 1];
        if (n > 1) b[(n - 2) * s] = (b[(n - 2) * s] - du[n - 2] * b[(n - 1) * s]) * dinv[n - 2];
        for (int i = n - 3; i >= 0; --i)
            b[i * s] = (b[i * s] - du[i] * b[(i + 1) * s] - du2[i] * b[(i + 2) * s]) * dinv[i];
    }
}

// solve_fluid.F90:110-160 (solq2j): v, y lines of n2 unknowns, k = 1..n3m
__global__ void k_tri_y2(Dev d, SubDev s) {
    FB_GRID_WAIT();
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (k > d.n3m) return;
    double *b = d.rhs2 + fidx(d, 1, k);
    b[0] = 0.0;
    for (int j = 2; j <= d.n2m; ++j) b[j - 1] = b[j - 1] * s.by2[j];
    b[d.n2 - 1] = 0.0;
    gtts2(s.y2, 0, b, 1);
}

// solve_fluid.F90:164-229 (solq2k) then helsolve.F90:32-33: v, z lines of
// n3m unknowns with the inflow/outflow terms, q2 += x, wall columns zeroed
__global__ void k_tri_z2(Dev d, SubDev s) {
    FB_GRID_WAIT();
    const int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (j > d.n2m) return;
    if (j == 1) {
        for (int k = 0; k <= d.n3; ++k) {
            Fv(d.q2, 1, k) = 0.0;
            Fv(d.q2, d.n2, k) = 0.0;
        }
        return;
    }
    double *b = d.rhs2 + fidx(d, j, 1);
    const size_t P = static_cast<size_t>(d.P);
    for (int k = 1; k <= d.n3m; ++k) b[(k - 1) * P] = b[(k - 1) * P] * s.bz2[k];
    b[0] = b[0] + d.dqb2s[j] * s.ugkks;
    b[(d.n3m - 1) * P] = b[(d.n3m - 1) * P] + d.dqb2n[j] * s.ugkkn;
    gtts2(s.z2, 0, b, P);
    for (int k = 1; k <= d.n3m; ++k) Fv(d.q2, j, k) = Fv(d.q2, j, k) + b[(k - 1) * P];
}

// solve_fluid.F90:61-104 (solq3j): w, y lines of n2m unknowns, k = 2..n3m
// (the k = 1 line of the reference is overwritten by solq3k and skipped)
__global__ void k_tri_y3(Dev d, SubDev s) {
    FB_GRID_WAIT();
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 2;
    if (k > d.n3m) return;
    double *b = d.rhs3 + fidx(d, 1, k);
    for (int j = 1; j <= d.n2m; ++j) b[j - 1] = b[j - 1] * s.by3[j];
    gtts2(s.y3, 0, b, 1);
}

// solve_fluid.F90:233-312 (solq3k): w, z lines of n3 unknowns with
// Dirichlet end rows, q3 += x, outflow row advanced by dqb3n
__global__ void k_tri_z3(Dev d, SubDev s) {
    FB_GRID_WAIT();
    const int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (j > d.n2m) return;
    double *b = d.rhs3 + fidx(d, j, 1);
    const size_t P = static_cast<size_t>(d.P);
    b[0] = d.dqb3s[j];
    for (int k = 2; k <= d.n3m; ++k) b[(k - 1) * P] = b[(k - 1) * P] * s.bz3[k];
    b[(d.n3 - 1) * P] = d.dqb3n[j];
    gtts2(s.z3, 0, b, P);
    for (int k = 1; k <= d.n3m; ++k) Fv(d.q3, j, k) = Fv(d.q3, j, k) + b[(k - 1) * P];
    Fv(d.q3, j, d.n3) = Fv(d.q3, j, d.n3) + d.dqb3n[j];
}

// ------------------------------------------------------------ Poisson

// divergence.F90:88-115 (divg)
// Blocks of 32 x 8 threads over 32 x (8 kDivK) cells: thread (x, y) takes j0 + x
// and the rows k0 + y + 8 i.  rmax (may be null): the maxima of |dph| over
// each row j (the rows of the INT8 transform's data operand) are accumulated
// into rmax[j - 1], one atomic per block and row, for the digit cut that follows
// extra (kernels.h): the grid has one row of blocks more (the first, so that it
// is not the grid's tail), whose first block
// runs boucqt (iobcs.F90:81-108; helsolve has used the increments, and nothing
// reads the boundary values before the next nl_rhs) and publishes the CFL number
// with the fixed-dt check of fluid_tsch.F90:49-55.
constexpr int kDivK = 4;
__device__ __forceinline__ void divg_extra(const Dev &d, int extra) {
    const int t = threadIdx.x + blockDim.x * threadIdx.y, nt = blockDim.x * blockDim.y;
    if (extra & kDivBoucqt)
        for (int j = t + 1; j <= d.n2m; j += nt) {
            const double a = d.qb2s[j] + d.dqb2s[j], b = d.qb3s[j] + d.dqb3s[j];
            const double e = d.qb2n[j] + d.dqb2n[j], f = d.qb3n[j] + d.dqb3n[j];
            d.qb2s[j] = a;   // (every load before the first store, which could alias them)
            d.qb3s[j] = b;
            d.qb2n[j] = e;
            d.qb3n[j] = f;
        }
    if ((extra & kDivCfl) && t == 0) {
        const double am = d.scal[S_CFLNEXT], cflm = am * d.dt;
        d.scal[S_CFLM] = cflm;
        d.scal[S_CFLRAW] = am;
        d.scal[S_Q3AVG] = d.scal[S_Q3NEXT];
        if (!(cflm <= d.cfllim)) raise_status(d, FB_ERR_CFL);
    }
}
__device__ __forceinline__ void divg_body(const Dev &d, double usdtal, double *rmax, int extra) {
    int by = blockIdx.y;
    if (extra && by-- == 0) {
        if (blockIdx.x == 0) divg_extra(d, extra);
        return;
    }
    const int jc = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int kb = by * blockDim.y * kDivK + threadIdx.y + 1;
    double m = 0.0;
    if (jc <= d.n2m) {
#pragma unroll
        for (int i = 0; i < kDivK; ++i) {
            const int kc = kb + static_cast<int>(blockDim.y) * i;
            if (kc > d.n3m) break;
            const double dqcap = (Fv(d.q2, jc + 1, kc) - Fv(d.q2, jc, kc)) * d.udx2m[jc] +
                                 (Fv(d.q3, jc, kc + 1) - Fv(d.q3, jc, kc)) * d.udx3m[kc];
            const double v = dqcap * usdtal;
            Fv(d.dph, jc, kc) = v;
            m = fmax(m, fabs(v));   // fmax drops a NaN, as the cut's maximum does
        }
    }
    if (!rmax) return;
    __shared__ double part[8][32];
    part[threadIdx.y][threadIdx.x] = m;
    __syncthreads();
    if (threadIdx.y == 0 && jc <= d.n2m) {
        for (int q = 1; q < 8; ++q) m = fmax(m, part[q][threadIdx.x]);
        if (m > 0.0) atomic_max_nonneg(rmax + jc - 1, m);
    }
}

__global__ void k_divg(Dev d, double usdtal, double *rmax, int extra) {
    FB_GRID_WAIT();
    divg_body(d, usdtal, rmax, extra);
}

// updvp.F90:5-59 (updvp) fused with updvp.F90:68-105 (prcalc) and the
// partial sums of pr_submean (updvp.F90:320-333).  Tiles of kNlJ x kNlK cells
// as in nl_rhs: dph with its halo in shared memory; the block partial sums
// of the pressure mean are finished by the case's last block.
struct UpTile {
    double dph[kNlK + 2][kNlS];   // dph tile + one-cell halo (rows k0-1.., cols j0-1..)
    double kc[6][kNlK];           // udx3c, apphk, acphk, amphk, zz(k), zz(k+1) at rows k0..
    double jc[6][kNlJ];           // udx2c, apphj, acphj, amphj, rc(j), rc(j+1) at columns j0..
};
constexpr size_t kUpSmem = 2 * sizeof(UpTile);
constexpr int kUpBlocksPerSM = 3;

// the TMA-staged form: the dph box of kNlTH x kNlTW (column c holds j = j0 - 2 + c)
struct alignas(128) UpTileT {
    alignas(128) double dph[kNlTH][kNlTW];
    double kc[6][kNlK];
    double jc[6][kNlJ];
};
constexpr size_t kUpSmemT = 2 * sizeof(UpTileT) + 128 + 128;   // tiles, two mbarriers, alignment slack

// the dph box of a tile, issued by one thread (see nl_issue_tma)
__device__ __forceinline__ void up_issue_tma(const NlMaps &m, UpTileT &t, uint32_t bar, int tile, int ntj) {
    const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(bar, kNlBoxBytes);
    tma_load_2d(smem_u32(&t.dph[0][0]), &m.dph, bar, j0 - 3, k0 - 1);
}

// the tile's coefficient vectors (cp.async) and the commit of the thread's group
template <class Tile>
__device__ __forceinline__ void up_prefetch_coef(const Dev &d, Tile &t, int j0, int k0, int tid) {
    if (tid < kNlK) {
        const int k = min(k0 + tid, d.n3m);
        cp8(&t.kc[0][tid], d.udx3c + k);
        cp8(&t.kc[1][tid], d.apphk + k);
        cp8(&t.kc[2][tid], d.acphk + k);
        cp8(&t.kc[3][tid], d.amphk + k);
        cp8(&t.kc[4][tid], d.zz + k);
        cp8(&t.kc[5][tid], d.zz + k + 1);
    } else if (tid < kNlK + kNlJ) {
        const int c = tid - kNlK, j = min(j0 + c, d.n2m);
        cp8(&t.jc[0][c], d.udx2c + j);
        cp8(&t.jc[1][c], d.apphj + j);
        cp8(&t.jc[2][c], d.acphj + j);
        cp8(&t.jc[3][c], d.amphj + j);
        cp8(&t.jc[4][c], d.rc + j);
        cp8(&t.jc[5][c], d.rc + j + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void up_prefetch(const Dev &d, UpTile &t, int tile, int ntj, int tid) {
    const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
    constexpr int kW = kNlJ + 2, kH = kNlK + 2;
    for (int e = tid; e < kW * kH; e += 256) {
        const int r = e / kW, c = e % kW;
        const int j = j0 - 1 + c, k = k0 - 1 + r;
        if (j >= 1 && j <= d.n2 && k >= 0 && k <= d.n3) cp8(&t.dph[r][c], d.dph + fidx(d, j, k));
        else t.dph[r][c] = 0.0;
    }
    up_prefetch_coef(d, t, j0, k0, tid);
}

// q2, q3, pr at this thread's cells of a tile, read before any is written
__device__ __forceinline__ void up_own(const Dev &d, int tile, int ntj, double (&q2)[kNlK / 8], double (&q3)[kNlK / 8],
                                       double (&pr)[kNlK / 8]) {
    const int jc = 1 + (tile % ntj) * kNlJ + threadIdx.x, k0 = 1 + (tile / ntj) * kNlK;
#pragma unroll
    for (int i = 0; i < kNlK / 8; ++i) {
        const int kc = k0 + threadIdx.y + 8 * i;
        const bool ok = jc <= d.n2m && kc <= d.n3m;
        const size_t x = fidx(d, min(jc, d.n2m), min(kc, d.n3m));
        q2[i] = ok ? d.q2[x] : 0.0;
        q3[i] = ok ? d.q3[x] : 0.0;
        pr[i] = ok ? d.pr[x] : 0.0;
    }
}

// pend: as for nl_rhs, pr - pravg of the previous substep is the pressure
// this update starts from (read before this grid's last block stores the new
// mean).  kTma: the dph tiles are TMA boxes on the mbarriers bars (maps m);
// a wait that gives up records FB_ERR_TIMEOUT and ends the block's tiles (the
// block still takes part in the mean)
// (kTma: the single-case kernel; it waits here for the kernel before it, the
// transform that writes dph, with everything but dph of its first tile loaded)
template <bool kTma, class Tile>
__device__ __forceinline__ void updvp_prcalc_body(const Dev &d, double al, double be, Tile *buf, bool pend, int slot,
                                                  const NlMaps *m = nullptr, uint64_t *bars = nullptr) {
    __shared__ double sh[32];
    __shared__ bool last;
    constexpr int kC0 = kTma ? 2 : 1;   // the tile column of j = j0
    const double pravg = pend ? d.scal[S_PRAVG] : 0.0;
    const int ntj = (d.n2m + kNlJ - 1) / kNlJ, ntk = (d.n3m + kNlK - 1) / kNlK, ntiles = ntj * ntk;
    const int t = threadIdx.x + blockDim.x * threadIdx.y, nt = blockDim.x * blockDim.y;
    const int b = blockIdx.x, nb = gridDim.x;
    constexpr int kC = kNlK / 8;
    double part = 0.0;
    int tile = blockIdx.x;
    double q2n[kC], q3n[kC], prn[kC];
    uint32_t bar0 = 0, bar1 = 0;
    if constexpr (kTma) {
        bar0 = smem_u32(bars);
        bar1 = smem_u32(bars + 1);
    }
    if constexpr (kTma) {
        if (tile < ntiles) {
            if (t == 0) {
                mbar_init(bar0, 1);
                mbar_init(bar1, 1);
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            }
            up_prefetch_coef(d, buf[0], 1 + (tile % ntj) * kNlJ, 1 + (tile / ntj) * kNlK, t);
            up_own(d, tile, ntj, q2n, q3n, prn);
        }
        FB_GRID_WAIT();
        if (tile < ntiles && t == 0) up_issue_tma(*m, buf[0], bar0, tile, ntj);
        __syncthreads();   // the barriers are initialised before any thread waits on them
    } else if (tile < ntiles) {
        up_prefetch(d, buf[0], tile, ntj, t);
        up_own(d, tile, ntj, q2n, q3n, prn);
    }
    for (int it = 0; tile < ntiles; ++it, tile += gridDim.x) {
        const Tile &u = buf[it & 1];
        double q2v[kC], q3v[kC], prv[kC];
#pragma unroll
        for (int i = 0; i < kC; ++i) {
            q2v[i] = q2n[i];
            q3v[i] = q3n[i];
            prv[i] = prn[i];
        }
        const int nxt = tile + gridDim.x;
        if (nxt < ntiles) {
            if constexpr (kTma) {
                if (t == 0) up_issue_tma(*m, buf[(it + 1) & 1], (it & 1) ? bar0 : bar1, nxt, ntj);
                up_prefetch_coef(d, buf[(it + 1) & 1], 1 + (nxt % ntj) * kNlJ, 1 + (nxt / ntj) * kNlK, t);
            } else {
                up_prefetch(d, buf[(it + 1) & 1], nxt, ntj, t);
            }
            up_own(d, nxt, ntj, q2n, q3n, prn);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        if constexpr (kTma) {
            const bool landed = mbar_wait((it & 1) ? bar1 : bar0, static_cast<uint32_t>(it >> 1) & 1u);
            if (__syncthreads_or(!landed)) {
                if (t == 0) atomicCAS(d.status, 0, FB_ERR_TIMEOUT);
                break;
            }
        } else {
            __syncthreads();
        }
        const int j0 = 1 + (tile % ntj) * kNlJ, k0 = 1 + (tile / ntj) * kNlK;
        const int jc = j0 + threadIdx.x;
#define TD(j, k) u.dph[(k) - k0 + 1][(j) - j0 + kC0]
        if (jc <= d.n2m) {
            const int cj = jc - j0;
            const int jm = jmv_(jc), jp = jpv_(d, jc);
            const double usujm = al * d.dt * u.jc[0][cj];
            const double apj = u.jc[1][cj], acj = u.jc[2][cj], amj = u.jc[3][cj];
            const double dyc = u.jc[5][cj] - u.jc[4][cj];
#pragma unroll
            for (int i = 0; i < kC; ++i) {
                const int kc = k0 + threadIdx.y + 8 * i;
                if (kc > d.n3m) break;
                const int r = kc - k0;
                const double locdph = TD(jc, kc);
                Fv(d.q2, jc, kc) = q2v[i] - (locdph - TD(jm, kc)) * usujm;
                if (kc >= 2) {
                    const double usukm = al * d.dt * u.kc[0][r];
                    Fv(d.q3, jc, kc) = q3v[i] - (TD(jc, kc) - TD(jc, kc - 1)) * usukm;
                }
                const int kp = kpv_(d, kc), km = kmv_(kc);
                const double pr0 = pend ? prv[i] - pravg : prv[i];
                const double p = pr0 + TD(jc, kc) -
                                 be * ((TD(jp, kc) * apj + TD(jc, kc) * acj + TD(jm, kc) * amj) +
                                       (TD(jc, kp) * u.kc[1][r] + TD(jc, kc) * u.kc[2][r] + TD(jc, km) * u.kc[3][r]));
                Fv(d.pr, jc, kc) = p;
                part = part + p * (u.kc[5][r] - u.kc[4][r]) * dyc;
            }
        }
#undef TD
        __syncthreads();   // this buffer is refilled two tiles on
    }
    const double bsum = block_reduce_fast<false>(part, sh);
    double *red = d.red + 2 * static_cast<size_t>(kRedSlot);
    if (t == 0) {
        red[b] = bsum;
        __threadfence();
        last = (atomicAdd(d.count + 2, 1u) == static_cast<unsigned>(nb - 1));
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double acc = 0.0;
    for (int i = t; i < nb; i += nt) acc = acc + __ldcg(red + i);
    acc = block_reduce_fast<false>(acc, sh);
    if (t == 0) {
        d.count[2] = 0u;
        const double avg = acc / (d.rext2 * d.alx3);
        d.scal[S_PRAVG] = avg;
        if (slot >= 0) d.scal[slot] = avg;
    }
}

__global__ void __launch_bounds__(256, kUpBlocksPerSM)
    k_updvp_prcalc_tma(const __grid_constant__ Dev d, const __grid_constant__ NlMaps m, double al, double be,
                       int pend, int slot) {
    extern __shared__ __align__(16) unsigned char up_smem[];
    const uint32_t raw = smem_u32(up_smem);
    unsigned char *base = up_smem + ((128u - (raw & 127u)) & 127u);   // the tiles on 128-byte boundaries
    updvp_prcalc_body<true>(d, al, be, reinterpret_cast<UpTileT *>(base), pend != 0, slot, &m,
                            reinterpret_cast<uint64_t *>(base + 2 * sizeof(UpTileT)));
}

// pr_submean (updvp.F90:336: the whole array) and boucqt (iobcs.F90:97-105)
// deferred: the means of RK3 substeps 1 and 2 were applied to the cells that
// updvp rewrites (j <= n2m, 1 <= k <= n3m) as it read them; the other
// entries of the array get all three subtractions here, in order.  boucqt has
// then run with divg.
__device__ __forceinline__ void submean_boucqt_body(const Dev &d, bool deferred = false) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int k = blockIdx.y * blockDim.y + threadIdx.y;
    const double pravg = d.scal[S_PRAVG];
    if (j <= d.n2 && k <= d.n3) {
        double p = Fv(d.pr, j, k);
        if (deferred && (j > d.n2m || k < 1 || k > d.n3m)) p = (p - d.scal[S_PRAVG1]) - d.scal[S_PRAVG2];
        Fv(d.pr, j, k) = p - pravg;
    }
    if (!deferred && blockIdx.y == 0 && threadIdx.y == 0 && j <= d.n2m) {
        d.qb2s[j] = d.qb2s[j] + d.dqb2s[j];
        d.qb3s[j] = d.qb3s[j] + d.dqb3s[j];
        d.qb2n[j] = d.qb2n[j] + d.dqb2n[j];
        d.qb3n[j] = d.qb3n[j] + d.dqb3n[j];
    }
}

__global__ void k_submean_boucqt(Dev d, int deferred) {
    FB_GRID_WAIT();
    submean_boucqt_body(d, deferred != 0);
}

// ------------------------------------------------------------ loads

// loads_transfer_c (loads_transfer.F90:143-185), per-marker part: the probe
// interpolation of v, w or p with first and second derivatives; the v and w
// groups also form checkbcs (ckbcs.F90:29-60) with the substep-1 weights.
// One (marker, quantity) per group of kLoadLanes lanes, support node m on
// lane m < kSD: the nodes' weights, moment terms and field reads are
// independent, and every sum over the nodes is formed in node order
// (group_sums), so each result is that of the sequential loops.  Every lane of
// a warp reaches every exchange: a group that stops (outside the channel, an
// error) carries on with its loads and stores switched off.
constexpr int kLoadLanes = kNodeLanes;
constexpr int kLoadMk = 2;   // markers per block: the three groups of a marker in one block
constexpr int kLoadThreads = 3 * kLoadMk * kLoadLanes;

// pend: the step's last pressure mean is still to be subtracted from pr (in row
// k = 0, which a probe beside the inflow reads, all three of them); the value is
// the one pr_submean would have stored.
// vals (may be null): the block's markers' values in shared memory, 24 each
template <bool kWait>
__device__ __forceinline__ void loads_probe_body(const Dev &d, bool pend, double *vals) {
    constexpr unsigned kAll = 0xffffffffu;
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    const int T = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = T / kLoadLanes, m = T % kLoadLanes;
    const int base = (threadIdx.x & 31) & ~(kLoadLanes - 1);
    __shared__ double bufs[3 * kLoadMk][10 * 18];
    double *buf = bufs[threadIdx.x / kLoadLanes];
    const bool have = t < 3 * d.nlm;
    const int tt = have ? t : 0;
    const int n = tt / 3, idir = tt % 3 + 1;
    const bool node = m < kSD;
    double *pb = d.probe + static_cast<size_t>(n) * 24;
    const double pos[2] = {d.lmcc[2 * n], d.lmcc[2 * n + 1]};
    const bool inside = (d.zz[1] < pos[1] && pos[1] < d.zz[d.n3]);
    // (an early look at the status: without a set-up of this step there are no
    // support nodes to read; the one behind the wait decides what is stored)
    const bool early = __shfl_sync(kAll, static_cast<int>(*d.status != 0), base) != 0;
    const bool live = have && inside && !early;

    const double hpr = d.ddmin * d.kprobe;
    const double probe[2] = {pos[0] + d.lmnor[2 * n] * hpr, pos[1] + d.lmnor[2 * n + 1] * hpr};
    int mj, mk;
    if (idir == 3) {
        mj = d.lmind[4 * n + 2];
        mk = d.lmind[4 * n + 1];
    } else {
        mj = d.lmind[4 * n + 2 * (idir - 1)];
        mk = d.lmind[4 * n + 2 * (idir - 1) + 1];
    }

    // probeind (loads_transfer.F90:238-281): the nearest y and z lines to the
    // probe within 5 lines of the marker's own; lane i holds lines js + i, ks + i
    constexpr int off = 5;
    const int js = mj - off, ks = mk - off;
    const bool inrange = live && js >= 1 && mj + off <= d.n2 && ks >= 1 && mk + off <= d.n3;
    const double *ya = (idir == 1) ? d.rc : d.rm;
    const double *za = (idir == 2) ? d.zz : d.zm;
    double vy = inf, vz = inf;
    if (inrange && m <= 2 * off) {
        vy = fabs(ya[js + m] - probe[0]);
        vz = fabs(za[ks + m] - probe[1]);
    }
    // a NaN distance never wins the strict comparison; one at the first line
    // keeps the first line
    const bool y0nan = isnan(__shfl_sync(kAll, vy, base)), z0nan = isnan(__shfl_sync(kAll, vz, base));
    const int iy = group_argmin(isnan(vy) ? inf : vy, m);
    const int iz = group_argmin(isnan(vz) ? inf : vz, m);
    const int ij = js + (y0nan ? 0 : iy), ik = ks + (z0nan ? 0 : iz);

    // MLS_SD_ind (MLSint.F90:4-104): node m = 3 (j - 1) + (k - 1) of the 3 x 3
    // support, moved inside the field
    const double *y, *z;
    int dimy, dimz;
    sd_axes(d, idir, y, dimy, z, dimz);
    const int sj = (ij == 1) ? 1 : (ij == d.n2m ? -1 : 0);
    const int sk = (ik == 1) ? 1 : (ik == d.n3m ? -1 : 0);
    const int mm = node ? m : 0;
    const int ej = ij + (mm / 3 + 1 + sj) - 2, ek = ik + (mm % 3 + 1 + sk) - 2;
    const bool bad = inrange && node && (ej < 1 || ej + 1 > dimy || ek < 1 || ek + 1 > dimz);
    const bool supported = group_none(bad, base) && inrange;
    const int ej0 = __shfl_sync(kAll, ej, base);
    const bool found = supported && ej0 >= 2, act = found && node;

    // MLS_SF_d (MLSint.F90:173-258) with compute_AB_d (:342-402)
    double sc0 = 0.0, sc1 = 0.0, w0 = 0.0, w1 = 0.0, w2 = 0.0;
    if (act) {
        sc0 = y[ej];
        sc1 = z[ek];
        const double sd0 = y[ej + 1] - y[ej], sd1 = z[ek + 1] - z[ek];
        double wc[2], dw[2];
        wkernel(d.wfun, probe[0] - sc0, d.radiusSD * sd0, wc[0], dw[0]);
        wkernel(d.wfun, probe[1] - sc1, d.radiusSD * sd1, wc[1], dw[1]);
        w0 = wc[0] * wc[1];
        w1 = wc[1] * dw[0];
        w2 = wc[0] * dw[1];
    }
    const double pk[3] = {1.0, sc0, sc1};
    // the moments of the weights and of their two derivatives; pk[a] pk[b] =
    // pk[b] pk[a]: the same terms, the same sums
    double mom[18];
    int q = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a; b < 3; ++b) {
            const double pp = pk[a] * pk[b];
            mom[q] = w0 * pp;
            mom[6 + q] = w1 * pp;
            mom[12 + q] = w2 * pp;
            ++q;
        }
    group_sums<18>(mom, m, buf);
    const double Aa[3][3] = {{mom[0], mom[1], mom[2]}, {mom[1], mom[3], mom[4]}, {mom[2], mom[4], mom[5]}};
    GeLu lu;
    ge_factor(Aa, lu);
    double gam[3][3];
    const double gps[3] = {1.0, probe[0], probe[1]};
    double g0[3];
    ge_apply(lu, gps, g0);
    {
        // the two derivatives' systems on the group's two halves
        const int l = (m < kNodeLanes / 2) ? 1 : 2;
        const double *ml = buf + 18 * kSD + 6 * l;   // (the sums, where group_sums left them)
        const double Al[3][3] = {{ml[0], ml[1], ml[2]}, {ml[1], ml[3], ml[4]}, {ml[2], ml[4], ml[5]}};
        double C[3], gx[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            double acc = 0.0;
#pragma unroll
            for (int b = 0; b < 3; ++b) acc = acc + Al[a][b] * g0[b];
            const double gpl = (a == l) ? 1.0 : 0.0;
            C[a] = gpl - acc;
        }
        ge_apply(lu, C, gx);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            gam[a][0] = g0[a];
            gam[a][1] = __shfl_sync(kAll, gx[a], base);
            gam[a][2] = __shfl_sync(kAll, gx[a], base + kNodeLanes / 2);
        }
    }
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double B0 = pk[a] * w0, B1 = pk[a] * w1, B2 = pk[a] * w2;
        p0 = p0 + gam[a][0] * B0;
        p1 = p1 + gam[a][1] * B0 + gam[a][0] * B1;
        p2 = p2 + gam[a][2] * B0 + gam[a][0] * B2;
    }
    // All of the above depends on the markers alone: kWait waits only here for
    // the kernel before it (updvp or pr_submean, which write q2, q3 and pr, or the
    // launch that sums the loads of the probes before)
    if (kWait) FB_GRID_WAIT();
    const int status = __ldcg(d.status);
    // checkbcs: the velocity at the marker from the substep-1 weights
    double prod = 0.0;
    if (live && idir <= 2 && node) {
        const int t2 = 2 * n + idir - 1;
        const int *eu = d.eulins + static_cast<size_t>(t2) * 2 * kSD;
        const double *q = (idir == 1) ? d.q2 : d.q3;
        prod = d.phi[static_cast<size_t>(t2) * kSD + m] * q[fidx(d, eu[m], eu[kSD + m])];
    }
    double f0 = 0.0, fym = 0.0, fzm = 0.0, g2r = 1.0, g3r = 1.0;
    if (act) {
        const double *f = (idir == 1) ? d.q2 : (idir == 2 ? d.q3 : d.pr);
        const bool late = pend && idir == 3;
        const double mean = late ? d.scal[S_PRAVG] : 0.0;   // (x - 0.0 is x)
        f0 = Fv(f, ej, ek) - mean;
        fym = Fv(f, ej - 1, ek) - mean;   // (ej >= 2)
        double fk = Fv(f, ej, ek - 1);
        if (late && ek == 1) fk = (fk - d.scal[S_PRAVG1]) - d.scal[S_PRAVG2];   // row 0: no updvp has rewritten it
        fzm = fk - mean;
        g2r = d.g2rc[ej];
        g3r = d.g3rc[ek];
    }
    const bool stopped = __shfl_sync(kAll, static_cast<int>(status != 0), base) != 0;
    const bool ok = live && !stopped, good = found && !stopped;
    if (have && m == 0) {
        if (idir == 1) {
            pb[23] = inside ? 0.0 : -1.0;
            if (vals) vals[24 * (threadIdx.x / (3 * kLoadLanes)) + 23] = inside ? 0.0 : -1.0;
            d.bcerrv[n] = 0.0;
        }
        if (idir == 2) d.bcerrw[n] = 0.0;
        if (ok && !good) raise_status(d, FB_ERR_MARKER_OUT);
    }
    // getpbup (loads_transfer.F90:285-357) for this quantity; the last two: the
    // partition of unity and checkbcs's velocity
    double o[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, p0, prod};
    if (act) {
        const double uk1 = (f0 - fym) * d.dx2 / g2r;
        const double uk2 = (f0 - fzm) * d.dx3 / g3r;
        o[0] = p0 * f0;
        o[1] = p1 * f0;
        o[2] = p2 * f0;
        o[3] = p1 * uk1;
        o[4] = p1 * uk2;
        o[5] = p2 * uk1;
        o[6] = p2 * uk2;
    }
    group_sums<9>(o, m, buf);
    if (good && m == 0 && !(fabs(1.0 - fabs(o[7])) <= 1.0e-10)) raise_status(d, FB_ERR_MLS);
    if (ok && idir <= 2 && m == 0) {
        if (idir == 1) d.bcerrv[n] = d.lmvel[2 * n] - o[8];
        else d.bcerrw[n] = d.lmvel[2 * n + 1] - o[8];
    }
    const double res = buf[9 * kSD + min(m, 8)];   // sum m
    if (good && m < 7) {
        pb[7 * (idir - 1) + m] = res;
        if (vals) vals[24 * (threadIdx.x / (3 * kLoadLanes)) + 7 * (idir - 1) + m] = res;
    }
}

// loads_transfer.F90:187-214 for marker n with probe values pb (ucy, ucz, pc of
// seven each) and tangent (tany, tanz): pressure extrapolation (Wang et al.
// 2019 eq. 20) and wall shear (eq. 26)
__device__ __forceinline__ void finish_marker(const Dev &d, int n, const double *pb, double tany, double tanz,
                                              double &press, double (&tau)[2]) {
    const double hpr = d.ddmin * d.kprobe, visc = d.visc;
    const double *ucy = pb, *ucz = pb + 7, *pc = pb + 14;
    const double nory = d.lmnor[2 * n], norz = d.lmnor[2 * n + 1];
    double dpdnw = d.lmacc[2 * n] * nory + d.lmacc[2 * n + 1] * norz;
    dpdnw = -1.0 * dpdnw;
    const double dpdne = pc[1] * nory + pc[2] * norz;
    press = pc[0] - 0.5 * (dpdnw + dpdne) * hpr;
    const double ducdn = (ucy[1] * tany * nory + ucy[2] * tany * norz + ucz[1] * tanz * nory +
                          ucz[2] * tanz * norz);
    const double d3ucdn3 = (pc[3] * nory * nory + pc[4] * nory * norz + pc[5] * norz * nory +
                            pc[6] * norz * norz) * 1.0 / visc;
    const double d2ucdn2 = (ucy[3] * tany * nory * nory + ucy[4] * tany * nory * norz +
                            ucy[5] * tany * norz * nory + ucy[6] * tany * norz * norz +
                            ucz[3] * tanz * nory * nory + ucz[4] * tanz * nory * norz +
                            ucz[5] * tanz * norz * nory + ucz[6] * tanz * norz * norz);
    const double ducdnm = ducdn - d2ucdn2 * hpr - 0.5 * d3ucdn3 * (hpr * hpr);
    tau[0] = visc * ducdnm * tany;
    tau[1] = visc * ducdnm * tanz;
}

// the tangent of the last marker up to n that has one of its own (zero if none)
__device__ __forceinline__ void carried_tangent(const Dev &d, int n, double &tany, double &tanz) {
    for (int m = n; m >= 0; --m) {
        const double *pm = d.probe + static_cast<size_t>(m) * 24;
        if (pm[23] > 0.5) {
            tany = pm[21];
            tanz = pm[22];
            return;
        }
    }
}

// the probes of kLoadMk markers per block, then each probed marker's own
// tangent (loads_transfer.F90:177-185) from its first two probes.  kFinish: a
// marker with a tangent of its own is finished here (press, tau), one outside
// the channel gets zeros, and only those whose tangent carries over from
// another marker are left to the launch that sums the loads.  The values go to
// d.lfin: only that launch knows that no probe has failed.
template <bool kFinish, bool kWait>
__device__ __forceinline__ void loads_probe_tan_body(const Dev &d, bool pend) {
    if (!d.nlm) return;
    __shared__ double vals[kLoadMk][24];
    loads_probe_body<kWait>(d, pend, kFinish ? &vals[0][0] : nullptr);
    __syncthreads();
    const int T = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = T / kLoadLanes;
    if (t >= 3 * d.nlm || t % 3 != 0 || T % kLoadLanes != 0 || *d.status) return;
    const int n = t / 3;
    double *pb = d.probe + static_cast<size_t>(n) * 24;
    const double *pv = kFinish ? vals[threadIdx.x / (3 * kLoadLanes)] : pb;
    double press = 0.0, tau[2] = {0.0, 0.0};
    bool done = true;
    if (pv[23] >= 0.0) {
        const double nory = d.lmnor[2 * n], norz = d.lmnor[2 * n + 1];
        const double vel0 = pv[0], vel1 = pv[7];
        const double veln_md = vel0 * nory + vel1 * norz;
        const double velt0 = vel0 - veln_md * nory, velt1 = vel1 - veln_md * norz;
        const double velt_md = sqrt(velt0 * velt0 + velt1 * velt1);
        if (velt_md != 0.0) {
            const double tany = velt0 / velt_md, tanz = velt1 / velt_md;
            pb[21] = tany;
            pb[22] = tanz;
            pb[23] = 1.0;
            if (kFinish) finish_marker(d, n, pv, tany, tanz, press, tau);
        } else {
            pb[23] = 0.0;
            done = false;
        }
    }
    if (kFinish && done) {
        d.lfin[3 * n] = press;
        d.lfin[3 * n + 1] = tau[0];
        d.lfin[3 * n + 2] = tau[1];
    }
}

template <bool kFinish>
__global__ void __launch_bounds__(kLoadThreads, 5) k_loads_probe(Dev d, int pend) {
    loads_probe_tan_body<kFinish, true>(d, pend != 0);
}

// loads_transfer_c (loads_transfer.F90:187-214): the tangent carries over
// from the previous marker when the probe's tangential velocity vanishes;
// pressure extrapolation (Wang et al. 2019 eq. 20) and wall shear (eq. 26).
// Also the L2 norms of checkbcs (ckbcs.F90:76-81).  Single block.
__device__ __forceinline__ void loads_finish_body(const Dev &d) {
    __shared__ double sh[32];
    __shared__ bool last;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    double sv = 0.0, sw = 0.0;
    if (n < d.nlm) {
        const double *pb = d.probe + static_cast<size_t>(n) * 24;
        if (*d.status == 0) {
            double press = 0.0, tau[2] = {0.0, 0.0};
            if (pb[23] >= 0.0) {
                double tany = 0.0, tanz = 0.0;
                carried_tangent(d, n, tany, tanz);
                finish_marker(d, n, pb, tany, tanz, press, tau);
            }
            d.press[n] = press;
            d.tau[2 * n] = tau[0];
            d.tau[2 * n + 1] = tau[1];
        }
        sv = d.bcerrv[n] * d.bcerrv[n];
        sw = d.bcerrw[n] * d.bcerrw[n];
    }
    // the L2 norms of checkbcs (ckbcs.F90:76-81): block partials, summed in
    // block order by the last block
    const double tv = block_reduce_fast<false>(sv, sh);
    const double tw = block_reduce_fast<false>(sw, sh);
    const int b = blockIdx.x, nb = gridDim.x;
    double *rv = d.red, *rw = d.red + kRedSlot;
    if (threadIdx.x == 0) {
        rv[b] = tv;
        rw[b] = tw;
        __threadfence();
        last = (atomicAdd(d.count + 1, 1u) == static_cast<unsigned>(nb - 1));
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double av = 0.0, aw = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        av = av + __ldcg(rv + i);
        aw = aw + __ldcg(rw + i);
    }
    av = block_reduce_fast<false>(av, sh);
    aw = block_reduce_fast<false>(aw, sh);
    if (threadIdx.x == 0) {
        d.count[1] = 0u;
        d.scal[S_NBCV] = sqrt(av) / static_cast<double>(d.nlm);
        d.scal[S_NBCW] = sqrt(aw) / static_cast<double>(d.nlm);
    }
}

constexpr int kLoadFin = 128;   // markers per block of the finish
__global__ void __launch_bounds__(kLoadFin) k_loads_finish(Dev d) {
    FB_GRID_WAIT();
    loads_finish_body(d);
}

// ------------------------------------------------------------ rigid body

// rigid.F90:341-369 (modfn) for the uncoupled 3-DOF system
__device__ void modfn(double K[6], const double t[6], const double FF[6], const double Mi[3], const Dev &d) {
    for (int i = 0; i < 3; ++i) {
        const double cube = t[i] * t[i] * t[i];
        const double lin = -d.kk[i] * t[i] + -d.cc[i] * t[i + 3];
        const double rhs = lin + -d.kk3[i] * cube + FF[i + 3];
        K[i] = t[i + 3];
        K[i + 3] = Mi[i] * rhs;
    }
}

// explicit RK4 (kinem_RK4) with loads frozen over the stages: the three degrees
// of freedom i (y, z, rotation) are independent (modfn); xns[i], xns[3 + i] are
// the new displacement and velocity
__device__ __forceinline__ void rigid_rk4(const Dev &d, int i, const double *rs, double Fy, double Fz, double M,
                                          double *xns) {
    const double dt = d.dt;
    const double csp = (i == 0) ? d.cmposi0 : (i == 1 ? d.cmposi1 : d.cmroti);
    double FFi, Mii;
    if (i == 0) {
        if (d.rtcoup) {
            FFi = Fy + M / d.rrr;
            Mii = 1.0 / ((d.rba1 / (d.rrr * d.rrr) + d.rba0) * d.rbden);
        } else {
            FFi = Fy;
            Mii = 1.0 / (d.rba0 * d.rbden);
        }
    } else if (i == 1) {
        FFi = Fz;
        Mii = 1.0 / (d.rba0 * d.rbden);
    } else {
        FFi = M;
        Mii = 1.0 / (d.rba1 * d.rbden);
    }
    const double kk = d.kk[i], cc = d.cc[i], kk3 = d.kk3[i];
    // modfn (rigid.F90) for component i: K_x = v, K_v = Mi (-kk x + -cc v + -kk3 x^3 + F)
    auto mod = [&](double x, double v, double &kx, double &kv) {
        const double cube = x * x * x;
        const double lin = -kk * x + -cc * v;
        const double rhs = lin + -kk3 * cube + FFi;
        kx = v;
        kv = Mii * rhs;
    };
    const double xo = rs[i] - csp, vo = rs[3 + i];
    double k1x, k1v, k2x, k2v, k3x, k3v, k4x, k4v;
    mod(xo, vo, k1x, k1v);
    mod(xo + k1x * dt / 2.0, vo + k1v * dt / 2.0, k2x, k2v);
    mod(xo + k2x * dt / 2.0, vo + k2v * dt / 2.0, k3x, k3v);
    mod(xo + k3x * dt, vo + k3v * dt, k4x, k4v);
    xns[i] = xo + dt * (k1x / 6.0 + k2x / 3.0 + k3x / 3.0 + k4x / 6.0);
    xns[3 + i] = vo + dt * (k1v / 6.0 + k2v / 3.0 + k3v / 3.0 + k4v / 6.0);
}

// the body's state cm[0..17] (rigid layout) after the RK4 update xn, and the
// rotation matrix of the step (get_rotmat); one thread
__device__ __forceinline__ void rigid_state(const Dev &d, const double *rs, const double *xns, const double *kin,
                                            const int *mcon, double *cm, double *rot) {
    const double dt = d.dt;
    const double csp[3] = {d.cmposi0, d.cmposi1, d.cmroti};
    double xn[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) xn[i] = xns[i];
    // P1, V1, A1 (rigid[9..17]) formed in shared memory (cm)
    for (int i = 0; i < 18; ++i) cm[i] = rs[i];
    double *P1 = cm + 9, *V1 = cm + 12, *A1 = cm + 15;
    if (!d.rtcoup) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            P1[i] = csp[i] + xn[i];
            V1[i] = xn[3 + i];
            A1[i] = (V1[i] - rs[3 + i]) / dt;
        }
    } else {
        P1[0] = csp[0] + xn[0];
        V1[0] = xn[3];
        A1[0] = (V1[0] - rs[3]) / dt;
        P1[1] = csp[1];
        V1[1] = 0.0;
        A1[1] = 0.0;
        P1[2] = csp[2] + xn[0] / d.rrr;
        V1[2] = V1[0] / d.rrr;
        A1[2] = A1[2] / d.rrr;  // as rigid.F90:296 (incoming value / rr)
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (mcon[i] == 1) {
            P1[i] = kin[i];
            V1[i] = kin[3 + i];
            A1[i] = kin[6 + i];
        }
    const double cmrot = P1[2] - rs[2];
    double sn, cs;
    sincos(cmrot, &sn, &cs);
    rot[0] = cs;
    rot[1] = -sn;
    rot[2] = sn;
    rot[3] = cs;
}

// a marker (y, z) carried by the body's motion P0 -> P1 (kinematics of
// rigid.F90:75-108): new position, velocity, acceleration
__device__ __forceinline__ void move_marker(const double *cm, const double *rot, double y, double z, double (&pos)[2],
                                            double (&vel)[2], double (&acc)[2]) {
    const double *P0 = cm, *P1 = cm + 9, *V1 = cm + 12, *A1 = cm + 15;
    const double rho0 = y - P0[0], rho1 = z - P0[1];
    const double c10 = -V1[2] * rho1, c11 = V1[2] * rho0;
    const double c20 = -A1[2] * rho1, c21 = A1[2] * rho0;
    const double c30 = -V1[2] * c11, c31 = V1[2] * c10;
    pos[0] = P1[0] + (rot[0] * rho0 + rot[1] * rho1);
    pos[1] = P1[1] + (rot[2] * rho0 + rot[3] * rho1);
    vel[0] = V1[0] + c10;
    vel[1] = V1[1] + c11;
    acc[0] = A1[0] + c20 + c30;
    acc[1] = A1[1] + c21 + c31;
}

// a vertex rotated about the updated centre (rigid.F90:110-121)
__device__ __forceinline__ void move_vertex(const double *cm, const double *rot, const double *v, double (&o)[2]) {
    const double *P1 = cm + 9;
    const double rho0 = v[0] - P1[0], rho1 = v[1] - P1[1];
    o[0] = P1[0] + (rot[0] * rho0 + rot[1] * rho1);
    o[1] = P1[1] + (rot[2] * rho0 + rot[3] * rho1);
}

// createnorm (rigid.F90:468-495): the normal of the segment a -> b
__device__ __forceinline__ void segment_normal(const double *a, const double *b, double (&nor)[2]) {
    const double v1[3] = {0.0 - 0.0, b[0] - a[0], b[1] - a[1]};
    const double v2[3] = {-1.0 - 0.0, (a[0] + b[0]) * 0.5 - a[0], (a[1] + b[1]) * 0.5 - a[1]};
    const double c0 = v1[1] * v2[2] - v1[2] * v2[1];
    const double c1 = v1[2] * v2[0] - v1[0] * v2[2];
    const double c2 = v1[0] * v2[1] - v1[1] * v2[0];
    const double den = sqrt(c0 * c0 + c1 * c1 + c2 * c2);
    nor[0] = c1 / den;
    nor[1] = c2 / den;
}

// the end of a step (one thread): body state, clock (main.F90:92), history row
__device__ __forceinline__ void commit_step(const Dev &d, int hist_rows, const double *cm, const double (&fv)[8],
                                            double t0, double stepd, double nbcv, double nbcw, double cflm,
                                            double solves) {
    for (int i = 0; i < 9; ++i) d.rigid[i] = cm[9 + i];
    const double t1 = t0 + d.dt;
    d.scal[S_TIME] = t1;
    const int row = static_cast<int>(stepd);
    if (hist_rows > 0) {
        double *h = d.hist + static_cast<size_t>(row % hist_rows) * FB_HIST_COLS;
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = fv[i];
        h[8] = t1;
        for (int i = 0; i < 9; ++i) h[9 + i] = cm[9 + i];
        h[18] = nbcv;
        h[19] = nbcw;
        h[20] = cflm;
        h[21] = d.dt;
        for (int i = 22; i < FB_HIST_COLS; ++i) h[i] = 0.0;  // diagnostics, when enabled
        h[30] = solves;
    }
    d.scal[S_STEP] = static_cast<double>(row + 1);
}

// rigid.F90:4-138 (rigid) with int_stress :373-464, kinem_RK4 :165-228 /
// kinem_RK4i :233-299, get_rotmat :142-161, createnorm :468-495; then the
// clock update of main.F90:92 and one history row.  Single block.
// mode RIGID_STEP: the reference's loose coupling (loads -> forces -> RK4 ->
// markers -> commit).  The strong coupling iteration splits it:
// RIGID_PLACE moves the markers to the state that the load fin[0..2] (Fy,
// Fz, M) gives, without committing; RIGID_FORCES integrates the loads of the
// markers at that new state (moment about the new centre) and evaluates the
// RK4 update they give into rigid[9..17] only; RIGID_COMMIT is RIGID_STEP
// with the load fin (markers restored to the start of the step first).
__device__ __forceinline__ void rigid_body(const Dev &d, int hist_rows, int mode, const double *fin,
                                           double *mbox = nullptr) {
    __shared__ double sh[32 * 5];
    __shared__ double cm[18];
    __shared__ double rot[4];
    __shared__ double xns[6];
    __shared__ double rs[18], kin[9];   // the body state and the prescribed kinematics, read once
    __shared__ int mcon[3];
    const int tid = threadIdx.x, nt = blockDim.x, nlm = d.nlm;
    double *R = d.rigid;
    const bool from_loads = (mode == RIGID_STEP || mode == RIGID_FORCES);
    if (tid < 18) rs[tid] = R[tid];
    else if (tid >= 32 && tid < 41) kin[tid - 32] = d.kinori[tid - 32];
    else if (tid >= 64 && tid < 67) mcon[tid - 64] = d.rbmcon[tid - 64];
    if (!from_loads) __syncthreads();   // (otherwise the block sums' barriers order them)
    double fyp = 0.0, fzp = 0.0, fyv = 0.0, fzv = 0.0, mom = 0.0;
    if (from_loads) {
        const double c0 = (mode == RIGID_FORCES) ? R[9] : R[0], c1 = (mode == RIGID_FORCES) ? R[10] : R[1];
        double f[5] = {0.0, 0.0, 0.0, 0.0, 0.0};   // fyp, fzp, fyv, fzv, mom
        for (int i = tid; i < nlm; i += nt) {
            const double p = d.press[i], A = d.lmA[i];
            const double Fp1 = -p * d.lmnor[2 * i] * A, Fp2 = -p * d.lmnor[2 * i + 1] * A;
            const double Fv1 = d.tau[2 * i] * A, Fv2 = d.tau[2 * i + 1] * A;
            f[0] = f[0] + Fp1;
            f[1] = f[1] + Fp2;
            f[2] = f[2] + Fv1;
            f[3] = f[3] + Fv2;
            const double r1 = d.lmcc[2 * i] - c0, r2 = d.lmcc[2 * i + 1] - c1;
            f[4] = f[4] + (r1 * (Fp2 + Fv2) - r2 * (Fp1 + Fv1));
        }
        block_sum_n<5>(f, sh);   // the five block sums (the same trees as one at a time)
        fyp = f[0];
        fzp = f[1];
        fyv = f[2];
        fzv = f[3];
        mom = f[4];
    }
    // the loads of the step (every thread forms the same values)
    const double time = d.scal[S_TIME];
    double Fy, Fz, M;
    if (from_loads) {
        const double fy = fyp + fyv, fz = fzp + fzv;
        const double g0 = (1.0 - 1.0 / d.rbden) * d.rba0 * d.rbgravF0;
        const double g1 = (1.0 - 1.0 / d.rbden) * d.rba0 * d.rbgravF1;
        Fy = fy + g0;
        Fz = fz + g1;
        M = mom;
    } else {
        Fy = fin[0];
        Fz = fin[1];
        M = fin[2];
    }
    if (tid == 0 && from_loads) {
        d.forces[0] = time;
        d.forces[1] = Fy;
        d.forces[2] = Fz;
        d.forces[3] = M;
        d.forces[4] = fyp;
        d.forces[5] = fzp;
        d.forces[6] = fyv;
        d.forces[7] = fzv;
    }
    if (tid < 3) rigid_rk4(d, tid, rs, Fy, Fz, M, xns);
    __syncthreads();
    if (tid == 0) {
        rigid_state(d, rs, xns, kin, mcon, cm, rot);
        for (int i = 9; i < 18; ++i) R[i] = cm[i];
    }
    __syncthreads();
    if (mode == RIGID_FORCES) return;   // the update the loads give, markers untouched
    // Each loop reads all of a thread's kRgU entries before it stores any: the
    // stores could alias the next loads, so a load after a store would wait
    // for the store's round trip.
    constexpr int kRgU = 4;
    for (int i0 = tid; i0 < nlm; i0 += kRgU * nt) {
        double y[kRgU], z[kRgU];
#pragma unroll
        for (int u = 0; u < kRgU; ++u) {
            const int i = min(i0 + u * nt, nlm - 1);
            y[u] = d.lmcc[2 * i];
            z[u] = d.lmcc[2 * i + 1];
        }
#pragma unroll
        for (int u = 0; u < kRgU; ++u) {
            const int i = i0 + u * nt;
            if (i >= nlm) break;
            double pos[2], vel[2], acc[2];
            move_marker(cm, rot, y[u], z[u], pos, vel, acc);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                d.lmcc[2 * i + q] = pos[q];
                d.lmvel[2 * i + q] = vel[q];
                d.lmacc[2 * i + q] = acc[q];
            }
        }
    }
    // vertices rotate about the updated centre (rigid.F90:110-121)
    for (int i0 = tid; i0 <= nlm; i0 += kRgU * nt) {
        double y[kRgU], z[kRgU];
#pragma unroll
        for (int u = 0; u < kRgU; ++u) {
            const int i = min(i0 + u * nt, nlm);
            y[u] = d.vert[2 * i];
            z[u] = d.vert[2 * i + 1];
        }
#pragma unroll
        for (int u = 0; u < kRgU; ++u) {
            const int i = i0 + u * nt;
            if (i > nlm) break;
            const double v[2] = {y[u], z[u]};
            double o[2];
            move_vertex(cm, rot, v, o);
            d.vert[2 * i] = o[0];
            d.vert[2 * i + 1] = o[1];
        }
    }
    __syncthreads();
    for (int i0 = tid; i0 < nlm; i0 += kRgU * nt) {
        double va[kRgU][4];   // vertices i and i + 1
#pragma unroll
        for (int u = 0; u < kRgU; ++u) {
            const int i = min(i0 + u * nt, nlm - 1);
#pragma unroll
            for (int q = 0; q < 4; ++q) va[u][q] = d.vert[2 * i + q];
        }
#pragma unroll
        for (int u = 0; u < kRgU; ++u) {
            const int i = i0 + u * nt;
            if (i >= nlm) break;
            double nor[2];
            segment_normal(va[u], va[u] + 2, nor);
            d.lmnor[2 * i] = nor[0];
            d.lmnor[2 * i + 1] = nor[1];
        }
    }
    if (mode == RIGID_PLACE) return;     // markers at the trial state; nothing committed
    if (tid == 0) {
        // every value read before the first store (see above)
        const double t0 = d.scal[S_TIME], stepd = d.scal[S_STEP];
        const double nbcv = d.scal[S_NBCV], nbcw = d.scal[S_NBCW], cflm = d.scal[S_CFLM];
        double fv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) fv[i] = d.forces[i];
        const double solves = (mode == RIGID_COMMIT) ? fin[3] : 1.0;   // fluid solves this step
        commit_step(d, hist_rows, cm, fv, t0, stepd, nbcv, nbcw, cflm, solves);
        if (mbox) {   // the synchronous call's status and forcecomp row, into mapped host memory
            volatile double *m = mbox;
            m[0] = static_cast<double>(*d.status);
#pragma unroll
            for (int i = 0; i < 8; ++i) m[1 + i] = fv[i];
            __threadfence_system();
        }
    }
}

__global__ void __launch_bounds__(512) k_rigid(Dev d, int hist_rows, int mode, const double *fin, double *mbox) {
    FB_GRID_WAIT();
    rigid_body(d, hist_rows, mode, fin, mbox);
}

// The end of a loosely coupled step behind k_loads_probe<true> in one block:
// the markers whose tangent carries over (loads_transfer.F90:187-214), the
// checkbcs norms, then rigid (RIGID_STEP).  It replaces two launches of the
// step's serial end; its marker and vertex arrays are staged at once and the
// normals formed from the vertices in registers, so that it makes one round
// trip to global memory where the two launches made seven.  In the step, 5.4 +
// 6.0 -> 6.0 us with 40 markers; the probes in front of it 9.7 -> 7.0 us.
constexpr int kCloseThreads = 512;
constexpr int kCloseMax = 2048;   // markers: a single block's worth (beyond, the two launches)
inline size_t close_smem(int nlm) { return static_cast<size_t>(4 * nlm + 2) * sizeof(double); }

__device__ __forceinline__ void close_body(const Dev &d, int hist_rows) {
    extern __shared__ __align__(16) double close_sm[];
    __shared__ double sh[32 * 7];
    __shared__ double cm[18], rot[4], xns[6], rs[18], kin[9];
    __shared__ int mcon[3];
    const int tid = threadIdx.x, nt = blockDim.x, nlm = d.nlm;
    double *pos0 = close_sm, *ver0 = close_sm + 2 * nlm;   // markers and vertices at the start
    for (int i = tid; i < 2 * nlm; i += nt) cp8(pos0 + i, d.lmcc + i);
    for (int i = tid; i < 2 * nlm + 2; i += nt) cp8(ver0 + i, d.vert + i);
    if (tid < 18) rs[tid] = d.rigid[tid];
    else if (tid >= 32 && tid < 41) kin[tid - 32] = d.kinori[tid - 32];
    else if (tid >= 64 && tid < 67) mcon[tid - 64] = d.rbmcon[tid - 64];
    const double time = d.scal[S_TIME], stepd = d.scal[S_STEP], cflm = d.scal[S_CFLM];
    const double c0 = d.rigid[0], c1 = d.rigid[1];
    FB_GRID_WAIT();   // (the probes before it write lfin, bcerrv, bcerrw, probe and the status)
    const bool good = *d.status == 0;   // else press and tau stay what they were
    double f[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};   // fyp, fzp, fyv, fzv, mom, the checkbcs sums
    for (int i = tid; i < nlm; i += nt) {
        const double p0 = d.press[i], t0 = d.tau[2 * i], t1 = d.tau[2 * i + 1];
        const double pn = d.lfin[3 * i], tn0 = d.lfin[3 * i + 1], tn1 = d.lfin[3 * i + 2];
        double p = good ? pn : p0, tau[2] = {good ? tn0 : t0, good ? tn1 : t1};
        const double A = d.lmA[i], ny = d.lmnor[2 * i], nz = d.lmnor[2 * i + 1];
        const double y = d.lmcc[2 * i], z = d.lmcc[2 * i + 1], ev = d.bcerrv[i], ew = d.bcerrw[i];
        const double *pb = d.probe + static_cast<size_t>(i) * 24;
        if (good && pb[23] == 0.0) {   // no tangent of its own
            double tany = 0.0, tanz = 0.0;
            carried_tangent(d, i, tany, tanz);
            finish_marker(d, i, pb, tany, tanz, p, tau);
        }
        if (good) {
            d.press[i] = p;
            d.tau[2 * i] = tau[0];
            d.tau[2 * i + 1] = tau[1];
        }
        const double Fp1 = -p * ny * A, Fp2 = -p * nz * A;
        const double Fv1 = tau[0] * A, Fv2 = tau[1] * A;
        f[0] = f[0] + Fp1;
        f[1] = f[1] + Fp2;
        f[2] = f[2] + Fv1;
        f[3] = f[3] + Fv2;
        const double r1 = y - c0, r2 = z - c1;
        f[4] = f[4] + (r1 * (Fp2 + Fv2) - r2 * (Fp1 + Fv1));
        f[5] = f[5] + ev * ev;
        f[6] = f[6] + ew * ew;
    }
    cp_wait();
    block_sum_n<7>(f, sh);   // (its barriers also publish the staged arrays)
    const double fy = f[0] + f[2], fz = f[1] + f[3];
    const double g0 = (1.0 - 1.0 / d.rbden) * d.rba0 * d.rbgravF0;
    const double g1 = (1.0 - 1.0 / d.rbden) * d.rba0 * d.rbgravF1;
    const double Fy = fy + g0, Fz = fz + g1, M = f[4];
    if (tid < 32) {
        if (tid < 3) rigid_rk4(d, tid, rs, Fy, Fz, M, xns);
        __syncwarp();
        if (tid == 0) rigid_state(d, rs, xns, kin, mcon, cm, rot);
    }
    __syncthreads();
    for (int i = tid; i <= nlm; i += nt) {
        double o[2];
        move_vertex(cm, rot, ver0 + 2 * i, o);
        d.vert[2 * i] = o[0];
        d.vert[2 * i + 1] = o[1];
        if (i == nlm) break;
        double b[2], nor[2], pos[2], vel[2], acc[2];
        move_vertex(cm, rot, ver0 + 2 * i + 2, b);
        segment_normal(o, b, nor);
        move_marker(cm, rot, pos0[2 * i], pos0[2 * i + 1], pos, vel, acc);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            d.lmnor[2 * i + q] = nor[q];
            d.lmcc[2 * i + q] = pos[q];
            d.lmvel[2 * i + q] = vel[q];
            d.lmacc[2 * i + q] = acc[q];
        }
    }
    if (tid == nt - 1) {
        const double nbcv = sqrt(f[5]) / static_cast<double>(nlm), nbcw = sqrt(f[6]) / static_cast<double>(nlm);
        d.scal[S_NBCV] = nbcv;
        d.scal[S_NBCW] = nbcw;
        const double fv[8] = {time, Fy, Fz, M, f[0], f[1], f[2], f[3]};
#pragma unroll
        for (int i = 0; i < 8; ++i) d.forces[i] = fv[i];
        for (int i = 9; i < 18; ++i) d.rigid[i] = cm[i];
        commit_step(d, hist_rows, cm, fv, time, stepd, nbcv, nbcw, cflm, 1.0);
    }
}

__global__ void __launch_bounds__(kCloseThreads, 2) k_step_close(Dev d, int hist_rows) {
    close_body(d, hist_rows);
}

// ------------------------------------------------------------ diagnostics

// ttime.F90:24-147: diagnostics of the end-of-step field for the fluid report
// (fluid_rep.out) -- vmaxv/vminv (vcheck.F90:4-80), cfl (cfl.F90) times dt,
// divgck (divergence.F90:49-82), kinen (utils_proc.F90:474-515) and the line
// vorticity of getintvort (utils_proc.F90:582-632) at row indz.  Eight block
// reductions; the last block writes history columns 22..29 of the step.
__device__ __forceinline__ void diag_body(const Dev &d, int hist_rows) {
    __shared__ double sh[32];
    __shared__ bool last;
    constexpr int kV = 8, kStride = 2048;  // partial v of block b at red[v * kStride + b]
    const int t = threadIdx.x, nt = blockDim.x, b = blockIdx.x, nb = gridDim.x;
    const long cells = static_cast<long>(d.n2m) * d.n3m;
    double v[kV] = {-100.0, -100.0, -100.0, -100.0, 1.0e-8, -100.0, 0.0, 0.0};
    for (long idx = static_cast<long>(b) * nt + t; idx < cells; idx += static_cast<long>(nb) * nt) {
        const int j = static_cast<int>(idx % d.n2m) + 1, k = static_cast<int>(idx / d.n2m) + 1;
        const int jp = j + 1, kp = k + 1;
        const double q2c = Fv(d.q2, j, k), q3c = Fv(d.q3, j, k);
        const double q2j = Fv(d.q2, jp, k), q3k = Fv(d.q3, j, kp);
        v[0] = fmax(v[0], fabs(q2c));
        v[1] = fmax(v[1], fabs(q3c));
        v[2] = fmax(v[2], -q2c);
        v[3] = fmax(v[3], -q3c);
        v[4] = fmax(v[4], fabs((q2c + q2j) * 0.5 * d.udx2m[j]) + fabs((q3c + q3k) * 0.5 * d.udx3m[k]));
        v[5] = fmax(v[5], fabs((q2j - q2c) * d.udx2m[j] + (q3k - q3c) * d.udx3m[k]));
        const double vol = (d.zz[kp] - d.zz[k]) * (d.rc[jp] - d.rc[j]);
        const double vccv = (q2c + q2j) * 0.5, vccw = (q3c + q3k) * 0.5;
        v[6] = v[6] + (vccv * vccv + vccw * vccw) * vol;
        if (k == d.indz) {
            const double dz = d.zz[kp] - d.zz[k];
            const double dwdy = (Fv(d.q3, jp, k) - q3c) / (d.rc[jp] - d.rc[j]);
            const double dvdz = (Fv(d.q2, j, kp) - q2c) / dz;
            v[7] = v[7] + (dwdy - dvdz) * (d.rc[jp] - d.rc[j]);
        }
    }
#pragma unroll
    for (int i = 0; i < kV; ++i) {
        const double r = (i < 6) ? block_reduce_fast<true>(v[i], sh) : block_reduce_fast<false>(v[i], sh);
        if (t == 0) d.red[i * kStride + b] = r;
    }
    if (t == 0) {
        __threadfence();
        last = (atomicAdd(d.count + 3, 1u) == static_cast<unsigned>(nb - 1));
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a[kV];
#pragma unroll
    for (int i = 0; i < kV; ++i) {
        double x = (i < 6) ? -1.0e300 : 0.0;
        for (int q = t; q < nb; q += nt) {
            const double y = __ldcg(d.red + i * kStride + q);
            x = (i < 6) ? fmax(x, y) : x + y;
        }
        a[i] = (i < 6) ? block_reduce_fast<true>(x, sh) : block_reduce_fast<false>(x, sh);
    }
    if (t == 0) {
        d.count[3] = 0u;
        if (hist_rows > 0) {
            const int row = static_cast<int>(d.scal[S_STEP]) - 1;  // the step k_rigid closed
            double *h = d.hist + static_cast<size_t>((row + hist_rows) % hist_rows) * FB_HIST_COLS;
            h[22] = a[4] * d.dt;                                   // cflm at the end of the step
            h[23] = a[5];                                          // dmax
            h[24] = 0.5 * a[6] / (d.rext2 * d.alx3);               // ektot
            h[25] = a[7];                                          // vorti
            h[26] = a[0];                                          // vmax(1), vmax(2)
            h[27] = a[1];
            h[28] = -a[2];                                         // vmin(1), vmin(2)
            h[29] = -a[3];
        }
    }
}

__global__ void __launch_bounds__(256) k_diag(Dev d, int hist_rows) {
    FB_GRID_WAIT();
    diag_body(d, hist_rows);
}

// ------------------------------------------------------------ grouped launches

// The same kernels over a group of cases of one launch geometry: blockIdx.z
// selects the case; its view (and substep n's constants, n 0-based) are
// staged in shared memory from the group's device array (the single-case
// kernels take them by value).

template <bool kCfl>
__global__ void __launch_bounds__(256, kNlBlocksPerSM) kg_nl_rhs(const GroupCase *__restrict__ g, int n, int pend,
                                                                 int extra) {
    extern __shared__ __align__(16) unsigned char nl_smem[];
    __shared__ Dev d;
    __shared__ SubDev s;
    if (!stage_case(g, &d, &s, n)) return;
    const int nb = gridDim.x - nl_more(extra);
    if (static_cast<int>(blockIdx.x) >= nb) {
        if ((extra & kNlBoucdq) && static_cast<int>(blockIdx.x) == nb) boucdq_body(d, s.ga, s.ro);
        else edge_means_body(d);
        return;
    }
    nl_rhs_body<kCfl>(d, s.al, s.ga, s.ro, reinterpret_cast<NlTile *>(nl_smem), pend != 0, nb);
}

__global__ void kg_mls_setup(const GroupCase *__restrict__ g) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    mls_setup_body<true>(d);
}

__global__ void kg_spread_chains(const GroupCase *__restrict__ g) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    spread_chains_body(d);
}

__global__ void kg_mls_interp(const GroupCase *__restrict__ g, int first) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    mls_interp_body<false>(d, first != 0, first != 0);   // (batches have a fixed dt)
}

__global__ void kg_mls_spread(const GroupCase *__restrict__ g) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    mls_spread_body<false>(d);
}

__global__ void kg_divg(const GroupCase *__restrict__ g, int n, int extra) {
    __shared__ Dev d;
    __shared__ SubDev s;
    if (!stage_case(g, &d, &s, n)) return;
    divg_body(d, s.usdtal, g[blockIdx.z].rmax_dph, extra);
}

__global__ void __launch_bounds__(256, kUpBlocksPerSM) kg_updvp_prcalc(const GroupCase *__restrict__ g, int n,
                                                                       int pend, int slot) {
    extern __shared__ __align__(16) unsigned char up_smem[];
    __shared__ Dev d;
    __shared__ SubDev s;
    if (!stage_case(g, &d, &s, n)) return;
    updvp_prcalc_body<false>(d, s.al, s.al * s.beta, reinterpret_cast<UpTile *>(up_smem), pend != 0, slot);
}

__global__ void kg_submean_boucqt(const GroupCase *__restrict__ g, int deferred) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    submean_boucqt_body(d, deferred != 0);
}

__global__ void __launch_bounds__(kLoadThreads, 5) kg_loads_probe(const GroupCase *__restrict__ g) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    loads_probe_tan_body<false, false>(d, false);
}

__global__ void __launch_bounds__(kLoadFin) kg_loads_finish(const GroupCase *__restrict__ g) {
    __shared__ Dev d;
    if (!stage_case(g, &d)) return;
    loads_finish_body(d);
}

// mode as k_rigid, with the case's trial load; the commit after a coupling
// iteration runs for every case (no gate)
__global__ void __launch_bounds__(512) kg_rigid(const GroupCase *__restrict__ g, int mode) {
    __shared__ Dev d;
    if (!stage_case(g, &d, nullptr, 0, mode == RIGID_PLACE || mode == RIGID_FORCES)) return;
    rigid_body(d, g[blockIdx.z].hist_rows, mode, g[blockIdx.z].fin);
}

__global__ void __launch_bounds__(256) kg_diag(const GroupCase *__restrict__ g) {
    __shared__ Dev d;
    if (!stage_case(g, &d, nullptr, 0, false)) return;
    diag_body(d, g[blockIdx.z].hist_rows);
}

// ------------------------------------------------------------ launchers

namespace {
inline dim3 grid2(int nx, int ny, dim3 b) { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y); }
}  // namespace

int stride_blocks(const Dev &d) {
    const long cells = static_cast<long>(d.n2m) * d.n3m;
    return static_cast<int>(std::min<long>((cells + 255) / 256, 148L * 8));
}

// grid-stride reductions of a group: the cases fill the GPU together, so each
// case takes fewer blocks (about eight cells per thread) and the block and
// last-block reductions are paid less often
int group_stride_blocks(const Dev &d) {
    const long cells = static_cast<long>(d.n2m) * d.n3m;
    return static_cast<int>(std::max<long>(1, std::min<long>((cells + 2047) / 2048, 148L * 8)));
}
// two blocks per SM, each on pairs of rows: few partials for the last block
// to gather, and few arrivals on the grid's counter
void launch_cfl(const Dev &d, cudaStream_t s) { pdl(k_cfl, dim3(std::min(d.n3m, 148 * 2)), dim3(256), 0, s, d); }
void launch_note(const Dev &d, cudaStream_t s) { pdl(k_note, dim3(1), dim3(32), 0, s, d.scal); }
void launch_boucdq(const Dev &d, double ga, double ro, cudaStream_t s) { pdl(k_boucdq, dim3(1), dim3(1024), 0, s, d, ga, ro); }
int nl_tiles(const Dev &d) { return ((d.n2m + kNlJ - 1) / kNlJ) * ((d.n3m + kNlK - 1) / kNlK); }

void launch_nl_rhs(const Dev &d, double al, double ga, double ro, cudaStream_t s, bool pend, const NlMaps &maps,
                   int extra) {
    const int more = nl_more(extra);
    // all resident at once; beside the marker set-up of the step (kNlMeans) a
    // sixteenth of the slots is left to its small blocks, which otherwise waited
    // for these persistent ones (none, 20, 37, 74 or 148 slots left: 1568, 1559,
    // 1562, 1572, 1592 us per step at 2048 x 1536; 20 and 37 do not differ by more
    // than two runs of one of them do)
    const int slots = 148 * kNlBlocksPerSM - more - ((extra & kNlMeans) ? 148 * kNlBlocksPerSM / 16 : 0);
    const int blocks = std::min(nl_tiles(d), slots) + more;
    pdl((extra & kNlCfl) ? k_nl_rhs_tma<true> : k_nl_rhs_tma<false>, dim3(blocks), dim3(32, 8), kNlSmemT, s, d, maps,
        al, ga, ro, pend ? 1 : 0, extra);
}

// q2, q3, pr, dph as 2-D FP64 tensors: x = j - 1 (j = 1 .. n2), y = k (0 .. n3),
// rows P doubles apart; a box is one tile with its halo (kNlTW x kNlTH)
int encode_nl_maps(NlMaps *m, const Dev &d) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn)
            return FB_ERR_CUDA;
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    const double *f[4] = {d.q2, d.q3, d.pr, d.dph};
    CUtensorMap *dst[4] = {&m->q2, &m->q3, &m->pr, &m->dph};
    for (int i = 0; i < 4; ++i) {
        if ((reinterpret_cast<uintptr_t>(f[i]) & 15u) || (static_cast<long>(d.P) * 8) % 16 || d.P < d.n2)
            return FB_ERR_STATE;
        const cuuint64_t dims[2] = {static_cast<cuuint64_t>(d.n2), static_cast<cuuint64_t>(d.n3) + 1u};
        const cuuint64_t strides[1] = {static_cast<cuuint64_t>(d.P) * 8u};
        const cuuint32_t box[2] = {static_cast<cuuint32_t>(kNlTW), static_cast<cuuint32_t>(kNlTH)};
        const cuuint32_t es[2] = {1, 1};
        const CUresult r = encode(dst[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double *>(f[i]), dims,
                                  strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return FB_ERR_CUDA;
    }
    return FB_OK;
}
void launch_lgrdist(const Dev &d, cudaStream_t s) {
    if (d.nlm) pdl(k_lgrdist, dim3((d.nlm + 127) / 128), dim3(128), 0, s, d);
}
namespace {
inline int setup_blocks(int nlm) { return (2 * nlm * kNodeLanes + kSetupThreads - 1) / kSetupThreads; }
}  // namespace
void launch_mls_setup(const Dev &d, cudaStream_t s, bool find) {
    if (d.nlm) pdl(find ? k_mls_setup<true> : k_mls_setup<false>, dim3(setup_blocks(d.nlm)), dim3(kSetupThreads),
                   0, s, d);
}
void launch_mls_interp(const Dev &d, cudaStream_t s, bool clear, bool cfl) {
    if (d.nlm)
        pdl(k_mls_interp, dim3((2 * d.nlm * kInterpLanes + 255) / 256), dim3(256), 0, s, d, clear ? 1 : 0, cfl ? 1 : 0);
}
void launch_table_clear(const Dev &d, cudaStream_t s) {
    if (d.nlm) pdl(k_table_clear, dim3((2 * d.nlm + 127) / 128), dim3(128), 0, s, d);
}
namespace {
inline int chain_blocks(int nlm) { return (2 * nlm * kSD * kNodeLanes + kChainThreads - 1) / kChainThreads; }
}  // namespace
void launch_spread_chains(const Dev &d, cudaStream_t s) {
    if (d.nlm) pdl(k_spread_chains, dim3(chain_blocks(d.nlm)), dim3(kChainThreads), 0, s, d);
}
void launch_mls_spread(const Dev &d, cudaStream_t s) {
    const int n = 2 * d.nlm * kSD;
    if (n) pdl(k_mls_spread, dim3((n + 127) / 128), dim3(128), 0, s, d);
}
void launch_helsolve(const Dev &d, const SubDev &sd, cudaStream_t s) {
    pdl(k_tri_y2, dim3((d.n3m + 63) / 64), dim3(64), 0, s, d, sd);
    pdl(k_tri_z2, dim3((d.n2m + 63) / 64), dim3(64), 0, s, d, sd);
    pdl(k_tri_y3, dim3((d.n3m + 63) / 64), dim3(64), 0, s, d, sd);
    pdl(k_tri_z3, dim3((d.n2m + 63) / 64), dim3(64), 0, s, d, sd);
}
namespace {
inline dim3 divg_grid(const Dev &d, int extra) {
    dim3 g = grid2(d.n2m, (d.n3m + kDivK - 1) / kDivK, dim3(32, 8));
    if (extra) ++g.y;
    return g;
}
}  // namespace
void launch_divg(const Dev &d, double usdtal, cudaStream_t s, double *rmax, int extra) {
    // (the row maxima's reduction assumes these blocks)
    pdl(k_divg, divg_grid(d, extra), dim3(32, 8), 0, s, d, usdtal, rmax, extra);
}
void launch_updvp_prcalc(const Dev &d, double al, double be, cudaStream_t s, bool pend, const NlMaps &maps, int slot) {
    const int blocks = std::min(nl_tiles(d), 148 * kUpBlocksPerSM);
    pdl(k_updvp_prcalc_tma, dim3(blocks), dim3(32, 8), kUpSmemT, s, d, maps, al, be, pend ? 1 : 0, slot);
}
void launch_submean_boucqt(const Dev &d, cudaStream_t s, bool deferred) {
    dim3 b(32, 8);
    pdl(k_submean_boucqt, dim3(grid2(d.n2, d.n3 + 1, b)), dim3(b), 0, s, d, deferred ? 1 : 0);
}
void launch_loads_probe(const Dev &d, cudaStream_t s, bool pend, bool finish) {
    pdl(finish ? k_loads_probe<true> : k_loads_probe<false>, dim3((d.nlm + kLoadMk - 1) / kLoadMk),
        dim3(kLoadThreads), 0, s, d, pend ? 1 : 0);
}
bool step_closes(int nlm) { return nlm > 0 && nlm <= kCloseMax; }
void launch_step_close(const Dev &d, int hist_rows, cudaStream_t s) {
    pdl(k_step_close, dim3(1), dim3(kCloseThreads), close_smem(d.nlm), s, d, hist_rows);
}
void launch_loads(const Dev &d, cudaStream_t s, bool pend) {
    if (!d.nlm) return;
    launch_loads_probe(d, s, pend, false);
    pdl(k_loads_finish, dim3((d.nlm + kLoadFin - 1) / kLoadFin), dim3(kLoadFin), 0, s, d);
}
void launch_diag(const Dev &d, int hist_rows, cudaStream_t s) {
    pdl(k_diag, dim3(std::min(stride_blocks(d), 2048)), dim3(256), 0, s, d, hist_rows);
}
// The end of a synchronous API call: the status word (and the forcecomp
// row) written by the GPU into mapped host memory, so that the host reads them
// after its stream synchronisation without a device-to-host copy
__global__ void k_publish(const int *status, const double *forces, double *mbox) {
    FB_GRID_WAIT();
    volatile double *m = mbox;
    m[0] = static_cast<double>(*status);
    if (forces)
        for (int i = 0; i < 8; ++i) m[1 + i] = forces[i];
    __threadfence_system();
}
void launch_publish(const Dev &d, bool forces, double *mbox, cudaStream_t s) {
    pdl(k_publish, dim3(1), dim3(1), 0, s, static_cast<const int *>(d.status),
        forces ? static_cast<const double *>(d.forces) : nullptr, mbox);
}

void launch_rigid(const Dev &d, int hist_rows, cudaStream_t s, int mode, const double *fin, double *mbox) {
    if (d.nlm) pdl(k_rigid, dim3(1), dim3(512), 0, s, d, hist_rows, mode, fin, mbox);
}


// grouped launchers: the geometry of the group's first case, gridDim.z = cases
namespace {
inline dim3 zgrid(dim3 g, const Group &gr) { return dim3(g.x, g.y, static_cast<unsigned>(gr.n)); }
}  // namespace

void glaunch_nl_rhs(const Group &g, int n, cudaStream_t s, bool pend, int extra) {
    // about two waves of resident blocks over the whole group
    const int per_case = std::max(1, std::min(nl_tiles(g.rep), (2 * 148 * kNlBlocksPerSM + g.n - 1) / g.n)) +
                         nl_more(extra);
    pdl((extra & kNlCfl) ? kg_nl_rhs<true> : kg_nl_rhs<false>, zgrid(dim3(per_case), g), dim3(32, 8), kNlSmem, s,
        g.cases, n, pend ? 1 : 0, extra);
}

cudaError_t kernels_configure() {
    cudaError_t e = cudaSuccess;
    auto allow = [&](auto kern, size_t smem) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    };
    allow(k_nl_rhs_tma<false>, kNlSmemT);
    allow(k_nl_rhs_tma<true>, kNlSmemT);
    allow(kg_nl_rhs<false>, kNlSmem);
    allow(kg_nl_rhs<true>, kNlSmem);
    allow(k_updvp_prcalc_tma, kUpSmemT);
    allow(kg_updvp_prcalc, kUpSmem);
    allow(k_step_close, close_smem(kCloseMax));
    return e;
}
void glaunch_marker_setup(const Group &g, cudaStream_t s) {
    const Dev &d = g.rep;
    if (!d.nlm) return;
    pdl(kg_mls_setup, zgrid(dim3(setup_blocks(d.nlm)), g), dim3(kSetupThreads), 0, s, g.cases);
    pdl(kg_spread_chains, zgrid(dim3(chain_blocks(d.nlm)), g), dim3(kChainThreads), 0, s, g.cases);
}
void glaunch_forcing(const Group &g, int n, cudaStream_t s) {
    const Dev &d = g.rep;
    if (!d.nlm) return;
    pdl(kg_mls_interp, zgrid(dim3((2 * d.nlm * kInterpLanes + 255) / 256), g), dim3(256), 0, s, g.cases,
        n == 0 ? 1 : 0);
    pdl(kg_mls_spread, zgrid(dim3((2 * d.nlm * kSD + 127) / 128), g), dim3(128), 0, s, g.cases);
}
void glaunch_divg(const Group &g, int n, cudaStream_t s, int extra) {
    pdl(kg_divg, zgrid(divg_grid(g.rep, extra), g), dim3(32, 8), 0, s, g.cases, n, extra);
}
void glaunch_updvp_prcalc(const Group &g, int n, cudaStream_t s, bool pend, int slot) {
    const int per_case = std::max(1, std::min(nl_tiles(g.rep), (2 * 148 * kUpBlocksPerSM + g.n - 1) / g.n));
    pdl(kg_updvp_prcalc, zgrid(dim3(per_case), g), dim3(32, 8), kUpSmem, s, g.cases, n, pend ? 1 : 0,
        slot);
}
void glaunch_submean_boucqt(const Group &g, cudaStream_t s, bool deferred) {
    dim3 b(32, 8);
    pdl(kg_submean_boucqt, zgrid(grid2(g.rep.n2, g.rep.n3 + 1, b), g), dim3(b), 0, s, g.cases, deferred ? 1 : 0);
}
void glaunch_loads(const Group &g, cudaStream_t s) {
    const Dev &d = g.rep;
    if (!d.nlm) return;
    pdl(kg_loads_probe, zgrid(dim3((d.nlm + kLoadMk - 1) / kLoadMk), g), dim3(kLoadThreads), 0, s, g.cases);
    pdl(kg_loads_finish, zgrid(dim3((d.nlm + kLoadFin - 1) / kLoadFin), g), dim3(kLoadFin), 0, s, g.cases);
}
void glaunch_rigid(const Group &g, cudaStream_t s, int mode) {
    if (g.rep.nlm) pdl(kg_rigid, zgrid(dim3(1), g), dim3(512), 0, s, g.cases, mode);
}
void glaunch_diag(const Group &g, cudaStream_t s) {
    pdl(kg_diag, zgrid(dim3(std::min(group_stride_blocks(g.rep), 2048)), g), dim3(256), 0, s, g.cases);
}

}  // namespace fb
