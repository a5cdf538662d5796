// batch.cu -- persistent batched CG over many independent systems (batch.cuh).
//
// One launch solves every bound system.  Each CTA (or each team of CTAs, for the
// largest systems: a whole cluster, then its halves, each from its own queue) takes the
// next job from an atomic queue and runs a complete preconditioned CG on it, with
// team-local reductions and no grid-wide synchronisation; when the queues are empty
// the CTA retires.  Jobs are ordered by estimated cost (the iteration count of the
// previous solve of the same system, when there was one), so the longest systems
// start first, and in the largest teams.
//
// Team step of one CG iteration (each warp of the team owns whole 32-row
// slices of the system's sliced-ELL matrix, dealt out over the CTAs first so that
// all SMs of a cluster get the same share; the thread that computes q for a
// row also updates that row's x, r, z and p, so only the dot products and the
// complete direction vector need team-wide synchronisation):
//   q = K p, <p,q>        -> team reduction 1 (alpha)
//   x, r, z, <r,z>, <r,r>  -> team reduction 2 (beta, stop test)
//   p = z + beta p        -> team barrier (p complete before the next gathers)
// Vectors written during the launch are gathered with ld.global.cg (L2, not the
// SM's L1, which is not coherent across the cluster's SMs); the matrix, the
// right-hand side and the preconditioner are read-only in the launch.
#include <cooperative_groups.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <functional>
#include <mutex>
#include <numeric>
#include <vector>

#include "batch.cuh"

namespace cg = cooperative_groups;

namespace pfg {
namespace {

constexpr int kMaxCluster = kMaxTeam;
constexpr int kAbortEvery = 64;   // iterations between two reads of the abort flag
// Mixed precision hands a system over to FP64 CG (from its current x) after
// kMaxFailures FP32 passes in a row that broke down, overflowed or diverged
// (|r| grew kDiverge-fold over its smallest value in the pass), or kMaxStall
// replacements in a row that did not cut the FP64 residual by 10 %: the FP32
// copy of a system conditioned beyond FP32 is not positive definite.
constexpr int kMaxFailures = 2;
constexpr int kMaxStall = 3;
constexpr float kDiverge = 1.0e3f;

struct TeamShared {
    double slot[2][kMaxCluster][4];   // CTA totals of team reductions, one row per rank (every CTA holds all)
    double wpart[2][32][4];           // per-warp partials (FP64), double-buffered
    float wpart32[2][32][4];          // per-warp compensated partials (s, c pairs), double-buffered
    uint64_t bar[kTeamSizes];         // mbarriers of teams smaller than the cluster, one per size
    long long limit;                  // clock cycles after which a wait on one of them gives up
    int lost;                         // a wait in one of this CTA's teams ran out (set from any of them, at any time)
    int gone;                         // the CTA has taken note: written between its own barriers
    double scalar[2][4];              // what thread 0 made of a reduction's totals, for the whole CTA
    int job;
};

struct Team {
    int rank;          // CTA rank in the team
    int size;          // CTAs in the team (1: a single CTA)
    int base;          // the team's first CTA in the cluster
    bool whole;        // the team is the whole cluster
    int level;         // mbarrier of this size
    unsigned parity;   // of the mbarrier's current phase
    int nred;          // reductions done on this job (alternates the double buffers)
    // a barrier of this team gave up (the same in every thread of the CTA)
    __device__ __forceinline__ bool gave_up(const TeamShared &sh) const { return size > 1 && !whole && sh.gone; }
};

// Barrier of the CTAs of a team, with release and acquire over the cluster: the
// hardware's cluster barrier for a whole cluster; for a part of one an mbarrier in every
// CTA's shared memory on which each CTA of the team arrives once and warp 0 waits.
// False, in every thread of the CTA alike: a wait ran out, here or in another CTA of
// the team.  The CTA then marks every CTA of the team lost and arrives on none of the
// team's barriers again, so that no other CTA passes one without it: their waits end too
// (the mark spares them the limit), and the job's record stays PFG_E_INTERNAL.  Nor does
// it write into another CTA's slots: one that has passed its last barrier may still be
// adding them.
__device__ __forceinline__ bool team_barrier(Team &tm, TeamShared &sh)
{
    if (tm.whole) {
        cg::this_cluster().sync();
        return true;
    }
    if (__syncthreads_or(*(volatile int *)&sh.lost)) {
        if (threadIdx.x == 0) sh.gone = 1;
        __syncthreads();
        return false;
    }
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&sh.bar[tm.level]);
    if ((int)threadIdx.x < tm.size) {
        uint32_t remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(bar), "r"(tm.base + (int)threadIdx.x));
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
    }
    uint32_t done = 1;
    if (threadIdx.x < 32) {
        done = 0;
        const long long t0 = clock64(), limit = sh.limit;
        while (!done && clock64() - t0 <= limit) {
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(tm.parity)
                : "memory");
            if (!done && *(volatile int *)&sh.lost) break;
        }
    }
    tm.parity ^= 1;
    if (__syncthreads_and(done)) return true;
    if ((int)threadIdx.x < tm.size)
        *(volatile int *)cg::this_cluster().map_shared_rank(&sh.lost, tm.base + (int)threadIdx.x) = 1;
    if (threadIdx.x == 0) sh.gone = 1;
    __syncthreads();
    return false;
}

__device__ __forceinline__ void team_sync(Team &tm, TeamShared &sh)
{
    if (tm.size > 1)
        team_barrier(tm, sh);
    else
        __syncthreads();
}

// Team-wide sums of NV = 1 or 2 FP64 values, left in v of thread 0 of every CTA (the
// same bits in each).  An FP64 instruction holds its quarter of the SM's pipe for 64
// cycles whichever warp issues it, so what follows the warps' own sums is done by
// one warp, and what a caller makes of the totals (a division is 660 cycles in one
// warp and 2,560 in all sixteen) by thread 0, which passes it on in sh.scalar: a
// 6-slice system's iteration 20.3 -> 14.1 us, in a cluster 25.2 -> 15.2.  In a cluster
// warp 0 pushes the CTA's totals into row `rank` of every CTA's slot table
// (distributed shared memory) and after the cluster barrier adds its own copy in a fixed
// order.  The buffers alternate between consecutive reductions: one is rewritten two
// reductions later, after a barrier of the reduction in between that its readers
// have passed.  Returns the buffer's index.
template <int NV>
__device__ __forceinline__ int team_reduce(double (&v)[NV], Team &tm, TeamShared &sh)
{
    static_assert(NV == 1 || NV == 2, "one or two values per reduction");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int buf = tm.nred++ & 1;
    const double part = lanes_sum<NV>(v, lane);
    if (NV == 1 ? lane == 0 : (lane & 15) == 0) sh.wpart[buf][wid][lane >> 4] = part;
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] = lane < nw ? sh.wpart[buf][lane][k] : 0.0;
        double t = lanes_sum<NV>(v, lane);
        v[0] = __shfl_sync(0xffffffffu, t, 0);
        if (NV == 2) v[NV - 1] = __shfl_sync(0xffffffffu, t, 16);
    }
    if (tm.size > 1) {
        cg::cluster_group cl = cg::this_cluster();
        if (wid == 0 && lane < tm.size && !tm.gave_up(sh)) {
            double *dst = cl.map_shared_rank(&sh.slot[buf][tm.rank][0], tm.base + lane);
#pragma unroll
            for (int k = 0; k < NV; ++k) dst[k] = v[k];
        }
        team_barrier(tm, sh);
        if (wid == 0) {
            // lane 16 k + r: value k of rank r
            const int r = lane & 15, k = NV == 2 ? lane >> 4 : 0;
            double t = r < tm.size ? sh.slot[buf][r][k] : 0.0;
#pragma unroll
            for (int o = kMaxCluster / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            v[0] = __shfl_sync(0xffffffffu, t, 0);
            if (NV == 2) v[NV - 1] = __shfl_sync(0xffffffffu, t, 16);
        }
    }
    return buf;
}

// The totals for all threads of the team.
template <int NV>
__device__ __forceinline__ void team_sum(double (&v)[NV], Team &tm, TeamShared &sh)
{
    const int buf = team_reduce<NV>(v, tm, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) sh.scalar[buf][k] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = sh.scalar[buf][k];
}

__device__ __forceinline__ void comp_warp_merge(Comp32 &t)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float s2 = __shfl_xor_sync(0xffffffffu, t.s, o);
        const float c2 = __shfl_xor_sync(0xffffffffu, t.c, o);
        comp_merge(t, s2, c2);
    }
}

// Team-wide compensated FP32 sums (Dot2 accumulators), rounded to float at the
// end; same structure as team_sum.
template <int NV>
__device__ __forceinline__ void team_sum_comp(Comp32 (&v)[NV], float (&tot)[NV], Team &tm, TeamShared &sh)
{
    static_assert(NV <= 2, "at most 2 compensated values per reduction");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int buf = tm.nred++ & 1;
#pragma unroll
    for (int k = 0; k < NV; ++k) comp_warp_merge(v[k]);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            sh.wpart32[buf][wid][2 * k] = v[k].s;
            sh.wpart32[buf][wid][2 * k + 1] = v[k].c;
        }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        v[k].s = lane < nw ? sh.wpart32[buf][lane][2 * k] : 0.f;
        v[k].c = lane < nw ? sh.wpart32[buf][lane][2 * k + 1] : 0.f;
        comp_warp_merge(v[k]);
    }
    if (tm.size > 1) {
        cg::cluster_group cl = cg::this_cluster();
        if (wid == 0 && lane < tm.size && !tm.gave_up(sh)) {
            double *dst = cl.map_shared_rank(&sh.slot[buf][tm.rank][0], tm.base + lane);
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                dst[2 * k] = (double)v[k].s;
                dst[2 * k + 1] = (double)v[k].c;
            }
        }
        team_barrier(tm, sh);
        if (tm.gave_up(sh)) {  // the same in every thread, as what follows from it has to be
#pragma unroll
            for (int k = 0; k < NV; ++k) tot[k] = __int_as_float(0x7fc00000);
            return;
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            v[k].s = lane < tm.size ? (float)sh.slot[buf][lane][2 * k] : 0.f;
            v[k].c = lane < tm.size ? (float)sh.slot[buf][lane][2 * k + 1] : 0.f;
            comp_warp_merge(v[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) tot[k] = __fadd_rn(v[k].s, v[k].c);
}

// Abort flag of the batch, read by rank 0 and agreed on by the team.
__device__ __forceinline__ bool team_abort(const BatchParams &P, Team &tm, TeamShared &sh)
{
    double f[1] = {(P.abort && tm.rank == 0 && threadIdx.x == 0) ? (double)(*P.abort != 0) : 0.0};
    team_sum<1>(f, tm, sh);
    return f[0] != 0.0;
}

template <typename T>
__device__ __forceinline__ void precond3(int pc, const T *__restrict__ dinv, int64_t row, const T (&r)[3],
                                         T (&z)[3])
{
    if (pc == PFG_PC_NONE) {
#pragma unroll
        for (int i = 0; i < 3; ++i) z[i] = r[i];
        return;
    }
    const T *D = dinv + row * 9;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        T s = T(0);
#pragma unroll
        for (int j = 0; j < 3; ++j) s = fma(__ldg(D + i * 3 + j), r[j], s);
        z[i] = s;
    }
}

// Gather of block column c of a vector written during the launch (L2 path).
template <typename T>
struct GatherCG {
    const T *v;
    __device__ __forceinline__ void operator()(int c, T (&xv)[3]) const
    {
        const T *q = v + 3 * (int64_t)c;
        xv[0] = __ldcg(q);
        xv[1] = __ldcg(q + 1);
        xv[2] = __ldcg(q + 2);
    }
};

struct Span {
    int64_t w0, nw;   // this thread's warp in the team, CTA by CTA in turn, and the team's warps
};

__device__ __forceinline__ Span team_span(const Team &tm, int warps_per_cta)
{
    return Span{(int64_t)(threadIdx.x >> 5) * tm.size + tm.rank, (int64_t)tm.size * warps_per_cta};
}

// Sum of squares of r = b - K x (FP64) over the team, r written out.
__device__ double residual64(const BatchMesh &D, const Span &sp, Team &tm, TeamShared &sh)
{
    // Local copies of the descriptor's pointers: stores through them cannot
    // alias the descriptor, so it is not re-read after every store.
    const int lane = threadIdx.x & 31;
    const SellView<double> A = D.A64;
    const double *__restrict__ b = D.b;
    const double *__restrict__ x = D.x;
    double *__restrict__ r = D.r64;
    double acc[1] = {0.0};
    for (int64_t s = sp.w0; s < A.ns; s += sp.nw) {
        double y[3];
        sell_row_product<3>(A, s, lane, GatherCG<double>{x}, y);
        const int64_t row = s * 32 + lane;
        if (row < A.nb) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int64_t i = 3 * row + k;
                const double rv = __ldg(b + i) - y[k];
                r[i] = rv;
                acc[0] = fma(rv, rv, acc[0]);
            }
        }
    }
    team_sum<1>(acc, tm, sh);
    return acc[0];
}

// Gather of block column c of the candidate solution x + x32.
struct GatherSum {
    const double *x;
    const float *x32;
    __device__ __forceinline__ void operator()(int c, double (&xv)[3]) const
    {
        const int64_t j = 3 * (int64_t)c;
#pragma unroll
        for (int k = 0; k < 3; ++k) xv[k] = __ldcg(x + j + k) + (double)__ldcg(x32 + j + k);
    }
};

// Sum of squares of b - K (x + x32) over the team; the candidate residual is
// written to q64 (unused by the mixed iterations), r64 keeps the residual of x.
__device__ double candidate_residual(const BatchMesh &D, const Span &sp, Team &tm, TeamShared &sh)
{
    const int lane = threadIdx.x & 31;
    const SellView<double> A = D.A64;
    const double *__restrict__ b = D.b;
    double *__restrict__ q = D.q64;
    const GatherSum src{D.x, D.x32};
    double acc[1] = {0.0};
    for (int64_t s = sp.w0; s < A.ns; s += sp.nw) {
        double y[3];
        sell_row_product<3>(A, s, lane, src, y);
        const int64_t row = s * 32 + lane;
        if (row < A.nb) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int64_t i = 3 * row + k;
                const double rv = __ldg(b + i) - y[k];
                q[i] = rv;
                acc[0] = fma(rv, rv, acc[0]);
            }
        }
    }
    team_sum<1>(acc, tm, sh);
    return acc[0];
}

__device__ void restore_fixed_rows(const BatchMesh &D, const Span &sp, int64_t nb)
{
    const uint8_t *__restrict__ fixed = D.fixed;
    const double *__restrict__ fixval = D.fixval;
    double *__restrict__ x = D.x;
    if (!fixed) return;
    const int lane = threadIdx.x & 31;
    for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
        const int64_t row = s * 32 + lane;
        if (row < nb)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int64_t i = 3 * row + k;
                if (fixed[i]) x[i] = fixval[i];
            }
    }
}

// ------------------------------------------------------------- FP64 CG
// Preconditioned CG on K x = b from the current x, counting on from `it`:
//   q = K p, <p,q>                      -> team reduction (alpha)
//   x += a p, r -= a q, z = M^-1 r, <r,z>, <r,r>   -> team reduction (beta, stop)
//   p = z + b p                         -> team barrier (p complete for the gathers)
// (The Chronopoulos-Gear form, one reduction per iteration, measured 8 % slower
// here: its extra live vectors cost registers the SpMV needs.)  A recursive
// residual at the tolerance is confirmed on the true residual, restarting from
// it otherwise (at most P.max_restarts).  Returns the status; `rel` = true
// |b - Kx| / |b| at exit.
template <int NT>
__device__ int cg64(const BatchParams &P, const BatchMesh &D, Team &tm, TeamShared &sh, int &it, int &restarts,
                    double &rel)
{
    const SellView<double> A = D.A64;
    const int64_t nb = A.nb;
    const int lane = threadIdx.x & 31;
    const Span sp = team_span(tm, NT / 32);
    const int pc = P.precond;
    const bool lead = tm.rank == 0 && threadIdx.x == 0;

    // r = b - K x0, z = M^-1 r, p = z
    double a3[3] = {0.0, 0.0, 0.0};
    {
        const double *__restrict__ b = D.b;
        const double *__restrict__ x = D.x;
        double *__restrict__ r = D.r64;
        double *__restrict__ z = D.z64;
        double *__restrict__ p = D.p64;
        const double *__restrict__ dinv = D.dinv64;
        for (int64_t s = sp.w0; s < A.ns; s += sp.nw) {
            double y[3];
            sell_row_product<3>(A, s, lane, GatherCG<double>{x}, y);
            const int64_t row = s * 32 + lane;
            if (row < nb) {
                double rv[3], zv[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double bi = __ldg(b + 3 * row + k);
                    rv[k] = bi - y[k];
                    a3[2] = fma(bi, bi, a3[2]);
                }
                precond3<double>(pc, dinv, row, rv, zv);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int64_t i = 3 * row + k;
                    r[i] = rv[k];
                    z[i] = zv[k];
                    p[i] = zv[k];
                    a3[0] = fma(rv[k], zv[k], a3[0]);
                    a3[1] = fma(rv[k], rv[k], a3[1]);
                }
            }
        }
    }
    double a1[1] = {a3[2]}, a01[2] = {a3[0], a3[1]};
    team_sum<1>(a1, tm, sh);
    team_sum<2>(a01, tm, sh);  // also completes p for the first gathers
    double rho = a01[0];
    const double bb = a1[0];
    const double tol_b = P.tol * sqrt(bb);
    int status = PFG_OK;
    rel = bb > 0.0 ? sqrt(a01[1] / bb) : 0.0;
    if (tm.gave_up(sh)) return PFG_E_INTERNAL;
    if (sqrt(a01[1]) <= tol_b) return PFG_OK;
    for (;;) {
        if (it >= P.itrmax) {
            status = PFG_W_NOT_CONVERGED;
            break;
        }
        // q = K p, <p, q>; the abort flag rides along every kAbortEvery iterations
        double a2[2] = {0.0, 0.0};
        if (P.abort && lead && it % kAbortEvery == 0) a2[1] = (double)(*P.abort != 0);
        {
            const double *__restrict__ p = D.p64;
            double *__restrict__ q = D.q64;
            for (int64_t s = sp.w0; s < A.ns; s += sp.nw) {
                double y[3];
                sell_row_product<3>(A, s, lane, GatherCG<double>{p}, y);
                const int64_t row = s * 32 + lane;
                if (row < nb)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const int64_t i = 3 * row + k;
                        q[i] = y[k];
                        a2[0] = fma(p[i], y[k], a2[0]);
                    }
            }
        }
        const int b2 = team_reduce<2>(a2, tm, sh);
        if (threadIdx.x == 0) {
            const bool ok = a2[1] == 0.0 && a2[0] > 0.0 && isfinite(a2[0]);
            sh.scalar[b2][0] = ok ? rho / a2[0] : 0.0;
            sh.scalar[b2][1] = tm.gave_up(sh)         ? (double)PFG_E_INTERNAL
                               : a2[1] != 0.0 ? (double)PFG_E_ABORTED
                               : ok           ? (double)PFG_OK
                                              : (double)PFG_E_BREAKDOWN;
        }
        __syncthreads();
        status = (int)sh.scalar[b2][1];
        if (status != PFG_OK) break;
        const double alpha = sh.scalar[b2][0];
        // x += alpha p, r -= alpha q, z = M^-1 r, <r, z>, <r, r>
        double a4[2] = {0.0, 0.0};
        {
            double *__restrict__ x = D.x;
            double *__restrict__ r = D.r64;
            double *__restrict__ z = D.z64;
            const double *__restrict__ p = D.p64;
            const double *__restrict__ q = D.q64;
            const double *__restrict__ dinv = D.dinv64;
            for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
                const int64_t row = s * 32 + lane;
                if (row >= nb) continue;
                double rv[3], zv[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int64_t i = 3 * row + k;
                    x[i] = fma(alpha, p[i], x[i]);
                    rv[k] = fma(-alpha, q[i], r[i]);
                    r[i] = rv[k];
                }
                precond3<double>(pc, dinv, row, rv, zv);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    z[3 * row + k] = zv[k];
                    a4[0] = fma(rv[k], zv[k], a4[0]);
                    a4[1] = fma(rv[k], rv[k], a4[1]);
                }
            }
        }
        const int b4 = team_reduce<2>(a4, tm, sh);  // x complete for a true residual
        if (threadIdx.x == 0) {
            const bool finite = isfinite(a4[0]) && isfinite(a4[1]);
            sh.scalar[b4][0] = a4[0] / rho;
            sh.scalar[b4][1] = a4[0];
            sh.scalar[b4][2] = !finite ? 2.0 : sqrt(a4[1]) <= tol_b ? 1.0 : 0.0;
        }
        __syncthreads();
        ++it;
        double beta = sh.scalar[b4][0];
        const double state = sh.scalar[b4][2];
        rho = sh.scalar[b4][1];
        if (tm.gave_up(sh)) {
            status = PFG_E_INTERNAL;
            break;
        }
        if (state == 2.0) {
            status = PFG_E_NONFINITE;
            break;
        }
        if (state == 1.0) {
            // recursive residual converged: confirm on the true residual
            const double rt = residual64(D, sp, tm, sh);
            rel = bb > 0.0 ? sqrt(rt / bb) : 0.0;
            if (tm.gave_up(sh)) return PFG_E_INTERNAL;
            if (sqrt(rt) <= tol_b) return PFG_OK;
            if (restarts >= P.max_restarts) {
                status = PFG_W_NOT_CONVERGED;
                break;
            }
            ++restarts;
            // restart from the true residual (r64 holds it): z = M^-1 r, p = z
            double ar[1] = {0.0};
            {
                const double *__restrict__ r = D.r64;
                double *__restrict__ z = D.z64;
                const double *__restrict__ dinv = D.dinv64;
                for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
                    const int64_t row = s * 32 + lane;
                    if (row >= nb) continue;
                    double rv[3], zv[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) rv[k] = r[3 * row + k];
                    precond3<double>(pc, dinv, row, rv, zv);
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        z[3 * row + k] = zv[k];
                        ar[0] = fma(rv[k], zv[k], ar[0]);
                    }
                }
            }
            team_sum<1>(ar, tm, sh);
            rho = ar[0];
            beta = 0.0;
        }
        // p = z + beta p (p = z after a restart)
        {
            double *__restrict__ p = D.p64;
            const double *__restrict__ z = D.z64;
            for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
                const int64_t row = s * 32 + lane;
                if (row >= nb) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int64_t i = 3 * row + k;
                    p[i] = beta == 0.0 ? z[i] : fma(beta, p[i], z[i]);
                }
            }
        }
        team_sync(tm, sh);
    }
    const double rt = residual64(D, sp, tm, sh);
    rel = bb > 0.0 ? sqrt(rt / bb) : 0.0;
    return status;
}

__device__ void finish_job(const BatchParams &P, int m, const BatchMesh &D, Team &tm, const TeamShared &sh,
                           int status, int it, int reps, int fallback, double rel)
{
    restore_fixed_rows(D, team_span(tm, blockDim.x / 32), D.A64.nb);
    if (tm.rank == 0 && threadIdx.x == 0) {
        BatchOut o;
        o.status = tm.gave_up(sh) ? PFG_E_INTERNAL : status;
        o.iterations = it;
        o.replacements = reps;
        o.team_size = tm.size;
        o.fallback = fallback;
        o.rel_residual = rel;
        P.out[m] = o;
    }
}

template <int NT>
__device__ void solve_fp64(const BatchParams &P, int m, Team &tm, TeamShared &sh, int fallback)
{
    const BatchMesh &D = P.mesh[m];
    int it = 0, restarts = 0;
    double rel = 0.0;
    const int status = cg64<NT>(P, D, tm, sh, it, restarts, rel);
    finish_job(P, m, D, tm, sh, status, it, restarts, fallback, rel);
}

// ------------------------------------------- FP32 CG with FP64 replacement
template <int NT>
__device__ void solve_mixed(const BatchParams &P, int m, Team &tm, TeamShared &sh)
{
    const BatchMesh &D = P.mesh[m];
    const SellView<float> A = D.A32;
    const int64_t nb = A.nb;
    const int lane = threadIdx.x & 31;
    const Span sp = team_span(tm, NT / 32);
    const int pc = P.precond;

    // FP64 residual of x0 and |b|
    double a2[2] = {0.0, 0.0};
    for (int64_t s = sp.w0; s < D.A64.ns; s += sp.nw) {
        double y[3];
        sell_row_product<3>(D.A64, s, lane, GatherCG<double>{D.x}, y);
        const int64_t row = s * 32 + lane;
        if (row < nb)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int64_t i = 3 * row + k;
                const double bi = __ldg(D.b + i);
                const double rv = bi - y[k];
                D.r64[i] = rv;
                D.x32[i] = 0.f;
                a2[0] = fma(rv, rv, a2[0]);
                a2[1] = fma(bi, bi, a2[1]);
            }
    }
    team_sum<2>(a2, tm, sh);
    const double bb = a2[1];
    const double tol_b = P.tol * sqrt(bb);
    double rel = bb > 0.0 ? sqrt(a2[0] / bb) : 0.0;
    int it = 0, reps = 0, status = PFG_OK, failures = 0, stall = 0, fallback = 0;
    double best_rt = a2[0], cur_rt = a2[0];
    bool converged = sqrt(a2[0]) <= tol_b;
    bool restart = true;   // the first pass starts from p = z
    float rho = 0.f, rmax = 0.f, rmin = 0.f;
    while (!converged && !tm.gave_up(sh)) {
        // (re)start from the FP64 residual: r32 = r64, z = M^-1 r, beta keeps p unless a restart
        {
            Comp32 c2[2] = {Comp32{0.f, 0.f}, Comp32{0.f, 0.f}};
            for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
                const int64_t row = s * 32 + lane;
                if (row >= nb) continue;
                float rv[3], zv[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    rv[k] = (float)D.r64[3 * row + k];
                    D.r32[3 * row + k] = rv[k];
                }
                precond3<float>(pc, D.dinv32, row, rv, zv);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    D.z32[3 * row + k] = zv[k];
                    comp_add_prod(c2[0], rv[k], zv[k]);
                    comp_add_prod(c2[1], rv[k], rv[k]);
                }
            }
            float t2[2];
            team_sum_comp<2>(c2, t2, tm, sh);
            const float beta = (!restart && rho != 0.f && isfinite(t2[0])) ? t2[0] / rho : 0.f;
            rho = t2[0];
            rmax = sqrtf(t2[1]);
            rmin = rmax;
            for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
                const int64_t row = s * 32 + lane;
                if (row >= nb) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int64_t i = 3 * row + k;
                    D.p32[i] = beta == 0.f ? D.z32[i] : fmaf(beta, D.p32[i], D.z32[i]);
                }
            }
            team_sync(tm, sh);
        }
        // FP32 iterations until the residual fell by delta (or trouble)
        bool poisoned = false, broke = false, diverged = false;
        for (;;) {
            if (it >= P.itrmax) break;
            if (P.abort && it % kAbortEvery == 0 && team_abort(P, tm, sh)) {
                status = PFG_E_ABORTED;
                break;
            }
            Comp32 c1[1] = {Comp32{0.f, 0.f}};
            for (int64_t s = sp.w0; s < A.ns; s += sp.nw) {
                float y[3];
                sell_row_product<3>(A, s, lane, GatherCG<float>{D.p32}, y);
                const int64_t row = s * 32 + lane;
                if (row < nb)
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const int64_t i = 3 * row + k;
                        D.q32[i] = y[k];
                        comp_add_prod(c1[0], D.p32[i], y[k]);
                    }
            }
            float pq[1];
            team_sum_comp<1>(c1, pq, tm, sh);
            if (!(pq[0] > 0.f) || !isfinite(pq[0])) {
                broke = true;
                break;
            }
            const float alpha = rho / pq[0];
            Comp32 c2[2] = {Comp32{0.f, 0.f}, Comp32{0.f, 0.f}};
            for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
                const int64_t row = s * 32 + lane;
                if (row >= nb) continue;
                float rv[3], zv[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int64_t i = 3 * row + k;
                    D.x32[i] = fmaf(alpha, D.p32[i], D.x32[i]);
                    rv[k] = fmaf(-alpha, D.q32[i], D.r32[i]);
                    D.r32[i] = rv[k];
                }
                precond3<float>(pc, D.dinv32, row, rv, zv);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    D.z32[3 * row + k] = zv[k];
                    comp_add_prod(c2[0], rv[k], zv[k]);
                    comp_add_prod(c2[1], rv[k], rv[k]);
                }
            }
            float t2[2];
            team_sum_comp<2>(c2, t2, tm, sh);
            ++it;
            if (!isfinite(t2[0]) || !isfinite(t2[1])) {
                poisoned = true;
                break;
            }
            const float rn = sqrtf(t2[1]);
            rmax = fmaxf(rmax, rn);
            rmin = fminf(rmin, rn);
            if (rn > kDiverge * rmin) {
                diverged = true;
                break;
            }
            if ((double)rn < P.delta * (double)rmax || (double)rn <= tol_b) {
                // residual replacement; the restart block recomputes rho and
                // keeps the direction through beta = rho_new / rho
                break;
            }
            const float beta = t2[0] / rho;
            rho = t2[0];
            for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
                const int64_t row = s * 32 + lane;
                if (row >= nb) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int64_t i = 3 * row + k;
                    D.p32[i] = fmaf(beta, D.p32[i], D.z32[i]);
                }
            }
            team_sync(tm, sh);
        }
        // Keep the FP32 correction only if it lowers the FP64 residual: the
        // candidate b - K (x + x32) goes to q64; on acceptance it becomes r64
        // and x32 is folded into x, otherwise x and r64 stay as they were.
        bool accepted = false;
        double rt = cur_rt;
        if (!poisoned) {
            rt = candidate_residual(D, sp, tm, sh);
            accepted = isfinite(rt) && rt < cur_rt;
        }
        for (int64_t s = sp.w0; s * 32 < nb; s += sp.nw) {
            const int64_t row = s * 32 + lane;
            if (row >= nb) continue;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int64_t i = 3 * row + k;
                if (accepted) {
                    D.x[i] += (double)D.x32[i];
                    D.r64[i] = D.q64[i];
                }
                D.x32[i] = 0.f;
            }
        }
        team_sync(tm, sh);
        ++reps;
        if (tm.gave_up(sh)) break;
        if (accepted) cur_rt = rt;
        rt = cur_rt;
        rel = bb > 0.0 ? sqrt(rt / bb) : 0.0;
        if (status == PFG_E_ABORTED) break;
        if (sqrt(rt) <= tol_b) {
            converged = true;
            break;
        }
        if (it >= P.itrmax) {
            status = PFG_W_NOT_CONVERGED;
            break;
        }
        if (rt < 0.81 * best_rt) {
            best_rt = rt;
            stall = 0;
        } else {
            ++stall;
        }
        restart = poisoned || broke || diverged || !accepted;
        failures = restart ? failures + 1 : 0;
        if (failures >= kMaxFailures || stall >= kMaxStall) {
            // FP32 cannot carry this system: FP64 CG from the current x
            fallback = 1;
            int restarts = 0;
            status = cg64<NT>(P, D, tm, sh, it, restarts, rel);
            break;
        }
    }
    finish_job(P, m, D, tm, sh, status, it, reps, fallback, rel);
}

template <bool MIXED, int NT>
__device__ __forceinline__ void solve_job(const BatchParams &P, int m, Team &tm, TeamShared &sh)
{
    if (MIXED && !(P.force64 && P.force64[m]))
        solve_mixed<NT>(P, m, tm, sh);
    else
        solve_fp64<NT>(P, m, tm, sh, MIXED ? 2 : 0);
}

template <bool MIXED, int NT>
__global__ void __launch_bounds__(NT, 1) k_batch_cg(const __grid_constant__ BatchParams P)
{
    __shared__ TeamShared sh;
    if (P.cluster > 1) {
        // team phases: the cluster takes jobs together, then its halves, ...
        cg::cluster_group cl = cg::this_cluster();
        const int me = (int)cl.block_rank();
        if (threadIdx.x == 0) {
            sh.lost = sh.gone = 0;
            sh.limit = P.wait_limit;
            for (int l = 0; l < kTeamSizes; ++l)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(&sh.bar[l])),
                             "r"(kMaxTeam >> l)
                             : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        cl.sync();
        int first = 0;
        for (int l = 0; l < kTeamSizes; first += P.n_team[l++]) {
            const int size = kMaxTeam >> l;
            if (P.n_team[l] == 0) continue;
            Team tm{me % size, size, me / size * size, size == P.cluster, l, 0, 0};
            // (a job that is taken by a team which then loses a CTA keeps the record
            // that every job starts with, PFG_E_INTERNAL; a lost CTA takes none)
            for (;;) {
                if (tm.rank == 0 && threadIdx.x == 0)
                    sh.job = *(volatile int *)&sh.lost ? P.n_team[l] : (int)atomicAdd(P.queue + l, 1u);
                if (!team_barrier(tm, sh)) break;
                const int job = *cl.map_shared_rank(&sh.job, tm.base);
                // every CTA has read the job before rank 0 overwrites it
                if (!team_barrier(tm, sh) || job >= P.n_team[l]) break;
                tm.nred = 0;
                solve_job<MIXED, NT>(P, P.order[first + job], tm, sh);
            }
        }
    }
    // single-CTA phase
    int n_solo = P.n_total, solo0 = 0;
    for (int l = 0; l < kTeamSizes; ++l) solo0 += P.n_team[l];
    n_solo -= solo0;
    for (;;) {
        if (threadIdx.x == 0) sh.job = (int)atomicAdd(P.queue + kTeamSizes, 1u);
        __syncthreads();
        const int job = sh.job;
        __syncthreads();
        if (job >= n_solo) break;
        Team tm{0, 1, 0, false, 0, 0, 0};
        solve_job<MIXED, NT>(P, P.order[solo0 + job], tm, sh);
    }
    // no CTA of a cluster leaves while another may still reach its shared memory
    if (P.cluster > 1) cg::this_cluster().sync();
}

}  // namespace
}  // namespace pfg

// ------------------------------------------------------------------ host side
namespace pfg {
namespace {

const void *batch_kernel(bool mixed, int threads)
{
    if (mixed) {
        if (threads == 256) return (const void *)k_batch_cg<true, 256>;
        if (threads == 512) return (const void *)k_batch_cg<true, 512>;
        return (const void *)k_batch_cg<true, 1024>;
    }
    if (threads == 256) return (const void *)k_batch_cg<false, 256>;
    if (threads == 512) return (const void *)k_batch_cg<false, 512>;
    return (const void *)k_batch_cg<false, 1024>;
}

int device_sms()
{
    int dev = 0, n = 0;
    PFG_CUDA(cudaGetDevice(&dev));
    PFG_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    return n;
}

void fill_launch(cudaLaunchConfig_t &lc, cudaLaunchAttribute &attr, int grid, int threads, int cluster,
                 cudaStream_t st)
{
    memset(&lc, 0, sizeof(lc));
    lc.gridDim = dim3((unsigned)grid, 1, 1);
    lc.blockDim = dim3((unsigned)threads, 1, 1);
    lc.dynamicSmemBytes = 0;
    lc.stream = st;
    lc.attrs = nullptr;
    lc.numAttrs = 0;
    if (cluster > 1) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)cluster;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        lc.attrs = &attr;
        lc.numAttrs = 1;
    }
}

// Persistent grid: as many CTAs (or clusters) as can be resident at once.
int persistent_grid(bool mixed, int threads, int cluster)
{
    const void *fn = batch_kernel(mixed, threads);
    const int sms = device_sms();
    if (cluster <= 1) {
        int per_sm = 0;
        PFG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0));
        return std::max(per_sm, 0) * sms;
    }
    cudaLaunchConfig_t lc;
    cudaLaunchAttribute attr;
    fill_launch(lc, attr, cluster * sms, threads, cluster, nullptr);
    int clusters = 0;
    PFG_CUDA(cudaOccupancyMaxActiveClusters(&clusters, fn, &lc));
    return std::max(clusters, 0) * cluster;
}

bool valid_config(const pfg_batch_config &c)
{
    return (c.threads == 256 || c.threads == 512 || c.threads == 1024) &&
           (c.cluster == 1 || c.cluster == 2 || c.cluster == 4 || c.cluster == 8) && c.team_fraction >= 0.0 &&
           c.team_fraction <= 1.0;
}

uint64_t mix(uint64_t h, uint64_t v)
{
    h ^= v + 0x9e3779b97f4a7c15ULL + (h << 6) + (h >> 2);
    return h;
}

}  // namespace
}  // namespace pfg

using namespace pfg;

struct pfg_batch {
    std::mutex mu;
    int device = 0;
    cudaStream_t st = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    std::vector<pfg_solver *> handles;
    std::vector<BatchSource> src;
    std::vector<int64_t> ndof, off;   // DOF of each system and its offset in the pooled vectors
    int64_t total = 0;                // pooled length (each system padded to 32 values)
    DevBuf<double> v64;               // x | r | p | q | z | s, `total` values each
    DevBuf<float> v32;                // x32 | r32 | p32 | q32 | z32
    DevBuf<double> d64;               // block-Jacobi inverses, 3 * total
    DevBuf<float> d32;
    int dinv_kind = -1;               // preconditioner the inverses hold
    DevBuf<BatchMesh> meshes;
    DevBuf<BatchOut> out;
    DevBuf<BatchOut> unsolved;        // what `out` holds until a system has been solved
    long long wait_limit = 1ll << 32; // clock cycles (about two seconds)
    DevBuf<int> order;
    DevBuf<unsigned> queue;
    std::vector<double> work;         // matrix blocks of each system (work per iteration)
    std::vector<int> last_iters;      // iterations of the previous solve (0: none yet)
    std::vector<int> iters64;         // iterations of the last FP64 solve of each system (0: none)
    std::vector<uint8_t> force64;     // mixed: systems to solve in FP64 (learned)
    DevBuf<uint8_t> force64_d;
    pfg_batch_config cfg{512, 4, 0.25};
    bool tuned = false;
    int *abort_h = nullptr;           // host-mapped abort flag
    int *abort_d = nullptr;
    cudaGraphExec_t graph = nullptr;
    uint64_t graph_key = 0;
    std::vector<BatchOut> out_h;

    ~pfg_batch()
    {
        if (graph) cudaGraphExecDestroy(graph);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (abort_h) cudaFreeHost(abort_h);
        if (st) cudaStreamDestroy(st);
    }
};

namespace {


void need(bool c, int code, const char *msg)
{
    if (!c) throw Error(code, msg);
}

struct RunSpec {
    bool mixed;
    int precond, itrmax;
    double tol, delta;
    int debug;
};

RunSpec run_spec(const pfg_solve_opts *opts)
{
    pfg_solve_opts o;
    if (opts)
        o = *opts;
    else {
        pfg_solve_opts_default(&o);
        o.algorithm = PFG_ALG_CG;
        o.precision = PFG_PREC_MIXED;
        o.precond = PFG_PC_BLOCK_JACOBI;
    }
    need(o.algorithm == PFG_ALG_CG, PFG_E_UNSUPPORTED,
         "batched solves run CG (the bound systems are symmetric positive definite)");
    need(o.precision == PFG_PREC_FP64 || o.precision == PFG_PREC_MIXED, PFG_E_ARG, "precision");
    need(o.precond == PFG_PC_NONE || o.precond == PFG_PC_JACOBI || o.precond == PFG_PC_BLOCK_JACOBI, PFG_E_ARG,
         "precond");
    need(o.itrmax > 0 && o.relative_er > 0.0, PFG_E_ARG, "itrmax and relative_er must be positive");
    need(o.reliable_delta > 0.0 && o.reliable_delta < 1.0, PFG_E_ARG, "reliable_delta must lie in (0, 1)");
    return RunSpec{o.precision == PFG_PREC_MIXED, o.precond, o.itrmax, o.relative_er, o.reliable_delta, o.debug};
}

struct TeamPlan {
    int cluster, grid;
    int n[kTeamSizes];  // systems, in the job order, for teams of 8, 4 and 2 CTAs
};

// Team sizes.  The n_team largest systems get a whole cluster; a system that would keep
// its team busy for more than `limit` of the balanced time (all costs over all
// CTAs) gets the next larger team, since one long system bounds the whole solve
// otherwise.  A team's CTAs keep at least a slice for each quarter of the SM (FP64)
// or each of sixteen warps (mixed, where the barriers weigh more).  No system gets a
// larger team than a costlier one: the job order lists the sizes in turn.
TeamPlan teams_within(const pfg_batch *b, const RunSpec &rs, const pfg_batch_config &c, const std::vector<int> &ord,
                      const std::vector<double> &cost, double total, int n_team, int cluster, int grid, double limit)
{
    TeamPlan p{cluster, grid, {}};
    int last = kMaxTeam;
    for (size_t k = 0; k < ord.size(); ++k) {
        const int m = ord[k];
        int size = (int)k < n_team ? c.cluster : 1;
        while (size < cluster && cost[m] > limit * size * total / grid &&
               b->ndof[m] >= (int64_t)2 * size * (rs.mixed ? 16 : 4) * 96)
            size *= 2;
        last = size = std::min(size, last);
        if (size == 1) break;
        for (int l = 0; l < kTeamSizes; ++l)
            if (size == kMaxTeam >> l) ++p.n[l];
    }
    return p;
}

// Time of a plan when every queue's jobs go to the team that is free first, as on the
// device.  An iteration in microseconds, fitted to 6, 11, 19, 37, 79 and 211 slices on
// 1, 2, 4 and 8 CTAs (FP64: the slices of the busiest quarter of an SM, and a
// cluster's barriers; larger teams up to 9 % more, as the odd slices' warps run alone).
double plan_time(const pfg_batch *b, const RunSpec &rs, const std::vector<int> &ord, const TeamPlan &p)
{
    std::vector<double> free_at((size_t)p.grid / p.cluster, 0.0);
    size_t k = 0;
    for (int size = p.cluster; size >= 1; size /= 2) {
        size_t n = ord.size() - k;
        for (int l = 0; l < kTeamSizes; ++l)
            if (size == kMaxTeam >> l) n = (size_t)p.n[l];
        std::make_heap(free_at.begin(), free_at.end(), std::greater<double>());
        for (size_t j = 0; j < n; ++j, ++k) {
            const int m = ord[k];
            const double ns = std::ceil((double)b->ndof[m] / 96.0);
            const bool f64 = !rs.mixed || b->force64[m];
            const double width = 3.0 * b->work[m] / (double)b->ndof[m];  // blocks in a row
            const double us = f64 ? (0.31 * width + 0.9) * std::ceil(ns / (4.0 * size)) + (size > 1 ? 5.0 : 1.0)
                                  : 1.65 * ns / (4.0 * size) + (size > 1 ? 8.0 : 4.5);
            std::pop_heap(free_at.begin(), free_at.end(), std::greater<double>());
            free_at.back() += (size > 2 ? 1.05 * us : us) * b->last_iters[m];
            std::push_heap(free_at.begin(), free_at.end(), std::greater<double>());
        }
        if (size > 1) {  // each team splits in two
            const size_t teams = free_at.size();
            free_at.resize(2 * teams);
            std::copy(free_at.begin(), free_at.begin() + teams, free_at.begin() + teams);
        }
    }
    return *std::max_element(free_at.begin(), free_at.end());
}

// The limit.  256 uneven slabs in pairs and single CTAs are 125 ms of FP64 work per SM
// and took 220 ms, the longest pair's time.  Limits of 0.5, 0.7, 0.85, 1.0 and 1.15 gave
// 181, 179, 181, 174 and 162 ms, and 179, 198, 203, 203 and 203 in clusters of four, so
// once a solve has counted the iterations the one of the shortest plan is taken (163-170
// ms); in a first solve, with costs guessed, 0.5 (291 -> 218 ms; 1.15 is the longest
// pair's time again).  Clusters of four fill 144 of the 152 SMs, of eight 120: pairs may
// grow to fours, for a first solve only if the longest clearly needs it, and
// fours don't grow.  Many systems for each CTA balance by themselves: no plans compared.
TeamPlan plan_teams(const pfg_batch *b, const RunSpec &rs, const pfg_batch_config &c, const std::vector<int> &ord,
                    const std::vector<double> &cost, int n_team, int grid)
{
    constexpr double kGuessed = 0.5, kWider = 0.9;
    const double total = std::accumulate(cost.begin(), cost.end(), 0.0);
    const int wider = c.cluster == 2 ? persistent_grid(rs.mixed, c.threads, 4) : 0;
    const bool known = std::all_of(b->last_iters.begin(), b->last_iters.end(), [](int it) { return it > 0; });
    if (!known || ord.size() > (size_t)16 * grid) {
        const bool wide = wider > 0 && cost[ord[0]] > kWider * 2 * total / grid;
        return teams_within(b, rs, c, ord, cost, total, n_team, wide ? 4 : c.cluster, wide ? wider : grid, kGuessed);
    }
    // (small systems in number give one plan, or a pair, whatever the limit: each is timed
    // once, which takes 30 us for 2,400 systems, all 26 took 0.8 ms of the solve's 11)
    std::vector<TeamPlan> plans;
    for (int cluster : {c.cluster, 4}) {
        if (cluster != c.cluster && wider <= 0) continue;
        for (double limit = 0.4; limit < 1.65; limit += 0.1) {
            const TeamPlan p = teams_within(b, rs, c, ord, cost, total, n_team, cluster,
                                            cluster == c.cluster ? grid : wider, limit);
            const bool seen = std::any_of(plans.begin(), plans.end(), [&](const TeamPlan &q) {
                return q.cluster == p.cluster && std::equal(p.n, p.n + kTeamSizes, q.n);
            });
            if (!seen) plans.push_back(p);
        }
        if (c.cluster == 4) break;
    }
    if (plans.size() == 1) return plans[0];
    size_t best = 0;
    double best_time = 0.0;
    for (size_t k = 0; k < plans.size(); ++k) {
        const double t = plan_time(b, rs, ord, plans[k]);
        if (k == 0 || t < best_time) {
            best = k;
            best_time = t;
        }
    }
    return plans[best];
}

// Launches one batched solve with configuration c (graph replay when the
// captured one matches); returns the device milliseconds of the launch.
double run_batch(pfg_batch *b, const RunSpec &rs, const pfg_batch_config &c)
{
    const int count = (int)b->src.size();
    // block-Jacobi inverses for the requested preconditioner
    if (rs.precond != PFG_PC_NONE && b->dinv_kind != rs.precond) {
        for (int m = 0; m < count; ++m)
            block_jacobi(*b->src[m].K, rs.precond, b->d64.p + 3 * b->off[m], b->d32.p + 3 * b->off[m], b->st);
        b->dinv_kind = rs.precond;
    }
    // longest estimated work first: blocks x iterations (previous solve, else sqrt of the rows)
    std::vector<int> ord((size_t)count);
    std::iota(ord.begin(), ord.end(), 0);
    std::vector<double> cost((size_t)count);
    for (int m = 0; m < count; ++m) {
        const double it = b->last_iters[m] > 0 ? (double)b->last_iters[m] : std::sqrt((double)b->ndof[m]);
        cost[m] = b->work[m] * it;
    }
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int d) { return cost[a] > cost[d]; });
    PFG_CUDA(cudaMemcpyAsync(b->order.p, ord.data(), count * sizeof(int), cudaMemcpyHostToDevice, b->st));
    int n_team = 0;
    if (c.cluster > 1) n_team = std::min(count, (int)std::lround(c.team_fraction * count));
    int cluster = c.cluster;
    int grid = persistent_grid(rs.mixed, c.threads, cluster);
    need(grid > 0, PFG_E_UNSUPPORTED, "batched kernel configuration cannot be resident on this GPU");
    TeamPlan plan{cluster, grid, {}};
    if (n_team > 0) plan = plan_teams(b, rs, c, ord, cost, n_team, grid);
    cluster = plan.cluster;
    grid = plan.grid;

    BatchParams P;
    P.mesh = b->meshes.p;
    P.out = b->out.p;
    P.order = b->order.p;
    std::copy(plan.n, plan.n + kTeamSizes, P.n_team);
    P.n_total = count;
    P.cluster = cluster;
    P.queue = b->queue.p;
    P.precond = rs.precond;
    P.itrmax = rs.itrmax;
    P.max_restarts = 5;
    P.tol = rs.tol;
    P.delta = rs.delta;
    P.abort = b->abort_d;
    P.wait_limit = b->wait_limit;
    P.force64 = rs.mixed ? b->force64_d.p : nullptr;
    if (rs.mixed)
        PFG_CUDA(cudaMemcpyAsync(b->force64_d.p, b->force64.data(), count, cudaMemcpyHostToDevice, b->st));

    uint64_t key = 0x51ab;
    for (uint64_t v : {(uint64_t)rs.mixed, (uint64_t)rs.precond, (uint64_t)rs.itrmax, (uint64_t)c.threads,
                       (uint64_t)cluster, (uint64_t)plan.n[0], (uint64_t)plan.n[1], (uint64_t)plan.n[2], (uint64_t)count, (uint64_t)grid,
                       (uint64_t)(uintptr_t)b->meshes.p, (uint64_t)(uintptr_t)b->v64.p,
                       (uint64_t)(uintptr_t)b->abort_d, (uint64_t)(uintptr_t)b->force64_d.p,
                       (uint64_t)b->wait_limit})
        key = mix(key, v);
    uint64_t tb, db;
    memcpy(&tb, &rs.tol, 8);
    memcpy(&db, &rs.delta, 8);
    key = mix(mix(key, tb), db);
    if (!b->graph || b->graph_key != key) {
        if (b->graph) cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
        cudaGraph_t g;
        PFG_CUDA(cudaStreamBeginCapture(b->st, cudaStreamCaptureModeThreadLocal));
        // x0 = 0 and the record of an unsolved system for every system, empty job
        // queues, then the persistent kernel
        cudaMemsetAsync(b->v64.p, 0, b->total * sizeof(double), b->st);
        cudaMemcpyAsync(b->out.p, b->unsolved.p, count * sizeof(BatchOut), cudaMemcpyDeviceToDevice, b->st);
        cudaMemsetAsync(b->queue.p, 0, (kTeamSizes + 1) * sizeof(unsigned), b->st);
        cudaLaunchConfig_t lc;
        cudaLaunchAttribute attr;
        fill_launch(lc, attr, grid, c.threads, cluster, b->st);
        void *args[] = {&P};
        const cudaError_t le = cudaLaunchKernelExC(&lc, batch_kernel(rs.mixed, c.threads), args);
        const cudaError_t ce = cudaStreamEndCapture(b->st, &g);
        PFG_CUDA(le);
        PFG_CUDA(ce);
        const cudaError_t ie = cudaGraphInstantiate(&b->graph, g, 0);
        cudaGraphDestroy(g);
        PFG_CUDA(ie);
        b->graph_key = key;
    }
    PFG_CUDA(cudaEventRecord(b->e0, b->st));
    PFG_CUDA(cudaGraphLaunch(b->graph, b->st));
    PFG_CUDA(cudaEventRecord(b->e1, b->st));
    b->out_h.resize((size_t)count);
    PFG_CUDA(cudaMemcpyAsync(b->out_h.data(), b->out.p, count * sizeof(BatchOut), cudaMemcpyDeviceToHost, b->st));
    PFG_CUDA(cudaStreamSynchronize(b->st));
    PFG_CUDA(cudaGetLastError());
    float ms = 0.f;
    PFG_CUDA(cudaEventElapsedTime(&ms, b->e0, b->e1));
    for (int m = 0; m < count; ++m) {
        const BatchOut &o = b->out_h[m];
        if (o.status == PFG_E_INTERNAL) continue;
        b->last_iters[m] = std::max(o.iterations, 1);
        if (!rs.mixed || o.fallback == 2) {
            if (o.status == PFG_OK) b->iters64[m] = o.iterations;
        } else if (o.fallback == 1) {
            b->force64[m] = 1;  // the FP32 operator failed on this system
        } else if (b->iters64[m] > 0 && o.iterations > 3 * b->iters64[m] / 2) {
            b->force64[m] = 1;  // FP32 needs 1.5x the FP64 iterations: no gain
        }
    }
    return (double)ms;
}

}  // namespace

extern "C" {

int pfg_batch_create(pfg_batch **out)
{
    return guard([&] {
        need(out != nullptr, PFG_E_ARG, "NULL batch pointer");
        pfg_batch *b = new pfg_batch();
        try {
            PFG_CUDA(cudaGetDevice(&b->device));
            PFG_CUDA(cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking));
            PFG_CUDA(cudaEventCreate(&b->e0));
            PFG_CUDA(cudaEventCreate(&b->e1));
            PFG_CUDA(cudaHostAlloc((void **)&b->abort_h, sizeof(int), cudaHostAllocMapped));
            *b->abort_h = 0;
            PFG_CUDA(cudaHostGetDevicePointer((void **)&b->abort_d, b->abort_h, 0));
            b->queue.alloc(kTeamSizes + 1);
        } catch (...) {
            delete b;
            throw;
        }
        *out = b;
    });
}

int pfg_batch_destroy(pfg_batch *b)
{
    return guard([&] {
        if (!b) return;
        {
            std::lock_guard<std::mutex> lk(b->mu);
            if (b->st) cudaStreamSynchronize(b->st);
        }
        delete b;
    });
}

int pfg_batch_set(pfg_batch *b, int64_t count, pfg_solver *const *handles)
{
    return guard([&] {
        need(b && handles && count > 0, PFG_E_ARG, "batch, handles and count > 0 required");
        need(count <= (int64_t)1 << 24, PFG_E_ARG, "too many systems in one batch");
        std::lock_guard<std::mutex> lk(b->mu);
        int dev = 0;
        PFG_CUDA(cudaGetDevice(&dev));
        need(dev == b->device, PFG_E_STATE, "batch used on another device than it was created on");
        std::vector<BatchSource> src((size_t)count);
        for (int64_t m = 0; m < count; ++m) {
            src[m] = batch_bind(handles[m]);
            need(src[m].device == b->device, PFG_E_ARG, "batch member on another device");
        }
        b->handles.assign(handles, handles + count);
        b->src = std::move(src);
        b->ndof.resize((size_t)count);
        b->off.resize((size_t)count);
        b->work.resize((size_t)count);
        b->last_iters.assign((size_t)count, 0);
        b->iters64.assign((size_t)count, 0);
        b->force64.assign((size_t)count, 0);
        b->force64_d.resize((size_t)count);
        int64_t tot = 0;
        for (int64_t m = 0; m < count; ++m) {
            const DevMatrix &K = *b->src[m].K;
            b->ndof[m] = K.ndof();
            b->off[m] = tot;
            b->work[m] = (double)K.nnzb;
            tot += (K.ndof() + 31) / 32 * 32;
        }
        b->total = tot;
        b->v64.resize((size_t)tot * 6);
        b->v32.resize((size_t)tot * 5);
        b->d64.resize((size_t)tot * 3);
        b->d32.resize((size_t)tot * 3);
        b->dinv_kind = -1;
        std::vector<BatchMesh> hm((size_t)count);
        for (int64_t m = 0; m < count; ++m) {
            const BatchSource &s = b->src[m];
            BatchMesh &d = hm[m];
            const int64_t o = b->off[m];
            d.A64 = s.K->sell<double>();
            d.A32 = s.K->sell<float>();
            d.b = s.b;
            d.fixed = s.fixed;
            d.fixval = s.fixval;
            d.x = b->v64.p + o;
            d.r64 = b->v64.p + tot + o;
            d.p64 = b->v64.p + 2 * tot + o;
            d.q64 = b->v64.p + 3 * tot + o;
            d.z64 = b->v64.p + 4 * tot + o;
            d.s64 = b->v64.p + 5 * tot + o;
            d.x32 = b->v32.p + o;
            d.r32 = b->v32.p + tot + o;
            d.p32 = b->v32.p + 2 * tot + o;
            d.q32 = b->v32.p + 3 * tot + o;
            d.z32 = b->v32.p + 4 * tot + o;
            d.dinv64 = b->d64.p + 3 * o;
            d.dinv32 = b->d32.p + 3 * o;
        }
        b->meshes.resize((size_t)count);
        b->out.resize((size_t)count);
        b->unsolved.resize((size_t)count);
        b->order.resize((size_t)count);
        PFG_CUDA(cudaMemcpyAsync(b->meshes.p, hm.data(), count * sizeof(BatchMesh), cudaMemcpyHostToDevice, b->st));
        BatchOut none{};
        none.status = PFG_E_INTERNAL;
        none.rel_residual = 1.0;  // of x = 0
        const std::vector<BatchOut> ho((size_t)count, none);
        PFG_CUDA(cudaMemcpyAsync(b->unsolved.p, ho.data(), count * sizeof(BatchOut), cudaMemcpyHostToDevice, b->st));
        PFG_CUDA(cudaStreamSynchronize(b->st));
        if (b->graph) cudaGraphExecDestroy(b->graph);
        b->graph = nullptr;
    });
}

int pfg_batch_set_config(pfg_batch *b, const pfg_batch_config *cfg)
{
    return guard([&] {
        need(b && cfg, PFG_E_ARG, "NULL argument");
        need(valid_config(*cfg), PFG_E_ARG, "threads 256/512/1024, cluster 1/2/4/8, team_fraction in [0, 1]");
        std::lock_guard<std::mutex> lk(b->mu);
        b->cfg = *cfg;
    });
}

int pfg_batch_get_config(pfg_batch *b, pfg_batch_config *cfg, int32_t *tuned)
{
    return guard([&] {
        need(b && cfg, PFG_E_ARG, "NULL argument");
        std::lock_guard<std::mutex> lk(b->mu);
        *cfg = b->cfg;
        if (tuned) *tuned = b->tuned ? 1 : 0;
    });
}

int pfg_batch_solve(pfg_batch *b, const pfg_solve_opts *opts, double *const *x_out, pfg_info *infos,
                    pfg_batch_info *binfo)
{
    int worst = PFG_OK;
    const int rc = guard([&] {
        need(b != nullptr, PFG_E_ARG, "NULL batch");
        std::lock_guard<std::mutex> lk(b->mu);
        need(!b->src.empty(), PFG_E_STATE, "solve before pfg_batch_set");
        const RunSpec rs = run_spec(opts);
        const double ms = run_batch(b, rs, b->cfg);
        const int count = (int)b->src.size();
        int64_t tot_it = 0;
        int max_it = 0, fallbacks = 0;
        double max_rel = 0.0;
        for (int m = 0; m < count; ++m) {
            const BatchOut &o = b->out_h[m];
            if (x_out && x_out[m])
                PFG_CUDA(cudaMemcpyAsync(x_out[m], b->v64.p + b->off[m], b->ndof[m] * sizeof(double),
                                         cudaMemcpyDeviceToHost, b->st));
            if (infos) {
                pfg_info &in = infos[m];
                memset(&in, 0, sizeof(in));
                in.status = o.status;
                in.iterations = o.iterations;
                in.replacements = o.replacements;
                in.kernel_launches = 1;
                in.rel_residual = o.rel_residual;
                in.iter_residual = o.rel_residual;
                in.solve_ms = ms;
                in.fallback = o.fallback;
            }
            tot_it += o.iterations;
            max_it = std::max(max_it, o.iterations);
            max_rel = std::max(max_rel, o.rel_residual);
            fallbacks += o.fallback != 0;
            if (o.status < 0 && (worst >= 0)) worst = o.status;
            if (o.status > 0 && worst == PFG_OK) worst = o.status;
        }
        PFG_CUDA(cudaStreamSynchronize(b->st));
        if (binfo) {
            memset(binfo, 0, sizeof(*binfo));
            binfo->config = b->cfg;
            binfo->launches = 1;
            binfo->max_iterations = max_it;
            binfo->total_iterations = tot_it;
            binfo->max_rel_residual = max_rel;
            binfo->solve_ms = ms;
            binfo->fallbacks = fallbacks;
        }
        if (worst < 0) {
            set_last_error("a batched system ended with status " + std::to_string(worst));
        }
    });
    if (rc != PFG_OK) return rc;
    return worst;
}

int pfg_batch_get_x(pfg_batch *b, int64_t index, double *x_out)
{
    return guard([&] {
        need(b && x_out, PFG_E_ARG, "NULL argument");
        std::lock_guard<std::mutex> lk(b->mu);
        need(index >= 0 && index < (int64_t)b->src.size(), PFG_E_ARG, "index out of range");
        PFG_CUDA(cudaMemcpyAsync(x_out, b->v64.p + b->off[index], b->ndof[index] * sizeof(double),
                                 cudaMemcpyDeviceToHost, b->st));
        PFG_CUDA(cudaStreamSynchronize(b->st));
    });
}

int pfg_batch_tune(pfg_batch *b, const pfg_solve_opts *opts, pfg_batch_config *best, double *best_ms)
{
    return guard([&] {
        need(b != nullptr, PFG_E_ARG, "NULL batch");
        std::lock_guard<std::mutex> lk(b->mu);
        need(!b->src.empty(), PFG_E_STATE, "tune before pfg_batch_set");
        const RunSpec rs = run_spec(opts);
        // one untimed solve fills the iteration counts the job order uses
        run_batch(b, rs, b->cfg);
        pfg_batch_config cur = b->cfg, top = b->cfg;
        double top_ms = 1e300;
        auto trial = [&](const pfg_batch_config &c) {
            if (!valid_config(c)) return;
            if (persistent_grid(rs.mixed, c.threads, c.cluster) <= 0) return;
            const double ms = run_batch(b, rs, c);
            if (rs.debug)
                fprintf(stderr, "[pfg] batch tune: threads %d cluster %d team share %.4f: %.2f ms\n", c.threads,
                        c.cluster, c.team_fraction, ms);
            if (ms < top_ms) {
                top_ms = ms;
                top = c;
            }
        };
        // stage 1: CTA size (block rows per CTA tile) x team size; stage 2: team share
        for (int nt : {256, 512, 1024})
            for (int cl : {1, 2, 4, 8}) {
                pfg_batch_config c = cur;
                c.threads = nt;
                c.cluster = cl;
                c.team_fraction = cl > 1 ? 0.125 : 0.0;
                trial(c);
            }
        cur = top;
        if (cur.cluster > 1)
            for (double f : {0.0625, 0.25, 0.5, 1.0}) {
                pfg_batch_config c = cur;
                c.team_fraction = f;
                trial(c);
            }
        b->cfg = top;
        b->tuned = true;
        if (best) *best = top;
        if (best_ms) *best_ms = top_ms;
    });
}

int pfg_batch_set_wait_limit(pfg_batch *b, int64_t cycles)
{
    return guard([&] {
        need(b != nullptr, PFG_E_ARG, "NULL batch");
        std::lock_guard<std::mutex> lk(b->mu);
        b->wait_limit = cycles;
    });
}

int pfg_batch_abort_flag(pfg_batch *b, volatile int32_t **flag)
{
    return guard([&] {
        need(b && flag, PFG_E_ARG, "NULL argument");
        *flag = (volatile int32_t *)b->abort_h;
    });
}

}  // extern "C"
